"""The room that a fused run's first launch makes for encounter candidates: a
system of 1M particles with box overlaps at 4.2 % a step is stepped once, not
made again with twice the room."""
import pytest
import torch

from mercuda_b200.backend import Backend
from mercuda_b200.system import make_system

pytestmark = pytest.mark.gpu


def held(lib, s):
    """Device memory that 30 steps (launches of 5 and 25) leave the library with."""
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    b = Backend("MVS", lib)
    b.configure()
    try:
        b.upload(s)
        b.mvs_advance(0.0, 8.0, 30, 0.005)
        assert [k for k, _ in b.advance_launches()] == [5, 25]
        return free0 - torch.cuda.mem_get_info()[0]
    finally:
        b.free()


def test_first_run_is_made_once(cuda_lib):
    systems = [make_system(seed=seed, n_particles=1_000_000, near_fraction=0.01) for seed in (1, 6)]
    held(cuda_lib, systems[0])
    calm = held(cuda_lib, make_system(seed=2, n_particles=1_000_000, near_fraction=0.0))
    for s in systems:
        assert held(cuda_lib, s) - calm < 64 << 20   # twice the room: 130 MB more
