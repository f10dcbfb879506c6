"""How many steps a launch of the fused MVS run takes: 18 KB of force rows of
eight doubles a body, so 31 steps of eight planets and 56 of four, as a caller's
steps_per_launch and as the longest run whose copies overlap its steps."""
import numpy as np
import pytest
import torch

from mercuda_b200.backend import Backend
from mercuda_b200.system import make_system

pytestmark = pytest.mark.gpu


@pytest.fixture()
def backend(cuda_lib):
    b = Backend("MVS", lib=cuda_lib)
    b.configure()
    yield b
    b.free()


@pytest.mark.parametrize("planets,limit", [(8, 31), (4, 56), (1, 64)])
def test_steps_of_one_launch(backend, planets, limit):
    backend.upload(make_system(seed=planets, n_particles=100, nplanets=planets))
    for asked in (limit, limit + 5):
        backend.mvs_advance(0.0, 8.0, limit + 1, 0.005, steps_per_launch=asked)
        assert [k for k, _ in backend.advance_launches()] == [limit, 1]


def test_overlapped_run_of_the_longest_launch(backend):
    """Page-locked arrays, two parts of the particles, 31 steps: two particle
    launches, one a part, and the states of the three calls in turn."""
    s = make_system(seed=9, n_particles=270_000, near_fraction=0.01)
    pins = []

    def pinned(a):
        pins.append(torch.empty(a.shape, dtype=torch.float64, pin_memory=True))
        pins[-1].numpy()[...] = a
        return pins[-1].numpy()

    backend.upload(s)
    ev0, st0 = backend.mvs_advance(0.0, 8.0, 31, 0.005)
    x0, v0 = backend.download()
    for name in ("m", "x", "v", "ngf", "rce", "rphys", "rcrit"):
        setattr(s, name, pinned(getattr(s, name)))
    out = (pinned(np.zeros((s.n, 3))), pinned(np.zeros((s.n, 3))))
    ev, st, x, v = backend.mvs_run(s, 0.0, 8.0, 31, 0.005, out=out)
    assert backend.timing()["particle_launches"] == 2
    assert ev.tobytes() == ev0.tobytes() and np.array_equal(st, st0)
    assert np.array_equal(x, x0) and np.array_equal(v, v0)
