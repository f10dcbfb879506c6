"""Calls on a device with little memory left: room that only makes a run faster
is not asked for, and the results do not depend on it. The sizes below leave
each call what it must have, and a quarter of that on top."""
import contextlib

import numpy as np
import pytest
import torch

from mercuda_b200.adjoint import mvs_trajectory
from mercuda_b200.backend import Batch
from mercuda_b200.system import make_system

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def little_room(lib, left):
    """The device with `left` bytes free, once the library holds nothing."""
    for free in ("mercury_cuda_free", "mercury_b200_batch_free", "mercury_b200_adjoint_free",
                 "mercury_b200_hybrid_adjoint_free"):
        getattr(lib, free)()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")
    try:
        assert torch.cuda.mem_get_info()[0] <= left
        yield
    finally:
        del held
        torch.cuda.empty_cache()


def test_adjoint_record_buffers(cuda_lib):
    """Four segments of 8 steps, 300,000 particles: 230 MB of records a segment;
    the same run with two record buffers as with four."""
    s = make_system(seed=3, n_particles=300_000, nplanets=2)
    nb = s.nbig
    t = [torch.tensor(a[nb:], device="cuda", requires_grad=True) for a in (s.x, s.v)]
    big = (s.m[:nb], s.x[:nb], s.v[:nb])

    def run():
        xf, vf = mvs_trajectory(*t, None, big, 8.0, 32, 8)
        g = torch.autograd.grad((xf ** 2).sum() + (vf ** 2).sum(), t)
        return [q.detach().cpu() for q in (xf, vf, *g)]

    cuda_lib.mercury_b200_adjoint_free()   # what an earlier test's run left
    torch.cuda.empty_cache()
    free0 = torch.cuda.mem_get_info()[0]
    roomy = run()
    assert free0 - torch.cuda.mem_get_info()[0] > 4 * 8 * 12 * 8 * 300_000
    needs = 300_000 * (2 * 8 * 12 * 8 + 4 * 76 + 10 * 8)
    with little_room(cuda_lib, int(1.25 * needs)):
        tight = run()
    assert all(torch.equal(a, b) for a, b in zip(roomy, tight))


def batch_run(systems, nsteps):
    b = Batch(systems, np.full(len(systems), 8.0))
    b.set(threads=128, steps_per_launch=64)
    ev, sy, st = b.advance(0.0, nsteps, 0.005)
    return ev.tobytes(), sy.tolist(), st.tolist(), b.download()


def test_batch_candidates(cuda_lib):
    """A million particles in four systems, 64 steps a launch: 302 bytes a
    particle is what an upload asks for, 2.56 candidates a particle (328 bytes)
    only a guess that saves making a run twice."""
    systems = [make_system(seed=20 + k, n_particles=250_000, nplanets=1) for k in range(4)]
    roomy = batch_run(systems, 64)
    with little_room(cuda_lib, int(1.25 * 302 * 1_000_000)):
        tight = batch_run(systems, 64)
        cuda_lib.mercury_b200_batch_free()
    cuda_lib.mercury_b200_batch_set(0, 0, -1)
    assert roomy[:3] == tight[:3]
    assert all(np.array_equal(p, q) for a, c in zip(roomy[3], tight[3]) for p, q in zip(a, c))


def test_large_batch_gives_way_to_a_small_one(cuda_lib):
    little = [make_system(seed=5, n_particles=1000, nplanets=1)]
    Batch(little, np.full(1, 8.0)).free()
    free0 = torch.cuda.mem_get_info()[0]
    Batch([make_system(seed=6, n_particles=500_000, nplanets=1)], np.full(1, 8.0))
    assert free0 - torch.cuda.mem_get_info()[0] > 500_000 * 302
    b = Batch(little, np.full(1, 8.0))
    assert free0 - torch.cuda.mem_get_info()[0] < 32 << 20
    b.free()
