"""Calls on a device with little memory left: room that only makes a run faster
is not asked for, and the results do not depend on it. The sizes below leave
each call what it must have, and a quarter of that on top."""
import contextlib

import pytest
import torch

from mercuda_b200.adjoint import mvs_trajectory
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

    free0 = torch.cuda.mem_get_info()[0]
    roomy = run()
    assert free0 - torch.cuda.mem_get_info()[0] > 4 * 8 * 12 * 8 * 300_000
    needs = 300_000 * (2 * 8 * 12 * 8 + 4 * 76 + 10 * 8)
    with little_room(cuda_lib, int(1.25 * needs)):
        tight = run()
    assert all(torch.equal(a, b) for a, b in zip(roomy, tight))
