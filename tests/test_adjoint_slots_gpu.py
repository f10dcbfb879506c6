"""The adjoint's slots: particle counts about a warp and a warp's share of slow
particles, all-slow and no-slow populations, more segments than record buffers.
Every particle's result is its own, so a run of many must equal runs of each
part bit for bit, and the final states those of the forward MVS run."""
import numpy as np
import pytest
import torch

from mercuda_b200.adjoint import mvs_trajectory
from mercuda_b200.system import make_system

pytestmark = pytest.mark.gpu


def run(s, rows, h, steps, every):
    nb = s.nbig
    t = [torch.tensor(a[rows], device="cuda", requires_grad=True) for a in (s.x[nb:], s.v[nb:], s.ngf[nb:, 4])]
    xf, vf = mvs_trajectory(*t, (s.m[:nb], s.x[:nb], s.v[:nb]), h, steps, every)
    g = torch.autograd.grad((xf ** 2).sum() + (vf ** 2).sum(), t)
    return [q.detach().cpu().numpy() for q in (xf, vf, *g)]


@pytest.mark.parametrize("count", [1, 7, 9, 33, 129])
@pytest.mark.parametrize("pe_max,pa", [(0.02, (2.0, 5.0)), (0.9, (0.4, 0.6)), (0.5, (0.5, 3.0))])
def test_slots_change_nothing(cuda_lib, oracle, count, pe_max, pa):
    s = make_system(seed=count, n_particles=count, nplanets=3, pe_max=pe_max, pa=pa)
    s.ngf[s.nbig:, 4] = 1e-14
    whole = run(s, slice(None), 8.0, 30, 4)
    for k in range(0, count, max(1, count // 3)):
        part = run(s, slice(k, k + 1), 8.0, 30, 4)
        assert all(np.array_equal(a[k:k + 1], b) for a, b in zip(whole, part))
    # 30 steps of the same map on the CPU: a few ulp of the drift's cosine,
    # amplified at most linearly along these short regular orbits
    ref = s.copy()
    oracle.mvs_run(ref, 0.0, 8.0, 30, 0.0)
    assert np.max(np.abs(whole[0] - ref.x[ref.nbig:])) <= 1e-9
