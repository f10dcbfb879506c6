"""Batches whose records, candidates or both outgrow the room their run starts
with: the run is made again with room, and every system's states and records
equal those of the system run alone."""
import numpy as np
import pytest

from mercuda_b200.backend import Backend, Batch
from mercuda_b200.system import make_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("near,steps", [(1.0, 16), (0.6, 40)])
def test_overflowing_batch(cuda_lib, near, steps, graph):
    """3 x 9,000 particles, near 1.0: every particle beside a planet of 1e-3
    masses, so 0.7 candidates a particle-step where 0.04 have room, and
    more records than the 4,096 that an upload makes room for."""
    kw = dict(near_fraction=near, nplanets=3, planet_kw=dict(mmin=1e-3, mmax=1e-3))
    systems = [make_system(seed=90 + k, n_particles=9000, **kw) for k in range(3)]
    h = np.array([8.0, 5.0, 11.0])
    cuda_lib.mercury_b200_batch_free()
    b = Batch(systems, h)
    b.set(threads=128, steps_per_launch=16, graph=graph)
    try:
        ev, sy, st = b.advance(0.0, steps, 0.005)
        ends = b.download()
    finally:
        b.set(threads=0, steps_per_launch=0, graph=1)
        b.free()
    assert len(ev) > 4096
    one = Backend("MVS", cuda_lib)
    one.configure()
    for k, s in enumerate(systems):
        one.upload(s)
        ev1, st1 = one.mvs_advance(0.0, float(h[k]), steps, 0.005)
        x1, v1 = one.download()
        assert np.array_equal(ends[k][0], x1) and np.array_equal(ends[k][1], v1)
        mine = sorted(zip(st[sy == k].tolist(), (e.tobytes() for e in ev[sy == k])))
        assert mine == sorted(zip(st1.tolist(), (e.tobytes() for e in ev1)))
    one.free()
