"""The batch's layout kernels: rows in and out at the edges of a block's share
of a system, one batch after a larger one, and a run whose records outgrow the
room it starts with."""
import numpy as np
import pytest

from mercuda_b200.backend import Batch
from mercuda_b200.system import make_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[1024, 0, 3], [1, 1015, 1016, 1017, 2040], [31, 32, 33, 5000], [7]])
def test_rows_round_trip(cuda_lib, sizes):
    systems = [make_system(seed=60 + k, n_particles=n, nplanets=1 + k % 8) for k, n in enumerate(sizes)]
    for s in systems:
        s.v[0] = 1e-5   # the central body's row comes back as it went in
    b = Batch(systems, np.full(len(systems), 8.0))
    try:
        for s, (x, v) in zip(systems, b.download()):
            assert np.array_equal(x, s.x) and np.array_equal(v, s.v)
    finally:
        b.free()


def test_smaller_batch_after_a_larger_one(cuda_lib):
    """The second run's states and records equal those of the batch alone."""
    big = [make_system(seed=70 + k, n_particles=900, near_fraction=0.1) for k in range(6)]
    small = [make_system(seed=80 + k, n_particles=40, near_fraction=0.5) for k in range(3)]
    h = np.array([8.0, 5.0, 11.0])

    def run():
        b = Batch(small, h)
        b.set(threads=128, steps_per_launch=8)
        ev = b.advance(0.0, 20, 0.005)
        return ev, b.download(), b

    (ev0, sy0, st0), ends0, b = run()
    b.free()
    b = Batch(big, np.full(6, 8.0))
    b.advance(0.0, 20, 0.005)
    (ev1, sy1, st1), ends1, b = run()
    b.free()
    assert ev0.tobytes() == ev1.tobytes() and np.array_equal(sy0, sy1) and np.array_equal(st0, st1)
    assert all(np.array_equal(p, q) for a, c in zip(ends0, ends1) for p, q in zip(a, c))
