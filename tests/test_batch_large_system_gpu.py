"""A batch with one system of more bodies than the layout kernel's blocks take
in one pass (1,024 blocks of 1,024 bodies): rows in and out."""
import numpy as np
import pytest

from mercuda_b200.backend import Batch
from mercuda_b200.system import make_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bodies", [1024 * 1024, 1024 * 1024 + 1, 2 * 1024 * 1024 + 1025])
def test_rows_of_a_large_system(cuda_lib, bodies):
    systems = [make_system(seed=1, n_particles=5, nplanets=2), make_system(seed=2, n_particles=bodies - 2, nplanets=1)]
    assert systems[1].n == bodies
    b = Batch(systems, np.full(2, 8.0))
    try:
        for s, (x, v) in zip(systems, b.download()):
            assert np.array_equal(x, s.x) and np.array_equal(v, s.v)
    finally:
        b.free()
