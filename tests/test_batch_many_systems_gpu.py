"""A batch whose step tables hold more than 2^31 doubles (1.9 million systems of
one planet, 64 steps a launch: 67 GB on the device)."""
import ctypes as C

import numpy as np
import pytest

from mercuda_b200.backend import PD, PI
from mercuda_b200.system import make_system

pytestmark = pytest.mark.gpu


def run(lib, n, m, x, v, steps):
    """The last states of n systems of a star and a planet."""
    f = lambda a: a.ctypes.data_as(PD)
    offsets = np.arange(n + 1, dtype=np.int32) * 2
    nbig = np.full(n, 2, dtype=np.int32)
    h = np.full(n, 8.0)
    r = np.zeros(2 * n)
    out = [np.zeros((2 * n, 3)) for _ in range(2)]
    nev = C.c_int(0)
    try:
        assert lib.mercury_b200_batch_upload(n, offsets.ctypes.data_as(PI), nbig.ctypes.data_as(PI), f(h), f(m), f(x),
                                             f(v), f(r), f(r)) == 0
        assert lib.mercury_b200_batch_advance(0.0, steps, 0.005, C.byref(nev)) == 0
        assert lib.mercury_b200_batch_download(f(out[0]), f(out[1])) == 0
    finally:
        lib.mercury_b200_batch_free()
    return out


def test_tables_beyond_32_bits(cuda_lib):
    n, few = 1_900_000, 1000
    systems = [make_system(seed=k, n_particles=0, nplanets=1) for k in range(few)]
    m, x, v = (np.concatenate([getattr(s, a) for s in systems]) for a in ("m", "x", "v"))
    cuda_lib.mercury_b200_batch_set(128, 64, -1)
    try:
        alone = run(cuda_lib, few, m, x, v, 64)
        many = run(cuda_lib, n, np.tile(m, n // few), np.tile(x, (n // few, 1)), np.tile(v, (n // few, 1)), 64)
    finally:
        cuda_lib.mercury_b200_batch_set(0, 0, -1)
    for a, b in zip(alone, many):
        assert not np.array_equal(a, np.zeros_like(a))
        assert np.array_equal(np.tile(a, (n // few, 1)), b)
