"""1/sqrt as IEEE division and square root round it, at the one operand of each
two binades where a residual correction alone does not: 4^k (1 - 2^-53), whose
root's significand is all ones. Bodies at such a squared distance from the
central body and from each other, through the force entry, bit for bit."""
import numpy as np
import pytest

from mercuda_b200.backend import Backend
from mercuda_b200.system import K2, System

pytestmark = pytest.mark.gpu


def norm2(d):
    return d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1] + d[..., 2] * d[..., 2]


def at_distance(rng, origin, s2):
    """A point whose rounded difference from `origin` has exactly the rounded square s2."""
    while True:
        u = rng.normal(size=3)
        x = origin + u / np.linalg.norm(u) * np.sqrt(s2)
        z = x[2] + np.spacing(x[2]) * np.arange(-40, 41)
        cand = np.column_stack([np.full(81, x[0]), np.full(81, x[1]), z])
        hit = np.flatnonzero(norm2(cand - origin) == s2)
        if len(hit):
            return cand[hit[0]]


def system():
    rng = np.random.default_rng(8)
    odd = [np.nextafter(4.0 ** k, 0.0) for k in (-2, -1, 0, 1, 2, 3)]
    zero = np.zeros(3)
    big = [zero, at_distance(rng, zero, odd[3])]
    big.append(at_distance(rng, big[1], odd[2]))      # a pair of Big bodies
    big.append(rng.normal(size=3) * 5)
    part = [at_distance(rng, c, s2) for s2 in odd for c in (zero, big[1], big[3]) for _ in range(8)]
    part += list(rng.normal(size=(16, 3)) * 3)
    x = np.array(big + part)
    n = len(x)
    m = np.zeros(n)
    m[:4] = K2 * np.array([1.0, 0.3, 0.01, 0.2])
    return System(m=m, x=x, v=np.zeros((n, 3)), nbig=4), odd


@pytest.mark.parametrize("algorithm", ["RADAU", "BS"])
def test_force_at_the_exception(cuda_lib, oracle, algorithm):
    s, odd = system()
    special = np.isin(norm2(s.x), odd) | np.isin(norm2(s.x - s.x[1]), odd) | np.isin(norm2(s.x - s.x[3]), odd)
    assert special[4:148].all() and special[1] and special[2]
    b = Backend(algorithm, cuda_lib)
    b.configure()
    try:
        b.upload(s)
        a = b.force()
    finally:
        b.free()
    want = oracle.force(s)
    assert np.array_equal(a[1:], want[1:])
