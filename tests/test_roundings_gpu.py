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


def hard_numerators(b, most=41):
    """For each divisor b a numerator of 53 bits whose quotient lies within
    `most` parts of 2^53 half ulps of the middle of two doubles: A 2^j = B M + d
    with the divisor's significand B, an odd M of 54 bits and a small d."""
    out = np.zeros(len(b))
    for i, q in enumerate(b):
        B = int(np.ldexp(np.frexp(q)[0], 53))
        B >>= (B & -B).bit_length() - 1
        for d in sorted(range(-most, most + 1), key=abs):
            j = 53 + (d & 1)
            M = -d * pow(B, -1, 1 << j) % (1 << j) if d else 0
            A = (B * M + d) >> j
            if d and M % 2 and M >> 53 == 1 and 0 < A < 1 << 53:
                out[i] = float(A)
                break
    return out


@pytest.mark.parametrize("term", ["yar", "pr"])
def test_quotients_next_to_a_middle(cuda_lib, oracle, term):
    """Radiation forces whose coefficient makes the quotient of the force law
    (yar / (r^2 |t|), K2 beta / (r r)) as hard to round as can be; the central
    mass is small enough to leave them alone in the sum."""
    rng = np.random.default_rng(12)
    n = 6000
    x = np.vstack([np.zeros(3), rng.normal(size=(n, 3)) * 2])
    v = np.vstack([np.zeros(3), rng.normal(size=(n, 3)) * 0.01])
    ngf = np.zeros((n + 1, 5))
    r2 = norm2(x[1:])
    if term == "yar":
        q = (x[1:, 0] * v[1:, 0] + x[1:, 1] * v[1:, 1] + x[1:, 2] * v[1:, 2]) / r2
        t = v[1:] - q[:, None] * x[1:]
        a = hard_numerators(r2 * np.sqrt(norm2(t)))
        ngf[1:, 4] = np.ldexp(a, -60)
    else:
        r = np.sqrt(r2)
        a = np.ldexp(hard_numerators(r * r), -70)
        beta = a / K2
        for step in (-1, 1):     # a neighbour whose product with K2 is the numerator
            other = beta + step * np.spacing(beta)
            beta = np.where((K2 * beta != a) & (K2 * other == a), other, beta)
        ngf[1:, 3] = beta
    assert (a > 0).mean() > 0.9
    m = np.zeros(n + 1)
    m[0] = 1e-200
    s = System(m=m, x=x, v=v, ngf=ngf, nbig=1)
    b = Backend("RADAU", cuda_lib)
    b.configure()
    try:
        b.upload(s)
        got = b.force()
    finally:
        b.free()
    assert np.array_equal(got[1:], oracle.force(s)[1:])
