"""The adaptive integrators' encounter and impact screens, one launch a step:
Big bodies at the edges of the block's shared tables (64 at a time), particle
counts at the edges of a block, massive Small bodies, no particles at all."""
import numpy as np
import pytest

from adaptive_cases import ALGORITHMS, compare_events, oracle_intervals, planar_body, run_intervals
from mercuda_b200.backend import Backend
from mercuda_b200.system import K2, System

pytestmark = pytest.mark.gpu


def crowded(nbig, count, massive):
    """A planet every few hundredths of an au, the Small bodies next to them
    and every 50th falling past the central body."""
    rng = np.random.default_rng(1000 * nbig + count)
    bodies = [(K2, [0.0] * 3, [0.0] * 3)]
    bodies += [planar_body(1e-9, 1.0 + 0.03 * k, 0.01, 0.4 * k) for k in range(nbig)]
    for j in range(count):
        _, x, v = bodies[1 + j % nbig]
        x, v = np.array(x) + rng.uniform(-0.03, 0.03, 3), np.array(v) * rng.uniform(0.9, 1.1, 3)
        if j % 50 == 7:
            x, v = x * 0.3, -x * rng.uniform(0.008, 0.012)
        bodies.append((1e-10 * K2 if massive and j % 3 == 0 else 0.0, list(x), list(v)))
    n = len(bodies)
    return System(m=np.array([b[0] for b in bodies]), x=np.array([b[1] for b in bodies]),
                  v=np.array([b[2] for b in bodies]), nbig=nbig + 1, ngf=np.zeros((n, 5)),
                  rce=np.full(n, 0.05), rphys=np.full(n, 1e-3))


@pytest.mark.parametrize("name", ["RADAU", "BS2"])
@pytest.mark.parametrize("nbig,count,massive", [(1, 1, False), (3, 0, False), (8, 127, True), (64, 128, False),
                                                (65, 129, False), (2, 400, True)])
def test_records(cuda_lib, oracle, name, nbig, count, massive):
    sys0 = crowded(nbig, count, massive)
    be = Backend(name, cuda_lib)
    be.configure()
    be.upload(sys0)
    got, _ = run_intervals(be, sys0.copy(), 0.0, 6.0, 6.0, 1.0, 1e-11, rcen=0.28)
    x, v = be.download()
    be.free()
    ref = sys0.copy()
    want, *_ = oracle_intervals(oracle, ref, ALGORITHMS[name], 0.0, 6.0, 6.0, 1.0, 1e-11, rcen=0.28)
    assert np.array_equal(x, ref.x) and np.array_equal(v, ref.v)
    assert count < 100 or {8} < {int(e["kind"]) for e in want}
    compare_events(got, want)
