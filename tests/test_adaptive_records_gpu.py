"""The records of an adaptive step whose screens were queued with the step: more
of them than the page-locked head holds (1,024), more than the event buffer
holds (made again with room), and screens queued for another central radius.
The yardstick is the same step's records from a run that asked for none before,
which queues nothing ahead; they equal the oracle's in the other tests."""
import numpy as np
import pytest

from adaptive_cases import planar_body
from mercuda_b200.backend import Backend
from mercuda_b200.system import K2, System

pytestmark = pytest.mark.gpu
RCEN = 0.4


def passing(count):
    """Eight planets, `count` Small bodies that each pass one of them within 0.3
    days, and some that fall past the central body meanwhile."""
    rng = np.random.default_rng(count)
    bodies = [(K2, [0.0] * 3, [0.0] * 3)] + [planar_body(1e-9, 1.0 + 0.1 * k, 0.01, 0.4 * k) for k in range(8)]
    m, x, v = (np.array([b[c] for b in bodies]) for c in range(3))
    at = rng.integers(1, 9, count)
    w = rng.normal(size=(count, 3)) * 0.01
    b = np.cross(w, rng.normal(size=(count, 3)))
    b *= (rng.uniform(0.005, 0.03, count) / np.linalg.norm(b, axis=1))[:, None]
    xs = x[at] + b - w * rng.uniform(0.0, 0.3, count)[:, None]
    vs = v[at] + w
    fall = np.arange(count) % 50 == 7
    xs[fall] *= 0.3
    vs[fall] = -xs[fall] * rng.uniform(0.03, 0.04, fall.sum())[:, None]
    n = 9 + count
    return System(m=np.concatenate([m, np.zeros(count)]), x=np.vstack([x, xs]), v=np.vstack([v, vs]), nbig=9,
                  ngf=np.zeros((n, 5)), rce=np.full(n, 0.05), rphys=np.full(n, 1e-4))


def steps(lib, name, sys0, radii):
    """Two steps of one tenth of a day; the records of each whose radius is not None."""
    b = Backend(name, lib)
    b.configure()
    try:
        b.upload(sys0)
        t, h, out = 0.0, 0.1, []
        for rcen in radii:
            hdid, _ = b.step(t, h, 1e-11)
            t += hdid
            out.append(None if rcen is None else sorted(e.tobytes() for e in b.events(t, hdid, rcen)))
        return out
    finally:
        b.free()


@pytest.fixture(params=["RADAU", "BS", "BS2"])
def case(request):
    return request.param, passing(6000)


@pytest.mark.parametrize("capacity", [0, 1, 1000, 1025])
def test_many_records(cuda_lib, case, capacity):
    name, sys0 = case
    want = steps(cuda_lib, name, sys0, [None, RCEN])[1]
    assert len(want) > 1500
    cuda_lib.mercury_b200_set_event_capacity(capacity)
    try:
        got = steps(cuda_lib, name, sys0, [RCEN, RCEN])[1]
    finally:
        cuda_lib.mercury_b200_set_event_capacity(0)
    assert got == want


def test_another_central_radius(cuda_lib, case):
    name, sys0 = case
    for first, second in ((RCEN, 0.35), (0.35, RCEN), (1e-4, 0.5)):
        want = steps(cuda_lib, name, sys0, [None, second])[1]
        assert steps(cuda_lib, name, sys0, [first, second])[1] == want
