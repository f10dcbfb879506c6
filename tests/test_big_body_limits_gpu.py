"""The Big-body CTA at the ends of its forms: 33 bodies with a slot for every
pair force, 34 without, and the 512 that an upload takes (224 KB of shared
memory), of Big bodies alone and with massive Small bodies among them."""
import numpy as np
import pytest

from mercuda_b200.backend import Backend, BackendError
from mercuda_b200.system import make_system

from test_mvs_gpu import REL_ONE_STEP, assert_events_equal, rel_err

pytestmark = pytest.mark.gpu


def system(nbig, massive):
    s = make_system(seed=nbig, n_particles=massive + 40, nplanets=nbig - 1, planet_kw=dict(mmin=1e-9, mmax=1e-8))
    s.m[s.nbig:s.nbig + massive] = 1e-12
    return s


@pytest.mark.parametrize("nbig,massive", [(32, 0), (33, 0), (34, 0), (20, 13), (20, 14), (512, 0), (300, 212)])
def test_one_step(cuda_lib, oracle, nbig, massive):
    s = system(nbig, massive)
    b = Backend("MVS", cuda_lib)
    b.configure()
    try:
        b.upload(s)
        b.step(0.0, 8.0, dtflag=0)
        x, v = b.download()
        ev = b.events(8.0, 8.0, 0.005)
    finally:
        b.free()
    ref = s.copy()
    rev, _ = oracle.mvs_run(ref, 0.0, 8.0, 1, 0.005, threads=4)
    assert rel_err(x, ref.x) <= REL_ONE_STEP
    assert rel_err(v, ref.v) <= REL_ONE_STEP
    assert_events_equal(ev, rev)


@pytest.mark.parametrize("nbig,massive", [(513, 0), (300, 213)])
def test_beyond_the_limit(cuda_lib, nbig, massive):
    s = system(nbig, massive)
    s.jcen[:] = [1e-6, 0.0, 0.0]
    b = Backend("MVS", cuda_lib)
    b.configure()
    try:
        with pytest.raises(BackendError):
            b.upload(s)
    finally:
        b.free()
