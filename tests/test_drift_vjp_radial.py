"""Drifts of radial orbits (kepler_adjoint.cuh, compiled for the host), whose end
point says nothing about the anomaly: wherever the universal Kepler equation is
solved from dt / r0, the walk back has to solve it too."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

HEADER = Path(__file__).resolve().parents[1] / "mercuda_b200" / "csrc" / "kepler_adjoint.cuh"
SOURCE = """
#include <cmath>
using namespace std;
#include "%s"
using namespace mb200;
// rows x, v, dt; returns the drifts solved from dt / r0, failed = those that the walk does not solve
extern "C" int solve(int n, double mu, const double* q, int* failed) {
    int solved = 0;
    *failed = 0;
    for (int k = 0; k < n; ++k, q += 7) {
        const double *x = q, *v = q + 3, dt = q[6], r0 = sqrt(dot3(x, x)), sig = dot3(x, v);
        const double al = 2 * mu / r0 - dot3(v, v);
        double s = dt / r0, G[6], x1[3];
        if (!universal_anomaly(r0, sig, al, mu, dt, s)) continue;
        ++solved;
        gfuncs(s, al, G);
        const double f = 1 - mu * G[2] / r0, g = r0 * G[1] + sig * G[2];
        for (int c = 0; c < 3; ++c) x1[c] = f * x[c] + g * v[c];
        *failed += !drift_anomaly(x, v, x1, r0, 1 / r0, sig, al, mu, 1 / mu, dt, s, G);
    }
    return solved;
}
"""
MU = 2.959122082855911e-4


@pytest.mark.parametrize("exact", [True, False])
def test_radial_drifts_are_solved(tmp_path, exact):
    (tmp_path / "radial.cpp").write_text(SOURCE % HEADER)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-o",
                    str(tmp_path / "radial.so"), str(tmp_path / "radial.cpp")], check=True, capture_output=True)
    lib = C.CDLL(str(tmp_path / "radial.so"))
    rng = np.random.default_rng(11)
    n = 100000
    e = rng.normal(size=(n, 3))
    e /= np.linalg.norm(e, axis=1)[:, None]
    r = 10 ** rng.uniform(-2, 1, n)
    k = np.sqrt(2 * MU / r) * rng.uniform(0.05, 1.55, n) / r
    if exact:   # v a power of two times x: equal products in x x v
        k = np.exp2(np.floor(np.log2(k)))
    q = np.zeros((n, 7))
    q[:, :3] = e * r[:, None]
    q[:, 3:6] = q[:, :3] * (k * rng.choice([-1.0, 1.0], n))[:, None]
    q[:, 6] = 10 ** rng.uniform(-2, 2, n) * rng.choice([-1.0, 1.0], n)
    failed = C.c_int()
    solved = lib.solve(n, C.c_double(MU), q.ctypes.data_as(C.POINTER(C.c_double)), C.byref(failed))
    assert solved > n // 2 and failed.value == 0, (solved, failed.value)
