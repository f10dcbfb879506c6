"""The anomaly of a recorded Kepler drift (kepler_adjoint.cuh, compiled for the
host) where one step from the end point's guess is taken to suffice, against a
root of the same equation found in 64-bit significands, on orbits from ordinary
to nearly radial ones, whose end point gives the anomaly to a few digits only.

Bar, for drifts with |alpha| s^2 < 1, where the G functions are sums of a series
(beyond, the rounding of the closed forms' argument grows with it): F(s) = r0 G1
+ sigma0 G2 + mu G3 - dt carries about ten roundings in each G and four in the
sum, all at most 2^-53 of r0 |s|, |sigma0| s^2 / 2, mu |s|^3 / 6 (or of the terms
themselves, hyperbolic ones grow beyond) and |dt|; twice that, over F', and two
roundings of s."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

HEADER = Path(__file__).resolve().parents[1] / "mercuda_b200" / "csrc" / "kepler_adjoint.cuh"
SOURCE = """
#include <cmath>
using namespace std;
typedef double plain;
#ifdef WIDE
#define double long double
#endif
#include "%s"
typedef double real;
#undef double
using namespace mb200;
// the equation's coefficients, the same doubles on both sides
plain dot(const plain* a, const plain* b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }
struct Orbit {
    plain r0, sig, al, mu, dt;
    Orbit(const plain* q, plain m) : r0(sqrt(dot(q, q))), sig(dot(q, q + 3)), mu(m), dt(q[6]) {
        al = 2 * m / r0 - dot(q + 3, q + 3);
    }
};
// rows x, v, dt, x1: out = anomaly, how it was found
extern "C" void anomaly(int n, double mu, const double* in, double* out) {
    for (int k = 0; k < n; ++k, in += 10, out += 2) {
        Orbit o(in, mu);
        real q[10], s, G[6];
        for (int c = 0; c < 10; ++c) q[c] = in[c];
        out[1] = drift_anomaly(q, q + 3, q + 7, o.r0, 1 / o.r0, o.sig, o.al, o.mu, 1 / o.mu, o.dt, s, G);
        out[0] = (double)s;
    }
}
// end positions into columns 7..9; out = the root, the bar's sum of terms, F', alpha s^2
extern "C" void root(int n, double mu, double* in, double* out) {
    for (int k = 0; k < n; ++k, in += 10, out += 4) {
        Orbit o(in, mu);
        real s = (real)o.dt / o.r0, G[6];
        const bool ok = universal_anomaly(o.r0, o.sig, o.al, o.mu, o.dt, s);
        gfuncs(s, o.al, G);
        const real f = 1 - (real)o.mu * G[2] / o.r0, g = o.r0 * G[1] + o.sig * G[2], a = fabs(s);
        for (int c = 0; c < 3; ++c) in[7 + c] = ok ? (double)(f * in[c] + g * in[3 + c]) : NAN;
        out[0] = (double)s;
        out[1] = (double)(o.r0 * fmax(fabs(G[1]), a) + fabs(o.sig) * fmax(G[2], a * a / 2) +
                          o.mu * fmax(fabs(G[3]), a * a * a / 6) + fabs(o.dt));
        out[2] = (double)(o.r0 * G[0] + o.sig * G[1] + o.mu * G[2]);
        out[3] = (double)(o.al * s * s);
    }
}
"""
MU = 2.959122082855911e-4


@pytest.fixture(scope="module")
def libs(tmp_path_factory):
    d = tmp_path_factory.mktemp("vjp")
    (d / "vjp.cpp").write_text(SOURCE % HEADER)
    out = []
    for name, flag in (("narrow", "-DNARROW"), ("wide", "-DWIDE")):
        subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", flag, "-o",
                        str(d / f"{name}.so"), str(d / "vjp.cpp")], check=True, capture_output=True)
        out.append(C.CDLL(str(d / f"{name}.so")))
    return out


@pytest.mark.parametrize("angle", [1.0, 1e-2, 1e-4, 1e-6, 1e-8, 1e-9, 1e-10, 2e-11])
def test_accepted_anomaly(libs, angle):
    narrow, wide = libs
    p = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))
    rng = np.random.default_rng(int(1 / angle) % 1000003)
    n = 20000
    e = rng.normal(size=(n, 3))
    e /= np.linalg.norm(e, axis=1)[:, None]
    r = 10 ** rng.uniform(-2, 1, n)
    vv = np.sqrt(2 * MU / r) * rng.uniform(0.05, 1.55, n)
    q = np.zeros((n, 10))
    q[:, :3] = e * r[:, None]
    q[:, 3:6] = vv[:, None] * (rng.choice([-1.0, 1.0], n)[:, None] * e + angle * rng.normal(size=(n, 3)))
    q[:, 6] = 10 ** rng.uniform(-2, 2, n) * rng.choice([-1.0, 1.0], n)
    want, got = np.zeros((n, 4)), np.zeros((n, 2))
    wide.root(n, C.c_double(MU), p(q), p(want))
    ok = np.isfinite(q).all(axis=1) & (np.abs(want[:, 3]) < 1.0)
    q, want, got = (np.ascontiguousarray(a[ok]) for a in (q, want, got))
    narrow.anomaly(len(q), C.c_double(MU), p(q), p(got))
    one = got[:, 1] == 2
    assert ok.sum() > 5000 and one.any()
    bar = 2.0 ** -53 * (28 * want[:, 1] / np.abs(want[:, 2]) + 2 * np.abs(want[:, 0]))
    worst = (np.abs(got[:, 0] - want[:, 0]) / bar)[one].max()
    assert worst <= 1.0, worst
