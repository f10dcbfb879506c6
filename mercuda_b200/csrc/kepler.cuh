// Universal-variable Kepler drift for one body, FP64, on the device.
//
// Restates SWIFT's drift_* routines as they appear in mercury6_2.for:7602-8330
// (Levison & Duncan) and mco_sine (mercury6_2.for:2940-2972), keeping every
// statement's operand order so that, with --fmad=false, each result rounds as
// the Fortran CPU build rounds it. The paths are: the elliptic small-step
// solver drift_kepmd when dm^2 <= 0.16, e^2 <= 0.36 and e^2 dm^2 < 0.0016;
// otherwise drift_kepu (seed from drift_kepu_guess, up to 7 quartic Newton
// iterations, then at most 401 Laguerre iterations); drift_one retries a
// failed drift as ten substeps and keeps the partial result, as every caller
// in the reference does.
#pragma once
#include "common.cuh"
#include "fp64.cuh"

namespace mb200 {

// drift_kepu_stumpff: argument quartering, degree-6 series, doubling back.
// Any finite argument falls below 0.1 within about 520 quarterings; the cap
// only stops a non-finite argument (which then yields a non-finite result and
// a failed drift) from looping forever.
constexpr int STUMPFF_MAX_QUARTERINGS = 2000;
__device__ __forceinline__ void stumpff(double x, double& c0, double& c1, double& c2, double& c3) {
    int n = 0;
    while (fabs(x) >= 0.1 && n < STUMPFF_MAX_QUARTERINGS) {
        n = n + 1;
        x = x * 0.25;
    }
    const double x2 = x * x, x3 = x * x2, x4 = x2 * x2, x5 = x2 * x3, x6 = x3 * x3;
    c2 = 1.147074559772972e-11 * x6 - 2.087675698786810e-9 * x5 + 2.755731922398589e-7 * x4 -
         2.480158730158730e-5 * x3 + 1.388888888888889e-3 * x2 - 4.166666666666667e-2 * x + 0.5;
    c3 = 7.647163731819816e-13 * x6 - 1.605904383682161e-10 * x5 + 2.505210838544172e-8 * x4 -
         2.755731922398589e-6 * x3 + 1.984126984126984e-4 * x2 - 8.333333333333333e-3 * x +
         1.666666666666667e-1;
    c1 = 1.0 - x * c3;
    c0 = 1.0 - x * c2;
#pragma unroll 1
    for (int i = n; i >= 1; --i) {
        c3 = (c2 + c0 * c3) * 0.25;
        c2 = c1 * c1 * 0.5;
        c1 = c0 * c1;
        c0 = 2.0 * c0 * c0 - 1.0;
    }
}

// drift_kepu_fchk: residual of the universal Kepler equation at s.
__device__ __forceinline__ double kepu_residual(double dt, double r0, double mu, double alpha, double u,
                                                double s) {
    double c0, c1, c2, c3;
    stumpff(s * s * alpha, c0, c1, c2, c3);
    c1 = c1 * s;
    c2 = c2 * s * s;
    c3 = c3 * s * s * s;
    return r0 * c1 + u * c2 + mu * c3 - dt;
}

// drift_kepu_p3solve: Cardano seed for alpha <= 0. Returns false when no real root.
static __device__ __noinline__ bool kepu_cubic_seed(double dt, double r0, double mu, double alpha, double u,
                                             double& s) {
    const double denom = (mu - alpha * r0) / 6.0;
    const double a2 = 0.5 * u / denom;
    const double a1 = r0 / denom;
    const double a0 = -dt / denom;
    const double q = (a1 - a2 * a2 / 3.0) / 3.0;
    const double r = (a1 * a2 - 3.0 * a0) / 6.0 - pow(a2, 3.0) / 27.0;
    const double sq2 = pow(q, 3.0) + r * r;
    if (sq2 >= 0.0) {
        const double sq = sqrt(sq2), third = 1.0 / 3.0;
        const double p1 = (r + sq) <= 0.0 ? -pow(-(r + sq), third) : pow(r + sq, third);
        const double p2 = (r - sq) <= 0.0 ? -pow(-(r - sq), third) : pow(r - sq, third);
        s = p1 + p2 - a2 / 3.0;
        return true;
    }
    s = 0.0;
    return false;
}

// drift_kepu_guess (with mco_sine for the elliptic long-step seed).
__device__ __forceinline__ double kepu_guess(double dt, double r0, double mu, double alpha, double u) {
    if (alpha > 0.0) {
        if (dt / r0 <= 0.4) return dt / r0 - (dt * dt * u) / (2.0 * r0 * r0 * r0);
        const double a = mu / alpha;
        const double en = sqrt(mu / (a * a * a));
        const double ec = 1.0 - r0 / a;
        const double es = u / (en * a * a);
        const double e = sqrt(ec * ec + es * es);
        double y = en * dt - es;
        // mco_sine
        const double pi = 3.141592653589793, twopi = 2.0 * pi;
        if (y > 0.0) y = fmod(y, twopi);
        else y = fmod(y, twopi) + twopi;
        const double cy = cos(y);
        const double sy = (y > pi) ? -sqrt(1.0 - cy * cy) : sqrt(1.0 - cy * cy);
        const double sigma = copysign(1.0, es * cy + ec * sy);
        const double x = y + sigma * 0.85 * e;
        return x / sqrt(alpha);
    }
    double s;
    if (!kepu_cubic_seed(dt, r0, mu, alpha, u, s)) s = dt / r0;
    return s;
}

// drift_kepu_new: quartic Newton, at most 7 passes. Returns true on convergence.
__device__ __forceinline__ bool kepu_newton(double& s, double dt, double r0, double mu, double alpha,
                                            double u, double& fp, double& c1, double& c2, double& c3) {
    const double tol = DANBYB * DANBYB;
#pragma unroll 1
    for (int nc = 0; nc <= 6; ++nc) {
        const double s2 = s * s;
        double c0;
        stumpff(s2 * alpha, c0, c1, c2, c3);
        c1 = c1 * s;
        c2 = c2 * s2;
        c3 = c3 * s * s2;
        const double f = r0 * c1 + u * c2 + mu * c3 - dt;
        fp = r0 * c0 + u * c1 + mu * c2;
        const double fpp = (mu - r0 * alpha) * c1 + u * c0;
        const double fppp = (mu - r0 * alpha) * c0 - u * alpha * c1;
        double ds = -(f / fp);
        ds = -(f / (fp + 0.5 * ds * fpp));
        ds = -(f / (fp + 0.5 * ds * fpp + ds * ds * fppp * 0.1666666666666667));
        s = s + ds;
        const double fdt = f / dt;
        if (fdt * fdt < tol) return true;
    }
    return false;
}

// drift_kepu_lag: Laguerre iteration (n = 5), at most 401 passes; rarely taken.
static __device__ __noinline__ bool kepu_laguerre(double& s, double dt, double r0, double mu, double alpha,
                                           double u, double& fp, double& c1, double& c2, double& c3) {
    const double ln = 5.0, tol = DANBYB * DANBYB;
#pragma unroll 1
    for (int nc = 0; nc <= 400; ++nc) {
        double c0;
        stumpff(s * s * alpha, c0, c1, c2, c3);
        c1 = c1 * s;
        c2 = c2 * s * s;
        c3 = c3 * s * s * s;
        const double f = r0 * c1 + u * c2 + mu * c3 - dt;
        fp = r0 * c0 + u * c1 + mu * c2;
        const double fpp = (-40.0 * alpha + mu) * c1 + u * c0;
        const double ds = -(ln * f / (fp + copysign(1.0, fp) *
                                                sqrt(fabs((ln - 1.0) * (ln - 1.0) * fp * fp -
                                                          (ln - 1.0) * ln * f * fpp))));
        s = s + ds;
        const double fdt = f / dt;
        if (fdt * fdt < tol) return true;
    }
    return false;
}

// drift_kepu: guess, Newton, and on failure the better of the two seeds for Laguerre.
__device__ __forceinline__ bool kepu(double dt, double r0, double mu, double alpha, double u, double& fp,
                                     double& c1, double& c2, double& c3) {
    double s = kepu_guess(dt, r0, mu, alpha, u);
    const double st = s;
    if (kepu_newton(s, dt, r0, mu, alpha, u, fp, c1, c2, c3)) return true;
    const double fo = kepu_residual(dt, r0, mu, alpha, u, st);
    const double fn = kepu_residual(dt, r0, mu, alpha, u, s);
    if (fabs(fo) < fabs(fn)) s = st;
    return kepu_laguerre(s, dt, r0, mu, alpha, u, fp, c1, c2, c3);
}

// Series for sin x of drift_kepmd (Horner form over 11!).
__device__ __forceinline__ double kepmd_sine(double x) {
    const double y = x * x;
    return x * (39916800.0 - y * (6652800.0 - y * (332640.0 - y * (7920.0 - y * (110.0 - y))))) /
           39916800.0;
}

// drift_dan. State (p, w) is updated in place; returns false (state untouched)
// when neither solver converged, which makes drift_one substep.
__device__ __forceinline__ bool drift_dan(double mu, double3& p, double3& w, double dt0) {
    double dt = dt0;
    const double r0 = sqrt(p.x * p.x + p.y * p.y + p.z * p.z);
    const double v0s = w.x * w.x + w.y * w.y + w.z * w.z;
    const double u = p.x * w.x + p.y * w.y + p.z * w.z;
    const double alpha = 2.0 * mu / r0 - v0s;
    double f, g, fdot, gdot;
    bool done = false;
    if (alpha > 0.0) {
        const double a = mu / alpha;
        const double asq = a * a;
        const double en = sqrt(mu / (a * asq));
        const double ec = 1.0 - r0 / a;
        const double es = u / (en * asq);
        const double esq = ec * ec + es * es;
        const double dm = dt * en - double(int(dt * en / TWOPI_SWIFT)) * TWOPI_SWIFT;
        dt = dm / en;
        if (!((dm * dm > 0.16) || (esq > 0.36)) && esq * dm * dm < 0.0016) {
            // drift_kepmd: cubic seed, one quartic Newton correction.
            const double fac1 = 1.0 / (1.0 - ec);
            const double q = fac1 * dm;
            const double fac2 = es * es * fac1 - ec / 3.0;
            double x = q * (1.0 - 0.5 * fac1 * q * (es - q * fac2));
            double s = kepmd_sine(x);
            double c = sqrt(1.0 - s * s);
            {
                const double ff = x - ec * s + es * (1.0 - c) - dm;
                const double ffp = 1.0 - ec * c + es * s;
                const double ffpp = ec * s + es * c;
                const double ffppp = ec * c - es * s;
                double dx = -(ff / ffp);
                dx = -(ff / (ffp + 0.5 * dx * ffpp));
                dx = -(ff / (ffp + 0.5 * dx * ffpp + 0.16666666666666666 * dx * dx * ffppp));
                x = x + dx;
            }
            s = kepmd_sine(x);
            c = sqrt(1.0 - s * s);
            const double fchk = (x - ec * s + es * (1.0 - c) - dm);
            if (fchk * fchk > DANBYB) return false;
            const double fp = 1.0 - ec * c + es * s;
            f = (a / r0) * (c - 1.0) + 1.0;
            g = dt + (s - x) / en;
            fdot = -(a / (r0 * fp)) * en * s;
            gdot = (c - 1.0) / fp + 1.0;
            done = true;
        }
    }
    if (!done) {
        double fp, c1, c2, c3;
        if (!kepu(dt, r0, mu, alpha, u, fp, c1, c2, c3)) return false;
        f = 1.0 - (mu / r0) * c2;
        g = dt - mu * c3;
        fdot = -(mu / (fp * r0)) * c1;
        gdot = 1.0 - (mu / fp) * c2;
    }
    const double3 p1 = make_double3(p.x * f + w.x * g, p.y * f + w.y * g, p.z * f + w.z * g);
    const double3 w1 = make_double3(p.x * fdot + w.x * gdot, p.y * fdot + w.y * gdot, p.z * fdot + w.z * gdot);
    p = p1;
    w = w1;
    return true;
}

// drift_dan's drift_kepmd branch for operands of moderate size, in straight
// line: every statement and rounding of the branch above, its sixteen divisions
// and four square roots by the sequences of fp64.cuh, which share reciprocals
// where the statements share a divisor (r0, en, a) or one is the product of
// others. rr = |p|^2 and rmu ~ 1/mu (within an ulp) come from the caller. False
// (state untouched) where drift_dan takes another branch, drift_kepmd does not
// converge or an operand is out of range; the caller then runs drift_dan.
// What bounds it is the issue of its FP64 instructions and the length of its
// chain. Five of the reciprocals are products and take a step more to be known to
// half an ulp: ten instructions, 2.59 -> 2.62 ms for 100 steps of 300,000 particles.
__device__ __forceinline__ bool narrow_range(double x) {   // positive, exponent -100 .. 99
    return (unsigned)__double2hiint(x) - ((1023u - 100u) << 20) < (200u << 20);
}
__device__ __forceinline__ double kepmd_sine_near(double x) {
    const double y = x * x;
    return quotient(x * (39916800.0 - y * (6652800.0 - y * (332640.0 - y * (7920.0 - y * (110.0 - y))))),
                    39916800.0, 1.0 / 39916800.0);
}
__device__ __forceinline__ bool drift_near(double mu, double rmu, double3& p, double3& w, double dt0, double rr) {
    double r0, yr;
    sqrt_recip(rr, r0, yr);
    const double v0s = w.x * w.x + w.y * w.y + w.z * w.z;
    const double u = p.x * w.x + p.y * w.y + p.z * w.z;
    const double alpha = quotient(2.0 * mu, r0, yr) - v0s;
    if (!(narrow_range(rr) && narrow_range(alpha) && narrow_range(mu))) return false;
    const double a = quotient(mu, alpha, recip_near(alpha));
    const double asq = a * a;
    const double acu = a * asq;
    double en, yen;
    sqrt_recip(quotient(mu, acu, recip_near(acu)), en, yen);
    const double ya = recip_fix(a, alpha * rmu);
    const double ec = 1.0 - quotient(r0, a, ya);
    const double es = quotient_of(u, en * asq, yen * (ya * ya));
    const double esq = ec * ec + es * es;
    // dt en: beyond one turn it fails the next test, and within one the whole
    // turns drift_dan takes off are none
    const double dm = dt0 * en;
    if (!(!((dm * dm > 0.16) || (esq > 0.36)) && esq * dm * dm < 0.0016)) return false;
    const double dt = quotient_fix(dm, en, yen, dt0);
    const double b = 1.0 - ec;   // r0 / a but for its rounding
    const double fac1 = recip_fix(b, recip_fix(b, a * yr));
    const double q = fac1 * dm;
    const double fac2 = es * es * fac1 - quotient(ec, 3.0, 1.0 / 3.0);
    double x = q * (1.0 - 0.5 * fac1 * q * (es - q * fac2));
    double s = kepmd_sine_near(x), c, y;
    sqrt_near(1.0 - s * s, c, y);
    {
        const double ff = x - ec * s + es * (1.0 - c) - dm;
        const double ffp = 1.0 - ec * c + es * s;
        const double ffpp = ec * s + es * c;
        const double ffppp = ec * c - es * s;
        double dx = -quotient(ff, ffp, recip_near(ffp));
        const double d2 = ffp + 0.5 * dx * ffpp;
        dx = -quotient(ff, d2, recip_near(d2));
        const double d3 = ffp + 0.5 * dx * ffpp + 0.16666666666666666 * dx * dx * ffppp;
        dx = -quotient(ff, d3, recip_near(d3));
        x = x + dx;
    }
    s = kepmd_sine_near(x);
    sqrt_near(1.0 - s * s, c, y);
    const double fchk = (x - ec * s + es * (1.0 - c) - dm);
    if (fchk * fchk > DANBYB) return false;
    const double fp = 1.0 - ec * c + es * s;
    const double yfp = recip_near(fp);
    const double f = quotient(a, r0, yr) * (c - 1.0) + 1.0;
    const double g = dt + quotient(s - x, en, yen);
    const double fdot = -quotient_of(a, r0 * fp, yr * yfp) * en * s;
    const double gdot = quotient(c - 1.0, fp, yfp) + 1.0;
    const double3 p1 = make_double3(p.x * f + w.x * g, p.y * f + w.y * g, p.z * f + w.z * g);
    const double3 w1 = make_double3(p.x * fdot + w.x * gdot, p.y * fdot + w.y * gdot, p.z * fdot + w.z * gdot);
    p = p1;
    w = w1;
    return true;
}

// The rest of drift_dan, drift_kepu's universal-variable solve, the same way:
// the statements of kepu_guess, kepu_newton and kepu_laguerre with the
// divisions and square roots of fp64.cuh. Particles on this path are few
// (1.6 % at the start of the 1M-particle workload, 5 % after 4,600 steps), but
// a warp of them takes several times an ordinary warp's time and, started
// first, still ends a launch of 16 to 31 steps last: what counts here is the
// length of the chain. Undecided (state untouched) where drift_kepmd applies or
// an operand is out of range: drift_dan then decides. Failed, as drift_dan would
// be with the same iterates, where Laguerre's 401 passes do not converge.
enum : int { DRIFT_FAILED = -1, DRIFT_UNDECIDED = 0, DRIFT_DONE = 1 };
// stumpff with the number of quarterings taken from the exponent (|x| 4^-n is
// exact either way), for |x| below 2^200.
__device__ __forceinline__ void stumpff_near(double x, double& c0, double& c1, double& c2, double& c3) {
    int n = 0;
    if (fabs(x) >= 0.1) {
        const int k = ((__double2hiint(x) >> 20) & 0x7ff) - 1023 + 4;   // |x| = m 2^(k - 4), 0.1 = 1.6 2^-4
        n = (k + 1) >> 1;
        x = x * __hiloint2double((1023 - 2 * n) << 20, 0);
        if (fabs(x) >= 0.1) {
            ++n;
            x = x * 0.25;
        }
    }
    const double x2 = x * x, x3 = x * x2, x4 = x2 * x2, x5 = x2 * x3, x6 = x3 * x3;
    c2 = 1.147074559772972e-11 * x6 - 2.087675698786810e-9 * x5 + 2.755731922398589e-7 * x4 -
         2.480158730158730e-5 * x3 + 1.388888888888889e-3 * x2 - 4.166666666666667e-2 * x + 0.5;
    c3 = 7.647163731819816e-13 * x6 - 1.605904383682161e-10 * x5 + 2.505210838544172e-8 * x4 -
         2.755731922398589e-6 * x3 + 1.984126984126984e-4 * x2 - 8.333333333333333e-3 * x +
         1.666666666666667e-1;
    c1 = 1.0 - x * c3;
    c0 = 1.0 - x * c2;
#pragma unroll 1
    for (int i = n; i >= 1; --i) {
        c3 = (c2 + c0 * c3) * 0.25;
        c2 = c1 * c1 * 0.5;
        c1 = c0 * c1;
        c0 = 2.0 * c0 * c0 - 1.0;
    }
}
__device__ __forceinline__ int drift_universal(double mu, double3& p, double3& w, double dt) {
    const double rr = p.x * p.x + p.y * p.y + p.z * p.z;
    double r0, yr;
    sqrt_recip(rr, r0, yr);
    const double v0s = w.x * w.x + w.y * w.y + w.z * w.z;
    const double u = p.x * w.x + p.y * w.y + p.z * w.z;
    const double alpha = quotient(2.0 * mu, r0, yr) - v0s;
    if (!(narrow_range(rr) && narrow_range(mu))) return DRIFT_UNDECIDED;
    double s;
    if (alpha > 0.0) {
        if (!narrow_range(alpha)) return DRIFT_UNDECIDED;
        const double a = quotient(mu, alpha, recip_near(alpha));
        const double asq = a * a;
        const double acu = a * asq;
        double en, yen;
        sqrt_recip(quotient(mu, acu, recip_near(acu)), en, yen);
        const double ya = recip_near(a);
        const double ec = 1.0 - quotient(r0, a, ya);
        const double es = quotient_of(u, en * asq, yen * (ya * ya));
        const double esq = ec * ec + es * es;
        const double turn = dt * en;
        const double dm = turn - double(int(quotient(turn, TWOPI_SWIFT, 1.0 / TWOPI_SWIFT))) * TWOPI_SWIFT;
        dt = quotient(dm, en, yen);
        if (!((dm * dm > 0.16) || (esq > 0.36)) && esq * dm * dm < 0.0016) return DRIFT_UNDECIDED;
        const double lead = quotient(dt, r0, yr);
        if (lead <= 0.4) {
            const double d = 2.0 * r0 * r0 * r0;
            s = lead - quotient(dt * dt * u, d, recip_near(d));
        } else {
            const double d = en * a * a;
            const double esg = quotient(u, d, recip_near(d));
            double y = en * dt - esg, e, ye;
            const double e2 = ec * ec + esg * esg;
            if (!mid_range(e2)) return DRIFT_UNDECIDED;
            sqrt_near(e2, e, ye);
            // mco_sine (fmod leaves an angle within one turn as it is)
            const double pi = 3.141592653589793, twopi = 2.0 * pi;
            const double ym = fabs(y) < twopi ? y : fmod(y, twopi);
            y = y > 0.0 ? ym : ym + twopi;
            const double cy = cos(y);
            const double sy = (y > pi) ? -sqrt(1.0 - cy * cy) : sqrt(1.0 - cy * cy);
            const double sigma = copysign(1.0, esg * cy + ec * sy);
            const double x = y + sigma * 0.85 * e;
            double sa, ysa;
            sqrt_recip(alpha, sa, ysa);
            s = quotient(x, sa, ysa);
        }
    } else {
        // NaN comes here too and fails below
        if (!kepu_cubic_seed(dt, r0, mu, alpha, u, s)) s = quotient(dt, r0, yr);
    }
    if (!mid_magnitude(dt)) return DRIFT_UNDECIDED;
    const double ydt = recip_near(dt), tol = DANBYB * DANBYB;
    double fp = 0.0, c0, c1 = 0.0, c2 = 0.0, c3 = 0.0;
    const double st = s, mra = mu - r0 * alpha;
    bool done = false;
#pragma unroll 1
    for (int nc = 0; nc <= 6 && !done; ++nc) {
        const double s2 = s * s;
        const double z = s2 * alpha;
        stumpff_near(z, c0, c1, c2, c3);
        c1 = c1 * s;
        c2 = c2 * s2;
        c3 = c3 * s * s2;
        const double f = r0 * c1 + u * c2 + mu * c3 - dt;
        fp = r0 * c0 + u * c1 + mu * c2;
        const double fpp = mra * c1 + u * c0;
        const double fppp = mra * c0 - u * alpha * c1;
        double ds = -quotient(f, fp, recip_near(fp));
        const double d2 = fp + 0.5 * ds * fpp;
        ds = -quotient(f, d2, recip_near(d2));
        const double d3 = fp + 0.5 * ds * fpp + ds * ds * fppp * 0.1666666666666667;
        ds = -quotient(f, d3, recip_near(d3));
        // z below 2^200, divisors and numerators of moderate size
        if (!(fabs(z) < 1e60 && fabs(f) < 1e60 && mid_magnitude(fp) && mid_magnitude(d2) && mid_magnitude(d3)))
            return DRIFT_UNDECIDED;
        s = s + ds;
        const double fdt = quotient(f, dt, ydt);
        done = fdt * fdt < tol;
    }
    if (!done) {
        // Laguerre from the better of the two ends
        const double fo = kepu_residual(dt, r0, mu, alpha, u, st);
        const double fn = kepu_residual(dt, r0, mu, alpha, u, s);
        if (fabs(fo) < fabs(fn)) s = st;
        const double ln = 5.0;
#pragma unroll 1
        for (int nc = 0; nc <= 400 && !done; ++nc) {
            const double z = s * s * alpha;
            stumpff_near(z, c0, c1, c2, c3);
            c1 = c1 * s;
            c2 = c2 * s * s;
            c3 = c3 * s * s * s;
            const double f = r0 * c1 + u * c2 + mu * c3 - dt;
            fp = r0 * c0 + u * c1 + mu * c2;
            const double fpp = (-40.0 * alpha + mu) * c1 + u * c0;
            const double q = fabs((ln - 1.0) * (ln - 1.0) * fp * fp - (ln - 1.0) * ln * f * fpp);
            double sq, ysq;
            sqrt_near(q, sq, ysq);
            const double d = fp + copysign(1.0, fp) * sq;
            if (!(fabs(z) < 1e60 && fabs(f) < 1e60 && mid_range(q) && mid_magnitude(d))) return DRIFT_UNDECIDED;
            s = s - quotient(ln * f, d, recip_near(d));
            const double fdt = quotient(f, dt, ydt);
            done = fdt * fdt < tol;
        }
        if (!done) return DRIFT_FAILED;
    }
    if (!mid_magnitude(fp)) return DRIFT_UNDECIDED;
    const double yfp = recip_near(fp);
    const double d = fp * r0;
    const double f = 1.0 - quotient(mu, r0, yr) * c2;
    const double g = dt - mu * c3;
    const double fdot = -quotient_of(mu, d, yfp * yr) * c1;
    const double gdot = 1.0 - quotient(mu, fp, yfp) * c2;
    const double3 p1 = make_double3(p.x * f + w.x * g, p.y * f + w.y * g, p.z * f + w.z * g);
    const double3 w1 = make_double3(p.x * fdot + w.x * gdot, p.y * fdot + w.y * gdot, p.z * fdot + w.z * gdot);
    p = p1;
    w = w1;
    return DRIFT_DONE;
}

// drift_one: the drift, else ten substeps of dt/10 (stopping at a failed one).
// The flag is discarded by all MVS/HYBRID callers (mdt_mvs, mdt_hy, mco_mvs2h).
// Written as one loop so that each solver is there once: attempt 0 is the whole
// step, attempts 1..10 the substeps. An orbit whose solves fail takes up to
// eleven rounds of 401 passes in every step, alone: one such among 1M particles
// made a run of 457 steps take 458 ms with drift_dan for every round behind a
// failed first one, 161 as here (runs without such an orbit 32 to 38).
struct DriftState {
    double3 p, w;
    int done;
};
static __device__ __noinline__ DriftState drift_plain(double mu, DriftState z, double dt) {
    z.done = drift_dan(mu, z.p, z.w, dt) ? DRIFT_DONE : DRIFT_FAILED;
    return z;
}
static __device__ __noinline__ DriftState drift_general(double mu, DriftState z, double dt) {
#pragma unroll 1
    for (int attempt = 0; attempt <= 10; ++attempt) {
        z.done = drift_universal(mu, z.p, z.w, dt);
        if (z.done == DRIFT_UNDECIDED) z = drift_plain(mu, z, dt);
        if (attempt == 0) dt = dt / 10.0;
        if ((z.done == DRIFT_DONE) == (attempt == 0)) break;
    }
    return z;
}
// With rr = |p|^2 at hand and rmu ~ 1/mu. The general solver is a call, so
// that its registers do not count against the straight-line path.
__device__ __forceinline__ void drift_one(double mu, double rmu, double3& p, double3& w, double dt, double rr) {
    if (drift_near(mu, rmu, p, w, dt, rr)) return;
    const DriftState z = drift_general(mu, DriftState{p, w, 0}, dt);
    p = z.p;
    w = z.w;
}
__device__ __forceinline__ void drift_one(double mu, double3& p, double3& w, double dt) {
    drift_one(mu, recip_near(mu), p, w, dt, p.x * p.x + p.y * p.y + p.z * p.z);
}

}  // namespace mb200
