// MVS kernels: the Big-body integrator (one CTA) and the fused test-particle
// step (kick, Kepler drift, encounter screen, interaction kick) for K steps
// per launch with the particle state in registers.
#include <stdexcept>

#include "kepler.cuh"
#include "mvs.cuh"
#include "mvs_device.cuh"

// Minimum resident CTAs per SM requested from ptxas for the particle kernel
// (bounds its registers per thread at 65536 / (128 * this)). 1M particles, 16
// steps: 0.90 ms a launch with 5 (96 registers), 0.885 with 6 (80), 0.89 with 7.
#ifndef MB200_PARTICLE_MIN_BLOCKS
#define MB200_PARTICLE_MIN_BLOCKS 6
#endif

namespace mb200 {
static_assert(sizeof(MercuryEvent) == 8 * sizeof(double2), "event records are eight double2 words");

namespace {

constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ double3 ld3(const double* p, int stride, int k) {
    return make_double3(p[k], p[stride + k], p[2 * stride + k]);
}
__device__ __forceinline__ void st3(double* p, int stride, int k, double3 v) {
    p[k] = v.x;
    p[stride + k] = v.y;
    p[2 * stride + k] = v.z;
}

// The order of doubles on integers: a >= b implies order_key(a) >= order_key(b)
// - 1 (only the high words count; the 1 is for -0 >= +0).
__device__ __forceinline__ int order_key(double x) {
    const int hi = __double2hiint(x);
    return hi ^ ((hi >> 31) & 0x7fffffff);
}

// ------------------------------------------------------------ Big bodies
// The Big-body step is one CTA's serial chain, and small runs, the per-step
// calls, batches and the adjoint's forward run all wait for it: what counts is
// its latency. Sums that the map takes in body order (Jacobi coordinates, the
// indirect terms, the pair forces) are made by one thread per body and
// coordinate, each adding its own prefix in that order from terms computed one
// per thread; everything that depends on the masses alone is computed once per
// launch; square roots and divisions are those of fp64.cuh; and what the next
// step does not wait for (boxes, details, encounter and impact screens) is
// done by warps beside the ones that compute the force. 8 planets: 19 us a
// step with those loops in one thread and plain divisions, 5.2 us so (half of it
// the innermost planet's universal-variable drift).

// Shared-memory workspace of the Big-body CTA. Arrays are found by their place
// in it (a table of pointers would live in local memory): [3][N] vectors, then
// [N] scalars, the pair terms last.
constexpr int BIG_PAIR_MAX = 33;   // bodies up to which every pair force has its slot
constexpr int BIG_THREADS = 256;   // a warp for each of eight planets' drifts
struct BigSmem {
    double* base;
    int N;
    int now;   // parity of the current step: its start state is XS(now), VS(now)
    __device__ double* vec(int q) const { return base + 3 * N * q; }
    __device__ double* scal(int q) const { return base + (3 * 17 + q) * N; }
    __device__ double* X() const { return vec(0); }
    __device__ double* V() const { return vec(1); }
    __device__ double* XJ() const { return vec(2); }    // Jacobi
    __device__ double* VJ() const { return vec(3); }
    __device__ double* ACC() const { return vec(4); }
    __device__ double* V0() const { return vec(5); }    // velocity after the first kick
    __device__ double* XS(int par) const { return vec(6 + par); }
    __device__ double* VS(int par) const { return vec(8 + par); }
    __device__ double* X0() const { return XS(now); }   // the kick leaves positions alone
    __device__ double* A1() const { return vec(10); }   // mfo_mvs's terms, see big_force_terms
    __device__ double* F0() const { return vec(11); }
    __device__ double* F2() const { return vec(12); }
    __device__ double* A3() const { return vec(13); }
    __device__ double* OT() const { return vec(14); }
    __device__ double* AO() const { return vec(15); }
    __device__ double* NG() const { return vec(16); }
    __device__ double* GM() const { return scal(0); }   // gm_j
    __device__ double* TH() const { return scal(1); }   // 1 / MI
    __device__ double* TJ() const { return scal(2); }   // m_j over the mass up to j
    __device__ double* MI() const { return scal(3); }   // mass inside j
    __device__ double* MS() const { return scal(4); }   // masses
    // N <= BIG_PAIR_MAX: for each coordinate c and body k a row of terms by
    // the other body (its index less 1), padded with zeros to whole chunks of eight:
    // signed pair forces, then mfo_mvs's second indirect term of the bodies up
    // to k; and one row a coordinate of the first indirect term
    __device__ int np() const { return term_row(N); }
    __device__ double* PT(int c, int k) const { return scal(5) + (c * N + k) * np(); }
    __device__ double* QT(int c, int k) const { return PT(3 + c, k); }
    __device__ double* RT(int c) const { return PT(6, 0) + c * np(); }
};
constexpr size_t big_smem_doubles(int N) {
    return (size_t)(17 * 3 + 5) * N + (N <= BIG_PAIR_MAX ? (size_t)(6 * N + 3) * term_row(N) + 1 : 0);
}
// For a launch of systems of up to N bodies: one of 33, with its pair terms, takes
// more than one of 34 to 183 without.
constexpr size_t big_smem_doubles_up_to(int N) {
    const size_t largest = big_smem_doubles(N), pairs = big_smem_doubles(N < BIG_PAIR_MAX ? N : BIG_PAIR_MAX);
    return largest > pairs ? largest : pairs;
}
// 512 bodies are the most that an upload takes
static_assert(sizeof(double) * big_smem_doubles_up_to(512) <= 227 * 1024, "shared memory of a CTA");

// Bodies held by the Big-body CTA (Big, then massive Small bodies).
__device__ __forceinline__ int big_count(const MvsBigArgs& A) { return A.nmass > A.nbig ? A.nmass : A.nbig; }

__device__ __forceinline__ void big_sync() {
    if (blockDim.x == 32) __syncwarp();
    else __syncthreads();
}
// The items [0, n) of a job that warp w does while others do theirs (0 and 1
// the force, 2 to 5 the screens and table rows, which take as long); one-warp
// CTAs and large systems take the jobs one after another with every thread.
template <class F> __device__ __forceinline__ void big_job(int w, int N, int n, F f) {
    const bool all = blockDim.x == 32 || N > BIG_PAIR_MAX;
    if (!all && (int)(threadIdx.x >> 5) != w) return;
    const int step = all ? blockDim.x : 32;
    for (int k = all ? threadIdx.x : threadIdx.x & 31; k < n; k += step) f(k);
}
// Every (body k in [k0, k1), coordinate c), each by one thread.
template <class F> __device__ __forceinline__ void big_each(int k0, int k1, F f) {
    for (int q = threadIdx.x; q < 3 * (k1 - k0); q += blockDim.x) {
        const int j = q / 3;
        f(k0 + j, q - 3 * j);
    }
}
__device__ __forceinline__ double rsqrt_any(double x) {
    double s, r;
    sqrt_recip_any(x, s, r);
    return r;
}

// What depends on the masses alone. S.MS() is filled; synchronized before.
__device__ void big_constants(const MvsBigArgs& A, BigSmem& S) {
    if (threadIdx.x == 0) {
        double minside = S.MS()[0], mtot = 0.0;   // mtot: Big bodies inside the next one
        for (int j = 1; j < A.nbig; ++j) {
            S.GM()[j] = minside;
            minside = minside + S.MS()[j];
            S.TH()[j] = minside;
            S.MI()[j] = mtot + S.MS()[0];
            mtot = j == 1 ? S.MS()[1] : mtot + S.MS()[j];
            S.TJ()[j] = mtot;
        }
    }
    big_sync();
    for (int j = 1 + threadIdx.x; j < A.nbig; j += blockDim.x) {
        S.GM()[j] = S.MS()[0] * S.TH()[j] / S.GM()[j];
        S.TJ()[j] = S.MS()[j] / (S.TJ()[j] + S.MS()[0]);
        S.TH()[j] = 1.0 / S.MI()[j];
    }
    big_sync();
}

// Prefix sums of the products that big_products left in F0 and F2, in body
// order: A3 and OT receive, for body j, the sum over bodies 1 .. j - 1. Six
// chains of adds; eight terms are fetched at a time (past the last body's they
// are not used).
__device__ __forceinline__ void big_scan(const MvsBigArgs& A, const BigSmem& S) {
    if (threadIdx.x >= 6) return;
    const int N = S.N, nbig = A.nbig, c = threadIdx.x % 3;
    const double* t = (threadIdx.x < 3 ? S.F0() : S.F2()) + c * N;
    double* out = (threadIdx.x < 3 ? S.A3() : S.OT()) + c * N;
    if (nbig < 3) return;
    double p = t[1];
    out[2] = p;
    for (int i0 = 2; i0 < nbig - 1; i0 += 8) {
        double u[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) u[q] = t[i0 + q];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            p = p + u[q];
            if (i0 + q + 1 < nbig) out[i0 + q + 1] = p;
        }
    }
}

// mco_h2j for the Big bodies (mercury6_2.for:2613-2682) from the products m_j
// x_j, m_j v_j in F0, F2. All threads; synchronized before and after.
__device__ __forceinline__ void big_h2j(const MvsBigArgs& A, const BigSmem& S) {
    const int N = S.N;
    big_scan(A, S);
    big_sync();
    big_each(1, A.nbig, [&](int j, int c) {
        const int z = c * N + j;
        const double x = S.X()[z], v = S.V()[z], th = S.TH()[j], px = S.A3()[z], pv = S.OT()[z];
        S.XJ()[z] = j >= 2 ? x - th * px : x;
        S.VJ()[z] = j >= 2 ? v - th * pv : v;
    });
    big_sync();
}
__device__ __forceinline__ void big_products(const MvsBigArgs& A, const BigSmem& S) {
    const int N = S.N;
    big_each(1, A.nbig, [&](int j, int c) {
        const int z = c * N + j;
        S.F0()[z] = S.MS()[j] * S.X()[z];
        S.F2()[z] = S.MS()[j] * S.V()[z];
    });
    big_sync();
}

// The drift of mdt_mvs, after h2j: Kepler drift of each Jacobi Big body with
// gm_j, j2h; each massive Small body drifts heliocentrically about the central
// mass (mercury6_2.for:4031-4052). All threads.
__device__ void big_drift(const MvsBigArgs& A, BigSmem& S, double h) {
    const int nbig = A.nbig, N = big_count(A);
    // bodies dealt out to the warps: those that need the universal-variable
    // solve (the innermost planets' steps are long for them) then take no
    // other body's time
    const int nw = blockDim.x >> 5, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int k = 1 + w + nw * lane; k < N; k += blockDim.x) {
        const bool big = k < nbig;
        double* px = big ? S.XJ() : S.X();
        double* pv = big ? S.VJ() : S.V();
        double3 p = ld3(px, N, k), w = ld3(pv, N, k);
        drift_one(big ? S.GM()[k] : S.MS()[0], p, w, h);
        st3(px, N, k, p);
        st3(pv, N, k, w);
        if (big) {
            const double tj = S.TJ()[k];
            st3(S.F0(), N, k, make_double3(tj * p.x, tj * p.y, tj * p.z));
            st3(S.F2(), N, k, make_double3(tj * w.x, tj * w.y, tj * w.z));
        }
    }
    big_sync();
    // mco_j2h (mercury6_2.for:2700-2770)
    big_scan(A, S);
    big_sync();
    big_each(1, nbig, [&](int j, int c) {
        const int z = c * N + j;
        const double x = S.XJ()[z], v = S.VJ()[z], px = S.A3()[z], pv = S.OT()[z];
        S.X()[z] = j >= 2 ? x + px : x;
        S.V()[z] = j >= 2 ? v + pv : v;
    });
    big_sync();
}

// The terms of mfo_obl and mfo_ngf (rare, hence a call).
static __device__ __noinline__ void big_extra_terms(const MvsBigArgs& A, const BigSmem S, const double* V_ngf) {
    const int nbig = A.nbig, nb = nbig - 1, N = big_count(A);
    const double* m = S.MS();
    if (A.obl)
        big_job(1, N, N - 1, [&](int q) {
            const int k = 1 + q;
            const double3 ao = oblate_accel(ld3(S.X(), N, k), A.jcen, m[0]);
            const double tmp4 = m[k] / m[0];
            st3(S.AO(), N, k, ao);
            st3(S.OT(), N, k, make_double3(tmp4 * ao.x, tmp4 * ao.y, tmp4 * ao.z));
        });
    if (A.ngflag == 1 || A.ngflag == 3)
        big_job(0, N, nb, [&](int q) {
            const int k = 1 + q;
            double3 g;
            if (!nongrav_accel(ld3(S.X(), N, k), ld3(V_ngf, N, k), A.ngf + 5 * k, g)) raise_fault(A.status, 2);
            st3(S.NG(), N, k, g);
        });
}

// mfo_mvs for the Big bodies plus the indirect term a0tp that every Small
// body receives (mercury6_2.for:4946-5070), with mfo_ngf for Big bodies, in two
// parts with a barrier of the caller's between: the terms, one per thread ...
// With massive Small bodies held (A.nmass > nbig) their oblateness terms
// enter acen in body order, as mfo_obl sums over every body
// (mercury6_2.for:5176-5230); their own accelerations follow from the force
// row (small_type_force).
__device__ void big_force_terms(const MvsBigArgs& A, BigSmem& S, const double* V_ngf) {
    const int nbig = A.nbig, nb = nbig - 1, N = big_count(A);
    const double* m = S.MS();
    big_job(0, N, nb, [&](int q) {
        const int k = 1 + q;
        const double3 p = ld3(S.X(), N, k), pj = ld3(S.XJ(), N, k);
        const double r2 = p.x * p.x + p.y * p.y + p.z * p.z;
        const double rj2 = pj.x * pj.x + pj.y * pj.y + pj.z * pj.z;
        // both square roots and both quotients in flight together; operands
        // out of range (k = 1 has no Jacobi terms) take the plain statements
        double s, r, rj;
        sqrt_recip(r2, s, r);
        sqrt_recip(rj2, s, rj);
        const bool fast = root_range(r2) && root_range(rj2);
        if (!fast) {
            r = div_plain(1.0, sqrt_plain(r2));
            rj = div_plain(1.0, sqrt_plain(rj2));
        }
        const double r3 = r * r * r, rj3 = rj * rj * rj;
        const double fac0 = m[k] * r3;
        const double fac12 = m[0] * rj3;
        const double f2 = m[k] * fac12, dr = (r2 - rj2) * 0.5, mi = S.MI()[k];
        double fac2 = quotient(f2, mi, S.TH()[k]), u = quotient_of(dr, rj2, rj * rj);
        if (!(fast && mid_magnitude(mi) && (mid_magnitude(f2) || f2 == 0.0) && (mid_magnitude(dr) || dr == 0.0))) {
            fac2 = div_plain(f2, mi);
            u = div_plain(dr, rj2);
        }
        const double q2 = u * u, q3 = u * q2, q4 = q2 * q2, q5 = q2 * q3, q6 = q3 * q3, q7 = q3 * q4;
        const double fac1 = 402.1875 * q7 - 187.6875 * q6 + 86.625 * q5 - 39.375 * q4 + 17.5 * q3 - 7.5 * q2 +
                            3.0 * u - 1.0;
        st3(S.F0(), N, k, make_double3(fac0 * p.x, fac0 * p.y, fac0 * p.z));
        st3(S.A1(), N, k, k == 1 ? make_double3(0.0, 0.0, 0.0)
                               : make_double3(fac12 * (pj.x + fac1 * p.x), fac12 * (pj.y + fac1 * p.y),
                                              fac12 * (pj.z + fac1 * p.z)));
        const double3 t2 = make_double3(fac2 * pj.x, fac2 * pj.y, fac2 * pj.z);
        st3(S.F2(), N, k, t2);
        if (N <= BIG_PAIR_MAX && k >= 2) {
            S.RT(0)[k - 1] = -(fac0 * p.x);
            S.RT(1)[k - 1] = -(fac0 * p.y);
            S.RT(2)[k - 1] = -(fac0 * p.z);
            for (int j = k; j < nbig; ++j) {
                S.QT(0, j)[k - 1] = t2.x;
                S.QT(1, j)[k - 1] = t2.y;
                S.QT(2, j)[k - 1] = t2.z;
            }
        }
    });
    if (N <= BIG_PAIR_MAX) {
        // a pair (i < k) once: the difference is the later body's less the
        // earlier one's in both sums
        big_job(1, N, nb * (nb - 1) / 2, [&](int q) {
            int i = 1, rem = q;
            while (rem >= nbig - 1 - i) { rem -= nbig - 1 - i; ++i; }
            const int k = i + 1 + rem;
            const double3 pk = ld3(S.X(), N, k), pi = ld3(S.X(), N, i);
            const double dx = pk.x - pi.x, dy = pk.y - pi.y, dz = pk.z - pi.z;
            const double s2 = dx * dx + dy * dy + dz * dz;
            const double s_1 = rsqrt_any(s2);
            const double s_3 = s_1 * s_1 * s_1;
            const double fk = m[i] * s_3, fi = m[k] * s_3;
            S.PT(0, k)[i - 1] = -(fk * dx);
            S.PT(1, k)[i - 1] = -(fk * dy);
            S.PT(2, k)[i - 1] = -(fk * dz);
            S.PT(0, i)[k - 1] = fi * dx;
            S.PT(1, i)[k - 1] = fi * dy;
            S.PT(2, i)[k - 1] = fi * dz;
        });
    } else {
        big_job(1, N, nb, [&](int q) {
            const int k = 1 + q;
            const double3 pk = ld3(S.X(), N, k);
            double3 a3 = make_double3(0.0, 0.0, 0.0);
            for (int i = 1; i < nbig; ++i) {
                if (i == k) continue;
                const double3 pi = ld3(S.X(), N, i);
                const bool lower = i < k;
                const double dx = lower ? pk.x - pi.x : pi.x - pk.x;
                const double dy = lower ? pk.y - pi.y : pi.y - pk.y;
                const double dz = lower ? pk.z - pi.z : pi.z - pk.z;
                const double s2 = dx * dx + dy * dy + dz * dz;
                const double s_1 = rsqrt_any(s2);
                const double s_3 = s_1 * s_1 * s_1;
                const double fac = m[i] * s_3;
                if (lower) { a3.x = a3.x - fac * dx; a3.y = a3.y - fac * dy; a3.z = a3.z - fac * dz; }
                else { a3.x = a3.x + fac * dx; a3.y = a3.y + fac * dy; a3.z = a3.z + fac * dz; }
            }
            st3(S.A3(), N, k, a3);
        });
    }
    if (A.obl || A.ngflag == 1 || A.ngflag == 3) big_extra_terms(A, S, V_ngf);
}

// ... and their sums in mfo_mvs's order: S.ACC() = (angf + 0) + a, and the force
// row's head {a0tp, acen} (of the step's table row, or null). The caller
// synchronizes after it.
__device__ void big_force_sum(const MvsBigArgs& A, BigSmem& S, double* row) {
    const int nbig = A.nbig, N = big_count(A);
    big_each(1, nbig, [&](int k, int c) {
        const double* F0 = S.F0() + c * N;
        double a0 = 0.0, a2 = 0.0, a3 = 0.0, acen = 0.0;
        if (N <= BIG_PAIR_MAX) {
            // every term of a row, the zeros too (x + 0 is x: no sum here is
            // -0), so that nothing depends on k: three chains of adds
            const double2 *p3 = reinterpret_cast<const double2*>(S.PT(c, k)),
                          *p2 = reinterpret_cast<const double2*>(S.QT(c, k)),
                          *p0 = reinterpret_cast<const double2*>(S.RT(c));
            for (int i0 = 1; i0 < nbig; i0 += 8, p3 += 4, p2 += 4, p0 += 4) {
                double2 t3[4], t2[4], t0[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    t3[q] = p3[q];
                    t2[q] = p2[q];
                    t0[q] = p0[q];
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    a3 = a3 + t3[q].x;
                    a2 = a2 + t2[q].x;
                    a0 = a0 + t0[q].x;
                    a3 = a3 + t3[q].y;
                    a2 = a2 + t2[q].y;
                    a0 = a0 + t0[q].y;
                }
            }
        } else {
            for (int i = 2; i < nbig; ++i) a0 = a0 - F0[i];
            for (int i = 2; i <= k; ++i) a2 = a2 + S.F2()[c * N + i];
            a3 = S.A3()[c * N + k];
        }
        double a = a0 + S.A1()[c * N + k] + a2 + a3;
        if (A.obl) {
            for (int i = 1; i < N; ++i) acen = acen - S.OT()[c * N + i];
            a = a + (S.AO()[c * N + k] - acen);
        }
        if (A.ngflag == 1 || A.ngflag == 3) a = S.NG()[c * N + k] + 0.0 + a;
        if (!isfinite(a)) raise_fault(A.status, 1);
        S.ACC()[c * N + k] = a;
        if (k == 1) {
            row[c] = a0 - F0[1];
            row[3 + c] = acen;
        }
    });
    if (nbig < 2)
        for (int c = threadIdx.x; c < 3; c += blockDim.x) {
            double acen = 0.0;
            if (A.obl)
                for (int i = 1; i < N; ++i) acen = acen - S.OT()[c * N + i];
            row[c] = 0.0;
            row[3 + c] = acen;
        }
}

// Force rows {x, m} of the Big bodies.
__device__ void write_force_rows(const MvsBigArgs& A, const BigSmem& S, double* row) {
    const int N = big_count(A);
    big_job(5, N, A.nbig - 1, [&](int q) {
        double* b = row + TAB_HEAD + q * TAB_BODY;
        b[0] = S.X()[q + 1];
        b[1] = S.X()[N + q + 1];
        b[2] = S.X()[2 * N + q + 1];
        b[3] = S.MS()[q + 1];
    });
}

// Accelerations of the massive Small bodies held by the CTA: the particles'
// mfo_mvs + mfo_ngf statements (small_body_force) against the force row just
// written. All threads; the row must be visible (after big_sync).
static __device__ __noinline__ void small_type_force(const MvsBigArgs& A, const BigSmem S, const double* row,
                                                     const double* V_ngf) {
    const int nbig = A.nbig, N = big_count(A), nb = nbig - 1;
    const bool ngf = A.ngflag == 1 || A.ngflag == 3;
    for (int k = nbig + threadIdx.x; k < N; k += blockDim.x) {
        const double3 x = ld3(S.X(), N, k), v = ld3(V_ngf, N, k);
        auto g = [&](int c) -> double { return A.ngf[5 * k + c]; };
        double3 a;
        if (ngf) a = A.obl ? small_body_force<true, true>(x, v, g, row, nb, A.jcen, A.m[0], A.status)
                           : small_body_force<true, false>(x, v, g, row, nb, A.jcen, A.m[0], A.status);
        else a = A.obl ? small_body_force<false, true>(x, v, g, row, nb, A.jcen, A.m[0], A.status)
                       : small_body_force<false, false>(x, v, g, row, nb, A.jcen, A.m[0], A.status);
        st3(S.ACC(), N, k, a);
    }
    big_sync();
}

// The whole force: terms, sums, table row. All threads; synchronized after.
__device__ void big_force(const MvsBigArgs& A, BigSmem& S, double* row) {
    big_force_terms(A, S, S.V());
    write_force_rows(A, S, row);
    big_sync();
    big_force_sum(A, S, row);
    big_sync();
    if (big_count(A) > A.nbig) small_type_force(A, S, row, S.V());
}

__device__ void big_load(const MvsBigArgs& A, BigSmem& S, double* smem) {
    const int N = big_count(A), tid = threadIdx.x, nt = blockDim.x;
    if (A.fresh_status && tid == 0) *A.status = DeviceStatus{};   // big_constants synchronizes
    S.base = smem;
    S.N = N;
    S.now = 0;
    for (int q = tid; q < 3 * N; q += nt) {
        S.X()[q] = A.in.x[q];
        S.V()[q] = A.in.v[q];
        S.ACC()[q] = A.in.a[q];
    }
    for (int k = tid; k < N; k += nt) S.MS()[k] = A.m[k];
    if (N <= BIG_PAIR_MAX)
        for (int q = tid; q < (6 * N + 3) * term_row(N); q += nt) S.PT(0, 0)[q] = 0.0;
    big_sync();
    big_constants(A, S);
}

// Boxes, details and mce_stat's pairs of step s (start states X0, V0 after the
// kick, end states X, V after the drift): jobs for the warps beside the force.
__device__ void big_screen(const MvsBigArgs& A, BigSmem& S, int s, double* row, double* det) {
    const int nbig = A.nbig, N = big_count(A), nb = nbig - 1;
    const double h = A.h, hm1 = 1.0 / h;
    big_job(2, N, nb, [&](int q) {
        const int k = 1 + q;
        double* b = row + TAB_HEAD + q * TAB_BODY;
        const double pad = A.rce[k] * 1.2;
        double xlo, xhi, ylo, yhi;
        box_extent(S.X0()[k], S.X()[k], S.V0()[k], S.V()[k], h, xlo, xhi);
        box_extent(S.X0()[N + k], S.X()[N + k], S.V0()[N + k], S.V()[N + k], h, ylo, yhi);
        xlo = xlo - pad; xhi = xhi + pad; ylo = ylo - pad; yhi = yhi + pad;
        b[4] = xlo; b[5] = xhi; b[6] = ylo; b[7] = yhi;
        reinterpret_cast<int4*>(row + TAB_HEAD + TAB_BODY * nb)[q] =
            make_int4(order_key(xlo) - 1, order_key(xhi), order_key(ylo) - 1, order_key(yhi));
        double* d = det + q * TAB_DETAIL;
        for (int c = 0; c < 3; ++c) {
            d[c] = S.X0()[c * N + k];
            d[3 + c] = S.V0()[c * N + k];
            d[6 + c] = S.X()[c * N + k];
            d[9 + c] = S.V()[c * N + k];
        }
        d[12] = A.rce[k];
        d[13] = A.rphys[k];
    });
    // mce_stat between Big bodies (pairs 1 <= i < j < nbig), then between
    // Big bodies and the massive Small bodies held (i < nbig <= j < N).
    const int npair_big = nb * (nb - 1) / 2;
    big_job(3, N, npair_big + nb * (N - nbig), [&](int q) {
        int i = 1, j;
        if (q < npair_big) {
            int rem = q;
            while (rem >= nbig - 1 - i) { rem -= nbig - 1 - i; ++i; }
            j = i + 1 + rem;
        } else {
            const int r = q - npair_big;
            i = 1 + r / (N - nbig);
            j = nbig + r % (N - nbig);
        }
        double lo_i, hi_i, lo_j, hi_j, ylo_i, yhi_i, ylo_j, yhi_j;
        const double pi_ = A.rce[i] * 1.2, pj_ = A.rce[j] * 1.2;
        box_extent(S.X0()[i], S.X()[i], S.V0()[i], S.V()[i], h, lo_i, hi_i);
        box_extent(S.X0()[N + i], S.X()[N + i], S.V0()[N + i], S.V()[N + i], h, ylo_i, yhi_i);
        box_extent(S.X0()[j], S.X()[j], S.V0()[j], S.V()[j], h, lo_j, hi_j);
        box_extent(S.X0()[N + j], S.X()[N + j], S.V0()[N + j], S.V()[N + j], h, ylo_j, yhi_j);
        lo_i = lo_i - pi_; hi_i = hi_i + pi_; ylo_i = ylo_i - pi_; yhi_i = yhi_i + pi_;
        lo_j = lo_j - pj_; hi_j = hi_j + pj_; ylo_j = ylo_j - pj_; yhi_j = yhi_j + pj_;
        if (!(hi_i >= lo_j && hi_j >= lo_i && yhi_i >= ylo_j && yhi_j >= ylo_i)) return;
        PairEnds I{ld3(S.X0(), N, i), ld3(S.V0(), N, i), ld3(S.X(), N, i), ld3(S.V(), N, i)};
        PairEnds J{ld3(S.X0(), N, j), ld3(S.V0(), N, j), ld3(S.X(), N, j), ld3(S.V(), N, j)};
        PairClass pc;
        if (!pair_classify(I, J, A.rce[i], A.rce[j], A.rphys[i], A.rphys[j], h, pc)) return;
        const int slot = atomicAdd(&A.status->events, 1);
        if (slot < A.event_cap) {
            pair_record(A.events + slot, I, J, pc, hm1, i + 1, j + 1, A.m[j] > A.m[i] && j < nbig);
            A.event_step[slot] = A.step0 + s;
            if (A.event_sys) A.event_sys[slot] = A.sys;
        } else {
            atomicExch(&A.status->overflow, 1);
        }
    });
}

// mce_cent over step s: its start state is in XS/VS[s & 1], its end state in
// XS/VS of the next step.
__device__ void big_central(const MvsBigArgs& A, BigSmem& S, int s) {
    const int N = big_count(A);
    const double *x0 = S.XS(s & 1), *v0 = S.VS(s & 1), *x1 = S.XS(~s & 1), *v1 = S.VS(~s & 1);
    big_job(4, N, N - 1, [&](int q) {
        const int k = 1 + q;
        double temp;
        if (!central_impact(ld3(x0, N, k), ld3(v0, N, k), ld3(x1, N, k), ld3(v1, N, k), A.m[0], A.m[k], A.h, A.rcen,
                            temp))
            return;
        const int slot = atomicAdd(&A.status->events, 1);
        if (slot < A.event_cap) {
            MercuryEvent rec = {};
            rec.i = 1;
            rec.j = k + 1;
            rec.kind = EV_CENTRAL;
            rec.time = temp;
            rec.distance = A.rcen;
            store_event(A.events + slot, rec);
            A.event_step[slot] = A.step0 + s;
            if (A.event_sys) A.event_sys[slot] = A.sys;
        } else {
            atomicExch(&A.status->overflow, 1);
        }
    });
}

// The Big-body integrator of one system (all threads of the CTA), with the
// massive Small bodies it holds (A.nmass > nbig).
__device__ void big_run(const MvsBigArgs& A, double* smem) {
    const int nbig = A.nbig, N = big_count(A), nb = nbig - 1;
    const int stride = tab_stride(nb);
    BigSmem S;
    big_load(A, S, smem);
    const double hby2 = 0.5 * A.h;
    // step -1 is the force alone, for the first kick of a fresh start
    for (int s = A.reset ? -1 : 0; s < A.nsteps; ++s) {
        double* row = A.tab + (size_t)(s + 1) * stride;
        if (s >= 0) {
            S.now = s & 1;
            double *XS = S.XS(S.now), *VS = S.VS(S.now);
            big_each(1, N, [&](int k, int c) {
                const int z = c * N + k;
                const double x = S.X()[z], v = S.V()[z], m = S.MS()[k];
                XS[z] = x;
                VS[z] = v;
                const double v0 = v + hby2 * S.ACC()[z];
                S.V()[z] = v0;
                S.V0()[z] = v0;
                S.F0()[z] = m * x;
                S.F2()[z] = m * v0;
            });
            big_sync();
        } else {
            big_products(A, S);
        }
        big_h2j(A, S);
        if (s >= 0) big_drift(A, S, A.h);
        big_force_terms(A, S, S.V());
        write_force_rows(A, S, row);
        if (s >= 0) big_screen(A, S, s, row, A.detail + (size_t)s * nb * TAB_DETAIL);
        if (A.central && s > 0) big_central(A, S, s - 1);
        big_sync();
        big_force_sum(A, S, row);
        big_sync();
        if (N > nbig) small_type_force(A, S, row, S.V());
        // each thread kicks the entries it takes into the next step itself
        if (s >= 0)
            big_each(1, N, [&](int k, int c) {
                const int z = c * N + k;
                S.V()[z] = S.V()[z] + hby2 * S.ACC()[z];
            });
    }
    if (A.central && A.nsteps > 0) {
        double *XS = S.XS(A.nsteps & 1), *VS = S.VS(A.nsteps & 1);
        big_each(1, N, [&](int k, int c) {
            const int z = c * N + k;
            XS[z] = S.X()[z];
            VS[z] = S.V()[z];
        });
        big_sync();
        big_central(A, S, A.nsteps - 1);
    }
    big_sync();
    for (int q = threadIdx.x; q < 3 * N; q += blockDim.x) {
        A.out.x[q] = S.X()[q];
        A.out.v[q] = S.V()[q];
        A.out.a[q] = S.ACC()[q];
    }
}

__global__ void __launch_bounds__(BIG_THREADS, 1) mvs_big_kernel(const __grid_constant__ MvsBigArgs A) {
    extern __shared__ double smem[];
    big_run(A, smem);
}

// ------------------------------------------------------------ test particles
// Warp-aggregated slot claim: one atomic per warp, slots in lane order by a
// ballot prefix count; -1 for lanes without a record or beyond capacity.
// Must be reached by all 32 lanes.
__device__ __forceinline__ int claim_slot(bool has, int cap, DeviceStatus* st, int* counter, int overflow_bit) {
    const unsigned mask = __ballot_sync(FULL, has);
    if (mask == 0) return -1;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(mask) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(counter, __popc(mask));
    base = __shfl_sync(FULL, base, leader);
    if (!has) return -1;
    const int slot = base + __popc(mask & ((1u << lane) - 1u));
    if (slot >= cap) {
        atomicOr(&st->overflow, overflow_bit);
        return -1;
    }
    return slot;
}

// Thread-private shared-memory columns of the particle kernels, one double per
// thread per column (column-major, so the lanes of a warp hit distinct banks).
// Only x, v, the cached acceleration and |x|^2 live in registers; what a step
// needs again after the drift waits here, which keeps the drift's register
// footprint small.
template <int STRIDE_> struct ColsOf {
    static constexpr int X0 = 0;       // 3: state after the first kick
    static constexpr int V0 = 3;       // 3
    static constexpr int VS = 6;       // 3: velocity at the start of the step (mce_cent)
    static constexpr int PAD = 9;      // 1.2 rce, mce_stat's margin
    static constexpr int NGF = 10;     // 5 coefficients
    __host__ __device__ static constexpr int count(bool ngf) { return ngf ? 15 : 10; }
    // column stride: the kernel's largest CTA, so that a column offset is a
    // constant (base already points at the thread's own entry)
    static constexpr int STRIDE = STRIDE_;
    volatile double* base;
    __device__ volatile double& at(int c) const { return base[c * STRIDE]; }
    __device__ double3 ld3(int c) const { return make_double3(at(c), at(c + 1), at(c + 2)); }
    __device__ void st3(int c, double3 v) const { at(c) = v.x; at(c + 1) = v.y; at(c + 2) = v.z; }
};

using Cols = ColsOf<128>;

// A particle between steps: what the next step takes from the one before.
struct Particle {
    double3 x, v, acc;
    double rr;          // |x|^2
    int kx, ky;         // order_key of x.x and x.y
    int rv;             // high word of x.v
    bool padded;        // rce != 0
    __device__ void derive() {
        rr = x.x * x.x + x.y * x.y + x.z * x.z;
        kx = order_key(x.x);
        ky = order_key(x.y);
        rv = __double2hiint(v.x * x.x + v.y * x.y + v.z * x.z);
    }
};

// What a step needs of its system.
struct StepEnv {
    double mu, rmu, h, hby2, rcen;
    int nb;
};

// Keys of a coordinate's extent over the step when the velocity turns within
// it (mce_box then adds the interpolated turning point) or the body has a
// margin of its own: an interval that contains mce_box's. The turning point is
// within |a1 - a0| + |h| min(|u0|, |u1|) / 2 of an end, without the division
// (1/16 more covers the roundings).
__device__ __forceinline__ void wide_keys(double a0, double a1, double u0, double u1, double h, double pad, int& klo,
                                          int& khi) {
    double e = pad;
    if ((__double2hiint(u0) ^ __double2hiint(u1)) < 0)
        e = e + 1.0625 * (fabs(a1 - a0) + 0.5 * fabs(h) * fmin(fabs(u0), fabs(u1)));
    klo = order_key(fmin(a0, a1) - e) - 1;
    khi = order_key(fmax(a0, a1) + e);
}

// The bodies of keys[0 .. n), n <= 32, whose box may overlap [kxlo, kxhi] x
// [kylo, kyhi], as a bit mask. Four compares chained through one predicate and
// one predicated OR a body.
__device__ __forceinline__ unsigned overlap_mask(const int4* keys, int n, int kxlo, int kxhi, int kylo, int kyhi) {
    unsigned mask = 0;
    auto test = [&](int b, unsigned bit) {
        const int4 k = keys[b];
        asm("{\n\t.reg .pred p;\n\t"
            "setp.ge.s32 p, %1, %2;\n\t"
            "setp.ge.and.s32 p, %3, %4, p;\n\t"
            "setp.ge.and.s32 p, %5, %6, p;\n\t"
            "setp.ge.and.s32 p, %7, %8, p;\n\t"
            "@p or.b32 %0, %0, %9;\n\t}"
            : "+r"(mask)
            : "r"(k.y), "r"(kxlo), "r"(kxhi), "r"(k.x), "r"(k.w), "r"(kylo), "r"(kyhi), "r"(k.z), "r"(bit));
    };
    // the usual planetary system without a loop, whose counter and branches are
    // 2.5 % of the kernel (1M particles, 160 steps: 8.78 ms so, 9.00 with the loop,
    // 8.90 with it unrolled by four)
    if (n == 8) {
#pragma unroll
        for (int b = 0; b < 8; ++b) test(b, 1u << b);
    } else {
#pragma unroll 1
        for (int b = 0; b < n; ++b) test(b, 1u << b);
    }
    return mask;
}

// One mdt_mvs step of one Small body: kick, Kepler drift, mce_stat's box
// screen, interaction force, kick, mce_cent. T holds the step's head, the
// bodies' force rows (ROW doubles apart) and their box keys; G the table row
// with the exact boxes. found(b, P, x0, v0) is called by the whole warp for
// each body with the lanes whose exact boxes overlap, struck(hit, time) once a
// step.
//
// The screens run in two passes. The first compares integers: order_key()
// keeps the order of doubles by their high words (a >= b implies key(a) >=
// key(b) - 1), and x at the step's start, |x|^2 and x.v come from the step
// before. What passes is tested with mce_box's and mce_cent's own statements.
// The kernel issues an FP64 instruction every other cycle and another kind in
// between, so both kinds count. Per warp-step of the benchmark's mixture of
// orbits, 8 planets: 729 FP64 of 1,535 instructions with exact boxes compared on
// the FP64 pipe and IEEE division calls, 564 of 1,116 so; 1M particles, 16 steps:
// 1.45 ms a launch before, 0.93 now.
template <bool NGF, bool OBL, bool CENTRAL, int ROW, class Cols, class Found, class Struck>
__device__ __forceinline__ void particle_step(Particle& P, bool ok, const Cols& cols, const double* T,
                                              const double* G, const StepEnv& E, const double* jcen,
                                              DeviceStatus* status, double mass, Found&& found, Struck&& struck) {
    double3& x = P.x;
    double3& v = P.v;
    const int nb = E.nb;
    const double h = E.h;
    int kxlo = 0, kxhi = 0, kylo = 0, kyhi = 0;
    const int rr0 = __double2hiint(P.rr), rv0 = P.rv;
    if (ok) {
        if (CENTRAL) cols.st3(Cols::VS, v);
        v.x = v.x + E.hby2 * P.acc.x;
        v.y = v.y + E.hby2 * P.acc.y;
        v.z = v.z + E.hby2 * P.acc.z;
        const int ux = __double2hiint(v.x), uy = __double2hiint(v.y);
        cols.st3(Cols::X0, x);
        cols.st3(Cols::V0, v);
        drift_one(E.mu, E.rmu, x, v, h, P.rr);
        P.rr = x.x * x.x + x.y * x.y + x.z * x.z;
        const int kx = order_key(x.x), ky = order_key(x.y);
        kxlo = min(P.kx, kx) - 1;
        kxhi = max(P.kx, kx);
        kylo = min(P.ky, ky) - 1;
        kyhi = max(P.ky, ky);
        P.kx = kx;
        P.ky = ky;
        if ((ux ^ __double2hiint(v.x)) < 0 || P.padded)
            wide_keys(cols.at(Cols::X0), x.x, cols.at(Cols::V0), v.x, h, cols.at(Cols::PAD), kxlo, kxhi);
        if ((uy ^ __double2hiint(v.y)) < 0 || P.padded)
            wide_keys(cols.at(Cols::X0 + 1), x.y, cols.at(Cols::V0 + 1), v.y, h, cols.at(Cols::PAD), kylo, kyhi);
    }
    for (int b0 = 0; b0 < nb; b0 += 32) {
        const int4* keys = reinterpret_cast<const int4*>(T + TAB_HEAD + ROW * nb) + b0;
        unsigned maybe = overlap_mask(keys, min(32, nb - b0), kxlo, kxhi, kylo, kyhi);
        if (!ok) maybe = 0;
        unsigned any = __reduce_or_sync(FULL, maybe);
        if (any == 0) continue;
        double bxlo = 0.0, bxhi = 0.0, bylo = 0.0, byhi = 0.0;
        const double3 x0 = cols.ld3(Cols::X0), v0 = cols.ld3(Cols::V0);
        if (maybe) {
            box_extent(x0.x, x.x, v0.x, v.x, h, bxlo, bxhi);
            box_extent(x0.y, x.y, v0.y, v.y, h, bylo, byhi);
            const double pad = cols.at(Cols::PAD);
            bxlo = bxlo - pad;
            bxhi = bxhi + pad;
            bylo = bylo - pad;
            byhi = byhi + pad;
        }
        do {
            const int b = __ffs(any) - 1;
            any &= any - 1;
            const double* row = G + TAB_HEAD + (b0 + b) * TAB_BODY;
            found(((maybe >> b) & 1u) && row[5] >= bxlo && bxhi >= row[4] && row[7] >= bylo && byhi >= row[6], b0 + b,
                  x0, v0);
        } while (any);
    }
    if (ok) {
        P.acc = small_body_force<NGF, OBL, ROW>(
            x, v, [&](int c) -> double { return cols.at(Cols::NGF + c); }, T, nb, jcen, E.mu, status);
        v.x = v.x + E.hby2 * P.acc.x;
        v.y = v.y + E.hby2 * P.acc.y;
        v.z = v.z + E.hby2 * P.acc.z;
    }
    if (CENTRAL) {
        // mce_cent's first test, (rv0 h <= 0 and rv1 h >= 0) or min |x|^2 <=
        // rcen^2, on high words: signs, with numbers that a product with h
        // could flush to zero (below 2^-767) counted as both
        P.rv = __double2hiint(v.x * x.x + v.y * x.y + v.z * x.z);
        const int hs = __double2hiint(h) & 0x80000000;
        double temp = 0.0;
        bool hit = false;
        if (ok && (((rv0 ^ hs) < 0x10000000 && (unsigned)(P.rv ^ hs) < 0x90000000u) ||
                   min(rr0, __double2hiint(P.rr)) <= __double2hiint(E.rcen * E.rcen) || fabs(h) < 1e-60)) {
            // a pericentre inside rcen needs |x0 x v0|^2 <= rcen^2 (v0^2 - 2 M
            // / r0) + 2 M rcen (the speed an orbit has at rcen): most passages
            // end here, without the square roots and divisions of the rest
            const CentralStart c = central_start(cols.ld3(Cols::X0), cols.ld3(Cols::VS));
            const double rcen2 = E.rcen * E.rcen;
            if (c.rr0 <= rcen2 || c.h2 <= 1.001 * (rcen2 * c.v2 + 2.0 * (E.mu + mass) * E.rcen))
                hit = central_finish(c, x, v, E.mu, mass, h, E.rcen, temp);
        }
        struck(hit, temp);
    }
}

// A central-body record (it carries no states: xi = xj = 0).
__device__ __forceinline__ void central_record(MercuryEvent* e, int id, double rcen, double temp) {
    *reinterpret_cast<int4*>(e) = make_int4(1, id, EV_CENTRAL, 0);
    reinterpret_cast<double2*>(e)[1] = make_double2(rcen, temp);
    for (int k = 2; k < 8; ++k) reinterpret_cast<double2*>(e)[k] = make_double2(0.0, 0.0);
}
__device__ __forceinline__ void candidate_record(EncounterCandidate* c, int4 head, double rce, double rphys,
                                                 double3 x0, double3 v0, double3 x, double3 v) {
    *reinterpret_cast<int4*>(c) = head;
    double2* w = reinterpret_cast<double2*>(c);
    w[1] = make_double2(rce, rphys);
    w[2] = make_double2(x0.x, x0.y);
    w[3] = make_double2(x0.z, v0.x);
    w[4] = make_double2(v0.y, v0.z);
    w[5] = make_double2(x.x, x.y);
    w[6] = make_double2(x.z, v.x);
    w[7] = make_double2(v.y, v.z);
}

// Rows of the Big bodies staged in shared memory: a table row without the
// exact boxes, {head, x y z m per body, box keys}.
constexpr int SROW_BODY = 4;
__host__ __device__ constexpr int srow_stride(int nb) { return TAB_HEAD + (SROW_BODY + TAB_KEYS) * nb; }

// Test-particle kernel: one particle slot per thread through all K steps; the
// Big-body rows of the K steps are staged in shared memory once per CTA.
//
// One slot per thread, not two: a warp's time on a tile is the time of its
// slowest particle, and a tile of particles that need the universal-variable
// drift takes several times an ordinary one. With two particles in turn in
// each thread such a tile alone took the whole launch (1M particles, 16 steps: 1.52 ms of a
// 1.52 ms launch; one slot a thread, 0.97 ms).
template <bool NGF, bool OBL, bool CENTRAL>
__global__ void __launch_bounds__(128, MB200_PARTICLE_MIN_BLOCKS) mvs_particle_kernel(MvsParticleArgs A) {
    extern __shared__ double smem[];
    const int nb = A.nb, gstride = tab_stride(nb), stride = srow_stride(nb);
    const int rows = A.nsteps + (A.reset ? 1 : 0);
    double* stab = smem;
    const Cols cols{smem + (size_t)rows * stride + threadIdx.x};
    const double* gtab = A.tab + (A.reset ? 0 : gstride);
    {
        // 16 bytes at a time: unit u of a staged row is the head's, a body's
        // half force row or a body's keys
        const int units = stride / 2, gunits = gstride / 2;
        const double2* src = reinterpret_cast<const double2*>(gtab);
        double2* dst = reinterpret_cast<double2*>(stab);
        for (int k = threadIdx.x; k < rows * units; k += blockDim.x) {
            const int r = k / units, u = k - r * units, q = u - TAB_HEAD / 2;
            const int g = q < 0 ? u : q < 2 * nb ? TAB_HEAD / 2 + (q >> 1) * (TAB_BODY / 2) + (q & 1)
                                                 : TAB_HEAD / 2 + nb * (TAB_BODY / 2) + (q - 2 * nb);
            dst[k] = src[(size_t)r * gunits + g];
        }
    }
    __syncthreads();
    const double* steps_tab = stab + (A.reset ? stride : 0);
    const double* steps_gtab = A.tab + gstride;
    const StepEnv E{A.mu, A.rmu, A.h, 0.5 * A.h, A.rcen, nb};
    const int lane = threadIdx.x & 31;
    // Warps claim tiles of 32 slots from a launch-wide counter: slots are ordered
    // slowest-first (Newton-path particles lead), so claiming dynamically
    // balances the SMs (longest-processing-time-first).
    const int ntiles = (A.np + 31) >> 5;
    const size_t S = A.npcap;
    int* const tiles = A.tiles ? A.tiles : &A.status->next_tile;
    for (;;) {
        int tile = 0;
        if (lane == 0) tile = atomicAdd(tiles, 1);
        tile = __shfl_sync(FULL, tile, 0);
        if (tile >= ntiles) break;
        const int p = tile * 32 + lane;
        const bool ok = p < A.np;
        Particle P{};
        if (ok) {
            const double* in = A.xin + p;
            P.x = make_double3(in[0], in[S], in[2 * S]);
            P.v = make_double3(in[3 * S], in[4 * S], in[5 * S]);
            P.acc = make_double3(in[6 * S], in[7 * S], in[8 * S]);
            const double pad = A.rce[p] * 1.2;
            cols.at(Cols::PAD) = pad;
            P.padded = pad != 0.0;
            if (NGF)
                for (int c = 0; c < 5; ++c) cols.at(Cols::NGF + c) = A.ngf[c * S + p];
            if (A.reset)
                P.acc = small_body_force<NGF, OBL, SROW_BODY>(
                    P.x, P.v, [&](int c) -> double { return cols.at(Cols::NGF + c); }, stab, nb, A.jcen, A.mu,
                    A.status);
            P.derive();
        }
#pragma unroll 1
        for (int s = 0; s < A.nsteps; ++s)
            particle_step<NGF, OBL, CENTRAL, SROW_BODY>(
                P, ok, cols, steps_tab + s * stride, steps_gtab + (size_t)s * gstride, E, A.jcen, A.status,
                CENTRAL && ok ? A.m[p] : 0.0,
                [&](bool cand, int b, double3 x0, double3 v0) {
                    const int slot = claim_slot(cand, A.cand_cap, A.status, &A.status->cands, 2);
                    if (slot >= 0)
                        candidate_record(A.cands + slot, make_int4(p, b, A.step0 + s, A.nbig + A.perm[p] + 1),
                                         A.rce[p], A.rphys[p], x0, v0, P.x, P.v);
                },
                [&](bool hit, double temp) {
                    const int slot = claim_slot(hit, A.event_cap, A.status, &A.status->events, 1);
                    if (slot >= 0) {
                        central_record(A.events + slot, A.nbig + A.perm[p] + 1, A.rcen, temp);
                        A.event_step[slot] = A.step0 + s;
                    }
                });
        if (ok) {
            double* out = A.xout + p;
            out[0] = P.x.x;
            out[S] = P.x.y;
            out[2 * S] = P.x.z;
            out[3 * S] = P.v.x;
            out[4 * S] = P.v.y;
            out[5 * S] = P.v.z;
            out[6 * S] = P.acc.x;
            out[7 * S] = P.acc.y;
            out[8 * S] = P.acc.z;
            if (A.rows_x) {
                // rows in particle order for the copy back to the host
                const size_t i = 3 * (size_t)A.perm[p];
                A.rows_x[i] = P.x.x;
                A.rows_x[i + 1] = P.x.y;
                A.rows_x[i + 2] = P.x.z;
                A.rows_v[i] = P.v.x;
                A.rows_v[i + 1] = P.v.y;
                A.rows_v[i + 2] = P.v.z;
            }
        }
    }
}

// ------------------------------------------------------------ output corrector
// The Big bodies' part of the corrector (mercury6_2.for:2200-2222 in
// mco_mvs2h, 2510-2532 in mco_h2mvs) from big.in into big.out, writing the
// force table of each of the four kicks.
__global__ void __launch_bounds__(BIG_THREADS, 1) mvs_corrector_big_kernel(const __grid_constant__ MvsBigArgs A, const __grid_constant__ CorrectorArgs K) {
    extern __shared__ double smem[];
    const int N = big_count(A);
    const int stride = tab_stride(A.nbig - 1);
    BigSmem S;
    big_load(A, S, smem);
    auto kick = [&](double hk, bool subtract) {
        big_each(1, N, [&](int k, int c) {
            const int z = c * N + k;
            const double term = hk * S.ACC()[z];
            S.V()[z] = subtract ? S.V()[z] - term : S.V()[z] + term;
        });
        big_sync();
    };
    // drift ha, kick, drift -2 ha, kick, drift ha, twice
#pragma unroll 1
    for (int q = 0; q < 6; ++q) {
        const int k = q / 3, part = q - 3 * k;
        big_products(A, S);
        big_h2j(A, S);
        big_drift(A, S, part == 1 ? -2.0 * K.ha[k] : K.ha[k]);
        if (part == 2) continue;
        big_force(A, S, A.tab + (size_t)(2 * k + part) * stride);
        kick(K.hb[k], part == 0 ? K.forward != 0 : K.forward == 0);
    }
    for (int q = threadIdx.x; q < 3 * N; q += blockDim.x) {
        A.out.x[q] = S.X()[q];
        A.out.v[q] = S.V()[q];
    }
}

// The Small bodies' part: heliocentric drifts with the central mass and the
// mfo_mvs + mfo_ngf kicks against the Big-body tables; one thread per slot.
template <bool NGF, bool OBL>
__global__ void __launch_bounds__(128) mvs_corrector_particle_kernel(CorrectorArgs K) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x, S = K.npcap;
    if (p >= K.np) return;
    const int stride = tab_stride(K.nb);
    double3 x = make_double3(K.xin[p], K.xin[S + p], K.xin[2 * S + p]);
    double3 v = make_double3(K.xin[3 * S + p], K.xin[4 * S + p], K.xin[5 * S + p]);
    auto g = [&](int c) -> double { return K.ngf[(size_t)c * S + p]; };
    auto kick = [&](const double* T, double hk, bool subtract) {
        const double3 a = small_body_force<NGF, OBL>(x, v, g, T, K.nb, K.jcen, K.mu, K.status);
        v.x = subtract ? v.x - hk * a.x : v.x + hk * a.x;
        v.y = subtract ? v.y - hk * a.y : v.y + hk * a.y;
        v.z = subtract ? v.z - hk * a.z : v.z + hk * a.z;
    };
#pragma unroll 1
    for (int k = 0; k < 2; ++k) {
        drift_one(K.mu, x, v, K.ha[k]);
        kick(K.tab + (size_t)(2 * k) * stride, K.hb[k], K.forward != 0);
        drift_one(K.mu, x, v, -2.0 * K.ha[k]);
        kick(K.tab + (size_t)(2 * k + 1) * stride, K.hb[k], K.forward == 0);
        drift_one(K.mu, x, v, K.ha[k]);
    }
    K.xout[p] = x.x;
    K.xout[S + p] = x.y;
    K.xout[2 * S + p] = x.z;
    K.xout[3 * S + p] = v.x;
    K.xout[4 * S + p] = v.y;
    K.xout[5 * S + p] = v.z;
}

// mce_stat's test for each encounter candidate of the last launch
// (mercury6_2.for:1815-1908) and the record it produces.
__global__ void __launch_bounds__(256) classify_kernel(ClassifyArgs A) {
    const int count = min(A.status->cands, A.cand_cap);
    const double hm1 = 1.0 / A.h;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) {
        const EncounterCandidate& c = A.cands[k];
        const double* d = A.detail + ((size_t)c.step * A.nb + c.body) * TAB_DETAIL;
        const PairEnds I{make_double3(d[0], d[1], d[2]), make_double3(d[3], d[4], d[5]),
                         make_double3(d[6], d[7], d[8]), make_double3(d[9], d[10], d[11])};
        const PairEnds J{make_double3(c.x0[0], c.x0[1], c.x0[2]), make_double3(c.v0[0], c.v0[1], c.v0[2]),
                         make_double3(c.x1[0], c.x1[1], c.x1[2]), make_double3(c.v1[0], c.v1[1], c.v1[2])};
        PairClass pc;
        if (!pair_classify(I, J, d[12], c.rce, d[13], c.rphys, A.h, pc)) continue;
        const int slot = atomicAdd(&A.status->events, 1);
        if (slot < A.event_cap) {
            pair_record(A.events + slot, I, J, pc, hm1, c.body + 2, c.id, false);
            A.event_step[slot] = c.step + A.step_base;
        } else {
            atomicOr(&A.status->overflow, 1);
        }
    }
}

// ------------------------------------------------------------ batched systems
__global__ void __launch_bounds__(32, 1) mvs_big_batch_kernel(BatchBigArgs B) {
    extern __shared__ double smem[];
    const int q = blockIdx.x;
    // in shared memory: registers and local copies of it would be read slower
    __shared__ MvsBigArgs A;
    if (threadIdx.x == 0) {
        A = B.proto[q];
        if (B.flip) {
            const BigState t = A.in;
            A.in = A.out;
            A.out = t;
        }
        A.nsteps = B.nsteps;
        A.reset = B.reset;
        A.central = B.central;
        A.step0 = B.step0;
        A.rcen = B.rcen;
        A.tab = B.tab + B.sys[q].tab_off;
        A.detail = B.detail + B.sys[q].det_off;
        A.events = B.events;
        A.event_step = B.event_step;
        A.event_sys = B.event_sys;
        A.event_cap = B.event_cap;
        A.status = B.status;
        A.sys = q;
    }
    __syncwarp();
    big_run(A, smem);
}

// Every test particle of every system: warps claim 32-slot tiles (each of a
// single system) from a launch-wide counter and run K steps per particle in
// registers (particle_step above); the step tables are read through the cache.
template <bool CENTRAL, int THREADS>
__global__ void __launch_bounds__(THREADS, 128 * MB200_PARTICLE_MIN_BLOCKS / THREADS)
    mvs_particle_batch_kernel(BatchParticleArgs A) {
    using Cols = ColsOf<THREADS>;
    __shared__ double col_mem[THREADS * Cols::count(false)];
    const Cols cols{col_mem + threadIdx.x};
    const int lane = threadIdx.x & 31;
    const size_t S2 = A.npcap;
    for (;;) {
        int tile = 0;
        if (lane == 0) tile = atomicAdd(&A.status->next_tile, 1);
        tile = __shfl_sync(FULL, tile, 0);
        if (tile >= A.ntiles) break;
        const BatchTile t = A.tiles[tile];
        const BatchSys S = A.sys[t.sys];
        const bool ok = lane < t.count;
        const int p = t.first + (ok ? lane : 0);
        const int stride = tab_stride(S.nb);
        const double* tab = A.tab + S.tab_off;
        const StepEnv E{S.mu, recip_fix(S.mu, recip_near(S.mu)), S.h, 0.5 * S.h, A.rcen, S.nb};
        const double* in = A.xin + p;
        Particle P;
        P.x = make_double3(in[0], in[S2], in[2 * S2]);
        P.v = make_double3(in[3 * S2], in[4 * S2], in[5 * S2]);
        P.acc = make_double3(in[6 * S2], in[7 * S2], in[8 * S2]);
        const double pad = A.rce[p] * 1.2;
        cols.at(Cols::PAD) = pad;
        P.padded = pad != 0.0;
        auto none = [](int) -> double { return 0.0; };
        if (A.reset && ok)
            P.acc = small_body_force<false, false>(P.x, P.v, none, tab, S.nb, nullptr, S.mu, A.status);
        P.derive();
#pragma unroll 1
        for (int s = 0; s < A.nsteps; ++s) {
            const double* T = tab + (size_t)(s + 1) * stride;
            particle_step<false, false, CENTRAL, TAB_BODY>(
                P, ok, cols, T, T, E, nullptr, A.status, 0.0,
                [&](bool cand, int b, double3 x0, double3 v0) {
                    const int slot = claim_slot(cand, A.cand_cap, A.status, &A.status->cands, 2);
                    if (slot >= 0)
                        candidate_record(A.cands + slot, make_int4(t.sys, b, A.step0 + s, S.nbig + A.local[p] + 1),
                                         A.rce[p], A.rphys[p], x0, v0, P.x, P.v);
                },
                [&](bool hit, double temp) {
                    const int slot = claim_slot(hit, A.event_cap, A.status, &A.status->events, 1);
                    if (slot >= 0) {
                        central_record(A.events + slot, S.nbig + A.local[p] + 1, A.rcen, temp);
                        A.event_step[slot] = A.step0 + s;
                        A.event_sys[slot] = t.sys;
                    }
                });
        }
        if (ok) {
            double* out = A.xout + p;
            out[0] = P.x.x;
            out[S2] = P.x.y;
            out[2 * S2] = P.x.z;
            out[3 * S2] = P.v.x;
            out[4 * S2] = P.v.y;
            out[5 * S2] = P.v.z;
            out[6 * S2] = P.acc.x;
            out[7 * S2] = P.acc.y;
            out[8 * S2] = P.acc.z;
        }
    }
}

// mce_stat's test for the candidates of the last batched launch.
__global__ void __launch_bounds__(256) classify_batch_kernel(BatchParticleArgs A) {
    const int count = min(A.status->cands, A.cand_cap);
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) {
        const EncounterCandidate& c = A.cands[k];
        const BatchSys S = A.sys[c.slot];
        const double* d = A.detail + S.det_off + ((size_t)(c.step - A.step0) * S.nb + c.body) * TAB_DETAIL;
        const PairEnds I{make_double3(d[0], d[1], d[2]), make_double3(d[3], d[4], d[5]),
                         make_double3(d[6], d[7], d[8]), make_double3(d[9], d[10], d[11])};
        const PairEnds J{make_double3(c.x0[0], c.x0[1], c.x0[2]), make_double3(c.v0[0], c.v0[1], c.v0[2]),
                         make_double3(c.x1[0], c.x1[1], c.x1[2]), make_double3(c.v1[0], c.v1[1], c.v1[2])};
        PairClass pc;
        if (!pair_classify(I, J, d[12], c.rce, d[13], c.rphys, S.h, pc)) continue;
        const int slot = atomicAdd(&A.status->events, 1);
        if (slot < A.event_cap) {
            pair_record(A.events + slot, I, J, pc, 1.0 / S.h, c.body + 2, c.id, false);
            A.event_step[slot] = c.step;
            A.event_sys[slot] = c.slot;
        } else {
            atomicOr(&A.status->overflow, 1);
        }
    }
}

template <bool NGF, bool OBL, bool CENTRAL>
void launch_variant(const MvsParticleArgs& a, cudaStream_t s, int threads) {
    auto kern = mvs_particle_kernel<NGF, OBL, CENTRAL>;
    const size_t smem = mvs_particle_smem(a.nb, a.nsteps, a.reset, threads, NGF);
    if (smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int tiles = (a.np + threads - 1) / threads;
    // the device's room for this launch shape, asked for when it changes (a
    // per-step host launches the same shape every time)
    static thread_local struct {
        int dev = -1, threads = 0, slots = 1;
        size_t smem = 0;
    } room;
    int dev = 0;
    cudaGetDevice(&dev);
    if (room.dev != dev || room.threads != threads || room.smem != smem) {
        int sms = 148, per_sm = 1;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
        room.dev = dev;
        room.threads = threads;
        room.smem = smem;
        room.slots = sms * (per_sm < 1 ? 1 : per_sm);
    }
    // All of them: the Big-body CTA of the next launch (another stream) needs
    // 38,912 registers, so it starts as these drain, and leaving one slot free
    // for it changes nothing (1M particles, 160 steps: 8.78 ms with, 8.79 without).
    const int grid = tiles < room.slots ? tiles : room.slots;
    if (grid > 0) kern<<<grid, threads, smem, s>>>(a);
}

}  // namespace

size_t mvs_particle_smem(int nb, int nsteps, int reset, int threads, bool ngf) {
    return sizeof(double) * ((size_t)srow_stride(nb) * (size_t)(nsteps + (reset ? 1 : 0)) +
                             (size_t)Cols::STRIDE * Cols::count(ngf));
}

namespace {
// Rows of 18 KB less the one for a fresh start's force, 1 to 64.
int steps_of_rows(int row_doubles) {
    const int k = (int)(18 * 1024 / (sizeof(double) * (size_t)row_doubles)) - 1;
    return k < 1 ? 1 : k > 64 ? 64 : k;
}
}  // namespace

// The most steps a launch takes: as many as there are rows {head, 8 doubles a
// body} in 18 KB, whatever else a table row holds: 31 steps of eight planets, 56
// of four (a CTA stages 14 KB of them).
int mvs_max_steps_per_launch(int nb) { return steps_of_rows(TAB_HEAD + TAB_BODY * nb); }

// The steps of a launch where the caller leaves it open: 18 KB of whole table
// rows, 25 steps of eight planets, 47 of four. Fewer launches re-order the slots
// and wait for their slowest tile less often, more sort particles that change
// path sooner. 457 steps of 1M particles take 30.0 ms with 16 steps a launch,
// 28.7 with 24 to 31, 29.0 with 40; a whole pass of 46 steps of 10,000 takes
// 0.81 ms with 25 (launches of 5, 25 and 16) and 0.84 with 31 (7, 31 and 8).
int mvs_usual_steps_per_launch(int nb) { return steps_of_rows(tab_stride(nb)); }

void launch_mvs_corrector(const MvsBigArgs& big, const CorrectorArgs& a, cudaStream_t s) {
    const int N = big.nmass > big.nbig ? big.nmass : big.nbig;
    const size_t smem = sizeof(double) * big_smem_doubles(N);
    if (smem > 48 * 1024)
        cudaFuncSetAttribute(mvs_corrector_big_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    mvs_corrector_big_kernel<<<1, BIG_THREADS, smem, s>>>(big, a);
    if (a.np <= 0) return;
    const int grid = (a.np + 127) / 128;
    if (a.ngf_on) {
        if (a.obl) mvs_corrector_particle_kernel<true, true><<<grid, 128, 0, s>>>(a);
        else mvs_corrector_particle_kernel<true, false><<<grid, 128, 0, s>>>(a);
    } else {
        if (a.obl) mvs_corrector_particle_kernel<false, true><<<grid, 128, 0, s>>>(a);
        else mvs_corrector_particle_kernel<false, false><<<grid, 128, 0, s>>>(a);
    }
}

void launch_mvs_big_batch(const BatchBigArgs& a, int nsys, int max_nbig, cudaStream_t s) {
    const size_t smem = sizeof(double) * big_smem_doubles_up_to(max_nbig);
    if (smem > 48 * 1024)
        cudaFuncSetAttribute(mvs_big_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (nsys > 0) mvs_big_batch_kernel<<<nsys, 32, smem, s>>>(a);
}

void launch_mvs_particles_batch(const BatchParticleArgs& a, cudaStream_t s, int threads) {
    if (a.ntiles <= 0) return;
    using Kernel = void (*)(BatchParticleArgs);
    const Kernel kern = threads <= 64    ? (a.central ? mvs_particle_batch_kernel<true, 64> : mvs_particle_batch_kernel<false, 64>)
                        : threads <= 128 ? (a.central ? mvs_particle_batch_kernel<true, 128> : mvs_particle_batch_kernel<false, 128>)
                                         : (a.central ? mvs_particle_batch_kernel<true, 256> : mvs_particle_batch_kernel<false, 256>);
    int dev = 0, sms = 148, per_sm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, 0);
    if (per_sm < 1) per_sm = 1;
    const int warps = threads / 32;
    const int want = (a.ntiles + warps - 1) / warps;
    const int slots = sms * per_sm;
    const int grid = want < slots ? want : slots;
    kern<<<grid, threads, 0, s>>>(a);
}

void launch_classify_batch(const BatchParticleArgs& a, cudaStream_t s) {
    classify_batch_kernel<<<296, 256, 0, s>>>(a);
}

void launch_classify(const ClassifyArgs& a, cudaStream_t s) {
    classify_kernel<<<296, 256, 0, s>>>(a);
}

void launch_mvs_big(const MvsBigArgs& a, cudaStream_t s) {
    const int N = a.nmass > a.nbig ? a.nmass : a.nbig;
    const size_t smem = sizeof(double) * big_smem_doubles(N);
    if (smem > 48 * 1024)
        cudaFuncSetAttribute(mvs_big_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    mvs_big_kernel<<<1, BIG_THREADS, smem, s>>>(a);
}

void launch_mvs_particles(const MvsParticleArgs& args, cudaStream_t s, int threads) {
    MvsParticleArgs a = args;
    a.rmu = 1.0 / a.mu;
    const bool ngf = a.ngf_on != 0;
    const bool obl = a.jcen[0] != 0.0 || a.jcen[1] != 0.0 || a.jcen[2] != 0.0;
    const bool cen = a.central != 0;
    if (ngf) {
        if (obl) cen ? launch_variant<true, true, true>(a, s, threads) : launch_variant<true, true, false>(a, s, threads);
        else cen ? launch_variant<true, false, true>(a, s, threads) : launch_variant<true, false, false>(a, s, threads);
    } else {
        if (obl) cen ? launch_variant<false, true, true>(a, s, threads) : launch_variant<false, true, false>(a, s, threads);
        else cen ? launch_variant<false, false, true>(a, s, threads) : launch_variant<false, false, false>(a, s, threads);
    }
}

}  // namespace mb200
