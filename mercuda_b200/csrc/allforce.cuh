// mfo_all (mercury6_2.for:4506-4571) on the device for the adaptive
// integrators, split as they use it: the massive set (Big bodies and massive
// Small bodies, [3][nsplit] arrays) by one CTA that also writes a table row
// of what every massless particle needs (the indirect sum sx, the oblateness
// reaction acen, the Big bodies' positions and masses), and the massless
// particles from that row. Every sum keeps mfo_grav's order: the indirect sum
// over all bodies by index (massless ones add exactly zero), direct terms with
// Big i outer and j > i inner.
#pragma once
#include "common.cuh"
#include "mvs_device.cuh"

namespace mb200 {

// Force configuration shared by every kernel that evaluates mfo_all.
struct ForceCfg {
    int nbig;      // Big bodies incl. the central body
    int nsplit;    // bodies [0, nsplit) are in the "big" arrays (Big + massive Small)
    int ngflag;
    int pn;
    int obl;
    double jcen[3];
    double m0;
};

// Table row for the particle kernels, in doubles:
// {sx, sy, sz, acen_x, acen_y, acen_z, pad, pad, [x, y, z, m] per Big body}.
constexpr int FT_HEAD = 8;
__host__ __device__ constexpr int force_row(int nb) { return FT_HEAD + 4 * nb; }

// c = 299792458*86400/(AU*0.01) AU/day as mfo_grav/mfo_pr compute it.
__device__ __forceinline__ double light_c() { return 299792458.0 * 86400.0 / (1.495978707e13 * 0.01); }

// mfo_pr's drag for one body (mercury6_2.for:5300-5343), given r = |x|.
static __device__ __noinline__ double3 pr_plain(double3 x, double3 v, double beta) {
    const double c = light_c(), sw = 0.3;
    const double r = sqrt(x.x * x.x + x.y * x.y + x.z * x.z);
    const double vr = (x.x * v.x + x.y * v.y + x.z * v.z) / r;
    const double ff = K2 * beta / (r * r);
    return make_double3(ff * ((1.0 - (1.0 + sw) * vr / c) * x.x / r - (1.0 + sw) * v.x / c),
                        ff * ((1.0 - (1.0 + sw) * vr / c) * x.y / r - (1.0 + sw) * v.y / c),
                        ff * ((1.0 - (1.0 + sw) * vr / c) * x.z / r - (1.0 + sw) * v.z / c));
}

// |x|, its square and reciprocal for the central terms, rounded as sqrt and
// 1/sqrt round them; mid: within fp64.cuh's range (else they were made by the
// plain statements).
struct Radius {
    double r2, r, ri;
    bool mid;
};
static __device__ __noinline__ Radius radius_plain(double r2) {
    const double r = sqrt(r2);
    return Radius{r2, r, 1.0 / r, false};
}
__device__ __forceinline__ Radius radius_of(const double3 x) {
    Radius R;
    R.r2 = x.x * x.x + x.y * x.y + x.z * x.z;
    sqrt_recip(R.r2, R.r, R.ri);
    R.mid = root_range(R.r2);
    return R.mid ? R : radius_plain(R.r2);
}

// The terms of mfo_all after the direct sums: indirect and central terms of
// mfo_grav (with the fused 1PN), then mfo_obl, mfo_ngf, mfo_pr.
// a holds the direct sum. The drag's eight divisions and the others are made
// by fp64.cuh's quotients from 1/r and the reciprocals of constants.
__device__ __forceinline__ double3 finish_force(double3 a, const double3 x, const double3 v, const Radius R,
                                               const double* T, const ForceCfg& f, double mj, const double* g,
                                               DeviceStatus* st) {
    const double ri = R.ri;
    const double r3 = ri * ri * ri;
    const double tmp1 = f.m0 * r3;
    const double c = light_c();
    if (f.pn == 0) {
        a.x = a.x + T[0] - tmp1 * x.x;
        a.y = a.y + T[1] - tmp1 * x.y;
        a.z = a.z + T[2] - tmp1 * x.z;
    } else {
        const double light2 = c * c;
        const double rv = 0.0 + x.x * v.x + x.y * v.y + x.z * v.z;
        const double v2 = 0.0 + v.x * v.x + v.y * v.y + v.z * v.z;
        const double ff = quotient(tmp1, light2, 1.0 / light2);
        const double radial = 4.0 * f.m0 * ri - v2;
        a.x = a.x + T[0] - tmp1 * x.x + ff * (radial * x.x + 4.0 * rv * v.x);
        a.y = a.y + T[1] - tmp1 * x.y + ff * (radial * x.y + 4.0 * rv * v.y);
        a.z = a.z + T[2] - tmp1 * x.z + ff * (radial * x.z + 4.0 * rv * v.z);
    }
    if (f.obl) {
        const double3 ao = oblate_accel(x, f.jcen, f.m0);
        a.x = a.x + (ao.x - T[3]);
        a.y = a.y + (ao.y - T[4]);
        a.z = a.z + (ao.z - T[5]);
    }
    if (f.ngflag == 1 || f.ngflag == 3) {
        double3 ng;
        if (!nongrav_near(x, v, R.r2, g, ng)) raise_fault(st, FAULT_NGF);
        a.x = a.x + ng.x;
        a.y = a.y + ng.y;
        a.z = a.z + ng.z;
    }
    if (f.ngflag == 2 || f.ngflag == 3) {
        double3 pr = make_double3(0.0, 0.0, 0.0);
        if (!(mj != 0.0 || g[3] == 0.0)) {
            const double sw = 0.3, yc = 1.0 / c;
            const double vr = quotient(x.x * v.x + x.y * v.y + x.z * v.z, R.r, ri);
            const double ff = quotient_of(K2 * g[3], R.r * R.r, ri * ri);
            const double rad = 1.0 - quotient((1.0 + sw) * vr, c, yc);
            pr.x = ff * (quotient(rad * x.x, R.r, ri) - quotient((1.0 + sw) * v.x, c, yc));
            pr.y = ff * (quotient(rad * x.y, R.r, ri) - quotient((1.0 + sw) * v.y, c, yc));
            pr.z = ff * (quotient(rad * x.z, R.r, ri) - quotient((1.0 + sw) * v.z, c, yc));
            if (!R.mid) pr = pr_plain(x, v, g[3]);
        }
        a.x = a.x + pr.x;
        a.y = a.y + pr.y;
        a.z = a.z + pr.z;
    }
    if (!isfinite(a.x) || !isfinite(a.y) || !isfinite(a.z)) raise_fault(st, FAULT_NONFINITE);
    return a;
}

// mfo_all for a massless Small body from a table row T (mfo_grav's direct sum
// over the Big bodies in index order, then finish_force).
template <int UNROLL = 4>
__device__ __forceinline__ double3 particle_allforce(const double3 x, const double3 v, const double* T, int nb,
                                                     const ForceCfg& f, double mj, const double* g,
                                                     DeviceStatus* st) {
    const Radius R = radius_of(x);
    if (R.r2 <= 0.0) raise_fault(st, FAULT_COINCIDENT);
    bool coincident = false;
    const double3 a = direct_terms<4, UNROLL>(x, T + FT_HEAD, nb, &coincident);
    if (coincident) raise_fault(st, FAULT_COINCIDENT);
    return finish_force(a, x, v, R, T, f, mj, g, st);
}

// mfo_all for body k of the massive set, positions X/V [3][ns] in memory,
// T the row being built (sx, acen already in it).
__device__ __forceinline__ double3 massive_allforce(int k, const double* X, const double* V, const double* m,
                                                    const double* ngfbig, const double* T, const ForceCfg& f,
                                                    DeviceStatus* st) {
    const int N = f.nsplit;
    const double3 x = make_double3(X[k], X[N + k], X[2 * N + k]);
    const double3 v = make_double3(V[k], V[N + k], V[2 * N + k]);
    const Radius R = radius_of(x);
    if (R.r2 <= 0.0) raise_fault(st, FAULT_COINCIDENT);
    double3 a = make_double3(0.0, 0.0, 0.0);
    const int last_i = k < f.nbig ? k : f.nbig;
    for (int i = 1; i < last_i; ++i) {  // earlier Big bodies: k is their "j"
        const double dx = x.x - X[i], dy = x.y - X[N + i], dz = x.z - X[2 * N + i];
        const double s2 = dx * dx + dy * dy + dz * dz;
        if (s2 <= 0.0) raise_fault(st, FAULT_COINCIDENT);
        const double s_1 = 1.0 / sqrt(s2);
        const double s_3 = s_1 * s_1 * s_1;
        const double tmp1 = s_3 * m[i];
        a.x = a.x - tmp1 * dx;
        a.y = a.y - tmp1 * dy;
        a.z = a.z - tmp1 * dz;
    }
    if (k < f.nbig)
        for (int j = k + 1; j < N; ++j) {  // later bodies: k is their Big "i"
            const double dx = X[j] - x.x, dy = X[N + j] - x.y, dz = X[2 * N + j] - x.z;
            const double s2 = dx * dx + dy * dy + dz * dz;
            if (s2 <= 0.0) raise_fault(st, FAULT_COINCIDENT);
            const double s_1 = 1.0 / sqrt(s2);
            const double s_3 = s_1 * s_1 * s_1;
            const double tmp2 = s_3 * m[j];
            a.x = a.x + tmp2 * dx;
            a.y = a.y + tmp2 * dy;
            a.z = a.z + tmp2 * dz;
        }
    return finish_force(a, x, v, R, T, f, m[k], ngfbig + 5 * k, st);
}

// Row head: sx (mfo_grav's indirect sum over every body, in index order; the
// massless particles add exactly zero) and acen (mfo_obl's reaction), from the
// massive set's positions. One thread.
static __device__ void row_head(const double* X, const double* m, const ForceCfg& f, double* T) {
    const int N = f.nsplit;
    double sx = 0.0, sy = 0.0, sz = 0.0, ax = 0.0, ay = 0.0, az = 0.0;
    for (int i = 1; i < N; ++i) {
        const double3 p = make_double3(X[i], X[N + i], X[2 * N + i]);
        const double s2 = p.x * p.x + p.y * p.y + p.z * p.z;
        const double s_1 = 1.0 / sqrt(s2);
        const double r3 = s_1 * s_1 * s_1;
        const double tmp1 = m[i] * r3;
        sx = sx - tmp1 * p.x;
        sy = sy - tmp1 * p.y;
        sz = sz - tmp1 * p.z;
        if (f.obl) {
            const double3 ao = oblate_accel(p, f.jcen, f.m0);
            const double tmp4 = m[i] / f.m0;
            ax = ax - tmp4 * ao.x;
            ay = ay - tmp4 * ao.y;
            az = az - tmp4 * ao.z;
        }
    }
    T[0] = sx; T[1] = sy; T[2] = sz;
    T[3] = ax; T[4] = ay; T[5] = az;
    T[6] = 0.0; T[7] = 0.0;
}

// ---- The massive set's mfo_all by a whole CTA, for sets of up to
// MASSIVE_PAR_MAX bodies. A force call is a link of the integrator's serial
// chain, so its latency counts: every pair's and body's terms are computed one
// per thread, signed, into rows of shared memory padded with zeros; one thread
// per body and coordinate adds a row up in mfo_grav's order (x + 0 is x, so
// nothing depends on which bodies act on which); one thread per body finishes
// with the central terms. The same roundings in the same order as the loops
// above. Eight planets, a call of RADAU: 4.6 us with sums in one thread and
// division calls, 1.9 us so.
constexpr int MASSIVE_PAR_MAX = 32;
__host__ __device__ constexpr int massive_rows_doubles(int N) {
    return N <= MASSIVE_PAR_MAX ? (3 * N + 6) * term_row(N) + 5 * N + 1 : 0;
}
struct MassiveRows {
    double* base;   // massive_rows_doubles(N) doubles, 16-byte aligned
    int N;
    __device__ double* pair(int c, int k) const { return base + (c * N + k) * term_row(N); }
    __device__ double* head(int c) const { return base + (3 * N + c) * term_row(N); }   // sx terms, then acen's
    __device__ double* sum() const { return base + (3 * N + 6) * term_row(N); }         // [3][N] direct sums
    __device__ double* rad() const { return sum() + 3 * N; }                            // [N] |x|, then 1/|x|
    __device__ void clear() const {
        for (int q = threadIdx.x; q < (3 * N + 6) * term_row(N); q += blockDim.x) base[q] = 0.0;
    }
};
__device__ __forceinline__ double row_sum(const double* row, int n) {
    const double2* p = reinterpret_cast<const double2*>(row);
    double a = 0.0;
    for (int i0 = 0; i0 < n; i0 += 8, p += 4) {
        const double2 t0 = p[0], t1 = p[1], t2 = p[2], t3 = p[3];
        a = a + t0.x; a = a + t0.y;
        a = a + t1.x; a = a + t1.y;
        a = a + t2.x; a = a + t2.y;
        a = a + t3.x; a = a + t3.y;
    }
    return a;
}
// One force call at X, V (shared, [3][N]; synchronized inside) into out
// [3][N] and table row T. Rows cleared once before the first call.
static __device__ __forceinline__ void massive_rows_call(const double* X, const double* V, double* out, double* T,
                                                         const double* mb, const double* ngf, const ForceCfg& f,
                                                         const MassiveRows M, double* head, DeviceStatus* st) {
    const int N = f.nsplit, tid = threadIdx.x, nt = blockDim.x, nw = nt >> 5;
    __syncthreads();
    // pairs (i < k, i Big) from the first thread on, bodies from the last warp
    const int npair = (N - 1) * (N - 2) / 2;
    for (int q = tid; q < npair; q += nt) {
        int i = 1, rem = q;
        while (rem >= N - 1 - i) { rem -= N - 1 - i; ++i; }
        const int k = i + 1 + rem;
        if (i >= f.nbig) continue;
        const double dx = X[k] - X[i], dy = X[N + k] - X[N + i], dz = X[2 * N + k] - X[2 * N + i];
        const Radius R = radius_of(make_double3(dx, dy, dz));
        if (R.r2 <= 0.0) raise_fault(st, FAULT_COINCIDENT);
        const double s_3 = R.ri * R.ri * R.ri;
        const double tk = s_3 * mb[i], ti = s_3 * mb[k];
        M.pair(0, k)[i - 1] = -(tk * dx);
        M.pair(1, k)[i - 1] = -(tk * dy);
        M.pair(2, k)[i - 1] = -(tk * dz);
        M.pair(0, i)[k - 1] = ti * dx;
        M.pair(1, i)[k - 1] = ti * dy;
        M.pair(2, i)[k - 1] = ti * dz;
    }
    for (int k = 1 + (nt - 1 - tid); k < N; k += nt) {
        const double3 p = make_double3(X[k], X[N + k], X[2 * N + k]);
        const Radius R = radius_of(p);
        if (R.r2 <= 0.0) raise_fault(st, FAULT_COINCIDENT);
        M.rad()[k] = R.r;
        M.rad()[N + k] = R.ri;
        const double r3 = R.ri * R.ri * R.ri;
        const double tmp1 = mb[k] * r3;
        M.head(0)[k - 1] = -(tmp1 * p.x);
        M.head(1)[k - 1] = -(tmp1 * p.y);
        M.head(2)[k - 1] = -(tmp1 * p.z);
        if (f.obl) {
            const double3 ao = oblate_accel(p, f.jcen, f.m0);
            const double tmp4 = mb[k] / f.m0;
            M.head(3)[k - 1] = -(tmp4 * ao.x);
            M.head(4)[k - 1] = -(tmp4 * ao.y);
            M.head(5)[k - 1] = -(tmp4 * ao.z);
        }
        if (k < f.nbig) {
            double* row = T + FT_HEAD + 4 * (k - 1);
            row[0] = p.x; row[1] = p.y; row[2] = p.z; row[3] = mb[k];
        }
    }
    __syncthreads();
    for (int q = tid; q < 3 * (N - 1); q += nt) {
        const int k = 1 + q / 3, c = q - 3 * (k - 1);
        M.sum()[c * N + k] = row_sum(M.pair(c, k), N - 1);
    }
    if (tid >= 32 * (nw - 1) && (tid & 31) < FT_HEAD) {
        const int c = tid & 31;
        const double h = c < 6 ? row_sum(M.head(c), N - 1) : 0.0;
        head[c] = h;
        T[c] = h;
    }
    __syncthreads();
    for (int k = 1 + tid; k < N; k += nt) {
        const double3 x = make_double3(X[k], X[N + k], X[2 * N + k]);
        const double3 v = make_double3(V[k], V[N + k], V[2 * N + k]);
        const double* s = M.sum();
        const double r2 = x.x * x.x + x.y * x.y + x.z * x.z;
        const Radius R{r2, M.rad()[k], M.rad()[N + k], mid_range(r2)};
        const double3 a = finish_force(make_double3(s[k], s[N + k], s[2 * N + k]), x, v, R, head, f, mb[k],
                                       ngf + 5 * k, st);
        out[k] = a.x; out[N + k] = a.y; out[2 * N + k] = a.z;
    }
    __syncthreads();
}

}  // namespace mb200
