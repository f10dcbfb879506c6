// Batched MVS systems: host orchestration of the extension entry points in
// include/mercury_b200.h (mercury_b200_batch_*). The reference integrates one
// system per process; these calls advance thousands of independent systems,
// each with its own Big bodies, particle count and step, in one pipelined run:
//
//   stream_big: Big-body CTAs of chunk c (every system) -> tables set c % 2
//   stream:     particles of chunk c (one launch over every system's tiles),
//               classification of its encounter candidates
//
// The chunk loop of a run is captured once into a CUDA graph and replayed for
// later runs of the same shape. The launch shape (steps per launch and the
// particle kernel's CTA size) is chosen by timing short trial runs before the
// first run (tune).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <tuple>
#include <vector>

#include "../../include/mercury_b200.h"
#include "context.cuh"
#include "mvs.cuh"

namespace mb200 {
namespace {

constexpr int BATCH_MAX_NBIG = 32;

struct Batch {
    int nsys = 0, nbody = 0, npcap = 0, ntiles = 0, nbigs = 0, max_nbig = 1, max_body = 1, K = 31;
    std::vector<int> body_off, nbig, np, first_slot, big_off;
    std::vector<double> h, mu;
    std::vector<BatchSys> sys;
    DBuf<BatchSys> d_sys;
    DBuf<int> d_body_end;
    DBuf<BatchTile> d_tiles;
    DBuf<MvsBigArgs> d_proto;
    DBuf<double> bigbuf[2];          // per system [9][nbig] at 9 * big_off
    DBuf<double> bm, brce, brphys;   // per system [nbig] at big_off
    DBuf<double> pstate[2];          // [9][npcap]
    DBuf<double> prce, prphys;
    DBuf<int> plocal;
    DBuf<double> tab[2], det[2];
    size_t tab_size = 0, det_size = 0;
    DBuf<MercuryEvent> events;
    DBuf<int> event_step, event_sys;
    DBuf<EncounterCandidate> cands;
    DBuf<DeviceStatus> status;
    DeviceStatus* status_host = nullptr;
    // the run's starting state; between runs the host arrays' rows as they are
    // (x, v, 3 a body, m, rce, rphys: the same size)
    DBuf<double> snap;
    int cur = 0;
    bool reset = true;
    int threads = 0;                 // 0: tune on the first run
    int tuned_K = 31, tuned_threads = 128;
    int forced_threads = 0, forced_K = 0, use_graph = 1;
    cudaStream_t stream = nullptr, stream_big = nullptr;
    cudaEvent_t t0 = nullptr, t1 = nullptr;
    std::vector<cudaEvent_t> big_done, part_done;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    std::tuple<int, int, int, int, int, double, long> graph_key{};
    long epoch = 0;                  // bumped whenever a buffer is reallocated
    float last_ms = 0.0f;
    int last_launches = 0;
    std::vector<MercuryEvent> host_events;
    std::vector<int> host_sys, host_step;

    void release() {
        release_buffers();
        nsys = nbody = npcap = ntiles = 0;
        host_events.clear();
        host_sys.clear();
        host_step.clear();
    }
    void release_buffers() {
        DBuf<double>* d[] = {&bigbuf[0], &bigbuf[1], &bm, &brce, &brphys, &pstate[0], &pstate[1],
                             &prce, &prphys, &tab[0], &tab[1], &det[0], &det[1], &snap};
        for (auto* b : d) b->release();
        d_sys.release();
        d_body_end.release();
        d_tiles.release();
        d_proto.release();
        plocal.release();
        events.release();
        event_step.release();
        event_sys.release();
        cands.release();
        status.release();
        drop_graph();
        ++epoch;
    }
    int record_cap() const { return (int)std::min({events.n, event_step.n, event_sys.n}); }
    // Room for that many records and candidates; what there was where it
    // cannot be had (the records' three arrays are always of one size).
    void room_for(size_t records, size_t candidates) {
        const size_t r0 = events.n, c0 = cands.n;
        auto reserve = [&](size_t r, size_t c) {
            events.reserve(r);
            event_step.reserve(r);
            event_sys.reserve(r);
            cands.reserve(c);
        };
        ++epoch;
        try {
            reserve(std::max(records, r0), candidates);
        } catch (const CudaError&) {
            cudaGetLastError();
            events.release();
            event_step.release();
            event_sys.release();
            cands.release();
            reserve(r0, c0);
            throw;
        }
    }
    void drop_graph() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        exec = nullptr;
        graph = nullptr;
    }
    void ensure_streams() {
        if (stream) return;
        check(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking), "stream");
        check(cudaStreamCreateWithFlags(&stream_big, cudaStreamNonBlocking), "stream");
        check(cudaEventCreate(&t0), "event");
        check(cudaEventCreate(&t1), "event");
        check(cudaMallocHost(reinterpret_cast<void**>(&status_host), sizeof(DeviceStatus)), "pinned");
    }
    void ensure_chunk_events(int n) {
        while ((int)big_done.size() < n) {
            cudaEvent_t a, b;
            check(cudaEventCreateWithFlags(&a, cudaEventDisableTiming), "event");
            check(cudaEventCreateWithFlags(&b, cudaEventDisableTiming), "event");
            big_done.push_back(a);
            part_done.push_back(b);
        }
    }
};

Batch& batch() {
    static Batch b;
    return b;
}

// Between the host arrays' rows (staged on the device) and the batch's
// layout, one block per system and BATCH_CHUNK bodies of it (systems of more
// than a million bodies: several chunks a block): Big bodies to
// [9][nbig] at 9 big_off, particles to their slots. GATHER takes positions and
// velocities back to rows.
constexpr int BATCH_CHUNK = 1024, BATCH_CHUNK_BLOCKS = 1024;
struct BatchRows {
    const BatchSys* sys;
    const int* body_end;      // first row past each system
    int row0, nchunks;        // the first system's first row; BATCH_CHUNKs of the largest system
    double *x, *v;            // rows, 3 a body
    const double *m, *rce, *rphys;
    double* big;
    double* part;
    size_t npcap;
    double *bm, *brce, *brphys, *prce, *prphys;
    int* local;
};
template <bool GATHER> __global__ void __launch_bounds__(128) batch_rows_kernel(BatchRows A) {
    const BatchSys S = A.sys[blockIdx.x];
    const int n = A.body_end[blockIdx.x] - S.body;
    auto move = [&](int j) {
        const size_t row = (size_t)(S.body - A.row0) + j;
        double* x = A.x + 3 * row;
        double* v = A.v + 3 * row;
        const bool is_big = j < S.nbig;
        const int q = j - S.nbig;
        const size_t slot = S.first_slot + q, st = is_big ? S.nbig : A.npcap;
        double* d = is_big ? A.big + 9 * (size_t)S.big_off + j : A.part + slot;
        for (int c = 0; c < 3; ++c) {
            if (GATHER) {
                x[c] = d[c * st];
                v[c] = d[(3 + c) * st];
            } else {
                d[c * st] = x[c];
                d[(3 + c) * st] = v[c];
                d[(6 + c) * st] = 0.0;
            }
        }
        if (GATHER) return;
        if (is_big) {
            A.bm[S.big_off + j] = A.m[row];
            A.brce[S.big_off + j] = A.rce[row];
            A.brphys[S.big_off + j] = A.rphys[row];
        } else {
            A.prce[slot] = A.rce[row];
            A.prphys[slot] = A.rphys[row];
            A.local[slot] = q;
        }
    };
    for (int c = blockIdx.y; c < A.nchunks; c += gridDim.y) {
        const int j0 = c * BATCH_CHUNK;
        if (j0 >= n) break;
        const int count = min(n - j0, BATCH_CHUNK);
        for (int j = threadIdx.x; j < count; j += blockDim.x) move(j0 + j);
    }
}
template <bool GATHER> void launch_batch_rows(Batch& B) {
    const size_t n = B.nbody - B.body_off[0];
    BatchRows a{};
    a.sys = B.d_sys.p;
    a.body_end = B.d_body_end.p;
    a.row0 = B.body_off[0];
    a.nchunks = (int)(((long long)B.max_body + BATCH_CHUNK - 1) / BATCH_CHUNK);
    a.x = B.snap.p;
    a.v = a.x + 3 * n;
    a.m = a.v + 3 * n;
    a.rce = a.m + n;
    a.rphys = a.rce + n;
    a.big = B.bigbuf[B.cur].p;
    a.part = B.pstate[B.cur].p;
    a.npcap = B.npcap;
    a.bm = B.bm.p;
    a.brce = B.brce.p;
    a.brphys = B.brphys.p;
    a.prce = B.prce.p;
    a.prphys = B.prphys.p;
    a.local = B.plocal.p;
    const dim3 grid(B.nsys, std::min(a.nchunks, BATCH_CHUNK_BLOCKS));
    batch_rows_kernel<GATHER><<<grid, 128, 0, B.stream>>>(a);
    check(cudaGetLastError(), "batch rows");
}

// Table and detail offsets of every system for K steps per chunk, and the
// sizes of one set.
void layout_tables(Batch& B, int K) {
    size_t t = 0, d = 0;
    for (int s = 0; s < B.nsys; ++s) {
        const int nb = B.nbig[s] - 1;
        B.sys[s].tab_off = t;
        B.sys[s].det_off = d;
        t += (size_t)(K + 1) * tab_stride(nb);
        d += (size_t)K * std::max(1, nb) * TAB_DETAIL;
    }
    B.tab_size = t;
    B.det_size = d;
    auto reserve = [&] {
        for (int k = 0; k < 2; ++k) {
            if (t > B.tab[k].n || d > B.det[k].n) ++B.epoch;
            B.tab[k].reserve(t);
            B.det[k].reserve(d);
        }
    };
    try {
        reserve();
    } catch (const CudaError&) {
        // the room for candidates may be an earlier run's guess
        cudaGetLastError();
        const size_t least = std::max(16384, B.npcap / 2);
        if (B.cands.n <= least) throw;
        B.cands.release();
        ++B.epoch;
        B.cands.reserve(least);
        reserve();
    }
    B.K = K;
    h2d(B.d_sys.p, B.sys.data(), sizeof(BatchSys) * B.nsys, B.stream);
}

BatchBigArgs big_chunk(Batch& B, int ch, int ks, int reset, int central, int s0, double rcen) {
    BatchBigArgs a{};
    a.proto = B.d_proto.p;
    a.sys = B.d_sys.p;
    a.flip = ((B.cur + ch) & 1) ? 1 : 0;
    a.nsteps = ks;
    a.reset = reset;
    a.central = central;
    a.step0 = s0;
    a.rcen = rcen;
    a.tab = B.tab[ch & 1].p;
    a.detail = B.det[ch & 1].p;
    a.events = B.events.p;
    a.event_step = B.event_step.p;
    a.event_sys = B.event_sys.p;
    a.event_cap = B.record_cap();
    a.status = B.status.p;
    return a;
}

BatchParticleArgs particle_chunk(Batch& B, int ch, int ks, int reset, int central, int s0, double rcen) {
    BatchParticleArgs a{};
    a.ntiles = B.ntiles;
    a.npcap = B.npcap;
    a.nsteps = ks;
    a.reset = reset;
    a.central = central;
    a.step0 = s0;
    a.rcen = rcen;
    a.sys = B.d_sys.p;
    a.tiles = B.d_tiles.p;
    const int in = (B.cur + ch) & 1;
    a.xin = B.pstate[in].p;
    a.xout = B.pstate[1 - in].p;
    a.rce = B.prce.p;
    a.rphys = B.prphys.p;
    a.local = B.plocal.p;
    a.tab = B.tab[ch & 1].p;
    a.detail = B.det[ch & 1].p;
    a.events = B.events.p;
    a.event_step = B.event_step.p;
    a.event_sys = B.event_sys.p;
    a.event_cap = B.record_cap();
    a.cands = B.cands.p;
    a.cand_cap = (int)B.cands.n;
    a.status = B.status.p;
    return a;
}

// The chunk loop of one run, enqueued on the two streams (also what a graph
// captures). Returns the number of kernels launched.
int enqueue_run(Batch& B, int nsteps, double rcen, int reset0, int central) {
    const int K = B.K, nchunks = (nsteps + K - 1) / K;
    int launches = 0;
    check(cudaMemsetAsync(B.status.p, 0, sizeof(DeviceStatus), B.stream), "memset");
    check(cudaEventRecord(B.big_done[0], B.stream), "event");  // fork point
    check(cudaStreamWaitEvent(B.stream_big, B.big_done[0], 0), "wait");
    for (int ch = 0; ch < nchunks; ++ch) {
        const int s0 = ch * K, ks = std::min(K, nsteps - s0);
        const int reset = (ch == 0 && reset0) ? 1 : 0;
        // the table set of this chunk is free once chunk ch - 2 was classified
        if (ch >= 2) check(cudaStreamWaitEvent(B.stream_big, B.part_done[ch - 2], 0), "wait");
        launch_mvs_big_batch(big_chunk(B, ch, ks, reset, central, s0, rcen), B.nsys, B.max_nbig, B.stream_big);
        ++launches;
        check(cudaEventRecord(B.big_done[ch], B.stream_big), "event");
        check(cudaStreamWaitEvent(B.stream, B.big_done[ch], 0), "wait");
        if (B.ntiles > 0) {
            check(cudaMemsetAsync(&B.status.p->next_tile, 0, sizeof(int), B.stream), "memset");
            const BatchParticleArgs pa = particle_chunk(B, ch, ks, reset, central, s0, rcen);
            launch_mvs_particles_batch(pa, B.stream, B.threads);
            launch_classify_batch(pa, B.stream);
            check(cudaMemsetAsync(&B.status.p->cands, 0, sizeof(int), B.stream), "memset");
            launches += 2;
        }
        check(cudaEventRecord(B.part_done[ch], B.stream), "event");
    }
    // join the Big-body stream
    check(cudaStreamWaitEvent(B.stream, B.big_done[nchunks - 1], 0), "wait");
    return launches;
}

// The launch shape of a batch: for every steps-per-launch K (8, 16, 31, 64)
// and particle CTA size (64, 128, 256) a short pipelined trial run of two
// chunks (Big-body CTAs on their stream ahead of the particle launches, as
// the real runs make them), timed with CUDA events; the fastest time per step
// wins. The trials start from the batch's state and it is restored after
// them (the snapshot), so tuning advances nothing. A forced CTA size or K
// (mercury_b200_batch_set) limits the search to it; the choice is kept and
// reported by mercury_b200_batch_timing.
void tune(Batch& B, double rcen, int nsteps) {
    std::vector<int> Ks = {8, 16, 31, 64};
    std::vector<int> Ts = {64, 128, 256};
    if (B.forced_K > 0) Ks = {B.forced_K};
    if (B.forced_threads > 0) Ts = {B.forced_threads};
    for (int& k : Ks) k = std::max(1, std::min(k, nsteps));
    std::sort(Ks.begin(), Ks.end());
    Ks.erase(std::unique(Ks.begin(), Ks.end()), Ks.end());
    B.threads = Ts[0];
    B.tuned_K = Ks[0];
    if (B.ntiles == 0 || (Ks.size() == 1 && Ts.size() == 1)) return;
    const size_t bigs = (size_t)B.nbigs;
    auto copy = [&](void* d, const void* src, size_t bytes) {
        check(cudaMemcpyAsync(d, src, bytes, cudaMemcpyDeviceToDevice, B.stream), "tune");
    };
    copy(B.snap.p, B.pstate[B.cur].p, sizeof(double) * 9 * B.npcap);
    copy(B.snap.p + 9 * (size_t)B.npcap, B.bigbuf[B.cur].p, sizeof(double) * 9 * bigs);
    B.ensure_chunk_events(2);
    double best = 1e300;
    for (int K : Ks) {
        layout_tables(B, K);
        const int steps = std::min(nsteps, 2 * K);
        for (int threads : Ts) {
            B.threads = threads;
            check(cudaEventRecord(B.t0, B.stream), "event");
            enqueue_run(B, steps, rcen, B.reset ? 1 : 0, 1);
            check(cudaEventRecord(B.t1, B.stream), "event");
            check(cudaEventSynchronize(B.t1), "tune");
            float ms = 0.0f;
            check(cudaEventElapsedTime(&ms, B.t0, B.t1), "tune");
            const double per_step = ms / steps;
            if (per_step < best) {
                best = per_step;
                B.tuned_K = K;
                B.tuned_threads = threads;
            }
            copy(B.pstate[B.cur].p, B.snap.p, sizeof(double) * 9 * B.npcap);
            copy(B.bigbuf[B.cur].p, B.snap.p + 9 * (size_t)B.npcap, sizeof(double) * 9 * bigs);
        }
    }
    B.threads = B.tuned_threads;
    check(cudaGetLastError(), "tune");
}

// The records in (system, step, min id, max id) order; equal keys keep the
// order in which they came.
void sort_batch_events(Batch& B) {
    struct Key {
        uint64_t where, pair;
        uint32_t at;
    };
    const size_t n = B.host_events.size();
    std::vector<Key> keys(n);
    for (size_t k = 0; k < n; ++k) {
        const MercuryEvent& e = B.host_events[k];
        keys[k] = Key{(uint64_t)(uint32_t)B.host_sys[k] << 32 | (uint32_t)B.host_step[k],
                      (uint64_t)(uint32_t)std::min(e.i, e.j) << 32 | (uint32_t)std::max(e.i, e.j), (uint32_t)k};
    }
    std::sort(keys.begin(), keys.end(), [](const Key& a, const Key& b) {
        return a.where != b.where ? a.where < b.where : a.pair != b.pair ? a.pair < b.pair : a.at < b.at;
    });
    std::vector<MercuryEvent> e(n);
    std::vector<int> sy(n), st(n);
    for (size_t k = 0; k < n; ++k) {
        e[k] = B.host_events[keys[k].at];
        sy[k] = B.host_sys[keys[k].at];
        st[k] = B.host_step[keys[k].at];
    }
    B.host_events.swap(e);
    B.host_sys.swap(sy);
    B.host_step.swap(st);
}

// Room for a run's records and one chunk's candidates, so that a run need not
// be made again: the package's workloads give up to 8 records and 400
// candidates per 10,000 particle-steps. Only a guess (the records are capped at
// 4M), so made out of a quarter of the free memory or not at all: an overflow
// still grows the buffers and redoes the run.
void size_records(Batch& B, int nsteps, int K) {
    const long long slots = B.npcap;
    const size_t records = (size_t)std::min<long long>(4 << 20, slots * nsteps / 1000);
    const size_t cands = (size_t)std::min<long long>(INT32_MAX / 2, slots * K / 25);
    if (records <= B.events.n && cands <= B.cands.n) return;
    size_t more = 0, free_b = 0, total_b = 0;
    if (records > B.events.n) more += records * (sizeof(MercuryEvent) + 2 * sizeof(int));
    if (cands > B.cands.n) more += cands * sizeof(EncounterCandidate);
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess || more > free_b / 4) return;
    try {
        B.room_for(records, cands);
    } catch (const CudaError&) {
        cudaGetLastError();
    }
}

}  // namespace
}  // namespace mb200

using namespace mb200;

extern "C" {

int mercury_b200_batch_upload(int nsys, const int* body_offset, const int* nbig, const double* h, const double* m,
                              const double* xx, const double* vv, const double* rce, const double* rphys) {
    Batch& B = batch();
    try {
        if (nsys < 1) throw std::runtime_error("batch needs at least one system");
        B.ensure_streams();
        // the buffers of an earlier batch may stay (below); its graph, records
        // and sizes do not
        B.drop_graph();
        B.host_events.clear();
        B.host_sys.clear();
        B.host_step.clear();
        ++B.epoch;
        B.nsys = 0;
        B.body_off.assign(body_offset, body_offset + nsys + 1);
        B.nbody = body_offset[nsys];
        B.nbig.assign(nbig, nbig + nsys);
        B.h.assign(h, h + nsys);
        B.np.resize(nsys);
        B.first_slot.resize(nsys);
        B.big_off.resize(nsys);
        B.mu.resize(nsys);
        B.sys.resize(nsys);
        B.max_nbig = 1;
        B.max_body = 1;
        int slots = 0, bigs = 0;
        std::vector<BatchTile> tiles;
        for (int s = 0; s < nsys; ++s) {
            const int n = B.body_off[s + 1] - B.body_off[s];
            if (n < 1 || B.nbig[s] < 1 || B.nbig[s] > n) throw std::runtime_error("invalid body counts of a system");
            if (B.nbig[s] > BATCH_MAX_NBIG) throw std::runtime_error("more than 32 Big bodies in a batched system");
            if (!(B.h[s] != 0.0) || !std::isfinite(B.h[s])) throw std::runtime_error("invalid step of a system");
            B.max_body = std::max(B.max_body, n);
            for (int j = B.body_off[s] + B.nbig[s]; j < B.body_off[s + 1]; ++j)
                if (m[j] != 0.0) throw std::runtime_error("batched systems take massless Small bodies only");
            B.np[s] = n - B.nbig[s];
            B.first_slot[s] = slots;
            B.big_off[s] = bigs;
            B.mu[s] = m[B.body_off[s]];
            B.max_nbig = std::max(B.max_nbig, B.nbig[s]);
            for (int t = 0; t < B.np[s]; t += 32) tiles.push_back(BatchTile{s, slots + t, std::min(32, B.np[s] - t), 0});
            slots += B.np[s];
            bigs += B.nbig[s];
            BatchSys& S = B.sys[s];
            S.mu = B.mu[s];
            S.h = B.h[s];
            S.nbig = B.nbig[s];
            S.nb = B.nbig[s] - 1;
            S.first_slot = B.first_slot[s];
            S.np = B.np[s];
            S.body = B.body_off[s];
            S.big_off = B.big_off[s];
        }
        B.npcap = std::max(1, slots);
        B.ntiles = (int)tiles.size();
        B.nbigs = bigs;
        auto reserve = [&] {
            B.d_sys.reserve(nsys);
            B.d_tiles.reserve(std::max(1, B.ntiles));
            B.d_proto.reserve(nsys);
            for (int k = 0; k < 2; ++k) {
                B.bigbuf[k].reserve((size_t)9 * bigs);
                B.pstate[k].reserve((size_t)9 * B.npcap);
            }
            B.bm.reserve(bigs);
            B.brce.reserve(bigs);
            B.brphys.reserve(bigs);
            B.prce.reserve(B.npcap);
            B.prphys.reserve(B.npcap);
            B.plocal.reserve(B.npcap);
            B.room_for(std::max(4096, B.npcap / 64), std::max(16384, B.npcap / 2));
            B.status.reserve(1);
            B.snap.reserve((size_t)9 * B.npcap + (size_t)9 * bigs);
            B.d_body_end.reserve(nsys);
            layout_tables(B, B.forced_K > 0 ? B.forced_K : 31);   // copies the systems' records
        };
        // An earlier batch's buffers stay for one of about its size (until
        // batch_free, or until room is short): programs upload batch after batch,
        // and allocating some hundred MB takes as long as copying them
        const size_t spare = (size_t)1 << 20;
        if (B.pstate[0].n > (size_t)9 * B.npcap / 4 * 5 + spare || B.bigbuf[0].n > (size_t)9 * bigs / 4 * 5 + spare)
            B.release_buffers();
        B.nsys = nsys;
        try {
            reserve();
        } catch (const CudaError&) {
            cudaGetLastError();
            B.release_buffers();
            reserve();
        }
        // every host array in one round of copies; layout on the device
        const size_t o = B.body_off[0], n = B.nbody - o;
        auto rows = [&](size_t at, const double* a, size_t width) {
            return HostSpan{B.snap.p + at * n, const_cast<double*>(a) + width * o, sizeof(double) * width * n};
        };
        std::vector<HostSpan> spans = {
            rows(0, xx, 3), rows(3, vv, 3), rows(6, m, 1), rows(7, rce, 1), rows(8, rphys, 1),
            {B.d_body_end.p, B.body_off.data() + 1, sizeof(int) * nsys}};
        if (B.ntiles) spans.push_back({B.d_tiles.p, tiles.data(), sizeof(BatchTile) * B.ntiles});
        copy_in(spans, B.stream);
        // per-system Big-body argument templates (in = set 0, out = set 1)
        std::vector<MvsBigArgs> proto(nsys);
        for (int s = 0; s < nsys; ++s) {
            MvsBigArgs& a = proto[s];
            a = MvsBigArgs{};
            a.nbig = B.nbig[s];
            a.h = B.h[s];
            a.m = B.bm.p + B.big_off[s];
            a.rce = B.brce.p + B.big_off[s];
            a.rphys = B.brphys.p + B.big_off[s];
            for (int k = 0; k < 2; ++k) {
                BigState& st = k ? a.out : a.in;
                double* base = B.bigbuf[k].p + 9 * (size_t)B.big_off[s];
                st.x = base;
                st.v = base + 3 * B.nbig[s];
                st.a = base + 6 * B.nbig[s];
            }
        }
        h2d(B.d_proto.p, proto.data(), sizeof(MvsBigArgs) * nsys, B.stream);
        B.cur = 0;
        launch_batch_rows<false>(B);
        check(cudaMemsetAsync(B.bigbuf[1].p, 0, sizeof(double) * 9 * bigs, B.stream), "upload");
        check(cudaMemsetAsync(B.pstate[1].p, 0, sizeof(double) * 9 * B.npcap, B.stream), "upload");
        check(cudaStreamSynchronize(B.stream), "upload");
        B.reset = true;
        B.threads = 0;
        B.tuned_K = 31;
        B.tuned_threads = 128;
        return 0;
    } catch (const std::exception& e) {
        B.nsys = 0;
        return report(e);
    }
}

int mercury_b200_batch_advance(double time, int nsteps, double rcen, int* nevents) {
    Batch& B = batch();
    try {
        if (B.nsys < 1) throw std::runtime_error("no batch uploaded");
        if (nsteps < 1) throw std::runtime_error("nsteps must be positive");
        if (B.threads == 0) tune(B, rcen, nsteps);
        int K = B.forced_K > 0 ? B.forced_K : B.tuned_K;
        K = std::max(1, std::min(K, nsteps));
        if (K != B.K) layout_tables(B, K);
        size_records(B, nsteps, K);
        const int nchunks = (nsteps + K - 1) / K;
        B.ensure_chunk_events(std::max(2, nchunks));
        const int reset0 = B.reset ? 1 : 0;
        // starting state, for a redo after an event-buffer overflow
        const size_t bigs = (size_t)B.nbigs;
        auto copy = [&](void* d, const void* s, size_t bytes) {
            check(cudaMemcpyAsync(d, s, bytes, cudaMemcpyDeviceToDevice, B.stream), "snapshot");
        };
        copy(B.snap.p, B.pstate[B.cur].p, sizeof(double) * 9 * B.npcap);
        copy(B.snap.p + 9 * (size_t)B.npcap, B.bigbuf[B.cur].p, sizeof(double) * 9 * bigs);
        int launches = 0;
        for (int attempt = 0;; ++attempt) {
            const auto key = std::make_tuple(nsteps, K, B.threads, reset0, B.cur, rcen, B.epoch);
            check(cudaEventRecord(B.t0, B.stream), "event");
            if (B.use_graph) {
                if (!B.exec || B.graph_key != key) {
                    B.drop_graph();
                    check(cudaStreamBeginCapture(B.stream, cudaStreamCaptureModeThreadLocal), "capture");
                    launches = enqueue_run(B, nsteps, rcen, reset0, 1);
                    check(cudaStreamEndCapture(B.stream, &B.graph), "capture");
                    check(cudaGraphInstantiate(&B.exec, B.graph, 0), "graph");
                    B.graph_key = key;
                }
                launches = 1 + (B.ntiles > 0 ? 2 : 0);
                launches = nchunks * launches;
                check(cudaGraphLaunch(B.exec, B.stream), "graph");
            } else {
                launches = enqueue_run(B, nsteps, rcen, reset0, 1);
            }
            check(cudaEventRecord(B.t1, B.stream), "event");
            check(cudaMemcpyAsync(B.status_host, B.status.p, sizeof(DeviceStatus), cudaMemcpyDeviceToHost, B.stream),
                  "status");
            check(cudaStreamSynchronize(B.stream), "advance");
            check(cudaGetLastError(), "advance");
            if (B.status_host->fault) throw std::runtime_error("MVS force failed");
            if (!B.status_host->overflow) break;
            if (attempt > 8) throw std::runtime_error("event buffer growth failed");
            copy(B.pstate[B.cur].p, B.snap.p, sizeof(double) * 9 * B.npcap);
            copy(B.bigbuf[B.cur].p, B.snap.p + 9 * (size_t)B.npcap, sizeof(double) * 9 * bigs);
            const int over = B.status_host->overflow;
            B.room_for(over & 1 ? std::max(2 * B.events.n, (size_t)B.status_host->events + 1024) : 0,
                       over & 2 ? 2 * B.cands.n + 4096 : 0);
        }
        check(cudaEventElapsedTime(&B.last_ms, B.t0, B.t1), "timer");
        B.last_launches = launches;
        B.cur = (B.cur + nchunks) & 1;
        B.reset = false;
        const int nev = B.status_host->events;
        B.host_events.resize(nev);
        B.host_sys.resize(nev);
        B.host_step.resize(nev);
        if (nev) {
            check(cudaMemcpy(B.host_events.data(), B.events.p, sizeof(MercuryEvent) * nev, cudaMemcpyDeviceToHost),
                  "events");
            check(cudaMemcpy(B.host_sys.data(), B.event_sys.p, sizeof(int) * nev, cudaMemcpyDeviceToHost), "events");
            check(cudaMemcpy(B.host_step.data(), B.event_step.p, sizeof(int) * nev, cudaMemcpyDeviceToHost),
                  "events");
        }
        // absolute times on each system's own clock (time = time + h per step)
        std::vector<std::vector<double>> tend(B.nsys);
        for (int k = 0; k < nev; ++k) {
            const int s = B.host_sys[k];
            if (tend[s].empty()) {
                tend[s].resize(nsteps);
                double tt = time;
                for (int q = 0; q < nsteps; ++q) {
                    tt = tt + B.h[s];
                    tend[s][q] = tt;
                }
            }
            MercuryEvent& e = B.host_events[k];
            const double te = tend[s][B.host_step[k]];
            if (e.kind == EV_CENTRAL) e.time = te - B.h[s] + e.time;
            else e.time = e.time + te;
        }
        sort_batch_events(B);
        *nevents = nev;
        return 0;
    } catch (const std::exception& e) {
        return report(e);
    }
}

int mercury_b200_batch_events(MercuryEvent* events, int* sys, int* steps, int cap) {
    Batch& B = batch();
    const int nev = (int)B.host_events.size();
    const int k = std::min(cap, nev);
    if (k > 0) {
        std::memcpy(events, B.host_events.data(), sizeof(MercuryEvent) * k);
        if (sys) std::memcpy(sys, B.host_sys.data(), sizeof(int) * k);
        if (steps) std::memcpy(steps, B.host_step.data(), sizeof(int) * k);
    }
    return nev;
}

int mercury_b200_batch_download(double* xx, double* vv) {
    Batch& B = batch();
    try {
        if (B.nsys < 1) throw std::runtime_error("no batch uploaded");
        const size_t o = B.body_off[0], n = B.nbody - o;   // rows before the first system are not the batch's
        launch_batch_rows<true>(B);
        copy_out({{B.snap.p, xx + 3 * o, 24 * n}, {B.snap.p + 3 * n, vv + 3 * o, 24 * n}}, B.stream);
        return 0;
    } catch (const std::exception& e) {
        return report(e);
    }
}

int mercury_b200_batch_set(int threads, int steps_per_launch, int use_graph) {
    Batch& B = batch();
    if (threads > 0 && threads != 64 && threads != 128 && threads != 256) return 1;
    if (threads >= 0) {
        B.forced_threads = threads;
        B.threads = 0;   // tuned again (over K only when threads is forced)
    }
    if (steps_per_launch >= 0) {
        B.forced_K = std::min(steps_per_launch, 64);
        B.threads = 0;
    }
    if (use_graph >= 0) B.use_graph = use_graph ? 1 : 0;
    return 0;
}

int mercury_b200_batch_timing(double* ms, int* launches, int* threads, int* steps_per_launch) {
    Batch& B = batch();
    if (ms) *ms = B.last_ms;
    if (launches) *launches = B.last_launches;
    if (threads) *threads = B.threads;
    if (steps_per_launch) *steps_per_launch = B.K;
    return 0;
}

void mercury_b200_batch_free(void) { batch().release(); }

}  // extern "C"
