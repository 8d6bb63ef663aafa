// kernels.cu -- the device kernels of the PDLP engine (sm_100a).
//
// Hot path, per linesearch trial (pdlp_engine/src/pdhg_kernel.cpp:47-277):
//   k_primal  over the A^T side: g = c + A'y, x' = clip(x - (eta/omega) tau g),
//             sum dx^2/tau; applies the iterate-average update owed by the last
//             commit (iterate_average.cpp:40-82) while x is in registers.
//   k_dual    over the A side: A x', extrapolation 2Ax' - Ax, dual prox
//             y' = max(v - s u, 0) + min(v - s l, 0), sum dy^2/sigma and
//             dy'(A dx); owed average update of y.
//   k_decide  per instance: the linesearch decision and commit (trial_control).
// Every check_frequency iterations (termination.cpp:66-325,
// infeasibility.cpp:51-192, pdlp_solver.cpp:354-476), in FP64 on the original
// problem:
//   k_check_prep   elementwise: original-coordinate copies of the current and
//                  averaged iterates and of the ray directions, and every
//                  reduction that needs no matrix product
//   k_check_spmv   both matrix passes at once, each gathering up to three
//                  vectors; the last CTA of an instance decides (best point,
//                  certificates, termination, restart)
//   k_check_apply  best-point copies, restarts, polishing entry, ray copies
//   k_refresh      A x after an iterate was replaced
//   k_finalize     clears the per-check flags
// Setup: Ruiz max-abs passes, scaled coefficients, Pock-Chambolle sums.
//
// Gathers go through the read-only path; matrix streams use 128-bit loads
// when the vector width allows. No atomics touch numerical data: the only
// atomic is the per-instance arrival counter.
#include "control.cuh"
#include "kernels.cuh"
#include "ndg.cuh"

#include <algorithm>
#include <cstdio>

namespace pdlpgpu {
namespace {

constexpr unsigned kFull = 0xffffffffu;

// ---------------------------------------------------------------------------
// Loads of V consecutive elements (V in {1, 2, 4}); the caller guarantees
// V-element alignment.
// ---------------------------------------------------------------------------
template <int V> __device__ __forceinline__ void ld(const int32_t* p, int32_t (&o)[V]);
template <> __device__ __forceinline__ void ld<1>(const int32_t* p, int32_t (&o)[1]) { o[0] = __ldg(p); }
template <> __device__ __forceinline__ void ld<2>(const int32_t* p, int32_t (&o)[2]) {
    const int2 v = __ldg(reinterpret_cast<const int2*>(p)); o[0] = v.x; o[1] = v.y;
}
template <> __device__ __forceinline__ void ld<4>(const int32_t* p, int32_t (&o)[4]) {
    const int4 v = __ldg(reinterpret_cast<const int4*>(p)); o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
}
template <int V> __device__ __forceinline__ void ld(const float* p, float (&o)[V]);
template <> __device__ __forceinline__ void ld<1>(const float* p, float (&o)[1]) { o[0] = __ldg(p); }
template <> __device__ __forceinline__ void ld<2>(const float* p, float (&o)[2]) {
    const float2 v = __ldg(reinterpret_cast<const float2*>(p)); o[0] = v.x; o[1] = v.y;
}
template <> __device__ __forceinline__ void ld<4>(const float* p, float (&o)[4]) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(p)); o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
}
template <int V> __device__ __forceinline__ void ld(const double* p, double (&o)[V]);
template <> __device__ __forceinline__ void ld<1>(const double* p, double (&o)[1]) { o[0] = __ldg(p); }
template <> __device__ __forceinline__ void ld<2>(const double* p, double (&o)[2]) {
    const double2 v = __ldg(reinterpret_cast<const double2*>(p)); o[0] = v.x; o[1] = v.y;
}
template <> __device__ __forceinline__ void ld<4>(const double* p, double (&o)[4]) {
    const double2 a = __ldg(reinterpret_cast<const double2*>(p));
    const double2 b = __ldg(reinterpret_cast<const double2*>(p + 2));
    o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
}

// Lane position inside a slice.
struct LanePos {
    int glog;     // log2 of the lane group
    int g;        // lane inside the group
    int line;     // local line index
    bool valid;   // the lane's line exists
};

__device__ __forceinline__ LanePos lane_pos(const SliceDesc& sd, int lane) {
    LanePos p;
    p.glog = slice_glog(sd.meta);
    const int r = lane >> p.glog;
    p.g = lane & ((1 << p.glog) - 1);
    p.line = sd.line0 + r;
    p.valid = r < slice_lines(sd.meta);
    return p;
}

// Sum of NQ products over the lane's entries of one line, then combined over
// the G lanes of the line with an xor butterfly (every lane ends with the same
// bits, so the result is deterministic). Up to kDepth vector loads of index
// and value are issued before their gathers, so a lane keeps several
// independent memory requests in flight instead of one load-gather chain.
// kDeep doubles the depth for FP32 vector loads (measured: the dual kernel
// gains, the primal kernel, whose lanes also stream five vectors, loses).
template <int V, int NQ, bool kDeep = false, class TA, class TV, class F>
__device__ __forceinline__ void line_sums(int64_t base, int steps, const LanePos& lp, int lane,
                                          int len, const int32_t* __restrict__ idx,
                                          const TV* __restrict__ val, TA (&acc)[NQ], F fetch) {
    // About four entries in flight per lane, eight for deep FP32 vector
    // loads (deeper FP64 or scalar pipelines spill at 64 registers).
    constexpr int kDepth = (kDeep && V >= 2 && sizeof(TV) == 4) ? 8 / V : (V >= 4 ? 1 : 4 / V);
    constexpr int kStep = kDepth * V;
    // Software pipeline: the index and value loads of the next group are in
    // flight while the current group's gathers are.
    auto load = [&](int s0, int32_t (&id)[kDepth][V], TV (&v)[kDepth][V]) {
#pragma unroll
        for (int u = 0; u < kDepth; ++u) {
            const int s = s0 + u * V;
            if (s < steps) {
                const int64_t p = base + static_cast<int64_t>(s) * 32 + lane * V;
                ld<V>(idx + p, id[u]);
                ld<V>(val + p, v[u]);
            } else {
#pragma unroll
                for (int q = 0; q < V; ++q) {
                    id[u][q] = 0;
                    v[u][q] = TV(0);
                }
            }
        }
    };
    int32_t id[kDepth][V];
    TV v[kDepth][V];
    load(0, id, v);
    for (int s0 = 0; s0 < steps; s0 += kStep) {
        int32_t nid[kDepth][V];
        TV nv[kDepth][V];
        load(s0 + kStep, nid, nv);
#pragma unroll
        for (int u = 0; u < kDepth; ++u) {
#pragma unroll
            for (int q = 0; q < V; ++q) {
                const int k = ((s0 + u * V + q) << lp.glog) + lp.g;
                if (k < len) fetch(acc, static_cast<TA>(v[u][q]), id[u][q]);
            }
        }
#pragma unroll
        for (int u = 0; u < kDepth; ++u)
#pragma unroll
            for (int q = 0; q < V; ++q) {
                id[u][q] = nid[u][q];
                v[u][q] = nv[u][q];
            }
    }
    for (int o = (1 << lp.glog) >> 1; o > 0; o >>= 1) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) acc[q] += __shfl_xor_sync(kFull, acc[q], o);
    }
}

// Block-wide deterministic sum of NQ doubles; the result is valid in thread 0.
template <int NQ>
__device__ __forceinline__ void block_sum(double (&v)[NQ]) {
    __shared__ double red[NQ][kWarps * 4];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int warps = blockDim.x >> 5;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(kFull, v[q], o);
    }
    if (lane == 0) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) red[q][warp] = v[q];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            double t = 0.0;
            for (int w = 0; w < warps; ++w) t += red[q][w];
            v[q] = t;
        }
    }
}

// Warp-0 deterministic sum over a range of per-CTA partials (stride `slots`).
__device__ __forceinline__ double warp_range_sum(const double* part, int begin, int end,
                                                 int slots, int slot) {
    const int lane = threadIdx.x & 31;
    double t = 0.0;
    for (int k = begin + lane; k < end; k += 32) t += part[static_cast<int64_t>(k) * slots + slot];
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(kFull, t, o);
    return t;
}

// Arrival counter: returns true in every thread of the CTA that arrives last
// among `expected` CTAs of the instance (and resets the counter for the next
// launch, which a kernel boundary orders). Partials written before the call
// are visible to that CTA. One thread arrives for the CTA with an
// acquire-release atomic at GPU scope: the barrier orders the other threads'
// writes before it, its release publishes them, and in the last CTA its
// acquire makes every earlier arrival's writes visible -- one round trip
// where a full fence and an atomic took two.
__device__ __forceinline__ bool arrive_last(int32_t* counter, int expected) {
    __shared__ int last;
    __syncthreads();
    if (threadIdx.x == 0) {
        int prev;
        asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(prev) : "l"(counter) : "memory");
        last = prev == expected - 1;
        if (last) *counter = 0;
    }
    __syncthreads();
    return last != 0;
}


// Programmatic dependent launch of the trial kernels (k_primal, k_dual,
// k_decide): each lets its successor start as its own CTAs leave, and reads what
// a trial kernel writes only after the wait, which returns once every earlier
// kernel has ended and its writes are visible. Before it only data that no
// trial kernel writes is read (heads, entries). Every CTA waits: a kernel's end
// then means that all before it have ended.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Non-binding L2 prefetch of [p, p + bytes), shrunk inward to 16-byte
// boundaries (so it never reaches outside the range) and cut into pieces of at
// most 32 KiB spread over the warp's lanes starting at lane `first`.
__device__ __forceinline__ void prefetch_range(const void* p, int64_t bytes, int first, int lane) {
    if (bytes <= 0) return;
    const uintptr_t a = (reinterpret_cast<uintptr_t>(p) + 15) & ~uintptr_t(15);
    const uintptr_t e = (reinterpret_cast<uintptr_t>(p) + static_cast<uintptr_t>(bytes)) & ~uintptr_t(15);
    if (e <= a) return;
    constexpr uintptr_t kPiece = 32768;
    const uintptr_t pieces = (e - a + kPiece - 1) / kPiece;
    for (uintptr_t k = (static_cast<unsigned>(first) + lane) % 32; k < pieces; k += 32) {
        const uintptr_t b = a + k * kPiece;
        const uint32_t n = static_cast<uint32_t>(e - b < kPiece ? e - b : kPiece);
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(b), "r"(n) : "memory");
    }
}

// The streams of an entry with more slices than warps, prefetched into L2 by the
// warp that starts its first record: its later slices find them there. `off`:
// the instance's first line.
template <class T, int NV>
__device__ __forceinline__ void prefetch_entry(const Side& side, int slice_begin, int slice_end, int64_t data_base,
                                               int64_t off, const T* vals, const T* const (&vecs)[NV], int nvec,
                                               int lane) {
    const SliceDesc first = side.slices[slice_begin], last = side.slices[slice_end - 1];
    const int64_t e0 = data_base + static_cast<int64_t>(first.data_off) * 32;
    const int64_t e1 = data_base + (static_cast<int64_t>(last.data_off) + last.steps) * 32;
    prefetch_range(side.idx + e0, (e1 - e0) * 4, 0, lane);
    prefetch_range(vals + e0, (e1 - e0) * static_cast<int64_t>(sizeof(T)), 8, lane);
    const int64_t l0 = off + first.line0, l1 = off + last.line0 + slice_lines(last.meta);
    for (int v = 0; v < nvec; ++v)
        prefetch_range(vecs[v] + l0, (l1 - l0) * static_cast<int64_t>(sizeof(T)), 16 + 2 * v, lane);
}

__device__ __forceinline__ bool check_have_avg(const InstanceCtl& c, const DeviceOptions& o) {
    if (c.check_kind == kCheckInitial) return c.have_avg_at_check != 0;
    return o.averaging && c.avg_weight != 0.0;
}

template <class T> __device__ __forceinline__ const T* matrix_values(const Side& s);
template <> __device__ __forceinline__ const double* matrix_values<double>(const Side& s) { return s.val_s64; }
template <> __device__ __forceinline__ const float* matrix_values<float>(const Side& s) { return s.val_s32; }


// ---------------------------------------------------------------------------
// The trial kernels: the primal half (pdhg_kernel.cpp:47-104), the dual half and
// the decision. A CTA takes every gridDim-th entry of the CTA map, as many
// CTAs as the device holds at once. What starts an entry -- a record per warp
// (WarpHead) and the instance's step (TrialParams) -- is brought into shared
// memory for up to kTrialTile entries at once, and an entry's first slots and
// indices are loaded while the gathers of the entry before it are in flight.
//
// Bound by latency: what a lane waits for is a gather of L2 under load (about
// 2000 cycles). Of the 38 us of a 200k x 400k FP64 trial (2M entries) the random
// gathers alone would take 14 (285 G a second measured), its 93 MB of streams 14
// at HBM's rate. A CTA per entry, each following map, instance, slice table and
// slots one after the other (14k cycles, three waves), and the decision in
// k_dual's last CTA (21k cycles, its partials a round trip to L2 per 32) took
// 60 us; FP32, 48 LPs of 200 to 20000 rows: 51 -> 40 us.
// ---------------------------------------------------------------------------
constexpr int kTrialTile = 32;
template <class T> constexpr int kTrialCtas = sizeof(T) == 8 ? 2 : 3;   // per SM: 128 and 80 registers a thread

template <class T>
struct alignas(16) TrialParams {
    T mult;      // the half's step
    T frac;      // of the pending average update
    int32_t parity, pending, active;
};

template <class T>
struct TrialShared {
    WarpHead heads[kTrialTile][kWarps];
    TrialParams<T> params[kTrialTile];
    double red[kTrialTile][kWarps][2];   // a record's sums
};

// The tile's records: entries blockIdx.x + (t0 + i) gridDim.x, i < n.
__device__ __forceinline__ void load_heads(const Side& side, int t0, int n, WarpHead (*heads)[kWarps]) {
    constexpr int kWords = kWarps * static_cast<int>(sizeof(WarpHead) / 16);
    for (int k = threadIdx.x; k < n * kWords; k += kThreads) {
        const int64_t e = blockIdx.x + static_cast<int64_t>(t0 + k / kWords) * gridDim.x;
        reinterpret_cast<int4*>(heads)[k] = __ldg(reinterpret_cast<const int4*>(side.heads + e * kWarps) + k % kWords);
    }
}

// Lane i's entry of the tile: its instance's step, and whether it runs.
template <class T, bool kDual>
__device__ __forceinline__ TrialParams<T> trial_params(const Global& g, int instance) {
    const InstanceCtl& c = g.ctl[instance];
    TrialParams<T> k;
    k.mult = static_cast<T>(kDual ? c.trial_eta * c.trial_omega : c.trial_eta / c.trial_omega);
    k.frac = static_cast<T>(c.avg_frac);
    k.parity = c.parity;
    k.pending = !g.measure && c.pending_avg != 0;
    k.active = g.measure || trial_active<T>(c);
    return k;
}

// A lane's place in its warp's current slice.
struct LineAt {
    LanePos lp;
    int steps, len;
    int base, line;   // the slice's first slot / 32; the line in its whole space

    __device__ __forceinline__ bool owner() const { return lp.valid && lp.g == 0; }
    __device__ __forceinline__ int64_t slot0() const { return static_cast<int64_t>(base) * 32; }
    __device__ __forceinline__ void at(const Side& side, int base32, int line0, int len0, int nsteps, int meta,
                                       int lane) {
        const SliceDesc sd{0, 0, nsteps, meta};
        lp = lane_pos(sd, lane);
        steps = nsteps;
        base = base32;
        line = line0 + lp.line;
        len = lp.valid ? side.line_len[len0 + lp.line] : 0;
    }
    __device__ __forceinline__ void first(const Side& side, const WarpHead& h, int lane) {
        at(side, h.base, h.line, h.len, h.steps, h.meta, lane);
    }
    // A later slice of the warp (CTAs with more slices than warps).
    __device__ __forceinline__ void later(const Side& side, int64_t data_base, int64_t off, int64_t len_base,
                                          int slice, int lane) {
        const SliceDesc sd = side.slices[slice];
        at(side, static_cast<int>(data_base / 32) + sd.data_off, static_cast<int>(off) + sd.line0,
           static_cast<int>(len_base) + sd.line0, sd.steps, sd.meta, lane);
    }
};

// A lane's entries in flight at once: four. With eight, which is a whole line for
// a lane of all but the longest lines, FP64 spills at 128 registers (a trial of
// 200k x 400k 40.3 us for 37.9) and FP32 has room for two CTAs an SM instead of
// three (48 LPs of 200 to 20000 rows 41.3 us for 39.6).
constexpr int kGroup = 4;
template <class T>
struct LineGroup {
    int32_t id[kGroup];
    T v[kGroup];

    __device__ __forceinline__ void load(const Side& side, const T* vals, const LineAt& a, int s0, int lane) {
#pragma unroll
        for (int u = 0; u < kGroup; ++u) {
            if (s0 + u < a.steps) {
                const int64_t p = a.slot0() + static_cast<int64_t>(s0 + u) * 32 + lane;
                id[u] = __ldg(side.idx + p);
                v[u] = __ldg(vals + p);
            }
        }
    }
};

// The line's product with the vector x, every lane of the line's group with the
// same bits: line_sums from a loaded first group.
template <class T>
__device__ __forceinline__ T line_product(LineGroup<T>& group, const Side& side, const T* vals, const LineAt& a,
                                          int lane, const T* x) {
    // The lane has an entry in step s while (s << glog) + g < len.
    const int mine = (a.len - a.lp.g + (1 << a.lp.glog) - 1) >> a.lp.glog;
    T sum = T(0);
    for (int s0 = 0;;) {
        T xs[kGroup];
#pragma unroll
        for (int u = 0; u < kGroup; ++u)
            if (s0 + u < mine) xs[u] = x[group.id[u]];
#pragma unroll
        for (int u = 0; u < kGroup; ++u)
            if (s0 + u < mine) sum += group.v[u] * xs[u];
        s0 += kGroup;
        if (s0 >= a.steps) break;
        group.load(side, vals, a, s0, lane);
    }
    for (int o = (1 << a.lp.glog) >> 1; o > 0; o >>= 1) sum += __shfl_xor_sync(kFull, sum, o);
    return sum;
}

// One half of a trial over the CTA's entries. `body(i, r, at, group, v)` runs the
// slices of entry i's record r; its NR sums are added over the lanes at once,
// over the entry's records in order at the end of the tile, and stored to
// part[NR * entry + q]: the warps wait for one another once a tile, not once an
// entry. A warp takes another record in each entry, since the last records of
// many entries have no slice.
template <class T, int NR, bool kDual, class Body>
__device__ __forceinline__ void trial_half(const Global& g, const Side& side, TrialShared<T>& sh, double* part,
                                           Body body) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const T* vals = matrix_values<T>(side);
    const int mine = (side.num_ctas - static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) - 1) /
                     static_cast<int>(gridDim.x);
    for (int t0 = 0; t0 < mine; t0 += kTrialTile) {
        const int n = min(kTrialTile, mine - t0);
        if (t0 > 0) __syncthreads();
        load_heads(side, t0, n, sh.heads);
        __syncthreads();
        // The first entry is opened before it is known whether it runs.
        LineAt at, next_at;
        LineGroup<T> group, next_group;
        auto record = [&](int i) { return (warp + 3 * i) % kWarps; };
        auto open = [&](int i, LineAt& a, LineGroup<T>& gr) {
            a.first(side, sh.heads[i][record(i)], lane);
            gr.load(side, vals, a, 0, lane);
        };
        open(0, at, group);
        if (t0 == 0) {
            pdl_wait();
            if (kDual) pdl_trigger();
        }
        if (static_cast<int>(threadIdx.x) < n)
            sh.params[threadIdx.x] = trial_params<T, kDual>(g, sh.heads[threadIdx.x][0].instance);
        __syncthreads();
        const unsigned runs = __ballot_sync(kFull, lane < n && sh.params[lane].active != 0);
        int i = __ffs(runs) - 1;
        if (i > 0) open(i, at, group);
        while (i >= 0) {
            const int next = __ffs(runs & ~((2u << i) - 1u)) - 1;
            if (next >= 0) open(next, next_at, next_group);
            double v[NR];
#pragma unroll
            for (int q = 0; q < NR; ++q) v[q] = 0.0;
            const int r = record(i);
            body(i, r, at, group, v);
#pragma unroll
            for (int q = 0; q < NR; ++q) {
                for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(kFull, v[q], o);
                if (lane == 0) sh.red[i][r][q] = v[q];
            }
            i = next;
            at = next_at;
            group = next_group;
        }
        __syncthreads();
        for (int k = threadIdx.x; k < n * NR; k += kThreads) {
            const int e = k / NR, q = k % NR;
            if (!((runs >> e) & 1u)) continue;
            double t = 0.0;
            for (int w = 0; w < kWarps; ++w) t += sh.red[e][w][q];
            part[NR * (blockIdx.x + static_cast<int64_t>(t0 + e) * gridDim.x) + q] = t;
        }
    }
}

template <class T>
__global__ void __launch_bounds__(kThreads, kTrialCtas<T>) k_primal(Global g, Work<T> w) {
    __shared__ TrialShared<T> sh;
    pdl_trigger();
    const int lane = threadIdx.x & 31;
    const T* vals = matrix_values<T>(g.at);
    auto body = [&](int i, int r, LineAt& at, LineGroup<T>& group, double (&moved)[1]) {
        const WarpHead& h = sh.heads[i][r];
        const TrialParams<T> k = sh.params[i];
        // Written by other kernels of the stream while this one may be
        // waiting: no __restrict__.
        const T* y = w.Y[k.parity] + h.other;
        const T* x = w.X[k.parity];
        T* xt = w.X[k.parity ^ 1];
        T* avg = w.avg_x;
        const InstanceInfo& inf = g.info[h.instance];
        if (h.many && r == 0) {
            const T* const vecs[7] = {x, w.c, w.xl, w.xu, w.tau, w.itau, avg};
            prefetch_entry<T, 7>(g.at, h.slice, h.slice_end, inf.at_data_base, inf.col_off, vals, vecs,
                                 k.pending ? 7 : 6, lane);
        }
        for (int s = h.slice; s < h.slice_end;) {
            // The epilogue's operands do not depend on the product: loaded
            // first, their latency overlaps the gathers'.
            T cj = T(0), prev = T(0), loj = T(0), hij = T(0), tj = T(0), itj = T(0), aj = T(0);
            if (at.owner()) {
                cj = __ldg(w.c + at.line);
                prev = x[at.line];
                loj = __ldg(w.xl + at.line);
                hij = __ldg(w.xu + at.line);
                tj = __ldg(w.tau + at.line);
                itj = __ldg(w.itau + at.line);
                if (k.pending) aj = avg[at.line];
            }
            const T sum = line_product(group, g.at, vals, at, lane, y);
            if (at.owner()) {
                const T gradient = cj + sum;
                const T upd = smax(loj, smin(prev - k.mult * tj * gradient, hij));
                xt[at.line] = upd;
                const double d = static_cast<double>(upd - prev);
                moved[0] += d * d * static_cast<double>(itj);
                if (k.pending) avg[at.line] = aj + k.frac * (prev - aj);
            }
            s += kWarps;
            if (s < h.slice_end) {
                at.later(g.at, inf.at_data_base, inf.col_off, inf.at_len_base, s, lane);
                group.load(g.at, vals, at, 0, lane);
            }
        }
    };
    trial_half<T, 1, false>(g, g.at, sh, g.part_primal, body);
}

// ---------------------------------------------------------------------------
// Dual half (pdhg_kernel.cpp:109-187) and the trial decision
// ---------------------------------------------------------------------------
template <class T>
__global__ void __launch_bounds__(kThreads, kTrialCtas<T>) k_dual(Global g, Work<T> w) {
    __shared__ TrialShared<T> sh;
    const int lane = threadIdx.x & 31;
    const T* vals = matrix_values<T>(g.a);
    auto body = [&](int i, int r, LineAt& at, LineGroup<T>& group, double (&red)[2]) {
        const WarpHead& h = sh.heads[i][r];
        const TrialParams<T> k = sh.params[i];
        const T* xt = w.X[k.parity ^ 1] + h.other;
        const T* y = w.Y[k.parity];
        T* yt = w.Y[k.parity ^ 1];
        const T* ax = w.AX[k.parity];
        T* axt = w.AX[k.parity ^ 1];
        T* avg = w.avg_y;
        const InstanceInfo& inf = g.info[h.instance];
        if (h.many && r == 0) {
            const T* const vecs[7] = {ax, y, w.rl, w.ru, w.sigma, w.isigma, avg};
            prefetch_entry<T, 7>(g.a, h.slice, h.slice_end, inf.a_data_base, inf.row_off, vals, vecs,
                                 k.pending ? 7 : 6, lane);
        }
        for (int s = h.slice; s < h.slice_end;) {
            T axi = T(0), sgi = T(0), prev = T(0), loi = T(0), hii = T(0), isi = T(0), ai = T(0);
            if (at.owner()) {
                axi = ax[at.line];
                sgi = __ldg(w.sigma + at.line);
                prev = y[at.line];
                loi = __ldg(w.rl + at.line);
                hii = __ldg(w.ru + at.line);
                isi = __ldg(w.isigma + at.line);
                if (k.pending) ai = avg[at.line];
            }
            const T sum = line_product(group, g.a, vals, at, lane, xt);
            if (at.owner()) {
                const T next = sum;
                const T dact = next - axi;
                const T ext = next + dact;
                const T step = smax(k.mult * sgi, min_dual_step<T>());
                const T v = prev + step * ext;
                const T upd = smax(v - step * hii, T(0)) + smin(v - step * loi, T(0));
                yt[at.line] = upd;
                axt[at.line] = next;
                const double d = static_cast<double>(upd - prev);
                red[0] += d * d * static_cast<double>(isi);
                red[1] += d * static_cast<double>(dact);
                if (k.pending) avg[at.line] = ai + k.frac * (prev - ai);
            }
            s += kWarps;
            if (s < h.slice_end) {
                at.later(g.a, inf.a_data_base, inf.row_off, inf.a_len_base, s, lane);
                group.load(g.a, vals, at, 0, lane);
            }
        }
    };
    trial_half<T, 2, true>(g, g.a, sh, g.part_dual, body);
}

// The two halves for long lines (V > 1: a mean of 12 entries, FP64 16, or more): a
// CTA per entry, four an SM, its slots streamed V at a time with a group ahead.
// Such matrices are streams more than gathers, and the bytes in flight count: on
// 1024 LPs of 200 to 50000 rows (145M entries, FP32, V = 4) these take 525 and
// 504 us where the kernels above, at two CTAs an SM, took 643 and 588.
template <class T, int V>
__global__ void __launch_bounds__(kThreads, 4) k_primal_wide(Global g, Work<T> w) {
    pdl_trigger();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const CtaWork cw = g.at.ctas[blockIdx.x];
    const InstanceCtl& c = g.ctl[cw.instance];
    if (!g.measure && !trial_active<T>(c)) return;
    const InstanceInfo inf = g.info[cw.instance];
    const int p = c.parity;
    const T mult = static_cast<T>(c.trial_eta / c.trial_omega);
    const bool pending = !g.measure && c.pending_avg != 0;
    const T frac = static_cast<T>(c.avg_frac);

    const T* y = w.Y[p] + inf.row_off;
    const T* x = w.X[p] + inf.col_off;
    T* __restrict__ xt = w.X[p ^ 1] + inf.col_off;
    const T* __restrict__ cv = w.c + inf.col_off;
    const T* __restrict__ lo = w.xl + inf.col_off;
    const T* __restrict__ hi = w.xu + inf.col_off;
    const T* __restrict__ tau = w.tau + inf.col_off;
    const T* __restrict__ itau = w.itau + inf.col_off;
    T* __restrict__ avg = w.avg_x + inf.col_off;
    const T* vals = matrix_values<T>(g.at);
    {
        const T* const vecs[7] = {x, cv, lo, hi, tau, itau, avg};
        if (warp == 0 && cw.slice_end > cw.slice_begin)
            prefetch_entry<T, 7>(g.at, cw.slice_begin, cw.slice_end, inf.at_data_base, 0, vals, vecs, pending ? 7 : 6, lane);
    }

    double moved[1] = {0.0};
    for (int s = cw.slice_begin + warp; s < cw.slice_end; s += kWarps) {
        const SliceDesc sd = g.at.slices[s];
        const LanePos lp = lane_pos(sd, lane);
        const bool owner = lp.valid && lp.g == 0;
        const int j = lp.line;
        const int len = lp.valid ? g.at.line_len[inf.at_len_base + j] : 0;
        // The epilogue's operands do not depend on the product: load them
        // first so their latency overlaps the gathers.
        T cj = T(0), prev = T(0), loj = T(0), hij = T(0), tj = T(0), itj = T(0), aj = T(0);
        if (owner) {
            cj = cv[j];
            prev = x[j];
            loj = lo[j];
            hij = hi[j];
            tj = tau[j];
            itj = itau[j];
            if (pending) aj = avg[j];
        }
        T sum[1] = {T(0)};
        line_sums<V, 1>(inf.at_data_base + static_cast<int64_t>(sd.data_off) * 32, sd.steps, lp,
                        lane, len, g.at.idx, vals, sum,
                        [&](T (&a)[1], T v, int i) { a[0] += v * y[i]; });
        if (owner) {
            const T gradient = cj + sum[0];
            const T upd = smax(loj, smin(prev - mult * tj * gradient, hij));
            xt[j] = upd;
            const double d = static_cast<double>(upd - prev);
            moved[0] += d * d * static_cast<double>(itj);
            if (pending) avg[j] = aj + frac * (prev - aj);
        }
    }
    block_sum<1>(moved);
    if (threadIdx.x == 0) g.part_primal[blockIdx.x] = moved[0];
}

template <class T, int V>
__global__ void __launch_bounds__(kThreads, 4) k_dual_wide(Global g, Work<T> w) {
    pdl_wait();
    pdl_trigger();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const CtaWork cw = g.a.ctas[blockIdx.x];
    InstanceCtl& c = g.ctl[cw.instance];
    if (!g.measure && !trial_active<T>(c)) return;
    const InstanceInfo inf = g.info[cw.instance];
    const int p = c.parity;
    const T dm = static_cast<T>(c.trial_eta * c.trial_omega);
    const bool pending = !g.measure && c.pending_avg != 0;
    const T frac = static_cast<T>(c.avg_frac);

    const T* xt = w.X[p ^ 1] + inf.col_off;
    const T* y = w.Y[p] + inf.row_off;
    T* __restrict__ yt = w.Y[p ^ 1] + inf.row_off;
    const T* ax = w.AX[p] + inf.row_off;
    T* __restrict__ axt = w.AX[p ^ 1] + inf.row_off;
    const T* __restrict__ lo = w.rl + inf.row_off;
    const T* __restrict__ hi = w.ru + inf.row_off;
    const T* __restrict__ sig = w.sigma + inf.row_off;
    const T* __restrict__ isig = w.isigma + inf.row_off;
    T* __restrict__ avg = w.avg_y + inf.row_off;
    const T* vals = matrix_values<T>(g.a);
    {
        const T* const vecs[7] = {ax, y, lo, hi, sig, isig, avg};
        if (warp == 0 && cw.slice_end > cw.slice_begin)
            prefetch_entry<T, 7>(g.a, cw.slice_begin, cw.slice_end, inf.a_data_base, 0, vals, vecs, pending ? 7 : 6, lane);
    }

    double red[2] = {0.0, 0.0};
    for (int s = cw.slice_begin + warp; s < cw.slice_end; s += kWarps) {
        const SliceDesc sd = g.a.slices[s];
        const LanePos lp = lane_pos(sd, lane);
        const bool owner = lp.valid && lp.g == 0;
        const int i = lp.line;
        const int len = lp.valid ? g.a.line_len[inf.a_len_base + i] : 0;
        T axi = T(0), sgi = T(0), prev = T(0), loi = T(0), hii = T(0), isi = T(0), ai = T(0);
        if (owner) {
            axi = ax[i];
            sgi = sig[i];
            prev = y[i];
            loi = lo[i];
            hii = hi[i];
            isi = isig[i];
            if (pending) ai = avg[i];
        }
        T sum[1] = {T(0)};
        line_sums<V, 1, true>(inf.a_data_base + static_cast<int64_t>(sd.data_off) * 32, sd.steps, lp,
                              lane, len, g.a.idx, vals, sum,
                              [&](T (&a)[1], T v, int j) { a[0] += v * xt[j]; });
        if (owner) {
            const T next = sum[0];
            const T dact = next - axi;
            const T ext = next + dact;
            const T step = smax(dm * sgi, min_dual_step<T>());
            const T v = prev + step * ext;
            const T upd = smax(v - step * hii, T(0)) + smin(v - step * loi, T(0));
            yt[i] = upd;
            axt[i] = next;
            const double d = static_cast<double>(upd - prev);
            red[0] += d * d * static_cast<double>(isi);
            red[1] += d * static_cast<double>(dact);
            if (pending) avg[i] = ai + frac * (prev - ai);
        }
    }
    block_sum<2>(red);
    if (threadIdx.x == 0) {
        g.part_dual[2 * blockIdx.x] = red[0];
        g.part_dual[2 * blockIdx.x + 1] = red[1];
    }
}

// warp_range_sum with up to 16 of a lane's partials in flight.
__device__ __forceinline__ double warp_range_sum_deep(const double* part, int begin, int end, int slots, int slot) {
    constexpr int kAhead = 16;
    const int lane = threadIdx.x & 31;
    double t = 0.0;
    for (int k = begin + lane; k < end; k += 32 * kAhead) {
        double v[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
            v[u] = k + 32 * u < end ? part[static_cast<int64_t>(k + 32 * u) * slots + slot] : 0.0;
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
            if (k + 32 * u < end) t += v[u];
    }
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(kFull, t, o);
    return t;
}

// The decision on a trial, a CTA per instance: the entries' partials are added
// in a fixed order, a warp per sum, then trial_control runs on a shared-memory
// copy of the control block (after a store to a global line the thread's next
// load of that line would be served by L2, and the decision reads back much of
// what it writes). The control block, the options (by reference from shared
// memory: a reference to the kernel parameter would copy it to local memory in
// every thread) and the step factors are there before the wait: only the
// previous decision writes the block, and k_dual lets this kernel start after
// its own wait, when that decision has ended.
constexpr int kDecideThreads = 96;
template <class T>
__global__ void __launch_bounds__(kDecideThreads) k_decide(Global g, DeviceOptions o) {
    __shared__ DeviceOptions so;
    __shared__ alignas(16) InstanceCtl sc;
    __shared__ double factors[2];
    __shared__ double sums[3];
    pdl_trigger();
    InstanceCtl* c = g.ctl + blockIdx.x;
    const InstanceInfo& inf = g.info[blockIdx.x];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = inf.n;
    const int begin = warp == 0 ? inf.at_cta_begin : inf.a_cta_begin;
    const int end = warp == 0 ? inf.at_cta_end : inf.a_cta_end;
    bool have = false;
    if (warp == 0) {
        if (lane < static_cast<int>(sizeof(InstanceCtl) / 16))
            reinterpret_cast<int4*>(&sc)[lane] = __ldcg(reinterpret_cast<const int4*>(c) + lane);
        __syncwarp();
        const int64_t k = sc.phase == kPhasePolish ? sc.polish_iteration : sc.iteration;
        have = k >= 0 && k < o.step_pow_entries;
        if (have && lane < 2) factors[lane] = __ldg(o.step_pow + 2 * k + lane);
    } else if (warp == 1 && lane == 0) {
        so = o;
    }
    pdl_wait();
    __syncthreads();
    if (!trial_active<T>(sc)) return;
    const double t = warp_range_sum_deep(warp == 0 ? g.part_primal : g.part_dual, begin, end, warp == 0 ? 1 : 2,
                                         warp == 2 ? 1 : 0);
    if (lane == 0) sums[warp] = t;
    __syncthreads();
    if (warp != 0) return;
    if (lane == 0) trial_control(sc, so, sums[0], sums[1], sums[2], n, have ? factors : nullptr);
    __syncwarp();
    copy_ctl_warp(c, &sc);
}

// Fused trials of small LPs (k_fused).
#include "fused.cuh"

// ---------------------------------------------------------------------------
// Check, elementwise part (termination.cpp rowPass/columnPass terms without a
// product, infeasibility.cpp normalisation and cone projections,
// pdlp_solver.cpp:373-389 and :455-459)
// ---------------------------------------------------------------------------
template <class T>
__global__ void __launch_bounds__(kThreads) k_check_prep(Global g, Work<T> w, DeviceOptions o) {
    const VecWork vw = g.vec[blockIdx.x];
    const InstanceCtl& c = g.ctl[vw.instance];
    if (c.stage != kStageCheck || c.check_kind == kCheckTransition || !precision_matches<T>(c)) return;
    const InstanceInfo inf = g.info[vw.instance];
    const int p = c.parity;
    const bool pending = c.pending_avg != 0;
    const T frac = static_cast<T>(c.avg_frac);
    const bool have_avg = check_have_avg(c, o);
    const bool rays =
        (c.check_kind == kCheckMain || c.check_kind == kCheckEvaluate) && o.detect_infeasibility;

    double acc[kPrepSlots];
#pragma unroll
    for (int q = 0; q < kPrepSlots; ++q) acc[q] = 0.0;

    if (!vw.is_row) {
        const int64_t off = inf.col_off;
        for (int j = vw.begin + threadIdx.x; j < vw.end; j += blockDim.x) {
            const int64_t k = off + j;
            const T x = w.X[p][k];
            T a = w.avg_x[k];
            if (pending) {
                a = a + frac * (x - a);
                w.avg_x[k] = a;
            }
            const double cs = g.cs[k];
            const double xo = cs * static_cast<double>(x);
            g.x_o[k] = xo;
            const double co = g.c_orig[k];
            acc[0] += co * xo;
            if (have_avg) {
                const double xao = cs * static_cast<double>(a);
                g.xa_o[k] = xao;
                acc[1] += co * xao;
            }
            if (rays) {
                const double d = cs * (static_cast<double>(x) - static_cast<double>(w.rx[k]));
                acc[2] += d * d;
                double q = d;
                if (isfinite(g.xu_orig[k])) q = smin(q, 0.0);
                if (isfinite(g.xl_orig[k])) q = smax(q, 0.0);
                const double drift = d - q;
                acc[3] += drift * drift;
                acc[4] += co * q;
                g.p_proj[k] = q;
            }
            if (c.check_kind == kCheckMain) {
                const double r = static_cast<double>(w.rx[k]);
                const double dc = static_cast<double>(x) - r;
                acc[5] += dc * dc;
                const double da = static_cast<double>(a) - r;
                acc[6] += da * da;
            }
        }
    } else {
        const int64_t off = inf.row_off;
        for (int i = vw.begin + threadIdx.x; i < vw.end; i += blockDim.x) {
            const int64_t k = off + i;
            const T y = w.Y[p][k];
            T a = w.avg_y[k];
            if (pending) {
                a = a + frac * (y - a);
                w.avg_y[k] = a;
            }
            const double rs = g.rs[k];
            const double lo = g.rl_orig[k], hi = g.ru_orig[k];
            const bool lo_f = isfinite(lo), hi_f = isfinite(hi);
            const double yo = rs * static_cast<double>(y);
            g.y_o[k] = yo;
            {
                double q = yo;
                if (!hi_f) q = smin(q, 0.0);
                if (!lo_f) q = smax(q, 0.0);
                const double drift = yo - q;
                acc[1] += drift * drift;
                if (q > 0.0) acc[0] += q * hi;
                else if (q < 0.0) acc[0] += q * lo;
            }
            if (have_avg) {
                const double yao = rs * static_cast<double>(a);
                g.ya_o[k] = yao;
                double q = yao;
                if (!hi_f) q = smin(q, 0.0);
                if (!lo_f) q = smax(q, 0.0);
                const double drift = yao - q;
                acc[3] += drift * drift;
                if (q > 0.0) acc[2] += q * hi;
                else if (q < 0.0) acc[2] += q * lo;
            }
            if (rays) {
                const double d = rs * (static_cast<double>(y) - static_cast<double>(w.ry[k]));
                g.dy_o[k] = d;
                acc[4] += d * d;
                double q = d;
                if (!hi_f) q = smin(q, 0.0);
                if (!lo_f) q = smax(q, 0.0);
                const double drift = d - q;
                acc[5] += drift * drift;
                if (q > 0.0) acc[6] += q * hi;
                else if (q < 0.0) acc[6] += q * lo;
            }
            if (c.check_kind == kCheckMain) {
                const double r = static_cast<double>(w.ry[k]);
                const double dc = static_cast<double>(y) - r;
                acc[7] += dc * dc;
                const double da = static_cast<double>(a) - r;
                acc[8] += da * da;
            }
        }
    }
    block_sum<kPrepSlots>(acc);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < kPrepSlots; ++q)
            g.part_prep[static_cast<int64_t>(blockIdx.x) * kPrepSlots + q] = acc[q];
    }
}

// ---------------------------------------------------------------------------
// Check, matrix passes and decision
// ---------------------------------------------------------------------------
// The decision of one check from its sums (pdlp_solver.cpp:239-476,
// feasibility_polishing.cpp:107-141). C/R: column- and row-side elementwise
// sums (kPrepSlots each), A3: row-pass sums, T6: column-pass sums.
// `ndg`: with normalised-gap restarts at a main check, the gaps of the
// current and average iterates (else null).
__device__ __noinline__ void check_decide(const DeviceOptions& o, InstanceCtl& c, int32_t n_cols,
                                          const double* C, const double* R, const double* A3,
                                          const double* T6, const double* ndg) {

    c.pending_avg = 0;
    const bool have_avg = check_have_avg(c, o);
    const Metrics cur = make_metrics(c, A3[0], R[0], R[1], C[0], T6[1], T6[0]);
    const Metrics avg = have_avg ? make_metrics(c, A3[1], R[2], R[3], C[1], T6[3], T6[2]) : cur;

    if (c.check_kind == kCheckEvaluate) {
        store_best(c, cur);
        for (int q = 3; q < 12; ++q) c.dbg[q] = 0.0;
        const double dn = sqrt(R[4]);
        if (o.detect_infeasibility && dn > 1e-300 && isfinite(dn)) {
            const double inv = 1.0 / dn;
            const double value = (T6[5] - R[6]) * inv;
            c.dbg[4] = value;
            c.dbg[5] = 1.0;
            if (isfinite(value) && value > 0.0) {
                c.dbg[5] = sqrt(T6[4] + R[5]) * inv / value;
                c.dbg[3] = c.dbg[5] <= o.infeasibility_tol ? 1.0 : 0.0;
            }
        }
        const double pn = sqrt(C[2]);
        if (o.detect_infeasibility && pn > 1e-300 && isfinite(pn)) {
            const double inv = 1.0 / pn;
            const double rate = C[4] * inv;
            c.dbg[7] = rate;
            c.dbg[8] = 1.0;
            if (isfinite(rate) && rate < 0.0) {
                c.dbg[8] = sqrt(C[3] + A3[2]) * inv / (-rate);
                c.dbg[6] = c.dbg[8] <= o.infeasibility_tol ? 1.0 : 0.0;
            }
        }
        c.stage = kStageTrial;
        c.phase = kPhaseDone;
        return;
    }

    if (c.check_kind == kCheckInitial) {
        // pdlp_solver.cpp:239-264 (a warm start competes with the cold point,
        // which sits in the average buffers).
        c.restart_src = 1;
        Metrics start = cur;
        c.best_src = 1;
        if (have_avg && avg.kkt < cur.kkt) {
            start = avg;
            c.best_src = 2;
            c.restart_src = 2;
            c.need_refresh = 1;
        }
        store_best(c, start);
        // A normalised gap needs a radius, which the starting point does not
        // have yet: only the artificial test can trigger the first restart.
        c.restart_baseline = o.ndg_restarts ? INFINITY : start.kkt;
        c.avg_weight = 0.0;
        c.have_avg_at_check = 0;
        if (is_optimal_best(c, o)) {
            finish(c, 0, kMsgInitialOptimal, false);
            return;
        }
        loop_top_main(c, o, n_cols);
        return;
    }

    if (c.check_kind == kCheckPolish) {   // feasibility_polishing.cpp:107-141
        if (c.polish_deadline_ns > 0 && now_ns() >= c.polish_deadline_ns) {
            end_polish(c, o);
            return;
        }
        if (cur.kkt < c.best_kkt) {
            c.best_src = 1;
            store_best(c, cur);
        }
        if (have_avg && avg.kkt < c.best_kkt) {
            c.best_src = 2;
            store_best(c, avg);
        }
        if (is_optimal_best(c, o) || c.polish_done_iterations == o.polishing_iterations) {
            end_polish(c, o);
            return;
        }
        c.stage = kStageTrial;
        return;
    }

    // Main check (pdlp_solver.cpp:354-476).
    if (cur.kkt < c.best_kkt) {
        c.best_src = 1;
        store_best(c, cur);
    }
    if (have_avg && avg.kkt < c.best_kkt) {
        c.best_src = 2;
        store_best(c, avg);
    }
    if (o.detect_infeasibility) {
        // Dual ray: value = inf_box (A'd)'x - support(d), both linear in d, so
        // the sums over the raw direction are scaled by 1/||d|| afterwards.
        const double dn = sqrt(R[4]);
        if (dn > 1e-300 && isfinite(dn)) {
            const double inv = 1.0 / dn;
            const double value = (T6[5] - R[6]) * inv;
            if (isfinite(value) && value > 0.0) {
                const double viol = sqrt(T6[4] + R[5]) * inv;
                if (viol / value <= o.infeasibility_tol) {
                    finish(c, 1, kMsgInfeasible, true);
                    c.save_ray = 1;
                    c.ray_kind = 1;
                    return;
                }
            }
        }
        const double pn = sqrt(C[2]);
        if (pn > 1e-300 && isfinite(pn)) {
            const double inv = 1.0 / pn;
            const double rate = C[4] * inv;
            if (isfinite(rate) && rate < 0.0) {
                const double viol = sqrt(C[3] + A3[2]) * inv;
                if (viol / (-rate) <= o.infeasibility_tol) {
                    finish(c, 2, kMsgUnbounded, true);
                    c.save_ray = 2;
                    c.ray_kind = 2;
                    return;
                }
            }
        }
    }
    if (is_optimal_best(c, o)) {
        finish(c, 0, kMsgOptimal, true);
        return;
    }
    double score;
    const int choice = ndg ? restart_choose(c, o, ndg[0], ndg[1], &score)
                           : restart_choose(c, o, cur.kkt, avg.kkt, &score);
    if (choice != 0) {
        const bool from_avg = choice == 2 && have_avg;
        update_weight(c.omega, o, sqrt(from_avg ? C[6] : C[5]), sqrt(from_avg ? R[8] : R[7]));
        c.trial_omega = c.omega;
        c.restart_src = from_avg ? 2 : 1;
        if (from_avg) c.need_refresh = 1;
        c.restart_baseline = score;
        c.avg_weight = 0.0;
        c.prev_candidate = INFINITY;
        c.since_restart = 0;
        ++c.restart_count;
    }
    if (o.mixed && !c.fp64_stage) {
        // Mixed precision: FP32 iterations go on while the best KKT score
        // keeps falling or is still far (above fp32_switch_kkt) from the
        // tolerance; after fp32_stall_checks checks without a 10% drop the
        // instance continues in FP64 from its last FP32 restart point (the
        // restart point this check may just have set), with a fresh average.
        if (!(c.best_kkt_at_stall > 0.0) || c.best_kkt < 0.9 * c.best_kkt_at_stall ||
            !(c.best_kkt <= o.fp32_switch_kkt)) {
            c.best_kkt_at_stall = c.best_kkt;
            c.stall_checks = 0;
        } else if (++c.stall_checks >= o.fp32_stall_checks) {
            c.to_fp64 = 1;
            c.need_refresh = 1;
            c.avg_weight = 0.0;
            c.since_restart = 0;
            c.prev_candidate = INFINITY;
            c.stall_checks = 0;
        }
    }
    loop_top_main(c, o, n_cols);
}

__device__ __noinline__ void check_control(const Global& g, const DeviceOptions& o, InstanceCtl& c,
                              const InstanceInfo& inf, const double* ndg) {
    // Column-side and row-side elementwise partials.
    double C[kPrepSlots], R[kPrepSlots], A3[3], T6[kCheckSlots];
    for (int q = 0; q < kPrepSlots; ++q) { C[q] = 0.0; R[q] = 0.0; }
    const int lane = threadIdx.x & 31;
    for (int q = 0; q < kPrepSlots; ++q) {
        double tc = 0.0, tr = 0.0;
        for (int k = inf.vec_cta_begin + lane; k < inf.vec_cta_end; k += 32) {
            const double v = g.part_prep[static_cast<int64_t>(k) * kPrepSlots + q];
            if (g.vec[k].is_row) tr += v; else tc += v;
        }
        for (int s = 16; s > 0; s >>= 1) {
            tc += __shfl_xor_sync(kFull, tc, s);
            tr += __shfl_xor_sync(kFull, tr, s);
        }
        C[q] = tc;
        R[q] = tr;
    }
    for (int q = 0; q < 3; ++q)
        A3[q] = warp_range_sum(g.part_check, inf.a_cta_begin, inf.a_cta_end, kCheckSlots, q);
    const int at0 = g.a.num_ctas + inf.at_cta_begin, at1 = g.a.num_ctas + inf.at_cta_end;
    for (int q = 0; q < kCheckSlots; ++q) T6[q] = warp_range_sum(g.part_check, at0, at1, kCheckSlots, q);
    if (lane != 0) return;
    check_decide(o, c, inf.n, C, R, A3, T6, ndg);
}

// The candidate coordinates of a main check in the scaled space of the
// iterations (x = x_o / cs, y = y_o / rs, c + A'y scaled by cs, A x by rs,
// bounds scaled like the iterates), from what the check stored in original
// coordinates; the restart point comes from the working arrays.
struct CheckNdgCoord {
    const Global* g;
    int64_t col0, row0, n;
    int which;    // 0 current, 1 average
    bool fp32;    // restart point in the FP32 working arrays
    __device__ NdgCoord operator()(int64_t k) const {
        NdgCoord q;
        if (k < n) {
            const int64_t j = col0 + k;
            const double cs = g->cs[j], ics = 1.0 / cs;
            q.v = (which ? g->xa_o[j] : g->x_o[j]) * ics;
            q.d = cs * g->ndg_g[which][j];
            q.lo = g->xl_orig[j] * ics;
            q.hi = g->xu_orig[j] * ics;
            q.r = fp32 ? static_cast<double>(g->rx32[j]) : g->rx64[j];
        } else {
            const int64_t i = row0 + (k - n);
            const double rs = g->rs[i];
            q.v = (which ? g->ya_o[i] : g->y_o[i]) * (1.0 / rs);
            q.d = rs * g->ndg_a[which][i];
            q.lo = g->rl_orig[i] * rs;
            q.hi = g->ru_orig[i] * rs;
            q.r = fp32 ? static_cast<double>(g->ry32[i]) : g->ry64[i];
        }
        return q;
    }
};

// Normalised gaps of the current and the average iterate (the same value
// twice without an average), computed by the whole CTA; out[0..1] in shared
// memory, valid after the CTA's next barrier.
__device__ __noinline__ void check_ndg(const Global& g, const DeviceOptions& o, const InstanceCtl& c,
                                       const InstanceInfo& inf, double* out) {
    __shared__ double scratch[16 * 32];
    const bool fp32 = o.mixed && !c.fp64_stage;
    CheckNdgCoord q{&g, inf.col_off, inf.row_off, inf.n, 0, fp32};
    const double cur = block_normalized_gap(inf.n, inf.m, c.omega, q, scratch, nullptr);
    double avg = cur;
    if (check_have_avg(c, o)) {
        q.which = 1;
        avg = block_normalized_gap(inf.n, inf.m, c.omega, q, scratch, nullptr);
    }
    if (threadIdx.x == 0) {
        out[0] = cur;
        out[1] = avg;
    }
}

template <int V>
__global__ void __launch_bounds__(kThreads) k_check_spmv(Global g, DeviceOptions o) {
    const bool a_side = blockIdx.x < static_cast<unsigned>(g.a.num_ctas);
    const int cta = a_side ? blockIdx.x : blockIdx.x - g.a.num_ctas;
    const CtaWork cw = (a_side ? g.a.ctas : g.at.ctas)[cta];
    InstanceCtl& c = g.ctl[cw.instance];
    if (c.stage != kStageCheck || c.check_kind == kCheckTransition) return;
    const InstanceInfo inf = g.info[cw.instance];
    const bool have_avg = check_have_avg(c, o);
    const bool rays =
        (c.check_kind == kCheckMain || c.check_kind == kCheckEvaluate) && o.detect_infeasibility;
    const bool ndg = o.ndg_restarts && o.restarts && c.check_kind == kCheckMain;

    double acc[kCheckSlots];
#pragma unroll
    for (int q = 0; q < kCheckSlots; ++q) acc[q] = 0.0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (a_side) {   // rowPass (termination.cpp:66-135) for current/average, A*d for the primal ray
        const double* xo = g.x_o + inf.col_off;
        const double* xa = g.xa_o + inf.col_off;
        const double* pp = g.p_proj + inf.col_off;
        for (int s = cw.slice_begin + warp; s < cw.slice_end; s += kWarps) {
            const SliceDesc sd = g.a.slices[s];
            const LanePos lp = lane_pos(sd, lane);
            const int len = lp.valid ? g.a.line_len[inf.a_len_base + lp.line] : 0;
            double sum[3] = {0.0, 0.0, 0.0};
            line_sums<V, 3>(inf.a_data_base + static_cast<int64_t>(sd.data_off) * 32, sd.steps,
                            lp, lane, len, g.a.idx, g.a.val_orig, sum,
                            [&](double (&a)[3], double v, int j) {
                                a[0] += v * xo[j];
                                if (have_avg) a[1] += v * xa[j];
                                if (rays) a[2] += v * pp[j];
                            });
            if (lp.valid && lp.g == 0) {
                const int64_t k = inf.row_off + lp.line;
                if (ndg) {
                    g.ndg_a[0][k] = sum[0];
                    if (have_avg) g.ndg_a[1][k] = sum[1];
                }
                const double lo = g.rl_orig[k], hi = g.ru_orig[k];
                const double e0 = sum[0] - smax(lo, smin(sum[0], hi));
                acc[0] += e0 * e0;
                if (have_avg) {
                    const double e1 = sum[1] - smax(lo, smin(sum[1], hi));
                    acc[1] += e1 * e1;
                }
                if (rays) {
                    double q = sum[2];
                    if (isfinite(hi)) q = smin(q, 0.0);
                    if (isfinite(lo)) q = smax(q, 0.0);
                    const double drift = sum[2] - q;
                    acc[2] += drift * drift;
                }
            }
        }
    } else {        // columnPass (termination.cpp:140-209), A'd for the dual ray
        const double* yo = g.y_o + inf.row_off;
        const double* ya = g.ya_o + inf.row_off;
        const double* dy = g.dy_o + inf.row_off;
        for (int s = cw.slice_begin + warp; s < cw.slice_end; s += kWarps) {
            const SliceDesc sd = g.at.slices[s];
            const LanePos lp = lane_pos(sd, lane);
            const int len = lp.valid ? g.at.line_len[inf.at_len_base + lp.line] : 0;
            double sum[3] = {0.0, 0.0, 0.0};
            line_sums<V, 3>(inf.at_data_base + static_cast<int64_t>(sd.data_off) * 32, sd.steps,
                            lp, lane, len, g.at.idx, g.at.val_orig, sum,
                            [&](double (&a)[3], double v, int i) {
                                a[0] += v * yo[i];
                                if (have_avg) a[1] += v * ya[i];
                                if (rays) a[2] += v * dy[i];
                            });
            if (lp.valid && lp.g == 0) {
                const int64_t k = inf.col_off + lp.line;
                const double co = g.c_orig[k];
                const double lo = g.xl_orig[k], hi = g.xu_orig[k];
                const bool lo_f = isfinite(lo), hi_f = isfinite(hi);
                for (int which = 0; which < 2; ++which) {
                    if (which == 1 && !have_avg) break;
                    const double reduced = co + sum[which];
                    if (ndg) g.ndg_g[which][k] = reduced;
                    double q = reduced;
                    if (!lo_f) q = smin(q, 0.0);
                    if (!hi_f) q = smax(q, 0.0);
                    const double drift = reduced - q;
                    acc[2 * which] += drift * drift;
                    if (q > 0.0) acc[2 * which + 1] += q * lo;
                    else if (q < 0.0) acc[2 * which + 1] += q * hi;
                }
                if (rays) {
                    const double r = sum[2];
                    double q = r;
                    if (!lo_f) q = smin(q, 0.0);
                    if (!hi_f) q = smax(q, 0.0);
                    const double drift = r - q;
                    acc[4] += drift * drift;
                    if (q > 0.0) acc[5] += q * lo;
                    else if (q < 0.0) acc[5] += q * hi;
                }
            }
        }
    }
    block_sum<kCheckSlots>(acc);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < kCheckSlots; ++q)
            g.part_check[static_cast<int64_t>(blockIdx.x) * kCheckSlots + q] = acc[q];
    }
    const int expected = (inf.a_cta_end - inf.a_cta_begin) + (inf.at_cta_end - inf.at_cta_begin);
    if (!arrive_last(g.count_check + cw.instance, expected)) return;
    // With normalised-gap restarts, k_check_ndg takes the decision.
    if (o.ndg_restarts) return;
    __shared__ DeviceOptions so;   // see k_decide
    if (threadIdx.x == 0) so = o;
    __syncthreads();
    if (threadIdx.x < 32) check_control(g, so, c, inf, nullptr);
}

// The check decision with normalised-gap restarts: one CTA per instance,
// after k_check_spmv. At a main check the CTA first computes the two
// candidates' normalised gaps from the products k_check_spmv stored.
__global__ void __launch_bounds__(kThreads) k_check_ndg(Global g, DeviceOptions o) {
    const int b = blockIdx.x;
    InstanceCtl& c = g.ctl[b];
    if (c.stage != kStageCheck || c.check_kind == kCheckTransition) return;
    const InstanceInfo inf = g.info[b];
    __shared__ DeviceOptions so;   // see k_decide
    __shared__ double gaps[2];
    if (threadIdx.x == 0) so = o;
    __syncthreads();
    const bool main = o.restarts && c.check_kind == kCheckMain;
    if (main) check_ndg(g, so, c, inf, gaps);
    __syncthreads();
    if (threadIdx.x < 32) check_control(g, so, c, inf, main ? gaps : nullptr);
}

// ---------------------------------------------------------------------------
// Check, application of the decisions
// ---------------------------------------------------------------------------
template <class T>
__global__ void __launch_bounds__(kThreads) k_check_apply(Global g, Work<T> w) {
    const VecWork vw = g.vec[blockIdx.x];
    const InstanceCtl& c = g.ctl[vw.instance];
    if (!(c.best_src || c.restart_src || c.to_polish || c.save_ray)) return;
    if (!precision_matches<T>(c)) return;
    const InstanceInfo inf = g.info[vw.instance];
    const int p = c.parity;
    if (!vw.is_row) {
        for (int j = vw.begin + threadIdx.x; j < vw.end; j += blockDim.x) {
            const int64_t k = inf.col_off + j;
            if (c.best_src == 1) g.best_x[k] = g.x_o[k];
            else if (c.best_src == 2) g.best_x[k] = g.xa_o[k];
            if (c.save_ray == 2)
                g.pray[k] = g.cs[k] * (static_cast<double>(w.X[p][k]) - static_cast<double>(w.rx[k]));
            if (c.restart_src) {
                if (c.restart_src == 2) w.X[p][k] = w.avg_x[k];
                w.rx[k] = w.X[p][k];
            }
            if (c.to_polish) {   // toScaled (scaling.cpp:39-53)
                w.X[p][k] = static_cast<T>(g.best_x[k] / g.cs[k]);
            }
        }
    } else {
        for (int i = vw.begin + threadIdx.x; i < vw.end; i += blockDim.x) {
            const int64_t k = inf.row_off + i;
            if (c.best_src == 1) g.best_y[k] = g.y_o[k];
            else if (c.best_src == 2) g.best_y[k] = g.ya_o[k];
            if (c.save_ray == 1) g.dray[k] = g.dy_o[k];
            if (c.restart_src) {
                if (c.restart_src == 2) w.Y[p][k] = w.avg_y[k];
                w.ry[k] = w.Y[p][k];
            }
            if (c.to_polish) {
                w.Y[p][k] = static_cast<T>(g.best_y[k] / g.rs[k]);
            }
        }
    }
}

// A x for the current iterate of instances whose iterate was replaced
// (CpuPdhgKernel::refreshActivity, pdhg_kernel.cpp:40-42).
template <class T, int V>
__global__ void __launch_bounds__(kThreads) k_refresh(Global g, Work<T> w) {
    const CtaWork cw = g.a.ctas[blockIdx.x];
    const InstanceCtl& c = g.ctl[cw.instance];
    // An instance moving to the FP64 stage gets its FP64 product here.
    if (!c.need_refresh || !(precision_matches<T>(c) || (sizeof(T) == 8 && c.to_fp64))) return;
    const InstanceInfo inf = g.info[cw.instance];
    const int p = c.parity;
    const T* __restrict__ x = w.X[p] + inf.col_off;
    T* __restrict__ ax = w.AX[p] + inf.row_off;
    const T* vals = matrix_values<T>(g.a);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int s = cw.slice_begin + warp; s < cw.slice_end; s += kWarps) {
        const SliceDesc sd = g.a.slices[s];
        const LanePos lp = lane_pos(sd, lane);
        const int len = lp.valid ? g.a.line_len[inf.a_len_base + lp.line] : 0;
        T sum[1] = {T(0)};
        line_sums<V, 1>(inf.a_data_base + static_cast<int64_t>(sd.data_off) * 32, sd.steps, lp,
                        lane, len, g.a.idx, vals, sum,
                        [&](T (&a)[1], T v, int j) { a[0] += v * x[j]; });
        if (lp.valid && lp.g == 0) ax[lp.line] = sum[0];
    }
}

// Clears the per-check flags, completes a move to the FP64 stage, and counts
// the unfinished instances (active[0]) and those among them in the FP64
// stage of a mixed solve (active[1]).
__global__ void k_finalize(Global g, int32_t count, int32_t* active) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= count) return;
    InstanceCtl& c = g.ctl[b];
    if (c.to_fp64) {
        c.fp64_stage = 1;
        c.to_fp64 = 0;
    }
    if (c.phase != kPhaseDone && active != nullptr) {
        atomicAdd(active, 1);
        if (c.fp64_stage && g.mixed) atomicAdd(active + 1, 1);
    }
    if (c.stage == kStageCheck && c.check_kind == kCheckTransition) c.stage = kStageTrial;
    c.best_src = 0;
    c.restart_src = 0;
    c.need_refresh = 0;
    c.to_polish = 0;
    c.save_ray = 0;
    c.il_sync = 0;
}

// Mixed precision: the FP64 stage starts from the last FP32 restart point.
__global__ void k_switch_fp64(Global g, Work<float> w32, Work<double> w64) {
    const VecWork vw = g.vec[blockIdx.x];
    const InstanceCtl& c = g.ctl[vw.instance];
    if (!c.to_fp64) return;
    const InstanceInfo inf = g.info[vw.instance];
    const int p = c.parity;
    if (!vw.is_row) {
        for (int j = vw.begin + threadIdx.x; j < vw.end; j += blockDim.x) {
            const int64_t k = inf.col_off + j;
            const double v = static_cast<double>(w32.rx[k]);
            w64.X[p][k] = v;
            w64.rx[k] = v;
        }
    } else {
        for (int i = vw.begin + threadIdx.x; i < vw.end; i += blockDim.x) {
            const int64_t k = inf.row_off + i;
            const double v = static_cast<double>(w32.ry[k]);
            w64.Y[p][k] = v;
            w64.ry[k] = v;
        }
    }
}

// ---------------------------------------------------------------------------
// Setup: Ruiz equilibration (scaling.cpp:55-107). Row maxima over the A side
// and column maxima over the A^T side read the same scale state, as the
// reference's single sweep does; max is exact, so the scale vectors equal the
// reference's bit for bit.
// ---------------------------------------------------------------------------
template <int V>
__global__ void __launch_bounds__(kThreads) k_ruiz_max(Global g, int a_ctas) {
    const bool a_side = blockIdx.x < static_cast<unsigned>(a_ctas);
    const Side side = a_side ? g.a : g.at;
    const CtaWork cw = side.ctas[a_side ? blockIdx.x : blockIdx.x - a_ctas];
    const InstanceInfo inf = g.info[cw.instance];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const double* line_scale = a_side ? g.rs + inf.row_off : g.cs + inf.col_off;
    const double* other = a_side ? g.cs + inf.col_off : g.rs + inf.row_off;
    double* out = a_side ? g.row_tmp + inf.row_off : g.col_tmp + inf.col_off;
    const int64_t dbase = a_side ? inf.a_data_base : inf.at_data_base;
    const int64_t lbase = a_side ? inf.a_len_base : inf.at_len_base;
    for (int s = cw.slice_begin + warp; s < cw.slice_end; s += kWarps) {
        const SliceDesc sd = side.slices[s];
        const LanePos lp = lane_pos(sd, lane);
        const int len = lp.valid ? side.line_len[lbase + lp.line] : 0;
        const double f = lp.valid ? line_scale[lp.line] : 0.0;
        double mx = 0.0;
        const int64_t base = dbase + static_cast<int64_t>(sd.data_off) * 32;
        for (int st = 0; st < sd.steps; st += V) {
            const int64_t pidx = base + static_cast<int64_t>(st) * 32 + lane * V;
            int32_t id[V];
            double v[V];
            ld<V>(side.idx + pidx, id);
            ld<V>(side.val_orig + pidx, v);
#pragma unroll
            for (int q = 0; q < V; ++q) {
                const int k = ((st + q) << lp.glog) + lp.g;
                if (k < len) {
                    // |a_ij| * r_i * c_j, multiplied in the reference's order
                    const double m = a_side ? fabs(v[q]) * f * other[id[q]]
                                            : fabs(v[q]) * other[id[q]] * f;
                    mx = smax(mx, m);
                }
            }
        }
        for (int o = (1 << lp.glog) >> 1; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(kFull, mx, o));
        if (lp.valid && lp.g == 0) out[lp.line] = mx;
    }
}

__global__ void k_ruiz_update(Global g) {
    const VecWork vw = g.vec[blockIdx.x];
    const InstanceInfo inf = g.info[vw.instance];
    double* scale = vw.is_row ? g.rs + inf.row_off : g.cs + inf.col_off;
    const double* mx = vw.is_row ? g.row_tmp + inf.row_off : g.col_tmp + inf.col_off;
    for (int k = vw.begin + threadIdx.x; k < vw.end; k += blockDim.x) {
        const double m = mx[k];
        if (m > 1e-30) scale[k] /= sqrt(m);
    }
}

// Scaled coefficients (SparseMatrix::scaled, sparse_matrix.cpp:243-274).
template <int V>
__global__ void __launch_bounds__(kThreads) k_scale_values(Global g, double* a_s64, double* at_s64,
                                                        float* a_s32, float* at_s32, int a_ctas) {
    const bool a_side = blockIdx.x < static_cast<unsigned>(a_ctas);
    const Side side = a_side ? g.a : g.at;
    const CtaWork cw = side.ctas[a_side ? blockIdx.x : blockIdx.x - a_ctas];
    const InstanceInfo inf = g.info[cw.instance];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const double* line_scale = a_side ? g.rs + inf.row_off : g.cs + inf.col_off;
    const double* other = a_side ? g.cs + inf.col_off : g.rs + inf.row_off;
    double* out64 = a_side ? a_s64 : at_s64;
    float* out32 = a_side ? a_s32 : at_s32;
    const int64_t dbase = a_side ? inf.a_data_base : inf.at_data_base;
    const int64_t lbase = a_side ? inf.a_len_base : inf.at_len_base;
    for (int s = cw.slice_begin + warp; s < cw.slice_end; s += kWarps) {
        const SliceDesc sd = side.slices[s];
        const LanePos lp = lane_pos(sd, lane);
        const int len = lp.valid ? side.line_len[lbase + lp.line] : 0;
        const double f = lp.valid ? line_scale[lp.line] : 0.0;
        const int64_t base = dbase + static_cast<int64_t>(sd.data_off) * 32;
        for (int st = 0; st < sd.steps; ++st) {
            const int64_t pidx = base + static_cast<int64_t>(st - st % V) * 32 + lane * V + st % V;
            const int k = (st << lp.glog) + lp.g;
            double r = 0.0;
            if (k < len) r = side.val_orig[pidx] * (f * other[side.idx[pidx]]);
            out64[pidx] = r;
            if (out32) out32[pidx] = static_cast<float>(r);
        }
    }
}

// Pock-Chambolle (preconditioner.cpp:31-80): row and column L1 sums of the
// scaled matrix, each over its own side.
template <class T, int V>
__global__ void __launch_bounds__(kThreads) k_precondition(Global g, Work<T> w, int a_ctas) {
    const bool a_side = blockIdx.x < static_cast<unsigned>(a_ctas);
    const Side side = a_side ? g.a : g.at;
    const CtaWork cw = side.ctas[a_side ? blockIdx.x : blockIdx.x - a_ctas];
    const InstanceInfo inf = g.info[cw.instance];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t dbase = a_side ? inf.a_data_base : inf.at_data_base;
    const int64_t lbase = a_side ? inf.a_len_base : inf.at_len_base;
    T* sc = a_side ? w.sigma + inf.row_off : w.tau + inf.col_off;
    T* isc = a_side ? w.isigma + inf.row_off : w.itau + inf.col_off;
    for (int s = cw.slice_begin + warp; s < cw.slice_end; s += kWarps) {
        const SliceDesc sd = side.slices[s];
        const LanePos lp = lane_pos(sd, lane);
        const int len = lp.valid ? side.line_len[lbase + lp.line] : 0;
        double sum[1] = {0.0};
        line_sums<V, 1>(dbase + static_cast<int64_t>(sd.data_off) * 32, sd.steps, lp, lane, len,
                        side.idx, side.val_s64, sum,
                        [&](double (&a)[1], double v, int) { a[0] += fabs(v); });
        if (lp.valid && lp.g == 0) {
            const double scale = sum[0] > 1e-12 ? 1.0 / sum[0] : 1.0;
            sc[lp.line] = static_cast<T>(scale);
            isc[lp.line] = static_cast<T>(1.0 / scale);
        }
    }
}

__device__ __forceinline__ double scale_bound(double b, double f) { return isfinite(b) ? b * f : b; }

__device__ __forceinline__ double initial_value(double lo, double hi) {   // pdlp_solver.cpp:30-41
    if (lo <= 0.0 && 0.0 <= hi) return 0.0;
    if (isfinite(lo)) return lo;
    if (isfinite(hi)) return hi;
    return 0.0;
}

__global__ void k_warp_heads(Global g) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const bool a_side = k < g.a.num_ctas * kWarps;
    const int i = a_side ? k : k - g.a.num_ctas * kWarps;
    const Side& side = a_side ? g.a : g.at;
    if (i >= side.num_ctas * kWarps) return;
    const CtaWork cw = side.ctas[i / kWarps];
    const InstanceInfo inf = g.info[cw.instance];
    const int s = cw.slice_begin + i % kWarps;
    const bool some = s < cw.slice_end;
    SliceDesc sd{};
    if (some) sd = side.slices[s];
    WarpHead h{};
    h.base = static_cast<int32_t>((a_side ? inf.a_data_base : inf.at_data_base) / 32) + sd.data_off;
    h.line = static_cast<int32_t>(a_side ? inf.row_off : inf.col_off) + sd.line0;
    h.len = static_cast<int32_t>(a_side ? inf.a_len_base : inf.at_len_base) + sd.line0;
    h.other = static_cast<int32_t>(a_side ? inf.col_off : inf.row_off);
    h.instance = cw.instance;
    h.steps = sd.steps;
    h.meta = sd.meta;
    h.slice = some ? s : cw.slice_end;
    h.slice_end = cw.slice_end;
    h.many = cw.slice_end - cw.slice_begin > kWarps;
    side.heads[i] = h;
}

// Scaled objective and bounds (scaling.cpp:109-135), the starting point
// (pdlp_solver.cpp:168-176) or a warm start, and its cold alternative.
template <class T>
__global__ void k_setup_vectors(Global g, Work<T> w) {
    const VecWork vw = g.vec[blockIdx.x];
    if (g.slot_mask != nullptr && g.slot_mask[vw.instance] == 0) return;
    const InstanceInfo inf = g.info[vw.instance];
    const bool warm = g.warm_x != nullptr || g.warm_y != nullptr;
    if (!vw.is_row) {
        for (int j = vw.begin + threadIdx.x; j < vw.end; j += blockDim.x) {
            const int64_t k = inf.col_off + j;
            const double f = g.cs[k];
            const double lo = scale_bound(g.xl_orig[k], 1.0 / f);
            const double hi = scale_bound(g.xu_orig[k], 1.0 / f);
            w.c[k] = static_cast<T>(g.c_orig[k] * f);
            w.xl[k] = static_cast<T>(lo);
            w.xu[k] = static_cast<T>(hi);
            const double cold = initial_value(lo, hi);
            double x0 = cold;
            if (g.warm_x != nullptr) {
                const double v = g.warm_x[k] / f;
                x0 = isfinite(v) ? smax(lo, smin(v, hi)) : cold;
            }
            w.X[0][k] = static_cast<T>(x0);
            w.X[1][k] = static_cast<T>(x0);
            w.rx[k] = static_cast<T>(x0);
            w.avg_x[k] = static_cast<T>(warm ? cold : 0.0);
        }
    } else {
        for (int i = vw.begin + threadIdx.x; i < vw.end; i += blockDim.x) {
            const int64_t k = inf.row_off + i;
            const double f = g.rs[k];
            w.rl[k] = static_cast<T>(scale_bound(g.rl_orig[k], f));
            w.ru[k] = static_cast<T>(scale_bound(g.ru_orig[k], f));
            double y0 = 0.0;
            if (g.warm_y != nullptr) {
                const double v = g.warm_y[k] / f;
                y0 = isfinite(v) ? v : 0.0;
            }
            w.Y[0][k] = static_cast<T>(y0);
            w.Y[1][k] = static_cast<T>(y0);
            w.ry[k] = static_cast<T>(y0);
            w.avg_y[k] = static_cast<T>(0.0);
            w.AX[0][k] = T(0);
            w.AX[1][k] = T(0);
        }
    }
}

// Shared-matrix batches: scales and preconditioner depend on A only, so the
// vectors of instance 0 are copied to every other instance.
__global__ void k_broadcast_scales(double* rs, double* cs, int64_t rows, int64_t cols, int32_t count) {
    const int64_t total = (rows + cols) * (count - 1);
    for (int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; t < total;
         t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t b = 1 + t / (rows + cols), e = t % (rows + cols);
        if (e < rows) rs[b * rows + e] = rs[e];
        else cs[b * cols + (e - rows)] = cs[e - rows];
    }
}

template <class T>
__global__ void k_broadcast_precond(T* sigma, T* isigma, T* tau, T* itau, int64_t rows, int64_t cols,
                                    int32_t count) {
    const int64_t total = (rows + cols) * (count - 1);
    for (int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; t < total;
         t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t b = 1 + t / (rows + cols), e = t % (rows + cols);
        if (e < rows) {
            sigma[b * rows + e] = sigma[e];
            isigma[b * rows + e] = isigma[e];
        } else {
            tau[b * cols + (e - rows)] = tau[e - rows];
            itau[b * cols + (e - rows)] = itau[e - rows];
        }
    }
}

// Plain product over one side, lines in internal order.
template <class T, int V>
__global__ void __launch_bounds__(kThreads) k_spmv(Global g, int transpose, const T* vals,
                                                   const T* v, T* out) {
    const Side side = transpose ? g.at : g.a;
    const CtaWork cw = side.ctas[blockIdx.x];
    const InstanceInfo inf = g.info[cw.instance];
    const T* src = v + (transpose ? inf.row_off : inf.col_off);
    T* dst = out + (transpose ? inf.col_off : inf.row_off);
    const int64_t dbase = transpose ? inf.at_data_base : inf.a_data_base;
    const int64_t lbase = transpose ? inf.at_len_base : inf.a_len_base;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int s = cw.slice_begin + warp; s < cw.slice_end; s += kWarps) {
        const SliceDesc sd = side.slices[s];
        const LanePos lp = lane_pos(sd, lane);
        const int len = lp.valid ? side.line_len[lbase + lp.line] : 0;
        T sum[1] = {T(0)};
        line_sums<V, 1>(dbase + static_cast<int64_t>(sd.data_off) * 32, sd.steps, lp, lane, len,
                        side.idx, vals, sum, [&](T (&a)[1], T x, int j) { a[0] += x * src[j]; });
        if (lp.valid && lp.g == 0) dst[lp.line] = sum[0];
    }
}


// The linesearch's step factors by iteration index (DeviceOptions::step_pow).
__global__ void k_step_pow(double* table, int64_t entries) {
    for (int64_t k = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; k < entries;
         k += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const double index = static_cast<double>(k) + 2.0;
        table[2 * k] = pow(index, -0.3);
        table[2 * k + 1] = pow(index, -0.6);
    }
}

// ---------------------------------------------------------------------------
// Power iteration on A'A (preconditioner.cpp:82-140), used only when the
// diagonal preconditioner is off. Per-instance state lives in ctl.dbg:
// [4] estimate, [5] previous, [6] scale 1/||z||, [7] state (0 running,
// 1 converged, 2 stopped on a zero vector, 3 budget exhausted), [8] unit flag.
// ---------------------------------------------------------------------------
__global__ void k_power_dot(Global g, const double* x, const double* z) {
    const VecWork vw = g.vec[blockIdx.x];
    const InstanceInfo inf = g.info[vw.instance];
    double acc[2] = {0.0, 0.0};
    if (!vw.is_row && g.ctl[vw.instance].dbg[7] == 0.0) {
        for (int j = vw.begin + threadIdx.x; j < vw.end; j += blockDim.x) {
            const double a = x[inf.col_off + j], b = z[inf.col_off + j];
            acc[0] += a * b;
            acc[1] += b * b;
        }
    }
    block_sum<2>(acc);
    if (threadIdx.x == 0) {
        g.part_prep[static_cast<int64_t>(blockIdx.x) * kPrepSlots] = acc[0];
        g.part_prep[static_cast<int64_t>(blockIdx.x) * kPrepSlots + 1] = acc[1];
    }
}

__global__ void k_power_step(Global g, int32_t count, int init, int it, int budget) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= count) return;
    InstanceCtl& c = g.ctl[b];
    if (c.dbg[7] != 0.0) return;
    const InstanceInfo inf = g.info[b];
    double xz = 0.0, zz = 0.0;
    for (int k = inf.vec_cta_begin; k < inf.vec_cta_end; ++k) {
        if (g.vec[k].is_row) continue;
        xz += g.part_prep[static_cast<int64_t>(k) * kPrepSlots];
        zz += g.part_prep[static_cast<int64_t>(k) * kPrepSlots + 1];
    }
    const double norm = sqrt(zz);
    if (init) {
        c.dbg[8] = norm == 0.0 ? 1.0 : 0.0;
        c.dbg[6] = norm > 0.0 ? 1.0 / norm : 0.0;
        return;
    }
    const double est = sqrt(smax(xz, 0.0));
    c.dbg[4] = est;
    if (norm == 0.0) {
        c.dbg[7] = 2.0;
        return;
    }
    c.dbg[6] = 1.0 / norm;
    c.dbg[8] = 0.0;
    if (it > 0 && est > 0.0 && fabs(est - c.dbg[5]) <= 1e-8 * est) {
        c.dbg[7] = 1.0;
        return;
    }
    c.dbg[5] = est;
    if (it == budget - 1) c.dbg[7] = 3.0;
}

__global__ void k_power_scale(Global g, double* x, const double* z) {
    const VecWork vw = g.vec[blockIdx.x];
    if (vw.is_row) return;
    const InstanceCtl& c = g.ctl[vw.instance];
    if (c.dbg[7] != 0.0) return;
    const InstanceInfo inf = g.info[vw.instance];
    const double s = c.dbg[6];
    const bool unit = c.dbg[8] != 0.0;
    const double u = inf.n > 0 ? 1.0 / sqrt(static_cast<double>(inf.n)) : 0.0;
    for (int j = vw.begin + threadIdx.x; j < vw.end; j += blockDim.x)
        x[inf.col_off + j] = unit ? u : z[inf.col_off + j] * s;
}

// pdlp_solver.cpp:188-202 and the StepController constructor (step_controller.cpp:17-28).
__global__ void k_power_finish(Global g, int32_t count, double safety, double min_scale) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= count) return;
    InstanceCtl& c = g.ctl[b];
    const double est = c.dbg[4];
    const bool converged = c.dbg[7] == 1.0 || c.dbg[7] == 2.0;
    const double safe = est > 0.0 ? 0.99 / (est * (converged ? 1.02 : 1.25)) : 1.0;
    c.eta_max = safe;
    c.eta = clampd(safety * safe, min_scale * safe, safe);
    c.trial_eta = c.eta;
    for (int q = 3; q < 12; ++q) c.dbg[q] = 0.0;
}

// The solve clock: the reference's clock starts when solve() is entered, so
// the host's setup time is carried in.
__global__ void k_stamp_clock(Global g, int32_t count, int64_t elapsed_ns, int64_t limit_ns) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= count) return;
    if (g.slot_mask != nullptr && g.slot_mask[b] == 0) return;
    InstanceCtl& c = g.ctl[b];
    c.start_ns = now_ns() - elapsed_ns;
    c.deadline_ns = limit_ns > 0 ? c.start_ns + limit_ns : 0;
}


// ---------------------------------------------------------------------------
// Sessions: order changes between the caller's layout and the internal one,
// the TerminationChecker normalisers (termination.cpp:58-62) and the initial
// control state, all on the device.
// ---------------------------------------------------------------------------
__global__ void k_permute(const double* __restrict__ src, double* __restrict__ dst,
                          const int32_t* __restrict__ perm, int64_t len, int32_t count, int mode) {
    const int64_t total = len * count;
    for (int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; t < total;
         t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t b = t / len, k = t - b * len;
        if (mode == 0) dst[t] = src[b * len + perm[k]];
        else if (mode == 1) dst[b * len + perm[k]] = src[t];
        else dst[t] = src[k];
    }
}

__global__ void __launch_bounds__(kThreads) k_norm_parts(Global g) {
    const VecWork vw = g.vec[blockIdx.x];
    if (g.slot_mask != nullptr && g.slot_mask[vw.instance] == 0) return;
    const InstanceInfo inf = g.info[vw.instance];
    double acc[1] = {0.0};
    if (!vw.is_row) {
        for (int j = vw.begin + threadIdx.x; j < vw.end; j += blockDim.x) {
            const double v = g.c_orig[inf.col_off + j];
            acc[0] += v * v;
        }
    } else {
        for (int i = vw.begin + threadIdx.x; i < vw.end; i += blockDim.x) {
            const double l = g.rl_orig[inf.row_off + i], u = g.ru_orig[inf.row_off + i];
            if (isfinite(l)) acc[0] += l * l;
            if (isfinite(u) && u != l) acc[0] += u * u;
        }
    }
    block_sum<1>(acc);
    if (threadIdx.x == 0) g.part_prep[static_cast<int64_t>(blockIdx.x) * kPrepSlots] = acc[0];
}

// The host's init_control, per instance on the device.
__global__ void k_init_ctl(Global g, DeviceOptions o, int32_t count, int32_t mixed, int32_t warm,
                           const double* warm_weight, double eta_max, double initial_weight,
                           double objective_offset) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= count) return;
    if (g.slot_mask != nullptr && g.slot_mask[b] == 0) return;
    const InstanceInfo inf = g.info[b];
    double rows = 0.0, cols = 0.0;
    for (int k = inf.vec_cta_begin; k < inf.vec_cta_end; ++k) {
        const double v = g.part_prep[static_cast<int64_t>(k) * kPrepSlots];
        if (g.vec[k].is_row) rows += v; else cols += v;
    }
    InstanceCtl c;
    memset(&c, 0, sizeof(c));
    c.phase = kPhaseMain;
    c.stage = kStageCheck;
    c.check_kind = kCheckInitial;
    c.need_refresh = 1;
    c.fp64_stage = mixed ? 0 : 1;
    c.status = -1;
    c.limit_status = 3;
    c.have_avg_at_check = warm;
    c.eta_max = eta_max;
    c.eta = clampd(o.initial_step_safety * eta_max, o.min_step_scale * eta_max, eta_max);
    c.omega = 1.0;
    set_weight(c.omega, o, initial_weight);
    if (warm_weight != nullptr && warm_weight[b] > 0.0) set_weight(c.omega, o, warm_weight[b]);
    c.trial_eta = c.ctl_eta = c.eta;
    c.trial_omega = c.ctl_omega = c.omega;
    c.best_pobj = nan("");
    c.best_dobj = -INFINITY;
    c.best_pres = c.best_dres = c.best_gap = c.best_kkt = INFINITY;
    c.restart_baseline = INFINITY;
    c.prev_candidate = INFINITY;
    c.pnorm = 1.0 + sqrt(rows);
    c.dnorm = 1.0 + sqrt(cols);
    c.objective_offset = objective_offset;
    g.ctl[b] = c;
}


// ---------------------------------------------------------------------------
// Streams: refill finished slots with the next instances of a queue.
// ---------------------------------------------------------------------------
__global__ void k_gather_slots(const double* __restrict__ src, const double* __restrict__ fam,
                               double* __restrict__ dst, const int32_t* __restrict__ perm,
                               const int64_t* __restrict__ inst, const int32_t* __restrict__ mask,
                               int64_t len, int32_t count) {
    const int64_t total = len * count;
    for (int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; t < total;
         t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t b = t / len, k = t - b * len;
        if (mask[b] == 0) continue;
        dst[t] = src != nullptr ? src[inst[b] * len + perm[k]] : fam[k];
    }
}

__global__ void k_scatter_slots(const double* __restrict__ src, double* __restrict__ out,
                                const int32_t* __restrict__ perm, const int64_t* __restrict__ inst,
                                const int32_t* __restrict__ mask, int64_t len, int32_t count) {
    const int64_t total = len * count;
    for (int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; t < total;
         t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t b = t / len, k = t - b * len;
        if (mask[b] == 0) continue;
        out[inst[b] * len + perm[k]] = src[t];
    }
}

// Marks every slot finished (no work) before a stream fills them.
__global__ void k_retire(Global g, int32_t count) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= count) return;
    InstanceCtl& c = g.ctl[b];
    c.phase = kPhaseDone;
    c.stage = kStageTrial;
    c.best_src = c.restart_src = c.need_refresh = c.to_polish = c.save_ray = 0;
}

__global__ void k_slot_done(Global g, int32_t count, int32_t* done) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b < count) done[b] = g.ctl[b].phase == kPhaseDone ? 1 : 0;
}

inline unsigned blocks_for(int64_t n, int per) { return static_cast<unsigned>((n + per - 1) / per); }

}  // namespace

// ---------------------------------------------------------------------------
// Launch wrappers
// ---------------------------------------------------------------------------
void launch_warp_heads(const Global& g, cudaStream_t s) {
    const int64_t n = static_cast<int64_t>(g.a.num_ctas + g.at.num_ctas) * kWarps;
    if (n > 0) k_warp_heads<<<blocks_for(n, 256), 256, 0, s>>>(g);
}

namespace {
// A trial kernel; `chained`: its predecessor in the stream is a trial kernel,
// so it may start while that one ends (see pdl_wait).
template <class... P, class... A>
void launch_trial(void (*kernel)(P...), int32_t ctas, int threads, bool chained, cudaStream_t s, A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(ctas));
    cfg.blockDim = dim3(static_cast<unsigned>(threads));
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = chained ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}
// As many CTAs as the device holds at once, at most one per entry of the map.
template <class T>
int32_t trial_ctas(const Global& g, const Side& side) {
    return std::min<int32_t>(side.num_ctas, g.sms * kTrialCtas<T>);
}
}  // namespace

template <class T>
void launch_primal(const Global& g, const Work<T>& w, const DeviceOptions&, int vw, cudaStream_t s, bool chained) {
    if (g.at.num_ctas == 0) return;
    switch (vw) {
        case 4: launch_trial(k_primal_wide<T, 4>, g.at.num_ctas, kThreads, chained, s, g, w); break;
        case 2: launch_trial(k_primal_wide<T, 2>, g.at.num_ctas, kThreads, chained, s, g, w); break;
        default: launch_trial(k_primal<T>, trial_ctas<T>(g, g.at), kThreads, chained, s, g, w); break;
    }
}

namespace {
// The fused kernel of a shape: staged ones by layout and by whether a worker
// has one slice a side (the code of one slice is a quarter as long, and a
// trial is as fast as its instructions come in) or up to kFusedLocal.
template <class T, bool kLimits>
auto fused_kernel(int vw, int cluster, const FusedShape& f) {
    if (f.mode == kFusedGlobal)
        return vw == 4 ? k_fused_global<T, 4, kLimits> : vw == 2 ? k_fused_global<T, 2, kLimits>
                                                                 : k_fused_global<T, 1, kLimits>;
    if (std::max(f.slices_p, f.slices_d) <= cluster * kFusedCtaWorkers)
        return f.mode == kFusedCopies ? k_fused<T, kFusedCopies, 1, kLimits> : k_fused<T, kFusedStaged, 1, kLimits>;
    return f.mode == kFusedCopies ? k_fused<T, kFusedCopies, kFusedLocal, kLimits>
                                  : k_fused<T, kFusedStaged, kFusedLocal, kLimits>;
}

template <class T>
auto fused_kernel(int vw, int cluster, const FusedShape& f) {
    return f.limits ? fused_kernel<T, true>(vw, cluster, f) : fused_kernel<T, false>(vw, cluster, f);
}

// The launch configuration of `count` clusters; false where the device
// refuses it.
template <class K>
bool fused_config(K kernel, int count, int cluster, const FusedShape& shape, cudaLaunchConfig_t& cfg,
                  cudaLaunchAttribute& attr) {
    const size_t smem = fused_smem_bytes(shape);
    cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(count * cluster));
    cfg.blockDim = dim3(kFusedThreads);
    cfg.dynamicSmemBytes = smem;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = static_cast<unsigned>(cluster);
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    // The limit is the kernel's, shared by every engine of the process, so all
    // set the same one: an engine that set its own size would lower it between
    // another's query and its launch. Clusters of 16 CTAs are beyond the
    // portable size of 8.
    static_assert(kFusedMaxSmemHost + sizeof(FusedCta) <= 227 * 1024, "beside the static shared memory");
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(kFusedMaxSmemHost)) == cudaSuccess &&
        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess)
        return true;
    cudaGetLastError();
    return false;
}
}  // namespace

template <class T>
cudaError_t launch_fused(const Global& g, const Work<T>& w, const DeviceOptions& o, int vw, int count,
                         int cluster, int max_trials, const FusedShape& shape, cudaStream_t s) {
    if (count <= 0) return cudaSuccess;
    auto* kernel = fused_kernel<T>(vw, cluster, shape);
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    if (!fused_config(kernel, count, cluster, shape, cfg, attr)) return cudaErrorInvalidConfiguration;
    cfg.stream = s;
    return cudaLaunchKernelEx(&cfg, kernel, g, w, o, vw == 4 ? 2 : vw == 2 ? 1 : 0, max_trials, shape);
}

template <class T>
int fused_max_clusters(int vw, int cluster, const FusedShape& shape) {
    auto* kernel = fused_kernel<T>(vw, cluster, shape);
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    if (!fused_config(kernel, 1, cluster, shape, cfg, attr)) return 0;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

template <class T>
void launch_dual(const Global& g, const Work<T>& w, const DeviceOptions& o, int vw, cudaStream_t s,
                 bool chained) {
    if (g.a.num_ctas == 0) return;
    switch (vw) {
        case 4: launch_trial(k_dual_wide<T, 4>, g.a.num_ctas, kThreads, chained, s, g, w); break;
        case 2: launch_trial(k_dual_wide<T, 2>, g.a.num_ctas, kThreads, chained, s, g, w); break;
        default: launch_trial(k_dual<T>, trial_ctas<T>(g, g.a), kThreads, chained, s, g, w); break;
    }
    if (!g.measure) launch_trial(k_decide<T>, g.instances, kDecideThreads, true, s, g, o);
}

template <class T>
void launch_check_prep(const Global& g, const Work<T>& w, const DeviceOptions& o, cudaStream_t s) {
    if (g.num_vec) k_check_prep<T><<<g.num_vec, kThreads, 0, s>>>(g, w, o);
}

void launch_check_spmv(const Global& g, const DeviceOptions& o, int vw, cudaStream_t s) {
    const int n = g.a.num_ctas + g.at.num_ctas;
    if (n == 0) return;
    switch (vw) {
        case 4: k_check_spmv<4><<<n, kThreads, 0, s>>>(g, o); break;
        case 2: k_check_spmv<2><<<n, kThreads, 0, s>>>(g, o); break;
        default: k_check_spmv<1><<<n, kThreads, 0, s>>>(g, o); break;
    }
}

void launch_check_ndg(const Global& g, const DeviceOptions& o, int32_t count, cudaStream_t s) {
    if (o.ndg_restarts && count > 0) k_check_ndg<<<count, kThreads, 0, s>>>(g, o);
}

template <class T>
void launch_check_apply(const Global& g, const Work<T>& w, const DeviceOptions&, cudaStream_t s) {
    if (g.num_vec) k_check_apply<T><<<g.num_vec, kThreads, 0, s>>>(g, w);
}

template <class T>
void launch_refresh(const Global& g, const Work<T>& w, const DeviceOptions&, int vw, cudaStream_t s) {
    if (g.a.num_ctas == 0) return;
    switch (vw) {
        case 4: k_refresh<T, 4><<<g.a.num_ctas, kThreads, 0, s>>>(g, w); break;
        case 2: k_refresh<T, 2><<<g.a.num_ctas, kThreads, 0, s>>>(g, w); break;
        default: k_refresh<T, 1><<<g.a.num_ctas, kThreads, 0, s>>>(g, w); break;
    }
}

void launch_finalize(const Global& g, int32_t count, int32_t* active, cudaStream_t s) {
    if (count) k_finalize<<<blocks_for(count, 256), 256, 0, s>>>(g, count, active);
}

void launch_switch_fp64(const Global& g, const Work<float>& w32, const Work<double>& w64,
                        cudaStream_t s) {
    if (g.num_vec) k_switch_fp64<<<g.num_vec, kThreads, 0, s>>>(g, w32, w64);
}

void launch_ruiz_max(const Global& g, int vw, int a_ctas, int at_ctas, cudaStream_t s) {
    if (a_ctas + at_ctas == 0) return;
    switch (vw) {
        case 4: k_ruiz_max<4><<<a_ctas + at_ctas, kThreads, 0, s>>>(g, a_ctas); break;
        case 2: k_ruiz_max<2><<<a_ctas + at_ctas, kThreads, 0, s>>>(g, a_ctas); break;
        default: k_ruiz_max<1><<<a_ctas + at_ctas, kThreads, 0, s>>>(g, a_ctas); break;
    }
}

void launch_ruiz_update(const Global& g, int vec_ctas, cudaStream_t s) {
    if (vec_ctas) k_ruiz_update<<<vec_ctas, kThreads, 0, s>>>(g);
}

void launch_scale_values(const Global& g, double* a_s64, double* at_s64, float* a_s32,
                         float* at_s32, int vw, int a_ctas, int at_ctas, cudaStream_t s) {
    if (a_ctas + at_ctas == 0) return;
    switch (vw) {
        case 4: k_scale_values<4><<<a_ctas + at_ctas, kThreads, 0, s>>>(g, a_s64, at_s64, a_s32, at_s32, a_ctas); break;
        case 2: k_scale_values<2><<<a_ctas + at_ctas, kThreads, 0, s>>>(g, a_s64, at_s64, a_s32, at_s32, a_ctas); break;
        default: k_scale_values<1><<<a_ctas + at_ctas, kThreads, 0, s>>>(g, a_s64, at_s64, a_s32, at_s32, a_ctas); break;
    }
}

template <class T>
void launch_precondition(const Global& g, const Work<T>& w, int enabled, int vw, int a_ctas,
                         int at_ctas, cudaStream_t s) {
    if (!enabled || a_ctas + at_ctas == 0) return;
    switch (vw) {
        case 4: k_precondition<T, 4><<<a_ctas + at_ctas, kThreads, 0, s>>>(g, w, a_ctas); break;
        case 2: k_precondition<T, 2><<<a_ctas + at_ctas, kThreads, 0, s>>>(g, w, a_ctas); break;
        default: k_precondition<T, 1><<<a_ctas + at_ctas, kThreads, 0, s>>>(g, w, a_ctas); break;
    }
}

template <class T>
void launch_setup_vectors(const Global& g, const Work<T>& w, cudaStream_t s) {
    if (g.num_vec) k_setup_vectors<T><<<g.num_vec, kThreads, 0, s>>>(g, w);
}

template <class T>
__global__ void k_fill(T* __restrict__ p, int64_t n, T v) {
    for (int64_t k = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; k < n;
         k += static_cast<int64_t>(gridDim.x) * blockDim.x)
        p[k] = v;
}

template <class T>
void launch_fill(T* p, int64_t n, T v, cudaStream_t s) {
    if (n > 0) k_fill<T><<<static_cast<int>(std::min<int64_t>(blocks_for(n, 256), 148 * 16)), 256, 0, s>>>(p, n, v);
}

void launch_broadcast_scales(const Global& g, const InstanceInfo& first, int32_t count,
                             int64_t rows, int64_t cols, cudaStream_t s) {
    (void)first;
    if (count > 1) k_broadcast_scales<<<592, 256, 0, s>>>(g.rs, g.cs, rows, cols, count);
}

template <class T>
void launch_broadcast_precond(const Work<T>& w, const InstanceInfo&, int32_t count, int64_t rows,
                              int64_t cols, cudaStream_t s) {
    if (count > 1)
        k_broadcast_precond<T><<<592, 256, 0, s>>>(w.sigma, w.isigma, w.tau, w.itau, rows, cols, count);
}

template <class T>
void launch_spmv(const Global& g, int transpose, int values, const T* v, T* out, int vw,
                 cudaStream_t s) {
    const Side& side = transpose ? g.at : g.a;
    if (side.num_ctas == 0) return;
    const T* vals;
    if constexpr (sizeof(T) == 8) {
        vals = values == 0 ? side.val_orig : side.val_s64;
    } else {
        vals = side.val_s32;
    }
    switch (vw) {
        case 4: k_spmv<T, 4><<<side.num_ctas, kThreads, 0, s>>>(g, transpose, vals, v, out); break;
        case 2: k_spmv<T, 2><<<side.num_ctas, kThreads, 0, s>>>(g, transpose, vals, v, out); break;
        default: k_spmv<T, 1><<<side.num_ctas, kThreads, 0, s>>>(g, transpose, vals, v, out); break;
    }
}

void launch_step_pow(double* table, int64_t entries, cudaStream_t s) {
    if (entries > 0) k_step_pow<<<blocks_for(entries, 256), 256, 0, s>>>(table, entries);
}

void launch_power_dot(const Global& g, const double* x, const double* z, cudaStream_t s) {
    if (g.num_vec) k_power_dot<<<g.num_vec, kThreads, 0, s>>>(g, x, z);
}
void launch_power_step(const Global& g, int32_t count, int init, int it, int budget, cudaStream_t s) {
    if (count) k_power_step<<<blocks_for(count, 128), 128, 0, s>>>(g, count, init, it, budget);
}
void launch_power_scale(const Global& g, double* x, const double* z, cudaStream_t s) {
    if (g.num_vec) k_power_scale<<<g.num_vec, kThreads, 0, s>>>(g, x, z);
}
void launch_power_finish(const Global& g, int32_t count, double safety, double min_scale, cudaStream_t s) {
    if (count) k_power_finish<<<blocks_for(count, 128), 128, 0, s>>>(g, count, safety, min_scale);
}
void launch_stamp_clock(const Global& g, int32_t count, int64_t elapsed_ns, int64_t limit_ns, cudaStream_t s) {
    if (count) k_stamp_clock<<<blocks_for(count, 128), 128, 0, s>>>(g, count, elapsed_ns, limit_ns);
}

void launch_permute(const double* src, double* dst, const int32_t* perm, int64_t len,
                    int32_t count, int mode, cudaStream_t s) {
    const int64_t total = len * count;
    if (total == 0) return;
    const unsigned blocks = static_cast<unsigned>(std::min<int64_t>((total + 255) / 256, 148 * 16));
    k_permute<<<blocks, 256, 0, s>>>(src, dst, perm, len, count, mode);
}
void launch_norm_parts(const Global& g, cudaStream_t s) {
    if (g.num_vec) k_norm_parts<<<g.num_vec, kThreads, 0, s>>>(g);
}
void launch_init_ctl(const Global& g, const DeviceOptions& o, int32_t count, int32_t mixed,
                     int32_t warm, const double* warm_weight, double eta_max,
                     double initial_weight, double objective_offset, cudaStream_t s) {
    if (count)
        k_init_ctl<<<blocks_for(count, 128), 128, 0, s>>>(g, o, count, mixed, warm, warm_weight,
                                                          eta_max, initial_weight, objective_offset);
}

void launch_gather_slots(const double* src, const double* fam, double* dst, const int32_t* perm,
                         const int64_t* inst, const int32_t* mask, int64_t len, int32_t count,
                         cudaStream_t s) {
    const int64_t total = len * count;
    if (total == 0) return;
    const unsigned blocks = static_cast<unsigned>(std::min<int64_t>((total + 255) / 256, 148 * 16));
    k_gather_slots<<<blocks, 256, 0, s>>>(src, fam, dst, perm, inst, mask, len, count);
}
void launch_scatter_slots(const double* src, double* out, const int32_t* perm, const int64_t* inst,
                          const int32_t* mask, int64_t len, int32_t count, cudaStream_t s) {
    const int64_t total = len * count;
    if (total == 0) return;
    const unsigned blocks = static_cast<unsigned>(std::min<int64_t>((total + 255) / 256, 148 * 16));
    k_scatter_slots<<<blocks, 256, 0, s>>>(src, out, perm, inst, mask, len, count);
}
void launch_retire(const Global& g, int32_t count, cudaStream_t s) {
    if (count) k_retire<<<blocks_for(count, 128), 128, 0, s>>>(g, count);
}
void launch_slot_done(const Global& g, int32_t count, int32_t* done, cudaStream_t s) {
    if (count) k_slot_done<<<blocks_for(count, 128), 128, 0, s>>>(g, count, done);
}

#define PDLPGPU_INSTANTIATE(T)                                                                      \
    template void launch_primal<T>(const Global&, const Work<T>&, const DeviceOptions&, int, cudaStream_t, bool); \
    template cudaError_t launch_fused<T>(const Global&, const Work<T>&, const DeviceOptions&, int, int, int, \
                                         int, const FusedShape&, cudaStream_t);                      \
    template int fused_max_clusters<T>(int, int, const FusedShape&);                                 \
    template void launch_dual<T>(const Global&, const Work<T>&, const DeviceOptions&, int, cudaStream_t, bool); \
    template void launch_check_prep<T>(const Global&, const Work<T>&, const DeviceOptions&, cudaStream_t);  \
    template void launch_check_apply<T>(const Global&, const Work<T>&, const DeviceOptions&, cudaStream_t); \
    template void launch_refresh<T>(const Global&, const Work<T>&, const DeviceOptions&, int, cudaStream_t); \
    template void launch_precondition<T>(const Global&, const Work<T>&, int, int, int, int, cudaStream_t);  \
    template void launch_setup_vectors<T>(const Global&, const Work<T>&, cudaStream_t);                    \
    template void launch_fill<T>(T*, int64_t, T, cudaStream_t);                                              \
    template void launch_broadcast_precond<T>(const Work<T>&, const InstanceInfo&, int32_t, int64_t, int64_t, cudaStream_t); \
    template void launch_spmv<T>(const Global&, int, int, const T*, T*, int, cudaStream_t);

PDLPGPU_INSTANTIATE(double)
PDLPGPU_INSTANTIATE(float)

}  // namespace pdlpgpu
