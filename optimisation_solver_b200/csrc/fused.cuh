// fused.cuh -- the trials of small LPs in one launch (included by kernels.cu,
// whose slice arithmetic it shares).
//
// One thread-block cluster per instance runs the trials of a check interval.
// A CTA has sixteen worker warps and one that decides; the instance's slices
// are dealt to the C CTAs in turn, and a CTA's to its workers in turn. A trial:
//   primal half of every slice (k_primal's arithmetic, its warp sum per
//   slice), the warp sums stored into every CTA          cluster barrier
//   dual half of every slice (k_dual's)                  cluster barrier
//   the decision, in every CTA on its own copy of the control block, while
//   the workers already gather the next primal half's sums from the trial
//   dual -- the one it needs unless the trial is rejected  CTA barrier
// A rejected trial (one in a hundred) gathers again. The decision adds each
// CTA-map entry's slice sums in slice order (k_primal's and k_dual's block
// sums: one slice per warp, warps in order), then the entries' three sums in
// k_dual's fixed order, so an instance's results are the two-kernel path's
// bit for bit; every CTA adds the same numbers, so all of them agree without
// being told. What that does not cover -- the check boundary, limits, a
// clock that has run out, non-finite sums -- goes through trial_control in rank
// 0, whose control block is then copied to the others. The clock is read by rank
// 0 while the workers run (1000 x 2000, FP64, 4000 trials with their checks: 4.9 us
// a trial with a time limit as without, 4.7 with a fixed step; 6.9 and 6.5 when
// all of those went through rank 0).
//
// Where the vectors live (chosen by Engine::choose_fused):
//   copies  every CTA holds the whole trial x and the whole y of both
//           parities; gathers are local, and the owner lane of a line writes
//           its new value into all C copies (a slice's lanes own consecutive
//           lines, so each remote store is one contiguous run). The slices,
//           the lines' constants, iterates and averages are staged in the
//           owner's shared memory. No trial touches global memory.
//   staged  as copies, but x and y go through L2: a gather is slower, a new
//           value is stored once instead of into every CTA. The better one
//           for sixteen CTAs and short lines, where a trial has as many stores as
//           gathers.
//   global  nothing is staged (more slices than four per warp, or no room).
// Vectors another CTA writes inside the launch are read through L2 (ld.cg);
// the barrier's release and acquire order them.
//
// Bound by latency: two cluster barriers and three dependent phases a trial.
// 100 trials, FP64, of a 40 x 70 planted LP (one CTA) 224 us, 1000 x 2000
// (4 CTAs) 399, a 2000-node flow LP (16 CTAs, staged) 801. With three barriers a
// trial, the decision by the workers and 32-bit indices from step-major global
// slices they were 383, 570 and 1133. Of 1000 x 2000's 7800 cycles a trial
// the sums and the decision take 2900, the dual gathers 1900, the primal 1100
// and waiting for the slowest CTA 1400.
#pragma once

constexpr int kFusedWorkers = kFusedCtaWorkers;
constexpr int kFusedThreads = 32 * (kFusedWorkers + 1);

// Every thread of every CTA of the cluster; the warp is reconverged first.
__device__ __forceinline__ void cluster_sync_all() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// Every thread of the CTA, from the workers' loop and the decider's.
__device__ __forceinline__ void cta_sync_all() {
    __syncwarp();
    asm volatile("barrier.cta.sync 1, %0;" ::"n"(kFusedThreads) : "memory");
}

// Every thread of the C CTAs. A cluster of one takes the CTA's barrier (the
// cluster's costs 490 cycles even then).
__device__ __forceinline__ void trial_sync(uint32_t C) {
    if (C == 1) cta_sync_all();
    else cluster_sync_all();
}

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

__device__ __forceinline__ uint32_t cluster_size() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}

// The lanes' values of one warp added by the butterfly of block_sum's first
// stage (every lane gets the sum).
template <int NQ>
__device__ __forceinline__ void warp_sum(double (&v)[NQ]) {
#pragma unroll
    for (int q = 0; q < NQ; ++q)
        for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(kFull, v[q], o);
}

// What the workers need of the control block for a trial.
struct alignas(16) FusedCtl {
    double mult_primal, mult_dual, frac;
    int active, parity, pending;
    int accepted;   // the trial before was accepted: its dual is the current one
    int slow;       // the decision goes through rank 0 (see FusedState)
    int expired;    // the time limit has passed; set by rank 0, never taken back
};

// The next trial's snapshot of an instance's control block.
__device__ __forceinline__ void fused_snapshot(const InstanceCtl& c, FusedCtl& f, bool fp64) {
    f.active = c.phase != kPhaseDone && c.stage == kStageTrial && (c.fp64_stage != 0) == fp64;
    f.parity = c.parity;
    f.pending = c.pending_avg;
    f.mult_primal = c.trial_eta / c.trial_omega;
    f.mult_dual = c.trial_eta * c.trial_omega;
    f.frac = c.avg_frac;
    f.accepted = 0;
    f.slow = 0;     // (expired is the clock's alone)
}

template <class T, int V>
__device__ __forceinline__ double fused_primal(const Global& g, const Work<T>& w, const CtaWork& cw,
                                               const InstanceInfo& inf, const FusedCtl& f, int lt) {
    const int p = f.parity;
    const T mult = static_cast<T>(f.mult_primal);
    const bool pending = f.pending != 0;
    const T frac = static_cast<T>(f.frac);
    const T* y = w.Y[p] + inf.row_off;
    const T* x = w.X[p] + inf.col_off;
    T* xt = w.X[p ^ 1] + inf.col_off;
    const T* cv = w.c + inf.col_off;
    const T* lo = w.xl + inf.col_off;
    const T* hi = w.xu + inf.col_off;
    const T* tau = w.tau + inf.col_off;
    const T* itau = w.itau + inf.col_off;
    T* avg = w.avg_x + inf.col_off;
    const T* vals = matrix_values<T>(g.at);
    double moved = 0.0;
    const int warp = lt >> 5, lane = lt & 31;
    for (int s = cw.slice_begin + warp; s < cw.slice_end; s += kWarps) {
        const SliceDesc sd = g.at.slices[s];
        const LanePos lp = lane_pos(sd, lane);
        const bool owner = lp.valid && lp.g == 0;
        const int j = lp.line;
        const int len = lp.valid ? g.at.line_len[inf.at_len_base + j] : 0;
        T cj = T(0), prev = T(0), loj = T(0), hij = T(0), tj = T(0), itj = T(0), aj = T(0);
        if (owner) {
            cj = cv[j];
            prev = __ldcg(x + j);
            loj = lo[j];
            hij = hi[j];
            tj = tau[j];
            itj = itau[j];
            if (pending) aj = __ldcg(avg + j);
        }
        T sum[1] = {T(0)};
        line_sums<V, 1>(inf.at_data_base + static_cast<int64_t>(sd.data_off) * 32, sd.steps, lp, lane, len,
                        g.at.idx, vals, sum, [&](T (&a)[1], T v, int i) { a[0] += v * __ldcg(y + i); });
        if (owner) {
            const T gradient = cj + sum[0];
            const T upd = smax(loj, smin(prev - mult * tj * gradient, hij));
            xt[j] = upd;
            const double d = static_cast<double>(upd - prev);
            moved += d * d * static_cast<double>(itj);
            if (pending) avg[j] = aj + frac * (prev - aj);
        }
    }
    return moved;
}

template <class T, int V>
__device__ __forceinline__ void fused_dual(const Global& g, const Work<T>& w, const CtaWork& cw,
                                           const InstanceInfo& inf, const FusedCtl& f, int lt,
                                           double (&red)[2]) {
    const int p = f.parity;
    const T dm = static_cast<T>(f.mult_dual);
    const bool pending = f.pending != 0;
    const T frac = static_cast<T>(f.frac);
    const T* xt = w.X[p ^ 1] + inf.col_off;
    const T* y = w.Y[p] + inf.row_off;
    T* yt = w.Y[p ^ 1] + inf.row_off;
    const T* ax = w.AX[p] + inf.row_off;
    T* axt = w.AX[p ^ 1] + inf.row_off;
    const T* lo = w.rl + inf.row_off;
    const T* hi = w.ru + inf.row_off;
    const T* sig = w.sigma + inf.row_off;
    const T* isig = w.isigma + inf.row_off;
    T* avg = w.avg_y + inf.row_off;
    const T* vals = matrix_values<T>(g.a);
    const int warp = lt >> 5, lane = lt & 31;
    for (int s = cw.slice_begin + warp; s < cw.slice_end; s += kWarps) {
        const SliceDesc sd = g.a.slices[s];
        const LanePos lp = lane_pos(sd, lane);
        const bool owner = lp.valid && lp.g == 0;
        const int i = lp.line;
        const int len = lp.valid ? g.a.line_len[inf.a_len_base + i] : 0;
        T axi = T(0), sgi = T(0), prev = T(0), loi = T(0), hii = T(0), isi = T(0), ai = T(0);
        if (owner) {
            axi = __ldcg(ax + i);
            sgi = sig[i];
            prev = __ldcg(y + i);
            loi = lo[i];
            hii = hi[i];
            isi = isig[i];
            if (pending) ai = __ldcg(avg + i);
        }
        T sum[1] = {T(0)};
        line_sums<V, 1, true>(inf.a_data_base + static_cast<int64_t>(sd.data_off) * 32, sd.steps, lp, lane, len,
                              g.a.idx, vals, sum, [&](T (&a)[1], T v, int j) { a[0] += v * __ldcg(xt + j); });
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
}


// Distributed shared memory of rank `r`: the address of `local` there, and
// stores.
__device__ __forceinline__ uint32_t rank_addr(const void* local, uint32_t r) {
    const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(local));
    uint32_t out;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(a), "r"(r));
    return out;
}
__device__ __forceinline__ void st_cluster(uint32_t addr, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ void st_cluster(uint32_t addr, int v) {
    asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void st_cluster(uint32_t addr, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
// The value v of element `e` of a copied vector, stored into all C copies.
template <class T>
__device__ __forceinline__ void store_copies(const T* elem, T v, uint32_t C) {
    for (uint32_t r = 0; r < C; ++r) st_cluster(rank_addr(elem, r), v);
}

// Step factors a CTA keeps in shared memory, of the iteration indices that come
// next; trials past them fetch as many again (past the options' table the
// slow decision computes them).
constexpr int kFusedFactors = 160;
__device__ __forceinline__ int fused_factors(const DeviceOptions& o, int64_t first) {
    const int64_t avail = first >= 0 && first < o.step_pow_entries ? o.step_pow_entries - first : 0;
    return static_cast<int>(avail < kFusedFactors ? avail : kFusedFactors);
}

// ---------------------------------------------------------------------------
// The decision, in the registers of a CTA's deciding warp (every lane holds
// the same values): the cases of trial_control that stay inside a check
// interval. `decide` returns false, with nothing changed, for the rest.
// ---------------------------------------------------------------------------
template <bool kLimits>
struct FusedState {
    double eta, omega_eval, omega_trial, eta_max;   // of the phase's controller
    double held;          // the trials' step while polishing with a fixed step (else eta is)
    double avg_weight, avg_frac;
    double sums[3];
    int64_t index0;       // iteration index at load
    int64_t to_check;     // accepted trials until the check boundary or the limit
    int parity, pending, rejected;
    int accepted, trials; // since the load
    bool polish;

    __device__ __forceinline__ void load(const InstanceCtl& c, const DeviceOptions& o) {
        polish = c.phase == kPhasePolish;
        eta = polish ? c.ctl_eta : c.eta;
        omega_eval = polish ? c.ctl_omega : c.omega;
        omega_trial = polish ? c.trial_omega : c.omega;
        if (kLimits) held = c.trial_eta;
        eta_max = c.eta_max;
        avg_weight = c.avg_weight;
        avg_frac = c.avg_frac;
        index0 = polish ? c.polish_iteration : c.iteration;
        const int64_t done = polish ? c.polish_done_iterations : c.iteration;
        to_check = o.check_frequency - count_mod(done, o.check_frequency);
        const int64_t left = (polish ? static_cast<int64_t>(o.polishing_iterations) : o.iteration_limit) - done;
        if (left < to_check) to_check = left;
        parity = c.parity;
        pending = c.pending_avg;
        rejected = c.trials_this_iter;
        accepted = trials = 0;
    }

    // trial_control's changes of `trials` trials.
    __device__ __forceinline__ void store(InstanceCtl& c, const DeviceOptions& o) const {
        if (trials == 0) return;
        c.dbg[0] = sums[0];
        c.dbg[1] = sums[1];
        c.dbg[2] = sums[2];
        c.trial_eta = step(o);
        if (polish) {
            c.ctl_eta = eta;
            c.polish_trials += trials;
            c.polish_iteration += accepted;
            c.polish_done_iterations += accepted;
        } else {
            c.eta = eta;
            c.trial_omega = omega_trial;
            c.step_trials += trials;
            c.iteration += accepted;
            c.since_restart += accepted;
        }
        if (c.fp64_stage && o.mixed) c.fp64_iterations += accepted;
        c.avg_weight = avg_weight;
        c.avg_frac = avg_frac;
        c.pending_avg = pending;
        c.parity = parity;
        c.trials_this_iter = rejected;
    }

    // The trials' step.
    __device__ __forceinline__ double step(const DeviceOptions& o) const {
        return kLimits && polish && !o.adaptive ? held : eta;
    }

    // Iteration index of the trial under way.
    __device__ __forceinline__ int64_t iteration() const { return index0 + accepted; }

    // `factors`: nfactors of them, from iteration index `first` on.
    __device__ __forceinline__ bool decide(const DeviceOptions& o, const double (&s)[3], const double* factors,
                                           int64_t first, int nfactors) {
        const int64_t k = iteration() - first;
        if (k >= nfactors || !(isfinite(s[0]) && isfinite(s[1]) && isfinite(s[2]))) return false;
        double next = eta;
        const bool accept =
            (kLimits && !o.adaptive) || evaluate_step(next, omega_eval, eta_max, o, s[0], s[1], s[2], iteration(), factors + 2 * k);
        if (accept ? to_check <= 1 : rejected + 1 >= o.max_trials) return false;
        eta = next;
        ++trials;
        pending = 0;
#pragma unroll
        for (int q = 0; q < 3; ++q) sums[q] = s[q];
        if (!accept) {
            ++rejected;
            return true;
        }
        parity ^= 1;
        rejected = 0;
        ++accepted;
        --to_check;
        const double weight = step(o);
        if (o.averaging && weight > 0.0) {   // average_add
            const double total = avg_weight + weight;
            avg_frac = weight / total;
            avg_weight = total;
            pending = 1;
        }
        return true;
    }
};

// A lane's share of the sums over the CTA-map entries: entries lane, lane + 32,
// ... in order, each the in-order total of its slices' warp sums (NV values a
// slice). Four entries' loads are in flight together. Table word: first
// slice << 4 | slice count.
template <int NV>
__device__ __forceinline__ void entry_sums(const int32_t* tab, int entries, const double* part, int lane,
                                           double (&s)[NV]) {
    if (entries <= 64) {   // short: little code before little work
        for (int e = lane; e < entries; e += 32) {
            const int first = tab[e] >> 4, count = tab[e] & 15;
            double v[NV];
#pragma unroll
            for (int q = 0; q < NV; ++q) v[q] = 0.0;
#pragma unroll 1
            for (int k = 0; k < count; ++k)
#pragma unroll
                for (int q = 0; q < NV; ++q) v[q] += part[(first + k) * NV + q];
#pragma unroll
            for (int q = 0; q < NV; ++q) s[q] += v[q];
        }
        return;
    }
    constexpr int kAhead = 4;
    for (int base = 0; base < entries; base += 32 * kAhead) {
        int word[kAhead];
        double v[kAhead][NV];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int e = base + 32 * u + lane;
            word[u] = e < entries ? tab[e] : 0;
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
#pragma unroll
            for (int q = 0; q < NV; ++q) v[u][q] = (word[u] & 15) ? part[(word[u] >> 4) * NV + q] : 0.0;
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
            for (int k = 1; k < (word[u] & 15); ++k)
#pragma unroll
                for (int q = 0; q < NV; ++q) v[u][q] += part[((word[u] >> 4) + k) * NV + q];
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
#pragma unroll
            for (int q = 0; q < NV; ++q) s[q] += v[u][q];
    }
}

// ---------------------------------------------------------------------------
// A staged slice: per lane a head word -- its line's length, and above it, in
// the lane that owns the line, the line's number plus one (else 0; both fit
// 16 bits, see choose_fused); the entries, indices in 16 bits; then per lane
// the line's constants and own vectors. (The cluster barriers acquire at
// cluster scope, after which the SM's L1 holds nothing of global memory, so
// what is not staged comes from L2 in every trial.)
// ---------------------------------------------------------------------------
template <class T>
struct FusedSlice {
    uint32_t* head;
    uint16_t* idx;   // [steps][32]
    T* val;
    T* k;            // constants [consts][32], then own vectors [own][32]
    int steps, glog;
    __device__ __forceinline__ int line(int lane) const { return static_cast<int>(head[lane] >> 16) - 1; }
};
// Where it lies: byte offset in the stage, steps and log2 of the lane group.
struct FusedPlace {
    int off, steps, glog;
};
template <class T>
__device__ __forceinline__ FusedSlice<T> fused_slice(unsigned char* stage, const FusedPlace& p) {
    FusedSlice<T> s;
    unsigned char* b = stage + p.off;
    s.head = reinterpret_cast<uint32_t*>(b);
    s.idx = reinterpret_cast<uint16_t*>(b + kFusedHeadBytes);
    s.val = reinterpret_cast<T*>(b + kFusedHeadBytes + 64 * p.steps);
    s.k = s.val + 32 * p.steps;
    s.steps = p.steps;
    s.glog = p.glog;
    return s;
}

template <class T>
__device__ __forceinline__ void fused_stage(const Side& side, const T* vals, int64_t data_base, int64_t len_base,
                                            int slice, unsigned char* stage, const FusedPlace& at,
                                            const T* const* consts, int nconsts, const T* const* own, int nown,
                                            int vlog, int lane) {
    const SliceDesc sd = side.slices[slice];
    const FusedSlice<T> s = fused_slice<T>(stage, at);
    const LanePos lp = lane_pos(sd, lane);
    const bool owner = lp.valid && lp.g == 0;
    const uint32_t len = lp.valid ? static_cast<uint32_t>(side.line_len[len_base + lp.line]) : 0u;
    s.head[lane] = len | (owner ? static_cast<uint32_t>(lp.line + 1) << 16 : 0u);
    const int64_t base = data_base + static_cast<int64_t>(sd.data_off) * 32;
    for (int st = 0; st < sd.steps; ++st) {   // step by step, whatever the matrix's load width V
        const int64_t q = base + (st >> vlog) * (32 << vlog) + (lane << vlog) + (st & ((1 << vlog) - 1));
        s.idx[32 * st + lane] = static_cast<uint16_t>(side.idx[q]);
        s.val[32 * st + lane] = vals[q];
    }
    for (int c = 0; c < nconsts; ++c) s.k[c * 32 + lane] = owner ? consts[c][lp.line] : T(0);
    for (int c = 0; c < nown; ++c) s.k[(nconsts + c) * 32 + lane] = owner ? own[c][lp.line] : T(0);
}

// line_sums over a staged slice: the same products added in the same order
// (steps 0, 1, ... of the lane, then the lane group's butterfly), with eight
// gathers in flight since the entries come from shared memory; `get(i)`
// gathers element i of the other side's vector.
template <class T, class Get>
__device__ __forceinline__ T staged_sum(const FusedSlice<T>& L, int lane, Get get) {
    constexpr int kAhead = 8;
    const int len = static_cast<int>(L.head[lane] & 0xffffu), g = lane & ((1 << L.glog) - 1);
    T acc = T(0);
    for (int s0 = 0; s0 < L.steps; s0 += kAhead) {
        T gv[kAhead], wv[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int st = s0 + u;
            gv[u] = T(0);
            wv[u] = T(0);
            if (st < L.steps && (st << L.glog) + g < len) {
                wv[u] = L.val[32 * st + lane];
                gv[u] = get(L.idx[32 * st + lane]);
            }
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int st = s0 + u;
            // (An FMA by name: left to the compiler, the eighth product of a
            // full group was rounded before it was added.)
            if (st < L.steps && (st << L.glog) + g < len) acc = fma(wv[u], gv[u], acc);
        }
    }
    for (int o = (1 << L.glog) >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
    return acc;
}

// What a CTA keeps in shared memory beside the staged slices, and where its
// instance's slices and entries lie.
struct FusedCta {
    DeviceOptions so;
    FusedCtl f;
    InstanceCtl ctl;
    double fac[2 * kFusedFactors];
};
struct FusedRange {
    int ps0, ps1, ds0, ds1;   // slices (contiguous in the CTA map: append_cta_map)
    int ne_p, ne_d;           // entries
};
// The tables and warp sums at the head of the dynamic shared memory: two
// sets of sums for the primal half (a CTA that has decided may be a half
// ahead of one that is still adding), one for the dual half.
struct FusedSums {
    double *p[2], *d;
    int32_t *tab_p, *tab_d;
};

__device__ __forceinline__ FusedSums fused_sums(unsigned char* smem, const FusedShape& fs) {
    FusedSums s;
    s.p[0] = reinterpret_cast<double*>(smem);
    s.p[1] = s.p[0] + fs.slices_p;
    s.d = s.p[1] + fs.slices_p;
    s.tab_p = reinterpret_cast<int32_t*>(s.d + 2 * fs.slices_d);
    s.tab_d = s.tab_p + fs.entries_p;
    return s;
}

// Fills them; the caller synchronises the CTA before they are read.
__device__ __forceinline__ FusedRange fused_setup(const Global& g, const DeviceOptions& o, const InstanceInfo& inf,
                                                  const InstanceCtl* cp, FusedCta& sc, const FusedSums& sums) {
    FusedRange r;
    r.ps0 = g.at.ctas[inf.at_cta_begin].slice_begin;
    r.ps1 = g.at.ctas[inf.at_cta_end - 1].slice_end;
    r.ds0 = g.a.ctas[inf.a_cta_begin].slice_begin;
    r.ds1 = g.a.ctas[inf.a_cta_end - 1].slice_end;
    r.ne_p = inf.at_cta_end - inf.at_cta_begin;
    r.ne_d = inf.a_cta_end - inf.a_cta_begin;
    if (threadIdx.x == 0) {
        sc.so = o;
        sc.f.expired = 0;
    }
    if (threadIdx.x < sizeof(InstanceCtl) / 16)
        reinterpret_cast<int4*>(&sc.ctl)[threadIdx.x] = reinterpret_cast<const int4*>(cp)[threadIdx.x];
    for (int e = threadIdx.x; e < r.ne_p; e += kFusedThreads) {
        const CtaWork cw = g.at.ctas[inf.at_cta_begin + e];
        sums.tab_p[e] = ((cw.slice_begin - r.ps0) << 4) | (cw.slice_end - cw.slice_begin);
    }
    for (int e = threadIdx.x; e < r.ne_d; e += kFusedThreads) {
        const CtaWork cw = g.a.ctas[inf.a_cta_begin + e];
        sums.tab_d[e] = ((cw.slice_begin - r.ds0) << 4) | (cw.slice_end - cw.slice_begin);
    }
    return r;
}

// The deciding warp of a CTA, from the first trial to the launch's end. kLimits:
// there is a time limit or the step is fixed. (Kernels of their own: the few
// instructions it takes would cost every trial 1 to 4%.)
template <bool kLimits>
__device__ __forceinline__ void fused_decider(InstanceCtl* cp, int32_t n_cols, bool fp64, int max_trials,
                                              FusedCta& sc, const FusedSums& sums, const FusedRange& range,
                                              uint32_t C, uint32_t rank) {
    const int lane = threadIdx.x & 31;
    DeviceOptions& so = sc.so;
    FusedCtl& f = sc.f;
    InstanceCtl& sctl = sc.ctl;
    // Its registers are never the workers'; its barriers match theirs one for
    // one.
    FusedState<kLimits> state;
    state.load(sctl, so);
    const bool timed = kLimits && so.time_limit > 0.0 && sctl.deadline_ns > 0;
    int64_t fac0 = 0;   // the factors kept are of iteration indices fac0, fac0 + 1, ..., nfac of them
    int nfac = 0;
    int widest = 16;   // the butterfly's first step that meets an entry
    while (widest > 0 && widest >= max(range.ne_p, range.ne_d)) widest >>= 1;
    for (int t = 0; t < max_trials && f.active; ++t) {
        // By index, not by trial: a slow decision inside an interval loads the
        // state anew, past the iteration that the launch began with.
        if (state.iteration() - fac0 >= nfac) {
            fac0 = state.iteration();
            nfac = fused_factors(so, fac0);
            for (int q = lane; q < 2 * nfac; q += 32) sc.fac[q] = so.step_pow[2 * fac0 + q];
            __syncwarp();
        }
        // The clock, once a trial, by one lane of one CTA, for all: `expired` is
        // stored before the first barrier and read between the two, so every CTA
        // sees the same (after the second, rank 0 may be in the next trial).
        if (timed && rank == 0 && !state.polish) {
            const bool over = __shfl_sync(kFull, now_ns() >= sctl.deadline_ns ? 1 : 0, 0) != 0;
            if (over && static_cast<uint32_t>(lane) < C)
                st_cluster(rank_addr(&f.expired, static_cast<uint32_t>(lane)), 1);
        }
        trial_sync(C);
        const bool expired = timed && f.expired != 0;
        trial_sync(C);
        const double* const sums_p = sums.p[t & 1];
        // k_dual's fixed-order sums (warp_range_sum_deep: a lane's entries in
        // order, then the butterfly; its steps that would only add the
        // zeros of lanes without entries are left out).
        double s[3], sp[1] = {0.0}, sd[2] = {0.0, 0.0};
        entry_sums<1>(sums.tab_p, range.ne_p, sums_p, lane, sp);
        entry_sums<2>(sums.tab_d, range.ne_d, sums.d, lane, sd);
        s[0] = sp[0];
        s[1] = sd[0];
        s[2] = sd[1];
        for (int d = widest; d > 0; d >>= 1) {
#pragma unroll
            for (int q = 0; q < 3; ++q) s[q] += __shfl_xor_sync(kFull, s[q], d);
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) s[q] = __shfl_sync(kFull, s[q], 0);
        const int before = state.accepted;
        if (!expired && state.decide(so, s, sc.fac, fac0, nfac)) {
            if (lane == 0) {
                const double step = state.step(so);
                f.mult_primal = step / state.omega_trial;
                f.mult_dual = step * state.omega_trial;
                f.frac = state.avg_frac;
                f.parity = state.parity;
                f.pending = state.pending;
                f.accepted = state.accepted != before;
            }
        } else {
            if (lane == 0) f.slow = 1;
            if (rank == 0) {
                if (lane == 0) {
                    state.store(sctl, so);
                    trial_control(sctl, so, s[0], s[1], s[2], n_cols);
                }
                __syncwarp();
                if (lane < static_cast<int>(sizeof(InstanceCtl) / 16)) {
                    const int4 word = reinterpret_cast<const int4*>(&sctl)[lane];
                    for (uint32_t r = 1; r < C; ++r)
                        asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(
                                         rank_addr(reinterpret_cast<const int4*>(&sctl) + lane, r)),
                                     "r"(word.x), "r"(word.y), "r"(word.z), "r"(word.w)
                                     : "memory");
                }
            }
            state.trials = 0;   // the control block is ahead of the registers
        }
        cta_sync_all();
        if (f.slow) {   // the same in every CTA: all of them decide alike
            cluster_sync_all();
            state.load(sctl, so);
            if (lane == 0) fused_snapshot(sctl, f, fp64);
            cta_sync_all();
        }
    }
    // Every CTA leaves the loop at the same trial; the barrier keeps
    // every CTA's shared memory alive until the last remote store into it
    // has landed.
    cluster_sync_all();
    if (rank == 0) {
        if (lane == 0) state.store(sctl, so);
        __syncwarp();
        copy_ctl_warp(cp, &sctl);
    }
}

template <class T, int M, int NL, bool kLimits>
__global__ void __launch_bounds__(kFusedThreads, 1) k_fused(Global g, Work<T> w, DeviceOptions o, int vlog,
                                                           int max_trials, FusedShape fs) {
    constexpr bool kCopies = M == kFusedCopies;
    constexpr bool kFp64 = sizeof(T) == 8;
    __shared__ alignas(16) FusedCta sc;
    extern __shared__ __align__(16) unsigned char fused_smem[];
    const FusedSums sums = fused_sums(fused_smem, fs);
    T* const copies = reinterpret_cast<T*>(fused_smem + fused_copies_offset(fs));
    unsigned char* const stage = fused_smem + fused_stage_offset(fs);
    const uint32_t C = cluster_size(), rank = cluster_rank();
    const int b = static_cast<int>(blockIdx.x / C);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool decider = warp == kFusedWorkers;
    InstanceCtl* cp = g.ctl + b;
    const InstanceInfo inf = g.info[b];
    const FusedRange range = fused_setup(g, o, inf, cp, sc, sums);
    const int ps0 = range.ps0, ps1 = range.ps1, ds0 = range.ds0, ds1 = range.ds1;
    // Worker w of CTA r serves slices w C + r, + 16 C, ... of each side.
    const int stride = static_cast<int>(C) * kFusedWorkers;
    const int slot = warp * static_cast<int>(C) + static_cast<int>(rank);
    T* const xg[2] = {w.X[0] + inf.col_off, w.X[1] + inf.col_off};
    T* const yg[2] = {w.Y[0] + inf.row_off, w.Y[1] + inf.row_off};
    // Copies: y of both parities, then the trial x.
    T* const yc[2] = {copies, copies + inf.m};
    T* const xc = copies + 2 * inf.m;
    if (kCopies)
        for (int q = threadIdx.x; q < inf.m; q += kFusedThreads) {
            yc[0][q] = yg[0][q];
            yc[1][q] = yg[1][q];
        }
    // Own vectors of a staged line: average and x of both parities; Ax of
    // both parities, average and, without copies of y, y of both.
    constexpr int kOwnP = fused_own_primal(M), kOwnD = fused_own_dual(M);
    const T* const own_p[3] = {w.avg_x + inf.col_off, xg[0], xg[1]};
    const T* const own_d[5] = {w.AX[0] + inf.row_off, w.AX[1] + inf.row_off, w.avg_y + inf.row_off, yg[0], yg[1]};
    FusedPlace pp[NL], pd[NL];
    int np = 0, nd = 0;   // the worker's slices of each side
    // The workers' shares of the stage, in worker order (lane q computes
    // worker q's bytes).
    auto bytes = [&](const SliceDesc* slices, int s, int s1, int words) {
        int need = 0;
        for (; s < s1; s += stride) need += fused_slice_bytes(slices[s].steps, words, sizeof(T));
        return need;
    };
    const int first = lane * static_cast<int>(C) + static_cast<int>(rank);
    int need = 0;
    if (lane < kFusedWorkers)
        need = bytes(g.at.slices, ps0 + first, ps1, kFusedPrimalConsts + kOwnP) +
               bytes(g.a.slices, ds0 + first, ds1, kFusedDualConsts + kOwnD);
    int incl = need;
    for (int d = 1; d < 32; d <<= 1) {
        const int t = __shfl_up_sync(kFull, incl, d);
        if (lane >= d) incl += t;
    }
    int off = __shfl_sync(kFull, incl - need, warp);
    const T* const cp_consts[kFusedPrimalConsts] = {w.c + inf.col_off, w.xl + inf.col_off, w.xu + inf.col_off,
                                                    w.tau + inf.col_off, w.itau + inf.col_off};
    const T* const cd_consts[kFusedDualConsts] = {w.sigma + inf.row_off, w.isigma + inf.row_off,
                                                  w.rl + inf.row_off, w.ru + inf.row_off};
    #pragma unroll
    for (int i = 0; i < NL; ++i) {
        const int s = ps0 + slot + i * stride;
        if (decider || s >= ps1) continue;
        const SliceDesc sd = g.at.slices[s];
        pp[i] = {off, sd.steps, slice_glog(sd.meta)};
        fused_stage<T>(g.at, matrix_values<T>(g.at), inf.at_data_base, inf.at_len_base, s, stage, pp[i], cp_consts,
                       kFusedPrimalConsts, own_p, kOwnP, vlog, lane);
        off += fused_slice_bytes(sd.steps, kFusedPrimalConsts + kOwnP, sizeof(T));
        np = i + 1;
    }
    #pragma unroll
    for (int i = 0; i < NL; ++i) {
        const int s = ds0 + slot + i * stride;
        if (decider || s >= ds1) continue;
        const SliceDesc sd = g.a.slices[s];
        pd[i] = {off, sd.steps, slice_glog(sd.meta)};
        fused_stage<T>(g.a, matrix_values<T>(g.a), inf.a_data_base, inf.a_len_base, s, stage, pd[i], cd_consts,
                       kFusedDualConsts, own_d, kOwnD, vlog, lane);
        off += fused_slice_bytes(sd.steps, kFusedDualConsts + kOwnD, sizeof(T));
        nd = i + 1;
    }
    __syncthreads();
    FusedCtl& f = sc.f;
    if (decider && lane == 0) fused_snapshot(sc.ctl, f, kFp64);
    // Remote shared memory is written only once every CTA of the cluster runs.
    cluster_sync_all();
    if (decider) {
        fused_decider<kLimits>(cp, inf.n, kFp64, max_trials, sc, sums, range, C, rank);
        return;
    }

    auto primal_sum = [&](const FusedSlice<T>& L, int parity) {
        const T* y = kCopies ? yc[parity] : yg[parity];
        if constexpr (kCopies) return staged_sum(L, lane, [&](int i) { return y[i]; });
        else return staged_sum(L, lane, [&](int i) { return __ldcg(y + i); });
    };
    // A slice's warp sums, into every CTA's arrays.
    auto publish = [&](double* at, double v) {
        if (static_cast<uint32_t>(lane) < C) st_cluster(rank_addr(at, static_cast<uint32_t>(lane)), v);
    };
    T ahead[NL];   // the slices' sums over the last trial's dual
    for (int t = 0; t < max_trials && f.active; ++t) {
        const int p = f.parity;
        const bool pending = f.pending != 0;
        const T frac = static_cast<T>(f.frac);
        double* const sums_p = sums.p[t & 1];
        // The lanes' terms of the slices' sums, added over the warp together
        // at the end of the dual half (no decision needs them before).
        double vp[NL], vd[NL][2];
        const bool have = t > 0 && f.accepted;
        const T mult = static_cast<T>(f.mult_primal);
#pragma unroll
        for (int i = 0; i < NL; ++i) {
            vp[i] = 0.0;
            if (i >= np) continue;
            const FusedSlice<T> L = fused_slice<T>(stage, pp[i]);
            const T sum = have ? ahead[i] : primal_sum(L, p);
            const int j = L.line(lane);
            if (j >= 0) {
                T* const own = L.k + 32 * kFusedPrimalConsts + lane;   // average, x, x
                const T cj = L.k[lane], loj = L.k[32 + lane], hij = L.k[64 + lane];
                const T tj = L.k[96 + lane], itj = L.k[128 + lane];
                const T prev = own[32 * (1 + p)];
                const T gradient = cj + sum;
                const T upd = smax(loj, smin(prev - mult * tj * gradient, hij));
                own[32 * (1 + (p ^ 1))] = upd;
                if (kCopies) store_copies<T>(xc + j, upd, C);
                else xg[p ^ 1][j] = upd;
                const double d = static_cast<double>(upd - prev);
                vp[i] = d * d * static_cast<double>(itj);
                if (pending) {
                    const T aj = own[0];
                    own[0] = aj + frac * (prev - aj);
                }
            }
        }
        trial_sync(C);
        const T dm = static_cast<T>(f.mult_dual);
#pragma unroll
        for (int i = 0; i < NL; ++i) {
            vd[i][0] = vd[i][1] = 0.0;
            if (i >= nd) continue;
            const FusedSlice<T> L = fused_slice<T>(stage, pd[i]);
            const T* xt = kCopies ? xc : xg[p ^ 1];
            T sum;
            if constexpr (kCopies) sum = staged_sum(L, lane, [&](int jj) { return xt[jj]; });
            else sum = staged_sum(L, lane, [&](int jj) { return __ldcg(xt + jj); });
            const int r = L.line(lane);
            if (r >= 0) {
                T* const own = L.k + 32 * kFusedDualConsts + lane;   // Ax, Ax, average (, y, y)
                const T sgi = L.k[lane], isi = L.k[32 + lane], loi = L.k[64 + lane], hii = L.k[96 + lane];
                const T axi = own[32 * p];
                const T prev = kCopies ? yc[p][r] : own[32 * (3 + p)];
                const T next = sum;
                const T dact = next - axi;
                const T ext = next + dact;
                const T step = smax(dm * sgi, min_dual_step<T>());
                const T u = prev + step * ext;
                const T upd = smax(u - step * hii, T(0)) + smin(u - step * loi, T(0));
                if (kCopies) {
                    store_copies<T>(yc[p ^ 1] + r, upd, C);
                } else {
                    own[32 * (3 + (p ^ 1))] = upd;
                    yg[p ^ 1][r] = upd;
                }
                own[32 * (p ^ 1)] = next;
                const double d = static_cast<double>(upd - prev);
                vd[i][0] = d * d * static_cast<double>(isi);
                vd[i][1] = d * static_cast<double>(dact);
                if (pending) {
                    const T ai = own[64];
                    own[64] = ai + frac * (prev - ai);
                }
            }
        }
        // Without a branch inside a butterfly its values overlap.
        static_assert(NL == 1 || NL == 4, "the sums below name four slices");
        {
            double v[3] = {vp[0], vd[0][0], vd[0][1]};
            warp_sum<3>(v);
            if (np > 0) publish(sums_p + slot, v[0]);
            if (nd > 0) {
                publish(sums.d + 2 * slot, v[1]);
                publish(sums.d + 2 * slot + 1, v[2]);
            }
        }
        if constexpr (NL == 4) {
            if (np > 1) {
                double v[3] = {vp[1], vp[2], vp[3]};
                warp_sum<3>(v);
#pragma unroll
                for (int i = 1; i < NL; ++i)
                    if (i < np) publish(sums_p + slot + i * stride, v[i - 1]);
            }
            if (nd > 1) {
                double v[6] = {vd[1][0], vd[1][1], vd[2][0], vd[2][1], vd[3][0], vd[3][1]};
                warp_sum<6>(v);
#pragma unroll
                for (int i = 1; i < NL; ++i)
                    if (i < nd) {
                        publish(sums.d + 2 * (slot + i * stride), v[2 * i - 2]);
                        publish(sums.d + 2 * (slot + i * stride) + 1, v[2 * i - 1]);
                    }
            }
        }
        trial_sync(C);
#pragma unroll
        for (int i = 0; i < NL; ++i)
            if (i < np) ahead[i] = primal_sum(fused_slice<T>(stage, pp[i]), p ^ 1);
        cta_sync_all();
        if (f.slow) {
            cluster_sync_all();
            cta_sync_all();
        }
    }
    cluster_sync_all();
    // The owner lanes write their lines' iterates and averages back.
#pragma unroll
    for (int i = 0; i < NL; ++i) {
        if (i >= np) continue;
        const FusedSlice<T> L = fused_slice<T>(stage, pp[i]);
        const int j = L.line(lane);
        if (j < 0) continue;
        const T* own = L.k + 32 * kFusedPrimalConsts + lane;
        w.avg_x[inf.col_off + j] = own[0];
        xg[0][j] = own[32];
        xg[1][j] = own[64];
    }
#pragma unroll
    for (int i = 0; i < NL; ++i) {
        if (i >= nd) continue;
        const FusedSlice<T> L = fused_slice<T>(stage, pd[i]);
        const int r = L.line(lane);
        if (r < 0) continue;
        const T* own = L.k + 32 * kFusedDualConsts + lane;
        w.AX[0][inf.row_off + r] = own[0];
        w.AX[1][inf.row_off + r] = own[32];
        w.avg_y[inf.row_off + r] = own[64];
        yg[0][r] = kCopies ? yc[0][r] : own[96];
        yg[1][r] = kCopies ? yc[1][r] : own[128];
    }
}

// The same with nothing staged: slices and vectors through L2 in every trial.
template <class T, int V, bool kLimits>
__global__ void __launch_bounds__(kFusedThreads, 1) k_fused_global(Global g, Work<T> w, DeviceOptions o, int,
                                                                  int max_trials, FusedShape fs) {
    constexpr bool kFp64 = sizeof(T) == 8;
    __shared__ alignas(16) FusedCta sc;
    extern __shared__ __align__(16) unsigned char fused_smem[];
    const FusedSums sums = fused_sums(fused_smem, fs);
    const uint32_t C = cluster_size(), rank = cluster_rank();
    const int b = static_cast<int>(blockIdx.x / C);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool decider = warp == kFusedWorkers;
    InstanceCtl* cp = g.ctl + b;
    const InstanceInfo inf = g.info[b];
    const FusedRange range = fused_setup(g, o, inf, cp, sc, sums);
    const int stride = static_cast<int>(C) * kFusedWorkers;
    const int slot = warp * static_cast<int>(C) + static_cast<int>(rank);
    __syncthreads();
    FusedCtl& f = sc.f;
    if (decider && lane == 0) fused_snapshot(sc.ctl, f, kFp64);
    cluster_sync_all();
    if (decider) {
        fused_decider<kLimits>(cp, inf.n, kFp64, max_trials, sc, sums, range, C, rank);
        return;
    }
    auto publish = [&](double* at, double v) {
        if (static_cast<uint32_t>(lane) < C) st_cluster(rank_addr(at, static_cast<uint32_t>(lane)), v);
    };
    for (int t = 0; t < max_trials && f.active; ++t) {
        double* const sums_p = sums.p[t & 1];
        for (int s = range.ps0 + slot; s < range.ps1; s += stride) {
            const CtaWork one{b, s, s + 1, 0};
            double v[1] = {fused_primal<T, V>(g, w, one, inf, f, lane)};
            warp_sum<1>(v);
            publish(sums_p + (s - range.ps0), v[0]);
        }
        trial_sync(C);
        for (int s = range.ds0 + slot; s < range.ds1; s += stride) {
            const CtaWork one{b, s, s + 1, 0};
            double r2[2] = {0.0, 0.0};
            fused_dual<T, V>(g, w, one, inf, f, lane, r2);
            warp_sum<2>(r2);
            publish(sums.d + 2 * (s - range.ds0), r2[0]);
            publish(sums.d + 2 * (s - range.ds0) + 1, r2[1]);
        }
        trial_sync(C);
        cta_sync_all();
        if (f.slow) {
            cluster_sync_all();
            cta_sync_all();
        }
    }
    cluster_sync_all();
}
