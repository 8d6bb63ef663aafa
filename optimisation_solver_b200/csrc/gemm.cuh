// gemm.cuh -- the tensor-core building blocks of the learned warm start:
// BF16 operands, FP32 accumulation in TMEM (tcgen05.mma), operands staged by
// TMA (cp.async.bulk.tensor, 128-byte swizzle) through mbarrier rings.
//
//   gemm_tile   one 128-row output tile per CTA; either operand may be stored
//               K-major ([row][K]) or row-major over its rows ([K][row]), so
//               a backward pass needs no transposed copies
//   last_layer  the network's wide last layer: a column tile of the output for
//               every row of the batch, stored, or in a training step straight
//               into the loss, its gradient and the bias update
//   adam_step   the weight gradients of a training step, each tile straight
//               into its weights' Adam step
//   gemm_pair   large plain products: two CTAs share a 256 x 256 tile
//               (cta_group::2), persistent, the epilogue of one tile under
//               the main loop of the next
//
// A dot product is accumulated in K order in steps of 16 by every one of
// them, so the kernel that computes a product does not change its bits.
//
// Every mbarrier wait gives up after two seconds of %globaltimer, records an
// error code and lets the CTA drain its copies, free its TMEM and return, so
// a fault in the pipeline cannot hang the device.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "team_walk.hpp"

namespace pdlpgpu_mlp_impl {

using bf16 = __nv_bfloat16;

constexpr int BM = 128;
constexpr int BK = 64;                       // 64 BF16 = one 128-byte swizzle row
constexpr int64_t kWaitNs = 2000000000LL;

// ---------------------------------------------------------------------------
// PTX helpers
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ int64_t gtimer() {
    int64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Programmatic dependent launch. A kernel lets its successor start only once
// all its CTAs hold their TMEM: a successor's CTA that took the columns
// first would wait for this grid to end while this grid waits for columns.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// One look at a barrier's phase; the thread sleeps in hardware for a while if
// it has not completed. (Polled without that, the waiting epilogue warps took
// issue slots from the one thread that feeds the tensor cores.)
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t phase) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(phase)
        : "memory");
    return ok != 0;
}

// Bounded wait: false (and an error code) after kWaitNs without completion.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t phase, int* err, int code) {
    if (mbar_try(bar, phase)) return true;
    const int64_t t0 = gtimer();
    while (true) {
        if (mbar_try(bar, phase)) return true;
        if (gtimer() - t0 > kWaitNs) {
            atomicExch(err, code);
            return false;
        }
    }
}

// The same for a whole warp: all lanes agree.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t phase, int* err, int code) {
    return __all_sync(0xffffffffu, mbar_wait(bar, phase, err, code)) != 0;
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar,
                                            int32_t x, int32_t y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y)
        : "memory");
}

__device__ __forceinline__ void prefetch_map(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// Shared-memory matrix descriptor, 128-byte swizzle, version 1.
// K-major: 128-byte rows of 64 K, 8-row groups 1024 bytes apart (SBO).
// Row-major over rows (MN-major): 128-byte rows of 64 consecutive tile rows,
// one per K; 8-K groups 1024 bytes apart (SBO), 64-row blocks of the tile
// `mn_block` bytes apart (LBO).
constexpr uint32_t kMnBlock = 64 * BK * 2;   // one 64 (rows) x BK box

template <bool kMn>
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((addr >> 4) & 0x3fff);                  // start address
    d |= static_cast<uint64_t>(kMn ? (kMnBlock >> 4) : 1) << 16;       // leading byte offset
    d |= static_cast<uint64_t>(1024 >> 4) << 32;                       // stride byte offset
    d |= static_cast<uint64_t>(1) << 46;                               // descriptor version
    d |= static_cast<uint64_t>(2) << 61;                               // SWIZZLE_128B
    return d;
}
// Byte step of 16 K inside a stage: along the 128-byte row, or two 8-K groups.
template <bool kMn> constexpr uint32_t kStepK = kMn ? 2048 : 32;

// Instruction descriptor: BF16 x BF16 -> FP32.
constexpr uint32_t instr_desc(int m, int n, bool a_mn, bool b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (a_mn ? 1u << 15 : 0u) | (b_mn ? 1u << 16 : 0u) |
           (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,"
        "%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
          "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
          "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t slot, uint32_t columns) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(columns));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_free(uint32_t tmem, uint32_t columns) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(columns));
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ uint8_t* align1024(uint8_t* p) {
    return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(p) + 1023) & ~uintptr_t(1023));
}

// True in one lane of the (converged) warp. The loading and the multiplying
// warp run their loops with all lanes, so that stages, descriptors and
// coordinates stay in uniform registers, and only the copies, MMAs and
// commits are issued by this lane; in a loop of one lane every operand of an
// MMA crosses to the uniform registers on its own.
__device__ __forceinline__ bool elect_one() {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok));
    return ok != 0;
}

// The ring position of a role: stage index and the parity of its barriers'
// current pass. Counted, not divided: one thread feeds the copies and one the
// tensor cores, and an integer division per K block there is time in which
// nothing is issued (a 128 x 128 tile took 0.37 us a block with two).
template <int S>
struct Ring {
    int s = 0;
    uint32_t phase = 0;
    bool wrapped = false;   // every stage has been used
    __device__ __forceinline__ void next() {
        if (++s == S) {
            s = 0;
            phase ^= 1;
            wrapped = true;
        }
    }
};

// Loads of one operand's part of a stage: rows [r0, r0 + kRows) of K block kb.
template <bool kMn, int kRows>
__device__ __forceinline__ void load_operand(uint32_t dst, const CUtensorMap* map, uint32_t bar, int kb, int r0) {
    if constexpr (kMn) {
#pragma unroll
        for (int q = 0; q < kRows / 64; ++q) tma_load_2d(dst + q * kMnBlock, map, bar, r0 + 64 * q, kb * BK);
    } else {
        tma_load_2d(dst, map, bar, kb * BK, r0);
    }
}

// ---------------------------------------------------------------------------
// Epilogues of gemm_tile. A warp gets one 32 x 32 block of the tile: acc(q)
// gives lane `lane` the four values of row 4 q + lane / 8 from column
// 4 (lane % 8) on, q < 8, so a warp's accesses are 128-byte row pieces.
// ---------------------------------------------------------------------------
// C[z][M][N] = acc: a K split's partial, or the product itself.
struct EpiStore {
    float* C;
    int64_t split_stride;
    __device__ __forceinline__ const float* sums() const { return C; }
    template <class Acc>
    __device__ __forceinline__ void block(int z, int row0, int col0, int M, int N, const Acc& acc) const {
        const int lane = threadIdx.x & 31;
        float* out = C + z * split_stride;
        const int col = col0 + 4 * (lane & 7);
        const bool wide = (N & 3) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int row = row0 + 4 * q + (lane >> 3);
            float v[4];
            acc(q, v);
            float* p = out + static_cast<int64_t>(row) * N + col;
            if (wide) {
                if (row < M && col < N) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
            } else if (row < M) {
                for (int k = 0; k < 4; ++k)
                    if (col + k < N) p[k] = v[k];
            }
        }
    }
};

// Branch-free FP32 quotient and square root with IEEE's rounding, for values
// away from underflow and overflow (Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34,
// 1990): an approximation is refined to a faithful result and one FMA with
// its exact remainder rounds it correctly. The operators compile to code with
// a branch per operation, which keeps the independent elements of a thread
// from overlapping.
__device__ __forceinline__ float quotient(float x, float c, float recip) {   // recip: 1 / c to half an ulp
    const float q = __fmul_rn(x, recip);
    return __fmaf_rn(__fmaf_rn(-q, c, x), recip, q);
}
__device__ __forceinline__ float quotient(float x, float c) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(c));
    y = __fmaf_rn(__fmaf_rn(-c, y, 1.0f), y, y);
    return quotient(x, c, y);
}
__device__ __forceinline__ float root(float a) {   // a > 0
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(a));
    float g = __fmul_rn(a, y), h = __fmul_rn(0.5f, y);
    const float r = __fmaf_rn(-g, h, 0.5f);
    g = __fmaf_rn(g, r, g);
    h = __fmaf_rn(h, r, h);
    return __fmaf_rn(__fmaf_rn(-g, g, a), h, g);
}

// One Adam step (Kingma and Ba, 2015) with bias correction.
struct AdamStep {
    float lr, b1, b2, eps, c1, c2, r1, r2;   // r = 1 / c
    __device__ __forceinline__ void moments(float g, float& m, float& v) const {
        m = __fmaf_rn(1.0f - b1, g, __fmul_rn(b1, m));
        v = __fmaf_rn(__fmul_rn(1.0f - b2, g), g, __fmul_rn(b2, v));
    }
    __device__ __forceinline__ float update(float m, float v) const {
        return lr * (m / c1) / (sqrtf(v / c2) + eps);
    }
    // The same value without a branch; `plain` is false where the
    // remainders could underflow (zeros are exact) and update() is needed.
    __device__ __forceinline__ float update_fast(float m, float v, bool& plain) const {
        const float mm = quotient(m, c1, r1), vv = quotient(v, c2, r2);
        const float s = v > 0.0f ? root(vv) : 0.0f;
        const float x = __fmul_rn(lr, mm);
        plain = plain && (v == 0.0f || (v > 1e-25f && v < 1e25f)) &&
                (m == 0.0f || (fabsf(m) > 1e-25f && fabsf(m) < 1e25f && fabsf(x) > 1e-25f));
        return quotient(x, s + eps);
    }
    __device__ __forceinline__ void operator()(float g, float& p, float& m, float& v) const {
        moments(g, m, v);
        p = p - update(m, v);
    }
    // Four elements, independent of one another.
    __device__ __forceinline__ void operator()(const float (&g)[4], float4& p, float4& m, float4& v) const {
        moments(g[0], m.x, v.x);
        moments(g[1], m.y, v.y);
        moments(g[2], m.z, v.z);
        moments(g[3], m.w, v.w);
        bool plain = true;
        float u[4] = {update_fast(m.x, v.x, plain), update_fast(m.y, v.y, plain), update_fast(m.z, v.z, plain),
                      update_fast(m.w, v.w, plain)};
        if (!plain) {
            u[0] = update(m.x, v.x);
            u[1] = update(m.y, v.y);
            u[2] = update(m.z, v.z);
            u[3] = update(m.w, v.w);
        }
        p.x -= u[0];
        p.y -= u[1];
        p.z -= u[2];
        p.w -= u[3];
    }
};

// ---------------------------------------------------------------------------
// gemm_tile: C tile (128 x kBN) = A rows x B rows over K
// ---------------------------------------------------------------------------
struct TileArgs {
    int M, N, K;
    int kb_per_split;   // K blocks of a split
    int splits;         // splits this CTA runs one after another (gridDim.z runs them side by side)
    int* err;
};

constexpr int kTileThreads = 256;

template <int kBN, int kStages>
constexpr int tile_smem() {
    return kStages * (BM * BK * 2 + kBN * BK * 2) + 1024 /*align*/ + 256 /*barriers*/;
}
// Accumulators of successive splits held side by side in TMEM.
template <int kBN, int kStages>
constexpr int tile_accs() {
    // An SM has 512 columns: two CTAs share it when their rings allow it.
    return tile_smem<kBN, kStages>() > 113 * 1024 ? 512 / kBN : 256 / kBN;
}

// Warp-specialised: warp 0 loads (it refills a stage as soon as the MMAs that
// read it have completed), warp 1 issues the MMAs, each by an elected lane, then
// all eight warps take the accumulator: warp w rows 32 (w % 4).., columns
// kBN / 2 (w / 4)... With several splits per CTA each has its own
// accumulator, and the epilogue adds them in split order; beyond
// tile_accs of them the running sum waits in C (gridDim.z = 1).
template <int kBN, int kStages, bool kAMn, bool kBMn, class Epi>
__device__ __forceinline__ void tile_product(const CUtensorMap& map_a, const CUtensorMap& map_b, const TileArgs& a,
                                             const Epi& epi, int m0, int n0, int z) {
    constexpr uint32_t kABytes = BM * BK * 2, kBBytes = kBN * BK * 2;
    constexpr int kAccs = tile_accs<kBN, kStages>();
    constexpr uint32_t kIdesc = instr_desc(BM, kBN, kAMn, kBMn);
    static_assert(kStages * (kABytes + kBBytes) >= 8 * 32 * 33 * 4, "the drained ring holds the epilogue's blocks");
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = align1024(smem_raw);
    uint8_t* sa = smem;
    uint8_t* sb = smem + kStages * kABytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sb + kStages * kBBytes);
    uint64_t* full = bars;                    // [kStages]
    uint64_t* empty = bars + kStages;         // [kStages]
    uint64_t* done = bars + 2 * kStages;      // [1]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kStages + 1);
    __shared__ int consumed_by_mma;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int total_kb = (a.K + BK - 1) / BK;
    const int z0 = z * a.splits;
    int columns = kBN;                        // TMEM: a power of two of at least 32 columns
    while (columns < kBN * min(a.splits, kAccs)) columns *= 2;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(smem_u32(&full[s]), 1);
            mbar_init(smem_u32(&empty[s]), 1);
        }
        mbar_init(smem_u32(done), 1);
        consumed_by_mma = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        prefetch_map(&map_a);
        prefetch_map(&map_b);
    }
    if (warp == 0) tmem_alloc(smem_u32(tmem_slot), columns);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_trigger();
    pdl_wait();

    const int row0 = m0 + (warp & 3) * 32;
    const int half0 = (warp >> 2) * (kBN / 2);

    bool good = true;
    int base = 0;                             // K blocks done by earlier groups of splits
    Ring<kStages> ring;                       // of the loading or the multiplying thread
    for (int g0 = 0; g0 < a.splits && good; g0 += kAccs) {
        const int g1 = min(a.splits, g0 + kAccs);
        const int kb0 = min(total_kb, (z0 + g0) * a.kb_per_split);
        const int nk = min(total_kb, (z0 + g1) * a.kb_per_split) - kb0;
        int issued = base;
        if (warp == 0 && nk > 0) {
            for (int kb = kb0; kb < kb0 + nk; ++kb, ring.next()) {
                const int s = ring.s;
                if (ring.wrapped && !warp_wait(smem_u32(&empty[s]), ring.phase ^ 1, a.err, 2)) break;
                if (elect_one()) {
                    const uint32_t fb = smem_u32(&full[s]);
                    mbar_expect_tx(fb, kABytes + kBBytes);
                    load_operand<kAMn, BM>(smem_u32(sa + s * kABytes), &map_a, fb, kb, m0);
                    load_operand<kBMn, kBN>(smem_u32(sb + s * kBBytes), &map_b, fb, kb, n0);
                }
                ++issued;
            }
        } else if (warp == 1 && nk > 0) {
            int i = base;
            uint32_t acc = tmem;              // the split's accumulator
            int left = a.kb_per_split;        // of the split
            uint32_t more = 0;                // accumulate onto what is there
            for (; i < base + nk; ++i, ring.next()) {
                const int s = ring.s;
                if (!warp_wait(smem_u32(&full[s]), ring.phase, a.err, 1)) break;
                tc_fence_after();
                const uint64_t da = smem_desc<kAMn>(smem_u32(sa + s * kABytes));
                const uint64_t db = smem_desc<kBMn>(smem_u32(sb + s * kBBytes));
                if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < BK / 16; ++kk)
                        mma_bf16(acc, da + kk * (kStepK<kAMn> >> 4), db + kk * (kStepK<kBMn> >> 4), kIdesc,
                                 kk > 0 ? 1u : more);
                    mma_commit(smem_u32(&empty[s]));
                }
                more = 1;
                if (--left == 0) {
                    left = a.kb_per_split;
                    acc += kBN;
                    more = 0;
                }
            }
            // Arrives once every MMA issued above has completed (by the lane
            // that issued them: elect.sync picks the same one every time).
            if (elect_one()) {
                consumed_by_mma = i;
                mma_commit(smem_u32(done));
            }
            __syncwarp();
        }
        __syncthreads();
        // After an error, copies the MMA warp never consumed may still be in
        // flight: the producer waits for them (bounded) before the stage
        // memory is reused below.
        if (warp == 0 && lane == 0)
            for (int i = consumed_by_mma; i < issued; ++i)
                mbar_wait(smem_u32(&full[i % kStages]), (i / kStages) & 1, a.err, 3);
        bool have = nk > 0;
        if (have) have = mbar_wait(smem_u32(done), (g0 / kAccs) & 1, a.err, 4);
        if (nk > 0) good = __syncthreads_and(have) != 0;
        else __syncthreads();
        tc_fence_after();

        // Each 32 x 32 block goes through shared memory (the drained ring).
        float* tile = reinterpret_cast<float*>(sa) + warp * 32 * 33;
        const int accs = nk > 0 ? (nk + a.kb_per_split - 1) / a.kb_per_split : 0;
#pragma unroll 1
        for (int c0 = half0; c0 < half0 + kBN / 2; c0 += 32) {
            float sum[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) sum[j] = 0.0f;
            if (g0 > 0) {   // the earlier groups' sum, which this warp stored
                const float* prior = epi.sums() + static_cast<int64_t>(row0 + lane) * a.N + n0 + c0;
                if (row0 + lane < a.M)
                    for (int j = 0; j < 32; ++j)
                        if (n0 + c0 + j < a.N) sum[j] = prior[j];
                __syncwarp();
            }
            for (int q = 0; q < accs; ++q) {
                uint32_t r[32];
                tmem_ld32(tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + q * kBN + c0, r);
#pragma unroll
                for (int j = 0; j < 32; ++j) sum[j] = have ? sum[j] + __uint_as_float(r[j]) : 0.0f;
            }
#pragma unroll
            for (int j = 0; j < 32; ++j) tile[lane * 33 + j] = sum[j];
            __syncwarp();
            epi.block(z, row0, n0 + c0, a.M, a.N, [&](int q, float (&v)[4]) {
                const float* t = tile + (4 * q + (lane >> 3)) * 33 + 4 * (lane & 7);
#pragma unroll
                for (int k = 0; k < 4; ++k) v[k] = t[k];
            });
            __syncwarp();
        }
        // The next group's copies reuse the memory the blocks went through.
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        base += nk;
    }
    __syncthreads();
    if (warp == 0) tmem_free(tmem, columns);
}

// The tile of CTA `pid` of tiles_m x tiles_n in grouped order: consecutive
// CTAs sweep 16 row tiles for each column tile, so the CTAs in flight share
// their A and B panels in L2.
__device__ __forceinline__ void tile_origin(int pid, int tiles_m, int tiles_n, int bn, int& m0, int& n0) {
    constexpr int kGroupM = 16;
    const int per_group = kGroupM * tiles_n;
    const int first_m = (pid / per_group) * kGroupM;
    const int group_m = min(tiles_m - first_m, kGroupM);
    m0 = (first_m + (pid % per_group) % group_m) * BM;
    n0 = ((pid % per_group) / group_m) * bn;
}

template <int kBN, int kStages, bool kAMn, bool kBMn, class Epi>
__global__ void __launch_bounds__(kTileThreads, tile_smem<kBN, kStages>() > 113 * 1024 ? 1 : 2)
gemm_tile(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, TileArgs a,
          Epi epi) {
    int m0, n0;
    tile_origin(static_cast<int>(blockIdx.x + blockIdx.y * gridDim.x), static_cast<int>(gridDim.x),
                static_cast<int>(gridDim.y), kBN, m0, n0);
    tile_product<kBN, kStages, kAMn, kBMn>(map_a, map_b, a, epi, m0, n0, static_cast<int>(blockIdx.z));
}

// ---------------------------------------------------------------------------
// adam_step: the rest of a training step in one launch -- the three weight
// gradients' products, each ending in Adam, and the hidden biases' sums and
// Adam steps. Bound by HBM: weights and moments read and written, 26 bytes a
// weight.
// ---------------------------------------------------------------------------
// The hidden biases: db[j] = sum_b dZ[b][j], rows in order, then stored
// (gradient mode) or Adam; and the loss, its CTAs' sums added in a fixed
// order over the batch.
struct BiasArgs {
    const float* dz[2];
    float *b[2], *m[2], *v[2];
    float* gb[2];
    int B, H;
    int gradient;
    AdamStep adam;
    const double* loss_part;
    int loss_ctas;
    float* loss;
};
// Warps of bias_and_loss: one for the loss, one per 32 hidden columns.
inline __host__ __device__ int bias_warps(int H) { return 1 + 2 * H / 32; }

__device__ __forceinline__ void bias_and_loss_warp(const BiasArgs& a, int job) {
    const int lane = threadIdx.x & 31;
    if (job == 0) {
        double l = 0.0;
        for (int k = lane; k < a.loss_ctas; k += 32) l += a.loss_part[k];
        for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
        if (lane == 0) *a.loss = static_cast<float>(l / a.B);
        return;
    }
    const int col = (job - 1) * 32 + lane;   // H is a multiple of 64
    const int layer = col / a.H, j = col - layer * a.H;
    const float* d = a.dz[layer] + j;
    float s = 0.0f;
    int b = 0;
    for (; b + 32 <= a.B; b += 32) {
        float r[32];
#pragma unroll
        for (int u = 0; u < 32; ++u) r[u] = d[static_cast<int64_t>(b + u) * a.H];
#pragma unroll
        for (int u = 0; u < 32; ++u) s += r[u];
    }
    for (; b < a.B; ++b) s += d[static_cast<int64_t>(b) * a.H];
    if (a.gradient) {
        if (a.gb[layer] != nullptr) a.gb[layer][j] = s;
        return;
    }
    float p = a.b[layer][j], m = a.m[layer][j], v = a.v[layer][j];
    a.adam(s, p, m, v);
    a.b[layer][j] = p;
    a.m[layer][j] = m;
    a.v[layer][j] = v;
}

struct AdamLayer {
    CUtensorMap d, a;           // D [batch][rows], A [batch][cols]: dW = D^T A
    CUtensorMap p, m, v;        // FP32 [rows][cols], boxes of 128 x 32, 128-byte swizzle
    CUtensorMap h;              // BF16 copy, boxes of 128 x 32, 64-byte swizzle
    int rows, cols;
    int tiles_n, tiles;         // of 128 x kAdamBN
};
struct AdamArgs {
    AdamLayer layer[3];
    AdamStep adam;
    BiasArgs bias;
    int K;                      // batch
    int tiles;
    int* err;
};

// Persistent: one CTA per SM walks the tiles of all three layers. The
// optimiser's state moves in chunks of 128 x 32 (16 KB each of p, m and v)
// by TMA through three slots of shared memory, each served by a team of eight
// epilogue warps that updates it in place. Warp 0 loads the operands, warp 1
// multiplies (two accumulators), warp 2 loads the chunks. In the epilogue
// lane = row, so the gradient stays in the registers tcgen05.ld put it in,
// and the swizzle keeps a warp's 32 rows of 128 bytes off each other's banks.
// Bound by HBM: 22.8M weights (22,000 x 512 x 22,016) take 124 us, 586 MB at
// 4.7 TB/s. With the state read and written through registers by a 128 x 128
// product's epilogue (16 warps an SM, half a block ahead) the same work took
// 190 us, 185 of them without arithmetic; with one team of warps 139; with
// 16-column chunks in six slots 147. The products, the copy of the gradient
// and the separate Adam kernels took about 240.
constexpr int kAdamBN = 64;
constexpr int kAdamStages = 2;
constexpr int kAdamSlots = 3;
constexpr int kAdamTeams = kAdamSlots;                    // of eight warps, a slot each
constexpr int kAdamThreads = 128 + kAdamTeams * 256;
constexpr uint32_t kAdamABytes = BM * BK * 2, kAdamBBytes = kAdamBN * BK * 2;
constexpr uint32_t kChunkBytes = BM * 32 * 4;             // of p, m or v
constexpr uint32_t kSlotBytes = 3 * kChunkBytes + BM * 32 * 2;
constexpr int kAdamSmem = kAdamStages * (kAdamABytes + kAdamBBytes) + kAdamSlots * kSlotBytes + 1024 + 256;

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, uint32_t src, int32_t x, int32_t y) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                     reinterpret_cast<uint64_t>(map)),
                 "r"(src), "r"(x), "r"(y)
                 : "memory");
}

// After a failed wait: time for copies in flight to land before the CTA ends.
__device__ __forceinline__ void drain_pause() {
    const int64_t t0 = gtimer();
    while (gtimer() - t0 < 10000000LL) {
    }
}

// Whether a wait succeeded in all 256 threads of an epilogue team, which
// leave together if one did not (they share barriers).
__device__ __forceinline__ bool all_good(bool good, int barrier) {
    uint32_t all;
    __syncwarp();
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "barrier.cta.red.and.pred q, %2, 256, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(all)
        : "r"(good ? 1u : 0u), "r"(barrier)
        : "memory");
    return all != 0;
}

__global__ void __launch_bounds__(kAdamThreads, 1) adam_step(const __grid_constant__ AdamArgs a) {
    constexpr uint32_t kIdesc = instr_desc(BM, kAdamBN, true, true);
    constexpr int S = kAdamStages;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = align1024(smem_raw);
    uint8_t* slots = smem;                                        // every part 1024-byte aligned
    uint8_t* sa = smem + kAdamSlots * kSlotBytes;
    uint8_t* sb = sa + S * kAdamABytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sb + S * kAdamBBytes);
    uint64_t *full = bars, *empty = bars + S, *acc_full = bars + 2 * S, *acc_empty = bars + 2 * S + 2;
    uint64_t *slot_full = bars + 2 * S + 4, *slot_empty = slot_full + kAdamSlots;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(slot_empty + kAdamSlots);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kbs = (a.K + BK - 1) / BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(smem_u32(&full[s]), 1);
            mbar_init(smem_u32(&empty[s]), 1);
        }
        for (int q = 0; q < 2; ++q) {
            mbar_init(smem_u32(&acc_full[q]), 1);
            mbar_init(smem_u32(&acc_empty[q]), kAdamTeams * 8);
        }
        for (int s = 0; s < kAdamSlots; ++s) {
            mbar_init(smem_u32(&slot_full[s]), 1);
            mbar_init(smem_u32(&slot_empty[s]), 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 3) tmem_alloc(smem_u32(tmem_slot), 2 * kAdamBN);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_trigger();
    pdl_wait();

    // Tile t of the call: its layer and origin. Columns run fastest, so the
    // CTAs in flight sweep whole rows of the state.
    auto locate = [&](int t, int& m0, int& n0) -> const AdamLayer& {
        int l = 0;
        while (t >= a.layer[l].tiles) t -= a.layer[l++].tiles;
        const AdamLayer& L = a.layer[l];
        m0 = t / L.tiles_n * BM;
        n0 = t % L.tiles_n * kAdamBN;
        return L;
    };
    const int step = static_cast<int>(gridDim.x);
    bool good = true;
    if (warp == 0) {
        Ring<S> ring;
        for (int t = blockIdx.x; t < a.tiles && good; t += step) {
            int m0, n0;
            const AdamLayer& L = locate(t, m0, n0);
            for (int kb = 0; kb < kbs; ++kb, ring.next()) {
                const int s = ring.s;
                if (ring.wrapped && !warp_wait(smem_u32(&empty[s]), ring.phase ^ 1, a.err, 2)) {
                    good = false;
                    break;
                }
                if (elect_one()) {
                    const uint32_t fb = smem_u32(&full[s]);
                    mbar_expect_tx(fb, kAdamABytes + kAdamBBytes);
                    load_operand<true, BM>(smem_u32(sa + s * kAdamABytes), &L.d, fb, kb, m0);
                    load_operand<true, kAdamBN>(smem_u32(sb + s * kAdamBBytes), &L.a, fb, kb, n0);
                }
            }
        }
    } else if (warp == 1) {
        int n = 0;
        Ring<S> ring;
        for (int t = blockIdx.x; t < a.tiles && good; t += step, ++n) {
            const int q = n & 1;
            if (n >= 2 && !warp_wait(smem_u32(&acc_empty[q]), ((n / 2) - 1) & 1, a.err, 5)) {
                good = false;
                break;
            }
            tc_fence_after();
            for (int kb = 0; kb < kbs; ++kb, ring.next()) {
                const int s = ring.s;
                if (!warp_wait(smem_u32(&full[s]), ring.phase, a.err, 1)) {
                    good = false;
                    break;
                }
                tc_fence_after();
                const uint64_t da = smem_desc<true>(smem_u32(sa + s * kAdamABytes));
                const uint64_t db = smem_desc<true>(smem_u32(sb + s * kAdamBBytes));
                if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < BK / 16; ++kk)
                        mma_bf16(tmem + q * kAdamBN, da + kk * (kStepK<true> >> 4), db + kk * (kStepK<true> >> 4), kIdesc,
                                 (kb > 0 || kk > 0) ? 1u : 0u);
                    mma_commit(smem_u32(&empty[s]));
                }
            }
            if (elect_one()) mma_commit(smem_u32(&acc_full[q]));
            __syncwarp();
        }
    } else if (warp == 2) {
        if (lane == 0) {
            int n = 0;
            for (int t = blockIdx.x; t < a.tiles && good; t += step) {
                int m0, n0;
                const AdamLayer& L = locate(t, m0, n0);
                for (int c = 0; c < kAdamBN && n0 + c < L.cols; c += 32, ++n) {
                    const int s = n % kAdamSlots;
                    if (n >= kAdamSlots && !mbar_wait(smem_u32(&slot_empty[s]), ((n / kAdamSlots) - 1) & 1, a.err, 6)) {
                        good = false;
                        break;
                    }
                    const uint32_t fb = smem_u32(&slot_full[s]), at = smem_u32(slots + s * kSlotBytes);
                    mbar_expect_tx(fb, 3 * kChunkBytes);
                    tma_load_2d(at, &L.p, fb, n0 + c, m0);
                    tma_load_2d(at + kChunkBytes, &L.m, fb, n0 + c, m0);
                    tma_load_2d(at + 2 * kChunkBytes, &L.v, fb, n0 + c, m0);
                }
            }
        }
    } else if (warp >= 4) {
        // Team t takes the chunks n = t, t + 3, ... through slot t, so one
        // team's arithmetic runs beside the others' waits.
        const int team = (warp - 4) >> 3;
        const int quad = warp & 3, part = (warp >> 2) & 1;   // rows 32 quad .., columns 16 part .. of a chunk
        const int row = quad * 32 + lane;
        uint8_t* const at = slots + team * kSlotBytes;
        // The biases' warps sit in the last CTAs, which have the fewest tiles.
        const int job = (static_cast<int>(gridDim.x) - 1 - static_cast<int>(blockIdx.x)) * 8 * kAdamTeams + (warp - 4);
        for (int b = job; b < bias_warps(a.bias.H); b += 8 * kAdamTeams * step) bias_and_loss_warp(a.bias, b);
        int m0 = 0, n0 = 0;
        const AdamLayer* L = nullptr;
        auto chunks = [&](int t) {
            L = &locate(t, m0, n0);
            return min(kAdamBN, L->cols - n0 + 31) / 32;
        };
        auto wait_tile = [&](int k) { return mbar_wait(smem_u32(&acc_full[k & 1]), (k / 2) & 1, a.err, 4); };
        auto wait_chunk = [&](int i) { return mbar_wait(smem_u32(&slot_full[team]), i & 1, a.err, 7); };
        auto agree = [&](bool ok) { return all_good(ok, 1 + team); };
        auto work = [&](int k, int chunk) {
            const int q = k & 1, c = 32 * chunk;
            tc_fence_after();
            uint32_t g[16];
            tmem_ld16(tmem + (static_cast<uint32_t>(quad * 32) << 16) + q * kAdamBN + c + 16 * part, g);
            uint32_t h[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int off = row * 128 + (((4 * part + j) ^ (row & 7)) << 4);
                float4* pp = reinterpret_cast<float4*>(at + off);
                float4* pm = reinterpret_cast<float4*>(at + kChunkBytes + off);
                float4* pv = reinterpret_cast<float4*>(at + 2 * kChunkBytes + off);
                float4 p = *pp, m = *pm, v = *pv;
                const float gj[4] = {__uint_as_float(g[4 * j]), __uint_as_float(g[4 * j + 1]),
                                     __uint_as_float(g[4 * j + 2]), __uint_as_float(g[4 * j + 3])};
                a.adam(gj, p, m, v);
                *pp = p;
                *pm = m;
                *pv = v;
                h[2 * j] = static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(p.x))) |
                           (static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(p.y))) << 16);
                h[2 * j + 1] = static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(p.z))) |
                               (static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(p.w))) << 16);
            }
            uint8_t* ph = at + 3 * kChunkBytes + row * 64;
#pragma unroll
            for (int j = 0; j < 2; ++j)
                *reinterpret_cast<uint4*>(ph + (((2 * part + j) ^ ((row >> 1) & 3)) << 4)) =
                    make_uint4(h[4 * j], h[4 * j + 1], h[4 * j + 2], h[4 * j + 3]);
            // The chunk goes out as the eight warps leave it, and the
            // slot is free once the store has read it.
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            asm volatile("bar.sync %0, 256;" ::"r"(1 + kAdamTeams + team) : "memory");
            if (quad == 0 && part == 0 && lane == 0) {
                const uint32_t src = smem_u32(at);
                tma_store_2d(&L->p, src, n0 + c, m0);
                tma_store_2d(&L->m, src + kChunkBytes, n0 + c, m0);
                tma_store_2d(&L->v, src + 2 * kChunkBytes, n0 + c, m0);
                tma_store_2d(&L->h, src + 3 * kChunkBytes, n0 + c, m0);
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                mbar_arrive(smem_u32(&slot_empty[team]));
            }
            __syncwarp();
        };
        // Every team is done with the tile's accumulator.
        auto leave = [&](int k) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&acc_empty[k & 1]));
        };
        good = team_walk(static_cast<int>(blockIdx.x), step, a.tiles, team, kAdamTeams, chunks, wait_tile, wait_chunk,
                         agree, work, leave);
        if (quad == 0 && part == 0 && lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    if (!good) drain_pause();
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 3) tmem_free(tmem, 2 * kAdamBN);
}

// ---------------------------------------------------------------------------
// last_layer: out = H W^T + bias over one tile of `bn` columns and all rows,
// 128 at a time. A forward pass stores it; a training step goes on to
//   e = out - target,  loss += w e^2,
//   d = 2 w e / batch (BF16 to memory),  db += d over the rows in order
// stores db or takes the bias's Adam step, and never stores the output.
// The layer is wide and its K short, so a CTA per SM takes one tile of about
// a 148th of the columns (22,016: 160) in a single wave: with 64-column
// tiles three CTAs an SM shared two-stage rings and the step took 35 us,
// with 128 x 128 tiles the forward pass ran 344 CTAs over 296 places.
// Warp 0 loads, warp 1 multiplies (two sets of accumulators while TMEM has
// room, so a row tile's products run under the previous one's epilogue);
// two teams of four epilogue warps take the 32-column blocks in turn.
// In a forward pass the row tiles may be dealt over gridDim.y CTAs (a batch of
// many rows and few columns); a training step adds the bias gradient over all
// rows in order and has one.
// ---------------------------------------------------------------------------
struct LastArgs {
    int M, N, K, bn;
    int kb_per_split, splits; // K splits, added in order (splits * bn <= 512)
    float* out;               // forward
    const float *target, *weight;
    float* bias;
    bf16* d;
    double* loss_part;        // [gridDim.x]
    float* gb;                // gradient mode: the bias gradient; else
    float *mb, *vb;           // the bias's Adam moments
    AdamStep adam;
    int* err;
};

constexpr int kLastStages = 4;
constexpr int kLastThreads = 384;
constexpr int kLastTmem = 512;                  // columns
inline int last_smem(int bn) { return kLastStages * (BM + bn) * BK * 2 + 2 * BM * 33 * 4 + 1024 + 256; }

template <bool kTrain>
__global__ void __launch_bounds__(kLastThreads, 1)
last_layer(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
           const __grid_constant__ LastArgs a) {
    constexpr uint32_t kABytes = BM * BK * 2;
    constexpr int S = kLastStages;
    const uint32_t b_bytes = static_cast<uint32_t>(a.bn) * BK * 2;   // a multiple of 4 KiB
    const uint32_t idesc = instr_desc(BM, a.bn, false, false);
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = align1024(smem_raw);
    uint8_t* sa = smem;
    uint8_t* sb = smem + S * kABytes;
    float* tiles = reinterpret_cast<float*>(sb + S * b_bytes);   // [team][128][33]
    uint64_t* bars = reinterpret_cast<uint64_t*>(tiles + 2 * BM * 33);
    uint64_t *full = bars, *empty = bars + S, *acc_full = bars + 2 * S, *acc_empty = bars + 2 * S + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * S + 4);
    __shared__ double part[8];
    __shared__ int consumed_by_mma;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = static_cast<int>(blockIdx.x) * a.bn;
    const int kbs = (a.K + BK - 1) / BK, mts = (a.M + BM - 1) / BM;
    const int sets = 2 * a.splits * a.bn <= kLastTmem ? 2 : 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(smem_u32(&full[s]), 1);
            mbar_init(smem_u32(&empty[s]), 1);
        }
        for (int q = 0; q < 2; ++q) {
            mbar_init(smem_u32(&acc_full[q]), 1);
            mbar_init(smem_u32(&acc_empty[q]), 8);
        }
        consumed_by_mma = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        prefetch_map(&map_a);
        prefetch_map(&map_b);
    }
    if (warp == 2) tmem_alloc(smem_u32(tmem_slot), kLastTmem);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_trigger();
    pdl_wait();

    int issued = 0;
    if (warp == 0) {
        Ring<S> ring;
        bool good = true;
        for (int mt = blockIdx.y; mt < mts && good; mt += gridDim.y)
            for (int kb = 0; kb < kbs; ++kb, ring.next()) {
                const int s = ring.s;
                if (ring.wrapped && !warp_wait(smem_u32(&empty[s]), ring.phase ^ 1, a.err, 2)) {
                    good = false;
                    break;
                }
                if (elect_one()) {
                    const uint32_t fb = smem_u32(&full[s]);
                    mbar_expect_tx(fb, kABytes + b_bytes);
                    tma_load_2d(smem_u32(sa + s * kABytes), &map_a, fb, kb * BK, mt * BM);
                    tma_load_2d(smem_u32(sb + s * b_bytes), &map_b, fb, kb * BK, n0);
                }
                ++issued;
            }
    } else if (warp == 1) {
        int i = 0;
        Ring<S> ring;
        bool good = true;
        for (int mt = blockIdx.y, t = 0; mt < mts && good; mt += gridDim.y, ++t) {
            const int q = sets == 2 ? t & 1 : 0;
            if (t >= sets && !warp_wait(smem_u32(&acc_empty[q]), ((sets == 2 ? t >> 1 : t) - 1) & 1, a.err, 5)) break;
            tc_fence_after();
            uint32_t acc = tmem + static_cast<uint32_t>(q * a.splits * a.bn), more = 0;
            int left = a.kb_per_split;
            for (int kb = 0; kb < kbs; ++kb, ++i, ring.next()) {
                const int s = ring.s;
                if (!warp_wait(smem_u32(&full[s]), ring.phase, a.err, 1)) {
                    good = false;
                    break;
                }
                tc_fence_after();
                const uint64_t da = smem_desc<false>(smem_u32(sa + s * kABytes));
                const uint64_t db = smem_desc<false>(smem_u32(sb + s * b_bytes));
                if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < BK / 16; ++kk)
                        mma_bf16(acc, da + kk * 2, db + kk * 2, idesc, kk > 0 ? 1u : more);
                    mma_commit(smem_u32(&empty[s]));
                }
                more = 1;
                if (--left == 0) {
                    left = a.kb_per_split;
                    acc += a.bn;
                    more = 0;
                }
            }
            if (elect_one()) mma_commit(smem_u32(&acc_full[q]));
            __syncwarp();
        }
        if (lane == 0) consumed_by_mma = i;
    } else if (warp >= 4) {
        const int quad = warp & 3, team = (warp - 4) >> 2;   // TMEM lanes 32 quad ..
        const int rr = lane >> 3, cc = 4 * (lane & 7);
        const int blocks = min(a.bn, a.N - n0) / 32;         // N and bn are multiples of 32
        float* tile = tiles + team * BM * 33;
        float* mine = tile + quad * 32 * 33;
        auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
        const bool wide = kTrain ? aligned(a.target) && aligned(a.weight) : aligned(a.out);
        const float batch = static_cast<float>(a.M);
        // A power of two divides exactly, so its reciprocal gives the same bits.
        const bool pow2 = (a.M & (a.M - 1)) == 0;
        const float inv_batch = 1.0f / batch;
        float loss[4] = {};
        float csum = 0.0f;     // block `team + 2 quad` of the tile, a lane per column
        // The targets of a block (128 rows x 32 columns), loaded one block ahead.
        float4 t[8] = {};
        auto load_targets = [&](int mt, int b) {
            if constexpr (kTrain) {
                const int m0 = mt * BM + quad * 32, col = n0 + 32 * b + cc;
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    const int row = m0 + 4 * r + rr;
                    if (row >= a.M) continue;
                    const float* p = a.target + static_cast<int64_t>(row) * a.N + col;
                    if (wide) t[r] = __ldcs(reinterpret_cast<const float4*>(p));
                    else t[r] = make_float4(p[0], p[1], p[2], p[3]);
                }
            }
        };
        if (team < blocks) load_targets(0, team);
        for (int mt = blockIdx.y, u = 0; mt < mts; mt += gridDim.y, ++u) {
            const int m0 = mt * BM, q = sets == 2 ? u & 1 : 0;
            const bool have = mbar_wait(smem_u32(&acc_full[q]), (sets == 2 ? u >> 1 : u) & 1, a.err, 4);
            tc_fence_after();
            __syncwarp();
            for (int b = team; b < blocks; b += 2) {
                const int col = n0 + 32 * b + cc;
                for (int z = 0; z < a.splits; ++z) {
                    uint32_t r[32];
                    tmem_ld32(tmem + (static_cast<uint32_t>(quad * 32) << 16) + (q * a.splits + z) * a.bn + 32 * b, r);
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const float v = have ? __uint_as_float(r[j]) : 0.0f;
                        mine[lane * 33 + j] = z == 0 ? v : mine[lane * 33 + j] + v;
                    }
                }
                __syncwarp();
                const float4 b4 = *reinterpret_cast<const float4*>(a.bias + col);
                const float bv[4] = {b4.x, b4.y, b4.z, b4.w};
                if constexpr (!kTrain) {
#pragma unroll
                    for (int r = 0; r < 8; ++r) {
                        const int row = m0 + quad * 32 + 4 * r + rr;
                        const float* p = mine + (4 * r + rr) * 33 + cc;
                        const float v[4] = {p[0] + bv[0], p[1] + bv[1], p[2] + bv[2], p[3] + bv[3]};
                        float* o = a.out + static_cast<int64_t>(row) * a.N + col;
                        if (row < a.M) {
                            if (wide) *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
                            else for (int k = 0; k < 4; ++k) o[k] = v[k];
                        }
                    }
                    __syncwarp();
                } else {
                    float4 w4;
                    if (wide) w4 = *reinterpret_cast<const float4*>(a.weight + col);
                    else w4 = make_float4(a.weight[col], a.weight[col + 1], a.weight[col + 2], a.weight[col + 3]);
                    const float wv[4] = {w4.x, w4.y, w4.z, w4.w};
                    // Every value is read before the first is written back,
                    // so the elements overlap.
                    float g[8][4];
#pragma unroll
                    for (int r = 0; r < 8; ++r)
#pragma unroll
                        for (int k = 0; k < 4; ++k) g[r][k] = mine[(4 * r + rr) * 33 + cc + k];
                    auto elements = [&](auto over_batch) {
#pragma unroll
                        for (int r = 0; r < 8; ++r) {
                            const bool valid = m0 + quad * 32 + 4 * r + rr < a.M;
                            const float tv[4] = {t[r].x, t[r].y, t[r].z, t[r].w};
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                const float e = (g[r][k] + bv[k]) - tv[k];
                                const float l = wv[k] * e * e;
                                loss[k] += valid ? l : 0.0f;
                                g[r][k] = over_batch(2.0f * wv[k] * e);
                            }
                        }
                    };
                    if (pow2) elements([&](float x) { return x * inv_batch; });
                    else elements([&](float x) { return x / batch; });
#pragma unroll
                    for (int r = 0; r < 8; ++r) {
                        const int row = m0 + quad * 32 + 4 * r + rr;
#pragma unroll
                        for (int k = 0; k < 4; ++k) mine[(4 * r + rr) * 33 + cc + k] = g[r][k];
                        uint2 u;
                        u.x = static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(g[r][0]))) |
                              (static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(g[r][1]))) << 16);
                        u.y = static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(g[r][2]))) |
                              (static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(g[r][3]))) << 16);
                        if (row < a.M) *reinterpret_cast<uint2*>(a.d + static_cast<int64_t>(row) * a.N + col) = u;
                    }
                    if (b + 2 < blocks) load_targets(mt, b + 2);
                    else if (mt + 1 < mts) load_targets(mt + 1, team);
                    // Column sums over the rows in order: one of the team's
                    // warps, a lane per column, between two barriers.
                    __syncwarp();
                    asm volatile("bar.sync %0, 128;" ::"r"(1 + team) : "memory");
                    if (quad == (b >> 1)) {
                        const int rows = min(BM, a.M - m0);
                        float s = csum;
#pragma unroll 16
                        for (int r = 0; r < rows; ++r) s += tile[r * 33 + lane];
                        csum = s;
                    }
                    __syncwarp();
                    asm volatile("bar.sync %0, 128;" ::"r"(1 + team) : "memory");
                }
            }
            // The accumulators are read out.
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&acc_empty[q]));
        }
        if constexpr (kTrain) {
            const int b = team + 2 * quad;
            if (b < blocks) {
                const int j = n0 + 32 * b + lane;
                if (a.gb != nullptr) {
                    a.gb[j] = csum;
                } else {
                    float p = a.bias[j], m = a.mb[j], v = a.vb[j];
                    a.adam(csum, p, m, v);
                    a.bias[j] = p;
                    a.mb[j] = m;
                    a.vb[j] = v;
                }
            }
            double l = static_cast<double>(loss[0]) + loss[1] + loss[2] + loss[3];
            for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
            if (lane == 0) part[warp - 4] = l;
        }
    }
    __syncthreads();
    if (warp == 0 && lane == 0) {
        for (int i = consumed_by_mma; i < issued; ++i)
            mbar_wait(smem_u32(&full[i % S]), (i / S) & 1, a.err, 3);
        if constexpr (kTrain) {
            double l = 0.0;
            for (int k = 0; k < 8; ++k) l += part[k];
            a.loss_part[blockIdx.x] = l;
        }
    }
    __syncthreads();
    if (warp == 2) tmem_free(tmem, kLastTmem);
}

// ---------------------------------------------------------------------------
// gemm_pair: C[M][N] = A[M][K] B[N][K]^T for products of many tiles. The two
// CTAs of a cluster sit on neighbouring SMs and share a 256 x 256 tile:
// cta_group::2 MMAs (M = 256, N = 256) read both CTAs' shared memory, each
// CTA loading only its own 128 rows of A and of B, and leave 128 rows of the
// tile in each CTA's TMEM. Half the operand bytes per product of a 128 x 128
// tile, which is what the single-CTA kernel is bound by. Persistent: the 512
// TMEM columns hold two accumulators, so a tile's epilogue (warps 4-7 of both
// CTAs) runs under the next tile's main loop. Bound by the copies into shared
// memory, 32 KB an SM and K block (about 80 bytes a cycle), and at 8192^3 by
// power: 720 to 742 us, 1482 to 1527 TFLOP/s, 0.89 to 0.92 of the measured dense
// BF16 peak; the 128 x 128 tiles of one CTA took 931 us there.
// ---------------------------------------------------------------------------
constexpr int kPairStages = 6;
constexpr int kPairThreads = 256;
constexpr int kPairSmem = kPairStages * 2 * (BM * BK * 2) + 4 * 32 * 33 * 4 + 1024 + 256;

struct PairArgs {
    int M, N, K;
    float* C;
    int* err;
};

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

// `bar` in the shared::cluster window: of either CTA.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar, int32_t x,
                                                 int32_t y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void mma_bf16_pair(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc,
                                              uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}
// Arrives on the barrier at this offset in both CTAs once the MMAs issued so
// far have completed.
__device__ __forceinline__ void mma_commit_pair(uint32_t bar) {
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
        "h"(static_cast<uint16_t>(3))
        : "memory");
}
__device__ __forceinline__ void mbar_arrive_rank0(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(map_rank(bar, 0)) : "memory");
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
gemm_pair(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, PairArgs a) {
    constexpr uint32_t kBytes = BM * BK * 2;   // 128 rows of either operand
    constexpr uint32_t kIdesc = instr_desc(256, 256, false, false);
    constexpr int S = kPairStages;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = align1024(smem_raw);
    uint8_t* sa = smem;
    uint8_t* sb = smem + S * kBytes;
    float* blocks = reinterpret_cast<float*>(sb + S * kBytes);   // [4][32][33]
    uint64_t* bars = reinterpret_cast<uint64_t*>(blocks + 4 * 32 * 33);
    uint64_t *full = bars, *empty = bars + S, *acc_full = bars + 2 * S, *acc_empty = bars + 2 * S + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * S + 4);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int pair = static_cast<int>(blockIdx.x) >> 1, pairs = static_cast<int>(gridDim.x) >> 1;
    const int tiles_m = (a.M + 255) / 256, tiles_n = (a.N + 255) / 256, tiles = tiles_m * tiles_n;
    const int total_kb = (a.K + BK - 1) / BK;
    // Grouped order: the tiles in flight share their A and B panels in L2.
    constexpr int kGroupM = 8;
    auto origin = [&](int t, int& m0, int& n0) {
        const int per_group = kGroupM * tiles_n, first = (t / per_group) * kGroupM;
        const int in = t % per_group, height = min(tiles_m - first, kGroupM);
        m0 = (first + in % height) * 256;
        n0 = (in / height) * 256;
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(smem_u32(&full[s]), 1);
            mbar_init(smem_u32(&empty[s]), 1);
        }
        for (int q = 0; q < 2; ++q) {
            mbar_init(smem_u32(&acc_full[q]), 1);
            mbar_init(smem_u32(&acc_empty[q]), 8);   // four epilogue warps in either CTA
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        prefetch_map(&map_a);
        prefetch_map(&map_b);
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();   // the peer's barriers and TMEM are ready
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        Ring<S> ring;
        bool good = true;
        for (int t = pair; t < tiles && good; t += pairs) {
            int m0, n0;
            origin(t, m0, n0);
            m0 += static_cast<int>(rank) * BM;
            n0 += static_cast<int>(rank) * BM;
            for (int kb = 0; kb < total_kb; ++kb, ring.next()) {
                const int s = ring.s;
                if (ring.wrapped && !warp_wait(smem_u32(&empty[s]), ring.phase ^ 1, a.err, 2)) {
                    good = false;
                    break;
                }
                if (elect_one()) {
                    // Both CTAs' bytes count on the even CTA's barrier.
                    if (rank == 0) mbar_expect_tx(smem_u32(&full[s]), 4 * kBytes);
                    const uint32_t fb = map_rank(smem_u32(&full[s]), 0);
                    tma_load_2d_pair(smem_u32(sa + s * kBytes), &map_a, fb, kb * BK, m0);
                    tma_load_2d_pair(smem_u32(sb + s * kBytes), &map_b, fb, kb * BK, n0);
                }
            }
        }
        if (!good) drain_pause();
    } else if (warp == 1) {
        if (rank == 0) {
            Ring<S> ring;
            int n = 0;           // accumulators used
            bool good = true;
            for (int t = pair; t < tiles && good; t += pairs, ++n) {
                const int q = n & 1;
                if (n >= 2 && !warp_wait(smem_u32(&acc_empty[q]), ((n / 2) - 1) & 1, a.err, 5)) {
                    good = false;
                    break;
                }
                tc_fence_after();
                for (int kb = 0; kb < total_kb; ++kb, ring.next()) {
                    const int s = ring.s;
                    if (!warp_wait(smem_u32(&full[s]), ring.phase, a.err, 1)) {
                        good = false;
                        break;
                    }
                    tc_fence_after();
                    const uint64_t da = smem_desc<false>(smem_u32(sa + s * kBytes));
                    const uint64_t db = smem_desc<false>(smem_u32(sb + s * kBytes));
                    if (elect_one()) {
#pragma unroll
                        for (int kk = 0; kk < BK / 16; ++kk)
                            mma_bf16_pair(tmem + q * 256, da + kk * 2, db + kk * 2, kIdesc, (kb > 0 || kk > 0) ? 1u : 0u);
                        mma_commit_pair(smem_u32(&empty[s]));
                    }
                }
                if (elect_one()) mma_commit_pair(smem_u32(&acc_full[q]));
                __syncwarp();
            }
            if (!good) drain_pause();
        }
    } else if (warp >= 4) {
        const int quad = warp & 3;
        float* block = blocks + quad * 32 * 33;
        const bool wide = (a.N & 3) == 0 && (reinterpret_cast<uintptr_t>(a.C) & 15) == 0;
        int n = 0;
        bool good = true;
        for (int t = pair; t < tiles && good; t += pairs, ++n) {
            int m0, n0;
            origin(t, m0, n0);
            const int row0 = m0 + static_cast<int>(rank) * BM + quad * 32;
            const int q = n & 1;
            good = warp_wait(smem_u32(&acc_full[q]), (n / 2) & 1, a.err, 4);
            if (!good) break;
            tc_fence_after();
#pragma unroll 1
            for (int c0 = 0; c0 < 256; c0 += 32) {
                {
                    uint32_t r[32];
                    tmem_ld32(tmem + (static_cast<uint32_t>(quad * 32) << 16) + q * 256 + c0, r);
                    if (c0 == 224) {   // read out: the accumulator is free
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive_rank0(smem_u32(&acc_empty[q]));
                    }
#pragma unroll
                    for (int j = 0; j < 32; ++j) block[lane * 33 + j] = __uint_as_float(r[j]);
                }
                __syncwarp();
                if (wide) {
                    const int col = n0 + c0 + 4 * (lane & 7);
#pragma unroll
                    for (int r = 0; r < 8; ++r) {
                        const int rr = 4 * r + (lane >> 3);
                        const float* b = block + rr * 33 + 4 * (lane & 7);
                        if (row0 + rr < a.M && col < a.N)
                            __stcs(reinterpret_cast<float4*>(a.C + static_cast<int64_t>(row0 + rr) * a.N + col),
                                   make_float4(b[0], b[1], b[2], b[3]));
                    }
                } else {
                    const int col = n0 + c0 + lane;
                    for (int rr = 0; rr < 32; ++rr)
                        if (row0 + rr < a.M && col < a.N)
                            a.C[static_cast<int64_t>(row0 + rr) * a.N + col] = block[rr * 33 + lane];
                }
                __syncwarp();
            }
        }
    }
    __syncwarp();
    __syncthreads();
    tc_fence_before();
    cluster_sync();   // no copy, MMA or arrival of the peer touches this CTA any more
    tc_fence_after();
    if (warp == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

}  // namespace pdlpgpu_mlp_impl
