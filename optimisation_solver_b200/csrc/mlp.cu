// mlp.cu -- the learned warm start's network, trained and evaluated with
// this library's own sm_100a kernels: the tensor-core products of gemm.cuh
// with their epilogues, and here what surrounds them -- the fixed-order sums
// of K splits with the layer's activation, the biases' sums and Adam steps,
// the codec between LP instances and the network, and the host side.
//
// A training step (10 launches, each a programmatic launch after the one
// before) stores no output, no FP32 output gradient, no weight gradient and
// no transposed operand: the last layer's product ends in the loss and its
// gradient, and a weight gradient's product ends in Adam.
#include "pdlpgpu_mlp.h"

#include "gemm.cuh"

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <initializer_list>
#include <mutex>
#include <random>
#include <string>
#include <utility>
#include <vector>

extern "C" void pdlpgpu_internal_set_error(const char* message);

namespace pdlpgpu_mlp_impl {

// ---------------------------------------------------------------------------
// Elementwise kernels
// ---------------------------------------------------------------------------
// The K splits' partials of four neighbouring elements added in split order
// (every load is in flight before the first add needs it).
__device__ __forceinline__ void split_sums(const float* partial, int splits, int64_t stride, int64_t t, float (&v)[4]) {
    v[0] = v[1] = v[2] = v[3] = 0.0f;
#pragma unroll 6
    for (int z = 0; z < splits; ++z) {
        const float4 p = *reinterpret_cast<const float4*>(partial + z * stride + t);
        v[0] += p.x;
        v[1] += p.y;
        v[2] += p.z;
        v[3] += p.w;
    }
}

__device__ __forceinline__ void store_bf16x4(bf16* out, const float (&v)[4]) {
    uint2 u;
    u.x = static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(v[0]))) |
          (static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(v[1]))) << 16);
    u.y = static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(v[2]))) |
          (static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(v[3]))) << 16);
    *reinterpret_cast<uint2*>(out) = u;
}

// h = relu(sum of the splits + bias), BF16. N (the hidden width) is a
// multiple of 64.
__global__ void __launch_bounds__(128) hidden_forward(const float* partial, int splits, int64_t stride, int N,
                                                      const float* bias, bf16* h) {
    pdl_trigger();
    pdl_wait();
    const int64_t t = 4 * (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x);
    if (t >= stride) return;
    float v[4];
    split_sums(partial, splits, stride, t, v);
    const float4 b = *reinterpret_cast<const float4*>(bias + t % N);
    v[0] += b.x;
    v[1] += b.y;
    v[2] += b.z;
    v[3] += b.w;
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = v[k] > 0.0f ? v[k] : 0.0f;
    store_bf16x4(h + t, v);
}

// dZ = (sum of the splits) * (H > 0), FP32 (the bias's sum) and BF16 (the
// products).
__global__ void __launch_bounds__(128) hidden_backward(const float* partial, int splits, int64_t stride, const bf16* h,
                                                       float* dz, bf16* dzh) {
    pdl_trigger();
    pdl_wait();
    const int64_t t = 4 * (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x);
    if (t >= stride) return;
    float v[4];
    split_sums(partial, splits, stride, t, v);
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = __bfloat162float(h[t + k]) > 0.0f ? v[k] : 0.0f;
    *reinterpret_cast<float4*>(dz + t) = make_float4(v[0], v[1], v[2], v[3]);
    store_bf16x4(dzh + t, v);
}

// The bias sums and the loss alone (gradient mode; adam_step does them in a
// training step).
__global__ void __launch_bounds__(32) bias_and_loss(BiasArgs a) {
    pdl_trigger();
    pdl_wait();
    bias_and_loss_warp(a, static_cast<int>(blockIdx.x));
}

// C = the splits' partials added in split order, four neighbouring elements a
// thread where C allows 16-byte stores, else one. Sixteen splits' loads are in
// flight before the first is added.
template <int kPer>
__global__ void __launch_bounds__(128) add_splits(const float* partial, int splits, int64_t total, float* C) {
    pdl_trigger();
    pdl_wait();
    const int64_t t = kPer * (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x);
    if (t >= total) return;
    if constexpr (kPer == 4) {
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 16
        for (int z = 0; z < splits; ++z) {
            const float4 p = *reinterpret_cast<const float4*>(partial + z * total + t);
            v.x += p.x;
            v.y += p.y;
            v.z += p.z;
            v.w += p.w;
        }
        *reinterpret_cast<float4*>(C + t) = v;
    } else {
        float v = 0.0f;
#pragma unroll 16
        for (int z = 0; z < splits; ++z) v += partial[z * total + t];
        C[t] = v;
    }
}

__global__ void to_bf16(const float* src, bf16* dst, int64_t n) {
    for (int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; t < n;
         t += static_cast<int64_t>(gridDim.x) * blockDim.x)
        dst[t] = __float2bfloat16_rn(src[t]);
}

// --- codec between LP instances and the network -----------------------------
// A CTA takes 1024 elements, four a thread, whose loads are in flight together: of
// long rows neighbouring elements of one row, so that no element divides its
// index; of rows of up to 512 elements whatever follows in the batch, with one
// division a thread. HBM-bound (20 bytes an element in, 8 to 12 out). Features of
// the flow family's 256 instances of 22,000 parameters: 10.4 us (a division per
// element 20.8); 65,536 rows of 8: 6.8, of 300 62 (a CTA a row 45 and 76, a
// division per element 6.8 and 68).
constexpr int kCodecThreads = 256;
constexpr int kCodecItems = 4;
constexpr int kCodecShort = 512;
struct CodecLaunch {
    bool wide;
    dim3 grid;
    CodecLaunch(int64_t width, int B) : wide(width > kCodecShort) {
        const int64_t per = kCodecThreads * kCodecItems, total = wide ? width : width * B;
        grid = dim3(static_cast<unsigned>((total + per - 1) / per),
                    wide ? static_cast<unsigned>(B < 65535 ? B : 65535) : 1u);
    }
};

// f(b, j) for the CTA's elements j < width of rows b < B: `load` of all items
// before `store` of the first.
template <bool kWide, class Load, class Store>
__device__ __forceinline__ void codec_rows(int B, int width, Load load, Store store) {
    if constexpr (kWide) {
        const int j0 = blockIdx.x * (kCodecThreads * kCodecItems) + threadIdx.x;
        for (int b = blockIdx.y; b < B; b += gridDim.y) {
            decltype(load(0, 0)) v[kCodecItems];
#pragma unroll
            for (int k = 0; k < kCodecItems; ++k)
                if (j0 + k * kCodecThreads < width) v[k] = load(b, j0 + k * kCodecThreads);
#pragma unroll
            for (int k = 0; k < kCodecItems; ++k)
                if (j0 + k * kCodecThreads < width) store(b, j0 + k * kCodecThreads, v[k]);
        }
    } else {
        const uint64_t t = uint64_t(blockIdx.x) * (kCodecThreads * kCodecItems) + threadIdx.x;
        const uint64_t b0 = (t >> 32) == 0 ? static_cast<uint32_t>(t) / static_cast<uint32_t>(width) : t / width;
        const int step_b = kCodecThreads / width, step_j = kCodecThreads % width;
        int b[kCodecItems], j[kCodecItems];
        b[0] = static_cast<int>(b0 < static_cast<uint64_t>(B) ? b0 : B);
        j[0] = static_cast<int>(t - b0 * width);
#pragma unroll
        for (int k = 1; k < kCodecItems; ++k) {
            j[k] = j[k - 1] + step_j;
            b[k] = b[k - 1] >= B - step_b ? B : b[k - 1] + step_b;
            if (j[k] >= width) {
                j[k] -= width;
                b[k] += b[k] < B ? 1 : 0;
            }
        }
        decltype(load(0, 0)) v[kCodecItems];
#pragma unroll
        for (int k = 0; k < kCodecItems; ++k)
            if (b[k] < B) v[k] = load(b[k], j[k]);
#pragma unroll
        for (int k = 0; k < kCodecItems; ++k)
            if (b[k] < B) store(b[k], j[k], v[k]);
    }
}

// Features: standardised instance parameters, BF16, zero-padded to `padded`.
// The parameters are the P of `first` and the Q of `second`, in that order
// (one array has Q = 0).
template <bool kWide>
__global__ void __launch_bounds__(kCodecThreads)
encode_features(int B, int padded, const double* first, int P, const double* second, int Q, const float* mean,
                const float* inv_std, bf16* out) {
    codec_rows<kWide>(
        B, padded,
        [&](int b, int k) {
            const int64_t r = b;
            if (k >= P + Q) return 0.0f;
            const double x = k < P ? first[r * P + k] : second[r * Q + (k - P)];
            return (static_cast<float>(x) - mean[k]) * inv_std[k];
        },
        [&](int b, int k, float v) { out[static_cast<int64_t>(b) * padded + k] = __float2bfloat16_rn(v); });
}

// Targets: primal / scale, standardised dual, standardised log weight, zeros.
template <bool kWide>
__global__ void __launch_bounds__(kCodecThreads)
encode_targets(int B, int O, const double* x, const double* y, const double* w, int n, int m, const double* scale,
               const float* ymean, const float* yinv, float wmean, float winv, float* out) {
    codec_rows<kWide>(
        B, O,
        [&](int b, int j) {
            const int64_t r = b;
            if (j < n) return static_cast<float>(x[r * n + j] / scale[j]);
            if (j < n + m) return (static_cast<float>(y[r * m + (j - n)]) - ymean[j - n]) * yinv[j - n];
            return j == n + m ? (logf(static_cast<float>(w[r])) - wmean) * winv : 0.0f;
        },
        [&](int b, int j, float v) { out[static_cast<int64_t>(b) * O + j] = v; });
}

// Warm start from network outputs: x = clamp(out, 0, 1) * scale, y and the
// weight de-standardised.
template <bool kWide>
__global__ void __launch_bounds__(kCodecThreads)
decode_warmstart(int B, const float* out, int n, int m, int O, const double* scale, const float* ymean,
                 const float* ystd, float wmean, float wstd, double* wx, double* wy, double* ww) {
    codec_rows<kWide>(
        B, n + m + 1,
        [&](int b, int j) {
            const float v = out[static_cast<int64_t>(b) * O + j];
            if (j < n) return static_cast<double>(fminf(fmaxf(v, 0.0f), 1.0f)) * scale[j];
            if (j < n + m) return static_cast<double>(v * ystd[j - n] + ymean[j - n]);
            return static_cast<double>(expf(v * wstd + wmean));
        },
        [&](int b, int j, double v) {
            const int64_t r = b;
            if (j < n) wx[r * n + j] = v;
            else if (j < n + m) wy[r * m + (j - n)] = v;
            else ww[r] = v;
        });
}

inline unsigned grid_for(int64_t n) {
    const int64_t b = (n + 255) / 256;
    return static_cast<unsigned>(b < 148 * 32 ? (b > 0 ? b : 1) : 148 * 32);
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
std::mutex g_encode_mutex;

bool encoder(std::string& err) {
    std::lock_guard<std::mutex> lock(g_encode_mutex);
    if (g_encode) return true;
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || fn == nullptr) {
        err = "cuTensorMapEncodeTiled unavailable";
        return false;
    }
    g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    return true;
}

// 2-D row-major [rows][cols] tensor map with boxes of box_rows x box_cols,
// swizzled over the box's rows of 64 or 128 bytes.
template <class T>
bool make_map(CUtensorMap& map, const T* base, int64_t rows, int64_t cols, int box_cols, int box_rows,
              std::string& err) {
    if (!encoder(err)) return false;
    if ((cols * sizeof(T)) % 16 != 0 || (reinterpret_cast<uintptr_t>(base) & 15) != 0) {
        err = "GEMM operand rows must be 16-byte multiples and 16-byte aligned";
        return false;
    }
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(cols * sizeof(T))};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(box_cols), static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r =
        g_encode(&map, sizeof(T) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                 const_cast<T*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                 box_cols * sizeof(T) == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                 CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        err = "cuTensorMapEncodeTiled failed";
        return false;
    }
    return true;
}

// An operand of `rows` tile rows over K: stored [rows][K], or [K][rows]
// (kMn), which is read in boxes of 64 rows x 64 K.
template <bool kMn>
bool operand_map(CUtensorMap& map, const bf16* base, int rows, int K, int tile_rows, std::string& err) {
    return kMn ? make_map(map, base, K, rows, BK, BK, err) : make_map(map, base, rows, K, BK, tile_rows, err);
}

// A kernel's dynamic shared memory limit, set once per device it runs on.
bool allow_smem(const void* kernel, int bytes, bool (&done)[64], std::string& msg) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (done[dev & 63]) return true;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) {
        msg = "cudaFuncSetAttribute failed";
        return false;
    }
    done[dev & 63] = true;
    return true;
}

// A launch; `after`: it may start while the previous kernel of the stream
// finishes (the kernel waits for it). cluster_x > 1: clusters along x.
template <class... P, class... A>
bool launch(void (*kernel)(P...), dim3 grid, int threads, int smem, cudaStream_t s, bool after, int cluster_x,
            A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(static_cast<unsigned>(threads));
    cfg.dynamicSmemBytes = static_cast<size_t>(smem);
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    unsigned n = 0;
    if (after) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster_x > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = static_cast<unsigned>(cluster_x);
        attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kernel, P(std::forward<A>(args))...) == cudaSuccess;
}

struct Splits {
    int count, per;   // splits that hold K blocks, K blocks of each (the last may be short)
};
Splits effective_splits(int K, int splits) {
    const int total_kb = (K + BK - 1) / BK;
    const int asked = std::max(1, std::min(splits, total_kb));
    const int per = (total_kb + asked - 1) / asked;
    return {(total_kb + per - 1) / per, per};
}

// gemm_tile over the whole product: `parallel` runs the splits side by side
// (one partial each), else every CTA runs its tile's splits one after another.
template <int kBN, int kStages, bool kAMn, bool kBMn, class Epi>
bool tile_gemm(const bf16* A, const bf16* B, int M, int N, int K, Splits sp, bool parallel, const Epi& epi, int* err,
               cudaStream_t s, bool after, std::string& msg) {
    static bool smem_set[64] = {false};
    constexpr int smem = tile_smem<kBN, kStages>();
    auto* kernel = gemm_tile<kBN, kStages, kAMn, kBMn, Epi>;
    if (!allow_smem(reinterpret_cast<const void*>(kernel), smem, smem_set, msg)) return false;
    CUtensorMap ma, mb;
    if (!operand_map<kAMn>(ma, A, M, K, BM, msg) || !operand_map<kBMn>(mb, B, N, K, kBN, msg)) return false;
    const TileArgs ta{M, N, K, sp.per, parallel ? 1 : sp.count, err};
    const dim3 grid((M + BM - 1) / BM, (N + kBN - 1) / kBN, parallel ? sp.count : 1);
    if (!launch(kernel, grid, kTileThreads, smem, s, after, 1, ma, mb, ta, epi)) {
        msg = "GEMM launch failed";
        return false;
    }
    return true;
}

// Error words of calls that have no model to keep one: a slot of this
// static array per call in flight, so calls of several threads do not see
// one another's errors. A slot is zero whenever it is free.
constexpr int kErrSlots = 64;
__device__ int g_gemm_err[kErrSlots];
// The partials of a call's K splits, M x N of every split (74 tiles in 16 splits:
// 78 MB): static, so that no call allocates, and of the call that holds slot 0.
constexpr int64_t kScratchTiles = 1184;   // of 128 x 128
__device__ float4 g_gemm_scratch[kScratchTiles * BM * 128 / 4];
std::mutex g_err_mutex;
uint64_t g_err_used = 0;

struct ErrSlot {
    int slot = -1;
    int* address = nullptr;
    bool owned = false;   // all slots taken: an allocation of its own
    ErrSlot() {
        {
            std::lock_guard<std::mutex> lock(g_err_mutex);
            for (int k = 0; k < kErrSlots && slot < 0; ++k)
                if (!((g_err_used >> k) & 1)) {
                    g_err_used |= uint64_t(1) << k;
                    slot = k;
                }
        }
        void* base = nullptr;
        if (slot >= 0) {
            if (cudaGetSymbolAddress(&base, g_gemm_err) == cudaSuccess) address = static_cast<int*>(base) + slot;
        } else if (cudaMalloc(&base, sizeof(int)) == cudaSuccess) {
            address = static_cast<int*>(base);
            owned = true;
            cudaMemset(address, 0, sizeof(int));
        }
    }
    // The scratch for partials, where this call holds it.
    float* scratch() const {
        void* base = nullptr;
        return slot == 0 && cudaGetSymbolAddress(&base, g_gemm_scratch) == cudaSuccess ? static_cast<float*>(base)
                                                                                       : nullptr;
    }
    // Waits for the default stream and returns the error word, clearing it;
    // a negative value is a CUDA error.
    int take() {
        int h = 0;
        if (cudaMemcpy(&h, address, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
        if (h != 0) cudaMemset(address, 0, sizeof(int));
        return h;
    }
    ~ErrSlot() {
        if (owned) cudaFree(address);
        if (slot >= 0) {
            std::lock_guard<std::mutex> lock(g_err_mutex);
            g_err_used &= ~(uint64_t(1) << slot);
        }
    }
    ErrSlot(const ErrSlot&) = delete;
    ErrSlot& operator=(const ErrSlot&) = delete;
};

// C = A B^T for the two entry points below. The rule, with times in us of the
// kernels that meet at each line:
//   one split, at least 56 tiles of 256 x 256 and 1792 tile x K-block steps:
//     gemm_pair (4096 x 2048 x 4096: 51, gemm_tile 63; 2048^3 21, 21;
//     4096 x 2048 x 512, below the line: 21 against 19)
//   several splits: gemm_tile with a CTA for every split of every tile, the
//     partials in `scratch` and added by add_splits, as long as the splits make
//     up for the waves of CTAs (K = 8000, in brackets each CTA its tile's splits
//     in turn: 60 tiles in 8 splits 30 [47], in 16 49 [72], 96 in 3 29 [35], in 12
//     59 [60]; beyond the line 104 in 8 50 [48], 147 in 2 41 [37]; 256 x 512 x
//     22000 in 18 takes 16). Six stages and an SM to itself while the CTAs fit the SMs once, else
//     three and two CTAs an SM (24 tiles in 8: 17, with six 22). The clusters of
//     CTAs that added their splits through distributed shared memory took 33 at
//     256 x 512 x 22000, 27 with wide loads, and 51 and 25 for two splits of one
//     tile (23 this way).
//   else gemm_tile, each CTA its tile's splits in turn: six stages and an SM
//     to itself while the tiles fit the SMs once or a tile has several splits
//     to keep apart in TMEM (3000 x 2000 x 4096 in 8: 88, with three stages
//     184), else three stages and two CTAs an SM (2560 x 1024 x 1024, 160
//     tiles: 14, with six 19).
constexpr int64_t kPairMinTiles = 56;
constexpr int64_t kPairMinSteps = 1792;

bool plain_gemm(const bf16* A, const bf16* B, float* C, int M, int N, int K, int splits, float* scratch, int* err,
                cudaStream_t s, std::string& msg) {
    if (K % 8 != 0) {
        msg = "GEMM K must be a multiple of 8";
        return false;
    }
    const Splits sp = effective_splits(K, splits);
    const int64_t pair_tiles = int64_t((M + 255) / 256) * ((N + 255) / 256);
    const int64_t tiles = int64_t((M + BM - 1) / BM) * ((N + 127) / 128);
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sp.count == 1 && pair_tiles >= kPairMinTiles && pair_tiles * ((K + BK - 1) / BK) >= kPairMinSteps) {
        static bool smem_set[64] = {false};
        if (!allow_smem(reinterpret_cast<const void*>(gemm_pair), kPairSmem, smem_set, msg)) return false;
        CUtensorMap ma, mb;
        if (!make_map(ma, A, M, K, BK, BM, msg) || !make_map(mb, B, N, K, BK, BM, msg)) return false;
        const PairArgs pa{M, N, K, C, err};
        const unsigned pairs = static_cast<unsigned>(std::min<int64_t>(pair_tiles, sms / 2));
        return launch(gemm_pair, dim3(2 * pairs), kPairThreads, kPairSmem, s, false, 1, ma, mb, pa);
    }
    const int64_t ctas = tiles * sp.count, waves = (ctas + 2 * sms - 1) / (2 * sms);
    if (sp.count > 1 && scratch != nullptr && ctas <= kScratchTiles && (ctas <= sms || 3 * waves <= sp.count)) {
        const int64_t total = int64_t(M) * N;
        const EpiStore epi{scratch, total};
        if (!(ctas <= sms ? tile_gemm<128, 6, false, false>(A, B, M, N, K, sp, true, epi, err, s, false, msg)
                          : tile_gemm<128, 3, false, false>(A, B, M, N, K, sp, true, epi, err, s, false, msg)))
            return false;
        const bool wide = total % 4 == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0;
        const int64_t threads = wide ? total / 4 : total;
        return launch(wide ? add_splits<4> : add_splits<1>, dim3(static_cast<unsigned>((threads + 127) / 128)), 128, 0, s,
                      true, 1, scratch, sp.count, total, C);
    }
    const EpiStore epi{C, 0};
    if (tiles <= sms || sp.count > 1)
        return tile_gemm<128, 6, false, false>(A, B, M, N, K, sp, false, epi, err, s, false, msg);
    return tile_gemm<128, 3, false, false>(A, B, M, N, K, sp, false, epi, err, s, false, msg);
}

int splits_for(int M, int N, int K) {
    const int tiles = ((M + BM - 1) / BM) * ((N + 127) / 128);
    const int kb = (K + BK - 1) / BK;
    int s = std::max(1, 148 / std::max(1, tiles));
    return std::min(s, std::max(1, kb / 4));
}

}  // namespace pdlpgpu_mlp_impl

using namespace pdlpgpu_mlp_impl;

struct pdlpgpu_mlp {
    int in = 0, hidden = 0, out = 0, batch = 0, device = 0;
    int sms = 148;
    cudaStream_t stream = nullptr;
    cudaEvent_t caller_done = nullptr;
    std::vector<void*> allocs;
    // parameters (FP32 master), BF16 copies, Adam moments, gradients
    float *W1 = nullptr, *b1 = nullptr, *W2 = nullptr, *b2 = nullptr, *W3 = nullptr, *b3 = nullptr;
    bf16 *W1h = nullptr, *W2h = nullptr, *W3h = nullptr;
    float *mW1, *vW1, *mb1, *vb1, *mW2, *vW2, *mb2, *vb2, *mW3, *vW3, *mb3, *vb3;
    // activations and scratch
    bf16 *H1 = nullptr, *H2 = nullptr;
    float *dZ1 = nullptr, *dZ2 = nullptr;
    bf16 *dOuth = nullptr, *dZ1h = nullptr, *dZ2h = nullptr;
    float* partial = nullptr;   // split-K partials of a [batch][hidden] product
    double* loss_part = nullptr;
    // What a call reports, read back in one copy: the loss and the pipeline's
    // error word; `report` is its pinned host copy.
    struct Report {
        float loss;
        int err;
    };
    Report *report_dev = nullptr, *report = nullptr;
    int* err = nullptr;         // &report_dev->err
    int64_t step = 0;           // Adam steps taken
    int64_t launches = 0;
    std::string msg;

    ~pdlpgpu_mlp() {
        for (void* p : allocs) cudaFree(p);
        if (report) cudaFreeHost(report);
        if (caller_done) cudaEventDestroy(caller_done);
        if (stream) cudaStreamDestroy(stream);
    }

    // The caller's device arguments (features, targets, parameters) are
    // usually written just before the call on the legacy default stream --
    // by pdlpgpu_encode_features, or by PyTorch, which enqueues there by
    // default -- and the model's own stream does not synchronise with it
    // implicitly (it is non-blocking): it waits for all work enqueued there
    // so far before it reads them.
    bool wait_for_caller() {
        if (!caller_done && cudaEventCreateWithFlags(&caller_done, cudaEventDisableTiming) != cudaSuccess)
            return false;
        return cudaEventRecord(caller_done, cudaStreamLegacy) == cudaSuccess &&
               cudaStreamWaitEvent(stream, caller_done, 0) == cudaSuccess;
    }

    template <class T>
    bool alloc(T*& p, int64_t n) {
        void* q = nullptr;
        if (cudaMalloc(&q, static_cast<size_t>(std::max<int64_t>(n, 1)) * sizeof(T)) != cudaSuccess) {
            msg = "cudaMalloc failed";
            return false;
        }
        cudaMemsetAsync(q, 0, static_cast<size_t>(std::max<int64_t>(n, 1)) * sizeof(T), stream);
        allocs.push_back(q);
        p = static_cast<T*>(q);
        return true;
    }

    // A launch after the previous one of the call (the call's first is
    // ordered after the caller's work instead, see wait_for_caller).
    template <class... P, class... A>
    bool enqueue(void (*kernel)(P...), int grid, int threads, A&&... args) {
        const bool after = launches++ > 0;
        if (launch(kernel, dim3(static_cast<unsigned>(grid)), threads, 0, stream, after, 1, std::forward<A>(args)...))
            return true;
        msg = "launch failed";
        return false;
    }

    template <int kStages, bool kAMn, bool kBMn, class Epi>
    bool product(const bf16* A, const bf16* B, int M, int N, int K, Splits sp, const Epi& epi) {
        const bool after = launches++ > 0;
        return tile_gemm<128, kStages, kAMn, kBMn>(A, B, M, N, K, sp, true, epi, err, stream, after, msg);
    }

    // partial[z] of a [batch][hidden] product over K, and its splits. With at
    // most one CTA per SM the ring is six stages deep (the copies in flight
    // bound a long K): 22,000 inputs, 512 wide, batch 256. More CTAs go two to an
    // SM with three stages, as in plain_gemm.
    template <bool kBMn>
    bool hidden_product(const bf16* A, const bf16* B, int K, Splits& sp) {
        sp = effective_splits(K, splits_for(batch, hidden, K));
        const EpiStore epi{partial, int64_t(batch) * hidden};
        const int64_t ctas = int64_t((batch + BM - 1) / BM) * ((hidden + 127) / 128) * sp.count;
        return ctas <= sms ? product<6, false, kBMn>(A, B, batch, hidden, K, sp, epi)
                           : product<3, false, kBMn>(A, B, batch, hidden, K, sp, epi);
    }

    int hidden_ctas() const { return static_cast<int>((int64_t(batch) * hidden / 4 + 127) / 128); }

    bool forward_hidden(const bf16* X) {
        const int64_t BH = int64_t(batch) * hidden;
        Splits sp;
        return hidden_product<false>(X, W1h, in, sp) &&
               enqueue(hidden_forward, hidden_ctas(), 128, partial, sp.count, BH, hidden, b1, H1) &&
               hidden_product<false>(H1, W2h, hidden, sp) &&
               enqueue(hidden_forward, hidden_ctas(), 128, partial, sp.count, BH, hidden, b2, H2);
    }

    // The last layer's column tile: the whole width over the SMs, in
    // 32-column blocks, at most 256 columns (one MMA).
    int last_bn() const { return std::min(256, ((out + sms - 1) / sms + 31) / 32 * 32); }
    int last_ctas() const { return (out + last_bn() - 1) / last_bn(); }

    // A forward pass of a batch of many rows may share the row tiles of wider
    // column tiles instead. What counts is the bytes a CTA copies into shared
    // memory, 128 + bn rows of both operands per K block and row tile
    // (a forward pass of 1024 x 512 x 64, batch 8192: 69 us, 203 with two CTAs; 2048 x
    // 1024 x 2048, batch 4096: 94 and 205). The K splits, and with them the
    // bits, stay.
    void forward_tile(int splits, int& bn, int& rows) const {
        const int mts = (batch + BM - 1) / BM;
        int64_t least = INT64_MAX;
        for (int n = last_bn(); n <= 256 && n * splits <= kLastTmem; n += 32) {
            const int ctas = (out + n - 1) / n, share = std::max(1, std::min(mts, sms / ctas));
            const int64_t cost = int64_t((mts + share - 1) / share) * (BM + n) * ((ctas * share + sms - 1) / sms);
            if (cost >= least) continue;
            least = cost;
            bn = n;
            rows = share;
        }
    }

    template <bool kTrain>
    bool last(LastArgs la) {
        int bn = last_bn(), rows = 1;   // CTAs that share the batch's row tiles
        const Splits sp = effective_splits(hidden, std::min(splits_for(batch, out, hidden), kLastTmem / bn));
        if (!kTrain) forward_tile(sp.count, bn, rows);
        la.M = batch;
        la.N = out;
        la.K = hidden;
        la.bn = bn;
        la.kb_per_split = sp.per;
        la.splits = sp.count;
        la.bias = b3;
        la.err = err;
        static bool smem_set[64] = {false};
        if (!allow_smem(reinterpret_cast<const void*>(last_layer<kTrain>), last_smem(256), smem_set, msg)) return false;
        CUtensorMap ma, mb;
        if (!make_map(ma, H2, batch, hidden, BK, BM, msg) || !make_map(mb, W3h, out, hidden, BK, bn, msg)) return false;
        ++launches;
        if (launch(last_layer<kTrain>, dim3(static_cast<unsigned>((out + bn - 1) / bn), static_cast<unsigned>(rows)),
                   kLastThreads, last_smem(bn), stream, true, 1, ma, mb, la))
            return true;
        msg = "GEMM launch failed";
        return false;
    }

    bool forward(const bf16* X, float* outputs) {
        LastArgs la{};
        la.out = outputs;
        return forward_hidden(X) && last<false>(la);
    }

    // Gradients wanted by the caller (any may be null), or, when `lr` is not
    // negative, an Adam step.
    struct Gradients {
        float *W1 = nullptr, *b1 = nullptr, *W2 = nullptr, *b2 = nullptr, *W3 = nullptr, *b3 = nullptr;
    };

    // dW = D^T A of a [batch][rows] and a [batch][cols] matrix, both operands
    // as they lie, into `grad`.
    bool weight_gradient(const bf16* D, const bf16* A, int rows, int cols, float* grad) {
        return grad == nullptr || product<3, true, true>(D, A, rows, cols, batch, effective_splits(batch, 1),
                                                         EpiStore{grad, 0});
    }
    bool adam_layer(AdamLayer& L, const bf16* D, const bf16* A, int rows, int cols, float* p, float* m, float* v,
                    bf16* h) {
        L.rows = rows;
        L.cols = cols;
        L.tiles_n = (cols + kAdamBN - 1) / kAdamBN;
        L.tiles = (rows + BM - 1) / BM * L.tiles_n;
        return operand_map<true>(L.d, D, rows, batch, BM, msg) && operand_map<true>(L.a, A, cols, batch, kAdamBN, msg) &&
               make_map(L.p, p, rows, cols, 32, BM, msg) && make_map(L.m, m, rows, cols, 32, BM, msg) &&
               make_map(L.v, v, rows, cols, 32, BM, msg) && make_map(L.h, h, rows, cols, 32, BM, msg);
    }

    bool step_or_gradients(const bf16* X, const float* target, const float* w, bool train, float lr,
                           const Gradients& g) {
        AdamStep adam{lr, 0.9f, 0.999f, 1e-8f, 1.0f, 1.0f, 1.0f, 1.0f};
        if (train) {
            adam.c1 = 1.0f - std::pow(adam.b1, static_cast<float>(step + 1));
            adam.c2 = 1.0f - std::pow(adam.b2, static_cast<float>(step + 1));
            adam.r1 = 1.0f / adam.c1;
            adam.r2 = 1.0f / adam.c2;
        }
        LastArgs la{};
        la.target = target;
        la.weight = w;
        la.d = dOuth;
        la.loss_part = loss_part;
        // In gradient mode the bias gradient always has a place to go: the
        // split-K partials are free while the last layer runs.
        la.gb = train ? nullptr : (g.b3 != nullptr ? g.b3 : partial);
        la.mb = mb3;
        la.vb = vb3;
        la.adam = adam;
        if (!forward_hidden(X) || !last<true>(la)) return false;
        // dH2 = dOut W3 and dH1 = dZ2 W2 read the weights as they are stored
        // (K x hidden), before the Adam steps below change them.
        const int64_t BH = int64_t(batch) * hidden;
        Splits sp;
        if (!hidden_product<true>(dOuth, W3h, out, sp) ||
            !enqueue(hidden_backward, hidden_ctas(), 128, partial, sp.count, BH, H2, dZ2, dZ2h) ||
            !hidden_product<true>(dZ2h, W2h, hidden, sp) ||
            !enqueue(hidden_backward, hidden_ctas(), 128, partial, sp.count, BH, H1, dZ1, dZ1h))
            return false;
        const BiasArgs ba{{dZ1, dZ2}, {b1, b2}, {mb1, mb2}, {vb1, vb2}, {g.b1, g.b2}, batch, hidden, !train, adam,
                          loss_part, last_ctas(), &report_dev->loss};
        if (!train)
            return weight_gradient(dOuth, H2, out, hidden, g.W3) && weight_gradient(dZ1h, X, hidden, in, g.W1) &&
                   weight_gradient(dZ2h, H1, hidden, hidden, g.W2) &&
                   enqueue(bias_and_loss, bias_warps(hidden), 32, ba);
        AdamArgs aa;
        if (!adam_layer(aa.layer[0], dZ2h, H1, hidden, hidden, W2, mW2, vW2, W2h) ||
            !adam_layer(aa.layer[1], dOuth, H2, out, hidden, W3, mW3, vW3, W3h) ||
            !adam_layer(aa.layer[2], dZ1h, X, hidden, in, W1, mW1, vW1, W1h))
            return false;
        aa.adam = adam;
        aa.bias = ba;
        aa.K = batch;
        aa.tiles = aa.layer[0].tiles + aa.layer[1].tiles + aa.layer[2].tiles;
        aa.err = err;
        static bool smem_set[64] = {false};
        if (!allow_smem(reinterpret_cast<const void*>(adam_step), kAdamSmem, smem_set, msg)) return false;
        ++launches;
        if (!launch(adam_step, dim3(static_cast<unsigned>(std::min(aa.tiles, sms))), kAdamThreads, kAdamSmem, stream,
                    true, 1, aa)) {
            msg = "Adam launch failed";
            return false;
        }
        ++step;   // a refused call does not count
        return true;
    }

    void refresh_bf16() {
        to_bf16<<<grid_for(int64_t(hidden) * in), 256, 0, stream>>>(W1, W1h, int64_t(hidden) * in);
        to_bf16<<<grid_for(int64_t(hidden) * hidden), 256, 0, stream>>>(W2, W2h, int64_t(hidden) * hidden);
        to_bf16<<<grid_for(int64_t(out) * hidden), 256, 0, stream>>>(W3, W3h, int64_t(out) * hidden);
    }

    // Whether the kernels can store to a caller's array (null: not asked for);
    // host memory that is not mapped for the device is refused here, instead of
    // faulting there.
    bool writable(std::initializer_list<const float*> arrays) {
        for (const float* p : arrays) {
            if (p == nullptr) continue;
            cudaPointerAttributes a;
            if (cudaPointerGetAttributes(&a, p) == cudaSuccess && a.type != cudaMemoryTypeUnregistered &&
                (reinterpret_cast<uintptr_t>(p) & 3) == 0)
                continue;
            cudaGetLastError();
            msg = "outputs must be float arrays in device memory";
            return false;
        }
        return true;
    }

    // Waits for the call; false on a CUDA error or a pipeline timeout.
    bool finish(const char* what, float* loss) {
        if (cudaMemcpyAsync(report, report_dev, sizeof(Report), cudaMemcpyDeviceToHost, stream) != cudaSuccess ||
            cudaStreamSynchronize(stream) != cudaSuccess) {
            msg = std::string(what) + ": " + cudaGetErrorString(cudaGetLastError());
            return false;
        }
        if (loss) *loss = report->loss;
        if (report->err != 0) {
            msg = std::string(what) + ": tensor-core pipeline wait timed out (code " + std::to_string(report->err) + ")";
            cudaMemsetAsync(err, 0, sizeof(int), stream);
            return false;
        }
        return true;
    }
};

namespace {
int fail(const std::string& m) {
    pdlpgpu_internal_set_error(m.c_str());
    return -1;
}
}  // namespace

extern "C" {

int32_t pdlpgpu_mlp_create(int32_t in, int32_t hidden, int32_t out, int32_t batch, uint64_t seed,
                           int32_t device, pdlpgpu_mlp** result) {
    if (in <= 0 || in % 8 != 0 || hidden <= 0 || hidden % 64 != 0 || out <= 0 || out % 64 != 0 ||
        batch <= 0 || batch % 8 != 0)
        return fail("mlp: in must be a multiple of 8, hidden and out of 64, batch of 8");
    auto* m = new pdlpgpu_mlp();
    m->in = in; m->hidden = hidden; m->out = out; m->batch = batch; m->device = device;
    if (cudaSetDevice(device) != cudaSuccess || cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess) {
        delete m;
        return fail("mlp: cannot use the device");
    }
    if (cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) m->sms = 148;
    const int64_t H = hidden, I = in, O = out, B = batch;
    bool ok = m->alloc(m->W1, H * I) && m->alloc(m->b1, H) && m->alloc(m->W2, H * H) &&
              m->alloc(m->b2, H) && m->alloc(m->W3, O * H) && m->alloc(m->b3, O) &&
              m->alloc(m->W1h, H * I) && m->alloc(m->W2h, H * H) && m->alloc(m->W3h, O * H);
    for (auto* q : {&m->mW1, &m->vW1}) ok = ok && m->alloc(*q, H * I);
    for (auto* q : {&m->mW2, &m->vW2}) ok = ok && m->alloc(*q, H * H);
    for (auto* q : {&m->mW3, &m->vW3}) ok = ok && m->alloc(*q, O * H);
    for (auto* q : {&m->mb1, &m->vb1, &m->mb2, &m->vb2}) ok = ok && m->alloc(*q, H);
    for (auto* q : {&m->mb3, &m->vb3}) ok = ok && m->alloc(*q, O);
    for (auto* q : {&m->H1, &m->H2, &m->dZ1h, &m->dZ2h}) ok = ok && m->alloc(*q, B * H);
    for (auto* q : {&m->dZ1, &m->dZ2}) ok = ok && m->alloc(*q, B * H);
    ok = ok && m->alloc(m->dOuth, B * O) && m->alloc(m->loss_part, m->last_ctas()) && m->alloc(m->report_dev, 1);
    // Split-K partials of the [B x H] products (at least O: see gb in step_or_gradients).
    int64_t parts = 1;
    for (int k : {in, hidden, out})
        parts = std::max<int64_t>(parts, effective_splits(k, splits_for(batch, hidden, k)).count);
    ok = ok && m->alloc(m->partial, std::max(parts * B * H, O));
    if (ok && cudaMallocHost(reinterpret_cast<void**>(&m->report), sizeof(pdlpgpu_mlp::Report)) != cudaSuccess) {
        m->msg = "cudaMallocHost failed";
        ok = false;
    }
    if (ok) m->err = &m->report_dev->err;
    if (!ok) {
        const std::string msg = m->msg;
        delete m;
        return fail("mlp: " + msg);
    }
    // He initialisation (normal, std sqrt(2/fan_in)), seeded.
    std::mt19937_64 rng(seed);
    auto init = [&](float* dst, int64_t rows, int64_t fan_in) {
        std::normal_distribution<float> nd(0.0f, std::sqrt(2.0f / static_cast<float>(fan_in)));
        std::vector<float> h(static_cast<size_t>(rows * fan_in));
        for (float& v : h) v = nd(rng);
        cudaMemcpyAsync(dst, h.data(), h.size() * sizeof(float), cudaMemcpyHostToDevice, m->stream);
        cudaStreamSynchronize(m->stream);
    };
    init(m->W1, H, I);
    init(m->W2, H, H);
    init(m->W3, O, H);
    m->refresh_bf16();
    if (cudaStreamSynchronize(m->stream) != cudaSuccess) {
        delete m;
        return fail("mlp: initialisation failed");
    }
    *result = m;
    return 0;
}

void pdlpgpu_mlp_destroy(pdlpgpu_mlp* m) { delete m; }

int32_t pdlpgpu_mlp_forward(pdlpgpu_mlp* m, const uint16_t* inputs, float* outputs) {
    if (!m) return -1;
    cudaSetDevice(m->device);
    m->launches = 0;
    if (outputs == nullptr || !m->writable({outputs})) return fail("mlp forward: outputs must be float arrays in device memory");
    if (!m->wait_for_caller()) return fail("mlp forward: stream wait failed");
    if (!m->forward(reinterpret_cast<const bf16*>(inputs), outputs)) return fail("mlp forward: " + m->msg);
    if (!m->finish("mlp forward", nullptr)) return fail(m->msg);
    return 0;
}

int32_t pdlpgpu_mlp_gradients(pdlpgpu_mlp* m, const uint16_t* inputs, const float* targets,
                              const float* w, float* dW1, float* db1, float* dW2, float* db2,
                              float* dW3, float* db3, float* loss) {
    if (!m) return -1;
    cudaSetDevice(m->device);
    m->launches = 0;
    if (!m->writable({dW1, db1, dW2, db2, dW3, db3})) return fail("mlp gradients: " + m->msg);
    if (!m->wait_for_caller()) return fail("mlp gradients: stream wait failed");
    const pdlpgpu_mlp::Gradients g{dW1, db1, dW2, db2, dW3, db3};
    if (!m->step_or_gradients(reinterpret_cast<const bf16*>(inputs), targets, w, false, 0.0f, g))
        return fail("mlp gradients: " + m->msg);
    if (!m->finish("mlp gradients", loss)) return fail(m->msg);
    return 0;
}

int32_t pdlpgpu_mlp_train_step(pdlpgpu_mlp* m, const uint16_t* inputs, const float* targets,
                               const float* w, float lr, float* loss) {
    if (!m) return -1;
    cudaSetDevice(m->device);
    m->launches = 0;
    if (!m->wait_for_caller()) return fail("mlp train: stream wait failed");
    if (!m->step_or_gradients(reinterpret_cast<const bf16*>(inputs), targets, w, true, lr, {}))
        return fail("mlp train: " + m->msg);
    if (!m->finish("mlp train", loss)) return fail(m->msg);
    return 0;
}

int32_t pdlpgpu_mlp_get_params(pdlpgpu_mlp* m, float* W1, float* b1, float* W2, float* b2,
                               float* W3, float* b3) {
    if (!m) return -1;
    cudaSetDevice(m->device);
    if (!m->wait_for_caller()) return fail("mlp get_params: stream wait failed");
    const int64_t H = m->hidden, I = m->in, O = m->out;
    auto cp = [&](float* dst, const float* src, int64_t n) {
        if (dst) cudaMemcpyAsync(dst, src, n * sizeof(float), cudaMemcpyDeviceToDevice, m->stream);
    };
    cp(W1, m->W1, H * I); cp(b1, m->b1, H); cp(W2, m->W2, H * H); cp(b2, m->b2, H);
    cp(W3, m->W3, O * H); cp(b3, m->b3, O);
    return cudaStreamSynchronize(m->stream) == cudaSuccess ? 0 : fail("mlp get_params failed");
}

int32_t pdlpgpu_mlp_set_params(pdlpgpu_mlp* m, const float* W1, const float* b1, const float* W2,
                               const float* b2, const float* W3, const float* b3) {
    if (!m) return -1;
    cudaSetDevice(m->device);
    if (!m->wait_for_caller()) return fail("mlp set_params: stream wait failed");
    const int64_t H = m->hidden, I = m->in, O = m->out;
    auto cp = [&](float* dst, const float* src, int64_t n) {
        if (src) cudaMemcpyAsync(dst, src, n * sizeof(float), cudaMemcpyDeviceToDevice, m->stream);
    };
    cp(m->W1, W1, H * I); cp(m->b1, b1, H); cp(m->W2, W2, H * H); cp(m->b2, b2, H);
    cp(m->W3, W3, O * H); cp(m->b3, b3, O);
    m->refresh_bf16();
    return cudaStreamSynchronize(m->stream) == cudaSuccess ? 0 : fail("mlp set_params failed");
}

int64_t pdlpgpu_mlp_launches(pdlpgpu_mlp* m) { return m ? m->launches : 0; }

int32_t pdlpgpu_gemm_bf16(int32_t M, int32_t N, int32_t K, const uint16_t* A, const uint16_t* B,
                          float* C, int32_t splits) {
    if (M <= 0 || N <= 0 || K <= 0) return fail("gemm: sizes must be positive");
    ErrSlot err;
    if (err.address == nullptr) return fail("gemm: no error word");
    std::string msg;
    bool ok = plain_gemm(reinterpret_cast<const bf16*>(A), reinterpret_cast<const bf16*>(B), C, M, N, K, splits,
                         err.scratch(), err.address, nullptr, msg);
    const int h = err.take();
    if (h > 0) msg = "tensor-core pipeline wait timed out (code " + std::to_string(h) + ")";
    ok = ok && h == 0;
    return ok ? 0 : fail("gemm: " + (msg.empty() ? std::string(cudaGetErrorString(cudaGetLastError())) : msg));
}


int32_t pdlpgpu_gemm_time(int32_t M, int32_t N, int32_t K, const uint16_t* A, const uint16_t* B,
                          float* C, int32_t splits, int32_t reps, double* ms_per_call) {
    if (M <= 0 || N <= 0 || K <= 0 || reps <= 0 || ms_per_call == nullptr)
        return fail("gemm_time: sizes and repetitions must be positive");
    ErrSlot err;
    if (err.address == nullptr) return fail("gemm_time: no error word");
    std::string msg;
    auto once = [&]() {
        return plain_gemm(reinterpret_cast<const bf16*>(A), reinterpret_cast<const bf16*>(B), C, M, N, K, splits,
                          err.scratch(), err.address, nullptr, msg);
    };
    bool ok = once();   // warm-up: tensor maps, instruction cache
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0);
    for (int r = 0; ok && r < reps; ++r) ok = once();
    cudaEventRecord(e1);
    cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    const int h = err.take();
    if (h > 0) msg = "tensor-core pipeline wait timed out (code " + std::to_string(h) + ")";
    ok = ok && h == 0;
    *ms_per_call = ms / reps;
    return ok ? 0 : fail("gemm_time: " + (msg.empty() ? std::string(cudaGetErrorString(cudaGetLastError())) : msg));
}

int32_t pdlpgpu_encode_features(const double* params, int32_t batch, int32_t count, int32_t padded,
                                const float* mean, const float* inv_std, uint16_t* out) {
    if (batch <= 0 || count <= 0 || padded < count) return fail("encode_features: bad sizes");
    const CodecLaunch c(padded, batch);
    (c.wide ? encode_features<true> : encode_features<false>)<<<c.grid, kCodecThreads>>>(
        batch, padded, params, count, nullptr, 0, mean, inv_std, reinterpret_cast<bf16*>(out));
    return cudaGetLastError() == cudaSuccess ? 0 : fail("encode_features: launch failed");
}

int32_t pdlpgpu_encode_feature_pair(const double* first, int32_t first_count, const double* second,
                                    int32_t second_count, int32_t batch, int32_t padded, const float* mean,
                                    const float* inv_std, uint16_t* out) {
    const int64_t count = static_cast<int64_t>(first_count) + second_count;
    if (batch <= 0 || first_count <= 0 || second_count <= 0 || padded < count)
        return fail("encode_feature_pair: bad sizes");
    const CodecLaunch c(padded, batch);
    (c.wide ? encode_features<true> : encode_features<false>)<<<c.grid, kCodecThreads>>>(
        batch, padded, first, first_count, second, second_count, mean, inv_std, reinterpret_cast<bf16*>(out));
    return cudaGetLastError() == cudaSuccess ? 0 : fail("encode_feature_pair: launch failed");
}

int32_t pdlpgpu_encode_targets(const double* primal, const double* dual, const double* weight,
                               int32_t batch, int32_t n, int32_t m, int32_t out_width,
                               const double* primal_scale, const float* dual_mean,
                               const float* dual_inv_std, float weight_mean, float weight_inv_std,
                               float* targets) {
    if (batch <= 0 || out_width < n + m + 1) return fail("encode_targets: bad sizes");
    const CodecLaunch c(out_width, batch);
    (c.wide ? encode_targets<true> : encode_targets<false>)<<<c.grid, kCodecThreads>>>(
        batch, out_width, primal, dual, weight, n, m, primal_scale, dual_mean, dual_inv_std, weight_mean,
        weight_inv_std, targets);
    return cudaGetLastError() == cudaSuccess ? 0 : fail("encode_targets: launch failed");
}

int32_t pdlpgpu_decode_warmstart(const float* outputs, int32_t batch, int32_t n, int32_t m,
                                 int32_t out_width, const double* primal_scale,
                                 const float* dual_mean, const float* dual_std, float weight_mean,
                                 float weight_std, double* primal, double* dual, double* weight) {
    if (batch <= 0 || out_width < n + m + 1) return fail("decode_warmstart: bad sizes");
    const CodecLaunch c(static_cast<int64_t>(n) + m + 1, batch);
    (c.wide ? decode_warmstart<true> : decode_warmstart<false>)<<<c.grid, kCodecThreads>>>(
        batch, outputs, n, m, out_width, primal_scale, dual_mean, dual_std, weight_mean, weight_std, primal, dual,
        weight);
    return cudaGetLastError() == cudaSuccess ? 0 : fail("decode_warmstart: launch failed");
}

}  // extern "C"
