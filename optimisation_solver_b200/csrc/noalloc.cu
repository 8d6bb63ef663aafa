// noalloc.cu -- one fused PDHG trial that allocates no device memory.
//
// Some callers cannot let a library call cudaMalloc: a serving process that
// owns every byte of device memory through its own pool and a fixed budget,
// or a solve loop that must not take the device-wide synchronisation an
// allocation can cause. pdlpgpu_trial_noalloc serves them: the caller passes
// every input and output as device memory it already owns, and the only
// scratch the kernels need -- one partial sum per CTA -- lives in the
// file-scope array below, which the driver places in device memory when it
// loads this library (each GPU that loads it keeps those 192 KiB until the
// process exits). Nothing here calls cudaMalloc, cudaFree or an allocating
// library routine.
//
// The computation is pdlpgpu_trial's (the reference's CpuPdhgKernel::trial,
// pdlp_engine/src/pdhg_kernel.cpp:47-187) on plain CSR inputs: blocks of
// lines, the primal half over the rows of A^T, the dual half over the rows
// of A, then one CTA adds the partial sums in a fixed order.
#include "pdlpgpu_components.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <mutex>
#include <string>
#include <vector>

extern "C" void pdlpgpu_internal_set_error(const char* message);

namespace {

constexpr int kNaThreads = 256;
constexpr int64_t kNaMaxLines = 8388608;            // the interface's bound; nothing here depends on it
constexpr int kNaGridCtas = 148 * 16;               // CTAs of a half at most (each loops over its blocks)
constexpr int kNaUnroll = 6;                        // entries a thread has in flight
constexpr int kNaChunk = 2 * kNaUnroll * kNaThreads;   // products in shared memory: 24 KiB
constexpr int kNaLong = 32;                         // longer pieces of a line are summed by a whole warp
constexpr unsigned kFull = 0xffffffffu;

// Slots [0, kNaGridCtas): primal partials; then two per dual CTA.
static __device__ __align__(256) double g_noalloc_scratch[3 * kNaGridCtas];

// Address of the array in each CUDA context it was looked up in. The key is
// the context's unique ID, not the device ordinal: after cudaDeviceReset, or
// under a caller's own driver context, the library's module is loaded again at
// another address, and a lookup made in an earlier context would be stale.
// Context IDs are never reused within a process, unlike context handles.
struct ScratchEntry {
    unsigned long long context_id;
    double* address;
};
std::mutex g_scratch_mutex;
std::vector<ScratchEntry> g_scratch_entries;
using CtxGetCurrent = int (*)(void**);                    // cuCtxGetCurrent(CUcontext*)
using CtxGetId = int (*)(void*, unsigned long long*);     // cuCtxGetId(CUcontext, id*)
CtxGetCurrent g_ctx_get_current = nullptr;
CtxGetId g_ctx_get_id = nullptr;

__device__ __forceinline__ double dmin(double a, double b) { return b < a ? b : a; }
__device__ __forceinline__ double dmax(double a, double b) { return a < b ? b : a; }

// Programmatic dependent launch: the dual half and the final sum are launched
// while their predecessor finishes, and wait here for its results. A kernel
// of this file lets its successor start only after its own wait, so whatever
// ran before the call, the primal half and the dual half complete in order.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Lines of a block of the two halves: a power of two from 32 to kNaThreads that gives every SM
// about two blocks where the problem is that small. Below 32 lines a block's
// few entries no longer fill the threads; above kNaThreads a thread would own
// several lines.
inline int block_lines(int64_t lines) {
    int per = 32;
    while (per < kNaThreads && int64_t(per) * 296 < lines) per *= 2;
    return per;
}

// The products of lines [line0, line0 + n) with v: thread t < n returns line
// line0 + t's. Lines are too short (5 to 10 entries on the LPs served) for a
// warp or even a lane group each, so the block streams its entries, which are
// contiguous in CSR, without regard to lines: coalesced index and value
// loads, kNaUnroll gathers in flight per thread, products into shared memory;
// then each thread adds its line's products in order (a line's piece of more
// than kNaLong products is added by its warp). The work per thread does not
// depend on how the entries are spread over the lines. Contains barriers.
// Bound by the latency of its gathers and the matrix stream. Measured on a
// 200,000 x 400,000 LP with 2M entries (91 MB): the call 43 us, the primal
// half 18 and the dual half 23; a warp per line in 1024-line CTAs took 424 us
// (179 each: 22 of 32 lanes idle, and 391 and 196 CTAs for 148 SMs), of which
// 19 went into adding the CTAs' partials in one thread.
__device__ __forceinline__ double block_products(const int64_t* __restrict__ start,
                                                 const int32_t* __restrict__ index,
                                                 const double* __restrict__ values, int64_t line0, int n,
                                                 const double* v, double* prod) {
    const int t = threadIdx.x, lane = t & 31;
    int64_t s = 0, e = 0;
    if (t < n) {
        s = start[line0 + t];
        e = start[line0 + t + 1];
    }
    const int64_t e0 = start[line0], e1 = start[line0 + n];
    double acc = 0.0;
    for (int64_t c0 = e0; c0 < e1; c0 += kNaChunk) {
        const int count = static_cast<int>(e1 - c0 < kNaChunk ? e1 - c0 : kNaChunk);
        for (int k0 = t; k0 < count; k0 += kNaUnroll * kNaThreads) {
            int32_t id[kNaUnroll];
            double w[kNaUnroll];
#pragma unroll
            for (int u = 0; u < kNaUnroll; ++u) {
                const int k = k0 + u * kNaThreads;
                id[u] = k < count ? index[c0 + k] : -1;
                w[u] = k < count ? values[c0 + k] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < kNaUnroll; ++u)
                if (id[u] >= 0) w[u] *= v[id[u]];
#pragma unroll
            for (int u = 0; u < kNaUnroll; ++u)
                if (id[u] >= 0) prod[k0 + u * kNaThreads] = w[u];
        }
        __syncthreads();
        const int a = static_cast<int>(s > c0 ? (s - c0 < count ? s - c0 : count) : 0);
        const int b = static_cast<int>(e > c0 ? (e - c0 < count ? e - c0 : count) : 0);
        const bool wide = b - a > kNaLong;
        if (!wide)
            for (int k = a; k < b; ++k) acc += prod[k];
        for (unsigned todo = __ballot_sync(kFull, wide); todo != 0; todo &= todo - 1) {
            const int owner = __ffs(todo) - 1;
            const int wa = __shfl_sync(kFull, a, owner), wb = __shfl_sync(kFull, b, owner);
            double part = 0.0;
            for (int k = wa + lane; k < wb; k += 32) part += prod[k];
            for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(kFull, part, o);
            if (lane == owner) acc += part;
        }
        __syncthreads();
    }
    return acc;
}

// The CTA's sums of two values a thread, in a fixed order.
__device__ __forceinline__ void cta_sum(double a, double b, double* out_a, double* out_b) {
    __shared__ double red[2][kNaThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(kFull, a, o);
        b += __shfl_xor_sync(kFull, b, o);
    }
    if (lane == 0) {
        red[0][warp] = a;
        red[1][warp] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double sa = 0.0, sb = 0.0;
        for (int w = 0; w < kNaThreads / 32; ++w) {
            sa += red[0][w];
            sb += red[1][w];
        }
        *out_a = sa;
        if (out_b != nullptr) *out_b = sb;
    }
}

__global__ void __launch_bounds__(kNaThreads, 4)
na_primal(int32_t cols, int per, const int64_t* at_start, const int32_t* at_index, const double* at_values,
          const double* c, const double* xl, const double* xu, const double* tau,
          const double* itau, const double* x, const double* y, double mult, double* x_out,
          double* scratch) {
    __shared__ double prod[kNaChunk];
    pdl_trigger();
    double moved = 0.0;
    const int64_t step = int64_t(gridDim.x) * per;
    for (int64_t line0 = int64_t(blockIdx.x) * per; line0 < cols; line0 += step) {
        const int n = static_cast<int>(line0 + per < cols ? per : cols - line0);
        const int64_t j = line0 + threadIdx.x;
        const bool own = static_cast<int>(threadIdx.x) < n;
        double cj = 0.0, prev = 0.0, lo = 0.0, hi = 0.0, tj = 0.0, itj = 0.0;
        if (own) {   // in flight during the gathers
            cj = c[j];
            prev = x[j];
            lo = xl[j];
            hi = xu[j];
            tj = tau[j];
            itj = itau[j];
        }
        const double g = cj + block_products(at_start, at_index, at_values, line0, n, y, prod);
        if (own) {
            const double upd = dmax(lo, dmin(prev - mult * tj * g, hi));
            x_out[j] = upd;
            const double d = upd - prev;
            moved += d * d * itj;
        }
    }
    cta_sum(moved, 0.0, scratch + blockIdx.x, nullptr);
}

__global__ void __launch_bounds__(kNaThreads, 4)
na_dual(int32_t rows, int per, const int64_t* a_start, const int32_t* a_index, const double* a_values,
        const double* rl, const double* ru, const double* sigma, const double* isigma,
        const double* y, const double* ax, const double* x_out, double dmult, double* y_out,
        double* ax_out, double* scratch) {
    __shared__ double prod[kNaChunk];
    pdl_wait();
    pdl_trigger();
    double moved = 0.0, inter = 0.0;
    const int64_t stride = int64_t(gridDim.x) * per;
    for (int64_t line0 = int64_t(blockIdx.x) * per; line0 < rows; line0 += stride) {
        const int n = static_cast<int>(line0 + per < rows ? per : rows - line0);
        const int64_t i = line0 + threadIdx.x;
        const bool own = static_cast<int>(threadIdx.x) < n;
        double axi = 0.0, sg = 0.0, isg = 0.0, prev = 0.0, lo = 0.0, hi = 0.0;
        if (own) {
            axi = ax[i];
            sg = sigma[i];
            isg = isigma[i];
            prev = y[i];
            lo = rl[i];
            hi = ru[i];
        }
        const double next = block_products(a_start, a_index, a_values, line0, n, x_out, prod);
        if (own) {
            const double dact = next - axi;
            const double ext = next + dact;
            const double step = dmax(dmult * sg, 1e-300);
            const double v = prev + step * ext;
            const double upd = dmax(v - step * hi, 0.0) + dmin(v - step * lo, 0.0);
            y_out[i] = upd;
            ax_out[i] = next;
            const double d = upd - prev;
            moved += d * d * isg;
            inter += d * dact;
        }
    }
    double* base = scratch + kNaGridCtas + 2 * blockIdx.x;
    cta_sum(moved, inter, base, base + 1);
}

// Adds the partials this call wrote, in a fixed order: thread t those of CTAs
// t, t + 256, ..., then the block.
__global__ void __launch_bounds__(kNaThreads)
na_reduce(int primal_ctas, int dual_ctas, const double* scratch, double* out) {
    pdl_wait();
    double p = 0.0, d = 0.0, it = 0.0;
    for (int k = threadIdx.x; k < primal_ctas; k += kNaThreads) p += scratch[k];
    for (int k = threadIdx.x; k < dual_ctas; k += kNaThreads) {
        d += scratch[kNaGridCtas + 2 * k];
        it += scratch[kNaGridCtas + 2 * k + 1];
    }
    cta_sum(p, d, out, out + 1);
    __syncthreads();
    cta_sum(it, 0.0, out + 2, nullptr);
}

// A launch that may start while the previous kernel of the stream finishes.
template <class... P, class... A>
cudaError_t launch_after(void (*kernel)(P...), int grid, cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(grid));
    cfg.blockDim = dim3(kNaThreads);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

bool driver_entry(const char* name, void** fn, std::string& error) {
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint(name, fn, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || *fn == nullptr) {
        error = std::string(name) + " unavailable";
        return false;
    }
    return true;
}

// Device address of the scratch array in the current context. The first call
// in each context does the lookup (with that context current); later calls
// reuse it.
double* scratch_in_current_context(std::string& error) {
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (g_ctx_get_current == nullptr || g_ctx_get_id == nullptr) {
        void* current = nullptr;
        void* id = nullptr;
        if (!driver_entry("cuCtxGetCurrent", &current, error) ||
            !driver_entry("cuCtxGetId", &id, error))
            return nullptr;
        g_ctx_get_current = reinterpret_cast<CtxGetCurrent>(current);
        g_ctx_get_id = reinterpret_cast<CtxGetId>(id);
    }
    void* context = nullptr;
    double* fresh = nullptr;
    if (g_ctx_get_current(&context) != 0) {
        error = "cuCtxGetCurrent failed";
        return nullptr;
    }
    if (context == nullptr) {
        // No context is current yet: the runtime makes the device's primary
        // context current while it resolves the symbol.
        const cudaError_t rc = cudaGetSymbolAddress(reinterpret_cast<void**>(&fresh), g_noalloc_scratch);
        if (rc != cudaSuccess) {
            error = std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(rc);
            return nullptr;
        }
        if (g_ctx_get_current(&context) != 0 || context == nullptr) {
            error = "no current CUDA context";
            return nullptr;
        }
    }
    unsigned long long id = 0;
    if (g_ctx_get_id(context, &id) != 0) {
        error = "cuCtxGetId failed";
        return nullptr;
    }
    for (const ScratchEntry& e : g_scratch_entries)
        if (e.context_id == id) return e.address;
    if (fresh == nullptr) {
        const cudaError_t rc = cudaGetSymbolAddress(reinterpret_cast<void**>(&fresh), g_noalloc_scratch);
        if (rc != cudaSuccess) {
            error = std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(rc);
            return nullptr;
        }
    }
    g_scratch_entries.push_back({id, fresh});
    return fresh;
}

int fail(const std::string& message) {
    pdlpgpu_internal_set_error(message.c_str());
    return -1;
}

}  // namespace

extern "C" int32_t pdlpgpu_trial_noalloc(
    int32_t rows, int32_t cols, const int64_t* a_row_start, const int32_t* a_col_index,
    const double* a_values, const int64_t* at_row_start, const int32_t* at_col_index,
    const double* at_values, const double* objective, const double* var_lower,
    const double* var_upper, const double* tau, const double* tau_inverse,
    const double* row_lower, const double* row_upper, const double* sigma,
    const double* sigma_inverse, const double* x, const double* y, const double* ax,
    double step, double weight, double* x_out, double* y_out, double* ax_out,
    double* reductions, void* stream) {
    if (rows < 0 || cols < 0) return fail("pdlpgpu_trial_noalloc: negative dimensions");
    if (rows > kNaMaxLines || cols > kNaMaxLines)
        return fail("pdlpgpu_trial_noalloc: at most 8388608 rows and 8388608 columns");
    if (!(weight > 0.0)) return fail("pdlpgpu_trial_noalloc: weight must be positive");
    // Every pointer a launch would dereference must be given: NULL is refused
    // here, before anything is enqueued, instead of faulting on the device.
    if (reductions == nullptr) return fail("pdlpgpu_trial_noalloc: reductions is NULL");
    if (cols > 0) {
        const void* column_side[] = {at_row_start, at_col_index, at_values, objective, var_lower,
                                     var_upper, tau, tau_inverse, x, x_out};
        for (const void* p : column_side)
            if (p == nullptr)
                return fail("pdlpgpu_trial_noalloc: a column-side pointer (A^T, objective, "
                            "variable bounds, tau, x, x_out) is NULL with cols > 0");
    }
    if (rows > 0) {
        const void* row_side[] = {a_row_start, a_col_index, a_values, row_lower, row_upper,
                                  sigma, sigma_inverse, y, ax, y_out, ax_out};
        for (const void* p : row_side)
            if (p == nullptr)
                return fail("pdlpgpu_trial_noalloc: a row-side pointer (A, row bounds, sigma, "
                            "y, ax, y_out, ax_out) is NULL with rows > 0");
    }
    std::string error;
    double* scratch = scratch_in_current_context(error);
    if (scratch == nullptr) return fail("pdlpgpu_trial_noalloc: " + error);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int per_p = block_lines(cols), per_d = block_lines(rows);
    const auto ctas = [](int64_t lines, int per) {
        return static_cast<int>(std::min<int64_t>((lines + per - 1) / per, kNaGridCtas));
    };
    const int pc = ctas(cols, per_p), dc = ctas(rows, per_d);
    // Only the first launch of the call is ordered after everything before
    // it; with neither rows nor columns that is the sum.
    cudaError_t rc = cudaSuccess;
    if (pc > 0) {
        na_primal<<<pc, kNaThreads, 0, s>>>(cols, per_p, at_row_start, at_col_index, at_values, objective,
                                            var_lower, var_upper, tau, tau_inverse, x, y,
                                            step / weight, x_out, scratch);
        rc = cudaGetLastError();
    }
    if (rc == cudaSuccess && dc > 0) {
        if (pc > 0)
            rc = launch_after(na_dual, dc, s, rows, per_d, a_row_start, a_col_index, a_values, row_lower,
                              row_upper, sigma, sigma_inverse, y, ax, x_out, step * weight, y_out, ax_out,
                              scratch);
        else
            na_dual<<<dc, kNaThreads, 0, s>>>(rows, per_d, a_row_start, a_col_index, a_values, row_lower,
                                              row_upper, sigma, sigma_inverse, y, ax, x_out, step * weight,
                                              y_out, ax_out, scratch);
    }
    if (rc == cudaSuccess) {
        if (pc > 0 || dc > 0) rc = launch_after(na_reduce, 1, s, pc, dc, scratch, reductions);
        else na_reduce<<<1, kNaThreads, 0, s>>>(pc, dc, scratch, reductions);
    }
    const cudaError_t last = cudaGetLastError();
    if (rc == cudaSuccess) rc = last;
    if (rc != cudaSuccess) return fail(std::string("pdlpgpu_trial_noalloc: ") + cudaGetErrorString(rc));
    return 0;
}
