// Shared helpers of the kernel sources: element types, conversions, the
// activation formulas and the C ABI's error convention.
//
// Every exported launcher returns 0 on success and a non-zero code otherwise;
// the text of the last failure is read with <lib>_last_error().  Launchers
// never allocate device memory, never synchronise and launch on the stream
// they are given.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>

typedef __nv_bfloat16 bf16;

// Element type codes of the C ABI.
enum { DT_F32 = 0, DT_BF16 = 1 };

// Epilogue codes of the linear kernels.
//   EPI_STORE      out = acc + bias
//   EPI_GELU_TANH  out = gelu_tanh(acc + bias)
//   EPI_GELU_ERF   out = gelu_erf(acc + bias)
//   EPI_ADD        out(fp32) += acc + bias        (residual sum kept in 32-bit)
//   EPI_RELU_SQ    out = max(acc + bias, 0)^2
//   EPI_SILU       out = u / (1 + exp(-u)), u = acc + bias
enum { EPI_STORE = 0, EPI_GELU_TANH = 1, EPI_GELU_ERF = 2, EPI_ADD = 3, EPI_RELU_SQ = 4, EPI_SILU = 5 };

template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<bf16>(bf16 v) { return __bfloat162float(v); }

template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ bf16 from_f32<bf16>(float v) { return __float2bfloat16_rn(v); }

// gelu, tanh form: 0.5 u (1 + tanh(0.7978845608 (u + 0.044715 u^3))), the
// formula of the reference's feed-forward (engine/include/gelu_math.h:6-11).
__device__ __forceinline__ float gelu_tanh_f(float u) {
    const float c = 0.7978845608f;
    const float k = 0.044715f;
    float arg = c * (u + k * u * u * u);
    return 0.5f * u * (1.0f + tanhf(arg));
}

// gelu, exact form: 0.5 u (1 + erf(u / sqrt(2))) (engine/src/gelu.c:5-9).
__device__ __forceinline__ float gelu_erf_f(float u) {
    return 0.5f * u * (1.0f + erff(u / sqrtf(2.0f)));
}

// gelu, tanh form, with the hardware's approximate tanh (relative error about 2^-11): the
// result is rounded to bfloat16 (2^-9) right after, and an exact tanh for every element of a
// feed-forward product costs more SM time than the product itself.  For kernels whose output is
// bfloat16 only.
__device__ __forceinline__ float gelu_tanh_fast(float u) {
    float t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(0.7978845608f * (u + 0.044715f * u * u * u)));
    return 0.5f * u * (1.0f + t);
}

template <int EPI> __device__ __forceinline__ float apply_activation(float v) {
    if (EPI == EPI_GELU_TANH) return gelu_tanh_f(v);
    if (EPI == EPI_GELU_ERF) return gelu_erf_f(v);
    if (EPI == EPI_RELU_SQ) return v > 0.0f ? v * v : 0.0f;
    if (EPI == EPI_SILU) return v / (1.0f + expf(-v));
    return v;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Sum over a block of up to 1024 threads; every thread gets the result.
// `scratch` holds 33 floats of shared memory.
__device__ __forceinline__ float block_sum(float v, float* scratch) {
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int n_warps = (blockDim.x + 31) >> 5;
    v = warp_sum(v);
    __syncthreads();                 // scratch may still be read from a previous call
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    if (warp == 0) {
        float t = lane < n_warps ? scratch[lane] : 0.0f;
        t = warp_sum(t);
        if (lane == 0) scratch[32] = t;
    }
    __syncthreads();
    return scratch[32];
}

// The same with one barrier, for a kernel's first use of `slots` (one float a warp): every thread adds the warps' sums itself,
// in warp order.
__device__ __forceinline__ float block_sum_once(float v, float* slots) {
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) slots[threadIdx.x >> 5] = v;
    __syncthreads();
    const int n_warps = (blockDim.x + 31) >> 5;
    float total = 0.0f;
    for (int w = 0; w < n_warps; w++) total += slots[w];
    return total;
}

// c[16 x 8] += a[16 x 16] b[16 x 8] over the lanes of a warp, bfloat16 operands, 32-bit sums.
__device__ __forceinline__ void mma_bf16_16816(float& c0, float& c1, float& c2, float& c3, uint32_t a0, uint32_t a1,
                                               uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                 "{%0, %1, %2, %3};"
                 : "+f"(c0), "+f"(c1), "+f"(c2), "+f"(c3)
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

#define MLLM_ERROR_BUFFER 512

// ---- programmatic dependent launch ---------------------------------------------------------
//
// A kernel launched with launch_kernel(true, ...) may be scheduled while the kernel before it
// on the stream still runs: its CTAs take the SMs that the earlier kernel's CTAs leave, set up
// what needs no memory of the step (barriers, tensor memory, index arithmetic) and then wait
// in wait_for_earlier_kernels(), which returns when every earlier kernel has completed and its
// writes are visible.  A kernel says with dependents_may_start(), at its start, that the next one
// may be scheduled as soon as all of its own CTAs run.  Both calls do nothing in a kernel that was
// launched the ordinary way, and stream capture keeps the dependency as an edge of the graph.
//
// Before it has passed that wait no thread writes global memory, and none reads what another
// kernel of the same step writes.  What it may read there:
//   - weights and what lies beside them, which no kernel writes;
//   - the step's arrays (positions, block tables, entries, work lists), which a step's first kernel
//     brings, but for the token ids, which resolve_tokens may write;
//   - where its caller says so (first_new, rows_ahead, state_ahead): cached rows of positions before an
//     entry's first new one, and the state that this kernel alone writes.  (A state that another kernel
//     of the step writes is not read ahead, whatever its caller knows about the steps.)
// The last two hold because steps are apart: control_kernel, which brings the arrays, waits for all
// kernels ahead and lets no dependents start, and the kernel behind it (resolve_tokens or an embedding)
// is launched AFTER_THE_KERNELS_AHEAD, so that everything behind that one runs when the arrays are there
// and every earlier step has ended.  An embedding whose first kernel is launched as a dependent must
// not say `begins_apart` (parts/base.py): the engine then puts resolve_tokens before it.
__device__ __forceinline__ void dependents_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_earlier_kernels() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// A kernel that reads weights before that wait takes what other kernels of the step wrote through a pointer that has passed
// here behind it: loads through a `const ... __restrict__` parameter count as loads of memory that nobody writes, and the
// compiler may move them ahead of the wait (a filter kernel read rows that the product before it had not yet written, once
// in a few replayed steps).
template <typename T> __device__ __forceinline__ T* behind_the_wait(T* p) {
    asm volatile("" : "+l"(p) : : "memory");
    return p;
}

// How a launch is made: as a dependent where `g_dependent_launch` of its library says so, or after the kernels ahead have ended.
// A kernel of few long blocks is launched the second way: as a dependent its blocks go to whatever SMs have room while other
// kernels' waiting blocks hold the rest, several to an SM, and stay there (per launch within a replayed step, early against
// not: a gated delta rule over two prompts of 1,000 tokens 680 against 513 us, latent attention of one token in 32 parts 23.5 against
// 12.4, a 32-bit product of 240 x 768 x 768 73 against 41).  So is the kernel behind the one that brings a step's
// arrays (see above).
constexpr bool AFTER_THE_KERNELS_AHEAD = false;

// (cluster: the CTAs of a thread block cluster, or x = 0 for a launch without clusters)
template <typename... Params, typename... Args>
static cudaError_t launch_kernel_in_clusters(bool dependent, dim3 cluster, void (*kernel)(Params...), dim3 grid, dim3 block,
                                             size_t shared_bytes, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t config = {};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = shared_bytes;
    config.stream = stream;
    cudaLaunchAttribute attributes[2];
    unsigned count = 0;
    if (dependent) {
        attributes[count].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attributes[count].val.programmaticStreamSerializationAllowed = 1;
        count++;
    }
    if (cluster.x != 0) {
        attributes[count].id = cudaLaunchAttributeClusterDimension;
        attributes[count].val.clusterDim.x = cluster.x;
        attributes[count].val.clusterDim.y = cluster.y;
        attributes[count].val.clusterDim.z = cluster.z;
        count++;
    }
    config.attrs = attributes;
    config.numAttrs = count;
    return cudaLaunchKernelEx(&config, kernel, Params(args)...);
}
template <typename... Params, typename... Args>
static cudaError_t launch_kernel(bool dependent, void (*kernel)(Params...), dim3 grid, dim3 block, size_t shared_bytes,
                                 cudaStream_t stream, Args... args) {
    return launch_kernel_in_clusters(dependent, dim3(0, 1, 1), kernel, grid, block, shared_bytes, stream, args...);
}

#define MLLM_DEFINE_ERROR_API(prefix)                                              \
    static thread_local char g_error_text[MLLM_ERROR_BUFFER] = "";                 \
    extern "C" const char* prefix##_last_error(void) { return g_error_text; }      \
    static int fail(const char* what) {                                            \
        snprintf(g_error_text, MLLM_ERROR_BUFFER, "%s", what);                     \
        return 1;                                                                  \
    }                                                                              \
    static int check_launch(const char* kernel) {                                  \
        cudaError_t e = cudaGetLastError();                                        \
        if (e == cudaSuccess) return 0;                                            \
        snprintf(g_error_text, MLLM_ERROR_BUFFER, "%s: %s", kernel,                \
                 cudaGetErrorString(e));                                           \
        return 2;                                                                  \
    }                                                                              \
    /* whether this library's kernels are launched as dependents (see above) */    \
    static int g_dependent_launch = 1;                                             \
    extern "C" void prefix##_set_dependent_launch(int on) { g_dependent_launch = on; } \
    static int launched(cudaError_t e, const char* kernel) {                       \
        if (e == cudaSuccess) return check_launch(kernel);                         \
        snprintf(g_error_text, MLLM_ERROR_BUFFER, "%s: %s", kernel,                \
                 cudaGetErrorString(e));                                           \
        return 2;                                                                  \
    }
