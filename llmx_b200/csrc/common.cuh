// Shared helpers of the sm_100a kernels: element types, conversions, reductions.
//
// Every exported function is `extern "C"`, takes raw device pointers and a
// stream, launches on that stream and returns the CUDA error code of the launch
// (0 on success).  Nothing here allocates.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include <stdlib.h>

#define LLMX_EXPORT extern "C" __attribute__((visibility("default")))

// Element type codes shared with the Python side.
enum : int { LLMX_F32 = 0, LLMX_BF16 = 1 };

// Error codes above the CUDA range, for argument refusals made on the host.
enum : int { LLMX_ERR_BAD_ARGUMENT = 10001, LLMX_ERR_UNSUPPORTED = 10002 };

__device__ __forceinline__ float to_float(float v) { return v; }
__device__ __forceinline__ float to_float(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T> __device__ __forceinline__ T from_float(float v);
template <> __device__ __forceinline__ float from_float<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_float<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

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

// Sum over a block of up to 1024 threads, in a fixed order (lane tree, then warps in index order),
// so a row's sum does not depend on what else the launch holds.  `scratch` holds 32 floats.
__device__ __forceinline__ float block_sum(float v, float* scratch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    const int nwarps = (blockDim.x + 31) >> 5;
    float total = 0.0f;
    for (int w = 0; w < nwarps; ++w) total += scratch[w];
    return total;
}

// a / b for b >= 1 (or infinite, or not a number) without a branch: the reciprocal refined by a Newton step, the quotient by its
// remainder (Markstein, "Computation of elementary functions on the IBM RISC System/6000", 1990): correctly rounded, a zero's
// sign included, wherever the remainder is a normal number (|a| >= 2^-100), below that within one unit in the last place.  So
// x / (1 + exp(-x)) has the division's bits for every x.  Where the refinement meets an infinity its first guess is the answer.
// (A division with a branch puts each of a thread's values behind its own: chains that could run side by side run one
// after another.)
__device__ __forceinline__ float quotient(float a, float b) {
    const float s = b > 0x1p100f ? 0x1p-64f : 1.0f;          // the reciprocal of what is left is no subnormal number
    const float a_s = a * s;
    b *= s;
    float r0;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(b));
    const float r = fmaf(fmaf(-b, r0, 1.0f), r0, r0);
    const float q0 = a_s * r;
    const float q = fmaf(fmaf(-b, q0, a_s), r, q0);
    return fabsf(q) <= 3.402823466e38f ? copysignf(q, a) : a_s * r0;
}

static inline int launch_status() { return (int)cudaGetLastError(); }

// Dynamic shared memory beyond 48 KB has to be allowed for a kernel, by a limit that belongs to the function and not to the thread
// or stream that sets it.  So every call allows the same: all that a block can have beside what the kernel declares.  (A call
// that set its own size would lower the limit under a launch that another thread had just made room for.)
template <auto KERNEL>
static inline cudaError_t allow_all_smem() {
    static const int most = [] {
        cudaFuncAttributes a = {};
        return cudaFuncGetAttributes(&a, KERNEL) == cudaSuccess ? 227 * 1024 - (int)a.sharedSizeBytes : 0;
    }();
    return cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
}
#define LLMX_ALLOW_SMEM(...)                                                          \
    do {                                                                              \
        if (const cudaError_t allowed = allow_all_smem<__VA_ARGS__>()) return (int)allowed; \
    } while (0)

// ---- programmatic dependent launch --------------------------------------------------------------
// Kernels of a step run one after another on one stream.  Launched with the "programmatic stream
// serialization" attribute, a kernel's blocks may be placed on the SMs and run their prologue (barriers,
// tensor memory, descriptor prefetch) while the kernel before it drains.  The rule every kernel here
// keeps: `pdl_trigger()` first (the next kernel may start arriving), then `pdl_wait()` before the first
// access to global memory another kernel writes or reads.  `pdl_wait()` returns only when the kernel
// before has finished and its writes are visible, so nothing after it can race; without the attribute
// both are no-ops.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

//
// `llmx_launch_overlap` (one per library, exported; build.py `set_overlap` writes it): 0 launches without the attribute, so
// that a kernel starts when everything before it on the stream has ended.
extern "C" {
__attribute__((visibility("default"), weak)) int llmx_launch_overlap = 1;
}

static inline bool llmx_pdl_enabled() {
    if (!llmx_launch_overlap) return false;
    static int on = -1;
    if (on < 0) {
        const char* e = getenv("LLMX_PDL");
        on = (e && e[0] == '0') ? 0 : 1;
    }
    return on == 1;
}

template <typename... KArgs, typename... Args>
static inline void launch_kernel(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                 Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = llmx_pdl_enabled() ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}
