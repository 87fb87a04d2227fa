// The activations that a product may apply to its result before it is stored as bfloat16, shared by the one-block product
// (gemm_tc.cu) and the product on pairs of SMs (gemm_tc_pair.cu).  All are 32-bit, with the fast exponential and
// reciprocal (a few units in the last place, far below the bfloat16 rounding that follows): with short inner widths the
// epilogue, not the products, sets the kernel's time.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace {

// SWIGLU  silu(g) * u                                                        of two products (gate rows, then up rows)
// CLAMPED g' sigmoid(alpha g') (u' + 1), g' = min(g, limit), u' = clamp(u, -limit, limit)    of two products
// RELU2   max(x, 0)^2                                                        of one product
enum : int { ACT_SWIGLU = 0, ACT_CLAMPED = 1, ACT_RELU2 = 2 };

struct ActEpilogue {
    int kind;
    float limit, alpha;
};

__device__ __forceinline__ float act_gated(const ActEpilogue& a, float g, float u) {
    if (a.kind == ACT_CLAMPED) {
        g = fminf(g, a.limit);
        u = fminf(fmaxf(u, -a.limit), a.limit);
        return __fdividef(g, 1.0f + __expf(-a.alpha * g)) * (u + 1.0f);
    }
    return __fdividef(g, 1.0f + __expf(-g)) * u;
}

// 32 tokens of one output column: out[j * stride] = act(g[j], u[j]) for j < left.  All values are made before any is stored, and
// a full run of tokens has no condition: with the condition around each store the compiler put each value's chain (exponential,
// reciprocal) behind its own branch, and a tile's epilogue took 13 us where its products over 1,024 take 4 (1,722 tokens x 2 x
// 3,072 over 1,024: 47.6 -> 24.6 us).
template <int N>
__device__ __forceinline__ void store_gated(const ActEpilogue& a, const uint32_t (&g)[N], const uint32_t (&u)[N], __nv_bfloat16* out,
                                            size_t stride, int left) {
    __nv_bfloat16 v[N];
    if (a.kind == ACT_CLAMPED) {
#pragma unroll
        for (int j = 0; j < N; ++j) v[j] = __float2bfloat16_rn(act_gated({ACT_CLAMPED, a.limit, a.alpha}, __uint_as_float(g[j]), __uint_as_float(u[j])));
    } else {
#pragma unroll
        for (int j = 0; j < N; ++j) v[j] = __float2bfloat16_rn(act_gated({ACT_SWIGLU, 0.0f, 0.0f}, __uint_as_float(g[j]), __uint_as_float(u[j])));
    }
    if (left >= N) {
#pragma unroll
        for (int j = 0; j < N; ++j) out[(size_t)j * stride] = v[j];
    } else {
#pragma unroll
        for (int j = 0; j < N; ++j)
            if (j < left) out[(size_t)j * stride] = v[j];
    }
}

__device__ __forceinline__ float act_single(float x) {
    const float m = fmaxf(x, 0.0f);
    return m * m;
}

}  // namespace
