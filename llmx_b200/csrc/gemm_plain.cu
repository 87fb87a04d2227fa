// Plain matrix product on the CUDA cores: C[M, N] (+)= A[M, K] * W[N, K]^T.
//
// This is the product of the true 32-bit path (32-bit inputs, explicit fmaf, no
// reduced-precision matrix mode) and the fallback of the bfloat16 path for widths a
// TMA descriptor cannot take (a row stride that is not a multiple of 16 bytes).
// Each output's sum runs over k in increasing order whatever M is, so a row's result
// does not depend on what else is in the batch (the reference's rule,
// src/backends/backend.hpp:141-150; its kernels: f32.gpu:1034-1084).
//
// Forms with the same bits: up to eight rows a thread an output column (`gemm_plain_few_kernel`, which reads its
// first weights before it waits for the kernel before: W must not be that kernel's output), more than 64 rows 128 x 64 tiles with two
// multiply-adds an instruction (`gemm_plain_many_kernel`), both for K in fours and aligned operands of one type; else 64 x 64 tiles.
#include "common.cuh"

namespace {
constexpr int BM = 64, BN = 64, BK = 16;

template <typename AT, typename WT>
__global__ void __launch_bounds__(256) gemm_plain_kernel(const AT* __restrict__ A, const WT* __restrict__ W,
                                                         float* __restrict__ C, int M, int N, int K, int accumulate) {
    pdl_trigger();
    pdl_wait();
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;

    for (int k0 = 0; k0 < K; k0 += BK) {
        // 64 x 16 elements per operand, 256 threads: four each, consecutive k fastest.
#pragma unroll
        for (int it = 0; it < 4; ++it) {
            const int e = threadIdx.x + it * 256;
            const int r = e >> 4, k = e & 15;
            const int gm = m0 + r, gn = n0 + r, gk = k0 + k;
            As[k][r] = (gm < M && gk < K) ? to_float(A[(size_t)gm * K + gk]) : 0.0f;
            Ws[k][r] = (gn < N && gk < K) ? to_float(W[(size_t)gn * K + gk]) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float a[4], w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[k][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = Ws[k][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int gm = m0 + ty * 4 + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gn = n0 + tx * 4 + j;
            if (gn >= N) continue;
            float* c = C + (size_t)gm * N + gn;
            *c = accumulate ? *c + acc[i][j] : acc[i][j];
        }
    }
}

__device__ __forceinline__ void four(const float* p, float (&v)[4]) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
}
__device__ __forceinline__ void four(const __nv_bfloat16* p, float (&v)[4]) {
    const uint2 x = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x.y));
    v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
}

// Many rows: 128 x 64 outputs a block, 8 x 4 a thread as pairs of neighbouring rows (two multiply-adds an instruction), the next
// 16 of K on their way in registers.  The same sums in the same order, bit for bit.  2,048 x 2,048 over 128: 51 -> 35 us.
constexpr int MM = 128, MN = 64, MK = 16;

template <typename AT, typename WT>
__global__ void __launch_bounds__(256) gemm_plain_many_kernel(const AT* __restrict__ A, const WT* __restrict__ W, float* __restrict__ C,
                                                              int M, int N, int K, int accumulate) {
    pdl_trigger();
    pdl_wait();
    __shared__ __align__(16) float As[MK][MM + 4], Ws[MK][MN + 4];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int m0 = blockIdx.y * MM, n0 = blockIdx.x * MN;
    // Thread t brings four values of K, 4 (t % 4) on, of rows t / 4 and t / 4 + 64 of A and t / 4 of W.
    const int kk = 4 * (threadIdx.x & 3), r = threadIdx.x >> 2;
    float ahead[3][4];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const int row = i < 2 ? m0 + r + 64 * i : n0 + r;
            ahead[i][0] = ahead[i][1] = ahead[i][2] = ahead[i][3] = 0.0f;
            if (k0 + kk < K && row < (i < 2 ? M : N)) {
                if (i < 2) four(A + (size_t)row * K + k0 + kk, ahead[i]);
                else four(W + (size_t)row * K + k0 + kk, ahead[i]);
            }
        }
    };
    unsigned long long acc[4][4];                        // [pair of rows][column]
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
    fetch(0);
    for (int k0 = 0; k0 < K; k0 += MK) {
        __syncthreads();
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            As[kk + u][r] = ahead[0][u];
            As[kk + u][r + 64] = ahead[1][u];
            Ws[kk + u][r] = ahead[2][u];
        }
        __syncthreads();
        if (k0 + MK < K) fetch(k0 + MK);
        const int steps = min(MK, K - k0);               // K is a multiple of four: whole runs of four, in increasing order
#pragma unroll
        for (int k = 0; k < MK; ++k) {
            if (k >= steps) break;
            const ulonglong2 a01 = *reinterpret_cast<const ulonglong2*>(&As[k][8 * ty]), a23 = *reinterpret_cast<const ulonglong2*>(&As[k][8 * ty + 4]);
            const unsigned long long a[4] = {a01.x, a01.y, a23.x, a23.y};
            const float4 w4 = *reinterpret_cast<const float4*>(&Ws[k][4 * tx]);
            const float w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                unsigned long long ww;
                asm("mov.b64 %0, {%1, %1};" : "=l"(ww) : "f"(w[j]));
#pragma unroll
                for (int i = 0; i < 4; ++i) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][j]) : "l"(a[i]), "l"(ww));
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int gm = m0 + 8 * ty + 2 * i + half;
            if (gm >= M) continue;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int gn = n0 + 4 * tx + j;
                if (gn >= N) continue;
                float lo, hi;
                asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(acc[i][j]));
                float* c = C + (size_t)gm * N + gn;
                const float v = half ? hi : lo;
                *c = accumulate ? *c + v : v;
            }
        }
}

// A few rows: a thread an output column, its weight row in pieces of four values, FEW_AHEAD pieces in flight before the
// first is used; A's rows lie in shared memory.  k runs in increasing order, as above, so a row's result is the same bit for
// bit whichever form runs.  Four rows, 4,096 columns over 256: 29 -> 9 us.
constexpr int FEW_ROWS = 8, FEW_COLS = 64, FEW_AHEAD = 8, FEW_BYTES = 40 * 1024;

template <typename AT, typename WT>
__global__ void __launch_bounds__(FEW_COLS) gemm_plain_few_kernel(const AT* __restrict__ A, const WT* __restrict__ W, float* __restrict__ C,
                                                                  int M, int N, int K, int accumulate) {
    pdl_trigger();
    extern __shared__ __align__(16) float rows[];        // [M][K]
    const int n = blockIdx.x * FEW_COLS + threadIdx.x;
    const WT* w = W + (size_t)min(n, N - 1) * K;
    float acc[FEW_ROWS] = {}, ahead[FEW_AHEAD][4];
    // No kernel writes the weights: the first pieces are asked for before the wait.
#pragma unroll
    for (int i = 0; i < FEW_AHEAD; ++i)
        if (4 * i < K) four(w + 4 * i, ahead[i]);
    pdl_wait();
    for (int i = threadIdx.x; i < M * K; i += FEW_COLS) rows[i] = to_float(A[i]);
    __syncthreads();
    for (int k0 = 0; k0 < K; k0 += 4 * FEW_AHEAD) {
        float now[FEW_AHEAD][4];
#pragma unroll
        for (int i = 0; i < FEW_AHEAD; ++i) {
#pragma unroll
            for (int u = 0; u < 4; ++u) now[i][u] = ahead[i][u];
            const int next = k0 + 4 * (FEW_AHEAD + i);
            if (next < K) four(w + next, ahead[i]);
        }
#pragma unroll
        for (int i = 0; i < FEW_AHEAD; ++i) {
            if (k0 + 4 * i >= K) continue;
#pragma unroll
            for (int m = 0; m < FEW_ROWS; ++m) {
                if (m >= M) continue;
                const float4 a = *reinterpret_cast<const float4*>(rows + m * K + k0 + 4 * i);
                acc[m] = fmaf(a.x, now[i][0], acc[m]);
                acc[m] = fmaf(a.y, now[i][1], acc[m]);
                acc[m] = fmaf(a.z, now[i][2], acc[m]);
                acc[m] = fmaf(a.w, now[i][3], acc[m]);
            }
        }
    }
    if (n >= N) return;
#pragma unroll
    for (int m = 0; m < FEW_ROWS; ++m) {
        if (m >= M) continue;
        float* c = C + (size_t)m * N + n;
        *c = accumulate ? *c + acc[m] : acc[m];
    }
}

// A few rows over a short K (the second half of a low-rank pair): 32 columns a block, whose weight rows the block copies to shared
// memory before it waits for the kernel before (a thread reading its own row asked for 16 bytes of 32 rows at a time); a thread
// then has a column of up to two rows (with one row three of the four warps repeat the first one's: the reads decide, not the
// multiply-adds).  The same order of k, the same bits.  Eight weights in a row, 1 to 8 rows, us against a column a thread:
//   4,096 columns    K 32 2.2/3.3   128 3.4/6.1   256 5.0/9.9   512 8.3/17.5
//   32,768 columns   K 32 3.9/5.2   128 8.9/13.7  256 17.8/23.9  512 33.8/42.7
//   65,536 columns   K 32 5.1/6.3   128 15.7/15.9  256 24.7/28.0  384 40.5/39.7  512 59.8/51.2
// The blocks' copies of more than 256 values a row leave room for two or three of them on an SM, and so many columns are more rounds of
// such blocks: there a column a thread is the faster one (at 128 values of 65,536 columns the two are equal).
constexpr int SHORT_COLS = 32, SHORT_THREADS = 128, SHORT_K = 512, SHORT_WIDE_K = 256, SHORT_MANY_COLS = 32768;

__global__ void __launch_bounds__(SHORT_THREADS) gemm_plain_short_kernel(const float* __restrict__ A, const float* __restrict__ W,
                                                                         float* __restrict__ C, int M, int N, int K, int accumulate) {
    pdl_trigger();
    extern __shared__ __align__(16) float short_mem[];   // weights [32][K + 4], then A's rows [M][K]
    const int n0 = blockIdx.x * SHORT_COLS, pieces = K / 4, stride = K + 4;
    float* rows = short_mem + SHORT_COLS * stride;
    for (int i = threadIdx.x; i < SHORT_COLS * pieces; i += SHORT_THREADS) {
        const int r = i / pieces, c = 4 * (i - r * pieces);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(short_mem + r * stride + c)),
                     "l"(W + (size_t)min(n0 + r, N - 1) * K + c) : "memory");
    }
    pdl_wait();
    for (int i = threadIdx.x; i < M * pieces; i += SHORT_THREADS)
        *reinterpret_cast<float4*>(rows + 4 * i) = *reinterpret_cast<const float4*>(A + 4 * i);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const int col = threadIdx.x & 31, m0 = threadIdx.x >> 5, n = n0 + col;
    const float* w = short_mem + col * stride;
    const float* a0 = rows + min(m0, M - 1) * K;
    const float* a1 = rows + min(m0 + 4, M - 1) * K;
    float acc0 = 0.0f, acc1 = 0.0f;
#pragma unroll 4
    for (int k = 0; k < K; k += 4) {
        const float4 x = *reinterpret_cast<const float4*>(w + k), y = *reinterpret_cast<const float4*>(a0 + k), z = *reinterpret_cast<const float4*>(a1 + k);
        acc0 = fmaf(y.x, x.x, acc0), acc1 = fmaf(z.x, x.x, acc1);
        acc0 = fmaf(y.y, x.y, acc0), acc1 = fmaf(z.y, x.y, acc1);
        acc0 = fmaf(y.z, x.z, acc0), acc1 = fmaf(z.z, x.z, acc1);
        acc0 = fmaf(y.w, x.w, acc0), acc1 = fmaf(z.w, x.w, acc1);
    }
    if (n >= N) return;
    if (m0 < M) {
        float* c = C + (size_t)m0 * N + n;
        *c = accumulate ? *c + acc0 : acc0;
    }
    if (m0 + 4 < M) {
        float* c = C + (size_t)(m0 + 4) * N + n;
        *c = accumulate ? *c + acc1 : acc1;
    }
}
}  // namespace

LLMX_EXPORT int llmx_gemm_plain(const void* A, int a_dtype, const void* W, int w_dtype, float* C, int M, int N, int K,
                                int accumulate, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return LLMX_ERR_BAD_ARGUMENT;
    const size_t few_bytes = (size_t)M * K * sizeof(float);
    if (M <= FEW_ROWS && K % 4 == 0 && K <= (N > SHORT_MANY_COLS ? SHORT_WIDE_K : SHORT_K) && a_dtype == LLMX_F32 && w_dtype == LLMX_F32 && !(((uintptr_t)A | (uintptr_t)W) & 15)) {
        const size_t bytes = ((size_t)SHORT_COLS * (K + 4) + (size_t)M * K) * sizeof(float);
        if (bytes > 48 * 1024) LLMX_ALLOW_SMEM(gemm_plain_short_kernel);
        launch_kernel(gemm_plain_short_kernel, dim3((N + SHORT_COLS - 1) / SHORT_COLS), dim3(SHORT_THREADS), bytes, stream, (const float*)A,
                      (const float*)W, C, M, N, K, accumulate);
        return launch_status();
    }
    if (M <= FEW_ROWS && K % 4 == 0 && few_bytes <= FEW_BYTES && !((uintptr_t)W & 15) && a_dtype == w_dtype) {
        const dim3 few((N + FEW_COLS - 1) / FEW_COLS);
        if (a_dtype == LLMX_F32)
            launch_kernel(gemm_plain_few_kernel<float, float>, few, dim3(FEW_COLS), few_bytes, stream, (const float*)A, (const float*)W, C, M, N, K, accumulate);
        else if (a_dtype == LLMX_BF16)
            launch_kernel(gemm_plain_few_kernel<__nv_bfloat16, __nv_bfloat16>, few, dim3(FEW_COLS), few_bytes, stream, (const __nv_bfloat16*)A, (const __nv_bfloat16*)W, C, M, N, K, accumulate);
        else
            return LLMX_ERR_UNSUPPORTED;
        return launch_status();
    }
    const long long many_rows = ((long long)M + MM - 1) / MM;
    if (M > BM && K % 4 == 0 && many_rows <= 65535 && !(((uintptr_t)A | (uintptr_t)W) & 15) && a_dtype == w_dtype) {
        const dim3 many((N + MN - 1) / MN, (unsigned)many_rows);
        if (a_dtype == LLMX_F32)
            launch_kernel(gemm_plain_many_kernel<float, float>, many, dim3(256), 0, stream, (const float*)A, (const float*)W, C, M, N, K, accumulate);
        else if (a_dtype == LLMX_BF16)
            launch_kernel(gemm_plain_many_kernel<__nv_bfloat16, __nv_bfloat16>, many, dim3(256), 0, stream, (const __nv_bfloat16*)A, (const __nv_bfloat16*)W, C, M, N, K, accumulate);
        else
            return LLMX_ERR_UNSUPPORTED;
        return launch_status();
    }
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (grid.y > 65535) return LLMX_ERR_UNSUPPORTED;
    if (a_dtype == LLMX_F32 && w_dtype == LLMX_F32)
        launch_kernel(gemm_plain_kernel<float, float>, dim3(grid), dim3(256), 0, stream, (const float*)A, (const float*)W, C, M, N, K, accumulate);
    else if (a_dtype == LLMX_BF16 && w_dtype == LLMX_BF16)
        launch_kernel(gemm_plain_kernel<__nv_bfloat16, __nv_bfloat16>, dim3(grid), dim3(256), 0, stream, (const __nv_bfloat16*)A, (const __nv_bfloat16*)W, C, M, N, K, accumulate);
    else
        return LLMX_ERR_UNSUPPORTED;
    return launch_status();
}
