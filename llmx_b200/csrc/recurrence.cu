// Linear recurrences over a matrix state per (request, head): decayed linear attention and the gated delta rule.
//
// Per head the state S is [D, V] (key width x value width), 32-bit, one per request in a state slot, and for the
// step's rows t of a request, in order:
//     a_t = decay_h (a constant per head)                  or  g_t (a gate per row and head)
//     u_t = v_t                                            or  beta_t * (v_t - a_t * S^T k_t)      (delta rule)
//     S  <- a_t * S + k_t u_t^T
//     o_t = S^T q_t                                        (the read-out sees the row's own write)
// Two more forms share the code.  The scaled form (a selective state space): a_t a gate per row and head,
// u_t = beta_t * v_t (beta the row's step size), and o_t += skip_h * v_t.  The delta rule with a decay per key
// channel: S <- diag(g_t) S with g_t [D] per row and head, then u_t = beta_t * (v_t - S^T k_t), S <- S + k_t u_t^T.
// Gated linear attention is that without the correction: S <- diag(g_t) S + k_t v_t^T; its gates are made by
// `llmx_channel_decay`.
// Column j of S (the D values that meet v's entry j) never meets another column, so the work is cut by columns:
// a few threads own one column, each holding a share of its values in registers for all of the request's rows;
// the two dot products are sums over a lane's values and then over the column's lanes by shuffles.  A block holds
// columns of one head (and of one request); the rows' q and k are read by every worker from the cache.  The state is
// read from `slot_in` (zeros at a request's first token, whatever the slot holds) and written to `slot_out` once,
// after the request's last row of the step.  State layout in a slot: [H][V][D] floats, so a worker's column is
// contiguous.
//
// The short convolution in front of the delta rule lives here too (`llmx_conv_prepare`): a causal filter of
// `taps` taps per channel over the request's rows, continued from the last taps-1 inputs kept in the state slot,
// then silu; q and k heads made unit vectors (x / sqrt(sum x^2 + 1e-6), q also times D^-1/2); beta = sigmoid(b);
// g = exp(-exp(A_log) * softplus(a + dt_bias)).  All of it 32-bit.  The filter may carry a bias per channel, the unit
// scaling may be left out (no q or k channels named), and the gates come in three kinds (`gate_kind`): 0, the delta
// rule's (g per head, then beta = sigmoid); 1, a selective state space's (dt = softplus(a + dt_bias) with no clamp,
// then g = exp(-exp(A_log) dt) and dt itself per head); 2, the delta rule's with a decay per key channel
// (beta = sigmoid per head, and g [heads * D] from a second matrix `decay_in` [rows, heads * D] with dt_bias
// [heads * D]).
#include "common.cuh"
#include <math.h>
#include <type_traits>

namespace {
constexpr int REC_THREADS = 128;
// What a row does to the state: a constant decay per head; the delta rule with one gate per row and head; a gate per
// row and head with the input scaled by beta and a skip term; the delta rule with a gate per row, head and key channel;
// such a gate alone.
constexpr int M_CONST = 0, M_DELTA = 1, M_SCALED = 2, M_DELTA_VEC = 3, M_VEC = 4;
constexpr bool has_channel_gate(int mode) { return mode == M_DELTA_VEC || mode == M_VEC; }
constexpr bool has_beta(int mode) { return mode != M_CONST && mode != M_VEC; }

// The form for steps of a row or a few: LANES (8) threads share one column of the state, each holding PER of its D
// values (D <= LANES * PER), so a sum over the lanes is three shuffle steps; a block of 128 threads owns 16 columns of
// one head.  A row's q, k, v and gates are fetched one row ahead.
template <int PER, int LANES, int MODE>
__global__ void __launch_bounds__(REC_THREADS)
recurrence_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v, int q_stride,
                  int k_stride, int v_stride, const float* __restrict__ decay, const float* __restrict__ gate,
                  const float* __restrict__ beta, int gate_stride, int beta_stride, const float* __restrict__ skip,
                  float* __restrict__ state, long long slot_floats,
                  const int* __restrict__ row_start, const int* __restrict__ row_count, const int* __restrict__ history,
                  const int* __restrict__ slot_in, const int* __restrict__ slot_out, float* __restrict__ out, int heads,
                  int qk_heads, int D, int V) {
    pdl_trigger();
    pdl_wait();
    constexpr int COLS = REC_THREADS / LANES;
    const int r = blockIdx.x;
    const int blocks_per_head = (V + COLS - 1) / COLS;
    const int h = blockIdx.y / blocks_per_head;
    const int col = (blockIdx.y % blocks_per_head) * COLS + threadIdx.x / LANES;
    const int lane = threadIdx.x % LANES;
    const int n = row_count[r];
    if (n <= 0) return;
    const bool live = col < V;
    const int j = live ? col : V - 1;                 // idle workers shadow a real column and store nothing
    const int a0 = row_start[r];
    const int hq = h / (heads / qk_heads);
    float S[PER];
    const float* sin_ = state + (size_t)slot_in[r] * slot_floats + ((size_t)h * V + j) * D;
    const bool fresh = history[r] == 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int d = lane + i * LANES;
        S[i] = (!fresh && d < D) ? sin_[d] : 0.0f;
    }
    constexpr bool VEC = has_channel_gate(MODE);
    constexpr int GP = VEC ? PER : 1;
    const float dec = MODE == M_CONST ? decay[h] : VEC ? 1.0f : 0.0f;
    const float sk = MODE == M_SCALED && skip != nullptr ? skip[h] : 0.0f;
    float kk[PER], qq[PER], nk[PER], nq[PER], gg[GP], ng[GP];
    float u = 0.0f, a = dec, bt = 0.0f, nu = 0.0f, na = dec, nb = 0.0f;
    auto fetch = [&](int t, float* fk, float* fq, float* fg, float& fu, float& fa, float& fb) {
        const size_t row = (size_t)(a0 + t);
        const float* qp = q + row * q_stride + (size_t)hq * D;
        const float* kp = k + row * k_stride + (size_t)hq * D;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int d = lane + i * LANES;
            fk[i] = d < D ? kp[d] : 0.0f;
            fq[i] = d < D ? qp[d] : 0.0f;
        }
        fu = v[row * v_stride + (size_t)h * V + j];
        if (MODE == M_DELTA || MODE == M_SCALED) fa = gate[row * gate_stride + h];
        if (has_beta(MODE)) fb = beta[row * beta_stride + h];
        if (VEC) {
            const float* gp = gate + row * gate_stride + (size_t)h * D;
#pragma unroll
            for (int i = 0; i < GP; ++i) {
                const int d = lane + i * LANES;
                fg[i] = d < D ? gp[d] : 1.0f;
            }
        }
    };
    fetch(0, kk, qq, gg, u, a, bt);
    for (int t = 0; t < n; ++t) {
        if (t + 1 < n) fetch(t + 1, nk, nq, ng, nu, na, nb);
        const float raw = u;
        if (VEC) {
#pragma unroll
            for (int i = 0; i < PER; ++i) S[i] *= gg[i < GP ? i : 0];
        }
        if (MODE == M_DELTA || MODE == M_DELTA_VEC) {
            float dot = 0.0f;
#pragma unroll
            for (int i = 0; i < PER; ++i) dot = fmaf(S[i], kk[i], dot);
#pragma unroll
            for (int o = LANES / 2; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
            u = bt * (u - a * dot);
        }
        if (MODE == M_SCALED) u = bt * u;
        float acc = 0.0f;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            S[i] = fmaf(a, S[i], kk[i] * u);
            acc = fmaf(S[i], qq[i], acc);
        }
#pragma unroll
        for (int o = LANES / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (MODE == M_SCALED) acc = fmaf(sk, raw, acc);
        if (live && lane == 0) out[(size_t)(a0 + t) * ((size_t)heads * V) + (size_t)h * V + j] = acc;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            kk[i] = nk[i];
            qq[i] = nq[i];
        }
#pragma unroll
        for (int i = 0; i < GP; ++i) gg[i] = ng[i];
        u = nu;
        a = (MODE == M_DELTA || MODE == M_SCALED) ? na : dec;
        bt = nb;
    }
    if (live) {
        float* sout = state + (size_t)slot_out[r] * slot_floats + ((size_t)h * V + j) * D;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int d = lane + i * LANES;
            if (d < D) sout[d] = S[i];
        }
    }
}

// The wide form for long runs of rows: 16 or 32 columns of one head a block.  A group of LANES lanes shares CPL columns: a lane
// reads PER values of a row's q and k (and gates) from shared memory once and uses them for its share of all the columns.
// (Shared memory gives a lane 4 bytes a cycle: one column a group of eight lanes was bound by that, 162 cycles a row and
// warp.)  A lane's values are pairs in 64-bit registers, two multiply-adds an instruction.  Four more warps bring the rows' q, k, v and gates to shared memory by cp.async, sixteen rows
// a buffer (four a warp), two or three buffers, handed over by named barriers: the workers address no global memory for
// their inputs.
//
// With a delta rule a row waits for the sum k . S over the group's lanes, and the next row for that row.  Four rows t are
// therefore taken at a time: p_t = k_t . S (after the decays of the rows up to t) against the state before the four, whose
// sums over the lanes go side by side, and what the rows between add to it, (k_t . k_s) u_s, comes from the six products
// of the four keys with one another -- the same for all columns, made by the warp that copied the four rows:
//     x_t = p_t;  for s < t:  x_t = a_s x_t + (k_t . k_s) u_s         (channel decays: inside p_t and the products)
//     u_t = beta_t (v_t - a_t x_t)
// The state then takes the four rows in order.  The read-outs, which nothing waits for, are summed over the lanes eight rows
// at a time.
//
// 16 heads of 128 x 128, 2,048 rows of one request, us before (a warp two columns, or with a correction one, copies by all
// threads) and now: constant decay 245 -> 166, delta rule 673 -> 259, scaled 265 -> 172, delta rule with channel decays 715 -> 307,
// channel decays alone 298 -> 186; 32 heads: 362 -> 235, 949 -> 362 and (channel decays) 1,037 -> 449; eight requests of 190 rows:
// 122 -> 110, 329 -> 159 and 339 -> 192.  A row's multiply-adds are 48 to 64 cycles of a warp, its reads of shared memory and
// shuffles 50 to 90 cycles of the SM; the rest is the chain of the four rows' corrections (delta rule) and the hand-over.
constexpr int WIDE_CH = 16, WIDE_SUMS = 8;
constexpr int WIDE_COPY_WARPS = 4, WIDE_COPY_ROWS = WIDE_CH / WIDE_COPY_WARPS;
constexpr int WIDE_GRAM = 8 * WIDE_COPY_WARPS;          // floats a buffer has for its keys' products: six (of eight) for four rows

__device__ __forceinline__ void barrier_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void barrier_arrive(int id, int threads) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

__device__ __forceinline__ void cp_async_4(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

__device__ __forceinline__ void cp_async_16f(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// Two 32-bit numbers in a 64-bit register, and operations on both.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pair(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float pair_sum(f32x2 v) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
    return lo + hi;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// A lane holds PER values of its column, d = 4 (lane + LANES i) + 0 .. 3; a row's vectors are padded with zeros to LANES PER values,
// so that a lane's share is whole 16-byte reads from shared memory without a condition (neighbouring lanes read a run).
template <int PER, int LANES>
__device__ __forceinline__ void read_share(const float* p, int sub, f32x2 (&out)[PER / 2]) {
#pragma unroll
    for (int i = 0; i < PER / 4; ++i) {
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(p + 4 * (sub + LANES * i));
        out[2 * i] = x.x, out[2 * i + 1] = x.y;
    }
}

// The sum of a lane's share of a dot product, in two chains.
template <int N>
__device__ __forceinline__ float share_dot(const f32x2 (&a)[N], const f32x2 (&b)[N]) {
    f32x2 s0 = mul2(a[0], b[0]), s1 = mul2(a[1], b[1]);
#pragma unroll
    for (int i = 2; i < N; i += 2) {
        s0 = fma2(a[i], b[i], s0);
        s1 = fma2(a[i + 1], b[i + 1], s1);
    }
    return pair_sum(add2(s0, s1));
}

template <int PER, int LANES, int CPL, int COLS, int MODE>
__global__ void __launch_bounds__(COLS / CPL * LANES + 32 * WIDE_COPY_WARPS, 1)
recurrence_wide_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v, int q_stride,
                       int k_stride, int v_stride, const float* __restrict__ decay, const float* __restrict__ gate,
                       const float* __restrict__ beta, int gate_stride, int beta_stride, const float* __restrict__ skip,
                       float* __restrict__ state, long long slot_floats,
                       const int* __restrict__ row_start, const int* __restrict__ row_count,
                       const int* __restrict__ history, const int* __restrict__ slot_in,
                       const int* __restrict__ slot_out, float* __restrict__ out, int heads, int qk_heads, int D, int V, int stages) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ __align__(16) float stage[];   // [stages]{[WIDE_CH][row_floats]: q (Dp), k (Dp), [gates per channel (Dp)], v (the block's columns), gate, beta, pad; gram}
    constexpr bool VEC = has_channel_gate(MODE), CORRECTED = MODE == M_DELTA || MODE == M_DELTA_VEC;
    constexpr int NV = VEC ? 3 : 2;                  // vectors of D values a row brings
    constexpr int WORKERS = COLS / CPL * LANES, THREADS = WORKERS + 32 * WIDE_COPY_WARPS;
    constexpr int BLK = PER == 16 ? 1 : 4;           // rows taken at a time (four of 16 values a lane: too many registers)
    constexpr int Dp = PER * LANES;                  // the vectors' padded length (the pad is cleared once and never written by the copies)
    constexpr int row_floats = NV * Dp + COLS + 4;   // a multiple of 4: every row starts on 16 bytes
    constexpr int stage_floats = WIDE_CH * row_floats + WIDE_GRAM;
    constexpr int P2 = PER / 2;
    constexpr int FULL = 1, EMPTY = 4;               // named barriers: buffer s is filled (FULL + s), is free again (EMPTY + s)
    const int r = blockIdx.x;
    const int blocks_per_head = (V + COLS - 1) / COLS;
    const int h = blockIdx.y / blocks_per_head;
    const int first_col = (blockIdx.y % blocks_per_head) * COLS;
    const int n = row_count[r];
    if (n <= 0) return;
    const int a0 = row_start[r];
    const int chunks = (n + WIDE_CH - 1) / WIDE_CH;
    if (D < Dp) {
        for (int i = threadIdx.x; i < stages * stage_floats; i += THREADS) stage[i] = 0.0f;
        __syncthreads();
    }

    if (threadIdx.x >= WORKERS) {
        // ---- a copying warp: four rows of every chunk, pieces of 16 bytes where addresses and widths allow it, else single
        // values.  A lane has one piece of a vector (more with wide vectors), of all four rows, and one of the rows' small pieces.
        const int lane = threadIdx.x & 31, first = (threadIdx.x - WORKERS) / 32 * WIDE_COPY_ROWS;
        const bool vec = D % 4 == 0 && q_stride % 4 == 0 && k_stride % 4 == 0 && ((uintptr_t)q & 15) == 0 && ((uintptr_t)k & 15) == 0 &&
                         (!VEC || (gate_stride % 4 == 0 && ((uintptr_t)gate & 15) == 0));
        const bool vec_v = V % 4 == 0 && v_stride % 4 == 0 && ((uintptr_t)v & 15) == 0 && first_col + COLS <= V;
        const size_t row0 = (size_t)(a0 + first);
        const int hq = h / (heads / qk_heads);
        const float* src[3] = {q + row0 * q_stride + (size_t)hq * D, k + row0 * k_stride + (size_t)hq * D,
                               VEC ? gate + row0 * gate_stride + (size_t)h * D : nullptr};
        const int strides[3] = {q_stride, k_stride, gate_stride};
        const float* src_v = v + row0 * v_stride + (size_t)h * V;
        const float* src_gate = MODE == M_DELTA || MODE == M_SCALED ? gate + row0 * gate_stride + h : nullptr;
        const float* src_beta = has_beta(MODE) ? beta + row0 * beta_stride + h : nullptr;
        auto issue = [&](int chunk, float* buf) {
            const int rows = min(WIDE_COPY_ROWS, n - chunk * WIDE_CH - first);      // negative where the last chunk ends before this warp's rows
            buf += first * row_floats;
            const size_t t0 = (size_t)chunk * WIDE_CH;
#pragma unroll
            for (int w = 0; w < NV; ++w) {
                const float* from = src[w] + t0 * strides[w];
#pragma unroll
                for (int t = 0; t < WIDE_COPY_ROWS; ++t) {
                    if (t >= rows) break;
                    float* to = buf + t * row_floats + w * Dp;
                    if (vec) {
#pragma unroll
                        for (int e = 0; e < Dp; e += 128)
                            if (e + 4 * lane < D) cp_async_16f(to + e + 4 * lane, from + e + 4 * lane);
                    } else {
                        for (int e = lane; e < D; e += 32) cp_async_4(to + e, from + e);
                    }
                    from += strides[w];
                }
            }
            const float* from = src_v + t0 * v_stride;
            if (vec_v) {
                constexpr int PIECES = COLS / 4;     // of a row: 32 lanes have four rows' at once
                static_assert(WIDE_COPY_ROWS * PIECES <= 32, "a lane a piece");
                const int t = lane / PIECES, e = 4 * (lane % PIECES);
                if (t < rows) cp_async_16f(buf + t * row_floats + NV * Dp + e, from + (size_t)t * v_stride + first_col + e);
            } else {
                for (int i = lane; i < WIDE_COPY_ROWS * COLS; i += 32)
                    if (i / COLS < rows)
                        cp_async_4(buf + i / COLS * row_floats + NV * Dp + i % COLS, from + (size_t)(i / COLS) * v_stride + min(first_col + i % COLS, V - 1));
            }
            if (src_gate != nullptr && lane < rows) cp_async_4(buf + lane * row_floats + NV * Dp + COLS, src_gate + (t0 + lane) * gate_stride);
            if (src_beta != nullptr && lane >= 16 && lane - 16 < rows)
                cp_async_4(buf + (lane - 16) * row_floats + NV * Dp + COLS + 1, src_beta + (t0 + lane - 16) * beta_stride);
        };
        for (int c = 0; c < stages - 1; ++c) {
            if (c < chunks) issue(c, stage + (size_t)c * stage_floats);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        int at = 0;                                  // c % stages
        for (int c = 0; c < chunks; ++c) {
            if (stages == 3) asm volatile("cp.async.wait_group 1;" ::: "memory");
            else asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncwarp();                            // this warp's rows of chunk c have landed
            float* buf = stage + (size_t)at * stage_floats;
            if constexpr (CORRECTED && BLK == 4) {
                // k_t . k_s for s < t, with channel decays (k_t g_t .. g_{s+1}) . k_s.  Rows that a last chunk does not have
                // give numbers that nobody reads.
                static_assert(WIDE_COPY_ROWS == BLK, "a copying warp's rows are the rows taken together");
                float g[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                for (int e = 0; e < Dp; e += 128) {
                    const int d = e + 4 * lane;
                    if (d >= Dp) continue;
                    const float* rowp = buf + first * row_floats + d;
                    float4 kr[4], gr[4];
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        kr[t] = *reinterpret_cast<const float4*>(rowp + t * row_floats + Dp);
                        if (VEC) gr[t] = *reinterpret_cast<const float4*>(rowp + t * row_floats + 2 * Dp);
                    }
#pragma unroll
                    for (int t = 1; t < 4; ++t) {
                        float4 w = kr[t];
#pragma unroll
                        for (int s = 2; s >= 0; --s) {
                            if (s >= t) continue;
                            if (VEC) w.x *= gr[s + 1].x, w.y *= gr[s + 1].y, w.z *= gr[s + 1].z, w.w *= gr[s + 1].w;
                            float& sum = g[t * (t - 1) / 2 + s];
                            sum = fmaf(w.x, kr[s].x, fmaf(w.y, kr[s].y, fmaf(w.z, kr[s].z, fmaf(w.w, kr[s].w, sum))));
                        }
                    }
                }
                // Sums over the lanes: each gives half of the sums it holds to its partner and takes the partner's share of the
                // other half until one is left; the lanes that hold the same one add theirs up.
                int index = 0;
#pragma unroll
                for (int o = 16, held = 8; o >= 1; o >>= 1) {
                    if (held == 1) {
                        g[0] += __shfl_xor_sync(0xffffffffu, g[0], o);
                        continue;
                    }
                    held >>= 1;
                    const bool high = lane & o;
                    if (high) index += held;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (i >= held) continue;
                        const float keep = high ? g[i + held] : g[i], give = high ? g[i] : g[i + held];
                        g[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                    }
                }
                if (lane % 4 == 0) buf[WIDE_CH * row_floats + 2 * first + index] = g[0];
            }
            __threadfence_block();
            barrier_arrive(FULL + at, THREADS);
            const int next = c + stages - 1, next_at = at == 0 ? stages - 1 : at - 1;      // next % stages
            if (next < chunks) {
                if (c > 0) barrier_sync(EMPTY + next_at, THREADS);        // the workers have left chunk c - 1
                issue(next, stage + (size_t)next_at * stage_floats);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            at = at + 1 == stages ? 0 : at + 1;
        }
        return;
    }

    // ---- the workers
    const int sub = threadIdx.x % LANES, mine = threadIdx.x / LANES * CPL;      // the group's first column in the block
    const int col = first_col + mine;                // columns past V shadow the last one and store nothing
    f32x2 S[CPL][P2];
#pragma unroll
    for (int w = 0; w < CPL; ++w) {
        const bool fresh = history[r] == 0;
        const float* from = state + (size_t)slot_in[r] * slot_floats + ((size_t)h * V + min(col + w, V - 1)) * D;
#pragma unroll
        for (int i = 0; i < P2; ++i) {
            const int d = 4 * (sub + LANES * (i / 2)) + 2 * (i % 2);
            S[w][i] = pair(!fresh && d < D ? from[d] : 0.0f, !fresh && d + 1 < D ? from[d + 1] : 0.0f);
        }
    }
    const float dec = MODE == M_CONST ? decay[h] : 1.0f;
    const float sk = MODE == M_SCALED && skip != nullptr ? skip[h] : 0.0f;
    for (int c = 0, at = 0; c < chunks; ++c, at = at + 1 == stages ? 0 : at + 1) {
        const float* buf = stage + (size_t)at * stage_floats;
        const int rows = min(WIDE_CH, n - c * WIDE_CH);
        barrier_sync(FULL + at, THREADS);
        // N rows from t0 on, their corrections together; leaves the lane's shares of the read-outs in acc.
        auto take = [&](int t0, auto count, float* acc) {
            constexpr int N = decltype(count)::value;
            const float* rowp = buf + (size_t)t0 * row_floats;
            f32x2 kk[N][P2], gg[VEC ? N : 1][P2];
            float u[N][CPL], a[N];
#pragma unroll
            for (int i = 0; i < N; ++i) {
                read_share<PER, LANES>(rowp + i * row_floats + Dp, sub, kk[i]);
                if constexpr (VEC) read_share<PER, LANES>(rowp + i * row_floats + 2 * Dp, sub, gg[i]);
                const float* smalls = rowp + i * row_floats + NV * Dp;
                a[i] = MODE == M_DELTA || MODE == M_SCALED ? smalls[COLS] : dec;
                if constexpr (!CORRECTED)
#pragma unroll
                    for (int w = 0; w < CPL; ++w) u[i][w] = MODE == M_SCALED ? smalls[COLS + 1] * smalls[mine + w] : smalls[mine + w];
            }
            if constexpr (CORRECTED) {
                static_assert(CPL <= 2, "a half of the group a column");
                float x[N][CPL];
#pragma unroll
                for (int w = 0; w < CPL; ++w) {
                    f32x2 decayed[P2];                   // channel decays: the state before the rows, decayed up to row i
#pragma unroll
                    for (int d = 0; d < P2; ++d) decayed[d] = S[w][d];
#pragma unroll
                    for (int i = 0; i < N; ++i) {
                        if constexpr (VEC)
#pragma unroll
                            for (int d = 0; d < P2; ++d) decayed[d] = mul2(decayed[d], gg[i][d]);    // past D everything is zero and stays so
                        x[i][w] = share_dot(decayed, kk[i]);
                    }
                }
                // The sums over the group's lanes; with two columns each half of the lanes ends with one column's.
                const bool second = CPL == 2 && (sub & (LANES / 2));
                float own[N];
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    own[i] = x[i][0];
                    if constexpr (CPL == 2) {
                        const float give = second ? x[i][0] : x[i][1];
                        own[i] = (second ? x[i][1] : x[i][0]) + __shfl_xor_sync(0xffffffffu, give, LANES / 2);
                    }
                }
#pragma unroll
                for (int o = LANES / CPL / 2; o > 0; o >>= 1)
#pragma unroll
                    for (int i = 0; i < N; ++i) own[i] += __shfl_xor_sync(0xffffffffu, own[i], o);
                const float* gram = buf + WIDE_CH * row_floats + 2 * t0;
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    const float* smalls = rowp + i * row_floats + NV * Dp;
                    float y = own[i];
#pragma unroll
                    for (int j = 0; j < i; ++j) y = fmaf(gram[i * (i - 1) / 2 + j], own[j], VEC ? y : a[j] * y);
                    own[i] = smalls[COLS + 1] * (smalls[mine + (second ? 1 : 0)] - a[i] * y);          // u_i from here on
                }
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    u[i][0] = own[i];
                    if constexpr (CPL == 2) {
                        const float other = __shfl_xor_sync(0xffffffffu, own[i], LANES / 2);
                        u[i][0] = second ? other : own[i];
                        u[i][1] = second ? own[i] : other;
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const f32x2 a2 = pair(a[i], a[i]);
                f32x2 qq[P2];
                read_share<PER, LANES>(rowp + i * row_floats, sub, qq);
#pragma unroll
                for (int w = 0; w < CPL; ++w) {
                    const f32x2 u2 = pair(u[i][w], u[i][w]);
#pragma unroll
                    for (int d = 0; d < P2; ++d) S[w][d] = fma2(VEC ? gg[VEC ? i : 0][d] : a2, S[w][d], mul2(kk[i][d], u2));
                    acc[i * CPL + w] = share_dot(S[w], qq);
                }
            }
        };
        auto store = [&](int t, int w, float sum) {
            if (MODE == M_SCALED) sum = fmaf(sk, buf[(size_t)t * row_floats + NV * Dp + mine + w], sum);
            if (col + w < V) out[(size_t)(a0 + c * WIDE_CH + t) * ((size_t)heads * V) + (size_t)h * V + col + w] = sum;
        };
        int t0 = 0;
        for (; t0 + WIDE_SUMS <= rows; t0 += WIDE_SUMS) {
            constexpr int SUMS = WIDE_SUMS * CPL;        // [row][column]
            static_assert(SUMS <= LANES, "a lane a sum");
            float acc[SUMS];
#pragma unroll
            for (int i = 0; i < WIDE_SUMS; i += BLK) take(t0 + i, std::integral_constant<int, BLK>{}, acc + i * CPL);
            // At each step a lane gives half of the sums it holds to its partner and takes the partner's share of the other
            // half; when one is left, the lanes that hold the same one add theirs up.
            int held = SUMS, index = 0;
#pragma unroll
            for (int o = LANES / 2; o >= 1; o >>= 1) {
                if (held == 1) {
                    acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
                    continue;
                }
                held >>= 1;
                const bool high = sub & o;
                if (high) index += held;
#pragma unroll
                for (int i = 0; i < SUMS / 2; ++i) {
                    if (i >= held) continue;
                    const float keep = high ? acc[i + held] : acc[i], give = high ? acc[i] : acc[i + held];
                    acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                }
            }
            if (sub % (LANES / SUMS) == 0) store(t0 + index / CPL, index % CPL, acc[0]);
        }
        for (; t0 < rows; ++t0) {                    // a request's last rows, one by one
            float acc[CPL];
            take(t0, std::integral_constant<int, 1>{}, acc);
#pragma unroll
            for (int w = 0; w < CPL; ++w) {
#pragma unroll
                for (int o = LANES / 2; o >= 1; o >>= 1) acc[w] += __shfl_xor_sync(0xffffffffu, acc[w], o);
                if (sub == 0) store(t0, w, acc[w]);
            }
        }
        if (c + stages < chunks) barrier_arrive(EMPTY + at, THREADS);
    }
#pragma unroll
    for (int w = 0; w < CPL; ++w) {
        if (col + w >= V) continue;
        float* to = state + (size_t)slot_out[r] * slot_floats + ((size_t)h * V + col + w) * D;
#pragma unroll
        for (int i = 0; i < P2; ++i) {
            const int d = 4 * (sub + LANES * (i / 2)) + 2 * (i % 2);
            float lo, hi;
            asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(S[w][i]));
            if (d < D) to[d] = lo;
            if (d + 1 < D) to[d + 1] = hi;
        }
    }
}

// One block per row (conv, activation, unit vectors, gates) and, after those, one block per request (the inputs the
// next step's convolution will need).
__device__ __forceinline__ float softplus_f(float z) { return z > 20.0f ? z : log1pf(expf(z)); }

__global__ void __launch_bounds__(256)
conv_prepare_kernel(const float* __restrict__ proj, int stride, int first, int channels, int q_channels, int k_channels,
                    const float* __restrict__ taps_w, const float* __restrict__ taps_b, int taps,
                    float* __restrict__ ready, const float* __restrict__ a_log, const float* __restrict__ dt_bias,
                    int b_off, int a_off, int gate_kind, const float* __restrict__ decay_in, int decay_stride,
                    float* __restrict__ gates, int gates_stride, int heads, int D, float q_factor,
                    float* __restrict__ state, long long slot_floats, long long conv_off,
                    const int* __restrict__ row_request, const int* __restrict__ row_start,
                    const int* __restrict__ row_count, const int* __restrict__ history, const int* __restrict__ slot_in,
                    const int* __restrict__ slot_out, int rows) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ float vals[];                  // the row's channels after the filter and silu
    const int keep = taps - 1;
    proj += first;                                   // the filtered channels start at column `first` of the projections
    if ((int)blockIdx.x >= rows) {
        const int r = blockIdx.x - rows;
        const int n = row_count[r], a0 = row_start[r], hist = history[r];
        if (n <= 0) return;
        const float* old = state + (size_t)slot_in[r] * slot_floats + conv_off;
        float* fresh = state + (size_t)slot_out[r] * slot_floats + conv_off;
        for (int c = threadIdx.x; c < channels; c += blockDim.x)
            for (int s = 0; s < keep; ++s) {         // slot_in and slot_out differ: the rows' blocks read the old inputs meanwhile
                const int ii = n - keep + s;         // the input's place relative to the step's first row
                float x = 0.0f;
                if (ii >= 0) x = proj[(size_t)(a0 + ii) * stride + c];
                else if (hist + ii >= 0) x = old[(size_t)(keep + ii) * channels + c];
                fresh[(size_t)s * channels + c] = x;
            }
        return;
    }
    const int row = blockIdx.x;
    const int r = row_request[row];
    const int i0 = row - row_start[r], hist = history[r];
    const float* old = state + (size_t)slot_in[r] * slot_floats + conv_off;
    for (int c = threadIdx.x; c < channels; c += blockDim.x) {
        float y = taps_b ? taps_b[c] : 0.0f;
        for (int jt = 0; jt < taps; ++jt) {
            const int ii = i0 - keep + jt;
            float x = 0.0f;
            if (ii >= 0) x = proj[(size_t)(row_start[r] + ii) * stride + c];
            else if (hist + ii >= 0) x = old[(size_t)(keep + ii) * channels + c];
            y = fmaf(taps_w[(size_t)c * taps + jt], x, y);
        }
        vals[c] = y / (1.0f + expf(-y));
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int unit_heads = (q_channels + k_channels) / D;          // q heads, then k heads
    for (int g = warp; g < unit_heads; g += warps) {
        float s = 0.0f;
        for (int d = lane; d < D; d += 32) s = fmaf(vals[g * D + d], vals[g * D + d], s);
        s = warp_sum(s);
        const float f = (g * D < q_channels ? q_factor : 1.0f) / sqrtf(s + 1e-6f);
        for (int d = lane; d < D; d += 32) ready[(size_t)row * channels + g * D + d] = vals[g * D + d] * f;
    }
    for (int c = q_channels + k_channels + threadIdx.x; c < channels; c += blockDim.x) ready[(size_t)row * channels + c] = vals[c];
    proj -= first;
    float* grow = gates + (size_t)row * gates_stride;
    if (gate_kind == 2) {
        for (int h = threadIdx.x; h < heads; h += blockDim.x)
            grow[h] = 1.0f / (1.0f + expf(-proj[(size_t)row * stride + b_off + h]));
        for (int c = threadIdx.x; c < heads * D; c += blockDim.x) {
            const float z = decay_in[(size_t)row * decay_stride + c] + dt_bias[c];
            grow[heads + c] = expf(-expf(a_log[c / D]) * softplus_f(z));
        }
        return;
    }
    for (int h = threadIdx.x; h < heads; h += blockDim.x) {
        const float z = proj[(size_t)row * stride + a_off + h] + dt_bias[h];
        if (gate_kind == 1) {
            const float dt = z > 20.0f ? z : log1pf(expf(z));      // the same function beyond 20 up to rounding: no clamp of dt itself
            grow[h] = expf(-expf(a_log[h]) * dt);
            grow[heads + h] = dt;
        } else {
            const float b = proj[(size_t)row * stride + b_off + h];
            grow[h] = expf(-expf(a_log[h]) * softplus_f(z));
            grow[heads + h] = 1.0f / (1.0f + expf(-b));
        }
    }
}

// The same where channels come in fours: a thread owns four neighbouring channels (16-byte reads and writes) of a run of rows,
// whose last taps - 1 inputs it keeps, so an input is read once for all the outputs it enters; the D / 4 lanes of a head sum
// its squares by shuffles.  A block has up to 1,024 channels of `run` rows, or those channels of a request's kept inputs, or
// the gates of the rows: a few rows (decoding) spread over as many blocks as the channels make, where one block a row
// took them 256 at a time, each waiting for the one before: 8 rows of
// 4,096 channels 28 -> 5.6 us, 4 rows of 8,192 and 6,144 channels 45 -> 5.9 us; 2,048 rows of 4,096 channels 51 -> 31 us, with
// a decay per key channel 76 -> 60, 1,201 rows of 8,192 with such decays 129 -> 73 us (bound by its exponentials and
// logarithms: 40 % of the issue slots with three blocks an SM).
constexpr int CONV_THREADS = 256, CONV_RUN = 16, CONV_TAPS = 4, CONV_AHEAD = 2;

__device__ __forceinline__ float4 load_four(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float silu_f(float y) { return quotient(y, 1.0f + expf(-y)); }

__global__ void __launch_bounds__(CONV_THREADS, 3)
conv_prepare_four_kernel(const float* __restrict__ proj, int stride, int first, int channels, int q_channels, int k_channels,
                         const float* __restrict__ taps_w, const float* __restrict__ taps_b, int taps,
                         float* __restrict__ ready, const float* __restrict__ a_log, const float* __restrict__ dt_bias,
                         int b_off, int a_off, int gate_kind, const float* __restrict__ decay_in, int decay_stride,
                         float* __restrict__ gates, int gates_stride, int heads, int D, float q_factor,
                         float* __restrict__ state, long long slot_floats, long long conv_off,
                         const int* __restrict__ row_request, const int* __restrict__ row_start,
                         const int* __restrict__ row_count, const int* __restrict__ history, const int* __restrict__ slot_in,
                         const int* __restrict__ slot_out, int rows, int run, int row_blocks, int gate_blocks) {
    pdl_trigger();
    const int keep = taps - 1;
    // The gates' blocks come first: they are the longest.
    const bool conv = (int)blockIdx.y >= gate_blocks;
    const int c = (((int)blockIdx.y - gate_blocks) * CONV_THREADS + (int)threadIdx.x) * 4;
    const bool mine = conv && c < channels;
    // The filter's weights are written by no kernel: they are read before the wait.  w[j]: tap j of the four channels.
    float4 w[CONV_TAPS], bias = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int j = 0; j < CONV_TAPS; ++j) w[j] = bias;
    if (mine) {
        float* wv = reinterpret_cast<float*>(w);
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int j = 0; j < CONV_TAPS; ++j)
                if (j < taps) wv[4 * j + u] = taps_w[(size_t)(c + u) * taps + j];
        if (taps_b) bias = load_four(taps_b + c);
    }
    pdl_wait();
    if ((int)blockIdx.x >= row_blocks) {
        // The inputs the next step's filter will need.
        if (!mine) return;
        const int r = blockIdx.x - row_blocks;
        const int n = row_count[r], a0 = row_start[r], hist = history[r];
        if (n <= 0) return;
        const float* old = state + (size_t)slot_in[r] * slot_floats + conv_off;
        float* fresh = state + (size_t)slot_out[r] * slot_floats + conv_off;
        for (int s = 0; s < keep; ++s) {             // slot_in and slot_out differ: the rows' blocks read the old inputs meanwhile
            const int ii = n - keep + s;
            float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (ii >= 0) x = load_four(proj + (size_t)(a0 + ii) * stride + first + c);
            else if (hist + ii >= 0) x = load_four(old + (size_t)(keep + ii) * channels + c);
            *reinterpret_cast<float4*>(fresh + (size_t)s * channels + c) = x;
        }
        return;
    }
    const int row0 = blockIdx.x * run, row_end = min(rows, row0 + run);
    if (!conv) {
        // Gates: `per` a row, a thread one of them for all of the block's rows.
        const int per = gate_kind == 2 ? heads * D : heads;
        const int g = (int)blockIdx.y * CONV_THREADS + (int)threadIdx.x;
        if (g >= per) return;
        const float rate = -expf(a_log[gate_kind == 2 ? g / D : g]), bias_g = dt_bias[g];
#pragma unroll 4
        for (int row = row0; row < row_end; ++row) {
            float* grow = gates + (size_t)row * gates_stride;
            const float* prow = proj + (size_t)row * stride;
            const float z = (gate_kind == 2 ? decay_in[(size_t)row * decay_stride + g] : prow[a_off + g]) + bias_g;
            const float beta = gate_kind != 1 && g < heads ? quotient(1.0f, 1.0f + expf(-prow[b_off + g])) : 0.0f;
            if (gate_kind == 2) {
                grow[heads + g] = expf(rate * softplus_f(z));
                if (g < heads) grow[g] = beta;
            } else if (gate_kind == 1) {
                const float dt = z > 20.0f ? z : log1pf(expf(z));      // the same function beyond 20 up to rounding: no clamp of dt itself
                grow[g] = expf(rate * dt);
                grow[heads + g] = dt;
            } else {
                grow[g] = expf(rate * softplus_f(z));
                grow[heads + g] = beta;
            }
        }
        return;
    }
    const bool unit = c < q_channels + k_channels;   // the same for all lanes of a head: heads are whole
    const float factor = c < q_channels ? q_factor : 1.0f;
    float4 x[CONV_TAPS];                             // x[j]: the input under tap j
    float4 ahead[CONV_AHEAD];                        // the next rows' inputs
#pragma unroll
    for (int i = 0; i < CONV_AHEAD; ++i)
        ahead[i] = mine && row0 + i < row_end ? load_four(proj + (size_t)(row0 + i) * stride + first + c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    int left = 0;                                    // rows of the request at hand that are still to come
#pragma unroll
    for (int j = 0; j < CONV_TAPS; ++j) x[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int row1 = row0; row1 < row_end; row1 += CONV_AHEAD)
#pragma unroll
    for (int turn = 0; turn < CONV_AHEAD; ++turn) {
        const int row = row1 + turn;
        if (row >= row_end) break;
        const float4 now = ahead[turn];
        if (mine && row + CONV_AHEAD < row_end) ahead[turn] = load_four(proj + (size_t)(row + CONV_AHEAD) * stride + first + c);
        if (left == 0) {
            // The first row of the block or of a request: the inputs before it, from earlier rows or the state.
            const int r = row_request[row];
            const int i0 = row - row_start[r], hist = history[r];
            left = row_count[r] - i0;
            if (mine) {
                const float* old = state + (size_t)slot_in[r] * slot_floats + conv_off;
#pragma unroll
                for (int j = 0; j < CONV_TAPS; ++j) {
                    const int ii = i0 - keep + j;        // tap j's input of this row, as this row's place in the request has it
                    if (j >= keep) continue;
                    x[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (ii >= 0) x[j] = load_four(proj + (size_t)(row_start[r] + ii) * stride + first + c);
                    else if (hist + ii >= 0) x[j] = load_four(old + (size_t)(keep + ii) * channels + c);
                }
            }
        }
        --left;
        float4 y = bias;
#pragma unroll
        for (int j = 0; j < CONV_TAPS; ++j) {
            if (j >= taps) continue;
            const float4 v = j == keep ? now : x[j];
            y.x = fmaf(w[j].x, v.x, y.x);
            y.y = fmaf(w[j].y, v.y, y.y);
            y.z = fmaf(w[j].z, v.z, y.z);
            y.w = fmaf(w[j].w, v.w, y.w);
        }
#pragma unroll
        for (int j = 0; j + 1 < CONV_TAPS; ++j)
            if (j < keep) x[j] = j + 1 == keep ? now : x[j + 1];
        y = make_float4(silu_f(y.x), silu_f(y.y), silu_f(y.z), silu_f(y.w));
        // Every lane takes part in the shuffles; only heads that are made unit vectors use the sum.
        float s = fmaf(y.x, y.x, fmaf(y.y, y.y, fmaf(y.z, y.z, y.w * y.w)));
        if (q_channels + k_channels > 0) {
            for (int o = D / 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (unit) {
                const float f = factor / sqrtf(s + 1e-6f);
                y.x *= f, y.y *= f, y.z *= f, y.w *= f;
            }
        }
        if (mine) *reinterpret_cast<float4*>(ready + (size_t)row * channels + c) = y;
    }
}

// Decays per key channel through a low-rank pair, in 32-bit: z = low W2^T + bias, decay = sigmoid(z)^(1 / tau); `low` is the
// pair's inner values (a run of columns of the projections), `w2t` W2 transposed [rank][channels].  In passing the same
// channels of q (columns q_off .. of the projections) are multiplied by `q_factor`.  A thread a channel, DECAY_ROWS rows.
constexpr int DECAY_ROWS = 8, DECAY_THREADS = 128, DECAY_RANK = 64;

__global__ void __launch_bounds__(DECAY_THREADS)
channel_decay_kernel(float* __restrict__ proj, int stride, int rows, int low_off, int rank, const float* __restrict__ w2t,
                     const float* __restrict__ bias, float inv_tau, float* __restrict__ decay, int channels, int q_off, float q_factor) {
    pdl_trigger();
    pdl_wait();
    __shared__ float low[DECAY_RANK][DECAY_ROWS];
    const int c = blockIdx.x * DECAY_THREADS + threadIdx.x;
    const int r0 = blockIdx.y * DECAY_ROWS, n = min(DECAY_ROWS, rows - r0);
    const float b = bias && c < channels ? bias[c] : 0.0f;
    float z[DECAY_ROWS], qv[DECAY_ROWS];
#pragma unroll
    for (int r = 0; r < DECAY_ROWS; ++r) {
        z[r] = b;
        qv[r] = c < channels && r < n ? proj[(size_t)(r0 + r) * stride + q_off + c] : 0.0f;      // on its way during the sums
    }
    for (int k0 = 0; k0 < rank; k0 += DECAY_RANK) {
        const int kn = min(DECAY_RANK, rank - k0);
        __syncthreads();
        for (int i = threadIdx.x; i < kn * DECAY_ROWS; i += DECAY_THREADS) {
            const int r = i / kn, k = i - r * kn;
            low[k][r] = r < n ? proj[(size_t)(r0 + r) * stride + low_off + k0 + k] : 0.0f;
        }
        __syncthreads();
        if (c < channels)
#pragma unroll 8
            for (int k = 0; k < kn; ++k) {
                const float w = w2t[(size_t)(k0 + k) * channels + c];
#pragma unroll
                for (int r = 0; r < DECAY_ROWS; ++r) z[r] = fmaf(low[k][r], w, z[r]);
            }
    }
    if (c >= channels) return;
#pragma unroll
    for (int r = 0; r < DECAY_ROWS; ++r) {
        if (r >= n) break;
        const float log_sigmoid = fminf(z[r], 0.0f) - log1pf(expf(-fabsf(z[r])));
        decay[(size_t)(r0 + r) * channels + c] = expf(log_sigmoid * inv_tau);
        proj[(size_t)(r0 + r) * stride + q_off + c] = qv[r] * q_factor;
    }
}

template <int MODE>
int launch_recurrence(int D, bool wide, int requests, cudaStream_t stream, const float* q, const float* k, const float* v,
                      int q_stride, int k_stride, int v_stride, const float* decay, const float* gate, const float* beta,
                      int gate_stride, int beta_stride, const float* skip, float* state, long long slot_floats, const int* row_start, const int* row_count,
                      const int* history, const int* slot_in, const int* slot_out, float* out, int heads, int qk_heads,
                      int V) {
#define LLMX_REC(P, L)                                                                                                    \
    do {                                                                                                                  \
        const long long by = (long long)heads * ((V + REC_THREADS / L - 1) / (REC_THREADS / L));                          \
        if (by > 65535) return LLMX_ERR_UNSUPPORTED;                                                                      \
        launch_kernel(recurrence_kernel<P, L, MODE>, dim3(requests, (unsigned)by), dim3(REC_THREADS), 0, stream, q, k, v,  \
                      q_stride, k_stride, v_stride, decay, gate, beta, gate_stride, beta_stride, skip, state,          \
                      slot_floats, row_start, row_count, history, slot_in, slot_out, out, heads, qk_heads, D, V);       \
        return launch_status();                                                                                           \
    } while (0)
    if (wide) {
#define LLMX_WIDE_COLS(P, L, W, C)                                                                                                \
    do {                                                                                                                  \
        const long long by = (long long)heads * ((V + C - 1) / C);                                                        \
        if (by > 65535) return LLMX_ERR_UNSUPPORTED;                                                                      \
        const size_t buffer = ((size_t)WIDE_CH * ((has_channel_gate(MODE) ? 3 : 2) * P * L + C + 4) + WIDE_GRAM) * sizeof(float); \
        const int stages = 3 * buffer <= 200 * 1024 ? 3 : 2;                                                              \
        const size_t smem = stages * buffer;                                                                              \
        if (smem > 200 * 1024) return LLMX_ERR_UNSUPPORTED;                                                               \
        if (smem > 48 * 1024) LLMX_ALLOW_SMEM(recurrence_wide_kernel<P, L, W, C, MODE>);                                  \
        launch_kernel(recurrence_wide_kernel<P, L, W, C, MODE>, dim3(requests, (unsigned)by), dim3(C / W * L + 32 * WIDE_COPY_WARPS), \
                      smem, stream, q, k, v, q_stride, k_stride, v_stride, decay, gate, beta, gate_stride, beta_stride, skip, state, \
                      slot_floats, row_start, row_count, history, slot_in, slot_out, out, heads, qk_heads, D, V, stages); \
        return launch_status();                                                                                           \
    } while (0)
        // 32 columns a block (its rows are copied half as often) once blocks of 16 would be more than the 148 SMs take at once.
#define LLMX_WIDE(P, L, W)                                                                                                \
    do {                                                                                                                  \
        if ((long long)requests * heads * ((V + 15) / 16) > 148) LLMX_WIDE_COLS(P, L, W, 32);                             \
        LLMX_WIDE_COLS(P, L, W, 16);                                                                                      \
    } while (0)
        // Values a lane, lanes, columns a group: without a correction more lanes and columns (nothing waits for the sums).
        constexpr bool corrected = MODE == M_DELTA || MODE == M_DELTA_VEC;
        if (D <= 32) LLMX_WIDE(4, 8, 1);
        if (D <= 64) LLMX_WIDE(4, 16, 2);
        if (D <= 128) {
            if constexpr (corrected) LLMX_WIDE(8, 16, 2);
            else LLMX_WIDE(4, 32, 4);
        }
        if (D <= 256) LLMX_WIDE_COLS(8, 32, 2, 16);
        if (D <= 512) LLMX_WIDE_COLS(16, 32, 1, 16);
#undef LLMX_WIDE_COLS
#undef LLMX_WIDE
    } else {
        if (D <= 16) LLMX_REC(2, 8);
        if (D <= 32) LLMX_REC(4, 8);
        if (D <= 64) LLMX_REC(8, 8);
        if (D <= 128) LLMX_REC(16, 8);
        if (D <= 256) LLMX_REC(32, 8);
        if (D <= 512) LLMX_REC(16, 32);          // a warp a column: 64 values a lane would not stay in registers
    }
#undef LLMX_REC
    return LLMX_ERR_UNSUPPORTED;
}
}  // namespace

// q, k [rows, qk_heads * D] and v [rows, heads * V] floats with row strides of their own (they may lie inside one wider
// matrix).  `mode` 0: a constant `decay` [heads].  1: the delta rule, `gate` and `beta` [rows, .] (row strides
// `gate_stride`, `beta_stride`, entry h).  2: the scaled form, a = gate, u = beta * v, out += skip_h * v (`skip` [heads]
// or null).  3: the delta rule with `gate` [rows, heads * D] (entry h * D + d), a decay per key channel.  4: `gate` as in 3,
// u = v (gated linear attention; no beta).  `state`: the
// slots' storage, `slot_floats` apart, the recurrence's [H][V][D] at its start; out [rows, heads * V] floats.  The
// metadata arrays are the step's, on the device.
LLMX_EXPORT int llmx_linear_recurrence(const float* q, const float* k, const float* v, int q_stride, int k_stride,
                                       int v_stride, int mode, const float* decay, const float* gate, const float* beta,
                                       int gate_stride, int beta_stride, const float* skip, float* state,
                                       long long slot_floats, const int* row_start, const int* row_count,
                                       const int* history, const int* slot_in, const int* slot_out, float* out,
                                       int requests, int heads, int qk_heads, int D, int V, int max_rows,
                                       cudaStream_t stream) {
    if (requests <= 0) return 0;
    if (heads <= 0 || qk_heads <= 0 || heads % qk_heads || D <= 0 || V <= 0 || D > 512) return LLMX_ERR_UNSUPPORTED;
    if (mode < 0 || mode > 4 || (mode == M_CONST ? decay == nullptr : (gate == nullptr || (beta == nullptr && has_beta(mode)))))
        return LLMX_ERR_BAD_ARGUMENT;
    // `max_rows`: the most rows one request brings.  Beyond eight the wide form runs, whose sums go in another order: a row's last
    // bits then depend on how its request was cut and on what else is in the step.  A caller that wants neither says 1.
    const bool wide = max_rows > 8;
#define LLMX_MODE(M)                                                                                                      \
    return launch_recurrence<M>(D, wide, requests, stream, q, k, v, q_stride, k_stride, v_stride, decay, gate, beta,      \
                                gate_stride, beta_stride, skip, state, slot_floats, row_start, row_count, history, slot_in, \
                                slot_out, out, heads, qk_heads, V)
    if (mode == M_CONST) LLMX_MODE(M_CONST);
    if (mode == M_DELTA) LLMX_MODE(M_DELTA);
    if (mode == M_SCALED) LLMX_MODE(M_SCALED);
    if (mode == M_DELTA_VEC) LLMX_MODE(M_DELTA_VEC);
    LLMX_MODE(M_VEC);
#undef LLMX_MODE
}

// proj [rows, stride]: columns first .. first + channels - 1 are filtered: q (q_channels), k (k_channels), each of whole
// heads of D values that are made unit vectors, and the rest; columns b_off + h and a_off + h hold the rows' beta and
// decay (or step size) projections.  ready [rows, channels] receives the channels after filter (+ `taps_b` if given),
// silu and unit scaling.  gates [rows, gates_stride]: kind 0: g [heads], beta [heads]; kind 1: g [heads], dt [heads];
// kind 2: beta [heads], g [heads * D] made from `decay_in` [rows, heads * D] (row stride `decay_stride`).
// taps_w [channels, taps].  The last taps-1 inputs of a request lie at `conv_off` floats into its state slot,
// [taps - 1][channels].
LLMX_EXPORT int llmx_conv_prepare(const float* proj, int stride, int first, int channels, int q_channels, int k_channels,
                                  const float* taps_w, const float* taps_b, int taps, float* ready, const float* a_log,
                                  const float* dt_bias, int b_off, int a_off, int gate_kind, const float* decay_in,
                                  int decay_stride, float* gates, int gates_stride, int heads, int D, float q_factor,
                                  float* state, long long slot_floats, long long conv_off, const int* row_request,
                                  const int* row_start, const int* row_count, const int* history, const int* slot_in,
                                  const int* slot_out, int rows, int requests, cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (taps < 1 || channels <= 0 || D <= 0 || q_channels % D || k_channels % D || q_channels + k_channels > channels ||
        gate_kind < 0 || gate_kind > 2 || (gate_kind == 2 && decay_in == nullptr))
        return LLMX_ERR_BAD_ARGUMENT;
    const size_t smem = (size_t)channels * sizeof(float);
    if (smem > 200 * 1024) return LLMX_ERR_UNSUPPORTED;
    // Fours: a head's lanes are a power of two of a warp's (without unit heads any width does), and every run of channels
    // starts on 16 bytes.
    const bool units = q_channels + k_channels > 0;
    if (taps <= CONV_TAPS && channels % 4 == 0 && stride % 4 == 0 && first % 4 == 0 && slot_floats % 4 == 0 && conv_off % 4 == 0 &&
        (!units || (D % 4 == 0 && D <= 128 && ((D / 4) & (D / 4 - 1)) == 0)) &&
        (((uintptr_t)proj | (uintptr_t)ready | (uintptr_t)state | (uintptr_t)taps_b) & 15) == 0) {
        const int per = gate_kind == 2 ? heads * D : heads, block = CONV_THREADS * 4;
        const int conv_blocks = (channels + block - 1) / block, gate_blocks = (per + CONV_THREADS - 1) / CONV_THREADS;
        // One row a block while there are fewer blocks than four to an SM, longer runs of rows beyond.
        int run = (int)((long long)rows * conv_blocks / 592);
        run = run < 1 ? 1 : run > CONV_RUN ? CONV_RUN : run;
        const int row_blocks = (rows + run - 1) / run;
        launch_kernel(conv_prepare_four_kernel, dim3(row_blocks + requests, gate_blocks + conv_blocks), dim3(CONV_THREADS), 0, stream, proj,
                      stride, first, channels, q_channels, k_channels, taps_w, taps_b, taps, ready, a_log, dt_bias, b_off, a_off,
                      gate_kind, decay_in, decay_stride, gates, gates_stride, heads, D, q_factor, state, slot_floats, conv_off,
                      row_request, row_start, row_count, history, slot_in, slot_out, rows, run, row_blocks, gate_blocks);
        return launch_status();
    }
    if (smem > 48 * 1024) LLMX_ALLOW_SMEM(conv_prepare_kernel);
    launch_kernel(conv_prepare_kernel, dim3(rows + requests), dim3(256), smem, stream, proj, stride, first, channels,
                  q_channels, k_channels, taps_w, taps_b, taps, ready, a_log, dt_bias, b_off, a_off, gate_kind, decay_in,
                  decay_stride, gates, gates_stride, heads, D, q_factor, state, slot_floats, conv_off, row_request,
                  row_start, row_count, history, slot_in, slot_out, rows);
    return launch_status();
}

// proj [rows, stride]: the pair's inner values in columns low_off .. low_off + rank - 1, q in columns q_off .. q_off + channels
// - 1 (multiplied in place by q_factor; the two runs must not overlap); w2t [rank, channels], bias [channels] or null;
// decay [rows, channels] = sigmoid(low w2t + bias)^inv_tau.
LLMX_EXPORT int llmx_channel_decay(float* proj, int stride, int rows, int low_off, int rank, const float* w2t, const float* bias,
                                   float inv_tau, float* decay, int channels, int q_off, float q_factor, cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (rank < 1 || channels < 1 || low_off < 0 || q_off < 0 || low_off + rank > stride || q_off + channels > stride ||
        (low_off < q_off + channels && q_off < low_off + rank) || w2t == nullptr)
        return LLMX_ERR_BAD_ARGUMENT;
    const long long by = ((long long)rows + DECAY_ROWS - 1) / DECAY_ROWS;
    if (by > 65535) return LLMX_ERR_UNSUPPORTED;
    launch_kernel(channel_decay_kernel, dim3((channels + DECAY_THREADS - 1) / DECAY_THREADS, (unsigned)by), dim3(DECAY_THREADS), 0, stream,
                  proj, stride, rows, low_off, rank, w2t, bias, inv_tau, decay, channels, q_off, q_factor);
    return launch_status();
}
