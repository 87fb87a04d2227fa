// The tiled form of the attention over [key ; value] rows (attention_split.cu) on the 5th-generation tensor cores: key and value
// widths of 128, bfloat16 queries and cache, pages of whole sixteens, and a plain softmax (no cap, sink, rotated values,
// second map or gate).
//
// A block takes 128 rows that share their keys: tokens of one request in a row times the heads of one key/value head
// (their number rounded up to a power of two), 64 keys a stage in two stages:
//     S[128, 64] = Q K^T (one product a stage)     O[128, 128] += P V, the weights P as three bfloat16 parts (24 bits), small ones first
//   warp 0      producer: a stage's sixteen copies (four runs of sixteen tokens x the row's four blocks of 64 values)
//   warp 1      the products, issued by one thread
//   warps 2-5   one thread a row: its queries to shared memory; a stage's scores from tensor memory, mask, online softmax in
//               32-bit (base 2), the weights' parts over the scores; at the end O / l
// 96 KB of shared memory and 256 columns of tensor memory (scores or weights 96, output 128) a block, so two blocks share an SM and
// one's softmax runs beside the other's products: what bounds it (1,024 cycles of products and about as many of softmax a
// stage).  2,048 rows of 16 heads over 4: 330 -> 61 us; 1,201 rows of 32 over 8: 240 -> 43 us (both against 64
// rows a block on mma.sync).
//
// Slots of the cache that no row of the block may see can hold anything: their values are overwritten with zeros before a
// product reads them.  Every wait on an mbarrier is bounded (tc_common.cuh).
#include "attn_parts.cuh"
#include <math.h>

namespace {

constexpr int D = 128, ROWS = 128, KEYS = 64, RUN = 16;       // RUN: tokens a copy brings
constexpr int BLOCK_BYTES = KEYS * 128, STAGE_BYTES = 4 * BLOCK_BYTES, STAGES = 2;       // 64 keys x 64 values; two blocks of the key, two of the value
constexpr int Q_BLOCK = ROWS * 128, Q_BYTES = 2 * Q_BLOCK;
constexpr int SMEM_BYTES = Q_BYTES + STAGES * STAGE_BYTES + 1024 + 256;
constexpr int THREADS = 192, ROW_WARPS = 4;
constexpr uint32_t TMEM_COLS = 256, TMEM_S = 0, P_PART = 32, TMEM_O = 128;
constexpr float RAISE = 8.0f;                 // the exponent's maximum follows the true one when it is 2^8 behind
enum : int { ERR_ROWS_PRODUCER = 461, ERR_ROWS_MMA = 462, ERR_ROWS_SOFTMAX = 463 };
constexpr uint32_t IDESC_QK = tc::instr_desc_bf16(ROWS, KEYS);
constexpr uint32_t IDESC_PV = tc::instr_desc_bf16(ROWS, D) | (1u << 16);       // values: the MN-major operand

__global__ void __launch_bounds__(THREADS, 2)
attention_rows_kernel(const __grid_constant__ CUtensorMap cache_map, const __nv_bfloat16* __restrict__ q, __nv_bfloat16* __restrict__ out,
                      const int* __restrict__ row_start, const int* __restrict__ row_count, const int* __restrict__ history,
                      const int* __restrict__ block_tables, int table_stride, int requests, int heads, int kv_heads, int page_size,
                      int window, int chunk, float scale_log2, int r_pad, int* error_word) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* stages = smem + Q_BYTES;
    uint64_t* bars = (uint64_t*)(stages + STAGES * STAGE_BYTES);
    uint64_t *full = bars, *empty = bars + 2;      // [2] a stage's keys and values have landed / its products have run
    uint64_t* q_full = bars + 4;                   // the rows' queries are in shared memory
    uint64_t* s_full = bars + 5;                   // a stage's scores are complete (after the last stage: the output)
    uint64_t* p_full = bars + 6;                   // a stage's weights are in tensor memory, the output rescaled if need be
    uint32_t* tmem_slot = (uint32_t*)(bars + 7);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 4; ++i) tc::mbar_init(&bars[i], 1);
        tc::mbar_init(q_full, ROW_WARPS);
        tc::mbar_init(s_full, 1);
        tc::mbar_init(p_full, ROW_WARPS);
        *abort_flag = 0;
        tc::fence_barrier_init();
        tc::tma_prefetch_desc(&cache_map);
    }
    if (warp == 1) {
        tc::tmem_alloc(tmem_slot, TMEM_COLS);
        tc::tmem_relinquish();
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_trigger();
    pdl_wait();

    // Which tile: the requests' tiles are numbered one request after the other, a request's last ones (with the most keys) first.
    const int ratio = heads / kv_heads, tok = ROWS / r_pad, g = blockIdx.y;
    int idx = blockIdx.x, r = 0, tiles_r = 0;
    for (; r < requests; ++r) {
        tiles_r = (row_count[r] + tok - 1) / tok;
        if (idx < tiles_r) break;
        idx -= tiles_r;
    }
    const bool active = r < requests;
    if (!active) r = 0;
    const int t0 = active ? (tiles_r - 1 - idx) * tok : 0, a0 = row_start[r], hist = history[r];
    const int n_tok = min(tok, row_count[r] - t0);
    auto lowest = [&](int p) {
        int lo = window > 0 ? max(0, p - window + 1) : 0;
        if (chunk > 0) lo = max(lo, p / chunk * chunk);
        return lo;
    };
    const int key_lo = lowest(hist + t0), key_end = hist + t0 + n_tok;       // the keys some row of the block sees
    const int begin = key_lo / KEYS * KEYS;
    const int n_iter = active ? (key_end - begin + KEYS - 1) / KEYS : 0;
    const int* table = block_tables + (size_t)r * table_stride;

    if (warp == 0) {
        // Lane l < 16: tokens 16 (l / 4) on of the stage, values 64 (l % 4) on of the row.  Tokens past the last key, or on a
        // page that a window has given back, are read from page 0 (and overwritten with zeros).
        bool ok = true;
        for (int j = 0; j < n_iter && ok; ++j) {
            const int st = j & 1, t = begin + j * KEYS + RUN * (lane >> 2);
            const int page = lane < 16 && t < key_end ? max(table[t / page_size], 0) : 0;
            ok = tc::mbar_wait_warp(&empty[st], ((j >> 1) & 1u) ^ 1u, abort_flag, error_word, ERR_ROWS_PRODUCER);
            if (!ok) break;
            if (lane == 0) tc::mbar_expect_tx(&full[st], STAGE_BYTES);
            __syncwarp();
            if (lane < 16)
                tc::tma_load_2d(stages + st * STAGE_BYTES + (lane & 3) * BLOCK_BYTES + (lane >> 2) * RUN * 128, &cache_map, (lane & 3) * 64,
                                (page * kv_heads + g) * page_size + t % page_size, &full[st]);
        }
    } else if (warp == 1) {
        if (tc::elect_one() && active) {
            const uint32_t ts = tmem_base + TMEM_S, to = tmem_base + TMEM_O, q_addr = tc::smem_u32(smem);
            bool ok = tc::mbar_wait(q_full, 0, abort_flag, error_word, ERR_ROWS_MMA);
            for (int j = 0; j < n_iter && ok; ++j) {
                const int st = j & 1;
                ok = tc::mbar_wait(&full[st], (j >> 1) & 1u, abort_flag, error_word, ERR_ROWS_MMA);
                if (!ok) break;
                tc::tc_fence_after();
                const uint32_t k_addr = tc::smem_u32(stages + st * STAGE_BYTES), v_addr = k_addr + 2 * BLOCK_BYTES;
                // The products of one thread run in the order they are issued: the weights these scores overwrite have been
                // read by the stage before's P V.
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk)
                    tc::mma_bf16_ss(ts, tc::smem_desc_k_sw128(q_addr + (kk >> 2) * Q_BLOCK + (kk & 3) * 32),
                                    tc::smem_desc_k_sw128(k_addr + (kk >> 2) * BLOCK_BYTES + (kk & 3) * 32), IDESC_QK, kk > 0 ? 1u : 0u);
                tc::mma_commit(s_full);
                ok = tc::mbar_wait(p_full, j & 1u, abort_flag, error_word, ERR_ROWS_MMA);
                if (!ok) break;
                tc::tc_fence_after();
#pragma unroll
                for (int part = 2; part >= 0; --part)
#pragma unroll
                    for (int kk = 0; kk < KEYS / 16; ++kk)
                        tc::mma_bf16_ts(to, ts + part * P_PART + kk * 8, attn::smem_desc_mn_sw128(v_addr + kk * 16 * 128, BLOCK_BYTES), IDESC_PV,
                                        (j > 0 || part < 2 || kk > 0) ? 1u : 0u);
                tc::mma_commit(&empty[st]);
            }
            if (ok) tc::mma_commit(s_full);
        }
    } else if (active) {
        const int quarter = warp & 3, row = quarter * 32 + lane;
        const int tk = row / r_pad, hd = row % r_pad;
        const bool valid = tk < n_tok && hd < ratio;
        const size_t at = ((size_t)(a0 + t0 + (valid ? tk : 0)) * heads + (size_t)g * ratio + (valid ? hd : 0)) * D;
        const uint32_t lanes = tmem_base + ((uint32_t)(quarter * 32) << 16);
        {
            const uint4* src = reinterpret_cast<const uint4*>(q + at);
#pragma unroll
            for (int c = 0; c < D / 8; ++c)
                *reinterpret_cast<uint4*>(smem + (c >> 3) * Q_BLOCK + attn::swz(row, c & 7)) = valid ? src[c] : make_uint4(0u, 0u, 0u, 0u);
        }
        tc::fence_proxy_async();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(q_full);

        const int pos = hist + t0 + tk, lo_key = lowest(pos);
        float m_used = -INFINITY, l_run = 0.0f;
        bool ok = true;
        for (int j = 0; j < n_iter; ++j) {
            const int key0 = begin + j * KEYS;
            if (key0 < key_lo || key0 + KEYS > key_end) {
                // Slots of the stage that no row may see: a zero weight must meet a finite value.  Thread t has key t % 64, half t / 64.
                ok = tc::mbar_wait_warp(&full[j & 1], (j >> 1) & 1u, abort_flag, error_word, ERR_ROWS_SOFTMAX);
                if (!ok) break;
                const int t = row % KEYS, key = key0 + t;
                if (key < key_lo || key >= key_end) {
                    uint4* v = reinterpret_cast<uint4*>(stages + (j & 1) * STAGE_BYTES + (2 + row / KEYS) * BLOCK_BYTES + t * 128);
#pragma unroll
                    for (int i = 0; i < 8; ++i) v[i] = make_uint4(0u, 0u, 0u, 0u);
                }
                tc::fence_proxy_async();
            }
            ok = tc::mbar_wait_warp(s_full, j & 1u, abort_flag, error_word, ERR_ROWS_SOFTMAX);
            if (!ok) break;
            tc::tc_fence_after();
            uint32_t sc[KEYS];
#pragma unroll
            for (int c = 0; c < KEYS; c += 32) tc::tmem_ld_32x32(lanes + TMEM_S + c, *reinterpret_cast<uint32_t(*)[32]>(&sc[c]));
            tc::tmem_wait_ld();
            if (key0 + KEYS - 1 > pos || key0 < lo_key) {
#pragma unroll
                for (int k = 0; k < KEYS; ++k)
                    if (key0 + k > pos || key0 + k < lo_key) sc[k] = __float_as_uint(-INFINITY);
            }
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int k = 0; k < KEYS; k += 8)
#pragma unroll
                for (int u = 0; u < 4; ++u) mx[u] = attn::max3(mx[u], __uint_as_float(sc[k + 2 * u]), __uint_as_float(sc[k + 2 * u + 1]));
            // The scale is positive: it is applied after the maximum and folded into the exponent's multiply-add.
            const float cand = fmaxf(m_used, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * scale_log2);
            const bool raise = j > 0 && __any_sync(0xffffffffu, cand > m_used + RAISE);
            const float factor = !raise || cand == -INFINITY ? 1.0f : exp2f(m_used - cand);
            if (j == 0 || raise) m_used = cand;
            const float base = m_used == -INFINITY ? 0.0f : m_used;
            float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int c = 0; c < KEYS; c += 32) {
                uint32_t p[3][16];
#pragma unroll
                for (int u = 0; u < 16; ++u) {
                    const float a = exp2f(fmaf(__uint_as_float(sc[c + 2 * u]), scale_log2, -base));
                    const float b = exp2f(fmaf(__uint_as_float(sc[c + 2 * u + 1]), scale_log2, -base));
                    sum[u & 3] += a + b;
                    attn::split3_pair(a, b, p[0][u], p[1][u], p[2][u]);
                }
#pragma unroll
                for (int k = 0; k < 3; ++k) tc::tmem_st_32x16(lanes + TMEM_S + k * P_PART + c / 2, p[k]);
            }
            if (raise) {
                // The output so far was summed against the old maximum.  P V of the stage before has finished (this stage's
                // scores were made after it) and this one's waits for the arrival below.
#pragma unroll 1
                for (int c = 0; c < D; c += 32) {
                    uint32_t v[32];
                    tc::tmem_ld_32x32(lanes + TMEM_O + c, v);
                    tc::tmem_wait_ld();
#pragma unroll
                    for (int k = 0; k < 32; ++k) v[k] = __float_as_uint(__uint_as_float(v[k]) * factor);
                    tc::tmem_st_32x32(lanes + TMEM_O + c, v);
                }
                l_run *= factor;
            }
            l_run += (sum[0] + sum[1]) + (sum[2] + sum[3]);
            tc::tmem_wait_st();
            tc::tc_fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(p_full);
        }
        if (ok) ok = tc::mbar_wait_warp(s_full, n_iter & 1u, abort_flag, error_word, ERR_ROWS_SOFTMAX);
        if (ok) {
            tc::tc_fence_after();
            const float inv = 1.0f / l_run;
#pragma unroll 1
            for (int c = 0; c < D; c += 32) {
                uint32_t v[32];
                tc::tmem_ld_32x32(lanes + TMEM_O + c, v);
                tc::tmem_wait_ld();
                if (valid) {
#pragma unroll
                    for (int d = 0; d < 32; d += 8) {
                        uint32_t w[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            w[u] = attn::pack_bf16(__uint_as_float(v[d + 2 * u]) * inv, __uint_as_float(v[d + 2 * u + 1]) * inv);
                        *reinterpret_cast<uint4*>(out + at + c + d) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                }
                __syncwarp();
            }
        }
        tc::tc_fence_before();
    }
    __syncthreads();
    if (warp == 1) {
        tc::tc_fence_after();
        tc::tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

}  // namespace

// q, out [rows, heads * 128] and cache [pool_rows, 256] (a page holds kv_heads runs of page_size [key ; value] rows) bfloat16;
// the metadata arrays are the step's, on the device.
LLMX_EXPORT int llmx_attention_rows_tc(const void* q, const void* cache, long long pool_rows, void* out, const int* row_start,
                                       const int* row_count, const int* history, const int* block_tables, int table_stride, int rows,
                                       int requests, int heads, int kv_heads, int page_size, int window, int chunk, float scale,
                                       int* error_word, cudaStream_t stream) {
    if (rows <= 0 || requests <= 0) return 0;
    if (heads <= 0 || kv_heads <= 0 || heads % kv_heads || heads / kv_heads > ROWS || kv_heads > 65535 || page_size <= 0 || page_size % RUN ||
        pool_rows <= 0 || pool_rows >= (1ll << 31) || !(scale > 0.0f) || (((uintptr_t)q | (uintptr_t)cache | (uintptr_t)out) & 15))
        return LLMX_ERR_UNSUPPORTED;
    int r_pad = 1;
    while (r_pad < heads / kv_heads) r_pad *= 2;
    const int tok = ROWS / r_pad;
    CUtensorMap map;
    if (int e = llmx_make_map_bf16_2d(&map, cache, (uint64_t)pool_rows, 2 * D, RUN, 64)) return e;
    if (cudaFuncSetAttribute(attention_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess) return (int)cudaGetLastError();
    launch_kernel(attention_rows_kernel, dim3((rows + tok - 1) / tok + requests, kv_heads), dim3(THREADS), (size_t)SMEM_BYTES, stream, map,
                  (const __nv_bfloat16*)q, (__nv_bfloat16*)out, row_start, row_count, history, block_tables, table_stride, requests, heads,
                  kv_heads, page_size, window, chunk, scale * attn::LOG2E, r_pad, error_word);
    return launch_status();
}
