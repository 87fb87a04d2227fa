// The tiled form of the attention over [key ; value] rows (attention_split.cu) on the 5th-generation tensor cores: key and value
// widths of 128, bfloat16 queries and cache, pages of whole sixteens, and a plain softmax (no cap, sink, rotated values,
// second map or gate).
//
// A tile is 128 rows that share their keys: tokens of one request in a row times the heads of one key/value head
// (their number rounded up to a power of two), 64 keys a stage in two stages:
//     S[128, 64] = Q K^T (one product a stage)     O[128, 128] = P V, the weights P as three bfloat16 parts (24 bits), small ones first
// A block has two tiles, each with keys and values of its own (their requests may differ), so that one's softmax runs beside
// the other's products; launches of few tiles give each an SM.
//   warp 0      producer: a stage's sixteen copies (four runs of sixteen tokens x the row's four blocks of 64 values), half a warp a tile
//   warp 1      the products of both tiles, issued by one thread in turn
//   warps 4-11  four a tile, one thread a row: its queries to shared memory; a stage's scores from tensor memory, mask, online
//               softmax in 32-bit (base 2), the weights' parts to tensor memory; the stage's output joins the row's sums; at the end O / l
// The tensor core cuts off what an addition shifts out of its accumulator.  A stage's output therefore starts from nothing and joins
// the 128 sums that the row's thread holds in registers by rounded additions; added up over the stages in tensor memory,
// 4,096 keys left 0.65 % of the results at another bfloat16 than the exact ones (values of mean 1; 0.28 % in the form on mma.sync, whose
// accumulators run through too, 0.002 % so), 16,384 keys 2.6 % (1.4 %; 0.005 %).
// A row's thread has no registers left for 64 scores: it reads them twice, for the maximum and, sixteen at a time, for the
// weights, whose parts lie where no unread score does.
// 192 KB of shared memory and all of tensor memory a block.  What bounds it: 1,024 cycles of products a tile and stage, two tiles
// taking turns, and the causal edge: the last tiles of a prompt see all keys.  2,048 rows of 16 heads over 4: 330 us on mma.sync,
// 95 so; 1,201 rows of 32 over 8: 240 -> 63 us (72 and 50 with sums and weights that were less exact).
//
// Slots of the cache that no row of the tile may see can hold anything: their values are overwritten with zeros before a
// product reads them.  Every wait on an mbarrier is bounded (tc_common.cuh).
#include "attn_parts.cuh"
#include <math.h>

namespace {

constexpr int D = 128, ROWS = 128, KEYS = 64, RUN = 16;       // RUN: tokens a copy brings
constexpr int BLOCK_BYTES = KEYS * 128, STAGE_BYTES = 4 * BLOCK_BYTES, STAGES = 2;       // 64 keys x 64 values; two blocks of the key, two of the value
constexpr int Q_BLOCK = ROWS * 128, Q_BYTES = 2 * Q_BLOCK;
constexpr int TILES = 2, TILE_BYTES = Q_BYTES + STAGES * STAGE_BYTES;
constexpr int SMEM_BYTES = TILES * TILE_BYTES + 1024 + 256;
// Three groups of four warps: the first copies and issues products (two of its warps idle), the others have a tile each.  The block is
// launched with 3 x 128 x 168 registers; the first group gives back what the rows' threads need for their 128 sums: 40 + 232 + 232 = 3 x 168.
constexpr int ROW_WARPS = 4, THREADS = (1 + TILES) * ROW_WARPS * 32, FEWER_REGISTERS = 40, MORE_REGISTERS = 232;
static_assert(FEWER_REGISTERS + TILES * MORE_REGISTERS <= (1 + TILES) * 168, "setmaxnreg draws on the block's registers at launch");
// Tensor memory of a tile: the weights' parts in columns 0 .. 95, the scores in 64 .. 127, the output of a stage in 128 .. 255.  The parts
// of scores 16 c .. 16 c + 15 end at column 64 + 8 c + 8: over scores that have been read.
constexpr uint32_t TMEM_COLS = 512, TILE_COLS = 256, P_PART = 32, TMEM_S = 64, TMEM_O = 128;
constexpr float RAISE = 8.0f;                 // the exponent's maximum follows the true one when it is 2^8 behind
enum : int { ERR_ROWS_PRODUCER = 461, ERR_ROWS_MMA = 462, ERR_ROWS_SOFTMAX = 463 };
constexpr uint32_t IDESC_QK = tc::instr_desc_bf16(ROWS, KEYS);
constexpr uint32_t IDESC_PV = tc::instr_desc_bf16(ROWS, D) | (1u << 16);       // values: the MN-major operand

__device__ __forceinline__ void tmem_st_32x8(uint32_t addr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}

// The lowest key that position p sees.
__device__ __forceinline__ int lowest_key(int p, int window, int chunk) {
    int lo = window > 0 ? max(0, p - window + 1) : 0;
    if (chunk > 0) lo = max(lo, p / chunk * chunk);
    return lo;
}

// A tile: its request, the place of its first token in the request's rows, its tokens, and the keys that some row of it sees.
struct Tile {
    int request, t0, n_tok, a0, hist, key_lo, key_end, begin, n_iter;
};

// The requests' tiles are numbered one request after the other, a request's last ones (with the most keys) first; beyond the last
// one there is nothing to do (n_iter 0).
__device__ __forceinline__ Tile find_tile(int idx, const int* row_start, const int* row_count, const int* history, int requests, int tok,
                                          int window, int chunk) {
    Tile w = {};
    int tiles_r = 0;
    for (; w.request < requests; ++w.request) {
        tiles_r = (row_count[w.request] + tok - 1) / tok;
        if (idx < tiles_r) break;
        idx -= tiles_r;
    }
    if (w.request >= requests) {
        w.request = 0;
        return w;
    }
    w.t0 = (tiles_r - 1 - idx) * tok;
    w.n_tok = min(tok, row_count[w.request] - w.t0);
    w.a0 = row_start[w.request];
    w.hist = history[w.request];
    w.key_lo = lowest_key(w.hist + w.t0, window, chunk);
    w.key_end = w.hist + w.t0 + w.n_tok;
    w.begin = w.key_lo / KEYS * KEYS;
    w.n_iter = (w.key_end - w.begin + KEYS - 1) / KEYS;
    return w;
}

__global__ void __launch_bounds__(THREADS, 1)
attention_rows_kernel(const __grid_constant__ CUtensorMap cache_map, const __nv_bfloat16* __restrict__ q, __nv_bfloat16* __restrict__ out,
                      const int* __restrict__ row_start, const int* __restrict__ row_count, const int* __restrict__ history,
                      const int* __restrict__ block_tables, int table_stride, int requests, int heads, int kv_heads, int page_size,
                      int window, int chunk, float scale_log2, int r_pad, int tiles_a_block, int* error_word) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    // Of each tile: [2] a stage's keys and values have landed / its products have run; the rows' queries are in shared memory; a stage's
    // scores are complete / its weights are in tensor memory and the output of the stage before has been read / its output is complete.
    struct Bars {
        uint64_t full[STAGES], empty[STAGES], q_full, s_full, p_full, o_full;
    };
    Bars* bars = (Bars*)(smem + TILES * TILE_BYTES);
    uint32_t* tmem_slot = (uint32_t*)(bars + TILES);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int t = 0; t < TILES; ++t) {
            for (int i = 0; i < STAGES; ++i) {
                tc::mbar_init(&bars[t].full[i], 1);
                tc::mbar_init(&bars[t].empty[i], 1);
            }
            tc::mbar_init(&bars[t].q_full, ROW_WARPS);
            tc::mbar_init(&bars[t].s_full, 1);
            tc::mbar_init(&bars[t].p_full, ROW_WARPS);
            tc::mbar_init(&bars[t].o_full, 1);
        }
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

    const int ratio = heads / kv_heads, tok = ROWS / r_pad, g = blockIdx.y;
    auto tile_of = [&](int t) -> Tile {
        if (t >= tiles_a_block) return Tile{};
        return find_tile(blockIdx.x * tiles_a_block + t, row_start, row_count, history, requests, tok, window, chunk);
    };

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(FEWER_REGISTERS));
        if (warp == 0) {
            // Lanes 16 t + l of tile t: tokens 16 (l / 4) on of the stage, values 64 (l % 4) on of the row.  Tokens past the last key, or on a
            // page that a window has given back, are read from page 0 (and overwritten with zeros).
            const int mine = lane >> 4, l = lane & 15;
            const Tile w = tile_of(mine);
            const int* table = block_tables + (size_t)w.request * table_stride;
            uint8_t* stages = smem + mine * TILE_BYTES + Q_BYTES;
            Bars& b = bars[mine];
            const int most = max(__shfl_sync(0xffffffffu, w.n_iter, 0), __shfl_sync(0xffffffffu, w.n_iter, 16));
            for (int j = 0; j < most; ++j) {
                const int st = j & 1, t = w.begin + j * KEYS + RUN * (l >> 2);
                const bool here = j < w.n_iter;
                const int page = here && t < w.key_end ? max(table[t / page_size], 0) : 0;
                bool ok = !here || tc::mbar_wait(&b.empty[st], ((j >> 1) & 1u) ^ 1u, abort_flag, error_word, ERR_ROWS_PRODUCER);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                if (here && l == 0) tc::mbar_expect_tx(&b.full[st], STAGE_BYTES);
                __syncwarp();
                if (here)
                    tc::tma_load_2d(stages + st * STAGE_BYTES + (l & 3) * BLOCK_BYTES + (l >> 2) * RUN * 128, &cache_map, (l & 3) * 64,
                                    (page * kv_heads + g) * page_size + t % page_size, &b.full[st]);
            }
        } else if (warp == 1) {
            int n_iter[TILES];
    #pragma unroll
            for (int t = 0; t < TILES; ++t) n_iter[t] = tile_of(t).n_iter;
            if (tc::elect_one()) {
                bool ok = true;
                auto scores = [&](int t, int j) {            // S = Q K^T of stage j
                    Bars& b = bars[t];
                    const int st = j & 1;
                    ok = tc::mbar_wait(&b.full[st], (j >> 1) & 1u, abort_flag, error_word, ERR_ROWS_MMA);
                    if (!ok) return;
                    tc::tc_fence_after();
                    const uint32_t q_addr = tc::smem_u32(smem + t * TILE_BYTES), k_addr = q_addr + Q_BYTES + st * STAGE_BYTES;
    #pragma unroll
                    for (int kk = 0; kk < D / 16; ++kk)
                        tc::mma_bf16_ss(tmem_base + t * TILE_COLS + TMEM_S, tc::smem_desc_k_sw128(q_addr + (kk >> 2) * Q_BLOCK + (kk & 3) * 32),
                                        tc::smem_desc_k_sw128(k_addr + (kk >> 2) * BLOCK_BYTES + (kk & 3) * 32), IDESC_QK, kk > 0 ? 1u : 0u);
                    tc::mma_commit(&b.s_full);
                };
    #pragma unroll 1
                for (int t = 0; t < TILES; ++t)
                    if (ok && n_iter[t] > 0) {
                        ok = tc::mbar_wait(&bars[t].q_full, 0, abort_flag, error_word, ERR_ROWS_MMA);
                        if (ok) scores(t, 0);
                    }
                for (int j = 0; ok && j < max(n_iter[0], n_iter[1]); ++j)
    #pragma unroll 1
                    for (int t = 0; t < TILES; ++t) {
                        if (!ok || j >= n_iter[t]) continue;
                        Bars& b = bars[t];
                        const int st = j & 1;
                        ok = tc::mbar_wait(&b.p_full, j & 1u, abort_flag, error_word, ERR_ROWS_MMA);
                        if (!ok) continue;
                        tc::tc_fence_after();
                        const uint32_t tile = tmem_base + t * TILE_COLS;
                        const uint32_t v_addr = tc::smem_u32(smem + t * TILE_BYTES + Q_BYTES + st * STAGE_BYTES) + 2 * BLOCK_BYTES;
    #pragma unroll
                        for (int part = 2; part >= 0; --part)
    #pragma unroll
                            for (int kk = 0; kk < KEYS / 16; ++kk)
                                tc::mma_bf16_ts(tile + TMEM_O, tile + part * P_PART + kk * 8, attn::smem_desc_mn_sw128(v_addr + kk * 16 * 128, BLOCK_BYTES),
                                                IDESC_PV, part < 2 || kk > 0 ? 1u : 0u);
                        tc::mma_commit(&b.empty[st]);
                        tc::mma_commit(&b.o_full);
                        // The products of one thread run in the order they are issued: the weights that the next scores overwrite have been
                        // read by P V.
                        if (j + 1 < n_iter[t]) scores(t, j + 1);
                    }
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(MORE_REGISTERS));
        const int t = (warp - 4) / ROW_WARPS;
        const Tile w = tile_of(t);
        Bars& b = bars[t];
        uint8_t* q_smem = smem + t * TILE_BYTES;
        const int quarter = warp & 3, row = quarter * 32 + lane;
        const int tk = row / r_pad, hd = row % r_pad;
        const bool valid = tk < w.n_tok && hd < ratio;
        const size_t at = ((size_t)(w.a0 + w.t0 + (valid ? tk : 0)) * heads + (size_t)g * ratio + (valid ? hd : 0)) * D;
        const uint32_t lanes = tmem_base + t * TILE_COLS + ((uint32_t)(quarter * 32) << 16);
        if (w.n_iter > 0) {
            {
                const uint4* src = reinterpret_cast<const uint4*>(q + at);
#pragma unroll
                for (int c = 0; c < D / 8; ++c)
                    *reinterpret_cast<uint4*>(q_smem + (c >> 3) * Q_BLOCK + attn::swz(row, c & 7)) = valid ? src[c] : make_uint4(0u, 0u, 0u, 0u);
            }
            tc::fence_proxy_async();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&b.q_full);
        }

        const int pos = w.hist + w.t0 + tk, lo_key = lowest_key(pos, window, chunk);
        float m_used = -INFINITY, l_run = 0.0f, o[D];
#pragma unroll
        for (int d = 0; d < D; ++d) o[d] = 0.0f;
        // What stage j made of the output joins the row's sums.
        auto take_output = [&](int j) -> bool {
            if (!tc::mbar_wait_warp(&b.o_full, j & 1u, abort_flag, error_word, ERR_ROWS_SOFTMAX)) return false;
            tc::tc_fence_after();
#pragma unroll
            for (int c = 0; c < D; c += 32) {
                uint32_t v[32];
                tc::tmem_ld_32x32(lanes + TMEM_O + c, v);
                tc::tmem_wait_ld();
#pragma unroll
                for (int k = 0; k < 32; ++k) o[c + k] += __uint_as_float(v[k]);
            }
            return true;
        };
        bool ok = true;
        for (int j = 0; j < w.n_iter; ++j) {
            const int key0 = w.begin + j * KEYS;
            if (key0 < w.key_lo || key0 + KEYS > w.key_end) {
                // Slots of the stage that no row may see: a zero weight must meet a finite value.  Thread r has key r % 64, half r / 64.
                ok = tc::mbar_wait_warp(&b.full[j & 1], (j >> 1) & 1u, abort_flag, error_word, ERR_ROWS_SOFTMAX);
                if (!ok) break;
                const int s = row % KEYS, key = key0 + s;
                if (key < w.key_lo || key >= w.key_end) {
                    uint4* v = reinterpret_cast<uint4*>(q_smem + Q_BYTES + (j & 1) * STAGE_BYTES + (2 + row / KEYS) * BLOCK_BYTES + s * 128);
#pragma unroll
                    for (int i = 0; i < 8; ++i) v[i] = make_uint4(0u, 0u, 0u, 0u);
                }
                tc::fence_proxy_async();
            }
            ok = j == 0 || take_output(j - 1);
            ok = ok && tc::mbar_wait_warp(&b.s_full, j & 1u, abort_flag, error_word, ERR_ROWS_SOFTMAX);
            if (!ok) break;
            tc::tc_fence_after();
            // Keys key0 + first .. key0 + last - 1 of the stage are the row's.
            const int first = lo_key - key0, last = pos + 1 - key0;
            const bool masked = first > 0 || last < KEYS;
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int c = 0; c < KEYS; c += 32) {
                uint32_t sc[32];
                tc::tmem_ld_32x32(lanes + TMEM_S + c, sc);
                tc::tmem_wait_ld();
                if (masked) {
#pragma unroll
                    for (int k = 0; k < 32; ++k)
                        if (c + k >= last || c + k < first) sc[k] = __float_as_uint(-INFINITY);
                }
#pragma unroll
                for (int k = 0; k < 32; k += 8)
#pragma unroll
                    for (int u = 0; u < 4; ++u) mx[u] = attn::max3(mx[u], __uint_as_float(sc[k + 2 * u]), __uint_as_float(sc[k + 2 * u + 1]));
            }
            // The scale is positive: it is applied after the maximum and folded into the exponent's multiply-add.
            const float cand = fmaxf(m_used, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * scale_log2);
            if (j == 0) {
                m_used = cand;
            } else if (__any_sync(0xffffffffu, cand > m_used + RAISE)) {
                const float factor = cand == -INFINITY ? 1.0f : exp2f(m_used - cand);       // the sums so far were made against the old maximum
                m_used = cand;
                l_run *= factor;
#pragma unroll
                for (int d = 0; d < D; ++d) o[d] *= factor;
            }
            const float base = m_used == -INFINITY ? 0.0f : m_used;
            float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int c = 0; c < KEYS; c += 16) {
                uint32_t sc[16], p[3][8];
                tc::tmem_ld_32x16(lanes + TMEM_S + c, sc);
                tc::tmem_wait_ld();
                if (masked) {
#pragma unroll
                    for (int k = 0; k < 16; ++k)
                        if (c + k >= last || c + k < first) sc[k] = __float_as_uint(-INFINITY);
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const float x = exp2f(fmaf(__uint_as_float(sc[2 * u]), scale_log2, -base));
                    const float y = exp2f(fmaf(__uint_as_float(sc[2 * u + 1]), scale_log2, -base));
                    sum[u & 3] += x + y;
                    attn::split3_pair(x, y, p[0][u], p[1][u], p[2][u]);
                }
#pragma unroll
                for (int k = 0; k < 3; ++k) tmem_st_32x8(lanes + k * P_PART + c / 2, p[k]);
            }
            l_run += (sum[0] + sum[1]) + (sum[2] + sum[3]);
            tc::tmem_wait_st();
            tc::tc_fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&b.p_full);
        }
        if (ok && w.n_iter > 0 && take_output(w.n_iter - 1) && valid) {
            const float inv = 1.0f / l_run;
#pragma unroll
            for (int d = 0; d < D; d += 8) {
                uint32_t v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = attn::pack_bf16(o[d + 2 * u] * inv, o[d + 2 * u + 1] * inv);
                *reinterpret_cast<uint4*>(out + at + d) = make_uint4(v[0], v[1], v[2], v[3]);
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
    // At most this many tiles.  Two to a block unless every tile can have an SM of its own.
    const long long tiles = ((long long)rows + tok - 1) / tok + requests;
    const int tiles_a_block = tiles * kv_heads > 148 ? TILES : 1;
    launch_kernel(attention_rows_kernel, dim3((unsigned)((tiles + tiles_a_block - 1) / tiles_a_block), kv_heads), dim3(THREADS), (size_t)SMEM_BYTES, stream,
                  map, (const __nv_bfloat16*)q, (__nv_bfloat16*)out, row_start, row_count, history, block_tables, table_stride, requests, heads,
                  kv_heads, page_size, window, chunk, scale * attn::LOG2E, r_pad, tiles_a_block, error_word);
    return launch_status();
}
