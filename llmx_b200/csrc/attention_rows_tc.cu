// The tiled form of the attention over [key ; value] rows (attention_split.cu) on the 5th-generation tensor cores: key and value
// widths of 128, bfloat16 queries and cache, pages of whole sixteens, and a plain softmax (no cap, sink, rotated values,
// second map or gate).
//
// A tile is 128 rows that share their keys: tokens of one request in a row times the heads of one key/value head
// (their number rounded up to a power of two), 48 keys a stage in three stages:
//     S[128, 48] = Q K^T (one product a stage)     O[128, 128] = P V, the weights P as three bfloat16 parts (24 bits), small ones first
// A block an SM stays for the whole launch and has two places, each with a tile, a producer, a thread that issues its products and
// four warps of rows of its own, so that one's softmax runs beside the other's products.  All tiles of all heads, a request's longest
// first, go to the places in turn: the first 148 to the blocks' first places, the next ones backwards to the second, so that few tiles
// have an SM each and many share theirs with one that is short where they are long (two neighbours in length on an SM: 2,048
// rows of 16 heads over 4 took 97 us instead of 70).
//   warps 0, 3   producers: a stage's twelve copies (three runs of sixteen tokens x the row's four blocks of 64 values)
//   warps 1, 2   the products, issued by one thread each
//   warps 4-11   four a place, one thread a row: its queries to shared memory; a stage's scores from tensor memory, mask, online
//                softmax in 32-bit (base 2), the weights' parts to tensor memory; the stage's output joins the row's sums; at the end O / l
// The tensor core cuts off what an addition shifts out of its accumulator.  A stage's output therefore starts from nothing and joins
// the 128 sums that the row's thread holds in registers by rounded additions; added up over the stages in tensor memory,
// 4,096 keys left 0.65 % of the results at another bfloat16 than the exact ones (values of mean 1; 0.28 % in the form on mma.sync, whose
// accumulators run through too, 0.002 % so), 16,384 keys 2.6 % (1.4 %; 0.004 %).
// With 48 keys a stage, scores, weights and output have tensor memory of their own: a stage's scores are made while the weights of
// the one before are.  209 KB of shared memory and all of tensor memory a block.  What bounds it: the products of an SM's two tiles (with
// two long ones on it the tensor pipe was busy 80 % of the cycles), and the causal edge: the last tiles of a prompt see all keys.
// 2,048 rows of 16 heads over 4: 330 us on mma.sync, 70 so; 1,201 rows of 32 over 8: 240 -> 59 (72 and 50 with sums and weights that
// were less exact); 64 rows of 16 over 4 16 us.
//
// Slots of the cache that no row of the tile may see can hold anything: their values are overwritten with zeros before a
// product reads them.  Every wait on an mbarrier is bounded (tc_common.cuh).
#include "attn_parts.cuh"
#include <math.h>

namespace {

constexpr int D = 128, ROWS = 128, KEYS = 48, RUN = 16;       // RUN: tokens a copy brings
constexpr int BLOCK_BYTES = KEYS * 128, STAGE_BYTES = 4 * BLOCK_BYTES, STAGES = 3;       // 48 keys x 64 values; two blocks of the key, two of the value
constexpr int Q_BLOCK = ROWS * 128, Q_BYTES = 2 * Q_BLOCK;
constexpr int PLACES = 2, PLACE_BYTES = Q_BYTES + STAGES * STAGE_BYTES, SMS = 148;
constexpr int SMEM_BYTES = PLACES * PLACE_BYTES + 1024 + 256;
// Three groups of four warps: the first copies and issues products, the others have the rows of a place each.  The block is
// launched with 3 x 128 x 168 registers; the first group gives back what the rows' threads need for their 128 sums: 40 + 232 + 232 = 3 x 168.
constexpr int ROW_WARPS = 4, THREADS = (1 + PLACES) * ROW_WARPS * 32, FEWER_REGISTERS = 40, MORE_REGISTERS = 232;
static_assert(FEWER_REGISTERS + PLACES * MORE_REGISTERS <= (1 + PLACES) * 168, "setmaxnreg draws on the block's registers at launch");
// Tensor memory of a place: the weights' parts in columns 0 .. 71, the scores in 80 .. 127, the output of a stage in 128 .. 255.
constexpr uint32_t TMEM_COLS = 512, PLACE_COLS = 256, P_PART = KEYS / 2, TMEM_S = 80, TMEM_O = 128;
static_assert(3 * P_PART <= TMEM_S && TMEM_S + KEYS <= TMEM_O, "weights, scores and output of a stage lie apart");
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
                      int window, int chunk, float scale_log2, int r_pad, int* error_word) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    // Of each place: a stage's keys and values have landed / its products have run; the rows' queries are in shared memory; a stage's
    // scores are complete / have been read / its weights are in tensor memory and the output of the stage before has been read / its
    // output is complete.
    struct Bars {
        uint64_t full[STAGES], empty[STAGES], q_full, s_full, s_free, p_full, o_full;
    };
    Bars* bars = (Bars*)(smem + PLACES * PLACE_BYTES);
    uint32_t* tmem_slot = (uint32_t*)(bars + PLACES);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int t = 0; t < PLACES; ++t) {
            for (int i = 0; i < STAGES; ++i) {
                tc::mbar_init(&bars[t].full[i], 1);
                tc::mbar_init(&bars[t].empty[i], 1);
            }
            tc::mbar_init(&bars[t].q_full, ROW_WARPS);
            tc::mbar_init(&bars[t].s_full, 1);
            tc::mbar_init(&bars[t].s_free, ROW_WARPS);
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

    // The place's tiles: the first places take theirs in order, the second ones backwards from twice the blocks, so that an SM's two
    // add up to about the same; every place then goes on by that many.  Number i is tile i / kv_heads of key/value head i % kv_heads.
    const int ratio = heads / kv_heads, tok = ROWS / r_pad;
    const int place = warp >= 4 ? (warp - 4) / ROW_WARPS : warp >= 2 ? 1 : 0;
    const int stride = PLACES * (int)gridDim.x, first_tile = place ? stride - 1 - (int)blockIdx.x : (int)blockIdx.x;
    auto tile_of = [&](int i) -> Tile { return find_tile(i / kv_heads, row_start, row_count, history, requests, tok, window, chunk); };
    Bars& b = bars[place];
    uint8_t* q_smem = smem + place * PLACE_BYTES;
    const uint32_t tile_tmem = tmem_base + place * PLACE_COLS;

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(FEWER_REGISTERS));
        if (warp == 0 || warp == 3) {
            // Lane l < 12: tokens 16 (l / 4) on of the stage, values 64 (l % 4) on of the row.  Tokens past the last key, or on a
            // page that a window has given back, are read from page 0 (and overwritten with zeros).
            const bool copies = lane < 4 * (KEYS / RUN);
            uint8_t* dst = q_smem + Q_BYTES + (lane & 3) * BLOCK_BYTES + (lane >> 2) * RUN * 128;
            bool ok = true;
            for (int i = first_tile, c = 0; ok; i += stride) {       // c: the place's stages so far
                const Tile w = tile_of(i);
                if (w.n_iter == 0) break;
                const int* table = block_tables + (size_t)w.request * table_stride;
                for (int j = 0; j < w.n_iter; ++j, ++c) {
                    const int st = c % STAGES, t = w.begin + j * KEYS + RUN * (lane >> 2);
                    const int page = copies && t < w.key_end ? max(table[t / page_size], 0) : 0;
                    ok = tc::mbar_wait_warp(&b.empty[st], ((c / STAGES) & 1u) ^ 1u, abort_flag, error_word, ERR_ROWS_PRODUCER);
                    if (!ok) break;
                    if (lane == 0) tc::mbar_expect_tx(&b.full[st], STAGE_BYTES);
                    __syncwarp();
                    if (copies)
                        tc::tma_load_2d(dst + st * STAGE_BYTES, &cache_map, (lane & 3) * 64, (page * kv_heads + i % kv_heads) * page_size + t % page_size,
                                        &b.full[st]);
                }
            }
        } else if (tc::elect_one()) {
            const uint32_t q_addr = tc::smem_u32(q_smem);
            auto scores = [&](int c) -> bool {               // S = Q K^T of stage c
                const int st = c % STAGES;
                if (!tc::mbar_wait(&b.full[st], (c / STAGES) & 1u, abort_flag, error_word, ERR_ROWS_MMA)) return false;
                tc::tc_fence_after();
                const uint32_t k_addr = q_addr + Q_BYTES + st * STAGE_BYTES;
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk)
                    tc::mma_bf16_ss(tile_tmem + TMEM_S, tc::smem_desc_k_sw128(q_addr + (kk >> 2) * Q_BLOCK + (kk & 3) * 32),
                                    tc::smem_desc_k_sw128(k_addr + (kk >> 2) * BLOCK_BYTES + (kk & 3) * 32), IDESC_QK, kk > 0 ? 1u : 0u);
                tc::mma_commit(&b.s_full);
                return true;
            };
            bool ok = true;
            for (int i = first_tile, c = 0, n = 0; ok; i += stride, ++n) {
                const int end = c + tile_of(i).n_iter;
                if (end == c) break;
                ok = tc::mbar_wait(&b.q_full, n & 1u, abort_flag, error_word, ERR_ROWS_MMA) && scores(c);
                for (; ok && c < end; ++c) {
                    // The next stage's scores as soon as these have been read, so that they are there when the weights are done.
                    if (c + 1 < end) ok = tc::mbar_wait(&b.s_free, c & 1u, abort_flag, error_word, ERR_ROWS_MMA) && scores(c + 1);
                    ok = ok && tc::mbar_wait(&b.p_full, c & 1u, abort_flag, error_word, ERR_ROWS_MMA);
                    if (!ok) break;
                    tc::tc_fence_after();
                    const uint32_t v_addr = q_addr + Q_BYTES + c % STAGES * STAGE_BYTES + 2 * BLOCK_BYTES;
#pragma unroll
                    for (int part = 2; part >= 0; --part)
#pragma unroll
                        for (int kk = 0; kk < KEYS / 16; ++kk)
                            tc::mma_bf16_ts(tile_tmem + TMEM_O, tile_tmem + part * P_PART + kk * 8,
                                            attn::smem_desc_mn_sw128(v_addr + kk * 16 * 128, BLOCK_BYTES), IDESC_PV, part < 2 || kk > 0 ? 1u : 0u);
                    tc::mma_commit(&b.empty[c % STAGES]);
                    tc::mma_commit(&b.o_full);
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(MORE_REGISTERS));
        const int quarter = warp & 3, row = quarter * 32 + lane;
        const int tk = row / r_pad, hd = row % r_pad;
        const uint32_t lanes = tile_tmem + ((uint32_t)(quarter * 32) << 16);
        bool ok = true;
        for (int i = first_tile, c = 0; ok; i += stride) {
            int n_iter, begin, key_lo, key_end, pos, at;         // at: the row of queries and outputs, or -1
            {
                const Tile w = tile_of(i);
                n_iter = w.n_iter, begin = w.begin, key_lo = w.key_lo, key_end = w.key_end, pos = w.hist + w.t0 + tk;
                at = tk < w.n_tok && hd < ratio ? (w.a0 + w.t0 + tk) * heads + i % kv_heads * ratio + hd : -1;
            }
            if (n_iter == 0) break;
            {
                // (All products of the tile before have run: its last output has been read.)
                const uint4* src = reinterpret_cast<const uint4*>(q + (size_t)max(at, 0) * D);
#pragma unroll
                for (int k = 0; k < D / 8; ++k)
                    *reinterpret_cast<uint4*>(q_smem + (k >> 3) * Q_BLOCK + attn::swz(row, k & 7)) = at >= 0 ? src[k] : make_uint4(0u, 0u, 0u, 0u);
            }
            tc::fence_proxy_async();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&b.q_full);

            const int lo_key = lowest_key(pos, window, chunk);
            float m_used = -INFINITY, l_run = 0.0f, o[D];
#pragma unroll
            for (int d = 0; d < D; ++d) o[d] = 0.0f;
            // What stage n made of the output joins the row's sums; that stage is then done with its weights too.
            auto take_output = [&](int n) -> bool {
                if (!tc::mbar_wait_warp(&b.o_full, n & 1u, abort_flag, error_word, ERR_ROWS_SOFTMAX)) return false;
                tc::tc_fence_after();
#pragma unroll
                for (int k = 0; k < D; k += 32) {
                    uint32_t v[32];
                    tc::tmem_ld_32x32(lanes + TMEM_O + k, v);
                    tc::tmem_wait_ld();
#pragma unroll
                    for (int u = 0; u < 32; ++u) o[k + u] += __uint_as_float(v[u]);
                }
                return true;
            };
            for (int j = 0; j < n_iter; ++j, ++c) {
                const int key0 = begin + j * KEYS;
                if (key0 < key_lo || key0 + KEYS > key_end) {
                    // Slots of the stage that no row may see: a zero weight must meet a finite value.  Thread r has key r % 48, half r / 48.
                    ok = tc::mbar_wait_warp(&b.full[c % STAGES], (c / STAGES) & 1u, abort_flag, error_word, ERR_ROWS_SOFTMAX);
                    if (!ok) break;
                    const int s = row % KEYS, key = key0 + s;
                    if (row < 2 * KEYS && (key < key_lo || key >= key_end)) {
                        uint4* v = reinterpret_cast<uint4*>(q_smem + Q_BYTES + c % STAGES * STAGE_BYTES + (2 + row / KEYS) * BLOCK_BYTES + s * 128);
#pragma unroll
                        for (int k = 0; k < 8; ++k) v[k] = make_uint4(0u, 0u, 0u, 0u);
                    }
                    tc::fence_proxy_async();
                }
                ok = tc::mbar_wait_warp(&b.s_full, c & 1u, abort_flag, error_word, ERR_ROWS_SOFTMAX);
                if (!ok) break;
                tc::tc_fence_after();
                uint32_t sc[KEYS];
                tc::tmem_ld_32x32(lanes + TMEM_S, *reinterpret_cast<uint32_t(*)[32]>(&sc[0]));
                tc::tmem_ld_32x16(lanes + TMEM_S + 32, *reinterpret_cast<uint32_t(*)[16]>(&sc[32]));
                tc::tmem_wait_ld();
                tc::tc_fence_before();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&b.s_free);
                // Keys key0 + first .. key0 + last - 1 of the stage are the row's.
                const int first = lo_key - key0, last = pos + 1 - key0;
                if (first > 0 || last < KEYS) {
#pragma unroll
                    for (int k = 0; k < KEYS; ++k)
                        if (k >= last || k < first) sc[k] = __float_as_uint(-INFINITY);
                }
                float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int k = 0; k < KEYS; k += 8)
#pragma unroll
                    for (int u = 0; u < 4; ++u) mx[u] = attn::max3(mx[u], __uint_as_float(sc[k + 2 * u]), __uint_as_float(sc[k + 2 * u + 1]));
                // The scale is positive: it is applied after the maximum and folded into the exponent's multiply-add.
                const float cand = fmaxf(m_used, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * scale_log2);
                ok = j == 0 || take_output(c - 1);
                if (!ok) break;
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
                for (int k = 0; k < KEYS; k += 16) {
                    uint32_t p[3][8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        const float x = exp2f(fmaf(__uint_as_float(sc[k + 2 * u]), scale_log2, -base));
                        const float y = exp2f(fmaf(__uint_as_float(sc[k + 2 * u + 1]), scale_log2, -base));
                        sum[u & 3] += x + y;
                        attn::split3_pair(x, y, p[0][u], p[1][u], p[2][u]);
                    }
#pragma unroll
                    for (int u = 0; u < 3; ++u) tmem_st_32x8(lanes + u * P_PART + k / 2, p[u]);
                }
                l_run += (sum[0] + sum[1]) + (sum[2] + sum[3]);
                tc::tmem_wait_st();
                tc::tc_fence_before();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&b.p_full);
            }
            ok = ok && take_output(c - 1);
            if (ok && at >= 0) {
                const float inv = 1.0f / l_run;
#pragma unroll
                for (int d = 0; d < D; d += 8) {
                    uint32_t v[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) v[u] = attn::pack_bf16(o[d + 2 * u] * inv, o[d + 2 * u + 1] * inv);
                    *reinterpret_cast<uint4*>(out + (size_t)at * D + d) = make_uint4(v[0], v[1], v[2], v[3]);
                }
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
        pool_rows <= 0 || pool_rows >= (1ll << 31) || (long long)rows * heads >= (1ll << 31) || !(scale > 0.0f) || (((uintptr_t)q | (uintptr_t)cache | (uintptr_t)out) & 15))
        return LLMX_ERR_UNSUPPORTED;
    static const bool enough = registers_reach(attention_rows_kernel, THREADS, FEWER_REGISTERS + PLACES * MORE_REGISTERS);
    if (!enough) return LLMX_ERR_UNSUPPORTED;
    int r_pad = 1;
    while (r_pad < heads / kv_heads) r_pad *= 2;
    const int tok = ROWS / r_pad;
    CUtensorMap map;
    if (int e = llmx_make_map_bf16_2d(&map, cache, (uint64_t)pool_rows, 2 * D, RUN, 64)) return e;
    if (cudaFuncSetAttribute(attention_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess) return (int)cudaGetLastError();
    const long long tiles = (((long long)rows + tok - 1) / tok + requests) * kv_heads;        // at most
    launch_kernel(attention_rows_kernel, dim3((unsigned)(tiles < SMS ? tiles : SMS)), dim3(THREADS), (size_t)SMEM_BYTES, stream,
                  map, (const __nv_bfloat16*)q, (__nv_bfloat16*)out, row_start, row_count, history, block_tables, table_stride, requests, heads,
                  kv_heads, page_size, window, chunk, scale * attn::LOG2E, r_pad, error_word);
    return launch_status();
}
