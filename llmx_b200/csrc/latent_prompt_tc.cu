// Latent attention for requests that bring many rows: keys and values made once a step, softmax attention over them on
// the 5th-generation tensor cores.
//
// A cached token is [c ; r] (C latent values, R rotated ones shared by the heads); head h's key is [Wuk_h c ; r], its
// value Wuv_h c.  The general form (latent_attention.cu) never makes them: every (row, head, key) costs 2 C + R
// multiply-adds over the latent itself.  For a request with many rows the other order is cheaper: a key and a value per
// (token, head) are made once, (D + V) C multiply-adds, and a (row, head, key) costs D + R + V.  Two kernels:
//
//   latent_expand   128 keys x one head a block: [K_h | V_h] = c [Wuk_h | Wuv_h]^T (bfloat16 in, 32-bit sums), written to
//                   a workspace as three bfloat16 parts a value
//   latent_prompt   128 rows x one head a block: S = Q K^T, online softmax, O += P V
//
// 32-bit factors on 16-bit operands.  Queries, keys, weights and values are 32-bit numbers here.  Each is cut into three
// bfloat16 parts of 8 significand bits (hi + mid + lo is the number itself, all 24 bits), and a product of two such
// numbers is the six products of parts that reach 2^-24 of it: lo hi, hi lo, mid mid, mid hi, hi mid, hi hi, small ones
// first.  The rotated key part is bfloat16 in the cache and needs three.  That is 6 (D + V) + 3 R = 1,728 multiply-adds
// a (row, head, key) for D = V = 128, R = 64, against 3 (2 C + R) = 3,264 of the general form, which also has 16 rows to
// an instruction where these have 128.
//
// What bounds `latent_prompt` is the tensor core and the turns it takes with the softmax: 84 products of a stage of 64
// keys (3,456 cycles at the full rate), then the 64 scores of a row are turned into weights by its thread.  The query's
// parts lie in tensor memory (288 columns), beside the scores / weights (96 columns: three parts of 64 weights over the
// scores they came from) and a stage's output (128 columns): all 512 columns, so one block per SM and one tile in flight.
//
// The tensor core cuts off what an addition shifts out of its accumulator.  A stage's output (and 64 columns of an expanded key or
// value, below) therefore starts from nothing
// and joins the row's sums, which its thread holds in registers, by a rounded addition, while the next stage's scores are
// made; added up over the stages in tensor memory, 3,500 keys cost five times the values (0.8 % against 0.15 %) that
// round to another bfloat16 than the exact ones.
//
// Both kernels together, 2,048 rows after nothing: 16 heads 247 us, 32 heads 402 us; 32 heads, 2,048 rows after 4,096 tokens
// under a window of 4,096: 1,068 us.  The general form: 2,639, 5,142 and 14,506 us.
//
// Shapes: D = V = 128, R a multiple of 8 up to 64, C a multiple of 64, pages of a multiple of 16 tokens, bfloat16 cache
// and maps.  Every wait on an mbarrier is bounded (tc_common.cuh).
#include "attn_parts.cuh"
#include <math.h>

namespace {

constexpr int D = 128;                        // unrotated key width = value width of a head
constexpr int ROWS = 128;                     // query rows (the products' M), keys of an expansion tile
constexpr int KEYS = 64;                      // keys a stage (N of Q K^T, K of P V)
constexpr int BLOCK_BYTES = KEYS * 128;       // 64 keys x 64 columns
constexpr int K_BLOCKS = 7, V_BLOCKS = 6;     // hi, mid, lo of the key (2 blocks each), the rotated part; hi, mid, lo of the value
constexpr int TOKEN_BLOCKS = K_BLOCKS + V_BLOCKS;         // blocks of 64 values the workspace has for a (token, head)
constexpr int STAGE_BYTES = TOKEN_BLOCKS * BLOCK_BYTES;
constexpr int STAGES = 2;
constexpr int PROMPT_SMEM = STAGES * STAGE_BYTES + 1024 + 256;
constexpr int PROMPT_THREADS = 192;           // producer warp, product warp, four warps of one row a thread
constexpr int ROW_WARPS = 4;
constexpr uint32_t TMEM_Q = 0, Q_PART = 96, Q_ROT = 64;   // a part of the query: 64 columns unrotated, 32 rotated
constexpr uint32_t TMEM_S = 288, P_PART = 32, TMEM_O = 384;
constexpr float RAISE = 8.0f;                 // the exponent's maximum follows the true one when it is 2^8 behind
enum : int { ERR_LAT_PRODUCER = 421, ERR_LAT_MMA = 422, ERR_LAT_ROWS = 423, ERR_LAT_EXPAND = 424 };

constexpr uint32_t IDESC_QK = tc::instr_desc_bf16(ROWS, KEYS);
constexpr uint32_t IDESC_PV = tc::instr_desc_bf16(ROWS, D) | (1u << 16);       // values: the MN-major operand
constexpr uint32_t IDESC_EXPAND = tc::instr_desc_bf16(ROWS, D);

__device__ __forceinline__ void tmem_st_32x1(uint32_t addr, uint32_t v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(addr), "r"(v) : "memory");
}

// Whether all 128 threads of four warps say so (named barrier `id`).
__device__ __forceinline__ bool all_four_warps(int id, bool mine) {
    uint32_t all;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, %2, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(all) : "r"(mine ? 1u : 0u), "r"(id) : "memory");
    return all != 0;
}

// The keys a request's rows see, from its first row's window to its last row's own; the workspace starts at the stage
// boundary below.
__device__ __forceinline__ int first_key(int pos_first, int window) {
    return window > 0 ? max(0, pos_first - window + 1) : 0;
}

// requests[4 i ..]: first row, rows, first workspace token, workspace tokens (a multiple of 128) of request i.
// 128 keys x one head: two products of 128 x 128 (key, value) over C in steps of 64 columns.  A step's products start from nothing, in
// one of two pairs of accumulators, and join the 128 sums that a thread holds in registers by rounded additions while the next step's
// run: over C / 16 additions in one accumulator, each of which the tensor core cuts off, 0.06 % of the attention's results at
// 128 to 512 keys rounded to another bfloat16 than the exact ones (general form 0.03 to 0.05 %), so 0.02 to 0.03 %.
//   warp 0      producer, warp 1 products; warps 2 and 3 idle
//   warps 4-7   the keys' sums, one thread a key; warps 8-11 the values'
// The three parts of the sums are laid out in shared memory (the operands' stages are free then) and leave by TMA, whole 128-byte
// lines.  Bound by the writes to the workspace (1,664 bytes a token and head), which one block an SM does not overlap with the next
// one's products: 2,048 tokens of 16 heads 35 us, 5,003 tokens of 32 133 us (27 and 96 with one accumulator and two blocks an SM).
constexpr int EXPAND_STAGE = 3 * ROWS * 128;                // 128 keys, 128 + 128 rows of the maps, 64 columns each
constexpr int EXPAND_STAGES = 4;
static_assert(EXPAND_STAGES * EXPAND_STAGE >= 2 * 6 * ROWS * 128, "the parts of 128 keys and values");
constexpr int EXPAND_SMEM = EXPAND_STAGES * EXPAND_STAGE + 1024 + 256;
// Launched with 3 x 128 x 168 registers; the first group gives back what the sums need: 40 + 232 + 232 = 3 x 168.
constexpr int EXPAND_THREADS = 3 * 128, FEWER_REGISTERS = 40, MORE_REGISTERS = 232;
static_assert(FEWER_REGISTERS + 2 * MORE_REGISTERS <= 3 * 168, "setmaxnreg draws on the block's registers at launch");

__global__ void __launch_bounds__(EXPAND_THREADS, 1)
latent_expand_kernel(const __grid_constant__ CUtensorMap cache_map, const __grid_constant__ CUtensorMap uk_map,
                     const __grid_constant__ CUtensorMap uv_map, const __grid_constant__ CUtensorMap expanded_map, const __nv_bfloat16* __restrict__ cache,
                     __nv_bfloat16* __restrict__ expanded, const int* __restrict__ requests,
                     const int* __restrict__ row_request, const int* __restrict__ positions,
                     const int* __restrict__ block_tables, int table_stride, int tokens, int head0, int C, int R,
                     int page_size, int window, int* error_word) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full = (uint64_t*)(smem + EXPAND_STAGES * EXPAND_STAGE);
    uint64_t* empty = full + EXPAND_STAGES;
    uint64_t *made = empty + EXPAND_STAGES, *taken = made + 2;          // [2] a step's products are complete / have joined the sums
    uint32_t* tmem_slot = (uint32_t*)(taken + 2);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < EXPAND_STAGES; ++i) {
            tc::mbar_init(&full[i], 1);
            tc::mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            tc::mbar_init(&made[i], 1);
            tc::mbar_init(&taken[i], 2 * ROW_WARPS);
        }
        *abort_flag = 0;
        tc::fence_barrier_init();
        tc::tma_prefetch_desc(&cache_map);
        tc::tma_prefetch_desc(&uk_map);
        tc::tma_prefetch_desc(&uv_map);
    }
    if (warp == 1) {
        tc::tmem_alloc(tmem_slot, 4 * D);
        tc::tmem_relinquish();
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_trigger();
    pdl_wait();

    const int* rq = requests + 4 * blockIdx.z;
    const int row0 = rq[0], rows = rq[1];
    const int lo = first_key(positions[row0], window), end = positions[row0 + rows - 1] + 1;
    const int key0 = lo / KEYS * KEYS + (int)blockIdx.x * ROWS;
    const int head = head0 + blockIdx.y;
    // Tokens past the request's last, and what its share of the workspace does not hold, are not made.
    const bool active = key0 < end && (int)(blockIdx.x + 1) * ROWS <= rq[3];
    const int* table = block_tables + (size_t)row_request[row0] * table_stride;
    const int n_steps = C / 64;

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(FEWER_REGISTERS));
        if (active && warp == 0) {
            // Lane l < 8: the sixteen keys from key0 + 16 l; a page that the window has given back (-1), or past the last key,
            // is read from page 0 and written as zeros.
            const int t = key0 + 16 * lane;
            const int page = lane < 8 && t < end ? max(table[t / page_size], 0) : 0;
            const int slot = page * page_size + t % page_size;
            for (int s = 0; s < n_steps; ++s) {
                const int st = s % EXPAND_STAGES;
                if (!tc::mbar_wait_warp(&empty[st], ((s / EXPAND_STAGES) & 1u) ^ 1u, abort_flag, error_word, ERR_LAT_EXPAND)) break;
                uint8_t* base = smem + st * EXPAND_STAGE;
                if (lane == 0) tc::mbar_expect_tx(&full[st], EXPAND_STAGE);
                __syncwarp();
                if (lane < 8) tc::tma_load_2d(base + lane * 16 * 128, &cache_map, s * 64, slot, &full[st]);
                else if (lane == 8) tc::tma_load_2d(base + ROWS * 128, &uk_map, s * 64, head * D, &full[st]);
                else if (lane == 9) tc::tma_load_2d(base + 2 * ROWS * 128, &uv_map, s * 64, head * D, &full[st]);
            }
        } else if (active && warp == 1) {
            if (tc::elect_one()) {
                for (int s = 0; s < n_steps; ++s) {
                    const int st = s % EXPAND_STAGES;
                    if (!tc::mbar_wait(&taken[s & 1], ((s >> 1) & 1u) ^ 1u, abort_flag, error_word, ERR_LAT_EXPAND) ||
                        !tc::mbar_wait(&full[st], (s / EXPAND_STAGES) & 1u, abort_flag, error_word, ERR_LAT_EXPAND))
                        break;
                    tc::tc_fence_after();
                    const uint32_t a = tc::smem_u32(smem + st * EXPAND_STAGE);
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                        for (int w = 0; w < 2; ++w)
                            tc::mma_bf16_ss(tmem_base + (2 * (s & 1) + w) * D, tc::smem_desc_k_sw128(a + kk * 32),
                                            tc::smem_desc_k_sw128(a + (1 + w) * ROWS * 128 + kk * 32), IDESC_EXPAND, kk > 0 ? 1u : 0u);
                    tc::mma_commit(&empty[st]);
                    tc::mma_commit(&made[s & 1]);
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(MORE_REGISTERS));
        if (active) {
            const int which = (warp - 4) / ROW_WARPS;          // 0: keys, 1: values
            const int quarter = warp & 3, row = quarter * 32 + lane, t = key0 + row;
            const bool real = t >= lo && t < end;
            const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
            if (which == 0) {
                __nv_bfloat16* dst = expanded + ((size_t)blockIdx.y * tokens + rq[2] + blockIdx.x * ROWS + row) * (TOKEN_BLOCKS * 64);
                uint4* rot = reinterpret_cast<uint4*>(dst + 3 * D);
                const uint4* src = reinterpret_cast<const uint4*>(
                    cache + ((size_t)(real ? table[t / page_size] : 0) * page_size + t % page_size) * (C + R) + C);
#pragma unroll
                for (int i = 0; i < 8; ++i) rot[i] = real && i * 8 < R ? src[i] : zero;
            }
            float sum[D];
#pragma unroll
            for (int d = 0; d < D; ++d) sum[d] = 0.0f;
            bool ok = true;
            for (int s = 0; s < n_steps; ++s) {
                ok = tc::mbar_wait_warp(&made[s & 1], (s >> 1) & 1u, abort_flag, error_word, ERR_LAT_EXPAND);
                if (!ok) break;
                tc::tc_fence_after();
#pragma unroll
                for (int c = 0; c < D; c += 32) {
                    uint32_t v[32];
                    tc::tmem_ld_32x32(tmem_base + (2 * (s & 1) + which) * D + c + ((uint32_t)(quarter * 32) << 16), v);
                    tc::tmem_wait_ld();
#pragma unroll
                    for (int k = 0; k < 32; ++k) sum[c + k] += __uint_as_float(v[k]);
                }
                tc::tc_fence_before();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&taken[s & 1]);
            }
            // The last step's products are complete, so all stages are free.  The four warps of keys, or of values, go on together or
            // not at all: they meet at a barrier below.
            uint8_t* parts = smem + which * 6 * ROWS * 128;
            if (all_four_warps(1 + which, ok)) {
#pragma unroll
                for (int c = 0; c < D; c += 8) {
                    uint32_t p[3][4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) attn::split3_pair(sum[c + 2 * u], sum[c + 2 * u + 1], p[0][u], p[1][u], p[2][u]);
#pragma unroll
                    for (int q = 0; q < 3; ++q)
                        *reinterpret_cast<uint4*>(parts + (2 * q + (c >> 6)) * ROWS * 128 + attn::swz(row, (c & 63) >> 3)) =
                            real ? make_uint4(p[q][0], p[q][1], p[q][2], p[q][3]) : zero;
                }
                tc::fence_proxy_async();
                all_four_warps(1 + which, true);
                if (quarter == 0 && lane == 0) {
                    for (int b = 0; b < 12; ++b)
                        asm volatile("cp.async.bulk.tensor.5d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5, %6}], [%1];"
                                     ::"l"(&expanded_map), "r"(tc::smem_u32(parts + (b >> 1) * ROWS * 128 + (b & 1) * BLOCK_BYTES)), "r"(0),
                                     "r"(rq[2] + (int)blockIdx.x * ROWS + (b & 1) * KEYS), "r"((which ? K_BLOCKS : 0) + (b >> 1)), "r"((int)blockIdx.y),
                                     "r"(0) : "memory");
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
                }
            }
            tc::tc_fence_before();
        }
    }
    __syncthreads();
    if (warp == 1) {
        tc::tc_fence_after();
        tc::tmem_dealloc(tmem_base, 4 * D);
    }
}

// tiles[4 i ..]: first row, rows (up to 128), first workspace token of its request, first row of its request.  The tiles
// of a request come with its last rows first (they see the most keys), a head's tiles before the next head's, so that the
// blocks in flight read few heads' keys and values: those stay in the L2 cache.
__global__ void __launch_bounds__(PROMPT_THREADS, 1)
latent_prompt_kernel(const __grid_constant__ CUtensorMap expanded_map, const float* __restrict__ q, int q_stride,
                     __nv_bfloat16* __restrict__ out, const int* __restrict__ tiles, const float* __restrict__ freq, int rot_pairs,
                     int rot_halves, float rot_mag, const int* __restrict__ positions, int heads, int head0, int R, int window,
                     float scale_log2, int* error_word) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = (uint64_t*)(smem + STAGES * STAGE_BYTES);
    uint64_t *k_full = bars, *v_full = bars + 2, *k_empty = bars + 4, *v_empty = bars + 6;
    uint64_t* q_full = bars + 8;                   // the query's parts are in tensor memory
    uint64_t* s_full = bars + 9;                   // a stage's scores are complete
    uint64_t* p_full = bars + 10;                  // a stage's weights are in tensor memory, the output of the stage before has been read
    uint64_t* o_full = bars + 11;                  // a stage's output is complete
    uint32_t* tmem_slot = (uint32_t*)(bars + 12);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 8; ++i) tc::mbar_init(&bars[i], 1);
        tc::mbar_init(q_full, ROW_WARPS);
        tc::mbar_init(s_full, 1);
        tc::mbar_init(p_full, ROW_WARPS);
        tc::mbar_init(o_full, 1);
        *abort_flag = 0;
        tc::fence_barrier_init();
        tc::tma_prefetch_desc(&expanded_map);
    }
    if (warp == 1) {
        tc::tmem_alloc(tmem_slot, 512);
        tc::tmem_relinquish();
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_trigger();
    pdl_wait();

    const int* tile = tiles + 4 * blockIdx.x;
    const int row0 = tile[0], n_rows = tile[1];
    const int base_key = first_key(positions[tile[3]], window) / KEYS * KEYS;         // the key of the request's first workspace token
    const int begin = first_key(positions[row0], window) / KEYS * KEYS;
    const int n_iter = (positions[row0 + n_rows - 1] + 1 - begin + KEYS - 1) / KEYS;

    if (warp == 0) {
        const int token0 = tile[2] + begin - base_key;
        const bool value = lane >= K_BLOCKS;
        uint64_t* full = value ? v_full : k_full;
        uint64_t* empty = value ? v_empty : k_empty;
        bool ok = true;
        for (int j = 0; j < n_iter && ok; ++j) {
            const int st = j & 1;
            // Keys and values have barriers of their own: the keys' buffer is free a product earlier than the values'.
            for (int half = 0; half < 2 && ok; ++half) {
                if ((int)value == half) {
                    ok = tc::mbar_wait(&empty[st], ((j >> 1) & 1u) ^ 1u, abort_flag, error_word, ERR_LAT_PRODUCER);
                    if (ok && (lane == 0 || lane == K_BLOCKS)) tc::mbar_expect_tx(&full[st], (value ? V_BLOCKS : K_BLOCKS) * BLOCK_BYTES);
                }
                ok = __all_sync(0xffffffffu, ok);
                if (ok && (int)value == half && lane < TOKEN_BLOCKS)
                    tc::tma_load_5d(smem + st * STAGE_BYTES + lane * BLOCK_BYTES, &expanded_map, 0, token0 + j * KEYS, lane, (int)blockIdx.y, 0, &full[st]);
            }
        }
    } else if (warp == 1) {
        if (tc::elect_one()) {
            const uint32_t tq = tmem_base + TMEM_Q, ts = tmem_base + TMEM_S, to = tmem_base + TMEM_O;
            // Which part of the one factor meets which of the other (0 hi, 1 mid, 2 lo), small products first.
            constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0};
            bool ok = tc::mbar_wait(q_full, 0, abort_flag, error_word, ERR_LAT_MMA);
            for (int j = 0; j < n_iter && ok; ++j) {
                const int st = j & 1;
                const uint32_t ph = (j >> 1) & 1u;
                ok = tc::mbar_wait(&k_full[st], ph, abort_flag, error_word, ERR_LAT_MMA);
                if (!ok) break;
                tc::tc_fence_after();
                // The products of one thread run in the order they are issued: the weights these scores overwrite have
                // been read by the stage before's P V.
                const uint32_t k_addr = tc::smem_u32(smem + st * STAGE_BYTES), v_addr = k_addr + K_BLOCKS * BLOCK_BYTES;
#pragma unroll
                for (int p = 0; p < 6; ++p) {
                    if (p == 0 || p == 3 || p == 5) {             // the rotated part with lo, mid, hi of the query
                        const int qp = p == 0 ? 2 : p == 3 ? 1 : 0;
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk)
                            tc::mma_bf16_ts(ts, tq + qp * Q_PART + Q_ROT + kk * 8, tc::smem_desc_k_sw128(k_addr + 6 * BLOCK_BYTES + kk * 32), IDESC_QK,
                                            (p > 0 || kk > 0) ? 1u : 0u);
                    }
#pragma unroll
                    for (int kk = 0; kk < 8; ++kk)
                        tc::mma_bf16_ts(ts, tq + PA[p] * Q_PART + kk * 8,
                                        tc::smem_desc_k_sw128(k_addr + (2 * PB[p] + (kk >> 2)) * BLOCK_BYTES + (kk & 3) * 32), IDESC_QK, 1u);
                }
                tc::mma_commit(s_full);
                tc::mma_commit(&k_empty[st]);
                ok = tc::mbar_wait(&v_full[st], ph, abort_flag, error_word, ERR_LAT_MMA) &&
                     tc::mbar_wait(p_full, j & 1u, abort_flag, error_word, ERR_LAT_MMA);
                if (!ok) break;
                tc::tc_fence_after();
#pragma unroll
                for (int p = 0; p < 6; ++p)
#pragma unroll
                    for (int kk = 0; kk < KEYS / 16; ++kk)
                        tc::mma_bf16_ts(to, ts + PA[p] * P_PART + kk * 8,
                                        attn::smem_desc_mn_sw128(v_addr + 2 * PB[p] * BLOCK_BYTES + kk * 16 * 128, BLOCK_BYTES), IDESC_PV,
                                        (p > 0 || kk > 0) ? 1u : 0u);
                tc::mma_commit(&v_empty[st]);
                tc::mma_commit(o_full);
            }
        }
    } else {
        const int quarter = warp & 3, row = quarter * 32 + lane, head = head0 + blockIdx.y;
        const bool valid = row < n_rows;
        const int r = row0 + (valid ? row : 0);
        const int pos = positions[r];
        const uint32_t lanes = tmem_base + ((uint32_t)(quarter * 32) << 16);
        const float* src = q + (size_t)r * q_stride + (size_t)head * (D + R);
        // ---- the query, scaled for exponentials of base 2, in three parts; its rotated part turned, and zeros up to 64
#pragma unroll 1
        for (int c = 0; c < D; c += 32) {
            uint32_t p[3][16];
#pragma unroll
            for (int u = 0; u < 16; ++u) {
                const float2 x = *reinterpret_cast<const float2*>(src + c + 2 * u);
                attn::split3_pair(valid ? x.x * scale_log2 : 0.0f, valid ? x.y * scale_log2 : 0.0f, p[0][u], p[1][u], p[2][u]);
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) tc::tmem_st_32x16(lanes + TMEM_Q + k * Q_PART + c / 2, p[k]);
        }
        auto turned = [&](int e) -> float {
            if (!valid || e >= R) return 0.0f;
            if (e >= 2 * rot_pairs) return src[D + e] * scale_log2;
            const bool second = rot_halves ? e >= rot_pairs : (e & 1);
            const int i = rot_halves ? (second ? e - rot_pairs : e) : e >> 1;
            const float other = src[D + (rot_halves ? (second ? i : i + rot_pairs) : e ^ 1)];
            float sn, cs;
            sincosf((float)pos * freq[i], &sn, &cs);
            sn *= rot_mag;
            cs *= rot_mag;
            return (second ? src[D + e] * cs + other * sn : src[D + e] * cs - other * sn) * scale_log2;
        };
#pragma unroll 1
        for (int e = 0; e < 64; e += 2) {
            uint32_t hi, mid, lo;
            attn::split3_pair(turned(e), turned(e + 1), hi, mid, lo);
            __syncwarp();
            tmem_st_32x1(lanes + TMEM_Q + Q_ROT + e / 2, hi);
            tmem_st_32x1(lanes + TMEM_Q + Q_PART + Q_ROT + e / 2, mid);
            tmem_st_32x1(lanes + TMEM_Q + 2 * Q_PART + Q_ROT + e / 2, lo);
        }
        tc::tmem_wait_st();
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(q_full);

        const int lo_key = first_key(pos, window);
        float m_used = -INFINITY, l_run = 0.0f, o[D];
#pragma unroll
        for (int d = 0; d < D; ++d) o[d] = 0.0f;
        // What stage j made of the output joins the row's sums.
        auto take_output = [&](int j) -> bool {
            if (!tc::mbar_wait_warp(o_full, j & 1u, abort_flag, error_word, ERR_LAT_ROWS)) return false;
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
        for (int j = 0; j < n_iter; ++j) {
            ok = j == 0 || take_output(j - 1);
            ok = ok && tc::mbar_wait_warp(s_full, j & 1u, abort_flag, error_word, ERR_LAT_ROWS);
            if (!ok) break;
            tc::tc_fence_after();
            const int key0 = begin + j * KEYS;
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
            const float cand = fmaxf(m_used, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])));
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
                    const float a = exp2f(__uint_as_float(sc[c + 2 * u]) - base), b = exp2f(__uint_as_float(sc[c + 2 * u + 1]) - base);
                    sum[u & 3] += a + b;
                    attn::split3_pair(a, b, p[0][u], p[1][u], p[2][u]);
                }
#pragma unroll
                for (int k = 0; k < 3; ++k) tc::tmem_st_32x16(lanes + TMEM_S + k * P_PART + c / 2, p[k]);
            }
            if (raise) {                             // the sums so far were made against the old maximum
#pragma unroll
                for (int d = 0; d < D; ++d) o[d] *= factor;
                l_run *= factor;
            }
            l_run += (sum[0] + sum[1]) + (sum[2] + sum[3]);
            tc::tmem_wait_st();
            tc::tc_fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(p_full);
        }
        if (ok && take_output(n_iter - 1) && valid) {
            const float inv = 1.0f / l_run;
            __nv_bfloat16* dst = out + ((size_t)r * heads + head) * D;
#pragma unroll
            for (int d = 0; d < D; d += 8) {
                uint32_t w[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) w[u] = attn::pack_bf16(o[d + 2 * u] * inv, o[d + 2 * u + 1] * inv);
                *reinterpret_cast<uint4*>(dst + d) = make_uint4(w[0], w[1], w[2], w[3]);
            }
        }
        tc::tc_fence_before();
    }
    __syncthreads();
    if (warp == 1) {
        tc::tc_fence_after();
        tc::tmem_dealloc(tmem_base, 512);
    }
}

// The workspace [heads, tokens, 13 blocks of 64 values] as (64 values) x (token) x (block) x (head), box 64 x 64 tokens.
int make_expanded_map(CUtensorMap* map, const void* base, uint64_t tokens, uint64_t heads) {
    llmx_encode_tiled_fn enc = llmx_encode_tiled();
    if (!enc) return 10003;
    const cuuint64_t dims[5] = {64, tokens, TOKEN_BLOCKS, heads, 1};
    const cuuint64_t strides[4] = {TOKEN_BLOCKS * 128, 128, tokens * TOKEN_BLOCKS * 128, heads * tokens * TOKEN_BLOCKS * 128};
    const cuuint32_t box[5] = {64, KEYS, 1, 1, 1};
    const cuuint32_t elem[5] = {1, 1, 1, 1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(base), dims, strides, box, elem,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : 10003;
}

}  // namespace

// Keys and values of heads head0 .. head0 + n_heads for the tokens that the requests' rows see.  cache [pool_tokens, C + R]
// and the maps [all heads * 128, C] are bfloat16; `expanded` [n_heads, tokens, 832] bfloat16; `max_tokens`: the largest of
// the requests' shares of it.  requests: device int32 [n_req, 4].
LLMX_EXPORT int llmx_latent_expand(const void* cache, long long pool_tokens, const void* w_uk, const void* w_uv, int all_heads,
                                   void* expanded, const int* requests, int n_req, int max_tokens, const int* row_request,
                                   const int* positions, const int* block_tables, int table_stride, int tokens, int head0,
                                   int n_heads, int C, int R, int page_size, int window, int* error_word, cudaStream_t stream) {
    if (n_req <= 0 || n_heads <= 0) return 0;
    if (C <= 0 || C % 64 || R < 0 || R > 64 || R % 8 || page_size <= 0 || page_size % 16 || n_req > 65535 || n_heads > 65535 ||
        pool_tokens <= 0 || tokens <= 0 || tokens % ROWS || max_tokens <= 0 || max_tokens % ROWS || head0 < 0 || head0 + n_heads > all_heads ||
        (((uintptr_t)cache | (uintptr_t)w_uk | (uintptr_t)w_uv | (uintptr_t)expanded) & 15))
        return LLMX_ERR_UNSUPPORTED;
    static const bool enough = registers_reach(latent_expand_kernel, EXPAND_THREADS, FEWER_REGISTERS + 2 * MORE_REGISTERS);
    if (!enough) return LLMX_ERR_UNSUPPORTED;
    CUtensorMap cache_map, uk_map, uv_map, expanded_map;
    if (int e = make_expanded_map(&expanded_map, expanded, (uint64_t)tokens, (uint64_t)n_heads)) return e;
    if (int e = llmx_make_map_bf16_2d(&cache_map, cache, (uint64_t)pool_tokens, (uint64_t)(C + R), 16, 64)) return e;
    if (int e = llmx_make_map_bf16_2d(&uk_map, w_uk, (uint64_t)all_heads * D, (uint64_t)C, D, 64)) return e;
    if (int e = llmx_make_map_bf16_2d(&uv_map, w_uv, (uint64_t)all_heads * D, (uint64_t)C, D, 64)) return e;
    LLMX_ALLOW_SMEM(latent_expand_kernel);
    launch_kernel(latent_expand_kernel, dim3(max_tokens / ROWS, n_heads, n_req), dim3(EXPAND_THREADS), (size_t)EXPAND_SMEM, stream, cache_map,
                  uk_map, uv_map, expanded_map, (const __nv_bfloat16*)cache, (__nv_bfloat16*)expanded, requests, row_request, positions, block_tables,
                  table_stride, tokens, head0, C, R, page_size, window, error_word);
    return launch_status();
}

// Attention of the tiles' rows over the expanded keys and values: q float [rows, q_stride], per head 128 unrotated then R
// rotated-part values; out [rows, heads, 128] bfloat16.  tiles: device int32 [n_tiles, 4].
LLMX_EXPORT int llmx_latent_prompt(const void* expanded, int tokens, const float* q, int q_stride, void* out, const int* tiles,
                                   int n_tiles, const float* freq, int rot_pairs, int rot_halves, float rot_mag, const int* positions,
                                   int heads, int head0, int n_heads, int R, int window, float scale, int* error_word,
                                   cudaStream_t stream) {
    if (n_tiles <= 0 || n_heads <= 0) return 0;
    if (R < 0 || R > 64 || R % 8 || 2 * rot_pairs > R || n_heads > 65535 || head0 < 0 || head0 + n_heads > heads || tokens <= 0 || q_stride % 2 ||
        (((uintptr_t)expanded | (uintptr_t)out) & 15) || ((uintptr_t)q & 7))
        return LLMX_ERR_UNSUPPORTED;
    CUtensorMap map;
    if (int e = make_expanded_map(&map, expanded, (uint64_t)tokens, (uint64_t)n_heads)) return e;
    LLMX_ALLOW_SMEM(latent_prompt_kernel);
    launch_kernel(latent_prompt_kernel, dim3(n_tiles, n_heads), dim3(PROMPT_THREADS), (size_t)PROMPT_SMEM, stream, map, q, q_stride,
                  (__nv_bfloat16*)out, tiles, freq, rot_pairs, rot_halves, rot_mag, positions, heads, head0, R, window,
                  scale * attn::LOG2E, error_word);
    return launch_status();
}
