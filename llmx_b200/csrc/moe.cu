// A mixture of experts whose routing is a table: token id -> the `top` experts that token uses (no router product), or
// row of the step -> experts, as a router (`llmx_moe_router`) wrote it on the device.
//
// A step's rows are sorted by expert on the device, so that nothing about the routing is read on the host and a step
// can be recorded and replayed.  A *pair* is (row, k): row r with the k-th expert of its token, numbered r * top + k.
//   llmx_moe_route       one block an expert walks the pairs in order and lists those that name it (so a list is in
//                        row order, whatever else the launch holds); for the products on the CUDA cores one more block cuts
//                        the lists into tiles of 32 pairs: (expert, first place in the list), compactly, with their number.
//   llmx_moe_product     gated: act[pair, f] = glu(h[row] . Wg_e[f], h[row] . Wu_e[f])       (gate and up rows stacked per expert;
//                        glu(g, u) = silu(g) u, or the clamped unit min(g, L) sigmoid(alpha min(g, L)) (clamp(u, -L, L) + 1));
//                        else y[pair, c] = act[pair] . Wd_e[c]                               (32-bit)
//   llmx_moe_gather      the pairs' rows, one expert's after the other's, for the next:
//   llmx_moe_product_tc  the same products on the tensor cores over sorted rows; the gated one leaves its rows sorted for the second
//   llmx_moe_combine     x[row]      += weight * sum_k y[row * top + k]                      (k in order: one order of sums)
// A pair may name an expert beyond those that have weights (an identity expert): it is in no list, the products leave its
// rows alone, and `llmx_moe_combine_weighted` takes the row's input in its place.
// Three forms of the products.  On the CUDA cores (32-bit weights and rows: the true 32-bit path; also bfloat16 shapes the tensor-core form
// does not take) a block has a tile of an expert's pairs and a tile of output columns, gathers its rows through the list and reads
// the expert's weights once a tile, explicit fmaf, k in increasing order; it checks its tiles' size against what the routing wrote
// (tiles[1]).  On the tensor cores (tcgen05.mma, bfloat16 in, 32-bit sums; K a multiple of 32) pairs of SMs walk parts of the lists.
// Steps of a few pairs (decoding) need no lists: their products are the experts' weights streamed once.
#include "tc_pair.cuh"
#include <math.h>
#include <type_traits>

namespace {
constexpr int TILE_ROWS = 32;     // pairs a tile holds

// The gated unit of an expert: silu(g) * u without a clamp, else the clamped one.
struct Glu {
    int clamped;
    float limit, alpha;
};
__device__ __forceinline__ float glu_f(const Glu& a, float g, float u) {
    if (!a.clamped) return quotient(g, 1.0f + expf(-g)) * u;
    g = fminf(g, a.limit);
    u = fminf(fmaxf(u, -a.limit), a.limit);
    return quotient(g, 1.0f + expf(-a.alpha * g)) * (u + 1.0f);
}

// A block's threads look up ROUTE_AHEAD pairs each before any is counted; the places follow the pairs' order: a ballot within a
// warp, a scan over the (turn, warp) counts of the chunk by the first warp.  4,096 pairs: 23.6 -> 6.1 us.
constexpr int ROUTE_THREADS = 1024, ROUTE_WARPS = ROUTE_THREADS / 32, ROUTE_AHEAD = 4;

__global__ void __launch_bounds__(ROUTE_THREADS)
route_kernel(const int* __restrict__ token_ids, const int* __restrict__ table, int top, int rows, int experts, int vocab,
             int* __restrict__ lists, int* __restrict__ counts) {
    pdl_trigger();
    pdl_wait();
    __shared__ int place[ROUTE_AHEAD * ROUTE_WARPS];     // counts, then the places where the turns' and warps' pairs begin
    __shared__ int total;
    const int e = blockIdx.x;
    const int pairs = rows * top;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int base = 0;
    for (int p0 = 0; p0 < pairs; p0 += ROUTE_THREADS * ROUTE_AHEAD) {
        int tok[ROUTE_AHEAD];
        bool mine[ROUTE_AHEAD];
#pragma unroll
        for (int i = 0; i < ROUTE_AHEAD; ++i) {
            const int p = p0 + i * ROUTE_THREADS + threadIdx.x;
            tok[i] = p >= pairs ? -1 : token_ids ? token_ids[p / top] : p / top;      // no ids: the table has a row for each row of the step
        }
#pragma unroll
        for (int i = 0; i < ROUTE_AHEAD; ++i) {
            const int p = p0 + i * ROUTE_THREADS + threadIdx.x;
            mine[i] = tok[i] >= 0 && tok[i] < vocab && table[(size_t)tok[i] * top + p % top] == e;
        }
        unsigned ballot[ROUTE_AHEAD];
#pragma unroll
        for (int i = 0; i < ROUTE_AHEAD; ++i) {
            ballot[i] = __ballot_sync(0xffffffffu, mine[i]);
            if (lane == 0) place[i * ROUTE_WARPS + warp] = __popc(ballot[i]);
        }
        __syncthreads();
        if (warp == 0) {
            int at = base;
#pragma unroll
            for (int i = 0; i < ROUTE_AHEAD; ++i) {
                const int n = place[i * ROUTE_WARPS + lane];
                int upto = n;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int below = __shfl_up_sync(0xffffffffu, upto, o);
                    if (lane >= o) upto += below;
                }
                place[i * ROUTE_WARPS + lane] = at + upto - n;
                at += __shfl_sync(0xffffffffu, upto, 31);
            }
            if (lane == 0) total = at;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ROUTE_AHEAD; ++i)
            if (mine[i])
                lists[(size_t)e * pairs + place[i * ROUTE_WARPS + warp] + __popc(ballot[i] & ((1u << lane) - 1u))] = p0 + i * ROUTE_THREADS + threadIdx.x;
        base = total;
        __syncthreads();                                 // the counts may be written again
    }
    if (threadIdx.x == 0) counts[e] = base;
}

// tiles: [0] their number, then (expert, first place) pairs from tiles[2] on.
__global__ void tiles_kernel(const int* __restrict__ counts, int experts, int* __restrict__ tiles, int tile_rows) {
    pdl_trigger();
    pdl_wait();
    if (threadIdx.x != 0) return;
    int n = 0;
    for (int e = 0; e < experts; ++e)
        for (int at = 0; at < counts[e]; at += tile_rows) {
            tiles[2 + 2 * n] = e;
            tiles[3 + 2 * n] = at;
            ++n;
        }
    tiles[0] = n;
    tiles[1] = tile_rows;
}

// ---- the product on the CUDA cores ---------------------------------------------------------------------------------
// A block: TILE_ROWS pairs x 64 output columns, K in steps of 16; a thread owns 2 pairs x 4 columns (and, GATED, the
// same of the up rows).  A's rows are gathered: pair p reads row p / a_div of `a`.
constexpr int CC_COLS = 64, CC_K = 16;

template <typename T, bool GATED, typename OutT>
__global__ void __launch_bounds__(256)
moe_cores_kernel(const T* __restrict__ a, int a_div, const T* __restrict__ w, const int* __restrict__ lists,
                 const int* __restrict__ counts, const int* __restrict__ tiles, int pairs, OutT* __restrict__ out, int N,
                 int K, Glu glu) {
    pdl_trigger();
    pdl_wait();
    if ((int)blockIdx.x >= tiles[0] || tiles[1] != TILE_ROWS) return;
    const int e = tiles[2 + 2 * blockIdx.x], at = tiles[3 + 2 * blockIdx.x];
    const int n_here = min(TILE_ROWS, counts[e] - at);
    const int* list = lists + (size_t)e * pairs + at;
    const int col0 = blockIdx.y * CC_COLS;
    __shared__ float As[CC_K][TILE_ROWS + 1];
    __shared__ float Ws[GATED ? 2 : 1][CC_K][CC_COLS + 1];
    __shared__ int src_pair[TILE_ROWS];
    if (threadIdx.x < TILE_ROWS) src_pair[threadIdx.x] = threadIdx.x < n_here ? list[threadIdx.x] : -1;
    __syncthreads();
    const int tr = threadIdx.x / 16, tc = threadIdx.x % 16;        // pairs 2 tr, 2 tr + 1; columns tc + 16 j
    float acc[2][4] = {}, acc2[2][4] = {};
    const T* wbase = w + (size_t)e * (GATED ? 2 : 1) * N * K;
    for (int k0 = 0; k0 < K; k0 += CC_K) {
        for (int i = threadIdx.x; i < TILE_ROWS * CC_K; i += 256) {
            const int r = i / CC_K, kk = i % CC_K;
            const int p = src_pair[r];
            As[kk][r] = (p >= 0 && k0 + kk < K) ? to_float(a[(size_t)(p / a_div) * K + k0 + kk]) : 0.0f;
        }
        for (int i = threadIdx.x; i < CC_COLS * CC_K; i += 256) {
            const int c = i / CC_K, kk = i % CC_K;
            const bool ok = col0 + c < N && k0 + kk < K;
            Ws[0][kk][c] = ok ? to_float(wbase[(size_t)(col0 + c) * K + k0 + kk]) : 0.0f;
            if (GATED) Ws[1][kk][c] = ok ? to_float(wbase[(size_t)(N + col0 + c) * K + k0 + kk]) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < CC_K; ++kk) {
            const float a0 = As[kk][2 * tr], a1 = As[kk][2 * tr + 1];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float b = Ws[0][kk][tc + 16 * j];
                acc[0][j] = fmaf(a0, b, acc[0][j]);
                acc[1][j] = fmaf(a1, b, acc[1][j]);
                if (GATED) {
                    const float b2 = Ws[1][kk][tc + 16 * j];
                    acc2[0][j] = fmaf(a0, b2, acc2[0][j]);
                    acc2[1][j] = fmaf(a1, b2, acc2[1][j]);
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int p = src_pair[2 * tr + i];
        if (p < 0) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int c = col0 + tc + 16 * j;
            if (c >= N) continue;
            float v = acc[i][j];
            if (GATED) v = glu_f(glu, v, acc2[i][j]);
            out[(size_t)p * N + c] = from_float<OutT>(v);
        }
    }
}

// ---- the product on the tensor cores -------------------------------------------------------------------------------
// The pairs' rows lie sorted by expert (`gather_kernel`, or as the gated product wrote them), so that both operands come by TMA.
// Pairs of SMs (a cluster of two blocks, tcgen05 `cta_group::2`) walk units: 256 weight rows x up to 256 of an expert's pairs; a
// block holds 128 of the weight rows and half of the pairs' rows, and its sums (128 x 256) twice in tensor memory, so that a unit is
// written out beside the next one's products.
//   warp 0 (both blocks)   TMA: K in steps of 64 through six stages; gated, the block's weight rows are runs of 16 gate rows and the
//                          16 up rows of the same outputs, so that a warp's 32 sums of a pair are 16 whole outputs; of the pairs' rows
//                          as many boxes of 32 as the unit's half has
//   warp 1 (first block)   the products, and a commit that frees a stage in both blocks
//   warps 2-9 (both)       sums to the output, of two warps with the same lanes each every other run of 32 pairs; gated, lanes i and
//                          i + 16 swap halves of their pairs, each makes 16 units of both
// An expert's list is cut into ceil(pairs / 256) equal parts: its weights are read that often, and none is left with a few
// pairs.  Units of one expert follow one another, its weight tiles fastest: what they share meets in the L2 cache.
// Bound, at a few dozen to a few hundred pairs an expert, by the experts' weights from memory and by the write-out: with one warp for a
// quarter of the lanes the tensor cores were busy a third of the time.  Measured against one SM a tile with rows gathered by cp.async, 16
// experts, two a token: 2,048 tokens, 2,048 -> 1,536 gated 98 us, one warp 80, two 71; back 51, 34 and 34; 1,201 tokens, 4,096 -> 3,072 gated
// 188 us -> 167 (one warp), back 87 -> 80.
constexpr int TC_LIST_TILE = 128;                                            // pairs a tile holds where tiles are asked for beside this form, which reads none
constexpr int TC_ROWS = 256, TC_K = 64, TC_M = 128, TC_BOX = 32;
constexpr int TC_W_BYTES = TC_M * TC_K * 2, TC_R_BYTES = TC_ROWS / 2 * TC_K * 2, TC_STAGE = TC_W_BYTES + TC_R_BYTES, TC_STAGES = 6;
constexpr int TC_EPI_WARPS = 8, TC_THREADS = 64 + TC_EPI_WARPS * 32;
// Four numbers of each expert that has pairs lie in shared memory, beside fewer stages if need be; of more than TC_MAX_LISTED, in memory.
constexpr int TC_MAX_LISTED = 8192, TC_BARS = 512;                           // barriers, what the block's scan carries from warp to warp
constexpr int tc_smem(int stages, int listed) { return stages * TC_STAGE + 1024 + TC_BARS + 4 * listed * (int)sizeof(int); }
constexpr int tc_stages(int listed) {
    int stages = TC_STAGES;
    while (tc_smem(stages, listed) > 227 * 1024) --stages;
    return stages;
}
static_assert(tc_stages(TC_MAX_LISTED) >= 3, "a stage in use and two on their way");
enum : int { ERR_MOE_PRODUCER = 441, ERR_MOE_MMA = 442, ERR_MOE_EPILOGUE = 443 };

// rows[place] = a[pair / a_div] for the pair at that place of the sorted lists; a block a place.  Bound by three reads that follow one
// another, from memory (counts, list, row).  Few experts: the first warp adds up their counts, 32 at a time.  MANY: the block's threads
// add up equal runs of experts side by side and the one whose run holds the place walks it (32 at a time the chain of reads is as long
// as there are experts: 80 pairs of 1,024 of them 19 us and of 8,192 105 us, the wait for the routing included, against 5 and 57).
constexpr int GATHER_THREADS = 128;                  // many blocks an SM: a block waits for one read after the other
template <bool MANY>
__global__ void __launch_bounds__(GATHER_THREADS)
gather_kernel(const uint4* __restrict__ a, int a_div, const int* __restrict__ lists, const int* __restrict__ counts, int experts, int pairs,
              uint4* __restrict__ rows, int per_row) {
    pdl_trigger();
    pdl_wait();
    const int place = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __shared__ int found, carry[GATHER_THREADS / 32];
    if (MANY) {
        const int run = (experts + GATHER_THREADS - 1) / GATHER_THREADS, e0 = threadIdx.x * run, e1 = min(e0 + run, experts);
        int mine = 0;
        for (int e = e0; e < e1; ++e) mine += counts[e];
        int upto = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int below = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += below;
        }
        if (lane == 31) carry[warp] = upto;
        if (threadIdx.x == 0) found = -1;
        __syncthreads();
        int at = place - (upto - mine);
        for (int w = 0; w < warp; ++w) at -= carry[w];
        if (at >= 0 && at < mine) {
            int e = e0;
            while (at >= counts[e]) at -= counts[e++];
            found = lists[(size_t)e * pairs + at];
        }
    } else if (warp == 0) {                          // the expert whose list holds the place
        int base = 0, pair = -1;
        for (int e0 = 0; e0 < experts && pair < 0; e0 += 32) {
            const int mine = e0 + lane < experts ? counts[e0 + lane] : 0;
            int upto = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int below = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += below;
            }
            const unsigned hit = __ballot_sync(0xffffffffu, place < base + upto);
            if (hit) {
                const int first = __ffs(hit) - 1;
                const int at = place - base - __shfl_sync(0xffffffffu, upto - mine, first);
                pair = lists[(size_t)(e0 + first) * pairs + at];
            }
            base += __shfl_sync(0xffffffffu, upto, 31);
        }
        if (lane == 0) found = pair;
    }
    __syncthreads();
    if (found < 0) return;                           // past the lists: pairs of experts without weights
    const uint4* src = a + (size_t)(found / a_div) * per_row;
    for (int i = threadIdx.x; i < per_row; i += GATHER_THREADS) rows[(size_t)place * per_row + i] = src[i];
}

// What the block's warps read of the experts, made by the block at its start: numbers [4][room] = how many pairs; rows before its own;
// parts of lists up to and with its own; and, MANY, which expert (only those with pairs are listed: when every role of every block walked
// the others, 8,192 experts, 80 pairs were 600 us of a product).  Few experts keep a place each and one warp's scan, 32 at a time: less
// code, which comes from memory too, and for 16 experts 1 to 2 us a launch less than the list.
constexpr int MANY_EXPERTS = 128;
__device__ __forceinline__ void number_experts(const int* __restrict__ counts, int experts, int* numbers, int lane) {
    int rows_before = 0, tiles_before = 0;
    for (int e0 = 0; e0 < experts; e0 += 32) {
        const int e = e0 + lane, c = e < experts ? counts[e] : 0;
        int rows_upto = c, tiles_upto = (c + TC_ROWS - 1) / TC_ROWS;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int r = __shfl_up_sync(0xffffffffu, rows_upto, o), t = __shfl_up_sync(0xffffffffu, tiles_upto, o);
            if (lane >= o) rows_upto += r, tiles_upto += t;
        }
        if (e < experts) numbers[e] = c, numbers[experts + e] = rows_before + rows_upto - c, numbers[2 * experts + e] = tiles_before + tiles_upto;
        rows_before += __shfl_sync(0xffffffffu, rows_upto, 31);
        tiles_before += __shfl_sync(0xffffffffu, tiles_upto, 31);
    }
}
// All threads of the block, each an equal run of the experts, so that counts are read side by side; `carry`: 3 ints a warp.  Returns how
// many are listed, `room` at most (counts that add up to more than the pairs are nobody's routing).
__device__ __forceinline__ int list_experts(const int* __restrict__ counts, int experts, int* numbers, int room, int* carry) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = (int)blockDim.x >> 5;
    const int run = (experts + (int)blockDim.x - 1) / (int)blockDim.x, e0 = (int)threadIdx.x * run, e1 = min(e0 + run, experts);
    int mine[3] = {0, 0, 0}, upto[3];
    for (int e = e0; e < e1; ++e) {
        const int c = counts[e];
        mine[0] += c > 0, mine[1] += c, mine[2] += (c + TC_ROWS - 1) / TC_ROWS;
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        upto[i] = mine[i];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int below = __shfl_up_sync(0xffffffffu, upto[i], o);
            if (lane >= o) upto[i] += below;
        }
        if (lane == 31) carry[3 * warp + i] = upto[i];
    }
    __syncthreads();
    int total = 0;
    for (int w = 0; w < warps; ++w) {
        if (w < warp) upto[0] += carry[3 * w], upto[1] += carry[3 * w + 1], upto[2] += carry[3 * w + 2];
        total += carry[3 * w];
    }
    int at = upto[0] - mine[0], row = upto[1] - mine[1], tile = upto[2] - mine[2];
    for (int e = e0; e < e1; ++e) {
        const int c = counts[e];
        if (c <= 0 || at >= room) continue;
        tile += (c + TC_ROWS - 1) / TC_ROWS;
        numbers[at] = c, numbers[room + at] = row, numbers[2 * room + at] = tile, numbers[3 * room + at] = e;
        row += c, ++at;
    }
    return min(total, room);
}

// More experts with pairs than shared memory has room for: their numbers, then how many they are, in memory; one block.
constexpr int LIST_THREADS = 1024;
__global__ void __launch_bounds__(LIST_THREADS) list_experts_kernel(const int* __restrict__ counts, int experts, int* __restrict__ numbers, int room) {
    pdl_trigger();
    pdl_wait();
    __shared__ int carry[3 * LIST_THREADS / 32];
    const int listed = list_experts(counts, experts, numbers, room, carry);
    if (threadIdx.x == 0) numbers[4 * (size_t)room] = listed;
}

// A pair of blocks' units.
template <bool MANY>
struct Units {
    const int* numbers;      // as above
    int room, listed, w_tiles, cur, step, place;
    // Unit `cur`: expert e, pairs at .. at + n - 1 of its list, rows from `row` on, weight tile w.
    __device__ __forceinline__ bool next(int& e, int& at, int& n, int& row, int& w) {
        const int* tile = numbers + 2 * room;
        const int t = cur / w_tiles;
        if (MANY)
            while (place + 8 <= listed && tile[place + 7] <= t) place += 8;
        while (place < listed && tile[place] <= t) ++place;
        if (place >= listed) return false;
        e = MANY ? numbers[3 * room + place] : place;
        w = cur % w_tiles;
        const int count = numbers[place], parts = (count + TC_ROWS - 1) / TC_ROWS;
        // Equal parts, multiples of 16 of at most 256 pairs: the last one is never empty, (parts - 1) * 256 being below the count.
        const int size = ((count + parts - 1) / parts + 15) & ~15;
        at = (t - (tile[place] - parts)) * size;
        n = min(size, count - at);
        row = numbers[room + place] + at;
        cur += step;
        return true;
    }
};

template <bool GATED, typename OutT, bool MANY>
__global__ void __launch_bounds__(TC_THREADS, 1)
moe_tc_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap r_map, const int* __restrict__ lists,
              const int* __restrict__ counts, int experts, int pairs, OutT* __restrict__ out, int out_sorted, int N, int K, Glu glu,
              int stages, int room, const int* __restrict__ made, int* error_word) {
    extern __shared__ uint8_t tc_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)tc_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full = (uint64_t*)(smem + stages * TC_STAGE);          // used in the first block
    uint64_t* empty = full + stages;                                // one in each block
    uint64_t* acc_full = empty + stages;                            // [2], one in each block
    uint64_t* acc_empty = acc_full + 2;                             // [2], used in the first block
    uint32_t* tmem_slot = (uint32_t*)(acc_empty + 2);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    int* carry = (int*)(smem + stages * TC_STAGE + 256);
    int* numbers = (int*)(smem + stages * TC_STAGE + TC_BARS);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const bool leader = rank == 0;
    if (threadIdx.x == 0) {
        for (int i = 0; i < stages; ++i) {
            tc::mbar_init(&full[i], 1);
            tc::mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            tc::mbar_init(&acc_full[i], 1);
            tc::mbar_init(&acc_empty[i], 2 * TC_EPI_WARPS);
        }
        *abort_flag = 0;
        tc::fence_barrier_init();
        tc::tma_prefetch_desc(&w_map);
        tc::tma_prefetch_desc(&r_map);
    }
    if (warp == 1) {
        tmem_alloc_pair(tmem_slot, 2 * TC_ROWS);
        tmem_relinquish_pair();
    }
    tc::tc_fence_before();
    __syncthreads();
    cluster_sync();           // both blocks' barriers exist before either signals the other
    tc::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_trigger();            // only now that this block holds its tensor memory (gemm_tc_pair.cu)
    pdl_wait();
    int listed = experts;
    if (MANY) listed = made ? made[4 * (size_t)room] : list_experts(counts, experts, numbers, room, carry);
    else if (warp == 2) number_experts(counts, experts, numbers, lane);
    __syncthreads();
    const int w_cols = GATED ? TC_M : 2 * TC_M;      // output columns of a unit
    const int steps = (K + TC_K - 1) / TC_K;
    Units<MANY> units{MANY && made ? made : numbers, MANY ? room : experts, listed, (N + w_cols - 1) / w_cols, (int)blockIdx.x >> 1, (int)gridDim.x >> 1, 0};
    int e, at, n, row, w;

    if (warp == 0) {
        if (tc::elect_one()) {
            int st = 0;
            uint32_t phase = 1;
            bool ok = true;
            while (ok && units.next(e, at, n, row, w)) {
                const int half = ((n + 15) & ~15) / 2, boxes = (half + TC_BOX - 1) / TC_BOX;
                const int first = row + (int)rank * half;
                const int col = w * w_cols + (int)rank * (GATED ? TC_M / 2 : TC_M);
                for (int s = 0; s < steps; ++s) {
                    ok = tc::mbar_wait(&empty[st], phase, abort_flag, error_word, ERR_MOE_PRODUCER);
                    if (!ok) break;
                    if (leader) tc::mbar_expect_tx(&full[st], 2 * (TC_W_BYTES + boxes * TC_BOX * TC_K * 2));
                    const uint32_t bar = peer_addr(&full[st], 0);
                    uint8_t* base = smem + st * TC_STAGE;
                    if (GATED) {
#pragma unroll
                        for (int i = 0; i < TC_M / 32; ++i) tma_load_3d_pair(base + i * 32 * TC_K * 2, &w_map, s * TC_K, col + 16 * i, 2 * e, bar);
                    } else {
                        tma_load_3d_pair(base, &w_map, s * TC_K, col, e, bar);
                    }
                    for (int i = 0; i < boxes; ++i)
                        tma_load_2d_pair(base + TC_W_BYTES + i * TC_BOX * TC_K * 2, &r_map, s * TC_K, first + i * TC_BOX, bar);
                    if (++st == stages) { st = 0; phase ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        if (leader && tc::elect_one()) {
            int st = 0;
            uint32_t phase = 0, acc = 0, acc_phase = 1;
            bool ok = true;
            while (ok && units.next(e, at, n, row, w)) {
                ok = tc::mbar_wait(&acc_empty[acc], acc_phase, abort_flag, error_word, ERR_MOE_MMA);
                if (!ok) break;
                tc::tc_fence_after();
                const uint32_t idesc = tc::instr_desc_bf16(2 * TC_M, (n + 15) & ~15), tmem_d = tmem_base + acc * TC_ROWS;
                for (int s = 0; s < steps; ++s) {
                    ok = tc::mbar_wait(&full[st], phase, abort_flag, error_word, ERR_MOE_MMA);
                    if (!ok) break;
                    tc::tc_fence_after();
                    const uint32_t addr = tc::smem_u32(smem + st * TC_STAGE);
                    const uint64_t desc_w = tc::smem_desc_k_sw128(addr), desc_r = tc::smem_desc_k_sw128(addr + TC_W_BYTES);
#pragma unroll
                    for (int k = 0; k < TC_K / 16; ++k)
                        mma_bf16_pair(tmem_d, desc_w + 2 * k, desc_r + 2 * k, idesc, (s > 0 || k > 0) ? 1u : 0u);
                    mma_commit_pair(&empty[st], 3);
                    if (++st == stages) { st = 0; phase ^= 1; }
                }
                if (!ok) break;
                mma_commit_pair(&acc_full[acc], 3);
                if (++acc == 2) { acc = 0; acc_phase ^= 1; }
            }
        }
    } else {
        const int quarter = warp & 3, share = (warp - 2) >> 2;        // the tensor-memory lanes that this warp may touch, and which pairs it has
        uint32_t acc = 0, acc_phase = 0;
        bool ok = true;
        while (ok && units.next(e, at, n, row, w)) {
            const int* list = lists + (size_t)e * pairs + at;
            const int c = w * w_cols + (GATED ? (int)rank * (TC_M / 2) + quarter * 16 + (lane & 15) : (int)rank * TC_M + quarter * 32 + lane);
            int dest[TC_ROWS / 64];                  // the rows that the lane's pairs go to: read while the products run
#pragma unroll
            for (int i = 0; i < TC_ROWS / 64; ++i) {
                const int p = 32 * share + 64 * i + lane;
                dest[i] = out_sorted ? row + p : p < n ? list[p] : 0;
            }
            ok = tc::mbar_wait_warp(&acc_full[acc], acc_phase, abort_flag, error_word, ERR_MOE_EPILOGUE);
            if (!ok) break;
            tc::tc_fence_after();
            const uint32_t taddr = tmem_base + acc * TC_ROWS + ((uint32_t)(quarter * 32) << 16);
#pragma unroll
            for (int i = 0; i < TC_ROWS / 64; ++i) {
                const int p0 = 32 * share + 64 * i, to = dest[i];
                if (p0 >= n) break;
                uint32_t r[32];
                tc::tmem_ld_32x32(taddr + p0, r);
                tc::tmem_wait_ld();
                if constexpr (GATED) {
                    const bool up = lane >= 16;      // this lane's sums are up rows; it makes the second half of the pairs
                    OutT x[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const float got = __shfl_xor_sync(0xffffffffu, __uint_as_float(up ? r[j] : r[16 + j]), 16);
                        const float own = __uint_as_float(up ? r[16 + j] : r[j]);
                        x[j] = from_float<OutT>(glu_f(glu, up ? got : own, up ? own : got));
                    }
                    const int half = up ? 16 : 0;
                    if (out_sorted && p0 + 32 <= n) {            // no condition a value: neighbouring rows
                        OutT* to_row = out + (size_t)(row + p0 + half) * N + c;
                        if (c < N)
#pragma unroll
                            for (int j = 0; j < 16; ++j) to_row[(size_t)j * N] = x[j];
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            const size_t dst = (size_t)__shfl_sync(0xffffffffu, to, half + j);
                            if (p0 + half + j < n && c < N) out[dst * N + c] = x[j];
                        }
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const size_t dst = (size_t)__shfl_sync(0xffffffffu, to, j);
                        if (p0 + j < n && c < N) out[dst * N + c] = from_float<OutT>(__uint_as_float(r[j]));
                    }
                }
            }
            tc::tc_fence_before();
            __syncwarp();
            if (lane == 0) arrive_at(peer_addr(&acc_empty[acc], 0));
            if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        }
    }
    tc::tc_fence_before();
    __syncthreads();
    cluster_sync();           // the partner no longer reads this block's shared memory or signals its barriers
    if (warp == 1) {
        tc::tc_fence_after();
        tmem_dealloc_pair(tmem_base, 2 * TC_ROWS);
    }
}

// A tensor map of three dimensions of bfloat16 (x contiguous), 128-byte swizzle.
static int make_map_3d(CUtensorMap* map, const void* base, uint64_t x, uint64_t y, uint64_t z, uint32_t bx, uint32_t by, uint32_t bz) {
    llmx_encode_tiled_fn enc = llmx_encode_tiled();
    if (!enc) return 10003;
    const cuuint64_t dims[3] = {x, y, z}, strides[2] = {x * 2, x * y * 2};
    const cuuint32_t box[3] = {bx, by, bz}, elem[3] = {1, 1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : 10003;
}

// ---- steps of a few pairs -------------------------------------------------------------------------------------------
// With a handful of pairs (decoding) nearly every pair has an expert of its own and the products are the experts'
// weights streamed once: a block takes one pair and 16 output columns, its row lies in shared memory, and a warp makes
// two columns, each lane reading 16-byte pieces of the weight rows (several in flight) and the lanes' sums meeting by
// shuffles in a fixed order.  The pair's expert is read from the table; no lists are needed.
constexpr int GV_COLS = 16;

__device__ __forceinline__ void fma8(float& acc, const uint4& w, const uint4& x) {
    const __nv_bfloat162* wp = reinterpret_cast<const __nv_bfloat162*>(&w);
    const __nv_bfloat162* xp = reinterpret_cast<const __nv_bfloat162*>(&x);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 a = __bfloat1622float2(wp[i]), b = __bfloat1622float2(xp[i]);
        acc = fmaf(a.x, b.x, acc);
        acc = fmaf(a.y, b.y, acc);
    }
}

template <bool GATED, typename OutT>
__global__ void __launch_bounds__(256)
moe_few_kernel(const __nv_bfloat16* __restrict__ a, int a_div, const __nv_bfloat16* __restrict__ w,
               const int* __restrict__ token_ids, const int* __restrict__ table, int top, int vocab, int experts,
               OutT* __restrict__ out, int N, int K, Glu glu) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ __align__(16) unsigned char few_smem[];
    uint4* row = reinterpret_cast<uint4*>(few_smem);                 // the pair's row, K bfloat16
    const int p = blockIdx.x;
    const int tok = token_ids ? token_ids[p / top] : p / top;
    const int e = (tok >= 0 && tok < vocab) ? table[(size_t)tok * top + p % top] : -1;
    if (e < 0 || e >= experts) return;
    const uint4* src = reinterpret_cast<const uint4*>(a + (size_t)(p / a_div) * K);
    for (int i = threadIdx.x; i < K / 8; i += 256) row[i] = src[i];
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const __nv_bfloat16* wbase = w + (size_t)e * (GATED ? 2 : 1) * N * K;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int c = blockIdx.y * GV_COLS + 2 * warp + j;
        if (c >= N) continue;
        const uint4* w0 = reinterpret_cast<const uint4*>(wbase + (size_t)c * K);
        const uint4* w1 = reinterpret_cast<const uint4*>(wbase + (size_t)(N + c) * K);
        float s0 = 0.0f, s1 = 0.0f;
#pragma unroll 4
        for (int i = lane; i < K / 8; i += 32) {
            const uint4 x = row[i];
            fma8(s0, w0[i], x);
            if (GATED) fma8(s1, w1[i], x);
        }
        s0 = warp_sum(s0);
        if (GATED) s1 = warp_sum(s1);
        if (lane == 0) out[(size_t)p * N + c] = from_float<OutT>(GATED ? glu_f(glu, s0, s1) : s0);
    }
}

// The same for steps of up to FEW_PAIRS pairs whose weight rows fit shared memory several times (K up to FEW_K): the experts
// that the pairs name, each once, as a stream.  A block an SM takes an equal run of the items (expert, two weight rows: the
// gate and up rows of a column, or two columns); one thread brings them by bulk copies of whole rows into a ring of up to
// 192 KB, so that the memory always has requests, and up to sixteen warps take the ring's places in turn: dot products with
// the rows of all pairs that name the expert (which the L1 cache holds), the lanes' sums met by shuffles in a fixed order.
// The warps' number divides the ring's places, so that a place is always the same warp's: a waiter tells uses of a place
// apart by parity only, and a warp that came to a place before its last use had landed would take it for the next.
// Eight pairs that name six experts, gate and up of K 4,096 and N 3,072: 70 -> 57 us, down 38.7 -> 32; two pairs 38.8 -> 22
// and 15.4 -> 12.6 us.  Bound by the dot products more than by the memory where an expert's rows meet several pairs.  Eight is the most it
// takes; beyond, stream / kernel above, gate and up, inputs out of the cache: K 4,096 nine pairs on nine experts 93 / 96 us, sixteen on
// twelve 123 / 133, on two 78 / 123; K 2,048 sixteen on sixteen 53 / 51, on two 29 / 39; down products equal or up to 40 % faster.
constexpr int FEW_PAIRS = 8, FEW_WARPS = 16, FEW_THREADS = 32 * FEW_WARPS + 32, FEW_PLACES = 32, FEW_K = 12288, FEW_RING = 192 * 1024;
enum : int { ERR_FEW_PRODUCER = 451, ERR_FEW_CONSUMER = 452 };

template <bool GATED, typename OutT>
__global__ void __launch_bounds__(FEW_THREADS, 1)
moe_few_stream_kernel(const __nv_bfloat16* __restrict__ a, int a_div, const __nv_bfloat16* __restrict__ w,
                      const int* __restrict__ token_ids, const int* __restrict__ table, int top, int vocab, int experts, int pairs,
                      OutT* __restrict__ out, int N, int K, Glu glu, int places, bool early, int* error_word) {
    const int workers = (int)blockDim.x / 32 - 1;
    extern __shared__ __align__(128) unsigned char ring[];
    __shared__ uint64_t full[FEW_PLACES], empty[FEW_PLACES];
    __shared__ int abort_word;
    // The experts that the pairs name, in the order of the first pair of each, and which pairs name each.
    __shared__ int expert_of[FEW_PAIRS], named;
    __shared__ unsigned pairs_of[FEW_PAIRS];
    volatile int* abort_flag = &abort_word;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < places; ++i) {
            tc::mbar_init(&full[i], 1);
            tc::mbar_init(&empty[i], 1);
        }
        abort_word = 0;
        tc::fence_barrier_init();
    }
    pdl_trigger();
    // `early`: no kernel that may still run writes the ids or the table (the caller says so: a step's tokens that a copy brought, a
    // table that came with the weights).  The stream of weights then starts while the kernel before still runs.
    if (!early) pdl_wait();
    if (warp == 0) {
        int mine = -1;
        if (lane < pairs) {
            const int tok = token_ids ? token_ids[lane / top] : lane / top;
            const int e = (tok >= 0 && tok < vocab) ? table[(size_t)tok * top + lane % top] : -1;
            if (e >= 0 && e < experts) mine = e;
        }
        const unsigned who = __match_any_sync(0xffffffffu, mine), before = (1u << lane) - 1;
        const bool first = mine >= 0 && !(who & before);
        const unsigned firsts = __ballot_sync(0xffffffffu, first);
        if (first) {
            expert_of[__popc(firsts & before)] = mine;
            pairs_of[__popc(firsts & before)] = who;
        }
        if (lane == 0) named = __popc(firsts);
    }
    __syncthreads();
    const int per_expert = GATED ? N : (N + 1) / 2;
    const int items = named * per_expert;
    const int per = (items + gridDim.x - 1) / gridDim.x;
    const int begin = blockIdx.x * per, count = min(items, begin + per) - begin;
    const size_t row_bytes = (size_t)K * 2;

    if (warp == workers) {
        if (tc::elect_one()) {
            int st = 0;
            uint32_t phase = 1;
            for (int n = 0; n < count; ++n) {
                if (!tc::mbar_wait(&empty[st], phase, abort_flag, error_word, ERR_FEW_PRODUCER)) break;
                const int it = begin + n, e = expert_of[it / per_expert];
                const int c = it % per_expert * (GATED ? 1 : 2);
                const __nv_bfloat16* w0 = w + ((size_t)e * (GATED ? 2 : 1) * N + c) * K;
                const __nv_bfloat16* w1 = GATED ? w0 + (size_t)N * K : c + 1 < N ? w0 + K : w0;
                unsigned char* dst = ring + (size_t)st * 2 * row_bytes;
                tc::mbar_expect_tx(&full[st], (uint32_t)(2 * row_bytes));
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                 ::"r"(tc::smem_u32(dst + i * row_bytes)), "l"(i ? w1 : w0), "r"((uint32_t)row_bytes), "r"(tc::smem_u32(&full[st])) : "memory");
                if (++st == places) { st = 0; phase ^= 1; }
            }
        }
        return;
    }
    if (early) pdl_wait();       // the rows, and the output's earlier readers
    for (int n = warp; n < count; n += workers) {
        const int st = n % places;
        if (!tc::mbar_wait_warp(&full[st], (n / places) & 1u, abort_flag, error_word, ERR_FEW_CONSUMER)) break;
        const uint4* w0 = reinterpret_cast<const uint4*>(ring + (size_t)st * 2 * row_bytes);
        const uint4* w1 = reinterpret_cast<const uint4*>(ring + (size_t)st * 2 * row_bytes + row_bytes);
        const int it = begin + n;
        const int c = it % per_expert * (GATED ? 1 : 2);
        unsigned left = pairs_of[it / per_expert];
        auto rows = [&](auto number) {                   // the next pairs of the expert
            constexpr int R = decltype(number)::value;
            int p[R];
            const uint4* x[R];
            float s0[R], s1[R];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                p[r] = __ffs(left) - 1;
                left &= left - 1;
                x[r] = reinterpret_cast<const uint4*>(a + (size_t)(p[r] / a_div) * K);
                s0[r] = s1[r] = 0.0f;
            }
#pragma unroll 4
            for (int i = lane; i < K / 8; i += 32) {
                const uint4 a0 = w0[i], a1 = w1[i];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const uint4 xv = x[r][i];
                    fma8(s0[r], a0, xv);
                    fma8(s1[r], a1, xv);
                }
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
                s0[r] = warp_sum(s0[r]);
                s1[r] = warp_sum(s1[r]);
                if (lane == 0) {
                    OutT* row = out + (size_t)p[r] * N;
                    row[c] = from_float<OutT>(GATED ? glu_f(glu, s0[r], s1[r]) : s0[r]);
                    if (!GATED && c + 1 < N) row[c + 1] = from_float<OutT>(s1[r]);
                }
            }
        };
        while (left) {
            const int k = __popc(left);
            if (k >= 4) rows(std::integral_constant<int, 4>{});
            else if (k >= 2) rows(std::integral_constant<int, 2>{});
            else rows(std::integral_constant<int, 1>{});
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&empty[st]);
    }
}

// Rows of whole groups of four values: a block a row and 1,024 of its values.  2,048 rows of 2,048, top 2: 25.6 -> 8.3 us.
__global__ void __launch_bounds__(256)
combine_vec_kernel(const float4* __restrict__ y, float4* __restrict__ x, int top, int n4, float weight) {
    pdl_trigger();
    pdl_wait();
    const int c = blockIdx.y * 256 + threadIdx.x;
    if (c >= n4) return;
    const size_t row = blockIdx.x;
    const float4* from = y + row * top * n4 + c;
    float4* to = x + row * n4 + c;
    float4 t = *to, s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
    for (int k = 0; k < top; ++k) {
        const float4 v = from[(size_t)k * n4];
        s = make_float4(s.x + v.x, s.y + v.y, s.z + v.z, s.w + v.w);
    }
    *to = make_float4(fmaf(weight, s.x, t.x), fmaf(weight, s.y, t.y), fmaf(weight, s.z, t.z), fmaf(weight, s.w, t.w));
}

__global__ void combine_kernel(const float* __restrict__ y, float* __restrict__ x, int top, int width, float weight,
                               long long n) {
    pdl_trigger();
    pdl_wait();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const long long row = i / width;
    const int c = (int)(i % width);
    float s = 0.0f;
    for (int k = 0; k < top; ++k) s += y[((size_t)row * top + k) * width + c];
    x[i] = fmaf(weight, s, x[i]);
}

// A router: logits z = h W^T + b in 32-bit (h may be bfloat16; the weights are 32-bit) and from them a choice of `top`
// outputs (the lower index first among equals) and their weights, in one of two ways:
//   over the chosen   the largest logits; weights: the softmax over the chosen logits alone
//   over all          s = softmax over all outputs; the largest s + correction among the outputs that may be chosen; weights:
//                     s / (sum of the chosen s + 1e-20) * scale.  With `group_keep` < `group_count` the outputs form equal
//                     groups of neighbours and only members of the groups with the largest best s + correction may be chosen
// `extra` more rows of W after the outputs' give one number a row each through a sigmoid (a gate on a part that runs beside
// the experts).  A block takes R rows of the step (1 when the rows are few, so that they spread over the SMs; 8 when they
// are many, so that a weight row is read once for 8 rows); a row's logits do not depend on what else the step holds.
struct RouterChoice {
    int over_all, group_count, group_keep;
    const float* correction;
    float scale;
};

// The best of v[0 .. n) over a warp: (value, index), the lower index among equals; index -1 when none exceeds minus infinity.
__device__ __forceinline__ void warp_best(const float* v, int n, int lane, float& bv, int& bi) {
    bv = -INFINITY;
    bi = -1;
    for (int e = lane; e < n; e += 32)
        if (v[e] > bv) bv = v[e], bi = e;                    // no number is never larger
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > bv || (ov == bv && oi >= 0 && (bi < 0 || oi < bi))) bv = ov, bi = oi;
    }
}
__device__ __forceinline__ void load4(const float* p, float (&v)[4]) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
}
__device__ __forceinline__ void load4(const __nv_bfloat16* p, float (&v)[4]) {
    const uint2 t = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&t.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&t.y));
    v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
}

template <typename T, int R, int VEC>
__global__ void __launch_bounds__(256)
router_kernel(const T* __restrict__ h, const float* __restrict__ w, const float* __restrict__ bias, int rows, int K, int experts,
              int top, int extra, RouterChoice rule, int* __restrict__ choice, float* __restrict__ weight, float* __restrict__ gate) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ float router_z[];                    // [R][experts + extra], then the warps' parts [8][experts + extra][R]
    const int row0 = blockIdx.x * R, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int outs = experts + extra;
    float* part = router_z + R * outs;
    // The inner width is cut into runs of VEC values, run p going to thread p mod 256: a warp holds every eighth group of
    // 32 runs, for all logits, so its loads of one turn (a run of each row, a run of each of four weight rows) do not wait
    // for one another.  Parts are summed lane tree first, then warps in order: one order whatever the step holds.
    constexpr int EC = R == 1 ? 8 : 4;                       // few rows: more weight rows a turn, so that more loads are in flight
    for (int e0 = 0; e0 < outs; e0 += EC) {
        float s[EC][R];
#pragma unroll
        for (int j = 0; j < EC; ++j)
#pragma unroll
            for (int r = 0; r < R; ++r) s[j][r] = 0.0f;
#pragma unroll(R == 1 ? 2 : 1)
        for (int k = VEC * (int)threadIdx.x; k < K; k += VEC * 256) {
            float xv[R][VEC];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (row0 + r < rows) {
                    if constexpr (VEC == 4) load4(h + (size_t)(row0 + r) * K + k, xv[r]);
                    else xv[r][0] = to_float(h[(size_t)(row0 + r) * K + k]);
                } else {
#pragma unroll
                    for (int i = 0; i < VEC; ++i) xv[r][i] = 0.0f;
                }
            }
#pragma unroll
            for (int j = 0; j < EC; ++j) {
                if (e0 + j >= outs) break;
                float wv[VEC];
                if constexpr (VEC == 4) load4(w + (size_t)(e0 + j) * K + k, wv);
                else wv[0] = w[(size_t)(e0 + j) * K + k];
#pragma unroll
                for (int r = 0; r < R; ++r)
#pragma unroll
                    for (int i = 0; i < VEC; ++i) s[j][r] = fmaf(xv[r][i], wv[i], s[j][r]);
            }
        }
#pragma unroll
        for (int j = 0; j < EC; ++j) {
            if (e0 + j >= outs) break;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float t = warp_sum(s[j][r]);
                if (lane == 0) part[((size_t)warp * outs + e0 + j) * R + r] = t;
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < R * outs; i += blockDim.x) {
        const int r = i / outs, e = i - r * outs;
        float t = 0.0f;
        for (int wp = 0; wp < 8; ++wp) t += part[((size_t)wp * outs + e) * R + r];
        router_z[i] = t + ((bias && e < experts) ? bias[e] : 0.0f);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < R * extra; i += blockDim.x) {
        const int r = i / extra, x = i - r * extra;
        if (row0 + r < rows) gate[(size_t)(row0 + r) * extra + x] = 1.0f / (1.0f + expf(-router_z[r * outs + experts + x]));
    }
    // A warp a row picks (R is at most the block's warps).  The warps' parts, which nobody reads any more, hold the row's
    // choice scores, the picked values and the groups' best scores.
    if (warp >= R || row0 + warp >= rows) return;
    float* z = router_z + warp * outs;                       // logits; over all: scores
    float* cs = part + (size_t)warp * 8 * outs;              // choice scores; a chosen one is struck out
    float* picked = cs + outs;
    float* best_of = picked + outs;
    int* mine = choice + (size_t)(row0 + warp) * top;
    float* wt = weight + (size_t)(row0 + warp) * top;
    if (rule.over_all) {
        float zmax = -INFINITY;
        for (int e = lane; e < experts; e += 32) zmax = fmaxf(zmax, z[e]);
        zmax = warp_max(zmax);
        float sum = 0.0f;
        for (int e = lane; e < experts; e += 32) {
            z[e] = expf(z[e] - zmax);
            sum += z[e];
        }
        sum = warp_sum(sum);
        for (int e = lane; e < experts; e += 32) {
            z[e] /= sum;
            cs[e] = z[e] + (rule.correction ? rule.correction[e] : 0.0f);
        }
        __syncwarp();
        if (rule.group_keep < rule.group_count) {
            const int size = experts / rule.group_count;
            for (int g = lane; g < rule.group_count; g += 32) {
                float b = -INFINITY;
                for (int i = 0; i < size; ++i) b = fmaxf(b, cs[g * size + i]);
                best_of[g] = b;
            }
            __syncwarp();
            for (int n = 0; n < rule.group_keep; ++n) {      // a kept group is marked by plus infinity once all lanes have looked
                float b = -INFINITY;
                int bi = -1;
                for (int g = lane; g < rule.group_count; g += 32)
                    if (best_of[g] > b && best_of[g] < INFINITY) b = best_of[g], bi = g;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const float ob = __shfl_xor_sync(0xffffffffu, b, o);
                    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                    if (ob > b || (ob == b && oi >= 0 && (bi < 0 || oi < bi))) b = ob, bi = oi;
                }
                __syncwarp();
                if (lane == 0 && bi >= 0) best_of[bi] = INFINITY;
                __syncwarp();
            }
            for (int e = lane; e < experts; e += 32)
                if (best_of[e / size] != INFINITY) cs[e] = -INFINITY;
            __syncwarp();
        }
    } else {
        for (int e = lane; e < experts; e += 32) cs[e] = z[e];
        __syncwarp();
    }
    for (int k = 0; k < top; ++k) {
        float bv;
        int best;
        warp_best(cs, experts, lane, bv, best);
        if (best < 0) {                                      // nothing left that is a number
            for (int e = 0; e < experts && best < 0; ++e)
                if (cs[e] != cs[e]) best = e;
            best = best < 0 ? 0 : best;
        }
        __syncwarp();
        if (lane == 0) {
            mine[k] = best;
            picked[k] = rule.over_all ? z[best] : bv;
            cs[best] = -INFINITY;
        }
        __syncwarp();
    }
    if (lane != 0) return;
    float sum = rule.over_all ? 1e-20f : 0.0f;
    const float zmax = picked[0];
    for (int k = 0; k < top; ++k) {
        if (!rule.over_all) picked[k] = zmax == -INFINITY ? 1.0f : expf(picked[k] - zmax);
        sum += picked[k];
    }
    for (int k = 0; k < top; ++k) wt[k] = picked[k] / sum * (rule.over_all ? rule.scale : 1.0f);
}

// x[row] += factor * sum_k pair_weight[row * top + k] * e_k + shared_gate[row] * shared[row], k in increasing order: e_k is
// the expert's output y[row * top + k], or, when `choice` names an expert beyond the `experts` that have weights, the row's
// input h[row].  `choice` null: every pair has an expert's output.  `shared` null: no such part.
template <typename T, int VEC>
__global__ void __launch_bounds__(256)
combine_weighted_kernel(const float* __restrict__ y, float* __restrict__ x, const float* __restrict__ pair_weight,
                        const int* __restrict__ choice, int experts, const T* __restrict__ h, const float* __restrict__ shared,
                        const float* __restrict__ shared_gate, int top, int width, float factor, long long pieces) {
    pdl_trigger();
    pdl_wait();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= pieces) return;
    const int per_row = width / VEC;
    const long long row = i / per_row;
    const int c = (int)(i - row * per_row) * VEC;
    auto read = [](auto* p, float (&v)[VEC]) {
        if constexpr (VEC == 4) load4(p, v);
        else v[0] = to_float(*p);
    };
    float s[VEC], v[VEC];
#pragma unroll
    for (int j = 0; j < VEC; ++j) s[j] = 0.0f;
    for (int k = 0; k < top; ++k) {
        const long long p = row * top + k;
        const float w = pair_weight[p];
        if (choice && choice[p] >= experts) read(h + (size_t)row * width + c, v);
        else read(y + (size_t)p * width + c, v);
#pragma unroll
        for (int j = 0; j < VEC; ++j) s[j] = fmaf(w, v[j], s[j]);
    }
    float* dst = x + (size_t)row * width + c;
    float t[VEC];
    read(dst, t);
#pragma unroll
    for (int j = 0; j < VEC; ++j) t[j] = fmaf(factor, s[j], t[j]);
    if (shared) {
        const float g = shared_gate[row];
        read(shared + (size_t)row * width + c, v);
#pragma unroll
        for (int j = 0; j < VEC; ++j) t[j] = fmaf(g, v[j], t[j]);
    }
    if constexpr (VEC == 4) *reinterpret_cast<float4*>(dst) = make_float4(t[0], t[1], t[2], t[3]);
    else dst[0] = t[0];
}

inline int max_tiles(int pairs, int experts, int tile_rows) { return (pairs + tile_rows - 1) / tile_rows + experts; }
}  // namespace

// h [rows, K] of `dtype`; w float32 [outputs + extra, K]; bias float32 [outputs] or null; choice int32 [rows, top]; weight float32
// [rows, top]; gate float32 [rows, extra] (extra 0: not used).  `over_all` 0: weights are the softmax over the chosen logits;
// 1: scores over all outputs, with `correction` [outputs] (or null) counting for the choice alone, `group_keep` of
// `group_count` groups, and `scale` on the weights.
LLMX_EXPORT int llmx_moe_router(const void* h, int dtype, const float* w, const float* bias, int rows, int K, int outputs, int top,
                                int extra, int over_all, const float* correction, int group_count, int group_keep, float scale,
                                int* choice, float* weight, float* gate, cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (K <= 0 || outputs <= 0 || top <= 0 || top > outputs || extra < 0 || extra > 128 || (extra > 0 && gate == nullptr) ||
        outputs + extra > 1024)
        return LLMX_ERR_BAD_ARGUMENT;
    if (over_all && (group_count <= 0 || outputs % group_count || group_keep <= 0 || group_keep > group_count ||
                     top > group_keep * (outputs / group_count)))
        return LLMX_ERR_BAD_ARGUMENT;
    const RouterChoice rule = {over_all, group_count, group_keep, correction, scale};
    // Eight rows a block when the rows are many (a weight row is then read once for eight rows), one when they are few.
    const bool vec = (K & 3) == 0 && !((uintptr_t)h & 15) && !((uintptr_t)w & 15);
    int R = rows > 64 ? 8 : 1;
    size_t smem = (size_t)9 * R * (outputs + extra) * sizeof(float);
    if (smem > 40 * 1024) R = 1, smem = (size_t)9 * (outputs + extra) * sizeof(float);
    if (smem > 40 * 1024) return LLMX_ERR_UNSUPPORTED;
    const dim3 grid((rows + R - 1) / R);
#define LLMX_ROUTER(T, RR, V) \
    launch_kernel(router_kernel<T, RR, V>, grid, dim3(256), smem, stream, (const T*)h, w, bias, rows, K, outputs, top, extra, rule, choice, weight, gate)
#define LLMX_ROUTER_T(T)                      \
    do {                                      \
        if (R == 8 && vec) LLMX_ROUTER(T, 8, 4); \
        else if (R == 8) LLMX_ROUTER(T, 8, 1);   \
        else if (vec) LLMX_ROUTER(T, 1, 4);      \
        else LLMX_ROUTER(T, 1, 1);               \
    } while (0)
    if (dtype == LLMX_BF16) LLMX_ROUTER_T(__nv_bfloat16);
    else if (dtype == LLMX_F32) LLMX_ROUTER_T(float);
    else return LLMX_ERR_UNSUPPORTED;
#undef LLMX_ROUTER_T
#undef LLMX_ROUTER
    return launch_status();
}

// x [rows, width] += factor * sum over k of pair_weight[rows * top] * (y [rows * top, width], or h [rows, width] of `h_dtype` where
// choice[rows * top] >= experts), k in increasing order, + shared_gate[rows] * shared [rows, width].  choice and h, shared and
// shared_gate: null when the design has no such experts, no such part.
LLMX_EXPORT int llmx_moe_combine_weighted(const float* y, float* x, const float* pair_weight, const int* choice, int experts,
                                          const void* h, int h_dtype, const float* shared, const float* shared_gate, int rows,
                                          int top, int width, float factor, cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (pair_weight == nullptr || top <= 0 || width <= 0 || (choice && h == nullptr) || (shared && shared_gate == nullptr))
        return LLMX_ERR_BAD_ARGUMENT;
    const bool vec = width % 4 == 0 && !(((uintptr_t)y | (uintptr_t)x | (uintptr_t)h | (uintptr_t)shared) & 15);
    const long long pieces = (long long)rows * (vec ? width / 4 : width);
    const dim3 grid((unsigned)((pieces + 255) / 256));
#define LLMX_COMBINE(T, V) \
    launch_kernel(combine_weighted_kernel<T, V>, grid, dim3(256), 0, stream, y, x, pair_weight, choice, experts, (const T*)h, shared, shared_gate, top, width, factor, pieces)
    if (h_dtype == LLMX_BF16 && vec) LLMX_COMBINE(__nv_bfloat16, 4);
    else if (h_dtype == LLMX_BF16) LLMX_COMBINE(__nv_bfloat16, 1);
    else if (vec) LLMX_COMBINE(float, 4);
    else LLMX_COMBINE(float, 1);
#undef LLMX_COMBINE
    return launch_status();
}

// The pairs a tile holds for the products on the CUDA cores, or of the tiles that go with the other form (it reads the counts alone).
LLMX_EXPORT int llmx_moe_tile_rows(int tensor_cores) { return tensor_cores ? TC_LIST_TILE : TILE_ROWS; }

// Whether the tensor-core form takes a product of these sizes and type.
LLMX_EXPORT int llmx_moe_tensor_cores_fit(int dtype, int K) { return dtype == LLMX_BF16 && K > 0 && K % 32 == 0; }

// token_ids int32 [rows]; table int32 [vocab, top]; lists int32 [experts, rows * top]; counts int32 [experts]; tiles int32
// [2 + 2 * (ceil(rows * top / tile_rows) + experts)], or null (the tensor cores' products read the counts alone).
LLMX_EXPORT int llmx_moe_route(const int* token_ids, const int* table, int top, int rows, int experts, int vocab, int* lists,
                               int* counts, int* tiles, int tile_rows, cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (top <= 0 || experts <= 0 || experts > 65535 || (tile_rows != TILE_ROWS && tile_rows != TC_LIST_TILE)) return LLMX_ERR_BAD_ARGUMENT;
    launch_kernel(route_kernel, dim3(experts), dim3(ROUTE_THREADS), 0, stream, token_ids, table, top, rows, experts, vocab, lists, counts);
    int status = launch_status();
    if (status) return status;
    if (tiles == nullptr) return 0;
    launch_kernel(tiles_kernel, dim3(1), dim3(32), 0, stream, (const int*)counts, experts, tiles, tile_rows);
    return launch_status();
}

// a [rows of `a_div` pairs each, K] and w [experts, (gated ? 2 : 1) * N, K] of `dtype`; out [pairs, N] of `out_dtype`
// (gated: silu(gate) * up, or the clamped unit of `limit` and `alpha` if `clamped`; else the plain product, float32).  The routing must have
// cut the lists into tiles of `llmx_moe_tile_rows(0)` pairs.
LLMX_EXPORT int llmx_moe_product(const void* a, int a_div, const void* w, int dtype, const int* lists, const int* counts,
                                 const int* tiles, int pairs, int experts, void* out, int out_dtype, int N, int K,
                                 int gated, int clamped, float limit, float alpha, cudaStream_t stream) {
    if (pairs <= 0) return 0;
    if (N <= 0 || K <= 0 || a_div <= 0) return LLMX_ERR_BAD_ARGUMENT;
    if (!gated && out_dtype != LLMX_F32) return LLMX_ERR_UNSUPPORTED;
    const Glu glu = {clamped, limit, alpha};
    dim3 grid(max_tiles(pairs, experts, TILE_ROWS), (N + CC_COLS - 1) / CC_COLS);
    if (grid.y > 65535) return LLMX_ERR_UNSUPPORTED;
#define LLMX_MOE(T, G, O) \
    launch_kernel(moe_cores_kernel<T, G, O>, dim3(grid), dim3(256), 0, stream, (const T*)a, a_div, (const T*)w, lists, counts, tiles, pairs, (O*)out, N, K, glu)
    if (dtype == LLMX_BF16 && gated && out_dtype == LLMX_BF16) LLMX_MOE(__nv_bfloat16, true, __nv_bfloat16);
    else if (dtype == LLMX_BF16 && gated && out_dtype == LLMX_F32) LLMX_MOE(__nv_bfloat16, true, float);
    else if (dtype == LLMX_BF16 && !gated) LLMX_MOE(__nv_bfloat16, false, float);
    else if (dtype == LLMX_F32 && gated && out_dtype == LLMX_F32) LLMX_MOE(float, true, float);
    else if (dtype == LLMX_F32 && !gated) LLMX_MOE(float, false, float);
    else return LLMX_ERR_UNSUPPORTED;
#undef LLMX_MOE
    return launch_status();
}

// rows [pairs, K] = the lists' rows of a [rows of `a_div` pairs each, K], bfloat16, one expert's after the other's.
LLMX_EXPORT int llmx_moe_gather(const void* a, int a_div, const int* lists, const int* counts, int experts, int pairs, void* rows, int K,
                                cudaStream_t stream) {
    if (pairs <= 0) return 0;
    if (K <= 0 || a_div <= 0 || experts <= 0) return LLMX_ERR_BAD_ARGUMENT;
    if (K % 8 || (((uintptr_t)a | (uintptr_t)rows) & 15)) return LLMX_ERR_UNSUPPORTED;
    launch_kernel(experts > MANY_EXPERTS ? gather_kernel<true> : gather_kernel<false>, dim3(pairs), dim3(GATHER_THREADS), 0, stream, (const uint4*)a,
                  a_div, lists, counts, experts, pairs, (uint4*)rows, K / 8);
    return launch_status();
}

// The same products on the tensor cores: rows [pairs, K] and w bfloat16, the rows sorted as the lists are; out [pairs, N] by pair or,
// `out_sorted`, in the rows' order.  `numbers`: int32 [4 m + 1] where m = min(pairs, experts) is more than TC_MAX_LISTED, else null.
LLMX_EXPORT int llmx_moe_product_tc(const void* rows, const void* w, const int* lists, const int* counts, int pairs, int experts, void* out,
                                    int out_dtype, int out_sorted, int N, int K, int gated, int clamped, float limit, float alpha,
                                    int* numbers, int* error_word, cudaStream_t stream) {
    if (pairs <= 0) return 0;
    if (N <= 0 || K <= 0 || experts <= 0) return LLMX_ERR_BAD_ARGUMENT;
    if (!gated && out_dtype != LLMX_F32) return LLMX_ERR_UNSUPPORTED;
    if (!llmx_moe_tensor_cores_fit(LLMX_BF16, K) || (((uintptr_t)rows | (uintptr_t)w) & 15)) return LLMX_ERR_UNSUPPORTED;
    const Glu glu = {clamped, limit, alpha};
    const int w_cols = gated ? TC_M : 2 * TC_M;
    const bool many = experts > MANY_EXPERTS;
    const int room = many && pairs < experts ? pairs : experts;   // experts that have a place
    const long long most = ((long long)pairs / TC_ROWS + room) * ((N + w_cols - 1) / w_cols);
    if (most >= (1ll << 31)) return LLMX_ERR_UNSUPPORTED;
    CUtensorMap w_map, r_map;
    const int per = gated ? 2 : 1;                   // gate rows and up rows are planes of their own
    if (int bad = make_map_3d(&w_map, w, K, N, (uint64_t)experts * per, TC_K, gated ? 16 : TC_M, per)) return bad;
    if (int bad = llmx_make_map_bf16_2d(&r_map, rows, (uint64_t)pairs, (uint64_t)K, TC_BOX, TC_K)) return bad;
    int device = 0, sms = 0;
    cudaGetDevice(&device);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || sms < 2) sms = 148;
    const bool apart = room > TC_MAX_LISTED;
    if (apart) {
        if (numbers == nullptr) return LLMX_ERR_BAD_ARGUMENT;
        launch_kernel(list_experts_kernel, dim3(1), dim3(LIST_THREADS), 0, stream, counts, experts, numbers, room);
        if (const int status = launch_status()) return status;
    }
    const int* made = apart ? numbers : nullptr;
    const int stages = tc_stages(apart ? 0 : room);
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)(2 * (most < sms / 2 ? most : sms / 2)));
    lc.blockDim = dim3(TC_THREADS);
    lc.dynamicSmemBytes = tc_smem(stages, apart ? 0 : room);
    lc.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr;
    lc.numAttrs = llmx_pdl_enabled() ? 2 : 1;
#define LLMX_MOE_TC_AS(G, O, M)                                                                                        \
    do {                                                                                                                \
        LLMX_ALLOW_SMEM(moe_tc_kernel<G, O, M>);                                                                        \
        cudaLaunchKernelEx(&lc, moe_tc_kernel<G, O, M>, w_map, r_map, lists, counts, experts, pairs, (O*)out, out_sorted, N, K, glu, stages, room, made, error_word); \
    } while (0)
#define LLMX_MOE_TC(G, O)                          \
    do {                                           \
        if (many) LLMX_MOE_TC_AS(G, O, true);      \
        else LLMX_MOE_TC_AS(G, O, false);          \
    } while (0)
    if (gated && out_dtype == LLMX_BF16) LLMX_MOE_TC(true, __nv_bfloat16);
    else if (gated) LLMX_MOE_TC(true, float);
    else LLMX_MOE_TC(false, float);
#undef LLMX_MOE_TC_AS
#undef LLMX_MOE_TC
    return launch_status();
}

// The same products for steps of a few pairs, without lists: a [rows of `a_div` pairs each, K] and w bfloat16 with K a
// multiple of 8; the pair's expert is read from the table.  `settled`: ids and table are written by none of the kernels launched since
// the stream was last waited for in full (a copy does): they may be read before the kernel before has ended.
LLMX_EXPORT int llmx_moe_product_few(const void* a, int a_div, const void* w, const int* token_ids, const int* table,
                                     int top, int vocab, int pairs, int experts, void* out, int out_dtype, int N, int K,
                                     int gated, int clamped, float limit, float alpha, int settled, int* error_word, cudaStream_t stream) {
    if (pairs <= 0) return 0;
    if (N <= 0 || K <= 0 || K % 8 || a_div <= 0 || top <= 0 || ((uintptr_t)a & 15) || ((uintptr_t)w & 15)) return LLMX_ERR_UNSUPPORTED;
    if (!gated && out_dtype != LLMX_F32) return LLMX_ERR_UNSUPPORTED;
    const Glu glu = {clamped, limit, alpha};
    const size_t smem = (size_t)K * 2;
    if (smem > 200 * 1024) return LLMX_ERR_UNSUPPORTED;
    const long long items = (long long)pairs * (gated ? N : (N + 1) / 2);
    if (pairs <= FEW_PAIRS && K <= FEW_K && items < (1ll << 31)) {
        int places = FEW_RING / (4 * K);
        places = places > FEW_PLACES ? FEW_PLACES : places;
        int workers = FEW_WARPS;                             // at least four: four places fit whatever K is
        while (places % workers) --workers;
        if (workers < 4) workers = 4, places = places / 4 * 4;
        const size_t ring = (size_t)places * 4 * K;
        const dim3 stream_grid((unsigned)(items < 148 ? items : 148));
#define LLMX_FEW(G, O)                                                                                                  \
    do {                                                                                                                \
        LLMX_ALLOW_SMEM(moe_few_stream_kernel<G, O>);                                                                   \
        launch_kernel(moe_few_stream_kernel<G, O>, stream_grid, dim3(32 * workers + 32), ring, stream, (const __nv_bfloat16*)a, a_div, \
                      (const __nv_bfloat16*)w, token_ids, table, top, vocab, experts, pairs, (O*)out, N, K, glu, places, settled != 0, error_word); \
    } while (0)
        if (gated && out_dtype == LLMX_BF16) LLMX_FEW(true, __nv_bfloat16);
        else if (gated) LLMX_FEW(true, float);
        else LLMX_FEW(false, float);
#undef LLMX_FEW
        return launch_status();
    }
    dim3 grid(pairs, (N + GV_COLS - 1) / GV_COLS);
    if (grid.y > 65535) return LLMX_ERR_UNSUPPORTED;
#define LLMX_FEW(G, O)                                                                                                  \
    do {                                                                                                                \
        if (smem > 48 * 1024) LLMX_ALLOW_SMEM(moe_few_kernel<G, O>);                                                    \
        launch_kernel(moe_few_kernel<G, O>, dim3(grid), dim3(256), smem, stream, (const __nv_bfloat16*)a, a_div,       \
                      (const __nv_bfloat16*)w, token_ids, table, top, vocab, experts, (O*)out, N, K, glu);              \
    } while (0)
    if (gated && out_dtype == LLMX_BF16) LLMX_FEW(true, __nv_bfloat16);
    else if (gated) LLMX_FEW(true, float);
    else LLMX_FEW(false, float);
#undef LLMX_FEW
    return launch_status();
}

// x [rows, width] += weight * sum over k of y [rows * top, width], k in increasing order.
LLMX_EXPORT int llmx_moe_combine(const float* y, float* x, int rows, int top, int width, float weight, cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (width > 0 && width % 4 == 0 && width <= 4 * 256 * 65535 && !(((uintptr_t)y | (uintptr_t)x) & 15)) {
        launch_kernel(combine_vec_kernel, dim3(rows, (width / 4 + 255) / 256), dim3(256), 0, stream, (const float4*)y, (float4*)x, top, width / 4, weight);
        return launch_status();
    }
    const long long n = (long long)rows * width;
    launch_kernel(combine_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, stream, y, x, top, width, weight, n);
    return launch_status();
}
