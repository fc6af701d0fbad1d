// The products of routed experts for many rows, on the tcgen05 tensor cores: rows sorted by expert, every expert's
// run of rows padded to whole tiles of 128, so that a tile has one expert and the product is an ordinary tiled one
// whose weight operand is chosen per row tile.
//
//   moe_sort      pairs (token, k-th choice) -> places in the sorted order. Two launches (three for steps of very many
//                 pairs or experts, whose counts and places are kernels of their own): a count per expert (each
//                 pair draws its rank within its expert with an atomic: the order within an expert is whatever the
//                 hardware made it, which no result depends on, a row's product being its own); the experts' first
//                 places (runs padded to 128 rows) and the expert of every row tile (-1 beyond the last); the rows
//                 themselves gathered into their places, multiplied by the pair's weight where the weight acts on
//                 the expert's input (rounded to bfloat16 like any stored activation).
//   gemm_grouped  out[p, :] = act(W[expert of p's tile] x[p, :]) for the sorted rows: TMA (128-byte swizzle) -> ring
//                 of stages -> tcgen05.mma 128 x 128 x 16 into tensor memory -> tcgen05.ld epilogue, one warp that
//                 loads, one that multiplies, four that store. The weights are one matrix [experts * N, K]; a tile's
//                 weight rows start at expert * N + its column. Long runs go to pairs of CTAs (below). Tiles beyond the last used one leave at once. Rows of
//                 padding hold whatever the buffer held; their results are never read. Gated: an expert's matrix holds gate
//                 and up rows in turns of 64, so that a tile of 128 columns has both of 64 features, and the activation
//                 is applied where the tile is stored.
//   moe_unsort    out[t] (+)= sum over k of sorted[place of pair t * top + k], in the order of k.
// All waits on barriers are bounded (tc::mbar_wait); a wait that runs out sets status word 1.
#define ABK_DEFINE_ERROR
#include "common.cuh"
#include "tc_common.cuh"
#include "tensor_map.cuh"

#define GG_ROWS 128
#define GG_BN 128
#define GG_K 64
#define GG_STAGES 4
#define GG_THREADS 192
enum { GG_NONE = 0, GG_RELU_SQUARED = 1, GG_SILU_GATED = 2, GG_CLAMPED_GATED = 3 };
#define GG_TURN (GG_BN / 2)  // rows of gate, then of up, of a gated matrix

// ---------------------------------------------------------------- sorting pairs by expert
__global__ void __launch_bounds__(256) moe_count_kernel(const int *pair_expert, int n_pairs, int *counts, int *rank) {
    pdl_wait();
    const int p = blockIdx.x * 256 + threadIdx.x;
    if (p >= n_pairs) return;
    const int e = pair_expert[p];
    rank[p] = e >= 0 ? atomicAdd(&counts[e], 1) : 0;
}

// The expert of row tile t, whose tiles start at tiles[expert]; -1 beyond the used ones.
__device__ __forceinline__ int expert_of_tile(const int *tiles, int experts, int t) {
    if (t >= tiles[experts]) return -1;
    int lo = 0, hi = experts - 1;  // the last expert whose first tile is <= t and that has tiles
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (tiles[mid] <= t) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// first[e]: the first sorted row of expert e; tile_expert[t]: the expert of row tile t, -1 beyond the used tiles.
__global__ void __launch_bounds__(256) moe_offsets_kernel(const int *counts, int experts, int *first, int *tile_expert,
                                                          int max_tiles) {
    extern __shared__ int mo_tiles[];  // [experts + 1] first tile of each expert
    pdl_wait();
    if (threadIdx.x == 0) {
        int tile = 0;
        for (int e = 0; e < experts; e++) {
            mo_tiles[e] = tile;
            first[e] = tile * GG_ROWS;
            tile += (counts[e] + GG_ROWS - 1) / GG_ROWS;
        }
        mo_tiles[experts] = tile;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < max_tiles; t += 256) tile_expert[t] = expert_of_tile(mo_tiles, experts, t);
}

// Both of the above, and the counts' zeros, by one CTA: a launch that may start while the kernel before still runs, in place of three that
// may not. With the gathering, 6,002 pairs, 16 experts, rows of 2,560: 9.8 us, with the three 16.4; 300 pairs: 3.1 and 9.1.
#define MP_THREADS 1024
#define MP_PAIRS 32768  // pairs that one CTA counts (moe_plans)
__global__ void __launch_bounds__(MP_THREADS) moe_plan_kernel(const int *pair_expert, int n_pairs, int experts, int *rank, int *first,
                                                              int *tile_expert, int max_tiles) {
    extern __shared__ int mp_tiles[];  // [experts + 1] first tile of each expert; [experts] pairs
    int *counts = mp_tiles + experts + 1;
    for (int e = threadIdx.x; e < experts; e += MP_THREADS) counts[e] = 0;
    __syncthreads();
    pdl_wait();
#pragma unroll 4
    for (int p = threadIdx.x; p < n_pairs; p += MP_THREADS) {
        const int e = pair_expert[p];
        rank[p] = e >= 0 ? atomicAdd(&counts[e], 1) : 0;
    }
    __syncthreads();
    if (threadIdx.x < 32) {  // a warp: the sums of 32 experts' tiles at a time
        int before = 0;
        for (int base = 0; base < experts; base += 32) {
            const int e = base + threadIdx.x, mine = e < experts ? (counts[e] + GG_ROWS - 1) / GG_ROWS : 0;
            int upto = mine;
#pragma unroll
            for (int m = 1; m < 32; m <<= 1) {
                const int other = __shfl_up_sync(0xffffffffu, upto, m);
                if ((int)threadIdx.x >= m) upto += other;
            }
            if (e < experts) mp_tiles[e] = before + upto - mine, first[e] = (before + upto - mine) * GG_ROWS;
            before += __shfl_sync(0xffffffffu, upto, 31);
        }
        if (threadIdx.x == 0) mp_tiles[experts] = before;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < max_tiles; t += MP_THREADS) tile_expert[t] = expert_of_tile(mp_tiles, experts, t);
}

// x row of pair p: x + (p / pairs_per_row) * ldx; its place: first[expert] + rank; sorted[place] = scale * x (bfloat16).
__global__ void __launch_bounds__(128) moe_gather_kernel(const __nv_bfloat16 *x, long long ldx, int pairs_per_row,
                                                         const int *pair_expert, const float *pair_scale, const int *rank,
                                                         const int *first, int *place, __nv_bfloat16 *sorted, int d) {
    const int p = blockIdx.x;
    pdl_wait();
    const int e = pair_expert[p];
    if (e < 0) {
        if (threadIdx.x == 0) place[p] = -1;
        return;
    }
    const int at = first[e] + rank[p];
    if (threadIdx.x == 0) place[p] = at;
    const __nv_bfloat16 *src = x + (long long)(p / pairs_per_row) * ldx;
    __nv_bfloat16 *dst = sorted + (long long)at * d;
    if (d % 8 == 0 && ldx % 8 == 0 && (((uintptr_t)x | (uintptr_t)sorted) & 15) == 0) {  // 16-byte pieces
        const float sc = pair_scale ? pair_scale[p] : 1.0f;
        for (int i = threadIdx.x * 8; i < d; i += 128 * 8) {
            uint4 raw = *(const uint4 *)(src + i);
            if (pair_scale) {
                __nv_bfloat162 *h = (__nv_bfloat162 *)&raw;
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const float2 f = __bfloat1622float2(h[u]);
                    h[u] = __floats2bfloat162_rn(sc * f.x, sc * f.y);
                }
            }
            *(uint4 *)(dst + i) = raw;
        }
    } else if (pair_scale) {
        const float sc = pair_scale[p];
        for (int i = threadIdx.x; i < d; i += 128) dst[i] = __float2bfloat16_rn(sc * __bfloat162float(src[i]));
    } else {
        for (int i = threadIdx.x; i < d; i += 128) dst[i] = src[i];
    }
}

// Pairs of a step and experts that one CTA plans: 16 experts, 32,768 pairs, with the gathering 45.4 us by one CTA and 47.4 by many, 8 experts 45.9
// and 47.2 (24,576: 32.9 and 36.8; all pairs of one expert 55.7 and 63.7; 64 experts 44 and 53); one CTA's shared memory and time grow with both.
static bool moe_plans(int n_pairs, int experts) { return n_pairs <= MP_PAIRS && experts <= 4096; }
// Kernels that abk_moe_sort launches.
extern "C" int abk_moe_sort_kernels(int n_pairs, int experts) { return n_pairs <= 0 ? 0 : moe_plans(n_pairs, experts) ? 2 : 3; }

// counts [experts], rank and place [n_pairs], first [experts], tile_expert [max_tiles] int32; sorted bfloat16
// [max_tiles * 128, d]. max_tiles >= ceil(n_pairs / 128) + experts.
extern "C" int abk_moe_sort(const void *x, long long ldx, int pairs_per_row, const int *pair_expert, const float *pair_scale,
                            int n_pairs, int experts, int d, int *counts, int *rank, int *first, int *place,
                            int *tile_expert, int max_tiles, void *sorted, void *stream) {
    if (n_pairs <= 0) return 0;
    if (max_tiles < (n_pairs + GG_ROWS - 1) / GG_ROWS + experts)
        ABK_REFUSE("moe_sort: %d row tiles do not hold %d pairs of %d experts", max_tiles, n_pairs, experts);
    if (experts > 8192) ABK_REFUSE("moe_sort: %d experts", experts);
    cudaStream_t s = (cudaStream_t)stream;
    if (moe_plans(n_pairs, experts)) {
        abk_launch(moe_plan_kernel, dim3(1), dim3(MP_THREADS), (size_t)(2 * experts + 1) * sizeof(int), s, pair_expert, n_pairs, experts, rank, first,
                   tile_expert, max_tiles);
    } else {
        cudaError_t err = cudaMemsetAsync(counts, 0, (size_t)experts * sizeof(int), s);
        if (err != cudaSuccess) return (int)err;
        moe_count_kernel<<<(n_pairs + 255) / 256, 256, 0, s>>>(pair_expert, n_pairs, counts, rank);
        moe_offsets_kernel<<<1, 256, (size_t)(experts + 1) * sizeof(int), s>>>(counts, experts, first, tile_expert, max_tiles);
    }
    abk_launch(moe_gather_kernel, dim3(n_pairs), dim3(128), 0, s, (const __nv_bfloat16 *)x, ldx, pairs_per_row < 1 ? 1 : pairs_per_row,
               pair_expert, pair_scale, (const int *)rank, (const int *)first, place, (__nv_bfloat16 *)sorted, d);
    return ABK_LAUNCH_RESULT();
}

// ---------------------------------------------------------------- the product
struct GemmGrouped {
    void *out;
    long long ldo;
    int N, K, k_blocks;
    const int *tile_expert;
    int *status;
    int vec;  // every 16-column run of an output row starts on a 16-byte boundary
    float limit;  // of the clamped activation
};

struct GroupedSmem {
    static constexpr int A_BYTES = GG_ROWS * GG_K * 2, B_BYTES = GG_BN * GG_K * 2;
    static constexpr int BYTES = GG_STAGES * (A_BYTES + B_BYTES) + 1024 /* alignment */ + 256 /* barriers */;
};

__device__ __forceinline__ void gg_store16(float *dst, const uint32_t *v) {
#pragma unroll
    for (int j = 0; j < 16; j += 4) *(uint4 *)(dst + j) = make_uint4(v[j], v[j + 1], v[j + 2], v[j + 3]);
}
__device__ __forceinline__ void gg_store16(__nv_bfloat16 *dst, const uint32_t *v) {
    uint32_t h[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
        __nv_bfloat162 t = __floats2bfloat162_rn(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
        h[j] = *(uint32_t *)&t;
    }
    *(uint4 *)dst = make_uint4(h[0], h[1], h[2], h[3]);
    *(uint4 *)(dst + 8) = make_uint4(h[4], h[5], h[6], h[7]);
}

template <typename TO, int ACT>
__global__ void __launch_bounds__(GG_THREADS) gemm_grouped_kernel(const __grid_constant__ CUtensorMap map_x,
                                                                  const __grid_constant__ CUtensorMap map_w, GemmGrouped g) {
    using S = GroupedSmem;
    // the tile's expert was written at least two launches back (the gather stands between): it may be read at once
    const int expert = g.tile_expert[blockIdx.x];
    if (expert < 0) return;
    extern __shared__ uint8_t gg_smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)gg_smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *a_tiles = smem, *b_tiles = smem + GG_STAGES * S::A_BYTES;
    uint64_t *full = (uint64_t *)(smem + GG_STAGES * (S::A_BYTES + S::B_BYTES));
    uint64_t *empty = full + GG_STAGES, *acc_ready = empty + GG_STAGES;
    uint32_t *tmem_holder = (uint32_t *)(acc_ready + 1);
    volatile int *flags = (volatile int *)(tmem_holder + 1);  // [0]: a wait ran out

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int p0 = blockIdx.x * GG_ROWS, q0 = blockIdx.y * GG_BN;
    const int w_row = expert * g.N + q0;
    if (threadIdx.x == 0) {
        for (int s = 0; s < GG_STAGES; s++) tc::mbar_init(&full[s], 1), tc::mbar_init(&empty[s], 1);
        tc::mbar_init(acc_ready, 1);
        flags[0] = 0;
        tc::mbar_init_fence();
        tc::tma_prefetch_map(&map_x), tc::tma_prefetch_map(&map_w);
    }
    if (warp == 1) tc::tmem_alloc(tmem_holder, GG_BN);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *tmem_holder;
    if (warp == 0) {
        if (lane == 0) {
            // the weights' first stages are asked for at once; the rows (the launch before wrote them) after the wait
            const int ahead = min(GG_STAGES, g.k_blocks);
            for (int i = 0; i < ahead; i++) {
                tc::mbar_expect_tx(&full[i], S::A_BYTES + S::B_BYTES);
                tc::tma_load_2d(b_tiles + i * S::B_BYTES, &map_w, i * GG_K, w_row, &full[i]);
            }
            pdl_wait();
            int issued = 0;
            for (int kb = 0; kb < g.k_blocks; kb++, issued++) {
                const int s = issued % GG_STAGES;
                if (issued >= ahead) {
                    if (!tc::mbar_wait(&empty[s], ((issued / GG_STAGES) & 1) ^ 1)) {
                        flags[0] = 1;
                        break;
                    }
                    tc::mbar_expect_tx(&full[s], S::A_BYTES + S::B_BYTES);
                    tc::tma_load_2d(b_tiles + s * S::B_BYTES, &map_w, kb * GG_K, w_row, &full[s]);
                }
                tc::tma_load_2d(a_tiles + s * S::A_BYTES, &map_x, kb * GG_K, p0, &full[s]);
            }
            if (flags[0]) {  // let the copies still in flight land before the CTA's memory goes away
                for (int i = max(0, issued - GG_STAGES); i < issued; i++) tc::mbar_wait(&full[i % GG_STAGES], (i / GG_STAGES) & 1);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc = tc::idesc_bf16_f32(GG_ROWS, GG_BN);
            int done = 0;
            for (int kb = 0; kb < g.k_blocks; kb++, done++) {
                const int s = done % GG_STAGES;
                if (!tc::mbar_wait(&full[s], (done / GG_STAGES) & 1)) {
                    flags[0] = 1;
                    break;
                }
                tc::fence_after_sync();
                const uint32_t a = tc::smem_addr(a_tiles + s * S::A_BYTES), b = tc::smem_addr(b_tiles + s * S::B_BYTES);
#pragma unroll
                for (int k = 0; k < GG_K / 16; k++)
                    tc::mma_ss(tmem, tc::smem_desc_k_sw128(a + k * 32), tc::smem_desc_k_sw128(b + k * 32), idesc, done > 0 || k > 0);
                tc::mma_commit(&empty[s]);
            }
            tc::mma_commit(acc_ready);
        }
    } else {
        // epilogue: warp w reads lanes 32 * (w % 4) .. + 31 of the accumulator
        const int quarter = warp & 3, row = quarter * 32 + lane;
        const bool ok = tc::mbar_wait(acc_ready, 0);
        if (!ok) flags[0] = 1;
        tc::fence_after_sync();
        TO *out = (TO *)g.out + (long long)(p0 + row) * g.ldo;
        if (ok && ACT >= GG_SILU_GATED) {
            const int f0 = q0 / 2;  // the tile's first feature
#pragma unroll 1
            for (int c0 = 0; c0 < GG_TURN; c0 += 16) {
                uint32_t v[16], u[16];
                tc::tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + c0, v);
                tc::tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + GG_TURN + c0, u);
                tc::tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; j++) {  // gate and up pass through bfloat16, as they do where they are stored in between
                    const float gate = __bfloat162float(__float2bfloat16_rn(__uint_as_float(v[j])));
                    const float up = __bfloat162float(__float2bfloat16_rn(__uint_as_float(u[j])));
                    v[j] = __float_as_uint(gated_mul(ACT == GG_CLAMPED_GATED ? ABK_CLAMPED : ABK_SILU, gate, up, g.limit));
                }
                if (g.vec) {
                    gg_store16(out + f0 + c0, v);
                } else {
#pragma unroll
                    for (int j = 0; j < 16; j++) out[f0 + c0 + j] = from_float<TO>(__uint_as_float(v[j]));
                }
            }
        } else if (ok) {
#pragma unroll 1
            for (int c0 = 0; c0 < GG_BN; c0 += 16) {
                if (q0 + c0 >= g.N) break;
                uint32_t v[16];
                tc::tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + c0, v);
                tc::tmem_ld_wait();
                if (ACT == GG_RELU_SQUARED) {
#pragma unroll
                    for (int j = 0; j < 16; j++) {
                        const float f = __uint_as_float(v[j]);
                        v[j] = __float_as_uint(f > 0.0f ? f * f : 0.0f);
                    }
                }
                if (g.vec && q0 + c0 + 16 <= g.N) {
                    gg_store16(out + q0 + c0, v);
                } else {
#pragma unroll
                    for (int j = 0; j < 16; j++)
                        if (q0 + c0 + j < g.N) out[q0 + c0 + j] = from_float<TO>(__uint_as_float(v[j]));
                }
            }
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (flags[0] && threadIdx.x == 0) atomicOr(g.status + 1, 1);
    if (warp == 1) {
        tc::fence_after_sync();
        tc::tmem_free(tmem, GG_BN);
    }
}

// The same product on pairs of CTAs (cta_group::2). A tile of 128 x 128 asks the L2 for 32 KB every 128 cycles of the tensor
// core, four times what an SM gets from it; a pair's tile of 256 x 256 asks for as much every 256 cycles of either SM, its CTAs
// are persistent, and one accumulator is stored while the other is filled. The pairs' rows are two neighbouring row tiles of
// one expert (the leader's and its peer's; an expert's odd last tile has a peer that stores nothing), listed in shared memory
// by every CTA for itself from the row tiles' experts. Measured, 16 experts, 6,002 rows of 2,560 into 2,432 and
// back: 89 and 114 us (840 and 656 TFLOP/s), where the tiles of 128 x 128 take 126 and 167.
#define GP_BN 256
#define GP_STAGES 6
#define GP_MAX_TILES 4096   // row tiles the list holds

struct GroupedPairSmem {
    static constexpr int A_BYTES = GG_ROWS * GG_K * 2, B_BYTES = (GP_BN / 2) * GG_K * 2;
    static constexpr int BYTES = GP_STAGES * (A_BYTES + B_BYTES) + 1024 /* alignment */ + 256 /* barriers */ + GP_MAX_TILES * 2;
};

template <typename TO, int ACT>
__global__ void __launch_bounds__(GG_THREADS) gemm_grouped_pair_kernel(const __grid_constant__ CUtensorMap map_x,
                                                                       const __grid_constant__ CUtensorMap map_w, GemmGrouped g, int max_tiles) {
    using S = GroupedPairSmem;
    extern __shared__ uint8_t gg_smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)gg_smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *a_tiles = smem, *b_tiles = smem + GP_STAGES * S::A_BYTES;
    uint64_t *full = (uint64_t *)(smem + GP_STAGES * (S::A_BYTES + S::B_BYTES));
    uint64_t *empty = full + GP_STAGES, *acc_full = empty + GP_STAGES, *acc_empty = acc_full + 2;
    uint32_t *tmem_holder = (uint32_t *)(acc_empty + 2);
    volatile int *flags = (volatile int *)(tmem_holder + 1);  // [0]: a wait ran out, [1]: entries of the list
    uint16_t *list = (uint16_t *)((uint8_t *)full + 256);     // first row tile * 2 + whether the next one is the expert's too

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)tc::cluster_rank();  // 0: the leader, 1: its peer
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    if (threadIdx.x == 0) {
        for (int s = 0; s < GP_STAGES; s++) tc::mbar_init(&full[s], 1), tc::mbar_init(&empty[s], 1);
        for (int b = 0; b < 2; b++) tc::mbar_init(&acc_full[b], 1), tc::mbar_init(&acc_empty[b], 8);  // every storing warp of both CTAs
        flags[0] = 0;
        tc::mbar_init_fence();
        tc::tma_prefetch_map(&map_x), tc::tma_prefetch_map(&map_w);
    }
    if (warp == 1) tc::tmem_alloc_pair(tmem_holder, 2 * GP_BN);
    if (warp == 2) {  // the tiles' experts were written at least two launches back: they may be read at once
        int count = 0, run_carry = 0;  // the run of one expert's tiles that reaches into these 32 from before
        for (int base = 0; base < max_tiles; base += 32) {
            const int t = base + lane, e = t < max_tiles ? g.tile_expert[t] : -1;
            const bool starts = t == 0 || (t < max_tiles && g.tile_expert[t - 1] != e);
            const unsigned run_starts = __ballot_sync(0xffffffffu, starts), upto = run_starts & (0xffffffffu >> (31 - lane));
            const int run = upto ? base + 31 - __clz(upto) : run_carry;
            run_carry = __shfl_sync(0xffffffffu, run, 31);
            const bool first = e >= 0 && ((t - run) & 1) == 0;
            const bool both = first && t + 1 < max_tiles && g.tile_expert[t + 1] == e;
            const unsigned firsts = __ballot_sync(0xffffffffu, first);
            if (first) list[count + __popc(firsts & ((1u << lane) - 1))] = (uint16_t)(2 * t + (both ? 1 : 0));
            count += __popc(firsts);
        }
        if (lane == 0) flags[1] = count;
    }
    tc::fence_before_sync();
    tc::cluster_sync();  // both CTAs' barriers are there before either signals the other's
    tc::fence_after_sync();
    const uint32_t tmem = *tmem_holder;
    const int m_tiles = flags[1], n_tiles = (g.N + GP_BN - 1) / GP_BN, tiles = m_tiles * n_tiles;

    if (warp == 0) {
        if (lane == 0 && pair < tiles) {
            // A stage is full when both CTAs' copies have landed: all of them report to the leader's barrier.
            constexpr uint32_t STAGE_BYTES = 2 * (S::A_BYTES + S::B_BYTES);
            const int ahead = min(GP_STAGES, g.k_blocks);
            {   // the weights of the first tile's first stages are asked for before pdl_wait(): nobody writes them
                const int w_row = g.tile_expert[list[pair % m_tiles] >> 1] * g.N + (pair / m_tiles) * GP_BN + rank * (GP_BN / 2);
                for (int i = 0; i < ahead; i++) {
                    if (rank == 0) tc::mbar_expect_tx(&full[i], STAGE_BYTES);
                    tc::tma_load_2d_pair(b_tiles + i * S::B_BYTES, &map_w, i * GG_K, w_row, tc::peer_smem(tc::smem_addr(&full[i]), 0));
                }
            }
            pdl_wait();
            int issued = 0;
            for (int t = pair; t < tiles && !flags[0]; t += pairs) {
                const int first = list[t % m_tiles] >> 1;
                // (the peer's rows of an odd last tile: the same rows again, which are there, and nothing is stored)
                const int p0 = (first + (rank && (list[t % m_tiles] & 1) ? 1 : 0)) * GG_ROWS;
                const int w_row = g.tile_expert[first] * g.N + (t / m_tiles) * GP_BN + rank * (GP_BN / 2);
                for (int kb = 0; kb < g.k_blocks; kb++, issued++) {
                    const int s = issued % GP_STAGES;
                    const uint32_t bar = tc::peer_smem(tc::smem_addr(&full[s]), 0);
                    if (issued >= ahead) {
                        if (!tc::mbar_wait(&empty[s], ((issued / GP_STAGES) & 1) ^ 1)) {  // (its own: the commit reaches both)
                            flags[0] = 1;
                            break;
                        }
                        if (rank == 0) tc::mbar_expect_tx(&full[s], STAGE_BYTES);
                        tc::tma_load_2d_pair(b_tiles + s * S::B_BYTES, &map_w, kb * GG_K, w_row, bar);
                    }
                    tc::tma_load_2d_pair(a_tiles + s * S::A_BYTES, &map_x, kb * GG_K, p0, bar);
                }
            }
        } else if (lane == 0) {
            pdl_wait();
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            constexpr uint32_t idesc = tc::idesc_bf16_f32(2 * GG_ROWS, GP_BN);
            int done = 0, it = 0;
            for (int t = pair; t < tiles && !flags[0]; t += pairs, it++) {
                const int b = it & 1;
                if (!tc::mbar_wait(&acc_empty[b], ((it >> 1) & 1) ^ 1)) {  // both CTAs are done with this accumulator
                    flags[0] = 1;
                    break;
                }
                tc::fence_after_sync();
                for (int kb = 0; kb < g.k_blocks; kb++, done++) {
                    const int s = done % GP_STAGES;
                    if (!tc::mbar_wait(&full[s], (done / GP_STAGES) & 1)) {
                        flags[0] = 1;
                        break;
                    }
                    tc::fence_after_sync();
                    const uint32_t a = tc::smem_addr(a_tiles + s * S::A_BYTES), bq = tc::smem_addr(b_tiles + s * S::B_BYTES);
#pragma unroll
                    for (int k = 0; k < GG_K / 16; k++)
                        tc::mma_ss_pair(tmem + b * GP_BN, tc::smem_desc_k_sw128(a + k * 32), tc::smem_desc_k_sw128(bq + k * 32), idesc, kb > 0 || k > 0);
                    tc::mma_commit_pair(&empty[s]);
                }
                if (flags[0]) break;
                tc::mma_commit_pair(&acc_full[b]);
            }
        }
    } else {
        const int quarter = warp & 3, row = quarter * 32 + lane;
        const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16);
        int it = 0;
        pdl_wait();
        for (int t = pair; t < tiles; t += pairs, it++) {
            const int b = it & 1, entry = list[t % m_tiles], q0 = (t / m_tiles) * GP_BN;
            const bool stores = rank == 0 || (entry & 1);
            TO *out = (TO *)g.out + ((long long)((entry >> 1) + rank) * GG_ROWS + row) * g.ldo;
            const bool ok = __all_sync(0xffffffffu, !flags[0] && tc::mbar_wait(&acc_full[b], (it >> 1) & 1));
            if (!ok) {
                flags[0] = 1;
                break;
            }
            tc::fence_after_sync();
            if constexpr (ACT >= GG_SILU_GATED) {
#pragma unroll 1
                for (int c0 = 0; c0 < GP_BN; c0 += 2 * GG_TURN)  // gate and up rows come in turns of 64
#pragma unroll 1
                    for (int c = 0; c < GG_TURN && q0 + c0 < g.N; c += 16) {
                        uint32_t v[16], u[16];
                        tc::tmem_ld16(lanes + b * GP_BN + c0 + c, v);
                        tc::tmem_ld16(lanes + b * GP_BN + c0 + GG_TURN + c, u);
                        tc::tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 16; j++) {  // gate and up pass through bfloat16, as they do where they are stored in between
                            const float gate = __bfloat162float(__float2bfloat16_rn(__uint_as_float(v[j])));
                            const float up = __bfloat162float(__float2bfloat16_rn(__uint_as_float(u[j])));
                            v[j] = __float_as_uint(gated_mul(ACT == GG_CLAMPED_GATED ? ABK_CLAMPED : ABK_SILU, gate, up, g.limit));
                        }
                        TO *dst = out + (q0 + c0) / 2 + c;
                        if (stores && g.vec) {
                            gg_store16(dst, v);
                        } else if (stores) {
#pragma unroll
                            for (int j = 0; j < 16; j++) dst[j] = from_float<TO>(__uint_as_float(v[j]));
                        }
                    }
            } else {
#pragma unroll 1
                for (int c0 = 0; c0 < GP_BN && q0 + c0 < g.N; c0 += 32) {
                    uint32_t v[32];
                    tc::tmem_ld16(lanes + b * GP_BN + c0, v);
                    tc::tmem_ld16(lanes + b * GP_BN + c0 + 16, v + 16);
                    tc::tmem_ld_wait();
                    if (ACT == GG_RELU_SQUARED) {
#pragma unroll
                        for (int j = 0; j < 32; j++) {
                            const float f = __uint_as_float(v[j]);
                            v[j] = __float_as_uint(f > 0.0f ? f * f : 0.0f);
                        }
                    }
#pragma unroll
                    for (int h = 0; h < 32; h += 16) {
                        if (stores && g.vec && q0 + c0 + h + 16 <= g.N) {
                            gg_store16(out + q0 + c0 + h, v + h);
                        } else if (stores) {
#pragma unroll
                            for (int j = 0; j < 16; j++)
                                if (q0 + c0 + h + j < g.N) out[q0 + c0 + h + j] = from_float<TO>(__uint_as_float(v[h + j]));
                        }
                    }
                }
            }
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive_in_cluster(tc::peer_smem(tc::smem_addr(&acc_empty[b]), 0));
        }
    }
    // Nobody leaves while the other CTA may still signal its barriers or write its tensor memory. (After a wait that ran
    // out, copies may still be on their way into this CTA's shared memory: give them a tenth of a millisecond.)
    if (flags[0]) {
        const uint64_t t0 = tc::global_ns();
        while (tc::global_ns() - t0 < 100000) __nanosleep(1000);
    }
    tc::fence_before_sync();
    tc::cluster_sync();
    if (flags[0] && threadIdx.x == 0) atomicOr(g.status + 1, 1);
    if (warp == 1) {
        tc::fence_after_sync();
        tc::tmem_free_pair(tmem, 2 * GP_BN);
    }
}

// x bfloat16 [max_tiles * 128, K] (sorted rows); w bfloat16 [experts, N, K]; out [max_tiles * 128, ldo] bfloat16 or
// (out_f32) float32; tile_expert int32 [max_tiles]; status int32 [>= 2]. Gated: N counts gate and up rows (a multiple of 128),
// out has N / 2 columns. in_pairs: 1 or 0 pins the kernel on pairs of CTAs or the one on single ones; -1: whichever is faster.
extern "C" int abk_gemm_grouped(const void *x, const void *w, void *out, long long ldo, int out_f32, int activation,
                                int max_tiles, int experts, int N, int K, const int *tile_expert, float limit, int *status, int in_pairs,
                                void *stream) {
    if (max_tiles <= 0 || N <= 0) return 0;
    if (K <= 0 || K % 8) ABK_REFUSE("gemm_grouped: K = %d must be a multiple of 8", K);
    const bool gated = activation == GG_SILU_GATED || activation == GG_CLAMPED_GATED;
    if (gated && (N % GG_BN || out_f32)) ABK_REFUSE("gemm_grouped: gate and up rows in turns of %d do not fit %d rows", GG_TURN, N);
    if (activation < GG_NONE || activation > GG_CLAMPED_GATED) ABK_REFUSE("gemm_grouped: activation %d is not built", activation);
    CUtensorMap mx, mw;
    int rc = tmap::bf16_rows_of_128_bytes(x, (long long)max_tiles * GG_ROWS, K, K, GG_ROWS, &mx);
    if (rc) return rc;
    rc = tmap::bf16_rows_of_128_bytes(w, (long long)experts * N, K, K, GG_BN, &mw);
    if (rc) return rc;
    GemmGrouped g;
    g.out = out, g.ldo = ldo, g.N = N, g.K = K, g.k_blocks = (K + GG_K - 1) / GG_K, g.tile_expert = tile_expert, g.status = status, g.limit = limit;
    g.vec = ((uintptr_t)out % 16 == 0) && (ldo * (out_f32 ? 4 : 2)) % 16 == 0;
    cudaStream_t s = (cudaStream_t)stream;
    // Which way: what counts is how often the GPU has to be filled, SMs with a tile of 128 x 128 each or pairs of SMs with one of
    // 256 x 256, since a pair's turn takes about as long as an SM's, and the launch some four us more (as much as a turn where
    // K is short). us with single CTAs and with pairs: 4 experts, 1,024 rows in all, N = K = 512: 5.7 and 9.0 (one turn either
    // way); 8 experts, 2,048 rows, 768 x 1,024: 9.7 and 12.9 (one); 4 experts, 4,096 rows: 18 and 14 (two and one); 16 experts,
    // 6,400 rows, 2,432 x 2,560: 139 and 91. Which expert has how many rows is not known here: half a tile of padding an expert
    // is the usual, and since a pair has rows of one expert only, few rows an expert may leave it half empty (16 experts of 1,024 x
    // 768, 129 rows each on average: 15.8 and 13.8, but 16 and 19 where one expert has half of all rows).
    const long long sms = abk_sm_count(), used = max_tiles - experts, row_tiles = used + experts / 2;
    const long long turns = (row_tiles * ((N + GG_BN - 1) / GG_BN) + sms - 1) / sms;
    const long long pair_turns = ((row_tiles > 2 * experts ? row_tiles : 2 * experts) * ((N + GP_BN - 1) / GP_BN) + sms - 1) / sms;
    const bool takes = N >= GP_BN && max_tiles <= GP_MAX_TILES;
    const bool wins = (2 * used >= 3 * experts || (used >= experts && (long long)N * K >= 4 << 20)) && pair_turns + (K < 512) < turns;
    if (in_pairs > 0 && !takes) ABK_REFUSE("gemm_grouped: pairs of CTAs take %d and more columns and up to %d row tiles", GP_BN, GP_MAX_TILES);
    if (takes && (in_pairs < 0 ? wins : in_pairs > 0)) {
        const int pairs = abk_sm_count() / 2;
#define GP_LAUNCH(TO, ACT)                                                                                                         \
    do {                                                                                                                           \
        if (cudaError_t e = abk_allow_shared_memory((const void *)gemm_grouped_pair_kernel<TO, ACT>, GroupedPairSmem::BYTES))      \
            return (int)e;                                                                                                         \
        abk_launch_clusters(gemm_grouped_pair_kernel<TO, ACT>, dim3(2 * pairs), dim3(GG_THREADS), (size_t)GroupedPairSmem::BYTES, s, 2, mx, mw, g, max_tiles); \
    } while (0)
        if (out_f32) { if (activation) GP_LAUNCH(float, 1); else GP_LAUNCH(float, 0); }
        else if (activation == GG_CLAMPED_GATED) GP_LAUNCH(__nv_bfloat16, GG_CLAMPED_GATED);
        else if (activation == GG_SILU_GATED) GP_LAUNCH(__nv_bfloat16, GG_SILU_GATED);
        else { if (activation) GP_LAUNCH(__nv_bfloat16, 1); else GP_LAUNCH(__nv_bfloat16, 0); }
#undef GP_LAUNCH
        return ABK_LAUNCH_RESULT();
    }
    dim3 grid(max_tiles, (N + GG_BN - 1) / GG_BN);
    if (grid.y > 65535) ABK_REFUSE("gemm_grouped: %d output features are more than a grid takes", N);
#define GG_LAUNCH(TO, ACT)                                                                                          \
    do {                                                                                                            \
        if (cudaError_t e = abk_allow_shared_memory((const void *)gemm_grouped_kernel<TO, ACT>, GroupedSmem::BYTES)) \
            return (int)e;                                                                                          \
        abk_launch(gemm_grouped_kernel<TO, ACT>, grid, dim3(GG_THREADS), (size_t)GroupedSmem::BYTES, s, mx, mw, g); \
    } while (0)
    if (out_f32) { if (activation) GG_LAUNCH(float, 1); else GG_LAUNCH(float, 0); }
    else if (activation == GG_CLAMPED_GATED) GG_LAUNCH(__nv_bfloat16, GG_CLAMPED_GATED);
    else if (activation == GG_SILU_GATED) GG_LAUNCH(__nv_bfloat16, GG_SILU_GATED);
    else { if (activation) GG_LAUNCH(__nv_bfloat16, 1); else GG_LAUNCH(__nv_bfloat16, 0); }
#undef GG_LAUNCH
    return ABK_LAUNCH_RESULT();
}

// ---------------------------------------------------------------- back to the tokens' order
// A CTA a token; VEC: four columns a thread as one 16-byte piece (d a multiple of 4).
template <bool VEC>
__global__ void __launch_bounds__(256) moe_unsort_kernel(const float *sorted, const int *place, float *out, int d, int top, int add) {
    pdl_wait();
    const long long t = blockIdx.x;
    constexpr int W = VEC ? 4 : 1;
    for (int j = threadIdx.x * W; j < d; j += 256 * W) {
        float acc[W];
        bool any = false;
        for (int k = 0; k < top; k++) {
            const int at = place[t * top + k];
            if (at < 0) continue;
            float v[W];
            if (VEC) {
                const float4 r = *(const float4 *)(sorted + (long long)at * d + j);
                v[0] = r.x, v[W > 1 ? 1 : 0] = r.y, v[W > 2 ? 2 : 0] = r.z, v[W > 3 ? 3 : 0] = r.w;
            } else {
                v[0] = sorted[(long long)at * d + j];
            }
#pragma unroll
            for (int u = 0; u < W; u++) acc[u] = any ? acc[u] + v[u] : v[u];
            any = true;
        }
#pragma unroll
        for (int u = 0; u < W; u++) {
            const float a = any ? acc[u] : 0.0f;
            out[t * d + j + u] = add ? out[t * d + j + u] + a : a;
        }
    }
}

extern "C" int abk_moe_unsort(const float *sorted, const int *place, float *out, int n_tokens, int d, int top, int add,
                              void *stream) {
    if (n_tokens <= 0 || d <= 0) return 0;
    if (d % 4 == 0 && (((uintptr_t)sorted | (uintptr_t)out) & 15) == 0)
        abk_launch(moe_unsort_kernel<true>, dim3(n_tokens), dim3(256), 0, (cudaStream_t)stream, sorted, place, out, d, top, add);
    else
        abk_launch(moe_unsort_kernel<false>, dim3(n_tokens), dim3(256), 0, (cudaStream_t)stream, sorted, place, out, d, top, add);
    return ABK_LAUNCH_RESULT();
}
