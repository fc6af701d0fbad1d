// out[M, N] = x[M, K] . w[N, K]^T of float32 operands on the tensor cores, with errors below those of eight float32 sums.
//
// A float32 number is the sum of three bfloat16 numbers (8 + 8 + 8 bits, each rounded to nearest: what is left over is below
// 2^-26 of it), x = x1 + x2 + x3, so x w is the six products x1 w1, x1 w2, x2 w1, x2 w2, x1 w3, x3 w1; the three left out are
// below 2^-26. The tensor cores multiply bfloat16 without rounding and add in float32, but cut a sum off where float32
// rounds it, and a sum over a long K cut off at every step of 16 drifts towards zero. So x1 w1 is added up in tensor memory over a few
// steps only; these short sums are added in registers, rounded. The five small products have an accumulator of their own, whose
// cuts are 2^-8 as large.
//
// Errors against 64 bits (2-norm, in units of 1e-8; K = 512, 768, 1024, 2048, 3072, 9728) with sums over 16, 32 and 64 of K, and of the eight
// rounded sums on the CUDA cores:
//     numbers of either sign   16: 7.5 8.2 9.0 11.6 13.7 23.3   32: 7.4 7.9 8.4  9.9 11.2 17.5   64: 8.6 8.9 9.1 9.9 10.6 14.5   15.2 18.3 20.9 29.1 35.5 62.5
//     their magnitudes         16: 5.1 4.8 5.5  6.2  6.0 10.2   32: 5.9 5.6 6.0  6.4  6.0  8.5   64: 9.0 8.8 9.0 9.0  8.8  9.8    5.9  6.0  7.4  9.6  9.9 18.8
// (numbers of one sign: the cuts all go one way, 1.6, 3.7 and 7.7e-8 too small, and 17e-8 with sums over 128). So the short sums grow with K, as
// the CUDA cores' errors do: over 16 below K = 1024, over 32 below 2048, else over 64, below the CUDA cores' in every one of these.
//
// An element is the sum of four running sums, over the quarters of K in order: ((q0 + q1) + q2) + q3, each over its short sums in
// order, then its small products. That order goes by K alone: a row's result does not depend on how many other rows
// are in the batch, whether a pair of CTAs walks all of K or a quarter, or where its tile lies.
// bfloat16 operands (those that the tensor-core product proper refuses: rows that start anywhere) have one part. Their eight sums on the CUDA
// cores lose less, a product being exact there too, so below K = 2048 their short sums, over 16 and from 1024 on over 32, are added in one running
// sum with what each addition rounds off beside it (Knuth's two-sum), added at the end; from there on they go as float32 ones, over 32. Errors of
// this and of the CUDA cores, K = 512, 1024, 2048, 3072: magnitudes 3.2 4.7 6.2 5.9 and 4.5 5.2 6.8 6.9e-8, either sign 3.5 4.6 9.5 10.9 and 6.9 8.7 11.7
// 14.4e-8. 2048 x 1024 x 1020 in 68 us, 273 x 686 x 2768 in 21 (the CUDA cores 148 and 76; two-sums over 16 at every K 68 and 89).
// A number that is not finite makes its products NaN in this form, and one below 1e-33 keeps fewer digits (its third part is too small for
// bfloat16): an element that came out not finite, or below 2^-96 but not zero, is taken again with the CUDA cores' eight sums, a tile at a time and
// behind all waits, so that no wait runs out meanwhile: 2000 x 6144 x 1024 in 170 us, with one row of NaN 400, with nothing but NaN 3,600 (the CUDA
// cores 691). What is left: factors below 1e-33 whose partners are beyond 2^14, so that the element is not small.
//
// What bounds it: the chain between the tensor cores and the warps that add up (0.3 us a short sum), and the way of the parts from
// the L2, 6 bytes a number, at some 30 bytes a cycle and SM (500 x 6144 x 1024 in 62 us, 9 of them for the parts; sums over 128 53, the CUDA
// cores 197; 4000 x 6144 x 1024 in 305 us, 253, 1,349). The adding warps report to their own CTA's barrier and the pair's idle warp passes
// that on: 16 warps' words to the other CTA's barrier, one by one, took 72 us for 63.
//
// Two kernels: one writes the operands' parts as three planes of bfloat16 each, the other multiplies them on pairs of CTAs. (As one kernel
// that splits what it fetches, weights again for every column of tiles: 500 x 6144 x 1024 in 71 us, bound by the instructions
// of the splitting and by the way of plain loads through what the stages leave of the L1.)
#pragma once
#include "bf16_parts.cuh"
#include "recurrence.cuh"
#include "tc_common.cuh"
#include "tensor_map.cuh"
#include <float.h>

#define GP_ADDERS 16                      // warps that add up what the tensor cores leave
#define GP_THREADS (32 * GP_ADDERS + 64)  // one that loads, one that multiplies
#define GP_ROWS 128                       // weight rows of a CTA: the accumulators' lanes
#define GP_K 64                           // of K at a time
#define GP_QUARTERS 4

// BN: rows of x in a tile of a pair of CTAs; each brings half of them.
template <int BN> struct GpShape {
    static constexpr int STAGES = 3, X_ROWS = BN / 2;
    static constexpr int W_PLANE = GP_ROWS * GP_K * 2, X_PLANE = X_ROWS * GP_K * 2, STAGE = 3 * (W_PLANE + X_PLANE);
    static constexpr int BYTES = STAGES * STAGE + 1024 /* alignment */ + 256 /* barriers */;
    // accumulators of x1 w1 (three or four in turn where they fit: 63.3 -> 62.4 us with tiles of 96; two with 128: 65.4 against 70.0)
    // and two of the small products
    static constexpr int SUMS = BN == 128 ? 2 : BN == 96 ? 3 : 4, SMALLS = 2, ACCUMULATORS = SUMS + SMALLS;
    static constexpr int TMEM = BN == 32 ? 256 : 512;
    static_assert(ACCUMULATORS * BN <= TMEM, "the accumulators fill tensor memory");
    static constexpr int COLS = BN / 4;                   // of the accumulator that a warp adds up
};

template <int N> __device__ __forceinline__ void gp_tmem_ld(uint32_t taddr, uint32_t *v);
template <> __device__ __forceinline__ void gp_tmem_ld<8>(uint32_t taddr, uint32_t *v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(taddr));
}

// ------------------------------------------------------------------ the parts of the operands
// Rows of `k` numbers, `ld` apart, as planes [rows][pitch] of bfloat16 (pitch: k up to a multiple of 8): three of float32 numbers, one of
// bfloat16 ones, which only get rows that TMA takes.
struct SplitRows {
    const void *from;
    __nv_bfloat16 *to;
    long long ld;
    int rows, vec;  // vec: the rows start on 16-byte boundaries, float32 ones of a multiple of four numbers
};
// Bound by memory: 4 bytes read and 6 written a number (6,644 rows of 1,024: 8.9 us). A thread has eight numbers of a row.
template <typename T> __global__ void __launch_bounds__(256) gemm_split_rows_kernel(SplitRows a, SplitRows b, int k, int pitch) {
    const int pieces = pitch / 8;
    pdl_wait();
    const long long na = (long long)a.rows * pieces, n = na + (long long)b.rows * pieces;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n; i += (long long)gridDim.x * 256) {
        const bool first = i < na;
        const SplitRows &o = first ? a : b;
        const long long j = first ? i : i - na, row = j / pieces;
        const int c = (int)(j - row * pieces) * 8;
        const T *from = (const T *)o.from + row * o.ld + c;
        __nv_bfloat16 *to = o.to + row * pitch + c;
        T v[8];
        if (sizeof(T) == 4 && o.vec) {
            *(float4 *)v = *(const float4 *)from;
            *(float4 *)(v + 4) = c + 4 < k ? *(const float4 *)(from + 4) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        } else {
#pragma unroll
            for (int e = 0; e < 8; e++) v[e] = c + e < k ? from[e] : from_float<T>(0.0f);
        }
        if constexpr (sizeof(T) == 4) {
            uint4 p1, p2, p3;
            split_pair(v[0], v[1], p1.x, p2.x, p3.x), split_pair(v[2], v[3], p1.y, p2.y, p3.y);
            split_pair(v[4], v[5], p1.z, p2.z, p3.z), split_pair(v[6], v[7], p1.w, p2.w, p3.w);
            const long long plane = (long long)o.rows * pitch;
            *(uint4 *)to = p1, *(uint4 *)(to + plane) = p2, *(uint4 *)(to + 2 * plane) = p3;
        } else {
            uint32_t word[4];
#pragma unroll
            for (int e = 0; e < 8; e += 2) {
                const __nv_bfloat162 two = __halves2bfloat162(v[e], v[e + 1]);
                word[e / 2] = *(const uint32_t *)&two;
            }
            *(uint4 *)to = make_uint4(word[0], word[1], word[2], word[3]);
        }
    }
}

// ------------------------------------------------------------------ the product
struct GemmSplit {
    const void *x, *w;
    void *out;
    int dtype, out_dtype;  // of x and w, ABK_F32 or ABK_BF16; of out
    int M, N, K, m_tiles, tiles;
    long long ldx, ldw, ldo;
    int *status;
    float *quarters;  // [GP_QUARTERS][M][N]
};

__device__ __forceinline__ void gp_put(const GemmSplit &g, int m, int n, float v) {
    if (g.out_dtype == ABK_F32) ((float *)g.out)[m * g.ldo + n] = v;
    else ((__nv_bfloat16 *)g.out)[m * g.ldo + n] = __float2bfloat16_rn(v);
}
__device__ __forceinline__ float gp_stored(const GemmSplit &g, int m, int n) {
    if (g.out_dtype == ABK_F32) return __ldcg((const float *)g.out + m * g.ldo + n);
    return __bfloat162float(__ldcg((const __nv_bfloat16 *)g.out + m * g.ldo + n));
}
// Whether a sum has to be taken again.
__device__ __forceinline__ bool gp_again(float v) { return !(fabsf(v) >= 0x1p-96f && fabsf(v) <= FLT_MAX) && v != 0.0f; }

// The elements of a tile of THREADS / 16 rows of x from m0 on and 128 rows of w from n0 on that have to be taken again, as gemm_simt.cu adds
// them up: eight sums, pieces of 16 of K, piece c to sum c % 8, in ascending order, then in pairs (up to K = 256 one sum). All threads of
// the CTA call it and THREADS of them work, one for a row of w and eight rows of x; bad: bit j for the thread's j-th. smem: GP_REDO_FLOATS.
#define GP_REDO_PITCH 20  // (eight rows' runs of four numbers lie in different banks)
#define GP_REDO_FLOATS(THREADS) ((128 + (THREADS) / 16) * GP_REDO_PITCH)
template <typename T, int THREADS> __device__ __forceinline__ void gp_redo(const GemmSplit &g, int m0, int n0, uint32_t bad, float *smem) {
    const int tid = threadIdx.x, n = tid & 127, row = tid / 128 * 8, sums = g.K <= 256 ? 1 : 8, pieces = (g.K + 15) / 16;
    const float *const ws = smem + n * GP_REDO_PITCH, *const xs = smem + (128 + row) * GP_REDO_PITCH;
    constexpr int MINE = (128 + THREADS / 16) * 16 / THREADS;  // numbers of a piece that a thread brings: asked for while the one before is multiplied
    float a[8], b[8], c[8], sum[8], next[MINE];
    auto ask = [&](int piece) {
        if (tid >= THREADS) return;
#pragma unroll
        for (int i = 0; i < MINE; i++) {
            const int e = tid + i * THREADS, r = e / 16, k = piece * 16 + e % 16;
            const bool of_w = r < 128, real = k < g.K && (of_w ? n0 + r < g.N : m0 + r - 128 < g.M);
            const T *from = of_w ? (const T *)g.w + (n0 + r) * g.ldw : (const T *)g.x + (m0 + r - 128) * g.ldx;
            next[i] = real ? to_float(from[k]) : 0.0f;
        }
    };
    for (int s = 0; s < sums; s++) {
#pragma unroll
        for (int j = 0; j < 8; j++) sum[j] = 0.0f;
        ask(s);
        for (int piece = s; piece < pieces; piece += sums) {
            __syncthreads();
            if (tid < THREADS) {
#pragma unroll
                for (int i = 0; i < MINE; i++) smem[(tid + i * THREADS) / 16 * GP_REDO_PITCH + (tid + i * THREADS) % 16] = next[i];
            }
            __syncthreads();
            if (piece + sums < pieces) ask(piece + sums);
            if (tid < THREADS) {
#pragma unroll
                for (int k = 0; k < 16; k += 4) {
                    const float4 v = *(const float4 *)(ws + k);
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        const float4 u = *(const float4 *)(xs + j * GP_REDO_PITCH + k);
                        sum[j] = fmaf(u.w, v.w, fmaf(u.z, v.z, fmaf(u.y, v.y, fmaf(u.x, v.x, sum[j]))));
                    }
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 8; j++) {  // ((s0 + s1) + (s2 + s3)) + ((s4 + s5) + (s6 + s7))
            if (s == 0) a[j] = sum[j];
            else if (s == 1) a[j] += sum[j];
            else if (s == 2 || s == 4) b[j] = sum[j];
            else if (s == 3) a[j] += b[j] + sum[j];
            else if (s == 5) b[j] += sum[j];
            else if (s == 6) c[j] = sum[j];
            else a[j] += b[j] + (c[j] + sum[j]);
        }
    }
    __syncthreads();  // (the next tile is staged in the same place)
    if (tid < THREADS)
#pragma unroll
        for (int j = 0; j < 8; j++)
            if (bad >> j & 1) gp_put(g, m0 + row + j, n0 + n, a[j]);
}

// The same for the tiles of a pair's CTA (item pair, pair + pairs, ...).
template <typename T, int BN> __device__ __noinline__ void gp_redo_items(const GemmSplit &g, int pair, int pairs, int items, int half, float *smem) {
    constexpr int THREADS = 32 * GP_ADDERS, ROWS = THREADS / 16;
    for (int item = pair; item < items; item += pairs) {
        const int m_end = min((item % g.m_tiles + 1) * BN, g.M), n0 = (item / g.m_tiles * 2 + half) * GP_ROWS, n = n0 + (threadIdx.x & 127);
        for (int m0 = item % g.m_tiles * BN; m0 < m_end; m0 += ROWS) {
            uint32_t bad = 0;
            if (threadIdx.x < THREADS && n < g.N)
                for (int j = 0, m = m0 + threadIdx.x / 128 * 8; j < 8 && m < m_end; j++, m++) bad |= (uint32_t)gp_again(gp_stored(g, m, n)) << j;
            if (__syncthreads_or(bad)) gp_redo<T, THREADS>(g, m0, n0, bad, smem);
        }
    }
}

template <int PARTS> struct GpOperand { typedef float T; };
template <> struct GpOperand<1> { typedef __nv_bfloat16 T; };

// A tile is 256 rows of w (128 of each CTA) and BN rows of x; pair c of CTAs takes items c, c + pairs, ... An item is a tile, or
// (QUARTERS) a quarter of K of one, whose sums go to `quarters` and are added up by the kernel behind.
// map_w, map_x: the planes, one below the other; PARTS: 3 of float32 operands, 1 of bfloat16 ones; STEPS: of 16 of K in a
// short sum, 1, 2 or 4; TWO_SUM: one running sum of all, with what its additions round off.
template <int BN, bool QUARTERS, int PARTS, int STEPS, bool TWO_SUM> __global__ void __launch_bounds__(GP_THREADS, 1) gemm_split_kernel(const __grid_constant__ CUtensorMap map_w,
                                                                                               const __grid_constant__ CUtensorMap map_x, const __grid_constant__ GemmSplit g) {
    using S = GpShape<BN>;
    constexpr int STAGES = S::STAGES, COLS = S::COLS, SUMS = S::SUMS, SMALLS = S::SMALLS;
    extern __shared__ uint8_t gp_smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)gp_smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t *full = (uint64_t *)(smem + STAGES * S::STAGE), *empty = full + STAGES;
    uint64_t *sum_ready = empty + STAGES, *sum_free = sum_ready + SUMS, *small_free = sum_free + SUMS;
    uint32_t *tmem_holder = (uint32_t *)(small_free + SMALLS);
    volatile int *gave_up = (volatile int *)(tmem_holder + 1), *again = gave_up + 1;  // again: some element has to be taken again
    typedef typename GpOperand<PARTS>::T T;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t half = tc::cluster_rank();  // 0: the leader
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) tc::mbar_init(&full[s], 1), tc::mbar_init(&empty[s], 1);
        // sum_free, small_free: every adding warp of the CTA, and, on the leader's, the peer's word that all of its own have
        for (int b = 0; b < SUMS; b++) tc::mbar_init(&sum_ready[b], 1), tc::mbar_init(&sum_free[b], GP_ADDERS + (half == 0));
        for (int b = 0; b < SMALLS; b++) tc::mbar_init(&small_free[b], GP_ADDERS + (half == 0));
        *gave_up = *again = 0;
        tc::mbar_init_fence();
        tc::tma_prefetch_map(&map_w), tc::tma_prefetch_map(&map_x);
    }
    if (warp == GP_ADDERS) tc::tmem_alloc_pair(tmem_holder, S::TMEM);
    tc::fence_before_sync();
    tc::cluster_sync();
    tc::fence_after_sync();
    const uint32_t tmem = *tmem_holder;

    const int pieces = (g.K + GP_K - 1) / GP_K;
    constexpr int sums_a_piece = GP_K / 16 / STEPS;
    const int items = QUARTERS ? g.tiles * GP_QUARTERS : g.tiles, pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const auto first_quarter = [&](int item) { return QUARTERS ? item / g.tiles : 0; };
    const auto last_quarter = [&](int item) { return QUARTERS ? item / g.tiles : GP_QUARTERS - 1; };
    const auto tile_of = [&](int item) { return QUARTERS ? item % g.tiles : item; };
    const auto begin_of = [&](int quarter) { return (int)((long long)pieces * quarter / GP_QUARTERS); };
    if (warp == GP_ADDERS) {
        if (lane == 0) {
            pdl_wait();
            int i = 0;
            bool ok = true;
            for (int item = pair; ok && item < items; item += pairs) {
                const int tile = tile_of(item), m0 = tile % g.m_tiles * BN + half * S::X_ROWS, n0 = (tile / g.m_tiles * 2 + half) * GP_ROWS;
                const int end = begin_of(last_quarter(item) + 1);
                for (int p = begin_of(first_quarter(item)); p < end; p++, i++) {
                    const int s = i % STAGES;
                    if (i >= STAGES && !tc::mbar_wait(&empty[s], ((i / STAGES) & 1) ^ 1)) {
                        ok = false;
                        break;
                    }
                    if (half == 0) tc::mbar_expect_tx(&full[s], PARTS * 2 * (S::W_PLANE + S::X_PLANE));  // both CTAs' copies report to the leader
                    const uint32_t bar = tc::peer_smem(tc::smem_addr(&full[s]), 0);
                    uint8_t *stage = smem + s * S::STAGE;
                    for (int t = 0; t < PARTS; t++) {
                        tc::tma_load_2d_pair(stage + t * S::W_PLANE, &map_w, p * GP_K, t * g.N + n0, bar);
                        tc::tma_load_2d_pair(stage + 3 * S::W_PLANE + t * S::X_PLANE, &map_x, p * GP_K, t * g.M + m0, bar);
                    }
                }
            }
            if (!ok) *gave_up = 1;
        }
        __syncwarp();
    } else if (warp == GP_ADDERS + 1) {
        if (lane == 0 && half == 0) {
            constexpr uint32_t idesc = tc::idesc_bf16_f32(2 * GP_ROWS, BN);
            int i = 0, sum_i = 0, quarter_i = 0;  // pieces, short sums and quarters so far
            bool ok = true;
            for (int item = pair; ok && item < items; item += pairs) {
                for (int q = first_quarter(item); ok && q <= last_quarter(item); q++, quarter_i++) {
                    const int q_begin = begin_of(q), q_end = begin_of(q + 1);
                    const uint32_t small = tmem + (SUMS + quarter_i % SMALLS) * BN;
                    if (PARTS == 3) ok = quarter_i < SMALLS || tc::mbar_wait(&small_free[quarter_i % SMALLS], ((quarter_i / SMALLS) & 1) ^ 1);
                    for (int p = q_begin; ok && p < q_end; p++, i++) {
                        const int s = i % STAGES;
                        if (!(ok = tc::mbar_wait(&full[s], (i / STAGES) & 1))) break;
                        tc::fence_after_sync();
                        const uint32_t at = tc::smem_addr(smem + s * S::STAGE);
                        const uint64_t w1 = tc::smem_desc_k_sw128(at), w2 = w1 + (S::W_PLANE >> 4), w3 = w2 + (S::W_PLANE >> 4);
                        const uint64_t x1 = w3 + (S::W_PLANE >> 4), x2 = x1 + (S::X_PLANE >> 4), x3 = x2 + (S::X_PLANE >> 4);
#pragma unroll
                        for (int k0 = 0; k0 < GP_K / 16; k0 += STEPS) {  // (16 of K: 32 bytes of a row)
                            const int b = sum_i % SUMS;
#pragma unroll
                            for (int k = k0; k < k0 + STEPS; k++) {
                                if (PARTS == 1) continue;  // (ahead of the wait: they keep the tensor cores busy while a sum is read)
                                tc::mma_ss_pair(small, w1 + 2 * k, x2 + 2 * k, idesc, p > q_begin || k > 0);
                                tc::mma_ss_pair(small, w2 + 2 * k, x1 + 2 * k, idesc, true);
                                tc::mma_ss_pair(small, w2 + 2 * k, x2 + 2 * k, idesc, true);
                                tc::mma_ss_pair(small, w1 + 2 * k, x3 + 2 * k, idesc, true);
                                tc::mma_ss_pair(small, w3 + 2 * k, x1 + 2 * k, idesc, true);
                            }
                            if (!(ok = sum_i < SUMS || tc::mbar_wait(&sum_free[b], ((sum_i / SUMS) & 1) ^ 1))) break;
                            tc::fence_after_sync();
#pragma unroll
                            for (int k = k0; k < k0 + STEPS; k++) tc::mma_ss_pair(tmem + b * BN, w1 + 2 * k, x1 + 2 * k, idesc, k > k0);
                            tc::mma_commit_pair(&sum_ready[b]), sum_i++;
                        }
                        if (ok) tc::mma_commit_pair(&empty[s]);
                    }
                }
            }
            if (!ok) *gave_up = 1;
        } else if (lane == 0) {  // the peer: what its adding warps have read, passed on to the leader
            int sum_i = 0, quarter_i = 0;
            bool ok = true;
            for (int item = pair; ok && item < items; item += pairs) {
                for (int q = first_quarter(item); ok && q <= last_quarter(item); q++, quarter_i++) {
                    const int sums = (begin_of(q + 1) - begin_of(q)) * sums_a_piece;
                    for (int n = 0; ok && n < sums; n++, sum_i++) {
                        ok = tc::mbar_wait(&sum_free[sum_i % SUMS], (sum_i / SUMS) & 1);
                        if (ok) tc::mbar_arrive_in_cluster(tc::peer_smem(tc::smem_addr(&sum_free[sum_i % SUMS]), 0));
                    }
                    if (PARTS == 3) ok = ok && tc::mbar_wait(&small_free[quarter_i % SMALLS], (quarter_i / SMALLS) & 1);
                    if (PARTS == 3 && ok) tc::mbar_arrive_in_cluster(tc::peer_smem(tc::smem_addr(&small_free[quarter_i % SMALLS]), 0));
                }
            }
            if (!ok) *gave_up = 1;
        }
        __syncwarp();
    } else {
        pdl_wait();
        // a warp has a quarter of the lanes (the weights' rows) and COLS columns (rows of x) of the accumulators
        const int lane_base = (warp & 3) * 32, col0 = (warp >> 2) * COLS;
        const uint32_t taddr = tmem + ((uint32_t)lane_base << 16) + col0;
        float sum[COLS], total[COLS];  // of the quarter, of those before; TWO_SUM: of all, and what its additions rounded off
        const f32x2 minus = pack2(-1.0f, -1.0f);
#pragma unroll
        for (int j = 0; j < COLS; j++) sum[j] = total[j] = 0.0f;
        int sum_i = 0, quarter_i = 0;
        bool ok = true, redo = false;
#pragma unroll 1
        for (int item = pair; ok && item < items; item += pairs) {
#pragma unroll 1
            for (int q = first_quarter(item); q <= last_quarter(item); q++, quarter_i++) {
                const int sums = (begin_of(q + 1) - begin_of(q)) * sums_a_piece;
#pragma unroll 1
                for (int n = 0; n < sums; n++, sum_i++) {
                    const int b = sum_i % SUMS;
                    ok = __all_sync(0xffffffffu, ok && tc::mbar_wait(&sum_ready[b], (sum_i / SUMS) & 1));
                    tc::fence_after_sync();
                    uint32_t v[8];
#pragma unroll
                    for (int c = 0; c < COLS; c += 8) {
                        gp_tmem_ld<8>(taddr + b * BN + c, v);
                        tc::tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 8; j += 2) {
                            float *const s2 = sum + c + j, *const t2 = total + c + j;
                            if constexpr (!TWO_SUM) {
                                s2[0] += __uint_as_float(v[j]), s2[1] += __uint_as_float(v[j + 1]);
                            } else {
                                const f32x2 a = pack2(s2[0], s2[1]), b2 = pack2(__uint_as_float(v[j]), __uint_as_float(v[j + 1]));
                                const f32x2 both = add2(a, b2), of_b = fma2(a, minus, both), of_a = fma2(of_b, minus, both);
                                const float2 r = unpack2(both), lost = unpack2(add2(pack2(t2[0], t2[1]), add2(fma2(of_a, minus, a), fma2(of_b, minus, b2))));
                                s2[0] = r.x, s2[1] = r.y, t2[0] = lost.x, t2[1] = lost.y;
                            }
                        }
                    }
                    if (!TWO_SUM && n + 1 == sums) {
#pragma unroll
                        for (int c = 0; c < COLS; c += 8) {
                            if constexpr (PARTS == 3) {
                                gp_tmem_ld<8>(taddr + (SUMS + quarter_i % SMALLS) * BN + c, v);
                                tc::tmem_ld_wait();
                            }
#pragma unroll
                            for (int j = 0; j < 8; j++) total[c + j] += PARTS == 3 ? sum[c + j] + __uint_as_float(v[j]) : sum[c + j], sum[c + j] = 0.0f;
                        }
                    }
                    tc::fence_before_sync();
                    __syncwarp();
                    if (lane == 0) {
                        tc::mbar_arrive(&sum_free[b]);
                        if (PARTS == 3 && n + 1 == sums) tc::mbar_arrive(&small_free[quarter_i % SMALLS]);
                    }
                }
            }
            if (ok) {
                const int tile = tile_of(item), m0 = tile % g.m_tiles * BN + col0, n = (tile / g.m_tiles * 2 + half) * GP_ROWS + lane_base + lane;
                const int cols = n < g.N ? g.M - m0 : 0;
                if constexpr (QUARTERS) {
                    float *out = g.quarters + ((long long)first_quarter(item) * g.M + m0) * g.N + n;
#pragma unroll
                    for (int j = 0; j < COLS; j++)
                        if (j < cols) out[(long long)j * g.N] = total[j];
                } else {
#pragma unroll
                    for (int j = 0; j < COLS; j++)
                        if (j < cols) {
                            const float v = TWO_SUM ? sum[j] + total[j] : total[j];
                            gp_put(g, m0 + j, n, v), redo |= gp_again(v);
                        }
                }
#pragma unroll
                for (int j = 0; j < COLS; j++) sum[j] = total[j] = 0.0f;
            }
        }
        if (!ok) *gave_up = 1;
        if (redo) *again = 1;
    }
    tc::fence_before_sync();
    tc::cluster_sync();  // (the pair's other CTA is done with this one's memory and barriers)
    if (*gave_up && threadIdx.x == 0) atomicOr(g.status + 1, 1);
    if (warp == GP_ADDERS) {
        tc::fence_after_sync();
        tc::tmem_free_pair(tmem, S::TMEM);
    }
    if (!QUARTERS && *again && !*gave_up) gp_redo_items<T, BN>(g, pair, pairs, items, half, (float *)smem);
}

// The four quarters' sums of every element, in order: a CTA has tiles of 16 rows and 128 columns, a thread a column and eight rows.
#define GP_SUM_THREADS 256
template <typename T> __global__ void __launch_bounds__(GP_SUM_THREADS) gemm_split_sum_kernel(const __grid_constant__ GemmSplit g) {  // T: of the operands
    __shared__ __align__(16) float smem[GP_REDO_FLOATS(GP_SUM_THREADS)];
    constexpr int ROWS = GP_SUM_THREADS / 16;
    const long long plane = (long long)g.M * g.N;
    const int m_tiles = (g.M + ROWS - 1) / ROWS, tiles = m_tiles * ((g.N + 127) / 128);
    pdl_wait();
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int m0 = tile % m_tiles * ROWS, n0 = tile / m_tiles * 128, m = m0 + threadIdx.x / 128 * 8, n = n0 + (threadIdx.x & 127);
        float q[8][GP_QUARTERS];
#pragma unroll
        for (int j = 0; j < 8; j++)
#pragma unroll
            for (int i = 0; i < GP_QUARTERS; i++) q[j][i] = m + j < g.M && n < g.N ? g.quarters[i * plane + (long long)(m + j) * g.N + n] : 0.0f;
        uint32_t bad = 0;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const float v = ((q[j][0] + q[j][1]) + q[j][2]) + q[j][3];
            if (m + j < g.M && n < g.N) gp_put(g, m + j, n, v), bad |= (uint32_t)gp_again(v) << j;
        }
        if (__syncthreads_or(bad)) gp_redo<T, GP_SUM_THREADS>(g, m0, n0, bad, smem);
    }
}

template <int BN, bool QUARTERS, int PARTS, int STEPS, bool TWO_SUM = false> static int gemm_split_launch(const CUtensorMap &map_w, const CUtensorMap &map_x, GemmSplit g, cudaStream_t s) {
    using S = GpShape<BN>;
    const cudaError_t e = abk_allow_shared_memory((const void *)gemm_split_kernel<BN, QUARTERS, PARTS, STEPS, TWO_SUM>, S::BYTES);
    if (e != cudaSuccess) return (int)e;
    const int pairs = abk_sm_count() / 2, items = QUARTERS ? g.tiles * GP_QUARTERS : g.tiles;
    abk_launch_clusters(gemm_split_kernel<BN, QUARTERS, PARTS, STEPS, TWO_SUM>, dim3(2 * (items < pairs ? items : pairs)), dim3(GP_THREADS), S::BYTES, s, 2, map_w, map_x, g);
    const int rc = ABK_LAUNCH_RESULT();
    if (rc || !QUARTERS) return rc;
    const long long blocks = ((long long)g.M + 15) / 16 * ((g.N + 127) / 128), most = 8LL * abk_sm_count();
    abk_launch(gemm_split_sum_kernel<typename GpOperand<PARTS>::T>, dim3((unsigned)(blocks < most ? blocks : most)), dim3(GP_SUM_THREADS), 0, s, g);
    return ABK_LAUNCH_RESULT();
}

#define GP_QUARTERS_BYTES (64LL << 20)  // sums of quarters in the scratch memory at most
static bool gp_may_quarter(int M, int N) { return 4LL * GP_QUARTERS * M * N <= GP_QUARTERS_BYTES; }

// Steps of 16 of K in a short sum, and whether bfloat16 operands are added up by two-sums.
static int gp_steps(int K, int parts) { return K < 1024 ? 1 : K < 2048 || parts == 1 ? 2 : 4; }
static bool gp_two_sum(int K, int parts) { return parts == 1 && K < 2048; }

// Rows of x in a tile, and whether pairs of CTAs take quarters of K: what takes least, by turns of the GPU's pairs times what a
// piece of 64 of K takes (measured with a turn each: 1.2 us for tiles of 32 rows, 1.25, 1.35, 1.5 for 128 with sums over 64, a fifth more
// over 32, half as much again over 16: the way from the L2 and the chain count for more than the products, 1,104 to 1,536 cycles), and the passes over the quarters'
// sums. 500 x 6144 x 1024 in tiles of 96: 62 us, of 128: 65, of 64: 81, in quarters 79; 500 x 1024 x 3072 in quarters with tiles of 128: 30 us, of
// 64: 41, whole: 63.
static void gp_choose(int M, int N, int K, int parts, bool may_quarter, int &bn, int &quarters) {
    static const struct { int bn; float us; } tile[4] = {{32, 1.2f}, {64, 1.25f}, {96, 1.35f}, {128, 1.5f}};
    const long long pairs = abk_sm_count() / 2;
    const float pieces = (float)((K + GP_K - 1) / GP_K) * (gp_steps(K, parts) == 4 ? 1.0f : gp_steps(K, parts) == 2 ? 1.2f : 1.6f);  // (in those of sums over 64)
    float best = 0.0f;
    bn = quarters = 0;
    for (const auto &t : tile) {
        if (gp_two_sum(K, parts) && t.bn == 128) continue;  // (not built: two numbers an output in registers)
        const long long tiles = ((long long)M + t.bn - 1) / t.bn * ((N + 2 * GP_ROWS - 1) / (2 * GP_ROWS));
        for (int q = 0; q < (may_quarter ? 2 : 1); q++) {
            const float us = q ? (float)((tiles * GP_QUARTERS + pairs - 1) / pairs) * pieces / GP_QUARTERS * t.us + 3.0f + (float)M * (float)N * 6.4e-6f
                               : (float)((tiles + pairs - 1) / pairs) * pieces * t.us;
            if (bn == 0 || us < best) best = us, bn = t.bn, quarters = q;
        }
    }
}

// The parts of this many numbers of an operand at most lie in the scratch memory at a time (96 MB); larger products go slab by slab.
#define GP_SLAB (16 << 20)
static int gp_slab_rows(int rows, int K, int multiple) {
    const int most = GP_SLAB / K / multiple * multiple;
    return rows < most ? rows : most > multiple ? most : multiple;
}
static long long gp_planes(int rows, int K) {  // bytes, up to a multiple of 1024
    return (3LL * rows * ((K + 7) / 8 * 8) * 2 + 1023) / 1024 * 1024;
}
static long long gemm_split_scratch(int M, int N, int K) {
    const int n_slab = gp_slab_rows(N, K, 256), m_slab = gp_slab_rows(M, K, 128);
    return gp_planes(n_slab, K) + gp_planes(m_slab, K) + (gp_may_quarter(m_slab, n_slab) ? 4LL * GP_QUARTERS * m_slab * n_slab : 0) + 1024;
}

// Kernels that gemm_split_run launches where the sizes choose the tile.
static int gemm_split_kernels(int M, int N, int K, int parts) {
    const int n_slab = gp_slab_rows(N, K, 256), m_slab = gp_slab_rows(M, K, 128);
    int kernels = 0, bn, quarters;
    for (int m = 0; m < M; m += m_slab)
        for (int n = 0; n < N; n += n_slab) {
            gp_choose(M - m < m_slab ? M - m : m_slab, N - n < n_slab ? N - n : n_slab, K, parts, !gp_two_sum(K, parts) && gp_may_quarter(m_slab, n_slab), bn, quarters);
            kernels += 2 + quarters;
        }
    return kernels;
}

// Where bn is 0 the sizes choose it and whether K is walked in quarters.
template <typename T> static int gemm_split_run(GemmSplit g, int bn, int quarters, void *scratch, cudaStream_t s) {
    const int pitch = (g.K + 7) / 8 * 8, n_slab = gp_slab_rows(g.N, g.K, 256), m_slab = gp_slab_rows(g.M, g.K, 128), M = g.M, N = g.N;
    constexpr int parts = sizeof(T) == 4 ? 3 : 1;
    if (g.K <= (GP_QUARTERS - 1) * GP_K) ABK_REFUSE("gemm: K = %d is too short for four quarters on the tensor cores", g.K);
    const int out_size = g.out_dtype == ABK_F32 ? 4 : 2;
    __nv_bfloat16 *const w_planes = (__nv_bfloat16 *)(((uintptr_t)scratch + 1023) & ~(uintptr_t)1023);
    __nv_bfloat16 *const x_planes = w_planes + gp_planes(n_slab, g.K) / 2;
    g.quarters = (float *)(x_planes + gp_planes(m_slab, g.K) / 2);
    const T *const x = (const T *)g.x, *const w = (const T *)g.w;
    char *const out = (char *)g.out;
    const bool may_quarter = !gp_two_sum(g.K, parts) && gp_may_quarter(m_slab, n_slab);
    const auto vec = [&](const T *from, long long ld) { return sizeof(T) == 4 && g.K % 4 == 0 && ld % 4 == 0 && !((uintptr_t)from & 15); };
    for (int m = 0; m < M; m += m_slab)
        for (int n = 0; n < N; n += n_slab) {
            g.M = M - m < m_slab ? M - m : m_slab, g.N = N - n < n_slab ? N - n : n_slab;
            g.x = x + m * g.ldx, g.w = w + n * g.ldw, g.out = out + (m * g.ldo + n) * out_size;
            const SplitRows rows_w = {g.w, w_planes, g.ldw, g.N, vec((const T *)g.w, g.ldw)};
            const SplitRows rows_x = {g.x, x_planes, g.ldx, n == 0 ? g.M : 0, vec((const T *)g.x, g.ldx)};
            const long long pieces = ((long long)rows_w.rows + rows_x.rows) * (pitch / 8), blocks = (pieces + 255) / 256, most = 16LL * abk_sm_count();
            abk_launch(gemm_split_rows_kernel<T>, dim3((unsigned)(blocks < most ? blocks : most)), dim3(256), 0, s, rows_w, rows_x, g.K, pitch);
            int rc = ABK_LAUNCH_RESULT();
            if (rc) return rc;
            int b = bn, in_quarters = quarters;
            if (!b) gp_choose(g.M, g.N, g.K, parts, may_quarter, b, in_quarters);
            if (in_quarters && !may_quarter) ABK_REFUSE("gemm: no room for the quarters of %d x %d sums", g.M, g.N);
            g.m_tiles = (g.M + b - 1) / b, g.tiles = g.m_tiles * ((g.N + 2 * GP_ROWS - 1) / (2 * GP_ROWS));
            const int steps = gp_steps(g.K, parts);
            CUtensorMap map_w, map_x;
            if ((rc = tmap::bf16_rows_of_128_bytes(w_planes, (long long)parts * g.N, g.K, pitch, GP_ROWS, &map_w))) return rc;
            if ((rc = tmap::bf16_rows_of_128_bytes(x_planes, (long long)parts * g.M, g.K, pitch, b / 2, &map_x))) return rc;
#define GP_AS(BN, STEPS) (in_quarters ? gemm_split_launch<BN, true, parts, STEPS>(map_w, map_x, g, s) : gemm_split_launch<BN, false, parts, STEPS>(map_w, map_x, g, s))
#define GP_CASE(BN)                                                                                                             \
    case BN:                                                                                                                    \
        if constexpr (parts == 3) rc = steps == 1 ? GP_AS(BN, 1) : steps == 2 ? GP_AS(BN, 2) : GP_AS(BN, 4);                    \
        else if (!gp_two_sum(g.K, parts)) rc = GP_AS(BN, 2);                                                                    \
        else if constexpr (BN < 128)                                                                                            \
            rc = steps == 1 ? gemm_split_launch<BN, false, 1, 1, true>(map_w, map_x, g, s) : gemm_split_launch<BN, false, 1, 2, true>(map_w, map_x, g, s); \
        else ABK_REFUSE("gemm: tiles of %d rows of bfloat16 numbers are not built for K = %d", BN, g.K);                        \
        break
            switch (b) {
                GP_CASE(32);
                GP_CASE(64);
                GP_CASE(96);
                GP_CASE(128);
                default: ABK_REFUSE("gemm: tiles of %d rows are not built", b);
            }
#undef GP_CASE
#undef GP_AS
            if (rc) return rc;
        }
    return 0;
}
