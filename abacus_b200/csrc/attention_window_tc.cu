// Causal attention of whole prompts with float32 softmax weights on the 5th-generation tensor cores (tcgen05): what
// attention_window.cu computes (a sliding window that also keeps a sequence's first keys, chunks, a sink, values of another
// size than keys; keys and values from the step's own rows), for heads of 64, 128 or 192, values of 64 or 128, no cap.
//
//   key j is seen from i when j <= i and (window == 0 or i - j < window or j < keep_first)
//                                    and (chunk == 0 or j / chunk == i / chunk)
//   p_j = exp(z_j - M) / (exp(sink - M) + sum_j exp(z_j - M)),  z_j = scale * (q . k_j),  out = sum_j p_j v_j
//
// A CTA has 256 query rows of one (sequence, head), two groups of 128, and walks the tiles of 64 keys any of them sees:
//   warp 0     TMA: the query tiles once, then a tile of keys and a tile of values per step into rings; both groups use
//              what comes in;
//   warp 1     issues tcgen05.mma: S = Q K^T of a group (128 x 64, into tensor memory), and O += P V with P from tensor
//              memory: the weights are float32, each as three bfloat16 parts that together hold its 24 bits (the value
//              rounded, the remainder rounded, the remainder of that), and the product is taken once with each;
//   warps 2-9  a thread a query row (four warps a group): reads its row of S, masks (only in tiles that some row does not
//              see whole), follows the row's maximum, and writes the three parts of the row's weights over its scores.
// While one group's rows are in the softmax the tensor cores work for the other. Bound by the softmax warps: 860 instructions a
// warp and tile (995 one weight at a time), two warps to a scheduler, where the products of both groups take 1,100 cycles (tensor pipe
// 31 % of active cycles). Two weights at a time need one multiply-add, sum or remainder for both and give the same bits. Measured one
// weight at a time: 3 prompts, 3,893 tokens, 32 query and 8 key heads of 128, a window of 1,024: 158 us (the warp-level kernel 377);
// 32 heads of 192 with values of 128, no window: 191 (506). Two at a time, the kernel alone in turns with the other: 155 -> 149 us and 190 ->
// 183; 16 query heads, one prompt of 2,048: 67.3 -> 64.1; 512 tokens, 16 heads of 192 with values of 64: 28.05 and 28.33. (The whole layers, with
// products and the host's step, change by less than their runs differ.) The pairs cost registers: the three instantiations
// for values of 64 spill 68 bytes a thread (3,893 tokens, 16 heads of 64, a window of 512: 68.2 -> 67.2 all the same).
// Tensor memory: two groups of 128 columns of output and of 96 columns of scores and weights, 512 in all, so a CTA to an SM.
// A value row beyond the sequence's end belongs to another sequence or to nothing, and a weight of zero times what is no
// number is none: the rows are set to zero in shared memory before the tile that crosses the end is multiplied.
// The reference of a row's exponentials follows the row's maximum only when that has outgrown it by 2^8, and is a whole power
// of two, so that O is rescaled (in tensor memory, exactly) on a few early steps only; the sink joins at the end.
// Every wait on an mbarrier is bounded; one that runs out sets status word 3 and the CTA winds down.
#define ABK_DEFINE_ERROR
#include "common.cuh"
#include "recurrence.cuh"
#include "tc_common.cuh"
#include "tensor_map.cuh"

#define WT_Q 128           // query rows of a group
#define WT_K 64            // keys of a tile
#define WT_THREADS 320
#define WT_BOX_Q (WT_Q * 128)  // bytes of a box of 64 columns of a query tile
#define WT_BOX_K (WT_K * 128)  // of a key or value tile

struct AttnWindowTc {
    __nv_bfloat16 *out;    // [tokens, n_heads * v_dim]
    int n_heads, n_kv_heads;
    int k_off, v_off;
    float scale_log2;      // positive
    int window, keep_first, chunk;
    const float *sink;     // [n_heads] or null
    const int *seq_start;  // [n_seqs + 1]
    int n_seqs, max_tiles;
    int *status;
};

// Shared-memory descriptor of the values as a B operand whose N dimension is contiguous ([key][value], boxes of 64 columns with
// the 128-byte swizzle): 8 keys are 1024 bytes apart, the next 64 columns a box on.
__device__ __forceinline__ uint64_t wt_values_desc(uint32_t addr) {
    uint64_t d = (uint64_t)((addr >> 4) & 0x3FFF);
    d |= (uint64_t)((WT_BOX_K >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
__device__ __forceinline__ uint64_t wt_k_major_desc(uint32_t base, uint32_t box_bytes, int k16) {
    return tc::smem_desc_k_sw128(base + (k16 / 4) * box_bytes + (k16 % 4) * 32);
}
// D[tmem] (+)= A[tmem] . B[smem]: A's rows in the lanes, two bfloat16 of K in a column.
__device__ __forceinline__ void wt_mma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, bool accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"((uint32_t)accumulate)
        : "memory");
}
__device__ __forceinline__ void wt_tmem_st16(uint32_t taddr, const uint32_t *v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
        "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
__device__ __forceinline__ float wt_ex2(float x) {  // 2^x by the special-function unit (-inf gives 0)
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// The tiles a CTA walks, and which of its two groups need one.
struct WindowTiles {
    int n, r0, window, keep_first, chunk, w_first, kept, count;
    __device__ __forceinline__ WindowTiles(const AttnWindowTc &p, int n_, int r0_) : n(n_), r0(r0_), window(p.window), keep_first(p.keep_first), chunk(p.chunk) {
        const int last = min(r0 + 2 * WT_Q - 1, n - 1);
        int lo = window > 0 && r0 - window + 1 > 0 ? r0 - window + 1 : 0;  // first key the first row sees in its window
        if (chunk > 0) lo = max(lo, r0 / chunk * chunk);                   // or in its chunk
        w_first = lo / WT_K;
        kept = window > 0 ? min((keep_first + WT_K - 1) / WT_K, w_first) : 0;
        count = kept + last / WT_K - w_first + 1;
    }
    __device__ __forceinline__ int key0(int i) const { return (i < kept ? i : w_first + i - kept) * WT_K; }
    __device__ __forceinline__ bool need(int g, int i) const {
        const int first = r0 + g * WT_Q, last = min(first + WT_Q - 1, n - 1), k0 = key0(i);
        if (first >= n || k0 > last) return false;
        if (i < kept) return true;
        if (chunk > 0 && k0 + WT_K - 1 < first / chunk * chunk) return false;
        return window <= 0 || k0 + WT_K - 1 > first - window || k0 < keep_first;
    }
};

template <int DB, int VB>  // boxes of 64 columns of a head and of its values
__global__ void __launch_bounds__(WT_THREADS, 1) attention_window_tc_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap kv_map,
                                                                            AttnWindowTc p) {
    constexpr int STAGES = DB == 3 ? 2 : 3;
    constexpr int Q_BYTES = DB * WT_BOX_Q, K_BYTES = DB * WT_BOX_K, V_BYTES = VB * WT_BOX_K;
    extern __shared__ __align__(1024) uint8_t wt_smem[];  // the kernel has no static shared memory: this starts aligned
    uint8_t *q_s = wt_smem, *k_s = q_s + 2 * Q_BYTES, *v_s = k_s + STAGES * K_BYTES;
    uint64_t *bars = (uint64_t *)(v_s + STAGES * V_BYTES);
    uint64_t *q_full = bars, *k_full = bars + 1, *k_empty = k_full + STAGES, *v_full = k_empty + STAGES, *v_empty = v_full + STAGES,
             *s_full = v_empty + STAGES, *p_full = s_full + 2, *o_step = p_full + 2;  // the last three: one a group
    uint32_t *tmem_holder = (uint32_t *)(o_step + 2);
    volatile int *failed = (volatile int *)(tmem_holder + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the CTAs in the order they start: the last tiles of the step's sequences, which see the most keys, first, all heads of a
    // tile together. (The step's index arrays come from further back than the kernel just before.)
    const int h = blockIdx.x % p.n_heads, kvh = h / (p.n_heads / p.n_kv_heads);
    int seq = -1, tile = p.max_tiles - 1 - (int)(blockIdx.x / p.n_heads), start = 0, n = 0;
    for (int s = 0; s < p.n_seqs; s++) {
        start = p.seq_start[s], n = p.seq_start[s + 1] - start;
        const int tiles = (n + 2 * WT_Q - 1) / (2 * WT_Q);
        if (tile < tiles) {
            seq = s;
            break;
        }
        tile -= tiles;
    }
    if (seq < 0) {
        pdl_wait();
        return;
    }
    const int r0 = tile * 2 * WT_Q;
    const WindowTiles t(p, n, r0);
    const bool two = r0 + WT_Q < n;  // the second group has rows
    if (threadIdx.x == 0) {
        *failed = 0;
        tc::mbar_init(q_full, 1);
        for (int s = 0; s < STAGES; s++)
            tc::mbar_init(&k_full[s], 1), tc::mbar_init(&k_empty[s], 1), tc::mbar_init(&v_full[s], 1), tc::mbar_init(&v_empty[s], 1);
        for (int g = 0; g < 2; g++) tc::mbar_init(&s_full[g], 1), tc::mbar_init(&p_full[g], WT_Q), tc::mbar_init(&o_step[g], 1);
        tc::mbar_init_fence();
        tc::tma_prefetch_map(&q_map), tc::tma_prefetch_map(&kv_map);
    }
    if (warp == 1) tc::tmem_alloc(tmem_holder, 512);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *tmem_holder;
    pdl_wait();  // q, k and v come from the kernel just before

    if (warp == 0) {
        if (lane == 0) {
            tc::mbar_expect_tx(q_full, (two ? 2 : 1) * Q_BYTES);
            for (int g = 0; g < (two ? 2 : 1); g++)
                for (int b = 0; b < DB; b++) tc::tma_load_2d(q_s + g * Q_BYTES + b * WT_BOX_Q, &q_map, (h * DB + b) * 64, start + r0 + g * WT_Q, q_full);
            int k_issued = 0, v_issued = 0;
            bool go = true;
            for (int i = 0; i < t.count && go; i++) {
                const int s = i % STAGES, y = start + t.key0(i);
                const uint32_t parity = ((i / STAGES) & 1) ^ 1;
                go = tc::mbar_wait(&k_empty[s], parity);
                if (!go) break;
                tc::mbar_expect_tx(&k_full[s], K_BYTES);
                for (int b = 0; b < DB; b++) tc::tma_load_2d(k_s + s * K_BYTES + b * WT_BOX_K, &kv_map, p.k_off + (kvh * DB + b) * 64, y, &k_full[s]);
                k_issued++;
                go = tc::mbar_wait(&v_empty[s], parity);
                if (!go) break;
                tc::mbar_expect_tx(&v_full[s], V_BYTES);
                for (int b = 0; b < VB; b++) tc::tma_load_2d(v_s + s * V_BYTES + b * WT_BOX_K, &kv_map, p.v_off + (kvh * VB + b) * 64, y, &v_full[s]);
                v_issued++;
            }
            if (!go) {  // let the copies in flight land before the CTA's memory goes away
                atomicOr(p.status + 3, 2);
                *failed = 1;
                tc::mbar_wait(q_full, 0);
                for (int i = max(0, k_issued - STAGES); i < k_issued; i++) tc::mbar_wait(&k_full[i % STAGES], (i / STAGES) & 1);
                for (int i = max(0, v_issued - STAGES); i < v_issued; i++) tc::mbar_wait(&v_full[i % STAGES], (i / STAGES) & 1);
            }
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc_s = tc::idesc_bf16_f32(WT_Q, WT_K), idesc_o = tc::idesc_bf16_f32(WT_Q, VB * 64) | (1u << 16);
        bool ok = __all_sync(0xffffffffu, tc::mbar_wait(q_full, 0));
        int done[2] = {0, 0};       // tiles whose second product is issued
        bool pending[2] = {false, false};
        // step i: each group's second product of the tile before, then its first product of this one
        for (int i = 0; i <= t.count && ok; i++) {
            const int s = i % STAGES, sp = (i + STAGES - 1) % STAGES;  // this tile's stage, and the stage of the one before
#pragma unroll
            for (int g = 0; g < 2; g++) {
                const uint32_t scores = tmem + 256 + g * 128, o = tmem + g * 128;
                if (pending[g]) {
                    ok = ok && tc::mbar_wait(&p_full[g], done[g] & 1);  // the weights are there, O is rescaled
                    ok = ok && tc::mbar_wait(&v_full[sp], ((i - 1) / STAGES) & 1);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    const int real = n - t.key0(i - 1);  // rows of the tile that are the sequence's
                    uint8_t *vs = v_s + sp * V_BYTES;
                    if (real < WT_K && (g == 0 || !t.need(0, i - 1))) {
                        for (int e = lane; e < (WT_K - real) * VB * 8; e += 32) {
                            const int row = real + e / (VB * 8), b = e / 8 % VB, c = e % 8;
                            *(uint4 *)(vs + b * WT_BOX_K + row * 128 + c * 16) = make_uint4(0, 0, 0, 0);
                        }
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        __syncwarp();
                    }
                    tc::fence_after_sync();
                    if (lane == 0) {
                        const uint32_t vb = tc::smem_addr(vs);
#pragma unroll
                        for (int part = 0; part < 3; part++)
#pragma unroll
                            for (int k16 = 0; k16 < WT_K / 16; k16++)
                                wt_mma_ts(o, scores + part * 32 + k16 * 8, wt_values_desc(vb + k16 * 2048), idesc_o, done[g] > 0 || part > 0 || k16 > 0);
                        tc::mma_commit(&o_step[g]);
                        if (g == 1 || !t.need(1, i - 1)) tc::mma_commit(&v_empty[sp]);  // the tile's values may be replaced
                    }
                    __syncwarp();
                    pending[g] = false, done[g]++;
                }
                if (i < t.count && t.need(g, i)) {
                    ok = ok && tc::mbar_wait(&k_full[s], (i / STAGES) & 1);
                    ok = ok && (done[g] == 0 || tc::mbar_wait(&o_step[g], (done[g] - 1) & 1));  // the weights have been read
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    tc::fence_after_sync();
                    if (lane == 0) {
                        const uint32_t qa = tc::smem_addr(q_s + g * Q_BYTES), kb = tc::smem_addr(k_s + s * K_BYTES);
#pragma unroll
                        for (int k16 = 0; k16 < DB * 4; k16++)
                            tc::mma_ss(scores, wt_k_major_desc(qa, WT_BOX_Q, k16), wt_k_major_desc(kb, WT_BOX_K, k16), idesc_s, k16 > 0);
                        tc::mma_commit(&s_full[g]);
                        if (g == 1 || !t.need(1, i)) tc::mma_commit(&k_empty[s]);  // the tile's keys may be replaced
                    }
                    __syncwarp();
                    pending[g] = true;
                }
            }
        }
        if (!ok && lane == 0) atomicOr(p.status + 3, 4), *failed = 1;
    } else {
        const int g = (warp - 2) >> 2, quarter = warp & 3, r = quarter * 32 + lane;  // (a warp reaches its own quarter of the lanes)
        const int row = r0 + g * WT_Q + r, warp_first = r0 + g * WT_Q + quarter * 32, warp_last = warp_first + 31;
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        const uint32_t scores = tmem + 256 + g * 128 + lane_base, o_row = tmem + g * 128 + lane_base;
        const int chunk0 = p.chunk > 0 ? row / p.chunk * p.chunk : 0;
        const int low = max(p.window > 0 ? row - p.window + 1 : 0, chunk0);  // first key the row sees but for the kept first ones
        float m = -INFINITY, l = 0.0f;  // the reference of the row's exponentials (in units of log2), and their sum
        int done = 0;
        bool ok = true;
        for (int i = 0; i < t.count && ok; i++) {
            if (!t.need(g, i)) continue;
            ok = __all_sync(0xffffffffu, tc::mbar_wait(&s_full[g], done & 1));
            if (!ok) break;
            tc::fence_after_sync();
            float s[WT_K];
#pragma unroll
            for (int c0 = 0; c0 < WT_K; c0 += 16) tc::tmem_ld16(scores + c0, (uint32_t *)(s + c0));
            tc::tmem_ld_wait();
            const int key0 = t.key0(i);
            // a tile whose every key every row of this warp sees needs no look at single keys
            const bool clear = i >= t.kept && key0 + WT_K - 1 <= warp_first && (p.window <= 0 || warp_last - key0 < p.window) &&
                               (p.chunk <= 0 || key0 >= warp_last / p.chunk * p.chunk);
            if (!clear) {
#pragma unroll
                for (int c = 0; c < WT_K; c++) {
                    const int j = key0 + c;
                    if (!(j <= row && (j >= low || (j < p.keep_first && j >= chunk0)))) s[c] = -INFINITY;
                }
            }
            float top0 = -INFINITY, top1 = -INFINITY, top2 = -INFINITY, top3 = -INFINITY;
#pragma unroll
            for (int c = 0; c < WT_K; c += 4) top0 = fmaxf(top0, s[c]), top1 = fmaxf(top1, s[c + 1]), top2 = fmaxf(top2, s[c + 2]), top3 = fmaxf(top3, s[c + 3]);
            const float cand = fmaxf(m, ceilf(fmaxf(fmaxf(top0, top1), fmaxf(top2, top3)) * p.scale_log2));
            // Each row for itself (the first tile: m is -inf), so that a row's bits know nothing of the rows beside it; the
            // vote only says whether any row of the warp has outputs to rescale (those of the others by one).
            const float m_new = cand > m + 8.0f ? cand : m, ref = m_new == -INFINITY ? 0.0f : m_new;
            const bool move = __any_sync(0xffffffffu, m_new != m);
            const float corr = m_new != m ? exp2f(m - ref) : 1.0f;  // (0 when m was -inf)
            m = m_new;
            // two weights at a time: an instruction for both where there is one (the same numbers, fewer to issue)
            const f32x2 scale2 = pack2(p.scale_log2, p.scale_log2), ref2 = pack2(-ref, -ref), minus = pack2(-1.0f, -1.0f);
            f32x2 sum2 = pack2(0.0f, 0.0f);
#pragma unroll
            for (int c0 = 0; c0 < WT_K; c0 += 32) {
                uint32_t hi[16], mid[16], lo[16];
#pragma unroll
                for (int c = 0; c < 32; c += 2) {
                    float2 x = unpack2(fma2(pack2(s[c0 + c], s[c0 + c + 1]), scale2, ref2));
                    x.x = wt_ex2(x.x), x.y = wt_ex2(x.y);
                    f32x2 x2 = pack2(x.x, x.y);
                    sum2 = add2(sum2, x2);
                    __nv_bfloat162 b = __floats2bfloat162_rn(x.x, x.y);
                    hi[c / 2] = *(const uint32_t *)&b;
                    x2 = fma2(pack2(__uint_as_float(hi[c / 2] << 16), __uint_as_float(hi[c / 2] & 0xffff0000u)), minus, x2);
                    x = unpack2(x2);
                    b = __floats2bfloat162_rn(x.x, x.y);
                    mid[c / 2] = *(const uint32_t *)&b;
                    x = unpack2(fma2(pack2(__uint_as_float(mid[c / 2] << 16), __uint_as_float(mid[c / 2] & 0xffff0000u)), minus, x2));
                    b = __floats2bfloat162_rn(x.x, x.y);
                    lo[c / 2] = *(const uint32_t *)&b;
                }
                wt_tmem_st16(scores + c0 / 2, hi), wt_tmem_st16(scores + 32 + c0 / 2, mid), wt_tmem_st16(scores + 64 + c0 / 2, lo);
            }
            const float2 sums = unpack2(sum2);
            l = l * corr + (sums.x + sums.y);
            if (done > 0 && move) {  // (the second product of the tile before is done: the first product of this one waited for it)
#pragma unroll 1
                for (int c0 = 0; c0 < VB * 64; c0 += 16) {
                    uint32_t v[16];
                    tc::tmem_ld16(o_row + c0, v);
                    tc::tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 16; e++) v[e] = __float_as_uint(__uint_as_float(v[e]) * corr);
                    wt_tmem_st16(o_row + c0, v);
                }
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc::fence_before_sync();
            tc::mbar_arrive(&p_full[g]);
            done++;
        }
        if (ok && done > 0) ok = __all_sync(0xffffffffu, tc::mbar_wait(&o_step[g], (done - 1) & 1));
        if (!ok) {
            if (lane == 0) atomicOr(p.status + 3, 8), *failed = 1;
        } else if (done > 0) {
            tc::fence_after_sync();
            const float sink2 = p.sink ? p.sink[h] * 1.4426950408889634f : -INFINITY, top = fmaxf(m, sink2);
            const float own = exp2f(m - top), inv = own / (l * own + (p.sink ? exp2f(sink2 - top) : 0.0f));
            __nv_bfloat16 *dst = p.out + ((long long)(start + row) * p.n_heads + h) * (VB * 64);
#pragma unroll 1
            for (int c0 = 0; c0 < VB * 64; c0 += 32) {
                uint32_t v[32], w[16];
                tc::tmem_ld16(o_row + c0, v);
                tc::tmem_ld16(o_row + c0 + 16, v + 16);
                tc::tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 16; e++) {
                    const __nv_bfloat162 b = __floats2bfloat162_rn(__uint_as_float(v[2 * e]) * inv, __uint_as_float(v[2 * e + 1]) * inv);
                    w[e] = *(const uint32_t *)&b;
                }
                if (row < n) {
#pragma unroll
                    for (int e = 0; e < 4; e++) *(uint4 *)(dst + c0 + 8 * e) = make_uint4(w[4 * e], w[4 * e + 1], w[4 * e + 2], w[4 * e + 3]);
                }
            }
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (*failed && threadIdx.x == 0) atomicOr(p.status + 3, 1);
    if (warp == 1) {
        tc::fence_after_sync();
        tc::tmem_free(tmem, 512);
    }
}

// max_tiles: an upper bound of the step's tiles of 256 rows, sum over its sequences of ceil(rows / 256) (CTAs beyond the
// real tiles return at once). n_rows: rows of qkv that may be read. status word 3 is set if a wait ran out.
extern "C" int abk_attention_window_tc(const void *qkv, long long row, int n_rows, void *out, int n_heads, int n_kv_heads, int head_dim, int v_dim,
                                       int k_off, int v_off, float scale, int window, int keep_first, const float *sink, const int *seq_start,
                                       int n_seqs, int max_tiles, int chunk, int *status, void *stream) {
    if (n_seqs <= 0 || max_tiles <= 0 || n_rows <= 0) return 0;
    if ((head_dim != 64 && head_dim != 128 && head_dim != 192) || (v_dim != 64 && v_dim != 128))
        ABK_REFUSE("attention_window_tc: heads of %d and values of %d are not 64, 128 or 192 and 64 or 128", head_dim, v_dim);
    if (!(scale > 0.0f)) ABK_REFUSE("attention_window_tc: the scale is not positive");
    if (row % 8 || k_off % 8 || v_off % 8 || ((uintptr_t)qkv & 15) || ((uintptr_t)out & 15)) ABK_REFUSE("attention_window_tc: rows of q, k and v are not 16-byte aligned");
    if (n_kv_heads < 1 || n_heads % n_kv_heads) ABK_REFUSE("attention_window_tc: %d query heads do not divide into %d kv heads", n_heads, n_kv_heads);
    if ((long long)max_tiles * n_heads > 0x7fffffffLL) ABK_REFUSE("attention_window_tc: %d tiles of %d heads exceed a grid", max_tiles, n_heads);
    CUtensorMap qm, kvm;
    int rc = tmap::bf16_rows_of_128_bytes(qkv, n_rows, row, row, WT_Q, &qm);
    if (!rc) rc = tmap::bf16_rows_of_128_bytes(qkv, n_rows, row, row, WT_K, &kvm);
    if (rc) return rc;
    AttnWindowTc p;
    p.out = (__nv_bfloat16 *)out, p.n_heads = n_heads, p.n_kv_heads = n_kv_heads, p.k_off = k_off, p.v_off = v_off;
    p.scale_log2 = scale * 1.4426950408889634f, p.window = window > 0 ? window : 0, p.keep_first = window > 0 && keep_first > 0 ? keep_first : 0;
    p.chunk = chunk > 0 ? chunk : 0, p.sink = sink, p.seq_start = seq_start, p.n_seqs = n_seqs, p.max_tiles = max_tiles, p.status = status;
#define WT_LAUNCH(DB, VB)                                                                                                          \
    do {                                                                                                                           \
        constexpr int smem = 2 * DB * WT_BOX_Q + (DB == 3 ? 2 : 3) * (DB + VB) * WT_BOX_K + 512;                                   \
        if (cudaError_t e = abk_allow_shared_memory((const void *)attention_window_tc_kernel<DB, VB>, smem)) return (int)e;        \
        abk_launch(attention_window_tc_kernel<DB, VB>, dim3((unsigned)(max_tiles * n_heads)), dim3(WT_THREADS), smem, (cudaStream_t)stream, qm, kvm, p); \
    } while (0)
    if (v_dim == 64) {
        if (head_dim == 64) WT_LAUNCH(1, 1);
        else if (head_dim == 128) WT_LAUNCH(2, 1);
        else WT_LAUNCH(3, 1);
    } else {
        if (head_dim == 64) WT_LAUNCH(1, 2);
        else if (head_dim == 128) WT_LAUNCH(2, 2);
        else WT_LAUNCH(3, 2);
    }
#undef WT_LAUNCH
    return ABK_LAUNCH_RESULT();
}
