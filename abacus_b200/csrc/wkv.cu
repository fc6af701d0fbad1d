// Time mixing with a decay per head, key channel and token ("wkv"): a recurrent mixer whose state is one [key, value]
// matrix per head and the token before,
//     o_t = (S_(t-1) + diag(u) k_t v_t^T)^T r_t,    S_t = diag(w_t) S_(t-1) + k_t v_t^T,    w_t = exp(-exp(z_t + w0)),
// float32, zero at a sequence's start and carried from step to step in the sequence's slot.
//
//   token_shift       per token the blends m_s = x + (x' - x) * mu_s of a row with the row before it (the sequence's
//                     last row of the step before, kept in its slot, for a step's first row; zeros at the start), one
//                     plane of the output per s. In a step of one token a sequence it also leaves the new last row.
//   token_shift_keep  the last row of every sequence of a step of prompts, into its slot.
//   wkv_block         prompts: blocks of four tokens (below)
//   wkv_step          a step of one token a sequence (below)
//   wkv_scan          a step of a few tokens a sequence, and prompts of heads too few to fill the GPU, in segments walked
//                     side by side: a CTA walks one sequence's (a segment's) tokens for one head and 16 (32 for heads
//                     of up to 32 channels) value columns. Its threads are those columns x 4, 8 or 16 parts of the key
//                     channels, so a thread keeps 4 to 16 state values in registers; the parts' partial outputs of a
//                     column meet by shuffles, four tokens at a time. Rows come 16 (8 for heads beyond 128 channels) tokens
//                     at a time: asked for a chunk ahead into registers, the decay made from its pre-activation on the way
//                     into shared memory, read from there as 16-byte pieces. A sequence that brings no token to the step
//                     is left alone.
#define ABK_DEFINE_ERROR
#include "recurrence.cuh"

// ---------------------------------------------------------------- the blends with the token before
struct TokenShift {
    const void *x;       // [tokens][d], as stored
    float *last;         // [slots][d]: the last row a sequence brought
    const float *mu;     // [blends][d]
    void *out;           // [blends][plane]: blend s of row t at out + s * plane + t * d
    long long plane;
    int d, blends, update;
    const int *token_seq, *seq_start, *seq_slot;
};

// A thread has one column (a CTA 128 of them: blockIdx.y counts the runs of columns), so that no load waits for a store.
template <typename T> __global__ void __launch_bounds__(128) token_shift_kernel(TokenShift p) {
    const int t = blockIdx.x, j = blockIdx.y * 128 + threadIdx.x;
    pdl_wait();
    const int seq = p.token_seq[t];
    if (seq < 0 || j >= p.d) return;
    const bool first = t == p.seq_start[seq];
    float *last = p.last + (long long)p.seq_slot[seq] * p.d;
    const T *x = (const T *)p.x + (long long)t * p.d;
    T *out = (T *)p.out + (long long)t * p.d;
    const float h = to_float(x[j]);
    const float before = first ? last[j] : to_float(x[j - p.d]);
    const float diff = before - h;
    for (int s = 0; s < p.blends; s++) out[s * p.plane + j] = from_float<T>(fmaf(diff, __ldg(p.mu + (long long)s * p.d + j), h));
    if (p.update) last[j] = h;  // (a step of one token a sequence: this row is the sequence's only one)
}

__device__ __forceinline__ void shift_open(uint4 raw, float *v) {
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int e = 0; e < 4; e++) v[2 * e] = __uint_as_float(w[e] << 16), v[2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u);
}
// The same for bfloat16 rows of a multiple of 8 columns and up to 8 blends: a thread has 8 consecutive columns of TOKENS
// tokens, read and written as 16-byte pieces, the blends' factors read once for all of them (16 bytes of a row go with 32 of each
// blend's factors), every load on its way before the first store. Long steps take four tokens: 3,571 tokens of 2,560, five blends,
// 110 MB, in 21.8 us with the rows that are kept; one token a thread, and the kept rows by one CTA a sequence, 43.5. At the line, 1,016 tokens
// by one and 1,024 by four, with the kept rows: 8.7 and 7.5 us, of 1,024 columns 5.3 and 4.2; below it one token a thread keeps the SMs full.
#define SHIFT_TOKENS 4
template <int BLENDS, int TOKENS> __global__ void __launch_bounds__(128) token_shift_bf16x8_kernel(TokenShift p, int n_tokens) {
    const int t0 = blockIdx.x * TOKENS, j = (blockIdx.y * 128 + threadIdx.x) * 8;
    float4 m[BLENDS][2];
    if (j < p.d) {
#pragma unroll
        for (int s = 0; s < BLENDS; s++)
            if (s < p.blends) m[s][0] = __ldg((const float4 *)(p.mu + (long long)s * p.d + j)), m[s][1] = __ldg((const float4 *)(p.mu + (long long)s * p.d + j + 4));
    }
    pdl_wait();
    if (j >= p.d) return;
    int seq[TOKENS];
    bool first[TOKENS];
    uint4 rows[TOKENS + 1];  // from the row before the first token on
#pragma unroll
    for (int i = 0; i < TOKENS; i++) seq[i] = t0 + i < n_tokens ? p.token_seq[t0 + i] : -1;
#pragma unroll
    for (int i = 0; i <= TOKENS; i++) {
        const int t = t0 + i - 1;
        rows[i] = make_uint4(0, 0, 0, 0);
        if (t >= 0 && t < n_tokens) rows[i] = *(const uint4 *)((const __nv_bfloat16 *)p.x + (long long)t * p.d + j);
    }
#pragma unroll
    for (int i = 0; i < TOKENS; i++) first[i] = seq[i] >= 0 && t0 + i == p.seq_start[seq[i]];
#pragma unroll
    for (int i = 0; i < TOKENS; i++) {
        if (seq[i] < 0) continue;
        float h[8], before[8];
        shift_open(rows[i + 1], h);
        float *last = p.last + (first[i] || p.update ? (long long)p.seq_slot[seq[i]] * p.d + j : 0);
        if (first[i]) {
            const float4 a = *(const float4 *)last, b = *(const float4 *)(last + 4);
            before[0] = a.x, before[1] = a.y, before[2] = a.z, before[3] = a.w, before[4] = b.x, before[5] = b.y, before[6] = b.z, before[7] = b.w;
        } else {
            shift_open(rows[i], before);
        }
        __nv_bfloat16 *out = (__nv_bfloat16 *)p.out + (long long)(t0 + i) * p.d + j;
#pragma unroll
        for (int s = 0; s < BLENDS; s++) {
            if (s >= p.blends) break;
            const float mu[8] = {m[s][0].x, m[s][0].y, m[s][0].z, m[s][0].w, m[s][1].x, m[s][1].y, m[s][1].z, m[s][1].w};
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const __nv_bfloat162 h2 = __floats2bfloat162_rn(fmaf(before[2 * e] - h[2 * e], mu[2 * e], h[2 * e]),
                                                                fmaf(before[2 * e + 1] - h[2 * e + 1], mu[2 * e + 1], h[2 * e + 1]));
                w[e] = *(const uint32_t *)&h2;
            }
            *(uint4 *)(out + s * p.plane) = make_uint4(w[0], w[1], w[2], w[3]);
        }
        if (p.update) {
            *(float4 *)last = make_float4(h[0], h[1], h[2], h[3]);
            *(float4 *)(last + 4) = make_float4(h[4], h[5], h[6], h[7]);
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(128) token_shift_keep_kernel(const T *x, float *last, int d, const int *seq_start,
                                                               const int *seq_slot) {
    const int seq = blockIdx.x, j = blockIdx.y * 128 + threadIdx.x;
    pdl_wait();
    const int row0 = seq_start[seq], n = seq_start[seq + 1] - row0;
    if (n <= 0 || j >= d) return;
    last[(long long)seq_slot[seq] * d + j] = to_float(x[(long long)(row0 + n - 1) * d + j]);
}

extern "C" int abk_token_shift(const void *x, int dtype, int n_tokens, int d, const float *mu, int blends, float *last, void *out,
                               long long plane, int update, const int *token_seq, const int *seq_start, const int *seq_slot,
                               void *stream) {
    if (n_tokens <= 0) return 0;
    if (blends < 1 || d < 1 || plane < (long long)n_tokens * d) ABK_REFUSE("token_shift: %d blends of %d columns", blends, d);
    TokenShift p;
    p.x = x, p.last = last, p.mu = mu, p.out = out, p.plane = plane, p.d = d, p.blends = blends, p.update = update;
    p.token_seq = token_seq, p.seq_start = seq_start, p.seq_slot = seq_slot;
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == ABK_BF16 && d % 8 == 0 && blends <= 8 && plane % 8 == 0 && ((uintptr_t)x | (uintptr_t)out | (uintptr_t)mu | (uintptr_t)last) % 16 == 0) {
        if (n_tokens >= 1024) abk_launch(token_shift_bf16x8_kernel<8, SHIFT_TOKENS>, dim3((n_tokens + SHIFT_TOKENS - 1) / SHIFT_TOKENS, (d / 8 + 127) / 128), dim3(128), 0, s, p, n_tokens);
        else abk_launch(token_shift_bf16x8_kernel<8, 1>, dim3(n_tokens, (d / 8 + 127) / 128), dim3(128), 0, s, p, n_tokens);
    } else if (dtype == ABK_BF16) abk_launch(token_shift_kernel<__nv_bfloat16>, dim3(n_tokens, (d + 127) / 128), dim3(128), 0, s, p);
    else abk_launch(token_shift_kernel<float>, dim3(n_tokens, (d + 127) / 128), dim3(128), 0, s, p);
    return ABK_LAUNCH_RESULT();
}

extern "C" int abk_token_shift_keep(const void *x, int dtype, int d, float *last, const int *seq_start, const int *seq_slot,
                                    int n_seqs, void *stream) {
    if (n_seqs <= 0 || d <= 0) return 0;
    if (d > 65535 * 128) ABK_REFUSE("token_shift: %d columns are more than a grid takes", d);
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == ABK_BF16)
        abk_launch(token_shift_keep_kernel<__nv_bfloat16>, dim3(n_seqs, (d + 127) / 128), dim3(128), 0, s, (const __nv_bfloat16 *)x, last, d, seq_start, seq_slot);
    else
        abk_launch(token_shift_keep_kernel<float>, dim3(n_seqs, (d + 127) / 128), dim3(128), 0, s, (const float *)x, last, d, seq_start, seq_slot);
    return ABK_LAUNCH_RESULT();
}

// ---------------------------------------------------------------- the activation inside the decay's pair of matrices
// dst = tanh(src) over `cols` columns of n rows (rows of any pitch): src float32 (a product's sums) or as stored, dst as
// stored (the second product's input).
template <typename TS, typename T>
__global__ void __launch_bounds__(256) tanh_rows_kernel(const TS *src, long long lds, T *dst, long long ldd, int cols, long long total) {
    pdl_wait();
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= total) return;
    const long long t = i / cols;
    const int j = (int)(i - t * cols);
    dst[t * ldd + j] = from_float<T>(tanhf(to_float(src[t * lds + j])));
}

extern "C" int abk_tanh_rows(const void *src, long long lds, int src_dtype, void *dst, long long ldd, int dtype, int n, int cols,
                             void *stream) {
    const long long total = (long long)n * cols;
    if (total <= 0) return 0;
    const dim3 grid((unsigned)((total + 255) / 256));
    cudaStream_t s = (cudaStream_t)stream;
    typedef __nv_bfloat16 bf;
    if (dtype == ABK_BF16 && src_dtype == ABK_BF16)
        abk_launch(tanh_rows_kernel<bf, bf>, grid, dim3(256), 0, s, (const bf *)src, lds, (bf *)dst, ldd, cols, total);
    else if (dtype == ABK_BF16)
        abk_launch(tanh_rows_kernel<float, bf>, grid, dim3(256), 0, s, (const float *)src, lds, (bf *)dst, ldd, cols, total);
    else if (src_dtype == ABK_F32)
        abk_launch(tanh_rows_kernel<float, float>, grid, dim3(256), 0, s, (const float *)src, lds, (float *)dst, ldd, cols, total);
    else
        ABK_REFUSE("tanh_rows: bfloat16 into float32 is not built");
    return ABK_LAUNCH_RESULT();
}

// ---------------------------------------------------------------- the recurrence
struct WkvScan {
    const void *proj;    // row t at proj + t * ld: r head h at r_at + h * dim, k at k_at + h * dim, v at v_at + h * dim
    long long ld;
    int r_at, k_at, v_at;
    int n_heads, dim;
    const float *pre;    // [tokens][heads * dim]: the decay's pre-activation z
    const float *w0;     // [heads * dim]
    const float *bonus;  // [heads * dim]
    float *state;        // [slots][heads][dim][dim] (key, value)
    float *out;          // [tokens][heads * dim]
    const int *seq_start, *seq_slot;
    int n_seqs, tiles, longest_first, vec;  // of the walk in blocks
    // Prompts in segments of `chunk` tokens, all at once (blockIdx.z counts the step's segments, sequence after sequence):
    // phase 1 walks each segment from an empty state and leaves its sum and the product of its decays,
    // wkv_segment_prefix turns the sums into the states at the segments' starts (and leaves the last in the slot), phase 2
    // walks each segment again from its start state for the outputs. chunk 0 (phase 0): a CTA walks a whole sequence.
    int chunk;
    float *sums;         // [segments][heads][dim][dim]
    float *prods;        // [segments][heads][dim]
};

// The segment blockIdx.z names: its sequence, its first row and its rows (0: none). Sequences are walked in order.
__device__ __forceinline__ void wkv_segment(const int *seq_start, int n_seqs, int chunk, int z, int &seq, int &row0, int &n) {
    n = 0;
    int first = 0;
    for (seq = 0; seq < n_seqs; seq++) {
        const int start = seq_start[seq], len = seq_start[seq + 1] - start, count = (len + chunk - 1) / chunk;
        if (z < first + count) {
            const int c = z - first;
            row0 = start + c * chunk, n = len - c * chunk < chunk ? len - c * chunk : chunk;
            return;
        }
        first += count;
    }
}

// N tokens of one thread's share: r, k, w point at the thread's channels of the first token (tokens `pitch` floats
// apart), v at its column's value (tokens `v_pitch` apart); the column's output goes to out if `writes`.
// SUMS: the state alone moves (a segment's own sum): no r, no output.
template <int DPT, int PARTS, int N, bool SUMS>
__device__ __forceinline__ void wkv_tokens(float *s, const float *u, const float *r, const float *k, const float *w, int pitch,
                                           const float *v, int v_pitch, bool writes, float *out, long long out_pitch) {
    if constexpr (SUMS) {
        float vv[N];
#pragma unroll
        for (int n = 0; n < N; n++) vv[n] = v[n * v_pitch];
#pragma unroll
        for (int i = 0; i < DPT / 4; i++) {
            float4 kk[N], ww[N];
#pragma unroll
            for (int n = 0; n < N; n++) kk[n] = *(const float4 *)(k + n * pitch + 4 * i), ww[n] = *(const float4 *)(w + n * pitch + 4 * i);
#pragma unroll
            for (int n = 0; n < N; n++) {
                s[4 * i] = fmaf(ww[n].x, s[4 * i], kk[n].x * vv[n]), s[4 * i + 1] = fmaf(ww[n].y, s[4 * i + 1], kk[n].y * vv[n]);
                s[4 * i + 2] = fmaf(ww[n].z, s[4 * i + 2], kk[n].z * vv[n]), s[4 * i + 3] = fmaf(ww[n].w, s[4 * i + 3], kk[n].w * vv[n]);
            }
        }
        return;
    }
    float vv[N], o[N];
#pragma unroll
    for (int n = 0; n < N; n++) vv[n] = v[n * v_pitch], o[n] = 0.0f;
#pragma unroll
    for (int i = 0; i < DPT / 4; i++) {
        float4 kk[N], rr[N], ww[N];
#pragma unroll
        for (int n = 0; n < N; n++) {
            kk[n] = *(const float4 *)(k + n * pitch + 4 * i), rr[n] = *(const float4 *)(r + n * pitch + 4 * i);
            ww[n] = *(const float4 *)(w + n * pitch + 4 * i);
        }
#pragma unroll
        for (int n = 0; n < N; n++) {
            const float a0 = kk[n].x * vv[n], a1 = kk[n].y * vv[n], a2 = kk[n].z * vv[n], a3 = kk[n].w * vv[n];
            o[n] = fmaf(rr[n].x, fmaf(u[4 * i], a0, s[4 * i]), o[n]);
            o[n] = fmaf(rr[n].y, fmaf(u[4 * i + 1], a1, s[4 * i + 1]), o[n]);
            o[n] = fmaf(rr[n].z, fmaf(u[4 * i + 2], a2, s[4 * i + 2]), o[n]);
            o[n] = fmaf(rr[n].w, fmaf(u[4 * i + 3], a3, s[4 * i + 3]), o[n]);
            s[4 * i] = fmaf(ww[n].x, s[4 * i], a0), s[4 * i + 1] = fmaf(ww[n].y, s[4 * i + 1], a1);
            s[4 * i + 2] = fmaf(ww[n].z, s[4 * i + 2], a2), s[4 * i + 3] = fmaf(ww[n].w, s[4 * i + 3], a3);
        }
    }
#pragma unroll
    for (int m = 1; m < PARTS; m <<= 1)
#pragma unroll
        for (int n = 0; n < N; n++) o[n] += __shfl_xor_sync(0xffffffffu, o[n], m);
    if (writes)
#pragma unroll
        for (int n = 0; n < N; n++) out[n * out_pitch] = o[n];
}

// DPT key channels a thread, PARTS threads a value column (DPT * PARTS >= dim); a CTA has COLS columns and stages TOK
// tokens at a time.
// The decay from its pre-activation: to the last bit where the model is float32; where the model's operands are bfloat16
// numbers, by the special-function unit (a few units in the last place of float32, in float32 arithmetic).
template <typename T> __device__ __forceinline__ float wkv_decay(float z) { return expf(-expf(z)); }
template <> __device__ __forceinline__ float wkv_decay<__nv_bfloat16>(float z) { return __expf(-__expf(z)); }

// PHASE: of a walk in segments (above), 0 where a CTA walks a whole sequence.
template <typename T, int DPT, int PARTS, int COLS, int TOK, int PHASE>
__global__ void __launch_bounds__(PARTS * COLS, 2) wkv_scan_kernel(WkvScan p) {
    constexpr bool SUMS = PHASE == 1;
    constexpr int DP = DPT * PARTS;             // key channels, padded
    constexpr int PITCH = PARTS * (DPT + 4);    // a token's channels in shared memory: a part's run, then 4 floats of
    constexpr int THREADS = PARTS * COLS;       // padding, so that the parts' 16-byte reads meet no bank twice
    constexpr int PER = TOK * DP / THREADS;     // elements of r (of k, of the decay) a thread stages a chunk
    constexpr int PER_V = (TOK * COLS + THREADS - 1) / THREADS;
    __shared__ __align__(16) float r_s[TOK][PITCH], k_s[TOK][PITCH], w_s[TOK][PITCH];
    __shared__ float v_s[TOK][COLS];
    const int tile = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, part = tid % PARTS, vc = tid / PARTS;
    const int col = tile * COLS + vc;
    float u[DPT];
#pragma unroll
    for (int i = 0; i < DPT; i++) {
        const int d = part * DPT + i;
        u[i] = d < p.dim ? p.bonus[(long long)h * p.dim + d] : 0.0f;
    }
    pdl_wait();
    int seq = blockIdx.z, row0, n;
    if constexpr (PHASE > 0) wkv_segment(p.seq_start, p.n_seqs, p.chunk, blockIdx.z, seq, row0, n);
    else row0 = p.seq_start[seq], n = p.seq_start[seq + 1] - row0;
    if (n <= 0) return;  // (a sequence of the step's padding: its slot is someone else's)
    float *state = PHASE == 0 ? p.state + ((long long)p.seq_slot[seq] * p.n_heads + h) * p.dim * p.dim
                                : p.sums + ((long long)blockIdx.z * p.n_heads + h) * p.dim * p.dim;
    float s[DPT];
#pragma unroll
    for (int i = 0; i < DPT; i++) {
        const int d = part * DPT + i;
        s[i] = PHASE != 1 && d < p.dim && col < p.dim ? state[(long long)d * p.dim + col] : 0.0f;
    }
    const T *proj = (const T *)p.proj;
    const long long hk = (long long)p.n_heads * p.dim;
    // A chunk's rows are asked for a chunk ahead and kept as they come: nothing is done to a loaded value before the
    // chunk is staged (an instruction that needs it would hold the warp until the load is back), so the loads' way from
    // memory lies under the chunk before. A thread stages one channel (THREADS is a multiple of the padded channels).
    static_assert(THREADS % DP == 0, "a thread stages one channel");
    T rr[PER], rk[PER], rv[PER_V];
    float rz[PER];
    const int my_d = tid % DP, my_ch = h * p.dim + (my_d < p.dim ? my_d : 0);
    const float my_w0 = p.w0[my_ch];
    float decayed = 1.0f;  // phase 1: the product of this thread's staged decays (one channel, its share of the tokens)
    auto fetch = [&](int c0) {
        const int cnt = n - c0 < TOK ? n - c0 : TOK;
#pragma unroll
        for (int it = 0; it < PER; it++) {
            // (every load is made, from a place that exists, and dropped where it is not wanted: loads that hang on no
            // branch are all in flight together)
            if (it * THREADS >= cnt * DP) break;  // (the same for every thread: the chunk has no such token)
            const int tok = (tid + it * THREADS) / DP;
            const long long row = row0 + c0 + (tok < cnt ? tok : cnt - 1);
            const T *r = proj + row * p.ld + my_ch;
            if (!SUMS) rr[it] = r[p.r_at];
            rk[it] = r[p.k_at], rz[it] = p.pre[row * hk + my_ch];
        }
#pragma unroll
        for (int it = 0; it < PER_V; it++) {
            if (it * THREADS >= cnt * COLS) break;
            const int e = tid + it * THREADS, tok = e / COLS, c = tile * COLS + e % COLS;
            rv[it] = proj[(long long)(row0 + c0 + (tok < cnt ? tok : cnt - 1)) * p.ld + p.v_at + (long long)h * p.dim + (c < p.dim ? c : 0)];
        }
    };
    fetch(0);
    for (int c0 = 0; c0 < n; c0 += TOK) {
        const int cnt = n - c0 < TOK ? n - c0 : TOK;
        __syncthreads();  // the chunk before is done with
#pragma unroll
        for (int it = 0; it < PER; it++) {
            if (it * THREADS >= cnt * DP) break;
            const int tok = (tid + it * THREADS) / DP, at = (my_d / DPT) * (DPT + 4) + my_d % DPT;
            const bool in = tok < cnt && my_d < p.dim;
            const float w = wkv_decay<T>(rz[it] + my_w0);
            if (!SUMS) r_s[tok][at] = in ? to_float(rr[it]) : 0.0f;
            if (SUMS && in) decayed *= w;
            k_s[tok][at] = in ? to_float(rk[it]) : 0.0f, w_s[tok][at] = w;
        }
#pragma unroll
        for (int it = 0; it < PER_V; it++) {
            const int e = tid + it * THREADS;
            if (e < cnt * COLS) v_s[e / COLS][e % COLS] = tile * COLS + e % COLS < p.dim ? to_float(rv[it]) : 0.0f;
        }
        __syncthreads();
        if (c0 + TOK < n) fetch(c0 + TOK);
        // four tokens at a time: their reads from shared memory and their shuffles overlap, and only the state's own
        // multiply-adds follow one another
        const int at = part * (DPT + 4);
        float *out = p.out + (long long)(row0 + c0) * hk + (long long)h * p.dim + col;
        const bool writes = part == 0 && col < p.dim && PHASE != 1;
        int tok = 0;
        for (; tok + 4 <= cnt; tok += 4)
            wkv_tokens<DPT, PARTS, 4, SUMS>(s, u, &r_s[tok][at], &k_s[tok][at], &w_s[tok][at], PITCH, &v_s[tok][vc], COLS, writes, out + tok * hk, hk);
        for (; tok < cnt; tok++)
            wkv_tokens<DPT, PARTS, 1, SUMS>(s, u, &r_s[tok][at], &k_s[tok][at], &w_s[tok][at], PITCH, &v_s[tok][vc], COLS, writes, out + tok * hk, hk);
    }
    if constexpr (PHASE == 2) return;  // (the states between segments are wkv_segment_prefix's)
#pragma unroll
    for (int i = 0; i < DPT; i++) {
        const int d = part * DPT + i;
        if (d < p.dim && col < p.dim) state[(long long)d * p.dim + col] = s[i];
    }
    if (PHASE == 1 && tile == 0) {
        // every thread staged the decays of one channel: the shares of a channel meet through shared memory
        __syncthreads();
        float *share = &r_s[0][0];
        share[tid] = decayed;
        __syncthreads();
        if (tid < DP && tid < p.dim) {
            float all = 1.0f;
            for (int o = tid; o < THREADS; o += DP) all *= share[o];
            p.prods[((long long)blockIdx.z * p.n_heads + h) * p.dim + tid] = all;
        }
    }
}

// A step of one token a sequence: the state comes and goes once, and that is all there is to do. A CTA has one (sequence, head) and
// 4 LPR of its value columns, a lane four of them in every 16th row (as a 16-byte piece where heads are a multiple of 4 channels),
// all rows asked for before the token's r, k and decay are made; the rows' sums of a column meet by shuffles and across the warps.
// (A sequence that brings several tokens after all is walked token by token.) Bound by the state's way in and out of memory: 64
// sequences, 40 heads of 64, 84 MB of it read and written in 14 to 15 us (part of it in the L2), 20 heads of 128 in 37; 8 sequences, 40
// heads of 64 4.3 us (wkv_scan, which has no more than a column a thread in flight: 57, 123 and 9.1).
template <typename T, int LPR, int ROWS, bool VEC>  // lanes of a row; rows of a thread
__global__ void __launch_bounds__(16 * LPR) wkv_step_kernel(WkvScan p) {
    constexpr int THREADS = 16 * LPR, WARPS = THREADS / 32, COLS = 4 * LPR;
    __shared__ float r_s[16 * ROWS], k_s[16 * ROWS], w_s[16 * ROWS], u_s[16 * ROWS];
    __shared__ __align__(16) float meet[WARPS][COLS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, D = p.dim, h = blockIdx.y, row = tid / LPR;
    const int col = blockIdx.x * COLS + tid % LPR * 4;
    const bool mine = col < D;
    const long long hk = (long long)p.n_heads * D;
    pdl_wait();
    const int seq = blockIdx.z, row0 = p.seq_start[seq], n = p.seq_start[seq + 1] - row0;
    if (n <= 0) return;  // (a sequence of the step's padding: its slot is someone else's)
    float *state = p.state + ((long long)p.seq_slot[seq] * p.n_heads + h) * D * D + col;
    float4 S[ROWS];
#pragma unroll
    for (int i = 0; i < ROWS; i++) {
        const float *src = state + (long long)(row + 16 * i) * D;
        S[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (!mine || row + 16 * i >= D) continue;
        if constexpr (VEC) S[i] = *(const float4 *)src;
        else S[i] = make_float4(src[0], col + 1 < D ? src[1] : 0.0f, col + 2 < D ? src[2] : 0.0f, col + 3 < D ? src[3] : 0.0f);
    }
    for (int t = 0; t < n; t++) {
        const T *proj = (const T *)p.proj + (long long)(row0 + t) * p.ld + h * D;
        float v[4];
#pragma unroll
        for (int x = 0; x < 4; x++) v[x] = col + x < D ? to_float(proj[p.v_at + col + x]) : 0.0f;
        for (int d = tid; d < 16 * ROWS; d += THREADS) {
            const bool in = d < D;
            r_s[d] = in ? to_float(proj[p.r_at + d]) : 0.0f, k_s[d] = in ? to_float(proj[p.k_at + d]) : 0.0f;
            w_s[d] = in ? wkv_decay<T>(p.pre[(row0 + t) * hk + h * D + d] + p.w0[h * D + d]) : 0.0f, u_s[d] = in ? p.bonus[h * D + d] : 0.0f;
        }
        __syncthreads();
        float o[4] = {};
#pragma unroll
        for (int i = 0; i < ROWS; i++) {
            const int d = row + 16 * i;
            const float r = r_s[d], k = k_s[d], w = w_s[d], u = u_s[d];
            float *s = (float *)&S[i];
#pragma unroll
            for (int x = 0; x < 4; x++) {
                const float a = k * v[x];
                o[x] = fmaf(r, fmaf(u, a, s[x]), o[x]), s[x] = fmaf(w, s[x], a);
            }
        }
#pragma unroll
        for (int m = LPR; m < 32; m <<= 1)
#pragma unroll
            for (int x = 0; x < 4; x++) o[x] += __shfl_xor_sync(0xffffffffu, o[x], m);
        if (lane < LPR) *(float4 *)&meet[warp][4 * lane] = make_float4(o[0], o[1], o[2], o[3]);
        __syncthreads();
        const int c = blockIdx.x * COLS + tid;
        if (tid < COLS && c < D) {
            float sum = meet[0][tid];
#pragma unroll
            for (int w = 1; w < WARPS; w++) sum += meet[w][tid];
            p.out[(row0 + t) * hk + (long long)h * D + c] = sum;
        }
    }
#pragma unroll
    for (int i = 0; i < ROWS; i++) {
        float *dst = state + (long long)(row + 16 * i) * D;
        if (!mine || row + 16 * i >= D) continue;
        if constexpr (VEC) {
            *(float4 *)dst = S[i];
        } else {
            dst[0] = S[i].x;
            if (col + 1 < D) dst[1] = S[i].y;
            if (col + 2 < D) dst[2] = S[i].z;
            if (col + 3 < D) dst[3] = S[i].w;
        }
    }
}

// The states at the segments' starts from the segments' own sums: along a sequence S <- prod * S + sum, the state before
// each segment left where its sum was, the last in the sequence's slot. A thread an element of the state; four segments'
// loads are on their way together.
__global__ void __launch_bounds__(256) wkv_segment_prefix_kernel(float *sums, const float *prods, float *state, const int *seq_start,
                                                                 const int *seq_slot, int n_heads, int dim, int chunk) {
    const int e = blockIdx.x * 256 + threadIdx.x, h = blockIdx.y, seq = blockIdx.z;
    pdl_wait();
    const int len = seq_start[seq + 1] - seq_start[seq];
    if (len <= 0 || e >= dim * dim) return;
    int first = 0;
    for (int q = 0; q < seq; q++) first += (seq_start[q + 1] - seq_start[q] + chunk - 1) / chunk;
    const int count = (len + chunk - 1) / chunk, d = e / dim;
    float *slot = state + ((long long)seq_slot[seq] * n_heads + h) * dim * dim + e;
    float S = *slot;
    for (int c0 = 0; c0 < count; c0 += 4) {
        float u[4], pr[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const long long at = (long long)(first + (c0 + i < count ? c0 + i : count - 1)) * n_heads + h;
            u[i] = sums[at * dim * dim + e], pr[i] = prods[at * dim + d];
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (c0 + i >= count) break;
            sums[((long long)(first + c0 + i) * n_heads + h) * dim * dim + e] = S;
            S = fmaf(pr[i], S, u[i]);
        }
    }
    *slot = S;
}

// ---------------------------------------------------------------- the recurrence, prompts: in blocks of four tokens
// With S the state before a block of four, G_i = w_1 .. w_i its decays up to token i (elementwise over the key channels) and
// G_ij = w_(j+1) .. w_i,
//     o_i = S^T (G_(i-1) r_i) + sum over j < i of [r_i . G_(i-1)j k_j] v_j + [r_i . u k_i] v_i,   S <- G_4 S + sum_j (G_4j k_j) v_j^T
// (decays multiplied, never divided). The nine vectors and ten numbers of a block know neither the state nor the values:
// four warps of the CTA make them, a block each, and put them into shared memory while the walking warps are at the four
// blocks before. What a walker does to the state is nine multiply-adds an element and four tokens (twelve token by token),
// two elements an instruction. P lanes share a value column, each with 4 J of its key channels (lane p: 4 p .. 4 p + 3 of
// every 4 P); a lane has C columns, and a piece of a vector it reads serves them all. Float32 throughout, the same numbers
// as token by token in another order of sums. Bound by instructions: a block costs a walker some 290 and a maker 600, and an
// SM with one CTA runs them at half its issue rate; 3 prompts, 3,571 tokens, 40 heads of 64: 245 us (segments walked twice
// token by token, with the states between them made from the segments' sums, took 480 + 253 + 42 us).
#define WB_TOKENS 4
#define WB_NUMBERS 12   // ten, and the next multiple of four
#define WB_WALKERS 4    // warps
#define WB_MAKERS 4     // warps, and blocks of a stage; two stages

template <int BYTES> struct WkvPiece;
template <> struct WkvPiece<2> { typedef uint16_t type; };
template <> struct WkvPiece<4> { typedef uint32_t type; };
template <> struct WkvPiece<8> { typedef uint2 type; };
template <> struct WkvPiece<16> { typedef uint4 type; };
struct __align__(16) WkvPiece32 { uint4 a, b; };
template <> struct WkvPiece<32> { typedef WkvPiece32 type; };
// N floats (1, 2, or a multiple of 4) as pieces of up to 16 bytes.
template <int N> __device__ __forceinline__ void wkv_load_floats(float *dst, const float *src) {
    if constexpr (N == 1) dst[0] = *src;
    else if constexpr (N == 2) *(float2 *)dst = *(const float2 *)src;
    else
#pragma unroll
        for (int i = 0; i < N; i += 4) *(float4 *)(dst + i) = *(const float4 *)(src + i);
}
template <int N> __device__ __forceinline__ void wkv_store_floats(float *dst, const float *src) {
    if constexpr (N == 1) *dst = src[0];
    else if constexpr (N == 2) *(float2 *)dst = make_float2(src[0], src[1]);
    else
#pragma unroll
        for (int i = 0; i < N; i += 4) *(float4 *)(dst + i) = make_float4(src[i], src[i + 1], src[i + 2], src[i + 3]);
}

template <typename T, int P, int J, int C>
__global__ void __launch_bounds__(32 * (WB_WALKERS + WB_MAKERS)) wkv_block_kernel(WkvScan p) {
    constexpr int DP = 4 * P * J, JL = DP / 32, COLS = WB_WALKERS * 32 / P * C, HEAD = 9 * DP + WB_NUMBERS, RS = HEAD + WB_TOKENS * COLS;
    extern __shared__ __align__(16) float wb_smem[];  // [2 stages][WB_MAKERS blocks][RS]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int h = blockIdx.x % p.n_heads, tile = blockIdx.x / p.n_heads % p.tiles, place = blockIdx.x / p.n_heads / p.tiles;
    const int col0 = tile * COLS, D = p.dim;
    const long long hk = (long long)p.n_heads * D;
    const bool makes = warp >= WB_WALKERS;
    float w0[JL], bonus[JL];
    if (makes) {
#pragma unroll
        for (int j = 0; j < JL; j++) {
            const int c = min(lane * JL + j, D - 1);
            w0[j] = p.w0[(long long)h * D + c], bonus[j] = p.bonus[(long long)h * D + c];  // weights: ahead of the wait
        }
    }
    pdl_wait();
    const int seq = p.longest_first ? sequence_place(p.seq_start, p.n_seqs, place) : place;
    const int row0 = p.seq_start[seq], n = p.seq_start[seq + 1] - row0;
    if (n <= 0) return;  // (a sequence of the step's padding: its slot is someone else's)
    const int n_blocks = (n + WB_TOKENS - 1) / WB_TOKENS, n_stages = (n_blocks + WB_MAKERS - 1) / WB_MAKERS;
    if (makes) {
        constexpr int VL = (WB_TOKENS * COLS + 31) / 32;  // values a lane brings
        typedef typename WkvPiece<sizeof(T) * JL>::type TPiece;
        const int mine = warp - WB_WALKERS;
        const int c_mine = lane * JL < D ? lane * JL : 0, k_from_r = p.k_at - p.r_at;  // (lanes beyond the head bring what is not used)
        const T *mine_proj = (const T *)p.proj + h * D + p.r_at + c_mine, *head_values = (const T *)p.proj + h * D + p.v_at;
        const float *mine_pre = p.pre + h * D + c_mine;
        struct __align__(16) Rows {  // a block's rows as they come
            T r_in[WB_TOKENS][JL], k_in[WB_TOKENS][JL];
            float z_in[WB_TOKENS][JL];
            T v_in[VL];
        } even, odd;
        auto ask = [&](Rows &w, int block) {
            if (block >= n_blocks) return;
            const int t0 = block * WB_TOKENS;
#pragma unroll
            for (int i = 0; i < WB_TOKENS; i++) {
                const long long row = row0 + min(t0 + i, n - 1);
                const T *src = mine_proj + row * p.ld;
                const float *z = mine_pre + row * hk;
                if (p.vec) {  // a lane's channels of a row as one piece
                    *(TPiece *)w.r_in[i] = *(const TPiece *)src, *(TPiece *)w.k_in[i] = *(const TPiece *)(src + k_from_r);
                    wkv_load_floats<JL>(w.z_in[i], z);
                } else {
#pragma unroll
                    for (int j = 0; j < JL; j++) {
                        const int c = min(lane * JL + j, D - 1) - c_mine;
                        w.r_in[i][j] = src[c], w.k_in[i][j] = src[k_from_r + c], w.z_in[i][j] = z[c];
                    }
                }
            }
#pragma unroll
            for (int e = 0; e < VL; e++) {
                const int at = lane + 32 * e, i = at / COLS, c = col0 + at % COLS;
                w.v_in[e] = head_values[(row0 + min(t0 + min(i, WB_TOKENS - 1), n - 1)) * p.ld + min(c, D - 1)];
            }
        };
        auto make = [&](const Rows &in, int block) {
            if (block >= n_blocks) return;
            float *rec = wb_smem + ((block / WB_MAKERS % 2) * WB_MAKERS + mine) * RS;
            const int count = min(WB_TOKENS, n - block * WB_TOKENS);
            float num[16], R[WB_TOKENS][JL], U[WB_TOKENS][JL], G[JL];
#pragma unroll
            for (int e = 0; e < 16; e++) num[e] = 0.0f;
#pragma unroll
            for (int j = 0; j < JL; j++) {
                const bool channel = lane * JL + j < D;
                G[j] = 1.0f;  // U[s]: G_(i-1)s k_s on the way
#pragma unroll
                for (int i = 0; i < WB_TOKENS; i++) {
                    const bool real = i < count && channel;
                    const float r = real ? to_float(in.r_in[i][j]) : 0.0f, k = real ? to_float(in.k_in[i][j]) : 0.0f;
                    const float w = real ? wkv_decay<T>(in.z_in[i][j] + w0[j]) : 1.0f;
                    R[i][j] = G[j] * r;
#pragma unroll
                    for (int s = 0; s < i; s++) {
                        num[i * (i + 1) / 2 + s] = fmaf(r, U[s][j], num[i * (i + 1) / 2 + s]);
                        U[s][j] *= w;
                    }
                    num[i * (i + 1) / 2 + i] = fmaf(r * bonus[j], k, num[i * (i + 1) / 2 + i]);
                    U[i][j] = k;
                    G[j] *= w;
                }
            }
#pragma unroll
            for (int i = 0; i < WB_TOKENS; i++)
                wkv_store_floats<JL>(rec + i * DP + lane * JL, R[i]), wkv_store_floats<JL>(rec + (4 + i) * DP + lane * JL, U[i]);
            wkv_store_floats<JL>(rec + 8 * DP + lane * JL, G);
            // the ten sums across the warp: half of a lane's handed over at each step, so that a pair of lanes ends with one
#pragma unroll
            for (int half = 8, bit = 16; half > 0; half >>= 1, bit >>= 1) {
                const bool up = lane & bit;
#pragma unroll
                for (int e = 0; e < half; e++) {
                    const float give = up ? num[e] : num[e + half], keep = up ? num[e + half] : num[e];
                    num[e] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
                }
            }
            num[0] += __shfl_xor_sync(0xffffffffu, num[0], 1);
            if (!(lane & 1) && (lane >> 1) < WB_NUMBERS) rec[9 * DP + (lane >> 1)] = num[0];  // (bit 16 counts eight, .., bit 2 one)
#pragma unroll
            for (int e = 0; e < VL; e++) {
                const int at = lane + 32 * e, i = at / COLS, c = col0 + at % COLS;
                if (at < WB_TOKENS * COLS) rec[HEAD + at] = i < count && c < D ? to_float(in.v_in[e]) : 0.0f;
            }
        };
        ask(even, mine);
        ask(odd, WB_MAKERS + mine);
        make(even, mine);
        for (int s = 0; s < n_stages; s++) {
            // stage s is made, and stage s - 1 has been read: its place is filled again, from rows asked for a stage ago
            __syncthreads();
            if (s & 1) ask(odd, (s + 2) * WB_MAKERS + mine), make(even, (s + 1) * WB_MAKERS + mine);
            else ask(even, (s + 2) * WB_MAKERS + mine), make(odd, (s + 1) * WB_MAKERS + mine);
        }
        return;
    }
    const int part = lane & (P - 1), own = tid / P * C, first_col = col0 + own;
    float *state = p.state + ((long long)p.seq_slot[seq] * p.n_heads + h) * D * D;
    f32x2 S[C][2 * J];
#pragma unroll
    for (int c = 0; c < C; c++)
#pragma unroll
        for (int j = 0; j < J; j++) {
            float v[4];
#pragma unroll
            for (int x = 0; x < 4; x++) {
                const int ch = 4 * (P * j + part) + x;
                v[x] = ch < D && first_col + c < D ? state[(long long)ch * D + first_col + c] : 0.0f;
            }
            S[c][2 * j] = pack2(v[0], v[1]), S[c][2 * j + 1] = pack2(v[2], v[3]);
        }
    constexpr int BITS = P == 16 ? 4 : 3, COL_STEPS = C == 4 ? 2 : C == 2 ? 1 : 0, TOK_STEPS = BITS - COL_STEPS < 2 ? BITS - COL_STEPS : 2;
    constexpr int REST = P >> (COL_STEPS + TOK_STEPS);  // lanes that end with the same sums
    const int my_c = part >> (BITS - COL_STEPS), my_t = (part / REST) & ((1 << TOK_STEPS) - 1);  // this lane's column and tokens
    const int my_col = first_col + my_c;
    float *out = p.out + (long long)row0 * hk + (long long)h * D + my_col;
    for (int s = 0; s < n_stages; s++) {
        __syncthreads();
#pragma unroll 1
        for (int b = 0; b < WB_MAKERS; b++) {
            const int left = n - (s * WB_MAKERS + b) * WB_TOKENS;
            if (left <= 0) break;
            const float *rec = wb_smem + ((s & 1) * WB_MAKERS + b) * RS, *vec = rec + 4 * part;
            float sums[C][4], vv[4][C];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                f32x2 a[C];
#pragma unroll
                for (int j = 0; j < J; j++) {
                    const ulonglong2 w = *(const ulonglong2 *)(vec + i * DP + 4 * P * j);
#pragma unroll
                    for (int c = 0; c < C; c++) {
                        a[c] = j == 0 ? mul2(w.x, S[c][0]) : fma2(w.x, S[c][2 * j], a[c]);
                        a[c] = fma2(w.y, S[c][2 * j + 1], a[c]);
                    }
                }
#pragma unroll
                for (int c = 0; c < C; c++) {
                    const float2 x = unpack2(a[c]);
                    sums[c][i] = x.x + x.y;
                }
                const float *vs = rec + HEAD + i * COLS + own;
                if constexpr (C == 4) {
                    const float4 x = *(const float4 *)vs;
                    vv[i][0] = x.x, vv[i][1] = x.y, vv[i][2] = x.z, vv[i][3] = x.w;
                } else if constexpr (C == 2) {
                    const float2 x = *(const float2 *)vs;
                    vv[i][0] = x.x, vv[i][1] = x.y;
                } else {
                    vv[i][0] = vs[0];
                }
            }
#pragma unroll
            for (int j = 0; j < J; j++) {
                const ulonglong2 w = *(const ulonglong2 *)(vec + 8 * DP + 4 * P * j);
#pragma unroll
                for (int c = 0; c < C; c++) S[c][2 * j] = mul2(w.x, S[c][2 * j]), S[c][2 * j + 1] = mul2(w.y, S[c][2 * j + 1]);
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                f32x2 vd[C];
#pragma unroll
                for (int c = 0; c < C; c++) vd[c] = pack2(vv[i][c], vv[i][c]);
#pragma unroll
                for (int j = 0; j < J; j++) {
                    const ulonglong2 w = *(const ulonglong2 *)(vec + (4 + i) * DP + 4 * P * j);
#pragma unroll
                    for (int c = 0; c < C; c++) S[c][2 * j] = fma2(w.x, vd[c], S[c][2 * j]), S[c][2 * j + 1] = fma2(w.y, vd[c], S[c][2 * j + 1]);
                }
            }
            // the sums across the column's lanes: columns handed over first, then tokens, then plain sums
#pragma unroll
            for (int step = 0; step < COL_STEPS; step++) {
                const int half = C >> (step + 1), bit = P >> (step + 1);
                const bool up = part & bit;
#pragma unroll
                for (int c = 0; c < half; c++)
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const float give = up ? sums[c][i] : sums[c + half][i], keep = up ? sums[c + half][i] : sums[c][i];
                        sums[c][i] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
                    }
            }
            // the block's own tokens, with the numbers: each lane for its column
            const float4 n0 = *(const float4 *)(rec + 9 * DP), n1 = *(const float4 *)(rec + 9 * DP + 4), n2 = *(const float4 *)(rec + 9 * DP + 8);
            float u[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                u[i] = vv[i][0];
#pragma unroll
                for (int c = 1; c < C; c++) u[i] = my_c == c ? vv[i][c] : u[i];
            }
            float add[4];
            add[0] = n0.x * u[0], add[1] = fmaf(n0.z, u[1], n0.y * u[0]), add[2] = fmaf(n1.y, u[2], fmaf(n1.x, u[1], n0.w * u[0]));
            add[3] = fmaf(n2.y, u[3], fmaf(n2.x, u[2], fmaf(n1.w, u[1], n1.z * u[0])));
            float o[4];
#pragma unroll
            for (int i = 0; i < 4; i++) o[i] = sums[0][i];
#pragma unroll
            for (int step = 0; step < TOK_STEPS; step++) {
                const int half = 2 >> step, bit = P >> (COL_STEPS + step + 1);
                const bool up = part & bit;
#pragma unroll
                for (int i = 0; i < half; i++) {
                    const float give = up ? o[i] : o[i + half], keep = up ? o[i + half] : o[i];
                    o[i] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
                    add[i] = up ? add[i + half] : add[i];
                }
            }
#pragma unroll
            for (int bit = REST >> 1; bit > 0; bit >>= 1)
#pragma unroll
                for (int i = 0; i < (4 >> TOK_STEPS); i++) o[i] += __shfl_xor_sync(0xffffffffu, o[i], bit);
            if ((part & (REST - 1)) == 0 && my_col < D) {
                constexpr int EACH = 4 >> TOK_STEPS;
#pragma unroll
                for (int i = 0; i < EACH; i++)
                    if (my_t * EACH + i < left) out[(my_t * EACH + i) * hk] = o[i] + add[i];
            }
            out += WB_TOKENS * hk;
        }
    }
#pragma unroll
    for (int c = 0; c < C; c++)
#pragma unroll
        for (int j = 0; j < J; j++) {
            const float2 x = unpack2(S[c][2 * j]), y = unpack2(S[c][2 * j + 1]);
            const float v[4] = {x.x, x.y, y.x, y.y};
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int ch = 4 * (P * j + part) + e;
                if (ch < D && first_col + c < D) state[(long long)ch * D + first_col + c] = v[e];
            }
        }
}

template <typename T, int P, int J, int C> static int wkv_block_launch(WkvScan p, cudaStream_t s) {
    constexpr int COLS = WB_WALKERS * 32 / P * C, RS = 9 * 4 * P * J + WB_NUMBERS + WB_TOKENS * COLS;
    size_t smem = (size_t)2 * WB_MAKERS * RS * sizeof(float);
    const long long sms = abk_sm_count();
    // a lane's JL channels of a row of r, k and the pre-activations as aligned pieces
    constexpr int JL = P * J / 8, BYTES = JL * (int)sizeof(T) > 16 ? 16 : JL * (int)sizeof(T), FLOATS = JL < 4 ? JL : 4;
    p.vec = p.dim % JL == 0 && (p.ld * sizeof(T)) % BYTES == 0 && !(((uintptr_t)p.proj + (size_t)p.r_at * sizeof(T)) % BYTES) &&
            !(((uintptr_t)p.proj + (size_t)p.k_at * sizeof(T)) % BYTES) && (p.dim * sizeof(T)) % BYTES == 0 &&
            !((uintptr_t)p.pre % (4 * FLOATS)) && p.dim % FLOATS == 0;
    p.tiles = (p.dim + COLS - 1) / COLS;
    const long long ctas = (long long)p.n_seqs * p.n_heads * p.tiles, share = (ctas + sms - 1) / sms;
    if (ctas > 0x7fffffffLL) ABK_REFUSE("wkv_scan: %lld CTAs are more than a grid takes", ctas);
    // CTAs that start while the kernel before still holds parts of the SMs gather where there is room: each asks for so much
    // shared memory that no SM takes more than its share
    const size_t least = share <= 4 ? (size_t)(228 * 1024 / (share + 1)) : 0;
    if (smem < least) smem = least;
    p.longest_first = p.n_seqs > 1 && p.n_seqs <= SEQUENCE_PLACE_MAX && share > 1;  // (a long walk that starts last would be walked alone)
    const cudaError_t e = abk_allow_shared_memory((const void *)wkv_block_kernel<T, P, J, C>, (int)smem);
    if (e != cudaSuccess) return (int)e;
    abk_launch(wkv_block_kernel<T, P, J, C>, dim3((unsigned)ctas), dim3(32 * (WB_WALKERS + WB_MAKERS)), smem, s, p);
    return ABK_LAUNCH_RESULT();
}

enum { WKV_TOKENS, WKV_BLOCKS, WKV_SEGMENTS, WKV_STEP };
// form: token by token; in blocks of four tokens; in segments of `chunk` tokens (`segments` of them at most, with room for their
// sums and products); or a step of one token a sequence.
extern "C" int abk_wkv_scan(const void *proj, long long ld, int dtype, int r_at, int k_at, int v_at, int n_heads, int dim,
                            const float *pre, const float *w0, const float *bonus, float *state, float *out,
                            const int *seq_start, const int *seq_slot, int n_seqs, int form, int chunk, int segments, float *sums,
                            float *prods, void *stream) {
    if (n_seqs <= 0) return 0;
    if (dim < 1 || dim > 256) ABK_REFUSE("wkv_scan: %d key channels a head are not 1 to 256", dim);
    if (n_heads < 1 || n_heads > 65535 || n_seqs > 65535) ABK_REFUSE("wkv_scan: %d heads, %d sequences", n_heads, n_seqs);
    WkvScan p;
    p.proj = proj, p.ld = ld, p.r_at = r_at, p.k_at = k_at, p.v_at = v_at, p.n_heads = n_heads, p.dim = dim;
    p.pre = pre, p.w0 = w0, p.bonus = bonus, p.state = state, p.out = out, p.seq_start = seq_start, p.seq_slot = seq_slot;
    p.n_seqs = n_seqs, p.tiles = 1, p.longest_first = 0, p.vec = 0, p.chunk = chunk, p.sums = sums, p.prods = prods;
    if (form < WKV_TOKENS || form > WKV_STEP) ABK_REFUSE("wkv_scan: form %d is not built", form);
    if (form == WKV_SEGMENTS && (chunk < 1 || segments < 1 || segments > 65535 || !sums || !prods))
        ABK_REFUSE("wkv_scan: %d segments of %d tokens", segments, chunk);
    cudaStream_t s = (cudaStream_t)stream;
    if (form == WKV_BLOCKS) {
        // Columns a lane has: as few as leave an SM one CTA, else as many as a head uses. The makers' work is every CTA's own,
        // and an SM's CTAs share its issue slots. One prompt of 500, us a walk with 1, 2, 4: 40 heads of 64 65, 54, 61 (160,
        // 80, 40 CTAs), 16 heads of 64 44, 54, 61, 32 heads of 128 261, 162, 87, 16 of 256 484, 254, 142, 80 of 32 46, 37, 53;
        // 500, 1,023 and 2,048 tokens, 40 heads of 64: 253, 271, 241; 8 prompts of 500: 312, 206, 152.
        const int each = dim <= 64 ? 16 : 8;  // columns a CTA has where a lane has one
        const long long heads = (long long)n_seqs * n_heads, sms = abk_sm_count();
        int lane_columns = 1;
        while (lane_columns < 4 && lane_columns * each < dim && heads * ((dim + lane_columns * each - 1) / (lane_columns * each)) > sms) lane_columns *= 2;
#define WB_LAUNCH_AS(T, P, J)                                     \
    (lane_columns == 1   ? wkv_block_launch<T, P, J, 1>(p, s)     \
     : lane_columns == 2 ? wkv_block_launch<T, P, J, 2>(p, s)     \
                         : wkv_block_launch<T, P, J, 4>(p, s))
#define WB_LAUNCH(T)                                              \
    (dim <= 32    ? WB_LAUNCH_AS(T, 8, 1)                         \
     : dim <= 64  ? WB_LAUNCH_AS(T, 8, 2)                         \
     : dim <= 128 ? WB_LAUNCH_AS(T, 16, 2)                        \
                  : WB_LAUNCH_AS(T, 16, 4))
        return dtype == ABK_BF16 ? WB_LAUNCH(__nv_bfloat16) : WB_LAUNCH(float);
#undef WB_LAUNCH
#undef WB_LAUNCH_AS
    }
    if (form == WKV_STEP) {
        const bool pieces = dim % 4 == 0 && !((uintptr_t)state & 15);
        const int wide = dim <= 32 ? 32 : 64;
        const dim3 tiles((dim + wide - 1) / wide, n_heads, n_seqs);
#define WST_LAUNCH_AS(T, LPR, ROWS)                                                                      \
    do {                                                                                                 \
        if (pieces) abk_launch(wkv_step_kernel<T, LPR, ROWS, true>, tiles, dim3(16 * LPR), 0, s, p);     \
        else abk_launch(wkv_step_kernel<T, LPR, ROWS, false>, tiles, dim3(16 * LPR), 0, s, p);           \
    } while (0)
#define WST_LAUNCH(LPR, ROWS)                                       \
    do {                                                            \
        if (dtype == ABK_BF16) WST_LAUNCH_AS(__nv_bfloat16, LPR, ROWS); \
        else WST_LAUNCH_AS(float, LPR, ROWS);                       \
    } while (0)
        if (dim <= 32) WST_LAUNCH(8, 2);
        else if (dim <= 64) WST_LAUNCH(16, 4);
        else if (dim <= 128) WST_LAUNCH(16, 8);
        else WST_LAUNCH(16, 16);
#undef WST_LAUNCH
#undef WST_LAUNCH_AS
        return ABK_LAUNCH_RESULT();
    }
    const int cols = dim <= 32 ? 32 : 16;  // value columns a CTA has
    dim3 grid((dim + cols - 1) / cols, n_heads, form == WKV_SEGMENTS ? segments : n_seqs);
#define WS_LAUNCH_AS(T, PHASE)                                                                               \
    do {                                                                                                     \
        if (dim <= 16) abk_launch(wkv_scan_kernel<T, 4, 4, 32, 16, PHASE>, grid, dim3(128), 0, s, p);        \
        else if (dim <= 32) abk_launch(wkv_scan_kernel<T, 8, 4, 32, 16, PHASE>, grid, dim3(128), 0, s, p);   \
        else if (dim <= 64) abk_launch(wkv_scan_kernel<T, 8, 8, 16, 16, PHASE>, grid, dim3(128), 0, s, p);   \
        else if (dim <= 128) abk_launch(wkv_scan_kernel<T, 8, 16, 16, 16, PHASE>, grid, dim3(256), 0, s, p); \
        else abk_launch(wkv_scan_kernel<T, 16, 16, 16, 8, PHASE>, grid, dim3(256), 0, s, p);                 \
    } while (0)
#define WS_LAUNCH(PHASE)                                        \
    do {                                                        \
        if (dtype == ABK_BF16) WS_LAUNCH_AS(__nv_bfloat16, PHASE); \
        else WS_LAUNCH_AS(float, PHASE);                        \
    } while (0)
    if (form != WKV_SEGMENTS) {
        WS_LAUNCH(0);
        return ABK_LAUNCH_RESULT();
    }
    WS_LAUNCH(1);  // the segments' sums, the states between them, the segments' outputs
    int rc = ABK_LAUNCH_RESULT();
    if (rc) return rc;
    abk_launch(wkv_segment_prefix_kernel, dim3((dim * dim + 255) / 256, n_heads, n_seqs), dim3(256), 0, s, sums, prods, state,
               seq_start, seq_slot, n_heads, dim, chunk);
    rc = ABK_LAUNCH_RESULT();
    if (rc) return rc;
    WS_LAUNCH(2);
#undef WS_LAUNCH
#undef WS_LAUNCH_AS
    return ABK_LAUNCH_RESULT();
}
