// The gated delta rule with a decay per key channel, as a recurrent mixer: the short causal convolution in
// front of it, the recurrence over a per-sequence state, and the gated per-head norm behind it.
//
// Per head, with a state S [key, value] in float32 that starts at zero and is carried from token to token:
//     S <- diag(g) S;   e = b (v - S^T k);   S <- S + k e^T;   o = S^T q
// q and k are unit vectors per head (x / sqrt(sum x^2 + 1e-6)), q also times key^-1/2; b = sigmoid(.) per head;
// g = exp(-exp(A) * softplus(a + bias)) per head and key channel (or, per_head, one for all of a head's channels).
// The convolution may also stand alone, without its SiLU (plain). Everything that enters the recurrence is
// float32; q, k and v come from the convolution in the model's storage type.
//
// A value column of S never meets another: column j needs S[:, j], v_j and the token's q, k, g, b. So a thread
// keeps (a part of) one column in registers and walks the sequence in order: prompts in blocks of four tokens, whose
// vectors a kernel makes ahead of the walk, and a step of one token a sequence in one kernel with its preparation. The
// state is stored [head, value, key], so a column is one contiguous run.
#define ABK_DEFINE_ERROR
#include "recurrence.cuh"

#define CONV_MAX_TAPS 8

// ------------------------------------------------------------------ short convolution + SiLU
// out[t, c] = silu(sum_j w[c, j] * in[position(t) - (taps - 1 - j), c]); inputs before the sequence's start are
// zero, inputs before this step's rows come from the slot's tail [taps - 1, channels] (the last inputs of the
// steps before). in: the first `channels` columns of rows of `ld` elements.
struct ShortConv {
    const void *in;
    long long ld;
    void *out;          // [tokens, channels]
    const float *w;     // [channels, taps]
    const float *tail;  // [slots, taps - 1, channels]
    const int *token_seq, *token_pos, *seq_slot, *seq_pos0;
    int channels, taps, n_tokens;
    float *new_tail;       // a step of one token a sequence: the kernel leaves the slot's new tail itself (the thread that
                           // read a channel's old tail writes its new one); null: short_conv_tail does it
    int plain;             // 1: the sum as it is, no SiLU behind it
};

template <typename T> __global__ void __launch_bounds__(128) short_conv_kernel(ShortConv p) {
    pdl_wait();
    const int t = blockIdx.x;
    const int c = blockIdx.y * blockDim.x + threadIdx.x;
    if (c >= p.channels) return;
    T *out = (T *)p.out + (long long)t * p.channels + c;
    const int seq = p.token_seq[t];
    if (seq < 0) {
        *out = from_float<T>(0.0f);
        return;
    }
    const int pos = p.token_pos[t], pos0 = p.seq_pos0[seq], taps = p.taps;
    const float *w = p.w + (long long)c * taps;
    const float *tail = p.tail + (long long)p.seq_slot[seq] * (taps - 1) * p.channels + c;
    float acc = 0.0f;
    float *left = p.new_tail ? p.new_tail + (long long)p.seq_slot[seq] * (taps - 1) * p.channels + c : nullptr;
    for (int j = 0; j < taps; j++) {
        const int back = taps - 1 - j, at = pos - back;
        float v = 0.0f;
        if (at >= pos0) v = to_float(((const T *)p.in)[(long long)(t - back) * p.ld + c]);
        else if (at >= 0) v = tail[(long long)(at - (pos0 - (taps - 1))) * p.channels];
        if (left && j > 0) left[(long long)(j - 1) * p.channels] = v;  // the input `back` tokens ago is back + 1 ago next time
        acc = fmaf(w[j], v, acc);
    }
    *out = from_float<T>(p.plain ? acc : silu_f(acc));
}

// The same with VEC channels a thread (16 bytes of the storage type), for channel counts and row pitches that are
// multiples of VEC with everything 16-byte aligned, for 2 to 4 taps. A thread has TOKENS tokens of its channels: the weights and
// the rows that its tokens share are read once, and all of its loads are in flight together. Long steps take four tokens (two in
// float32, and from 2,400 CTAs on two such turns, the weights read once for both: 5,672 tokens of 4,096 float32 channels 50 us, with one turn
// 60, token by token 58; 1,024 of 1,024, 1,024 CTAs, 4.5, 4.1 and 5.6), short ones one: 1,016 tokens of 4,096 bfloat16 channels by one
// 21 us, 1,024 by four 11; float32 15 and 11. 1,999 tokens of 4,096 bfloat16 channels, four taps: 20.4 us, 5,672 tokens 57; with each token's rows fetched
// one token after the other, and the division in full, 23.1 and 60.
#define CONV_TOKENS 4
template <typename T, int VEC> struct ConvVector;
template <> struct ConvVector<__nv_bfloat16, 8> {
    static __device__ __forceinline__ void open(uint4 raw, float *v) {
        const __nv_bfloat162 *h = (const __nv_bfloat162 *)&raw;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const float2 f = __bfloat1622float2(h[u]);
            v[2 * u] = f.x, v[2 * u + 1] = f.y;
        }
    }
    static __device__ __forceinline__ void store(__nv_bfloat16 *p, const float *v) {
        uint4 raw;
        __nv_bfloat162 *h = (__nv_bfloat162 *)&raw;
#pragma unroll
        for (int u = 0; u < 4; u++) h[u] = __floats2bfloat162_rn(v[2 * u], v[2 * u + 1]);
        *(uint4 *)p = raw;
    }
};
template <> struct ConvVector<float, 4> {
    static __device__ __forceinline__ void open(uint4 raw, float *v) {
        v[0] = __uint_as_float(raw.x), v[1] = __uint_as_float(raw.y), v[2] = __uint_as_float(raw.z), v[3] = __uint_as_float(raw.w);
    }
    static __device__ __forceinline__ void store(float *p, const float *v) { *(float4 *)p = make_float4(v[0], v[1], v[2], v[3]); }
};

template <typename T, int VEC, int TAPS, int TOKENS, int TURNS> __global__ void __launch_bounds__(128) short_conv_vec_kernel(ShortConv p) {
    const int c = (blockIdx.y * blockDim.x + threadIdx.x) * VEC;
    float w[VEC * TAPS];  // this thread's weights lie together: VEC channels of TAPS taps, a multiple of 16 bytes
    if (c < p.channels) {
#pragma unroll
        for (int i = 0; i < VEC * TAPS / 4; i++) {
            const float4 f = *(const float4 *)(p.w + (long long)c * TAPS + 4 * i);  // weights: ahead of the wait
            w[4 * i] = f.x, w[4 * i + 1] = f.y, w[4 * i + 2] = f.z, w[4 * i + 3] = f.w;
        }
    }
    pdl_wait();
    if (c >= p.channels) return;
    for (int turn = 0; turn < TURNS; turn++) {
        const int t0 = (blockIdx.x * TURNS + turn) * TOKENS;
        if (t0 >= p.n_tokens) return;
        int seq[TOKENS], pos[TOKENS], pos0[TOKENS];
        uint4 rows[TOKENS + TAPS - 1];  // rows t0 - (TAPS - 1) .. t0 + TOKENS - 1 of the step
#pragma unroll
        for (int i = 0; i < TOKENS; i++) {
            seq[i] = t0 + i < p.n_tokens ? p.token_seq[t0 + i] : -1;
            pos[i] = t0 + i < p.n_tokens ? p.token_pos[t0 + i] : 0;
        }
#pragma unroll
        for (int i = 0; i < TOKENS + TAPS - 1; i++) {
            const int t = t0 + i - (TAPS - 1);
            rows[i] = make_uint4(0, 0, 0, 0);
            if (t >= 0 && t < p.n_tokens) rows[i] = *(const uint4 *)((const T *)p.in + (long long)t * p.ld + c);
        }
#pragma unroll
        for (int i = 0; i < TOKENS; i++) pos0[i] = seq[i] >= 0 ? p.seq_pos0[seq[i]] : 0;
#pragma unroll
        for (int i = 0; i < TOKENS; i++) {
            if (t0 + i >= p.n_tokens) break;
            float acc[VEC];
#pragma unroll
            for (int u = 0; u < VEC; u++) acc[u] = 0.0f;
            if (seq[i] >= 0) {
                const float *tail = p.tail + (p.new_tail || pos[i] - pos0[i] < TAPS - 1 ? (long long)p.seq_slot[seq[i]] * (TAPS - 1) * p.channels + c : 0);
#pragma unroll
                for (int j = 0; j < TAPS; j++) {
                    const int back = TAPS - 1 - j, at = pos[i] - back;
                    float v[VEC];
                    if (at >= pos0[i]) ConvVector<T, VEC>::open(rows[i + j], v);
                    else if (at >= 0) {
#pragma unroll
                        for (int u = 0; u < VEC; u++) v[u] = tail[(long long)(at - (pos0[i] - (TAPS - 1))) * p.channels + u];
                    } else {
#pragma unroll
                        for (int u = 0; u < VEC; u++) v[u] = 0.0f;
                    }
                    if (p.new_tail && j > 0) {  // the input `back` tokens ago is back + 1 ago next time
                        float *left = p.new_tail + (long long)p.seq_slot[seq[i]] * (TAPS - 1) * p.channels + (long long)(j - 1) * p.channels + c;
#pragma unroll
                        for (int u = 0; u < VEC; u++) left[u] = v[u];
                    }
#pragma unroll
                    for (int u = 0; u < VEC; u++) acc[u] = fmaf(w[u * TAPS + j], v[u], acc[u]);
                }
#pragma unroll
                for (int u = 0; u < VEC; u++) acc[u] = p.plain ? acc[u] : silu_f(acc[u]);
            }
            ConvVector<T, VEC>::store((T *)p.out + (long long)(t0 + i) * p.channels + c, acc);
        }
    }
}

// update_tail: every sequence of the step brings one token, and the kernel leaves the slots' new tails itself.
extern "C" int abk_short_conv(const void *in, long long ld, void *out, int dtype, const float *w, float *tail,
                              const int *token_seq, const int *token_pos, const int *seq_slot, const int *seq_pos0,
                              int n_tokens, int channels, int taps, int update_tail, int plain, void *stream) {
    if (n_tokens <= 0 || channels <= 0) return 0;
    if (taps < 1 || taps > CONV_MAX_TAPS) ABK_REFUSE("short convolution: %d taps, the kernel takes 1 to %d", taps, CONV_MAX_TAPS);
    ShortConv p;
    p.in = in, p.ld = ld, p.out = out, p.w = w, p.tail = tail, p.token_seq = token_seq, p.token_pos = token_pos;
    p.seq_slot = seq_slot, p.seq_pos0 = seq_pos0, p.channels = channels, p.taps = taps, p.n_tokens = n_tokens;
    p.plain = plain;
    p.new_tail = update_tail && taps > 1 ? tail : nullptr;
    dim3 grid(n_tokens, (channels + 127) / 128);
    if (grid.y > 65535) ABK_REFUSE("short convolution: %d channels are more than a grid takes", channels);
    cudaStream_t s = (cudaStream_t)stream;
    const int vec = dtype == ABK_BF16 ? 8 : 4;
    if (channels % vec == 0 && ld % vec == 0 && taps >= 2 && taps <= 4 && !(((uintptr_t)in | (uintptr_t)out | (uintptr_t)w) & 15)) {
        const int strips = (channels / vec + 127) / 128, many = n_tokens < 1024 ? 1 : dtype == ABK_BF16 ? CONV_TOKENS : CONV_TOKENS / 2;
        const int turns = dtype == ABK_F32 && many > 1 && (long long)n_tokens / many * strips >= 2400 ? 2 : 1;
        dim3 tiles((n_tokens + many * turns - 1) / (many * turns), strips);
#define CONV_AS(T, VEC, TAPS, TOKENS, TURNS) abk_launch(short_conv_vec_kernel<T, VEC, TAPS, TOKENS, TURNS>, tiles, dim3(128), 0, s, p)
#define CONV_LAUNCH(TAPS)                                                   \
    if (dtype == ABK_BF16) {                                                \
        if (many == 1) CONV_AS(__nv_bfloat16, 8, TAPS, 1, 1);               \
        else CONV_AS(__nv_bfloat16, 8, TAPS, CONV_TOKENS, 1);               \
    } else {                                                                \
        if (many == 1) CONV_AS(float, 4, TAPS, 1, 1);                       \
        else if (turns == 1) CONV_AS(float, 4, TAPS, CONV_TOKENS / 2, 1);   \
        else CONV_AS(float, 4, TAPS, CONV_TOKENS / 2, 2);                   \
    }
        if (taps == 2) { CONV_LAUNCH(2) } else if (taps == 3) { CONV_LAUNCH(3) } else { CONV_LAUNCH(4) }
#undef CONV_LAUNCH
#undef CONV_AS
        return ABK_LAUNCH_RESULT();
    }
    if (dtype == ABK_BF16) abk_launch(short_conv_kernel<__nv_bfloat16>, grid, dim3(128), 0, s, p);
    else abk_launch(short_conv_kernel<float>, grid, dim3(128), 0, s, p);
    return ABK_LAUNCH_RESULT();
}

// The tails after the step: for every sequence and channel the last taps - 1 inputs, from this step's rows and,
// where the step brought fewer, from the old tail moved up. One thread reads all it needs before it writes.
template <typename T>
__global__ void short_conv_tail_kernel(const T *in, long long ld, float *tail, const int *seq_start, const int *seq_slot,
                                       const int *seq_pos0, int n_seqs, int channels, int taps) {
    pdl_wait();
    const int i = blockIdx.y, c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= channels || i >= n_seqs) return;
    const int row0 = seq_start[i], n = seq_start[i + 1] - row0;
    if (n <= 0) return;
    float *mine = tail + (long long)seq_slot[i] * (taps - 1) * channels + c;
    float keep[CONV_MAX_TAPS];
    for (int a = 0; a < taps - 1; a++) {
        const int back = taps - 1 - a;  // this place holds the input `back` tokens before the next one
        if (back <= n) keep[a] = to_float(in[(long long)(row0 + n - back) * ld + c]);
        else keep[a] = seq_pos0[i] + n - back >= 0 ? mine[(long long)(a + n) * channels] : 0.0f;
    }
    for (int a = 0; a < taps - 1; a++) mine[(long long)a * channels] = keep[a];
}

extern "C" int abk_short_conv_tail(const void *in, long long ld, int dtype, float *tail, const int *seq_start,
                                   const int *seq_slot, const int *seq_pos0, int n_seqs, int channels, int taps,
                                   void *stream) {
    if (n_seqs <= 0 || channels <= 0 || taps <= 1) return 0;
    if (taps > CONV_MAX_TAPS) ABK_REFUSE("short convolution: %d taps, the kernel takes 1 to %d", taps, CONV_MAX_TAPS);
    if (n_seqs > 65535) ABK_REFUSE("short convolution: %d sequences are more than a grid takes", n_seqs);
    dim3 grid((channels + 127) / 128, n_seqs);
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == ABK_BF16)
        abk_launch(short_conv_tail_kernel<__nv_bfloat16>, grid, dim3(128), 0, s, (const __nv_bfloat16 *)in, ld, tail,
                   seq_start, seq_slot, seq_pos0, n_seqs, channels, taps);
    else
        abk_launch(short_conv_tail_kernel<float>, grid, dim3(128), 0, s, (const float *)in, ld, tail, seq_start, seq_slot,
                   seq_pos0, n_seqs, channels, taps);
    return ABK_LAUNCH_RESULT();
}

// ------------------------------------------------------------------ the tokens' records of the chunked form
// Every (token, head) is prepared in parallel, a warp each: the unit vectors q and k (q times key^-1/2), the decays g, the
// value row and the write strength b, as one float32 record
//     [ k | q | g | v (vp) | b, 0, 0, 0 ]     vp = the value size padded to a multiple of 4
// in which k, q and g each lie as `parts` runs of 32 channels with 4 floats of padding behind each run (zeros
// beyond the key size; parts = 1, 2, 4 or 8).
#define SCAN_ROWS 32    // key channels of a run
#define SCAN_RUN 36     // with its padding

static inline int delta_parts(int key) { return key <= 32 ? 1 : key <= 64 ? 2 : key <= 128 ? 4 : 8; }
static inline int delta_record_floats(int key, int value) { return 3 * delta_parts(key) * SCAN_RUN + ((value + 3) & ~3) + 4; }

struct DeltaPrepare {
    const void *qkv;        // [tokens, ld_qkv]: q heads (kv_heads x key), k heads, v heads (heads x value), after the convolution
    long long ld_qkv;
    const void *decay_in;   // row t at decay_in + t * ld_decay, heads * key float32: a, before bias and softplus; with
    long long ld_decay;     // per_head: one a per head, `heads` of them in the storage type, and dt_bias [heads]
    int per_head;
    const void *beta_in;    // row t, head h at beta_in[t * ld_beta + h], before the sigmoid
    long long ld_beta;
    const float *a_log;     // [heads]
    const float *dt_bias;   // [heads * key]
    float *records;         // [tokens, heads, record] (or, of blocks of tokens, [blocks, heads, record])
    const int *token_seq;
    long long pairs;        // tokens (or blocks) * heads
    int heads, kv_heads, key, value, parts, record;
    float q_scale;          // key^-1/2
};

__device__ __forceinline__ float softplus_f(float z) { return z > 20.0f ? z : log1pf(expf(z)); }

template <typename T> __global__ void __launch_bounds__(128) delta_prepare_kernel(DeltaPrepare p) {
    const long long pair = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    pdl_wait();
    if (pair >= p.pairs) return;
    const long long row = pair / p.heads;
    const int h = (int)(pair - row * p.heads), K = p.key, V = p.value, region = p.parts * SCAN_RUN;
    float *rec = p.records + pair * p.record;
    if (p.token_seq[row] < 0) return;  // padding: its record is never read
    const int kvh = h / (p.heads / p.kv_heads);
    const T *qr = (const T *)p.qkv + row * p.ld_qkv + (long long)kvh * K;
    const T *kr = qr + (long long)p.kv_heads * K;
    const T *vr = (const T *)p.qkv + row * p.ld_qkv + 2LL * p.kv_heads * K + (long long)h * V;
    const float rate = expf(p.a_log[h]);
    // one decay for all of the head's key channels (the chunked form takes no others)
    const float head_decay = expf(-rate * softplus_f(to_float(((const T *)p.decay_in)[row * p.ld_decay + h]) + p.dt_bias[h]));
    float qq = 0.0f, kk = 0.0f;
    for (int i = lane; i < K; i += 32) {
        const float qv = to_float(qr[i]), kv = to_float(kr[i]);
        qq = fmaf(qv, qv, qq), kk = fmaf(kv, kv, kk);
    }
    qq = warp_sum(qq), kk = warp_sum(kk);
    const float qn = p.q_scale / sqrtf(qq + 1e-6f), kn = 1.0f / sqrtf(kk + 1e-6f);
    for (int at = lane; at < region; at += 32) {  // a place within a region: run at / 36, channel at % 36 of it
        const int i = (at / SCAN_RUN) * SCAN_ROWS + at % SCAN_RUN;
        const bool real = at % SCAN_RUN < SCAN_ROWS && i < K;
        rec[at] = real ? to_float(kr[i]) * kn : 0.0f;
        rec[region + at] = real ? to_float(qr[i]) * qn : 0.0f;
        rec[2 * region + at] = real ? head_decay : 0.0f;
    }
    const int vp = p.record - 3 * region - 4;
    for (int j = lane; j < vp; j += 32) rec[3 * region + j] = j < V ? to_float(vr[j]) : 0.0f;
    if (lane < 4) {
        const float z = to_float(((const T *)p.beta_in)[row * p.ld_beta + h]);
        rec[3 * region + vp + lane] = lane == 0 ? 1.0f / (1.0f + expf(-z)) : 0.0f;
    }
}

struct DeltaScan {
    const float *records;   // the step's records: a token's and head's (chunks), or a block's and head's
    float *state;           // [slots, heads, value, key]
    float *out;             // [tokens, heads * value]
    const int *seq_start, *seq_slot;
    int heads, key, value, parts, record;
    int n_seqs, tiles, longest_first;  // of the blocks' walk
    int vec;                // the state's columns are read and written as 16-byte pieces (aligned, a multiple of 4 channels)
};

// ------------------------------------------------------------------ the recurrence, token by token and in blocks of 4
// What the token-by-token walk waits for is the chain state -> sum over the key channels -> e -> state: with the sums
// crossing lanes it is some 150 cycles a token whatever the arithmetic. Four tokens unrolled take the chain once. With S
// the state before them, G_i = g_1 .. g_i the decays up to token i (elementwise over the key channels) and
// G_ij = g_(j+1) .. g_i, everything the block reads of S are eight vectors' products with it, all at once:
//     e_i = b_i (v_i - S^T (G_i k_i) - sum over j < i of [k_i . G_ij k_j] e_j)
//     o_i =          S^T (G_i q_i) + sum over j <= i of [q_i . G_ij k_j] e_j      S <- G_4 S + sum over j of (G_4j k_j) e_j^T
// (decays multiplied, never divided: every factor is at most 1). The vectors and the sixteen numbers in brackets know
// neither the state nor the values: delta_block_prepare makes them for all blocks side by side, and delta_block_scan walks
// the blocks. 13 multiply-adds a state element and 4 tokens where the walk token by token takes 16. Float32 throughout, the
// same numbers in another order of sums.
#define DB_TOKENS 4
#define DB_STAGE 2     // blocks that come in together
#define DB_STAGES 3    // of those in flight or in use

static inline int delta_pad_key(int key) { return key <= 32 ? 32 : key <= 64 ? 64 : key <= 128 ? 128 : 256; }
// A block's record, float32: [G_i k_i] x 4, [G_i q_i] x 4, [G_4j k_j] x 4, G_4 (each of the padded key size, zeros, or in
// G_4 ones, beyond the key size), then b_i [k_i . G_ij k_j] (10, 20, 21, 30, 31, 32), [q_i . G_ij k_j] (00, 10, 11, 20 .. 33),
// b (4), then the values [4][vp].
#define DB_NUMBERS 20
static inline long long delta_block_floats(int key, int value) { return 13LL * delta_pad_key(key) + DB_NUMBERS + DB_TOKENS * ((value + 3) & ~3); }

// Which sequence has the step's block `b`, and which rows: whole warps call it. False: no sequence has.
template <int TOKENS> __device__ __forceinline__ bool delta_block_locate(const int *seq_start, int n_seqs, int b, int &row0, int &count) {
    const int lane = threadIdx.x & 31;
    for (int base = 0; base < n_seqs; base += 32) {
        const int q = base + lane;
        const int first = q < n_seqs ? seq_start[q] : 0, n = q < n_seqs ? seq_start[q + 1] - first : 0;
        const int blocks = n > 0 ? (n + TOKENS - 1) / TOKENS : 0;
        int upto = blocks;
#pragma unroll
        for (int m = 1; m < 32; m <<= 1) {
            const int other = __shfl_up_sync(0xffffffffu, upto, m);
            if (lane >= m) upto += other;
        }
        const unsigned hit = __ballot_sync(0xffffffffu, b < upto);
        if (hit) {
            const int src = __ffs(hit) - 1;
            const int at = (b - (upto - blocks)) * TOKENS;
            row0 = __shfl_sync(0xffffffffu, first + at, src);
            count = __shfl_sync(0xffffffffu, min(TOKENS, n - at), src);
            return true;
        }
        b -= __shfl_sync(0xffffffffu, upto, 31);
    }
    return false;
}

// A warp a (block, head); a lane has the channels lane, lane + 32, .. Every load is made before the first use.
template <typename T, int J, bool PER_HEAD> __global__ void __launch_bounds__(128) delta_block_prepare_kernel(DeltaPrepare p, const int *seq_start, int n_seqs) {
    constexpr int DP = 32 * J;
    const long long pair = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    pdl_wait();
    if (pair >= p.pairs) return;
    const int b = (int)(pair / p.heads), h = (int)(pair - (long long)b * p.heads), K = p.key, V = p.value;
    int row0, count;
    if (!delta_block_locate<DB_TOKENS>(seq_start, n_seqs, b, row0, count)) return;
    float *rec = p.records + pair * p.record;
    const int kvh = h / (p.heads / p.kv_heads);
    T q_in[DB_TOKENS][J], k_in[DB_TOKENS][J], b_in[DB_TOKENS], h_in[DB_TOKENS];
    float d_in[DB_TOKENS][J], bias[J];
#pragma unroll
    for (int i = 0; i < DB_TOKENS; i++) {
        const long long row = row0 + min(i, count - 1);
        const T *qr = (const T *)p.qkv + row * p.ld_qkv + (long long)kvh * K, *kr = qr + (long long)p.kv_heads * K;
#pragma unroll
        for (int j = 0; j < J; j++) {
            const int c = min(lane + 32 * j, K - 1);
            q_in[i][j] = qr[c], k_in[i][j] = kr[c];
            if (!PER_HEAD) d_in[i][j] = ((const float *)p.decay_in)[row * p.ld_decay + (long long)h * K + c];
        }
        b_in[i] = ((const T *)p.beta_in)[row * p.ld_beta + h];
        if (PER_HEAD) h_in[i] = ((const T *)p.decay_in)[row * p.ld_decay + h];
    }
#pragma unroll
    for (int j = 0; j < J; j++) bias[j] = PER_HEAD ? p.dt_bias[h] : p.dt_bias[h * K + min(lane + 32 * j, K - 1)];
    const float rate = expf(p.a_log[h]);
    const int vp = (V + 3) & ~3;
    float *vals = rec + 13 * DP + DB_NUMBERS;
#pragma unroll
    for (int i = 0; i < DB_TOKENS; i++) {
        const T *vr = (const T *)p.qkv + (long long)(row0 + min(i, count - 1)) * p.ld_qkv + 2LL * p.kv_heads * K + (long long)h * V;
        for (int j = lane; j < vp; j += 32) vals[i * vp + j] = i < count && j < V ? to_float(vr[j]) : 0.0f;
    }
    float q[DB_TOKENS][J], k[DB_TOKENS][J], g[DB_TOKENS][J], beta[DB_TOKENS];
#pragma unroll
    for (int i = 0; i < DB_TOKENS; i++) {
        const bool real = i < count;
        float qq = 0.0f, kk = 0.0f, head_decay = 1.0f;
        if (PER_HEAD) head_decay = expf(-rate * softplus_f(to_float(h_in[i]) + bias[0]));
#pragma unroll
        for (int j = 0; j < J; j++) {
            const bool in = real && lane + 32 * j < K;
            q[i][j] = in ? to_float(q_in[i][j]) : 0.0f, k[i][j] = in ? to_float(k_in[i][j]) : 0.0f;
            const float decay = PER_HEAD ? head_decay : expf(-rate * softplus_f(d_in[i][j] + bias[j]));
            g[i][j] = in ? decay : 1.0f;
            qq = fmaf(q[i][j], q[i][j], qq), kk = fmaf(k[i][j], k[i][j], kk);
        }
        qq = warp_sum(qq), kk = warp_sum(kk);
        const float qn = p.q_scale / sqrtf(qq + 1e-6f), kn = 1.0f / sqrtf(kk + 1e-6f);
#pragma unroll
        for (int j = 0; j < J; j++) q[i][j] *= qn, k[i][j] *= kn;
        beta[i] = real ? 1.0f / (1.0f + expf(-to_float(b_in[i]))) : 0.0f;
    }
    float kk[6] = {}, qk[10] = {};
#pragma unroll
    for (int j = 0; j < J; j++) {
        const int c = lane + 32 * j;
        float G = 1.0f, carried[DB_TOKENS];  // carried[s]: G_is k_s
#pragma unroll
        for (int i = 0; i < DB_TOKENS; i++) {
            G *= g[i][j];
            rec[i * DP + c] = G * k[i][j];
            rec[(4 + i) * DP + c] = G * q[i][j];
#pragma unroll
            for (int s = 0; s < i; s++) {
                carried[s] *= g[i][j];
                kk[i * (i - 1) / 2 + s] = fmaf(k[i][j], carried[s], kk[i * (i - 1) / 2 + s]);
            }
            carried[i] = k[i][j];
#pragma unroll
            for (int s = 0; s <= i; s++) qk[i * (i + 1) / 2 + s] = fmaf(q[i][j], carried[s], qk[i * (i + 1) / 2 + s]);
        }
#pragma unroll
        for (int s = 0; s < DB_TOKENS; s++) rec[(8 + s) * DP + c] = carried[s];
        rec[12 * DP + c] = G;
    }
    float mine = 0.0f;  // lane n keeps number n
#pragma unroll
    for (int i = 1; i < DB_TOKENS; i++)
#pragma unroll
        for (int s = 0; s < i; s++) {
            const float v = beta[i] * warp_sum(kk[i * (i - 1) / 2 + s]);
            if (lane == i * (i - 1) / 2 + s) mine = v;
        }
#pragma unroll
    for (int n = 0; n < 10; n++) {
        const float v = warp_sum(qk[n]);
        if (lane == 6 + n) mine = v;
    }
#pragma unroll
    for (int i = 0; i < DB_TOKENS; i++)
        if (lane == 16 + i) mine = beta[i];
    if (lane < DB_NUMBERS) rec[13 * DP + lane] = mine;
}

__device__ __forceinline__ void scan_copy_16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// Four of a state column's channels from `ch` on; beyond the key size, or where the column is none, zeros.
__device__ __forceinline__ float4 delta_load_state(const float *column, int ch, int K, bool real, int vec) {
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (!real) return v;
    const float *src = column + ch;
    if (vec) {
        if (ch < K) v = *(const float4 *)src;
    } else {
        if (ch < K) v.x = src[0];
        if (ch + 1 < K) v.y = src[1];
        if (ch + 2 < K) v.z = src[2];
        if (ch + 3 < K) v.w = src[3];
    }
    return v;
}
__device__ __forceinline__ void delta_store_state(float *column, int ch, int K, float4 v, int vec) {
    float *dst = column + ch;
    if (vec) {
        if (ch < K) *(float4 *)dst = v;
    } else {
        if (ch < K) dst[0] = v.x;
        if (ch + 1 < K) dst[1] = v.y;
        if (ch + 2 < K) dst[2] = v.z;
        if (ch + 3 < K) dst[3] = v.w;
    }
}

// P lanes share a value column, each with 4 J of its key channels (lane p: 4 p .. 4 p + 3 of every 4 P, so that together
// they read a vector as whole lines); a lane has C columns, 4 J C numbers of state in registers, and every piece of a
// vector it reads serves them all: a 16-byte read costs the warp four cycles of shared memory whatever the lanes share, so
// C, not the columns of a warp (32 C / P), decides what shared memory costs a column. A block: its eight vectors against
// the columns; the 8 C partial sums of a lane meet by shuffles that hand half of them over at each of the first steps, so
// that at the end a lane has one column's four sums with the keys or with the queries; the lanes with the first solve for
// e, all get it, the lanes with the others write o. The CTA's last warp does nothing but bring the records in, so that the
// others' instructions are the recurrence's alone.
// Bound by the chain where sequences are few: one prompt of 1,999 tokens, 16 heads of 128 x 128: 298 us, 1,110 cycles a
// block at one walking warp a scheduler (the walk token by token with two barriers a token, which stood here: 1,560 us);
// towards the multiply-adds where they are many: 8 prompts, 5,672 tokens, 32 heads, 701 us.
template <int P, int J, int C>
__global__ void __launch_bounds__(160) delta_block_scan_kernel(DeltaScan p) {
    extern __shared__ __align__(16) float smem[];  // [DB_STAGES][DB_STAGE] records, of the values this CTA's columns
    constexpr int DP = 4 * P * J, HEAD = 13 * DP + DB_NUMBERS;
    const int walkers = blockDim.x - 32, cols = walkers / P * C, vp = (p.value + 3) & ~3;  // this CTA's columns
    const int RS = HEAD + DB_TOKENS * cols;
    const int tid = threadIdx.x, lane = tid & 31, part = lane & (P - 1);
    const int h = blockIdx.x % p.heads, tile = blockIdx.x / p.heads % p.tiles, place = blockIdx.x / p.heads / p.tiles;
    const int col0 = tile * cols, first_col = col0 + tid / P * C;  // this lane's columns: first_col ..
    const int K = p.key, V = p.value;
    pdl_wait();
    const int seq = p.longest_first ? sequence_place(p.seq_start, p.n_seqs, place) : place;
    const int row0 = p.seq_start[seq], n = p.seq_start[seq + 1] - row0;
    if (n <= 0) return;
    const int n_blocks = (n + DB_TOKENS - 1) / DB_TOKENS;
    if (tid >= walkers) {  // the records: a stage ahead of the walkers, two in flight
        int first_block = 0;
        for (int q = lane; q < seq; q += 32) first_block += (max(p.seq_start[q + 1] - p.seq_start[q], 0) + DB_TOKENS - 1) / DB_TOKENS;
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) first_block += __shfl_xor_sync(0xffffffffu, first_block, m);
        const uint32_t base_s = (uint32_t)__cvta_generic_to_shared(smem);
        const int own = min(cols, vp - col0);  // columns whose values the record holds (a multiple of 4)
        auto fetch = [&](int first) {          // blocks first .. first + DB_STAGE - 1
            const int count = min(DB_STAGE, n_blocks - first), stage = first / DB_STAGE % DB_STAGES;
            for (int b = 0; b < count; b++) {
                const float *rec = p.records + ((long long)(first_block + first + b) * p.heads + h) * p.record;
                const uint32_t dst = base_s + (stage * DB_STAGE + b) * RS * 4;
                for (int e = lane; e < HEAD / 4; e += 32) scan_copy_16(dst + e * 16, rec + e * 4);
                for (int e = lane; e < own; e += 32) {  // own / 4 pieces of each of the four tokens
                    const int t = e / (own / 4), c = e - t * (own / 4);
                    scan_copy_16(dst + (HEAD + t * cols + c * 4) * 4, rec + HEAD + t * vp + col0 + c * 4);
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");  // (a group each time, empty beyond the last block)
        };
        fetch(0);
        fetch(DB_STAGE);
        for (int b0 = 0; b0 < n_blocks; b0 += DB_STAGE) {
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncthreads();  // this stage is here, and the one before it has been read by all: its place is filled again
            fetch(b0 + 2 * DB_STAGE);
        }
        return;
    }
    float *head_state = p.state + ((long long)p.seq_slot[seq] * p.heads + h) * V * K;
    f32x2 S[C][2 * J];
#pragma unroll
    for (int c = 0; c < C; c++)
#pragma unroll
        for (int j = 0; j < J; j++) {
            const float4 v = delta_load_state(head_state + (long long)(first_col + c) * K, 4 * (P * j + part), K, first_col + c < V, p.vec);
            S[c][2 * j] = pack2(v.x, v.y), S[c][2 * j + 1] = pack2(v.z, v.w);
        }
    // every lane's place after the shuffles: its column, and whether its sums are with the queries
    constexpr int COL_STEPS = C == 4 ? 2 : C == 2 ? 1 : 0;
    constexpr int SPLIT = P >> (COL_STEPS + 1);   // the lane bit that tells sums with queries from sums with keys
    static_assert(SPLIT >= 1, "a lane has a column to itself at the end");
    const int my_c = part / (2 * SPLIT);          // (the first steps' bits, highest first, count the columns)
    const bool reads = (part & SPLIT) != 0;
    const int my_col = first_col + my_c;
    const long long hv = (long long)p.heads * V;
    float *out = p.out + (long long)row0 * hv + (long long)h * V + my_col;

    for (int b0 = 0, stage = 0; b0 < n_blocks; b0 += DB_STAGE, stage = stage == DB_STAGES - 1 ? 0 : stage + 1) {
        __syncthreads();
        const int count = min(DB_STAGE, n_blocks - b0);
        for (int b = 0; b < count; b++, out += DB_TOKENS * hv) {
            const float *rec = smem + (stage * DB_STAGE + b) * RS;
            const float *vec = rec + 4 * part;
            float sums[C][8];
#pragma unroll
            for (int r = 0; r < 8; r++) {
                f32x2 a[C];
#pragma unroll
                for (int j = 0; j < J; j++) {
                    const ulonglong2 w = *(const ulonglong2 *)(vec + r * DP + 4 * P * j);
#pragma unroll
                    for (int c = 0; c < C; c++) {
                        a[c] = j == 0 ? mul2(w.x, S[c][0]) : fma2(w.x, S[c][2 * j], a[c]);
                        a[c] = fma2(w.y, S[c][2 * j + 1], a[c]);
                    }
                }
#pragma unroll
                for (int c = 0; c < C; c++) {
                    const float2 x = unpack2(a[c]);
                    sums[c][r] = x.x + x.y;
                }
            }
            // what does not wait for the sums: the state's decay, the block's numbers and values, and (few channels a lane)
            // the vectors of the update, read while the shuffles are under way
            constexpr bool AHEAD = J <= 2;
            ulonglong2 u[AHEAD ? 4 : 1][J];
            if constexpr (AHEAD) {
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < J; j++) u[i][j] = *(const ulonglong2 *)(vec + (8 + i) * DP + 4 * P * j);
            }
#pragma unroll
            for (int j = 0; j < J; j++) {
                const ulonglong2 w = *(const ulonglong2 *)(vec + 12 * DP + 4 * P * j);
#pragma unroll
                for (int c = 0; c < C; c++) S[c][2 * j] = mul2(w.x, S[c][2 * j]), S[c][2 * j + 1] = mul2(w.y, S[c][2 * j + 1]);
            }
            const float4 n0 = *(const float4 *)(rec + 13 * DP), n1 = *(const float4 *)(rec + 13 * DP + 4), n2 = *(const float4 *)(rec + 13 * DP + 8);
            const float4 n3 = *(const float4 *)(rec + 13 * DP + 12), bt = *(const float4 *)(rec + 13 * DP + 16);
            const float *vv = rec + HEAD + my_col - col0;
            const float v0 = vv[0], v1 = vv[cols], v2 = vv[2 * cols], v3 = vv[3 * cols];
            // hand over: columns first, then keys' sums against queries', then plain sums
#pragma unroll
            for (int step = 0; step < COL_STEPS; step++) {
                const int half = C >> (step + 1), bit = P >> (step + 1);
                const bool up = part & bit;
#pragma unroll
                for (int c = 0; c < half; c++)
#pragma unroll
                    for (int r = 0; r < 8; r++) {
                        const float give = up ? sums[c][r] : sums[c + half][r], keep = up ? sums[c + half][r] : sums[c][r];
                        sums[c][r] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
                    }
            }
            float mine[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float give = reads ? sums[0][i] : sums[0][4 + i], keep = reads ? sums[0][4 + i] : sums[0][i];
                mine[i] = keep + __shfl_xor_sync(0xffffffffu, give, SPLIT);
            }
#pragma unroll
            for (int m = SPLIT >> 1; m > 0; m >>= 1)
#pragma unroll
                for (int i = 0; i < 4; i++) mine[i] += __shfl_xor_sync(0xffffffffu, mine[i], m);
            float e[4];  // (meant where the sums are with the keys)
            e[0] = bt.x * (v0 - mine[0]);
            e[1] = fmaf(-n0.x, e[0], bt.y * (v1 - mine[1]));
            e[2] = fmaf(-n0.z, e[1], fmaf(-n0.y, e[0], bt.z * (v2 - mine[2])));
            e[3] = fmaf(-n1.y, e[2], fmaf(-n1.x, e[1], fmaf(-n0.w, e[0], bt.w * (v3 - mine[3]))));
            float all[C][4], mine_e[4];
#pragma unroll
            for (int c = 0; c < C; c++) {
                const int src = (lane & ~(P - 1)) | c * 2 * SPLIT;
#pragma unroll
                for (int i = 0; i < 4; i++) all[c][i] = __shfl_sync(0xffffffffu, e[i], src);
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                f32x2 ee[C];
#pragma unroll
                for (int c = 0; c < C; c++) ee[c] = pack2(all[c][i], all[c][i]);
#pragma unroll
                for (int j = 0; j < J; j++) {
                    const ulonglong2 w = AHEAD ? u[AHEAD ? i : 0][j] : *(const ulonglong2 *)(vec + (8 + i) * DP + 4 * P * j);
#pragma unroll
                    for (int c = 0; c < C; c++) S[c][2 * j] = fma2(w.x, ee[c], S[c][2 * j]), S[c][2 * j + 1] = fma2(w.y, ee[c], S[c][2 * j + 1]);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                float x = all[0][i];
#pragma unroll
                for (int c = 1; c < C; c++) x = my_c == c ? all[c][i] : x;
                mine_e[i] = x;
            }
            float o[4];
            o[0] = fmaf(n1.z, mine_e[0], mine[0]);
            o[1] = fmaf(n2.x, mine_e[1], fmaf(n1.w, mine_e[0], mine[1]));
            o[2] = fmaf(n2.w, mine_e[2], fmaf(n2.z, mine_e[1], fmaf(n2.y, mine_e[0], mine[2])));
            o[3] = fmaf(n3.w, mine_e[3], fmaf(n3.z, mine_e[2], fmaf(n3.y, mine_e[1], fmaf(n3.x, mine_e[0], mine[3]))));
            const int left = n - (b0 + b) * DB_TOKENS;
            if (reads && my_col < V) {  // SPLIT lanes have the same column: each writes its share of the four tokens
                if constexpr (SPLIT >= 4) {
                    const float lo = part & 1 ? o[1] : o[0], hi = part & 1 ? o[3] : o[2];
                    if ((part & (SPLIT - 1)) < 4 && (part & 3) < left) out[(part & 3) * hv] = part & 2 ? hi : lo;
                } else {
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        if ((i & (SPLIT - 1)) == (part & (SPLIT - 1)) && i < left) out[i * hv] = o[i];
                }
            }
        }
    }
#pragma unroll
    for (int c = 0; c < C; c++)
#pragma unroll
        for (int j = 0; j < J; j++) {
            if (first_col + c >= V) continue;
            const float2 x = unpack2(S[c][2 * j]), y = unpack2(S[c][2 * j + 1]);
            delta_store_state(head_state + (long long)(first_col + c) * K, 4 * (P * j + part), K, make_float4(x.x, x.y, y.x, y.y), p.vec);
        }
}

// A step of one token a sequence: the state comes and goes once, and that is all there is to do, so the preparation is in
// the same kernel. A CTA has one (sequence, head) and some of its columns; it makes the token's k, q, g, b in shared memory
// (its columns' CTAs each for themselves: a few hundred channels), then every warp takes 8 columns at a time, LPC lanes a
// column with 4 J channels each: with a = g k and r = g q as above, S^T a and S^T r, then S <- g S + k e. (A sequence that
// brings several tokens after all is walked token by token.) Bound by HBM: 64 sequences, 32 heads of 128 x 128, 268 MB of
// state in 61 us with its wait (the walk above's general form and its preparation: 103 us).
template <typename T, int LPC, int J>
__global__ void __launch_bounds__(256) delta_step_kernel(DeltaPrepare p, DeltaScan q) {
    constexpr int DP = LPC * 4 * J, SIDE = 32 / LPC, ROUNDS = 8 / SIDE;  // columns side by side, and one after another
    __shared__ __align__(16) float ks[DP], qs[DP], gs[DP];
    __shared__ float meet[2][8], numbers[2];
    const int seq = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, K = p.key, V = p.value;
    const int n_warps = blockDim.x >> 5;
    pdl_wait();
    const int row0 = q.seq_start[seq], n = q.seq_start[seq + 1] - row0;
    if (n <= 0) return;
    float *head_state = q.state + ((long long)q.seq_slot[seq] * p.heads + h) * V * K;
    const int kvh = h / (p.heads / p.kv_heads), part = lane % LPC, side = lane / LPC;
    const float rate = expf(p.a_log[h]);
    for (int t = 0; t < n; t++) {
        const long long row = row0 + t;
        const T *qr = (const T *)p.qkv + row * p.ld_qkv + (long long)kvh * K, *kr = qr + (long long)p.kv_heads * K;
        const T *vr = (const T *)p.qkv + row * p.ld_qkv + 2LL * p.kv_heads * K + (long long)h * V;
        const float beta = 1.0f / (1.0f + expf(-to_float(((const T *)p.beta_in)[row * p.ld_beta + h])));
        float qq = 0.0f, kk = 0.0f;
        for (int c = tid; c < DP; c += blockDim.x) {
            const float qv = c < K ? to_float(qr[c]) : 0.0f, kv = c < K ? to_float(kr[c]) : 0.0f;
            float g = 1.0f;
            if (p.per_head) g = expf(-rate * softplus_f(to_float(((const T *)p.decay_in)[row * p.ld_decay + h]) + p.dt_bias[h]));
            else if (c < K) g = expf(-rate * softplus_f(((const float *)p.decay_in)[row * p.ld_decay + (long long)h * K + c] + p.dt_bias[h * K + c]));
            qs[c] = qv, ks[c] = kv, gs[c] = g;
            qq = fmaf(qv, qv, qq), kk = fmaf(kv, kv, kk);
        }
        qq = warp_sum(qq), kk = warp_sum(kk);
        if (lane == 0) meet[0][warp] = qq, meet[1][warp] = kk;
        __syncthreads();
        if (tid == 0) {
            qq = kk = 0.0f;
            for (int w = 0; w < n_warps; w++) qq += meet[0][w], kk += meet[1][w];
            numbers[0] = p.q_scale / sqrtf(qq + 1e-6f), numbers[1] = 1.0f / sqrtf(kk + 1e-6f);
        }
        __syncthreads();
        const float qn = numbers[0], kn = numbers[1];
        float4 k4[J], g4[J], a4[J], r4[J];
        float kq = 0.0f;
#pragma unroll
        for (int j = 0; j < J; j++) {
            const int c = 4 * (part + LPC * j);
            const float4 kv = *(const float4 *)(ks + c), qv = *(const float4 *)(qs + c), g = *(const float4 *)(gs + c);
            k4[j] = make_float4(kv.x * kn, kv.y * kn, kv.z * kn, kv.w * kn), g4[j] = g;
            const float4 r = make_float4(qv.x * qn, qv.y * qn, qv.z * qn, qv.w * qn);
            kq = fmaf(k4[j].x, r.x, fmaf(k4[j].y, r.y, fmaf(k4[j].z, r.z, fmaf(k4[j].w, r.w, kq))));
            a4[j] = make_float4(g.x * k4[j].x, g.y * k4[j].y, g.z * k4[j].z, g.w * k4[j].w);
            r4[j] = make_float4(g.x * r.x, g.y * r.y, g.z * r.z, g.w * r.w);
        }
#pragma unroll
        for (int m = 1; m < LPC; m <<= 1) kq += __shfl_xor_sync(0xffffffffu, kq, m);
        for (int col0 = (blockIdx.z * n_warps + warp) * 8; col0 < V; col0 += gridDim.z * n_warps * 8) {
            float4 s[ROUNDS][J];
            float vv[ROUNDS], a[ROUNDS], r[ROUNDS];
#pragma unroll
            for (int u = 0; u < ROUNDS; u++) {
                const int col = col0 + u * SIDE + side;
#pragma unroll
                for (int j = 0; j < J; j++) s[u][j] = delta_load_state(head_state + (long long)col * K, 4 * (part + LPC * j), K, col < V, q.vec);
                vv[u] = col < V ? to_float(vr[col]) : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < ROUNDS; u++) {
                a[u] = r[u] = 0.0f;
#pragma unroll
                for (int j = 0; j < J; j++) {
                    a[u] = fmaf(a4[j].x, s[u][j].x, fmaf(a4[j].y, s[u][j].y, fmaf(a4[j].z, s[u][j].z, fmaf(a4[j].w, s[u][j].w, a[u]))));
                    r[u] = fmaf(r4[j].x, s[u][j].x, fmaf(r4[j].y, s[u][j].y, fmaf(r4[j].z, s[u][j].z, fmaf(r4[j].w, s[u][j].w, r[u]))));
                }
            }
#pragma unroll
            for (int m = 1; m < LPC; m <<= 1)
#pragma unroll
                for (int u = 0; u < ROUNDS; u++) a[u] += __shfl_xor_sync(0xffffffffu, a[u], m), r[u] += __shfl_xor_sync(0xffffffffu, r[u], m);
#pragma unroll
            for (int u = 0; u < ROUNDS; u++) {
                const int col = col0 + u * SIDE + side;
                if (col >= V) continue;
                const float e = beta * (vv[u] - a[u]);
                if (part == u % LPC) q.out[row * p.heads * V + (long long)h * V + col] = fmaf(kq, e, r[u]);
#pragma unroll
                for (int j = 0; j < J; j++)
                    delta_store_state(head_state + (long long)col * K, 4 * (part + LPC * j), K,
                                      make_float4(fmaf(k4[j].x, e, g4[j].x * s[u][j].x), fmaf(k4[j].y, e, g4[j].y * s[u][j].y),
                                                  fmaf(k4[j].z, e, g4[j].z * s[u][j].z), fmaf(k4[j].w, e, g4[j].w * s[u][j].w)), q.vec);
            }
        }
        __syncthreads();  // (a further token's k, q, g come into the same memory)
    }
}

#include "delta_chunk.cuh"

// Whether a step's prompts go in chunks of 16 tokens (delta_chunk.cuh) rather than in blocks of four: where the longest prompt's chain counts
// for more than what the GPU has to do meanwhile, that is by the value columns an SM has on average while the longest walks. In us, blocks
// against chunks, both kernels each, keys and values of 128 (limit 48 columns), columns in brackets: 16 heads, one prompt of 1,999 tokens (14) 325
// and 208; prompts of 167, 32, 32 and 1,998 (15) 562 and 253; three of 900 (42) 309 and 265; 8 heads, six of 800 (42) 280 and 235, seven
// of 700 (48) 253 and 255, eight of 101 (55) 46 and 55; 32 heads, two of 250 (55) 95 and 106; 16 heads, four of 700 (55) 255 and 266.
// Of 64 (limit 24): 32 heads, one of 1,999 (14) 263 and 238; 8 heads, seven of 700 (24) 120 and 109; 32 heads, 35, 699, 1,223, 135, 71, 111 and
// 28 (26) 273 and 297; 32 heads, three of 900 (42) 229 and 241, four of 700 (55) 191 and 216. And prompts of 48 tokens on: 16 heads of 128, one of 50
// 21 and 22, of 100 28 and 25. Over 225 steps of one to eight prompts of 16 to 2,048 tokens this takes 31.3 ms, the faster form each time 31.2;
// none of them is more than 3 % slower than blocks, which take 39.4.
static bool delta_in_chunks(int n_tokens, int longest, int heads, int per_head, int key, int value) {
    if (per_head || !delta_chunk_takes(key, value) || longest < 48) return false;
    return (long long)heads * value * n_tokens <= (long long)(key == 64 ? 24 : 48) * abk_sm_count() * longest;
}

static long long delta_chunk_scratch(int n_tokens, int n_seqs, int heads, int key, int value) {
    return ((long long)n_tokens / DK_TOKENS + n_seqs) * heads * delta_chunk_floats(key, value);
}

static long long delta_block_scratch(int n_tokens, int n_seqs, int heads, int key, int value) {
    return ((long long)n_tokens / DB_TOKENS + n_seqs) * heads * delta_block_floats(key, value);
}

// Floats of scratch memory the recurrence needs for n_tokens tokens of n_seqs sequences, the longest of `longest`: the records of the blocks or
// chunks (form as in abk_delta_scan), none where no sequence brings more than a token; chunks: the tokens' records of abk_delta_chunks.
extern "C" long long abk_delta_scan_scratch(int n_tokens, int n_seqs, int longest, int heads, int key, int value, int chunks, int form) {
    if (chunks) return (long long)n_tokens * heads * delta_record_floats(key, value);
    if (n_tokens <= n_seqs) return 0;
    const long long in_chunks = delta_chunk_scratch(n_tokens, n_seqs, heads, key, value), in_blocks = delta_block_scratch(n_tokens, n_seqs, heads, key, value);
    if (form == 16) return in_chunks;
    // (a state that is not 16-byte aligned goes in blocks whatever the sizes)
    return form != 4 && in_chunks > in_blocks && delta_in_chunks(n_tokens, longest, heads, 0, key, value) ? in_chunks : in_blocks;
}

static int delta_chunk_run(DeltaPrepare q, DeltaScan p, const int *seq_start, int dtype, int n_tokens, int n_seqs, cudaStream_t s) {
    q.record = p.record = (int)delta_chunk_floats(q.key, q.value), q.pairs = ((long long)n_tokens / DK_TOKENS + n_seqs) * q.heads;
    if (q.pairs > 0x7fffffffLL) ABK_REFUSE("delta rule: %lld (chunk, head) pairs are more than a grid takes", q.pairs);
#define CHUNK_PREPARE_AS(T, J) abk_launch(delta_chunk_prepare_kernel<T, J>, dim3((unsigned)q.pairs), dim3(256), 0, s, q, seq_start, n_seqs)
#define CHUNK_PREPARE(J)                                           \
    do {                                                           \
        if (dtype == ABK_BF16) CHUNK_PREPARE_AS(__nv_bfloat16, J); \
        else CHUNK_PREPARE_AS(float, J);                           \
    } while (0)
    if (q.key == 64) CHUNK_PREPARE(2);
    else CHUNK_PREPARE(4);
#undef CHUNK_PREPARE
#undef CHUNK_PREPARE_AS
    const int rc = ABK_LAUNCH_RESULT();
    if (rc) return rc;
    const int lanes = q.key / 4, cols = DK_WARPS * 128 / lanes, sms = abk_sm_count();
    p.tiles = (q.value + cols - 1) / cols, p.n_seqs = n_seqs;
    const long long ctas = (long long)n_seqs * q.heads * p.tiles, share = (ctas + sms - 1) / sms;
    if (ctas > 0x7fffffffLL) ABK_REFUSE("delta rule: %lld blocks are more than a grid takes", ctas);
    size_t smem = (size_t)(DK_STAGES * (49 * q.key + 32 * cols) + 16 * cols) * 4;
    // (as the walk in blocks: no SM takes more CTAs than its share, and the longest sequence starts first)
    const size_t least = share <= 4 ? (size_t)(228 * 1024 / (share + 1)) : 0;
    if (smem < least) smem = least;
    p.longest_first = n_seqs > 1 && n_seqs <= SEQUENCE_PLACE_MAX && share > 1;
#define CHUNK_WALK(P)                                                                                        \
    do {                                                                                                     \
        const cudaError_t e = abk_allow_shared_memory((const void *)delta_chunk_walk_kernel<P>, (int)smem);  \
        if (e != cudaSuccess) return (int)e;                                                                 \
        abk_launch(delta_chunk_walk_kernel<P>, dim3((unsigned)ctas), dim3(32 * DK_WARPS + 32), smem, s, p);  \
    } while (0)
    if (lanes == 16) CHUNK_WALK(16);
    else CHUNK_WALK(32);
#undef CHUNK_WALK
    return ABK_LAUNCH_RESULT();
}

// longest: tokens of the longest sequence. form: 0 by size; 4: prompts in blocks of four tokens; 16: in chunks of 16 (refused where they are not built).
extern "C" int abk_delta_scan(const void *qkv, long long ld_qkv, int dtype, const void *decay_in, long long ld_decay, int per_head, const void *beta_in,
                              long long ld_beta, const float *a_log, const float *dt_bias, float *state, float *out,
                              const int *token_seq, const int *seq_start, const int *seq_slot, int n_tokens, int n_seqs,
                              int heads, int kv_heads, int key, int value, float *records, long long records_floats,
                              int longest, int form, void *stream) {
    if (n_seqs <= 0 || n_tokens <= 0) return 0;
    if (key < 1 || key > 256) ABK_REFUSE("delta rule: key size %d, the kernel takes 1 to 256", key);
    if (kv_heads < 1 || heads % kv_heads) ABK_REFUSE("delta rule: %d heads do not divide into %d key heads", heads, kv_heads);
    if (heads > 65535 || value > 65535 * 16) ABK_REFUSE("delta rule: %d heads of %d values are more than a grid takes", heads, value);
    if (form == 16 && (per_head || !delta_chunk_takes(key, value) || ((uintptr_t)state & 15)))
        ABK_REFUSE("delta rule: no chunks of 16 tokens for keys of %d and values of %d%s", key, value, per_head ? " with one decay a head" : "");
    const long long need = abk_delta_scan_scratch(n_tokens, n_seqs, longest, heads, key, value, 0, form);
    if (need > records_floats || (need && ((uintptr_t)records & 15)))
        ABK_REFUSE("delta rule: the scratch memory holds %lld floats, the step needs %lld (16-byte aligned)", records_floats, need);
    cudaStream_t s = (cudaStream_t)stream;
    DeltaPrepare q;
    q.qkv = qkv, q.ld_qkv = ld_qkv, q.decay_in = decay_in, q.ld_decay = ld_decay, q.per_head = per_head, q.beta_in = beta_in, q.ld_beta = ld_beta, q.a_log = a_log;
    q.dt_bias = dt_bias, q.records = records, q.token_seq = token_seq, q.pairs = ((long long)n_tokens / DB_TOKENS + n_seqs) * heads;
    q.heads = heads, q.kv_heads = kv_heads, q.key = key, q.value = value, q.parts = 0, q.record = (int)delta_block_floats(key, value);
    q.q_scale = 1.0f / sqrtf((float)key);
    DeltaScan p;
    p.records = records, p.state = state, p.out = out, p.seq_start = seq_start, p.seq_slot = seq_slot;
    p.heads = heads, p.key = key, p.value = value, p.parts = 0, p.record = q.record;
    p.vec = key % 4 == 0 && !((uintptr_t)state & 15);
    if (n_tokens <= n_seqs) {  // a token a sequence (or fewer)
        // (a CTA a head where that fills the GPU, else one for every 64 of its columns)
        const int slices = (long long)n_seqs * heads >= 2LL * abk_sm_count() ? 1 : (value + 63) / 64;
        const dim3 grid(n_seqs, heads, slices < 1 ? 1 : slices > 65535 ? 65535 : slices);
        // (as many warps as have columns: 256 sequences, 40 heads of 32 x 32 in 30 us, with eight 53)
        const int warps = value > 56 ? 8 : value < 1 ? 1 : (value + 7) / 8;
#define STEP_LAUNCH(LPC, J)                                                                                          \
    do {                                                                                                             \
        if (dtype == ABK_BF16) abk_launch(delta_step_kernel<__nv_bfloat16, LPC, J>, grid, dim3(32 * warps), 0, s, q, p); \
        else abk_launch(delta_step_kernel<float, LPC, J>, grid, dim3(32 * warps), 0, s, q, p);                       \
    } while (0)
        if (key <= 32) STEP_LAUNCH(8, 1);
        else if (key <= 64) STEP_LAUNCH(16, 1);
        else if (key <= 128) STEP_LAUNCH(32, 1);
        else STEP_LAUNCH(32, 2);
#undef STEP_LAUNCH
        return ABK_LAUNCH_RESULT();
    }
    if (form == 16 || (form == 0 && delta_in_chunks(n_tokens, longest, heads, per_head, key, value) && !((uintptr_t)state & 15)))
        return delta_chunk_run(q, p, seq_start, dtype, n_tokens, n_seqs, s);
    const long long blocks = (q.pairs + 3) / 4;
    if (blocks > 0x7fffffffLL) ABK_REFUSE("delta rule: %lld (block, head) pairs are more than a grid takes", q.pairs);
    const int kp4 = delta_pad_key(key) / 32;
#define PREPARE_LAUNCH_AS(T, J)                                                                                                          \
    do {                                                                                                                                 \
        if (per_head) abk_launch(delta_block_prepare_kernel<T, J, true>, dim3((unsigned)blocks), dim3(128), 0, s, q, seq_start, n_seqs); \
        else abk_launch(delta_block_prepare_kernel<T, J, false>, dim3((unsigned)blocks), dim3(128), 0, s, q, seq_start, n_seqs);         \
    } while (0)
#define PREPARE_LAUNCH(J)                                           \
    do {                                                            \
        if (dtype == ABK_BF16) PREPARE_LAUNCH_AS(__nv_bfloat16, J); \
        else PREPARE_LAUNCH_AS(float, J);                           \
    } while (0)
    if (kp4 == 1) PREPARE_LAUNCH(1);
    else if (kp4 == 2) PREPARE_LAUNCH(2);
    else if (kp4 == 4) PREPARE_LAUNCH(4);
    else PREPARE_LAUNCH(8);
#undef PREPARE_LAUNCH
#undef PREPARE_LAUNCH_AS
    int rc = ABK_LAUNCH_RESULT();
    if (rc) return rc;
    // A warp's columns, 4 or 8: the fewer, the more warps share the work and the less each waits for in a block; the more,
    // the less a column costs. Heads of 128 x 128, one prompt: of 1,999 tokens and 16 heads 298 us against 366, of 1,500
    // tokens and 32 heads 331 against 286; 8 prompts, 5,672 tokens, 32 heads: 960 against 701. Four columns therefore up to
    // what gives every SM one CTA of them, and where keys are long and prompts short, whose state is most of the work (100 prompts
    // of 20 tokens, 4 heads of 256 x 512: 417 us against 482).
    const long long columns = (long long)n_seqs * heads * value, sms = abk_sm_count();
    const int per_warp = columns <= 16 * sms || (key > 128 && n_tokens <= 32LL * n_seqs) ? 4 : 8;
    int warps = 4;
    while (warps > 1 && warps * per_warp >= 2 * value) warps /= 2;  // (no CTA of which less than half is used)
    const int cols = warps * per_warp;
    size_t smem = (size_t)DB_STAGES * DB_STAGE * (13 * delta_pad_key(key) + DB_NUMBERS + DB_TOKENS * cols) * sizeof(float);
    // The walk's CTAs start while the preparation's last ones still hold parts of the SMs, and gather where there is room
    // (one prompt: 601 us against 383): each asks for so much shared memory that no SM takes more than its share.
    p.tiles = (value + cols - 1) / cols, p.n_seqs = n_seqs;
    const long long ctas = (long long)n_seqs * heads * p.tiles, share = (ctas + sms - 1) / sms;
    const size_t least = share <= 4 ? (size_t)(228 * 1024 / (share + 1)) : 0;
    if (smem < least) smem = least;
    if (ctas > 0x7fffffffLL) ABK_REFUSE("delta rule: %lld blocks are more than a grid takes", ctas);
    // (a long walk that starts last would be walked alone: the 8 prompts above 701 us against 1,001 in the step's order)
    p.longest_first = n_seqs > 1 && n_seqs <= SEQUENCE_PLACE_MAX && share > 1;
#define SCAN_LAUNCH(P, J, C)                                                                               \
    do {                                                                                                   \
        cudaError_t e = abk_allow_shared_memory((const void *)delta_block_scan_kernel<P, J, C>, (int)smem); \
        if (e != cudaSuccess) return (int)e;                                                               \
        abk_launch(delta_block_scan_kernel<P, J, C>, dim3((unsigned)ctas), dim3(warps * 32 + 32), smem, s, p); \
    } while (0)
    const int kind = (kp4 == 1 ? 0 : kp4 == 2 ? 2 : kp4 == 4 ? 4 : 6) + (per_warp == 8);
    switch (kind) {
    case 0: SCAN_LAUNCH(8, 1, 1); break;
    case 1: SCAN_LAUNCH(8, 1, 2); break;
    case 2: SCAN_LAUNCH(16, 1, 2); break;
    case 3: SCAN_LAUNCH(16, 1, 4); break;
    case 4: SCAN_LAUNCH(16, 2, 2); break;
    case 5: SCAN_LAUNCH(16, 2, 4); break;
    case 6: SCAN_LAUNCH(16, 4, 2); break;
    default: SCAN_LAUNCH(16, 4, 4); break;
    }
#undef SCAN_LAUNCH
    return ABK_LAUNCH_RESULT();
}

// ------------------------------------------------------------------ one decay a head, prompts: in chunks
// With one decay g_t for all of a head's key channels the recurrence of a chunk of DC_TOKENS tokens that starts from S0
// unrolls, G_t the product of the chunk's decays up to t and r(t, s) = G_t / G_s:
//     u_t = b_t (v_t - G_t S0^T k_t - sum over s < t of r(t, s) (k_s . k_t) u_s)
//     o_t = G_t S0^T q_t + sum over s <= t of r(t, s) (k_s . q_t) u_s        S_end = G_end S0 + sum_s r(end, s) k_s u_s^T
// The first line is a triangular system (I + M) U = diag(b) (V - diag(G) K S0), M(t, s) = b_t r(t, s) (k_t . k_s) for
// s < t, whose matrix knows neither the state nor the values. delta_chunk_tables makes T = (I + M)^-1 diag(b) and
// Q(t, s) = r(t, s) (q_t . k_s) for every chunk and head side by side; delta_chunk_scan walks a sequence's chunks for one
// head and DC_VT value columns (the columns of a state do not meet) with four products a chunk:
//     [K; Q] S0,   U = T (V - diag(G) K S0),   O = diag(G) Q S0 + Q U,   S_end = G_end S0 + K^T diag(r(end, .)) U.
// Float32 throughout; the same numbers as token by token, summed in another order. A decay below e^-80 counts as e^-80.
#define DC_TOKENS 64
#define DC_VT 16
#define DC_P (DC_TOKENS + 1)

struct DeltaChunks {
    DeltaScan s;
    float *work;   // per (chunk, head): one table [64][64] (Q on and below the diagonal, T below its diagonal transposed
    int n_seqs, max_chunks;   // above it), the logarithms of G [64], T's diagonal [64] (the write strengths)
};
#define DC_WORK (DC_TOKENS * DC_TOKENS + 2 * DC_TOKENS)

__device__ __forceinline__ bool dc_locate(const DeltaChunks &p, int chunk, int &t0, int &nt) {
    for (int q = 0; q < p.n_seqs; q++) {
        const int first = p.s.seq_start[q], n = p.s.seq_start[q + 1] - first;
        const int chunks = (n + DC_TOKENS - 1) / DC_TOKENS;
        if (chunk < chunks) {
            t0 = first + chunk * DC_TOKENS, nt = min(DC_TOKENS, n - chunk * DC_TOKENS);
            return true;
        }
        chunk -= chunks;
    }
    return false;
}

// 16 bytes from global to shared memory, or 16 bytes of zeros.
__device__ __forceinline__ void dc_copy_16(float *dst, const float *src, bool real) {
    const int bytes = real ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}

__global__ void __launch_bounds__(256) delta_chunk_tables_kernel(DeltaChunks p) {
    extern __shared__ __align__(16) float dc_smem[];
    const int h = blockIdx.y, parts = p.s.parts, region = parts * SCAN_RUN, RP = 2 * region + 4, vp = p.s.record - 3 * region - 4;
    float *kq = dc_smem;                      // [64][RP]: k's runs, then q's, as in the records (see delta_chunk_scan)
    float *m = kq + DC_TOKENS * RP;           // [64][65]: M, strictly below the diagonal
    float *x = m + DC_TOKENS * DC_P;          // [64][65]: T
    float *lg = x + DC_TOKENS * DC_P, *beta = lg + DC_TOKENS;
    pdl_wait();
    int t0, nt;
    if (!dc_locate(p, blockIdx.x, t0, nt)) return;
    const int row_pieces = 2 * region / 4;
    for (int e = threadIdx.x; e < DC_TOKENS * row_pieces; e += 256) {
        const int t = e / row_pieces, c = e - t * row_pieces;
        const float *rec = p.s.records + ((long long)(t0 + min(t, nt - 1)) * p.s.heads + h) * p.s.record;
        dc_copy_16(kq + t * RP + 4 * c, rec + 4 * c, t < nt);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (threadIdx.x < DC_TOKENS) {
        const float *rec = p.s.records + ((long long)(t0 + min((int)threadIdx.x, nt - 1)) * p.s.heads + h) * p.s.record;
        lg[threadIdx.x] = threadIdx.x < nt ? fmaxf(logf(rec[2 * region]), -80.0f) : 0.0f;
        beta[threadIdx.x] = threadIdx.x < nt ? rec[3 * region + vp] : 0.0f;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0) {
        float sum = 0.0f;
        for (int t = 0; t < DC_TOKENS; t++) sum += lg[t], lg[t] = sum;   // (beyond nt: the last real one's)
    }
    __syncthreads();
    float *work = p.work + ((long long)blockIdx.x * p.s.heads + h) * DC_WORK;
    // a thread: one row t and every fourth column s
    const int t = threadIdx.x >> 2, sg = threadIdx.x & 3;
    for (int j = 0; j < DC_TOKENS / 4; j++) {
        const int c = sg + 4 * j;
        float kk = 0.0f, qk = 0.0f;
        if (c <= t && t < nt) {
            const float *kt = kq + t * RP, *kc = kq + c * RP;
            for (int r = 0; r < parts; r++) {
#pragma unroll
                for (int i = r * SCAN_RUN; i < r * SCAN_RUN + SCAN_ROWS; i += 4) {
                    const float4 a = *(const float4 *)(kc + i), b = *(const float4 *)(kt + i), q = *(const float4 *)(kt + region + i);
                    kk = fmaf(b.w, a.w, fmaf(b.z, a.z, fmaf(b.y, a.y, fmaf(b.x, a.x, kk))));
                    qk = fmaf(q.w, a.w, fmaf(q.z, a.z, fmaf(q.y, a.y, fmaf(q.x, a.x, qk))));
                }
            }
        }
        const float r = c <= t && t < nt ? expf(lg[t] - lg[c]) : 0.0f;
        m[t * DC_P + c] = c < t ? beta[t] * r * kk : 0.0f;
        if (c <= t) work[t * DC_TOKENS + c] = r * qk;
    }
    __syncthreads();
    // (I + M) X = diag(b): a thread a column, down its rows
    if (threadIdx.x < DC_TOKENS) {
        const int j = threadIdx.x;
        for (int r = 0; r < DC_TOKENS; r++) {
            float v = r == j ? beta[j] : 0.0f;
            if (r > j) {
                float acc = 0.0f;
                for (int c = j; c < r; c++) acc = fmaf(m[r * DC_P + c], x[c * DC_P + j], acc);
                v = -acc;
            }
            x[r * DC_P + j] = r >= j ? v : 0.0f;
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < DC_TOKENS * DC_TOKENS; e += 256) {  // T below its diagonal, transposed, above the table's
        const int r = e / DC_TOKENS, c = e % DC_TOKENS;
        if (c > r) work[e] = x[c * DC_P + r];
    }
    if (threadIdx.x < DC_TOKENS) {
        work[DC_TOKENS * DC_TOKENS + threadIdx.x] = lg[threadIdx.x];
        work[DC_TOKENS * DC_TOKENS + DC_TOKENS + threadIdx.x] = beta[threadIdx.x];
    }
}

// The rows of k and q lie in shared memory as in their records: runs of 32 channels with 4 floats of padding (zeros
// beyond the key size), k's runs and then q's, a row every 2 * region + 4 floats; so a chunk comes in as 16-byte copies
// that are all in flight together. Channel c of run r is at r * SCAN_RUN + c; the state's columns lie the same way,
// [run][32][DC_VT], rows beyond the key size zero.
#define DC_TP (DC_TOKENS + 4)   // a row of T or Q in shared memory
__global__ void __launch_bounds__(256) delta_chunk_scan_kernel(DeltaChunks p) {
    extern __shared__ __align__(16) float dc_smem[];
    const int K = p.s.key, V = p.s.value, h = blockIdx.y, seq = blockIdx.x, v0 = blockIdx.z * DC_VT;
    const int parts = p.s.parts, region = parts * SCAN_RUN, RP = 2 * region + 4, vp = p.s.record - 3 * region - 4;
    float *st = dc_smem;                          // [parts * 32][DC_VT]: the state's columns
    float *rs = st + parts * SCAN_ROWS * DC_VT;   // [64][DC_VT]: V, then V - diag(G) K S0
    float *us = rs + DC_TOKENS * DC_VT;           // [64][DC_VT]: U
    float *os = us + DC_TOKENS * DC_VT;           // [64][DC_VT]: diag(G) Q S0
    float *tq = os + DC_TOKENS * DC_VT;           // [64][DC_TP]: Q on and below the diagonal, T transposed above it
    float *lg = tq + DC_TOKENS * DC_TP;           // [64], then T's diagonal [64]
    float *td = lg + DC_TOKENS;
    float *kq = td + DC_TOKENS;                   // [64][RP]: k's runs, then q's
    pdl_wait();
    const int first = p.s.seq_start[seq], n = p.s.seq_start[seq + 1] - first;
    if (n <= 0) return;  // the sequence brings no token: its state stays as it is
    int chunk = 0;
    for (int q = 0; q < seq; q++) chunk += (p.s.seq_start[q + 1] - p.s.seq_start[q] + DC_TOKENS - 1) / DC_TOKENS;
    float *state = p.s.state + ((long long)p.s.seq_slot[seq] * p.s.heads + h) * V * K;
    for (int e = threadIdx.x; e < parts * SCAN_ROWS * DC_VT; e += 256) {
        const int c = e / (parts * SCAN_ROWS), i = e - c * (parts * SCAN_ROWS);
        st[i * DC_VT + c] = v0 + c < V && i < K ? state[(long long)(v0 + c) * K + i] : 0.0f;
    }
    const int row_pieces = 2 * region / 4;
    for (int t0 = first; t0 < first + n; t0 += DC_TOKENS, chunk++) {
        const int nt = min(DC_TOKENS, first + n - t0);
        const float *work = p.work + ((long long)chunk * p.s.heads + h) * DC_WORK;
        __syncthreads();  // the chunk before has been read
        for (int e = threadIdx.x; e < DC_TOKENS * row_pieces; e += 256) {
            const int t = e / row_pieces, c = e - t * row_pieces;
            const float *rec = p.s.records + ((long long)(t0 + min(t, nt - 1)) * p.s.heads + h) * p.s.record;
            dc_copy_16(kq + t * RP + 4 * c, rec + 4 * c, t < nt);
        }
        for (int e = threadIdx.x; e < DC_TOKENS * (DC_TOKENS / 4); e += 256) {
            const int r = e / (DC_TOKENS / 4), c = e - r * (DC_TOKENS / 4);
            dc_copy_16(tq + r * DC_TP + 4 * c, work + r * DC_TOKENS + 4 * c, true);
        }
        if (threadIdx.x < 2 * DC_TOKENS / 4) dc_copy_16(lg + 4 * threadIdx.x, work + DC_TOKENS * DC_TOKENS + 4 * threadIdx.x, true);
        {   // the values' columns: a row is DC_VT / 4 pieces, zeros beyond the record's values and the chunk's tokens
            const int t = threadIdx.x >> 2, c = (threadIdx.x & 3) * 4;
            const float *rec = p.s.records + ((long long)(t0 + min(t, nt - 1)) * p.s.heads + h) * p.s.record;
            dc_copy_16(rs + t * DC_VT + c, rec + 3 * region + min(v0 + c, vp - 4), t < nt && v0 + c < vp);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        {   // [K; Q] S0: a thread one of the 128 rows and 8 columns
            const int row = threadIdx.x >> 1, cg = (threadIdx.x & 1) * 8, t = row & (DC_TOKENS - 1);
            const float *a = kq + t * RP + (row < DC_TOKENS ? 0 : region);
            float acc[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
            for (int r = 0; r < parts; r++) {
                const float *ar = a + r * SCAN_RUN, *sr = st + r * SCAN_ROWS * DC_VT + cg;
#pragma unroll 8
                for (int i = 0; i < SCAN_ROWS; i++) {
                    const float w = ar[i];
                    const float4 s0 = *(const float4 *)(sr + i * DC_VT), s1 = *(const float4 *)(sr + i * DC_VT + 4);
                    acc[0] = fmaf(w, s0.x, acc[0]), acc[1] = fmaf(w, s0.y, acc[1]), acc[2] = fmaf(w, s0.z, acc[2]), acc[3] = fmaf(w, s0.w, acc[3]);
                    acc[4] = fmaf(w, s1.x, acc[4]), acc[5] = fmaf(w, s1.y, acc[5]), acc[6] = fmaf(w, s1.z, acc[6]), acc[7] = fmaf(w, s1.w, acc[7]);
                }
            }
            const float G = expf(lg[t]);
#pragma unroll
            for (int u = 0; u < 8; u++) {
                if (row < DC_TOKENS) rs[t * DC_VT + cg + u] -= G * acc[u];
                else os[t * DC_VT + cg + u] = G * acc[u];
            }
        }
        __syncthreads();
        const int t = threadIdx.x >> 2, c4 = (threadIdx.x & 3) * 4;   // a thread: one token and 4 columns
        {   // U = T R
            float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            for (int c = 0; c <= t; c++) {
                const float w = c < t ? tq[c * DC_TP + t] : td[t];
                const float4 r = *(const float4 *)(rs + c * DC_VT + c4);
                acc[0] = fmaf(w, r.x, acc[0]), acc[1] = fmaf(w, r.y, acc[1]), acc[2] = fmaf(w, r.z, acc[2]), acc[3] = fmaf(w, r.w, acc[3]);
            }
            *(float4 *)(us + t * DC_VT + c4) = make_float4(acc[0], acc[1], acc[2], acc[3]);
        }
        __syncthreads();
        {   // O = diag(G) Q S0 + Q U
            float4 o = *(const float4 *)(os + t * DC_VT + c4);
            for (int c = 0; c <= t; c++) {
                const float w = tq[t * DC_TP + c];
                const float4 u = *(const float4 *)(us + c * DC_VT + c4);
                o.x = fmaf(w, u.x, o.x), o.y = fmaf(w, u.y, o.y), o.z = fmaf(w, u.z, o.z), o.w = fmaf(w, u.w, o.w);
            }
            if (t < nt) {
                float *out = p.s.out + (long long)(t0 + t) * p.s.heads * V + (long long)h * V + v0 + c4;
                if (v0 + c4 < V) out[0] = o.x;
                if (v0 + c4 + 1 < V) out[1] = o.y;
                if (v0 + c4 + 2 < V) out[2] = o.z;
                if (v0 + c4 + 3 < V) out[3] = o.w;
            }
        }
        // S_end = G_end S0 + K^T diag(r(end, .)) U: a thread a key channel and 8 columns (its own elements of the state)
        const float lg_end = lg[nt - 1], G_end = expf(lg_end);
        for (int i = threadIdx.x >> 1; i < parts * SCAN_ROWS; i += 128) {
            const int cg = (threadIdx.x & 1) * 8, at = (i / SCAN_ROWS) * SCAN_RUN + i % SCAN_ROWS;
            float acc[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
            for (int c = 0; c < nt; c++) {
                const float w = kq[c * RP + at] * expf(lg_end - lg[c]);
                const float4 u0 = *(const float4 *)(us + c * DC_VT + cg), u1 = *(const float4 *)(us + c * DC_VT + cg + 4);
                acc[0] = fmaf(w, u0.x, acc[0]), acc[1] = fmaf(w, u0.y, acc[1]), acc[2] = fmaf(w, u0.z, acc[2]), acc[3] = fmaf(w, u0.w, acc[3]);
                acc[4] = fmaf(w, u1.x, acc[4]), acc[5] = fmaf(w, u1.y, acc[5]), acc[6] = fmaf(w, u1.z, acc[6]), acc[7] = fmaf(w, u1.w, acc[7]);
            }
#pragma unroll
            for (int u = 0; u < 8; u++) st[i * DC_VT + cg + u] = fmaf(G_end, st[i * DC_VT + cg + u], acc[u]);
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < K * DC_VT; e += 256) {
        const int c = e / K, i = e - c * K;
        if (v0 + c < V) state[(long long)(v0 + c) * K + i] = st[i * DC_VT + c];
    }
}

// The delta rule with one decay a head over a step that brings prompts, in chunks of 64 tokens: the preparation of
// abk_delta_scan, then the chunks' tables side by side, then the sequences' chunks in order. work: float32 scratch of at
// least max_chunks * heads * (64 * 64 + 2 * 64), max_chunks >= ceil(tokens / 64) + sequences.
extern "C" int abk_delta_chunks(const void *qkv, long long ld_qkv, int dtype, const void *decay_in, long long ld_decay,
                                const void *beta_in, long long ld_beta, const float *a_log, const float *dt_bias, float *state,
                                float *out, const int *token_seq, const int *seq_start, const int *seq_slot, int n_tokens,
                                int n_seqs, int heads, int kv_heads, int key, int value, float *records,
                                long long records_floats, int max_chunks, float *work, long long work_floats, void *stream) {
    if (n_seqs <= 0 || n_tokens <= 0 || max_chunks <= 0) return 0;
    if (key < 1 || key > 256) ABK_REFUSE("delta rule: key size %d, the kernel takes 1 to 256", key);
    if (kv_heads < 1 || heads % kv_heads) ABK_REFUSE("delta rule: %d heads do not divide into %d key heads", heads, kv_heads);
    if (heads > 65535 || n_seqs > 65535 || value > 65535 * DC_VT) ABK_REFUSE("delta rule: %d heads of %d values, %d sequences are more than a grid takes", heads, value, n_seqs);
    const int parts = delta_parts(key), record = delta_record_floats(key, value);
    if ((long long)n_tokens * heads * record > records_floats || ((uintptr_t)records & 15))
        ABK_REFUSE("delta rule: the scratch memory holds %lld floats, the step needs %lld (16-byte aligned)", records_floats,
                   (long long)n_tokens * heads * record);
    if ((long long)max_chunks * heads * DC_WORK > work_floats || ((uintptr_t)work & 15))
        ABK_REFUSE("delta rule: the chunks' scratch memory holds %lld floats, the step needs %lld (16-byte aligned)", work_floats,
                   (long long)max_chunks * heads * DC_WORK);
    cudaStream_t s = (cudaStream_t)stream;
    DeltaPrepare q;
    q.qkv = qkv, q.ld_qkv = ld_qkv, q.decay_in = decay_in, q.ld_decay = ld_decay, q.per_head = 1, q.beta_in = beta_in, q.ld_beta = ld_beta, q.a_log = a_log;
    q.dt_bias = dt_bias, q.records = records, q.token_seq = token_seq, q.pairs = (long long)n_tokens * heads;
    q.heads = heads, q.kv_heads = kv_heads, q.key = key, q.value = value, q.parts = parts, q.record = record;
    q.q_scale = 1.0f / sqrtf((float)key);
    const long long blocks = (q.pairs + 3) / 4;
    if (blocks > 0x7fffffffLL) ABK_REFUSE("delta rule: %lld (token, head) pairs are more than a grid takes", q.pairs);
    if (dtype == ABK_BF16) abk_launch(delta_prepare_kernel<__nv_bfloat16>, dim3((unsigned)blocks), dim3(128), 0, s, q);
    else abk_launch(delta_prepare_kernel<float>, dim3((unsigned)blocks), dim3(128), 0, s, q);
    int rc = ABK_LAUNCH_RESULT();
    if (rc) return rc;
    DeltaChunks p;
    p.s.records = records, p.s.state = state, p.s.out = out, p.s.seq_start = seq_start, p.s.seq_slot = seq_slot;
    p.s.heads = heads, p.s.key = key, p.s.value = value, p.s.parts = parts, p.s.record = record, p.s.vec = 0;
    p.work = work, p.n_seqs = n_seqs, p.max_chunks = max_chunks;
    const size_t smem_t = (size_t)(DC_TOKENS * (2 * parts * SCAN_RUN + 4) + 2 * DC_TOKENS * DC_P + 2 * DC_TOKENS) * sizeof(float);
    const size_t smem_s = (size_t)(parts * SCAN_ROWS * DC_VT + 3 * DC_TOKENS * DC_VT + DC_TOKENS * DC_TP + 2 * DC_TOKENS +
                                   DC_TOKENS * (2 * parts * SCAN_RUN + 4)) * sizeof(float);
    // Two CTAs of the walk fit an SM (heads of 128 channels: 111 KB each), which a step of many sequences needs; a step
    // whose CTAs are fewer than the SMs asks for more than half an SM's shared memory instead, so that each CTA has an SM
    // to itself (measured, one prompt of 2,048 tokens, 64 CTAs: 3.03 ms a step of four layers against 3.37 when the
    // scheduler may pair them)
    size_t smem_walk = smem_s;
    if ((long long)n_seqs * heads * ((value + DC_VT - 1) / DC_VT) <= abk_sm_count() && smem_walk < 116 * 1024) smem_walk = 116 * 1024;
    cudaError_t e = abk_allow_shared_memory((const void *)delta_chunk_tables_kernel, (int)smem_t);
    if (e == cudaSuccess) e = abk_allow_shared_memory((const void *)delta_chunk_scan_kernel, (int)smem_walk);
    if (e != cudaSuccess) return (int)e;
    abk_launch(delta_chunk_tables_kernel, dim3(max_chunks, heads), dim3(256), smem_t, s, p);
    abk_launch(delta_chunk_scan_kernel, dim3(n_seqs, heads, (value + DC_VT - 1) / DC_VT), dim3(256), smem_walk, s, p);
    return ABK_LAUNCH_RESULT();
}

// ------------------------------------------------------------------ gated per-head norm
// out[t, h, :] = o[t, h, :] / sqrt(mean(o^2) + eps) * w * act(gate[t, h, :]); one warp per (token, head). A token's
// gates lie at gate + t * ld_gate, float32 or (TG) in the storage type. act: sigmoid, or (silu) z sigmoid(z). w: [value],
// shared by the heads, or (w_per_head) [heads * value].
template <typename T, typename TG>
__global__ void __launch_bounds__(128) gated_head_norm_kernel(const float *o, const TG *gate, long long ld_gate, int heads,
                                                              const float *w, T *out, long long n_heads_total, int value,
                                                              float eps, int silu, int w_per_head) {
    pdl_wait();
    const long long head = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (head >= n_heads_total) return;
    const float *src = o + head * value;
    const TG *gs = gate + (head / heads) * ld_gate + (head % heads) * value;
    if (w_per_head) w += (head % heads) * value;
    float ss = 0.0f;
    for (int j = lane; j < value; j += 32) ss = fmaf(src[j], src[j], ss);
    ss = warp_sum(ss);
    const float scale = 1.0f / sqrtf(ss / (float)value + eps);
    for (int j = lane; j < value; j += 32) {
        const float z = to_float(gs[j]), sg = sigmoid_f(z);
        out[head * value + j] = from_float<T>(src[j] * scale * w[j] * (silu ? z * sg : sg));
    }
}

// The same for heads of 32 to 512 values, a power of two, everything aligned for pieces of four: LANES lanes a head, PIECES pieces of four values
// each, so that a warp's loads are whole lines and all in flight together; a CTA has a token's heads blockIdx.y * 256 / LANES on.
// 3,571 tokens of 40 heads of 64, bfloat16 gates and results: 16.0 us; 64 tokens of 32 heads of 128: 1.7 (a warp a head, number
// by number, each head's place by a division of 64 bits: 46 and 3.5; with the exponential and the reciprocal of the special-function unit,
// which are up to 4e-6 off far from zero, 12.3 and 1.6).
template <typename T, typename TG, int LANES, int PIECES>
__global__ void __launch_bounds__(256) gated_head_norm_vec_kernel(const float *o, const TG *gate, long long ld_gate, int heads, const float *w, T *out,
                                                                  float eps, int silu, int w_per_head) {
    constexpr int V = 4 * LANES * PIECES;
    const int h = blockIdx.y * (256 / LANES) + threadIdx.x / LANES, part = threadIdx.x & (LANES - 1);
    pdl_wait();
    const bool real = h < heads;  // (lanes beyond the last head take it along, for the shuffles)
    const int head = real ? h : heads - 1;
    const long long t = blockIdx.x;
    const float *src = o + (t * heads + head) * V + 4 * part, *ws = w + (w_per_head ? head * V : 0) + 4 * part;
    const TG *gs = gate + t * ld_gate + head * V + 4 * part;
    float4 v[PIECES], z[PIECES];
#pragma unroll
    for (int i = 0; i < PIECES; i++) {
        v[i] = *(const float4 *)(src + 4 * LANES * i);
        if constexpr (sizeof(TG) == 4) {
            z[i] = *(const float4 *)(gs + 4 * LANES * i);
        } else {
            const uint2 raw = *(const uint2 *)(gs + 4 * LANES * i);
            z[i] = make_float4(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u), __uint_as_float(raw.y << 16), __uint_as_float(raw.y & 0xffff0000u));
        }
    }
    float ss = 0.0f;
#pragma unroll
    for (int i = 0; i < PIECES; i++) ss = fmaf(v[i].x, v[i].x, fmaf(v[i].y, v[i].y, fmaf(v[i].z, v[i].z, fmaf(v[i].w, v[i].w, ss))));
#pragma unroll
    for (int m = LANES / 2; m > 0; m >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, m);
    const float scale = 1.0f / sqrtf(ss / (float)V + eps);
    if (!real) return;
    T *dst = out + (t * heads + head) * V + 4 * part;
#pragma unroll
    for (int i = 0; i < PIECES; i++) {
        const float4 g = *(const float4 *)(ws + 4 * LANES * i);
        const float x[4] = {v[i].x * scale * g.x, v[i].y * scale * g.y, v[i].z * scale * g.z, v[i].w * scale * g.w}, zz[4] = {z[i].x, z[i].y, z[i].z, z[i].w};
        float r[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const float sg = sigmoid_f(zz[u]);
            r[u] = x[u] * (silu ? zz[u] * sg : sg);
        }
        if constexpr (sizeof(T) == 4) {
            *(float4 *)(dst + 4 * LANES * i) = make_float4(r[0], r[1], r[2], r[3]);
        } else {
            const __nv_bfloat162 a = __floats2bfloat162_rn(r[0], r[1]), b = __floats2bfloat162_rn(r[2], r[3]);
            *(uint2 *)(dst + 4 * LANES * i) = make_uint2(*(const uint32_t *)&a, *(const uint32_t *)&b);
        }
    }
}

extern "C" int abk_gated_head_norm(const float *o, const void *gate, long long ld_gate, int gate_stored, const float *w, void *out,
                                   int dtype, int n_tokens, int heads, int value, float eps, int silu, int w_per_head,
                                   void *stream) {
    const long long total = (long long)n_tokens * heads;
    if (total <= 0) return 0;
    const long long blocks = (total + 3) / 4;
    if (blocks > 0x7fffffffLL) ABK_REFUSE("gated norm: %lld heads are more than a grid takes", total);
    cudaStream_t s = (cudaStream_t)stream;
    typedef __nv_bfloat16 bf;
    const bool gate16 = dtype == ABK_BF16 && gate_stored;  // 16-bit gates; pieces of four are 8 bytes of them
    const bool aligned = !(((uintptr_t)o | (uintptr_t)w) & 15) && !((uintptr_t)out & (dtype == ABK_BF16 ? 7 : 15)) && !((uintptr_t)gate & (gate16 ? 7 : 15)) &&
                         ld_gate % 4 == 0;
    if (aligned && (value == 32 || value == 64 || value == 128 || value == 256 || value == 512) && heads <= 65535) {
        const int lanes = value / 4 < 32 ? value / 4 : 32, per = 256 / lanes;
        const dim3 grid(n_tokens, (heads + per - 1) / per);
#define NORM_AS(T, TG, LANES, PIECES)                                                                                                        \
    abk_launch(gated_head_norm_vec_kernel<T, TG, LANES, PIECES>, grid, dim3(256), 0, s, o, (const TG *)gate, ld_gate, heads, w, (T *)out, eps, \
               silu, w_per_head)
#define NORM_LAUNCH(T, TG)                         \
    switch (value) {                               \
    case 32: NORM_AS(T, TG, 8, 1); break;          \
    case 64: NORM_AS(T, TG, 16, 1); break;         \
    case 128: NORM_AS(T, TG, 32, 1); break;        \
    case 256: NORM_AS(T, TG, 32, 2); break;        \
    default: NORM_AS(T, TG, 32, 4);                \
    }
        if (gate16) { NORM_LAUNCH(bf, bf) }
        else if (dtype == ABK_BF16) { NORM_LAUNCH(bf, float) }
        else { NORM_LAUNCH(float, float) }
#undef NORM_LAUNCH
#undef NORM_AS
        return ABK_LAUNCH_RESULT();
    }
    if (dtype == ABK_BF16 && gate_stored)
        abk_launch(gated_head_norm_kernel<bf, bf>, dim3((unsigned)blocks), dim3(128), 0, s, o, (const bf *)gate, ld_gate, heads, w,
                   (bf *)out, total, value, eps, silu, w_per_head);
    else if (dtype == ABK_BF16)
        abk_launch(gated_head_norm_kernel<bf, float>, dim3((unsigned)blocks), dim3(128), 0, s, o, (const float *)gate, ld_gate, heads, w,
                   (bf *)out, total, value, eps, silu, w_per_head);
    else
        abk_launch(gated_head_norm_kernel<float, float>, dim3((unsigned)blocks), dim3(128), 0, s, o, (const float *)gate, ld_gate, heads, w,
                   (float *)out, total, value, eps, silu, w_per_head);
    return ABK_LAUNCH_RESULT();
}
