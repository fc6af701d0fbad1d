// The gated delta rule over prompts in chunks of 16 tokens, in float32 on the CUDA cores (included by delta_rule.cu).
//
// With S [key, value] the state before a chunk, a_i = G_i k_i, r_i = G_i q_i and G_ij as in the blocks of four, the chunk's corrections E (a
// row a token) solve a triangular system whose matrix knows neither the state nor the values:
//     (I + L) E = diag(b) (V - A S),   L_is = b_i [k_i . G_is k_s],   O = R S + M E,   M_is = [q_i . G_is k_s] (s <= i)
// so with U0 = (I + L)^-1 diag(b) V and W = (I + L)^-1 diag(b) A, made for all chunks side by side,
//     E = U0 - W S,     O = M U0 + (R - M W) S,     S <- G_16 S + K~^T E,   K~_s = G_16,s k_s.
// (Decays multiplied, never divided.) The walk is then two products with the state and one into it a chunk, and its chain one
// latency for 16 tokens: one prompt of 1,999 tokens, 16 heads of 128 x 128, in 143 us (2,200 cycles a chunk at one walking warp a
// scheduler, half of them issuing; the walk in blocks of four 290), after 68 us for the records (blocks 36). Float32 throughout. (The
// products in three bfloat16 parts on warp-level tensor cores, the state in registers as their operand, took 156 us: an SM gives one
// such product in nine cycles, 40 float32 multiply-adds a cycle, and its 288 products a chunk and 16 columns were all of the time.)
// Errors against 64 bits (2-norm, 16 heads of 128 x 128, 1,999 tokens, results and states), blocks of four and chunks: slow decays 19.0 20.4 and
// 19.1 20.5e-7, none 17.0 18.7 and 16.0 17.6e-7; decays of a few tokens 1.50 1.15 and 1.64 1.42e-7, of one 1.24 1.05 and 1.39 1.42e-7 (a
// token's key is decayed by up to fifteen rounded products, in blocks by three and the state by one a block).
#pragma once

#define DK_TOKENS 16
#define DK_WARPS 4    // walking warps of a CTA
#define DK_STAGES 4   // chunks that are in shared memory or on their way

static inline bool delta_chunk_takes(int key, int value) { return (key == 64 || key == 128) && value % 4 == 0; }
// A record, float32, of a chunk and a head: [-W; R - M W] [32][key], K~ [16][key], G_16 [key], [U0; M U0] [32][value].
static inline long long delta_chunk_floats(int key, int value) { return 49LL * key + 32LL * value; }

// The sum over 2 BIT lanes of v[0 .. N): at the end a lane has N / (2 BIT) of them, v[0 ..], from its place among the lanes times that on.
template <int N, int BIT> __device__ __forceinline__ void hand_over(float *v, int lane) {
    const bool up = lane & BIT;
#pragma unroll
    for (int i = 0; i < N / 2; i++) {
        const float give = up ? v[i] : v[i + N / 2], keep = up ? v[i + N / 2] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, give, BIT);
    }
    if constexpr (BIT > 1) hand_over<N / 2, BIT / 2>(v, lane);
}

// A CTA a (chunk, head): the tokens' vectors two a warp; the pairs' products two rows s a warp, carried from token to token; then a
// thread a column of A and one of V down the triangular system. Bound by its instructions, 21,000 a CTA, spills among them: three CTAs an SM leave
// a thread 80 registers, and the pairs' 64 sums, or the system's four runs of sixteen, do not fit (keys of 128: 528 bytes stored and 572
// loaded a thread, of 64: 172 and 168).
template <typename T, int J> __global__ void __launch_bounds__(256, 3) delta_chunk_prepare_kernel(DeltaPrepare p, const int *seq_start, int n_seqs) {
    constexpr int K = 32 * J;
    __shared__ __align__(16) float ks[DK_TOKENS * K], qs[DK_TOKENS * K], gs[DK_TOKENS * K], L[256], M[256], beta[DK_TOKENS];  // (L times b_i)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, V = p.value;
    const int b = (int)(blockIdx.x / p.heads), h = (int)(blockIdx.x - (unsigned)b * p.heads);
    pdl_wait();
    int row0, count;
    if (!delta_block_locate<DK_TOKENS>(seq_start, n_seqs, b, row0, count)) return;
    const int kvh = h / (p.heads / p.kv_heads);
    const float rate = expf(p.a_log[h]);
    {
        T q_in[2][J], k_in[2][J], b_in[2];
        float d_in[2][J], bias[J];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const long long row = row0 + min(2 * warp + u, count - 1);
            const T *qr = (const T *)p.qkv + row * p.ld_qkv + (long long)kvh * K, *kr = qr + (long long)p.kv_heads * K;
#pragma unroll
            for (int j = 0; j < J; j++) {
                const int c = lane + 32 * j;
                q_in[u][j] = qr[c], k_in[u][j] = kr[c], d_in[u][j] = ((const float *)p.decay_in)[row * p.ld_decay + (long long)h * K + c];
            }
            b_in[u] = ((const T *)p.beta_in)[row * p.ld_beta + h];
        }
#pragma unroll
        for (int j = 0; j < J; j++) bias[j] = p.dt_bias[h * K + lane + 32 * j];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int i = 2 * warp + u;
            const bool real = i < count;
            float q[J], k[J], qq = 0.0f, kk = 0.0f;
#pragma unroll
            for (int j = 0; j < J; j++) {
                q[j] = real ? to_float(q_in[u][j]) : 0.0f, k[j] = real ? to_float(k_in[u][j]) : 0.0f;
                qq = fmaf(q[j], q[j], qq), kk = fmaf(k[j], k[j], kk);
            }
            qq = warp_sum(qq), kk = warp_sum(kk);
            const float qn = p.q_scale / sqrtf(qq + 1e-6f), kn = 1.0f / sqrtf(kk + 1e-6f);
#pragma unroll
            for (int j = 0; j < J; j++) {
                const int at = i * K + lane + 32 * j;
                qs[at] = q[j] * qn, ks[at] = k[j] * kn;
                gs[at] = real ? expf(-rate * softplus_f(d_in[u][j] + bias[j])) : 1.0f;
            }
            if (lane == 0) beta[i] = real ? 1.0f / (1.0f + expf(-to_float(b_in[u]))) : 0.0f;
        }
    }
    __syncthreads();
    float *const rec = p.records + (long long)blockIdx.x * p.record;
    {   // rows s and 15 - s of the pairs (s, i >= s): k_s carried along, its products with k_i and q_i; 64 sums that lanes hand over by halves
        const int s[2] = {warp, DK_TOKENS - 1 - warp};
        float carried[2][J], sums[64];
#pragma unroll
        for (int v = 0; v < 64; v++) sums[v] = 0.0f;
#pragma unroll
        for (int j = 0; j < J; j++) carried[0][j] = carried[1][j] = 0.0f;
#pragma unroll
        for (int i = 0; i < DK_TOKENS; i++) {
            if (i < s[0]) continue;
            float k[J], q[J], g[J];
#pragma unroll
            for (int j = 0; j < J; j++) {
                const int at = i * K + lane + 32 * j;
                k[j] = ks[at], q[j] = qs[at], g[j] = gs[at];
            }
#pragma unroll
            for (int u = 0; u < 2; u++) {
                if (i < s[u]) continue;
#pragma unroll
                for (int j = 0; j < J; j++) {
                    carried[u][j] = i == s[u] ? k[j] : carried[u][j] * g[j];
                    sums[32 * u + i] = fmaf(k[j], carried[u][j], sums[32 * u + i]), sums[32 * u + 16 + i] = fmaf(q[j], carried[u][j], sums[32 * u + 16 + i]);
                }
            }
        }
        hand_over<64, 16>(sums, lane);
#pragma unroll
        for (int u = 0; u < 2; u++) {  // this lane's: sums 2 lane, 2 lane + 1
            const int i = (2 * lane + u) & 15, col = lane & 16 ? s[1] : s[0];
            if (lane & 8) M[i * 16 + col] = sums[u];
            else L[i * 16 + col] = i > col ? beta[i] * sums[u] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < 2; u++)
#pragma unroll
            for (int j = 0; j < J; j++) rec[(32 + s[u]) * K + lane + 32 * j] = carried[u][j];
    }
    __syncthreads();
    // down the system: a thread a column of A and one of V (each number of L and M read for both)
    for (int c = threadIdx.x; c < max(K, V); c += 256) {
        float w[DK_TOKENS], r[DK_TOKENS], y[DK_TOKENS], o[DK_TOKENS], G = 1.0f;
        const bool key = c < K, value = c < V;
#pragma unroll
        for (int i = 0; i < DK_TOKENS; i++) {
            w[i] = r[i] = 0.0f;
            if (key) {
                G *= gs[i * K + c];
                w[i] = -beta[i] * (G * ks[i * K + c]), r[i] = G * qs[i * K + c];
            }
        }
        {
            const T *vr = (const T *)p.qkv + row0 * p.ld_qkv + 2LL * p.kv_heads * K + (long long)h * V + (value ? c : 0);
            T v[DK_TOKENS];
#pragma unroll
            for (int i = 0; i < DK_TOKENS; i++) v[i] = vr[min(i, count - 1) * p.ld_qkv];
#pragma unroll
            for (int i = 0; i < DK_TOKENS; i++) y[i] = beta[i] * to_float(v[i]);  // (beyond the last token beta is 0)
        }
#pragma unroll
        for (int i = 0; i < DK_TOKENS; i++) {
            float sum = 0.0f;
#pragma unroll
            for (int s = 0; s <= i; s += 4) {
                const float4 l4 = *(const float4 *)(L + i * 16 + s), m4 = *(const float4 *)(M + i * 16 + s);
                const float l[4] = {l4.x, l4.y, l4.z, l4.w}, m[4] = {m4.x, m4.y, m4.z, m4.w};
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    if (s + t < i) {
                        w[i] = fmaf(-l[t], w[s + t], w[i]), y[i] = fmaf(-l[t], y[s + t], y[i]);
                        r[i] = fmaf(m[t], w[s + t], r[i]), sum = fmaf(m[t], y[s + t], sum);
                    } else if (s + t == i) {
                        r[i] = fmaf(m[t], w[i], r[i]), sum = fmaf(m[t], y[i], sum);
                    }
                }
            }
            o[i] = sum;
        }
        if (key) {
#pragma unroll
            for (int i = 0; i < DK_TOKENS; i++) rec[i * K + c] = w[i], rec[(16 + i) * K + c] = r[i];
            rec[48 * K + c] = G;
        }
        if (value) {
            float *to = rec + 49 * K + c;
#pragma unroll
            for (int i = 0; i < DK_TOKENS; i++) to[(long long)i * V] = y[i], to[(long long)(16 + i) * V] = o[i];
        }
    }
}

// P lanes (16 for keys of 64, 32 for 128) have four value columns of a state, four channels each: sixteen numbers in registers, so that 16
// bytes of a record's row serve 16 multiply-adds (a 16-byte read costs the SM four cycles for a warp, whatever its lanes share). A
// warp needs no other for its columns: the lanes' sums for E are handed over by halves, E goes through shared memory to all of its
// lanes, and O's sums follow behind the state. The CTA's last warp does nothing but bring the records in.
template <int P> __global__ void __launch_bounds__(32 * DK_WARPS + 32) delta_chunk_walk_kernel(DeltaScan p) {
    constexpr int K = 4 * P, COLS = DK_WARPS * 128 / P, AT_K = 32 * K, AT_G = 48 * K, AT_U = 49 * K, STAGE = AT_U + 32 * COLS, MINE = 64 / P;
    extern __shared__ __align__(16) float dk_smem[];  // [DK_STAGES][STAGE], then [groups of four columns][16 tokens][4]: E
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, part = lane & (P - 1), group = tid / P;
    const int h = blockIdx.x % p.heads, tile = blockIdx.x / p.heads % p.tiles, place = blockIdx.x / p.heads / p.tiles;
    const int V = p.value, col0 = tile * COLS, first_col = col0 + 4 * group;
    pdl_wait();
    const int seq = p.longest_first ? sequence_place(p.seq_start, p.n_seqs, place) : place;
    const int row0 = p.seq_start[seq], n = p.seq_start[seq + 1] - row0;
    if (n <= 0) return;
    const int n_chunks = (n + DK_TOKENS - 1) / DK_TOKENS;
    if (warp == DK_WARPS) {
        int first_chunk = 0;
        for (int q = lane; q < seq; q += 32) first_chunk += (max(p.seq_start[q + 1] - p.seq_start[q], 0) + DK_TOKENS - 1) / DK_TOKENS;
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) first_chunk += __shfl_xor_sync(0xffffffffu, first_chunk, m);
        const float *records = p.records + ((long long)first_chunk * p.heads + h) * p.record;
        const long long next_record = (long long)p.heads * p.record;
        const int own = min(COLS, V - col0) / 4;  // pieces of a row of [U0; M U0]
        auto fetch = [&](int c) {
            if (c < n_chunks) {
                const float *rec = records + c * next_record;
                const uint32_t dst = (uint32_t)__cvta_generic_to_shared(dk_smem + c % DK_STAGES * STAGE);
#pragma unroll 7
                for (int e = lane; e < 49 * K / 4; e += 32) scan_copy_16(dst + e * 16, rec + e * 4);
#pragma unroll
                for (int e = lane; e < 32 * COLS / 4; e += 32)
                    if (e % (COLS / 4) < own) scan_copy_16(dst + (AT_U + e * 4) * 4, rec + AT_U + e / (COLS / 4) * V + col0 + e % (COLS / 4) * 4);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");  // (a group each time, empty beyond the last chunk)
        };
#pragma unroll 1
        for (int c = 0; c < DK_STAGES - 1; c++) fetch(c);
#pragma unroll 1
        for (int c = 0; c < n_chunks; c++) {
            asm volatile("cp.async.wait_group %0;" ::"n"(DK_STAGES - 2) : "memory");
            __syncthreads();  // this chunk is here, and the one before it has been read by all: its place is filled again
            fetch(c + DK_STAGES - 1);
        }
        return;
    }
    const bool real = first_col < V;
    float *const state = p.state + ((long long)p.seq_slot[seq] * p.heads + h) * V * K + (long long)first_col * K + 4 * part;
    f32x2 S[4][2];  // [column][pair of channels]
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const float4 v = real ? *(const float4 *)(state + c * K) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        S[c][0] = pack2(v.x, v.y), S[c][1] = pack2(v.z, v.w);
    }
    float *const es = dk_smem + DK_STAGES * STAGE + group * 64;
    const long long hv = (long long)p.heads * V;
    // The sums over the P lanes: at each step a lane hands over the half of its rows that is not its own token's. Every lane takes the rows
    // in its own order, row i ^ my_token as its i-th, so that what it hands over is always its second half; at the end it has its
    // token's four columns (P = 16) or two of them.
    const int my_token = MINE * part / 4, my_c = MINE * part & 3;
    int row_at[DK_TOKENS];
#pragma unroll
    for (int i = 0; i < DK_TOKENS; i++) row_at[i] = (i ^ my_token) * K;
    auto meet = [&](float *v) {
#pragma unroll
        for (int i = 0; i < 32; i++) v[i] += __shfl_xor_sync(0xffffffffu, v[i + 32], P / 2);
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] += __shfl_xor_sync(0xffffffffu, v[i + 16], P / 4);
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] += __shfl_xor_sync(0xffffffffu, v[i + 8], P / 8);
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] += __shfl_xor_sync(0xffffffffu, v[i + 4], P / 16);
        if constexpr (P == 32) hand_over<4, 1>(v, lane);
    };
    float *out = p.out + ((long long)row0 + my_token) * hv + (long long)h * V + first_col + my_c;
    for (int c = 0; c < n_chunks; c++, out += DK_TOKENS * hv) {
        __syncthreads();
        const float *const stage = dk_smem + c % DK_STAGES * STAGE, *const x = stage + 4 * part, *const u0 = stage + AT_U + my_token * COLS + 4 * group + my_c;
        auto products = [&](int first, float *v) {  // 16 rows from `first` on with this lane's channels of its four columns
#pragma unroll
            for (int i = 0; i < DK_TOKENS; i++) {
                const ulonglong2 w = *(const ulonglong2 *)(x + first * K + row_at[i]);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float2 a = unpack2(fma2(w.y, S[j][1], mul2(w.x, S[j][0])));
                    v[4 * i + j] = a.x + a.y;
                }
            }
        };
        float e[64], o[64];
        products(0, e);
        products(16, o);  // (before the state moves on; its sums meet behind the state)
        meet(e);
#pragma unroll
        for (int i = 0; i < MINE; i++) es[MINE * part + i] = e[i] + u0[i];
        __syncwarp();
        const float4 G = *(const float4 *)(x + AT_G);
        float s[4][4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float2 a = unpack2(S[j][0]), b = unpack2(S[j][1]);
            s[j][0] = G.x * a.x, s[j][1] = G.y * a.y, s[j][2] = G.z * b.x, s[j][3] = G.w * b.y;
        }
#pragma unroll
        for (int i = 0; i < DK_TOKENS; i++) {
            const float4 k = *(const float4 *)(x + AT_K + i * K), ev = *(const float4 *)(es + 4 * i);
            const float et[4] = {ev.x, ev.y, ev.z, ev.w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                s[j][0] = fmaf(k.x, et[j], s[j][0]), s[j][1] = fmaf(k.y, et[j], s[j][1]);
                s[j][2] = fmaf(k.z, et[j], s[j][2]), s[j][3] = fmaf(k.w, et[j], s[j][3]);
            }
        }
#pragma unroll
        for (int j = 0; j < 4; j++) S[j][0] = pack2(s[j][0], s[j][1]), S[j][1] = pack2(s[j][2], s[j][3]);
        meet(o);
        if (real && c * DK_TOKENS + my_token < n) {
#pragma unroll
            for (int i = 0; i < MINE; i++) out[i] = o[i] + u0[16 * COLS + i];
        }
        __syncwarp();  // (E is written again)
    }
    if (real) {
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const float2 a = unpack2(S[c][0]), b = unpack2(S[c][1]);
            *(float4 *)(state + c * K) = make_float4(a.x, a.y, b.x, b.y);
        }
    }
}
