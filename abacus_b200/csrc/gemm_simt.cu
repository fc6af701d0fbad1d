// out[M, N] = x[M, K] . w[N, K]^T with float32 multiply-adds, for any M, N, K.
//
// This is the matrix product of the true 32-bit path (no TF32), and the fallback of the bfloat16 path for shapes the tensor-core
// kernel refuses. Large products go to the tensor cores, with smaller errors (gemm_split.cuh); here an output element is the sum of eight running
// sums: K in pieces of 16, piece c to sum c % 8, each sum over its k in ascending order, then in pairs,
// ((s0 + s1) + (s2 + s3)) + ((s4 + s5) + (s6 + s7)); up to K = 256 it is one sum over k in ascending order (a chain of that
// length needs no cutting, and the small products of small models keep the order they had). So a row's result does not
// depend on where its tile lies. Nor does it on how many other rows are in the batch as long as the product goes the same way: a row of a step that
// is large enough for the tensor cores differs from the same row alone by the two orders' rounding (some 2e-7), so a prompt in one step
// and token by token are not bit-equal where a product has 512 inputs and more and gemm_split_wins takes the step's rows.
// Formula: src/model.c:299, 302, 307, 309, 324 (weights are [out, in] row-major, no bias).
//
// A warp has one tile of outputs and one of their sums. It stages its own pieces, 16 bytes at a time by cp.async (rows of 20
// floats: eight rows' pieces lie in different banks), one to three ahead, and waits for no other warp on the way. With eight
// sums a CTA's eight warps have them all of one tile, and meet at the end: a product of a few hundred rows has too few outputs
// to fill 148 SMs with warps whose lanes hold enough of them. Shared memory gives a warp a number a lane and cycle, and an
// SM's four schedulers share it; a lane with 16 x 8 outputs needs 24 numbers for 128 multiply-adds (0.75 of what the
// schedulers could use up), one with 8 x 8 needs 16 for 64 (all of it). Measured (launches in a row): 500 x 6144 x
// 1024 in 197 us and 500 x 1024 x 3072 in 97 (32 TFLOP/s; tiles of 64 x 64 of a whole CTA with one sum and 4 x 4 outputs a
// lane: 322 and 220 us), 1 x 1024 x 3072 in 12 us (214). Multiply-adds of three registers alone run at 60 TFLOP/s here; the
// rest goes to their registers' banks and to waiting for the next piece. Half the tile, twice the CTAs an SM: 259 and 134 us.
// With one sum a CTA is one warp, so that an SM holds ten of them and takes the next when one is done; small tiles, since K
// is too short to cut and many warps must share the outputs: 2048 x 4096 x 128 in 65 us, 2048 x 4096 x 64 in 36, 1 x 8192 x 128 in
// 3.6 (a CTA's tile of 64 x 64 and 4 x 4 outputs a lane: 98, 52 and 10.8; one warp of eight of a CTA of 160 KB: 330, 184 and 26).
#define ABK_DEFINE_ERROR
#include "common.cuh"
#include "gemm_split.cuh"

#define GS_WARPS 8      // of a CTA that cuts its sums
#define GS_BK 16
#define GS_PITCH 20     // floats of a staged row
#define GS_ONE_SUM 256  // up to this K an element is one sum

__device__ __forceinline__ void gs_copy_16(float *dst, const float *src, bool real) {
    const int bytes = real ? 16 : 0;  // 0: zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}

// How a warp brings its pieces. GS_PIECES: float32 operands whose rows start on 16-byte boundaries, K a multiple of 4, by
// cp.async; GS_VALUES: any others, number by number, the next piece asked for into registers while this one is multiplied.
// (Loads that the warp waited for one after the other: 500 x 1024 x 1023 float32 in 134 us and 500 x 1024 x 1020 bfloat16 in
// 144, now 42 and 43; 2048 x 2048 x 130 float32 954, now 45.)
enum { GS_PIECES, GS_VALUES };

// TM x TN: outputs a lane has, rows 4 apart and columns 8 apart; a tile has 4 TM x 8 TN. WARPS: GS_WARPS sums an element, or 1.
// STAGES: pieces of a warp in flight or in use.
template <typename TX, typename TW, typename TO, int TM, int TN, int WARPS, int STAGES, int LOADS>
__global__ void __launch_bounds__(32 * WARPS) gemm_simt_kernel(const TX *__restrict__ x, const TW *__restrict__ w, TO *__restrict__ out, int M,
                                                               int N, int K, long long ldx, long long ldw, long long ldo) {
    constexpr int BM = 4 * TM, BN = 8 * TN, STAGE = (BM + BN) * GS_PITCH;
    extern __shared__ __align__(16) float gs_smem[];  // [warps][stages][BM rows of x, then BN of w][20]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tx = lane & 7, ty = lane >> 3;
    const int m_tiles = (M + BM - 1) / BM, m0 = (int)(blockIdx.x % m_tiles) * BM, n0 = (int)(blockIdx.x / m_tiles) * BN;
    float *mine = gs_smem + warp * STAGES * STAGE;
    const int r_mine = lane >> 2, c_mine = (lane & 3) * 4;  // a lane's pieces: every 8th row from here
    const TX *x_mine = x + (long long)(m0 + r_mine) * ldx + c_mine;
    const TW *w_mine = w + (long long)(n0 + r_mine) * ldw + c_mine;
    const int r_single = lane >> 4, c_single = lane & 15;  // a lane's numbers where they come one by one: every 2nd row
    pdl_wait();
    const int pieces = (K + GS_BK - 1) / GS_BK;
    auto fetch = [&](int piece, int stage) {
        if (piece < pieces) {
            float *dst = mine + stage * STAGE;
            const int k0 = piece * GS_BK;
            const bool in = k0 + c_mine < K;
#pragma unroll
            for (int i = 0; i < BM / 8; i++) {
                const bool real = in && m0 + r_mine + 8 * i < M;
                gs_copy_16(dst + (r_mine + 8 * i) * GS_PITCH + c_mine, real ? (const float *)x_mine + 8 * i * ldx + k0 : (const float *)x, real);
            }
#pragma unroll
            for (int i = 0; i < BN / 8; i++) {
                const bool real = in && n0 + r_mine + 8 * i < N;
                gs_copy_16(dst + (BM + r_mine + 8 * i) * GS_PITCH + c_mine, real ? (const float *)w_mine + 8 * i * ldw + k0 : (const float *)w, real);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");  // (a group each time, empty beyond the last piece)
    };
    TX x_next[LOADS == GS_VALUES ? BM / 2 : 1];
    TW w_next[LOADS == GS_VALUES ? BN / 2 : 1];
    auto ask = [&](int piece) {
        const int k = piece * GS_BK + c_single;
        long long x_step = 2 * ldx, w_step = 2 * ldw;
        asm volatile("" : "+l"(x_step), "+l"(w_step));  // (or every row's address is kept in registers from piece to piece)
        const TX *xp = x + (long long)(m0 + r_single) * ldx + k;
        const TW *wp = w + (long long)(n0 + r_single) * ldw + k;
#pragma unroll
        for (int i = 0; i < BM / 2; i++, xp += x_step) x_next[i] = k < K && m0 + r_single + 2 * i < M ? *xp : from_float<TX>(0.0f);
#pragma unroll
        for (int i = 0; i < BN / 2; i++, wp += w_step) w_next[i] = k < K && n0 + r_single + 2 * i < N ? *wp : from_float<TW>(0.0f);
    };
    auto put = [&](int stage) {
        float *dst = mine + stage * STAGE + r_single * GS_PITCH + c_single;
#pragma unroll
        for (int i = 0; i < BM / 2; i++) dst[2 * i * GS_PITCH] = to_float(x_next[i]);
#pragma unroll
        for (int i = 0; i < BN / 2; i++) dst[(BM + 2 * i) * GS_PITCH] = to_float(w_next[i]);
    };
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) acc[i][j] = 0.0f;
    if constexpr (LOADS == GS_VALUES) {
        if (warp < pieces) ask(warp), put(0);
    } else {
#pragma unroll
        for (int s = 0; s < STAGES - 1; s++) fetch(warp + s * WARPS, s);
    }
    int stage = 0;
    for (int piece = warp; piece < pieces; piece += WARPS) {
        if constexpr (LOADS == GS_VALUES) {
            if (piece + WARPS < pieces) ask(piece + WARPS);
        } else {
            fetch(piece + (STAGES - 1) * WARPS, stage == 0 ? STAGES - 1 : stage - 1);
            asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 1) : "memory");
        }
        __syncwarp();
        const float *xs = mine + stage * STAGE + ty * GS_PITCH, *ws = mine + stage * STAGE + (BM + tx) * GS_PITCH;
#pragma unroll
        for (int k = 0; k < GS_BK; k += 2) {
            float2 a[TM], b[TN];
#pragma unroll
            for (int j = 0; j < TN; j++) b[j] = *(const float2 *)(ws + j * 8 * GS_PITCH + k);
#pragma unroll
            for (int i = 0; i < TM; i++) a[i] = *(const float2 *)(xs + i * 4 * GS_PITCH + k);
#pragma unroll
            for (int i = 0; i < TM; i++)
#pragma unroll
                for (int j = 0; j < TN; j++) acc[i][j] = fmaf(a[i].y, b[j].y, fmaf(a[i].x, b[j].x, acc[i][j]));
        }
        if constexpr (LOADS == GS_VALUES) {
            if (piece + WARPS < pieces) put(stage == STAGES - 1 ? 0 : stage + 1);
        }
        __syncwarp();  // the next iteration fills this stage again
        stage = stage == STAGES - 1 ? 0 : stage + 1;
    }
    if constexpr (WARPS == 1) {
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
            for (int j = 0; j < TN; j++)
                if (m0 + ty + 4 * i < M && n0 + tx + 8 * j < N) out[(long long)(m0 + ty + 4 * i) * ldo + n0 + tx + 8 * j] = from_float<TO>(acc[i][j]);
    } else {
        __syncthreads();
        constexpr int PITCH = BN + 8, TILE = BM * PITCH;  // (four rows' runs of eight columns lie in different banks)
        float *sums = gs_smem;  // [warps][BM][PITCH]
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
            for (int j = 0; j < TN; j++) sums[warp * TILE + (ty + 4 * i) * PITCH + tx + 8 * j] = acc[i][j];
        __syncthreads();
        for (int e = threadIdx.x; e < BM * BN; e += 32 * WARPS) {
            const int r = e / BN, c = e % BN;
            const float *s = sums + r * PITCH + c;
            if (m0 + r < M && n0 + c < N)
                out[(long long)(m0 + r) * ldo + n0 + c] = from_float<TO>(((s[0] + s[TILE]) + (s[2 * TILE] + s[3 * TILE])) + ((s[4 * TILE] + s[5 * TILE]) + (s[6 * TILE] + s[7 * TILE])));
        }
    }
}

template <typename TX, typename TW, typename TO, int TM, int TN, int WARPS, int STAGES, int LOADS>
static int gemm_simt_launch(const void *x, const void *w, void *out, int M, int N, int K, long long ldx, long long ldw, long long ldo, cudaStream_t s) {
    constexpr int BM = 4 * TM, BN = 8 * TN;
    constexpr int ring = WARPS * STAGES * (BM + BN) * GS_PITCH * 4, sums = WARPS == 1 ? 0 : WARPS * BM * (BN + 8) * 4, least = ring > sums ? ring : sums;
    const long long tiles = ((long long)M + BM - 1) / BM * (((long long)N + BN - 1) / BN);
    if (tiles > 0x7fffffffLL) ABK_REFUSE("gemm: %d x %d outputs are more than one launch takes", M, N);
    const dim3 grid((unsigned)tiles);
    // One warp a CTA: those that start while the kernel before still holds parts of the SMs gather where there is room (500 x
    // 2048 x 256, seven an SM: 25.5 us against 20.2), so each asks for so much shared memory that no SM takes more than its share.
    const long long share = (tiles + abk_sm_count() - 1) / abk_sm_count();
    const int even = WARPS == 1 && share <= 10 ? 228 * 1024 / (int)(share + 1) : 0, smem = even > least ? even : least;
    const cudaError_t e = abk_allow_shared_memory((const void *)gemm_simt_kernel<TX, TW, TO, TM, TN, WARPS, STAGES, LOADS>, smem);
    if (e != cudaSuccess) return (int)e;
    abk_launch(gemm_simt_kernel<TX, TW, TO, TM, TN, WARPS, STAGES, LOADS>, grid, dim3(32 * WARPS), smem, s, (const TX *)x, (const TW *)w, (TO *)out, M, N, K,
               ldx, ldw, ldo);
    return ABK_LAUNCH_RESULT();
}

// The product on the tensor cores (gemm_split.cuh), for any M and N and K from 193 on (every quarter of K has a piece of 64). bn: rows of x in a tile (32, 64, 96, 128), quarters: pairs of CTAs take
// quarters of K (not of bfloat16 operands below K = 2048, nor are there tiles of 128 then); 0, 0: by size. scratch: abk_gemm_split_scratch bytes.
extern "C" int abk_gemm_split(const void *x, const void *w, int dtype, void *out, int out_dtype, int M, int N, int K, long long ldx, long long ldw,
                              long long ldo, int bn, int quarters, void *scratch, int *status, void *stream) {
    const GemmSplit g = {x, w, out, dtype, out_dtype, M, N, K, 0, 0, ldx, ldw, ldo, status, nullptr};
    return dtype == ABK_F32 ? gemm_split_run<float>(g, bn, quarters, scratch, (cudaStream_t)stream)
                            : gemm_split_run<__nv_bfloat16>(g, bn, quarters, scratch, (cudaStream_t)stream);
}
extern "C" long long abk_gemm_split_scratch(int M, int N, int K) { return gemm_split_scratch(M, N, K); }

// Whether a product goes to the tensor cores: more than a handful of rows (up to 32 rows the plain kernel reads the weights once and
// writes nothing beside: 17 x 6144 x 1024 in 19 us against 23), and enough to do for two or three launches in place of one, whose
// host side takes some 12 us more: 64 x 6144 x 1024 in 27 us against 32, 100 x 4096 x 1024 in 21 against 36, 500 x 1024 x 1024 in 20 against
// 35; below that there is little to win (64 x 1024 x 1024: 12.8 against 13.4; 500 x 256 x 512: 10.3 against 7.9). 64 columns are one of the plain
// kernel's tiles and a quarter of a pair's: 6300 x 64 x 1024 in 39 us against 36, x 72 in 39 against 67. Up to 64 rows are one of its tiles too, and
// weights beyond the L2 are written and read again as parts: 33 x 40960 x 1024 in 145 against 157, x 65536 in 231 against 223; 40 x
// 16384 x 700 in 46 against 50, 33 x 24000 x 512 in 59 against 53. (bfloat16: 33 x 24000 x 513 in 50 against 77.)
static bool gemm_split_wins(int dtype, int M, int N, int K) {
    return M > 32 && N > 64 && K >= 512 && (long long)M * N * K >= 400000000LL && (dtype == ABK_BF16 || M > 64 || N < (K < 1024 ? 20000 : 65536));
}
// Bytes of scratch memory with which abk_gemm_simt goes to the tensor cores (0: it does not); dtype: of x and w.
extern "C" long long abk_gemm_simt_scratch(int M, int N, int K, int dtype) { return gemm_split_wins(dtype, M, N, K) ? gemm_split_scratch(M, N, K) : 0; }
// Kernels that abk_gemm_simt launches, given that scratch memory; dtype: of x and w.
extern "C" int abk_gemm_simt_kernels(int dtype, int M, int N, int K) {
    return M <= 0 || N <= 0 ? 0 : gemm_split_wins(dtype, M, N, K) ? gemm_split_kernels(M, N, K, dtype == ABK_F32 ? 3 : 1) : 1;
}

// x_dtype/w_dtype/out_dtype: ABK_F32 or ABK_BF16. Supported: all-float32; bf16 x and w with bf16 or f32 out.
// scratch: at least abk_gemm_simt_scratch bytes, or null (then every product runs on the CUDA cores); status: int32 [>= 2], word 1
// is set if a wait ran out.
extern "C" int abk_gemm_simt(const void *x, int x_dtype, const void *w, int w_dtype, void *out, int out_dtype, int M,
                             int N, int K, long long ldx, long long ldw, long long ldo, void *scratch, long long scratch_bytes, int *status,
                             void *stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) ABK_REFUSE("gemm: K = %d", K);
    cudaStream_t s = (cudaStream_t)stream;
    typedef __nv_bfloat16 bf;
    if (N > 65535 * 64) ABK_REFUSE("gemm: %d output columns are more than one launch takes", N);
    if (scratch && x_dtype == w_dtype && (x_dtype == ABK_BF16 || out_dtype == ABK_F32) && gemm_split_wins(x_dtype, M, N, K)) {
        if (scratch_bytes < gemm_split_scratch(M, N, K))
            ABK_REFUSE("gemm: %lld bytes of scratch memory for %d x %d x %d, which takes %lld", scratch_bytes, M, N, K, gemm_split_scratch(M, N, K));
        const GemmSplit g = {x, w, out, x_dtype, out_dtype, M, N, K, 0, 0, ldx, ldw, ldo, status, nullptr};
        return x_dtype == ABK_F32 ? gemm_split_run<float>(g, 0, 0, scratch, s) : gemm_split_run<bf>(g, 0, 0, scratch, s);
    }
    const bool one = K <= GS_ONE_SUM;
    const long long large = ((M + 63LL) / 64) * ((N + 63LL) / 64), small = ((M + 15LL) / 16) * ((N + 15LL) / 16), sms = abk_sm_count();
    // Eight sums: tiles of 64 x 64 where they fill two thirds of the SMs, else of 32 x 32 (of 16 x 16 for up to 16 rows): 64 x
    // 1024 x 3072, 16 large tiles or 64 of 32 x 32, in 114 or 34 us. One sum: tiles of 16 x 16 while an SM has up to seven of
    // them, else of 32 x 32: 100 x 2048 x 256 in 8.2 us against 10.8, 200 x 2048 x 256 in 16.1 against 12.6 (of 64 x 64: 56).
    const int tile = one ? small <= 7 * sms ? 16 : 32 : large >= sms * 2 / 3 ? 64 : M > 16 ? 32 : 16;
#define GS_LAUNCH(TX, TW, TO, LARGE, STAGES, LOADS)                                                                    \
    (one ? tile == 32 ? gemm_simt_launch<TX, TW, TO, 8, 4, 1, STAGES, LOADS>(x, w, out, M, N, K, ldx, ldw, ldo, s)     \
                      : gemm_simt_launch<TX, TW, TO, 4, 2, 1, STAGES, LOADS>(x, w, out, M, N, K, ldx, ldw, ldo, s)     \
     : tile == 64 ? gemm_simt_launch<TX, TW, TO, LARGE, 8, GS_WARPS, 2, LOADS>(x, w, out, M, N, K, ldx, ldw, ldo, s)   \
     : tile == 32 ? gemm_simt_launch<TX, TW, TO, 8, 4, GS_WARPS, 2, LOADS>(x, w, out, M, N, K, ldx, ldw, ldo, s)       \
                  : gemm_simt_launch<TX, TW, TO, 4, 2, GS_WARPS, 2, LOADS>(x, w, out, M, N, K, ldx, ldw, ldo, s))
    // (large tiles of 32 x 64 where the next piece needs room in the registers)
    if (x_dtype == ABK_F32 && w_dtype == ABK_F32 && out_dtype == ABK_F32) {
        const bool aligned = K % 4 == 0 && ldx % 4 == 0 && ldw % 4 == 0 && !(((uintptr_t)x | (uintptr_t)w) & 15);
        return aligned ? GS_LAUNCH(float, float, float, 16, 4, GS_PIECES) : GS_LAUNCH(float, float, float, 8, 2, GS_VALUES);
    }
    if (x_dtype == ABK_BF16 && w_dtype == ABK_BF16 && out_dtype == ABK_BF16) return GS_LAUNCH(bf, bf, bf, 8, 2, GS_VALUES);
    if (x_dtype == ABK_BF16 && w_dtype == ABK_BF16 && out_dtype == ABK_F32) return GS_LAUNCH(bf, bf, float, 8, 2, GS_VALUES);
#undef GS_LAUNCH
    ABK_REFUSE("gemm: dtype combination x=%d w=%d out=%d is not built", x_dtype, w_dtype, out_dtype);
}
