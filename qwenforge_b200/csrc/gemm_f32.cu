// True 32-bit matrix product of the float32 path:  C[M][N] = A[M][K] * W[N][K]^T (+ bias[N]).
// FFMA only, no tensor cores, no TF32. Every output element is one chain of fused multiply-adds
// over k = 0 .. K-1 in that order, whatever M, the tiling or the batch: a row's result is bitwise
// the same however the rows were grouped into calls.
#include "mma.cuh"

// Two neighbouring float32 as one 64-bit register pair: one instruction multiplies and adds both, each rounded as fmaf rounds it.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 both(float x) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float2 halves(f32x2 x) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(x));
    return r;
}

// A block makes a BM x BN tile with WM x WN warps; a warp makes (4 TM) x (8 TN) of it, its 4 x 8 lanes TM x TN each in runs of four rows
// and columns (two columns, where a lane's are no whole fours), so that the lanes of a warp read a k's rows and columns of both operands as whole
// pieces without conflicts. Which rows and columns a lane has: neighbouring lanes share one of the two, and a 16-byte load of eight pieces takes two cycles of
// the shared memory, four where eight neighbours have eight (32 x 64 tiles 12 to 15% faster so, the larger ones up to 2%; 64 x 64 in few rounds
// 1.5% slower, so not there). 16
// or 32 columns of K at a time, the next ones on their way through registers: they are turned on the way into shared memory, where
// the rows of every eight k are swapped among themselves so that a warp's stores of four k a lane meet all 32 banks. Rows go two to
// a register pair, and a column's number twice into one.
// What bounds it is the multiply-add pipe (72 TFLOP/s; 79% of its cycles on 96 x 128 tiles) and, for small tiles, the shared memory's loads
// (90% on 64 x 64), then the last tiles' round. 1,031 rows of the 0.5B model's products (30.6 GFLOP): 1,441 microseconds with 64 x 64
// tiles read by single words, 840 with 64 x 128 and 64 x 64 tiles whose stores met half the banks, 714 so; 1,031 x 22,016 x 2,048
// 1,911 before and 1,631 (57 TFLOP/s).
template <int TM, int TN, int WM, int WN, int BK>
__global__ void __launch_bounds__(32 * WM * WN, TM * TN >= 128 ? 256 / (32 * WM * WN) : TM * TN >= 64 ? 384 / (32 * WM * WN) : 512 / (32 * WM * WN))
gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                float* __restrict__ C, int M, int N, int K, int lda, int ldw, int ldc, int vec) {
    constexpr int THREADS = 32 * WM * WN, BM = 4 * TM * WM, BN = 8 * TN * WN, LA = BM + 4, LW = BN + 4, Q = BK / 4, SWAP = BK == 16 ? 8 : 4;
    constexpr int A_EACH = BM * Q / THREADS, W_EACH = BN * Q / THREADS, RW = TN % 4 ? 2 : 4;
    static_assert(TM % 4 == 0 && TN % 2 == 0 && BM * Q % THREADS == 0 && BN * Q % THREADS == 0 && BM % 16 == 0 && BN % 16 == 0, "whole runs");
    __shared__ __align__(16) float a_s[2][BK][LA], w_s[2][BK][LW];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    constexpr bool SHARED = !(TM == 8 && TN == 4);
    const int row0 = (warp / WN) * 4 * TM + (SHARED ? lane >> 1 & 3 : lane >> 3) * 4;
    const int col0 = (warp % WN) * 8 * TN + (SHARED ? (lane & 1) | (lane >> 2 & 6) : lane & 7) * RW;
    f32x2 acc[TM / 2][TN];            // rows 2 i and 2 i + 1 of column j
#pragma unroll
    for (int i = 0; i < TM / 2; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;

    // four neighbouring k of a row per piece; rows beyond M or N and columns beyond K are zeros
    float4 a_next[A_EACH], w_next[W_EACH];
    auto piece = [&](const float* X, int ld, int row, int rows, int k) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row < rows) {
            const float* p = X + (size_t)row * ld + k;
            if (vec) {
                if (k < K) v = *reinterpret_cast<const float4*>(p);
            } else {
                if (k < K) v.x = p[0];
                if (k + 1 < K) v.y = p[1];
                if (k + 2 < K) v.z = p[2];
                if (k + 3 < K) v.w = p[3];
            }
        }
        return v;
    };
    auto fetch = [&](int k0) {
#pragma unroll
        for (int u = 0; u < A_EACH; ++u) {
            const int i = threadIdx.x + u * THREADS;
            a_next[u] = piece(A, lda, m0 + i / Q, M, k0 + (i % Q) * 4);
        }
#pragma unroll
        for (int u = 0; u < W_EACH; ++u) {
            const int i = threadIdx.x + u * THREADS;
            w_next[u] = piece(W, ldw, n0 + i / Q, N, k0 + (i % Q) * 4);
        }
    };
    auto stash = [&](int buf) {
        const int k = (threadIdx.x % Q) * 4, swap = k / 8 * SWAP;
#pragma unroll
        for (int u = 0; u < A_EACH; ++u) {
            const int r = ((threadIdx.x + u * THREADS) / Q) ^ swap;
            a_s[buf][k][r] = a_next[u].x, a_s[buf][k + 1][r] = a_next[u].y;
            a_s[buf][k + 2][r] = a_next[u].z, a_s[buf][k + 3][r] = a_next[u].w;
        }
#pragma unroll
        for (int u = 0; u < W_EACH; ++u) {
            const int r = ((threadIdx.x + u * THREADS) / Q) ^ swap;
            w_s[buf][k][r] = w_next[u].x, w_s[buf][k + 1][r] = w_next[u].y;
            w_s[buf][k + 2][r] = w_next[u].z, w_s[buf][k + 3][r] = w_next[u].w;
        }
    };
    fetch(0);
    stash(0);
    __syncthreads();
    for (int k0 = 0, buf = 0; k0 < K; k0 += BK, buf ^= 1) {
        if (k0 + BK < K) fetch(k0 + BK);
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            f32x2 a[TM / 2];
            float w[TN];
#pragma unroll
            for (int i = 0; i < TM; i += 4) {   // runs of four rows, 16 rows apart
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&a_s[buf][k][(row0 + 4 * i) ^ (k / 8 * SWAP)]);
                a[i / 2] = v.x, a[i / 2 + 1] = v.y;
            }
#pragma unroll
            for (int j = 0; j < TN; j += RW) {   // runs of four columns, 32 apart, or of two, 16 apart
                const float* p = &w_s[buf][k][(col0 + 8 * j) ^ (k / 8 * SWAP)];
                if (RW == 4) { const float4 v = *reinterpret_cast<const float4*>(p); w[j] = v.x, w[j + 1] = v.y, w[(j + 2) % TN] = v.z, w[(j + 3) % TN] = v.w; }
                else { const float2 v = *reinterpret_cast<const float2*>(p); w[j] = v.x, w[j + 1] = v.y; }
            }
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const f32x2 wj = both(w[j]);
#pragma unroll
                for (int i = 0; i < TM / 2; ++i) acc[i][j] = fma2(a[i], wj, acc[i][j]);
            }
        }
        if (k0 + BK < K) {
            stash(buf ^ 1);      // (read in the turn before, which ended with a barrier)
            __syncthreads();
        }
    }
#pragma unroll
    for (int i = 0; i < TM / 2; ++i) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int gm = m0 + row0 + (i / 2) * 16 + (2 * i) % 4 + h;
            if (gm >= M) continue;
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const float2 v = halves(acc[i][j]);
                const int gn = n0 + col0 + j / RW * 8 * RW + j % RW;
                if (gn < N) C[(size_t)gm * ldc + gn] = (h ? v.y : v.x) + (bias ? bias[gn] : 0.f);
            }
        }
    }
}

// The same product for 16 rows or fewer (decode steps), where tiles of 64 rows would be mostly padding and a handful of
// blocks would stream all the weights. A block takes 8 * NPT weight rows and all (up to 16) token rows: thread (n, m)
// owns the output elements (n + 8 i, m), each still ONE chain of fused multiply-adds over k = 0 .. K-1 in that order
// (zeros beyond K add nothing), so its bits are those of the kernel above. The chain is what bounds a block (4 cycles
// per k), so products of few weight rows are spread over N / 8 blocks (NPT = 1) and the others give a thread four
// chains (NPT = 4); the next columns of both operands arrive by cp.async, two stages ahead of the multiplication.
#define FR_N 8
#define FR_M 16
#define FR_STAGES 3
template <int NPT, int KC>
__global__ void __launch_bounds__(FR_N * FR_M)
gemm_f32_few_rows_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                         float* __restrict__ C, int M, int N, int K, int lda, int ldw, int ldc) {
    constexpr int LD = KC + 4;         // rows 16 bytes apart in the banks: 8 weight rows and 4 token rows read without conflicts
    constexpr int WR = FR_N * NPT;     // weight rows of a block
    __shared__ __align__(16) float w_s[FR_STAGES][WR][LD];
    __shared__ __align__(16) float a_s[FR_STAGES][FR_M][LD];
    const int n = threadIdx.x % FR_N, m = threadIdx.x / FR_N;
    const int n0 = blockIdx.x * WR;
    // whole 16-byte pieces go by cp.async when rows and K allow it; otherwise element by element
    const bool vec = (K % 4 == 0) && (lda % 4 == 0) && (ldw % 4 == 0) && ((((uintptr_t)A) | ((uintptr_t)W)) % 16 == 0);
    auto fetch = [&](int k0, int buf) {
        if (k0 >= K) return;
        if (vec) {
            for (int i = threadIdx.x; i < (WR + FR_M) * (KC / 4); i += FR_N * FR_M) {
                const int r = i / (KC / 4), k = (i % (KC / 4)) * 4;
                const bool is_w = r < WR;
                const int row = is_w ? n0 + r : r - WR;
                const bool ok = (is_w ? row < N : row < M) && k0 + k < K;
                const float* src = is_w ? W + (size_t)row * ldw + k0 + k : A + (size_t)row * lda + k0 + k;
                cp_async_16(is_w ? &w_s[buf][r][k] : &a_s[buf][r - WR][k], ok ? src : W, ok);
            }
        } else {
            for (int i = threadIdx.x; i < (WR + FR_M) * KC; i += FR_N * FR_M) {
                const int r = i / KC, k = i % KC;
                const bool is_w = r < WR;
                const int row = is_w ? n0 + r : r - WR;
                const bool ok = (is_w ? row < N : row < M) && k0 + k < K;
                const float v = ok ? (is_w ? W[(size_t)row * ldw + k0 + k] : A[(size_t)row * lda + k0 + k]) : 0.f;
                if (is_w) w_s[buf][r][k] = v;
                else a_s[buf][r - WR][k] = v;
            }
        }
    };
    float acc[NPT];
#pragma unroll
    for (int i = 0; i < NPT; ++i) acc[i] = 0.f;
    fetch(0, 0);
    cp_async_commit();
    fetch(KC, 1);
    cp_async_commit();
    for (int k0 = 0, turn = 0; k0 < K; k0 += KC, ++turn) {
        const int buf = turn % FR_STAGES;
        fetch(k0 + 2 * KC, (turn + 2) % FR_STAGES);   // its stage was read two turns ago, before that turn's last barrier
        cp_async_commit();
        cp_async_wait<2>();
        __syncthreads();
#pragma unroll 4
        for (int k = 0; k < KC; k += 4) {
            const float4 a = *reinterpret_cast<const float4*>(&a_s[buf][m][k]);
#pragma unroll
            for (int i = 0; i < NPT; ++i) {
                const float4 w = *reinterpret_cast<const float4*>(&w_s[buf][n + FR_N * i][k]);
                acc[i] = fmaf(a.x, w.x, acc[i]);
                acc[i] = fmaf(a.y, w.y, acc[i]);
                acc[i] = fmaf(a.z, w.z, acc[i]);
                acc[i] = fmaf(a.w, w.w, acc[i]);
            }
        }
        __syncthreads();
    }
    cp_async_wait<0>();
    if (m < M) {
#pragma unroll
        for (int i = 0; i < NPT; ++i) {
            const int col = n0 + n + FR_N * i;
            if (col < N) C[(size_t)m * ldc + col] = acc[i] + (bias ? bias[col] : 0.f);
        }
    }
}

// The tile with which the busiest SM is done first: a first wait and a time per tile, measured at K = 896 in microseconds (between events, a launch's
// 8 to 10 among them, 1 and 18 tiles per SM of 64 x 64 40 and 392, of 128 x 128 97 and 1,364, of 96 x 128 82 and 995, of 96 x 64 53 and 566, of
// 96 x 96 67 and 825: a time per tile is a seventeenth of the difference; 1,031 x 1,152 x 896 in one round of 96 x 96 61 microseconds, in three of
// 64 x 64 73). The 32 x 64 tile's time is the one that it had before its lanes shared operands; now 30 and 229, 11.7 a tile, with which it
// would be taken in more places (700 x 2,048 x 2,048 165 / 155, 300 x 2,560 x 2,048 116 / 100, but 330 x 9,728 x 896 153 / 156). Never the
// fastest by more than a twentieth: 64 x 128 and 64 x 256 with two or four warps, 32 x 64 with two warps, 128 x 64. (With K a tile's time grows
// and its wait does not: the waits, which count here as at K = 896, decide between tiles whose rounds take nearly the same time.)
static const struct { int bm, bn; float wait, each; } f32_tiles[] = {{96, 128, 18.f, 53.7f}, {128, 128, 13.5f, 74.5f}, {96, 64, 15.f, 30.f},
                                                                     {64, 64, 8.5f, 20.8f}, {32, 64, 8.f, 14.3f}, {96, 96, 17.f, 44.2f}};
static int best_tile(int M, int N) {
    const int sms = qf_sm_count() > 0 ? qf_sm_count() : 1;
    int best = 0;
    float least = 0.f;
    for (int i = 0; i < 6; ++i) {
        const long long count = (long long)((M + f32_tiles[i].bm - 1) / f32_tiles[i].bm) * ((N + f32_tiles[i].bn - 1) / f32_tiles[i].bn);
        const float time = f32_tiles[i].wait + (float)((count + sms - 1) / sms) * f32_tiles[i].each;
        if (i == 0 || time < least) best = i, least = time;
    }
    return best;
}
// Which tile a product of more than 16 rows takes: 1,000 x its rows + its columns.
QF_EXPORT int qf_gemm_f32_tile(int M, int N) { return f32_tiles[best_tile(M, N)].bm * 1000 + f32_tiles[best_tile(M, N)].bn; }

QF_EXPORT int qf_gemm_f32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda,
                          int ldw, int ldc, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (M <= 16) {
        if (N <= 4096) gemm_f32_few_rows_kernel<1, 128><<<(N + 7) / 8, FR_N * FR_M, 0, stream>>>(A, W, bias, C, M, N, K, lda, ldw, ldc);
        else gemm_f32_few_rows_kernel<4, 64><<<(N + 31) / 32, FR_N * FR_M, 0, stream>>>(A, W, bias, C, M, N, K, lda, ldw, ldc);
        return (int)cudaGetLastError();
    }
    const int vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
    const int best = best_tile(M, N);
    const dim3 grid((N + f32_tiles[best].bn - 1) / f32_tiles[best].bn, (M + f32_tiles[best].bm - 1) / f32_tiles[best].bm);
#define QF_F32(TM, TN, BK) gemm_f32_kernel<TM, TN, 2, 2, BK><<<grid, 128, 0, stream>>>(A, W, bias, C, M, N, K, lda, ldw, ldc, vec)
    if (best == 0) QF_F32(12, 8, 16);
    else if (best == 1) QF_F32(16, 8, 16);
    else if (best == 2) QF_F32(12, 4, 16);
    else if (best == 3) QF_F32(8, 4, 32);
    else if (best == 4) QF_F32(4, 4, 32);
    else QF_F32(12, 6, 16);
#undef QF_F32
    return (int)cudaGetLastError();
}
