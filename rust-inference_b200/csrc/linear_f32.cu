// y[M, N] = x[M, K] . W[N, K]^T in true float32 (FMA on the CUDA cores, no tensor
// cores, no reduced-precision mode).  Every output element is the sum over
// k = 0..K-1 in that order with one accumulator, whatever M, N and the tile a
// row falls into: a token's result does not depend on what it is batched with.
// Formula: thanhauco/rust-inference src/ops/linear.rs:7-20.
#include "common.cuh"

#define LF_BM 64
#define LF_BN 64
#define LF_BK 16
#define LF_THREADS 256

__global__ void __launch_bounds__(LF_THREADS)
linear_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y, int M, int N, int K,
                  int vec_ok, long long ldx, long long ldy, long long x_batch, long long w_batch, long long y_batch) {
    // blockIdx.z: one product of a batch (a head); rows of x and y may lie ldx / ldy elements apart
    x += (size_t)blockIdx.z * x_batch;
    w += (size_t)blockIdx.z * w_batch;
    y += (size_t)blockIdx.z * y_batch;
    __shared__ float xs[LF_BK][LF_BM + 4];
    __shared__ float ws[LF_BK][LF_BN + 4];
    int m0 = blockIdx.y * LF_BM, n0 = blockIdx.x * LF_BN;
    int tid = threadIdx.x;
    int tx = tid % 16, ty = tid / 16;          // thread owns rows ty*4.., cols tx*4..
    int lrow = tid / 4, lk = (tid % 4) * 4;    // loader: row of the tile, 4 consecutive k
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.0f;

    for (int k0 = 0; k0 < K; k0 += LF_BK) {
        float xv[4], wv[4];
        int gm = m0 + lrow, gn = n0 + lrow, gk = k0 + lk;
        if (vec_ok && gk + 3 < K) {
            float4 a = gm < M ? *(const float4*)(x + (size_t)gm * ldx + gk) : make_float4(0, 0, 0, 0);
            float4 b = gn < N ? *(const float4*)(w + (size_t)gn * K + gk) : make_float4(0, 0, 0, 0);
            xv[0] = a.x; xv[1] = a.y; xv[2] = a.z; xv[3] = a.w;
            wv[0] = b.x; wv[1] = b.y; wv[2] = b.z; wv[3] = b.w;
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                xv[i] = (gm < M && gk + i < K) ? x[(size_t)gm * ldx + gk + i] : 0.0f;
                wv[i] = (gn < N && gk + i < K) ? w[(size_t)gn * K + gk + i] : 0.0f;
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; i++) {
            xs[lk + i][lrow] = xv[i];
            ws[lk + i][lrow] = wv[i];
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < LF_BK; kk++) {
            float4 a = *(const float4*)&xs[kk][ty * 4];
            float4 b = *(const float4*)&ws[kk][tx * 4];
            float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        int gm = m0 + ty * 4 + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            int gn = n0 + tx * 4 + j;
            if (gn < N) y[(size_t)gm * ldy + gn] = acc[i][j];
        }
    }
}

// The same for more rows: 128 x 16 TN outputs a block, eight rows and TN columns a thread, two neighbouring columns an instruction
// (fma.rn.f32x2 rounds each as fmaf does), the next 16 k on their way in registers and two buffers in shared memory.  What
// bounds it: the multiply-adds (one instruction of two takes two cycles of a scheduler) and, at half their rate, the words that a
// thread reads from shared memory for them: 16 for 64 with TN = 8, where the kernel above reads 8 for 16.  Every output is the
// same chain of multiply-adds over ascending k: the same bits.  512 tokens of width 4,096 and 6,144 outputs:
// 643 us, 40 TFLOP/s, where the kernel above takes 893 us; 2,048 tokens 2,140 (48 TFLOP/s) and 2,961 us.
#define LW_BM 128
#define LW_THREADS 256
template <int TN>
__global__ void __launch_bounds__(LW_THREADS, 2)
linear_f32_wide_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y, int M, int N, int K,
                       int vec_ok, long long ldx, long long ldy, long long x_batch, long long w_batch, long long y_batch) {
    constexpr int BN = 16 * TN, BK = LF_BK;
    constexpr int WPER = BN * BK / 4 / LW_THREADS + (BN * BK / 4 % LW_THREADS ? 1 : 0);      // 16-byte pieces of W per thread
    x += (size_t)blockIdx.z * x_batch;
    w += (size_t)blockIdx.z * w_batch;
    y += (size_t)blockIdx.z * y_batch;
    __shared__ __align__(16) float xs[2][BK][LW_BM + 4];
    __shared__ __align__(16) float ws[2][BK][BN + 4];
    const int m0 = blockIdx.y * LW_BM, n0 = blockIdx.x * BN;
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;       // rows 4 ty .. and 64 + 4 ty .., columns 2 tx + 32 j ..
    float xr[2][4], wr[WPER][4];
    auto piece = [&](const float* p, int row, int rows, long long ld, int k, float (&v)[4]) {
        if (vec_ok && k + 3 < K) {
            const float4 f = row < rows ? *(const float4*)(p + (size_t)row * ld + k) : make_float4(0, 0, 0, 0);
            v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++) v[i] = (row < rows && k + i < K) ? p[(size_t)row * ld + k + i] : 0.0f;
        }
    };
    auto fetch = [&](int k0) {
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int i = tid + e * LW_THREADS;
            piece(x, m0 + i / 4, M, ldx, k0 + (i % 4) * 4, xr[e]);
        }
#pragma unroll
        for (int e = 0; e < WPER; e++) {
            const int i = tid + e * LW_THREADS;
            if (i < BN * 4) piece(w, n0 + i / 4, N, K, k0 + (i % 4) * 4, wr[e]);
        }
    };
    auto store = [&](int buf) {
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int i = tid + e * LW_THREADS;
#pragma unroll
            for (int c = 0; c < 4; c++) xs[buf][(i % 4) * 4 + c][i / 4] = xr[e][c];
        }
#pragma unroll
        for (int e = 0; e < WPER; e++) {
            const int i = tid + e * LW_THREADS;
            if (i < BN * 4)
#pragma unroll
                for (int c = 0; c < 4; c++) ws[buf][(i % 4) * 4 + c][i / 4] = wr[e][c];
        }
    };
    typedef unsigned long long f32x2;
    f32x2 acc[8][TN / 2];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < TN / 2; j++) acc[i][j] = 0ull;
    fetch(0);
    store(0);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < K; k0 += BK) {
        const bool more = k0 + BK < K;
        if (more) fetch(k0 + BK);
#pragma unroll
        for (int kk = 0; kk < BK; kk++) {
            const float4 a0 = *(const float4*)&xs[buf][kk][ty * 4], a1 = *(const float4*)&xs[buf][kk][64 + ty * 4];
            f32x2 b[TN / 2];
#pragma unroll
            for (int j = 0; j < TN / 2; j++) b[j] = *(const f32x2*)&ws[buf][kk][2 * tx + 32 * j];
            const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
            for (int i = 0; i < 8; i++) {
                f32x2 aa;
                asm("mov.b64 %0, {%1, %1};" : "=l"(aa) : "f"(av[i]));
#pragma unroll
                for (int j = 0; j < TN / 2; j++) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][j]) : "l"(aa), "l"(b[j]));
            }
        }
        if (more) store(buf ^ 1);
        __syncthreads();
        buf ^= 1;
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int gm = m0 + (i / 4) * 64 + ty * 4 + i % 4;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < TN / 2; j++) {
            float lo, hi;
            asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(acc[i][j]));
            const int gn = n0 + 2 * tx + 32 * j;
            if (gn < N) y[(size_t)gm * ldy + gn] = lo;
            if (gn + 1 < N) y[(size_t)gm * ldy + gn + 1] = hi;
        }
    }
}

// Which kernel: the one whose busiest SM has the least to do, in outputs times what one costs there.  Measured at K = 4,096: a
// block of the wide kernel 430 us with TN = 8, 334 with 6, 250 with 4 (26 to 30 ns an output, with one or more blocks on
// the SM alike); one of the first kernel 146 us among several (36 ns an output) and 334 us alone, so it is left for few rows
// of more outputs than the SMs take at once.  64 rows of 4,096 outputs: 250 us with TN = 4, 334 with the first; 512 rows of 4,096:
// 455 with TN = 8, 479 with 4, 586 with the first.
static int lf_launch(const float* x, const float* w, float* y, int M, int N, int K, int heads, int vec_ok, long long ldx, long long ldy,
                     long long x_head, long long w_head, long long y_head, cudaStream_t stream) {
    static int sms = 0;
    if (!sms) {
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        sms = n > 0 ? n : 148;
    }
    auto cost = [&](int bm, int bn, double each) {
        const long long blocks = (long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn) * heads;
        return (double)((blocks + sms - 1) / sms) * bm * bn * each;
    };
    const double alone = 2.3 * LF_BM * LF_BN * 1.36, first = cost(LF_BM, LF_BN, 1.36);
    const double c[4] = {first < alone ? alone : first, cost(LW_BM, 64, 1.17), cost(LW_BM, 96, 1.06), cost(LW_BM, 128, 1.0)};
    int best = 0;
    for (int i = 1; i < 4; i++)
        if (c[i] < c[best]) best = i;
    const int bm = best ? LW_BM : LF_BM, bn = best == 0 ? LF_BN : best == 1 ? 64 : best == 2 ? 96 : 128;
    const dim3 grid((N + bn - 1) / bn, (M + bm - 1) / bm, heads);
#define LW_GO(TN) linear_f32_wide_kernel<TN><<<grid, LW_THREADS, 0, stream>>>(x, w, y, M, N, K, vec_ok, ldx, ldy, x_head, w_head, y_head)
    if (best == 0) linear_f32_kernel<<<grid, LF_THREADS, 0, stream>>>(x, w, y, M, N, K, vec_ok, ldx, ldy, x_head, w_head, y_head);
    else if (best == 1) LW_GO(4);
    else if (best == 2) LW_GO(6);
    else LW_GO(8);
#undef LW_GO
    RI_CHECK_LAUNCH("linear_f32");
    return 0;
}

extern "C" int ri_linear_f32(const float* x, const float* w, float* y, int M, int N, int K, cudaStream_t stream) {
    if (M == 0 || N == 0) return 0;
    RI_REQUIRE(M > 0 && N > 0 && K > 0, "linear_f32: bad sizes M=%d N=%d K=%d", M, N, K);
    RI_REQUIRE((M + LF_BM - 1) / LF_BM <= 65535, "linear_f32: too many rows (%d)", M);
    int vec_ok = (K % 4 == 0) && (((uintptr_t)x | (uintptr_t)w) % 16 == 0);
    return lf_launch(x, w, y, M, N, K, 1, vec_ok, K, N, 0, 0, 0, stream);
}

// One product per head: y[m, h, :] = x[m, h, :] . W[h]^T with W [heads, N, K] dense, x rows of K elements that start
// ldx apart per token and x_head apart per head, y likewise (ldy, y_head).  The arithmetic of an output element is
// that of ri_linear_f32.
extern "C" int ri_linear_heads_f32(const float* x, const float* w, float* y, int M, int heads, int N, int K, long long ldx,
                                   long long x_head, long long ldy, long long y_head, cudaStream_t stream) {
    if (M == 0 || N == 0 || heads == 0) return 0;
    RI_REQUIRE(M > 0 && N > 0 && K > 0 && heads > 0, "linear_heads_f32: bad sizes M=%d heads=%d N=%d K=%d", M, heads, N, K);
    RI_REQUIRE((M + LF_BM - 1) / LF_BM <= 65535 && heads <= 65535, "linear_heads_f32: too many rows or heads (%d, %d)", M, heads);
    int vec_ok = (K % 4 == 0) && (ldx % 4 == 0) && (x_head % 4 == 0) && (((uintptr_t)x | (uintptr_t)w) % 16 == 0);
    return lf_launch(x, w, y, M, N, K, heads, vec_ok, ldx, ldy, x_head, (long long)N * K, y_head, stream);
}
