// y[M, N] = x[M, K] . W[N, K]^T in true float32, in two forms that K and W alone decide between.
// `ri_linear_f32`, `ri_linear_heads_f32`: multiply-adds on the CUDA cores.  Every output element is the sum over
// k = 0..K-1 in that order with one accumulator, whatever M, N and the tile a row falls into: a token's result does not
// depend on what it is batched with.
// `ri_linear_f32_tc`: exact cuts of the float32 values into bfloat16 on the tensor cores (linear_f32_tc.cuh), likewise the same chains for
// every output whatever M, N and the tile.
// Formula: thanhauco/rust-inference src/ops/linear.rs:7-20.
#include "common.cuh"
#include "linear_f32_tc.cuh"
#include <cuda.h>

#define LF_BK 16
#define LF_THREADS 256

// A block has 16 TM rows of 16 TN outputs, a thread TM rows and TN columns of them, two neighbouring columns an instruction
// (fma.rn.f32x2 rounds each as fmaf does), the next 16 k on their way in registers and two buffers in shared memory.
// blockIdx.z: one product of a batch (a head); rows of x and y may lie ldx / ldy elements apart.  What bounds it: with many blocks the
// multiply-adds (one instruction of two takes two cycles of a scheduler) and, at half their rate for TM = TN = 8, the
// words that a thread reads from shared memory for them; with a block an SM the trip of the next 16 k and the barrier behind it.
// Every output is one chain of multiply-adds over ascending k: the same bits from every tile.  Width 4,096, where 64 x 64
// outputs a block with one buffer and one multiply-add an instruction took: 512 tokens and 6,144 outputs 641 us (40 TFLOP/s), 885;
// 512 and 12,288 1,194, 1,576; up to 128 tokens and 4,096 outputs, weights in the L2 cache 152 to 171 (TM = TN = 4), 228 to 280,
// and from memory 190, 332.
template <int TM, int TN>
__global__ void __launch_bounds__(LF_THREADS, TM == 8 ? 2 : 4)
linear_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y, int M, int N, int K,
                  int vec_ok, long long ldx, long long ldy, long long x_batch, long long w_batch, long long y_batch) {
    constexpr int BM = 16 * TM, BN = 16 * TN, BK = LF_BK;
    constexpr int XPER = BM * BK / 4 / LF_THREADS;                                            // 16-byte pieces of X per thread
    constexpr int WPER = BN * BK / 4 / LF_THREADS + (BN * BK / 4 % LF_THREADS ? 1 : 0);      // ... and of W
    x += (size_t)blockIdx.z * x_batch;
    w += (size_t)blockIdx.z * w_batch;
    y += (size_t)blockIdx.z * y_batch;
    __shared__ __align__(16) float xs[2][BK][BM + 4];
    __shared__ __align__(16) float ws[2][BK][BN + 4];
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;       // rows 4 ty .. and 64 + 4 ty .., columns 2 tx + 32 j ..
    float xr[XPER][4], wr[WPER][4];
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
        for (int e = 0; e < XPER; e++) {
            const int i = tid + e * LF_THREADS;
            piece(x, m0 + i / 4, M, ldx, k0 + (i % 4) * 4, xr[e]);
        }
#pragma unroll
        for (int e = 0; e < WPER; e++) {
            const int i = tid + e * LF_THREADS;
            if (i < BN * 4) piece(w, n0 + i / 4, N, K, k0 + (i % 4) * 4, wr[e]);
        }
    };
    auto store = [&](int buf) {
#pragma unroll
        for (int e = 0; e < XPER; e++) {
            const int i = tid + e * LF_THREADS;
#pragma unroll
            for (int c = 0; c < 4; c++) xs[buf][(i % 4) * 4 + c][i / 4] = xr[e][c];
        }
#pragma unroll
        for (int e = 0; e < WPER; e++) {
            const int i = tid + e * LF_THREADS;
            if (i < BN * 4)
#pragma unroll
                for (int c = 0; c < 4; c++) ws[buf][(i % 4) * 4 + c][i / 4] = wr[e][c];
        }
    };
    typedef unsigned long long f32x2;
    f32x2 acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; i++)
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
            const float4 a0 = *(const float4*)&xs[buf][kk][ty * 4], a1 = *(const float4*)&xs[buf][kk][(TM == 8 ? 64 : 0) + ty * 4];
            f32x2 b[TN / 2];
#pragma unroll
            for (int j = 0; j < TN / 2; j++) b[j] = *(const f32x2*)&ws[buf][kk][2 * tx + 32 * j];
            const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
            for (int i = 0; i < TM; i++) {
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
    for (int i = 0; i < TM; i++) {
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

// Which tile: the one with the least time on the busiest SM, `alone` for its first block and `more` for each further one.  Measured
// in us at K = 4,096 with 1 to 28 blocks an SM (tiles 64 x 64, 128 x 64, 128 x 96, 128 x 128): 162 to 190 from the L2 cache and from
// memory, then 135 a block; 245 to 270 and 213; 334 to 356 and 290; 430 to 454 and 374.  Where they cross, 64 rows by 12,288 outputs: 287
// (64 x 64, two blocks), 451, 344, 434; 129 rows by 6,144 291, 442, 359, 453; 512 rows by 4,096 563, 477, 645, 455.
static int lf_launch(const float* x, const float* w, float* y, int M, int N, int K, int heads, int vec_ok, long long ldx, long long ldy,
                     long long x_head, long long w_head, long long y_head, cudaStream_t stream) {
    static int sms = 0;
    if (!sms) {
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        sms = n > 0 ? n : 148;
    }
    struct Tile {
        int bm, bn;
        double alone, more;
    };
    static const Tile tiles[4] = {{64, 64, 170, 135}, {128, 64, 265, 213}, {128, 96, 350, 290}, {128, 128, 445, 374}};
    int best = 0;
    double least = 0;
    for (int i = 0; i < 4; i++) {
        const long long blocks = (long long)((M + tiles[i].bm - 1) / tiles[i].bm) * ((N + tiles[i].bn - 1) / tiles[i].bn) * heads;
        const double time = tiles[i].alone + tiles[i].more * (double)((blocks + sms - 1) / sms - 1);
        if (i == 0 || time < least) {
            best = i;
            least = time;
        }
    }
    const dim3 grid((N + tiles[best].bn - 1) / tiles[best].bn, (M + tiles[best].bm - 1) / tiles[best].bm, heads);
#define LF_GO(TM, TN) linear_f32_kernel<TM, TN><<<grid, LF_THREADS, 0, stream>>>(x, w, y, M, N, K, vec_ok, ldx, ldy, x_head, w_head, y_head)
    if (best == 0) LF_GO(4, 4);
    else if (best == 1) LF_GO(8, 4);
    else if (best == 2) LF_GO(8, 6);
    else LF_GO(8, 8);
#undef LF_GO
    RI_CHECK_LAUNCH("linear_f32");
    return 0;
}

extern "C" int ri_linear_f32(const float* x, const float* w, float* y, int M, int N, int K, cudaStream_t stream) {
    if (M == 0 || N == 0) return 0;
    RI_REQUIRE(M > 0 && N > 0 && K > 0, "linear_f32: bad sizes M=%d N=%d K=%d", M, N, K);
    RI_REQUIRE((M + 63) / 64 <= 65535, "linear_f32: too many rows (%d)", M);
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
    RI_REQUIRE((M + 63) / 64 <= 65535 && heads <= 65535, "linear_heads_f32: too many rows or heads (%d, %d)", M, heads);
    int vec_ok = (K % 4 == 0) && (ldx % 4 == 0) && (x_head % 4 == 0) && (((uintptr_t)x | (uintptr_t)w) % 16 == 0);
    return lf_launch(x, w, y, M, N, K, heads, vec_ok, ldx, ldy, x_head, (long long)N * K, y_head, stream);
}

// ---- the tensor cores' form ------------------------------------------------------------------------------------------------
typedef CUresult (*lt_encode_tiled_fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                       const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                       CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

template <int CH, int GROUPS, int BUFS>
static int lt_launch(const CUtensorMap& map_w, const CUtensorMap& map_x, const float* x, const float* w, float* y, int M, int N, int K,
                     int tn, int* err, cudaStream_t stream) {
    auto kernel = linear_f32_tc_kernel<CH, GROUPS, BUFS>;
    const int stage = LT_W_BYTES + 3 * 64 * tn;
    int stages = LT_SMEM_MAX / stage, wstages = (512 - (BUFS + 1) * tn) / LT_W_COLS;
    if (stages > LT_MAX_STAGES) stages = LT_MAX_STAGES;
    if (wstages > LT_MAX_WSTAGES) wstages = LT_MAX_WSTAGES;
    // A wait knows a barrier's phases by their parity only, so that whoever waits must know the phase before to be over.  A place of the
    // first ring is always the same group's, which has waited for it there; copies into the place of stage s start when the
    // products up to s - stages are done, so that the second ring's phase before last is over if it has half as many places.
    stages -= stages % GROUPS;
    RI_REQUIRE(tn <= 32 * CH && stages >= GROUPS && wstages >= GROUPS && 2 * wstages >= stages, "linear_f32_tc: %d tokens a block", tn);
    cudaError_t e = cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LT_SMEM_MAX);
    if (e != cudaSuccess) RI_FAIL((int)e, "linear_f32_tc: %s", cudaGetErrorString(e));
    ri_launch_pdl(kernel, dim3((N + LT_ROWS - 1) / LT_ROWS, (M + tn - 1) / tn), dim3(128 * GROUPS + LT_SUMS), (size_t)stages * stage, stream,
                  map_w, map_x, x, w, y, M, N, K, tn, stages, wstages, (long long)K, (long long)N, err);
    RI_CHECK_LAUNCH("linear_f32_tc");
    return 0;
}

// The most tokens a block takes: the largest variant's warps hand registers over, whose sum has to be what they are launched with, so that it
// is left out where the compiler gave it another number.
static int lt_most_tokens() {
    static int most = 0;
    if (!most) {
        cudaFuncAttributes attr;
        cudaError_t e = cudaFuncGetAttributes(&attr, (const void*)linear_f32_tc_kernel<6, 2, 1>);
        if (e != cudaSuccess) RI_FAIL(0, "linear_f32_tc: %s", cudaGetErrorString(e));
        most = attr.numRegs == 128 ? LT_MAX_TOKENS : 128;
    }
    return most;
}

// Tokens a block: the multiple of 16, up to `most`, with the least time, rounds of blocks (one an SM) times what a round takes, some 57 us +
// 0.285 a token at K = 4,096 where the blocks fill the device (16 tokens 55, 128 and 48 blocks 68, 176 and 48 blocks 69, 176 and 144 blocks 112).
extern "C" int ri_linear_f32_tc_tokens(int rows, int N, int sms, int most) {
    int tn = 16;
    double least = 0;
    for (int t = 16; t <= most; t += 16) {
        const long long blocks = (long long)((N + LT_ROWS - 1) / LT_ROWS) * ((rows + t - 1) / t);
        const double time = (double)((blocks + sms - 1) / sms) * (57 + 0.285 * t);
        if (t == 16 || time < least) {
            tn = t;
            least = time;
        }
    }
    return tn;
}

// `parts`: scratch for the cut rows of x, 6 bytes for each of K rounded up to 32 and each of `part_rows` rows; more rows than that are
// taken in several launches.  K a multiple of 4, x and w on 16 bytes.
//
// Cold, with the cut of x, in us at K = 4,096, tensor cores / multiply-adds: 512 tokens and 6,144 outputs 112 / 639,
// 512 and 4,096 87 / 449, 300 and 6,144 85 / 450, 128 and 6,144 68 / 265, 16 and 6,144 55 / 184, 1 and 4,096 53 / 184; K = 2,048, 300 and 4,096 42 / 180;
// K = 512, 300 and 4,096 16 / 47, 1 and 4,096 9.6 / 24.
// 2-norm of the error against float64 over that of the result, normal values: 2.2e-7 / 1.15e-6 at K = 4,096, 9.0e-8 / 4.1e-7 at 512,
// 6.2e-8 / 2.0e-7 at 128; with one entry that is not zero 2.60e-8 / 2.53e-8, two 2.6e-8 / 3.1e-8, four 2.7e-8 / 4.0e-8, 32 4.4e-8 / 1.0e-7; all of
// one sign and size, K = 4,096, 1.2e-7 / 8.6e-7.  With all terms in one sum of 32 k, parts cut towards zero: 1.0e-7 for one entry, 1.1e-7 for four.
extern "C" int ri_linear_f32_tc(const float* x, const float* w, float* y, void* parts, int part_rows, int M, int N, int K, int* err_flag,
                                cudaStream_t stream) {
    if (M == 0 || N == 0) return 0;
    RI_REQUIRE(M > 0 && N > 0 && K > 0 && part_rows > 0, "linear_f32_tc: bad sizes M=%d N=%d K=%d", M, N, K);
    RI_REQUIRE(K % 4 == 0 && (((uintptr_t)x | (uintptr_t)w | (uintptr_t)parts) & 15) == 0, "linear_f32_tc: rows of whole 16-byte pieces are needed");
    static lt_encode_tiled_fn encode = nullptr;
    static int sms = 0;
    if (!sms) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult res;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &res);
        if (e != cudaSuccess || res != cudaDriverEntryPointSuccess || !fn) RI_FAIL(-1, "linear_f32_tc: the driver has no cuTensorMapEncodeTiled");
        encode = (lt_encode_tiled_fn)fn;
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        sms = n > 0 ? n : 148;
    }
    const int most = lt_most_tokens();
    if (!most) return -1;
    const int Kp = (K + LT_K - 1) / LT_K * LT_K;
    const cuuint32_t one[3] = {1, 1, 1};
    CUtensorMap map_w;
    {
        cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)N}, strides[1] = {(cuuint64_t)K * 4};
        cuuint32_t box[2] = {LT_K, LT_ROWS};
        CUresult r = encode(&map_w, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(w), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) RI_FAIL(-1, "linear_f32_tc: cuTensorMapEncodeTiled failed with %d (N=%d, K=%d)", (int)r, N, K);
    }
    for (int at = 0; at < M; at += part_rows) {
        const int rows = M - at < part_rows ? M - at : part_rows;
        const int tn = ri_linear_f32_tc_tokens(rows, N, sms, most);
        RI_REQUIRE((rows + tn - 1) / tn <= 65535, "linear_f32_tc: too many rows (%d)", M);
        CUtensorMap map_x;
        cuuint64_t dims[3] = {(cuuint64_t)Kp, (cuuint64_t)rows, 3}, strides[2] = {(cuuint64_t)Kp * 2, (cuuint64_t)Kp * 2 * rows};
        cuuint32_t box[3] = {LT_K, (cuuint32_t)tn, 3};
        CUresult r = encode(&map_x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, parts, dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) RI_FAIL(-1, "linear_f32_tc: cuTensorMapEncodeTiled failed with %d (M=%d, K=%d)", (int)r, rows, K);
        const float* xs = x + (size_t)at * K;
        float* ys = y + (size_t)at * N;
        const long long pieces = (long long)rows * (Kp / 8);
        RI_REQUIRE((pieces + 255) / 256 < (1ll << 31), "linear_f32_tc: too many rows (%d)", M);
        ri_launch_pdl(linear_f32_cut_kernel, dim3((unsigned)((pieces + 255) / 256)), dim3(256), 0, stream, xs, (uint4*)parts, rows, K, Kp / 8);
        RI_CHECK_LAUNCH("linear_f32_cut");
        int rc;
        if (tn <= 64) rc = lt_launch<2, 4, 4>(map_w, map_x, xs, w, ys, rows, N, K, tn, err_flag, stream);
        else if (tn <= 128) rc = lt_launch<4, 2, 2>(map_w, map_x, xs, w, ys, rows, N, K, tn, err_flag, stream);
        else rc = lt_launch<6, 2, 1>(map_w, map_x, xs, w, ys, rows, N, K, tn, err_flag, stream);
        if (rc) return rc;
    }
    return 0;
}
