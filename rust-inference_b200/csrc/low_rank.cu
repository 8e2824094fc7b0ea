// The outer products of low-rank projections, up to two of them in one launch:
//     y_i[t, :] = W_i x[t, col_i .. col_i + K_i - 1]        W_i [N_i, K_i], K_i up to 128 (multiples of 8), bfloat16, float32 sums
// x is the stacked projection that holds the inner parts as columns (rows ldx apart): no copy of them is made.
// What bounds it: for a step's few tokens the launch and one trip to memory, for a prompt writing y.  A block takes MT tokens and 64
// outputs, all K at once (mma.sync m16n8k16), in the order in which `ops.linear` would add them up, whose bits these are.  W's tile, which no
// kernel of the step writes, is on its way before the kernel in front is done.
// Two products of 64 to 2,048 columns, us: 2,048 tokens 11 (two copies, two library products and their gaps 23), 8 tokens 1.6 behind the
// product in front (two copies and two weight-streaming products 10).
#include "common.cuh"
#include "mma_helpers.cuh"

#define LR_COLS 64
#define LR_MAX_K 128
#define LR_PITCH (LR_MAX_K + 8)

struct LrSet {
    const bf16* w;
    bf16* y;
    int col, K, N;
    int streamed;                                  // (up to 16 tokens) the sums' order is the weight-streaming product's
};

template <int MT>
__global__ void __launch_bounds__(128)
low_rank_kernel(const bf16* __restrict__ x, long long ldx, int tokens, LrSet first, LrSet second) {
    __shared__ __align__(16) bf16 ws[LR_COLS][LR_PITCH];
    __shared__ __align__(16) bf16 xs[MT][LR_PITCH];
    const LrSet p = blockIdx.z == 0 ? first : second;
    const int n0 = blockIdx.x * LR_COLS, t0 = blockIdx.y * MT;
    pdl_trigger();
    if (n0 >= p.N) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int K32 = (p.K + 31) & ~31, pieces = K32 / 8;
    for (int i = tid; i < LR_COLS * pieces; i += 128) {
        const int n = i / pieces, k = (i - n * pieces) * 8;
        const bool there = n0 + n < p.N && k < p.K;
        cp_async16(&ws[n][k], there ? p.w + (size_t)(n0 + n) * p.K + k : p.w, there);
    }
    pdl_wait();
    for (int i = tid; i < MT * pieces; i += 128) {
        const int m = i / pieces, k = (i - m * pieces) * 8;
        const bool there = t0 + m < tokens && k < p.K;
        cp_async16(&xs[m][k], there ? x + (size_t)(t0 + m) * ldx + p.col + k : x, there);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    // a warp has 16 tokens and all 64 outputs (MT 64), or 16 outputs of the block's 16 tokens
    constexpr int NT = MT == 64 ? 8 : 2;
    const int m0 = MT == 64 ? warp * 16 : 0, c0 = MT == 64 ? 0 : warp * 16;
    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; n++)
#pragma unroll
        for (int i = 0; i < 4; i++) acc[n][i] = 0.0f;
    const bool streamed = MT == 16 && p.streamed;
    if (streamed) {
        // As linear_skinny.cu: W is the product's first operand, and of every 32 k a thread's eight neighbouring ones go four to the first
        // mma.sync and four to the second.  acc[n]: outputs rho, rho + 8 of the warp's 16, tokens 8 n + 2 (lane & 3), + 1
        const int quad = lane >> 2, qc = lane & 3, rho = (quad >> 1) | ((quad & 1) << 2);
        for (int k = qc * 8; k < K32; k += 32) {
            const uint4 a = *reinterpret_cast<const uint4*>(&ws[c0 + rho][k]), b = *reinterpret_cast<const uint4*>(&ws[c0 + rho + 8][k]);
#pragma unroll
            for (int n = 0; n < 2; n++) {
                const uint4 v = *reinterpret_cast<const uint4*>(&xs[n * 8 + quad][k]);
                mma_bf16(acc[n], a.x, b.x, a.y, b.y, v.x, v.y);
                mma_bf16(acc[n], a.z, b.z, a.w, b.w, v.z, v.w);
            }
        }
    } else {
        for (int k = 0; k < K32; k += 16) {
            unsigned a0, a1, a2, a3;
            ldmatrix_x4(a0, a1, a2, a3, &xs[m0 + (lane & 15)][k + (lane >> 4) * 8]);
#pragma unroll
            for (int n = 0; n < NT; n += 2) {
                unsigned b0, b1, b2, b3;
                ldmatrix_x4(b0, b1, b2, b3, &ws[c0 + n * 8 + (lane & 7) + (lane >> 4) * 8][k + ((lane >> 3) & 1) * 8]);
                mma_bf16(acc[n], a0, a1, a2, a3, b0, b1);
                mma_bf16(acc[n + 1], a0, a1, a2, a3, b2, b3);
            }
        }
    }
    __syncthreads();                               // the tiles have been read: x's place takes the results
    bf16(*ys)[LR_COLS + 8] = reinterpret_cast<bf16(*)[LR_COLS + 8]>(&xs[0][0]);
    static_assert(LR_COLS + 8 <= LR_PITCH, "the results fit");
    if (streamed) {
        const int quad = lane >> 2, rho = (quad >> 1) | ((quad & 1) << 2);
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
            for (int i = 0; i < 4; i++) ys[n * 8 + (lane & 3) * 2 + (i & 1)][c0 + rho + (i >> 1) * 8] = __float2bfloat16(acc[n][i]);
    } else
#pragma unroll
    for (int n = 0; n < NT; n++)
#pragma unroll
        for (int h = 0; h < 2; h++)
            *reinterpret_cast<unsigned*>(&ys[m0 + (lane >> 2) + 8 * h][c0 + n * 8 + (lane & 3) * 2]) = pack_bf16(acc[n][2 * h], acc[n][2 * h + 1]);
    __syncthreads();
    for (int i = tid; i < MT * (LR_COLS / 8); i += 128) {
        const int m = i / (LR_COLS / 8), c = (i % (LR_COLS / 8)) * 8;
        if (t0 + m < tokens && n0 + c < p.N) *reinterpret_cast<uint4*>(p.y + (size_t)(t0 + m) * p.N + n0 + c) = *reinterpret_cast<const uint4*>(&ys[m][c]);
    }
}

// x [tokens, ldx], w_i [N_i, K_i], y_i [tokens, N_i] bfloat16; N_1 = 0: one product.  streamed_i: up to 16 tokens whose sums take the order
// of ri_linear_skinny
extern "C" int ri_low_rank(const void* x, long long ldx, int tokens, int col0, int K0, const void* w0, void* y0, int N0, int streamed0,
                           int col1, int K1, const void* w1, void* y1, int N1, int streamed1, cudaStream_t stream) {
    if (tokens == 0) return 0;
    RI_REQUIRE(tokens > 0 && N0 > 0 && N1 >= 0 && K0 > 0 && K0 <= LR_MAX_K && (N1 == 0 || (K1 > 0 && K1 <= LR_MAX_K)), "low_rank: bad sizes");
    RI_REQUIRE(ldx % 8 == 0 && col0 % 8 == 0 && K0 % 8 == 0 && N0 % 8 == 0 && (N1 == 0 || (col1 % 8 == 0 && K1 % 8 == 0 && N1 % 8 == 0)) &&
                   (((uintptr_t)x | (uintptr_t)w0 | (uintptr_t)y0 | (uintptr_t)w1 | (uintptr_t)y1) & 15) == 0,
               "low_rank: rows of whole 16-byte pieces are needed");
    RI_REQUIRE(tokens <= 16 || !(streamed0 || streamed1), "low_rank: %d tokens in the order of the weight-streaming product", tokens);
    const LrSet a{(const bf16*)w0, (bf16*)y0, col0, K0, N0, streamed0}, b{(const bf16*)w1, (bf16*)y1, col1, K1, N1, streamed1};
    const int most = N0 > N1 ? N0 : N1;
    if (tokens <= 64) {
        const dim3 grid((most + LR_COLS - 1) / LR_COLS, (tokens + 15) / 16, N1 ? 2 : 1);
        ri_launch_pdl(low_rank_kernel<16>, grid, dim3(128), 0, stream, (const bf16*)x, ldx, tokens, a, b);
    } else {
        RI_REQUIRE((tokens + 63) / 64 <= 65535, "low_rank: too many tokens (%d)", tokens);
        const dim3 grid((most + LR_COLS - 1) / LR_COLS, (tokens + 63) / 64, N1 ? 2 : 1);
        ri_launch_pdl(low_rank_kernel<64>, grid, dim3(128), 0, stream, (const bf16*)x, ldx, tokens, a, b);
    }
    RI_CHECK_LAUNCH("low_rank");
    return 0;
}
