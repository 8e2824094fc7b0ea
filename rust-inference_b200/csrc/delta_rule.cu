// The gated delta rule: a recurrent mixer with a matrix-valued state per (sequence, head), and the short causal
// convolution in front of it.
//
// `short_conv`: per channel c a convolution over time with `taps` weights w[c, 0 .. taps-1] (the last one is the
// current token's), zeros before a sequence's start, then silu:
//     y_t[c] = silu( sum_j w[c, j] x_(t - (taps-1-j))[c] )                    float32, j ascending
// The inputs of a sequence's last taps-1 tokens are its state ([slots, taps-1, C] float32, oldest first), so a prompt,
// its pieces and single tokens give the same bits.  x is a block of columns of a projection (compute type T).
//
// `delta_rule_recurrent`: per head h with q/k head h / (H / G), for every new token in order
//     qn = q / sqrt(sum q^2 + 1e-6) * qscale,   kn = k / sqrt(sum k^2 + 1e-6)
//     g[d] = exp(-exp(A_log[h]) * softplus(z[h, d] + dt_bias[h, d]))          decay of key channel d
//            (or one decay per head, g = exp(-exp(A_log[h]) * softplus(z[h] + dt_bias[h])), for all its channels)
//     beta = sigmoid(b[h])
//     S[d, j] <- g[d] S[d, j];   u[j] = beta (v[j] - sum_d S[d, j] kn[d]);   S[d, j] <- S[d, j] + kn[d] u[j]
//     o[j] = sum_d S[d, j] qn[d]                                              (reads the current token's write)
//          = sum_d (g[d] S_old[d, j]) qn[d] + u[j] (kn . qn)                   (the form the kernel computes)
// all in float32; S [dim, vdim] lives in the sequence's slot of `state` [slots, H, dim, vdim].
// What does not depend on the token before (unit vectors, decays, beta) is computed for all tokens at once by a kernel
// of its own; the recurrence kernels only walk the tokens.  There a block owns some value columns of one (sequence, head), and
// the key channels of a column are spread over 4 to 32 neighbouring lanes' registers (single tokens: over a block's warps).  Every
// sum over d has one order that depends on the head's size only, so the result does not depend on how a sequence's tokens
// were cut into steps.
#include "common.cuh"

__device__ __forceinline__ float dr_silu(float z) { return z / (1.0f + expf(-z)); }
__device__ __forceinline__ float dr_softplus(float z) { return fmaxf(z, 0.0f) + log1pf(expf(-fabsf(z))); }

template <typename T>
__global__ void __launch_bounds__(256)
short_conv_kernel(const T* __restrict__ x, long long ld, int col0, const float* __restrict__ w, float* __restrict__ y,
                  float* __restrict__ state, const int* __restrict__ tok_seq, const int* __restrict__ seq_slot,
                  const int* __restrict__ seq_start, int tokens, int C, int taps, int update) {
    pdl_trigger();
    pdl_wait();
    const int c = blockIdx.y * blockDim.x + threadIdx.x;
    const int t = blockIdx.x;
    if (c >= C) return;
    const int b = tok_seq[t];
    const int t0 = seq_start[b];
    const int slot = seq_slot[b];
    float* st = state + (size_t)slot * (taps - 1) * C + c;
    float acc = 0.0f;
    for (int j = 0; j < taps; j++) {
        const int r = (t - t0) - (taps - 1 - j);                 // index among the step's tokens of this sequence
        const float v = r >= 0 ? ld_f(x + (size_t)(t0 + r) * ld + col0 + c) : st[(size_t)(taps - 1 + r) * C];
        acc = fmaf(w[(size_t)c * taps + j], v, acc);
    }
    y[(size_t)t * C + c] = dr_silu(acc);
    if (update) {                                                // one token per sequence: this thread alone owns st
        for (int j = 0; j + 1 < taps - 1; j++) st[(size_t)j * C] = st[(size_t)(j + 1) * C];
        if (taps > 1) st[(size_t)(taps - 2) * C] = ld_f(x + (size_t)t * ld + col0 + c);
    }
}

// bfloat16 inputs, eight neighbouring channels per thread (16-byte loads of the inputs, of the weights in their
// transposed copy wt [taps, C], of the state; two 16-byte stores): an element's arithmetic and its order are the scalar
// kernel's.  For C, ld and col0 multiples of 8 and 16-byte aligned bases.
__global__ void __launch_bounds__(128)
short_conv_x8_kernel(const __nv_bfloat16* __restrict__ x, long long ld, int col0, const float* __restrict__ wt,
                     float* __restrict__ y, float* __restrict__ state, const int* __restrict__ tok_seq,
                     const int* __restrict__ seq_slot, const int* __restrict__ seq_start, int C, int taps, int update) {
    pdl_trigger();
    pdl_wait();
    const int c = (blockIdx.y * blockDim.x + threadIdx.x) * 8;
    const int t = blockIdx.x;
    if (c >= C) return;
    const int b = tok_seq[t];
    const int t0 = seq_start[b];
    float* st = state + (size_t)seq_slot[b] * (taps - 1) * C + c;
    float acc[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    float cur[8];
    for (int j = 0; j < taps; j++) {
        const int r = (t - t0) - (taps - 1 - j);
        float v[8];
        if (r >= 0) {
            const uint4 raw = *reinterpret_cast<const uint4*>(x + (size_t)(t0 + r) * ld + col0 + c);
            const unsigned u[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
            for (int e = 0; e < 4; e++) {
                v[2 * e] = __uint_as_float(u[e] << 16);
                v[2 * e + 1] = __uint_as_float(u[e] & 0xffff0000u);
            }
        } else {
            const float4 a = *reinterpret_cast<const float4*>(st + (size_t)(taps - 1 + r) * C);
            const float4 bq = *reinterpret_cast<const float4*>(st + (size_t)(taps - 1 + r) * C + 4);
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = bq.x; v[5] = bq.y; v[6] = bq.z; v[7] = bq.w;
        }
        const float4 w0 = *reinterpret_cast<const float4*>(wt + (size_t)j * C + c);
        const float4 w1 = *reinterpret_cast<const float4*>(wt + (size_t)j * C + c + 4);
        const float wv[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
        for (int e = 0; e < 8; e++) {
            acc[e] = fmaf(wv[e], v[e], acc[e]);
            cur[e] = v[e];                                        // after the last tap: the current token's inputs
        }
    }
    float o[8];
#pragma unroll
    for (int e = 0; e < 8; e++) o[e] = dr_silu(acc[e]);
    *reinterpret_cast<float4*>(y + (size_t)t * C + c) = make_float4(o[0], o[1], o[2], o[3]);
    *reinterpret_cast<float4*>(y + (size_t)t * C + c + 4) = make_float4(o[4], o[5], o[6], o[7]);
    if (update && taps > 1) {
        for (int j = 0; j + 1 < taps - 1; j++) {
            *reinterpret_cast<float4*>(st + (size_t)j * C) = *reinterpret_cast<const float4*>(st + (size_t)(j + 1) * C);
            *reinterpret_cast<float4*>(st + (size_t)j * C + 4) = *reinterpret_cast<const float4*>(st + (size_t)(j + 1) * C + 4);
        }
        *reinterpret_cast<float4*>(st + (size_t)(taps - 2) * C) = make_float4(cur[0], cur[1], cur[2], cur[3]);
        *reinterpret_cast<float4*>(st + (size_t)(taps - 2) * C + 4) = make_float4(cur[4], cur[5], cur[6], cur[7]);
    }
}

// The same with CONV_TOKENS neighbouring tokens per thread, for prompts with four taps: the weights and the tokens before are read once for
// all of them, and the tokens' loads are on their way together.  What bounds it: the functions of silu, and memory.  2,048 tokens of 4,096 channels (50 MB): 19 us,
// 20 to 22 with a token per thread, whose weights come from L2 again for every token (134 MB), and with eight.  An element's arithmetic and its order are the same.
// From CONV_MANY elements on: below it the blocks are too few (us, this / a token per thread: 1,000 tokens of 256 channels 5.4 / 4.6, 320 of 4,096 7.2 / 6.3)
// or take a second round for a few (2.5 million elements 9.6 / 8.9); 3.3 million 10.5 / 11.0, 6.1 million 15.2 / 16.3, 24 million 53 / 62.
#define CONV_MANY (3 << 20)
#define CONV_TOKENS 4
__global__ void __launch_bounds__(128)
short_conv_x8_many_kernel(const __nv_bfloat16* __restrict__ x, long long ld, int col0, const float* __restrict__ wt, float* __restrict__ y,
                          const float* __restrict__ state, const int* __restrict__ tok_seq, const int* __restrict__ seq_slot,
                          const int* __restrict__ seq_start, int tokens, int C) {
    constexpr int TAPS = 4;
    pdl_trigger();
    const int c = (blockIdx.y * blockDim.x + threadIdx.x) * 8, first = blockIdx.x * CONV_TOKENS;
    if (c >= C) return;
    float w[TAPS][8];
#pragma unroll
    for (int j = 0; j < TAPS; j++) {
        *reinterpret_cast<float4*>(&w[j][0]) = *reinterpret_cast<const float4*>(wt + (size_t)j * C + c);
        *reinterpret_cast<float4*>(&w[j][4]) = *reinterpret_cast<const float4*>(wt + (size_t)j * C + c + 4);
    }
    int seq[CONV_TOKENS], nth[CONV_TOKENS];                      // each token's sequence, and its place among the step's tokens of it
#pragma unroll
    for (int i = 0; i < CONV_TOKENS; i++) seq[i] = tok_seq[min(first + i, tokens - 1)];
#pragma unroll
    for (int i = 0; i < CONV_TOKENS; i++) nth[i] = min(first + i, tokens - 1) - seq_start[seq[i]];
    pdl_wait();
    uint4 raw[CONV_TOKENS + TAPS - 1];
#pragma unroll
    for (int i = 0; i < CONV_TOKENS + TAPS - 1; i++)
        raw[i] = *reinterpret_cast<const uint4*>(x + (size_t)min(max(first + i - (TAPS - 1), 0), tokens - 1) * ld + col0 + c);
#pragma unroll
    for (int i = 0; i < CONV_TOKENS; i++) {
        if (first + i >= tokens) break;
        float acc[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int j = 0; j < TAPS; j++) {
            const int r = nth[i] - (TAPS - 1 - j);
            float v[8];
            const unsigned u[4] = {raw[i + j].x, raw[i + j].y, raw[i + j].z, raw[i + j].w};
#pragma unroll
            for (int e = 0; e < 4; e++) {
                v[2 * e] = __uint_as_float(u[e] << 16);
                v[2 * e + 1] = __uint_as_float(u[e] & 0xffff0000u);
            }
            if (r < 0) {                                         // before the step's tokens of the sequence: from its state
                const float* st = state + ((size_t)seq_slot[seq[i]] * (TAPS - 1) + (TAPS - 1 + r)) * C + c;
                *reinterpret_cast<float4*>(&v[0]) = *reinterpret_cast<const float4*>(st);
                *reinterpret_cast<float4*>(&v[4]) = *reinterpret_cast<const float4*>(st + 4);
            }
#pragma unroll
            for (int e = 0; e < 8; e++) acc[e] = fmaf(w[j][e], v[e], acc[e]);
        }
        float* to = y + (size_t)(first + i) * C + c;
        *reinterpret_cast<float4*>(to) = make_float4(dr_silu(acc[0]), dr_silu(acc[1]), dr_silu(acc[2]), dr_silu(acc[3]));
        *reinterpret_cast<float4*>(to + 4) = make_float4(dr_silu(acc[4]), dr_silu(acc[5]), dr_silu(acc[6]), dr_silu(acc[7]));
    }
}

template <typename T>
__global__ void __launch_bounds__(256)
short_conv_state_kernel(const T* __restrict__ x, long long ld, int col0, float* __restrict__ state,
                        const int* __restrict__ seq_slot, const int* __restrict__ seq_start, int C, int taps) {
    pdl_trigger();
    pdl_wait();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int b = blockIdx.y;
    if (c >= C) return;
    const int t0 = seq_start[b], n = seq_start[b + 1] - t0;
    float* st = state + (size_t)seq_slot[b] * (taps - 1) * C + c;
    for (int j = 0; j < taps - 1; j++) {                         // ascending: an old entry is read before it is overwritten
        const int r = n - (taps - 1) + j;
        st[(size_t)j * C] = r >= 0 ? ld_f(x + (size_t)(t0 + r) * ld + col0 + c) : st[(size_t)(j + n) * C];
    }
}

// wt: the weights once more as [taps, C] (may be null: then the scalar kernel runs)
extern "C" int ri_short_conv(const void* x, long long ld, int col0, const float* w, const float* wt, float* y, float* state,
                             const int* tok_seq, const int* seq_slot, const int* seq_start, int tokens, int seqs, int C,
                             int taps, int single, int dtype, cudaStream_t stream) {
    if (tokens == 0) return 0;
    RI_REQUIRE(tokens > 0 && seqs > 0 && C > 0 && taps >= 1, "short_conv: bad sizes");
    RI_REQUIRE(seqs <= 65535 && C <= 65535 * 256, "short_conv: too many sequences or channels for one launch");
    RI_REQUIRE(dtype == RI_DTYPE_F32 || dtype == RI_DTYPE_BF16, "short_conv: unknown dtype %d", dtype);
    const int upd = single && tokens == seqs ? 1 : 0;
    const dim3 grid(tokens, (C + 255) / 256);
    const bool x8 = dtype == RI_DTYPE_BF16 && wt && C % 8 == 0 && ld % 8 == 0 && col0 % 8 == 0 &&
                    (((uintptr_t)x | (uintptr_t)wt | (uintptr_t)y | (uintptr_t)state) & 15) == 0;
    if (x8 && taps == 4 && !upd && (long long)tokens * C >= CONV_MANY)
        ri_launch_pdl(short_conv_x8_many_kernel, dim3((tokens + CONV_TOKENS - 1) / CONV_TOKENS, (C / 8 + 127) / 128), dim3(128), 0, stream,
                      (const __nv_bfloat16*)x, ld, col0, wt, y, (const float*)state, tok_seq, seq_slot, seq_start, tokens, C);
    else if (x8)
        ri_launch_pdl(short_conv_x8_kernel, dim3(tokens, (C / 8 + 127) / 128), dim3(128), 0, stream, (const __nv_bfloat16*)x, ld,
                      col0, wt, y, state, tok_seq, seq_slot, seq_start, C, taps, upd);
    else if (dtype == RI_DTYPE_F32)
        ri_launch_pdl(short_conv_kernel<float>, grid, dim3(256), 0, stream, (const float*)x, ld, col0, w, y, state, tok_seq,
                      seq_slot, seq_start, tokens, C, taps, upd);
    else
        ri_launch_pdl(short_conv_kernel<__nv_bfloat16>, grid, dim3(256), 0, stream, (const __nv_bfloat16*)x, ld, col0, w, y,
                      state, tok_seq, seq_slot, seq_start, tokens, C, taps, upd);
    RI_CHECK_LAUNCH("short_conv");
    if (!upd && taps > 1) {
        const dim3 g2((C + 255) / 256, seqs);
        if (dtype == RI_DTYPE_F32)
            ri_launch_pdl(short_conv_state_kernel<float>, g2, dim3(256), 0, stream, (const float*)x, ld, col0, state, seq_slot,
                          seq_start, C, taps);
        else
            ri_launch_pdl(short_conv_state_kernel<__nv_bfloat16>, g2, dim3(256), 0, stream, (const __nv_bfloat16*)x, ld, col0,
                          state, seq_slot, seq_start, C, taps);
        RI_CHECK_LAUNCH("short_conv_state");
    }
    return 0;
}

// ---- what the recurrence reads, made ready for all tokens at once ------------------------------------------------------
// One block per token: q and k of every q/k head become unit vectors in place (q also times qscale), the decays
// g[h, d] = exp(-exp(A_log[h]) softplus(z[h, d] + dt_bias[h, d])) with d < ddim (ddim = dim, or 1: one decay per head),
// beta[h] = sigmoid(b[h]) and the products k . q of the unit vectors are written as float32 (`beta` [tokens, H + G]: the
// betas, then the products).  Row t of z starts ldz elements after row t - 1.
template <typename T>
__global__ void __launch_bounds__(128)
delta_prep_kernel(float* __restrict__ qkv, int C, int q_col, int k_col, const T* __restrict__ proj, long long ld, int b_col,
                  const T* __restrict__ z, long long ldz, const float* __restrict__ dt_bias, const float* __restrict__ a_log,
                  float qscale, float* __restrict__ decay, float* __restrict__ beta, int H, int G, int dim, int ddim) {
    pdl_trigger();
    pdl_wait();
    const int t = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* row = qkv + (size_t)t * C;
    // (a token's work is spread over gridDim.y blocks when the step has few tokens)
    for (int g = blockIdx.y * 4 + warp; g < G; g += 4 * gridDim.y) {      // a warp per q/k head: both unit vectors and their product
        float* q = row + q_col + g * dim;
        float* k = row + k_col + g * dim;
        float sq = 0.0f, sk = 0.0f, qk = 0.0f;
        for (int d = lane; d < dim; d += 32) {
            sq = fmaf(q[d], q[d], sq);
            sk = fmaf(k[d], k[d], sk);
            qk = fmaf(q[d], k[d], qk);
        }
        const float iq = qscale / sqrtf(warp_sum(sq) + 1e-6f), ik = 1.0f / sqrtf(warp_sum(sk) + 1e-6f);
        qk = warp_sum(qk);
        for (int d = lane; d < dim; d += 32) {
            q[d] *= iq;
            k[d] *= ik;
        }
        if (lane == 0) beta[(size_t)t * (H + G) + H + g] = qk * iq * ik;
    }
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < H * ddim; i += blockDim.x * gridDim.y) {
        const float rate = expf(a_log[i / ddim]);
        decay[(size_t)t * H * ddim + i] = expf(-rate * dr_softplus(ld_f(z + (size_t)t * ldz + i) + dt_bias[i]));
    }
    for (int h = blockIdx.y * blockDim.x + threadIdx.x; h < H; h += blockDim.x * gridDim.y)
        beta[(size_t)t * (H + G) + h] = 1.0f / (1.0f + expf(-ld_f(proj + (size_t)t * ld + b_col + h)));
}

// The same, bit for bit, for heads of whole groups of four channels (up to 128 PIECES of them): a lane's channels of q and k are asked for
// together, a thread has four neighbouring decays, whose rate is taken once.  What bounds it: memory and, beside it, the functions of the decays.  2,048
// tokens, 8 q/k heads and 16 heads of 128 (73 MB), behind the convolution: 14 us, 28 a channel at a time.
__device__ __forceinline__ float4 dr_ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 dr_ld4(const __nv_bfloat16* p) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
}
template <typename T, int PIECES>
__global__ void __launch_bounds__(256)
delta_prep_vec_kernel(float* __restrict__ qkv, int C, int q_col, int k_col, const T* __restrict__ proj, long long ld, int b_col,
                      const T* __restrict__ z, long long ldz, const float* __restrict__ dt_bias, const float* __restrict__ a_log,
                      float qscale, float* __restrict__ decay, float* __restrict__ beta, int H, int G, int dim) {
    pdl_trigger();
    pdl_wait();
    const int t = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* row = qkv + (size_t)t * C;
    for (int g = blockIdx.y * 8 + warp; g < G; g += 8 * gridDim.y) {      // a warp per q/k head: both unit vectors and their product
        float* q = row + q_col + g * dim;
        float* k = row + k_col + g * dim;
        float a[4 * PIECES], b[4 * PIECES];                     // channels lane, lane + 32, ..: a lane's sums go over them in that order
#pragma unroll
        for (int p = 0; p < 4 * PIECES; p++) {
            const int d = p * 32 + lane;
            a[p] = d < dim ? q[d] : 0.0f;
            b[p] = d < dim ? k[d] : 0.0f;
        }
        float sq = 0.0f, sk = 0.0f, qk = 0.0f;
#pragma unroll
        for (int p = 0; p < 4 * PIECES; p++) {
            sq = fmaf(a[p], a[p], sq);
            sk = fmaf(b[p], b[p], sk);
            qk = fmaf(a[p], b[p], qk);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            sq += __shfl_xor_sync(0xffffffffu, sq, o);
            sk += __shfl_xor_sync(0xffffffffu, sk, o);
            qk += __shfl_xor_sync(0xffffffffu, qk, o);
        }
        const float iq = qscale / sqrtf(sq + 1e-6f), ik = 1.0f / sqrtf(sk + 1e-6f);
#pragma unroll
        for (int p = 0; p < 4 * PIECES; p++) {
            const int d = p * 32 + lane;
            if (d < dim) {
                q[d] = a[p] * iq;
                k[d] = b[p] * ik;
            }
        }
        if (lane == 0) beta[(size_t)t * (H + G) + H + g] = qk * iq * ik;
    }
    for (int i = 4 * (blockIdx.y * blockDim.x + threadIdx.x); i < H * dim; i += 4 * blockDim.x * gridDim.y) {
        const float4 zz = dr_ld4(z + (size_t)t * ldz + i), bias = dr_ld4(dt_bias + i);
        const float rate = expf(a_log[i / dim]);
        *reinterpret_cast<float4*>(decay + (size_t)t * H * dim + i) =
            make_float4(expf(-rate * dr_softplus(zz.x + bias.x)), expf(-rate * dr_softplus(zz.y + bias.y)),
                        expf(-rate * dr_softplus(zz.z + bias.z)), expf(-rate * dr_softplus(zz.w + bias.w)));
    }
    for (int h = blockIdx.y * blockDim.x + threadIdx.x; h < H; h += blockDim.x * gridDim.y)
        beta[(size_t)t * (H + G) + h] = 1.0f / (1.0f + expf(-ld_f(proj + (size_t)t * ld + b_col + h)));
}

// ---- the recurrence -------------------------------------------------------------------------------------------------
#define DR_CT 128               // computing threads
// buffers of staged tokens and how many of them are being filled, for ST staging threads (128; 64 or 32 where many blocks wait)
#define DR_RING(ST) ((ST) == 128 ? 6 : 4)
#define DR_AHEAD(ST) ((ST) == 128 ? 4 : 3)

// two float32 multiply-adds (products) per instruction, each rounded as fmaf (a product) rounds it
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 dr_fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 dr_mul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 dr_pack2(float x, float y) {
    f32x2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
    return d;
}
__device__ __forceinline__ void dr_unpack2(f32x2 v, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v)); }
__device__ __forceinline__ float dr_sum2(f32x2 v) {
    float x, y;
    dr_unpack2(v, x, y);
    return x + y;
}

// BYTES from global to shared memory without a register in between; `valid` false: zeros, nothing is read
template <int BYTES>
__device__ __forceinline__ void dr_copy(void* dst, const void* src, bool valid) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(valid ? 16 : 0) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d), "l"(src), "r"(valid ? 4 : 0) : "memory");
}

// Barriers between the computing and the staging warps of a block: `arrive` goes on, `sync` waits for everybody
__device__ __forceinline__ void dr_bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void dr_bar_arrive(int id, int threads) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// SPLIT: neighbouring lanes that share COLS (one or two) neighbouring value columns (a block owns COLS DR_CT / SPLIT columns); R:
// key channels per lane (dim <= SPLIT R; lane `part` has channels 4 SPLIT i + 4 part .. + 3, so that the lanes of a column
// read neighbouring 16-byte pieces of a staged vector); GROUP: tokens staged at a time.
// What bounds it: the chain from token to token, S' = g S, p = S'^T k, u = beta (v - p), S = S' + k u^T (a multiply-add takes six
// cycles, a shuffle 24), and beside it reading a token's vectors from shared memory, 32 words a cycle for an SM whether the
// lanes of a warp want the same words or not.  The read-out after the write, o = S^T q, is taken as S'^T q + u (k . q): both sums
// run over the same S' side by side (their shuffles travel together), and the next token's vectors are in registers before
// this token's sums are taken.  With two columns the first shuffle of a sum leaves the even lanes with the first column and the
// odd ones with the second, and one more brings the other's u.  A sum over d is taken in four partial sums per lane (two pairs
// of channels by turns), then over the lanes, neighbours first: the same bits with one column per lane as with two.
// Four more warps of the block copy the tokens into a ring of buffers, several groups on their way together, and write
// the outputs of the groups that have been computed, so that neither a group's trip to memory nor its outputs stand
// between the tokens (with one group's loads in registers every group took a trip to memory, 2.5 us).
// SCALAR (one decay per head): the sums run over the undecayed state and are multiplied by the decay afterwards,
// S'^T k = g (S^T k); only its one number per token is staged.
// 2,048 tokens with the preparation: 16 heads of 128 x 128 744 -> 435 us, 8 heads 592 -> 395 us, 8 of 64 x 64 453 -> 335 us, 16 of 128 x
// 128 with one decay per head 586 -> 455 us; four sequences of 512 tokens and 16 heads 503 -> 314 us.  (Before: 16 lanes a column,
// one multiply-add an instruction, the tokens staged by the warps that compute.)  What is left is some 370 cycles a token: the
// chain of about 210 and the instructions that do not fit beside it, one warp to a scheduler.
template <int R, int SPLIT, int COLS, int GROUP, bool SCALAR, bool VEC, int ST>
__global__ void __launch_bounds__(DR_CT + ST)
delta_rule_kernel(const float* qkv, int C, int q_col, int k_col, int v_col, const float* decay, const float* beta, float* state,
                  float* __restrict__ o, const int* __restrict__ seq_slot, const int* __restrict__ seq_start, int H, int G, int dim,
                  int vdim) {
    constexpr int DIMC = R * SPLIT;
    constexpr int BCOLS = COLS * DR_CT / SPLIT;
    constexpr int RING = DR_RING(ST), FILL = DR_AHEAD(ST);
    constexpr int KP = DIMC / 4;                                           // staged pieces of four channels per token
    constexpr int PER = (GROUP * KP + ST - 1) / ST;                  // ... and per thread
    constexpr int VPER = (GROUP * BCOLS + ST - 1) / ST;
    constexpr int VECS = SCALAR ? 2 : 3;                                   // k, q, and the decays g
    constexpr bool AHEAD = R <= 16;                                        // the next token's vectors in registers
    constexpr int ALL = DR_CT + ST;
    extern __shared__ __align__(16) float dr_dyn[];
    float (*s_x)[GROUP][VECS][DIMC] = reinterpret_cast<float (*)[GROUP][VECS][DIMC]>(dr_dyn);                             // [RING]
    float (*s_c)[GROUP][4] = reinterpret_cast<float (*)[GROUP][4]>(dr_dyn + RING * GROUP * VECS * DIMC);                  // beta, k . q, the decay (SCALAR)
    float (*s_v)[GROUP][BCOLS] = reinterpret_cast<float (*)[GROUP][BCOLS]>(dr_dyn + RING * GROUP * (VECS * DIMC + 4));
    float (*s_o)[GROUP][BCOLS] = reinterpret_cast<float (*)[GROUP][BCOLS]>(dr_dyn + RING * GROUP * (VECS * DIMC + 4 + BCOLS));
    static_assert(3 * GROUP <= ST, "a thread per staged beta, product and decay");
    // (the kernel after this one is let in only when the walk is over, see below)
    const int b = blockIdx.z, h = blockIdx.y, j0 = blockIdx.x * BCOLS;
    const int kvh = h / (H / G);
    pdl_wait();
    const int t0 = seq_start[b], t1 = seq_start[b + 1];
    if (t0 >= t1) return;                     // a sequence without tokens keeps its state (the whole block leaves)
    const int st_id = threadIdx.x - DR_CT;                                 // among the staging threads
    // Copies of a group of tokens into its buffer (VEC: 16 bytes, else words): past the sequence's tokens and the columns
    // something that exists is copied and not used, past the head's channels zeros are written (the state is zero there).
    auto copy = [&](int buf, int base) {
#pragma unroll
        for (int e = 0; e < PER; e++) {
            const int idx = st_id + e * ST;
            const int g = idx / KP, d = (idx % KP) * 4, t = min(base + g, t1 - 1);
            if (g < GROUP) {
                const float* src[3] = {qkv + (size_t)t * C + k_col + kvh * dim + d, qkv + (size_t)t * C + q_col + kvh * dim + d,
                                       decay + (SCALAR ? 0 : ((size_t)t * H + h) * dim + d)};
#pragma unroll
                for (int w = 0; w < VECS; w++) {
                    if (VEC) {
                        dr_copy<16>(&s_x[buf][g][w][d], d < dim ? src[w] : qkv, d < dim);
                    } else {
#pragma unroll
                        for (int i = 0; i < 4; i++) dr_copy<4>(&s_x[buf][g][w][d + i], d + i < dim ? src[w] + i : qkv, d + i < dim);
                    }
                }
            }
        }
#pragma unroll
        for (int e = 0; e < VPER; e++) {
            const int idx = st_id + e * ST;
            if (idx < GROUP * BCOLS)
                dr_copy<4>(&(&s_v[buf][0][0])[idx], qkv + (size_t)min(base + idx / BCOLS, t1 - 1) * C + v_col + h * vdim + min(j0 + idx % BCOLS, vdim - 1), true);
        }
        if (st_id < (SCALAR ? 3 : 2) * GROUP) {      // betas, products k . q, decays
            const int g = st_id % GROUP, which = st_id / GROUP, t = min(base + g, t1 - 1);
            dr_copy<4>(&s_c[buf][g][which], which < 2 ? beta + (size_t)t * (H + G) + (which == 0 ? h : H + kvh) : decay + (size_t)t * H + h, true);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    if (threadIdx.x >= DR_CT) {
        // ---- the staging warps.  Barriers 1 + buf: the buffer is full; 1 + RING + buf: it was read, its outputs are there ----------------
        auto write_out = [&](int buf, int base) {
            for (int i = st_id; i < GROUP * BCOLS; i += ST) {
                const int g = i / BCOLS, c = i % BCOLS;
                if (base + g < t1 && j0 + c < vdim) o[((size_t)(base + g) * H + h) * vdim + j0 + c] = s_o[buf][g][c];
            }
        };
        const int groups = (t1 - t0 + GROUP - 1) / GROUP;
        for (int i = 0; i < FILL; i++) {
            if (i < groups) copy(i, t0 + i * GROUP);
            else asm volatile("cp.async.commit_group;\n" ::: "memory");
        }
        for (int n = 0; n < groups; n++) {
            asm volatile("cp.async.wait_group %0;\n" ::"n"(FILL - 1) : "memory");
            dr_bar_arrive(1 + n % RING, ALL);
            const int m = n + FILL, buf = m % RING;                    // the group whose copies start now
            if (m >= RING) {                                               // (m - RING < groups: FILL < RING)
                dr_bar_sync(1 + RING + buf, ALL);
                write_out(buf, t0 + (m - RING) * GROUP);
            }
            if (m < groups) copy(buf, t0 + m * GROUP);
            else asm volatile("cp.async.commit_group;\n" ::: "memory");
        }
        for (int m = groups + FILL > RING ? groups + FILL - RING : 0; m < groups; m++) {      // the groups that the loop has not written
            dr_bar_sync(1 + RING + m % RING, ALL);
            write_out(m % RING, t0 + m * GROUP);
        }
        return;
    }
    // ---- the computing warps ----------------------------------------------------------------------------------------------------
    const int part = threadIdx.x % SPLIT, first = COLS * (threadIdx.x / SPLIT);   // this lane's channels; its first column
    const int odd = COLS == 2 ? part & 1 : 0, col = first + odd;           // the column whose sums this lane ends with
    const int j = j0 + first;
    float* st = state + ((size_t)seq_slot[b] * H + h) * dim * vdim;
    const bool whole = COLS == 2 && vdim % 2 == 0 && ((uintptr_t)state & 7) == 0;     // the state's rows start on 8 bytes
    f32x2 S[COLS][R / 2];
#pragma unroll
    for (int i = 0; i < R; i += 2) {
        const int d = 4 * SPLIT * (i / 4) + 4 * part + (i & 3);
        if (whole) {
            const float2 x = j < vdim && d < dim ? *reinterpret_cast<const float2*>(st + (size_t)d * vdim + j) : make_float2(0.0f, 0.0f);
            const float2 y = j < vdim && d + 1 < dim ? *reinterpret_cast<const float2*>(st + (size_t)(d + 1) * vdim + j) : make_float2(0.0f, 0.0f);
            S[0][i / 2] = dr_pack2(x.x, y.x);
            S[COLS - 1][i / 2] = dr_pack2(COLS == 2 ? x.y : x.x, COLS == 2 ? y.y : y.x);
        } else {
#pragma unroll
            for (int c = 0; c < COLS; c++)
                S[c][i / 2] = dr_pack2(j + c < vdim && d < dim ? st[(size_t)d * vdim + j + c] : 0.0f,
                                       j + c < vdim && d + 1 < dim ? st[(size_t)(d + 1) * vdim + j + c] : 0.0f);
        }
    }
    struct Token {                                                         // a token's vectors in registers
        f32x2 x[VECS][R / 2];
        float v, beta, kq, g;
    };
    auto load = [&](Token& t, int buf, int g) {
#pragma unroll
        for (int w = 0; w < VECS; w++)
#pragma unroll
            for (int i = 0; i < R; i += 4) {
                const ulonglong2 p = *reinterpret_cast<const ulonglong2*>(&s_x[buf][g][w][4 * SPLIT * (i / 4) + 4 * part]);
                t.x[w][i / 2] = p.x;
                t.x[w][i / 2 + 1] = p.y;
            }
        t.v = s_v[buf][g][col];
        t.beta = s_c[buf][g][0];
        t.kq = s_c[buf][g][1];
        if (SCALAR) t.g = s_c[buf][g][2];
    };
    auto partial = [&](const f32x2* s, const f32x2* x) {                   // this lane's share of a column's sum
        f32x2 p0 = dr_mul2(s[0], x[0]), p1 = dr_mul2(s[1], x[1]);
#pragma unroll
        for (int i = 2; i < R / 2; i += 2) {
            p0 = dr_fma2(s[i], x[i], p0);
            p1 = dr_fma2(s[i + 1], x[i + 1], p1);
        }
        return dr_sum2(p0) + dr_sum2(p1);
    };
    auto step = [&](const Token& t, int buf, int g) {
        const f32x2 *k = t.x[0], *q = t.x[1];
        if (!SCALAR) {
#pragma unroll
            for (int i = 0; i < R / 2; i++)
#pragma unroll
                for (int c = 0; c < COLS; c++) S[c][i] = dr_mul2(t.x[VECS - 1][i], S[c][i]);
        }
        float p[COLS], a[COLS];
#pragma unroll
        for (int c = 0; c < COLS; c++) p[c] = partial(S[c], k);
#pragma unroll
        for (int c = 0; c < COLS; c++) a[c] = partial(S[c], q);
        if (SCALAR) {
            const f32x2 gs = dr_pack2(t.g, t.g);
#pragma unroll
            for (int i = 0; i < R / 2; i++)
#pragma unroll
                for (int c = 0; c < COLS; c++) S[c][i] = dr_mul2(gs, S[c][i]);
        }
        float pred = p[0], acc = a[0];
        if (COLS == 2) {
            pred = (odd ? p[COLS - 1] : p[0]) + __shfl_xor_sync(0xffffffffu, odd ? p[0] : p[COLS - 1], 1);
            acc = (odd ? a[COLS - 1] : a[0]) + __shfl_xor_sync(0xffffffffu, odd ? a[0] : a[COLS - 1], 1);
        }
#pragma unroll
        for (int sh = COLS; sh < SPLIT; sh <<= 1) {
            const float x = __shfl_xor_sync(0xffffffffu, pred, sh), y = __shfl_xor_sync(0xffffffffu, acc, sh);
            pred += x;
            acc += y;
        }
        if (SCALAR) acc *= t.g;
        const float u = t.beta * (SCALAR ? fmaf(-t.g, pred, t.v) : t.v - pred);
        float ub[COLS];
        ub[0] = u;
        if (COLS == 2) {
            const float other = __shfl_xor_sync(0xffffffffu, u, 1);
            ub[0] = odd ? other : u;
            ub[COLS - 1] = odd ? u : other;
        }
#pragma unroll
        for (int c = 0; c < COLS; c++) {
            const f32x2 uu = dr_pack2(ub[c], ub[c]);
#pragma unroll
            for (int i = 0; i < R / 2; i++) S[c][i] = dr_fma2(k[i], uu, S[c][i]);
        }
        acc = fmaf(u, t.kq, acc);
        if (part < COLS) s_o[buf][g][col] = acc;
    };
    int nth = 0;
    for (int base = t0; base < t1; base += GROUP, nth++) {
        const int buf = nth % RING, n = min(GROUP, t1 - base);
        dr_bar_sync(1 + buf, ALL);
        if (AHEAD) {
            Token one, two;
            load(one, buf, 0);
#pragma unroll 1
            for (int g = 0; g < n; g += 2) {
                load(two, buf, g + 1);
                step(one, buf, g);
                if (g + 2 < GROUP) load(one, buf, g + 2);
                if (g + 1 < n) step(two, buf, g + 1);
            }
        } else {
#pragma unroll 1
            for (int g = 0; g < n; g++) {
                Token one;
                load(one, buf, g);
                step(one, buf, g);
            }
        }
        dr_bar_arrive(1 + RING + buf, ALL);
    }
    pdl_trigger();               // the next kernel may come in once the walk is over
#pragma unroll
    for (int i = 0; i < R; i += 2) {
        const int d = 4 * SPLIT * (i / 4) + 4 * part + (i & 3);
        float x[COLS], y[COLS];
#pragma unroll
        for (int c = 0; c < COLS; c++) dr_unpack2(S[c][i / 2], x[c], y[c]);
        if (whole) {
            if (j < vdim && d < dim) *reinterpret_cast<float2*>(st + (size_t)d * vdim + j) = make_float2(x[0], x[COLS - 1]);
            if (j < vdim && d + 1 < dim) *reinterpret_cast<float2*>(st + (size_t)(d + 1) * vdim + j) = make_float2(y[0], y[COLS - 1]);
        } else {
#pragma unroll
            for (int c = 0; c < COLS; c++) {
                if (j + c < vdim && d < dim) st[(size_t)d * vdim + j + c] = x[c];
                if (j + c < vdim && d + 1 < dim) st[(size_t)(d + 1) * vdim + j + c] = y[c];
            }
        }
    }
}

// The same for steps in which every sequence brings one token.  What bounds it: the state's trip to memory and back, and for few
// sequences the trips in front of it.  A lane has one value column, a warp 32 neighbouring ones (whole 128-byte lines of the
// state's rows) with the key channels of PP neighbouring `parts` of the kernel above (R channels each); a block has all channels of its
// columns.  The warps' sums meet in shared memory, and every warp adds them up in the order of that kernel: the same bits.
// A step of 1 / 8 / 24 / 64 sequences with the preparation, us: 16 heads of 128 x 128 5.7 / 9.0 / 17 / 37, where the kernel above with
// a token at a time took 6.5 / 13 / 31 / 75; 8 heads of 64 x 64 4.8 / 5.1 / 5.8 / 8.4 (5.7 / 5.7 / 6.7 / 9.3).
template <int R, int SPLIT, int PP, bool SCALAR>
__global__ void __launch_bounds__(32 * SPLIT / PP)
delta_single_kernel(const float* qkv, int C, int q_col, int k_col, int v_col, const float* decay, const float* beta, float* state,
                    float* __restrict__ o, const int* __restrict__ seq_slot, const int* __restrict__ seq_start, int H, int G, int dim,
                    int vdim) {
    constexpr int WARPS = SPLIT / PP, N = R * PP;                          // a lane's channels
    static_assert(N <= 32 && (PP == 1 || PP == 2), "a lane per staged channel");
    __shared__ __align__(16) float s_x[WARPS][3][N];                       // k, q and the decays of the warp's channels
    __shared__ float s_sum[2][WARPS][32];
    pdl_trigger();
    const int b = blockIdx.z, h = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int kvh = h / (H / G), j = blockIdx.x * 32 + lane;
    auto channel = [&](int n) { return 4 * SPLIT * ((n % R) / 4) + 4 * (PP * warp + n / R) + (n & 3); };
    const int t0 = seq_start[b], t1 = seq_start[b + 1];
    float* st = state + ((size_t)seq_slot[b] * H + h) * dim * vdim + j;
    pdl_wait();
    if (t0 >= t1) return;                     // a sequence without tokens keeps its state (the whole block leaves)
    const float* row = qkv + (size_t)t0 * C;
    const int mine = channel(lane % N);
    const bool own = lane < N && mine < dim;
    const float kx = own ? row[k_col + kvh * dim + mine] : 0.0f;
    const float qx = own ? row[q_col + kvh * dim + mine] : 0.0f;
    const float gx = own && !SCALAR ? decay[((size_t)t0 * H + h) * dim + mine] : 0.0f;
    const float v = j < vdim ? row[v_col + h * vdim + j] : 0.0f;
    const float bt = beta[(size_t)t0 * (H + G) + h], kq = beta[(size_t)t0 * (H + G) + H + kvh];
    const float gs = SCALAR ? decay[(size_t)t0 * H + h] : 1.0f;
    float S[N];
#pragma unroll
    for (int n = 0; n < N; n++) S[n] = j < vdim && channel(n) < dim ? st[(size_t)channel(n) * vdim] : 0.0f;
    if (lane < N) {
        s_x[warp][0][lane] = kx;
        s_x[warp][1][lane] = qx;
        s_x[warp][2][lane] = gx;
    }
    __syncwarp();
    if (!SCALAR) {
#pragma unroll
        for (int n = 0; n < N; n++) S[n] = __fmul_rn(s_x[warp][2][n], S[n]);
    }
#pragma unroll
    for (int w = 0; w < 2; w++) {                                          // S^T k, S^T q
        float part[PP];
#pragma unroll
        for (int p = 0; p < PP; p++) {
            float e[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                e[i] = __fmul_rn(S[p * R + i], s_x[warp][w][p * R + i]);
#pragma unroll
                for (int c = 4; c < R; c += 4) e[i] = fmaf(S[p * R + c + i], s_x[warp][w][p * R + c + i], e[i]);
            }
            part[p] = (e[0] + e[1]) + (e[2] + e[3]);
        }
        s_sum[w][warp][lane] = PP == 2 ? part[0] + part[PP - 1] : part[0];
    }
    __syncthreads();
    auto total = [&](int w) {
        float x[WARPS];
#pragma unroll
        for (int i = 0; i < WARPS; i++) x[i] = s_sum[w][i][lane];
#pragma unroll
        for (int m = 1; m < WARPS; m <<= 1)
#pragma unroll
            for (int i = 0; i < WARPS; i += 2 * m) x[i] += x[i + m];
        return x[0];
    };
    const float pred = total(0);
    const float u = bt * (SCALAR ? fmaf(-gs, pred, v) : v - pred);
#pragma unroll
    for (int n = 0; n < N; n++) {
        const float x = fmaf(s_x[warp][0][n], u, SCALAR ? __fmul_rn(gs, S[n]) : S[n]);
        if (j < vdim && channel(n) < dim) st[(size_t)channel(n) * vdim] = x;
    }
    if (warp == 0 && j < vdim) {
        float acc = total(1);
        if (SCALAR) acc *= gs;
        o[((size_t)t0 * H + h) * vdim + j] = fmaf(u, kq, acc);
    }
}

// qkv [tokens, C] float32 (the convolution's output; its q and k columns are made unit vectors in place): q of q/k head g
// at columns q_col + g dim .., k at k_col + g dim .., v of head h at v_col + h vdim ..;  proj [tokens, ld] (compute type):
// beta's logit of head h at column b_col + h;  z [tokens, H ddim] (compute type, rows ldz apart): the decay's projection,
// dt_bias [H ddim] and a_log [H] float32, ddim = dim (a decay per key channel) or 1 (one per head);  decay [tokens, H ddim] and beta [tokens, H + G]: float32 scratch that this call fills;
// state [slots, H, dim, vdim] float32, updated in place;  o [tokens, H, vdim] float32.
extern "C" int ri_delta_rule_recurrent(float* qkv, int C, int q_col, int k_col, int v_col, const void* proj, long long ld,
                                       int b_col, const void* z, long long ldz, int ddim, const float* dt_bias,
                                       const float* a_log, float qscale,
                                       float* decay, float* beta, float* state, float* o, const int* seq_slot,
                                       const int* seq_start, int tokens, int seqs, int H, int G, int dim, int vdim,
                                       int single, int dtype, cudaStream_t stream) {
    if (seqs == 0 || tokens == 0) return 0;
    RI_REQUIRE(seqs > 0 && tokens > 0 && H > 0 && G > 0 && H % G == 0 && dim > 0 && vdim > 0, "delta_rule_recurrent: bad sizes");
    RI_REQUIRE(seqs <= 65535 && H <= 65535, "delta_rule_recurrent: %d sequences, %d heads: too many for one launch", seqs, H);
    RI_REQUIRE(ddim == dim || ddim == 1, "delta_rule_recurrent: %d decays per head of %d key channels", ddim, dim);
    RI_REQUIRE(dim <= 512, "delta_rule_recurrent: %d key channels per head (up to 512 are built)", dim);
    const uintptr_t z_align = dtype == RI_DTYPE_F32 ? 15 : 7;
    const bool fours = ddim == dim && dim % 4 == 0 && C % 4 == 0 && q_col % 4 == 0 && k_col % 4 == 0 && ldz % 4 == 0 &&
                       (((uintptr_t)qkv | (uintptr_t)decay | (uintptr_t)dt_bias) & 15) == 0 && ((uintptr_t)z & z_align) == 0;
    const int spread = tokens >= 256 ? 1 : (H * dim + 127) / 128 > 16 ? 16 : (H * dim + 127) / 128;
    const dim3 pgrid(tokens, spread);
    RI_REQUIRE(dtype == RI_DTYPE_F32 || dtype == RI_DTYPE_BF16, "delta_rule_recurrent: unknown dtype %d", dtype);
    if (fours) {
        const dim3 g(tokens, tokens >= 256 ? 1 : (H * dim + 1023) / 1024);
#define DP_GO1(T, P) ri_launch_pdl(delta_prep_vec_kernel<T, P>, g, dim3(256), 0, stream, qkv, C, q_col, k_col, (const T*)proj, ld, b_col, \
                                   (const T*)z, ldz, dt_bias, a_log, qscale, decay, beta, H, G, dim)
#define DP_GO(T) do { if (dim <= 128) DP_GO1(T, 1); else if (dim <= 256) DP_GO1(T, 2); else DP_GO1(T, 4); } while (0)
        if (dtype == RI_DTYPE_F32) DP_GO(float);
        else DP_GO(__nv_bfloat16);
#undef DP_GO
#undef DP_GO1
    } else if (dtype == RI_DTYPE_F32)
        ri_launch_pdl(delta_prep_kernel<float>, pgrid, dim3(128), 0, stream, qkv, C, q_col, k_col, (const float*)proj, ld,
                      b_col, (const float*)z, ldz, dt_bias, a_log, qscale, decay, beta, H, G, dim, ddim);
    else
        ri_launch_pdl(delta_prep_kernel<__nv_bfloat16>, pgrid, dim3(128), 0, stream, qkv, C, q_col, k_col,
                      (const __nv_bfloat16*)proj, ld, b_col, (const __nv_bfloat16*)z, ldz, dt_bias, a_log, qscale, decay, beta, H,
                      G, dim, ddim);
    RI_CHECK_LAUNCH("delta_prep");
    // A prompt's recurrence kernel is launched the ordinary way, not as a dependent launch: its few long-lived blocks (a chain of
    // dependent instructions, one warp per scheduler) must spread one per SM, and blocks that come in while the kernel
    // before still holds most SMs pile up on the first SMs that get free and stay there (2,048 tokens of 8 heads of
    // 128 x 128: 0.97 ms as a dependent launch, 0.59 ms as an ordinary one).
    // (Single tokens: a dependent launch as everything else.)
#define DS_GO(R, SPLIT, PP, SC)                                                                                            \
    ri_launch_pdl(delta_single_kernel<R, SPLIT, PP, SC>, dim3((vdim + 31) / 32, H, seqs), dim3(32 * SPLIT / PP), 0, stream, (const float*)qkv, \
                  C, q_col, k_col, v_col, (const float*)decay, (const float*)beta, state, o, seq_slot, seq_start, H, G, dim, vdim)
    if (single) {
        if (ddim == 1 && dim > 1) {
            if (dim <= 16) DS_GO(4, 4, 1, true);
            else if (dim <= 32) DS_GO(4, 8, 1, true);
            else if (dim <= 64) DS_GO(4, 16, 2, true);
            else if (dim <= 128) DS_GO(4, 32, 2, true);
            else if (dim <= 256) DS_GO(16, 16, 1, true);
            else DS_GO(32, 16, 1, true);
        } else {
            if (dim <= 16) DS_GO(4, 4, 1, false);
            else if (dim <= 32) DS_GO(4, 8, 1, false);
            else if (dim <= 64) DS_GO(8, 8, 1, false);
            else if (dim <= 128) DS_GO(8, 16, 1, false);
            else if (dim <= 256) DS_GO(16, 16, 1, false);
            else DS_GO(32, 16, 1, false);
        }
        RI_CHECK_LAUNCH("delta_rule_recurrent");
        return 0;
    }
#undef DS_GO
    // 16-byte copies of four channels where every row of q, k and the decays starts on 16 bytes
    const bool vec = dim % 4 == 0 && C % 4 == 0 && q_col % 4 == 0 && k_col % 4 == 0 && (((uintptr_t)qkv | (uintptr_t)decay) & 15) == 0;
    static int sms = 0;
    if (!sms) {
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        sms = n > 0 ? n : 148;
    }
    // One column a lane where all blocks of a prompt's step then still have an SM to themselves, two otherwise (one a lane / two;
    // 2,048 tokens: 8 heads of 128 x 128 395 / 418 us, 8 of 64 x 64 335 / 357, 16 of 128 x 128 516 / 435, four sequences
    // of 512 tokens and 16 heads 490 / 314).  With one decay per head half as many channels a lane (16 heads of 128 x 128: 455
    // us, with eight channels 516): there is a third less to read.
#define DR_GO(R, SPLIT, COLS, GROUP, SC, VEC, ST)                                                                          \
    do {                                                                                                                 \
        constexpr int bcols = COLS * DR_CT / SPLIT;                                                                      \
        constexpr size_t sm = (size_t)DR_RING(ST) * GROUP * ((SC ? 2 : 3) * R * SPLIT + 4 + 2 * bcols) * sizeof(float);   \
        const dim3 grid((vdim + bcols - 1) / bcols, H, seqs);                                                            \
        cudaError_t e = sm > 48 * 1024 ? cudaFuncSetAttribute(delta_rule_kernel<R, SPLIT, COLS, GROUP, SC, VEC, ST>,      \
                                                              cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm) : cudaSuccess; \
        if (e != cudaSuccess) RI_FAIL((int)e, "delta_rule_recurrent: %s", cudaGetErrorString(e));                        \
        delta_rule_kernel<R, SPLIT, COLS, GROUP, SC, VEC, ST><<<grid, dim3(DR_CT + ST), sm, stream>>>(                    \
            (const float*)qkv, C, q_col, k_col, v_col, (const float*)decay, (const float*)beta, state, o, seq_slot,      \
            seq_start, H, G, dim, vdim);                                                                                 \
    } while (0)
#define DR_BY_VEC(R, SPLIT, COLS, GROUP, SC, ST)                                                                         \
    do {                                                                                                                 \
        if (vec) DR_GO(R, SPLIT, COLS, GROUP, SC, true, ST);                                                             \
        else DR_GO(R, SPLIT, COLS, GROUP, SC, false, ST);                                                                \
    } while (0)
    auto blocks = [&](int columns) { return (long long)((vdim + columns - 1) / columns) * H * seqs; };
    // With many blocks fewer staging threads, so that more blocks fit an SM (ST / 128 threads; 64 sequences of 4 tokens; 16 heads of 128 x 128
    // with one decay per head 114 us, with 128 staging threads 130; 8 heads of 256 x 128 95 / 127 us).  Not for the eight channels a lane of per-channel
    // decays: a long prompt beside many single tokens would have its blocks pile up on few SMs (500 tokens and 32 times one, 16
    // heads of 128 x 128: 151 / 133 us).
    auto many = [&](int columns) { return blocks(columns) > 4ll * sms; };
#define DR_CHANNEL(R, SPLIT, GROUP, FEWER)                                                                               \
    do {                                                                                                                 \
        if (blocks(DR_CT / SPLIT) <= sms) DR_BY_VEC(R, SPLIT, 1, GROUP, false, 128);                                     \
        else if (FEWER == 128 || !many(2 * DR_CT / SPLIT)) DR_BY_VEC(R, SPLIT, 2, GROUP, false, 128);                    \
        else DR_BY_VEC(R, SPLIT, 2, GROUP, false, FEWER);                                                                \
    } while (0)
#define DR_HEAD(R, SPLIT, GROUP, FEWER)                                                                                  \
    do {                                                                                                                 \
        if (!many(2 * DR_CT / SPLIT)) DR_BY_VEC(R, SPLIT, 2, GROUP, true, 128);                                          \
        else DR_BY_VEC(R, SPLIT, 2, GROUP, true, FEWER);                                                                 \
    } while (0)
    if (ddim == 1 && dim > 1) {
        if (dim <= 16) DR_HEAD(4, 4, 16, 64);
        else if (dim <= 32) DR_HEAD(4, 8, 16, 64);
        else if (dim <= 64) DR_HEAD(4, 16, 16, 64);
        else if (dim <= 128) DR_HEAD(4, 32, 8, 32);
        else if (dim <= 256) DR_HEAD(16, 16, 4, 64);
        else DR_HEAD(32, 16, 2, 64);
    } else {
        if (dim <= 16) DR_CHANNEL(4, 4, 16, 64);
        else if (dim <= 32) DR_CHANNEL(4, 8, 16, 64);
        else if (dim <= 64) DR_CHANNEL(8, 8, 16, 128);
        else if (dim <= 128) DR_CHANNEL(8, 16, 8, 128);
        else if (dim <= 256) DR_CHANNEL(16, 16, 4, 64);
        else DR_CHANNEL(32, 16, 2, 64);
    }
#undef DR_HEAD
#undef DR_CHANNEL
#undef DR_BY_VEC
#undef DR_GO
    RI_CHECK_LAUNCH("delta_rule_recurrent");
    return 0;
}
