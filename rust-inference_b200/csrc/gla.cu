// Gated linear attention: a matrix-valued state per (sequence, head) that every token decays, feeds and reads.
//
//   a_t[d] = sigmoid(z_t[d] + bias[d])^(1/tau)                     decay of key channel d, in (0, 1)
//   S_t[d, j] = a_t[d] S_(t-1)[d, j] + k_t[d] v_t[j]               state [dim, vdim], float32, zero at a sequence's start
//   o_t[j] = sum over d of S_t[d, j] (q_t[d] qscale)               d ascending, one accumulator
// then per head  y_t = o_t / sqrt(mean_j(o_t[j]^2) + eps) * gain * silu(g_t)   (`gla_head_norm_gate`).
//
// `gla_recurrent`: a block owns one (sequence, head, tile of value columns j) and walks the sequence's new
// tokens in order with its part of the state in registers (heads of up to 128 key channels) or in shared memory, loaded
// from / stored to the sequence's slot of the state tensor at the ends.  The decay is computed as
// exp(log_sigmoid(z) / tau) with float32 functions (for steps of many tokens by `gla_decay`, once for all blocks of a head); q, k, v and z
// come from bfloat16 or float32 projections and are widened once.  A token's result depends on the tokens before it only through the state, so prompts,
// pieces of prompts and single tokens give the same bits.
//
// The same kernels run a second form (`gates` given): one decay per token and head instead of one per key channel, and
// a factor on the key,
//   S_t[d, j] = a_t S_(t-1)[d, j] + (b_t k_t[d]) v_t[j],      (a_t, b_t) = gates[t, h, 0..1], float32, made by the caller,
// optionally with one more column j = vdim whose value is 1 for every token (`ones`): that column of the state is the
// running sum n_t = a_t n_(t-1) + b_t k_t, and its output n_t . q_t, which a normaliser behind the kernel reads.  State
// and output are then [.., vdim + 1] wide.
//
//   proj [tokens, ld]: q of head h at columns q_col + h dim .., k at k_col + h dim .., v at v_col + h vdim ..
//   z    [tokens, H dim] (the low-rank decay projection, bias not yet added);  bias [H dim] float32
//   state [slots, H, dim, vdim] float32;  o [tokens, H, vdim] float32
#include "common.cuh"

#define GLA_TILE 64

__device__ __forceinline__ float gla_decay(float z, float inv_tau) {
    // log(sigmoid(z)) = min(z, 0) - log1p(exp(-|z|))
    const float ls = fminf(z, 0.0f) - log1pf(expf(-fabsf(z)));
    return expf(ls * inv_tau);
}

// two float32 multiply-adds (products) per instruction, each rounded as fmaf (a product) rounds it
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 gla_fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 gla_mul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 gla_pack2(float x, float y) {
    f32x2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
    return d;
}
__device__ __forceinline__ void gla_unpack2(f32x2 v, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v)); }

// eight neighbouring elements as they come from memory, widened (and cleared where they are not the token's own) only when they
// are stored into a buffer.  VEC: on 16 bytes.
template <typename T, bool VEC>
struct GlaPiece {
    alignas(16) T v[8];
    __device__ __forceinline__ void load(const T* p, int valid) {            // valid: elements that may be read, at least 1
        if (VEC) {
#pragma unroll
            for (int i = 0; i < (int)(sizeof(T) / 2); i++) reinterpret_cast<uint4*>(v)[i] = reinterpret_cast<const uint4*>(p)[i];
        } else {
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = p[min(i, valid - 1)];
        }
    }
};

// exp(log_sigmoid(z + bias) / tau) of a prompt's tokens: float32 [tokens, HD], HD = heads x key channels
template <typename T>
__global__ void __launch_bounds__(256)
gla_decay_kernel(const T* z, const float* __restrict__ bias, float inv_tau, float* __restrict__ decay, int HD) {
    pdl_trigger();
    const int d = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
    const float b0 = d < HD ? bias[d] : 0.0f, b1 = d + 1 < HD ? bias[d + 1] : 0.0f;
    pdl_wait();
    const size_t at = (size_t)blockIdx.y * HD + d;
    if (d < HD) decay[at] = gla_decay(ld_f(z + at) + b0, inv_tau);
    if (d + 1 < HD) decay[at + 1] = gla_decay(ld_f(z + at + 1) + b1, inv_tau);
}

// BYTES from global to shared memory without a register in between
template <int BYTES>
__device__ __forceinline__ void gla_copy(void* dst, const void* src) {
    if (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// Barriers between the computing and the staging warps of a block: `arrive` goes on, `sync` waits for everybody
__device__ __forceinline__ void gla_bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void gla_bar_arrive(int id, int threads) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// The kernel for heads of up to 128 key channels (DIMC: that rounded up to 64 or 128; channels past `dim` hold zeros and stay
// zero).  What bounds it: reading a token's vectors from shared memory, 32 words a cycle for an SM whether the lanes of a warp
// want the same words or not, and the multiply-adds, three per element of the state and token.  A thread keeps four key channels
// of four neighbouring columns in registers, LP = DIMC / 4 lanes share the columns: per token 16 words for 24
// instructions of two multiply-adds (eight channels of one column: 26 words for 12, 243 cycles of shared memory a token and SM
// where this takes some 80).  A block's four computing warps, one for each scheduler of an SM, own 512 / LP columns; a
// head of 64 x 128 is four blocks.
// Four more warps of the block stage GROUP tokens at a time into a ring of GLA_RING buffers and write the outputs of the groups
// that have been computed, so that nothing of a group's trip to memory, its conversions and its outputs stands between the
// tokens.  The copies of GLA_AHEAD groups are on their way together (cp.async into slots of the thread's own, widened from there:
// with the next group's loads in registers every group of 16 tokens took a trip to memory, 2.5 us).  A group that the sequence
// does not fill is padded with tokens of decay 1, key 0 and value 0, which leave the state as it is.
//     S[d, j] = a[d] S[d, j] + k[d] v[j];  acc_j += S[d, j] q[d]
// A thread's sum of a column runs over its channels in order (even and odd ones apart, then added); the LP lanes' sums go
// down a tree (neighbours first), for four tokens and columns side by side: every step halves the number of sums a lane still
// holds, so that each lane ends with one.  Every token's sum thus has one order that depends on the head's size only: prompts,
// pieces of prompts and single tokens (`gla_single`, below) give the same bits.
// Steps of few tokens come without decays (`decay` null): the staging warps then take them from z, every block of a head its own.
// 2,048 tokens of 32 heads of 64 x 128, with the decays' kernel: 608 -> 203 us (99 ns a token); three sequences of 2,302 tokens in
// all 645 -> 207 us; 16 heads of 128 x 129 with one decay 445 -> 278 us.  (Before: one column and four channels a thread, the
// tokens staged and the decays taken by the same warps of every block.)
#define GLA_CT 128              // computing threads
#define GLA_ST 128              // staging threads
#define GLA_RING 3
#define GLA_AHEAD 3
template <typename T, int DIMC, int GROUP, bool VEC>
__global__ void __launch_bounds__(GLA_CT + GLA_ST)
gla_walk_kernel(const T* proj, long long ld, int q_col, int k_col, int v_col, const T* z, const float* __restrict__ bias,
                float inv_tau, float qscale, const float* decay, float* state, float* __restrict__ o,
                const int* __restrict__ seq_slot, const int* __restrict__ seq_start, int H, int dim, int vdim_in, const float* gates,
                int gate_pitch, int ones) {
    constexpr int LP = DIMC / 4;                                             // lanes that share four columns
    constexpr int WCOLS = 4 * (32 / LP), BCOLS = 4 * (GLA_CT / LP);          // columns per warp and per block
    constexpr int KP = DIMC / 8, VP = BCOLS / 8;                             // staged pieces of eight per token
    constexpr int PER = (GROUP * KP + GLA_ST - 1) / GLA_ST;                  // ... and per thread
    static_assert(GROUP * VP <= GLA_ST && GROUP % 4 == 0, "a piece of values per thread; tokens in fours");
    constexpr int ROW = 3 * DIMC + BCOLS;                                    // a staged token: decay, key, query, values
    constexpr int ALL = GLA_CT + GLA_ST;
    extern __shared__ __align__(16) float gla_dyn[];                         // [ring][GROUP][ROW], outputs [ring][GROUP][BCOLS]
    const int vdim = vdim_in + ones;                                         // columns of the state and of the output
    const int b = blockIdx.z, h = blockIdx.y, j0 = blockIdx.x * BCOLS;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t0 = seq_start[b], t1 = seq_start[b + 1];
    const int slot = seq_slot[b];
    pdl_wait();
    if (t0 >= t1) return;                     // (a sequence without tokens keeps its state; the whole block leaves)

    const int st_id = threadIdx.x - GLA_CT;                                  // among the staging threads
    const bool own_decays = !decay && !gates;
    GlaPiece<T, VEC> rk[PER], rq[PER], rz[PER], rv;
    GlaPiece<float, VEC> ra[PER];
    float ga[PER], gb[PER], bs[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {             // (a thread's pieces are of the same channels in every token)
        const int d = ((int)threadIdx.x % KP) * 8 + i;
        bs[i] = own_decays && d < dim ? bias[h * dim + d] : 0.0f;
    }
    static_assert(GLA_ST % KP == 0 && GLA_CT % KP == 0, "a staging thread's channels");
    // Loads are never under a condition (a load that is gets waited for where it stands): past the group, the sequence or the
    // head something that exists is read and left out by `store`.
    auto fetch = [&](int base) {              // the raw values of tokens base .. base + GROUP - 1 into registers
#pragma unroll
        for (int e = 0; e < PER; e++) {
            const int idx = st_id + e * GLA_ST;
            const int t = min(base + idx / KP, t1 - 1), d = (idx % KP) * 8 < dim ? (idx % KP) * 8 : 0;
            const T* row = proj + (size_t)t * ld + h * dim + d;
            rk[e].load(row + k_col, dim - d);
            rq[e].load(row + q_col, dim - d);
            if (gates) {
                ga[e] = gates[((size_t)t * H + h) * gate_pitch];
                gb[e] = gates[((size_t)t * H + h) * gate_pitch + 1];
            } else if (own_decays) {
                rz[e].load(z + ((size_t)t * H + h) * dim + d, dim - d);
            } else {
                ra[e].load(decay + ((size_t)t * H + h) * dim + d, dim - d);
            }
        }
        const int t = min(base + st_id / VP, t1 - 1), jj = min(j0 + (st_id % VP) * 8, (vdim_in - 1) & ~7);
        rv.load(proj + (size_t)t * ld + v_col + h * vdim_in + jj, vdim_in - jj);
    };
    auto decays = [&](int base) {             // the decays from z, of the tokens that there are
        if (!own_decays) return;
#pragma unroll
        for (int e = 0; e < PER; e++)
            if (base + (st_id + e * GLA_ST) / KP < t1)
#pragma unroll
                for (int i = 0; i < 8; i++) ra[e].v[i] = gla_decay(ld_f(&rz[e].v[i]) + bs[i], inv_tau);
    };
    auto store = [&](int buf, int base) {     // ... and from there into a buffer
        float* to = gla_dyn + buf * GROUP * ROW;
#pragma unroll
        for (int e = 0; e < PER; e++) {
            const int idx = st_id + e * GLA_ST;
            const int g = idx / KP, d = (idx % KP) * 8;
            if (g < GROUP) {
                // a token past the sequence's end: decay 1, key 0 (the state stays); a channel past dim: all zero
                const bool live = base + g < t1;
                float a[8], k[8], q[8];
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const bool own = d + i < dim;
                    k[i] = !(live && own) ? 0.0f : gates ? ld_f(&rk[e].v[i]) * gb[e] : ld_f(&rk[e].v[i]);
                    q[i] = !(live && own) ? 0.0f : ld_f(&rq[e].v[i]) * qscale;
                    if (gates) a[i] = ga[e];
                    else a[i] = ra[e].v[i];
                    a[i] = !own ? 0.0f : live ? a[i] : 1.0f;
                }
                float* row = to + g * ROW + d;
#pragma unroll
                for (int i = 0; i < 8; i += 4) {
                    *reinterpret_cast<float4*>(row + i) = make_float4(a[i], a[i + 1], a[i + 2], a[i + 3]);
                    *reinterpret_cast<float4*>(row + DIMC + i) = make_float4(k[i], k[i + 1], k[i + 2], k[i + 3]);
                    *reinterpret_cast<float4*>(row + 2 * DIMC + i) = make_float4(q[i], q[i + 1], q[i + 2], q[i + 3]);
                }
            }
        }
        if (st_id < GROUP * VP) {
            const int jj = j0 + (st_id % VP) * 8;
            float* row = to + (st_id / VP) * ROW + 3 * DIMC + (st_id % VP) * 8;
            const bool live = base + st_id / VP < t1;      // (a value of a token past the end may be infinite, and 0 times that a NaN)
            float x[8];
#pragma unroll
            for (int i = 0; i < 8; i++) x[i] = !live ? 0.0f : jj + i < vdim_in ? ld_f(&rv.v[i]) : jj + i < vdim ? 1.0f : 0.0f;      // the column of ones
#pragma unroll
            for (int i = 0; i < 8; i += 4) *reinterpret_cast<float4*>(row + i) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
        }
    };
    float* outs = gla_dyn + GLA_RING * GROUP * ROW;
    if (threadIdx.x >= GLA_CT) {
        // ---- the staging warps.  Barriers 1 + buf: the buffer is full; 1 + GLA_RING + buf: it was read, its outputs are there ----------
        // VEC: this thread's pieces of the groups on their way, [GLA_AHEAD][16 bytes of a piece][staging thread]
        constexpr int PT = sizeof(T) / 2;                                    // 16-byte pieces of eight elements
        constexpr int EACH = 2 * PT + 2, SLOT = PER * EACH + PT;
        uint4* raw = reinterpret_cast<uint4*>(outs + GLA_RING * GROUP * BCOLS);
        auto piece16 = [&](int slot_, int i) -> uint4& { return raw[(slot_ * SLOT + i) * GLA_ST + st_id]; };
        auto issue = [&](int slot_, int base) {
#pragma unroll
            for (int e = 0; e < PER; e++) {
                const int idx = st_id + e * GLA_ST;
                const int t = min(base + idx / KP, t1 - 1), d = (idx % KP) * 8 < dim ? (idx % KP) * 8 : 0;
                const T* row = proj + (size_t)t * ld + h * dim + d;
#pragma unroll
                for (int i = 0; i < PT; i++) {
                    gla_copy<16>(&piece16(slot_, e * EACH + i), reinterpret_cast<const uint4*>(row + k_col) + i);
                    gla_copy<16>(&piece16(slot_, e * EACH + PT + i), reinterpret_cast<const uint4*>(row + q_col) + i);
                }
                if (own_decays) {
                    const T* zz = z + ((size_t)t * H + h) * dim + d;
#pragma unroll
                    for (int i = 0; i < PT; i++) gla_copy<16>(&piece16(slot_, e * EACH + 2 * PT + i), reinterpret_cast<const uint4*>(zz) + i);
                } else if (!gates) {
                    const float* dec = decay + ((size_t)t * H + h) * dim + d;
                    gla_copy<16>(&piece16(slot_, e * EACH + 2 * PT), dec);
                    gla_copy<16>(&piece16(slot_, e * EACH + 2 * PT + 1), dec + 4);
                } else {
                    const float* two = gates + ((size_t)t * H + h) * gate_pitch;
                    gla_copy<4>(&piece16(slot_, e * EACH + 2 * PT).x, two);
                    gla_copy<4>(&piece16(slot_, e * EACH + 2 * PT).y, two + 1);
                }
            }
            const int t = min(base + st_id / VP, t1 - 1), jj = min(j0 + (st_id % VP) * 8, (vdim_in - 1) & ~7);
#pragma unroll
            for (int i = 0; i < PT; i++)
                gla_copy<16>(&piece16(slot_, PER * EACH + i), reinterpret_cast<const uint4*>(proj + (size_t)t * ld + v_col + h * vdim_in + jj) + i);
        };
        auto take = [&](int slot_) {          // a slot's pieces into the registers that `store` widens
#pragma unroll
            for (int e = 0; e < PER; e++) {
#pragma unroll
                for (int i = 0; i < PT; i++) {
                    reinterpret_cast<uint4*>(rk[e].v)[i] = piece16(slot_, e * EACH + i);
                    reinterpret_cast<uint4*>(rq[e].v)[i] = piece16(slot_, e * EACH + PT + i);
                }
                const uint4 lo = piece16(slot_, e * EACH + 2 * PT);
                if (gates) {
                    ga[e] = __uint_as_float(lo.x);
                    gb[e] = __uint_as_float(lo.y);
                } else if (own_decays) {
#pragma unroll
                    for (int i = 0; i < PT; i++) reinterpret_cast<uint4*>(rz[e].v)[i] = piece16(slot_, e * EACH + 2 * PT + i);
                } else {
                    reinterpret_cast<uint4*>(ra[e].v)[0] = lo;
                    reinterpret_cast<uint4*>(ra[e].v)[1] = piece16(slot_, e * EACH + 2 * PT + 1);
                }
            }
#pragma unroll
            for (int i = 0; i < PT; i++) reinterpret_cast<uint4*>(rv.v)[i] = piece16(slot_, PER * EACH + i);
        };
        auto write_out = [&](int buf, int base) {
            for (int i = st_id; i < GROUP * BCOLS; i += GLA_ST) {
                const int g = i / BCOLS, c = i % BCOLS;
                if (base + g < t1 && j0 + c < vdim) o[((size_t)(base + g) * H + h) * vdim + j0 + c] = outs[(buf * GROUP + g) * BCOLS + c];
            }
        };
        if (VEC) {
            for (int i = 0; i < GLA_AHEAD; i++) {
                if (t0 + i * GROUP < t1) issue(i, t0 + i * GROUP);
                asm volatile("cp.async.commit_group;\n" ::: "memory");
            }
        } else {
            fetch(t0);
        }
        int n = 0;
        for (int base = t0; base < t1; base += GROUP, n++) {
            const int buf = n % GLA_RING;
            if (VEC) {
                asm volatile("cp.async.wait_group %0;\n" ::"n"(GLA_AHEAD - 1) : "memory");
                take(n % GLA_AHEAD);
                if (base + GLA_AHEAD * GROUP < t1) issue(n % GLA_AHEAD, base + GLA_AHEAD * GROUP);
                asm volatile("cp.async.commit_group;\n" ::: "memory");
            }
            decays(base);
            if (n >= GLA_RING) {
                gla_bar_sync(1 + GLA_RING + buf, ALL);
                write_out(buf, base - GLA_RING * GROUP);
            }
            store(buf, base);
            gla_bar_arrive(1 + buf, ALL);
            if (!VEC && base + GROUP < t1) fetch(base + GROUP);
        }
        for (int m = n > GLA_RING ? n - GLA_RING : 0; m < n; m++) {
            gla_bar_sync(1 + GLA_RING + m % GLA_RING, ALL);
            write_out(m % GLA_RING, t0 + m * GROUP);
        }
        return;
    }
    // ---- the computing warps ----------------------------------------------------------------------------------------------------
    const int part = lane % LP, col = warp * WCOLS + 4 * (lane / LP);        // this thread's channels 4 part .. and columns col ..
    const int j = j0 + col, d0 = 4 * part;
    float* st = state + ((size_t)slot * H + h) * dim * vdim;
    f32x2 S[4][2];                            // [column][pair of channels]
    const bool whole = vdim % 4 == 0 && ((uintptr_t)state & 15) == 0;        // the state's rows start on 16 bytes, columns come in fours
    float4 x4[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float* row = st + (size_t)(d0 + i) * vdim + j;
        x4[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (d0 + i < dim) {
            if (whole) {
                if (j < vdim) x4[i] = *reinterpret_cast<const float4*>(row);
            } else {
                if (j < vdim) x4[i].x = row[0];
                if (j + 1 < vdim) x4[i].y = row[1];
                if (j + 2 < vdim) x4[i].z = row[2];
                if (j + 3 < vdim) x4[i].w = row[3];
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 2; i++) {
        S[0][i] = gla_pack2(x4[2 * i].x, x4[2 * i + 1].x);
        S[1][i] = gla_pack2(x4[2 * i].y, x4[2 * i + 1].y);
        S[2][i] = gla_pack2(x4[2 * i].z, x4[2 * i + 1].z);
        S[3][i] = gla_pack2(x4[2 * i].w, x4[2 * i + 1].w);
    }
    struct Token {                            // a token's decay, key and query (this thread's channels) and its four values
        ulonglong2 a, k, q;
        float4 v;
    };
    auto load = [&](Token& x, const float* row) {
        x.a = *reinterpret_cast<const ulonglong2*>(row + d0);
        x.k = *reinterpret_cast<const ulonglong2*>(row + DIMC + d0);
        x.q = *reinterpret_cast<const ulonglong2*>(row + 2 * DIMC + d0);
        x.v = *reinterpret_cast<const float4*>(row + 3 * DIMC + col);
    };
    auto token = [&](const Token& x, float* out) {
        const float v[4] = {x.v.x, x.v.y, x.v.z, x.v.w};
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const f32x2 vv = gla_pack2(v[c], v[c]);
            S[c][0] = gla_fma2(x.a.x, S[c][0], gla_mul2(x.k.x, vv));
            S[c][1] = gla_fma2(x.a.y, S[c][1], gla_mul2(x.k.y, vv));
        }
#pragma unroll
        for (int c = 0; c < 4; c++) {
            float lo, hi;
            gla_unpack2(gla_fma2(S[c][1], x.q.y, gla_mul2(S[c][0], x.q.x)), lo, hi);
            out[c] = lo + hi;
        }
    };
    // the token of four and the column of four whose output this lane ends with (lanes 16 .. of 32 hold copies)
    const int my_t = 2 * (part & 1) + ((part >> 1) & 1), my_c = 2 * ((part >> 2) & 1) + ((part >> 3) & 1);
    int n = 0;
    for (int base = t0; base < t1; base += GROUP, n++) {
        const int buf = n % GLA_RING;
        gla_bar_sync(1 + buf, ALL);
        const float* rows = gla_dyn + buf * GROUP * ROW;
        Token x[2];                       // the token at hand and the next one, on its way from shared memory
        load(x[0], rows);
#pragma unroll
        for (int g = 0; g < GROUP; g += 4) {
            if (g > 0 && base + g >= t1) break;
            float v[16];
#pragma unroll
            for (int t = 0; t < 4; t++) {
                if (g + t + 1 < GROUP) load(x[(t + 1) & 1], rows + (g + t + 1) * ROW);
                token(x[t & 1], v + 4 * t);
            }
#pragma unroll
            for (int m = 1, k = 8; m < 16; m <<= 1, k >>= 1) {
                const bool upper = (lane & m) != 0;
#pragma unroll
                for (int i = 0; i < k; i++) {
                    const float give = upper ? v[i] : v[i + k], keep = upper ? v[i + k] : v[i];
                    v[i] = keep + __shfl_xor_sync(0xffffffffu, give, m);
                }
            }
            if (LP == 32) v[0] += __shfl_xor_sync(0xffffffffu, v[0], 16);
            if (part < 16) outs[(buf * GROUP + g + my_t) * BCOLS + col + my_c] = v[0];
        }
        gla_bar_arrive(1 + GLA_RING + buf, ALL);
    }
    pdl_trigger();                            // the next kernel may come in once the walk is over
#pragma unroll
    for (int i = 0; i < 4; i++) {
        float x[4], y[4];
#pragma unroll
        for (int c = 0; c < 4; c++) gla_unpack2(S[c][i / 2], x[c], y[c]);
        const float4 w = i & 1 ? make_float4(y[0], y[1], y[2], y[3]) : make_float4(x[0], x[1], x[2], x[3]);
        float* row = st + (size_t)(d0 + i) * vdim + j;
        if (d0 + i < dim) {
            if (whole) {
                if (j < vdim) *reinterpret_cast<float4*>(row) = w;
            } else {
                if (j < vdim) row[0] = w.x;
                if (j + 1 < vdim) row[1] = w.y;
                if (j + 2 < vdim) row[2] = w.z;
                if (j + 3 < vdim) row[3] = w.w;
            }
        }
    }
}

// The same for steps in which every sequence brings one token.  What bounds it: the state's trip to memory and back, and for
// few sequences the chain of trips in front of it, so a token's own loads start first and the decays' exponentials run under
// the state's loads.  A warp has eight key channels of 32 neighbouring columns (whole 128-byte lines of the state's rows,
// whatever the columns' number), a lane one column; lanes 0..7 take the decays of its channels, 8..15 its keys, 16..23 its
// queries, one each.  A block has all channels of its columns; its warps' sums are added down the walk's tree: the same bits.
// A step of single tokens of 1 / 8 / 24 / 64 sequences, 32 heads of 64 x 128: 2.4 / 5.0 / 11.8 / 29 us, where 16 columns a block
// with four channels a thread took 2.4 / 7.2 / 18 / 46; 32 heads of 128 x 128 2.9 / 8.8 / 23 / 79 (2.9 / 10.3 / 27 / 87).  With
// four channels a warp, twice the threads: 2.4 / 6.7 / 17 / 42 and 2.9 / 16 / 47 / 151.
template <typename T, int DIMC>
__global__ void __launch_bounds__(4 * DIMC)
gla_single_kernel(const T* proj, long long ld, int q_col, int k_col, int v_col, const T* z, const float* __restrict__ bias, float inv_tau,
                  float qscale, float* state, float* __restrict__ o, const int* __restrict__ seq_slot, const int* __restrict__ seq_start,
                  int H, int dim, int vdim_in, const float* gates, int gate_pitch, int ones) {
    constexpr int WARPS = DIMC / 8;
    __shared__ __align__(16) float s_x[WARPS][3][8];                         // decay, key, query of the warp's channels
    __shared__ float s_sum[WARPS][32];
    pdl_trigger();
    const int vdim = vdim_in + ones;
    const int b = blockIdx.z, h = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int j = blockIdx.x * 32 + lane, d0 = 8 * warp;
    const int what = lane >> 3, d = d0 + (lane & 7);
    const bool own = what < 3 && d < dim;
    const int t0 = seq_start[b], t1 = seq_start[b + 1];
    float* st = state + ((size_t)seq_slot[b] * H + h) * dim * vdim + (size_t)d0 * vdim + j;
    const float add = own && what == 0 && !gates ? bias[h * dim + d] : 0.0f;
    pdl_wait();
    if (t0 >= t1) return;                     // (a sequence without tokens keeps its state; the whole block leaves)
    const T* row = proj + (size_t)t0 * ld;
    const T* src = (what == 0 && !gates ? z + (size_t)t0 * H * dim : row + (what == 2 ? q_col : k_col)) + h * dim + d;
    const T raw = own ? *src : T(0.0f);
    const float a = gates ? gates[((size_t)t0 * H + h) * gate_pitch] : 0.0f;
    const float kb = gates ? gates[((size_t)t0 * H + h) * gate_pitch + 1] : 1.0f;
    const float v = j < vdim_in ? ld_f(row + v_col + h * vdim_in + j) : j < vdim ? 1.0f : 0.0f;        // the column of ones
    float S[8];
#pragma unroll
    for (int i = 0; i < 8; i++) S[i] = j < vdim && d0 + i < dim ? st[(size_t)i * vdim] : 0.0f;
    if (what < 3) {
        float x = ld_f(&raw);
        if (what == 0) x = gates ? a : gla_decay(x + add, inv_tau);
        else if (what == 1) x = gates ? x * kb : x;
        else x *= qscale;
        s_x[warp][what][lane & 7] = own ? x : 0.0f;
    }
    __syncwarp();
    float part[2];
#pragma unroll
    for (int p = 0; p < 2; p++) {
        const float4 g = *reinterpret_cast<const float4*>(&s_x[warp][0][4 * p]), k = *reinterpret_cast<const float4*>(&s_x[warp][1][4 * p]),
                     q = *reinterpret_cast<const float4*>(&s_x[warp][2][4 * p]);
        float* x = S + 4 * p;
        x[0] = fmaf(g.x, x[0], __fmul_rn(k.x, v));
        x[1] = fmaf(g.y, x[1], __fmul_rn(k.y, v));
        x[2] = fmaf(g.z, x[2], __fmul_rn(k.z, v));
        x[3] = fmaf(g.w, x[3], __fmul_rn(k.w, v));
        part[p] = fmaf(x[2], q.z, __fmul_rn(x[0], q.x)) + fmaf(x[3], q.w, __fmul_rn(x[1], q.y));
    }
    s_sum[warp][lane] = part[0] + part[1];
#pragma unroll
    for (int i = 0; i < 8; i++)
        if (j < vdim && d0 + i < dim) st[(size_t)i * vdim] = S[i];
    __syncthreads();
    if (warp == 0 && j < vdim) {
        float x[WARPS];
#pragma unroll
        for (int w = 0; w < WARPS; w++) x[w] = s_sum[w][lane];
#pragma unroll
        for (int m = 1; m < WARPS; m <<= 1)
#pragma unroll
            for (int w = 0; w < WARPS; w += 2 * m) x[w] += x[w + m];
        o[((size_t)t0 * H + h) * vdim + j] = x[0];
    }
}

template <typename T, int DIMC>
static int gla_single_go(const void* proj, long long ld, int q_col, int k_col, int v_col, const void* z, const float* bias, float tau,
                         float qscale, float* state, float* o, const int* seq_slot, const int* seq_start, int seqs, int H, int dim,
                         int vdim_in, const float* gates, int gate_pitch, int ones, cudaStream_t stream) {
    ri_launch_pdl(gla_single_kernel<T, DIMC>, dim3((vdim_in + ones + 31) / 32, H, seqs), dim3(4 * DIMC), 0, stream, (const T*)proj, ld, q_col,
                  k_col, v_col, (const T*)z, bias, 1.0f / tau, qscale, state, o, seq_slot, seq_start, H, dim, vdim_in, gates, gate_pitch, ones);
    RI_CHECK_LAUNCH("gla_recurrent");
    return 0;
}

template <typename T, int DIMC, int GROUP, bool VEC>
static int gla_walk_go(const void* proj, long long ld, int q_col, int k_col, int v_col, const void* z, const float* bias, float tau,
                       float qscale, const float* decay, float* state, float* o, const int* seq_slot, const int* seq_start, int seqs,
                       int H, int dim, int vdim_in, const float* gates, int gate_pitch, int ones, int sms, cudaStream_t stream) {
    constexpr int BCOLS = GLA_CT * 16 / DIMC, PER = (GROUP * (DIMC / 8) + GLA_ST - 1) / GLA_ST, PT = sizeof(T) / 2;
    constexpr size_t RAW = VEC ? (size_t)GLA_AHEAD * (PER * (2 * PT + 2) + PT) * GLA_ST * 16 : 0;      // the slots of pieces
    constexpr size_t need = (size_t)GLA_RING * GROUP * (3 * DIMC + 2 * BCOLS) * sizeof(float) + RAW;
    const dim3 grid((vdim_in + ones + BCOLS - 1) / BCOLS, H, seqs);
    // No more blocks than SMs: more than half of an SM's shared memory for each, so that no two share one (behind a small product
    // two had: 300 tokens of 32 heads of 64 x 128, the layer 151 -> 111 us)
    constexpr size_t alone = 116 * 1024;
    const size_t sm = need < alone && (long long)grid.x * H * seqs <= sms ? alone : need;
    // (the same bound from every thread)
    cudaError_t e = cudaFuncSetAttribute(gla_walk_kernel<T, DIMC, GROUP, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(need < alone ? alone : need));
    if (e != cudaSuccess) RI_FAIL((int)e, "gla_recurrent: %s", cudaGetErrorString(e));
    // A prompt's kernel is launched the ordinary way, not as a dependent launch: its long-lived blocks must spread over the
    // SMs, and blocks that come in while the kernel before still holds most SMs pile up on the first that get free.
    gla_walk_kernel<T, DIMC, GROUP, VEC><<<grid, dim3(GLA_CT + GLA_ST), sm, stream>>>((const T*)proj, ld, q_col, k_col, v_col, (const T*)z,
                  bias, 1.0f / tau, qscale, decay, state, o, seq_slot, seq_start, H, dim, vdim_in, gates, gate_pitch, ones);
    RI_CHECK_LAUNCH("gla_recurrent");
    return 0;
}

// Any number of key channels: the state tile [dim][GLA_TILE] lives in shared memory.
template <typename T>
__global__ void __launch_bounds__(GLA_TILE)
gla_recurrent_kernel(const T* __restrict__ proj, long long ld, int q_col, int k_col, int v_col, const T* __restrict__ z,
                     const float* __restrict__ bias, float inv_tau, float qscale, float* __restrict__ state,
                     float* __restrict__ o, const int* __restrict__ seq_slot, const int* __restrict__ seq_start, int H,
                     int dim, int vdim_in, const float* __restrict__ gates, int gate_pitch, int ones) {
    const int vdim = vdim_in + ones;
    extern __shared__ float gla_smem[];
    float* S = gla_smem;                              // [dim][GLA_TILE]
    float* tok = S + (size_t)dim * GLA_TILE;          // two buffers of [3][dim]: decay, key, query
    pdl_trigger();
    const int b = blockIdx.z, h = blockIdx.y;
    const int j = blockIdx.x * GLA_TILE + threadIdx.x;
    const bool mine = j < vdim;
    const int t0 = seq_start[b], t1 = seq_start[b + 1];
    const int slot = seq_slot[b];
    pdl_wait();
    float* st = state + ((size_t)slot * H + h) * dim * vdim;
    for (int d = 0; d < dim; d++) S[d * GLA_TILE + threadIdx.x] = mine ? st[(size_t)d * vdim + j] : 0.0f;
    for (int t = t0; t < t1; t++) {
        float* cur = tok + (size_t)((t - t0) & 1) * 3 * dim;
        const T* row = proj + (size_t)t * ld;
        const float ga = gates ? gates[((size_t)t * H + h) * gate_pitch] : 1.0f;
        const float gb = gates ? gates[((size_t)t * H + h) * gate_pitch + 1] : 1.0f;
        for (int d = threadIdx.x; d < dim; d += GLA_TILE) {
            cur[d] = gates ? ga : gla_decay(ld_f(z + ((size_t)t * H + h) * dim + d) + bias[h * dim + d], inv_tau);
            cur[dim + d] = gates ? ld_f(row + k_col + h * dim + d) * gb : ld_f(row + k_col + h * dim + d);
            cur[2 * dim + d] = ld_f(row + q_col + h * dim + d) * qscale;
        }
        const float v = !mine ? 0.0f : (j < vdim_in ? ld_f(row + v_col + h * vdim_in + j) : 1.0f);
        __syncthreads();              // the token's vectors are there (the other buffer is free again after this barrier)
        float acc = 0.0f;
        for (int d = 0; d < dim; d++) {
            const float s = fmaf(cur[d], S[d * GLA_TILE + threadIdx.x], cur[dim + d] * v);
            S[d * GLA_TILE + threadIdx.x] = s;
            acc = fmaf(s, cur[2 * dim + d], acc);
        }
        if (mine) o[((size_t)t * H + h) * vdim + j] = acc;
    }
    if (mine)
        for (int d = 0; d < dim; d++) st[(size_t)d * vdim + j] = S[d * GLA_TILE + threadIdx.x];
}

static int gla_recurrent_go(const void* proj, long long ld, int q_col, int k_col, int v_col, const void* z,
                            const float* bias, float tau, float qscale, float* decay, float* state, float* o, const int* seq_slot,
                            const int* seq_start, int tokens, int seqs, int H, int dim, int vdim_in, int single, int dtype,
                            const float* gates, int gate_pitch, int ones, cudaStream_t stream) {
    // single: every sequence brings one token (no staging of groups; the same results)
    if (seqs == 0) return 0;
    const int vdim = vdim_in + ones;                 // what the grid covers
    RI_REQUIRE(seqs > 0 && H > 0 && dim > 0 && vdim_in > 0 && tau > 0.0f, "gla_recurrent: bad sizes");
    RI_REQUIRE(gates ? gate_pitch >= 2 : (z && bias && !ones), "gla_recurrent: a decay per channel (z, bias) or per token (gates)");
    RI_REQUIRE(seqs <= 65535 && H <= 65535, "gla_recurrent: %d sequences, %d heads: too many for one launch", seqs, H);
    RI_REQUIRE(dtype == RI_DTYPE_F32 || dtype == RI_DTYPE_BF16, "gla_recurrent: unknown dtype %d", dtype);
    if (dim <= 128) {
        if (decay) {
            const int HD = H * dim;
            for (int t = 0; t < tokens; t += 65535) {        // (a grid's second dimension)
                const dim3 g((HD + 511) / 512, tokens - t < 65535 ? tokens - t : 65535);
                const size_t at = (size_t)t * HD;
                if (dtype == RI_DTYPE_F32)
                    ri_launch_pdl(gla_decay_kernel<float>, g, dim3(256), 0, stream, (const float*)z + at, bias, 1.0f / tau, decay + at, HD);
                else
                    ri_launch_pdl(gla_decay_kernel<__nv_bfloat16>, g, dim3(256), 0, stream, (const __nv_bfloat16*)z + at, bias, 1.0f / tau,
                                  decay + at, HD);
                RI_CHECK_LAUNCH("gla_decay");
            }
        }
        const bool vec = dim % 8 == 0 && vdim_in % 8 == 0 && ld % 8 == 0 && q_col % 8 == 0 && k_col % 8 == 0 && v_col % 8 == 0 &&
                         (((uintptr_t)proj | (uintptr_t)z | (uintptr_t)decay) & 15) == 0;
        // Tokens staged at a time: 16, or eight for heads of more than 64 channels where there are more blocks than SMs (a block
        // with 16 has an SM for itself, 135 KB; two fit with eight) or where sequences bring few tokens.  16 / 8 at a time, bfloat16: 32
        // heads of 128 x 128 2,048 tokens 402 / 361 us, 64 sequences of 4 tokens 344 / 186; but 16 heads of 128 x 64 (64 blocks)
        // 2,048 tokens 201 / 239, and for heads of 64 channels 172 / 255 (32 of 64 x 128).
        static int sms = 0;
        if (!sms) {
            int dev = 0, n = 0;
            cudaGetDevice(&dev);
            cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
            sms = n > 0 ? n : 148;
        }
        const bool eight = dim > 64 && ((long long)((vdim + 15) / 16) * H * seqs > sms || tokens <= 16 * (long long)seqs);
#define GLA_GO3(T, DIMC, GROUP, VEC)                                                                                           \
        return gla_walk_go<T, DIMC, GROUP, VEC>(proj, ld, q_col, k_col, v_col, z, bias, tau, qscale, decay, state, o, seq_slot, \
                                                seq_start, seqs, H, dim, vdim_in, gates, gate_pitch, ones, sms, stream)
#define GLA_GO2(T, DIMC, GROUP)                                                                                                \
        do {                                                                                                                   \
            if (vec) GLA_GO3(T, DIMC, GROUP, true);                                                                            \
            else GLA_GO3(T, DIMC, GROUP, false);                                                                               \
        } while (0)
#define GLA_GO0(T, DIMC)                                                                                                       \
        return gla_single_go<T, DIMC>(proj, ld, q_col, k_col, v_col, z, bias, tau, qscale, state, o, seq_slot, seq_start, seqs, H, \
                                      dim, vdim_in, gates, gate_pitch, ones, stream)
#define GLA_GO1(T)                                                                                                             \
        do {                                                                                                                   \
            if (single) { if (dim <= 64) GLA_GO0(T, 64); else GLA_GO0(T, 128); }                                               \
            else if (dim <= 64) GLA_GO2(T, 64, 16);                                                                            \
            else if (eight) GLA_GO2(T, 128, 8);                                                                                \
            else GLA_GO2(T, 128, 16);                                                                                          \
        } while (0)
        if (dtype == RI_DTYPE_F32) GLA_GO1(float);
        else GLA_GO1(__nv_bfloat16);
#undef GLA_GO0
#undef GLA_GO1
#undef GLA_GO2
#undef GLA_GO3
    }
    const size_t smem = ((size_t)dim * GLA_TILE + 6 * (size_t)dim) * sizeof(float);
    RI_REQUIRE(smem <= 200 * 1024, "gla_recurrent: %d key channels per head do not fit in shared memory", dim);
    const dim3 grid((vdim + GLA_TILE - 1) / GLA_TILE, H, seqs);
    cudaError_t e = cudaSuccess;
#define GLA_GO(T)                                                                                                          \
    do {                                                                                                                   \
        if (smem > 48 * 1024) e = cudaFuncSetAttribute(gla_recurrent_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
        if (e != cudaSuccess) RI_FAIL((int)e, "gla_recurrent: %s", cudaGetErrorString(e));                                 \
        ri_launch_pdl(gla_recurrent_kernel<T>, grid, dim3(GLA_TILE), smem, stream, (const T*)proj, ld, q_col, k_col, v_col, \
                      (const T*)z, bias, 1.0f / tau, qscale, state, o, seq_slot, seq_start, H, dim, vdim_in, gates,        \
                      gate_pitch, ones);                                                                                   \
    } while (0)
    if (dtype == RI_DTYPE_F32) GLA_GO(float);
    else GLA_GO(__nv_bfloat16);
#undef GLA_GO
    RI_CHECK_LAUNCH("gla_recurrent");
    return 0;
}

// decay: float32 scratch [tokens, H, dim] that a call for prompts (not `single`) with up to 128 key channels fills, or null: then
// every block takes its tokens' decays itself
extern "C" int ri_gla_recurrent(const void* proj, long long ld, int q_col, int k_col, int v_col, const void* z,
                                const float* bias, float tau, float qscale, float* decay, float* state, float* o, const int* seq_slot,
                                const int* seq_start, int tokens, int seqs, int H, int dim, int vdim, int single, int dtype,
                                cudaStream_t stream) {
    return gla_recurrent_go(proj, ld, q_col, k_col, v_col, z, bias, tau, qscale, decay, state, o, seq_slot, seq_start, tokens, seqs, H,
                            dim, vdim, single, dtype, nullptr, 0, 0, stream);
}

// The second form: gates [tokens, H, gate_pitch] float32 with the decay at [0] and the key's factor at [1]; ones: the
// state [slots, H, dim, vdim + 1] and the output [tokens, H, vdim + 1] carry the column of ones.
extern "C" int ri_gla_recurrent_scalar(const void* proj, long long ld, int q_col, int k_col, int v_col, const float* gates,
                                       int gate_pitch, int ones, float qscale, float* state, float* o, const int* seq_slot,
                                       const int* seq_start, int tokens, int seqs, int H, int dim, int vdim, int single, int dtype,
                                       cudaStream_t stream) {
    RI_REQUIRE(gates != nullptr && (ones == 0 || ones == 1), "gla_recurrent_scalar: gates are needed");
    return gla_recurrent_go(proj, ld, q_col, k_col, v_col, nullptr, nullptr, 1.0f, qscale, nullptr, state, o, seq_slot, seq_start, tokens,
                            seqs, H, dim, vdim, single, dtype, gates, gate_pitch, ones, stream);
}

// four neighbouring elements as they come from memory
template <typename T> struct GlaFour;
template <> struct GlaFour<float> {
    float4 v;
    __device__ __forceinline__ void load(const float* p) { v = *reinterpret_cast<const float4*>(p); }
    __device__ __forceinline__ float4 value() const { return v; }
    static __device__ __forceinline__ void store(float* p, const float (&r)[4]) { *reinterpret_cast<float4*>(p) = make_float4(r[0], r[1], r[2], r[3]); }
};
template <> struct GlaFour<__nv_bfloat16> {
    uint2 v;
    __device__ __forceinline__ void load(const __nv_bfloat16* p) { v = *reinterpret_cast<const uint2*>(p); }
    __device__ __forceinline__ float4 value() const {
        return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
    }
    static __device__ __forceinline__ void store(__nv_bfloat16* p, const float (&r)[4]) {
        const __nv_bfloat162 a = __floats2bfloat162_rn(r[0], r[1]), b = __floats2bfloat162_rn(r[2], r[3]);
        *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const unsigned*>(&a), *reinterpret_cast<const unsigned*>(&b));
    }
};

// y[t, h, j] = T( o[t, h, j] / sqrt(mean_j o[t, h, :]^2 + eps) * gain[j] * f(g[t, h vdim + j]) ),  f: silu (fn 1) or
// sigmoid (fn 0); a warp per (token, head), the sum of squares over the warp's tree.
template <typename T>
__global__ void gla_head_norm_gate_kernel(const float* __restrict__ o, const float* __restrict__ gain, float eps,
                                          const T* __restrict__ g, long long ldg, T* __restrict__ y, int H, int vdim,
                                          int fn, size_t units) {
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const size_t unit = (size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (unit >= units) return;
    const size_t t = unit / H;
    const int h = (int)(unit - t * H);
    const float* op = o + unit * vdim;
    float ss = 0.0f;
    for (int j = lane; j < vdim; j += 32) ss += op[j] * op[j];
    const float inv = 1.0f / sqrtf(warp_sum(ss) / (float)vdim + eps);
    for (int j = lane; j < vdim; j += 32) {
        const float zg = ld_f(g + t * ldg + (size_t)h * vdim + j);
        const float s = 1.0f / (1.0f + expf(-zg));
        st_f(y + unit * vdim + j, op[j] * inv * gain[j] * (fn == 1 ? zg * s : s));
    }
}

// The same, bit for bit, for rows of whole groups of four columns, up to 128 PIECES: a lane has four neighbouring columns (PIECES times).  Its
// part of the sum goes over the columns lane, lane + 32, .. all the same, which it reads beside them from the same lines.  What bounds it:
// memory, and the gate's functions beside it.  2,302 tokens of 32 heads of 128 columns (75 MB): 21 us, 31 with a column a lane and
// trip; two or four rows a warp with their loads on their way together take 21 and 23.
template <typename T, int PIECES>
__global__ void __launch_bounds__(256)
gla_head_norm_gate_vec_kernel(const float* __restrict__ o, const float* __restrict__ gain, float eps, const T* __restrict__ g, long long ldg,
                              T* __restrict__ y, int H, int vdim, int fn, size_t units) {
    pdl_trigger();
    const int lane = threadIdx.x & 31;
    pdl_wait();
    const size_t unit = (size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (unit >= units) return;
    const size_t t = unit / H;
    const int h = (int)(unit - t * H);
    float4 v[PIECES], gn[PIECES];
    float part[4 * PIECES];
    GlaFour<T> z[PIECES];
#pragma unroll
    for (int p = 0; p < 4 * PIECES; p++) part[p] = p * 32 + lane < vdim ? o[unit * vdim + p * 32 + lane] : 0.0f;
#pragma unroll
    for (int p = 0; p < PIECES; p++) {
        const int j = p * 128 + 4 * lane, at = j < vdim ? j : 0;
        v[p] = *reinterpret_cast<const float4*>(o + unit * vdim + at);
        z[p].load(g + t * ldg + (size_t)h * vdim + at);
        gn[p] = *reinterpret_cast<const float4*>(gain + at);
    }
    float ss = 0.0f;
#pragma unroll
    for (int p = 0; p < 4 * PIECES; p++) ss = fmaf(part[p], part[p], ss);
    const float inv = 1.0f / sqrtf(warp_sum(ss) / (float)vdim + eps);
#pragma unroll
    for (int p = 0; p < PIECES; p++) {
        const int j = p * 128 + 4 * lane;
        if (j >= vdim) break;
        const float4 zg = z[p].value();
        const float x[4] = {v[p].x, v[p].y, v[p].z, v[p].w}, gg[4] = {gn[p].x, gn[p].y, gn[p].z, gn[p].w}, zz[4] = {zg.x, zg.y, zg.z, zg.w};
        float r[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float s = 1.0f / (1.0f + expf(-zz[i]));
            r[i] = x[i] * inv * gg[i] * (fn == 1 ? zz[i] * s : s);
        }
        GlaFour<T>::store(y + unit * vdim + j, r);
    }
}

extern "C" int ri_gla_head_norm_gate(const float* o, const float* gain, float eps, const void* g, long long ldg, void* y,
                                     int tokens, int H, int vdim, int fn, int dtype, cudaStream_t stream) {
    if (tokens == 0) return 0;
    RI_REQUIRE(tokens > 0 && H > 0 && vdim > 0, "gla_head_norm_gate: bad sizes");
    const size_t units = (size_t)tokens * H;
    const unsigned blocks = (unsigned)((units + 7) / 8);
    const uintptr_t align = dtype == RI_DTYPE_F32 ? 15 : 7;
    if (vdim % 4 == 0 && vdim <= 256 && ldg % 4 == 0 && (((uintptr_t)o | (uintptr_t)gain) & 15) == 0 && (((uintptr_t)g | (uintptr_t)y) & align) == 0 &&
        (dtype == RI_DTYPE_F32 || dtype == RI_DTYPE_BF16)) {
#define HN_GO1(T, P) ri_launch_pdl(gla_head_norm_gate_vec_kernel<T, P>, dim3(blocks), dim3(256), 0, stream, o, gain, eps, (const T*)g, ldg, (T*)y, H, vdim, fn, units)
#define HN_GO(T) do { if (vdim <= 128) HN_GO1(T, 1); else HN_GO1(T, 2); } while (0)
        if (dtype == RI_DTYPE_F32) HN_GO(float);
        else HN_GO(__nv_bfloat16);
#undef HN_GO
#undef HN_GO1
        RI_CHECK_LAUNCH("gla_head_norm_gate");
        return 0;
    }
    if (dtype == RI_DTYPE_F32)
        ri_launch_pdl(gla_head_norm_gate_kernel<float>, dim3(blocks), dim3(256), 0, stream, o, gain, eps, (const float*)g, ldg, (float*)y, H, vdim, fn, units);
    else if (dtype == RI_DTYPE_BF16)
        ri_launch_pdl(gla_head_norm_gate_kernel<__nv_bfloat16>, dim3(blocks), dim3(256), 0, stream, o, gain, eps, (const __nv_bfloat16*)g, ldg, (__nv_bfloat16*)y, H, vdim, fn, units);
    else RI_FAIL(-1, "gla_head_norm_gate: unknown dtype %d", dtype);
    RI_CHECK_LAUNCH("gla_head_norm_gate");
    return 0;
}
