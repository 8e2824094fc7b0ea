// The float32 product y[M, N] = x[M, K] . W[N, K]^T on the 5th-generation tensor cores (tcgen05), in full 32-bit precision.
//
// Every float32 is the sum of three bfloat16, each the rest's nearest (8 significant bits and a sign: the sum is exact), and a product of
// two such sums is taken as six of its nine terms:
//     x w = hi hi + (hi mid + mid hi) + (mid mid + hi lo + lo hi)
// What is left out is 2^-24.2 of a product at most, of either sign (mid is 2^-8 of the value's power of two at most, lo 2^-17).  Both values are
// taken times 2^16, exactly, so that a part's last bit, 2^-149 at the least, is one that bfloat16 has (2^-133).
//
// The tensor cores multiply bfloat16 exactly and add in float32, but they cut a sum off instead of rounding it.  So the terms go two ways.
// hi hi, whose products have 16 bits, is added up there for LT_K = 32 k only, into an accumulator that starts at zero; a few products of
// like size fit its 24 bits as they are.  Then the sum is read back and added to a float32 register, rounded to nearest, over ascending k.  The
// others, some 2^-8 of the product, are added up there over all k: what is cut off is 2^-31 of a product.  Their sum joins the register at
// the end, then 2^-32 takes the powers of two back.  Every output is these two chains whatever M, N and the tile a row falls into: a
// token's result does not depend on what it is batched with.
//
// Waits are bounded (error 5): whoever gives up says so in shared memory, the others end when they next have to wait, the copies that were
// started are waited for once more, and the block ends as usual with a wrong result.  -DLF_TEST_DROP_COPY_K=<k> (tests only; nothing
// in an ordinary build) makes the first block leave out the copy of W of its first stage in launches with K == k, so that this path can be run.
#pragma once
#include "common.cuh"
#include "mma_helpers.cuh"
#include "tcgen05_helpers.cuh"

#define LT_K 32                            // k per stage and per sum of the tensor cores
#define LT_ROWS 128                        // rows of W per block (the product's M)
#define LT_W_BYTES (LT_ROWS * LT_K * 4)    // ... of a stage, as they are
#define LT_MAX_TOKENS 176                  // tokens per block (the product's N), at most
#define LT_MAX_STAGES 8
#define LT_MAX_WSTAGES 8
#define LT_W_COLS 48                       // tensor-memory columns of a stage's rows of W: three parts of 32 k
#define LT_SUMS 256                        // threads that add up
#define LT_MAX_GROUPS 4
#define LT_SMEM_MAX (224 * 1024)

// shared-memory matrix descriptor: K-major rows of 64 bytes, 64-byte swizzle (layout type 4), descriptor version 1, 512 bytes
// between groups of 8 rows
__device__ __forceinline__ unsigned long long lt_desc(unsigned addr) {
    unsigned long long d = 0;
    d |= (unsigned long long)((addr & 0x3FFFF) >> 4);
    d |= (unsigned long long)(16 >> 4) << 16;
    d |= (unsigned long long)(512 >> 4) << 32;
    d |= 1ull << 46;
    d |= 4ull << 61;
    return d;
}

__device__ __forceinline__ void lt_ld16(unsigned taddr, unsigned (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr) : "memory");
}
__device__ __forceinline__ void lt_st8(unsigned taddr, const uint4& a, const uint4& b) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n"
                 ::"r"(taddr), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w) : "memory");
}
// D += A B with A in the tensor memory; ACC 0: D = A B
template <int ACC>
__device__ __forceinline__ void lt_mma(unsigned d, unsigned a, unsigned long long b, unsigned idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}\n"
        ::"r"(d), "r"(a), "l"(b), "r"(idesc), "n"(ACC), "r"(0u) : "memory");
}
__device__ __forceinline__ bool lt_elect() {
    unsigned one;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(one));
    return one != 0;
}

__device__ __forceinline__ unsigned lt_nearest2(float a, float b) {          // a in the low half
    unsigned r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(r) : "f"(b), "f"(a));
    return r;
}
// a pair of values without the pair of parts that `h` holds (exact)
__device__ __forceinline__ unsigned long long lt_rest2(unsigned long long v, unsigned h) {
    return ffma2(pack2(__uint_as_float(h << 16), __uint_as_float(h & 0xffff0000u)), pack2(-1.0f, -1.0f), v);
}
// eight neighbouring k of a row, times 2^16, as three times eight bfloat16.  A value that leaves the range on the way is no number in one
// of its parts, and so are the outputs that it is part of (see the end of the kernel).
__device__ __forceinline__ void lt_cut(const float (&v)[8], uint4& hi, uint4& mid, uint4& lo) {
    unsigned h[4], m[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        unsigned long long rest = fmul2(pack2(v[2 * i], v[2 * i + 1]), pack2(65536.0f, 65536.0f));
        float a, b;
        unpack2(rest, a, b);
        h[i] = lt_nearest2(a, b);
        rest = lt_rest2(rest, h[i]);
        unpack2(rest, a, b);
        m[i] = lt_nearest2(a, b);
        rest = lt_rest2(rest, m[i]);
        unpack2(rest, a, b);
        l[i] = lt_nearest2(a, b);
    }
    hi = make_uint4(h[0], h[1], h[2], h[3]);
    mid = make_uint4(m[0], m[1], m[2], m[3]);
    lo = make_uint4(l[0], l[1], l[2], l[3]);
}

// The three parts of x, [3, M, Kp] with Kp = K rounded up to whole stages (zeros past K, a multiple of four)
__global__ void __launch_bounds__(256)
linear_f32_cut_kernel(const float* x, uint4* __restrict__ parts, int M, int K, int pieces) {
    pdl_trigger();
    pdl_wait();
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= (long long)M * pieces) return;
    const int m = (int)(i / pieces), k = (int)(i % pieces) * 8;
    const float* row = x + (size_t)m * K + k;
    const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const float4 a = k < K ? *reinterpret_cast<const float4*>(row) : none, b = k + 4 < K ? *reinterpret_cast<const float4*>(row + 4) : none;
    const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    uint4 hi, mid, lo;
    lt_cut(v, hi, mid, lo);
    const long long part = (long long)M * pieces;
    parts[i] = hi;
    parts[i + part] = mid;
    parts[i + 2 * part] = lo;
}

struct LtTail {
    unsigned long long full[LT_MAX_STAGES], w_full[LT_MAX_WSTAGES], w_empty[LT_MAX_WSTAGES], acc_full[LT_MAX_GROUPS], acc_empty[LT_MAX_GROUPS], turn[LT_MAX_GROUPS],
        drained[LT_MAX_GROUPS];
    unsigned tmem_base;
    int dead;
};

__device__ __forceinline__ bool lt_test(unsigned long long* bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return __all_sync(0xffffffffu, ok);
}
// A warp's wait: false when it ran out (after some milliseconds), or when somebody else has given up
__device__ __forceinline__ bool lt_wait_on(unsigned long long* bar, unsigned parity, int* dead, int* err) {
    unsigned start;
    asm volatile("mov.u32 %0, %globaltimer_lo;\n" : "=r"(start));
    for (unsigned now = start; now - start < 4000000u;) {
#pragma unroll 1
        for (int i = 0; i < 32; i++)
            if (lt_test(bar, parity)) return true;
        if (__any_sync(0xffffffffu, *(volatile int*)dead)) return false;
        asm volatile("mov.u32 %0, %globaltimer_lo;\n" : "=r"(now));
        now = __shfl_sync(0xffffffffu, now, 0);
        start = __shfl_sync(0xffffffffu, start, 0);
    }
    atomicExch(err, 5);
    *(volatile int*)dead = 1;
    return false;
}
__device__ __forceinline__ bool lt_wait(unsigned long long* bar, unsigned parity, LtTail& tail, int* err) {
    return lt_test(bar, parity) || lt_wait_on(bar, parity, &tail.dead, err);
}
__device__ __forceinline__ void lt_arrive(unsigned long long* bar) {
    asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void lt_tma_3d(void* dst, const CUtensorMap* map, int x, int y, int z, unsigned long long* bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n"
                 ::"r"(smem_u32(dst)), "l"((unsigned long long)map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar)) : "memory");
}

// A block: 128 rows of W as the product's M side, from the tensor memory; `tn` tokens (a multiple of 16, up to 32 CH) as its N side, from
// shared memory.  A ring of `stages` holds LT_K k of W as they are (128-byte swizzle) and of the three parts of x (64-byte swizzle), copied
// by TMA; another of `wstages` the parts of W in the tensor memory, and there BUFS buffers hold hi hi's sums and one more the small terms'.
//   4 GROUPS warps  take the stages by turns, four a stage: a lane reads its row of W from shared memory, cuts it and puts the parts
//                   into the tensor memory; one of the four then issues the twelve tcgen05.mma of the stage, in its turn: the small
//                   terms' sum is one chain over the stages of all groups
//   8 warps         read a stage's sums back and add them to their registers: a lane has a row of W, two warps share its tokens; two of
//                   them then start the copies into the place that the stage has left
// x is cut once, by a kernel of its own: cut in here by every block, with loads into registers, the loads' trips and the words
// written to shared memory took more time than the products (233 us and 197 where this took 114 and 93, see linear_f32.cu).
// What bounds it: with many tokens a block the tensor cores (twelve products of 128 x tn x 16 a stage, 1,060 cycles at 176 tokens, where one
// buffer for hi hi's sums is enough: they are read back under the next stage's small terms); with few tokens the hand-overs alone, some 700
// cycles a stage, where the copies of W would take 300.
template <int CH, int GROUPS, int BUFS>
__global__ void __launch_bounds__(128 * GROUPS + LT_SUMS, 1)
linear_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const float* x,
                     const float* __restrict__ w, float* __restrict__ y, int M, int N, int K, int tn, int stages, int wstages,
                     long long ldx, long long ldy, int* __restrict__ err) {
    constexpr bool SPLIT = CH == 6;                                // registers: 88 and 168 instead of 128 each
    static_assert(BUFS == GROUPS || BUFS == 1, "a buffer of sums is always the same group's, or each stage's issuer has waited for the one before");
    static_assert(!SPLIT || GROUPS == 2, "256 threads of 88 and 256 of 168 registers are what 512 of 128 have");
    extern __shared__ __align__(1024) unsigned char lt_smem[];
    __shared__ LtTail tail;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int x_part = tn * 64, x_bytes = 3 * x_part;
    unsigned char* x_ring = lt_smem + stages * LT_W_BYTES;
    const int n0 = blockIdx.x * LT_ROWS, m0 = blockIdx.y * tn;
    const int steps = (K + LT_K - 1) / LT_K;
    if (smem_u32(lt_smem) & 1023u) {                               // the swizzle's period
        if (tid == 0) atomicExch(err, 6);
        return;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tail.tmem_base)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (tid == 32) {
        for (int s = 0; s < stages; s++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 2;\n" ::"r"(smem_u32(&tail.full[s])));
        for (int s = 0; s < wstages; s++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;\n" ::"r"(smem_u32(&tail.w_full[s])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&tail.w_empty[s])));
        }
        for (int b = 0; b < BUFS; b++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&tail.acc_full[b])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 8;\n" ::"r"(smem_u32(&tail.acc_empty[b])));
        }
        for (int g = 0; g < GROUPS; g++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&tail.turn[g])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&tail.drained[g])));
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        tail.dead = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = tail.tmem_base, small = tmem + BUFS * tn, w_cols = small + tn;      // the sums, then the stages' rows of W
    pdl_wait();

    if (warp < 4 * GROUPS) {
        // ---- W, products -----------------------------------------------------------------------------------------------------
        if (SPLIT) asm volatile("setmaxnreg.dec.sync.aligned.u32 88;\n");
        const int quad = warp & 3, group = warp >> 2;
        const unsigned char* src = lt_smem + (quad * 32 + lane) * 128;
        const int swz = (lane & 7) << 4;
        const unsigned idesc = instr_desc(LT_ROWS, tn, 0);
        const unsigned long long x0 = lt_desc(smem_u32(x_ring));
        const bool one = lt_elect();
        int slot = group % stages, wslot = group % wstages;        // of stage s = group, group + GROUPS, ..
        unsigned parity = 0, wparity = 0;
        for (int s = group; s < steps; s += GROUPS) {
            if (!lt_wait(&tail.full[slot], parity, tail, err)) break;
            float v[LT_K / 8][8];
#pragma unroll
            for (int c = 0; c < LT_K / 4; c++)
                *reinterpret_cast<float4*>(&v[c / 2][4 * (c & 1)]) = *reinterpret_cast<const float4*>(src + slot * LT_W_BYTES + ((c << 4) ^ swz));
            if (s >= wstages && !lt_wait(&tail.w_empty[wslot], wparity ^ 1, tail, err)) break;
            tc_fence_after();
            const unsigned wh = w_cols + wslot * LT_W_COLS, to = wh + ((unsigned)(quad * 32) << 16);
#pragma unroll
            for (int p = 0; p < LT_K / 8; p += 2) {
                uint4 hi[2], mid[2], lo[2];
                lt_cut(v[p], hi[0], mid[0], lo[0]);
                lt_cut(v[p + 1], hi[1], mid[1], lo[1]);
                lt_st8(to + p * 4, hi[0], hi[1]);
                lt_st8(to + p * 4 + 16, mid[0], mid[1]);
                lt_st8(to + p * 4 + 32, lo[0], lo[1]);
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) lt_arrive(&tail.w_full[wslot]);
            if (quad == group) {                                   // (the issuing warps on different schedulers)
                const int buf = s % BUFS, before = (group + GROUPS - 1) % GROUPS;
                if (!lt_wait(&tail.w_full[wslot], wparity, tail, err)) break;
                if (s > 0 && !lt_wait(&tail.turn[before], (unsigned)(((s - 1) / GROUPS) & 1), tail, err)) break;
                tc_fence_after();
                const unsigned wm = wh + 16, wl = wh + 32;
                const unsigned long long xh = x0 + (unsigned long long)(slot * (x_bytes >> 4)), xm = xh + (x_part >> 4), xl = xm + (x_part >> 4);
                if (one) {
                    if (s == 0) lt_mma<0>(small, wl, xh, idesc);
                    else lt_mma<1>(small, wl, xh, idesc);
                    lt_mma<1>(small, wl + 8, xh + 2, idesc);
                    lt_mma<1>(small, wh, xl, idesc);
                    lt_mma<1>(small, wh + 8, xl + 2, idesc);
                    lt_mma<1>(small, wm, xm, idesc);
                    lt_mma<1>(small, wm + 8, xm + 2, idesc);
                    lt_mma<1>(small, wm, xh, idesc);
                    lt_mma<1>(small, wm + 8, xh + 2, idesc);
                    lt_mma<1>(small, wh, xm, idesc);
                    lt_mma<1>(small, wh + 8, xm + 2, idesc);
                }
                __syncwarp();
                // hi hi, when the sums of the stage that had the buffer have been read (beside the small terms' products)
                if (s >= BUFS && !lt_wait(&tail.acc_empty[buf], (unsigned)((s / BUFS - 1) & 1), tail, err)) break;
                tc_fence_after();
                if (one) {
                    lt_mma<0>(tmem + buf * tn, wh, xh, idesc);
                    lt_mma<1>(tmem + buf * tn, wh + 8, xh + 2, idesc);
                    umma_commit(&tail.w_empty[wslot]);
                    umma_commit(&tail.acc_full[buf]);
                    tc_fence_before();
                    lt_arrive(&tail.turn[group]);
                }
                __syncwarp();
            }
            if ((slot += GROUPS) >= stages) {
                slot -= stages;
                parity ^= 1;
            }
            if ((wslot += GROUPS) >= wstages) {
                wslot -= wstages;
                wparity ^= 1;
            }
        }
        if (quad == group && one) {                                    // no product is under way when the tensor memory goes back
            umma_commit(&tail.drained[group]);
            ri_mbar_wait(&tail.drained[group], 0);
        }
        __syncwarp();
    } else {
        // ---- sums, copies ------------------------------------------------------------------------------------------------------
        if (SPLIT) asm volatile("setmaxnreg.inc.sync.aligned.u32 168;\n");
        const int quad = warp & 3, half = (warp >> 2) & 1;         // lanes 32 quad .. of the tensor memory; tokens `from` .. of the sums
        const int from = half ? (tn / 16 + 1) / 2 * 16 : 0, to = half ? tn : (tn / 16 + 1) / 2 * 16;
        // the last two warps of the second half, which has the fewer tokens, copy: one W, one x
        const int copier = half && quad >= 2 && lt_elect() ? quad - 1 : 0;
        auto copy = [&](int s, int slot) {
            if (copier == 1) {
                tc_expect_tx(&tail.full[slot], (unsigned)LT_W_BYTES);
#ifdef LF_TEST_DROP_COPY_K
                if (K == LF_TEST_DROP_COPY_K && blockIdx.x == 0 && blockIdx.y == 0 && s == 0) return;      // tests only: see the top
#endif
                tc_tma_2d(lt_smem + slot * LT_W_BYTES, &map_w, s * LT_K, n0, &tail.full[slot]);
            } else if (copier == 2) {
                tc_expect_tx(&tail.full[slot], (unsigned)x_bytes);
                lt_tma_3d(x_ring + slot * x_bytes, &map_x, s * LT_K, m0, 0, &tail.full[slot]);
            }
        };
        if (copier) {
            asm volatile("fence.proxy.async.global;\n" ::: "memory");      // x's parts were written by ordinary stores
            for (int s = 0; s < stages && s < steps; s++) copy(s, s);
        }
        __syncwarp();
        unsigned long long acc[CH][8];                             // pairs of neighbouring tokens
#pragma unroll
        for (int c = 0; c < CH; c++)
#pragma unroll
            for (int i = 0; i < 8; i++) acc[c][i] = 0ull;
        // adds the sums in the tensor memory's columns from `taddr` on to the registers
        auto add = [&](unsigned taddr) {
#pragma unroll
            for (int c = 0; c < CH; c += 2) {
                if (from + 16 * c >= to) break;
                unsigned r[2][16];
                lt_ld16(taddr + 16 * c, r[0]);
                lt_ld16(taddr + 16 * c + 16, r[1]);                // (past the tokens: columns that exist and are not used)
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 2; e++)
#pragma unroll
                    for (int i = 0; i < 8; i++) acc[c + e][i] = fadd2(acc[c + e][i], pack2(__uint_as_float(r[e][2 * i]), __uint_as_float(r[e][2 * i + 1])));
            }
        };
        const unsigned mine = from + ((unsigned)(quad * 32) << 16);
        int slot = 0, s = 0;
        for (; s < steps; s++) {
            const int buf = s % BUFS;
            if (!lt_wait(&tail.acc_full[buf], (unsigned)((s / BUFS) & 1), tail, err)) break;
            tc_fence_after();
            add(tmem + buf * tn + mine);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) lt_arrive(&tail.acc_empty[buf]);
            if (s + stages < steps) copy(s + stages, slot);        // the products of stage s have been read and taken
            __syncwarp();
            if (++slot == stages) slot = 0;
        }
        add(small + mine);                                         // (the last stage's products were issued behind all others)
        if (copier && s < steps)                                   // somebody gave up: what was started lands first
            for (int i = s; i < s + stages && i < steps; i++) ri_mbar_wait(&tail.full[i % stages], (unsigned)((i / stages) & 1));
        __syncwarp();
        pdl_trigger();
        const int n = n0 + quad * 32 + lane;
        if (n < N) {
#pragma unroll
            for (int c = 0; c < CH; c++) {
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const int t = from + 16 * c + i;
                    if (t >= to || m0 + t >= M) break;
                    float lo, hi;
                    unpack2(acc[c][i / 2], lo, hi);
                    float v = (i & 1 ? hi : lo) * 2.3283064365386963e-10f;      // 2^-32
                    // An infinity's parts are no numbers, so its products are none either, and with the powers of two values from 2^112 and
                    // sums from 2^96 on leave the range: what is not finite is taken again, as the chain of multiply-adds over ascending k (until
                    // it is no number, which it then stays).  A thread walks W's row alone for it: no matter for single outputs, but 24 ms
                    // where all 512 x 6,144 of K = 4,096 are out of range.
                    if (!(fabsf(v) <= 3.402823466e38f)) {
                        const float *a = x + (size_t)(m0 + t) * ldx, *b = w + (size_t)n * K;
                        v = 0.0f;
#pragma unroll 1
                        for (int k = 0; k < K && v == v; k += 4) {           // (K is a multiple of four here)
                            const float4 p = *reinterpret_cast<const float4*>(a + k), q = *reinterpret_cast<const float4*>(b + k);
                            v = fmaf(p.w, q.w, fmaf(p.z, q.z, fmaf(p.y, q.y, fmaf(p.x, q.x, v))));
                        }
                    }
                    y[(size_t)(m0 + t) * ldy + n] = v;
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512) : "memory");
}
