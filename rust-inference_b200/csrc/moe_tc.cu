// The routed feed-forward's grouped products on the 5th-generation tensor cores (tcgen05), for steps with many pairs per
// expert (prompts): y[out(r), :] = W[e] a[r, :] for every row r of the plan's tiles of MT_ROWS rows (`moe_plan`), with
// out(r) = perm[r] (`scatter`) or r; and the same with the gate of the experts' feed-forward in its epilogue,
// y[r, i] = f(gate_i) * up_i for W[e] = [gate rows; up rows].  `moe_gather` brings the tokens' rows into the plan's order first.
//
// What bounds it: the tensor cores and, behind them, the shared memory's 128 bytes a cycle.  Two blocks on neighbouring SMs (a
// thread-block cluster) work on one tile with tcgen05.mma.cta_group::2: 256 rows x 256 outputs, of which a block copies and
// keeps 128 rows of a and 128 rows of W (32 KB for 64 k) and accumulates its 128 rows x 256 outputs.  Per 64 k that is 32 KB
// written and 32 KB read in 512 cycles of the tensor core.  A block alone with 128 x 256 has 48 KB written and 48 KB read
// for the same products: it took 0.48 us per 64 k where the products need 0.27.
// The pair stays on its SMs (six stages of 32 KB) and takes tiles one after the other, some row tiles of the plan for one
// range of outputs before the next (`mt_place`), so that the row tiles of an expert, which lie next to each other, read the
// expert's matrix at the same time (one trip to memory); two accumulators of 256 columns fill the tensor memory, so that a tile's
// epilogue runs beside the next tile's products.  In each block:
//   warps 0, 6  one lane of each starts copies: 128 rows of a as one TMA box of 64 k, and 128 rows of W as another (with the gate the
//               first block the gate rows and the second the up rows of the same channels, so that a channel's two sums meet
//               in one thread); they signal the first block's barrier
//   warp 1      of the first block: one lane issues tcgen05.mma (256 x 256 x 16, kind::f16), four a stage, and the commits that
//               hand back the stage and hand over the accumulator, to both blocks
//   warps 2..5  the epilogue of the block's own 128 rows: a thread reads a row of the accumulator (a lane of the tensor memory)
//               32 columns at a time and puts it into shared memory, from which a warp stores whole 128-byte lines
// 128-byte swizzle everywhere; rows past a tile's own are whatever follows, k past K reads as zeros, outputs past N are
// computed and not written.
// The rows are gathered by a kernel of their own (60 MB, 12 us for the step below) because gathering in this one costs more: TMA's
// gather4 brings four rows an instruction but takes some 40 cycles for each (0.78 us per 64 k), and with cp.async every
// hand-over to the tensor core waits for the copies under way (fence.proxy.async; 1.5 us per 64 k).
// The warps that issue walk their loops whole and one lane of them issues, and a wait that is over costs one instruction: with one lane
// in the loop every product took some 60 cycles to issue and every wait 200, more than the 512 that a stage's products take
// (now some 550 a stage).  Layer below: 556 us with one lane and all row tiles for one range of outputs, 534 without, 519 with the row
// tiles in groups of 12 (520 in groups of 6 and of 18: what a group reads of a stays in L2).
// 2,048 tokens of width 4,096, 16 experts of 1,376 channels, 4 choices (7,300 rows, 246 GFLOP in both products): 165 us and 95 us
// in a cold pass, 0.95 PFLOP/s, where mma.sync tiles of 64 rows x 64 outputs took 687 and 401 us and the gate's own kernel 38.
// The plan has wide tiles from 48 pairs per expert on, where they also lay for the tiles before these.  Gather and both products, wide / tiles
// of 32 rows: width 4,096, 16 experts of 1,376: 25 pairs per expert 177 / 180 us, 48 pairs 169 / 237; width 2,048, 32 experts of
// 704: 12 pairs 116 / 100, 50 pairs 114 / 138.  So the two forms meet at some 25 pairs, and from there to 47 the plan takes the
// slower one by up to 40 %; a wide step costs the host a launch more, which is what bounds small ones.
//
// Waits are bounded (error 5): whoever gives up says so in shared memory, the other roles end when they next have to wait, the copies
// under way land (`mt_land`), and the blocks end as usual with a wrong result.  -DMT_TEST_STOP_COPY_K=<k> (tests only; nothing in
// an ordinary build) makes one copying warp of each block of the first pair give up before the fourth stage in launches with K == k, a's
// in the first block and W's in the second, so that this path can be run with copies that nobody else completes.
#include "common.cuh"
#include "mma_helpers.cuh"
#include <cuda.h>

#define MT_ROWS 256                        // rows of a tile (the product's M), half of them per block
#define MT_HALF (MT_ROWS / 2)
#define MT_COLS 256                        // rows of W per tile (the product's N), half of them copied by each block
#define MT_STAGE_K 64                      // k per stage: 128 bytes, one swizzle row
#define MT_A_BYTES (MT_HALF * 128)
#define MT_W_BYTES (MT_COLS / 2 * 128)
#define MT_STAGE_BYTES (MT_A_BYTES + MT_W_BYTES)
#define MT_STAGES 6
#define MT_THREADS 224
#define MT_PITCH 36                        // floats between rows of an epilogue warp's 32 x 32 block
#define MT_EPI_BYTES (4 * 32 * MT_PITCH * 4)
#define MT_SMEM (MT_STAGES * MT_STAGE_BYTES + MT_EPI_BYTES + 256)

__device__ __forceinline__ unsigned long long mt_desc(unsigned addr) {
    // shared-memory matrix descriptor: K-major, 128-byte swizzle (layout type 2), descriptor version 1, 1024 bytes between
    // groups of 8 rows
    unsigned long long d = 0;
    d |= (unsigned long long)((addr & 0x3FFFF) >> 4);
    d |= (unsigned long long)(16 >> 4) << 16;
    d |= (unsigned long long)(1024 >> 4) << 32;
    d |= 1ull << 46;
    d |= 2ull << 61;
    return d;
}
template <int ACC>
__device__ __forceinline__ void mt_mma(unsigned tmem_d, unsigned long long a, unsigned long long b) {
    constexpr unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((MT_COLS >> 3) << 17) | ((MT_ROWS >> 4) << 24);
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}\n"
        ::"r"(tmem_d), "l"(a), "l"(b), "r"(idesc), "n"(ACC), "r"(0u) : "memory");
}
// arrives on the barrier at this place in both blocks when the products issued so far are done
__device__ __forceinline__ void mt_commit(unsigned long long* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n"
                 ::"r"(smem_u32(bar)), "h"((unsigned short)3) : "memory");
}
// `bar`: an address in the cluster's shared memory (the first block's barrier)
__device__ __forceinline__ void mt_box(unsigned dst, const CUtensorMap* map, int x, int y, unsigned bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];\n"
                 ::"r"(dst), "l"((unsigned long long)map), "r"(x), "r"(y), "r"(bar) : "memory");
}
// the address of this block's `p` in block `rank` of the cluster
__device__ __forceinline__ unsigned mt_in_block(const void* p, unsigned rank) {
    unsigned a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ void mt_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void mt_ld32(unsigned taddr, float (&v)[32]) {
    unsigned r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

// four neighbouring outputs of a row, of which `valid` lie inside it; `whole`: rows start on multiples of four elements
__device__ __forceinline__ void mt_store4(float* p, float4 v, int valid, bool whole) {
    if (whole && valid >= 4) {
        *reinterpret_cast<float4*>(p) = v;
        return;
    }
    if (valid > 0) p[0] = v.x;
    if (valid > 1) p[1] = v.y;
    if (valid > 2) p[2] = v.z;
    if (valid > 3) p[3] = v.w;
}
__device__ __forceinline__ void mt_store4(bf16* p, float4 v, int valid, bool whole) {
    if (whole && valid >= 4) {
        *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
        return;
    }
    if (valid > 0) st_f(p, v.x);
    if (valid > 1) st_f(p + 1, v.y);
    if (valid > 2) st_f(p + 2, v.z);
    if (valid > 3) st_f(p + 3, v.w);
}

// xg[r] = x[perm[r] / div] for the plan's rows, in pieces of 16 bytes
__global__ void __launch_bounds__(256)
moe_gather_kernel(const uint4* x, long long ldx, uint4* __restrict__ xg, const int* perm, const int* meta, int div, int pieces) {
    pdl_trigger();
    pdl_wait();
    const int rows = meta[1];
    for (int r = blockIdx.x; r < rows; r += gridDim.x) {
        const uint4* src = x + (long long)(perm[r] / div) * ldx;
        uint4* dst = xg + (long long)r * pieces;
        for (int i = threadIdx.x; i < pieces; i += blockDim.x) dst[i] = src[i];
    }
}

struct MtGate {
    int kind;                              // 0 none; 1 silu(g) u; 2 gelu in its tanh form times u; 3 the clamped swish
    float limit, alpha;
};
__device__ __forceinline__ float mt_gate(float g, float u, const MtGate& c) {
    if (c.kind == 3) {
        g = fminf(g, c.limit);
        u = fminf(fmaxf(u, -c.limit), c.limit) + 1.0f;
        return (g / (1.0f + expf(-c.alpha * g))) * u;
    }
    if (c.kind == 2) return 0.5f * g * (1.0f + tanhf(0.7978845608028654f * (g + 0.044715f * g * g * g))) * u;
    return g / (1.0f + expf(-g)) * u;
}

// The order of the tiles: MT_GROUP row tiles for one range of outputs after the other, then the next MT_GROUP.  What a group reads
// of a (MT_GROUP x 256 rows of 8 KB at width 4,096: 25 MB) stays in L2 over all ranges, and its experts' matrices are read once.
#define MT_GROUP 12
__device__ __forceinline__ void mt_place(int t, int row_tiles, int col_tiles, int& m, int& c) {
    const int g = t / (MT_GROUP * col_tiles), rest = t - g * MT_GROUP * col_tiles, here = min(MT_GROUP, row_tiles - g * MT_GROUP);
    c = rest / here;
    m = g * MT_GROUP + rest - c * here;
}

struct MtTail {
    unsigned long long full[MT_STAGES], empty[MT_STAGES], acc_full[2], acc_empty[2], drained;
    unsigned tmem_base;
    int dead, peer_dead;                   // somebody has given up in this block; in the other one (written by it when its roles are over)
    int fills[2];                          // how often the block's copying warps have filled a stage: a, W
};
static_assert(sizeof(MtTail) <= 256, "the tail fits behind the stages");

__device__ __forceinline__ bool mt_test(unsigned long long* bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return __all_sync(0xffffffffu, ok);
}
// A warp's wait: false when it ran out, or when it took long and somebody in the block has given up meanwhile.  Whoever finds the
// barrier over goes on, so that the copying warps may stop at different stages: `mt_land` sees to what is then under way.
__device__ __forceinline__ bool mt_wait(unsigned long long* bar, unsigned parity, MtTail& tail, int* err) {
    if (mt_test(bar, parity)) return true;
    if (!__all_sync(0xffffffffu, ri_mbar_wait(bar, parity))) {
        atomicExch(err, 5);
        *(volatile int*)&tail.dead = 1;
        return false;
    }
    return __all_sync(0xffffffffu, *(volatile int*)&tail.dead == 0);
}
__device__ __forceinline__ bool mt_elect() {
    unsigned one;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(one));
    return one != 0;
}

// After somebody has given up: the copies that were started land before either block leaves.  One thread of both blocks calls this, behind
// a barrier of the cluster, when no product is under way.  A stage is full when all four copies into it (a and W of both blocks) are, but
// the four warps may have stopped at different stages; so each block makes up what its own warps have not started of the stages
// that somebody has (any rows do), after which every such barrier completes, and the first block, whose barriers they are, waits for
// the last round of them.  No two warps are a whole round apart: a stage is filled again only when its products, which need all four
// copies, are done.
__device__ __forceinline__ void mt_land(const CUtensorMap* map_a, const CUtensorMap* map_w, MtTail& tail, unsigned ring, unsigned rank) {
    int most = 0;
    for (unsigned r = 0; r < 2; r++)
        for (int i = 0; i < 2; i++) {
            int f;
            asm volatile("ld.shared::cluster.s32 %0, [%1];\n" : "=r"(f) : "r"(mt_in_block(&tail.fills[i], r)) : "memory");
            most = max(most, f);
        }
    for (int i = 0; i < 2; i++)
        for (int f = tail.fills[i]; f < most; f++) {
            const int s = f % MT_STAGES;
            if (i == 0 && rank == 0)
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(&tail.full[s])), "r"(2 * MT_STAGE_BYTES) : "memory");
            mt_box(ring + s * MT_STAGE_BYTES + (i ? MT_A_BYTES : 0), i ? map_w : map_a, 0, 0, mt_in_block(&tail.full[s], 0));
        }
    if (rank == 0)
        for (int f = max(0, most - MT_STAGES); f < most; f++) ri_mbar_wait(&tail.full[f % MT_STAGES], (unsigned)((f / MT_STAGES) & 1));
}

// N: outputs per row (with a gate: channels, W has 2 N rows per expert); y rows start ldy elements apart
template <typename TO, bool GATED>
__global__ void __launch_bounds__(MT_THREADS, 1)
moe_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, TO* __restrict__ y, long long ldy,
              const int* perm, const int* tiles, const int* meta, int N, int K, int scatter, int whole_rows, MtGate gate,
              int* __restrict__ err) {
    extern __shared__ __align__(1024) unsigned char mt_smem[];
    if (smem_u32(mt_smem) & 1023u) {                               // the swizzle's period (the same place in both blocks)
        if (threadIdx.x == 0) atomicExch(err, 6);
        return;
    }
    MtTail& tail = *reinterpret_cast<MtTail*>(mt_smem + MT_STAGES * MT_STAGE_BYTES + MT_EPI_BYTES);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    unsigned rank;
    asm volatile("mov.u32 %0, %cluster_ctarank;\n" : "=r"(rank));
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tail.tmem_base)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
    }
    if (tid == 32) {
        for (int s = 0; s < MT_STAGES; s++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&tail.full[s])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&tail.empty[s])));
        }
        for (int b = 0; b < 2; b++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&tail.acc_full[b])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 8;\n" ::"r"(smem_u32(&tail.acc_empty[b])));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&tail.drained)));
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        tail.dead = tail.peer_dead = 0;
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    mt_cluster_sync();                             // both blocks' barriers are set up before either copies
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const unsigned tmem = tail.tmem_base;
    pdl_trigger();                                 // every block of this grid is on its SM from the start
    pdl_wait();
    const int row_tiles = meta[0];
    const int cols = GATED ? MT_COLS / 2 : MT_COLS;                // outputs per tile
    const int col_tiles = (N + cols - 1) / cols;
    const int total = row_tiles * col_tiles;
    const int steps = (K + MT_STAGE_K - 1) / MT_STAGE_K;
    const int first = blockIdx.x >> 1, stride = gridDim.x >> 1;    // the pair's tiles

    if (warp == 0 || warp == 6) {
        // ---- copies: the first warp a, the last one W ----------------------------------------------------------------------
        const bool one = mt_elect();
        const unsigned ring = smem_u32(mt_smem) + (warp == 0 ? 0 : MT_A_BYTES), bars = mt_in_block(&tail.full[0], 0);
        int s = 0, laps = 0;                                       // the ring's place, and how often it has been filled
        bool ok = true;
        for (int t = first; t < total && ok; t += stride) {
            int m, c;
            mt_place(t, row_tiles, col_tiles, m, c);
            const int e = tiles[3 * m], r0 = tiles[3 * m + 1] + (int)rank * MT_HALF, n0 = c * cols;
            const int w0 = GATED ? e * 2 * N + (int)rank * N + n0 : e * N + n0 + (int)rank * (MT_COLS / 2);
            for (int k = 0; k < steps; k++) {
                if (laps > 0 && !mt_wait(&tail.empty[s], (unsigned)((laps - 1) & 1), tail, err)) { ok = false; break; }
#ifdef MT_TEST_STOP_COPY_K
                if (K == MT_TEST_STOP_COPY_K && blockIdx.x < 2 && warp == 6 * rank && laps * MT_STAGES + s == 3) {      // tests only: see the top
                    atomicExch(err, 5);
                    *(volatile int*)&tail.dead = 1;
                    ok = false;
                    break;
                }
#endif
                if (one) {
                    if (warp == 6) {
                        mt_box(ring + s * MT_STAGE_BYTES, &map_w, k * MT_STAGE_K, w0, bars + s * 8);
                    } else {
                        if (rank == 0)                             // what both blocks copy
                            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n"
                                         ::"r"(smem_u32(&tail.full[s])), "r"(2 * MT_STAGE_BYTES) : "memory");
                        mt_box(ring + s * MT_STAGE_BYTES, &map_a, k * MT_STAGE_K, r0, bars + s * 8);
                    }
                }
                if (++s == MT_STAGES) {
                    s = 0;
                    laps++;
                }
            }
        }
        if (one) tail.fills[warp == 0 ? 0 : 1] = laps * MT_STAGES + s;
        __syncwarp();
    } else if (warp == 1) {
        // ---- products ----------------------------------------------------------------------------------------------------
        if (rank == 0) {
            // (the whole warp walks the loop and one lane issues: what the products take is the same for all lanes, and stays so)
            const bool one = mt_elect();
            const unsigned long long a0 = mt_desc(smem_u32(mt_smem)), w0 = mt_desc(smem_u32(mt_smem + MT_A_BYTES));
            int nth = 0, s = 0;
            unsigned lap = 0;
            bool ok = true;
            for (int t = first; t < total && ok; t += stride, nth++) {
                const int buf = nth & 1;
                if (nth >= 2 && !mt_wait(&tail.acc_empty[buf], (unsigned)((nth / 2 - 1) & 1), tail, err)) break;
                for (int k = 0; k < steps; k++) {
                    if (!mt_wait(&tail.full[s], lap & 1, tail, err)) { ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    if (one) {
                        const unsigned long long off = (unsigned long long)(s * (MT_STAGE_BYTES >> 4));
                        const unsigned d = tmem + buf * MT_COLS;
                        if (k == 0) mt_mma<0>(d, a0 + off, w0 + off);
                        else mt_mma<1>(d, a0 + off, w0 + off);
#pragma unroll
                        for (int j = 1; j < MT_STAGE_K / 16; j++) mt_mma<1>(d, a0 + off + j * 2, w0 + off + j * 2);
                        mt_commit(&tail.empty[s]);
                    }
                    if (++s == MT_STAGES) {
                        s = 0;
                        lap++;
                    }
                }
                if (ok && one) mt_commit(&tail.acc_full[buf]);
            }
            if (one) {
                mt_commit(&tail.drained);                          // no product is under way when the tensor memory goes back
                ri_mbar_wait(&tail.drained, 0);
            }
            __syncwarp();
        }
    } else {
        // ---- epilogue: warp w reads the lanes 32 (w % 4) .. + 31 of the tensor memory -----------------------------------------
        const int quad = warp & 3;
        float* block = reinterpret_cast<float*>(mt_smem + MT_STAGES * MT_STAGE_BYTES) + quad * 32 * MT_PITCH;
        const int sub = lane >> 3, c4 = (lane & 7) * 4;            // what this lane stores: rows sub, sub + 4, .., four columns
        int nth = 0;
        for (int t = first; t < total; t += stride, nth++) {
            const int buf = nth & 1;
            int m, c;
            mt_place(t, row_tiles, col_tiles, m, c);
            const int n0 = c * cols;
            const int r0 = tiles[3 * m + 1], rows = tiles[3 * m + 2];
            const int base = (int)rank * MT_HALF + quad * 32;      // the warp's first row of the tile
            int out[8];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int r = base + 4 * i + sub;
                out[i] = r < rows ? (scatter ? perm[r0 + r] : r0 + r) : -1;
            }
            if (!mt_wait(&tail.acc_full[buf], (unsigned)((nth / 2) & 1), tail, err)) break;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const unsigned taddr = tmem + buf * MT_COLS + ((unsigned)(quad * 32) << 16);
            if (base < rows) {
#pragma unroll 1
                for (int c = 0; c < cols; c += 32) {
                    if (n0 + c >= N) break;
                    float v[32];
                    mt_ld32(taddr + c, v);
                    if (GATED) {
                        float u[32];
                        mt_ld32(taddr + cols + c, u);
#pragma unroll
                        for (int i = 0; i < 32; i++) v[i] = mt_gate(v[i], u[i], gate);
                    }
                    __syncwarp();                                  // the block was read
#pragma unroll
                    for (int i = 0; i < 32; i += 4)
                        *reinterpret_cast<float4*>(block + lane * MT_PITCH + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
                    __syncwarp();
                    const int valid = N - (n0 + c + c4);
#pragma unroll
                    for (int i = 0; i < 8; i++)
                        if (out[i] >= 0)
                            mt_store4(y + (long long)out[i] * ldy + n0 + c + c4, *reinterpret_cast<const float4*>(block + (4 * i + sub) * MT_PITCH + c4), valid, whole_rows);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(mt_in_block(&tail.acc_empty[buf], 0)) : "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (rank == 1 && tid == 0) ri_mbar_wait(&tail.drained, 0);     // the last commit has reached this block as well
    if (tid == 0) asm volatile("st.shared::cluster.s32 [%0], %1;\n" ::"r"(mt_in_block(&tail.peer_dead, rank ^ 1)), "r"(*(volatile int*)&tail.dead) : "memory");
    __syncwarp();
    mt_cluster_sync();                             // nobody leaves while the other block may still signal its barriers
    // (from here on a block may be gone, unless both know that somebody gave up: nothing of the other one's is read before that is known)
    if (*(volatile int*)&tail.dead | *(volatile int*)&tail.peer_dead) {
        if (tid == 0) mt_land(&map_a, &map_w, tail, smem_u32(mt_smem), rank);
        __syncthreads();
        mt_cluster_sync();
    }
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512) : "memory");
}

// ---- host ----------------------------------------------------------------------------------------------------------------
typedef CUresult (*mt_encode_tiled_fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                       const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                       CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// a row-major bfloat16 matrix [rows, K] with rows ld elements apart, copied in boxes of box_rows rows x 64 k
static int mt_tensor_map(CUtensorMap* map, const void* p, long long rows, int K, long long ld, int box_rows) {
    static mt_encode_tiled_fn encode = nullptr;
    if (!encode) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult res;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &res);
        if (e != cudaSuccess || res != cudaDriverEntryPointSuccess || !fn) RI_FAIL(-1, "moe_tc: the driver has no cuTensorMapEncodeTiled");
        encode = (mt_encode_tiled_fn)fn;
    }
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {MT_STAGE_K, (cuuint32_t)box_rows};
    cuuint32_t elem[2] = {1, 1};
    CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(p), dims, strides, box, elem,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) RI_FAIL(-1, "moe_tc: cuTensorMapEncodeTiled failed with %d (rows=%lld, K=%d)", (int)r, rows, K);
    return 0;
}

// a [a_rows, lda] bfloat16, w [E, N, K] (gate 0) or [E, 2 N, K] (gate rows, then up rows; gate 1 silu, 2 gelu_tanh, 3 clamped
// swish); y [.., ldy] bfloat16 or float32 (out_f32; without a gate only).  The plan's tiles have MT_ROWS rows.  x not null: row r
// of a is scratch that becomes x[perm[r] / div] first, for the plan's rows (x [.., ldx] bfloat16).
extern "C" int ri_moe_tc(const void* x, long long ldx, int div, void* a, long long a_rows, long long lda, const void* w, void* y,
                         long long ldy, const int* perm, const int* tiles, const int* meta, int max_tiles, int E, int N, int K, int scatter, int out_f32, int gate,
                         float limit, float alpha, int* err_flag, cudaStream_t stream) {
    if (max_tiles == 0 || a_rows == 0) return 0;
    RI_REQUIRE(max_tiles > 0 && a_rows > 0 && E > 0 && N > 0 && K > 0, "moe_tc: bad sizes");
    RI_REQUIRE(K % 8 == 0 && lda % 8 == 0 && lda >= K && (((uintptr_t)a | (uintptr_t)w) & 15) == 0, "moe_tc: rows of whole 16-byte pieces are needed");
    RI_REQUIRE(gate >= 0 && gate <= 3 && !(gate && out_f32), "moe_tc: gate function %d", gate);
    const long long w_rows = (long long)E * N * (gate ? 2 : 1);
    RI_REQUIRE(w_rows < (1ll << 31) && a_rows < (1ll << 31), "moe_tc: too many rows");
    if (x) {
        RI_REQUIRE(div > 0 && lda == K && ldx % 8 == 0 && ldx >= K && ((uintptr_t)x & 15) == 0, "moe_tc: rows of whole 16-byte pieces are needed");
        ri_launch_pdl(moe_gather_kernel, dim3((unsigned)(a_rows < 8192 ? a_rows : 8192)), dim3(256), 0, stream, (const uint4*)x, ldx / 8, (uint4*)a,
                      perm, meta, div, K / 8);
        RI_CHECK_LAUNCH("moe_gather");
    }
    static int sms = 0;
    if (!sms) {
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        const void* kernels[3] = {(const void*)moe_tc_kernel<float, false>, (const void*)moe_tc_kernel<bf16, false>, (const void*)moe_tc_kernel<bf16, true>};
        for (const void* k : kernels) {
            cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, MT_SMEM);
            if (e != cudaSuccess) RI_FAIL((int)e, "moe_tc: %s", cudaGetErrorString(e));
        }
        sms = n > 0 ? n : 148;
    }
    CUtensorMap map_a, map_w;
    int rc = mt_tensor_map(&map_a, a, a_rows, K, lda, MT_HALF);
    if (rc) return rc;
    rc = mt_tensor_map(&map_w, w, w_rows, K, K, MT_COLS / 2);
    if (rc) return rc;
    const int cols = gate ? MT_COLS / 2 : MT_COLS;
    const long long most = (long long)max_tiles * ((N + cols - 1) / cols);
    RI_REQUIRE(most < (1ll << 31), "moe_tc: too many tiles");
    const long long pairs = sms / 2 > 0 ? sms / 2 : 1;
    const int whole = (ldy % 4 == 0 && ((uintptr_t)y & 15) == 0) ? 1 : 0;
    const MtGate g{gate, limit, alpha};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(2 * (most < pairs ? most : pairs)));
    cfg.blockDim = dim3(MT_THREADS);
    cfg.dynamicSmemBytes = MT_SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = ri_pdl_enabled();
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 2;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
#define MT_GO(TO, GATED)                                                                                                  \
    cudaLaunchKernelEx(&cfg, moe_tc_kernel<TO, GATED>, map_a, map_w, (TO*)y, ldy, perm, tiles, meta, N, K, scatter, whole, g, err_flag)
    cudaError_t le = gate ? MT_GO(bf16, true) : out_f32 ? MT_GO(float, false) : MT_GO(bf16, false);
#undef MT_GO
    if (le != cudaSuccess) RI_FAIL((int)le, "moe_tc: %s", cudaGetErrorString(le));
    RI_CHECK_LAUNCH("moe_tc");
    return 0;
}
