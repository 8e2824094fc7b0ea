// Prefill attention over latent rows on the 5th-generation tensor cores (tcgen05): keys of 256 elements whose first VD (up to
// 192) elements are the values (latent attention: one pool, handed out as keys and values), bfloat16, pages of 32 tokens.
//
// What bounds it: the tensor cores and the shared memory they read (per 64 keys and 128 queries 768 cycles for Q K^T, whose 64
// columns read 6 KB of operands every 16 k, and 384 for P V); the softmax of one query tile runs beside the products of the
// other.  One block of 352 threads per SM takes work items (256 rows of a sequence and a head: two query tiles of 128) one
// after the other, as the kernel for heads of 64 and 128 does (attention_prefill_tc.cu has the order of items and the reasons
// for the hand-overs); what differs:
//   * a tile of 64 rows of 256 elements is loaded ONCE and serves as the keys of Q K^T (K-major, 16 steps of 16 elements) and,
//     its first VD elements, as the values of P V (MN-major, straight from the [key][element] tile);
//   * tensor memory holds one S buffer of 64 columns per query tile and two outputs of VD columns: 512 columns at VD = 192;
//     Q K^T of block j + 1 is issued as soon as the tile's threads hold S of block j in their registers;
//   * shared memory holds the queries (128 KB), two key/value tiles (64 KB) and one P buffer per query tile (32 KB).
// Warps 0..3 own query tile 0 (thread = row), 4..7 tile 1; a lane of warp 8 issues tile 0's products, one of warp 9 tile 1's, one of
// warp 10 starts every copy (TMA tensor copies, 128-byte swizzle).  Barriers:
//   s_full[t]  (tcgen05.commit)  S_t of a block is in tensor memory
//   s_read[t]  (4 arrivals)      the tile's threads hold it in registers: it may be overwritten
//   p_ready[t] (4 arrivals)      the tile's threads have written P_t
//   pv_done[t] (tcgen05.commit)  O_t holds that block: P_t and O_t may be touched
//   full[s] (TMA), empty[s] (both issuing lanes)   a key/value tile has landed in stage s; stage s is free
//   q_full[t] (TMA), q_empty[t] (tcgen05.commit), o_free[t] (4 arrivals)   as in attention_prefill_tc.cu
// A barrier waited on by parity is never two phases ahead of a waiter: its next phase needs something that the waiter does after
// the wait.  Waits are bounded and end in an error code (5): the thread that gave up says so in shared memory, no further copy or
// product is started, the rows' threads run through without waiting, and the block ends as usual with a wrong result.
// 2,048 tokens of 32 heads (rows of 256, values of 192, 60 GFLOP): 94 us, 640 TFLOP/s, where the mma.sync kernel took 574 us.
#include "common.cuh"
#include "mma_helpers.cuh"
#include "tcgen05_helpers.cuh"
#include <cuda.h>
#include <float.h>

#define LA_DH 256
#define LA_SLABS 4                          // 64-element (128-byte) slabs of a row
#define LA_PAGE 32
#define LA_BM 128                           // queries per tile
#define LA_BN 64                            // keys per step
#define LA_Q_SLAB (LA_BM * 128)
#define LA_KV_SLAB (LA_BN * 128)
#define LA_Q_BYTES (LA_SLABS * LA_Q_SLAB)
#define LA_KV_BYTES (LA_SLABS * LA_KV_SLAB)
#define LA_P_BYTES (LA_BM * 128)
#define LA_STAGES 2
#define LA_OFF_KV (2 * LA_Q_BYTES)
#define LA_OFF_P (LA_OFF_KV + LA_STAGES * LA_KV_BYTES)
#define LA_OFF_TAIL (LA_OFF_P + 2 * LA_P_BYTES)
#define LA_THREADS 352
#define LA_LAZY 8.0f                        // log2 of how far a score may exceed the running maximum
struct LaTail {
    unsigned long long s_full[2], s_read[2], p_ready[2], pv_done[2], full[LA_STAGES], empty[LA_STAGES], q_full[2], q_empty[2], o_free[2];
    unsigned tmem_base;
    volatile int dead;
};
#define LA_SMEM (LA_OFF_TAIL + 256)
static_assert(sizeof(LaTail) <= 256 && LA_SMEM <= 227 * 1024, "shared memory of a block");
#define LA_S_COL(t) ((t) * LA_BN)
#define LA_O_COL(t) (2 * LA_BN + (t) * 192)

struct LaItem {
    int h, kvh, t_first, len, rows, n_tiles, pos_first, pos_last, key_lo, kb0, n_blocks, n_blocks_0;
    const int* table;
};
struct LaWork {
    const int *page_table, *seq_slot, *seq_start, *seq_len;
    int seqs, H, KV, mpps, groups_max, n_items, window;
    const float* sink;
};
__device__ __forceinline__ bool la_item(const LaWork& w, int k, LaItem& it) {
    const int G = (int)gridDim.x;
    const int id = (k & 1) ? k * G + G - 1 - (int)blockIdx.x : k * G + (int)blockIdx.x;
    if (id >= w.n_items) return false;
    const int per = w.seqs * w.H;
    const int g_rev = id / per, rem = id - g_rev * per;
    const int b = rem / w.H;
    it.h = rem - b * w.H;
    const int group = w.groups_max - 1 - g_rev;
    const int t_begin = w.seq_start[b], n_new = w.seq_start[b + 1] - t_begin;
    if (group * 2 * LA_BM >= n_new) return false;
    it.len = w.seq_len[b];
    const int r_base = group * 2 * LA_BM;
    it.t_first = t_begin + r_base;
    it.rows = min(2 * LA_BM, n_new - r_base);
    it.n_tiles = it.rows > LA_BM ? 2 : 1;
    it.pos_first = it.len - n_new + r_base;
    it.pos_last = it.pos_first + it.rows - 1;
    it.key_lo = ri_first_visible(it.pos_first, w.window);
    it.kb0 = it.key_lo / LA_BN;
    it.n_blocks = it.pos_last / LA_BN + 1 - it.kb0;
    it.n_blocks_0 = it.n_tiles > 1 ? min(it.n_blocks, (it.pos_first + LA_BM - 1) / LA_BN + 1 - it.kb0) : it.n_blocks;
    it.kvh = it.h / (w.H / w.KV);
    it.table = w.page_table + (size_t)w.seq_slot[b] * w.mpps;
    return true;
}
__device__ __forceinline__ int la_tile_blocks(const LaItem& it, int t) { return t < it.n_tiles ? (t == 0 ? it.n_blocks_0 : it.n_blocks) : 0; }

// Which of two phases completes first: 1 or 2 (1 if both have), 0 when neither did in time (as ri_mbar_wait)
__device__ __forceinline__ int la_either(unsigned long long* bar1, unsigned parity1, unsigned long long* bar2, unsigned parity2) {
    auto test = [](unsigned long long* bar, unsigned parity) {
        unsigned ok;
        asm volatile("{\n.reg .pred p;\nmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
                     : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
        return ok != 0;
    };
    unsigned long long start = 0;
    for (int i = 0;; i++) {
        if (test(bar1, parity1)) return 1;
        if (test(bar2, parity2)) return 2;
        if ((i & 63) == 63) {
            const unsigned long long now = ri_globaltimer();
            if (start == 0) start = now;
            else if (now - start > 4000000ull) return 0;
        }
    }
}

template <int VD>
__global__ void __launch_bounds__(LA_THREADS, 1)
attention_latent_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_kv, bf16* __restrict__ out,
                           const LaWork work, int num_pages, float scale_log2, int* __restrict__ err) {
    extern __shared__ __align__(1024) unsigned char la_smem[];
    if (smem_u32(la_smem) & 1023u) {
        if (threadIdx.x == 0) atomicExch(err, 6);
        return;
    }
    LaTail& tail = *reinterpret_cast<LaTail*>(la_smem + LA_OFF_TAIL);
    const int H = work.H, KV = work.KV, window = work.window;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    unsigned char* kv_tiles = la_smem + LA_OFF_KV;
    const int rounds = (work.n_items + (int)gridDim.x - 1) / (int)gridDim.x;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tail.tmem_base)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (warp == 10 && lane == 0) {
        asm volatile("prefetch.tensormap [%0];\n" ::"l"((unsigned long long)&map_q) : "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"((unsigned long long)&map_kv) : "memory");
        auto init = [&](unsigned long long* bar, int n) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(n)); };
        for (int i = 0; i < 2; i++) {
            init(&tail.s_full[i], 1);
            init(&tail.s_read[i], 4);
            init(&tail.p_ready[i], 4);
            init(&tail.pv_done[i], 1);
            init(&tail.q_full[i], 1);
            init(&tail.q_empty[i], 1);
            init(&tail.o_free[i], 4);
        }
        for (int i = 0; i < LA_STAGES; i++) {
            init(&tail.full[i], 1);
            init(&tail.empty[i], 2);                                 // both issuing lanes, always
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        tail.dead = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = tail.tmem_base;
    bool dead = false;
    auto wait = [&](unsigned long long* bar, unsigned parity) {
        if (!dead && !ri_mbar_wait(bar, parity)) { atomicExch(err, 5); tail.dead = 1; dead = true; }
    };
    int started = 0, q_started = 0;
    if (warp == 10) {
        if (lane == 0) {
            // ---- the copying lane -------------------------------------------------------------------------------------
            int base = 0, n_it = 0;                // blocks of keys and items before the one at hand
            auto gone = [&]() { dead = dead || tail.dead != 0; return dead; };
            for (int k = 0; k < rounds && !gone(); k++) {
                LaItem it;
                if (!la_item(work, k, it)) continue;
                // (the queries of a later item wait for the item before's last product Q K^T: they go in behind the keys
                // that take the first stages which that item gives back)
                auto load_q = [&]() {
                    for (int t = 0; t < 2; t++) {
                        if (n_it > 0) wait(&tail.q_empty[t], (unsigned)((n_it - 1) & 1));
                        if (gone()) return;
                        tc_expect_tx(&tail.q_full[t], LA_Q_BYTES);
                        for (int sl = 0; sl < LA_SLABS; sl++)
                            tc_tma_2d(la_smem + t * LA_Q_BYTES + sl * LA_Q_SLAB, &map_q, it.h * LA_DH + sl * 64, it.t_first + t * LA_BM, &tail.q_full[t]);
                        q_started = 2 * n_it + t + 1;
                    }
                };
                if (n_it == 0) load_q();
                const int q_after = min(LA_STAGES - 1, it.n_blocks - 1);
                for (int j = 0; j < it.n_blocks; j++) {
                    const int gj = base + j, st = gj % LA_STAGES, kb = it.kb0 + j;
                    int id[2];
                    for (int p = 0; p < 2; p++) {                    // the two pages (-1: none, or wholly before the first visible key)
                        const int pg = kb * 2 + p;
                        id[p] = -1;
                        if (pg * LA_PAGE < it.len && (pg + 1) * LA_PAGE > it.key_lo) {
                            id[p] = it.table[pg];
                            if (id[p] < 0 || id[p] >= num_pages) {
                                atomicExch(err, 4);
                                id[p] = -1;
                            }
                        }
                    }
                    if (gj >= LA_STAGES) wait(&tail.empty[st], (unsigned)((gj / LA_STAGES - 1) & 1));
                    if (gone()) break;
                    tc_expect_tx(&tail.full[st], (unsigned)(((id[0] >= 0) + (id[1] >= 0)) * LA_SLABS * LA_PAGE * 128));
                    for (int p = 0; p < 2; p++)
                        if (id[p] >= 0)
                            for (int sl = 0; sl < LA_SLABS; sl++)
                                tc_tma_2d(kv_tiles + st * LA_KV_BYTES + sl * LA_KV_SLAB + p * (LA_PAGE * 128), &map_kv, sl * 64,
                                          (id[p] * KV + it.kvh) * LA_PAGE, &tail.full[st]);
                    started = gj + 1;
                    if (n_it > 0 && j == q_after) load_q();
                    if (gone()) break;
                }
                base += it.n_blocks;
                n_it++;
            }
        }
    } else if (warp >= 8) {
        if (lane == 0) {
            // ---- the issuing lane of query tile t ------------------------------------------------------------------------
            const int t = warp - 8;
            const unsigned long long qd = smem_desc(smem_u32(la_smem + t * LA_Q_BYTES), 16, 1024);
            const unsigned long long kd = smem_desc(smem_u32(kv_tiles), 16, 1024);
            const unsigned long long pd = smem_desc(smem_u32(la_smem + LA_OFF_P + t * LA_P_BYTES), 16, 1024);
            const unsigned long long vd = smem_desc(smem_u32(kv_tiles), LA_KV_SLAB, 1024);
            constexpr unsigned IDESC_QK = instr_desc(LA_BM, LA_BN, 0), IDESC_PV = instr_desc(LA_BM, VD, 1);
            const unsigned s_col = tmem + LA_S_COL(t), o_col = tmem + LA_O_COL(t);
            int c = 0, base = 0, n_it = 0, n_mine = 0;     // this tile's blocks, all blocks, items, this tile's items so far
            for (int k = 0; k < rounds && !dead; k++) {
                LaItem it;
                if (!la_item(work, k, it)) continue;
                const int mine = la_tile_blocks(it, t);
                wait(&tail.q_full[t], (unsigned)(n_it & 1));
                auto issue_qk = [&](int jb) {
                    const int idx = c + jb, gj = base + jb, st = gj % LA_STAGES;
                    if (idx >= 1) wait(&tail.s_read[t], (unsigned)((idx - 1) & 1));
                    wait(&tail.full[st], (unsigned)((gj / LA_STAGES) & 1));
                    if (dead) return;
                    tc_fence_after();
                    const unsigned long long off = (unsigned long long)(st * (LA_KV_BYTES >> 4));
#pragma unroll
                    for (int i = 0; i < LA_DH / 16; i++)
                        umma_bf16(s_col, qd + (unsigned)(((i >> 2) * LA_Q_SLAB + (i & 3) * 32) >> 4),
                                  kd + off + (unsigned)(((i >> 2) * LA_KV_SLAB + (i & 3) * 32) >> 4), IDESC_QK, i > 0);
                    umma_commit(&tail.s_full[t]);
                    if (jb + 1 == mine) umma_commit(&tail.q_empty[t]);
                };
                if (mine == 0) umma_commit(&tail.q_empty[t]);
                if (mine > 0) issue_qk(0);
                for (int j = 0; j < mine && !dead; j++) {
                    const int idx = c + j, gj = base + j, st = gj % LA_STAGES;
                    // Q K^T of the next block beside this one's softmax, if its keys are there before P is
                    bool early = false;
                    if (j + 1 < mine) {
                        const int which = la_either(&tail.full[(gj + 1) % LA_STAGES], (unsigned)(((gj + 1) / LA_STAGES) & 1), &tail.p_ready[t], (unsigned)(idx & 1));
                        if (which == 0) { atomicExch(err, 5); tail.dead = 1; dead = true; }
                        early = which == 1;
                        if (early) issue_qk(j + 1);
                    }
                    wait(&tail.p_ready[t], (unsigned)(idx & 1));
                    // the first product of an item overwrites O_t: the threads must have read the item before out of it
                    if (j == 0 && n_mine > 0) wait(&tail.o_free[t], (unsigned)((n_mine - 1) & 1));
                    if (dead) break;
                    tc_fence_after();
                    const unsigned long long off = (unsigned long long)(st * (LA_KV_BYTES >> 4));
#pragma unroll
                    for (int i = 0; i < LA_BN / 16; i++)
                        umma_bf16(o_col, pd + (unsigned)((i * 32) >> 4), vd + off + (unsigned)((i * 16 * 128) >> 4), IDESC_PV, (j > 0 || i > 0) ? 1u : 0u);
                    umma_commit(&tail.pv_done[t]);
                    umma_commit(&tail.empty[st]);                    // this tile is done with block j
                    if (j + 1 < mine && !early) issue_qk(j + 1);
                }
                // blocks that this tile leaves out: both tiles hand a stage back, once the block has landed
                for (int j = mine; j < it.n_blocks && !dead; j++) {
                    const int gj = base + j, st = gj % LA_STAGES;
                    wait(&tail.full[st], (unsigned)((gj / LA_STAGES) & 1));
                    if (!dead) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(&tail.empty[st])) : "memory");
                }
                c += mine;
                base += it.n_blocks;
                n_it++;
                n_mine += mine > 0 ? 1 : 0;
            }
            // no product is under way when the tensor memory goes back: the rows' threads have waited for the last P V of
            // every item, and after a wait that ran out
            if (dead || tail.dead) {
                umma_commit(&tail.q_empty[t]);
                ri_mbar_wait(&tail.q_empty[t], (unsigned)(n_it & 1));
            }
        }
    } else {
        // ---- a query row of tile t ------------------------------------------------------------------------------------------
        const int t = warp >> 2, row = tid & (LA_BM - 1);
        const unsigned tmem_row = tmem + ((unsigned)((warp & 3) * 32) << 16);
        unsigned char* p_row = la_smem + LA_OFF_P + t * LA_P_BYTES + row * 128;
        int c = 0, base = 0;
        for (int k = 0; k < rounds; k++) {
            LaItem it;
            if (!la_item(work, k, it)) continue;
            const int mine = la_tile_blocks(it, t);
            if (mine == 0) {
                base += it.n_blocks;
                continue;
            }
            const int row_of = t * LA_BM + row, my_pos = it.pos_first + row_of;
            const int tile_first = my_pos - row, tile_last = min(tile_first + LA_BM - 1, it.pos_last);
            const bool real_row = row_of < it.rows;
            float m = -FLT_MAX, l = 0.0f;
            for (int j = 0; j < mine; j++) {
                const int kb = it.kb0 + j, idx = c + j, gj = base + j;
                wait(&tail.s_full[t], (unsigned)(idx & 1));
                dead = dead || tail.dead != 0;
                tc_fence_after();
                float s[LA_BN];
                {
                    unsigned a[32], b[32];
                    tmem_ld32_start(tmem_row + LA_S_COL(t), a);
                    tmem_ld32_start(tmem_row + LA_S_COL(t) + 32, b);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 32; i++) {
                        s[i] = __uint_as_float(a[i]);
                        s[32 + i] = __uint_as_float(b[i]);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(&tail.s_read[t])) : "memory");
                // a block of keys needs the mask if some query of this tile does not see all of it
                if ((kb * LA_BN + LA_BN - 1 > tile_first) || (window != 0 && kb * LA_BN < ri_first_visible(tile_last, window))) {
                    const int first_vis = ri_first_visible(my_pos, window);
#pragma unroll
                    for (int i = 0; i < LA_BN; i++) s[i] = ri_sees(kb * LA_BN + i, my_pos, first_vis, 0) ? s[i] : -FLT_MAX;
                }
                float mx4[4];
#pragma unroll
                for (int q4 = 0; q4 < 4; q4++) mx4[q4] = max3(s[q4 * 16], s[q4 * 16 + 1], s[q4 * 16 + 2]);
#pragma unroll
                for (int q4 = 0; q4 < 4; q4++) {
#pragma unroll
                    for (int i = 3; i < 15; i += 2) mx4[q4] = max3(mx4[q4], s[q4 * 16 + i], s[q4 * 16 + i + 1]);
                    mx4[q4] = fmaxf(mx4[q4], s[q4 * 16 + 15]);
                }
                float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
                mx = mx == -FLT_MAX ? -FLT_MAX : mx * scale_log2;      // scale > 0
                // P_t and O_t: the block before must be through P V (its P buffer is this one)
                if (idx > 0) wait(&tail.pv_done[t], (unsigned)((idx - 1) & 1));
                // (a row past the item's rows has no say: a sequence's bits do not depend on what stands behind it)
                const bool raise = real_row && (mx > m + LA_LAZY || (m == -FLT_MAX && mx != -FLT_MAX));
                if (__any_sync(0xffffffffu, raise)) {
                    const float m_new = fmaxf(m, mx);
                    const float corr = m_new == m ? 1.0f : ((m == -FLT_MAX) ? 0.0f : ex2_approx(m - m_new));
                    m = m_new;
                    l *= corr;
                    if (j > 0) {
                        tc_fence_after();
#pragma unroll
                        for (int cc = 0; cc < VD / 32; cc++) {
                            float ob[32];
                            tmem_ld32(tmem_row + LA_O_COL(t) + cc * 32, ob);
#pragma unroll
                            for (int i = 0; i < 32; i++) ob[i] *= corr;
                            tmem_st32(tmem_row + LA_O_COL(t) + cc * 32, ob);
                        }
                        tmem_st_wait();
                    }
                }
                const float neg_m = (m == -FLT_MAX) ? 0.0f : -m;
                {
                    // a masked score is -FLT_MAX: times the (positive) scale and less any maximum its exponential is zero
                    const unsigned long long sc2 = pack2(scale_log2, scale_log2), nm2 = pack2(neg_m, neg_m);
                    unsigned long long l2[2] = {pack2(0.0f, 0.0f), pack2(0.0f, 0.0f)};
#pragma unroll
                    for (int cc = 0; cc < LA_BN / 8; cc++) {
                        unsigned w[4];
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            float x0, x1;
                            unpack2(ffma2(pack2(s[cc * 8 + 2 * e], s[cc * 8 + 2 * e + 1]), sc2, nm2), x0, x1);
                            const float p0 = ex2_approx(x0), p1 = ex2_approx(x1);
                            l2[e & 1] = fadd2(l2[e & 1], pack2(p0, p1));
                            w[e] = pack_bf16(p0, p1);
                        }
                        *(uint4*)(p_row + ((cc ^ (row & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                    float a0, a1, b0, b1;
                    unpack2(l2[0], a0, a1);
                    unpack2(l2[1], b0, b1);
                    l += (a0 + a1) + (b0 + b1);
                }
                // Rows of the tile past the sequence's end or before the first key that any query of the item sees may hold
                // anything, and 0 times a NaN is a NaN: each tile's threads zero the values' part before they say that P is
                // written.  (The other tile's Q K^T may read them as keys meanwhile: keys that are masked.)
                const int from = it.len - kb * LA_BN, upto = it.key_lo - kb * LA_BN;
                if (from < LA_BN || upto > 0) {
                    const int st = gj % LA_STAGES;
                    wait(&tail.full[st], (unsigned)((gj / LA_STAGES) & 1));
                    unsigned char* tile = kv_tiles + st * LA_KV_BYTES;
                    for (int r = row >> 3; r < LA_BN; r += LA_BM / 8)
                        if (r >= from || r < upto)
#pragma unroll
                            for (int sl = 0; sl < VD / 64; sl++) *(uint4*)(tile + sl * LA_KV_SLAB + r * 128 + ((row & 7) << 4)) = make_uint4(0, 0, 0, 0);
                }
                fence_async_smem();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(&tail.p_ready[t])) : "memory");
            }
            // ---- out = O / l ------------------------------------------------------------------------------------------------
            wait(&tail.pv_done[t], (unsigned)((c + mine - 1) & 1));
            tc_fence_after();
            const bool store = real_row && !dead;
            if (work.sink && m != -FLT_MAX) l += ex2_approx(work.sink[it.h] * 1.4426950408889634f - m);
            const float inv = 1.0f / l;
            bf16* dst = out + ((size_t)(it.t_first + (store ? row_of : 0)) * H + it.h) * LA_DH;
#pragma unroll
            for (int cc = 0; cc < LA_DH / 32; cc++) {
                float o[32];
                if (cc < VD / 32) tmem_ld32(tmem_row + LA_O_COL(t) + cc * 32, o);        // the whole warp, whether the row is a query or not
                if (store) {
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        uint4 w = make_uint4(0, 0, 0, 0);                               // (behind the values' elements: zeros)
                        if (cc < VD / 32)
                            w = make_uint4(pack_bf16(o[i] * inv, o[i + 1] * inv), pack_bf16(o[i + 2] * inv, o[i + 3] * inv),
                                           pack_bf16(o[i + 4] * inv, o[i + 5] * inv), pack_bf16(o[i + 6] * inv, o[i + 7] * inv));
                        *(uint4*)(dst + cc * 32 + i) = w;
                    }
                }
            }
            // O_t is in my registers: the next item's first product may overwrite it
            tc_fence_before();
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(&tail.o_free[t])) : "memory");
            c += mine;
            base += it.n_blocks;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (tail.dead) {
        // somebody gave up: the copies that were started are waited for once more before the shared memory goes back
        if (warp == 10 && lane == 0) {
            for (int g = started > LA_STAGES ? started - LA_STAGES : 0; g < started; g++) ri_mbar_wait(&tail.full[g % LA_STAGES], (unsigned)((g / LA_STAGES) & 1));
            for (int g = q_started > 2 ? q_started - 2 : 0; g < q_started; g++) ri_mbar_wait(&tail.q_full[g % 2], (unsigned)((g / 2) & 1));
        }
        __syncthreads();
    }
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512) : "memory");
}

// ---- host -------------------------------------------------------------------------------------------------------------------
typedef CUresult (*la_encode_tiled_fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                       const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                       CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
// a row-major bfloat16 matrix [rows, cols], copied in boxes of box_rows rows x 64 elements; rows past the last read as zeros
static int la_tensor_map(CUtensorMap* map, const void* p, long long rows, long long cols, int box_rows) {
    static la_encode_tiled_fn encode = nullptr;
    if (!encode) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult res;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &res);
        if (e != cudaSuccess || res != cudaDriverEntryPointSuccess || !fn) RI_FAIL(-1, "attention_latent_tc: the driver has no cuTensorMapEncodeTiled");
        encode = (la_encode_tiled_fn)fn;
    }
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    cuuint32_t elem[2] = {1, 1};
    CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(p), dims, strides, box, elem,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) RI_FAIL(-1, "attention_latent_tc: cuTensorMapEncodeTiled failed with %d", (int)r);
    return 0;
}

// q, out [tokens, H, 256] bfloat16; pool [pages, KV, 32, 256]; v_dims (1 .. 192): the leading elements of a row that are its
// value; the result's other elements are zeros.  max_new: the most tokens one sequence brings in this step.
extern "C" int ri_attention_latent_tc(const void* q, const void* pool, void* out, const int* page_table, const int* seq_slot,
                                      const int* seq_start, const int* seq_len, int tokens, int seqs, int max_new, int H, int KV,
                                      int mpps, int page_size, int num_pages, float scale, int window, const float* sink, int v_dims,
                                      int* err_flag, cudaStream_t stream) {
    if (seqs == 0 || max_new == 0 || tokens == 0) return 0;
    RI_REQUIRE(page_size == LA_PAGE, "attention_latent_tc: pages of %d tokens, this kernel needs %d", page_size, LA_PAGE);
    RI_REQUIRE(H > 0 && KV > 0 && H % KV == 0, "attention_latent_tc: %d heads over %d kv heads", H, KV);
    RI_REQUIRE(tokens > 0 && max_new > 0 && max_new <= tokens, "attention_latent_tc: %d tokens, at most %d of one sequence", tokens, max_new);
    RI_REQUIRE(scale > 0.0f, "attention_latent_tc: the score scale must be positive");
    RI_REQUIRE(v_dims > 0 && v_dims <= 192, "attention_latent_tc: values of %d elements (up to 192 are built)", v_dims);
    RI_REQUIRE((((uintptr_t)q | (uintptr_t)pool | (uintptr_t)out) & 15) == 0, "attention_latent_tc: q, out and the pool must be 16-byte aligned");
    const int groups_max = (max_new + 2 * LA_BM - 1) / (2 * LA_BM);
    const long long n_items = (long long)groups_max * seqs * H;
    RI_REQUIRE(n_items < (1ll << 30), "attention_latent_tc: %lld work items", n_items);
    RI_REQUIRE((long long)num_pages * KV * LA_PAGE < (1ll << 31), "attention_latent_tc: a pool of %d pages", num_pages);
    CUtensorMap map_q, map_kv;
    int rc = la_tensor_map(&map_q, q, tokens, (long long)H * LA_DH, LA_BM);
    if (rc) return rc;
    rc = la_tensor_map(&map_kv, pool, (long long)num_pages * KV * LA_PAGE, LA_DH, LA_PAGE);
    if (rc) return rc;
    static int sms = 0;
    if (!sms) {
        const void* kernels[3] = {(const void*)attention_latent_tc_kernel<64>, (const void*)attention_latent_tc_kernel<128>, (const void*)attention_latent_tc_kernel<192>};
        for (const void* k : kernels) {
            cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, LA_SMEM);
            if (e != cudaSuccess) RI_FAIL((int)e, "attention_latent_tc: %s", cudaGetErrorString(e));
        }
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        sms = n > 0 ? n : 148;
    }
    const LaWork work{page_table, seq_slot, seq_start, seq_len, seqs, H, KV, mpps, groups_max, (int)n_items, window, sink};
    const int blocks = n_items < sms ? (int)n_items : sms;
    const float scale_log2 = scale * 1.4426950408889634f;
#define LA_GO(VD) attention_latent_tc_kernel<VD><<<blocks, LA_THREADS, LA_SMEM, stream>>>(map_q, map_kv, (bf16*)out, work, num_pages, scale_log2, err_flag)
    if (v_dims <= 64) LA_GO(64);
    else if (v_dims <= 128) LA_GO(128);
    else LA_GO(192);
#undef LA_GO
    RI_CHECK_LAUNCH("attention_latent_tc");
    return 0;
}
