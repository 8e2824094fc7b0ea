// Causal grouped-query attention over the paged cache, one fixed order of arithmetic per row.
//
// This is the attention of the float32 path, and of bfloat16 models whose head size or page size the
// tensor-core kernels do not take.  A "row" is one (new token, query head).  What a row computes, and
// in which order, depends on the row's own position and on the cache's page size only: the keys it
// sees are walked in strips (32 consecutive keys of one page, at fixed places of the sequence), and
// for every strip
//     score_j = (sum over d ascending of q[d] k_j[d], one accumulator) * scale       lane j = key j of the strip
//     (with a soft cap c > 0: score_j <- c tanh(score_j / c);  with a distance bias: score_j += bias[h][pos - j])
//     m' = max(m, max_j score_j);  c = exp(m - m');  p_j = exp(score_j - m')
//     l = l c + (sum of the p_j over the warp's shuffle tree);  acc[d] = acc[d] c, then += p_j v_j[d] for j ascending
// with exp the full-precision function, as thanhauco/rust-inference's CPU attention does a page at a
// time (src/attention.rs:111-150).  So the logits of a token are the same bits however the tokens were cut
// into steps and whatever else is in the batch.
//
// Work is shared between rows, not split inside one: a block takes up to `tile_q` consecutive new tokens
// of one sequence and up to `group_chunk` query heads of one kv head, stages each strip of keys and
// values once in shared memory (as float32) for all of them, and every warp then takes the rows
// w, w + 8, ... four or two at a time (query heads of one token: what is read of a key or a value from shared memory
// serves them all): a row belongs to one warp from start to end, its running maximum, sum and output live in shared
// memory between strips.  Keys and values are thus read from memory once per
// (tile, kv head) where one block per (token, head) would read them tile_q x group size times.
//
//   q, out  [tokens, H, Dh];  k_pool, v_pool [pages, KV, page_size, Dh]
//   sequence b: slot seq_slot[b], new tokens seq_start[b] .. seq_start[b+1]-1 of the packed arrays,
//   length seq_len[b] after the step; new token i sits at position seq_len[b] - n_b + i and sees keys
//   max(0, pos-window+1) .. pos  (window 0: all keys 0..pos) and, beside a window, the sequence's first `keep` keys.
//   kv head = h / (H / KV).
// A page index outside the pool (or -1) among the pages a tile needs: error word 4, the strip is left
// out.  Pages wholly before the first key that the tile sees are not looked up (a window group may have
// given them back).
#include "common.cuh"
#include "distance_bias.cuh"
#include <float.h>
#include <math.h>

#define AR_WARPS 8
#define AR_STRIP 32
#define AR_MAX_DH 640
#define AR_MAX_TILE 16
#define AR_SMEM_BUDGET (200 * 1024)

template <typename T> struct ArVec;                    // four consecutive elements from global memory as floats
template <> struct ArVec<float> {
    static __device__ __forceinline__ float4 load(const float* p) { return *reinterpret_cast<const float4*>(p); }
};
template <> struct ArVec<__nv_bfloat16> {
    static __device__ __forceinline__ float4 load(const __nv_bfloat16* p) {
        const uint2 raw = *reinterpret_cast<const uint2*>(p);
        const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&raw.x);
        const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162*>(&raw.y);
        return make_float4(__low2float(a), __high2float(a), __low2float(b), __high2float(b));
    }
};

__host__ __device__ inline int ar_key_pitch(int Dh, bool vec4) { return vec4 ? Dh + 4 : Dh + 1; }    // floats per staged key

// One strip of keys for R (1, 2 or 4) rows that follow each other in shared memory and see the same keys j_lo .. j_hi of
// the strip, except hole_lo .. hole_hi - 1 (between the kept first keys and the window; a key in the hole has weight 0):
// scores (lane j = key j), the online-softmax update of each row's maximum and sum, and the rows' outputs
// (a lane owns head elements lane, lane + 32, ...; the keys are added in rising order).
template <bool VEC4, int R>
__device__ __forceinline__ void ar_strip(const float* __restrict__ qs, float* __restrict__ accs, float* __restrict__ ms,
                                         float* __restrict__ ls, const float* __restrict__ ks, const float* __restrict__ vs,
                                         int row, int Dh, int kpitch, int j_lo, int j_hi, int hole_lo, int hole_hi, float scale, float softcap, int lane,
                                         const float* __restrict__ bias_row, int bias_len, int distance) {
    // bias_row: the distance bias of the first row's head (the next row's follows it), or null; distance: of key `lane`
    const bool mine = lane >= j_lo && lane <= j_hi && !(lane >= hole_lo && lane < hole_hi);
    float s[R];
#pragma unroll
    for (int r = 0; r < R; r++) s[r] = -INFINITY;
    if (mine) {
        const float* qr = qs + (size_t)row * Dh;
        const float* kr = ks + lane * kpitch;
        float dot[R];
#pragma unroll
        for (int r = 0; r < R; r++) dot[r] = 0.0f;
        if (VEC4) {
            for (int c = 0; c < Dh; c += 4) {
                const float4 k4 = *reinterpret_cast<const float4*>(kr + c);
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const float4 a = *reinterpret_cast<const float4*>(qr + (size_t)r * Dh + c);
                    dot[r] = fmaf(a.x, k4.x, dot[r]);
                    dot[r] = fmaf(a.y, k4.y, dot[r]);
                    dot[r] = fmaf(a.z, k4.z, dot[r]);
                    dot[r] = fmaf(a.w, k4.w, dot[r]);
                }
            }
        } else {
            for (int d = 0; d < Dh; d++) {
                const float kd = kr[d];
#pragma unroll
                for (int r = 0; r < R; r++) dot[r] = fmaf(qr[(size_t)r * Dh + d], kd, dot[r]);
            }
        }
#pragma unroll
        for (int r = 0; r < R; r++) s[r] = dot[r] * scale;
        if (softcap > 0.0f) {
#pragma unroll
            for (int r = 0; r < R; r++) s[r] = softcap * tanhf(s[r] / softcap);
        }
        if (bias_row) {
#pragma unroll
            for (int r = 0; r < R; r++) s[r] += ri_bias_at(bias_row + (size_t)r * ri_bias_pitch(bias_len), bias_len, distance);
        }
    }
    float corr[R], p[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        const float m_old = ms[row + r];
        const float m_new = fmaxf(m_old, warp_max(s[r]));
        corr[r] = expf(m_old - m_new);                            // 0 at the row's first strip (m_old is -inf)
        p[r] = mine ? expf(s[r] - m_new) : 0.0f;
        const float p_sum = warp_sum(p[r]);
        __syncwarp();
        if (lane == 0) {
            ms[row + r] = m_new;
            ls[row + r] = ls[row + r] * corr[r] + p_sum;
        }
    }
    // the outputs: four head elements per lane and row at a time, the strip's keys in rising order
    float* ar = accs + (size_t)row * Dh;
    for (int d0 = 0; d0 < Dh; d0 += 128) {
        float a[R][4];
#pragma unroll
        for (int r = 0; r < R; r++)
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const int d = d0 + c * 32 + lane;
                a[r][c] = d < Dh ? ar[(size_t)r * Dh + d] * corr[r] : 0.0f;
            }
        for (int j = j_lo; j <= j_hi; j++) {
            float pj[R];
#pragma unroll
            for (int r = 0; r < R; r++) pj[r] = __shfl_sync(0xffffffffu, p[r], j);
            const float* vr = vs + j * Dh + d0 + lane;
#pragma unroll
            for (int c = 0; c < 4; c++)
                if (d0 + c * 32 + lane < Dh) {
                    const float v = vr[c * 32];
#pragma unroll
                    for (int r = 0; r < R; r++) a[r][c] = fmaf(pj[r], v, a[r][c]);
                }
        }
#pragma unroll
        for (int r = 0; r < R; r++)
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const int d = d0 + c * 32 + lane;
                if (d < Dh) ar[(size_t)r * Dh + d] = a[r][c];
            }
    }
}

// VEC4: the head size is a multiple of 4 (vector loads, and a staged key's row starts on 16 bytes)
template <typename T, bool VEC4>
__global__ void __launch_bounds__(32 * AR_WARPS)
attention_rows_kernel(const T* __restrict__ q, const T* __restrict__ k_pool, const T* __restrict__ v_pool,
                      T* __restrict__ out, const int* __restrict__ page_table, const int* __restrict__ seq_slot,
                      const int* __restrict__ seq_start, const int* __restrict__ seq_len, int H, int KV, int Dh,
                      int mpps, int page_size, int num_pages, int tile_q, int group_chunk, float scale, int window,
                      int keep, const float* __restrict__ sink, float softcap, DistBias bias, int* __restrict__ err) {
    extern __shared__ __align__(16) float ar_smem[];
    const int b = blockIdx.z;
    const int t_begin = seq_start[b], n_new = seq_start[b + 1] - t_begin;
    const int r_base = blockIdx.x * tile_q;
    if (r_base >= n_new) return;
    const int nq = min(tile_q, n_new - r_base);
    const int G = H / KV, chunks = (G + group_chunk - 1) / group_chunk;
    const int kvh = blockIdx.y / chunks, g0 = (blockIdx.y % chunks) * group_chunk;
    const int ng = min(group_chunk, G - g0);
    const int rows = nq * ng, rows_max = tile_q * group_chunk;
    const int kpitch = ar_key_pitch(Dh, VEC4);
    float* ks = ar_smem;                              // [32][kpitch]
    float* vs = ks + AR_STRIP * kpitch;               // [32][Dh]
    float* qs = vs + AR_STRIP * Dh;                   // [rows][Dh]
    float* accs = qs + (size_t)rows_max * Dh;         // [rows][Dh]
    float* ms = accs + (size_t)rows_max * Dh;         // [rows]
    float* ls = ms + rows_max;                        // [rows]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int len = seq_len[b];
    const int pos0 = len - n_new + r_base, pos_last = pos0 + nq - 1;       // positions of the tile's queries
    const int key_lo = ri_first_visible(pos0, window);
    const int* table = page_table + (size_t)seq_slot[b] * mpps;

    // row = i * ng + g: new token r_base + i, query head kvh * G + g0 + g
    for (int idx = tid; idx < rows * Dh; idx += blockDim.x) {
        const int row = idx / Dh, d = idx - row * Dh;
        const int i = row / ng, g = row - i * ng;
        qs[idx] = ld_f(q + ((size_t)(t_begin + r_base + i) * H + kvh * G + g0 + g) * Dh + d);
        accs[idx] = 0.0f;
    }
    for (int row = tid; row < rows; row += blockDim.x) {
        ms[row] = -INFINITY;
        ls[row] = 0.0f;
    }

    // strips: 32 consecutive keys of one page (the last strip of a page may be shorter), at places that
    // depend on the page size only
    const int window_strip = key_lo - (key_lo % page_size) % AR_STRIP;      // start of the strip that holds key_lo
    int key0 = keep > 0 ? 0 : window_strip;
    while (key0 <= pos_last) {
        if (key0 >= keep && key0 < window_strip) {                    // past the strips of the kept keys
            key0 = window_strip;
            continue;
        }
        const int page_idx = key0 / page_size, in_page = key0 - page_idx * page_size;
        const int width = min(AR_STRIP, page_size - in_page);
        const int page = page_idx < mpps ? table[page_idx] : -1;
        if (page < 0 || page >= num_pages) {
            if (tid == 0) atomicExch(err, 4);
            key0 += width;
            continue;
        }
        __syncthreads();                                              // the strip before has been used (and q, acc are set)
        const size_t base = (((size_t)page * KV + kvh) * page_size + in_page) * Dh;
        if (VEC4) {
            const int per = Dh >> 2;
            for (int idx = tid; idx < width * per; idx += blockDim.x) {
                const int r = idx / per, c = idx - r * per;
                *reinterpret_cast<float4*>(ks + r * kpitch + 4 * c) = ArVec<T>::load(k_pool + base + (size_t)r * Dh + 4 * c);
                *reinterpret_cast<float4*>(vs + r * Dh + 4 * c) = ArVec<T>::load(v_pool + base + (size_t)r * Dh + 4 * c);
            }
        } else {
            for (int idx = tid; idx < width * Dh; idx += blockDim.x) {
                const int r = idx / Dh, d = idx - r * Dh;
                ks[r * kpitch + d] = ld_f(k_pool + base + idx);
                vs[idx] = ld_f(v_pool + base + idx);
            }
        }
        __syncthreads();
        // A warp takes four query heads of one token at a time (they see the same keys), or two where fours would leave warps idle:
        // a key or a value read from shared memory then serves all of them; each row's own arithmetic and its order are
        // what they would be alone
        const int per_unit = nq * ((ng + 3) >> 2) >= AR_WARPS ? 4 : 2;
        const int units = (ng + per_unit - 1) / per_unit;
        for (int unit = warp; unit < nq * units; unit += AR_WARPS) {
            const int i = unit / units, g_first = per_unit * (unit - i * units);
            const int pos = pos0 + i;
            const int first = ri_first_visible(pos, window);
            // the token's keys in this strip: from the window's first one (or, where kept keys are, from the strip's start)
            // to its own; between the kept ones and the window lies a hole
            const int hole_lo = max(keep - key0, 0), hole_hi = first - key0;
            const int j_lo = hole_lo > 0 ? 0 : max(hole_hi, 0);
            int j_hi = min(pos - key0, width - 1);
            if (hole_hi > j_hi) j_hi = min(j_hi, hole_lo - 1);
            if (j_lo > j_hi) continue;                                // none: the rows' state stays as it is
            const int distance = pos - key0 - lane;
            const int g_end = min(g_first + per_unit, ng);
            for (int g = g_first; g < g_end;) {
                const int row_a = i * ng + g;
                const float* bias_row = bias.table ? ri_bias_row(bias, kvh * G + g0 + g) : nullptr;
#define AR_STRIP_GO(R) \
    ar_strip<VEC4, R>(qs, accs, ms, ls, ks, vs, row_a, Dh, kpitch, j_lo, j_hi, hole_lo, hole_hi, scale, softcap, lane, bias_row, \
                      bias.len, distance); \
    g += R
                if (g + 3 < g_end) { AR_STRIP_GO(4); }
                else if (g + 1 < g_end) { AR_STRIP_GO(2); }
                else { AR_STRIP_GO(1); }
#undef AR_STRIP_GO
            }
        }
        key0 += width;
    }
    __syncthreads();
    for (int row = warp; row < rows; row += AR_WARPS) {
        const int i = row / ng, g = row - i * ng;
        float l = ls[row];
        // a sink: one more term exp(sink[head]) in the denominator, with no key and no value (not scaled)
        if (sink && l > 0.0f) l += expf(sink[kvh * G + g0 + g] - ms[row]);
        const float inv = l > 0.0f ? 1.0f / l : 0.0f;                 // no key at all: only after error 4
        T* dst = out + ((size_t)(t_begin + r_base + i) * H + kvh * G + g0 + g) * Dh;
        for (int d = lane; d < Dh; d += 32) st_f(dst + d, accs[(size_t)row * Dh + d] * inv);
    }
}

// The same rows, the same arithmetic and order of every row, for float32 steps of more than a few rows: a block takes AT_ROWS rows of one kv head
// (tile_q tokens of all its query heads) and walks the strips with the scores and the outputs in registers, four rows of two keys and four
// rows of DH / 16 elements a thread.  What bounds it: the words that come from shared memory, 32 a cycle for an SM whether the lanes of a warp want
// the same ones or not: 0.75 words a multiply-add of the scores and 0.375 of the outputs, where a lane with one key and four rows takes 1.25 for
// either; for few blocks the chain of a strip.  The next strip's keys are copied under the softmax and the outputs, its values under the scores.
// Cold, us, this / a row at a time, heads over kv heads of size: 32 / 8 of 128, 512 tokens 141 / 283, 32 behind 300 64 / 160, 8 sequences of one token
// behind 300 57 / 60; 16 / 2 of 64, 300 tokens 45 / 176; 16 / 1 of 256, 300 tokens 92 / 256.  Tiles of 64 rows (0.5 and 0.25 words) leave two blocks
// to an SM and take 172, 96, 84; 62; 141.
#define AT_ROWS 32
#define AT_MIN_ROWS 10             // ... and with fewer rows, down to eight, from AT_MIN_WORK elements of queries on
#define AT_MIN_WORK 65536
#define AT_THREADS 128
#define AT_P_PITCH 36
template <bool V> struct AtFlag { static constexpr bool value = V; };
template <int DH>
constexpr int at_smem_floats() { return AT_ROWS * (DH + 4) + AR_STRIP * (DH + 4) + AR_STRIP * DH + AT_ROWS * AT_P_PITCH + 2 * AT_ROWS; }

__device__ __forceinline__ void at_copy16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void at_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void at_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

template <int DH>
__global__ void __launch_bounds__(AT_THREADS, DH <= 128 ? 4 : 2)
attention_tile_kernel(const float* __restrict__ q, const float* __restrict__ k_pool, const float* __restrict__ v_pool, float* __restrict__ out,
                      const int* __restrict__ page_table, const int* __restrict__ seq_slot, const int* __restrict__ seq_start,
                      const int* __restrict__ seq_len, int H, int KV, int mpps, int page_size, int num_pages, int tile_q, float scale, int window,
                      int keep, const float* __restrict__ sink, float softcap, DistBias bias, int* __restrict__ err) {
    constexpr int PITCH = DH + 4, DC = DH / 64;                   // DC pieces of four elements a thread
    constexpr int LANES = 16, KEYS = 2, PR = 4;                   // lanes that share four rows, keys of each; rows of outputs
    static_assert(AT_ROWS * LANES == 4 * AT_THREADS && LANES * KEYS == AR_STRIP && 8 * PR == AT_ROWS, "the threads cover the tile");
    extern __shared__ __align__(16) float ar_smem[];
    const int b = blockIdx.z, kvh = blockIdx.y;
    const int t_begin = seq_start[b], n_new = seq_start[b + 1] - t_begin;
    const int r_base = (gridDim.x - 1 - blockIdx.x) * tile_q;     // the longest walks first
    if (r_base >= n_new) return;
    const int nq = min(tile_q, n_new - r_base), G = H / KV, rows = nq * G;
    float* qs = ar_smem;                                          // [AT_ROWS][PITCH]
    float* ks = qs + AT_ROWS * PITCH;                             // [32][PITCH]
    float* vs = ks + AR_STRIP * PITCH;                            // [32][DH]
    float* ps = vs + AR_STRIP * DH;                               // [AT_ROWS][AT_P_PITCH]
    float* s_corr = ps + AT_ROWS * AT_P_PITCH;                    // [AT_ROWS], at the end the rows' factors
    unsigned* s_mask = reinterpret_cast<unsigned*>(s_corr + AT_ROWS);
    const int tid = threadIdx.x;
    const int len = seq_len[b];
    const int pos0 = len - n_new + r_base, pos_last = pos0 + nq - 1;       // positions of the tile's queries
    const int key_lo = ri_first_visible(pos0, window);
    const int* table = page_table + (size_t)seq_slot[b] * mpps;
    for (int i = tid; i < AT_ROWS * (DH / 4); i += AT_THREADS) {
        const int row = i / (DH / 4), c = (i % (DH / 4)) * 4, tok = row / G;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (row < rows) v = *reinterpret_cast<const float4*>(q + ((size_t)(t_begin + r_base + tok) * H + kvh * G + row - tok * G) * DH + c);
        *reinterpret_cast<float4*>(qs + row * PITCH + c) = v;
    }
    // strips of 32 keys, whole ones: pages hold a multiple of 32
    const int window_strip = key_lo - (key_lo % page_size) % AR_STRIP;      // start of the strip that holds key_lo
    auto next = [&](int& key0) -> long long {                     // the first strip from key0 on that has a page: its elements' place, or -1
        while (key0 <= pos_last) {
            if (key0 >= keep && key0 < window_strip) {            // past the strips of the kept keys
                key0 = window_strip;
                continue;
            }
            const int page_idx = key0 / page_size;
            const int page = page_idx < mpps ? table[page_idx] : -1;
            if (page >= 0 && page < num_pages) return (((long long)page * KV + kvh) * page_size + key0 - page_idx * page_size) * DH;
            if (tid == 0) atomicExch(err, 4);
            key0 += AR_STRIP;
        }
        return -1;
    };
    auto copy_k = [&](long long at) {
        if (at >= 0)
            for (int i = tid; i < AR_STRIP * (DH / 4); i += AT_THREADS) at_copy16(ks + i / (DH / 4) * PITCH + (i % (DH / 4)) * 4, k_pool + at + (size_t)i * 4);
        at_commit();
    };
    auto copy_v = [&](long long at) {
        if (at >= 0)
            for (int i = tid; i < AR_STRIP * (DH / 4); i += AT_THREADS) at_copy16(vs + i * 4, v_pool + at + (size_t)i * 4);
        at_commit();
    };
    // scores: rows 4 ty .., keys tx, tx + LANES, ..;  outputs: rows PR ry .., elements 4 rx + 64 c ..
    const int ty = tid / LANES, tx = tid % LANES, ry = tid >> 4, rx = tid & 15;
    float m[4], l[4];
    int pos[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        m[i] = -INFINITY;
        l[i] = 0.0f;
        pos[i] = 4 * ty + i < rows ? pos0 + (4 * ty + i) / G : -1;      // -1: no such row, it sees nothing
    }
    float o[PR][DC][4];
#pragma unroll
    for (int r = 0; r < PR; r++)
#pragma unroll
        for (int c = 0; c < DC; c++)
#pragma unroll
            for (int e = 0; e < 4; e++) o[r][c][e] = 0.0f;
    int key0 = keep > 0 ? 0 : window_strip;
    long long at = next(key0);
    copy_k(at);
    copy_v(at);
    while (at >= 0) {
        int key1 = key0 + AR_STRIP;
        const long long at1 = next(key1);
        at_wait<1>();                                             // the keys
        __syncthreads();
        float s[4][KEYS];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < KEYS; j++) s[i][j] = 0.0f;
#pragma unroll 4
        for (int d = 0; d < DH; d += 4) {
            float4 a[4], k[KEYS];
#pragma unroll
            for (int i = 0; i < 4; i++) a[i] = *reinterpret_cast<const float4*>(qs + (4 * ty + i) * PITCH + d);
#pragma unroll
            for (int j = 0; j < KEYS; j++) k[j] = *reinterpret_cast<const float4*>(ks + (tx + LANES * j) * PITCH + d);
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < KEYS; j++) {
                    s[i][j] = fmaf(a[i].x, k[j].x, s[i][j]);
                    s[i][j] = fmaf(a[i].y, k[j].y, s[i][j]);
                    s[i][j] = fmaf(a[i].z, k[j].z, s[i][j]);
                    s[i][j] = fmaf(a[i].w, k[j].w, s[i][j]);
                }
        }
        __syncthreads();                                          // the keys were read, the weights of the strip before too
        copy_k(at1);
        const bool all = key0 + AR_STRIP - 1 <= pos0 && key0 >= ri_first_visible(pos_last, window);      // every row sees every key
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int row = 4 * ty + i;
            const int first = ri_first_visible(max(pos[i], 0), window);
            // the row's keys in this strip, as for a row alone
            const int hole_lo = max(keep - key0, 0), hole_hi = first - key0;
            const int j_lo = hole_lo > 0 ? 0 : max(hole_hi, 0);
            int j_hi = min(pos[i] - key0, AR_STRIP - 1);
            if (hole_hi > j_hi) j_hi = min(j_hi, hole_lo - 1);
            const bool any = pos[i] >= 0 && j_lo <= j_hi;
            const float* bias_row = bias.table && any ? ri_bias_row(bias, kvh * G + row % G) : nullptr;
            bool mine[KEYS];
            float most = -INFINITY;
#pragma unroll
            for (int j = 0; j < KEYS; j++) {
                const int key = tx + LANES * j;
                mine[j] = any && key >= j_lo && key <= j_hi && !(key >= hole_lo && key < hole_hi);
                float v = s[i][j] * scale;
                if (softcap > 0.0f) v = softcap * tanhf(v / softcap);
                if (bias_row && mine[j]) v += ri_bias_at(bias_row, bias.len, pos[i] - key0 - key);
                s[i][j] = mine[j] ? v : -INFINITY;
                most = fmaxf(most, s[i][j]);
            }
#pragma unroll
            for (int w = LANES / 2; w > 0; w >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, w));
            const float m_new = fmaxf(m[i], most);
            const float corr = any ? expf(m[i] - m_new) : 1.0f;
            float p[KEYS];
#pragma unroll
            for (int j = 0; j < KEYS; j++) p[j] = mine[j] ? expf(s[i][j] - m_new) : 0.0f;
            float sum = p[0] + p[1];                              // the tree of a warp with a key a lane: sixteen apart, eight, four ..
#pragma unroll
            for (int w = LANES / 2; w > 0; w >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, w);
            if (any) {
                l[i] = l[i] * corr + sum;
                m[i] = m_new;
            }
#pragma unroll
            for (int j = 0; j < KEYS; j++) ps[row * AT_P_PITCH + tx + LANES * j] = p[j];
            if (tx == 0) {
                s_corr[row] = corr;
                s_mask[row] = any ? (0xffffffffu >> (31 - j_hi)) & (0xffffffffu << j_lo) : 0u;
            }
        }
        at_wait<1>();                                             // the values
        __syncthreads();
        unsigned mask[PR];
#pragma unroll
        for (int r = 0; r < PR; r++) {
            const float corr = s_corr[PR * ry + r];
            mask[r] = s_mask[PR * ry + r];
#pragma unroll
            for (int c = 0; c < DC; c++)
#pragma unroll
                for (int e = 0; e < 4; e++) o[r][c][e] *= corr;
        }
        auto outputs = [&](auto every) {                          // every: all rows see all keys (a key that a row does not see may hold anything)
#pragma unroll 2
            for (int j0 = 0; j0 < AR_STRIP; j0 += 4) {
                float p[PR][4];
#pragma unroll
                for (int r = 0; r < PR; r++) *reinterpret_cast<float4*>(p[r]) = *reinterpret_cast<const float4*>(ps + (PR * ry + r) * AT_P_PITCH + j0);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    float v[DC][4];
#pragma unroll
                    for (int c = 0; c < DC; c++) *reinterpret_cast<float4*>(v[c]) = *reinterpret_cast<const float4*>(vs + (j0 + j) * DH + 64 * c + 4 * rx);
#pragma unroll
                    for (int r = 0; r < PR; r++) {
                        if (!decltype(every)::value && !((mask[r] >> (j0 + j)) & 1u)) continue;
#pragma unroll
                        for (int c = 0; c < DC; c++)
#pragma unroll
                            for (int e = 0; e < 4; e++) o[r][c][e] = fmaf(p[r][j], v[c][e], o[r][c][e]);
                    }
                }
            }
        };
        if (all) outputs(AtFlag<true>());
        else outputs(AtFlag<false>());
        __syncthreads();                                          // the values were read
        copy_v(at1);
        key0 = key1;
        at = at1;
    }
    at_wait<0>();
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int row = 4 * ty + i;
        // a sink: one more term exp(sink[head]) in the denominator, with no key and no value (not scaled)
        if (sink && l[i] > 0.0f) l[i] += expf(sink[kvh * G + row % G] - m[i]);
        if (tx == 0) s_corr[row] = l[i] > 0.0f ? 1.0f / l[i] : 0.0f;      // no key at all: only after error 4
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < PR; r++) {
        const int row = PR * ry + r, tok = row / G;
        if (row >= rows) break;
        const float inv = s_corr[row];
        float* dst = out + ((size_t)(t_begin + r_base + tok) * H + kvh * G + row - tok * G) * DH + 4 * rx;
#pragma unroll
        for (int c = 0; c < DC; c++)
            *reinterpret_cast<float4*>(dst + 64 * c) = make_float4(o[r][c][0] * inv, o[r][c][1] * inv, o[r][c][2] * inv, o[r][c][3] * inv);
    }
}

// how a launch is cut: rows per block from the shared memory that the staged strip leaves
static void ar_geometry(int G, int Dh, int max_new, bool vec4, int* tile_q, int* group_chunk, size_t* smem) {
    const size_t strip = (size_t)AR_STRIP * (ar_key_pitch(Dh, vec4) + Dh) * sizeof(float);
    const size_t per_row = (size_t)(2 * Dh + 2) * sizeof(float);
    int rows_max = (int)((AR_SMEM_BUDGET - strip) / per_row);          // at least 7 (head size 640)
    int gc = G < rows_max ? G : rows_max;
    int tq = rows_max / gc;
    tq = tq > AR_MAX_TILE ? AR_MAX_TILE : tq;
    tq = tq > max_new ? max_new : tq;
    tq = tq < 1 ? 1 : tq;
    *tile_q = tq;
    *group_chunk = gc;
    *smem = strip + (size_t)tq * gc * per_row;
}

template <typename T, bool VEC4>
static int ar_launch(const void* q, const void* k_pool, const void* v_pool, void* out, const int* page_table,
                     const int* seq_slot, const int* seq_start, const int* seq_len, int seqs, int max_new, int H, int KV,
                     int Dh, int mpps, int page_size, int num_pages, float scale, int window, int keep, const float* sink,
                     float softcap, DistBias bias, int* err_flag, cudaStream_t stream) {
    int tile_q, group_chunk;
    size_t smem;
    const int G = H / KV;
    ar_geometry(G, Dh, max_new, VEC4, &tile_q, &group_chunk, &smem);
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(attention_rows_kernel<T, VEC4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             AR_SMEM_BUDGET + 1024);
        if (e != cudaSuccess) RI_FAIL((int)e, "attention_rows: shared memory limit: %s", cudaGetErrorString(e));
        configured = true;
    }
    const long long gy = (long long)KV * ((G + group_chunk - 1) / group_chunk);
    RI_REQUIRE(gy <= 65535 && seqs <= 65535, "attention_rows: %d heads, %d sequences: too many for one launch", H, seqs);
    dim3 grid((max_new + tile_q - 1) / tile_q, (unsigned)gy, seqs);
    attention_rows_kernel<T, VEC4><<<grid, 32 * AR_WARPS, smem, stream>>>(
        (const T*)q, (const T*)k_pool, (const T*)v_pool, (T*)out, page_table, seq_slot, seq_start, seq_len, H, KV, Dh, mpps,
        page_size, num_pages, tile_q, group_chunk, scale, window, keep, sink, softcap, bias, err_flag);
    RI_CHECK_LAUNCH("attention_rows");
    return 0;
}

template <int DH>
static int at_launch(const void* q, const void* k_pool, const void* v_pool, void* out, const int* page_table, const int* seq_slot,
                     const int* seq_start, const int* seq_len, int seqs, int max_new, int H, int KV, int mpps, int page_size, int num_pages,
                     float scale, int window, int keep, const float* sink, float softcap, DistBias bias, int* err_flag, cudaStream_t stream) {
    constexpr int smem = at_smem_floats<DH>() * (int)sizeof(float);
    cudaError_t e = cudaFuncSetAttribute(attention_tile_kernel<DH>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) RI_FAIL((int)e, "attention_rows: shared memory limit: %s", cudaGetErrorString(e));
    const int tile_q = AT_ROWS / (H / KV);
    attention_tile_kernel<DH><<<dim3((max_new + tile_q - 1) / tile_q, KV, seqs), AT_THREADS, smem, stream>>>(
        (const float*)q, (const float*)k_pool, (const float*)v_pool, (float*)out, page_table, seq_slot, seq_start, seq_len, H, KV, mpps, page_size,
        num_pages, tile_q, scale, window, keep, sink, softcap, bias, err_flag);
    RI_CHECK_LAUNCH("attention_tile");
    return 0;
}

// q, out [tokens, H, Dh]; max_new = the most tokens one sequence brings in this step
// sink [H] float32 or null: a learned term per head that joins the softmax's denominator only
// softcap > 0: score <- softcap * tanh(score / softcap) after the scale (0: none)
// dist_bias (float32, bias_len entries a head between their padding) or null: added to the score by the query's distance to the key (distance_bias.cuh)
extern "C" int ri_attention_rows(const void* q, const void* k_pool, const void* v_pool, void* out, const int* page_table,
                                 const int* seq_slot, const int* seq_start, const int* seq_len, int seqs, int max_new,
                                 int H, int KV, int Dh, int mpps, int page_size, int num_pages, float scale, int window,
                                 const float* sink, float softcap, const float* dist_bias, int bias_len, int keep, int dtype,
                                 int* err_flag, cudaStream_t stream) {
    if (seqs == 0 || max_new == 0) return 0;
    RI_REQUIRE(keep >= 0, "attention_rows: %d kept keys", keep);
    if (window <= 0) keep = 0;                 // nothing is out of sight, or the mask is one of chunks
    RI_REQUIRE(seqs > 0 && max_new > 0 && H > 0 && KV > 0 && Dh > 0 && page_size > 0 && mpps > 0, "attention_rows: bad sizes");
    RI_REQUIRE(H % KV == 0, "attention_rows: %d heads are not a multiple of %d kv heads", H, KV);
    RI_REQUIRE(Dh <= AR_MAX_DH, "attention_rows: head_dim %d exceeds the limit %d", Dh, AR_MAX_DH);
    RI_REQUIRE(!dist_bias || bias_len > 0, "attention_rows: a distance bias needs its length");
    const DistBias bias{dist_bias, bias_len};
    const bool f32 = dtype == RI_DTYPE_F32;
    RI_REQUIRE(f32 || dtype == RI_DTYPE_BF16, "attention_rows: unknown dtype %d", dtype);
    // vector loads need rows of the pools and of q that start on 16 bytes (float32) or 8 bytes (bfloat16)
    const uintptr_t align = f32 ? 15 : 7;
    const bool vec4 = Dh % 4 == 0 && (((uintptr_t)q | (uintptr_t)k_pool | (uintptr_t)v_pool) & align) == 0;
    // Tiles of rows (the same bits) from ten rows a kv head on, from eight where the blocks are many: a row at a time is the shorter chain, but takes
    // more words from shared memory a row.  Pools from memory, behind 300 keys, tiles / a row at a time, us: eight rows of 8 kv heads of 128 50 / 42, of 64
    // 50 / 46, of 192 68 / 66, of 768 166 / 205, of 48 of 256 elements 78 / 99; ten rows of 8 kv heads of 64 38 / 49, of 128 (five query heads each)
    // 50 / 47, of 192 68 / 74; 16 rows of 8 kv heads of 128 50 / 51, of 192 70 / 84.  Behind a few keys only the chain counts: 12 rows behind none 9.7 / 7.9,
    // 16 9.7 / 8.9, 24 10.2 / 12.1.
    const long long rows = (long long)max_new * (H / KV);
    const bool many = rows >= AT_MIN_ROWS || (rows >= 8 && rows * KV * seqs * Dh >= AT_MIN_WORK);
    if (f32 && vec4 && ((uintptr_t)out & 15) == 0 && page_size % AR_STRIP == 0 && H / KV <= AT_ROWS && many && KV <= 65535 && seqs <= 65535) {
#define AT_GO(D) at_launch<D>(q, k_pool, v_pool, out, page_table, seq_slot, seq_start, seq_len, seqs, max_new, H, KV, mpps, page_size, num_pages, \
                              scale, window, keep, sink, softcap, bias, err_flag, stream)
        if (Dh == 64) return AT_GO(64);
        if (Dh == 128) return AT_GO(128);
        if (Dh == 256) return AT_GO(256);
#undef AT_GO
    }
#define AR_GO(T, V) ar_launch<T, V>(q, k_pool, v_pool, out, page_table, seq_slot, seq_start, seq_len, seqs, max_new, H, KV, \
                                    Dh, mpps, page_size, num_pages, scale, window, keep, sink, softcap, bias, err_flag, stream)
    if (f32) return vec4 ? AR_GO(float, true) : AR_GO(float, false);
    return vec4 ? AR_GO(__nv_bfloat16, true) : AR_GO(__nv_bfloat16, false);
#undef AR_GO
}
