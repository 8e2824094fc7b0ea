// A routed feed-forward (mixture of experts): router, plan of the step, grouped products, combination.
//
// `moe_route`   per token: logits z = R x (float32), scores s = softmax(z) over all N outputs of the router (or the
//               sigmoid of each), choice scores s + correction, optionally only within the best groups of neighbouring
//               outputs (`MoeRule`), the `top` largest of them (ties: the lower index), and as weights the chosen
//               outputs' scores s divided by their sum (+ 1e-20) or as they are, times a constant.  Or the choice is by
//               the logits themselves and the weights are the softmax over the chosen ones alone.  The logits may have a
//               bias.  Every sum has a fixed order.
// `moe_plan`    the step's (token, choice) pairs grouped by expert: `perm` lists the pairs of expert 0, then of expert
//               1 and so on (pairs whose choice is not one of the first E outputs, identity experts, are left out), and
//               `tiles` cuts every expert's run into tiles of MOE_BM rows: (expert, first row in perm, rows).  One
//               block; which pair lands where inside an expert's run is not fixed, and no result depends on it: a
//               row of a product is computed alone.
// `moe_grouped_linear`  y[out(r), :] = W[e] a[in(r), :] for every row r of every tile, W [E, N, K]; in(r) = perm[r] /
//               div (gather: a token's row for each of its pairs) or r, out(r) = perm[r] (scatter: back to the pair's
//               own place) or r.  float32: FMA tiles, k ascending in one accumulator per output; bfloat16: mma.sync
//               m16n8k16 with float32 accumulators (steps with many pairs per expert: moe_tc.cu).  The grid covers the most tiles a step can have; blocks past the
//               plan's count leave at once (the count stays on the device: no trip to the host, and the step can be
//               replayed from a graph).
// `moe_combine` y[t] = sum_j w[t, j] (choice j an identity expert ? x[t] : pair_out[t top + j]) (+ extra[t]),
//               j ascending, float32, rounded once.
// Without a router, a table names every token id's experts (`ri_moe_plan_table`) and the weights are equal.
#include "common.cuh"
#include "mma_helpers.cuh"

#define MOE_BM 32
#define MOE_BM_WIDE 256              // tiles for moe_tc.cu
#define MOE_BN 64
#define MOE_ROUTE_WARPS 4

// A warp per token.  The logits are taken four router outputs at a time: a lane walks its own k (four neighbouring ones
// per trip with 16-byte loads where the rows allow it, else one) and keeps four sums, so that twenty loads are on their
// way together; a sum's order depends on the row's size alone.  Then the warp does the softmax and the choice.
__device__ __forceinline__ float4 moe_ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 moe_ld4(const bf16* p) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&u.x), b = *reinterpret_cast<const __nv_bfloat162*>(&u.y);
    return make_float4(__low2float(a), __high2float(a), __low2float(b), __high2float(b));
}

__device__ __forceinline__ void moe_st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void moe_st4(bf16* p, float4 v) {
    *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
}

// How scores become a choice and weights.  mode 0: scores are the softmax over all outputs; mode 1: the sigmoid of every
// output on its own; mode 2: the logits themselves, without a correction, and the weights are the softmax over the chosen
// outputs alone (times `scale`).  `bias` [N] (or null) is added to the logits first.  Choice scores are the scores plus the correction.  groups > 1: the outputs form `groups` equal runs
// of neighbours, a run's score is the sum of its `gtop` largest choice scores, and only the outputs of the `keep` best
// runs can be chosen (ties: the lower index, for runs as for outputs).  The weights are the chosen outputs' scores
// (without the correction) times `scale`, divided by their sum first when `renorm` is set.
struct MoeRule {
    int mode, groups, keep, gtop, renorm;
    float scale;
    const float* bias;
};

// One warp: s [N] holds the logits on entry, c [N] and gs [groups] are scratch.
__device__ __forceinline__ void moe_choose(float* s, float* c, float* gs, const float* __restrict__ correction,
                                           int* __restrict__ idx, float* __restrict__ weight, int t, int N, int top, int lane,
                                           const MoeRule rule) {
    if (rule.bias) {
        for (int n = lane; n < N; n += 32) s[n] += rule.bias[n];
        __syncwarp();
    }
    if (rule.mode == 2) {
        for (int n = lane; n < N; n += 32) c[n] = s[n];
    } else if (rule.mode == 0) {
        float mx = -INFINITY;
        for (int n = lane; n < N; n += 32) mx = fmaxf(mx, s[n]);
        mx = warp_max(mx);
        float sum = 0.0f;
        for (int n = lane; n < N; n += 32) {
            const float e = expf(s[n] - mx);
            s[n] = e;
            sum += e;
        }
        sum = warp_sum(sum);
        for (int n = lane; n < N; n += 32) {
            s[n] = s[n] / sum;
            c[n] = s[n] + correction[n];
        }
    } else {
        for (int n = lane; n < N; n += 32) {
            s[n] = 1.0f / (1.0f + expf(-s[n]));
            c[n] = s[n] + correction[n];
        }
    }
    __syncwarp();
    if (rule.groups > 1) {
        const int size = N / rule.groups;
        for (int g = lane; g < rule.groups; g += 32) {
            // the gtop largest of the run, one after the other in the order (value descending, index ascending)
            float total = 0.0f, last = INFINITY;
            int last_at = -1;
            for (int r = 0; r < rule.gtop && r < size; r++) {
                float best = -INFINITY;
                int at = -1;
                for (int n = 0; n < size; n++) {
                    const float v = c[g * size + n];
                    const bool after = v < last || (v == last && n > last_at);
                    if (after && (at < 0 || v > best)) {
                        best = v;
                        at = n;
                    }
                }
                if (at < 0) break;
                total += best;
                last = best;
                last_at = at;
            }
            gs[g] = total;
        }
        __syncwarp();
        if (lane == 0) {
            for (int r = 0; r < rule.keep; r++) {
                float best = -INFINITY;
                int at = -1;
                for (int g = 0; g < rule.groups; g++)
                    if (gs[g] != INFINITY && (at < 0 || gs[g] > best)) {
                        best = gs[g];
                        at = g;
                    }
                if (at >= 0) gs[at] = INFINITY;           // kept
            }
        }
        __syncwarp();
        for (int n = lane; n < N; n += 32)
            if (gs[n / size] != INFINITY) c[n] = -INFINITY;
        __syncwarp();
    }
    float picked_sum = 0.0f, mine = 0.0f;                 // mine: lane j's is the j-th choice's score (of up to 32)
    for (int j = 0; j < top; j++) {
        float best = -INFINITY;
        int at = 0x7fffffff;
        for (int n = lane; n < N; n += 32)
            if (c[n] > best) {                        // ascending n: the first of equals stays
                best = c[n];
                at = n;
            }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oa = __shfl_xor_sync(0xffffffffu, at, o);
            if (ob > best || (ob == best && oa < at)) {
                best = ob;
                at = oa;
            }
        }
        if (at >= N) at = 0;                           // no finite score left (NaN inputs): still a valid index
        const float picked = s[at];
        if (lane == 0) {
            idx[(size_t)t * top + j] = at;
            if (top > 32) weight[(size_t)t * top + j] = picked;
            c[at] = -INFINITY;
        }
        if (lane == j) mine = picked;
        picked_sum += picked;
        __syncwarp();
    }
    if (top <= 32) {                                      // (more choices than lanes: from memory, below)
        float div = rule.renorm ? picked_sum + 1e-20f : 1.0f;
        if (rule.mode == 2) {
            // the first choice has the largest logit
            mine = expf(mine - __shfl_sync(0xffffffffu, mine, 0));
            div = 0.0f;
            for (int j = 0; j < top; j++) div += __shfl_sync(0xffffffffu, mine, j);
        }
        if (lane < top) weight[(size_t)t * top + lane] = mine / div * rule.scale;
    } else if (lane == 0 && rule.mode == 2) {
        // the first choice has the largest logit
        float* w = weight + (size_t)t * top;
        const float mx = w[0];
        float sum = 0.0f;
        for (int j = 0; j < top; j++) {
            w[j] = expf(w[j] - mx);
            sum += w[j];
        }
        for (int j = 0; j < top; j++) w[j] = w[j] / sum * rule.scale;
    } else if (lane == 0) {
        const float div = rule.renorm ? picked_sum + 1e-20f : 1.0f;
        for (int j = 0; j < top; j++) weight[(size_t)t * top + j] = weight[(size_t)t * top + j] / div * rule.scale;
    }
}

template <typename T>
__global__ void __launch_bounds__(32 * MOE_ROUTE_WARPS)
moe_route_kernel(const T* __restrict__ x, const float* __restrict__ router, const float* __restrict__ correction,
                 int* __restrict__ idx, float* __restrict__ weight, int tokens, int D, int N, int top, int vec, MoeRule rule) {
    extern __shared__ float moe_sm[];                 // per warp: scores [N], choice scores [N], runs' scores [groups]
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t = blockIdx.x * MOE_ROUTE_WARPS + warp;
    if (t >= tokens) return;
    float* s = moe_sm + (size_t)warp * (2 * N + rule.groups);
    float* c = s + N;
    const T* xr = x + (size_t)t * D;
    for (int n0 = 0; n0 < N; n0 += 4) {
        const float* w[4];
#pragma unroll
        for (int j = 0; j < 4; j++) w[j] = router + (size_t)min(n0 + j, N - 1) * D;     // past the last output: its sum is dropped
        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (vec) {
            // four trips' loads (twenty of them) are issued before the first product needs one: the loop is written out so
            const float4 zero4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            for (int k0 = 4 * lane; k0 < D; k0 += 4 * 128) {
                float4 xv[4], wv[4][4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int k = k0 + 128 * u;
                    const bool ok = k < D;
                    xv[u] = ok ? moe_ld4(xr + k) : zero4;
#pragma unroll
                    for (int j = 0; j < 4; j++) wv[u][j] = ok ? *reinterpret_cast<const float4*>(w[j] + k) : zero4;
                }
#pragma unroll
                for (int u = 0; u < 4; u++)
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        acc[j] = fmaf(xv[u].x, wv[u][j].x, acc[j]);
                        acc[j] = fmaf(xv[u].y, wv[u][j].y, acc[j]);
                        acc[j] = fmaf(xv[u].z, wv[u][j].z, acc[j]);
                        acc[j] = fmaf(xv[u].w, wv[u][j].w, acc[j]);
                    }
            }
        } else {
#pragma unroll 4
            for (int k = lane; k < D; k += 32) {
                const float xv = ld_f(xr + k);
#pragma unroll
                for (int j = 0; j < 4; j++) acc[j] = fmaf(xv, w[j][k], acc[j]);
            }
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float v = warp_sum(acc[j]);
            if (lane == 0 && n0 + j < N) s[n0 + j] = v;
        }
    }
    __syncwarp();
    moe_choose(s, c, c + N, correction, idx, weight, t, N, top, lane, rule);
}

// The same with a block of 1,024 threads per token, for routers small enough that all their partial sums fit in shared
// memory: a warp takes (output, run of MOE_ROUTE_RUN segments of 128 k) items, so the whole router is asked for at once instead of row after
// row (one trip to memory instead of dozens: the warp-per-token form took 75 us whatever the number of tokens); a lane adds up
// its four k of every segment of a run, the run's sum is the warp's tree, an output's logit the sum of its runs in ascending order.
#define MOE_ROUTE_RUN 4
#define MOE_ROUTE_WIDE_THREADS 1024
#define MOE_ROUTE_WIDE_ITEMS 8192
#define MOE_ROUTE_AHEAD 2
template <typename T>
__global__ void __launch_bounds__(MOE_ROUTE_WIDE_THREADS)
moe_route_wide_kernel(const T* __restrict__ x, const float* __restrict__ router, const float* __restrict__ correction,
                      int* __restrict__ idx, float* __restrict__ weight, int D, int N, int top, MoeRule rule) {
    extern __shared__ float moe_sm[];                 // partial sums [N][segs], scores [N], choice scores [N], runs' scores
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t = blockIdx.x;
    const int runs = (D + 128 * MOE_ROUTE_RUN - 1) / (128 * MOE_ROUTE_RUN);
    float* part = moe_sm;
    float* s = part + (size_t)N * runs;
    float* c = s + N;
    const T* xr = x + (size_t)t * D;
    const float4 zero4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    // MOE_ROUTE_AHEAD items' loads are on their way together
    constexpr int WARPS = MOE_ROUTE_WIDE_THREADS / 32;
    for (int item0 = warp; item0 < N * runs; item0 += WARPS * MOE_ROUTE_AHEAD) {
        float4 xv[MOE_ROUTE_AHEAD][MOE_ROUTE_RUN], wv[MOE_ROUTE_AHEAD][MOE_ROUTE_RUN];
#pragma unroll
        for (int u = 0; u < MOE_ROUTE_AHEAD; u++) {
            const int item = min(item0 + u * WARPS, N * runs - 1), n = item / runs, k0 = (item - n * runs) * 128 * MOE_ROUTE_RUN + 4 * lane;
#pragma unroll
            for (int i = 0; i < MOE_ROUTE_RUN; i++) {
                const int k = k0 + 128 * i;
                xv[u][i] = k < D ? moe_ld4(xr + k) : zero4;
                wv[u][i] = k < D ? *reinterpret_cast<const float4*>(router + (size_t)n * D + k) : zero4;
            }
        }
#pragma unroll
        for (int u = 0; u < MOE_ROUTE_AHEAD; u++) {
            const int item = item0 + u * WARPS;
            float a = 0.0f;
#pragma unroll
            for (int i = 0; i < MOE_ROUTE_RUN; i++) {
                a = fmaf(xv[u][i].x, wv[u][i].x, a);
                a = fmaf(xv[u][i].y, wv[u][i].y, a);
                a = fmaf(xv[u][i].z, wv[u][i].z, a);
                a = fmaf(xv[u][i].w, wv[u][i].w, a);
            }
            a = warp_sum(a);
            if (lane == 0 && item < N * runs) part[item] = a;
        }
    }
    __syncthreads();
    for (int n = threadIdx.x; n < N; n += MOE_ROUTE_WIDE_THREADS) {
        float a = 0.0f;
        for (int g = 0; g < runs; g++) a += part[n * runs + g];
        s[n] = a;
    }
    __syncthreads();
    if (warp > 0) return;
    moe_choose(s, c, c + N, correction, idx, weight, t, N, top, lane, rule);
}

// The same for many tokens: a block takes MOE_ROUTE_TILE tokens, so that a piece of the router that a warp has loaded serves
// all of them (a block per token reads the whole router from L2 for every token).  What bounds it: the router's way from L2, the
// multiply-adds and the trees, and for few blocks the trips to memory, one for each item of a warp.  A warp takes a run for four outputs, its
// loads on their way together, and keeps the 16 sums of four tokens and four outputs in registers; they go down the warp's tree side by side,
// every step halving the number of values a lane still holds, so that lanes 2 i and 2 i + 1 end with the sum of token i / 4 and output i % 4.  The
// additions of a sum and their order are those of the kernel above: the same bits.
// Cold, width 4,096 and 18 outputs, 256 / 512 / 2,048 tokens: 16.6 / 18.4 / 35 us; with a tree for every segment of 128 k 23.5 / 23.6 / 53.
// (Eight tokens and eight outputs a warp's item, a segment at a time: 26.7 / 28.6 / 35.5.)
#define MOE_ROUTE_TILE 4
#define MOE_ROUTE_TILE_THREADS 256
template <typename T> struct MoePiece;                // four neighbouring elements as they come from memory
template <> struct MoePiece<float> {
    float4 v;
    __device__ __forceinline__ void load(const float* p) { v = moe_ld4(p); }
    __device__ __forceinline__ float4 value() const { return v; }
};
template <> struct MoePiece<bf16> {
    uint2 v;
    __device__ __forceinline__ void load(const bf16* p) { v = *reinterpret_cast<const uint2*>(p); }
    __device__ __forceinline__ float4 value() const {
        return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
    }
};
template <typename T>
__global__ void __launch_bounds__(MOE_ROUTE_TILE_THREADS, 2)
moe_route_tile_kernel(const T* x, const float* __restrict__ router, const float* __restrict__ correction, int* __restrict__ idx,
                      float* __restrict__ weight, int tokens, int D, int N, int top, MoeRule rule) {
    extern __shared__ float moe_sm[];                 // partial sums [runs][TILE][N4], per token: scores, choice scores, groups' scores
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t0 = blockIdx.x * MOE_ROUTE_TILE;
    const int runs = (D + 128 * MOE_ROUTE_RUN - 1) / (128 * MOE_ROUTE_RUN), quads = (N + 3) / 4, N4 = 4 * quads;
    float* part = moe_sm;
    float* scores = part + (size_t)runs * MOE_ROUTE_TILE * N4;
    constexpr int AHEAD = sizeof(T) == 2 ? MOE_ROUTE_RUN : MOE_ROUTE_RUN / 2;      // segments whose loads are on their way together
    for (int item = warp; item < runs * quads; item += MOE_ROUTE_TILE_THREADS / 32) {
        const int run = item / quads, q = item - run * quads;
        float v[4 * MOE_ROUTE_TILE];
#pragma unroll
        for (int i = 0; i < 4 * MOE_ROUTE_TILE; i++) v[i] = 0.0f;
#pragma unroll
        for (int i0 = 0; i0 < MOE_ROUTE_RUN; i0 += AHEAD) {
            MoePiece<T> xv[AHEAD][MOE_ROUTE_TILE];
            float4 wv[AHEAD][4];
#pragma unroll
            for (int i = 0; i < AHEAD; i++) {
                const int k = (run * MOE_ROUTE_RUN + i0 + i) * 128 + 4 * lane, at = k < D ? k : 0;      // past the row: zeros in place of x
#pragma unroll
                for (int n = 0; n < 4; n++) wv[i][n] = *reinterpret_cast<const float4*>(router + (size_t)min(4 * q + n, N - 1) * D + at);
#pragma unroll
                for (int j = 0; j < MOE_ROUTE_TILE; j++) xv[i][j].load(x + (size_t)min(t0 + j, tokens - 1) * D + at);
            }
#pragma unroll
            for (int i = 0; i < AHEAD; i++) {
                const bool ok = (run * MOE_ROUTE_RUN + i0 + i) * 128 + 4 * lane < D;
                if (!ok)
#pragma unroll
                    for (int n = 0; n < 4; n++) wv[i][n] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
                for (int j = 0; j < MOE_ROUTE_TILE; j++) {
                    const float4 a = ok ? xv[i][j].value() : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
                    for (int n = 0; n < 4; n++) {
                        float c = v[4 * j + n];
                        c = fmaf(a.x, wv[i][n].x, c);
                        c = fmaf(a.y, wv[i][n].y, c);
                        c = fmaf(a.z, wv[i][n].z, c);
                        v[4 * j + n] = fmaf(a.w, wv[i][n].w, c);
                    }
                }
            }
        }
#pragma unroll
        for (int o = 16; o > 1; o >>= 1) {
            const bool upper = (lane & o) != 0;
#pragma unroll
            for (int i = 0; i < o / 2; i++) {
                const float give = upper ? v[i] : v[i + o / 2];
                const float keep = upper ? v[i + o / 2] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
        }
        v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
        if ((lane & 1) == 0) part[((size_t)run * MOE_ROUTE_TILE + (lane >> 3)) * N4 + 4 * q + ((lane >> 1) & 3)] = v[0];
    }
    __syncthreads();
    const int pitch = 2 * N + rule.groups;
    for (int i = threadIdx.x; i < MOE_ROUTE_TILE * N; i += MOE_ROUTE_TILE_THREADS) {
        const int j = i / N, n = i - j * N;
        float a = 0.0f;
#pragma unroll 8
        for (int g = 0; g < runs; g++) a += part[((size_t)g * MOE_ROUTE_TILE + j) * N4 + n];
        scores[j * pitch + n] = a;
    }
    __syncthreads();
    static_assert(MOE_ROUTE_TILE <= MOE_ROUTE_TILE_THREADS / 32, "a warp per token");
    if (warp >= MOE_ROUTE_TILE || t0 + warp >= tokens) return;
    float* s = scores + (size_t)warp * pitch;
    moe_choose(s, s + N, s + 2 * N, correction, idx, weight, t0 + warp, N, top, lane, rule);
}

static int moe_sms() {
    static int sms = 0;
    if (!sms) {
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        sms = n > 0 ? n : 148;
    }
    return sms;
}

extern "C" int ri_moe_route_rule(const void* x, const float* router, const float* correction, int* idx, float* weight,
                                 int tokens, int D, int N, int top, int mode, int groups, int keep, int gtop, float scale,
                                 int renorm, const float* bias, int dtype, cudaStream_t stream) {
    if (tokens == 0) return 0;
    RI_REQUIRE(mode >= 0 && mode <= 2, "moe_route: score rule %d", mode);
    RI_REQUIRE(mode == 2 || correction, "moe_route: score rule %d needs its correction", mode);
    RI_REQUIRE(groups >= 1 && N % groups == 0 && keep >= 1 && keep <= groups && gtop >= 1,
               "moe_route: %d outputs in %d groups of which %d are kept", N, groups, keep);
    RI_REQUIRE(top <= keep * (N / groups), "moe_route: top %d of the %d outputs of the kept groups", top, keep * (N / groups));
    MoeRule rule;
    rule.mode = mode; rule.groups = groups; rule.keep = keep; rule.gtop = gtop; rule.renorm = renorm; rule.scale = scale;
    rule.bias = bias;
    RI_REQUIRE(tokens > 0 && D > 0 && N > 0 && top > 0 && top <= N, "moe_route: bad sizes (top %d of %d)", top, N);
    RI_REQUIRE(N <= 4096, "moe_route: %d router outputs (up to 4096 are built)", N);
    const size_t smem = (size_t)MOE_ROUTE_WARPS * (2 * N + groups) * sizeof(float);
    const dim3 grid((tokens + MOE_ROUTE_WARPS - 1) / MOE_ROUTE_WARPS);
    // (which form runs depends on sizes, the number of tokens among them, and addresses; the two forms that the tokens decide between give
    // the same bits)
    const int vec = (D % 4 == 0 && (((uintptr_t)router | (uintptr_t)x) & 15) == 0) ? 1 : 0;
    cudaError_t e = cudaSuccess;
    const long long items = (long long)N * ((D + 127) / 128);
    // Blocks of four tokens from where blocks of one token, which have an SM each, need a second round of the SMs.  Cold, 148 SMs, width 4,096 and
    // 18 outputs: one token a block 14.4 us up to 148 tokens and 22.5 for 200, four 16.6 for 256; width 2,048 and 34 outputs 14.4, 22.5, 16.4.
    const long long runs = (D + 128 * MOE_ROUTE_RUN - 1) / (128 * MOE_ROUTE_RUN);
    const size_t tile_sm = ((size_t)runs * MOE_ROUTE_TILE * ((N + 3) / 4 * 4) + (size_t)MOE_ROUTE_TILE * (2 * N + groups)) * sizeof(float);
    if (vec && items <= MOE_ROUTE_WIDE_ITEMS && tokens > moe_sms() && tile_sm <= 96 * 1024) {
        const dim3 tiles((tokens + MOE_ROUTE_TILE - 1) / MOE_ROUTE_TILE);
        if (dtype == RI_DTYPE_F32) {
            if (tile_sm > 48 * 1024) e = cudaFuncSetAttribute(moe_route_tile_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tile_sm);
            if (e != cudaSuccess) RI_FAIL((int)e, "moe_route: %s", cudaGetErrorString(e));
            ri_launch_pdl(moe_route_tile_kernel<float>, tiles, dim3(MOE_ROUTE_TILE_THREADS), tile_sm, stream, (const float*)x, router,
                          correction, idx, weight, tokens, D, N, top, rule);
        } else if (dtype == RI_DTYPE_BF16) {
            if (tile_sm > 48 * 1024) e = cudaFuncSetAttribute(moe_route_tile_kernel<bf16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tile_sm);
            if (e != cudaSuccess) RI_FAIL((int)e, "moe_route: %s", cudaGetErrorString(e));
            ri_launch_pdl(moe_route_tile_kernel<bf16>, tiles, dim3(MOE_ROUTE_TILE_THREADS), tile_sm, stream, (const bf16*)x, router,
                          correction, idx, weight, tokens, D, N, top, rule);
        } else RI_FAIL(-1, "moe_route: unknown dtype %d", dtype);
        RI_CHECK_LAUNCH("moe_route");
        return 0;
    }
    if (vec && items <= MOE_ROUTE_WIDE_ITEMS && tokens <= 65535 * 32) {
        const size_t sm = (size_t)(N * runs + 2 * N + groups) * sizeof(float);
        if (dtype == RI_DTYPE_F32)
            ri_launch_pdl(moe_route_wide_kernel<float>, dim3(tokens), dim3(MOE_ROUTE_WIDE_THREADS), sm, stream, (const float*)x,
                          router, correction, idx, weight, D, N, top, rule);
        else if (dtype == RI_DTYPE_BF16)
            ri_launch_pdl(moe_route_wide_kernel<bf16>, dim3(tokens), dim3(MOE_ROUTE_WIDE_THREADS), sm, stream, (const bf16*)x,
                          router, correction, idx, weight, D, N, top, rule);
        else RI_FAIL(-1, "moe_route: unknown dtype %d", dtype);
        RI_CHECK_LAUNCH("moe_route");
        return 0;
    }
    if (dtype == RI_DTYPE_F32) {
        if (smem > 48 * 1024) e = cudaFuncSetAttribute(moe_route_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) RI_FAIL((int)e, "moe_route: %s", cudaGetErrorString(e));
        ri_launch_pdl(moe_route_kernel<float>, grid, dim3(32 * MOE_ROUTE_WARPS), smem, stream, (const float*)x, router,
                      correction, idx, weight, tokens, D, N, top, vec, rule);
    } else if (dtype == RI_DTYPE_BF16) {
        if (smem > 48 * 1024) e = cudaFuncSetAttribute(moe_route_kernel<bf16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) RI_FAIL((int)e, "moe_route: %s", cudaGetErrorString(e));
        ri_launch_pdl(moe_route_kernel<bf16>, grid, dim3(32 * MOE_ROUTE_WARPS), smem, stream, (const bf16*)x, router,
                      correction, idx, weight, tokens, D, N, top, vec, rule);
    } else RI_FAIL(-1, "moe_route: unknown dtype %d", dtype);
    RI_CHECK_LAUNCH("moe_route");
    return 0;
}

// ---- the plan ---------------------------------------------------------------------------------------------------------
// meta[0] = number of tiles, meta[1] = number of rows in perm.  tiles [max_tiles][3].
// With a `table` [vocab, top] of experts by token id (no router) the pairs' experts are looked up here, idx[t top + j] =
// table[ids[t]][j], and written to idx_out for whoever reads the choice later.
struct MoeTable {
    const int* ids;
    const int* table;            // null: idx holds the choice
    int vocab, top;
    int* idx_out;
    int* err;
};
__global__ void __launch_bounds__(1024)
moe_plan_kernel(const int* idx, int* __restrict__ perm, int* __restrict__ tiles, int* __restrict__ meta,
                int pairs, int E, int max_tiles, int bm, MoeTable by_id) {
    extern __shared__ int plan_sm[];                  // counts, offsets, tiles before, next free place: [E] each
    int* counts = plan_sm;
    int* offsets = counts + E;
    int* first_tile = offsets + E;
    int* next = first_tile + E;
    pdl_trigger();
    const int lane = threadIdx.x & 31;
    for (int e = threadIdx.x; e < E; e += blockDim.x) counts[e] = 0;
    pdl_wait();
    __syncthreads();
    if (by_id.table) idx = by_id.idx_out;             // (a thread reads back only what it wrote itself)
    for (int p = threadIdx.x; p < pairs; p += blockDim.x) {
        if (by_id.table) {
            const int t = p / by_id.top, id = by_id.ids[t];
            int chosen = -1;
            if (id >= 0 && id < by_id.vocab) chosen = by_id.table[(size_t)id * by_id.top + (p - t * by_id.top)];
            if (chosen < 0 || chosen >= E) {
                atomicExch(by_id.err, id >= 0 && id < by_id.vocab ? 8 : 1);
                chosen = -1;
            }
            by_id.idx_out[p] = chosen;
        }
        const int e = idx[p];
        if (e >= 0 && e < E) atomicAdd(&counts[e], 1);
    }
    __syncthreads();
    if (threadIdx.x < 32) {                           // one warp: the experts' runs and their first tiles, 32 experts a trip
        int off = 0, n = 0;
        for (int e0 = 0; e0 < E; e0 += 32) {
            const int e = e0 + lane, c = e < E ? counts[e] : 0;
            int rows = c, tl = (c + bm - 1) / bm;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int r = __shfl_up_sync(0xffffffffu, rows, o), t = __shfl_up_sync(0xffffffffu, tl, o);
                if (lane >= o) {
                    rows += r;
                    tl += t;
                }
            }
            if (e < E) {
                offsets[e] = next[e] = off + rows - c;
                first_tile[e] = n + tl - (c + bm - 1) / bm;
            }
            off += __shfl_sync(0xffffffffu, rows, 31);
            n += __shfl_sync(0xffffffffu, tl, 31);
        }
        if (lane == 0) {
            meta[0] = n < max_tiles ? n : max_tiles;
            meta[1] = off;
        }
    }
    __syncthreads();
    for (int e = threadIdx.x >> 5; e < E; e += blockDim.x >> 5) {      // a warp per expert: its tiles
        const int c = counts[e];
        for (int i = lane; i * bm < c && first_tile[e] + i < max_tiles; i += 32) {
            int* tile = tiles + 3 * (first_tile[e] + i);
            tile[0] = e;
            tile[1] = offsets[e] + i * bm;
            tile[2] = min(bm, c - i * bm);
        }
    }
    for (int p = threadIdx.x; p < pairs; p += blockDim.x) {
        const int e = idx[p];
        if (e >= 0 && e < E) perm[atomicAdd(&next[e], 1)] = p;
    }
}

// bm: rows per tile, MOE_BM (32) or MOE_BM_WIDE (256: many pairs per expert, bfloat16 with 16-byte rows, moe_tc.cu)
extern "C" int ri_moe_max_tiles(int pairs, int E, int bm) { return (pairs + bm - 1) / bm + E; }

extern "C" int ri_moe_plan(const int* idx, int* perm, int* tiles, int* meta, int pairs, int E, int max_tiles, int bm,
                           cudaStream_t stream) {
    if (pairs == 0) return 0;
    RI_REQUIRE(bm == MOE_BM || bm == MOE_BM_WIDE, "moe_plan: tiles of %d rows are not built", bm);
    RI_REQUIRE(pairs > 0 && E > 0 && max_tiles >= ri_moe_max_tiles(pairs, E, bm), "moe_plan: bad sizes");
    const size_t smem = (size_t)4 * E * sizeof(int);
    RI_REQUIRE(E <= 4095, "moe_plan: %d experts (up to 4095 are built)", E);
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(moe_plan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) RI_FAIL((int)e, "moe_plan: %s", cudaGetErrorString(e));
    }
    ri_launch_pdl(moe_plan_kernel, dim3(1), dim3(1024), smem, stream, idx, perm, tiles, meta, pairs, E, max_tiles, bm,
                  MoeTable{nullptr, nullptr, 0, 0, nullptr, nullptr});
    RI_CHECK_LAUNCH("moe_plan");
    return 0;
}

// The plan of a step whose experts a table names: ids [tokens] int32, table [vocab, top] int32; idx [tokens, top] gets the
// choice.  A token id outside the table: error word 1; an expert that does not exist: error word 8 (the pair is left out).
extern "C" int ri_moe_plan_table(const int* ids, const int* table, int vocab, int top, int* idx, int* perm, int* tiles, int* meta,
                                 int tokens, int E, int max_tiles, int bm, int* err_flag, cudaStream_t stream) {
    if (tokens == 0) return 0;
    RI_REQUIRE(bm == MOE_BM || bm == MOE_BM_WIDE, "moe_plan: tiles of %d rows are not built", bm);
    RI_REQUIRE(tokens > 0 && top > 0 && vocab > 0 && (long long)tokens * top < (1ll << 31), "moe_plan: bad sizes");
    const int pairs = tokens * top;
    RI_REQUIRE(E > 0 && max_tiles >= ri_moe_max_tiles(pairs, E, bm), "moe_plan: bad sizes");
    const size_t smem = (size_t)4 * E * sizeof(int);
    RI_REQUIRE(E <= 4095, "moe_plan: %d experts (up to 4095 are built)", E);
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(moe_plan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) RI_FAIL((int)e, "moe_plan: %s", cudaGetErrorString(e));
    }
    ri_launch_pdl(moe_plan_kernel, dim3(1), dim3(1024), smem, stream, (const int*)nullptr, perm, tiles, meta, pairs, E, max_tiles,
                  bm, MoeTable{ids, table, vocab, top, idx, err_flag});
    RI_CHECK_LAUNCH("moe_plan");
    return 0;
}

// ---- grouped products ---------------------------------------------------------------------------------------------------
template <typename TO>
__device__ __forceinline__ void moe_store(TO* p, float v) { st_f(p, v); }

// float32: 128 threads, each 4 rows x 4 columns of the 32 x 64 tile; k ascending, one accumulator per output
template <typename TO>
__global__ void __launch_bounds__(128)
moe_grouped_f32_kernel(const float* __restrict__ a, long long lda, const float* __restrict__ w, TO* __restrict__ y,
                       long long ldy, const int* __restrict__ perm, const int* __restrict__ tiles,
                       const int* __restrict__ meta, int N, int K, int gather_div, int scatter) {
    constexpr int BK = 16;
    __shared__ float As[BK][MOE_BM + 1], Ws[BK][MOE_BN + 1];
    __shared__ int s_in[MOE_BM], s_out[MOE_BM];
    pdl_trigger();
    pdl_wait();
    if ((int)blockIdx.x >= meta[0]) return;
    const int e = tiles[3 * blockIdx.x], r0 = tiles[3 * blockIdx.x + 1], rows = tiles[3 * blockIdx.x + 2];
    const int n0 = blockIdx.y * MOE_BN;
    for (int i = threadIdx.x; i < MOE_BM; i += blockDim.x) {
        const int p = i < rows ? perm[r0 + i] : 0;
        s_in[i] = gather_div > 0 ? p / gather_div : r0 + i;
        s_out[i] = scatter ? p : r0 + i;
    }
    __syncthreads();
    const float* we = w + (size_t)e * N * K;
    const int ty = threadIdx.x / 16, tx = threadIdx.x % 16;
    float acc[4][4] = {};
    for (int k0 = 0; k0 < K; k0 += BK) {
        for (int i = threadIdx.x; i < MOE_BM * BK; i += blockDim.x) {
            const int r = i / BK, k = i % BK;
            As[k][r] = (r < rows && k0 + k < K) ? a[(size_t)s_in[r] * lda + k0 + k] : 0.0f;
        }
        for (int i = threadIdx.x; i < MOE_BN * BK; i += blockDim.x) {
            const int n = i / BK, k = i % BK;
            Ws[k][n] = (n0 + n < N && k0 + k < K) ? we[(size_t)(n0 + n) * K + k0 + k] : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; k++) {
            float av[4], wv[4];
#pragma unroll
            for (int i = 0; i < 4; i++) av[i] = As[k][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; j++) wv[j] = Ws[k][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int r = ty * 4 + i;
        if (r >= rows) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int n = n0 + tx * 4 + j;
            if (n < N) moe_store(y + (size_t)s_out[r] * ldy + n, acc[i][j]);
        }
    }
}

// bfloat16: 4 warps; warp w owns columns 16 w .. 16 w + 15 of the tile and all 32 rows (2 x 2 mma tiles per k16).
// VEC (K a multiple of 8, 16-byte aligned rows): the tiles of A and W come by cp.async through a ring of STAGES
// stages of 64 k each, so that all others are on their way while one is multiplied; otherwise element by element.
// STAGES: four where all blocks find a place at once with four on an SM (56 KB each: 96 KB of the experts' matrices on their way),
// three where five on an SM save a round of blocks (`moe_stages`).  A few tokens are bound by reading those matrices.  First product with
// the gate, four / three stages: 24 tokens of one choice, 8 experts of 1,376 channels and width 4,096 (344 blocks) 53 / 56 us; 24 tokens of four
// choices, 16 experts (688 blocks, two rounds of four an SM, one of five) 92 / 76 us, 32 experts of 704 and width 2,048 alike; second
// product (1,024 blocks, two rounds either way) 41.4 / 44.4 us.
// GATED: W [E, 2 N, K] holds an expert's gate rows, then its up rows; a tile takes 32 channels, the gate rows as its columns
// 0 .. 31 and the up rows as 32 .. 63, and the epilogue puts the two float32 sums of a channel together.
#define MOE_BK 64
#define MOE_PITCH (MOE_BK + 8)
#define MOE_SMEM(stages) ((stages) * (MOE_BM + MOE_BN) * MOE_PITCH * 2)
struct MoeGate {
    int kind;                              // 0 none; 1 silu(g) u; 2 gelu in its tanh form times u; 3 the clamped swish
    float limit, alpha;
};
__device__ __forceinline__ float moe_gate(float g, float u, const MoeGate& c) {
    if (c.kind == 3) {
        g = fminf(g, c.limit);
        u = fminf(fmaxf(u, -c.limit), c.limit) + 1.0f;
        return (g / (1.0f + expf(-c.alpha * g))) * u;
    }
    if (c.kind == 2) return 0.5f * g * (1.0f + tanhf(0.7978845608028654f * (g + 0.044715f * g * g * g))) * u;
    return g / (1.0f + expf(-g)) * u;
}
template <typename TO, bool VEC, bool GATED, int STAGES>
__global__ void __launch_bounds__(128)
moe_grouped_bf16_kernel(const bf16* __restrict__ a, long long lda, const bf16* __restrict__ w, TO* __restrict__ y,
                        long long ldy, const int* __restrict__ perm, const int* __restrict__ tiles,
                        const int* __restrict__ meta, int N, int K, int gather_div, int scatter, MoeGate gate) {
    constexpr int ST = VEC ? STAGES : 1;
    extern __shared__ __align__(16) unsigned char moe_grouped_sm[];
    bf16 (*As)[MOE_BM][MOE_PITCH] = reinterpret_cast<bf16 (*)[MOE_BM][MOE_PITCH]>(moe_grouped_sm);
    bf16 (*Ws)[MOE_BN][MOE_PITCH] = reinterpret_cast<bf16 (*)[MOE_BN][MOE_PITCH]>(moe_grouped_sm + ST * MOE_BM * MOE_PITCH * 2);
    __shared__ int s_in[MOE_BM], s_out[MOE_BM];
    pdl_trigger();
    pdl_wait();
    if ((int)blockIdx.x >= meta[0]) return;
    const int e = tiles[3 * blockIdx.x], r0 = tiles[3 * blockIdx.x + 1], rows = tiles[3 * blockIdx.x + 2];
    constexpr int COLS = GATED ? MOE_BN / 2 : MOE_BN;                 // outputs per tile
    const int n0 = blockIdx.y * COLS;
    for (int i = threadIdx.x; i < MOE_BM; i += blockDim.x) {
        const int p = i < rows ? perm[r0 + i] : 0;
        s_in[i] = gather_div > 0 ? p / gather_div : r0 + i;
        s_out[i] = scatter ? p : r0 + i;
    }
    __syncthreads();
    const bf16* we = w + (size_t)e * N * K * (GATED ? 2 : 1);
    // the row of W behind column n of the tile, and whether there is one
    auto w_row = [&](int n) { return GATED && n >= COLS ? N + n0 + n - COLS : n0 + n; };
    auto w_ok = [&](int n) { return n0 + (GATED ? n % COLS : n) < N; };
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int quad = lane >> 2, qc = lane & 3;
    float acc[2][2][4] = {};
    const bf16 zero = __float2bfloat16_rn(0.0f);
    auto copy_stage = [&](int st, int k0) {        // VEC: 16-byte pieces, zeros past the tile's rows, N and K
#pragma unroll
        for (int pass = 0; pass < 2; pass++) {
            const int i = threadIdx.x + pass * 128;
            const int r = i / 8, kc = (i % 8) * 8;
            const bool ok = r < rows && k0 + kc < K;
            cp_async16(&As[st][r][kc], ok ? a + (size_t)s_in[r] * lda + k0 + kc : a, ok);
        }
#pragma unroll
        for (int pass = 0; pass < 4; pass++) {
            const int i = threadIdx.x + pass * 128;
            const int n = i / 8, kc = (i % 8) * 8;
            const bool ok = w_ok(n) && k0 + kc < K;
            cp_async16(&Ws[st][n][kc], ok ? we + (size_t)w_row(n) * K + k0 + kc : we, ok);
        }
    };
    auto multiply = [&](int st) {
#pragma unroll
        for (int kk = 0; kk < MOE_BK; kk += 16) {
            unsigned af[2][4], bfr[2][2];
#pragma unroll
            for (int mi = 0; mi < 2; mi++) {
                af[mi][0] = *reinterpret_cast<const unsigned*>(&As[st][mi * 16 + quad][kk + qc * 2]);
                af[mi][1] = *reinterpret_cast<const unsigned*>(&As[st][mi * 16 + quad + 8][kk + qc * 2]);
                af[mi][2] = *reinterpret_cast<const unsigned*>(&As[st][mi * 16 + quad][kk + qc * 2 + 8]);
                af[mi][3] = *reinterpret_cast<const unsigned*>(&As[st][mi * 16 + quad + 8][kk + qc * 2 + 8]);
            }
#pragma unroll
            for (int ni = 0; ni < 2; ni++) {
                bfr[ni][0] = *reinterpret_cast<const unsigned*>(&Ws[st][warp * 16 + ni * 8 + quad][kk + qc * 2]);
                bfr[ni][1] = *reinterpret_cast<const unsigned*>(&Ws[st][warp * 16 + ni * 8 + quad][kk + qc * 2 + 8]);
            }
#pragma unroll
            for (int mi = 0; mi < 2; mi++)
#pragma unroll
                for (int ni = 0; ni < 2; ni++)
                    mma_bf16(acc[mi][ni], af[mi][0], af[mi][1], af[mi][2], af[mi][3], bfr[ni][0], bfr[ni][1]);
        }
    };
    const int nk = (K + MOE_BK - 1) / MOE_BK;
    if (VEC) {
        for (int st = 0; st < STAGES - 1; st++) {
            if (st < nk) copy_stage(st, st * MOE_BK);
            cp_async_commit();
        }
        for (int it = 0; it < nk; it++) {
            cp_async_wait<STAGES - 2>();
            __syncthreads();                         // stage `it` has landed for everyone; the stage of it - 1 is free
            const int ahead = it + STAGES - 1;
            if (ahead < nk) copy_stage(ahead % STAGES, ahead * MOE_BK);
            cp_async_commit();
            multiply(it % STAGES);
        }
        cp_async_wait<0>();
    } else {
        for (int it = 0; it < nk; it++) {
            const int k0 = it * MOE_BK;
            for (int i = threadIdx.x; i < MOE_BM * MOE_BK; i += blockDim.x) {
                const int r = i / MOE_BK, k = i % MOE_BK;
                As[0][r][k] = (r < rows && k0 + k < K) ? a[(size_t)s_in[r] * lda + k0 + k] : zero;
            }
            for (int i = threadIdx.x; i < MOE_BN * MOE_BK; i += blockDim.x) {
                const int n = i / MOE_BK, k = i % MOE_BK;
                Ws[0][n][k] = (w_ok(n) && k0 + k < K) ? we[(size_t)w_row(n) * K + k0 + k] : zero;
            }
            __syncthreads();
            multiply(0);
            __syncthreads();
        }
    }
    if (GATED) {
        float (*sums)[MOE_BN + 1] = reinterpret_cast<float (*)[MOE_BN + 1]>(moe_grouped_sm);
        static_assert(MOE_BM * (MOE_BN + 1) * 4 <= MOE_SMEM(1), "the tile's sums fit in the stages");
        __syncthreads();                             // the last stage was read
#pragma unroll
        for (int mi = 0; mi < 2; mi++)
#pragma unroll
            for (int ni = 0; ni < 2; ni++)
#pragma unroll
                for (int c = 0; c < 4; c++)
                    sums[mi * 16 + quad + (c >> 1) * 8][warp * 16 + ni * 8 + qc * 2 + (c & 1)] = acc[mi][ni][c];
        __syncthreads();
        for (int i = threadIdx.x; i < rows * COLS; i += blockDim.x) {
            const int r = i / COLS, c = i % COLS;
            if (n0 + c < N) moe_store(y + (size_t)s_out[r] * ldy + n0 + c, moe_gate(sums[r][c], sums[r][COLS + c], gate));
        }
        return;
    }
#pragma unroll
    for (int mi = 0; mi < 2; mi++)
#pragma unroll
        for (int ni = 0; ni < 2; ni++)
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const int r = mi * 16 + quad + (c >> 1) * 8;
                const int n = n0 + warp * 16 + ni * 8 + qc * 2 + (c & 1);
                if (r < rows && n < N) moe_store(y + (size_t)s_out[r] * ldy + n, acc[mi][ni][c]);
            }
}

// rounds of blocks that the SMs take with four (four stages) and five (three stages) on each
static int moe_stages(long long blocks) {
    const int sms = moe_sms();
    return (blocks + 5 * sms - 1) / (5 * sms) < (blocks + 4 * sms - 1) / (4 * sms) ? 3 : 4;
}
template <typename TO, bool VEC, bool GATED, int STAGES>
static int moe_grouped_launch(dim3 grid, cudaStream_t stream, const void* a, long long lda, const void* w, void* y, long long ldy,
                              const int* perm, const int* tiles, const int* meta, int N, int K, int gather_div, int scatter, MoeGate gate) {
    constexpr int sm = MOE_SMEM(VEC ? STAGES : 1);
    if (sm > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(moe_grouped_bf16_kernel<TO, VEC, GATED, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
        if (e != cudaSuccess) RI_FAIL((int)e, "moe_grouped: %s", cudaGetErrorString(e));
    }
    ri_launch_pdl(moe_grouped_bf16_kernel<TO, VEC, GATED, STAGES>, grid, dim3(128), (size_t)sm, stream, (const bf16*)a, lda, (const bf16*)w,
                  (TO*)y, ldy, perm, tiles, meta, N, K, gather_div, scatter, gate);
    return 0;
}
// likely: the tiles that a step of so many pairs has as a rule (the grid covers the most it can have)
template <typename TO, bool VEC, bool GATED>
static int moe_grouped_go(dim3 grid, int likely, cudaStream_t stream, const void* a, long long lda, const void* w, void* y, long long ldy,
                          const int* perm, const int* tiles, const int* meta, int N, int K, int gather_div, int scatter, MoeGate gate) {
    if (VEC && moe_stages((long long)likely * grid.y) == 3)
        return moe_grouped_launch<TO, VEC, GATED, 3>(grid, stream, a, lda, w, y, ldy, perm, tiles, meta, N, K, gather_div, scatter, gate);
    return moe_grouped_launch<TO, VEC, GATED, 4>(grid, stream, a, lda, w, y, ldy, perm, tiles, meta, N, K, gather_div, scatter, gate);
}

// a [rows, lda] and w [E, N, K] in the compute type; y [.., ldy] float32 (out_f32) or the compute type
// bm: the tile height that the plan was made with (plans with tiles of MOE_BM_WIDE rows are for moe_tc.cu); likely: how many of the
// max_tiles tiles the step has as a rule (it chooses between forms with the same results)
extern "C" int ri_moe_grouped_linear(const void* a, long long lda, const void* w, void* y, long long ldy, const int* perm,
                                     const int* tiles, const int* meta, int max_tiles, int likely, int bm, int N, int K, int gather_div,
                                     int scatter, int out_f32, int dtype, cudaStream_t stream) {
    if (max_tiles == 0) return 0;
    RI_REQUIRE(bm == MOE_BM, "moe_grouped_linear: tiles of %d rows", bm);
    RI_REQUIRE(max_tiles > 0 && N > 0 && K > 0 && gather_div >= 0, "moe_grouped_linear: bad sizes");
    const dim3 grid(max_tiles, (N + MOE_BN - 1) / MOE_BN);
    RI_REQUIRE(grid.y <= 65535, "moe_grouped_linear: %d outputs are too many for one launch", N);
    if (dtype == RI_DTYPE_F32) {
        RI_REQUIRE(out_f32, "moe_grouped_linear: a float32 product writes float32");
        ri_launch_pdl(moe_grouped_f32_kernel<float>, grid, dim3(128), 0, stream, (const float*)a, lda, (const float*)w,
                      (float*)y, ldy, perm, tiles, meta, N, K, gather_div, scatter);
    } else if (dtype == RI_DTYPE_BF16) {
        const bool vec = K % 8 == 0 && lda % 8 == 0 && (((uintptr_t)a | (uintptr_t)w) & 15) == 0;
        const MoeGate none{0, 0.0f, 0.0f};
        int rc = out_f32 ? (vec ? moe_grouped_go<float, true, false>(grid, likely, stream, a, lda, w, y, ldy, perm, tiles, meta, N, K, gather_div, scatter, none)
                                : moe_grouped_go<float, false, false>(grid, likely, stream, a, lda, w, y, ldy, perm, tiles, meta, N, K, gather_div, scatter, none))
                         : (vec ? moe_grouped_go<bf16, true, false>(grid, likely, stream, a, lda, w, y, ldy, perm, tiles, meta, N, K, gather_div, scatter, none)
                                : moe_grouped_go<bf16, false, false>(grid, likely, stream, a, lda, w, y, ldy, perm, tiles, meta, N, K, gather_div, scatter, none));
        if (rc) return rc;
    } else RI_FAIL(-1, "moe_grouped_linear: unknown dtype %d", dtype);
    RI_CHECK_LAUNCH("moe_grouped_linear");
    return 0;
}

// bfloat16: w [E, 2 N, K] (an expert's gate rows, then its up rows), y [.., ldy] = f(gate) * up' with gate function 1 silu, 2
// gelu_tanh, 3 the clamped swish with `limit` and `alpha`
extern "C" int ri_moe_grouped_gated(const void* a, long long lda, const void* w, void* y, long long ldy, const int* perm,
                                    const int* tiles, const int* meta, int max_tiles, int likely, int bm, int N, int K, int gather_div,
                                    int gate, float limit, float alpha, cudaStream_t stream) {
    if (max_tiles == 0) return 0;
    RI_REQUIRE(bm == MOE_BM, "moe_grouped_gated: tiles of %d rows", bm);
    RI_REQUIRE(max_tiles > 0 && N > 0 && K > 0 && gather_div >= 0 && gate >= 1 && gate <= 3, "moe_grouped_gated: bad sizes or gate");
    const dim3 grid(max_tiles, (N + MOE_BN / 2 - 1) / (MOE_BN / 2));
    RI_REQUIRE(grid.y <= 65535, "moe_grouped_gated: %d channels are too many for one launch", N);
    const bool vec = K % 8 == 0 && lda % 8 == 0 && (((uintptr_t)a | (uintptr_t)w) & 15) == 0;
    const MoeGate g{gate, limit, alpha};
    int rc = vec ? moe_grouped_go<bf16, true, true>(grid, likely, stream, a, lda, w, y, ldy, perm, tiles, meta, N, K, gather_div, 0, g)
                 : moe_grouped_go<bf16, false, true>(grid, likely, stream, a, lda, w, y, ldy, perm, tiles, meta, N, K, gather_div, 0, g);
    if (rc) return rc;
    RI_CHECK_LAUNCH("moe_grouped_gated");
    return 0;
}

// ---- combination ----------------------------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256)
moe_combine_kernel(const float* __restrict__ pair_out, const int* __restrict__ idx, const float* __restrict__ weight,
                   const T* __restrict__ x, const T* __restrict__ extra, T* __restrict__ y, int D, int top, int E) {
    pdl_trigger();
    pdl_wait();
    const int t = blockIdx.x;
    const float equal = 1.0f / (float)top;               // every choice's weight where none are given
    for (int d = blockIdx.y * blockDim.x + threadIdx.x; d < D; d += gridDim.y * blockDim.x) {
        float acc = 0.0f;
        for (int j = 0; j < top; j++) {
            const int e = idx ? idx[(size_t)t * top + j] : 0;
            const float v = (e >= E) ? ld_f(x + (size_t)t * D + d) : pair_out[((size_t)t * top + j) * D + d];
            acc = fmaf(weight ? weight[(size_t)t * top + j] : equal, v, acc);
        }
        if (extra) acc += ld_f(extra + (size_t)t * D + d);
        st_f(y + (size_t)t * D + d, acc);
    }
}

// Rows of whole groups of four elements: four neighbouring ones per thread, the loads of four choices on their way together
// (2,048 tokens of 4 choices and width 4,096, 170 MB: 75 -> 35 us).  The same additions in the same order.
template <typename T>
__global__ void __launch_bounds__(256)
moe_combine_vec4_kernel(const float* pair_out, const int* idx, const float* weight, const T* x, const T* extra, T* __restrict__ y,
                        int D, int top, int E) {
    pdl_trigger();
    pdl_wait();
    const int t = blockIdx.x;
    const float equal = 1.0f / (float)top;
    for (int d = 4 * (blockIdx.y * blockDim.x + threadIdx.x); d < D; d += 4 * gridDim.y * blockDim.x) {
        float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
        for (int j = 0; j < top; j++) {
            const int e = idx ? idx[(size_t)t * top + j] : 0;
            const float w = weight ? weight[(size_t)t * top + j] : equal;
            const float4 v = (e >= E) ? moe_ld4(x + (size_t)t * D + d) : moe_ld4(pair_out + ((size_t)t * top + j) * D + d);
            acc.x = fmaf(w, v.x, acc.x);
            acc.y = fmaf(w, v.y, acc.y);
            acc.z = fmaf(w, v.z, acc.z);
            acc.w = fmaf(w, v.w, acc.w);
        }
        if (extra) {
            const float4 v = moe_ld4(extra + (size_t)t * D + d);
            acc.x += v.x;
            acc.y += v.y;
            acc.z += v.z;
            acc.w += v.w;
        }
        moe_st4(y + (size_t)t * D + d, acc);
    }
}

// weight null: every choice has weight 1 / top; idx null: no choice is an identity expert (x is not read)
extern "C" int ri_moe_combine(const float* pair_out, const int* idx, const float* weight, const void* x, const void* extra,
                              void* y, int tokens, int D, int top, int E, int dtype, cudaStream_t stream) {
    if (tokens == 0) return 0;
    RI_REQUIRE(tokens > 0 && D > 0 && top > 0, "moe_combine: bad sizes");
    if (D % 4 == 0 && (((uintptr_t)pair_out | (uintptr_t)x | (uintptr_t)extra | (uintptr_t)y) & 15) == 0 &&
        (dtype == RI_DTYPE_F32 || dtype == RI_DTYPE_BF16)) {
        // (one group per thread: a block per 1,024 elements of a token)
        const dim3 grid4(tokens, (D + 1023) / 1024 > 64 ? 64 : (D + 1023) / 1024);
        if (dtype == RI_DTYPE_F32)
            ri_launch_pdl(moe_combine_vec4_kernel<float>, grid4, dim3(256), 0, stream, pair_out, idx, weight, (const float*)x,
                          (const float*)extra, (float*)y, D, top, E);
        else
            ri_launch_pdl(moe_combine_vec4_kernel<bf16>, grid4, dim3(256), 0, stream, pair_out, idx, weight, (const bf16*)x,
                          (const bf16*)extra, (bf16*)y, D, top, E);
        RI_CHECK_LAUNCH("moe_combine");
        return 0;
    }
    const dim3 grid(tokens, tokens >= 512 ? 1 : (D + 255) / 256 > 64 ? 64 : (D + 255) / 256);    // few tokens: a row over several blocks
    if (dtype == RI_DTYPE_F32)
        ri_launch_pdl(moe_combine_kernel<float>, grid, dim3(256), 0, stream, pair_out, idx, weight, (const float*)x,
                      (const float*)extra, (float*)y, D, top, E);
    else if (dtype == RI_DTYPE_BF16)
        ri_launch_pdl(moe_combine_kernel<bf16>, grid, dim3(256), 0, stream, pair_out, idx, weight, (const bf16*)x,
                      (const bf16*)extra, (bf16*)y, D, top, E);
    else RI_FAIL(-1, "moe_combine: unknown dtype %d", dtype);
    RI_CHECK_LAUNCH("moe_combine");
    return 0;
}

extern "C" int ri_moe_route(const void* x, const float* router, const float* correction, int* idx, float* weight,
                            int tokens, int D, int N, int top, int dtype, cudaStream_t stream) {
    return ri_moe_route_rule(x, router, correction, idx, weight, tokens, D, N, top, 0, 1, 1, 1, 1.0f, 1, nullptr, dtype, stream);
}
