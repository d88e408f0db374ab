// Routed feed-forward: the router's choice, the rows sorted by expert for the grouped tensor-core
// products (gemm_tc.cu), the experts' products of a few tokens, and the plain expert products.
//
//   route        scores s = softmax(z) over all E experts (float32); experts lie in `groups` equal
//                groups of neighbours, a group scores its best expert, only the `keep` best groups
//                stay eligible; the `top` best eligible experts are taken, weight = their score
//                (divided by the sum of the taken scores when `renorm` is set).  Ties go to the lower
//                index.  One warp per token.  On request it also counts the choices per expert.
//   plan_rows, place_rows   every expert's (token, choice) pairs in a run of rows of their own (see below)
//   expert_rows_bf16        up and down products of a few tokens, bfloat16, a warp per four output rows
//   expert_tiles            the same with an expert's matrix read once for all the pairs that chose it
//   expert_up    act[t, c, :] = f(W_up[e(t,c)] h[t])             c < top, f = gelu (erf or tanh form)
//   expert_down  part[c][t, :] = weight(t,c) * W_down[e(t,c)] act[t, c, :]   float32 parts, one per choice,
//                which the consumer (the norm that takes the branch) adds in index order
//   act_rows     f applied in place to [T, F] rows (the shared expert's hidden layer)
//   A gated expert's first matrix holds gate and up rows (w_up [E, 2F, D]): act = silu(gate) * up.  On request the pair's
//   weight multiplies the expert's input instead of its output: the products are linear, so it multiplies what they give
//   before the activation, in float32.
//
// expert_up / expert_down are one warp per output value with the reduction in a fixed lane order, so a
// token's result depends on its own row alone; they serve the 32-bit engine and sizes the others do not
// take, and are what the faster products are held to.
#include "common.cuh"
#include <math.h>

namespace aien {

// kind 0: gelu (erf form), 1: gelu (tanh form), 2: the square of relu
__device__ __forceinline__ float act_apply(float z, int kind) {
    if (kind == 2) { const float r = fmaxf(z, 0.f); return r * r; }
    if (kind == 1) return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
    return 0.5f * z * (1.0f + erff(z * 0.7071067811865476f));
}

// ---------------------------------------------------------------- router
constexpr int ROUTE_MAX_EXPERTS = 1024;

// One warp per token, its scores in registers: lane l holds experts l, l + 32, ...  What bounds a router is the chain of its `top` choices, one
// after another, and a choice is two warp reductions in hardware: the largest key (unsigned, in the order of the floats), then the
// lowest expert that has it.  Before, every choice went through shared memory and ten shuffles, the weights back through global memory.
// B200, us, before and so: 2,048 tokens, 6 of 64 experts in 4 of 8 groups 14.7 and 7.1; 8 of 256 20.4 and 12.5; 64 tokens, 6 of 64 6.5 and 2.6;
// 9 tokens, 4 of 16 with sigmoid scores 3.3 and 1.6; 16 tokens, 8 of 1,024 7.4 and 5.3.  Choices and weights of numbers are the same to the bit.
constexpr int ROUTE_WARPS = 4;                                            // tokens per CTA
constexpr uint32_t ROUTE_TAKEN = 0, ROUTE_OUT = 1, ROUTE_NAN = 2;         // chosen before, not eligible, not a number: below the key of every float

// The order of the floats.  What is not a number is chosen only when no number is left, whatever its sign: one expert's NaN does not
// reach the weights of a token that has numbers to choose from.
__device__ __forceinline__ uint32_t route_key(float v) {
    const uint32_t u = __float_as_uint(v + 0.0f);                         // -0 and 0 are one
    return v != v ? ROUTE_NAN : (u & 0x80000000u) != 0 ? ~u : u | 0x80000000u;
}

// The largest key's index (ties to the lower), which is then taken.
template <int NR>
__device__ __forceinline__ int route_pick(uint32_t (&key)[NR], int lane) {
    uint32_t k = key[0];
    int e = lane;
#pragma unroll
    for (int j = 1; j < NR; ++j)
        if (key[j] > k) { k = key[j]; e = lane + 32 * j; }
    const uint32_t most = __reduce_max_sync(0xffffffffu, k);
    const int pick = __reduce_min_sync(0xffffffffu, k == most ? e : 0x7fffffff);
#pragma unroll
    for (int j = 0; j < NR; ++j)
        if (pick == lane + 32 * j) key[j] = ROUTE_TAKEN;
    return pick;
}

// The score of expert `pick` from the lane that holds it.
template <int NR>
__device__ __forceinline__ float route_score(const float (&s)[NR], int pick, int lane) {
    float w = s[0];
#pragma unroll
    for (int j = 1; j < NR; ++j)
        if (pick == lane + 32 * j) w = s[j];
    return __shfl_sync(0xffffffffu, w, pick & 31);
}

// s = softmax of a row's E numbers
template <int NR>
__device__ __forceinline__ void route_softmax(float (&s)[NR], const float* zr, int E, int lane) {
    float m = -INFINITY;
#pragma unroll
    for (int j = 0; j < NR; ++j) {
        s[j] = lane + 32 * j < E ? __ldcg(zr + lane + 32 * j) : -INFINITY;
        m = fmaxf(m, s[j]);
    }
    m = warp_max(m);
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < NR; ++j)
        if (lane + 32 * j < E) { s[j] = expf(s[j] - m); sum += s[j]; }
    sum = warp_sum(sum);
    const float inv = 1.0f / sum;
#pragma unroll
    for (int j = 0; j < NR; ++j) s[j] *= inv;
}

template <int NR>
__global__ void __launch_bounds__(ROUTE_WARPS * 32)
moe_route_kernel(const float* __restrict__ z, int T, int E, int groups, int keep, int top, int renorm,
                 int* __restrict__ ids, float* __restrict__ wts, int* __restrict__ expert_count) {
    __shared__ float held[ROUTE_WARPS][NR * 32];              // the groups' scores and choices, then the chosen weights
    __shared__ int chosen[ROUTE_WARPS][NR * 32];
    griddep_launch();
    griddep_wait();
    const int t = blockIdx.x * ROUTE_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (t >= T) return;
    float* w_at = held[threadIdx.x >> 5];
    int* id_at = chosen[threadIdx.x >> 5];
    float s[NR];
    uint32_t key[NR];
    route_softmax<NR>(s, z + (size_t)t * E, E, lane);
#pragma unroll
    for (int j = 0; j < NR; ++j) key[j] = lane + 32 * j < E ? route_key(s[j]) : ROUTE_TAKEN;
    if (groups > 1 && keep < groups) {                        // only the `keep` best groups' experts may be chosen
        const int per = E / groups;
#pragma unroll
        for (int j = 0; j < NR; ++j) w_at[lane + 32 * j] = s[j];
        __syncwarp();
        uint32_t gkey[NR];
#pragma unroll
        for (int i = 0; i < NR; ++i) {
            const int g = lane + 32 * i;
            gkey[i] = ROUTE_TAKEN;
            if (g < groups) {
                float best = -INFINITY;
                for (int j = 0; j < per; ++j) best = fmaxf(best, w_at[g * per + j]);
                gkey[i] = route_key(best);
            }
        }
        for (int r = 0; r < keep; ++r) route_pick<NR>(gkey, lane);
        __syncwarp();
#pragma unroll
        for (int i = 0; i < NR; ++i) id_at[lane + 32 * i] = gkey[i] == ROUTE_TAKEN;
        __syncwarp();
#pragma unroll
        for (int j = 0; j < NR; ++j)
            if (lane + 32 * j < E && !id_at[(lane + 32 * j) / per]) key[j] = ROUTE_OUT;
        __syncwarp();
    }
    float wsum = 0.f;
    for (int r = 0; r < top; ++r) {
        const int e = route_pick<NR>(key, lane);
        const float w = route_score<NR>(s, e, lane);
        wsum += w;
        if (lane == 0) { id_at[r] = e; w_at[r] = w; }
    }
    __syncwarp();
    for (int r = lane; r < top; r += 32) {
        ids[(size_t)t * top + r] = id_at[r];
        wts[(size_t)t * top + r] = renorm ? w_at[r] / wsum : w_at[r];
        if (expert_count != nullptr) atomicAdd(expert_count + id_at[r], 1);     // for the plan of the grouped products
    }
}

// The router with a correction on the choice and experts that return their input.  s = softmax(z[t][0..E)) (rows ldz
// apart), or s = sigmoid(z) of every output by itself (`sigmoid`; without a correction the choice then goes by z, which has
// the same order and does not saturate); the `top` experts with the largest s + correction are chosen (ties to the lower index); a choice weighs s,
// divided by the sum of the chosen s plus renorm_eps when `renorm` is set.  Experts from `real` on have no tensors:
// their output is their input, so their weights are summed into w_same[t] and the choice is handed on as expert 0
// with weight zero (the expert products need no case for it).
template <int NR>
__global__ void __launch_bounds__(ROUTE_WARPS * 32)
moe_route_biased_kernel(const float* __restrict__ z, long ldz, int T, int E, int real, int top, int renorm, float renorm_eps,
                        const void* __restrict__ correction, int cdt, int sigmoid, int* __restrict__ ids, float* __restrict__ wts,
                        float* __restrict__ w_same, int* __restrict__ expert_count) {
    __shared__ float held[ROUTE_WARPS][NR * 32];
    __shared__ int chosen[ROUTE_WARPS][NR * 32];
    griddep_launch();
    const int t = blockIdx.x * ROUTE_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (t >= T) return;
    const float* zr = z + (size_t)t * ldz;
    float* w_at = held[threadIdx.x >> 5];
    int* id_at = chosen[threadIdx.x >> 5];
    float s[NR];
    uint32_t key[NR];
    if (!sigmoid) route_softmax<NR>(s, zr, E, lane);
#pragma unroll
    for (int j = 0; j < NR; ++j) {
        const int e = lane + 32 * j;
        key[j] = ROUTE_TAKEN;
        if (e < E) {
            const float v = sigmoid ? __ldcg(zr + e) : s[j];
            if (sigmoid) s[j] = 1.0f / (1.0f + expf(-v));
            key[j] = route_key(correction != nullptr ? s[j] + load_dyn(correction, cdt, e) : v);
        }
    }
    float wsum = 0.f;
    for (int r = 0; r < top; ++r) {
        const int e = route_pick<NR>(key, lane);
        const float w = route_score<NR>(s, e, lane);
        wsum += w;
        if (lane == 0) { id_at[r] = e; w_at[r] = w; }
    }
    __syncwarp();
    const float div = renorm ? wsum + renorm_eps : 1.0f;
    for (int r = lane; r < top; r += 32) {
        const float w = w_at[r] / div;
        const int e = id_at[r], to = e < real ? e : 0;
        w_at[r] = w;
        ids[(size_t)t * top + r] = to;
        wts[(size_t)t * top + r] = e < real ? w : 0.f;
        if (expert_count != nullptr) atomicAdd(expert_count + to, 1);
    }
    if (w_same == nullptr) return;
    __syncwarp();
    if (lane == 0) {
        float same = 0.f;
        if (real < E)
            for (int r = 0; r < top; ++r)
                if (id_at[r] >= real) same += w_at[r];
        w_same[t] = same;
    }
}

// BODY with NR bound: registers of a lane for E experts
#define ROUTE_DISPATCH(E, BODY)                             \
    do {                                                    \
        if ((E) <= 32) { constexpr int NR = 1; BODY; }      \
        else if ((E) <= 64) { constexpr int NR = 2; BODY; } \
        else if ((E) <= 128) { constexpr int NR = 4; BODY; }\
        else if ((E) <= 256) { constexpr int NR = 8; BODY; }\
        else { constexpr int NR = 32; BODY; }               \
    } while (0)

// ---------------------------------------------------------------- plain expert products
// One warp per output value; 8 warps a CTA take 8 consecutive output rows of one (token, choice).
// Row of w_up that makes gate (up: + up_step) number f of a gated expert: runs of `group` gate and up rows in turn, or all
// gate rows ahead of all up rows (group 0).
__device__ __forceinline__ int gated_row(int f, int F, int group, int* up_step) {
    *up_step = group > 0 ? group : F;
    return group > 0 ? (f / group) * 2 * group + f % group : f;
}

template <typename TH, typename TW, typename TO>
__global__ void __launch_bounds__(256)
moe_expert_up_kernel(const TH* __restrict__ h, long h_stride, const TW* __restrict__ w_up, const int* __restrict__ ids,
                     const float* __restrict__ in_wts, TO* __restrict__ act, int top, int D, int F, int act_kind, int gated, int group) {
    griddep_launch();
    griddep_wait();
    const int pair = blockIdx.x;                       // t * top + c
    const int t = pair / top;
    const int f = blockIdx.y * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (f >= F) return;
    const int e = __ldcg(ids + pair);
    const TH* hr = h + (size_t)t * h_stride;
    const float scale = in_wts != nullptr ? __ldcg(in_wts + pair) : 1.0f;
    if (gated) {
        int up_step;
        const int r = gated_row(f, F, group, &up_step);
        const TW* wg = w_up + ((size_t)e * 2 * F + r) * D;
        const TW* wu = wg + (size_t)up_step * D;
        float g = 0.f, u = 0.f;
        for (int i = lane; i < D; i += 32) {
            const float hv = ld_act(hr + i);
            g = fmaf(to_f(wg[i]), hv, g);
            u = fmaf(to_f(wu[i]), hv, u);
        }
        g = warp_sum(g) * scale;
        u = warp_sum(u) * scale;
        if (lane == 0) act[(size_t)pair * F + f] = from_f<TO>(g / (1.0f + expf(-g)) * u);
        return;
    }
    const TW* wr = w_up + ((size_t)e * F + f) * D;
    float acc = 0.f;
    for (int i = lane; i < D; i += 32) acc = fmaf(to_f(wr[i]), ld_act(hr + i), acc);
    acc = warp_sum(acc) * scale;
    if (lane == 0) act[(size_t)pair * F + f] = from_f<TO>(act_apply(acc, act_kind));
}

template <typename TA, typename TW>
__global__ void __launch_bounds__(256)
moe_expert_down_kernel(const TA* __restrict__ act, const TW* __restrict__ w_down, const int* __restrict__ ids,
                       const float* __restrict__ wts, float* __restrict__ parts, int T, int top, int D, int F) {
    griddep_launch();
    griddep_wait();
    const int pair = blockIdx.x;
    const int t = pair / top, c = pair - t * top;
    const int n = blockIdx.y * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (n >= D) return;
    const int e = __ldcg(ids + pair);
    const TW* wr = w_down + ((size_t)e * D + n) * F;
    const TA* ar = act + (size_t)pair * F;
    float acc = 0.f;
    for (int i = lane; i < F; i += 32) acc = fmaf(to_f(wr[i]), ld_act(ar + i), acc);
    acc = warp_sum(acc);
    if (lane == 0) parts[((size_t)c * T + t) * D + n] = acc * (wts != nullptr ? __ldcg(wts + pair) : 1.0f);
}

// ---------------------------------------------------------------- rows sorted by expert, for the grouped product
// Pair p = t * top + c chose expert ids[p].  Every expert's pairs get a run of rows that starts at a multiple of 128
// (the row tile of the grouped tensor-core product); the runs follow one another in expert order.
//   tile_group[i] = expert of row tile i (-1 beyond the last run, whose rows are not written at all);
//   row_dest[r] = c * T + t, the row of the [top, T, D] parts that the pair in row r belongs to (-1: padding);
//   row_scale[r] = the pair's weight;  a_sorted[r, :] = the pair's token's row of h.
// Which row of its run a pair gets depends on the order the threads arrive in; no result depends on it, since a row
// of a product depends on that row alone.
constexpr int SORT_THREADS = 1024;

// Two launches.  The router's choice has counted the pairs of every expert (expert_count).  moe_plan_rows (one CTA): the first row of every expert's run, a cursor
// into it, the experts of the row tiles, -1 as the destination of the padding rows; the counts are zeroed for the
// next step.  moe_place_rows (64 threads a pair): the pair takes the next row of its expert's run and its token's
// row of h is copied there, with the pair's destination and weight.  Padding rows of a_sorted are left as they are:
// a row of a product depends on that row alone, and their results are never stored.
__global__ void __launch_bounds__(SORT_THREADS)
moe_plan_rows_kernel(int* __restrict__ expert_count, int E, int max_tiles, int* __restrict__ cursor, int* __restrict__ tile_group,
                     int* __restrict__ row_dest) {
    __shared__ int count[ROUTE_MAX_EXPERTS];
    __shared__ int start[ROUTE_MAX_EXPERTS];
    __shared__ int used_rows;
    griddep_launch();
    griddep_wait();
    const int tid = threadIdx.x;
    for (int e = tid; e < E; e += SORT_THREADS) { count[e] = __ldcg(expert_count + e); expert_count[e] = 0; }
    __syncthreads();
    if (tid == 0) {
        int row = 0;
        for (int e = 0; e < E; ++e) {
            start[e] = row;
            row += (count[e] + 127) & ~127;
        }
        used_rows = row;
    }
    __syncthreads();
    for (int e = tid; e < E; e += SORT_THREADS) cursor[e] = start[e];
    for (int i = (used_rows >> 7) + tid; i < max_tiles; i += SORT_THREADS) tile_group[i] = -1;
    for (int e = tid; e < E; e += SORT_THREADS) {
        const int first = start[e] >> 7, n = (count[e] + 127) >> 7;
        for (int i = 0; i < n; ++i) tile_group[first + i] = e;
    }
    for (int e = tid >> 7; e < E; e += SORT_THREADS >> 7) {
        const int r = start[e] + count[e] + (tid & 127);
        if (r < start[e] + ((count[e] + 127) & ~127)) row_dest[r] = -1;
    }
}

__global__ void __launch_bounds__(256)
moe_place_rows_kernel(const __nv_bfloat16* __restrict__ h, long h_stride, const int* __restrict__ ids, const float* __restrict__ wts,
                      int* __restrict__ cursor, int P, int T, int top, __nv_bfloat16* __restrict__ a_sorted, int D,
                      int* __restrict__ row_dest, float* __restrict__ row_scale) {
    __shared__ int rows[4];
    griddep_launch();
    griddep_wait();
    const int sub = threadIdx.x >> 6, lane = threadIdx.x & 63;
    const int p = blockIdx.x * 4 + sub;
    if (p < P && lane == 0) {
        const int r = atomicAdd(cursor + __ldcg(ids + p), 1);
        const int t = p / top, c = p - t * top;
        row_dest[r] = c * T + t;
        row_scale[r] = __ldcg(wts + p);
        rows[sub] = r;
    }
    __syncthreads();
    if (p >= P) return;
    const int r = rows[sub];
    const int vec = D >> 3;
    const uint4* src = reinterpret_cast<const uint4*>(h + (size_t)(p / top) * h_stride);
    uint4* dst = reinterpret_cast<uint4*>(a_sorted + (size_t)r * D);
    for (int v0 = lane; v0 < vec; v0 += 256) {
        uint4 val[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int v = v0 + 64 * j;
            val[j] = v < vec ? __ldcg(src + v) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int v = v0 + 64 * j;
            if (v < vec) dst[v] = val[j];
        }
    }
}

// ---------------------------------------------------------------- expert products of a few tokens (bfloat16)
// A step that decodes brings few (token, choice) pairs, each with a whole expert's matrices to read:
// the products are bound by that stream.  One warp per output value, 16-byte loads, ROWS output rows
// of one pair per warp so that as many loads are in flight; K is a multiple of 8.
__device__ __forceinline__ float dot8(const uint4 w, const uint4 a) {
    const __nv_bfloat162* wp = reinterpret_cast<const __nv_bfloat162*>(&w);
    const __nv_bfloat162* ap = reinterpret_cast<const __nv_bfloat162*>(&a);
    float acc = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 wf = __bfloat1622float2(wp[j]), af = __bfloat1622float2(ap[j]);
        acc = fmaf(wf.x, af.x, acc);
        acc = fmaf(wf.y, af.y, acc);
    }
    return acc;
}

constexpr int SV_ROWS = 4;        // output rows per warp

// MODE 0: act[pair, f] = f(w[e, f, :] . x[pair / top, :])   (x = the tokens' rows, K = D)
//         (wts given: times wts[pair] before f)
// MODE 1: parts[c, t, n] = wts[pair] * (w[e, n, :] . x[pair, :])  (x = the pairs' hidden rows, K = F; wts null: no factor)
// MODE 2: a gated expert: rows of w as gated_row says, act[pair, f] = silu(gate) * up (wts given: both times wts[pair] first)
template <int MODE>
__global__ void __launch_bounds__(256)
moe_expert_rows_bf16_kernel(const __nv_bfloat16* __restrict__ x, long x_stride, const __nv_bfloat16* __restrict__ w,
                            const int* __restrict__ ids, const float* __restrict__ wts, void* __restrict__ out,
                            int T, int top, int N, int K, int act_kind, int group) {
    griddep_launch();
    constexpr int OUTS = MODE == 2 ? SV_ROWS / 2 : SV_ROWS;      // results a warp makes; a gated one takes two rows
    const int pair = blockIdx.x;
    const int lane = threadIdx.x & 31;
    const int n0 = (blockIdx.y * 8 + (threadIdx.x >> 5)) * OUTS;
    griddep_wait();
    if (n0 >= N) return;
    const int e = __ldcg(ids + pair);
    const int t = pair / top;
    const __nv_bfloat16* xr = x + (size_t)(MODE == 1 ? pair : t) * x_stride;
    const __nv_bfloat16* wr[SV_ROWS];
    bool in[SV_ROWS];
#pragma unroll
    for (int j = 0; j < SV_ROWS; ++j) {
        const int n = n0 + (MODE == 2 ? j >> 1 : j);
        in[j] = n < N;
        if (MODE == 2) {
            int up_step;
            const int r = gated_row(in[j] ? n : n0, N, group, &up_step);
            wr[j] = w + ((size_t)e * 2 * N + r + ((j & 1) ? up_step : 0)) * K;
        } else {
            wr[j] = w + ((size_t)e * N + (in[j] ? n : n0)) * K;
        }
    }
    float acc[SV_ROWS];
#pragma unroll
    for (int j = 0; j < SV_ROWS; ++j) acc[j] = 0.f;
    for (int k = lane * 8; k < K; k += 256) {
        const uint4 a = __ldcg(reinterpret_cast<const uint4*>(xr + k));
        uint4 wv[SV_ROWS];
#pragma unroll
        for (int j = 0; j < SV_ROWS; ++j)
            wv[j] = in[j] ? __ldg(reinterpret_cast<const uint4*>(wr[j] + k)) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int j = 0; j < SV_ROWS; ++j) acc[j] += dot8(wv[j], a);
    }
#pragma unroll
    for (int j = 0; j < SV_ROWS; ++j) acc[j] = warp_sum(acc[j]);
    if (lane == 0) {
        const float scale = wts != nullptr ? __ldcg(wts + pair) : 1.0f;
#pragma unroll
        for (int j = 0; j < OUTS; ++j) {
            if (n0 + j >= N) break;
            if (MODE == 0) {
                reinterpret_cast<__nv_bfloat16*>(out)[(size_t)pair * N + n0 + j] = __float2bfloat16_rn(act_apply(acc[j] * scale, act_kind));
            } else if (MODE == 2) {
                const float g = acc[2 * j] * scale, u = acc[2 * j + 1] * scale;
                reinterpret_cast<__nv_bfloat16*>(out)[(size_t)pair * N + n0 + j] = __float2bfloat16_rn(g / (1.0f + expf(-g)) * u);
            } else {
                const int c = pair - t * top;
                reinterpret_cast<float*>(out)[((size_t)c * T + t) * N + n0 + j] = acc[j] * scale;
            }
        }
    }
}

// The same results with every expert's matrix read once: a CTA has 16 rows of one expert's matrix and serves all pairs that chose
// it, sixteen at a time (a token chooses an expert once, but choices without tensors of their own arrive as expert 0 with
// weight zero), each of its four warps a quarter of the columns, on the tensor cores
// (mma.sync.m16n8k16, rows of W on the left, pairs on the right; both sides' columns in the order in which 16-byte loads give them).
// Sixteen products start from zero, eight of their sums meet in a tree, the trees (128 columns each) are added in float32, and so are the
// quarters, with what the tensor core cuts off a sum on the average added back.  Relative 2-norm of the down product's results against 64 bits,
// a row a pair and so: K = 1,024 6.7e-8 and 6.7e-8, 2,048 7.5e-8 and 7.3e-8, 4,096 8.7e-8 and 8.5e-8; numbers of one sign, K = 2,048
// 3.1e-8 and 2.9e-8 (every sum of sixteen added to one accumulator: 8.7e-8, 1.1e-7, 1.6e-7 and 5.4e-8).
// A CTA finds its pairs in the list of choices and leaves where there are none; `early`: the first
// columns of W are asked for before the kernel ahead has made the choices (where most experts are chosen).
// What bounds moe_expert_rows_bf16_kernel is instructions: two a number of W and pair (9 tokens, 4 of 16 gated experts of 2,048 x
// 1,024, 36 pairs: 33.6 and 31.6 us for the two products of 124 and 62 MB); 24 and 15 so.
constexpr int ET_WARPS = 4, ET_PAIRS = 16, ET_LIST = 256;       // pairs at a time; most pairs of a step
constexpr int ET_U = 2;                                         // k-steps of 64 whose loads are in flight together
constexpr float ET_LOST = 1.6e-8f;                              // what the tensor core cuts off a sum of sixteen products, on the average of its size

// sixteen products, from zero
__device__ __forceinline__ void et_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    d[0] = d[1] = d[2] = d[3] = 0.f;
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

struct EtTile { uint4 w[2][2]; };                               // row g, row g + 8; columns 16 c .. 16 c + 7, .. + 15 of a k-step

__device__ __forceinline__ void et_load(EtTile& t, const __nv_bfloat16* r0, const __nv_bfloat16* r1, int k, int K) {
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        const bool in = k + 8 * p < K;
        t.w[0][p] = in ? __ldg(reinterpret_cast<const uint4*>(r0 + k + 8 * p)) : make_uint4(0u, 0u, 0u, 0u);
        t.w[1][p] = in ? __ldg(reinterpret_cast<const uint4*>(r1 + k + 8 * p)) : make_uint4(0u, 0u, 0u, 0u);
    }
}

// The sums of ET_U k-steps' products, made from zero in a tree, are added to acc.  MODE as for moe_expert_rows_bf16_kernel.  NT: eights of pairs.
template <int NT>
__device__ __forceinline__ void et_products(float (&acc)[NT][4], const EtTile (&t)[ET_U], const __nv_bfloat16* const (&xr)[NT], const int (&k)[ET_U], int K) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        float sum[ET_U][4];
#pragma unroll
        for (int u = 0; u < ET_U; ++u) {
            float d[2][2][4];
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                const bool in = xr[nt] != nullptr && k[u] + 8 * p < K;
                const uint4 x = in ? __ldcg(reinterpret_cast<const uint4*>(xr[nt] + k[u] + 8 * p)) : make_uint4(0u, 0u, 0u, 0u);
                et_mma(d[p][0], t[u].w[0][p].x, t[u].w[1][p].x, t[u].w[0][p].y, t[u].w[1][p].y, x.x, x.y);
                et_mma(d[p][1], t[u].w[0][p].z, t[u].w[1][p].z, t[u].w[0][p].w, t[u].w[1][p].w, x.z, x.w);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) sum[u][e] = (d[0][0][e] + d[0][1][e]) + (d[1][0][e] + d[1][1][e]);
        }
        static_assert(ET_U == 2, "two sums");
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[nt][e] += sum[0][e] + sum[1][e];
    }
}

template <int MODE, int NT>
__device__ __forceinline__ void et_serve(const __nv_bfloat16* __restrict__ x, long x_stride, const __nv_bfloat16* r0, const __nv_bfloat16* r1, EtTile (&first)[ET_U],
                                         bool early, const int* pairs, int count, const float* __restrict__ wts, void* __restrict__ out, float* red, int row0,
                                         int T, int top, int N, int K, int act_kind, int s0, int s1) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
    const __nv_bfloat16* xr[NT];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        const int i = nt * 8 + g;
        xr[nt] = i < count ? x + (size_t)(MODE == 1 ? pairs[i] : pairs[i] / top) * x_stride : nullptr;
    }
    float acc[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
    for (int s = s0; s < s1; s += ET_U) {
        EtTile t[ET_U];
        int k[ET_U];
#pragma unroll
        for (int u = 0; u < ET_U; ++u) {
            k[u] = s + u < s1 ? (s + u) * 64 + c * 16 : K;
            if (early && s == s0) t[u] = first[u];
            else et_load(t[u], r0, r1, k[u], K);
        }
        et_products<NT>(acc, t, xr, k, K);
    }
    // [quarter][nt][e][lane]: thread (warp e, lane) adds the four quarters of its value; silu(gate) * up wants e and e + 2
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) red[((warp * NT + nt) * 4 + e) * 32 + lane] = acc[nt][e];
    __syncthreads();
    auto total = [&](int nt, int e) {
        const float* q = red + (nt * 4 + e) * 32 + lane;
        static_assert(ET_WARPS == 4, "four quarters");
        const float a = q[0] + q[NT * 128], b = q[2 * NT * 128] + q[3 * NT * 128], v = a + b, held = v - a;
        // with what a + b lost to rounding, so that less than half of a last place counts; an infinite sum stays one
        return fabsf(v) <= 3.402823466e38f ? v + fmaf(ET_LOST, v, (a - (v - held)) + (b - held)) : v;
    };
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        if (MODE == 2 && warp >= 2) break;
        const int i = nt * 8 + 2 * c + (warp & 1);                             // the pair; rows g (e = 0, 1) and g + 8 (e = 2, 3)
        if (i >= count) continue;
        const int pair = pairs[i];
        const float scale = wts != nullptr ? __ldcg(wts + pair) : 1.0f;
        if (MODE == 2) {
            const float gate = total(nt, warp) * scale, up = total(nt, warp + 2) * scale;
            const int f = row0 / 2 + g;
            if (f < N) reinterpret_cast<__nv_bfloat16*>(out)[(size_t)pair * N + f] = __float2bfloat16_rn(gate / (1.0f + expf(-gate)) * up);
            continue;
        }
        const int n = row0 + g + (warp >= 2 ? 8 : 0);
        if (n >= N) continue;
        const float v = total(nt, warp) * scale;
        if (MODE == 0) {
            reinterpret_cast<__nv_bfloat16*>(out)[(size_t)pair * N + n] = __float2bfloat16_rn(act_apply(v, act_kind));
        } else {
            const int t = pair / top;
            reinterpret_cast<float*>(out)[((size_t)(pair - t * top) * T + t) * N + n] = v;
        }
    }
}

template <int MODE>
__global__ void __launch_bounds__(ET_WARPS * 32)
moe_expert_tiles_kernel(const __nv_bfloat16* __restrict__ x, long x_stride, const __nv_bfloat16* __restrict__ w, const int* __restrict__ ids,
                        const float* __restrict__ wts, void* __restrict__ out, int T, int top, int N, int K, int act_kind, int early, int per) {
    __shared__ int pairs[ET_LIST];
    __shared__ int s_count;
    __shared__ float red[2][ET_WARPS * 2 * 4 * 32];                            // of a tile and the one after it
    griddep_launch();
    const int e = blockIdx.y, P = T * top, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
    const int rows = MODE == 2 ? 2 * N : N, tiles = (rows + 15) / 16, tile0 = blockIdx.x * per, tile1 = tile0 + per < tiles ? tile0 + per : tiles;
    const __nv_bfloat16* we = w + (size_t)e * rows * K;
    // rows beyond the last are computed and not stored
    auto row = [&](int tile, int r) { return we + (size_t)(tile * 16 + r < rows ? tile * 16 + r : 0) * K; };
    const int steps = (K + 63) / 64, s0 = steps * warp / ET_WARPS, s1 = steps * (warp + 1) / ET_WARPS;
    EtTile first[ET_U];
    if (early) {
#pragma unroll
        for (int u = 0; u < ET_U; ++u) et_load(first[u], row(tile0, g), row(tile0, g + 8), s0 + u < s1 ? (s0 + u) * 64 + c * 16 : K, K);
    }
    griddep_wait();
    if (warp == 0) {
        int n = 0;
        for (int base = 0; base < P; base += 32) {
            const bool hit = base + lane < P && __ldcg(ids + base + lane) == e;
            const uint32_t m = __ballot_sync(0xffffffffu, hit);
            if (hit) pairs[n + __popc(m & ((1u << lane) - 1u))] = base + lane;
            n += __popc(m);
        }
        if (lane == 0) s_count = n;
    }
    __syncthreads();
    const int count = s_count;
    if (count == 0) return;
    int turn = 0;
    for (int tile = tile0; tile < tile1; ++tile)
        for (int p0 = 0; p0 < count; p0 += ET_PAIRS, turn ^= 1) {
            const bool asked = early && tile == tile0 && p0 == 0;
            const int n = count - p0 < ET_PAIRS ? count - p0 : ET_PAIRS;
            if (n <= 8) et_serve<MODE, 1>(x, x_stride, row(tile, g), row(tile, g + 8), first, asked, pairs + p0, n, wts, out, red[turn], tile * 16, T, top, N, K, act_kind, s0, s1);
            else et_serve<MODE, 2>(x, x_stride, row(tile, g), row(tile, g + 8), first, asked, pairs + p0, n, wts, out, red[turn], tile * 16, T, top, N, K, act_kind, s0, s1);
        }
}

template <typename T>
__global__ void act_rows_kernel(T* __restrict__ a, size_t n, int act_kind) {
    griddep_launch();
    griddep_wait();
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        a[i] = from_f<T>(act_apply(ld_act(a + i), act_kind));
}

}  // namespace aien

using namespace aien;

// expert_count (may be null): E ints that hold zero on entry; every choice adds one to its expert's
// (aien_moe_plan_rows reads them and leaves zeros behind).
AIEN_API int aien_moe_route(const float* z, int T, int E, int groups, int keep, int top, int renorm, int* ids, float* wts,
                            int* expert_count, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (E <= 0 || E > ROUTE_MAX_EXPERTS || groups <= 0 || E % groups != 0 || keep <= 0 || keep > groups || top <= 0 ||
        top > keep * (E / groups)) return AIEN_E_SHAPE;
    ROUTE_DISPATCH(E, (launch_chain(moe_route_kernel<NR>, dim3((unsigned)((T + ROUTE_WARPS - 1) / ROUTE_WARPS)), dim3(ROUTE_WARPS * 32), (size_t)0, stream, z, T, E,
                                    groups, keep, top, renorm, ids, wts, expert_count)));
    return launch_status();
}

// z float32 [T, ldz]: the first E numbers of a row are the router's; correction [E] in c_dt (or null); experts from
// `real` on return their input (w_same float32 [T], needed when real < E).
AIEN_API int aien_moe_route_biased(const float* z, long ldz, int T, int E, int real, int top, int renorm, float renorm_eps,
                                   const void* correction, int c_dt, int sigmoid, int* ids, float* wts, float* w_same, int* expert_count,
                                   cudaStream_t stream) {
    if (T <= 0) return 0;
    if (E <= 0 || E > ROUTE_MAX_EXPERTS || real <= 0 || real > E || top <= 0 || top > E || (real < E && w_same == nullptr)) return AIEN_E_SHAPE;
    ROUTE_DISPATCH(E, (moe_route_biased_kernel<NR><<<(unsigned)((T + ROUTE_WARPS - 1) / ROUTE_WARPS), ROUTE_WARPS * 32, 0, stream>>>(      // plain: see griddep_wait
        z, ldz, T, E, real, top, renorm, renorm_eps, correction, c_dt, sigmoid, ids, wts, w_same, expert_count)));
    return launch_status();
}

// h [T, D] (row stride h_stride), w_up [E, F, D], act [T * top, F]; act_kind 0: erf gelu, 1: tanh gelu, 2: relu squared.
// gated != 0: w_up [E, 2F, D] with gate and up rows in runs of `group` (0: all gate rows first).  in_wts [T * top] or null:
// the pair's weight multiplies the expert's input.
AIEN_API int aien_moe_expert_up(const void* h, int h_dt, long h_stride, const void* w_up, int w_dt, const int* ids, const float* in_wts,
                                void* act, int act_dt, int T, int top, int D, int F, int act_kind, int gated, int group, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (T * (long)top > 2147483647L || D <= 0 || F <= 0 || (F + 7) / 8 > 65535 || group < 0 || (group > 0 && F % group)) return AIEN_E_SHAPE;
    dim3 grid(T * top, (F + 7) / 8);
    AIEN_DISPATCH_DTYPE(h_dt, TH, AIEN_DISPATCH_DTYPE(w_dt, TW, AIEN_DISPATCH_DTYPE(act_dt, TO,
        (launch_chain(moe_expert_up_kernel<TH, TW, TO>, grid, dim3(256), 0, stream,
                      (const TH*)h, h_stride, (const TW*)w_up, ids, in_wts, (TO*)act, top, D, F, act_kind, gated, group)))));
    return launch_status();
}

// act [T * top, F], w_down [E, D, F], parts float32 [top, T, D].
AIEN_API int aien_moe_expert_down(const void* act, int act_dt, const void* w_down, int w_dt, const int* ids, const float* wts,
                                  float* parts, int T, int top, int D, int F, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (T * (long)top > 2147483647L || D <= 0 || F <= 0 || (D + 7) / 8 > 65535) return AIEN_E_SHAPE;
    dim3 grid(T * top, (D + 7) / 8);
    AIEN_DISPATCH_DTYPE(act_dt, TA, AIEN_DISPATCH_DTYPE(w_dt, TW,
        (launch_chain(moe_expert_down_kernel<TA, TW>, grid, dim3(256), 0, stream,
                      (const TA*)act, (const TW*)w_down, ids, wts, parts, T, top, D, F))));
    return launch_status();
}

// expert_count: what aien_moe_route counted (left zero); cursor: E ints of scratch; tile_group: max_tiles; row_dest: max_tiles * 128.
AIEN_API int aien_moe_plan_rows(int* expert_count, int E, int max_tiles, int* cursor, int* tile_group, int* row_dest, cudaStream_t stream) {
    if (E <= 0 || E > ROUTE_MAX_EXPERTS || max_tiles <= 0) return AIEN_E_SHAPE;
    launch_chain(moe_plan_rows_kernel, dim3(1), dim3(SORT_THREADS), 0, stream, expert_count, E, max_tiles, cursor, tile_group, row_dest);
    return launch_status();
}

AIEN_API int aien_moe_place_rows(const void* h, long h_stride, const int* ids, const float* wts, int* cursor, int T, int top,
                                 void* a_sorted, int D, int* row_dest, float* row_scale, cudaStream_t stream) {
    if (T <= 0) return 0;
    const long P = (long)T * top;
    if (top <= 0 || P > 2147483647L / 2) return AIEN_E_SHAPE;
    if (D <= 0 || (D & 7) || (h_stride & 7) || ((uintptr_t)h & 15) || ((uintptr_t)a_sorted & 15)) return AIEN_E_ALIGN;
    launch_chain(moe_place_rows_kernel, dim3((unsigned)((P + 3) / 4)), dim3(256), 0, stream, (const __nv_bfloat16*)h, h_stride, ids, wts,
                 cursor, (int)P, T, top, (__nv_bfloat16*)a_sorted, D, row_dest, row_scale);
    return launch_status();
}

// The expert products of a few tokens, bfloat16: mode 0 = up with activation (out bfloat16 [T*top, N], K = D), mode 2 = the
// same for gated experts (w [E, 2N, K], runs of `group` gate and up rows), in both wts (or null) multiplies the input; mode 1 =
// down into float32 parts [top, T, N] (K = F) times wts (or null).  K a multiple of 8, 16-byte aligned rows.
AIEN_API int aien_moe_expert_rows_bf16(int mode, const void* x, long x_stride, const void* w, const int* ids, const float* wts,
                                       void* out, int T, int top, int E, int N, int K, int act_kind, int group, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (N <= 0 || K <= 0 || (K & 7) || (x_stride & 7) || ((uintptr_t)x & 15) || ((uintptr_t)w & 15)) return AIEN_E_ALIGN;
    const int outs = 8 * (mode == 2 ? SV_ROWS / 2 : SV_ROWS);
    const int tiles = (N + outs - 1) / outs;
    if (tiles > 65535 || (long)T * top > 2147483647L || group < 0 || (group > 0 && N % group)) return AIEN_E_SHAPE;
    // Every expert's matrix once for all its pairs where enough pairs share an expert, by the experts that T tokens reach on the
    // average: 1.4 pairs an expert and more.  us, a row a pair and an expert's tile (up and down product): 16 gated experts of
    // 2,048 x 1,024, 4 a token, 4 tokens (1.5 pairs) 21.5 and 21.2, 13.9 and 13.2; 9 (2.4) 33.0 and 24.5, 23.7 and 15.2; 16 49.7 and 26.5, 34.9
    // and 15.7; 64 of 2,048 x 768, 6 a token, 4 tokens (1.2) 18.4 and 16.2, 16.6 and 19.7; 9 (1.4) 33.0 and 24.4, 28.2 and 28.1; 16 56.6 and
    // 33.7, 44.4 and 38.9.  More experts than 64 (128, 8 a token, 16 tokens, 1.6 pairs: 85 and 87) cost their CTAs.
    double missed = 1.0;
    for (int t = 0; t < T && t <= ET_PAIRS; ++t) missed *= 1.0 - (double)(top < E ? top : E) / (E > 0 ? E : 1);
    const double reached = (1.0 - missed) * E;
    if (E > 0 && E <= 64 && T <= ET_PAIRS && T * top <= ET_LIST && (mode != 2 || group == 8) && (double)T * top >= 1.4 * reached) {
        const int early = T * top >= 2 * E;          // most experts are chosen: a CTA need not wait for the choices to ask for its first rows
        // A tile of a short K is over before its CTA has found its pairs, so a CTA takes two or four in turn while a thousand CTAs are left
        // (64 experts, 9 tokens, K = 768: 34.9 us with one, 29.3 with two, 28.1 with four)
        const long tiles16 = ((mode == 2 ? 2L * N : N) + 15) / 16;
        const int per = K > 1024 || tiles16 * reached < 2048 ? 1 : tiles16 * reached < 4096 ? 2 : 4;
        const dim3 tile_grid((unsigned)((tiles16 + per - 1) / per), E);
#define ME_CASE(M)                                                                                                       \
    launch_chain(moe_expert_tiles_kernel<M>, tile_grid, dim3(ET_WARPS * 32), 0, stream, (const __nv_bfloat16*)x, x_stride, \
                 (const __nv_bfloat16*)w, ids, wts, out, T, top, N, K, act_kind, early, per)
        if (mode == 0) ME_CASE(0);
        else if (mode == 2) ME_CASE(2);
        else ME_CASE(1);
#undef ME_CASE
        return launch_status();
    }
    dim3 grid(T * top, tiles);
#define MR_CASE(M)                                                                                                       \
    launch_chain(moe_expert_rows_bf16_kernel<M>, grid, dim3(256), 0, stream, (const __nv_bfloat16*)x, x_stride,           \
                 (const __nv_bfloat16*)w, ids, wts, out, T, top, N, K, act_kind, group)
    if (mode == 0) MR_CASE(0);
    else if (mode == 2) MR_CASE(2);
    else MR_CASE(1);
#undef MR_CASE
    return launch_status();
}

AIEN_API int aien_act_rows(void* a, int dt, size_t n, int act_kind, cudaStream_t stream) {
    if (n == 0) return 0;
    const int blocks = (int)((n + 255) / 256 < 148 * 16 ? (n + 255) / 256 : 148 * 16);
    AIEN_DISPATCH_DTYPE(dt, TT, (launch_chain(act_rows_kernel<TT>, dim3(blocks), dim3(256), 0, stream, (TT*)a, n, act_kind)));
    return launch_status();
}
