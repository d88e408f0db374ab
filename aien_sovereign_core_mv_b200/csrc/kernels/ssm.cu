// State-space recurrences with a float32 state per request: the selective scan (a state per channel) and the
// state-space-duality form (a state matrix per head), and the gate and grouped norm that follows the latter.
//
//   selective scan   per channel c and state n, token by token:
//                      dt = softplus(dtz[c] + dt_bias[c]);
//                      S[c][n] = exp(dt * A[c][n]) * S[c][n] + dt * x[c] * B[n];
//                      y[c] = sum_n S[c][n] * C[n] + D[c] * x[c];  out[c] = y[c] * silu(z[c])
//   duality form     per head h (group g = h / (heads / groups)) with S [N][V], token by token:
//                      dt = softplus(dtr[h] + dt_bias[h]) and exp(-A[h] * dt) (made once per token and head, likewise);
//                      S = exp(-A[h] * dt) * S + dt * B[g] x[h]^T;  y[h] = S^T C[g] + D[h] * x[h]
//   gate and norm    v = y * silu(z); every one of `groups` equal parts of the row divided by its own root mean
//                    square (eps inside the root), times the weight, times a constant
//
// The state of request s lives in row slot_map[s] of `state` (rows of state_stride floats, the recurrence's part from
// s_off on); a portion whose first token has position 0 starts from zeros.  A few neighbouring lanes own a channel (or a
// column of a head's state), keep its N state values in registers between them and walk the portion's tokens in order: a
// token's result depends only on the tokens before it.  The order of the float32 additions in it may depend on the step: the
// scan has eight or sixteen lanes a channel by the channels of all its requests, a step of single tokens four, and whether
// portions are cut into segments goes by the step's size too.
// Everything here is float32 in both engine precisions; only the result leaves in the compute dtype, and where that is
// bfloat16 the scan's decays come from the special-function unit (see decay_exp).
//
// The portion-parallel forms cut a portion into segments that run side by side: every segment first runs from a zero
// state and records the product of its decays and its end state; the segments' starting states then follow one from
// another; a second pass repeats the segment from its true starting state and writes the results.
#include "common.cuh"
#include "gated_rows.cuh"
#include <math.h>

namespace aien {

__device__ __forceinline__ float ssm_silu(float z) { return z / (1.0f + expf(-z)); }
__device__ __forceinline__ float ssm_softplus(float a) { return a > 20.f ? a : log1pf(expf(a)); }

constexpr int SSM_THREADS = 128;

// mode 0: the whole portion from the slot's state, results and new state written (the plain form).
// mode 1: segment `blockIdx.z` of the portion from zeros; writes its decay product and end state to scratch.
// mode 2: segment from the state the combine step left for it; writes results (the combine step wrote the slot).
struct Segments {
    int mode;
    int seg_len;
    float* decay;       // [segments][lanes]   product of the decays over the segment
    float* end;         // [segments][lanes]   mode 1: end state from zeros; after the combine: the state at the segment's end
    int nseg;           // the most segments one portion has (grid z); request s's segments start at q_start[s] / seg_len + s
};

// ---- the selective scan
// LANES neighbouring lanes share one channel: lane ln keeps the CH state values n = ln * CH .. ln * CH + CH - 1 in
// registers (N <= LANES * CH) and walks the portion's tokens in order.  One request has few walkers (4,096 channels with
// 8 lanes are two warps a scheduler), so what bounds a walk is the length of a token's dependent instructions, then their
// number (at the limit one exponential per token and state value, 16 a clock and SM).  Hence:
//   * the rows of a stage of tokens arrive in shared memory by cp.async while the stage before is worked on;
//   * all that does not depend on the state is made for the whole stage before and after its walk, by all threads: the
//     step size (softplus) and its product with x before, the sum over a channel's lanes, the skip and the gate after;
//   * inside the walk, eight tokens at a time, only one multiply-add a state value depends on the token before.
// 2,048 tokens of 4,096 channels with 16 states each, one request, B200: 764 us, and 26 us for the step sizes, with the
// rows fetched into registers four tokens ahead; 147 us so, 7 of them the gate's exponential and division
// (31 instructions a token and warp, of which half a dozen in the prologue and epilogue of a stage; 16 lanes: 180 us, 4: 216 us).
// With few channels a portion is cut into segments (see kernels.selective_scan_segments): 126 us with four lanes a channel, of
// which the passes take 50 and 70; there 68 and 72 % of the issue slots are used (36 and 54 instructions a token and warp of eight
// channels) and 66 and 53 % of the special-function unit (profiles/layer_kernels__ncu_counters.md).
template <int LANES, int CH>
struct ScanCfg {
    static constexpr int NP = LANES * CH;
    static constexpr int TOKENS = NP > 32 || LANES == 4 ? 16 : 32;      // of a stage; two stages and the sums fit in 48 KB
    static constexpr int CPB = SSM_THREADS / LANES;                     // channels of a CTA
    static constexpr int ROWS = TOKENS * CPB;                           // one of dt, x, z
    static constexpr int STAGE = 3 * ROWS + TOKENS * 2 * NP;            // dt | x | z | (B | C) per token
};

__device__ __forceinline__ void scan_cp(float* dst, const float* src, bool wide, bool in) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    if (wide) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(in ? 16 : 0) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(in ? 4 : 0) : "memory");
}

struct ScanRowsIn {
    const float* x; long ldx; const float* dtz; long lddt; const float* bc; long ldbc; int b_off, c_off; const float* z; long ldz;
    bool wide, wide_bc;
};

// The rows of tokens t .. t + TOKENS - 1 of channels c0 .. c0 + CPB - 1, in pieces of UNIT (dt, x, z) and UBC (B, C)
// numbers; zeros behind t1 and behind the last channel.  FIRST: no z and no C, which only results need.
template <int LANES, int CH, int UNIT, int UBC, bool FIRST>
__device__ __forceinline__ void scan_fetch_units(float* __restrict__ buf, const ScanRowsIn& in, int c0, int inner, int N, int t, int t1) {
    using C = ScanCfg<LANES, CH>;
    constexpr int per = C::CPB / UNIT, pb = C::NP / UBC, pr = FIRST ? pb : 2 * pb;
    const float* src[3] = {in.dtz, in.x, in.z};
    const long ld[3] = {in.lddt, in.ldx, in.ldz};
#pragma unroll
    for (int a = 0; a < (FIRST ? 2 : 3); ++a)
#pragma unroll 1
        for (int i = threadIdx.x; i < C::TOKENS * per; i += SSM_THREADS) {
            const int tok = i / per, c = i % per * UNIT;
            const bool ok = t + tok < t1 && c0 + c < inner;
            scan_cp(buf + a * C::ROWS + tok * C::CPB + c, ok ? src[a] + (t + tok) * ld[a] + c0 + c : src[a], UNIT == 4, ok);
        }
    float* rows = buf + 3 * C::ROWS;
#pragma unroll 1
    for (int i = threadIdx.x; i < C::TOKENS * pr; i += SSM_THREADS) {
        const int tok = i / pr, r = i % pr, which = r >= pb, n = (r - which * pb) * UBC;
        const bool ok = t + tok < t1 && n < N;
        scan_cp(rows + tok * 2 * C::NP + which * C::NP + n, ok ? in.bc + (t + tok) * in.ldbc + (which ? in.c_off : in.b_off) + n : in.bc, UBC == 4, ok);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

template <int LANES, int CH, bool FIRST>
__device__ __forceinline__ void scan_fetch(float* __restrict__ buf, const ScanRowsIn& in, int c0, int inner, int N, int t, int t1) {
    if (in.wide && in.wide_bc) scan_fetch_units<LANES, CH, 4, 4, FIRST>(buf, in, c0, inner, N, t, t1);
    else if (in.wide_bc) scan_fetch_units<LANES, CH, 1, 4, FIRST>(buf, in, c0, inner, N, t, t1);
    else scan_fetch_units<LANES, CH, 1, 1, FIRST>(buf, in, c0, inner, N, t, t1);
}

// exp for the decays: full precision where the result leaves in float32; through the special-function unit (relative
// error near 2^-21) where it leaves in bfloat16, whose own rounding is a hundred times coarser.  There the rate comes
// times log2(e).
template <typename TO> __device__ __forceinline__ float decay_rate(float a) { return a; }
template <> __device__ __forceinline__ float decay_rate<__nv_bfloat16>(float a) { return a * 1.4426950408889634f; }
template <typename TO> __device__ __forceinline__ float decay_exp(float v) { return expf(v); }
template <> __device__ __forceinline__ float decay_exp<__nv_bfloat16>(float v) {
    float e;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(v));
    return e;
}

// FIRST: the first pass over segments (Segments, mode 1): no results, and a channel's decay over the segment is one exponential
// a state value of the sum of its step sizes.
template <int LANES, int CH, bool FIRST, typename TO>
__global__ void __launch_bounds__(SSM_THREADS)
selective_scan_kernel(ScanRowsIn in, const float* __restrict__ A, const void* __restrict__ dt_bias, const void* __restrict__ D, int pdt,
                      float* __restrict__ state, size_t state_stride, size_t s_off, const int* __restrict__ slots,
                      const int* __restrict__ q_start, const int* __restrict__ positions, TO* __restrict__ out, long ldo, int inner, int N, Segments sg) {
    using C = ScanCfg<LANES, CH>;
    constexpr int U = 8;
    __shared__ __align__(16) float bufs[2][C::STAGE];
    __shared__ __align__(16) float2 steps[C::ROWS];                    // (dt, dt * x) per token and channel
    __shared__ __align__(16) float sums[C::TOKENS * SSM_THREADS];      // a lane's part of y per token
    const int s = blockIdx.y, seg = sg.mode == 0 ? 0 : blockIdx.z;
    griddep_launch();
    griddep_wait();
    int t0 = __ldcg(q_start + s), t1 = __ldcg(q_start + s + 1);
    if (t1 <= t0) return;
    const bool fresh = __ldcg(positions + t0) == 0;
    const size_t seg0 = sg.mode == 0 ? 0 : (size_t)(t0 / sg.seg_len + s);         // the request's first segment in the scratch
    if (sg.mode != 0) {
        t0 += seg * sg.seg_len;
        if (t0 >= t1) return;                                           // a segment beyond the portion's end
        if (t0 + sg.seg_len < t1) t1 = t0 + sg.seg_len;
    }
    const int cl = threadIdx.x / LANES, ln = threadIdx.x % LANES, n0 = ln * CH;
    const int c0 = blockIdx.x * C::CPB, c = c0 + cl < inner ? c0 + cl : inner - 1;      // lanes beyond the last channel write nothing
    const bool live = c0 + cl < inner;
    scan_fetch<LANES, CH, FIRST>(bufs[0], in, c0, inner, N, t0, t1);
    float* st = state + (size_t)slots[s] * state_stride + s_off + (size_t)c * N + n0;
    const size_t so = ((seg0 + seg) * inner + c) * N + n0;
    const float* init = sg.mode == 2 ? (seg > 0 ? sg.end + so - (size_t)inner * N : sg.decay + so) : st;      // see segment_combine_kernel
    const bool zero = FIRST || (sg.mode == 0 && fresh);
    float S[CH], a[CH], dts = 0.f;
#pragma unroll
    for (int i = 0; i < CH; ++i) {
        const bool in_n = n0 + i < N;
        a[i] = in_n ? decay_rate<TO>(A[(size_t)c * N + n0 + i]) : 0.f;
        S[i] = (in_n && !zero) ? init[i] : 0.f;
    }
    // outside the walk a thread serves channel threadIdx.x % CPB of every LANES-th token
    const int ec = threadIdx.x % C::CPB, e0 = threadIdx.x / C::CPB;
    const int eg = c0 + ec < inner ? c0 + ec : inner - 1;
    const float dskip = load_dyn(D, pdt, eg), bias = load_dyn(dt_bias, pdt, eg);
    int b = 0;
    for (int t = t0; t < t1; t += C::TOKENS, b ^= 1) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (t + C::TOKENS < t1) scan_fetch<LANES, CH, FIRST>(bufs[b ^ 1], in, c0, inner, N, t + C::TOKENS, t1);
        const int n_tok = t1 - t < C::TOKENS ? t1 - t : C::TOKENS;
        const float* rows = bufs[b];
#pragma unroll
        for (int k = 0; k < C::TOKENS / LANES; ++k) {
            const int tok = e0 + k * LANES, i = tok * C::CPB + ec;
            const float dt = tok < n_tok ? ssm_softplus(rows[i] + bias) : 0.f;
            steps[i] = make_float2(dt, dt * rows[C::ROWS + i]);
        }
        __syncthreads();
        const float* sbc = rows + 3 * C::ROWS + n0;
        auto token = [&](int tok) {                                     // the lane's part of y
            const float2 dd = steps[tok * C::CPB + cl];
            const float* br = sbc + tok * 2 * C::NP;
            if (FIRST) dts += dd.x;
            if (CH % 2 == 0) {
                float2 ys = make_float2(0.f, 0.f);
                __align__(16) float bv[CH], cv[CH];
#pragma unroll
                for (int i = 0; i < CH; i += CH % 4 == 0 ? 4 : 2) {
                    if (CH % 4 == 0) {
                        *reinterpret_cast<float4*>(bv + i) = *reinterpret_cast<const float4*>(br + i);
                        if (!FIRST) *reinterpret_cast<float4*>(cv + i) = *reinterpret_cast<const float4*>(br + C::NP + i);
                    } else {
                        *reinterpret_cast<float2*>(bv + i) = *reinterpret_cast<const float2*>(br + i);
                        if (!FIRST) *reinterpret_cast<float2*>(cv + i) = *reinterpret_cast<const float2*>(br + C::NP + i);
                    }
                }
#pragma unroll
                for (int i = 0; i < CH; i += 2) {
                    const float2 b2 = make_float2(bv[i], bv[(i + 1) % CH]), c2 = FIRST ? b2 : make_float2(cv[i], cv[(i + 1) % CH]);
                    const float2 p = __fmul2_rn(make_float2(dd.x, dd.x), make_float2(a[i], a[(i + 1) % CH]));
                    const float2 e = make_float2(decay_exp<TO>(p.x), decay_exp<TO>(p.y));
                    const float2 S2 = __ffma2_rn(e, make_float2(S[i], S[(i + 1) % CH]), __fmul2_rn(make_float2(dd.y, dd.y), b2));
                    S[i] = S2.x; S[(i + 1) % CH] = S2.y;
                    if (!FIRST) ys = __ffma2_rn(S2, c2, ys);
                }
                return ys.x + ys.y;
            }
            float y = 0.f;
#pragma unroll
            for (int i = 0; i < CH; ++i) {
                S[i] = fmaf(decay_exp<TO>(dd.x * a[i]), S[i], dd.y * br[i]);
                if (!FIRST) y = fmaf(S[i], br[C::NP + i], y);
            }
            return y;
        };
        int g = 0;
        for (; g + U <= n_tok; g += U) {
            float y[U];
#pragma unroll
            for (int u = 0; u < U; ++u) y[u] = token(g + u);
#pragma unroll
            for (int u = 0; u < U; ++u) if (!FIRST) sums[(g + u) * SSM_THREADS + threadIdx.x] = y[u];
        }
        // the rest of a portion; the tokens behind its end have no step: 0 times an infinite rate is no decay
#pragma unroll 1
        for (; g < n_tok; ++g) {
            const float y = token(g);
            if (!FIRST) sums[g * SSM_THREADS + threadIdx.x] = y;
        }
        if (FIRST) continue;
        __syncthreads();
        if (c0 + ec < inner) {
#pragma unroll
            for (int k = 0; k < C::TOKENS / LANES; ++k) {
                const int tok = e0 + k * LANES, i = tok * C::CPB + ec;
                const float4* p = reinterpret_cast<const float4*>(sums + tok * SSM_THREADS + ec * LANES);
                float y = 0.f;
#pragma unroll
                for (int j = 0; j < LANES / 4; ++j) { const float4 v = p[j]; y += (v.x + v.y) + (v.z + v.w); }
                if (tok < n_tok) out[(size_t)(t + tok) * ldo + c0 + ec] = from_f<TO>(fmaf(dskip, rows[C::ROWS + i], y) * ssm_silu(rows[2 * C::ROWS + i]));
            }
        }
    }
    if (!live || sg.mode == 2) return;
#pragma unroll
    for (int i = 0; i < CH; ++i)
        if (n0 + i < N) {
            if (FIRST) { sg.decay[so + i] = decay_exp<TO>(dts * a[i]); sg.end[so + i] = S[i]; }
            else st[i] = S[i];
        }
}

// One token a request (as many tokens as requests): a thread group lives for one token, so what counts is how many are resident and how much each
// moves.  Four (sixteen) lanes a channel, no shared memory; 64 requests x 4,096 channels x 16 states (33.5 MB of
// state read and written): 12.8 us with float4 moves and 15.9 without, against 17.5 us with the step sizes in a launch of their own and
// 52 us for the walk's kernel.
// VEC: a lane's state values, rates, B and C as float4 (they lie on 16-byte boundaries and N = LANES CH).
template <int LANES, int CH, bool VEC, typename TO>
__global__ void __launch_bounds__(SSM_THREADS)
selective_scan_token_kernel(ScanRowsIn in, const float* __restrict__ A, const void* __restrict__ dt_bias, const void* __restrict__ D, int pdt,
                            float* __restrict__ state, size_t state_stride, size_t s_off, const int* __restrict__ slots,
                            const int* __restrict__ q_start, const int* __restrict__ positions, TO* __restrict__ out, long ldo, int inner, int N) {
    const int s = blockIdx.y, t0 = q_start[s], t1 = q_start[s + 1], gid = blockIdx.x * SSM_THREADS + threadIdx.x;
    if (t1 <= t0) return;
    const bool live = gid / LANES < inner;
    const int c = live ? gid / LANES : inner - 1, ln = gid % LANES, n0 = ln * CH;   // lanes beyond the last channel repeat it and write nothing
    float* st = state + (size_t)slots[s] * state_stride + s_off + (size_t)c * N + n0;
    const bool zero = positions[t0] == 0;
    __align__(16) float S[CH], a[CH];
    if (VEC) {
#pragma unroll
        for (int i = 0; i < CH; i += 4) {
            *reinterpret_cast<float4*>(S + i) = zero ? make_float4(0.f, 0.f, 0.f, 0.f) : *reinterpret_cast<const float4*>(st + i);
            *reinterpret_cast<float4*>(a + i) = *reinterpret_cast<const float4*>(A + (size_t)c * N + n0 + i);
        }
#pragma unroll
        for (int i = 0; i < CH; ++i) a[i] = decay_rate<TO>(a[i]);
    } else {
#pragma unroll
        for (int i = 0; i < CH; ++i) {
            const bool ok = n0 + i < N;
            S[i] = (ok && !zero) ? st[i] : 0.f;
            a[i] = ok ? decay_rate<TO>(A[(size_t)c * N + n0 + i]) : 0.f;
        }
    }
    int t = t0;
    do {                                            // once, unless a step of as many tokens as requests has an empty request beside a portion
        const float* br = in.bc + t * in.ldbc + in.b_off + n0;
        const float* cr = in.bc + t * in.ldbc + in.c_off + n0;
        __align__(16) float bv[CH], cv[CH];
        if (VEC) {
#pragma unroll
            for (int i = 0; i < CH; i += 4) {
                *reinterpret_cast<float4*>(bv + i) = *reinterpret_cast<const float4*>(br + i);
                *reinterpret_cast<float4*>(cv + i) = *reinterpret_cast<const float4*>(cr + i);
            }
        } else {
#pragma unroll
            for (int i = 0; i < CH; ++i) {
                const bool ok = n0 + i < N;
                bv[i] = ok ? br[i] : 0.f;
                cv[i] = ok ? cr[i] : 0.f;
            }
        }
        const float x = in.x[t * in.ldx + c], z = in.z[t * in.ldz + c];
        const float dt = ssm_softplus(in.dtz[t * in.lddt + c] + load_dyn(dt_bias, pdt, c)), dx = dt * x;
        float y = 0.f;
#pragma unroll
        for (int i = 0; i < CH; ++i) {
            S[i] = fmaf(decay_exp<TO>(dt * a[i]), S[i], dx * bv[i]);
            y = fmaf(S[i], cv[i], y);
        }
#pragma unroll
        for (int o = 1; o < LANES; o <<= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
        if (ln == 0 && live) out[t * ldo + c] = from_f<TO>(fmaf(load_dyn(D, pdt, c), x, y) * ssm_silu(z));
    } while (++t < t1);
    if (!live) return;
    if (VEC) {
#pragma unroll
        for (int i = 0; i < CH; i += 4) *reinterpret_cast<float4*>(st + i) = *reinterpret_cast<const float4*>(S + i);
    } else {
#pragma unroll
        for (int i = 0; i < CH; ++i) if (n0 + i < N) st[i] = S[i];
    }
}

// Between the two passes: end[k] becomes the state at the end of segment k with the true start, one after another;
// the state the portion started from moves into decay[0] (the second pass reads no slot) and the state after the
// portion's last token into the slot.  lanes = values per request (inner * N, or heads * N * V).
__global__ void __launch_bounds__(256)
segment_combine_kernel(float* __restrict__ state, size_t state_stride, size_t s_off, const int* __restrict__ slots,
                       const int* __restrict__ q_start, const int* __restrict__ positions, Segments sg, size_t lanes) {
    const int s = blockIdx.y;
    const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
    griddep_launch();
    griddep_wait();
    if (i >= lanes) return;
    const int t0 = q_start[s], n_tok = q_start[s + 1] - t0;
    if (n_tok <= 0) return;
    const int used = (n_tok + sg.seg_len - 1) / sg.seg_len;
    const size_t seg0 = (size_t)(t0 / sg.seg_len + s);
    float* slot = state + (size_t)slots[s] * state_stride + s_off + i;
    const float init = positions[t0] == 0 ? 0.f : *slot;
    float cur = init;
    for (int k = 0; k < used; ++k) {
        const size_t o = (seg0 + k) * lanes + i;
        cur = fmaf(sg.decay[o], cur, sg.end[o]);
        sg.end[o] = cur;
    }
    sg.decay[seg0 * lanes + i] = init;
    *slot = cur;
}

// steps[t][h] = softplus(dtr[t][h] + bias[h]) and steps[t][heads + h] = exp(-A[h] * that): once per token and head.
__global__ void __launch_bounds__(256)
ssd_steps_kernel(const float* __restrict__ dtr, long lddt, const float* __restrict__ A, const void* __restrict__ bias, int pdt,
                 float* __restrict__ steps, int T, int heads) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    griddep_launch();
    griddep_wait();
    if (i >= T * heads) return;
    const int t = i / heads, h = i - t * heads;
    const float dt = ssm_softplus(ld_act(dtr + (size_t)t * lddt + h) + load_dyn(bias, pdt, h));
    steps[(size_t)t * 2 * heads + h] = dt;
    steps[(size_t)t * 2 * heads + heads + h] = expf(-A[h] * dt);
}

// LANES neighbouring lanes share one (head, value column): lane ln keeps the CH state values n = ln * CH .. ln * CH + CH - 1
// of S[:, v] in registers (N <= LANES * CH) and the partial sums of y meet by shuffles.  The slot holds S as
// [heads][value column][N], so the lanes read one contiguous row.  VEC: B, C and the state move as float4.  U tokens are
// fetched ahead of their arithmetic.
constexpr int SSD_THREADS = 256;

template <int LANES, int CH, int U, bool VEC>
__global__ void __launch_bounds__(SSD_THREADS)
ssd_scan_kernel(const float* __restrict__ xbc, long ld, int x_off, int b_off, int c_off,
                const float* __restrict__ steps, const void* __restrict__ D, int pdt, float* __restrict__ state, size_t state_stride, size_t s_off,
                const int* __restrict__ slots, const int* __restrict__ q_start, const int* __restrict__ positions,
                float* __restrict__ y_out, long ldy, int heads, int V, int G, int N, Segments sg, int longest) {
    const int s = blockIdx.y, gid = blockIdx.x * SSD_THREADS + threadIdx.x;
    const int cols = heads * V;
    const bool live = gid / LANES < cols;
    const int col = live ? gid / LANES : cols - 1, ln = gid % LANES;       // lanes beyond the last column repeat it and write nothing
    const int h = col / V, g = h / (heads / G), n0 = ln * CH;
    int t0 = q_start[s];
    int t1 = q_start[s + 1];
    if (t1 <= t0 || t1 - t0 > longest) return;
    const bool fresh = positions[t0] == 0;
    const int seg = sg.mode == 0 ? 0 : blockIdx.z;
    const size_t seg0 = sg.mode == 0 ? 0 : (size_t)(t0 / sg.seg_len + s);
    if (sg.mode != 0) {
        t0 += seg * sg.seg_len;
        if (t0 + sg.seg_len < t1) t1 = t0 + sg.seg_len;              // a segment beyond the portion's end walks no token
    }
    float* st = state + (size_t)slots[s] * state_stride + s_off + (size_t)col * N + n0;
    const size_t lanes = (size_t)cols * N;
    const size_t so = (seg0 + seg) * lanes + (size_t)col * N + n0;
    const bool mine = t0 < t1 || sg.mode == 0;
    float S[CH];
    float P = 1.f;
    const float* init = sg.mode == 2 ? (seg > 0 ? sg.end + so - lanes : sg.decay + so) : st;
    const bool zero = !mine || sg.mode == 1 || (sg.mode == 0 && fresh);
    if (VEC) {
#pragma unroll
        for (int i = 0; i < CH; i += 4) {
            float4 v4 = make_float4(0.f, 0.f, 0.f, 0.f);
            if (!zero && n0 + i < N) v4 = *reinterpret_cast<const float4*>(init + i);
            S[i] = v4.x;
            if (i + 1 < CH) S[i + 1] = v4.y;
            if (i + 2 < CH) S[i + 2] = v4.z;
            if (i + 3 < CH) S[i + 3] = v4.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < CH; ++i) S[i] = (!zero && n0 + i < N) ? init[i] : 0.f;
    }
    const float dskip = load_dyn(D, pdt, h);
    for (int t = t0; t < t1; t += U) {
        float dtu[U], eu[U], xu[U], bv[U][CH], cv[U][CH];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int tt = t + u < t1 ? t + u : t1 - 1;
            dtu[u] = steps[(size_t)tt * 2 * heads + h];
            eu[u] = steps[(size_t)tt * 2 * heads + heads + h];
            xu[u] = xbc[(size_t)tt * ld + x_off + col];
            const float* br = xbc + (size_t)tt * ld + b_off + (size_t)g * N + n0;
            const float* cr = xbc + (size_t)tt * ld + c_off + (size_t)g * N + n0;
            if (VEC) {
#pragma unroll
                for (int i = 0; i < CH; i += 4) {
                    float4 b4 = make_float4(0.f, 0.f, 0.f, 0.f), c4 = b4;
                    if (n0 + i < N) { b4 = *reinterpret_cast<const float4*>(br + i); c4 = *reinterpret_cast<const float4*>(cr + i); }
                    bv[u][i] = b4.x; cv[u][i] = c4.x;
                    if (i + 1 < CH) { bv[u][i + 1] = b4.y; cv[u][i + 1] = c4.y; }
                    if (i + 2 < CH) { bv[u][i + 2] = b4.z; cv[u][i + 2] = c4.z; }
                    if (i + 3 < CH) { bv[u][i + 3] = b4.w; cv[u][i + 3] = c4.w; }
                }
            } else {
#pragma unroll
                for (int i = 0; i < CH; ++i) { const bool in = n0 + i < N; bv[u][i] = in ? br[i] : 0.f; cv[u][i] = in ? cr[i] : 0.f; }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (t + u < t1) {
                const float e = eu[u], dx = dtu[u] * xu[u];
                float y = 0.f;
#pragma unroll
                for (int i = 0; i < CH; ++i) {
                    S[i] = fmaf(e, S[i], dx * bv[u][i]);
                    y = fmaf(S[i], cv[u][i], y);
                }
                if (sg.mode == 1) {
                    P *= e;
                } else {
#pragma unroll
                    for (int o = 1; o < LANES; o <<= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
                    if (ln == 0 && live) y_out[(size_t)(t + u) * ldy + col] = fmaf(dskip, xu[u], y);
                }
            }
        }
    }
    if (!live || !mine) return;
    if (sg.mode == 1) {
#pragma unroll
        for (int i = 0; i < CH; ++i) if (n0 + i < N) { sg.decay[so + i] = P; sg.end[so + i] = S[i]; }
    } else if (sg.mode == 0) {
#pragma unroll
        for (int i = 0; i < CH; ++i) if (n0 + i < N) st[i] = S[i];
    }
}

// The duality form where a request brings one token and a state column 128 numbers: what counts is the state, read and written
// once, and how much of it is on its way at a time.  A warp has eight columns of a head, a float4 of each a lane, all requested
// before the token's numbers, and makes the head's step size and decay itself; the eight sums over the lanes are folded
// together (nine shuffles, added in the order of a butterfly a column).  64 requests x 32 heads of 64 x 128 (134 MB of
// state read and written), B200: 51 us with one column a warp, and 2 for the steps
// in a launch of their own; 24 us so (5.6 TB/s).
constexpr int SSD_TOKEN_COLS = 8;

__global__ void __launch_bounds__(SSD_THREADS)
ssd_token_kernel(const float* __restrict__ xbc, long ld, int x_off, int b_off, int c_off, const float* __restrict__ dtr, long lddt,
                 const float* __restrict__ A, const void* __restrict__ dt_bias, const void* __restrict__ D, int pdt,
                 float* __restrict__ state, size_t state_stride, size_t s_off, const int* __restrict__ slots, const int* __restrict__ q_start,
                 const int* __restrict__ positions, float* __restrict__ y_out, long ldy, int heads, int V, int G, int longest) {
    constexpr int COLS = SSD_TOKEN_COLS, N = 128;
    const int s = blockIdx.y, lane = threadIdx.x & 31, col0 = (blockIdx.x * (SSD_THREADS / 32) + (threadIdx.x >> 5)) * COLS;
    const int t0 = q_start[s], t1 = q_start[s + 1];
    if (t1 <= t0 || t1 - t0 > longest || col0 >= heads * V) return;
    const int h = col0 / V, g = h / (heads / G);
    float* st = state + (size_t)slots[s] * state_stride + s_off + (size_t)col0 * N + lane * 4;
    const bool fresh = positions[t0] == 0;
    float4 S[COLS];
#pragma unroll
    for (int i = 0; i < COLS; ++i) S[i] = fresh ? make_float4(0.f, 0.f, 0.f, 0.f) : *reinterpret_cast<const float4*>(st + i * N);
    const float dskip = load_dyn(D, pdt, h), rate = -A[h], bias = load_dyn(dt_bias, pdt, h);
    for (int t = t0; t < t1; ++t) {                 // once, unless a step of as many tokens as requests has an empty request beside a portion
        const float* row = xbc + (size_t)t * ld;
        const float4 b = *reinterpret_cast<const float4*>(row + b_off + (size_t)g * N + lane * 4);
        const float4 c = *reinterpret_cast<const float4*>(row + c_off + (size_t)g * N + lane * 4);
        const float x = row[x_off + col0 + (lane & (COLS - 1))];
        const float dt = ssm_softplus(dtr[(size_t)t * lddt + h] + bias), e = expf(rate * dt);
        float y[COLS];
#pragma unroll
        for (int i = 0; i < COLS; ++i) {
            const float dx = dt * __shfl_sync(0xffffffffu, x, i);
            S[i].x = fmaf(e, S[i].x, dx * b.x);
            S[i].y = fmaf(e, S[i].y, dx * b.y);
            S[i].z = fmaf(e, S[i].z, dx * b.z);
            S[i].w = fmaf(e, S[i].w, dx * b.w);
            y[i] = fmaf(S[i].w, c.w, fmaf(S[i].z, c.z, fmaf(S[i].y, c.y, S[i].x * c.x)));
        }
        // lane bits 0, 1, 2 choose the column (4, 2, 1) that the lane goes on with
#pragma unroll
        for (int k = COLS / 2, bit = 1; k > 0; k >>= 1, bit <<= 1) {
            const bool upper = lane & bit;
#pragma unroll
            for (int i = 0; i < k; ++i) {
                const float mine = upper ? y[i + k] : y[i], other = upper ? y[i] : y[i + k];
                y[i] = mine + __shfl_xor_sync(0xffffffffu, other, bit);
            }
        }
        float sum = y[0] + __shfl_xor_sync(0xffffffffu, y[0], 8);
        sum += __shfl_xor_sync(0xffffffffu, sum, 16);
        const int col = (lane & 1) * 4 + (lane & 2) + ((lane >> 2) & 1);
        const float xc = __shfl_sync(0xffffffffu, x, col);
        if (lane < COLS) y_out[(size_t)t * ldy + col0 + col] = fmaf(dskip, xc, sum);
    }
#pragma unroll
    for (int i = 0; i < COLS; ++i) *reinterpret_cast<float4*>(st + i * N) = S[i];
}

// out[t] = the three bfloat16 parts of x[t]'s numbers, part by part: x = p0 + p1 + p2 up to 2^-25 of x (each part rounds
// what the ones before leave).  With the weights three times side by side a product on the tensor cores then has float32
// rows on the left (parts_product.cu).  x may come as partial products over ranges of K: the product that makes it has
// few columns (160 over 4,096: 32 tiles at 2,048 tokens, 28 us) and is cut over the whole GPU (14 us, and 1.7 more here).
__global__ void __launch_bounds__(256)
split_rows_kernel(const float* __restrict__ x, long ldx, int P, size_t part_stride, __nv_bfloat16* __restrict__ out, float* __restrict__ rest,
                  int T, int n, int m) {
    const long i = (long)blockIdx.x * 256 + threadIdx.x;
    griddep_launch();
    griddep_wait();
    if (i >= (long)T * (n + m)) return;
    const int t = (int)(i / (n + m)), c = (int)(i - (long)t * (n + m));
    const float* xc = x + t * ldx + c;
    float v = ld_act(xc);
    for (int p0 = 1; p0 < P; p0 += 4) {                         // partial products in order, four loads in flight
        float w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = p0 + j < P ? ld_act(xc + (p0 + j) * part_stride) : 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) v += w[j];
    }
    if (c >= n) {
        rest[(size_t)t * m + c - n] = v;
        return;
    }
    __nv_bfloat16 p0 = __float2bfloat16_rn(v);
    if (fabsf(__bfloat162float(p0)) == INFINITY && fabsf(v) < INFINITY) p0 = __float2bfloat16_rz(v);        // the largest numbers round beyond the type
    const float r0 = fabsf(v) < INFINITY ? v - __bfloat162float(p0) : 0.f;                                  // an infinity (or NaN) is whole in its first part
    const __nv_bfloat16 p1 = __float2bfloat16_rn(r0);
    __nv_bfloat16* o = out + (size_t)t * 3 * n + c;
    o[0] = p0;
    o[n] = p1;
    o[2 * n] = __float2bfloat16_rn(r0 - __bfloat162float(p1));
}

// out[t][o_off + c] = (y * silu(z))[c] / rms(part of c) * w[c] * mult; one CTA per (token, part)
template <typename TO>
__global__ void __launch_bounds__(256)
gate_group_norm_kernel(const float* __restrict__ y, long ldy, const float* __restrict__ z, long ldz, const void* __restrict__ w, int wdt,
                       float eps, float mult, TO* __restrict__ out, long ldo, int part) {
    __shared__ float red[32];
    const int t = blockIdx.x, c0 = blockIdx.y * part;
    float ss = 0.f;
    for (int i = threadIdx.x; i < part; i += 256) {
        const float v = y[(size_t)t * ldy + c0 + i] * ssm_silu(z[(size_t)t * ldz + c0 + i]);
        ss = fmaf(v, v, ss);
    }
    const float r = mult / sqrtf(block_sum(ss, red) / (float)part + eps);
    for (int i = threadIdx.x; i < part; i += 256) {
        const float v = y[(size_t)t * ldy + c0 + i] * ssm_silu(z[(size_t)t * ldz + c0 + i]);
        out[(size_t)t * ldo + c0 + i] = from_f<TO>(v * r * load_dyn(w, wdt, c0 + i));
    }
}

}  // namespace aien

using namespace aien;

// Floats of scratch that the portion-parallel forms need: T tokens of S requests in segments of seg_len tokens.
AIEN_API long aien_ssm_segments_scratch(int T, int S, int seg_len, long lanes) { return 2L * (T / seg_len + S) * lanes; }

struct ScanArgs {
    ScanRowsIn in; const float* A; const void* dt_bias; const void* D; int p_dt; float* state; size_t state_stride, s_off; const int* slots;
    const int* q_start; const int* positions; void* out; long ldo; int T, S, inner, N; Segments sg; cudaStream_t stream;
};

template <int LANES, int CH, typename TO>
static void launch_selective_scan(const ScanArgs& a) {
    using C = ScanCfg<LANES, CH>;
    Segments sg = a.sg;
    const dim3 grid((unsigned)((a.inner + C::CPB - 1) / C::CPB), a.S, sg.mode == 0 ? 1 : sg.nseg);
    const long ctas = (long)grid.x * grid.y * grid.z;
    auto pass = [&](auto kern, int resident) {
        if (sg.mode != 0 && fills_gpu(ctas, resident))                  // see griddep_wait
            launch_chain(kern, grid, dim3(SSM_THREADS), (size_t)0, a.stream, a.in, a.A, a.dt_bias, a.D, a.p_dt, a.state, a.state_stride, a.s_off, a.slots, a.q_start,
                         a.positions, (TO*)a.out, a.ldo, a.inner, a.N, sg);
        else
            kern<<<grid, SSM_THREADS, 0, a.stream>>>(a.in, a.A, a.dt_bias, a.D, a.p_dt, a.state, a.state_stride, a.s_off, a.slots, a.q_start, a.positions, (TO*)a.out,
                                                     a.ldo, a.inner, a.N, sg);
    };
    if (sg.mode != 0) {
        const size_t lanes = (size_t)a.inner * a.N;
        static const int resident = resident_ctas(selective_scan_kernel<LANES, CH, true, TO>, SSM_THREADS, 0);
        pass(selective_scan_kernel<LANES, CH, true, TO>, resident);
        launch_chain(segment_combine_kernel, dim3((unsigned)((lanes + 255) / 256), a.S), dim3(256), (size_t)0, a.stream, a.state, a.state_stride, a.s_off, a.slots,
                     a.q_start, a.positions, sg, lanes);
        sg.mode = 2;
    }
    static const int resident = resident_ctas(selective_scan_kernel<LANES, CH, false, TO>, SSM_THREADS, 0);
    pass(selective_scan_kernel<LANES, CH, false, TO>, resident);
}

template <int LANES, int CH, typename TO>
static void launch_selective_scan_token(const ScanArgs& a) {
    const unsigned gx = (unsigned)(((long)a.inner * LANES + SSM_THREADS - 1) / SSM_THREADS);
    const bool vec = CH % 4 == 0 && a.N == LANES * CH && a.in.wide_bc && ((a.state_stride | a.s_off) & 3) == 0 &&
                     ((reinterpret_cast<uintptr_t>(a.state) | reinterpret_cast<uintptr_t>(a.A)) & 15) == 0;
    const auto kern = vec ? selective_scan_token_kernel<LANES, CH, CH % 4 == 0, TO> : selective_scan_token_kernel<LANES, CH, false, TO>;
    kern<<<dim3(gx, a.S), SSM_THREADS, 0, a.stream>>>(
        a.in, a.A, a.dt_bias, a.D, a.p_dt, a.state, a.state_stride, a.s_off, a.slots, a.q_start, a.positions, (TO*)a.out, a.ldo, a.inner, a.N);
}

// Eight lanes a channel; with fewer than 2,048 channels in the step, whose walkers would leave SM schedulers without a
// warp, and with many state values, sixteen.  In segments of 16 states beyond 512 channels four with four states each, whose
// instructions per state are fewer: segments are of one length, so what counts is their number.  Whole portions keep eight: their longest
// one may be all that still walks, and four lanes take half as long again a token (4,096 channels, us with eight and four: requests of
// 900, 100, 100 and 100 tokens 83 and 113, of 700, 500 and 300 77 and 93; three of 500 88 and 76, which the step's sizes do not tell apart).
// In segments of up to 512 channels eight from 512 tokens on (1,024 tokens: 26 us with sixteen, 23).
template <typename TO>
static int dispatch_selective_scan(const ScanArgs& a) {
    const int N = a.N;
    const bool few = (long)a.inner * a.S < 2048;
    if (N > 128) return AIEN_E_SHAPE;
    if (a.T == a.S) {
        if (N <= 4) launch_selective_scan_token<4, 1, TO>(a);
        else if (N <= 8) launch_selective_scan_token<4, 2, TO>(a);
        else if (N <= 16) launch_selective_scan_token<4, 4, TO>(a);
        else if (N <= 32) launch_selective_scan_token<4, 8, TO>(a);
        else if (N <= 64) launch_selective_scan_token<16, 4, TO>(a);
        else launch_selective_scan_token<16, 8, TO>(a);
        return 0;
    }
    if (N <= 8) launch_selective_scan<8, 1, TO>(a);
    else if (N <= 16) {
        const long channels = (long)a.inner * a.S;
        const bool few_cut = channels <= 512 && a.T >= 512L * a.S;
        if (a.sg.mode != 0 && channels > 512) launch_selective_scan<4, 4, TO>(a);
        else if (few && !(a.sg.mode != 0 && few_cut)) launch_selective_scan<16, 1, TO>(a);
        else launch_selective_scan<8, 2, TO>(a);
    }
    else if (N <= 32) { if (few) launch_selective_scan<16, 2, TO>(a); else launch_selective_scan<8, 4, TO>(a); }
    else if (N <= 64) launch_selective_scan<16, 4, TO>(a);
    else launch_selective_scan<16, 8, TO>(a);
    return 0;
}

// x [T, ldx] (after convolution and silu), dtz [T, lddt] = W_dt dt before its bias, bc [T, ldbc] with B at b_off and C at
// c_off (N numbers each, N <= 128), z [T, ldz] the gate's input, A float32 [inner, N] (negative rates), dt_bias and D
// [inner] in p_dt.  T is the number of tokens in the step.  seg_len > 0: portions are cut into nseg segments of seg_len tokens
// that run side by side (scratch float32, aien_ssm_segments_scratch(T, S, seg_len, inner * N) numbers); nseg * seg_len must cover
// the longest portion.
AIEN_API int aien_selective_scan(const float* x, long ldx, const float* dtz, long lddt, const float* bc, long ldbc, int b_off, int c_off,
                                 const float* z, long ldz, const float* A, const void* dt_bias, const void* D, int p_dt,
                                 float* state, size_t state_stride, size_t s_off, const int* slots, const int* q_start,
                                 const int* positions, void* out, int o_dt, long ldo, int T, int S, int inner, int N,
                                 int seg_len, int nseg, float* scratch, cudaStream_t stream) {
    if (S <= 0 || T <= 0) return 0;
    if (inner <= 0 || N <= 0 || S > 65535 || nseg > 65535) return AIEN_E_SHAPE;
    Segments sg{0, 0, nullptr, nullptr, 1};
    if (seg_len > 0 && nseg > 1) {
        if (scratch == nullptr) return AIEN_E_SHAPE;
        sg = Segments{1, seg_len, scratch, scratch + (size_t)(T / seg_len + S) * (size_t)inner * N, nseg};
    }
    const bool wide = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(dtz) | reinterpret_cast<uintptr_t>(z)) & 15) == 0 &&
                      ((ldx | lddt | ldz | inner) & 3) == 0;
    const bool wide_bc = (reinterpret_cast<uintptr_t>(bc) & 15) == 0 && ((ldbc | b_off | c_off | N) & 3) == 0;
    const ScanArgs a{{x, ldx, dtz, lddt, bc, ldbc, b_off, c_off, z, ldz, wide, wide_bc}, A, dt_bias, D, p_dt, state, state_stride, s_off, slots,
                     q_start, positions, out, ldo, T, S, inner, N, sg, stream};
    int rc = 0;
    AIEN_DISPATCH_DTYPE(o_dt, TO, (rc = dispatch_selective_scan<TO>(a)));
    if (rc != 0) return rc;
    return launch_status();
}

// steps [T][2 * heads]: the step sizes softplus(dtr + dt_bias) and the decays exp(-A * that) of a step's tokens.
AIEN_API int aien_ssd_steps(const float* dtr, long lddt, const float* A, const void* dt_bias, int p_dt, float* steps, int T, int heads,
                            cudaStream_t stream) {
    if (T <= 0 || heads <= 0) return T == 0 ? 0 : AIEN_E_SHAPE;
    launch_chain(ssd_steps_kernel, dim3((unsigned)(((long)T * heads + 255) / 256)), dim3(256), (size_t)0, stream, dtr, lddt, A, dt_bias, p_dt, steps, T, heads);
    return launch_status();
}

struct SsdArgs {
    const float* xbc; long ld; int x_off, b_off, c_off; const float* dtr; long lddt; const float* A; const void* dt_bias; const void* D;
    int p_dt; float* state; size_t state_stride, s_off; const int* slots; const int* q_start; const int* positions; float* y; long ldy;
    int T, S, heads, V, G, N; Segments sg; int longest; float* steps; cudaStream_t stream;
};

template <int LANES, int CH, int U, bool VEC>
static void launch_ssd_scan(const SsdArgs& a) {
    auto kern = ssd_scan_kernel<LANES, CH, U, VEC>;
    const long threads = (long)a.heads * a.V * LANES;
    const unsigned gx = (unsigned)((threads + SSD_THREADS - 1) / SSD_THREADS);
    Segments sg = a.sg;
    const dim3 grid(gx, a.S, sg.mode == 0 ? 1 : sg.nseg);
    ssd_steps_kernel<<<(unsigned)(((long)a.T * a.heads + 255) / 256), 256, 0, a.stream>>>(a.dtr, a.lddt, a.A, a.dt_bias, a.p_dt, a.steps, a.T, a.heads);
    kern<<<grid, SSD_THREADS, 0, a.stream>>>(a.xbc, a.ld, a.x_off, a.b_off, a.c_off, a.steps, a.D, a.p_dt, a.state,
                                             a.state_stride, a.s_off, a.slots, a.q_start, a.positions, a.y, a.ldy, a.heads, a.V, a.G, a.N, sg, a.longest);
    if (sg.mode == 0) return;
    const size_t lanes = (size_t)a.heads * a.N * a.V;
    segment_combine_kernel<<<dim3((unsigned)((lanes + 255) / 256), a.S), 256, 0, a.stream>>>(a.state, a.state_stride, a.s_off, a.slots, a.q_start,
                                                                                             a.positions, sg, lanes);
    sg.mode = 2;
    kern<<<grid, SSD_THREADS, 0, a.stream>>>(a.xbc, a.ld, a.x_off, a.b_off, a.c_off, a.steps, a.D, a.p_dt, a.state,
                                             a.state_stride, a.s_off, a.slots, a.q_start, a.positions, a.y, a.ldy, a.heads, a.V, a.G, a.N, sg, a.longest);
}

// xbc [T, ld] (after convolution and silu): x (heads * V) at x_off, B (G * N) at b_off, C (G * N) at c_off; dtr [T, lddt]
// the raw step sizes, one per head; A float32 [heads] (positive rates exp(A_log)); dt_bias and D [heads] in p_dt;
// y float32 [T, ldy]; N <= 256; steps: float32 scratch of T * 2 * heads numbers (the step sizes and decays of the step's
// tokens).  The slot holds S as [heads][V][N].  Segments as for aien_selective_scan, with heads * N * V state values per
// request.  longest > 0: requests that bring more tokens are served elsewhere and left alone here (but for their steps).
AIEN_API int aien_ssd_scan(const float* xbc, long ld, int x_off, int b_off, int c_off, const float* dtr, long lddt, const float* A,
                           const void* dt_bias, const void* D, int p_dt, float* state, size_t state_stride, size_t s_off,
                           const int* slots, const int* q_start, const int* positions, float* y, long ldy, int T, int S, int heads, int V,
                           int G, int N, int seg_len, int nseg, float* scratch, float* steps, int longest, cudaStream_t stream) {
    if (S <= 0 || T <= 0) return 0;
    if (longest <= 0) longest = 0x7fffffff;
    if (heads <= 0 || V <= 0 || G <= 0 || heads % G || N <= 0 || N > 256 || S > 65535 || nseg > 65535 || steps == nullptr) return AIEN_E_SHAPE;
    Segments sg{0, 0, nullptr, nullptr, 1};
    if (seg_len > 0 && nseg > 1) {
        if (scratch == nullptr) return AIEN_E_SHAPE;
        sg = Segments{1, seg_len, scratch, scratch + (size_t)(T / seg_len + S) * (size_t)heads * N * V, nseg};
    }
    const SsdArgs a{xbc, ld, x_off, b_off, c_off, dtr, lddt, A, dt_bias, D, p_dt, state, state_stride, s_off, slots, q_start, positions,
                    y, ldy, T, S, heads, V, G, N, sg, longest, steps, stream};
    // float4 moves: every lane's first state value, B and C value on a 16-byte boundary, whole groups of four inside N
    const bool vec = N >= 128 && N % 4 == 0 && ld % 4 == 0 && b_off % 4 == 0 && c_off % 4 == 0 && state_stride % 4 == 0 && s_off % 4 == 0 &&
                     ((uintptr_t)xbc & 15) == 0 && ((uintptr_t)state & 15) == 0 && (scratch == nullptr || ((uintptr_t)scratch & 15) == 0);
    if ((T == S || longest == 1) && vec && N == 128 && V % SSD_TOKEN_COLS == 0) {
        if (T != S) ssd_steps_kernel<<<(unsigned)(((long)T * heads + 255) / 256), 256, 0, stream>>>(dtr, lddt, A, dt_bias, p_dt, steps, T, heads);
        const unsigned gx = (unsigned)(((long)heads * V / SSD_TOKEN_COLS + SSD_THREADS / 32 - 1) / (SSD_THREADS / 32));
        ssd_token_kernel<<<dim3(gx, S), SSD_THREADS, 0, stream>>>(xbc, ld, x_off, b_off, c_off, dtr, lddt, A, dt_bias, D, p_dt, state, state_stride,
                                                                  s_off, slots, q_start, positions, y, ldy, heads, V, G, longest);
        return launch_status();
    }
    if (T == S || longest == 1) {                     // single tokens: no rows fetched ahead (fewer registers, more CTAs resident)
        if (N <= 8) launch_ssd_scan<8, 1, 1, false>(a);
        else if (N <= 16) launch_ssd_scan<8, 2, 1, false>(a);
        else if (N <= 32) launch_ssd_scan<32, 1, 1, false>(a);
        else if (N <= 64) launch_ssd_scan<32, 2, 1, false>(a);
        else if (N <= 128) { if (vec) launch_ssd_scan<32, 4, 1, true>(a); else launch_ssd_scan<32, 4, 1, false>(a); }
        else { if (vec && N % 8 == 0) launch_ssd_scan<32, 8, 1, true>(a); else launch_ssd_scan<32, 8, 1, false>(a); }
        return launch_status();
    }
    if (N <= 8) launch_ssd_scan<8, 1, 4, false>(a);
    else if (N <= 16) launch_ssd_scan<8, 2, 4, false>(a);
    else if (N <= 32) launch_ssd_scan<32, 1, 4, false>(a);
    else if (N <= 64) launch_ssd_scan<32, 2, 4, false>(a);
    else if (N <= 128) { if (vec) launch_ssd_scan<32, 4, 4, true>(a); else launch_ssd_scan<32, 4, 4, false>(a); }
    else { if (vec && N % 8 == 0) launch_ssd_scan<32, 8, 2, true>(a); else launch_ssd_scan<32, 8, 2, false>(a); }
    return launch_status();
}

// x float32 [T, ldx] (or P partial products of it, part_stride numbers apart); out bfloat16 [T, 3 n] of the first n columns,
// rest float32 [T, m] (may be null with m = 0) the m columns behind them.
AIEN_API int aien_split_rows(const float* x, long ldx, int P, size_t part_stride, void* out, float* rest, int T, int n, int m, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (n <= 0 || m < 0 || P < 1 || (m > 0 && rest == nullptr) || ((long)T * (n + m) + 255) / 256 > 2147483647L) return AIEN_E_SHAPE;
    launch_chain(split_rows_kernel, dim3((unsigned)(((long)T * (n + m) + 255) / 256)), dim3(256), (size_t)0, stream, x, ldx, P, part_stride, (__nv_bfloat16*)out, rest, T,
                 n, m);
    return launch_status();
}

// y float32 [T, ldy], z float32 [T, ldz] (the gate's input), w [width] in w_dt; the row is `groups` equal parts.
// out [T, ldo] in o_dt = (y * silu(z)) / rms(its part) * w * mult.
AIEN_API int aien_gate_group_norm(const float* y, long ldy, const float* z, long ldz, const void* w, int w_dt, float eps, float mult,
                                  void* out, int o_dt, long ldo, int T, int width, int groups, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (groups <= 0 || width <= 0 || width % groups || groups > 65535) return AIEN_E_SHAPE;
    const int part = width / groups;
    AIEN_DISPATCH_DTYPE(o_dt, TO,
        if (gated_rows_take(y, ldy, z, ldz, (const TO*)out, ldo, part))
            launch_gated_rows<true>(y, ldy, z, ldz, w, w_dt, eps, mult, (TO*)out, ldo, T, groups, part, stream);
        else
            (gate_group_norm_kernel<TO><<<dim3(T, groups), 256, 0, stream>>>(y, ldy, z, ldz, w, w_dt, eps, mult, (TO*)out, ldo, part)));
    return launch_status();
}
