// A short causal convolution over time on every channel of a projection, carried across steps, with what two kinds
// of mixer do to the result in the same kernel.
//
//   y_t[c] = sum_j w[c][j] * u_(t - taps + 1 + j)[c],   j = 0 .. taps-1,  zeros before the sequence's start.
//
// u are rows of a float32 projection [T, ld] (several convolved blocks of channels side by side).  The last taps-1
// rows of u of every request live in a float32 state slot [taps-1][C] (C = all convolved channels of the mixer; row
// taps-2 is the newest; rows that would lie before position 0 hold zeros).  One CTA serves one token, except at the
// start of a portion: the CTA of a portion's first token also serves the next taps-2 tokens (the only ones that read
// the slot) and then writes the slot's new contents, so no other CTA reads a slot while it is rewritten.  The sum runs
// over j in rising order whatever the cut of the prompt, so a token's value does not depend on the cut.
//
// attn_conv_prepare: q | k | v blocks; then an RMS norm over the whole q row and the whole k row (plain weights), each
// value head divided by its root mean square; q leaves in the compute dtype, k and v go to the token's cache slot.
// delta_conv_prepare: q | k | v blocks; silu; q and k made unit vectors per head (x / sqrt(sum x^2 + 1e-6)), q times
// dim^-1/2; besides, per value head, beta = sigmoid(b) and the decay g = exp(-exp(A_log) * softplus(a + dt_bias)).
// All of it is float32.
#include "common.cuh"
#include <math.h>

namespace aien {

constexpr int SC_MAX_TAPS = 8;
constexpr int SC_THREADS = 256;
constexpr int SC_THREADS_WIDE = 1024;       // for a step of few tokens: its CTAs are too few to hide a row's loads behind one another

inline int conv_threads(int T, int C) { return (T <= 2 * 148 && C >= 2048) ? SC_THREADS_WIDE : SC_THREADS; }

struct ConvRow {
    int t, first, last, slot;
    bool fresh;
};

// The same for a number of taps known when the kernel is compiled: the addresses are one pointer a source and a stride,
// a token with all its taps inside the step (every token but a portion's first ones) reads without a test, and four
// bfloat16 weights are one load.  What the kernel spends is instructions, not bytes: with the taps a run-time number
// it issued several hundred a channel.
template <int TAPS>
__device__ __forceinline__ float conv_fixed(const float* __restrict__ proj, long ld, int off, int cc, const void* __restrict__ w, int wdt,
                                            const float* __restrict__ st, int C, int c0, const ConvRow& r) {
    const int t_first = r.t - (TAPS - 1);
    float u[TAPS], wv[TAPS];
    if (t_first >= r.first) {
        const float* p = proj + (long)t_first * ld + off + cc;
#pragma unroll
        for (int j = 0; j < TAPS; ++j) u[j] = __ldcg(p + (long)j * ld);
    } else {
#pragma unroll
        for (int j = 0; j < TAPS; ++j) {
            const int tt = t_first + j;
            if (tt >= r.first) u[j] = __ldcg(proj + (long)tt * ld + off + cc);
            else u[j] = r.fresh ? 0.f : st[(long)((TAPS - 1) + (tt - r.first)) * C + c0 + cc];
        }
    }
    if (wdt == AIEN_DT_F32) {
        const float* wf = reinterpret_cast<const float*>(w) + (size_t)cc * TAPS;
#pragma unroll
        for (int j = 0; j < TAPS; ++j) wv[j] = wf[j];
    } else if (TAPS == 4 && (reinterpret_cast<uintptr_t>(w) & 7) == 0) {
        const uint2 raw = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(w) + (size_t)cc * 4);
        const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
        const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
        wv[0] = lo.x; wv[1] = lo.y; wv[2 % TAPS] = hi.x; wv[3 % TAPS] = hi.y;
    } else {
        const __nv_bfloat16* wh = reinterpret_cast<const __nv_bfloat16*>(w) + (size_t)cc * TAPS;
#pragma unroll
        for (int j = 0; j < TAPS; ++j) wv[j] = __bfloat162float(wh[j]);
    }
    float y = 0.f;
#pragma unroll
    for (int j = 0; j < TAPS; ++j) y = fmaf(wv[j], u[j], y);
    return y;
}

// channel cc of the convolved block that starts at column `off` of proj and at channel `c0` of the state
__device__ __forceinline__ float conv_value(const float* __restrict__ proj, long ld, int off, int cc, const void* __restrict__ w, int wdt,
                                            int taps, const float* __restrict__ st, int C, int c0, const ConvRow& r) {
    switch (taps) {
        case 2: return conv_fixed<2>(proj, ld, off, cc, w, wdt, st, C, c0, r);
        case 3: return conv_fixed<3>(proj, ld, off, cc, w, wdt, st, C, c0, r);
        case 4: return conv_fixed<4>(proj, ld, off, cc, w, wdt, st, C, c0, r);
        default: break;
    }
    float y = 0.f;
    for (int j = 0; j < taps; ++j) {
        const int tt = r.t - (taps - 1) + j;
        float u;
        if (tt >= r.first) u = ld_act(proj + (size_t)tt * ld + off + cc);
        else if (r.fresh) u = 0.f;
        else u = st[(size_t)((taps - 1) + (tt - r.first)) * C + c0 + cc];
        y = fmaf(load_dyn(w, wdt, (size_t)cc * taps + j), u, y);
    }
    return y;
}

// the slot's new rows for one block of channels, by the thread that owns the channel
__device__ __forceinline__ void conv_state_update(const float* __restrict__ proj, long ld, int off, int n, int taps,
                                                  float* __restrict__ st, int C, int c0, const ConvRow& r) {
    for (int cc = threadIdx.x; cc < n; cc += blockDim.x) {
        float keep[SC_MAX_TAPS];
        for (int k = 0; k < taps - 1; ++k) {
            const int tt = r.last - (taps - 1) + k;
            if (tt >= r.first) keep[k] = ld_act(proj + (size_t)tt * ld + off + cc);
            else keep[k] = r.fresh ? 0.f : st[(size_t)((taps - 1) + (tt - r.first)) * C + c0 + cc];
        }
        for (int k = 0; k < taps - 1; ++k) st[(size_t)k * C + c0 + cc] = keep[k];
    }
}

// which rows this CTA serves: returns the count (0: another CTA serves this token)
__device__ __forceinline__ int conv_rows(int t, int taps, const int* seq_of_token, const int* q_start, const int* positions,
                                         const int* slot_map, ConvRow& r) {
    const int s = seq_of_token[t];
    r.first = q_start[s];
    r.last = q_start[s + 1];
    r.slot = slot_map[s];
    r.fresh = positions[r.first] == 0;
    r.t = t;
    const int k = t - r.first;
    if (k > 0 && k < taps - 1) return 0;
    if (k > 0) return 1;
    const int n = r.last - r.first;
    return taps - 1 < 1 ? 1 : (n < taps - 1 ? n : taps - 1);
}

template <typename TQ, typename TKV>
__global__ void __launch_bounds__(SC_THREADS_WIDE)
attn_conv_prepare_kernel(const float* __restrict__ proj, long ld, int q_off, int k_off, int v_off, int Cq, int Ck, int Cv,
                         const void* __restrict__ wq, const void* __restrict__ wk, const void* __restrict__ wv, int wdt, int taps,
                         const void* __restrict__ qn, const void* __restrict__ kn, int ndt, float eps, int G, int V, int value_norm,
                         float* __restrict__ state, const int* __restrict__ state_slots, const int* __restrict__ seq_of_token,
                         const int* __restrict__ q_start, const int* __restrict__ positions, const int* __restrict__ kv_slots,
                         TKV* __restrict__ k_cache, TKV* __restrict__ v_cache, TQ* __restrict__ q_out, long ldq) {
    extern __shared__ float vals[];               // q | k | v of the row at hand
    __shared__ float red[32];
    ConvRow r;
    const int rows = conv_rows(blockIdx.x, taps, seq_of_token, q_start, positions, state_slots, r);
    if (rows == 0) return;
    const bool own_kv = Ck > 0;
    const int C = Cq + Ck + Cv;
    float* st = state + (size_t)r.slot * (size_t)(taps - 1) * C;
    const int t0 = r.t;
    for (int i = 0; i < rows; ++i) {
        r.t = t0 + i;
        float sq = 0.f, sk = 0.f;
        for (int c = threadIdx.x; c < C; c += blockDim.x) {
            float y;
            if (c < Cq) { y = conv_value(proj, ld, q_off, c, wq, wdt, taps, st, C, 0, r); sq = fmaf(y, y, sq); }
            else if (c < Cq + Ck) { y = conv_value(proj, ld, k_off, c - Cq, wk, wdt, taps, st, C, Cq, r); sk = fmaf(y, y, sk); }
            else y = conv_value(proj, ld, v_off, c - Cq - Ck, wv, wdt, taps, st, C, Cq + Ck, r);
            vals[c] = y;
        }
        const float rq = 1.0f / sqrtf(block_sum(sq, red) / (float)Cq + eps);
        for (int c = threadIdx.x; c < Cq; c += blockDim.x)
            q_out[(size_t)r.t * ldq + c] = from_f<TQ>(vals[c] * rq * load_dyn(qn, ndt, c));
        if (own_kv) {
            const float rk = 1.0f / sqrtf(block_sum(sk, red) / (float)Ck + eps);
            const int slot = kv_slots[r.t];
            if (slot >= 0) {
                for (int c = threadIdx.x; c < Ck; c += blockDim.x)
                    k_cache[(size_t)slot * Ck + c] = from_f<TKV>(vals[Cq + c] * rk * load_dyn(kn, ndt, c));
                const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
                for (int g = warp; g < G; g += nwarps) {
                    const float* v = vals + Cq + Ck + (size_t)g * V;
                    float rv = 1.f;
                    if (value_norm) {
                        float sv = 0.f;
                        for (int d = lane; d < V; d += 32) sv = fmaf(v[d], v[d], sv);
                        rv = 1.0f / sqrtf(warp_sum(sv) / (float)V + eps);
                    }
                    for (int d = lane; d < V; d += 32) v_cache[(size_t)slot * Cv + (size_t)g * V + d] = from_f<TKV>(v[d] * rv);
                }
            }
        }
        __syncthreads();
    }
    if (t0 == r.first && taps > 1) {
        conv_state_update(proj, ld, q_off, Cq, taps, st, C, 0, r);
        if (own_kv) {
            conv_state_update(proj, ld, k_off, Ck, taps, st, C, Cq, r);
            conv_state_update(proj, ld, v_off, Cv, taps, st, C, Cq + Ck, r);
        }
    }
}

__device__ __forceinline__ float silu_f(float z) { return z / (1.0f + expf(-z)); }

// out float32 [T, Cq+Ck+Cv] (q | k | v prepared), gb float32 [T, 2*heads] (decay g | beta)
__global__ void __launch_bounds__(SC_THREADS_WIDE)
delta_conv_prepare_kernel(const float* __restrict__ proj, long ld, int q_off, int k_off, int v_off, int b_off, int a_off,
                          int G, int D, int heads, int V,
                          const void* __restrict__ wq, const void* __restrict__ wk, const void* __restrict__ wv, int wdt, int taps,
                          const void* __restrict__ a_log, const void* __restrict__ dt_bias, int pdt,
                          float* __restrict__ state, size_t state_stride, const int* __restrict__ state_slots,
                          const int* __restrict__ seq_of_token, const int* __restrict__ q_start, const int* __restrict__ positions,
                          float* __restrict__ out, long ldo, float* __restrict__ gb, long ldgb) {
    extern __shared__ float vals[];
    ConvRow r;
    const int rows = conv_rows(blockIdx.x, taps, seq_of_token, q_start, positions, state_slots, r);
    if (rows == 0) return;
    const int Cq = G * D, Ck = G * D, Cv = heads * V, C = Cq + Ck + Cv;
    float* st = state + (size_t)r.slot * state_stride;
    const int t0 = r.t;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const float qmul = 1.0f / sqrtf((float)D);
    for (int i = 0; i < rows; ++i) {
        r.t = t0 + i;
        for (int c = threadIdx.x; c < C; c += blockDim.x) {
            float y;
            if (c < Cq) y = conv_value(proj, ld, q_off, c, wq, wdt, taps, st, C, 0, r);
            else if (c < Cq + Ck) y = conv_value(proj, ld, k_off, c - Cq, wk, wdt, taps, st, C, Cq, r);
            else y = conv_value(proj, ld, v_off, c - Cq - Ck, wv, wdt, taps, st, C, Cq + Ck, r);
            y = silu_f(y);
            if (c >= Cq + Ck) out[(size_t)r.t * ldo + c] = y;
            else vals[c] = y;
        }
        for (int h = threadIdx.x; h < heads; h += blockDim.x) {
            const float a = ld_act(proj + (size_t)r.t * ld + a_off + h) + load_dyn(dt_bias, pdt, h);
            const float sp = a > 20.f ? a : log1pf(expf(a));
            gb[(size_t)r.t * ldgb + h] = expf(-expf(load_dyn(a_log, pdt, h)) * sp);
            gb[(size_t)r.t * ldgb + heads + h] = 1.0f / (1.0f + expf(-ld_act(proj + (size_t)r.t * ld + b_off + h)));
        }
        __syncthreads();
        for (int g = warp; g < 2 * G; g += nwarps) {            // q heads then k heads, each a unit vector
            const float* v = vals + (size_t)g * D;
            float ss = 0.f;
            for (int d = lane; d < D; d += 32) ss = fmaf(v[d], v[d], ss);
            const float m = (g < G ? qmul : 1.0f) / sqrtf(warp_sum(ss) + 1e-6f);
            for (int d = lane; d < D; d += 32) out[(size_t)r.t * ldo + (size_t)g * D + d] = v[d] * m;
        }
        __syncthreads();
    }
    if (t0 == r.first && taps > 1) {
        conv_state_update(proj, ld, q_off, Cq, taps, st, C, 0, r);
        conv_state_update(proj, ld, k_off, Ck, taps, st, C, Cq, r);
        conv_state_update(proj, ld, v_off, Cv, taps, st, C, Cq + Ck, r);
    }
}

// One block of C convolved channels with a bias and an activation of its own:
// out[t][c] = f(conv(c) + bias[c]), f the identity (act 0) or silu (act 1); float32 out, and on request the same rows
// once more in bfloat16 (the operand of a product that follows).
__global__ void __launch_bounds__(SC_THREADS_WIDE)
conv_act_kernel(const float* __restrict__ proj, long ld, int off, int C, const void* __restrict__ w, int wdt,
                const void* __restrict__ bias, int bdt, int taps, int act, float* __restrict__ state, size_t state_stride,
                const int* __restrict__ state_slots, const int* __restrict__ seq_of_token, const int* __restrict__ q_start,
                const int* __restrict__ positions, float* __restrict__ out, long ldo, __nv_bfloat16* __restrict__ out16, long ldo16) {
    ConvRow r;
    const int rows = conv_rows(blockIdx.x, taps, seq_of_token, q_start, positions, state_slots, r);
    if (rows == 0) return;
    float* st = state + (size_t)r.slot * state_stride;
    const int t0 = r.t;
    for (int i = 0; i < rows; ++i) {
        r.t = t0 + i;
        for (int c = threadIdx.x; c < C; c += blockDim.x) {
            float y = conv_value(proj, ld, off, c, w, wdt, taps, st, C, 0, r);
            if (bias != nullptr) y += load_dyn(bias, bdt, c);
            y = act == 1 ? silu_f(y) : y;
            out[(size_t)r.t * ldo + c] = y;
            if (out16 != nullptr) out16[(size_t)r.t * ldo16 + c] = __float2bfloat16_rn(y);
        }
    }
    __syncthreads();
    if (t0 == r.first && taps > 1) conv_state_update(proj, ld, off, C, taps, st, C, 0, r);
}

// ---- channels four at a time, tokens in runs
// conv_act and delta_conv_prepare for 2 to 4 taps and rows that 16-byte loads take.  The kernels above spend a thread and
// taps loads on every (token, channel) and leave the whole beginning of a portion to one CTA; what these rows cost at
// least is being read and written once.  So a thread owns four neighbouring channels over a run of tokens: a row is loaded
// once, the taps - 1 rows before it wait in registers, the weights are read once per run.
//
// Token t belongs to run t / run, except that the run holding a portion's first token also serves the portion's next
// taps - 2 tokens: only these read the request's slot, which the same thread rewrites afterwards.
// The sums run over the taps in rising order, as above, so the two forms agree to the bit.
// 2,048 tokens, B200: conv_act of 4,096 channels with both outputs (84 MB): 62 us before, 24 so; delta_conv_prepare of 4,096 channels
// (67 MB): 63 us before, 27 so.
constexpr int CR_THREADS = 128;

struct ConvBlock {                              // up to three blocks of convolved channels side by side
    int off, c0, n;                             // first column of proj, first channel, channels
    const void* w;
};

struct ConvRunArgs {
    const float* proj; long ld; ConvBlock blk[3]; int C, wdt; const void* bias; int bdt, act; float* state; size_t state_stride;
    const int* slots; const int* seq_of_token; const int* q_start; const int* positions; float* out; long ldo; __nv_bfloat16* out16; long ldo16;
    int T, run;
    // delta_conv_prepare: heads of D channels in the first two blocks become unit vectors, and the gates
    int D, heads, a_off, b_off; const void* a_log; const void* dt_bias; int pdt; float* gb; long ldgb;
};

__device__ __forceinline__ float4 f4(float a) { return make_float4(a, a, a, a); }

template <int TAPS, bool DELTA>
__global__ void __launch_bounds__(CR_THREADS)
conv_runs_kernel(const ConvRunArgs a) {
    griddep_launch();
    const int lo = blockIdx.y * a.run, hi = lo + a.run < a.T ? lo + a.run : a.T;
    if (DELTA && blockIdx.x == gridDim.x - 1) {                             // one CTA per run makes the gates
        for (int i = threadIdx.x; i < (hi - lo) * a.heads; i += CR_THREADS) {
            const int t = lo + i / a.heads, h = i % a.heads;
            const float z = ld_act(a.proj + (size_t)t * a.ld + a.a_off + h) + load_dyn(a.dt_bias, a.pdt, h);
            const float sp = z > 20.f ? z : log1pf(expf(z));
            a.gb[(size_t)t * a.ldgb + h] = expf(-expf(load_dyn(a.a_log, a.pdt, h)) * sp);
            a.gb[(size_t)t * a.ldgb + a.heads + h] = 1.0f / (1.0f + expf(-ld_act(a.proj + (size_t)t * a.ld + a.b_off + h)));
        }
        return;
    }
    const int c = (blockIdx.x * CR_THREADS + threadIdx.x) * 4;
    const bool live = c < a.C;
    if (!DELTA && !live) return;                                            // with unit vectors the lanes of a warp stay together
    const int bi = !DELTA || c < a.blk[1].c0 ? 0 : c < a.blk[2].c0 ? 1 : 2;
    const int off = bi == 0 ? a.blk[0].off : bi == 1 ? a.blk[1].off : a.blk[2].off;
    const int c0 = bi == 0 ? 0 : bi == 1 ? a.blk[1].c0 : a.blk[2].c0;
    const void* w = bi == 0 ? a.blk[0].w : bi == 1 ? a.blk[1].w : a.blk[2].w;
    const int cc = live ? c - c0 : 0;
    const float* src = a.proj + off + cc;
    float wv[TAPS][4], bias[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        bias[k] = a.bias != nullptr ? load_dyn(a.bias, a.bdt, cc + k) : 0.f;
#pragma unroll
        for (int j = 0; j < TAPS; ++j) wv[j][k] = load_dyn(w, a.wdt, (size_t)(cc + k) * TAPS + j);
    }
    const float qmul = DELTA ? 1.0f / sqrtf((float)a.D) : 1.f;
    float4 u[TAPS - 1];                                                     // the rows before the token at hand, the oldest first
    int first = -1, last = 0;
    float* st = nullptr;
    bool fresh = false, owns = false;                                       // owns: this run holds the portion's first token
    // row tt of the request at hand, from before its portion too
    auto row = [&](int tt) {
        if (tt >= first) return __ldcg(reinterpret_cast<const float4*>(src + (size_t)tt * a.ld));
        if (fresh) return f4(0.f);
        return *reinterpret_cast<const float4*>(st + (size_t)(TAPS - 1 + tt - first) * a.C + c);
    };
    // the slot's new rows: those of the portion's last tokens, where the portion is short the slot's own moved up
    auto leave = [&]() {
        if (!owns || !live) return;
        float4 keep[TAPS - 1];
#pragma unroll
        for (int k = 0; k < TAPS - 1; ++k) keep[k] = row(last - (TAPS - 1) + k);
#pragma unroll
        for (int k = 0; k < TAPS - 1; ++k) *reinterpret_cast<float4*>(st + (size_t)k * a.C + c) = keep[k];
    };
    for (int t = lo; t < a.T; ++t) {
        if (t >= hi && !(owns && t < last && t - first < TAPS - 1)) break;  // past the run: only the rest of a beginning that started in it
        if (first < 0 || t >= last) {                                       // another request
            leave();
            const int s = a.seq_of_token[t];
            first = a.q_start[s];
            last = a.q_start[s + 1];
            fresh = a.positions[first] == 0;
            st = a.state + (size_t)a.slots[s] * a.state_stride;
            owns = first >= lo;
            if (!owns && t - first < TAPS - 1) {                            // the beginning belongs to the run before
                t = first + TAPS - 1;
                if (t >= last) {                                            // a short portion, served whole there
                    t = last - 1;
                    first = -1;
                    owns = false;
                    continue;
                }
                if (t >= hi) break;
            }
#pragma unroll
            for (int j = 0; j < TAPS - 1; ++j) u[j] = live ? row(t - (TAPS - 1) + j) : f4(0.f);
        }
        const float4 x = live ? __ldcg(reinterpret_cast<const float4*>(src + (size_t)t * a.ld)) : f4(0.f);
        float y[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int j = 0; j < TAPS; ++j) {
            const float4 r = j < TAPS - 1 ? u[j % (TAPS - 1)] : x;
            y[0] = fmaf(wv[j][0], r.x, y[0]);
            y[1] = fmaf(wv[j][1], r.y, y[1]);
            y[2] = fmaf(wv[j][2], r.z, y[2]);
            y[3] = fmaf(wv[j][3], r.w, y[3]);
        }
#pragma unroll
        for (int j = 0; j + 1 < TAPS - 1; ++j) u[j] = u[j + 1];
        u[TAPS - 2] = x;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (a.bias != nullptr) y[k] += bias[k];
            if (DELTA || a.act == 1) y[k] = silu_f(y[k]);
        }
        if (DELTA) {                                                        // the lanes of one head meet: D / 4 of them, a power of two
            float ss = fmaf(y[0], y[0], y[1] * y[1]) + fmaf(y[2], y[2], y[3] * y[3]);
            for (int o = a.D / 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            if (bi < 2) {
                const float m = (bi == 0 ? qmul : 1.0f) / sqrtf(ss + 1e-6f);
#pragma unroll
                for (int k = 0; k < 4; ++k) y[k] *= m;
            }
        }
        if (live) {
            *reinterpret_cast<float4*>(a.out + (size_t)t * a.ldo + c) = make_float4(y[0], y[1], y[2], y[3]);
            if (!DELTA && a.out16 != nullptr) {
                const __nv_bfloat162 p0 = __floats2bfloat162_rn(y[0], y[1]), p1 = __floats2bfloat162_rn(y[2], y[3]);
                *reinterpret_cast<uint2*>(a.out16 + (size_t)t * a.ldo16 + c) =
                    make_uint2(*reinterpret_cast<const uint32_t*>(&p0), *reinterpret_cast<const uint32_t*>(&p1));
            }
        }
    }
    leave();
}

// Whether rows and state take 16-byte accesses at every fourth channel.
static bool conv_runs_take(const ConvRunArgs& a, int taps) {
    if (taps < 2 || taps > 4 || a.C % 4 || a.ld % 4 || a.ldo % 4 || a.state_stride % 4) return false;
    if ((reinterpret_cast<uintptr_t>(a.proj) | reinterpret_cast<uintptr_t>(a.out) | reinterpret_cast<uintptr_t>(a.state)) & 15) return false;
    if (a.out16 != nullptr && ((reinterpret_cast<uintptr_t>(a.out16) & 7) || a.ldo16 % 4)) return false;
    for (const ConvBlock& b : a.blk) if (b.off % 4 || b.n % 4) return false;
    return true;
}

template <bool DELTA>
static void launch_conv_runs(ConvRunArgs& a, int taps, cudaStream_t stream) {
    const int gx = (a.C / 4 + CR_THREADS - 1) / CR_THREADS + (DELTA ? 1 : 0);
    // longer runs read the rows before them less often; four CTAs an SM are wanted first
    a.run = 1;
    while (a.run < 16 && (long)gx * ((a.T + 2 * a.run - 1) / (2 * a.run)) >= 4 * 148) a.run *= 2;
    const dim3 grid(gx, (a.T + a.run - 1) / a.run);
    const auto kern = taps == 2 ? conv_runs_kernel<2, DELTA> : taps == 3 ? conv_runs_kernel<3, DELTA> : conv_runs_kernel<4, DELTA>;
    kern<<<grid, CR_THREADS, 0, stream>>>(a);                               // plain: see griddep_wait
}

}  // namespace aien

using namespace aien;

template <typename TQ, typename TKV>
static int launch_attn_conv_prepare(size_t smem, cudaStream_t stream, int T, const float* proj, long ld, int q_off, int k_off, int v_off,
                                    int Cq, int Ck, int Cv, const void* wq, const void* wk, const void* wv, int wdt, int taps,
                                    const void* qn, const void* kn, int ndt, float eps, int G, int V, int value_norm, float* state,
                                    const int* state_slots, const int* seq_of_token, const int* q_start, const int* positions,
                                    const int* kv_slots, TKV* k_cache, TKV* v_cache, TQ* q_out, long ldq) {
    auto kern = attn_conv_prepare_kernel<TQ, TKV>;
    if (smem > 48 * 1024 && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return AIEN_E_STATE;
    kern<<<T, conv_threads(T, Cq + Ck + Cv), smem, stream>>>(proj, ld, q_off, k_off, v_off, Cq, Ck, Cv, wq, wk, wv, wdt, taps, qn, kn, ndt, eps, G, V,
                                          value_norm, state, state_slots, seq_of_token, q_start, positions, kv_slots, k_cache, v_cache,
                                          q_out, ldq);
    return 0;
}

// proj float32 [T, ld] with the q block at q_off (Cq channels) and, when the run keeps its own keys and values
// (Ck > 0), k at k_off (Ck = G * head size) and v at v_off (Cv = G * V).  Convolution weights [C, taps] in w_dt, norm
// weights in n_dt.  state float32 [slots][taps-1][Cq+Ck+Cv]; kv_slots[t]: cache slot of token t (-1: write nothing).
AIEN_API int aien_attn_conv_prepare(const float* proj, long ld, int q_off, int k_off, int v_off, int Cq, int Ck, int Cv,
                                    const void* wq, const void* wk, const void* wv, int w_dt, int taps,
                                    const void* qn, const void* kn, int n_dt, float eps, int G, int V, int value_norm,
                                    float* state, const int* state_slots, const int* seq_of_token, const int* q_start,
                                    const int* positions, const int* kv_slots, void* k_cache, void* v_cache, int kv_dt,
                                    void* q_out, int q_dt, long ldq, int T, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (taps < 1 || taps > SC_MAX_TAPS || Cq <= 0 || Ck < 0 || Cv < 0 || (Ck > 0 && (G <= 0 || Cv != G * V))) return AIEN_E_SHAPE;
    if (taps > 1 && state == nullptr) return AIEN_E_SHAPE;
    const size_t smem = (size_t)(Cq + Ck + Cv) * sizeof(float);
    if (smem > 200 * 1024) return AIEN_E_SHAPE;
    int rc = 0;
    AIEN_DISPATCH_DTYPE(q_dt, TQ, AIEN_DISPATCH_DTYPE(kv_dt, TKV,
        (rc = launch_attn_conv_prepare<TQ, TKV>(smem, stream, T, proj, ld, q_off, k_off, v_off, Cq, Ck, Cv, wq, wk, wv, w_dt, taps, qn, kn,
                                                n_dt, eps, G, V, value_norm, state, state_slots, seq_of_token, q_start, positions,
                                                kv_slots, (TKV*)k_cache, (TKV*)v_cache, (TQ*)q_out, ldq))));
    if (rc != 0) return rc;
    return launch_status();
}

// proj float32 [T, ld]: q (G*D) at q_off, k (G*D) at k_off, v (heads*V) at v_off, beta's input (heads) at b_off, the
// decay's input (heads) at a_off.  state float32 rows of state_stride numbers whose first (taps-1)*(2*G*D + heads*V)
// are the convolution's.  out float32 [T, ldo] = q | k | v prepared; gb float32 [T, ldgb] = decay | beta.
AIEN_API int aien_delta_conv_prepare(const float* proj, long ld, int q_off, int k_off, int v_off, int b_off, int a_off,
                                     int G, int D, int heads, int V, const void* wq, const void* wk, const void* wv, int w_dt, int taps,
                                     const void* a_log, const void* dt_bias, int p_dt, float* state, size_t state_stride,
                                     const int* state_slots, const int* seq_of_token, const int* q_start, const int* positions,
                                     float* out, long ldo, float* gb, long ldgb, int T, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (taps < 1 || taps > SC_MAX_TAPS || G <= 0 || D <= 0 || heads <= 0 || V <= 0 || heads % G) return AIEN_E_SHAPE;
    const size_t smem = (size_t)(2 * G * D) * sizeof(float);
    if (smem > 200 * 1024) return AIEN_E_SHAPE;
    ConvRunArgs a{proj, ld, {{q_off, 0, G * D, wq}, {k_off, G * D, G * D, wk}, {v_off, 2 * G * D, heads * V, wv}}, 2 * G * D + heads * V, w_dt, nullptr, 0, 1,
                  state, state_stride, state_slots, seq_of_token, q_start, positions, out, ldo, nullptr, 0, T, 1,
                  D, heads, a_off, b_off, a_log, dt_bias, p_dt, gb, ldgb};
    // the lanes of a head meet by shuffles: D / 4 of them, a power of two, a head inside one warp
    if (D >= 8 && D <= 128 && (D & (D - 1)) == 0 && T <= 65535 && conv_runs_take(a, taps)) {
        launch_conv_runs<true>(a, taps, stream);
        return launch_status();
    }
    auto kern = delta_conv_prepare_kernel;
    if (smem > 48 * 1024 && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return AIEN_E_STATE;
    kern<<<T, conv_threads(T, 2 * G * D + heads * V), smem, stream>>>(proj, ld, q_off, k_off, v_off, b_off, a_off, G, D, heads, V, wq, wk, wv, w_dt, taps, a_log, dt_bias,
                                          p_dt, state, state_stride, state_slots, seq_of_token, q_start, positions, out, ldo, gb, ldgb);
    return launch_status();
}

// proj float32 [T, ld] with the C convolved channels from column `off` on; weights [C, taps] in w_dt, bias [C] in b_dt (or
// null); state float32 rows of state_stride numbers whose first (taps-1)*C are the convolution's; out float32 [T, ldo];
// out16 (or null) bfloat16 [T, ldo16]: the same rows rounded.
AIEN_API int aien_conv_act(const float* proj, long ld, int off, int C, const void* w, int w_dt, const void* bias, int b_dt, int taps,
                           int act, float* state, size_t state_stride, const int* state_slots, const int* seq_of_token,
                           const int* q_start, const int* positions, float* out, long ldo, void* out16, long ldo16, int T,
                           cudaStream_t stream) {
    if (T <= 0) return 0;
    if (taps < 1 || taps > SC_MAX_TAPS || C <= 0 || (act != 0 && act != 1)) return AIEN_E_SHAPE;
    if (taps > 1 && state == nullptr) return AIEN_E_SHAPE;
    ConvRunArgs a{proj, ld, {{off, 0, C, w}, {0, C, 0, nullptr}, {0, C, 0, nullptr}}, C, w_dt, bias, b_dt, act, state, state_stride, state_slots,
                  seq_of_token, q_start, positions, out, ldo, (__nv_bfloat16*)out16, ldo16, T, 1, 0, 0, 0, 0, nullptr, nullptr, 0, nullptr, 0};
    if (T <= 65535 && conv_runs_take(a, taps)) {
        launch_conv_runs<false>(a, taps, stream);
        return launch_status();
    }
    conv_act_kernel<<<T, conv_threads(T, C), 0, stream>>>(proj, ld, off, C, w, w_dt, bias, b_dt, taps, act, state, state_stride, state_slots,
                                                          seq_of_token, q_start, positions, out, ldo, (__nv_bfloat16*)out16, ldo16);
    return launch_status();
}
