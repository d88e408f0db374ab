// Portions of prompts through recurrences with a state matrix and one decay per head and token, sixteen tokens at a time.
//
//   S <- g S + k u^T ,  o = S^T q        u = v (linear attention; state-space duality with k = B, q = C, v = dt x), or
//                                        u = beta (v - (g S)^T k) (the delta rule)
//
// Written out over a block of 16 tokens that finds the state S0, with G_i the product of the decays up to token i and
// G_i/G_j the product of those behind j up to i:
//   p_i = S0^T k_i ,  r_i = S0^T q_i
//   u_i = beta_i (v_i - G_i p_i - sum_{j<i} G_i/G_j (k_i.k_j) u_j)   that is   u = M (v - G p)
//   o_i = G_i r_i + sum_{j<=i} G_i/G_j (q_i.k_j) u_j                 that is   o = G r + A u
//   S   = G_16 S0 + sum_j G_16/G_j k_j u_j^T
// A, M (16 x 16, lower triangular), G and G_16/G_j depend on the rows alone.  A first kernel makes them for every block
// and head side by side (M by forward substitution in float32); a second one walks a request's blocks in order with a CTA
// for 16 columns of a head's state.  There S0^T [q | k] and the update are matrix products over the 16 columns, and what
// a token waits for is one sixteenth of a block's chain instead of a chain of its own.
//
// The products run on the tensor cores (mma.sync tf32) with every float32 operand cut in two: x = hi + lo, hi the nearest
// number of 11 bits, lo the rest, and x y = hi hi + hi lo + lo hi; what is dropped is 2^-22 of a product and has no sign
// of its own.  The two small products have accumulators of their own: the tensor cores cut off what does not fit 24 bits
// where a multiply-add rounds, which adds up where everything is of one sign (see bw_total).  tcgen05 would have to find the state in
// shared memory for every block's product; here the eight warps share its rows and each keeps its own as accumulators:
// [16 columns] x [8 rows] fragments whose register order is the order of the left operand once the rows of a fragment are
// counted 0 2 4 6 1 3 5 7 on both sides.  The update is accumulated from zero and added to the decayed state by float32
// multiply-adds, so the state is rounded once per block.  The decays' products are sums of two numbers until they are
// written, and G_16 stays one: rounded, it would be off by the same factor in every block where the decay is constant.
//
// Relative error (2-norm) of the results and the last states against 64 bits, 2,048 tokens, and in brackets that of the
// float32 kernels that go token by token or, for one decay per head, by chunks of 64:
//   one decay per head, 1 - 2^-5 .. 1 - 2^-8          0.8e-7 and 0.8e-7  (1.7e-7 and 1.3e-7)
//   one decay per head, 1 - 1e-4                      0.9e-7 and 1.7e-7  (2.7e-7 and 3.2e-7)
//   duality, rows of silu, drawn step sizes           0.9e-7 and 1.0e-7  (0.9e-7 and 3.0e-7)
//   delta rule, rows of silu, drawn decays            1.4e-7 and 1.4e-7  (2.1e-7 and 3.1e-7)
//   delta rule, rows of either sign, decays 0.74 .. 1 1.3e-7 and 1.1e-7  (1.1e-7 and 0.8e-7)
// With one accumulator, nothing added back and rounded products of decays the first two were 6.8e-7 and 2.3e-6.
//
// Walk and coefficients back to back, B200: 2,048 tokens, 16 heads of 128 x 128, one request, the delta rule 170 us, 16 of them the
// coefficients (603 token by token); linear attention 159 and 31.  2,000 tokens of three requests, 32 heads of 128 x 64, state-space duality:
// 112 and 7 us (540 token by token; 22 more with the longest request's CTAs the last to start); linear attention, 1,900 tokens of two requests, 16
// heads of 128 x 128: 127 and 30 us (237 by chunks).  What bounds the walk is a block's chain of dependent instructions (405 a warp; issue
// slots 55 to 58 % used with two CTAs on an SM, profiles/layer_kernels__ncu_counters.md), not its barriers or its rows: fetched two
// blocks ahead instead of one, with one barrier a block instead of two, and with products of different sums between dependent
// ones it gains 4 us in 128.  (The choices of a form below were measured at 148, 110 and 86 us, with one accumulator a sum.)
#include "common.cuh"
#include <math.h>

namespace aien {

constexpr int BW_B = 16;                       // tokens of a block
constexpr int BW_WARPS = 8;
constexpr int BW_THREADS = 32 * BW_WARPS;
constexpr int BW_LD = 20;                      // floats between rows of A and M: no bank twice in a quarter warp
constexpr int BW_TAIL = 2 * BW_B + 4;                     // G | G_16 / G_j | what G_16 lacks, padded
constexpr int BW_COEF = 2 * BW_B * BW_B + BW_TAIL;       // A | M and the tail per block and head

__device__ __forceinline__ void bw_split(float x, uint32_t& hi, uint32_t& lo) {
    hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
    lo = __float_as_uint(x - __uint_as_float(hi));
}

__device__ __forceinline__ void bw_mma(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// a product of decays as the sum of two numbers
struct BwDecay {
    float h = 1.f, l = 0.f;
    __device__ __forceinline__ void by(float g) {
        const float p = h * g;
        l = fmaf(l, g, fmaf(h, g, -p));
        h = p;
    }
    __device__ __forceinline__ float times(float x) const { return fmaf(h, x, l * x); }
};

__device__ __forceinline__ void bw_cp16(float* dst, const float* src, bool in) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(in ? 16 : 0) : "memory");
}

__device__ __forceinline__ void bw_cp16(float* dst, const float* src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

struct BlockWalk {
    const float* rows; long ld; int q_off, k_off, v_off;        // q, k: G heads of N numbers; v: `heads` heads of V
    const float* gates; long ldg; int g_off, w_off;             // decay of head h in column g_off + h; its weight (beta, or the step size) in w_off + h (w_off < 0: 1)
    const float* decay;                                         // or one decay per head for all tokens
    float* act_rows; long ld_act;                               // with `act`: silu of q | k | v goes here first and is read from here
    int act, delta;
    float* coef;
    const void* skip_any; int skip_dt;       // o += skip[h] * v (null: no such term)
    float* state; size_t state_stride, s_off; int state_vn;     // state_vn: a head's state is [V][N], else [N][V]
    const int* slots; const int* q_start; const int* positions;
    float* out; long ldo;
    int T, S, heads, G, N, V;
    int alone;                               // requests of one token that are served elsewhere: left out here
};

// the request whose blocks include block slot b; request s's blocks start at q_start[s] / 16 + s
__device__ __forceinline__ int bw_first_block(const int* q_start, int s) { return q_start[s] / BW_B + s; }

__device__ __forceinline__ float bw_silu(float z) { return z / (1.0f + expf(-z)); }

// G_i from the product of the decays behind the block's first token, and for the last what its rounding lacks
__device__ __forceinline__ void bw_write_decay(float* c, int i, BwDecay d, float g0) {
    d.by(g0);
    const float g = d.h + d.l;
    c[512 + i] = g;
    if (i == BW_B - 1) c[512 + 2 * BW_B] = d.l - (g - d.h);
}

// One CTA per (block, q/k head): its dot products once, then A, M and the decays of every head that shares the q/k head.
// Its life is one chain (loads, silu, dot products, coefficients), so other CTAs have to fill it: without the delta rule,
// whose solve takes 64 registers, six to an SM and, with few heads a q/k head, all threads on the coefficients: linear
// attention with the silu of all rows, 1,900 tokens, 16 heads of 128 x 128: 35 us with four and half a warp, 28.5 so.
template <bool DELTA>
__global__ void __launch_bounds__(256, DELTA ? 4 : 6)
block_coef_kernel(const BlockWalk a) {
    extern __shared__ __align__(16) float bw_smem[];
    __shared__ float dots[DELTA ? 2 : 1][BW_B * BW_B];                      // q_i . k_j and k_i . k_j
    const int slot = blockIdx.x, kvh = blockIdx.y;
    griddep_launch();
    int lo = 0, hi = a.S - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (bw_first_block(a.q_start, mid) <= slot) lo = mid; else hi = mid - 1;
    }
    const int s = lo, t0 = a.q_start[s] + (slot - bw_first_block(a.q_start, s)) * BW_B, end = a.q_start[s + 1];
    const int n = end - t0 < BW_B ? end - t0 : BW_B;
    if (n <= 0 || (a.alone && end - a.q_start[s] == 1)) return;
    const int per = a.heads / a.G, N = a.N, LDN = N + 4;
    float* sq = bw_smem;                                        // [16][N + 4]
    float* sk = sq + BW_B * LDN;
    float* sg = sk + BW_B * LDN;                                // [16][per] decays, then [16][per] weights
    float* sw = sg + BW_B * per;
    float* sl = sw + BW_B * per;                                // [per][16][16] the strictly lower part of I + L (the delta rule)
    const int tid = threadIdx.x;
    for (int i = tid; i < BW_B * (N / 4); i += 256) {
        const int t = i / (N / 4), c = (i - t * (N / 4)) * 4;
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f), k = q;
        if (t < n) {
            const float* r = a.rows + (size_t)(t0 + t) * a.ld + (size_t)kvh * N + c;
            q = __ldcg(reinterpret_cast<const float4*>(r + a.q_off));
            k = __ldcg(reinterpret_cast<const float4*>(r + a.k_off));
            if (a.act) {
                q = make_float4(bw_silu(q.x), bw_silu(q.y), bw_silu(q.z), bw_silu(q.w));
                k = make_float4(bw_silu(k.x), bw_silu(k.y), bw_silu(k.z), bw_silu(k.w));
                float* w = a.act_rows + (size_t)(t0 + t) * a.ld_act + (size_t)kvh * N + c;
                *reinterpret_cast<float4*>(w) = q;
                *reinterpret_cast<float4*>(w + a.G * N) = k;
            }
        }
        *reinterpret_cast<float4*>(sq + t * LDN + c) = q;
        *reinterpret_cast<float4*>(sk + t * LDN + c) = k;
    }
    if (a.act) {
        const int cols = per * a.V / 4;
        for (int i = tid; i < n * cols; i += 256) {
            const int t = i / cols, c = kvh * per * a.V + (i - t * cols) * 4;
            const float4 v = __ldcg(reinterpret_cast<const float4*>(a.rows + (size_t)(t0 + t) * a.ld + a.v_off + c));
            *reinterpret_cast<float4*>(a.act_rows + (size_t)(t0 + t) * a.ld_act + 2 * a.G * N + c) =
                make_float4(bw_silu(v.x), bw_silu(v.y), bw_silu(v.z), bw_silu(v.w));
        }
    }
    for (int i = tid; i < BW_B * per; i += 256) {
        const int t = i / per, h = kvh * per + i - t * per;
        float g = 1.f, w = 0.f;
        if (t < n) {
            g = a.gates != nullptr ? ld_act(a.gates + (size_t)(t0 + t) * a.ldg + a.g_off + h) : a.decay[h];
            w = a.w_off >= 0 ? ld_act(a.gates + (size_t)(t0 + t) * a.ldg + a.w_off + h) : 1.f;
        }
        sg[i] = g;
        sw[i] = w;
    }
    __syncthreads();
    {
        const int i = tid >> 4, j = tid & 15;
        const float4* q4 = reinterpret_cast<const float4*>(sq + i * LDN);
        const float4* ki4 = reinterpret_cast<const float4*>(sk + i * LDN);
        const float4* kj4 = reinterpret_cast<const float4*>(sk + j * LDN);
        float x0 = 0.f, x1 = 0.f, x2 = 0.f, x3 = 0.f, y0 = 0.f, y1 = 0.f, y2 = 0.f, y3 = 0.f;
#pragma unroll 4
        for (int c = 0; c < N / 4; ++c) {
            const float4 q = q4[c], b = kj4[c];
            x0 = fmaf(q.x, b.x, x0); x1 = fmaf(q.y, b.y, x1); x2 = fmaf(q.z, b.z, x2); x3 = fmaf(q.w, b.w, x3);
            if (DELTA) {
                const float4 k = ki4[c];
                y0 = fmaf(k.x, b.x, y0); y1 = fmaf(k.y, b.y, y1); y2 = fmaf(k.z, b.z, y2); y3 = fmaf(k.w, b.w, y3);
            }
        }
        dots[0][tid] = (x0 + x1) + (x2 + x3);
        if (DELTA) dots[DELTA ? 1 : 0][tid] = (y0 + y1) + (y2 + y3);
    }
    __syncthreads();
    if (per * BW_B * 4 <= 256) {                                // few heads: a thread owns numbers (i, j), and its product of decays
        for (int u = tid; u < per * BW_B * BW_B; u += 256) {
            const int hh = u >> 8, i = (u >> 4) & 15, j = u & 15;
            float* c = a.coef + ((size_t)slot * a.heads + kvh * per + hh) * BW_COEF;
            const float wj = DELTA ? 1.f : sw[j * per + hh];
            BwDecay ratio;
            for (int r = j + 1; r <= i; ++r) ratio.by(sg[r * per + hh]);
            c[i * 16 + j] = i >= j ? ratio.times(dots[0][i * 16 + j]) * wj : 0.f;
            if (DELTA) sl[u] = i > j ? ratio.times(dots[DELTA ? 1 : 0][i * 16 + j]) * sw[i * per + hh] : 0.f;
            if (i == BW_B - 1) c[512 + 16 + j] = ratio.times(wj);
            if (j == 0) bw_write_decay(c, i, ratio, sg[hh]);
        }
    } else {                                                    // a thread owns column j of one head's matrices: the product of the decays grows by one factor a row
        for (int u = tid; u < per * BW_B; u += 256) {
            const int hh = u >> 4, j = u & 15;
            float* c = a.coef + ((size_t)slot * a.heads + kvh * per + hh) * BW_COEF;
            const float wj = DELTA ? 1.f : sw[j * per + hh];
            BwDecay ratio;
#pragma unroll
            for (int i = 0; i < BW_B; ++i) {
                if (i > j) ratio.by(sg[i * per + hh]);
                c[i * 16 + j] = i >= j ? ratio.times(dots[0][i * 16 + j]) * wj : 0.f;
                if (DELTA) sl[hh * 256 + i * 16 + j] = i > j ? ratio.times(dots[DELTA ? 1 : 0][i * 16 + j]) * sw[i * per + hh] : 0.f;
                if (j == 0) bw_write_decay(c, i, ratio, sg[hh]);
            }
            c[512 + 16 + j] = ratio.times(wj);
        }
    }
    if (!DELTA) return;
    __syncthreads();
    // (I + L)^-1 column by column: a thread owns one column of one head
    for (int u = tid; u < per * BW_B; u += 256) {
        const int hh = u >> 4, col = u & 15;
        const float* L = sl + hh * 256;
        const float beta = sw[col * per + hh];
        float x[BW_B];
#pragma unroll
        for (int r = 0; r < BW_B; ++r) {
            float v = r == col ? 1.f : 0.f;
#pragma unroll
            for (int m = 0; m < r; ++m) v = fmaf(-L[r * 16 + m], x[m], v);
            x[r] = v;
        }
        float* c = a.coef + ((size_t)slot * a.heads + kvh * per + hh) * BW_COEF + 256;
#pragma unroll
        for (int r = 0; r < BW_B; ++r) c[r * 16 + col] = x[r] * beta;
    }
}

// NT: fragments of 8 rows that a warp owns; N <= 64 NT.  MT: a CTA has 16 MT columns of the state.
// HELP: with helper warps (see block_walk_kernel).
template <int NT, int MT, bool DELTA, bool HELP>
struct BwSmem {
    static constexpr int STAGES = DELTA ? 3 : 4, TURNS = HELP || !DELTA ? 2 : 1;  // TURNS: sums of r (and u) for so many blocks
    static constexpr int LDN = 64 * NT + 8;                     // floats between rows of q and k: a half warp's 8-byte reads meet no bank twice
    static constexpr int LDV = 16 * MT + 8, LDP = 16 * MT + 4;  // floats between rows of v and u, and of the partial sums
    static constexpr int QK = BW_B * LDN;
    static constexpr int M_AT = 2 * QK + BW_B * LDV + BW_B * BW_LD, G_AT = M_AT + (DELTA ? BW_B * BW_LD : 0);
    static constexpr int STAGE = G_AT + BW_TAIL;                // q | k | v | A | M (the delta rule) | G | G_16 / G_j, what G_16 lacks
    static constexpr int PART = BW_WARPS * BW_B * LDP;
    static constexpr int U = DELTA ? BW_B * LDV : 0;
    static constexpr int TOTAL = STAGES * STAGE + (DELTA ? PART : 0) + TURNS * (PART + U);            // partial sums of p, and of r, and u
};

template <int NT, int MT, bool DELTA, bool HELP>
__device__ __forceinline__ void bw_fetch(float* __restrict__ buf, const BlockWalk& a, const float* rows, long ld, int q_col, int k_col, int v_col,
                                         int cols, const float* coef, int t, int t1, int tid) {
    using C = BwSmem<NT, MT, DELTA, HELP>;
    constexpr int pieces = 16 * NT;                             // 16-byte pieces of a padded row
#pragma unroll
    for (int i = tid; i < BW_B * pieces; i += BW_THREADS) {
        const int tok = i / pieces, c = i % pieces * 4;
        const bool in = t + tok < t1 && c < a.N;
        const float* r = in ? rows + (size_t)(t + tok) * ld + c : rows;
        bw_cp16(buf + tok * C::LDN + c, r + (in ? q_col : 0), in);
        bw_cp16(buf + C::QK + tok * C::LDN + c, r + (in ? k_col : 0), in);
    }
    float* sA = buf + 2 * C::QK + BW_B * C::LDV;
    if (tid < 64 * MT) {
        const int tok = tid / (4 * MT), c = tid % (4 * MT) * 4;
        const bool in = t + tok < t1 && c < cols;
        bw_cp16(buf + 2 * C::QK + tok * C::LDV + c, in ? rows + (size_t)(t + tok) * ld + v_col + c : rows, in);
    } else if (tid < 64 * MT + 64) {
        const int e = tid - 64 * MT;
        bw_cp16(sA + (e >> 2) * BW_LD + (e & 3) * 4, coef + e * 4, true);
    } else if (DELTA && tid < 64 * MT + 128) {
        const int e = tid - 64 * MT - 64;
        bw_cp16(sA + BW_B * BW_LD + (e >> 2) * BW_LD + (e & 3) * 4, coef + 256 + e * 4, true);
    }
    if (tid < BW_TAIL / 4) bw_cp16(buf + C::G_AT + tid * 4, coef + 512 + tid * 4, true);
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// What the tensor cores cut off a sum lies between nothing and one unit of its 24 bits: on the average over mantissas 0.36 x
// 2^-23 of it, and 0.54 x 2^-23 where the sum takes two steps, the first of half the size.  The mean is added back with the
// small products; what is left has no sign.
template <int STEPS>
__device__ __forceinline__ float bw_total(float c, float d) {
    return c + fmaf(c, (STEPS == 2 ? 0.54f : 0.36f) * 1.1920929e-7f, d);
}

// Partial products S0^T x of a warp's rows, x the q or k rows of a block (IN of them): [16 MT columns] x [16 tokens] into
// part[token][column].  A product whose sum the one before it adds to waits for that, so products of different sums stand between.
template <int NT, int MT, int IN>
__device__ __forceinline__ void bw_read_out(const float* const (&x)[IN], const uint32_t (&sh)[MT][NT][4], const uint32_t (&sl)[MT][NT][4],
                                            float* const (&part)[IN], int row0, int g, int t) {
    using C = BwSmem<NT, MT, true, false>;
    constexpr int HALVES = 2 / MT;                              // of the tokens at a time: as many accumulators with 32 columns as with 16
#pragma unroll
    for (int h0 = 0; h0 < 2; h0 += HALVES) {
        float acc[IN][MT][HALVES][4] = {}, low[IN][MT][HALVES][4] = {};
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            uint32_t bh[IN][HALVES][2], bl[IN][HALVES][2];
#pragma unroll
            for (int i = 0; i < IN; ++i)
#pragma unroll
                for (int h = 0; h < HALVES; ++h) {
                    const float2 v = *reinterpret_cast<const float2*>(x[i] + ((h0 + h) * 8 + g) * C::LDN + row0 + nt * 8 + 2 * t);
                    bw_split(v.x, bh[i][h][0], bl[i][h][0]);
                    bw_split(v.y, bh[i][h][1], bl[i][h][1]);
                }
#pragma unroll
            for (int step = 0; step < 3; ++step)
#pragma unroll
                for (int i = 0; i < IN; ++i)
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                        for (int h = 0; h < HALVES; ++h) {
                            if (step == 0) bw_mma(low[i][mt][h], sl[mt][nt], bh[i][h]);
                            if (step == 1) bw_mma(acc[i][mt][h], sh[mt][nt], bh[i][h]);
                            if (step == 2) bw_mma(low[i][mt][h], sh[mt][nt], bl[i][h]);
                        }
        }
#pragma unroll
        for (int i = 0; i < IN; ++i)
#pragma unroll
            for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                for (int h = 0; h < HALVES; ++h) {
                    float* p = part[i] + ((h0 + h) * 8 + 2 * t) * C::LDP + mt * 16 + g;
                    p[0] = bw_total<NT>(acc[i][mt][h][0], low[i][mt][h][0]);
                    p[C::LDP] = bw_total<NT>(acc[i][mt][h][1], low[i][mt][h][1]);
                    p[8] = bw_total<NT>(acc[i][mt][h][2], low[i][mt][h][2]);
                    p[C::LDP + 8] = bw_total<NT>(acc[i][mt][h][3], low[i][mt][h][3]);
                }
    }
}

template <int LDP>
__device__ __forceinline__ float bw_sum_parts(const float* __restrict__ part, int tok, int col) {
    float v[BW_WARPS];
#pragma unroll
    for (int w = 0; w < BW_WARPS; ++w) v[w] = part[(w * BW_B + tok) * LDP + col];
    return ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
}

// Barriers of part of a CTA: `sync` waits, `arrive` does not.
__device__ __forceinline__ void bw_sync(int id, int threads) { asm volatile("barrier.cta.sync.aligned %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void bw_arrive(int id, int threads) { asm volatile("barrier.cta.arrive.aligned %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
constexpr int BW_BAR_STATE = 1, BW_BAR_FULL = 2, BW_BAR_DONE = 5;              // FULL + stage, DONE + block & 1

// Columns col0 .. col0 + cols - 1 of a head's state through a portion token by token in plain float32, from the slot's state as
// the portion found it; a warp a column, its lanes the rows.  A block multiplies all its tokens with zeros above the
// diagonal and adds products of halves, which holds for finite numbers only: an infinity or NaN would reach the block's
// earlier tokens, and an infinity become NaN.  One anywhere in a CTA's rows, gates or state shows in a result or in the
// last state, so the CTA then walks its columns again here, where a token's number reaches what follows it and nothing else.
template <bool DELTA>
__device__ __noinline__ void bw_walk_tokens(const BlockWalk& a, const float* rows, long ld, int q_col, int k_col, int v_col, int s, int h, int col0, int cols) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t0 = a.q_start[s], t1 = a.q_start[s + 1];
    const long sr = a.state_vn ? 1 : a.V, sc = a.state_vn ? a.N : 1;
    const float skip = a.skip_any != nullptr ? load_dyn(a.skip_any, a.skip_dt, h) : 0.f;
    const bool fresh = a.positions[t0] == 0;
    for (int c = warp; c < cols; c += blockDim.x >> 5) {
        float* st = a.state + (size_t)a.slots[s] * a.state_stride + a.s_off + (size_t)h * a.N * a.V + (col0 + c) * sc;
        float S[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) S[i] = !fresh && lane + 32 * i < a.N ? st[(lane + 32 * i) * sr] : 0.f;
        for (int t = t0; t < t1; ++t) {
            const float* r = rows + (size_t)t * ld;
            const float v = r[v_col + c], g = a.gates != nullptr ? a.gates[(size_t)t * a.ldg + a.g_off + h] : a.decay[h];
            const float w = a.w_off >= 0 ? a.gates[(size_t)t * a.ldg + a.w_off + h] : 1.f;
            float k[4], q[4], sk = 0.f, sq = 0.f, kq = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const bool in = lane + 32 * i < a.N;
                k[i] = in ? r[k_col + lane + 32 * i] : 0.f;
                q[i] = in ? r[q_col + lane + 32 * i] : 0.f;
                if (DELTA) {
                    sk = fmaf(S[i], k[i], sk);
                    sq = fmaf(S[i], q[i], sq);
                    kq = fmaf(k[i], q[i], kq);
                }
            }
            float o;
            if (DELTA) {
                const float u = w * (v - g * warp_sum(sk));
                o = fmaf(warp_sum(kq), u, g * warp_sum(sq));
#pragma unroll
                for (int i = 0; i < 4; ++i) if (lane + 32 * i < a.N) S[i] = fmaf(k[i], u, g * S[i]);
            } else {
                const float u = w * v;
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (lane + 32 * i < a.N) {
                        S[i] = fmaf(g, S[i], u * k[i]);
                        sq = fmaf(S[i], q[i], sq);
                    }
                o = warp_sum(sq);
            }
            if (a.skip_any != nullptr) o = fmaf(skip, v, o);
            if (lane == 0) a.out[(size_t)t * a.ldo + (size_t)h * a.V + col0 + c] = o;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) if (lane + 32 * i < a.N) st[(lane + 32 * i) * sr] = S[i];
    }
}

// The request with the n-th longest portion (of equal ones the first counts as the longer), for up to 32 requests; beyond, the
// n-th: CTAs start in this order, so a walk of many blocks does not begin when the short ones have ended.
__device__ __forceinline__ int bw_nth_longest(const int* __restrict__ q_start, int S, int n) {
    if (S == 1 || S > 32) return n;
    const int lane = threadIdx.x & 31, len = lane < S ? q_start[lane + 1] - q_start[lane] : -1;
    int rank = 0;
    for (int j = 0; j < S; ++j) {
        const int other = __shfl_sync(0xffffffffu, len, j);
        rank += other > len || (other == len && j < lane);
    }
    return __ffs(__ballot_sync(0xffffffffu, lane < S && rank == n)) - 1;
}

__device__ __forceinline__ bool bw_finite(float x) { return fabsf(x) <= 3.402823466e38f; }

// Eight warps hold the state, bring the blocks and make the results.  Without the delta rule a block's u depends on no state, so
// a block's results (the sums over the warps' rows, and A u in float32 multiply-adds: cut in two tf32 numbers it was further from 64
// bits where portions are short, 1.0e-7 and 0.9e-7 for 17 tokens) are made beside the next block, behind its one barrier.
// With HELP eight more bring the blocks and turn a
// block's partial sums into results while the state warps, which then do only what the next block waits for, are at the next
// one.  A helper passes DONE of block i before it refills the stage of block i - 1 (whose update came before) with block
// i + 2, makes block i's results and then reports block i + 2 FULL, so the state warps write block i + 2's sums over block
// i's only after these were read.  That shortens the delta rule's long chain where a CTA has its SM to itself (185 -> 148 us
// for 2,048 tokens of 16 heads); with two CTAs on an SM, and without the delta rule, the extra warps only get in the
// way (linear attention, 1,900 tokens of two requests: 88 -> 107 us).  The least number of CTAs an SM keeps the compiler from
// saving registers: with 80 a thread and three CTAs on an SM the same walk took 100 us, with 126 it takes 86.
template <int NT, int MT, bool DELTA, bool HELP>
__global__ void __launch_bounds__((HELP ? 2 : 1) * BW_THREADS, HELP ? 1 : 2)
block_walk_kernel(const __grid_constant__ BlockWalk a) {
    using C = BwSmem<NT, MT, DELTA, HELP>;
    constexpr int COLS = 16 * MT;
    constexpr bool PIPE = !DELTA;                               // a block's results are made beside the next block
    static_assert(!PIPE || (MT == 1 && !HELP), "without the delta rule 16 columns and no helpers");
    extern __shared__ __align__(16) float bw_smem[];
    float* part_p = bw_smem + C::STAGES * C::STAGE;
    float* parts_r = part_p + (DELTA ? C::PART : 0);
    float* us = parts_r + C::TURNS * C::PART;
    griddep_launch();
    griddep_wait();
    const int s = bw_nth_longest(a.q_start, a.S, blockIdx.z), h = blockIdx.y, kvh = h / (a.heads / a.G), t0 = a.q_start[s], t1 = a.q_start[s + 1];
    if (t1 <= t0 || (a.alone && t1 - t0 == 1)) return;
    const int tid = threadIdx.x & (BW_THREADS - 1), warp = tid >> 5, lane = tid & 31;
    const int col0 = blockIdx.x * COLS, cols = a.V - col0 < COLS ? a.V - col0 : COLS;

    const float* rows = a.act ? a.act_rows : a.rows;
    const long ld = a.act ? a.ld_act : a.ld;
    const int q_col = (a.act ? 0 : a.q_off) + kvh * a.N, k_col = (a.act ? a.G * a.N : a.k_off) + kvh * a.N;
    const int v_col = (a.act ? 2 * a.G * a.N : a.v_off) + h * a.V + col0;
    const float* coef = a.coef + ((size_t)bw_first_block(a.q_start, s) * a.heads + h) * BW_COEF;
    const size_t coef_step = (size_t)a.heads * BW_COEF;
    // What a thread copies of a whole block lies in the same place of every block: one address a row piece and one of v, A or M,
    // moved on by a block each time.  (Looked up block by block, the copies took a fifth of the walk's instructions.)
    constexpr int PIECES = 16 * NT, ROWS = BW_THREADS / PIECES;  // 16-byte pieces of a row of q or k; rows at a time
    const int mrow = tid / PIECES, mcol = tid % PIECES * 4, side = tid - 64 * MT;
    const float* from = rows + (size_t)(t0 + mrow) * ld + q_col + mcol;
    const float* from2 = side < 0 ? rows + (size_t)(t0 + tid / (4 * MT)) * ld + v_col + tid % (4 * MT) * 4 : coef + side * 4;
    const bool has = mcol < a.N, has2 = side < 0 ? tid % (4 * MT) * 4 < cols : side < (DELTA ? 128 : 64);
    const long from2_step = side < 0 ? BW_B * ld : (long)coef_step, k_minus_q = k_col - q_col;
    const int to2 = side < 0 ? 2 * C::QK + tid / (4 * MT) * C::LDV + tid % (4 * MT) * 4
                             : 2 * C::QK + BW_B * C::LDV + (side >> 2) * BW_LD + (side & 3) * 4;          // M's rows follow A's
    auto fetch = [&](int t, int stage) {                        // the next block in order, which starts at token t
        float* buf = bw_smem + stage * C::STAGE;
        if (t + BW_B <= t1) {
            if (has) {
                float* to = buf + mrow * C::LDN + mcol;
#pragma unroll
                for (int i = 0; i < BW_B / ROWS; ++i) {
                    bw_cp16(to + i * ROWS * C::LDN, from + i * ROWS * ld);
                    bw_cp16(to + C::QK + i * ROWS * C::LDN, from + k_minus_q + i * ROWS * ld);
                }
            }
            if (has2) bw_cp16(buf + to2, from2);
            if (tid < BW_TAIL / 4) bw_cp16(buf + C::G_AT + tid * 4, coef + 512 + tid * 4);
            asm volatile("cp.async.commit_group;" ::: "memory");
        } else {
            bw_fetch<NT, MT, DELTA, HELP>(buf, a, rows, ld, q_col, k_col, v_col, cols, coef, t, t1, tid);
        }
        from += BW_B * ld;
        from2 += from2_step;
        coef += coef_step;
    };
    if (a.N < 64 * NT || cols < COLS) {                         // columns that no block brings
        for (int i = threadIdx.x; i < C::STAGES * C::STAGE; i += (HELP ? 2 : 1) * BW_THREADS) bw_smem[i] = 0.f;
        __syncthreads();
    }
    const float skip = a.skip_any != nullptr ? load_dyn(a.skip_any, a.skip_dt, h) : 0.f;
    bool odd = false;                                           // a number that is not finite has been seen
    auto results = [&](int t, int stage, int turn) {            // thread = column tid % COLS of token tid / COLS and, with MT, eight on
        const int col = tid % COLS, tok = tid / COLS;
        const float* sv = bw_smem + stage * C::STAGE + 2 * C::QK;
        const float* sA = sv + BW_B * C::LDV;
        const float* gam = bw_smem + stage * C::STAGE + C::G_AT;
        const float* u = (DELTA ? us + turn * C::U : sv) + col;
        float o0[MT], o1[MT];
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            o0[m] = gam[tok + 8 * m] * bw_sum_parts<C::LDP>(parts_r + turn * C::PART, tok + 8 * m, col);
            o1[m] = skip * sv[(tok + 8 * m) * C::LDV + col];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float u0 = u[(4 * j) * C::LDV], u1 = u[(4 * j + 1) * C::LDV], u2 = u[(4 * j + 2) * C::LDV], u3 = u[(4 * j + 3) * C::LDV];
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const float4 w = *reinterpret_cast<const float4*>(sA + (tok + 8 * m) * BW_LD + 4 * j);
                o0[m] = fmaf(w.x, u0, o0[m]);
                o1[m] = fmaf(w.y, u1, o1[m]);
                o0[m] = fmaf(w.z, u2, o0[m]);
                o1[m] = fmaf(w.w, u3, o1[m]);
            }
        }
#pragma unroll
        for (int m = 0; m < MT; ++m)
            if (t + tok + 8 * m < t1 && col < cols) {
                const float o = o0[m] + o1[m];
                odd |= !bw_finite(o);
                a.out[(size_t)(t + tok + 8 * m) * a.ldo + (size_t)h * a.V + col0 + col] = o;
            }
    };

    if (HELP && threadIdx.x >= BW_THREADS) {
        const bool more = t0 + BW_B < t1;
        fetch(t0, 0);
        if (more) {
            fetch(t0 + BW_B, 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        bw_arrive(BW_BAR_FULL, 2 * BW_THREADS);
        if (more) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            bw_arrive(BW_BAR_FULL + 1, 2 * BW_THREADS);
        }
        int b = 0, turn = 0;
        for (int t = t0; t < t1; t += BW_B, turn ^= 1) {
            const int ahead = b == 0 ? 2 : b - 1;               // the stage of the block before, for the one two blocks on
            bw_sync(BW_BAR_DONE + turn, 2 * BW_THREADS);
            if (t + 2 * BW_B < t1) fetch(t + 2 * BW_B, ahead);
            results(t, b, turn);
            if (t + 2 * BW_B < t1) {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
                bw_arrive(BW_BAR_FULL + ahead, 2 * BW_THREADS);
            }
            b = b == 2 ? 0 : b + 1;
        }
        if (__syncthreads_or(odd)) bw_walk_tokens<DELTA>(a, rows, ld, q_col, k_col, v_col, s, h, col0, cols);
        return;
    }

    // ---------------------------------------------------------------------- the state
    // thread (g, tq) of a warp holds columns g and g + 8 of every 16, rows 2 tq and 2 tq + 1 of every fragment
    if (!HELP) {
        fetch(t0, 0);
        if (t0 + BW_B < t1) fetch(t0 + BW_B, 1);
        else asm volatile("cp.async.commit_group;" ::: "memory");
    }
    const int g = lane >> 2, tq = lane & 3, row0 = warp * 8 * NT;
    float* st = a.state + (size_t)a.slots[s] * a.state_stride + a.s_off + (size_t)h * a.N * a.V;
    const long sr = a.state_vn ? 1 : a.V, sc = a.state_vn ? a.N : 1;
    const bool fresh = a.positions[t0] == 0;
    float S[MT][NT][4];
#pragma unroll
    for (int f = 0; f < MT * NT; ++f)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int row = row0 + f % NT * 8 + 2 * tq + (e & 1), col = f / NT * 16 + g + (e >> 1) * 8;
            S[f / NT][f % NT][e] = (!fresh && row < a.N && col < cols) ? st[row * sr + (col0 + col) * sc] : 0.f;
        }
    int b = 0, turn = 0;
    for (int t = t0; t < t1; t += BW_B) {
        if (HELP) {
            bw_sync(BW_BAR_FULL + b, 2 * BW_THREADS);
        } else {
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncthreads();                                    // the block's rows are here, and everyone has left the block before
            const int ahead = b + 2 < C::STAGES ? b + 2 : b + 2 - C::STAGES;
            if (t + 2 * BW_B < t1) fetch(t + 2 * BW_B, ahead);
            else asm volatile("cp.async.commit_group;" ::: "memory");
        }
        const float* sq = bw_smem + b * C::STAGE;
        const float* sk = sq + C::QK;
        const float* sv = sk + C::QK;
        const float* sM = sq + C::M_AT;
        const float* gam = sq + C::G_AT;
        const float* suf = gam + BW_B;
        uint32_t sh[MT][NT][4], sl[MT][NT][4];
#pragma unroll
        for (int f = 0; f < MT * NT; ++f) {                     // rows 2 tq are the operand's k index tq, rows 2 tq + 1 its tq + 4
            const float(&x)[4] = S[f / NT][f % NT];
            uint32_t(&xh)[4] = sh[f / NT][f % NT], (&xl)[4] = sl[f / NT][f % NT];
            bw_split(x[0], xh[0], xl[0]);
            bw_split(x[2], xh[1], xl[1]);
            bw_split(x[1], xh[2], xl[2]);
            bw_split(x[3], xh[3], xl[3]);
        }
        const float* u = sv;
        if (DELTA) {
            float* su = us + turn * C::U;
            const float* const in[2] = {sk, sq};
            float* const to[2] = {part_p + warp * BW_B * C::LDP, parts_r + turn * C::PART + warp * BW_B * C::LDP};
            bw_read_out<NT, MT, 2>(in, sh, sl, to, row0, g, tq);
            HELP ? bw_sync(BW_BAR_STATE, BW_THREADS) : __syncthreads();
            // thread: token lane % 16 of column tid / 16 of every 16; the 16 tokens of a column meet in half a warp
            const int tok = lane & 15;
            const float4* m4 = reinterpret_cast<const float4*>(sM + tok * BW_LD);
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
                const int col = mt * 16 + (tid >> 4);
                const float e = sv[tok * C::LDV + col] - gam[tok] * bw_sum_parts<C::LDP>(part_p, tok, col);
                float u0 = 0.f, u1 = 0.f;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float4 m = m4[j];
                    u0 = fmaf(m.x, __shfl_sync(0xffffffffu, e, 4 * j, 16), u0);
                    u1 = fmaf(m.y, __shfl_sync(0xffffffffu, e, 4 * j + 1, 16), u1);
                    u0 = fmaf(m.z, __shfl_sync(0xffffffffu, e, 4 * j + 2, 16), u0);
                    u1 = fmaf(m.w, __shfl_sync(0xffffffffu, e, 4 * j + 3, 16), u1);
                }
                su[tok * C::LDV + col] = u0 + u1;
            }
            u = su;
        }
        if (!DELTA) {
            const float* const in[1] = {sq};
            float* const to[1] = {parts_r + turn * C::PART + warp * BW_B * C::LDP};
            bw_read_out<NT, MT, 1>(in, sh, sl, to, row0, g, tq);
        }
        if (HELP) bw_sync(BW_BAR_STATE, BW_THREADS);            // u and the partial sums of r are there
        else if (!PIPE) __syncthreads();
        else if (t > t0) results(t - BW_B, b == 0 ? C::STAGES - 1 : b - 1, turn ^ 1);
        if (HELP) bw_arrive(BW_BAR_DONE + turn, 2 * BW_THREADS);
        uint32_t kh[2][NT][2], kl[2][NT][2];
#pragma unroll
        for (int ks = 0; ks < 2; ++ks)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                bw_split(sk[(ks * 8 + tq) * C::LDN + row0 + nt * 8 + g], kh[ks][nt][0], kl[ks][nt][0]);
                bw_split(sk[(ks * 8 + tq + 4) * C::LDN + row0 + nt * 8 + g], kh[ks][nt][1], kl[ks][nt][1]);
            }
        const float total = gam[BW_B - 1], rest = gam[2 * BW_B];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
            float up[NT][4] = {}, low[NT][4] = {};
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) {
                const int ta = ks * 8 + tq;
                const float w0 = suf[ta], w1 = suf[ta + 4];
                const float* u0 = u + ta * C::LDV + mt * 16 + g;
                uint32_t ah[4], al[4];
                bw_split(u0[0] * w0, ah[0], al[0]);
                bw_split(u0[8] * w0, ah[1], al[1]);
                bw_split(u0[4 * C::LDV] * w1, ah[2], al[2]);
                bw_split(u0[4 * C::LDV + 8] * w1, ah[3], al[3]);
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) bw_mma(low[nt], al, kh[ks][nt]);
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) bw_mma(up[nt], ah, kh[ks][nt]);
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) bw_mma(low[nt], ah, kl[ks][nt]);
            }
            if (!HELP && !PIPE && mt == MT - 1) results(t, b, 0);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) S[mt][nt][e] = fmaf(total, S[mt][nt][e], fmaf(rest, S[mt][nt][e], bw_total<2>(up[nt][e], low[nt][e])));
        }
        b = b == C::STAGES - 1 ? 0 : b + 1;
        if (C::TURNS == 2) turn ^= 1;
    }
    if (PIPE) {
        __syncthreads();                                        // the last block's partial sums are there
        results(t0 + (t1 - t0 - 1) / BW_B * BW_B, b == 0 ? C::STAGES - 1 : b - 1, turn ^ 1);
    }
#pragma unroll
    for (int f = 0; f < MT * NT; ++f)
#pragma unroll
        for (int e = 0; e < 4; ++e) odd |= !bw_finite(S[f / NT][f % NT][e]);
    if (__syncthreads_or(odd)) {
        bw_walk_tokens<DELTA>(a, rows, ld, q_col, k_col, v_col, s, h, col0, cols);
        return;
    }
#pragma unroll
    for (int f = 0; f < MT * NT; ++f)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int row = row0 + f % NT * 8 + 2 * tq + (e & 1), col = f / NT * 16 + g + (e >> 1) * 8;
            if (row < a.N && col < cols) st[row * sr + (col0 + col) * sc] = S[f / NT][f % NT][e];
        }
}

template <int NT, int MT, bool DELTA, bool HELP>
static int launch_block_walk(const BlockWalk& a, cudaStream_t stream) {
    constexpr int bytes = BwSmem<NT, MT, DELTA, HELP>::TOTAL * 4;
    auto kern = block_walk_kernel<NT, MT, DELTA, HELP>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return AIEN_E_STATE;
    constexpr int threads = (HELP ? 2 : 1) * BW_THREADS;
    static const int resident = resident_ctas(kern, threads, bytes);
    const dim3 grid((a.V + 16 * MT - 1) / (16 * MT), a.heads, a.S);
    if (resident == 1) launch_chain(kern, grid, dim3(threads), (size_t)bytes, stream, a);         // see griddep_wait
    else kern<<<grid, threads, bytes, stream>>>(a);
    return launch_status();
}

// Without the delta rule 16 columns a CTA are the faster whatever the load (2,000 tokens of three requests, 32 heads of 128 x
// 64: 110 us, with 32 columns 139; 1,900 of two, 16 heads of 128 x 128: 86 and 102): a CTA's chain is the longer with 32.  The
// delta rule has twice the work per block on the rows of q and k, which 32 columns share: where more CTAs than SMs walk
// anyway, a layer of 1,239 tokens of two requests, 32 heads of 128 x 128, takes 356 us with 32 columns and 388 with 16 (1,186
// of five requests, 16 heads: 173 and 182).  With fewer, a CTA of 16 columns and helpers has an SM to itself.
template <int NT>
static int dispatch_block_walk(const BlockWalk& a, cudaStream_t stream) {
    int sms = 148, dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
    if (!a.delta) return launch_block_walk<NT, 1, false, false>(a, stream);
    if ((long)((a.V + 15) / 16) * a.heads * (a.S - a.alone) <= sms) return launch_block_walk<NT, 1, true, true>(a, stream);
    return a.V <= 16 ? launch_block_walk<NT, 1, true, false>(a, stream) : launch_block_walk<NT, 2, true, false>(a, stream);
}

}  // namespace aien

using namespace aien;

// Whether the walk takes these sizes; the rows besides have to start on 16-byte boundaries (aien_block_walk refuses others).
AIEN_API int aien_block_walk_supports(int heads, int G, int N, int V, int delta) {
    if (heads <= 0 || G <= 0 || heads % G || N <= 0 || N > 128 || N % 4 || V <= 0 || V % 4 || heads > 65535) return 0;
    const long smem = 2L * BW_B * (N + 4) + (2L * BW_B + (delta ? 256 : 0)) * (heads / G);       // as the launch of block_coef_kernel counts
    return smem * 4 <= 160 * 1024;
}

// rows float32 [T, ld] with q (G heads of N numbers) at q_off, k at k_off, v (`heads` heads of V) at v_off; act: they pass
// silu first.  gates float32 [T, ldg]: decay of head h at g_off + h and (w_off >= 0) its weight at w_off + h: beta with
// delta, else a factor on v; gates null: decay[heads] for every token.  skip (in skip_dt, or null): o += skip[h] v.
// state: rows of state_stride floats, a head's matrix at s_off + h N V, [V][N] with state_vn, else [N][V].  Request s (tokens
// q_start[s] .. q_start[s+1]) continues from slot slots[s], from zeros where its first position is 0.  out float32 [T, ldo].
// alone: how many requests bring one token and are served elsewhere; 0: none is left out.
// scratch: float32, (T / 16 + S) * heads * 548 numbers (the blocks' coefficients) and with act T * (2 G N + heads V) more.
AIEN_API int aien_block_walk(const float* rows, long ld, int q_off, int k_off, int v_off, int act, const float* gates, long ldg, int g_off,
                             int w_off, const float* decay, int delta, const void* skip, int skip_dt, float* state, size_t state_stride,
                             size_t s_off, int state_vn, const int* slots, const int* q_start, const int* positions, float* out, long ldo,
                             int T, int S, int heads, int G, int N, int V, int alone, float* scratch, cudaStream_t stream) {
    if (S <= 0 || T <= 0) return 0;
    if (!aien_block_walk_supports(heads, G, N, V, delta) || S > 65535 || G > 65535 || scratch == nullptr || (gates == nullptr && decay == nullptr)) return AIEN_E_SHAPE;
    if ((reinterpret_cast<uintptr_t>(rows) | reinterpret_cast<uintptr_t>(scratch)) & 15 || (ld | q_off | k_off | v_off) & 3) return AIEN_E_ALIGN;
    const long blocks = T / BW_B + S, coefs = blocks * heads * BW_COEF;
    BlockWalk a{rows, ld, q_off, k_off, v_off, gates, ldg, g_off, w_off, decay, scratch + coefs, 2L * G * N + (long)heads * V, act, delta, scratch,
                skip, skip_dt, state, state_stride, s_off, state_vn, slots, q_start, positions, out, ldo, T, S, heads, G, N, V, alone};
    const int per = heads / G, smem = 4 * (2 * BW_B * (N + 4) + 2 * BW_B * per + (delta ? 256 * per : 0));
    auto coef = delta ? block_coef_kernel<true> : block_coef_kernel<false>;
    if (smem > 48 * 1024 && cudaFuncSetAttribute(coef, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return AIEN_E_STATE;
    coef<<<dim3((unsigned)blocks, G), 256, smem, stream>>>(a);              // plain: see griddep_wait
    const int rc = launch_status();
    if (rc != 0) return rc;
    return N <= 64 ? dispatch_block_walk<1>(a, stream) : dispatch_block_walk<2>(a, stream);
}
