// The gated delta rule: per value head a float32 state S [D][V] that every token first decays, then corrects along
// its key, then reads with its query:
//     S <- g S ;   u = beta (v - S^T k) ;   S <- S + k u^T ;   o = S^T q
// (g a decay in (0, 1], beta in (0, 1), k a unit vector; heads/G value heads share one q/k head).  Column j of S
// never meets another column: S^T k, u, the update and S^T q are all per column.  So a thread owns part of one column
// in registers and a portion is walked token by token with no barrier inside a chunk of tokens.  Both products are
// taken from the state as the token finds it, in one pass over the registers:
//     a = S^T k ,  b = S^T q ,  c = k . q ;   u = beta (v - g a) ;   o = g b + c u ;   S <- g S + k u^T
// which is the same arithmetic with the decay drawn out of the sums.  A warp holds 32/RS columns x RS row ranges (the
// partial sums meet through log2(RS) shuffles), a CTA four warps' columns of one head of one request.  What the
// walk is bound by is the reading of k and q from shared memory, once per token and thread: the row ranges lie
// DPT + 4 floats apart there, so that the 16-byte reads of a warp fall into different banks.  q, k, v, g and beta of
// the next chunk of tokens arrive through cp.async while the current one is walked, and the next token's are taken
// into registers while the current one's sums are on their way.  Every operation is float32 and a token's are the
// same whatever the cut of the prompt or the batch, so its output depends on the tokens before it only through S.
// (Single tokens have a kernel of their own, which adds a column's products in another order.)
//
// The state lives in the request's slot between steps (a portion whose first token has position 0 starts from zero).
//
// grouped_gated_rmsnorm: out = o / sqrt(mean_group(o^2) + eps) * w[c mod group] * act(gate), the norm taken over
// every group of `group` neighbouring columns (one head) with one weight vector shared by the groups.
#include "common.cuh"
#include "gated_rows.cuh"
#include <math.h>

namespace aien {

constexpr int DR_THREADS = 128;

__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

template <int DPT, int RS>
struct DeltaCfg {
    static constexpr int DP = RS * DPT;                        // rows of S, padded
    static constexpr int PS = DPT == 4 ? 4 : DPT + 4;          // floats between two row ranges of k (or q) in shared memory
    static constexpr int CW = 32 / RS;                         // columns per warp
    static constexpr int COLS = (DR_THREADS / 32) * CW;        // columns of S per CTA
    static constexpr int KQ = RS * PS;                         // floats of k (or q) per token, padded
    static constexpr int ROW = 2 * KQ + COLS + 4;              // floats per token: k | q | v | g, beta, -, -
    static constexpr int TC = 2 * 16 * ROW * 4 <= 48 * 1024 ? 16 : 8;   // tokens per chunk: two chunks within 48 KB
};

// What one thread copies for every token of a chunk: up to NE pieces, found once per kernel (where in the token's
// row of the source, where in its row of shared memory, 16 bytes or 4), so that a chunk's copies are an address
// and a cp.async each.  The walk shares its warps with the copies, so their instructions count.
template <int DPT, int RS>
struct DeltaPieces {
    using C = DeltaCfg<DPT, RS>;
    static constexpr int NE = (2 * C::DP + C::COLS + 2 + DR_THREADS - 1) / DR_THREADS;
    const float* src[NE];
    long stride[NE];
    int dst[NE];
    int kind[NE];                                              // 0: none, 1: 4 bytes, 2: 16 bytes; +4: always zero

    __device__ __forceinline__ void find(bool vec, const float* qkv, long ld, int q_col, int k_col, int v_col, const float* gb,
                                         long ldgb, int h, int heads, int D, int V, int col0) {
        const int unit = vec ? 4 : 1;
        const int n_kq = C::DP / unit, n_v = C::COLS / unit;
#pragma unroll
        for (int i = 0; i < NE; ++i) {
            const int e = threadIdx.x + i * DR_THREADS;
            src[i] = qkv; stride[i] = ld; dst[i] = 0; kind[i] = 0;
            if (e < 2 * n_kq) {
                const int which = e >= n_kq, r = (e - which * n_kq) * unit;        // 0: k, 1: q; row r
                dst[i] = which * C::KQ + (r / DPT) * C::PS + (r % DPT);
                src[i] = qkv + (which ? q_col : k_col) + r;
                kind[i] = (vec ? 2 : 1) + (r < D ? 0 : 4);
            } else if (e < 2 * n_kq + n_v) {
                const int c = (e - 2 * n_kq) * unit;
                dst[i] = 2 * C::KQ + c;
                src[i] = qkv + v_col + col0 + c;
                kind[i] = (vec ? 2 : 1) + (col0 + c < V ? 0 : 4);
            } else if (e < 2 * n_kq + n_v + 2) {
                const int w = e - 2 * n_kq - n_v;                                   // 0: decay, 1: beta
                dst[i] = 2 * C::KQ + C::COLS + w;
                src[i] = gb + w * heads + h;
                stride[i] = ldgb;
                kind[i] = 1;
            }
        }
    }

    __device__ __forceinline__ void fetch(float* __restrict__ buf, int t, int t1) const {
#pragma unroll 4
        for (int tok = 0; tok < C::TC; ++tok) {
            const int tt = t + tok;
#pragma unroll
            for (int i = 0; i < NE; ++i) {
                if (kind[i] == 0) continue;
                float* d = buf + tok * C::ROW + dst[i];
                const bool wide = (kind[i] & 2) != 0;
                if (tt < t1 && kind[i] < 4) {
                    const float* sp = src[i] + (size_t)tt * stride[i];
                    if (wide) cp_async16(d, sp);
                    else cp_async4(d, sp);
                } else if (wide) {
                    *reinterpret_cast<float4*>(d) = make_float4(0.f, 0.f, 0.f, 0.f);
                } else {
                    *d = 0.f;
                }
            }
        }
        cp_async_commit();
    }
};

template <int DPT, int RS>
__global__ void __launch_bounds__(DR_THREADS)
delta_rule_kernel(const float* __restrict__ qkv, long ld, int q_off, int k_off, int v_off, const float* __restrict__ gb, long ldgb,
                  float* __restrict__ state, size_t state_stride, size_t s_off, const int* __restrict__ slot_map,
                  const int* __restrict__ q_start, const int* __restrict__ positions, float* __restrict__ o, long ldo,
                  int heads, int G, int D, int V, int longest) {
    using C = DeltaCfg<DPT, RS>;
    constexpr int N4 = DPT / 4;
    __shared__ __align__(16) float bufs[2][C::TC * C::ROW];
    const int s = blockIdx.z, h = blockIdx.y, kvh = h / (heads / G);
    const int t0 = q_start[s], t1 = q_start[s + 1];
    if (t1 <= t0 || t1 - t0 > longest) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rs = lane / C::CW, cw = lane % C::CW;
    const int col0 = blockIdx.x * C::COLS, cl = warp * C::CW + cw, col = col0 + cl;
    const bool col_ok = col < V;
    const int i0 = rs * DPT;
    float* S = state + (size_t)slot_map[s] * state_stride + s_off + (size_t)h * D * V;
    const int q_col = q_off + kvh * D, k_col = k_off + kvh * D, v_col = v_off + h * V;

    // 16-byte copies where every piece of four neighbours starts on a 16-byte boundary and lies inside or outside whole
    const bool vec = ((reinterpret_cast<uintptr_t>(qkv) & 15) == 0) && ((ld | q_col | k_col | v_col | D | V) & 3) == 0;
    DeltaPieces<DPT, RS> pieces;
    pieces.find(vec, qkv, ld, q_col, k_col, v_col, gb, ldgb, h, heads, D, V, col0);
    pieces.fetch(bufs[0], t0, t1);
    // the thread's rows of its column, two to a register pair: the sums and the update run on packed pairs
    // (fma.rn.f32x2, each half rounded as the single operation is), which halves the instructions of the walk
    float2 Sr[2 * N4];
    const bool fresh = positions[t0] == 0;
#pragma unroll
    for (int i = 0; i < 2 * N4; ++i) {
        Sr[i].x = (!fresh && col_ok && i0 + 2 * i < D) ? S[(size_t)(i0 + 2 * i) * V + col] : 0.f;
        Sr[i].y = (!fresh && col_ok && i0 + 2 * i + 1 < D) ? S[(size_t)(i0 + 2 * i + 1) * V + col] : 0.f;
    }

    float4 kc[N4], qc[N4];
    float vj, g, beta;
    auto take = [&](const float* row) {                        // one token's numbers into registers
        const float4* kk = reinterpret_cast<const float4*>(row + rs * C::PS);
        const float4* qq = reinterpret_cast<const float4*>(row + C::KQ + rs * C::PS);
#pragma unroll
        for (int i = 0; i < N4; ++i) { kc[i] = kk[i]; qc[i] = qq[i]; }
        vj = row[2 * C::KQ + cl];
        g = row[2 * C::KQ + C::COLS];
        beta = row[2 * C::KQ + C::COLS + 1];
    };

    int b = 0;
    for (int t = t0; t < t1; t += C::TC, b ^= 1) {
        cp_async_wait_all();
        __syncthreads();                                        // chunk b has arrived; everyone is done with chunk b^1
        if (t + C::TC < t1) pieces.fetch(bufs[b ^ 1], t + C::TC, t1);
        const int n = t1 - t < C::TC ? t1 - t : C::TC;
        take(bufs[b]);
        for (int tt = 0; tt < n; ++tt) {
            float2 a0 = make_float2(0.f, 0.f), a1 = a0, b0 = a0, b1 = a0, c0 = a0, c1 = a0;
#pragma unroll
            for (int i = 0; i < N4; ++i) {
                const float2 k0 = make_float2(kc[i].x, kc[i].y), k1 = make_float2(kc[i].z, kc[i].w);
                const float2 q0 = make_float2(qc[i].x, qc[i].y), q1 = make_float2(qc[i].z, qc[i].w);
                a0 = __ffma2_rn(Sr[2 * i], k0, a0); a1 = __ffma2_rn(Sr[2 * i + 1], k1, a1);
                b0 = __ffma2_rn(Sr[2 * i], q0, b0); b1 = __ffma2_rn(Sr[2 * i + 1], q1, b1);
                c0 = __ffma2_rn(k0, q0, c0); c1 = __ffma2_rn(k1, q1, c1);
            }
            float sa = (a0.x + a0.y) + (a1.x + a1.y), sb = (b0.x + b0.y) + (b1.x + b1.y), sc = (c0.x + c0.y) + (c1.x + c1.y);
#pragma unroll
            for (int off = C::CW; off < 32; off <<= 1) {
                sa += __shfl_xor_sync(0xffffffffu, sa, off);
                sb += __shfl_xor_sync(0xffffffffu, sb, off);
                sc += __shfl_xor_sync(0xffffffffu, sc, off);
            }
            const float gg = g;
            const float u = beta * (vj - gg * sa);
            const float oj = fmaf(sc, u, gg * sb);
            const float2 g2 = make_float2(gg, gg), u2 = make_float2(u, u);
#pragma unroll
            for (int i = 0; i < N4; ++i) {
                Sr[2 * i] = __ffma2_rn(make_float2(kc[i].x, kc[i].y), u2, __fmul2_rn(g2, Sr[2 * i]));
                Sr[2 * i + 1] = __ffma2_rn(make_float2(kc[i].z, kc[i].w), u2, __fmul2_rn(g2, Sr[2 * i + 1]));
            }
            if (tt + 1 < n) take(bufs[b] + (tt + 1) * C::ROW);  // the next token's, while this one's output leaves
            if (rs == 0 && col_ok) o[(size_t)(t + tt) * ldo + (size_t)h * V + col] = oj;
        }
    }
    if (col_ok) {
#pragma unroll
        for (int i = 0; i < 2 * N4; ++i) {
            if (i0 + 2 * i < D) S[(size_t)(i0 + 2 * i) * V + col] = Sr[i].x;
            if (i0 + 2 * i + 1 < D) S[(size_t)(i0 + 2 * i + 1) * V + col] = Sr[i].y;
        }
    }
}

// One token a request: what counts is the state, read and written once, and how much of it is on its way at a time.  A CTA has a
// head's whole state in registers (V / 4 threads across a row, 16 rows or fewer a thread), all of it requested before the
// token's rows arrive; the sums over a column meet in shared memory, once.  64 requests, 16 heads of 128 x 128 (134 MB
// of state read and written), B200: 81 us by delta_rule_kernel, whose threads read 4 bytes of every row they own; 26 us so
// (5.1 TB/s).  Relative 2-norm of the results against 64 bits 8.2e-8 both ways (1.0e-7 with a thread's sixteen rows in one chain, 1 us
// slower as it spilled).
constexpr int DT_THREADS = 256, DT_ROWS = 16;

template <int LANES>
__global__ void __launch_bounds__(DT_THREADS, 2)
delta_token_kernel(const float* __restrict__ qkv, long ld, int q_off, int k_off, int v_off, const float* __restrict__ gb, long ldgb,
                   float* __restrict__ state, size_t state_stride, size_t s_off, const int* __restrict__ slot_map,
                   const int* __restrict__ q_start, const int* __restrict__ positions, float* __restrict__ o, long ldo,
                   int heads, int G, int D, int longest) {
    constexpr int RG = DT_THREADS / LANES, V = 4 * LANES, ROWS = 128 / RG < DT_ROWS ? 128 / RG : DT_ROWS;
    __shared__ __align__(16) float rows[2][128];               // k, q
    __shared__ __align__(16) float sums[2][RG][V];             // S^T k and S^T q, by row groups
    static_assert((ROWS == 8 || ROWS == 16) && RG % 4 == 0, "a tree of fours");
    __shared__ float dots[RG];
    const int s = blockIdx.y, h = blockIdx.x, kvh = h / (heads / G), tid = threadIdx.x;
    const int t0 = q_start[s], t1 = q_start[s + 1];
    if (t1 <= t0 || t1 - t0 > longest) return;
    const int rg = tid / LANES, c = tid % LANES * 4;
    float* st = state + (size_t)slot_map[s] * state_stride + s_off + (size_t)h * D * V + c;
    const bool fresh = positions[t0] == 0;
    float4 S[ROWS];
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
        const int d = rg + RG * j;
        S[j] = (!fresh && d < D) ? *reinterpret_cast<const float4*>(st + (size_t)d * V) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (int t = t0; t < t1; ++t) {                 // once, unless a step of as many tokens as requests has an empty request beside a portion
        const float* row = qkv + (size_t)t * ld;
        {
            const int which = tid >> 7, d = tid & 127;
            rows[which][d] = d < D ? row[(which ? q_off : k_off) + kvh * D + d] : 0.f;
        }
        const float4 v = *reinterpret_cast<const float4*>(row + v_off + (size_t)h * V + c);
        const float g = gb[(size_t)t * ldgb + h], beta = gb[(size_t)t * ldgb + heads + h];
        __syncthreads();
        // sums of four rows, the fours in a tree, the row groups in another: short chains, whose rounding is that of the walk's
        auto four_rows = [&](const float (&x)[128], int j0) {
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int j = j0; j < j0 + 4; ++j) {
                const float k = x[rg + RG * j];
                a.x = fmaf(S[j].x, k, a.x); a.y = fmaf(S[j].y, k, a.y); a.z = fmaf(S[j].z, k, a.z); a.w = fmaf(S[j].w, k, a.w);
            }
            return a;
        };
        auto over_rows = [&](const float (&x)[128]) {
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int j = 0; j < ROWS; j += 8) {
                const float4 p = four_rows(x, j), q = four_rows(x, j + 4);
                a.x += p.x + q.x; a.y += p.y + q.y; a.z += p.z + q.z; a.w += p.w + q.w;
            }
            return a;
        };
        *reinterpret_cast<float4*>(&sums[0][rg][c]) = over_rows(rows[0]);
        *reinterpret_cast<float4*>(&sums[1][rg][c]) = over_rows(rows[1]);
        float kq = 0.f;
        if (c == 0) {
#pragma unroll
            for (int j = 0; j < ROWS; j += 4) {
                float d = 0.f;
#pragma unroll
                for (int i = j; i < j + 4; ++i) d = fmaf(rows[0][rg + RG * i], rows[1][rg + RG * i], d);
                kq += d;
            }
            dots[rg] = kq;
        }
        __syncthreads();
        auto over_groups = [&](const float (&part)[RG][V]) {
            float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int r = 0; r < RG; r += 4) {
                const float4 x = *reinterpret_cast<const float4*>(&part[r][c]), y = *reinterpret_cast<const float4*>(&part[r + 1][c]);
                const float4 z = *reinterpret_cast<const float4*>(&part[r + 2][c]), w = *reinterpret_cast<const float4*>(&part[r + 3][c]);
                t.x += (x.x + y.x) + (z.x + w.x); t.y += (x.y + y.y) + (z.y + w.y);
                t.z += (x.z + y.z) + (z.z + w.z); t.w += (x.w + y.w) + (z.w + w.w);
            }
            return t;
        };
        const float4 a = over_groups(sums[0]), b = over_groups(sums[1]);
        kq = 0.f;
#pragma unroll
        for (int r = 0; r < RG; r += 4) kq += (dots[r] + dots[r + 1]) + (dots[r + 2] + dots[r + 3]);
        const float4 u = make_float4(beta * (v.x - g * a.x), beta * (v.y - g * a.y), beta * (v.z - g * a.z), beta * (v.w - g * a.w));
        if (rg == 0) {
            float* dst = o + (size_t)t * ldo + (size_t)h * V + c;
            dst[0] = fmaf(kq, u.x, g * b.x); dst[1] = fmaf(kq, u.y, g * b.y); dst[2] = fmaf(kq, u.z, g * b.z); dst[3] = fmaf(kq, u.w, g * b.w);
        }
#pragma unroll
        for (int j = 0; j < ROWS; ++j) {
            const float k = rows[0][rg + RG * j];
            S[j].x = fmaf(k, u.x, g * S[j].x); S[j].y = fmaf(k, u.y, g * S[j].y);
            S[j].z = fmaf(k, u.z, g * S[j].z); S[j].w = fmaf(k, u.w, g * S[j].w);
        }
        if (t + 1 < t1) __syncthreads();                        // the rows are read before the next token's arrive
    }
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
        const int d = rg + RG * j;
        if (d < D) *reinterpret_cast<float4*>(st + (size_t)d * V) = S[j];
    }
}

__device__ __forceinline__ float gate_act(float z, int kind) {
    const float sg = 1.0f / (1.0f + expf(-z));
    return kind == 1 ? z * sg : sg;
}

// one warp per (token, group)
template <typename TP, typename TO>
__global__ void __launch_bounds__(256)
grouped_gated_rmsnorm_kernel(const float* __restrict__ o, long ldo, const TP* __restrict__ gate, long ldg, const void* __restrict__ w,
                             int wdt, float eps, TO* __restrict__ out, long ldout, int T, int groups, int group, int act) {
    const size_t unit = (size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (unit >= (size_t)T * groups) return;
    const int lane = threadIdx.x & 31;
    const size_t t = unit / groups;
    const int g = (int)(unit - t * groups);
    const float* row = o + t * ldo + (size_t)g * group;
    float ss = 0.f;
    for (int d = lane; d < group; d += 32) { const float v = ld_act(row + d); ss = fmaf(v, v, ss); }
    const float scale = 1.0f / sqrtf(warp_sum(ss) / (float)group + eps);
    for (int d = lane; d < group; d += 32) {
        const float z = ld_act(gate + t * ldg + (size_t)g * group + d);
        out[t * ldout + (size_t)g * group + d] = from_f<TO>(ld_act(row + d) * scale * load_dyn(w, wdt, d) * gate_act(z, act));
    }
}

// The same with four neighbouring numbers a lane, read once: groups of up to 256 numbers, multiples of 4, rows that
// four-number accesses take.  2,048 tokens, 16 groups of 128 (42 MB), B200: 21 us a number at a time, 12 so.
template <typename TP, typename TO>
__global__ void __launch_bounds__(256)
grouped_gated_rmsnorm_vec_kernel(const float* __restrict__ o, long ldo, const TP* __restrict__ gate, long ldg, const void* __restrict__ w,
                                 int wdt, float eps, TO* __restrict__ out, long ldout, int T, int groups, int group, int act) {
    const size_t unit = (size_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    griddep_launch();
    griddep_wait();
    if (unit >= (size_t)T * groups) return;
    const int lane = threadIdx.x & 31;
    const size_t t = unit / groups;
    const int c0 = (int)(unit - t * groups) * group;
    float v[2][4], z[2][4];
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int d = (lane + 32 * k) * 4;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
        if (d < group) {
            a = ld_act4(o + t * ldo + c0 + d);
            b = ld_act4(gate + t * ldg + c0 + d);
        }
        v[k][0] = a.x; v[k][1] = a.y; v[k][2] = a.z; v[k][3] = a.w;
        z[k][0] = b.x; z[k][1] = b.y; z[k][2] = b.z; z[k][3] = b.w;
#pragma unroll
        for (int e = 0; e < 4; ++e) ss = fmaf(v[k][e], v[k][e], ss);
    }
    const float scale = 1.0f / sqrtf(warp_sum(ss) / (float)group + eps);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int d = (lane + 32 * k) * 4;
        if (d >= group) break;
        float y[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) y[e] = v[k][e] * scale * load_dyn(w, wdt, d + e) * gate_act(z[k][e], act);
        store4(out + t * ldout + c0 + d, y);
    }
}

}  // namespace aien

using namespace aien;

template <int DPT, int RS>
static void launch_delta_rule(cudaStream_t stream, const float* qkv, long ld, int q_off, int k_off, int v_off, const float* gb,
                              long ldgb, float* state, size_t state_stride, size_t s_off, const int* slot_map, const int* q_start,
                              const int* positions, float* o, long ldo, int S, int heads, int G, int D, int V, int longest) {
    constexpr int COLS = DeltaCfg<DPT, RS>::COLS;
    dim3 grid((V + COLS - 1) / COLS, heads, S);
    delta_rule_kernel<DPT, RS><<<grid, DR_THREADS, 0, stream>>>(qkv, ld, q_off, k_off, v_off, gb, ldgb, state, state_stride, s_off,
                                                                slot_map, q_start, positions, o, ldo, heads, G, D, V, longest);
}

// qkv float32 [T, ld]: prepared q (G*D) at q_off, k (G*D) at k_off, v (heads*V) at v_off; gb float32 [T, ldgb]: decay
// of head h at column h, beta at heads + h.  state: float32 rows of state_stride numbers per slot, S [heads][D][V] at
// s_off.  T: the step's tokens.  Request s of the step (tokens q_start[s] .. q_start[s+1]) continues from slot slot_map[s].  o float32 [T, ldo].
// longest > 0: requests that bring more tokens are served elsewhere and left alone here.
AIEN_API int aien_delta_rule(const float* qkv, long ld, int q_off, int k_off, int v_off, const float* gb, long ldgb, float* state,
                             size_t state_stride, size_t s_off, const int* slot_map, const int* q_start, const int* positions,
                             float* o, long ldo, int T, int S, int heads, int G, int D, int V, int longest, cudaStream_t stream) {
    if (S <= 0) return 0;
    if (longest <= 0) longest = 0x7fffffff;
    if (heads <= 0 || G <= 0 || heads % G || D <= 0 || D > 256 || V <= 0 || S > 65535 || heads > 65535) return AIEN_E_SHAPE;
    // single tokens, and states whose rows are 64 or 128 columns and start on 16-byte boundaries (D <= 128: a thread's share fits its registers)
    if ((T == S || longest == 1) && (V == 128 || V == 64) && D <= 128 && ((ld | v_off) & 3) == 0 && ((state_stride | s_off) & 3) == 0 &&
        ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(state)) & 15) == 0) {
        const auto kern = V == 128 ? delta_token_kernel<32> : delta_token_kernel<16>;
        kern<<<dim3(heads, S), DT_THREADS, 0, stream>>>(qkv, ld, q_off, k_off, v_off, gb, ldgb, state, state_stride, s_off, slot_map, q_start, positions,
                                                        o, ldo, heads, G, D, longest);
        return launch_status();
    }
#define DR_CASE(N, R) launch_delta_rule<N, R>(stream, qkv, ld, q_off, k_off, v_off, gb, ldgb, state, state_stride, s_off, slot_map, q_start, positions, o, ldo, S, heads, G, D, V, longest)
    if (D <= 16) DR_CASE(4, 4);
    else if (D <= 32) DR_CASE(8, 4);
    else if (D <= 64) DR_CASE(8, 8);
    else if (D <= 96) DR_CASE(12, 8);
    else if (D <= 128) DR_CASE(16, 8);
    else if (D <= 192) DR_CASE(24, 8);
    else DR_CASE(32, 8);
#undef DR_CASE
    return launch_status();
}

// o float32 [T, groups*group]; gate [T, *] in g_dt; w [group]; act 0: sigmoid(gate), 1: silu(gate).
AIEN_API int aien_grouped_gated_rmsnorm(const float* o, long ldo, const void* gate, int g_dt, long ldg, const void* w, int w_dt, float eps,
                                        void* out, int o_dt, long ldout, int T, int groups, int group, int act, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (groups <= 0 || group <= 0) return AIEN_E_SHAPE;
    const size_t units = (size_t)T * groups;
    const unsigned blocks = (unsigned)((units + 7) / 8);
    const bool four = group % 4 == 0 && group <= 256 && ((ldo | ldg | ldout) & 3) == 0 && (reinterpret_cast<uintptr_t>(o) & 15) == 0 &&
                      reinterpret_cast<uintptr_t>(gate) % (g_dt == AIEN_DT_F32 ? 16 : 8) == 0 && reinterpret_cast<uintptr_t>(out) % (o_dt == AIEN_DT_F32 ? 16 : 8) == 0;
    if (four) {
        AIEN_DISPATCH_DTYPE(g_dt, TP, AIEN_DISPATCH_DTYPE(o_dt, TO,
            (launch_chain(grouped_gated_rmsnorm_vec_kernel<TP, TO>, dim3(blocks), dim3(256), (size_t)0, stream, o, ldo, (const TP*)gate, ldg, w, w_dt, eps, (TO*)out,
                          ldout, T, groups, group, act))));
        return launch_status();
    }
    AIEN_DISPATCH_DTYPE(g_dt, TP, AIEN_DISPATCH_DTYPE(o_dt, TO,
        (grouped_gated_rmsnorm_kernel<TP, TO><<<blocks, 256, 0, stream>>>(o, ldo, (const TP*)gate, ldg, w, w_dt, eps, (TO*)out, ldout, T,
                                                                         groups, group, act))));
    return launch_status();
}
