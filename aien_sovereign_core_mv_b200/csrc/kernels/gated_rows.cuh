// A row (or one of its equal parts) normed and gated, four neighbouring numbers a thread: the row is read once and waits
// in registers for its root mean square.  The plain kernels of the three forms read it twice, a number at a time, and are
// bound by the number of their loads; these are bound by the bytes.
//   GATE_FIRST   v = o * silu(gate);  out = v / rms(v) * w * mult
//   otherwise    out = o / rms(o) * w * sigmoid(gate) * mult
// 2,000 rows of 2,048, B200 (41 MB): 17 and 20 us a number at a time, 9.3 us so.
#pragma once
#include "common.cuh"

namespace aien {

constexpr int GATED_ROWS_THREADS = 256, GATED_ROWS_MAX = 4096;

__device__ __forceinline__ void store4(float* p, const float (&v)[4]) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void store4(__nv_bfloat16* p, const float (&v)[4]) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}

// NV: groups of four numbers a thread holds (a part has at most 1,024 NV numbers); grid (rows, parts)
template <int NV, bool GATE_FIRST, typename TG, typename TO>
__global__ void __launch_bounds__(GATED_ROWS_THREADS)
gated_rows_kernel(const float* __restrict__ o, long ldo, const TG* __restrict__ gate, long ldg, const void* __restrict__ w, int wdt, float eps,
                  float mult, TO* __restrict__ out, long ldout, int part) {
    __shared__ float red[32];
    griddep_launch();
    griddep_wait();
    const size_t t = blockIdx.x;
    const int c0 = blockIdx.y * part;
    float v[NV][4], g[NV][4];
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int i = (threadIdx.x + k * GATED_ROWS_THREADS) * 4;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), z = a;
        if (i < part) {
            a = ld_act4(o + t * ldo + c0 + i);
            z = ld_act4(gate + t * ldg + c0 + i);
        }
        v[k][0] = a.x; v[k][1] = a.y; v[k][2] = a.z; v[k][3] = a.w;
        g[k][0] = z.x; g[k][1] = z.y; g[k][2] = z.z; g[k][3] = z.w;
    }
#pragma unroll
    for (int k = 0; k < NV; ++k)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            g[k][e] = (GATE_FIRST ? g[k][e] : 1.0f) / (1.0f + expf(-g[k][e]));
            if (GATE_FIRST) v[k][e] *= g[k][e];
            ss = fmaf(v[k][e], v[k][e], ss);
        }
    const float r = mult / sqrtf(block_sum(ss, red) / (float)part + eps);
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int i = (threadIdx.x + k * GATED_ROWS_THREADS) * 4;
        if (i >= part) break;
        float y[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) y[e] = v[k][e] * r * load_dyn(w, wdt, c0 + i + e) * (GATE_FIRST ? 1.0f : g[k][e]);
        store4(out + t * ldout + c0 + i, y);
    }
}

// Whether rows of `part` numbers start on boundaries that four-number accesses take.
template <typename TG, typename TO>
inline bool gated_rows_take(const float* o, long ldo, const TG* gate, long ldg, const TO* out, long ldout, int part) {
    return part % 4 == 0 && part >= 256 && part <= GATED_ROWS_MAX && ((ldo | ldg | ldout) & 3) == 0 && (reinterpret_cast<uintptr_t>(o) & 15) == 0 &&
           reinterpret_cast<uintptr_t>(gate) % (4 * sizeof(TG)) == 0 && reinterpret_cast<uintptr_t>(out) % (4 * sizeof(TO)) == 0;
}

template <bool GATE_FIRST, typename TG, typename TO>
inline void launch_gated_rows(const float* o, long ldo, const TG* gate, long ldg, const void* w, int wdt, float eps, float mult, TO* out, long ldout,
                              int rows, int parts, int part, cudaStream_t stream) {
    const dim3 grid(rows, parts);
    const auto kern = part <= 1024 ? gated_rows_kernel<1, GATE_FIRST, TG, TO> : part <= 2048 ? gated_rows_kernel<2, GATE_FIRST, TG, TO>
                                                                                             : gated_rows_kernel<4, GATE_FIRST, TG, TO>;
    launch_chain(kern, grid, dim3(GATED_ROWS_THREADS), (size_t)0, stream, o, ldo, gate, ldg, w, wdt, eps, mult, out, ldout, part);
}

}  // namespace aien
