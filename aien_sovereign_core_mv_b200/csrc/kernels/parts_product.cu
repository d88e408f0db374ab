// out = x W^T for float32 rows x and a bfloat16 matrix W with the rounding of float32 multiply-adds, on the tensor cores.
//
// x comes as the sum of three bfloat16 rows (split_rows, up to 2^-25 of it): x W^T = p0 W^T + p1 W^T + p2 W^T, every product
// exact.  What is left is how they are added.  The tensor cores cut the sum of 16 products off at 24 bits and never round up, so
// a long accumulation in them loses in one direction: over K = 128 in a tcgen05 accumulator the result is off by 6.6e-7 (K = 256:
// 1.3e-6), by 0.9e-7 with float32 multiply-adds.  So every 16 products of p0 start from zero and are added outside, by
// float32 additions; the products of p1 and p2 are 2^-8 and less of them and stay in accumulators of their own.  tcgen05
// would have to pass every such piece through tensor memory; mma.sync leaves it in registers.
//
// A CTA makes 128 x 64 results, its eight warps 32 x 32 each, in steps of 32 columns of K through three stages of shared
// memory; 128 registers and 105 KB, so two CTAs an SM take turns at waiting.  What bounds it is the rate of mma.sync and the
// additions beside it.  Relative error and time on a B200, in brackets of multiply-adds on the CUDA cores and of a tcgen05
// accumulator: 2,048 x 4,096 x 128 0.62e-7, 31 us (0.93e-7, 101 us; 6.6e-7, 12 us); 2,048 x 8,192 x 256 0.80e-7, 107 us
// (1.07e-7, 381 us; 12.8e-7, 31 us); one row of 4,096 x 128 6.3 us (10.4; 6.3).
#include "common.cuh"

namespace aien {

constexpr int PP_BM = 128, PP_BN = 64, PP_BK = 32, PP_STAGES = 3, PP_THREADS = 256;
constexpr int PP_LD = PP_BK + 8;                                          // numbers between rows: eight rows' 16 bytes meet no bank twice
constexpr int PP_STAGE = (3 * PP_BM + PP_BN) * PP_LD;                     // p0 | p1 | p2 | W

__device__ __forceinline__ void pp_ldmatrix(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}

__device__ __forceinline__ void pp_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__global__ void __launch_bounds__(PP_THREADS, 2)
parts_product_kernel(const __nv_bfloat16* __restrict__ parts, const __nv_bfloat16* __restrict__ W, long ldw, float* __restrict__ out, long ldo,
                     int M, int N, int K, int pairs) {
    extern __shared__ __align__(16) __nv_bfloat16 pp_smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, wm = (warp & 3) * 32, wn = (warp >> 2) * 32;
    const int m0 = blockIdx.y * PP_BM, n0 = blockIdx.x * PP_BN, steps = (K + PP_BK - 1) / PP_BK;
    const uint32_t smem = (uint32_t)__cvta_generic_to_shared(pp_smem);
    griddep_launch();
    // K is a multiple of 8, so a piece of 8 numbers lies inside or outside whole
    auto fetch = [&](int step) {
        if (step < steps) {
            const uint32_t stage = smem + (uint32_t)(step % PP_STAGES * PP_STAGE) * 2;
#pragma unroll
            for (int i = tid; i < (3 * PP_BM + PP_BN) * (PP_BK / 8); i += PP_THREADS) {
                const int r = i / (PP_BK / 8), c = i % (PP_BK / 8) * 8, k = step * PP_BK + c;
                const bool a = r < 3 * PP_BM;
                const int row = a ? m0 + r % PP_BM : n0 + r - 3 * PP_BM;
                const bool in = k < K && row < (a ? M : N);
                const __nv_bfloat16* src = !in ? W : a ? parts + ((size_t)row * 3 + r / PP_BM) * K + k : W + row * ldw + k;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(stage + (uint32_t)(r * PP_LD + c) * 2), "l"(src), "r"(in ? 16 : 0) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float acc[2][4][4] = {}, low[2][4][4] = {};
    fetch(0);
    fetch(1);
    for (int step = 0; step < steps; ++step) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                                                 // this step's rows are here, and everyone has left the stage two steps on
        fetch(step + 2);
        const uint32_t stage = smem + (uint32_t)(step % PP_STAGES * PP_STAGE) * 2;
#pragma unroll
        for (int k0 = 0; k0 < PP_BK; k0 += 16) {
            uint32_t b[2][4];                                            // 16 columns each: of the first 8 k 0..7, k 8..15, of the others likewise
#pragma unroll
            for (int j = 0; j < 2; ++j)
                pp_ldmatrix(b[j], stage + (uint32_t)((3 * PP_BM + wn + j * 16 + (lane >> 4) * 8 + (lane & 7)) * PP_LD + k0 + ((lane >> 3) & 1) * 8) * 2);
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) {
                uint32_t a[3][4];
#pragma unroll
                for (int p = 0; p < 3; ++p)
                    pp_ldmatrix(a[p], stage + (uint32_t)((p * PP_BM + wm + mt * 16 + (lane & 15)) * PP_LD + k0 + (lane >> 4) * 8) * 2);
#pragma unroll
                for (int nt = 0; nt < 4; ++nt) {
                    const uint32_t b0 = b[nt >> 1][(nt & 1) * 2], b1 = b[nt >> 1][(nt & 1) * 2 + 1];
                    float c[4] = {0.f, 0.f, 0.f, 0.f};
                    pp_mma(c, a[0], b0, b1);
                    pp_mma(low[mt][nt], a[2], b0, b1);
                    pp_mma(low[mt][nt], a[1], b0, b1);
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[mt][nt][e] += c[e];
                }
            }
        }
    }
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int row = m0 + wm + mt * 16 + half * 8 + (lane >> 2);
            if (row >= M) continue;
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                const int col = n0 + wn + nt * 8 + (lane & 3) * 2;
                const float2 v = make_float2(acc[mt][nt][2 * half] + low[mt][nt][2 * half], acc[mt][nt][2 * half + 1] + low[mt][nt][2 * half + 1]);
                float* o = out + row * ldo + col;
                if (pairs && col < N) {
                    *reinterpret_cast<float2*>(o) = v;
                } else {
                    if (col < N) o[0] = v.x;
                    if (col + 1 < N) o[1] = v.y;
                }
            }
        }
}

}  // namespace aien

using namespace aien;

// parts bfloat16 [M, 3 K], the three parts of a row side by side (aien_split_rows); W bfloat16 [N, K] (row stride ldw); out
// float32 [M, N] (row stride ldo).  K and ldw are multiples of 8, parts and W start on 16-byte boundaries.
AIEN_API int aien_parts_product(const void* parts, const void* W, long ldw, float* out, long ldo, int M, int N, int K, cudaStream_t stream) {
    if (M <= 0) return 0;
    if (N <= 0 || K <= 0 || (K & 7) || (M + PP_BM - 1) / PP_BM > 65535) return AIEN_E_SHAPE;
    if ((ldw & 7) || ((reinterpret_cast<uintptr_t>(parts) | reinterpret_cast<uintptr_t>(W)) & 15)) return AIEN_E_ALIGN;
    constexpr int bytes = PP_STAGES * PP_STAGE * 2;
    if (cudaFuncSetAttribute(parts_product_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return AIEN_E_STATE;
    const int pairs = ((ldo | N) & 1) == 0 && (reinterpret_cast<uintptr_t>(out) & 7) == 0;
    parts_product_kernel<<<dim3((N + PP_BN - 1) / PP_BN, (M + PP_BM - 1) / PP_BM), PP_THREADS, bytes, stream>>>(      // plain: see griddep_wait
        (const __nv_bfloat16*)parts, (const __nv_bfloat16*)W, ldw, out, ldo, M, N, K, pairs);
    return launch_status();
}
