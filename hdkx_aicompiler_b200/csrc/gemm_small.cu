// Dense layers of a few hundred tiles ([M,K] x [N,K]^T + c, a classifier's head) in one launch on the CUDA cores, with the operands
// rounded as the tensor-core path rounds them.
//
// The tensor-core path converts both operands into a workspace, builds two tensor maps and launches two kernels, the second of which is
// a chain of latencies at this size: 32 x 1000 x 512 in tf32 takes 2.2 + 7.0 us on the device and 9 of the host, this kernel 6.5
// and 3.6. Products of tf32 (or bf16) values are exact in fp32, so every term is added with one rounding.
//
// What bounds it: one way to memory and back per pass, then the shared-memory loads of a lane's 4 x 4 outputs (eight per 64 FMA). A
// block loads its 48 rows (up to 512 k at a time, every load in flight at once), rounds them on the way into shared memory, its
// eight warps take a 64-wide part of k each (four k per shared-memory load) and the parts are added in warp order.
#include "common.cuh"
#include "conv_common.cuh"
#include "sm100.cuh"
#include "tf32.cuh"

#include <cuda_bf16.h>

namespace kxc_b200 {
namespace {

constexpr int kThreads = 256, kWarps = kThreads / 32;
constexpr int kTM = 32, kTN = 16, kTK = 512;   // tile, and the k of one pass
constexpr int kPitch = kTK + 4;                // floats: eight rows of 16 bytes fall on all banks
constexpr int kRowsPerWarp = (kTM + kTN) / kWarps;
constexpr int kVecs = kTK / 128;               // 16-byte loads of a lane per row
constexpr int kSmemBytes = (kTM + kTN) * kPitch * 4;
static_assert(kWarps * kTM * kTN <= (kTM + kTN) * kPitch, "the parts reuse the operands' memory");

template <bool kBF16>
__device__ __forceinline__ float round_operand(float x) {
    if constexpr (kBF16) return __bfloat162float(__float2bfloat16_rn(x));
    else return tf32_rne(x);
}

// kBlocks: resident per SM, what the rule below counts on. (128 registers, tf32 with or without the bound; bf16 takes 161 for one block,
// which is faster while there is a tile per SM, 32x2016x512 6.0 / 6.3 us and 32x2016x1024 10.4 / 11.2, but would be two waves beyond that,
// 128x1000x512 11.1 / 9.2.)
template <bool kBF16, int kBlocks>
__global__ void __launch_bounds__(kThreads, kBlocks) gemm_small_kernel(const float* __restrict__ a, const float* __restrict__ b, const float* __restrict__ c,
                                                              float* __restrict__ out, int M, int N, int K, int vec) {
    extern __shared__ __align__(16) float rows[];  // kTM rows of a, then kTN rows of b
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.y * kTM, n0 = blockIdx.x * kTN;
    const int lr = lane & 7, lc = lane >> 3;  // outputs (lr + 8 i, lc + 4 j)
    float acc[4][4] = {};
    sm100::pdl_wait();
    for (int k0 = 0; k0 < K; k0 += kTK) {
        float4 v[kRowsPerWarp][kVecs];
#pragma unroll
        for (int r = 0; r < kRowsPerWarp; ++r) {
            const int row = warp * kRowsPerWarp + r;
            const bool from_a = row < kTM;
            const int index = from_a ? m0 + row : n0 + row - kTM;
            const bool there = index < (from_a ? M : N);
            const float* src = (from_a ? a : b) + (int64_t)(there ? index : 0) * K;
#pragma unroll
            for (int q = 0; q < kVecs; ++q) {
                const int k = k0 + 4 * lane + 128 * q;
                v[r][q] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (!there) continue;
                if (vec) {  // (K is a multiple of four)
                    if (k < K) v[r][q] = __ldg(reinterpret_cast<const float4*>(src + k));
                } else {
                    if (k < K) v[r][q].x = __ldg(src + k);
                    if (k + 1 < K) v[r][q].y = __ldg(src + k + 1);
                    if (k + 2 < K) v[r][q].z = __ldg(src + k + 2);
                    if (k + 3 < K) v[r][q].w = __ldg(src + k + 3);
                }
            }
        }
        if (k0 > 0) __syncthreads();  // the previous pass has been read
#pragma unroll
        for (int r = 0; r < kRowsPerWarp; ++r)
#pragma unroll
            for (int q = 0; q < kVecs; ++q) {
                const float4 x = v[r][q];
                *reinterpret_cast<float4*>(rows + (warp * kRowsPerWarp + r) * kPitch + 4 * lane + 128 * q) =
                    make_float4(round_operand<kBF16>(x.x), round_operand<kBF16>(x.y), round_operand<kBF16>(x.z), round_operand<kBF16>(x.w));
            }
        __syncthreads();
        const int left = K - k0 - warp * (kTK / kWarps);  // of this warp's part
        const int steps = left >= kTK / kWarps ? kTK / kWarps / 4 : (left + 3) / 4;
        const float* pa = rows + lr * kPitch + warp * (kTK / kWarps);
        const float* pb = rows + (kTM + lc) * kPitch + warp * (kTK / kWarps);
#pragma unroll 4
        for (int s = 0; s < steps; ++s) {
            float4 x[4], y[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                x[i] = *reinterpret_cast<const float4*>(pa + i * 8 * kPitch + 4 * s);
                y[i] = *reinterpret_cast<const float4*>(pb + i * 4 * kPitch + 4 * s);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[i][j] = fmaf(x[i].x, y[j].x, acc[i][j]);
                    acc[i][j] = fmaf(x[i].y, y[j].y, acc[i][j]);
                    acc[i][j] = fmaf(x[i].z, y[j].z, acc[i][j]);
                    acc[i][j] = fmaf(x[i].w, y[j].w, acc[i][j]);
                }
        }
    }
    __syncthreads();
    float* parts = rows;  // [warp][row][column]
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) parts[(warp * kTM + lr + 8 * i) * kTN + lc + 4 * j] = acc[i][j];
    __syncthreads();
#pragma unroll
    for (int o = threadIdx.x; o < kTM * kTN; o += kThreads) {
        const int m = m0 + o / kTN, n = n0 + o % kTN;
        if (m >= M || n >= N) continue;
        float sum = parts[o];
#pragma unroll
        for (int w = 1; w < kWarps; ++w) sum = __fadd_rn(sum, parts[w * kTM * kTN + o]);
        if (c != nullptr) sum = __fadd_rn(sum, __ldg(c + n));
        out[(int64_t)m * N + n] = sum;
    }
}

}  // namespace

// While all tiles are resident at once, two blocks per SM for one pass over k and one for two: then a call of the operator, which is
// bound by its host side, always gains. On the device alone, in a captured graph or behind a full queue, it gains with one pass and a
// tile per SM and trades otherwise. us, a call / its device time, other path : this one:
//                    tf32                          bf16
//   32x1008x512      13.5 / 9.1 : 8.2 / 6.1        12.9 / 8.1 : 8.5 / 5.9
//   128x1000x512     13.6 / 10.3 : 9.8 / 9.4       12.9 / 9.0 : 9.6 / 9.2
//   32x3200x64       12.5 / 5.9 : 8.2 / 7.2        12.9 / 5.5 : 8.4 / 6.7
//   32x1008x640      13.5 / 9.3 : 9.8 / 9.5        12.7 / 8.8 : 9.3 / 9.0
//   32x1008x1024     14.0 / 10.6 : 10.9 / 10.7     14.0 / 9.4 : 10.5 / 10.3
//   32x128x1024      13.1 / 8.6 : 10.7 / 10.6      13.5 / 7.9 : 10.3 / 10.2
//   32x2016x1024     16.5 / 12.8 : 11.1 / 10.8     13.9 / 11.1 : 10.6 / 10.4
//   128x1000x1024, beyond the line: 11.5 : 17.4 on the device
// A result that overlaps an operand needs the other path, which has read both (into its workspace) before it stores anything.
bool gemm_small_applicable(const float* a, const float* b, const float* out, const kxc_b200_gemm_desc& g) {
    auto overlaps = [&](const float* x, int64_t rows) {
        const auto o = reinterpret_cast<uintptr_t>(out), q = reinterpret_cast<uintptr_t>(x);
        return o < q + (uintptr_t)rows * g.k * 4 && q < o + (uintptr_t)g.m * g.n * 4;
    };
    if (overlaps(a, g.m) || overlaps(b, g.n)) return false;
    if (!g.transB || g.k > 2 * kTK || (g.precision != KXC_B200_PREC_TF32 && g.precision != KXC_B200_PREC_BF16)) return false;
    const int64_t tiles = ((int64_t)g.m + kTM - 1) / kTM * (((int64_t)g.n + kTN - 1) / kTN);
    return tiles <= (g.k > kTK ? 1 : 2) * kNumSMs;
}

int32_t gemm_small(const float* a, const float* b, const float* c, float* out, const kxc_b200_gemm_desc& g, cudaStream_t s) {
    const int vec = (g.k & 3) == 0 && aligned16(a) && aligned16(b) ? 1 : 0;
    const dim3 grid((unsigned)((g.n + kTN - 1) / kTN), (unsigned)((g.m + kTM - 1) / kTM));
    auto go = [&](auto kernel, PerDeviceOnce& once) -> int32_t {
        KXC_TRY(smem_opt_in(once, kernel, kSmemBytes));
        KXC_CUDA_TRY(launch_kernel(kernel, grid, dim3(kThreads), kSmemBytes, s, /*pdl=*/true, 1, a, b, c, out, g.m, g.n, g.k, vec));
        return check_launch("gemm_small");
    };
    static PerDeviceOnce once_bf16, once_bf16_two, once_tf32;
    if (g.precision != KXC_B200_PREC_BF16) return go(gemm_small_kernel<false, 2>, once_tf32);
    return (int64_t)grid.x * grid.y <= kNumSMs ? go(gemm_small_kernel<true, 1>, once_bf16) : go(gemm_small_kernel<true, 2>, once_bf16_two);
}

}  // namespace kxc_b200
