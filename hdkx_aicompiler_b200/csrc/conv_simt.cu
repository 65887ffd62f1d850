// CUDA-core (SIMT) contraction kernels in the reference's own operation order.
//
// These are the KXC_B200_PREC_FP32 mode of nn_conv2d / nn_gemm and the integer-exact form of the
// int8 convolution. Each output element is one thread's sequential reduction
//   acc = 0; for rc, rh, rw: acc = acc + (inb ? x : 0) * w          include/te/topi/nn.h:107-158
// with separately rounded multiply and add (__fmul_rn/__fadd_rn are never contracted into FMA), so
// fp32 results are bit-identical to the reference's CPU lowering. They also serve shapes the
// tensor-core path does not take (dilation, channel counts that do not fill a K block).
#include "common.cuh"
#include "sm100.cuh"
#include "conv_common.cuh"

#include <type_traits>

namespace kxc_b200 {
namespace {

constexpr int kThreads = 128;

template <typename TIn, typename TAcc>
__device__ __forceinline__ TAcc mac_exact(TAcc acc, TIn x, TIn w);
template <>
__device__ __forceinline__ float mac_exact<float, float>(float acc, float x, float w) {
    return __fadd_rn(acc, __fmul_rn(x, w));
}
template <>
__device__ __forceinline__ int32_t mac_exact<int8_t, int32_t>(int32_t acc, int8_t x, int8_t w) {
    return acc + (int32_t)x * (int32_t)w;
}

// One thread per output element, ow fastest so a warp reads contiguous input columns; the weight
// address is warp-uniform for most warps (broadcast load).
template <typename TIn, typename TAcc, typename Epilogue>
__global__ void __launch_bounds__(kThreads) conv2d_direct_kernel(const TIn* __restrict__ data,
                                                                 const TIn* __restrict__ weight, ConvDims d,
                                                                 Epilogue epi) {
    sm100::pdl_wait();
    const int64_t total = (int64_t)d.N * d.O * d.OH * d.OW;
    for (int64_t lin = (int64_t)blockIdx.x * kThreads + threadIdx.x; lin < total; lin += (int64_t)gridDim.x * kThreads) {
        const int ow = (int)(lin % d.OW);
        int64_t t = lin / d.OW;
        const int oh = (int)(t % d.OH);
        t /= d.OH;
        const int o = (int)(t % d.O);
        const int n = (int)(t / d.O);
        const TIn* xn = data + (int64_t)n * d.C * d.H * d.W;
        const TIn* wo = weight + (int64_t)o * d.C * d.KH * d.KW;
        TAcc acc = 0;
        for (int rc = 0; rc < d.C; ++rc) {
            const TIn* xc = xn + (int64_t)rc * d.H * d.W;
            const TIn* wc = wo + rc * d.KH * d.KW;
            for (int rh = 0; rh < d.KH; ++rh) {
                const int ih = oh * d.SH + rh * d.DH - d.PH;
                const bool inb_h = (ih >= 0) && (ih < d.H);
                for (int rw = 0; rw < d.KW; ++rw) {
                    const int iw = ow * d.SW + rw * d.DW - d.PW;
                    const bool inb = inb_h && (iw >= 0) && (iw < d.W);
                    const TIn xv = inb ? __ldg(xc + (int64_t)ih * d.W + iw) : (TIn)0;
                    acc = mac_exact<TIn, TAcc>(acc, xv, __ldg(wc + rh * d.KW + rw));
                }
            }
        }
        epi(acc, lin, o);
    }
}

// Register-tiled fp32 form of the same reduction, on packed pairs. A block computes kTO*kOG output channels x kTP*kPG
// consecutive output pixels (flattened over n, oh, ow), a thread kTO x kTP of them. Every output element is still ONE
// sequential chain acc = acc + x * w over rc, rh, rw with separately rounded multiply and add, so the bits are those of the
// one-thread-per-output kernel above.
//
// What bounds it: the FMA pipe. Two roundings per term are two instructions, and a scalar multiply + add pair reaches only
// 88 of the 128 lanes per clock of an SM (three register operands each, in a pure register loop); the packed f32x2 forms
// reach 125, i.e. 62.5 terms per clock and SM = 36.4 TFLOP/s at 1.965 GHz, and leave half of the issue slots to the loads.
// ptxas fuses mul.rn.f32x2 + add.rn.f32x2 into one fused multiply-add, which rounds once and changes the bits. The product
// is therefore formed as fma(x, w, -0) with a -0 that is a kernel argument (fma(x, w, -0) is the rounded product for every
// x and w, the signs of zeros included), which nothing can fold.
// Measured, 128 -> 128 channels 3x3 at 28x28 and 32 images: 646 us with scalar arithmetic, 275 us = 26.9 TFLOP/s now, 0.74 of
// the packed bound at 1.965 GHz. ncu: the pipe is busy for 97 % of the clocks on the SMs that work throughout and 85 % on average, as
// there are 2.65 blocks for each SM, two of them at a time, at 1.89 GHz. ResNet-18 at 32 images 11.3 -> 4.4 ms. Weights doubled in shared
// memory or channels and pixels paired crosswise to spare the register moves, unrolling two stages and rolling the k loop up gained nothing.
//
// Half of the warps compute, the other half feed them: the im2col values of KC consecutive k = (rc, rh, rw) by 4-byte
// cp.async (zeros outside the image and past the last k: acc + 0 is the identity, acc is never -0) and the weights, into a ring of
// shared-memory stages handed over with named barriers. Filters of width 3 and 7 copy their weights in the same way and keep
// the copies of kBufs - 2 stages in flight: small tiles alone on their SM were bound by one stage's way from L2
// (512 -> 512 3x3 at 7x7, one image: 55 us, 51 with them, 37 on 16x16 tiles). The others, whose K is
// short, take them through registers a stage ahead (4-byte copies there: 10 to 25 % slower). With the same warps doing both, the
// gather's dependent address arithmetic held up the FMA pipe (175 clocks per k where the arithmetic alone takes 140 with
// one warp on a scheduler); as separate warps it runs in the issue slots that the packed instructions leave. A stage is
// whole filter rows (four of 3 taps, two of 7, sixteen of 1), so that a row's pointer and bounds are found once and a tap
// costs a bit test and the copy; other widths find every tap in a table.
constexpr int kExactMaxTaps = 64; // the table's size

__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ uint64_t mac2_exact(uint64_t acc, uint64_t x, uint64_t w, uint64_t neg_zero) {
    uint64_t prod, sum;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(prod) : "l"(x), "l"(w), "l"(neg_zero));
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(sum) : "l"(acc), "l"(prod));
    return sum;
}
// 4 bytes to shared memory: the value at src, or zero where !valid (src is not read then); nothing where !active
__device__ __forceinline__ void cp_async4_zfill(uint32_t dst, const float* src, uint32_t valid, bool active) {
    asm volatile(
        "{\n\t.reg .pred ignore, act;\n\tsetp.eq.u32 ignore, %2, 0;\n\tsetp.ne.u32 act, %3, 0;\n\t"
        "@act cp.async.ca.shared.global [%0], [%1], 4, ignore;\n\t}" ::"r"(dst), "l"(src), "r"(valid), "r"((uint32_t)active));
}

__device__ __forceinline__ void named_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void named_arrive(int id, int threads) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

template <int kTO, int kTP, int kOG, int kPG>
struct ExactTile {
    static constexpr int kThreads = kOG * kPG;  // of each role
    static constexpr int kO = kTO * kOG;
    static constexpr int kP = kTP * kPG;
};

// kKW: the filter width at compile time (1, 3, 7; horizontal dilation 1), 0 = any
template <int kKW, int kMul>
struct ExactStage {
    static constexpr int kRows = kMul * (kKW == 7 ? 2 : kKW == 3 ? 4 : 16);  // filter rows of a stage (kKW = 0: taps)
    static constexpr int kK = kRows * (kKW > 0 ? kKW : 1);
    // a warp copies the weights of kWK consecutive k of 32 / kWK channels: 8 to 32 bytes in a row on the global side, and rows
    // of the stage that are 32 / kWK words longer than its channels spread them over all banks
    static constexpr bool kAsync = kKW >= 3;
    static constexpr int kWK = kK % 8 == 0 ? 8 : kK % 4 == 0 ? 4 : 2;
    static constexpr int kWO = kAsync ? 32 / kWK : 0;
    static constexpr int kVec = kK % 4 == 0 ? 4 : 2;  // through registers: weights of one global load
};

template <int kKW, int kTO, int kTP, int kOG, int kPG, int kMul, int kDeep>
struct ExactSmem {
    using Tile = ExactTile<kTO, kTP, kOG, kPG>;
    using Stage = ExactStage<kKW, kMul>;
    static constexpr int kBufs = Stage::kAsync ? kDeep : 3;
    static constexpr int kWPitch = Tile::kO + Stage::kWO;
    static constexpr int kXs = Stage::kK * Tile::kP, kWs = Stage::kK * kWPitch;  // words of a buffer
    static constexpr int kBytes = kBufs * (kXs + kWs) * 4;
};

// Blocks of an SM: as the cost tables were measured. The small tiles of kExactCosts have four (the 32x64 tile would take 72 registers for
// 1x1 and 76 for any width without the bound, and three would be resident: 64 -> 128 channels 3x5 at 14x14, 16 images 58.2 / 56.5 us with
// four, 32 -> 64 5x5 at 28x28, 4 images 28.7 / 27.3).
template <int kKW, int kTO, int kTP, int kOG, int kPG, int kMul, int kDeep, typename Epilogue>
__global__ void __launch_bounds__(2 * kOG * kPG, !ExactStage<kKW, kMul>::kAsync && kTO * kTP <= 16 ? 4 : 2)
    conv2d_tiled_f32_kernel(const float* __restrict__ data, const float* __restrict__ weight, ConvDims d, float neg_zero_arg,
                            Epilogue epi) {
    sm100::pdl_wait();
    using Tile = ExactTile<kTO, kTP, kOG, kPG>;
    using Stage = ExactStage<kKW, kMul>;
    using Smem = ExactSmem<kKW, kTO, kTP, kOG, kPG, kMul, kDeep>;
    constexpr int kBufs = Smem::kBufs, kVec = Stage::kVec;
    constexpr int kT = Tile::kThreads, kTileO = Tile::kO, kTileP = Tile::kP, KC = Stage::kK, kWPitch = Smem::kWPitch;
    constexpr int kLag = kBufs - 2;  // stages whose copies are in flight behind the one that is handed over
    // threads that share the gather of one pixel, and the filter rows each takes of a stage
    constexpr int kShare = kT / kTileP > 1 ? kT / kTileP : 1;
    constexpr int kSub = kShare < Stage::kRows ? kShare : Stage::kRows;
    constexpr int kRowsPer = Stage::kRows / kSub;
    constexpr int kWLoads = kTileO * KC / (Stage::kAsync ? 1 : kVec);  // weight copies (loads) of a stage
    constexpr int kWPer = (kWLoads + kT - 1) / kT;
    static_assert(kTO % 2 == 0 && kTP % 2 == 0 && kTileP <= kT && Stage::kRows % kSub == 0 && kTileO % 8 == 0, "tile shape");
    static_assert(kBufs >= 3 && 2 * kBufs < 16, "ring: two named barriers a buffer");
    extern __shared__ __align__(16) float exact_smem[];
    float* const xs = exact_smem;                     // [kBufs][KC][kTileP]
    float* const ws = exact_smem + kBufs * Smem::kXs;  // [kBufs][KC][kWPitch]
    __shared__ int tap_off[kKW > 0 ? 1 : kExactMaxTaps];

    const int K = d.C * d.KH * d.KW;
    const int stages = (K + KC - 1) / KC;
    const int plane_in = d.H * d.W, plane_out = d.OH * d.OW;
    const int64_t P = (int64_t)d.N * plane_out;
    const int o0 = blockIdx.y * kTileO;
    const int64_t p0 = (int64_t)blockIdx.x * kTileP;
    const int tid = threadIdx.x % kT;
    if (kKW == 0) {
        for (int t = threadIdx.x; t < d.KH * d.KW; t += 2 * kT) tap_off[t] = (t / d.KW) * d.DH * d.W + (t % d.KW) * d.DW;
        __syncthreads();
    }
    if (threadIdx.x >= kT) {
    // gather role: pixel gp, kRowsPer consecutive filter rows (kKW = 0: taps) of every stage
    const int gp = tid % kTileP, gsub = tid / kTileP;
    const bool gather = kSub * kTileP == kT || gsub < kSub;
    const int period = kKW > 0 ? d.KH : d.KH * d.KW;  // rows (taps) of one input channel
    uint64_t inside = 0;                       // kKW = 0: taps inside the image; else filter columns inside it
    int ih0 = -0x40000000;                     // no row of it is inside
    const float* src = data;                   // the next row's first input (kKW = 0: the channel's plane at the first tap)
    {
        const int64_t p = p0 + gp;
        if (gather && p < P) {
            const int n = (int)(p / plane_out);
            const int rem = (int)(p - (int64_t)n * plane_out);
            const int oh = rem / d.OW, ow = rem - oh * d.OW;
            const int iw0 = ow * d.SW - d.PW;
            ih0 = oh * d.SH - d.PH;
            src = data + (int64_t)n * d.C * plane_in + (int64_t)ih0 * d.W + iw0;
            if (kKW > 0) {
                for (int rw = 0; rw < kKW; ++rw)
                    if (iw0 + rw >= 0 && iw0 + rw < d.W) inside |= 1ull << rw;
            } else {
                for (int rh = 0, t = 0; rh < d.KH; ++rh)
                    for (int rw = 0; rw < d.KW; ++rw, ++t) {
                        const int ih = ih0 + rh * d.DH, iw = iw0 + rw * d.DW;
                        if (ih >= 0 && ih < d.H && iw >= 0 && iw < d.W) inside |= 1ull << t;
                    }
            }
        }
    }
    const int row_step = kKW > 0 ? d.DH * d.W : 0;                      // to the next row of the same channel
    const int64_t wrap_step = (int64_t)plane_in - (int64_t)(period - 1) * row_step;  // from its last row to the next channel
    int left = d.C * period;                                          // rows up to the end of K
    int gt = 0, ih = ih0;
    auto advance = [&](int rows) {  // a few rows ahead
        const int c = rows / period, t = rows - c * period;
        src += (int64_t)c * plane_in + (int64_t)t * row_step;
        gt += t;
        left -= rows;
        if (gt >= period) {
            gt -= period;
            src += wrap_step - row_step;
        }
        ih = ih0 + gt * d.DH;
    };
    if (kSub > 1) advance(gsub * kRowsPer);
    const uint32_t gdst0 = (uint32_t)__cvta_generic_to_shared(xs + gsub * kRowsPer * (kKW > 0 ? kKW : 1) * kTileP + gp);

    // row i (of kRowsPer) of the next stage into buffer `buf`; afterwards the state stands at the following row
    auto gather_row = [&](int buf, int i) {
        const uint32_t dst = gdst0 + (uint32_t)((buf * KC + i * (kKW > 0 ? kKW : 1)) * kTileP * 4);
        if constexpr (kKW > 0) {
            const uint32_t cols = ((unsigned)ih < (unsigned)d.H && left > 0) ? (uint32_t)inside : 0u;
#pragma unroll
            for (int rw = 0; rw < kKW; ++rw) cp_async4_zfill(dst + rw * kTileP * 4, src + rw, cols & (1u << rw), gather);
        } else {
            cp_async4_zfill(dst, src + tap_off[gt], left > 0 ? (uint32_t)(inside >> gt) & 1u : 0u, gather);
        }
        const bool wrap = ++gt == period;
        gt = wrap ? 0 : gt;
        ih = wrap ? ih0 : ih + d.DH;
        src += wrap ? wrap_step : (int64_t)row_step;
        --left;
        if (kSub > 1 && i == kRowsPer - 1) advance(Stage::kRows - kRowsPer);
    };
    int buf = 0;
    auto hand_over = [&](int s) {  // stage s - kLag has landed
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (s >= kLag) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kLag) : "memory");
            named_arrive(1 + (buf >= kLag ? buf - kLag : buf - kLag + kBufs), 2 * kT);
        }
        buf = buf + 1 == kBufs ? 0 : buf + 1;
    };
    if constexpr (Stage::kAsync) {
        // weights: a warp copies blocks of kWK consecutive k of kWO channels; the pointers advance by a stage at a time
        const float* wsrc[kWPer];
        uint32_t wdst[kWPer];
        int wleft[kWPer];  // k up to the end of K; 0: no such channel
#pragma unroll
        for (int i = 0; i < kWPer; ++i) {
            const int block = tid / 32 + i * (kT / 32), l = tid & 31;
            const int k = block % (KC / Stage::kWK) * Stage::kWK + l % Stage::kWK;
            const int o = block / (KC / Stage::kWK) * Stage::kWO + l / Stage::kWK;
            const bool there = o < kTileO && o0 + o < d.O;
            wsrc[i] = there ? weight + (int64_t)(o0 + o) * K + k : weight;
            wdst[i] = (uint32_t)__cvta_generic_to_shared(ws + k * kWPitch + o);
            wleft[i] = there ? K - k : 0;
        }
        for (int s = 0; s < stages; ++s) {
            if (s >= kBufs) named_sync(1 + kBufs + buf, 2 * kT);  // the stage that lay here has been read
#pragma unroll
            for (int i = 0; i < kWPer; ++i) {
                const bool in_tile = kWLoads % kT == 0 || tid + i * kT < kWLoads;
                cp_async4_zfill(wdst[i] + (uint32_t)(buf * Smem::kWs * 4), wsrc[i], wleft[i] > 0 ? 1u : 0u, in_tile);
                wsrc[i] += wleft[i] > 0 ? KC : 0;
                wleft[i] -= KC;
            }
#pragma unroll
            for (int i = 0; i < kRowsPer; ++i) gather_row(buf, i);
            hand_over(s);
        }
    } else {
        // through registers: up to kWPer loads of kVec consecutive k of one channel; consecutive threads take consecutive channels
        const bool w_vec = K % kVec == 0 && (reinterpret_cast<uintptr_t>(weight) & (kVec * 4 - 1)) == 0;
        float wreg[kWPer][kVec];
        auto load_weights = [&](int k0) {
#pragma unroll
            for (int i = 0; i < kWPer; ++i) {
                const int q = tid + i * kT;
                const int o = o0 + q % kTileO, k = k0 + (q / kTileO) * kVec;
#pragma unroll
                for (int v = 0; v < kVec; ++v) wreg[i][v] = 0.0f;
                if (o < d.O && k < K && (kWLoads % kT == 0 || q < kWLoads)) {
                    const float* src = weight + (int64_t)o * K + k;
                    if (w_vec && kVec == 4) {
                        const float4 v = __ldg(reinterpret_cast<const float4*>(src));
                        wreg[i][0] = v.x; wreg[i][1] = v.y; wreg[i][kVec - 2] = v.z; wreg[i][kVec - 1] = v.w;
                    } else if (w_vec) {
                        const float2 v = __ldg(reinterpret_cast<const float2*>(src));
                        wreg[i][0] = v.x; wreg[i][1] = v.y;
                    } else {
#pragma unroll
                        for (int v = 0; v < kVec; ++v)
                            if (k + v < K) wreg[i][v] = __ldg(src + v);
                    }
                }
            }
        };
        load_weights(0);
        for (int s = 0; s < stages; ++s) {
            if (s >= kBufs) named_sync(1 + kBufs + buf, 2 * kT);
#pragma unroll
            for (int i = 0; i < kRowsPer; ++i) gather_row(buf, i);
#pragma unroll
            for (int i = 0; i < kWPer; ++i) {
                const int q = tid + i * kT;
                if (kWLoads % kT != 0 && q >= kWLoads) break;
                float* dst = ws + (buf * KC + (q / kTileO) * kVec) * kWPitch + q % kTileO;
#pragma unroll
                for (int v = 0; v < kVec; ++v) dst[v * kWPitch] = wreg[i][v];
            }
            load_weights((s + 1) * KC);
            hand_over(s);
        }
    }
    // the last stages, each as soon as it has landed (handed over together, short reductions waited for all their copies: 16 -> 16
    // channels 3x3 at 9x9 4.03 / 3.91 us)
    auto hand_over_last = [&](auto behind) {
        constexpr int kBehind = decltype(behind)::value;
        if (stages > kBehind) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kBehind) : "memory");
            named_arrive(1 + (stages - 1 - kBehind) % kBufs, 2 * kT);
        }
    };
    static_assert(kLag <= 3, "stages handed over after the loop");
    if constexpr (kLag > 2) hand_over_last(std::integral_constant<int, 2>{});
    if constexpr (kLag > 1) hand_over_last(std::integral_constant<int, 1>{});
    hand_over_last(std::integral_constant<int, 0>{});
    return;
    }

    const int pg = tid % kPG, og = tid / kPG;
    const uint64_t neg_zero = pack2(neg_zero_arg, neg_zero_arg);
    uint64_t acc[kTO][kTP / 2];
#pragma unroll
    for (int j = 0; j < kTO; ++j)
#pragma unroll
        for (int e = 0; e < kTP / 2; ++e) acc[j][e] = 0ull;
    int buf = 0;
    for (int s = 0; s < stages; ++s) {
        named_sync(1 + buf, 2 * kT);
#pragma unroll
        for (int k = 0; k < KC; ++k) {
            uint64_t x[kTP / 2], w[kTO];
            // the thread's pixels: groups of four consecutive ones kPG * 4 apart, then (kTP % 4 == 2) one pair
#pragma unroll
            for (int e = 0; e < kTP / 4; ++e) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(xs + (buf * KC + k) * kTileP + e * kPG * 4 + pg * 4);
                x[2 * e] = v.x;
                x[2 * e + 1] = v.y;
            }
            if constexpr (kTP % 4 != 0) x[kTP / 2 - 1] = *reinterpret_cast<const uint64_t*>(xs + (buf * KC + k) * kTileP + (kTP / 4) * kPG * 4 + pg * 2);
#pragma unroll
            for (int j = 0; j < kTO / 4; ++j) {
                const float4 v = *reinterpret_cast<const float4*>(ws + (buf * KC + k) * kWPitch + og * kTO + 4 * j);
                w[4 * j] = pack2(v.x, v.x);
                w[4 * j + 1] = pack2(v.y, v.y);
                w[4 * j + 2] = pack2(v.z, v.z);
                w[4 * j + 3] = pack2(v.w, v.w);
            }
            if constexpr (kTO % 4 != 0) {
                const float2 v = *reinterpret_cast<const float2*>(ws + (buf * KC + k) * kWPitch + og * kTO + kTO - 2);
                w[kTO - 2] = pack2(v.x, v.x);
                w[kTO - 1] = pack2(v.y, v.y);
            }
#pragma unroll
            for (int j = 0; j < kTO; ++j)
#pragma unroll
                for (int e = 0; e < kTP / 2; ++e) acc[j][e] = mac2_exact(acc[j][e], x[e], w[j], neg_zero);
        }
        if (s + kBufs < stages) named_arrive(1 + kBufs + buf, 2 * kT);
        buf = buf + 1 == kBufs ? 0 : buf + 1;
    }

    // Four consecutive pixels of one image are one 16-byte access where planes and pointers allow it. A pixel's place is found once
    // for all channels, and the residual of four channels is fetched before the first of their results is stored: with a 64-bit
    // division and one load in flight per result, short reductions were nothing but epilogue (19 -> 476 channels 1x1 over 81x81,
    // 18 images, with a residual: 625 us, now 301; over 80x82 418 and 277). All channels at once were slower in long ones
    // (128 -> 128 3x3 at 28x28, 32 images: 280 against 275 us, for registers), lanes that trade pixels so that a warp stores whole
    // rows in all of them (715 us).
    const bool vec = (plane_out & 3) == 0 && epi.aligned16();
    const int64_t image_step = (int64_t)d.O * plane_out;
#pragma unroll
    for (int g = 0; g < (kTP + 2) / 4; ++g) {
        const bool quad = 4 * g + 4 <= kTP;
        const int width = quad ? 4 : 2;
        const bool whole = quad && vec;
        int64_t base[4] = {-1, -1, -1, -1};  // where the thread's pixels lie in channel 0; -1: nowhere
#pragma unroll
        for (int e = 0; e < width; ++e) {
            const uint32_t p = (uint32_t)p0 + g * kPG * 4 + pg * width + e;  // (P is below 2^31)
            const uint32_t n = p / (uint32_t)plane_out;
            if (p < (uint32_t)P) base[e] = n * image_step + (p - n * plane_out);
        }
        if (base[0] < 0) continue;
        constexpr int kBatch = kTO < 4 ? kTO : 4;  // channels whose residual is in flight together
#pragma unroll
        for (int j0 = 0; j0 < kTO; j0 += kBatch) {
            float r[kBatch][4] = {};
#pragma unroll
            for (int i = 0; i < kBatch; ++i) {
                const int o = o0 + og * kTO + j0 + i;
                if (o >= d.O) continue;
                if (whole) {
                    epi.fetch4(r[i], base[0] + (int64_t)o * plane_out);
                } else {
#pragma unroll
                    for (int e = 0; e < width; ++e)
                        if (base[e] >= 0) r[i][e] = epi.fetch(base[e] + (int64_t)o * plane_out);
                }
            }
#pragma unroll
            for (int i = 0; i < kBatch; ++i) {
                const int o = o0 + og * kTO + j0 + i;
                if (o >= d.O) continue;
                float v[4] = {0.f, 0.f, 0.f, 0.f};
                asm("mov.b64 {%0, %1}, %2;" : "=f"(v[0]), "=f"(v[1]) : "l"(acc[j0 + i][2 * g]));
                if (quad) asm("mov.b64 {%0, %1}, %2;" : "=f"(v[2]), "=f"(v[3]) : "l"(acc[j0 + i][quad ? 2 * g + 1 : 0]));
#pragma unroll
                for (int e = 0; e < width; ++e) v[e] = epi.finish(v[e], r[i][e], o);
                if (whole) {
                    *reinterpret_cast<float4*>(epi.out + base[0] + (int64_t)o * plane_out) = make_float4(v[0], v[1], v[2], v[3]);
                } else {
#pragma unroll
                    for (int e = 0; e < width; ++e)
                        if (base[e] >= 0) epi.out[base[e] + (int64_t)o * plane_out] = v[e];
                }
            }
        }
    }
}

struct EpilogueF32 {
    const float* bias;
    const float* residual;
    float* out;
    int relu;
    __device__ __forceinline__ float fetch(int64_t lin) const { return residual ? __ldg(residual + lin) : 0.0f; }
    __device__ __forceinline__ void fetch4(float (&r)[4], int64_t lin) const {  // lin: a multiple of four
        if (residual) {
            const float4 q = __ldg(reinterpret_cast<const float4*>(residual + lin));
            r[0] = q.x; r[1] = q.y; r[2] = q.z; r[3] = q.w;
        }
    }
    // the result of channel o: r as fetched
    __device__ __forceinline__ float finish(float v, float r, int o) const {
        if (bias) v = __fadd_rn(v, __ldg(bias + o));
        if (residual) v = __fadd_rn(v, r);
        if (relu) v = v > 0.0f ? v : 0.0f;
        return v;
    }
    __device__ __forceinline__ void operator()(float acc, int64_t lin, int o) const { out[lin] = finish(acc, fetch(lin), o); }
    __device__ __forceinline__ bool aligned16() const {
        return ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(residual)) & 15u) == 0;
    }
};

struct EpilogueS8 {
    const int32_t* bias;
    const int32_t* multiplier;
    const int32_t* shift;
    int8_t* out;
    int relu;
    __device__ __forceinline__ void operator()(int32_t acc, int64_t lin, int o) const {
        out[lin] = requantize_s8(acc + __ldg(bias + o), __ldg(multiplier + o), __ldg(shift + o), relu);
    }
};

// nn_dense / nn_gemm in reference order, for what the packed kernel does not take: acc = 0; acc += a[i,k]*b[j,k]; (*alpha); + (beta*)c[j]
// (include/te/topi/nn.h:48-101, src/relay/op/nn/dense.cc:34-61).
__global__ void __launch_bounds__(kThreads) gemm_direct_kernel(const float* __restrict__ a, const float* __restrict__ b,
                                                               const float* __restrict__ c, float* __restrict__ out,
                                                               int M, int N, int K, float alpha, float beta, int transB,
                                                               int has_c) {
    sm100::pdl_wait();
    const int64_t total = (int64_t)M * N;
    for (int64_t lin = (int64_t)blockIdx.x * kThreads + threadIdx.x; lin < total; lin += (int64_t)gridDim.x * kThreads) {
        const int j = (int)(lin % N);
        const int i = (int)(lin / N);
        float acc = 0.0f;
        if (transB) {
            for (int k = 0; k < K; ++k) acc = __fadd_rn(acc, __fmul_rn(__ldg(a + (int64_t)i * K + k), __ldg(b + (int64_t)j * K + k)));
        } else {
            for (int k = 0; k < K; ++k) acc = __fadd_rn(acc, __fmul_rn(__ldg(a + (int64_t)i * K + k), __ldg(b + (int64_t)k * N + j)));
        }
        if (has_c) {
            if ((double)alpha != 1.0) acc = __fmul_rn(acc, alpha);
            float bias = __ldg(c + j);
            if ((double)beta != 1.0) bias = __fmul_rn(bias, beta);
            acc = __fadd_rn(acc, bias);
        }
        out[lin] = acc;
    }
}

int grid_for(int64_t items) {
    int64_t blocks = (items + kThreads - 1) / kThreads;
    const int64_t cap = (int64_t)kNumSMs * 16;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    return (int)blocks;
}

// Tile of the packed kernel. The sum over k is one chain per output and cannot be split, so a launch's parallelism is its
// outputs: large tiles for large launches, smaller ones where they would leave SMs idle. The estimate is the number of
// blocks on the busiest SM times the clocks a block takes there per k (`alone`: a single block on its SM, latencies showing;
// `shared`: per block when there are several). Filters of width 3 and 7: fits over 156 convolutions of 1 to 64 images timed
// with every tile, 4 to 7 % off (10 % at 16x16); what they choose is 0.1 % behind the fastest tile on average and 1.08 times as
// fast as the best of the first four tiles. The others, where the epilogue weighs as much as the sum: as measured on ResNet-18.
//   tile (channels x pixels)    64x128   64x96  32x64  16x32  16x16  32x96  32x32  32x128
//   FMA-pipe bound                 128      96     32      8      4     48     16      64
struct ExactCost {
    int tile_o, tile_p;
    double alone, shared;
};
constexpr ExactCost kExactCosts[] = {{64, 128, 157.0, 150.0}, {64, 96, 126.0, 120.0}, {32, 64, 59.0, 45.0}, {16, 32, 31.0, 20.5}};
constexpr ExactCost kExactWideCosts[] = {{64, 128, 162.8, 153.6}, {64, 96, 127.2, 120.0}, {32, 64, 49.2, 46.4}, {16, 32, 21.7, 18.4},
                                         {16, 16, 14.8, 11.8},    {32, 96, 71.2, 67.2},   {32, 32, 32.1, 27.2}, {32, 128, 88.2, 83.2}};

template <int kCount>
int pick_exact_tile(const ConvDims& d, const ExactCost (&costs)[kCount]) {
    const int64_t P = (int64_t)d.N * d.OH * d.OW;
    int best = 0;
    double best_cost = 0.0;
    for (int i = 0; i < kCount; ++i) {
        const ExactCost& c = costs[i];
        const int64_t blocks = ((P + c.tile_p - 1) / c.tile_p) * ((d.O + c.tile_o - 1) / c.tile_o);
        const int64_t per_sm = (blocks + kNumSMs - 1) / kNumSMs;
        const double cost = per_sm <= 1 ? c.alone : (double)per_sm * c.shared;
        if (i == 0 || cost < best_cost) {
            best = i;
            best_cost = cost;
        }
    }
    return best;
}

template <int kKW, int kTO, int kTP, int kOG, int kPG, int kMul, int kDeep>
int32_t launch_exact(const float* data, const float* weight, const ConvDims& d, const EpilogueF32& epi, cudaStream_t s) {
    using Tile = ExactTile<kTO, kTP, kOG, kPG>;
    constexpr int kBytes = ExactSmem<kKW, kTO, kTP, kOG, kPG, kMul, kDeep>::kBytes;
    auto kernel = conv2d_tiled_f32_kernel<kKW, kTO, kTP, kOG, kPG, kMul, kDeep, EpilogueF32>;
    static PerDeviceOnce smem_once;
    KXC_TRY(smem_opt_in(smem_once, kernel, kBytes));
    const int64_t P = (int64_t)d.N * d.OH * d.OW;
    const dim3 grid((unsigned)((P + Tile::kP - 1) / Tile::kP), (unsigned)((d.O + Tile::kO - 1) / Tile::kO), 1u);
    KXC_CUDA_TRY(launch_kernel(kernel, grid, dim3(2 * Tile::kThreads), kBytes, s, /*pdl=*/true, 1, data, weight, d, -0.0f, epi));
    return check_launch("nn_conv2d (fp32, tiled)");
}

template <int kKW>
int32_t launch_exact_width(const float* data, const float* weight, const ConvDims& d, const EpilogueF32& epi, cudaStream_t s) {
    if constexpr (kKW >= 3) {
        switch (pick_exact_tile(d, kExactWideCosts)) {
            case 4: return launch_exact<kKW, 2, 2, 8, 8, 4, 5>(data, weight, d, epi, s);
            case 5: return launch_exact<kKW, 4, 6, 8, 16, 1, 4>(data, weight, d, epi, s);
            case 6: return launch_exact<kKW, 4, 2, 8, 16, 2, 5>(data, weight, d, epi, s);
            case 7: return launch_exact<kKW, 4, 8, 8, 16, 1, 4>(data, weight, d, epi, s);
            default: break;
        }
    }
    switch (kKW >= 3 ? pick_exact_tile(d, kExactWideCosts) : pick_exact_tile(d, kExactCosts)) {
        case 0: return launch_exact<kKW, 8, 8, 8, 16, 1, 3>(data, weight, d, epi, s);
        case 1: return launch_exact<kKW, 8, 6, 8, 16, 1, 3>(data, weight, d, epi, s);
        case 2: return launch_exact<kKW, 4, 4, 8, 16, 2, 5>(data, weight, d, epi, s);
        default: return launch_exact<kKW, 2, 2, 8, 16, 4, 5>(data, weight, d, epi, s);
    }
}

// one thread per output for a handful of them, filters of more than 64 taps and extents beyond 32-bit offsets
bool tiled_f32_ok(const ConvDims& d) {
    const int64_t P = (int64_t)d.N * d.OH * d.OW;
    return P * d.O >= 64 && d.KH * d.KW <= kExactMaxTaps && P <= 0x7fffffffll && (int64_t)d.H * d.W <= 0x3fffffffll &&
           (int64_t)d.C * d.KH * d.KW <= 0x3fffffffll && (d.O + 15) / 16 <= 65535 &&
           (int64_t)d.KH * d.DH * d.W + (int64_t)d.KW * d.DW <= 0x3fffffffll;
}

int32_t launch_tiled_f32(const float* data, const float* weight, const ConvDims& d, const EpilogueF32& epi, cudaStream_t s) {
    switch (d.DW == 1 ? d.KW : 0) {
        case 1: return launch_exact_width<1>(data, weight, d, epi, s);
        case 3: return launch_exact_width<3>(data, weight, d, epi, s);
        case 7: return launch_exact_width<7>(data, weight, d, epi, s);
        default: return launch_exact_width<0>(data, weight, d, epi, s);
    }
}

}  // namespace

int32_t conv2d_fp32_exact(const float* data, const float* weight, const float* bias, const float* residual, float* out,
                          const ConvDims& d, int relu, cudaStream_t s) {
    const int64_t total = (int64_t)d.N * d.O * d.OH * d.OW;
    if (total == 0) return KXC_B200_OK;
    EpilogueF32 epi{bias, residual, out, relu};
    if (tiled_f32_ok(d)) return launch_tiled_f32(data, weight, d, epi, s);
    KXC_CUDA_TRY(launch_kernel(conv2d_direct_kernel<float, float, EpilogueF32>, dim3(grid_for(total)), dim3(kThreads), 0, s, /*pdl=*/true, 1, data,
                               weight, d, epi));
    return check_launch("nn_conv2d (fp32)");
}

int32_t conv2d_s8_exact(const int8_t* data, const int8_t* weight, const int32_t* bias, const int32_t* multiplier,
                        const int32_t* shift, int8_t* out, const ConvDims& d, int relu, cudaStream_t s) {
    const int64_t total = (int64_t)d.N * d.O * d.OH * d.OW;
    if (total == 0) return KXC_B200_OK;
    EpilogueS8 epi{bias, multiplier, shift, out, relu};
    KXC_CUDA_TRY(launch_kernel(conv2d_direct_kernel<int8_t, int32_t, EpilogueS8>, dim3(grid_for(total)), dim3(kThreads), 0, s, /*pdl=*/true, 1, data,
                               weight, d, epi));
    return check_launch("nn_conv2d_s8 (direct)");
}

int32_t gemm_fp32_exact(const float* a, const float* b, const float* c, float* out, const kxc_b200_gemm_desc& g,
                        cudaStream_t s) {
    const int64_t total = (int64_t)g.m * g.n;
    if (total == 0) return KXC_B200_OK;
    // [M,K] x [N,K]^T + c is a 1x1 convolution over M images of one pixel, in the same order (32 x 1000 x 512: 76 -> 20 us)
    const bool plain = !g.has_c || ((double)g.alpha == 1.0 && (double)g.beta == 1.0);
    const ConvDims d{g.m, g.k, 1, 1, g.n, 1, 1, 1, 1, 0, 0, 1, 1, 1, 1};
    if (g.transB && plain && g.k > 0 && tiled_f32_ok(d)) return launch_tiled_f32(a, b, d, EpilogueF32{g.has_c ? c : nullptr, nullptr, out, 0}, s);
    KXC_CUDA_TRY(launch_kernel(gemm_direct_kernel, dim3(grid_for(total)), dim3(kThreads), 0, s, /*pdl=*/true, 1, a, b, c, out, g.m, g.n, g.k, g.alpha,
                               g.beta, g.transB, g.has_c));
    return check_launch("nn_gemm (fp32)");
}

}  // namespace kxc_b200
