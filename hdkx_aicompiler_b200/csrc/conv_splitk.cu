// Implicit-GEMM convolution / dense layer whose reduction is split over the CTAs of a cluster (see conv_tc.cuh for the GEMM
// view). For launches with fewer tiles than SMs: the deep layers of a small batch are 8 to 64 tiles of 36 to 72 K blocks, and
// one CTA walks its K blocks at the rate its own operand stream arrives (~50 B/clk), 16 to 24 us for 72 blocks whatever the
// rest of the chip does. ResNet-18 bf16 on one image: 221 -> 130 us (layer 4: 24 -> 7.5 us per convolution, layer 3: 14.5 -> 7.4).
//
// One cluster = one output tile of 128 pixels x BN channels; CTA r of S takes the K blocks [r*K/S, (r+1)*K/S) through the same
// TMA -> tcgen05.mma pipeline and owns the r-th S-th of the rows. It writes its partial sums into its own (by then idle) operand
// ring; each warp sends the rows of its 32 x 32 piece to their owners as bulk copies between the CTAs' shared memories, counted on the
// owner's mbarrier, and the owner adds the S parts in rank order and applies the epilogue. No partial sum touches global memory,
// nothing is atomic, and the result does not depend on timing.
// The other ways to exchange them were slower: owners that fetch the parts after a cluster barrier, a few 16-byte loads per
// thread in flight (whole networks, us before / now: bf16 one image 127.3 / 121.0, 8: 161.9 / 155.7; tf32 one image 168.0 / 157.8,
// 4: 204.0 / 189.5, 32: 491.6 / 476.7), and 16-byte st.async from the accumulator to the owners (slower than the fetches from two
// images on, tf32 32: 524).
//
// Both issuing loops run on whole warps (elect_one in sm100.cuh): ResNet-18 tf32 one image 147.4 -> 134.8 us, bf16 109.7 -> 102.4; 512 -> 512 3x3
// at 7x7, tf32, 8 images 14.4 -> 11.8.
//
//   warp 0      TMA producer; loads the weights of the first stages before it waits for the previous kernel (weights of a
//               plan do not come from that kernel), so only the pixels are on the critical path of a layer
//   warp 1      MMA issuer, TMEM owner
//   warps 2..9  accumulator -> shared memory -> owners, then reduction and epilogue, 8 channels of one pixel per thread and step
//
// The shape of the launch (S, BN) comes from choose_split or, with two outputs, tc_setup_dual in conv_tc.cu. Waits are bounded as in conv_tc.cu; the cluster
// barriers are reached by every thread of every CTA whether or not a wait ran out.
#include "conv_tc.cuh"

#include <cuda_bf16.h>

#include <mutex>

#include "common.cuh"
#include "conv_epilogue.cuh"
#include "sm100.cuh"

namespace kxc_b200 {
namespace {

using namespace sm100;

constexpr int kSplitThreads = 320;
constexpr int kKB = 128;  // bytes of a K block
constexpr int kSplitSmem = 227 * 1024 - 2048;

template <int BN, bool kX3, bool kDual = false>
struct SplitGeom {
    static constexpr int kATile = 128 * kKB;
    static constexpr int kBTile = BN * kKB;
    static constexpr int kABytes = (kX3 ? 2 : 1) * kATile;
    static constexpr int kStageBytes = kABytes + (kX3 ? 2 : 1) * kBTile;
    // A CTA's own sums: [BN / 32][128 rows][128 bytes], at the start of the ring. What it receives: [BN / 32][other ranks][rows][128
    // bytes], at most 7 x 16 or 6 x 19 rows (256 channels: up to 3 x 32), one rank more with a second output.
    static constexpr int kSumBytes = 128 * BN * 4;
    static constexpr int kMaxParts = BN == 256 ? 4 : kMaxSplit;
    static constexpr int kRecvRows = kDual ? 133 : (BN == 256 ? 96 : 114);
    static constexpr int kRecvBytes = kRecvRows * BN * 4;
    // It lies behind the ring, ready from the start, where that costs one of eight stages; else behind the CTA's own sums, from when
    // the cluster's MMAs have read the rings (128 channels with five of seven stages and a buffer: 2 to 3 % slower in long reductions).
    static constexpr bool kOwnBuffer = BN == 64 && !kX3;
    static constexpr int kStagesRaw = (kSplitSmem - 1024 - (kOwnBuffer ? kRecvBytes : 0)) / kStageBytes;
    static constexpr int kStages = kStagesRaw > 8 ? 8 : kStagesRaw;
    static constexpr int kRecvOffset = kOwnBuffer ? kStages * kStageBytes : kSumBytes;
    static constexpr int kUsed = kRecvOffset + kRecvBytes > kStages * kStageBytes ? kRecvOffset + kRecvBytes : kStages * kStageBytes;
    static constexpr int kSmemBytes = kUsed + 1024;
    static_assert(kSmemBytes <= kSplitSmem && (kDual ? 2 : 1) * kSumBytes <= (kOwnBuffer ? kStages * kStageBytes : kSumBytes), "shared memory of one CTA");
};

// `bytes` (a multiple of 16) into a CTA of the cluster, counted on the mbarrier `cluster_bar` of that CTA
__device__ __forceinline__ void bulk_copy_to_cta(uint32_t cluster_dst, uint32_t src, uint32_t bytes, uint32_t cluster_bar) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(cluster_dst), "r"(src),
                 "r"(bytes), "r"(cluster_bar)
                 : "memory");
}

// byte offset of 16-byte piece 0..7 in a row of 32 sums (pieces rotate with the tile's row, so that both a warp of rows and a warp of
// pieces touch all banks)
__device__ __forceinline__ uint32_t piece_off(int row, int piece) { return (uint32_t)((piece ^ (row & 7)) << 4); }

// 8 consecutive channels [c0, c0 + 8) of one pixel: a thread's share of a step
struct Item {
    bool mine;
    int second, piece, local, row;  // second output; piece of 8 columns; row of the owner's share, of the tile
    int c0, n, oh, ow;
};

// what the epilogue of an item reads from global memory, fetched while the sums are still on their way
template <int kOutMode>
struct Ahead {
    float bias[8];
    uint32_t res[kOutMode == kOutNHWC_BF16 ? 4 : 8];  // bf16 pairs or fp32
};

template <int kOutMode>
__device__ __forceinline__ void fetch_ahead(const TcParams& p, const Item& it, const float* bias, const void* residual, Ahead<kOutMode>& a) {
    if (!it.mine) return;
    const int nch = p.Cout - it.c0 < 8 ? p.Cout - it.c0 : 8;
    const size_t pix = ((size_t)it.n * p.OH + it.oh) * p.OW + it.ow;
    if (bias != nullptr) {
        if (nch == 8 && p.vec_ok) {
            const float4 x = __ldg(reinterpret_cast<const float4*>(bias + it.c0)), y = __ldg(reinterpret_cast<const float4*>(bias + it.c0) + 1);
            a.bias[0] = x.x; a.bias[1] = x.y; a.bias[2] = x.z; a.bias[3] = x.w;
            a.bias[4] = y.x; a.bias[5] = y.y; a.bias[6] = y.z; a.bias[7] = y.w;
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) a.bias[j] = j < nch ? __ldg(bias + it.c0 + j) : 0.0f;
        }
    }
    if (residual == nullptr) return;
    if constexpr (kOutMode == kOutNHWC_BF16) {
        const __nv_bfloat16* res = static_cast<const __nv_bfloat16*>(residual) + pix * p.Cout + it.c0;
        if (nch == 8 && (p.Cout & 7) == 0 && p.vec_ok) {
            const uint4 r = __ldg(reinterpret_cast<const uint4*>(res));
            a.res[0] = r.x; a.res[1] = r.y; a.res[2] = r.z; a.res[3] = r.w;
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t lo = 2 * k < nch ? __ldg(reinterpret_cast<const unsigned short*>(res) + 2 * k) : 0u;
                const uint32_t hi = 2 * k + 1 < nch ? __ldg(reinterpret_cast<const unsigned short*>(res) + 2 * k + 1) : 0u;
                a.res[k] = lo | (hi << 16);
            }
        }
    } else {
        const size_t plane = kOutMode == kOutNCHW_F32 ? (size_t)p.OH * p.OW : 1;
        const float* res = static_cast<const float*>(residual) + (kOutMode == kOutNCHW_F32 ? ((size_t)it.n * p.Cout + it.c0) * plane + (size_t)it.oh * p.OW + it.ow
                                                                                           : pix * p.Cout + it.c0);
        if (kOutMode == kOutNHWC_F32 && nch == 8 && (p.Cout & 3) == 0 && p.vec_ok) {
            const uint4 x = __ldg(reinterpret_cast<const uint4*>(res)), y = __ldg(reinterpret_cast<const uint4*>(res) + 1);
            a.res[0] = x.x; a.res[1] = x.y; a.res[2] = x.z; a.res[3] = x.w;
            a.res[4] = y.x; a.res[5] = y.y; a.res[6] = y.z; a.res[7] = y.w;
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) a.res[j] = j < nch ? __float_as_uint(__ldg(res + j * plane)) : 0u;
        }
    }
}

// +bias -> +residual -> ReLU -> store of an item
template <int kOutMode, bool kSplitOut>
__device__ __forceinline__ void epilogue8(const TcParams& p, float (&f)[8], const Ahead<kOutMode>& a, bool has_bias, bool has_res, void* out_ptr,
                                          int relu, const Item& it) {
    const int c0 = it.c0;
    const int nch = p.Cout - c0 < 8 ? p.Cout - c0 : 8;
    const size_t pix = ((size_t)it.n * p.OH + it.oh) * p.OW + it.ow;
    if (has_bias) {
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = __fadd_rn(f[j], a.bias[j]);
    }
    if (has_res) {
        if constexpr (kOutMode == kOutNHWC_BF16) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                f[2 * k] = __fadd_rn(f[2 * k], bf16_lo(a.res[k]));
                f[2 * k + 1] = __fadd_rn(f[2 * k + 1], bf16_hi(a.res[k]));
            }
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) f[j] = __fadd_rn(f[j], __uint_as_float(a.res[j]));
        }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = relu && !(f[j] > 0.0f) ? 0.0f : f[j];
    if constexpr (kOutMode == kOutNCHW_F32) {
        const size_t plane = (size_t)p.OH * p.OW;
        float* out = static_cast<float*>(out_ptr) + ((size_t)it.n * p.Cout + c0) * plane + (size_t)it.oh * p.OW + it.ow;
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (j < nch) out[j * plane] = f[j];
    } else if constexpr (kOutMode == kOutNHWC_BF16) {
        __nv_bfloat16* out = static_cast<__nv_bfloat16*>(out_ptr) + pix * p.Cout + c0;
        if (nch == 8 && (p.Cout & 7) == 0 && p.vec_ok) {
            *reinterpret_cast<uint4*>(out) = make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (j < nch) out[j] = __float2bfloat16_rn(f[j]);
        }
    } else {  // kOutNHWC_F32
        const size_t off = pix * p.Cout + c0;
        const bool whole = nch == 8 && (p.Cout & 3) == 0;
        if (p.round_out_tf32) {
#pragma unroll
            for (int j = 0; j < 8; ++j) f[j] = tf32_rne(f[j]);
        }
        auto store = [&](float* dst, const float (&v)[8], bool wide) {
            if (wide) {
                reinterpret_cast<float4*>(dst)[0] = make_float4(v[0], v[1], v[2], v[3]);
                reinterpret_cast<float4*>(dst)[1] = make_float4(v[4], v[5], v[6], v[7]);
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (j < nch) dst[j] = v[j];
            }
        };
        if constexpr (kSplitOut) {
            if (p.out_hi != nullptr) {
                float h[8], l[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    h[j] = tf32_rne(f[j]);
                    l[j] = tf32_low_part(f[j], h[j]);
                }
                store(p.out_hi + off, h, whole);
                store(p.out_hi + p.out_lo_offset + off, l, whole);
            }
            if (out_ptr == nullptr) return;
        }
        store(static_cast<float*>(out_ptr) + off, f, whole && p.vec_ok);
    }
}

// kDual, kX3: as in conv_tc.cu (second output through tmB2 / out2; high and low operand parts).
template <MmaKind kKind, int BN, int kOutMode, bool kDual, bool kX3>
__global__ void __launch_bounds__(kSplitThreads, 1) conv_splitk_kernel(const __grid_constant__ TcParams p) {
    using G = SplitGeom<BN, kX3, kDual>;
    static_assert(!(kDual && kX3), "one of the two");
    constexpr int kStages = G::kStages;
    constexpr uint32_t kTmemCols = (kDual || kX3 ? 2 : 1) * BN;
    constexpr uint32_t kFmt = kKind == MmaKind::F16 ? kFmtBF16 : kFmtTF32;
    constexpr uint32_t kIdesc = make_instr_desc(kFmt, kAccF32, BN, 128u);
    [[maybe_unused]] constexpr uint32_t kIdescWide = make_instr_desc(kFmt, kAccF32, 2 * BN <= 256 ? 2 * BN : 256, 128u);

    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bar_full[kStages];
    __shared__ __align__(8) uint64_t bar_empty[kStages];
    __shared__ __align__(8) uint64_t bar_acc;
    __shared__ __align__(8) uint64_t bar_recv;
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);  // (a uniform value, as the compiler then knows)
    const int lane = threadIdx.x & 31;
    const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int rank = (int)cluster_cta_rank();
    const int S = p.split;
    const int tile = (int)blockIdx.x / S;
    // The tile's rows that hold pixels are shared out: `rows` to an owner, fewer or none to the last ones. (All 128 shared out and sent,
    // whatever they held / these: dense 1 x 4096 x 1024 tf32 14.6 / 13.4 us with its conversion; ResNet-18 bf16 one image 120.8 / 118.4,
    // 8: 155.7 / 151.5, tf32 4: 191.7 / 185.1, three passes 4: 283.8 / 276.5.)
    const int rows_used = p.BW * p.BH * p.BNI;
    const int rows = (rows_used + S - 1) / S;
    const int rest = rows_used - rank * rows;
    const int my_rows = rest < 0 ? 0 : (rest < rows ? rest : rows);
    const int parts = S - 1 + (kDual ? 1 : 0);  // received per 32 columns: the other ranks' in order, the last rank's second output
    const uint32_t recv = ring + (uint32_t)G::kRecvOffset;

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < kStages; ++s) {
            mbar_init(smem_u32(&bar_full[s]), 1);
            mbar_init(smem_u32(&bar_empty[s]), 1);
        }
        mbar_init(smem_u32(&bar_acc), 1);
        mbar_init(smem_u32(&bar_recv), 1);
        mbar_fence_init();
        mbar_arrive_expect_tx(smem_u32(&bar_recv), (uint32_t)((rank == S - 1 ? S - 1 : parts) * my_rows * BN * 4));
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(&tmem_base_slot), kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_base_slot, 0);
    volatile int* abort_ptr = &abort_flag;
    // First cluster barrier: every CTA's receive buffer and its mbarrier are ready. Arrived at here, or when the ring is idle.
    if constexpr (G::kOwnBuffer) cluster_arrive();
    pdl_launch_dependents();

    const int kb_main = p.taps_h * p.taps_w * p.cblocks;
    const int kb_all = kb_main + (kDual ? p.cblocks : 0);
    // The second output's few blocks go to the last rank alone: its sum is formed in the order of a launch of its own, and the
    // main sum's parts are those of a launch without it in as many parts (bit-identical then).
    const int kb0 = rank * kb_main / S, kb1 = rank == S - 1 ? kb_all : (rank + 1) * kb_main / S;
    const int ct = tile % p.tiles_c;
    int r = tile / p.tiles_c;
    const int tw = r % p.tiles_w; r /= p.tiles_w;
    const int th = r % p.tiles_h;
    const int tn = r / p.tiles_h;
    const int ow0 = tw * p.BW, oh0 = th * p.BH, n0 = tn * p.BNI;

    if (warp == 0) {
        // The three-pass form of 128 channels keeps a loop of one lane: its stages of 64 KB, asked for any faster, arrive later (512 -> 512 at 7x7,
        // 32 images 45.5 us, 47.2 with the whole warp; 51.2 with the pixels' loads before the weights').
        constexpr bool kWhole = !(kX3 && BN == 128);
        const bool lead = kWhole ? elect_one() : lane == 0;
        auto converge = [] {
            if constexpr (kWhole) __syncwarp();
        };
        if (kWhole || lead) {
            if (lead) {
                tma_prefetch_desc(&p.tmB);
                tma_prefetch_desc(&p.tmA[0]);
                if constexpr (kDual || kX3) tma_prefetch_desc(&p.tmB2);
            }
            const uint32_t tx_bytes = (uint32_t)((kX3 ? 2 : 1) * (rows_used * kKB + G::kBTile));
            auto load_weights = [&](int kb, int stage) {
                const uint32_t full = smem_u32(&bar_full[stage]);
                const uint32_t dst = ring + (uint32_t)stage * G::kStageBytes + G::kABytes;
                if (!lead) return;
                mbar_arrive_expect_tx(full, tx_bytes);
                if (kDual && kb >= kb_main) {
                    tma_load_2d(dst, &p.tmB2, full, (kb - kb_main) * p.kb_elems, ct * BN);
                } else {
                    tma_load_2d(dst, &p.tmB, full, kb * p.kb_elems, ct * BN);
                    if constexpr (kX3) tma_load_2d(dst + G::kBTile, &p.tmB2, full, kb * p.kb_elems, ct * BN);
                }
            };
            auto load_pixels = [&](int kb, int stage) {
                int cb, kh, kw;
                if (kDual && kb >= kb_main) {  // the 1x1 convolution reads the centre tap
                    cb = kb - kb_main;
                    kh = p.taps_h / 2;
                    kw = p.taps_w / 2;
                } else {
                    const int tap = kb / p.cblocks;
                    cb = kb - tap * p.cblocks;
                    kh = tap / p.taps_w;
                    kw = tap - kh * p.taps_w;
                }
                const int dh = kh * p.dil_h - p.pad_h, dw = kw * p.dil_w - p.pad_w;
                int map = 0, ch = dh, cw = dw;
                if (p.stride == 2) {
                    const int hp = dh & 1, wp = dw & 1;
                    map = hp * 2 + wp;
                    ch = (dh - hp) >> 1;
                    cw = (dw - wp) >> 1;
                }
                const uint32_t full = smem_u32(&bar_full[stage]);
                const uint32_t dst = ring + (uint32_t)stage * G::kStageBytes;
                if (!lead) return;
                tma_load_4d(dst, &p.tmA[map], full, cb * p.kb_elems, ow0 + cw, oh0 + ch, n0);
                if constexpr (kX3) tma_load_4d(dst + G::kATile, &p.tmA[map], full, cb * p.kb_elems, ow0 + cw, oh0 + ch, n0 + p.N);
            };
            const int early = p.weights_ready ? (kb1 - kb0 < kStages ? kb1 - kb0 : kStages) : 0;
            for (int i = 0; i < early; ++i) load_weights(kb0 + i, i);
            converge();
            pdl_wait();  // the pixels come from the previous kernel
            for (int i = 0; i < early; ++i) load_pixels(kb0 + i, i);
            converge();
            int stage = early == kStages ? 0 : early;
            uint32_t phase = early == kStages ? 1u : 0u;
            for (int kb = kb0 + early; kb < kb1; ++kb) {
                if (!(kWhole ? mbar_wait_warp(smem_u32(&bar_empty[stage]), phase ^ 1u, abort_ptr) : mbar_wait_bounded(smem_u32(&bar_empty[stage]), phase ^ 1u, abort_ptr))) break;
                load_weights(kb, stage);
                load_pixels(kb, stage);
                converge();
                if (++stage == kStages) { stage = 0; phase ^= 1u; }
            }
        }
    } else if (warp == 1) {
        const bool lead = elect_one();
        int stage = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (int kb = kb0; kb < kb1; ++kb) {
            if (!mbar_wait_warp(smem_u32(&bar_full[stage]), phase, abort_ptr)) {
                ok = false;
                break;
            }
            tc_fence_after_sync();
            const bool second = kDual && kb >= kb_main;
            const bool first_of_sum = kb == kb0 || (kDual && kb == kb_main);
            const uint32_t d = tmem_base + (second ? (uint32_t)BN : 0u);
            const uint32_t a_addr = ring + (uint32_t)stage * G::kStageBytes;
            const uint64_t a_desc = make_smem_desc(a_addr, kKB), b_desc = make_smem_desc(a_addr + G::kABytes, kKB);
            if (lead) {
#pragma unroll
                for (int k = 0; k < kKB / 32; ++k) {
                    const uint64_t a_k = a_desc + (uint64_t)(2 * k), b_k = b_desc + (uint64_t)(2 * k);
                    const uint32_t accumulate = first_of_sum && k == 0 ? 0u : 1u;
                    if constexpr (kX3) {
                        umma<kKind>(d, a_k, b_k, kIdescWide, accumulate);
                        umma<kKind>(d + (uint32_t)BN, a_k + (uint64_t)(G::kATile >> 4), b_k, kIdesc, 1u);
                    } else {
                        umma<kKind>(d, a_k, b_k, kIdesc, accumulate);
                    }
                }
                umma_commit(smem_u32(&bar_empty[stage]));
            }
            __syncwarp();
            if (++stage == kStages) { stage = 0; phase ^= 1u; }
        }
        if (ok && lead) umma_commit(smem_u32(&bar_acc));
    } else {
        // this CTA's partial sums into its ring and on to the owners of their rows: every load has landed and every MMA has read it
        // once bar_acc completes
        const int quad = warp & 3, half = (warp - 2) >> 2;
        const int row = quad * 32 + lane;
        pdl_wait();  // residual reads and output writes must not overtake earlier kernels
        bool ok = mbar_wait_bounded(smem_u32(&bar_acc), 0, abort_ptr);
        ok = __all_sync(0xffffffffu, ok);
        if constexpr (!G::kOwnBuffer) cluster_arrive();
        tc_fence_after_sync();
        // lanes 0 to 7: the owners of the warp's rows, and the rows of them
        const int owner = quad * 32 / rows + lane;
        const int from = owner * rows > quad * 32 ? owner * rows : quad * 32;
        int upto = (owner + 1) * rows < quad * 32 + 32 ? (owner + 1) * rows : quad * 32 + 32;
        if (upto > rows_used) upto = rows_used;
        const bool sends = lane < kMaxSplit && from < upto && owner != rank;
        const uint32_t to = map_to_cta(recv, sends ? (uint32_t)owner : 0u), to_bar = map_to_cta(smem_u32(&bar_recv), sends ? (uint32_t)owner : 0u);
        const int slot = rank < owner ? rank : rank - 1;  // of this rank among the owner's parts
        bool ready = false;
#pragma unroll 1
        for (int a = 0; a < (kDual ? 2 : 1); ++a) {
            if (a == 1 && rank != S - 1) continue;
#pragma unroll 1
            for (int i = 0; i < BN / 64; ++i) {
                const int cg = half * (BN / 64) + i;  // 32 columns
                const uint32_t t_addr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(a * BN + cg * 32);
                const uint32_t own = ring + (uint32_t)(a * G::kSumBytes + cg * 128 * 128);
                if (ok) {
                    uint32_t v[32];
                    tmem_ld_32x32(t_addr, v);
                    if constexpr (kX3) {
                        uint32_t u[32];
                        tmem_ld_32x32(t_addr + (uint32_t)BN, u);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__fadd_rn(__uint_as_float(v[j]), __uint_as_float(u[j])));
                    } else {
                        tmem_ld_wait();
                    }
#pragma unroll
                    for (int g = 0; g < 8; ++g)
                        st_shared_v4(own + (uint32_t)(row * 128) + piece_off(row, g), make_uint4(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]));
                }
                fence_proxy_async_shared();
                __syncwarp();
                if (!ready) cluster_wait();
                ready = true;
                if (ok && sends)
                    bulk_copy_to_cta(to + (uint32_t)(((cg * parts + (a == 1 ? S - 1 : slot)) * rows + from - owner * rows) * 128),
                                     own + (uint32_t)(from * 128), (uint32_t)((upto - from) * 128), to_bar);
                __syncwarp();
            }
        }
        tc_fence_before_sync();
    }
    // Every thread: one item of 8 channels per step, its bias and residual fetched a step (or the exchange) ahead.
    constexpr int kPieces = BN / 8;
    const int box_hw = p.BH * p.BW;
    const int items = my_rows * kPieces;
    auto item_of = [&](int step) {
        Item it{};
        int idx = step * 256 + (int)threadIdx.x - 64;
        it.mine = idx < items * (kDual ? 2 : 1);
        if (!it.mine) return it;
        it.second = kDual ? idx / items : 0;
        idx -= it.second * items;
        // neighbouring threads: neighbouring channels of a pixel (NHWC) or neighbouring pixels (NCHW)
        it.piece = kOutMode == kOutNCHW_F32 ? idx / my_rows : idx % kPieces;
        it.local = kOutMode == kOutNCHW_F32 ? idx % my_rows : idx / kPieces;
        it.row = rank * rows + it.local;
        const int n_l = it.row / box_hw;
        const int rem = it.row - n_l * box_hw;
        const int h_l = rem / p.BW;
        it.n = n0 + n_l;
        it.oh = oh0 + h_l;
        it.ow = ow0 + rem - h_l * p.BW;
        it.c0 = ct * BN + it.piece * 8;
        it.mine = it.n < p.N && it.oh < p.OH && it.ow < p.OW && it.c0 < p.Cout;
        return it;
    };
    auto fetch = [&](const Item& it, Ahead<kOutMode>& a) {
        fetch_ahead<kOutMode>(p, it, kDual && it.second ? p.bias2 : p.bias, kDual && it.second ? nullptr : p.residual, a);
    };
    Item cur{};
    Ahead<kOutMode> ahead{};
    bool live = false;
    if (warp >= 2) {
        cur = item_of(0);
        fetch(cur, ahead);
        live = mbar_wait_bounded(smem_u32(&bar_recv), 0, abort_ptr);
        asm volatile("fence.acq_rel.cluster;" ::: "memory");
        live = !named_barrier_or(1, 256, !live);  // ... and the CTA's own sums are in place
    } else {
        __syncwarp();
        if constexpr (!G::kOwnBuffer) cluster_arrive();
        cluster_wait();
    }
    // Second cluster barrier: this CTA has what it waited for, or has given up. The epilogue's arithmetic and stores are not waited
    // for by the others; nobody's shared memory goes while parts are read out of it or on their way to it.
    __syncwarp();
    cluster_arrive();
    const int steps = live ? (items * (kDual ? 2 : 1) + 255) / 256 : 0;
#pragma unroll 1
    for (int step = 0; step < steps; ++step) {
        const Item next = item_of(step + 1);
        Ahead<kOutMode> next_ahead{};
        fetch(next, next_ahead);
        if (cur.mine) {
            float f[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
            const int cg = cur.piece >> 2;
            const uint32_t off0 = piece_off(cur.row, 2 * (cur.piece & 3)), off1 = piece_off(cur.row, 2 * (cur.piece & 3) + 1);
            auto add = [&](uint32_t at) {
                const uint4 x = ld_shared_v4(at + off0), y = ld_shared_v4(at + off1);
                f[0] += __uint_as_float(x.x); f[1] += __uint_as_float(x.y); f[2] += __uint_as_float(x.z); f[3] += __uint_as_float(x.w);
                f[4] += __uint_as_float(y.x); f[5] += __uint_as_float(y.y); f[6] += __uint_as_float(y.z); f[7] += __uint_as_float(y.w);
            };
            const uint32_t own = ring + (uint32_t)(cur.second * G::kSumBytes + (cg * 128 + cur.row) * 128);
            const uint32_t got = recv + (uint32_t)((cg * parts * rows + cur.local) * 128);
            if (kDual && cur.second) {
                add(rank == S - 1 ? own : got + (uint32_t)((S - 1) * rows * 128));
                epilogue8<kOutMode, false>(p, f, ahead, p.bias2 != nullptr, false, p.out2, p.relu2, cur);
            } else {
#pragma unroll 4
                for (int s = 0; s < S; ++s) add(s == rank ? own : got + (uint32_t)((s < rank ? s : s - 1) * rows * 128));
                epilogue8<kOutMode, kX3>(p, f, ahead, p.bias != nullptr, p.residual != nullptr, p.out, p.relu, cur);
            }
        }
        cur = next;
        ahead = next_ahead;
    }
    if (*abort_ptr) {  // loads already issued may still be landing (see conv_tc.cu)
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    __syncwarp();
    cluster_wait();
    if (*abort_ptr) {  // ... and so may parts that the others sent before they arrived
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    tc_fence_after_sync();
    if (warp == 1) {
        __syncwarp();
        tmem_dealloc(tmem_base, kTmemCols);
    }
    if (threadIdx.x == 0 && *abort_ptr && p.status != nullptr) atomicExch(p.status, KXC_B200_ERR_DEVICE_WAIT);
}

template <MmaKind kKind, int BN, int kOutMode, bool kDual, bool kX3>
int32_t launch_split(const TcParams& p, cudaStream_t s) {
    using G = SplitGeom<BN, kX3, kDual>;
    if (p.split > G::kMaxParts) return fail(KXC_B200_ERR_INVALID, "split-reduction conv: %d parts of %d channels", p.split, BN);
    auto kernel = conv_splitk_kernel<kKind, BN, kOutMode, kDual, kX3>;
    static PerDeviceOnce smem_once;
    KXC_TRY(smem_opt_in(smem_once, kernel, G::kSmemBytes));
    const int tiles = p.tiles_c * p.tiles_w * p.tiles_h * p.tiles_n;
    KXC_CUDA_TRY(launch_kernel(kernel, dim3((unsigned)(tiles * p.split)), dim3(kSplitThreads), G::kSmemBytes, s, /*pdl=*/true, p.split, p));
    return check_launch("conv_splitk_kernel");
}

template <MmaKind kKind, int kOutMode, bool kX3>
int32_t launch_by_width(const TcConfig& cfg, const TcParams& p, cudaStream_t s) {
    if constexpr (kKind == MmaKind::F16 && kOutMode == kOutNHWC_BF16) {
        if (cfg.dual) return launch_split<kKind, 64, kOutMode, true, false>(p, s);  // (the only width of it, tc_setup_dual)
    }
    if (cfg.dual) return fail(KXC_B200_ERR_INVALID, "split-reduction conv: no two-output form for this configuration");
    if constexpr (!kX3) {
        if (cfg.bn == 256) return launch_split<kKind, 256, kOutMode, false, kX3>(p, s);
    }
    return cfg.bn == 64 ? launch_split<kKind, 64, kOutMode, false, kX3>(p, s) : launch_split<kKind, 128, kOutMode, false, kX3>(p, s);
}

}  // namespace

int tc_split_capacity(int split) {
    if (split < 2 || split > kMaxSplit) return 0;
    static std::mutex mu;
    static int known[PerDeviceOnce::kMaxDevices][kMaxSplit + 1] = {};  // clusters + 1
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= PerDeviceOnce::kMaxDevices) return 0;
    std::lock_guard<std::mutex> lock(mu);
    int& n = known[dev][split];
    if (n == 0) {
        using G = SplitGeom<64, false>;  // every form of the kernel takes an SM to itself
        auto kernel = conv_splitk_kernel<MmaKind::F16, 64, kOutNHWC_BF16, false, false>;
        cudaLaunchConfig_t lc = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)split;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        lc.gridDim = dim3((unsigned)(kNumSMs / split * split));
        lc.blockDim = dim3(kSplitThreads);
        lc.dynamicSmemBytes = G::kSmemBytes;
        lc.attrs = attr;
        lc.numAttrs = 1;
        int found = 0;
        if (cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel), cudaFuncAttributeMaxDynamicSharedMemorySize, G::kSmemBytes) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&found, kernel, &lc) != cudaSuccess || found < 0) {
            cudaGetLastError();
            return 0;  // not kept: the next call asks again
        }
        n = (found < kNumSMs / split ? found : kNumSMs / split) + 1;
    }
    return n - 1;
}

int32_t tc_launch_split(const TcConfig& cfg, const TcParams& p, cudaStream_t s) {
    if (p.split < 2 || p.split > kMaxSplit || (cfg.bn != 64 && (cfg.dual || (cfg.bn != 128 && (cfg.bn != 256 || cfg.x3)))) || cfg.kb_bytes != kKB)
        return fail(KXC_B200_ERR_INVALID, "split-reduction conv: %d parts, %d channels, %d-byte K blocks", p.split, cfg.bn, cfg.kb_bytes);
    if (cfg.dtype == kTcBF16) {
        switch (cfg.out_mode) {
            case kOutNHWC_BF16: return launch_by_width<MmaKind::F16, kOutNHWC_BF16, false>(cfg, p, s);
            case kOutNHWC_F32: return launch_by_width<MmaKind::F16, kOutNHWC_F32, false>(cfg, p, s);
            case kOutNCHW_F32: return launch_by_width<MmaKind::F16, kOutNCHW_F32, false>(cfg, p, s);
            default: break;
        }
    } else if (cfg.dtype == kTcTF32) {
        switch (cfg.out_mode) {
            case kOutNHWC_F32:
                return cfg.x3 ? launch_by_width<MmaKind::TF32, kOutNHWC_F32, true>(cfg, p, s) : launch_by_width<MmaKind::TF32, kOutNHWC_F32, false>(cfg, p, s);
            case kOutNCHW_F32:
                return cfg.x3 ? launch_by_width<MmaKind::TF32, kOutNCHW_F32, true>(cfg, p, s) : launch_by_width<MmaKind::TF32, kOutNCHW_F32, false>(cfg, p, s);
            default: break;
        }
    }
    return fail(KXC_B200_ERR_INVALID, "split-reduction conv: output mode %d does not fit dtype %d", (int)cfg.out_mode, (int)cfg.dtype);
}

}  // namespace kxc_b200
