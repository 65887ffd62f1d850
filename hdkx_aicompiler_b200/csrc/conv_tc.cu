// Implicit-GEMM convolution / dense on tcgen05 tensor cores with TMEM accumulators and TMA operand
// loads (see conv_tc.cuh for the GEMM view). Persistent, warp-specialised CTAs, one per SM:
//
//   warp 0      TMA producer   its elected lane issues cp.async.bulk.tensor loads into a ring of swizzled
//                              shared-memory stages, each guarded by a full/empty mbarrier pair
//   warp 1      MMA issuer     its elected lane (elect_one in sm100.cuh: both loops run on the whole warp; int8 256 -> 256 3x3 at 14x14,
//                              256 images, a loop of one lane 26.4 us, so 23.1) issues tcgen05.mma (M = 128, N = BN, K = 32 bytes per
//                              instruction) into one of two TMEM accumulators; tcgen05.commit
//                              releases stages and publishes finished accumulators; owns TMEM alloc
//   warps 2..9  epilogue       tcgen05.ld the accumulator (two warps per 32-lane quadrant, each half
//                              of the columns),
//                              +bias -> +residual -> ReLU (or int8 requantize), store; overlaps the
//                              next tile's main loop through the second accumulator
//
// Every wait is bounded (sm100::mbar_wait_bounded); a wait that runs out sets the CTA's abort flag
// and the global status word, every role leaves its loop, TMEM is released and the kernel returns.
#include "conv_tc.cuh"

#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <cstdlib>
#include <mutex>

#include "common.cuh"
#include "conv_epilogue.cuh"
#include "sm100.cuh"

namespace kxc_b200 {
namespace {

using namespace sm100;

constexpr int kTcThreads = 320;  // 2 control warps + 8 epilogue warps
constexpr int kStoreBoxBytes = 32 * 128;
constexpr int kSmemLimit = 227 * 1024;

template <int KB_BYTES, int BN, int kCtas, int kMT = 1, bool kX3 = false, bool kNchw = false>
struct StageGeom {
    static constexpr int kATileBytes = 128 * KB_BYTES;
    static constexpr int kABytes = (kX3 ? 2 : kMT) * kATileBytes;  // kMT pixel tiles share one B tile; x3: high, low part
    static constexpr int kBTileBytes = (BN / kCtas) * KB_BYTES;  // a CTA of a pair holds half of the B tile's rows
    static constexpr int kBBytes = (kX3 ? 2 : 1) * kBTileBytes;
    static constexpr int kStageBytes = kABytes + kBBytes;
    // per epilogue warp a 4 KiB box (32 pixels x 64 channels, SWIZZLE_128B) that TMA stores read; its first half
    // doubles as the staging tile of the per-thread store path
    // (fp32 NHWC: all of it; into the reference's layout it holds the bias, the three-pass kernels' only use for it there)
    static constexpr int kEpilogueBytes = kX3 && kNchw ? kStoreBoxBytes : 8 * kStoreBoxBytes;
    static constexpr int kStagesRaw = (kSmemLimit - 2048 - kEpilogueBytes) / kStageBytes;
    static constexpr int kStages = kStagesRaw > 8 ? 8 : kStagesRaw;
    static constexpr int kSmemBytes = kStages * kStageBytes + kEpilogueBytes + 1024;  // + slack to align the ring to 1024 B
};

// kCtas = 2: the CTAs of a cluster of two work as a pair on 256 output pixels x BN channels. Each loads its own
// 128-pixel A tile and HALF of the B tile; the leader (cluster rank 0) issues tcgen05.mma.cta_group::2
// (M = 256), which reads both CTAs' shared memory and writes each CTA's 128 rows into that CTA's TMEM.
// Both CTAs' loads count on the leader's "full" barrier; commits arrive on both CTAs' barriers; the
// peer's epilogue warps release accumulators on the leader's "accumulator empty" barrier.
//
// kDual: a second output, the 1x1 convolution of the same stride over the same input (TcParams::tmB2 ...). Its
// reduction is appended to the K loop as `cblocks` extra stages that load the centre tap's pixels again together
// with the second weight tensor's rows and accumulate into a second TMEM accumulator; the epilogue drains both.
//
// kMT = 2: a work item is TWO pixel tiles per CTA against one B tile. Their MMAs alternate between two
// accumulators, which gives the tensor core two independent accumulate chains (a pair's M = 256 instruction has
// a long dependent-issue latency) and halves the B traffic per pixel.
//
// kX3 (three-pass tf32): every stage carries the high and low parts of both operands, so a tap's pixels and weights cross
// L2 -> shared memory twice instead of three times and no partial sum leaves the chip. The B tile is [w_hi; w_lo] (2 BN
// rows): ONE instruction of N = 2 BN multiplies a_hi with both and fills the accumulators hi*hi | hi*lo side by side, a
// second of N = BN adds a_lo * w_hi to the latter. The two sums meet in one rounded fp32 add in the epilogue. A stage of four K steps
// is 448 cycles of the tensor pipe with 64 channels (64 + 48 a step) and 768 with 128, but takes 850 and 1150: what crosses shared
// memory, 56 or 80 KB of operands that the instructions read and 48 or 64 KB of copies, does so at 125 to 128 bytes a cycle.
// Pairs (64 channels): 44 and 40 KB a stage and CTA, whose half of the B tile is [w_hi; w_lo] of 32 channels. The wide instruction then
// gives hi*hi | hi*lo of either half, so lo*hi has columns of its own and the epilogue adds three sums. 680 to 790 cycles a stage: ResNet-18's layers, us,
// 32 images 28x28 45.3 -> 40.0 (128 channels a tile before), 56x56 50.5 -> 47.5, 64 images 14x14 81 -> 73; whole networks 32: 873 -> 841, 48: 1260 -> 1204.
template <MmaKind kKind, int KB_BYTES, int BN, int kOutMode, int kCtas, bool kDual = false, int kMT = 1, bool kX3 = false>
__global__ void __launch_bounds__(kTcThreads, 1) conv_igemm_kernel(const __grid_constant__ TcParams p) {
    using G = StageGeom<KB_BYTES, BN, kCtas, kMT, kX3, kOutMode == kOutNCHW_F32>;
    static_assert(!(kDual && kMT != 1), "the two-output kernel works on one pixel tile at a time");
    static_assert(!kX3 || (kKind == MmaKind::TF32 && !kDual && kMT == 1 && BN <= 128 / kCtas), "three-pass form: tf32, one pixel tile, pairs of 64 channels");
    constexpr bool kPair = kCtas == 2;
    constexpr int kStages = G::kStages;
    constexpr int kAccCols = (kX3 && kPair ? 3 : (kDual || kX3 ? 2 : kMT)) * BN;  // TMEM columns of one accumulator buffer
    // two accumulator buffers (the epilogue of one work item overlaps the next item's main loop) where TMEM's 512
    // columns allow it, else one
    constexpr int kBufs = 2 * kAccCols <= 512 ? 2 : 1;
    constexpr uint32_t kTmemUsed = kBufs * kAccCols;
    constexpr uint32_t kTmemCols = kTmemUsed <= 128 ? 128u : (kTmemUsed <= 256 ? 256u : 512u);  // allocations are powers of two
    static_assert(kTmemUsed <= 512, "TMEM has 512 columns");
    static_assert(!kDual || (!kPair && kOutMode == kOutNHWC_BF16), "the dual kernel exists for single CTAs and bf16 NHWC output");
    constexpr uint32_t kIdesc =
        make_instr_desc(kKind == MmaKind::F16 ? kFmtBF16 : (kKind == MmaKind::TF32 ? kFmtTF32 : kFmtS8),
                        kKind == MmaKind::I8 ? kAccS32 : kAccF32, BN, 128u * kCtas);
    [[maybe_unused]] constexpr uint32_t kIdescWide = make_instr_desc(kFmtTF32, kAccF32, 2 * BN <= 256 ? 2 * BN : 256, 128u * kCtas);  // x3: [w_hi; w_lo]

    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bar_full[kStages];
    __shared__ __align__(8) uint64_t bar_empty[kStages];
    __shared__ __align__(8) uint64_t bar_acc_full[2];
    __shared__ __align__(8) uint64_t bar_acc_empty[2];
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;
    [[maybe_unused]] __shared__ int requant_ok;

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);  // (a uniform value, as the compiler then knows)
    const int lane = threadIdx.x & 31;
    const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t cta_rank = kPair ? cluster_cta_rank() : 0u;
    const bool leader = cta_rank == 0;

    if (threadIdx.x == 0) {
        abort_flag = 0;
        if constexpr (kKind == MmaKind::I8) requant_ok = 1;
        for (int s = 0; s < kStages; ++s) {
            mbar_init(smem_u32(&bar_full[s]), 1);
            mbar_init(smem_u32(&bar_empty[s]), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(smem_u32(&bar_acc_full[a]), 1);
            mbar_init(smem_u32(&bar_acc_empty[a]), 8 * kCtas);  // one arrival per epilogue warp (of both CTAs)
        }
        mbar_fence_init();
    }
    if (warp == 1) {
        if constexpr (kPair) {
            tmem_alloc_pair(smem_u32(&tmem_base_slot), kTmemCols);
            tmem_relinquish_pair();
        } else {
            tmem_alloc(smem_u32(&tmem_base_slot), kTmemCols);
            tmem_relinquish();
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if constexpr (kPair) cluster_sync_all();  // the peer's barriers are initialised before anything signals them
    tc_fence_after_sync();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_base_slot, 0);
    volatile int* abort_ptr = &abort_flag;
    auto wait = [&](uint64_t* bar, uint32_t phase) { return mbar_wait_warp(smem_u32(bar), phase, abort_ptr); };
    pdl_launch_dependents();  // the next kernel's CTAs may take over SMs this grid has left; they wait before touching memory

    const int num_kb_main = p.taps_h * p.taps_w * p.cblocks;
    const int num_kb = num_kb_main + (kDual ? p.cblocks : 0);
    // Work items: (channel tile, group of kCtas consecutive pixel tiles). A pair whose second pixel tile
    // does not exist loads a box beyond the last image (all zeros) and stores nothing for it.
    const int m_tiles = p.tiles_w * p.tiles_h * p.tiles_n;
    const int total_tiles = p.tiles_c * ((m_tiles + kCtas * kMT - 1) / (kCtas * kMT));
    const int first_tile = kPair ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
    const int tile_step = kPair ? (int)(gridDim.x >> 1) : (int)gridDim.x;
    const int rows_used = p.BW * p.BH * p.BNI;

    if (warp == 0) {
        // ------------------------------ TMA producer ------------------------------
        const bool lead = elect_one();
        if (lead) {
            tma_prefetch_desc(&p.tmB);
            tma_prefetch_desc(&p.tmA[0]);
            if constexpr (kDual || kX3) tma_prefetch_desc(&p.tmB2);
        }
        const uint32_t tx_bytes = (uint32_t)((kX3 ? 2 : kMT) * rows_used * KB_BYTES + G::kBBytes);
        pdl_wait();  // the activations come from the previous kernel
        int stage = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (int item = first_tile; ok && item < total_tiles; item += tile_step) {
            const int tile = p.reverse ? total_tiles - 1 - item : item;
            const int ct = tile % p.tiles_c;
            int ow0[kMT], oh0[kMT], n0[kMT];
#pragma unroll
            for (int t = 0; t < kMT; ++t) {
                int r = ((tile / p.tiles_c) * kCtas + (int)cta_rank) * kMT + t;
                const int tw = r % p.tiles_w; r /= p.tiles_w;
                const int th = r % p.tiles_h;
                const int tn = r / p.tiles_h;
                ow0[t] = tw * p.BW; oh0[t] = th * p.BH; n0[t] = tn * p.BNI;
            }
            const int co0 = ct * BN + (int)cta_rank * (BN / kCtas);
            int kb = 0;
            for (int kh = 0; ok && kh < p.taps_h; ++kh) {
                for (int kw = 0; ok && kw < p.taps_w; ++kw) {
                    const int dh = kh * p.dil_h - p.pad_h;
                    const int dw = kw * p.dil_w - p.pad_w;
                    int map = 0, ch = dh, cw = dw;  // offsets of this tap's box from the tile's first pixel
                    if (p.stride == 2) {
                        const int hp = dh & 1, wp = dw & 1;
                        map = hp * 2 + wp;
                        ch = (dh - hp) >> 1;
                        cw = (dw - wp) >> 1;
                    }
                    for (int cb = 0; cb < p.cblocks; ++cb, ++kb) {
                        if (!wait(&bar_empty[stage], phase ^ 1u)) {
                            ok = false;
                            break;
                        }
                        const uint32_t full = smem_u32(&bar_full[stage]);
                        const uint32_t a_dst = ring + (uint32_t)stage * G::kStageBytes;
                        if (!lead) {
                        } else if constexpr (kPair) {
                            if (leader) mbar_arrive_expect_tx(full, 2u * tx_bytes);
                            const uint32_t full0 = map_to_cta(full, 0);
#pragma unroll
                            for (int t = 0; t < kMT; ++t)
                                tma_load_4d_pair(a_dst + t * G::kATileBytes, &p.tmA[map], full0, cb * p.kb_elems, ow0[t] + cw,
                                                 oh0[t] + ch, n0[t]);
                            if constexpr (kX3)
                                tma_load_4d_pair(a_dst + G::kATileBytes, &p.tmA[map], full0, cb * p.kb_elems, ow0[0] + cw, oh0[0] + ch, n0[0] + p.N);
                            tma_load_2d_pair(a_dst + G::kABytes, &p.tmB, full0, kb * p.kb_elems, co0);
                            if constexpr (kX3) tma_load_2d_pair(a_dst + G::kABytes + G::kBTileBytes, &p.tmB2, full0, kb * p.kb_elems, co0);
                        } else {
                            mbar_arrive_expect_tx(full, tx_bytes);
#pragma unroll
                            for (int t = 0; t < kMT; ++t)
                                tma_load_4d(a_dst + t * G::kATileBytes, &p.tmA[map], full, cb * p.kb_elems, ow0[t] + cw, oh0[t] + ch,
                                            n0[t]);
                            tma_load_2d(a_dst + G::kABytes, &p.tmB, full, kb * p.kb_elems, co0);
                            if constexpr (kX3) {
                                tma_load_4d(a_dst + G::kATileBytes, &p.tmA[map], full, cb * p.kb_elems, ow0[0] + cw, oh0[0] + ch,
                                            n0[0] + p.N);
                                tma_load_2d(a_dst + G::kABytes + G::kBTileBytes, &p.tmB2, full, kb * p.kb_elems, co0);
                            }
                        }
                        __syncwarp();
                        if (++stage == kStages) { stage = 0; phase ^= 1u; }
                    }
                }
            }
            if constexpr (kDual) {
                // second output: the centre tap's pixels (the 1x1 convolution's only tap) against tmB2
                const int dh = (p.taps_h / 2) * p.dil_h - p.pad_h, dw = (p.taps_w / 2) * p.dil_w - p.pad_w;  // 0, 0
                int map = 0, ch = oh0[0] + dh, cw = ow0[0] + dw;
                if (p.stride == 2) {
                    const int hp = dh & 1, wp = dw & 1;
                    map = hp * 2 + wp;
                    ch = oh0[0] + ((dh - hp) >> 1);
                    cw = ow0[0] + ((dw - wp) >> 1);
                }
                for (int cb = 0; ok && cb < p.cblocks; ++cb) {
                    if (!wait(&bar_empty[stage], phase ^ 1u)) {
                        ok = false;
                        break;
                    }
                    const uint32_t full = smem_u32(&bar_full[stage]);
                    const uint32_t a_dst = ring + (uint32_t)stage * G::kStageBytes;
                    if (lead) {
                        mbar_arrive_expect_tx(full, tx_bytes);
                        tma_load_4d(a_dst, &p.tmA[map], full, cb * p.kb_elems, cw, ch, n0[0]);
                        tma_load_2d(a_dst + G::kABytes, &p.tmB2, full, cb * p.kb_elems, co0);
                    }
                    __syncwarp();
                    if (++stage == kStages) { stage = 0; phase ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------ MMA issuer ------------------------------
        if (leader) {
            const bool lead = elect_one();
            int stage = 0;
            uint32_t phase = 0;
            int acc = 0;
            uint32_t acc_phase = 0;
            bool ok = true;
            for (int tile = first_tile; ok && tile < total_tiles; tile += tile_step) {
                if (!wait(&bar_acc_empty[acc], acc_phase ^ 1u)) break;
                tc_fence_after_sync();
                const uint32_t d_main = tmem_base + (uint32_t)(acc * kAccCols);
                for (int kb = 0; kb < num_kb; ++kb) {
                    const bool second = kDual && kb >= num_kb_main;
                    const uint32_t d_tmem = second ? d_main + (uint32_t)BN : d_main;
                    const int kb_local = second ? kb - num_kb_main : kb;
                    if (!wait(&bar_full[stage], phase)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    const uint32_t a_addr = ring + (uint32_t)stage * G::kStageBytes;
                    const uint64_t a_desc = make_smem_desc(a_addr, KB_BYTES);
                    const uint64_t b_desc = make_smem_desc(a_addr + G::kABytes, KB_BYTES);
                    if (lead) {
#pragma unroll
                        for (int k = 0; k < KB_BYTES / 32; ++k) {
                            if constexpr (kX3) {
                                const uint64_t a_k = a_desc + (uint64_t)(2 * k), b_k = b_desc + (uint64_t)(2 * k), a_lo = a_k + (uint64_t)(G::kATileBytes >> 4);
                                if constexpr (kPair) {
                                    umma_pair<kKind>(d_tmem, a_k, b_k, kIdescWide, (kb_local | k) != 0 ? 1u : 0u);
                                    umma_pair<kKind>(d_tmem + (uint32_t)(2 * BN), a_lo, b_k, kIdesc, (kb_local | k) != 0 ? 1u : 0u);
                                } else {
                                    umma<kKind>(d_tmem, a_k, b_k, kIdescWide, (kb_local | k) != 0 ? 1u : 0u);
                                    umma<kKind>(d_tmem + (uint32_t)BN, a_lo, b_k, kIdesc, 1u);
                                }
                            } else {
#pragma unroll
                                for (int t = 0; t < kMT; ++t) {
                                    // advancing 32 bytes along K inside the swizzle span = +2 in the (addr >> 4) field;
                                    // the next pixel tile of the stage is kATileBytes further on
                                    const uint64_t a_k = a_desc + (uint64_t)(2 * k) + (uint64_t)(t * (G::kATileBytes >> 4));
                                    const uint32_t d_t = d_tmem + (uint32_t)(t * BN);
                                    if constexpr (kPair)
                                        umma_pair<kKind>(d_t, a_k, b_desc + (uint64_t)(2 * k), kIdesc, (kb_local | k) != 0 ? 1u : 0u);
                                    else
                                        umma<kKind>(d_t, a_k, b_desc + (uint64_t)(2 * k), kIdesc, (kb_local | k) != 0 ? 1u : 0u);
                                }
                            }
                        }
                        if constexpr (kPair) umma_commit_pair(smem_u32(&bar_empty[stage]), 3);
                        else umma_commit(smem_u32(&bar_empty[stage]));
                    }
                    __syncwarp();
                    if (++stage == kStages) { stage = 0; phase ^= 1u; }
                }
                if (!ok) break;
                if (lead) {
                    if constexpr (kPair) umma_commit_pair(smem_u32(&bar_acc_full[acc]), 3);
                    else umma_commit(smem_u32(&bar_acc_full[acc]));
                }
                __syncwarp();
                if (++acc == kBufs) {
                    acc = 0;
                    acc_phase ^= 1u;
                }
            }
        }
    } else {
        // ------------------------------ epilogue ------------------------------
        const int quad = warp & 3;  // TMEM lanes [32*quad, 32*quad+32) are the ones this warp may read
        const int half = (warp - 2) >> 2;  // which half of the tile's columns this warp handles
        constexpr int kChunksPerWarp = BN / 64;
        const int row = quad * 32 + lane;
        const int box_hw = p.BH * p.BW;
        const int n_l = row / box_hw;
        const int rem = row - n_l * box_hw;
        const int h_l = rem / p.BW;
        const int w_l = rem - h_l * p.BW;
        const bool fast = (kOutMode == kOutNHWC_BF16) && p.vec_ok && ((p.Cout & 31) == 0);
        const bool wide = kOutMode == kOutNHWC_F32 && p.vec_ok && (p.Cout & 3) == 0;  // fp32 NHWC in 16-byte pieces
        const bool has_res = p.residual != nullptr;
        const EpiParams ep = {p.bias, p.residual, p.out, p.Cout, p.relu};
        const uint32_t stage_tile = ring + (uint32_t)(kStages * G::kStageBytes) + (uint32_t)((warp - 2) * kStoreBoxBytes);
        // Residual-free launches with store maps: the warp's values go into its swizzled box and leave by TMA store
        // (boxes are 64 channels wide: a warp needs an even number of 32-column chunks, which the 192-wide tile lacks)
        const bool boxed = fast && p.store_box && !has_res && (BN >= 128) && (kChunksPerWarp % 2 == 0);
        pdl_wait();  // residual reads and output writes must not overtake earlier kernels
        // int8: the per-channel constants of the high-word requantize, prepared once per CTA in shared memory (the store boxes
        // are not used by this type) instead of three loads, a shift and a select per value of every chunk. One channel whose
        // shift or bias the short formula does not cover, or more channels than fit, and all chunks take the general one.
        // (256 -> 256 channels, 14x14, 256 images: 31 -> 28 us)
        [[maybe_unused]] const int4* q_tab = nullptr;
        if constexpr (kKind == MmaKind::I8) {
            const int padded = p.tiles_c * BN;
            int4* tab = reinterpret_cast<int4*>(smem_raw + (ring - smem_u32(smem_raw)) + kStages * G::kStageBytes);
            const int64_t max_abs_acc = 128ll * 128 * p.taps_h * p.taps_w * p.cblocks * p.kb_elems;
            if (padded * (int)sizeof(int4) <= G::kEpilogueBytes && max_abs_acc < (1ll << 31)) {
                for (int c = (int)threadIdx.x - 64; c < padded; c += 256) {
                    if (c >= p.Cout) tab[c] = make_int4(0, 0, 0, 0);
                    else if (!requant_prepare(__ldg(p.bias_i32 + c), __ldg(p.multiplier + c), __ldg(p.shift + c), max_abs_acc, &tab[c])) requant_ok = 0;
                }
                named_barrier(1, 256);
                if (*(volatile int*)&requant_ok) q_tab = tab;
            }
        }
        // The reference's layout: the bias in shared memory (the store boxes are not used here either), padded to whole tiles
        [[maybe_unused]] const uint32_t bias_tab = ring + (uint32_t)(kStages * G::kStageBytes);
        [[maybe_unused]] bool small_nchw = false;  // nchw_store32's conditions
        if constexpr (kOutMode == kOutNCHW_F32) {
            const int padded = p.tiles_c * BN;
            small_nchw = padded * 4 <= G::kEpilogueBytes && (unsigned long long)p.N * p.Cout * p.OH * p.OW < (1ull << 30);
            if (small_nchw) {
                float* tab = reinterpret_cast<float*>(smem_raw + (bias_tab - smem_u32(smem_raw)));
                for (int c = (int)threadIdx.x - 64; c < padded; c += 256) tab[c] = p.bias != nullptr && c < p.Cout ? __ldg(p.bias + c) : 0.0f;
                named_barrier(1, 256);
            }
        }
        int acc = 0;
        uint32_t acc_phase = 0;
        bool alive = true;
        for (int item = first_tile; alive && item < total_tiles; item += tile_step) {
          const int tile = p.reverse ? total_tiles - 1 - item : item;
          const int ct = tile % p.tiles_c;
#pragma unroll 1
          for (int t = 0; t < kMT; ++t) {
            int r = ((tile / p.tiles_c) * kCtas + (int)cta_rank) * kMT + t;
            const int tw = r % p.tiles_w; r /= p.tiles_w;
            const int th = r % p.tiles_h;
            const int tn = r / p.tiles_h;
            const int n = tn * p.BNI + n_l, oh = th * p.BH + h_l, ow = tw * p.BW + w_l;
            const bool valid = (row < rows_used) && (n < p.N) && (oh < p.OH) && (ow < p.OW);
            const size_t pix = ((size_t)n * p.OH + oh) * p.OW + ow;
            const int col0 = half * kChunksPerWarp * 32;  // first column of this warp inside the tile
            const int c_base = ct * BN + col0;
            uint4 res_cur[4] = {};
            float nchw_cur[32] = {}, nchw_next[32] = {};  // kOutNCHW_F32 only
            [[maybe_unused]] const uint32_t nchw_step = (uint32_t)(p.OH * p.OW) * 4u;
            [[maybe_unused]] const uint32_t nchw_off = small_nchw ? (uint32_t)(n * p.Cout + c_base) * nchw_step + (uint32_t)(oh * p.OW + ow) * 4u : 0u;
            if constexpr (kOutMode == kOutNCHW_F32) {
                if (has_res && c_base < p.Cout) {
                    if (!small_nchw) residual_fetch_nchw(p, c_base, valid, n, oh, ow, nchw_cur);
                    else if (valid) nchw_fetch32(static_cast<const char*>(p.residual), nchw_off, nchw_step, p.Cout - c_base, nchw_cur);
                    __syncwarp();  // (lanes beyond the image's edge skipped the loads; the reads of tensor memory want the whole warp)
                }
            }
            [[maybe_unused]] size_t at32[8];  // kOutNHWC_F32 only
            [[maybe_unused]] uint4 res32[8] = {}, next32[8] = {};
            if constexpr (kOutMode == kOutNHWC_F32) {
                if (wide) {
                    make_row_map_f32(pix, valid, p.Cout, lane, at32);
                    if (has_res && c_base < p.Cout) residual_fetch_rows_f32(p, at32, c_base, lane, res32);
                }
            }
            RowMap rows;
            if (fast && !boxed) {
                rows = make_row_map(pix, valid, lane);
                if (has_res && c_base < p.Cout) residual_fetch_rows(ep, rows, c_base, lane, res_cur);
            }
            if (t == 0) {
                bool ok = mbar_wait_bounded(smem_u32(&bar_acc_full[acc]), acc_phase, abort_ptr);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) {
                    alive = false;
                    break;
                }
                tc_fence_after_sync();
            }
            // (x3 pairs: of either half of the channels hi*hi and hi*lo, then lo*hi of all)
            const uint32_t t_addr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(acc * kAccCols + t * BN + col0 + (kX3 && kPair ? half * (BN / 2) : 0));
            [[maybe_unused]] const uint32_t u_addr = t_addr + (uint32_t)(kPair ? BN / 2 : BN), w_addr = t_addr + (uint32_t)(2 * BN - half * (BN / 2));
            if (kOutMode == kOutNCHW_F32 && small_nchw) {
                if constexpr (kOutMode == kOutNCHW_F32) {
                    // unrolled: the two chunks of residual values in flight then need not be moved
#pragma unroll
                    for (int i = 0; i < kChunksPerWarp; ++i) {
                        const int c0 = c_base + i * 32;
                        if (c0 >= p.Cout) break;
                        uint32_t v[32];
                        tmem_ld_32x32(t_addr + (uint32_t)(i * 32), v);
                        float(&res)[32] = i & 1 ? nchw_next : nchw_cur;
                        float(&res_ahead)[32] = i & 1 ? nchw_cur : nchw_next;
                        if (has_res && valid && i + 1 < kChunksPerWarp && c0 + 32 < p.Cout)
                            nchw_fetch32(static_cast<const char*>(p.residual), nchw_off + (uint32_t)(i + 1) * 32u * nchw_step, nchw_step, p.Cout - c0 - 32, res_ahead);
                        __syncwarp();
                        if constexpr (kX3) {
                            uint32_t u[32];
                            tmem_ld_32x32(u_addr + (uint32_t)(i * 32), u);
                            if constexpr (kPair) {
                                uint32_t w[32];
                                tmem_ld_32x32(w_addr + (uint32_t)(i * 32), w);
                                tmem_ld_wait();
#pragma unroll
                                for (int j = 0; j < 32; ++j) u[j] = __float_as_uint(__fadd_rn(__uint_as_float(u[j]), __uint_as_float(w[j])));
                            }
                            tmem_ld_wait();
#pragma unroll
                            for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__fadd_rn(__uint_as_float(v[j]), __uint_as_float(u[j])));
                        }
                        tmem_ld_wait();
                        if (valid)
                            nchw_store32(static_cast<char*>(p.out), nchw_off + (uint32_t)i * 32u * nchw_step, nchw_step, p.Cout - c0, v,
                                         bias_tab + (uint32_t)c0 * 4u, p.bias != nullptr, res, has_res, p.relu != 0);
                        __syncwarp();
                    }
                }
            } else
#pragma unroll 1
            for (int i = 0; i < kChunksPerWarp; ++i) {
                const int c0 = c_base + i * 32;
                uint32_t v[32];
                tmem_ld_32x32(t_addr + (uint32_t)(i * 32), v);
                uint4 res_next[4] = {};
                if (fast && has_res && (i + 1 < kChunksPerWarp) && (c0 + 32 < p.Cout))
                    residual_fetch_rows(ep, rows, c0 + 32, lane, res_next);
                if constexpr (kOutMode == kOutNHWC_F32) {
                    if (wide && has_res && i + 1 < kChunksPerWarp && c0 + 32 < p.Cout) residual_fetch_rows_f32(p, at32, c0 + 32, lane, next32);
                }
                if constexpr (kOutMode == kOutNCHW_F32) {
                    if (has_res && i + 1 < kChunksPerWarp && c0 + 32 < p.Cout) residual_fetch_nchw(p, c0 + 32, valid, n, oh, ow, nchw_next);
                }
                if constexpr (kX3) {
                    uint32_t u[32];
                    tmem_ld_32x32(u_addr + (uint32_t)(i * 32), u);
                    if constexpr (kPair) {
                        uint32_t w[32];
                        tmem_ld_32x32(w_addr + (uint32_t)(i * 32), w);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 32; ++j) u[j] = __float_as_uint(__fadd_rn(__uint_as_float(u[j]), __uint_as_float(w[j])));
                    }
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__fadd_rn(__uint_as_float(v[j]), __uint_as_float(u[j])));
                }
                tmem_ld_wait();
                if (boxed) {
                    if ((i & 1) == 0) {  // a new 64-channel group: the previous store must have read the box
                        if (lane == 0) bulk_wait_group_read<0>();
                        __syncwarp();
                    }
                    if (c0 < p.Cout) epilogue_box_bf16(ep, v, c0, stage_tile, (i & 1) * 4, lane);
                    if (i & 1) {
                        fence_proxy_async_shared();
                        __syncwarp();
                        // lane 0's pixel is the first of the warp's 32: the box origin (a pair's missing second tile
                        // lies beyond the last image and stores nothing)
                        if (lane == 0 && c0 < p.Cout && n < p.N) {
                            tma_store_4d(&p.tmOut, stage_tile, c0 - 32, ow, oh, n);
                            bulk_commit_group();
                        }
                    }
                } else if (fast) {
                    if (c0 < p.Cout) epilogue_coalesced_bf16<32>(ep, v, c0, stage_tile, lane, rows, res_cur, has_res);
                } else if (wide) {
                    if constexpr (kOutMode == kOutNHWC_F32) {
                        if (c0 < p.Cout) epilogue_coalesced_f32<kX3>(p, v, c0, stage_tile, lane, at32, res32, has_res);
                    }
                } else if (kKind == MmaKind::I8 && q_tab != nullptr) {
                    if constexpr (kKind == MmaKind::I8) {
                        if (valid && c0 < p.Cout) {
                            const int32_t lo_cap = p.relu ? 0 : INT32_MIN;
                            uint32_t qw[8];
#pragma unroll
                            for (int j = 0; j < 32; j += 4) {
                                const uint32_t vv[4] = {v[j], v[j + 1], v[j + 2], v[j + 3]};
                                const int4 qq[4] = {q_tab[c0 + j], q_tab[c0 + j + 1], q_tab[c0 + j + 2], q_tab[c0 + j + 3]};
                                qw[j >> 2] = requant4_prepared(vv, qq, lo_cap);
                            }
                            store_chunk_s8<kOutMode>(p, qw, c0, p.Cout - c0 < 32 ? p.Cout - c0 : 32, n, oh, ow);
                        }
                    }
                } else {
                    epilogue_chunk<kOutMode, kX3>(p, v, c0, valid, n, oh, ow, nchw_cur);
                }
#pragma unroll
                for (int g = 0; g < 4; ++g) res_cur[g] = res_next[g];
                if constexpr (kOutMode == kOutNHWC_F32) {
#pragma unroll
                    for (int g = 0; g < 8; ++g) res32[g] = next32[g];
                }
                if constexpr (kOutMode == kOutNCHW_F32) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) nchw_cur[j] = nchw_next[j];
                }
            }
            if constexpr (kDual) {
                // second output: same rows and channels from the accumulator next to the main one; no residual
                const EpiParams ep2 = {p.bias2, nullptr, p.out2, p.Cout, p.relu2};
                const uint4 none[4] = {};
#pragma unroll 1
                for (int i = 0; i < kChunksPerWarp; ++i) {
                    const int c0 = c_base + i * 32;
                    uint32_t v[32];
                    tmem_ld_32x32(t_addr + (uint32_t)(BN + i * 32), v);
                    tmem_ld_wait();
                    if (boxed) {
                        if ((i & 1) == 0) {
                            if (lane == 0) bulk_wait_group_read<0>();
                            __syncwarp();
                        }
                        if (c0 < p.Cout) epilogue_box_bf16(ep2, v, c0, stage_tile, (i & 1) * 4, lane);
                        if (i & 1) {
                            fence_proxy_async_shared();
                            __syncwarp();
                            if (lane == 0 && c0 < p.Cout && n < p.N) {
                                tma_store_4d(&p.tmOut2, stage_tile, c0 - 32, ow, oh, n);
                                bulk_commit_group();
                            }
                        }
                    } else if (c0 < p.Cout) {
                        epilogue_coalesced_bf16<32>(ep2, v, c0, stage_tile, lane, rows, none, false);
                    }
                }
            }
          }  // pixel tiles of the work item
            if (!alive) break;
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                if constexpr (kPair) mbar_arrive_cluster(map_to_cta(smem_u32(&bar_acc_empty[acc]), 0));
                else mbar_arrive(smem_u32(&bar_acc_empty[acc]));
            }
            if (++acc == kBufs) {
                acc = 0;
                acc_phase ^= 1u;
            }
        }
        if (boxed && lane == 0) bulk_wait_group_all();  // the stores have read shared memory and written the output
    }

    // ------------------------------ teardown ------------------------------
    if (*abort_ptr) {
        // Loads that were already issued may still be landing in shared memory: give them time
        // (bounded) before the CTA's shared memory is released.
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    tc_fence_before_sync();
    __syncthreads();
    // Neither CTA of a pair may release its TMEM or shared memory while the other can still signal or read it.
    if constexpr (kPair) cluster_sync_all();
    tc_fence_after_sync();
    if (warp == 1) {
        __syncwarp();
        if constexpr (kPair) tmem_dealloc_pair(tmem_base, kTmemCols);
        else tmem_dealloc(tmem_base, kTmemCols);
    }
    if (threadIdx.x == 0 && *abort_ptr && p.status != nullptr) atomicExch(p.status, KXC_B200_ERR_DEVICE_WAIT);
}

template <MmaKind kKind, int KB_BYTES, int BN, int kOutMode, int kCtas, bool kDual = false, int kMT = 1, bool kX3 = false>
int32_t launch_one(const TcParams& p, cudaStream_t stream) {
    using G = StageGeom<KB_BYTES, BN, kCtas, kMT, kX3, kOutMode == kOutNCHW_F32>;
    auto kernel = conv_igemm_kernel<kKind, KB_BYTES, BN, kOutMode, kCtas, kDual, kMT, kX3>;
    static PerDeviceOnce smem_once;
    static std::mutex units_mu;
    static int max_units[PerDeviceOnce::kMaxDevices] = {0};  // per device: clusters of two (kCtas = 2) resident at once
    int dev = 0;
    KXC_TRY(smem_opt_in(smem_once, kernel, G::kSmemBytes, &dev));
    const long long m_tiles = (long long)p.tiles_w * p.tiles_h * p.tiles_n;
    const long long tiles = (long long)p.tiles_c * ((m_tiles + kCtas * kMT - 1) / (kCtas * kMT));
    if (tiles <= 0) return KXC_B200_OK;
    int units = kNumSMs;
    if constexpr (kCtas == 2) {
        std::lock_guard<std::mutex> lock(units_mu);
        if (max_units[dev] == 0) {
            cudaLaunchConfig_t lc = {};
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = 2;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            lc.gridDim = dim3(kNumSMs);
            lc.blockDim = dim3(kTcThreads);
            lc.dynamicSmemBytes = G::kSmemBytes;
            lc.attrs = attr;
            lc.numAttrs = 1;
            int n = 0;
            const cudaError_t e = cudaOccupancyMaxActiveClusters(&n, kernel, &lc);
            if (e != cudaSuccess || n <= 0)
                return fail(KXC_B200_ERR_CUDA, "cudaOccupancyMaxActiveClusters: %s (%d clusters)", cudaGetErrorString(e), n);
            max_units[dev] = n < kNumSMs / 2 ? n : kNumSMs / 2;
        }
        units = max_units[dev];
    }
    const int grid = kCtas * (int)(tiles < units ? tiles : units);
    KXC_CUDA_TRY(launch_kernel(kernel, dim3(grid), dim3(kTcThreads), G::kSmemBytes, stream, /*pdl=*/true, kCtas, p));
    return check_launch("conv_igemm_kernel");
}

template <MmaKind kKind, int KB_BYTES, int BN, int kCtas>
int32_t launch_by_out(const TcConfig& cfg, const TcParams& p, cudaStream_t s) {
    if constexpr (kKind == MmaKind::I8) {
        switch (cfg.out_mode) {
            case kOutNHWC_S8: return launch_one<kKind, KB_BYTES, BN, kOutNHWC_S8, kCtas>(p, s);
            case kOutNCHW_S8: return launch_one<kKind, KB_BYTES, BN, kOutNCHW_S8, kCtas>(p, s);
            default: break;
        }
    } else {
        switch (cfg.out_mode) {
            case kOutNHWC_BF16: return launch_one<kKind, KB_BYTES, BN, kOutNHWC_BF16, kCtas>(p, s);
            case kOutNHWC_F32: return launch_one<kKind, KB_BYTES, BN, kOutNHWC_F32, kCtas>(p, s);
            case kOutNCHW_F32: return launch_one<kKind, KB_BYTES, BN, kOutNCHW_F32, kCtas>(p, s);
            default: break;
        }
    }
    return fail(KXC_B200_ERR_INVALID, "tensor-core conv: output mode %d does not fit dtype %d", (int)cfg.out_mode, (int)cfg.dtype);
}

template <int KB_BYTES, int BN, int kCtas>
int32_t launch_x3(const TcConfig& cfg, const TcParams& p, cudaStream_t s) {
    switch (cfg.out_mode) {
        case kOutNHWC_F32: return launch_one<MmaKind::TF32, KB_BYTES, BN, kOutNHWC_F32, kCtas, false, 1, true>(p, s);
        case kOutNCHW_F32: return launch_one<MmaKind::TF32, KB_BYTES, BN, kOutNCHW_F32, kCtas, false, 1, true>(p, s);
        default: return fail(KXC_B200_ERR_INVALID, "tensor-core conv: output mode %d has no three-pass form", (int)cfg.out_mode);
    }
}

template <MmaKind kKind, int KB_BYTES>
int32_t launch_by_bn(const TcConfig& cfg, const TcParams& p, cudaStream_t s) {
    if (cfg.x3) {
        if constexpr (kKind == MmaKind::TF32) {
            if constexpr (KB_BYTES == 128) {
                if (cfg.ctas == 2 && cfg.mt == 1 && !cfg.dual && cfg.bn == 64) return launch_x3<KB_BYTES, 64, 2>(cfg, p, s);
            }
            if (cfg.ctas == 1 && cfg.mt == 1 && !cfg.dual && (cfg.bn == 64 || cfg.bn == 128))
                return cfg.bn == 64 ? launch_x3<KB_BYTES, 64, 1>(cfg, p, s) : launch_x3<KB_BYTES, 128, 1>(cfg, p, s);
        }
        return fail(KXC_B200_ERR_INVALID, "tensor-core conv: no three-pass kernel for this configuration");
    }
    if constexpr (KB_BYTES == 128 && kKind == MmaKind::F16) {
        if (cfg.dual) {
            if ((cfg.bn != 128 && cfg.bn != 192) || cfg.ctas != 1 || cfg.out_mode != kOutNHWC_BF16 || !p.vec_ok || (p.Cout & 31) != 0)
                return fail(KXC_B200_ERR_INVALID, "tensor-core conv: the two-output kernel needs a 128- or 192-wide tile, bf16 NHWC output and aligned pointers");
            return cfg.bn == 192 ? launch_one<kKind, KB_BYTES, 192, kOutNHWC_BF16, 1, true>(p, s)
                                 : launch_one<kKind, KB_BYTES, 128, kOutNHWC_BF16, 1, true>(p, s);
        }
    }
    if (cfg.dual) return fail(KXC_B200_ERR_INVALID, "tensor-core conv: no two-output kernel for this configuration");
    if constexpr (KB_BYTES == 128 && kKind == MmaKind::F16) {
        if (cfg.mt == 2) {
            if (cfg.bn != 128 || cfg.out_mode != kOutNHWC_BF16)
                return fail(KXC_B200_ERR_INVALID, "tensor-core conv: two pixel tiles per work item exist for the 128-wide bf16 NHWC kernel");
            return cfg.ctas == 2 ? launch_one<kKind, KB_BYTES, 128, kOutNHWC_BF16, 2, false, 2>(p, s)
                                 : launch_one<kKind, KB_BYTES, 128, kOutNHWC_BF16, 1, false, 2>(p, s);
        }
    }
    if constexpr (KB_BYTES == 128 && kKind != MmaKind::F16) {
        if (cfg.mt == 2 && cfg.ctas == 1) {
            if constexpr (kKind == MmaKind::I8) {
                if (cfg.bn == 128 && cfg.out_mode == kOutNHWC_S8) return launch_one<kKind, KB_BYTES, 128, kOutNHWC_S8, 1, false, 2>(p, s);
            } else if (cfg.out_mode == kOutNHWC_F32) {
                if (cfg.bn == 64) return launch_one<kKind, KB_BYTES, 64, kOutNHWC_F32, 1, false, 2>(p, s);
                if (cfg.bn == 128) return launch_one<kKind, KB_BYTES, 128, kOutNHWC_F32, 1, false, 2>(p, s);
            } else if (cfg.out_mode == kOutNCHW_F32) {
                if (cfg.bn == 64) return launch_one<kKind, KB_BYTES, 64, kOutNCHW_F32, 1, false, 2>(p, s);
                if (cfg.bn == 128) return launch_one<kKind, KB_BYTES, 128, kOutNCHW_F32, 1, false, 2>(p, s);
            }
        }
    }
    if (cfg.mt != 1) return fail(KXC_B200_ERR_INVALID, "tensor-core conv: no multi-tile kernel for this configuration");
    if constexpr (KB_BYTES == 128) {
        if (cfg.ctas == 2) {  // pairs exist for the wide tiles only (tc_setup_conv)
            switch (cfg.bn) {
                case 128: return launch_by_out<kKind, KB_BYTES, 128, 2>(cfg, p, s);
                case 256: return launch_by_out<kKind, KB_BYTES, 256, 2>(cfg, p, s);
                default: return fail(KXC_B200_ERR_INVALID, "tensor-core conv: no CTA-pair kernel for N tile %d", cfg.bn);
            }
        }
    }
    if (cfg.ctas != 1) return fail(KXC_B200_ERR_INVALID, "tensor-core conv: no CTA-pair kernel for %d-byte K blocks", KB_BYTES);
    switch (cfg.bn) {
        case 64: return launch_by_out<kKind, KB_BYTES, 64, 1>(cfg, p, s);
        case 128: return launch_by_out<kKind, KB_BYTES, 128, 1>(cfg, p, s);
        case 192:
            if constexpr (KB_BYTES == 128) return launch_by_out<kKind, KB_BYTES, 192, 1>(cfg, p, s);
            return fail(KXC_B200_ERR_INVALID, "tensor-core conv: the 192-wide tile exists for 128-byte K blocks only");
        case 256: return launch_by_out<kKind, KB_BYTES, 256, 1>(cfg, p, s);
        default: return fail(KXC_B200_ERR_INVALID, "tensor-core conv: unsupported N tile %d", cfg.bn);
    }
}

template <MmaKind kKind>
int32_t launch_by_kb(const TcConfig& cfg, const TcParams& p, cudaStream_t s) {
    switch (cfg.kb_bytes) {
        case 32: return launch_by_bn<kKind, 32>(cfg, p, s);
        case 64: return launch_by_bn<kKind, 64>(cfg, p, s);
        case 128: return launch_by_bn<kKind, 128>(cfg, p, s);
        default: return fail(KXC_B200_ERR_INVALID, "tensor-core conv: unsupported K block of %d bytes", cfg.kb_bytes);
    }
}

}  // namespace

int32_t tc_launch(const TcConfig& cfg, const TcParams& p, cudaStream_t stream) {
    if (p.split > 1) return tc_launch_split(cfg, p, stream);
    switch (cfg.dtype) {
        case kTcBF16: return launch_by_kb<MmaKind::F16>(cfg, p, stream);
        case kTcTF32: return launch_by_kb<MmaKind::TF32>(cfg, p, stream);
        case kTcS8: return launch_by_kb<MmaKind::I8>(cfg, p, stream);
    }
    return fail(KXC_B200_ERR_INVALID, "tensor-core conv: unknown dtype");
}

namespace {
// What the two searches over tile boxes look up instead of dividing in every one of up to 620 boxes (an operator call spent 2 to
// 7 us of host time on them): tiles over the rows by box height, and images per box and tiles over the images by box area.
struct BoxTables {
    int tiles_h[129], bni[129], tiles_n[129];
    BoxTables(int N, int OH) {
        for (int bh = 1; bh <= 128 && bh <= OH; ++bh) tiles_h[bh] = (OH + bh - 1) / bh;
        for (int area = 1; area <= 128; ++area) {
            int bn = 128 / area;
            if (bn > N) bn = N;
            if (bn < 1) bn = 1;
            bni[area] = bn;
            tiles_n[area] = (N + bn - 1) / bn;
        }
    }
};
}  // namespace

void tc_pick_tile(int N, int OH, int OW, int* BW, int* BH, int* BNI) {
    const BoxTables tables(N, OH);
    long long best = -1;
    int bw_best = 1, bh_best = 1, area_best = 0, skew_best = 0;
    for (int bw = 1; bw <= OW && bw <= 128; ++bw) {
        const long long tiles_w = (OW + bw - 1) / bw;
        for (int bh = 1, area = bw; bh <= OH && area <= 128; ++bh, area += bw) {
            const long long tiles = tiles_w * tables.tiles_h[bh] * tables.tiles_n[area];
            // prefer fewer tiles, i.e. more of the 128 rows in use; on ties the box with the most pixels per image (neighbouring
            // filter taps of one tile then re-read the same cache lines), then the squarer one (smaller halo)
            const int skew = bw > bh ? bw - bh : bh - bw;
            if (best < 0 || tiles < best || (tiles == best && (area > area_best || (area == area_best && skew < skew_best)))) {
                best = tiles;
                bw_best = bw; bh_best = bh; area_best = area; skew_best = skew;
            }
        }
    }
    *BW = bw_best; *BH = bh_best; *BNI = tables.bni[bw_best * bh_best];
}

int32_t tc_make_tmap(CUtensorMap* out, TcDType dtype, int rank, void* base, const uint64_t* dims,
                     const uint64_t* strides_bytes, const uint32_t* box, int swizzle_bytes) {
    static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    });
    if (!encode) return fail(KXC_B200_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    const CUtensorMapDataType dt = dtype == kTcBF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                                    : (dtype == kTcTF32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_UINT8);
    const CUtensorMapSwizzle sw = swizzle_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                                                       : (swizzle_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
    cuuint64_t gdims[5];
    cuuint64_t gstrides[4];
    cuuint32_t gbox[5];
    cuuint32_t estr[5];
    for (int i = 0; i < rank; ++i) {
        gdims[i] = dims[i];
        gbox[i] = box[i];
        estr[i] = 1;
        if (i + 1 < rank) gstrides[i] = strides_bytes[i];
    }
    const CUresult r = encode(out, dt, (cuuint32_t)rank, base, gdims, gstrides, gbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        return fail(KXC_B200_ERR_CUDA,
                    "cuTensorMapEncodeTiled failed (%d): rank %d dims [%llu,%llu,%llu,%llu] box [%u,%u,%u,%u] stride0 %llu", (int)r,
                    rank, (unsigned long long)dims[0], (unsigned long long)(rank > 1 ? dims[1] : 0),
                    (unsigned long long)(rank > 2 ? dims[2] : 0), (unsigned long long)(rank > 3 ? dims[3] : 0), box[0],
                    rank > 1 ? box[1] : 0, rank > 2 ? box[2] : 0, rank > 3 ? box[3] : 0,
                    (unsigned long long)(rank > 1 ? strides_bytes[0] : 0));
    }
    return KXC_B200_OK;
}

int32_t tc_status_word(int** out) {
    static std::mutex mu;
    static int* words[64] = {nullptr};
    int dev = 0;
    KXC_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(KXC_B200_ERR_INVALID, "device ordinal %d out of range", dev);
    std::lock_guard<std::mutex> lock(mu);
    if (!words[dev]) {
        KXC_CUDA_TRY(cudaMalloc(&words[dev], sizeof(int)));
        KXC_CUDA_TRY(cudaMemset(words[dev], 0, sizeof(int)));
    }
    *out = words[dev];
    return KXC_B200_OK;
}

int32_t tc_bind_store(TcParams* p, const TcConfig& cfg) {
    p->store_box = 0;
    static const bool enabled = [] {
        const char* e = getenv("KXC_B200_TMA_STORE");
        return !(e != nullptr && e[0] == '0');
    }();
    auto pow2 = [](int v) { return v > 0 && (v & (v - 1)) == 0; };
    if (!enabled || cfg.dtype != kTcBF16 || cfg.out_mode != kOutNHWC_BF16 || cfg.bn < 128 || cfg.bn == 192 || p->out == nullptr || (p->Cout & 63) != 0 ||
        !pow2(p->BW) || !pow2(p->BH) || !pow2(p->BNI) || p->BW * p->BH * p->BNI != 128 || p->BW > 32)
        return KXC_B200_OK;
    // a warp's 32 consecutive tile rows as a box of the output tensor
    const int hw = p->BW * p->BH;
    const uint32_t sub_w = (uint32_t)p->BW;
    const uint32_t sub_h = (uint32_t)(hw >= 32 ? 32 / p->BW : p->BH);
    const uint32_t sub_n = (uint32_t)(hw >= 32 ? 1 : 32 / hw);
    const uint64_t px = (uint64_t)p->Cout * 2;
    const uint64_t dims[4] = {(uint64_t)p->Cout, (uint64_t)p->OW, (uint64_t)p->OH, (uint64_t)p->N};
    const uint64_t strides[3] = {px, (uint64_t)p->OW * px, (uint64_t)p->OH * p->OW * px};
    const uint32_t box[4] = {64u, sub_w, sub_h, sub_n};
    KXC_TRY(tc_make_tmap(&p->tmOut, kTcBF16, 4, p->out, dims, strides, box, 128));
    if (cfg.dual) {
        if (p->out2 == nullptr) return KXC_B200_OK;
        KXC_TRY(tc_make_tmap(&p->tmOut2, kTcBF16, 4, p->out2, dims, strides, box, 128));
    }
    p->store_box = 1;
    return KXC_B200_OK;
}

namespace {
// Tile box of a launch that writes the reference's layout: a warp's 32 pixels leave as one 4-byte store per channel, in runs of
// BW consecutive addresses (BW * BH when the box spans the rows), and every run costs its own 32-byte sectors. The box with
// the fewest tiles may have runs of one to three pixels, so waves and sectors are weighed together: a tile's main loop is its K
// blocks at the rate they arrive, its epilogue 80 cycles per channel or, if that is more, 12 per sector of a warp's store, which
// overlaps the next tile's main loop. Runs of 8 to 32 pixels took the same time per tile (62 to 66 cycles per channel at 256
// channels without a residual; 88, 95 and 107 at 32, 16 and 8 with one), runs of 4 twice that. Among 60 launches timed with up to 30
// boxes each, a cost per sector alone traded whole waves for longer runs: 31 -> 331 1x1 stride 2, 56x54, 61 images, 1x14x9 boxes
// 52 us and 1x4x27 60; 20 -> 463 on 101x103, 53 images, 158 and 172. In launches of one wave the box hardly matters (64 -> 64
// 3x3 at 56x56, one image: 11.0 to 11.3 us from 128 down to 28 pixels a box). All of these were measured with 64-bit addresses in the
// epilogue; nchw_store32 takes up to 0.6 of its time (95 -> 120 1x1 at 33x36, 50 images 21.3 -> 12.9 us a launch), so the weights given to
// it here are too high by as much and have not been fitted again.
void pick_tile_nchw(int N, int OH, int OW, int Cout, int num_kb, int kb_bytes, int* BW, int* BH, int* BNI) {
    const int bn_out = Cout <= 64 ? 64 : (Cout <= 128 ? 128 : 256);
    const int tiles_c = (Cout + bn_out - 1) / bn_out;
    const double main_loop = (double)num_kb * kb_bytes / 128.0 * (bn_out == 64 ? 550 : (bn_out == 128 ? 590 : 620));  // (choose_split's figures)
    const BoxTables tables(N, OH);
    double best = -1.0;
    for (int bw = 1; bw <= OW && bw <= 128; ++bw) {
        const long long tiles_w = (OW + bw - 1) / bw;
        int run = 0;
        double epilogue = 0.0, slower = 0.0, once = 0.0;
        for (int bh = 1, area = bw; bh <= OH && area <= 128; ++bh, area += bw) {
            const long long tiles = tiles_w * tables.tiles_h[bh] * tables.tiles_n[area];
            const long long waves = (tiles * tiles_c + kNumSMs - 1) / kNumSMs;
            int r = bw == OW ? area : bw;
            if (r > 32) r = 32;
            if (r != run) {
                run = r;
                const double sectors = 32.0 * (run / 8.0 + 0.9) / run;
                epilogue = bn_out * (12.0 * sectors > 80.0 ? 12.0 * sectors : 80.0);
                slower = main_loop > epilogue ? main_loop : epilogue;
                once = 10.0 * sectors;
            }
            // (tie-breakers: longer runs, then fewer tiles on the same number of waves)
            const double cost = main_loop + (double)(waves - 1) * slower + epilogue + once + 1e-3 * (double)tiles;
            if (best < 0.0 || cost < best) {
                best = cost;
                *BW = bw; *BH = bh; *BNI = tables.bni[area];
            }
        }
    }
}

// The weights of a split launch: boxes of cfg->bn rows x one K block of `k_elems` elements per output channel.
int32_t weight_map(CUtensorMap* m, const TcConfig* cfg, const TcParams* p, const void* w, int k_elems) {
    const uint64_t dims[2] = {(uint64_t)k_elems, (uint64_t)p->Cout};
    const uint64_t strides[1] = {(uint64_t)k_elems * tc_elem_bytes(cfg->dtype)};
    const uint32_t box[2] = {(uint32_t)p->kb_elems, (uint32_t)cfg->bn};
    return tc_make_tmap(m, cfg->dtype, 2, const_cast<void*>(w), dims, strides, box, 128);
}

// Whether `tiles` clusters of s CTAs fit on the chip at once, and the cycles that the last ones start later. Clusters of an odd
// number of CTAs leave halves of SM pairs behind: behind a kernel that is still draining, 44 of 45 clusters of three took 1 to
// 17 us longer than fewer clusters do, 25 and 26 of 26 clusters of five 2 and 5 us (32 of 33 clusters of four 0.3); behind one
// that leaves the shared memory free, nothing.
bool split_fits(long long tiles, int s, long long* late) {
    const int held = tc_split_capacity(s);
    *late = (s & 1) != 0 && tiles > held - 2 ? 3800 : 0;
    return tiles * s <= kNumSMs && tiles <= held;
}

// Whether a set-up launch (tile width, store form and so on already chosen for the persistent kernel) is better off with its
// reduction split over a cluster, and the set-up of that form: the cheaper of the two in modelled cycles, the split one 5 % ahead.
// The figures are fits over 320 launches timed in every form that fits the chip (7 layers in a row, NHWC, and one layer
// into NCHW; 16 to 144 K blocks; 1 to 96 images), in clocks of 1.9 GHz, and older than the loops of whole warps, which take 400 to 490 clocks a block at 64
// and 128 channels in either form (tc_modelled_clocks below, which only the choice of CTA pairs uses): this model splits from 14 K blocks on in two parts of one
// wave, that one from 18 to 24. Which is right there has not been timed:
//   a K block of 128 bytes per row     550 / 590 / 500 / 620 at 64 / 128 / 192 / 256 channels, 650 at 256 in the split kernel;
//                                      760 with two bf16 pixel tiles, 820 / 1100 with two tf32 ones; three passes 830 / 1050, split 830 / 930, pairs
//                                      660 (of the loops of whole warps: 148 launches that pairs took over were 1.11 times as fast with them in
//                                      the mean, 0.94 to 1.8, the 22 that would be split 1.18, 0.98 to 1.8)
//   what follows the last K block      unsplit 0 / 2000 / 4000 / 8000 (the epilogue of that many channels), 2800 more with two pixel
//                                      tiles; split 3000 / 5500 / 10000 (the exchange of the partial sums over distributed shared
//                                      memory and the epilogue, which grow with the width; refitted over 170 layers when the
//                                      exchange changed, 7000 / 13000 before: 0.1 % behind the fastest form, 0.5 with the old ones;
//                                      tf32 512 -> 512 1x1 at 7x7, 32 images: 14.0 unsplit, 11.7 in two parts of 128 channels);
//                                      7000 and 13000 still into the reference's layout, whose 4-byte stores weigh more (tf32 66
//                                      channels 3x3 stride 2 at 23x22, 43 images: 16.4 unsplit, 18.4 split by the lower figures);
//                                      4000 more into the reference's layout, for more than 64 channels, when the weights cannot
//                                      be fetched ahead of the previous kernel's end (87 operator calls: 14 were slower than
//                                      unsplit without it, tf32 42 -> 113 3x3 at 11x11, 30 images, 16.1 against 14.0 us; 5 with it;
//                                      427 -> 36 1x1 at 8x7, 7 images, 11.6 split, 12.4 unsplit)
// Into NCHW what this chooses was 1.4 % behind the fastest form on average, and one launch behind the unsplit one by more than
// 1 %, both with the epilogue of 64-bit addresses, which unsplit launches below 4 GiB have left since (nchw_store32): the unsplit tails
// and the figures into NCHW have not been fitted again. (One figure for every width, 3000, made wide splits of short reductions slower than no split: bf16
// 1024 -> 1024 1x1 at 7x7 and 24 images 14.7 us per layer in two parts of 256 channels, 11.3 unsplit; 256 -> 256 3x3 at
// 14x14 and 32 images 19.4 and 17.8.) A launch is kept to the clusters that the chip holds at once (split_fits; a dense
// layer of 16 tiles in clusters of eight that did not all fit: 8.8 -> 12 us).
int32_t choose_split(TcParams* p, TcConfig* cfg, const void* w, const void* w_lo, int k_elems) {
    p->split = 0;
    if (cfg->dtype == kTcS8 || cfg->kb_bytes != 128) return KXC_B200_OK;
    const long long m_tiles = (long long)p->tiles_w * p->tiles_h * p->tiles_n;
    const int kb = p->taps_h * p->taps_w * p->cblocks;
    const bool wide_items = cfg->mt == 2;
    const long long block = cfg->x3 ? (cfg->ctas == 2 ? 660 : (cfg->bn == 64 ? 830 : 1050))
                            : wide_items ? (cfg->dtype == kTcBF16 ? 760 : (cfg->bn == 64 ? 820 : 1100))
                                         : (cfg->bn == 64 ? 550 : (cfg->bn == 128 ? 590 : (cfg->bn == 192 ? 500 : 620)));
    const long long tail = (cfg->bn == 64 ? 0 : (cfg->bn == 128 ? 2000 : (cfg->bn == 192 ? 4000 : 8000))) + (wide_items ? 2800 : 0);
    const long long group = (long long)cfg->ctas * cfg->mt;
    const long long items = p->tiles_c * ((m_tiles + group - 1) / group), slots = kNumSMs / cfg->ctas;
    long long best = ((items + slots - 1) / slots * kb * block + tail) * 95 / 100;
    cfg->clocks = (double)best * 100.0 / 95.0;
    if (cfg->out_mode != kOutNCHW_F32) {  // (the epilogue, ~30 clocks a channel of a pixel tile, where it outlasts the main loop)
        const long long epilogue = 30ll * cfg->bn * cfg->mt;
        if (epilogue > kb * block) cfg->clocks = (double)((items + slots - 1) / slots * epilogue + tail);
    }
    if (kb < 12) return KXC_B200_OK;  // two or three microseconds as it is
    const bool nchw = cfg->out_mode == kOutNCHW_F32;
    const long long cold = nchw && !p->weights_ready && p->Cout > 64 ? 4000 : 0;
    int split = 0, width = 0;
    for (int bn = 64; bn <= 256 && (bn == 64 || bn / 2 < p->Cout) && !(bn == 256 && cfg->x3); bn *= 2) {
        const long long tiles = m_tiles * ((p->Cout + bn - 1) / bn);
        const long long split_block = cfg->x3 ? (bn == 64 ? 830 : 930) : (bn == 64 ? 550 : (bn == 128 ? 590 : 650));
        const long long split_tail = bn == 64 ? 3000 : (nchw ? (bn == 128 ? 7000 : 13000) : (bn == 128 ? 5500 : 10000));
        for (int s = 2; s <= (bn == 256 ? 4 : kMaxSplit); ++s) {  // (what shared memory holds of the parts)
            long long late = 0;
            if (!split_fits(tiles, s, &late)) continue;
            const long long span = (long long)((kb + s - 1) / s) * split_block + split_tail + cold + late;
            if (span < best) {
                best = span;
                split = s;
                width = bn;
            }
        }
    }
    if (split == 0) return KXC_B200_OK;
    p->split = split;
    cfg->clocks = (double)best;
    cfg->bn = width; cfg->ctas = 1; cfg->mt = 1;
    p->tiles_c = (p->Cout + width - 1) / width;
    KXC_TRY(weight_map(&p->tmB, cfg, p, w, k_elems));
    return w_lo != nullptr ? weight_map(&p->tmB2, cfg, p, w_lo, k_elems) : KXC_B200_OK;
}
}  // namespace

bool tc_cta_pairs() {
    static const bool on = [] {
        const char* e = getenv("KXC_B200_CTA_PAIR");
        return !(e != nullptr && e[0] == '0');
    }();
    return on;
}

// Per form: what a launch costs besides, a K block, the epilogue of a tile (it overlaps the next tile's main loop) NHWC and what a residual adds to it,
// and both into the reference's layout. Fits over the launches of 381 drawn layers (plans' layers with and without a residual, graph outputs,
// operators with their conversion apart; 1 to 512 images), 2 to 9 % rms each. Choosing between this and the channel-major kernel's clocks (box_cost
// there, 12 % rms) lost 1.004 to 1.02 in the mean of each kind of layer against the faster form of each; weighted ratios of older models with lines
// of their own per kind of layer 1.02 to 1.04.
double tc_modelled_clocks(const TcParams& p, const TcConfig& cfg, bool residual) {
    struct Form {
        double once, block, epilogue, with_residual, planes, planes_with_residual;
    };
    const bool bf16 = cfg.dtype == kTcBF16;
    static constexpr Form kWhole[2][3] = {{{2640, 405, 2720, 0, 2865, 593}, {2700, 427, 6230, 680, 5200, 2080}, {1420, 596, 14080, 2720, 11900, 9160}},    // tf32 64, 128, 256
                                          {{2620, 417, 2660, 0, 2750, 470}, {2700, 430, 4500, 680, 5200, 2080}, {5480, 590, 6680, 3020, 12950, 8470}}};   // bf16
    static constexpr Form kTwoTiles[2] = {{2050, 703, 6150, 0, 6600, 490}, {5740, 791, 8070, 1630, 5110, 2360}};                                          // tf32 64, 128
    static constexpr Form kTwoTilesBf16 = {500, 859, 7770, 2280, 7770, 2280}, k192 = {2530, 477, 5180, 1510, 10630, 5920};
    static constexpr Form kSplit[2][3] = {{{4520, 401, 4580, 0, 5000, 380}, {5580, 482, 6570, 0, 6530, 660}, {5850, 660, 12950, 0, 9000, 3600}},           // tf32
                                          {{4660, 489, 3680, 0, 4830, 140}, {5720, 425, 6450, 0, 4820, 2280}, {6100, 751, 10590, 0, 6660, 3610}}};         // bf16
    const int width = cfg.bn == 64 ? 0 : (cfg.bn == 128 ? 1 : 2);
    const Form& f = p.split > 1 ? kSplit[bf16][width] : (cfg.mt == 2 ? (bf16 ? kTwoTilesBf16 : kTwoTiles[width == 0 ? 0 : 1]) : (cfg.bn == 192 ? k192 : kWhole[bf16][width]));
    const long long m_tiles = (long long)p.tiles_w * p.tiles_h * p.tiles_n;
    const int kb = p.taps_h * p.taps_w * p.cblocks;
    const long long group = (long long)cfg.ctas * cfg.mt, items = p.tiles_c * ((m_tiles + group - 1) / group), slots = kNumSMs / cfg.ctas;
    const double waves = p.split > 1 ? 1.0 : (double)((items + slots - 1) / slots);
    const double main_loop = f.block * (p.split > 1 ? (kb + p.split - 1) / p.split : kb);
    const double epilogue = cfg.out_mode == kOutNCHW_F32 ? f.planes + (residual ? f.planes_with_residual : 0.0) : f.epilogue + (residual ? f.with_residual : 0.0);
    return f.once + main_loop + (waves - 1.0) * (main_loop > epilogue ? main_loop : epilogue) + epilogue;
}

bool tc_dual_applicable(TcDType dtype, TcOutMode out_mode, int cpad, int Cout, int KH, int KW, int stride, int pad_h, int pad_w,
                        int dil_h, int dil_w) {
    // the second output's only tap must be the main filter's centre tap
    return dtype == kTcBF16 && out_mode == kOutNHWC_BF16 && (cpad * 2) % 128 == 0 && Cout % 32 == 0 && (KH & 1) && (KW & 1) &&
           dil_h == 1 && dil_w == 1 && pad_h == KH / 2 && pad_w == KW / 2 && (stride == 1 || stride == 2);
}

int32_t tc_setup_dual(TcParams* p, TcConfig* cfg, const void* act_nhwc, const void* w_packed, const void* w2_packed, int N,
                      int H, int W, int cpad, int Cout, int KH, int KW, int stride, int pad_h, int pad_w) {
    KXC_TRY(tc_setup_conv(p, cfg, kTcBF16, kOutNHWC_BF16, act_nhwc, w_packed, N, H, W, cpad, Cout, KH, KW, stride, pad_h, pad_w, 1, 1));
    cfg->ctas = 1; cfg->mt = 1; cfg->dual = 1;
    p->split = 0;  // (that of the main convolution alone)
    const long long m_tiles = (long long)p->tiles_w * p->tiles_h * p->tiles_n;
    auto waves = [](long long items) { return (items + kNumSMs - 1) / kNumSMs; };
    // Split over clusters as in choose_split, by the clusters of this form and with the second output's K blocks behind the last
    // rank's own. Its partial sums double the exchange, which leaves nothing to gain for tiles wider than 64 channels:
    // 256 -> 512 at 14x14, block of four layers, us unsplit / 64 wide / 128 wide: one image 35.0 / 24.8 / 26.9, 8 images
    // 35.5 / 30.9 / 32.9, 16 images 41.2 / 37.1 / 37.1, 24 images 45.3 / - / 45.3; 128 -> 256 at 28x28: 4 images
    // 28.9 / 27.2 / 29.3, 8 images 33.1 / 31.5 / 33.3. Of short reductions (nine K blocks: 3x3
    // over 64 channels) only parts of two K blocks pay, and the margin leaves those: of 85 drawn blocks (32 to 512 outputs, 8x8 to 109x109, 1 to
    // 42 images; blocks of four layers) 56 split into five and more parts were 1.06 to 1.25 times as fast, 1.15 in the mean; 12 in three parts 0.95 to
    // 1.11, 17 in two 0.92 to 0.99 and one 1.03. ResNet-18 at one image 115.8 / 111.8 us.
    const int kb = KH * KW * p->cblocks;
    const long long tiles64 = m_tiles * ((Cout + 63) / 64);
    long long best = (waves(m_tiles * ((Cout + 127) / 128)) * (kb + p->cblocks) * 590 + 4000) * 95 / 100;
    const long long margin = kb < 12 ? 2900 : 0;
    for (int s = 2; kb >= 8 && s <= kMaxSplit; ++s) {
        long long late = 0;
        if (!split_fits(tiles64, s, &late)) continue;
        const long long span = (long long)(kb - (s - 1) * kb / s + p->cblocks) * 550 + 4400 + late + margin;
        if (span < best) {
            best = span;
            p->split = s;
        }
    }
    if (p->split > 1) {
        cfg->bn = 64;
        p->tiles_c = (Cout + 63) / 64;
        KXC_TRY(weight_map(&p->tmB, cfg, p, w_packed, KH * KW * cpad));
        return weight_map(&p->tmB2, cfg, p, w2_packed, cpad);
    }
    // The two accumulators of a buffer share TMEM: 128-wide tiles (two buffers of 2 x 128 columns), single CTAs. When
    // that leaves a launch with a second, mostly empty wave and 192-wide tiles fit one wave (256 -> 512 channels at 128
    // images: 196 tiles against 147 for 148 SMs), the 192-wide form is taken: one buffer of 2 x 192 columns, so the
    // epilogue no longer overlaps the next item's MMAs, which a CTA with a single work item does not miss.
    int bn = 128;
    {
        const long long t128 = m_tiles * ((Cout + 127) / 128), t192 = m_tiles * ((Cout + 191) / 192);
        static const bool model = [] { const char* e = getenv("KXC_B200_TILE_MODEL"); return !(e != nullptr && e[0] == '0'); }();
        if (model && p->kb_elems * 2 == 128 && waves(t192) == 1 && waves(t128) >= 2) bn = 192;  // (192-wide tiles need 128-byte K blocks)
    }
    cfg->bn = bn;
    p->tiles_c = (Cout + bn - 1) / bn;
    const uint64_t ktot = (uint64_t)KH * KW * cpad;
    const uint64_t bdims[2] = {ktot, (uint64_t)Cout};
    const uint64_t bstrides[1] = {ktot * 2};
    const uint32_t bbox[2] = {(uint32_t)p->kb_elems, (uint32_t)bn};
    KXC_TRY(tc_make_tmap(&p->tmB, kTcBF16, 2, const_cast<void*>(w_packed), bdims, bstrides, bbox, 128));
    const uint64_t b2dims[2] = {(uint64_t)cpad, (uint64_t)Cout};
    const uint64_t b2strides[1] = {(uint64_t)cpad * 2};
    return tc_make_tmap(&p->tmB2, kTcBF16, 2, const_cast<void*>(w2_packed), b2dims, b2strides, bbox, 128);
}

int32_t tc_setup_conv(TcParams* p, TcConfig* cfg, TcDType dtype, TcOutMode out_mode, const void* act_nhwc,
                      const void* w_packed, int N, int H, int W, int cpad, int Cout, int KH, int KW, int stride, int pad_h,
                      int pad_w, int dil_h, int dil_w, int* status_word, int map_images) {
    if (map_images <= 0) map_images = N;
    const int eb = tc_elem_bytes(dtype);
    if (stride != 1 && stride != 2) return fail(KXC_B200_ERR_UNSUPPORTED, "tensor-core conv: stride %d", stride);
    const int row_bytes = cpad * eb;
    int kb_bytes;
    if (row_bytes == 32 || row_bytes == 64) kb_bytes = row_bytes;
    else if (row_bytes % 128 == 0) kb_bytes = 128;
    else return fail(KXC_B200_ERR_INVALID, "tensor-core conv: %d padded channels x %d bytes is not a K-block multiple", cpad, eb);
    const int OH = (int)conv_out_dim(H, KH, stride, pad_h, dil_h);
    const int OW = (int)conv_out_dim(W, KW, stride, pad_w, dil_w);
    if (OH <= 0 || OW <= 0) return fail(KXC_B200_ERR_INVALID, "tensor-core conv: empty output");

    p->N = N; p->OH = OH; p->OW = OW; p->Cout = Cout;
    p->taps_h = KH; p->taps_w = KW; p->stride = stride;
    p->pad_h = pad_h; p->pad_w = pad_w; p->dil_h = dil_h; p->dil_w = dil_w;
    p->kb_elems = kb_bytes / eb;
    p->cblocks = row_bytes / kb_bytes;
    if (out_mode == kOutNCHW_F32)
        pick_tile_nchw(N, OH, OW, Cout, KH * KW * p->cblocks, kb_bytes, &p->BW, &p->BH, &p->BNI);
    else
        tc_pick_tile(N, OH, OW, &p->BW, &p->BH, &p->BNI);
    p->tiles_w = (OW + p->BW - 1) / p->BW;
    p->tiles_h = (OH + p->BH - 1) / p->BH;
    p->tiles_n = (N + p->BNI - 1) / p->BNI;

    int bn = Cout <= 64 ? 64 : (Cout <= 128 ? 128 : 256);
    // A launch with a handful of tiles (the dense layer of a small batch: 1 pixel tile x 4 channel tiles) is bound by
    // the latency of each CTA's own operand stream: narrower tiles spread the weight rows over more SMs.
    {
        const long long mt = (long long)p->tiles_w * p->tiles_h * p->tiles_n;
        while (bn > 64 && mt * ((Cout + bn - 1) / bn) < 32) bn /= 2;
        // Into the reference's layout a narrower tile is the better one as long as all are resident at once: their K blocks
        // arrive at nearly the same rate, and the epilogue that follows the last one is half as long. (252 -> 160 1x1 at 9x9,
        // tf32, 42 images: 10.1 us 64 wide, 14.8 256 wide; 84 -> 433 1x1 at 7x10, bf16, 12 images: 7.2 and 8.6 128 wide.)
        if (out_mode == kOutNCHW_F32) {
            while (bn > 64 && mt * ((Cout + bn / 2 - 1) / (bn / 2)) <= kNumSMs) bn /= 2;
        }
    }
    // CTA pairs (tcgen05 cta_group::2): each CTA fetches half of the B tile, which relieves the L2 -> shared-memory
    // fill rate that bounds the wide tiles.
    const long long m_tiles = (long long)p->tiles_w * p->tiles_h * p->tiles_n;
    // Measured: pairs gain 5-7 % with the 256-wide tile, so that one uses them. With the 128-wide one they lost 3-10 % when one lane issued and
    // are level since (ResNet-18 bf16, 1024 images 3322 us, with them 3328; 64 to 256 level). "2" forces them for 128 too.
    static const bool pair_all = [] { const char* e = getenv("KXC_B200_CTA_PAIR"); return e != nullptr && e[0] == '2'; }();
    int ctas = (tc_cta_pairs() && bn >= (pair_all ? 128 : 256) && kb_bytes == 128 && m_tiles >= 2) ? 2 : 1;
    // Launches with few tiles (small per-GPU batches in the deep layers): the 256-wide tile leaves SMs idle, e.g. 98 tiles
    // (49-50 pairs) on 148 SMs. 512 channels in 192-wide tiles on 49 pixel tiles are 147 CTAs, one wave, and an
    // M = 128, K = 16 instruction takes ~99 cycles at N = 192 against ~131 at N = 256 (measured). The narrower tile is
    // taken when the modelled makespan (waves x cycles per instruction) gains 10 %: layer 4 at 128 / 256 images per GPU
    // 37 -> 35 / 61 -> 57 us. (A 128-wide tile was measured slower there, 38 -> 45 us: without the pair's halved weight
    // fetch each CTA's operand stream from L2 becomes the limit.) KXC_B200_TILE_MODEL=0 keeps the widest tile.
    static const bool tile_model = [] {
        const char* e = getenv("KXC_B200_TILE_MODEL");
        return !(e != nullptr && e[0] == '0');
    }();
    if (tile_model && bn == 256 && kb_bytes == 128 && (dtype == kTcBF16 || dtype == kTcS8)) {
        auto waves = [](long long items, long long slots) { return (items + slots - 1) / slots; };
        const long long span256 = ctas == 2 ? waves(((m_tiles + 1) / 2) * ((Cout + 255) / 256), kNumSMs / 2) * 131
                                            : waves(m_tiles * ((Cout + 255) / 256), kNumSMs) * 131;
        const long long span192 = waves(m_tiles * ((Cout + 191) / 192), kNumSMs) * 99;
        int pick = 256;
        if (span192 * 10 <= span256 * 9) pick = 192;
        if (pick != 256) {
            bn = pick;
            ctas = 1;
        }
    }
    cfg->dtype = dtype; cfg->kb_bytes = kb_bytes; cfg->bn = bn; cfg->out_mode = out_mode; cfg->ctas = ctas;
    // Two pixel tiles per work item for the 128-wide bf16 tile: measured 0.285/0.277/0.284 -> 0.231/0.221/0.234 ms on the
    // 128->128 layers. With the
    // 256-wide tile TMEM holds only one buffer of two accumulators and the lost epilogue overlap costs more than the
    // second chain brings (0.168 -> 0.211 ms), so that form is not instantiated. KXC_B200_MT=1 switches it off.
    static const bool mt_enabled = [] {
        const char* e = getenv("KXC_B200_MT");
        return !(e != nullptr && e[0] == '1');
    }();
    cfg->mt = (mt_enabled && bn == 128 && dtype == kTcBF16 && out_mode == kOutNHWC_BF16 && kb_bytes == 128 && m_tiles >= 2 * ctas) ? 2 : 1;
    // tf32 and int8: the tiles of such a launch reach shared memory at 7 to 8 TB/s over all SMs whatever the MMAs do, and two
    // pixel tiles against one weight tile are 20 / 24 KB per tile instead of 24 / 32 (64 / 128 channels). Taken when the
    // modelled makespan gains: a stage of two tiles cost 820 / 1100 cycles against 490 / 655 when one lane issued (a whole warp: 703 / 791 against 405 / 427,
    // tc_modelled_clocks; not fitted again). ResNet-18 tf32, 32 images: layer 1 42 -> 34 us per convolution, layer 2 31 -> 30; int8 128 -> 128, 28x28, 256
    // images: 52 -> 46.
    if (mt_enabled && ctas == 1 && kb_bytes == 128 &&
        ((dtype == kTcTF32 && (bn == 64 || bn == 128)) || (dtype == kTcS8 && bn == 128 && out_mode == kOutNHWC_S8))) {
        const long long tc = (Cout + bn - 1) / bn;
        auto waves = [](long long items) { return (items + kNumSMs - 1) / kNumSMs; };
        if (waves((m_tiles + 1) / 2 * tc) * (bn == 64 ? 820 : 1100) < waves(m_tiles * tc) * (bn == 64 ? 490 : 655)) cfg->mt = 2;
    }
    p->tiles_c = (Cout + bn - 1) / bn;

    const uint32_t box[4] = {(uint32_t)p->kb_elems, (uint32_t)p->BW, (uint32_t)p->BH, (uint32_t)p->BNI};
    uint8_t* base = const_cast<uint8_t*>(static_cast<const uint8_t*>(act_nhwc));
    if (stride == 1) {
        const uint64_t dims[4] = {(uint64_t)cpad, (uint64_t)W, (uint64_t)H, (uint64_t)map_images};
        const uint64_t strides[3] = {(uint64_t)row_bytes, (uint64_t)W * row_bytes, (uint64_t)H * W * row_bytes};
        KXC_TRY(tc_make_tmap(&p->tmA[0], dtype, 4, base, dims, strides, box, kb_bytes));
        for (int i = 1; i < 4; ++i) p->tmA[i] = p->tmA[0];
    } else {
        // One map per (row parity, column parity): the stride-2 walk over the input becomes a unit-stride
        // walk over the pixels of one parity class.
        for (int hp = 0; hp < 2; ++hp)
            for (int wp = 0; wp < 2; ++wp) {
                const int hc = (H - hp + 1) / 2, wc = (W - wp + 1) / 2;
                CUtensorMap* m = &p->tmA[hp * 2 + wp];
                if (hc <= 0 || wc <= 0)
                    return fail(KXC_B200_ERR_UNSUPPORTED, "tensor-core conv: stride 2 over a %dx%d input", H, W);
                const uint64_t dims[4] = {(uint64_t)cpad, (uint64_t)wc, (uint64_t)hc, (uint64_t)map_images};
                const uint64_t strides[3] = {(uint64_t)2 * row_bytes, (uint64_t)2 * W * row_bytes, (uint64_t)H * W * row_bytes};
                KXC_TRY(tc_make_tmap(m, dtype, 4, base + ((size_t)hp * W + wp) * row_bytes, dims, strides, box, kb_bytes));
            }
    }
    const uint64_t ktot = (uint64_t)KH * KW * cpad;
    const uint64_t bdims[2] = {ktot, (uint64_t)Cout};
    const uint64_t bstrides[1] = {ktot * eb};
    const uint32_t bbox[2] = {(uint32_t)p->kb_elems, (uint32_t)(bn / ctas)};
    KXC_TRY(tc_make_tmap(&p->tmB, dtype, 2, const_cast<void*>(w_packed), bdims, bstrides, bbox, kb_bytes));
    if (status_word != nullptr) {
        p->status = status_word;
    } else {
        KXC_TRY(tc_status_word(&p->status));
    }
    return choose_split(p, cfg, w_packed, nullptr, KH * KW * cpad);
}

int32_t tc_finish_x3(TcParams* p, TcConfig* cfg, const void* w_hi, const void* w_lo, int Cout, int k_elems) {
    // The tile whose waves cost least. Single CTAs: by 950 cycles a stage with 64 channels and 1400 with 128 (of the loops of one lane, not fitted again); pairs
    // of 64 channels where by what the forms measured since (660, and 760 / 1030 for single ones, over ResNet-18's layers of 1 to 64 images) they are ahead. 250 launches of
    // 150 drawn layers (operators and plans, 1 to 64 images, 32 to 512 channels): pairs took 62, 1.09 times as fast in the mean, 0.98 to 1.30 (a
    // 64 -> 128 3x3 at 80x79, one image, before it was split in two). Fewer than 12 K blocks lose up to 10 % (the stem 73 / 78 us), 1x1 layers were 0.94 to 1.04 times as fast. Pairs of 128 channels
    // have one accumulator buffer and were level or behind (28x28, 32 images 45 / 52).
    const long long m_tiles = (long long)p->tiles_w * p->tiles_h * p->tiles_n;
    auto waves = [&](int bn) { return (m_tiles * ((Cout + bn - 1) / bn) + kNumSMs - 1) / kNumSMs; };
    int bn = Cout > 64 && waves(128) * 1400 <= waves(64) * 950 ? 128 : 64;
    const long long pair_waves = ((m_tiles + 1) / 2 * ((Cout + 63) / 64) + kNumSMs / 2 - 1) / (kNumSMs / 2);
    const bool pair = cfg->kb_bytes == 128 && m_tiles > 1 && p->taps_h * p->taps_w > 1 && p->taps_h * p->taps_w * p->cblocks >= 12 &&
                      pair_waves * 660 < waves(bn) * (bn == 64 ? 760 : 1030) && tc_cta_pairs() && tc_split_capacity(2) > 0;
    if (pair) bn = 64;
    cfg->bn = bn; cfg->ctas = pair ? 2 : 1; cfg->mt = 1; cfg->dual = 0; cfg->x3 = 1;
    p->tiles_c = (Cout + bn - 1) / bn;
    const uint64_t ktot = (uint64_t)k_elems;
    const uint64_t bdims[2] = {ktot, (uint64_t)Cout};
    const uint64_t bstrides[1] = {ktot * 4};
    const uint32_t bbox[2] = {(uint32_t)p->kb_elems, (uint32_t)(bn / cfg->ctas)};
    KXC_TRY(tc_make_tmap(&p->tmB, kTcTF32, 2, const_cast<void*>(w_hi), bdims, bstrides, bbox, cfg->kb_bytes));
    KXC_TRY(tc_make_tmap(&p->tmB2, kTcTF32, 2, const_cast<void*>(w_lo), bdims, bstrides, bbox, cfg->kb_bytes));
    return choose_split(p, cfg, w_hi, w_lo, k_elems);
}

int32_t tc_setup_conv_x3(TcParams* p, TcConfig* cfg, TcOutMode out_mode, const void* act_hi, const void* w_hi, const void* w_lo, int N,
                         int H, int W, int cpad, int Cout, int KH, int KW, int stride, int pad_h, int pad_w, int dil_h, int dil_w) {
    // The maps cover 2N images: an image's low part is addressed N images further on. A box that runs past image N reads
    // low parts into rows that are not stored.
    KXC_TRY(tc_setup_conv(p, cfg, kTcTF32, out_mode, act_hi, w_hi, N, H, W, cpad, Cout, KH, KW, stride, pad_h, pad_w, dil_h, dil_w, nullptr,
                          2 * N));
    return tc_finish_x3(p, cfg, w_hi, w_lo, Cout, KH * KW * cpad);
}

}  // namespace kxc_b200
