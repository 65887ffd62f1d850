// Convolution with the output CHANNELS as the MMA's rows and the pixels as its columns, on tcgen05 + TMEM: D[128 channels, N pixels] =
// W[128, K] x X[N, K]^T. Into the reference's layout (NCHW; bf16 / tf32 with fp32 results, int8) and, for layers of plans, into NHWC.
//
// The implicit-GEMM kernel (conv_tc.cu) has the pixels as rows, so a thread of its epilogue owns one pixel of every plane. For
// results in planes that costs three things this arrangement does not have:
//
//   * M = 128 pixels per tile whatever the image: here N is any multiple of 16 up to 256, which fits odd planes in whole waves;
//   * a table of requantize constants in shared memory that every thread reads for every value: here a thread IS a channel and
//     keeps its constants in registers;
//   * for int8 single-byte stores at plane pitch, or a second pass that transposes: here a thread holds consecutive pixels of its
//     channel, and a small staging tile turns them into runs of a plane.
//
// A 3x3 filter's nine taps share their pixels. A channel block's pixels come as ONE box with the filter's halo (stride 2: one box
// per row / column parity), HB x WB pixels of 128 bytes side by side in shared memory, and a tap is a view of that box at a row
// offset (the swizzle is a function of the address, so a view may start at any 128-byte row; conv_direct.cu does the same). The
// columns of the accumulator are then the box's pixels in flat order: WB - BW of every WB are not results and are not stored.
// Where that waste costs more than loading every tap by itself (small planes, wide filters) each tap is a box of its own; both are the
// same list of loads and of taps per load (CmParams).
//
// Channels beyond the last whole 32 bytes of a pixel are not multiplied: the last channel block of a tap issues only the
// instructions that have channels (72 tf32 channels: 9 of 12).
//
// CTA pairs (tcgen05 cta_group::2; NHWC results of more than 128 channels): 256 channels and two boxes of pixels to a tile. Each CTA holds its 128
// channels' weights and one box, an instruction reads both boxes, and each CTA's tensor memory takes its channels of both. Weights, most of what a
// tile loads, then serve twice the pixels that a CTA's shared memory and ring hold. The leader issues, all loads count on its barriers,
// commits arrive on both CTAs', and the second CTA's epilogue releases accumulators on the leader's (as in conv_tc.cu).
//
// Roles: warp 0 loads pixels, warp 1 issues MMAs and owns TMEM, warp 2 loads weights (a ring of its own, ahead of the previous kernel's
// end where the weights are old), the others are the epilogue: warp (quad, part) takes TMEM lanes = channels [32 quad, 32 quad + 32) and
// every second (int8: fourth) chunk of 32 columns. Two accumulators of 256 columns. Every wait is bounded.
//
// What bounds it: the instructions where N is large (142 clocks for N = 224 in a launch of seven tiles a CTA; 112 alone, with nothing else in shared
// memory), the issuing warp where it is small (elect_one in sm100.cuh; ~100 clocks for the hand-over of a group of taps; a loop that
// waited and committed per tap took 300 a tap), in fp32 launches of many tiles the epilogue's 4-byte accesses (~18 clocks per channel and 32
// pixels with a residual, as in the pixel-major kernel). Device time of a call, pixel-major kernel / this one, us: tf32 72 -> 120 3x3
// at 45x51, 9 images, with a residual 26.9 / 17.5 (135 tiles of 51x3 pixels in one wave, before 208 tiles of 51x2 in two); int8 128 -> 128 3x3
// at 28x28, 256 images 67.3 / 41.1 (a transposition of 13 us and single-byte stores fell away; 28x7 tiles, 1024 of them in seven waves).
// Into NHWC the gain is the loads of a 3x3 layer, one box for nine taps instead of nine: tf32 128 -> 128 3x3 at 28x28, 32 images, a launch
// of a plan 31.0 / 20.0 with a residual, 27.4 / 18.1 without; 256 images 130.8 / 98.5.
#include "conv_chmajor.cuh"

#include <cuda_bf16.h>

#include <climits>
#include <cstring>
#include <mutex>

#include "common.cuh"
#include "conv_epilogue.cuh"
#include "sm100.cuh"

namespace kxc_b200 {
namespace {

using namespace sm100;

// Epilogue warps: sixteen for int8, whose arithmetic bounds it; eight for fp32, whose threads then have the registers to keep two chunks of
// residual values in flight beside the one they work on.
template <MmaKind kKind>
constexpr int kEpiWarps = kKind == MmaKind::I8 ? 16 : 8;
template <MmaKind kKind>
constexpr int kThreads = (3 + kEpiWarps<kKind>) * 32;
constexpr int kRow = 128;               // bytes of a pixel's (a filter's) channel block
constexpr int kM = 128;                 // channels per tile
constexpr int kMaxN = 256;
constexpr int kMaxSlots = 8;
constexpr int kAccCols = 256;
constexpr int kChunk = 32;                                     // columns that an epilogue warp takes at a time
constexpr int kF32Tile = 32 * kChunk * 4;                      // a warp's staging tile: 32 channels
constexpr int kS8Pitch = kChunk + 4, kS8Tile = 32 * kS8Pitch;
constexpr int kSmemLimit = 227 * 1024 - 1024;                  // (static shared memory: barriers)

template <MmaKind kKind>
constexpr int kStagingBytes = kEpiWarps<kKind> * (kKind == MmaKind::I8 ? kS8Tile : kF32Tile);

// (pair form, as tma_load_4d_pair)
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap* m, uint32_t cluster_bar, int c0, int c1, int c2) {
    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst),
                 "l"(reinterpret_cast<uint64_t>(m)), "r"(cluster_bar), "r"(c0), "r"(c1), "r"(c2)
                 : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* m, uint32_t bar, int c0, int c1, int c2) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst),
                 "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
                 : "memory");
}

// Predicated accesses: a branch around each of a lane's stores cost 50 to 70 clocks, with 16 of them to a chunk of columns.
__device__ __forceinline__ float ldg_if(bool there, const float* a) {
    float v = 0.0f;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %1, 0;\n\t@p ld.global.nc.f32 %0, [%2];\n\t}" : "+f"(v) : "r"((int)there), "l"(a));
    return v;
}
__device__ __forceinline__ float4 ldg4_if(bool there, const float* a) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t@p ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%5];\n\t}"
                 : "+f"(v.x), "+f"(v.y), "+f"(v.z), "+f"(v.w) : "r"((int)there), "l"(a));
    return v;
}
__device__ __forceinline__ void stg_if(bool there, float* a, float v) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %0, 0;\n\t@p st.global.f32 [%1], %2;\n\t}" ::"r"((int)there), "l"(a), "f"(v));
}
__device__ __forceinline__ void stg4_if(bool there, float* a, float x, float y, float z, float w) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %0, 0;\n\t@p st.global.v4.f32 [%1], {%2, %3, %4, %5};\n\t}" ::"r"((int)there), "l"(a),
                 "f"(x), "f"(y), "f"(z), "f"(w));
}
__device__ __forceinline__ uint4 ldg16_if(bool there, const char* a) {
    uint4 v = make_uint4(0, 0, 0, 0);
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t@p ld.global.nc.v4.b32 {%0, %1, %2, %3}, [%5];\n\t}"
                 : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w) : "r"((int)there), "l"(a));
    return v;
}
__device__ __forceinline__ void stg16_if(bool there, char* a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %0, 0;\n\t@p st.global.v4.b32 [%1], {%2, %3, %4, %5};\n\t}" ::"r"((int)there), "l"(a),
                 "r"(x), "r"(y), "r"(z), "r"(w));
}
__device__ __forceinline__ void stg_word_if(bool there, int8_t* a, uint32_t v) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %0, 0;\n\t@p st.global.b32 [%1], %2;\n\t}" ::"r"((int)there), "l"(a), "r"(v));
}
__device__ __forceinline__ void stg_byte_if(bool there, int8_t* a, uint32_t v) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %0, 0;\n\t@p st.global.b8 [%1], %2;\n\t}" ::"r"((int)there), "l"(a), "r"(v));
}
// the formula for every shift, bias and accumulator, out of the way of the short one
__device__ __noinline__ uint32_t requantize_any(uint32_t acc, int32_t bias, int32_t mult, int32_t shift, int relu) {
    return (uint32_t)(uint8_t)requantize_s8((int32_t)(acc + (uint32_t)bias), mult, shift, relu);
}

// First result of a tile's box of pixels; a box beyond the last one (the second of a pair's last tile) lies beyond the last image.
struct Corner {
    int ow0, oh0, n0;
};
__device__ __forceinline__ Corner corner_of(const CmParams& p, int box) {
    const int row = (int)p.by_w.quotient((unsigned)box), n = (int)p.by_h.quotient((unsigned)row);
    return {(box - row * p.tiles_w) * p.BW, (row - n * p.tiles_h) * p.BH, n * p.BNI};
}

// One instruction of M = 128; the upper words of both descriptors are the same constant.
template <MmaKind kKind, bool kPair>
__device__ __forceinline__ void mma_step(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc, uint32_t accumulate) {
    if constexpr (kPair) umma_pair<kKind>(d, (uint64_t)hi << 32 | a_lo, (uint64_t)hi << 32 | b_lo, idesc, accumulate);
    else umma<kKind>(d, (uint64_t)hi << 32 | a_lo, (uint64_t)hi << 32 | b_lo, idesc, accumulate);
}
template <bool kPair>
__device__ __forceinline__ void commit(uint32_t bar) {
    if constexpr (kPair) umma_commit_pair(bar, 3);
    else umma_commit(bar);
}

// How results leave. Planes: the reference's layout, element by element, neighbouring lanes side by side. PlanesVec: rows, planes and
// pointers are such that four columns of an accumulator at a time are four consecutive elements of a plane or none, 16-byte accesses for
// fp32, words for int8. Pixels (bf16 and tf32 plans): NHWC, bf16 or fp32; the staging tile turns 32 channels x 32 pixels, and lanes take 16
// bytes of a pixel each.
enum class CmForm { Planes, PlanesVec, Pixels };
template <MmaKind kKind, CmForm kForm, bool kPair>
__global__ void __launch_bounds__(kThreads<kKind>, 1) conv_chmajor_kernel(const __grid_constant__ CmParams p) {
    constexpr bool kVec = kForm == CmForm::PlanesVec;
    constexpr int kCtas = kPair ? 2 : 1;
    static_assert(kForm != CmForm::Pixels || kKind != MmaKind::I8, "int8 results leave in planes");
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bar_px_full[kMaxSlots], bar_px_empty[kMaxSlots];
    __shared__ __align__(8) uint64_t bar_w_full[kMaxSlots], bar_w_empty[kMaxSlots];
    __shared__ __align__(8) uint64_t bar_acc_full[2], bar_acc_empty[2];
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);  // (a uniform value, as the compiler then knows)
    const int lane = threadIdx.x & 31;
    const int rank = kPair ? (int)cluster_cta_rank() : 0;
    // pixels, weights, staging: an MMA may read up to 15 rows past a pixel slot (N is rounded up) and up to 120 past a weight slot
    // (rows beyond the last channel); both stay inside this allocation, and those columns and rows are not stored
    const uint32_t px_smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t w_smem = px_smem + (uint32_t)(p.px_slots * p.px_slot_bytes);
    const uint32_t staging = w_smem + (uint32_t)(p.w_slots * p.w_slot_bytes);

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < p.px_slots; ++s) {
            mbar_init(smem_u32(&bar_px_full[s]), 1);
            mbar_init(smem_u32(&bar_px_empty[s]), 1);
        }
        for (int s = 0; s < p.w_slots; ++s) {
            mbar_init(smem_u32(&bar_w_full[s]), 1);
            mbar_init(smem_u32(&bar_w_empty[s]), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(smem_u32(&bar_acc_full[a]), 1);
            mbar_init(smem_u32(&bar_acc_empty[a]), kCtas * kEpiWarps<kKind>);
        }
        mbar_fence_init();
    }
    if (warp == 1) {
        if constexpr (kPair) {
            tmem_alloc_pair(smem_u32(&tmem_base_slot), 2 * kAccCols);
            tmem_relinquish_pair();
        } else {
            tmem_alloc(smem_u32(&tmem_base_slot), 2 * kAccCols);
            tmem_relinquish();
        }
    }
    if (p.zero_bytes > 0) {  // the halo behind a box, which no load writes
        uint8_t* boxes = smem_raw + (px_smem - smem_u32(smem_raw)) + p.px_bytes;
        for (int s = 0; s < p.px_slots; ++s)
            for (int i = (int)threadIdx.x * 16; i < p.zero_bytes; i += kThreads<kKind> * 16)
                *reinterpret_cast<uint4*>(boxes + (size_t)s * p.px_slot_bytes + i) = make_uint4(0, 0, 0, 0);
        fence_proxy_async_shared();
    }
    tc_fence_before_sync();
    __syncthreads();
    if constexpr (kPair) cluster_sync_all();  // the other CTA's barriers are initialised before anything signals them
    tc_fence_after_sync();
    const uint32_t tmem_base = tmem_base_slot;
    volatile int* abort_ptr = &abort_flag;
    pdl_launch_dependents();

    auto wait = [&](uint64_t* bar, uint32_t phase) { return mbar_wait_warp(smem_u32(bar), phase, abort_ptr); };
    const int items = p.tiles_c * ((p.tiles_w * p.tiles_h * p.tiles_n + kCtas - 1) / kCtas);
    const int first = kPair ? (int)(blockIdx.x >> 1) : (int)blockIdx.x, step = kPair ? (int)(gridDim.x >> 1) : (int)gridDim.x;

    if (warp == 0) {
        const bool lead = elect_one();
        if (lead) tma_prefetch_desc(&p.tmA[0]);
        pdl_wait();
        int slot = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (int item = first; ok && item < items; item += step) {
            const Corner t = corner_of(p, (int)p.by_c.quotient((unsigned)item) * kCtas + rank);
            for (int cb = 0; ok && cb < p.cblocks; ++cb)
                for (int l = 0; l < p.loads; ++l) {
                    if (!wait(&bar_px_empty[slot], phase ^ 1u)) {
                        ok = false;
                        break;
                    }
                    const uint32_t full = smem_u32(&bar_px_full[slot]);
                    const uint32_t dst = px_smem + (uint32_t)(slot * p.px_slot_bytes);
                    if (lead) {
                        if constexpr (kPair) {  // (both CTAs' bytes count on the leader's barrier)
                            if (rank == 0) mbar_arrive_expect_tx(full, 2u * (uint32_t)p.px_bytes);
                            tma_load_4d_pair(dst, &p.tmA[p.load_map[l]], map_to_cta(full, 0), cb * p.kb_elems, t.ow0 + p.load_w[l], t.oh0 + p.load_h[l], t.n0);
                        } else {
                            mbar_arrive_expect_tx(full, (uint32_t)p.px_bytes);
                            tma_load_4d(dst, &p.tmA[p.load_map[l]], full, cb * p.kb_elems, t.ow0 + p.load_w[l], t.oh0 + p.load_h[l], t.n0);
                        }
                    }
                    __syncwarp();
                    if (++slot == p.px_slots) { slot = 0; phase ^= 1u; }
                }
        }
    } else if (warp == 2) {
        const bool lead = elect_one();
        if (lead) tma_prefetch_desc(&p.tmW);
        if (!p.weights_ready) pdl_wait();
        int slot = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (int item = first; ok && item < items; item += step) {
            const int co0 = ((item - (int)p.by_c.quotient((unsigned)item) * p.tiles_c) * kCtas + rank) * kM;
            for (int cb = 0; ok && cb < p.cblocks; ++cb)
                for (int g = 0; g < p.groups; ++g) {
                    if (!wait(&bar_w_empty[slot], phase ^ 1u)) {
                        ok = false;
                        break;
                    }
                    const uint32_t full = smem_u32(&bar_w_full[slot]);
                    const int count = p.group[g].count;
                    if (lead) {
                        if (rank == 0) mbar_arrive_expect_tx(full, (uint32_t)(kCtas * count * p.w_tap_bytes));
                        for (int j = 0; j < count; ++j) {
                            const uint32_t dst = w_smem + (uint32_t)(slot * p.w_slot_bytes + j * p.w_tap_bytes);
                            if constexpr (kPair) tma_load_3d_pair(dst, &p.tmW, map_to_cta(full, 0), cb * p.kb_elems, co0, p.group[g].tap[j]);
                            else tma_load_3d(dst, &p.tmW, full, cb * p.kb_elems, co0, p.group[g].tap[j]);
                        }
                    }
                    __syncwarp();
                    if (++slot == p.w_slots) { slot = 0; phase ^= 1u; }
                }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            const bool lead = elect_one();
            const uint32_t idesc = make_instr_desc(kKind == MmaKind::F16 ? kFmtBF16 : (kKind == MmaKind::TF32 ? kFmtTF32 : kFmtS8),
                                                   kKind == MmaKind::I8 ? kAccS32 : kAccF32, (uint32_t)p.n_cols, kCtas * kM);
            const uint32_t hi = desc_hi(8 * kRow, kLayoutSw128);
            const uint32_t px_lo0 = desc_lo(px_smem, 16), w_lo0 = desc_lo(w_smem, 16);
            const uint32_t tap_step = (uint32_t)p.w_tap_bytes >> 4;
            const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
            const int groups = p.groups, w_slots = p.w_slots, px_slots = p.px_slots;
            int ps = 0, ws = 0, acc = 0;
            uint32_t pphase = 0, wphase = 0, acc_phase = 0;
            uint32_t px_lo = px_lo0, w_lo = w_lo0;
            bool ok = true;
            for (int item = first; ok && item < items; item += step) {
                if (!wait(&bar_acc_empty[acc], acc_phase ^ 1u)) break;
                tc_fence_after_sync();
                const uint32_t d = tmem + (uint32_t)(acc * kAccCols);
                uint32_t accumulate = 0;
                for (int cb = 0; ok && cb < p.cblocks; ++cb) {
                    const int steps = cb + 1 == p.cblocks ? p.last_steps : kRow / 32;
                    CmParams::Group g = p.group[0];
                    for (int i = 0; i < groups; ++i) {
                        const CmParams::Group next = p.group[i + 1];  // (one more than there are: read ahead of its use)
                        if ((g.first && !wait(&bar_px_full[ps], pphase)) || !wait(&bar_w_full[ws], wphase)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after_sync();
                        if (lead) {
#pragma unroll
                            for (int j = 0; j < CmParams::kMaxGroup; ++j) {
                                if (j >= g.count) break;
                                const uint32_t a = w_lo + (uint32_t)j * tap_step, b = px_lo + g.shift[j];
                                if (steps == kRow / 32) {
#pragma unroll
                                    for (int k = 0; k < kRow / 32; ++k) mma_step<kKind, kPair>(d, a + 2 * k, b + 2 * k, hi, idesc, k == 0 && j == 0 ? accumulate : 1u);
                                } else {
                                    mma_step<kKind, kPair>(d, a, b, hi, idesc, j == 0 ? accumulate : 1u);
                                    if (steps > 1) mma_step<kKind, kPair>(d, a + 2, b + 2, hi, idesc, 1u);
                                    if (steps > 2) mma_step<kKind, kPair>(d, a + 4, b + 4, hi, idesc, 1u);
                                }
                            }
                            commit<kPair>(smem_u32(&bar_w_empty[ws]));
                            if (g.last) commit<kPair>(smem_u32(&bar_px_empty[ps]));
                        }
                        __syncwarp();
                        accumulate = 1;
                        w_lo += (uint32_t)p.w_slot_bytes >> 4;
                        if (++ws == w_slots) { ws = 0; wphase ^= 1u; w_lo = w_lo0; }
                        if (g.last) {
                            px_lo += (uint32_t)p.px_slot_bytes >> 4;
                            if (++ps == px_slots) { ps = 0; pphase ^= 1u; px_lo = px_lo0; }
                        }
                        g = next;
                    }
                }
                if (!ok) break;
                if (lead) commit<kPair>(smem_u32(&bar_acc_full[acc]));
                __syncwarp();
                acc ^= 1;
                if (acc == 0) acc_phase ^= 1u;
            }
        }
    } else {
        constexpr int kEpiParts = kEpiWarps<kKind> / 4;
        constexpr int kMine = (kMaxN / kChunk + kEpiParts - 1) / kEpiParts;  // chunks of a warp at most
        const int quad = warp & 3, part = (warp - 3) >> 2;
        const int chunks = (p.n_cols + kChunk - 1) / kChunk;
        uint8_t* tile = smem_raw + (staging - smem_u32(smem_raw)) + (warp - 3) * (kKind == MmaKind::I8 ? kS8Tile : kF32Tile);
        const uint32_t plane = (uint32_t)(p.OH * p.OW);
        // A lane stores the columns from `col` on of a chunk (four with kVec, else one) for every kLanesC-th channel from `sub` on.
        constexpr int kLanesPx = kVec ? kChunk / 4 : kChunk, kLanesC = 32 / kLanesPx, kStores = 32 / kLanesC;
        const int col = lane % kLanesPx * (kVec ? 4 : 1), sub = lane / kLanesPx;
        // where those columns lie in their box: (second box) << 28 | image << 16 | row << 8 | column, -1: not a result
        int place[kMine];
#pragma unroll
        for (int i = 0; i < kMine; ++i) {
            int j = (part + i * kEpiParts) * kChunk + col;
            const int second = kPair && j >= p.n_cols / 2 ? 1 : 0;
            j -= second * (p.n_cols / 2);
            const int hw = p.HB * p.WB, n_l = j / hw, r = j - n_l * hw, h_l = r / p.WB, w_l = r - h_l * p.WB;
            place[i] = n_l < p.BNI && h_l < p.BH && w_l < p.BW ? second << 28 | n_l << 16 | h_l << 8 | w_l : -1;
        }
        // of this lane's channel, in the tile `held`: the bias; int8: also K = bias * M + rounding term as in requant_prepare, M, shift - 1
        int held = -1;
        [[maybe_unused]] float bias_f = 0.0f;
        [[maybe_unused]] int32_t bias = 0, mult = 0, shift = 2, down = 1;
        [[maybe_unused]] int64_t add = 0;
        [[maybe_unused]] bool fast = false;
        pdl_wait();  // residual reads and result writes must not overtake earlier kernels
        int acc = 0;
        uint32_t acc_phase = 0;
        for (int item = first; item < items; item += step) {
            const int group = (int)p.by_c.quotient((unsigned)item), ct = (item - group * p.tiles_c) * kCtas + rank;
            const Corner t = corner_of(p, group * kCtas);
            [[maybe_unused]] Corner t2 = t;
            if constexpr (kPair) t2 = corner_of(p, group * kCtas + 1);
            // the pixel of this lane's columns of chunk i, and whether there is one
            auto pixel_of = [&](int i, int* n, int* oh, int* ow) {
                int at = place[0];
#pragma unroll
                for (int k = 1; k < kMine; ++k) at = i == k ? place[k] : at;
                const bool second = kPair && (at >> 28 & 1) != 0;
                *n = (second ? t2.n0 : t.n0) + (at >> 16 & 0xfff); *oh = (second ? t2.oh0 : t.oh0) + (at >> 8 & 255); *ow = (second ? t2.ow0 : t.ow0) + (at & 255);
                return at >= 0 && *n < p.N && *oh < p.OH && *ow < p.OW;
            };
            const int c0 = ct * kM + quad * 32;
            const int nch = p.Cout - c0 < 32 ? p.Cout - c0 : 32;
            const uint32_t t_addr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(acc * kAccCols);
            // the element that this lane's columns of chunk i have in its first channel, and whether there is one
            auto pixel = [&](int i, uint32_t* off) {
                int n, oh, ow;
                const bool there = pixel_of(i, &n, &oh, &ow);
                *off = ((uint32_t)(n * p.Cout + c0 + sub) * (uint32_t)p.OH + (uint32_t)oh) * (uint32_t)p.OW + (uint32_t)ow;
                return there;
            };
            auto wait = [&] {
                const bool ok = __all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&bar_acc_full[acc]), acc_phase, abort_ptr));
                if (ok) tc_fence_after_sync();
                return ok;
            };
            auto release = [&] {  // this warp has read its part of the accumulator
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) {
                    if constexpr (kPair) mbar_arrive_cluster(map_to_cta(smem_u32(&bar_acc_empty[acc]), 0));
                    else mbar_arrive(smem_u32(&bar_acc_empty[acc]));
                }
            };
            const int mine = nch > 0 && part < chunks ? (chunks - part + kEpiParts - 1) / kEpiParts : 0;
            if constexpr (kForm == CmForm::Pixels) {
                constexpr int kElems = kKind == MmaKind::F16 ? 8 : 4, kLanes = 32 / kElems;  // channels of an access, lanes of a pixel
                constexpr int kPx = 32 / kLanes, kSteps = 32 / kPx;                         // pixels of a warp's access
                const int ch = lane % kLanes * kElems, px = lane / kLanes;
                const bool has_bias = p.bias != nullptr, has_res = p.residual != nullptr, relu = p.relu != 0, round = p.round_out_tf32 != 0;
                constexpr int kBytes = kKind == MmaKind::F16 ? 2 : 4;
                if (ct != held) {
                    held = ct;
                    if (has_bias) bias_f = lane < nch ? __ldg(p.bias + c0 + lane) : 0.0f;
                }
                // the element of this warp's first channel in the pixel of this lane's column, all ones: no pixel
                auto element = [&](int i) {
                    int n, oh, ow;
                    const bool there = pixel_of(i, &n, &oh, &ow);
                    const uint32_t e = ((uint32_t)(n * p.OH + oh) * (uint32_t)p.OW + (uint32_t)ow) * (uint32_t)p.Cout + (uint32_t)c0;
                    return there ? e : 0xffffffffu;
                };
                auto fetch = [&](int i, uint4(&res)[kSteps]) {
                    const uint32_t mine_at = element(i);
#pragma unroll
                    for (int k = 0; k < kSteps; ++k) {
                        const uint32_t e = __shfl_sync(0xffffffffu, mine_at, k * kPx + px);
                        res[k] = ldg16_if(e != 0xffffffffu && ch < nch, static_cast<const char*>(p.residual) + (size_t)(e + (uint32_t)ch) * kBytes);
                    }
                };
                uint4 res[kSteps] = {}, next[kSteps] = {};
                if (has_res && mine > 0) fetch(0, res);
                __syncwarp();
                if (!wait()) break;
#pragma unroll 1
                for (int i = 0; i < mine; ++i) {
                    uint32_t v[32];
                    tmem_ld_32x32(t_addr + (uint32_t)((part + i * kEpiParts) * kChunk), v);
                    if (has_res && i + 1 < mine) fetch(i + 1, next);
                    const uint32_t mine_at = element(i);
                    __syncwarp();
                    tmem_ld_wait();
                    if (i + 1 == mine) release();
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const float x = __uint_as_float(v[j]);
                        *reinterpret_cast<float*>(tile + j * 128 + lane * 4) = has_bias ? __fadd_rn(x, bias_f) : x;
                    }
                    __syncwarp();
#pragma unroll
                    for (int k = 0; k < kSteps; ++k) {
                        const uint8_t* row = tile + (k * kPx + px) * 128 + ch * 4;
                        float x[kElems];
#pragma unroll
                        for (int g = 0; g < kElems / 4; ++g) {
                            const float4 r = *reinterpret_cast<const float4*>(row + 16 * g);
                            x[4 * g] = r.x; x[4 * g + 1] = r.y; x[4 * g + 2] = r.z; x[4 * g + 3] = r.w;
                        }
                        const uint32_t rw[4] = {res[k].x, res[k].y, res[k].z, res[k].w};
                        if (has_res) {
#pragma unroll
                            for (int e = 0; e < kElems; ++e)
                                x[e] = __fadd_rn(x[e], kElems == 4 ? __uint_as_float(rw[e]) : ((e & 1) != 0 ? bf16_hi(rw[e >> 1]) : bf16_lo(rw[e >> 1])));
                        }
                        if (relu) {
#pragma unroll
                            for (int e = 0; e < kElems; ++e) x[e] = x[e] > 0.0f ? x[e] : 0.0f;
                        }
                        uint32_t o[4];
                        if constexpr (kElems == 8) {
#pragma unroll
                            for (int e = 0; e < 4; ++e) o[e] = pack_bf16(x[2 * e], x[2 * e + 1]);
                        } else {
#pragma unroll
                            for (int e = 0; e < 4; ++e) o[e] = __float_as_uint(round ? tf32_rne(x[e]) : x[e]);
                        }
                        const uint32_t e = __shfl_sync(0xffffffffu, mine_at, k * kPx + px);
                        stg16_if(e != 0xffffffffu && ch < nch, static_cast<char*>(p.out) + (size_t)(e + (uint32_t)ch) * kBytes, o[0], o[1], o[2], o[3]);
                    }
                    __syncwarp();
#pragma unroll
                    for (int k = 0; k < kSteps; ++k) res[k] = next[k];
                }
            } else if constexpr (kKind != MmaKind::I8) {
                const float* res_base = static_cast<const float*>(p.residual);
                float* out = static_cast<float*>(p.out);
                const bool has_bias = p.bias != nullptr, has_res = res_base != nullptr, relu = p.relu != 0;
                if (ct != held) {
                    held = ct;
                    if (has_bias) bias_f = lane < nch ? __ldg(p.bias + c0 + lane) : 0.0f;
                }
                auto fetch = [&](int i, float(&res)[32]) {
                    uint32_t off;
                    const bool valid = pixel(i, &off);
#pragma unroll
                    for (int k = 0; k < kStores; ++k, off += kLanesC * plane) {
                        const bool there = valid && kLanesC * k + sub < nch;
                        if constexpr (kVec) {
                            const float4 r = ldg4_if(there, res_base + off);
                            res[4 * k] = r.x; res[4 * k + 1] = r.y; res[4 * k + 2] = r.z; res[4 * k + 3] = r.w;
                        } else {
                            res[k] = ldg_if(there, res_base + off);
                        }
                    }
                };
                float res[32] = {}, next[32] = {};
                if (has_res && mine > 0) fetch(0, res);
                __syncwarp();
                if (!wait()) break;
#pragma unroll 1
                for (int i = 0; i < mine; ++i) {
                    uint32_t v[32];
                    tmem_ld_32x32(t_addr + (uint32_t)((part + i * kEpiParts) * kChunk), v);
                    if (has_res && i + 1 < mine) fetch(i + 1, next);
                    __syncwarp();
                    tmem_ld_wait();
                    if (i + 1 == mine) release();
                    // in: lane = channel, 128-byte rows, 16-byte piece g of row r at g ^ (r & 7) (no bank conflicts either way)
#pragma unroll
                    for (int g = 0; g < 8; ++g) {
                        float4 o;
                        o.x = __uint_as_float(v[4 * g]); o.y = __uint_as_float(v[4 * g + 1]);
                        o.z = __uint_as_float(v[4 * g + 2]); o.w = __uint_as_float(v[4 * g + 3]);
                        if (has_bias) {
                            o.x = __fadd_rn(o.x, bias_f); o.y = __fadd_rn(o.y, bias_f);
                            o.z = __fadd_rn(o.z, bias_f); o.w = __fadd_rn(o.w, bias_f);
                        }
                        *reinterpret_cast<float4*>(tile + lane * 128 + ((g ^ (lane & 7)) << 4)) = o;
                    }
                    __syncwarp();
                    float x[32];
#pragma unroll
                    for (int k = 0; k < kStores; ++k) {
                        const int c = kLanesC * k + sub;
                        const uint8_t* row = tile + c * 128 + (((col >> 2) ^ (c & 7)) << 4);
                        if constexpr (kVec) {
                            const float4 r = *reinterpret_cast<const float4*>(row);
                            x[4 * k] = r.x; x[4 * k + 1] = r.y; x[4 * k + 2] = r.z; x[4 * k + 3] = r.w;
                        } else {
                            x[k] = *reinterpret_cast<const float*>(row + (col & 3) * 4);
                        }
                    }
                    __syncwarp();
                    if (has_res) {
#pragma unroll
                        for (int k = 0; k < 32; ++k) x[k] = __fadd_rn(x[k], res[k]);
                    }
                    if (relu) {
#pragma unroll
                        for (int k = 0; k < 32; ++k) x[k] = fmaxf(x[k], 0.0f);  // (NaN and -0 give 0, as x > 0 ? x : 0 does)
                    }
                    uint32_t off;
                    const bool valid = pixel(i, &off);
#pragma unroll
                    for (int k = 0; k < kStores; ++k, off += kLanesC * plane) {
                        const bool there = valid && kLanesC * k + sub < nch;
                        if constexpr (kVec) stg4_if(there, out + off, x[4 * k], x[4 * k + 1], x[4 * k + 2], x[4 * k + 3]);
                        else stg_if(there, out + off, x[k]);
                    }
#pragma unroll
                    for (int k = 0; k < 32; ++k) res[k] = next[k];
                }
            } else {
                if (ct != held) {
                    held = ct;
                    bias = 0; mult = 0; shift = 2;
                    if (lane < nch) {
                        bias = __ldg(p.bias_i32 + c0 + lane);
                        mult = __ldg(p.multiplier + c0 + lane);
                        shift = __ldg(p.shift + c0 + lane);
                    }
                    int4 q;
                    fast = __all_sync(0xffffffffu, requant_prepare(bias, mult, shift, p.max_abs_acc, &q) && p.max_abs_acc < (1ll << 31));
                    add = (int64_t)(((uint64_t)(uint32_t)q.z << 32) | (uint32_t)q.y);
                    down = q.w;
                }
                const int32_t lo_cap = p.relu ? 0 : INT32_MIN;
                if (!wait()) break;
#pragma unroll 1
                for (int i = 0; i < mine; ++i) {
                    uint32_t v[32], w[8];
                    tmem_ld_32x32(t_addr + (uint32_t)((part + i * kEpiParts) * kChunk), v);
                    tmem_ld_wait();
                    if (i + 1 == mine) release();
                    if (fast) {
#pragma unroll
                        for (int g = 0; g < 8; ++g) {
                            int32_t r[4];
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                const int32_t hi = (int32_t)(((int64_t)(int32_t)v[4 * g + k] * mult + add) >> 32);
                                r[k] = max(hi >> down, lo_cap);
                            }
                            uint32_t hi16;
                            asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(hi16) : "r"(r[3]), "r"(r[2]), "r"(0));
                            asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(w[g]) : "r"(r[1]), "r"(r[0]), "r"(hi16));
                        }
                    } else {
#pragma unroll
                        for (int g = 0; g < 8; ++g) {
                            w[g] = 0;
#pragma unroll
                            for (int k = 0; k < 4; ++k)
                                w[g] |= requantize_any(v[4 * g + k], bias, mult, shift, p.relu) << (8 * k);
                        }
                    }
#pragma unroll
                    for (int g = 0; g < 8; ++g) *reinterpret_cast<uint32_t*>(tile + lane * kS8Pitch + 4 * g) = w[g];
                    __syncwarp();
                    uint32_t off;
                    const bool valid = pixel(i, &off);
                    int8_t* out = static_cast<int8_t*>(p.out);
                    if constexpr (kVec) {
                        uint32_t x[kStores];
#pragma unroll
                        for (int k = 0; k < kStores; ++k) x[k] = *reinterpret_cast<const uint32_t*>(tile + (kLanesC * k + sub) * kS8Pitch + col);
#pragma unroll
                        for (int k = 0; k < kStores; ++k, off += kLanesC * plane)
                            stg_word_if(valid && kLanesC * k + sub < nch, out + off, x[k]);
                    } else {
                        uint32_t x[kStores];
#pragma unroll
                        for (int k = 0; k < kStores; ++k) x[k] = tile[k * kS8Pitch + lane];
#pragma unroll
                        for (int k = 0; k < kStores; ++k, off += plane)
                            stg_byte_if(valid && k < nch, out + off, x[k]);
                    }
                    __syncwarp();
                }
            }
            if (mine == 0) release();
            acc ^= 1;
            if (acc == 0) acc_phase ^= 1u;
        }
    }

    if (*abort_ptr) {  // loads in flight may still land in shared memory: give them time (bounded) before it is released
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    tc_fence_before_sync();
    __syncthreads();
    // neither CTA of a pair may release its tensor or shared memory while the other one can still signal or read it
    if constexpr (kPair) cluster_sync_all();
    tc_fence_after_sync();
    if (warp == 1) {
        __syncwarp();
        if constexpr (kPair) tmem_dealloc_pair(tmem_base, 2 * kAccCols);
        else tmem_dealloc(tmem_base, 2 * kAccCols);
    }
    if (threadIdx.x == 0 && *abort_ptr && p.status != nullptr) atomicExch(p.status, KXC_B200_ERR_DEVICE_WAIT);
}

template <MmaKind kKind, CmForm kForm, bool kPair>
int32_t launch(const CmParams& p, cudaStream_t stream) {
    static PerDeviceOnce smem_once;
    auto kernel = conv_chmajor_kernel<kKind, kForm, kPair>;
    KXC_TRY(smem_opt_in(smem_once, kernel, kSmemLimit));
    const int ctas = kPair ? 2 : 1;
    const long long boxes = (long long)p.tiles_w * p.tiles_h * p.tiles_n, items = p.tiles_c * ((boxes + ctas - 1) / ctas);
    if (items <= 0) return KXC_B200_OK;
    const int bytes = 1024 + p.px_slots * p.px_slot_bytes + p.w_slots * p.w_slot_bytes + kStagingBytes<kKind>;
    if (bytes > kSmemLimit || boxes + 1 > INT_MAX || items > INT_MAX) return fail(KXC_B200_ERR_INVALID, "channel-major conv: %d bytes of shared memory, %lld tiles", bytes, items);
    // (pairs: as many as are resident at once, every form of these kernels takes an SM to itself)
    const int units = kPair ? tc_split_capacity(2) : kNumSMs;
    if (units <= 0) return fail(KXC_B200_ERR_CUDA, "channel-major conv: no room for CTA pairs");
    KXC_CUDA_TRY(launch_kernel(kernel, dim3((unsigned)(ctas * (items < units ? items : units))), dim3(kThreads<kKind>), bytes, stream, /*pdl=*/true, ctas, p));
    return check_launch("conv_chmajor_kernel");
}

template <MmaKind kKind>
int32_t launch_kind(const CmParams& p, cudaStream_t stream) {
    // four columns at a time: every row of a result plane starts and ends on a multiple of four, in the accumulator (WB) as in memory
    const uintptr_t addr = reinterpret_cast<uintptr_t>(p.out) | reinterpret_cast<uintptr_t>(p.residual);
    const bool vec = (p.OW & 3) == 0 && (p.BW & 3) == 0 && (p.WB & 3) == 0 && (addr & (kKind == MmaKind::I8 ? 3u : 15u)) == 0;
    if constexpr (kKind != MmaKind::I8) {
        if (p.pixels) {
            if ((addr & 15u) != 0 || p.Cout % (kKind == MmaKind::F16 ? 8 : 4) != 0) return fail(KXC_B200_ERR_INVALID, "channel-major conv: NHWC results need 16-byte pixels");
            return p.ctas == 2 ? launch<kKind, CmForm::Pixels, true>(p, stream) : launch<kKind, CmForm::Pixels, false>(p, stream);
        }
    }
    return vec ? launch<kKind, CmForm::PlanesVec, false>(p, stream) : launch<kKind, CmForm::Planes, false>(p, stream);
}

int div_up(int a, int b) { return (a + b - 1) / b; }
// work items of a launch: tiles of one CTA, or of a pair
long long tiles(const CmGeometry& g, int BW, int BH, int BNI, int ctas) {
    const long long boxes = (long long)div_up(g.OW, BW) * div_up(g.OH, BH) * div_up(g.N, BNI);
    return (long long)div_up(g.Cout, ctas * kM) * ((boxes + ctas - 1) / ctas);
}
long long tiles(const CmPlan& plan) { return tiles(plan.g, plan.c.BW, plan.c.BH, plan.c.BNI, plan.c.ctas); }
int floor_half(int v) { return (v - (v & 1)) / 2; }

// The taps of a filter as loads: those that share a box (all of them at stride 1, those of one row and column parity at stride 2) or
// each by itself. Offsets are from the tile's first pixel, in pixels of the load's map.
struct Grouping {
    int loads = 0, most = 0;                  // most taps of a load
    int extra_h = 0, extra_w = 0;             // how much larger than the tile a box is
    int first[CmParams::kMaxLoads], map[CmParams::kMaxLoads], h[CmParams::kMaxLoads], w[CmParams::kMaxLoads];
    int taps = 0, index[CmParams::kMaxTaps], dh[CmParams::kMaxTaps], dw[CmParams::kMaxTaps];
};
bool group_taps(const CmGeometry& g, bool shared, Grouping* out) {
    if (g.KH * g.KW > CmParams::kMaxTaps || (!shared && g.KH * g.KW > CmParams::kMaxLoads)) return false;
    for (int par = 0; par < (g.stride == 2 ? 4 : 1); ++par) {
        bool open = false;
        for (int kh = 0; kh < g.KH; ++kh)
            for (int kw = 0; kw < g.KW; ++kw) {
                int dh = kh * g.dil_h - g.pad_h, dw = kw * g.dil_w - g.pad_w;
                if (g.stride == 2) {
                    if ((dh & 1) * 2 + (dw & 1) != par) continue;
                    dh = floor_half(dh);
                    dw = floor_half(dw);
                }
                if (!shared || !open) {  // (taps come in ascending order: the first one has the smallest row, and below its column)
                    out->first[out->loads] = out->taps;
                    out->map[out->loads] = par;
                    out->h[out->loads] = dh;
                    out->w[out->loads] = dw;
                    ++out->loads;
                    open = true;
                }
                const int l = out->loads - 1;
                if (out->taps - out->first[l] + 1 > out->most) out->most = out->taps - out->first[l] + 1;
                out->index[out->taps] = kh * g.KW + kw;
                out->dh[out->taps] = dh - out->h[l];
                out->dw[out->taps] = dw - out->w[l];
                if (out->dh[out->taps] > out->extra_h) out->extra_h = out->dh[out->taps];
                if (out->dw[out->taps] > out->extra_w) out->extra_w = out->dw[out->taps];
                ++out->taps;
            }
    }
    return true;
}

struct Box {
    double cost = -1.0, clocks = -1.0;
    int BW = 0, BH = 0, BNI = 0, HB = 0, WB = 0, n = 0, zero_rows = 0, px_slots = 0, w_slots = 0, group = 0;
};

// Columns of a loaded box: a multiple of four where the rows of the result are (kVec). A pair's box that spans the plane shares its padding: what
// lies behind a row, and behind an image, is what lies before the next one, and a tap's view runs on into it (7x7 planes of a 3x3
// filter: 8x8 pixels instead of 9x9, two images in 119 columns instead of 142).
int box_width(const CmGeometry& g, const Grouping& t, int ctas, int BW) {
    if (ctas == 2) return BW + t.extra_w - (g.stride == 1 && BW == g.OW && t.extra_w >= g.pad_w ? g.pad_w : 0);
    return (g.OW & 3) == 0 && (BW & 3) == 0 ? div_up(BW + t.extra_w, 4) * 4 : BW + t.extra_w;
}
int box_height(const CmGeometry& g, const Grouping& t, int ctas, int BH) {
    return BH + t.extra_h - (ctas == 2 && g.stride == 1 && BH == g.OH && t.extra_h >= g.pad_h ? g.pad_h : 0);
}

// Modelled cycles of a launch and the slots of its rings for one tile box; false where shared memory does not hold it.
bool box_cost(const CmGeometry& g, const Grouping& t, int staging, int ctas, int BW, int BH, int BNI, Box* b) {
    b->BW = BW; b->BH = BH; b->BNI = BNI;
    b->HB = box_height(g, t, ctas, BH); b->WB = box_width(g, t, ctas, BW);
    const int n = ((BNI - 1) * b->HB + BH - 1) * b->WB + BW;  // the last pixel's flat place, and one
    const int step = 16 / ctas;  // (of a pair's columns each CTA's box has half)
    if (n > kMaxN / ctas || b->WB > 256 || b->HB > 256) return false;
    b->n = div_up(n, step) * step;
    const int rows_w = g.Cout < kM ? div_up(g.Cout, 8) * 8 : kM, rows_px = b->HB * b->WB * BNI;
    const int last = n + t.extra_h * b->WB + t.extra_w;  // rows that the last tap's view reaches
    b->zero_rows = ctas == 2 && last > rows_px ? last - rows_px : 0;
    const int px_bytes = div_up((rows_px + b->zero_rows) * kRow, 1024) * 1024, tap_bytes = rows_w * kRow;
    const int budget = kSmemLimit - 1024 - staging;
    int px_slots, w_slots;
    b->group = 1;
    if (t.taps == t.loads) {
        px_slots = w_slots = budget / (px_bytes + tap_bytes);
    } else {
        // the taps that share a box in as few groups as leave two slots of each ring; what is left goes to the pixels, then the weights
        b->group = t.most < CmParams::kMaxGroup ? t.most : (t.most % 3 == 0 ? 3 : CmParams::kMaxGroup);
        px_slots = 2;
        while (b->group > 1 && 2 * (px_bytes + b->group * tap_bytes) > budget) --b->group;
        w_slots = (budget - 2 * px_bytes) / (b->group * tap_bytes);
        while (px_slots < 4 && (budget - (px_slots + 1) * px_bytes) / (b->group * tap_bytes) >= 3) w_slots = (budget - ++px_slots * px_bytes) / (b->group * tap_bytes);
    }
    if (px_slots < 2 || w_slots < 2) return false;
    b->px_slots = px_slots < kMaxSlots ? px_slots : kMaxSlots;
    b->w_slots = w_slots < kMaxSlots ? w_slots : kMaxSlots;
    int groups = 0;
    for (int l = 0; l < t.loads; ++l) groups += div_up((l + 1 < t.loads ? t.first[l + 1] : t.taps) - t.first[l], b->group);
    const long long items = tiles(g, BW, BH, BNI, ctas);
    // What a tile costs: its rows at the rate the copies reach shared memory, or its instructions, 64 + n / 2 clocks each, and the hand-over of a
    // group; then its epilogue, which overlaps the next tile. (Boxes chosen so over 200 drawn layers. A fit of the loops of one lane: the boxes of single CTAs, and the
    // lines of cm_wanted but that of the pairs, still go by it.)
    const double fill = (double)g.cblocks * ((double)t.loads * rows_px + (double)t.taps * rows_w) * 2.6;
    const double mma = (double)t.taps * ((g.cblocks - 1) * 4 + g.last_steps) * (64.0 + 0.5 * b->n);
    const double main_loop = (fill > mma ? fill : mma) + 100.0 * g.cblocks * groups;
    const double epilogue = 1500.0 + 700.0 * div_up(div_up(b->n, kChunk), g.epi_parts);
    const double waves = (double)((items + kNumSMs / ctas - 1) / (kNumSMs / ctas));
    b->cost = main_loop + (waves - 1.0) * (main_loop > epilogue ? main_loop : epilogue) + epilogue + 1e-3 * (double)items;
    // The same in clocks of 1.85 GHz, with what a launch costs besides: fitted to 753 launches of 381 drawn layers in either form (9 to 12 % rms) after the
    // loops had come to run on whole warps; for the choice between pairs and the others. (A pair's instruction takes a clock for each
    // column of a box, 45 at least; a single one half that.)
    if (g.eb > 1) {
        const bool pair = ctas == 2;
        const double rows = (double)g.cblocks * ((double)t.loads * rows_px + (double)t.taps * rows_w) * (pair ? 0.82 : 1.15);
        const double steps = (double)t.taps * ((g.cblocks - 1) * 4 + g.last_steps) * (pair ? (b->n > 45 ? b->n : 45.0) : 4.0 + 0.463 * b->n);
        const double loop = (rows > steps ? rows : steps) + (pair ? 190.0 : 553.0) * g.cblocks * groups;
        const double end = 390.0 + (!g.pixels ? 2600.0 : (g.eb == 2 ? 1610.0 : 2730.0)) * div_up(div_up(b->n * ctas, kChunk), g.epi_parts);
        b->clocks = (pair ? 6580.0 : 2810.0) + loop + (waves - 1.0) * (loop > end ? loop : end) + end;
    }
    return true;
}

// The tile box of a launch, of single CTAs or of pairs; false where the form does not apply.
bool choose(CmPlan* plan, TcDType dtype, const ConvDims& d, bool pixels, int ctas) {
    CmGeometry* g = &plan->g;
    CmChoice* best = &plan->c;
    const int eb = tc_elem_bytes(dtype), N = d.N, C = d.C, KH = d.KH, KW = d.KW;
    g->N = N; g->H = d.H; g->W = d.W; g->Cout = d.O; g->KH = KH; g->KW = KW; g->stride = d.SH;
    g->pad_h = d.PH; g->pad_w = d.PW; g->dil_h = d.DH; g->dil_w = d.DW;
    g->OH = d.OH; g->OW = d.OW; g->pixels = pixels ? 1 : 0; g->eb = eb;
    // (elements are counted in 32 bits)
    if (d.SH != d.SW || (d.SH != 1 && d.SH != 2) || g->OH <= 0 || g->OW <= 0 || (unsigned long long)N * d.O * g->OH * g->OW >= (1ull << 32)) return false;
    g->kb_elems = kRow / eb;
    g->cblocks = div_up(C, g->kb_elems);
    g->last_steps = div_up((C - (g->cblocks - 1) * g->kb_elems) * eb, 32);
    g->epi_parts = (dtype == kTcS8 ? kEpiWarps<MmaKind::I8> : kEpiWarps<MmaKind::F16>) / 4;
    const int staging = dtype == kTcS8 ? kStagingBytes<MmaKind::I8> : kStagingBytes<MmaKind::F16>;
    best->cost = -1.0;
    best->ctas = ctas;
    const int columns = kMaxN / ctas;
    for (int shared = ctas == 2 ? 1 : 0; shared < 2; ++shared) {
        Grouping t;
        if ((shared && KH * KW == 1) || !group_taps(*g, shared != 0, &t)) continue;
        // widths and heights that divide the plane evenly, from the widest that fits down
        for (int tw = div_up(d.OW, columns), last_w = 0; tw <= d.OW; ++tw) {
            const int BW = (d.OW & 3) == 0 ? div_up(div_up(d.OW, tw), 4) * 4 : div_up(d.OW, tw);
            if (BW == last_w) continue;
            last_w = BW;
            if (BW < 8 && tw > 1) break;
            if (BW > columns) continue;
            const int WB = box_width(*g, t, ctas, BW), most_h = (columns - BW) / WB + 1;
            for (int th = div_up(d.OH, most_h), last_h = 0; th <= d.OH; ++th) {
                const int BH = div_up(d.OH, th);
                if (BH == last_h) continue;
                last_h = BH;
                if (th > 1 && BW * BH < 48 / ctas && best->cost >= 0.0) break;
                int most = 1;
                if (BH == d.OH) {
                    most = 1 + (columns - ((BH - 1) * WB + BW)) / (box_height(*g, t, ctas, BH) * WB);
                    if (most > N) most = N;
                }
                for (int bni = most; bni >= 1; bni = bni > 1 ? bni / 2 : 0) {
                    Box b;
                    if (!box_cost(*g, t, staging, ctas, BW, BH, bni, &b)) continue;
                    if (best->cost < 0.0 || (ctas == 2 ? b.clocks < best->clocks : b.cost < best->cost)) {
                        best->cost = b.cost; best->clocks = b.clocks;
                        best->shared = shared;
                        best->BW = BW; best->BH = BH; best->BNI = bni; best->HB = b.HB; best->WB = b.WB; best->n = b.n; best->zero_rows = b.zero_rows;
                        best->px_slots = b.px_slots; best->w_slots = b.w_slots; best->group = b.group;
                    }
                }
            }
        }
    }
    return best->cost >= 0.0;
}

}  // namespace

// Integers take this form wherever it applies: of 260 drawn layers (device time of a call, against the pixel-major forms of results in planes: byte
// stores, or NHWC and a transposition) it was the faster one by 1.32 in the geometric mean; seven lost more than 2 %, 1x1 layers to 32 and fewer
// channels up to 6 % (53 -> 8 of stride 2 at 80x78, 68 images: 19.2 -> 20.4), 180 -> 17 3x3 at 16x16, 51 images 12.6 -> 15.4, 64 -> 64 3x3 at 12x13,
// 165 images 12.2 -> 14.0. A model of the pixel-major forms, fitted to the same layers, chose worse than not choosing.
//
// With fp32 results into planes the pixel-major kernel has less to hand over per K block, splits long reductions of few tiles over
// clusters and takes 64 channels at a time, so modelled clocks decide. Its model ends with the last K block; 30 clocks per channel of a
// tile stand for the epilogue of an unsplit one. Over 225 drawn layers (operators with a residual and graph outputs, tf32 and bf16) the choice was
// 5.6 % ahead of the pixel-major kernel alone; six lost more than 2 %, one-wave 1x1 layers at the line up to 19 % (tf32 32 -> 505 at 21x20, 7 images
// 6.9 / 8.5, bf16 436 -> 442 at 17x17, 13 images 12.4 / 13.1), 384 -> 61 1x1 at 57x54, 24 images, bf16, 57.7 / 63.5. Few channels (24 -> 30
// 3x3 at 92x95, 32 images, 12 % slower) leave three quarters of the epilogue's warps idle in a launch that it bounds: those keep the pixel-major kernel.
// One wave of 1x1 tiles, which share no loads, has to be further ahead: tf32 322 -> 473 at 19x22, 8 images 14.9 pixel-major / 17.1 us, 311 -> 448 of
// stride 2 at 39x40, 9 images 18.7 / 21.2, bf16 141 -> 129 at 84x84, 2 images 13.6 / 14.8; 110 -> 364 at 14x13, 15 images 11.6 / 11.3 and all of 22 drawn
// layers of more waves (0.997 to 1.8 times) still take this form. Where the pixel-major kernel's K blocks are narrower than 128 bytes (up to 32 bf16 or
// 16 tf32 channels) its main loop is not modelled: those layers stay with it unless this whole launch is shorter than that epilogue (2 of 340
// drawn ones; bf16 22 -> 254 1x1 at 28x29, 20 images, 13.3 / 10.4). Of 160 forced over, 1x1 layers to few channels lost, up to 0.69 times as
// fast, and wide filters gained, 1.18 times in the mean of all: a model for them has yet to be fitted.
//
// NHWC results (layers of plans): each form's modelled clocks, the pixel-major one's with its epilogue, weighted by what launches of plans
// measured. 3x3 layers, whose pixels the pixel-major kernel loads nine times over, are ahead of their model: tf32 128 -> 128 at 28x28 and
// 256 -> 256 at 14x14 gained up to the line, 512 -> 512 at 7x7 (two images to a tile, the weights' rows bound both forms) lost where the model said
// so: 32 images 39.7 / 77.1 us, 256 images 103.5 / 154.0. Split reductions of 1x1 layers lose 8 to 17 % up to a ratio of 1 (64 x 768 -> 160 at 7x7
// 14.2 / 15.2) and gain from 1.15 on. Splits of wider filters over three and more CTAs are left only where the models cross; 40 drawn layers
// of ratios 0.86 to 1.02 were 0.985 to 1.43 times as fast here (bf16 192 -> 160 3x3 at 13x11, 28 images, ratio 0.997: 18.9 / 15.2 us). Launches of one channel
// block that read and write more than they multiply are the epilogue's, of which 32 channels use a quarter: tf32 1x1 layers up to a ratio
// of 1.5 (32 -> 32 at 90x88, 45 images 161.8 / 225.8, 32 -> 40 at 76x79, 56 images 160.8 / 174.1; all 23 drawn ones lost) and 3x3 layers of 17 to 32 channels
// from about 100 tiles on (32 -> 32 at 40x42, 61 images 66.9 / 81.2, 0.82 to 1.10; fewer tiles 1.04 to 1.18), bf16 1x1 layers of 17 to 32 channels and more
// than one wave (64 -> 32 at 95x95, 33 images 92.4 / 100.4, 0.92 to 0.95; 16 channels gain 16 to 23 %). bf16 1x1 layers to
// more channels gain from a ratio of 1.6 on (1.0 to 1.25 times, with a residual and without; below it 0.92 to 1.02: 384 -> 384 at 17x14, 63 images, 52.0 /
// 56.4). Of 840 drawn layers these lines let 264 through, which were 1.12 times as fast (seven lost more than 3 %, the worst tf32 64 -> 32 3x3 of stride 2 at
// 45x48, 39 images, 29.5 / 32.6).
// CTA pairs: 3x3 layers of stride 1 and at least four channel blocks, where their fitted clocks (box_cost) are 5.5 % below the other form's
// (tc_modelled_clocks, or those of single CTAs), not where the reduction is split over three and more. Of 200 drawn layers and those of ResNet-18 at 1 to 512
// images 73 took them, 1.12 times as fast in the mean (0.86 to 1.37; four lost more than 3 %): 512 -> 512 at 7x7, 64 images, bf16 23.2 / 16.9 us (split
// in two), tf32 35.3 / 28.1; 256 -> 256 at 14x14, 128 images, 28.7 / 25.7 and 52.6 / 45.0. 110 others that took them: 1.12 (0.93 to 1.37, two lost more than
// 3 %), 48 of other paddings and dilations 1.08 (0.93 to 1.33, six). With fewer channel blocks they lost up to 20 % (32 -> 256 at
// 17x15, 97 images, tf32 15.8 / 19.9), at stride 2 up to 35 % (256 -> 512 at 14x14, 256 images, tf32 52.7 / 71.2), with 5x5 filters up to 40 %; into planes one
// of 71 layers gained, int8 planes lost 13 % in the mean. Filters of two to nine taps that are not 3x3, which the fit has none of: 80 that it would take
// over were 0.97 times as fast in the mean (288 -> 288 1x5 at 15x17, 41 images, tf32 27.4 / 42.7; 192 -> 192 5x1 at 17x15, 118 images, 28.9 / 42.4).
// ResNet-18 tf32 32 images 476.8 / 419.6 us, 64: 739 / 661, 256: 2156 / 2028; bf16 32: 265.7 / 254.2, 128: 552 / 545. bf16 layers of stride 2
// keep the pixel-major kernel: with a 1x1 layer beside them they are one launch of it (two outputs), and alone they give the same bits as there.
const CmPlan* cm_wanted(TcDType dtype, const ConvDims& d, int weights_ready, TcOutMode out_mode, bool residual) {
    // The choices of the last geometries: sets of four, so that the layers of a network called one by one keep theirs (of 11 ResNet-18 layers
    // in 128 single entries, two met in 45 of 128 combinations of batch and precision, and each call of these chose anew: 3 to 20 us).
    struct Entry {
        int key[18] = {-1};
        bool use = false;
        CmPlan plan;
    };
    struct Set {
        Entry way[4];
        unsigned next = 0;
    };
    static thread_local Set sets[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    const int key[18] = {(int)dtype, d.N, d.C, d.H, d.W, d.O, d.KH, d.KW, d.SH, d.SW, d.PH, d.PW, d.DH, d.DW, weights_ready, (int)out_mode, (int)residual, dev};
    uint32_t hash = 0;  // (each step carries the upper bits down: extents are multiples of large powers of two)
    for (const int v : key) {
        hash = (hash ^ (uint32_t)v) * 0x9e3779b1u;
        hash ^= hash >> 15;
    }
    Set& set = sets[hash % 64];
    for (Entry& w : set.way)
        if (memcmp(w.key, key, sizeof(key)) == 0) return w.use ? &w.plan : nullptr;
    Entry& e = set.way[set.next++ % 4];  // (in turn: the oldest)
    memcpy(e.key, key, sizeof(key));
    const bool pixels = out_mode == kOutNHWC_BF16 || out_mode == kOutNHWC_F32;
    e.use = choose(&e.plan, dtype, d, pixels, 1);
    if (e.use && dtype != kTcS8) {
        TcParams p{};
        TcConfig cfg{};
        int word = 0;
        p.weights_ready = weights_ready;
        void* placeholder = reinterpret_cast<void*>((uintptr_t)4096);  // (an address for the tensor maps of a launch that is not made)
        const int32_t rc = tc_setup_conv(&p, &cfg, dtype, out_mode, placeholder, placeholder, d.N, d.H, d.W, tc_channel_pad(dtype, d.C), d.O, d.KH,
                                         d.KW, d.SH, d.PH, d.PW, d.DH, d.DW, &word);
        if (out_mode == kOutNCHW_F32) {
            const double epilogue = p.split > 1 ? 0.0 : 30.0 * (d.O < cfg.bn ? d.O : cfg.bn);
            const CmChoice& c = e.plan.c;
            const double ahead = d.KH * d.KW == 1 && tiles(e.plan) <= kNumSMs ? 2800.0 : 1000.0;
            e.use = rc == KXC_B200_OK && (d.O > 32 || e.plan.g.cblocks > 1) && c.cost + ahead < cfg.clocks + epilogue;
        } else {
            const double ahead = d.KH * d.KW == 1 ? (p.split > 1 ? 1.15 : (dtype == kTcBF16 && d.O > 32 ? 1.6 : 0.80))
                                                  : (p.split > 2 ? 1.0 : (d.SH == 1 ? 0.83 : 0.95));
            const long long items = tiles(e.plan);
            const bool few = d.O > 16 && d.O <= 32;  // channels
            bool stays = dtype == kTcBF16 && d.SH == 2;
            if (e.plan.g.cblocks == 1 && d.SH == 1) {
                if (dtype == kTcTF32) stays = d.KH * d.KW == 1 ? cfg.clocks < 1.5 * e.plan.c.cost : few && d.KH * d.KW <= 9 && items > 100;
                else if (few && d.KH * d.KW == 1 && items > kNumSMs) stays = true;
            }
            e.use = rc == KXC_B200_OK && cfg.clocks >= ahead * e.plan.c.cost && !stays;
            CmPlan pair;
            if (rc == KXC_B200_OK && d.O > kM && e.plan.g.cblocks >= 4 && d.KH == 3 && d.KW == 3 && d.SH == 1 && p.split <= 2 && tc_cta_pairs() && tc_split_capacity(2) > 0 &&
                choose(&pair, dtype, d, true, 2)) {
                const double other = e.use ? e.plan.c.clocks : tc_modelled_clocks(p, cfg, residual);
                if (pair.c.clocks < 0.945 * other) {
                    e.plan = pair;
                    e.use = true;
                }
            }
        }
        // (what a failed query of the device decided is not kept)
        if (rc != KXC_B200_OK || tc_split_capacity(2) <= 0) e.key[0] = -1;
    }
    return e.use ? &e.plan : nullptr;
}

int cm_weight_pad(TcDType t, int c, const CmPlan& plan) {
    const int e128 = kRow / tc_elem_bytes(t);
    return plan.c.ctas * tiles(plan) > kNumSMs ? div_up(c, e128) * e128 : cm_channel_pad(t, c);
}

int32_t cm_setup(CmParams* p, TcDType dtype, const CmPlan& plan, const void* act_nhwc, const void* w_packed, int cpad, int w_cpad, int* status_word) {
    const CmGeometry& g = plan.g;
    const CmChoice& c = plan.c;
    Grouping t;
    if (!group_taps(g, c.shared != 0, &t)) return fail(KXC_B200_ERR_INVALID, "channel-major conv: %dx%d filter", g.KH, g.KW);
    const int eb = tc_elem_bytes(dtype);
    const uint64_t px = (uint64_t)cpad * eb, tap = (uint64_t)w_cpad * eb;
    if (px % 16 != 0 || tap % 16 != 0) return fail(KXC_B200_ERR_INVALID, "channel-major conv: %d, %d padded channels x %d bytes", cpad, w_cpad, eb);
    p->N = g.N; p->OH = g.OH; p->OW = g.OW; p->Cout = g.Cout;
    p->kb_elems = g.kb_elems; p->cblocks = g.cblocks; p->last_steps = g.last_steps;
    p->BW = c.BW; p->BH = c.BH; p->BNI = c.BNI; p->HB = c.HB; p->WB = c.WB; p->ctas = c.ctas; p->n_cols = c.ctas * c.n;
    p->tiles_w = div_up(g.OW, c.BW);
    p->tiles_h = div_up(g.OH, c.BH); p->tiles_n = div_up(g.N, c.BNI); p->tiles_c = div_up(g.Cout, c.ctas * kM);
    p->by_c = Divisor((unsigned)p->tiles_c); p->by_w = Divisor((unsigned)p->tiles_w); p->by_h = Divisor((unsigned)p->tiles_h);
    const int rows_w = g.Cout < kM ? div_up(g.Cout, 8) * 8 : kM;
    p->px_bytes = c.HB * c.WB * c.BNI * kRow;
    p->zero_bytes = c.zero_rows * kRow;
    p->px_slot_bytes = div_up(p->px_bytes + p->zero_bytes, 1024) * 1024;
    p->w_tap_bytes = rows_w * kRow;
    p->w_slot_bytes = c.group * p->w_tap_bytes;
    p->px_slots = c.px_slots; p->w_slots = c.w_slots;
    p->loads = t.loads; p->groups = 0;
    for (int l = 0; l < t.loads; ++l) {
        p->load_map[l] = (unsigned char)t.map[l];
        p->load_h[l] = t.h[l];
        p->load_w[l] = t.w[l];
        const int end = l + 1 < t.loads ? t.first[l + 1] : t.taps;
        for (int j = t.first[l]; j < end; j += c.group) {
            CmParams::Group& w = p->group[p->groups++];
            w.count = (unsigned char)(end - j < c.group ? end - j : c.group);
            w.first = j == t.first[l];
            w.last = j + c.group >= end;
            for (int k = 0; k < w.count; ++k) {
                w.tap[k] = (unsigned char)t.index[j + k];
                w.shift[k] = (unsigned short)((t.dh[j + k] * c.WB + t.dw[j + k]) * (kRow >> 4));
            }
        }
    }
    p->max_abs_acc = 128ll * 128 * g.KH * g.KW * cpad;
    const uint32_t box[4] = {(uint32_t)g.kb_elems, (uint32_t)c.WB, (uint32_t)c.HB, (uint32_t)c.BNI};
    uint8_t* base = const_cast<uint8_t*>(static_cast<const uint8_t*>(act_nhwc));
    for (int par = 0; par < (g.stride == 2 ? 4 : 1); ++par) {
        const int hp = par >> 1, wp = par & 1, s = g.stride;
        const int hc = (g.H - hp + s - 1) / s, wc = (g.W - wp + s - 1) / s;
        if (hc <= 0 || wc <= 0) return fail(KXC_B200_ERR_UNSUPPORTED, "channel-major conv: stride 2 over a %dx%d input", g.H, g.W);
        const uint64_t dims[4] = {(uint64_t)cpad, (uint64_t)wc, (uint64_t)hc, (uint64_t)g.N};
        const uint64_t strides[3] = {px * s, px * s * g.W, px * g.H * g.W};
        KXC_TRY(tc_make_tmap(&p->tmA[par], dtype, 4, base + ((size_t)hp * g.W + wp) * px, dims, strides, box, kRow));
    }
    const uint64_t wdims[3] = {(uint64_t)w_cpad, (uint64_t)g.Cout, (uint64_t)(g.KH * g.KW)};
    const uint64_t wstr[2] = {tap * g.KH * g.KW, tap};
    const uint32_t wbox[3] = {(uint32_t)g.kb_elems, (uint32_t)rows_w, 1u};
    KXC_TRY(tc_make_tmap(&p->tmW, dtype, 3, const_cast<void*>(w_packed), wdims, wstr, wbox, kRow));
    p->status = status_word;
    return status_word != nullptr ? KXC_B200_OK : tc_status_word(&p->status);
}

int32_t cm_launch(TcDType dtype, const CmParams& p, cudaStream_t stream) {
    switch (dtype) {
        case kTcBF16: return launch_kind<MmaKind::F16>(p, stream);
        case kTcTF32: return launch_kind<MmaKind::TF32>(p, stream);
        case kTcS8: return launch_kind<MmaKind::I8>(p, stream);
    }
    return fail(KXC_B200_ERR_INVALID, "channel-major conv: dtype");
}

}  // namespace kxc_b200
