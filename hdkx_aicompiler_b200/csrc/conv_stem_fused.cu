// 7x7 stride-2 "stem" convolution + bias + ReLU + max_pool2d(3x3, stride 2, pad 1) in ONE kernel that reads the
// graph input as the reference hands it over (NCHW fp32, include/te/topi/nn.h:107-158 / :161-229) and writes the
// pooled NHWC activation (bf16, or fp32 holding tf32 values): neither a packed copy of the input nor the convolution's output
// touches HBM.
//
// Work split of a CTA (22 warps, tf32 14), all roles running concurrently on a ring of input strips:
//   warp 0        loads the 28 KiB (tf32: 56) of weights once and the fp32 rows of the strips, eight at a time (bulk copies)
//   last 4 warps  converters: round the rows to the operand type and write the packed layout [row][pixel][4 channels] (8 bytes
//                 per pixel, zero border) that the tensor core reads
//   warp 1        issues tcgen05.mma, owns TMEM
//   the others    epilogue: accumulator -> 3x3 maximum -> +bias, ReLU, rounding -> store
//
// MMA formulation. In the packed layout the K vector of output pixel (oh, ow) for filter row r is the 8 pixels x 4
// channels starting at packed pixel (2*oh + r, 2*ow): with the unswizzled K-major operand layout (rows 16 bytes
// apart) the A operand of 128 consecutive output columns is a window of ONE packed input row (conv_stem.cu). The
// older kernel issues 14 instructions of N = 64 per output row, which the tensor core cannot run faster than about
// 74 cycles each however short their math is (32 cycles). Here one instruction serves SEVERAL output rows: packed
// input row t contributes, through filter row r = t - 2j, to every output row j of a block of three for which
// 0 <= r <= 6, and these rows' accumulators lie side by side in TMEM. So the B operand of the instruction for input
// row t is the stack [W(r_max); W(r_max - 2); ...] of the filter rows of t's parity (N = 64, 128 or 192) and D spans
// the matching accumulator slots: 24 instructions per three output rows instead of 42, most of them wide enough to
// run at the tensor pipe's full rate. Input rows are walked in ascending order and each slot's first contribution
// (r = 0) is an instruction of its own with the accumulate flag off, so every output element sums its 28 K chunks in
// exactly the order the one-row-at-a-time kernel uses: the two kernels give identical bits.
//
// Pooling in the epilogue: a thread owns one convolution column's 16 (tf32: 32) channels. The vertical maximum of a pooled row's three
// convolution rows is one three-operand instruction on the accumulators; the last of them stays in registers for the next pooled
// row. Then the bias, the rounding, and the horizontal maximum with two shuffles per register and pair of columns (the neighbour in
// another warp comes through a slot in shared memory and a 128-thread barrier). Adding the bias and rounding are monotonic and keep the
// order of signs, so that maximum, ReLU included, equals the reference's ReLU-then-fold `m = (m > v) ? m : v` (NaN -> 0, -0 -> +0
// included): 0 is a neutral element after the bias and one final max with 0 is the ReLU.
//
// tf32. A pixel is 16 bytes, so consecutive output columns (two pixels) are 32 bytes apart and the rows of a core matrix, which lie
// 16 bytes apart, cannot be every second pixel. The even and the odd pixels of a row therefore lie in two planes: one K step
// (eight tf32 values) is the pixel pair (2j, 2j + 1) = entry i + j of either plane, the distance of the planes being the
// operand's leading byte offset. Four K steps per filter row instead of two, 46 instructions per three output rows; strips of two
// pooled rows, which is what shared memory holds. The order of the sums is that of the implicit-GEMM kernel over the packed
// input, which this replaces together with the packing and the pooling kernel, and so are the bits. ResNet-18 tf32, the three
// launches / this one, us: 4 images 28.6 / 18.3, 32: 119 / 54.
//
// What bounds it, by the clocks that each role waits (bf16, 512 images; of 7500 a strip): the epilogue's chain of accumulator reads, barrier
// and shuffles (6300 clocks of work), the issue of the MMAs (5200), the converters (4700). Before the rows came by bulk copies (they came
// by each converter's own cp.async, read back one at a time) and the maximum moved in front of bias and rounding a strip took 9400: the epilogue worked for
// 8100, the converters for 7000. A launch in ResNet-18, us, before / now: bf16 1 image 11.9 / 9.9, 32: 34.2 / 25.1, 128: 74.5 / 61.5; tf32 1: 16.9 / 12.7, 32:
// 55.3 / 38.1, 128: 154.9 / 111.8; whole networks gain 2 to 4.5 % (at 1024 images, where the power limit sets the clock, they are level). Tried: fp32 rows prefetched in registers instead
// (two rows ahead: 10500 clocks a strip, memory latency), packed pixels stored without bank conflicts (no change).
//
// bf16 strips have four pooled rows; two where that leaves no SM a second strip (up to five images of 224 x 224), whose time is
// then one strip's latency: 13.1 -> 9.6 us.
// Every wait is bounded (sm100::mbar_wait_bounded); a wait that runs out is reported through the status word.
#include "conv_stem.cuh"

#include <cuda_bf16.h>

#include "common.cuh"
#include "conv_epilogue.cuh"
#include "sm100.cuh"

namespace kxc_b200 {
namespace {

using namespace sm100;

constexpr int kEpilogueWarp0 = 2, kConverterWarps = 4;
constexpr int kBN = 64;             // output channels
constexpr int kKH = 7;
constexpr int kBlockRows = 3;       // output rows per accumulator buffer
constexpr int kBufCols = 256;       // TMEM columns per buffer (3 slots of 64 used)
constexpr int kStages = 2;          // packed strips in shared memory (the tensor core reads one while the next is written)
constexpr int kEvenRows = 4 * kBN, kOddRows = 3 * kBN;     // stacked filter rows: r = 6,4,2,0 and r = 5,3,1
constexpr int kMaxC = 3;

template <bool kF32, int kPooled>
struct StemGeom {
    // Output channels of an epilogue warp. bf16: 16 warps of 16 (ResNet-18, 32 images 27.6 -> 25.1 us against 8 of 32, 128: 68 -> 61). tf32
    // keeps twice the registers per channel and would spill: 32 images 41 us with 16 channels, 38 with 32.
    static constexpr int kPartCols = kF32 ? 32 : 16, kEpilogueWarps = 4 * (kBN / kPartCols);
    static constexpr int kConverterWarp0 = kEpilogueWarp0 + kEpilogueWarps;
    static constexpr int kThreads = (kConverterWarp0 + kConverterWarps) * 32;  // loader, MMA issuer, epilogue warps, converters
    static constexpr int kConvRows = 2 * kPooled + 1;             // conv rows 2 kPooled s - 1 ... (the first one recomputed)
    static constexpr int kInRows = 2 * (kConvRows - 1) + kKH;     // packed input rows
    static constexpr int kMaxWidth = kF32 ? 224 : 244;
    static constexpr int kMaxRowBytes = kF32 ? 232 * 16 : 2048;
    // + slack for what the M = 128 rows read past the last row's end
    static constexpr int kStripBytes = ((kInRows * kMaxRowBytes + (kF32 ? 1024 : 4096) + 1023) / 1024) * 1024;
    static constexpr int kSteps = kF32 ? 4 : 2;                   // K steps (32 bytes) of a filter row
    static constexpr int kWeightBytes = 2 * kSteps * (kEvenRows + kOddRows) * 16;
    static constexpr int kExchBytes = 2 * 4 * kBN * (kF32 ? 4 : 2);  // [parity][channel part][quadrant] x one column's channels
    // fp32 rows on their way to the converters: a ring of slots, each two rows per converter warp of every channel plane
    static constexpr int kSlots = kF32 ? 2 : 3, kSlotRows = 2 * kConverterWarps;
    static constexpr int kSlotBytes = kMaxC * kSlotRows * kMaxWidth * 4;
    static constexpr int kStagingBytes = kSlots * kSlotBytes;
    static constexpr int kBiasBytes = kBN * 4;
    static constexpr int kSmemBytes = kWeightBytes + kStages * kStripBytes + kExchBytes + kStagingBytes + kBiasBytes + 1024;
    static_assert(kSmemBytes <= 227 * 1024 - 256, "shared memory of one CTA");
};

// The instruction list of a block of R output rows (see the file comment), built at compile time so that the issue
// loop is straight-line code with immediate operands: a single thread can then issue an MMA every ~25 cycles. (A loop
// that fetches its operands from a table costs ~140 cycles per instruction in one issuing thread, twice what the
// tensor core needs for the instruction itself.)
constexpr int kMaxEntries = 48;     // MMA instructions of a three-row block (24 for bf16)
struct MmaEntry {
    int t, cp;        // packed input row relative to the block's first one; which pair of K chunks
    uint32_t b_rel;   // low descriptor word of the stacked weights, relative to the weights' base address
    int d_off, n, acc;
};
struct MmaTable {
    MmaEntry e[kMaxEntries];
    int len;
};
__host__ __device__ constexpr MmaTable make_mma_table(int R, int steps) {
    MmaTable tb{};
    int n = 0;
    for (int t = 0; t <= 2 * (R - 1) + (kKH - 1); ++t) {
        const int jmin = t > kKH - 1 ? (t - (kKH - 1) + 1) / 2 : 0;
        const int jmax = (t / 2) < (R - 1) ? (t / 2) : (R - 1);
        const int odd = t & 1;
        const int r_first = t - 2 * jmin;  // filter row of the first (lowest) slot: the largest of the range
        const int q = odd ? (kKH - 2 - r_first) / 2 : (kKH - 1 - r_first) / 2;
        const int cnt = jmax - jmin + 1;
        const uint32_t lbo = (uint32_t)(odd ? kOddRows : kEvenRows) * 16u;
        const uint32_t wbase = (odd ? 2u * (uint32_t)steps * kEvenRows * 16u : 0u) + (uint32_t)q * kBN * 16u;
        for (int cp = 0; cp < steps; ++cp) {
            const uint32_t b_addr = wbase + (uint32_t)cp * 2u * lbo;
            const uint32_t lbo_field = (lbo >> 4) << 16;
            const bool first_touch = cp == 0 && !odd && t == 2 * jmax;  // slot jmax receives filter row 0 here
            if (first_touch) {
                if (cnt > 1) tb.e[n++] = MmaEntry{t, cp, (b_addr >> 4) | lbo_field, jmin * kBN, (cnt - 1) * kBN, 1};
                tb.e[n++] = MmaEntry{t, cp, ((b_addr + (uint32_t)(cnt - 1) * kBN * 16u) >> 4) | lbo_field, jmax * kBN, kBN, 0};
            } else {
                tb.e[n++] = MmaEntry{t, cp, (b_addr >> 4) | lbo_field, jmin * kBN, cnt * kBN, 1};
            }
        }
    }
    tb.len = n;
    return tb;
}

template <bool kF32, int kAcc>
__device__ __forceinline__ void umma_imm(uint32_t d_tmem, uint32_t a_lo, uint32_t hi, uint32_t b_lo, uint32_t idesc) {
    // both descriptors share the upper word (unswizzled, 8-row groups 128 B apart); the accumulate flag is an immediate
    if constexpr (kF32) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.eq.u32 p, 1, %5;\n\tmov.b64 da, {%1, %2};\n\tmov.b64 db, {%3, %2};\n\t"
            "tcgen05.mma.cta_group::1.kind::tf32 [%0], da, db, %4, p;\n\t}" ::"r"(d_tmem), "r"(a_lo), "r"(hi), "r"(b_lo), "r"(idesc), "n"(kAcc)
            : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.eq.u32 p, 1, %5;\n\tmov.b64 da, {%1, %2};\n\tmov.b64 db, {%3, %2};\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}" ::"r"(d_tmem), "r"(a_lo), "r"(hi), "r"(b_lo), "r"(idesc), "n"(kAcc)
            : "memory");
    }
}

template <bool kF32, int R, int I = 0>
__device__ __forceinline__ void issue_block(uint32_t d0, uint32_t a_lo0, uint32_t row16, uint32_t hi, uint32_t w_lo) {
    constexpr MmaTable tb = make_mma_table(R, kF32 ? 4 : 2);
    if constexpr (I < tb.len) {
        constexpr MmaEntry e = tb.e[I];
        constexpr uint32_t idesc = make_instr_desc(kF32 ? kFmtTF32 : kFmtBF16, kAccF32, (uint32_t)e.n);
        // a K step further: four bf16 pixels in a row, or the next entry of both planes
        umma_imm<kF32, e.acc>(d0 + (uint32_t)e.d_off, a_lo0 + (uint32_t)e.t * row16 + (uint32_t)(e.cp * (kF32 ? 1 : 2)), hi, w_lo + e.b_rel, idesc);
        issue_block<kF32, R, I + 1>(d0, a_lo0, row16, hi, w_lo);
    }
}

__device__ __forceinline__ void tmem_ld_part(uint32_t taddr, uint32_t (&v)[32]) { tmem_ld_32x32(taddr, v); }
__device__ __forceinline__ void tmem_ld_part(uint32_t taddr, uint32_t (&v)[16]) { tmem_ld_32x16(taddr, v); }

// As fmaxf(fmaxf(a, b), c): an operand that is no number is passed over.
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// (x, y) + (bx, by), each as __fadd_rn
__device__ __forceinline__ void add_pair(float& x, float& y, float bx, float by) {
    asm("{\n\t.reg .b64 a, b;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 b, {%2, %3};\n\tadd.rn.f32x2 a, a, b;\n\tmov.b64 {%0, %1}, a;\n\t}" : "+f"(x), "+f"(y) : "f"(bx), "f"(by));
}

__device__ __forceinline__ float4 lds16_if(bool there, uint32_t a) {
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t@p ld.shared.v4.f32 {%0, %1, %2, %3}, [%5];\n\t}"
                 : "+f"(v.x), "+f"(v.y), "+f"(v.z), "+f"(v.w) : "r"((int)there), "r"(a));
    return v;
}
__device__ __forceinline__ void bulk_copy_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
                 "r"(bytes), "r"(bar)
                 : "memory");
}

template <bool kF32, int kPooledRows>
__global__ void __launch_bounds__(StemGeom<kF32, kPooledRows>::kThreads, 1) conv_stem_pool_nchw_kernel(const __grid_constant__ TcParams p) {
    using G = StemGeom<kF32, kPooledRows>;
    constexpr int kConvRows = G::kConvRows, kStripBytes = G::kStripBytes, kWeightBytes = G::kWeightBytes, kSlots = G::kSlots, kSlotRows = G::kSlotRows, kSlotBytes = G::kSlotBytes;
    constexpr int kThreads = G::kThreads, kPartCols = G::kPartCols, kEpilogueWarps = G::kEpilogueWarps, kConverterWarp0 = G::kConverterWarp0;
    constexpr uint32_t kTmemCols = 2 * kBufCols;

    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bar_w;
    __shared__ __align__(8) uint64_t bar_full[kStages];
    __shared__ __align__(8) uint64_t bar_empty[kStages];
    __shared__ __align__(8) uint64_t bar_rows_full[kSlots], bar_rows_empty[kSlots];
    __shared__ __align__(8) uint64_t bar_acc_full[2];
    __shared__ __align__(8) uint64_t bar_acc_empty[2];
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;

    // (a uniform value, as the compiler then knows, and so all addresses that follow from it: 128 images 61.0 -> 53.9 us, 1024 500 -> 434)
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;
    const uint32_t w_smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t strip_smem = w_smem + kWeightBytes;
    const uint32_t exch_smem = strip_smem + kStages * kStripBytes;
    const uint32_t staging_smem = exch_smem + G::kExchBytes;
    const uint32_t bias_smem = staging_smem + G::kStagingBytes;  // (the epilogue's registers are taken)

    const int row_bytes = p.aux_row_bytes;  // packed row: Wp pixels
    const int Hp = p.aux_hp;
    const int H = p.aux_h, W = p.aux_w_px, C = p.aux_c;
    const int strips_per_image = p.OH / (2 * kPooledRows);
    const int total_strips = strips_per_image * p.N;

    if (threadIdx.x == 0) {
        abort_flag = 0;
        mbar_init(smem_u32(&bar_w), 1);
        for (int s = 0; s < kStages; ++s) {
            mbar_init(smem_u32(&bar_full[s]), kConverterWarps);
            mbar_init(smem_u32(&bar_empty[s]), 1);
        }
        for (int s = 0; s < kSlots; ++s) {
            mbar_init(smem_u32(&bar_rows_full[s]), 1);
            mbar_init(smem_u32(&bar_rows_empty[s]), kConverterWarps);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(smem_u32(&bar_acc_full[a]), 1);
            mbar_init(smem_u32(&bar_acc_empty[a]), kEpilogueWarps);
        }
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(&tmem_base_slot), kTmemCols);
        tmem_relinquish();
    }
    // Zero borders and slack: the converters only ever write the pixels of the image; the MMA of the last output
    // columns reads a little past a row's end (finite values that feed accumulator rows nobody stores).
    for (uint32_t i = threadIdx.x; i < (uint32_t)(kStages * kStripBytes / 16); i += kThreads) {
        const uint32_t addr = strip_smem + i * 16;
        asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(addr), "r"(0u) : "memory");
    }
    fence_proxy_async_shared();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_base_slot, 0);
    volatile int* abort_ptr = &abort_flag;
    pdl_launch_dependents();

    // Strip s of an image, four pooled rows: conv rows 8s-1 .. 8s+7 (local j = 0..8; j = 0 is skipped for s = 0, it is the pool's
    // padding row), packed input rows from max(16s - 2, 0); blocks of up to three conv rows.
    const float* x = static_cast<const float*>(p.aux_in);
    const bool vec = (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
    const size_t plane = (size_t)H * W;
    // rows [row_lo, row_hi) of a strip's rows_in local packed rows come from the image planes at `base` (+ local row * W); the others
    // are padding rows (zeros)
    auto strip_geom = [&](int strip, const float** base, int* row_lo, int* row_hi) {
        const int n = strip / strips_per_image;
        const int s = strip - n * strips_per_image;
        const int row0 = s > 0 ? 4 * kPooledRows * s - 2 : 0;
        int rows_in = (s > 0 ? 2 * (kConvRows - 1) : 2 * (kConvRows - 2)) + kKH;
        if (row0 + rows_in > Hp) rows_in = Hp - row0;
        const int h0 = row0 - p.pad_h;  // image row of local row 0
        *row_lo = h0 < 0 ? -h0 : 0;
        *row_hi = (H - h0) < rows_in ? (H - h0) : rows_in;
        *base = x + (size_t)n * C * plane + (ptrdiff_t)h0 * W;
        return rows_in;
    };
    if (warp == 0) {
        // ------------------------------ loader ------------------------------
        // A slot's rows of a plane lie one after the other in the image: one bulk copy per channel.
        if (lane == 0) {
            mbar_arrive_expect_tx(smem_u32(&bar_w), (uint32_t)kWeightBytes);
            bulk_copy_g2s(w_smem, p.aux_w, (uint32_t)kWeightBytes, smem_u32(&bar_w));  // the plan's (TcParams::weights_ready)
            pdl_wait();
            int slot = 0;
            uint32_t phase = 0;
            bool ok = vec;
            for (int strip = blockIdx.x; ok && strip < total_strips; strip += gridDim.x) {
                const float* base;
                int row_lo, row_hi;
                const int rows_in = strip_geom(strip, &base, &row_lo, &row_hi);
                for (int r0 = 0; r0 < rows_in; r0 += kSlotRows) {
                    if (!mbar_wait_bounded(smem_u32(&bar_rows_empty[slot]), phase ^ 1u, abort_ptr)) {
                        ok = false;
                        break;
                    }
                    const int lo = r0 > row_lo ? r0 : row_lo, hi = r0 + kSlotRows < row_hi ? r0 + kSlotRows : row_hi;
                    const uint32_t bytes = hi > lo ? (uint32_t)(hi - lo) * (uint32_t)W * 4u : 0u;
                    const uint32_t full = smem_u32(&bar_rows_full[slot]);
                    mbar_arrive_expect_tx(full, bytes * (uint32_t)C);
                    if (bytes != 0)
                        for (int c = 0; c < C; ++c)
                            bulk_copy_g2s(staging_smem + (uint32_t)(slot * kSlotBytes) + (uint32_t)((c * kSlotRows + lo - r0) * W) * 4u,
                                          base + c * plane + (ptrdiff_t)lo * W, bytes, full);
                    if (++slot == kSlots) { slot = 0; phase ^= 1u; }
                }
            }
        }
    } else if (warp >= kConverterWarp0) {
        // ------------------------------ converters ------------------------------
        // A warp takes two rows of every slot; a lane the rows' 4-pixel items `lane` and `lane + 32`, read without a branch, so that a row's reads
        // are in flight together (one at a time they took half of the converters' clocks).
        const int cw = warp - kConverterWarp0;
        const int wq = W >> 2;  // 4-pixel items per row
        static_assert(G::kMaxWidth / 4 <= 64, "two items a lane");
        pdl_wait();
        int stage = 0, slot = 0;
        uint32_t phase = 0, rows_phase = 0;
        bool ok = true;
        for (int strip = blockIdx.x; ok && strip < total_strips; strip += gridDim.x) {
            const float* base;
            int row_lo, row_hi;
            const int rows_in = strip_geom(strip, &base, &row_lo, &row_hi);
            // warp-uniform outcome: no lane may leave while the others go on to the __syncwarp below
            if (!__all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&bar_empty[stage]), phase ^ 1u, abort_ptr))) break;
            const uint32_t strip0 = strip_smem + (uint32_t)stage * kStripBytes + (kF32 ? 0u : (uint32_t)p.pad_w * 8u);
            for (int r0 = 0; r0 < rows_in; r0 += kSlotRows) {
                if (vec && !__all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&bar_rows_full[slot]), rows_phase, abort_ptr))) {
                    ok = false;
                    break;
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int row = r0 + h * kConverterWarps + cw;
                    const bool inside = row >= row_lo && row < row_hi;
                    float4 v[2][kMaxC];
                    if (vec) {
                        const uint32_t src = staging_smem + (uint32_t)(slot * kSlotBytes) + (uint32_t)((h * kConverterWarps + cw) * W) * 4u + (uint32_t)lane * 16u;
#pragma unroll
                        for (int i = 0; i < 2; ++i)
#pragma unroll
                            for (int c = 0; c < kMaxC; ++c)
                                v[i][c] = lds16_if(inside && c < C && lane + 32 * i < wq, src + (uint32_t)(c * kSlotRows * W) * 4u + (uint32_t)i * 512u);
                    } else {
#pragma unroll
                        for (int i = 0; i < 2; ++i)
#pragma unroll
                            for (int c = 0; c < kMaxC; ++c) {
                                v[i][c] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                                if (inside && c < C && lane + 32 * i < wq) {
                                    const float* at = base + c * plane + (ptrdiff_t)row * W + 4 * (lane + 32 * i);
                                    v[i][c] = make_float4(__ldg(at), __ldg(at + 1), __ldg(at + 2), __ldg(at + 3));
                                }
                            }
                    }
                    if (row >= rows_in) continue;
                    const uint32_t dst0 = strip0 + (uint32_t)row * (uint32_t)row_bytes;
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int q = lane + 32 * i;
                        if (q >= wq) continue;
                        const uint32_t dst = dst0 + (kF32 ? 0u : (uint32_t)q * 32u);
                        const float* f0 = reinterpret_cast<const float*>(&v[i][0]);
                        const float* f1 = reinterpret_cast<const float*>(&v[i][1]);
                        const float* f2 = reinterpret_cast<const float*>(&v[i][2]);
                        if constexpr (kF32) {
#pragma unroll
                            for (int px = 0; px < 4; ++px) {
                                const uint32_t at = (uint32_t)(4 * q + px + p.pad_w);  // even pixels, then odd ones
                                asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(dst + (at & 1u) * (uint32_t)(row_bytes >> 1) + (at >> 1) * 16u),
                                             "f"(tf32_rne(f0[px])), "f"(tf32_rne(f1[px])), "f"(tf32_rne(f2[px])), "f"(0.0f)
                                             : "memory");
                            }
                        } else {
                            uint32_t o[8];
#pragma unroll
                            for (int px = 0; px < 4; ++px) {
                                o[2 * px] = pack_bf16(f0[px], f1[px]);
                                o[2 * px + 1] = pack_bf16(f2[px], 0.0f);
                            }
                            // 16-byte stores where the padding leaves two pixels on such a boundary
                            if ((p.pad_w & 1) != 0) {
                                asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(dst), "r"(o[0]), "r"(o[1]) : "memory");
                                asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(dst + 8u), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]) : "memory");
                                asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(dst + 24u), "r"(o[6]), "r"(o[7]) : "memory");
                            } else {
                                asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]) : "memory");
                                asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(dst + 16u), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]) : "memory");
                            }
                        }
                    }
                }
                if (vec) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&bar_rows_empty[slot]));
                    if (++slot == kSlots) { slot = 0; rows_phase ^= 1u; }
                }
            }
            if (!ok) break;
            fence_proxy_async_shared();  // the tensor core reads these bytes through the async proxy
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bar_full[stage]));
            if (++stage == kStages) { stage = 0; phase ^= 1u; }
        }
    } else if (warp == 1) {
        // ------------------------------ MMA issuer ------------------------------
        // The whole warp walks the loop (uniform control flow); one elected lane issues the instructions.
        {
            bool ok = __all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&bar_w), 0, abort_ptr));
            const uint32_t ab_hi = desc_hi(128, 0);  // unswizzled, 8-row groups 128 B apart (A and B alike)
            const uint32_t w_lo = (w_smem & 0x3ffffu) >> 4;
            const uint32_t row16 = (uint32_t)(row_bytes >> 4);
            int stage = 0;
            uint32_t phase = 0;
            uint32_t blk = 0;
            for (int strip = blockIdx.x; ok && strip < total_strips; strip += gridDim.x) {
                const int s = strip % strips_per_image;
                if (!__all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&bar_full[stage]), phase, abort_ptr))) break;
                tc_fence_after_sync();
                const uint32_t strip_base = strip_smem + (uint32_t)stage * kStripBytes;
                for (int j0 = (s > 0 ? 0 : 1); j0 < kConvRows; j0 += kBlockRows, ++blk) {
                    const int R = kConvRows - j0 < kBlockRows ? kConvRows - j0 : kBlockRows;
                    const uint32_t buf = blk & 1u;
                    if (!__all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&bar_acc_empty[buf]), ((blk >> 1) & 1u) ^ 1u, abort_ptr))) { ok = false; break; }
                    tc_fence_after_sync();
                    const int in_row0 = s > 0 ? 2 * j0 : 2 * j0 - 2;  // local packed row of filter row 0 of conv row j0
                    const uint32_t a_lo0 = desc_lo(strip_base + (uint32_t)(in_row0 * row_bytes), kF32 ? (uint32_t)row_bytes >> 1 : 16u);
                    const uint32_t d0 = tmem_base + buf * kBufCols;
                    if (elect_one()) {
                        if (R == 3) issue_block<kF32, 3>(d0, a_lo0, row16, ab_hi, w_lo);
                        else if (R == 2) issue_block<kF32, 2>(d0, a_lo0, row16, ab_hi, w_lo);
                        else issue_block<kF32, 1>(d0, a_lo0, row16, ab_hi, w_lo);
                        umma_commit(smem_u32(&bar_acc_full[buf]));
                    }
                    __syncwarp();
                }
                if (!ok) break;
                if (elect_one()) umma_commit(smem_u32(&bar_empty[stage]));
                __syncwarp();
                if (++stage == kStages) { stage = 0; phase ^= 1u; }
            }
        }
    } else {
        // ------------------------------ epilogue ------------------------------
        // TMEM lane quadrant (warp & 3) x one channel part of kPartCols channels per warp.
        const int quad = warp & 3;
        const int part = (warp - kEpilogueWarp0) >> 2;
        const int ow = quad * 32 + lane;
        const int c0 = part * kPartCols;
        const int POH = p.OH / 2, POW = p.OW / 2;
        constexpr int kRegs = kF32 ? kPartCols : kPartCols / 2;  // registers of a column's pooled values: fp32, or bf16 pairs
        constexpr int kHalf = kRegs / 2;
        constexpr uint32_t kColBytes = kRegs * 4;
        char* pooled = static_cast<char*>(p.out) + (size_t)c0 * (kF32 ? 4 : 2);
        const uint32_t lane_base = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0;
        const bool odd = (lane & 1) != 0;
        pdl_wait();
        if (ow < kPartCols) {  // the bias of this part's channels, for its four warps
            const float b = p.bias != nullptr ? __ldg(p.bias + c0 + ow) : 0.0f;
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(bias_smem + (uint32_t)(c0 + ow) * 4u), "f"(b) : "memory");
        }
        named_barrier(1 + part, 128);
        uint32_t blk = 0;
        uint32_t fin = 0;  // pooled rows finished so far (parity picks the exchange slot)
        bool bad = false;  // a wait ran out: carried to the next 128-thread barrier, where the four warps of this part leave together
        int jj = 0, rows = 0, left = 0;  // the next row's slot in its accumulator block, the block's rows, the strip's rows from this block on
        auto open_block = [&]() {  // before a row's first read
            if (jj != 0) return;
            rows = left < kBlockRows ? left : kBlockRows;
            if (!bad) bad = !__all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&bar_acc_full[blk & 1u]), (blk >> 1) & 1u, abort_ptr));
            tc_fence_after_sync();
        };
        auto next_addr = [&]() { return lane_base + (blk & 1u) * kBufCols + (uint32_t)(jj * kBN); };
        auto close_row = [&]() {  // after the row's values have arrived: hand the buffer back with its last row
            if (++jj < rows) return;
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bar_acc_empty[blk & 1u]));
            ++blk;
            left -= rows;
            jj = 0;
        };
        // One pooled row: the rows `held` (its first, read before), and the next two, the second of which stays in `last`. The vertical maximum is
        // that of the unrounded sums; bias and rounding are monotonic, so they follow it once.
        auto pooled_row = [&](int n, int ph, const uint32_t (&held)[kPartCols], uint32_t (&last)[kPartCols]) -> bool {
            uint32_t mid[kPartCols];
            open_block();
            tmem_ld_part(next_addr(), mid);
            if (jj + 1 < rows) {  // both in one block
                ++jj;
                tmem_ld_part(next_addr(), last);
                tmem_ld_wait();
            } else {
                tmem_ld_wait();
                close_row();
                open_block();
                tmem_ld_part(next_addr(), last);
                tmem_ld_wait();
            }
            close_row();
            uint32_t m[kRegs];
#pragma unroll
            for (int g = 0; g < kPartCols / 4; ++g) {
                float b[4], s4[4];
                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(b[0]), "=f"(b[1]), "=f"(b[2]), "=f"(b[3]) : "r"(bias_smem + (uint32_t)(c0 + 4 * g) * 4u));
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    s4[k] = max3(__uint_as_float(held[4 * g + k]), __uint_as_float(mid[4 * g + k]), __uint_as_float(last[4 * g + k]));
                add_pair(s4[0], s4[1], b[0], b[1]);
                add_pair(s4[2], s4[3], b[2], b[3]);
                if constexpr (kF32) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) m[4 * g + k] = __float_as_uint(s4[k]);
                } else {
                    m[2 * g] = pack_bf16(s4[0], s4[1]);
                    m[2 * g + 1] = pack_bf16(s4[2], s4[3]);
                }
            }
            auto slot_of = [&](int q) { return exch_smem + ((((fin & 1u) * (uint32_t)(64 / kPartCols) + (uint32_t)part) * 4u + (uint32_t)q) * kColBytes); };
            if (lane == 31) {  // the left neighbour of the next quadrant's first column
                const uint32_t slot = slot_of(quad);
#pragma unroll
                for (int g = 0; g < kRegs / 4; ++g)
                    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(slot + g * 16u), "r"(m[4 * g]), "r"(m[4 * g + 1]), "r"(m[4 * g + 2]), "r"(m[4 * g + 3])
                                 : "memory");
            }
            if (named_barrier_or(1 + part, 128, bad)) return false;
            // Horizontal maximum over conv columns 2m-1, 2m, 2m+1 for pooled column m, shared by the two lanes of a pair: the even
            // lane (column 2m) takes the lower half of the part's channels, the odd lane (column 2m+1) the upper half, so each register
            // costs two shuffles per PAIR of lanes and every lane stores.
            uint32_t edge[kHalf];  // column 2m-1 for lanes 0 and 1: the previous quadrant's last column (or padding)
#pragma unroll
            for (int e = 0; e < kHalf; ++e) edge[e] = 0u;
            if (lane < 2 && quad > 0) {
                const uint32_t slot = slot_of(quad - 1) + (odd ? kColBytes / 2 : 0u);
#pragma unroll
                for (int g = 0; g < kHalf / 4; ++g)
                    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                                 : "=r"(edge[4 * g]), "=r"(edge[4 * g + 1]), "=r"(edge[4 * g + 2]), "=r"(edge[4 * g + 3])
                                 : "r"(slot + g * 16u));
            }
            uint32_t res[kHalf];
#pragma unroll
            for (int e = 0; e < kHalf; ++e) {
                const uint32_t lo = m[e], hi = m[e + kHalf];
                const uint32_t mine = odd ? hi : lo;
                const uint32_t partner = __shfl_xor_sync(0xffffffffu, odd ? lo : hi, 1);  // the pair's other column, my half
                uint32_t prev = __shfl_up_sync(0xffffffffu, odd ? mine : partner, 2);     // the previous pair's odd column, my half
                if (lane < 2) prev = edge[e];
                if constexpr (kF32) {
                    const float f = fmaxf(max3(__uint_as_float(mine), __uint_as_float(partner), __uint_as_float(prev)), 0.0f);  // ReLU
                    res[e] = __float_as_uint(p.round_out_tf32 ? tf32_rne(f) : f);
                } else {
                    const __nv_bfloat162 zero2 = __floats2bfloat162_rn(0.0f, 0.0f);
                    __nv_bfloat162 f = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&mine), *reinterpret_cast<const __nv_bfloat162*>(&partner));
                    f = __hmax2(f, *reinterpret_cast<const __nv_bfloat162*>(&prev));
                    f = __hmax2(f, zero2);  // ReLU
                    res[e] = *reinterpret_cast<uint32_t*>(&f);
                }
            }
            if ((ow & ~1) < p.OW) {  // (columns beyond the image feed no pooled one: OW is even)
                uint4* dst = reinterpret_cast<uint4*>(pooled + ((((size_t)n * POH + ph) * POW + (ow >> 1)) * kBN) * (kF32 ? 4 : 2) + (odd ? kColBytes / 2 : 0u));
#pragma unroll
                for (int g = 0; g < kHalf / 4; ++g) dst[g] = make_uint4(res[4 * g], res[4 * g + 1], res[4 * g + 2], res[4 * g + 3]);
            }
            ++fin;
            return true;
        };
        for (int strip = blockIdx.x; strip < total_strips; strip += gridDim.x) {
            const int n = strip / strips_per_image;
            const int s = strip - n * strips_per_image;
            uint32_t u[kPartCols], v[kPartCols];
            left = s > 0 ? kConvRows : kConvRows - 1;
            if (s > 0) {
                open_block();
                tmem_ld_part(next_addr(), u);
                tmem_ld_wait();
                close_row();
            } else {  // the pool's padding row
#pragma unroll
                for (int e = 0; e < kPartCols; ++e) u[e] = 0xff800000u;
            }
            bool go = true;
#pragma unroll 1
            for (int k = 0; k < kPooledRows; k += 2) go = go && pooled_row(n, kPooledRows * s + k, u, v) && pooled_row(n, kPooledRows * s + k + 1, v, u);
            if (!go) break;
        }
    }

    if (*abort_ptr) {
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    if (warp == 1) {
        __syncwarp();
        tmem_dealloc(tmem_base, kTmemCols);
    }
    if (threadIdx.x == 0 && *abort_ptr && p.status != nullptr) atomicExch(p.status, KXC_B200_ERR_DEVICE_WAIT);
}

// Stem weights, filter rows stacked by parity: [r = 6,4,2,0 | r = 5,3,1], each stack in core-matrix order
// [k-chunks][stack rows][16 bytes] with stack row = (position in the stack) * 64 + cout; element e of bf16 chunk j (of 4) = pixel
// 2j + e/4, channel e%4, of tf32 chunk j (of 8) = pixel j, channel e; zero for kw >= KW or c >= C.
template <typename T>
__global__ void stem_pack_weights_stacked_kernel(const float* __restrict__ w, T* __restrict__ out, int O, int C, int KW) {
    constexpr int kElems = 16 / (int)sizeof(T), kPixels = kElems / 4, kChunks = 8 / kPixels;
    const int total = kChunks * (kEvenRows + kOddRows) * kElems;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const bool odd = i >= kChunks * kEvenRows * kElems;
        const int li = odd ? i - kChunks * kEvenRows * kElems : i;
        const int rows = odd ? kOddRows : kEvenRows;
        const int e = li % kElems;
        const int row = (li / kElems) % rows;
        const int jc = (li / kElems) / rows;
        const int o = row & (kBN - 1), pos = row / kBN;
        const int r = odd ? (kKH - 2) - 2 * pos : (kKH - 1) - 2 * pos;
        const int kw = kPixels * jc + (e >> 2), c = e & 3;
        float f = 0.0f;
        if (o < O && c < C && kw < KW) f = w[((o * C + c) * kKH + r) * KW + kw];
        if constexpr (sizeof(T) == 4) out[i] = tf32_rne(f);
        else out[i] = __float2bfloat16_rn(f);
    }
}

template <bool kF32, int kPooled>
int32_t launch(const TcParams& p, cudaStream_t stream) {
    constexpr int kBytes = StemGeom<kF32, kPooled>::kSmemBytes;
    static PerDeviceOnce smem_once;
    auto kernel = conv_stem_pool_nchw_kernel<kF32, kPooled>;
    KXC_TRY(smem_opt_in(smem_once, kernel, kBytes));
    const long long strips = (long long)(p.OH / (2 * kPooled)) * p.N;
    const int grid = (int)(strips < kNumSMs ? strips : kNumSMs);
    KXC_CUDA_TRY(launch_kernel(kernel, dim3(grid), dim3(StemGeom<kF32, kPooled>::kThreads), kBytes, stream, /*pdl=*/true, 1, p));
    return check_launch("conv_stem_pool_nchw_kernel");
}

}  // namespace

bool stem_pool_nchw_applicable(TcDType dtype, int C, int O, int KH, int KW, int W, int OH, int OW, int Wp) {
    if (dtype != kTcBF16 && dtype != kTcTF32) return false;
    const bool f32 = dtype == kTcTF32;
    const int row_bytes = Wp * (f32 ? 16 : 8), pooled = f32 ? 2 : 4;
    return C >= 1 && C <= kMaxC && W <= (f32 ? StemGeom<true, 2>::kMaxWidth : StemGeom<false, 4>::kMaxWidth) && O == kBN && KH == kKH && KW <= 8 && (W % 4) == 0 && (OH % (2 * pooled)) == 0 &&
           (OW % 2) == 0 && OW <= 128 && row_bytes <= (f32 ? StemGeom<true, 2>::kMaxRowBytes : StemGeom<false, 4>::kMaxRowBytes) && row_bytes % 32 == 0;
}

size_t stem_stacked_weight_bytes(TcDType dtype) {
    return dtype == kTcTF32 ? (size_t)StemGeom<true, 2>::kWeightBytes : (size_t)StemGeom<false, 4>::kWeightBytes;
}

int32_t stem_stacked_pack_weights(TcDType dtype, const float* w, void* out, int O, int C, int KW, cudaStream_t s) {
    const int grid = (8 * (kEvenRows + kOddRows) * 4 + 255) / 256;
    if (dtype == kTcTF32) stem_pack_weights_stacked_kernel<float><<<grid, 256, 0, s>>>(w, static_cast<float*>(out), O, C, KW);
    else stem_pack_weights_stacked_kernel<__nv_bfloat16><<<grid, 256, 0, s>>>(w, static_cast<__nv_bfloat16*>(out), O, C, KW);
    return check_launch("stem_pack_weights_stacked");
}

int32_t stem_pool_nchw_setup(TcParams* p, TcDType dtype, const void* packed_w, int N, int C, int H, int W, int OH, int OW, int pad_h, int pad_w,
                             int Hp, int Wp) {
    p->N = N; p->OH = OH; p->OW = OW; p->Cout = kBN;
    p->taps_h = kKH; p->taps_w = 1; p->stride = 2;
    p->pad_h = pad_h; p->pad_w = pad_w; p->dil_h = 1; p->dil_w = 1;
    p->BW = 128; p->BH = kBlockRows; p->BNI = 1;
    p->tiles_w = 1; p->tiles_h = OH; p->tiles_n = N; p->tiles_c = 1;
    p->aux_in = nullptr;  // the graph input: bound at run time
    p->aux_w = packed_w;
    p->aux_row_bytes = Wp * (dtype == kTcTF32 ? 16 : 8);
    p->aux_hp = Hp;
    p->aux_c = C; p->aux_h = H; p->aux_w_px = W;
    KXC_TRY(tc_status_word(&p->status));
    return KXC_B200_OK;
}

int32_t stem_pool_nchw_launch(TcDType dtype, const TcParams& p, cudaStream_t stream) {
    if ((dtype == kTcBF16 && !p.vec_ok) || p.out == nullptr || p.aux_in == nullptr)
        return fail(KXC_B200_ERR_INVALID, "fused stem conv + pool: missing tensors or pointers that are not 16-byte aligned");
    if (!p.relu) return fail(KXC_B200_ERR_INVALID, "fused stem conv + pool: the pooling shortcut relies on the ReLU in between");
    if (p.N <= 0 || p.OH <= 0) return KXC_B200_OK;
    if (dtype == kTcTF32) return launch<true, 2>(p, stream);
    // two pooled rows per strip where every strip then has an SM to itself
    return (long long)(p.OH / 4) * p.N <= kNumSMs ? launch<false, 2>(p, stream) : launch<false, 4>(p, stream);
}

}  // namespace kxc_b200
