// Layout / precision conversion kernels (HBM-bound, coalesced on both sides through a shared-memory
// transpose tile).
#include "layout.cuh"

#include <cuda_bf16.h>

#include "common.cuh"
#include "divisor.cuh"
#include "sm100.cuh"
#include "tf32.cuh"

namespace kxc_b200 {
namespace {

template <typename TOut>
__device__ __forceinline__ TOut convert_to(float v);
template <>
__device__ __forceinline__ __nv_bfloat16 convert_to<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <>
__device__ __forceinline__ float convert_to<float>(float v) { return tf32_rne(v); }

// what single-pass tf32 drops
struct Tf32Lo {
    float v;
};
template <>
__device__ __forceinline__ Tf32Lo convert_to<Tf32Lo>(float v) {
    return Tf32Lo{tf32_low_part(v, tf32_rne(v))};
}

struct PackArgs {
    const void* w = nullptr;
    void* out = nullptr;
    void* lo = nullptr;   // three-pass tf32: the low parts
    int64_t groups = 0;   // threads that have work for every piece of a filter (pack_weights_block)
    int C = 0, taps = 0, cpad = 0;
    int per_thread = 0;       // taps
    Divisor pieces, per_row;  // of a filter; groups of channels of an output channel
    unsigned blocks = 0;
};

// Weights OIHW -> [O][KH*KW][cpad] (channels c >= C zero): a thread takes some taps (PackArgs::per_thread) of one output channel and kVec
// input channels, so that its reads are consecutive words, about ten of them in flight at once, and its stores are whole 32-bit words side
// by side with its neighbours'. The warps of the pieces of 32 groups are neighbours: they read the same sectors. One way to memory and
// back bounds it. (With a thread per whole filter there was one after the other for every nine taps, on few blocks where the channels are
// few: 3 -> 32 channels 31x31 at 64x64, bf16 442 us a call so, 333 now, int8 428 and 326; 3 -> 64 7x7 stride 2 at 224x224, bf16 28.5 and 24.7.)
// Nine taps of fp32, five of bf16, three of int8, but nine where that still makes 48 blocks: 100 -> 200 3x3 at 41x43, 16 images, int8 36 us a
// call with nine and 28 with three, since the convolution's CTAs, set up meanwhile, leave less room to a conversion that takes long; 256 ->
// 256 3x3 at 14x14, 16 images, 14.9 with nine and 16.4 with three, whose blocks cost more than their shorter chain gains.
template <typename T>
constexpr int kPackTaps = sizeof(T) == 4 ? 9 : sizeof(T) == 2 ? 5 : 3;
template <typename TIn, typename TOut, bool kSplit>
__device__ __forceinline__ void pack_weights_block(const TIn* __restrict__ w, TOut* __restrict__ out, TOut* __restrict__ lo, const PackArgs& a,
                                                   unsigned block) {
    constexpr int kVec = 4 / (int)sizeof(TOut);
    const unsigned warp = block * 8 + threadIdx.x / 32, set = a.pieces.quotient(warp);
    const int64_t g = (int64_t)set * 32 + threadIdx.x % 32;
    if (g >= a.groups) return;
    const int C = a.C, taps = a.taps, cpad = a.cpad, first = (int)(warp - set * a.pieces.d) * a.per_thread;
    const int o = a.groups < 1ll << 31 ? (int)a.per_row.quotient((unsigned)g) : (int)(g / a.per_row.d);
    const int c0 = (int)(g - (int64_t)o * a.per_row.d) * kVec;
    const TIn* src = w + ((int64_t)o * C + c0) * taps + first;
    TOut* dst = out + ((int64_t)o * taps + first) * cpad + c0;
    [[maybe_unused]] const int64_t lo_off = kSplit ? lo - out : 0;
    if constexpr (kVec == 4) {  // (a loop: the registers of 36 loads would cost the transposition blocks)
        const int count = taps - first < a.per_thread ? taps - first : a.per_thread;
#pragma unroll 9
        for (int t = 0; t < count; ++t) {
            alignas(4) TOut v[kVec];
#pragma unroll
            for (int e = 0; e < kVec; ++e) v[e] = c0 + e < C ? __ldg(src + (int64_t)e * taps + t) : (TIn)0;
            *reinterpret_cast<uint32_t*>(dst + (int64_t)t * cpad) = *reinterpret_cast<const uint32_t*>(v);
        }
    } else {
        TIn x[kPackTaps<TOut>][kVec];
#pragma unroll
        for (int t = 0; t < kPackTaps<TOut>; ++t)
#pragma unroll
            for (int e = 0; e < kVec; ++e) x[t][e] = first + t < taps && c0 + e < C ? __ldg(src + (int64_t)e * taps + t) : (TIn)0;
#pragma unroll
        for (int t = 0; t < kPackTaps<TOut>; ++t) {
            if (first + t >= taps) break;
            alignas(4) TOut v[kVec];
#pragma unroll
            for (int e = 0; e < kVec; ++e) v[e] = convert_to<TOut>(x[t][e]);
            *reinterpret_cast<uint32_t*>(dst + (int64_t)t * cpad) = *reinterpret_cast<const uint32_t*>(v);
            if constexpr (kSplit) dst[lo_off + (int64_t)t * cpad] = convert_to<Tf32Lo>(x[t][0]).v;
        }
    }
}

// Activations NCHW fp32 -> NHWC of the operand type and, in the first blocks of the same launch, the weights of the convolution
// that follows. One launch instead of two (each cost 2 to 3 us of launch and drain beside 2 to 5 us of work: conv 72 -> 120 3x3
// at 45x51, 9 images, tf32: 38.9 -> 32.3 us a call). A block turns kCT channels x 2048 / kCT pixels through shared memory with
// eight loads in flight per thread; stores are channel pairs, 128 bytes per pixel (kCT = 64 for more than 32 bf16 channels, which are
// padded to whole 64s then, else 32: fp32 counts are padded to 32s, 66 channels at 23x22, 43 images: 5.7 us with 64, 4.7 with 32).
// Bound by memory: 4 bytes read and 2, 4 or 8 written per value.
//
// Programmatic launch on both sides: the blocks wait for the previous kernel before they touch memory, and with `overlap` then
// let the next kernel's CTAs set themselves up. Weights packed here are not TcParams::weights_ready for the kernel after it (it
// waits before it reads them); those of a plan have been packed before its first step begins. A launch that packs a plan's weights does not let go
// early: the kernel after the next may read them ahead.
//
// kSub: only the pixels that a 1x1 convolution of stride `st` without padding reads, so that it runs with stride 1 over a quarter of the
// pixels: rows it skips are never touched, and a quarter is written (67 -> 56 at 91x94, 60 images, bf16: 102 -> 49 us a call).
struct PixelArgs {
    int plane = 0, W = 0, st = 1;  // elements of an input plane and columns of it; stride
    Divisor by_ow;                 // columns of the pixels read
};
template <typename TOut, bool kSplit, int kCT, bool kSub>
__global__ void __launch_bounds__(256) convert_operands_kernel(const float* __restrict__ in, TOut* __restrict__ out, TOut* __restrict__ lo, int C,
                                                               int HW, int cpad, Divisor tiles_hw, Divisor tiles_c, PackArgs pack, int overlap,
                                                               PixelArgs px) {
    constexpr int kPT = 2048 / kCT;
    sm100::pdl_wait();
    if (overlap) sm100::pdl_launch_dependents();
    if (blockIdx.x < pack.blocks) {
        pack_weights_block<float, TOut, kSplit>(static_cast<const float*>(pack.w), static_cast<TOut*>(pack.out), static_cast<TOut*>(pack.lo),
                                                pack, blockIdx.x);
        return;
    }
    __shared__ float tile[kCT][kPT + 1];
    const unsigned t = blockIdx.x - pack.blocks;
    const unsigned row = tiles_hw.quotient(t);
    const int hw0 = (int)(t - row * tiles_hw.d) * kPT;
    const int n = (int)tiles_c.quotient(row);
    const int c0 = (int)(row - n * tiles_c.d) * kCT;
    const int plane = kSub ? px.plane : HW;
    int place = hw0 + (int)threadIdx.x % kPT;  // (256 is a multiple of kPT: a thread has one pixel)
    const bool there = place < HW;
    if constexpr (kSub) {
        const int row = (int)px.by_ow.quotient((unsigned)place);
        place = (row * px.W + place - row * (int)px.by_ow.d) * px.st;
    }
    const float* src = in + ((int64_t)n * C + c0) * plane + place;
    const int64_t dst = ((int64_t)n * HW + hw0) * cpad + c0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int i = (int)threadIdx.x + 256 * k, p = i % kPT, c = i / kPT;
        tile[c][p] = c0 + c < C && there ? __ldg(src + (int64_t)c * plane) : 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int i = (int)threadIdx.x + 256 * k, c = i % (kCT / 2) * 2, p = i / (kCT / 2);
        if (hw0 + p >= HW || c0 + c >= cpad) continue;  // (cpad is even)
        const float x = tile[c][p], y = tile[c + 1][p];
        const int64_t at = dst + (int64_t)p * cpad + c;
        if constexpr (sizeof(TOut) == 2) {
            *reinterpret_cast<__nv_bfloat162*>(out + at) = __nv_bfloat162(convert_to<TOut>(x), convert_to<TOut>(y));
        } else {
            *reinterpret_cast<float2*>(out + at) = make_float2(convert_to<float>(x), convert_to<float>(y));
            if constexpr (kSplit) *reinterpret_cast<float2*>(lo + at) = make_float2(convert_to<Tf32Lo>(x).v, convert_to<Tf32Lo>(y).v);
        }
    }
}

// Weights alone: constants of a plan, packed once.
template <typename TIn, typename TOut, bool kSplit>
__global__ void __launch_bounds__(256) pack_weights_kernel(PackArgs pack) {
    sm100::pdl_wait();
    pack_weights_block<TIn, TOut, kSplit>(static_cast<const TIn*>(pack.w), static_cast<TOut*>(pack.out), static_cast<TOut*>(pack.lo), pack, blockIdx.x);
}

// The same for rows that need no reordering: [rows, cols] -> two times [rows, cpad]. cols % 4 == 0 and cols == cpad take
// 16-byte accesses (bound by memory: 4 bytes read and 8 written per value).
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ in, float* __restrict__ hi, float* __restrict__ lo, int64_t rows,
                                                         int cols, int cpad) {
    sm100::pdl_wait();
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (cols == cpad && (cols & 3) == 0) {
        for (const int64_t total = rows * cols / 4; i < total; i += step) {
            const float4 v = __ldg(reinterpret_cast<const float4*>(in) + i);
            reinterpret_cast<float4*>(hi)[i] = make_float4(convert_to<float>(v.x), convert_to<float>(v.y), convert_to<float>(v.z), convert_to<float>(v.w));
            reinterpret_cast<float4*>(lo)[i] = make_float4(convert_to<Tf32Lo>(v.x).v, convert_to<Tf32Lo>(v.y).v, convert_to<Tf32Lo>(v.z).v,
                                                           convert_to<Tf32Lo>(v.w).v);
        }
        return;
    }
    for (const int64_t total = rows * cpad; i < total; i += step) {
        const int c = (int)(i % cpad);
        const int64_t r = i / cpad;
        const float v = c < cols ? in[r * cols + c] : 0.0f;
        hi[i] = convert_to<float>(v);
        lo[i] = convert_to<Tf32Lo>(v).v;
    }
}

// int8 form: 64 channels x 64 pixels per block, four bytes per thread on both sides (64-byte runs in HBM instead of the
// 32-byte runs an element-wise kernel makes of 1-byte elements). Tiles ceil(HW/64) x ceil(cpad/64) x N, block 256.
// It is a batched byte transpose [C][HW] -> [HW][cpad] (rows c >= C read as zero), so it also serves NHWC -> NCHW with
// the roles of the two extents exchanged (source rows `pitch` bytes apart); vec_out = 0 when the destination rows are not 4-byte multiples.
__device__ __forceinline__ void transpose_s8_tile(const int8_t* __restrict__ in, int8_t* __restrict__ out, int C, int HW, int pitch, int cpad,
                                                  int vec_in, int vec_out, int hw_tile, int c_tile, int n) {
    __shared__ __align__(4) int8_t tile[64][68];
    const int hw0 = hw_tile * 64, c0 = c_tile * 64;
    const int8_t* src = in + (size_t)n * C * pitch;
    int8_t* dst = out + (size_t)n * HW * cpad;
    const int q = threadIdx.x & 15, r = threadIdx.x >> 4;  // 16 four-byte columns x 16 rows per pass
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int c = c0 + r + 16 * k, hw = hw0 + 4 * q;
        uint32_t v = 0;
        if (c < C) {
            const int8_t* s4 = src + (size_t)c * pitch + hw;
            if (vec_in && hw + 3 < HW) {
                v = __ldg(reinterpret_cast<const uint32_t*>(s4));
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (hw + e < HW) v |= (uint32_t)(uint8_t)__ldg(s4 + e) << (8 * e);
            }
        }
        *reinterpret_cast<uint32_t*>(&tile[r + 16 * k][4 * q]) = v;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int hw = hw0 + r + 16 * k, c = c0 + 4 * q;
        if (hw < HW && c < cpad) {
            const int hl = r + 16 * k;
            const uint32_t v = (uint32_t)(uint8_t)tile[4 * q][hl] | ((uint32_t)(uint8_t)tile[4 * q + 1][hl] << 8) |
                               ((uint32_t)(uint8_t)tile[4 * q + 2][hl] << 16) | ((uint32_t)(uint8_t)tile[4 * q + 3][hl] << 24);
            int8_t* d4 = dst + (size_t)hw * cpad + c;
            if (vec_out) {  // cpad is a multiple of 4: the four bytes are in or out together
                *reinterpret_cast<uint32_t*>(d4) = v;
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (c + e < cpad) d4[e] = (int8_t)(v >> (8 * e));
            }
        }
    }
}

// The same transpose for pitches that are multiples of four: R rows of `pitch` bytes, the first W of them used (the rest may be
// read) -> W rows of `opitch` bytes, zero from byte R on. A thread turns 4 x 4 byte blocks in registers (a byte gather out of
// shared memory, as above, held the kernel to 3 TB/s: 17 us for 25.7 MB in and out, this one 12 to 13), reads V bytes of four
// rows at a time and parks whole words in shared memory; word (column p, quad q) lies at q ^ f(p), so that a warp's stores,
// whose columns are V apart, fall on 16 banks and its reads, one column per 16 lanes, on 32.
// Tile 64 rows x TP columns: ceil(W/TP) x ceil(max(R, opitch)/64) x batch of them, block 256.
template <int V, int TP>
__device__ __forceinline__ void transpose_bytes_tile(const int8_t* __restrict__ in, int8_t* __restrict__ out, int R, int W, int pitch, int opitch,
                                                     int w_tile, int r_tile, int batch) {
    __shared__ uint32_t tile[TP * 16];
    const int w0 = w_tile * TP, r0 = r_tile * 64;
    const int8_t* src = in + (int64_t)batch * R * pitch;
    int8_t* dst = out + (int64_t)batch * W * opitch;
    auto slot = [](int p, int q) { return p * 16 + (q ^ (((p >> 2) ^ (p >> 4)) & 15)); };
    constexpr int kWords = V / 4, kVecs = TP / V;
#pragma unroll
    for (int u = threadIdx.x; u < 16 * kVecs; u += 256) {
        const int q = u / kVecs, p = (u % kVecs) * V;  // four rows, V columns
        uint32_t a[4][kWords] = {};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (r0 + 4 * q + k < R && w0 + p < W) {  // (pitch % V == 0: the vector lies inside its row)
                const int8_t* row = src + (int64_t)(r0 + 4 * q + k) * pitch + w0 + p;
                if constexpr (V == 16) {
                    const uint4 v = __ldg(reinterpret_cast<const uint4*>(row));
                    a[k][0] = v.x; a[k][1] = v.y; a[k][2] = v.z; a[k][3] = v.w;
                } else {
                    a[k][0] = __ldg(reinterpret_cast<const uint32_t*>(row));
                }
            }
        }
#pragma unroll
        for (int x = 0; x < kWords; ++x) {
            const uint32_t lo01 = __byte_perm(a[0][x], a[1][x], 0x5140), hi01 = __byte_perm(a[0][x], a[1][x], 0x7362);
            const uint32_t lo23 = __byte_perm(a[2][x], a[3][x], 0x5140), hi23 = __byte_perm(a[2][x], a[3][x], 0x7362);
            const int c = p + 4 * x;
            tile[slot(c, q)] = __byte_perm(lo01, lo23, 0x5410);
            tile[slot(c + 1, q)] = __byte_perm(lo01, lo23, 0x7632);
            tile[slot(c + 2, q)] = __byte_perm(hi01, hi23, 0x5410);
            tile[slot(c + 3, q)] = __byte_perm(hi01, hi23, 0x7632);
        }
    }
    __syncthreads();
#pragma unroll 4
    for (int u = threadIdx.x; u < TP * 16; u += 256) {
        const int p = u >> 4, q = u & 15;
        if (w0 + p < W && r0 + 4 * q < opitch) *reinterpret_cast<uint32_t*>(dst + (int64_t)(w0 + p) * opitch + r0 + 4 * q) = tile[slot(p, q)];
    }
}

// int8 NCHW -> NHWC of the pixels a 1x1 convolution of stride `st` (no padding) reads: out[n][p][c] =
// in[n][c][(p / OW) * st][(p % OW) * st], p = oh * OW + ow. Tiles ceil(OH*OW/64) x ceil(cpad/64) x N, block 256: the same
// 64 x 64 byte transpose as above with gathered source pixels; the rows the convolution skips are never touched.
__device__ __forceinline__ void subsample_s8_tile(const int8_t* __restrict__ in, int8_t* __restrict__ out, int C, int H, int W, int OH, int OW,
                                                  int st, int cpad, int p_tile, int c_tile, int n) {
    __shared__ __align__(4) int8_t tile[64][68];
    const int p0 = p_tile * 64, c0 = c_tile * 64;
    const int P = OH * OW;
    const int8_t* src = in + (size_t)n * C * H * W;
    int8_t* dst = out + (size_t)n * P * cpad;
    const int q = threadIdx.x & 15, r = threadIdx.x >> 4;
    int off[4];  // source offsets of this thread's four pixels inside a channel plane (-1: beyond the last pixel)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int p = p0 + 4 * q + e;
        off[e] = p < P ? (p / OW) * st * W + (p % OW) * st : -1;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int c = c0 + r + 16 * k;
        uint32_t v = 0;
        if (c < C) {
            const int8_t* plane = src + (size_t)c * H * W;
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (off[e] >= 0) v |= (uint32_t)(uint8_t)__ldg(plane + off[e]) << (8 * e);
        }
        *reinterpret_cast<uint32_t*>(&tile[r + 16 * k][4 * q]) = v;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int p = p0 + r + 16 * k, c = c0 + 4 * q;
        if (p < P && c < cpad) {  // cpad is a multiple of 4
            const int pl = r + 16 * k;
            const uint32_t v = (uint32_t)(uint8_t)tile[4 * q][pl] | ((uint32_t)(uint8_t)tile[4 * q + 1][pl] << 8) |
                               ((uint32_t)(uint8_t)tile[4 * q + 2][pl] << 16) | ((uint32_t)(uint8_t)tile[4 * q + 3][pl] << 24);
            *reinterpret_cast<uint32_t*>(dst + (size_t)p * cpad + c) = v;
        }
    }
}

// How the tiles of an int8 transposition are turned
enum TransposeForm : int { kTurnBytes, kTurnWords, kTurnVectors, kTurnSubsampled };

struct TransposeArgs {
    const int8_t* in;
    int8_t* out;
    int R, W, pitch, opitch;  // R rows of `pitch` bytes, W of them used -> W rows of `opitch` bytes
    int vec_in, vec_out;      // kTurnBytes
    int H, OH, OW, stride;    // kTurnSubsampled (W: the input's columns)
    Divisor tiles_w, tiles_r;
};

// The int8 counterpart of convert_operands_kernel: the activations' byte transposition and the weights of the same convolution.
// Also the way back (results NHWC -> NCHW, without weights). (128 -> 128 3x3 at 28x28, 256 images: 74.0 -> 68.6 us a call.)
template <int kForm, int TP>
__global__ void __launch_bounds__(256) transpose_bytes_kernel(TransposeArgs a, PackArgs pack, int overlap) {
    sm100::pdl_wait();
    if (overlap) sm100::pdl_launch_dependents();
    if (blockIdx.x < pack.blocks) {
        pack_weights_block<int8_t, int8_t, false>(static_cast<const int8_t*>(pack.w), static_cast<int8_t*>(pack.out), nullptr, pack, blockIdx.x);
        return;
    }
    const unsigned t = blockIdx.x - pack.blocks;
    const unsigned row = a.tiles_w.quotient(t);
    const int tw = (int)(t - row * a.tiles_w.d), n = (int)a.tiles_r.quotient(row), tr = (int)(row - n * a.tiles_r.d);
    if constexpr (kForm == kTurnVectors) transpose_bytes_tile<16, TP>(a.in, a.out, a.R, a.W, a.pitch, a.opitch, tw, tr, n);
    else if constexpr (kForm == kTurnWords) transpose_bytes_tile<4, TP>(a.in, a.out, a.R, a.W, a.pitch, a.opitch, tw, tr, n);
    else if constexpr (kForm == kTurnBytes) transpose_s8_tile(a.in, a.out, a.R, a.W, a.pitch, a.opitch, a.vec_in, a.vec_out, tw, tr, n);
    else subsample_s8_tile(a.in, a.out, a.R, a.H, a.W, a.OH, a.OW, a.stride, a.opitch, tw, tr, n);
}

template <typename TOut>
__global__ void convert_rows_kernel(const float* __restrict__ in, TOut* __restrict__ out, int64_t rows, int cols, int cpad) {
    sm100::pdl_wait();
    const int64_t total = rows * cpad;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int c = (int)(i % cpad);
        const int64_t r = i / cpad;
        out[i] = convert_to<TOut>(c < cols ? in[r * cols + c] : 0.0f);
    }
}

// Both operands of a dense layer (rows of the same length) in one launch: [rows_a, cols] and [rows_b, cols] -> operand type.
// cols == cpad and a multiple of four (the launcher checks the addresses): 16-byte reads, no division (32x512 and 1000x512
// fp32 -> tf32: 1.7 + 4.4 us in two launches of the kernel above).
template <typename TOut>
__global__ void __launch_bounds__(256) convert_two_kernel(const float* __restrict__ a, TOut* __restrict__ out_a, int64_t quads_a,
                                                          const float* __restrict__ b, TOut* __restrict__ out_b, int64_t quads_b) {
    sm100::pdl_wait();
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < quads_a + quads_b; i += step) {
        const bool first = i < quads_a;
        const int64_t q = first ? i : i - quads_a;
        const float4 v = __ldg(reinterpret_cast<const float4*>(first ? a : b) + q);
        alignas(16) TOut o[4] = {convert_to<TOut>(v.x), convert_to<TOut>(v.y), convert_to<TOut>(v.z), convert_to<TOut>(v.w)};
        TOut* dst = (first ? out_a : out_b) + 4 * q;
        if constexpr (sizeof(TOut) == 4) *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(o);
        else *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(o);
    }
}

int grid_1d(int64_t items, int threads) {
    int64_t b = (items + threads - 1) / threads;
    const int64_t cap = (int64_t)kNumSMs * 16;
    if (b > cap) b = cap;
    if (b < 1) b = 1;
    return (int)b;
}

template <typename T>
PackArgs pack_args(const WeightPack* w) {
    PackArgs p;
    if (w == nullptr || (int64_t)w->O * w->taps * w->cpad == 0) return p;
    p.w = w->w; p.out = w->out; p.lo = w->lo;
    p.C = w->C; p.taps = w->taps; p.cpad = w->cpad;
    p.per_row = Divisor((unsigned)(w->cpad / (4 / (int)sizeof(T))));
    p.groups = (int64_t)w->O * p.per_row.d;
    p.per_thread = sizeof(T) == 1 && p.groups >= 48 * 256 ? 9 : kPackTaps<T>;  // (reasons at pack_weights_block)
    p.pieces = Divisor((unsigned)((w->taps + p.per_thread - 1) / p.per_thread));
    p.blocks = (unsigned)(((p.groups + 31) / 32 * p.pieces.d + 7) / 8);
    return p;
}

// Tiles of an activation conversion and the blocks that pack weights, as one grid dimension.
int32_t one_dim_grid(int64_t tiles_a, int64_t tiles_b, int64_t batch, unsigned pack_blocks, unsigned* grid) {
    const int64_t blocks = tiles_a * tiles_b * batch + pack_blocks;
    if (blocks > 0x7fffffffll) return fail(KXC_B200_ERR_UNSUPPORTED, "layout transform: %lld tiles exceed the grid limit", (long long)blocks);
    *grid = (unsigned)blocks;
    return KXC_B200_OK;
}

template <typename TOut, bool kSplit, bool kSub>
int32_t launch_convert(const float* in, void* out, void* lo, int N, int C, int HW, int cpad, const WeightPack* w, cudaStream_t s, bool overlap,
                       const PixelArgs& px = PixelArgs()) {
    const PackArgs pack = pack_args<TOut>(w);
    auto go = [&](auto kernel, int ct) -> int32_t {
        const int tiles_hw = (int)(((int64_t)HW + 2048 / ct - 1) / (2048 / ct)), tiles_c = (cpad + ct - 1) / ct;
        unsigned grid = 0;
        KXC_TRY(one_dim_grid(tiles_hw, tiles_c, N, pack.blocks, &grid));
        KXC_CUDA_TRY(launch_kernel(kernel, dim3(grid), dim3(256), 0, s, /*pdl=*/true, 1, in, static_cast<TOut*>(out), static_cast<TOut*>(lo), C, HW,
                                   cpad, Divisor(tiles_hw), Divisor(tiles_c), pack, overlap ? 1 : 0, px));
        return check_launch("convert_operands");
    };
    if constexpr (sizeof(TOut) == 2) {
        if (cpad > 32) return go(convert_operands_kernel<TOut, kSplit, 64, kSub>, 64);
    }
    return go(convert_operands_kernel<TOut, kSplit, 32, kSub>, 32);
}

// Byte transposition of `batch` matrices, by words turned in registers where pitches and addresses allow it.
int32_t launch_transpose(const int8_t* in, int8_t* out, int batch, int R, int W, int pitch, int opitch, const WeightPack* w, cudaStream_t s,
                         bool overlap) {
    const PackArgs pack = pack_args<int8_t>(w);
    const uintptr_t ia = reinterpret_cast<uintptr_t>(in), oa = reinterpret_cast<uintptr_t>(out);
    TransposeArgs a{};
    a.in = in; a.out = out; a.R = R; a.W = W; a.pitch = pitch; a.opitch = opitch;
    auto go = [&](auto kernel, int tp, int rows) -> int32_t {
        a.tiles_w = Divisor((unsigned)(((int64_t)W + tp - 1) / tp));
        a.tiles_r = Divisor((unsigned)(((int64_t)rows + 63) / 64));
        unsigned grid = 0;
        KXC_TRY(one_dim_grid(a.tiles_w.d, a.tiles_r.d, batch, pack.blocks, &grid));
        KXC_CUDA_TRY(launch_kernel(kernel, dim3(grid), dim3(256), 0, s, /*pdl=*/true, 1, a, pack, overlap ? 1 : 0));
        return check_launch("transpose_bytes");
    };
    if ((pitch & 3) == 0 && (opitch & 3) == 0 && (ia & 3u) == 0 && (oa & 3u) == 0) {
        const int rows = R > opitch ? R : opitch;
        const bool wide = (pitch & 15) == 0 && (ia & 15u) == 0;
        if (W <= 64) return wide ? go(transpose_bytes_kernel<kTurnVectors, 64>, 64, rows) : go(transpose_bytes_kernel<kTurnWords, 64>, 64, rows);
        if (W <= 128) return wide ? go(transpose_bytes_kernel<kTurnVectors, 128>, 128, rows) : go(transpose_bytes_kernel<kTurnWords, 128>, 128, rows);
        return wide ? go(transpose_bytes_kernel<kTurnVectors, 256>, 256, rows) : go(transpose_bytes_kernel<kTurnWords, 256>, 256, rows);
    }
    a.vec_in = (pitch & 3) == 0 && (ia & 3u) == 0;
    a.vec_out = (opitch & 3) == 0 && (oa & 3u) == 0;
    return go(transpose_bytes_kernel<kTurnBytes, 64>, 64, opitch);
}

}  // namespace

int32_t convert_operands(const void* in, void* out, void* lo, TcDType dtype, int N, int C, int HW, int cpad, const WeightPack* w, cudaStream_t s,
                         bool overlap) {
    if (N == 0) return KXC_B200_OK;
    if (N > 65535) return fail(KXC_B200_ERR_UNSUPPORTED, "layout transform: batch %d exceeds the grid limit", N);
    const float* f = static_cast<const float*>(in);
    switch (dtype) {
        case kTcBF16: return launch_convert<__nv_bfloat16, false, false>(f, out, nullptr, N, C, HW, cpad, w, s, overlap);
        case kTcTF32:
            return lo != nullptr ? launch_convert<float, true, false>(f, out, lo, N, C, HW, cpad, w, s, overlap)
                                 : launch_convert<float, false, false>(f, out, nullptr, N, C, HW, cpad, w, s, overlap);
        case kTcS8: return launch_transpose(static_cast<const int8_t*>(in), static_cast<int8_t*>(out), N, C, HW, HW, cpad, w, s, overlap);
    }
    return fail(KXC_B200_ERR_INVALID, "convert_operands: dtype");
}

int32_t convert_rows_two(const float* a, void* out_a, int64_t rows_a, const float* b, void* out_b, int64_t rows_b, TcDType dtype, int cols,
                         int cpad, cudaStream_t s) {
    const uintptr_t addr = reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b);
    if (cols != cpad || (cols & 3) != 0 || (addr & 15u) != 0 || rows_a + rows_b == 0 || (dtype != kTcBF16 && dtype != kTcTF32)) {
        KXC_TRY(convert_rows(a, out_a, dtype, rows_a, cols, cpad, s));
        return convert_rows(b, out_b, dtype, rows_b, cols, cpad, s);
    }
    const int64_t qa = rows_a * cols / 4, qb = rows_b * cols / 4;
    const int grid = grid_1d(qa + qb, 256);
    if (dtype == kTcBF16)
        KXC_CUDA_TRY(launch_kernel(convert_two_kernel<__nv_bfloat16>, dim3(grid), dim3(256), 0, s, /*pdl=*/true, 1, a,
                                   static_cast<__nv_bfloat16*>(out_a), qa, b, static_cast<__nv_bfloat16*>(out_b), qb));
    else
        KXC_CUDA_TRY(launch_kernel(convert_two_kernel<float>, dim3(grid), dim3(256), 0, s, /*pdl=*/true, 1, a, static_cast<float*>(out_a), qa, b,
                                   static_cast<float*>(out_b), qb));
    return check_launch("convert_rows_two");
}

int32_t split_rows(const float* in, float* hi, float* lo, int64_t rows, int cols, int cpad, cudaStream_t s) {
    if (rows * cpad == 0) return KXC_B200_OK;
    const bool vec = cols == cpad && (cols & 3) == 0;
    if (vec && ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(hi) | reinterpret_cast<uintptr_t>(lo)) & 15u) != 0) {
        // a caller's matrix that is not 16-byte aligned: element by element
        KXC_TRY(convert_rows(in, hi, kTcTF32, rows, cols, cpad, s, false));
        return convert_rows(in, lo, kTcTF32, rows, cols, cpad, s, true);
    }
    KXC_CUDA_TRY(launch_kernel(split_rows_kernel, dim3(grid_1d(vec ? rows * cols / 4 : rows * cpad, 256)), dim3(256), 0, s, /*pdl=*/true, 1, in, hi,
                               lo, rows, cols, cpad));
    return check_launch("split_rows");
}

int32_t convert_operands_subsample(const float* in, void* out, void* lo, TcDType dtype, int N, int C, int H, int W, int OH, int OW, int stride, int cpad,
                                   const WeightPack* w, cudaStream_t s, bool overlap) {
    if (N == 0) return KXC_B200_OK;
    if (N > 65535 || (long long)H * W > 0x7fffffffll) return fail(KXC_B200_ERR_UNSUPPORTED, "layout transform: %d images of %dx%d", N, H, W);
    PixelArgs px;
    px.plane = H * W; px.W = W; px.st = stride; px.by_ow = Divisor((unsigned)OW);
    if (dtype == kTcBF16) return launch_convert<__nv_bfloat16, false, true>(in, out, nullptr, N, C, OH * OW, cpad, w, s, overlap, px);
    return lo != nullptr ? launch_convert<float, true, true>(in, out, lo, N, C, OH * OW, cpad, w, s, overlap, px)
                         : launch_convert<float, false, true>(in, out, nullptr, N, C, OH * OW, cpad, w, s, overlap, px);
}

int32_t convert_operands_s8_subsample(const int8_t* in, int8_t* out, int N, int C, int H, int W, int OH, int OW, int stride, int cpad,
                                      const WeightPack* w, cudaStream_t s, bool overlap) {
    if (N == 0 || C == 0 || OH == 0 || OW == 0) return KXC_B200_OK;
    if ((cpad & 3) != 0 || (reinterpret_cast<uintptr_t>(out) & 3u) != 0 || N > 65535 || (long long)H * W > 0x7fffffffll)
        return fail(KXC_B200_ERR_UNSUPPORTED, "convert_operands_s8_subsample: %d padded channels, %d images", cpad, N);
    const PackArgs pack = pack_args<int8_t>(w);
    TransposeArgs a{};
    a.in = in; a.out = out; a.R = C; a.W = W; a.opitch = cpad;
    a.H = H; a.OH = OH; a.OW = OW; a.stride = stride;
    a.tiles_w = Divisor((unsigned)((OH * OW + 63) / 64));
    a.tiles_r = Divisor((unsigned)((cpad + 63) / 64));
    unsigned grid = 0;
    KXC_TRY(one_dim_grid(a.tiles_w.d, a.tiles_r.d, N, pack.blocks, &grid));
    KXC_CUDA_TRY(launch_kernel(transpose_bytes_kernel<kTurnSubsampled, 64>, dim3(grid), dim3(256), 0, s, /*pdl=*/true, 1, a, pack, overlap ? 1 : 0));
    return check_launch("convert_operands_s8_subsample");
}

int32_t nhwc_to_nchw_s8(const int8_t* in, int8_t* out, int N, int C, int pitch, int HW, cudaStream_t s) {
    if (N == 0 || C == 0 || HW == 0) return KXC_B200_OK;
    // source rows = pixels (C bytes of `pitch`), destination rows = channels (HW bytes each)
    return launch_transpose(in, out, N, HW, C, pitch, HW, nullptr, s, false);
}

int32_t pack_weights_ohwi(const WeightPack& w, TcDType dtype, cudaStream_t s) {
    auto go = [&](auto kernel, const PackArgs& p) -> int32_t {
        if (p.blocks == 0) return KXC_B200_OK;
        KXC_CUDA_TRY(launch_kernel(kernel, dim3(p.blocks), dim3(256), 0, s, /*pdl=*/true, 1, p));
        return check_launch("pack_weights");
    };
    switch (dtype) {
        case kTcBF16: return go(pack_weights_kernel<float, __nv_bfloat16, false>, pack_args<__nv_bfloat16>(&w));
        case kTcTF32:
            return w.lo != nullptr ? go(pack_weights_kernel<float, float, true>, pack_args<float>(&w))
                                   : go(pack_weights_kernel<float, float, false>, pack_args<float>(&w));
        case kTcS8: return go(pack_weights_kernel<int8_t, int8_t, false>, pack_args<int8_t>(&w));
    }
    return fail(KXC_B200_ERR_INVALID, "pack_weights: dtype");
}

int32_t convert_rows(const float* in, void* out, TcDType dtype, int64_t rows, int cols, int cpad, cudaStream_t s, bool tf32_lo) {
    const int64_t total = rows * cpad;
    if (total == 0) return KXC_B200_OK;
    const int grid = grid_1d(total, 256);
    if (dtype == kTcBF16)
        KXC_CUDA_TRY(launch_kernel(convert_rows_kernel<__nv_bfloat16>, dim3(grid), dim3(256), 0, s, /*pdl=*/true, 1, in,
                                   static_cast<__nv_bfloat16*>(out), rows, cols, cpad));
    else if (dtype == kTcTF32 && tf32_lo)
        KXC_CUDA_TRY(launch_kernel(convert_rows_kernel<Tf32Lo>, dim3(grid), dim3(256), 0, s, /*pdl=*/true, 1, in, static_cast<Tf32Lo*>(out), rows,
                                   cols, cpad));
    else if (dtype == kTcTF32)
        KXC_CUDA_TRY(launch_kernel(convert_rows_kernel<float>, dim3(grid), dim3(256), 0, s, /*pdl=*/true, 1, in, static_cast<float*>(out), rows, cols,
                                   cpad));
    else
        return fail(KXC_B200_ERR_INVALID, "convert_rows: dtype");
    return check_launch("convert_rows");
}

}  // namespace kxc_b200
