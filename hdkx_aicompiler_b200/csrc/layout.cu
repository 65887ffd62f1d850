// Layout / precision conversion kernels (HBM-bound, coalesced on both sides through a shared-memory
// transpose tile).
#include "layout.cuh"

#include <cuda_bf16.h>

#include "common.cuh"
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

template <typename TIn, typename TOut>
__device__ __forceinline__ TOut convert_elem(TIn v) { return convert_to<TOut>((float)v); }
template <>
__device__ __forceinline__ int8_t convert_elem<int8_t, int8_t>(int8_t v) { return v; }

// `overlap` (here and in pack_weights_kernel): the next kernel's CTAs may set themselves up while this one runs; they wait for its
// end before they read. Never for weights that a kernel reads ahead of its predecessor's end: those of a plan
// (TcParams::weights_ready) and of the row-stacked kernels.
// grid (ceil(HW/32), ceil(cpad/32), N), block (32, 8)
template <typename TIn, typename TOut>
__global__ void nchw_to_nhwc_kernel(const TIn* __restrict__ in, TOut* __restrict__ out, int C, int HW, int cpad, int overlap) {
    if (overlap) sm100::pdl_launch_dependents();
    __shared__ TIn tile[32][33];
    const int n = blockIdx.z;
    const int hw0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
    const TIn* src = in + (size_t)n * C * HW;
    TOut* dst = out + (size_t)n * HW * cpad;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int c = c0 + threadIdx.y + 8 * k, hw = hw0 + threadIdx.x;
        tile[threadIdx.y + 8 * k][threadIdx.x] = (c < C && hw < HW) ? src[(size_t)c * HW + hw] : (TIn)0;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int hw = hw0 + threadIdx.y + 8 * k, c = c0 + threadIdx.x;
        if (hw < HW && c < cpad) dst[(size_t)hw * cpad + c] = convert_elem<TIn, TOut>(tile[threadIdx.x][threadIdx.y + 8 * k]);
    }
}

// Both tf32 parts of every value in one pass over the input (three-pass tf32). Same grid and block.
__global__ void nchw_to_nhwc_split_kernel(const float* __restrict__ in, float* __restrict__ hi, float* __restrict__ lo, int C, int HW, int cpad) {
    __shared__ float tile[32][33];
    const int n = blockIdx.z;
    const int hw0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
    const float* src = in + (size_t)n * C * HW;
    const size_t dst = (size_t)n * HW * cpad;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int c = c0 + threadIdx.y + 8 * k, hw = hw0 + threadIdx.x;
        tile[threadIdx.y + 8 * k][threadIdx.x] = (c < C && hw < HW) ? src[(size_t)c * HW + hw] : 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int hw = hw0 + threadIdx.y + 8 * k, c = c0 + threadIdx.x;
        if (hw < HW && c < cpad) {
            const float v = tile[threadIdx.x][threadIdx.y + 8 * k];
            hi[dst + (size_t)hw * cpad + c] = convert_to<float>(v);
            lo[dst + (size_t)hw * cpad + c] = convert_to<Tf32Lo>(v).v;
        }
    }
}

// The same for rows that need no reordering: [rows, cols] -> two times [rows, cpad]. cols % 4 == 0 and cols == cpad take
// 16-byte accesses (bound by memory: 4 bytes read and 8 written per value).
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ in, float* __restrict__ hi, float* __restrict__ lo, int64_t rows,
                                                         int cols, int cpad) {
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
// 32-byte runs the element-wise kernel makes of 1-byte elements). grid (ceil(HW/64), ceil(cpad/64), N), block 256.
// It is a batched byte transpose [C][HW] -> [HW][cpad] (rows c >= C read as zero), so it also serves NHWC -> NCHW with
// the roles of the two extents exchanged (source rows `pitch` bytes apart); vec_out = 0 when the destination rows are not 4-byte multiples.
// rows_on_x (here and in transpose_bytes_kernel): the first two grid dimensions are exchanged, see transpose_grid.
__global__ void __launch_bounds__(256) nchw_to_nhwc_s8_kernel(const int8_t* __restrict__ in, int8_t* __restrict__ out, int C, int HW,
                                                               int pitch, int cpad, int vec_in, int vec_out, int rows_on_x) {
    __shared__ __align__(4) int8_t tile[64][68];
    const int n = blockIdx.z;
    const int hw0 = (int)(rows_on_x ? blockIdx.y : blockIdx.x) * 64, c0 = (int)(rows_on_x ? blockIdx.x : blockIdx.y) * 64;
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
// Tile 64 rows x TP columns. grid (ceil(W/TP), ceil(max(R, opitch)/64), batch), block 256.
template <int V, int TP>
__global__ void __launch_bounds__(256) transpose_bytes_kernel(const int8_t* __restrict__ in, int8_t* __restrict__ out, int R, int W, int pitch,
                                                               int opitch, int rows_on_x) {
    __shared__ uint32_t tile[TP * 16];
    const int w0 = (int)(rows_on_x ? blockIdx.y : blockIdx.x) * TP, r0 = (int)(rows_on_x ? blockIdx.x : blockIdx.y) * 64;
    const int8_t* src = in + (int64_t)blockIdx.z * R * pitch;
    int8_t* dst = out + (int64_t)blockIdx.z * W * opitch;
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

// Grid of a batched transpose: column tiles, row tiles, batch. The row tiles of a whole plane (NHWC -> NCHW: pixels) can be more
// than the 65535 that the second dimension holds; they change places with the column tiles then, of which there are few.
dim3 transpose_grid(int cols, int rows, int batch, int* rows_on_x) {
    *rows_on_x = rows > 65535 ? 1 : 0;
    return *rows_on_x ? dim3((unsigned)rows, (unsigned)cols, (unsigned)batch) : dim3((unsigned)cols, (unsigned)rows, (unsigned)batch);
}

// Batched byte transpose of `batch` matrices; false when the pitches or addresses do not suit the kernel above.
bool transpose_bytes(const int8_t* in, int8_t* out, int batch, int R, int W, int pitch, int opitch, cudaStream_t s) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(in);
    if ((pitch & 3) != 0 || (opitch & 3) != 0 || (a & 3u) != 0 || (reinterpret_cast<uintptr_t>(out) & 3u) != 0) return false;
    const bool wide = (pitch & 15) == 0 && (a & 15u) == 0;
    const int tp = W <= 64 ? 64 : (W <= 128 ? 128 : 256);
    int rows_on_x = 0;
    const dim3 grid = transpose_grid((W + tp - 1) / tp, ((R > opitch ? R : opitch) + 63) / 64, batch, &rows_on_x);
    auto go = [&](auto kernel) { kernel<<<grid, 256, 0, s>>>(in, out, R, W, pitch, opitch, rows_on_x); };
    if (wide) {
        if (tp == 64) go(transpose_bytes_kernel<16, 64>);
        else if (tp == 128) go(transpose_bytes_kernel<16, 128>);
        else go(transpose_bytes_kernel<16, 256>);
    } else {
        if (tp == 64) go(transpose_bytes_kernel<4, 64>);
        else if (tp == 128) go(transpose_bytes_kernel<4, 128>);
        else go(transpose_bytes_kernel<4, 256>);
    }
    return true;
}

// int8 NCHW -> NHWC of the pixels a 1x1 convolution of stride `st` (no padding) reads: out[n][p][c] =
// in[n][c][(p / OW) * st][(p % OW) * st], p = oh * OW + ow. grid (ceil(OH*OW/64), ceil(cpad/64), N), block 256: the same
// 64 x 64 byte transpose as above with gathered source pixels; the rows the convolution skips are never touched.
__global__ void __launch_bounds__(256) nchw_to_nhwc_s8_subsample_kernel(const int8_t* __restrict__ in, int8_t* __restrict__ out, int C,
                                                                         int H, int W, int OH, int OW, int st, int cpad) {
    __shared__ __align__(4) int8_t tile[64][68];
    const int n = blockIdx.z;
    const int p0 = blockIdx.x * 64, c0 = blockIdx.y * 64;
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

template <typename TIn, typename TOut>
__global__ void pack_weights_kernel(const TIn* __restrict__ w, TOut* __restrict__ out, int O, int C, int KH, int KW, int cpad, int overlap) {
    if (overlap) sm100::pdl_launch_dependents();
    const int64_t total = (int64_t)O * KH * KW * cpad;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int c = (int)(i % cpad);
        int64_t t = i / cpad;
        const int kw = (int)(t % KW); t /= KW;
        const int kh = (int)(t % KH);
        const int o = (int)(t / KH);
        out[i] = c < C ? convert_elem<TIn, TOut>(w[(((int64_t)o * C + c) * KH + kh) * KW + kw]) : convert_elem<TIn, TOut>((TIn)0);
    }
}

template <typename TOut>
__global__ void convert_rows_kernel(const float* __restrict__ in, TOut* __restrict__ out, int64_t rows, int cols, int cpad) {
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

}  // namespace

int32_t nchw_to_nhwc(const void* in, void* out, TcDType dtype, int N, int C, int HW, int cpad, cudaStream_t s, bool tf32_lo, bool overlap) {
    if (N == 0) return KXC_B200_OK;
    if (N > 65535) return fail(KXC_B200_ERR_UNSUPPORTED, "layout transform: batch %d exceeds the grid limit", N);
    const dim3 grid((HW + 31) / 32, (cpad + 31) / 32, N), block(32, 8);
    switch (dtype) {
        case kTcBF16:
            nchw_to_nhwc_kernel<float, __nv_bfloat16><<<grid, block, 0, s>>>(static_cast<const float*>(in), static_cast<__nv_bfloat16*>(out), C, HW, cpad, overlap ? 1 : 0);
            break;
        case kTcTF32:
            if (tf32_lo)
                nchw_to_nhwc_kernel<float, Tf32Lo><<<grid, block, 0, s>>>(static_cast<const float*>(in), static_cast<Tf32Lo*>(out), C, HW, cpad, overlap ? 1 : 0);
            else
                nchw_to_nhwc_kernel<float, float><<<grid, block, 0, s>>>(static_cast<const float*>(in), static_cast<float*>(out), C, HW, cpad, overlap ? 1 : 0);
            break;
        case kTcS8:
            if (transpose_bytes(static_cast<const int8_t*>(in), static_cast<int8_t*>(out), N, C, HW, HW, cpad, s)) break;
            if ((cpad & 3) == 0 && (reinterpret_cast<uintptr_t>(out) & 3u) == 0) {
                const int vec_in = ((HW & 3) == 0 && (reinterpret_cast<uintptr_t>(in) & 3u) == 0) ? 1 : 0;
                int rows_on_x = 0;
                const dim3 g = transpose_grid((HW + 63) / 64, (cpad + 63) / 64, N, &rows_on_x);
                nchw_to_nhwc_s8_kernel<<<g, 256, 0, s>>>(static_cast<const int8_t*>(in), static_cast<int8_t*>(out), C, HW, HW, cpad, vec_in, 1, rows_on_x);
            } else {
                nchw_to_nhwc_kernel<int8_t, int8_t><<<grid, block, 0, s>>>(static_cast<const int8_t*>(in), static_cast<int8_t*>(out), C, HW, cpad, overlap ? 1 : 0);
            }
            break;
    }
    return check_launch("nchw_to_nhwc");
}

int32_t nchw_to_nhwc_split(const float* in, float* hi, float* lo, int N, int C, int HW, int cpad, cudaStream_t s) {
    if (N == 0) return KXC_B200_OK;
    if (N > 65535) return fail(KXC_B200_ERR_UNSUPPORTED, "layout transform: batch %d exceeds the grid limit", N);
    nchw_to_nhwc_split_kernel<<<dim3((HW + 31) / 32, (cpad + 31) / 32, N), dim3(32, 8), 0, s>>>(in, hi, lo, C, HW, cpad);
    return check_launch("nchw_to_nhwc_split");
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
        convert_two_kernel<__nv_bfloat16><<<grid, 256, 0, s>>>(a, static_cast<__nv_bfloat16*>(out_a), qa, b, static_cast<__nv_bfloat16*>(out_b), qb);
    else
        convert_two_kernel<float><<<grid, 256, 0, s>>>(a, static_cast<float*>(out_a), qa, b, static_cast<float*>(out_b), qb);
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
    split_rows_kernel<<<grid_1d(vec ? rows * cols / 4 : rows * cpad, 256), 256, 0, s>>>(in, hi, lo, rows, cols, cpad);
    return check_launch("split_rows");
}

int32_t nchw_to_nhwc_s8_subsample(const int8_t* in, int8_t* out, int N, int C, int H, int W, int OH, int OW, int stride, int cpad,
                                  cudaStream_t s) {
    if (N == 0 || C == 0 || OH == 0 || OW == 0) return KXC_B200_OK;
    if ((cpad & 3) != 0 || (reinterpret_cast<uintptr_t>(out) & 3u) != 0 || N > 65535 || (long long)H * W > 0x7fffffffll)
        return fail(KXC_B200_ERR_UNSUPPORTED, "nchw_to_nhwc_s8_subsample: %d padded channels, %d images", cpad, N);
    nchw_to_nhwc_s8_subsample_kernel<<<dim3((OH * OW + 63) / 64, (cpad + 63) / 64, N), 256, 0, s>>>(in, out, C, H, W, OH, OW, stride, cpad);
    return check_launch("nchw_to_nhwc_s8_subsample");
}

int32_t nhwc_to_nchw_s8(const int8_t* in, int8_t* out, int N, int C, int pitch, int HW, cudaStream_t s) {
    if (N == 0 || C == 0 || HW == 0) return KXC_B200_OK;
    // source rows = pixels (C bytes of `pitch`), destination rows = channels (HW bytes each)
    if (!transpose_bytes(in, out, N, HW, C, pitch, HW, s)) {
        const int vec_in = ((pitch & 3) == 0 && (reinterpret_cast<uintptr_t>(in) & 3u) == 0) ? 1 : 0;
        const int vec_out = ((HW & 3) == 0 && (reinterpret_cast<uintptr_t>(out) & 3u) == 0) ? 1 : 0;
        int rows_on_x = 0;
        const dim3 g = transpose_grid((C + 63) / 64, (HW + 63) / 64, N, &rows_on_x);
        nchw_to_nhwc_s8_kernel<<<g, 256, 0, s>>>(in, out, HW, C, pitch, HW, vec_in, vec_out, rows_on_x);
    }
    return check_launch("nhwc_to_nchw_s8");
}

int32_t pack_weights_ohwi(const void* w, void* out, TcDType dtype, int O, int C, int KH, int KW, int cpad, cudaStream_t s, bool tf32_lo, bool overlap) {
    const int64_t total = (int64_t)O * KH * KW * cpad;
    const int grid = grid_1d(total, 256);
    switch (dtype) {
        case kTcBF16:
            pack_weights_kernel<float, __nv_bfloat16><<<grid, 256, 0, s>>>(static_cast<const float*>(w), static_cast<__nv_bfloat16*>(out), O, C, KH, KW, cpad, overlap ? 1 : 0);
            break;
        case kTcTF32:
            if (tf32_lo)
                pack_weights_kernel<float, Tf32Lo><<<grid, 256, 0, s>>>(static_cast<const float*>(w), static_cast<Tf32Lo*>(out), O, C, KH, KW, cpad, overlap ? 1 : 0);
            else
                pack_weights_kernel<float, float><<<grid, 256, 0, s>>>(static_cast<const float*>(w), static_cast<float*>(out), O, C, KH, KW, cpad, overlap ? 1 : 0);
            break;
        case kTcS8:
            pack_weights_kernel<int8_t, int8_t><<<grid, 256, 0, s>>>(static_cast<const int8_t*>(w), static_cast<int8_t*>(out), O, C, KH, KW, cpad, overlap ? 1 : 0);
            break;
    }
    return check_launch("pack_weights");
}

int32_t convert_rows(const float* in, void* out, TcDType dtype, int64_t rows, int cols, int cpad, cudaStream_t s, bool tf32_lo) {
    const int64_t total = rows * cpad;
    if (total == 0) return KXC_B200_OK;
    const int grid = grid_1d(total, 256);
    if (dtype == kTcBF16)
        convert_rows_kernel<__nv_bfloat16><<<grid, 256, 0, s>>>(in, static_cast<__nv_bfloat16*>(out), rows, cols, cpad);
    else if (dtype == kTcTF32 && tf32_lo)
        convert_rows_kernel<Tf32Lo><<<grid, 256, 0, s>>>(in, static_cast<Tf32Lo*>(out), rows, cols, cpad);
    else if (dtype == kTcTF32)
        convert_rows_kernel<float><<<grid, 256, 0, s>>>(in, static_cast<float*>(out), rows, cols, cpad);
    else
        return fail(KXC_B200_ERR_INVALID, "convert_rows: dtype");
    return check_launch("convert_rows");
}

}  // namespace kxc_b200
