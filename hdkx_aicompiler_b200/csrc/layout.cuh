// Layout / precision conversions at the edges of the tensor-core path.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "conv_tc.cuh"

namespace kxc_b200 {

// The weights of a convolution: OIHW (fp32 or int8) -> [O][taps][cpad] in the operand type; `lo` (tf32 only, may be null): the
// tf32 rounding of what the tf32 rounding dropped.
struct WeightPack {
    const void* w;
    void* out;
    void* lo;
    int O, C, taps, cpad;
};
int32_t pack_weights_ohwi(const WeightPack& w, TcDType dtype, cudaStream_t s);

// NCHW (fp32 or int8) -> NHWC with `cpad` channels (zero filled), converted to the tensor-core
// operand type: bf16 (round to nearest even), tf32 kept in fp32 storage (low 13 mantissa bits
// rounded away, nearest even; `lo`, if not null, as for the weights), or int8 (copied). `weights` (may be null) are packed by the
// same launch. `overlap`: the next kernel's CTAs may set themselves up meanwhile; not when it reads `weights` ahead of this launch's end.
int32_t convert_operands(const void* in, void* out, void* lo, TcDType dtype, int N, int C, int HW, int cpad, const WeightPack* weights,
                         cudaStream_t s, bool overlap);

// The int8 form of it for only the pixels a 1x1 convolution of stride `stride` without padding reads:
// out[n][oh][ow][c] = in[n][c][oh*stride][ow*stride], channels zero-filled up to cpad (a multiple of 4).
int32_t convert_operands_s8_subsample(const int8_t* in, int8_t* out, int N, int C, int H, int W, int OH, int OW, int stride, int cpad,
                                      const WeightPack* weights, cudaStream_t s, bool overlap);

// bf16 and tf32: `lo` as for convert_operands.
int32_t convert_operands_subsample(const float* in, void* out, void* lo, TcDType dtype, int N, int C, int H, int W, int OH, int OW, int stride, int cpad,
                                   const WeightPack* weights, cudaStream_t s, bool overlap);

// convert_rows of two matrices with rows of the same length, in one launch where extents and addresses allow it.
int32_t convert_rows_two(const float* a, void* out_a, int64_t rows_a, const float* b, void* out_b, int64_t rows_b, TcDType dtype, int cols,
                         int cpad, cudaStream_t s);

// Three-pass tf32 operands: the tf32 rounding of every value (hi) and the tf32 rounding of what that dropped (lo).
int32_t split_rows(const float* in, float* hi, float* lo, int64_t rows, int cols, int cpad, cudaStream_t s);

// int8 NHWC [N][HW][C of pitch] -> NCHW [N][C][HW] (the reference layout of a requantized result).
int32_t nhwc_to_nchw_s8(const int8_t* in, int8_t* out, int N, int C, int pitch, int HW, cudaStream_t s);

// Row-major [rows, cols] fp32 -> [rows, cpad] operand type (dense operands).
int32_t convert_rows(const float* in, void* out, TcDType dtype, int64_t rows, int cols, int cpad, cudaStream_t s, bool tf32_lo = false);

}  // namespace kxc_b200
