// Convolution with the output channels as the MMA's rows (conv_chmajor.cu): into the reference's layout bf16 and tf32 operands with fp32
// results, int8 with requantized ones; into NHWC bf16 and tf32. Activations NHWC of `cpad` channels, weights [Cout][KH * KW][w_cpad], both of the operand
// type and in multiples of 16 bytes.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "conv_tc.cuh"
#include "divisor.cuh"

namespace kxc_b200 {

struct alignas(64) CmParams {
    static constexpr int kMaxTaps = 64, kMaxLoads = 25, kMaxGroup = 4;
    // taps of one loaded box whose weights share a slot of their ring
    struct Group {
        unsigned short shift[kMaxGroup];  // first row of a tap's view of its box, in units of 16 bytes
        unsigned char tap[kMaxGroup];     // its place in the packed weights
        unsigned char count, first, last, pad;  // taps; the first and the last group of its box
    };
    CUtensorMap tmA[4];  // stride 1: [0]; stride 2: one map per (row parity, column parity) of the input
    CUtensorMap tmW;     // channels, output channels, taps
    int N, OH, OW, Cout;
    int kb_elems, cblocks, last_steps;  // elements of a channel block; blocks; MMAs of the last block
    int BW, BH, BNI;                    // tile box: columns x rows x images of results
    int HB, WB;                         // rows and columns of a loaded box (the tile and the halo of its taps)
    int ctas;                           // 2: a pair of CTAs, 256 channels and two boxes to a tile
    int n_cols;                         // columns of the accumulator: flat pixels of the loaded boxes, a multiple of 16
    int tiles_w, tiles_h, tiles_n, tiles_c;
    Divisor by_c, by_w, by_h;           // of the first three extents of a tile's number: tiles_c, tiles_w, tiles_h
    int zero_bytes;                     // behind a box: padding that its last taps read
    int px_bytes, px_slot_bytes, px_slots, w_tap_bytes, w_slot_bytes, w_slots;
    int loads, groups;                  // per channel block
    int relu;
    int pixels;                         // bf16 and tf32: results NHWC, bf16 or fp32 (round_out_tf32: rounded to tf32), else planes
    int round_out_tf32;
    int weights_ready;                  // as TcParams::weights_ready
    long long max_abs_acc;              // int8: bound of an accumulator
    const float* bias;
    const int32_t* bias_i32;
    const int32_t* multiplier;
    const int32_t* shift;
    const void* residual;
    void* out;
    int* status;
    int load_h[kMaxLoads], load_w[kMaxLoads];  // first row and column of the box, from the tile's first pixel (paddings and dilations have 24 bits)
    unsigned char load_map[kMaxLoads];
    Group group[kMaxTaps + 1];
};

struct CmGeometry {
    int N, H, W, Cout, KH, KW, stride, pad_h, pad_w, dil_h, dil_w, OH, OW, pixels, eb, kb_elems, cblocks, last_steps, epi_parts;
};
struct CmChoice {
    double cost, clocks;  // modelled clocks of single CTAs; of either form (box_cost)
    int shared, ctas, BW, BH, BNI, HB, WB, n, zero_rows, px_slots, w_slots, group;
};

struct CmPlan {
    CmGeometry g;
    CmChoice c;
};

// Whether a convolution into the reference's layout or NHWC (`out_mode`) takes this form, and its tile box; null: it does not. Looked up in the calling thread's
// last choices, which depend on the geometry and the device alone; valid until the thread's next call.
const CmPlan* cm_wanted(TcDType dtype, const ConvDims& d, int weights_ready, TcOutMode out_mode = kOutNCHW_F32, bool residual = false);
// `status_word`: as in tc_setup_conv.
int32_t cm_setup(CmParams* p, TcDType dtype, const CmPlan& plan, const void* act_nhwc, const void* w_packed, int cpad, int w_cpad, int* status_word = nullptr);
int32_t cm_launch(TcDType dtype, const CmParams& p, cudaStream_t stream);

// Channels that an operator pads its pixels to: whole 32-byte sectors (pixels of 16 bytes more made the copies up to twice as long: tf32 1 -> 76
// 5x5 at 46x44, 28 images, a call 31.7 -> 21.1 us; int8 44 -> 46 3x3 of stride 2 at 53x56, 85 images 31.6 -> 23.5; none of 420 drawn layers lost 2 %).
inline int cm_channel_pad(TcDType t, int c) {
    const int e32 = 32 / tc_elem_bytes(t);
    return (c + e32 - 1) / e32 * e32;
}
// ... and its filters' taps. Of a launch with more tiles than SMs, which loads them once per tile: whole rows of 128 bytes, the copies' unit
// (int8, a call, with sectors / so: 11 -> 137 5x5 at 20x19, 235 images 98.3 / 50.1 us, 16 -> 158 5x5 at 63x65, 18 images 65.2 / 39.0). One wave
// does not earn back the longer packing (64 -> 32 3x3 at 8x11, one image 7.3 / 7.6).
int cm_weight_pad(TcDType t, int c, const CmPlan& plan);

}  // namespace kxc_b200
