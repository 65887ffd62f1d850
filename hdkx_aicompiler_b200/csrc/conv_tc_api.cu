// Per-operator glue between the reference-layout entry points (NCHW fp32 / int8 tensors) and the
// tensor-core implicit-GEMM kernel: operand conversion into a stream-ordered workspace, parameter
// set-up, launch. Shapes the tensor-core path does not take fall back to the CUDA-core kernels
// (still on the GPU; there is no CPU path).
#include <cstdlib>

#include "common.cuh"
#include "conv_chmajor.cuh"
#include "conv_common.cuh"
#include "conv_tc.cuh"
#include "layout.cuh"
#include "sm100.cuh"
#include "conv_rowstack.cuh"
#include "conv_stem.cuh"

#include <mutex>

namespace kxc_b200 {

namespace {

// The library's own stream-ordered memory pool, one per device, that keeps what it has allocated (release threshold =
// unlimited). The device's default pool gives freed memory back to the driver at the next synchronisation, so a caller that
// synchronises between calls would pay a fresh device allocation (milliseconds for tens of MB) inside every call.
int32_t scratch_pool(cudaMemPool_t* out) {
    static std::mutex mu;
    static cudaMemPool_t pools[PerDeviceOnce::kMaxDevices] = {};
    int dev = 0;
    KXC_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= PerDeviceOnce::kMaxDevices) return fail(KXC_B200_ERR_INVALID, "device ordinal %d out of range", dev);
    std::lock_guard<std::mutex> lock(mu);
    if (pools[dev] == nullptr) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.handleTypes = cudaMemHandleTypeNone;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        KXC_CUDA_TRY(cudaMemPoolCreate(&pool, &props));
        uint64_t keep = UINT64_MAX;
        KXC_CUDA_TRY(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
        pools[dev] = pool;
    }
    *out = pools[dev];
    return KXC_B200_OK;
}

// Stream-ordered scratch: allocated and freed on the caller's stream, so the call stays asynchronous.
struct StreamScratch {
    void* ptr = nullptr;
    cudaStream_t stream;
    explicit StreamScratch(cudaStream_t s) : stream(s) {}
    int32_t alloc(size_t bytes) {
        cudaMemPool_t pool = nullptr;
        KXC_TRY(scratch_pool(&pool));
        cudaError_t e = cudaMallocFromPoolAsync(&ptr, bytes, pool, stream);
        if (e != cudaSuccess) {
            ptr = nullptr;
            cudaGetLastError();  // reported here: a launch after it (a caller's smaller request) has its own result
            return fail(KXC_B200_ERR_NOMEM, "workspace of %zu bytes: %s", bytes, cudaGetErrorString(e));
        }
        return KXC_B200_OK;
    }
    ~StreamScratch() {
        if (ptr) cudaFreeAsync(ptr, stream);
    }
};

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

bool tc_shape_ok(const ConvDims& d) {
    return d.SH == d.SW && (d.SH == 1 || d.SH == 2) && !(d.SH == 2 && (d.H < 2 || d.W < 2)) && d.N <= 65535;
}

// A 1x1 convolution of stride > 1 without padding reads one pixel in stride^2; the same over those pixels alone.
bool subsampled(const ConvDims& d) {
    return d.KH == 1 && d.KW == 1 && d.PH == 0 && d.PW == 0 && d.SH == d.SW && d.SH > 1 && d.N <= 65535;
}
ConvDims without_stride(ConvDims d) {
    d.H = d.OH;
    d.W = d.OW;
    d.SH = d.SW = 1;
    return d;
}

}  // namespace

int32_t conv2d_tensor_core(const float* data, const float* weight, const float* bias, const float* residual, float* out,
                           const ConvDims& whole, int relu, int precision, cudaStream_t s) {
    if (!tc_shape_ok(whole)) return conv2d_fp32_exact(data, weight, bias, residual, out, whole, relu, s);
    // A 1x1 convolution of stride 2 without padding reads a quarter of the pixels: only those are converted, and the kernel has stride 1
    const bool sub = subsampled(whole);
    const ConvDims d = sub ? without_stride(whole) : whole;
    auto convert = [&](void* act, void* lo, TcDType dt, int cpad, const WeightPack* pack) {
        return sub ? convert_operands_subsample(data, act, lo, dt, d.N, d.C, whole.H, whole.W, d.OH, d.OW, whole.SH, cpad, pack, s, true)
                   : convert_operands(data, act, lo, dt, d.N, d.C, d.H * d.W, cpad, pack, s, true);
    };
    if (precision == KXC_B200_PREC_TF32X3) {
        // x*w ~ x_hi*w_hi + x_hi*w_lo + x_lo*w_hi, summed in one launch (conv_tc.cu)
        const int cpad = tc_channel_pad(kTcTF32, d.C);
        const size_t act = (size_t)d.N * d.H * d.W * cpad;
        const size_t w_bytes = align_up((size_t)d.O * d.KH * d.KW * cpad * 4, 1024);
        StreamScratch ws(s);
        KXC_TRY(ws.alloc(align_up(2 * act * 4, 1024) + 2 * w_bytes));
        float* act_hi = static_cast<float*>(ws.ptr);
        uint8_t* w_hi = static_cast<uint8_t*>(ws.ptr) + align_up(2 * act * 4, 1024);
        uint8_t* w_lo = w_hi + w_bytes;
        const WeightPack pack{weight, w_hi, w_lo, d.O, d.C, d.KH * d.KW, cpad};
        KXC_TRY(convert(act_hi, act_hi + act, kTcTF32, cpad, &pack));
        TcParams p{};
        TcConfig cfg{};
        KXC_TRY(tc_setup_conv_x3(&p, &cfg, kOutNCHW_F32, act_hi, w_hi, w_lo, d.N, d.H, d.W, cpad, d.O, d.KH, d.KW, d.SH, d.PH, d.PW, d.DH,
                                 d.DW));
        p.bias = bias;
        p.residual = residual;
        p.out = out;
        p.relu = relu;
        tc_finish_params(&p);
        return tc_launch(cfg, p, s);
    }
    const TcDType dt = precision == KXC_B200_PREC_BF16 ? kTcBF16 : kTcTF32;
    const int eb = tc_elem_bytes(dt);
    const CmPlan* cm = cm_wanted(dt, d, 0);
    const int cpad = cm != nullptr ? cm_channel_pad(dt, d.C) : tc_channel_pad(dt, d.C);
    const int w_cpad = cm != nullptr ? cm_weight_pad(dt, d.C, *cm) : cpad;
    const size_t act_bytes = align_up((size_t)d.N * d.H * d.W * cpad * eb, 1024);
    const size_t w_bytes = align_up((size_t)d.O * d.KH * d.KW * w_cpad * eb, 1024);
    StreamScratch ws(s);
    KXC_TRY(ws.alloc(act_bytes + w_bytes));
    uint8_t* act = static_cast<uint8_t*>(ws.ptr);
    uint8_t* wp = act + act_bytes;
    const WeightPack pack{weight, wp, nullptr, d.O, d.C, d.KH * d.KW, w_cpad};
    KXC_TRY(convert(act, nullptr, dt, cpad, &pack));
    if (cm != nullptr) {
        CmParams p{};
        KXC_TRY(cm_setup(&p, dt, *cm, act, wp, cpad, w_cpad));
        p.bias = bias;
        p.residual = residual;
        p.out = out;
        p.relu = relu;
        return cm_launch(dt, p, s);
    }
    TcParams p{};
    TcConfig cfg{};
    KXC_TRY(tc_setup_conv(&p, &cfg, dt, kOutNCHW_F32, act, wp, d.N, d.H, d.W, cpad, d.O, d.KH, d.KW, d.SH, d.PH, d.PW, d.DH,
                          d.DW));
    p.bias = bias;
    p.residual = residual;
    p.out = out;
    p.relu = relu;
    tc_finish_params(&p);
    return tc_launch(cfg, p, s);
}

int32_t conv2d_s8_dispatch(const int8_t* data, const int8_t* weight, const int32_t* bias, const int32_t* multiplier,
                           const int32_t* shift, int8_t* out, const ConvDims& d, int relu, int force_simt, int nhwc,
                           cudaStream_t s) {
    const TcDType dt = kTcS8;
    const int cpad = tc_channel_pad(dt, d.C);
    // few-channel stride-2 first layer (the 7x7 stem): pixels packed to 8 bytes, direct kernel, K = 7 x 64 bytes instead of
    // 49 taps x 32 padded channels. Both layouts of the entry point take it (NHWC: data [N,H,W,C], weight [O,KH,KW,C]).
    const int stem_hp = (d.H + 2 * d.PH + 1) & ~1;
    const int stem_wp = ((d.W + 2 * d.PW > 2 * (d.OW - 1) + 8 ? d.W + 2 * d.PW : 2 * (d.OW - 1) + 8) + 3) / 4 * 4;
    const bool stem_ok = !force_simt && tc_shape_ok(d) && d.SH == 2 && d.SW == 2 && d.DH == 1 && d.DW == 1 &&
                         stem_direct_s8_applicable(d.C, d.O, d.KH, d.KW, 2, 1, d.W, d.OW, stem_wp);
    auto run_stem = [&](bool nhwc_layout) -> int32_t {
        const size_t x_bytes = align_up((size_t)d.N * stem_hp * stem_wp * 8, 1024);
        const size_t w_bytes = align_up(stem_direct_weight_bytes(d.KH), 1024);
        StreamScratch ws(s);
        KXC_TRY(ws.alloc(x_bytes + w_bytes));
        uint8_t* px = static_cast<uint8_t*>(ws.ptr);
        uint8_t* pw = px + x_bytes;
        KXC_TRY(stem_direct_s8_pack(data, weight, px, pw, d.N, d.C, d.H, d.W, d.O, d.KH, d.KW, stem_hp, stem_wp, d.PH, d.PW, nhwc_layout, s));
        TcParams p{};
        KXC_TRY(stem_direct_setup(&p, px, pw, d.N, d.OH, d.OW, d.KH, stem_hp, stem_wp));
        p.bias_i32 = bias;
        p.multiplier = multiplier;
        p.shift = shift;
        p.out = out;
        p.relu = relu;
        tc_finish_params(&p);
        return stem_direct_s8_launch(p, nhwc_layout, s);
    };
    if (nhwc) {
        // operands already NHWC / OHWI with the kernel's channel granularity: straight to the tensor-core kernel
        if (force_simt || !tc_shape_ok(d)) return fail(KXC_B200_ERR_UNSUPPORTED, "nn_conv2d_s8: the NHWC form exists for the tensor-core path only");
        if (stem_ok && d.C <= 8 && aligned16(out)) return run_stem(true);
        if (cpad != d.C || (d.O & 15) != 0 || !aligned16(data) || !aligned16(weight) || !aligned16(out))
            return fail(KXC_B200_ERR_INVALID, "nn_conv2d_s8: NHWC operands need C = 32/64/128k channels, O a multiple of 16 and 16-byte aligned pointers");
        TcParams p{};
        // 64 -> 64 channels, 3x3, stride 1: the row-stacked kernel (one box load per tile instead of nine)
        static const bool rowstack_enabled = [] {
            const char* e = getenv("KXC_B200_ROWSTACK_S8");
            return !(e != nullptr && e[0] == '0');
        }();
        if (rowstack_enabled && rowstack3x3_s8_applicable(d.C, d.O, d.KH, d.KW, d.SH, d.PH, d.PW, d.DH, d.DW)) {
            KXC_TRY(rowstack3x3_s8_setup(&p, data, weight, d.N, d.H, d.W));
            p.bias_i32 = bias;
            p.multiplier = multiplier;
            p.shift = shift;
            p.out = out;
            p.relu = relu;
            tc_finish_params(&p);
            return rowstack3x3_s8_launch(p, s);
        }
        TcConfig cfg{};
        KXC_TRY(tc_setup_conv(&p, &cfg, dt, kOutNHWC_S8, data, weight, d.N, d.H, d.W, cpad, d.O, d.KH, d.KW, d.SH, d.PH, d.PW, d.DH,
                              d.DW));
        p.bias_i32 = bias;
        p.multiplier = multiplier;
        p.shift = shift;
        p.out = out;
        p.relu = relu;
        tc_finish_params(&p);
        return tc_launch(cfg, p, s);
    }
    if (force_simt || !tc_shape_ok(d)) return conv2d_s8_exact(data, weight, bias, multiplier, shift, out, d, relu, s);
    if (stem_ok) return run_stem(false);
    // (a quarter of the conversion and of the kernel's loads for the downsample branches of a ResNet)
    const bool subsample = subsampled(d);
    const ConvDims dc = subsample ? without_stride(d) : d;  // what the kernel convolves
    auto convert = [&](uint8_t* act, int pad, const WeightPack* pack) {
        return subsample ? convert_operands_s8_subsample(data, reinterpret_cast<int8_t*>(act), d.N, d.C, d.H, d.W, d.OH, d.OW, d.SH, pad, pack, s, true)
                         : convert_operands(data, act, nullptr, dt, d.N, d.C, d.H * d.W, pad, pack, s, true);
    };
    if (const CmPlan* cm = cm_wanted(dt, dc, 0)) {
        const int cm_pad = cm_channel_pad(dt, d.C), w_cpad = cm_weight_pad(dt, d.C, *cm);
        const size_t cm_act = align_up((size_t)d.N * dc.H * dc.W * cm_pad, 1024);
        StreamScratch ws(s);
        KXC_TRY(ws.alloc(cm_act + align_up((size_t)d.O * d.KH * d.KW * w_cpad, 1024)));
        uint8_t* act = static_cast<uint8_t*>(ws.ptr);
        uint8_t* wp = act + cm_act;
        const WeightPack pack{weight, wp, nullptr, d.O, d.C, d.KH * d.KW, w_cpad};
        KXC_TRY(convert(act, cm_pad, &pack));
        CmParams p{};
        KXC_TRY(cm_setup(&p, dt, *cm, act, wp, cm_pad, w_cpad));
        p.bias_i32 = bias;
        p.multiplier = multiplier;
        p.shift = shift;
        p.out = out;
        p.relu = relu;
        return cm_launch(dt, p, s);
    }
    // What is left: filters of more taps than the channel-major kernel lists or too far apart for its boxes, results of 2^32 elements and more.
    const size_t act_bytes = align_up((size_t)d.N * dc.H * dc.W * cpad, 1024);
    const size_t w_bytes = align_up((size_t)d.O * d.KH * d.KW * cpad, 1024);
    // Result layout. A thread of the epilogue owns one pixel, so its NCHW stores are single bytes whose neighbours in
    // memory belong to the next pixel of the same tile row: runs of BW bytes. The other way is to store NHWC into the
    // workspace, pixels padded to 16 channels, and to let a byte transpose write the reference layout, which costs a launch
    // (1 to 3 us) and the result's bytes twice more. Measured on 60 filters of 81 and 121 taps, us a call with byte stores / by way of NHWC:
    //   narrow boxes (BW <= 2)         24 -> 401 at 13x13, 66 images: 80.3 / 71.5; 17 -> 33 at 5x5, 128 images: 36.3 / 34.3; 20 -> 100 at 7x7, 64
    //                                  images (two pixels to an image's box, odd channels) 34.5 / 35.1
    //   results of 1 MiB and more      3 -> 210 at 20x17, 88 images: 110.3 / 97.1, others between 0.95 and 1.03 times; planes no multiple of four
    //                                  (byte-wise transpose): 3 -> 223 at 39x42, 112 images 303 / 340
    //   smaller ones                   32.9 / 33.7 to 47.2 / 49.4
    int bw = 0, bh = 0, bni = 0;
    tc_pick_tile(d.N, d.OH, d.OW, &bw, &bh, &bni);
    const int out_pitch = (d.O + 15) / 16 * 16;
    const long long plane = (long long)d.OH * d.OW;
    const bool narrow = bw <= 2;
    bool two_step = (narrow && ((d.O & 15) == 0 || bw * bh == 1)) || (plane * d.N * d.O >= (1 << 20) && ((plane & 3) == 0 || narrow));
    const size_t out_bytes = two_step ? align_up((size_t)d.N * d.OH * d.OW * out_pitch, 1024) : 0;
    StreamScratch ws(s);
    int32_t rc = ws.alloc(act_bytes + w_bytes + out_bytes);
    if (rc != KXC_B200_OK && two_step) {  // no room for the second copy of the result: byte stores
        two_step = false;
        rc = ws.alloc(act_bytes + w_bytes);
    }
    KXC_TRY(rc);
    uint8_t* act = static_cast<uint8_t*>(ws.ptr);
    uint8_t* wp = act + act_bytes;
    int8_t* out_nhwc = reinterpret_cast<int8_t*>(wp + w_bytes);
    const WeightPack pack{weight, wp, nullptr, d.O, d.C, d.KH * d.KW, cpad};
    KXC_TRY(convert(act, cpad, &pack));
    TcParams p{};
    TcConfig cfg{};
    KXC_TRY(tc_setup_conv(&p, &cfg, dt, two_step ? kOutNHWC_S8 : kOutNCHW_S8, act, wp, d.N, dc.H, dc.W, cpad, d.O, d.KH, d.KW, dc.SH, d.PH, d.PW, d.DH,
                          d.DW));
    p.bias_i32 = bias;
    p.multiplier = multiplier;
    p.shift = shift;
    p.out = two_step ? out_nhwc : out;
    p.out_pitch = two_step ? out_pitch : 0;
    p.relu = relu;
    tc_finish_params(&p);
    KXC_TRY(tc_launch(cfg, p, s));
    if (two_step) return nhwc_to_nchw_s8(out_nhwc, out, d.N, d.O, out_pitch, d.OH * d.OW, s);
    return KXC_B200_OK;
}

int32_t gemm_tensor_core(const float* a, const float* b, const float* c, float* out, const kxc_b200_gemm_desc& g,
                         cudaStream_t s) {
    // alpha/beta scaling is a separately rounded multiply in the reference; only the common
    // alpha = beta = 1 form is fused into the tensor-core epilogue.
    if ((g.has_c && ((double)g.alpha != 1.0 || (double)g.beta != 1.0)) || g.m > 65535 * 128)
        return gemm_fp32_exact(a, b, c, out, g, s);
    if (gemm_small_applicable(a, b, out, g)) return gemm_small(a, b, g.has_c ? c : nullptr, out, g, s);
    if (g.precision == KXC_B200_PREC_TF32X3) {
        const int kpad = tc_channel_pad(kTcTF32, g.k);
        const size_t a_elems = (size_t)g.m * kpad;  // the low part of A follows its high part at once (tc_setup_conv_x3)
        const size_t b_bytes = align_up((size_t)g.n * kpad * 4, 1024);
        StreamScratch ws(s);
        KXC_TRY(ws.alloc(align_up(2 * a_elems * 4, 1024) + 2 * b_bytes));
        float* a_hi = static_cast<float*>(ws.ptr);
        float* b_hi = reinterpret_cast<float*>(static_cast<uint8_t*>(ws.ptr) + align_up(2 * a_elems * 4, 1024));
        float* b_lo = b_hi + b_bytes / 4;
        KXC_TRY(split_rows(a, a_hi, a_hi + a_elems, g.m, g.k, kpad, s));
        if (g.transB)
            KXC_TRY(split_rows(b, b_hi, b_lo, g.n, g.k, kpad, s));
        else
            KXC_TRY(convert_operands(b, b_hi, b_lo, kTcTF32, 1, g.k, g.n, kpad, nullptr, s, false));
        TcParams p{};
        TcConfig cfg{};
        KXC_TRY(tc_setup_conv_x3(&p, &cfg, kOutNHWC_F32, a_hi, b_hi, b_lo, g.m, 1, 1, kpad, g.n, 1, 1, 1, 0, 0, 1, 1));
        p.bias = g.has_c ? c : nullptr;
        p.out = out;
        tc_finish_params(&p);
        return tc_launch(cfg, p, s);
    }
    const TcDType dt = g.precision == KXC_B200_PREC_BF16 ? kTcBF16 : kTcTF32;
    const int eb = tc_elem_bytes(dt);
    const int kpad = tc_channel_pad(dt, g.k);
    const size_t a_bytes = align_up((size_t)g.m * kpad * eb, 1024);
    const size_t b_bytes = align_up((size_t)g.n * kpad * eb, 1024);
    StreamScratch ws(s);
    KXC_TRY(ws.alloc(a_bytes + b_bytes));
    uint8_t* ap = static_cast<uint8_t*>(ws.ptr);
    uint8_t* bp = ap + a_bytes;
    if (g.transB) {
        KXC_TRY(convert_rows_two(a, ap, g.m, b, bp, g.n, dt, g.k, kpad, s));  // b is [N, K]
    } else {
        KXC_TRY(convert_rows(a, ap, dt, g.m, g.k, kpad, s));
        KXC_TRY(convert_operands(b, bp, nullptr, dt, 1, g.k, g.n, kpad, nullptr, s, true));  // b is [K, N] -> [N, Kpad]
    }
    TcParams p{};
    TcConfig cfg{};
    // A dense layer is a 1x1 convolution over an M x 1 x 1 "image" batch.
    KXC_TRY(tc_setup_conv(&p, &cfg, dt, kOutNHWC_F32, ap, bp, g.m, 1, 1, kpad, g.n, 1, 1, 1, 0, 0, 1, 1));
    p.bias = g.has_c ? c : nullptr;
    p.out = out;
    p.relu = 0;
    tc_finish_params(&p);
    return tc_launch(cfg, p, s);
}

}  // namespace kxc_b200

using namespace kxc_b200;

// Reads (and clears) the device status words written by a tensor-core kernel whose bounded wait ran
// out: the regular one and the one of the static-scratch entry point. Synchronises the stream.
// 0 = every kernel so far completed its protocol. Allocates nothing once the regular word exists.
extern "C" int32_t kxc_b200_device_status(void* stream, int32_t* status_out) {
    KXC_TRY(require_device());
    int* words[2] = {nullptr, nullptr};
    KXC_TRY(tc_status_word(&words[0]));
    KXC_TRY(static_scratch_status_word(&words[1]));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int host[2] = {0, 0};
    for (int i = 0; i < 2; ++i)
        if (words[i]) KXC_CUDA_TRY(cudaMemcpyAsync(&host[i], words[i], sizeof(int), cudaMemcpyDeviceToHost, s));
    KXC_CUDA_TRY(cudaStreamSynchronize(s));
    for (int i = 0; i < 2; ++i)
        if (host[i] != 0) KXC_CUDA_TRY(cudaMemsetAsync(words[i], 0, sizeof(int), s));
    const int combined = host[0] | host[1];
    if (status_out) *status_out = combined;
    if (combined != 0)
        return fail(KXC_B200_ERR_DEVICE_WAIT, "a tensor-core kernel gave up a bounded wait (status %d%s)", combined,
                    host[1] != 0 ? ", static-scratch entry point" : "");
    return KXC_B200_OK;
}

// ---- self tests -----------------------------------------------------------------------------------------
namespace kxc_b200 {
namespace {
// One CTA waits, through the same bounded wait every tensor-core kernel uses, on an mbarrier that nothing ever
// arrives on. After `limit_ns` the wait gives up, the kernel reports into the status word and returns normally.
__global__ void bounded_wait_selftest_kernel(uint64_t limit_ns, int* status, int* gave_up) {
    __shared__ __align__(8) uint64_t bar;
    __shared__ int abort_flag;
    if (threadIdx.x == 0) {
        abort_flag = 0;
        sm100::mbar_init(sm100::smem_u32(&bar), 1);
        sm100::mbar_fence_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const bool arrived = sm100::mbar_wait_bounded(sm100::smem_u32(&bar), 0, &abort_flag, limit_ns);
        *gave_up = arrived ? 0 : 1;
        if (!arrived) atomicExch(status, KXC_B200_ERR_DEVICE_WAIT);
    }
}
}  // namespace
}  // namespace kxc_b200

extern "C" int32_t kxc_b200_selftest_bounded_wait(int64_t limit_ns, void* stream, int32_t* gave_up_out) {
    KXC_TRY(require_device());
    if (limit_ns <= 0 || limit_ns > 100000000ll) return fail(KXC_B200_ERR_INVALID, "selftest_bounded_wait: limit must be in (0, 100 ms]");
    int* word = nullptr;
    KXC_TRY(tc_status_word(&word));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int* flag = nullptr;
    KXC_CUDA_TRY(cudaMallocAsync(&flag, sizeof(int), s));
    KXC_CUDA_TRY(cudaMemsetAsync(flag, 0, sizeof(int), s));
    bounded_wait_selftest_kernel<<<1, 32, 0, s>>>((uint64_t)limit_ns, word, flag);
    const int32_t rc = check_launch("bounded_wait_selftest_kernel");
    int host = 0;
    cudaError_t e = cudaMemcpyAsync(&host, flag, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaFreeAsync(flag, s);
    if (rc != KXC_B200_OK) return rc;
    if (e != cudaSuccess) return fail(KXC_B200_ERR_CUDA, "selftest_bounded_wait: %s", cudaGetErrorString(e));
    if (gave_up_out) *gave_up_out = host;
    return KXC_B200_OK;
}
