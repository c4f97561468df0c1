// Launchers of the denoiser's tensor-core convolutions (gs_conv.cu).
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace gs {
namespace conv {

// One 3x3 "same" convolution, NHWC bf16 in, per output pixel
//   out[c] = epilogue(sum over taps and input channels + bias[c]).
struct ConvArgs {
    const __nv_bfloat16* x;     // input (Cin channels), or the full-resolution term of load mode 1
    const __nv_bfloat16* xh;    // load mode 1: half-resolution term, upsampled 2x (nearest) and added to x
    int n, h, w;                // batch and spatial size (input = output; h, w even in load mode 1)
    const uint8_t* wimage;      // packed weights (launch_pack_weights)
    const float* bias;          // Cout floats or null
    int relu;                   // max(., 0) after the bias
    const __nv_bfloat16* mask;  // Cout-channel tensor: outputs where mask <= 0 become 0 (ReLU backward); or null
    __nv_bfloat16* out_bf16;    // Cout channels, or null
    float* out_f32;             // Cout channels, or null
    int unit_rows;              // rows that stay in one CTA: 1, 2 (pool_out) or 16 (head_x)
    uint32_t* err;              // bit 0 set if a bounded wait ran out
    int row_offset;             // the units' row bands start at -row_offset (0: at row 0)
    int max_sms;                // SMs of the device
    int out_wide;               // out_bf16 is 32-byte aligned (set by launch_fwd)
    // (Cin = 16, Cout = 32, forward): also the 2x2 average of the bf16 output, n x h/2 x w/2 (h, w
    // even, unit_rows 2), summed from zero in row order and rounded once
    __nv_bfloat16* pool_out;
    // Denoised-mode head (Cout = 16, forward, head_x set): the epilogue writes head_out16 =
    // RGBA16F (head_x[5..7] + o[0..2], head_x[3] + o[3]) instead of the outputs above and,
    // per 16x16 tile of GL rows (unit_rows = 16 and row_offset aligning the bands with
    // them), tile_err = mean(max(o[4], 0)) * 0.001, counting tiles at or above err_budget.
    const __nv_bfloat16* head_x;   // the network input (16 channels per pixel)
    uint16_t* head_out16;
    float* tile_err;
    uint32_t* fallback_count;
    float err_budget;
    int tiles_x;
};

// dw[tap * Cin + cin][cout] += sum over pixels of X[p + tap][cin] * dy[p][cout],
// db[cout] += sum over pixels of dy[p][cout].
struct WgradArgs {
    const __nv_bfloat16* x;     // layer input (as ConvArgs::x)
    const __nv_bfloat16* xh;    // load mode 1 (as ConvArgs::xh)
    int n, h, w;
    const __nv_bfloat16* dy;    // gradient of the layer output (Cout channels)
    float* dw;                  // 9 * Cin * Cout floats, accumulated
    float* db;                  // Cout floats, accumulated, or null
    uint32_t* err;
};

// Supported (cin, cout, load mode): (16, 32, 0), (32, 32, 0), (32, 16, 0), (32, 32, 1).
// Return the number of kernels launched, or -1 for an unsupported shape.
int launch_fwd(int cin, int cout, int load_mode, const ConvArgs& a, cudaStream_t s);
// max_ctas: the SMs of the device (one persistent CTA each)
int launch_wgrad(int cin, int cout, int load_mode, const WgradArgs& a, int max_ctas, cudaStream_t s);
// transposed: the image of the layer's input gradient
int launch_pack_weights(const float* w, int cin, int cout, int transposed, uint8_t* image, cudaStream_t s);
// Byte offset of weight (tap = 3 ky + kx, ci, co) in the K-major B image: K = 3 kx x cin, N = 3 x cout with the
// columns of ky = 2, 1, 0 side by side.
__host__ __device__ constexpr int wimage_offset(int tap, int ci, int co, int cin, int cout) {
    const int k = (tap % 3) * cin + ci, n = (2 - tap / 3) * cout + co;
    return (k >> 3) * (3 * cout * 16) + (n >> 3) * 128 + (n & 7) * 16 + (k & 7) * 2;
}
size_t weight_image_bytes(int cin, int cout);

}  // namespace conv
}  // namespace gs
