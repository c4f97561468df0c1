// Denoiser kernels other than the convolutions (gs_denoise.cu).
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

namespace gs {
namespace dn {

constexpr int kInC = 16;    // input features (8 used)
constexpr int kHidC = 32;   // hidden channels
constexpr int kOutC = 16;   // output channels (5 used)

void set_gauss_window(cudaStream_t s);
int launch_upsample_grad(const __nv_bfloat16* du, const __nv_bfloat16* e3, int n, int h, int w, __nv_bfloat16* dz3,
                         cudaStream_t s);
int launch_skip_pool_grad(const __nv_bfloat16* du, const __nv_bfloat16* dp1, const __nv_bfloat16* e1, int n, int h,
                          int w, __nv_bfloat16* dz1, cudaStream_t s);
// o: 16 channels f32, x: the input features; part: 9 planes of n * h * w floats (or null: no SSIM term)
int launch_ssim_partials(const float* o, const __nv_bfloat16* x, const float4* target, int n, int h, int w, float* part,
                         float* acc, cudaStream_t s);
int launch_loss_grad(const float* o, const __nv_bfloat16* x, const float4* target, const float* part, int n, int h,
                     int w, float inv_l1, float ssim_scale, float err_scale, __nv_bfloat16* dout, float* acc,
                     cudaStream_t s);
// Where each layer's weights lie in the parameter vector and the bf16 operand
// images they are packed into (conv::wimage_offset); cut_cout >= 0: the output
// channel left out of the transposed image.
struct ParamImages {
    struct Layer {
        int first, cin, cout, cut_cout;
        uint8_t* image;
        uint8_t* image_t;
    };
    Layer layer[8];
    int layers;
};
int launch_adam(const ParamImages& im, float* w, const float* g, float* m, float* v, int count, float lr, float b1,
                float b2, float eps, float bc1, float bc2, cudaStream_t s);
int launch_pack_params(const ParamImages& im, float* w, int count, cudaStream_t s);

}  // namespace dn
}  // namespace gs
