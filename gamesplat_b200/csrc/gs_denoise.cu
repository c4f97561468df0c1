// Elementwise and reduction kernels of the stochastic-splat denoiser: the
// backward passes of pooling and upsampling (the input features are written by
// the TAA pass, the 2x average pooling by conv1's epilogue), the output head
// of training, the L1 + SSIM training loss with
// its gradient and Adam.  The convolutions are in gs_conv.cu; in the denoised
// render mode the last convolution's epilogue writes the frame and the
// per-tile error estimate that picks the tiles the sorted-alpha rasterizer
// renders again (conv::ConvArgs::head_x).
//
// Network (NHWC bf16 activations, FP32 accumulation):
//   x   16 ch  = noisy RGB, alpha, expected depth, reprojected history RGB, 8 zero channels
//   e1  = relu(conv1(x))            32 ch, full resolution
//   p1  = avgpool2(e1)              32 ch, half
//   e2  = relu(conv2(p1))           32 ch, half
//   e3  = relu(conv3(e2))           32 ch, half
//   d4  = relu(conv4(up2(e3) + e1)) 32 ch, full (U-Net skip)
//   o   = conv5(d4)                 16 ch (f32): 0..3 RGBA residual, 4 error estimate
//   RGBA = (history RGB, alpha) + o[0..3];  error = o[4] (1000 x squared error)
#include <cuda_bf16.h>

#include "gs_conv.h"
#include "gs_denoise.h"

namespace gs {
namespace dn {

__device__ __forceinline__ float bf(const __nv_bfloat16& v) { return __bfloat162float(v); }

// 8 channels (16 bytes) as floats and back.
__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
    const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 t = __bfloat1622float2(p[i]);
        f[2 * i] = t.x;
        f[2 * i + 1] = t.y;
    }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
    uint4 v;
    __nv_bfloat162* p = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
    for (int i = 0; i < 4; ++i) p[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
    return v;
}

constexpr int kHidQ = kHidC / 8;   // 16-byte granules of a hidden pixel

// Backward of the decoder input u = up2(e3) + e1 for its e3 term, with the
// ReLU of e3: dz3[q] = (e3[q] > 0) * sum of du over the 2x2 block of q.  A
// thread takes 8 channels of a pixel (16-byte loads): bound by the bytes of du
// (8 crops of 256x256: 25 us when a thread took one 2-byte channel, 6.4 us now).
__global__ void upsample_grad_kernel(const uint4* __restrict__ du, const uint4* __restrict__ e3, int n, int h, int w,
                                     uint4* __restrict__ dz3) {
    const int hh = h / 2, hw = w / 2;
    const size_t total = (size_t)n * hh * hw * kHidQ;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int c = (int)(i % kHidQ);
        const size_t op = i / kHidQ;
        const int ox = (int)(op % hw);
        const size_t row = op / hw;   // b * hh + oy: the source rows are 2 * row and 2 * row + 1 (h even)
        float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, e[8];
#pragma unroll
        for (int dy = 0; dy < 2; ++dy)
#pragma unroll
            for (int dx = 0; dx < 2; ++dx) {
                float v[8];
                unpack8(__ldg(du + ((2 * row + dy) * w + 2 * ox + dx) * kHidQ + c), v);
#pragma unroll
                for (int k = 0; k < 8; ++k) s[k] += v[k];
            }
        unpack8(__ldg(e3 + i), e);
#pragma unroll
        for (int k = 0; k < 8; ++k) s[k] = e[k] > 0.0f ? s[k] : 0.0f;
        dz3[i] = pack8(s);
    }
}

// Gradient of e1 (skip term du plus the pooling term dp1 / 4) through the
// ReLU of e1: dz1 = (e1 > 0) * (du + dp1[p / 2] / 4).  8 channels a thread, as
// above (85 us with one, 17 us now).
__global__ void skip_pool_grad_kernel(const uint4* __restrict__ du, const uint4* __restrict__ dp1,
                                      const uint4* __restrict__ e1, int n, int h, int w, uint4* __restrict__ dz1) {
    const int hw = w / 2;
    const size_t total = (size_t)n * h * w * kHidQ;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int c = (int)(i % kHidQ);
        const size_t p = i / kHidQ;
        const int x = (int)(p % w);
        const size_t row = p / w;   // b * h + y, h even
        float d[8], q[8], e[8];
        unpack8(__ldg(du + i), d);
        unpack8(__ldg(dp1 + ((row >> 1) * hw + (x >> 1)) * kHidQ + c), q);
        unpack8(__ldg(e1 + i), e);
#pragma unroll
        for (int k = 0; k < 8; ++k) d[k] = e[k] > 0.0f ? d[k] + 0.25f * q[k] : 0.0f;
        dz1[i] = pack8(d);
    }
}

// ---------------------------------------------------------------------------
// Output head and the training loss.
// ---------------------------------------------------------------------------
// pred of pixel i: (history RGB, alpha) + o[0..3].  wide: o and x are 16-byte
// aligned (the denoiser's own buffers are; a caller's need not be).
__device__ __forceinline__ float4 head_rgba(const float* __restrict__ o, const __nv_bfloat16* __restrict__ x, size_t i,
                                            bool wide) {
    const float* oi = o + i * kOutC;
    const __nv_bfloat16* xi = x + i * kInC;
    if (wide) {
        const float4 r = __ldg(reinterpret_cast<const float4*>(oi));
        float f[8];
        unpack8(__ldg(reinterpret_cast<const uint4*>(xi)), f);
        return make_float4(f[5] + r.x, f[6] + r.y, f[7] + r.z, f[3] + r.w);
    }
    return make_float4(bf(xi[5]) + oi[0], bf(xi[6]) + oi[1], bf(xi[7]) + oi[2], bf(xi[3]) + oi[3]);
}

// The SSIM window: a separable Gaussian (11 taps, sigma 1.5, zero outside the
// image), along x and then along y.
__constant__ float c_gauss[11];

// The loss kernels work on tiles of 32 x 16 pixels with a 5-pixel halo in
// shared memory, so that the moment maps (15 of them) and the blurred partials
// (9) never go through memory: as whole-image passes they were four blurs over
// 24 float maps, 447 us of a training step on 8 crops of 256x256, and now the
// two kernels' reads are the images and 9 floats a pixel between them.
constexpr int kLossTx = 32, kLossTy = 16, kLossThreads = 128;
constexpr int kLossRows = kLossTy + 10, kLossCols = kLossTx + 10;
constexpr int kLossStride = kLossCols + 1;   // 43 = 11 mod 32: the x pass reads (8 rows x 4 segments a warp) from 32 banks
constexpr int kLossHStride = kLossTx + 1;

struct LossTile {
    int b, x0, y0;
};
__device__ __forceinline__ LossTile loss_tile(int h, int w) {
    const int tx = (w + kLossTx - 1) / kLossTx, ty = (h + kLossTy - 1) / kLossTy;
    const int t = (int)blockIdx.x;
    return {t / (tx * ty), (t % tx) * kLossTx, (t / tx) % ty * kLossTy};
}

// Blur along x of 18 staged values into 8 outputs, taps in order.
__device__ __forceinline__ void blur8(const float (&v)[18], float* dst) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        float s = 0.0f;
#pragma unroll
        for (int k = 0; k < 11; ++k) s = fmaf(c_gauss[k], v[i + k], s);
        dst[i] = s;
    }
}
// Blur along y of column `col`, rows r0 .. r0 + 3 of the tile.
__device__ __forceinline__ void blur4(const float (*hb)[kLossHStride], int col, int r0, float (&out)[4]) {
    float v[14];
#pragma unroll
    for (int i = 0; i < 14; ++i) v[i] = hb[r0 + i][col];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float s = 0.0f;
#pragma unroll
        for (int k = 0; k < 11; ++k) s = fmaf(c_gauss[k], v[i + k], s);
        out[i] = s;
    }
}

// Sum of a and b over the CTA into acc[0] and acc[1].
__device__ __forceinline__ void block_sum2(float a, float b, float* acc) {
    __shared__ float s_sum[2][kLossThreads / 32];
    for (int off = 16; off; off >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, off);
        b += __shfl_xor_sync(0xffffffffu, b, off);
    }
    if ((threadIdx.x & 31) == 0) {
        s_sum[0][threadIdx.x >> 5] = a;
        s_sum[1][threadIdx.x >> 5] = b;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        float t = 0.0f;
        for (int k = 0; k < kLossThreads / 32; ++k) t += s_sum[threadIdx.x][k];
        atomicAdd(acc + threadIdx.x, t);
    }
}

constexpr float kC1 = 0.0001f, kC2 = 0.0009f;   // (0.01)^2, (0.03)^2 for a data range of 1

// Per RGB channel the moments (pred, target, pred^2, target^2, pred target),
// blurred; then SSIM per interior pixel (pixels closer than 5 to the border
// are left out) and its partial derivatives with respect to mu_x, E[x^2] and
// E[xy], to part[(3 c + q) npix + pixel]; the SSIM sum and count go to
// acc[0], acc[1].  8 crops of 256x256: 40 us, with loss_grad_kernel 66 us; 447 us of
// blurs through 24 maps in memory, 59 and 67 us for the rest before tiles.
__global__ void __launch_bounds__(kLossThreads) ssim_partials_kernel(const float* __restrict__ o,
                                                                     const __nv_bfloat16* __restrict__ x,
                                                                     const float4* __restrict__ target, int n, int h,
                                                                     int w, bool wide, float* __restrict__ part,
                                                                     float* __restrict__ acc) {
    __shared__ float s_p[3][kLossRows][kLossStride], s_t[3][kLossRows][kLossStride];
    __shared__ float s_h[5][kLossRows][kLossHStride];
    const LossTile tile = loss_tile(h, w);
    const int t = threadIdx.x;
    const size_t image = (size_t)tile.b * h * w, npix = (size_t)n * h * w;
    for (int i = t; i < kLossRows * kLossCols; i += kLossThreads) {
        const int r = i / kLossCols, c = i % kLossCols, yy = tile.y0 - 5 + r, xx = tile.x0 - 5 + c;
        float4 p = make_float4(0.f, 0.f, 0.f, 0.f), q = p;
        if (xx >= 0 && xx < w && yy >= 0 && yy < h) {
            const size_t at = image + (size_t)yy * w + xx;
            p = head_rgba(o, x, at, wide);
            q = __ldg(target + at);
        }
        s_p[0][r][c] = p.x;
        s_p[1][r][c] = p.y;
        s_p[2][r][c] = p.z;
        s_t[0][r][c] = q.x;
        s_t[1][r][c] = q.y;
        s_t[2][r][c] = q.z;
    }
    __syncthreads();
    const int hr = t >> 2, seg = (t & 3) * 8, col = t & 31, r0 = (t >> 5) * 4;
    float local = 0.0f, cnt = 0.0f;
    for (int c = 0; c < 3; ++c) {
        if (hr < kLossRows) {
            float p[18], q[18], v[18];
#pragma unroll
            for (int i = 0; i < 18; ++i) {
                p[i] = s_p[c][hr][seg + i];
                q[i] = s_t[c][hr][seg + i];
            }
            blur8(p, &s_h[0][hr][seg]);
            blur8(q, &s_h[1][hr][seg]);
#pragma unroll
            for (int i = 0; i < 18; ++i) v[i] = __fmul_rn(p[i], p[i]);
            blur8(v, &s_h[2][hr][seg]);
#pragma unroll
            for (int i = 0; i < 18; ++i) v[i] = __fmul_rn(q[i], q[i]);
            blur8(v, &s_h[3][hr][seg]);
#pragma unroll
            for (int i = 0; i < 18; ++i) v[i] = __fmul_rn(p[i], q[i]);
            blur8(v, &s_h[4][hr][seg]);
        }
        __syncthreads();
        float m[5][4];
#pragma unroll
        for (int k = 0; k < 5; ++k) blur4(s_h[k], col, r0, m[k]);
        __syncthreads();
        const int xx = tile.x0 + col;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int yy = tile.y0 + r0 + i;
            if (xx >= w || yy >= h) continue;
            const bool inside = xx >= 5 && xx < w - 5 && yy >= 5 && yy < h - 5;
            const float mx = m[0][i], my = m[1][i];
            const float sxx = m[2][i] - mx * mx, syy = m[3][i] - my * my, sxy = m[4][i] - mx * my;
            const float A1 = 2.0f * mx * my + kC1, A2 = 2.0f * sxy + kC2;
            const float B1 = mx * mx + my * my + kC1, B2 = sxx + syy + kC2;
            const float S = (A1 * A2) / (B1 * B2);
            float dmx = 0.0f, dxx = 0.0f, dxy = 0.0f;
            if (inside) {
                local += S;
                cnt += 1.0f;
                const float dS_dA1 = A2 / (B1 * B2), dS_dA2 = A1 / (B1 * B2);
                const float dS_dB1 = -S / B1, dS_dB2 = -S / B2;
                // A1(mx), A2(sxy(mx)), B1(mx), B2(sxx(mx)); sxx = E[x^2] - mx^2, sxy = E[xy] - mx my
                dxx = dS_dB2;                                   // dB2 / dE[x^2] = 1
                dxy = 2.0f * dS_dA2;                            // dA2 / dE[xy] = 2
                dmx = dS_dA1 * 2.0f * my + dS_dA2 * (-2.0f * my) + dS_dB1 * 2.0f * mx + dS_dB2 * (-2.0f * mx);
            }
            float* q = part + (size_t)(3 * c) * npix + image + (size_t)yy * w + xx;
            q[0] = dmx;
            q[npix] = dxx;
            q[2 * npix] = dxy;
        }
    }
    block_sum2(local, cnt, acc);
}

// Gradient of the loss
//   L = mean |pred - t| (RGBA) + ssim_w (1 - mean SSIM) + err_w mean (o4 - 1000 e)^2,
//   e = mean over RGBA of (pred - t)^2 (not differentiated),
// with respect to o (16 channels, bf16 for the backward convolutions); the
// partials, blurred here (the adjoint of the moments' blur), give
// dSSIM/dpred = B_mu + 2 pred B_xx + t B_xy; part null: no SSIM term.
// acc[2] += sum |pred - t|, acc[3] += sum (o4 - 1000 e)^2.  The SSIM count
// acc[1] is the one of ssim_partials_kernel (read by the host as ssim_count).
__global__ void __launch_bounds__(kLossThreads) loss_grad_kernel(const float* __restrict__ o,
                                                                 const __nv_bfloat16* __restrict__ x,
                                                                 const float4* __restrict__ target,
                                                                 const float* __restrict__ part, int n, int h, int w,
                                                                 bool wide, float inv_l1, float ssim_scale,
                                                                 float err_scale, __nv_bfloat16* __restrict__ dout,
                                                                 float* __restrict__ acc) {
    __shared__ float s_m[3][kLossRows][kLossStride];
    __shared__ float s_h[3][kLossRows][kLossHStride];
    const LossTile tile = loss_tile(h, w);
    const int t = threadIdx.x;
    const size_t image = (size_t)tile.b * h * w, npix = (size_t)n * h * w;
    const int hr = t >> 2, seg = (t & 3) * 8, col = t & 31, r0 = (t >> 5) * 4;
    float bl[3][3][4];   // blurred partials: channel, partial, row
    if (part) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            for (int i = t; i < kLossRows * kLossCols; i += kLossThreads) {
                const int r = i / kLossCols, cc = i % kLossCols, yy = tile.y0 - 5 + r, xx = tile.x0 - 5 + cc;
                const bool in = xx >= 0 && xx < w && yy >= 0 && yy < h;
                const float* q = part + (size_t)(3 * c) * npix + image + (in ? (size_t)yy * w + xx : 0);
#pragma unroll
                for (int k = 0; k < 3; ++k) s_m[k][r][cc] = in ? __ldg(q + k * npix) : 0.0f;
            }
            __syncthreads();
            if (hr < kLossRows) {
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    float v[18];
#pragma unroll
                    for (int i = 0; i < 18; ++i) v[i] = s_m[k][hr][seg + i];
                    blur8(v, &s_h[k][hr][seg]);
                }
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < 3; ++k) blur4(s_h[k], col, r0, bl[c][k]);
        }
    }
    float l1 = 0.0f, le = 0.0f;
    const int xx = tile.x0 + col;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int yy = tile.y0 + r0 + i;
        if (xx >= w || yy >= h) continue;
        const size_t at = image + (size_t)yy * w + xx;
        const float4 p = head_rgba(o, x, at, wide), q = __ldg(target + at);
        const float pv[4] = {p.x, p.y, p.z, p.w}, tv[4] = {q.x, q.y, q.z, q.w};
        float g[kOutC];
#pragma unroll
        for (int c = 0; c < kOutC; ++c) g[c] = 0.0f;
        float e = 0.0f;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const float d = pv[c] - tv[c];
            l1 += fabsf(d);
            e += d * d;
            g[c] = inv_l1 * (d > 0.0f ? 1.0f : d < 0.0f ? -1.0f : 0.0f);
        }
        e *= 0.25f;
        if (part) {
#pragma unroll
            for (int c = 0; c < 3; ++c)
                g[c] += -ssim_scale * (bl[c][0][i] + 2.0f * pv[c] * bl[c][1][i] + tv[c] * bl[c][2][i]);
        }
        const float r = o[at * kOutC + 4] - 1000.0f * e;
        le += r * r;
        g[4] = err_scale * 2.0f * r;
        uint4* op = reinterpret_cast<uint4*>(dout + at * kOutC);
#pragma unroll
        for (int k = 0; k < kOutC / 8; ++k) op[k] = pack8(reinterpret_cast<const float(&)[8]>(g[8 * k]));
    }
    block_sum2(l1, le, acc + 2);
}

// Adam (Kingma & Ba, bias-corrected) on the FP32 masters, and the packing of
// the weights into the convolutions' operand images (forward, and transposed
// for the input gradient), one launch over the whole parameter vector: as ten
// packing launches behind the Adam kernel they were 34 us of a step.
template <bool kAdam>
__global__ void update_pack_kernel(ParamImages im, float* __restrict__ w, const float* __restrict__ g,
                                   float* __restrict__ m, float* __restrict__ v, int count, float lr, float b1, float b2,
                                   float eps, float bc1, float bc2) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        float wi = w[i];
        if (kAdam) {
            const float gi = g[i];
            const float mi = b1 * m[i] + (1.0f - b1) * gi;
            const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
            m[i] = mi;
            v[i] = vi;
            const float mh = mi / bc1, vh = vi / bc2;
            wi -= lr * mh / (sqrtf(vh) + eps);
            w[i] = wi;
        }
        int l = 0;
        while (l + 1 < im.layers && i >= im.layer[l + 1].first) ++l;
        const ParamImages::Layer& L = im.layer[l];
        const int k = i - L.first;
        if (k >= 9 * L.cin * L.cout) continue;   // a bias
        const int co = k % L.cout, ci = (k / L.cout) % L.cin, tap = k / (L.cin * L.cout);
        const __nv_bfloat16 h = __float2bfloat16_rn(wi);
        *reinterpret_cast<__nv_bfloat16*>(L.image + conv::wimage_offset(tap, ci, co, L.cin, L.cout)) = h;
        // cut_cout: the output channel whose gradient stops at this layer
        *reinterpret_cast<__nv_bfloat16*>(L.image_t + conv::wimage_offset(8 - tap, co, ci, L.cout, L.cin)) =
            co == L.cut_cout ? __float2bfloat16_rn(0.0f) : h;
    }
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
static int grid_for(size_t n, int threads = 256) {
    size_t b = (n + threads - 1) / threads;
    return (int)(b < 148 * 16 ? (b ? b : 1) : 148 * 16);
}

void set_gauss_window(cudaStream_t s) {
    float g[11], sum = 0.0f;
    for (int k = -5; k <= 5; ++k) {
        g[k + 5] = expf(-(float)(k * k) / (2.0f * 1.5f * 1.5f));
        sum += g[k + 5];
    }
    for (float& v : g) v /= sum;
    cudaMemcpyToSymbolAsync(c_gauss, g, sizeof(g), 0, cudaMemcpyHostToDevice, s);
}

int launch_upsample_grad(const __nv_bfloat16* du, const __nv_bfloat16* e3, int n, int h, int w, __nv_bfloat16* dz3,
                         cudaStream_t s) {
    upsample_grad_kernel<<<grid_for((size_t)n * (h / 2) * (w / 2) * kHidQ), 256, 0, s>>>(
        reinterpret_cast<const uint4*>(du), reinterpret_cast<const uint4*>(e3), n, h, w, reinterpret_cast<uint4*>(dz3));
    return 1;
}
int launch_skip_pool_grad(const __nv_bfloat16* du, const __nv_bfloat16* dp1, const __nv_bfloat16* e1, int n, int h,
                          int w, __nv_bfloat16* dz1, cudaStream_t s) {
    skip_pool_grad_kernel<<<grid_for((size_t)n * h * w * kHidQ), 256, 0, s>>>(
        reinterpret_cast<const uint4*>(du), reinterpret_cast<const uint4*>(dp1), reinterpret_cast<const uint4*>(e1), n,
        h, w, reinterpret_cast<uint4*>(dz1));
    return 1;
}
static unsigned loss_tiles(int n, int h, int w) {
    return (unsigned)n * (unsigned)((w + kLossTx - 1) / kLossTx) * (unsigned)((h + kLossTy - 1) / kLossTy);
}
static bool wide_rows(const float* o, const __nv_bfloat16* x) { return (((uintptr_t)o | (uintptr_t)x) & 15u) == 0u; }
int launch_ssim_partials(const float* o, const __nv_bfloat16* x, const float4* target, int n, int h, int w, float* part,
                         float* acc, cudaStream_t s) {
    ssim_partials_kernel<<<loss_tiles(n, h, w), kLossThreads, 0, s>>>(o, x, target, n, h, w, wide_rows(o, x), part, acc);
    return 1;
}
int launch_loss_grad(const float* o, const __nv_bfloat16* x, const float4* target, const float* part, int n, int h,
                     int w, float inv_l1, float ssim_scale, float err_scale, __nv_bfloat16* dout, float* acc,
                     cudaStream_t s) {
    loss_grad_kernel<<<loss_tiles(n, h, w), kLossThreads, 0, s>>>(o, x, target, part, n, h, w, wide_rows(o, x), inv_l1,
                                                                 ssim_scale, err_scale, dout, acc);
    return 1;
}
int launch_adam(const ParamImages& im, float* w, const float* g, float* m, float* v, int count, float lr, float b1,
                float b2, float eps, float bc1, float bc2, cudaStream_t s) {
    update_pack_kernel<true><<<grid_for(count), 256, 0, s>>>(im, w, g, m, v, count, lr, b1, b2, eps, bc1, bc2);
    return 1;
}
int launch_pack_params(const ParamImages& im, float* w, int count, cudaStream_t s) {
    update_pack_kernel<false><<<grid_for(count), 256, 0, s>>>(im, w, nullptr, nullptr, nullptr, count, 0.f, 0.f, 0.f, 0.f,
                                                              1.f, 1.f);
    return 1;
}
}  // namespace dn
}  // namespace gs
