// Display transform of the linear RGBA16F frame: the gsanim 0.3 "layers"
// display pass (renderer_display_appearance, src/renderer.cpp:2120-2137;
// shaders/accum.glsl:201-240) or, without a LUT, the plain blit
// (shaders/accum.glsl:181-192).  One thread per pixel; the sampler is
// non-filtering at the frame's own resolution, so every output pixel reads
// its own input pixel.
//
// Per pixel: radiance = rgb * exp2(exposure_ev);
//   s = clamp((log2(max(radiance, exp2(log2_min))) - log2_min) / (log2_max - log2_min), 0, 1);
//   p = s * (lut_size - 1); trilinear lookup of the uint16 RGB lattice
//   (entry / 65535) between floor(p) and min(floor(p) + 1, lut_size - 1)
//   with weights fract(p), mixed x, then y, then z; alpha = 1.
// exp2 and log2 are the deterministic exp / log of gs_common.cuh scaled by
// ln 2 (the CPU oracle uses the same operations), so results are bit-exact
// against it.
#include <cuda_fp16.h>

#include "gs_common.cuh"
#include "gs_display.h"

namespace gs {

__device__ __forceinline__ float det_exp2f(float x) { return det_expf(mul(x, kLn2f)); }
__device__ __forceinline__ float det_log2f(float x) { return mul(det_logf(x), kInvLn2); }

// The table the display kernel reads: the uploaded uint16 lattice as floats
// (entry / 65535, the division the shader does per fetch), 16 bytes a point.
// The lattice arrives in the last 6 of every 16 bytes of the table's memory and
// is converted in place from the first point on, a thread a point: a launch
// takes the points whose 16 bytes end before the first unconverted entry (5 / 8 of
// what is left), so nothing it writes is read any more; the last points are one
// CTA's, which reads them all before it writes.
constexpr int kTableThreads = 1024;
__global__ void __launch_bounds__(kTableThreads) display_table_kernel(const uint16_t* lut, size_t first, size_t last,
                                                                      float4* table) {
    const size_t i = first + (size_t)blockIdx.x * kTableThreads + threadIdx.x;
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (i < last) {
        const uint16_t* a = lut + i * 3;
        v = make_float4(dv((float)a[0], 65535.0f), dv((float)a[1], 65535.0f), dv((float)a[2], 65535.0f), 0.0f);
    }
    __syncthreads();
    if (i < last) table[i] = v;
}

uint16_t* display_lattice(float4* table, int lut_size) {
    const size_t points = (size_t)lut_size * lut_size * lut_size;
    return reinterpret_cast<uint16_t*>(reinterpret_cast<char*>(table) + 10 * points);
}

int launch_display_table(float4* table, int lut_size, cudaStream_t s) {
    const size_t points = (size_t)lut_size * lut_size * lut_size;
    int launches = 0;
    for (size_t first = 0, last; first < points; first = last, ++launches) {
        last = points - first <= (size_t)kTableThreads ? points : (10 * points + 6 * first) / 16;
        const size_t grid = (last - first + kTableThreads - 1) / kTableThreads;
        display_table_kernel<<<(unsigned)grid, kTableThreads, 0, s>>>(display_lattice(table, lut_size), first, last, table);
    }
    return launches;
}

// g_mix with the weights 1 - a and a in hand.
__device__ __forceinline__ float mix_w(float x, float y, float wx, float wy) { return add(mul(x, wx), mul(y, wy)); }

// Bound by instruction issue (~600 warp instructions a pixel, most of them
// the three deterministic logarithms and their divisions), not by the 24
// bytes a pixel moves: 35 us at 1920x1080 with a 33^3 table, against 72 us
// when every fetch was three uint16 loads and three divisions by 65535 (24 of
// each a pixel).  Points interleaved with their +x neighbour (one 32-byte load
// for two fetches) measured the same 35 us with twice the table.
__global__ void __launch_bounds__(256) display_lut_kernel(DisplayParams p) {
    const size_t npix = (size_t)p.width * p.height;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npix) return;
    uint2 h = __ldg(reinterpret_cast<const uint2*>(p.in_rgba16f) + i);
    const float gain = det_exp2f(p.exposure_ev);
    const float lo_clamp = det_exp2f(p.log2_min);
    const float range = sub(p.log2_max, p.log2_min);
    const int n = p.lut_size, nn = n * n;
    const float top = (float)(n - 1);
    for (;;) {
        const size_t next = i + stride;
        const bool more = next < npix;
        uint2 hn = make_uint2(0u, 0u);
        if (more) hn = __ldg(reinterpret_cast<const uint2*>(p.in_rgba16f) + next);
        const float2 rg = __half22float2(*reinterpret_cast<const __half2*>(&h.x));
        const float2 ba = __half22float2(*reinterpret_cast<const __half2*>(&h.y));
        if (!p.table) {
            p.out_rgba32f[i] = make_float4(rg.x, rg.y, ba.x, ba.y);
        } else {
            const float rad[3] = {mul(rg.x, gain), mul(rg.y, gain), mul(ba.x, gain)};
            int lo[3], up[3];
            float f[3], e[3];   // weights of the upper and the lower lattice point
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                float s = g_clamp(dv(sub(det_log2f(g_max(rad[c], lo_clamp)), p.log2_min), range), 0.0f, 1.0f);
                if (s != s) s = 0.0f;   // NaN input: first lattice entry (as the oracle)
                const float pc = mul(s, top);
                const float fl = floorf(pc);
                lo[c] = (int)fl;
                up[c] = lo[c] + 1 < n ? 1 : 0;
                f[c] = sub(pc, fl);
                e[c] = sub(1.0f, f[c]);
            }
            const int base = lo[2] * nn + lo[1] * n + lo[0];
            const int dx = up[0], dy = up[1] ? n : 0, dz = up[2] ? nn : 0;
            const float4* t = p.table + base;
            const float4 l000 = __ldg(t), l100 = __ldg(t + dx), l010 = __ldg(t + dy), l110 = __ldg(t + dy + dx);
            const float4 l001 = __ldg(t + dz), l101 = __ldg(t + dz + dx), l011 = __ldg(t + dz + dy),
                         l111 = __ldg(t + dz + dy + dx);
            const float ex = e[0], fx = f[0], ey = e[1], fy = f[1], ez = e[2], fz = f[2];
            auto trilinear = [&](float a000, float a100, float a010, float a110, float a001, float a101, float a011,
                                 float a111) {
                const float a = mix_w(mix_w(a000, a100, ex, fx), mix_w(a010, a110, ex, fx), ey, fy);
                const float b = mix_w(mix_w(a001, a101, ex, fx), mix_w(a011, a111, ex, fx), ey, fy);
                return mix_w(a, b, ez, fz);
            };
            const float o[3] = {trilinear(l000.x, l100.x, l010.x, l110.x, l001.x, l101.x, l011.x, l111.x),
                                trilinear(l000.y, l100.y, l010.y, l110.y, l001.y, l101.y, l011.y, l111.y),
                                trilinear(l000.z, l100.z, l010.z, l110.z, l001.z, l101.z, l011.z, l111.z)};
            p.out_rgba32f[i] = make_float4(o[0], o[1], o[2], 1.0f);
        }
        if (!more) break;
        i = next;
        h = hn;
    }
}

int launch_display(const DisplayParams& p, uint32_t num_sms, cudaStream_t s) {
    const size_t npix = (size_t)p.width * p.height;
    if (npix == 0) return 0;
    size_t grid = (npix + 255) / 256;
    if (grid > (size_t)num_sms * 16) grid = (size_t)num_sms * 16;
    display_lut_kernel<<<(unsigned)grid, 256, 0, s>>>(p);
    return 1;
}

}  // namespace gs
