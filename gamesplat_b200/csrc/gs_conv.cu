// 3x3 "same" convolutions of the denoiser on the fifth-generation tensor
// cores (tcgen05.mma, BF16 operands, FP32 accumulators in TMEM).
//
// Tensors are NHWC bf16.  Weights are kept as FP32 masters in [tap][cin][cout]
// order (tap = ky * 3 + kx, ky = 0 the row above); each step packs them into
// the byte image of the shared-memory operand the kernels copy verbatim.
//
// conv_fwd_kernel (also the input gradient, with the transposed weights):
// implicit GEMM with M = 128 output pixels of one image row, N = Cout,
// K = 9 taps x Cin.  A persistent CTA walks column strips of 128 pixels down
// its share of the rows; input rows (130 pixels with the halo) pass through a
// ring of shared-memory slots in the K-major core-matrix layout, rows of
// 16 bytes one pixel apart, so the A operand of tap (ky, kx) is the slot of row
// y - 1 + ky started kx pixels (kx * 16 bytes) further: no im2col copy.  The
// warps have fixed roles that meet only at mbarriers: 8 load rows, one thread
// issues the 9 * Cin / 16 MMAs of a row into one of 4 TMEM accumulators, and 4
// read accumulators back (thread t = TMEM lane t = pixel t) for the epilogue
// (bias, ReLU, ReLU mask, bf16 / f32 store).
//
// conv_wgrad_kernel: the weight gradient, K = pixels; see there.
//
// Every wait is bounded; a wait that runs out sets err[0] and the kernel
// frees its TMEM and returns.
#include <cuda_bf16.h>

#include "gs_conv.h"
#include "gs_internal.h"
#include "gs_umma.cuh"

namespace gs {
namespace conv {

constexpr int kHaloRows = 136;                  // 130 used (pixels x0-1 .. x0+128)
// One 8-channel column of a halo row (kHaloRows pixels of 16 bytes) plus
// padding.  Consecutive threads copy the kG columns of a pixel, then the next
// pixel's; a quarter warp's eight 16-byte copies hit distinct banks when the
// columns are 8 banks apart for kG = 4 (stride = 32 mod 128 bytes) and 16
// banks apart for kG = 2 (64 mod 128).  It is also the MMA descriptors'
// K-direction stride.
__host__ __device__ constexpr int col_bytes(int cin) { return kHaloRows * 16 + (cin / 8 == 2 ? 64 : 32); }
constexpr uint32_t kWaitLimit = 1u << 22;

__host__ __device__ constexpr int wimage_bytes(int cin, int cout) { return 9 * cin * cout * 2; }

// Roles of the forward kernel's warps (an epilogue warp's number is its TMEM lane quadrant).
constexpr int kEpiWarps = 4, kLoadWarps = 8, kMmaWarp = kEpiWarps + kLoadWarps;
constexpr int kFwdThreads = (kMmaWarp + 1) * 32;
constexpr int kLoaders = kLoadWarps * 16;   // threads of a load group: the two groups take rows in turn
constexpr int kSlots = 8;                   // halo rows in the ring
constexpr int kAccs = 4;                    // TMEM accumulators of 32 columns

// Dynamic shared memory of the forward kernel: the halo rows and the weight image.
__host__ __device__ constexpr int fwd_smem_bytes(int cin, int cout) {
    return kSlots * (cin / 8) * col_bytes(cin) + wimage_bytes(cin, cout);
}

// 16-byte asynchronous global -> shared copy (zero-filled when src_bytes is 0).
__device__ __forceinline__ void cp_async16(void* dst, const void* src, uint32_t src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(src_bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all_but_one() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Wait for phase `phase` of a barrier, suspended for up to a microsecond between tests; false after a second or so.
__device__ __forceinline__ bool mbar_wait_suspend(uint64_t* bar, uint32_t phase) {
    for (uint32_t i = 0; i < (1u << 20); ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(phase), "r"(1000u)
            : "memory");
        if (ok) return true;
    }
    return false;
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// 32 bytes to global memory (32-byte aligned).
__device__ __forceinline__ void st_global32(void* p, const uint4& a, const uint4& b) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(a.x), "r"(a.y), "r"(a.z),
                 "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
                 : "memory");
}

__device__ __forceinline__ uint4 bf16x8_add(uint4 a, uint4 b) {
    uint4 r;
    const __nv_bfloat162* pa = reinterpret_cast<const __nv_bfloat162*>(&a);
    const __nv_bfloat162* pb = reinterpret_cast<const __nv_bfloat162*>(&b);
    __nv_bfloat162* pr = reinterpret_cast<__nv_bfloat162*>(&r);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 fa = __bfloat1622float2(pa[i]), fb = __bfloat1622float2(pb[i]);
        pr[i] = __floats2bfloat162_rn(fa.x + fb.x, fa.y + fb.y);
    }
    return r;
}

// 8 channels (16 bytes) of input pixel (n, y, x), zero outside the image.
// kLoad 1: the decoder input, nearest 2x upsampling of `xh` (half
// resolution) plus `x` at full resolution.
template <int kCin, int kLoad>
__device__ __forceinline__ uint4 load_granule(const ConvArgs& a, int n, int y, int x, int g) {
    if (y < 0 || y >= a.h || x < 0 || x >= a.w) return make_uint4(0u, 0u, 0u, 0u);
    const size_t pix = ((size_t)n * a.h + y) * a.w + x;
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(a.x + pix * kCin) + g);
    if (kLoad == 0) return v;
    const int hh = a.h >> 1, hw = a.w >> 1;
    const size_t hp = ((size_t)n * hh + min(y >> 1, hh - 1)) * hw + min(x >> 1, hw - 1);
    return bf16x8_add(v, __ldg(reinterpret_cast<const uint4*>(a.xh + hp * kCin) + g));
}

// A run of rows [y0, y1) of one strip; a CTA's share of the units is a sequence of them.
struct ConvRun {
    int n, x0, y0, y1;
};

// The runs of a CTA: units (unit_rows rows of a strip, bands shifted up by
// row_offset) are numbered strip by strip, and CTA b takes an equal share.
struct ConvRuns {
    int strips_x, bands, u, u1, unit_rows, row_offset, h;
    __device__ __forceinline__ ConvRuns(const ConvArgs& a)
        : strips_x((a.w + 127) / 128), bands((a.h + a.row_offset + a.unit_rows - 1) / a.unit_rows),
          unit_rows(a.unit_rows), row_offset(a.row_offset), h(a.h) {
        const long long total = (long long)a.n * strips_x * bands;
        u = (int)(total * blockIdx.x / gridDim.x);
        u1 = (int)(total * (blockIdx.x + 1) / gridDim.x);
    }
    __device__ __forceinline__ bool next(ConvRun& r) {
        if (u >= u1) return false;
        const int strip = u / bands, b0 = u - strip * bands;
        const int ue = min(u1, (strip + 1) * bands);
        r.n = strip / strips_x;
        r.x0 = (strip % strips_x) * 128;
        r.y0 = max(0, b0 * unit_rows - row_offset);
        r.y1 = min(h, (ue - strip * bands) * unit_rows - row_offset);
        u = ue;
        return true;
    }
};

// Bound by HBM: every input row of a strip is read once (and 2 more at each
// end of a run), every output written once in 32-byte sectors.  Before, a CTA
// of 128 threads did copy, MMAs and epilogue of a row in turn, at ~6 us a row
// (four CTAs an SM) for 16 KB moved; with the roles apart four rows are in flight
// per CTA (two CTAs an SM) and the MMAs of a row overlap the epilogue of the
// ones before.  Times before and after at launch_fwd.
template <int kCin, int kCout, int kLoad>
__global__ void __launch_bounds__(kFwdThreads, 2) conv_fwd_kernel(ConvArgs a) {
    static_assert(kCin % 16 == 0 && (kCout == 16 || kCout == 32), "channel counts");
    constexpr int kG = kCin / 8;                         // 16-byte columns per pixel
    constexpr int kColBytes = col_bytes(kCin);
    constexpr int kSlot = kG * kColBytes;                // one halo row
    constexpr int kW = wimage_bytes(kCin, kCout);
    constexpr uint32_t kIdesc = umma::idesc_bf16(128, kCout, 0, 0);
    extern __shared__ __align__(128) uint8_t smem[];
    uint8_t* s_w = smem + kSlots * kSlot;
    __shared__ __align__(8) uint64_t s_full[kSlots], s_empty[kSlots];        // a row has landed; its MMAs are done
    __shared__ __align__(8) uint64_t s_afull[kAccs], s_aempty[kAccs];        // an accumulator is done; it was read
    __shared__ uint32_t s_taddr;
    __shared__ float s_bias[kCout];
    constexpr bool kPool = kCin == 16 && kCout == 32;   // the pooled output (conv1 of the denoiser)
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    if (tid == 0) {
        for (int k = 0; k < kSlots; ++k) {
            mbar_init(&s_full[k], kLoaders);
            mbar_init(&s_empty[k], 1);
        }
        for (int k = 0; k < kAccs; ++k) {
            mbar_init(&s_afull[k], 1);
            mbar_init(&s_aempty[k], kEpiWarps * 32);
        }
        mbar_fence_init();
    }
    if (warp == kMmaWarp) umma::tmem_alloc(&s_taddr, kAccs * 32);
    pdl_wait();   // launched as a programmatic dependent: nothing above touches global memory
    // weights: the packed image, copied verbatim; the bias
    for (int i = tid; i < kW / 16; i += kFwdThreads)
        reinterpret_cast<uint4*>(s_w)[i] = __ldg(reinterpret_cast<const uint4*>(a.wimage) + i);
    if (tid < kCout) s_bias[tid] = a.bias ? __ldg(a.bias + tid) : 0.0f;
    umma::fence_smem_to_async();
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t taddr = s_taddr;
    ConvRuns runs(a);
    ConvRun r;
    bool failed = false;

    if (warp >= kEpiWarps && warp < kMmaWarp) {
        // ---- load: entry e of the ring (the run's rows y0 - 1 .. y1, then the next run's) by group e & 1
        const int lt = (tid - kEpiWarps * 32) % kLoaders;
        const uint32_t group = (uint32_t)((tid - kEpiWarps * 32) / kLoaders);
        uint32_t e = 0;
        int pending = -1;   // slot of this group's copied row that is not announced yet
        while (!failed && runs.next(r)) {
            for (int yy = r.y0 - 1; yy <= r.y1 && !failed; ++yy, ++e) {
                if ((e & 1u) != group) continue;
                const int slot = (int)(e % kSlots);
                if (e >= kSlots && !mbar_wait_suspend(&s_empty[slot], (e / kSlots - 1u) & 1u)) {
                    failed = true;
                    break;
                }
                uint8_t* dst = smem + slot * kSlot;
                const bool row_in = yy >= 0 && yy < a.h;
                const __nv_bfloat16* rowp = a.x + ((size_t)r.n * a.h + (row_in ? yy : 0)) * a.w * kCin;
                if (kLoad == 0) {
                    // copied asynchronously; announced once the group's next row is on its way
                    for (int q = lt; q < 130 * kG; q += kLoaders) {
                        const int hp = q / kG, g = q - hp * kG, x = r.x0 - 1 + hp;
                        const bool in = row_in && x >= 0 && x < a.w;
                        cp_async16(dst + g * kColBytes + hp * 16, in ? rowp + (size_t)x * kCin + g * 8 : a.x, in ? 16u : 0u);
                    }
                    cp_async_commit();
                    if (pending >= 0) {
                        cp_async_wait_all_but_one();
                        umma::fence_smem_to_async();
                        mbar_arrive(&s_full[pending]);
                    }
                    pending = slot;
                } else {
                    // x + the 2x nearest upsampling of xh (FP32 sum rounded to bf16): all of a
                    // thread's granules loaded before the first is stored
                    constexpr int kPer = (130 * kG + kLoaders - 1) / kLoaders;
                    const int hh = a.h >> 1, hw = a.w >> 1;
                    const __nv_bfloat16* hrow = a.xh + ((size_t)r.n * hh + (row_in ? min(yy >> 1, hh - 1) : 0)) * hw * kCin;
                    uint4 v[kPer], u[kPer];
#pragma unroll
                    for (int k = 0; k < kPer; ++k) {
                        const int q = lt + k * kLoaders, hp = q / kG, g = q - hp * kG, x = r.x0 - 1 + hp;
                        v[k] = u[k] = make_uint4(0u, 0u, 0u, 0u);
                        if (row_in && x >= 0 && x < a.w && q < 130 * kG) {
                            v[k] = __ldg(reinterpret_cast<const uint4*>(rowp + (size_t)x * kCin) + g);
                            u[k] = __ldg(reinterpret_cast<const uint4*>(hrow + (size_t)min(x >> 1, hw - 1) * kCin) + g);
                        }
                    }
#pragma unroll
                    for (int k = 0; k < kPer; ++k) {
                        const int q = lt + k * kLoaders, hp = q / kG, g = q - hp * kG;
                        if (q < 130 * kG) *reinterpret_cast<uint4*>(dst + g * kColBytes + hp * 16) = bf16x8_add(v[k], u[k]);
                    }
                    umma::fence_smem_to_async();
                    mbar_arrive(&s_full[slot]);
                }
            }
        }
        cp_async_wait_all();
        if (pending >= 0) {
            umma::fence_smem_to_async();
            mbar_arrive(&s_full[pending]);
        }
    } else if (warp == kMmaWarp) {
        // ---- multiply: one thread
        if (lane == 0) {
            const uint32_t halo_base = smem_u32(smem), w_base = smem_u32(s_w);
            uint32_t e = 0, m = 0;   // ring entry of the row above; output rows so far
            while (!failed && runs.next(r)) {
                for (int y = r.y0; y < r.y1; ++y, ++e, ++m) {
                    bool ok = true;
                    for (uint32_t k = y == r.y0 ? 0u : 2u; k < 3u && ok; ++k)
                        ok = mbar_wait_suspend(&s_full[(e + k) % kSlots], ((e + k) / kSlots) & 1u);
                    const uint32_t acc = m % kAccs;
                    if (ok && m >= kAccs) ok = mbar_wait_suspend(&s_aempty[acc], (m / kAccs - 1u) & 1u);
                    if (!ok) {
                        failed = true;
                        break;
                    }
                    umma::fence_after_sync();
                    uint32_t accumulate = 0;
#pragma unroll
                    for (int ky = 0; ky < 3; ++ky) {
                        const uint32_t slot = halo_base + ((e + (uint32_t)ky) % kSlots) * (uint32_t)kSlot;
#pragma unroll
                        for (int kx = 0; kx < 3; ++kx) {
#pragma unroll
                            for (int kb = 0; kb < kCin / 16; ++kb) {
                                const uint64_t ad = umma::smem_desc(slot + (uint32_t)(2 * kb * kColBytes + kx * 16),
                                                                    (uint32_t)kColBytes, 128u);
                                const int k0 = (ky * 3 + kx) * kCin + kb * 16;
                                const uint64_t bd = umma::smem_desc(w_base + (uint32_t)((k0 >> 3) * kCout * 16),
                                                                    (uint32_t)(kCout * 16), 128u);
                                umma::mma_bf16(taddr + acc * 32u, ad, bd, kIdesc, accumulate);
                                accumulate = 1;
                            }
                        }
                    }
                    umma::commit(&s_empty[e % kSlots]);   // this row was the last to read the row above it
                    umma::commit(&s_afull[acc]);
                }
                if (!failed) {   // the run's last two halo rows
                    umma::commit(&s_empty[e % kSlots]);
                    umma::commit(&s_empty[(e + 1u) % kSlots]);
                    e += 2u;
                }
            }
            // every MMA of this CTA, and the last commit's arrival, is done before its shared memory and TMEM go
            if (!failed && m > 0 && !mbar_wait_suspend(&s_empty[(e - 1u) % kSlots], ((e - 1u) / kSlots) & 1u)) failed = true;
        }
        __syncwarp();
    } else {
        // ---- epilogue: thread t holds pixel x0 + t of a row
        uint32_t m = 0;
        float err_sum = 0.0f, err_cnt = 0.0f;   // head mode: this thread's column of the band, in row order
        uint32_t even[kPool ? 16 : 1];          // the bf16 outputs of the even row above (pooled output)
        while (!failed && runs.next(r)) {
            const int x = r.x0 + tid;
            for (int y = r.y0; y < r.y1; ++y, ++m) {
                const uint32_t acc = m % kAccs;
                const size_t o = ((size_t)r.n * a.h + y) * a.w + x;
                if (!mbar_wait_suspend(&s_afull[acc], (m / kAccs) & 1u)) {
                    failed = true;
                    break;
                }
                umma::fence_after_sync();
                const uint32_t acc_addr = taddr + acc * 32u + ((uint32_t)(warp * 32) << 16);
                float v[32];
                if (kCout == 32) umma::tmem_ld32(acc_addr, *reinterpret_cast<float(*)[32]>(v));
                else umma::tmem_ld16(acc_addr, *reinterpret_cast<float(*)[16]>(v));
                umma::fence_before_sync();
                mbar_arrive(&s_aempty[acc]);
                uint32_t pk[kCout / 2];
                if (a.bias) {
#pragma unroll
                    for (int c = 0; c < kCout; ++c) v[c] += s_bias[c];
                }
                if (a.relu) {
#pragma unroll
                    for (int c = 0; c < kCout; ++c) v[c] = fmaxf(v[c], 0.0f);
                }
                if (x < a.w) {
                    if (a.mask) {
                        const uint4* mp = reinterpret_cast<const uint4*>(a.mask + o * kCout);
#pragma unroll
                        for (int q = 0; q < kCout / 8; ++q) {
                            const uint4 mv = __ldg(mp + q);
                            const __nv_bfloat16* mb = reinterpret_cast<const __nv_bfloat16*>(&mv);
#pragma unroll
                            for (int i = 0; i < 8; ++i)
                                if (!(__bfloat162float(mb[i]) > 0.0f)) v[q * 8 + i] = 0.0f;
                        }
                    }
                    if (kCout == 16 && a.head_x) {
                        // the denoised frame's pixel (head_rgba of the output step) and its error estimate
                        const uint4 xv = __ldg(reinterpret_cast<const uint4*>(a.head_x + o * 16));
                        const __nv_bfloat16* xb = reinterpret_cast<const __nv_bfloat16*>(&xv);
                        const float4 px = make_float4(__bfloat162float(xb[5]) + v[0], __bfloat162float(xb[6]) + v[1],
                                                      __bfloat162float(xb[7]) + v[2], __bfloat162float(xb[3]) + v[3]);
                        __half2 h01 = __floats2half2_rn(px.x, px.y), h23 = __floats2half2_rn(px.z, px.w);
                        uint2 pk2;
                        pk2.x = *reinterpret_cast<uint32_t*>(&h01);
                        pk2.y = *reinterpret_cast<uint32_t*>(&h23);
                        reinterpret_cast<uint2*>(a.head_out16)[o] = pk2;
                        err_sum += fmaxf(v[4], 0.0f);
                        err_cnt += 1.0f;
                    }
                }
#pragma unroll
                for (int i = 0; i < kCout / 2; ++i) {
                    __nv_bfloat162 b2 = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
                    pk[i] = *reinterpret_cast<uint32_t*>(&b2);
                }
                if (a.out_bf16 && x < a.w) {
                    uint4* op = reinterpret_cast<uint4*>(a.out_bf16 + o * kCout);
#pragma unroll
                    for (int q = 0; q < kCout / 16; ++q) {
                        const uint4 lo = make_uint4(pk[8 * q], pk[8 * q + 1], pk[8 * q + 2], pk[8 * q + 3]);
                        const uint4 hi = make_uint4(pk[8 * q + 4], pk[8 * q + 5], pk[8 * q + 6], pk[8 * q + 7]);
                        if (a.out_wide) {
                            st_global32(op + 2 * q, lo, hi);
                        } else {
                            op[2 * q] = lo;
                            op[2 * q + 1] = hi;
                        }
                    }
                }
                if (a.out_f32 && x < a.w) {
                    float4* op = reinterpret_cast<float4*>(a.out_f32 + o * kCout);
#pragma unroll
                    for (int q = 0; q < kCout / 4; ++q)
                        op[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                }
                if (kPool && a.pool_out) {
                    // 2x2 average of the bf16 outputs: (0 + (y, x) + (y, x + 1) + (y + 1, x) + (y + 1, x + 1)) * 0.25,
                    // the right neighbour's by lane shuffles (runs hold whole row pairs)
                    if ((y & 1) == 0) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) even[i] = pk[i];
                    } else {
                        const bool write = (x & 1) == 0 && x < a.w;
                        uint4* dp = reinterpret_cast<uint4*>(
                            a.pool_out + (((size_t)r.n * (a.h >> 1) + (y >> 1)) * (a.w >> 1) + (x >> 1)) * kCout);
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            uint32_t res[4];
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const uint32_t up = even[4 * q + i], down = pk[4 * q + i];
                                const uint32_t t4[4] = {up, __shfl_xor_sync(0xffffffffu, up, 1), down,
                                                        __shfl_xor_sync(0xffffffffu, down, 1)};
                                float acc0 = 0.0f, acc1 = 0.0f;
#pragma unroll
                                for (int k = 0; k < 4; ++k) {
                                    const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&t4[k]));
                                    acc0 += f.x;
                                    acc1 += f.y;
                                }
                                __nv_bfloat162 r2 = __floats2bfloat162_rn(0.25f * acc0, 0.25f * acc1);
                                res[i] = *reinterpret_cast<uint32_t*>(&r2);
                            }
                            if (write) dp[q] = make_uint4(res[0], res[1], res[2], res[3]);
                        }
                    }
                }
                if (kCout == 16 && a.head_x && (y + 1 == r.y1 || (y + 1 + a.row_offset) % 16 == 0)) {
                    // end of a band: per tile (16 threads = 16 columns) the sum of the error estimates and the
                    // pixel count, each over 16 lanes in a fixed order, then the tile's mean
#pragma unroll
                    for (int off = 8; off; off >>= 1) {
                        err_sum += __shfl_xor_sync(0xffffffffu, err_sum, off);
                        err_cnt += __shfl_xor_sync(0xffffffffu, err_cnt, off);
                    }
                    const int tx = (r.x0 >> 4) + (tid >> 4);
                    if ((tid & 15) == 0 && tx < a.tiles_x && err_cnt > 0.0f) {
                        const int band = (y + a.row_offset) / 16;
                        const int ty = (a.h + a.row_offset) / 16 - 1 - band;   // GL tile row of this band
                        const uint32_t tile = (uint32_t)(ty * a.tiles_x + tx);
                        const float mse = err_sum / err_cnt * 0.001f;
                        if (a.tile_err) a.tile_err[tile] = mse;
                        if (mse >= a.err_budget) a.fallback_tiles[atomicAdd(a.fallback_count, 1u)] = tile;
                    }
                    err_sum = err_cnt = 0.0f;
                }
            }
        }
    }
    if (failed && (lane == 0 || warp != kMmaWarp)) atomicOr(a.err, 1u);
    umma::fence_before_sync();
    __syncthreads();
    if (warp == kMmaWarp) {
        umma::fence_after_sync();
        umma::tmem_dealloc(taddr, kAccs * 32);
    }
}

// ---------------------------------------------------------------------------
// Weight gradient.
// ---------------------------------------------------------------------------
// dW[ky][kx][ci][co] = sum over pixels of X[p + (ky - 1, kx - 1)][ci] dY[p][co]:
// K = pixels, both operands MN-major (8 channels of a pixel are 16 bytes, as
// NHWC stores them).  A CTA takes strips of 128 pixels by up to 4 rows; the
// strip's X rows with their halo sit in shared memory once, row slot after row
// slot, so that the 16 row groups of one M = 128 operand, all a column of
// 8 channels apart, are the rows y - 1, y, y + 1 (and what lies below them:
// rows of D past 3 x Cin, never read) and tap kx is the same operand started
// kx pixels further.  Per output row: 3 taps x 8 K-steps MMAs into 3
// accumulators.  Two stages: the strip after the next is copied (cp.async)
// while one is multiplied, and MMAs of consecutive strips queue without a
// wait between them.  The bias gradient is summed from the staged dY by the
// threads while the MMAs run.  Bound by the shared-memory reads of the MMAs
// and the L2 reads of the strips (1.5 reads of X for 4 rows); 8 x 256 x 256
// pixels, 32 -> 32 channels: 262 us (load mode 1) when every tap was gathered
// from global memory and nothing overlapped; figures now at launch_wgrad.
constexpr int kWgThreads = 256;
constexpr int kWgPx = 128;    // pixels of a strip
constexpr int kWgRows = 4;    // output rows of a strip, at most
// A channel group of a dY row: 2 or 4 of them are copied by a quarter warp (as col_bytes)
__host__ __device__ constexpr int wg_dcol(int cout) { return kWgPx * 16 + (cout / 8 == 2 ? 64 : 32); }
// row slots of a stage: the rows of a strip, its halo, and what an M = 128 operand of the last row spans
__host__ __device__ constexpr int wg_slots(int cin) { return kWgRows - 1 + 128 / cin; }
__host__ __device__ constexpr int wg_x_bytes(int cin) { return wg_slots(cin) * (cin / 8) * col_bytes(cin); }
__host__ __device__ constexpr int wg_stage_bytes(int cin, int cout) {
    return wg_x_bytes(cin) + kWgRows * (cout / 8) * wg_dcol(cout);
}

template <int kCin, int kCout, int kLoad>
__global__ void __launch_bounds__(kWgThreads) conv_wgrad_kernel(WgradArgs a, int rows) {
    constexpr int kG = kCin / 8, kGo = kCout / 8;
    constexpr int kCol = col_bytes(kCin), kSlot = kG * kCol, kDcol = wg_dcol(kCout), kDrow = kGo * kDcol;
    constexpr int kStage = wg_stage_bytes(kCin, kCout), kX = wg_x_bytes(kCin);
    constexpr uint32_t kIdesc = umma::idesc_bf16(128, kCout, 1, 1);
    constexpr int kCols = 128;   // TMEM: 3 accumulators of kCout columns
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t s_bar[2];   // MMA completion, one per stage
    __shared__ uint32_t s_taddr;
    __shared__ float s_db[kWgThreads / 32][kCout];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    if (tid == 0) {
        mbar_init(&s_bar[0], 1);
        mbar_init(&s_bar[1], 1);
        mbar_fence_init();
    }
    if (warp == 0) umma::tmem_alloc(&s_taddr, kCols);
    // the slots no strip fills are operands too (their products are never read)
    for (int i = tid; i < 2 * kStage / 16; i += kWgThreads) reinterpret_cast<uint4*>(smem)[i] = make_uint4(0u, 0u, 0u, 0u);
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t taddr = s_taddr, base = smem_u32(smem);
    const int strips_x = (a.w + kWgPx - 1) / kWgPx, bands = (a.h + rows - 1) / rows;
    const int total = a.n * bands * strips_x;
    const ConvArgs ca{a.x, a.xh, a.n, a.h, a.w};

    struct Strip {
        int n, y0, x0, rows, px;   // px: pixels in whole K-steps
    };
    auto strip_at = [&](int item) {
        Strip s;
        s.x0 = (item % strips_x) * kWgPx;
        const int q = item / strips_x;
        s.n = q / bands;
        s.y0 = (q % bands) * rows;
        s.rows = min(rows, a.h - s.y0);
        s.px = (min(kWgPx, a.w - s.x0) + 15) & ~15;
        return s;
    };
    // X rows y0 - 1 .. y0 + rows (zero outside the image) into slots 0 ..., dY rows behind them
    auto load = [&](int stage, int item) {
        const Strip s = strip_at(item);
        uint8_t* xs = smem + stage * kStage;
        uint8_t* ds = xs + kX;
        const int row_q = (s.px + 2) * kG;
        for (int r = 0; r < s.rows + 2; ++r) {
            const int y = s.y0 - 1 + r;
            if (kLoad == 0) {
                const bool row_in = y >= 0 && y < a.h;
                const __nv_bfloat16* rowp = a.x + ((size_t)s.n * a.h + (row_in ? y : 0)) * a.w * kCin;
                for (int q = tid; q < row_q; q += kWgThreads) {
                    const int hp = q / kG, g = q % kG, x = s.x0 - 1 + hp;
                    const bool in = row_in && x >= 0 && x < a.w;
                    cp_async16(xs + r * kSlot + g * kCol + hp * 16, in ? rowp + (size_t)x * kCin + g * 8 : a.x,
                               in ? 16u : 0u);
                }
            } else {
                for (int q = tid; q < row_q; q += kWgThreads) {
                    const int hp = q / kG, g = q % kG;
                    *reinterpret_cast<uint4*>(xs + r * kSlot + g * kCol + hp * 16) =
                        load_granule<kCin, kLoad>(ca, s.n, y, s.x0 - 1 + hp, g);
                }
            }
        }
        for (int r = 0; r < s.rows; ++r) {
            const __nv_bfloat16* rowp = a.dy + ((size_t)s.n * a.h + s.y0 + r) * a.w * kCout;
            for (int q = tid; q < s.px * kGo; q += kWgThreads) {
                const int k = q / kGo, g = q % kGo, x = s.x0 + k;
                const bool in = x < a.w;
                cp_async16(ds + r * kDrow + g * kDcol + k * 16, in ? rowp + (size_t)x * kCout + g * 8 : a.dy, in ? 16u : 0u);
            }
        }
        cp_async_commit();
    };

    uint32_t phase[2] = {0u, 0u};
    bool failed = false, any = false;
    float db[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};   // of channel group tid % kGo
    int stage = 0;
    if ((int)blockIdx.x < total) load(0, blockIdx.x);
    for (int item = blockIdx.x; item < total; item += gridDim.x, stage ^= 1) {
        asm volatile("cp.async.wait_all;" ::: "memory");   // this strip, copied while the last one was multiplied
        umma::fence_smem_to_async();
        if (__syncthreads_or(failed)) {
            failed = true;
            break;
        }
        const Strip s = strip_at(item);
        if (tid == 0) {
            umma::fence_after_sync();
            const uint32_t xa = base + (uint32_t)(stage * kStage), da = xa + (uint32_t)kX;
            for (int r = 0; r < s.rows; ++r)
                for (int kk = 0; kk < s.px / 16; ++kk) {
                    const uint64_t bd = umma::smem_desc(da + (uint32_t)(r * kDrow + kk * 256), 128u, (uint32_t)kDcol);
#pragma unroll
                    for (int kx = 0; kx < 3; ++kx) {
                        const uint64_t ad =
                            umma::smem_desc(xa + (uint32_t)(r * kSlot + kx * 16 + kk * 256), 128u, (uint32_t)kCol);
                        umma::mma_bf16(taddr + (uint32_t)(kx * kCout), ad, bd, kIdesc, (any || r + kk > 0) ? 1u : 0u);
                    }
                }
            umma::commit(&s_bar[stage]);
        }
        if (a.db) {   // pixels past the row are zero
            const uint8_t* ds = smem + stage * kStage + kX + (tid % kGo) * kDcol;
            for (int r = 0; r < s.rows; ++r)
                for (int k = tid / kGo; k < s.px; k += kWgThreads / kGo) {
                    const uint4 v = *reinterpret_cast<const uint4*>(ds + r * kDrow + k * 16);
                    const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 f = __bfloat1622float2(p[e]);
                        db[2 * e] += f.x;
                        db[2 * e + 1] += f.y;
                    }
                }
        }
        const int next = item + (int)gridDim.x;
        if (next < total) {
            // the other stage: its MMAs (the previous strip's) read it to the end, and every
            // thread is past its sum over it (the barrier above)
            if (any) {
                if (!mbar_wait_bounded(&s_bar[stage ^ 1], phase[stage ^ 1], kWaitLimit)) failed = true;
                phase[stage ^ 1] ^= 1u;
            }
            load(stage ^ 1, next);
        }
        any = true;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (any && !failed) {   // the last strip's MMAs complete after all earlier ones
        if (!mbar_wait_bounded(&s_bar[stage ^ 1], phase[stage ^ 1], kWaitLimit)) failed = true;
    }
    if (__syncthreads_or(failed)) failed = true;
    umma::fence_after_sync();
    if (any && !failed) {
        // D rows m = ky * kCin + ci < 3 kCin of tap column kx; warps 0..3 read taps 0 and 1, warps 4..7 tap 2
        const int m = (warp & 3) * 32 + lane;
        const bool vec = (reinterpret_cast<uintptr_t>(a.dw) & 15u) == 0u;
        if ((warp & 3) * 32 < 3 * kCin) {
            for (int kx = warp < 4 ? 0 : 2; kx < (warp < 4 ? 2 : 3); ++kx) {
                float v[32];
                const uint32_t at = taddr + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(kx * kCout);
                if (kCout == 32) umma::tmem_ld32(at, *reinterpret_cast<float(*)[32]>(v));
                else umma::tmem_ld16(at, *reinterpret_cast<float(*)[16]>(v));
                if (m < 3 * kCin) {
                    float* dst = a.dw + ((size_t)((m / kCin) * 3 + kx) * kCin + m % kCin) * kCout;
                    if (vec) {
#pragma unroll
                        for (int c = 0; c < kCout / 4; ++c)
                            atomicAdd(reinterpret_cast<float4*>(dst) + c,
                                      make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]));
                    } else {
#pragma unroll
                        for (int c = 0; c < kCout; ++c) atomicAdd(dst + c, v[c]);
                    }
                }
            }
        }
    }
    if (a.db) {
        // lanes of one channel group, then the warps
#pragma unroll
        for (int e = 0; e < 8; ++e) {
#pragma unroll
            for (int off = 16; off >= kGo; off >>= 1) db[e] += __shfl_xor_sync(0xffffffffu, db[e], off);
            if (lane < kGo) s_db[warp][lane * 8 + e] = db[e];
        }
        __syncthreads();
        if (tid < kCout && any && !failed) {
            float sum = 0.0f;
            for (int q = 0; q < kWgThreads / 32; ++q) sum += s_db[q][tid];
            atomicAdd(a.db + tid, sum);
        }
    }
    if (failed && tid == 0) atomicOr(a.err, 1u);
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) umma::tmem_dealloc(taddr, kCols);
}

// ---------------------------------------------------------------------------
// Weight packing: FP32 masters [tap][cin][cout] -> the bf16 B-operand image of
// the forward convolution, or of the transposed convolution that gives the
// input gradient (cin' = cout, cout' = cin, tap' = 8 - tap).  For the
// stage-level convolutions; the denoiser packs its layers together
// (dn::launch_pack_params).
// ---------------------------------------------------------------------------
__global__ void pack_weights_kernel(const float* __restrict__ w, int cin, int cout, int transposed,
                                    uint8_t* __restrict__ image) {
    const int total = 9 * cin * cout;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const int co = i % cout, ci = (i / cout) % cin, tap = i / (cin * cout);
        const float v = w[i];
        int k, nn, cdim;
        if (!transposed) {
            k = tap * cin + ci;
            nn = co;
            cdim = cout;
        } else {
            k = (8 - tap) * cout + co;
            nn = ci;
            cdim = cin;
        }
        *reinterpret_cast<__nv_bfloat16*>(image + wimage_offset(k, nn, cdim)) = __float2bfloat16_rn(v);
    }
}

template <int kCin, int kCout, int kLoad>
static int launch_fwd_t(ConvArgs a, cudaStream_t s) {
    const long strips = (long)a.n * ((a.w + 127) / 128);
    const long units = strips * ((a.h + a.row_offset + a.unit_rows - 1) / a.unit_rows);
    const size_t smem = (size_t)fwd_smem_bytes(kCin, kCout);
    a.out_wide = (reinterpret_cast<uintptr_t>(a.out_bf16) & 31u) == 0u ? 1 : 0;
    static bool attr = false;
    if (!attr) {
        cudaFuncSetAttribute(conv_fwd_kernel<kCin, kCout, kLoad>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem);
        attr = true;
    }
    // two CTAs an SM; on small images one unit each at most
    const long ctas = 2L * a.max_sms;
    launch_pdl(conv_fwd_kernel<kCin, kCout, kLoad>, dim3((unsigned)(units < ctas ? units : ctas)), dim3(kFwdThreads), smem,
               s, a);
    return 1;
}

template <int kCin, int kCout, int kLoad>
static int launch_wgrad_t(const WgradArgs& a, int max_ctas, cudaStream_t s) {
    // Rows of a strip: 4 (1.5 reads of X), fewer where that leaves less than
    // two strips an SM: a 64 x 64 image of 8 has 128 strips of 4 rows.
    const long strips = (long)a.n * ((a.w + kWgPx - 1) / kWgPx);
    int rows = kWgRows;
    while (rows > 1 && strips * ((a.h + rows - 1) / rows) < 2L * max_ctas) rows >>= 1;
    const long total = strips * ((a.h + rows - 1) / rows);
    const size_t smem = 2 * (size_t)wg_stage_bytes(kCin, kCout);
    static bool attr = false;
    if (!attr) {
        cudaFuncSetAttribute(conv_wgrad_kernel<kCin, kCout, kLoad>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem);
        attr = true;
    }
    conv_wgrad_kernel<kCin, kCout, kLoad><<<(unsigned)(total < max_ctas ? total : max_ctas), kWgThreads, smem, s>>>(a, rows);
    return 1;
}

int launch_fwd(int cin, int cout, int load_mode, const ConvArgs& a, cudaStream_t s) {
    if (a.n <= 0 || a.h <= 0 || a.w <= 0) return 0;
    if (load_mode == 0) {
        if (cin == 16 && cout == 32) return launch_fwd_t<16, 32, 0>(a, s);
        if (cin == 32 && cout == 32) return launch_fwd_t<32, 32, 0>(a, s);
        if (cin == 32 && cout == 16) return launch_fwd_t<32, 16, 0>(a, s);
    } else {
        if (cin == 32 && cout == 32) return launch_fwd_t<32, 32, 1>(a, s);
    }
    return -1;
}

int launch_wgrad(int cin, int cout, int load_mode, const WgradArgs& a, int max_ctas, cudaStream_t s) {
    if (a.n <= 0 || a.h <= 0 || a.w <= 0) return 0;
    if (load_mode == 0) {
        if (cin == 16 && cout == 32) return launch_wgrad_t<16, 32, 0>(a, max_ctas, s);
        if (cin == 32 && cout == 32) return launch_wgrad_t<32, 32, 0>(a, max_ctas, s);
        if (cin == 32 && cout == 16) return launch_wgrad_t<32, 16, 0>(a, max_ctas, s);
    } else {
        if (cin == 32 && cout == 32) return launch_wgrad_t<32, 32, 1>(a, max_ctas, s);
    }
    return -1;
}

int launch_pack_weights(const float* w, int cin, int cout, int transposed, uint8_t* image, cudaStream_t s) {
    const int total = 9 * cin * cout;
    pack_weights_kernel<<<(total + 255) / 256, 256, 0, s>>>(w, cin, cout, transposed, image);
    return 1;
}

size_t weight_image_bytes(int cin, int cout) { return (size_t)wimage_bytes(cin, cout); }

}  // namespace conv
}  // namespace gs
