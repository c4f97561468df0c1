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
// y - 1 + ky started kx pixels (kx * 16 bytes) further: no im2col copy.  An MMA
// takes a row for the three output rows it belongs to at once (N = 3 Cout, the
// weights of ky = 2, 1, 0 side by side, the accumulators of consecutive rows
// adjacent in TMEM).  The warps have fixed roles that meet only at mbarriers:
// some load rows, one thread issues MMAs into a ring of 8 TMEM accumulators,
// some read accumulators back (a thread = a TMEM lane = a pixel) for the
// epilogue (bias, ReLU, ReLU mask, bf16 / f32 store).
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

// The forward kernel's warps: 12 that read accumulators back or load rows (see Roles), and the one that multiplies.
constexpr int kMmaWarp = 12;
constexpr int kFwdThreads = (kMmaWarp + 1) * 32;
constexpr int kGroup = 128;                 // threads that load a row, or that read one back
constexpr int kSlots = 8;                   // halo rows in the ring
constexpr int kAhead = 3;                   // rows copied behind the one announced next
constexpr uint32_t kAccs = 8;               // TMEM accumulators of Cout columns
// Barriers of finished rows.  While an accumulator is unread the MMAs stop at
// the first terms of the row kAccs later, and a run of R rows is R + 2 entries:
// past the entry that completes a row, the MMAs can finish 2 kAccs + 5 more
// (runs of one row; 13 in runs of two, 7 in long ones) before that row's reader
// has tested its barrier, which must not complete a second time until then.
constexpr uint32_t kDone = 32;
static_assert(kDone > 2 * kAccs + 5, "a finished row's barrier outlasts its reader's wait");

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
template <int kPending>
__device__ __forceinline__ void cp_async_wait_but() { asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory"); }
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
// One arrival for a warp, behind what all its lanes did before.
__device__ __forceinline__ void mbar_arrive_warp(uint64_t* bar) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
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

// Load mode 1 adds two tensors on the way in, through registers: two groups of
// loading threads take rows in turn and one group runs the epilogues.  Load
// mode 0 copies asynchronously and one group keeps four rows in flight; a layer
// of 32 outputs then has two groups for its epilogues (rows in turn, row pairs
// for the pooled output), one of 16 outputs one (the denoised frame's head
// sums a tile's rows in order).
template <int kCout, int kLoad>
struct Roles {
    static constexpr int kEpiGroups = kLoad == 0 && kCout == 32 ? 2 : 1;
    static constexpr int kLoadGroups = kLoad == 0 ? 1 : 2;
    static constexpr int kFirstLoader = kEpiGroups * kGroup;   // threads
    static_assert(kFirstLoader + kLoadGroups * kGroup <= kMmaWarp * 32, "room for the loaders");
};

// Bound by HBM: every input row of a strip is read once (and 2 more at each
// end of a run), every output written once in 32-byte sectors.  An M = 128, K =
// 16 MMA with both operands in shared memory takes ~50 cycles for N up to 64
// and 59 for N = 96 (its A operand is what it reads), so one MMA for three
// output rows takes a row 7 instead of 18 of them.  1920 x 1080, the layers of the
// denoised frame: 16 -> 32 pooled 61 us, 32 -> 32 at half size 25, 32 -> 32 from two
// inputs 86, 32 -> 16 with the head 80 (99, 46, 164, 94 at one MMA a tap and no
// roles); read and written bytes pass at ~4 TB/s.
template <int kCin, int kCout, int kLoad, bool kPool>
__global__ void __launch_bounds__(kFwdThreads, 2) conv_fwd_kernel(ConvArgs a) {
    static_assert(kCin % 16 == 0 && (kCout == 16 || kCout == 32), "channel counts");
    using R = Roles<kCout, kLoad>;
    constexpr int kG = kCin / 8;                         // 16-byte columns per pixel
    constexpr int kColBytes = col_bytes(kCin);
    constexpr int kSlot = kG * kColBytes;                // one halo row
    constexpr int kW = wimage_bytes(kCin, kCout);
    constexpr int kN = 3 * kCout;                        // columns of the weight image
    extern __shared__ __align__(128) uint8_t smem[];
    uint8_t* s_w = smem + kSlots * kSlot;
    // a row has landed; its MMAs are done (its slot is free and the output row above it complete: one commit, which
    // takes the tensor core ~70 cycles, says both); an accumulator was read
    __shared__ __align__(8) uint64_t s_full[kSlots], s_done[kDone], s_aempty[kAccs];
    __shared__ uint32_t s_taddr;
    __shared__ __align__(16) float s_bias[kCout];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    if (tid == 0) {
        for (int k = 0; k < kSlots; ++k) {
            mbar_init(&s_full[k], kGroup / 32);
        }
        for (uint32_t k = 0; k < kDone; ++k) mbar_init(&s_done[k], 1);
        for (uint32_t k = 0; k < kAccs; ++k) mbar_init(&s_aempty[k], kGroup / 32);
        mbar_fence_init();
    }
    if (warp == kMmaWarp) umma::tmem_alloc(&s_taddr, kAccs * kCout);
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

    if (tid >= R::kFirstLoader && tid < R::kFirstLoader + R::kLoadGroups * kGroup) {
        // ---- load: entries of the ring are the run's rows y0 - 1 .. y1, then the next run's; entry e by
        // group e % kLoadGroups
        const int lt = (tid - R::kFirstLoader) % kGroup;
        const uint32_t group = (uint32_t)((tid - R::kFirstLoader) / kGroup);
        uint32_t e = 0;
        while (!failed && runs.next(r)) {
            for (int yy = r.y0 - 1; yy <= r.y1; ++yy, ++e) {
                if (R::kLoadGroups > 1 && e % R::kLoadGroups != group) continue;
                const uint32_t slot = e % kSlots;
                if (e >= kSlots && !mbar_wait_suspend(&s_done[(e - kSlots) % kDone], ((e - kSlots) / kDone) & 1u)) {
                    failed = true;
                    break;
                }
                uint8_t* dst = smem + slot * kSlot;
                const bool row_in = yy >= 0 && yy < a.h;
                const __nv_bfloat16* rowp = a.x + ((size_t)r.n * a.h + (row_in ? yy : 0)) * a.w * kCin;
                if (kLoad == 0) {
                    // copied asynchronously; announced once kAhead more rows are on their way
                    for (int q = lt; q < 130 * kG; q += kGroup) {
                        const int hp = q / kG, g = q - hp * kG, x = r.x0 - 1 + hp;
                        const bool in = row_in && x >= 0 && x < a.w;
                        cp_async16(dst + g * kColBytes + hp * 16, in ? rowp + (size_t)x * kCin + g * 8 : a.x, in ? 16u : 0u);
                    }
                    cp_async_commit();
                    if (e >= kAhead) {
                        cp_async_wait_but<kAhead>();
                        umma::fence_smem_to_async();
                        mbar_arrive_warp(&s_full[(e - kAhead) % kSlots]);
                    }
                } else {
                    // x + the 2x nearest upsampling of xh (FP32 sum rounded to bf16): all of a
                    // thread's granules loaded before the first is stored
                    constexpr int kPer = (130 * kG + kGroup - 1) / kGroup;
                    const int hh = a.h >> 1, hw = a.w >> 1;
                    const __nv_bfloat16* hrow = a.xh + ((size_t)r.n * hh + (row_in ? min(yy >> 1, hh - 1) : 0)) * hw * kCin;
                    uint4 v[kPer], u[kPer];
#pragma unroll
                    for (int k = 0; k < kPer; ++k) {
                        const int q = lt + k * kGroup, hp = q / kG, g = q - hp * kG, x = r.x0 - 1 + hp;
                        v[k] = u[k] = make_uint4(0u, 0u, 0u, 0u);
                        if (row_in && x >= 0 && x < a.w && q < 130 * kG) {
                            v[k] = __ldg(reinterpret_cast<const uint4*>(rowp + (size_t)x * kCin) + g);
                            u[k] = __ldg(reinterpret_cast<const uint4*>(hrow + (size_t)min(x >> 1, hw - 1) * kCin) + g);
                        }
                    }
#pragma unroll
                    for (int k = 0; k < kPer; ++k) {
                        const int q = lt + k * kGroup, hp = q / kG, g = q - hp * kG;
                        if (q < 130 * kG) *reinterpret_cast<uint4*>(dst + g * kColBytes + hp * 16) = bf16x8_add(v[k], u[k]);
                    }
                    umma::fence_smem_to_async();
                    mbar_arrive_warp(&s_full[slot]);
                }
            }
        }
        if (kLoad == 0) {   // the rows not announced yet
            cp_async_wait_all();
            umma::fence_smem_to_async();
            for (uint32_t k = e > kAhead ? e - kAhead : 0u; k < e; ++k) mbar_arrive_warp(&s_full[k % kSlots]);
        }
    } else if (warp == kMmaWarp) {
        // ---- multiply: the warp in step, one lane issuing
        const uint32_t elected = lane == 0 ? 1u : 0u;
        const uint64_t ad0 = umma::smem_desc(smem_u32(smem), (uint32_t)kColBytes, 128u);
        const uint64_t bd0 = umma::smem_desc(smem_u32(s_w), (uint32_t)(kN * 16), 128u);
        uint32_t e = 0, m = 0;   // ring entry; output rows of earlier runs
        while (!failed && runs.next(r)) {
            const int rows = r.y1 - r.y0;
            for (int i = -1; i <= rows; ++i, ++e) {   // input row y0 + i: output rows i - 1, i, i + 1 of the run
                bool ok = mbar_wait_suspend(&s_full[e % kSlots], (e / kSlots) & 1u);
                const bool fresh = i + 1 < rows;      // row i + 1 gets its first terms
                const uint32_t mf = m + (uint32_t)(i + 1);
                if (ok && fresh && mf >= kAccs) ok = mbar_wait_suspend(&s_aempty[mf % kAccs], (mf / kAccs - 1u) & 1u);
                if (__any_sync(0xffffffffu, !ok)) {
                    failed = true;
                    break;
                }
                umma::fence_after_sync();
                const int lo = max(i - 1, 0), hi = min(i + 1, rows - 1);
                // accumulators p0 .. of the ring for output rows lo .. hi, the weights' columns from block nb
                // (0: ky = 2); the rows past the ring's end are a second MMA
                const uint32_t p0 = (m + (uint32_t)lo) % kAccs, c = (uint32_t)(hi - lo + 1), nb = (uint32_t)(lo - (i - 1));
                const uint64_t ad = ad0 + (uint64_t)((e % kSlots) * (uint32_t)(kSlot >> 4));
                auto mma_rows = [&](int k, uint32_t p, uint32_t rows_n, uint32_t block, uint32_t accumulate) {
                    const int kx = k / (kCin / 16), kb = k % (kCin / 16);
                    umma::mma_bf16_elect(taddr + p * (uint32_t)kCout,
                                         ad + (uint64_t)((2 * kb * kColBytes + kx * 16) >> 4),
                                         bd0 + (uint64_t)(((kx * kCin + kb * 16) >> 3) * kN) + block * (uint32_t)kCout,
                                         umma::idesc_bf16(128, kCout, 0, 0) + ((rows_n - 1u) * (uint32_t)(kCout >> 3) << 17),
                                         accumulate, elected);
                };
                {   // K-step 0: the fresh row's accumulator is written, the others are added to
                    const uint32_t old = fresh ? c - 1u : c, c1 = min(old, kAccs - p0), c2 = old - c1;
                    if (c1) mma_rows(0, p0, c1, nb, 1u);
                    if (c2) mma_rows(0, 0u, c2, nb + c1, 1u);
                    if (fresh) mma_rows(0, mf % kAccs, 1u, 2u, 0u);
                }
                const uint32_t c1 = min(c, kAccs - p0), c2 = c - c1;
#pragma unroll
                for (int k = 1; k < 3 * (kCin / 16); ++k) mma_rows(k, p0, c1, nb, 1u);
                if (c2) {
#pragma unroll
                    for (int k = 1; k < 3 * (kCin / 16); ++k) mma_rows(k, 0u, c2, nb + c1, 1u);
                }
                umma::commit_elect(&s_done[e % kDone], elected);
            }
            m += (uint32_t)rows;
        }
        // every MMA of this CTA, and the last commit's arrival, is done before its shared memory and TMEM go, after a
        // wait that ran out too (entry e then has issued nothing)
        if (e > 0 && !mbar_wait_suspend(&s_done[(e - 1u) % kDone], ((e - 1u) / kDone) & 1u)) failed = true;
        __syncwarp();
    } else if (tid < R::kFirstLoader) {
        // ---- epilogue: thread t of a group holds pixel x0 + t of a row (its TMEM lane: warp % 4)
        const uint32_t group = (uint32_t)(tid / kGroup);
        const int t = tid % kGroup;
        uint32_t m = 0, e = 2;   // output rows; the ring entry whose MMAs complete row m
        float err_sum = 0.0f, err_cnt = 0.0f;   // head mode: this thread's column of the band, in row order
        uint32_t even[kPool ? 16 : 1];          // the bf16 outputs of the even row above (pooled output)
        while (!failed && runs.next(r)) {
            const int x = r.x0 + t;
            const bool in = x < a.w;
            uint4 x_next = make_uint4(0u, 0u, 0u, 0u);
            if (kCout == 16 && a.head_x && in)
                x_next = __ldg(reinterpret_cast<const uint4*>(a.head_x + (((size_t)r.n * a.h + r.y0) * a.w + x) * 16));
            for (int y = r.y0; y < r.y1; ++y, ++m, ++e) {
                if (R::kEpiGroups > 1 && ((m >> (kPool ? 1 : 0)) & 1u) != group) continue;
                const uint32_t acc = m % kAccs;
                const size_t o = ((size_t)r.n * a.h + y) * a.w + x;
                // what the epilogue reads from memory comes while the row is multiplied
                constexpr int kMaskQ = kPool ? 1 : kCout / 8;
                uint4 mask[kMaskQ];
                if (!kPool && a.mask && in) {
#pragma unroll
                    for (int q = 0; q < kMaskQ; ++q) mask[q] = __ldg(reinterpret_cast<const uint4*>(a.mask + o * kCout) + q);
                }
                // (the head's features a row ahead: its rows take the group one after another)
                const uint4 xv = x_next;
                if (kCout == 16 && a.head_x && in && y + 1 < r.y1)
                    x_next = __ldg(reinterpret_cast<const uint4*>(a.head_x + (o + a.w) * 16));
                if (!mbar_wait_suspend(&s_done[e % kDone], (e / kDone) & 1u)) {
                    failed = true;
                    break;
                }
                umma::fence_after_sync();
                const uint32_t acc_addr = taddr + acc * (uint32_t)kCout + ((uint32_t)((warp & 3) * 32) << 16);
                float v[32];
                if (kCout == 32) umma::tmem_ld32(acc_addr, *reinterpret_cast<float(*)[32]>(v));
                else umma::tmem_ld16(acc_addr, *reinterpret_cast<float(*)[16]>(v));
                umma::fence_before_sync();
                mbar_arrive_warp(&s_aempty[acc]);
                if (a.bias) {
                    const float4* sb = reinterpret_cast<const float4*>(s_bias);
#pragma unroll
                    for (int q = 0; q < kCout / 4; ++q) {
                        const float4 b4 = sb[q];
                        const float2 lo = __fadd2_rn(make_float2(v[4 * q], v[4 * q + 1]), make_float2(b4.x, b4.y));
                        const float2 hi = __fadd2_rn(make_float2(v[4 * q + 2], v[4 * q + 3]), make_float2(b4.z, b4.w));
                        v[4 * q] = lo.x;
                        v[4 * q + 1] = lo.y;
                        v[4 * q + 2] = hi.x;
                        v[4 * q + 3] = hi.y;
                    }
                }
                if (kCout == 16 && a.head_x && in) {
                    // the denoised frame's pixel (head_rgba of the output step) and its error estimate
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
                if (!kPool && a.out_f32 && in) {
                    float4* op = reinterpret_cast<float4*>(a.out_f32 + o * kCout);
#pragma unroll
                    for (int q = 0; q < kCout / 4; ++q) {
                        float f[4] = {v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]};
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            if (a.relu) f[i] = fmaxf(f[i], 0.0f);
                            if (a.mask) {
                                const __nv_bfloat16* mb = reinterpret_cast<const __nv_bfloat16*>(&mask[q >> 1]);
                                if (!(__bfloat162float(mb[4 * (q & 1) + i]) > 0.0f)) f[i] = 0.0f;
                            }
                        }
                        op[q] = make_float4(f[0], f[1], f[2], f[3]);
                    }
                }
                if (a.out_bf16 || kPool) {
                    uint32_t pk[kCout / 2];
#pragma unroll
                    for (int i = 0; i < kCout / 2; ++i) {
                        // ReLU and mask on the rounded pairs: rounding keeps the sign and zero
                        __nv_bfloat162 b2 = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
                        if (a.relu) b2 = __hmax2(b2, __floats2bfloat162_rn(0.0f, 0.0f));
                        pk[i] = *reinterpret_cast<uint32_t*>(&b2);
                        if (!kPool && a.mask)
                            pk[i] &= __hgt2_mask(reinterpret_cast<const __nv_bfloat162*>(&mask[i >> 2])[i & 3],
                                                 __floats2bfloat162_rn(0.0f, 0.0f));
                    }
                    if (in) {
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
                    if constexpr (kPool) {
                        // 2x2 average of the bf16 outputs: (0 + (y, x) + (y, x + 1) + (y + 1, x) + (y + 1, x + 1)) * 0.25,
                        // the right neighbour's by lane shuffles (runs hold whole row pairs)
                        if ((y & 1) == 0) {
#pragma unroll
                            for (int i = 0; i < 16; ++i) even[i] = pk[i];
                        } else {
                            const bool write = (x & 1) == 0 && in;
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
                }
                if (kCout == 16 && a.head_x && (y + 1 == r.y1 || (y + 1 + a.row_offset) % 16 == 0)) {
                    // end of a band: per tile (16 threads = 16 columns) the sum of the error estimates and the
                    // pixel count, each over 16 lanes in a fixed order, then the tile's mean
#pragma unroll
                    for (int off = 8; off; off >>= 1) {
                        err_sum += __shfl_xor_sync(0xffffffffu, err_sum, off);
                        err_cnt += __shfl_xor_sync(0xffffffffu, err_cnt, off);
                    }
                    const int tx = (r.x0 >> 4) + (t >> 4);
                    if ((t & 15) == 0 && tx < a.tiles_x && err_cnt > 0.0f) {
                        const int band = (y + a.row_offset) / 16;
                        const int ty = (a.h + a.row_offset) / 16 - 1 - band;   // GL tile row of this band
                        const uint32_t tile = (uint32_t)(ty * a.tiles_x + tx);
                        const float mse = err_sum / err_cnt * 0.001f;
                        a.tile_err[tile] = mse;
                        if (mse >= a.err_budget) atomicAdd(a.fallback_count, 1u);
                    }
                    err_sum = err_cnt = 0.0f;
                }
            }
            e += 2u;
        }
    }
    if (failed) atomicOr(a.err, 1u);
    umma::fence_before_sync();
    __syncthreads();
    if (warp == kMmaWarp) {
        umma::fence_after_sync();
        umma::tmem_dealloc(taddr, kAccs * kCout);
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
// wait between them.  Eight warps copy and sum the bias gradient from the staged
// dY; a ninth issues the MMAs, which a copying warp did before, holding up its
// own copies.  The strips pass at ~115 cycles an MMA, more loading warps or
// less issue work change nothing, and an aligned operand takes ~50: presumably the
// reads of tap kx, whose operand starts kx x 16 bytes off a 128-byte line.  8 x 256 x 256
// pixels, 32 -> 16, 32 -> 32 (load mode 1) and 16 -> 32 channels: 41 / 59 / 41 us;
// 52 / 106 / 53 with the MMAs on a copying warp and one granule of mode 1 loaded at
// a time, 262 (mode 1) when every tap was gathered from global memory and
// nothing overlapped.  16 copying warps: 44 / 56 / 46.
constexpr int kWgThreads = 256;   // that copy and sum; one more warp multiplies
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
__global__ void __launch_bounds__(kWgThreads + 32) conv_wgrad_kernel(WgradArgs a, int rows) {
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
    for (int i = tid; i < 2 * kStage / 16; i += kWgThreads + 32) reinterpret_cast<uint4*>(smem)[i] = make_uint4(0u, 0u, 0u, 0u);
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t taddr = s_taddr, base = smem_u32(smem);
    const int strips_x = (a.w + kWgPx - 1) / kWgPx, bands = (a.h + rows - 1) / rows;
    const int total = a.n * bands * strips_x;

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
        for (int r = 0; kLoad == 0 && r < s.rows + 2; ++r) {
            const int y = s.y0 - 1 + r;
            {
                const bool row_in = y >= 0 && y < a.h;
                const __nv_bfloat16* rowp = a.x + ((size_t)s.n * a.h + (row_in ? y : 0)) * a.w * kCin;
                for (int q = tid; q < row_q; q += kWgThreads) {
                    const int hp = q / kG, g = q % kG, x = s.x0 - 1 + hp;
                    const bool in = row_in && x >= 0 && x < a.w;
                    cp_async16(xs + r * kSlot + g * kCol + hp * 16, in ? rowp + (size_t)x * kCin + g * 8 : a.x,
                               in ? 16u : 0u);
                }
            }
        }
        if (kLoad == 1) {
            // two rows at a time, all of a thread's granules loaded before the first is stored
            constexpr int kPer = ((kWgPx + 2) * kG + kWgThreads - 1) / kWgThreads;
            const int hh = a.h >> 1, hw = a.w >> 1;
            for (int r0 = 0; r0 < s.rows + 2; r0 += 2) {
                uint4 v[2][kPer], u[2][kPer];
#pragma unroll
                for (int d = 0; d < 2; ++d) {
                    const int y = s.y0 - 1 + r0 + d;
                    const bool row_in = r0 + d < s.rows + 2 && y >= 0 && y < a.h;
                    const size_t row = ((size_t)s.n * a.h + (row_in ? y : 0)) * a.w;
                    const size_t hrow = ((size_t)s.n * hh + (row_in ? min(y >> 1, hh - 1) : 0)) * hw;
#pragma unroll
                    for (int k = 0; k < kPer; ++k) {
                        const int q = tid + k * kWgThreads, hp = q / kG, g = q % kG, x = s.x0 - 1 + hp;
                        v[d][k] = u[d][k] = make_uint4(0u, 0u, 0u, 0u);
                        if (row_in && q < row_q && x >= 0 && x < a.w) {
                            v[d][k] = __ldg(reinterpret_cast<const uint4*>(a.x + (row + x) * kCin) + g);
                            u[d][k] = __ldg(reinterpret_cast<const uint4*>(a.xh + (hrow + min(x >> 1, hw - 1)) * kCin) + g);
                        }
                    }
                }
#pragma unroll
                for (int d = 0; d < 2; ++d)
#pragma unroll
                    for (int k = 0; k < kPer; ++k) {
                        const int q = tid + k * kWgThreads, hp = q / kG, g = q % kG;
                        if (r0 + d < s.rows + 2 && q < row_q)
                            *reinterpret_cast<uint4*>(xs + (r0 + d) * kSlot + g * kCol + hp * 16) =
                                bf16x8_add(v[d][k], u[d][k]);
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
    const bool multiplies = warp == kWgThreads / 32;   // the last warp; the others load and sum
    const uint32_t elected = lane == 0 ? 1u : 0u;
    if (!multiplies && (int)blockIdx.x < total) load(0, blockIdx.x);
    for (int item = blockIdx.x; item < total; item += gridDim.x, stage ^= 1) {
        asm volatile("cp.async.wait_all;" ::: "memory");   // this strip, copied while the last one was multiplied
        umma::fence_smem_to_async();
        if (__syncthreads_or(failed)) {
            failed = true;
            break;
        }
        const Strip s = strip_at(item);
        if (multiplies) {
            umma::fence_after_sync();
            const uint32_t xa = base + (uint32_t)(stage * kStage), da = xa + (uint32_t)kX;
            const uint64_t ad0 = umma::smem_desc(xa, 128u, (uint32_t)kCol), bd0 = umma::smem_desc(da, 128u, (uint32_t)kDcol);
            const int steps = s.px / 16;
            for (int r = 0; r < s.rows; ++r) {
                uint64_t ad = ad0 + (uint64_t)((r * kSlot) >> 4), bd = bd0 + (uint64_t)((r * kDrow) >> 4);
                for (int kk = 0; kk < steps; ++kk, ad += 16, bd += 16)
#pragma unroll
                    for (int kx = 0; kx < 3; ++kx)
                        umma::mma_bf16_elect(taddr + (uint32_t)(kx * kCout), ad + (uint64_t)kx, bd, kIdesc,
                                             (any || r + kk > 0) ? 1u : 0u, elected);
            }
            umma::commit_elect(&s_bar[stage], elected);
        }
        if (a.db && !multiplies) {   // pixels past the row are zero
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
        if (next < total && !multiplies) {
            // the other stage: its MMAs (the previous strip's) read it to the end, and every
            // thread is past its sum over it (the barrier above)
            if (any) {
                if (!mbar_wait_bounded(&s_bar[stage ^ 1], phase[stage ^ 1], kWaitLimit)) failed = true;
                phase[stage ^ 1] ^= 1u;
            }
            if (!failed) load(stage ^ 1, next);   // else those MMAs may still read it
        }
        any = true;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (any && !multiplies) {   // the last strip's MMAs complete after all earlier ones; also after a wait that ran out
        if (!mbar_wait_bounded(&s_bar[stage ^ 1], phase[stage ^ 1], kWaitLimit)) failed = true;
    }
    if (__syncthreads_or(failed)) failed = true;
    umma::fence_after_sync();
    if (any && !failed && !multiplies) {
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
            if (lane < kGo && !multiplies) s_db[warp][lane * 8 + e] = db[e];
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
        const int at = transposed ? wimage_offset(8 - tap, co, ci, cout, cin) : wimage_offset(tap, ci, co, cin, cout);
        *reinterpret_cast<__nv_bfloat16*>(image + at) = __float2bfloat16_rn(w[i]);
    }
}

static int current_device() {
    int dev = -1;
    cudaGetDevice(&dev);
    return dev;
}

template <int kCin, int kCout, int kLoad, bool kPool = false>
static int launch_fwd_t(ConvArgs a, cudaStream_t s) {
    const long strips = (long)a.n * ((a.w + 127) / 128);
    const long units = strips * ((a.h + a.row_offset + a.unit_rows - 1) / a.unit_rows);
    const size_t smem = (size_t)fwd_smem_bytes(kCin, kCout);
    a.out_wide = (reinterpret_cast<uintptr_t>(a.out_bf16) & 31u) == 0u ? 1 : 0;
    static OncePerDevice attr;
    attr(current_device(), [&] {
        cudaFuncSetAttribute(conv_fwd_kernel<kCin, kCout, kLoad, kPool>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem);
    });
    // two CTAs an SM; on small images one unit each at most
    const long ctas = 2L * a.max_sms;
    launch_pdl(conv_fwd_kernel<kCin, kCout, kLoad, kPool>, dim3((unsigned)(units < ctas ? units : ctas)), dim3(kFwdThreads), smem,
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
    static OncePerDevice attr;
    attr(current_device(), [&] {
        cudaFuncSetAttribute(conv_wgrad_kernel<kCin, kCout, kLoad>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem);
    });
    conv_wgrad_kernel<kCin, kCout, kLoad><<<(unsigned)(total < max_ctas ? total : max_ctas), kWgThreads + 32, smem, s>>>(a, rows);
    return 1;
}

int launch_fwd(int cin, int cout, int load_mode, const ConvArgs& a, cudaStream_t s) {
    if (a.n <= 0 || a.h <= 0 || a.w <= 0) return 0;
    if (load_mode == 0) {
        if (cin == 16 && cout == 32 && a.pool_out) return launch_fwd_t<16, 32, 0, true>(a, s);
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
