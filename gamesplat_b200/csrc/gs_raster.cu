// Tile rasterizer: replaces the reference's GL instanced-quad draw, fragment
// shader and fixed-function blender (shaders/splat.glsl:39-145,
// src/renderer.cpp:266-320, 1687-1720).
//
// One CTA per 16x16 pixel tile, two pixels per thread, each warp an 8x8 pixel
// block (GL window coordinates, row 0 at the bottom; the image is written
// top row first).  Control flow is warp-uniform: lanes never diverge around
// the per-splat loop (per-pixel work is predicated or selected), a warp skips
// splats whose rectangle misses its block and leaves the loop when all its
// pixels are done.  The tile's splat list (descending sorted position) is
// walked front to back (reverse of the reference's back-to-front draw order,
// so equal depth keys are visited in descending splat index, which
// reproduces "later instance on top").  Batches of 128 64-byte RasterRecords
// are gathered into shared memory by cp.async, 16 bytes a lane, double buffered
// so the next batch lands while the current one is composited.  (One TMA bulk
// copy a record is one instruction where this takes four, but the copy engine of
// an SM works off some one every 11 cycles, and that was what the rasterizers
// waited for: 250 us against 210 us for 3M Gaussians in the room at 1080p, 644
// against 531 us for 6M at 2160p.)  When a batch lands, one thread per record
// turns its pixel rectangle into tile-relative column and row bit masks, written
// into the staged record next to g, b, so a pixel's coverage test is one
// operation; drops the 8x8 blocks that its ellipse cannot reach; and each warp
// lists the records it has to shade.
//
// The two pixels of a thread share a column; their arithmetic runs as packed
// f32x2 operations (add/mul/fma .rn on float pairs, each element rounded like
// the scalar operation), which halves the issue slots of the per-pixel math.
// CTA b rasterizes tile
// tile_order[b]: the heaviest tiles first, so they do not form the last wave.
//
// Alpha mode: premultiplied "over" in FP32, front to back:
//   C += T * alpha * rgb,  T -= T * alpha,  output (C + T*bg, 1 - T),
// which equals the reference's back-to-front ONE / ONE_MINUS_SRC_ALPHA
// blend into a (bg,bg,bg,0) target up to FP32 rounding.  A warp stops once
// T < 2^-13 for all its pixels: the skipped remainder is below T * max(rgb, bg).
// Coverage (quad rectangle) and the two discards (power > 0, power < cutoff)
// are evaluated bit-exactly like the CPU oracle, on the quadratic form s with
// the bounds of RasterRecord; alpha = min(2^(s * -0.5 log2(e) + log2(opacity)),
// 0.99) uses the hardware exp2.
//
// Two-sample mode (the input of the denoised mode): the stochastic sample
// rule below for two seeds at once, on un-jittered records (the alpha
// binning), alpha evaluated once per (pixel, splat) and hashed per seed; a
// pixel stops when both samples are decided.  Writes the mean colour of the
// two samples (background where none kept), the fraction that kept a
// fragment and the mean window depth (1 where none kept), all in float.
//
// Stochastic mode: a fragment is kept iff hash13(fragcoord, id + seed) <
// alpha; the depth test (LESS, writes on) keeps the kept fragment with the
// smallest (D24 depth, instance index).  Walking front to back, a warp stops
// once a splat's D24 exceeds the kept ones of all its pixels by more than 8 (the
// float depth-to-D24 mapping is monotone to within 5 units, so a pixel whose
// kept depth was exceeded by 8 keeps nothing of a later splat either).  Deterministic exp and
// hash, so the kept set matches the oracle bit for bit.
#include <cuda_fp16.h>

#include <type_traits>

#include "gs_common.cuh"
#include "gs_copy.cuh"
#include "gs_internal.h"

namespace gs {

constexpr int kRasterThreads = kTileW * kTileH / 2;   // two pixels per thread
constexpr int kBatch = 128;
constexpr float kTransmittanceMin = 1.0f / 8192.0f;
constexpr uint32_t kDepthMargin = 8;
constexpr float kNegHalfLog2e = -0.72134752044448170368f;   // -0.5 / ln(2)

// hash13(x, y, z) (shaders/splat.glsl:121-125), split by what its terms
// depend on: p0 = fract(0.1031 x), p1 = fract(0.1031 y) and the products that
// hold only them belong to the pixel (computed once per tile), p2 =
// fract(0.1031 z) to the splat and sample (once per splat for all the pixels of
// a warp); the rest, per (pixel, splat, sample), is the same operations in the
// same order:  d = p0 (p1 + 33.33) + p1 (p2 + 33.33) + p2 (p0 + 33.33),
// hash = fract((p0 + d + p1 + d) (p2 + d)).
struct PixelHash {
    float p0, p1, t1, p0c;   // p0, p1, p0 (p1 + 33.33), p0 + 33.33
};

__device__ __forceinline__ PixelHash pixel_hash(float x, float y) {
    PixelHash h;
    h.p0 = g_fract(mul(x, 0.1031f));
    h.p1 = g_fract(mul(y, 0.1031f));
    h.t1 = mul(h.p0, add(h.p1, 33.33f));
    h.p0c = add(h.p0, 33.33f);
    return h;
}

// Both pixels of a thread (they share a column, hence p0): the same operations
// in the same order, two to an instruction.
struct PixelHash2 {
    float p0, p0c;
    float2 p1, t1;
};

__device__ __forceinline__ float hash_z(float z) { return g_fract(mul(z, 0.1031f)); }

__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float2 f2(float x) { return make_float2(x, x); }

// The multiplications stay scalar: a packed one is contracted with the packed
// addition of its result (whatever -fmad says), which the hash does not stand.
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return make_float2(mul(a.x, b.x), mul(a.y, b.y)); }

__device__ __forceinline__ float2 hash13(const PixelHash2& h, float p2) {
    const float m = mul(p2, h.p0c);
    const float2 d = __fadd2_rn(__fadd2_rn(h.t1, mul2(h.p1, f2(add(p2, 33.33f)))), f2(m));
    const float2 x = mul2(__fadd2_rn(__fadd2_rn(f2(h.p0), d), __fadd2_rn(h.p1, d)), __fadd2_rn(f2(p2), d));
    return make_float2(g_fract(x.x), g_fract(x.y));
}

// Fragment tests of one pixel: covered (all bits it needs are among the
// record's) and 0 <= s <= s_max, as one unsigned comparison (a negative s has
// the top bit set, a NaN compares above s_max).  The bounds of RasterRecord
// also admit s = -0 and the negative subnormal of the last place; s, a sum of
// conic_x dx^2 >= +0, a product and conic_z dy^2 >= +0, never is -0, and is that
// subnormal only if all terms are below 2^-125, a splat of sigma above 2^38
// pixels.  These tests are the loop's comparisons, on the rasterizers' busiest
// pipe, the ALU's (64 % before them): 310 -> 287 us for the alpha frame of
// raster_kernel.
template <class M>
__device__ __forceinline__ bool frag_live(M bits, M need, float s, float s_max) {
    return (need & ~bits) == (M)0 && __float_as_uint(s) <= __float_as_uint(s_max);
}

// The kept fragment of one (pixel, sample); best_id 0xFFFFFFFF (beyond every
// index) and the far plane's D24 while there is none.
struct StochState {
    uint32_t best_d24, best_id;
    float r, g, b;
};

constexpr uint32_t kFarD24 = 16777215u;

__device__ __forceinline__ void write_pixel_stoch2(const RasterParams& p, int px, int py, const StochState (&S)[2]) {
    const size_t o = (size_t)(p.height - 1 - py) * p.width + px;
    float c[2][3], a[2], d[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const bool kept = S[k].best_id != 0xFFFFFFFFu;
        c[k][0] = kept ? S[k].r : p.bg;
        c[k][1] = kept ? S[k].g : p.bg;
        c[k][2] = kept ? S[k].b : p.bg;
        a[k] = kept ? 1.0f : 0.0f;
        d[k] = __fdiv_rn((float)S[k].best_d24, 16777215.0f);
    }
    p.out_rgba32f[o] = make_float4(mul(add(c[0][0], c[1][0]), 0.5f), mul(add(c[0][1], c[1][1]), 0.5f),
                                   mul(add(c[0][2], c[1][2]), 0.5f), mul(add(a[0], a[1]), 0.5f));
    p.out_depth[o] = mul(add(d[0], d[1]), 0.5f);
}

__device__ __forceinline__ void write_rgba16f(uint16_t* out, size_t o, float r, float g, float b, float a) {
    __half2 h01 = __floats2half2_rn(r, g), h23 = __floats2half2_rn(b, a);
    uint2 packed;
    packed.x = *reinterpret_cast<uint32_t*>(&h01);
    packed.y = *reinterpret_cast<uint32_t*>(&h23);
    reinterpret_cast<uint2*>(out)[o] = packed;
}

__device__ __forceinline__ void write_pixel_stoch(const RasterParams& p, int px, int py, const StochState& S) {
    const size_t o = (size_t)(p.height - 1 - py) * p.width + px;
    float4 c;
    if (S.best_id == 0xFFFFFFFFu) c = make_float4(p.bg, p.bg, p.bg, 0.0f);
    else c = make_float4(S.r, S.g, S.b, 1.0f);
    if (p.rgba8) {
        c.x = rintf(g_clamp(c.x, 0.0f, 1.0f) * 255.0f) / 255.0f;
        c.y = rintf(g_clamp(c.y, 0.0f, 1.0f) * 255.0f) / 255.0f;
        c.z = rintf(g_clamp(c.z, 0.0f, 1.0f) * 255.0f) / 255.0f;
        c.w = rintf(g_clamp(c.w, 0.0f, 1.0f) * 255.0f) / 255.0f;
    }
    if (p.out_rgba32f) p.out_rgba32f[o] = c;
    if (p.out_depth) p.out_depth[o] = (float)S.best_d24 / 16777215.0f;
    if (p.accum_out) {   // the frame's running mean, as accum_kernel computes it from the sample
        const float nn = g_max(p.accum_n, 1.0f);
        const float4 h = p.accum_in ? p.accum_in[o] : c;
        p.accum_out[o] = make_float4(add(h.x, dv(sub(c.x, h.x), nn)), add(h.y, dv(sub(c.y, h.y), nn)),
                                     add(h.z, dv(sub(c.z, h.z), nn)), add(h.w, dv(sub(c.w, h.w), nn)));
    }
    if (p.out_rgba16f) write_rgba16f(p.out_rgba16f, o, c.x, c.y, c.z, c.w);
}

// Tile shapes: kTw x kTh pixels, four 8x8 warp blocks (16x16, 32x8, 8x32).
// Coverage masks: column bits from bit 0, row bits from bit RowShift (16 for
// 16x16 tiles, whose masks fit 32 bits; 32 for the others, in 64 bits).
template <int kTw, int kTh>
struct TileShape {
    static_assert(kTw * kTh == 256 && kTw % 8 == 0 && kTh % 8 == 0, "four 8x8 blocks");
    static constexpr int kBx = kTw / 8;          // blocks per row
    static constexpr int kRowShift = kTw == 16 && kTh == 16 ? 16 : 32;
    using Mask = typename std::conditional<kRowShift == 16, uint32_t, unsigned long long>::type;
};

// Tile-relative coverage of a record's pixel rectangle: column bits
// [0, kTw), row bits [RowShift, RowShift + kTh) (bit k = tile column / GL row
// k).  Empty rectangles give 0.
template <int kTw, int kTh>
__device__ __forceinline__ typename TileShape<kTw, kTh>::Mask rect_bits(uint32_t rect_x, uint32_t rect_y, int x0,
                                                                        int y0) {
    using S = TileShape<kTw, kTh>;
    using M = typename S::Mask;
    const int i0 = min(max((int)(rect_x & 0xFFFFu) - x0, 0), kTw), i1 = min(max((int)(rect_x >> 16) - x0, 0), kTw);
    const int j0 = min(max((int)(rect_y & 0xFFFFu) - y0, 0), kTh), j1 = min(max((int)(rect_y >> 16) - y0, 0), kTh);
    if (i1 <= i0 || j1 <= j0) return (M)0;
    const unsigned long long cols = (1ull << i1) - (1ull << i0);
    const unsigned long long rows = (1ull << j1) - (1ull << j0);
    return (M)(cols | (rows << S::kRowShift));
}

// Minimum of the splat's quadratic form q(d) = A dx^2 + B dx dy + C dy^2 (A, C > 0)
// over the box [X0,X1] x [Y0,Y1] of pixel-centre offsets, or more where that
// is above every value in [0, inf) that q takes there: q(t d) = t^2 q(d), so a point of
// the box with such a value has one no larger on an edge that faces the
// origin, and along an edge q is convex with its minimum at the clamped
// stationary point.  X and Y are those edges' coordinates; a box that spans an
// axis gives an inner line instead, one that holds the origin gives q(0) = 0.
// ia = -B / 2A, ic = -B / 2C.
__device__ __forceinline__ float min_q_box(float A, float B, float C, float ia, float ic, float X0, float X1, float Y0,
                                           float Y1) {
    const float X = fminf(fmaxf(0.0f, X0), X1), Y = fminf(fmaxf(0.0f, Y0), Y1);
    const float dy = fminf(fmaxf(ic * X, Y0), Y1), dx = fminf(fmaxf(ia * Y, X0), X1);
    return fminf(fmaf(fmaf(C, dy, B * X), dy, A * X * X), fmaf(fmaf(A, dx, B * Y), dx, C * Y * Y));
}

// One CTA of 128 threads per 16x16 tile; warp w owns the 8x8 block
// (w & 1, w >> 1); lane l shades pixels (l & 7, l >> 3) and (l & 7, (l >> 3) + 4)
// of it: the two pixels share a column, hence dx, the column test and the
// first term of the Gaussian exponent.
// Shared memory of one CTA's tile: two staging buffers of records, the records'
// warp-block masks and the warps' lists.
// A staged record and 16 bytes of padding: at an 80-byte stride the 16-byte
// loads of 8 consecutive records (one record per thread in the staging pass)
// fall in distinct banks, and a 32-bit field of 32 consecutive records spreads
// over 8 banks instead of 2.
struct __align__(16) StagedRecord {
    RasterRecord r;
    uint4 pad;
};

// State batches (kStates > 0): the colours of kStates frames of one geometry
// per record, channel by channel, staged beside the record.
template <int kStates>
struct StateColours {
    static constexpr int kQuads = 3 * kStates / 4;
    float4 col[2][kBatch][kQuads];
};
template <>
struct StateColours<0> {};

template <int kMode, int kTw = 16, int kTh = 16, int kStates = 0>
struct __align__(128) RasterShared : StateColours<kStates> {
    StagedRecord rec[2][kBatch];
    uint8_t mask[kBatch];
    // per warp the staged records it shades, as byte offsets from the first, nearest first
    __align__(16) uint16_t list[4][kBatch];
};

// One 16x16 tile, the whole CTA (used by the per-frame kernel, one tile per
// CTA, and by the batch kernel, many frames' tiles per CTA in turn).
// kStates > 0 (alpha): kStates frames that share geometry, order and alpha and
// differ in colour; the coverage, the exponential and the transmittance of a
// (pixel, splat) pair are evaluated once for all of them.
template <int kMode, int kTw = 16, int kTh = 16, int kStates = 0>  // kMode: 0 alpha, 1 stochastic, 2 two samples
__device__ __forceinline__ void raster_tile(const RasterParams& p, const uint32_t tile,
                                            RasterShared<kMode, kTw, kTh, kStates>& sh,
                                            uint16_t* const* outs = nullptr) {
    using Shape = TileShape<kTw, kTh>;
    using Mask = typename Shape::Mask;
    constexpr int kRs = Shape::kRowShift;
    static_assert(kMode == 0 || (kTw == 16 && kTh == 16), "the stochastic modes rasterize 16x16 tiles");
    const int tx = (int)(tile % (uint32_t)p.tiles_x), ty = (int)(tile / (uint32_t)p.tiles_x);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int x0 = tx * kTw, y0 = ty * kTh;
    const int lx = (warp % Shape::kBx) * 8 + (lane & 7), ly0 = (warp / Shape::kBx) * 8 + (lane >> 3), ly1 = ly0 + 4;
    const int px = x0 + lx, py0 = y0 + ly0, py1 = y0 + ly1;
    const bool in0 = px < p.width && py0 < p.height, in1 = px < p.width && py1 < p.height;
    // coverage bits a pixel needs: its tile column and its tile row
    const Mask need0 = ((Mask)1 << lx) | ((Mask)1 << (kRs + ly0)), need1 = ((Mask)1 << lx) | ((Mask)1 << (kRs + ly1));
    const uint2 range = p.tile_ranges[tile];
    const uint32_t n = range.y > range.x ? range.y - range.x : 0u;
    const uint32_t* __restrict__ vals = p.tile_plan->vfinal;

    const float fcx = (float)px + 0.5f, fcy0 = (float)py0 + 0.5f, fcy1 = (float)py1 + 0.5f;
    const float2 fcy = make_float2(fcy0, fcy1);
    // the stochastic modes' hash terms of the two pixels
    PixelHash2 pixh;
    if (kMode != 0) {
        const PixelHash a0 = pixel_hash(fcx, fcy0), a1 = pixel_hash(fcx, fcy1);
        pixh.p0 = a0.p0;
        pixh.p0c = a0.p0c;
        pixh.p1 = make_float2(a0.p1, a1.p1);
        pixh.t1 = make_float2(a0.t1, a1.t1);
    }
    // alpha state of the two pixels (x: pixel 0, y: pixel 1); pixels outside
    // the image start "done" (T = 0) and are never written
    float2 T = make_float2(in0 ? 1.0f : 0.0f, in1 ? 1.0f : 0.0f);
    float2 C0 = f2(0.0f), C1 = f2(0.0f), C2 = f2(0.0f);
    // state batches: per pixel and channel the frames' colours in pairs
    float2 CS[kStates ? 2 : 1][3][kStates ? kStates / 2 : 1];
    if (kStates)
#pragma unroll
        for (int k = 0; k < 3 * (kStates ? kStates / 2 : 1); ++k) (&CS[0][0][0])[k] = (&CS[kStates ? 1 : 0][0][0])[k] = f2(0.0f);
    // stochastic state of the pixels, per sample; pixels outside the image start
    // with nothing left to find and are never written
    constexpr int kSeeds = kMode == 2 ? 2 : 1;
    StochState S0[2], S1[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        S0[k] = {in0 ? kFarD24 : 0u, 0xFFFFFFFFu, 0.0f, 0.0f, 0.0f};
        S1[k] = {in1 ? kFarD24 : 0u, 0xFFFFFFFFu, 0.0f, 0.0f, 0.0f};
    }
    uint32_t last_z = 0;   // D24 of the last splat this warp went through
    const uint32_t nb = (n + kBatch - 1) / kBatch;

    // A warp copies the 32 records of a batch that it stages, 4 lanes a record
    // (16 bytes each); the list entries of the next batch are loaded a batch ahead.
    static_assert(kBatch == kRasterThreads, "one record a thread in the staging pass");
    auto entry = [&](uint32_t b) -> uint32_t {
        const uint32_t i = b * kBatch + threadIdx.x;
        return i < n ? min(vals[range.x + i], p.record_cap - 1u) : 0u;
    };
    uint32_t ahead = entry(0);
    auto issue = [&](uint32_t b) {
        const uint32_t cnt = min((uint32_t)kBatch, n - b * kBatch);
        const uint32_t mine = ahead;
        ahead = entry(b + 1);
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) {
            const uint32_t r = 8 * j + (lane >> 2), i = warp * 32 + r;
            const uint32_t s = __shfl_sync(0xffffffffu, mine, r);
            if (i < cnt)
                cp_async16(reinterpret_cast<uint4*>(&sh.rec[b & 1][i].r) + (lane & 3),
                           reinterpret_cast<const uint4*>(p.records + s) + (lane & 3));
        }
        if constexpr (kStates > 0) {
            constexpr uint32_t kQ = 3 * kStates / 4;   // 16-byte pieces of a record's colours
#pragma unroll
            for (uint32_t j = 0; j < kQ; ++j) {
                const uint32_t r = (32 * j + lane) / kQ, q = (32 * j + lane) % kQ, i = warp * 32 + r;
                const uint32_t s = __shfl_sync(0xffffffffu, mine, r);
                if (i < cnt) cp_async16(&sh.col[b & 1][i][q], p.colours + (size_t)s * kQ + q);
            }
        }
    };
    auto pixels_done = [&]() -> bool {
        if (kMode == 0) return fmaxf(T.x, T.y) < kTransmittanceMin;
        // a pixel's samples are decided once splats are beyond their kept depths
        // (+ margin): no later one passes the depth test
        uint32_t far = max(S0[0].best_d24, S1[0].best_d24);
        if (kMode == 2) far = max(far, max(S0[1].best_d24, S1[1].best_d24));
        return last_z > far + kDepthMargin;
    };

    if (nb > 0) issue(0);
    cp_async_commit();
    for (uint32_t b = 0; b < nb; ++b) {
        if (b + 1 < nb) issue(b + 1);
        cp_async_commit();
        cp_async_wait<1>();
        __syncwarp();
        const uint32_t cnt = min((uint32_t)kBatch, n - b * kBatch);
        const StagedRecord* recs = sh.rec[b & 1];
        // Coverage bits of each staged record and which of the four 8x8 warp
        // blocks it can shade (one thread per record): blocks its rectangle
        // touches, minus those where the splat's ellipse q(d) <= s_max misses
        // every covered pixel centre (tested with a 2 % + 0.02 margin over
        // s_max, far above the rounding of q and of the exact per-pixel sum).
        if (const uint32_t i = threadIdx.x; i < cnt) {
            const RasterRecord* R = &recs[i].r;
            const uint2 rr = reinterpret_cast<const uint2*>(R)[5];
            Mask bits;
            float cen_x, cen_y;
            if (kMode == 1) {
                // envelope record: this sample's quad (same computation as
                // the per-sample binning of the oracle) and jittered centre
                PixelRect q;
                const bool qok = quad_rect(R->cx, R->cy, R->log2_opacity, __uint_as_float(rr.y), __uint_as_float(rr.x),
                                           p.jitter_x, p.jitter_y, p.vp_w, p.vp_h, p.clip_y_sign, p.width, p.height,
                                           &q);
                bits = qok ? rect_bits<kTw, kTh>((uint32_t)q.i0 | ((uint32_t)q.i1 << 16),
                                                 (uint32_t)q.j0 | ((uint32_t)q.j1 << 16), x0, y0)
                           : (Mask)0;
                cen_x = add(R->cx, p.jitter_x);
                cen_y = add(R->cy, p.jitter_y);
            } else {
                bits = rect_bits<kTw, kTh>(rr.x, rr.y, x0, y0);
                cen_x = R->cx;
                cen_y = R->cy;
            }
            {
                // what the loop wants of the record, in place: the coverage bits next to
                // g, b and, in the stochastic modes, the sample's centre, the hash terms of
                // the splat and the bound of alpha (once a record here, not once a warp)
                RasterRecord* W = const_cast<RasterRecord*>(R);
                W->rect_x = (uint32_t)bits;
                if (kRs == 32) W->rect_y = (uint32_t)((unsigned long long)bits >> 32);
                if (kMode == 1) {
                    W->cx = cen_x;
                    W->cy = cen_y;
                }
                if (kMode != 0) {
                    const float id = (float)R->splat_id;
                    W->log2_opacity = hash_z(add(id, p.frame_seed));
                    if (kMode == 2) W->hash_z = hash_z(add(id, p.frame_seed2));
                    W->rect_y = __float_as_uint(g_min(R->opacity, 0.99f));
                }
            }
            // block w = (w % kBx, w / kBx): bit w set iff its 8 columns and 8 rows are covered
            uint32_t blocks = 0u;
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                const int bxw = w % Shape::kBx, byw = w / Shape::kBx;
                if (((bits >> (8 * bxw)) & 0xFFu) != 0u && ((bits >> (kRs + 8 * byw)) & 0xFFu) != 0u) blocks |= 1u << w;
            }
            const float4 q0 = reinterpret_cast<const float4*>(R)[0];
            const float2 q1 = reinterpret_cast<const float2*>(R)[2];
            const float A = q0.z, B = q0.w, C = q1.x;
            if (blocks && A > 0.0f && C > 0.0f) {
                const float ia = __fdividef(-0.5f * B, A), ic = __fdividef(-0.5f * B, C);
                const float thr = fmaf(R->s_max, 1.02f, 0.02f);
                for (uint32_t todo_w = blocks; todo_w; todo_w &= todo_w - 1u) {
                    const int w = __ffs(todo_w) - 1;
                    const int bxw = w % Shape::kBx, byw = w / Shape::kBx;
                    const uint32_t cb = (uint32_t)(bits >> (8 * bxw)) & 0xFFu;
                    const uint32_t rb = (uint32_t)(bits >> (kRs + 8 * byw)) & 0xFFu;
                    const float bx = (float)(x0 + 8 * bxw) + 0.5f - cen_x;
                    const float by = (float)(y0 + 8 * byw) + 0.5f - cen_y;
                    const float m = min_q_box(A, B, C, ia, ic, bx + (float)(__ffs(cb) - 1), bx + (float)(31 - __clz(cb)),
                                              by + (float)(__ffs(rb) - 1), by + (float)(31 - __clz(rb)));
                    if (m > thr) blocks &= ~(1u << w);
                }
            }
            sh.mask[i] = (uint8_t)blocks;
        }
        __syncthreads();
        // Warp-uniform control flow only; per-pixel work is predicated.
        bool warp_done = __all_sync(0xffffffffu, pixels_done());
        if (!warp_done) {
            // the warp's list of the batch
            uint16_t* list = sh.list[warp];
            uint32_t mine_n = 0;
            for (uint32_t c = 0; c < cnt; c += 32) {
                const bool mine = c + lane < cnt && ((sh.mask[c + lane] >> warp) & 1u);
                const uint32_t m = __ballot_sync(0xffffffffu, mine);
                if (mine)
                    list[mine_n + (uint32_t)__popc(m & ((1u << lane) - 1u))] =
                        (uint16_t)((c + lane) * (uint32_t)sizeof(StagedRecord));
                mine_n += (uint32_t)__popc(m);
            }
            __syncwarp();
            // one splat of the list into both pixels' state
            auto shade = [&](uint32_t off) {
                const char* rec = reinterpret_cast<const char*>(recs) + off;
                const float4 q0 = reinterpret_cast<const float4*>(rec)[0];
                const float4 q1 = reinterpret_cast<const float4*>(rec)[1];
                const uint4 q2u = reinterpret_cast<const uint4*>(rec)[2];
                Mask bits;
                if (kRs == 32) bits = (Mask)((unsigned long long)q2u.z | ((unsigned long long)q2u.w << 32));
                else bits = (Mask)q2u.z;
                const float dx = sub(fcx, q0.x);
                const float t0 = mul(mul(q0.z, dx), dx);
                const float m = mul(q0.w, dx);
                const float2 dy = __fadd2_rn(fcy, f2(-q0.y));
                const float2 sq = __fadd2_rn(__fadd2_rn(f2(t0), __fmul2_rn(f2(m), dy)),
                                             __fmul2_rn(__fmul2_rn(f2(q1.x), dy), dy));
                const bool live0 = frag_live(bits, need0, sq.x, q1.z);
                const bool live1 = frag_live(bits, need1, sq.y, q1.z);
                if constexpr (kMode == 0) {
                    const float2 q2 = make_float2(__uint_as_float(q2u.x), __uint_as_float(q2u.y));
                    const float2 arg = __ffma2_rn(sq, f2(kNegHalfLog2e), f2(q1.y));
                    const float a0 = live0 ? fminf(ex2_approx(arg.x), 0.99f) : 0.0f;
                    const float a1 = live1 ? fminf(ex2_approx(arg.y), 0.99f) : 0.0f;
                    const float2 w = __fmul2_rn(make_float2(a0, a1), T);
                    if constexpr (kStates > 0) {
                        const float4* col = sh.col[b & 1][off / (uint32_t)sizeof(StagedRecord)];
                        const float2 w0 = f2(w.x), w1 = f2(w.y);
#pragma unroll
                        for (int ch = 0; ch < 3; ++ch)
#pragma unroll
                            for (int k = 0; k < kStates / 4; ++k) {
                                const float4 c4 = col[ch * (kStates / 4) + k];
                                const float2 lo = make_float2(c4.x, c4.y), hi = make_float2(c4.z, c4.w);
                                CS[0][ch][2 * k] = __ffma2_rn(w0, lo, CS[0][ch][2 * k]);
                                CS[0][ch][2 * k + 1] = __ffma2_rn(w0, hi, CS[0][ch][2 * k + 1]);
                                CS[1][ch][2 * k] = __ffma2_rn(w1, lo, CS[1][ch][2 * k]);
                                CS[1][ch][2 * k + 1] = __ffma2_rn(w1, hi, CS[1][ch][2 * k + 1]);
                            }
                    } else {
                        C0 = __ffma2_rn(w, f2(q1.w), C0);
                        C1 = __ffma2_rn(w, f2(q2.x), C1);
                        C2 = __ffma2_rn(w, f2(q2.y), C2);
                    }
                    T = __ffma2_rn(w, f2(-1.0f), T);
                } else {
                    const float2 q2 = make_float2(__uint_as_float(q2u.x), __uint_as_float(q2u.y));
                    const uint4 q3 = reinterpret_cast<const uint4*>(rec)[3];
                    const uint32_t z24 = q3.x, id = q3.y;
                    last_z = z24;
                    // The depth test first (the tie by index only for a fragment that is
                    // kept), then the hashes, and the exponential for those below alpha's
                    // bound: alpha = min(opacity * exp(power), 0.99) with power <= 0 (exp <= 1
                    // there, also for the deterministic exp) never exceeds min(opacity, 0.99).
                    bool want0[kSeeds], want1[kSeeds], any = false;
#pragma unroll
                    for (int k = 0; k < kSeeds; ++k) {
                        want0[k] = live0 && z24 <= S0[k].best_d24;
                        want1[k] = live1 && z24 <= S1[k].best_d24;
                        any = any || want0[k] || want1[k];
                    }
                    if (any) {
                        const float bound = __uint_as_float(q2u.w), op = __uint_as_float(q3.w);
                        float2 rnd[kSeeds];
                        bool any0 = false, any1 = false;
#pragma unroll
                        for (int k = 0; k < kSeeds; ++k) {
                            rnd[k] = hash13(pixh, k ? __uint_as_float(q3.z) : q1.y);
                            want0[k] = want0[k] && rnd[k].x < bound;
                            want1[k] = want1[k] && rnd[k].y < bound;
                            any0 = any0 || want0[k];
                            any1 = any1 || want1[k];
                        }
                        auto keep = [&](StochState& S, bool want, float r, float alpha) {
                            if (want && r < alpha && (z24 < S.best_d24 || id < S.best_id))
                                S = {z24, id, q1.w, q2.x, q2.y};
                        };
                        if (any0) {
                            const float alpha = g_min(mul(op, det_expf(mul(-0.5f, sq.x))), 0.99f);
#pragma unroll
                            for (int k = 0; k < kSeeds; ++k) keep(S0[k], want0[k], rnd[k].x, alpha);
                        }
                        if (any1) {
                            const float alpha = g_min(mul(op, det_expf(mul(-0.5f, sq.y))), 0.99f);
#pragma unroll
                            for (int k = 0; k < kSeeds; ++k) keep(S1[k], want1[k], rnd[k].y, alpha);
                        }
                    }
                }
            };
            // kTrip splats per trip: one load of their offsets, one loop test and one
            // warp vote (trips of 2 / 4 / 8 measured at 3M room 1080p: alpha 269 / 266 /
            // 255 us, four stochastic samples 1390 / 1357 / 1475 us; eight state frames of
            // 1M take 1577 / 1515 / 1480 us a batch; 16 to a trip was slower again, 264 us)
            constexpr uint32_t kTrip = kMode == 0 ? 8 : 4;
            struct __align__(2 * kTrip) Trip { uint32_t pair[kTrip / 2]; };
            uint32_t k = 0;
            for (; k + kTrip <= mine_n; k += kTrip) {
                const Trip t = *reinterpret_cast<const Trip*>(list + k);
#pragma unroll
                for (uint32_t i = 0; i < kTrip / 2; ++i) {
                    shade(t.pair[i] & 0xFFFFu);
                    shade(t.pair[i] >> 16);
                }
                if (__all_sync(0xffffffffu, pixels_done())) { warp_done = true; break; }
            }
            if (!warp_done) {
                for (; k < mine_n; ++k) shade(list[k]);
                warp_done = __all_sync(0xffffffffu, pixels_done());
            }
        }
        if (__syncthreads_and(warp_done)) break;
    }
    cp_async_wait<0>();   // a batch that was not needed
    if constexpr (kStates > 0) {
        const size_t o0 = (size_t)(p.height - 1 - py0) * p.width + px;
        const size_t o1 = (size_t)(p.height - 1 - py1) * p.width + px;
#pragma unroll
        for (int k = 0; k < kStates; ++k) {
            uint16_t* out = outs[k];
            if (!out) continue;   // a group's unused places
            auto at = [&](int pix, int ch) { return (k & 1) ? CS[pix][ch][k / 2].y : CS[pix][ch][k / 2].x; };
            if (in0)
                write_rgba16f(out, o0, __fmaf_rn(T.x, p.bg, at(0, 0)), __fmaf_rn(T.x, p.bg, at(0, 1)),
                              __fmaf_rn(T.x, p.bg, at(0, 2)), 1.0f - T.x);
            if (in1)
                write_rgba16f(out, o1, __fmaf_rn(T.y, p.bg, at(1, 0)), __fmaf_rn(T.y, p.bg, at(1, 1)),
                              __fmaf_rn(T.y, p.bg, at(1, 2)), 1.0f - T.y);
        }
    } else if (kMode == 0) {
        const size_t o0 = (size_t)(p.height - 1 - py0) * p.width + px;
        const size_t o1 = (size_t)(p.height - 1 - py1) * p.width + px;
        const float2 bg = f2(p.bg);
        const float2 r = __ffma2_rn(T, bg, C0), g = __ffma2_rn(T, bg, C1), bb = __ffma2_rn(T, bg, C2);
        if (in0) write_rgba16f(p.out_rgba16f, o0, r.x, g.x, bb.x, 1.0f - T.x);
        if (in1) write_rgba16f(p.out_rgba16f, o1, r.y, g.y, bb.y, 1.0f - T.y);
    } else if (kMode == 2) {
        if (in0) write_pixel_stoch2(p, px, py0, S0);
        if (in1) write_pixel_stoch2(p, px, py1, S1);
    } else {
        if (in0) write_pixel_stoch(p, px, py0, S0[0]);
        if (in1) write_pixel_stoch(p, px, py1, S1[0]);
    }
}

// Bound by instructions issued (76 % of the slots; the ALU pipe, comparisons,
// selects and integers, is at 50 %, the exponentials' at 42 %) and the two barriers
// of a batch, a quarter of the stalls: one splat into two pixels is some 40 instructions, of
// which the fused multiply-adds, packed two pixels to one, are the smaller part.
// What is the same for the pixels of a warp is therefore done once a record in
// the staging pass, the warp's splats are listed before they are shaded, and the
// stochastic modes leave a pixel's termination to the warp's vote.  Room of 3M
// Gaussians, 1920x1080: alpha 310 -> 210 us, four stochastic samples 1644 -> 1200
// us, two samples and their fallback (denoised mode) 1057 -> 605 us; 6M at
// 3840x2160 798 -> 531 us.
template <int kMode, int kTw = 16, int kTh = 16>
__global__ void __launch_bounds__(kRasterThreads) raster_kernel(RasterParams p) {
    pdl_wait();
    __shared__ RasterShared<kMode, kTw, kTh> sh;
    const uint32_t tile = p.tile_order[blockIdx.x];
    // denoised mode's fallback: all tiles in the frame's order, heaviest first, those
    // within the budget leaving at once (a list of the others in the order in which
    // the network finished them left the SMs idle for a third of the pass)
    if (p.tile_err && !(p.tile_err[tile] >= p.err_budget)) return;
    raster_tile<kMode, kTw, kTh>(p, tile, sh);
}

// Many frames in one persistent launch: work item w is tile
// frames[f].tile_order[w - first[f]] of the frame f with first[f] <= w <
// first[f + 1]; CTAs take items by ticket until all are done.  Every frame of
// a launch has the launch's tile shape.
template <int kMode, int kTw = 16, int kTh = 16>
__global__ void __launch_bounds__(kRasterThreads) raster_batch_kernel(const RasterParams* __restrict__ frames,
                                                                      const uint32_t* __restrict__ first,
                                                                      uint32_t nframes, uint32_t* __restrict__ ticket) {
    __shared__ RasterShared<kMode, kTw, kTh> sh;
    __shared__ uint32_t s_item;
    const uint32_t total = first[nframes];
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(ticket, 1u);
        __syncthreads();
        const uint32_t w = s_item;
        if (w >= total) break;
        uint32_t lo = 0, hi = nframes;   // last f with first[f] <= w
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (first[mid] <= w) lo = mid;
            else hi = mid;
        }
        const RasterParams p = frames[lo];
        raster_tile<kMode, kTw, kTh>(p, p.tile_order[w - first[lo]], sh);
        __syncthreads();
    }
}

// A state batch: CTA b takes group b % groups of the frames on tile
// tile_order[b / groups], so the heaviest tiles of every group start first.
// Per (pixel, splat) pair the alpha work (~45 instructions) is shared by the
// group and a frame adds its three colour FMAs: 8 frames a group (24 KB of
// staged colours, 48 accumulators) against one frame a tile in the batch
// kernel.  1M Gaussians, 1920x1080, 16 blended frames: the call 6620 us when
// every frame rasterized alone (3534 us of it) and was recoloured alone, 1633 us
// in groups, 1446 us with the rasterizer's lists and cp.async; 4 CTAs an SM (128
// registers, 56 bytes spilled) against 3 (142) then 1367 -> 1306 us, 5 (96): 1452.
template <int kStates, int kTw, int kTh>
__global__ void __launch_bounds__(kRasterThreads, kStates == 8 ? 4 : 6)
    raster_states_kernel(RasterParams p, StateOuts outs, int first, uint32_t groups) {
    pdl_wait();
    __shared__ RasterShared<0, kTw, kTh, kStates> sh;
    __shared__ uint16_t* s_out[kStates];
    const uint32_t group = blockIdx.x % groups;
    if (threadIdx.x < kStates) s_out[threadIdx.x] = outs.out[first + (int)group * kStates + (int)threadIdx.x];
    __syncthreads();   // a tile without entries goes through raster_tile without meeting a barrier
    p.colours += (size_t)group * p.record_cap * (3 * kStates / 4);
    raster_tile<0, kTw, kTh, kStates>(p, p.tile_order[blockIdx.x / groups], sh, s_out);
}

template <int kStates>
static void launch_states(const RasterParams& p, const StateOuts& outs, int first, uint32_t groups, cudaStream_t s) {
    const dim3 grid((uint32_t)p.tiles_x * (uint32_t)p.tiles_y * groups), block(kRasterThreads);
    if (p.tile_w == 32) launch_pdl(raster_states_kernel<kStates, 32, 8>, grid, block, 0, s, p, outs, first, groups);
    else if (p.tile_w == 8) launch_pdl(raster_states_kernel<kStates, 8, 32>, grid, block, 0, s, p, outs, first, groups);
    else launch_pdl(raster_states_kernel<kStates, 16, 16>, grid, block, 0, s, p, outs, first, groups);
}

int launch_raster_states(const RasterParams& p, const StateOuts& outs, int frames, cudaStream_t s) {
    if (p.tiles_x <= 0 || p.tiles_y <= 0) return 0;
    const int g8 = state_groups8(frames), g4 = state_groups4(frames);
    if (g8) launch_states<8>(p, outs, 0, (uint32_t)g8, s);
    if (g4) {
        RasterParams q = p;
        q.colours += (size_t)g8 * p.record_cap * 6u;
        launch_states<4>(q, outs, 8 * g8, (uint32_t)g4, s);
    }
    return (g8 ? 1 : 0) + g4;
}

void raster_batch_occupancy(int* blocks_per_sm) {
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, raster_batch_kernel<0, 16, 16>, kRasterThreads, 0);
}

int launch_raster_batch_alpha(const RasterParams* frames, const uint32_t* first, uint32_t nframes, uint32_t* ticket,
                              uint32_t grid, int tile_w, cudaStream_t s) {
    if (nframes == 0) return 0;
    if (tile_w == 32) raster_batch_kernel<0, 32, 8><<<grid, kRasterThreads, 0, s>>>(frames, first, nframes, ticket);
    else if (tile_w == 8) raster_batch_kernel<0, 8, 32><<<grid, kRasterThreads, 0, s>>>(frames, first, nframes, ticket);
    else raster_batch_kernel<0, 16, 16><<<grid, kRasterThreads, 0, s>>>(frames, first, nframes, ticket);
    return 1;
}

int launch_raster_alpha(const RasterParams& p, cudaStream_t s) {
    const uint32_t tiles = (uint32_t)p.tiles_x * (uint32_t)p.tiles_y;
    if (tiles == 0) return 0;
    if (p.tile_w == 32) raster_kernel<0, 32, 8><<<tiles, kRasterThreads, 0, s>>>(p);
    else if (p.tile_w == 8) raster_kernel<0, 8, 32><<<tiles, kRasterThreads, 0, s>>>(p);
    else launch_pdl(raster_kernel<0, 16, 16>, dim3(tiles), dim3(kRasterThreads), 0, s, p);
    return 1;
}

int launch_raster_stochastic2(const RasterParams& p, cudaStream_t s) {
    const uint32_t tiles = (uint32_t)p.tiles_x * (uint32_t)p.tiles_y;
    if (tiles == 0) return 0;
    launch_pdl(raster_kernel<2>, dim3(tiles), dim3(kRasterThreads), 0, s, p);
    return 1;
}

int launch_raster_stochastic(const RasterParams& p, cudaStream_t s) {
    const uint32_t tiles = (uint32_t)p.tiles_x * (uint32_t)p.tiles_y;
    if (tiles == 0) return 0;
    launch_pdl(raster_kernel<1>, dim3(tiles), dim3(kRasterThreads), 0, s, p);
    return 1;
}

}  // namespace gs
