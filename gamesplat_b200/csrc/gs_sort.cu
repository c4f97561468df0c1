// Onesweep LSD radix sort of (uint32 key, uint32 value) pairs for the B200, and
// the two-pass sort of tile entries.
//
// Same result as the reference's 4 x (histogram, single-workgroup prefix,
// bitmask-rank scatter) passes (shaders/sort.glsl:26-163,
// src/renderer.cpp:1873-1962): a stable ascending sort, equal keys in input
// order.  Structure:
//   1. sort_hist_kernel   - one read of the keys builds the digit histograms
//                           of every pass (warp-private shared histograms);
//      (skipped when the producer of the keys already accumulated them);
//   2. sort_pass_kernel   - every CTA derives the pass plan from the
//                           histograms (passes whose digit is the same for all
//                           keys are skipped: identity for a stable sort;
//                           ping-pong assignment of the active passes; when none
//                           is left and the caller needs the result in a given
//                           buffer, the last pass copies), then CTAs take tiles
//                           in ticket order, rank keys within each warp,
//                           publish per-digit counts, reorder the tile by digit
//                           in shared memory, resolve their global offsets by a
//                           two-level look-back (bounded spin) and write runs
//                           coalesced.
// Tile entries (tile id, sorted position) take tile_pass_kernel: the position
// and the upper id bits share a word, the lower 8 id bits travel beside it as a
// byte to the first pass only, and the second pass marks each tile's range.
// Element counts are read on the device, so nothing here synchronises with
// the host.
#include "gs_common.cuh"
#include "gs_internal.h"

namespace gs {

constexpr int kSortWarps = kSortThreads / 32;
constexpr uint32_t kGroupTiles = 16;   // tiles whose counts one group word sums up

int sort_passes(int begin_bit, int end_bit) { return (end_bit - begin_bit + kRadixBits - 1) / kRadixBits; }

size_t sort_status_words(uint32_t count_cap) {
    size_t tiles = ((size_t)count_cap + kSortTile - 1) / kSortTile;
    if (tiles == 0) tiles = 1;
    return tiles * kRadix;
}

// How a pass over n pairs is cut into tiles: as many full waves of the grid as
// the largest tile needs, all tiles of one size, so that no wave is nearly
// empty (2.0M pairs in 4096-pair tiles were 497 tiles on 444 CTAs: two waves,
// 27 us a pass).  The smallest tile bounds the look-back words: a pass uses
// tiles + tiles / 16 rows of kRadix (or 2 kRadix) words, within the 4 rows of
// kRadix per 4096 pairs that sort_status_words() * 4 allots.
struct TileCut {
    uint32_t items, size, count;   // pairs per thread, pairs per tile, tiles
};
template <int kMin, int kMax>
__device__ __forceinline__ TileCut cut_tiles(uint32_t n) {
    const uint32_t lanes = gridDim.x * (uint32_t)kSortThreads;
    const uint32_t waves = max(1u, (n + lanes * kMax - 1u) / (lanes * kMax));
    const uint32_t per = lanes * waves;
    TileCut c;
    c.items = min(max((n + per - 1u) / per, (uint32_t)kMin), (uint32_t)kMax);
    c.size = c.items * (uint32_t)kSortThreads;
    c.count = (n + c.size - 1u) / c.size;
    return c;
}

__device__ __forceinline__ uint32_t digit_of(uint32_t key, int shift, uint32_t dmask) { return (key >> shift) & dmask; }

__global__ void __launch_bounds__(kSortThreads) sort_hist_kernel(SortParams p, int npasses) {
    __shared__ uint32_t wh[kSortWarps][4][kRadix];  // warp-private histograms, 32 KB
    const int warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < kSortWarps * 4 * kRadix; i += kSortThreads) (&wh[0][0][0])[i] = 0u;
    __syncthreads();
    const uint32_t n = p.count_ptr ? *p.count_ptr : p.count_cap;
    const uint32_t stride = gridDim.x * blockDim.x;
    // Vector loads only when the caller's key pointer is 16-byte aligned.
    const uint32_t n4 = (((uintptr_t)p.keys_in & 15u) == 0u) ? (n >> 2) : 0u;
    const uint4* k4 = reinterpret_cast<const uint4*>(p.keys_in);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += stride) {
        uint4 k = __ldg(k4 + i);
        for (int ps = 0; ps < npasses; ++ps) {
            int shift = p.begin_bit + ps * kRadixBits;
            uint32_t dmask = (1u << min(kRadixBits, p.end_bit - shift)) - 1u;
            atomicAdd(&wh[warp][ps][digit_of(k.x, shift, dmask)], 1u);
            atomicAdd(&wh[warp][ps][digit_of(k.y, shift, dmask)], 1u);
            atomicAdd(&wh[warp][ps][digit_of(k.z, shift, dmask)], 1u);
            atomicAdd(&wh[warp][ps][digit_of(k.w, shift, dmask)], 1u);
        }
    }
    for (uint32_t i = (n4 << 2) + blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        uint32_t k = __ldg(p.keys_in + i);
        for (int ps = 0; ps < npasses; ++ps) {
            int shift = p.begin_bit + ps * kRadixBits;
            uint32_t dmask = (1u << min(kRadixBits, p.end_bit - shift)) - 1u;
            atomicAdd(&wh[warp][ps][digit_of(k, shift, dmask)], 1u);
        }
    }
    __syncthreads();
    for (int ps = 0; ps < npasses; ++ps) {
        uint32_t sum = 0;
        for (int w = 0; w < kSortWarps; ++w) sum += wh[w][ps][threadIdx.x];
        if (sum) atomicAdd(&p.hist[ps * kRadix + threadIdx.x], sum);
    }
}

// ---------------------------------------------------------------------------
// Parts of a pass.  kD = digits per thread (a thread owns digits kD t ..).
// ---------------------------------------------------------------------------
template <int kBits>
struct PassShared {
    static constexpr int kR = 1 << kBits;
    static constexpr int kMaskWords = kSortWarps * kR;
    uint16_t cnt[kSortWarps][kR];               // a warp's count of each digit, then its run's start in the tile
    uint32_t base[kR];                          // global position of a digit's run minus its position in the tile
    uint32_t scan_tmp[33];
    uint32_t tile;
};

// Per warp and digit the lanes that hold the digit, zero between items.  The
// masks are done with when the tile is reordered and share its space: with 51
// KB a CTA (26 KB for tile entries) the next kernel, launched while a sort
// drains, finds 92 KB of L1 on the SM; with 68 KB it found 28 KB, and the
// binning's gathers, each holding an L1 line while it is in flight, took 120 us
// instead of 70.
template <int kBits>
__device__ __forceinline__ void clear_masks(uint32_t* mask) {
    for (int i = threadIdx.x; i < PassShared<kBits>::kMaskWords; i += kSortThreads) mask[i] = 0u;
}
template <int kBits>
__device__ __forceinline__ void clear_counts(PassShared<kBits>& sh) {
    uint32_t* c = reinterpret_cast<uint32_t*>(&sh.cnt[0][0]);
    for (int i = threadIdx.x; i < kSortWarps * PassShared<kBits>::kR / 2; i += kSortThreads) c[i] = 0u;
}

// Rank of one item among the warp's items of its digit so far: the lanes that
// hold the digit find each other through a shared word they all set their bit
// in (one shared atomic and ~15 instructions; a ballot per digit bit took
// ~60), their first lane advances the count.
template <int kBits>
__device__ __forceinline__ uint32_t rank_item(PassShared<kBits>& sh, uint32_t* masks, int warp, int lane, uint32_t d,
                                              bool valid) {
    uint32_t* mask = masks + (warp << kBits) + d;
    if (valid) atomicOr(mask, 1u << lane);
    __syncwarp();
    const uint32_t peers = valid ? *mask : 0u;
    const uint32_t before = valid ? sh.cnt[warp][d] : 0u;
    __syncwarp();
    if (valid && lane == __ffs(peers) - 1) {
        sh.cnt[warp][d] = (uint16_t)(before + (uint32_t)__popc(peers));
        *mask = 0u;
    }
    __syncwarp();
    return before + (uint32_t)__popc(peers & ((1u << lane) - 1u));
}

// Exclusive scan of kD values per thread, in digit order.
template <int kD>
__device__ __forceinline__ void scan_digits(const uint32_t (&v)[kD], uint32_t (&out)[kD], uint32_t* tmp) {
    uint32_t sum = 0, total;
#pragma unroll
    for (int q = 0; q < kD; ++q) sum += v[q];
    uint32_t run = block_excl_scan(sum, tmp, &total);
#pragma unroll
    for (int q = 0; q < kD; ++q) {
        out[q] = run;
        run += v[q];
    }
}

// The thread's digits over the warps: totals of the tile, then (behind the
// digits' starts in the tile) every warp's run start in place of its count.
template <int kBits, int kD>
__device__ __forceinline__ void tile_counts(const PassShared<kBits>& sh, uint32_t (&total)[kD]) {
#pragma unroll
    for (int q = 0; q < kD; ++q) {
        total[q] = 0u;
#pragma unroll
        for (int w = 0; w < kSortWarps; ++w) total[q] += sh.cnt[w][threadIdx.x * kD + q];
    }
}
template <int kBits, int kD>
__device__ __forceinline__ void tile_runs(PassShared<kBits>& sh, const uint32_t (&start)[kD]) {
#pragma unroll
    for (int q = 0; q < kD; ++q) {
        uint32_t run = start[q];
#pragma unroll
        for (int w = 0; w < kSortWarps; ++w) {
            uint16_t& c = sh.cnt[w][threadIdx.x * kD + q];
            const uint32_t n = c;
            c = (uint16_t)run;
            run += n;
        }
    }
}

// 16-bit values by item, two to a register (items are unrolled).
template <int kN>
struct Halves {
    uint32_t r[(kN + 1) / 2];
    __device__ __forceinline__ uint32_t get(int k) const { return (k & 1) ? r[k >> 1] >> 16 : r[k >> 1] & 0xFFFFu; }
    __device__ __forceinline__ void set(int k, uint32_t v) {   // even items before odd ones
        r[k >> 1] = (k & 1) ? r[k >> 1] | (v << 16) : v;
    }
};

// Look-back words of a pass: rows of kR words, the tiles' first (every tile
// publishes its counts), then one row per group of 16 tiles (its last tile
// publishes the group's sum, then its inclusive prefix).  A tile sums the at
// most 15 tiles before it in its group and looks back over groups: with all
// tiles of a wave ranked at about the same time a plain look-back over tiles
// advances 8 tiles an L2 round trip, ~20 us for 440 tiles.
template <int kD>
__device__ __forceinline__ void publish(u64* row, const uint32_t (&v)[kD], uint32_t tag, uint32_t flag) {
#pragma unroll
    for (int q = 0; q < kD; ++q) st_relaxed64(row + threadIdx.x * kD + q, status_word(tag, flag, v[q]));
}

template <int kD>
__device__ __forceinline__ void lookback(u64* status, uint32_t tile, uint32_t tiles, uint32_t tag,
                                         const uint32_t (&own)[kD], uint32_t (&excl)[kD], uint32_t* error_flags) {
    constexpr uint32_t kR = kD * kSortThreads;
    constexpr int kStep = kD == 1 ? 8 : 4;
    const uint32_t group = tile / kGroupTiles, first = group * kGroupTiles;
    u64* groups = status + (size_t)tiles * kR;
    const u64* col = status + threadIdx.x * kD;
    bool timed_out = false;
#pragma unroll
    for (int q = 0; q < kD; ++q) excl[q] = 0u;
    for (uint32_t j = first; j < tile; j += kStep) {
        u64 w[kStep][kD];
#pragma unroll
        for (int k = 0; k < kStep; ++k)
#pragma unroll
            for (int q = 0; q < kD; ++q)
                w[k][q] = j + k < tile ? ld_relaxed64(col + (size_t)(j + k) * kR + q) : status_word(tag, kFlagAgg, 0u);
#pragma unroll
        for (int k = 0; k < kStep; ++k)
#pragma unroll
            for (int q = 0; q < kD; ++q) {
                uint32_t spins = 0;
                while ((uint32_t)(w[k][q] >> 32) != tag) {   // not published yet
                    if (++spins > kSpinLimit) {
                        timed_out = true;
                        w[k][q] = 0;
                        break;
                    }
                    if (spins > 64) __nanosleep(32);
                    w[k][q] = ld_relaxed64(col + (size_t)(j + k) * kR + q);
                }
                excl[q] += (uint32_t)w[k][q] & kValMask;
            }
    }
    const bool leader = tile % kGroupTiles == kGroupTiles - 1u;
    uint32_t sum[kD];
    if (leader) {
#pragma unroll
        for (int q = 0; q < kD; ++q) sum[q] = excl[q] + own[q];
        publish<kD>(groups + (size_t)group * kR, sum, tag, group == 0u ? kFlagInc : kFlagAgg);
    }
    if (group > 0u) {
#pragma unroll
        for (int q = 0; q < kD; ++q)
            excl[q] += lookback_vec<8>(groups + threadIdx.x * kD + q, kR, group, tag, &timed_out);
        if (leader) {
#pragma unroll
            for (int q = 0; q < kD; ++q) sum[q] = excl[q] + own[q];
            publish<kD>(groups + (size_t)group * kR, sum, tag, kFlagInc);
        }
    }
    if (timed_out) atomicOr(error_flags, kErrSortLookback);
}

// Pass plan, recomputed by every CTA of every pass kernel from the digit
// histograms: a pass is skipped when one digit holds every key (a stable sort
// by a constant digit is the identity); active passes ping-pong between the
// writable buffers (with land_in_buf0 the last one writes buffer 0).
struct PassIO {
    const uint32_t* kin;
    const uint32_t* vin;
    uint32_t* kout;
    uint32_t* vout;
    const uint32_t* kfinal;
    const uint32_t* vfinal;
    bool active;
    bool copy_needed;
};

// own: this pass's histogram at the thread's digits.
template <int kBits>
__device__ __forceinline__ PassIO plan_passes(const SortParams& p, int npasses, int pass, uint32_t n,
                                              uint32_t (&own)[(1 << kBits) / kSortThreads]) {
    constexpr int kD = (1 << kBits) / kSortThreads;
    uint32_t h[4][kD];
#pragma unroll
    for (int ps = 0; ps < 4; ++ps)   // all in flight at once
#pragma unroll
        for (int q = 0; q < kD; ++q) h[ps][q] = ps < npasses ? p.hist[(ps << kBits) + threadIdx.x * kD + q] : 0u;
    uint32_t active = 0;
#pragma unroll
    for (int ps = 0; ps < 4; ++ps) {
        bool all = false;
#pragma unroll
        for (int q = 0; q < kD; ++q) {
            all |= h[ps][q] == n;
            if (ps == pass) own[q] = h[ps][q];
        }
        if (ps < npasses && !__syncthreads_or(all)) active |= 1u << ps;
    }
    const int m = __popc(active);
    PassIO io{};
    const uint32_t* kcur = p.keys_in;
    const uint32_t* vcur = p.vals_in;
    int j = 0;
    for (int ps = 0; ps < npasses; ++ps) {
        if (!((active >> ps) & 1u)) continue;
        const int dst = p.land_in_buf0 ? ((m - 1 - j) & 1) : (j & 1);
        if (ps == pass) {
            io.kin = kcur;
            io.vin = vcur;
            io.kout = p.keys_buf[dst];
            io.vout = p.vals_buf[dst];
        }
        kcur = p.keys_buf[dst];
        vcur = p.vals_buf[dst];
        ++j;
    }
    io.active = (active >> pass) & 1u;
    io.copy_needed = p.land_in_buf0 && m == 0;
    io.kfinal = io.copy_needed ? p.keys_buf[0] : kcur;
    io.vfinal = io.copy_needed ? p.vals_buf[0] : vcur;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        SortPlan* pl = p.plan;
        pl->kfinal = io.kfinal;
        pl->vfinal = io.vfinal;
        pl->count = n;
    }
    return io;
}

// kBits 8 (any bit range) or 9 (the depth keys, whose range after the bias is
// 27 bits in practice: three passes).  Per tile: ~3 us of loads and ranking,
// the rest latency of the scans, the look-back and the scatter, with the data
// in L2; three CTAs an SM hide each other's.  Times at launch_sort.
constexpr int kPairMin = 9, kPairMax = 20;    // items per thread (9: see cut_tiles, rows of 512 words)
static_assert(PassShared<9>::kMaskWords <= kPairMax * kSortThreads, "the masks fit the reordered keys' space");
template <int kBits>
constexpr size_t pair_smem() { return sizeof(PassShared<kBits>) + 2 * (size_t)kPairMax * kSortThreads * 4; }

template <int kBits>
__global__ void __launch_bounds__(kSortThreads, 3) sort_pass_kernel(SortParams p, int pass, int npasses) {
    constexpr int kD = (1 << kBits) / kSortThreads;
    constexpr int kMin = kBits == 9 ? kPairMin : 5;
    pdl_wait();
    pdl_trigger();
    extern __shared__ __align__(16) uint8_t s_raw[];
    PassShared<kBits>& sh = *reinterpret_cast<PassShared<kBits>*>(s_raw);
    uint32_t* s_keys = reinterpret_cast<uint32_t*>(s_raw + sizeof(PassShared<kBits>));   // the tile reordered by digit
    uint32_t* s_vals = s_keys + kPairMax * kSortThreads;

    uint32_t ticket = 0;
    if (threadIdx.x == 0) ticket = atomicAdd(&p.plan->ticket[pass], 1u);
    const uint32_t n = p.count_ptr ? *p.count_ptr : p.count_cap;
    uint32_t own[kD];
    const PassIO io = plan_passes<kBits>(p, npasses, pass, n, own);
    if (!io.active) {
        if (io.copy_needed && pass == npasses - 1)
            for (uint32_t i = blockIdx.x * kSortThreads + threadIdx.x; i < n; i += gridDim.x * kSortThreads) {
                p.keys_buf[0][i] = p.keys_in[i];
                p.vals_buf[0][i] = p.vals_in[i];
            }
        return;
    }
    const uint32_t* __restrict__ kin = io.kin;
    const uint32_t* __restrict__ vin = io.vin;
    uint32_t* __restrict__ kout = io.kout;
    uint32_t* __restrict__ vout = io.vout;
    const int shift = p.begin_bit + pass * kBits;
    const uint32_t dmask = (1u << min(kBits, p.end_bit - shift)) - 1u, bias = p.key_bias;
    const TileCut cut = cut_tiles<kMin, kPairMax>(n);
    const uint32_t tag = sort_tag(p.epoch, (uint32_t)pass);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t gdigit[kD];   // global start of the thread's digits
    scan_digits<kD>(own, gdigit, sh.scan_tmp);

    for (;;) {
        if (threadIdx.x == 0) sh.tile = ticket;
        clear_counts(sh);
        clear_masks<kBits>(s_keys);
        __syncthreads();
        const uint32_t tile = sh.tile;
        if (tile >= cut.count) break;
        const uint32_t first = tile * cut.size, wfirst = first + (uint32_t)warp * cut.items * 32u + (uint32_t)lane;
        uint32_t key[kPairMax];
        Halves<kPairMax> rank, at;   // rank in the warp, then position in the reordered tile
#pragma unroll
        for (int k = 0; k < kPairMax; ++k) {
            const uint32_t idx = wfirst + (uint32_t)k * 32u;
            key[k] = k < cut.items && idx < n ? kin[idx] : 0u;
        }
#pragma unroll
        for (int k = 0; k < kPairMax; ++k) {
            if (k >= cut.items) break;
            rank.set(k, rank_item<kBits>(sh, s_keys, warp, lane, digit_of(key[k] + bias, shift, dmask), wfirst + (uint32_t)k * 32u < n));
        }
        __syncthreads();
        uint32_t total[kD], start[kD];
        tile_counts(sh, total);
        publish<kD>(p.status + (size_t)tile * (kD * kSortThreads), total, tag, kFlagAgg);
        scan_digits<kD>(total, start, sh.scan_tmp);
        tile_runs(sh, start);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kPairMax; ++k) {
            if (k >= cut.items) break;
            const uint32_t o = rank.get(k) + sh.cnt[warp][digit_of(key[k] + bias, shift, dmask)];
            if (wfirst + (uint32_t)k * 32u < n) s_keys[o] = key[k];
            at.set(k, o);
        }
        // the values come in, and the next ticket, while the look-back waits
        uint32_t val[kPairMax];
#pragma unroll
        for (int k = 0; k < kPairMax; ++k) {
            const uint32_t idx = wfirst + (uint32_t)k * 32u;
            val[k] = k < cut.items && idx < n ? vin[idx] : 0u;
        }
        if (threadIdx.x == 0) ticket = cut.count > gridDim.x ? atomicAdd(&p.plan->ticket[pass], 1u) : cut.count;
        uint32_t excl[kD];
        lookback<kD>(p.status, tile, cut.count, tag, total, excl, p.error_flags);
#pragma unroll
        for (int q = 0; q < kD; ++q) sh.base[threadIdx.x * kD + q] = gdigit[q] + excl[q] - start[q];
#pragma unroll
        for (int k = 0; k < kPairMax; ++k) {
            if (k >= cut.items) break;
            if (wfirst + (uint32_t)k * 32u < n) s_vals[at.get(k)] = val[k];
        }
        __syncthreads();
        const uint32_t count = min(cut.size, n - first);
        for (uint32_t i = threadIdx.x; i < count; i += kSortThreads) {
            const uint32_t k = s_keys[i];
            const uint32_t o = sh.base[digit_of(k + bias, shift, dmask)] + i;
            if (o < n) {  // always true unless a look-back wait ran out
                kout[o] = k;
                vout[o] = s_vals[i];
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Tile entries, in the order the binning wrote them, to lists per tile.  Two
// passes over one 32-bit word per entry: (upper tile-id bits << vbits) | sorted
// position.  kPass 0 sorts by the lower 8 id bits, which come as a byte beside
// the word; kPass 1 by the upper bits.  An entry's lower bits are known in the
// second pass from where it stands (the first pass put equal ones together), so
// only positions are written at the end, and each CTA marks where the tiles
// begin and end in the runs it writes: per entry 22 bytes move (5 + 5 + 4 + 4 +
// 4, the expansion's write included) instead of 44 with (id, position) pairs
// and a pass over the sorted ids for the ranges.
// A range is kept as (~start, end) under maxima until tile_order_kernel turns
// it round: zero means no entries.
// ---------------------------------------------------------------------------
constexpr int kEntryMin = 5, kEntryMax = 16;

static_assert(PassShared<8>::kMaskWords <= kEntryMax * kSortThreads, "the masks fit the reordered words' space");

struct EntryShared {
    PassShared<8> pass;
    uint32_t word[kEntryMax * kSortThreads];
    uint8_t low[kEntryMax * kSortThreads];    // lower id bits of the reordered entries
    uint32_t low_start[257];                  // kPass 1: where the entries of each lower digit start
};

template <int kPass>
__global__ void __launch_bounds__(kSortThreads, 4) tile_pass_kernel(TileSortParams p) {
    pdl_wait();
    pdl_trigger();
    extern __shared__ __align__(16) uint8_t s_raw[];
    EntryShared& es = *reinterpret_cast<EntryShared*>(s_raw);
    PassShared<8>& sh = es.pass;
    uint32_t ticket = 0;
    if (threadIdx.x == 0) ticket = atomicAdd(&p.plan->ticket[kPass], 1u);
    const uint32_t n = *p.count_ptr;
    const uint32_t own[1] = {p.hist[kPass * kRadix + threadIdx.x]};
    const uint32_t low_count[1] = {kPass == 1 ? p.hist[threadIdx.x] : 0u};
    const uint32_t* __restrict__ in = p.words[kPass];
    uint32_t* __restrict__ out = p.words[kPass + 1];
    const uint32_t vmask = p.vbits >= 32 ? 0xFFFFFFFFu : (1u << p.vbits) - 1u;
    const TileCut cut = cut_tiles<kEntryMin, kEntryMax>(n);
    const uint32_t tag = sort_tag(p.epoch, (uint32_t)kPass);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t gdigit[1];
    scan_digits<1>(own, gdigit, sh.scan_tmp);
    if (kPass == 1) {
        uint32_t s[1];
        scan_digits<1>(low_count, s, sh.scan_tmp);
        es.low_start[threadIdx.x] = s[0];
        if (threadIdx.x == 0) es.low_start[256] = n;
    } else if (p.last_pass == 0 && blockIdx.x == 0 && threadIdx.x < p.num_tiles && own[0]) {
        p.ranges[threadIdx.x] = make_uint2(~gdigit[0], gdigit[0] + own[0]);   // at most 256 tiles: this pass is all
    }
    if (blockIdx.x == 0 && threadIdx.x == 0 && p.last_pass == kPass) {
        p.plan->vfinal = out;
        p.plan->count = n;
    }

    for (;;) {
        if (threadIdx.x == 0) sh.tile = ticket;
        clear_counts(sh);
        clear_masks<8>(es.word);
        __syncthreads();
        const uint32_t tile = sh.tile;
        if (tile >= cut.count) break;
        const uint32_t first = tile * cut.size, wfirst = first + (uint32_t)warp * cut.items * 32u + (uint32_t)lane;
        uint32_t word[kEntryMax];
        Halves<kEntryMax> rank;
        uint32_t dig[kPass == 0 ? kEntryMax / 4 : 1] = {};   // four lower digits to a register
#pragma unroll
        for (int k = 0; k < kEntryMax; ++k) {
            const uint32_t idx = wfirst + (uint32_t)k * 32u;
            const bool in_range = k < cut.items && idx < n;
            if (kPass == 0) dig[k >> 2] |= (in_range ? (uint32_t)__ldg(p.low + idx) : 0u) << (8 * (k & 3));
            word[k] = in_range ? in[idx] : 0u;
        }
        auto digit = [&](int k) -> uint32_t {
            if constexpr (kPass == 0) return (dig[k >> 2] >> (8 * (k & 3))) & 255u;
            else return word[k] >> p.vbits;
        };
#pragma unroll
        for (int k = 0; k < kEntryMax; ++k) {
            if (k >= cut.items) break;
            rank.set(k, rank_item<8>(sh, es.word, warp, lane, digit(k), wfirst + (uint32_t)k * 32u < n));
        }
        __syncthreads();
        uint32_t total[1], start[1];
        tile_counts(sh, total);
        publish<1>(p.status + (size_t)tile * kSortThreads, total, tag, kFlagAgg);
        scan_digits<1>(total, start, sh.scan_tmp);
        tile_runs(sh, start);
        __syncthreads();
        // The lower digit at the tile's first entry: the last one that starts at or before it.  Most tiles hold
        // entries of that digit alone (6.5M entries: 25 000 a digit): their ranges are their digits' runs.
        uint32_t low = 0;
        bool one_low = false;
        if (kPass == 1) {
            int hi = 255;
            while ((int)low < hi) {
                const int mid = ((int)low + hi + 1) >> 1;
                if (es.low_start[mid] <= first) low = (uint32_t)mid;
                else hi = mid - 1;
            }
            one_low = es.low_start[low + 1u] >= min(first + cut.size, n);
        }
        const uint32_t tile_low = low;
#pragma unroll
        for (int k = 0; k < kEntryMax; ++k) {
            if (k >= cut.items) break;
            const uint32_t idx = wfirst + (uint32_t)k * 32u;
            if (idx < n) {
                const uint32_t d = digit(k);
                const uint32_t o = rank.get(k) + sh.cnt[warp][d];
                es.word[o] = word[k];
                if (kPass == 0) {
                    es.low[o] = (uint8_t)d;
                } else if (!one_low) {
                    while (low < 255u && es.low_start[low + 1u] <= idx) ++low;
                    es.low[o] = (uint8_t)low;
                }
            }
        }
        if (threadIdx.x == 0) ticket = cut.count > gridDim.x ? atomicAdd(&p.plan->ticket[kPass], 1u) : cut.count;
        uint32_t excl[1];
        lookback<1>(p.status, tile, cut.count, tag, total, excl, p.error_flags);
        sh.base[threadIdx.x] = gdigit[0] + excl[0] - start[0];
        __syncthreads();
        const uint32_t count = min(cut.size, n - first);
        if (kPass == 1 && one_low) {
            const uint32_t id = (threadIdx.x << 8) | tile_low, o = gdigit[0] + excl[0];
            if (total[0] && id < p.num_tiles && o + total[0] <= n) {
                atomicMax(&p.ranges[id].x, ~o);
                atomicMax(&p.ranges[id].y, o + total[0]);
            }
            for (uint32_t i = threadIdx.x; i < count; i += kSortThreads) {
                const uint32_t w = es.word[i], o2 = sh.base[w >> p.vbits] + i;
                if (o2 < n) out[o2] = w & vmask;   // o2 >= n: a look-back wait ran out
            }
        } else for (uint32_t i0 = 0; i0 < count; i0 += kSortThreads) {   // whole warps: the neighbours come by shuffles
            const uint32_t i = i0 + threadIdx.x;
            const bool valid = i < count;
            const uint32_t w = valid ? es.word[i] : 0u, l = valid ? es.low[i] : 0u;
            const uint32_t d = kPass == 0 ? l : w >> p.vbits;
            const uint32_t o = valid ? sh.base[d] + i : n;
            if (o < n) out[o] = p.last_pass == kPass ? w & vmask : w;   // o >= n: a look-back wait ran out
            if (kPass == 1) {
                const uint32_t id = valid ? (d << 8) | l : 0xFFFFFFFFu;
                uint32_t prev = __shfl_up_sync(0xffffffffu, id, 1), next = __shfl_down_sync(0xffffffffu, id, 1);
                if (lane == 0) prev = i > 0u && valid ? ((es.word[i - 1u] >> p.vbits) << 8) | es.low[i - 1u] : 0xFFFFFFFFu;
                if (lane == 31)
                    next = i + 1u < count ? ((es.word[i + 1u] >> p.vbits) << 8) | es.low[i + 1u] : 0xFFFFFFFFu;
                if (o < n && id < p.num_tiles) {
                    if (prev != id) atomicMax(&p.ranges[id].x, ~o);
                    if (next != id) atomicMax(&p.ranges[id].y, o + 1u);
                }
            }
        }
        __syncthreads();
    }
}

// Per device: a pass kernel's shared-memory opt-in, then its occupancy.
constexpr int kMaxDevices = 64;
struct PassLaunch {
    int blocks_per_sm[kMaxDevices] = {};
    template <class K>
    uint32_t resident(K* kernel, size_t smem, uint32_t num_sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        int& b = blocks_per_sm[dev >= 0 && dev < kMaxDevices ? dev : 0];
        if (b == 0 || dev >= kMaxDevices) {
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            int n = 0;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kSortThreads, smem);
            b = n > 0 ? n : 1;
        }
        return num_sms * (uint32_t)b;
    }
};

static uint32_t pass_grid(uint32_t resident, uint32_t count_cap, int min_items) {
    const uint32_t tile = (uint32_t)min_items * kSortThreads, tiles = count_cap / tile + (count_cap % tile ? 1u : 0u);
    return resident < tiles ? resident : (tiles ? tiles : 1u);
}

template <int kBits>
static int launch_passes(const SortParams& p, uint32_t num_sms, cudaStream_t s) {
    static PassLaunch at;
    const int npasses = (p.end_bit - p.begin_bit + kBits - 1) / kBits;
    const uint32_t grid = pass_grid(at.resident(sort_pass_kernel<kBits>, pair_smem<kBits>(), num_sms), p.count_cap,
                                    kBits == 9 ? kPairMin : 5);
    for (int ps = 0; ps < npasses; ++ps) {
        // Passes after the first overlap their launch with the previous pass's
        // tail (programmatic dependent launch); so does the first pass when the
        // caller asks (the frame's sorts: every kernel of a frame starts with
        // griddepcontrol.wait).  The stage-level entry points launch it
        // ordinarily behind the caller's work.
        if (ps == 0 && !p.first_pdl)
            sort_pass_kernel<kBits><<<grid, kSortThreads, pair_smem<kBits>(), s>>>(p, ps, npasses);
        else
            launch_pdl(sort_pass_kernel<kBits>, dim3(grid), dim3(kSortThreads), pair_smem<kBits>(), s, p, ps, npasses);
    }
    return npasses;
}

int launch_sort(const SortParams& p, uint32_t num_sms, cudaStream_t s) {
    int launches = 0;
    if (!p.hist_ready) {
        uint32_t hist_grid = num_sms * 2;
        uint32_t hist_need = (p.count_cap / 4 + kSortThreads - 1) / kSortThreads;
        if (hist_grid > hist_need) hist_grid = hist_need > 0 ? hist_need : 1;
        sort_hist_kernel<<<hist_grid, kSortThreads, 0, s>>>(p, sort_passes(p.begin_bit, p.end_bit));
        ++launches;
    }
    return launches + launch_passes<kRadixBits>(p, num_sms, s);
}

// 2.0M depth keys (3M Gaussians, 1080p): 80 us for the three 9-bit passes and
// the skipped one, against 108 us for four of 8 bits in 4096-pair tiles with a
// plain look-back; 4M keys 134 against 164 us.
int launch_depth_sort(const SortParams& p, uint32_t num_sms, cudaStream_t s) {
    return launch_passes<kDepthBits>(p, num_sms, s);
}

// 6.5M entries (8160 tiles): 43 + 50 us and no range pass, with the order 104
// us; as (id, position) pairs 133 us.  25M entries (32 400 tiles): 460 against
// 511 us.
int launch_tile_sort(const TileSortParams& p, uint32_t num_sms, cudaStream_t s) {
    static PassLaunch at[2];
    const uint32_t g0 = pass_grid(at[0].resident(tile_pass_kernel<0>, sizeof(EntryShared), num_sms), p.count_cap, kEntryMin);
    launch_pdl(tile_pass_kernel<0>, dim3(g0), dim3(kSortThreads), sizeof(EntryShared), s, p);
    if (p.last_pass == 0) return 1;
    const uint32_t g1 = pass_grid(at[1].resident(tile_pass_kernel<1>, sizeof(EntryShared), num_sms), p.count_cap, kEntryMin);
    launch_pdl(tile_pass_kernel<1>, dim3(g1), dim3(kSortThreads), sizeof(EntryShared), s, p);
    return 2;
}

}  // namespace gs

// ---------------------------------------------------------------------------
// Stage-level C entry point: sort caller-owned device buffers.
// Scratch layout: SortPlan | 4x256 histograms | error word | look-back words
// (all passes share them) | temporary keys | temporary values (256-byte aligned).
// ---------------------------------------------------------------------------
namespace {
size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }
struct SortScratch {
    size_t plan, hist, err, status, tkeys, tvals, total, control_bytes;
};
SortScratch sort_scratch_layout(uint32_t n) {
    SortScratch l{};
    size_t off = 0;
    l.plan = off; off += align256(sizeof(gs::SortPlan));
    l.hist = off; off += align256(4 * 256 * 4);
    l.err = off; off += align256(4);
    l.status = off; off += align256(gs::sort_status_words(n) * 4 * sizeof(unsigned long long));
    l.control_bytes = off;
    l.tkeys = off; off += align256((size_t)n * 4);
    l.tvals = off; off += align256((size_t)n * 4);
    l.total = off;
    return l;
}
}  // namespace

extern "C" size_t gs_sort_pairs_scratch_bytes(uint32_t n) { return sort_scratch_layout(n).total; }

extern "C" int gs_sort_pairs(const uint32_t* keys_in, const uint32_t* vals_in, uint32_t* keys_out, uint32_t* vals_out,
                             uint32_t n, int begin_bit, int end_bit, void* scratch, size_t scratch_bytes,
                             void* stream) {
    if (begin_bit < 0 || end_bit > 32 || end_bit <= begin_bit) return GS_ERR_BAD_ARG;
    if (n == 0) return GS_OK;
    if (n > (1u << 30) - 1) return GS_ERR_TOO_LARGE;
    if (!keys_in || !vals_in || !keys_out || !vals_out || !scratch) return GS_ERR_BAD_ARG;
    if ((const void*)keys_in == (const void*)keys_out || (const void*)vals_in == (const void*)vals_out)
        return GS_ERR_BAD_ARG;
    const SortScratch l = sort_scratch_layout(n);
    if (scratch_bytes < l.total) return GS_ERR_BAD_ARG;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    char* base = static_cast<char*>(scratch);
    if (cudaMemsetAsync(base, 0, l.control_bytes, s) != cudaSuccess) return GS_ERR_CUDA;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    gs::SortParams p{};
    p.keys_in = keys_in;
    p.vals_in = vals_in;
    p.keys_buf[0] = keys_out;
    p.vals_buf[0] = vals_out;
    p.keys_buf[1] = reinterpret_cast<uint32_t*>(base + l.tkeys);
    p.vals_buf[1] = reinterpret_cast<uint32_t*>(base + l.tvals);
    p.land_in_buf0 = 1;
    p.count_ptr = nullptr;
    p.count_cap = n;
    p.begin_bit = begin_bit;
    p.end_bit = end_bit;
    p.hist = reinterpret_cast<uint32_t*>(base + l.hist);
    p.plan = reinterpret_cast<gs::SortPlan*>(base + l.plan);
    p.status = reinterpret_cast<unsigned long long*>(base + l.status);
    p.epoch = 1;
    p.error_flags = reinterpret_cast<uint32_t*>(base + l.err);
    gs::launch_sort(p, sms > 0 ? (uint32_t)sms : 148u, s);
    return cudaGetLastError() == cudaSuccess ? GS_OK : GS_ERR_CUDA;
}
