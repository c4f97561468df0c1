// Internal interfaces between the C++ host orchestration (gs_host.cpp) and the
// CUDA kernels.  Not part of the public C ABI (include/gs_api.h).
#pragma once
#include <atomic>
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/gs_api.h"

namespace gs {

// Device error flags (gs_stats.error_flags).
enum : uint32_t {
    kErrCullLookback = 1u << 0,
    kErrSortLookback = 1u << 1,
    kErrBinLookback = 1u << 2,
    kErrTileOverflow = 1u << 4,
    kErrGpsWait = 1u << 5,
    kErrCullStage = 1u << 6,
};

// Small per-frame device control block.  Zeroed at the start of each frame
// (one memset), except where noted.
struct FrameCounters {
    uint32_t visible_count;      // cull output (shaders/cull.glsl:230)
    uint32_t diag[8];            // SplatDiagnostics (shaders/cull.glsl:296-318)
    uint32_t error_flags;        // gs::kErr* bits
    uint32_t cull_ticket;        // tile tickets for persistent kernels
    uint32_t bin_ticket;
    uint32_t tile_entries;       // (tile, splat) pairs produced by binning
    uint32_t tile_overflow;      // entries that did not fit
    uint32_t gps_work[2];        // [0] requested work items, [1] overflow (gps.glsl work_count)
    uint32_t raster_ticket;
    uint32_t fallback_tiles;     // denoised mode: tiles over the error budget
    uint32_t pad[1];
};

// Device-resident state of one radix sort: the tile tickets of its passes and
// where its result is.  Zeroed before each sort.
struct SortPlan {
    const uint32_t* kfinal;      // where the sorted keys are
    const uint32_t* vfinal;      // where the sorted values are
    uint32_t ticket[4];
    uint32_t count;
};

// Look-back words carry a frame's epoch (1 .. kEpochs - 1, round again) in their
// upper half, those of the sorts the epoch and the pass, so that one frame's
// words, or the zeros of memory never written, are not another's.
constexpr uint32_t kEpochs = 1u << 30;
constexpr uint32_t next_epoch(uint32_t epoch) { return epoch + 1u < kEpochs ? epoch + 1u : 1u; }
__host__ __device__ constexpr uint32_t sort_tag(uint32_t epoch, uint32_t pass) { return (epoch << 2) | pass; }

// Onesweep radix sort configuration.
constexpr int kSortThreads = 256;
constexpr int kSortTile = 4096;   // pairs per 4 x kRadix look-back words (sort_status_words() * 4 words in all)
constexpr int kRadixBits = 8;
constexpr int kRadix = 1 << kRadixBits;
// Depth keys are 0xFFFFFFFF - bits(depth) with depth >= 0.2 for every visible
// row (the near test of the cull).  Adding bits(0.2f) (modulo 2^32) keeps their
// order and lifts the keys of depths below ~13 000 into the top 2^27 of the
// range: their upper 5 bits are equal, so three passes of 9 bits sort them and
// the fourth, of 5, is skipped.
constexpr int kDepthBits = 9;
constexpr int kDepthRadix = 1 << kDepthBits;
constexpr uint32_t kDepthKeyBias = 0x3E4CCCCDu;   // bits of 0.2f

// Cull configuration.  Visibility pass: 256-thread CTAs that take tiles of 8 to
// 20 rows a thread, cut so that they fill whole rounds (launch_cull).  Projection
// pass: 128-thread CTAs, each warp stages and projects 32 visible rows at a time.
constexpr int kCullVisThreads = 256;
constexpr int kCullVisItems = 8;     // rows a thread: the fewest of a tile, and the most
constexpr int kVisItemsMax = 20;
constexpr int kVisPerSm = 4;         // resident CTAs
constexpr int kCullVisTile = kCullVisThreads * kCullVisItems;   // the smallest tile: sizes the status words
constexpr int kCullThreads = 128;
constexpr int kHalfRowChunks = 9;   // 144-byte FP16-SH row: position/opacity, scale, rotation, 48 half SH

// Binning configuration: 8 sorted splats per thread, 1024 per CTA tile; the
// expansion takes the global entry range in chunks of 1024 entries.
constexpr int kBinThreads = 128;
constexpr int kBinItems = 8;
constexpr int kBinTile = kBinThreads * kBinItems;
constexpr int kBinChunk = 8 * kBinThreads;     // entries expanded per round
constexpr int kTileW = 16;
constexpr int kTileH = 16;

// Raster record: one per visible splat in depth-sorted order, 64 bytes,
// gathered into shared memory by cp.async.
//
// The rasterizer tests the splat's quadratic form s = conic(d) (the power is
// -0.5 s) instead of the power: "power <= 0 && !(power < cutoff)" holds
// exactly when -2^-149 <= s <= s_max, with s_max = -2 cutoff, or the smallest
// subnormal when cutoff == 0 (multiplying by -0.5 is exact except for
// subnormal s, and those cases are what the two bounds absorb).  The test made
// is 0 <= s <= s_max (frag_live, which says why no splat reaches the rest).
//
// Stochastic envelope records (BinParams::envelope) reuse three slots:
// log2_opacity holds radius_x, rect_x holds the bits of ndc_z and rect_y the
// bits of radius_y; cx, cy are un-jittered.
struct __align__(16) RasterRecord {
    float cx, cy, conic_x, conic_2y;     // centre (+jitter), conic.x, 2*conic.y
    float conic_z, log2_opacity, s_max, r;
    float g, b;
    uint32_t rect_x;                     // i0 | i1 << 16  (candidate pixel columns: quad coverage
    uint32_t rect_y;                     // j0 | j1 << 16   intersected with the alpha >= 1/255 box, GL rows)
    uint32_t depth24;                    // window depth as D24 (stochastic depth test)
    uint32_t splat_id;                   // original Gaussian index
    float hash_z;                        // 0; the two-sample rasterizer's staging keeps the second seed's hash here
    float opacity;
};
static_assert(sizeof(RasterRecord) == 64, "RasterRecord must be 64 bytes");

struct CullParams {
    const float4* rows;          // N x 16 float4 (GpuGaussian)
    const float4* heads;         // N float4: the first 16 bytes of every row (position, opacity), kept beside the rows
    uint32_t n;
    gs_camera cam;               // the frame's CameraUniforms, by value (constant-bank operands)
    int sh_degree;
    float sh_lod_distance;
    int collect_stats;
    int write_invisible;         // also write the reference's invisible record
    float4* projected;           // N x 4 float4 (CullProjectedSplatData)
    uint32_t* keys_out;          // compacted visible keys, index order
    uint32_t* ids_out;           // compacted visible ids
    unsigned long long* status;  // per-tile look-back words (epoch-tagged)
    uint32_t epoch;
    uint32_t* key_hist;          // 4 x kDepthRadix digit histograms of key + kDepthKeyBias (zeroed per frame)
    // gsanim int8 appearance deltas (shaders/cull.glsl:125-164); null = none
    const int8_t* anim_deltas;   // [(state-1) * n + row] * 48 + j
    const float* anim_scales;    // 48 (device)
    int anim_state_a, anim_state_b;
    float anim_weight;
    // gsanim 0.3 appearance layers (shaders/cull.glsl:141-148, 354-416); layer_count 0 = none
    const uint16_t* layer_halves;   // [(l * n + row) * 48 + j] IEEE half bits
    const float* layer_weights;     // [l * 3 + c] (device)
    int layer_count;
    int half_rows;               // rows are 144-byte FP16-SH rows (kHalfRowChunks float4 each)
    FrameCounters* fc;
};

struct SortParams {
    const uint32_t* keys_in;     // input pairs (never written)
    const uint32_t* vals_in;
    uint32_t* keys_buf[2];       // writable ping-pong buffers (keys_buf[1] may alias keys_in
    uint32_t* vals_buf[2];       //  when land_in_buf0 == 0)
    int land_in_buf0;            // 1: the result must end in keys_buf[0]/vals_buf[0]
    const uint32_t* count_ptr;   // device-side element count
    uint32_t count_cap;          // capacity (grid sizing)
    int begin_bit, end_bit;
    uint32_t* hist;              // digit histograms of the passes (zeroed before the sort)
    int hist_ready;              // 1: the producer of the keys already filled `hist`
    SortPlan* plan;              // zeroed before the sort
    unsigned long long* status;  // look-back words, tagged with the epoch and the pass
    uint32_t epoch;
    uint32_t* error_flags;
    uint32_t key_bias = 0;       // digits are those of key + key_bias (modulo 2^32)
    int first_pdl = 0;           // 1: the first pass too is a programmatic dependent launch
};

// Tile entries whose id's upper bits and sorted position fit one word.
struct TileSortParams {
    const uint8_t* low;          // lower 8 id bits of every entry
    uint32_t* words[3];          // (id >> 8) << vbits | position: input, after the first pass, after the second
    int vbits;
    int last_pass;               // 0: at most 256 tiles, one pass; its output and the second's are bare positions
    const uint32_t* count_ptr;   // entries (device)
    uint32_t count_cap;
    const uint32_t* hist;        // 2 x 256: lower and upper digits of the ids
    SortPlan* plan;              // zeroed before the sort; vfinal = the sorted positions
    unsigned long long* status;
    uint32_t epoch;
    uint32_t* error_flags;
    uint2* ranges;               // per tile (~start, end), zeroed before the sort
    uint32_t num_tiles;
};

struct BinParams {
    const SortPlan* depth_plan;      // sorted ids at depth_plan->vfinal
    const float4* projected;
    float vp_w, vp_h, clip_y_sign;   // CameraUniforms viewport and clip_y_sign of the frame
    float jitter_x, jitter_y;
    int width, height, tiles_x, tiles_y;
    int tile_shift_x, tile_shift_y;  // log2 of the tile width and height
    RasterRecord* records;           // N_vis records (sorted order)
    uint32_t* entry_keys;            // tile id per entry (entry_vbits < 0), or its lower 8 bits, a byte per entry
    uint32_t* entry_vals;            // sorted position per entry, with (id >> 8) << entry_vbits above it
    int entry_vbits;
    uint32_t entry_cap;
    uint4* item_info;                // per binned item: first entry, tx0 | ty0 << 16, width in tiles (0: none)
    uint32_t* chunk_first;           // per expansion chunk: the item owning its first entry
    uint32_t chunk_cap;              // chunk_first capacity (entry_cap / kBinChunk + 2)
    uint32_t* tile_hist;             // 3 x 256 digit histograms of the tile ids (zeroed per pass)
    unsigned long long* status;      // per-CTA-tile look-back words (epoch-tagged)
    uint32_t epoch;
    FrameCounters* fc;
    // 1: stochastic envelope mode.  Tiles are chosen for every sub-pixel
    // jitter in [-0.5, 0.5]^2 at once and the records keep the un-jittered
    // quad (centre, radii, ndc_z), so one binning serves all samples of a
    // frame; the rasterizer derives each sample's coverage.
    int envelope;
};

struct RasterParams {
    const RasterRecord* records;
    uint32_t record_cap;             // records allocated (bounds every record index)
    const SortPlan* tile_plan;       // tile-sorted entry values at tile_plan->vfinal
    const uint2* tile_ranges;        // [start, end) per tile
    const uint32_t* tile_order;      // tiles by descending work (CTA b rasterizes tile_order[b])
    const float* tile_err;           // optional: only tiles with tile_err[tile] >= err_budget are drawn
    float err_budget;
    const float4* colours;           // state batches: per record the colours of kStates frames (StateBatch)
    int width, height, tiles_x, tiles_y;
    int tile_w, tile_h;              // tile shape: 16x16, or 32x8 / 8x32 (alpha mode)
    float bg;
    // stochastic mode (envelope records): the sample's jitter and seed, and
    // the viewport of the quad computation
    float jitter_x, jitter_y, frame_seed;
    float frame_seed2;               // two-sample mode: the second sample's seed (frame_seed is the first's)
    float vp_w, vp_h, clip_y_sign;
    uint16_t* out_rgba16f;           // width*height*4 halves, top row first
    float4* out_rgba32f;             // optional float copy (stochastic sample), top row first
    float* out_depth;                // optional window depth (stochastic), top row first
    // optional running mean of the samples (stochastic): accum_out = h + (sample - h) / max(accum_n, 1)
    // with h = accum_in, or the sample itself when accum_in is null (accum_kernel's arithmetic)
    const float4* accum_in;
    float4* accum_out;
    float accum_n;
    int rgba8;                       // quantise stochastic sample like RGBA8 UNORM
    FrameCounters* fc;
};

// Launch with programmatic stream serialization: the kernel may be scheduled
// while its predecessor in the stream finishes, and calls pdl_wait() before
// it reads or writes anything the predecessor touches.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                              Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// What has to be done once on every device a process launches on (a kernel's
// shared-memory limit is an attribute per device): runs `set` unless it has run
// for `device`.  The mark comes after it, so that a thread which finds the mark
// finds the attribute; threads that meet before it set the same twice.
class OncePerDevice {
public:
    template <class F>
    void operator()(int device, F&& set) {
        const uint64_t bit = device >= 0 && device < 64 ? 1ull << device : 0ull;   // others: every time
        if (done_.load() & bit) return;
        set();
        done_.fetch_or(bit);
    }

private:
    std::atomic<uint64_t> done_{0};
};

// Every device allocation of the library goes through here: cudaMalloc, with
// a failed call's error cleared (it is reported through the return value),
// and the allocation-failure injection of gs_debug_fail_alloc.
cudaError_t device_malloc(void** p, size_t bytes);

// Launchers (each returns the number of kernels it launched).
int launch_cull(const CullParams& p, uint32_t num_sms, cudaStream_t s);
int launch_gather_heads(const float4* rows, float4* heads, uint32_t n, uint32_t num_sms, cudaStream_t s,
                        uint32_t row_chunks = 16);
int launch_pack_half_rows(const float4* rows, float4* half_rows, uint32_t n, uint32_t num_sms, cudaStream_t s);
// State batches (gs_render_anim_batch): frames of one geometry that differ in
// colours only.  The frames are taken in groups of 8 (the last one of 4 when
// that holds the rest); a group's colours lie together per record, channel
// by channel: 3 x group-width floats, group after group, cap records each.  1M
// Gaussians, 1920x1080: one to four frames take 534, 558, 588, 611 us in a group of
// 4 (667, 1087, 1479, 1923 when each was drawn alone), five to eight 732 to 792 in
// one of 8.
constexpr int kMaxBatchFrames = 256;
struct StateBatch {
    int32_t a[kMaxBatchFrames], b[kMaxBatchFrames];   // appearance states of each frame and
    float w[kMaxBatchFrames];                         // their blend weight (gs_set_anim_state)
};
struct StateOuts {
    uint16_t* out[kMaxBatchFrames];
};
inline int state_groups8(int frames) { return frames / 8 + (frames % 8 > 4 ? 1 : 0); }
inline int state_groups4(int frames) { return frames % 8 > 0 && frames % 8 <= 4 ? 1 : 0; }
inline size_t state_colour_floats(size_t cap, int frames) {
    return cap * (24u * (size_t)state_groups8(frames) + 12u * (size_t)state_groups4(frames));
}
int launch_recolour_states(const CullParams& p, const RasterRecord* records, const StateBatch& st, int frames,
                           float* colours, uint32_t num_sms, cudaStream_t s);
int launch_sort(const SortParams& p, uint32_t num_sms, cudaStream_t s);         // 8-bit digits, any bit range
int launch_depth_sort(const SortParams& p, uint32_t num_sms, cudaStream_t s);   // 9-bit digits, histograms ready
int launch_tile_sort(const TileSortParams& p, uint32_t num_sms, cudaStream_t s);
int launch_bin(const BinParams& p, uint32_t n_cap, uint32_t num_sms, cudaStream_t s);
int launch_tile_ranges(const SortPlan* tile_plan, const FrameCounters* fc, uint32_t entry_cap, uint2* ranges,
                       uint32_t num_tiles, uint32_t num_sms, cudaStream_t s);
// turned: the ranges are (~start, end) (launch_tile_sort) and are turned round here
int launch_tile_order(uint2* ranges, uint32_t num_tiles, uint32_t* order, bool turned, cudaStream_t s);
int launch_raster_alpha(const RasterParams& p, cudaStream_t s);
int launch_raster_stochastic(const RasterParams& p, cudaStream_t s);
int launch_raster_stochastic2(const RasterParams& p, cudaStream_t s);
// alpha frames[f] for f < nframes in one persistent launch (first: nframes + 1
// prefix sums of the frames' tile counts, device; ticket: a zeroed device word)
int launch_raster_batch_alpha(const RasterParams* frames, const uint32_t* first, uint32_t nframes, uint32_t* ticket,
                              uint32_t grid, int tile_w, cudaStream_t s);
void raster_batch_occupancy(int* blocks_per_sm);
// the frames of a state batch into outs (p.colours: launch_recolour_states' buffer of p.record_cap records a group)
int launch_raster_states(const RasterParams& p, const StateOuts& outs, int frames, cudaStream_t s);

int launch_wait_probe(const unsigned long long* status, FrameCounters* fc, uint32_t epoch, int which, uint32_t limit,
                      cudaStream_t s);

size_t sort_status_words(uint32_t count_cap);   // a quarter of a sort's look-back words
int sort_passes(int begin_bit, int end_bit);
}  // namespace gs
