// Device-side layout of one fused batch launch: the per-sample programs the
// kernel executes and the launch-wide parameters.  Host code fills these from
// the public descriptors (include/mlxd_b200.h) after validating them.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cstring>

namespace mlxd {

constexpr int kTileH = 16;    // copies and rotations: output rows per CTA
constexpr int kTileW = 64;    // and output pixels per tile of a copy
constexpr int kThreads = 256;

// Resize kernel (resize_strip.cu): a warp walks down a strip of output columns.
constexpr int kStripThreads = 128;
constexpr int kStripCtas = 5;         // per SM
constexpr int kStripRow = 241;        // source bytes of a strip: 16 units of 16 bytes, whichever byte of a unit they start at
constexpr int kStripMaxRows = 32;     // output rows per warp
constexpr int kStripSlots = 14;       // source rows of a part, which are in shared memory together
constexpr int kStripMaxSteps = 320;   // steps of a warp's walk
constexpr int kStripMaxPx = 256;      // output columns per strip
// Horizontal weights per strip: 32 * ceil(px / 32) columns of floor(2r) + 2 taps.  A
// shrink by r has px * r <= kStripRow, so 2 * 241 + 2 * 256 columns and taps bound them
// twice over; below 32 columns r is at most kStripRow / (kStripMinPx + 1).
// A strip of fewer columns is left to resize_walk.cu: a shrink along a row alone by 6 (12
// columns a strip) is 6 % faster in strips, by 7 (10 columns) 25 % slower, by 15 (4) 45 %.
constexpr int kStripMinPx = 11;
constexpr int kStripMaxTaps = 32 * (2 * kStripRow / (kStripMinPx + 1) + 4);

// Resize kernel of strong shrinks and what goes with them (resize_walk.cu): a CTA walks down
// a chunk of columns.
constexpr int kWalkThreads = 128;
constexpr int kWalkRow = 832;       // floats per row in shared memory: source bytes of a chunk, alignment included
constexpr int kWalkMaxRows = 32;    // output rows per CTA
constexpr int kWalkMaxSteps = 1024; // source rows walked per CTA
constexpr int kWalkMaxPx = 128;     // output columns per CTA
// Horizontal weights per CTA: px columns of floor(2r) + 2 taps.  A shrink by r has
// px * r <= kWalkRow (the chunk's source columns), so 2 * kWalkRow + 2 * kWalkMaxPx
// bounds them; an enlargement has 4 * kWalkMaxPx.
constexpr int kWalkMaxTaps = 2 * kWalkRow + 2 * kWalkMaxPx;
constexpr int kPadChunks = 128;     // CTAs that fill the rows below one sample
constexpr int kWalkPadPx = 256;     // columns per strip of padding

// kModeResizeDirect: a resize whose taps do not fit one chunk of the resize
// kernel: one column's 2r + 2 source columns exceed kWalkRow bytes (shrink ratios r
// above 412, 205, 136, 102 along a row for 1 to 4 channels) or one row's 2r + 11
// steps exceed kWalkMaxSteps (above 506 down the rows).  Every output pixel is then
// filtered straight from global memory by resize_direct_kernel.
// kModeResizeWide: a resize that resize_walk.cu runs: one too strong for resize_strip.cu, or
// one of a batch that goes there (launch_plan.cu: choose_resize_kernel).
enum Mode : int32_t { kModeCopy = 0, kModeResize = 1, kModeAffine = 2, kModeResizeDirect = 3, kModeResizeWide = 4 };

// One sample's program.  Coordinates name four nested images:
//   source [src_h, src_w] -> pre window [pre_h, pre_w] (+mirror)
//   -> geometric output [geom_h, geom_w] -> post window [post_h, post_w] (+mirror)
// and the post window lands in the top-left corner of the slot [slot_h, slot_w].
struct __align__(16) DevSample {
  const uint8_t* src;
  void* dst;
  int32_t src_h, src_w;
  int32_t pre_x, pre_y, pre_w, pre_h;
  int32_t geom_w, geom_h;
  int32_t post_x, post_y, post_w, post_h;
  int32_t slot_h, slot_w;
  int32_t mode;
  int32_t pre_flip, post_flip;
  int32_t cap_x;          // resize: bound on the horizontal tap count
  int32_t walk_px;        // resize kernels: most output columns of a strip (chunk),
  int32_t walk_chunks;    // strips that share the post window's columns,
  int32_t walk_rows;      // output rows per warp (CTA)
  union {
    float mx[6];          // affine
    struct {
      float axis_x[2], axis_y[2];   // resizes: Axis::ratio and Axis::fs
      float stage_cost;             // the planner's, of four output rows of a strip
    };
  };
  // resize_strip.cu: output rows whose source rows are in shared memory together (1, 2 or 4), those
  // source rows << 8, and steps of a warp's walk << 16, at most
  int32_t walk_sizes;
};

// What the resize kernel of one launch is sized by: the largest needs of its samples.
struct StripPlan {
  int32_t bytes;      // shared memory of a strip, without cast tables (0: no sample runs the kernel)
  int32_t steps;      // steps of a warp's walk
  int32_t cells_y;    // grid of cells of every sample, the most rows and the most columns of any of them;
  int32_t cells_x;    // or 0 rows: cells_x CTAs per sample, which counts its own cells off
  // with LaunchParams::pad_apart, set at launch: CTAs that walk; the first blocks, which hold
  // all of these; and the share of those blocks that fill, times 2^32
  uint32_t walks, mixed_blocks, fill_ratio;
  int32_t linear;        // blocks are numbered through, not by three coordinates (set at launch)
};

// The same for resize_walk.cu.
struct WalkPlan {
  int32_t px;         // columns of the widest chunk (0: no sample runs the resize kernel)
  int32_t taps;       // horizontal weights of a chunk
  int32_t steps;      // source rows of a walk
  int32_t cells_y;    // grid of cells of every sample, the most rows and the most columns of any of them;
  int32_t cells_x;    // or 0 rows: cells_x CTAs per sample, which counts its own cells off
};

// Both, and the samples the second one runs for.
struct ResizePlan {
  StripPlan strip;
  WalkPlan wide;
  int32_t first_wide, wides;   // all of them are among these samples
  int32_t first_band, bands;   // and the samples of the band kernel (and the direct one) among these
  int32_t first_affine, affines;   // and those of affine.cu among these
  bool enlarges;      // most resizes enlarge along the row
};

__host__ __device__ inline bool is_resize(const DevSample& s) {
  return s.mode == kModeResize || s.mode == kModeResizeWide || s.mode == kModeResizeDirect;
}

// Strips of padding beside the post window.
__host__ __device__ inline int walk_strips(const DevSample& s) {
  return (s.slot_w - s.post_w + kWalkPadPx - 1) / kWalkPadPx;
}

// The cast of a float32 batch as steps that give the table's values bit for bit (context.cu:
// cast_steps): x = v * r, then for kCastNormalise (x + neg_mean) * s, each factor a sum of two
// floats, every float twice as an operand of the packed instructions.
enum CastMode : int32_t { kCastTable = 0, kCastScale = 1, kCastNormalise = 2 };
struct CastSteps {
  float r_hi[2], r_lo[2];
  float neg_mean[4][2], s_hi[4][2], s_lo[4][2];
  int32_t mode;   // kCastTable: no such steps, or the channel reduction's
};

struct LaunchParams {
  const DevSample* samples;   // in device memory, or null: `carried`
  const DevSample* carried;   // in host memory, for the launch to take along (carried_samples)
  int32_t n;
  int32_t first;              // the launch's samples are these from `first` on
  int32_t tiles_y, tiles_x;   // tile grid of the largest slot
  int32_t c_in;               // channels of every source
  int32_t c_out;              // 1 when gray, else c_in
  int32_t gray;
  int32_t gray_m[3];
  int32_t gray_bias;
  int32_t out_f32;
  const float* lut;           // [c_out][256] cast table, device
  CastSteps cast;
  int32_t pad_px;             // pad value as a pixel
  int32_t* status;            // device word, non-zero once a self-check failed
  int32_t band_tiles;         // band kernel: tiles per CTA along a row band (set at launch)
  int32_t bands_x;            // band kernel: CTAs per row band
  WalkPlan walk;              // resize_walk.cu: ResizePlan::wide
  int32_t pad_apart;          // the rows below each post window are filled apart from the cells around them
  int32_t fill_every;         // resize kernels, then: every so many CTAs, from the first on, one of them fills
  int32_t direct;             // some sample is kModeResizeDirect: resize_direct_kernel runs last
};

// Sample records as a kernel's parameter: up to K of them, or (0) none, where they are read
// from LaunchParams::samples.  A kernel may have 32 764 bytes of parameters; each launch
// moves all of them, so there are two sizes.  4 images of 480x640 to 224x224 take 10.8 us a pass
// with 24, 13.2 with 128, 15.3 with a table copied ahead of the kernel; 32 of 200-500 px 17.5 with
// 128 and 20.9 with a table.  240, the most that fit, in place of 128 take 0.5 to 1 us off
// batches of 129 to 240 (160 of 64x64 28.5 us a pass, 27.5; 240 of 200-500 px 77.2, 76.4) and put up to
// 2 on those of 25 to 128 (64 of 64x64 18.4 us, 20.1; 128 of 256x256 rotated 45.2, 46.8).
constexpr int kFewSamples = 24, kMoreSamples = 128;

template <int K>
struct Records {
  DevSample at[K];
  __device__ __forceinline__ const DevSample* of(const LaunchParams& p, unsigned t) const { return at + p.first + t; }
  __device__ __forceinline__ const DevSample* whole(const LaunchParams& p, unsigned t) const { return of(p, t); }
};

template <>
struct Records<0> {
  __device__ __forceinline__ const DevSample* of(const LaunchParams& p, unsigned t) const { return p.samples + p.first + t; }
  // The record asked for as a whole, for a CTA that reads it field by field as it decides what it
  // needs, and waited for each of its four sectors: 512 full-HD frames 1100 -> 1097 us.  CTAs of
  // little work wait longer for what is asked: with it, those that fill padding and the bands took
  // 1.02 to 1.34 times as long (200 one-channel images of 200-400 px padded to the largest, bytes,
  // 87 us, 64 without; 500 of 200-500 px, shorter side 128, 178 and 163).
  __device__ __forceinline__ const DevSample* whole(const LaunchParams& p, unsigned t) const {
    const DevSample* const s = of(p, t);
#ifdef __CUDA_ARCH__
    asm volatile("prefetch.global.L1 [%0];" ::"l"(reinterpret_cast<const char*>(s) + 32 * (threadIdx.x & 3)));
#endif
    return s;
  }
};

// launch(records) with the records of a launch's samples.
template <class F>
inline cudaError_t with_records(const LaunchParams& p, F&& launch) {
  if (p.samples) {
    return launch(Records<0>{});
  }
  const int count = p.first + p.n;
  if (count <= kFewSamples) {
    Records<kFewSamples> r;
    std::memcpy(r.at, p.carried, sizeof(DevSample) * count);
    return launch(r);
  }
  Records<kMoreSamples> r;
  std::memcpy(r.at, p.carried, sizeof(DevSample) * count);
  return launch(r);
}

// Channels of cast tables that a resize kernel keeps in shared memory.
__host__ __device__ inline int table_channels(const LaunchParams& p) {
  return p.out_f32 && p.cast.mode == kCastTable ? p.c_out : 0;
}

// Whether launches can carry their samples: those of the kernels for strong shrinks are read from a table.
inline bool carried_samples(const LaunchParams& p, const ResizePlan& plan) {
  return p.n <= kMoreSamples && plan.wide.px == 0 && !p.direct;
}

// Launch the kernels the parameters call for: the resize kernel or, without a
// resize and when p.pad_apart is set, pad_fill_kernel, affine_kernel, the band kernel,
// resize_direct_kernel.
cudaError_t launch_fused_batch(const LaunchParams& p, const ResizePlan& plan, cudaStream_t stream);
cudaError_t launch_resize_strip(const LaunchParams& p, const StripPlan& plan, cudaStream_t stream);
cudaError_t launch_affine(const LaunchParams& p, cudaStream_t stream);
cudaError_t launch_resize_walk(const LaunchParams& p, bool fills_padding, cudaStream_t stream);

// axis_x, axis_y (the divisions of make_axis(), correctly rounded here as there) and
// cap_x of a resize.
void set_axes(DevSample& s);

// The kernel that runs a resize, its axes set.
Mode resize_mode(DevSample& s, int channels);

// Split the resize samples of a batch into CTAs (DevSample::walk_*) and size
// the launches.
void plan_resize(DevSample* samples, int n, int channels, ResizePlan& plan);

// Samples by which the distance of two taps of an axis of n source samples can exceed
// its exact value, beyond the one that the bounds below always add: a tap's position
// goes through at most four float32 roundings (and the ratio's), each of them half a
// unit in the last place of n, together below n * 2^-22, at either end.
__host__ __device__ constexpr int32_t axis_slack(int32_t n) {
  return n >> 21;
}

// Shared memory of a CTA of resize_strip.cu, laid out for its own sample: in an unlike batch
// the samples have their largest needs in different places, and every CTA has room for the
// largest sum.  256 of 256-800 px to 224x224: 51 KB with room for the largest of each, 44.7 so, of which
// five fit an SM: 113.3 us a pass and 105.4.
struct StripSmem {
  unsigned mid;      // per warp: float4 [256]
  unsigned lut;      // float [tables][256]
  unsigned ring;     // per warp: source rows [slots]
  unsigned weights;  // per warp: {wa, wa, wb, wb} per step
  unsigned places;   // per warp: {address of lane 0's word A, funnel shift} per step
  unsigned parts;    // per warp: {first, last source row} per part
  unsigned hx;       // {tap offset | taps << 16, column} per column
  unsigned hw;       // float [tap][columns]
  unsigned count;    // per warp: byte [kStripMaxRows]  steps of every output row
  unsigned ring_bytes, parts_bytes;
  int steps, slots, part_rows;
};

constexpr unsigned kStripSlotBytes = 272;                // a row's 16 units of 16 bytes, and the word behind them
constexpr unsigned kStripMidBytes = 256 * 16;            // four rows of 256 byte columns

__host__ __device__ inline unsigned strip_layout(const DevSample& s, int tables, unsigned base, StripSmem* out) {
  constexpr unsigned kWarps = kStripThreads / 32;
  StripSmem sm;
  sm.steps = s.walk_sizes >> 16;
  sm.slots = (s.walk_sizes >> 8) & 255;
  sm.part_rows = s.walk_sizes & 255;
  sm.ring_bytes = (unsigned)sm.slots * kStripSlotBytes;
  sm.parts_bytes = (unsigned)s.walk_rows * 8u >> (sm.part_rows >> 1);   // (walk_rows is a multiple of four)
  const unsigned columns = (unsigned)(s.walk_px + 31) / 32 * 32;
  sm.mid = base;
  sm.lut = sm.mid + kWarps * kStripMidBytes;
  sm.ring = sm.lut + (unsigned)tables * 1024u;
  sm.weights = sm.ring + kWarps * sm.ring_bytes;
  sm.places = sm.weights + kWarps * (unsigned)sm.steps * 16u;
  sm.parts = sm.places + kWarps * (unsigned)sm.steps * 8u;
  sm.hx = sm.parts + kWarps * sm.parts_bytes;
  sm.hw = sm.hx + columns * 8u;
  sm.count = sm.hw + columns * (unsigned)s.cap_x * 4u;
  if (out) {
    *out = sm;
  }
  return (sm.count + kWarps * kStripMaxRows + 15u - base) & ~15u;
}

// Which kernels a launch needs and their grids; call after plan_resize with the
// host copy of the sample table.
void choose_kernels(LaunchParams& p, ResizePlan& plan, const DevSample* host_samples, int n);

// Conservative per-axis bounds used by the host planner.
struct AxisPlan {
  int32_t cap;      // tap-count bound
  int32_t extent;   // bound on source samples touched by `sub` outputs
};
AxisPlan plan_axis(int32_t n_src, int32_t n_dst, int32_t sub);

} // namespace mlxd
