// Host side of a launch: which kernels run it, and how the resize samples are
// split into CTAs.
//
// Reference behaviour the kernels reproduce (paths inside mlx-data):
//   resize             mlx/data/core/image/ImageTransform.cpp:41-62 (triangle filter, clamp to edge)
//   crop               mlx/data/core/image/ImageTransform.cpp:64-73, mlx/data/Array.cpp:544-583
//   affine / rotate    mlx/data/core/image/ImageTransform.cpp:75-121
//   hflip              mlx/data/core/image/ImageTransform.cpp:123-140
//   channel_reduction  mlx/data/core/image/ImageTransform.cpp:142-182
//   batch + pad        mlx/data/Array.cpp:465-498, mlx/data/core/BatchShape.cpp:26-45
//   cast               README.md:55-57 (x.astype(float32) / 255 and its normalised form)
#include <algorithm>
#include <cmath>

#include "fused_batch.h"

namespace mlxd {

void choose_kernels(LaunchParams& p, const DevSample* host_samples, int n) {
  p.bands = 0;
  p.direct = 0;
  unsigned long long rows = 0, below = 0;
  for (int i = 0; i < n; i++) {
    const DevSample& s = host_samples[i];
    p.bands |= s.mode != kModeResize;   // a direct sample's padding is the band kernel's too
    p.direct |= s.mode == kModeResizeDirect;
    rows += (unsigned long long)s.slot_h;
    below += (unsigned long long)(s.slot_h > s.post_h ? s.slot_h - s.post_h : 0);
  }
  // The rows below a sample's post window are one contiguous run of its slot;
  // when those runs are at least an eighth of the batch they get a linear fill
  // of their own (CTAs of the resize kernel, else pad_fill_kernel), which writes
  // at memory speed.
  p.pad_apart = n > 0 && below * 8 >= rows ? 1 : 0;
  p.walk.cells_y = p.walk.cells_x = 0;
  long long own = 0;
  for (int i = 0; i < n; i++) {
    const DevSample& s = host_samples[i];
    if (s.mode == kModeResize) {
      const int h = p.pad_apart ? s.post_h : s.slot_h;
      const int cells_y = (h + s.walk_rows - 1) / s.walk_rows;
      const int cells_x = s.walk_chunks + walk_strips(s);
      p.walk.cells_y = std::max(p.walk.cells_y, cells_y);
      p.walk.cells_x = std::max(p.walk.cells_x, cells_x);
      own = std::max(own, (long long)cells_y * cells_x);
    }
  }
  // A tall strong shrink beside a wide one would multiply the rows of the one by the
  // columns of the other, for every sample: 1022 images of 32-120 px, one of 22400x60
  // and one of 60x22400, to 224x224, take 27.2 ms a pass in one grid and 1.71 when every
  // sample counts its own cells.  That costs each CTA a division by its sample's count
  // (128 images enlarged to 224x224: 58 us a pass instead of 55), so it is left to batches
  // whose common grid has twice the cells of the largest sample.
  if ((long long)p.walk.cells_y * p.walk.cells_x >= 2 * own && own <= 0x7fffffff) {
    p.walk.cells_y = 0;
    p.walk.cells_x = (int32_t)own;
  }
}

AxisPlan plan_axis(int32_t n_src, int32_t n_dst, int32_t sub) {
  AxisPlan a;
  if (n_src <= n_dst) {
    a.cap = 4;
    a.extent = sub + 4;
    return a;
  }
  // Output o reads taps ceil(u - R) .. floor(u + R) with u = (o + 0.5) * ratio - 0.5
  // and R = ratio: at most floor(2R) + 1 of them, and `sub` consecutive
  // outputs span at most (sub - 1) * ratio + 2R + 1 source samples.  One more
  // of each covers the float32 rounding of u and R in the kernel.
  const double ratio = (double)n_src / (double)n_dst;
  a.cap = (int32_t)std::floor(2.0 * ratio) + 2;
  a.extent = (int32_t)std::ceil((double)(sub - 1) * ratio + 2.0 * ratio) + 2;
  return a;
}

// Source bytes of `px` output columns, from the word that holds the first one.
static long long walk_row_bytes(const DevSample& s, int channels, int px) {
  const long long cols = std::min(plan_axis(s.pre_w, s.geom_w, px).extent, s.pre_w);
  return cols * channels + 6;
}

// Steps of a walk over `rows` output rows: every source row once, again once
// per output row whose neighbours on both sides reach it, one per output row
// at least.  (Enlargements walk the two rows of every output row.)
static long long walk_steps(const DevSample& s, int rows) {
  const long long extent = plan_axis(s.pre_h, s.geom_h, rows).extent;
  return s.pre_h <= s.geom_h ? 4LL * rows + 4 : extent + rows + 8;
}

bool walk_fits(const DevSample& s, int channels) {
  return walk_row_bytes(s, channels, 1) <= kWalkRow && walk_steps(s, 1) <= kWalkMaxSteps &&
      (long long)s.src_w * channels < (1LL << 31);
}

// Chunks of at most `px` columns and walks of at most `rows` rows, smaller
// where the source footprint asks for it.
static void split_walk(DevSample& s, int channels, int px, int rows) {
  if (walk_row_bytes(s, channels, px) > kWalkRow) {
    // (px + 1) * ratio + 3 source columns at most (plan_axis), then down to what fits
    const double ratio = (double)s.pre_w / (double)s.geom_w;
    const int guess = s.pre_w <= s.geom_w ? px : (int)(kWalkRow / channels / ratio);
    px = std::max(1, std::min(px, guess));
    while (px > 1 && walk_row_bytes(s, channels, px) > kWalkRow) {
      px--;
    }
  }
  while (rows > 1 && walk_steps(s, rows) > kWalkMaxSteps / 4) {
    rows /= 2;
  }
  s.walk_chunks = (s.post_w + px - 1) / px;
  s.walk_px = (s.post_w + s.walk_chunks - 1) / s.walk_chunks;
  s.walk_rows = rows;
}

void plan_walk(DevSample* samples, int n, int channels, WalkPlan& plan) {
  // The largest cells that still give every one of a B200's 148 SMs two CTAs (another
  // count would only choose other cells).  A CTA
  // builds its tables and walks 2 r source rows (shrink ratio r) before its first
  // output row is complete, so smaller cells cost more as soon as the SMs have
  // work: 512 frames of 1080x1920 to 512x512 take 1.37 ms in 128x32 cells, 1.46
  // in 128x16, 1.58 in 64x32, 3.4 in 64x4; 32 images of 200-500 px to 224x224
  // 32 us in 448 CTAs of 128x32 and in 1792 of 128x8, 52 us in 64x4.  One 480x640
  // image to 224x224 fills no wave of any size and is quickest in the smallest
  // cells: 14.4 us a call in 64x4, 18 in 128x8.
  static const int kCells[][2] = {{kWalkMaxPx, 32}, {kWalkMaxPx, 16}, {kWalkMaxPx, 8}, {64, 8}, {64, 4}};
  constexpr long long kWantCtas = 148 * 2;
  for (const auto& cell : kCells) {
    long long ctas = 0;
    plan = WalkPlan{0, 0, 0, 0, 0};
    for (int i = 0; i < n; i++) {
      DevSample& s = samples[i];
      if (s.mode == kModeResize) {
        split_walk(s, channels, cell[0], cell[1]);
        ctas += (long long)s.walk_chunks * ((s.post_h + s.walk_rows - 1) / s.walk_rows);
        plan.px = std::max(plan.px, s.walk_px);
        plan.taps = std::max(plan.taps, s.walk_px * s.cap_x);
        plan.steps = std::max(plan.steps, (int32_t)walk_steps(s, s.walk_rows));
      }
    }
    if (ctas == 0 || ctas >= kWantCtas) {
      return;
    }
  }
}

} // namespace mlxd
