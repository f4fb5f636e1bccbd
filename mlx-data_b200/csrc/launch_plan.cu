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

// The grid of one resize kernel: `rows` and `columns` of cells of a sample.
namespace {
struct Cells {
  int32_t y = 0, x = 0;
  long long own = 0;   // of the largest sample

  void add(int rows, int columns) {
    y = std::max(y, rows);
    x = std::max(x, columns);
    own = std::max(own, (long long)rows * columns);
  }
  // A tall strong shrink beside a wide one would multiply the rows of the one by the
  // columns of the other, for every sample: 1022 images of 32-120 px, one of 22400x60
  // and one of 60x22400, to 224x224, take 27.2 ms a pass in one grid and 1.71 when every
  // sample counts its own cells.  That costs each CTA a division by its sample's count
  // (128 images enlarged to 224x224: 58 us a pass instead of 55), so it is left to batches
  // whose common grid has twice the cells of the largest sample.
  void put(int32_t& cells_y, int32_t& cells_x) const {
    const bool each = (long long)y * x >= 2 * own && own <= 0x7fffffff;
    cells_y = each ? 0 : y;
    cells_x = each ? (int32_t)own : x;
  }
};
} // namespace

void choose_kernels(LaunchParams& p, ResizePlan& plan, const DevSample* host_samples, int n) {
  p.direct = 0;
  plan.first_band = plan.bands = plan.first_affine = plan.affines = 0;
  unsigned long long rows = 0, below = 0;
  for (int i = 0; i < n; i++) {
    const DevSample& s = host_samples[i];
    if (s.mode == kModeAffine) {
      plan.first_affine = plan.affines == 0 ? i : plan.first_affine;
      plan.affines = i + 1 - plan.first_affine;
    } else if (s.mode != kModeResize && s.mode != kModeResizeWide) {   // a direct sample's padding is the band kernel's too
      plan.first_band = plan.bands == 0 ? i : plan.first_band;
      plan.bands = i + 1 - plan.first_band;
    }
    p.direct |= s.mode == kModeResizeDirect;
    rows += (unsigned long long)s.slot_h;
    below += (unsigned long long)(s.slot_h > s.post_h ? s.slot_h - s.post_h : 0);
  }
  // The rows below a sample's post window are one contiguous run of its slot;
  // when those runs are at least an eighth of the batch they get a linear fill
  // of their own (CTAs of a resize kernel, else pad_fill_kernel), which writes
  // at memory speed.
  p.pad_apart = n > 0 && below * 8 >= rows ? 1 : 0;
  Cells strip, wide;
  plan.first_wide = plan.wides = 0;
  int enlarged = 0, resized = 0;
  for (int i = 0; i < n; i++) {
    const DevSample& s = host_samples[i];
    const int h = p.pad_apart ? s.post_h : s.slot_h;
    resized += is_resize(s);
    enlarged += is_resize(s) && s.pre_w < s.geom_w;
    if (s.mode == kModeResize) {
      const int cell_rows = s.walk_rows * (kStripThreads / 32);
      strip.add((h + cell_rows - 1) / cell_rows, s.walk_chunks + walk_strips(s));
    } else if (s.mode == kModeResizeWide) {
      wide.add((h + s.walk_rows - 1) / s.walk_rows, s.walk_chunks + walk_strips(s));
      plan.first_wide = plan.wides == 0 ? i : plan.first_wide;
      plan.wides = i + 1 - plan.first_wide;
    }
  }
  strip.put(plan.strip.cells_y, plan.strip.cells_x);
  wide.put(plan.wide.cells_y, plan.wide.cells_x);
  plan.enlarges = 2 * enlarged > resized;
  p.walk = plan.wide;
}

AxisPlan plan_axis(int32_t n_src, int32_t n_dst, int32_t sub) {
  AxisPlan a;
  const int32_t slack = axis_slack(n_src);
  if (n_src <= n_dst) {
    a.cap = 4 + slack;
    a.extent = sub + 4 + slack;
    return a;
  }
  // Output o reads taps ceil(u - R) .. floor(u + R) with u = (o + 0.5) * ratio - 0.5
  // and R = ratio: at most floor(2R) + 1 of them, and `sub` consecutive
  // outputs span at most (sub - 1) * ratio + 2R + 1 source samples.  One more
  // of each and the slack cover the float32 rounding of u and R in the kernel.
  const double ratio = (double)n_src / (double)n_dst;
  a.cap = (int32_t)std::floor(2.0 * ratio) + 2 + slack;
  a.extent = (int32_t)std::ceil((double)(sub - 1) * ratio + 2.0 * ratio) + 2 + slack;
  return a;
}

// Source bytes of `px` output columns, from the word that holds the first one.
static long long walk_row_bytes(const DevSample& s, int channels, int px) {
  const long long cols = std::min(plan_axis(s.pre_w, s.geom_w, px).extent, s.pre_w);
  return cols * channels + 6;
}

// Steps of a walk over `rows` output rows: every source row once, again once
// per output row whose neighbours on both sides reach it, one per output row
// at least.  (Enlargements walk the two rows of every output row.)  Rounding lets
// neighbours reach that much further into each other.
static long long walk_steps(const DevSample& s, int rows) {
  const long long extent = plan_axis(s.pre_h, s.geom_h, rows).extent;
  const long long again = (long long)rows * axis_slack(s.pre_h);
  return again + (s.pre_h <= s.geom_h ? 4LL * rows + 4 : extent + rows + 8);
}

// Whether one output column and one output row fit a chunk of resize_walk.cu.
static bool walk_fits(const DevSample& s, int channels) {
  return walk_row_bytes(s, channels, 1) <= kWalkRow && walk_steps(s, 1) <= kWalkMaxSteps && s.cap_x <= kWalkMaxTaps;
}

// Source columns of `px` output columns of a strip.  The last of them is centred
// (px - 1) ratios behind the first, and both reach one radius further; two more
// columns and the slack cover the ends' fractions and the float32 rounding of the kernel.
static int strip_columns(const DevSample& s, int px) {
  const float ratio = s.axis_x[0];
  const float span = std::min(1e6f, (float)(px - 1) * ratio + 2.0f * std::max(1.0f, ratio));
  const int whole = (int)span;
  return whole + (whole < span) + 2 + axis_slack(s.pre_w);
}

// The widest strip that fits; 0 when not even one column does.
static int strip_most_px(const DevSample& s, int channels) {
  const int most = std::min(s.post_w, kStripMaxPx);
  if ((long long)s.pre_w * channels <= kStripRow) {
    return most;
  }
  const int columns = kStripRow / channels;
  const float ratio = s.axis_x[0];
  const float guess = ((float)(columns - 2) - 2.0f * std::max(1.0f, ratio)) / ratio + 1.0f;
  int px = guess < (float)most ? std::max(0, (int)guess) : most;
  while (px > 0 && strip_columns(s, px) > columns) {
    px--;
  }
  return px;
}

// Bound on the source rows that `rows` output rows read.
static int strip_span(const DevSample& s, int rows) {
  const float ratio = s.axis_y[0];
  const float span = (float)(rows - 1) * ratio + 2.0f * (ratio > 1.0f ? ratio : 1.0f);
  return (int)(span < 1e6f ? span : 1e6f) + 2 + axis_slack(s.pre_h);
}

// walk_steps() from the ratio in the sample's record.
static int strip_steps(const DevSample& s, int rows) {
  const int slack = axis_slack(s.pre_h);
  if (s.pre_h <= s.geom_h) {
    return rows * (4 + slack) + 4;
  }
  const float span = (float)(rows + 1) * s.axis_y[0];
  const int whole = (int)span;
  return whole + (whole < span) + slack + 2 + rows * (1 + slack) + 8;
}

void set_axes(DevSample& s) {
  s.axis_x[0] = (float)s.pre_w / (float)s.geom_w;
  s.axis_x[1] = s.pre_w > s.geom_w ? std::min(1.0f, (float)s.geom_w / (float)s.pre_w) : 1.0f;
  s.axis_y[0] = (float)s.pre_h / (float)s.geom_h;
  s.axis_y[1] = s.pre_h > s.geom_h ? std::min(1.0f, (float)s.geom_h / (float)s.pre_h) : 1.0f;
  // plan_axis(): floor(2r) + 2 taps, which rounding r to a float cannot make fewer
  s.cap_x = (s.pre_w > s.geom_w ? (int32_t)(2.0f * s.axis_x[0]) + 2 : 4) + axis_slack(s.pre_w);
}

Mode resize_mode(DevSample& s, int channels) {
  if ((long long)s.src_w * channels >= (1LL << 31)) {
    return kModeResizeDirect;
  }
  const int px = strip_most_px(s, channels);
  s.walk_px = px;   // for split_strips
  if (px >= std::min(s.post_w, kStripMinPx) && s.cap_x * 32 * ((px + 31) / 32) <= kStripMaxTaps &&
      strip_span(s, 1) <= kStripSlots) {
    return kModeResize;
  }
  return walk_fits(s, channels) ? kModeResizeWide : kModeResizeDirect;
}

// Instructions of a warp per stage of four output rows of a strip, as measured by taking
// parts of the kernel away: the steps down the source rows, then passes of 32 columns.
static float stage_rows_cost(const DevSample& s) {
  return std::max(s.axis_y[0], 1.5f) * 120.0f + 150.0f;
}

static float stage_pass_cost(const DevSample& s) {
  return std::max(s.axis_x[0], 1.0f) * 34.0f + 107.0f;
}

// How many strips: the fewer, the fewer walks down the source rows; the horizontal
// half works on 32 columns at a time, so strips of whole 32s waste no lanes.  More
// strips than the least can at best save the passes above `whole`, which most often
// does not make up for one more walk: then nothing else is tried.
static void split_strips(DevSample& s) {
  const int most = s.walk_px;
  const float rows = stage_rows_cost(s), pass = stage_pass_cost(s);
  const int least = most >= s.post_w ? 1 : (s.post_w + most - 1) / most;
  const int whole = (s.post_w + 31) >> 5;
  s.walk_px = least == 1 ? s.post_w : (s.post_w + least - 1) / least;
  const int passes = (s.walk_px + 31) >> 5;
  float best = (float)least * (rows + (float)passes * pass);
  const float bound = (float)(least + 1) * rows + (float)whole * pass;
  for (int p = passes - 1; p > 0 && best > bound; p--) {
    const int strips = (s.post_w + 32 * p - 1) / (32 * p);
    const int px = (s.post_w + strips - 1) / strips;
    const float cost = (float)strips * (rows + (float)((px + 31) >> 5) * pass);
    if (cost < best) {
      best = cost;
      s.walk_px = px;
    }
  }
  s.walk_chunks = s.walk_px == s.post_w ? 1 : (s.post_w + s.walk_px - 1) / s.walk_px;
  s.stage_cost = rows + (float)((s.walk_px + 31) >> 5) * pass;
}

// Chunks of at most `px` columns and walks of at most `rows` rows, smaller
// where the source footprint asks for it.
static void split_walk(DevSample& s, int channels, int px, int rows) {
  px = std::min(px, kWalkMaxTaps / s.cap_x);   // (acts on axes with slack alone)
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

static void plan_strips(DevSample* samples, int n, StripPlan& plan) {
  constexpr int kWarps = kStripThreads / 32;
  // (Five CTAs an SM leave 45.7 KB each, which a batch of strong shrinks down the rows among many
  // taps can still exceed; walks cut until five fit took 138.8 us where four took 117.)
  constexpr float kWarpsAtOnce = 148 * kStripCtas * kWarps;
  plan = StripPlan{};
  double total = 0.0;
  const DevSample* last = nullptr;   // the sample before: like ones are split once
  int last_most = 0;
  for (int i = 0; i < n; i++) {
    DevSample& s = samples[i];
    if (s.mode != kModeResize) {
      continue;
    }
    const int most = s.walk_px;
    if (last && most == last_most && s.post_w == last->post_w && s.pre_h == last->pre_h && s.axis_x[0] == last->axis_x[0] &&
        s.axis_y[0] == last->axis_y[0]) {
      s.walk_px = last->walk_px;
      s.walk_chunks = last->walk_chunks;
      s.walk_sizes = last->walk_sizes;
      s.stage_cost = last->stage_cost;
    } else {
      split_strips(s);
      const int part = strip_span(s, 4) <= kStripSlots ? 4 : strip_span(s, 2) <= kStripSlots ? 2 : 1;
      s.walk_sizes = part | strip_span(s, part) << 8;
    }
    total += (double)(s.walk_chunks * ((s.post_h + 3) / 4)) * s.stage_cost;
    last = &s;
    last_most = most;
  }
  if (total == 0.0) {
    return;
  }
  // Walks of about the same work in all samples, so that a large or strongly shrunk one
  // does not hold up the end: one and a half rounds of them over the device's warps, but
  // not below kLeast, about three times what a walk's tables take, as long as all warps
  // have one.  96 images of 240-640 px to 224x224: 51 us a pass so, 56 in one round, 66
  // where every walk has 8 rows; 256 of 256-800 px: 121, 125 in two and a half rounds,
  // 149 in eight.
  constexpr float kRounds = 1.5f, kLeast = 2500.0f;
  const float each = (float)total / kWarpsAtOnce;
  float walk = std::max(each / kRounds, std::min(each, kLeast));
  for (;;) {
    long long ctas = 0;
    bool longest = true;
    plan.steps = 0;
    plan.bytes = 0;
    int stages = 0, post_h = 0, even = 0, down = 0;   // of the sample before
    for (int i = 0; i < n; i++) {
      DevSample& s = samples[i];
      if (s.mode != kModeResize) {
        continue;
      }
      const int most = (int)std::min(8.0f, std::max(1.0f, walk / s.stage_cost));
      if (most != stages || s.post_h != post_h) {
        // as few CTAs as that makes, with the rows dealt evenly, in fours
        stages = most;
        post_h = s.post_h;
        down = (post_h + 4 * kWarps * stages - 1) / (4 * kWarps * stages);
        even = (post_h + 4 * kWarps * down - 1) / (4 * kWarps * down) * 4;
        down = (post_h + even * kWarps - 1) / (even * kWarps);
      }
      longest = longest && stages == 8;
      int rows = even;
      int steps = strip_steps(s, rows);
      while (rows > 4 && steps > kStripMaxSteps) {
        rows -= 4;
        steps = strip_steps(s, rows);
      }
      s.walk_rows = rows;
      plan.steps = std::max(plan.steps, steps);
      s.walk_sizes = (s.walk_sizes & 0xffff) | steps << 16;
      plan.bytes = std::max(plan.bytes, (int32_t)strip_layout(s, 0, 0u, nullptr));
      ctas += s.walk_chunks * (long long)(rows == even ? down : (post_h + rows * kWarps - 1) / (rows * kWarps));
    }
    // A small batch: whole CTAs make the one round a little more than one, which takes as
    // long as two; longer walks until it is one.  4 and 8 images of 900x1100 px, shorter
    // side 224: 20.5 and 28.9 us a pass before, 18.4 and 24.6 so (896 CTAs for 740 places
    // in the second); beyond 1.3 rounds it costs more than it gives (32 images of 200-500
    // px to 224x224, 1.4 rounds: 23.9 and 24.4).
    if (walk > kLeast || ctas <= 148 * kStripCtas || 10 * ctas > 13 * 148 * kStripCtas || longest) {
      return;
    }
    walk *= 1.15f;
  }
}

// Two CTAs for every one of a B200's 148 SMs (another count would only choose other cells).
constexpr long long kWideWantCtas = 148 * 2;

static void plan_wide(DevSample* samples, int n, int channels, WalkPlan& plan) {
  // The largest cells that still give every SM two CTAs.
  static const int kCells[][2] = {{kWalkMaxPx, 32}, {kWalkMaxPx, 16}, {kWalkMaxPx, 8}, {64, 8}, {64, 4}};
  for (const auto& cell : kCells) {
    long long ctas = 0;
    plan = WalkPlan{0, 0, 0, 0, 0};
    for (int i = 0; i < n; i++) {
      DevSample& s = samples[i];
      if (s.mode == kModeResizeWide) {
        split_walk(s, channels, cell[0], cell[1]);
        ctas += (long long)s.walk_chunks * ((s.post_h + s.walk_rows - 1) / s.walk_rows);
        plan.px = std::max(plan.px, s.walk_px);
        plan.taps = std::max(plan.taps, s.walk_px * s.cap_x);
        plan.steps = std::max(plan.steps, (int32_t)walk_steps(s, s.walk_rows));
      }
    }
    if (ctas == 0 || ctas >= kWideWantCtas) {
      return;
    }
  }
}

// Chunks of resize_walk.cu across a resize, as split_walk() makes them but for a column
// or two, and the warps of a chunk that have a word of its source rows.
static int wide_chunks(const DevSample& s, int channels, int& warps) {
  const float ratio = s.axis_x[0], reach = 2.0f * std::max(ratio, 1.0f);
  const float columns = (float)((kWalkRow - 6) / channels - 2);
  const int px = (int)std::max(1.0f, std::min((float)kWalkMaxPx, (columns - reach) / ratio + 1.0f));
  const int chunks = (s.post_w + px - 1) / px;
  const float width = (float)((s.post_w + chunks - 1) / chunks - 1) * ratio + reach + 1.0f;
  warps = ((int)std::min((float)s.pre_w, width) * channels + 255) / 256;
  return chunks;
}

// What a resize adds to a launch of either kernel, in picoseconds: per strip (chunk) and
// stage of four output rows the steps down the source rows, then the passes of 32
// columns (the warps of the chunk, which all wait for the busiest).  Fitted to 1376 uniform
// batches of 1 to 1024 images, 0.2:1 to 8:1, 1 to 4 channels, both output types, timed in
// both kernels: they hold to 12 % in the mean; the strips' are a tenth lower, since a batch
// in doubt is theirs.  With four channels all units of a pixel column lie in one half of
// the banks, where the columns of a shrink meet.
static float strip_time(const DevSample& s, int channels) {
  const float rx = s.axis_x[0], ry = std::max(s.axis_y[0], 1.5f);
  const float pass = channels < 4 ? 180.0f + 65.0f * std::max(rx, 1.0f) : rx < 1.0f ? 400.0f : 640.0f + 110.0f * rx;
  return (float)(s.walk_chunks * ((s.post_h + 3) / 4)) * (420.0f * ry + (float)((s.walk_px + 31) >> 5) * pass);
}

static float wide_time(const DevSample& s, int channels) {
  int warps;
  const int chunks = wide_chunks(s, channels, warps);
  return (float)(chunks * ((s.post_h + 3) / 4)) * (760.0f * std::max(s.axis_y[0], 1.5f) + 1100.0f * (float)warps);
}

// Cells of a resize with walks of at most `most` rows.
static float wide_cells(const DevSample& s, int channels, float most) {
  int warps;
  const float rows = std::max(1.0f, std::min(most, (float)(kWalkMaxSteps / 4) / std::max(s.axis_y[0], 1.0f)));
  return (float)wide_chunks(s, channels, warps) * std::ceil((float)s.post_h / rows);
}

// A batch that resize_walk.cu has to run a part of: whether it should run all of it.  Two
// kernels run one after the other and each leaves the GPU part empty at its end: two
// launches took 1.13 times as long as one over 143 batches of shrinks by 1 to 12 (2 images
// 24.3 us and 15.0, 262 images 499 and 407).  Two are better where one launch
// - would be flooded: every sample gets as many cells as the largest, and an empty CTA takes
//   0.8 ns (255 images of 256-500 px, one 20000x300, one 300x20000, to 224x224: 201 000 CTAs,
//   387 us in one launch, 228 in two);
// - would fill less than one round of CTAs with the longest walks, of 32 rows, while the
//   strong shrinks by themselves are cut into short ones (plan_wide): 173 images shrunk by 1
//   to 4 and three by more, to 41x41: 38.7 us in one, 31.0 in two; 17 to 231x231 49.7 and 41.5.
static bool one_launch(const DevSample* samples, int n, int channels) {
  float cells = 0.0f, most = 0.0f, strong = 0.0f;
  int resizes = 0, light = 0;
  const int stride = std::max(1, n / 32);
  for (int i = 0; i < n; i++) {
    const DevSample& s = samples[i];
    const bool is_strong = s.mode == kModeResizeWide;
    resizes += is_strong || s.mode == kModeResize;
    if (is_strong || (s.mode == kModeResize && light++ % stride == 0)) {   // the light ones are counted from a few
      const float own = wide_cells(s, channels, kWalkMaxRows);
      cells += is_strong ? own : own * (float)stride;
      most = std::max(most, own);
      strong += is_strong ? wide_cells(s, channels, 16.0f) : 0.0f;
    }
  }
  const float grid = most * (float)resizes;
  const bool flooded = grid > 4.0f * cells && grid > 32768.0f;
  const bool part_filled = cells >= kWideWantCtas && cells < 2.2f * kWideWantCtas && strong < kWideWantCtas;
  return !flooded && !part_filled;
}

// Which kernel runs a resize that both can, decided for the batch.  One with strong
// shrinks: one_launch().  With four channels the columns of a shrink by two or three meet in
// one or two of the banks' eight places: a batch with a quarter of those is resize_walk.cu's
// (96 images to 224x224 133 us in strips at 2:1 and 110 there, 178 and 148 at 3:1).  Any
// other goes where it takes less time, into strips when in doubt: what a small launch takes
// beyond the sums is a few us less there, and with cells for less than one round of CTAs
// resize_walk.cu is the slower one although the sums are equal (53 batches: 1.1 to 1.27
// times as long; 8 images shrunk by 3 to 6 to 288x288: 42.2 us and 33.6).  Up to three
// channels strips win by 1.0 to 2.5 where the image shrinks by less than three, with four
// where it is enlarged by 1.3 at least, so the times are made up only when a quarter of a
// batch is beyond that, and for 32 to 63 of its samples (512 images of 748x748x3 to
// 136x136: 564 us in strips, 386 in resize_walk.cu; 564 of 507x507x3 to 136x136, bytes, 339
// and 276).
static void choose_resize_kernel(DevSample* samples, int n, int channels) {
  int strips = 0, strong = 0, doubt = 0, meet = 0;
  const float edge = channels == 4 ? 0.75f : 3.0f;
  for (int i = 0; i < n; i++) {
    const DevSample& s = samples[i];
    const int can = s.mode == kModeResize;
    strips += can;
    doubt += can & ((s.axis_x[0] >= edge) | (s.axis_y[0] >= 3.0f));
    meet += can & (s.axis_x[0] > 1.75f) & (s.axis_x[0] < 3.5f);
    strong += s.mode == kModeResizeWide;
  }
  if (strips == 0 || (strong == 0 && 4 * doubt <= strips)) {
    return;
  }
  if (strong > 0) {
    if (!one_launch(samples, n, channels)) {
      return;
    }
  } else if (channels < 4 || 4 * meet <= strips) {
    constexpr float kInDoubt = 3e6f;
    float in_strips = 0.0f, in_wide = 0.0f, cells = 0.0f, strip = 0.0f, wide = 0.0f, own = 0.0f;
    const DevSample* last = nullptr;
    const int stride = std::max(1, n / 32);
    for (int i = 0; i < n; i += stride) {
      DevSample& s = samples[i];
      if (s.mode != kModeResize) {
        continue;
      }
      if (!last || s.post_w != last->post_w || s.post_h != last->post_h || s.axis_x[0] != last->axis_x[0] ||
          s.axis_y[0] != last->axis_y[0] || s.pre_w != last->pre_w) {
        split_strips(s);
        strip = strip_time(s, channels);
        wide = wide_time(s, channels);
        own = wide_cells(s, channels, kWalkMaxRows);
        last = &s;
      }
      in_strips += strip;
      in_wide += wide;
      cells += own;
    }
    const bool few = cells * (float)stride < 3 * kWideWantCtas;   // six CTAs an SM
    if (few || in_strips < in_wide + kInDoubt / (float)stride) {
      return;
    }
  }
  for (int i = 0; i < n; i++) {
    if (samples[i].mode == kModeResize && walk_fits(samples[i], channels)) {
      samples[i].mode = kModeResizeWide;
    }
  }
}

// Copies among resizes (images that have the size already) as resizes by 1 along both axes,
// with weights of 1 and the same bytes: a launch of the band kernel behind the strips takes
// 10 us and more, a strip of a copy not much more than the copy.  96 images to a shorter
// side of 320, one of which has it, 50.4 us of kernels, 41.6 so.  Copies that add up to more
// than the launch keep it, as do those beside samples that need it anyway.
static void join_copies(DevSample* samples, int n, int channels) {
  constexpr float kMost = 10e6f;
  int copies = 0, strips = 0;
  for (int i = 0; i < n; i++) {
    copies += samples[i].mode == kModeCopy;
    strips += samples[i].mode == kModeResize;
    if (samples[i].mode == kModeAffine || samples[i].mode == kModeResizeDirect) {
      return;
    }
  }
  if (copies == 0 || strips == 0) {
    return;
  }
  float cost = 0.0f;
  for (int pass = 0; pass < 2; pass++) {
    for (int i = 0; i < n; i++) {
      if (samples[i].mode != kModeCopy) {
        continue;
      }
      DevSample s = samples[i];
      set_axes(s);
      s.mode = resize_mode(s, channels);
      if (pass == 1) {
        samples[i] = s;
        continue;
      }
      if (s.mode != kModeResize) {   // (a side so long that no strip holds a column: walk_px is 0)
        return;
      }
      split_strips(s);
      cost += strip_time(s, channels);
      if (cost > kMost) {
        return;
      }
    }
  }
}

void plan_resize(DevSample* samples, int n, int channels, ResizePlan& plan) {
  join_copies(samples, n, channels);
  choose_resize_kernel(samples, n, channels);
  plan_strips(samples, n, plan.strip);
  plan_wide(samples, n, channels, plan.wide);
}

} // namespace mlxd
