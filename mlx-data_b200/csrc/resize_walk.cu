// The resize kernel of strong shrinks and of the batches with them (kModeResizeWide): one
// CTA of kWalkThreads walks down one chunk of output columns (walk_px of them at most) of
// one sample, walk_rows output rows, in stages of four rows.
//
// Vertical half of a stage.  A thread owns two 32-bit words of the chunk's
// source bytes (eight byte columns) and walks down the source rows.  Each warp
// copies its own words of the rows to come into a ring in shared memory
// (cp.async, kAhead rows in flight; nobody else reads them, so the walk needs no
// barrier, and no register waits for memory).  Every byte is converted to float
// once; a source row is a tap of two output rows at most (any shrink or
// enlargement), so two accumulators per byte column are enough: the output row
// being finished (A) and the next one (B).  The walk follows a table of steps
// {weight in A, weight in B, row fetched ahead} built per CTA; completed rows go
// to shared memory two by two, (row, row + 1) of a byte column side by side, so
// that the horizontal half loads the operands of its packed multiply-adds as
// they are.  A row that three outputs touch (tap weights of about 0 at the ends)
// is stepped over twice.
//
// Horizontal half, after a barrier: a thread takes one output column of the
// stage's four rows over all channels, quantises, casts through the table and
// stores into the batch tensor.
//
// Arithmetic: every output is a chain acc = fma(w_k, v_k, acc) from 0 in
// increasing tap order, vertical axis first, quantised as (int)(acc + 0.5).
// Steps that are no tap of an accumulator enter it with weight 0, which leaves
// it unchanged.
//
// What bounds it (1080x1920x3 to 512x512, 512 images, when it ran those too: 1.37 ms, before: 1.75 ms in
// 16x64-pixel passes staged by bulk copies and filtered from there): the shared-
// memory pipe, 89 % busy, of whose wavefronts the horizontal taps are about 45 %
// (half of them bank conflicts of columns 2.1 apart), the stores of the row pairs
// 20 %; instructions per 16x64 pixels are 6.6 k, before 10.2 k.  Why this split:
// a walk converts a byte once instead of once per pair of output rows that it
// feeds, keeps no source footprint on chip beyond the rows in flight, and has two
// barriers per four output rows.  The rows in flight lie in shared memory because
// the same walk with the rows fetched ahead in registers waited for them at every
// move of a register between steps (1.62 - 1.89 ms).  One set of float rows and
// two barriers a stage leave room for six CTAs per SM; the clamped tap loop of
// chunks at an image's edge costs two instructions a tap.
//
// Unlike samples whose rows do and do not start on a word, with CTAs that fill padding among
// them, keep several paths of the kernel in the instruction cache at a time.  So where the cast is
// computed the horizontal half is there once for both kinds of rows, and an instance knows its way
// of casting.  346 images of 880-1730 px, shorter side 323, padded and normalised: with the casts by
// steps beside the look-ups in both halves 1357 us (0.67 stalls an issue for want of
// instructions), look-ups alone 1320 (0.23), so 1300; 64 of 1400 px to 300x300 216, 223 and 216.
// The way of casting alone known, the half still twice: 1471 and 236.  With the channel reduction
// 226 us and 202.  Byte batches and look-ups, whose code is shorter, keep the half twice (300 of
// 880-1730 px to 323x323, bytes, 908 us, 921 with one; 128 of 900 px to 64x64, looked up, 147.7 and 149.7).
#include <algorithm>

#include "fused_batch.h"
#include "kernel_common.cuh"
#include "resize_common.cuh"

namespace mlxd {
namespace {

constexpr int kStageRows = 4;
constexpr int kAhead = 7;                         // source rows in flight behind the one being filtered
constexpr int kSlots = kAhead + 1;                // a slot is written again one step after it was read
constexpr unsigned kWarpSlot = 68 * 4;            // a warp's 64 words of a row, one more, padding
constexpr unsigned kSlotBytes = kWalkThreads / 32 * kWarpSlot;
constexpr unsigned kPairBytes = kWalkRow * 8u;    // one pair of float rows in shared memory
constexpr unsigned kMidBytes = kStageRows / 2 * kPairBytes;

struct WalkSmem {
  unsigned mid;     // float2 [kStageRows / 2][kWalkRow]
  unsigned ring;    // source words [kSlots][warp][68]
  unsigned lut;     // float [table_channels][256]
  unsigned steps;   // 32 bytes per step, kAhead leading entries that only name rows
  unsigned count;   // int [kWalkMaxRows]  steps of every output row
  unsigned hx;      // {first tap's byte offset in a row pair, signed, tap count << 16} per column
  unsigned hw;      // float [tap][walk_px]
};

__host__ __device__ constexpr size_t walk_layout(int tables, const WalkPlan& w, unsigned base, WalkSmem* out) {
  WalkSmem sm{};
  size_t off = 0;
  sm.mid = base;
  off += kMidBytes;
  sm.ring = base + (unsigned)off;
  off += kSlots * kSlotBytes;
  sm.lut = base + (unsigned)off;
  off += (size_t)tables * 1024;
  sm.steps = base + (unsigned)off;
  off += (size_t)(w.steps + 2 * kAhead) * 32;
  sm.count = base + (unsigned)off;
  off += kWalkMaxRows * 4;
  sm.hx = base + (unsigned)off;
  off += (size_t)w.px * 4;
  sm.hw = base + (unsigned)off;
  off += (size_t)w.taps * 4;
  if (out) {
    *out = sm;
  }
  return (off + 15) & ~(size_t)15;
}

// One thread's filter state.
struct Walker {
  const uint8_t* src;       // word A in the window's row 0; word B is 128 bytes on
  unsigned pitch;
  int word;                 // index of word A in a row; word B is 32 on
  bool ok_a, ok_b;          // the words hold bytes of the chunk
  unsigned ring;            // word A in slot 0 of the ring
  unsigned free_slot;       // offset of the slot read in the step before
  unsigned tp;              // next step
  f32x2 acc_a[4], acc_b[4]; // bytes (0,1), (2,3) of word A, then of word B
};

// Step table entry i: +0 {wa, wa, wb, wb} of step i - kAhead, +16 source row of
// step i, +20 words of that row, +24 funnel shift and +28 ring offset of step
// i - kAhead.

__device__ __forceinline__ void copy_word(unsigned dst, const uint8_t* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}

// This warp's words of a source row into the slot at offset `slot`: those that
// hold a byte of the chunk, nothing before or behind them is read.
template <bool SHIFT>
__device__ __forceinline__ void fetch(const Walker& k, unsigned row, int words, unsigned slot) {
  const uint8_t* g = k.src + (size_t)row * k.pitch;
  if (SHIFT) {
    g = reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(g) & ~(uintptr_t)3);
  }
  const unsigned d = k.ring + slot;
  if (k.word < words) {
    copy_word(d, g);
  }
  if (k.word + 32 < words) {
    copy_word(d + 128, g + 128);
  }
  if (SHIFT && (threadIdx.x & 31) == 0 && k.word + 64 < words) {
    copy_word(d + 256, g + 256);   // lane 31's word B starts in this one's neighbour
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// Rows x (first) and y (second) of one word's four byte columns.
__device__ __forceinline__ void store_pair(unsigned a, f32x2 x01, f32x2 x23, f32x2 y01, f32x2 y23) {
  float x0, x1, x2, x3, y0, y1, y2, y3;
  unpack2(x01, x0, x1);
  unpack2(x23, x2, x3);
  unpack2(y01, y0, y1);
  unpack2(y23, y2, y3);
  sts_v4(a, x0, y0, x1, y1);
  sts_v4(a + 16, x2, y2, x3, y3);
}

// What every step does: this row's eight bytes as floats (v) and its weights;
// the row kAhead steps on is set under way.
template <bool SHIFT>
__device__ __forceinline__ void walk_load(Walker& k, f32x2 (&v)[4], f32x2& wa, f32x2& wb) {
  const f32x2 minus_two23 = pack2(-8388608.0f, -8388608.0f);
  uint32_t row_ahead, words_ahead, shift, slot;
  lds_v4u32<16>(k.tp, row_ahead, words_ahead, shift, slot);
  asm volatile("cp.async.wait_group %0;" ::"n"(kAhead - 1) : "memory");
  if (SHIFT) {
    __syncwarp();   // words copied by other lanes
  }
  const unsigned r = k.ring + slot;
  uint32_t xa = lds_u32<0>(r), xb = lds_u32<128>(r);
  if (SHIFT) {
    xa = __funnelshift_r(xa, lds_u32<4>(r), shift);
    xb = __funnelshift_r(xb, lds_u32<132>(r), shift);
  }
  lds_v2u64<0>(k.tp, wa, wb);
  k.tp += 32;
  fetch<SHIFT>(k, row_ahead, (int)words_ahead, k.free_slot);
  k.free_slot = slot;
  v[0] = bytes_to_f32x2<0, 1>(xa, minus_two23);
  v[1] = bytes_to_f32x2<2, 3>(xa, minus_two23);
  v[2] = bytes_to_f32x2<0, 1>(xb, minus_two23);
  v[3] = bytes_to_f32x2<2, 3>(xb, minus_two23);
}

// The steps of one output row; leaves the completed row in `done`.
template <bool SHIFT>
__device__ __forceinline__ void walk_row(Walker& k, int steps, f32x2 (&done)[4]) {
  f32x2 v[4], wa, wb;
#pragma unroll 1
  for (; steps > 1; steps--) {
    walk_load<SHIFT>(k, v, wa, wb);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      ffma2(k.acc_a[i], v[i], wa);
      ffma2(k.acc_b[i], v[i], wb);
    }
  }
  walk_load<SHIFT>(k, v, wa, wb);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    done[i] = fma2(v[i], wa, k.acc_a[i]);
    k.acc_a[i] = fma2(v[i], wb, k.acc_b[i]);
    k.acc_b[i] = 0;
  }
}

// The next `rows` output rows, whose step counts lie at shared address `count`,
// stored in pairs from st (word A) and st + 1024 (word B) on.
template <bool SHIFT>
__device__ __forceinline__ void walk_pairs(Walker& k, unsigned st, unsigned count, int rows) {
#pragma unroll 1
  for (; rows > 0; rows -= 2) {
    uint32_t n0, n1;
    lds_v2u32<0>(count, n0, n1);
    f32x2 x[4], y[4] = {0, 0, 0, 0};
    walk_row<SHIFT>(k, (int)n0, x);
    if (rows > 1) {
      walk_row<SHIFT>(k, (int)n1, y);
    }
    // (the second row of an incomplete pair is never used)
    if (k.ok_a) {
      store_pair(st, x[0], x[1], y[0], y[1]);
    }
    if (k.ok_b) {
      store_pair(st + 1024, x[2], x[3], y[2], y[3]);
    }
    st += kPairBytes;
    count += 8;
  }
}

// One tap of the horizontal filter: all channels of a source pixel in the four
// rows, at shared address a, weight w.  acc[2 * c + h]: rows 2h, 2h + 1 of
// channel c.
template <int C>
__device__ __forceinline__ void tap(unsigned a, float w, f32x2 (&acc)[2 * C]) {
  const f32x2 ww = pack2(w, w);
  if (C == 4) {
    f32x2 x, y;
    lds_v2u64<0>(a, x, y);
    ffma2(acc[0], x, ww);
    ffma2(acc[2 % (2 * C)], y, ww);
    lds_v2u64<16>(a, x, y);
    ffma2(acc[4 % (2 * C)], x, ww);
    ffma2(acc[6 % (2 * C)], y, ww);
    lds_v2u64<(int)kPairBytes>(a, x, y);
    ffma2(acc[1], x, ww);
    ffma2(acc[3 % (2 * C)], y, ww);
    lds_v2u64<(int)kPairBytes + 16>(a, x, y);
    ffma2(acc[5 % (2 * C)], x, ww);
    ffma2(acc[7 % (2 * C)], y, ww);
  } else {
    ffma2(acc[0], lds_u64<0>(a), ww);
    ffma2(acc[1], lds_u64<(int)kPairBytes>(a), ww);
    if (C > 1) {
      ffma2(acc[2 % (2 * C)], lds_u64<8>(a), ww);
      ffma2(acc[3 % (2 * C)], lds_u64<(int)kPairBytes + 8>(a), ww);
    }
    if (C > 2) {
      ffma2(acc[4 % (2 * C)], lds_u64<16>(a), ww);
      ffma2(acc[5 % (2 * C)], lds_u64<(int)kPairBytes + 16>(a), ww);
    }
  }
}

// What the tables of a chunk leave for the walk.
struct Chunk {
  WalkSmem sm;
  const uint8_t* g0;   // first word (or byte, when shifted) of the chunk in the window's row 0
  unsigned pitch;
  int common, nwords;  // bytes of the first word before the chunk; words of a row
  int nr, nc, y0, x0, x1;
  int first_col, last_col;   // shared addresses of the chunk's first and last column in the first row pair
  bool edge_x, pre_flip;
};

// The stages of one chunk, tables in place.  Its rows start on a word, or not, or (kAnyRows)
// `shifted` says.
enum RowStart { kWordRows, kShiftedRows, kAnyRows };
template <int C, bool GRAY, bool U8, int CAST, RowStart ROWS>
__device__ __forceinline__ void walk_stages(const DevSample& s, const LaunchParams& p, const Chunk& c, bool shifted) {
  constexpr int CO = GRAY ? 1 : C;
  const bool shift = ROWS == kAnyRows ? shifted : ROWS == kShiftedRows;
  const int tid = threadIdx.x;
  const int first_word = (tid >> 5) * 64;
  const bool warp_works = first_word < c.nwords;
  Walker k = {};
  k.pitch = c.pitch;
  k.word = first_word + (tid & 31);
  k.src = c.g0 + 4 * k.word;
  k.ok_a = k.word < c.nwords;
  k.ok_b = k.word + 32 < c.nwords;
  k.ring = c.sm.ring + (unsigned)(tid >> 5) * kWarpSlot + (unsigned)(tid & 31) * 4u;
  k.free_slot = kAhead * kSlotBytes;
  k.tp = c.sm.steps + kAhead * 32u;
  if (warp_works) {
#pragma unroll 1
    for (int j = 0; j < kAhead; j++) {
      const unsigned e = c.sm.steps + 32u * j;
      if (shift) {
        fetch<true>(k, lds_u32<16>(e), (int)lds_u32<20>(e), (unsigned)j * kSlotBytes);
      } else {
        fetch<false>(k, lds_u32<16>(e), (int)lds_u32<20>(e), (unsigned)j * kSlotBytes);
      }
    }
  }
  const size_t row_stride = (size_t)s.slot_w * CO;
  const bool post_flip = s.post_flip != 0;
  void* const dst = s.dst;   // (a copy: the stores could otherwise have changed it)
  const bool vec_ok = (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
  const unsigned hstep = (unsigned)s.walk_px * 4u;
  const int tap_step = c.pre_flip ? -8 * C : 8 * C;
  const unsigned mid = c.sm.mid;
  for (int r0 = 0; r0 < c.nr; r0 += kStageRows) {
    const int rows = min(kStageRows, c.nr - r0);
    if (warp_works) {
      const unsigned st = mid + (unsigned)k.word * 32u, count = c.sm.count + 4u * (unsigned)r0;
      if (shift) {
        walk_pairs<true>(k, st, count, rows);
      } else {
        walk_pairs<false>(k, st, count, rows);
      }
    }
    __syncthreads();
    for (int x = tid; x < c.nc; x += kWalkThreads) {
      const uint32_t hx = lds_u32<0>(c.sm.hx + 4u * (unsigned)x);
      const int cnt = (int)(hx >> 16);
      unsigned wq = c.sm.hw + 4u * (unsigned)x;
      f32x2 acc[2 * C];
#pragma unroll
      for (int i = 0; i < 2 * C; i++) {
        acc[i] = 0;
      }
      if (!c.edge_x) {
        unsigned a = mid + (hx & 0xffffu);
        for (int t = 0; t < cnt; t++) {
          tap<C>(a, __uint_as_float(lds_u32<0>(wq)), acc);
          a += tap_step;
          wq += hstep;
        }
      } else {
        // taps beyond the image read its first or last column, which is then the chunk's
        int a = (int)mid + (int16_t)(hx & 0xffffu);
        for (int t = 0; t < cnt; t++) {
          tap<C>((unsigned)clampi(a, c.first_col, c.last_col), __uint_as_float(lds_u32<0>(wq)), acc);
          a += tap_step;
          wq += hstep;
        }
      }
      const int ox = post_flip ? c.x1 - 1 - x : c.x0 + x;
      store_column<C, GRAY, U8, CAST>(
          p, c.sm.lut, acc, rows, dst, (size_t)(c.y0 + r0) * row_stride + (size_t)ox * CO, row_stride, vec_ok);
    }
    __syncthreads();
  }
}

// Rows [y0, y1) x columns [x0, x1) of the slot, all inside the post window.
template <int C, bool GRAY, bool U8, int CAST>
__device__ __forceinline__ void walk_chunk(
    const DevSample& s, const LaunchParams& p, const WalkSmem& sm, int y0, int y1, int x0, int x1) {
  constexpr int CO = GRAY ? 1 : C;
  const int tid = threadIdx.x;
  const int nr = y1 - y0;
  const int nc = x1 - x0;
  const int px = s.walk_px;
  const int by = s.post_y + y0;
  const int bx = s.post_x + (s.post_flip ? s.post_w - x1 : x0);   // first geometric column
  const int pre_w = s.pre_w, pre_h = s.pre_h;
  const bool pre_flip = s.pre_flip != 0;
  const Axis ay = make_axis(pre_h, s.geom_h);
  const Axis ax = make_axis(pre_w, s.geom_w);

  // ---- source columns of the chunk ----------------------------------------------
  int f0, l0, f1, l1;
  axis_range(ax, bx, f0, l0);
  axis_range(ax, bx + nc - 1, f1, l1);
  int clo = clampi(f0, 0, pre_w - 1);
  int chi = clampi(l1, 0, pre_w - 1);
  if (pre_flip) {
    const int t = clo;
    clo = pre_w - 1 - chi;
    chi = pre_w - 1 - t;
  }
  const bool edge_x = f0 < 0 || l1 > pre_w - 1;
  const int wbytes = (chi - clo + 1) * C;
  const unsigned pitch = (unsigned)s.src_w * C;
  const uint8_t* g0 = s.src + ((size_t)s.pre_y * s.src_w + (s.pre_x + clo)) * C;
  const unsigned phase0 = (unsigned)(reinterpret_cast<uintptr_t>(g0) & 3);
  // Rows a multiple of 4 bytes apart all start at the same byte of a word, so
  // whole words are taken from the word that holds the first byte; otherwise a
  // row's words are put together from two.  (Four channels are read back 16
  // bytes at a time, so there the first byte comes first.)
  const bool shifted = (pitch & 3) != 0 || (C == 4 && phase0 != 0);
  const int common = shifted ? 0 : (int)phase0;
  const int nwords = (common + wbytes + 3) >> 2;

  // ---- tables ---------------------------------------------------------------------
  // (the float rows are not in use yet: the per-row scratch lies there)
  int* r_lo = sp<int>(sm.mid);
  int* r_hi = r_lo + kWalkMaxRows;
  float* r_sum = reinterpret_cast<float*>(r_hi + kWalkMaxRows);
  int* r_off = reinterpret_cast<int*>(r_sum + kWalkMaxRows);   // kWalkMaxRows + 1 entries
  if (tid < nr) {
    int lo, hi;
    axis_range(ay, by + tid, lo, hi);
    float sum = 0.0f;
    if (!ay.identity) {
      const float u = axis_center(ay, by + tid);
      for (int k = lo; k <= hi; k++) {
        sum = __fadd_rn(sum, axis_tent(ay, u, k));
      }
    }
    r_lo[tid] = lo;
    r_hi[tid] = hi;
    r_sum[tid] = sum;
  }
  for (int x = tid; x < nc; x += kWalkThreads) {
    int lo, hi;
    axis_range(ax, bx + x, lo, hi);
    int cnt = hi - lo + 1;
    cnt = cnt > s.cap_x ? s.cap_x : cnt;
    const int col = pre_flip ? pre_w - 1 - lo : lo;   // may lie outside the image by the filter's radius
    sp<uint32_t>(sm.hx)[x] = (uint32_t)(((common + (col - clo) * C) * 8) & 0xffff) | ((uint32_t)cnt << 16);
    float* w = sp<float>(sm.hw) + x;
    if (ax.identity) {
      w[0] = 1.0f;
    } else {
      const float u = axis_center(ax, bx + x);
      float sum = 0.0f;
      for (int k = 0; k < cnt; k++) {
        const float v = axis_tent(ax, u, lo + k);
        w[k * px] = v;
        sum = __fadd_rn(sum, v);
      }
      for (int k = 0; k < cnt; k++) {
        w[k * px] = __fdiv_rn(w[k * px], sum);
      }
    }
  }
  if (!U8 && CAST == kCastTable) {
    for (int i = tid; i < CO * 256; i += kWalkThreads) {
      sp<float>(sm.lut)[i] = __ldg(p.lut + i);
    }
  }
  __syncthreads();
  // Steps of output row a: source rows first_a .. hi_a, where first_a continues
  // behind hi_(a-1) but goes back to the first tap of row a + 1 if that lies
  // before (its weight in row a is then 0: row a had it already).
  auto first_row = [&](int a) {
    int f = a == 0 ? r_lo[0] : r_hi[a - 1] + 1;
    if (a + 1 < nr) {
      f = min(f, r_lo[a + 1]);
    }
    return min(f, r_hi[a]);
  };
  if (tid < 32) {
    static_assert(kWalkMaxRows <= 32, "one lane per output row");
    const int own = tid < nr ? r_hi[tid] - first_row(tid) + 1 : 0;
    int n = own;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, n, d);
      n += tid >= d ? t : 0;
    }
    r_off[tid] = n - own;
    if (tid == 31) {
      r_off[32] = n;
    }
    sp<int>(sm.count)[tid] = own;
  }
  __syncthreads();
  const int steps = r_off[32];
  if (steps > p.walk.steps || nwords * 4 > kWalkRow) {
    if (tid == 0) {
      atomicOr(p.status, 8);
    }
    return;
  }
  // words of a row that hold bytes of the chunk
  auto row_words = [&](int row) {
    const unsigned phase = (phase0 + (unsigned)row * pitch) & 3u;
    return shifted ? (int)((phase + wbytes + 3) >> 2) : nwords;
  };
  for (int i = tid; i < nr * 4; i += kWalkThreads) {
    const int a = i >> 2;
    const int f = first_row(a);
    const int hi = r_hi[a];
    const int prev = a == 0 ? r_lo[0] - 1 : r_hi[a - 1];
    for (int row = f + (i & 3); row <= hi; row += 4) {
      const int at = r_off[a] + row - f;
      float wa = 0.0f, wb = 0.0f;
      if (row > prev && row >= r_lo[a]) {
        wa = ay.identity ? 1.0f : __fdiv_rn(axis_tent(ay, axis_center(ay, by + a), row), r_sum[a]);
      }
      if (a + 1 < nr && row >= r_lo[a + 1]) {
        wb = ay.identity ? 1.0f : __fdiv_rn(axis_tent(ay, axis_center(ay, by + a + 1), row), r_sum[a + 1]);
      }
      const int seen = clampi(row, 0, pre_h - 1);
      uint32_t* e = sp<uint32_t>(sm.steps + (unsigned)(at + kAhead) * 32u);
      *reinterpret_cast<float4*>(e) = make_float4(wa, wa, wb, wb);
      e[6] = ((phase0 + (unsigned)seen * pitch) & 3u) * 8u;
      e[7] = (unsigned)(at % kSlots) * kSlotBytes;
      uint32_t* r = sp<uint32_t>(sm.steps + (unsigned)at * 32u);
      r[4] = (uint32_t)seen;
      r[5] = (uint32_t)row_words(seen);
    }
  }
  if (tid < kAhead) {   // no rows to fetch ahead of the last steps
    uint32_t* r = sp<uint32_t>(sm.steps + (unsigned)(steps + tid) * 32u);
    r[4] = 0;
    r[5] = 0;
  }
  __syncthreads();

  const Chunk c = {sm, g0 - common, pitch, common, nwords, nr, nc, y0, x0, x1, (int)sm.mid + common * 8,
                   (int)sm.mid + (common + (chi - clo) * C) * 8, edge_x, pre_flip};
  if (!U8 && (GRAY || CAST != kCastTable)) {
    walk_stages<C, GRAY, U8, CAST, kAnyRows>(s, p, c, shifted);
  } else if (shifted) {
    walk_stages<C, GRAY, U8, CAST, kShiftedRows>(s, p, c, true);
  } else {
    walk_stages<C, GRAY, U8, CAST, kWordRows>(s, p, c, false);
  }
}

// One cell: walk_rows rows x one chunk (or one strip of padding) of a slot.
// OWN: samples count their own cells off (WalkPlan::cells_y of 0).  CAST: how its floats are cast.
template <int C, bool GRAY, bool U8, int CAST, bool OWN>
__global__ void __launch_bounds__(kWalkThreads, 6) resize_walk_kernel(const __grid_constant__ LaunchParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int CO = GRAY ? 1 : C;
  unsigned t = blockIdx.x;
  if (p.pad_apart && p.fill_every > 0) {   // (0: the other resize kernel fills)
    const unsigned fills = (unsigned)p.n * kPadChunks, every = (unsigned)p.fill_every;
    if (t % every == 0 && t / every < fills) {
      pad_below_any<kWalkThreads>(p, Records<0>(), t / every);
      return;
    }
    t -= min(t / every + 1, fills);
  }
  const unsigned cell = t % p.walk.cells_x;
  t /= p.walk.cells_x;
  int cx = (int)cell;
  int cy = OWN ? 0 : (int)(t % p.walk.cells_y);
  const DevSample& s = p.samples[p.first + (OWN ? t : t / p.walk.cells_y)];
  if (s.mode != kModeResizeWide) {
    return;   // the other kernels'
  }
  const int slot_h = s.slot_h, slot_w = s.slot_w, post_h = s.post_h, post_w = s.post_w;
  const int chunks = s.walk_chunks;
  if (OWN) {
    const unsigned cells_x = (unsigned)(chunks + walk_strips(s));
    cx = (int)(cell % cells_x);
    cy = (int)(cell / cells_x);
    if (cy >= (slot_h + s.walk_rows - 1) / s.walk_rows) {
      return;
    }
  }
  const int y0 = cy * s.walk_rows;
  // the chunks share the post window's columns evenly; strips of kWalkPadPx behind it
  const bool strip = cx >= chunks;
  const int x0 = strip ? post_w + (cx - chunks) * kWalkPadPx : (int)((long long)post_w * cx / chunks);
  const int x1 = strip ? min(x0 + kWalkPadPx, slot_w) : (int)((long long)post_w * (cx + 1) / chunks);
  if (y0 >= slot_h || x0 >= x1) {
    return;
  }
  const int y1 = min(y0 + s.walk_rows, slot_h);
  const int vy1 = min(y1, post_h);
  const int fill_y0 = strip ? y0 : max(y0, post_h);   // rows of the cell that are padding
  const int fill_y1 = p.pad_apart ? vy1 : y1;         // rows below the post window are the fill CTAs' then
  if (!strip && y0 < vy1) {
    WalkSmem sm;
    walk_layout(!U8 && CAST == kCastTable ? CO : 0, p.walk, smem_addr(smem_raw), &sm);
    walk_chunk<C, GRAY, U8, CAST>(s, p, sm, y0, vy1, x0, x1);
  }
  if (fill_y0 < fill_y1) {
    if (U8) {
      fill_rect_u8<CO>(reinterpret_cast<uint8_t*>(s.dst), slot_w, fill_y0, fill_y1, x0, x1, p.pad_px);
    } else {
      float padf[4];
#pragma unroll
      for (int c = 0; c < 4; c++) {
        padf[c] = c < CO ? __ldg(p.lut + c * 256 + p.pad_px) : 0.0f;
      }
      fill_rect_f32<CO>(reinterpret_cast<float*>(s.dst), slot_w, fill_y0, fill_y1, x0, x1, padf);
    }
  }
}

// No plan needs more shared memory than this.
constexpr size_t kWalkMaxSmem = walk_layout(4, WalkPlan{kWalkMaxPx, kWalkMaxTaps, kWalkMaxSteps, 0, 0}, 0u, nullptr);

template <int C, bool GRAY, bool U8, int CAST, bool OWN>
cudaError_t launch_kernel(const LaunchParams& p, unsigned blocks, size_t smem, cudaStream_t stream) {
  // Only strong shrinks need more than the 48 KB that every kernel may have.  The
  // limit belongs to the kernel on the current device and is shared by all host
  // threads, so each of them sets the same value: one that set its own launch's
  // need could lower the limit between another's setting and its launch.
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(
        resize_walk_kernel<C, GRAY, U8, CAST, OWN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWalkMaxSmem);
    if (e != cudaSuccess) {
      return e;
    }
  }
  resize_walk_kernel<C, GRAY, U8, CAST, OWN><<<blocks, kWalkThreads, smem, stream>>>(p);
  return cudaGetLastError();
}

template <int C, bool GRAY, bool U8, int CAST>
cudaError_t launch_cast(const LaunchParams& p, unsigned blocks, size_t smem, cudaStream_t stream) {
  return p.walk.cells_y == 0 ? launch_kernel<C, GRAY, U8, CAST, true>(p, blocks, smem, stream)
                          : launch_kernel<C, GRAY, U8, CAST, false>(p, blocks, smem, stream);
}

template <int C, bool GRAY, bool U8>
cudaError_t launch(const LaunchParams& p, unsigned blocks, size_t smem, cudaStream_t stream) {
  if constexpr (!GRAY && !U8) {
    if (p.cast.mode == kCastScale) {
      return launch_cast<C, GRAY, U8, kCastScale>(p, blocks, smem, stream);
    }
    if (p.cast.mode == kCastNormalise) {
      return launch_cast<C, GRAY, U8, kCastNormalise>(p, blocks, smem, stream);
    }
  }
  return launch_cast<C, GRAY, U8, kCastTable>(p, blocks, smem, stream);
}

} // namespace

cudaError_t launch_resize_walk(const LaunchParams& p_in, bool fills_padding, cudaStream_t stream) {
  LaunchParams p = p_in;
  p.fill_every = 0;
  unsigned long long blocks = (unsigned long long)p.n * std::max(p.walk.cells_y, 1) * p.walk.cells_x;
  if (blocks == 0) {
    return cudaSuccess;
  }
  if (p.pad_apart && fills_padding) {
    // Filling is bound by memory writes, walking by the SMs: the fill CTAs go
    // among the others, evenly, instead of into a launch of their own.  64 images
    // of 160-1024 px padded to the largest (2 GB written): 384 us a pass (in a
    // launch before this one, when it took 398: 449).  Where they are more than
    // the walking CTAs (small slots) all of them come first: 64 images of 100-400
    // px, shorter side 128, 74 us a pass, 256 of 30-120 px, shorter side 32, 87.
    const unsigned long long fills = (unsigned long long)p.n * kPadChunks;
    blocks += fills;
    p.fill_every = (int32_t)std::max<unsigned long long>(1, std::min<unsigned long long>(blocks / fills, 1u << 30));
  }
  if (blocks > 0x7fffffffULL) {
    return cudaErrorInvalidConfiguration;
  }
  const size_t smem = walk_layout(table_channels(p), p.walk, 0u, nullptr);
  const unsigned b = (unsigned)blocks;
  if (p.out_f32) {
    if (p.gray) {
      return launch<3, true, false>(p, b, smem, stream);
    }
    switch (p.c_in) {
      case 1:
        return launch<1, false, false>(p, b, smem, stream);
      case 2:
        return launch<2, false, false>(p, b, smem, stream);
      case 3:
        return launch<3, false, false>(p, b, smem, stream);
      default:
        return launch<4, false, false>(p, b, smem, stream);
    }
  }
  if (p.gray) {
    return launch<3, true, true>(p, b, smem, stream);
  }
  switch (p.c_in) {
    case 1:
      return launch<1, false, true>(p, b, smem, stream);
    case 2:
      return launch<2, false, true>(p, b, smem, stream);
    case 3:
      return launch<3, false, true>(p, b, smem, stream);
    default:
      return launch<4, false, true>(p, b, smem, stream);
  }
}

} // namespace mlxd
