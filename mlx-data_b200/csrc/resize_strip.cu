// The resize kernel: a warp walks down one strip of a sample - up to 241 source
// bytes, up to 256 output columns - in stages of four output rows, on its own.  A
// CTA's warps take one strip, one below the other.
//
// Vertical half of a stage.  The stage's source rows lie in shared memory, copied
// there two rows an instruction (cp.async, lanes 0-15 one row, 16-31 the next, 16
// bytes each) while the stage before was in its horizontal half.  A lane owns two
// 32-bit words of a row (words l and l + 32) and walks down the rows.  A source row
// is a tap of two output rows at most (any shrink or enlargement), so two
// accumulators per byte column are enough: the output row being finished (A) and
// the next one (B).  The walk follows a table of steps {weight in A, weight in B,
// place of the row}; a row that three outputs touch (tap weights of about 0 at the
// ends) is stepped over twice.  The four finished rows of a byte column go to shared
// memory as one 16-byte unit.
//
// Horizontal half: a lane takes one output column of the four rows over all
// channels (32 columns a pass), quantises, casts through the table and stores into
// the batch tensor.
//
// Arithmetic: every output is a chain acc = fma(w_k, v_k, acc) from 0 in
// increasing tap order, vertical axis first, quantised as (int)(acc + 0.5).
// Steps that are no tap of an accumulator enter it with weight 0, which leaves
// it unchanged.  A byte is a multiply-add's operand as it is: its bits are the
// float byte * 2^-149, so the vertical weights are kept times 2^127, their sums come
// out times 2^-22 and the horizontal weights are kept times 2^22 - powers of two
// throughout, so every rounding falls as without them.
//
// What bounds it (1080x1920x3 to 512x512, 512 images: 1.12 ms, 1.16 where casts are looked
// up; 1.37 in resize_walk.cu, which runs a whole CTA down 832 bytes): the latency of its own
// results and of shared memory at 19 warps an SM (1.8 and 1.2 of 7.4 cycles an instruction);
// instructions issue in 61 % of the cycles, the shared-memory pipe is 66 % busy (58 and 76 with
// look-ups, 89 there).  Per 32 columns x 4 rows a warp executes 810 instructions (780 with look-ups,
// 830 there), of them about 310 on the steps, 110 on copies and the skeleton of a stage, the rest on taps,
// casts and stores.  Why this
// split: two 4-byte cp.async a row cost the pipe nine wavefronts, one 16-byte cp.async
// for two rows about two a row; a unit of four rows halves the loads of the taps, and
// dealing columns to lanes by bank takes most of their conflicts; a CTA-wide walk meets
// two barriers a stage and leaves warps idle where a chunk's words are no multiple of its
// 128 lanes.  Five CTAs per SM at 96 registers, for which most instances of one to three
// channels spill 4 to 8 bytes; six spill the walk (1.55 ms), four wait (1.36).
// The tables of a CTA took a fifth of the time before the taps of a pass were shared by
// its warps, the steps dealt flat over the lanes and the axes' ratios divided on the
// host (1.25 ms).
#include <algorithm>

#include "fused_batch.h"
#include "kernel_common.cuh"
#include "resize_common.cuh"

namespace mlxd {
namespace {

constexpr int kWarps = kStripThreads / 32;
constexpr unsigned kSlotBytes = kStripSlotBytes, kMidBytes = kStripMidBytes;
constexpr float kScaleY = 0x1p127f, kScaleX = 0x1p22f;

__device__ __forceinline__ void copy16(unsigned dst, uintptr_t src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// One lane's state of the walk.
struct Walker {
  uintptr_t base;           // this lane's unit of the window's row 0, its first byte as the strip's is aligned
  unsigned pitch;
  int row_max;              // the window's last row
  int from;                 // the unit holds bytes of the strip if the row starts at more than this within 16 bytes
  unsigned dst;             // its place in the ring's first pair of rows
  unsigned tp, ip;          // weights of the next step, place of the one after it
  uint32_t place, shift;    // of the next step
  unsigned part;            // next part: source rows
  unsigned lane4;
  unsigned sel[4];          // prmt selectors: byte j is byte j ^ (lane / 2 % 4) of a word
  f32x2 acc_a[4], acc_b[4]; // bytes (0, 1), (2, 3) of word A, then of word B
};

// Source rows [first, last] of a part into the ring.  A unit is copied only when it
// holds a byte of the strip; units are aligned, so no copy leaves the 16 bytes
// around such a byte.
__device__ __forceinline__ void fetch_rows(const Walker& k, int first, int last) {
  const int half = (threadIdx.x >> 4) & 1;
  unsigned dst = k.dst;
#pragma unroll 1
  for (int row = first + half; row <= last; row += 2) {
    const uintptr_t g = k.base + (size_t)(unsigned)clampi(row, 0, k.row_max) * k.pitch;
    if ((int)(g & 15) > k.from) {
      copy16(dst, g & ~(uintptr_t)15);
    }
    dst += 2 * kSlotBytes;
  }
}

__device__ __forceinline__ void fetch_part(Walker& k) {
  uint32_t first, last;
  lds_v2u32<0>(k.part, first, last);
  k.part += 8;
  fetch_rows(k, (int)first, (int)last);
}

// Two bytes of a word as the low bits of two floats.
__device__ __forceinline__ f32x2 pick_bytes(uint32_t word, unsigned s0, unsigned s1) {
  return pack2(__uint_as_float(__byte_perm(word, 0u, s0)), __uint_as_float(__byte_perm(word, 0u, s1)));
}

// Step I from here: the row's eight bytes (v) and its weights.  The place of the step
// after it is read under way, so that a step starts with its words.
template <bool SHIFT, int I>
__device__ __forceinline__ void walk_load(Walker& k, f32x2 (&v)[4], f32x2& wa, f32x2& wb) {
  const unsigned r = k.place + k.lane4;
  uint32_t xa = lds_u32<0>(r), xb = lds_u32<128>(r);
  if (SHIFT) {
    xa = __funnelshift_r(xa, lds_u32<4>(r), k.shift);
    xb = __funnelshift_r(xb, lds_u32<132>(r), k.shift);
    lds_v2u32<8 * I>(k.ip, k.place, k.shift);
  } else {
    k.place = lds_u32<8 * I>(k.ip);
  }
  lds_v2u64<16 * I>(k.tp, wa, wb);
  v[0] = pick_bytes(xa, k.sel[0], k.sel[1]);
  v[1] = pick_bytes(xa, k.sel[2], k.sel[3]);
  v[2] = pick_bytes(xb, k.sel[0], k.sel[1]);
  v[3] = pick_bytes(xb, k.sel[2], k.sel[3]);
}

template <bool SHIFT, int I>
__device__ __forceinline__ void walk_step(Walker& k) {
  f32x2 v[4], wa, wb;
  walk_load<SHIFT, I>(k, v, wa, wb);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    ffma2(k.acc_a[i], v[i], wa);
    ffma2(k.acc_b[i], v[i], wb);
  }
}

// The steps of one output row; leaves the completed row in `done`.
template <bool SHIFT>
__device__ __forceinline__ void walk_row(Walker& k, int steps, float (&done)[8]) {
#pragma unroll 1
  for (; steps > 2; steps -= 2) {
    walk_step<SHIFT, 0>(k);
    walk_step<SHIFT, 1>(k);
    k.tp += 32;
    k.ip += 16;
  }
  if (steps > 1) {
    walk_step<SHIFT, 0>(k);
    k.tp += 16;
    k.ip += 8;
  }
  f32x2 v[4], wa, wb;
  walk_load<SHIFT, 0>(k, v, wa, wb);
  k.tp += 16;
  k.ip += 8;
  float w, w_;
  unpack2(wa, w, w_);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    // (single multiply-adds, so that the row's values need not leave as register pairs)
    float v0, v1, a0, a1;
    unpack2(v[i], v0, v1);
    unpack2(k.acc_a[i], a0, a1);
    done[2 * i] = __fmaf_rn(v0, w, a0);
    done[2 * i + 1] = __fmaf_rn(v1, w, a1);
    k.acc_a[i] = fma2(v[i], wb, k.acc_b[i]);
    k.acc_b[i] = 0;
  }
}

// The vertical half of a stage: `rows` output rows of packed step counts.
template <bool SHIFT>
__device__ __forceinline__ void walk_stage(Walker& k, unsigned st, unsigned steps, int rows, int part_rows) {
  float done[4][8];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    if (j < rows) {
      if ((j & (part_rows - 1)) == 0) {
        if (j > 0) {
          __syncwarp();   // nobody reads the rows before any more
          fetch_part(k);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();     // the rows as copied by all lanes
      }
      walk_row<SHIFT>(k, (int)(steps >> (8 * j)) & 255, done[j]);
    } else {
#pragma unroll
      for (int i = 0; i < 8; i++) {
        done[j][i] = 0.0f;
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const unsigned d = st ^ (16u * j);
    sts_v4(d, done[0][j], done[1][j], done[2][j], done[3][j]);
    sts_v4(d + 2048u, done[0][4 + j], done[1][4 + j], done[2][4 + j], done[3][4 + j]);
  }
}

// One tap of the horizontal filter: all channels of a source pixel in the four
// rows, at shared address a, weight w.  acc[2 * c + h]: rows 2h, 2h + 1 of
// channel c.
template <int C>
__device__ __forceinline__ void tap(unsigned a, float w, f32x2 (&acc)[2 * C]) {
  const f32x2 ww = pack2(w, w);
  f32x2 x, y;
  lds_v2u64<0>(a, x, y);
  ffma2(acc[0], x, ww);
  ffma2(acc[1], y, ww);
  if (C > 1) {
    lds_v2u64<16>(a, x, y);
    ffma2(acc[2 % (2 * C)], x, ww);
    ffma2(acc[3 % (2 * C)], y, ww);
  }
  if (C > 2) {
    lds_v2u64<32>(a, x, y);
    ffma2(acc[4 % (2 * C)], x, ww);
    ffma2(acc[5 % (2 * C)], y, ww);
  }
  if (C > 3) {
    lds_v2u64<48>(a, x, y);
    ffma2(acc[6 % (2 * C)], x, ww);
    ffma2(acc[7 % (2 * C)], y, ww);
  }
}

__device__ __forceinline__ Axis planned_axis(const float (&planned)[2], int n, int m) {
  Axis a;
  a.identity = n == m;
  a.ratio = planned[0];
  a.fs = planned[1];
  a.radius = a.ratio > 1.0f ? a.ratio : 1.0f;
  return a;
}

// What a warp knows of its strip once the tables are in place.
struct Strip {
  unsigned mid, hx, hw;      // shared addresses
  unsigned count;            // steps of its output rows
  int rows, passes, part_rows;
  int y0, x0, x1;            // its part of the slot
  int first_col, last_col;   // shared addresses of its first and last source column
  bool edge_x, shifted;
};

template <int C, bool GRAY, bool U8>
__device__ __forceinline__ void walk_strip(
    const DevSample& s, const LaunchParams& p, unsigned lut, const Strip& c, Walker& k) {
  constexpr int CO = GRAY ? 1 : C;
  const int lane = threadIdx.x & 31;
  const size_t row_stride = (size_t)s.slot_w * CO;
  const bool post_flip = s.post_flip != 0;
  void* const dst = s.dst;   // (a copy: the stores could otherwise have changed it)
  const bool vec_ok = (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
  const unsigned hstep = (unsigned)c.passes * 128u;
  const int tap_step = s.pre_flip ? -16 * C : 16 * C;
  // where byte 0 of word A goes; the others are 16 bytes on each, exclusive-or, so that
  // eight neighbouring lanes meet no bank twice
  const unsigned st = c.mid + (unsigned)lane * 64u + (unsigned)((lane >> 1) & 3) * 16u;
  lds_v2u32<0>(k.ip, k.place, k.shift);
  k.ip += 8;
#pragma unroll 1
  for (int r0 = 0; r0 < c.rows; r0 += 4) {
    const int rows = min(4, c.rows - r0);
    const unsigned steps = __shfl_sync(0xffffffffu, lds_u32<0>(c.count + (unsigned)r0), 0);
    if (c.shifted) {
      walk_stage<true>(k, st, steps, rows, c.part_rows);
    } else {
      walk_stage<false>(k, st, steps, rows, c.part_rows);
    }
    __syncwarp();
    if (r0 + 4 < c.rows) {
      fetch_part(k);
    }
    const size_t row_at = (size_t)(c.y0 + r0) * row_stride;
#pragma unroll 1
    for (int pass = 0; pass < c.passes; pass++) {
      const unsigned e = (unsigned)(pass * 32 + lane);
      uint32_t hx, col;
      lds_v2u32<0>(c.hx + 8u * e, hx, col);
      const int cnt = (int)(hx >> 16);
      unsigned wq = c.hw + 4u * e;
      f32x2 acc[2 * C];
#pragma unroll
      for (int i = 0; i < 2 * C; i++) {
        acc[i] = 0;
      }
      if (!c.edge_x) {
        unsigned a = c.mid + (hx & 0xffffu);
#pragma unroll 1
        for (int t = 0; t < cnt; t++) {
          tap<C>(a, __uint_as_float(lds_u32<0>(wq)), acc);
          a += tap_step;
          wq += hstep;
        }
      } else {
        // taps beyond the image read its first or last column, which is then the strip's
        int a = (int)c.mid + (int16_t)(hx & 0xffffu);
#pragma unroll 1
        for (int t = 0; t < cnt; t++) {
          tap<C>((unsigned)clampi(a, c.first_col, c.last_col), __uint_as_float(lds_u32<0>(wq)), acc);
          a += tap_step;
          wq += hstep;
        }
      }
      if (cnt > 0) {
        const int ox = post_flip ? c.x1 - 1 - (int)col : c.x0 + (int)col;
        store_column<C, GRAY, U8>(p, lut, acc, rows, dst, row_at + (size_t)ox * CO, row_stride, vec_ok);
      }
    }
  }
}

// Rows [y0, y1) x columns [x0, x1) of the slot, all inside the post window: a strip.
template <int C, bool GRAY, bool U8>
__device__ __forceinline__ void walk_cell(
    const DevSample& s, const LaunchParams& p, const StripPlan& plan, const StripSmem& sm, int y0, int y1, int x0, int x1) {
  constexpr int CO = GRAY ? 1 : C;
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // (so that what depends on it is known to be uniform)
  const int nc = x1 - x0;
  const int bx = s.post_x + (s.post_flip ? s.post_w - x1 : x0);   // first geometric column
  const int ra = y0 + warp * s.walk_rows;
  const int rows = min(s.walk_rows, y1 - ra);                     // this warp's, if any
  const int by = s.post_y + ra;
  const int pre_w = s.pre_w, pre_h = s.pre_h;
  const bool pre_flip = s.pre_flip != 0;
  const Axis ay = planned_axis(s.axis_y, pre_h, s.geom_h);
  const Axis ax = planned_axis(s.axis_x, pre_w, s.geom_w);
  // the cast table's values set out here and are stored behind the other tables
  constexpr int kLutQuads = U8 ? 0 : CO * 64;
  const bool looks_up = p.cast.mode == kCastTable;
  float4 lut[2] = {};
#pragma unroll
  for (int i = 0; i < 2; i++) {
    if (looks_up && tid + i * kStripThreads < kLutQuads) {
      lut[i] = __ldg(reinterpret_cast<const float4*>(p.lut) + tid + i * kStripThreads);
    }
  }
  const unsigned pitch = (unsigned)s.src_w * C;
  const bool shifted = (pitch & 3) != 0;   // rows start at different bytes of a word

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
  const int wbytes = (chi - clo + 1) * C;
  const uintptr_t g0 = reinterpret_cast<uintptr_t>(s.src) + ((size_t)s.pre_y * s.src_w + (s.pre_x + clo)) * C;
  const int common = shifted ? 0 : (int)(g0 & 3);
  Strip c;
  c.passes = (nc + 31) >> 5;
  if (wbytes > kStripRow) {
    if (tid == 0) {
      atomicOr(p.status, 8);
    }
    return;
  }
  c.part_rows = sm.part_rows;
  c.mid = sm.mid + (unsigned)warp * kMidBytes;
  c.hx = sm.hx;
  c.hw = sm.hw;
  c.count = sm.count + (unsigned)warp * kStripMaxRows;
  c.rows = rows;
  c.y0 = ra;
  c.x0 = x0;
  c.x1 = x1;
  c.first_col = (int)c.mid + common * 16;
  c.last_col = c.first_col + (chi - clo) * C * 16;
  c.edge_x = f0 < 0 || l1 > pre_w - 1;
  c.shifted = shifted;
  Walker k;
  const unsigned ring = sm.ring + (unsigned)warp * sm.ring_bytes;
  const unsigned unit = (unsigned)(lane & 15) * 16u;
  k.base = g0 + unit;
  k.pitch = pitch;
  k.row_max = pre_h - 1;
  k.from = (int)unit - wbytes;
  k.dst = ring + (unsigned)(lane >> 4) * kSlotBytes + unit;
  k.lane4 = (unsigned)lane * 4u;
  k.tp = sm.weights + (unsigned)(warp * sm.steps) * 16u;
  k.ip = sm.places + (unsigned)(warp * sm.steps) * 8u;
  k.part = sm.parts + (unsigned)warp * sm.parts_bytes;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    k.sel[j] = 0x4440u + (unsigned)(j ^ ((lane >> 1) & 3));
    k.acc_a[j] = 0;
    k.acc_b[j] = 0;
  }

  // ---- this warp's rows ---------------------------------------------------------------
  // Steps of output row a: source rows first .. hi, where first continues behind the
  // row before but goes back to the first tap of row a + 1 if that lies before (its
  // weight in row a is then 0: row a had it already).
  bool bad = false;
  if (rows > 0) {
    static_assert(kStripMaxRows <= 32, "one lane per output row");
    int lo = 0, hi = -1;
    if (lane < rows) {
      axis_range(ay, by + lane, lo, hi);
    }
    const int hi_before = __shfl_up_sync(0xffffffffu, hi, 1);
    const int lo_after = __shfl_down_sync(0xffffffffu, lo, 1);
    int f = lane == 0 ? lo : hi_before + 1;
    if (lane + 1 < rows) {
      f = min(f, lo_after);
    }
    f = min(f, hi);
    // parts: the source rows of part_rows output rows are in the ring together
    const int last_of_part = min(lane | (c.part_rows - 1), rows - 1);
    const int part_first = __shfl_sync(0xffffffffu, f, lane & ~(c.part_rows - 1));
    const int part_last = __shfl_sync(0xffffffffu, hi, last_of_part);
    const int own = lane < rows ? hi - f + 1 : 0;
    int sum = own;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, sum, d);
      sum += lane >= d ? t : 0;
    }
    bad = __any_sync(0xffffffffu, lane < rows && (sum > min(sm.steps, plan.steps) || part_last - part_first >= sm.slots || own > 255));
    if (!bad) {
      fetch_rows(k, __shfl_sync(0xffffffffu, part_first, 0), __shfl_sync(0xffffffffu, part_last, 0));
      if (lane < rows) {
        sp<uint8_t>(c.count)[lane] = (uint8_t)own;
        if ((lane & (c.part_rows - 1)) == 0) {
          sp<int>(k.part)[2 * (lane / c.part_rows)] = part_first;
          sp<int>(k.part)[2 * (lane / c.part_rows) + 1] = part_last;
        }
      }
      // (the float rows are not in use yet: scratch of the step table)
      const unsigned row_tables = c.mid, owners = c.mid + 48u * kStripMaxRows;
      float u = (float)(by + lane), total = 1.0f;
      if (!ay.identity) {
        u = axis_center(ay, by + lane);
        total = 0.0f;
#pragma unroll 1
        for (int t = lo; t <= hi; t++) {
          total = __fadd_rn(total, axis_tent(ay, u, t));
        }
      }
      const float u_after = __shfl_down_sync(0xffffffffu, u, 1);
      const float total_after = __shfl_down_sync(0xffffffffu, total, 1);
      const int at = sum - own;
      if (lane < rows) {
        const bool next = lane + 1 < rows;
        const unsigned e = row_tables + 48u * (unsigned)lane;
        sts_v4(e, __int_as_float(f - at), __int_as_float(lane == 0 ? lo : max(lo, hi_before + 1)),
               __int_as_float(next ? lo_after : 0x7fffffff), __int_as_float(part_first));
        sts_v4(e + 16u, u, total, next ? u_after : 0.0f, next ? total_after : 1.0f);
        for (int i = 0; i < own; i++) {
          *sp<uint8_t>(owners + (unsigned)(at + i)) = (uint8_t)lane;
        }
      }
      const int steps = __shfl_sync(0xffffffffu, sum, 31);
      __syncwarp();
#pragma unroll 1
      for (int i = lane; i < steps; i += 32) {
        const unsigned e = row_tables + 48u * *sp<uint8_t>(owners + (unsigned)i);
        uint32_t base, from, from_b, origin;
        lds_v4u32<0>(e, base, from, from_b, origin);
        const float4 w = *sp<float4>(e + 16u);   // centre and sum of the row, of the row after it
        const int row = (int)base + i;
        const float ta = row >= (int)from ? axis_tent(ay, w.x, row) : 0.0f;
        const float tb = row >= (int)from_b ? axis_tent(ay, w.z, row) : 0.0f;
        const float wa = __fmul_rn(__fdiv_rn(ta, w.y), kScaleY);
        const float wb = __fmul_rn(__fdiv_rn(tb, w.w), kScaleY);
        sts_v4(k.tp + 16u * (unsigned)i, wa, wa, wb, wb);
        const unsigned o = ((unsigned)g0 + (unsigned)clampi(row, 0, pre_h - 1) * pitch) & 15u;
        uint32_t* place = sp<uint32_t>(k.ip + 8u * (unsigned)i);
        place[0] = ring + (unsigned)(row - (int)origin) * kSlotBytes + (o & 12u);
        place[1] = (o & 3u) * 8u;
      }
      k.part += 8;
    } else if (lane == 0) {
      atomicOr(p.status, 8);
    }
  }

  // ---- columns: a pass to a warp, or one's taps to two or all of them -----------------
  const int columns = c.passes * 32;
  const int sharers = c.passes == 1 ? kWarps : c.passes == 2 ? kWarps / 2 : 1;
  const int share = sharers == 1 ? 0 : warp / c.passes;
#pragma unroll 1
  for (int pass = sharers == 1 ? warp : warp % c.passes; pass < c.passes; pass += kWarps) {
    const int x = pass * 32 + lane;
    const bool valid = x < nc;
    int lo = 0, hi = -1;
    if (valid) {
      axis_range(ax, bx + x, lo, hi);
    }
    int cnt = hi - lo + 1;
    cnt = cnt > s.cap_x ? s.cap_x : cnt;
    const int at = common + ((pre_flip ? pre_w - 1 - lo : lo) - clo) * C;   // may lie outside the image by the filter's radius
    // Which lane takes which column: columns sorted by the bank of their first
    // tap are dealt to the four groups of eight lanes that a 16-byte load serves
    // at a time, so that a group's columns meet in as few banks as possible.
    const unsigned all = __ballot_sync(0xffffffffu, valid);
    const unsigned b0 = __ballot_sync(0xffffffffu, (at & 1) != 0);
    const unsigned b1 = __ballot_sync(0xffffffffu, (at & 2) != 0);
    const unsigned b2 = __ballot_sync(0xffffffffu, (at & 4) != 0);
    const unsigned e2 = at & 4 ? b2 : ~b2, e1 = at & 2 ? b1 : ~b1, e0 = at & 1 ? b0 : ~b0;
    const unsigned below = (1u << lane) - 1u;
    const unsigned less = (at & 4 ? ~b2 : 0u) | (e2 & ((at & 2 ? ~b1 : 0u) | (e1 & (at & 1 ? ~b0 : 0u))));
    const int place = valid ? __popc(all & (less | (e2 & e1 & e0 & below))) : __popc(all) + __popc(~all & below);
    // In an enlargement neighbouring columns read the same pixels, which one access serves:
    // there they stay together (141 images of 41x41x4 to 174x174: 61.8 us dealt, 41.4 so).
    const int e = pass * 32 + (ax.ratio < 1.0f ? lane : (place & 3) * 8 + (place >> 2));
    if (share == 0) {
      uint32_t* hx = sp<uint32_t>(c.hx + 8u * (unsigned)e);
      hx[0] = (uint32_t)((at * 16) & 0xffff) | ((uint32_t)cnt << 16);
      hx[1] = (uint32_t)x;
    }
    float* w = sp<float>(c.hw) + e;
    float u = (float)(bx + x), sum = 1.0f;
    if (!ax.identity) {
      u = axis_center(ax, bx + x);
      sum = 0.0f;
#pragma unroll 1
      for (int t = 0; t < cnt; t++) {
        sum = __fadd_rn(sum, axis_tent(ax, u, lo + t));
      }
    }
#pragma unroll 1
    for (int t = share; t < cnt; t += sharers) {
      w[t * columns] = __fmul_rn(__fdiv_rn(axis_tent(ax, u, lo + t), sum), kScaleX);
    }
  }
#pragma unroll
  for (int i = 0; i < 2; i++) {
    if (looks_up && tid + i * kStripThreads < kLutQuads) {
      sp<float4>(sm.lut)[tid + i * kStripThreads] = lut[i];
    }
  }
  __syncthreads();
  if (rows > 0 && !bad) {
    walk_strip<C, GRAY, U8>(s, p, sm.lut, c, k);
  }
}

// One cell: a strip (or one of padding) of a slot.
// OWN: samples count their own cells off (StripPlan::cells_y of 0).
template <int C, bool GRAY, bool U8, bool OWN, int K>
__global__ void __launch_bounds__(kStripThreads, kStripCtas)
    resize_strip_kernel(
        const __grid_constant__ LaunchParams p, const __grid_constant__ StripPlan plan,
        const __grid_constant__ Records<K> records) {
  extern __shared__ __align__(64) unsigned char smem_raw[];
  constexpr int CO = GRAY ? 1 : C;
  unsigned t = blockIdx.x;
  int cx = (int)blockIdx.x, cy = (int)blockIdx.y;
  unsigned cell = 0;
  if (p.pad_apart) {
    // the first mixed_blocks hold all that walk and, evenly among them, fill_ratio / 2^32 that fill
    const bool mixed = t < plan.mixed_blocks;
    const unsigned fills = mixed ? (unsigned)((unsigned long long)t * plan.fill_ratio >> 32) : t - plan.walks;
    if (!mixed || (unsigned)((unsigned long long)(t + 1) * plan.fill_ratio >> 32) != fills) {
      pad_below_any<kStripThreads>(p, records, fills);
      return;
    }
    t -= fills;
  }
  if (plan.linear) {
    cell = t % plan.cells_x;
    t /= plan.cells_x;
    if (!OWN) {
      cx = (int)cell;
      cy = (int)(t % plan.cells_y);
      t /= plan.cells_y;
    }
  } else {
    t = blockIdx.z;
  }
  // (strips that end in the channel reduction and look casts up gain nothing: 500 of 400x400 to
  // 224x224 204.6 us with the whole record asked for, 202.6 without)
  const DevSample& s = *(GRAY && !U8 ? records.of(p, t) : records.whole(p, t));
  if (s.mode != kModeResize) {
    return;   // the other kernels'
  }
  const int slot_h = s.slot_h, slot_w = s.slot_w, post_h = s.post_h, post_w = s.post_w;
  const int chunks = s.walk_chunks;
  const int cell_rows = s.walk_rows * kWarps;
  if (OWN) {
    const unsigned cells_x = (unsigned)(chunks + walk_strips(s));
    cx = (int)(cell % cells_x);
    cy = (int)(cell / cells_x);
    if (cy >= (slot_h + cell_rows - 1) / cell_rows) {
      return;
    }
  }
  const int y0 = cy * cell_rows;
  const bool pad = cx >= chunks;   // a strip of kWalkPadPx columns of padding
  const int x0 = pad ? post_w + (cx - chunks) * kWalkPadPx : cx * s.walk_px;
  const int x1 = pad ? min(x0 + kWalkPadPx, slot_w) : min(x0 + s.walk_px, post_w);
  if (y0 >= slot_h || x0 >= x1) {
    return;
  }
  const int y1 = min(y0 + cell_rows, slot_h);
  const int vy1 = min(y1, post_h);
  const int fill_y0 = pad ? y0 : max(y0, post_h);     // rows of the cell that are padding
  const int fill_y1 = p.pad_apart ? vy1 : y1;         // rows below the post window are the fill CTAs' then
  if (!pad && y0 < vy1) {
    StripSmem sm;
    strip_layout(s, table_channels(p), smem_addr(smem_raw), &sm);
    walk_cell<C, GRAY, U8>(s, p, plan, sm, y0, vy1, x0, x1);
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
constexpr size_t kStripMaxSmem = kWarps * (kMidBytes + kStripSlots * kSlotBytes + kStripMaxSteps * 24u + kStripMaxRows * 9u) +
    4 * 1024 + kStripMaxPx * 8 + kStripMaxTaps * 4;

template <int C, bool GRAY, bool U8, bool OWN, int K>
cudaError_t launch_kernel(
    const LaunchParams& p, const StripPlan& plan, dim3 blocks, size_t smem, const Records<K>& records, cudaStream_t stream) {
  // More than the 48 KB that every kernel may have is asked for.  The limit belongs to
  // the kernel on the current device and is shared by all host threads, so each of
  // them sets the same value: one that set its own launch's need could lower the
  // limit between another's setting and its launch.
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(
        resize_strip_kernel<C, GRAY, U8, OWN, K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStripMaxSmem);
    if (e != cudaSuccess) {
      return e;
    }
  }
  resize_strip_kernel<C, GRAY, U8, OWN, K><<<blocks, kStripThreads, smem, stream>>>(p, plan, records);
  return cudaGetLastError();
}

template <int C, bool GRAY, bool U8>
cudaError_t launch(const LaunchParams& p, const StripPlan& plan, dim3 blocks, size_t smem, cudaStream_t stream) {
  return with_records(p, [&](const auto& records) {
    return plan.cells_y == 0 ? launch_kernel<C, GRAY, U8, true>(p, plan, blocks, smem, records, stream)
                             : launch_kernel<C, GRAY, U8, false>(p, plan, blocks, smem, records, stream);
  });
}

} // namespace

cudaError_t launch_resize_strip(const LaunchParams& p, const StripPlan& plan_in, cudaStream_t stream) {
  StripPlan plan = plan_in;
  unsigned long long blocks = (unsigned long long)p.n * std::max(plan.cells_y, 1) * plan.cells_x;
  if (blocks == 0) {
    return cudaSuccess;
  }
  if (p.pad_apart) {
    // Filling is bound by memory writes, walking by the SMs: the fill CTAs go among
    // the others instead of into a launch of their own.  The walks take long, so the
    // last of them start when a quarter of the filling is still to come: 64 images of
    // 160-1024 px padded to the largest (2 GB written) take 377 us a pass so, 385 / 396
    // / 404 with the walks among the first 50 / 25 / 5 % of the fill CTAs, 392 among all.
    const unsigned long long fills = (unsigned long long)p.n * kPadChunks;
    const unsigned long long among = fills / 4 * 3;
    plan.walks = (uint32_t)blocks;
    plan.mixed_blocks = (uint32_t)(blocks + among);
    plan.fill_ratio = (uint32_t)(((among << 32) + blocks + among - 1) / (blocks + among));
    blocks += fills;
  }
  if (blocks > 0x7fffffffULL) {
    return cudaErrorInvalidConfiguration;
  }
  // Blocks name their cell by three coordinates, which saves two divisions, where they can.
  plan.linear = p.pad_apart || plan.cells_y == 0 || plan.cells_y > 65535 || p.n > 65535;
  const dim3 b = plan.linear ? dim3((unsigned)blocks) : dim3((unsigned)plan.cells_x, (unsigned)plan.cells_y, (unsigned)p.n);
  const size_t smem = (size_t)plan.bytes + (size_t)table_channels(p) * 1024;
  if (p.out_f32) {
    if (p.gray) {
      return launch<3, true, false>(p, plan, b, smem, stream);
    }
    switch (p.c_in) {
      case 1:
        return launch<1, false, false>(p, plan, b, smem, stream);
      case 2:
        return launch<2, false, false>(p, plan, b, smem, stream);
      case 3:
        return launch<3, false, false>(p, plan, b, smem, stream);
      default:
        return launch<4, false, false>(p, plan, b, smem, stream);
    }
  }
  if (p.gray) {
    return launch<3, true, true>(p, plan, b, smem, stream);
  }
  switch (p.c_in) {
    case 1:
      return launch<1, false, true>(p, plan, b, smem, stream);
    case 2:
      return launch<2, false, true>(p, plan, b, smem, stream);
    case 3:
      return launch<3, false, true>(p, plan, b, smem, stream);
    default:
      return launch<4, false, true>(p, plan, b, smem, stream);
  }
}

} // namespace mlxd
