// The kernels around the resize kernels (resize_strip.cu, resize_walk.cu) and the rotations
// (affine.cu): bands of copies (crop / flip / batch only), padding of ragged batches, and
// resizes whose taps fit no chunk of resize_walk.cu.
//
// Copies: one CTA per band of up to eight kTileH x kTileW tiles of one sample's slot;
// the source is read through the read-only path, four pixels per thread, and stored 16
// bytes at a time; pad-only bands are plain 16-byte stores.  The rows below a sample in
// a ragged batch go out through a linear fill kernel when the launch has no resize (else
// CTAs of a resize kernel write them).  A resize too strong for both resize kernels is
// filtered pixel by pixel from global memory by a kernel of its own.
#include "fused_batch.h"
#include "kernel_common.cuh"

namespace mlxd {
namespace {

// N floats that start HEAD floats before a 16-byte boundary: whole 16-byte units
// where they lie, single floats around them.
template <int N, int HEAD>
__device__ __forceinline__ void store_run(float* dst, const float* v) {
#pragma unroll
  for (int i = 0; i < HEAD; i++) {
    dst[i] = v[i];
  }
#pragma unroll
  for (int i = HEAD; i + 4 <= N; i += 4) {
    *reinterpret_cast<float4*>(dst + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
  }
#pragma unroll
  for (int i = HEAD + (N - HEAD) / 4 * 4; i < N; i++) {
    dst[i] = v[i];
  }
}

// Copies (crop / flip / batch only): rows [y0, vy1) x columns [xa, xb) of the slot, a
// thread takes four adjacent pixels of a row, which come as aligned words.  The cast
// table is read from shared memory (lut_s); the four pixels leave as 16-byte stores
// when the row segment allows it.
template <int C, bool GRAY, bool U8>
__device__ void copy_rows(
    const DevSample& s, const LaunchParams& p, unsigned lut_s, int y0, int vy1, int xa, int xb) {
  constexpr int CO = GRAY ? 1 : C;
  const int nvx = xb - xa;
  const int nvy = vy1 - y0;
  const int quads = (nvx + 3) >> 2;
  float* base = reinterpret_cast<float*>(s.dst);
  const size_t row_floats = (size_t)s.slot_w * CO;
  const bool vec_ok = (row_floats & 3) == 0 && ((xa * CO) & 3) == 0 && (reinterpret_cast<uintptr_t>(base) & 15) == 0;
  // last 4-byte word of the source image: nothing behind it is read
  const uintptr_t last_word = (reinterpret_cast<uintptr_t>(s.src) + (size_t)s.src_h * s.src_w * C - 1) & ~(uintptr_t)3;
  for (int i = threadIdx.x; i < nvy * quads; i += kThreads) {
    const int ry = i / quads;
    const int q = i - ry * quads;
    const int x_first = xa + 4 * q;
    const int npx = min(4, xb - x_first);
    const int gy = s.post_y + y0 + ry;
    unsigned px[4][C];   // source bytes of the four pixels
    // pre_flip is folded into post_flip for copies: the source pixels of columns
    // x_first .. x_first + 3 are adjacent, ascending or (mirrored) descending
    const int gx_a = s.post_x + (s.post_flip ? (s.post_w - 1 - x_first) : x_first);
    const int sx_lo = s.pre_x + (s.post_flip ? gx_a - (npx - 1) : gx_a);
    const uintptr_t g =
        reinterpret_cast<uintptr_t>(s.src) + ((size_t)(s.pre_y + gy) * s.src_w + sx_lo) * C;
    const uint32_t* w = reinterpret_cast<const uint32_t*>(g & ~(uintptr_t)3);
    const unsigned sh = (unsigned)(g & 3) * 8u;
    const int need = (int)(g & 3) + npx * C;   // bytes from the first word on
    uint32_t x[C + 1];
#pragma unroll
    for (int k = 0; k < C + 1; k++) {
      const bool take = 4 * k < need && reinterpret_cast<uintptr_t>(w + k) <= last_word;
      x[k] = take ? __ldg(w + k) : 0u;
    }
    uint32_t v[C];   // the 4 * C bytes from g on
#pragma unroll
    for (int k = 0; k < C; k++) {
      v[k] = __funnelshift_r(x[k], x[k + 1], sh);
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
#pragma unroll
      for (int ch = 0; ch < C; ch++) {
        const int byte = j * C + ch;
        // mirrored: output pixel j is source pixel npx - 1 - j; places a row's last
        // quad leaves over index the cast table too, so they get some byte of the quad
        const int back = ((npx - 1 - j) & 3) * C + ch;
        unsigned val = (v[byte >> 2] >> (8 * (byte & 3))) & 0xffu;
        if (s.post_flip) {
          val = 0;
#pragma unroll
          for (int o = 0; o < 4; o++) {
            const int from = o * C + ch;
            val = back == from ? (v[from >> 2] >> (8 * (from & 3))) & 0xffu : val;
          }
        }
        px[j][ch] = val;
      }
    }
    if (U8) {
      // uint8 batch: the 4 * CO bytes as CO aligned words when the row segment allows it
      unsigned by[4 * CO];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if (GRAY) {
          by[j] = gray_mix(p, px[j][0], px[j][1 % C], px[j][2 % C]);
        } else {
#pragma unroll
          for (int ch = 0; ch < C; ch++) {
            by[(j * CO + ch) % (4 * CO)] = px[j][ch];
          }
        }
      }
      uint8_t* dst8 = reinterpret_cast<uint8_t*>(s.dst) + ((size_t)(y0 + ry) * s.slot_w + x_first) * CO;
      if (npx == 4 && (reinterpret_cast<uintptr_t>(dst8) & 3) == 0) {
#pragma unroll
        for (int k = 0; k < CO; k++) {
          reinterpret_cast<uint32_t*>(dst8)[k] =
              by[4 * k] | (by[4 * k + 1] << 8) | (by[4 * k + 2] << 16) | (by[4 * k + 3] << 24);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 4; j++) {
          if (j < npx) {
#pragma unroll
            for (int ch = 0; ch < CO; ch++) {
              dst8[j * CO + ch] = (uint8_t)by[j * CO + ch];
            }
          }
        }
      }
    } else {
      float out[4][CO];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if (GRAY) {
          out[j][0] = __uint_as_float(lds_u32<0>(lut_s + 4u * gray_mix(p, px[j][0], px[j][1 % C], px[j][2 % C])));
        } else {
#pragma unroll
          for (int ch = 0; ch < C; ch++) {
            out[j][ch % CO] = __uint_as_float(lds_u32<0>(lut_s + (unsigned)ch * 1024u + 4u * px[j][ch]));
          }
        }
      }
      float* dst = base + ((size_t)(y0 + ry) * s.slot_w + x_first) * CO;
      if (vec_ok && npx == 4) {
        const float* o = &out[0][0];
#pragma unroll
        for (int k = 0; k < CO; k++) {
          reinterpret_cast<float4*>(dst)[k] = make_float4(o[4 * k], o[4 * k + 1], o[4 * k + 2], o[4 * k + 3]);
        }
      } else if (CO > 1 && npx == 4) {
        // A row that starts off a 16-byte boundary (odd widths).  Single floats alone, a
        // lane's 4 * CO apart from the next lane's, bring each 32-byte sector to L2 once per
        // float in it: 64 mirrored images of 719x1279x3 487 us a pass, 259 with these units.
        const float* o = &out[0][0];
        switch ((reinterpret_cast<uintptr_t>(dst) >> 2) & 3) {
          case 0:
            store_run<4 * CO, 0>(dst, o);
            break;
          case 1:
            store_run<4 * CO, 3>(dst, o);
            break;
          case 2:
            store_run<4 * CO, 2>(dst, o);
            break;
          default:
            store_run<4 * CO, 1>(dst, o);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 4; j++) {
          if (j < npx) {
#pragma unroll
            for (int ch = 0; ch < CO; ch++) {
              dst[j * CO + ch] = out[j][ch];
            }
          }
        }
      }
    }
  }
}

// One CTA: rows [y0, y0 + kTileH) of one slot, columns of p.band_tiles tiles.
template <int C, bool GRAY, bool U8, int K>
__device__ void run_band(const LaunchParams& p, const Records<K>& records, float* lut_s) {
  unsigned t = blockIdx.x;
  const int tb = t % p.bands_x;
  t /= p.bands_x;
  const int ty = t % p.tiles_y;
  const int n = t / p.tiles_y;
  if (n >= p.n) {
    return;
  }
  const DevSample* const sample = records.of(p, (unsigned)n);
  if (sample->mode != kModeCopy && sample->mode != kModeResizeDirect) {
    return;   // the other kernels'
  }
  const DevSample s = *sample;
  const int y0 = ty * kTileH;
  const int x0 = tb * p.band_tiles * kTileW;
  if (y0 >= s.slot_h || x0 >= s.slot_w) {
    return;
  }
  const int y1 = min(y0 + kTileH, s.slot_h);
  const int x1 = min(x0 + p.band_tiles * kTileW, s.slot_w);
  const int vy1 = min(y1, s.post_h);
  const int vx1 = min(x1, s.post_w);
  const bool has_valid = (y0 < vy1) && (x0 < vx1);
  constexpr int CO = GRAY ? 1 : C;
  float padf[4];
#pragma unroll
  for (int c = 0; c < 4; c++) {
    padf[c] = (!U8 && c < CO) ? __ldg(p.lut + c * 256 + p.pad_px) : 0.0f;
  }
  float* out = reinterpret_cast<float*>(s.dst);
  // pad value into a rectangle of the slot, float32 or uint8
  auto pad_rect = [&](int ya, int yb, int xa, int xb) {
    if (U8) {
      fill_rect_u8<CO>(reinterpret_cast<uint8_t*>(s.dst), s.slot_w, ya, yb, xa, xb, p.pad_px);
    } else {
      fill_rect_f32<CO>(out, s.slot_w, ya, yb, xa, xb, padf);
    }
  };
  if (!has_valid) {
    // bands below the post window are filled apart when p.pad_apart is set
    if (!(p.pad_apart && y0 >= s.post_h)) {
      pad_rect(y0, y1, x0, x1);
    }
    return;
  }
  if (!U8) {
    for (int i = threadIdx.x; i < CO * 256; i += kThreads) {
      lut_s[i] = __ldg(p.lut + i);
    }
  }
  if (s.mode != kModeResizeDirect) {
    __syncthreads();
    copy_rows<C, GRAY, U8>(s, p, smem_addr(lut_s), y0, vy1, x0, vx1);
  }
  // (the post window of a kModeResizeDirect sample is resize_direct_kernel's)
  // pad the part of the band outside the post window
  if (!p.pad_apart) {
    pad_rect(vy1, y1, x0, x1);
  }
  pad_rect(y0, vy1, vx1, x1);
}

template <int K>
__global__ void __launch_bounds__(kThreads, 3) fused_fast_kernel(
    const __grid_constant__ LaunchParams p, const __grid_constant__ Records<K> records) {
  __shared__ __align__(16) float lut_s[4 * 256];
  if (p.c_in == 3) {
    run_band<3, false, false>(p, records, lut_s);
  } else if (p.c_in == 1) {
    run_band<1, false, false>(p, records, lut_s);
  } else {
    run_band<4, false, false>(p, records, lut_s);
  }
}

// Two-channel images, float32 batches.  Rare; kept out of the kernel above so
// that its register allocation is decided by the common cases alone.
template <int K>
__global__ void __launch_bounds__(kThreads, 3) fused_fast_c2_kernel(
    const __grid_constant__ LaunchParams p, const __grid_constant__ Records<K> records) {
  __shared__ __align__(16) float lut_s[2 * 256];
  run_band<2, false, false>(p, records, lut_s);
}

// uint8 batches (no cast): stand-alone ops, images between two geometric ops,
// pipelines that cast on the host.  Kernels of their own for the same reason
// as the channel-reduction one.
template <int K>
__global__ void __launch_bounds__(kThreads, 3) fused_fast_u8_kernel(
    const __grid_constant__ LaunchParams p, const __grid_constant__ Records<K> records) {
  __shared__ __align__(16) float lut_s[4];
  if (p.c_in == 3) {
    if (p.gray) {
      run_band<3, true, true>(p, records, lut_s);
    } else {
      run_band<3, false, true>(p, records, lut_s);
    }
  } else if (p.c_in == 1) {
    run_band<1, false, true>(p, records, lut_s);
  } else if (p.c_in == 2) {
    run_band<2, false, true>(p, records, lut_s);
  } else {
    run_band<4, false, true>(p, records, lut_s);
  }
}

template <int K>
__global__ void __launch_bounds__(kThreads, 6) pad_fill_kernel(
    const __grid_constant__ LaunchParams p, const __grid_constant__ Records<K> records) {
  pad_below_any<kThreads>(p, records, blockIdx.x);
}

// Launches that end in the channel reduction: three channels in, one out.  A
// kernel of its own, so that the usual one's register allocation is not touched.
template <int K>
__global__ void __launch_bounds__(kThreads, 3) fused_fast_gray_kernel(
    const __grid_constant__ LaunchParams p, const __grid_constant__ Records<K> records) {
  __shared__ __align__(16) float lut_s[256];
  run_band<3, true, false>(p, records, lut_s);
}

} // namespace

// ---- resizes whose taps do not fit a chunk of resize_walk.cu ------------------------------
//
// One thread per pixel of the post window, every tap read from global memory.
// The arithmetic is that of the resize kernels, value by value: per source column
// the vertical sum (multiply-adds in tap order, the first of them a product, taps
// outside the window reading the clamped row), then the horizontal multiply-adds
// over those sums in tap order onto zero, weights tent / sum with the sum taken in
// tap order.  Such samples are rare and small on the output side (launch_plan.cu: walk_fits: shrink
// ratios above 100 along a row, 500 down the rows), so nothing is staged or shared.
template <int C>
__device__ void direct_pixel(const DevSample& s, const LaunchParams& p, int ox, int oy) {
  const Axis ay = make_axis(s.pre_h, s.geom_h);
  const Axis ax = make_axis(s.pre_w, s.geom_w);
  const int gy = s.post_y + oy;
  const int gx = s.post_x + (s.post_flip ? s.post_w - 1 - ox : ox);
  int ylo, yhi, xlo, xhi;
  axis_range(ay, gy, ylo, yhi);
  axis_range(ax, gx, xlo, xhi);
  const int cy = yhi - ylo + 1;
  int cx = xhi - xlo + 1;
  cx = cx > s.cap_x ? s.cap_x : cx;
  const float uy = axis_center(ay, gy);
  const float ux = axis_center(ax, gx);
  float sum_y = 0.0f, sum_x = 0.0f;
  if (!ay.identity) {
    for (int k = 0; k < cy; k++) {
      sum_y = __fadd_rn(sum_y, axis_tent(ay, uy, ylo + k));
    }
  }
  if (!ax.identity) {
    for (int j = 0; j < cx; j++) {
      sum_x = __fadd_rn(sum_x, axis_tent(ax, ux, xlo + j));
    }
  }
  float acc_h[C];
#pragma unroll
  for (int c = 0; c < C; c++) {
    acc_h[c] = 0.0f;
  }
  for (int j = 0; j < cx; j++) {
    const float wx = ax.identity ? 1.0f : __fdiv_rn(axis_tent(ax, ux, xlo + j), sum_x);
    const int seen = clampi(xlo + j, 0, s.pre_w - 1);
    const int col = s.pre_x + (s.pre_flip ? s.pre_w - 1 - seen : seen);
    float acc_v[C];
#pragma unroll
    for (int c = 0; c < C; c++) {
      acc_v[c] = 0.0f;
    }
    for (int k = 0; k < cy; k++) {
      const float wy = ay.identity ? 1.0f : __fdiv_rn(axis_tent(ay, uy, ylo + k), sum_y);
      const int row = s.pre_y + clampi(ylo + k, 0, s.pre_h - 1);
      const uint8_t* px = s.src + ((size_t)row * s.src_w + col) * C;
#pragma unroll
      for (int c = 0; c < C; c++) {
        const float v = (float)__ldg(px + c);
        acc_v[c] = k == 0 ? __fmul_rn(v, wy) : __fmaf_rn(v, wy, acc_v[c]);
      }
    }
#pragma unroll
    for (int c = 0; c < C; c++) {
      acc_h[c] = __fmaf_rn(acc_v[c], wx, acc_h[c]);
    }
  }
  unsigned q[C];
#pragma unroll
  for (int c = 0; c < C; c++) {
    q[c] = quantise_sat(acc_h[c]);
  }
  const size_t at = (size_t)oy * s.slot_w + ox;
  if (p.gray) {
    const unsigned g = gray_mix(p, q[0], q[1 % C], q[2 % C]);
    if (p.out_f32) {
      reinterpret_cast<float*>(s.dst)[at] = __ldg(p.lut + g);
    } else {
      reinterpret_cast<uint8_t*>(s.dst)[at] = (uint8_t)g;
    }
  } else {
#pragma unroll
    for (int c = 0; c < C; c++) {
      if (p.out_f32) {
        reinterpret_cast<float*>(s.dst)[at * C + c] = __ldg(p.lut + c * 256 + q[c]);
      } else {
        reinterpret_cast<uint8_t*>(s.dst)[at * C + c] = (uint8_t)q[c];
      }
    }
  }
}

constexpr int kDirectChunks = 64;   // CTAs per sample

__global__ void __launch_bounds__(kThreads) resize_direct_kernel(const __grid_constant__ LaunchParams p) {
  const DevSample& s = *Records<0>().of(p, blockIdx.y);
  if (s.mode != kModeResizeDirect) {
    return;
  }
  const int vh = s.post_h < s.slot_h ? s.post_h : s.slot_h;
  const int vw = s.post_w < s.slot_w ? s.post_w : s.slot_w;
  const long long count = (long long)vh * vw;
  for (long long i = (long long)blockIdx.x * kThreads + threadIdx.x; i < count; i += (long long)kDirectChunks * kThreads) {
    const int oy = (int)(i / vw);
    const int ox = (int)(i - (long long)oy * vw);
    if (p.c_in == 3) {
      direct_pixel<3>(s, p, ox, oy);
    } else if (p.c_in == 1) {
      direct_pixel<1>(s, p, ox, oy);
    } else if (p.c_in == 2) {
      direct_pixel<2>(s, p, ox, oy);
    } else {
      direct_pixel<4>(s, p, ox, oy);
    }
  }
}

template <int K>
static void launch_fill(const LaunchParams& p, const Records<K>& records, cudaStream_t stream) {
  pad_fill_kernel<K><<<(unsigned)p.n * kPadChunks, kThreads, 0, stream>>>(p, records);
}

template <int K>
static void launch_band_kernel(const LaunchParams& p, const Records<K>& records, unsigned blocks, cudaStream_t stream) {
  if (!p.out_f32) {
    fused_fast_u8_kernel<K><<<blocks, kThreads, 0, stream>>>(p, records);
  } else if (p.c_in == 2) {
    fused_fast_c2_kernel<K><<<blocks, kThreads, 0, stream>>>(p, records);
  } else if (p.gray) {
    fused_fast_gray_kernel<K><<<blocks, kThreads, 0, stream>>>(p, records);
  } else {
    fused_fast_kernel<K><<<blocks, kThreads, 0, stream>>>(p, records);
  }
}

static cudaError_t launch_bands(LaunchParams p, cudaStream_t stream) {
  static thread_local int configured_device = -1;
  static thread_local int sm_count = 0;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) {
    return e;
  }
  if (configured_device != dev) {
    e = cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) {
      return e;
    }
    configured_device = dev;
  }
  // Tiles per CTA along a row band: as many as keeps about eight waves of CTAs
  // on the device (3 CTAs per SM), at most 8.
  const long long tiles = (long long)p.n * p.tiles_y * p.tiles_x;
  const long long want_ctas = (long long)sm_count * 3 * 8;
  int band = (int)(tiles / (want_ctas > 0 ? want_ctas : 1));
  band = band < 1 ? 1 : (band > 8 ? 8 : band);
  band = band > p.tiles_x ? p.tiles_x : band;
  p.band_tiles = band;
  p.bands_x = (p.tiles_x + band - 1) / band;
  const unsigned long long blocks = (unsigned long long)p.n * p.tiles_y * p.bands_x;
  if (blocks == 0) {
    return cudaSuccess;
  }
  if (blocks > 0x7fffffffULL) {
    return cudaErrorInvalidConfiguration;
  }
  return with_records(p, [&](const auto& records) {
    launch_band_kernel(p, records, (unsigned)blocks, stream);
    return cudaGetLastError();
  });
}

cudaError_t launch_fused_batch(const LaunchParams& described, const ResizePlan& plan, cudaStream_t stream) {
  LaunchParams p = described;
  if (p.n <= 0) {
    return cudaSuccess;
  }
  if (plan.enlarges) {
    // With two taps a column a resize is bound by the issue of instructions, and a look-up
    // has fewer: 128 images of 32x32 to 224x224 take 33.2 us with the table, 34.7 without.
    p.cast.mode = kCastTable;
  }
  const bool strips = plan.strip.bytes > 0, wides = plan.wide.px > 0;
  if (p.pad_apart && !strips && !wides) {   // a resize kernel fills the padding itself
    const cudaError_t e = with_records(p, [&](const auto& records) {
      launch_fill(p, records, stream);
      return cudaGetLastError();
    });
    if (e != cudaSuccess) {
      return e;
    }
  }
  if (strips) {
    const cudaError_t e = launch_resize_strip(p, plan.strip, stream);
    if (e != cudaSuccess) {
      return e;
    }
  }
  if (wides) {
    LaunchParams q = p;
    if (strips) {
      q.first += plan.first_wide;
      q.n = plan.wides;
    }
    const cudaError_t e = launch_resize_walk(q, !strips, stream);
    if (e != cudaSuccess) {
      return e;
    }
  }
  if (plan.affines > 0) {
    LaunchParams q = p;
    q.first += plan.first_affine;
    q.n = plan.affines;
    const cudaError_t e = launch_affine(q, stream);
    if (e != cudaSuccess) {
      return e;
    }
  }
  if (plan.bands > 0) {
    p.first += plan.first_band;
    p.n = plan.bands;
    const cudaError_t e = launch_bands(p, stream);
    if (e != cudaSuccess) {
      return e;
    }
  }
  if (p.direct) {
    resize_direct_kernel<<<dim3(kDirectChunks, (unsigned)p.n), kThreads, 0, stream>>>(p);
    return cudaGetLastError();
  }
  return cudaSuccess;
}

} // namespace mlxd
