// Nearest-neighbour affine samples (rotations): a warp takes four rows of the slot, 32 pixels
// of them at a time, a pixel a lane and row, so that the words of a load lie in different
// banks.  Their bytes go through shared memory, out of which they are cast and stored 16
// aligned bytes a lane, eight lanes to 128 consecutive bytes of a row; the next pixels' words
// set out before.
//
// The coordinate is built from float products and float sums in the order of the reference
// expression, no multiply-add contracted.  Its last step, trunc(((double)f + 0.5) + half),
// is a float sum here: c = half + 0.5 is exact (sides below 2^23), and f + c rounded toward
// zero has the truncation of the exact sum, since whole numbers of that size are floats;
// beyond it both are outside.  The double sums are exact too, or round by less than
// 2^-30, which reaches a whole number from below only where f itself is the whole distance:
// -2^-26 < f < 0 beside a whole c.  A warp that meets such an f takes the doubles.
//
// What bounds it (128 images of 512x512x3, an angle each, 448x448 floats: 102.5 us, 92.5 with the
// records as parameters, 113 in bands of CTA-wide 16x64-pixel tiles, four neighbouring pixels a
// lane): the latency of the loads at 24 warps an SM, the L1 pipe 60 % busy, DRAM 3.8 TB/s.
// The tiles' loads met 5.6 times in the banks (3 here), their stores brought sectors to L2
// by halves (15.2 M sectors, 9.6 here), and the coordinate took double additions and 64-bit
// conversions.  Bytes through shared memory make all stores whole lines whatever the row
// starts at: 128 of 511x511x3 to 447x447 109.7 us, 128 before; four channels 107 and 160,
// one channel 53.7 and 73.7, bytes 70 and 88.  Without the next words under way: 107 us;
// two rows of 16 pixels a load 107 to 112; eight by four with 8-byte loads 143.
#include <algorithm>
#include <type_traits>

#include "fused_batch.h"
#include "kernel_common.cuh"

namespace mlxd {
namespace {

constexpr int kAffineThreads = 128;
constexpr int kAffineCtas = 6;      // per SM
constexpr int kAffineRows = 4;      // of a warp
static_assert(kTileH == kAffineThreads / 32 * kAffineRows, "a CTA's rows are a band");

// Source pixel of a point (fx, fy) of an affine sample in the pre window (of half sides wh,
// hh): two double additions, then truncation toward zero, as in the reference expression;
// {-1, -1} where it falls outside.
__device__ __noinline__ int2 affine_exact(float fx, float fy, float wh, float hh, int pre_w, int pre_h) {
  const long long ax = (long long)__dadd_rn(__dadd_rn((double)fx, 0.5), (double)wh);
  const long long ay = (long long)__dadd_rn(__dadd_rn((double)fy, 0.5), (double)hh);
  const bool outside = ax < 0 || ay < 0 || ax >= pre_w || ay >= pre_h;
  return outside ? make_int2(-1, -1) : make_int2((int)ax, (int)ay);
}

// A window (or matrix) that affine_rows does not take: pixel by pixel.
template <int C, bool GRAY, bool U8>
__device__ __noinline__ void affine_pixels(const DevSample* sample, const LaunchParams& p, int y0, int vy1, int xa, int xb) {
  constexpr int CO = GRAY ? 1 : C;
  const DevSample& s = *sample;
  const float twh = (float)((double)s.geom_w / 2.0), thh = (float)((double)s.geom_h / 2.0);
  const float wh = (float)((double)s.pre_w / 2.0), hh = (float)((double)s.pre_h / 2.0);
  for (int y = y0; y < vy1; y++) {
    for (int x = xa + (int)threadIdx.x; x < xb; x += kAffineThreads) {
      const float dxf = __fsub_rn((float)(s.post_x + (s.post_flip ? s.post_w - 1 - x : x)), twh);
      const float dyf = __fsub_rn((float)(s.post_y + y), thh);
      const float fx = __fadd_rn(__fadd_rn(__fmul_rn(s.mx[0], dxf), __fmul_rn(s.mx[1], dyf)), s.mx[2]);
      const float fy = __fadd_rn(__fadd_rn(__fmul_rn(s.mx[3], dxf), __fmul_rn(s.mx[4], dyf)), s.mx[5]);
      const int2 at = affine_exact(fx, fy, wh, hh, s.pre_w, s.pre_h);
      const int ix = s.pre_x + (s.pre_flip ? s.pre_w - 1 - at.x : at.x);
      const uint8_t* const g = s.src + ((size_t)(s.pre_y + at.y) * s.src_w + ix) * C;
      unsigned px[C];
#pragma unroll
      for (int ch = 0; ch < C; ch++) {
        px[ch] = at.x < 0 ? 0u : __ldg(g + ch);
      }
      const unsigned gray = GRAY ? gray_mix(p, px[0], px[1 % C], px[2 % C]) : 0u;
      const size_t to = ((size_t)y * s.slot_w + x) * CO;
#pragma unroll
      for (int ch = 0; ch < CO; ch++) {
        const unsigned v = GRAY ? gray : px[ch];
        if (U8) {
          reinterpret_cast<uint8_t*>(s.dst)[to + ch] = (uint8_t)v;
        } else {
          reinterpret_cast<float*>(s.dst)[to + ch] = __ldg(p.lut + 256 * ch + v);
        }
      }
    }
  }
}

// What affine_rows takes: sides below 2^23, a pre window of less than 2^31 bytes, and a
// matrix whose products with them cannot overflow.
template <int C>
__device__ __forceinline__ bool affine_rows_take(const DevSample& s) {
  bool numbers = true;
#pragma unroll
  for (int i = 0; i < 6; i++) {
    numbers = numbers && fabsf(s.mx[i]) <= 0x1p40f;   // (false for a NaN)
  }
  return numbers && s.pre_w < (1 << 23) && s.pre_h < (1 << 23) && (size_t)s.pre_h * s.src_w * C < (1ull << 31);
}

// Whether a cast is computed; others look bytes up.
template <bool GRAY, bool U8>
__device__ __forceinline__ bool affine_scales(const LaunchParams& p) {
  return !GRAY && !U8 && p.cast.mode == kCastScale;
}

// Words of a lane's four pixels.
struct AffinePiece {
  uint32_t w0[4], w1[4];
  unsigned shift[4];
};

// Rows [ya, ya + rows) x columns [xa, xb) of the slot, inside the post window, by one warp.
// `patch`: shared address of its four rows of bytes.
template <int C, bool GRAY, bool U8>
__device__ __forceinline__ void affine_rows(
    const DevSample& s, const LaunchParams& p, unsigned lut_s, unsigned patch, int ya, int rows, int xa, int xb) {
  constexpr int CO = GRAY ? 1 : C;
  constexpr unsigned kRow = CO <= 2 ? 96u : 160u;   // bytes of a patch row: 8 words beyond a multiple of 16
  const int lane = threadIdx.x & 31;
  const float twh = (float)((double)s.geom_w / 2.0);
  const float thh = (float)((double)s.geom_h / 2.0);
  const float wh = (float)((double)s.pre_w / 2.0);
  const float hh = (float)((double)s.pre_h / 2.0);
  const float cx = __fadd_rn(wh, 0.5f), cy = __fadd_rn(hh, 0.5f);
  const int pre_w = s.pre_w, pre_h = s.pre_h;
  const float m0 = s.mx[0], m2 = s.mx[2], m3 = s.mx[3], m5 = s.mx[5];
  float m1y[4], m4y[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float dyf = __fsub_rn((float)(s.post_y + ya + i), thh);
    m1y[i] = __fmul_rn(s.mx[1], dyf);
    m4y[i] = __fmul_rn(s.mx[4], dyf);
  }
  // the window's first pixel: the word that holds it, and its offset there; a mirrored
  // window runs back from its last column
  const uintptr_t g0 = reinterpret_cast<uintptr_t>(s.src) + ((size_t)s.pre_y * s.src_w + s.pre_x) * C;
  const char* const words = reinterpret_cast<const char*>(g0 & ~(uintptr_t)3);
  const unsigned pitch = (unsigned)s.src_w * C;
  const unsigned first = (unsigned)(g0 & 3) + (s.pre_flip ? (unsigned)(pre_w - 1) * C : 0u);
  const int dir = s.pre_flip ? -C : C;
  const int dgx = s.post_flip ? -1 : 1;
  const int gx0 = (s.post_flip ? s.post_x + s.post_w - 1 : s.post_x) + dgx * (xa + lane);
  // Out of the patch a lane stores units of row `yo`, four elements that start on a multiple
  // of four: the segment's first element is `mis` elements into a unit, and so is every
  // piece's; it is `step` further in the next row.
  const int yo = lane >> 3;
  constexpr int kSize = U8 ? 1 : 4;
  uint8_t* const seg = reinterpret_cast<uint8_t*>(s.dst) + ((size_t)(ya + yo) * s.slot_w + xa) * (CO * kSize);
  const int step = (int)(((size_t)s.slot_w * CO) & 3);
  const int mis = (int)(reinterpret_cast<uintptr_t>(seg) / kSize & 3);
  unsigned to[4];   // this lane's pixel in the rows of the patch
#pragma unroll
  for (int i = 0; i < 4; i++) {
    to[i] = patch + (unsigned)i * kRow + (unsigned)((mis + (i - yo) * step) & 3) + (unsigned)(lane * CO);
  }
  const unsigned from = patch + (unsigned)yo * kRow + 4u * (unsigned)(lane & 7);
  // cast tables of the elements of a lane's first unit; 8 units on, the channel is two further of three
  unsigned table[CO];
#pragma unroll
  for (int b = 0; b < CO; b++) {
    table[b] = lut_s + 1024u * ((unsigned)(4 * (lane & 7) + 4 * CO - mis + b) % CO);
  }
  // the cast of unit j: x / scale alone by its steps, others through the tables, which lie
  // on multiples of 1024 bytes
  const bool scales = affine_scales<GRAY, U8>(p);
  const f32x2 r_hi = pack2(p.cast.r_hi[0], p.cast.r_hi[1]), r_lo = pack2(p.cast.r_lo[0], p.cast.r_lo[1]);
  auto cast = [&](uint32_t word, int j) {
    float f[4];
    if (scales) {
      const f32x2 minus_two23 = pack2(-8388608.0f, -8388608.0f);
      const f32x2 a = bytes_to_f32x2<0, 1>(word, minus_two23), b = bytes_to_f32x2<2, 3>(word, minus_two23);
      unpack2(fma2(a, r_hi, mul2(a, r_lo)), f[0], f[1]);
      unpack2(fma2(b, r_hi, mul2(b, r_lo)), f[2], f[3]);
    } else {
#pragma unroll
      for (int b = 0; b < 4; b++) {
        const uint32_t four = b == 0 ? word << 2 : word >> (8 * b - 2);
        f[b] = __uint_as_float(lds_u32<0>((four & 0x3fcu) | table[(b + 32 * j) % CO]));
      }
    }
    return make_float4(f[0], f[1], f[2], f[3]);
  };
  const int width = xb - xa;
  auto fetch = [&](AffinePiece& k, int x0) {
    const float dxf = __fsub_rn((float)(gx0 + dgx * x0), twh);
    const float m0x = __fmul_rn(m0, dxf), m3x = __fmul_rn(m3, dxf);
    int sx[4], sy[4];
    int least = 0;   // as whole numbers, negative floats are the less the closer to zero
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const float fx = __fadd_rn(__fadd_rn(m0x, m1y[i]), m2);
      const float fy = __fadd_rn(__fadd_rn(m3x, m4y[i]), m5);
      least = min(least, min(__float_as_int(fx), __float_as_int(fy)));
      sx[i] = __float2int_rz(__fadd_rz(fx, cx));
      sy[i] = __float2int_rz(__fadd_rz(fy, cy));
    }
    if (__any_sync(0xffffffffu, least < __float_as_int(-0x1p-26f))) {
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int2 at = affine_exact(
            __fadd_rn(__fadd_rn(m0x, m1y[i]), m2), __fadd_rn(__fadd_rn(m3x, m4y[i]), m5), wh, hh, pre_w, pre_h);
        sx[i] = at.x;
        sy[i] = at.y;
      }
    }
    // a pixel's C bytes, from the one or two aligned words that hold them
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const bool inside = (unsigned)sx[i] < (unsigned)pre_w && (unsigned)sy[i] < (unsigned)pre_h;
      const unsigned off = first + (unsigned)sy[i] * pitch + (unsigned)(sx[i] * dir);
      const uint32_t* const w = reinterpret_cast<const uint32_t*>(words + (off & ~3u));
      k.shift[i] = 8u * off;
      k.w0[i] = inside ? __ldg(w) : 0u;
      const bool more = C == 1 ? false : C == 2 ? (off & 3u) == 3u : C == 3 ? (off & 2u) != 0 : (off & 3u) != 0;
      k.w1[i] = inside && more ? __ldg(w + 1) : 0u;
    }
  };
  auto finish = [&](const AffinePiece& k, int x0) {
    const int n = min(32, width - x0);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t v = __funnelshift_r(k.w0[i], k.w1[i], k.shift[i]);
      if (GRAY) {
        sts_u8(to[i], gray_mix(p, v & 0xffu, (v >> 8) & 0xffu, (v >> 16) & 0xffu));
      } else {
#pragma unroll
        for (int ch = 0; ch < CO; ch++) {
          sts_u8(to[i] + (unsigned)ch, v >> (8 * ch));
        }
      }
    }
    __syncwarp();
    uint8_t* const d0 = seg + (ptrdiff_t)(x0 * CO - mis) * kSize + 4 * (lane & 7) * kSize;
    if (x0 > 0 && n == 32 && rows == 4 && x0 + 32 < width) {
      // inside a row every unit is whole: the one that the piece before began with has its first bytes from there
#pragma unroll
      for (int j = 0; j < CO; j++) {
        const uint32_t word = lds_u32<0>(from + 32u * j);
        if (U8) {
          reinterpret_cast<uint32_t*>(d0)[8 * j] = word;
        } else {
          reinterpret_cast<float4*>(d0)[8 * j] = cast(word, j);
        }
      }
    } else {
      // elements of the row that are in the patch and not stored yet: [begin, end); what the next piece completes is its
      const int begin = x0 > 0 ? 0 : mis;
      const int end = yo >= rows ? 0 : x0 + 32 < width ? 32 * CO : mis + n * CO;
#pragma unroll
      for (int j = 0; j < CO + 1; j++) {
        const int e = 4 * (8 * j + (lane & 7));
        if (e < end) {
          const uint32_t word = lds_u32<0>(from + 32u * j);
          const bool whole = e >= begin && e + 4 <= end;
          if (U8) {
            uint8_t* const d = d0 + 32 * j;
            if (whole) {
              *reinterpret_cast<uint32_t*>(d) = word;
            } else {
#pragma unroll
              for (int b = 0; b < 4; b++) {
                if (e + b >= begin && e + b < end) {
                  d[b] = (uint8_t)(word >> (8 * b));
                }
              }
            }
          } else {
            float* const d = reinterpret_cast<float*>(d0) + 32 * j;
            const float4 v = cast(word, j);
            if (whole) {
              *reinterpret_cast<float4*>(d) = v;
            } else {
              const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
              for (int b = 0; b < 4; b++) {
                if (e + b >= begin && e + b < end) {
                  d[b] = f[b];
                }
              }
            }
          }
        }
      }
    }
    // the bytes behind the last whole unit, to the front of the row
    const uint32_t rest = lds_u32<0>(patch + (unsigned)yo * kRow + 32u * CO);
    __syncwarp();
    if ((lane & 7) == 0) {
      *sp<uint32_t>(patch + (unsigned)yo * kRow) = rest;
    }
    __syncwarp();
  };
  AffinePiece even, odd;
  fetch(even, 0);
#pragma unroll 1
  for (int x0 = 0; x0 < width; x0 += 64) {
    const bool more = x0 + 32 < width;
    if (more) {
      fetch(odd, x0 + 32);
    }
    finish(even, x0);
    if (x0 + 64 < width) {
      fetch(even, x0 + 64);
    }
    if (more) {
      finish(odd, x0 + 32);
    }
  }
}

// One CTA: rows [y0, y0 + kTileH) of one slot, `columns` columns.
template <int C, bool GRAY, bool U8, int K>
__global__ void __launch_bounds__(kAffineThreads, kAffineCtas)
    affine_kernel(
        const __grid_constant__ LaunchParams p, int columns, int bands_x, const __grid_constant__ Records<K> records) {
  constexpr int CO = GRAY ? 1 : C;
  __shared__ __align__(1024) float lut_s[U8 ? 1 : CO * 256];
  __shared__ __align__(16) unsigned char patch[kAffineThreads / 32][640];
  unsigned t = blockIdx.x;
  const int tb = (int)(t % bands_x);
  t /= bands_x;
  const int y0 = (int)(t % p.tiles_y) * kTileH;
  const DevSample* const sample = records.of(p, t / p.tiles_y);
  // (a record of the table is copied whole, in one wait: 200 images of 512x512 146 us, 153 field by
  // field; one of the parameters is read as constants: 128 images 92.5 us, 97 copied)
  typename std::conditional<K == 0, const DevSample, const DevSample&>::type s = *sample;
  if (s.mode != kModeAffine) {
    return;   // the other kernels'
  }
  const int slot_h = s.slot_h, slot_w = s.slot_w, post_h = s.post_h, post_w = s.post_w;
  const int x0 = tb * columns;
  if (y0 >= slot_h || x0 >= slot_w) {
    return;
  }
  const int y1 = min(y0 + kTileH, slot_h), x1 = min(x0 + columns, slot_w);
  const int vy1 = min(y1, post_h), vx1 = min(x1, post_w);
  if (y0 < vy1 && x0 < vx1) {
    if (affine_rows_take<C>(s)) {
      if (!U8 && !affine_scales<GRAY, U8>(p)) {
        for (int i = threadIdx.x; i < CO * 64; i += kAffineThreads) {
          reinterpret_cast<float4*>(lut_s)[i] = __ldg(reinterpret_cast<const float4*>(p.lut) + i);
        }
        __syncthreads();
      }
      const int warp = threadIdx.x >> 5, ya = y0 + kAffineRows * warp;
      if (ya < vy1) {
        affine_rows<C, GRAY, U8>(
            s, p, smem_addr(lut_s), smem_addr(patch[warp]), ya, min(kAffineRows, vy1 - ya), x0, vx1);
      }
    } else {
      affine_pixels<C, GRAY, U8>(sample, p, y0, vy1, x0, vx1);
    }
  }
  // padding: right of the post window, and below it unless that is filled apart
  const int below = max(y0, min(y1, post_h)), right = max(x0, min(x1, post_w));
  auto pad = [&](int ya, int yb, int xa, int xb) {
    if (ya >= yb || xa >= xb) {
      return;
    }
    if (U8) {
      fill_rect_u8<CO>(reinterpret_cast<uint8_t*>(s.dst), slot_w, ya, yb, xa, xb, p.pad_px);
    } else {
      float padf[4];
#pragma unroll
      for (int c = 0; c < 4; c++) {
        padf[c] = c < CO ? __ldg(p.lut + c * 256 + p.pad_px) : 0.0f;
      }
      fill_rect_f32<CO>(reinterpret_cast<float*>(s.dst), slot_w, ya, yb, xa, xb, padf);
    }
  };
  pad(y0, below, right, x1);
  if (!p.pad_apart) {
    pad(below, y1, x0, x1);
  }
}

template <int C, bool GRAY, bool U8, int K>
void launch_one(
    const LaunchParams& p, unsigned blocks, int columns, int bands_x, const Records<K>& records, cudaStream_t stream) {
  affine_kernel<C, GRAY, U8, K><<<blocks, kAffineThreads, 0, stream>>>(p, columns, bands_x, records);
}

template <int C, bool GRAY, bool U8>
cudaError_t launch(const LaunchParams& p, unsigned blocks, int columns, int bands_x, cudaStream_t stream) {
  return with_records(p, [&](const auto& records) {
    launch_one<C, GRAY, U8>(p, blocks, columns, bands_x, records, stream);
    return cudaGetLastError();
  });
}

template <bool U8>
cudaError_t launch_type(const LaunchParams& p, unsigned blocks, int columns, int bands_x, cudaStream_t stream) {
  if (p.gray) {
    return launch<3, true, U8>(p, blocks, columns, bands_x, stream);
  }
  switch (p.c_in) {
    case 1:
      return launch<1, false, U8>(p, blocks, columns, bands_x, stream);
    case 2:
      return launch<2, false, U8>(p, blocks, columns, bands_x, stream);
    case 3:
      return launch<3, false, U8>(p, blocks, columns, bands_x, stream);
    default:
      return launch<4, false, U8>(p, blocks, columns, bands_x, stream);
  }
}

} // namespace

cudaError_t launch_affine(const LaunchParams& p, cudaStream_t stream) {
  // Whole rows to a warp, so that what it works out ahead of them serves many pixels, as long
  // as that makes half a round of CTAs; else as few pieces of 32 pixels as make it.  4 images
  // of 710x710x3 to 455x455: 13.6 us so, 14.2 with a round, 14.7 with two, 15.7 with a quarter;
  // 64 of 333x333x1 to 301x301, bytes: 17.6, 17.5, 19.0, 18.0.
  const int slot_w = p.tiles_x * kTileW;
  const long long bands = (long long)p.n * p.tiles_y;
  const long long want = 148 * kAffineCtas / 2;
  const int pieces = (slot_w + 31) / 32;
  const int splits = (int)std::max<long long>(1, std::min<long long>(pieces, (want + bands - 1) / bands));
  const int columns = (pieces + splits - 1) / splits * 32;
  const int bands_x = (slot_w + columns - 1) / columns;
  const unsigned long long blocks = (unsigned long long)bands * bands_x;
  if (blocks == 0) {
    return cudaSuccess;
  }
  if (blocks > 0x7fffffffULL) {
    return cudaErrorInvalidConfiguration;
  }
  return p.out_f32 ? launch_type<false>(p, (unsigned)blocks, columns, bands_x, stream)
                   : launch_type<true>(p, (unsigned)blocks, columns, bands_x, stream);
}

} // namespace mlxd
