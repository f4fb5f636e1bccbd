// What the two resize kernels share: packed float arithmetic, quantisation and
// the way of four finished rows into the batch tensor.
#pragma once

#include "fused_batch.h"
#include "kernel_common.cuh"

namespace mlxd {

// (int)(acc + 0.5) of both lanes as the low mantissa bits of 2^23 + that
// integer.  acc is never negative and at most 255 (1 + 1e-4) here - pixels
// times weights that sum to 1 within the rounding of a few hundred terms - so
// acc + 0.5 < 256 and the clamp to [0, 255] of the definition never acts.
__device__ __forceinline__ void quantise2(f32x2 acc, unsigned& q0, unsigned& q1) {
  const f32x2 half = pack2(0.5f, 0.5f), two23 = pack2(8388608.0f, 8388608.0f);
  f32x2 t;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(t) : "l"(acc), "l"(half));
  asm("add.rz.f32x2 %0, %1, %2;" : "=l"(t) : "l"(t), "l"(two23));
  float a, b;
  unpack2(t, a, b);
  q0 = __float_as_uint(a);
  q1 = __float_as_uint(b);
}

constexpr unsigned kTwo23Bits = 0x4B000000u;

__device__ __forceinline__ void sts_v4(unsigned a, float x, float y, float z, float w) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}

template <int OFF>
__device__ __forceinline__ void lds_v4u32(unsigned a, uint32_t& x, uint32_t& y, uint32_t& z, uint32_t& w) {
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4+%5];" : "=r"(x), "=r"(y), "=r"(z), "=r"(w) : "r"(a), "n"(OFF));
}

__device__ __forceinline__ f32x2 both(const float (&pair)[2]) {
  return pack2(pair[0], pair[1]);
}

#pragma nv_diagnostic push
#pragma nv_diag_suppress 128   // (where the way of casting is known, the look-ups below are never reached)

// One output column of four rows: filter sums acc[2 * c + h] (rows 2h and 2h + 1
// of channel c) quantised, reduced to grey, cast and stored.  `at` is the first
// row's place in the batch tensor in elements; the first `rows` rows are stored.
//
// The cast is computed where its steps are known (CastSteps), else looked up in a table in
// shared memory: 32 values meet three to four times in its banks, so a look-up takes the
// shared-memory pipe, of which a shrink has least to spare, as long as three other accesses.
// 512 images of 1080x1920x3 to 512x512: 1105 us, 1146 with the table; 256 random crops to
// 224x224 113 and 115; one image 9.6 and 10.0; in resize_walk.cu 64 of 1400 px to 300x300 216 and 223.  CAST: the way is known at compile time (a
// CastMode), or -1.
template <int C, bool GRAY, bool U8, int CAST = -1>
__device__ __forceinline__ void store_column(
    const LaunchParams& p, unsigned lut, const f32x2 (&acc)[2 * C], int rows, void* dst, size_t at, size_t row_stride,
    bool vec_ok) {
  constexpr int CO = GRAY ? 1 : C;
  const int mode = CAST < 0 ? p.cast.mode : CAST;
  if (!U8 && !GRAY && mode != kCastTable) {
    const f32x2 half = pack2(0.5f, 0.5f), two23 = pack2(8388608.0f, 8388608.0f), minus_two23 = pack2(-8388608.0f, -8388608.0f);
    f32x2 v[2 * C];
#pragma unroll
    for (int i = 0; i < 2 * C; i++) {
      f32x2 t = add2(acc[i], half);   // quantise2()
      asm("add.rz.f32x2 %0, %1, %2;" : "=l"(t) : "l"(t), "l"(two23));
      t = add2(t, minus_two23);
      v[i] = fma2(t, both(p.cast.r_hi), mul2(t, both(p.cast.r_lo)));
    }
    if (mode == kCastNormalise) {
#pragma unroll
      for (int i = 0; i < 2 * C; i++) {
        const f32x2 t = add2(v[i], both(p.cast.neg_mean[i / 2]));
        v[i] = fma2(t, both(p.cast.s_hi[i / 2]), mul2(t, both(p.cast.s_lo[i / 2])));
      }
    }
    float* d = reinterpret_cast<float*>(dst) + at;
#pragma unroll
    for (int r = 0; r < 4; r++, d += row_stride) {
      if (r < rows) {
        float o[C];
#pragma unroll
        for (int ch = 0; ch < C; ch++) {
          float lo, hi;
          unpack2(v[2 * ch + r / 2], lo, hi);
          o[ch] = r & 1 ? hi : lo;
        }
        if (C == 4 && vec_ok) {
          *reinterpret_cast<float4*>(d) = make_float4(o[0], o[1 % C], o[2 % C], o[3 % C]);
        } else {
#pragma unroll
          for (int ch = 0; ch < C; ch++) {
            d[ch] = o[ch];
          }
        }
      }
    }
    return;
  }
  unsigned q[4][C];   // 2^23 bits + value
#pragma unroll
  for (int ch = 0; ch < C; ch++) {
    quantise2(acc[2 * ch], q[0][ch], q[1][ch]);
    quantise2(acc[2 * ch + 1], q[2][ch], q[3][ch]);
  }
#pragma unroll
  for (int r = 0; r < 4; r++) {
    if (r < rows) {   // (rows beyond the last hold anything: they must not index the cast table)
      if (U8) {
        uint8_t* d = reinterpret_cast<uint8_t*>(dst) + at + r * row_stride;
        if (GRAY) {
          d[0] = (uint8_t)gray_mix(p, q[r][0] & 0xffu, q[r][1 % C] & 0xffu, q[r][2 % C] & 0xffu);
        } else {
#pragma unroll
          for (int ch = 0; ch < C; ch++) {
            d[ch] = (uint8_t)q[r][ch];
          }
        }
      } else {
        float v[CO];
        if (GRAY) {
          v[0] = __uint_as_float(
              lds_u32<0>(lut + 4u * gray_mix(p, q[r][0] & 0xffu, q[r][1 % C] & 0xffu, q[r][2 % C] & 0xffu)));
        } else {
#pragma unroll
          for (int ch = 0; ch < C; ch++) {
            v[ch % CO] = __uint_as_float(lds_u32<0>((lut + 1024u * ch - 4u * kTwo23Bits) + 4u * q[r][ch]));
          }
        }
        float* d = reinterpret_cast<float*>(dst) + at + r * row_stride;
        if (CO == 4 && vec_ok) {
          *reinterpret_cast<float4*>(d) = make_float4(v[0], v[1 % CO], v[2 % CO], v[3 % CO]);
        } else {
#pragma unroll
          for (int ch = 0; ch < CO; ch++) {
            d[ch] = v[ch];
          }
        }
      }
    }
  }
}

#pragma nv_diagnostic pop

} // namespace mlxd
