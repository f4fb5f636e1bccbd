// Device helpers shared by the kernels of the library.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "fused_batch.h"

namespace mlxd {

__device__ __forceinline__ int clampi(int v, int lo, int hi) {
  return v < lo ? lo : (v > hi ? hi : v);
}

// Geometry of one axis of a triangle-filter resize, n source -> m output
// samples.  Every step is one correctly rounded float32 operation in a fixed
// order (no contraction), so host and device agree bit for bit:
//   ratio = n / m, u(o) = (o + 0.5) * ratio - 0.5, radius = max(1, ratio),
//   taps i = ceil(u - radius) .. floor(u + radius),
//   k_i = max(0, 1 - |i - u| * min(1, m / n)), w_i = k_i / sum(k).
struct Axis {
  float ratio, fs, radius;
  bool identity;
};

__device__ __forceinline__ Axis make_axis(int n, int m) {
  Axis a;
  a.identity = n == m;
  a.ratio = __fdiv_rn((float)n, (float)m);
  const float scale = __fdiv_rn((float)m, (float)n);
  a.fs = scale < 1.0f ? scale : 1.0f;
  a.radius = a.ratio > 1.0f ? a.ratio : 1.0f;
  return a;
}

__device__ __forceinline__ float axis_center(const Axis& a, int o) {
  return __fsub_rn(__fmul_rn(__fadd_rn((float)o, 0.5f), a.ratio), 0.5f);
}

// Un-clamped first and last tap of output sample o.
__device__ __forceinline__ void axis_range(const Axis& a, int o, int& lo, int& hi) {
  if (a.identity) {
    lo = hi = o;
    return;
  }
  const float u = axis_center(a, o);
  lo = (int)ceilf(__fsub_rn(u, a.radius));
  hi = (int)floorf(__fadd_rn(u, a.radius));
}

// Un-normalised tent value of source sample i for the output centred at u.
__device__ __forceinline__ float axis_tent(const Axis& a, float u, int i) {
  const float d = fabsf(__fsub_rn((float)i, u));
  const float v = __fsub_rn(1.0f, __fmul_rn(d, a.fs));
  return v > 0.0f ? v : 0.0f;
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Typed view of a shared-space address.
template <typename T>
__device__ __forceinline__ T* sp(unsigned a) {
  return reinterpret_cast<T*>(__cvta_shared_to_generic(a));
}

// Two float lanes in one 64-bit register, the operand form of the packed
// instructions; keeping values packed avoids repacking moves around them.
typedef unsigned long long f32x2;

// d = a * b + d on both lanes (each lane is an IEEE fused multiply-add,
// identical to fmaf).
__device__ __forceinline__ void ffma2(f32x2& d, f32x2 a, f32x2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}

__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}

// d = a * b + c on both lanes.
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// Bytes B0 and B1 of a word as two packed floats, exactly: each byte is placed
// in the mantissa of 2^23 and 2^23 is subtracted (one packed add for both).
template <int B0, int B1>
__device__ __forceinline__ f32x2 bytes_to_f32x2(uint32_t word, f32x2 minus_two23) {
  const float x0 = __uint_as_float(__byte_perm(word, 0x4B000000u, 0x7540u + B0));
  const float x1 = __uint_as_float(__byte_perm(word, 0x4B000000u, 0x7540u + B1));
  f32x2 r = pack2(x0, x1);
  asm("add.rn.f32x2 %0, %0, %1;" : "+l"(r) : "l"(minus_two23));
  return r;
}

// (int)(acc + 0.5) clamped to [0, 255]: the float-to-uint8 conversion truncates
// toward zero and saturates at both ends, which is that clamp.
__device__ __forceinline__ unsigned quantise_sat(float acc) {
  unsigned q;
  asm("cvt.rzi.u8.f32 %0, %1;" : "=r"(q) : "f"(__fadd_rn(acc, 0.5f)));
  return q;
}

// Shared-memory loads by 32-bit shared-space address plus a constant offset.
// Spelling the inner loops with these keeps their address arithmetic to the
// pointer increments written out in the loops.
template <int OFF>
__device__ __forceinline__ uint32_t lds_u32(unsigned a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(v) : "r"(a), "n"(OFF));
  return v;
}

__device__ __forceinline__ void sts_u8(unsigned a, uint32_t v) {
  asm volatile("st.shared.u8 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

template <int OFF>
__device__ __forceinline__ void lds_v2u32(unsigned a, uint32_t& x, uint32_t& y) {
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2+%3];" : "=r"(x), "=r"(y) : "r"(a), "n"(OFF));
}

template <int OFF>
__device__ __forceinline__ f32x2 lds_u64(unsigned a) {
  f32x2 v;
  asm volatile("ld.shared.u64 %0, [%1+%2];" : "=l"(v) : "r"(a), "n"(OFF));
  return v;
}

template <int OFF>
__device__ __forceinline__ void lds_v2u64(unsigned a, f32x2& x, f32x2& y) {
  asm volatile("ld.shared.v2.u64 {%0, %1}, [%2+%3];" : "=l"(x), "=l"(y) : "r"(a), "n"(OFF));
}

// Channel reduction of one quantised pixel: 16.16 fixed point, truncating
// division, clamped (core::image::channel_reduction,
// mlx/data/core/image/ImageTransform.cpp:159-180).
__device__ __forceinline__ unsigned gray_mix(const LaunchParams& p, unsigned r, unsigned g, unsigned b) {
  int v = ((int)r * p.gray_m[0] + (int)g * p.gray_m[1] + (int)b * p.gray_m[2] + p.gray_bias) / 65536;
  v = v <= 255 ? v : 255;
  v = v >= 0 ? v : 0;
  return (unsigned)v;
}

template <int CO>
__device__ __forceinline__ float pad_pick(const float (&padf)[4], int m) {
  if (CO == 1) {
    return padf[0];
  }
  float v = padf[0];
  v = m == 1 ? padf[1] : v;
  v = m == 2 ? padf[2] : v;
  if (CO > 3) {
    v = m == 3 ? padf[3] : v;
  }
  return v;
}

// Pad value (already cast) into the rectangle [ya, yb) x [xa, xb) of a slot
// with CO channels, 16-byte stores wherever the row segment allows.
//
// When the row pitch is a multiple of 16 bytes every row of the rectangle
// starts at the same offset within a 16-byte unit, so a thread works out its
// column position and its four values once and walks down the rows with
// nothing but stores; the CTA's threads are dealt over (column position, row
// phase) so that narrow rectangles still use all of them.
template <int CO>
__device__ __forceinline__ void fill_rect_f32(
    float* base, int slot_w, int ya, int yb, int xa, int xb, const float (&padf)[4]) {
  if (ya >= yb || xa >= xb) {
    return;
  }
  const int n_threads = (int)blockDim.x;
  const int L = (xb - xa) * CO;
  const int ny = yb - ya;
  const size_t row_floats = (size_t)slot_w * CO;
  float* row0 = base + ((size_t)ya * slot_w + xa) * CO;
  if ((row_floats & 3) == 0) {
    const int mis = (int)((reinterpret_cast<uintptr_t>(row0) >> 2) & 3);
    int head = (4 - mis) & 3;
    head = head > L ? L : head;
    const int nvec = (L - head) >> 2;
    if (nvec > 0) {
      const int lanes_q = nvec >= n_threads ? n_threads : nvec;
      const int phases = n_threads / lanes_q;
      const int r0 = (int)threadIdx.x / lanes_q;
      if (r0 < phases) {
        for (int q = (int)threadIdx.x - r0 * lanes_q; q < nvec; q += lanes_q) {
          const int j = head + 4 * q;
          const int m = j % CO;
          const float4 v = make_float4(
              pad_pick<CO>(padf, m), pad_pick<CO>(padf, (m + 1) % CO), pad_pick<CO>(padf, (m + 2) % CO),
              pad_pick<CO>(padf, (m + 3) % CO));
          float* p = row0 + (size_t)r0 * row_floats + j;
          for (int ry = r0; ry < ny; ry += phases, p += (size_t)phases * row_floats) {
            *reinterpret_cast<float4*>(p) = v;
          }
        }
      }
    }
    // the few floats before the first and after the last aligned unit of each row
    const int tail = head + 4 * nvec;
    const int loose = head + (L - tail);
    for (int i = threadIdx.x; i < ny * loose; i += n_threads) {
      const int ry = i / loose;
      const int k = i - ry * loose;
      const int j = k < head ? k : tail + (k - head);
      row0[(size_t)ry * row_floats + j] = pad_pick<CO>(padf, j % CO);
    }
    return;
  }
  const int Q = ((L + 3) >> 2) + 2;
  for (int i = threadIdx.x; i < ny * Q; i += n_threads) {
    const int ry = i / Q;
    const int q = i - ry * Q;
    float* rowp = row0 + (size_t)ry * row_floats;
    const int mis = (int)((reinterpret_cast<uintptr_t>(rowp) >> 2) & 3);
    int head = (4 - mis) & 3;
    head = head > L ? L : head;
    const int nvec = (L - head) >> 2;
    if (q == 0) {
      for (int j = 0; j < head; j++) {
        rowp[j] = pad_pick<CO>(padf, j % CO);
      }
    } else if (q <= nvec) {
      const int j = head + 4 * (q - 1);
      const int m = j % CO;
      *reinterpret_cast<float4*>(rowp + j) = make_float4(
          pad_pick<CO>(padf, m), pad_pick<CO>(padf, (m + 1) % CO), pad_pick<CO>(padf, (m + 2) % CO),
          pad_pick<CO>(padf, (m + 3) % CO));
    } else if (q == nvec + 1) {
      for (int j = head + 4 * nvec; j < L; j++) {
        rowp[j] = pad_pick<CO>(padf, j % CO);
      }
    }
  }
}

// The same for a uint8 slot: every byte of the padding is the pad pixel, so the
// aligned middle of every row goes out as 16-byte stores of one pattern.
template <int CO>
__device__ __forceinline__ void fill_rect_u8(
    uint8_t* base, int slot_w, int ya, int yb, int xa, int xb, int pad_px) {
  if (ya >= yb || xa >= xb) {
    return;
  }
  const int L = (xb - xa) * CO;
  const int ny = yb - ya;
  const size_t row_bytes = (size_t)slot_w * CO;
  const unsigned w = (unsigned)(pad_px & 0xff) * 0x01010101u;
  const uint4 v = make_uint4(w, w, w, w);
  for (int ry = (int)threadIdx.x >> 5; ry < ny; ry += (int)blockDim.x >> 5) {     // a warp per row
    uint8_t* rowp = base + (size_t)(ya + ry) * row_bytes + (size_t)xa * CO;
    const int mis = (int)(reinterpret_cast<uintptr_t>(rowp) & 15);
    int head = (16 - mis) & 15;
    head = head > L ? L : head;
    const int nvec = (L - head) >> 4;
    const int lane = (int)threadIdx.x & 31;
    for (int q = lane; q < nvec; q += 32) {
      *reinterpret_cast<uint4*>(rowp + head + 16 * q) = v;
    }
    const int tail = head + 16 * nvec;
    for (int k = lane; k < head + (L - tail); k += 32) {
      rowp[k < head ? k : tail + (k - head)] = (uint8_t)pad_px;
    }
  }
}

// The padding below a sample of a ragged batch.  Rows of a slot are contiguous,
// so everything below the sample's post window down to the end of the slot is one
// contiguous run of floats: written here as a linear fill (16-byte stores,
// consecutive threads on consecutive addresses, kPadChunks CTAs per sample), which
// runs at memory speed (7.7 TB/s; the 16-row strips of the band kernel 4.5).  The
// strips to the right of the post window are the band kernel's, or cells of the
// resize kernel.  THREADS is a CTA's thread count: read from blockDim, it made the
// fill kernel spill (64 images of 64x64 in slots of 4000x100: 99.3 us a pass, 96.5 so).
template <int CO, int THREADS, int K>
__device__ __forceinline__ void pad_below(const LaunchParams& p, const Records<K>& records, unsigned block) {
  const int n = (int)(block / kPadChunks);
  const int chunk = (int)(block % kPadChunks);
  if (n >= p.n) {
    return;
  }
  const DevSample* s = records.of(p, (unsigned)n);
  const int slot_h = s->slot_h, slot_w = s->slot_w;
  const int post_h = s->post_h < slot_h ? s->post_h : slot_h;
  const int first_row = post_h;
  if (first_row >= slot_h) {
    return;
  }
  float padf[4];
#pragma unroll
  for (int c = 0; c < 4; c++) {
    padf[c] = c < CO ? __ldg(p.lut + c * 256 + p.pad_px) : 0.0f;
  }
  const size_t row_floats = (size_t)slot_w * CO;
  float* run = reinterpret_cast<float*>(s->dst) + (size_t)first_row * row_floats;   // starts on a pixel: channel 0
  const size_t len = (size_t)(slot_h - first_row) * row_floats;
  const size_t mis = (reinterpret_cast<uintptr_t>(run) >> 2) & 3;
  size_t head = (4 - mis) & 3;
  head = head > len ? len : head;
  const size_t nvec = (len - head) >> 2;
  // this CTA's share of the aligned units
  const size_t q0 = nvec * (size_t)chunk / kPadChunks;
  const size_t q1 = nvec * (size_t)(chunk + 1) / kPadChunks;
  for (size_t q = q0 + threadIdx.x; q < q1; q += THREADS) {
    const size_t j = head + 4 * q;
    const int m = (int)(j % CO);
    *reinterpret_cast<float4*>(run + j) = make_float4(
        pad_pick<CO>(padf, m), pad_pick<CO>(padf, (m + 1) % CO), pad_pick<CO>(padf, (m + 2) % CO),
        pad_pick<CO>(padf, (m + 3) % CO));
  }
  if (chunk == 0) {
    // the floats before the first and after the last aligned unit
    const size_t tail = head + 4 * nvec;
    for (size_t k = threadIdx.x; k < head + (len - tail); k += THREADS) {
      const size_t j = k < head ? k : tail + (k - head);
      run[j] = pad_pick<CO>(padf, (int)(j % CO));
    }
  }
}

// The same for a uint8 batch: a linear fill of bytes.
template <int THREADS, int K>
__device__ __forceinline__ void pad_below_u8(const LaunchParams& p, const Records<K>& records, unsigned block) {
  const int n = (int)(block / kPadChunks);
  const int chunk = (int)(block % kPadChunks);
  if (n >= p.n) {
    return;
  }
  const DevSample* s = records.of(p, (unsigned)n);
  const int slot_h = s->slot_h, slot_w = s->slot_w;
  const int post_h = s->post_h < slot_h ? s->post_h : slot_h;
  const int first_row = post_h;
  if (first_row >= slot_h) {
    return;
  }
  const size_t row_bytes = (size_t)slot_w * p.c_out;
  uint8_t* run = reinterpret_cast<uint8_t*>(s->dst) + (size_t)first_row * row_bytes;
  const size_t len = (size_t)(slot_h - first_row) * row_bytes;
  const size_t mis = reinterpret_cast<uintptr_t>(run) & 15;
  size_t head = (16 - mis) & 15;
  head = head > len ? len : head;
  const size_t nvec = (len - head) >> 4;
  const unsigned w = (unsigned)(p.pad_px & 0xff) * 0x01010101u;
  const uint4 v = make_uint4(w, w, w, w);
  const size_t q0 = nvec * (size_t)chunk / kPadChunks;
  const size_t q1 = nvec * (size_t)(chunk + 1) / kPadChunks;
  for (size_t q = q0 + threadIdx.x; q < q1; q += THREADS) {
    *reinterpret_cast<uint4*>(run + head + 16 * q) = v;
  }
  if (chunk == 0) {
    const size_t tail = head + 16 * nvec;
    for (size_t k = threadIdx.x; k < head + (len - tail); k += THREADS) {
      run[k < head ? k : tail + (k - head)] = (uint8_t)p.pad_px;
    }
  }
}

// Block `block` of n * kPadChunks.
template <int THREADS, int K>
__device__ __forceinline__ void pad_below_any(const LaunchParams& p, const Records<K>& records, unsigned block) {
  if (!p.out_f32) {
    pad_below_u8<THREADS>(p, records, block);
  } else if (p.c_out == 3) {
    pad_below<3, THREADS>(p, records, block);
  } else if (p.c_out == 1) {
    pad_below<1, THREADS>(p, records, block);
  } else if (p.c_out == 2) {
    pad_below<2, THREADS>(p, records, block);
  } else {
    pad_below<4, THREADS>(p, records, block);
  }
}

} // namespace mlxd
