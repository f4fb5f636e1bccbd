// Context, lanes, descriptor planning and the enqueue path of the C ABI.
#include "context.h"

#include <map>

#ifdef __SSE2__
#include <emmintrin.h>
#endif
#include <sched.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <thread>

namespace mlxd {

namespace {
thread_local std::string g_error;
}

const std::string& error_text() {
  return g_error;
}

void set_error(const std::string& msg) {
  g_error = msg;
}

int fail(int code, const std::string& msg) {
  g_error = msg;
  return code;
}

int fail_cuda(cudaError_t e, const char* what) {
  g_error = std::string(what) + ": " + cudaGetErrorString(e);
  return e == cudaErrorMemoryAllocation ? MLXD_ERR_NOMEM : MLXD_ERR_CUDA;
}

bool LutKey::operator<(const LutKey& o) const {
  return std::memcmp(this, &o, sizeof(LutKey)) < 0;
}

namespace {
struct PinnedBlock {
  size_t bytes;
  intptr_t device_delta;   // device-side address minus host address
};
std::mutex g_pinned_mu;
std::map<uintptr_t, PinnedBlock> g_pinned;
}  // namespace

void pinned_registry_add(void* host, size_t bytes, void* device_side) {
  std::lock_guard<std::mutex> g(g_pinned_mu);
  g_pinned[reinterpret_cast<uintptr_t>(host)] =
      PinnedBlock{bytes, static_cast<intptr_t>(reinterpret_cast<uintptr_t>(device_side) - reinterpret_cast<uintptr_t>(host))};
}

void pinned_registry_remove(void* host) {
  std::lock_guard<std::mutex> g(g_pinned_mu);
  g_pinned.erase(reinterpret_cast<uintptr_t>(host));
}

const uint8_t* pinned_registry_lookup(const void* host) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(host);
  std::lock_guard<std::mutex> g(g_pinned_mu);
  auto it = g_pinned.upper_bound(a);
  if (it == g_pinned.begin()) {
    return nullptr;
  }
  --it;
  if (a >= it->first + it->second.bytes) {
    return nullptr;
  }
  return reinterpret_cast<const uint8_t*>(a + it->second.device_delta);
}

int arena_reserve(mlxd_ctx* ctx, Arena& a, size_t bytes, bool pinned, cudaStream_t stream_to_drain) {
  if (bytes <= a.cap) {
    return MLXD_OK;
  }
  // Work already queued may still read the old block.
  if (stream_to_drain) {
    MLXD_CUDA(cudaStreamSynchronize(stream_to_drain));
  }
  size_t want = bytes + bytes / 4;
  want = (want + 4095) & ~(size_t)4095;
  void* p = nullptr;
  if (pinned) {
    MLXD_CUDA(cudaHostAlloc(&p, want, cudaHostAllocDefault));
    if (a.ptr) {
      cudaFreeHost(a.ptr);
    }
  } else {
    if (a.ptr) {
      cudaFree(a.ptr);
      ctx->reserved -= a.cap;
      a.ptr = nullptr;
      a.cap = 0;
    }
    MLXD_CUDA(cudaMalloc(&p, want));
    ctx->reserved += want;
  }
  a.ptr = p;
  a.cap = want;
  return MLXD_OK;
}

// "sample <i>: <what>" as the thread's error text.  Only failing calls come
// here, so a call that succeeds builds no string at all.
static int bad_sample(int i, const char* what) {
  return fail(MLXD_ERR_INVALID, "sample " + std::to_string(i) + ": " + what);
}

static int check_sample(const mlxd_sample_desc& d, int i, const mlxd_batch_desc* b, int slot_h, int slot_w) {
  if (!d.src) {
    return bad_sample(i, "null source");
  }
  if (d.src_h <= 0 || d.src_w <= 0) {
    return bad_sample(i, "image: cannot create image with 0 or negative dimension");
  }
  if (d.pre_w <= 0 || d.pre_h <= 0 || d.pre_x < 0 || d.pre_y < 0 ||
      (int64_t)d.pre_x + d.pre_w > d.src_w || (int64_t)d.pre_y + d.pre_h > d.src_h) {
    return bad_sample(i, "window before the geometric op leaves the source image");
  }
  if (d.geom < MLXD_GEOM_NONE || d.geom > MLXD_GEOM_AFFINE) {
    return bad_sample(i, "unknown geometric op");
  }
  if (d.geom_w <= 0 || d.geom_h <= 0) {
    return bad_sample(i, "image: cannot create image with 0 or negative dimension");
  }
  if (d.geom == MLXD_GEOM_NONE && (d.geom_w != d.pre_w || d.geom_h != d.pre_h)) {
    return bad_sample(i, "geom_w, geom_h must equal pre_w, pre_h without a geometric op");
  }
  if (d.post_w <= 0 || d.post_h <= 0 || d.post_x < 0 || d.post_y < 0 ||
      (int64_t)d.post_x + d.post_w > d.geom_w || (int64_t)d.post_y + d.post_h > d.geom_h) {
    return bad_sample(i, "window after the geometric op leaves its output");
  }
  if (d.post_w > slot_w || d.post_h > slot_h) {
    return bad_sample(i, "result is larger than its slot in the batch");
  }
  if ((int64_t)d.src_h * d.src_w * b->channels >= ((int64_t)1 << 40)) {
    return bad_sample(i, "source image too large");
  }
  return MLXD_OK;
}

int plan_one_sample(const mlxd_sample_desc& d, int i, const mlxd_batch_desc* b, const DevSample* before, DevSample& out) {
  {
    int rc = check_sample(d, i, b, b->slot_h, b->slot_w);
    if (rc != MLXD_OK) {
      return rc;
    }
    DevSample& s = out;
    std::memset(&s, 0, sizeof(s));
    s.src = d.src;
    s.src_h = d.src_h;
    s.src_w = d.src_w;
    s.pre_x = d.pre_x;
    s.pre_y = d.pre_y;
    s.pre_w = d.pre_w;
    s.pre_h = d.pre_h;
    s.pre_flip = d.pre_flip ? 1 : 0;
    s.geom_w = d.geom_w;
    s.geom_h = d.geom_h;
    s.post_x = d.post_x;
    s.post_y = d.post_y;
    s.post_w = d.post_w;
    s.post_h = d.post_h;
    s.post_flip = d.post_flip ? 1 : 0;
    s.slot_h = b->slot_h;
    s.slot_w = b->slot_w;
    std::memcpy(s.mx, d.mx, sizeof(s.mx));
    s.cap_x = 1;
    if (d.geom == MLXD_GEOM_RESIZE) {
      if (d.pre_w == d.geom_w && d.pre_h == d.geom_h) {
        s.mode = kModeCopy;  // identity on both axes
      } else {
        if (before && is_resize(*before) && s.pre_w == before->pre_w && s.pre_h == before->pre_h &&
            s.geom_w == before->geom_w && s.geom_h == before->geom_h && s.post_w == before->post_w &&
            s.src_w == before->src_w) {
          // like the sample before it, as in a batch of frames
          std::memcpy(s.mx, before->mx, sizeof(s.mx));
          s.cap_x = before->cap_x;
          s.walk_px = before->walk_px;
          s.mode = before->mode;
        } else {
          set_axes(s);
          s.mode = resize_mode(s, b->channels);
        }
      }
    } else if (d.geom == MLXD_GEOM_AFFINE) {
      s.mode = kModeAffine;
    } else {
      s.mode = kModeCopy;
    }
    if (s.mode == kModeCopy && s.pre_flip) {
      // Without a geometric op the two mirrors compose into one.
      s.pre_flip = 0;
      s.post_flip ^= 1;
      s.post_x = s.geom_w - s.post_x - s.post_w;
    }
  }
  return MLXD_OK;
}

int plan_into(const mlxd_sample_desc* samples, int n, const mlxd_batch_desc* b, DevSample* out, ResizePlan& plan) {
  bool resizes = false;
  for (int i = 0; i < n; i++) {
    const int rc = plan_one_sample(samples[i], i, b, i > 0 ? &out[i - 1] : nullptr, out[i]);
    if (rc != MLXD_OK) {
      return rc;
    }
    resizes |= is_resize(out[i]);
  }
  plan = ResizePlan{};
  if (resizes) {
    plan_resize(out, n, b->channels, plan);
  }
  return MLXD_OK;
}

int plan_samples(
    const mlxd_sample_desc* samples, int n, const mlxd_batch_desc* b, DevSample* out, ResizePlan& plan) {
  const int rc = plan_into(samples, n, b, out, plan);
  // Test hook (MLXD_TEST_SHORT_PLAN=1, read per launch): room for one step a walk.
  // Every resize CTA that has more finds that before it copies or filters anything,
  // sets the status word and returns, so the kernel's self-check and the way from it
  // to the caller's error code can be exercised without a fault or a hang.
  const char* hook = std::getenv("MLXD_TEST_SHORT_PLAN");
  if (rc == MLXD_OK && hook && hook[0] == '1') {
    plan.strip.steps = std::min(plan.strip.steps, 1);
    plan.wide.steps = std::min(plan.wide.steps, 1);
  }
  return rc;
}

// floor() and ceil() without a library call.
static int64_t floor_to(double x) {
  const int64_t t = (int64_t)x;
  return t - (x < (double)t);
}

static int64_t ceil_to(double x) {
  const int64_t t = (int64_t)x;
  return t + (x > (double)t);
}

// Source samples of an n_src -> n_dst axis that outputs [o_lo, o_hi) can read,
// widened by `margin` on both sides (none: the exact span, for statistics) and clipped
// to the axis.
static void axis_span(int64_t n_src, int64_t n_dst, int64_t o_lo, int64_t o_hi, int margin, int64_t& lo, int64_t& hi) {
  if (o_lo == 0 && o_hi == n_dst) {
    lo = 0;   // the first and the last output reach beyond the axis
    hi = n_src;
    return;
  }
  if (n_src == n_dst) {
    lo = o_lo;
    hi = o_hi;
  } else {
    const double ratio = (double)n_src / (double)n_dst;
    const double radius = ratio > 1.0 ? ratio : 1.0;
    const int around = margin > 0 ? margin + axis_slack((int32_t)n_src) : 0;
    lo = floor_to((o_lo + 0.5) * ratio - 0.5 - radius) - around;
    hi = ceil_to((o_hi - 0.5) * ratio - 0.5 + radius) + 1 + around;
  }
  lo = std::max<int64_t>(lo, 0);
  hi = std::min<int64_t>(hi, n_src);
}

void needed_region(const DevSample& s, int margin, int32_t& r0, int32_t& r1, int32_t& c0, int32_t& c1) {
  int64_t rlo = 0, rhi = s.pre_h, clo = 0, chi = s.pre_w;  // in pre-window coordinates
  if (s.mode == kModeCopy) {
    rlo = s.post_y;
    rhi = (int64_t)s.post_y + s.post_h;
    clo = s.post_x;
    chi = (int64_t)s.post_x + s.post_w;
  } else if (s.mode != kModeAffine) {   // the resizes
    axis_span(s.pre_h, s.geom_h, s.post_y, (int64_t)s.post_y + s.post_h, margin, rlo, rhi);
    axis_span(s.pre_w, s.geom_w, s.post_x, (int64_t)s.post_x + s.post_w, margin, clo, chi);
    if (s.pre_flip) {
      const int64_t a = s.pre_w - chi, b = s.pre_w - clo;
      clo = a;
      chi = b;
    }
  }
  r0 = (int32_t)(s.pre_y + rlo);
  r1 = (int32_t)(s.pre_y + rhi);
  c0 = (int32_t)(s.pre_x + clo);
  c1 = (int32_t)(s.pre_x + chi);
}

void compute_cast_table(const mlxd_batch_desc* b, int c_out, float* table) {
  // Every entry is the chain of float32 operations numpy performs:
  // float(v) / divisor, then - mean, then / std.
  for (int c = 0; c < c_out; c++) {
    for (int v = 0; v < 256; v++) {
      volatile float x = (float)v;
      volatile float q = x / b->divisor;
      if (b->normalise) {
        volatile float t = q - b->mean[c];
        q = t / b->std_[c];
      }
      table[(size_t)c * 256 + v] = q;
    }
  }
}

// A division of a float x by a float d, correctly rounded, is fma(x, hi, x * lo) with
// hi + lo = 1 / d to 48 bits, unless the quotient lies within 2^-48 of the middle between
// two floats: so every value is compared with the table's, and a cast with one that differs
// (or with infinities) keeps the table.  So does one with a NaN, of which arithmetic on the GPU
// keeps neither sign nor payload, and the channel reduction's: its values are whole numbers,
// which index the table as they are.
void cast_steps(const mlxd_batch_desc* b, int c_out, const float* table, CastSteps& steps) {
  std::memset(&steps, 0, sizeof(steps));
  if (b->gray) {
    return;
  }
  auto reciprocal = [](float d, float (&hi)[2], float (&lo)[2]) {
    const double r = 1.0 / (double)d;
    hi[0] = hi[1] = (float)r;
    lo[0] = lo[1] = (float)(r - (double)hi[0]);
  };
  reciprocal(b->divisor, steps.r_hi, steps.r_lo);
  for (int c = 0; c < c_out && b->normalise; c++) {
    steps.neg_mean[c][0] = steps.neg_mean[c][1] = -b->mean[c];
    reciprocal(b->std_[c], steps.s_hi[c], steps.s_lo[c]);
  }
  for (int c = 0; c < c_out; c++) {
    for (int v = 0; v < 256; v++) {
      const volatile float x = (float)v;
      const volatile float low = x * steps.r_lo[0];
      float y = std::fma((float)x, steps.r_hi[0], (float)low);
      if (b->normalise) {
        const volatile float t = y + steps.neg_mean[c][0];
        const volatile float t_low = t * steps.s_lo[c][0];
        y = std::fma((float)t, steps.s_hi[c][0], (float)t_low);
      }
      if (y != y || std::memcmp(&y, &table[(size_t)c * 256 + v], sizeof(y)) != 0) {
        return;
      }
    }
  }
  steps.mode = b->normalise ? kCastNormalise : kCastScale;
}

static LutKey cast_key(const mlxd_batch_desc* b, int c_out) {
  LutKey key;
  std::memset(&key, 0, sizeof(key));
  key.c_out = c_out;
  key.normalise = b->normalise ? 1 : 0;
  key.gray = b->gray ? 1 : 0;
  std::memcpy(&key.divisor_bits, &b->divisor, 4);
  if (key.normalise) {
    std::memcpy(key.mean_bits, b->mean, 4 * c_out);
    std::memcpy(key.std_bits, b->std_, 4 * c_out);
  }
  return key;
}

// Fixed storage: mlxd_fused_batch_noalloc comes here.  The host's part of such a call, one sample
// cast and normalised in three channels: 6.0 us where the cast is compared each time, 2.0 so (1.6 of
// them its table).
void kept_cast_steps(const mlxd_batch_desc* b, int c_out, const float* table, CastSteps& steps) {
  constexpr int kKept = 8;
  static LutKey keys[kKept];   // (c_out of 0: not in use yet)
  static CastSteps kept[kKept];
  static int next = 0;
  static std::mutex mu;
  const LutKey key = cast_key(b, c_out);
  std::lock_guard<std::mutex> g(mu);
  for (int i = 0; i < kKept; i++) {
    if (std::memcmp(&keys[i], &key, sizeof(key)) == 0) {
      steps = kept[i];
      return;
    }
  }
  cast_steps(b, c_out, table, steps);
  keys[next] = key;
  kept[next] = steps;
  next = (next + 1) % kKept;
}

LutUse::LutUse(mlxd_ctx* ctx) {
  bool full;
  {
    std::lock_guard<std::mutex> g(ctx->lut_mu);
    full = ctx->luts.size() >= kMaxCastTables;
  }
  if (full) {
    std::unique_lock<std::shared_mutex> alone(ctx->lut_users);
    std::lock_guard<std::mutex> g(ctx->lut_mu);
    if (ctx->luts.size() >= kMaxCastTables) {
      DeviceGuard on_device(ctx->device);
      cudaDeviceSynchronize();
      for (auto& kv : ctx->luts) {
        cudaFree(kv.second.values);
      }
      ctx->luts.clear();
    }
  }
  hold_ = std::shared_lock<std::shared_mutex>(ctx->lut_users);
}

int get_lut(mlxd_ctx* ctx, const mlxd_batch_desc* b, int c_out, CastTable& out) {
  const LutKey key = cast_key(b, c_out);
  std::lock_guard<std::mutex> g(ctx->lut_mu);
  auto it = ctx->luts.find(key);
  if (it != ctx->luts.end()) {
    out = it->second;
    return MLXD_OK;
  }
  std::vector<float> table((size_t)c_out * 256);
  compute_cast_table(b, c_out, table.data());
  float* d = nullptr;
  MLXD_CUDA(cudaMalloc(&d, table.size() * sizeof(float)));
  cudaError_t e = cudaMemcpy(d, table.data(), table.size() * sizeof(float), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    cudaFree(d);
    return fail_cuda(e, "cudaMemcpy(cast table)");
  }
  out.values = d;
  cast_steps(b, c_out, table.data(), out.steps);
  ctx->luts[key] = out;
  return MLXD_OK;
}

int describe_launch(const mlxd_batch_desc* b, int n, LaunchParams& p) {
  if (b->channels < 1 || b->channels > 4) {
    return fail(MLXD_ERR_INVALID, "image: channels must be 0 < c <= 4");
  }
  if (b->gray && b->channels != 3) {
    return fail(MLXD_ERR_INVALID, "image::channelReduction: expected a 3 channel uint8 array");
  }
  if (b->slot_h <= 0 || b->slot_w <= 0) {
    return fail(MLXD_ERR_INVALID, "batch slot must have positive height and width");
  }
  if (b->out_dtype != MLXD_U8 && b->out_dtype != MLXD_F32) {
    return fail(MLXD_ERR_INVALID, "unknown output dtype");
  }
  std::memset(&p, 0, sizeof(p));
  p.n = n;
  p.tiles_y = (b->slot_h + kTileH - 1) / kTileH;
  p.tiles_x = (b->slot_w + kTileW - 1) / kTileW;
  p.c_in = b->channels;
  p.c_out = b->gray ? 1 : b->channels;
  p.gray = b->gray ? 1 : 0;
  p.gray_m[0] = b->gray_m[0];
  p.gray_m[1] = b->gray_m[1];
  p.gray_m[2] = b->gray_m[2];
  p.gray_bias = b->gray_bias;
  p.out_f32 = b->out_dtype == MLXD_F32;
  p.pad_px = (int32_t)(uint8_t)(int32_t)b->pad_value;
  if (p.out_f32 && !(b->divisor != 0.0f)) {
    return fail(MLXD_ERR_INVALID, "cast divisor must be non-zero");
  }
  return MLXD_OK;
}

int prepare_launch(mlxd_ctx* ctx, const mlxd_batch_desc* b, int n, LaunchParams& p) {
  const int rc = describe_launch(b, n, p);
  if (rc != MLXD_OK || !p.out_f32) {
    return rc;
  }
  CastTable cast;
  const int got = get_lut(ctx, b, p.c_out, cast);
  p.lut = cast.values;
  p.cast = cast.steps;
  return got;
}

// Threads that pack one batch's pageable sources (the caller included):
// MLXD_PACK_THREADS, default 4, at most 32.
static int pack_threads() {
  static const int n = [] {
    const char* v = std::getenv("MLXD_PACK_THREADS");
    const int want = v && *v ? std::atoi(v) : 4;
    return want < 1 ? 1 : (want > 32 ? 32 : want);
  }();
  return n;
}

// Rows out of a source, back to back, into a page-locked block (16-byte aligned, with room up
// to the next multiple of 16), by stores past the caches: the copy engine reads lines that a
// core holds modified at a third of the bus's rate.  Where one row ends and the next begins
// inside 64 bytes they are put together first, so that whole lines leave.  32 images of 256-640
// px, 12.3 MB: packing 290 us by memcpy, 200 so, the copy after it 650 and 230.  On a host
// without SSE2 the stores are plain ones.
static void pack_rows(uint8_t* to, const uint8_t* from, size_t pitch, size_t row_bytes, size_t rows) {
  if (row_bytes == pitch) {   // one piece
    row_bytes *= rows;
    rows = 1;
  }
  alignas(64) uint8_t buffer[64];
  size_t held = 0;
  auto stream = [](uint8_t* d, const uint8_t* s, size_t n) {   // n: a multiple of 64
#ifdef __SSE2__
    for (size_t i = 0; i < n; i += 64) {
      const __m128i a = _mm_loadu_si128(reinterpret_cast<const __m128i*>(s + i));
      const __m128i b = _mm_loadu_si128(reinterpret_cast<const __m128i*>(s + i + 16));
      const __m128i c = _mm_loadu_si128(reinterpret_cast<const __m128i*>(s + i + 32));
      const __m128i e = _mm_loadu_si128(reinterpret_cast<const __m128i*>(s + i + 48));
      _mm_stream_si128(reinterpret_cast<__m128i*>(d + i), a);
      _mm_stream_si128(reinterpret_cast<__m128i*>(d + i + 16), b);
      _mm_stream_si128(reinterpret_cast<__m128i*>(d + i + 32), c);
      _mm_stream_si128(reinterpret_cast<__m128i*>(d + i + 48), e);
    }
#else
    std::memcpy(d, s, n);
#endif
  };
  for (size_t r = 0; r < rows; r++) {
    const uint8_t* s = from + r * pitch;
    size_t left = row_bytes;
    while (left > 0) {
      if (held == 0 && left >= 64) {   // straight through
        const size_t n = left & ~(size_t)63;
        stream(to, s, n);
        to += n;
        s += n;
        left -= n;
        continue;
      }
      const size_t n = std::min(left, 64 - held);
      std::memcpy(buffer + held, s, n);
      s += n;
      left -= n;
      held += n;
      if (held == 64) {
        stream(to, buffer, 64);
        to += 64;
        held = 0;
      }
    }
  }
  if (held > 0) {
    std::memcpy(to, buffer, held);
  }
#ifdef __SSE2__
  _mm_sfence();
#endif
}

int enqueue_on_lane(
    mlxd_ctx* ctx, Lane& lane, const mlxd_sample_desc* samples, int n, const mlxd_batch_desc* batch,
    const std::vector<void*>* per_sample_dst) {
  if (!samples || !batch || n < 0) {
    return fail(MLXD_ERR_INVALID, "null descriptor or negative sample count");
  }
  if (n == 0) {
    return MLXD_OK;
  }
  if (!batch->dst && !per_sample_dst) {
    return fail(MLXD_ERR_INVALID, "null batch destination");
  }
  MLXD_ON_DEVICE(ctx->device);
  LutUse table_in_use(ctx);
  LaunchParams p;
  int rc = prepare_launch(ctx, batch, n, p);
  if (rc != MLXD_OK) {
    return rc;
  }
  const std::unique_ptr<DevSample[]> dev(new DevSample[n]);   // (planning sets all of a record)
  p.status = lane.d_status;
  ResizePlan plan;
  rc = plan_samples(samples, n, batch, dev.get(), plan);
  if (rc != MLXD_OK) {
    return rc;
  }
  choose_kernels(p, plan, dev.get(), n);
  const size_t esize = p.out_f32 ? 4 : 1;
  const size_t slot_bytes = (size_t)batch->slot_h * batch->slot_w * p.c_out * esize;
  const size_t out_bytes = slot_bytes * n;
  const bool host_src = batch->src_mem == MLXD_MEM_HOST;
  const bool host_dst = batch->dst_mem == MLXD_MEM_HOST;
  if (per_sample_dst && host_dst) {
    return fail(MLXD_ERR_INVALID, "per-sample destinations must be device memory");
  }

  std::lock_guard<std::mutex> guard(lane.mu);
  const int slot = lane.next_slot;
  lane.next_slot = (slot + 1) % kDescSlots;
  // The pinned descriptor table of this slot may still be in flight.
  MLXD_CUDA(cudaEventSynchronize(lane.desc_copied[slot]));
  harvest_timing(ctx, lane, slot, true);
  // descriptors, then (for host sources) the table of the gather kernel
  const size_t desc_bytes = (sizeof(DevSample) * n + 255) & ~(size_t)255;
  const size_t block_bytes = desc_bytes + sizeof(GatherPiece) * n;
  rc = arena_reserve(ctx, lane.h_desc[slot], block_bytes, true, lane.stream);
  if (rc != MLXD_OK) {
    return rc;
  }
  rc = arena_reserve(ctx, lane.d_desc[slot], block_bytes, false, lane.stream);
  if (rc != MLXD_OK) {
    return rc;
  }

  // Stage host sources: only the rows the chain reads, each block 256-byte aligned.
  struct Piece {
    size_t offset, row_bytes, rows, from_pitch, first_row;
    const uint8_t* from;
  };
  std::vector<Piece> pieces;
  size_t stage_bytes = 0;
  uint64_t algo_src = 0;
  for (int i = 0; i < n; i++) {
    int32_t r0, r1, c0, c1;
    needed_region(dev[i], 0, r0, r1, c0, c1);
    algo_src += (uint64_t)(r1 - r0) * (uint64_t)(c1 - c0) * p.c_in;
  }
  ctx->algo_src += algo_src;
  ctx->algo_dst += out_bytes;
  // Page-locked sources that the GPU can address are packed by a kernel that
  // reads exactly the needed rectangles (gather.cu); anything else goes
  // through the copy engines.  MLXD_HOST_GATHER=0 turns the kernel path off.
  bool gather = false;
  std::vector<const uint8_t*> src_dev;
  if (host_src) {
    static const bool gather_enabled = [] {
      const char* v = std::getenv("MLXD_HOST_GATHER");
      return !(v && *v == '0');
    }();
    gather = gather_enabled;
    src_dev.resize(n);
    // sources in blocks from mlxd_pinned_alloc: a table look-up, no driver call
    for (int i = 0; i < n && gather; i++) {
      src_dev[i] = pinned_registry_lookup(samples[i].src);
      gather = src_dev[i] != nullptr;
    }
  }
  bool bounce = false;              // some source lies in ordinary (pageable) host memory
  std::vector<char> direct_copy;    // per sample: page-locked memory the copy engines can read
  unsigned int host_flags = 0;
  if (host_src) {
    pieces.resize(n);
    direct_copy.assign(n, 0);
    for (int i = 0; i < n; i++) {
      int32_t r0, r1, c0, c1;
      needed_region(dev[i], 2, r0, r1, c0, c1);
      // A strided (2-D) copy moves fewer bytes but runs slower per byte than a
      // contiguous one: trim columns only when that drops at least the
      // configured share of every row (MLXD_TRIM_PERCENT, default 60).
      static const int trim_percent = [] {
        const char* v = std::getenv("MLXD_TRIM_PERCENT");
        return v && *v ? std::atoi(v) : 60;
      }();
      // (sources in ordinary host memory are packed by the calling thread into a
      // page-locked block, which drops the columns for free)
      const bool direct = !gather && cudaHostGetFlags(&host_flags, const_cast<uint8_t*>(samples[i].src)) == cudaSuccess;
      if (!gather && !direct) {
        cudaGetLastError();
        bounce = true;
      }
      if (direct && (int64_t)(dev[i].src_w - (c1 - c0)) * 100 < (int64_t)trim_percent * dev[i].src_w) {
        c0 = 0;
        c1 = dev[i].src_w;
      }
      direct_copy[i] = direct;
      // The staged block is an image of its own: rows [r0, r1), columns
      // [c0, c1) of the source, tightly packed.
      pieces[i].offset = stage_bytes;
      pieces[i].row_bytes = (size_t)(c1 - c0) * p.c_in;
      pieces[i].rows = (size_t)(r1 - r0);
      pieces[i].from_pitch = (size_t)dev[i].src_w * p.c_in;
      pieces[i].from = samples[i].src + pieces[i].from_pitch * (size_t)r0 + (size_t)c0 * p.c_in;
      stage_bytes += (pieces[i].row_bytes * pieces[i].rows + 255) & ~(size_t)255;
      dev[i].src_w = c1 - c0;
      dev[i].pre_x -= c0;
      pieces[i].first_row = (size_t)r0;
    }
    rc = arena_reserve(ctx, lane.d_src, stage_bytes + 256, false, lane.stream);
    if (rc != MLXD_OK) {
      return rc;
    }
    for (int i = 0; i < n; i++) {
      // Base of a virtual image whose rows from r0 on are the staged block.
      dev[i].src = static_cast<const uint8_t*>(lane.d_src.ptr) + pieces[i].offset -
          pieces[i].row_bytes * pieces[i].first_row;
    }
  }
  uint8_t* out_base = static_cast<uint8_t*>(batch->dst);
  if (host_dst) {
    rc = arena_reserve(ctx, lane.d_out, out_bytes, false, lane.stream);
    if (rc != MLXD_OK) {
      return rc;
    }
    out_base = static_cast<uint8_t*>(lane.d_out.ptr);
  }
  for (int i = 0; i < n; i++) {
    dev[i].dst = per_sample_dst ? (*per_sample_dst)[i] : static_cast<void*>(out_base + slot_bytes * i);
  }

  std::memcpy(lane.h_desc[slot].ptr, dev.get(), sizeof(DevSample) * n);
  size_t upload = sizeof(DevSample) * n;
  uint32_t gather_rows = 0;
  if (gather) {
    GatherPiece* gp = reinterpret_cast<GatherPiece*>(static_cast<uint8_t*>(lane.h_desc[slot].ptr) + desc_bytes);
    for (int i = 0; i < n; i++) {
      gp[i].src = src_dev[i] + (pieces[i].from - samples[i].src);
      gp[i].dst = static_cast<uint8_t*>(lane.d_src.ptr) + pieces[i].offset;
      gp[i].src_pitch = pieces[i].from_pitch;
      gp[i].rows = (uint32_t)pieces[i].rows;
      gp[i].row_bytes = (uint32_t)pieces[i].row_bytes;
      gp[i].first_row = gather_rows;
      gp[i].pad_ = 0;
      gather_rows += (uint32_t)pieces[i].rows;
    }
    upload = block_bytes;
  }
  MLXD_CUDA(cudaMemcpyAsync(lane.d_desc[slot].ptr, lane.h_desc[slot].ptr, upload, cudaMemcpyHostToDevice, lane.stream));
  MLXD_CUDA(cudaEventRecord(lane.desc_copied[slot], lane.stream));
  const bool timed = ctx->timing.load() != 0;
  lane.in_timed[slot] = false;
  lane.out_timed[slot] = false;
  bool sent_early = false;   // all sources are on their way already
  // A call that fails while copies out of the lane's block are queued waits for them: the next
  // one writes into it, and src_copied, which it waits for, does not tell of these.
  struct Drain {
    cudaStream_t stream;
    bool armed;
    ~Drain() {
      if (armed) {
        cudaStreamSynchronize(stream);
      }
    }
  } block_in_use{lane.stream, false};
  if (bounce) {
    // Pack the rectangles of the pageable sources into the lane's page-locked
    // block (the calling thread does the copying), then one copy for all of
    // them.  The block may still be feeding the previous batch of this lane.
    rc = arena_reserve(ctx, lane.h_src, stage_bytes + 256, true, lane.stream);
    if (rc != MLXD_OK) {
      return rc;
    }
    MLXD_CUDA(cudaEventSynchronize(lane.src_copied));
    block_in_use.armed = true;
    const auto t0 = std::chrono::steady_clock::now();
    // The calling thread and up to pack_threads - 1 helpers started for this
    // batch take samples off a shared counter; packing is plain row copies.
    std::atomic<int> next{0};
    uint8_t* const block = static_cast<uint8_t*>(lane.h_src.ptr);
    // Where all sources are packed, the calling thread sends off what is ready between its
    // own samples, in parts of two megabytes, so that the copy runs beside the packing.  One batch
    // of 32 images of 256-640 px (12.3 MB): 905 us, 797 so; two of 48 1425 and 1180; four lanes at
    // once, which fill each other's gaps, 2508 and 2450.
    constexpr size_t kPart = size_t(2) << 20;
    sent_early = stage_bytes >= 2 * kPart && std::find(direct_copy.begin(), direct_copy.end(), 1) == direct_copy.end();
    const std::unique_ptr<std::atomic<bool>[]> packed(new std::atomic<bool>[n]());
    int sent = 0;
    size_t sent_bytes = 0;
    cudaError_t sending = cudaSuccess;
    auto send = [&](size_t least) {
      int ready = sent;
      while (ready < n && packed[ready].load(std::memory_order_acquire)) {
        ready++;
      }
      const size_t end = ready == n ? stage_bytes : pieces[ready].offset;
      if (sending == cudaSuccess && end >= sent_bytes + least) {
        if (timed && sent == 0) {
          sending = cudaEventRecord(lane.in_begin[slot], lane.stream);
          lane.in_timed[slot] = sending == cudaSuccess;
        }
        sending = sending != cudaSuccess ? sending : cudaMemcpyAsync(
            static_cast<uint8_t*>(lane.d_src.ptr) + sent_bytes, block + sent_bytes, end - sent_bytes, cudaMemcpyHostToDevice,
            lane.stream);
        sent = ready;
        sent_bytes = end;
      }
    };
    auto pack = [&](bool caller) {
      for (int i = next.fetch_add(1); i < n; i = next.fetch_add(1)) {
        if (direct_copy[i]) {
          continue;
        }
        pack_rows(block + pieces[i].offset, pieces[i].from, pieces[i].from_pitch, pieces[i].row_bytes, pieces[i].rows);
        packed[i].store(true, std::memory_order_release);
        if (caller && sent_early) {
          send(kPart);
        }
      }
    };
    const int helpers = stage_bytes >= (size_t(8) << 20) ? std::min(pack_threads() - 1, n - 1) : 0;
    std::vector<std::thread> crew;
    crew.reserve(helpers > 0 ? helpers : 0);
    for (int t = 0; t < helpers; t++) {
      crew.emplace_back(pack, false);
    }
    pack(true);
    for (auto& th : crew) {
      th.join();
    }
    if (sent_early) {
      send(1);
      MLXD_CUDA(sending);
    }
    ctx->host_stage_ns += (uint64_t)std::chrono::duration_cast<std::chrono::nanoseconds>(
        std::chrono::steady_clock::now() - t0).count();
  }
  if (timed && host_src && !sent_early) {
    MLXD_CUDA(cudaEventRecord(lane.in_begin[slot], lane.stream));
    lane.in_timed[slot] = true;
  }
  if (gather) {
    const GatherPiece* gd =
        reinterpret_cast<const GatherPiece*>(static_cast<const uint8_t*>(lane.d_desc[slot].ptr) + desc_bytes);
    MLXD_CUDA(launch_gather_rows(gd, n, gather_rows, lane.stream));
    ctx->launches += 1;
    uint64_t moved = 0;
    for (int i = 0; i < n; i++) {
      moved += (uint64_t)pieces[i].row_bytes * pieces[i].rows;
    }
    ctx->h2d += moved;
  } else if (host_src) {
    bool all_bounced = true;
    for (int i = 0; i < n; i++) {
      all_bounced = all_bounced && !direct_copy[i];
    }
    if (sent_early) {
      // (nothing is left)
    } else if (all_bounced) {
      MLXD_CUDA(cudaMemcpyAsync(lane.d_src.ptr, lane.h_src.ptr, stage_bytes, cudaMemcpyHostToDevice, lane.stream));
    } else {
      for (int i = 0; i < n; i++) {
        uint8_t* to = static_cast<uint8_t*>(lane.d_src.ptr) + pieces[i].offset;
        const size_t bytes = pieces[i].row_bytes * pieces[i].rows;
        if (!direct_copy[i]) {
          MLXD_CUDA(cudaMemcpyAsync(
              to, static_cast<uint8_t*>(lane.h_src.ptr) + pieces[i].offset, bytes, cudaMemcpyHostToDevice, lane.stream));
        } else if (pieces[i].row_bytes == pieces[i].from_pitch) {
          MLXD_CUDA(cudaMemcpyAsync(to, pieces[i].from, bytes, cudaMemcpyHostToDevice, lane.stream));
        } else {
          MLXD_CUDA(cudaMemcpy2DAsync(
              to, pieces[i].row_bytes, pieces[i].from, pieces[i].from_pitch, pieces[i].row_bytes, pieces[i].rows,
              cudaMemcpyHostToDevice, lane.stream));
        }
      }
    }
    if (bounce) {
      MLXD_CUDA(cudaEventRecord(lane.src_copied, lane.stream));
      block_in_use.armed = false;
    }
    ctx->h2d += stage_bytes;
  }
  p.samples = static_cast<const DevSample*>(lane.d_desc[slot].ptr);
  if (timed) {
    MLXD_CUDA(cudaEventRecord(lane.k_begin[slot], lane.stream));
  }
  MLXD_CUDA(launch_fused_batch(p, plan, lane.stream));
  if (timed) {
    MLXD_CUDA(cudaEventRecord(lane.k_end[slot], lane.stream));
    lane.k_pending[slot] = true;
  }
  if (host_dst) {
    MLXD_CUDA(cudaMemcpyAsync(batch->dst, lane.d_out.ptr, out_bytes, cudaMemcpyDeviceToHost, lane.stream));
    ctx->d2h += out_bytes;
    if (timed) {
      MLXD_CUDA(cudaEventRecord(lane.out_end[slot], lane.stream));
      lane.out_timed[slot] = true;
    }
  }
  lane.h_status[1] = 1;
  const cudaError_t brought =
      cudaMemcpyAsync(lane.h_status, lane.d_status, kStatusWords * sizeof(int32_t), cudaMemcpyDeviceToHost, lane.stream);
  if (brought != cudaSuccess) {
    lane.h_status[1] = 0;
    return fail_cuda(brought, "cudaMemcpyAsync(status)");
  }
  MLXD_CUDA(cudaEventRecord(lane.done, lane.stream));
  ctx->batches += 1;
  ctx->samples += n;
  ctx->launches += 1;
  return MLXD_OK;
}

void harvest_timing(mlxd_ctx* ctx, Lane& lane, int slot, bool block) {
  if (!lane.k_pending[slot]) {
    return;
  }
  if (block) {
    if (cudaEventSynchronize(lane.k_end[slot]) != cudaSuccess) {
      return;
    }
  } else if (cudaEventQuery(lane.k_end[slot]) != cudaSuccess) {
    return;
  }
  if (lane.out_timed[slot]) {
    const cudaError_t oe = block ? cudaEventSynchronize(lane.out_end[slot]) : cudaEventQuery(lane.out_end[slot]);
    if (oe != cudaSuccess) {
      return;
    }
  }
  float ms = 0.0f;
  if (cudaEventElapsedTime(&ms, lane.k_begin[slot], lane.k_end[slot]) == cudaSuccess) {
    ctx->kernel_ns += (uint64_t)((double)ms * 1e6);
    ctx->timed_launches += 1;
  }
  if (lane.in_timed[slot] && cudaEventElapsedTime(&ms, lane.in_begin[slot], lane.k_begin[slot]) == cudaSuccess) {
    ctx->h2d_ns += (uint64_t)((double)ms * 1e6);
  }
  if (lane.out_timed[slot] && cudaEventElapsedTime(&ms, lane.k_end[slot], lane.out_end[slot]) == cudaSuccess) {
    ctx->d2h_ns += (uint64_t)((double)ms * 1e6);
  }
  lane.in_timed[slot] = false;
  lane.out_timed[slot] = false;
  lane.k_pending[slot] = false;
}

int wait_lane(mlxd_ctx* ctx, Lane& lane, int timeout_ms) {
  MLXD_ON_DEVICE(ctx->device);
  const auto start = std::chrono::steady_clock::now();
  if (timeout_ms < 0) {
    // No deadline.  Blocked in the driver a thread wakes 200 us and more after the GPU's
    // interrupt (a virtual machine's processor sleeps meanwhile), so it first looks a while at
    // the word that the lane's last copy clears, without asking the driver from every lane.
    // One batch of 8 full-HD frames 1027 us, 696 so.  It gives its processor to any thread that
    // has work: where decoding, packing and waiting threads share two processors, four batches of 32
    // numpy images take 4924 us blocked at once and 4673 so, two of 32 JPEG files 43.5 ms and
    // 42.5; on four processors 3913 and 3562, 21.8 and 21.7.
    const volatile int32_t* const under_way = lane.h_status + 1;
    for (int i = 0; *under_way != 0; i++) {
#ifdef __SSE2__
      _mm_pause();
#endif
      if (i % 64 == 63) {
        if (std::chrono::steady_clock::now() - start > std::chrono::microseconds(kLookMicroseconds)) {
          break;
        }
        sched_yield();
      }
    }
    // (the event is next; with several batches in flight on the lane the word may be cleared by an earlier one)
    cudaError_t e = cudaErrorNotReady;
    for (int i = 0; i < 64 && e == cudaErrorNotReady && *under_way == 0; i++) {
      e = cudaEventQuery(lane.done);
    }
    if (e != cudaSuccess) {
      MLXD_CUDA(cudaEventSynchronize(lane.done));
    }
  }
  for (;;) {
    cudaError_t e = cudaEventQuery(lane.done);
    if (e == cudaSuccess) {
      break;
    }
    if (e != cudaErrorNotReady) {
      return fail_cuda(e, "cudaEventQuery(lane)");
    }
    if (timeout_ms >= 0) {
      const auto el = std::chrono::duration_cast<std::chrono::milliseconds>(
          std::chrono::steady_clock::now() - start).count();
      if (el >= timeout_ms) {
        return fail(MLXD_ERR_TIMEOUT, "lane still busy after " + std::to_string(timeout_ms) + " ms");
      }
    }
    std::this_thread::sleep_for(std::chrono::microseconds(20));
  }
  {
    std::lock_guard<std::mutex> guard(lane.mu);
    for (int s = 0; s < kDescSlots; s++) {
      harvest_timing(ctx, lane, s, false);
    }
  }
  if (*lane.h_status != 0) {
    // Reported once: the word is cleared so that later batches on this lane
    // start clean (other lanes have words of their own).
    const int32_t seen = *lane.h_status;
    *lane.h_status = 0;
    cudaMemsetAsync(lane.d_status, 0, sizeof(int32_t), lane.stream);
    return fail(MLXD_ERR_DEVICE, "kernel self-check failed (status " + std::to_string(seen) + ")");
  }
  return MLXD_OK;
}

} // namespace mlxd
