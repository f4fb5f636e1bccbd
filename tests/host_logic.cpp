// The host side of the C ABI (context.cu, api.cu, launch_plan.cu, noalloc.cu) against a CUDA
// runtime made up here: device memory is host memory, a stream is a list of work that runs when
// it is waited for, kernels are functions below.  So what a call queues, and what another caller
// does in between, is the same in every run, and calls can be made to fail.
//
// Usage: host_logic SCENARIO; exits with 0 if it holds, else prints what does not.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <string>
#include <vector>

#include "context.h"

using namespace mlxd;

// ---------------------------------------------------------------- the runtime
struct CUstream_st {
  std::deque<std::function<void()>> work;
  uint64_t queued = 0, done = 0;
};
struct CUevent_st {
  CUstream_st* stream = nullptr;
  uint64_t at = 0;
};

namespace {

std::vector<std::string> calls;              // what was queued and waited for, in order
std::function<cudaError_t(const std::string&)> before = [](const std::string&) { return cudaSuccess; };
std::function<void()> looked = [] {};        // after an event was looked at
std::function<void(const LaunchParams&)> kernel = [](const LaunchParams&) {};
CUstream_st legacy;

CUstream_st* of(cudaStream_t s) {
  return s ? s : &legacy;
}

void queue(cudaStream_t s, std::function<void()> f) {
  of(s)->work.push_back(std::move(f));
  of(s)->queued++;
}

void run(cudaStream_t s) {
  while (!of(s)->work.empty()) {
    const auto f = of(s)->work.front();
    of(s)->work.pop_front();
    f();
    of(s)->done++;
  }
}

// Notes a call and lets the scenario act before it, or make it fail.
cudaError_t note(const std::string& what) {
  calls.push_back(what);
  return before(what);
}

#define FAKE(what)                        \
  const cudaError_t fails__ = note(what); \
  if (fails__ != cudaSuccess) return fails__

} // namespace

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "made up"; }
cudaError_t cudaDeviceGetPCIBusId(char* s, int, int) { *s = 0; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { *p = std::aligned_alloc(256, (n + 255) & ~size_t(255)); return cudaSuccess; }
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) { *d = h; return cudaSuccess; }
cudaError_t cudaHostGetFlags(unsigned*, void*) { return cudaErrorInvalidValue; }   // all of it is pageable
cudaError_t cudaGetSymbolAddress(void** p, const void* s) { *p = const_cast<void*>(s); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemset(void* d, int v, size_t n) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = new CUstream_st; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { delete s; return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* c) { *c = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { FAKE("wait stream"); run(s); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = new CUevent_st; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete e; return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  FAKE("record");
  queue(s, [] {});
  e->stream = of(s);
  e->at = of(s)->queued;
  return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e) {
  FAKE("query");
  const bool ready = !e->stream || e->stream->done >= e->at;
  if (!ready) {
    run(e->stream);   // the GPU goes on meanwhile
  }
  looked();
  return ready ? cudaSuccess : cudaErrorNotReady;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  FAKE("wait event");
  if (e->stream && e->stream->done < e->at) {
    run(e->stream);
  }
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind kind, cudaStream_t stream) {
  FAKE(kind == cudaMemcpyHostToDevice ? "copy in" : "copy out");
  queue(stream, [=] { std::memcpy(d, s, n); });
  return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void*, size_t, const void*, size_t, size_t, size_t, cudaMemcpyKind, cudaStream_t) { std::abort(); }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t stream) {
  FAKE("set");
  queue(stream, [=] { std::memset(d, v, n); });
  return cudaSuccess;
}
}

namespace mlxd {
cudaError_t launch_fused_batch(const LaunchParams& p, const ResizePlan&, cudaStream_t stream) {
  FAKE(p.samples ? "kernel" : "kernel with records");
  LaunchParams q = p;
  queue(stream, [q] { kernel(q); });
  return cudaSuccess;
}
cudaError_t launch_gather_rows(const GatherPiece*, int, uint32_t, cudaStream_t) { std::abort(); }
int capture_batch(LaunchParams&, const ResizePlan&, const DevSample*, const mlxd_batch_desc*, cudaStream_t) { std::abort(); }
} // namespace mlxd

// ---------------------------------------------------------------- scenarios
namespace {

int failures = 0;

void check(bool holds, const char* what, int line) {
  if (!holds) {
    std::printf("line %d: %s (%s)\n", line, what, mlxd_last_error());
    failures++;
  }
}
#define CHECK(x) check((x), #x, __LINE__)

mlxd_ctx* context() {
  mlxd_ctx* ctx = nullptr;
  CHECK(mlxd_ctx_create(0, 1, &ctx) == MLXD_OK);
  return ctx;
}

mlxd_sample_desc whole(const uint8_t* src, int h, int w) {
  mlxd_sample_desc d{};
  d.src = src;
  d.src_h = d.pre_h = d.geom_h = d.post_h = h;
  d.src_w = d.pre_w = d.geom_w = d.post_w = w;
  return d;
}

mlxd_batch_desc batch_of(void* dst, int h, int w, int c) {
  mlxd_batch_desc b{};
  b.dst = dst;
  b.slot_h = h;
  b.slot_w = w;
  b.channels = c;
  b.out_dtype = MLXD_U8;
  b.divisor = 1.0f;
  b.src_mem = b.dst_mem = MLXD_MEM_HOST;
  return b;
}

// Another caller queues a batch on a lane at any look of a wait for it.
void wait_beside_another_caller() {
  uint8_t src[64 * 3] = {}, dst[2][64 * 3];
  const mlxd_sample_desc d = whole(src, 8, 8);
  const mlxd_batch_desc b[2] = {batch_of(dst[0], 8, 8, 3), batch_of(dst[1], 8, 8, 3)};
  for (const int32_t status : {0, 8}) {
    for (int step = 1; step <= 4; step++) {
      mlxd_ctx* ctx = context();
      kernel = [&](const LaunchParams& p) { *p.status |= status; };
      CHECK(mlxd_fused_batch(ctx, 0, &d, 1, &b[0]) == MLXD_OK);
      run(ctx->lanes[0]->stream);
      kernel = [](const LaunchParams&) {};
      int left = step;
      looked = [&] {
        if (--left == 0) {
          CHECK(mlxd_fused_batch(ctx, 0, &d, 1, &b[1]) == MLXD_OK);
        }
      };
      const int rc = mlxd_batch_wait(ctx, 0, -1);
      CHECK(rc == (status ? MLXD_ERR_DEVICE : MLXD_OK));
      CHECK(!status || std::strstr(mlxd_last_error(), "(status 8)"));
      looked = [] {};
      if (!status) {
        CHECK(mlxd_batch_wait(ctx, 0, -1) == MLXD_OK);
        CHECK(ctx->lanes[0]->stream->work.empty());
      }
      mlxd_ctx_destroy(ctx);
    }
  }
}

// Copies out of sources that no strip can take, beside a resize that runs in strips, stay copies.
void copies_of_huge_sources_beside_a_resize() {
  uint8_t src[4] = {}, dst[4];   // (planning reads no pixels)
  struct Case { int w, channels; bool joins; };
  for (const Case& k : {Case{1 << 30, 3, false}, Case{(1 << 29) + 5, 4, false}, Case{1 << 29, 1, false}, Case{1 << 28, 4, false},
                        Case{1 << 27, 4, false}, Case{4000, 3, true}}) {
    mlxd_sample_desc d[2] = {whole(src, 2, k.w), whole(src, 40, 30)};
    d[0].post_x = k.w - 9;
    d[0].post_w = 8;
    d[1].geom = MLXD_GEOM_RESIZE;
    d[1].geom_w = d[1].post_w = 8;
    d[1].geom_h = d[1].post_h = 20;
    const mlxd_batch_desc b = batch_of(dst, 20, 8, k.channels);
    DevSample out[2];
    ResizePlan plan;
    CHECK(plan_into(d, 2, &b, out, plan) == MLXD_OK);
    CHECK(out[0].mode == (k.joins ? kModeResize : kModeCopy));
    CHECK(out[1].mode == kModeResize);
    CHECK(out[0].post_x == k.w - 9 && out[0].post_w == 8 && out[0].post_h == 2);
  }
}

// A copy that fails after others of the same batch were queued: the call ends only when those,
// which read the lane's block, have run.
void failed_copy_of_a_part() {
  const int h = 1100, w = 700, n = 3;   // a part each, packed by the caller alone
  std::vector<uint8_t> src((size_t)h * w * 3, 7), dst(src.size() * n);
  std::vector<mlxd_sample_desc> d(n, whole(src.data(), h, w));
  const mlxd_batch_desc b = batch_of(dst.data(), h, w, 3);
  for (int bad = 3; bad <= 4; bad++) {   // (the first is the descriptors')
    mlxd_ctx* ctx = context();
    int copies = 0;
    calls.clear();
    before = [&](const std::string& call) {
      return call == "copy in" && ++copies == bad ? cudaErrorInvalidValue : cudaSuccess;
    };
    CHECK(mlxd_fused_batch(ctx, 0, d.data(), n, &b) == MLXD_ERR_CUDA);
    before = [](const std::string&) { return cudaSuccess; };
    CHECK(copies == bad);
    CHECK(ctx->lanes[0]->stream->work.empty());
    // and the lane goes on
    CHECK(mlxd_fused_batch(ctx, 0, d.data(), n, &b) == MLXD_OK);
    CHECK(mlxd_batch_wait(ctx, 0, -1) == MLXD_OK);
    mlxd_ctx_destroy(ctx);
  }
}

// What a call queues besides events.
std::vector<std::string> queued() {
  std::vector<std::string> out;
  for (const std::string& c : calls) {
    if (c != "record" && c != "query" && c.rfind("wait", 0) != 0) {
      out.push_back(c);
    }
  }
  return out;
}

// Timed calls queue the same copies and kernels as others, and each is counted once.
void timed_calls_take_the_same_way() {
  const int h = 1100, w = 700, n = 3;
  std::vector<uint8_t> src((size_t)h * w * 3, 7), dst(src.size() * 129);
  const mlxd_batch_desc host = batch_of(dst.data(), h, w, 3);
  mlxd_batch_desc device = batch_of(dst.data(), 8, 8, 3);
  device.src_mem = device.dst_mem = MLXD_MEM_DEVICE;
  std::vector<mlxd_sample_desc> frames(n, whole(src.data(), h, w)), tiny(129, whole(src.data(), 8, 8));
  std::vector<std::string> way[2];
  for (int timed = 0; timed < 2; timed++) {
    mlxd_ctx* ctx = context();
    CHECK(mlxd_ctx_set_timing(ctx, timed) == MLXD_OK);
    calls.clear();
    for (int i = 0; i < 6; i++) {   // (more than there are slots)
      for (const int k : {1, 24, 128, 129}) {
        CHECK(mlxd_fused_batch_on_stream(ctx, nullptr, tiny.data(), k, &device) == MLXD_OK);
        run(nullptr);
      }
      CHECK(mlxd_fused_batch(ctx, 0, frames.data(), n, &host) == MLXD_OK);
      CHECK(mlxd_batch_wait(ctx, 0, -1) == MLXD_OK);
    }
    way[timed] = queued();
    mlxd_stats stats;
    CHECK(mlxd_stats_get(ctx, &stats) == MLXD_OK);
    CHECK(stats.timed_launches == (timed ? 30u : 0u));
    CHECK(stats.kernel_ns == stats.timed_launches * 1000000u);   // (a made-up event is 1 ms from any other)
    CHECK(stats.h2d_ns == (timed ? 6000000u : 0u));
    mlxd_ctx_destroy(ctx);
  }
  CHECK(way[0] == way[1]);
}

// Casts that give NaN are looked up: steps on the GPU would give other NaNs than the table's.
void casts_with_nan_keep_the_table() {
  const float nan = std::nanf("");
  struct Case { float divisor, mean, std; int normalise, mode; };
  for (const Case& k : {Case{255.0f, 0.0f, 1.0f, 0, kCastScale}, Case{255.0f, 0.4f, 0.2f, 1, kCastNormalise},
                        Case{nan, 0.0f, 1.0f, 0, kCastTable}, Case{-nan, 0.4f, 0.2f, 1, kCastTable},
                        Case{255.0f, 0.4f, nan, 1, kCastTable}, Case{255.0f, 0.4f, -nan, 1, kCastTable},
                        Case{255.0f, nan, 0.2f, 1, kCastTable}, Case{255.0f, 0.0f, 0.0f, 1, kCastTable}}) {
    mlxd_batch_desc b = batch_of(nullptr, 8, 8, 3);
    b.out_dtype = MLXD_F32;
    b.divisor = k.divisor;
    b.normalise = k.normalise;
    for (int c = 0; c < 3; c++) {
      b.mean[c] = c == 1 ? k.mean : 0.5f;
      b.std_[c] = c == 1 ? k.std : 0.25f;
    }
    float table[3 * 256];
    CastSteps steps;
    compute_cast_table(&b, 3, table);
    cast_steps(&b, 3, table, steps);
    CHECK(steps.mode == k.mode);
  }
}

mlxd_batch_desc cast_batch(int c, int normalise, float divisor, float mean, float std) {
  mlxd_batch_desc b = batch_of(nullptr, 8, 8, c);
  b.src_mem = b.dst_mem = MLXD_MEM_DEVICE;
  b.out_dtype = MLXD_F32;
  b.divisor = divisor;
  b.normalise = normalise;
  for (int i = 0; i < 4; i++) {
    b.mean[i] = mean + 0.01f * (float)i;
    b.std_[i] = std + 0.01f * (float)i;
  }
  return b;
}

// Least microseconds of a call.
template <class F>
double least_us(F&& f) {
  double best = 1e9;
  for (int i = 0; i < 2000; i++) {
    const auto t = std::chrono::steady_clock::now();
    f();
    best = std::min(best, std::chrono::duration<double, std::micro>(std::chrono::steady_clock::now() - t).count());
  }
  return best;
}

// Calls without a context's cache: each has the steps of its own cast, in whatever order casts come,
// and a cast that comes again is not compared value by value again.
void casts_without_a_cache() {
  std::vector<mlxd_batch_desc> casts;
  for (int c = 1; c <= 4; c++) {
    casts.push_back(cast_batch(c, 0, 255.0f, 0.0f, 0.0f));
    casts.push_back(cast_batch(c, 0, 1e-39f, 0.0f, 0.0f));
    casts.push_back(cast_batch(c, 1, 255.0f, 0.4f, 0.2f));
    casts.push_back(cast_batch(c, 1, 255.0f, 0.4f, 0.3f));
  }
  casts.push_back(cast_batch(3, 1, 255.0f, 0.4f, 0.2f));
  casts.back().gray = 1;
  uint8_t src[8 * 8 * 4] = {};
  std::vector<uint8_t> dst(8 * 8 * 16);
  LaunchParams launched;
  kernel = [&](const LaunchParams& p) { launched = p; };
  const mlxd_sample_desc d = whole(src, 8, 8);
  auto call = [&](const mlxd_batch_desc& cast) {
    mlxd_batch_desc b = cast;
    b.dst = dst.data();
    CHECK(mlxd_fused_batch_noalloc(0, nullptr, &d, 1, &b) == MLXD_OK);
    run(nullptr);
    calls.clear();
  };
  unsigned order = 1;
  for (int i = 0; i < 400; i++) {
    order = order * 1664525u + 1013904223u;
    const mlxd_batch_desc& b = casts[i < 100 ? i % casts.size() : (order >> 8) % (i < 250 ? 4 : casts.size())];
    call(b);
    const int c_out = b.gray ? 1 : b.channels;
    float table[4 * 256];
    CastSteps steps;
    compute_cast_table(&b, c_out, table);
    cast_steps(&b, c_out, table, steps);
    CHECK(std::memcmp(&steps, &launched.cast, sizeof(steps)) == 0);
    CHECK(std::memcmp(table, launched.lut, sizeof(float) * 256 * c_out) == 0);
  }
  mlxd_batch_desc bytes = cast_batch(3, 0, 1.0f, 0.0f, 0.0f);
  bytes.out_dtype = MLXD_U8;
  const mlxd_batch_desc floats = cast_batch(3, 1, 255.0f, 0.4f, 0.2f);
  float table[4 * 256];
  CastSteps steps;
  const double with_cast = least_us([&] { call(floats); }), without = least_us([&] { call(bytes); });
  const double table_us = least_us([&] { compute_cast_table(&floats, 3, table); });
  const double steps_us = least_us([&] { cast_steps(&floats, 3, table, steps); });
  std::printf("float call %.2f us, byte call %.2f, table %.2f, steps %.2f\n", with_cast, without, table_us, steps_us);
  CHECK(with_cast - without - table_us < 0.5 * steps_us);
}

// Pageable sources through the lane's block: windows whose rows are shorter and longer than 64
// bytes and start anywhere, in batches below and above what is sent in parts.
void packed_sources() {
  const int sizes[][4] = {{9, 5, 9, 5}, {40, 33, 31, 21}, {40, 33, 40, 33}, {300, 400, 299, 133}, {1300, 1111, 1207, 1111}, {900, 1001, 900, 777}};
  for (int c = 1; c <= 4; c++) {
    std::vector<std::vector<uint8_t>> src, got;
    std::vector<mlxd_sample_desc> d;
    for (const auto& k : sizes) {
      src.emplace_back((size_t)k[0] * k[1] * c);
      for (size_t i = 0; i < src.back().size(); i++) {
        src.back()[i] = (uint8_t)(i * 2654435761u >> 13);
      }
    }
    for (size_t i = 0; i < src.size(); i++) {
      const auto& k = sizes[i];
      d.push_back(whole(src[i].data(), k[0], k[1]));
      d.back().post_y = k[0] - k[2];
      d.back().post_x = k[1] - k[3];
      d.back().post_h = k[2];
      d.back().post_w = k[3];
    }
    std::vector<uint8_t> dst((size_t)1300 * 1111 * c * d.size());
    const mlxd_batch_desc b = batch_of(dst.data(), 1300, 1111, c);
    got.resize(d.size());
    kernel = [&](const LaunchParams& p) {   // the window of every sample, from where the launch has its source
      for (int i = 0; i < p.n; i++) {
        const DevSample& s = p.samples[i];
        for (int y = 0; y < s.post_h; y++) {
          const uint8_t* row = s.src + ((size_t)(s.pre_y + s.post_y + y) * s.src_w + s.pre_x + s.post_x) * c;
          got[i].insert(got[i].end(), row, row + (size_t)s.post_w * c);
        }
      }
    };
    mlxd_ctx* ctx = context();
    for (size_t n : {size_t(1), size_t(4), d.size()}) {
      for (auto& g : got) {
        g.clear();
      }
      CHECK(mlxd_fused_batch(ctx, 0, d.data(), (int)n, &b) == MLXD_OK);
      CHECK(mlxd_batch_wait(ctx, 0, -1) == MLXD_OK);
      for (size_t i = 0; i < n; i++) {
        const auto& k = sizes[i];
        std::vector<uint8_t> want;
        for (int y = k[0] - k[2]; y < k[0]; y++) {
          const uint8_t* row = src[i].data() + ((size_t)y * k[1] + k[1] - k[3]) * c;
          want.insert(want.end(), row, row + (size_t)k[3] * c);
        }
        CHECK(want == got[i]);
      }
    }
    mlxd_ctx_destroy(ctx);
  }
  kernel = [](const LaunchParams&) {};
}

} // namespace

int main(int argc, char** argv) {
  const std::map<std::string, void (*)()> scenarios = {
      {"wait_beside_another_caller", wait_beside_another_caller},
      {"copies_of_huge_sources_beside_a_resize", copies_of_huge_sources_beside_a_resize},
      {"failed_copy_of_a_part", failed_copy_of_a_part},
      {"timed_calls_take_the_same_way", timed_calls_take_the_same_way},
      {"casts_with_nan_keep_the_table", casts_with_nan_keep_the_table},
      {"casts_without_a_cache", casts_without_a_cache},
      {"packed_sources", packed_sources},
  };
  const auto it = argc == 2 ? scenarios.find(argv[1]) : scenarios.end();
  if (it == scenarios.end()) {
    return 2;
  }
  it->second();
  return failures ? 1 : 0;
}
