// mlxd_fused_batch_on_stream on a stream under capture.
//
// A graph may run long after the call and any number of times, so nothing of it may
// point into memory that the context uses again: not a slot of the descriptor ring, not
// the cache of cast tables, and no event of the ring may become part of the capture
// (waiting for a captured event is an error from then on).  Here the program table and
// the cast table live in an allocation of the graph's own - an allocation node ahead of
// the kernel, a free node behind it - and their bytes in the parameters of the kernels
// that write them there, which the graph keeps.  No call in here is one that a capture
// forbids.
#include <algorithm>
#include <cstring>

#include "context.h"

namespace mlxd {
namespace {

constexpr int kPutThreads = 256;

// 16 KB of a table: a kernel may take 32 764 bytes of parameters.
struct TablePiece {
  uint4 units[1024];
};

__global__ void __launch_bounds__(kPutThreads) put_table_kernel(
    const __grid_constant__ TablePiece piece, uint4* dst, int units) {
  for (int i = threadIdx.x; i < units; i += kPutThreads) {
    dst[i] = piece.units[i];
  }
}

cudaError_t put_table(const void* from, unsigned char* to, size_t bytes, cudaStream_t stream) {
  for (size_t at = 0; at < bytes; at += sizeof(TablePiece)) {
    TablePiece piece;
    const size_t here = std::min(bytes - at, sizeof(TablePiece));
    std::memcpy(&piece, static_cast<const unsigned char*>(from) + at, here);
    put_table_kernel<<<1, kPutThreads, 0, stream>>>(piece, reinterpret_cast<uint4*>(to + at), (int)(here / 16));
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
      return e;
    }
  }
  return cudaSuccess;
}

} // namespace

int capture_batch(
    LaunchParams& p, const ResizePlan& plan, const DevSample* samples, const mlxd_batch_desc* batch, cudaStream_t stream) {
  static_assert(sizeof(DevSample) % 16 == 0, "tables are written in units of 16 bytes");
  const size_t table_bytes = sizeof(DevSample) * p.n;
  std::vector<float> cast(p.out_f32 ? (size_t)p.c_out * 256 : 0);
  if (p.out_f32) {
    compute_cast_table(batch, p.c_out, cast.data());
    kept_cast_steps(batch, p.c_out, cast.data(), p.cast);
  }
  const size_t cast_bytes = cast.size() * sizeof(float);
  void* block = nullptr;
  MLXD_CUDA(cudaMallocAsync(&block, table_bytes + cast_bytes, stream));
  unsigned char* const to = static_cast<unsigned char*>(block);
  p.samples = static_cast<const DevSample*>(block);
  p.lut = reinterpret_cast<const float*>(to + table_bytes);
  cudaError_t e = put_table(samples, to, table_bytes, stream);
  if (e == cudaSuccess) {
    e = put_table(cast.data(), to + table_bytes, cast_bytes, stream);
  }
  if (e == cudaSuccess) {
    e = launch_fused_batch(p, plan, stream);
  }
  const cudaError_t freed = cudaFreeAsync(block, stream);
  MLXD_CUDA(e);
  MLXD_CUDA(freed);
  return MLXD_OK;
}

} // namespace mlxd
