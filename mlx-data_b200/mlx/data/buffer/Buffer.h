// Random-access pipeline node (mlx/data/buffer/Buffer.h:11-20).
#pragma once

#include "mlx/data/Sample.h"

namespace mlx {
namespace data {
namespace buffer {

class Buffer {
 public:
  virtual Sample get(int64_t idx) const = 0;
  virtual int64_t size() const = 0;
  // The sample get(idx) would return, when this node holds it in memory for as
  // long as it lives; nullptr otherwise.  Throws what get(idx) throws.
  virtual const Sample* peek(int64_t idx) const {
    (void)idx;
    return nullptr;
  }
  virtual ~Buffer() {}
};

} // namespace buffer
} // namespace data
} // namespace mlx
