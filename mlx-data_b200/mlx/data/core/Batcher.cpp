#include "mlx/data/core/Batcher.h"

#include <optional>
#include <stdexcept>

#include "mlx/data/core/Utils.h"

namespace mlx {
namespace data {
namespace core {

namespace {

// One entry of a sample whose images may still be programs rather than pixels.
// Samples have a handful of keys and a batch many samples, so an entry names its
// key by the string of the sample or op it comes from (both outlive the batch),
// holds its program in place, and a sample is a flat list of entries: executing
// a batch of images symbolically allocates once per sample.
struct Entry {
  const std::string* key;
  std::shared_ptr<Array> array;            // set when concrete
  std::optional<gpu::LazyImage> lazy;      // set when pending
};
using LazySample = std::vector<Entry>;

Entry* find(LazySample& s, const std::string& key) {
  for (auto& e : s) {
    if (e.key == &key || *e.key == key) {
      return &e;
    }
  }
  return nullptr;
}

bool gpu_image(const std::shared_ptr<Array>& a) {
  return a && a->type() == UInt8 && a->ndim() == 3 && a->shape(2) >= 1 && a->shape(2) <= 4 && a->size() > 0;
}

std::shared_ptr<Array> lazy_pixels(const Entry& e) {
  if (e.array) {
    return e.array;
  }
  if (e.lazy->untouched()) {
    return std::make_shared<Array>(e.lazy->source());
  }
  return e.lazy->materialise();
}

LazySample open(const Sample& raw, size_t room) {
  LazySample s;
  s.reserve(raw.size() + room);
  for (auto& kv : raw) {
    s.push_back(Entry{&kv.first, kv.second, std::nullopt});
  }
  return s;
}

void run_op(LazySample& s, const op::FusableOp& op) {
  Entry* in = find(s, op.input_key());
  if (!in) {
    throw std::runtime_error("key <" + op.input_key() + "> expected");
  }
  std::shared_ptr<Array> pixels;         // the result: an array
  std::optional<gpu::LazyImage> lazy;    // or a program
  if (!in->lazy && !gpu_image(in->array)) {
    // videos, non-uint8 arrays, token arrays, malformed images: the op decides (and throws)
    pixels = op.apply_key(in->array);
  } else {
    // the op gets a copy: when it does not join, the program it was given is still needed
    if (in->lazy) {
      lazy = in->lazy;
    } else {
      lazy.emplace(in->array);
    }
    Sample concrete_entries;
    if (op.reads_sample()) {
      for (auto& e : s) {
        if (e.array) {
          concrete_entries[*e.key] = e.array;
        }
      }
    }
    // An image that claims padding takes no further op except more padding:
    // compute it before the op gets to draw anything.
    bool joined = !(lazy->extended() && !op.extends_only()) && op.fold_in(*lazy, concrete_entries);
    if (!joined && !lazy->untouched()) {
      // the program is full: compute what we have, start a new one
      lazy.emplace(lazy_pixels(*in));
      joined = op.fold_in(*lazy, concrete_entries);
    }
    if (!joined) {
      // not an op the kernels run (padding in front, a slice of the channels): the host op on the pixels
      lazy.reset();
      pixels = op.apply_key(lazy_pixels(*in));
    }
  }
  Entry* out = find(s, op.output_key());
  if (!out) {
    s.push_back(Entry{&op.output_key(), nullptr, std::nullopt});
    out = &s.back();
  }
  out->array = std::move(pixels);
  out->lazy = std::move(lazy);
}

} // namespace

Batcher::Batcher(
    std::vector<std::shared_ptr<op::FusableOp>> ops,
    std::unordered_map<std::string, double> pad_values,
    std::unordered_map<std::string, int> batch_dims,
    std::vector<CastRequest> casts)
    : ops_(std::move(ops)),
      pad_values_(std::move(pad_values)),
      batch_dims_(std::move(batch_dims)),
      casts_(std::move(casts)),
      placement_(gpu::Runtime::get().placement()) {}

Sample Batcher::run(const std::vector<Sample>& raw) const {
  std::vector<const Sample*> at;
  at.reserve(raw.size());
  for (auto& s : raw) {
    at.push_back(&s);
  }
  return run(at);
}

Sample Batcher::run(const std::vector<const Sample*>& raw) const {
  if (raw.empty()) {
    return Sample();
  }
  // 1. symbolic execution, sample-major like a pull pipeline
  std::vector<LazySample> lazy;
  lazy.reserve(raw.size());
  for (auto* s : raw) {
    lazy.push_back(open(*s, ops_.size()));
    for (auto& op : ops_) {
      run_op(lazy.back(), *op);
    }
  }
  // 2. per key of the first sample: one batch tensor.  Casts come after the batch in
  // the chain: what they make goes in last, in their order, over a batch of that key.
  Sample out;
  std::vector<std::shared_ptr<Array>> cast_results(casts_.size());
  std::vector<Entry*> col;
  std::vector<gpu::LazyImage> made;             // programs of entries that are plain arrays, or were computed on their own
  std::vector<const gpu::LazyImage*> images;
  for (auto& first_entry : lazy.front()) {
    const std::string& key = *first_entry.key;
    col.clear();
    col.reserve(lazy.size());
    for (auto& s : lazy) {
      Entry* e = find(s, key);
      if (!e) {
        throw std::runtime_error("mergeBatch: inconsistent sample keys in batch (unknown key: <" + key + ">)");
      }
      col.push_back(e);
    }
    double pad = 0.0;
    if (auto p = pad_values_.find(key); p != pad_values_.end()) {
      pad = p->second;
    }
    const auto dim = batch_dims_.find(key);
    bool on_gpu = dim == batch_dims_.end();
    for (auto* e : col) {
      on_gpu = on_gpu && (e->lazy || gpu_image(e->array));
    }
    if (on_gpu) {
      made.clear();
      made.reserve(col.size());   // `images` points into it
      images.clear();
      images.reserve(col.size());
      bool same = true;
      for (auto* e : col) {
        if (e->lazy && e->lazy->extension_matches(pad)) {
          images.push_back(&*e->lazy);
        } else {
          // (explicit padding with another value than the batch's: that image is computed on its own first)
          made.push_back(gpu::LazyImage(e->lazy ? e->lazy->materialise() : e->array));
          images.push_back(&made.back());
        }
        same = same && images.back()->source_channels() == images.front()->source_channels() &&
            images.back()->is_gray() == images.front()->is_gray();
      }
      if (!same) {
        throw std::runtime_error("BatchShape: batched arrays expected to have consistent shapes");
      }
      bool replaced = false;
      for (size_t k = 0; k < casts_.size(); k++) {
        const CastRequest& c = casts_[k];
        if (c.ikey == key) {
          cast_results[k] = gpu::Runtime::get().batch(images, pad, &c.spec, placement_);
          replaced = replaced || c.okey.empty() || c.okey == key;
        }
      }
      if (!replaced) {
        out[key] = gpu::Runtime::get().batch(images, pad, nullptr, placement_);
      }
      continue;
    }
    std::vector<std::shared_ptr<Array>> arrs;
    arrs.reserve(col.size());
    for (auto* e : col) {
      arrs.push_back(lazy_pixels(*e));
    }
    std::shared_ptr<Array> merged =
        dim == batch_dims_.end() ? array::batch(arrs, pad) : array::batch(arrs, dim->second, pad);
    out[key] = merged;
    for (size_t k = 0; k < casts_.size(); k++) {
      if (casts_[k].ikey == key) {
        cast_results[k] = gpu::Runtime::get().cast(merged, casts_[k].spec);
      }
    }
  }
  for (size_t k = 0; k < casts_.size(); k++) {
    if (cast_results[k]) {
      out[casts_[k].okey.empty() ? casts_[k].ikey : casts_[k].okey] = cast_results[k];
    }
  }
  return out;
}

std::vector<int64_t> folded_shape(
    const std::vector<std::shared_ptr<op::FusableOp>>& ops, const Sample& raw, const std::string& key) {
  LazySample lazy = open(raw, ops.size());
  for (auto& op : ops) {
    run_op(lazy, *op);
  }
  const Entry* e = find(lazy, key);
  if (!e) {
    throw std::runtime_error("key <" + key + "> expected");
  }
  if (e->lazy) {
    return {e->lazy->height(), e->lazy->width(), e->lazy->channels()};
  }
  return e->array->shape();
}

Sample merge_batch(
    const std::vector<Sample>& samples,
    const std::unordered_map<std::string, double>& pad_values,
    const std::unordered_map<std::string, int>& batch_dims) {
  return Batcher({}, pad_values, batch_dims).run(samples);
}

} // namespace core
} // namespace data
} // namespace mlx
