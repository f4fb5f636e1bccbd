#include "mlx/data/core/Batcher.h"

#include <stdexcept>

#include "mlx/data/core/Utils.h"

namespace mlx {
namespace data {
namespace core {

namespace {

// One entry of a sample whose images may still be programs rather than pixels.
// Samples have a handful of keys and a batch many samples, and on small images this
// work is what a batch takes.  So an entry names its key by the string of the sample or op
// it comes from and the sample's own array by its place there (all of them outlive the
// batch); the entries of all samples lie in one vector, their programs in another.
struct Entry {
  const std::string* key;
  const std::shared_ptr<Array>* held;      // the sample's array, where the entry is still that
  std::shared_ptr<Array> made;             // an op's array
  gpu::LazyImage* lazy;                    // set when pending

  const std::shared_ptr<Array>& array() const { return held ? *held : made; }
  bool concrete() const { return !lazy; }
};

// The entries of one sample: the last ones made, as long as it is being run.
struct LazySample {
  Entry* first;
  size_t count;
};

// Programs of a batch; they stay where they are.
class Programs {
 public:
  explicit Programs(size_t samples) : room_(samples) {}

  gpu::LazyImage* add(const gpu::LazyImage& program) {
    if (blocks_.empty() || blocks_.back().size() == blocks_.back().capacity()) {
      blocks_.emplace_back();
      blocks_.back().reserve(room_);
    }
    blocks_.back().push_back(program);
    return &blocks_.back().back();
  }

 private:
  size_t room_;
  std::vector<std::vector<gpu::LazyImage>> blocks_;
};

// The array as a program's source, without a share in it: whoever holds it outlives the
// batch, and programs are copied without counting.
std::shared_ptr<const Array> unowned(const std::shared_ptr<Array>& a) {
  return std::shared_ptr<const Array>(std::shared_ptr<const void>(), a.get());
}

Entry* find(const LazySample& s, const std::string& key) {
  for (size_t i = 0; i < s.count; i++) {
    Entry& e = s.first[i];
    if (e.key == &key || *e.key == key) {
      return &e;
    }
  }
  return nullptr;
}

bool gpu_image(const std::shared_ptr<Array>& a) {
  if (!a || a->type() != UInt8) {
    return false;
  }
  const std::vector<int64_t>& shape = a->shape();
  return shape.size() == 3 && shape[2] >= 1 && shape[2] <= 4 && shape[0] > 0 && shape[1] > 0;
}

std::shared_ptr<Array> lazy_pixels(const Entry& e) {
  if (e.concrete()) {
    return e.array();
  }
  if (e.lazy->untouched()) {
    return std::make_shared<Array>(e.lazy->source());
  }
  return e.lazy->materialise();
}

// Entries of `raw` behind the others in `all`, which has room for them and for a new one
// per op.
LazySample open(const Sample& raw, std::vector<Entry>& all) {
  const size_t at = all.size();
  for (auto& kv : raw) {
    all.push_back(Entry{&kv.first, &kv.second, nullptr, nullptr});
  }
  return LazySample{all.data() + at, raw.size()};
}

// A program of its own array, which lives as long as the entry it goes into.
void start_program(Entry& e, std::shared_ptr<Array> pixels, Programs& programs) {
  e.made = std::move(pixels);
  e.held = nullptr;
  e.lazy = programs.add(gpu::LazyImage(unowned(e.made)));
}

void run_op(LazySample& s, const Sample& raw, const op::FusableOp& op, std::vector<Entry>& all, Programs& programs) {
  Entry* in = find(s, op.input_key());
  if (!in) {
    throw std::runtime_error("key <" + op.input_key() + "> expected");
  }
  // the entry that takes the result; a new one is the sample's last
  Entry* out = in;
  if (&op.output_key() != &op.input_key()) {
    out = find(s, op.output_key());
    if (!out) {
      all.push_back(Entry{&op.output_key(), nullptr, nullptr, nullptr});
      s.count++;
      out = &s.first[s.count - 1];
    }
  }
  auto set_pixels = [&](std::shared_ptr<Array> pixels) {
    out->lazy = nullptr;
    out->held = nullptr;
    out->made = std::move(pixels);
  };
  if (!in->lazy && !gpu_image(in->array())) {
    // videos, non-uint8 arrays, token arrays, malformed images: the op decides (and throws)
    set_pixels(op.apply_key(in->array()));
    return;
  }
  Sample concrete_entries;
  const Sample* entries = &concrete_entries;
  if (op.reads_sample()) {
    // (the sample itself, as long as what the op reads is as it came)
    const std::string* reads = op.reads_key();
    const Entry* read = reads ? find(s, *reads) : nullptr;
    if (read && read->held && !read->lazy) {
      entries = &raw;
    } else {
      for (size_t i = 0; i < s.count; i++) {
        const Entry& e = s.first[i];
        if (e.concrete() && e.array()) {
          concrete_entries[*e.key] = e.array();
        }
      }
    }
  }
  // A program is recorded in place where the result replaces it: an op that does not
  // join leaves it as it is.
  std::shared_ptr<Array> keep = out == in ? nullptr : in->made;
  if (!in->lazy) {
    gpu::LazyImage* started = programs.add(gpu::LazyImage(unowned(in->array())));
    if (out == in) {
      in->lazy = started;
    } else {
      out->lazy = started;
      out->held = in->held;
      out->made = std::move(keep);
    }
  } else if (out != in) {
    out->lazy = programs.add(*in->lazy);
    out->held = in->held;
    out->made = std::move(keep);
  }
  // An image that claims padding takes no further op except more padding:
  // compute it before the op gets to draw anything.
  bool joined = !(out->lazy->extended() && !op.extends_only()) && op.fold_in(*out->lazy, *entries);
  if (!joined && !out->lazy->untouched()) {
    // the program is full: compute what we have, start a new one
    start_program(*out, lazy_pixels(*out), programs);
    joined = op.fold_in(*out->lazy, *entries);
  }
  if (!joined) {
    // not an op the kernels run (padding in front, a slice of the channels): the host op on the pixels
    set_pixels(op.apply_key(lazy_pixels(*out)));
  }
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
  size_t entries = 0;
  for (auto* s : raw) {
    entries += s->size() + ops_.size();
  }
  std::vector<Entry> all;
  all.reserve(entries);   // never grows beyond it: samples point into it
  Programs programs(raw.size());
  for (auto* s : raw) {
    lazy.push_back(open(*s, all));
    for (auto& op : ops_) {
      run_op(lazy.back(), *s, *op, all, programs);
    }
  }
  // 2. per key of the first sample: one batch tensor.  Casts come after the batch in
  // the chain: what they make goes in last, in their order, over a batch of that key.
  Sample out;
  std::vector<std::shared_ptr<Array>> cast_results(casts_.size());
  std::vector<Entry*> col;
  std::vector<std::shared_ptr<Array>> computed;   // images computed on their own
  std::vector<const gpu::LazyImage*> images;
  for (size_t k = 0; k < lazy.front().count; k++) {
    const size_t place = k;
    const std::string& key = *lazy.front().first[k].key;
    col.clear();
    col.reserve(lazy.size());
    for (auto& s : lazy) {
      // (most often where the first sample has it)
      Entry* e = place < s.count && *s.first[place].key == key ? &s.first[place] : find(s, key);
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
      on_gpu = on_gpu && (e->lazy || gpu_image(e->array()));
    }
    if (on_gpu) {
      computed.clear();
      images.clear();
      images.reserve(col.size());
      bool same = true;
      for (auto* e : col) {
        if (e->lazy && e->lazy->extension_matches(pad)) {
          images.push_back(e->lazy);
        } else if (e->lazy) {
          // (explicit padding with another value than the batch's: that image is computed on its own first)
          computed.push_back(e->lazy->materialise());
          images.push_back(programs.add(gpu::LazyImage(unowned(computed.back()))));
        } else {
          images.push_back(programs.add(gpu::LazyImage(unowned(e->array()))));
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
  std::vector<Entry> all;
  all.reserve(raw.size() + ops.size());
  Programs programs(1);
  LazySample lazy = open(raw, all);
  for (auto& op : ops) {
    run_op(lazy, raw, *op, all, programs);
  }
  const Entry* e = find(lazy, key);
  if (!e) {
    throw std::runtime_error("key <" + key + "> expected");
  }
  if (e->lazy) {
    return {e->lazy->height(), e->lazy->width(), e->lazy->channels()};
  }
  return e->array()->shape();
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
