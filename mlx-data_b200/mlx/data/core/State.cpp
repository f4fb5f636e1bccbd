#include "mlx/data/core/State.h"

#include <atomic>
#include <mutex>

namespace mlx {
namespace data {
namespace core {

namespace {
State& process_state() {
  static State s;
  return s;
}
std::mutex& process_mutex() {
  static std::mutex m;
  return m;
}

// The process's version, for threads to see without the lock whether they have it.
std::atomic<int64_t> current_version{0};

const std::shared_ptr<State>& mine() {
  static thread_local std::shared_ptr<State> state;
  if (!state || state->version != current_version.load(std::memory_order_acquire)) {
    std::lock_guard<std::mutex> g(process_mutex());
    state = std::make_shared<State>(process_state());
  }
  return state;
}
} // namespace

void set_state(int64_t seed) {
  std::lock_guard<std::mutex> g(process_mutex());
  State& s = process_state();
  s.randomGenerator = std::mt19937(seed);
  s.version++;
  current_version.store(s.version, std::memory_order_release);
}

std::shared_ptr<State> get_state() {
  return mine();
}

State& thread_state() {
  return *mine();
}

} // namespace core
} // namespace data
} // namespace mlx
