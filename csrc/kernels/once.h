// Work that is needed once per (device, slot), from any thread.
#pragma once
#include <atomic>
#include <mutex>

namespace orinfer {

template <int DEVICES, int SLOTS>
class OncePerSlot {
 public:
  // 0 once `set` has returned 0 for this pair, in this call or an earlier one; otherwise what it
  // returned, and the next caller tries again.  Nobody gets a 0 before `set` is through.  Outside
  // the table it runs on every call.
  template <class Set>
  int run(int device, int slot, Set&& set) {
    if (device < 0 || device >= DEVICES || slot < 0 || slot >= SLOTS) return set();
    std::atomic<bool>& done = done_[device][slot];
    if (done.load(std::memory_order_acquire)) return 0;
    std::lock_guard<std::mutex> lock(mutex_);
    if (done.load(std::memory_order_relaxed)) return 0;
    const int r = set();
    if (r == 0) done.store(true, std::memory_order_release);
    return r;
  }

 private:
  std::mutex mutex_;
  std::atomic<bool> done_[DEVICES][SLOTS] = {};
};

}  // namespace orinfer
