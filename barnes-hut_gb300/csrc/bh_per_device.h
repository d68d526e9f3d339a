// A positive number asked once of each device ordinal and kept.  Threads that
// ask for the first time at once store the same answer.
#pragma once

#include <atomic>

namespace bh {

class PerDevice {
  public:
    // `ask()` for `dev`'s answer, below 1 where it cannot be had (not kept);
    // then, and for ordinals outside the table, `otherwise`.
    template <typename F>
    int get(int dev, int otherwise, F ask)
    {
        const bool kept = dev >= 0 && dev < kMaxDevices;
        int v = kept ? cache_[dev].load(std::memory_order_relaxed) : 0;
        if (v > 0) return v;
        v = ask();
        if (v < 1) return otherwise;
        if (kept) cache_[dev].store(v, std::memory_order_relaxed);
        return v;
    }

  private:
    static constexpr int kMaxDevices = 64;
    std::atomic<int> cache_[kMaxDevices] = {};
};

}  // namespace bh
