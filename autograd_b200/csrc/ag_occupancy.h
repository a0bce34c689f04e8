// Answers of an occupancy query, kept per kernel and device.  Host C++ only.
#pragma once

#include <atomic>
#include <cstddef>
#include <cstdint>

// How many CTAs of one kernel an SM holds, by threads and dynamic shared memory of the launch.  Any number of threads
// may ask at once: an answer is a single word, and two threads that both miss store the same answer.  A program uses
// few row lengths per kernel, so a handful of answers is kept; with one, two row lengths in turn would pay the query
// at every launch (several microseconds against a launch of about two).  A static object of this type is zero: empty.
class AgOccupancy {
 public:
  static constexpr int kSlots = 8;

  // query() -> CTAs per SM; what is below 1 (an error) is handed through and not kept.
  template <typename Query>
  int get(int threads, size_t smem, Query query) {
    const uint64_t key = ((uint64_t)smem << 12 | (uint64_t)threads) << 8;
    int free = -1;
    for (int i = 0; i < kSlots; ++i) {
      const uint64_t word = slot_[i].load(std::memory_order_relaxed);
      if (word >> 8 == key >> 8 && (word & 255u)) return (int)(word & 255u);
      if (!word && free < 0) free = i;
    }
    const int occ = query();
    if (occ < 1) return occ;
    if (free < 0) free = (int)((key >> 8) * 0x9E3779B97F4A7C15ull >> 61);
    slot_[free].store(key | (uint64_t)(occ < 255 ? occ : 255), std::memory_order_relaxed);
    return occ;
  }

 private:
  std::atomic<uint64_t> slot_[kSlots];
};
