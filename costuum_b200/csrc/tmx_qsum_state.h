// Which batch the buffers of the Q sums are ready for (plain C++, no CUDA).
#pragma once
#include <cstdint>

// The counters behind the partial sums start at zero for a batch and are zero
// again after it, wherever the batch's size puts them. That no longer holds
// when a buffer could not be grown (the old one is gone by then) or when a batch
// ended early with rounds launched.
struct TmxQsumState {
  int64_t n = -1;    // grains the buffers are laid out and cleared for; -1: none
  bool open = false; // rounds of a batch that has not ended may have run

  // Start of a batch's first round; returns whether rounds of a batch that
  // ended early may still run (the caller waits for them).
  bool begin() {
    const bool left = open;
    if (left) {
      n = -1;
    }
    open = true;
    return left;
  }
  void end() { open = false; }

  // grow() makes the buffers large enough, clear() zeroes the counters; both
  // return 0 or an error, after which nothing counts as laid out.
  template <class Grow, class Clear> int layout(int64_t grains, Grow grow, Clear clear) {
    if (n == grains) {
      return 0;
    }
    n = -1;
    int rc = grow();
    if (rc == 0) {
      rc = clear();
    }
    if (rc == 0) {
      n = grains;
    }
    return rc;
  }
};
