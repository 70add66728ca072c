// Things put aside for reuse, per device (plain C++, no CUDA).
#pragma once
#include <mutex>

// At most Keep of them per device, on the first Devices devices; the last one
// put aside is taken first. Nothing is allocated and nothing needs a destructor,
// so that a process may end with some left.
template <class T, int Keep, int Devices> class TmxIdle {
public:
  // false: no place, the caller keeps it
  bool put(int device, const T &t) {
    if (device < 0 || device >= Devices) {
      return false;
    }
    std::lock_guard<std::mutex> lock(mutex_);
    if (count_[device] == Keep) {
      return false;
    }
    item_[device][count_[device]++] = t;
    return true;
  }
  // false: none left
  bool take(int device, T &t) {
    if (device < 0 || device >= Devices) {
      return false;
    }
    std::lock_guard<std::mutex> lock(mutex_);
    if (count_[device] == 0) {
      return false;
    }
    t = item_[device][--count_[device]];
    return true;
  }

private:
  std::mutex mutex_;
  T item_[Devices][Keep] = {};
  int count_[Devices] = {};
};
