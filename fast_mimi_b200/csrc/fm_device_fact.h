// A number that belongs to a device, asked for once and then kept.  Host code only.
#pragma once

#include <atomic>

namespace fm {

// Any thread may ask; what a question that failed would have said is not kept.  For objects of static storage duration.
class DeviceFact {
 public:
  // ask() -> the number, or a negative one where it could not be found out, which get() hands on.
  template <typename Ask>
  int get(int device, Ask ask) {
    if (device < 0 || device >= kDevices) return ask();
    const int kept = known_[device].load(std::memory_order_relaxed);
    if (kept != 0) return kept - 1;
    const int answer = ask();
    if (answer >= 0) known_[device].store(answer + 1, std::memory_order_relaxed);
    return answer;
  }

 private:
  static constexpr int kDevices = 64;
  std::atomic<int> known_[kDevices] = {};      // the number + 1; 0: not known
};

}  // namespace fm
