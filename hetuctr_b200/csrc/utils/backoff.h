// Something that normally pays and costs when it fails: after a failure it is left alone for one use, then for two, four, ... and
// 1024 at most, until it works again.
#pragma once
#include <algorithm>
#include <cstdint>

namespace hetuCTR {

class Backoff {
 public:
  bool tryNow() {
    if (pause_ == 0) return true;
    pause_--;
    return false;
  }
  void worked() { next_ = 1; }
  void failed() {
    pause_ = next_;
    next_ = std::min<uint32_t>(2 * next_, 1024);
  }

 private:
  uint32_t pause_ = 0, next_ = 1;
};

}  // namespace hetuCTR
