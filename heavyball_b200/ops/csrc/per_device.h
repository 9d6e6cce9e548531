// Values that a launcher finds out, or settings that it makes, once for every device it launches on.  A kernel's opt-in shared
// memory size and its occupancy belong to a device: set up on the first GPU of a process only, they are missing on the second.
#pragma once

#include <mutex>
#include <unordered_map>

namespace hb {

template <class Value>
class PerDevice {
 public:
  // *out <- the value of `device`, made by `make(Value&)` the first time.  `make` returns `ok` or an error, which is passed on and
  // not remembered: the next call tries again.
  template <class Status, class Make>
  Status get(int device, Status ok, Value* out, Make make) {
    std::lock_guard<std::mutex> lock(mutex_);
    auto it = values_.find(device);
    if (it == values_.end()) {
      Value v{};
      const Status s = make(v);
      if (s != ok) return s;
      it = values_.emplace(device, v).first;
    }
    *out = it->second;
    return ok;
  }

 private:
  std::mutex mutex_;
  std::unordered_map<int, Value> values_;
};

}  // namespace hb
