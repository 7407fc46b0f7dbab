// Values that belong to one device of the process: kernel attributes set
// there (a shared-memory opt-in is part of a device's context, so setting it
// on one device leaves the others without it), SM counts, resident grids.
#pragma once

#include <map>
#include <mutex>
#include <utility>

namespace silkb {

template <class T>
class PerDevice {
 public:
  // The value of device `dev`, from make() on the first call for it; a make()
  // that throws stores nothing and is run again by the next call.  Safe from
  // several threads; the reference stays valid.
  template <class Make>
  const T& get(int dev, Make&& make) {
    std::lock_guard<std::mutex> lock(mutex_);
    auto it = values_.find(dev);
    if (it == values_.end()) it = values_.emplace(dev, std::forward<Make>(make)()).first;
    return it->second;
  }

 private:
  std::mutex mutex_;
  std::map<int, T> values_;
};

}  // namespace silkb
