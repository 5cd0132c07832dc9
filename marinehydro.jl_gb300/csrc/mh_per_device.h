// mh_per_device.h -- values that belong to one CUDA device of the process (occupancy tables, SM
// counts; the function attributes set along with them).  No CUDA in here.
#pragma once

#include <map>
#include <mutex>

namespace mh {

// get(device, make): the value made by make() at the first call for `device`, which has to be the
// current one then; any number of threads
template <typename T>
class PerDevice {
 public:
  template <typename Make>
  const T& get(int device, Make make) {
    std::lock_guard<std::mutex> lock(mutex_);
    auto it = values_.find(device);
    if (it == values_.end()) it = values_.emplace(device, make()).first;
    return it->second;  // a map's elements stay where they are
  }

 private:
  std::mutex mutex_;
  std::map<int, T> values_;
};

}  // namespace mh
