// Values that are computed once per device and then only read.
#pragma once

#include <map>
#include <memory>
#include <mutex>

namespace ptd {

template <class T>
class PerDevice {
 public:
  // The device's value; the first caller's `fill` computes it while others
  // wait, so nobody reads one in the making. References stay valid.
  template <class Fill>
  const T &get(int device, Fill &&fill) {
    std::lock_guard<std::mutex> lock(m_);
    std::unique_ptr<const T> &p = values_[device];
    if (!p) {
      auto t = std::make_unique<T>();
      fill(*t);
      p = std::move(t);
    }
    return *p;
  }

 private:
  std::mutex m_;
  std::map<int, std::unique_ptr<const T>> values_;
};

}  // namespace ptd
