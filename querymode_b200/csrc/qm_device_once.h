// qm_device_once.h — what is set up once per device.
#pragma once

#include <map>
#include <mutex>

// Kernel attributes belong to one device: raised where a kernel first runs,
// they stay at their defaults on every other.  set(device) runs once for each
// device, and again after a failure (a non-zero error).
struct qm_kernel_setup {
  int error;
  int per_sm;  // blocks per SM
};

class qm_device_once {
  std::mutex mu;
  std::map<int, qm_kernel_setup> done;

 public:
  template <class SET>
  qm_kernel_setup get(int device, SET set) {
    std::lock_guard<std::mutex> lk(mu);
    const auto it = done.find(device);
    if (it != done.end()) return it->second;
    const qm_kernel_setup r = set();
    if (r.error == 0) done[device] = r;
    return r;
  }
};
