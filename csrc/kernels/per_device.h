// State that belongs to a device and is made once on each: kernel attributes and what follows from them. A process may drive several devices
// from several threads.
#pragma once
#include <mutex>

namespace skein {

constexpr int MAX_DEVICES = 64;

// value of the device, made by the first caller there whose `make` gives more than 0; what it gives otherwise (an error) is returned and tried again
class PerDevice {
 public:
  template <typename Make>
  int get(int device, Make make) {
    if (device < 0 || device >= MAX_DEVICES) return -4;
    std::lock_guard<std::mutex> lock(mu_);
    if (value_[device] <= 0) value_[device] = make();
    return value_[device];
  }

 private:
  std::mutex mu_;
  int value_[MAX_DEVICES] = {};
};

}  // namespace skein
