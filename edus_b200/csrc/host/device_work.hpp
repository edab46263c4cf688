// device_work.hpp — how many calls of this process have work on a device.
//
// A whole run in one launch (loop.cu) holds its SMs until it ends, its blocks
// waiting for one another: beside other work it would wait for room, or keep the others out
// for a quarter of a second at a time. Its caller takes that form only where nothing
// else of the process is at work on the device, and the captured launch per stage, whose
// small kernels interleave, where something is. One count per device, held by each
// call for its duration (an asynchronous run: until it has ended), is all that is shared;
// work that begins later does not change a run that has chosen.
#pragma once
#include <atomic>

namespace edus {

class DeviceWork {
 public:
  explicit DeviceWork(int device) : n_(device >= 0 && device < kDevices ? &count_[device] : nullptr) {
    alone_ = n_ && n_->fetch_add(1) == 0;
  }
  ~DeviceWork() {
    if (n_) n_->fetch_sub(1);
  }
  DeviceWork(const DeviceWork&) = delete;
  DeviceWork& operator=(const DeviceWork&) = delete;
  // nothing else was at work when this began
  bool alone() const { return alone_; }

 private:
  static constexpr int kDevices = 64;
  inline static std::atomic<int> count_[kDevices] = {};
  std::atomic<int>* n_;
  bool alone_ = false;
};

}  // namespace edus
