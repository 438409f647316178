// A set-up that CUDA keeps for each device (a kernel's shared-memory opt-in),
// done once per device and process.
#pragma once
#include <atomic>

namespace hobak {

class OncePerDevice {
 public:
  // setUp() returns 0 on success; it runs again on a device where it failed.
  // Batches are created and stepped from several host threads: two of them may
  // both run it, which these set-ups allow.
  template <typename SetUp>
  int operator()(int device, SetUp setUp) {
    const bool known = device >= 0 && device < kDevices;
    if (known && done_[device].load()) return 0;
    const int rc = setUp();
    if (rc == 0 && known) done_[device].store(true);
    return rc;
  }

 private:
  static constexpr int kDevices = 64;  // past them it runs each time
  std::atomic<bool> done_[kDevices] = {};
};

}  // namespace hobak
