// loop_gate.h -- keeps cooperative launches away from serving loops on one
// device.  Plain C++, so that the rule can be run without a device.
#pragma once

#include <mutex>

namespace sp {

// A cooperative launch needs its SMs at once, and a serving loop holds them for
// as long as requests come: a cooperative launch behind a loop would wait as
// long.  So a loop counts from before it is launched, a cooperative launch is
// made only while none counts, and a loop is launched behind the cooperative
// launches made before it (the caller's event).
class LoopGate {
 public:
  // launch() a loop, returning 0 if it is on its way
  template <typename F>
  int start_loop(const F &launch) {
    std::lock_guard<std::mutex> lk(mu_);
    const int rc = launch();
    if (!rc) loops_++;
    return rc;
  }
  void stop_loop() {
    std::lock_guard<std::mutex> lk(mu_);
    loops_--;
  }
  // launch() unless a loop counts; *taken: whether it was called
  template <typename F>
  int launch_alone(const F &launch, bool *taken) {
    std::lock_guard<std::mutex> lk(mu_);
    *taken = loops_ == 0;
    return *taken ? launch() : 0;
  }

 private:
  std::mutex mu_;
  int loops_ = 0;
};

}  // namespace sp
