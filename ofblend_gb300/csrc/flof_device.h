// flof_device.h -- host-side state kept per device (no CUDA in here: contexts
// on several devices of one process do not share it).
#pragma once

#include <condition_variable>
#include <mutex>

namespace flof {

constexpr int MAX_DEVICES = 64;

// A value per device, formed by init() at the first request for that device;
// requests from several threads wait for it.
template <class T>
class PerDevice {
  std::once_flag once_[MAX_DEVICES];
  T value_[MAX_DEVICES] = {};

 public:
  template <class Init>
  T get(int device, Init &&init) {
    if (device < 0 || device >= MAX_DEVICES) return init();
    std::call_once(once_[device], [&] { value_[device] = init(); });
    return value_[device];
  }
};

// The SMs of one device as the resident solves in flight on it share them: at
// most one block per SM in sum, waits in the order of arrival.
class SmShares {
  std::mutex mu_;
  std::condition_variable cv_;
  int used_ = 0;
  unsigned long long next_ = 0, serving_ = 0;

 public:
  void acquire(int n, int sms) {
    std::unique_lock<std::mutex> lk(mu_);
    const unsigned long long mine = next_++;
    cv_.wait(lk, [&] { return serving_ == mine && used_ + n <= sms; });
    ++serving_;
    used_ += n;
    cv_.notify_all();
  }
  void release(int n) {
    {
      std::lock_guard<std::mutex> lk(mu_);
      used_ -= n;
    }
    cv_.notify_all();
  }
};

inline SmShares &sm_shares(int device) {
  static SmShares shares[MAX_DEVICES + 1];  // the last for any device beyond
  return shares[device >= 0 && device < MAX_DEVICES ? device : MAX_DEVICES];
}

}  // namespace flof
