// The state that csrc/flof_device.h keeps per device: exit status 0 when every
// check holds.
#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>

#include "flof_device.h"

#define CHECK(x) \
  if (!(x)) return std::printf("line %d: %s\n", __LINE__, #x), 1

int main() {
  // a value is formed once per device, whichever device asked first
  flof::PerDevice<int> v;
  std::atomic<int> formed{0};
  auto ask = [&](int d) { return v.get(d, [&] { return ++formed, 100 + d; }); };
  std::vector<std::thread> ts;
  std::atomic<int> wrong{0};
  for (int k = 0; k < 8; ++k)
    ts.emplace_back([&, k] {
      for (int r = 0; r < 100; ++r) wrong += ask(k % 3) != 100 + k % 3;
    });
  for (auto &t : ts) t.join();
  CHECK(wrong == 0);
  CHECK(formed == 3);
  CHECK(ask(1000) == 1100);  // a device beyond the table: formed each time

  // a busy device holds up its own solves, in the order of arrival, and no
  // other device's
  flof::SmShares &dev = flof::sm_shares(0);
  dev.acquire(140, 152);
  std::atomic<int> big{0}, small{0};
  std::thread a([&] {
    dev.acquire(38, 152);
    big = 1;
  });
  std::this_thread::sleep_for(std::chrono::milliseconds(100));
  std::thread b([&] {  // would fit, but came second
    dev.acquire(1, 152);
    small = 1;
  });
  flof::sm_shares(1).acquire(152, 152);  // returns at once
  flof::sm_shares(1).release(152);
  std::this_thread::sleep_for(std::chrono::milliseconds(100));
  CHECK(big == 0 && small == 0);
  dev.release(26);  // 38 free: the first exactly
  a.join();
  std::this_thread::sleep_for(std::chrono::milliseconds(100));
  CHECK(big == 1 && small == 0);
  dev.release(38);
  b.join();
  dev.release(114 + 1);
  dev.acquire(152, 152);  // all of it is back
  dev.release(152);
  return 0;
}
