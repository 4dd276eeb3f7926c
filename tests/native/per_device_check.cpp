// PerDevice: set-up runs once on each device, again after it failed, and
// every time on a device past the table.
#include <cstdio>
#include <thread>
#include <vector>

#include "per_device.hpp"

enum Err { kOk = 0, kBad = 3 };

#define CHECK(x)                                     \
  do {                                               \
    if (!(x)) return std::printf("%s\n", #x), 1;     \
  } while (0)

int main() {
  dense_b200::PerDevice devices;
  int runs[128] = {};
  auto on = [&](int dev, Err result) { return devices.once(dev, [&] { return ++runs[dev], result; }); };
  CHECK(on(0, kOk) == kOk && on(0, kBad) == kOk && runs[0] == 1);
  CHECK(on(1, kOk) == kOk && runs[1] == 1);  // a second device is set up as well
  CHECK(on(2, kBad) == kBad && on(2, kOk) == kOk && on(2, kBad) == kOk && runs[2] == 2);
  CHECK(on(63, kOk) == kOk && on(63, kOk) == kOk && runs[63] == 1);
  CHECK(on(100, kOk) == kOk && on(100, kBad) == kBad && runs[100] == 2);
  std::vector<std::thread> threads;
  for (int i = 0; i < 8; ++i) threads.emplace_back([&] { on(5, kOk); });
  for (auto& t : threads) t.join();
  CHECK(runs[5] == 1);
  return 0;
}
