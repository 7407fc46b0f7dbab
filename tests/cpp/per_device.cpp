// PerDevice (csrc/per_device.hpp) without a GPU: one value for each device,
// made once there, also when several threads ask at once, and made again
// after a make that threw.
#include <atomic>
#include <cstdio>
#include <stdexcept>
#include <thread>
#include <vector>

#include "per_device.hpp"

int main() {
  silkb::PerDevice<int> value;
  std::atomic<int> made[3] = {};
  std::atomic<bool> wrong{false};
  std::vector<std::thread> pool;
  for (int t = 0; t < 8; ++t)
    pool.emplace_back([&] {
      for (int k = 0; k < 3000; ++k) {
        const int dev = k % 3;
        if (value.get(dev, [&, dev] { return ++made[dev], 10 + dev; }) != 10 + dev) wrong = true;
      }
    });
  for (auto& t : pool) t.join();
  if (wrong || made[0] != 1 || made[1] != 1 || made[2] != 1) return 1;
  bool threw = false;
  try {
    value.get(7, []() -> int { throw std::runtime_error("not there"); });
  } catch (const std::runtime_error&) {
    threw = true;
  }
  if (!threw || value.get(7, [] { return 5; }) != 5) return 2;
  std::puts("ok");
  return 0;
}
