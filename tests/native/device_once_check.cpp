// OncePerDevice: once for each device whatever the thread, again after a
// failure, every time beyond the table.
#include <atomic>
#include <cstdio>
#include <stdexcept>
#include <thread>
#include <vector>

#include "ek_device.h"

int main() {
  ek::OncePerDevice once;
  std::atomic<int> n[2] = {{0}, {0}};
  std::vector<std::thread> t;
  for (int k = 0; k < 8; ++k)
    t.emplace_back([&, k] {
      for (int r = 0; r < 100; ++r) once((k + r) & 1, [&] { ++n[(k + r) & 1]; });
    });
  for (std::thread &x : t) x.join();
  int tries = 0;
  for (int k = 0; k < 3; ++k) try {
      once(2, [&] {
        if (++tries == 1) throw std::runtime_error("first");
      });
    } catch (const std::runtime_error &) {
    }
  int far = 0;
  for (int k = 0; k < 3; ++k) once(1 << 20, [&] { ++far; });
  std::printf("%d %d %d %d\n", n[0].load(), n[1].load(), tries, far);
  return !(n[0] == 1 && n[1] == 1 && tries == 2 && far == 3);
}
