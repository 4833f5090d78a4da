// DeviceOnce (csrc/device_once.h) on the CPU: set once a device, after a
// failure again, beyond the devices it remembers each time.
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>

#include "device_once.h"

#define CHECK(x)                                     \
  do {                                               \
    if (!(x)) {                                      \
      std::printf("line %d: %s\n", __LINE__, #x);    \
      std::exit(1);                                  \
    }                                                \
  } while (0)

int main() {
  nn::DeviceOnce once;
  int calls[70] = {};
  auto run = [&](int d, int result) { return once(d, 0, [&] { return ++calls[d], result; }); };
  CHECK(run(0, 0) == 0 && run(0, 7) == 0 && calls[0] == 1);   // remembered
  CHECK(run(1, 0) == 0 && calls[1] == 1);                     // another device is set for itself
  CHECK(run(2, 5) == 5 && run(2, 0) == 0 && calls[2] == 2);   // a failure is not kept
  CHECK(run(2, 5) == 0 && calls[2] == 2);
  CHECK(run(63, 0) == 0 && run(63, 9) == 0 && calls[63] == 1);
  CHECK(run(64, 0) == 0 && run(64, 3) == 3 && calls[64] == 2);
  nn::DeviceOnce other;                                       // a kernel's bits are its own
  CHECK(other(0, 0, [] { return 4; }) == 4);
  nn::DeviceOnce shared;
  std::vector<std::thread> threads;
  std::atomic<int> sets{0};
  for (int t = 0; t < 8; ++t)
    threads.emplace_back([&, t] {
      for (int k = 0; k < 1000; ++k) shared(t % 4, 0, [&] { return ++sets, 0; });
    });
  for (auto& t : threads) t.join();
  CHECK(sets >= 4 && sets <= 8);
  std::puts("ok");
}
