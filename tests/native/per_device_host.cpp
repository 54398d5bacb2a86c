// Set-up per device (csrc/per_device.h): every device gets its own, once, also
// from several threads; a set-up that throws is not taken for done.
#include <cstdio>
#include <thread>
#include <vector>

#include "per_device.h"

using namespace bem2d_gpu;

int main() {
  static PerDeviceOnce once;
  static PerDevice<int> width(16);
  std::atomic<int> calls[70] = {};
  std::vector<std::thread> ts;
  for (int t = 0; t < 8; ++t)
    ts.emplace_back([&, t] {
      for (int i = 0; i < 1000; ++i) {
        const int dev = (i + t) % 4;
        once(dev, [&] {
          ++calls[dev];
          width[dev] = 8 + dev;
        });
        if (width[dev] != 8 + dev) calls[69] = 1;  // seen before it was set
      }
    });
  for (auto& t : ts) t.join();
  bool ok = calls[69] == 0;
  for (int d = 0; d < 4; ++d) ok = ok && calls[d] == 1;
  ok = ok && width[4] == 16;  // untouched
  // a set-up that fails by an exception runs again
  int tries = 0;
  for (int i = 0; i < 3; ++i) {
    try {
      once(5, [&] {
        if (++tries == 1) throw 1;
      });
    } catch (int) {
    }
  }
  ok = ok && tries == 2;
  // beyond the table: every time, no write outside it
  int far = 0;
  for (int i = 0; i < 3; ++i) once(kMaxDevices, [&] { ++far; });
  once(-1, [&] { ++far; });
  ok = ok && far == 4;
  width[kMaxDevices + 5] = 3;
  ok = ok && width[0] == 8;
  std::puts(ok ? "ok" : "FAILED");
  return ok ? 0 : 1;
}
