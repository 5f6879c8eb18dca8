// Once a device: a second device is set too, a failure is tried again, unknown devices are set every time.
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>

#include "per_device.h"

static void require(bool ok, const char* what) {
  if (!ok) {
    std::printf("failed: %s\n", what);
    std::exit(1);
  }
}

int main() {
  PerDevice p;
  int calls = 0;
  auto ok = [&] { ++calls; return 0; };
  require(p.once(0, ok) == 0 && p.once(0, ok) == 0 && calls == 1, "once a device");
  require(p.once(1, ok) == 0 && calls == 2 && p.once(63, ok) == 0 && calls == 3, "a second device");
  require(p.once(2, [&] { ++calls; return 7; }) == 7 && p.once(2, ok) == 0 && calls == 5 && p.once(2, ok) == 0 && calls == 5, "a failure is tried again");
  require(p.once(64, ok) == 0 && p.once(64, ok) == 0 && p.once(-1, ok) == 0 && calls == 8, "devices without a place are set each time");
  PerDevice q;
  std::atomic<int> sets{0};
  std::vector<std::thread> threads;
  for (int i = 0; i < 8; ++i)
    threads.emplace_back([&, i] {
      for (int k = 0; k < 1000; ++k) q.once(i % 4, [&] { ++sets; return 0; });
    });
  for (auto& t : threads) t.join();
  require(sets >= 4 && sets <= 8, "threads");
  std::printf("ok\n");
  return 0;
}
