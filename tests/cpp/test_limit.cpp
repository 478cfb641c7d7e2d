// Two threads that raise a kernel's shared-memory limit at the same time: the limit that is left is the one on record.
// Thread A (100) is held inside its set call until thread B (50) has come back, or for a fifth of a second.
#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>

#include "raise_limit.hpp"

int main() {
  std::atomic<int> record{0};
  std::atomic<bool> inside{false}, back{false};
  int limit = 0;
  std::thread a([&] {
    b200cp::raise_limit(record, 100, [&](int n) {
      limit = n;
      inside = true;
      const auto end = std::chrono::steady_clock::now() + std::chrono::milliseconds(200);
      while (!back && std::chrono::steady_clock::now() < end) std::this_thread::yield();
      return 0;
    });
  });
  std::thread b([&] {
    while (!inside) std::this_thread::yield();
    b200cp::raise_limit(record, 50, [&](int n) { limit = n; return 0; });
    back = true;
  });
  a.join();
  b.join();
  int refused = 0;
  const int e = b200cp::raise_limit(record, 200, [&](int) { ++refused; return 1; });
  std::printf("record %d limit %d refused %d\n", record.load(), limit, refused);
  return record == 100 && limit == 100 && refused == 1 && e == 1 ? 0 : 1;
}
