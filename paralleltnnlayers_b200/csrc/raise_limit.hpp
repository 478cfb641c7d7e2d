// A limit that host threads raise (dynamic shared memory of a kernel).
#pragma once

#include <atomic>
#include <mutex>

namespace b200cp {

inline std::mutex& limit_mutex() {   // one for all limits (a template's own would be one per `set`)
  static std::mutex mu;
  return mu;
}
// Raises a limit to at least `value` with `set`, once per value that exceeds the recorded one.  The record and the limit change
// together: two threads that raise it at the same time would else leave the smaller limit under the larger record.
template <typename Set>
auto raise_limit(std::atomic<int>& record, int value, Set set) -> decltype(set(value)) {
  using Error = decltype(set(value));
  if (record.load(std::memory_order_acquire) >= value) return Error{};
  std::lock_guard<std::mutex> lk(limit_mutex());
  if (record.load(std::memory_order_relaxed) >= value) return Error{};
  const Error e = set(value);
  if (e == Error{}) record.store(value, std::memory_order_release);
  return e;
}

}  // namespace b200cp
