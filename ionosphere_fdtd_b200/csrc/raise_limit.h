// A kernel function's limit that is only ever raised, by any of the host's threads.
#pragma once

#include <stddef.h>

#include <mutex>

namespace ifdtd {

inline std::mutex g_limit_lock;

// Raise a limit to `bytes` unless it is that high already.  get(&now) reads it and
// set(bytes) writes it; both return an error code, 0 for success.  Reading and raising
// are one step to other threads: without the lock the thread that needs less could
// write last, and a caller that asks once would never raise it again.
template <typename Get, typename Set>
auto raise_limit(size_t bytes, Get get, Set set) -> decltype(set(bytes)) {
  std::lock_guard<std::mutex> hold(g_limit_lock);
  size_t now = 0;
  const auto e = get(&now);
  if (static_cast<int>(e) != 0 || now >= bytes) return e;
  return set(bytes);
}

}  // namespace ifdtd
