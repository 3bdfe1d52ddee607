// Host work dealt out to threads, behind entry points that C callers (ctypes among them) use: no exception leaves it.
#pragma once

#include <atomic>
#include <thread>
#include <vector>

#include "common.cuh"

namespace orca {

// work(0), ..., work(n - 1), the first on the calling thread.  A share whose thread cannot be started (a limit on
// threads or on address space) is done by the calling thread.
template <class F>
int on_threads(int n, F work, const char *who) {
  std::atomic<bool> failed(false);
  auto share = [&](int t) noexcept {
    try {
      work(t);
    } catch (...) {
      failed = true;
    }
  };
  std::vector<std::thread> pool;
  try {
    pool.reserve(n > 1 ? n - 1 : 0);
    for (int t = 1; t < n; ++t) pool.emplace_back(share, t);
  } catch (...) {
  }
  if (n > 0) share(0);
  for (int t = (int)pool.size() + 1; t < n; ++t) share(t);
  for (std::thread &t : pool) t.join();
  return failed ? set_error(ORCA_E_CAPACITY, "%s: out of host memory", who) : ORCA_OK;
}

}  // namespace orca
