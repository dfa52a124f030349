// host_threads.h -- host work on several threads.
#pragma once
#include <functional>
#include <system_error>
#include <thread>
#include <vector>

namespace sf {
// run worker on this thread and up to n - 1 others; fewer where the system gives no more
// (an exception out of a C entry point, or past a pool of running threads, ends the process)
template <typename F>
void on_threads(int n, F &worker) {
  std::vector<std::thread> pool;
  pool.reserve(n > 1 ? n - 1 : 0);
  try {
    while ((int)pool.size() + 1 < n) pool.emplace_back(std::ref(worker));
  } catch (const std::system_error &) {
  }
  worker();
  for (std::thread &t : pool) t.join();
}
}  // namespace sf
