// Work shared by a few host threads, of which any number may not come to be.
#pragma once
#include <system_error>
#include <thread>
#include <vector>

namespace mrl {

// Runs work(0) on the calling thread and work(1) to work(n - 1) on threads of their own, as far as the system
// lets them start: every call of `work` has to go on until nothing is left to do.
template <class Work>
void on_threads(int n, Work work) {
  std::vector<std::thread> pool;
  try {
    pool.reserve(n > 0 ? (size_t)n : 0);
    for (int t = 1; t < n; t++) pool.emplace_back(work, t);
  } catch (const std::system_error&) {   // no more threads: those there are do it all
  }
  work(0);
  for (std::thread& th : pool) th.join();
}

}  // namespace mrl
