// Work on the trees of a forest that is being loaded, on a few host threads.
#pragma once

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <exception>
#include <system_error>
#include <thread>
#include <vector>

namespace b2fil {

// Threads that work of about 50 ns and more on each of so many nodes is worth.  Smaller forests gain 0.3 ms at
// most (300 trees of depth 6: 3.1 ms on two threads, 3.4 on one), less than a thread that gets its turn late costs.
inline int pack_threads(int64_t n_nodes, int n_trees)
{
  const int hw = static_cast<int>(std::thread::hardware_concurrency());
  return n_nodes < 100000 ? 1 : std::max(1, std::min({hw, 16, n_trees}));
}

// fn(t) for every tree, on a few threads.  What fn throws is thrown again here.
template <typename F>
void for_each_tree(int n_trees, int n_threads, F&& fn)
{
  std::atomic<int> next{0};
  std::atomic<bool> failed{false};
  std::exception_ptr error;
  auto work = [&] {
    try {
      for (int t; !failed.load() && (t = next.fetch_add(1)) < n_trees;) fn(t);
    } catch (...) {
      if (!failed.exchange(true)) error = std::current_exception();
    }
  };
  std::vector<std::thread> threads;
  threads.reserve(n_threads);
  try {
    for (int i = 1; i < n_threads; ++i) threads.emplace_back(work);
  } catch (const std::system_error&) {
    // fewer threads then
  }
  work();
  for (std::thread& t : threads) t.join();
  if (error) std::rethrow_exception(error);
}

}  // namespace b2fil
