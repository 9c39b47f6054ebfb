// Test-only: the copy threads of cuml_b200/csrc/host_pool.hpp without a GPU.
#include <sys/wait.h>
#include <unistd.h>

#include <cstring>

#include "../../cuml_b200/csrc/host_pool.hpp"

using namespace b2fil;

namespace {
// A job of n items that counts how often each was done, with or without a watcher.
bool job_is_done_once(size_t n, bool watched)
{
  std::vector<std::atomic<int>> count(n);
  std::atomic<size_t> done{0};
  auto item = [&](size_t i) {
    count[i].fetch_add(1);
    done.fetch_add(1);
  };
  bool seen_all = false;
  if (watched) {
    CopyPool::get(4).run(n, item, [&] { return seen_all = done.load() == n; });
  } else {
    CopyPool::get(4).run(n, item);
  }
  for (auto& c : count)
    if (c.load() != 1) return false;
  return !watched || seen_all;
}
bool jobs(int rounds, size_t most)
{
  bool ok = true;
  for (int k = 0; k < rounds; ++k) ok = job_is_done_once((k * 37) % most, k & 1) && ok;
  return ok;
}
}  // namespace

extern "C" {
// Jobs of 0 to `most` items from `threads` threads at a time: every item exactly once.
int pool_check_jobs(int threads, int rounds, int most)
{
  std::atomic<int> bad{0};
  std::vector<std::thread> t;
  for (int i = 0; i < threads; ++i)
    t.emplace_back([&] { if (!jobs(rounds, static_cast<size_t>(most))) bad.fetch_add(1); });
  for (auto& x : t) x.join();
  return bad.load();
}
// The same in a forked child, which has no copy threads: 0 when it finished its jobs.
int pool_check_fork(int rounds)
{
  if (!jobs(3, 100)) return 1;
  const pid_t pid = fork();
  if (pid == 0) {
    alarm(60);  // a child that waits for threads it does not have ends here
    _exit(jobs(rounds, 300) ? 0 : 2);
  }
  int status = 0;
  waitpid(pid, &status, 0);
  return WIFEXITED(status) ? WEXITSTATUS(status) : 3;
}
size_t pool_check_pinned_size(size_t bytes) { return pinned_size(bytes); }
}
