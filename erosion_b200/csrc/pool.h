// A pool of host threads for one call (batch.cu).
#pragma once
#include <algorithm>
#include <atomic>
#include <exception>
#include <stdexcept>
#include <system_error>
#include <thread>
#include <vector>

namespace eb {

// Runs f(order[0]), f(order[1]), ... on up to `threads` host threads, each of which calls
// enter() first; the first exception is thrown again once all have ended.  A thread that
// the system refuses is done without: the others take its jobs.
template <class Enter, class F>
void on_pool(int threads, const std::vector<int>& order, Enter&& enter, F&& f) {
  const int n = (int)order.size();
  std::atomic<int> next{0};
  std::atomic<bool> stop{false};
  std::vector<std::exception_ptr> errs(std::max(1, std::min(threads, n)));
  std::vector<std::thread> pool;
  pool.reserve(errs.size());
  for (size_t t = 0; t < errs.size(); ++t) {
    try {
      pool.emplace_back([&, t] {
        try {
          enter();
          for (int i; !stop && (i = next++) < n;) f(order[i]);
        } catch (...) {
          errs[t] = std::current_exception();
          stop = true;
        }
      });
    } catch (const std::system_error&) {
      break;
    }
  }
  if (pool.empty()) throw std::runtime_error("no host thread could be started");
  for (auto& th : pool) th.join();
  for (auto& e : errs)
    if (e) std::rethrow_exception(e);
}

}  // namespace eb
