// Host threads whose exceptions reach the caller: one that leaves a std::thread,
// or a thread destroyed while it can still be joined, ends the process, and the
// C entry points return error codes instead.
#pragma once
#include <exception>
#include <system_error>
#include <thread>
#include <vector>

namespace acg {

// body(0) .. body(count - 1), the first on this thread and each other on its own
// (on this thread too, where no thread can be started).  Returns when all are
// done; the exception of the lowest index is thrown again.
template <typename F>
void run_threads(int count, F&& body) {
  std::vector<std::exception_ptr> error(count);
  auto run = [&](int i) {
    try {
      body(i);
    } catch (...) {
      error[i] = std::current_exception();
    }
  };
  std::vector<std::thread> pool;
  pool.reserve(count);
  int started = 1;
  try {
    for (; started < count; ++started) pool.emplace_back(run, started);
  } catch (const std::system_error&) {
  }
  if (count > 0) run(0);
  for (int i = started; i < count; ++i) run(i);
  for (auto& t : pool) t.join();
  for (const auto& e : error)
    if (e) std::rethrow_exception(e);
}

}  // namespace acg
