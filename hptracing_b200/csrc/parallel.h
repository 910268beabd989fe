// Runs a function on several host threads.
#pragma once

#include <exception>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace hpt {

// f() on up to n threads (the caller's among them; fewer where the system
// has no more threads), then joins them. The first exception of any of them
// is rethrown here, so none ends the process.
template <class F>
void run_threads(int n, F&& f) {
  std::exception_ptr error;
  std::mutex mu;
  auto guarded = [&] {
    try {
      f();
    } catch (...) {
      std::lock_guard<std::mutex> lk(mu);
      if (!error) error = std::current_exception();
    }
  };
  std::vector<std::thread> pool;
  pool.reserve(n > 1 ? n - 1 : 0);
  for (int i = 1; i < n; ++i) {
    try {
      pool.emplace_back(guarded);
    } catch (const std::system_error&) {
      break;
    }
  }
  guarded();
  for (std::thread& t : pool) t.join();
  if (error) std::rethrow_exception(error);
}

}  // namespace hpt
