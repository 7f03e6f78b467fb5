// Host work in parts.  Plain C++, no CUDA calls.
#pragma once

#include <cstdint>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

namespace ct {

// f(0) .. f(n - 1): f(0) on the calling thread, the others on threads of their
// own, or here too where one cannot be started.  Returns when all have ended;
// the first exception of any of them is thrown then.
template <typename Thread = std::thread, typename F>
void run_parts(uint32_t n, F f) {
  std::mutex mu;
  std::exception_ptr error;
  auto part = [&](uint32_t i) {
    try {
      f(i);
    } catch (...) {
      std::lock_guard<std::mutex> lk(mu);
      if (!error) error = std::current_exception();
    }
  };
  std::vector<Thread> pool;
  uint32_t started = 1;
  try {
    pool.reserve(n);
    for (; started < n; ++started) pool.emplace_back(part, started);
  } catch (...) {
  }
  for (uint32_t i = 0; i < n; i = i == 0 ? started : i + 1) part(i);
  for (auto& t : pool) t.join();
  if (error) std::rethrow_exception(error);
}

}  // namespace ct
