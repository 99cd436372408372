// host_threads.h -- a host pass cut into parts, a thread each.
#pragma once

#include <exception>
#include <thread>
#include <vector>

namespace op2b {

// part(0) ... part(n - 1), each once: part 0 by the caller, the others by
// threads of their own.  Where a thread cannot be had (a process at its
// limit: std::thread throws, and no exception may leave a C entry point) the
// caller runs what is left.
template <class Part>
void on_threads(size_t n, const Part &part) {
  std::vector<std::thread> th;
  size_t t = 1;
  try {
    for (; t < n; t++) th.emplace_back([&part, t] { part(t); });
  } catch (const std::exception &) {
  }
  part(0);
  for (; t < n; t++) part(t);
  for (std::thread &x : th) x.join();
}

}  // namespace op2b
