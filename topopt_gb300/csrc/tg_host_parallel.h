// tg_host_parallel.h -- a loop over host threads.
#pragma once
#include <algorithm>
#include <cstdint>
#include <exception>
#include <thread>
#include <vector>

namespace tg {

constexpr int kHostParts = 16;

// fn(lo, hi, part) over [0, n) split across host threads, part < kHostParts.  The loops
// it runs are byte and integer work with per-part results combined exactly, so the
// outcome does not depend on the split.  Serial where the whole is less than 2^20 nodes'
// worth: starting sixteen threads took 0.5 to 1.8 ms, a loop over 200,000 nodes 0.2.
// What fn throws in any part (a row buffer that cannot be allocated) is thrown here,
// the first part's, once every thread has ended.
template <class F>
void host_parallel(int64_t n, int64_t nodes, F&& fn) {
  const unsigned hc = std::thread::hardware_concurrency();
  const int nt = int(std::max(1u, std::min(unsigned(kHostParts), hc)));
  if (nodes < (int64_t(1) << 20) || nt == 1) {
    fn(int64_t(0), n, 0);
    return;
  }
  std::exception_ptr failed[kHostParts];
  const int64_t chunk = (n + nt - 1) / nt;
  auto run = [&](int t) {
    const int64_t lo = t * chunk, hi = std::min(n, lo + chunk);
    if (lo >= hi) return;
    try {
      fn(lo, hi, t);
    } catch (...) {
      failed[t] = std::current_exception();
    }
  };
  std::thread th[kHostParts];
  int started = 0;
  try {
    for (; started < nt; ++started) th[started] = std::thread(run, started);
  } catch (...) {
    // No thread to be had (many jobs building at once): the rest runs here.
  }
  for (int t = started; t < nt; ++t) run(t);
  for (int t = 0; t < started; ++t) th[t].join();
  for (const std::exception_ptr& e : failed)
    if (e) std::rethrow_exception(e);
}

}  // namespace tg
