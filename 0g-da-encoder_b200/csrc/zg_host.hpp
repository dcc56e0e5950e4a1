// Host threads of a call: parsing, and the copies between a caller's pageable
// memory and pinned staging.
#pragma once
#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <thread>
#include <vector>

namespace zg {

// Runs fn(i) for i < n on up to `most` host threads, `grain` indexes at a time
// (the caller's thread alone when there is one grain or threads cannot be
// had). false if a call threw (out of memory); the other indexes still run.
template <class F>
bool host_parallel(size_t n, size_t grain, size_t most, F fn) {
  std::atomic<size_t> next{0};
  std::atomic<bool> ok{true};
  auto work = [&] {
    for (size_t b; (b = next.fetch_add(grain)) < n;)
      for (size_t i = b; i < std::min(n, b + grain); ++i) {
        try {
          fn(i);
        } catch (...) {
          ok = false;
        }
      }
  };
  const size_t blocks = (n + grain - 1) / grain;
  const size_t want = std::min<size_t>({most, std::max(1u, std::thread::hardware_concurrency()), blocks});
  std::vector<std::thread> more;
  try {
    more.reserve(want);
    for (size_t t = 1; t < want; ++t) more.emplace_back(work);
  } catch (...) {
  }
  work();
  for (std::thread& t : more) t.join();
  return ok;
}

// Threads that copy `bytes` between pageable and pinned memory. Starting and
// joining threads costs 15 us each and slows the CUDA calls that follow by up
// to 1.4 ms (16 threads), so small copies stay on the caller's thread: 6.6 MB
// of rows and 4 MB of payload of a 128 x 1024 recovery take 1.77 ms with one
// thread, 1.80, 1.91, 2.02 and 2.57 with 2, 4, 8 and 16 (12.6 MB: 2.32, 2.23,
// 2.18, 2.44, 2.87); 50 and 32 MB of a 1024 x 1024 one 20.9, 17.5, 15.6, 13.3
// and 14.0 ms (a B200 host of 16 cores; calls that zero-filled a buffer for the
// result and copied it once more: without that 1.37, 1.90 and 8.3 ms).
constexpr size_t COPY_SERIAL_BELOW = size_t(16) << 20;
constexpr size_t COPY_THREADS = 8;
inline size_t copy_threads(size_t bytes) { return bytes < COPY_SERIAL_BELOW ? 1 : COPY_THREADS; }

// memcpy by copy_threads(n) threads
inline void host_copy(void* dst, const void* src, size_t n) {
  constexpr size_t part = size_t(1) << 20;
  const size_t threads = copy_threads(n);
  if (threads == 1) {
    memcpy(dst, src, n);
    return;
  }
  host_parallel((n + part - 1) / part, 1, threads, [&](size_t i) {
    memcpy((uint8_t*)dst + i * part, (const uint8_t*)src + i * part, std::min(part, n - i * part));
  });
}

// copy(i), i < n, of `each` bytes by copy_threads(n * each) threads, some 256 KiB
// at a time
template <class F>
void host_copies(size_t n, size_t each, F copy) {
  host_parallel(n, std::max<size_t>(1, (size_t(1) << 18) / std::max<size_t>(1, each)), copy_threads(n * each), copy);
}

}  // namespace zg
