// The host threads of csrc/zg_host.hpp: which copies start threads, that every
// byte arrives, and that a throwing call is reported.
#include <cstdio>
#include <mutex>
#include <set>
#include <stdexcept>

#include "../../0g-da-encoder_b200/csrc/zg_host.hpp"
using namespace zg;

int main() {
  int bad = 0;
  auto check = [&](bool ok, const char* what, size_t n) {
    if (!ok) {
      printf("%s at %zu\n", what, n);
      ++bad;
    }
  };
  // rows of 32 KB: a 128 x 1024 recovery's 203 and 384, the line, and past it
  std::mutex mu;
  for (size_t rows : {1, 203, 384, 511, 512, 513}) {
    std::set<std::thread::id> ids;
    std::vector<int> times(rows, 0);
    host_copies(rows, 32768, [&](size_t i) {
      std::lock_guard<std::mutex> g(mu);
      ids.insert(std::this_thread::get_id());
      ++times[i];
    });
    check(std::all_of(times.begin(), times.end(), [](int x) { return x == 1; }), "a row not copied once", rows);
    check(ids.size() <= (rows * 32768 < COPY_SERIAL_BELOW ? 1 : COPY_THREADS), "too many threads", rows);
    if (rows * 32768 < COPY_SERIAL_BELOW) check(*ids.begin() == std::this_thread::get_id(), "another thread", rows);
  }
  for (size_t n : {size_t(0), size_t(1), COPY_SERIAL_BELOW - 1, COPY_SERIAL_BELOW, COPY_SERIAL_BELOW + 12345}) {
    std::vector<uint8_t> a(n + 1, 7), b(n + 1, 9);
    for (size_t i = 0; i < n; ++i) a[i] = (uint8_t)(i * 2654435761u >> 13);
    host_copy(b.data(), a.data(), n);
    check(std::equal(a.begin(), a.begin() + n, b.begin()) && b[n] == 9, "bytes differ", n);
  }
  for (size_t most : {1, 4}) {
    std::atomic<int> ran{0};
    const bool ok = host_parallel(100, 8, most, [&](size_t i) {
      ++ran;
      if (i == 41) throw std::bad_alloc();
    });
    check(!ok && ran == 100, "a throwing call", most);
  }
  return bad != 0;
}
