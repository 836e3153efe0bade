// Reading the transforms' sums from the device into the host's, chunk by chunk: host code alone (a test
// builds it without a device).
#pragma once

#include <algorithm>

namespace pxr {

constexpr long long CHUNK = 1LL << 18;  // doubles: 2 MiB

// n doubles, in chunks through two buffers in turn, one filled while the other is added. fetch(at, count,
// buffer): starts a chunk's copy; wait(): until what was started is done; add(at, count, buffer): adds a
// chunk that was fetched whole; clear(count): starts the clearing of the first `count` doubles at the source.
// fetch, wait and clear return 0 or an error. What has been added is cleared, on an error too, so that a
// second read takes the rest and nothing twice; *taken, kept by the caller between reads, is how many doubles
// have been added and could not be cleared. (One clearing a read: with one a chunk a
// read of 161 MB took 12.7 ms, with one 11.3 to 12.6.)
template <typename Fetch, typename Wait, typename Add, typename Clear>
int read_add(long long n, long long *taken, double *const buffer[2], Fetch fetch, Wait wait, Add add,
             Clear clear) {
  auto settle = [&]() {
    if (*taken == 0) return 0;
    const int r = clear(*taken);
    if (r == 0) *taken = 0;
    return r;
  };
  if (int r = settle()) return r;
  auto start = [&](long long at) { return fetch(at, std::min(CHUNK, n - at), buffer[(at / CHUNK) & 1]); };
  int r = n > 0 ? start(0) : 0;
  for (long long at = 0; at < n && r == 0; at += CHUNK) {
    if ((r = wait())) break;
    if (at + CHUNK < n) r = start(at + CHUNK);
    *taken = std::min(n, at + CHUNK);
    add(at, *taken - at, buffer[(at / CHUNK) & 1]);
  }
  if (r) wait();  // what was started may still write the buffer
  const int cleared = settle();
  return r ? r : cleared;
}

}  // namespace pxr
