// The transforms' chunked read-out (read_add, photonoxide_b200/csrc/readout.h) against a device played by
// host arrays: read whole, and with each of its calls failing in turn and a second read after it. Prints the
// cases that leave a sum not added or added twice, and the count of cases.
#include <cstdio>
#include <cstring>
#include <vector>

#include "readout.h"

int main() {
  long long bad = 0, cases = 0;
  for (long long n : {1LL, 7LL, pxr::CHUNK, pxr::CHUNK + 1, 4 * pxr::CHUNK + 12345}) {
    const long long chunks = (n + pxr::CHUNK - 1) / pxr::CHUNK;
    // the call that fails (-1: none): a chunk's copy, a wait, the clearing
    for (long long broken = -1; broken < 3 * chunks; broken++) {
      std::vector<double> device(n), host(n), want(n), a(pxr::CHUNK), b(pxr::CHUNK);
      for (long long q = 0; q < n; q++) {
        device[q] = 1.0 + q;
        host[q] = 0.5 * q;
        want[q] = host[q] + device[q];
      }
      double *buffer[2] = {a.data(), b.data()};
      bool healthy = false;  // the second read's device
      long long waits = 0, clears = 0, taken = 0;
      auto fails = [&](int call, long long number) { return !healthy && broken == 3 * number + call; };
      auto fetch = [&](long long at, long long m, double *to) {
        if (fails(0, at / pxr::CHUNK)) return 1;
        std::memcpy(to, device.data() + at, m * 8);
        return 0;
      };
      auto wait = [&]() { return fails(1, waits++) ? 1 : 0; };
      auto clear = [&](long long m) {
        if (fails(2, clears++)) return 1;
        std::memset(device.data(), 0, m * 8);
        return 0;
      };
      auto add = [&](long long at, long long m, const double *from) {
        for (long long q = 0; q < m; q++) host[at + q] += from[q];
      };
      const int r = pxr::read_add(n, &taken, buffer, fetch, wait, add, clear);
      cases++;
      if (r == 0 && broken >= 0 && !(broken % 3 == 2 && broken / 3 >= clears)) bad++;
      if (r != 0 && broken < 0) bad++;
      healthy = true;
      if (pxr::read_add(n, &taken, buffer, fetch, wait, add, clear) != 0 || taken != 0) bad++;
      for (long long q = 0; q < n; q++)
        if (host[q] != want[q] || device[q] != 0.0) {
          bad++;
          break;
        }
    }
  }
  std::printf("%lld %lld\n", bad, cases);
}
