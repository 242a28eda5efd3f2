// The word a solve publishes and the host's test of it (kernels.cuh), on the
// host: prints "bad <n>", the iterations at which the test was wrong.
#include <cstdio>
#include <initializer_list>

#include "kernels.cuh"

int main() {
  int bad = 0;
  for (long long start : {0LL, (1LL << 25) - 3, (1LL << 26) - 3, (1LL << 27) - 3, (1LL << 31) - 9})
    for (int d = 0; d < 6; ++d) {
      const long long done = start + d;  // tests that have run
      const unsigned w = gsb::published_word(static_cast<int>(done), false, 0);
      bad += (w & 1u) != 0;
      // the host waits for the test of an iteration at most two ahead, or one it has seen
      for (long long want = done > 3 ? done - 3 : 0; want <= done + 2; ++want)
        bad += gsb::published_reached(w, static_cast<unsigned>(want)) != (done >= want);
      for (int status = 0; status < 7; ++status) {
        const unsigned s = gsb::published_word(static_cast<int>(done), true, status);
        bad += (s & 1u) == 0 || static_cast<int>(s >> 28) != status;
      }
    }
  std::printf("bad %d\n", bad);
  return 0;
}
