// Host check of parallel_chunks (ffv_internal.h) about the sizes where it changes over: every
// element once, in the chunk that its thread index names, for any number of threads.
#include <stdio.h>

#include <atomic>
#include <vector>

#include "ffv_internal.h"

int main() {
  int failures = 0;
  for (int64_t n : {0, 1, 7, 511, 512, 513, 2047, 2048, 2049, 5000})
    for (int nth : {1, 2, 3, 16, 64}) {
      std::vector<std::atomic<int>> hits(n + 1);
      const int64_t chunk = (n + nth - 1) / nth;
      std::atomic<int> bad(0), calls(0);
      parallel_chunks(n, nth, [&](int t, int64_t a, int64_t b) {
        calls++;
        if (a != std::min(n, t * chunk) || b != std::min(n, (t + 1) * chunk)) bad++;
        for (int64_t i = a; i < b; i++) hits[i]++;
      });
      for (int64_t i = 0; i < n; i++) bad += hits[i] != 1;
      bad += calls != nth;
      if (bad) {
        printf("n %lld threads %d: %d\n", (long long)n, nth, (int)bad);
        failures++;
      }
    }
  printf("%d failures\n", failures);
  return failures != 0;
}
