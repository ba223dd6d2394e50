// Host check of the rule that hands an event to the rounds kernel (rounds_take),
// built with nvcc and run on the CPU by tests/test_rounds_rule.py.  What the
// launchers count on, in every mode: the rule falls with R, and along the sizes of
// one list it changes at most once, from refusing to taking; and an event in a call of several is never
// taken where it would not be alone (a call lasts as long as its slowest event).
// Prints "ok <checks>".
#include <cstdio>

#include "fjg_kernels.cuh"

using namespace fjg;

int main() {
  const double radii[] = {0.0, 0.2, 0.4, 0.5, 0.6, 0.7, 0.8, 0.9, 1.0, 1.1, 1.3, 1.5, 1.8, 2.1, 4.0};
  long checks = 0;
  for (int mode = kRoundsNone; mode <= kRoundsServeOne; ++mode)
    for (int algo = -1; algo <= 1; ++algo) {
      for (int q = 0; q <= kLargeQueue; ++q) {
        const int lo = q == 0 ? 1 : (128 << q) + 1, hi = q == kLargeQueue ? 9000 : 256 << q;
        for (double R : radii) {
          int changes = 0;
          for (int n = lo; n <= hi; ++n, ++checks) {
            changes += n > lo && rounds_take(mode, n, algo, R) != rounds_take(mode, n - 1, algo, R);
            if (n > lo && !rounds_take(mode, n, algo, R) && rounds_take(mode, n - 1, algo, R)) {
              std::printf("mode %d algo %d R %g: %d taken, %d not\n", mode, algo, R, n - 1, n);
              return 1;
            }
            for (double S : radii)
              if (S < R && rounds_take(mode, n, algo, R) && !rounds_take(mode, n, algo, S)) {
                std::printf("mode %d algo %d n %d: taken at R %g, not at %g\n", mode, algo, n, R, S);
                return 1;
              }
            const bool several = mode == kRoundsFew || mode == kRoundsSome;
            if (several && rounds_take(mode, n, algo, R) && !rounds_take(kRoundsOne, n, algo, R)) {
              std::printf("mode %d algo %d n %d R %g: taken among others, not alone\n", mode, algo, n, R);
              return 1;
            }
          }
          if (changes > 1) {
            std::printf("mode %d algo %d R %g: %d changes in list %d\n", mode, algo, R, changes, q);
            return 1;
          }
        }
      }
    }
  std::printf("ok %ld\n", checks);
  return 0;
}
