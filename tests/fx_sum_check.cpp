// Host check of the exact sums of csrc/tpm_fx.cuh (fx_add, fx_total): of any
// number of terms, the correctly rounded sum, in any order.  Prints "ok" or the
// first failure.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "tpm_fx.cuh"

using namespace tpm;

static double total(const std::vector<long long> &v, int k) {
  FxSum s = {};
  int biased = 0;
  for (long long t : v) {
    fx_add(s, t < 0 || biased % 3 ? t + kFxBias : t);
    biased += t < 0 || biased % 3;
  }
  return fx_total(s, biased, k);
}

int main() {
  std::mt19937_64 rng(11);
  long bad = 0;
  for (int bits : {40, 57, 62})
    for (int n : {0, 1, 2, 6, 7, 8, 62, 63, 64, 500, 70000})
      for (int kind = 0; kind < 5; ++kind)
        for (int rep = 0; rep < (n > 1000 ? 3 : 400); ++rep) {
          std::vector<long long> v(n);
          __int128 exact = 0;
          for (long long &t : v) {
            const long long r = (long long)(rng() >> (64 - bits));
            t = kind == 0 ? r                                  // positive
                : kind == 1 ? (rng() & 1 ? r : -r)             // both signs
                : kind == 2 ? (1ll << bits) - 1                // the largest
                : kind == 3 ? -((1ll << bits) - 1)
                            : (rng() & 1 ? 1ll : -1ll) << (rng() % bits);
            exact += t;
          }
          const double want = (double)exact, a = total(v, 0);  // (rounds to nearest)
          std::shuffle(v.begin(), v.end(), rng);
          const double b = total(v, 0);
          if ((std::memcmp(&a, &want, 8) || std::memcmp(&b, &a, 8)) && !(want == 0 && a == 0))
            if (bad++ < 10) std::printf("bits %d n %d kind %d: %a %a, exact %a\n", bits, n, kind, a, b, want);
        }
  // ties and what breaks them, around the width that fx_to takes
  for (int s = 0; s < 31; ++s)
    for (int sign : {-1, 1})
      for (long long off : {-1ll, 0ll, 1ll}) {
        const __int128 x = sign * ((((__int128)1 << 52) + 1) * ((__int128)1 << (11 + s)) +
                                   ((__int128)1 << (10 + s)) + off);
        const FxSum f = {(unsigned long long)x, (unsigned)(x >> 64)};
        const double got = fx_total(f, 0, 0), want = (double)x;
        if (got != want && bad++ < 10) std::printf("tie %d %d %lld: %a, %a\n", s, sign, off, got, want);
      }
  if (!bad) std::printf("ok\n");
  return bad != 0;
}
