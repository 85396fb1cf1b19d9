// Prints "precision n M M1" for every n in 8193..131072 at which the mixed
// Bluestein split changes; the factor lengths come as arguments.
#include <cstdio>
#include <cstdlib>
#include "gfft_bssplit.h"

int main(int argc, char** argv) {
  std::vector<int64_t> lengths;
  for (int i = 1; i < argc; ++i) lengths.push_back(std::atoll(argv[i]));
  for (int prec = 0; prec < 2; ++prec) {
    gfft::BsSplit last;
    for (int64_t n = 8193; n <= 131072; ++n) {
      const gfft::BsSplit s = gfft::bs_split(lengths, n, gfft::bs_split_wide(prec == 1));
      if (s.m == last.m && s.m1 == last.m1) continue;
      std::printf("%d %lld %lld %lld\n", prec, (long long)n, (long long)s.m, (long long)s.m1);
      last = s;
    }
  }
  return 0;
}
