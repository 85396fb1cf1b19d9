// The mixed Bluestein FFT length and its split.  Host-only C++ (no CUDA), so
// the rule is unit-tested on its own.
#pragma once
#include <cstdint>
#include <vector>

namespace gfft {

struct BsSplit {
  int64_t m = 0;   // FFT length M = M1 M2; 0: no product reaches 2n - 1
  int64_t m1 = 0;  // M1: the column length of the first and last pass
};

// The smallest product M >= 2n - 1 of two of `lengths` (ascending); among its
// splits the most balanced one with M1 <= wide, else the most balanced.
inline BsSplit bs_split(const std::vector<int64_t>& lengths, int64_t n, int64_t wide) {
  BsSplit best;
  for (size_t i = 0; i < lengths.size(); ++i)
    for (size_t j = i; j < lengths.size(); ++j) {
      const int64_t a = lengths[i], m = a * lengths[j];
      if (m < 2 * n - 1) continue;
      const bool better = (a <= wide) != (best.m1 <= wide) ? a <= wide : a > best.m1;
      if (best.m == 0 || m < best.m || (m == best.m && better)) best = BsSplit{m, a};
    }
  return best;
}

// M1 is the column length of two passes, M2 that of one, and a tile of long
// columns leaves one or two CTAs on an SM.  The bounds on M1, by timing every
// product whose split they change (batches of 2^24 complex64 or 2^23 complex128
// elements, the most balanced split -> this one, us):
//   complex64, 256: 40993 (M = 82944, 288 x 288 -> 192 x 432) 549 -> 452; under
//     a forced mixed length 45007 573 -> 430, 48017 566 -> 444, 50789 584 -> 395,
//     52433 588 -> 433, 54001 558 -> 436, 57347 538 -> 492, 58963 583 -> 485;
//   complex128, 288: 68023 (138240, 320 x 432 -> 288 x 480) 567 -> 465, 73013
//     (147456, 384 x 384 -> 288 x 512) 596 -> 473; forced 50789 572 -> 426, 52433
//     582 -> 434, 58963 586 -> 416, 64007 575 -> 476; 40993 stays at 288 x 288 (192 x
//     432 took 479 against 457).
// Eight transforms at a time: complex128 1.15-1.7x faster, complex64 between
// 0.92x (40993: 24.6 -> 26.7 us) and 1.2x.  Errors: 0.85-0.99 of the balanced
// split's, complex128 68023 1.05 (1.50e-15 -> 1.57e-15).
inline int64_t bs_split_wide(bool c128) { return c128 ? 288 : 256; }

}  // namespace gfft
