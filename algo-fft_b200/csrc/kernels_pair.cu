// Packed-pair kernels of the multi-pass complex64 powers of two: two passes
// for 2^15..2^20, three for 2^21..2^24 (gfft_pairpass.cuh).
#include "gfft_internal.h"
#include "gfft_pairpass.cuh"

namespace gfft {
namespace {

// What bounds these passes: HBM up to 256-row columns (6.2-6.7 TB/s of their
// own traffic), beyond that the two or three CTAs per SM that registers and
// shared memory allow, and in long runs the 1 kW power cap, which takes the SM
// clock from 1965 to about 1600 MHz.  So the tiles take the schedule with the
// fewest stages (32 x 16, 32 x 32) although 8 x 8 x 8 is faster in a burst:
// it moves half as much through shared memory.
//
// 512 MiB batches, scalar kernels before -> now: 2^15 356 -> 337 us, 2^16 367
// -> 329, 2^17 371 -> 342, 2^18 389 -> 348, 2^19 420 -> 384, 2^20 466 -> 429,
// 2^21 546 -> 516, 2^22 585 -> 513, 2^23 605 -> 544, 2^24 615 -> 559; rel-L2
// errors 2.5-5.7e-7 -> 1.7-4.6e-7 (twiddles from rounded table entries).
//
// 2^17..2^19 keep the scalar second pass (radix 32, 512 and 1024 rows: 176 and
// 201 us per 512 MiB against 182 and 219 in pairs, and more threads per column
// for small batches); at 2^20 its product-tree twiddles would cost accuracy
// (6e-7 against 3.2e-7), so the pairs serve both passes.
//
// Tile of a pass over columns of L rows: elements per thread, column pairs,
// resident CTAs asked for.
template <int L> struct Tile;
template <> struct Tile<128> { static constexpr int E = 16, NP = 16, MB = 4; };
template <> struct Tile<256> { static constexpr int E = 16, NP = 8, MB = 4; };
template <> struct Tile<512> { static constexpr int E = 32, NP = 8, MB = 3; };
template <> struct Tile<1024> { static constexpr int E = 32, NP = 4, MB = 3; };
// Passes of fewer than kFew such tiles, too few for the SMs, take the fewest
// columns: one transform spreads over more SMs.  The stages are the same, so a
// transform's result does not depend on the batch it is in.
// Below the line: one 2^16 alone 28 -> 23 us, 2^17 29 -> 26; at it, 16 x 2^15
// took 11.9 us with the large tiles, 12.4 with the small ones.
constexpr int kFew = 128;
template <int L>
struct Few {
  static constexpr int E = Tile<L>::E, NP = 4, MB = Tile<L>::MB;
};

// Prefix product of the last stage (its radix is L / it).
template <int L, int EPT>
constexpr int last_prefix() {
  int p = 1;
  while (p * Sched<L, EPT>::radix_at(p) < L) p *= Sched<L, EPT>::radix_at(p);
  return p;
}

// PDL: the launch may begin while its predecessor drains (the kernel waits for
// it before it reads).
template <auto* FN, int TPB, int SMEM, bool PDL>
cudaError_t go(const PairPassParams& p, int64_t tiles, cudaStream_t st) {
  if (tiles > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
  if constexpr (SMEM > 48 * 1024) {
    const cudaError_t e = raise_smem<FN>(SMEM);
    if (e != cudaSuccess) return e;
  }
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(tiles));
  cfg.blockDim = dim3(TPB);
  cfg.dynamicSmemBytes = SMEM;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = PDL ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, FN, p);
}

// Pass 1 over columns of N1 rows, `cols` of them per transform.
template <int N1, int64_t COLS, int DIR>
cudaError_t first_pass(const PairPassParams& p, int64_t nb, cudaStream_t st) {
  using A = Tile<N1>;
  using F = Few<N1>;
  if (nb * (COLS / (2 * A::NP)) >= kFew) {
    using S = PairShape<N1, A::E, A::NP>;
    return go<&k_pair_tp1<N1, COLS, A::E, A::NP, DIR, A::MB>, S::TPB, S::SMEM, false>(p, nb * (COLS / (2 * A::NP)), st);
  }
  using S = PairShape<N1, F::E, F::NP>;
  return go<&k_pair_tp1<N1, COLS, F::E, F::NP, DIR, F::MB>, S::TPB, S::SMEM, false>(p, nb * (COLS / (2 * F::NP)), st);
}

template <int N1, int N2, int DIR>
cudaError_t launch_tp(const PairPassParams& p, int pass, int64_t nb, cudaStream_t st) {
  if (pass == 1) return first_pass<N1, N2, DIR>(p, nb, st);
  using B = Tile<N2>;
  using F = Few<N2>;
  if (nb * (N1 / (2 * B::NP)) >= kFew) {
    using S = PairShape<N2, B::E, B::NP>;
    return go<&k_pair_tp2<N1, N2, B::E, B::NP, DIR, B::MB>, S::TPB, S::SMEM, true>(p, nb * (N1 / (2 * B::NP)), st);
  }
  using S = PairShape<N2, F::E, F::NP>;
  return go<&k_pair_tp2<N1, N2, F::E, F::NP, DIR, F::MB>, S::TPB, S::SMEM, true>(p, nb * (N1 / (2 * F::NP)), st);
}

template <int N1, int N2, int DIR>
cudaError_t launch_first(const PairPassParams& p, int, int64_t nb, cudaStream_t st) {
  return first_pass<N1, N2, DIR>(p, nb, st);
}

template <int N1, int M1, int M2, int DIR>
cudaError_t launch_tp3(const PairPassParams& p, int pass, int64_t nb, cudaStream_t st) {
  if (pass == 1) return first_pass<N1, int64_t(M1) * M2, DIR>(p, nb, st);
  using B = Tile<M1>;
  using D = Tile<M2>;
  using SB = PairShape<M1, B::E, B::NP>;
  using SD = PairShape<M2, D::E, D::NP>;
  if (pass == 2)
    return go<&k_pair_tp3b<N1, M1, M2, B::E, B::NP, DIR, B::MB>, SB::TPB, SB::SMEM, true>(
        p, nb * (int64_t(M2) * N1 / (2 * B::NP)), st);
  return go<&k_pair_tp3c<N1, M1, M2, D::E, D::NP, DIR, D::MB>, SD::TPB, SD::SMEM, true>(
      p, nb * (int64_t(M1) * N1 / (2 * D::NP)), st);
}

// first_only: the scalar kernel runs the second pass
template <int N1, int N2>
PairKernel two_pass(int te, int emax) {
  return PairKernel{N1, N2, 0, te, emax, last_prefix<N1, Tile<N1>::E>(), false,
                    {&launch_tp<N1, N2, -1>, &launch_tp<N1, N2, 1>}};
}
template <int N1, int N2>
PairKernel first_only(int te, int emax) {
  return PairKernel{N1, N2, 0, te, emax, last_prefix<N1, Tile<N1>::E>(), true,
                    {&launch_first<N1, N2, -1>, &launch_first<N1, N2, 1>}};
}
template <int N1, int M1, int M2>
PairKernel three_pass(int te = 0, int emax = 0) {
  return PairKernel{N1, M1, M2, te, emax, last_prefix<N1, Tile<N1>::E>(), false,
                    {&launch_tp3<N1, M1, M2, -1>, &launch_tp3<N1, M1, M2, 1>}};
}

}  // namespace

// One per length; te / emax: the scalar tile for buffers off 16 bytes (the
// fastest scalar variant of the length).  2^21 is the longest that the
// allocation-free entry holds, so its plan has two-pass tables too.
const PairKernel* find_pair(int64_t n) {
  static const PairKernel k[] = {
      two_pass<128, 256>(4096, 16),  two_pass<256, 256>(8192, 32),   first_only<256, 512>(8192, 32),
      first_only<512, 512>(8192, 32),  first_only<512, 1024>(8192, 32),  two_pass<1024, 1024>(8192, 16),
      three_pass<128, 128, 128>(8192, 16), three_pass<256, 128, 128>(),    three_pass<256, 256, 128>(),
      three_pass<256, 256, 256>()};
  for (const PairKernel& e : k)
    if (int64_t(e.n1) * e.m1 * (e.m2 ? e.m2 : 1) == n) return &e;
  return nullptr;
}

}  // namespace gfft
