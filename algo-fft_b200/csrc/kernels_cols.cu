// Power-of-two column batches: FFTs of length L <= 4096 down columns whose
// rows are `pitch` elements apart (the strided batches of
// gfft_exec_strided_batch and every non-contiguous axis of the N-D plans,
// plan_strided.go:35-99, plan_2d.go:161-400, plan_nd.go:188-460).  A CTA
// owns a tile of NC adjacent columns of one array, so each row of the tile
// is one run of NC contiguous elements in HBM; the column FFTs run the
// compile-time register/shared-memory stages of the two-pass kernel
// (col_stage) with the pitch taken at run time, reading and writing the
// columns in place of their natural order.  Lengths that are not powers of
// two use the runtime-radix column kernel.
#include "gfft_internal.h"
#include "gfft_pairpass.cuh"
#include "gfft_twopass.cuh"
#include <algorithm>

namespace gfft {
namespace {

// NC = columns per tile: about 8192 (complex64) / 4096 (complex128)
// elements per tile, 4..32 columns (32-byte rows at least); EPT as the
// two-pass tile rule.
template <typename C, int L>
struct ColTile {
  static constexpr int TE = sizeof(C) == 8 ? 8192 : 4096;
  static constexpr int NC0 = TE / L < 4 ? (sizeof(C) == 8 ? 4 : 2) : (TE / L > 32 ? 32 : TE / L);
  static constexpr int NC = NC0;
  static constexpr int EPT = (L / 16 >= 8) ? 16 : (L / 8 >= 2 ? L / 8 : 2);
  using S = ColShape<L, EPT, NC, sizeof(C)>;
};

template <typename C, int L, int DIR>
__global__ void __launch_bounds__(ColTile<C, L>::S::TPB)
k_pow2_cols(const C* src, C* dst, int64_t ncols, int64_t pitch, int64_t dist, int64_t tiles_per_array,
            const C* __restrict__ tw, typename RealOf<C>::type scale) {
  using T = ColTile<C, L>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* sh = reinterpret_cast<C*>(smem_raw);
  const int64_t arr = blockIdx.x / tiles_per_array;
  const int64_t col0 = (blockIdx.x % tiles_per_array) * int64_t(T::NC);
  const int c = threadIdx.x % T::NC, t = threadIdx.x / T::NC;
  const bool active = col0 + c < ncols && threadIdx.x < T::S::TPB;
  const C* in = src + arr * dist + col0;
  C* out = dst + arr * dist + col0;
  const BigTwiddle bt{nullptr, nullptr, 0};
  C v[T::EPT];
  col_stage<C, L, T::EPT, T::NC, DIR, 1, LOAD_EVICT, OUT_COLUMNS, 0, 0>(v, in, out, sh, t, c, active, tw, scale, bt,
                                                                         0, pitch);
}

template <typename C, int L, int DIR>
cudaError_t launch_cols(const void* src, void* dst, int64_t count, int64_t dist, int64_t ncols, int64_t pitch,
                        const void* tw, double scale, cudaStream_t st) {
  using T = ColTile<C, L>;
  static const cudaError_t attr =
      T::S::SMEM > 48 * 1024
          ? cudaFuncSetAttribute(&k_pow2_cols<C, L, DIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, T::S::SMEM)
          : cudaSuccess;
  if (attr != cudaSuccess) return attr;
  const int64_t tpa = (ncols + T::NC - 1) / T::NC;
  const int64_t tiles = tpa * count;
  if (tiles <= 0) return cudaSuccess;
  if (tiles > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
  k_pow2_cols<C, L, DIR><<<unsigned(tiles), T::S::TPB, T::S::SMEM, st>>>(
      static_cast<const C*>(src), static_cast<C*>(dst), ncols, pitch, dist, tpa, static_cast<const C*>(tw),
      typename RealOf<C>::type(scale));
  return cudaGetLastError();
}

using ColFn = cudaError_t (*)(const void*, void*, int64_t, int64_t, int64_t, int64_t, const void*, double,
                              cudaStream_t);

template <typename C, int DIR>
ColFn pick(int64_t L) {
  switch (L) {
    case 2: return &launch_cols<C, 2, DIR>;
    case 4: return &launch_cols<C, 4, DIR>;
    case 8: return &launch_cols<C, 8, DIR>;
    case 16: return &launch_cols<C, 16, DIR>;
    case 32: return &launch_cols<C, 32, DIR>;
    case 64: return &launch_cols<C, 64, DIR>;
    case 128: return &launch_cols<C, 128, DIR>;
    case 256: return &launch_cols<C, 256, DIR>;
    case 512: return &launch_cols<C, 512, DIR>;
    case 1024: return &launch_cols<C, 1024, DIR>;
    case 2048: return &launch_cols<C, 2048, DIR>;
    case 4096: return &launch_cols<C, 4096, DIR>;
  }
  return nullptr;
}

// ---- complex64 on packed column pairs ---------------------------------------
//
// The same columns two at a time in packed FP32 arithmetic (gfft_pairpass.cuh),
// for arrays on 16 bytes with an even pitch, distance and column count; the
// scalar tile serves the others (the middle axis of a real array has an odd
// pitch) and complex128.  Whole 2-D transforms, before -> now: 8 x 4096 x 4096
// 1070 -> 1007 us, 16 x 2048 x 2048 485 -> 456, 64 x 1024 x 1024 416 -> 394, 256 x
// 512 x 512 384 -> 368, 64 x 256 x 256 26.6 -> 24.6; rel-L2 errors 3.1-4.8e-7 ->
// 2.5-4.5e-7.  In long runs the power cap holds the clock near 1.6 GHz, so the
// tiles with the fewest stages win (512 rows: 32 x 16).  4096 rows as two passes
// of 64 through a workspace measured slower (1040-1085 us) than the one-pass
// tile in place.  128 rows stay on the scalar tile (16 x 16 in pairs: 64 x 128 x
// 2048 91 -> 96 us, 8 x 128^3 136 -> 143).  A length has one tile shape, so an
// array's result does not depend on its batch; the price is on one small array
// of 2048 rows (512 columns: 12.3 -> 14.4 us).
template <int L> struct PairTile;
template <> struct PairTile<32> { static constexpr int E = 8, NP = 16, MB = 8; };
template <> struct PairTile<64> { static constexpr int E = 8, NP = 16, MB = 8; };
template <> struct PairTile<256> { static constexpr int E = 16, NP = 8, MB = 4; };
template <> struct PairTile<512> { static constexpr int E = 32, NP = 8, MB = 3; };
template <> struct PairTile<1024> { static constexpr int E = 16, NP = 4, MB = 2; };
template <> struct PairTile<2048> { static constexpr int E = 16, NP = 4, MB = 1; };
template <> struct PairTile<4096> { static constexpr int E = 16, NP = 2, MB = 1; };

struct PairColsParams {
  const float4* src;
  float4* dst;
  int64_t dist;           // arrays, in pairs
  unsigned pitch, pairs;  // rows, in pairs; pairs per row
  unsigned tiles;         // tiles per array
  const float2* tw;       // W_L
  float scale;
};

template <int L, int DIR>
__global__ void __launch_bounds__(PairShape<L, PairTile<L>::E, PairTile<L>::NP>::TPB, PairTile<L>::MB)
k_pair_cols(PairColsParams p) {
  using T = PairTile<L>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const unsigned arr = blockIdx.x / p.tiles, first = (blockIdx.x % p.tiles) * T::NP;
  const bool active = first + threadIdx.x % T::NP < p.pairs;
  const int64_t off = int64_t(arr) * p.dist + first;
  const PairStridedLoad<PairNoTwiddle> ld{{}, p.src + off, p.pitch, active};
  const PairStridedStore<(DIR > 0)> st{p.dst + off, p.pitch, active, p.scale};
  pair_columns<L, T::E, T::NP, DIR>(reinterpret_cast<float4*>(smem_raw), p.tw, ld, st);
}

template <int L, int DIR>
cudaError_t launch_pair_cols(PairColsParams p, int64_t count, cudaStream_t st) {
  using T = PairTile<L>;
  using S = PairShape<L, T::E, T::NP>;
  p.tiles = (p.pairs + T::NP - 1) / T::NP;
  const int64_t grid = count * int64_t(p.tiles);
  if (grid <= 0) return cudaSuccess;
  if (grid > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
  if constexpr (S::SMEM > 48 * 1024) {
    const cudaError_t e = raise_smem<&k_pair_cols<L, DIR>>(S::SMEM);
    if (e != cudaSuccess) return e;
  }
  k_pair_cols<L, DIR><<<unsigned(grid), S::TPB, S::SMEM, st>>>(p);
  return cudaGetLastError();
}

template <int DIR>
cudaError_t exec_pair_cols(const PairColsParams& p, int64_t n, int64_t count, cudaStream_t st) {
  switch (n) {
    case 32: return launch_pair_cols<32, DIR>(p, count, st);
    case 64: return launch_pair_cols<64, DIR>(p, count, st);
    case 256: return launch_pair_cols<256, DIR>(p, count, st);
    case 512: return launch_pair_cols<512, DIR>(p, count, st);
    case 1024: return launch_pair_cols<1024, DIR>(p, count, st);
    case 2048: return launch_pair_cols<2048, DIR>(p, count, st);
    case 4096: return launch_pair_cols<4096, DIR>(p, count, st);
  }
  return cudaErrorNotSupported;
}

}  // namespace

bool pow2_cols_supported(int64_t n) { return n >= 2 && n <= 4096 && (n & (n - 1)) == 0; }

cudaError_t exec_pow2_cols(int prec, int dir, void* dst, const void* src, int64_t count, int64_t dist, int64_t ncols,
                           int64_t pitch, const void* tw_n, int64_t n, cudaStream_t st) {
  // pairs: 16-byte rows throughout, and row offsets of a tile within 32 bits
  if (prec == kC64 && n >= 32 && n != 128 && ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0 &&
      ((ncols | pitch | dist) & 1) == 0 && ncols <= pitch && pitch < (int64_t(1) << 32) / n) {
    PairColsParams p{};
    p.src = static_cast<const float4*>(src);
    p.dst = static_cast<float4*>(dst);
    p.dist = dist / 2;
    p.pitch = unsigned(pitch / 2);
    p.pairs = unsigned(ncols / 2);
    p.tw = static_cast<const float2*>(tw_n);
    p.scale = dir < 0 ? 1.f : float(1.0 / double(n));
    return dir < 0 ? exec_pair_cols<-1>(p, n, count, st) : exec_pair_cols<1>(p, n, count, st);
  }
  ColFn f = prec == kC64 ? (dir < 0 ? pick<float2, -1>(n) : pick<float2, 1>(n))
                         : (dir < 0 ? pick<double2, -1>(n) : pick<double2, 1>(n));
  if (!f) return cudaErrorNotSupported;
  return f(src, dst, count, dist, ncols, pitch, tw_n, dir < 0 ? 1.0 : 1.0 / double(n), st);
}

}  // namespace gfft
