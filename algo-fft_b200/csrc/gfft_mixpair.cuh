// The compiled mixed-radix column tiles (gfft_mixcols.cuh) on packed column
// pairs, complex64: the same schedules and index maps, 16 columns as 8 pairs
// of 16 bytes (real parts, imaginary parts), the same threads per column.
//
// The scalar tiles are bound by instruction issue (68-75 % of the slots, 2-4
// warp instructions per element and pass); packed FP32 halves their arithmetic
// and 16-byte exchanges halve their shared-memory instructions.  Stage twiddles
// come from rounded table entries (PairPowers).
#pragma once
#include "gfft_mixbs.cuh"
#include "gfft_pairpass.cuh"

namespace gfft {

constexpr int kMixPairs = 8;  // column pairs per tile

template <typename SC, int TT>
struct MixPairTile {
  static constexpr int L = SC::L, NP = kMixPairs;
  static constexpr int T = TT > 0 ? TT : L / SC::rmax();
  static constexpr int TPB = T * NP;
  static constexpr int SMEM = L * NP * 16;
  __host__ __device__ static constexpr int q_at(int s) { return (L / SC::radix(s) + T - 1) / T; }
  __host__ __device__ static constexpr int vmax() {
    int m = 1;
    for (int s = 0; s < SC::NS; ++s) m = q_at(s) * SC::radix(s) > m ? q_at(s) * SC::radix(s) : m;
    return m;
  }
  // resident CTAs asked of the register allocation: the elements of a thread
  // plus 56 registers, within 200 KB of shared memory
  static constexpr int WARP_TPB = (TPB + 31) / 32 * 32;
  static constexpr int BY_REGS = 65536 / (WARP_TPB * (4 * vmax() + 56));
  static constexpr int BY_SMEM = 200 * 1024 / SMEM;
  static constexpr int MINB0 = BY_REGS < BY_SMEM ? BY_REGS : BY_SMEM;
  static constexpr int MINB = MINB0 < 1 ? 1 : MINB0 > 10 ? 10 : MINB0;
  // one row is one 128-byte bank row: 8 lanes on consecutive pairs of a row, or
  // on consecutive rows of a pair, cover it
  __device__ static __forceinline__ int phys(int row, int c) { return row * NP + (c ^ (row & 7)); }
  __device__ static __forceinline__ Pair get(const float4* sh, int row, int c) {
    const float4 f = sh[phys(row, c)];
    return Pair{V2(float2{f.x, f.y}), V2(float2{f.z, f.w})};
  }
  __device__ static __forceinline__ void put(float4* sh, int row, int c, Pair a) {
    sh[phys(row, c)] = float4{a.x.v.x, a.x.v.y, a.y.v.x, a.y.v.y};
  }
};

// One stage, then the next (see mix_stage).  ld(row, c) gives the first
// stage's inputs (LD::kShared: from the tile itself); the last stage hands
// st(row, c, value) its outputs (ST::kShared: back into the tile), after the
// scaling of ST::Factors.
template <typename SC, typename TL, int DIR, int S, typename LD, typename ST>
__device__ __forceinline__ void mix_pair_stage(Pair* v, float4* sh, int t, int c, const float2* __restrict__ tw,
                                               const LD& ld, const ST& st) {
  constexpr int L = SC::L, T = TL::T, RS = SC::radix(S), P = SC::prefix(S), NB = L / RS, Q = (NB + T - 1) / T;
  constexpr bool GUARD = NB % T != 0, FIRST = S == 0, LAST = S == SC::NS - 1;
  constexpr bool READ_SH = !FIRST || LD::kShared;
  if constexpr (LAST && ST::ROWS_FIRST) {
    t = threadIdx.x % T;
    c = threadIdx.x / T;
  }
  [[maybe_unused]] typename ST::template Factors<RS, P, DIR> f[LAST ? Q : 1];
  if constexpr (LAST) {
#pragma unroll
    for (int q = 0; q < Q; ++q) f[q].begin(st, GUARD && t + q * T >= NB ? 0 : t + q * T, c);
  }
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int i = t + q * T;
    if (GUARD && i >= NB) break;
#pragma unroll
    for (int r = 0; r < RS; ++r) {
      if constexpr (FIRST) v[q * RS + r] = ld(i + r * NB, c);
      else v[q * RS + r] = TL::get(sh, i + r * NB, c);
    }
    if constexpr (P > 1) {
      PairPowers<RS> pw;
      pw.template load<DIR>(tw, (i % P) * (L / (P * RS)));
      pw.apply(v + q * RS);
    }
    pdft<RS, DIR>(v + q * RS);
    if constexpr (LAST) f[q].scale(v + q * RS);
  }
  if constexpr (LAST) {
    if constexpr (ST::kShared && READ_SH) __syncthreads();
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int i = t + q * T;
      if (GUARD && i >= NB) break;
#pragma unroll
      for (int r = 0; r < RS; ++r) st(i + r * P, c, v[q * RS + r]);
    }
  } else {
    if constexpr (READ_SH) __syncthreads();
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int i = t + q * T;
      if (GUARD && i >= NB) break;
      const int k = i % P, j = (i - k) * RS + k;
#pragma unroll
      for (int r = 0; r < RS; ++r) TL::put(sh, j + r * P, c, v[q * RS + r]);
    }
    __syncthreads();
    mix_pair_stage<SC, TL, DIR, S + 1>(v, sh, t, c, tw, ld, st);
  }
}

// Columns as rows of L elements, times W_N^(k row) for column k = col0 + its
// index, straight from registers: runs of T elements of a column (whole
// sectors where T is a multiple of 4).
template <typename SC>
struct MixPairStoreT {
  static constexpr bool ROWS_FIRST = true, kShared = false;
  static constexpr int L = SC::L;
  float2* out;  // of the tile's column 0
  BigTwiddle bt;
  unsigned col0;
  template <int RS, int P, int DIR>
  struct Factors {
    Pair b, s, s4;
    __device__ __forceinline__ void begin(const MixPairStoreT& st, int row0, int c) {
      const unsigned k = st.col0 + 2 * c;
      auto both = [&](unsigned e) {  // W^(k e), W^((k + 1) e)
        const float2 w = pair_twiddle<DIR>(st.bt, k * e);
        return two(w, cmul(w, pair_twiddle<DIR>(st.bt, e)));
      };
      b = both(row0);
      s = both(P);
      if constexpr (RS > 4) s4 = both(4 * P);
    }
    __device__ __forceinline__ void scale(Pair* v) const { pair_scale_powers<RS>(v, b, s, s4); }
  };
  __device__ __forceinline__ void operator()(int row, int c, Pair o) const {
    float2* p = out + 2 * c * L + row;
    __stcg(p, float2{o.x.v.x, o.y.v.x});
    __stcg(p + L, float2{o.x.v.y, o.y.v.y});
  }
};

struct MixPairNoFactors {
  static constexpr bool ROWS_FIRST = false;
  template <int RS, int P, int DIR> using Factors = PairNoFactors;
};

// ---- Bluestein chain (k_mix_bs) ---------------------------------------------
// M1 and M2 are multiples of 16: every tile is whole and every row of the
// scratch and work buffers starts on 16 bytes, and so do the chirps and
// filters; the user's transforms may start anywhere and move in 8 bytes where
// they do not (y16).  The middle and last passes only: the first pass waits on
// its chirped loads, and the fewer warps of the pairs wait longer (12 x 12: 63
// -> 70 us, 16 x 10: 60 -> 95).

struct MixPairRowsIn {  // rows `pitch` pairs apart
  static constexpr bool kShared = false;
  const float4* in;
  unsigned pitch;
  __device__ __forceinline__ Pair operator()(int row, int c) const {
    return pair_of(__ldcg(in + (unsigned(row) * pitch + unsigned(c))));
  }
};

template <typename TL>
struct MixPairTileIn {
  static constexpr bool kShared = true;
  const float4* sh;
  __device__ __forceinline__ Pair operator()(int row, int c) const { return TL::get(sh, row, c); }
};

// w[m], w[m + 1] (m even; the tables are padded to even lengths)
__device__ __forceinline__ Pair bs_pair(const float2* w, unsigned m, int inv) {
  Pair p = pair_of(__ldg(reinterpret_cast<const float4*>(w + m)));
  if (inv) p.y = -p.y;
  return p;
}

template <typename TL>
struct MixPairBsFilter : MixPairNoFactors {
  static constexpr bool kShared = true;
  float4* sh;
  const float2* f;
  unsigned m1, col0, M;
  int inv;
  __device__ __forceinline__ void operator()(int row, int c, Pair v) const {
    const unsigned k = col0 + 2 * unsigned(c) + m1 * unsigned(row);
    Pair q;
    if (inv) q = two(cconj(__ldg(f + (k == 0 ? 0 : M - k))), cconj(__ldg(f + (M - k - 1))));
    else q = bs_pair(f, k, 0);
    TL::put(sh, row, c, pmul(v, q));
  }
};

struct MixPairBsOut : MixPairNoFactors {
  static constexpr bool kShared = false;
  float2* y;
  const float2* w;
  unsigned n, m2, col0;
  float scale;
  int inv;
  bool y16;
  __device__ __forceinline__ void operator()(int row, int c, Pair v) const {
    const unsigned k = col0 + 2 * unsigned(c) + m2 * unsigned(row);
    if (k >= n) return;
    const V2 s(float2{scale, scale});
    Pair o = pmul(v, bs_pair(w, k, inv));
    o = Pair{o.x * s, o.y * s};
    if (y16 && k + 1 < n) {
      __stcs(reinterpret_cast<float4*>(y + k), pair_raw(o));
      return;
    }
    st_stream(y + k, float2{o.x.v.x, o.y.v.x});
    if (k + 1 < n) st_stream(y + k + 1, float2{o.x.v.y, o.y.v.y});
  }
};

template <typename SC, int KIND, int TT>
__global__ void __launch_bounds__(MixPairTile<SC, TT>::TPB, MixPairTile<SC, TT>::MINB) k_mix_bs_pair(MixBsParams p) {
  static_assert(KIND == BSK_MID || KIND == BSK_OUT, "the first pass stays scalar");
  if constexpr (KIND != BSK_OUT) asm volatile("griddepcontrol.launch_dependents;");
  if constexpr (KIND != BSK_IN) asm volatile("griddepcontrol.wait;" ::: "memory");  // the pass before this one
  using TL = MixPairTile<SC, TT>;
  constexpr int L = SC::L, NC = 2 * TL::NP;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float4* sh = reinterpret_cast<float4*>(smem_raw);
  int64_t off_y, s;
  unsigned col0, n, M;
  const float2 *w, *f;
  BigTwiddle bt = p.bt;
  float oscale;
  if (p.items) {
    const MixBsItem m = p.items[p.blk[blockIdx.x]];
    col0 = unsigned(int(blockIdx.x) - m.first[KIND]) * NC;
    off_y = m.off;
    s = m.s;
    n = unsigned(m.n);
    M = unsigned(m.M);
    const float2* tab = static_cast<const float2*>(p.tab);
    w = tab + m.chirp;
    f = tab + m.filt;
    bt = BigTwiddle{tab + m.lo, tab + m.hi, m.shift};
    oscale = float(p.inv ? 1.0 / double(m.n) : 1.0);
  } else {
    const unsigned b = blockIdx.x / unsigned(p.tiles);
    col0 = (blockIdx.x % unsigned(p.tiles)) * NC;
    off_y = b * p.odist;
    s = b * p.M;
    n = unsigned(p.n);
    M = unsigned(p.M);
    w = static_cast<const float2*>(p.w);
    f = static_cast<const float2*>(p.f);
    oscale = float(p.scale);  // batch mode: the direction's own tables
  }
  const unsigned ncols = M / L;  // M2 for BSK_OUT, M1 for BSK_MID
  const int c = threadIdx.x % TL::NP, t = threadIdx.x / TL::NP;
  const float2* tw = static_cast<const float2*>(p.tw);
  Pair v[TL::vmax()];
  if constexpr (KIND == BSK_MID) {
    const MixPairRowsIn ld{reinterpret_cast<const float4*>(static_cast<const float2*>(p.scratch) + s + col0), ncols / 2};
    const MixPairBsFilter<TL> fwd{{}, sh, f, ncols, col0, M, p.inv};
    mix_pair_stage<SC, TL, -1, 0>(v, sh, t, c, tw, ld, fwd);
    __syncthreads();
    const MixPairTileIn<TL> back{sh};
    const MixPairStoreT<SC> st{static_cast<float2*>(p.work) + s + int64_t(col0) * L, bt, col0};
    mix_pair_stage<SC, TL, +1, 0>(v, sh, t, c, tw, back, st);
  } else {
    const MixPairRowsIn ld{reinterpret_cast<const float4*>(static_cast<const float2*>(p.work) + s + col0), ncols / 2};
    float2* y = static_cast<float2*>(p.y) + off_y;
    const MixPairBsOut st{{}, y, w, n, ncols, col0, float(double(oscale) / double(M)), p.inv,
                          (reinterpret_cast<uintptr_t>(y) & 15) == 0};
    mix_pair_stage<SC, TL, +1, 0>(v, sh, t, c, tw, ld, st);
  }
}

}  // namespace gfft
