// Column passes of the multi-pass complex64 transforms on packed column pairs.
//
// A tile is NP pairs of adjacent columns of L rows.  Stages are the Stockham
// stages of the scalar column tiles (same index maps); element (row, pair) is
// 16 bytes in global and in shared memory, so every access is one 16-byte
// instruction for two elements and every butterfly one packed instruction.
//
// The four-step twiddle W_N^(n2 k1) is applied where the first pass stores
// (scaling in the second pass's loads measured slower: 512 rows 6.5 -> 5.0
// TB/s).  Columns leave transposed straight from the last stage's registers:
// it takes its rows with consecutive threads on consecutive rows of one pair,
// so a warp stores 256-byte runs of each column and the extra exchange of a
// transposed store is gone.  With three passes W_M^(m2 k'1), one factor per
// row for the whole tile, is applied as the last pass loads.
#pragma once
#include "gfft_pair.cuh"

namespace gfft {

// W_N^m from the split table, m < N < 2^32.
template <int DIR>
__device__ __forceinline__ float2 pair_twiddle(const BigTwiddle& bt, unsigned m) {
  const float2* lo = static_cast<const float2*>(bt.lo);
  const float2* hi = static_cast<const float2*>(bt.hi);
  float2 w = cmul(__ldg(hi + (m >> bt.shift)), __ldg(lo + (m & ((1u << bt.shift) - 1))));
  if constexpr (DIR > 0) w.y = -w.y;
  return w;
}
__device__ __forceinline__ Pair two(float2 a, float2 b) { return Pair{V2(float2{a.x, b.x}), V2(float2{a.y, b.y})}; }

// t[k], t[k + 1] (k even) of a table.
template <int DIR>
__device__ __forceinline__ Pair pair_table(const float2* t, unsigned k) {
  const float4 f = __ldg(reinterpret_cast<const float4*>(t + k));
  if constexpr (DIR > 0) return Pair{V2(float2{f.x, f.z}), V2(float2{-f.y, -f.w})};
  else return pair_of(f);
}

// v[r] *= b s^r, r < RS <= 32, from b, s and s4 = s^4, each looked up: a factor
// is at most RS / 4 + 2 rounded products away from them (RS / 4 - 2 for the
// power of s4, two for that of s, two that join them with b; 6 at RS = 16, 10 at
// 32), where powers of s alone would multiply its rounding error by r.
template <int RS>
__device__ __forceinline__ void pair_scale_powers(Pair* v, Pair b, Pair s, Pair s4) {
  Pair lo[4];
  lo[1] = s;
  if constexpr (RS > 2) lo[2] = pmul(s, s);
  if constexpr (RS > 3) lo[3] = pmul(lo[2], s);
  Pair h = b, q4 = s4;  // q4 = s^(4j)
#pragma unroll
  for (int j = 0; j < (RS + 3) / 4; ++j) {
    if (j > 0) h = pmul(b, q4);
#pragma unroll
    for (int i = 0; i < 4 && 4 * j + i < RS; ++i) v[4 * j + i] = pmul(v[4 * j + i], i == 0 ? h : pmul(h, lo[i]));
    if (j > 0 && 4 * j + 4 < RS) q4 = pmul(q4, s4);
  }
}

// Load policies: ld(row, c) reads a row of pair c; twiddle(v, t, c) scales the
// first stage's RS inputs of rows t + r STRIDE.
struct PairNoTwiddle {
  template <int RS, int STRIDE, int DIR>
  __device__ __forceinline__ void twiddle(Pair*, int, int) const {}
};
// W_M^(k row) for one k and every column of the tile
struct PairRowTwiddle {
  BigTwiddle bt;
  unsigned k;
  template <int RS, int STRIDE, int DIR>
  __device__ __forceinline__ void twiddle(Pair* v, int t, int) const {
    const Pair s4 = RS > 4 ? pbroadcast(pair_twiddle<DIR>(bt, k * STRIDE * 4)) : Pair{};
    pair_scale_powers<RS>(v, pbroadcast(pair_twiddle<DIR>(bt, k * t)), pbroadcast(pair_twiddle<DIR>(bt, k * STRIDE)),
                          s4);
  }
};

template <typename TW>
struct PairLoad : TW {
  const float2* in;  // row 0, column 0 of the tile
  int64_t pitch;
  __device__ __forceinline__ Pair operator()(int row, int c) const {
    const float4* p = reinterpret_cast<const float4*>(in + row * pitch) + c;
    return pair_of(__ldcg(p));
  }
};

// Store policies: ROWS_FIRST takes the last stage's rows with consecutive
// threads on consecutive rows of one pair.
struct PairNoFactors {
  template <typename ST>
  __device__ __forceinline__ void begin(const ST&, int, int) {}
  __device__ __forceinline__ void scale(Pair*) const {}
};
template <bool SCALE, bool CG>
struct PairStoreRows {
  static constexpr bool ROWS_FIRST = false;
  template <int RS, int P, int DIR> using Factors = PairNoFactors;
  float2* out;
  int64_t pitch;
  float scale;
  __device__ __forceinline__ void operator()(int row, int c, Pair o) const {
    if constexpr (SCALE) {
      const V2 s(float2{scale, scale});
      o = Pair{o.x * s, o.y * s};
    }
    float4* p = reinterpret_cast<float4*>(out + row * pitch) + c;
    if constexpr (CG) __stcg(p, pair_raw(o));
    else __stcs(p, pair_raw(o));
  }
};
// column c of the tile times W_N^(k row), k = col0 + its index, as a row of
// `pitch` elements.  The table lookups are issued (begin) before the last
// stage reads its inputs; s[k] = W_N^(k P) and s4[k] = W_N^(4 k P) come from
// tables of their own, one load for both columns.
struct PairStoreTransposed {
  static constexpr bool ROWS_FIRST = true;
  float2* out;  // of column 0
  int64_t pitch;
  BigTwiddle bt;
  const float2 *ts, *ts4;
  unsigned col0;
  template <int RS, int P, int DIR>
  struct Factors {
    Pair b, s, s4;
    __device__ __forceinline__ void begin(const PairStoreTransposed& st, int row0, int c) {
      const unsigned k = st.col0 + 2 * c;
      float2 w = __ldg(static_cast<const float2*>(st.bt.lo) + row0);  // row0 < L <= sqrt N: W_N^row0
      if constexpr (DIR > 0) w.y = -w.y;
      const float2 b0 = pair_twiddle<DIR>(st.bt, k * row0);
      b = two(b0, cmul(b0, w));
      s = pair_table<DIR>(st.ts, k);
      if constexpr (RS > 4) s4 = pair_table<DIR>(st.ts4, k);
    }
    __device__ __forceinline__ void scale(Pair* v) const { pair_scale_powers<RS>(v, b, s, s4); }
  };
  __device__ __forceinline__ void operator()(int row, int c, Pair o) const {
    float2* p = out + 2 * c * pitch + row;
    __stcg(p, float2{o.x.v.x, o.y.v.x});
    __stcg(p + pitch, float2{o.x.v.y, o.y.v.y});
  }
};

template <int L, int EPT, int NP, int DIR, int P, typename LD, typename ST>
__device__ __forceinline__ void pair_stage(Pair* v, float4* sh, int t, int c, const float2* __restrict__ tw,
                                           const LD& ld, const ST& st) {
  using S = PairShape<L, EPT, NP>;
  using SC = Sched<L, EPT>;
  constexpr int T = S::T, RS = SC::radix_at(P), Q = EPT / RS, STRIDE = L / RS;
  constexpr bool FIRST = P == 1, LAST = P * RS == L;
  if constexpr (LAST && ST::ROWS_FIRST) {
    t = threadIdx.x % T;
    c = threadIdx.x / T;
  }
  [[maybe_unused]] typename ST::template Factors<RS, P, DIR> f[LAST ? Q : 1];
  if constexpr (LAST)
#pragma unroll
    for (int q = 0; q < Q; ++q) f[q].begin(st, t + q * T, c);
  if constexpr (FIRST) {
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
      for (int r = 0; r < RS; ++r) v[q * RS + r] = ld(t + q * T + r * STRIDE, c);
  } else {
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
      for (int r = 0; r < RS; ++r) {
        const float4 x = sh[S::phys(t + q * T + r * STRIDE, c)];
        v[q * RS + r] = Pair{V2(float2{x.x, x.y}), V2(float2{x.z, x.w})};
      }
  }
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    if constexpr (FIRST) {
      ld.template twiddle<RS, STRIDE, DIR>(v + q * RS, t + q * T, c);
    } else {
      PairPowers<RS> pw;
      pw.template load<DIR>(tw, ((t + q * T) & (P - 1)) * (L / (P * RS)));
      pw.apply(v + q * RS);
    }
    pdft<RS, DIR>(v + q * RS);
    if constexpr (LAST) f[q].scale(v + q * RS);
  }
  if constexpr (LAST) {
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
      for (int r = 0; r < RS; ++r) st(t + q * T + r * P, c, v[q * RS + r]);
  } else {
    if constexpr (!FIRST) __syncthreads();
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int i = t + q * T, k = i & (P - 1), j = (i - k) * RS + k;
#pragma unroll
      for (int r = 0; r < RS; ++r) {
        const Pair a = v[q * RS + r];
        sh[S::phys(j + r * P, c)] = float4{a.x.v.x, a.x.v.y, a.y.v.x, a.y.v.y};
      }
    }
    __syncthreads();
    pair_stage<L, EPT, NP, DIR, P * RS>(v, sh, t, c, tw, ld, st);
  }
}

template <int L, int EPT, int NP, int DIR, typename LD, typename ST>
__device__ __forceinline__ void pair_columns(float4* sh, const float2* __restrict__ tw, const LD& ld, const ST& st) {
  Pair v[EPT];
  pair_stage<L, EPT, NP, DIR, 1>(v, sh, threadIdx.x / NP, threadIdx.x % NP, tw, ld, st);
}

// Rows at a run-time pitch (in pairs; a tile spans less than 2^32 pairs), for
// tiles whose last pairs may lie beyond the array (active = false).
template <typename TW>
struct PairStridedLoad : TW {
  const float4* in;
  unsigned pitch;
  bool active;
  __device__ __forceinline__ Pair operator()(int row, int c) const {
    return active ? pair_of(__ldcg(in + (unsigned(row) * pitch + unsigned(c)))) : Pair{V2(0.0), V2(0.0)};
  }
};
template <bool SCALE>
struct PairStridedStore {
  static constexpr bool ROWS_FIRST = false;
  template <int RS, int P, int DIR> using Factors = PairNoFactors;
  float4* out;
  unsigned pitch;
  bool active;
  float scale;
  __device__ __forceinline__ void operator()(int row, int c, Pair o) const {
    if constexpr (SCALE) {
      const V2 s(float2{scale, scale});
      o = Pair{o.x * s, o.y * s};
    }
    if (active) __stcs(out + (unsigned(row) * pitch + unsigned(c)), pair_raw(o));
  }
};

struct PairPassParams {
  const float2* src;
  float2* dst;
  float2* scratch;
  int64_t idist, odist;
  const float2 *tw1, *tw2, *tw3;  // W_L of the passes
  BigTwiddle bt, btm;             // W_N, W_M (three passes)
  const float2 *ts, *ts4;         // W_N^(k P1), W_N^(4 k P1), P1 = prefix product of pass 1's last stage
  float scale;
};

// Two passes, N = N1 N2: Y[n2][k1] = columns of x, x W_N^(n2 k1); X[k1 + N1 k2]
// = columns of Y.  One tile per CTA, tiles of a transform adjacent.
template <int N1, int64_t N2, int EPT, int NP, int DIR, int MINB>
__global__ void __launch_bounds__(PairShape<N1, EPT, NP>::TPB, MINB) k_pair_tp1(PairPassParams p) {
  asm volatile("griddepcontrol.launch_dependents;");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int TILES = int(N2 / (2 * NP));
  const int64_t b = blockIdx.x / TILES;
  const int col0 = int(blockIdx.x % TILES) * 2 * NP;
  const PairLoad<PairNoTwiddle> ld{{}, p.src + b * p.idist + col0, N2};
  const PairStoreTransposed st{p.scratch + b * (int64_t(N1) * N2) + int64_t(col0) * N1, N1, p.bt, p.ts, p.ts4,
                               unsigned(col0)};
  pair_columns<N1, EPT, NP, DIR>(reinterpret_cast<float4*>(smem_raw), p.tw1, ld, st);
}
template <int N1, int N2, int EPT, int NP, int DIR, int MINB>
__global__ void __launch_bounds__(PairShape<N2, EPT, NP>::TPB, MINB) k_pair_tp2(PairPassParams p) {
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the pass before this one
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int TILES = N1 / (2 * NP);
  const int64_t b = blockIdx.x / TILES;
  const int col0 = int(blockIdx.x % TILES) * 2 * NP;
  const PairLoad<PairNoTwiddle> ld{{}, p.scratch + b * (int64_t(N1) * N2) + col0, N1};
  const PairStoreRows<(DIR > 0), false> st{p.dst + b * p.odist + col0, N1, p.scale};
  pair_columns<N2, EPT, NP, DIR>(reinterpret_cast<float4*>(smem_raw), p.tw2, ld, st);
}

// Three passes, N = N1 M, M = M1 M2 (index maps of k_tp3): pass 1 as above
// with N2 = M; pass 2 over m1, in place on Y[M2 m1 + m2][k1]; pass 3 over m2,
// x W_M^(m2 k'1), natural order.
template <int N1, int M1, int M2, int EPT, int NP, int DIR, int MINB>
__global__ void __launch_bounds__(PairShape<M1, EPT, NP>::TPB, MINB) k_pair_tp3b(PairPassParams p) {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int G = N1 / (2 * NP), TILES = M2 * G;
  const int64_t b = blockIdx.x / TILES;
  const int r = int(blockIdx.x % TILES), m2 = r / G, col0 = (r % G) * 2 * NP;
  float2* y = p.scratch + b * (int64_t(N1) * M1 * M2) + int64_t(m2) * N1 + col0;
  const PairLoad<PairNoTwiddle> ld{{}, y, int64_t(M2) * N1};
  const PairStoreRows<false, true> st{y, int64_t(M2) * N1, 1.f};
  pair_columns<M1, EPT, NP, DIR>(reinterpret_cast<float4*>(smem_raw), p.tw2, ld, st);
}
template <int N1, int M1, int M2, int EPT, int NP, int DIR, int MINB>
__global__ void __launch_bounds__(PairShape<M2, EPT, NP>::TPB, MINB) k_pair_tp3c(PairPassParams p) {
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the pass before this one
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int G = N1 / (2 * NP), TILES = M1 * G;
  const int64_t b = blockIdx.x / TILES;
  const int r = int(blockIdx.x % TILES), k1 = r / G, col0 = (r % G) * 2 * NP;
  const PairLoad<PairRowTwiddle> ld{{p.btm, unsigned(k1)},
                                          p.scratch + b * (int64_t(N1) * M1 * M2) + int64_t(M2) * k1 * N1 + col0, N1};
  const PairStoreRows<(DIR > 0), false> st{p.dst + b * p.odist + int64_t(N1) * k1 + col0, int64_t(N1) * M1, p.scale};
  pair_columns<M2, EPT, NP, DIR>(reinterpret_cast<float4*>(smem_raw), p.tw3, ld, st);
}

}  // namespace gfft
