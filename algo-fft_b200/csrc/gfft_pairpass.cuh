#pragma once
#include "gfft_pair.cuh"
namespace gfft {
enum { PAIR_COLS = 0, PAIR_TWT = 1 };

template <int L, int EPT, int NP, int DIR, int P, int MODE, bool TF, typename LD, typename ST>
__device__ __forceinline__ void pair_stage(Pair* v, float4* sh, int t, int c, const float2* __restrict__ tw, LD& ld, ST& st) {
  using S = PairShape<L, EPT, NP>;
  using SC = Sched<L, EPT>;
  constexpr int T = S::T, RS = SC::radix_at(P), Q = EPT / RS, STRIDE = L / RS;
  constexpr bool FIRST = P == 1, LAST = P * RS == L;
  if constexpr (LAST && TF) {  // whole columns per warp from here on
    t = threadIdx.x % T;
    c = threadIdx.x / T;
  }
  if constexpr (LAST) st.template begin<Q, T, P>(t, c);
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
        const float4 f = sh[S::phys(t + q * T + r * STRIDE, c)];
        v[q * RS + r] = Pair{V2(float2{f.x, f.y}), V2(float2{f.z, f.w})};
      }
  }
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    if constexpr (P > 1) {
      const int k = (t + q * T) & (P - 1);
      PairPowers<RS> pw;
      pw.template load<DIR>(tw, k * (L / (P * RS)));
      pw.apply(v + q * RS);
    }
    pdft<RS, DIR>(v + q * RS);
  }
  if constexpr (LAST) {
    st.template finish<Q, RS, T, P>(v, t, c);
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
    pair_stage<L, EPT, NP, DIR, P * RS, MODE, TF>(v, sh, t, c, tw, ld, st);
  }
}

template <bool CG> struct PairLoad {
  const float2* in; int64_t pitch;
  __device__ __forceinline__ Pair operator()(int row, int c) const {
    const float4* p = reinterpret_cast<const float4*>(in + row * pitch) + c;
    return pair_of(CG ? __ldcg(p) : __ldcs(p));
  }
};
template <int DIR> struct PairStoreCols {
  float2* out; int64_t pitch; float scale;
  template <int Q, int T, int P> __device__ __forceinline__ void begin(int, int) {}
  template <int Q, int RS, int T, int P> __device__ __forceinline__ void finish(Pair* v, int t, int c) {
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
      for (int r = 0; r < RS; ++r) {
        Pair o = v[q * RS + r];
        if constexpr (DIR > 0) { const V2 s(float2{scale, scale}); o = Pair{o.x * s, o.y * s}; }
        __stcs(reinterpret_cast<float4*>(out + int64_t(t + q * T + r * P) * pitch) + c, pair_raw(o));
      }
  }
};
// times W_N^{n2 k1}, stored as rows of length N1: Y[n2][k1]
template <int DIR> struct PairStoreTwT {
  float2* y; int64_t n1; int col0; BigTwiddle bt;
  float2 s0, s1, b0[16], b1[16];
  template <int Q, int T, int P> __device__ __forceinline__ void begin(int t, int c) {
    const int64_t m = col0 + 2 * c;
    s0 = big_twiddle<float2, DIR>(bt, m * P); s1 = big_twiddle<float2, DIR>(bt, (m + 1) * P);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      b0[q] = big_twiddle<float2, DIR>(bt, m * (t + q * T)); b1[q] = big_twiddle<float2, DIR>(bt, (m + 1) * (t + q * T));
    }
  }
  template <int Q, int RS, int T, int P> __device__ __forceinline__ void finish(Pair* v, int t, int c) {
    Pair pw[RS];
    pw[1] = (Pair{V2(float2{s0.x, s1.x}), V2(float2{s0.y, s1.y})});
#pragma unroll
    for (int r = 2; r < RS; ++r) pw[r] = pmul(pw[r / 2], pw[r - r / 2]);
    float2* y0 = y + int64_t(col0 + 2 * c) * n1;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const Pair b = (Pair{V2(float2{b0[q].x, b1[q].x}), V2(float2{b0[q].y, b1[q].y})});
#pragma unroll
      for (int r = 0; r < RS; ++r) {
        const Pair o = pmul(v[q * RS + r], r == 0 ? b : pmul(b, pw[r]));
        const int row = t + q * T + r * P;
        __stcg(y0 + row, float2{o.x.v.x, o.y.v.x});
        __stcg(y0 + n1 + row, float2{o.x.v.y, o.y.v.y});
      }
    }
  }
};
struct PairParams { const float2* src; float2* dst; float2* scratch; int64_t idist, odist; const float2* tw1; const float2* tw2; BigTwiddle bt; float scale; };

template <int N1, int N2, int EPT, int NP, int DIR, bool TF, int MINB>
__global__ void __launch_bounds__(PairShape<N1, EPT, NP>::TPB, MINB) k_pair1(PairParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float4* sh = reinterpret_cast<float4*>(smem_raw);
  constexpr int TILES = N2 / (2 * NP);
  const int64_t bl = blockIdx.x / TILES;
  const int col0 = int(blockIdx.x % TILES) * 2 * NP;
  PairLoad<false> ld{p.src + bl * p.idist + col0, N2};
  PairStoreTwT<DIR> st; st.y = p.scratch + bl * int64_t(N1) * N2; st.n1 = N1; st.col0 = col0; st.bt = p.bt;
  Pair v[EPT];
  pair_stage<N1, EPT, NP, DIR, 1, PAIR_TWT, TF>(v, sh, threadIdx.x / NP, threadIdx.x % NP, p.tw1, ld, st);
}
template <int N1, int N2, int EPT, int NP, int DIR, int MINB>
__global__ void __launch_bounds__(PairShape<N2, EPT, NP>::TPB, MINB) k_pair2(PairParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float4* sh = reinterpret_cast<float4*>(smem_raw);
  constexpr int TILES = N1 / (2 * NP);
  const int64_t bl = blockIdx.x / TILES;
  const int col0 = int(blockIdx.x % TILES) * 2 * NP;
  PairLoad<true> ld{p.scratch + bl * int64_t(N1) * N2 + col0, N1};
  PairStoreCols<DIR> st{p.dst + bl * p.odist + col0, N1, p.scale};
  Pair v[EPT];
  pair_stage<N2, EPT, NP, DIR, 1, PAIR_COLS, false>(v, sh, threadIdx.x / NP, threadIdx.x % NP, p.tw2, ld, st);
}
}
