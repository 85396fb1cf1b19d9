// Single-CTA complex64 transforms on packed pairs within one transform.
//
// N = R1 R2 R3 with R1 = 2 EP.  Index maps (decimation in frequency):
//   n = M n1 + m, m = R3 n2 + n3, M = R2 R3;   k = K1 + R1 (k2 + R2 k3).
// Stage 1: thread m holds x[M n1 + m] for every n1.  A radix-2 step over
// (n1, n1 + EP) gives the inputs of two EP-point DFTs, whose outputs are the
// even K1 and the odd K1; they run as the two lanes of packed arithmetic, and
// so do the stages after it: the pair (2 k1, 2 k1 + 1) stays together.
// Stages 2 and 3 are DFTs over n2 and n3 of each pair, with the twiddles
// W_N^(K1 m) and W_M^(k2 n3) applied where a stage's outputs are written.
// Each exchange goes through shared memory in 16-byte pairs, in place (a
// stage writes the slots it read), so a transform needs one barrier per
// exchange.  The inverse of a product (convolution) runs the same stages
// backwards from the registers stage 3 ends in, without reordering the bins.
#pragma once
#include "gfft_pair.cuh"

namespace gfft {

template <int N_, int EP_, int R2_, int R3_>
struct PairRow {
  static constexpr int N = N_, EP = EP_, R2 = R2_, R3 = R3_;
  static constexpr int R1 = 2 * EP, M = R2 * R3;
  static constexpr int T = M;                        // threads
  static constexpr int Q2 = EP / R2, Q3 = EP / R3;   // butterflies per thread of stages 2 and 3
  static constexpr int SMEM = N / 2 * 16;
  static_assert(R1 * R2 * R3 == N && EP % R2 == 0 && EP % R3 == 0 && R3 >= 8 && EP >= 8, "unsupported split");

  // Slot of pair k1 (K1 = 2 k1, 2 k1 + 1) at m: runs of consecutive m (stages
  // 1 and 2) and of consecutive k1 (stage 3) both cover all 16-byte slots of a
  // bank row in 8 lanes.
  __device__ static __forceinline__ int slot(int k1, int m) { return k1 * M + (m ^ (k1 & 7)); }
  __device__ static __forceinline__ void put(float4* sh, int s, Pair a) {
    sh[s] = float4{a.x.v.x, a.x.v.y, a.y.v.x, a.y.v.y};
  }
  __device__ static __forceinline__ Pair get(const float4* sh, int s) {
    const float4 f = sh[s];
    return Pair{V2(float2{f.x, f.y}), V2(float2{f.z, f.w})};
  }

  // (n1, n1 + EP) -> lanes: s = x0 + x1, d = (x0 - x1) W_R1^(n1), and back
  template <int J, int DIR>
  __device__ static __forceinline__ Pair split(float2 x0, float2 x1) {
    const float2 s = cadd(x0, x1), d = twc<R1, J, DIR>(csub(x0, x1));
    return Pair{V2(float2{s.x, d.x}), V2(float2{s.y, d.y})};
  }
  template <int J, int DIR>
  __device__ static __forceinline__ void join(Pair p, float2* x0, float2* x1) {
    const float2 s{p.x.v.x, p.y.v.x}, d = twc<R1, J, DIR>(float2{p.x.v.y, p.y.v.y});
    *x0 = cadd(s, d);
    *x1 = csub(s, d);
  }
  template <int DIR, int J, typename LD>
  __device__ static __forceinline__ void load_all(Pair* v, int t, const LD& ld) {
    if constexpr (J < EP) {
      v[J] = split<J, DIR>(ld(J * M + t), ld((J + EP) * M + t));
      load_all<DIR, J + 1>(v, t, ld);
    }
  }
  template <int DIR, int J, typename ST>
  __device__ static __forceinline__ void store_all(const Pair* v, int t, const ST& st) {
    if constexpr (J < EP) {
      float2 x0, x1;
      join<J, DIR>(v[J], &x0, &x1);
      st(J * M + t, x0);
      st((J + EP) * M + t, x1);
      store_all<DIR, J + 1>(v, t, st);
    }
  }

  // v[k] *= (W_N^(2k t), W_N^((2k+1) t)) (conjugated for DIR > 0)
  template <int DIR>
  __device__ static __forceinline__ void twiddle1(Pair* v, int t, const float2* __restrict__ tw) {
    PairPowers<EP> pw;
    pw.template load<DIR>(tw, 2 * t);
    float2 w = __ldg(tw + t);
    if constexpr (DIR > 0) w.y = -w.y;
    const Pair one_w{V2(float2{1.f, w.x}), V2(float2{0.f, w.y})};
#pragma unroll
    for (int b = 0; b < PairPowers<EP>::NH; ++b) {
      const Pair h = b == 0 ? one_w : pmul(one_w, pw.hi[b]);
#pragma unroll
      for (int a = 0; a < 8; ++a) v[8 * b + a] = pmul(v[8 * b + a], a == 0 ? h : pmul(pw.lo[a], h));
    }
  }

  // Forward: ld(n) -> registers v[q R3 + k3] = bins (K1 = 2 k1 + lane, k2, k3)
  // with u = t + q T, k1 = u mod EP, k2 = u / EP.
  template <int DIR, typename LD>
  __device__ static __forceinline__ void forward(Pair* v, float4* sh, int t, const float2* __restrict__ tw,
                                                 const LD& ld) {
    load_all<DIR, 0>(v, t, ld);
    pdft<EP, DIR>(v);
    twiddle1<DIR>(v, t, tw);
#pragma unroll
    for (int k = 0; k < EP; ++k) put(sh, slot(k, t), v[k]);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < Q2; ++q) {
      const int u = t + q * T, n3 = u % R3, k1 = u / R3;
#pragma unroll
      for (int r = 0; r < R2; ++r) v[q * R2 + r] = get(sh, slot(k1, r * R3 + n3));
    }
#pragma unroll
    for (int q = 0; q < Q2; ++q) {
      const int u = t + q * T, n3 = u % R3, k1 = u / R3;
      pdft<R2, DIR>(v + q * R2);
      PairPowers<R2> pw;
      pw.template load<DIR>(tw, R1 * n3);
      pw.apply(v + q * R2);
#pragma unroll
      for (int r = 0; r < R2; ++r) put(sh, slot(k1, r * R3 + n3), v[q * R2 + r]);
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < Q3; ++q) {
      const int u = t + q * T, k1 = u % EP, k2 = u / EP;
#pragma unroll
      for (int r = 0; r < R3; ++r) v[q * R3 + r] = get(sh, slot(k1, k2 * R3 + r));
    }
#pragma unroll
    for (int q = 0; q < Q3; ++q) pdft<R3, DIR>(v + q * R3);
  }

  // The stages of forward() backwards, from the bins it leaves in v to
  // st(n, value); unscaled.
  template <int DIR, typename ST>
  __device__ static __forceinline__ void backward(Pair* v, float4* sh, int t, const float2* __restrict__ tw,
                                                  const ST& st) {
#pragma unroll
    for (int q = 0; q < Q3; ++q) {
      const int u = t + q * T, k1 = u % EP, k2 = u / EP;
      pdft<R3, DIR>(v + q * R3);
      PairPowers<R3> pw;
      pw.template load<DIR>(tw, R1 * k2);
      pw.apply(v + q * R3);
#pragma unroll
      for (int r = 0; r < R3; ++r) put(sh, slot(k1, k2 * R3 + r), v[q * R3 + r]);
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < Q2; ++q) {
      const int u = t + q * T, n3 = u % R3, k1 = u / R3;
#pragma unroll
      for (int r = 0; r < R2; ++r) v[q * R2 + r] = get(sh, slot(k1, r * R3 + n3));
    }
#pragma unroll
    for (int q = 0; q < Q2; ++q) {
      const int u = t + q * T, n3 = u % R3, k1 = u / R3;
      pdft<R2, DIR>(v + q * R2);
#pragma unroll
      for (int r = 0; r < R2; ++r) put(sh, slot(k1, r * R3 + n3), v[q * R2 + r]);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < EP; ++k) v[k] = get(sh, slot(k, t));
    twiddle1<DIR>(v, t, tw);
    pdft<EP, DIR>(v);
    store_all<DIR, 0>(v, t, st);
  }
};

}  // namespace gfft
