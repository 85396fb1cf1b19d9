// Pairs of complex64 elements in packed FP32 arithmetic, and column-tile
// FFT stages on them.
//
// sm_100a issues two FP32 operations of one thread as one instruction when
// the operands sit in 64-bit register pairs (add/sub/mul/fma .f32x2).  The
// FMA pipe runs no faster for it (measured: 117-127 lane operations per SM
// cycle either way), but the instruction count halves, and the column passes
// are bound by instruction issue and the latencies around it.  The two
// halves of a pair are the same row of two adjacent columns, real parts and
// imaginary parts in one register pair each, so every butterfly, rotation
// and twiddle of a column FFT is the same packed instruction for both.
#pragma once
#include "gfft_math.cuh"
#include "gfft_sched.cuh"

namespace gfft {

// Two FP32 lanes.
struct V2 {
  float2 v;
  V2() = default;
  __device__ __forceinline__ constexpr V2(float2 a) : v(a) {}
  __device__ __forceinline__ constexpr explicit V2(double a) : v{float(a), float(a)} {}
};

__device__ __forceinline__ V2 operator+(V2 a, V2 b) { return V2(__fadd2_rn(a.v, b.v)); }
__device__ __forceinline__ V2 operator*(V2 a, V2 b) { return V2(__fmul2_rn(a.v, b.v)); }
__device__ __forceinline__ V2 fma2(V2 a, V2 b, V2 c) { return V2(__ffma2_rn(a.v, b.v, c.v)); }
// Negation is an operand modifier of the packed instructions (an fma2 of a
// negated operand ran at the rate of the plain one).
__device__ __forceinline__ V2 operator-(V2 a) { return V2(float2{-a.v.x, -a.v.y}); }
__device__ __forceinline__ V2 operator-(V2 a, V2 b) { return a + (-b); }

// The same row of two adjacent columns.
struct Pair {
  V2 x, y;
};
template <> struct RealOf<Pair> { using type = V2; };

__device__ __forceinline__ Pair pmul(Pair a, Pair w) {
  return Pair{fma2(-a.y, w.y, a.x * w.x), fma2(a.y, w.x, a.x * w.y)};
}
__device__ __forceinline__ Pair pbroadcast(float2 w) {  // one factor for both lanes
  return Pair{V2(float2{w.x, w.x}), V2(float2{w.y, w.y})};
}

// a + DIR i b and a - DIR i b
template <int DIR>
__device__ __forceinline__ Pair padd_i(Pair a, Pair b) {
  if constexpr (DIR > 0) return Pair{a.x - b.y, a.y + b.x};
  else return Pair{a.x + b.y, a.y - b.x};
}

// a * exp(DIR 2 pi i M / R)
template <int R, int M, int DIR>
__device__ __forceinline__ Pair ptwc(Pair a) {
  constexpr int m = ((M % R) + R) % R;
  if constexpr (m == 0) return a;
  else if constexpr (2 * m == R) return Pair{-a.x, -a.y};
  else if constexpr (4 * m == R) {
    if constexpr (DIR > 0) return Pair{-a.y, a.x};
    else return Pair{a.y, -a.x};
  } else if constexpr (4 * m == 3 * R) {
    if constexpr (DIR > 0) return Pair{a.y, -a.x};
    else return Pair{-a.y, a.x};
  } else {
    constexpr double c = root_cos<R>(m);
    constexpr double s = DIR * root_sin<R>(m);
    return Pair{fma2(a.y, V2(-s), a.x * V2(c)), fma2(a.x, V2(s), a.y * V2(c))};
  }
}

template <int R, int R1, int R2, int DIR, int IDX = 0>
__device__ __forceinline__ void ptwiddle_block(Pair* a) {
  if constexpr (IDX < R) {
    constexpr int n2 = IDX / R1, k1 = IDX % R1;
    a[IDX] = ptwc<R, n2 * k1, DIR>(a[IDX]);
    ptwiddle_block<R, R1, R2, DIR, IDX + 1>(a);
  }
}

// Odd prime radix (3, 5, 7): dft_odd on pairs.
template <int R, int K, int J>
__device__ __forceinline__ void podd_accum(Pair& a, Pair& b, const Pair* s, const Pair* d) {
  if constexpr (J <= (R - 1) / 2) {
    const V2 c(cos_r<R>((J * K) % R)), sn(sin_r<R>((J * K) % R));
    a = Pair{fma2(s[J].x, c, a.x), fma2(s[J].y, c, a.y)};
    if constexpr (J == 1) b = Pair{d[J].x * sn, d[J].y * sn};
    else b = Pair{fma2(d[J].x, sn, b.x), fma2(d[J].y, sn, b.y)};
    podd_accum<R, K, J + 1>(a, b, s, d);
  }
}
template <int R, int K, int DIR>
__device__ __forceinline__ void podd_out(Pair* v, const Pair* s, const Pair* d, Pair x0) {
  if constexpr (K <= (R - 1) / 2) {
    Pair a = x0, b;
    podd_accum<R, K, 1>(a, b, s, d);
    v[K] = padd_i<DIR>(a, b);
    v[R - K] = padd_i<-DIR>(a, b);
    podd_out<R, K + 1, DIR>(v, s, d, x0);
  }
}

// In-register DFT of R pairs (7-smooth R up to 64), natural order.
template <int R, int DIR>
__device__ __forceinline__ void pdft(Pair* v) {
  if constexpr (R == 1) {
  } else if constexpr (R == 2) {
    const Pair a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  } else if constexpr (R == 4) {
    const Pair t0 = cadd(v[0], v[2]), t1 = csub(v[0], v[2]);
    const Pair t2 = cadd(v[1], v[3]), d = csub(v[1], v[3]);
    v[0] = cadd(t0, t2);
    v[2] = csub(t0, t2);
    v[1] = padd_i<DIR>(t1, d);
    v[3] = padd_i<-DIR>(t1, d);
  } else if constexpr (R == 3 || R == 5 || R == 7) {
    constexpr int H = (R - 1) / 2;
    Pair s[H + 1], d[H + 1];
#pragma unroll
    for (int j = 1; j <= H; ++j) {
      s[j] = cadd(v[j], v[R - j]);
      d[j] = csub(v[j], v[R - j]);
    }
    const Pair x0 = v[0];
    Pair sum = x0;
#pragma unroll
    for (int j = 1; j <= H; ++j) sum = cadd(sum, s[j]);
    podd_out<R, 1, DIR>(v, s, d, x0);
    v[0] = sum;
  } else {
    constexpr int R1 = dft_split(R), R2 = R / R1;
    Pair a[R];
#pragma unroll
    for (int n2 = 0; n2 < R2; ++n2) {
      Pair t[R1];
#pragma unroll
      for (int n1 = 0; n1 < R1; ++n1) t[n1] = v[R2 * n1 + n2];
      pdft<R1, DIR>(t);
#pragma unroll
      for (int k1 = 0; k1 < R1; ++k1) a[n2 * R1 + k1] = t[k1];
    }
    ptwiddle_block<R, R1, R2, DIR>(a);
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) {
      Pair t[R2];
#pragma unroll
      for (int n2 = 0; n2 < R2; ++n2) t[n2] = a[n2 * R1 + k1];
      pdft<R2, DIR>(t);
#pragma unroll
      for (int k2 = 0; k2 < R2; ++k2) v[k1 + R1 * k2] = t[k2];
    }
  }
}

// Powers w^r, r < RS <= 64, of one factor per thread from exactly rounded
// table entries: lo[1], lo[2], lo[4] and hi[h] = w^(8h) are loaded, the others
// are products of two (w^r = lo[r mod 8] hi[r / 8]).  A tree that starts from
// w alone multiplies its rounding error by r.
template <int RS>
struct PairPowers {
  static constexpr int NL = RS < 8 ? RS : 8, NH = (RS + 7) / 8;
  Pair lo[NL], hi[NH];
  // tw[i step] = w^i
  template <int DIR>
  __device__ __forceinline__ void load(const float2* __restrict__ tw, int step) {
    auto get = [&](int i) {
      float2 f = __ldg(tw + i * step);
      if constexpr (DIR > 0) f.y = -f.y;
      return pbroadcast(f);
    };
#pragma unroll
    for (int r = 1; r < NL; r *= 2) lo[r] = get(r);
    if constexpr (NL > 3) lo[3] = pmul(lo[2], lo[1]);
    if constexpr (NL > 5) lo[5] = pmul(lo[4], lo[1]);
    if constexpr (NL > 6) lo[6] = pmul(lo[4], lo[2]);
    if constexpr (NL > 7) lo[7] = pmul(lo[4], lo[3]);
#pragma unroll
    for (int h = 1; h < NH; ++h) hi[h] = get(8 * h);
  }
  // v[r] *= w^r
  __device__ __forceinline__ void apply(Pair* v) const {
#pragma unroll
    for (int r = 1; r < RS; ++r) {
      const int a = r % 8, b = r / 8;
      if (b == 0) v[r] = pmul(v[r], lo[a]);
      else if (a == 0) v[r] = pmul(v[r], hi[b]);
      else v[r] = pmul(v[r], pmul(lo[a], hi[b]));
    }
  }
};

// Global accesses of one row of a pair of columns: 16 bytes (re0, im0, re1, im1).
__device__ __forceinline__ Pair pair_of(float4 f) { return Pair{V2(float2{f.x, f.z}), V2(float2{f.y, f.w})}; }
__device__ __forceinline__ float4 pair_raw(Pair p) { return float4{p.x.v.x, p.y.v.x, p.x.v.y, p.y.v.y}; }

// Tile of NP column pairs of length L in shared memory, 16 bytes (re0, re1,
// im0, im1) per row and pair.  An 8-lane group of a 16-byte access must cover
// the 8 slots of 16 bytes of a 128-byte bank row.  The slot of (row, c) is
// chosen so that three patterns do: consecutive c then consecutive rows (stage
// reads, direct loads), consecutive c then rows EPT apart (the first stage's
// writes) and consecutive rows of one c (a last stage that stores whole
// columns).
template <int L, int EPT, int NP>
struct PairShape {
  static_assert(NP == 2 || NP == 4 || NP == 8 || NP == 16 || NP == 32, "2 to 32 column pairs per tile");
  static constexpr int T = L / EPT;
  static constexpr int TPB = T * NP;
  static constexpr int SMEM = L * NP * 16;
  static constexpr int LE = EPT == 4 ? 2 : EPT == 8 ? 3 : EPT == 16 ? 4 : 5;
  __device__ static __forceinline__ int phys(int row, int c) {
    if constexpr (NP == 2) return (row ^ ((row >> LE) & 3)) * 2 + (c ^ ((row >> 2) & 1));
    else if constexpr (NP == 4) return (row ^ ((row >> LE) & 1)) * 4 + (c ^ ((row >> 1) & 3));
    else return row * NP + (c ^ (row & 7));
  }
};

}  // namespace gfft
