// Convolution and correlation (K11): Convolve / Convolve128 (convolve.go),
// ConvolveReal (convolve_real.go), CrossCorrelate / AutoCorrelate
// (correlate.go), and a batched ConvolveReal with one shared kernel.
//
// Same algorithm as the reference: complex convolution at the exact length
// len(a)+len(b)-1 (so it may run Bluestein), real convolution at
// NextPow2(len(a)+len(b)-1) (at least 2) -- except for long real signals
// with a short kernel (len(b) - 1 <= L/4 for an L <= 2^15 block and more
// than two blocks of output), which run overlap-save (k_conv_pair for
// float32, k_conv_os for float64): the same linear convolution from
// single-CTA transforms.  The two forward transforms run
// as one batch of two, the pointwise product is one elementwise kernel
// (internal/fft/complex_mul.go:23), the inverse writes straight into a
// padded buffer whose head is the result.  Plans come from a process-wide
// cache keyed by (precision, kind, length) instead of being rebuilt on
// every call as the reference does (convolve.go:23, convolve_real.go:30).
#include <map>
#include <mutex>
#include <tuple>
#include "gfft_internal.h"
#include "gfft_pairrow.cuh"
#include "gfft_real.cuh"

namespace gfft {

namespace {

std::mutex g_cache_mu;
std::map<std::tuple<int, int, int64_t>, gfft_plan*> g_cplx;     // (device, prec, n)
std::map<std::tuple<int, int, int64_t>, gfft_plan_real*> g_real;  // (device, prec, n)

gfft_status cached_plan(int prec, int64_t n, gfft_plan** out) {
  int dev = 0;
  GFFT_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> g(g_cache_mu);
  auto key = std::make_tuple(dev, prec, n);
  auto it = g_cplx.find(key);
  if (it != g_cplx.end()) {
    *out = it->second;
    return GFFT_OK;
  }
  gfft_plan_options o{};
  o.device = dev;
  gfft_status s = gfft_plan_new(out, prec, n, &o);
  if (s == GFFT_OK) g_cplx[key] = *out;
  return s;
}

gfft_status cached_real_plan(int prec, int64_t n, gfft_plan_real** out) {
  int dev = 0;
  GFFT_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> g(g_cache_mu);
  auto key = std::make_tuple(dev, prec, n);
  auto it = g_real.find(key);
  if (it != g_real.end()) {
    *out = it->second;
    return GFFT_OK;
  }
  gfft_plan_options o{};
  o.device = dev;
  gfft_status s = gfft_plan_real_new(out, prec, n, &o);
  if (s == GFFT_OK) g_real[key] = *out;
  return s;
}

unsigned grid1(int64_t total) { return unsigned(std::max<int64_t>(1, std::min<int64_t>((total + 255) / 256, 148 * 32))); }

// rows of `w` elements: row r = src_r padded with zeros (reverse+conj when
// `rev` is set: the correlate operand of correlate.go:26-32).
template <typename T>
__global__ void k_pad(T* dst, int64_t w, const T* src, int64_t len, int64_t sdist, int64_t rows, bool rev) {
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < rows * w; e += int64_t(gridDim.x) * blockDim.x) {
    const int64_t r = e / w, i = e % w;
    T v{};
    if (i < len) v = src[r * sdist + (rev ? len - 1 - i : i)];
    dst[e] = v;
  }
}

template <typename T>
__global__ void k_pad_conj(T* dst, int64_t w, const T* src, int64_t len) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < w; i += int64_t(gridDim.x) * blockDim.x)
    dst[i] = i < len ? cconj(src[len - 1 - i]) : T{0, 0};
}

// A[r][k] *= B[r*bdist + k]: each of `rows` spectra of w bins times the
// shared spectrum B (bdist = 0) or its own row of B (bdist = w).
template <typename C>
__global__ void k_cmul_rows(C* A, const C* B, int64_t w, int64_t rows, int64_t bdist) {
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < rows * w; e += int64_t(gridDim.x) * blockDim.x) {
    const int64_t r = e / w, k = e % w;
    A[e] = cmul(A[e], B[r * bdist + k]);
  }
}

template <typename T>
__global__ void k_take_rows(T* dst, int64_t ddist, const T* src, int64_t sdist, int64_t len, int64_t rows) {
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < rows * len; e += int64_t(gridDim.x) * blockDim.x) {
    const int64_t r = e / len, i = e % len;
    dst[r * ddist + i] = src[r * sdist + i];
  }
}

// ---- overlap-save for long real signals ------------------------------------
//
// Block j of a signal produces outputs [j B, j B + B) from the input window
// [j B - (nb - 1), j B - (nb - 1) + L), B = L - (nb - 1): a real transform of
// length L = 2H of the window, the product with the kernel's spectrum (L/2+1
// bins, shared by every block and signal, L2-resident), and the inverse
// real transform, whose samples from nb - 1 on are the linear convolution.
// One CTA slot per block does all of it in shared memory: the window loads
// straight into the first Stockham stage, the R2C recombination, the
// product and the C2R packing happen pairwise (k, H - k) between the two
// half-length transforms, and the last stage stores the B new samples.
// HBM sees L/B reads and one write per output sample.

template <typename R>
struct WindowLoad {
  static constexpr bool kShared = false;
  const R* x;
  int64_t pos0, len;
  bool valid;
  __device__ __forceinline__ Cx<R> operator()(int e) const {
    const int64_t p = pos0 + 2 * int64_t(e);
    Cx<R> v{R(0), R(0)};
    if (valid) {
      if (p >= 0 && p < len) v.x = x[p];
      if (p + 1 >= 0 && p + 1 < len) v.y = x[p + 1];
    }
    return v;
  }
};

template <typename C, int N, int EPT>
struct SharedLoad {
  static constexpr bool kShared = true;
  const C* sh;
  __device__ __forceinline__ C operator()(int e) const { return sh[Pow2Shape<N, EPT, sizeof(C)>::pad(e)]; }
};

template <typename R>
struct WindowStore {
  static constexpr bool kShared = false;
  R* y;
  int64_t pos0, len;  // output index of window sample 0, outputs per signal
  int skip;           // the first nb - 1 window samples are wrapped: not outputs
  R scale;
  bool valid;
  __device__ __forceinline__ void operator()(int e, Cx<R> v) const {
    if (!valid) return;
    const int w = 2 * e;
    const int64_t o = pos0 + w;
    if (w >= skip && o < len) y[o] = v.x * scale;
    if (w + 1 >= skip && o + 1 < len) y[o + 1] = v.y * scale;
  }
};

template <typename C, int H, int EPT>
__global__ void __launch_bounds__(Pow2Shape<H, EPT, sizeof(C)>::TPB)
k_conv_os(const typename RealOf<C>::type* a, typename RealOf<C>::type* dst, int64_t na, int64_t a_dist,
          int64_t dst_dist, int64_t nout, int64_t nblk, int64_t total, int nb, const C* __restrict__ tw,
          const C* __restrict__ wt, const C* __restrict__ hs) {
  using R = typename RealOf<C>::type;
  using S = Pow2Shape<H, EPT, sizeof(C)>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* sh = reinterpret_cast<C*>(smem_raw) + (threadIdx.x / S::T) * S::STRIDE;
  const int t = threadIdx.x % S::T;
  const int64_t g = int64_t(blockIdx.x) * S::B + threadIdx.x / S::T;  // block over all signals
  const bool valid = g < total;
  const int64_t sig = valid ? g / nblk : 0, j = valid ? g % nblk : 0;
  const int64_t B = 2 * int64_t(H) - (nb - 1);
  const int64_t pos0 = j * B - (nb - 1);
  WindowLoad<R> ld{a + sig * a_dist, pos0, na, valid};
  PaddedStore<C, H, EPT> st{sh};
  pow2_fft<C, H, EPT, -1>(sh, t, tw, ld, st);
  xsync<S::T>();
  // Z (half-length spectrum) -> X (real spectrum) -> X * Hs -> packed Z'
  const C z0 = sh[0];
  const C x0 = cmul(C{z0.x + z0.y, R(0)}, __ldg(hs));
  const C xh = cmul(C{z0.x - z0.y, R(0)}, __ldg(hs + H));
  C zp[EPT];
#pragma unroll
  for (int i = 0; i < EPT; ++i) {
    const int k = t + i * S::T;
    const C zk = sh[S::pad(k)], zhk = sh[S::pad(k == 0 ? 0 : H - k)];
    const C xk = k == 0 ? x0 : cmul(r2c_bin(z0, zk, zhk, __ldg(wt + k), k, H), __ldg(hs + k));
    const C xhk = k == 0 ? xh : cmul(r2c_bin(z0, zhk, zk, __ldg(wt + H - k), H - k, H), __ldg(hs + H - k));
    zp[i] = c2r_packed(xk, xhk, x0, xh, __ldg(wt + k), k);
  }
  xsync<S::T>();
#pragma unroll
  for (int i = 0; i < EPT; ++i) sh[S::pad(t + i * S::T)] = zp[i];
  xsync<S::T>();
  SharedLoad<C, H, EPT> ld2{sh};
  WindowStore<R> st2{dst + sig * dst_dist, j * B - (nb - 1), nout, nb - 1, R(1.0 / double(H)), valid};
  pow2_fft<C, H, EPT, +1>(sh, t, tw, ld2, st2);
}

template <typename C, int H, int EPT>
cudaError_t launch_conv_os(const void* a, void* dst, int64_t na, int64_t a_dist, int64_t dst_dist, int64_t nout,
                           int64_t nblk, int64_t count, int nb, const void* tw, const void* wt, const void* hs,
                           cudaStream_t st) {
  using S = Pow2Shape<H, EPT, sizeof(C)>;
  static const cudaError_t attr =
      S::SMEM > 48 * 1024
          ? cudaFuncSetAttribute(&k_conv_os<C, H, EPT>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM)
          : cudaSuccess;
  if (attr != cudaSuccess) return attr;
  using R = typename RealOf<C>::type;
  const int64_t total = count * nblk;
  k_conv_os<C, H, EPT><<<unsigned((total + S::B - 1) / S::B), S::TPB, S::SMEM, st>>>(
      static_cast<const R*>(a), static_cast<R*>(dst), na, a_dist, dst_dist, nout, nblk, total, nb,
      static_cast<const C*>(tw), static_cast<const C*>(wt), static_cast<const C*>(hs));
  return cudaGetLastError();
}

// Which calls run overlap-save, and the window of the float64 kernel: the
// smallest power of two with at most an eighth of each window wrapped (L >= 8
// (nb - 1)), else at most a quarter, at least 4096, at most 2^15 (float64:
// 2^14, what one CTA transforms as L / 2 complex points); 0 = one transform of
// the whole signal (short signals, long kernels).  In float32 it bounds how far
// two blocks that share a transform may reach (os_points).
template <typename R>
int64_t os_length(int64_t na, int64_t nb) {
  const int64_t lmax = sizeof(R) == 4 ? 32768 : 16384;
  for (const int64_t wrap : {8, 4}) {
    int64_t L = 4096;
    while (L < wrap * (nb - 1)) L <<= 1;
    if (L <= lmax && na + nb - 1 > 2 * L) return L;
  }
  return 0;
}

cudaError_t dispatch_conv_os(int64_t L, const double* a, double* dst, int64_t na, int64_t a_dist, int64_t dst_dist,
                             int64_t nout, int64_t nblk, int64_t count, int nb, const void* tw, const void* wt,
                             const void* hs, cudaStream_t st) {
  using C = double2;
  switch (L) {
    case 4096: return launch_conv_os<C, 2048, 16>(a, dst, na, a_dist, dst_dist, nout, nblk, count, nb, tw, wt, hs, st);
    case 8192: return launch_conv_os<C, 4096, 16>(a, dst, na, a_dist, dst_dist, nout, nblk, count, nb, tw, wt, hs, st);
    case 16384: return launch_conv_os<C, 8192, 16>(a, dst, na, a_dist, dst_dist, nout, nblk, count, nb, tw, wt, hs, st);
  }
  return cudaErrorInvalidValue;
}

// ---- float32 overlap-save: two blocks per transform -------------------------
//
// Blocks j and j + 1 of one signal (windows of N samples, B = N - (nb - 1) new
// outputs each) are the real and the imaginary part of one complex transform
// of N points.  The kernel is real, so its spectrum multiplies both parts
// alike, and the inverse gives both blocks' outputs: no real-spectrum
// recombination exists, and the bins never need their natural order -- the
// inverse runs the forward stages backwards from the registers they end in.
// Against the half-length form it replaced (recombination of bins k and H - k
// through shared memory, five table loads per bin) this costs four exchanges
// through shared memory instead of seven and two table loads per bin pair.
// The two blocks are neighbours in one signal: non-finite values and rounding
// errors reach both blocks and no further, and no value crosses between signals.
//
// Bound: the FMA pipe and the phases of one or a few CTAs per SM.  64 signals
// of 2^20 with 4097 taps: 0.440 ms before (2^15-sample half-length blocks),
// 0.290 ms now (N = 16384; FMA pipe busy 43 %), rel-L2 error 7.6e-7 -> 3.1e-7;
// 32 x 2^20 with 513 taps 0.165 -> 0.098 ms, with 33 taps 0.152 -> 0.080 (N =
// 2048), with 1025 taps 0.169 -> 0.107 (N = 4096).
using ConvRow16k = PairRow<16384, 32, 16, 16>;
using ConvRow8k = PairRow<8192, 16, 16, 16>;
using ConvRow4k = PairRow<4096, 16, 16, 8>;
using ConvRow2k = PairRow<2048, 16, 8, 8>;

// e in [lo, hi) of a window is a sample of the signal, else zero
struct PairWindowLoad {
  const float *a, *b;  // window sample 0 of the two blocks
  unsigned lo_a, n_a, lo_b, n_b;
  __device__ __forceinline__ float2 operator()(int e) const {
    return float2{unsigned(e) - lo_a < n_a ? __ldg(a + e) : 0.f, unsigned(e) - lo_b < n_b ? __ldg(b + e) : 0.f};
  }
};

struct PairWindowStore {
  float *a, *b;  // output of window sample 0 of the two blocks
  unsigned skip, n_a, n_b;  // the first nb - 1 window samples are wrapped: not outputs
  __device__ __forceinline__ void operator()(int e, float2 v) const {
    const unsigned o = unsigned(e) - skip;
    if (o < n_a) __stcs(a + e, v.x);
    if (o < n_b) __stcs(b + e, v.y);
  }
};

// Spectrum of the kernel, scaled by 1/N, in the register order of
// K::forward: entry i T + t is pair i of thread t.
template <typename K>
__global__ void __launch_bounds__(K::T) k_conv_spectrum(const float* b, int nb, const float2* __restrict__ tw,
                                                        float4* hs) {
  asm volatile("griddepcontrol.launch_dependents;");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float4* sh = reinterpret_cast<float4*>(smem_raw);
  Pair v[K::EP];
  K::template forward<-1>(v, sh, threadIdx.x, tw,
                          [&](int e) { return float2{e < nb ? __ldg(b + e) : 0.f, 0.f}; });
  const V2 s(1.0 / double(K::N));
#pragma unroll
  for (int i = 0; i < K::EP; ++i) K::put(hs, i * K::T + threadIdx.x, Pair{v[i].x * s, v[i].y * s});
}

__device__ __forceinline__ int64_t clamp_to(int64_t v, int64_t hi) { return v < 0 ? 0 : (v > hi ? hi : v); }

// One CTA per pair of blocks; npair pairs per signal.  ahead > 0: the CTA asks
// for the samples of CTA blockIdx + ahead to be brought into L2.
template <typename K, int MINB>
__global__ void __launch_bounds__(K::T, MINB)
k_conv_pair(const float* a, float* dst, int64_t na, int64_t a_dist, int64_t dst_dist, int64_t nout, int npair, int nb,
            const float2* __restrict__ tw, const float4* hs, int ahead) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float4* sh = reinterpret_cast<float4*>(smem_raw);
  const int t = threadIdx.x;
  const int skip = nb - 1, B = K::N - skip;
  if (ahead > 0 && unsigned(ahead) < gridDim.x - blockIdx.x) {
    const int g = blockIdx.x + ahead;
    const int64_t p0 = int64_t(g % npair) * 2 * B - skip;
    const int64_t lo = clamp_to(p0, na), hi = clamp_to(p0 + B + K::N, na);
    const float* x = a + (g / npair) * a_dist;
    const uintptr_t q0 = (reinterpret_cast<uintptr_t>(x + lo) + 15) & ~uintptr_t(15);
    const uintptr_t q1 = reinterpret_cast<uintptr_t>(x + hi) & ~uintptr_t(15);
    if (q1 > q0) prefetch_range(reinterpret_cast<const void*>(q0), int64_t(q1 - q0), t, K::T);
  }
  const int sig = blockIdx.x / npair;
  const int64_t pa = int64_t(blockIdx.x % npair) * 2 * B - skip, pb = pa + B;  // window sample 0
  const float* x = a + sig * a_dist;
  float* y = dst + sig * dst_dist;
  Pair v[K::EP];
  {
    const int64_t la = clamp_to(-pa, K::N), lb = clamp_to(-pb, K::N);
    const PairWindowLoad ld{x + pa, x + pb, unsigned(la), unsigned(clamp_to(na - pa - la, K::N - la)), unsigned(lb),
                            unsigned(clamp_to(na - pb - lb, K::N - lb))};
    K::template forward<-1>(v, sh, t, tw, ld);
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the kernel's spectrum
#pragma unroll
  for (int i = 0; i < K::EP; ++i) v[i] = pmul(v[i], K::get(hs, i * K::T + t));
  const PairWindowStore st{y + pa, y + pb, unsigned(skip), unsigned(clamp_to(nout - pa - skip, B)),
                           unsigned(clamp_to(nout - pb - skip, B))};
  K::template backward<+1>(v, sh, t, tw, st);
}

template <typename K, int MINB, bool PREFETCH>
cudaError_t launch_conv_pair(const float* a, float* dst, int64_t na, int64_t a_dist, int64_t dst_dist, int64_t nout,
                             int64_t count, const float* b, int nb, const float2* tw, float4* hs, cudaStream_t st) {
  cudaError_t e = raise_smem<&k_conv_spectrum<K>>(K::SMEM);
  if (e == cudaSuccess) e = raise_smem<&k_conv_pair<K, MINB>>(K::SMEM);
  if (e != cudaSuccess) return e;
  static const int64_t resident = resident_ctas(&k_conv_pair<K, MINB>, K::T, K::SMEM);
  const int64_t B = K::N - (nb - 1), npair = ((nout + B - 1) / B + 1) / 2;
  if (npair > 0x7fffffffLL / count) return cudaErrorInvalidConfiguration;
  k_conv_spectrum<K><<<1, K::T, K::SMEM, st>>>(b, nb, tw, hs);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  // programmatic launch: the forward transforms of the first wave overlap the
  // one-CTA transform of the kernel
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(count * npair));
  cfg.blockDim = dim3(K::T);
  cfg.dynamicSmemBytes = K::SMEM;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, &k_conv_pair<K, MINB>, a, dst, na, a_dist, dst_dist, nout, int(npair), nb, tw,
                            static_cast<const float4*>(hs), PREFETCH && count * npair > resident ? int(resident) : 0);
}

// Transform length of the float32 blocks.  A non-finite or loud sample reaches
// every output of the two blocks that share its transform (its rounding error,
// where it is finite).  Two blocks of N points span 2 N - (nb - 1) samples, so
// the lengths with 2 N <= Lb keep that within fewer than Lb samples, the window
// of one block of os_length.  Among them the one whose waves of CTAs take the
// least time (so a signal's last bits depend on how many share the call): `us`
// is one full wave (148 SMs x resident CTAs), measured on 32 and 64 signals of
// 2^20 (33 taps: 2048 points 0.080 ms, 4096 0.085; 513 taps: 4096 points 0.171,
// 8192 0.205, 16384 0.261 ms; 4097 taps: 8192 points 0.349, 16384 0.306 ms); a
// length serves kernels that wrap at most half of its window.  Prefetching the
// next CTA's samples gained 8 % at 16384 points, 3 % at 8192 and lost 4 % at
// 4096.
int os_points(int64_t Lb, int64_t nout, int64_t count, int64_t nb) {
  static const struct {
    int n, resident;
    double us;
  } kRows[] = {{2048, 8, 10.0}, {4096, 4, 10.7}, {8192, 2, 13.7}, {16384, 1, 16.4}};
  int best = 0;
  double cost = 0;
  for (const auto& r : kRows) {
    if (2 * r.n > Lb || 2 * (nb - 1) > r.n) continue;
    const int64_t B = r.n - (nb - 1), pairs = count * (((nout + B - 1) / B + 1) / 2), wave = 148 * r.resident;
    const double c = double((pairs + wave - 1) / wave) * r.us;
    if (best == 0 || c < cost) {
      cost = c;
      best = r.n;
    }
  }
  return best;
}

}  // namespace

// Complex: dst[0, L) = IFFT_L(FFT_L(a) * FFT_L(b)), L = na + nb - 1.
template <typename C>
static gfft_status convolve_dev(int prec, C* dst, const C* a, int64_t na, const C* b, int64_t nb, bool correlate,
                                cudaStream_t st) {
  const int64_t L = na + nb - 1;
  gfft_plan* p = nullptr;
  gfft_status s = cached_plan(prec, L, &p);
  if (s != GFFT_OK) return s;
  C* work = nullptr;
  GFFT_CUDA(ws_alloc(reinterpret_cast<void**>(&work), size_t(2 * L) * sizeof(C), st));
  k_pad<C><<<grid1(L), 256, 0, st>>>(work, L, a, na, 0, 1, false);
  if (correlate)
    k_pad_conj<C><<<grid1(L), 256, 0, st>>>(work + L, L, b, nb);
  else
    k_pad<C><<<grid1(L), 256, 0, st>>>(work + L, L, b, nb, 0, 1, false);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) s = core_exec(&p->core, -1, work, work, 2, L, L, st);
  if (e == cudaSuccess && s == GFFT_OK) {
    k_cmul_rows<C><<<grid1(L), 256, 0, st>>>(work, work + L, L, 1, 0);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess && s == GFFT_OK) s = core_exec(&p->core, +1, dst, work, 1, L, L, st);
  cudaFreeAsync(work, st);
  if (e != cudaSuccess) return cuda_status(e, "convolve");
  return s;
}

// Real: `count` signals (a_len reals, a_dist apart) convolved with one kernel
// b; outputs of a_len + b_len - 1 reals, dst_dist apart.  F = NextPow2.
template <typename R>
static gfft_status convolve_real_dev(int prec, R* dst, int64_t dst_dist, const R* a, int64_t na, int64_t a_dist,
                                     int64_t count, const R* b, int64_t nb, cudaStream_t st) {
  using C = Cx<R>;
  const int64_t L = na + nb - 1;
  // long signals: overlap-save blocks (same linear convolution, transforms of
  // 2^11..2^14 complex points, float64 2^12..2^14 reals, instead of one of
  // NextPow2(na + nb - 1))
  const int64_t Lb = os_length<R>(na, nb);
  if constexpr (sizeof(R) == 4) {
    if (Lb) {
      const int N = os_points(Lb, L, count, nb);
      gfft_plan* tp = nullptr;  // its W_N table
      gfft_status s = cached_plan(prec, N, &tp);
      if (s != GFFT_OK) return s;
      if (tp->core.algo == Algo::Pow2Smem) {
        float4* hs = nullptr;
        GFFT_CUDA(ws_alloc(reinterpret_cast<void**>(&hs), size_t(N) * sizeof(float2), st));
        const float2* tw = static_cast<const float2*>(tp->core.tw);
        const int64_t dd = count == 1 ? L : dst_dist;
        cudaError_t e;
        if (N == 2048)
          e = launch_conv_pair<ConvRow2k, 8, false>(a, dst, na, a_dist, dd, L, count, b, int(nb), tw, hs, st);
        else if (N == 4096)
          e = launch_conv_pair<ConvRow4k, 4, false>(a, dst, na, a_dist, dd, L, count, b, int(nb), tw, hs, st);
        else if (N == 8192)
          e = launch_conv_pair<ConvRow8k, 2, true>(a, dst, na, a_dist, dd, L, count, b, int(nb), tw, hs, st);
        else
          e = launch_conv_pair<ConvRow16k, 1, true>(a, dst, na, a_dist, dd, L, count, b, int(nb), tw, hs, st);
        cudaFreeAsync(hs, st);
        if (e != cudaSuccess) return cuda_status(e, "k_conv_pair");
        return GFFT_OK;
      }
    }
  } else if (Lb) {
    gfft_plan_real* bp = nullptr;
    gfft_status s = cached_real_plan(prec, Lb, &bp);
    if (s != GFFT_OK) return s;
    if (bp->child.algo == Algo::Pow2Smem) {
      const int64_t hb = Lb / 2 + 1;
      R* kpad = nullptr;
      GFFT_CUDA(ws_alloc(reinterpret_cast<void**>(&kpad), size_t(Lb) * sizeof(R) + size_t(hb) * sizeof(C), st));
      C* hs = reinterpret_cast<C*>(kpad + Lb);
      k_pad<R><<<grid1(Lb), 256, 0, st>>>(kpad, Lb, b, nb, 0, 1, false);
      cudaError_t e = cudaGetLastError();
      if (e == cudaSuccess) s = real_forward(bp, 0, hs, kpad, 1, Lb, hb, st);
      if (e == cudaSuccess && s == GFFT_OK) {
        const int64_t B = Lb - (nb - 1), nblk = (L + B - 1) / B;
        e = dispatch_conv_os(Lb, a, dst, na, a_dist, count == 1 ? L : dst_dist, L, nblk, count, int(nb), bp->child.tw,
                             bp->wt, hs, st);
      }
      cudaFreeAsync(kpad, st);
      if (e != cudaSuccess) return cuda_status(e, "k_conv_os");
      return s;
    }
  }
  int64_t F = 2;
  while (F < L) F <<= 1;  // convolve_real.go:23-28
  const int64_t h1 = F / 2 + 1;
  gfft_plan_real* p = nullptr;
  gfft_status s = cached_real_plan(prec, F, &p);
  if (s != GFFT_OK) return s;
  // [count + 1 padded rows of F reals | count + 1 spectra of h1 bins]
  R* pad = nullptr;
  const size_t pad_bytes = size_t(count + 1) * size_t(F) * sizeof(R);
  GFFT_CUDA(ws_alloc(reinterpret_cast<void**>(&pad), pad_bytes + size_t(count + 1) * size_t(h1) * sizeof(C), st));
  C* spec = reinterpret_cast<C*>(reinterpret_cast<char*>(pad) + pad_bytes);
  k_pad<R><<<grid1(count * F), 256, 0, st>>>(pad, F, a, na, a_dist, count, false);
  k_pad<R><<<grid1(F), 256, 0, st>>>(pad + count * F, F, b, nb, 0, 1, false);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) s = real_forward(p, 0, spec, pad, count + 1, F, h1, st);
  if (e == cudaSuccess && s == GFFT_OK) {
    k_cmul_rows<C><<<grid1(count * h1), 256, 0, st>>>(spec, spec + count * h1, h1, count, 0);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess && s == GFFT_OK) s = real_inverse(p, pad, spec, count, F, h1, st);
  if (e == cudaSuccess && s == GFFT_OK) {
    k_take_rows<R><<<grid1(count * L), 256, 0, st>>>(dst, dst_dist, pad, F, L, count);
    e = cudaGetLastError();
  }
  cudaFreeAsync(pad, st);
  if (e != cudaSuccess) return cuda_status(e, "convolve_real");
  return s;
}

// convolve.go:10-21 / convolve_real.go:10-22 argument checks.
static gfft_status conv_args(const void* dst, int64_t dst_len, const void* a, int64_t na, const void* b, int64_t nb) {
  if (!dst || !a || !b) return GFFT_ERR_NIL_SLICE;
  if (na <= 0 || nb <= 0) return GFFT_ERR_INVALID_LENGTH;
  if (dst_len != na + nb - 1) return GFFT_ERR_LENGTH_MISMATCH;
  return GFFT_OK;
}

static gfft_status conv_any(int prec, bool real, bool corr, void* dst, int64_t dst_len, const void* a, int64_t na,
                            const void* b, int64_t nb, cudaStream_t st) {
  gfft_status s = conv_args(dst, dst_len, a, na, b, nb);
  if (s != GFFT_OK) return s;
  if (prec != GFFT_COMPLEX64 && prec != GFFT_COMPLEX128) return GFFT_ERR_INVALID_ARGUMENT;
  if (real) {
    if (prec == kC64)
      return convolve_real_dev<float>(prec, static_cast<float*>(dst), 0, static_cast<const float*>(a), na, 0, 1,
                                      static_cast<const float*>(b), nb, st);
    return convolve_real_dev<double>(prec, static_cast<double*>(dst), 0, static_cast<const double*>(a), na, 0, 1,
                                     static_cast<const double*>(b), nb, st);
  }
  if (prec == kC64)
    return convolve_dev<float2>(prec, static_cast<float2*>(dst), static_cast<const float2*>(a), na,
                                static_cast<const float2*>(b), nb, corr, st);
  return convolve_dev<double2>(prec, static_cast<double2*>(dst), static_cast<const double2*>(a), na,
                               static_cast<const double2*>(b), nb, corr, st);
}

static gfft_status conv_host(int prec, bool real, bool corr, void* dst, int64_t dst_len, const void* a, int64_t na,
                             const void* b, int64_t nb) {
  gfft_status s = conv_args(dst, dst_len, a, na, b, nb);
  if (s != GFFT_OK) return s;
  if (prec != GFFT_COMPLEX64 && prec != GFFT_COMPLEX128) return GFFT_ERR_INVALID_ARGUMENT;
  const size_t es = elem_bytes(prec) / (real ? 2 : 1);
  cudaStream_t st = nullptr;
  GFFT_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  char* buf = nullptr;
  cudaError_t e = cudaMallocAsync(reinterpret_cast<void**>(&buf), size_t(na + nb + dst_len) * es, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(buf, a, size_t(na) * es, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(buf + na * es, b, size_t(nb) * es, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) {
    s = conv_any(prec, real, corr, buf + (na + nb) * es, dst_len, buf, na, buf + na * es, nb, st);
    if (s == GFFT_OK) e = cudaMemcpyAsync(dst, buf + (na + nb) * es, size_t(dst_len) * es, cudaMemcpyDeviceToHost, st);
  }
  if (buf) cudaFreeAsync(buf, st);
  cudaError_t e2 = cudaStreamSynchronize(st);
  cudaStreamDestroy(st);
  if (e != cudaSuccess) return cuda_status(e, "convolve host path");
  if (e2 != cudaSuccess) return cuda_status(e2, "cudaStreamSynchronize");
  return s;
}

}  // namespace gfft

using namespace gfft;

extern "C" {

gfft_status gfft_convolve(int32_t precision, void* dst, int64_t dst_len, const void* a, int64_t a_len, const void* b,
                          int64_t b_len, void* stream) {
  clear_error();
  return conv_any(precision, false, false, dst, dst_len, a, a_len, b, b_len, static_cast<cudaStream_t>(stream));
}

gfft_status gfft_correlate(int32_t precision, void* dst, int64_t dst_len, const void* a, int64_t a_len, const void* b,
                           int64_t b_len, void* stream) {
  clear_error();
  return conv_any(precision, false, true, dst, dst_len, a, a_len, b, b_len, static_cast<cudaStream_t>(stream));
}

gfft_status gfft_convolve_real(int32_t precision, void* dst, int64_t dst_len, const void* a, int64_t a_len,
                               const void* b, int64_t b_len, void* stream) {
  clear_error();
  return conv_any(precision, true, false, dst, dst_len, a, a_len, b, b_len, static_cast<cudaStream_t>(stream));
}

gfft_status gfft_convolve_host(int32_t precision, void* dst, int64_t dst_len, const void* a, int64_t a_len,
                               const void* b, int64_t b_len) {
  clear_error();
  return conv_host(precision, false, false, dst, dst_len, a, a_len, b, b_len);
}

gfft_status gfft_correlate_host(int32_t precision, void* dst, int64_t dst_len, const void* a, int64_t a_len,
                                const void* b, int64_t b_len) {
  clear_error();
  return conv_host(precision, false, true, dst, dst_len, a, a_len, b, b_len);
}

gfft_status gfft_convolve_real_host(int32_t precision, void* dst, int64_t dst_len, const void* a, int64_t a_len,
                                    const void* b, int64_t b_len) {
  clear_error();
  return conv_host(precision, true, false, dst, dst_len, a, a_len, b, b_len);
}

gfft_status gfft_convolve_real_batch(int32_t precision, void* dst, int64_t dst_dist, const void* a, int64_t a_len,
                                     int64_t a_dist, int64_t count, const void* b, int64_t b_len, void* stream) {
  clear_error();
  if (!dst || !a || !b) return GFFT_ERR_NIL_SLICE;
  if (a_len <= 0 || b_len <= 0 || count < 1) return GFFT_ERR_INVALID_LENGTH;
  if (a_dist < a_len || dst_dist < a_len + b_len - 1) return GFFT_ERR_INVALID_STRIDE;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (precision == GFFT_COMPLEX64)
    return convolve_real_dev<float>(precision, static_cast<float*>(dst), dst_dist, static_cast<const float*>(a),
                                    a_len, a_dist, count, static_cast<const float*>(b), b_len, st);
  if (precision == GFFT_COMPLEX128)
    return convolve_real_dev<double>(precision, static_cast<double*>(dst), dst_dist, static_cast<const double*>(a),
                                     a_len, a_dist, count, static_cast<const double*>(b), b_len, st);
  return GFFT_ERR_INVALID_ARGUMENT;
}

}  // extern "C"
