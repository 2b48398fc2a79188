// Batched complex128 discrete Fourier transforms for the spectra of
// propagated correlation functions (lime/fft.py:9-56: g(w) = fftshift(fft(f))
// dx exp(-i w x0)).  Power-of-two lengths up to 8192 run as one CTA per
// transform, decimation in time with three radix-2 stages a pass in
// registers and one exchange through shared memory between passes; the first
// pass reads global memory, the last one writes it.  Other lengths up to 4096
// go through Bluestein's chirp-z identity
//     X_k = c_k sum_j (x_j c_j) conj(c_{k-j}),   c_j = exp(-i pi j^2 / n)
// as a circular convolution of length m = 2^ceil(log2(2n - 1)): the chirp, the
// forward transforms (the filter's among them) and the inverse transforms are
// a launch each.  The output can be written fftshift-ed and multiplied by a
// per-position factor (dx exp(-i w_k x0) for lime's fft).
//
// Bound: the FP64 pipe (1.68 lanes per clock and SM; everything else is
// nearly free beside it), so the butterflies are counted in FP64
// instructions: u + w v and u - w v are 8 fma, or 6 where the second is
// 2 u - (u + w v); the first pass's factors 1 and -i are 4 additions, and the
// factors come from a table that the compiler fills (a sincospi in each
// butterfly took 40 of 48).  The 6-fma form in all stages leaves an rms error
// 4 to 5 % above that of u +- t with a rounded t = w v, the 8-fma form one 3 to
// 4 % below; the first stage of a pass takes the former, the two others the
// latter, and the error is at or below the one of u +- t at every length.  256
// transforms of 4096: 719 -> 100 us, 40 + 4 FP64 instructions a point being
// 92 us (33.5 + 4 and 91 us with 6 fma throughout); 100 of length 999: 554 -> 62
// us, 3 launches for 6.

#include "common.cuh"

namespace lime {
namespace fft {

constexpr int kThreads = 512;
constexpr int kMaxPow2 = 8192;
constexpr int kRoots = kMaxPow2 / 2;

// exp(-2 pi i j / 8192), j = 0 .. 4095, from the Taylor series of the first
// octant in 62-bit fixed point (error under 2^-59), rounded once; read as double2
struct alignas(sizeof(double2)) Roots {
  double v[2 * kRoots];
};
static_assert(alignof(Roots) >= alignof(double2), "root() loads 16 bytes at a time");
constexpr long long fixmul(long long a, long long b) { return (long long)(((__int128)a * b) >> 62); }
constexpr Roots make_roots() {
  Roots r{};
  const unsigned long long pi = 0xC90FDAA22168C235ull;   // pi 2^62
  for (int j = 0; j <= kRoots / 4; ++j) {
    const long long x = (long long)(((unsigned __int128)pi * (unsigned)j) >> 12);   // 2 pi j / 8192
    const long long x2 = fixmul(x, x);
    long long c = 1ll << 62, s = x, tc = c, ts = x;
    for (int k = 1; k <= 11; ++k) {
      tc = -fixmul(tc, x2) / ((2 * k - 1) * (2 * k));
      ts = -fixmul(ts, x2) / ((2 * k) * (2 * k + 1));
      c += tc;
      s += ts;
    }
    const double one = 4611686018427387904.0;   // 2^62
    const double cd = (double)c / one, sd = (double)s / one;
    // octants: (c, -s) at j; (s, -c) at 2048 - j; (-s, -c) at 2048 + j; (-c, -s) at 4096 - j
    const int h = kRoots / 2;
    r.v[2 * j] = cd;
    r.v[2 * j + 1] = -sd;
    r.v[2 * (h - j)] = sd;
    r.v[2 * (h - j) + 1] = -cd;
    r.v[2 * (h + j)] = -sd;
    r.v[2 * (h + j) + 1] = -cd;
    if (j > 0) {
      r.v[2 * (kRoots - j)] = -cd;
      r.v[2 * (kRoots - j) + 1] = -sd;
    }
  }
  r.v[1] = 0.0;
  r.v[kRoots] = 0.0;
  return r;
}
__device__ const Roots g_roots = make_roots();

__device__ __forceinline__ double2 root(int j) { return reinterpret_cast<const double2*>(g_roots.v)[j]; }
__device__ __forceinline__ unsigned bitrev(unsigned v, int bits) { return bits == 0 ? 0u : __brev(v) >> (32 - bits); }
// place of element i in shared memory: the low three bits take in the higher
// ones, so that the bit-reversed stores of the first pass (one low part for
// all lanes) spread over the banks
__device__ __forceinline__ int sw(int i) { return i ^ (((i >> 3) ^ (i >> 6) ^ (i >> 9)) & 7); }

// (u, v) <- (u + w v, u - w v)
__device__ __forceinline__ void bfly(double2& u, double2& v, double2 w) {
  const double2 r = make_double2(fma(-w.y, v.y, fma(w.x, v.x, u.x)), fma(w.y, v.x, fma(w.x, v.y, u.y)));
  v = make_double2(fma(w.y, v.y, fma(-w.x, v.x, u.x)), fma(-w.y, v.x, fma(-w.x, v.y, u.y)));
  u = r;
}
// the same with 6 instructions for 8; the second result takes over the first one's rounding error
__device__ __forceinline__ void bfly_6(double2& u, double2& v, double2 w) {
  const double2 r = make_double2(fma(-w.y, v.y, fma(w.x, v.x, u.x)), fma(w.y, v.x, fma(w.x, v.y, u.y)));
  v = make_double2(fma(2.0, u.x, -r.x), fma(2.0, u.y, -r.y));
  u = r;
}
// with -i w
__device__ __forceinline__ void bfly_mi(double2& u, double2& v, double2 w) { bfly(u, v, make_double2(w.y, -w.x)); }
__device__ __forceinline__ void bfly_1(double2& u, double2& v) {
  const double2 r = cadd(u, v);
  v = csub(u, v);
  u = r;
}
__device__ __forceinline__ void bfly_mi1(double2& u, double2& v) {
  const double2 r = make_double2(u.x + v.y, u.y - v.x);
  v = make_double2(u.x - v.y, u.y + v.x);
  u = r;
}

// the first K stages of 2^K elements (factors exp(-i pi m / 2^stage))
template <int K>
__device__ __forceinline__ void first_stages(double2 (&v)[8]) {
#pragma unroll
  for (int m = 0; m < (1 << K); m += 2) bfly_1(v[m], v[m + 1]);
  if (K > 1)
#pragma unroll
    for (int m = 0; m < (1 << K); m += 4) {
      bfly_1(v[m], v[m + 2]);
      bfly_mi1(v[m + 1], v[m + 3]);
    }
  if (K > 2) {
    const double2 w = root(kRoots / 4);
    bfly_1(v[0], v[4]);
    bfly(v[1], v[5], w);
    bfly_mi1(v[2], v[6]);
    bfly_mi(v[3], v[7], w);
  }
}

template <int K, class Load, class Store>
__device__ __forceinline__ void first_pass(double2* s, int L, const Load& load, const Store& store) {
  const int groups = 1 << (L - K);
  for (int r = threadIdx.x; r < groups; r += blockDim.x) {
    double2 v[8];
#pragma unroll
    for (int m = 0; m < (1 << K); ++m) v[m] = load((int)(__brev((unsigned)m) >> (32 - K)) * groups + r);
    first_stages<K>(v);
    const int q = (int)bitrev((unsigned)r, L - K);
#pragma unroll
    for (int m = 0; m < (1 << K); ++m) {
      if (L == K) store(m, v[m]);
      else s[sw((q << K) + m)] = v[m];
    }
  }
}

// y_k = sum_j load(j) exp(-2 pi i j k / 2^L), store(k, y_k), by one CTA; s: 2^L elements
template <class Load, class Store>
__device__ void transform(double2* s, int L, const Load& load, const Store& store) {
  const int n = 1 << L;
  if (L == 0) {
    if (threadIdx.x == 0) store(0, load(0));
    return;
  }
  const int K = L % 3 == 0 ? 3 : L % 3;
  if (K == 3) first_pass<3>(s, L, load, store);
  else if (K == 2) first_pass<2>(s, L, load, store);
  else first_pass<1>(s, L, load, store);
  for (int h = 1 << K, lh = K; h < n; h <<= 3, lh += 3) {
    __syncthreads();
    const bool last = h << 3 == n;
    for (int q = threadIdx.x; q < n >> 3; q += blockDim.x) {
      const int pos = q & (h - 1), base = ((q - pos) << 3) + pos;
      // factors of the stages of half length h, 2 h, 4 h at pos
      const int j3 = pos << (10 - lh);
      const double2 w1 = root(j3 << 2), w2 = root(j3 << 1), w3 = root(j3), w3a = root(j3 + kRoots / 4);
      double2 v[8];
#pragma unroll
      for (int m = 0; m < 8; ++m) v[m] = s[sw(base + (m << lh))];
#pragma unroll
      for (int m = 0; m < 8; m += 2) bfly_6(v[m], v[m + 1], w1);
#pragma unroll
      for (int m = 0; m < 8; m += 4) {
        bfly(v[m], v[m + 2], w2);
        bfly_mi(v[m + 1], v[m + 3], w2);
      }
      bfly(v[0], v[4], w3);
      bfly(v[1], v[5], w3a);
      bfly_mi(v[2], v[6], w3);
      bfly_mi(v[3], v[7], w3a);
#pragma unroll
      for (int m = 0; m < 8; ++m) {
        if (last) store(base + (m << lh), v[m]);
        else s[sw(base + (m << lh))] = v[m];
      }
    }
  }
}

struct Pass {
  int n, log2n;              // transform length (Bluestein: the convolution's m)
  int len, inverse;          // data length, sign of the transform
  const double2* x; int64_t x_s, x_bs;
  double2* y; int64_t y_s, y_bs;
  int shift;                 // write output k at (k + len/2) % len
  const double2* post;       // per output position factor (after the shift), or null
  double2* conv;             // Bluestein: [batch][m]
  double2* chirp;            // Bluestein: c_j, j < len, then the filter's spectrum k = 0 .. m/2
};

// an inverse transform is the conjugate of the transform of the conjugate
__device__ __forceinline__ double2 conj_if(double2 v, int on) { return on ? cconj(v) : v; }

__device__ __forceinline__ void put(const Pass& p, int64_t b, int k, double2 v) {
  int ks = k;
  if (p.shift) {
    ks = k + p.len / 2;
    if (ks >= p.len) ks -= p.len;
  }
  if (p.post) v = cmul(v, p.post[ks]);
  p.y[b * p.y_bs + (int64_t)ks * p.y_s] = v;
}

__global__ void __launch_bounds__(kThreads) pow2_kernel(Pass p) {
  extern __shared__ double2 s[];
  const int64_t b = blockIdx.x;
  const double2* x = p.x + b * p.x_bs;
  transform(s, p.log2n, [&](int j) { return conj_if(x[(int64_t)j * p.x_s], p.inverse); },
            [&](int k, double2 v) { put(p, b, k, conj_if(v, p.inverse)); });
}

// c_j = exp(-+ i pi j^2 / len), the argument reduced exactly (j^2 mod 2 len)
__global__ void chirp_kernel(Pass p) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= p.len) return;
  const int64_t r = ((int64_t)j * j) % (2 * (int64_t)p.len);
  double sn, cs;
  sincospi((double)r / (double)p.len, &sn, &cs);
  p.chirp[j] = make_double2(cs, p.inverse ? sn : -sn);
}

// block b < batch: the spectrum of x_j c_j; the last block: half the
// spectrum of the filter conj(c_j), wrapped circularly (even, so its spectrum
// is too, and with the chirp it fits one row of the workspace)
__global__ void __launch_bounds__(kThreads) chirp_forward_kernel(Pass p) {
  extern __shared__ double2 s[];
  const int64_t b = blockIdx.x;
  const int len = p.len, m = p.n;
  if (b + 1 == gridDim.x) {
    double2* spec = p.chirp + len;
    transform(s, p.log2n,
              [&](int j) {
                const int k = j < len ? j : j > m - len ? m - j : -1;
                return k < 0 ? cz() : cconj(p.chirp[k]);
              },
              [&](int k, double2 v) { if (2 * k <= m) spec[k] = v; });
    return;
  }
  const double2* x = p.x + b * p.x_bs;
  double2* c = p.conv + b * m;
  transform(s, p.log2n, [&](int j) { return j < len ? cmul(x[(int64_t)j * p.x_s], p.chirp[j]) : cz(); },
            [&](int k, double2 v) { c[k] = v; });
}

// X_k = c_k conv_k / m from the product of the spectra
__global__ void __launch_bounds__(kThreads) chirp_inverse_kernel(Pass p) {
  extern __shared__ double2 s[];
  const int64_t b = blockIdx.x;
  const int len = p.len, m = p.n;
  const double2* c = p.conv + b * m;
  const double2* spec = p.chirp + len;
  const double scale = 1.0 / (double)m;   // a power of two
  transform(s, p.log2n, [&](int k) { return cconj(cmul(c[k], spec[2 * k <= m ? k : m - k])); },
            [&](int k, double2 v) { if (k < len) put(p, b, k, cmul(cscale(cconj(v), scale), p.chirp[k])); });
}

int log2_exact(int n) {
  int l = 0;
  while ((1 << l) < n) ++l;
  return (1 << l) == n ? l : -1;
}

int bluestein_len(int n) {
  int m = 1;
  while (m < 2 * n - 1) m <<= 1;
  return m;
}

}  // namespace fft
}  // namespace lime

using namespace lime;

extern "C" size_t lime_fft_f64_workspace(int32_t n, int32_t batch) {
  if (n <= 0 || batch <= 0) return 0;
  if (fft::log2_exact(n) >= 0) return 0;
  const int m = fft::bluestein_len(n);
  return ((size_t)batch + 1) * m * sizeof(double2);
}

extern "C" int lime_fft_f64(const LimeFftDesc* d, void* stream) {
  if (!d || d->n <= 0 || d->batch <= 0 || !d->x || !d->y) return LIME_ERR_ARG;
  if ((d->inverse & ~1) || (d->shift & ~1)) return LIME_ERR_ARG;
  const int n = d->n;
  cudaStream_t st = (cudaStream_t)stream;
  const int l2 = fft::log2_exact(n);
  const int m = l2 >= 0 ? n : fft::bluestein_len(n);
  if (m > fft::kMaxPow2) return LIME_ERR_UNSUPPORTED;
  if (l2 < 0 && (!d->workspace || d->workspace_bytes < lime_fft_f64_workspace(n, d->batch)))
    return LIME_ERR_WORKSPACE;
  fft::Pass p{};
  p.n = m; p.log2n = fft::log2_exact(m); p.len = n; p.inverse = d->inverse;
  p.x = reinterpret_cast<const double2*>(d->x); p.x_s = d->x_s; p.x_bs = d->x_bs;
  p.y = reinterpret_cast<double2*>(d->y); p.y_s = d->y_s; p.y_bs = d->y_bs;
  p.shift = d->shift;
  p.post = reinterpret_cast<const double2*>(d->post);
  const size_t smem = (size_t)m * sizeof(double2);
  // (one value for every length: calls of other threads set the same attribute)
  constexpr int kMost = fft::kMaxPow2 * (int)sizeof(double2);
  // a thread takes 8 elements of a pass
  const int nt = m / 8 < 32 ? 32 : m / 8 < fft::kThreads ? m / 8 : fft::kThreads;
  if (l2 >= 0) {
    LIME_CUDA_TRY(cudaFuncSetAttribute(fft::pow2_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost));
    fft::pow2_kernel<<<d->batch, nt, smem, st>>>(p);
    LIME_CUDA_TRY(cudaGetLastError());
    count_launch();
    return LIME_OK;
  }
  p.conv = reinterpret_cast<double2*>(d->workspace);      // [batch][m]
  p.chirp = p.conv + (size_t)d->batch * m;                 // [m]: n + m/2 + 1 <= m, n is not a power of two
  LIME_CUDA_TRY(cudaFuncSetAttribute(fft::chirp_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost));
  LIME_CUDA_TRY(cudaFuncSetAttribute(fft::chirp_inverse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost));
  fft::chirp_kernel<<<(n + 63) / 64, 64, 0, st>>>(p);
  LIME_CUDA_TRY(cudaGetLastError());
  fft::chirp_forward_kernel<<<d->batch + 1, nt, smem, st>>>(p);
  LIME_CUDA_TRY(cudaGetLastError());
  fft::chirp_inverse_kernel<<<d->batch, nt, smem, st>>>(p);
  LIME_CUDA_TRY(cudaGetLastError());
  count_launch(3);
  return LIME_OK;
}
