// Strided batched complex128 GEMM for the Liouville-space Green's-function
// route and the eigenbasis transforms of the Redfield solver
// (lime/oqs.py:169-366: U(t) = U1 exp(w t) U1^-1, expect, the 2- and 4-point
// correlation functions, and the basis changes V^dag X V of
// lime/phys.py:706-718).  Every contraction there is
//     C[z][i][j] = sum_k op(A)[z][i][k] s[z][k] op(B)[z][k][j]
// with op = identity or complex conjugate, an optional per-(z, k) complex
// scale s (the exp(w_j t_z) of the spectral propagator), and arbitrary
// element strides for rows, columns and the batch index (0 broadcasts), so
// a (D, D, Nt) propagator contracts with a block of vectors without any
// transposition.  FP64 on the tiled GEMM of gemm_f64.cuh (64 x 64 tiles), or
// one thread an element for outputs that would leave most of a tile empty;
// both add the K terms of an element in the same order.

#include "gemm_f64.cuh"

namespace lime {
namespace zg {

struct Args {
  int M, N, K;
  int conj_a, conj_b;
  const double2* A; int64_t a_rs, a_cs, a_bs;
  const double2* B; int64_t b_rs, b_cs, b_bs;
  const double2* S; int64_t s_ks, s_bs;
  double2* C; int64_t c_rs, c_cs, c_bs;
  int z0;
};

__global__ void __launch_bounds__(rf::kThreads) zgemm_kernel(Args a) {
  const int64_t z = (int64_t)a.z0 + blockIdx.z;
  const double2* A = a.A + z * a.a_bs;
  const double2* B = a.B + z * a.b_bs;
  const double2* S = a.S ? a.S + z * a.s_bs : nullptr;
  double2* C = a.C + z * a.c_bs;
  auto la = [&](int i, int k) -> double2 {
    double2 v = A[(int64_t)i * a.a_rs + (int64_t)k * a.a_cs];
    if (a.conj_a) v.y = -v.y;
    if (S != nullptr) v = cmul(v, S[(int64_t)k * a.s_ks]);
    return v;
  };
  auto lb = [&](int k, int j) -> double2 {
    double2 v = B[(int64_t)k * a.b_rs + (int64_t)j * a.b_cs];
    if (a.conj_b) v.y = -v.y;
    return v;
  };
  auto epi = [&](int i, int j, double2 v) { C[(int64_t)i * a.c_rs + (int64_t)j * a.c_cs] = v; };
  rf::gemm_tile(a.M, a.N, a.K, blockIdx.y * rf::kTile, blockIdx.x * rf::kTile, la, lb, epi);
}

// One thread an element, its operands through L1.  The FP64 pipe is the
// bound in both kernels (4 K DFMA an element) and a tile computes its
// padding: a 20 x 20 basis change of 100 states, 131 us on tiles, takes 10 us.
__global__ void __launch_bounds__(128) zgemm_element_kernel(Args a, int64_t total) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int j = (int)(e % a.N);
    const int64_t zi = e / a.N;
    const int i = (int)(zi % a.M);
    const int64_t z = zi / a.M;
    const double2* A = a.A + z * a.a_bs + (int64_t)i * a.a_rs;
    const double2* B = a.B + z * a.b_bs + (int64_t)j * a.b_cs;
    const double2* S = a.S ? a.S + z * a.s_bs : nullptr;
    double2 acc = cz();
#pragma unroll 4
    for (int k = 0; k < a.K; ++k) {
      double2 x = A[(int64_t)k * a.a_cs], y = B[(int64_t)k * a.b_rs];
      if (a.conj_a) x.y = -x.y;
      if (S != nullptr) x = cmul(x, S[(int64_t)k * a.s_ks]);
      if (a.conj_b) y.y = -y.y;
      cfma(acc, x, y);
    }
    a.C[z * a.c_bs + (int64_t)i * a.c_rs + (int64_t)j * a.c_cs] = acc;
  }
}

// Addresses of a strided operand, [lo, hi] in elements.
struct Span {
  const double2 *lo, *hi;
};
static Span span(const double2* p, int64_t d0, int64_t s0, int64_t d1, int64_t s1, int64_t d2, int64_t s2) {
  Span r{p, p};
  const int64_t len[3] = {(d0 - 1) * s0, (d1 - 1) * s1, (d2 - 1) * s2};
  for (int64_t v : len) (v < 0 ? r.lo : r.hi) += v;
  return r;
}
static bool meets(const Span& a, const Span& b) { return a.lo <= b.hi && b.lo <= a.hi; }

}  // namespace zg
}  // namespace lime

using namespace lime;

extern "C" int lime_zgemm_strided_f64(const LimeZgemmDesc* d, void* stream) {
  if (!d || d->M <= 0 || d->N <= 0 || d->K <= 0 || d->batch <= 0) return LIME_ERR_ARG;
  if (!d->A || !d->B || !d->C) return LIME_ERR_ARG;
  if ((d->conj_a & ~1) || (d->conj_b & ~1)) return LIME_ERR_ARG;
  zg::Args a{};
  a.M = d->M; a.N = d->N; a.K = d->K;
  a.conj_a = d->conj_a; a.conj_b = d->conj_b;
  a.A = reinterpret_cast<const double2*>(d->A); a.a_rs = d->a_rs; a.a_cs = d->a_cs; a.a_bs = d->a_bs;
  a.B = reinterpret_cast<const double2*>(d->B); a.b_rs = d->b_rs; a.b_cs = d->b_cs; a.b_bs = d->b_bs;
  a.S = reinterpret_cast<const double2*>(d->scale); a.s_ks = d->s_ks; a.s_bs = d->s_bs;
  a.C = reinterpret_cast<double2*>(d->C); a.c_rs = d->c_rs; a.c_cs = d->c_cs; a.c_bs = d->c_bs;
  cudaStream_t st = (cudaStream_t)stream;
  const unsigned gx = (unsigned)((d->N + rf::kTile - 1) / rf::kTile);
  const unsigned gy = (unsigned)((d->M + rf::kTile - 1) / rf::kTile);
  if (gy > 65535u) return LIME_ERR_UNSUPPORTED;
  // elements: while the tiles hold more than twice the outputs, or leave
  // most SMs without one (fewer than 76 tiles, half of the 152 SMs: an SM's
  // share of elements is then the smaller).  Not where C lies over an operand:
  // a tile reads all of its operands before it writes (C = A B in the place of
  // A works up to 64 x 64), an element's thread would write while others read.
  const int64_t outputs = (int64_t)d->M * d->N * d->batch, tiles = (int64_t)gx * gy * d->batch;
  const zg::Span c = zg::span(a.C, a.M, a.c_rs, a.N, a.c_cs, d->batch, a.c_bs);
  const bool apart = !zg::meets(c, zg::span(a.A, a.M, a.a_rs, a.K, a.a_cs, d->batch, a.a_bs)) &&
                     !zg::meets(c, zg::span(a.B, a.K, a.b_rs, a.N, a.b_cs, d->batch, a.b_bs)) &&
                     !(a.S && zg::meets(c, zg::span(a.S, a.K, a.s_ks, d->batch, a.s_bs, 1, 0)));
  if (apart && (tiles * rf::kTile * rf::kTile > 2 * outputs || tiles < 76)) {
    const int64_t blocks = (outputs + 127) / 128;
    zg::zgemm_element_kernel<<<(unsigned)(blocks < 1 << 20 ? blocks : 1 << 20), 128, 0, st>>>(a, outputs);
    LIME_CUDA_TRY(cudaGetLastError());
    count_launch();
    return LIME_OK;
  }
  int64_t launches = 0;
  for (int z0 = 0; z0 < d->batch; z0 += 65535) {
    a.z0 = z0;
    const unsigned gz = (unsigned)((d->batch - z0) < 65535 ? (d->batch - z0) : 65535);
    zg::zgemm_kernel<<<dim3(gx, gy, gz), rf::kThreads, 0, st>>>(a);
    LIME_CUDA_TRY(cudaGetLastError());
    ++launches;
  }
  count_launch(launches);
  return LIME_OK;
}
