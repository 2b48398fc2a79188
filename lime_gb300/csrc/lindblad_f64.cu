// FP64 Lindblad adjoint with dense collapse operators (one CTA per density
// matrix: CTA-wide complex GEMMs, register-tiled, operands staged through
// shared memory; without them see lindblad_adjoint_rows_f64.cu) and the
// preparation of the generators.
//
// GB300 executes FP64 at a small fraction of its tensor rate, so this path is
// DFMA-bound; its job is to be exact.

#include "adjoint_f64.cuh"

namespace lime {
namespace f64 {

constexpr int kThreads = 256;
constexpr int kKC = 16;  // k-chunk of the shared-memory tiles

// C (+)= A * op(B), all n x n, row-major, global memory; whole CTA.
// op(B) = B (conjb = false) or B^dag (conjb = true).
template <int TM>
__device__ void cta_cgemm(const double2* __restrict__ A, const double2* __restrict__ B,
                          bool conjb, double2* __restrict__ C, bool accumulate, int n,
                          double2* smem) {
  constexpr int T = 16 * TM;
  double2* As = smem;                   // [T][kKC + 1]
  double2* Bs = smem + T * (kKC + 1);   // [kKC][T + 1]
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  for (int i0 = 0; i0 < n; i0 += T) {
    for (int j0 = 0; j0 < n; j0 += T) {
      double2 acc[TM][TM];
#pragma unroll
      for (int u = 0; u < TM; ++u)
#pragma unroll
        for (int v = 0; v < TM; ++v) acc[u][v] = cz();
      for (int k0 = 0; k0 < n; k0 += kKC) {
        for (int idx = threadIdx.x; idx < T * kKC; idx += kThreads) {
          const int r = idx / kKC, c = idx % kKC;
          const int gi = i0 + r, gk = k0 + c;
          As[r * (kKC + 1) + c] = (gi < n && gk < n) ? A[(int64_t)gi * n + gk] : cz();
        }
        if (!conjb) {
          for (int idx = threadIdx.x; idx < T * kKC; idx += kThreads) {
            const int r = idx / T, c = idx % T;
            const int gk = k0 + r, gj = j0 + c;
            Bs[r * (T + 1) + c] = (gk < n && gj < n) ? B[(int64_t)gk * n + gj] : cz();
          }
        } else {
          // op(B)[k][j] = conj(B[j][k]); read along k for coalescing
          for (int idx = threadIdx.x; idx < T * kKC; idx += kThreads) {
            const int c = idx / kKC, r = idx % kKC;
            const int gk = k0 + r, gj = j0 + c;
            Bs[r * (T + 1) + c] = (gk < n && gj < n) ? cconj(B[(int64_t)gj * n + gk]) : cz();
          }
        }
        __syncthreads();
#pragma unroll 4
        for (int kk = 0; kk < kKC; ++kk) {
          double2 a[TM], b[TM];
#pragma unroll
          for (int u = 0; u < TM; ++u) a[u] = As[(ty + 16 * u) * (kKC + 1) + kk];
#pragma unroll
          for (int v = 0; v < TM; ++v) b[v] = Bs[kk * (T + 1) + tx + 16 * v];
#pragma unroll
          for (int u = 0; u < TM; ++u)
#pragma unroll
            for (int v = 0; v < TM; ++v) cfma(acc[u][v], a[u], b[v]);
        }
        __syncthreads();
      }
#pragma unroll
      for (int u = 0; u < TM; ++u) {
#pragma unroll
        for (int v = 0; v < TM; ++v) {
          const int gi = i0 + ty + 16 * u, gj = j0 + tx + 16 * v;
          if (gi < n && gj < n) {
            double2* c = C + (int64_t)gi * n + gj;
            *c = accumulate ? cadd(*c, acc[u][v]) : acc[u][v];
          }
        }
      }
    }
  }
  __syncthreads();
}

// ---------------------------------------------------------------- adjoint
// One generator in the Hermitian form f = -i(G x - x G^dag) + M o x + sum_k L_k x L_k^dag.
struct Gen {
  const double2* g;
  const double2* m;   // may be null
  const double2* l;   // k dense operators, may be null
  int k;
};

// out = gen(x); X, Y, J are n x n scratch.  Whole CTA; ends synchronised.
template <int TM>
__device__ void apply_gen(const Gen& G, const double2* x, double2* out, double2* X, double2* Y, double2* J, int n,
                          double2* smem) {
  const int64_t nn = (int64_t)n * n;
  cta_cgemm<TM>(G.g, x, false, X, false, n, smem);
  for (int k = 0; k < G.k; ++k) {
    const double2* L = G.l + k * nn;
    cta_cgemm<TM>(L, x, false, Y, false, n, smem);
    cta_cgemm<TM>(Y, L, true, J, k > 0, n, smem);
  }
  for (int64_t e = threadIdx.x; e < nn; e += kThreads) {
    const int i = (int)(e / n), j = (int)(e % n);
    const double2 a = X[e], b = X[(int64_t)j * n + i];
    double2 f = make_double2(a.y + b.y, b.x - a.x);   // -i (X - X^dag)
    if (G.m) f = cadd(f, cmul(G.m[e], x[e]));
    if (G.k > 0) f = cadd(f, J[e]);
    out[e] = f;
  }
  __syncthreads();
}

// Parameter-gradient contributions of one stage: abar = adjoint of the stage
// derivative, y = stage state (both Hermitian).  Thread-strided over rows.
__device__ void grad_terms(const double2* abar, const double2* y, int n, double* gd, double* gb, double* gg) {
  for (int k = threadIdx.x; k < n; k += kThreads) {
    double sd = 0.0, sg = 0.0, sb = 0.0;
    for (int x = 0; x < n; ++x) {
      const double2 a = abar[(int64_t)k * n + x], v = y[(int64_t)k * n + x];
      sd += a.x * v.y - a.y * v.x;                 // Im(conj(a) y)
      if (x != k) sg -= a.x * v.x + a.y * v.y;      // -Re(conj(a) y), off-diagonal
      if (k + 1 < n) {
        const double2 a2 = abar[(int64_t)(k + 1) * n + x], v2 = y[(int64_t)(k + 1) * n + x];
        sb += (a.x * v2.y - a.y * v2.x) + (a2.x * v.y - a2.y * v.x);
      }
    }
    gd[k] += 2.0 * sd;
    gg[k] += sg;
    if (k + 1 < n) gb[k] += 2.0 * sb;
  }
}

template <int TM>
__global__ void __launch_bounds__(kThreads) lindblad_adjoint_f64_kernel(AdjArgs a) {
  extern __shared__ double2 smem[];
  const int b = blockIdx.x;
  const int n = a.n;
  const int64_t nn = (int64_t)n * n;
  const int p = b % a.param_batch;
  const Gen F{a.heff + p * a.heff_stride, a.m ? a.m + p * a.m_stride : nullptr,
              a.ld ? a.ld + p * a.ld_stride : nullptr, a.k_dense};
  const Gen A{a.heff_adj + p * a.heff_adj_stride, a.m_adj ? a.m_adj + p * a.m_adj_stride : nullptr,
              a.ld_adj ? a.ld_adj + p * a.ld_adj_stride : nullptr, a.k_dense};
  double2* ws = a.ws + (int64_t)b * adj_ws_mats(a.seg_steps, a.k_dense) * nn;
  double2* seg = ws;                              // rho_{step0 + s}, s < seg_steps
  double2* y2 = ws + (int64_t)a.seg_steps * nn;
  double2* y3 = y2 + nn;
  double2* y4 = y3 + nn;
  double2* kk = y4 + nn;
  double2* ab = kk + nn;
  double2* yb = ab + nn;
  double2* lnew = yb + nn;
  double2* X = lnew + nn;
  double2* lam_s = X + nn;
  double2* Y = lam_s + nn;
  double2* J = Y + nn;
  double2* lam = a.lam + (int64_t)b * nn;
  const double2* obs_ops = a.obs_ops ? a.obs_ops + p * a.obs_stride : nullptr;
  const double dt = a.dt, dt2 = a.dt / 2.0;

  // ---- forward recompute of the segment from its checkpoint ----
  for (int64_t e = threadIdx.x; e < nn; e += kThreads) seg[e] = a.ckpt[(int64_t)b * nn + e];
  __syncthreads();
  for (int s = 0; s + 1 < a.seg_steps; ++s) {
    const double2* r = seg + (int64_t)s * nn;
    double2* nxt = seg + (int64_t)(s + 1) * nn;
    // nxt accumulates k1 + 2k2 + 2k3 + k4 ; y2 holds the current stage input
    apply_gen<TM>(F, r, kk, X, Y, J, n, smem);
    for (int64_t e = threadIdx.x; e < nn; e += kThreads) { nxt[e] = kk[e]; y2[e] = cadd(r[e], cscale(kk[e], dt2)); }
    __syncthreads();
    apply_gen<TM>(F, y2, kk, X, Y, J, n, smem);
    for (int64_t e = threadIdx.x; e < nn; e += kThreads) { nxt[e] = cadd(nxt[e], cscale(kk[e], 2.0)); y2[e] = cadd(r[e], cscale(kk[e], dt2)); }
    __syncthreads();
    apply_gen<TM>(F, y2, kk, X, Y, J, n, smem);
    for (int64_t e = threadIdx.x; e < nn; e += kThreads) { nxt[e] = cadd(nxt[e], cscale(kk[e], 2.0)); y2[e] = cadd(r[e], cscale(kk[e], dt)); }
    __syncthreads();
    apply_gen<TM>(F, y2, kk, X, Y, J, n, smem);
    for (int64_t e = threadIdx.x; e < nn; e += kThreads) {
      const double2 sum = cadd(nxt[e], kk[e]);
      nxt[e] = cadd(r[e], cscale(make_double2(sum.x / 6., sum.y / 6.), dt));
    }
    __syncthreads();
  }

  // ---- backward through the segment ----
  double* GD = a.g_diag + (int64_t)b * n;
  double* GB = a.g_bond + (int64_t)b * (n > 1 ? n - 1 : 1);
  double* GG = a.g_gamma + (int64_t)b * n;
  for (int s = a.seg_steps - 1; s >= 0; --s) {
    const int gstep = a.step0 + s;   // the step rho_{gstep} -> rho_{gstep+1}
    // source: observable recorded after this step, Tr(E rho_{gstep+1})
    if (a.n_obs > 0 && ((gstep + 1) % a.obs_every) == 0) {
      const int slot = (gstep + 1) / a.obs_every - 1;
      const double2* gr = a.obs_grad + ((int64_t)b * a.obs_per_inst + slot) * a.n_obs;
      for (int64_t e = threadIdx.x; e < nn; e += kThreads) {
        const int i = (int)(e / n), j = (int)(e % n);
        double2 add = cz();
        for (int o = 0; o < a.n_obs; ++o) {
          // Hermitian part of g E^dag: (g conj(E_ji) + conj(g) E_ij) / 2
          double2 eji, eij;
          if (a.obs_diag) {
            const double2 d = (i == j) ? obs_ops[(int64_t)o * n + i] : cz();
            eji = d; eij = d;
          } else {
            eji = obs_ops[o * nn + (int64_t)j * n + i];
            eij = obs_ops[o * nn + (int64_t)i * n + j];
          }
          const double2 g = gr[o];
          add = cadd(add, cscale(cadd(cmul(g, cconj(eji)), cmul(cconj(g), eij)), 0.5));
        }
        lam[e] = cadd(lam[e], add);
      }
      __syncthreads();
    }
    const double2* r = seg + (int64_t)s * nn;
    // stage states y2, y3, y4 (y1 = r)
    apply_gen<TM>(F, r, kk, X, Y, J, n, smem);
    for (int64_t e = threadIdx.x; e < nn; e += kThreads) y2[e] = cadd(r[e], cscale(kk[e], dt2));
    __syncthreads();
    apply_gen<TM>(F, y2, kk, X, Y, J, n, smem);
    for (int64_t e = threadIdx.x; e < nn; e += kThreads) y3[e] = cadd(r[e], cscale(kk[e], dt2));
    __syncthreads();
    apply_gen<TM>(F, y3, kk, X, Y, J, n, smem);
    for (int64_t e = threadIdx.x; e < nn; e += kThreads) y4[e] = cadd(r[e], cscale(kk[e], dt));
    __syncthreads();
    // adjoint stages
    for (int64_t e = threadIdx.x; e < nn; e += kThreads) {
      lam_s[e] = lam[e];
      ab[e] = cscale(lam[e], dt / 6.0);
    }
    __syncthreads();
    apply_gen<TM>(A, ab, yb, X, Y, J, n, smem);                   // ybar4
    grad_terms(ab, y4, n, GD, GB, GG);
    __syncthreads();
    for (int64_t e = threadIdx.x; e < nn; e += kThreads) {
      lnew[e] = cadd(lam_s[e], yb[e]);
      ab[e] = cadd(cscale(lam_s[e], dt / 3.0), cscale(yb[e], dt));
    }
    __syncthreads();
    apply_gen<TM>(A, ab, yb, X, Y, J, n, smem);                   // ybar3
    grad_terms(ab, y3, n, GD, GB, GG);
    __syncthreads();
    for (int64_t e = threadIdx.x; e < nn; e += kThreads) {
      lnew[e] = cadd(lnew[e], yb[e]);
      ab[e] = cadd(cscale(lam_s[e], dt / 3.0), cscale(yb[e], dt2));
    }
    __syncthreads();
    apply_gen<TM>(A, ab, yb, X, Y, J, n, smem);                   // ybar2
    grad_terms(ab, y2, n, GD, GB, GG);
    __syncthreads();
    for (int64_t e = threadIdx.x; e < nn; e += kThreads) {
      lnew[e] = cadd(lnew[e], yb[e]);
      ab[e] = cadd(cscale(lam_s[e], dt / 6.0), cscale(yb[e], dt2));
    }
    __syncthreads();
    apply_gen<TM>(A, ab, yb, X, Y, J, n, smem);                   // ybar1
    grad_terms(ab, r, n, GD, GB, GG);
    __syncthreads();
    for (int64_t e = threadIdx.x; e < nn; e += kThreads) lam[e] = cadd(lnew[e], yb[e]);
    __syncthreads();
  }
}

// Heff = H - (i/2) sum_k L_k^dag L_k ;  M = sum_k l_k l_k^dag, one CTA per
// generator.  The dense part sum_k L_k^dag L_k arrives in heff (a strided
// batched GEMM run before this kernel) or is absent (k_dense = 0).  For the
// diagonal operators the diagonal sums dg[i] = sum_k |l_k[i]|^2 (which are
// both the diagonal of sum_k L_k^dag L_k and of M) are formed once per
// generator in shared memory, k in order, then the site-dephasing rate r_i;
// when every diagonal operator has at most one nonzero entry (site
// dephasing) the off-diagonal terms l_k[i] conj(l_k[j]) of M are exact zeros
// and are not summed.
__global__ void __launch_bounds__(kThreads) prepare_kernel(LimePrepareDesc d) {
  extern __shared__ double dg[];    // [n]
  const int b = blockIdx.x;
  const int n = d.n;
  const int nn = n * n;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const double2* H = reinterpret_cast<const double2*>(d.h) + b * d.h_stride;
  const double2* lg = d.l_diag ? reinterpret_cast<const double2*>(d.l_diag) + b * d.l_diag_stride : nullptr;
  const double* rate = d.dephasing ? d.dephasing + b * d.dephasing_stride : nullptr;
  double2* heff = reinterpret_cast<double2*>(d.heff) + (int64_t)b * nn;
  double2* M = reinterpret_cast<double2*>(d.m) + (int64_t)b * nn;
  __shared__ int spread;   // some l_k has two or more nonzero entries
  if (t == 0) spread = 0;
  for (int i = t; i < n; i += kThreads) {
    double s = 0.0;
    for (int k = 0; k < d.k_diag; ++k) {
      const double2 v = lg[(int64_t)k * n + i];
      s += v.x * v.x + v.y * v.y;
    }
    dg[i] = rate ? s + rate[i] : s;
  }
  __syncthreads();
  // one warp per operator counts its nonzero entries
  for (int k = warp; k < d.k_diag; k += kThreads / 32) {
    int cnt = 0;
    for (int i0 = 0; i0 < n; i0 += 32) {   // every lane takes part in each ballot
      const int i = i0 + lane;
      const double2 v = i < n ? lg[(int64_t)k * n + i] : cz();
      cnt += __popc(__ballot_sync(0xffffffffu, v.x != 0.0 || v.y != 0.0));
    }
    if (lane == 0 && cnt > 1) atomicOr(&spread, 1);
  }
  __syncthreads();
  for (int e = t; e < nn; e += kThreads) {
    const int i = e / n, j = e - i * n;
    double2 g = d.k_dense > 0 ? heff[e] : cz();   // (sum_k L_k^dag L_k)_ij of the dense operators
    double2 mm = cz();
    if (i == j) {
      g.x += dg[i];
      mm.x = dg[i];
    } else if (spread) {
      for (int k = 0; k < d.k_diag; ++k) {
        const double2* l = lg + (int64_t)k * n;
        cfma(mm, l[i], cconj(l[j]));
      }
    }
    // H - (i/2) g  =  (H.re + g.im/2, H.im - g.re/2)
    const double2 h = H[e];
    heff[e] = make_double2(h.x + 0.5 * g.y, h.y - 0.5 * g.x);
    M[e] = mm;
  }
}

}  // namespace f64
}  // namespace lime

using namespace lime;

extern "C" int lime_lindblad_prepare_f64(const LimePrepareDesc* d, void* stream) {
  if (!d || d->n <= 0 || d->batch <= 0 || d->k_dense < 0 || d->k_diag < 0) return LIME_ERR_ARG;
  if (!d->h || !d->heff || !d->m) return LIME_ERR_ARG;
  if ((d->k_dense > 0 && !d->l_dense) || (d->k_diag > 0 && !d->l_diag)) return LIME_ERR_ARG;
  if (d->h_stride < 0 || d->l_dense_stride < 0 || d->l_diag_stride < 0 || d->dephasing_stride < 0)
    return LIME_ERR_ARG;
  if ((size_t)d->n * sizeof(double) > 48 * 1024) return LIME_ERR_UNSUPPORTED;
  cudaStream_t st = (cudaStream_t)stream;
  if (d->k_dense > 0) {
    // heff[b] = sum_k L_k^dag L_k = [L_1; ..; L_K]^dag [L_1; ..; L_K] (K n x n
    // stacked), one strided batched FP64 GEMM over the generators
    LimeZgemmDesc g{};
    const int64_t n = d->n;
    g.M = d->n; g.N = d->n; g.K = (int32_t)(d->k_dense * n); g.batch = d->batch;
    g.conj_a = 1;
    g.A = d->l_dense; g.a_rs = 1; g.a_cs = n; g.a_bs = d->l_dense_stride;
    g.B = d->l_dense; g.b_rs = n; g.b_cs = 1; g.b_bs = d->l_dense_stride;
    g.C = d->heff; g.c_rs = n; g.c_cs = 1; g.c_bs = n * n;
    const int rc = lime_zgemm_strided_f64(&g, stream);
    if (rc != LIME_OK) return rc;
  }
  f64::prepare_kernel<<<d->batch, f64::kThreads, (size_t)d->n * sizeof(double), st>>>(*d);
  LIME_CUDA_TRY(cudaGetLastError());
  count_launch();
  return LIME_OK;
}

extern "C" size_t lime_lindblad_adjoint_f64_workspace(int32_t n, int32_t batch, int32_t seg_steps, int32_t k_dense) {
  if (n <= 0 || batch <= 0 || seg_steps <= 0 || k_dense < 0) return 0;
  return (size_t)batch * (size_t)f64::adj_ws_mats(seg_steps, k_dense) * (size_t)n * n * sizeof(double2);
}

template <int TM>
static int launch_adj(f64::AdjArgs& args, int batch, cudaStream_t st) {
  const size_t smem = (size_t)(16 * TM) * (f64::kKC + 1) * sizeof(double2) +
                      (size_t)f64::kKC * (16 * TM + 1) * sizeof(double2);
  auto kern = f64::lindblad_adjoint_f64_kernel<TM>;
  LIME_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kern<<<batch, f64::kThreads, smem, st>>>(args);
  LIME_CUDA_TRY(cudaGetLastError());
  count_launch();
  return LIME_OK;
}

extern "C" int lime_lindblad_adjoint_f64(const LimeAdjointDesc* d, void* stream) {
  if (!d) return LIME_ERR_ARG;
  if (d->n <= 0 || d->batch <= 0 || d->seg_steps <= 0 || d->step0 < 0 || d->k_dense < 0 || d->n_obs < 0)
    return LIME_ERR_ARG;
  if (d->step0 + d->seg_steps > d->total_steps) return LIME_ERR_ARG;
  if (!d->ckpt || !d->lam || !d->heff || !d->heff_adj || !d->workspace) return LIME_ERR_ARG;
  if (!d->grad_diag || !d->grad_bond || !d->grad_gamma) return LIME_ERR_ARG;
  if (d->k_dense > 0 && (!d->l_dense || !d->l_dense_adj)) return LIME_ERR_ARG;
  if ((d->m == nullptr) != (d->m_adj == nullptr)) return LIME_ERR_ARG;
  if (d->n_obs > 0 && (!d->obs_ops || !d->obs_grad)) return LIME_ERR_ARG;
  if (d->heff_stride < 0 || d->m_stride < 0 || d->l_dense_stride < 0 || d->heff_adj_stride < 0 ||
      d->m_adj_stride < 0 || d->l_dense_adj_stride < 0 || d->obs_stride < 0)
    return LIME_ERR_ARG;
  const int pb = d->param_batch > 0 ? d->param_batch : d->batch;
  if (pb > d->batch) return LIME_ERR_ARG;
  if (d->workspace_bytes < lime_lindblad_adjoint_f64_workspace(d->n, d->batch, d->seg_steps, d->k_dense))
    return LIME_ERR_WORKSPACE;
  f64::AdjArgs a{};
  a.n = d->n; a.param_batch = pb; a.seg_steps = d->seg_steps; a.step0 = d->step0;
  a.total_steps = d->total_steps; a.k_dense = d->k_dense; a.n_obs = d->n_obs; a.obs_diag = d->obs_diag;
  a.obs_every = d->obs_every > 0 ? d->obs_every : 1;
  a.obs_per_inst = d->total_steps / a.obs_every;
  a.dt = d->dt; a.sixth = sixth_of(d->dt);
  a.ckpt = reinterpret_cast<const double2*>(d->ckpt);
  a.lam = reinterpret_cast<double2*>(d->lam);
  a.heff = reinterpret_cast<const double2*>(d->heff); a.heff_stride = d->heff_stride;
  a.m = reinterpret_cast<const double2*>(d->m); a.m_stride = d->m_stride;
  a.ld = reinterpret_cast<const double2*>(d->l_dense); a.ld_stride = d->l_dense_stride;
  a.heff_adj = reinterpret_cast<const double2*>(d->heff_adj); a.heff_adj_stride = d->heff_adj_stride;
  a.m_adj = reinterpret_cast<const double2*>(d->m_adj); a.m_adj_stride = d->m_adj_stride;
  a.ld_adj = reinterpret_cast<const double2*>(d->l_dense_adj); a.ld_adj_stride = d->l_dense_adj_stride;
  a.obs_ops = reinterpret_cast<const double2*>(d->obs_ops); a.obs_stride = d->obs_stride;
  a.obs_grad = reinterpret_cast<const double2*>(d->obs_grad);
  a.g_diag = d->grad_diag; a.g_bond = d->grad_bond; a.g_gamma = d->grad_gamma;
  a.ws = reinterpret_cast<double2*>(d->workspace);
  cudaStream_t st = (cudaStream_t)stream;
  // Without dense operators the products run over the generators' nonzero
  // entries; a dense Heff costs half the tiles' FP64 work there too.
  if (d->k_dense == 0) return f64::launch_adjoint_rows(a, d->batch, st);
  if (d->n <= 16) return launch_adj<1>(a, d->batch, st);
  if (d->n <= 32) return launch_adj<2>(a, d->batch, st);
  return launch_adj<4>(a, d->batch, st);
}
