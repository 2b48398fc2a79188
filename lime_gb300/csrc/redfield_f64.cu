// Bloch-Redfield generator assembly and FP64 RK4 on vec(rho) (sm_103a).
//
// Generator (lime/oqs.py:528-579), in the eigenbasis of H with row-major
// Liouville index (a, b) -> a N + b (lime/superoperator.py:131-151):
//   L[ab, cd] = -i (E_a - E_b) d_ac d_bd - d_bd P_ac - d_ac Q_db
//               + sum_k ( A_k[a,c] conj(Lam_k[b,d]) + Lam_k[a,c] A_k[d,b] )
// with Lam_k = C_k o A_k, P = sum_k A_k Lam_k, Q = sum_k Lam_k^dag A_k.  This
// is the closed form of -1j op2sop(diag E) - sum_k op2sop(A_k)(left(Lam_k) -
// right(Lam_k^dag)); the O(N^4 K) sum is one GEMM U (N^2 x 2K) . V (2K x N^2)
// whose epilogue scatters (a,c),(d,b) to (ab, cd) and adds the local terms.
//
// Time stepping (lime/oqs.py:373-472): RK4 on the right-hand-side block
// P (D x R, column r = vec rho_r) with one GEMM Y = L S per stage and the
// stage combination fused into the GEMM epilogue.  FP64 throughout; this is
// the exact path (DFMA-bound on GB300).

#include "gemm_f64.cuh"
#include "redfield_vec_f64.cuh"

#include <math.h>

namespace lime {
namespace rf {

// ---------------------------------------------------------------- assembly
__global__ void lam_kernel(int n, int k, const double2* A, const double* C, int64_t c_stride, double2* Lam) {
  const int64_t nn = (int64_t)n * n;
  const int64_t total = (int64_t)k * nn;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x)
    Lam[e] = cscale(A[e], C[(e / nn) * c_stride + e % nn]);
}

// P = sum_k A_k Lam_k, Q = sum_k Lam_k^dag A_k (one element per thread)
__global__ void pq_kernel(int n, int k, const double2* A, const double2* Lam, double2* P, double2* Q) {
  const int64_t nn = (int64_t)n * n;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < nn; e += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(e / n), j = (int)(e % n);
    double2 p = cz(), q = cz();
    for (int kk = 0; kk < k; ++kk) {
      const double2* Ak = A + kk * nn;
      const double2* Lk = Lam + kk * nn;
      for (int m = 0; m < n; ++m) {
        cfma(p, Ak[(int64_t)i * n + m], Lk[(int64_t)m * n + j]);
        cfma(q, cconj(Lk[(int64_t)m * n + i]), Ak[(int64_t)m * n + j]);
      }
    }
    P[e] = p;
    Q[e] = q;
  }
}

struct BuildArgs {
  int n, k;
  const double* E;
  const double2* A;
  const double2* Lam;
  const double2* P;
  const double2* Q;
  double2* R;
};

__global__ void __launch_bounds__(kThreads) assemble_kernel(BuildArgs a) {
  const int n = a.n, K = a.k;
  const int64_t nn = (int64_t)n * n;
  const int D = n * n;
  // U[(a,c), kk] = kk < K ? A_kk[a,c] : Lam_{kk-K}[a,c]
  auto la = [&](int row, int kk) -> double2 {
    return kk < K ? a.A[kk * nn + row] : a.Lam[(kk - K) * nn + row];
  };
  // V[kk, (d,b)] = kk < K ? conj(Lam_kk[b,d]) : A_{kk-K}[d,b]
  auto lb = [&](int kk, int col) -> double2 {
    const int d = col / n, b = col % n;
    return kk < K ? cconj(a.Lam[kk * nn + (int64_t)b * n + d]) : a.A[(kk - K) * nn + col];
  };
  auto epi = [&](int row, int col, double2 v) {
    const int ai = row / n, ci = row % n, di = col / n, bi = col % n;
    if (bi == di) v = csub(v, a.P[(int64_t)ai * n + ci]);
    if (ai == ci) v = csub(v, a.Q[(int64_t)di * n + bi]);
    if (ai == ci && bi == di) v = cadd(v, make_double2(0.0, -(a.E[ai] - a.E[bi])));
    a.R[(int64_t)(ai * n + bi) * D + (ci * n + di)] = v;
  };
  gemm_tile(D, D, 2 * K, blockIdx.y * kTile, blockIdx.x * kTile, la, lb, epi);
}

// out[slot][r][o] = sum_ij E_o[j][i] rho_r[i][j] over kept states hist[slot][D][R],
// one warp each: D / 32 terms a lane, where one thread summing all D left the
// chip idle for 144 us a step at D = 400
__global__ void observe_kernel(int n, int R, int n_obs, int slots, const double2* Eops, const double2* hist,
                               double2* out) {
  const int64_t D = (int64_t)n * n, total = (int64_t)slots * R * n_obs;
  const int lane = threadIdx.x & 31;
  const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t t = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); t < total; t += nw) {
    const int o = (int)(t % n_obs);
    const int64_t sr = t / n_obs;
    const int r = (int)(sr % R);
    const double2* P = hist + (sr / R) * D * R + r;
    double2 s = cz();
    for (int64_t e = lane; e < D; e += 32) {
      const int64_t j = e / n, i = e - j * n;
      cfma(s, Eops[o * D + e], P[(i * n + j) * R]);
    }
    for (int w = 16; w > 0; w >>= 1) {
      s.x += __shfl_xor_sync(0xffffffffu, s.x, w);
      s.y += __shfl_xor_sync(0xffffffffu, s.y, w);
    }
    if (lane == 0) out[t] = s;
  }
}

static int observe(int n, int R, int n_obs, int slots, const double2* E, const double2* hist, double2* out,
                   cudaStream_t st) {
  const int64_t warps = (int64_t)slots * R * n_obs, blocks = (warps + 3) / 4;
  observe_kernel<<<(unsigned)(blocks < 65535 ? blocks : 65535), 128, 0, st>>>(n, R, n_obs, slots, E, hist, out);
  LIME_CUDA_TRY(cudaGetLastError());
  count_launch();
  return LIME_OK;
}

}  // namespace rf
}  // namespace lime

using namespace lime;

extern "C" size_t lime_redfield_build_f64_workspace(int32_t n, int32_t k) {
  if (n <= 0 || k <= 0) return 0;
  const size_t nn = (size_t)n * n;
  return ((size_t)k * nn + 2 * nn) * sizeof(double2);
}

extern "C" int lime_redfield_build_f64(const LimeRedfieldBuildDesc* d, void* stream) {
  if (!d || d->n <= 0 || d->k <= 0 || d->spec_stride < 0) return LIME_ERR_ARG;
  if (!d->evals || !d->a_eig || !d->spec || !d->R || !d->workspace) return LIME_ERR_ARG;
  if ((int64_t)d->n * d->n > 46340) return LIME_ERR_UNSUPPORTED;   // D^2 must fit 31-bit tiles
  if (d->workspace_bytes < lime_redfield_build_f64_workspace(d->n, d->k)) return LIME_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  const int n = d->n, k = d->k;
  const size_t nn = (size_t)n * n;
  double2* Lam = reinterpret_cast<double2*>(d->workspace);
  double2* P = Lam + (size_t)k * nn;
  double2* Q = P + nn;
  const double2* A = reinterpret_cast<const double2*>(d->a_eig);
  const int eb = (int)(((size_t)k * nn + 255) / 256);
  rf::lam_kernel<<<eb < 4096 ? eb : 4096, 256, 0, st>>>(n, k, A, d->spec, d->spec_stride, Lam);
  LIME_CUDA_TRY(cudaGetLastError());
  const int pb = (int)((nn + 255) / 256);
  rf::pq_kernel<<<pb, 256, 0, st>>>(n, k, A, Lam, P, Q);
  LIME_CUDA_TRY(cudaGetLastError());
  rf::BuildArgs a{n, k, d->evals, A, Lam, P, Q, reinterpret_cast<double2*>(d->R)};
  const int D = n * n;
  dim3 grid((D + rf::kTile - 1) / rf::kTile, (D + rf::kTile - 1) / rf::kTile);
  rf::assemble_kernel<<<grid, rf::kThreads, 0, st>>>(a);
  LIME_CUDA_TRY(cudaGetLastError());
  count_launch(3);
  return LIME_OK;
}

extern "C" int lime_redfield_assemble_f64(const LimeRedfieldAssembleDesc* d, void* stream) {
  if (!d || d->n <= 0 || d->k <= 0) return LIME_ERR_ARG;
  if (!d->evals || !d->a_eig || !d->lam || !d->p || !d->q || !d->R) return LIME_ERR_ARG;
  if ((int64_t)d->n * d->n > 46340) return LIME_ERR_UNSUPPORTED;
  const int D = d->n * d->n;
  rf::BuildArgs a{d->n, d->k, d->evals, reinterpret_cast<const double2*>(d->a_eig),
                  reinterpret_cast<const double2*>(d->lam), reinterpret_cast<const double2*>(d->p),
                  reinterpret_cast<const double2*>(d->q), reinterpret_cast<double2*>(d->R)};
  dim3 grid((D + rf::kTile - 1) / rf::kTile, (D + rf::kTile - 1) / rf::kTile);
  rf::assemble_kernel<<<grid, rf::kThreads, 0, (cudaStream_t)stream>>>(a);
  LIME_CUDA_TRY(cudaGetLastError());
  count_launch();
  return LIME_OK;
}

extern "C" size_t lime_redfield_rk4_f64_workspace(int32_t n, int32_t n_rhs) {
  if (n <= 0 || n_rhs <= 0) return 0;
  const size_t tiled = (size_t)3 * n * n * n_rhs * sizeof(double2);
  if ((int64_t)n * n > 46340 || !rfv::supported(n * n, n_rhs)) return tiled;
  return tiled + rfv::workspace(n * n, n_rhs);
}

// The time loop in single launches: a chunk is as many steps as the kept
// states have slots for, and at most about a tenth of a second by the plan's
// count of a stage's clocks.
static int rk4_vec(const LimeRedfieldRK4Desc* d, const rfv::Plan& plan, int32_t* status, uint32_t max_wait,
                   cudaStream_t st) {
  const int n = d->n, D = n * n, R = d->n_rhs;
  const size_t DR = (size_t)D * R;
  const int obs_every = d->obs_every > 0 ? d->obs_every : 1;
  rfv::Run r{};
  r.D = D; r.R = R; r.n_steps = d->n_steps; r.dt = d->dt;
  r.L = reinterpret_cast<const double2*>(d->R);
  r.P = reinterpret_cast<double2*>(d->rho);
  r.ws = reinterpret_cast<double2*>(d->workspace) + 3 * DR;
  r.states = reinterpret_cast<double2*>(d->states); r.states_every = d->states_every;
  r.obs_every = d->n_obs > 0 ? obs_every : 0;
  r.status = status; r.max_wait = max_wait > 0 ? max_wait : rfv::kPollLimit;
  // the caller's states serve the observables when they are the same steps
  const bool own = d->n_obs > 0 && !(d->states && d->states_every == obs_every);
  double2* out = reinterpret_cast<double2*>(d->obs_out);
  const double2* E = reinterpret_cast<const double2*>(d->obs_ops);
  int rc = rfv::begin(plan, r, st);
  if (rc != LIME_OK) return rc;
  constexpr double kLaunchClocks = 2e8;
  int64_t chunk = (int64_t)fmax(1.0, fmin((double)d->n_steps, kLaunchClocks / (4.0 * plan.clocks)));
  if (own && chunk > (int64_t)rfv::kHistory * obs_every) chunk = (int64_t)rfv::kHistory * obs_every;
  for (int64_t s0 = 0; s0 < d->n_steps; s0 += chunk) {
    const int steps = (int)(d->n_steps - s0 < chunk ? d->n_steps - s0 : chunk);
    double2* hist = own ? rfv::history(r) : nullptr;
    rc = rfv::launch(plan, r, (int)s0, steps, hist, st);
    if (rc != LIME_OK) return rc;
    const int64_t k0 = s0 / obs_every, slots = (s0 + steps) / obs_every - k0;
    if (own && slots > 0) {
      rc = rf::observe(n, R, d->n_obs, (int)slots, E, hist, out + k0 * R * d->n_obs, st);
      if (rc != LIME_OK) return rc;
    }
  }
  if (d->n_obs > 0 && !own && d->n_steps / obs_every > 0)
    return rf::observe(n, R, d->n_obs, d->n_steps / obs_every, E, r.states, out, st);
  return LIME_OK;
}

// withhold: the plan lacks its last CTA, whose words the others wait for
static int rk4_f64(const LimeRedfieldRK4Desc* d, int32_t* status, uint32_t max_wait, bool withhold, void* stream) {
  if (!d || d->n <= 0 || d->n_rhs <= 0 || d->n_steps < 0 || d->n_obs < 0) return LIME_ERR_ARG;
  if (!d->R || !d->rho || !d->workspace) return LIME_ERR_ARG;
  if (d->n_obs > 0 && (!d->obs_ops || !d->obs_out)) return LIME_ERR_ARG;
  if (d->states && d->states_every <= 0) return LIME_ERR_ARG;
  if ((int64_t)d->n * d->n > 46340) return LIME_ERR_UNSUPPORTED;
  const int D = d->n * d->n, R = d->n_rhs;
  const size_t DR = (size_t)D * R;
  if (d->workspace_bytes < 3 * DR * sizeof(double2)) return LIME_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  // Few right-hand sides: one launch for the time loop, where the workspace
  // has room for its exchange (a caller that sized it for the tiled path
  // alone stays there).  From kMaxRhs right-hand sides on a tile's columns
  // are used and the tiled GEMM is as near to the FP64 bound.
  if (d->n_steps > 0 && d->workspace_bytes >= lime_redfield_rk4_f64_workspace(d->n, R)) {
    int dev = 0, sms = 0;
    LIME_CUDA_TRY(cudaGetDevice(&dev));
    LIME_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    rfv::Plan plan;
    const bool one = rfv::plan(D, R, sms, &plan);
    if (withhold) {
      if (!one || plan.mode != rfv::kGrid) return LIME_ERR_UNSUPPORTED;
      --plan.ctas;
    }
    if (one) return rk4_vec(d, plan, status, max_wait, st);
  }
  if (withhold) return LIME_ERR_UNSUPPORTED;
  double2* P = reinterpret_cast<double2*>(d->rho);
  double2* acc = reinterpret_cast<double2*>(d->workspace);
  double2* S0 = acc + DR;
  double2* S1 = S0 + DR;
  const int obs_every = d->obs_every > 0 ? d->obs_every : 1;
  dim3 grid((R + rf::kTile - 1) / rf::kTile, (D + rf::kTile - 1) / rf::kTile);
  int64_t launches = 0;
  for (int step = 0; step < d->n_steps; ++step) {
    const double2* S = P;
    for (int s = 0; s < 4; ++s) {
      double2* Sn = (s % 2 == 0) ? S0 : S1;
      rf::StageArgs a{D, R, s, d->dt, reinterpret_cast<const double2*>(d->R), S, P, acc, Sn};
      rf::stage_kernel<<<grid, rf::kThreads, 0, st>>>(a);
      LIME_CUDA_TRY(cudaGetLastError());
      ++launches;
      S = Sn;
    }
    if (d->n_obs > 0 && ((step + 1) % obs_every) == 0) {
      const int slot = (step + 1) / obs_every - 1;
      // obs_out layout [slot][R][n_obs]
      const int rc = rf::observe(d->n, R, d->n_obs, 1, reinterpret_cast<const double2*>(d->obs_ops), P,
                                 reinterpret_cast<double2*>(d->obs_out) + (size_t)slot * R * d->n_obs, st);
      if (rc != LIME_OK) return rc;
    }
    if (d->states && ((step + 1) % d->states_every) == 0) {
      const int slot = (step + 1) / d->states_every - 1;
      LIME_CUDA_TRY(cudaMemcpyAsync(reinterpret_cast<double2*>(d->states) + (size_t)slot * DR, P,
                                    DR * sizeof(double2), cudaMemcpyDeviceToDevice, st));
    }
  }
  count_launch(launches);
  return LIME_OK;
}

extern "C" int lime_redfield_rk4_f64(const LimeRedfieldRK4Desc* d, void* stream) {
  return rk4_f64(d, nullptr, 0, false, stream);
}

extern "C" int lime_redfield_rk4_f64_status(const LimeRedfieldRK4Desc* d, int32_t* status, uint32_t max_wait,
                                            void* stream) {
  return rk4_f64(d, status, max_wait, false, stream);
}

extern "C" int lime_redfield_wait_selftest(const LimeRedfieldRK4Desc* d, int32_t* status, uint32_t max_wait,
                                           void* stream) {
  if (!status || max_wait == 0) return LIME_ERR_ARG;
  return rk4_f64(d, status, max_wait, true, stream);
}
