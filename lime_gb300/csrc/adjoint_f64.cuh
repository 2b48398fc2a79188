// Arguments of the FP64 Lindblad adjoint kernels.
#pragma once

#include "common.cuh"

namespace lime {
namespace f64 {

struct AdjArgs {
  int n, param_batch, seg_steps, step0, total_steps, k_dense, n_obs, obs_diag, obs_every, obs_per_inst;
  double dt;
  Sixth sixth;
  const double2* ckpt;
  double2* lam;
  const double2* heff; int64_t heff_stride;
  const double2* m; int64_t m_stride;
  const double2* ld; int64_t ld_stride;
  const double2* heff_adj; int64_t heff_adj_stride;
  const double2* m_adj; int64_t m_adj_stride;
  const double2* ld_adj; int64_t ld_adj_stride;
  const double2* obs_ops; int64_t obs_stride;
  const double2* obs_grad;
  double* g_diag;
  double* g_bond;
  double* g_gamma;
  double2* ws;
};

// workspace per instance, n x n complex matrices: the segment's states and
// the work matrices of either kernel
__host__ __device__ inline int64_t adj_ws_mats(int seg_steps, int k_dense) {
  return (int64_t)seg_steps + (k_dense > 0 ? 11 : 10);
}

// one segment without dense operators (lindblad_adjoint_rows_f64.cu)
int launch_adjoint_rows(const AdjArgs& a, int batch, cudaStream_t st);

}  // namespace f64
}  // namespace lime
