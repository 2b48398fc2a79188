// Discrete FP64 adjoint of the Lindblad RK4 steps without dense collapse
// operators (no counterpart in the reference, which has no gradients).
//
// One CTA owns one density matrix.  As in the forward kernel the FP64 pipe is
// the bound, so both generators (Heff and its adjoint -Heff^dag) run over
// their nonzero entries, element by element of the upper triangle and one
// real component at a time (rows_f64.cuh).  Per step: the three stage states
// again, four adjoint stages, and per stage the products that the gradients
// sum.  Those are added per element over a step, the steps' sums per element
// over the segment, and the elements once at its end: one sum per element
// over all stages has up to 1.3 times the rounding error of sums by rows at
// each stage, the two levels have 0.7 to 1.05 times.  The states and adjoint
// stage inputs are full matrices, double buffered so that a stage costs one
// barrier, in shared memory as far as they fit (n up to 41), else in the
// caller's workspace.
//
// Measured against tiled GEMMs of the full Heff in every stage, with the
// gradient sums in n threads: 32 matrices of 25 levels, 16 steps, 7.35 -> 0.57
// ms (43 000 clocks of FP64 a step and matrix are 0.35 ms).

#include "adjoint_f64.cuh"
#include "rows_f64.cuh"

#include <type_traits>

namespace lime {
namespace f64 {

constexpr int kAdjThreads = 512;
constexpr int kAdjRowCap = 2048;       // entries of each generator's list in shared memory
constexpr size_t kAdjSmem = 224 * 1024;

// kE > 0: kE items a thread, the diagonal coefficients of both generators in
// registers; kE = 0: any number, coefficients formed at each use.
template <int kE>
__global__ void __launch_bounds__(kAdjThreads, 1) adjoint_rows_kernel(AdjArgs a, int row_cap, size_t smem_bytes) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ RowsBuild rb;
  using Idx = typename std::conditional<kE == 0, int64_t, int>::type;
  const int t = threadIdx.x, nt = blockDim.x, lane = t & 31, warp = t >> 5, nw = nt >> 5;
  const int b = blockIdx.x, n = a.n, p = b % a.param_batch;
  const int64_t nn = (int64_t)n * n;
  const Idx ld2 = 2 * (Idx)n;
  const double2* heff = a.heff + p * a.heff_stride;
  const double2* hadj = a.heff_adj + p * a.heff_adj_stride;
  const double2* m = a.m ? a.m + p * a.m_stride : nullptr;
  const double2* madj = a.m_adj ? a.m_adj + p * a.m_adj_stride : nullptr;
  const double2* obs_ops = a.obs_ops ? a.obs_ops + p * a.obs_stride : nullptr;
  double2* seg = a.ws + (int64_t)b * adj_ws_mats(a.seg_steps, 0) * nn;   // rho_{step0 + s}, s < seg_steps
  double2* ws = seg + (int64_t)a.seg_steps * nn;                        // 10 matrices
  double2* lam_io = a.lam + (int64_t)b * nn;

  // ---- shared memory: the row lists, then matrices while they fit, else
  // their places in the workspace
  double2* sp = reinterpret_cast<double2*>(smem);
  int64_t left = (int64_t)(smem_bytes / 16);
  auto take = [&](int64_t count, double2* global) {
    if (count > left) return global;
    double2* at = sp;
    sp += count;
    left -= count;
    return at;
  };
  const bool small = n <= kRowsSmemMax;
  double2* const dF = take(small ? n : 0, ws);
  double2* const dA = take(small ? n : 0, ws);
  double2* const vF = take(row_cap, ws);
  double2* const vA = take(row_cap, ws);
  double2* const abA = take(nn, ws + 2 * nn);
  double2* const abB = take(nn, ws + 3 * nn);
  double2* const y2 = take(nn, ws + 4 * nn);
  double2* const y3 = take(nn, ws + 5 * nn);
  double2* const y4 = take(nn, ws + 6 * nn);
  double2* const xs = take(nn, nullptr);                 // the step's state (else read from seg)
  // one double an item: lam, a running sum, and the gradients' products
  double* const half = reinterpret_cast<double*>(ws + 7 * nn);
  const int64_t hn = (nn + 1) / 2;
  double* const lam = reinterpret_cast<double*>(take(hn, reinterpret_cast<double2*>(half)));
  double* const sum = reinterpret_cast<double*>(take(hn, reinterpret_cast<double2*>(half + nn)));
  double* const VW = half + 2 * nn;   // a step's sums of the products
  double* const BS = half + 3 * nn;
  double* const VWs = half + 4 * nn;  // the segment's
  double* const BSs = half + 5 * nn;
  const auto entF = [&](int i, int c) { return heff[(int64_t)i * n + c]; };
  const auto entA = [&](int i, int c) { return hadj[(int64_t)i * n + c]; };
  const auto nonzero = [](double2 v) { return v.x != 0.0 || v.y != 0.0; };
  const Rows F = build_rows(entF, [&](int i, int c) { return nonzero(entF(i, c)); },
                            [&](int i, int c) { return entF(i, c).y != 0.0; }, n, (int)ld2, vF, row_cap, ws, dF, &rb);
  const Rows A = build_rows(entA, [&](int i, int c) { return nonzero(entA(i, c)); },
                            [&](int i, int c) { return entA(i, c).y != 0.0; }, n, (int)ld2, vA, row_cap, ws + nn, dA,
                            &rb);
  const auto coef = [&](const Rows& R, const double2* M, const Item& it) {
    return diag_coef(R.d[it.p], R.d[it.q], M ? M[(int64_t)it.p * n + it.q] : cz());
  };
  constexpr int kReg = kE > 0 ? kE : 1;
  double2 cF[kReg], cA[kReg];
  if (kE > 0) {
#pragma unroll
    for (int u = 0; u < kReg; ++u) {
      const int e = t + u * nt;
      cF[u] = cA[u] = cz();
      if (e < nn) {
        const Item it = item_of(e / n, e % n);
        cF[u] = coef(F, m, it);
        cA[u] = coef(A, madj, it);
      }
    }
  }
  // body(item number, item, register slot) over this thread's items
  const auto items = [&](const auto& body) {
    if (kE > 0) {
#pragma unroll
      for (int u = 0; u < kReg; ++u) {
        const int e = t + u * nt;
        if (e < nn) body((Idx)e, item_of(e / n, e % n), u);
      }
    } else {
      for (int64_t e = t; e < nn; e += nt) body((Idx)e, item_of((int)(e / n), (int)(e % n)), 0);
    }
  };
  const auto rhs = [&](const Rows& R, const double2 (&c)[kReg], const double2* M, const double2* x, const Item& it,
                       int u) {
    const Item i1[1] = {it};
    const double2 c1[1] = {kE > 0 ? c[u] : coef(R, M, it)};
    double f1[1];
    rhs_items<1, false, Idx>(R, c1, reinterpret_cast<const double*>(x), ld2, i1, f1);
    return f1[0];
  };
  const auto own = [&](const double2* x, const Item& it) {
    return reinterpret_cast<const double*>(x)[(Idx)it.p * ld2 + 2 * it.q + it.im];
  };
  const auto put = [&](double2* x, const Item& it, double v) {
    double* o = reinterpret_cast<double*>(x);
    o[(Idx)it.p * ld2 + 2 * it.q + it.im] = v;
    if (it.p != it.q) o[(Idx)it.q * ld2 + 2 * it.p + it.im] = it.im ? -v : v;
    else o[(Idx)it.p * ld2 + 2 * it.q + 1] = 0.0;
  };
  const double dt = a.dt, dt2 = a.dt / 2.0, dt3 = a.dt / 3.0, dt6 = a.dt / 6.0;

  // ---- forward recompute of the segment from its checkpoint
  items([&](Idx e, const Item& it, int) {
    const double v = own(a.ckpt + (int64_t)b * nn, it);
    put(seg, it, v);
    if (xs) put(xs, it, v);
    lam[e] = own(lam_io, it);
    VWs[e] = 0.0;
    BSs[e] = 0.0;
  });
  __syncthreads();
  for (int s = 0; s + 1 < a.seg_steps; ++s) {
    const double2* const r = xs ? xs : seg + (int64_t)s * nn;
    double2* const nxt = seg + (int64_t)(s + 1) * nn;
    items([&](Idx e, const Item& it, int u) {
      const double f = rhs(F, cF, m, r, it, u);
      sum[e] = f;
      put(y2, it, fma(dt2, f, own(r, it)));
    });
    __syncthreads();
    items([&](Idx e, const Item& it, int u) {
      const double f = rhs(F, cF, m, y2, it, u);
      sum[e] = fma(2.0, f, sum[e]);
      put(y3, it, fma(dt2, f, own(r, it)));
    });
    __syncthreads();
    items([&](Idx e, const Item& it, int u) {
      const double f = rhs(F, cF, m, y3, it, u);
      sum[e] = fma(2.0, f, sum[e]);
      put(y4, it, fma(dt, f, own(r, it)));
    });
    __syncthreads();
    items([&](Idx e, const Item& it, int u) {
      const double f = rhs(F, cF, m, y4, it, u);
      const double v = rk4_final_f64(own(r, it), sum[e] + f, a.sixth);
      put(nxt, it, v);
      if (xs) put(xs, it, v);
    });
    __syncthreads();
  }

  // ---- backward through the segment
  // the products of adjoint stage input ab and stage state y that the
  // gradients sum: Im(conj(ab_pq) y_pq) with the items of the upper triangle,
  // Re(conj(ab_pq) y_pq) with those of the lower one (both Hermitian), the
  // bond's at every element
  enum { kFirst, kNext, kLast };   // stage of the step
  const auto products = [&](Idx e, const Item& it, const double2* ab, const double2* y, int stage) {
    const auto add = [&](double* part, double* total, const auto& term) {
      const double v = term(stage == kFirst ? 0.0 : part[e]);
      if (stage == kLast) total[e] += v;
      else part[e] = v;
    };
    if (it.p != it.q) {
      const double2 av = ab[(Idx)it.p * n + it.q], yv = y[(Idx)it.p * n + it.q];
      add(VW, VWs, [&](double v) {
        return it.im ? fma(av.x, yv.x, fma(av.y, yv.y, v)) : fma(av.x, yv.y, fma(-av.y, yv.x, v));
      });
    }
    const Idx k = it.im ? it.q : it.p, x = it.im ? it.p : it.q;
    if (k + 1 < n) {
      const double2 a1 = ab[k * n + x], a2 = ab[(k + 1) * n + x], v1 = y[k * n + x], v2 = y[(k + 1) * n + x];
      add(BS, BSs, [&](double v) {
        return fma(a1.x, v2.y, fma(-a1.y, v2.x, fma(a2.x, v1.y, fma(-a2.y, v1.x, v))));
      });
    }
  };
  for (int s = a.seg_steps - 1; s >= 0; --s) {
    const int gstep = a.step0 + s;   // the step rho_{gstep} -> rho_{gstep+1}
    const double2* const rs = seg + (int64_t)s * nn;
    const double2* const r = xs ? xs : rs;
    const bool source = a.n_obs > 0 && (gstep + 1) % a.obs_every == 0;
    const double2* gr =
        source ? a.obs_grad + ((int64_t)b * a.obs_per_inst + (gstep + 1) / a.obs_every - 1) * a.n_obs : nullptr;
    if (xs && s + 1 < a.seg_steps) {
      items([&](Idx, const Item& it, int) { put(xs, it, own(rs, it)); });
      __syncthreads();
    }
    items([&](Idx e, const Item& it, int u) {
      const double f = rhs(F, cF, m, r, it, u);
      put(y2, it, fma(dt2, f, own(r, it)));
      if (source) {
        // Hermitian part of g E^dag: (g conj(E_qp) + conj(g) E_pq) / 2
        double add = 0.0;
        for (int o = 0; o < a.n_obs; ++o) {
          double2 eqp = cz(), epq = cz();
          if (!a.obs_diag) {
            eqp = obs_ops[o * nn + (int64_t)it.q * n + it.p];
            epq = obs_ops[o * nn + (int64_t)it.p * n + it.q];
          } else if (it.p == it.q) {
            eqp = epq = obs_ops[(int64_t)o * n + it.p];
          }
          if (!nonzero(eqp) && !nonzero(epq)) continue;
          const double2 g = gr[o];
          add += 0.5 * (it.im ? (g.y * eqp.x - g.x * eqp.y) + (g.x * epq.y - g.y * epq.x)
                              : (g.x * eqp.x + g.y * eqp.y) + (g.x * epq.x + g.y * epq.y));
        }
        lam[e] += add;
      }
      put(abA, it, dt6 * lam[e]);
    });
    __syncthreads();
    items([&](Idx, const Item& it, int u) { put(y3, it, fma(dt2, rhs(F, cF, m, y2, it, u), own(r, it))); });
    __syncthreads();
    items([&](Idx, const Item& it, int u) { put(y4, it, fma(dt, rhs(F, cF, m, y3, it, u), own(r, it))); });
    __syncthreads();
    // ab_4 = dt/6 lam; ab_3 = dt/3 lam + dt yb_4; ab_2 = dt/3 lam + dt/2 yb_3; ab_1 = dt/6 lam + dt/2 yb_2
    items([&](Idx e, const Item& it, int u) {
      const double yb = rhs(A, cA, madj, abA, it, u);
      sum[e] = lam[e] + yb;
      put(abB, it, fma(dt, yb, dt3 * lam[e]));
      products(e, it, abA, y4, kFirst);
    });
    __syncthreads();
    items([&](Idx e, const Item& it, int u) {
      const double yb = rhs(A, cA, madj, abB, it, u);
      sum[e] += yb;
      put(abA, it, fma(dt2, yb, dt3 * lam[e]));
      products(e, it, abB, y3, kNext);
    });
    __syncthreads();
    items([&](Idx e, const Item& it, int u) {
      const double yb = rhs(A, cA, madj, abA, it, u);
      sum[e] += yb;
      put(abB, it, fma(dt2, yb, dt6 * lam[e]));
      products(e, it, abA, y2, kNext);
    });
    __syncthreads();
    items([&](Idx e, const Item& it, int u) {
      const double yb = rhs(A, cA, madj, abB, it, u);
      lam[e] = sum[e] + yb;
      products(e, it, abB, r, kLast);
    });
    __syncthreads();
  }

  // ---- adjoint state and the gradients' sums, a warp a row
  items([&](Idx e, const Item& it, int) { put(lam_io, it, lam[e]); });
  double* const GD = a.g_diag + (int64_t)b * n;
  double* const GB = a.g_bond + (int64_t)b * (n > 1 ? n - 1 : 1);
  double* const GG = a.g_gamma + (int64_t)b * n;
  for (int k = warp; k < n; k += nw) {
    double d = 0.0, g = 0.0, w = 0.0;
    for (int x = lane; x < n; x += 32) {
      const int64_t up = x > k ? (int64_t)k * n + x : (int64_t)x * n + k;   // item (min, max)
      const int64_t lo = x > k ? (int64_t)x * n + k : (int64_t)k * n + x;   // item (max, min)
      if (x != k) {
        d += x > k ? VWs[up] : -VWs[up];
        g -= VWs[lo];
      }
      w += BSs[(int64_t)k * n + x];
    }
    for (int o = 16; o > 0; o >>= 1) {
      d += __shfl_xor_sync(0xffffffffu, d, o);
      g += __shfl_xor_sync(0xffffffffu, g, o);
      w += __shfl_xor_sync(0xffffffffu, w, o);
    }
    if (lane == 0) {
      GD[k] += 2.0 * d;
      GG[k] += g;
      if (k + 1 < n) GB[k] += 2.0 * w;
    }
  }
}

template <int kE>
static int launch_rows(const AdjArgs& a, int batch, int threads, int row_cap, size_t smem, cudaStream_t st) {
  auto kern = adjoint_rows_kernel<kE>;
  // (one value for every shape: calls of other threads set the same attribute)
  LIME_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAdjSmem));
  kern<<<batch, threads, smem, st>>>(a, row_cap, smem);
  LIME_CUDA_TRY(cudaGetLastError());
  count_launch();
  return LIME_OK;
}

int launch_adjoint_rows(const AdjArgs& a, int batch, cudaStream_t st) {
  const int64_t n = a.n, nn = n * n;
  const int row_cap = (int)(n > kRowsSmemMax ? 0 : n * (n - 1) < kAdjRowCap ? n * (n - 1) : kAdjRowCap);
  // lists, diagonals, six matrices and two item arrays, as far as they fit
  const int64_t want = 16 * (2 * row_cap + 2 * (n > kRowsSmemMax ? 0 : n) + 6 * nn + 2 * ((nn + 1) / 2));
  const size_t smem = (size_t)(want < (int64_t)kAdjSmem ? want : (int64_t)kAdjSmem);
  const int threads = (int)(nn >= kAdjThreads ? kAdjThreads : (nn + 31) / 32 * 32);
  const int64_t per = (nn + threads - 1) / threads;
  return per <= 1   ? launch_rows<1>(a, batch, threads, row_cap, smem, st)
         : per <= 2 ? launch_rows<2>(a, batch, threads, row_cap, smem, st)
         : per <= 4 ? launch_rows<4>(a, batch, threads, row_cap, smem, st)
                    : launch_rows<0>(a, batch, threads, row_cap, smem, st);
}

}  // namespace f64
}  // namespace lime
