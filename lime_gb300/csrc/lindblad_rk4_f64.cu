// Plain FP64 Lindblad RK4 propagator (sm_103a).
//
// One CTA, or a cluster of 2, 4 or 8 CTAs, owns one density matrix for the
// whole time loop.  Every thread owns up to E of the n^2 real numbers of the
// Hermitian state (rows_f64.cuh; the host splits non-Hermitian inputs): their
// value, RK4 accumulator and diagonal coefficient stay in registers, the
// stage input is a full matrix in shared memory (or, for a cluster and for
// n > 64, in the caller's workspace, read through L2), double-buffered so
// that a stage costs one barrier.  The right-hand side runs over the nonzero
// entries of the generator; the RK4 combination (lime/phys.py:636-649), the
// trace check and the observables of lime/phys.py:837-844 follow in the same
// thread; with one item a thread, where the time is one stage's latency, the
// narrow observables and the trace check are a helper warp's.
//
// Bound: the FP64 pipe, so the work of one matrix is its DFMA count and a
// batch smaller than the chip is spread over clusters.  Measured per RK4 step
// against tiled GEMMs of the full Heff and L_k over one CTA: 16-site chain,
// one instance, 58 -> 5.0 us (a stage's DFMA alone take 0.57 us of its 1.2);
// 64-site chain, 512 instances, 4.9 -> 0.24 ms; 37 levels with three dense
// operators, 48 instances, 5.6 -> 0.61 ms.

#include "rows_f64.cuh"

#include <math.h>

#include <type_traits>

namespace lime {
namespace f64 {

constexpr int kMaxThreads = 512;
constexpr int kMaxObs = 512;       // observables whose nonzero range is kept
constexpr int kNarrow = 4;         // widest diagonal observable summed by one thread
constexpr int kMaxFlagOps = 512;   // collapse operators that can take the entry lists
constexpr int kSparseRow = 2;      // entries a row of an operator that takes them

// Workspace layout per instance (complex elements), n x n matrices:
//   rs0 | rs1 | acc, f (n^2 doubles each) | generator values | Y0 | Y1
// (Y only with dense operators).
__host__ __device__ inline int64_t ws_mats(int k_dense) { return k_dense > 0 ? 6 : 4; }

struct RK4Args {
  int n, param_batch, n_steps, k_dense, n_obs, obs_diag, states_every, states_per_inst, step0;
  double dt, trace_tol;
  Sixth sixth;
  double2* rho;
  const double2* heff;    int64_t heff_stride;
  const double2* m;       int64_t m_stride;
  const double2* l_dense; int64_t l_dense_stride;
  const double2* obs_ops; int64_t obs_stride;
  double2* obs_out;       int obs_every, obs_per_inst;
  double2* states;
  double2* ws;
  double* tr0;
  int32_t* status;
  int n_drive;
  const double2* drive_ops;
  const double* drive_coef;
  int b0;                 // first instance of the launch (the batch's pointers start there)
  // shared-memory plan (RK4Plan)
  int cluster, ld, vcap, row_cap, y_smem;
  // extents for the bounds-checked build (elements of obs_out and states)
  size_t obs_elems = kNoExtent, states_elems = kNoExtent;
};

struct Head {
  RowsBuild rb;
  int max_row, n_dense;
  int dense_op[kMaxFlagOps];
  short2 obs_rng[kMaxObs];
};

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// sum of the warp's values
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// kE > 0: kE elements a thread in registers; kE = 0: any number, state and
// accumulators in global memory.  kCg: the stage input and Y are shared by
// the CTAs of a cluster (read through L2).
template <int kE, bool kCg>
__global__ void __launch_bounds__(kE == 1 ? kMaxThreads + 32 : kMaxThreads, 1) lindblad_rk4_f64_kernel(RK4Args a) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ Head S;
  // worker threads 0 .. nt - 1; kHelp: one more warp, the helper, takes the
  // narrow observables and the trace, else warp 0 does
  constexpr bool kHelp = kE == 1;
  const int t = threadIdx.x, nt = kHelp ? blockDim.x - 32 : blockDim.x, lane = t & 31, warp = t >> 5, nw = nt >> 5;
  const bool helper = kHelp && warp == nw;
  const bool side = warp == (kHelp ? nw : 0);
  const int nwa = blockDim.x >> 5;
  const int C = kCg ? a.cluster : 1;
  const int rank = kCg ? (int)(blockIdx.x % C) : 0;
  const int b = kCg ? (int)(blockIdx.x / C) : (int)blockIdx.x;
  const int n = a.n, ld = a.ld;
  const int64_t nn = (int64_t)n * n;
  const int p = (a.b0 + b) % a.param_batch;
  double2* rho = a.rho + b * nn;
  const double2* heff0 = a.heff + p * a.heff_stride;
  const double2* m = a.m ? a.m + p * a.m_stride : nullptr;
  const double2* ldn = a.l_dense ? a.l_dense + p * a.l_dense_stride : nullptr;
  const double2* obs_ops = a.obs_ops ? a.obs_ops + p * a.obs_stride : nullptr;
  double2* ws = a.ws + (int64_t)b * ws_mats(a.k_dense) * nn;

  // ---- shared memory: stage inputs, Y, generator values, diagonal, operator entries, their counts
  const bool small = n <= kRowsSmemMax;
  constexpr bool kSm = !kCg && kE > 0;                 // stage inputs in shared memory
  using Idx = typename std::conditional<kE == 0, int64_t, int>::type;
  double2* sp = reinterpret_cast<double2*>(smem);
  const Idx ld2 = 2 * (Idx)ld, half = (kSm ? (Idx)n * ld : (Idx)nn) * 2;   // doubles a row, a buffer
  double* const xb = kSm ? reinterpret_cast<double*>(smem) : reinterpret_cast<double*>(ws);
  if (kSm) sp += 2 * n * ld;
  double2* Y = ws + 4 * nn;
  int ycap = 2;
  if (!kCg && a.y_smem > 0) {
    Y = sp;
    sp += (int64_t)a.y_smem * nn;
    ycap = a.y_smem;
  }
  double2* v_s = sp;
  sp += a.vcap;
  double2* d_s = sp;
  sp += small ? n : 0;
  double2* lv = sp;
  sp += a.row_cap * n;
  uint32_t* lk = reinterpret_cast<uint32_t*>(sp);
  int* lcnt = reinterpret_cast<int*>(lk + a.row_cap * n);

  // ---- generator rows (driven: the union of the patterns)
  const double* coef = a.drive_coef ? a.drive_coef + (int64_t)a.step0 * a.n_drive : nullptr;
  auto entry = [&](int i, int c) -> double2 {
    double2 v = heff0[(int64_t)i * n + c];
    for (int q = 0; q < a.n_drive; ++q) v = csub(v, cscale(a.drive_ops[q * nn + (int64_t)i * n + c], coef[q]));
    return v;
  };
  auto nz = [&](int i, int c) -> bool {
    double2 v = heff0[(int64_t)i * n + c];
    bool on = v.x != 0.0 || v.y != 0.0;
    for (int q = 0; q < a.n_drive; ++q) {
      v = a.drive_ops[q * nn + (int64_t)i * n + c];
      on |= v.x != 0.0 || v.y != 0.0;
    }
    return on;
  };
  auto im = [&](int i, int c) -> bool {
    bool on = heff0[(int64_t)i * n + c].y != 0.0;
    for (int q = 0; q < a.n_drive; ++q) on |= a.drive_ops[q * nn + (int64_t)i * n + c].y != 0.0;
    return on;
  };
  const Rows R = build_rows(entry, nz, im, n, (int)ld2, v_s, a.vcap, ws + 3 * nn, d_s, &S.rb);

  // ---- collapse operators: those with at most kSparseRow entries a row go
  // into the rows' entry lists (operator, column, value) while they fit, the
  // others run as the two products (L rho) L^dag
  if (t == 0) S.n_dense = 0;
  const int K = a.k_dense;
  const bool lists = a.row_cap > 0 && K <= kMaxFlagOps;
  if (lists) {
    for (int i = t; i < n; i += blockDim.x) lcnt[i] = 0;
    for (int k = 0; k < K; ++k) {
      __syncthreads();
      if (t == 0) S.max_row = 0;
      __syncthreads();
      const double2* L = ldn + k * nn;
      int most = 0;
      for (int i = warp; i < n; i += nwa) {
        int c = 0;
        for (int c0 = 0; c0 < n; c0 += 32) {
          const int cc = c0 + lane;
          const double2 v = cc < n ? L[(int64_t)i * n + cc] : cz();
          c += __popc(__ballot_sync(0xffffffffu, v.x != 0.0 || v.y != 0.0));
        }
        if (c > kSparseRow || c + lcnt[i] > a.row_cap) most = 1;
      }
      if (lane == 0 && most) atomicOr(&S.max_row, 1);
      __syncthreads();
      if (S.max_row) {
        if (t == 0) S.dense_op[S.n_dense++] = k;
      } else {
        for (int i = warp; i < n; i += nwa) {
          int c = lcnt[i];
          for (int c0 = 0; c0 < n; c0 += 32) {
            const int cc = c0 + lane;
            const double2 v = cc < n ? L[(int64_t)i * n + cc] : cz();
            const bool on = v.x != 0.0 || v.y != 0.0;
            const unsigned bal = __ballot_sync(0xffffffffu, on);
            if (on) {
              const int q = c + __popc(bal & ((1u << lane) - 1u));
              lv[q * n + i] = v;
              lk[q * n + i] = ((uint32_t)k << 16) | (uint32_t)cc;
            }
            c += __popc(bal);
          }
          __syncwarp();
          if (lane == 0) lcnt[i] = c;
        }
      }
    }
  }
  __syncthreads();
  const int n_dense = lists ? S.n_dense : K;
  const bool jumps = lists && n_dense < K;
  auto dense_l = [&](int q) { return ldn + (lists ? S.dense_op[q] : q) * nn; };

  // ---- range of the nonzero entries of diagonal observables
  if (a.obs_diag && n <= 32767) {
    for (int o = warp; o < min(a.n_obs, kMaxObs); o += nwa) {
      int lo = n, hi = -1;
      for (int i = lane; i < n; i += 32) {
        const double2 v = obs_ops[(int64_t)o * n + i];
        if (v.x != 0.0 || v.y != 0.0) {
          lo = min(lo, i);
          hi = max(hi, i);
        }
      }
      lo = __reduce_min_sync(0xffffffffu, lo);
      hi = __reduce_max_sync(0xffffffffu, hi);
      if (lane == 0) S.obs_rng[o] = make_short2((short)lo, (short)hi);
    }
  }

  // ---- state: items e0 + q * nt + t, item (i, j) = (e / n, e % n)
  const int64_t per = (nn + C - 1) / C;
  const int64_t e0 = rank * per, e1 = nn < e0 + per ? nn : e0 + per;
  double* acc_g = reinterpret_cast<double*>(ws + 2 * nn);
  double* f_g = acc_g + nn;
  constexpr int kReg = kE > 0 ? kE : 1;
  constexpr bool kRegF = kE == 1 || kE == 2;   // f of the dense operators in registers, else in f_g
  double r_r[kReg], r_a[kReg];
  double2 r_c[kReg];
  uint32_t ij[kReg];
  auto coef_of = [&](const Item& it) {
    return diag_coef(R.d[it.p], R.d[it.q], m ? m[(int64_t)it.p * n + it.q] : cz());
  };
  auto valid = [&](int q) { return !helper && e0 + q * nt + t < e1; };
  auto unpack = [&](uint32_t v) { return item_of((int)(v >> 16), (int)(v & 0xffffu)); };
  auto own_of = [&](double2* z, const Item& it) {
    return reinterpret_cast<double*>(z + (int64_t)it.p * n + it.q) + (it.im ? 1 : 0);
  };
  if (!helper)
    for (int64_t e = t + (int64_t)rank * nt; e < nn; e += (int64_t)C * nt) {
      const int i = (int)(e / n), j = (int)(e - (int64_t)i * n);
      const double2 v = rho[e];
      double* o = xb + (Idx)i * ld2 + 2 * j;
      o[0] = v.x;
      o[1] = v.y;
      if (i == j) o[half + 1] = 0.0;   // no item writes Im rho_ii
    }
  if (kE > 0) {
#pragma unroll
    for (int q = 0; q < kReg; ++q) {
      const int64_t e = e0 + q * nt + t;
      ij[q] = 0;                 // a thread without item q computes item (0, 0) and drops it
      r_c[q] = cz();
      if (!helper && e < e1) {
        const int i = (int)(e / n), j = (int)(e - (int64_t)i * n);
        ij[q] = ((uint32_t)i << 16) | (uint32_t)j;
        const Item it = item_of(i, j);
        r_r[q] = *own_of(rho, it);
        r_c[q] = coef_of(it);
      }
    }
  }
  const bool tracer = rank == 0 && side;
  double tr0 = 0.0;
  if (tracer) {
    if (a.step0 == 0) {
      for (int i = lane; i < n; i += 32) tr0 += rho[(int64_t)i * n + i].x;
      tr0 = warp_sum(tr0);
      if (lane == 0) a.tr0[b] = tr0;
    } else {
      tr0 = a.tr0[b];
    }
  }
  const double tr_tol = a.trace_tol * fmax(1.0, fabs(tr0));
  auto stage_sync = [&]() {
    if (kCg) cluster_sync();
    else __syncthreads();
  };
  stage_sync();

  const double dt = a.dt, dt2 = a.dt / 2.0;
  int flags = 0, cur = 0;
  // trace of the state after the last step: the helper sums its lanes' parts
  // and compares while the workers are a stage further
  bool tr_pending = false;
  double tr_part = 0.0;
  auto check_trace = [&]() {
    if (fabs(warp_sum(tr_part) - tr0) > tr_tol) flags |= LIME_FLAG_TRACE_DRIFT;
    tr_pending = false;
  };
  for (int step = 0; step < a.n_steps; ++step) {
    const int gstep = a.step0 + step;
    if (a.n_drive > 0 && step > 0) {
      // driven generator (lime/oqs.py:1716-1722): Heff(t) = Heff0 - sum_i f_i(t) H_i
      // with f_i evaluated at the end of the step
      coef = a.drive_coef + (int64_t)gstep * a.n_drive;
      refill_rows(R, entry, (int)ld2);
      stage_sync();
      if (kE > 0) {
#pragma unroll
        for (int q = 0; q < kReg; ++q)
          r_c[q] = coef_of(unpack(ij[q]));
      }
    }
    const bool store = a.states && ((gstep + 1) % a.states_every) == 0;
    const int sslot = store ? (gstep + 1) / a.states_every - 1 : 0;
    double2* sdst = store ? a.states + ((int64_t)b * a.states_per_inst + sslot) * nn : nullptr;
    const bool sok = store && in_bounds((((size_t)b * a.states_per_inst + sslot) * nn) * 16, (size_t)nn * 16,
                                        a.states_elems * 16, a.status);
#pragma unroll 1
    for (int s = 0; s < 4; ++s) {
      const double* x = xb + cur * half;
      double* xn = xb + (cur ^ 1) * half;
      if (s == 1 && tr_pending) check_trace();
      // the jump terms of the listed operators
      auto listed = [&](const Item& it, double f) -> double {
        double j = 0.0;
        int u = 0, w = 0;
        const int cu = lcnt[it.p], cw = lcnt[it.q];
        while (u < cu && w < cw) {
          const uint32_t ku = lk[u * n + it.p], kw = lk[w * n + it.q];
          if ((ku >> 16) < (kw >> 16)) ++u;
          else if ((ku >> 16) > (kw >> 16)) ++w;
          else {
            for (int w2 = w; w2 < cw; ++w2) {
              const uint32_t k2 = lk[w2 * n + it.q];
              if ((k2 >> 16) != (ku >> 16)) break;
              const double2 r = ldz<kCg>(
                  reinterpret_cast<const double2*>(x + (Idx)(ku & 0xffffu) * ld2 + 2 * (int)(k2 & 0xffffu)));
              const double2 z = cmul(lv[u * n + it.p], cconj(lv[w2 * n + it.q]));
              j = it.im ? fma(z.x, r.y, fma(z.y, r.x, j)) : fma(z.x, r.x, fma(-z.y, r.y, j));
            }
            ++u;
          }
        }
        return f + j;
      };
      // f of all items (kE > 0) or of one, without the dense operators
      double f_r[kReg];
      auto rhs_all = [&]() {
        Item it[kReg];
#pragma unroll
        for (int q = 0; q < kReg; ++q) it[q] = unpack(ij[q]);
        rhs_items<kReg, kCg, Idx>(R, r_c, x, ld2, it, f_r);
        if (jumps)
#pragma unroll
          for (int q = 0; q < kReg; ++q) f_r[q] = listed(it[q], f_r[q]);
      };
      auto rhs_one = [&](const Item& it) -> double {
        const Item i1[1] = {it};
        const double2 c1[1] = {coef_of(it)};
        double f1[1];
        rhs_items<1, kCg, Idx>(R, c1, x, ld2, i1, f1);
        return jumps ? listed(it, f1[0]) : f1[0];
      };
      // RK4 combination: the item's next stage input
      auto combine = [&](double& r, double& ac, double f) -> double {
        if (s == 0) {
          ac = f;
          return fma(dt2, f, r);
        }
        if (s < 3) {
          ac = fma(2.0, f, ac);
          return fma(s == 2 ? dt : dt2, f, r);
        }
        r = rk4_final_f64(r, ac + f, a.sixth);
        if (!isfinite(r)) flags |= LIME_FLAG_NONFINITE;
        return r;
      };
      auto put = [&](const Item& it, double v) {
        xn[(Idx)it.p * ld2 + 2 * it.q + it.im] = v;
        if (it.p != it.q) xn[(Idx)it.q * ld2 + 2 * it.p + it.im] = it.im ? -v : v;
        if (s == 3 && sok) {
          double* so = reinterpret_cast<double*>(sdst);
          const int64_t su = 2 * ((int64_t)it.p * n + it.q), sl = 2 * ((int64_t)it.q * n + it.p);
          so[su + it.im] = v;
          if (it.p != it.q) so[sl + it.im] = it.im ? -v : v;
          else so[su + 1] = 0.0;
        }
      };
      if (n_dense > 0) {
        if (kE > 0 && !helper) {
          rhs_all();
          if (!kRegF)
#pragma unroll
            for (int q = 0; q < kReg; ++q)
              if (e0 + q * nt + t < e1) f_g[e0 + q * nt + t] = f_r[q];
        }
        for (int k0 = 0; k0 < n_dense; k0 += ycap) {
          const int kb = min(ycap, n_dense - k0);
          // Y_q = L_q rho_s
          const int64_t tot = (int64_t)kb * nn;
          for (int64_t y = helper ? tot : t + (int64_t)rank * nt; y < tot; y += (int64_t)C * nt) {
            const int q = (int)(y / nn);
            const int64_t e = y - q * nn;
            const int i = (int)(e / n), j = (int)(e - (int64_t)i * n);
            const double2* L = dense_l(k0 + q) + (int64_t)i * n;
            double2 s0 = cz();
#pragma unroll 4
            for (int k = 0; k < n; ++k)
              cfma(s0, L[k], ldz<kCg>(reinterpret_cast<const double2*>(x + (Idx)k * ld2 + 2 * j)));
            Y[y] = s0;
          }
          stage_sync();
          // f_pq += sum_q sum_b Y_q[p][b] conj(L_q[q][b]), an operator's sum and
          // theirs by themselves (added term by term to f they have 2.7 times
          // the rounding error)
          auto jump = [&](const Item& it, double f) -> double {
            double all = 0.0;
            for (int q = 0; q < kb; ++q) {
              const double2* L = dense_l(k0 + q) + (int64_t)it.q * n;
              const double2* y = Y + q * nn + (int64_t)it.p * n;
              double j = 0.0;
#pragma unroll 4
              for (int k = 0; k < n; ++k) {
                const double2 yv = ldz<kCg>(y + k), lv2 = L[k];
                j = fma(it.im ? yv.y : yv.x, lv2.x, j);
                j = fma(it.im ? -yv.x : yv.y, lv2.y, j);
              }
              all += j;
            }
            return f + all;
          };
          if (kRegF) {
#pragma unroll
            for (int q = 0; q < kReg; ++q)
              if (valid(q)) f_r[q] = jump(unpack(ij[q]), f_r[q]);
          } else {
            for (int64_t e = helper ? e1 : e0 + t; e < e1; e += nt) {
              const Item it = item_of((int)(e / n), (int)(e % n));
              f_g[e] = jump(it, kE == 0 && k0 == 0 ? rhs_one(it) : f_g[e]);
            }
          }
          if (k0 + ycap < n_dense) stage_sync();   // Y is read before the next operators overwrite it
        }
      }
      if (kE > 0) {
        if (n_dense == 0 && !helper) rhs_all();
#pragma unroll
        for (int q = 0; q < kReg; ++q) {
          if (!valid(q)) continue;
          const double f = (n_dense > 0 && !kRegF) ? f_g[e0 + q * nt + t] : f_r[q];
          put(unpack(ij[q]), combine(r_r[q], r_a[q], f));
        }
      } else {
        for (int64_t e = helper ? e1 : e0 + t; e < e1; e += nt) {
          const Item it = item_of((int)(e / n), (int)(e % n));
          const double f = n_dense > 0 ? f_g[e] : rhs_one(it);
          double* own = own_of(rho, it);
          double r = *own, ac = s > 0 ? acc_g[e] : 0.0;
          const double v = combine(r, ac, f);
          if (s < 3) acc_g[e] = ac;
          else *own = r;
          put(it, v);
        }
      }
      cur ^= 1;
      stage_sync();
    }
    const double* x = xb + cur * half;
    auto elem = [&](int i, int j) { return ldz<kCg>(reinterpret_cast<const double2*>(x + (Idx)i * ld2 + 2 * j)); };
    // observables after the step (the next write to this buffer is behind the next stage's barrier)
    if (a.n_obs > 0 && ((gstep + 1) % a.obs_every) == 0) {
      const int oslot = (gstep + 1) / a.obs_every - 1;
      const size_t base = ((size_t)b * a.obs_per_inst + oslot) * a.n_obs;
      const bool ranged = a.obs_diag && n <= 32767;
      if (ranged && side) {
        // one observable a lane: rho_ii is real
        for (int o = rank * 32 + lane; o < min(a.n_obs, kMaxObs); o += C * 32) {
          const short2 rg = S.obs_rng[o];
          if (rg.y - rg.x >= kNarrow) continue;
          double2 v = cz();
          for (int i = rg.x; i <= rg.y; ++i) {
            const double2 z = obs_ops[(int64_t)o * n + i];
            const double r = elem(i, i).x;
            if (i == rg.x) v = cscale(z, r);
            else v = make_double2(fma(z.x, r, v.x), fma(z.y, r, v.y));
          }
          if (in_bounds((base + o) * 16, 16, a.obs_elems * 16, a.status)) a.obs_out[base + o] = v;
        }
      }
      for (int o = helper ? a.n_obs : rank * nw + warp; o < a.n_obs; o += C * nw) {
        double2 v = cz();
        if (a.obs_diag) {
          if (ranged && o < kMaxObs && S.obs_rng[o].y - S.obs_rng[o].x < kNarrow) continue;
          const double2* E = obs_ops + (int64_t)o * n;
          for (int i = lane; i < n; i += 32) cfma(v, E[i], elem(i, i));
        } else {
          // Tr(E rho) = sum E[j][i] rho[i][j] with rho[i][j] = conj(rho[j][i])
          const double2* E = obs_ops + o * nn;
          for (int j = 0; j < n; ++j)
            for (int i = lane; i < n; i += 32) {
              const double2 z = E[(int64_t)j * n + i];
              if (z.x != 0.0 || z.y != 0.0) cfma(v, z, cconj(elem(j, i)));
            }
        }
        v.x = warp_sum(v.x);
        v.y = warp_sum(v.y);
        if (lane == 0 && in_bounds((base + o) * 16, 16, a.obs_elems * 16, a.status)) a.obs_out[base + o] = v;
      }
    }
    if (tracer && a.trace_tol > 0.0) {
      tr_part = 0.0;
      for (int i = lane; i < n; i += 32) tr_part += elem(i, i).x;
      tr_pending = true;
    }
  }
  if (tr_pending) check_trace();
  // ---- final state (kE = 0 kept the items' own words in place)
  for (int64_t e = helper ? nn : t + (int64_t)rank * nt; e < nn; e += (int64_t)C * nt) {
    const int i = (int)(e / n), j = (int)(e - (int64_t)i * n);
    rho[e] = ldz<kCg>(reinterpret_cast<const double2*>(xb + cur * half + (Idx)i * ld2 + 2 * j));
  }
  if (flags) atomicOr(a.status, flags);
}

// Shared-memory plan and grid of one call.
struct RK4Plan {
  int e, nt, cluster, ld, vcap, row_cap, y_smem;
  size_t smem;
};

constexpr size_t kSmemMax = 227 * 1024 - sizeof(Head) - 1024;

// How a launch with clusters of c CTAs is laid out.
//  - items a thread: the fewest of 1, 2, 4, 8 that 512 threads cover.
//  - shared memory: the stage inputs, the generator's values as full rows if
//    they fit, Y of up to four operators, the entry lists.
static RK4Plan plan_rk4(int n, int c, int k_dense) {
  RK4Plan P{};
  const int64_t nn = (int64_t)n * n;
  P.cluster = c;
  const int64_t per = (nn + P.cluster - 1) / P.cluster;
  const int64_t items = (per + kMaxThreads - 1) / kMaxThreads;
  P.e = items <= 1 ? 1 : items <= 2 ? 2 : items <= 4 ? 4 : items <= 8 ? 8 : 0;
  if (n > 65535 || (P.cluster == 1 && n > 64)) P.e = 0;
  P.nt = P.e == 0 ? kMaxThreads : (int)(((per + P.e - 1) / P.e + 31) / 32 * 32);
  if (k_dense > 0 && P.nt < 128) P.nt = 128;   // threads without an item still form rows of Y
  const bool rs_smem = P.cluster == 1 && P.e > 0;
  P.ld = rs_smem ? (n | 1) : n;      // odd: the transposed stores of a warp spread over the banks
  int64_t left = (int64_t)kSmemMax;
  auto take = [&](int64_t bytes) {
    if (bytes > left) return false;
    left -= bytes;
    return true;
  };
  if (rs_smem) take(2 * (int64_t)n * P.ld * 16);
  if (n <= kRowsSmemMax) {
    take((int64_t)n * 20);           // diagonal, entry counts
    if (k_dense > 0) {
      P.row_cap = (int)(32768 / ((int64_t)n * 20));
      if (P.row_cap > 32) P.row_cap = 32;
      if (!take((int64_t)P.row_cap * n * 20)) P.row_cap = 0;
    }
    // full complex rows, n (n - 1) double2, if they fit
    const int64_t full = (int64_t)n * (n - 1);
    P.vcap = (int)(full * 16 <= left && full <= 8192 ? full : left / 2 / 16 < 8192 ? left / 2 / 16 : 8192);
    take((int64_t)P.vcap * 16);
    while (rs_smem && P.y_smem < 4 && P.y_smem < k_dense && take(nn * 16)) ++P.y_smem;
  }
  P.smem = (size_t)((int64_t)kSmemMax - left);
  return P;
}

// A batch runs as rounds of one CTA an instance while they fill the chip,
// and what is left over (or a batch smaller than the chip) as launches of
// clusters, one round each: kRoom[c] clusters of c CTAs with an SM each fit
// at once (occupancy calculator; 152 SMs).  The split is the cheapest by this
// count of a stage's clocks: 64 an FP64 instruction and warp of the busiest of
// an SM's four partitions, plus the cluster's exchange through L2 (3000
// measured, with the four barriers of dense operators 12000, against 600 for
// a barrier of one CTA) and a launch's share.  Without dense operators the
// entries of a row are not known here; 12 FP64 instructions an item stand for
// a chain, whatever the generator: rows with more entries (2 (n - 1)
// instructions for real long-range couplings, 4 (n - 1) for a complex Heff,
// listed operators) get smaller clusters than their work would pay for.  A
// cluster leaves every CTA at least 512 items (128 with dense operators): below
// that, on a chain, the exchange costs more than it divides.
// Measured against one launch with one cluster size (a power of two, and one
// CTA an instance from 77 on), 37 levels with three dense operators: 170
// instances, 6 steps, 16.1 -> 9.9 ms; 48, 20 steps, 14.3 -> 12.3; 64-site
// chains, 160, 8 steps, 1.22 -> 0.89, 512, 8 steps, 2.20 -> 2.09.
constexpr int kMaxCluster = 8;
constexpr int kRoom[kMaxCluster + 1] = {0, 152, 76, 46, 36, 28, 23, 15, 15};

static double stage_clocks(int n, int c, int k_dense) {
  const RK4Plan P = plan_rk4(n, c, k_dense);
  const int64_t nn = (int64_t)n * n, per = (nn + c - 1) / c, rows = (int64_t)k_dense * nn;
  // instructions of the busiest partition for `work` thread items in rounds of the CTA's threads
  const auto busiest = [&](int64_t work) {
    return (double)(work / P.nt) * ((P.nt / 32 + 3) / 4) + (double)(((work % P.nt + 31) / 32 + 3) / 4);
  };
  const double item = busiest(per), y = busiest((rows + c - 1) / c);
  return 64.0 * (item * (k_dense > 0 ? (4.0 + 2.0 * k_dense) * n : 12.0) + y * 4.0 * n) +
         (c == 1 ? 600.0 : k_dense > 0 ? 12000.0 : 3000.0);
}

struct RK4Part {
  int b0, count, cluster;
};

// parts of a batch, at most kMaxParts
constexpr int kMaxParts = 4;
static int split_batch(int n, int batch, int k_dense, int n_steps, RK4Part* out) {
  const int64_t nn = (int64_t)n * n, least = k_dense > 0 ? 128 : 512;
  double t[kMaxCluster + 1];
  int most = 1;
  for (int c = 1; c <= kMaxCluster && (c == 1 || nn >= c * least); ++c) {
    t[c] = stage_clocks(n, c, k_dense) + 60000.0 / (4.0 * n_steps);
    most = c;
  }
  // best[r]: cheapest rounds for r instances; a remainder of parts parts
  const int room = kRoom[1], rest = batch % room, full = batch - rest;
  double best[kMaxParts + 1][kRoom[1] + 1];
  int pick[kMaxParts + 1][kRoom[1] + 1];
  for (int k = 0; k <= kMaxParts; ++k)
    for (int r = 0; r <= rest; ++r) {
      best[k][r] = r == 0 ? 0.0 : 1e300;
      pick[k][r] = 0;
      if (k > 0 && r > 0)
        for (int c = 1; c <= most; ++c) {
          const double v = t[c] + best[k - 1][r > kRoom[c] ? r - kRoom[c] : 0];
          if (v < best[k][r]) {
            best[k][r] = v;
            pick[k][r] = c;
          }
        }
    }
  // one launch for the remainder, unless several are a tenth cheaper
  int one = 1;
  for (int c = 2; c <= most; ++c)
    if (rest <= kRoom[c] && t[c] < t[one]) one = c;
  const bool several = best[kMaxParts - 1][rest] * 1.1 < t[one];
  if (rest == 0 || (!several && one == 1)) {   // whole rounds, or a last one that clusters do not shorten
    out[0] = {0, batch, 1};
    return 1;
  }
  int parts = 0, b = 0, r = rest;
  if (full > 0) {
    out[parts++] = {0, full, 1};
    b = full;
  }
  for (int k = kMaxParts - 1; r > 0; --k) {
    const int c = several ? pick[k][r] : one, m = r < kRoom[c] ? r : kRoom[c];
    out[parts++] = {b, m, c};
    b += m;
    r -= m;
  }
  return parts;
}

template <int kE, bool kCg>
static int launch_rk4(const RK4Args& a, const RK4Plan& P, int batch, cudaStream_t st) {
  auto kern = lindblad_rk4_f64_kernel<kE, kCg>;
  // (one value for every shape: calls of other threads set the same attribute)
  LIME_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)((int64_t)batch * P.cluster));
  cfg.blockDim = dim3(P.nt + (kE == 1 ? 32 : 0));
  cfg.dynamicSmemBytes = P.smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = P.cluster;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = kCg ? 1 : 0;
  LIME_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, a));
  LIME_CUDA_TRY(cudaGetLastError());
  count_launch();
  return LIME_OK;
}

}  // namespace f64
}  // namespace lime

using namespace lime;

extern "C" size_t lime_lindblad_rk4_f64_workspace(int32_t n, int32_t batch, int32_t k_dense) {
  if (n <= 0 || batch <= 0 || k_dense < 0) return 0;
  const size_t mats = (size_t)f64::ws_mats(k_dense) * (size_t)n * n * sizeof(double2);
  return (size_t)batch * (mats + sizeof(double));
}

extern "C" int lime_lindblad_rk4_f64(const LimeLindbladDesc* d, void* stream) {
  if (!d) return LIME_ERR_ARG;
  if (d->n <= 0 || d->batch <= 0 || d->n_steps < 0 || d->k_dense < 0 || d->n_obs < 0) return LIME_ERR_ARG;
  if (!d->rho || !d->heff || !d->status || !d->workspace) return LIME_ERR_ARG;
  if (d->k_dense > 0 && !d->l_dense) return LIME_ERR_ARG;
  if (d->n_obs > 0 && (!d->obs_ops || !d->obs_out)) return LIME_ERR_ARG;
  if (d->states && d->states_every <= 0) return LIME_ERR_ARG;
  if (d->heff_stride < 0 || d->m_stride < 0 || d->l_dense_stride < 0 || d->obs_stride < 0) return LIME_ERR_ARG;
  const int pb = d->param_batch > 0 ? d->param_batch : d->batch;
  if (pb > d->batch) return LIME_ERR_ARG;
  if (!(d->dt == d->dt)) return LIME_ERR_ARG;
  if (d->n_drive < 0 || (d->n_drive > 0 && (!d->drive_ops || !d->drive_coef))) return LIME_ERR_ARG;
  if (d->workspace_bytes < lime_lindblad_rk4_f64_workspace(d->n, d->batch, d->k_dense))
    return LIME_ERR_WORKSPACE;
  if (d->n_steps == 0) return LIME_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t nn = (int64_t)d->n * d->n;
  f64::RK4Args a{};
  a.n = d->n; a.param_batch = pb; a.k_dense = d->k_dense; a.n_obs = d->n_obs; a.obs_diag = d->obs_diag;
  a.states_every = d->states ? d->states_every : 1;
  a.states_per_inst = d->states ? d->n_steps / d->states_every : 0;
  a.dt = d->dt; a.sixth = sixth_of(d->dt); a.trace_tol = d->trace_tol;
  a.rho = reinterpret_cast<double2*>(d->rho);
  a.heff = reinterpret_cast<const double2*>(d->heff); a.heff_stride = d->heff_stride;
  a.m = reinterpret_cast<const double2*>(d->m); a.m_stride = d->m_stride;
  a.l_dense = reinterpret_cast<const double2*>(d->l_dense); a.l_dense_stride = d->l_dense_stride;
  a.obs_ops = reinterpret_cast<const double2*>(d->obs_ops); a.obs_stride = d->obs_stride;
  a.obs_out = reinterpret_cast<double2*>(d->obs_out);
  a.obs_every = d->obs_every > 0 ? d->obs_every : 1;
  a.obs_per_inst = d->n_steps / a.obs_every;
  a.states = reinterpret_cast<double2*>(d->states);
  a.obs_elems = (size_t)d->batch * a.obs_per_inst * (d->n_obs > 0 ? d->n_obs : 0);
  a.states_elems = (size_t)d->batch * a.states_per_inst * nn;
  a.ws = reinterpret_cast<double2*>(d->workspace);
  a.tr0 = reinterpret_cast<double*>(reinterpret_cast<char*>(d->workspace) +
                                    (size_t)d->batch * f64::ws_mats(d->k_dense) * nn * sizeof(double2));
  a.status = d->status;
  a.n_drive = d->n_drive;
  a.drive_ops = reinterpret_cast<const double2*>(d->drive_ops);
  a.drive_coef = d->drive_coef;
  // bounded launches: at most ~2^27 complex MACs of GEMM per instance per launch
  const double per_step = 4.0 * (1 + 2 * d->k_dense) * (double)nn * d->n;
  int chunk = (int)fmax(1.0, fmin((double)d->n_steps, 134217728.0 / per_step));
  f64::RK4Part part[f64::kMaxParts];
  const int parts = f64::split_batch(d->n, d->batch, d->k_dense, d->n_steps, part);
  for (int i = 0; i < parts; ++i) {
    const f64::RK4Plan P = f64::plan_rk4(d->n, part[i].cluster, d->k_dense);
    const int64_t skip = part[i].b0 - a.b0;
    a.b0 = part[i].b0;
    a.rho += skip * nn;
    a.ws += skip * f64::ws_mats(d->k_dense) * nn;
    a.tr0 += skip;
    if (a.obs_out) a.obs_out += skip * a.obs_per_inst * a.n_obs;
    if (a.states) a.states += skip * a.states_per_inst * nn;
    a.obs_elems -= (size_t)skip * a.obs_per_inst * a.n_obs;
    a.states_elems -= (size_t)skip * a.states_per_inst * nn;
    a.cluster = P.cluster; a.ld = P.ld; a.vcap = P.vcap; a.row_cap = P.row_cap; a.y_smem = P.y_smem;
    const auto run = P.cluster > 1 ? (P.e == 1   ? f64::launch_rk4<1, true>
                                      : P.e == 2 ? f64::launch_rk4<2, true>
                                      : P.e == 4 ? f64::launch_rk4<4, true>
                                      : P.e == 8 ? f64::launch_rk4<8, true>
                                                 : f64::launch_rk4<0, true>)
                                   : (P.e == 1   ? f64::launch_rk4<1, false>
                                      : P.e == 2 ? f64::launch_rk4<2, false>
                                      : P.e == 4 ? f64::launch_rk4<4, false>
                                      : P.e == 8 ? f64::launch_rk4<8, false>
                                                 : f64::launch_rk4<0, false>);
    for (int s0 = 0; s0 < d->n_steps; s0 += chunk) {
      a.step0 = s0;
      a.n_steps = (d->n_steps - s0 < chunk) ? d->n_steps - s0 : chunk;
      LIME_TRY(run(a, P, part[i].count, st));
    }
  }
  return LIME_OK;
}
