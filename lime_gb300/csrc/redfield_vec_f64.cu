// FP64 RK4 on vec(rho) under a dense generator for a few right-hand sides
// (lime/oqs.py:373-472, whose loop is one matrix-vector product a stage).
//
// One launch runs the time loop.  The 2 D R real numbers of the state are the
// outputs; a CTA owns a contiguous range of them, keeps its rows of the
// generator in shared memory (while they fit) and the stage input of all
// rows, and a team of threads shares the dot product of each output, so that
// all four FP64 partitions of the SM work whatever the number of rows.  The
// stage inputs are exchanged
//   kSolo     in the shared memory of one CTA,
//   kCluster  by stores into the shared memory of 8 CTAs and their barrier,
//   kGrid     through L2 between all SMs: an output travels as one 16-byte
//             word {value, stage number}, so the reader polls the data itself
//             and no fence or barrier stands between writer and reader.  The
//             launch is cooperative (all CTAs resident), the polls are
//             bounded.  A CTA whose wait runs out raises LIME_FLAG_TIMEOUT
//             and leaves NaN in its part of the state and of every state
//             that the launch should still have kept.
// Two buffers suffice: a CTA writes the input of stage s + 2 only after it
// has read all of stage s + 1, which its owners wrote after reading all of s.
//
// Bound: 4 D^2 R DFMA a stage at 1.68 lanes per clock and SM, and the latency
// of the exchange.  Measured against one 64 x 64 tiled GEMM launch a stage
// (one CTA per 64 rows, 63 of 64 columns padding), one right-hand side: D =
// 400 (kGrid) 1632 -> 3.7 us a stage, of which the DFMA are 1.3; D = 36
// (kCluster) 198 -> 2.0 us.

#include "redfield_vec_f64.cuh"

#include <math.h>

namespace lime {
namespace rfv {

struct Args {
  int D, R, F, outs, team, red, l_smem, cluster;
  int step0, n_steps, states_every, obs_every;
  double dt;
  Sixth sixth;
  const double2* L;
  double2* P;
  ulonglong2* xch;       // [2][F]
  double2* states;
  double2* hist;
  int32_t* status;
  uint32_t max_wait;
};

__device__ __forceinline__ ulonglong2 ld_tagged(const ulonglong2* p) {
  ulonglong2 v;
  asm volatile("{\n\t.reg .b128 r;\n\tld.relaxed.gpu.global.b128 r, [%2];\n\tmov.b128 {%0, %1}, r;\n\t}"
               : "=l"(v.x), "=l"(v.y)
               : "l"(p)
               : "memory");
  return v;
}
__device__ __forceinline__ void st_tagged(ulonglong2* p, double value, unsigned long long tag) {
  asm volatile("{\n\t.reg .b128 r;\n\tmov.b128 r, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], r;\n\t}" ::"l"(p),
               "l"(__double_as_longlong(value)), "l"(tag)
               : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void st_peer(double* local, int peer, double v) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(local);
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(peer));
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(r), "d"(v) : "memory");
}
__device__ __forceinline__ double flip(double x, int mask) {
  return __hiloint2double(__double2hiint(x) ^ mask, __double2loint(x));
}

constexpr int kPoll = 4;   // words a thread has in flight

template <int kMode>
__global__ void __launch_bounds__(kThreads, 1) rk4_kernel(Args a) {
  extern __shared__ __align__(16) double sm[];
  __shared__ int expired;
  const int t = threadIdx.x, D = a.D, R = a.R, F = a.F, T = a.team, g = a.red;
  const int f0 = blockIdx.x * a.outs, O = min(a.outs, F - f0) > 0 ? min(a.outs, F - f0) : 0;
  const int row0 = f0 / (2 * R), rows = O > 0 ? (f0 + O - 1) / (2 * R) - row0 + 1 : 0;
  constexpr int kBuf = kMode == kCluster ? 2 : 1;

  // ---- shared memory: stage inputs [buffer][r][2 D], partial sums, the outputs' values and accumulators, rows
  double* xs = sm;
  double* part = xs + (size_t)kBuf * F;
  double* val = part + (max(kThreads, a.outs) + 1) / 2 * 2;   // rows stay 16-byte aligned
  double* acc = val + a.outs;
  double2* Ls = reinterpret_cast<double2*>(acc + a.outs);
  const double2* L = a.L + (int64_t)row0 * D;
  if (a.l_smem) {
    for (int e = t; e < rows * D; e += kThreads) Ls[e] = L[e];
    L = Ls;
  }
  const double* P = reinterpret_cast<const double*>(a.P);
  // place of flat number f = (k R + r) 2 + c in xs: [r][2 k + c]
  auto at = [&](int f) { return R == 1 ? f : ((f >> 1) % R) * 2 * D + (f / (2 * R)) * 2 + (f & 1); };
  for (int f = t; f < F; f += kThreads) xs[at(f)] = P[f];
  for (int j = t; j < O; j += kThreads) {
    val[j] = P[f0 + j];
    acc[j] = 0.0;
  }
  if (t == 0) expired = 0;
  if (kMode == kCluster) cluster_sync();   // peers are running before the first remote store
  __syncthreads();

  const double dt = a.dt, dt2 = a.dt / 2.0;
  unsigned long long tag = (unsigned long long)a.step0 * 4u;   // of the input of the current stage
  int cur = 0;
  for (int step = 0; step < a.n_steps; ++step) {
    const int done = a.step0 + step + 1;
    const bool store = a.states != nullptr && done % a.states_every == 0;
    const bool keep = a.hist != nullptr && done % a.obs_every == 0;
    double* so = store ? reinterpret_cast<double*>(a.states) + (int64_t)(done / a.states_every - 1) * F : nullptr;
    double* ho = keep ? reinterpret_cast<double*>(a.hist) +
                            (int64_t)(done / a.obs_every - 1 - a.step0 / a.obs_every) * F
                      : nullptr;
#pragma unroll 1
    for (int s = 0; s < 4; ++s) {
      if (kMode == kGrid && (step > 0 || s > 0)) {
        const ulonglong2* src = a.xch + (size_t)(tag & 1) * F;
        for (int b = t; b < F; b += kThreads * kPoll) {
          ulonglong2 v[kPoll];
          uint32_t tries = 0;
          bool all;
          do {
            all = true;
#pragma unroll
            for (int u = 0; u < kPoll; ++u)
              if (b + u * kThreads < F) v[u] = ld_tagged(src + b + u * kThreads);
#pragma unroll
            for (int u = 0; u < kPoll; ++u)
              if (b + u * kThreads < F) all &= v[u].y == tag;
          } while (!all && ++tries < a.max_wait);
          if (!all) {
            expired = 1;
            break;
          }
#pragma unroll
          for (int u = 0; u < kPoll; ++u)
            if (b + u * kThreads < F) xs[at(b + u * kThreads)] = __longlong_as_double((long long)v[u].x);
        }
        __syncthreads();
        if (expired) {
          const double nan = __longlong_as_double(0x7ff8000000000000LL);
          if (t == 0 && a.status != nullptr) atomicOr(a.status, LIME_FLAG_TIMEOUT);
          for (int j = t; j < O; j += kThreads) {
            reinterpret_cast<double*>(a.P)[f0 + j] = nan;
            for (int k = done; k <= a.step0 + a.n_steps; ++k) {
              if (a.states != nullptr && k % a.states_every == 0)
                reinterpret_cast<double*>(a.states)[(int64_t)(k / a.states_every - 1) * F + f0 + j] = nan;
              if (a.hist != nullptr && k % a.obs_every == 0)
                reinterpret_cast<double*>(a.hist)[(int64_t)(k / a.obs_every - 1 - a.step0 / a.obs_every) * F + f0 + j] =
                    nan;
            }
          }
          return;
        }
      }
      const double* x = xs + (kMode == kCluster ? (size_t)cur * F : 0);
      // ---- partial dot products
      for (int j0 = 0; j0 < O; j0 += kThreads / T) {
        const int j = j0 + t / T, l = t % T;
        if (t < kThreads / T * T && j < O) {
          const int f = f0 + j, row = f / (2 * R), r = (f >> 1) % R, c = f & 1;
          const double2* lr = L + (int64_t)(row - row0) * D;
          const double* xr = x + (size_t)r * 2 * D;
          const int neg = c ? 0 : (int)0x80000000;
          double sum = 0.0;
#pragma unroll 4
          for (int k = l; k < D; k += T) {
            const double2 h = lr[k];
            sum = fma(h.x, xr[2 * k + c], sum);
            sum = fma(h.y, flip(xr[2 * k + 1 - c], neg), sum);
          }
          part[j * T + l] = sum;
        }
      }
      __syncthreads();
      ++tag;
      // ---- sums, RK4 combination, next stage input
      for (int j0 = 0; j0 < O; j0 += kThreads / g) {
        const int j = j0 + t / g, i = t % g;
        const bool on = j < O;
        double f = 0.0;
        if (on) {
          f = part[j * T + i];
          for (int q = i + g; q < T; q += g) f += part[j * T + q];
        }
        for (int o = g >> 1; o > 0; o >>= 1) f += __shfl_xor_sync(0xffffffffu, f, o);
        double nx = 0.0, p = 0.0, ac = 0.0;
        if (on) {
          p = val[j];
          ac = acc[j];
          if (s == 0) {
            ac = f;
            nx = fma(dt2, f, p);
          } else if (s < 3) {
            ac = fma(2.0, f, ac);
            nx = fma(s == 2 ? dt : dt2, f, p);
          } else {
            nx = rk4_final_f64(p, ac + f, a.sixth);
          }
        }
        __syncwarp();
        if (on) {
          if (i == 0) {
            if (s == 3) val[j] = nx;
            else acc[j] = ac;
          }
          if (kMode == kCluster) {
            for (int q = i; q < a.cluster; q += g) st_peer(xs + (size_t)(cur ^ 1) * F + at(f0 + j), q, nx);
          } else if (i == 0) {
            if (kMode == kGrid) st_tagged(a.xch + (size_t)(tag & 1) * F + f0 + j, nx, tag);
            else xs[at(f0 + j)] = nx;
          }
          if (s == 3 && i == 0) {
            if (so) so[f0 + j] = nx;
            if (ho) ho[f0 + j] = nx;
          }
        }
      }
      cur ^= 1;
      if (kMode == kCluster) cluster_sync();
      if (kMode == kSolo) __syncthreads();
    }
  }
  __syncthreads();
  for (int j = t; j < O; j += kThreads) reinterpret_cast<double*>(a.P)[f0 + j] = val[j];
}

constexpr size_t kSmemMax = 226 * 1024;

// A stage's clocks in each mode: FP64 work over the CTAs plus a fixed part
// (reduction, barriers, exchange), the fixed parts as measured.
constexpr double kSoloCost = 900, kClusterCost = 1700, kGridCost = 3600;

static bool plan_mode(int D, int R, Mode mode, int ctas, Plan* P) {
  const int F = 2 * D * R;
  P->mode = mode;
  P->outs = (F + ctas - 1) / ctas;
  P->ctas = mode == kCluster ? ctas : (F + P->outs - 1) / P->outs;
  int T = P->outs >= kThreads ? 1 : kThreads / P->outs;
  if (T > D) T = D;
  T = (D + (D + T - 1) / T - 1) / ((D + T - 1) / T);   // the fewest threads with as many terms each
  P->team = T;
  int g = 1;
  while (g < 16 && 2 * g <= T && 2 * g * P->outs <= kThreads) g <<= 1;
  P->red = g;
  const int parts = ((P->outs > kThreads ? P->outs : kThreads) + 1) / 2 * 2;
  const size_t base = ((size_t)(mode == kCluster ? 2 : 1) * F + parts + 2 * (size_t)P->outs) * 8;
  const size_t rows = (size_t)(P->outs + 2 * R - 2) / (2 * R) + 1;
  const size_t lb = rows * D * 16;
  if (base > kSmemMax) return false;
  P->l_smem = base + lb <= kSmemMax;
  P->smem = base + (P->l_smem ? lb : 0);
  return true;
}

bool supported(int D, int R) { return R >= 1 && R <= kMaxRhs && (int64_t)D * R <= 12800; }

bool plan(int D, int R, int sms, Plan* out) {
  if (!supported(D, R)) return false;
  const double work = 4.0 * (double)D * D * R / 1.68;
  const double solo = work + kSoloCost, cluster = work / kMaxCluster + kClusterCost, grid = work / sms + kGridCost;
  const Mode m = solo <= cluster && solo <= grid ? kSolo : cluster <= grid ? kCluster : kGrid;
  out->clocks = m == kSolo ? solo : m == kCluster ? cluster : grid;
  return plan_mode(D, R, m, m == kSolo ? 1 : m == kCluster ? kMaxCluster : sms, out);
}

size_t workspace(int D, int R) {
  const size_t dr = (size_t)D * R * 16;
  return 4 * dr + kHistory * dr;
}

int begin(const Plan& p, const Run& r, cudaStream_t st) {
  if (p.mode != kGrid) return LIME_OK;
  LIME_CUDA_TRY(cudaMemsetAsync(r.ws, 0, (size_t)4 * r.D * r.R * 16, st));
  return LIME_OK;
}

template <int kMode>
static int launch_mode(const Plan& p, const Args& a, cudaStream_t st) {
  auto kern = rk4_kernel<kMode>;
  // (one value for every shape: calls of other threads set the same attribute)
  LIME_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)p.ctas);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  if (kMode == kCluster) {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = p.ctas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  } else {
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
  }
  cfg.attrs = at;
  cfg.numAttrs = kMode == kSolo ? 0 : 1;
  LIME_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, a));
  LIME_CUDA_TRY(cudaGetLastError());
  count_launch();
  return LIME_OK;
}

int launch(const Plan& p, const Run& r, int step0, int steps, double2* hist, cudaStream_t st) {
  Args a{};
  a.D = r.D; a.R = r.R; a.F = 2 * r.D * r.R;
  a.outs = p.outs; a.team = p.team; a.red = p.red; a.l_smem = p.l_smem; a.cluster = p.ctas;
  a.step0 = step0; a.n_steps = steps;
  a.states = r.states; a.states_every = r.states_every > 0 ? r.states_every : 1;
  a.hist = hist; a.obs_every = r.obs_every > 0 ? r.obs_every : 1;
  a.dt = r.dt; a.sixth = sixth_of(r.dt); a.L = r.L; a.P = r.P;
  a.xch = reinterpret_cast<ulonglong2*>(r.ws);
  a.status = r.status; a.max_wait = r.max_wait;
  return p.mode == kSolo ? launch_mode<kSolo>(p, a, st)
                         : p.mode == kCluster ? launch_mode<kCluster>(p, a, st) : launch_mode<kGrid>(p, a, st);
}

}  // namespace rfv
}  // namespace lime
