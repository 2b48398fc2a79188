// FP64 RK4 of a few right-hand sides under a dense generator: the whole time
// loop in one launch (redfield_vec_f64.cu).
#pragma once

#include "common.cuh"

namespace lime {
namespace rfv {

enum Mode { kSolo = 0, kCluster = 1, kGrid = 2 };
constexpr int kThreads = 256;
constexpr int kMaxCluster = 8;
constexpr int kMaxRhs = 8;
constexpr int kHistory = 32;   // states kept in the workspace for the observables of one launch

struct Plan {
  Mode mode;
  int ctas;       // of the launch
  int outs;       // real outputs of a CTA (the last one may have fewer)
  int team;       // threads that share an output's dot product
  int red;        // lanes that add a team's partial sums
  int l_smem;     // the CTA's rows of the generator are kept in shared memory
  size_t smem;
  double clocks;  // of a stage, predicted
};

// shapes whose stage input fits the shared memory of an SM beside the rest
bool supported(int D, int R);
// false: the shape is left to the tiled GEMM per stage
bool plan(int D, int R, int sms, Plan* out);
// bytes behind the 3 D R complex of the tiled path: exchange and history
size_t workspace(int D, int R);

struct Run {
  int D, R, n_steps;
  double dt;
  const double2* L;
  double2* P;            // D x R, in and out
  void* ws;              // workspace(D, R) bytes, 16-byte aligned
  double2* states; int states_every;
  // observables: every obs_every steps hist holds the state (the caller evaluates them per chunk)
  int obs_every;         // 0: none
  int32_t* status;       // LIME_FLAG_TIMEOUT when a wait runs out, or null
  uint32_t max_wait;     // polls of a wait
};
constexpr uint32_t kPollLimit = 1u << 21;   // about two seconds

// runs steps [step0, step0 + steps); hist: slots of D x R, the first one for
// the first multiple of obs_every after step0
int launch(const Plan& p, const Run& r, int step0, int steps, double2* hist, cudaStream_t st);
// clears the exchange buffer of a call (before its first launch)
int begin(const Plan& p, const Run& r, cudaStream_t st);
inline double2* history(const Run& r) {
  return reinterpret_cast<double2*>(reinterpret_cast<char*>(r.ws) + (size_t)4 * r.D * r.R * 16);
}

}  // namespace rfv
}  // namespace lime
