// Per-grid-point convergence state and the step update shared by the step kernels.
#pragma once

#include "pkde_internal.cuh"

namespace pkde {

// Convergence state of every grid point (DensityState, GradeProEstimator.jl:515-615),
// plus the outputs: density, selected step, and the last step's means.
struct StepState {
  double *f1, *f2, *minima, *density, *mu_last;
  uint16_t *c_low, *c_over;
  uint8_t *flags;
  int32_t *selected;
};

struct StabilityResult {
  bool more_stable;
  double new_min;
  uint16_t c_low, c_over;
  uint8_t flag;
};

// The logarithms of the first and second differences of f (DirectSpace.jl:1092-1100), in
// FP64.  Explicit-rounding intrinsics keep the operation order of the reference.
__device__ __forceinline__ void log_differences(double f, double f1, double f2, double dlogt, double &d1, double &d2) {
  d1 = log(fabs(__ddiv_rn(__dsub_rn(f, f1), __dmul_rn(2.0, dlogt))));
  d2 = log(fabs(__ddiv_rn(__dadd_rn(__dsub_rn(f, __dmul_rn(2.0, f1)), f2), __dmul_rn(dlogt, dlogt))));
}

// find_stability (DirectSpace.jl:975-1031) from those logarithms.
__device__ __forceinline__ StabilityResult decide_stability(double d1, double d2, double eps, int64_t steps_low,
                                                            int64_t steps_over, double minimum, uint16_t c_low,
                                                            uint16_t c_over, uint8_t flag) {
  StabilityResult r{false, nan(""), c_low, c_over, flag};
  if (!flag) {
    if (d2 < eps) {
      if (((d1 < minimum) || isnan(minimum)) && ((int64_t)c_over <= steps_over)) {
        r.more_stable = true;
        r.new_min = d1;
        r.c_over = 0;
      } else {
        r.c_over = (uint16_t)(c_over + 1);
      }
    } else {
      r.c_low = (uint16_t)(c_low + 1);
      if ((int64_t)r.c_low > steps_low) {
        r.flag = 1;
        minimum = nan("");
      }
    }
  } else {
    if ((d2 < eps) && isnan(minimum)) {
      r.more_stable = true;
      r.new_min = d1;
    }
  }
  if (isnan(r.new_min)) r.new_min = minimum;
  return r;
}

__device__ __forceinline__ StabilityResult find_stability(double f, double f1, double f2, double dlogt, double eps,
                                                          int64_t steps_low, int64_t steps_over, double minimum,
                                                          uint16_t c_low, uint16_t c_over, uint8_t flag) {
  double d1, d2;
  log_differences(f, f1, f2, dlogt, d1, d2);
  return decide_stability(d1, d2, eps, steps_low, steps_over, minimum, c_low, c_over, flag);
}

// One step of update_state! (GradeProEstimator.jl:638-669) at grid point i:
// v = scaled bootstrap variance of the VMR (DirectSpace.jl:579), mu = the means.
// CG = true: the state was written by other CTAs of the same kernel, so it is read
// through L2 (ld.global.cg) and never from a possibly stale L1 line.
template <class T, bool CG>
__device__ __forceinline__ T ld_state(const T *p) {
  if constexpr (CG) return __ldcg(p);
  return *p;
}
template <bool CG = false>
__device__ __forceinline__ void step_update(const StepState &cs, int64_t i, double mu, double v, double dlogt,
                                            double eps, int64_t steps_low, int64_t steps_over, int step) {
  const double f = isfinite(v) ? log(v) : nan("");
  const double f1 = ld_state<double, CG>(cs.f1 + i), f2 = ld_state<double, CG>(cs.f2 + i);
  const uint16_t cl = ld_state<unsigned short, CG>(reinterpret_cast<const unsigned short *>(cs.c_low + i));
  const uint16_t co = ld_state<unsigned short, CG>(reinterpret_cast<const unsigned short *>(cs.c_over + i));
  const uint8_t fl = (uint8_t)ld_state<unsigned char, CG>(reinterpret_cast<const unsigned char *>(cs.flags + i));
  StabilityResult r =
      find_stability(f, f1, f2, dlogt, eps, steps_low, steps_over, ld_state<double, CG>(cs.minima + i), cl, co, fl);
  cs.c_low[i] = r.c_low;
  cs.c_over[i] = r.c_over;
  cs.flags[i] = r.flag;
  cs.minima[i] = r.new_min;
  if (r.more_stable) {
    cs.density[i] = mu;
    cs.selected[i] = step;
  }
  cs.f2[i] = f1;
  cs.f1[i] = f;
  cs.mu_last[i] = mu;
}

// persistent step engine (pkde_engine.cu)
struct EngineArgs {
  const pkde_grid *grid;
  int npairs, nboot, S;
  const double2 *spectra;
  const double *fz, *fw;  // per-step factor tables [S][tab_stride], axis j at aoff[j]
  int64_t tab_stride;
  int64_t aoff[4];
  const double *cw, *vscale, *dlogt;  // host arrays of S values
  double inv_n, eps;
  int64_t steps_low, steps_over;
  StepState cs;
  // schedule parameters (0: default): ring-slot MB, tiles per axis-pass item, pipeline
  // delay between the passes of a batch
  int tune_slot_mb = 0, tune_tpi = 0, tune_delay = 0, tune_qextra = 0;
};
bool engine_ok(const pkde_grid *g);
// Every axis on the register power-of-two tiles (the engine's lean instantiation).
bool engine_register_only(const pkde_grid *g);
// Per-shape schedule parameters: from the context's cache, else (autotuning on) timed
// trial runs of the estimation's first bandwidth steps.  Overwrites the estimation's
// convergence state (the caller initialises it afterwards).
void autotune_engine(pkde_ctx *ctx, EngineArgs &args, cudaStream_t st);
void run_engine(pkde_ctx *ctx, const EngineArgs &args, cudaStream_t st);
// The error flags of the engine launches queued since the last check: call after the stream
// has synchronised; throws if a launch gave up on a dependency wait.
void check_engine_flags(pkde_ctx *ctx);
// Device bytes of the estimation's ring slots under its schedule parameters.
size_t engine_ring_bytes(const EngineArgs &args);
// Ring slots of at most this size are always allowed; wider ones only within a memory budget.
constexpr int kNarrowSlotMB = 64;
// Several estimations in one persistent launch (their EngineArgs are independent).
void run_engine_batch(pkde_ctx *ctx, const EngineArgs *args, int count, cudaStream_t st);

// How the step engine transforms an axis (its arithmetic): register power-of-two tiles, N = R M
// mixed-radix tiles (R = 3 or 5), or plain Stockham stages (R = 1, pow2 false).
struct EngineAxis {
  bool ok, pow2;
  int R;
};
EngineAxis engine_axis(const pkde_grid *g, int j);
// Combine twiddles of N = R M: (cos, sin)(2 pi n1 k2 / N) as [n1 - 1][k2].
const double2 *combine_twiddles_device(pkde_ctx *ctx, int R, int M, cudaStream_t st);

// Bandwidth steps of N-D estimations in chunks of steps (pkde_chunk.cu).
struct ChunkArgs {
  const pkde_grid *grid;
  int npairs, nboot, S;
  int level;  // of the scratch
  const double2 *spectra;
  const double *fz, *fw;
  int64_t tab_stride;
  int64_t aoff[4];
  const double *cw, *vscale, *dlogt;  // device arrays of S values
  double inv_n, eps;
  int64_t steps_low, steps_over;
  StepState cs;
};
bool chunk_ok(const pkde_grid *g);
// Names an estimation's shape in the schedule file as one that runs in chunks.
void record_chunked(pkde_ctx *ctx, const pkde_grid *g, int npairs);
// Scratch at a memory level (0: the largest chunks .. kChunkLevels - 1).  Serving lanes, and contexts
// that leave the choice of buffer sizes to fixed defaults (pkde_set_autotune), start at kServeLevel;
// PKDE_RING_BUDGET_MB lowers to kCapLevel at most, whose scratch is always allowed, as the engine's ring of
// eight slots of kNarrowSlotMB is (512 x 512, 64 bootstraps, 200 steps: 53 ms within 256 MB, 62 within
// 64 MB, 61 in the engine with those slots).
constexpr int kChunkLevels = 5, kServeLevel = 3, kCapLevel = 3;
size_t chunk_scratch_bytes(const pkde_grid *g, int npairs, int S, int level);
// Whether density and selected step come out final (else the caller initialises the state
// before and fills the points without a selected step after).
bool chunk_keeps_all(const pkde_grid *g, int npairs, int S, int level);
void run_chunk(pkde_ctx *ctx, const ChunkArgs *args, int count, char *const *scratch, cudaStream_t st);

// Bandwidth steps of 1-D estimations (pkde_steps1d.cu).  f_out and mu_out: S x n1, each
// step's log scaled variance and means; cw and vscale: device arrays of S values.
struct Steps1dArgs {
  int n1, npairs, nboot, S;
  int fused;  // 1: the step engine's power-of-two arithmetic, 0: every VMR operation rounded by itself
  int64_t n;
  const double2 *spectra;
  const double *fz, *fw;
  int64_t tab_stride;
  const double *cw, *vscale;
  double *f_out, *mu_out;
  double2 *state;  // steps1d_state_bytes
};
bool steps1d_ok(const pkde_grid *g);
size_t steps1d_job_bytes();
size_t steps1d_state_bytes(int n1, int npairs, int64_t S);
// Descriptors (count x steps1d_job_bytes()) and launches of several estimations.
struct Steps1dPlan {
  static constexpr int kClasses = 7;  // kernels
  int first[kClasses + 1], S[kClasses];
  size_t smem[kClasses];
  struct Len {
    int n, first, count, S;
  };
  std::vector<Len> len;  // the jobs of the last class by length
};
void steps1d_describe(pkde_ctx *ctx, const Steps1dArgs *args, int count, void *host_jobs, Steps1dPlan &plan,
                      cudaStream_t st);
void steps1d_run(pkde_ctx *ctx, const Steps1dPlan &plan, const void *dev_jobs, cudaStream_t st);
// The convergence state machine over all steps (density and selected step of every point).
struct ConvergeJob {
  int64_t G, steps_low, steps_over;
  const double *f, *mu, *dlogt;  // f and means of every step, S x G
  double eps;
  int S;
  StepState cs;
};
void converge_steps(pkde_ctx *ctx, const std::vector<ConvergeJob> &jobs, cudaStream_t st);

// power-of-two path (pkde_step.cu)
bool pow2_path_ok(const pkde_grid *g);
void axis_pass_pow2(pkde_ctx *ctx, const LineSet &ls, const double2 *in, double2 *out, const double *const *factors,
                    const double *scal, int nfac, cudaStream_t st);
void vmr_pass_pow2(pkde_ctx *ctx, int n1, const double2 *in, int npairs, int b0, int nboot, int64_t rows,
                   const double *fz, const double *fw, double cz, double cw, double inv_n, int64_t G, double *wstate,
                   int first, cudaStream_t st);
void means_pass_pow2(pkde_ctx *ctx, int n1, const double2 *in, int64_t rows, const double *fz, double cz,
                     const double *wstate, int64_t G, int nboot, double vscale, double dlogt, double eps,
                     int64_t steps_low, int64_t steps_over, const StepState &cs, int step, cudaStream_t st);

}  // namespace pkde
