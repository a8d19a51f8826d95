// engine.h -- host-side solver context, plans and Parareal engine of libccfv.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <map>
#include <memory>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/ccfv.h"
#include "ccfv_internal.h"

namespace ccfv {

// Device memory owned by the library; freed on destruction.
struct DevBuf {
  void *p = nullptr;
  size_t bytes = 0;
  DevBuf() = default;
  DevBuf(const DevBuf &) = delete;
  DevBuf &operator=(const DevBuf &) = delete;
  ~DevBuf() { if (p) cudaFree(p); }
  cudaError_t alloc(size_t b);
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
  }
  template <typename T> T *as() const { return reinterpret_cast<T *>(p); }
};

// Line-invariant LU factors of one constant tridiagonal system (device, T[3L]).
struct SolverTable {
  DevBuf buf;
  double sm_fac = 0, sm_inv_den = 0;
};

// The sweep launches of a sequence of steps over a set of fields: kinds x(dt/2),
// y(dt), x(dt/2), and, where the x sweeps of neighbouring steps fuse
// (SWEEP_FILTER_XX), the last one of a step with the first of the next.
struct StepPlan {
  DevBuf mem;             // descriptors SweepField[kinds][nf], then the stencil tables
  int nf = 0;
  bool fused = false;     // steps run x y (xx y)* x: 2 n + 1 passes, else 3 n
  int groups_per_field[4] = {0, 0, 0, 0};
  LaunchGeom geom[4];
  PlanFields by_value[4];  // the same fields as a kernel argument
  bool pp = false;        // out-of-place sequence (SweepField::pp)
  // lines of the per-line stencil tables per sub-step kind (0: none), which the
  // descriptors point to.  The fused pass's table (fmem) is made by the first
  // sequence of several steps.
  int lines[4] = {0, 0, 0, 0};
  DevBuf fmem;
  bool fused_filled = false;
};

// One field of a plan: swept in place on A (B == nullptr), or an out-of-place
// sequence of passes over the pair A/B that starts from in0 (SweepField::pp).
// ends: > 0, a sequence of that many steps ends in A (the parity offset is
// chosen so); 0: its first pass writes B.  t0: the field's time origin.
struct PlanField {
  void *A = nullptr;
  double t0 = 0.0;
  void *B = nullptr;
  const void *in0 = nullptr;
  int ends = 0;
};
// Passes over the field of n steps.
inline int plan_passes(bool fused, int n) { return fused ? 2 * n + 1 : 3 * n; }

}  // namespace ccfv

struct ccfv_ctx {
  ccfv_grid grid;
  int device = 0;
  ccfv::DevBuf status;  // unsigned status word + partial-sum scratch
  // keyed by (dir, sub-step, FP64, diffusion theta) / (dt, FP64, 0, theta)
  std::map<std::tuple<int, double, int, double>, std::unique_ptr<ccfv::SolverTable>> tables;
  std::map<std::tuple<double, int, int, double>, std::unique_ptr<ccfv::StepPlan>> step_plans;
  // Parareal slice states and scratch
  ccfv::DevBuf U, F, Gold, W, C64, C32, norms, partial, counter, io, aux;
  ccfv::DevBuf FS, W2;  // ping-pong partners of the fine slices and the coarse work field
  ccfv::DevBuf pp64, pp32;  // ping-pong partner of single-field calls (FP64, FP32)
  size_t slices_cap = 0;
  std::unique_ptr<ccfv::StepPlan> fine_plan;
  double fine_plan_key[4] = {0, 0, 0, 0};
  const void *fine_plan_bufs[3] = {nullptr, nullptr, nullptr};
  int fine_plan_slices = 0;
  std::string last_error;
  bool force_general = false;  // test hook: route every sweep through the per-cell kernel
};

namespace ccfv {

int set_error(ccfv_ctx *ctx, int code, const std::string &msg);
// `theta` is the implicit weight of the diffusion sub-step: 0.5 is the
// reference's Crank-Nicolson; 1 is backward Euler (L-stable), which the
// coarse propagator may use (ccfv_parareal_opts::coarse_theta).
const SolverTable *get_table(ccfv_ctx *ctx, int dir, double Dt, bool fp64, int *status,
                             double theta = 0.5);
SweepField make_field(const ccfv_grid &g, int dir, double Dt, double ta_rel, double tb_rel,
                      void *data, const SolverTable *tab, int dsrc, double theta = 0.5);
// inplace: the sweep overwrites its input (the filter kernel's segments of a
// line then form one cluster, at most MAX_CLUSTER CTAs).
LaunchGeom step_geom(const ccfv_grid &g, int dir, double Dt, int dsrc, bool fp64,
                     bool inplace = true, double theta = 0.5);
// Diffusion weight of a Parareal run's coarse propagator of step dtc
// (ccfv_parareal_opts::coarse_theta; 0 selects 0.5).
double coarse_theta(const ccfv_parareal_opts &o, const ccfv_grid &g, double dtc);
// Whether coarse_theta holds an accepted value.
inline bool coarse_theta_ok(double th) {
  return th == 0.0 || th == CCFV_COARSE_THETA_AUTO || (th >= 0.5 && th <= 1.0);
}
void filter_field(const ccfv_grid &g, SweepField &f, bool fp64, const LaunchGeom &G);
// for_class: keep the choice for the line-length classes of this grid (the
// batched engine) instead of its exact line lengths (ccfv_autotune).
int autotune(ccfv_ctx *ctx, double dt, bool fp64, cudaStream_t st, int *chosen,
             bool for_class = false);
// Whether the line-length class of L has a tuned segment length.
bool class_tuned(int L, bool fp64);
// The next power of two >= L (at least 64): the batched engine's tuning class.
int line_class(int L);
int batch_solve(int n, const ccfv_problem *probs, ccfv_stats *stats, int device,
                cudaStream_t st, std::string *errmsg);
// homogeneous: the source term is left out (the linear part of the step,
// which the delta form of Parareal applies to slice increments).
// nsteps: steps of the sequence that it is built for (it serves others too; not
// 1: any sequence).
int build_step_plan(ccfv_ctx *ctx, StepPlan *plan, double dt, bool fp64,
                    const std::vector<std::pair<void *, double>> &fields, int nsteps,
                    bool homogeneous = false, double theta = 0.5);
int build_step_plan(ccfv_ctx *ctx, StepPlan *plan, double dt, bool fp64,
                    const std::vector<PlanField> &fields, int nsteps, bool homogeneous = false,
                    double theta = 0.5);
// nsteps steps of dt from t0 on fields first .. first+count-1 of a plan.  io:
// buffers of a single field that replace the plan's; y_in_place: the last
// step's y sweep writes over its input, so that the sequence ends in the
// other buffer than its number of passes says.
int run_steps(ccfv_ctx *ctx, StepPlan &plan, bool fp64, int first, int count, double t0,
              double dt, int nsteps, cudaStream_t st, const FieldIo &io = FieldIo(),
              bool y_in_place = false);
// nsteps steps of the field `src` into d_C (null: d_C in place).
int steps(ccfv_ctx *ctx, void *d_C, bool fp64, double t0, double dt, int nsteps, cudaStream_t st,
          double theta = 0.5, const void *src = nullptr);
// Whether the x sweeps of neighbouring steps of dt fuse into one pass, and its
// geometry.
bool fused_x_geom(const ccfv_grid &g, double dt, bool fp64, bool inplace, double theta,
                  LaunchGeom *G);
int coarse_fp32(ccfv_ctx *ctx, double *d_C, double tn, double DT, int m, cudaStream_t st,
                double theta = 0.5);
int fine_slices(ccfv_ctx *ctx, double *d_fields, int n, double t0, double slice_dt, double DT,
                int J, cudaStream_t st);
int correct(ccfv_ctx *ctx, int form, double *U, const double *Fv, double *Gold, double *W,
            double *sq_update, double *sq_state, cudaStream_t st);
int parareal(ccfv_ctx *ctx, const ccfv_parareal_opts *o, const double *C0, double *C_T,
             ccfv_stats *stats, cudaStream_t st);
int exact_ref(ccfv_ctx *ctx, double *d_C, double t, cudaStream_t st);
int gaussians(ccfv_ctx *ctx, double *d_C, int ng, const double *params, int img, cudaStream_t st);
int norms(ccfv_ctx *ctx, const double *a, const double *b, double *rel_l2, double *max_abs,
          cudaStream_t st);
constexpr int RED_BLOCKS_MAX = 592;

}  // namespace ccfv
