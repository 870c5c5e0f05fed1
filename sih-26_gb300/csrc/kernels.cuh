// kernels.cuh -- the device control block and the launchers of every engine kernel.
//
// The loop state of the reference's PDHG (src/pdhg/pdhg.cpp:181-197: eta, omega, iteration,
// restarts, the restart KKT, the best residuals) lives in ONE device struct, `Ctl`, which
// the kernels read and the last block of each reducing kernel updates. The host never
// touches it inside the loop; it reads a copy of it (a snapshot) every few steps.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "chunks.cuh"
#include "slices.cuh"
#include "tiles.cuh"

namespace sgb {

// Mirrors sankhya::pdhg::Residuals (src/pdhg/pdhg_evaluate.hpp:19-70).
struct Residuals {
  double primal, dual, gap;
  double primal_objective, dual_objective;
  double absolute_primal, absolute_dual;
  double gap_as_verified, complementarity;
};

__host__ __device__ inline double worst(const Residuals& r) {
  double w = r.primal;
  if (w < r.dual) w = r.dual;
  if (w < r.gap) w = r.gap;
  return w;
}

// src/pdhg/pdhg_evaluate.hpp:57-60; tolerances from include/sankhya/tolerances.hpp:19,22,108.
__host__ __device__ inline bool meets_request(const Residuals& r, double tolerance) {
  return r.primal <= tolerance && r.dual <= tolerance && r.gap <= tolerance &&
         r.absolute_primal <= 1e-7;
}
// src/pdhg/pdhg_evaluate.hpp:65-69.
__host__ __device__ inline bool meets_project_standard(const Residuals& r) {
  return r.absolute_primal <= 1e-7 && r.absolute_dual <= 1e-7 && r.gap_as_verified <= 1e-9 &&
         r.complementarity <= 1e-6;
}

// kRestartRound: the mixed method's inner loop decided a restart, which ends a refinement
// round (the anchor moves to the current iterate and the correction is rescaled).
enum DoneCode : int {
  kRunning = 0, kConverged = 1, kIterationLimit = 2, kFault = 3, kRestartRound = 4
};

constexpr int kLogRing = 64;

// One iteration-table row (Logger::iteration, src/pdhg/pdhg.cpp:399-400).
struct EvalRecord {
  long long iteration;
  double primal_objective;  // minimise space, unscaled
  double primal, dual, gap;
};

// Ticket slots (last-block counters), one per reducing kernel.
enum Ticket : int { kTicketDual = 0, kTicketEvalRows = 1, kTicketPrimal = 2, kTicketEvalCols = 3,
                    kTicketApply = 4, kTicketCount = 5 };

struct Ctl {
  // Step size and primal weight, src/pdhg/pdhg.cpp:181-186.
  double eta, omega, spectral_norm, eta_ceiling, restart_kkt, tolerance;
  long long iteration, averaged, last_restart, restarts, attempts, evaluations;
  long long iteration_limit;
  int cur;          // which of the two x / y buffers holds the current iterate
  int pending_add;  // the last step was accepted and its iterate is not yet in the sums
  int eval_now;     // an evaluation is due: set by the step decision, cleared by the
                    // evaluation's last kernel; steps do nothing while it is set
  int done;         // DoneCode
  int use_restarts, stop_at_request, no_information, accepted;
  int copy_best;    // 0: nothing; 1: the current candidate; 2: the average candidate
  int do_restart;
  int final_mode;   // the evaluation kernels evaluate (best_x, best_y) only
  int stop_rule;    // 0: the reference's stopping test; 1: relative KKT only
  int error;        // a bounded wait gave up (kCopyFault, kMeetFault: the host stops with an error)
  int inner_mode;   // the mixed method's inner loop: a restart ends the round
  double movement, interaction;  // of the last attempted step
  double mv_primal;              // primal half of the movement, from k_primal's last block
  // Mixed method, one refinement round (the FP32 inner loop reads these): the primal and
  // dual scale factors of the correction problem, the scaled problem's bound and cost
  // norms, the scaled objective at the round's anchor, and the round's KKT target.
  double dp, dd, bound_norm_s, cost_norm_s, pobj0, round_target;
  Residuals best;
  Residuals final_residuals;
  double model_objective;  // sum of the original-sense costs times best_x (final mode)
  long long log_count;
  EvalRecord log[kLogRing];
  unsigned int ticket[kTicketCount];
};

constexpr int kEvalColSlots = 16;  // doubles per block in the column-evaluation partials
constexpr int kEvalRowSlots = 8;

struct StepBuffers {
  Ctl* ctl;
  SliceSet csc, csr;  // scaled
  double* x[2];
  double* y[2];
  double* x_sum;
  double* y_sum;
  // x' - x per column, written by k_primal and gathered by k_dual, which forms A (2 x' - x) as
  // A x + 2 A (x' - x) with A x carried per row (double-buffered with x): half the gathered bytes and
  // half the products of gathering both. A carried sum's rounding cannot build up: every evaluation,
  // at most 40 accepted steps apart, stores A x afresh.
  double* dx;
  double* ax[2];
  const double *c, *l, *u, *rl, *ru;  // scaled problem
  double* chunk_primal;  // [csc.nchunks]
  double* chunk_dual;    // [csr.nchunks * 2]
  double* part_steps;    // [(the larger grid + 2 csc.nlong + csr.nlong) * 3] (step_totals)
  unsigned long long* arrivals;  // GridMeet's counter
  // The step-size factors by iteration count (decisions.cuh, step_factors).
  const double2* step_factors;
  long long step_factors_n;
};

struct EvalBuffers {
  Ctl* ctl;
  SliceSet csc, csr;  // UNSCALED values
  const double* x[2];
  const double* y[2];
  double* x_sum;
  double* y_sum;
  double *x_rst, *y_rst;
  double* ax[2];                  // the steps' carried scaled A x (StepBuffers)
  const double *dr, *dc;          // row / column scale (Dr, Dc)
  const double* cost;             // minimise-space unscaled cost
  const double* col_cost;         // original-sense cost (for the model objective)
  const double *l, *u, *rl, *ru;  // unscaled bounds
  double bound_norm, cost_norm, sense;
  double *xu[2], *yu[2];  // unscaled candidates (current, average)
  double* reduced;        // reduced cost of candidate 0
  double* best_x;
  double* best_y;
  double* part_rows0;  // [grid_rows * kEvalRowSlots]
  double* part_cols;   // [(grid_cols + 1) * kEvalColSlots]; the last slot holds long columns
  double* part_rows1;  // [grid_rows * kEvalRowSlots]
  double* chunk_cols;  // [csc.nchunks * 2]
  double* chunk_rows;  // [csr.nchunks * 2]
  int grid_rows, grid_cols;
  int m, n;
};

// ---- Launchers (pdhg_kernels.cu) ---------------------------------------------------------
void launch_pdhg_step(const StepBuffers& b, cudaStream_t s);
// The resident form (slices.cuh): up to `attempts` attempted steps in one kernel, which ends at once
// when an evaluation falls due; `smem` is resident_smem of the largest block.
void launch_pdhg_resident(const StepBuffers& b, int attempts, int smem, cudaStream_t s);
// Dynamic shared memory of a resident block with these slices and entry rows of the two layouts, in
// a problem of m rows and n columns; and whether the device can run the cluster with it.
int resident_smem(int m, int n, int col_rows, int col_slices, int row_rows, int row_slices);
bool resident_fits(const StepBuffers& b, int smem);
void launch_primal_pass(const StepBuffers& b, cudaStream_t s);
void launch_dual_pass(const StepBuffers& b, cudaStream_t s);
// Kernels launched per attempted step inside a graph (2 step + 4 evaluation kernels).
// A step graph holds `steps` attempted steps (k_primal + k_dual) and, after every
// kEvalStride of them, the four evaluation kernels. A step that falls due for an evaluation
// sets ctl->eval_now; the steps after it in the graph return at once until the evaluation
// kernels have run and cleared the flag, so the iterates, step sizes and evaluation points
// are those of one evaluation after every due step. The stride divides the 40-step
// evaluation cadence, so on accepted steps the due step ends a stride and nothing is
// skipped. Off a due step the four evaluation kernels return at once.
constexpr int kEvalStride = 8;
inline long long graph_kernel_launches(int steps) {
  return 2LL * steps + 4LL * ((steps + kEvalStride - 1) / kEvalStride);
}
// Running count of kernel launches issued by the launchers of this file (host side).
long long kernel_launch_count();
// The evaluation tick (no-op on the device unless ctl->eval_now or ctl->final_mode).
void launch_evaluation(const EvalBuffers& e, cudaStream_t s);

// Setup kernels.
// The preconditioner (src/la/scaling.cpp:111-159) on both sliced layouts: raw values in, scaled
// values, Dr and Dc (ones on entry) out, and the scaled values' magnitude range.
struct ScalingBuffers {
  SliceSet csr, csc;
  const double *csr_raw, *csc_raw;
  double *csr_val, *csc_val;
  double *row_factor[2], *col_factor[2];  // the rounds' factors, alternating
  double *dr, *dc;
  double* minmax;      // 2 * scale_blocks(csc)
  double* minmax_out;  // {max, min}
  long long nnz;
};
int scale_blocks(const SliceSet& S);
// The setup of a resident LP in one kernel: the preconditioner, the scaled vectors (cs, ls, us, rls,
// rus as launch_scale_vectors forms them) and the power iteration of `steps` steps from `start`
// (n entries). norms[2 k] = |v_k|^2 for k = 0 .. steps, as the power iteration over launches leaves
// them. `smem` and the cluster are the resident step's.
struct ResidentSetup {
  ScalingBuffers scaling;
  const double *cost, *l, *u, *rl, *ru;
  double *cs, *ls, *us, *rls, *rus;
  const double* start;
  double* norms;
  int steps;
};
void launch_resident_setup(const ResidentSetup& r, int threads, int smem, cudaStream_t s);
int resident_threads(const StepBuffers& b);
// Up to `attempts` attempted steps in one cooperative launch, which ends early where an evaluation
// falls due; pdhg_steps_fit: whether the device runs its blocks at once.
void launch_pdhg_steps(const StepBuffers& b, int attempts, cudaStream_t s);
bool pdhg_steps_fit(const StepBuffers& b);
// Launches the passes by themselves to no effect. A kernel's first launch waits for the device's other
// kernels (its code is loaded then), which a solve beside them must not.
void launch_load_passes(cudaStream_t s);
// Asks whether every SM has room for a block of a cooperative grid, without waiting for one (k_room):
// span receives what crowded(), on the host's copy, decides by.
void launch_room(unsigned long long* span, int sms, cudaStream_t s);
bool crowded(const unsigned long long* span);
void launch_scaling(const ScalingBuffers& b, cudaStream_t s);
// The sliced copy of a compressed layout's indices and values, and the values back.
void launch_slice_fill(const SliceSet& S, const int* ptr, const int* idx, const double* val,
                       int* sidx, double* sval, cudaStream_t s);
void launch_slice_unfill(const SliceSet& S, const int* ptr, const double* sval, double* val,
                         cudaStream_t s);
void launch_scale_vectors(int m, int n, const double* cost, const double* l, const double* u,
                          const double* rl, const double* ru, const double* dr, const double* dc,
                          double* cs, double* ls, double* us, double* rls, double* rus,
                          cudaStream_t s);
// Fixed device scratch of the allocation-free product: chunk partials for at most
// kNoAllocMaxChunks pieces of long rows and its completion counter. Set up once per device
// (the symbol addresses, and the counter cleared to zero) under a lock; later calls only read
// the cached addresses.
constexpr int kNoAllocMaxChunks = 16384;
cudaError_t noalloc_scratch(int device, cudaStream_t s, double** chunks, unsigned int** ticket);

// table[e] = step_factors(e) for e < n (decisions.cuh).
void launch_step_factors(double2* table, long long n, cudaStream_t s);
// y = A x (CSR gives A x; CSC gives A^T x). chunk holds a.nchunks doubles; ticket is one device
// counter that is zero on entry and on exit.
void launch_spmv(const SliceSet& a, const double* x, double* y, double* chunk,
                 unsigned int* ticket, cudaStream_t s);
// y = (A x) * *by.
void launch_spmv_scaled(const SliceSet& a, const double* x, double* y, double* chunk,
                        unsigned int* ticket, const double* by, cudaStream_t s);
// y = A x, norm[0] = sum y^2, norm[1] = 1 / its root; part holds a.grid doubles.
void launch_spmv_norm(const SliceSet& a, const double* x, double* y, double* chunk,
                      unsigned int* ticket, double* part, double* norm, cudaStream_t s);
// out[0] = sum v^2, out[1] = 1 / its root, deterministic; part holds grid doubles.
void launch_sumsq(const double* v, int count, double* part, double* out, unsigned int* ticket,
                  cudaStream_t s, int grid);
void launch_project_start(int n, const double* l, const double* u, double* x, cudaStream_t s);
void launch_fill(double* v, int count, double value, cudaStream_t s);

// The FP64 step passes (pass 0 = column pass, 1 = row pass): the elements of the gathered
// vector's window that fit a block.
int fp64_window_capacity(int pass);
// Sets the dynamic shared-memory limits of the FP64 kernels on the current device (once per
// device); false if the device refused.
bool configure_fp64_kernels();
// Fills dst[k] = src[map[k]] in FP32 (the values of a split layout's part), k < count.
void launch_gather_values(const double* src, const int* map, float* dst, long long count,
                          cudaStream_t s);

}  // namespace sgb
