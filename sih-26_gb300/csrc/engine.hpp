// engine.hpp -- host side of the GB300 PDHG engine (one LP, one device).
#pragma once

#include <cuda_runtime.h>

#include <functional>
#include <string>
#include <vector>

#include "chunks.cuh"
#include "kernels.cuh"
#include "mixed.cuh"
#include "sankhya_gb300.h"

namespace sgb {

// A named NVTX range for the lifetime of the object, marking an engine phase on a profiler's
// timeline (nsys, or ncu's --nvtx filters). The names follow SANKHYA's profiler scopes. With no
// tool attached NVTX calls return at once; without the NVTX headers this is empty.
struct Trace {
  explicit Trace(const char* name);
  ~Trace();
  Trace(const Trace&) = delete;
  Trace& operator=(const Trace&) = delete;
};

// Raised inside the engine and turned into a status code at the C boundary.
struct EngineError {
  int code;
  std::string message;
};

// Throws EngineError on any CUDA failure, with the call site in the message.
void cuda_check(cudaError_t err, const char* what, const char* file, int line);
#define SGB_CUDA(call) ::sgb::cuda_check((call), #call, __FILE__, __LINE__)

// A device allocation. allocate() keeps the one it has where that is large enough and not more than
// kKeepFactor times too large (or kKeepBytes), so an engine that is loaded again with a problem of
// like size allocates nothing; a much smaller problem gives the memory back. The contents are
// undefined after it either way. The caller sees to it that no work on the old contents is left.
constexpr size_t kKeepFactor = 4, kKeepBytes = 1u << 20;

template <typename T>
struct DeviceArray {
  T* ptr = nullptr;
  size_t count = 0;
  size_t capacity = 0;
  DeviceArray() = default;
  DeviceArray(const DeviceArray&) = delete;
  DeviceArray& operator=(const DeviceArray&) = delete;
  ~DeviceArray() { release(); }
  void allocate(size_t n);
  void upload(const T* host, size_t n, cudaStream_t s);
  // n entries followed by `pad` zeroed ones (count stays n).
  void allocate_padded(size_t n, size_t pad, cudaStream_t s);
  void upload_padded(const T* host, size_t n, size_t pad, cudaStream_t s);
  void release();
};

// Entries of the step-size factor table (decisions.cuh, step_factors): 16 MB of double2.
constexpr long long kStepFactorTable = 1LL << 20;

class Engine {
 public:
  explicit Engine(int device);
  ~Engine();

  void load(const sankhya_gb300_lp& lp);
  void solve(const sankhya_gb300_params& params, sankhya_gb300_result* result);
  void solution(double* col_value, double* col_dual, double* row_dual);
  void scaling(long long seed, double* row_scale, double* col_scale, double* scaled_values,
               double* spectral_norm);
  void spmv(int op, int scaled, const double* in, double* out);
  // The same product on caller-owned DEVICE buffers, enqueued on `stream` (nullptr: the legacy default
  // stream) with the fixed scratch of noalloc_scratch(): allocates no memory.
  void spmv_noalloc(int op, int scaled, const double* in, double* out, cudaStream_t stream);
  void time_kernels(int reps, double* ms);

  int device() const { return device_; }

 private:
  void require_loaded() const;
  void precondition(long long seed);
  double power_iteration(long long seed);
  ScalingBuffers scaling_buffers() const;
  // The preconditioning and the spectral-norm estimate, over launches or resident.
  double scale_and_norm(long long seed);
  void draw_power_start(long long seed);
  double norm_from_steps();
  void init_iterates(const sankhya_gb300_params& p);
  // `steps` attempted steps with their evaluations on the stream, and the control block's copy to the
  // snapshot slot. together: in cooperative launches (or the resident kernel), else pass by pass.
  void enqueue_steps(int steps, int slot, bool together);
  int enqueue_mixed_steps(int steps, int slot, bool together);  // its kernels
  void build_graphs(int steps);
  void build_mixed_graphs(int steps);
  void destroy_graphs();
  void fill_buffers();
  void fill_mixed_buffers();
  void allocate_mixed();
  // Runs runs of steps, each enqueued by enqueue(slot), until the control block behind `snapshot`
  // says done, the time limit passes or the interrupt flag is raised.
  void run_steps(const sankhya_gb300_params& p, double t0, const std::function<void(int)>& enqueue,
                 Ctl* snapshot, bool forward_log, long long iteration_offset, int* stop_status);
  void final_evaluation();
  void setup(const sankhya_gb300_params& p, sankhya_gb300_result* r, double* norm);
  void solve_fp64(const sankhya_gb300_params& p, sankhya_gb300_result* r, double t0);
  void solve_mixed(const sankhya_gb300_params& p, sankhya_gb300_result* r, double t0);
  void report(const sankhya_gb300_params& p, const Ctl& c, bool converged, long long iterations,
              long long restarts, int stop_status, sankhya_gb300_result* r);

  int device_ = 0;
  cudaStream_t stream_ = nullptr;
  int num_sms_ = 0;
  bool loaded_ = false;
  bool solved_ = false;
  bool scaled_ = false;

  // Problem dimensions and host-side scalars.
  int m_ = 0, n_ = 0;
  long long nnz_ = 0;
  double sense_ = 1.0, offset_ = 0.0;
  double bound_norm_ = 0.0, cost_norm_ = 0.0;
  int nlong_csr_ = 0, nlong_csc_ = 0;
  int nchunks_csr_ = 0, nchunks_csc_ = 0;
  // The FP32 evaluation kernels' tile layout (`lanes` threads per row).
  int ntiles_csr_f_ = 0, ntiles_csc_f_ = 0;
  int lanes_csr_f_ = 1, lanes_csc_f_ = 1;
  int grid_csr_f_ = 1, grid_csc_f_ = 1;
  DeviceArray<Tile> csc_tiles_f_, csr_tiles_f_;
  // The FP64 passes' sliced layouts (slices.cuh) of A by columns and by rows, with the values
  // unscaled (evaluation) and scaled (iterations).
  struct SliceDev {
    DeviceArray<unsigned short> meta;
    DeviceArray<unsigned int> base;
    DeviceArray<int> idx, seg_start, block_start;
    DeviceArray<double> raw, scaled;
    DeviceArray<SliceItem> items;
    DeviceArray<unsigned int> tickets;
    DeviceArray<LongRow> longs;
    DeviceArray<SliceSeg> segs;
    SliceSet view{};      // val = the scaled values
    double staged = 0.0;  // share of the nonzeros gathered from a staged window
    int most_rows = 0, most_slices = 0;  // entry rows and slices of the largest block
  };
  SliceDev sl_csc_, sl_csr_;
  void plan_sliced(SliceDev& D, const std::vector<int>& ptr, const int* idx, int lines,
                   int extent, int pass, int window_cap, int resident);
  // The FP32 step passes' chunk layouts (chunks.cuh): CSC (column pass) and CSR (row pass).
  // A split layout owns its main and outer index arrays (and the maps from their entries to
  // the full layout's, through which each solve fills their values); otherwise it reads the
  // full layout's arrays.
  struct ChunkDev {
    DeviceArray<Tile> chunks;
    DeviceArray<int2> orounds;
    DeviceArray<LongRow> longs;
    DeviceArray<ChunkSeg> segs;
    DeviceArray<int> seg_start, oround_start;
    DeviceArray<int> ptr, idx, map, optr, oidx, omap;
    DeviceArray<float> fval, foval, fouter;
    DeviceArray<int> osorted;  // the outer entries by column within a round,
    DeviceArray<unsigned short> opos;  // their places in the order of the rows
    DeviceArray<float> fosorted;
    DeviceArray<double> pieces;  // piece partials
    // Packed entries of a narrow layout, allocated and filled when the mixed method first runs; the
    // values each solve.
    DeviceArray<float> pval;
    DeviceArray<unsigned short> pidx;
    DeviceArray<int> lo;
    bool narrow = false;
    int nchunks = 0;
    int nlong = 0, npieces = 0, wmax = 0, grid = 1, smem = 0, nrows = 0;
    bool split = false;
    long long nmain = 0, nouter = 0;
    double staged = 0.0;    // share of the nonzeros gathered from a staged window
    double coverage = 0.0;  // share the windows would hold over the whole layout
  };
  ChunkDev ck_csc_f_, ck_csr_f_;
  void plan_layout(ChunkDev& D, const std::vector<int>& ptr, const int* idx, int lines,
                   int extent, int pass, int window_cap);
  void fill_split_values();
  ChunkSet chunk_set(const ChunkDev& D, const int* full_ptr, const int* full_idx,
                            const float* full_val) const;

  // Pattern (shared by scaled and unscaled values).
  DeviceArray<int> csc_ptr_, csc_idx_, csr_ptr_, csr_idx_;
  DeviceArray<LongRow> csc_longs_, csr_longs_;
  // Scaled values in the compressed layouts' order (scaling() and the mixed method's FP32
  // copies), allocated and filled when they are asked for.
  DeviceArray<double> csc_s_, csr_s_;
  void unslice_scaled();
  // Unscaled vectors.
  DeviceArray<double> cost_, col_cost_, l_, u_, rl_, ru_;
  // The step-size factors for iteration counts below kStepFactorTable (filled once).
  DeviceArray<double2> step_factors_;
  // Scaled vectors and scaling.
  DeviceArray<double> cs_, ls_, us_, rls_, rus_, dr_, dc_;
  DeviceArray<double> row_factor_[2], col_factor_[2], minmax_;
  // Iterates.
  DeviceArray<double> x0_, x1_, y0_, y1_, x_sum_, y_sum_, x_rst_, y_rst_;
  DeviceArray<double> xu0_, xu1_, yu0_, yu1_, reduced_, best_x_, best_y_;
  DeviceArray<double> dx_;         // x' - x per column
  DeviceArray<double> ax0_, ax1_;  // scaled A x per row, with x0_ and x1_
  // Reductions.
  DeviceArray<double> part_primal_, part_dual_, part_rows0_, part_cols_, part_rows1_;
  DeviceArray<double> chunk_primal_, chunk_dual_, chunk_cols_, chunk_rows_, chunk_spmv_;
  DeviceArray<double> scalars_, power_v_, power_av_, power_norms_;
  DeviceArray<unsigned int> tickets_;  // setup-kernel last-block counters
  DeviceArray<Ctl> ctl_;

  Ctl* snapshot_ = nullptr;  // pinned host, two slots
  cudaGraphExec_t graph_exec_[2] = {nullptr, nullptr};
  int graph_steps_ = 0;
  int graph_launches_ = 0;  // engine kernels per step graph
  bool steps_ = false;      // FP64 steps run in launch_pdhg_steps' kernel
  // The current solve found other kernels on SMs (launch_room): its steps run pass by pass instead, with
  // the same sums, and without a graph, whose instantiation would wait for those kernels.
  bool crowded_ = false;
  DeviceArray<unsigned long long> room_;
  DeviceArray<double> part_steps_, part_steps_f_, scaled_norms_;
  bool steps_f_ = false;    // the mixed method's steps run in launch_mixed_steps' kernel
  int mgraph_launches_ = 0;  // engine kernels per mixed step graph
  DeviceArray<unsigned long long> arrivals_;
  bool resident_ = false;   // FP64 steps run in the resident kernel,
  int resident_smem_ = 0;   // with this much shared memory a block
  cudaEvent_t done_event_[2] = {nullptr, nullptr};
  cudaEvent_t timing_[2] = {nullptr, nullptr};
  long long launches_ = 0;  // engine kernels launched by the current solve
  long long graphs_launched_ = 0;

  StepBuffers step_{};
  EvalBuffers eval_{};

  // Mixed method (allocated on its first solve).
  int last_precision_ = SANKHYA_GB300_FP64;
  bool mixed_ready_ = false;
  MixedBuffers mixed_{};
  DeviceArray<float> csc_f_, csr_f_;
  DeviceArray<float> u0f_, u1f_, v0f_, v1f_, usumf_, vsumf_, urstf_, vrstf_;
  DeviceArray<float> cf_, lf_, uf_, gu_, gl_, yhat_, uc0_, uc1_, vc0_, vc1_, ubest_, vbest_;
  DeviceArray<float> csf_;   // scaled cost in FP32
  DeviceArray<float> duf_;           // u' - u per column
  DeviceArray<float> auf0_, auf1_;   // A u per row, double-buffered with u
  DeviceArray<double> anchor_x_, anchor_y_, ax64_, aty64_;
  DeviceArray<Ctl> ctl_mixed_;
  Ctl* snapshot_mixed_ = nullptr;  // pinned host, two slots
  cudaGraphExec_t mgraph_exec_[2] = {nullptr, nullptr};
  int mgraph_steps_ = 0;
  double bound_norm_s_ = 0.0, cost_norm_s_ = 0.0;  // scaled problem norms
  long long extra_launches_ = 0;
};

// The sliced layout of one matrix layout (layout.cu): windows of at most `wmax` elements are
// kept where they hold at least `window_min` of the entries; at most `sms` blocks, or `resident`
// of them.
struct SlicePlan {
  int nslices = 0, nchunks = 0, wmax = 0, grid = 1, threads = 128;
  long long long_base = 0, entries = 0;  // first entry of the long region; entries stored
  double staged = 0.0;
  std::vector<unsigned short> meta;
  std::vector<unsigned int> base;
  std::vector<SliceItem> items;
  std::vector<LongRow> longs;
  std::vector<SliceSeg> segs;
  std::vector<int> seg_start, block_start;
};
SlicePlan plan_slices(const std::vector<int>& ptr, const int* idx, int lines, int extent, int wmax,
                      double window_min, int sms, int np, int resident = 0);

size_t estimate_memory(long long rows, long long cols, long long nnz, int precision);

// The step passes' chunk layout of one matrix layout (layout.cu): `ptr` / `idx` its lines
// and indices over a gathered vector of `extent` elements, `cap` entries per chunk, `wmax`
// the window capacity, `grid` blocks, `elem_bytes` the gathered element's size. Windows are
// kept over every entry when they hold at least `full_min` of them; between `split_min` and
// that, the layout is split into main and outer parts; below it, nothing is staged. A split
// layout's outer entries are summed in rounds of at most `outer_round_cap` entries.
struct ChunkPlan {
  int cap = 0, grid = 1, wmax = 0, npieces = 0;
  bool split = false, error = false;
  double coverage = 0.0, staged = 0.0;
  std::vector<Tile> chunks;
  std::vector<int2> orounds;
  std::vector<LongRow> longs;
  std::vector<ChunkSeg> segs;
  std::vector<int> seg_start, oround_start;
  std::vector<int> ptr, idx, map, optr, oidx, omap;  // split layouts only
  // The windows hold every entry of the (main) chunks of whole rows; lo: their starts by chunk.
  bool narrow = false;
  std::vector<int> lo;
};
ChunkPlan plan_chunks(const std::vector<int>& ptr, const int* idx, int lines, int extent, int cap,
                      int wmax, int grid, int elem_bytes, double split_min, double full_min,
                      int outer_round_cap);

// Throws EngineError (ARGUMENT / MODEL) when an LP is malformed. `matrix_known`: the same arrays
// have passed already (a batch's LPs may share them), so their entries are not walked again.
void validate_lp(const sankhya_gb300_lp& lp, bool matrix_known = false);

// Row tiles of a CSR / CSC pattern (see tiles.cuh).
void build_tiles(const std::vector<int>& ptr, int lines, int lanes, int threads,
                 std::vector<Tile>* tiles, std::vector<LongRow>* longs, int* nchunks);

// Gathered-vector windows of one tile layout (see tiles.cuh): `idx` is the layout's index
// array over a gathered vector of `extent` elements, `wmax` the window capacity.
// Returns the number of nonzeros whose index falls in their tile's window.
long long build_windows(const std::vector<Tile>& tiles, const int* idx, int extent, int wmax,
                        std::vector<int>* tile_win, std::vector<int2>* windows);

}  // namespace sgb
