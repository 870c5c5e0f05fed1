// pdhg_kernels.cu -- the FP64 hot path of the GB300 PDHG engine.
//
// Per attempted step (src/pdhg/pdhg.cpp:220-335) there are TWO kernels, both on the sliced
// rows of slices.cuh (the FP32 method's step kernels run on the warp chunks of chunks.cuh
// instead):
//   k_primal  one pass over the CSC copy of Ahat: A^T y gathered per column, fused with the
//             projected primal update x' = proj(x - tau (c + A^T y)), dx = x' - x (written
//             once per column for the row pass), the primal half of the movement, and the
//             deferred x_sum update.
//   k_dual    one pass over the CSR copy: A dx gathered per row, A (2x' - x) = A x + 2 A dx
//             with A x carried, fused with the Moreau dual update, the dual movement and the
//             interaction dy^T A dx; its last block sums every block's partials in a fixed
//             order and takes the step-size decision on the device.
// Small LPs run a period's steps in one resident cluster kernel (k_pdhg_resident), larger ones
// in one cooperative launch (k_pdhg_steps), with the same arithmetic per item.
// The evaluation tick (src/pdhg/pdhg.cpp:341-483, src/pdhg/pdhg_evaluate.cpp) is three
// fused passes over the UNSCALED values plus one vector pass; it runs only when the step
// decision asks for it and otherwise returns at once.
//
// GB300 executes FP64 at about 1/64 of its FP32 rate, so this method is bound by the FP64
// pipe rather than by HBM: the kernels are written to spend as few FP64 instructions per
// entry as the method allows (one FMA per entry and product), to divide only where a row
// is not an equality, and to keep every reduction deterministic.
#include "common.cuh"
#include "decisions.cuh"
#include "kernels.cuh"
#include "slices.cuh"

#include <algorithm>
#include <cstdio>
#include <mutex>

namespace sgb {

namespace {

long long g_launches = 0;

constexpr int kScratch = 16 * (kSliceThreads / 32);
// Entry rows per piece of the passes that gather a pair per entry (a row pass that gathered
// (2x' - x, x' - x), 500,000 x 1M block-angular LP: 86.5 us with 8, 86.6 with 6, 90.7 with 4; Zipf
// rows 60.3, 62.8, 63.8 us).
constexpr int kPairPiece = kPiece;

// Per-device state: whether the kernels' shared-memory limits are set on the device, and
// its occupancy and SM count (an engine on device 1 needs its own opt-in).
constexpr int kMaxDevices = 64;
struct DeviceConfig {
  bool configured;
  int sms;
};
std::mutex g_config_mutex;
DeviceConfig g_config[kMaxDevices];

int current_device() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  return dev >= 0 && dev < kMaxDevices ? dev : -1;
}

int device_sms() {
  const int dev = current_device();
  if (dev < 0) return 1;
  std::lock_guard<std::mutex> lock(g_config_mutex);
  if (g_config[dev].sms == 0) {
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
      cudaGetLastError();
      sms = 1;
    }
    g_config[dev].sms = sms > 0 ? sms : 1;
  }
  return g_config[dev].sms;
}

__device__ __forceinline__ void raise_error(Ctl* c) {
  c->error = kCopyFault;
  c->done = kFault;
}

// The reference's stopping test (src/pdhg/pdhg.cpp:424-425), or relative KKT alone.
__device__ bool fp64_stop_test(const Ctl* c, const Residuals& r) {
  return c->stop_rule == 1 ? worst(r) <= c->tolerance
                           : meets_request(r, c->tolerance) &&
                                 (c->stop_at_request || meets_project_standard(r));
}

// The three sums of a step's decision, a warp each (the block's first 96 threads): the primal movement,
// the dual movement over omega, the interaction. From the blocks' partials, those of the long columns
// (half: which of their two sets) and those of the long rows; entries that a column or a row does not
// have, or a block past its layout's grid, stay zero. The order is the same whichever kernel adds.
__device__ __forceinline__ void step_totals(const StepBuffers& b, int half, double omega,
                                            double inv_omega, double* s_sums) {
  if (threadIdx.x >= 96) return;
  const int q = static_cast<int>(threadIdx.x) >> 5;
  const int G = max(b.csc.grid, b.csr.grid), nc = b.csc.nlong;
  const double sum = table_sum(G + nc + b.csr.nlong, [&](int k) {
    const int skip = k < G ? 0 : (k < G + nc ? half * nc : nc);
    return __ldcg(b.part_steps + 3 * (k + skip) + q);
  });
  if ((threadIdx.x & 31) == 0) {
    s_sums[q] = q == 0 ? 0.5 * omega * sum : (q == 1 ? 0.5 * sum * inv_omega : sum);
  }
}

// ---- k_primal ----------------------------------------------------------------------------
__global__ void __launch_bounds__(kSliceThreads, 1) k_primal(StepBuffers b) {
  if (b.ctl == nullptr) return;  // launch_load_passes
  extern __shared__ __align__(128) unsigned char dsmem[];
  __shared__ double scratch[kScratch];
  SliceStart<kPiece> start;
  start_slices(b.csc, start);
  grid_dependency_wait();  // the previous kernels' results (launch_after)
  Ctl* ctl = b.ctl;
  // Every control field the pass reads, loaded together before the first test.
  const int done = ctl->done, eval_now = ctl->eval_now, cur = ctl->cur;
  const bool add = ctl->pending_add != 0;
  const long long iteration = ctl->iteration, limit = ctl->iteration_limit;
  const double omega = ctl->omega, eta = ctl->eta;
  if (done != kRunning || eval_now != 0 || iteration >= limit) {
    // src/pdhg/pdhg.cpp:206
    if (done == kRunning && eval_now == 0 && blockIdx.x == 0 && threadIdx.x == 0) {
      ctl->done = kIterationLimit;
    }
    return;
  }
  const double* __restrict__ x = b.x[cur];
  double* __restrict__ xn = b.x[cur ^ 1];
  const double* __restrict__ y = b.y[cur];
  // Formed once per block: an FP64 division per thread would hold GB300's slow FP64 pipe.
  __shared__ double s_tau;
  if (threadIdx.x == 0) s_tau = eta / omega;
  __syncthreads();
  const double tau = s_tau;
  double mv[1] = {0.0};  // sum of dx^2
  auto fetch = [&](int i) { return __ldg(y + i); };
  auto mac = [](double v, double g, double* acc) { acc[0] = fma(v, g, acc[0]); };
  // Operands of column j: x, c, l, u and (when the last step is still to be added) x_sum.
  auto load = [&](int j, double* o) {
    o[0] = x[j];
    o[1] = b.c[j];
    o[2] = b.l[j];
    o[3] = b.u[j];
    o[4] = add ? b.x_sum[j] : 0.0;
  };
  auto epi = [&](int j, const double* s, const double* o) {
    const double xj = o[0];
    if (add) b.x_sum[j] = o[4] + xj;
    const double gradient = o[1] + s[0];
    // Unfused, as src/pdhg/pdhg.cpp:232-233 rounds it.
    const double xnj = clamp_box(__dsub_rn(xj, __dmul_rn(tau, gradient)), o[2], o[3]);
    xn[j] = xnj;
    const double d = xnj - xj;
    b.dx[j] = d;
    mv[0] = fma(d, d, mv[0]);
  };
  auto finish = [&](int l, int j, const double* s, const double* o) {
    const double sum = mv[0];
    mv[0] = 0.0;
    epi(j, s, o);
    b.part_steps[3 * (max(b.csc.grid, b.csr.grid) + l)] = mv[0];
    mv[0] = sum;
  };
  if (!run_slices<true, 1, 5>(b.csc, start, y, fetch, dsmem, b.chunk_primal, mac, load, epi,
                              finish) &&
      threadIdx.x == 0) {
    raise_error(ctl);
  }
  // Each block publishes its partial, and k_dual's last block sums them (step_totals). No block of
  // this pass waits for another.
  double out[1];
  block_sum<1>(mv, scratch, out);
  if (threadIdx.x == 0) b.part_steps[3 * blockIdx.x] = out[0];
}

// ---- k_dual ------------------------------------------------------------------------------
__global__ void __launch_bounds__(kSliceThreads, 1) k_dual(StepBuffers b) {
  if (b.ctl == nullptr) return;  // launch_load_passes
  extern __shared__ __align__(128) unsigned char dsmem[];
  __shared__ double scratch[kScratch];
  SliceStart<kPiece> start;
  start_slices(b.csr, start);
  grid_dependency_wait();  // the previous kernels' results (launch_after)
  Ctl* ctl = b.ctl;
  const int done = ctl->done, eval_now = ctl->eval_now, cur = ctl->cur;
  const bool add = ctl->pending_add != 0;
  const double omega = ctl->omega, eta = ctl->eta;
  if (done != kRunning || eval_now != 0) return;
  // What the last block's decision needs beside the sums, formed now.
  __shared__ StepPrep s_prep;
  __shared__ double s_sums[3];
  if (threadIdx.x == blockDim.x - 1) {
    s_prep.set(ctl, step_factors(ctl->iteration, b.step_factors, b.step_factors_n));
  }
  const double* __restrict__ y = b.y[cur];
  double* __restrict__ yn = b.y[cur ^ 1];
  const double* __restrict__ dx = b.dx;
  const double* __restrict__ ax = b.ax[cur];
  double* __restrict__ axn = b.ax[cur ^ 1];
  const double sigma = eta * omega;
  __syncthreads();
  const double inv_sigma = s_prep.inv_sigma;
  double acc2[2] = {0.0, 0.0};  // sum dy^2, sum dy (A dx)
  auto fetch = [&](int j) { return __ldg(dx + j); };
  auto mac = [](double v, double g, double* acc) { acc[0] = fma(v, g, acc[0]); };
  // Operands of row i: y, rl, ru, (when the last step is still to be added) y_sum, and A x.
  auto load = [&](int i, double* o) {
    o[0] = y[i];
    o[1] = b.rl[i];
    o[2] = b.ru[i];
    o[3] = add ? b.y_sum[i] : 0.0;
    o[4] = ax[i];
  };
  auto epi = [&](int i, const double* s, const double* o) {
    const double yi = o[0];
    if (add) b.y_sum[i] = o[3] + yi;
    // Unfused, as the reference rounds it (src/pdhg/pdhg.cpp:244-245): a fused
    // v - sigma * (v / sigma) would leave the division's rounding error on a free row.
    axn[i] = o[4] + s[0];
    const double v = __dadd_rn(yi, __dmul_rn(sigma, fma(2.0, s[0], o[4])));
    const double p = row_projection(v, sigma, inv_sigma, o[1], o[2]);
    const double yni = __dsub_rn(v, __dmul_rn(sigma, p));
    yn[i] = yni;
    const double d = yni - yi;
    acc2[0] = fma(d, d, acc2[0]);
    acc2[1] = fma(d, s[0], acc2[1]);
  };
  auto finish = [&](int l, int i, const double* s, const double* o) {
    const double sums[2] = {acc2[0], acc2[1]};
    acc2[0] = acc2[1] = 0.0;
    epi(i, s, o);
    const int at = max(b.csc.grid, b.csr.grid) + 2 * b.csc.nlong + l;
    for (int q = 0; q < 2; ++q) {
      b.part_steps[3 * at + 1 + q] = acc2[q];
      acc2[q] = sums[q];
    }
  };
  if (!run_slices<true, 1, 5>(b.csr, start, dx, fetch, dsmem, b.chunk_dual, mac, load, epi,
                              finish) &&
      threadIdx.x == 0) {
    raise_error(ctl);
  }
  double out[2];
  block_sum<2>(acc2, scratch, out);
  __shared__ int s_last;
  if (threadIdx.x == 0) {
    b.part_steps[3 * blockIdx.x + 1] = out[0];
    b.part_steps[3 * blockIdx.x + 2] = out[1];
    __threadfence();
    s_last = atomicAdd(&ctl->ticket[kTicketDual], 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  step_totals(b, 0, omega, s_prep.inv_omega, s_sums);
  __syncthreads();
  if (threadIdx.x == 0) {
    ctl->ticket[kTicketDual] = 0;
    if (ctl->done == kRunning) {
      ctl->mv_primal = s_sums[0];
      step_decision(ctl, s_sums[0] + s_sums[1], fabs(s_sums[2]), s_prep);
    }
  }
}

// ---- The resident step (slices.cuh) -----------------------------------------------------------
// The passes of k_primal and k_dual, item for item, in one cluster. Every block keeps a copy of the
// control block and takes the same step decision from the same sums, in the same order, so the
// blocks agree on every branch. The warps' partial sums go to every block, into one of two tables
// by step: a block may be in the next column pass while another still adds the last step's.
constexpr int kResidentWarps = kResidentThreads / 32;
constexpr int kResidentTable = kResidentBlocks * kResidentWarps;

// Copies a block's state to (or, WRITE, from) shared memory: the slots' items of `src`.
template <bool WRITE>
__device__ __forceinline__ void local_items(const LocalSlices& L, double* slots, double* global) {
  for (int k = static_cast<int>(threadIdx.x); k < L.n * 32; k += static_cast<int>(blockDim.x)) {
    const unsigned m = L.meta[k];
    if (m == kNoRow) continue;
    const int item = slice_row(L.s0 + k / 32, m);
    if (WRITE) {
      global[item] = slots[k];
    } else {
      slots[k] = global[item];
    }
  }
}

__global__ void __launch_bounds__(kResidentThreads, 1) k_pdhg_resident(StepBuffers b, int attempts) {
  extern __shared__ __align__(128) unsigned char dsmem[];
  __shared__ Ctl s_ctl;
  __shared__ StepPrep s_prep;
  __shared__ double s_tau, s_sigma, s_sums[3];
  __shared__ double s_part[2][3][kResidentTable];
  static_assert(sizeof(Ctl) % sizeof(unsigned long long) == 0, "copied by words");
  constexpr int kWords = static_cast<int>(sizeof(Ctl) / sizeof(unsigned long long));
  const int T = static_cast<int>(blockDim.x), t = static_cast<int>(threadIdx.x);
  const int C = static_cast<int>(gridDim.x), W = T >> 5, lane = t & 31, warp = t >> 5;
  const int m = b.csr.nrows, n = b.csc.nrows;
  unsigned long long* const words = reinterpret_cast<unsigned long long*>(&s_ctl);
  for (int k = t; k < kWords; k += T) {
    words[k] = reinterpret_cast<const volatile unsigned long long*>(b.ctl)[k];
  }
  // Shared memory: the gathered vectors at the same place in every block, then the block's own.
  double2* const xd = reinterpret_cast<double2*>(dsmem);
  double* const ys[2] = {reinterpret_cast<double*>(xd + n), reinterpret_cast<double*>(xd + n) + m};
  unsigned char* mem = dsmem + (static_cast<size_t>(n) * 16 + static_cast<size_t>(m) * 16);
  LocalSlices cs, rs;
  mem = fill_local(b.csc, cs, mem);
  mem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(mem) + 15) & ~uintptr_t(15));
  mem = fill_local(b.csr, rs, mem);
  double* const own = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(mem) + 15) & ~uintptr_t(15));
  const int nc = cs.n * 32, nr = rs.n * 32;
  double* const x[2] = {own, own + nc};
  double *const xsum = own + 2 * nc, *const c = own + 3 * nc, *const lo = own + 4 * nc,
         *const up = own + 5 * nc;
  double *const ysum = own + 6 * nc, *const rl = ysum + nr, *const ru = ysum + 2 * nr;
  __syncthreads();
  const int first = s_ctl.cur;
  local_items<false>(cs, x[first], b.x[first]);
  local_items<false>(cs, xsum, b.x_sum);
  local_items<false>(cs, c, const_cast<double*>(b.c));
  local_items<false>(cs, lo, const_cast<double*>(b.l));
  local_items<false>(cs, up, const_cast<double*>(b.u));
  local_items<false>(rs, ysum, b.y_sum);
  local_items<false>(rs, rl, const_cast<double*>(b.rl));
  local_items<false>(rs, ru, const_cast<double*>(b.ru));
  for (int i = t; i < m; i += T) ys[first][i] = b.y[first][i];
  if (t == 0) {
    if (s_ctl.done == kRunning && s_ctl.eval_now == 0 &&
        s_ctl.iteration >= s_ctl.iteration_limit) {
      s_ctl.done = kIterationLimit;  // src/pdhg/pdhg.cpp:206
    }
    s_tau = s_ctl.eta / s_ctl.omega;
    s_sigma = s_ctl.eta * s_ctl.omega;
  }
  cluster_meet();  // every block has read the control block, and may be written to
  for (int a = 0; a < attempts; ++a) {
    if (s_ctl.done != kRunning || s_ctl.eval_now != 0) break;
    const int cur = s_ctl.cur;
    const bool add = s_ctl.pending_add != 0;
    const double tau = s_tau, sigma = s_sigma, omega = s_ctl.omega;
    double(*const part)[kResidentTable] = s_part[a & 1];
    if (t == T - 1) {
      s_prep.set(&s_ctl, step_factors(s_ctl.iteration, b.step_factors, b.step_factors_n));
    }
    {
      const double* y = ys[cur];
      double mv = 0.0;
      for (int s = warp; s < cs.n; s += W) {
        const unsigned meta = cs.meta[s * 32 + lane];
        if (meta == kNoRow) continue;
        const int len = static_cast<int>(meta >> 8), e = cs.base[s] * 32 + lane, k = s * 32 + lane;
        double g = 0.0;
#pragma unroll 4
        for (int q = 0; q < len; ++q) g = fma(cs.val[e + q * 32], y[cs.idx[e + q * 32]], g);
        const double xj = x[cur][k];
        if (add) xsum[k] = xsum[k] + xj;
        const double xnj = clamp_box(__dsub_rn(xj, __dmul_rn(tau, c[k] + g)), lo[k], up[k]);
        x[cur ^ 1][k] = xnj;
        const double d = xnj - xj;
        const double2 both = make_double2(fma(2.0, xnj, -xj), d);
        double2* const at = xd + slice_row(cs.s0 + s, meta);
        for (int r = 0; r < C; ++r) cluster_store(cluster_addr(at, r), both);
        mv = fma(d, d, mv);
      }
      __syncwarp();
      if (__any_sync(0xffffffffu, mv != 0.0)) mv = warp_sum(mv);  // an idle warp adds nothing
      if (lane < C) {
        cluster_store(cluster_addr(&part[0][static_cast<int>(blockIdx.x) * W + warp], lane), mv);
      }
    }
    cluster_meet();
    {
      const double* y = ys[cur];
      double* const yn = ys[cur ^ 1];
      double dy2 = 0.0, ia = 0.0;
      for (int s = warp; s < rs.n; s += W) {
        const unsigned meta = rs.meta[s * 32 + lane];
        if (meta == kNoRow) continue;
        const int len = static_cast<int>(meta >> 8), e = rs.base[s] * 32 + lane, k = s * 32 + lane;
        double s0 = 0.0, s1 = 0.0;
#pragma unroll 4
        for (int q = 0; q < len; ++q) {
          const double v = rs.val[e + q * 32];
          const double2 p = xd[rs.idx[e + q * 32]];
          s0 = fma(v, p.x, s0);
          s1 = fma(v, p.y, s1);
        }
        const int i = slice_row(rs.s0 + s, meta);
        const double yi = y[i];
        if (add) ysum[k] = ysum[k] + yi;
        const double v = __dadd_rn(yi, __dmul_rn(sigma, s0));
        const double p = row_projection(v, sigma, s_prep.inv_sigma, rl[k], ru[k]);
        const double yni = __dsub_rn(v, __dmul_rn(sigma, p));
        for (int r = 0; r < C; ++r) cluster_store(cluster_addr(yn + i, r), yni);
        const double d = yni - yi;
        dy2 = fma(d, d, dy2);
        ia = fma(d, s1, ia);
      }
      __syncwarp();
      double both[2] = {dy2, ia};
      if (__any_sync(0xffffffffu, dy2 != 0.0 || ia != 0.0)) {
        warp_sums<2>(both);
        dy2 = __shfl_sync(0xffffffffu, both[0], 0);
        ia = __shfl_sync(0xffffffffu, both[0], 16);
      }
      if (lane < C) {
        const int at = static_cast<int>(blockIdx.x) * W + warp;
        cluster_store(cluster_addr(&part[1][at], lane), dy2);
        cluster_store(cluster_addr(&part[2][at], lane), ia);
      }
    }
    cluster_meet();
    // A warp per sum: the primal movement, the dual movement over omega, the interaction.
    if (t < 96) {
      const int q = t >> 5;
      const double sum = table_sum(C * W, [&](int k) { return part[q][k]; });
      if (lane == 0) s_sums[q] = q == 0 ? 0.5 * omega * sum : (q == 1 ? 0.5 * sum * s_prep.inv_omega : sum);
    }
    __syncthreads();
    if (t == 0) {
      s_ctl.mv_primal = s_sums[0];
      step_decision(&s_ctl, s_sums[0] + s_sums[1], fabs(s_sums[2]), s_prep);
      if (s_ctl.eval_now == 0 && s_ctl.iteration >= s_ctl.iteration_limit) {
        s_ctl.done = kIterationLimit;
      }
      // eta / omega, rounded as the launch's first step has it: where a period is cut must not show.
      s_tau = divide(s_ctl.eta, s_ctl.omega, s_prep.inv_omega);
      s_sigma = s_ctl.eta * s_ctl.omega;
    }
    __syncthreads();
  }
  // The current iterate, the sums and the control block go back; the other buffers are written
  // before they are read again.
  const int last = s_ctl.cur;
  local_items<true>(cs, x[last], b.x[last]);
  local_items<true>(cs, xsum, b.x_sum);
  local_items<true>(rs, ysum, b.y_sum);
  for (int k = t; k < nr; k += T) {
    const unsigned meta = rs.meta[k];
    if (meta == kNoRow) continue;
    const int i = slice_row(rs.s0 + k / 32, meta);
    b.y[last][i] = ys[last][i];
  }
  if (blockIdx.x == 0) {
    for (int k = t; k < kWords; k += T) reinterpret_cast<unsigned long long*>(b.ctl)[k] = words[k];
  }
}

// ---- The steps of a period in one launch ---------------------------------------------------------
// k_primal and k_dual, item for item, by one cooperative grid whose blocks meet between the passes;
// every block takes the step decision from the same partials. The next pass's first entries are
// under way while a block waits. Operands a thread reads of its own rows it wrote itself; gathered
// vectors are read with ld_live.
__global__ void __launch_bounds__(kSliceThreads, 1) k_pdhg_steps(StepBuffers b, int attempts) {
  __shared__ double scratch[3 * (kSliceThreads / 32)];
  __shared__ Ctl s_ctl;
  __shared__ StepPrep s_prep;
  __shared__ double s_tau, s_sigma, s_sums[3];
  constexpr int kWords = static_cast<int>(sizeof(Ctl) / sizeof(unsigned long long));
  const int t = static_cast<int>(threadIdx.x), T = static_cast<int>(blockDim.x);
  const int block = static_cast<int>(blockIdx.x), G = static_cast<int>(gridDim.x);
  unsigned long long* const words = reinterpret_cast<unsigned long long*>(&s_ctl);
  for (int k = t; k < kWords; k += T) {
    words[k] = reinterpret_cast<const volatile unsigned long long*>(b.ctl)[k];
  }
  GridMeet grid;
  grid.start(b.arrivals);
  const auto meet = [&] {
    if (grid.meet(&b.ctl->error)) return true;
    if (t == 0) b.ctl->done = kFault;  // the kernels that follow do nothing
    return false;
  };
  __syncthreads();
  if (t == 0) {
    if (s_ctl.done == kRunning && s_ctl.eval_now == 0 &&
        s_ctl.iteration >= s_ctl.iteration_limit) {
      s_ctl.done = kIterationLimit;  // src/pdhg/pdhg.cpp:206
    }
    s_tau = s_ctl.eta / s_ctl.omega;
    s_sigma = s_ctl.eta * s_ctl.omega;
  }
  __syncthreads();
  SliceStart<kPiece> cols;
  if (block < b.csc.grid) start_slices(b.csc, cols);
  for (int a = 0; a < attempts; ++a) {
    if (s_ctl.done != kRunning || s_ctl.eval_now != 0) break;
    const int cur = s_ctl.cur;
    const bool add = s_ctl.pending_add != 0;
    const double* y = b.y[cur];
    double sums[3] = {0.0, 0.0, 0.0};  // dx^2, dy^2, dy (A dx)
    if (t == T - 1) {
      s_prep.set(&s_ctl, step_factors(s_ctl.iteration, b.step_factors, b.step_factors_n));
    }
    {
      const double* x = b.x[cur];
      double* xn = b.x[cur ^ 1];
      const double tau = s_tau;
      auto fetch = [&](int i) { return ld_live(y + i); };
      auto mac = [](double v, double g, double* acc) { acc[0] = fma(v, g, acc[0]); };
      auto load = [&](int j, double* o) {
        o[0] = x[j];
        o[1] = b.c[j];
        o[2] = b.l[j];
        o[3] = b.u[j];
        o[4] = add ? b.x_sum[j] : 0.0;
      };
      auto epi = [&](int j, const double* s, const double* o) {
        const double xj = o[0];
        if (add) b.x_sum[j] = o[4] + xj;
        const double gradient = o[1] + s[0];
        const double xnj = clamp_box(__dsub_rn(xj, __dmul_rn(tau, gradient)), o[2], o[3]);
        xn[j] = xnj;
        const double d = xnj - xj;
        b.dx[j] = d;
        sums[0] = fma(d, d, sums[0]);
      };
      auto finish = [&](int l, int j, const double* s, const double* o) {
        const double sum = sums[0];
        sums[0] = 0.0;
        epi(j, s, o);
        b.part_steps[3 * (G + (a & 1) * b.csc.nlong + l)] = sums[0];
        sums[0] = sum;
      };
      if (block < b.csc.grid) {
        run_slices<false, 1, 5>(b.csc, cols, y, fetch, nullptr, b.chunk_primal, mac, load, epi,
                                finish);
      }
    }
    {
      SliceStart<kPiece> rows;
      if (block < b.csr.grid) start_slices(b.csr, rows);
      if (!meet()) return;
      const double* dx = b.dx;
      const double* ax = b.ax[cur];
      double* axn = b.ax[cur ^ 1];
      double* yn = b.y[cur ^ 1];
      const double sigma = s_sigma, inv_sigma = s_prep.inv_sigma;
      auto fetch = [&](int j) { return ld_live(dx + j); };
      auto mac = [](double v, double g, double* acc) { acc[0] = fma(v, g, acc[0]); };
      auto load = [&](int i, double* o) {
        o[0] = y[i];
        o[1] = b.rl[i];
        o[2] = b.ru[i];
        o[3] = add ? b.y_sum[i] : 0.0;
        o[4] = ax[i];
      };
      auto epi = [&](int i, const double* s, const double* o) {
        const double yi = o[0];
        if (add) b.y_sum[i] = o[3] + yi;
        axn[i] = o[4] + s[0];
        const double v = __dadd_rn(yi, __dmul_rn(sigma, fma(2.0, s[0], o[4])));
        const double p = row_projection(v, sigma, inv_sigma, o[1], o[2]);
        const double yni = __dsub_rn(v, __dmul_rn(sigma, p));
        yn[i] = yni;
        const double d = yni - yi;
        sums[1] = fma(d, d, sums[1]);
        sums[2] = fma(d, s[0], sums[2]);
      };
      auto finish = [&](int l, int i, const double* s, const double* o) {
        const double keep[2] = {sums[1], sums[2]};
        sums[1] = sums[2] = 0.0;
        epi(i, s, o);
        for (int q = 1; q < 3; ++q) {
          b.part_steps[3 * (G + 2 * b.csc.nlong + l) + q] = sums[q];
          sums[q] = keep[q - 1];
        }
      };
      if (block < b.csr.grid) {
        run_slices<false, 1, 5>(b.csr, rows, dx, fetch, nullptr, b.chunk_dual, mac, load, epi,
                                finish);
      }
    }
    double part[3];
    block_sum<3>(sums, scratch, part);
    if (t == 0) {
      for (int q = 0; q < 3; ++q) b.part_steps[3 * block + q] = part[q];
    }
    if (block < b.csc.grid) start_slices(b.csc, cols);
    if (!meet()) return;
    // The long columns' partials of this attempt: a block still at the last decision reads the other
    // half.
    step_totals(b, a & 1, s_ctl.omega, s_prep.inv_omega, s_sums);
    __syncthreads();
    if (t == 0) {
      s_ctl.mv_primal = s_sums[0];
      step_decision(&s_ctl, s_sums[0] + s_sums[1], fabs(s_sums[2]), s_prep);
      if (s_ctl.eval_now == 0 && s_ctl.iteration >= s_ctl.iteration_limit) {
        s_ctl.done = kIterationLimit;
      }
      // eta / omega, rounded as the launch's first step has it: where a period is cut must not show.
      s_tau = divide(s_ctl.eta, s_ctl.omega, s_prep.inv_omega);
      s_sigma = s_ctl.eta * s_ctl.omega;
    }
    __syncthreads();
  }
  if (block == 0) {
    for (int k = t; k < kWords; k += T) reinterpret_cast<unsigned long long*>(b.ctl)[k] = words[k];
  }
}

// ---- Room for a cooperative grid -------------------------------------------------------------
// A cooperative launch starts when every SM has room for its block: beside a kernel that holds SMs for
// seconds (a batch in another thread) it would wait for that kernel's end, where launches of single
// passes share what is free. So a solve asks first. A block here takes all of an SM's shared memory, so
// that no other block is resident beside it, notes when it started and stays kRoomStay ns; it waits
// for nobody. span[0] = ~(first start), span[1] = last start: where SMs are held, blocks start that
// late or later.
constexpr long long kRoomStay = 8000;
__device__ __forceinline__ long long global_ns() {
  long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
__global__ void k_room(unsigned long long* span) {
  const long long start = global_ns();
  atomicMax(span, ~static_cast<unsigned long long>(start));
  atomicMax(span + 1, static_cast<unsigned long long>(start));
  for (int polls = 0; polls < 100000 && global_ns() - start < kRoomStay; ++polls) {
  }
}

// ---- Evaluation ----------------------------------------------------------------------------
__device__ __forceinline__ bool eval_active(const Ctl* c) {
  return c->final_mode != 0 || (c->eval_now != 0 && c->done == kRunning);
}

// E0: rows, no matrix. Unscaled y candidates, the row half of the dual objective and dual
// violation (src/pdhg/pdhg_evaluate.cpp:80-98), and |y - y_restart|^2.
__global__ void __launch_bounds__(kTileThreads) k_eval_rows0(EvalBuffers e) {
  __shared__ double scratch[kScratch];
  const Ctl* c = e.ctl;
  if (!eval_active(c)) return;
  const bool fin = c->final_mode != 0;
  const int cur = c->cur;
  const bool avg = !fin && c->averaged > 0;
  const bool pend = c->pending_add != 0;
  const double count = static_cast<double>(c->averaged);
  double acc[5] = {0.0, 0.0, 0.0, 0.0, 0.0};  // support0, viol0, support1, viol1, dy^2
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < e.m; i += gridDim.x * blockDim.x) {
    double cand[2];
    int nc = 1;
    if (fin) {
      cand[0] = e.best_y[i];
    } else {
      const double yc = e.y[cur][i];
      cand[0] = yc * e.dr[i];
      if (avg) {
        const double sum = pend ? e.y_sum[i] + yc : e.y_sum[i];
        cand[1] = (sum / count) * e.dr[i];
        nc = 2;
      }
      const double d = yc - e.y_rst[i];
      acc[4] += d * d;
    }
    const double rl = e.rl[i], ru = e.ru[i];
    for (int q = 0; q < nc; ++q) {
      const double yi = cand[q];
      e.yu[q][i] = yi;
      if (yi > 0.0) {
        if (finite_bound(ru)) acc[2 * q] += yi * ru; else acc[2 * q + 1] += yi * yi;
      } else if (yi < 0.0) {
        if (finite_bound(rl)) acc[2 * q] += yi * rl; else acc[2 * q + 1] += yi * yi;
      }
    }
  }
  double out[5];
  block_sum<5>(acc, scratch, out);
  if (threadIdx.x == 0) {
    for (int q = 0; q < 5; ++q) e.part_rows0[blockIdx.x * kEvalRowSlots + q] = out[q];
  }
}

// E1: columns over the unscaled CSC. Reduced costs d = c + A^T y of both candidates, the
// column half of the dual violation / dual objective / complementarity, the primal objective
// (src/pdhg/pdhg_evaluate.cpp:54-78,111-139) and |x - x_restart|^2.
__global__ void __launch_bounds__(kSliceThreads, 1) k_eval_cols(EvalBuffers e) {
  __shared__ double scratch[kScratch];
  Ctl* c = e.ctl;
  if (!eval_active(c)) return;
  const bool fin = c->final_mode != 0;
  const int cur = c->cur;
  const bool avg = !fin && c->averaged > 0;
  const bool pend = c->pending_add != 0;
  const double count = static_cast<double>(c->averaged);
  const double* __restrict__ yu0 = e.yu[0];
  const double* __restrict__ yu1 = e.yu[1];
  // sums: viol0, bc0, pobj0, viol1, bc1, pobj1, dx^2, model objective; maxes: comp0, comp1
  double acc[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  double cmax[2] = {0.0, 0.0};
  auto fetch = [&](int i) { return make_double2(yu0[i], avg ? yu1[i] : 0.0); };
  auto mac = [&](double v, double2 g, double* a) {
    a[0] = fma(v, g.x, a[0]);
    if (avg) a[1] = fma(v, g.y, a[1]);
  };
  auto load = [](int, double*) {};
  auto epi = [&](int j, const double* s, const double*) {
    const double cj = e.cost[j], lj = e.l[j], uj = e.u[j];
    double xc[2];
    const int nc = avg ? 2 : 1;
    if (fin) {
      xc[0] = e.best_x[j];
      acc[7] += e.col_cost[j] * xc[0];
    } else {
      const double xj = e.x[cur][j];
      xc[0] = xj * e.dc[j];
      if (avg) {
        const double sum = pend ? e.x_sum[j] + xj : e.x_sum[j];
        xc[1] = (sum / count) * e.dc[j];
      }
      const double d = xj - e.x_rst[j];
      acc[6] += d * d;
    }
    for (int q = 0; q < nc; ++q) {
      const double d = cj + s[q];
      if (q == 0) e.reduced[j] = d;
      e.xu[q][j] = xc[q];
      if (d > 0.0) {
        if (finite_bound(lj)) acc[3 * q + 1] += d * lj; else acc[3 * q] += d * d;
      } else if (d < 0.0) {
        if (finite_bound(uj)) acc[3 * q + 1] += d * uj; else acc[3 * q] += d * d;
      }
      if (lj != uj) {
        const double ls = finite_bound(lj) ? xc[q] - lj : HUGE_VAL;
        const double us = finite_bound(uj) ? uj - xc[q] : HUGE_VAL;
        cmax[q] = dmax(cmax[q], fabs(d) * dmin(ls, us));
      }
      acc[3 * q + 2] += cj * xc[q];
    }
  };
  SliceStart<kPairPiece> start;
  start_slices(e.csc, start);
  run_slices<false, 2, 0, double2>(e.csc, start, nullptr, fetch, nullptr, e.chunk_cols, mac, load, epi);
  double out[8], mout[2];
  block_sum<8>(acc, scratch, out);
  block_max<2>(cmax, scratch, mout);
  __shared__ int s_last;
  if (threadIdx.x == 0) {
    double* p = e.part_cols + blockIdx.x * kEvalColSlots;
    for (int q = 0; q < 8; ++q) p[q] = out[q];
    p[8] = mout[0];
    p[9] = mout[1];
    __threadfence();
    s_last = atomicAdd(&c->ticket[kTicketEvalCols], 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // Last block: long columns into the extra slot e.part_cols[grid_cols].
  for (int q = 0; q < 8; ++q) acc[q] = 0.0;
  cmax[0] = cmax[1] = 0.0;
  run_slice_long_rows<2, 0>(e.csc, e.chunk_cols, load, epi);
  block_sum<8>(acc, scratch, out);
  block_max<2>(cmax, scratch, mout);
  if (threadIdx.x == 0) {
    double* p = e.part_cols + e.grid_cols * kEvalColSlots;
    for (int q = 0; q < 8; ++q) p[q] = out[q];
    p[8] = mout[0];
    p[9] = mout[1];
    c->ticket[kTicketEvalCols] = 0;
  }
}

__device__ Residuals assemble(double pviol, double cviol, double rviol, double bc, double support,
                              double pobj, double comp, double bound_norm, double cost_norm) {
  Residuals r;
  r.absolute_primal = sqrt(pviol);
  r.primal = r.absolute_primal / (1.0 + bound_norm);
  r.absolute_dual = sqrt(cviol + rviol);
  r.dual = r.absolute_dual / (1.0 + cost_norm);
  r.complementarity = comp;
  r.primal_objective = pobj;
  r.dual_objective = bc - support;
  const double gap = fabs(r.primal_objective - r.dual_objective);
  r.gap = gap / (1.0 + fabs(r.primal_objective) + fabs(r.dual_objective));
  r.gap_as_verified = gap / dmax(1.0, fabs(r.primal_objective));
  return r;
}

// E2: rows over the unscaled CSR. Activities of both candidates, primal violation and the
// row complementarity (src/pdhg/pdhg_evaluate.cpp:29-45,99-110). The last block assembles
// the Residuals and takes the best / stop / restart decisions (src/pdhg/pdhg.cpp:349-483).
__global__ void __launch_bounds__(kSliceThreads, 1) k_eval_rows1(EvalBuffers e) {
  __shared__ double scratch[kScratch];
  Ctl* c = e.ctl;
  if (!eval_active(c)) return;
  const bool fin = c->final_mode != 0;
  const bool avg = !fin && c->averaged > 0;
  const double* __restrict__ xu0 = e.xu[0];
  const double* __restrict__ xu1 = e.xu[1];
  double* __restrict__ ax = e.ax[c->cur];
  double acc[2] = {0.0, 0.0};
  double cmax[2] = {0.0, 0.0};
  auto fetch = [&](int j) { return make_double2(xu0[j], avg ? xu1[j] : 0.0); };
  auto mac = [&](double v, double2 g, double* a) {
    a[0] = fma(v, g.x, a[0]);
    if (avg) a[1] = fma(v, g.y, a[1]);
  };
  auto load = [](int, double*) {};
  auto epi = [&](int i, const double* s, const double*) {
    if (!fin) ax[i] = e.dr[i] * s[0];  // the scaled A x of the current iterate, afresh
    const double rl = e.rl[i], ru = e.ru[i];
    const int nc = avg ? 2 : 1;
    for (int q = 0; q < nc; ++q) {
      const double a = s[q];
      double violation = 0.0;
      if (finite_bound(rl)) violation = dmax(violation, rl - a);
      if (finite_bound(ru)) violation = dmax(violation, a - ru);
      acc[q] += violation * violation;
      if (rl != ru) {
        const double ls = finite_bound(rl) ? a - rl : HUGE_VAL;
        const double us = finite_bound(ru) ? ru - a : HUGE_VAL;
        cmax[q] = dmax(cmax[q], fabs(e.yu[q][i]) * dmin(ls, us));
      }
    }
  };
  SliceStart<kPairPiece> start;
  start_slices(e.csr, start);
  run_slices<false, 2, 0, double2>(e.csr, start, nullptr, fetch, nullptr, e.chunk_rows, mac, load, epi);
  double mout[2], sums[2];
  block_max<2>(cmax, scratch, mout);
  block_sum<2>(acc, scratch, sums);
  __shared__ int s_last;
  if (threadIdx.x == 0) {
    double* p = e.part_rows1 + blockIdx.x * kEvalRowSlots;
    p[0] = sums[0];
    p[1] = sums[1];
    p[2] = mout[0];
    p[3] = mout[1];
    __threadfence();
    s_last = atomicAdd(&c->ticket[kTicketEvalRows], 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();

  // ---- Last block: long rows, then every partial in a fixed order. ----
  acc[0] = acc[1] = 0.0;
  cmax[0] = cmax[1] = 0.0;
  run_slice_long_rows<2, 0>(e.csr, e.chunk_rows, load, epi);
  double s[15];
#pragma unroll
  for (int q = 0; q < 15; ++q) s[q] = 0.0;
  double m4[4] = {cmax[0], cmax[1], 0.0, 0.0};
  s[5] = acc[0];
  s[6] = acc[1];
  for (int b = threadIdx.x; b < e.grid_rows; b += blockDim.x) {
    for (int q = 0; q < 5; ++q) s[q] += __ldcg(e.part_rows0 + b * kEvalRowSlots + q);
    s[5] += __ldcg(e.part_rows1 + b * kEvalRowSlots + 0);
    s[6] += __ldcg(e.part_rows1 + b * kEvalRowSlots + 1);
    m4[0] = dmax(m4[0], __ldcg(e.part_rows1 + b * kEvalRowSlots + 2));
    m4[1] = dmax(m4[1], __ldcg(e.part_rows1 + b * kEvalRowSlots + 3));
  }
  for (int b = threadIdx.x; b <= e.grid_cols; b += blockDim.x) {
    for (int q = 0; q < 8; ++q) s[7 + q] += __ldcg(e.part_cols + b * kEvalColSlots + q);
    m4[2] = dmax(m4[2], __ldcg(e.part_cols + b * kEvalColSlots + 8));
    m4[3] = dmax(m4[3], __ldcg(e.part_cols + b * kEvalColSlots + 9));
  }
  double t15[15];
  block_sum<15>(s, scratch, t15);
  double t4[4];
  block_max<4>(m4, scratch, t4);
  if (threadIdx.x != 0) return;
  c->ticket[kTicketEvalRows] = 0;
  // t15: [0] support0 [1] rviol0 [2] support1 [3] rviol1 [4] dy^2 [5] pviol0 [6] pviol1
  //      [7] cviol0 [8] bc0 [9] pobj0 [10] cviol1 [11] bc1 [12] pobj1 [13] dx^2 [14] model obj
  const Residuals cur = assemble(t15[5], t15[7], t15[1], t15[8], t15[0], t15[9],
                                 dmax(t4[0], t4[2]), e.bound_norm, e.cost_norm);
  if (fin) {
    c->final_residuals = cur;
    c->model_objective = t15[14];
    return;
  }
  Residuals av;
  if (avg) {
    av = assemble(t15[6], t15[10], t15[3], t15[11], t15[2], t15[12], dmax(t4[1], t4[3]),
                  e.bound_norm, e.cost_norm);
  }
  tick_decisions(c, cur, avg ? &av : nullptr, fp64_stop_test, t15[13], t15[4], 1e-6, 1e6);
}

// E4: the vector half of the decisions: best point copy, restart anchors, zeroed sums. The
// last block to finish clears the evaluation flags, which lets the next step run.
__global__ void k_eval_apply(EvalBuffers e) {
  Ctl* c = e.ctl;
  if (c->eval_now == 0 || c->final_mode != 0) return;
  const int copy = c->copy_best;
  const bool restart = c->do_restart != 0;
  const int cur = c->cur;
  const int total = (copy == 0 && !restart) ? 0 : (e.m > e.n ? e.m : e.n);
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < total; k += gridDim.x * blockDim.x) {
    if (k < e.n) {
      if (copy) e.best_x[k] = e.xu[copy - 1][k];
      if (restart) {
        e.x_rst[k] = e.x[cur][k];
        e.x_sum[k] = 0.0;
      }
    }
    if (k < e.m) {
      if (copy) e.best_y[k] = e.yu[copy - 1][k];
      if (restart) {
        e.y_rst[k] = e.y[cur][k];
        e.y_sum[k] = 0.0;
      }
    }
  }
  clear_evaluation_flags(c);
}

// ---- Setup kernels (src/la/scaling.cpp) ----------------------------------------------------

// The scaling rounds run on the sliced layouts: every load and store of the values coalesced, a
// line's magnitudes added in ascending index order, the reference's
// accumulation order. (One thread per line on the compressed layouts read 32 scattered
// entries per load: 101 us for the factors of one layout and 123 us to apply them on the
// 500,000 x 1M block-angular LP, and 1.35 and 2.5 ms where a Zipf row of 6,674 entries held one
// thread.) One kernel per layout and round applies the round's factors, takes the next round's
// from the values it has in registers and folds its own into the accumulated scale, so a
// round reads and writes each layout's values once.
enum ScaleMode { kScaleMax = 0, kScaleSum = 1, kScaleNone = 2 };

struct ScaleArgs {
  SliceSet S;            // the layout; S.val is not used
  const double* in;      // the values before the round
  double* out;           // and after it (may be `in`)
  const double* line;    // the round's factors of the layout's lines (nullptr: first, no apply)
  const double* other;   // and of the other side
  double* next;          // the next round's line factors (not for kScaleNone)
  double* scale;         // accumulated line scale, multiplied by `line`
  int line_is_row;
  // kScaleNone: per-block {max, -min} magnitudes of the final values, or nullptr.
  double* minmax;
};

// value <- (value * row factor) * column factor (src/la/scaling.cpp:21-28).
__device__ __forceinline__ double scaled_value(double v, double lp, double op, int line_is_row) {
  return line_is_row ? (v * lp) * op : (v * op) * lp;
}

// The pass factor of a line: 1 / sqrt of its maximum (Ruiz) or sum (Pock-Chambolle) of
// magnitudes, 1 for an empty line.
__device__ __forceinline__ double pass_factor(double acc) {
  return acc > 0.0 ? 1.0 / sqrt(acc) : 1.0;
}

constexpr int kScaleThreads = 256;

// The scaled data of one column or row (src/la/scaling.cpp:124-145). An absent bound is stored as
// an IEEE infinity (the reference keeps +-1e30 as is and tests it with is_finite_bound each time),
// so the step kernels project with min/max.
__device__ __forceinline__ void scale_column(double d, double cost, double l, double u, double* cs,
                                             double* ls, double* us) {
  *cs = cost * d;
  const double inv = 1.0 / d;
  *ls = finite_bound(l) ? l * inv : -HUGE_VAL;
  *us = finite_bound(u) ? u * inv : HUGE_VAL;
}
__device__ __forceinline__ void scale_row(double d, double rl, double ru, double* rls,
                                          double* rus) {
  *rls = finite_bound(rl) ? rl * d : -HUGE_VAL;
  *rus = finite_bound(ru) ? ru * d : HUGE_VAL;
}

// Maximum and minimum of non-negative doubles by their bits (which order as the values do): the
// integer pipe's, where FP64 compares would take as long as the rounds' multiplications.
__device__ __forceinline__ double max_magnitude(double a, double b) {
  return __longlong_as_double(max(__double_as_longlong(a), __double_as_longlong(b)));
}
__device__ __forceinline__ double min_magnitude(double a, double b) {
  return __longlong_as_double(min(__double_as_longlong(a), __double_as_longlong(b)));
}

template <int MODE, bool APPLY>
__global__ void __launch_bounds__(kScaleThreads) k_scale_round(ScaleArgs a) {
  __shared__ double scratch[2 * (kScaleThreads / 32)];
  const int lane = static_cast<int>(threadIdx.x) & 31;
  const int warp = static_cast<int>(threadIdx.x) >> 5;
  const int slice_blocks = (a.S.nslices + kScaleThreads / 32 - 1) / (kScaleThreads / 32);
  double most = 0.0, least = HUGE_VAL;  // kScaleNone: the magnitudes' range
  const auto take = [&](double mag, double& acc) {
    if (MODE == kScaleMax) acc = max_magnitude(acc, mag);
    if (MODE == kScaleSum) acc = acc + mag;
    if (MODE == kScaleNone) {
      most = max_magnitude(most, mag);
      least = min_magnitude(least, mag);
    }
  };
  if (static_cast<int>(blockIdx.x) < slice_blocks) {
    const int s = static_cast<int>(blockIdx.x) * (kScaleThreads / 32) + warp;
    if (s < a.S.nslices) {
      const unsigned m = __ldg(a.S.meta + static_cast<size_t>(s) * 32 + lane);
      if (m != kNoRow) {
        const int len = static_cast<int>(m >> 8), row = slice_row(s, m);
        const size_t at = static_cast<size_t>(__ldg(a.S.base + s)) * 32 + lane;
        const double lp = APPLY ? a.line[row] : 1.0;
        double acc = 0.0;
#pragma unroll 4
        for (int k = 0; k < len; ++k) {
          double v = ld_stream(a.in + at + static_cast<size_t>(k) * 32);
          if (APPLY) {
            const int o = ld_stream(a.S.idx + at + static_cast<size_t>(k) * 32);
            v = scaled_value(v, lp, __ldg(a.other + o), a.line_is_row);
            a.out[at + static_cast<size_t>(k) * 32] = v;
          }
          take(fabs(v), acc);
        }
        if (APPLY) a.scale[row] *= lp;
        if (MODE != kScaleNone) a.next[row] = pass_factor(acc);
      }
    }
  } else {
    // A block per long row: its warps take 32-entry runs in turn; the sum is taken by one warp
    // in index order.
    const int r = static_cast<int>(blockIdx.x) - slice_blocks;
    const SliceItem first = a.S.items[r];
    // Items of one row follow one another: only the row's first runs, over all its entries.
    if (r > 0 && a.S.items[r - 1].row == first.row) {
      if (MODE == kScaleNone && a.minmax != nullptr && threadIdx.x == 0) {
        a.minmax[2 * blockIdx.x] = 0.0;
        a.minmax[2 * blockIdx.x + 1] = -HUGE_VAL;
      }
      return;
    }
    int count = 0;
    for (int q = r; q < a.S.nitems && a.S.items[q].row == first.row; ++q) count += a.S.items[q].count;
    const size_t at = static_cast<size_t>(a.S.long_base) + static_cast<size_t>(first.begin);
    const double lp = APPLY ? a.line[first.row] : 1.0;
    double acc = 0.0;
    for (int k = static_cast<int>(threadIdx.x); k < count; k += kScaleThreads) {
      double v = ld_stream(a.in + at + k);
      if (APPLY) {
        v = scaled_value(v, lp, __ldg(a.other + ld_stream(a.S.idx + at + k)), a.line_is_row);
        a.out[at + k] = v;
      }
      if (MODE != kScaleSum) take(fabs(v), acc);
    }
    if (MODE == kScaleMax) {
      double v[1] = {acc}, total[1];
      block_max<1>(v, scratch, total);
      acc = total[0];
    }
    if (MODE == kScaleSum) {
      __syncthreads();  // the block's stores to `out` before warp 0 reads them
      const double* src = APPLY ? a.out : a.in;
      if (warp == 0) {
        double v = lane < count ? fabs(__ldcg(src + at + lane)) : 0.0;
        for (int k = 0; k < count; k += 32) {
          const int kn = k + 32 + lane;
          const double ahead = kn < count ? fabs(__ldcg(src + at + kn)) : 0.0;
          const int n = count - k < 32 ? count - k : 32;
          for (int q = 0; q < n; ++q) acc = acc + __shfl_sync(0xffffffffu, v, q);
          v = ahead;
        }
      }
    }
    if (threadIdx.x == 0) {
      if (APPLY) a.scale[first.row] *= lp;
      if (MODE != kScaleNone) a.next[first.row] = pass_factor(acc);
    }
  }
  if (MODE == kScaleNone && a.minmax != nullptr) {
    double mm[2] = {most, -least}, out[2];
    block_max<2>(mm, scratch, out);
    if (threadIdx.x == 0) {
      a.minmax[2 * blockIdx.x] = out[0];
      a.minmax[2 * blockIdx.x + 1] = out[1];
    }
  }
}

// out[0] = max, out[1] = min of the magnitudes from the blocks' {max, -min} pairs (0 when there
// are none). One block.
__global__ void __launch_bounds__(kScaleThreads) k_minmax_final(const double* part, int count,
                                                               long long entries, double* out) {
  __shared__ double scratch[2 * (kScaleThreads / 32)];
  double a[2] = {0.0, -HUGE_VAL};
  for (int b = static_cast<int>(threadIdx.x); b < count; b += kScaleThreads) {
    a[0] = dmax(a[0], part[2 * b]);
    a[1] = dmax(a[1], part[2 * b + 1]);
  }
  double o[2];
  block_max<2>(a, scratch, o);
  if (threadIdx.x == 0) {
    out[0] = o[0];
    out[1] = entries > 0 ? -o[1] : 0.0;
  }
}

// The sliced copy of a compressed layout (load), one warp per slice or item; and back, the
// values only (the scaled values in the caller's or the FP32 layouts' order).
template <bool BACK>
__global__ void __launch_bounds__(256) k_slice_copy(SliceSet S, const int* __restrict__ ptr,
                                                    int* idx, double* val, int* sidx,
                                                    double* sval) {
  const int lane = static_cast<int>(threadIdx.x) & 31;
  const int w = static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (w < S.nslices) {
    const unsigned m = S.meta[static_cast<size_t>(w) * 32 + lane];
    if (m == kNoRow) return;
    const int len = static_cast<int>(m >> 8), a = ptr[slice_row(w, m)];
    const size_t at = static_cast<size_t>(S.base[w]) * 32 + lane;
    for (int k = 0; k < len; ++k) {
      const size_t q = at + static_cast<size_t>(k) * 32;
      if (BACK) {
        val[a + k] = sval[q];
      } else {
        sidx[q] = idx[a + k];
        sval[q] = val[a + k];
      }
    }
    return;
  }
  if (w - S.nslices >= S.nitems) return;
  const SliceItem it = S.items[w - S.nslices];
  // An item's place in its row: the entries of the row's items before it.
  int before = 0;
  for (int q = w - S.nslices - 1; q >= 0 && S.items[q].row == it.row; --q) before += S.items[q].count;
  const int a = ptr[it.row] + before;
  const size_t at = static_cast<size_t>(S.long_base) + static_cast<size_t>(it.begin);
  for (int k = lane; k < it.count; k += 32) {
    if (BACK) {
      val[a + k] = sval[at + k];
    } else {
      sidx[at + k] = idx[a + k];
      sval[at + k] = val[a + k];
    }
  }
}

// src/la/scaling.cpp:124-145.
__global__ void k_scale_vectors(int m, int n, const double* cost, const double* l,
                                const double* u, const double* rl, const double* ru,
                                const double* dr, const double* dc, double* cs, double* ls,
                                double* us, double* rls, double* rus) {
  const int total = m > n ? m : n;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < total; k += gridDim.x * blockDim.x) {
    if (k < n) scale_column(dc[k], cost[k], l[k], u[k], cs + k, ls + k, us + k);
    if (k < m) scale_row(dr[k], rl[k], ru[k], rls + k, rus + k);
  }
}

// The whole setup of a resident LP, in its cluster (slices.cuh): every block scales its slices of
// both layouts in shared memory, the lines' factors and then the power iteration's vectors copied
// to every block as they are formed: latency alone, two cluster barriers a step. A call on 50 x 100
// (80 iterations) takes 1.29 ms so, 1.70 ms with the eighty-odd launches of the other path.
template <bool SUM>
__device__ __forceinline__ void local_factors(const LocalSlices& L, double* factors, int C) {
  const int W = static_cast<int>(blockDim.x) >> 5, warp = static_cast<int>(threadIdx.x) >> 5;
  const int lane = static_cast<int>(threadIdx.x) & 31;
  for (int s = warp; s < L.n; s += W) {
    const unsigned meta = L.meta[s * 32 + lane];
    if (meta == kNoRow) continue;
    const int len = static_cast<int>(meta >> 8), e = L.base[s] * 32 + lane;
    double acc = 0.0;
    for (int q = 0; q < len; ++q) {
      const double mag = fabs(L.val[e + q * 32]);
      acc = SUM ? acc + mag : max_magnitude(acc, mag);
    }
    const double f = pass_factor(acc);
    double* const at = factors + slice_row(L.s0 + s, meta);
    for (int r = 0; r < C; ++r) cluster_store(cluster_addr(at, r), f);
  }
}

// Applies a round's factors to the block's slices and to its lines' accumulated scale.
__device__ __forceinline__ void local_apply(const LocalSlices& L, const double* line,
                                            const double* other, double* scale, int line_is_row) {
  const int W = static_cast<int>(blockDim.x) >> 5, warp = static_cast<int>(threadIdx.x) >> 5;
  const int lane = static_cast<int>(threadIdx.x) & 31;
  for (int s = warp; s < L.n; s += W) {
    const unsigned meta = L.meta[s * 32 + lane];
    if (meta == kNoRow) continue;
    const int len = static_cast<int>(meta >> 8), e = L.base[s] * 32 + lane;
    const double lp = line[slice_row(L.s0 + s, meta)];
    for (int q = 0; q < len; ++q) {
      L.val[e + q * 32] = scaled_value(L.val[e + q * 32], lp, other[L.idx[e + q * 32]], line_is_row);
    }
    scale[s * 32 + lane] *= lp;
  }
}

// The block's lines' sums of the matrix times v, times `by`, to every block's `out`; returns this
// thread's sum of their squares.
__device__ __forceinline__ double local_product(const LocalSlices& L, const double* v, double by,
                                                double* out, int C) {
  const int W = static_cast<int>(blockDim.x) >> 5, warp = static_cast<int>(threadIdx.x) >> 5;
  const int lane = static_cast<int>(threadIdx.x) & 31;
  double sq = 0.0;
  for (int s = warp; s < L.n; s += W) {
    const unsigned meta = L.meta[s * 32 + lane];
    if (meta == kNoRow) continue;
    const int len = static_cast<int>(meta >> 8), e = L.base[s] * 32 + lane;
    double acc = 0.0;
#pragma unroll 4
    for (int q = 0; q < len; ++q) acc = fma(L.val[e + q * 32], v[L.idx[e + q * 32]], acc);
    acc *= by;
    double* const at = out + slice_row(L.s0 + s, meta);
    for (int r = 0; r < C; ++r) cluster_store(cluster_addr(at, r), acc);
    sq = fma(acc, acc, sq);
  }
  return sq;
}

__global__ void __launch_bounds__(kResidentThreads, 1) k_resident_setup(ResidentSetup r) {
  extern __shared__ __align__(128) unsigned char dsmem[];
  __shared__ double s_part[2][2][kResidentTable];
  __shared__ double s_norm2, s_inv;
  const ScalingBuffers& b = r.scaling;
  const int T = static_cast<int>(blockDim.x), t = static_cast<int>(threadIdx.x);
  const int C = static_cast<int>(gridDim.x), W = T >> 5, lane = t & 31, warp = t >> 5;
  const int m = b.csr.nrows, n = b.csc.nrows;
  double* const fc[2] = {reinterpret_cast<double*>(dsmem), reinterpret_cast<double*>(dsmem) + n};
  double* const fr[2] = {fc[1] + n, fc[1] + n + m};
  SliceSet csc = b.csc, csr = b.csr;
  csc.val = b.csc_raw;
  csr.val = b.csr_raw;
  LocalSlices cs, rs;
  unsigned char* mem = fill_local(csc, cs, dsmem + static_cast<size_t>(m + n) * 16);
  mem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(mem) + 15) & ~uintptr_t(15));
  mem = fill_local(csr, rs, mem);
  double* const dc = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(mem) + 15) & ~uintptr_t(15));
  double* const dr = dc + cs.n * 32;
  for (int k = t; k < cs.n * 32; k += T) dc[k] = 1.0;
  for (int k = t; k < rs.n * 32; k += T) dr[k] = 1.0;
  cluster_meet();
  local_factors<false>(cs, fc[0], C);
  local_factors<false>(rs, fr[0], C);
  cluster_meet();
  for (int round = 0; round < 11; ++round) {
    const int now = round & 1, then = now ^ 1;
    local_apply(cs, fc[now], fr[now], dc, 0);
    local_apply(rs, fr[now], fc[now], dr, 1);
    // A lane takes the next factor of the lines it has just scaled.
    if (round < 9) {
      local_factors<false>(cs, fc[then], C);
      local_factors<false>(rs, fr[then], C);
    } else if (round == 9) {
      local_factors<true>(cs, fc[then], C);
      local_factors<true>(rs, fr[then], C);
    }
    cluster_meet();
  }
  // The scaled matrix, the scales and the scaled vectors go out; the magnitudes' range.
  double most = 0.0, least = HUGE_VAL;
  for (int side = 0; side < 2; ++side) {
    const LocalSlices& L = side ? rs : cs;
    const SliceSet& S = side ? csr : csc;
    double* const out = side ? b.csr_val : b.csc_val;
    const size_t at = static_cast<size_t>(S.base[L.s0]) * 32;
    for (int s = warp; s < L.n; s += W) {
      const unsigned meta = L.meta[s * 32 + lane];
      if (meta == kNoRow) continue;
      const int len = static_cast<int>(meta >> 8), e = L.base[s] * 32 + lane;
      for (int q = 0; q < len; ++q) {
        const double v = L.val[e + q * 32];
        out[at + static_cast<size_t>(e + q * 32)] = v;
        if (side == 0) {
          most = max_magnitude(most, fabs(v));
          least = min_magnitude(least, fabs(v));
        }
      }
      const int item = slice_row(L.s0 + s, meta);
      if (side == 0) {
        const double d = dc[s * 32 + lane];
        b.dc[item] = d;
        scale_column(d, r.cost[item], r.l[item], r.u[item], r.cs + item, r.ls + item, r.us + item);
      } else {
        const double d = dr[s * 32 + lane];
        b.dr[item] = d;
        scale_row(d, r.rl[item], r.ru[item], r.rls + item, r.rus + item);
      }
    }
  }
  __syncwarp();
  most = warp_max(most);
  least = -warp_max(-least);
  if (lane == 0) {
    const int at = static_cast<int>(blockIdx.x) * W + warp;
    cluster_store(cluster_addr(&s_part[0][0][at], 0), most);
    cluster_store(cluster_addr(&s_part[0][1][at], 0), -least);
  }
  // The power iteration (src/la/scaling.cpp:161-194): v in fc[0], A v in fr[0], every block's copy
  // of the start its own.
  double* const v = fc[0];
  double* const av = fr[0];
  double sq = 0.0;
  for (int j = t; j < n; j += T) {
    v[j] = r.start[j];
    sq = fma(v[j], v[j], sq);
  }
  sq = warp_sum(sq);
  if (lane == 0) s_part[1][0][warp] = sq;
  cluster_meet();
  if (blockIdx.x == 0 && t < 32) {
    double a = 0.0, c = -HUGE_VAL;
    for (int k = lane; k < C * W; k += 32) {
      a = dmax(a, s_part[0][0][k]);
      c = dmax(c, s_part[0][1][k]);
    }
    a = warp_max(a);
    c = warp_max(c);
    if (lane == 0) {
      b.minmax_out[0] = a;
      b.minmax_out[1] = b.nnz > 0 ? -c : 0.0;
    }
  }
  int entries = W;  // of the table that holds the current |v|^2
  for (int step = 0;; ++step) {
    const double* const table = s_part[(step + 1) & 1][0];
    if (t < 32) {
      double sum = 0.0;
      for (int k = lane; k < entries; k += 32) sum += table[k];
      sum = warp_sum(sum);
      if (lane == 0) {
        s_norm2 = sum;
        s_inv = 1.0 / sqrt(sum);
      }
    }
    __syncthreads();
    if (blockIdx.x == 0 && t == 0) r.norms[2 * step] = s_norm2;
    if (step == r.steps) break;
    local_product(rs, v, s_inv, av, C);
    cluster_meet();
    double out = local_product(cs, av, 1.0, v, C);
    __syncwarp();
    if (__any_sync(0xffffffffu, out != 0.0)) out = warp_sum(out);
    if (lane < C) {
      cluster_store(cluster_addr(&s_part[step & 1][0][static_cast<int>(blockIdx.x) * W + warp], lane),
                    out);
    }
    entries = C * W;
    cluster_meet();
  }
}

// y = A x, a short row summed in ascending index order. SCALE multiplies every row's sum by
// *by; NORM leaves the sum of y^2 in norm[0] and the reciprocal of its root in norm[1]
// (part holds a double per block). The vector is gathered from L1 and L2 (x may lie at any
// 8-byte boundary, so no window is staged from it).
template <bool SCALE, bool NORM>
__global__ void __launch_bounds__(kSliceThreads, 1) k_spmv(SliceSet a, const double* x, double* y,
                                                           double* chunk, unsigned int* ticket,
                                                           const double* by, double* part,
                                                           double* norm) {
  __shared__ double scratch[kSliceThreads / 32];
  const double scale = SCALE ? *by : 1.0;
  double sq[1] = {0.0};
  auto fetch = [&](int c) { return __ldg(x + c); };
  auto mac = [](double v, double g, double* acc) { acc[0] = fma(v, g, acc[0]); };
  auto load = [](int, double*) {};
  auto epi = [&](int r, const double* s, const double*) {
    const double v = SCALE ? s[0] * scale : 0.0 + s[0];
    y[r] = v;
    if (NORM) sq[0] = fma(v, v, sq[0]);
  };
  SliceStart<kPiece> start;
  start_slices(a, start);
  run_slices<false, 1, 0, double>(a, start, nullptr, fetch, nullptr, chunk, mac, load, epi);
  if (NORM) {
    if (!arrive_last<1>(sq, scratch, part, ticket)) return;
    sq[0] = 0.0;
    run_slice_long_rows<1, 0>(a, chunk, load, epi);
    double longs[1], total[1];
    block_sum<1>(sq, scratch, longs);
    sum_partials<1>(part, gridDim.x, scratch, total);
    if (threadIdx.x == 0) {
      *ticket = 0;
      norm[0] = total[0] + longs[0];
      norm[1] = 1.0 / sqrt(norm[0]);
    }
    return;
  }
  if (a.nlong == 0) return;
  __shared__ int s_last;
  __syncthreads();  // the block's piece partials before thread 0's fence
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  run_slice_long_rows<1, 0>(a, chunk, load, epi);
  if (threadIdx.x == 0) *ticket = 0;
}

// norm[0] = sum v^2, norm[1] = 1 / its root.
__global__ void k_sumsq(const double* v, int count, double* part, double* out,
                        unsigned int* ticket) {
  __shared__ double scratch[kTileThreads / 32];
  double acc[1] = {0.0};
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) {
    acc[0] = fma(v[k], v[k], acc[0]);
  }
  double o[1];
  block_sum<1>(acc, scratch, o);
  __shared__ bool is_last;
  if (threadIdx.x == 0) {
    part[blockIdx.x] = o[0];
    __threadfence();
    is_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  double a[1] = {0.0};
  for (int b = threadIdx.x; b < gridDim.x; b += blockDim.x) a[0] += __ldcg(part + b);
  block_sum<1>(a, scratch, o);
  if (threadIdx.x == 0) {
    out[0] = o[0];
    out[1] = 1.0 / sqrt(o[0]);
    *ticket = 0;
  }
}

__global__ void k_project_start(int n, const double* l, const double* u, double* x) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    x[k] = clamp_box(0.0, l[k], u[k]);
  }
}

__global__ void k_fill(double* v, int count, double value) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) {
    v[k] = value;
  }
}

int elementwise_grid(int count) {
  int blocks = (count + 255) / 256;
  const int cap = device_sms() * 8;
  if (blocks > cap) blocks = cap;
  return blocks < 1 ? 1 : blocks;
}

__global__ void k_gather_values(const double* __restrict__ src, const int* __restrict__ map,
                                float* __restrict__ dst, long long count) {
  for (long long k = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; k < count;
       k += static_cast<long long>(gridDim.x) * blockDim.x) {
    dst[k] = static_cast<float>(src[map[k]]);
  }
}

}  // namespace

bool configure_fp64_kernels() {
  const int dev = current_device();
  if (dev < 0) return false;
  std::lock_guard<std::mutex> lock(g_config_mutex);
  DeviceConfig& c = g_config[dev];
  if (c.configured) return true;
  const cudaError_t errs[] = {
      cudaFuncSetAttribute(k_primal, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           max_dynamic_smem(reinterpret_cast<const void*>(k_primal))),
      cudaFuncSetAttribute(k_dual, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           max_dynamic_smem(reinterpret_cast<const void*>(k_dual))),
      cudaFuncSetAttribute(k_room, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           max_dynamic_smem(reinterpret_cast<const void*>(k_room))),
      cudaFuncSetAttribute(k_pdhg_resident, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           max_dynamic_smem(reinterpret_cast<const void*>(k_pdhg_resident))),
      cudaFuncSetAttribute(k_pdhg_resident, cudaFuncAttributeNonPortableClusterSizeAllowed, 1),
      cudaFuncSetAttribute(k_resident_setup, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           max_dynamic_smem(reinterpret_cast<const void*>(k_resident_setup))),
      cudaFuncSetAttribute(k_resident_setup, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)};
  for (cudaError_t e : errs) {
    if (e != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
  }
  c.configured = true;
  return true;
}

long long kernel_launch_count() { return g_launches; }

int fp64_window_capacity(int pass) {
  configure_fp64_kernels();
  return pass == 0
             ? window_capacity(reinterpret_cast<const void*>(k_primal), kSliceBarBytes,
                               sizeof(double))
             : window_capacity(reinterpret_cast<const void*>(k_dual), kSliceBarBytes,
                               sizeof(double));
}

void launch_primal_pass(const StepBuffers& b, cudaStream_t s) {
  // As many threads as k_pdhg_steps has, so that the warps' slices, and every sum, are the same.
  launch_after(k_primal, b.csc.grid, kSliceThreads, slice_smem<double>(b.csc.wmax), s, b);
  ++g_launches;
}

void launch_dual_pass(const StepBuffers& b, cudaStream_t s) {
  launch_after(k_dual, b.csr.grid, kSliceThreads, slice_smem<double>(b.csr.wmax), s, b);
  ++g_launches;
}

int resident_threads(const StepBuffers& b) {
  return std::min(kResidentThreads, std::max(b.csc.threads, b.csr.threads));
}

void launch_resident_setup(const ResidentSetup& r, int threads, int smem, cudaStream_t s) {
  ++g_launches;
  launch_cluster(k_resident_setup, r.scaling.csc.grid, threads, smem, s, r);
}

int resident_smem(int m, int n, int col_rows, int col_slices, int row_rows, int row_slices) {
  return 16 * n + 16 * m + local_slices_bytes(col_rows, col_slices) +
         local_slices_bytes(row_rows, row_slices) + 32 + 8 * 32 * (6 * col_slices + 3 * row_slices);
}

bool resident_fits(const StepBuffers& b, int smem) {
  return b.csc.grid == b.csr.grid &&
         smem <= max_dynamic_smem(reinterpret_cast<const void*>(k_pdhg_resident)) &&
         smem <= max_dynamic_smem(reinterpret_cast<const void*>(k_resident_setup)) &&
         cluster_fits(k_pdhg_resident, b.csc.grid, resident_threads(b), smem) &&
         cluster_fits(k_resident_setup, b.csc.grid, resident_threads(b), smem);
}

void launch_pdhg_resident(const StepBuffers& b, int attempts, int smem, cudaStream_t s) {
  ++g_launches;
  launch_cluster(k_pdhg_resident, b.csc.grid, resident_threads(b), smem, s, b, attempts);
}

void launch_load_passes(cudaStream_t s) {
  g_launches += 2;
  k_primal<<<1, 32, 0, s>>>(StepBuffers{});
  k_dual<<<1, 32, 0, s>>>(StepBuffers{});
}

void launch_room(unsigned long long* span, int sms, cudaStream_t s) {
  configure_fp64_kernels();
  ++g_launches;
  cudaMemsetAsync(span, 0, 2 * sizeof(unsigned long long), s);
  k_room<<<sms, 1, max_dynamic_smem(reinterpret_cast<const void*>(k_room)), s>>>(span);
}

bool crowded(const unsigned long long* span) {
  return span[1] - ~span[0] >= static_cast<unsigned long long>(kRoomStay / 2);
}

bool pdhg_steps_fit(const StepBuffers& b) {
  return grid_fits(k_pdhg_steps, std::max(b.csc.grid, b.csr.grid), kSliceThreads, 0);
}

void launch_pdhg_steps(const StepBuffers& b, int attempts, cudaStream_t s) {
  ++g_launches;
  launch_grid(k_pdhg_steps, std::max(b.csc.grid, b.csr.grid), kSliceThreads, 0, s, b, attempts);
}

void launch_pdhg_step(const StepBuffers& b, cudaStream_t s) {
  launch_primal_pass(b, s);
  launch_dual_pass(b, s);
}

void launch_gather_values(const double* src, const int* map, float* dst, long long count,
                          cudaStream_t s) {
  if (count <= 0) return;
  ++g_launches;
  k_gather_values<<<elementwise_grid(static_cast<int>(std::min<long long>(count, 1 << 30))),
                           256, 0, s>>>(src, map, dst, count);
}

void launch_evaluation(const EvalBuffers& e, cudaStream_t s) {
  g_launches += 4;
  k_eval_rows0<<<e.grid_rows, kTileThreads, 0, s>>>(e);
  k_eval_cols<<<e.grid_cols, e.csc.threads, 0, s>>>(e);
  k_eval_rows1<<<e.grid_rows, e.csr.threads, 0, s>>>(e);
  const int total = e.m > e.n ? e.m : e.n;
  k_eval_apply<<<elementwise_grid(total), 256, 0, s>>>(e);
}

int scale_blocks(const SliceSet& S) {
  return (S.nslices + kScaleThreads / 32 - 1) / (kScaleThreads / 32) + S.nitems;
}

namespace {

template <int MODE, bool APPLY>
void scale_round(const ScaleArgs& a, cudaStream_t s) {
  const int grid = scale_blocks(a.S);
  if (grid == 0) return;
  ++g_launches;
  k_scale_round<MODE, APPLY><<<grid, kScaleThreads, 0, s>>>(a);
}

}  // namespace

void launch_scaling(const ScalingBuffers& b, cudaStream_t s) {
  // Factors of the raw values, then 11 rounds: ten Ruiz rounds and the Pock-Chambolle round
  // apply factors; each takes the next round's, the last none.
  const auto args = [&](int side, int round) {
    ScaleArgs a{};
    a.S = side ? b.csc : b.csr;
    a.in = round <= 0 ? (side ? b.csc_raw : b.csr_raw) : (side ? b.csc_val : b.csr_val);
    a.out = side ? b.csc_val : b.csr_val;
    const int now = round & 1, then = now ^ 1;
    a.line = side ? b.col_factor[now] : b.row_factor[now];
    a.other = side ? b.row_factor[now] : b.col_factor[now];
    a.next = side ? b.col_factor[then] : b.row_factor[then];
    a.scale = side ? b.dc : b.dr;
    a.line_is_row = side ? 0 : 1;
    return a;
  };
  for (int side = 0; side < 2; ++side) {
    ScaleArgs a = args(side, -1);  // next = the factors of round 0
    scale_round<kScaleMax, false>(a, s);
  }
  for (int round = 0; round < 11; ++round) {
    for (int side = 0; side < 2; ++side) {
      ScaleArgs a = args(side, round);
      if (round < 9) {
        scale_round<kScaleMax, true>(a, s);
      } else if (round == 9) {
        scale_round<kScaleSum, true>(a, s);
      } else {
        a.minmax = side ? b.minmax : nullptr;
        scale_round<kScaleNone, true>(a, s);
      }
    }
  }
  ++g_launches;
  k_minmax_final<<<1, kScaleThreads, 0, s>>>(b.minmax, scale_blocks(b.csc), b.nnz, b.minmax_out);
}

void launch_slice_fill(const SliceSet& S, const int* ptr, const int* idx, const double* val,
                       int* sidx, double* sval, cudaStream_t s) {
  const int warps = S.nslices + S.nitems;
  if (warps == 0) return;
  ++g_launches;
  k_slice_copy<false><<<(warps + 7) / 8, 256, 0, s>>>(S, ptr, const_cast<int*>(idx),
                                                      const_cast<double*>(val), sidx, sval);
}

void launch_slice_unfill(const SliceSet& S, const int* ptr, const double* sval, double* val,
                         cudaStream_t s) {
  const int warps = S.nslices + S.nitems;
  if (warps == 0) return;
  ++g_launches;
  k_slice_copy<true><<<(warps + 7) / 8, 256, 0, s>>>(S, ptr, nullptr, val, nullptr,
                                                     const_cast<double*>(sval));
}

void launch_scale_vectors(int m, int n, const double* cost, const double* l, const double* u,
                          const double* rl, const double* ru, const double* dr, const double* dc,
                          double* cs, double* ls, double* us, double* rls, double* rus,
                          cudaStream_t s) {
  ++g_launches;
  k_scale_vectors<<<elementwise_grid(m > n ? m : n), 256, 0, s>>>(m, n, cost, l, u, rl, ru, dr, dc,
                                                                  cs, ls, us, rls, rus);
}

__global__ void k_step_factors(double2* table, long long n) {
  for (long long e = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; e < n;
       e += static_cast<long long>(gridDim.x) * blockDim.x) {
    table[e] = step_factors(step_factor_index(e - 1));
  }
}

void launch_step_factors(double2* table, long long n, cudaStream_t s) {
  if (n <= 0) return;
  ++g_launches;
  k_step_factors<<<std::max(1, device_sms()) * 8, 256, 0, s>>>(table, n);
}

namespace {

// A product combines its rows of several pieces in its last block. Their counters are the step
// kernels', which may run beside a product on another stream: it leaves them alone.
SliceSet without_tickets(SliceSet a) {
  a.tickets = nullptr;
  return a;
}

}  // namespace

void launch_spmv(const SliceSet& layout, const double* x, double* y, double* chunk,
                 unsigned int* ticket, cudaStream_t s) {
  const SliceSet a = without_tickets(layout);
  if (a.nrows == 0) return;
  ++g_launches;
  k_spmv<false, false><<<a.grid, a.threads, 0, s>>>(a, x, y, chunk, ticket, nullptr, nullptr,
                                                    nullptr);
}

void launch_spmv_scaled(const SliceSet& layout, const double* x, double* y, double* chunk,
                        unsigned int* ticket, const double* by, cudaStream_t s) {
  const SliceSet a = without_tickets(layout);
  ++g_launches;
  k_spmv<true, false><<<a.grid, a.threads, 0, s>>>(a, x, y, chunk, ticket, by, nullptr, nullptr);
}

void launch_spmv_norm(const SliceSet& layout, const double* x, double* y, double* chunk,
                      unsigned int* ticket, double* part, double* norm, cudaStream_t s) {
  const SliceSet a = without_tickets(layout);
  ++g_launches;
  k_spmv<false, true><<<a.grid, a.threads, 0, s>>>(a, x, y, chunk, ticket, nullptr, part, norm);
}

namespace {

// The allocation-free product's scratch: file-scope device arrays, never cudaMalloc'd.
// g_noalloc_ticket[0] is the product's completion counter.
static __device__ __align__(256) double g_noalloc_chunks[kNoAllocMaxChunks];
static __device__ __align__(256) unsigned int g_noalloc_ticket[4];

constexpr int kNoAllocMaxDevices = 64;
struct NoAllocSlot {
  bool ready;
  double* chunks;
  unsigned int* ticket;
};
std::mutex g_noalloc_mutex;
NoAllocSlot g_noalloc_slots[kNoAllocMaxDevices];

}  // namespace

cudaError_t noalloc_scratch(int device, cudaStream_t s, double** chunks, unsigned int** ticket) {
  if (device < 0 || device >= kNoAllocMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  NoAllocSlot& slot = g_noalloc_slots[device];
  if (!slot.ready) {
    cudaError_t err = cudaSetDevice(device);
    if (err != cudaSuccess) return err;
    void* c = nullptr;
    void* t = nullptr;
    err = cudaGetSymbolAddress(&c, g_noalloc_chunks);
    if (err != cudaSuccess) return err;
    err = cudaGetSymbolAddress(&t, g_noalloc_ticket);
    if (err != cudaSuccess) return err;
    // The completion counter must start at zero; k_spmv's last block puts it back to zero.
    // The chunk partials need no clearing: each is written before it is read.
    err = cudaMemsetAsync(t, 0, sizeof(g_noalloc_ticket), s);
    if (err != cudaSuccess) return err;
    err = cudaStreamSynchronize(s);
    if (err != cudaSuccess) return err;
    slot.chunks = static_cast<double*>(c);
    slot.ticket = static_cast<unsigned int*>(t);
    slot.ready = true;
  }
  *chunks = slot.chunks;
  *ticket = slot.ticket;
  return cudaSuccess;
}

void launch_sumsq(const double* v, int count, double* part, double* out, unsigned int* ticket,
                  cudaStream_t s, int grid) {
  ++g_launches;
  k_sumsq<<<grid, kTileThreads, 0, s>>>(v, count, part, out, ticket);
}

void launch_project_start(int n, const double* l, const double* u, double* x, cudaStream_t s) {
  ++g_launches;
  k_project_start<<<elementwise_grid(n), 256, 0, s>>>(n, l, u, x);
}

void launch_fill(double* v, int count, double value, cudaStream_t s) {
  if (count <= 0) return;
  ++g_launches;
  k_fill<<<elementwise_grid(count), 256, 0, s>>>(v, count, value);
}

}  // namespace sgb
