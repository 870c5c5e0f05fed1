// qp_kernels.cu -- kernels of the convex-QP engine (layout and schedule in qp.cuh).
//
// Arithmetic follows src/qp/qp_condat_vu.cpp:257-326 term by term. The element-wise steps
// round as the reference's do; the sums over a row or column accumulate with FMA in a fixed
// order (the entries' order for one lane, then a fixed tree over the lanes and over the chunks
// of a long item), which differs from the reference's sequential sums by a few ulps.
//
// GB300 retires about two FP64 lane operations per clock per SM, and these passes are bound
// by that pipe rather than by HBM: the per-item epilogue costs as much as a dozen entries of
// the sums. So the epilogues are written for few FP64 instructions, each with the reference's
// rounding:
//   - absent bounds are stored as -inf / +inf (the load maps every bound that
//     is_finite_bound calls absent), so the projection is two compares;
//   - the cost and Q are stored times the sense (exact), so the gradient
//     (sense c + sense Qx) + A'y is two additions with the same bits;
//   - 2 x' - x is one FMA (2 x' is exact);
//   - v / sigma is divide() (common.cuh), the correctly rounded quotient from the reciprocal;
//   - the projections compare on the integer units (clamp_box_or_nan).
#include "qp.cuh"

#include <algorithm>

#include "chunks.cuh"

namespace sgb {
namespace {

long long g_qp_launches = 0;

// The gradient of the minimisation-space objective, (sense c + sense (Qx)_j) + (A'y)_j, from
// the stored sense c and the sum over sense Q.
__device__ __forceinline__ double qp_gradient(double cmin, double qxmin, double aty) {
  return __dadd_rn(__dadd_rn(cmin, qxmin), aty);
}

// proj_[lo, hi](v) for bounds stored with absent sides as infinities: the reference's project
// (src/qp/qp_condat_vu.cpp:60-64), a NaN left as it is.
__device__ __forceinline__ double box(double v, double lo, double hi) {
  return clamp_box_or_nan(v, lo, hi);
}

// A residual into a running maximum held as the bit pattern of a non-negative double (the
// order of such patterns is the order of the values). A NaN is left out, as std::max(a, NaN)
// leaves a in the reference's loops.
__device__ __forceinline__ void max_bits(unsigned long long* slot, double v) {
  if (v > 0.0) atomicMax(slot, static_cast<unsigned long long>(__double_as_longlong(v)));
}

// The skip test of every step and check kernel: nothing once the stopping test held, nothing
// past the iteration limit. Uniform over the grid (ctl changes only between kernels).
__device__ __forceinline__ bool qp_skip(const QpCtl* ctl, int k) {
  const volatile QpCtl* c = ctl;
  return c->done != 0 || c->base + k + 1 > c->limit;
}

// ---- One-lane sums ------------------------------------------------------------------------
// sum over entries [b, e) of values[q] * vec[index[q]], in entry order, FMA-accumulated onto
// acc. Pairs of entries from an even position on are read as one double2 and one int2 (the
// arrays come from cudaMalloc, so an even position is 16- and 8-byte aligned): two memory
// instructions fewer per pair, the same sum in the same order.
__device__ __forceinline__ double seq_dot(const double* values, const int* index,
                                          const double* vec, int b, int e, double acc) {
  int q = b;
  if ((q & 1) && q < e) {
    acc = fma(values[q], vec[index[q]], acc);
    ++q;
  }
  for (; q + 1 < e; q += 2) {
    const double2 vv = *reinterpret_cast<const double2*>(values + q);
    const int2 ii = *reinterpret_cast<const int2*>(index + q);
    acc = fma(vv.x, vec[ii.x], acc);
    acc = fma(vv.y, vec[ii.y], acc);
  }
  if (q < e) acc = fma(values[q], vec[index[q]], acc);
  return acc;
}

// ---- Staged one-lane sums ----------------------------------------------------------------
// A warp's 32 consecutive items own one contiguous slice of each matrix array. The warp copies
// the slice into its part of shared memory with coalesced loads, then each lane sums its own
// item there in entry order: the same sums, in the same order, as the direct one-lane loop.
// A lane with no item (past the end, or a long item of the chunked path) passes an empty
// range. All 32 lanes must call.

__device__ __forceinline__ void stage_slice(const double* values, const int* index, int begin,
                                            int count, double* sv, int* si) {
  const int lane = threadIdx.x & 31;
#pragma unroll 4
  for (int k = lane; k < count; k += 32) {
    sv[k] = __ldg(values + begin + k);
    si[k] = __ldg(index + begin + k);
  }
}

__device__ __forceinline__ double* stage_values() {
  extern __shared__ __align__(16) unsigned char qp_smem[];
  return reinterpret_cast<double*>(qp_smem) + (threadIdx.x >> 5) * kQpStage;
}

__device__ __forceinline__ int* stage_index() {
  extern __shared__ __align__(16) unsigned char qp_smem[];
  return reinterpret_cast<int*>(qp_smem + kQpWarps * kQpStage * sizeof(double)) +
         (threadIdx.x >> 5) * kQpStage;
}

// (A v)_i over row i's entries [b, e) of the CSR.
__device__ __forceinline__ double staged_row_sum(const QpDev& d, const double* v, int i, int b,
                                                 int e) {
  const int lane = threadIdx.x & 31;
  const int r0 = i - lane;
  int wb = 0, we = 0;
  if (r0 < d.m) {
    wb = d.a_rs[r0];
    we = d.a_rs[min(r0 + 32, d.m)];
  }
  double ax = 0.0;
  if (we - wb <= kQpStage) {
    double* sv = stage_values();
    int* si = stage_index();
    stage_slice(d.a_rv, d.a_ci, wb, we - wb, sv, si);
    __syncwarp();
    for (int q = b - wb; q < e - wb; ++q) ax = fma(sv[q], v[si[q]], ax);
  } else {
    for (int q = b; q < e; ++q) ax = fma(d.a_rv[q], v[d.a_ci[q]], ax);
  }
  return ax;
}

// (Q x)_j over row j of Q's entries [qb, qe) and (A'y)_j over column j of A's [ab, ae).
__device__ __forceinline__ void staged_column_sums(const QpDev& d, const double* x, int j, int qb,
                                                   int qe, int ab, int ae, double* qx,
                                                   double* aty) {
  const int lane = threadIdx.x & 31;
  const int c0 = j - lane;
  int qwb = 0, qwe = 0, awb = 0, awe = 0;
  if (c0 < d.n) {
    const int cn = min(c0 + 32, d.n);
    qwb = d.q_rs[c0];
    qwe = d.q_rs[cn];
    awb = d.a_cs[c0];
    awe = d.a_cs[cn];
  }
  const int lq = qwe - qwb, la = awe - awb;
  double sq = 0.0, sa = 0.0;
  if (lq + la <= kQpStage) {
    double* sv = stage_values();
    int* si = stage_index();
    stage_slice(d.q_v, d.q_ci, qwb, lq, sv, si);
    stage_slice(d.a_cv, d.a_ri, awb, la, sv + lq, si + lq);
    __syncwarp();
    for (int q = qb - qwb; q < qe - qwb; ++q) sq = fma(sv[q], x[si[q]], sq);
    for (int a = lq + ab - awb; a < lq + ae - awb; ++a) sa = fma(sv[a], d.y[si[a]], sa);
  } else {
    for (int q = qb; q < qe; ++q) sq = fma(d.q_v[q], x[d.q_ci[q]], sq);
    for (int a = ab; a < ae; ++a) sa = fma(d.a_cv[a], d.y[d.a_ri[a]], sa);
  }
  *qx = sq;
  *aty = sa;
}

// ---- Sliced items -----------------------------------------------------------------------------
// A lane's item in slice s: its meta word, unpacked.
struct QpPlace {
  int item, len1, len2;  // item valid where `has`
  bool has;
  __device__ __forceinline__ void set(int s, unsigned m) {
    has = m != kQpNoItem;
    item = (s / (kQpGroup / 32)) * kQpGroup + static_cast<int>(m & 127u);
    len1 = has ? static_cast<int>((m >> 8) & 255u) : 0;
    len2 = has ? static_cast<int>(m >> 16) : 0;
  }
};

__device__ __forceinline__ unsigned qp_meta(const QpSliceSet& S, int s, int s1) {
  return s < s1 ? __ldg(S.meta + static_cast<size_t>(s) * 32 + (threadIdx.x & 31)) : kQpNoItem;
}

// A warp's walk over its block's slices: the slice at hand, and the first piece of what is summed
// next (slices.cuh). PART 0 is the first part and then the second of each slice, 1 and 2 one part.
template <int PART>
struct QpWalk {
  int s, s1;
  QpPlace p;
  size_t at1, at2;
  PieceIndices<kPiece> ix;
  unsigned m;  // of the next slice
  unsigned b1, b2;
  int step;

  __device__ __forceinline__ void fetch(const QpSliceSet& S, int next) {
    m = kQpNoItem;
    b1 = b2 = 0;
    if (next < s1) {
      m = __ldg(S.meta + static_cast<size_t>(next) * 32 + (threadIdx.x & 31));
      if (PART != 2) b1 = __ldg(S.base1 + next);
      if (PART != 1) b2 = __ldg(S.base2 + next);
    }
  }
  __device__ __forceinline__ void unpack() {
    p.set(s, m);
    at1 = static_cast<size_t>(b1) * 32 + (threadIdx.x & 31);
    at2 = static_cast<size_t>(b2) * 32 + (threadIdx.x & 31);
  }
  __device__ __forceinline__ void start(const QpSliceSet& S) {
    step = static_cast<int>(blockDim.x >> 5);
    const bool mine = static_cast<int>(blockIdx.x) < S.blocks;
    s = mine ? __ldg(S.block_start + blockIdx.x) + static_cast<int>(threadIdx.x >> 5) : 0;
    s1 = mine ? __ldg(S.block_start + blockIdx.x + 1) : 0;
    fetch(S, s);
    unpack();
    if (PART == 2) {
      ix.load(S.idx2 + at2, p.len2);
    } else {
      ix.load(S.idx1 + at1, p.len1);
    }
    fetch(S, s + step);
  }
  // The next slice's first piece, once its record has arrived.
  __device__ __forceinline__ void after(const QpSliceSet& S, const int** idx, int* left) const {
    QpPlace n;
    n.set(0, m);
    if (PART == 2) {
      *idx = S.idx2 + static_cast<size_t>(b2) * 32 + (threadIdx.x & 31);
      *left = n.len2;
    } else {
      *idx = S.idx1 + static_cast<size_t>(b1) * 32 + (threadIdx.x & 31);
      *left = n.len1;
    }
  }
  // The item's sums over the parts of PART, FMA-accumulated in entry order, of the vectors that
  // get1(c) and get2(c) read.
  template <typename Get1, typename Get2>
  __device__ __forceinline__ void sums(const QpSliceSet& S, Get1 get1, Get2 get2, double* sum1,
                                       double* sum2) {
    const int* ni;
    int nl;
    after(S, &ni, &nl);
    double a1 = 0.0, a2 = 0.0;
    if (PART != 2) {
      slice_sum<double>(S.idx1 + at1, S.val1 + at1, p.len1, __reduce_max_sync(0xffffffffu, p.len1),
                        ix, PART == 0 ? S.idx2 + at2 : ni, PART == 0 ? p.len2 : nl,
                        get1, [&](double v, double g) { a1 = fma(v, g, a1); });
    }
    if (PART != 1) {
      slice_sum<double>(S.idx2 + at2, S.val2 + at2, p.len2, __reduce_max_sync(0xffffffffu, p.len2),
                        ix, ni, nl, get2, [&](double v, double g) { a2 = fma(v, g, a2); });
    }
    *sum1 = a1;
    *sum2 = a2;
  }
  __device__ __forceinline__ void advance(const QpSliceSet& S) {
    s += step;
    unpack();
    fetch(S, s + step);
  }
};

// ---- Column pass ------------------------------------------------------------------------

// A gathered entry: of a vector that the running kernel does not write, or of one that it does.
template <bool LIVE>
__device__ __forceinline__ double gathered(const double* p) {
  return LIVE ? ld_live(p) : __ldg(p);
}

// The epilogue's operands of column j.
struct ColumnOps {
  double x, c, lower, upper;
  __device__ __forceinline__ void load(const QpDev& d, const double* xv, int j) {
    x = xv[j];
    c = d.cost[j];
    lower = d.col_lower[j];
    upper = d.col_upper[j];
  }
};

// The epilogue of column j, run by one lane. Returns the check's residual (check form) and the
// objective term c_j x_j + 0.5 x_j (Qx)_j (check and report forms).
template <int MODE>
__device__ __forceinline__ void column_epilogue(const QpDev& d, double tau, int j,
                                                const ColumnOps& o, double* xn, double qx,
                                                double aty, double* residual, double* obj) {
  const double xj = o.x;
  const double c = o.c;  // sense c; qx is (sense Q x)_j
  if (MODE == kQpStep) {
    const double g = qp_gradient(c, qx, aty);
    const double t = __dsub_rn(xj, __dmul_rn(tau, g));
    const double xnj = box(t, o.lower, o.upper);
    xn[j] = xnj;
    d.xbar[j] = fma(2.0, xnj, -xj);
  } else {
    if (MODE == kQpCheck) {
      const double g = qp_gradient(c, qx, aty);
      const double stepped = box(__dsub_rn(xj, g), o.lower, o.upper);
      *residual = fabs(__dsub_rn(xj, stepped));
    } else {
      // c + Qx = sense (sense c + sense Qx), exactly.
      d.col_dual[j] =
          __dadd_rn(__dmul_rn(d.sense, __dadd_rn(c, qx)), __dmul_rn(d.sense, aty));
    }
    *obj = d.sense * (c * xj + 0.5 * xj * qx);
  }
}

// The sum over entries [from, to) of values[e] * vec[index[e]], in every lane: lane l takes entries l,
// l + 32, ... (The compiler's unrolled loop: batches with predicated ends were slower, 23.4
// against 21.4 us an iteration of 5,000 Zipf rows in chunks of 2,048.)
template <bool LIVE>
__device__ __forceinline__ double chunk_sum(const double* values, const int* index,
                                            const double* vec, int from, int to) {
  if (from >= to) return 0.0;
  double sum = 0.0;
#pragma unroll 4
  for (int e = from + static_cast<int>(threadIdx.x & 31); e < to; e += 32) {
    sum = fma(values[e], gathered<LIVE>(vec + index[e]), sum);
  }
  return warp_sum(sum);
}

// The sum of the partials of ch's item, in every lane of the warp that brought the last.
__device__ __forceinline__ double2 chunk_total(const double2* part, const QpChunk& ch) {
  __threadfence();
  double2 sum = make_double2(0.0, 0.0);
  for (int c = ch.first + static_cast<int>(threadIdx.x & 31); c < ch.first + ch.count; c += 32) {
    const double2 p = __ldcg(&part[c]);
    sum.x += p.x;
    sum.y += p.y;
  }
  return make_double2(warp_sum(sum.x), warp_sum(sum.y));
}

// Long columns: one warp per chunk of the column's entries (row j of Q, then column j of A); the
// last chunk of a column to finish adds the chunks' sums in order and runs its epilogue. LIVE: the
// vectors are the running kernel's own (ld_live).
template <int MODE, bool LIVE>
__device__ __forceinline__ void long_column(const QpDev& d, QpCtl* ctl, double tau, int w,
                                            const double* x, double* xn) {
  const int lane32 = threadIdx.x & 31;
  const QpChunk ch = d.col_chunks[w];
  const int j = ch.item;
  const int qb = d.q_rs[j], lq = d.q_rs[j + 1] - qb, ab = d.a_cs[j];
  double qx = chunk_sum<LIVE>(d.q_v, d.q_ci, x, qb + ch.begin, qb + min(ch.end, lq));
  double aty = chunk_sum<LIVE>(d.a_cv, d.a_ri, d.y, ab + max(ch.begin - lq, 0), ab + ch.end - lq);
  int last = 1;
  if (ch.count > 1) {
    if (lane32 == 0) {
      __stcg(&d.chunk_part[w], make_double2(qx, aty));
      __threadfence();
      last = atomicAdd(&d.col_tickets[ch.slot], 1u) == static_cast<unsigned>(ch.count - 1);
    }
    last = __shfl_sync(0xffffffffu, last, 0);
    if (!last) return;
    const double2 all = chunk_total(d.chunk_part, ch);
    qx = all.x;
    aty = all.y;
    if (lane32 == 0) d.col_tickets[ch.slot] = 0u;
  }
  if (lane32 == 0) {
    double residual = 0.0, obj = 0.0;
    ColumnOps o;
    o.load(d, x, j);
    column_epilogue<MODE>(d, tau, j, o, xn, qx, aty, &residual, &obj);
    if (MODE == kQpCheck) max_bits(&ctl->dual_bits, residual);
    if (MODE != kQpStep) d.long_col_obj[ch.slot] = obj;
  }
}

// The step form of the block's columns on sliced items.
template <int MODE, bool LIVE>
__device__ __forceinline__ void sliced_columns(const QpDev& d, QpWalk<0>& walk, double tau,
                                               const double* x, double* xn, double* residual,
                                               double* obj) {
  for (; walk.s < walk.s1; walk.advance(d.cols)) {
    const QpPlace p = walk.p;
    ColumnOps o;
    if (p.has) o.load(d, x, p.item);
    double qx, aty, r = 0.0, t = 0.0;
    walk.sums(d.cols, [&](int c) { return gathered<LIVE>(x + c); },
              [&](int c) { return gathered<LIVE>(d.y + c); }, &qx, &aty);
    if (p.has) column_epilogue<MODE>(d, tau, p.item, o, xn, qx, aty, &r, &t);
    if (MODE != kQpStep) {
      *residual = r > *residual ? r : *residual;
      *obj += t;
    }
  }
}

// G = 0: the short columns on sliced items, in blocks of kQpSliceThreads.
template <int G>
constexpr int qp_threads() {
  return G == 0 ? kQpSliceThreads : kQpThreads;
}

template <int G, int MODE>
__global__ void __launch_bounds__(qp_threads<G>()) k_qp_column(QpDev d, QpCtl* ctl, int k, int src) {
  if (ctl == nullptr) return;  // qp_launch_load_passes
  // The first entries are under way before the wait: no kernel of the solve writes the matrix.
  QpWalk<0> walk;
  if (G == 0) walk.start(d.cols);
  grid_dependency_launch();
  grid_dependency_wait();
  if (MODE != kQpReport && qp_skip(ctl, k)) return;
  const double tau = ctl->tau;
  const double* x = src ? d.x1 : d.x0;
  double* xn = src ? d.x0 : d.x1;
  const int lane32 = threadIdx.x & 31;
  if (G == 0 && static_cast<int>(blockIdx.x) < d.col_short_blocks) {
    double residual = 0.0, obj = 0.0;
    sliced_columns<MODE, false>(d, walk, tau, x, xn, &residual, &obj);
    if (MODE != kQpStep) {
      __shared__ double scratch[kQpSliceThreads / 32];
      if (MODE == kQpCheck) {
        const double w = warp_max(residual);
        if (lane32 == 0) max_bits(&ctl->dual_bits, w);
      }
      double v[1] = {obj}, total[1];
      block_sum<1>(v, scratch, total);
      if (threadIdx.x == 0) d.obj_part[blockIdx.x] = total[0];
    }
    return;
  }
  if (G > 0 && static_cast<int>(blockIdx.x) < d.col_short_blocks) {
    // Short columns: G lanes per column, in column order.
    constexpr int kG = G > 0 ? G : 1;
    const int gid = static_cast<int>(blockIdx.x) * kQpThreads + static_cast<int>(threadIdx.x);
    const int j = gid / kG, lane = gid % kG;
    int qb = 0, qe = 0, ab = 0, ae = 0;
    bool active = j < d.n;
    if (active) {
      qb = d.q_rs[j];
      qe = d.q_rs[j + 1];
      ab = d.a_cs[j];
      ae = d.a_cs[j + 1];
      if ((qe - qb) + (ae - ab) > kQpLongPerLane * kG) {  // a long column: the chunk path's
        active = false;
        qb = qe = ab = ae = 0;
      }
    }
    double qx = 0.0, aty = 0.0;
    if (G == 1 && d.stage) {
      staged_column_sums(d, x, j, qb, qe, ab, ae, &qx, &aty);
    } else if (G == 1) {
      qx = seq_dot(d.q_v, d.q_ci, x, qb, qe, 0.0);
      aty = seq_dot(d.a_cv, d.a_ri, d.y, ab, ae, 0.0);
    } else {
      for (int e = qb + lane; e < qe; e += kG) qx = fma(d.q_v[e], x[d.q_ci[e]], qx);
      for (int e = ab + lane; e < ae; e += kG) aty = fma(d.a_cv[e], d.y[d.a_ri[e]], aty);
      qx = group_sum<kG>(qx);
      aty = group_sum<kG>(aty);
    }
    double residual = 0.0, obj = 0.0;
    if (active && lane == 0) {
      ColumnOps o;
      o.load(d, x, j);
      column_epilogue<MODE>(d, tau, j, o, xn, qx, aty, &residual, &obj);
    }
    if (MODE != kQpStep) {
      __shared__ double scratch[kQpThreads / 32];
      if (MODE == kQpCheck) {
        const double w = warp_max(residual);
        if (lane32 == 0) max_bits(&ctl->dual_bits, w);
      }
      double v[1] = {obj}, total[1];
      block_sum<1>(v, scratch, total);
      if (threadIdx.x == 0) d.obj_part[blockIdx.x] = total[0];
    }
    return;
  }
  const int w = (static_cast<int>(blockIdx.x) - d.col_short_blocks) * (qp_threads<G>() / 32) +
                static_cast<int>(threadIdx.x >> 5);
  if (w < d.ncol_chunks) long_column<MODE, false>(d, ctl, tau, w, x, xn);
}

// ---- Row pass ---------------------------------------------------------------------------

// The epilogue's operands of row i.
struct RowOps {
  double y, lower, upper;
  __device__ __forceinline__ void load(const QpDev& d, int i) {
    y = d.y[i];
    lower = d.row_lower[i];
    upper = d.row_upper[i];
  }
};

// y' = v - sigma proj(v / sigma), v = y + sigma (A xbar)_i (src/qp/qp_condat_vu.cpp:270-276).
__device__ __forceinline__ double row_step(double sigma, double inv_sigma, const RowOps& o,
                                           double ax) {
  const double v = __dadd_rn(o.y, __dmul_rn(sigma, ax));
  const double p = box(divide(v, sigma, inv_sigma), o.lower, o.upper);
  return __dsub_rn(v, __dmul_rn(sigma, p));
}

template <int MODE>
__device__ __forceinline__ double row_epilogue(const QpDev& d, double sigma, double inv_sigma,
                                               int i, const RowOps& o, double ax) {
  if (MODE == kQpStep) {
    d.y[i] = row_step(sigma, inv_sigma, o, ax);
    return 0.0;
  }
  const double projected = box(ax, o.lower, o.upper);
  return fabs(__dsub_rn(ax, projected));
}

// Long rows, a warp per chunk, as the long columns.
template <int MODE, bool LIVE>
__device__ __forceinline__ void long_row(const QpDev& d, QpCtl* ctl, double sigma, double inv_sigma,
                                         int w, const double* v) {
  const int lane32 = threadIdx.x & 31;
  const QpChunk ch = d.row_chunks[w];
  const int i = ch.item, b = d.a_rs[i];
  double ax = chunk_sum<LIVE>(d.a_rv, d.a_ci, v, b + ch.begin, b + ch.end);
  int last = 1;
  if (ch.count > 1) {
    if (lane32 == 0) {
      __stcg(&d.row_chunk_part[w], make_double2(ax, 0.0));
      __threadfence();
      last = atomicAdd(&d.row_tickets[ch.slot], 1u) == static_cast<unsigned>(ch.count - 1);
    }
    last = __shfl_sync(0xffffffffu, last, 0);
    if (!last) return;
    ax = chunk_total(d.row_chunk_part, ch).x;
    if (lane32 == 0) d.row_tickets[ch.slot] = 0u;
  }
  if (lane32 == 0) {
    RowOps o;
    o.load(d, i);
    const double residual = row_epilogue<MODE>(d, sigma, inv_sigma, i, o, ax);
    if (MODE == kQpCheck) max_bits(&ctl->primal_bits, residual);
  }
}

// The block's rows on sliced items; returns this thread's largest residual (check form).
template <int MODE, bool LIVE>
__device__ __forceinline__ double sliced_rows(const QpDev& d, QpWalk<2>& walk, double sigma,
                                              double inv_sigma, const double* v) {
  double residual = 0.0;
  for (; walk.s < walk.s1; walk.advance(d.rows)) {
    const QpPlace p = walk.p;
    RowOps o;
    if (p.has) o.load(d, p.item);
    double none, ax;
    walk.sums(d.rows, [](int) { return 0.0; }, [&](int c) { return gathered<LIVE>(v + c); }, &none,
              &ax);
    if (p.has) {
      const double r = row_epilogue<MODE>(d, sigma, inv_sigma, p.item, o, ax);
      residual = r > residual ? r : residual;
    }
  }
  return residual;
}

template <int G, int MODE>
__global__ void __launch_bounds__(qp_threads<G>()) k_qp_row(QpDev d, QpCtl* ctl, int k, int src) {
  if (ctl == nullptr) return;  // qp_launch_load_passes
  QpWalk<2> walk;
  if (G == 0) walk.start(d.rows);
  grid_dependency_launch();
  grid_dependency_wait();
  if (qp_skip(ctl, k)) return;
  const double sigma = ctl->sigma, inv_sigma = ctl->inv_sigma;
  const double* v = MODE == kQpStep ? d.xbar : (src ? d.x1 : d.x0);
  const int lane32 = threadIdx.x & 31;
  if (G == 0 && static_cast<int>(blockIdx.x) < d.row_short_blocks) {
    const double residual = sliced_rows<MODE, false>(d, walk, sigma, inv_sigma, v);
    if (MODE == kQpCheck) {
      const double w = warp_max(residual);
      if (lane32 == 0) max_bits(&ctl->primal_bits, w);
    }
    return;
  }
  if (G > 0 && static_cast<int>(blockIdx.x) < d.row_short_blocks) {
    constexpr int kG = G > 0 ? G : 1;
    const int gid = static_cast<int>(blockIdx.x) * kQpThreads + static_cast<int>(threadIdx.x);
    const int i = gid / kG, lane = gid % kG;
    int b = 0, e = 0;
    bool active = i < d.m;
    if (active) {
      b = d.a_rs[i];
      e = d.a_rs[i + 1];
      if (e - b > kQpLongPerLane * kG) {
        active = false;
        b = e = 0;
      }
    }
    double ax = 0.0;
    if (G == 1 && d.stage) {
      ax = staged_row_sum(d, v, i, b, e);
    } else if (G == 1) {
      ax = seq_dot(d.a_rv, d.a_ci, v, b, e, 0.0);
    } else {
      for (int q = b + lane; q < e; q += kG) ax = fma(d.a_rv[q], v[d.a_ci[q]], ax);
      ax = group_sum<kG>(ax);
    }
    double residual = 0.0;
    if (active && lane == 0) {
      RowOps o;
      o.load(d, i);
      residual = row_epilogue<MODE>(d, sigma, inv_sigma, i, o, ax);
    }
    if (MODE == kQpCheck) {
      const double w = warp_max(residual);
      if (lane32 == 0) max_bits(&ctl->primal_bits, w);
    }
    return;
  }
  const int w = (static_cast<int>(blockIdx.x) - d.row_short_blocks) * (qp_threads<G>() / 32) +
                static_cast<int>(threadIdx.x >> 5);
  if (w < d.nrow_chunks) long_row<MODE, false>(d, ctl, sigma, inv_sigma, w, v);
}

// ---- The steps of a period in one launch ---------------------------------------------------------
// Iterations k0 .. of the graph by one cooperative grid: blocks meet between the passes, and each
// warp has its next pass's first entries under way while it waits. A meeting takes 1.6 us of 152
// blocks; between two launches lie the drain of one, the start of the next and its first loads.
// An iteration over uniform rows: 8.9 us at 20,000 x 40,003 (14 us with launches), 14.2 us at 60,000.
__global__ void __launch_bounds__(kQpSliceThreads, 1) k_qp_steps(QpDev d, QpCtl* ctl, int k0,
                                                                 int count) {
  if (ctl->done != 0 || ctl->error != 0) return;
  const long long left = ctl->limit - (ctl->base + k0);
  const int iterations = left < count ? static_cast<int>(left) : count;
  if (iterations <= 0) return;
  const double tau = ctl->tau, sigma = ctl->sigma, inv_sigma = ctl->inv_sigma;
  const int gw = static_cast<int>((threadIdx.x >> 5) * gridDim.x + blockIdx.x);
  const int warps = static_cast<int>((blockDim.x >> 5) * gridDim.x);
  GridMeet grid;
  grid.start(&ctl->arrivals);
  QpWalk<0> cols;
  cols.start(d.cols);
  for (int i = 0; i < iterations; ++i) {
    const bool odd = (k0 + i) & 1;
    const double* x = odd ? d.x1 : d.x0;
    double* xn = odd ? d.x0 : d.x1;
    for (int w = gw; w < d.ncol_chunks; w += warps) {
      long_column<kQpStep, true>(d, ctl, tau, w, x, xn);
    }
    sliced_columns<kQpStep, true>(d, cols, tau, x, xn, nullptr, nullptr);
    if (d.m > 0) {
      QpWalk<2> rows;
      rows.start(d.rows);
      if (!grid.meet(&ctl->error)) return;
      for (int w = gw; w < d.nrow_chunks; w += warps) {
        long_row<kQpStep, true>(d, ctl, sigma, inv_sigma, w, d.xbar);
      }
      sliced_rows<kQpStep, true>(d, rows, sigma, inv_sigma, d.xbar);
    }
    if (i + 1 == iterations) return;
    cols.start(d.cols);
    if (!grid.meet(&ctl->error)) return;
  }
}

// ---- The resident iterations (slices.cuh) ------------------------------------------------------
// The step forms of the two passes, item for item, in one block with everything in shared memory.
// One part of the slices: the entries, indices as 16 bits, and the slices' first entry rows.
struct QpLocal {
  const double* val;
  const unsigned short* idx;
  const int* base;
  __device__ __forceinline__ double dot(int s, int len, const double* v) const {
    const int e = base[s] * 32 + (threadIdx.x & 31);
    double acc = 0.0;
#pragma unroll 4
    for (int q = 0; q < len; ++q) acc = fma(val[e + q * 32], v[idx[e + q * 32]], acc);
    return acc;
  }
};

__device__ __forceinline__ unsigned char* qp_fill_local(const int* idx, const double* val,
                                                        const unsigned* base, int slices,
                                                        unsigned char* mem, QpLocal* out) {
  const int rows = static_cast<int>(base[slices]);
  double* const v = reinterpret_cast<double*>(mem);
  int* const b = reinterpret_cast<int*>(v + rows * 32);
  unsigned short* const i = reinterpret_cast<unsigned short*>(b + ((slices + 4) & ~3));
  const int T = static_cast<int>(blockDim.x), t = static_cast<int>(threadIdx.x);
  for (int k = t; k < rows * 32; k += T) {
    v[k] = val[k];
    i[k] = static_cast<unsigned short>(idx[k]);
  }
  for (int k = t; k <= slices; k += T) b[k] = static_cast<int>(base[k]);
  *out = QpLocal{v, i, b};
  return reinterpret_cast<unsigned char*>(i + ((rows * 32 + 7) & ~7));
}

// A warp holds one slice of columns and one of rows (kQpResidentItems), a lane its column's and its
// row's data in registers.
__global__ void __launch_bounds__(kResidentThreads, 1) k_qp_resident(QpDev d, QpCtl* ctl, int k0,
                                                                     int count, int src) {
  extern __shared__ __align__(16) unsigned char qp_smem[];
  if (ctl->done != 0) return;
  const long long left = ctl->limit - (ctl->base + k0);
  const int iterations = left < count ? static_cast<int>(left) : count;
  if (iterations <= 0) return;
  const double tau = ctl->tau, sigma = ctl->sigma, inv_sigma = ctl->inv_sigma;
  const int T = static_cast<int>(blockDim.x), t = static_cast<int>(threadIdx.x);
  const int warp = t >> 5, m = d.m, n = d.n;
  double* const xs0 = reinterpret_cast<double*>(qp_smem);
  double* const xs1 = xs0 + n;
  double* const xbar = xs0 + 2 * n;
  double* const ys = xs0 + 3 * n;
  for (int j = t; j < n; j += T) {
    xs0[j] = d.x0[j];
    xs1[j] = d.x1[j];
  }
  for (int i = t; i < m; i += T) ys[i] = d.y[i];
  unsigned char* mem = qp_smem + ((3 * n + m) * 8 + 15) / 16 * 16;
  QpLocal q, a, r;
  mem = qp_fill_local(d.cols.idx1, d.cols.val1, d.cols.base1, d.cols.nslices, mem, &q);
  mem = qp_fill_local(d.cols.idx2, d.cols.val2, d.cols.base2, d.cols.nslices, mem, &a);
  if (m > 0) qp_fill_local(d.rows.idx2, d.rows.val2, d.rows.base2, d.rows.nslices, mem, &r);
  QpPlace col, row;
  col.set(warp, qp_meta(d.cols, warp, d.cols.nslices));
  row.set(warp, qp_meta(d.rows, warp, m > 0 ? d.rows.nslices : 0));
  ColumnOps o{0.0, 0.0, 0.0, 0.0};
  if (col.has) o.load(d, src ? d.x1 : d.x0, col.item);
  RowOps w{0.0, 0.0, 0.0};
  if (row.has) w.load(d, row.item);
  __syncthreads();
  for (int i = 0; i < iterations; ++i) {
    const bool odd = (src + i) & 1;
    if (col.has) {
      const double qx = q.dot(warp, col.len1, odd ? xs1 : xs0), aty = a.dot(warp, col.len2, ys);
      const double g = qp_gradient(o.c, qx, aty);
      const double xnj = box(__dsub_rn(o.x, __dmul_rn(tau, g)), o.lower, o.upper);
      (odd ? xs0 : xs1)[col.item] = xnj;
      xbar[col.item] = fma(2.0, xnj, -o.x);
      o.x = xnj;
    }
    __syncthreads();
    if (row.has) {
      w.y = row_step(sigma, inv_sigma, w, r.dot(warp, row.len2, xbar));
      ys[row.item] = w.y;
    }
    __syncthreads();
  }
  for (int j = t; j < n; j += T) {
    d.x0[j] = xs0[j];
    d.x1[j] = xs1[j];
    d.xbar[j] = xbar[j];
  }
  for (int i = t; i < m; i += T) d.y[i] = ys[i];
}

// ---- Decision -----------------------------------------------------------------------------

// Sum of the objective partials in a fixed order (short-path blocks, then the long columns
// by slot), plus the offset. One block.
__device__ double objective_total(const QpDev& d) {
  __shared__ double scratch[kQpThreads / 32];
  double s = 0.0;
  for (int b = static_cast<int>(threadIdx.x); b < d.col_short_blocks; b += kQpThreads) {
    s += d.obj_part[b];
  }
  double v[1] = {s}, total[1];
  block_sum<1>(v, scratch, total);
  double obj = total[0];
  if (threadIdx.x == 0) {
    for (int q = 0; q < d.nlong_cols; ++q) obj += d.long_col_obj[q];
    obj += d.offset;
  }
  return obj;
}

__global__ void __launch_bounds__(kQpThreads) k_qp_decide(QpDev d, QpCtl* ctl, int k, int p) {
  grid_dependency_launch();
  grid_dependency_wait();
  if (qp_skip(ctl, k)) return;
  const double obj = objective_total(d);
  if (threadIdx.x != 0) return;
  const long long t = ctl->base + k + 1;
  const double pr = __longlong_as_double(static_cast<long long>(ctl->primal_bits));
  const double dr = __longlong_as_double(static_cast<long long>(ctl->dual_bits));
  ctl->primal = pr;
  ctl->dual = dr;
  ctl->objective = obj;
  ctl->checked = t;
  d.hist[p] = QpHist{t, pr, dr, obj};
  ctl->primal_bits = 0ull;
  ctl->dual_bits = 0ull;
  // src/qp/qp_condat_vu.cpp:323-326.
  if (pr <= ctl->tolerance && dr <= ctl->tolerance) {
    ctl->done = 1;
    ctl->iterations = t;
  }
}

__global__ void k_qp_objective(QpDev d, QpCtl* ctl) {
  grid_dependency_launch();
  grid_dependency_wait();
  const double obj = objective_total(d);
  if (threadIdx.x == 0) ctl->objective = obj;
}

__global__ void k_qp_advance(QpCtl* ctl, int graph_iterations) {
  grid_dependency_launch();
  grid_dependency_wait();
  if (ctl->done) return;
  const long long next = ctl->base + graph_iterations;
  ctl->base = next < ctl->limit ? next : ctl->limit;
}

// ---- Setup --------------------------------------------------------------------------------

// The sliced copy of one part, a warp per slice.
__global__ void __launch_bounds__(kQpThreads) k_qp_slice_fill(QpSliceSet S, int part,
                                                              const int* starts, const int* index,
                                                              const double* values, int* idx,
                                                              double* val) {
  const int s = static_cast<int>(blockIdx.x) * kQpWarps + static_cast<int>(threadIdx.x >> 5);
  if (s >= S.nslices) return;
  QpPlace p;
  p.set(s, qp_meta(S, s, S.nslices));
  if (!p.has) return;
  const int len = part == 1 ? p.len1 : p.len2;
  const size_t at =
      static_cast<size_t>(part == 1 ? S.base1[s] : S.base2[s]) * 32 + (threadIdx.x & 31);
  const int from = starts[p.item];
  for (int k = 0; k < len; ++k) {
    idx[at + static_cast<size_t>(k) * 32] = index[from + k];
    val[at + static_cast<size_t>(k) * 32] = values[from + k];
  }
}

// One product of the power iterations (qp_launch_product): the short items on the slices or, without
// them, with `lanes` threads each, and a warp per chunk of a long item; the vector is normalised where an
// item's sum leaves the warp, so no pass over it is spent on that.
template <int SIDE>
__global__ void __launch_bounds__(kQpSliceThreads, 1) k_qp_product(QpDev d, const double* v,
                                                                const double* norm2, double* out,
                                                                int lanes, double* next,
                                                                double* part,
                                                                unsigned int* ticket) {
  __shared__ double scratch[2 * (kQpSliceThreads / 32)];
  __shared__ double s_inv;
  const QpSliceSet& S = SIDE == kQpRows ? d.rows : d.cols;
  const int count = SIDE == kQpRows ? d.m : d.n;
  const int* starts = SIDE == kQpRows ? d.a_rs : (SIDE == kQpCols ? d.a_cs : d.q_rs);
  const int* index = SIDE == kQpRows ? d.a_ci : (SIDE == kQpCols ? d.a_ri : d.q_ci);
  const double* values = SIDE == kQpRows ? d.a_rv : (SIDE == kQpCols ? d.a_cv : d.q_v);
  const int longest = kQpLongPerLane * (SIDE == kQpRows ? d.row_lanes : d.col_lanes);
  QpWalk<SIDE == kQpHessian ? 1 : 2> walk;
  if (S.nslices > 0) walk.start(S);
  if (threadIdx.x == 0) s_inv = norm2 != nullptr ? 1.0 / sqrt(*norm2) : 1.0;
  __syncthreads();
  const double inv = s_inv;
  const int lane = threadIdx.x & 31;
  constexpr int kWarps = kQpSliceThreads / 32;
  const int warps = static_cast<int>(gridDim.x) * kWarps;
  const int warp = static_cast<int>(blockIdx.x) * kWarps + static_cast<int>(threadIdx.x >> 5);
  double acc[2] = {0.0, 0.0};  // sum out^2, sum out (v inv)
  const auto put = [&](int item, double sum) {
    const double o = sum * inv;
    out[item] = o;
    if (next != nullptr) {
      acc[0] = fma(o, o, acc[0]);
      if (SIDE == kQpHessian) acc[1] = fma(o, v[item] * inv, acc[1]);
    }
  };
  if (S.nslices > 0) {
    for (; walk.s < walk.s1; walk.advance(S)) {
      const QpPlace p = walk.p;
      double sum1, sum2;
      walk.sums(S, [&](int c) { return __ldg(v + c); }, [&](int c) { return __ldg(v + c); }, &sum1,
                &sum2);
      if (p.has) put(p.item, SIDE == kQpHessian ? sum1 : sum2);
    }
  } else {
    // Every warp runs the same number of rounds, so its lanes stay together for the sums.
    const int per = 32 / lanes, sub = lane & (lanes - 1);
    for (long long i0 = static_cast<long long>(warp) * per; i0 < count;
         i0 += static_cast<long long>(warps) * per) {
      const int item = static_cast<int>(i0) + lane / lanes;
      double sum = 0.0;
      int all = 0;
      if (item < count) {
        all = starts[item + 1] - starts[item];
        if (SIDE == kQpCols) all += d.q_rs[item + 1] - d.q_rs[item];
        if (SIDE == kQpHessian) all += d.a_cs[item + 1] - d.a_cs[item];
      }
      const bool mine = item < count && all <= longest;
      if (mine) {
        for (int e = starts[item] + sub; e < starts[item + 1]; e += lanes) {
          sum = fma(values[e], v[index[e]], sum);
        }
      }
      for (int o = lanes >> 1; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (mine && sub == 0) put(item, sum);
    }
  }
  // Long items, a warp per chunk, as in the passes; a chunk of a column holds entries of Q, then of A.
  // What the warp that finishes an item adds to the norms goes to the item's own place.
  const QpChunk* chunks = SIDE == kQpRows ? d.row_chunks : d.col_chunks;
  const int nchunks = SIDE == kQpRows ? d.nrow_chunks : d.ncol_chunks;
  double2* chunk_part = SIDE == kQpRows ? d.row_chunk_part : d.chunk_part;
  unsigned int* tickets = SIDE == kQpRows ? d.row_tickets : d.col_tickets;
  for (int c = warp; c < nchunks; c += warps) {
    const QpChunk ch = chunks[c];
    const int lq = SIDE == kQpRows ? 0 : d.q_rs[ch.item + 1] - d.q_rs[ch.item];
    const int from = SIDE == kQpHessian ? ch.begin : max(ch.begin - lq, 0);
    const int to = SIDE == kQpHessian ? min(ch.end, lq) : ch.end - lq;
    const int at = starts[ch.item];
    double sum = chunk_sum<false>(values, index, v, at + from, at + to);
    int last = 0;
    if (lane == 0) {
      __stcg(&chunk_part[c], make_double2(sum, 0.0));
      __threadfence();
      last = atomicAdd(&tickets[ch.slot], 1u) == static_cast<unsigned>(ch.count - 1);
    }
    if (!__shfl_sync(0xffffffffu, last, 0)) continue;
    sum = chunk_total(chunk_part, ch).x;
    if (lane != 0) continue;
    tickets[ch.slot] = 0u;
    const double keep[2] = {acc[0], acc[1]};
    acc[0] = acc[1] = 0.0;
    put(ch.item, sum);
    if (next != nullptr) {
      for (int q = 0; q < 2; ++q) part[2 * (gridDim.x + ch.slot) + q] = acc[q];
    }
    acc[0] = keep[0];
    acc[1] = keep[1];
  }
  if (next == nullptr) return;
  double total[2];
  block_sum<2>(acc, scratch, total);
  __shared__ int s_last;
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = total[0];
    part[2 * blockIdx.x + 1] = total[1];
    __threadfence();
    s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  acc[0] = acc[1] = 0.0;
  const int parts = static_cast<int>(gridDim.x) + (SIDE == kQpRows ? d.nlong_rows : d.nlong_cols);
  for (int b = static_cast<int>(threadIdx.x); b < parts; b += kQpSliceThreads) {
    acc[0] += __ldcg(part + 2 * b);
    acc[1] += __ldcg(part + 2 * b + 1);
  }
  block_sum<2>(acc, scratch, total);
  if (threadIdx.x == 0) {
    next[0] = total[0];
    next[1] = total[1];
    *ticket = 0u;
  }
}

__global__ void __launch_bounds__(kQpThreads) k_qp_dot_partial(const double* a, const double* b,
                                                               int n, double* partials) {
  __shared__ double scratch[kQpThreads / 32];
  double s = 0.0;
  for (int i = static_cast<int>(blockIdx.x) * kQpThreads + static_cast<int>(threadIdx.x); i < n;
       i += kQpDotBlocks * kQpThreads) {
    s = fma(a[i], b[i], s);
  }
  double v[1] = {s}, total[1];
  block_sum<1>(v, scratch, total);
  if (threadIdx.x == 0) partials[blockIdx.x] = total[0];
}

__global__ void __launch_bounds__(kQpThreads) k_qp_dot_final(const double* partials, double* out) {
  __shared__ double scratch[kQpThreads / 32];
  double s = 0.0;
  for (int i = static_cast<int>(threadIdx.x); i < kQpDotBlocks; i += kQpThreads) s += partials[i];
  double v[1] = {s}, total[1];
  block_sum<1>(v, scratch, total);
  if (threadIdx.x == 0) *out = total[0];
}

__global__ void k_qp_row_dual(QpDev d, double* row_dual) {
  for (int i = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x); i < d.m;
       i += static_cast<int>(gridDim.x * blockDim.x)) {
    row_dual[i] = __dmul_rn(-d.sense, d.y[i]);
  }
}

__global__ void k_qp_init(QpDev d) {
  const int stride = static_cast<int>(gridDim.x * blockDim.x);
  for (int j = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x); j < d.n; j += stride) {
    d.x0[j] = box(0.0, d.col_lower[j], d.col_upper[j]);
    d.x1[j] = 0.0;
    d.xbar[j] = 0.0;
  }
  for (int i = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x); i < d.m; i += stride) {
    d.y[i] = 0.0;
  }
}

int grid_for(int n) { return n <= 0 ? 0 : std::min((n + kQpThreads - 1) / kQpThreads, 4096); }

template <int MODE>
void column_pass(const QpDev& d, QpCtl* ctl, int k, int src, cudaStream_t s) {
  const bool sliced = d.cols.nslices > 0;
  const int warps = (sliced ? kQpSliceThreads : kQpThreads) / 32;
  const int grid = d.col_short_blocks + (d.ncol_chunks + warps - 1) / warps;
  if (grid == 0) return;
  const int smem = d.stage ? kQpStageBytes : 0;
  switch (sliced ? 0 : d.col_lanes) {
    case 0:
      launch_after(k_qp_column<0, MODE>, grid, kQpSliceThreads, 0, s, d, ctl, k, src);
      break;
    case 1: launch_after(k_qp_column<1, MODE>, grid, kQpThreads, smem, s, d, ctl, k, src); break;
    case 2: launch_after(k_qp_column<2, MODE>, grid, kQpThreads, 0, s, d, ctl, k, src); break;
    case 4: launch_after(k_qp_column<4, MODE>, grid, kQpThreads, 0, s, d, ctl, k, src); break;
    case 8: launch_after(k_qp_column<8, MODE>, grid, kQpThreads, 0, s, d, ctl, k, src); break;
    case 16: launch_after(k_qp_column<16, MODE>, grid, kQpThreads, 0, s, d, ctl, k, src); break;
    default: launch_after(k_qp_column<32, MODE>, grid, kQpThreads, 0, s, d, ctl, k, src); break;
  }
  ++g_qp_launches;
}

template <int MODE>
void row_pass(const QpDev& d, QpCtl* ctl, int k, int src, cudaStream_t s) {
  const bool sliced = d.rows.nslices > 0;
  const int warps = (sliced ? kQpSliceThreads : kQpThreads) / 32;
  const int grid = d.row_short_blocks + (d.nrow_chunks + warps - 1) / warps;
  if (grid == 0) return;
  const int smem = d.stage ? kQpStageBytes : 0;
  switch (sliced ? 0 : d.row_lanes) {
    case 0:
      launch_after(k_qp_row<0, MODE>, grid, kQpSliceThreads, 0, s, d, ctl, k, src);
      break;
    case 1: launch_after(k_qp_row<1, MODE>, grid, kQpThreads, smem, s, d, ctl, k, src); break;
    case 2: launch_after(k_qp_row<2, MODE>, grid, kQpThreads, 0, s, d, ctl, k, src); break;
    case 4: launch_after(k_qp_row<4, MODE>, grid, kQpThreads, 0, s, d, ctl, k, src); break;
    case 8: launch_after(k_qp_row<8, MODE>, grid, kQpThreads, 0, s, d, ctl, k, src); break;
    case 16: launch_after(k_qp_row<16, MODE>, grid, kQpThreads, 0, s, d, ctl, k, src); break;
    default: launch_after(k_qp_row<32, MODE>, grid, kQpThreads, 0, s, d, ctl, k, src); break;
  }
  ++g_qp_launches;
}

}  // namespace

void qp_launch_column_pass(const QpDev& d, QpCtl* ctl, int mode, int k, int src,
                           cudaStream_t s) {
  if (mode == kQpStep) column_pass<kQpStep>(d, ctl, k, src, s);
  else if (mode == kQpCheck) column_pass<kQpCheck>(d, ctl, k, src, s);
  else column_pass<kQpReport>(d, ctl, k, src, s);
  if (mode == kQpReport) {
    launch_after(k_qp_objective, 1, kQpThreads, 0, s, d, ctl);
    ++g_qp_launches;
  }
}

void qp_launch_row_pass(const QpDev& d, QpCtl* ctl, int mode, int k, int src, cudaStream_t s) {
  if (mode == kQpStep) row_pass<kQpStep>(d, ctl, k, src, s);
  else row_pass<kQpCheck>(d, ctl, k, src, s);
}

long long qp_resident_smem(int m, int n, long long rows_q, long long rows_a, long long rows_r) {
  const auto part = [](long long rows, int items) {
    const int slices = (items + kQpGroup - 1) / kQpGroup * (kQpGroup / 32);
    return rows * 32 * 10 + ((slices + 4) & ~3) * 4 + 16;
  };
  return 8LL * (3 * n + m) + 16 + part(rows_q, n) + part(rows_a, n) +
         (m > 0 ? part(rows_r, m) : 0);
}

bool qp_resident_fits(long long smem) {
  return smem <= max_dynamic_smem(reinterpret_cast<const void*>(k_qp_resident));
}

void qp_launch_resident(const QpDev& d, QpCtl* ctl, int k0, int count, int src, int smem,
                        cudaStream_t s) {
  const int warps = std::max(2, std::max(d.cols.nslices, d.rows.nslices));
  k_qp_resident<<<1, std::min(kResidentThreads, warps * 32), smem, s>>>(d, ctl, k0, count, src);
  ++g_qp_launches;
}

bool qp_steps_fit(const QpDev& d) {
  return d.cols.nslices > 0 && (d.m == 0 || d.rows.nslices > 0) &&
         grid_fits(k_qp_steps, std::max(d.cols.blocks, d.rows.blocks), kQpSliceThreads, 0);
}

void qp_launch_load_passes(cudaStream_t s) {
  k_qp_column<0, kQpStep><<<1, 32, 0, s>>>(QpDev{}, nullptr, 0, 0);
  k_qp_row<0, kQpStep><<<1, 32, 0, s>>>(QpDev{}, nullptr, 0, 0);
  g_qp_launches += 2;
}

void qp_launch_steps(const QpDev& d, QpCtl* ctl, int k0, int count, cudaStream_t s) {
  launch_grid(k_qp_steps, std::max(d.cols.blocks, d.rows.blocks), kQpSliceThreads, 0, s, d, ctl, k0,
              count);
  ++g_qp_launches;
}

void qp_launch_decide(const QpDev& d, QpCtl* ctl, int k, int p, cudaStream_t s) {
  launch_after(k_qp_decide, 1, kQpThreads, 0, s, d, ctl, k, p);
  ++g_qp_launches;
}

void qp_launch_advance(QpCtl* ctl, int graph_iterations, cudaStream_t s) {
  launch_after(k_qp_advance, 1, 1, 0, s, ctl, graph_iterations);
  ++g_qp_launches;
}

int qp_product_blocks(const QpDev& d) {
  constexpr int kWarps = kQpSliceThreads / 32;
  // A sliced side's blocks each take their own slices; otherwise the warps stride over the items.
  const int warps = std::max({d.ncol_chunks, d.nrow_chunks, d.cols.nslices > 0 ? 0 : d.n / 32,
                              d.rows.nslices > 0 ? 0 : d.m / 32, 1});
  return std::max({std::min((warps + kWarps - 1) / kWarps, 2048), d.cols.blocks, d.rows.blocks});
}

void qp_launch_product(const QpDev& d, int side, const double* v, const double* norm2, double* out,
                       int lanes, double* next, double* part, unsigned int* ticket,
                       cudaStream_t s) {
  const int grid = qp_product_blocks(d);
  const auto launch = [&](auto kernel) {
    kernel<<<grid, kQpSliceThreads, 0, s>>>(d, v, norm2, out, lanes, next, part, ticket);
  };
  if (side == kQpRows) {
    launch(k_qp_product<kQpRows>);
  } else if (side == kQpCols) {
    launch(k_qp_product<kQpCols>);
  } else {
    launch(k_qp_product<kQpHessian>);
  }
  ++g_qp_launches;
}

void qp_launch_slice_fill(const QpDev& d, bool cols, int* idx1, double* val1, int* idx2,
                          double* val2, cudaStream_t s) {
  const QpSliceSet& S = cols ? d.cols : d.rows;
  if (S.nslices == 0) return;
  const int grid = (S.nslices + kQpWarps - 1) / kQpWarps;
  if (cols) {
    k_qp_slice_fill<<<grid, kQpThreads, 0, s>>>(S, 1, d.q_rs, d.q_ci, d.q_v, idx1, val1);
    ++g_qp_launches;
  }
  k_qp_slice_fill<<<grid, kQpThreads, 0, s>>>(S, 2, cols ? d.a_cs : d.a_rs,
                                              cols ? d.a_ri : d.a_ci, cols ? d.a_cv : d.a_rv,
                                              idx2, val2);
  ++g_qp_launches;
}

void qp_launch_dot(const double* a, const double* b, int n, double* partials, double* out,
                   cudaStream_t s) {
  k_qp_dot_partial<<<kQpDotBlocks, kQpThreads, 0, s>>>(a, b, n, partials);
  k_qp_dot_final<<<1, kQpThreads, 0, s>>>(partials, out);
  g_qp_launches += 2;
}

void qp_launch_row_dual(const QpDev& d, double* row_dual, cudaStream_t s) {
  if (d.m <= 0) return;
  k_qp_row_dual<<<grid_for(d.m), kQpThreads, 0, s>>>(d, row_dual);
  ++g_qp_launches;
}

void qp_launch_init(const QpDev& d, cudaStream_t s) {
  const int grid = grid_for(std::max(d.m, d.n));
  if (grid == 0) return;
  k_qp_init<<<grid, kQpThreads, 0, s>>>(d);
  ++g_qp_launches;
}

long long qp_kernel_launch_count() { return g_qp_launches; }

cudaError_t qp_configure_kernels() {
  cudaError_t err = cudaSuccess;
  const auto opt = [&](const void* f) {
    const cudaError_t e =
        cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, kQpStageBytes);
    if (err == cudaSuccess) err = e;
  };
  err = cudaFuncSetAttribute(k_qp_resident, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             max_dynamic_smem(reinterpret_cast<const void*>(k_qp_resident)));
  opt(reinterpret_cast<const void*>(k_qp_column<1, kQpStep>));
  opt(reinterpret_cast<const void*>(k_qp_column<1, kQpCheck>));
  opt(reinterpret_cast<const void*>(k_qp_column<1, kQpReport>));
  opt(reinterpret_cast<const void*>(k_qp_row<1, kQpStep>));
  opt(reinterpret_cast<const void*>(k_qp_row<1, kQpCheck>));
  return err;
}

}  // namespace sgb
