// qp_layout.hpp -- the host-side layouts of the convex-QP engine, with no CUDA in them: what
// QpEngine::load and QpEngine::layout build from a sankhya_gb300_qp_problem (qp.cu), kept
// apart so that the CPU tests can check them (tests/host/qp_layout_export.cpp).
#pragma once

#include <algorithm>
#include <cmath>
#include <limits>
#include <utility>
#include <vector>

#include "sankhya_gb300.h"

namespace sgb {

// Entries a chunk of a long row or column holds at most, and the lanes past which an item is
// long: an item with more than kQpLongPerLane entries per lane goes to the chunked path.
constexpr int kQpChunk = 2048;
// The chunks of the passes, by the entries of A: a warp's chunk is a chain of loads, and a chunk costs
// a partial and a ticket. us an iteration of rows drawn by Zipf's law with chunks of 256, 512, 1,024
// and 2,048: 16.8, 17.4, 18.9, 21.4 (200,000 entries); 39.8, 35.7, 32.5, 34.3 (2 million).
constexpr int kQpShortChunk = 512, kQpMidChunk = 1024;
constexpr long long kQpShortChunkNnz = 1LL << 20;
constexpr int kQpLongPerLane = 64;

// One chunk of a long row or column: entries [begin, end) of the item's entry sequence (for
// a column: the entries of row j of Q, then those of column j of A).
struct QpChunk {
  int item;
  int begin, end;
  int first;  // the item's first chunk (partials slot)
  int count;  // the item's chunk count
  int slot;   // the item's ticket and long-item slot
};

// What the kernels read, built on the host.
struct QpHostLayout {
  // A by rows: a counting-sort transpose in column order keeps each row's columns ascending.
  std::vector<int> row_starts, row_cols;
  std::vector<double> row_values;
  // sense Q by rows, both triangles: a stored entry (i, j) is Q_ij and, off the diagonal, Q_ji
  // (src/qp/qp_condat_vu.cpp:145-160); columns ascending inside each row.
  std::vector<int> q_starts, q_cols;
  std::vector<double> q_values;
  // Entries per column (its row of Q and its column of A) and per row.
  std::vector<int> col_len, row_len;
  // The cost times the sense, and every bound that is_finite_bound calls absent as an
  // infinity on its side (include/sankhya/types.hpp:88-96).
  std::vector<double> cost, col_lower, col_upper, row_lower, row_upper;
};

inline bool qp_finite_bound(double v) { return !(std::isinf(v) || std::fabs(v) >= 1e30); }

// Builds every array of QpHostLayout. The problem must have passed the engine's load checks.
inline void qp_build_layout(const sankhya_gb300_qp_problem& p, QpHostLayout* out) {
  const sankhya_gb300_lp& lp = p.lp;
  const int m = lp.rows, n = lp.cols;
  const long long nnz = lp.col_starts[n];
  const long long hz = p.hessian_starts != nullptr ? p.hessian_starts[n] : 0;
  const double sense = lp.sense < 0.0 ? -1.0 : 1.0;

  out->row_starts.assign(static_cast<size_t>(m) + 1, 0);
  std::vector<int>& rptr = out->row_starts;
  for (long long k = 0; k < nnz; ++k) ++rptr[static_cast<size_t>(lp.row_index[k]) + 1];
  for (int i = 0; i < m; ++i) rptr[i + 1] += rptr[i];
  std::vector<int> next(rptr.begin(), rptr.end() - 1);
  out->row_cols.assign(static_cast<size_t>(nnz), 0);
  out->row_values.assign(static_cast<size_t>(nnz), 0.0);
  for (int j = 0; j < n; ++j) {
    for (int k = lp.col_starts[j]; k < lp.col_starts[j + 1]; ++k) {
      const int slot = next[lp.row_index[k]]++;
      out->row_cols[slot] = j;
      out->row_values[slot] = lp.values[k];
    }
  }

  // Walking the stored columns in order puts each row's entries in ascending column order for
  // a lower triangle; any other input is sorted per row.
  out->q_starts.assign(static_cast<size_t>(n) + 1, 0);
  std::vector<int>& qptr = out->q_starts;
  for (int j = 0; j < n && hz > 0; ++j) {
    for (int k = p.hessian_starts[j]; k < p.hessian_starts[j + 1]; ++k) {
      const int i = p.hessian_index[k];
      ++qptr[static_cast<size_t>(i) + 1];
      if (i != j) ++qptr[static_cast<size_t>(j) + 1];
    }
  }
  for (int j = 0; j < n; ++j) qptr[j + 1] += qptr[j];
  const long long qz = qptr[n];
  std::vector<int> qnext(qptr.begin(), qptr.end() - 1);
  std::vector<int>& qidx = out->q_cols;
  std::vector<double>& qval = out->q_values;
  qidx.assign(static_cast<size_t>(qz), 0);
  qval.assign(static_cast<size_t>(qz), 0.0);
  for (int j = 0; j < n && hz > 0; ++j) {
    for (int k = p.hessian_starts[j]; k < p.hessian_starts[j + 1]; ++k) {
      const int i = p.hessian_index[k];
      const double v = sense * p.hessian_values[k];
      int slot = qnext[i]++;
      qidx[slot] = j;
      qval[slot] = v;
      if (i != j) {
        slot = qnext[j]++;
        qidx[slot] = i;
        qval[slot] = v;
      }
    }
  }
  for (int r = 0; r < n; ++r) {
    const int b = qptr[r], e = qptr[r + 1];
    bool sorted = true;
    for (int k = b + 1; k < e && sorted; ++k) sorted = qidx[k - 1] <= qidx[k];
    if (sorted) continue;
    std::vector<std::pair<int, double>> row;
    for (int k = b; k < e; ++k) row.push_back({qidx[k], qval[k]});
    std::stable_sort(row.begin(), row.end(),
                     [](const auto& a, const auto& c) { return a.first < c.first; });
    for (int k = b; k < e; ++k) {
      qidx[k] = row[k - b].first;
      qval[k] = row[k - b].second;
    }
  }

  out->col_len.assign(static_cast<size_t>(n), 0);
  out->row_len.assign(static_cast<size_t>(m), 0);
  for (int j = 0; j < n; ++j) {
    out->col_len[j] = (qptr[j + 1] - qptr[j]) + (lp.col_starts[j + 1] - lp.col_starts[j]);
  }
  for (int i = 0; i < m; ++i) out->row_len[i] = rptr[i + 1] - rptr[i];

  constexpr double kInf = std::numeric_limits<double>::infinity();
  out->cost.resize(static_cast<size_t>(n));
  out->col_lower.resize(static_cast<size_t>(n));
  out->col_upper.resize(static_cast<size_t>(n));
  out->row_lower.resize(static_cast<size_t>(m));
  out->row_upper.resize(static_cast<size_t>(m));
  for (int j = 0; j < n; ++j) {
    out->cost[j] = sense * lp.col_cost[j];
    out->col_lower[j] = qp_finite_bound(lp.col_lower[j]) ? lp.col_lower[j] : -kInf;
    out->col_upper[j] = qp_finite_bound(lp.col_upper[j]) ? lp.col_upper[j] : kInf;
  }
  for (int i = 0; i < m; ++i) {
    out->row_lower[i] = qp_finite_bound(lp.row_lower[i]) ? lp.row_lower[i] : -kInf;
    out->row_upper[i] = qp_finite_bound(lp.row_upper[i]) ? lp.row_upper[i] : kInf;
  }
}

// The chunks, of at most `chunk` entries, of the items longer than kQpLongPerLane * lanes entries, in
// item order; *nlong receives the number of such items (their slots are 0 .. *nlong - 1 in item
// order).
inline void qp_build_chunks(const std::vector<int>& len, int lanes, std::vector<QpChunk>* out,
                            int* nlong, int chunk = kQpChunk) {
  out->clear();
  *nlong = 0;
  for (int item = 0; item < static_cast<int>(len.size()); ++item) {
    const int l = len[item];
    if (l <= kQpLongPerLane * lanes) continue;
    const int count = (l + chunk - 1) / chunk;
    const int first = static_cast<int>(out->size());
    for (int c = 0; c < count; ++c) {
      out->push_back(QpChunk{item, c * chunk, std::min(l, (c + 1) * chunk), first, count, *nlong});
    }
    ++*nlong;
  }
}

// ---- Sliced items ----------------------------------------------------------------------------
// The one-lane passes' layout of the matrix: a slice is 32 items that one warp sums, one item per
// lane, with lane l's k-th entry at 32 (base + k) + l, so that a slice's entries are one run.
// Items of at most kQpLongPerLane entries are dealt to slices by length, longest first, inside
// groups of kQpGroup consecutive items: a warp takes as long as its longest item. A column's
// entries are its row of Q and its column of A, stored apart; a row has the second part only.
constexpr int kQpGroup = 128;
constexpr unsigned kQpNoItem = 0xffffffffu;

struct QpSlices {
  int nslices = 0;
  // Per slice and lane: the item's place in its group (7 bits), its entries of the first part
  // (from bit 8) and of the second (from bit 16); kQpNoItem where there is no short item.
  std::vector<unsigned> meta;
  std::vector<unsigned> base1, base2;  // per slice: first entry / 32 of each part; nslices + 1
  std::vector<int> block_start;        // block b's slices: [block_start[b], block_start[b + 1])
};

// starts1 may be null (no first part). At most `blocks` blocks, cut by cost (entry rows, and an
// epilogue's worth per slice), of at least four slices on average.
inline void qp_build_slices(const int* starts1, const int* starts2, int count, int blocks,
                            QpSlices* out) {
  const int groups = (count + kQpGroup - 1) / kQpGroup, per = kQpGroup / 32;
  out->nslices = groups * per;
  const size_t ns = static_cast<size_t>(out->nslices);
  out->meta.assign(ns * 32, kQpNoItem);
  out->base1.assign(ns + 1, 0);
  out->base2.assign(ns + 1, 0);
  unsigned t1 = 0, t2 = 0;
  const auto len1 = [&](int i) { return starts1 != nullptr ? starts1[i + 1] - starts1[i] : 0; };
  const auto len2 = [&](int i) { return starts2[i + 1] - starts2[i]; };
  for (int g = 0; g < groups; ++g) {
    const int i0 = g * kQpGroup, i1 = std::min(count, i0 + kQpGroup);
    int start[kQpLongPerLane + 2] = {0};
    for (int i = i0; i < i1; ++i) {
      const int len = len1(i) + len2(i);
      if (len <= kQpLongPerLane) ++start[kQpLongPerLane - len + 1];
    }
    for (int k = 0; k <= kQpLongPerLane; ++k) start[k + 1] += start[k];
    unsigned* meta = out->meta.data() + static_cast<size_t>(g) * kQpGroup;
    for (int i = i0; i < i1; ++i) {
      const int a = len1(i), b = len2(i);
      if (a + b > kQpLongPerLane) continue;
      meta[start[kQpLongPerLane - a - b]++] = static_cast<unsigned>(i - i0) |
                                              static_cast<unsigned>(a) << 8 |
                                              static_cast<unsigned>(b) << 16;
    }
    for (int s = 0; s < per; ++s) {
      unsigned w1 = 0, w2 = 0;
      for (int l = 0; l < 32; ++l) {
        const unsigned m = meta[s * 32 + l];
        if (m == kQpNoItem) continue;
        w1 = std::max(w1, (m >> 8) & 255u);
        w2 = std::max(w2, m >> 16);
      }
      t1 += w1;
      t2 += w2;
      out->base1[static_cast<size_t>(g) * per + s + 1] = t1;
      out->base2[static_cast<size_t>(g) * per + s + 1] = t2;
    }
  }
  const int G = std::max(1, std::min(blocks, (out->nslices + 3) / 4));
  const auto cost = [&](int s) {
    return static_cast<double>(out->base1[static_cast<size_t>(s)]) +
           static_cast<double>(out->base2[static_cast<size_t>(s)]) + 8.0 * s;
  };
  out->block_start.assign(static_cast<size_t>(G) + 1, out->nslices);
  int s = 0;
  for (int b = 0; b < G; ++b) {
    out->block_start[static_cast<size_t>(b)] = s;
    const double upto = cost(out->nslices) * (b + 1) / G;
    while (s < out->nslices && b + 1 < G && cost(s) + cost(s + 1) < 2.0 * upto) ++s;
  }
}

// Lanes per item from the mean entries per item: the smallest power of two that leaves each
// lane at most 32 entries of a typical item. The passes wait on memory and on the FP64 pipe,
// where a lane that sits out the epilogue costs as much as a working one, so few lanes win:
// on the 1M x 2M QP (15 entries per column, 20 per row) one lane per column and per row runs
// 2.4 and 2.6 times faster than four and eight. Items longer than kQpLongPerLane lanes' worth
// go to the chunked path whatever the lanes.
inline int qp_auto_lanes(double mean) {
  int g = 1;
  while (g < 32 && 32.0 * g < mean) g *= 2;
  return g;
}

}  // namespace sgb
