// layout.cu -- host planning of the step passes' chunk layouts (see chunks.cuh).
//
// plan_chunks() takes one layout of the matrix (the CSR copy for the row pass, the CSC copy
// for the column pass) and decides, once at load time:
//   * the chunks (rows cut at kChunkRows rows and `cap` entries, long rows into pieces);
//   * each chunk's window of the gathered vector (build_windows, the same rule as the tile
//     layouts), and from the share of entries the windows hold whether the layout stages
//     windows at all, stages them over every entry, or is SPLIT into a main part gathered
//     from windows only and an outer part gathered from L2;
//   * which chunks each block of the grid owns (a cost model: entries plus a fixed cost per
//     window staged), the block's segments, and for a split layout the block's outer chunks.
// plan_slices() plans the FP64 passes' sliced layouts (slices.cuh) the same way.
// Everything here is plain host code: the engine uploads the result, and
// tests/host/layout_check.cu checks the chunk layouts on the CPU.
#include "engine.hpp"

#include <algorithm>
#include <cstdio>
#include <cstdlib>

namespace sgb {

namespace {

// Consecutive rows while the chunk has at most kChunkRows rows and `cap` entries, and every
// row of it shares `row_win` (nullptr: no window constraint); a row longer than `cap` becomes
// pieces of `cap` entries, listed as a LongRow.
void cut_chunks(const std::vector<int>& ptr, int r_begin, int r_end, int cap,
                const std::vector<int>* row_win, std::vector<Tile>* chunks,
                std::vector<LongRow>* longs, int* npieces) {
  int r = r_begin;
  while (r < r_end) {
    const int len = ptr[r + 1] - ptr[r];
    if (len > cap) {
      LongRow lr{r, *npieces, 0};
      for (int k = ptr[r]; k < ptr[r + 1]; k += cap) {
        const int k1 = std::min(k + cap, ptr[r + 1]);
        chunks->push_back(Tile{r, -(*npieces) - 1, k, k1});
        ++*npieces;
        ++lr.nchunks;
      }
      longs->push_back(lr);
      ++r;
      continue;
    }
    const int begin = r;
    const int w = row_win ? (*row_win)[r] : 0;
    ++r;
    while (r < r_end && r - begin < kChunkRows && ptr[r + 1] - ptr[r] <= cap &&
           ptr[r + 1] - ptr[begin] <= cap && (row_win == nullptr || (*row_win)[r] == w)) {
      ++r;
    }
    chunks->push_back(Tile{begin, r, ptr[begin], ptr[r]});
  }
}

// The start lo (a multiple of 4, within [0, ext4 - wmax]) for which [lo, lo + wmax) holds the
// most of the sorted indices v, centred among the starts that do; *count receives that most.
int best_start(const std::vector<int>& v, int wmax, int ext4, int* count) {
  int best = 0, bl = 0, br = 0;
  for (int r = 0, l = 0; r < static_cast<int>(v.size()); ++r) {
    while (v[r] - v[l] >= wmax) ++l;
    if (r - l + 1 > best) {
      best = r - l + 1;
      bl = l;
      br = r;
    }
  }
  *count = best;
  long long lo = 0;
  if (best > 0) {
    const long long lo_min = static_cast<long long>(v[br]) - wmax + 1, lo_max = v[bl];
    lo = lo_min + (lo_max - lo_min) / 2;
  }
  lo = std::max(0LL, std::min(lo, static_cast<long long>(ext4 - wmax)));
  return static_cast<int>(lo) & ~3;
}

int held_by(const Tile& t, const int* idx, int lo, int len) {
  int held = 0;
  for (int k = t.k0; k < t.k1; ++k) {
    held += static_cast<unsigned>(idx[k] - lo) < static_cast<unsigned>(len);
  }
  return held;
}

// Windows of a chunk sequence, in chunk order. A chunk keeps the window its block holds
// while that window holds all but 2% of what the chunk's own best window would. Otherwise the
// window that best serves the next kLookahead chunks together is weighed against the one held
// over those chunks, and replaces it only if it holds 3% more of their entries: a chunk's own
// best window is tuned to its few scattered entries, and restaging costs a block barrier and
// a copy of the whole window, so a window changes only where the pattern moves (a new period
// of a block-angular matrix, say). A chunk whose best window holds fewer than 1/8 of its
// entries gathers from global memory. Returns the entries that fall inside their chunk's
// window.
long long plan_windows(const std::vector<Tile>& chunks, const int* idx, int extent, int wmax,
                       std::vector<int>* chunk_win, std::vector<int2>* windows) {
  constexpr int kLookahead = 32;
  const int nchunks = static_cast<int>(chunks.size());
  chunk_win->assign(static_cast<size_t>(nchunks), -1);
  windows->clear();
  if (wmax <= 0 || nchunks == 0 || extent <= 0) return 0;
  const int ext4 = (extent + 3) & ~3;
  long long covered = 0;
  if (ext4 <= wmax) {  // the whole vector fits: one window for every chunk
    windows->push_back(make_int2(0, ext4));
    chunk_win->assign(static_cast<size_t>(nchunks), 0);
    for (const Tile& t : chunks) covered += t.k1 - t.k0;
    return covered;
  }
  std::vector<int> v;
  int current = -1;
  int weighed_until = 0;  // the held window was last weighed over the chunks before this one
  for (int c = 0; c < nchunks; ++c) {
    const Tile& tl = chunks[static_cast<size_t>(c)];
    const int entries = tl.k1 - tl.k0;
    if (entries == 0) {
      (*chunk_win)[static_cast<size_t>(c)] = current;
      continue;
    }
    v.assign(idx + tl.k0, idx + tl.k1);
    std::sort(v.begin(), v.end());
    int best = 0;
    best_start(v, wmax, ext4, &best);
    if (best * 8 < entries) continue;  // gathers from global memory
    const int2 cw = current >= 0 ? (*windows)[static_cast<size_t>(current)] : make_int2(0, 0);
    const int held = current >= 0 ? held_by(tl, idx, cw.x, cw.y) : 0;
    // Within the chunks a weighing already covered, only a collapse of the held share
    // brings the window up again.
    if (current >= 0 && (held >= best - 0.02 * entries || (c < weighed_until && 2 * held >= best))) {
      (*chunk_win)[static_cast<size_t>(c)] = current;
      continue;
    }
    // The window that best serves this chunk and the next ones together.
    const int c_end = std::min(nchunks, c + kLookahead);
    v.clear();
    for (int d = c; d < c_end; ++d) {
      v.insert(v.end(), idx + chunks[static_cast<size_t>(d)].k0,
               idx + chunks[static_cast<size_t>(d)].k1);
    }
    std::sort(v.begin(), v.end());
    int union_best = 0;
    const int lo = best_start(v, wmax, ext4, &union_best);
    if (current >= 0) {
      long long held_cur = 0, held_new = 0;
      for (int d = c; d < c_end; ++d) {
        held_cur += held_by(chunks[static_cast<size_t>(d)], idx, cw.x, cw.y);
        held_new += held_by(chunks[static_cast<size_t>(d)], idx, lo, wmax);
      }
      if (static_cast<double>(held_new) <= held_cur + 0.03 * static_cast<double>(v.size())) {
        (*chunk_win)[static_cast<size_t>(c)] = current;
        weighed_until = c_end;
        continue;
      }
    }
    weighed_until = c_end;
    windows->push_back(make_int2(lo, wmax));
    current = static_cast<int>(windows->size()) - 1;
    (*chunk_win)[static_cast<size_t>(c)] = current;
  }
  for (int c = 0; c < nchunks; ++c) {
    const int w = (*chunk_win)[static_cast<size_t>(c)];
    if (w < 0) continue;
    const int2 r = (*windows)[static_cast<size_t>(w)];
    covered += held_by(chunks[static_cast<size_t>(c)], idx, r.x, r.y);
  }
  return covered;
}

}  // namespace

ChunkPlan plan_chunks(const std::vector<int>& ptr, const int* idx, int lines, int extent, int cap,
                      int wmax, int grid, int elem_bytes, double split_min, double full_min,
                      int outer_round_cap) {
  ChunkPlan p;
  p.cap = cap;
  p.grid = std::max(1, grid);
  const long long nnz = lines > 0 ? ptr[lines] : 0;
  // Base chunks over the whole layout and their windows.
  std::vector<Tile> base;
  std::vector<LongRow> base_longs;
  int base_pieces = 0;
  cut_chunks(ptr, 0, lines, cap, nullptr, &base, &base_longs, &base_pieces);
  std::vector<int> tile_win;
  std::vector<int2> windows;
  long long covered = 0;
  if (wmax > 0 && nnz > 0) {
    covered = plan_windows(base, idx, extent, wmax, &tile_win, &windows);
  } else {
    tile_win.assign(base.size(), -1);
  }
  const double share = nnz > 0 ? static_cast<double>(covered) / static_cast<double>(nnz) : 0.0;
  p.coverage = share;
  std::vector<int> chunk_win;
  if (windows.empty() || share < split_min) {
    // No staging: every gather from L2.
    p.chunks = base;
    p.longs = base_longs;
    p.npieces = base_pieces;
    chunk_win.assign(p.chunks.size(), -1);
    windows.clear();
    p.staged = 0.0;
  } else if (share >= full_min) {
    p.chunks = base;
    p.longs = base_longs;
    p.npieces = base_pieces;
    chunk_win = tile_win;
    p.staged = share;
  } else {
    // Split: a row's window is its base chunk's; long rows keep every entry in the main part
    // and gather from global memory.
    p.split = true;
    std::vector<int> row_win(static_cast<size_t>(lines), -1);
    for (size_t t = 0; t < base.size(); ++t) {
      const Tile& tl = base[t];
      if (tl.r1 < 0) continue;
      for (int r = tl.r0; r < tl.r1; ++r) row_win[r] = tile_win[t];
    }
    p.ptr.assign(static_cast<size_t>(lines) + 1, 0);
    p.optr.assign(static_cast<size_t>(lines) + 1, 0);
    long long in_window = 0;
    for (int r = 0; r < lines; ++r) {
      const int w = row_win[r];
      const int lo = w >= 0 ? windows[w].x : 0, len = w >= 0 ? windows[w].y : 0;
      for (int k = ptr[r]; k < ptr[r + 1]; ++k) {
        const bool inside = w < 0 || static_cast<unsigned>(idx[k] - lo) < static_cast<unsigned>(len);
        if (inside) {
          p.idx.push_back(idx[k]);
          p.map.push_back(k);
          in_window += w >= 0;
        } else {
          p.oidx.push_back(idx[k]);
          p.omap.push_back(k);
        }
      }
      p.ptr[r + 1] = static_cast<int>(p.idx.size());
      p.optr[r + 1] = static_cast<int>(p.oidx.size());
    }
    cut_chunks(p.ptr, 0, lines, cap, &row_win, &p.chunks, &p.longs, &p.npieces);
    chunk_win.resize(p.chunks.size());
    for (size_t c = 0; c < p.chunks.size(); ++c) {
      const Tile& tl = p.chunks[c];
      chunk_win[c] = tl.r1 < 0 ? -1 : row_win[tl.r0];
    }
    p.staged = nnz > 0 ? static_cast<double>(in_window) / static_cast<double>(nnz) : 0.0;
  }
  // Window capacity actually used.
  p.wmax = 0;
  for (const int2& w : windows) p.wmax = std::max(p.wmax, w.y);

  // Blocks: cut the chunk sequence where the running cost reaches the average. A chunk costs
  // its entries plus a fixed overhead; staging a window costs its bytes / 32 entries (it is
  // copied from L2 at a multiple of the matrix stream's speed).
  const int G = p.grid;
  const long long T = static_cast<long long>(p.chunks.size());
  const double per_chunk = 16.0;
  const double stage_cost = static_cast<double>(p.wmax) * elem_bytes / 32.0;
  double total = 0.0;
  long long stages = 0;
  for (long long c = 0; c < T; ++c) {
    total += (p.chunks[c].k1 - p.chunks[c].k0) + per_chunk;
    if (chunk_win[c] >= 0 && (c == 0 || chunk_win[c] != chunk_win[c - 1])) ++stages;
  }
  const double target = (total + stage_cost * static_cast<double>(stages + G)) / G;
  std::vector<long long> bstart(static_cast<size_t>(G) + 1, T);
  bstart[0] = 0;
  {
    int b = 0;
    double acc = 0.0;
    int held = -2;  // the window the current block holds (-2: none yet)
    for (long long c = 0; c < T; ++c) {
      if (chunk_win[c] >= 0 && chunk_win[c] != held) acc += stage_cost;
      held = chunk_win[c] >= 0 ? chunk_win[c] : held;
      acc += (p.chunks[c].k1 - p.chunks[c].k0) + per_chunk;
      if (acc >= target && b + 1 < G && c + 1 < T) {
        bstart[++b] = c + 1;
        acc = 0.0;
        held = -2;
      }
    }
    for (int q = b + 1; q <= G; ++q) bstart[q] = T;
  }
  // Segments.
  p.seg_start.assign(static_cast<size_t>(G) + 1, 0);
  for (int b = 0; b < G; ++b) {
    p.seg_start[b] = static_cast<int>(p.segs.size());
    long long c = bstart[b];
    while (c < bstart[b + 1]) {
      long long e = c + 1;
      while (e < bstart[b + 1] && chunk_win[e] == chunk_win[c]) ++e;
      ChunkSeg sg{static_cast<int>(c), static_cast<int>(e), 0, 0};
      if (chunk_win[c] >= 0) {
        sg.lo = windows[chunk_win[c]].x;
        sg.len = windows[chunk_win[c]].y;
      }
      p.segs.push_back(sg);
      c = e;
    }
  }
  p.seg_start[G] = static_cast<int>(p.segs.size());
  p.lo.assign(static_cast<size_t>(T), 0);
  p.narrow = p.wmax > 0 && p.wmax <= 65536 && (p.split || covered == nnz);
  for (const ChunkSeg& sg : p.segs) {
    for (int c = sg.c0; c < sg.c1; ++c) {
      p.lo[static_cast<size_t>(c)] = sg.lo;
      if (p.chunks[static_cast<size_t>(c)].r1 >= 0 && sg.len <= 0) p.narrow = false;
    }
  }
  // Outer rounds: block b sums the outer entries of rows [row_begin[b], row_begin[b + 1]),
  // where row_begin[b] is the first row of its first chunk. Its main chunks lie inside that
  // range (a piece of a long row may not, but pieces read no outer sum), and every row of it
  // is written, zero where it has no outer entry. A round is a run of those rows whose outer
  // entries fit the block's staging space (outer_round_cap entries).
  if (p.split) {
    std::vector<int> row_begin(static_cast<size_t>(G) + 1, lines);
    for (int b = 0; b < G; ++b) row_begin[b] = bstart[b] < T ? p.chunks[bstart[b]].r0 : lines;
    p.oround_start.assign(static_cast<size_t>(G) + 1, 0);
    for (int b = 0; b < G; ++b) {
      p.oround_start[b] = static_cast<int>(p.orounds.size());
      int r = row_begin[b];
      while (r < row_begin[b + 1]) {
        int e = r;
        while (e < row_begin[b + 1] && p.optr[e + 1] - p.optr[r] <= outer_round_cap) ++e;
        if (e == r) {  // one row with more outer entries than the staging space holds
          std::fprintf(stderr, "plan_chunks: row %d has %d outer entries (> %d)\n", r,
                       p.optr[r + 1] - p.optr[r], outer_round_cap);
          p.error = true;
          break;
        }
        p.orounds.push_back(make_int2(r, e));
        r = e;
      }
    }
    p.oround_start[G] = static_cast<int>(p.orounds.size());
    if (row_begin[0] != 0) p.error = true;
  }
  if (std::getenv("SANKHYA_GB300_LAYOUT_LOG") != nullptr) {
    std::fprintf(stderr,
                 "plan_chunks: %d lines, %lld entries, cap %d, wmax %d: coverage %.4f, %s, "
                 "staged %.4f, %zu chunks, %zu windows, %zu segments, %zu outer entries, "
                 "%zu outer rounds, %d pieces\n",
                 lines, nnz, cap, p.wmax, p.coverage,
                 p.split ? (p.narrow ? "split, packed" : "split")
                         : (p.wmax == 0 ? "unstaged" : (p.narrow ? "windowed, packed" : "windowed")),
                 p.staged,
                 p.chunks.size(), windows.size(), p.segs.size(), p.oidx.size(),
                 p.orounds.size(), p.npieces);
  }
  return p;
}

// The sliced layout of one matrix layout (slices.cuh): rows dealt to slices by length inside
// each group, the long rows' items, the windows over the groups and the blocks' segments.
// `np` products are accumulated per entry by the kernel that runs on it (the cost model: a
// slice costs its longest row's entries times np FP64 instructions, plus its epilogue).
SlicePlan plan_slices(const std::vector<int>& ptr, const int* idx, int lines, int extent, int wmax,
                      double window_min, int sms, int np, int resident) {
  SlicePlan p;
  const int ngroups = (lines + kGroupRows - 1) / kGroupRows;
  const long long nnz = lines > 0 ? ptr[lines] : 0;
  p.nslices = ngroups * kGroupSlices;
  p.meta.assign(static_cast<size_t>(p.nslices) * 32, kNoRow);
  p.base.assign(static_cast<size_t>(p.nslices) + 1, 0);
  std::vector<double> cost(static_cast<size_t>(p.nslices) + 1, 0.0);
  std::vector<Tile> groups(static_cast<size_t>(ngroups));
  long long rows32 = 0;  // entries stored so far, / 32
  long long lentries = 0;
  for (int g = 0; g < ngroups; ++g) {
    const int r0 = g * kGroupRows, r1 = std::min(lines, r0 + kGroupRows);
    groups[static_cast<size_t>(g)] = Tile{r0, r1, ptr[r0], ptr[r1]};
    // A counting sort by length, longest first, rows of equal length in row order.
    int start[kSliceLong + 2] = {0};
    for (int r = r0; r < r1; ++r) {
      const int len = ptr[r + 1] - ptr[r];
      if (len <= kSliceLong) ++start[kSliceLong - len + 1];
    }
    for (int k = 0; k <= kSliceLong; ++k) start[k + 1] += start[k];
    unsigned short* meta = p.meta.data() + static_cast<size_t>(g) * kGroupRows;
    for (int r = r0; r < r1; ++r) {
      const int len = ptr[r + 1] - ptr[r];
      if (len > kSliceLong) {
        const int pieces = (len + kSlicePiece - 1) / kSlicePiece;
        if (pieces > 1) p.longs.push_back(LongRow{r, p.nchunks, pieces});
        for (int c = 0; c < pieces; ++c) {
          const int b = c * kSlicePiece, e = std::min(len, b + kSlicePiece);
          p.items.push_back(SliceItem{r, pieces > 1 ? p.nchunks++ : -1,
                                      static_cast<int>(lentries) + b, e - b,
                                      pieces > 1 ? static_cast<int>(p.longs.size()) - 1 : -1});
        }
        lentries += len;
        continue;
      }
      meta[start[kSliceLong - len]++] =
          static_cast<unsigned short>(static_cast<unsigned>(r - r0) | (static_cast<unsigned>(len) << 8));
    }
    for (int q = 0; q < kGroupSlices; ++q) {
      const unsigned short head = meta[q * 32];
      const int width = head == kNoRow ? 0 : head >> 8;
      p.base[static_cast<size_t>(g) * kGroupSlices + q] = static_cast<unsigned>(rows32);
      rows32 += width;
      const size_t at = static_cast<size_t>(g) * kGroupSlices + q;
      cost[at + 1] = cost[at] + static_cast<double>(width) * np + 12.0;
    }
  }
  p.base[static_cast<size_t>(p.nslices)] = static_cast<unsigned>(rows32);
  p.long_base = rows32 * 32;
  p.entries = p.long_base + lentries;

  // Windows, over the groups; kept where they hold at least window_min of the entries.
  std::vector<int> group_win;
  std::vector<int2> windows;
  long long covered = build_windows(groups, idx, extent, wmax, &group_win, &windows);
  if (nnz > 0 && static_cast<double>(covered) < window_min * static_cast<double>(nnz)) {
    group_win.assign(group_win.size(), -1);
    windows.clear();
    covered = 0;
  }
  p.staged = nnz > 0 ? static_cast<double>(covered) / static_cast<double>(nnz) : 0.0;
  for (const int2& w : windows) p.wmax = std::max(p.wmax, w.y);

  // Blocks: at most one per SM and not under four slices each (a small matrix spreads over the
  // SMs: the FP64 pipe of each is the bound even there), cut where the running cost passes the
  // next share; a block has as many warps as its slices or items keep busy, at most
  // kSliceThreads threads. A resident layout's blocks are its cluster's.
  const int wanted = (std::max(p.nslices, static_cast<int>(p.items.size())) + 3) / 4;
  const int G = resident > 0 ? resident : std::max(1, std::min(wanted, sms));
  p.grid = G;
  p.seg_start.assign(static_cast<size_t>(G) + 1, 0);
  p.block_start.assign(static_cast<size_t>(G) + 1, p.nslices);
  int s0 = 0, most = 1;
  for (int b = 0; b < G; ++b) {
    p.seg_start[static_cast<size_t>(b)] = static_cast<int>(p.segs.size());
    p.block_start[static_cast<size_t>(b)] = s0;
    const double upto = cost[static_cast<size_t>(p.nslices)] * (b + 1) / G;
    int s1 = s0;
    while (s1 < p.nslices &&
           (b + 1 == G ||
            cost[static_cast<size_t>(s1)] + cost[static_cast<size_t>(s1) + 1] < 2.0 * upto)) {
      ++s1;
    }
    most = std::max(most, s1 - s0);
    const auto window = [&](int s) { return group_win[static_cast<size_t>(s / kGroupSlices)]; };
    for (int s = s0; s < s1;) {
      int e = s + 1;
      while (e < s1 && window(e) == window(s)) ++e;
      SliceSeg sg{s, e, 0, 0};
      if (window(s) >= 0) {
        sg.lo = windows[static_cast<size_t>(window(s))].x;
        sg.len = windows[static_cast<size_t>(window(s))].y;
      }
      p.segs.push_back(sg);
      s = e;
    }
    // A block of items only still visits them: they belong to its first segment.
    if (static_cast<int>(p.segs.size()) == p.seg_start[static_cast<size_t>(b)]) {
      p.segs.push_back(SliceSeg{0, 0, 0, 0});
    }
    s0 = s1;
  }
  p.seg_start[static_cast<size_t>(G)] = static_cast<int>(p.segs.size());
  most = std::max(most, (static_cast<int>(p.items.size()) + G - 1) / G);
  p.threads = std::min(kSliceThreads, std::max(128, (most + 3) / 4 * 128));

  return p;
}

}  // namespace sgb
