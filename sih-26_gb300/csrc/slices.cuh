// slices.cuh -- sliced rows: the FP64 sparse-product engine.
//
// A SLICE is 32 rows (of the CSR copy, or columns of the CSC copy) that one warp sums, one row
// per lane, with the entries stored so that lane l's k-th entry is at base + 32 k + l: a slice's
// entries are one contiguous run. A lane walks its own row in ascending index order with FMA, so
// every short row is summed in the reference's order. (Splitting the rows of a small matrix over
// 2 to 8 lanes to shorten their walk was slower at every size tried, down to 50 x 100: the lanes
// that sit out the epilogue cost the FP64 pipe as much as working ones.)
//
// Rows are dealt to slices inside GROUPS of kGroupRows consecutive rows, longest first, so the
// rows of a slice have nearly the same length: GB300 retires two FP64 lane operations per clock
// per SM and charges a warp instruction in full whatever its active lanes, so a slice costs its
// longest row. (Rows of 9 to 31 entries, the 1M x 2M block-angular LP: in row order the 32
// lanes of a warp wait for about 30 entries where the mean is 20; dealt by length inside 128
// rows, for about 21.) A group spans 128 rows only, so the rows of a slice stay close together:
// the per-row operands of the epilogue are read from the same few cache lines by the group's
// four slices, and the group's gathers share a window.
//
// A row of more than kSliceLong entries is LONG: a whole warp sums it (lane l takes entries l,
// l + 32, ...; a fixed tree adds the lanes) from a region of its own behind the slices, in
// pieces of kSlicePiece entries when it is longer than that; the pieces of a row are combined in
// order by the kernel's last block.
//
// PIECES. A warp takes a slice in pieces of up to kPiece entry rows: a piece's values and gathers are
// requested together, then the next piece's indices (of this slice, or the first of the warp's
// next), then the products are added, so a warp waits for memory once per piece. The first
// indices are requested before the kernel may read anything that an earlier one wrote, since the
// matrix never changes between the kernels of a graph. Each count of rows has its own code:
// predicated-off FP64 instructions hold the pipe like working ones.
//
// WINDOWS. A random 8-byte gather from L1 or L2 costs a tag lookup and a sector each, 32 per
// warp-wide gather at one per clock per SM; from shared memory a warp-wide gather of
// doubles costs about 7 clocks of bank conflicts. So a block keeps a window [lo, lo + len) of
// the gathered vector in shared memory where the layout's windows hold enough of its entries
// (build_windows over the groups; Engine::plan_sliced), copied in by one bulk copy per segment of
// groups.
//
// Block b owns a contiguous run of slices, cut by cost, and its warps take them in turn: every sum and every block partial is taken in a fixed order, so runs are
// bit-reproducible. Warps do not wait for one another except where the window changes. Every
// wait is bounded: a wait that gives up raises the block's abort flag, the block's remaining
// slices are skipped, a copy still in flight is given a bounded time to land, and the caller
// records the error.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "chunks.cuh"
#include "common.cuh"
#include "tiles.cuh"

namespace sgb {

constexpr int kGroupRows = 128;
constexpr int kGroupSlices = kGroupRows / 32;
constexpr int kSliceLong = 64;     // entries past which a row is long
constexpr int kSlicePiece = kCap;  // entries per piece of a long row
constexpr int kSliceThreads = 768;   // the largest block of a slice kernel: 85 registers a thread
constexpr int kPiece = 8;            // entry rows (32 entries each) per piece, at most
constexpr unsigned short kNoRow = 0xffff;

// A piece of a long row (or all of it): entries [begin, begin + count) of the layout's long
// region. slot < 0: the whole row, whose epilogue the warp runs; otherwise the partial slot.
struct SliceItem {
  int row;
  int slot;
  int begin;
  int count;
  int longs;  // slot >= 0: the row's LongRow
};

// Consecutive slices of one block that gather from the same window (len = 0: none).
struct SliceSeg {
  int s0, s1;
  int lo, len;
};

struct SliceSet {
  // Per slice and lane: the row's place in its group (7 bits) and its length (from bit 8), or
  // kNoRow (no row, or a long one).
  const unsigned short* meta;
  const unsigned int* base;  // per slice: first entry / 32; nslices + 1
  const int* idx;
  const double* val;
  const SliceItem* items;
  const LongRow* longs;      // rows of several pieces
  // Per such row, zero between passes: the warp that brings its last partial finishes the row. Null
  // in the kernels that leave these rows to run_slice_long_rows.
  unsigned int* tickets;
  const SliceSeg* segs;
  const int* seg_start;      // per block: its segments [seg_start[b], seg_start[b + 1])
  const int* block_start;    // per block: its slices [block_start[b], block_start[b + 1])
  long long long_base;       // first entry of the long region
  int nslices, nitems, nlong, nchunks, nrows;
  int wmax;                  // window capacity in gathered elements (0: none)
  int grid, threads;
};

// Dynamic shared memory of a slice kernel with a window: its mbarrier, then the window.
constexpr int kSliceBarBytes = 128;
template <typename G>
__host__ __device__ constexpr int slice_smem(int wmax) {
  return wmax > 0 ? kSliceBarBytes + ((wmax * static_cast<int>(sizeof(G)) + 127) & ~127) : 0;
}

// The row a meta word of slice s names.
__device__ __forceinline__ int slice_row(int s, unsigned m) {
  return (s / kGroupSlices) * kGroupRows + static_cast<int>(m & 127u);
}

// The indices of a lane's next piece: its first P of `left` entries from `idx` on.
template <int P>
struct PieceIndices {
  int c[P];
  __device__ __forceinline__ void load(const int* __restrict__ idx, int left) {
#pragma unroll
    for (int u = 0; u < P; ++u) c[u] = u < left ? ld_stream(idx + u * 32) : 0;
  }
};

// N entry rows: the lane's `left` entries' values from `val` on, gathered with get(c) and added with
// mac(v, g); `p` holds the piece's indices on entry and the next piece's on exit.
template <int N, typename G, int P, typename Get, typename Mac>
__device__ __forceinline__ void slice_piece(const double* __restrict__ val, int left,
                                            PieceIndices<P>& p, const int* next_idx, int next_left,
                                            Get get, Mac mac) {
  if constexpr (N <= P) {
    double v[N > 0 ? N : 1];
    G g[N > 0 ? N : 1];
#pragma unroll
    for (int u = 0; u < N; ++u) {
      const bool in = u < left;
      v[u] = in ? ld_stream(val + u * 32) : 0.0;
      g[u] = in ? get(p.c[u]) : G{};
    }
    p.load(next_idx, next_left);
#pragma unroll
    for (int u = 0; u < N; ++u) mac(v[u], g[u]);
  }
}

// A lane's `len` entries of a slice `width` entry rows wide, the first at idx / val; `p` as above,
// (next_idx, next_left) the first piece of what the warp sums next.
template <typename G, int P, typename Get, typename Mac>
__device__ __forceinline__ void slice_sum(const int* idx, const double* val, int len, int width,
                                          PieceIndices<P>& p, const int* next_idx, int next_left,
                                          Get get, Mac mac) {
  static_assert(P <= 8, "a case per count");
  int k = 0;
  do {
    const bool more = k + P < width;
    const int* ni = more ? idx + (k + P) * 32 : next_idx;
    const int nl = more ? len - k - P : next_left;
    const double* v = val + k * 32;
    const int left = len - k;
    switch (min(width - k, P)) {
      case 0: p.load(ni, nl); break;
      case 1: slice_piece<1, G>(v, left, p, ni, nl, get, mac); break;
      case 2: slice_piece<2, G>(v, left, p, ni, nl, get, mac); break;
      case 3: slice_piece<3, G>(v, left, p, ni, nl, get, mac); break;
      case 4: slice_piece<4, G>(v, left, p, ni, nl, get, mac); break;
      case 5: slice_piece<5, G>(v, left, p, ni, nl, get, mac); break;
      case 6: slice_piece<6, G>(v, left, p, ni, nl, get, mac); break;
      case 7: slice_piece<7, G>(v, left, p, ni, nl, get, mac); break;
      default: slice_piece<8, G>(v, left, p, ni, nl, get, mac); break;
    }
    k += P;
  } while (k < width);
}

// A lane's place in slice s of a layout: its meta word and the slice's first entry.
struct SlicePlace {
  unsigned m;
  size_t at;
  int len;
  __device__ __forceinline__ void load(const SliceSet& S, int s, int s1) {
    const int lane = static_cast<int>(threadIdx.x) & 31;
    m = kNoRow;
    at = 0;
    if (s < s1) {
      m = __ldg(S.meta + static_cast<size_t>(s) * 32 + lane);
      at = static_cast<size_t>(__ldg(S.base + s)) * 32 + lane;
    }
    len = m != kNoRow ? static_cast<int>(m >> 8) : 0;
  }
};

// What a warp holds of its first slice when its kernel starts to wait for the ones before it.
template <int P>
struct SliceStart {
  int s, s1;
  SlicePlace place;
  PieceIndices<P> indices;
};

template <int P>
__device__ __forceinline__ void start_slices(const SliceSet& S, SliceStart<P>& st) {
  st.s = __ldg(S.block_start + blockIdx.x) + (static_cast<int>(threadIdx.x) >> 5);
  st.s1 = __ldg(S.block_start + blockIdx.x + 1);
  st.place.load(S, st.s, st.s1);
  st.indices.load(S.idx + st.place.at, st.place.len);
}

// One long item, by the whole warp.
constexpr int kSliceBatch = 8;

template <int NP, int NR, typename G, typename Get, typename Mac, typename Load, typename Epi,
          typename Finish>
__device__ __forceinline__ void slice_item(const SliceSet& S, const SliceItem& it,
                                           double* chunk_part, Get get, Mac mac, Load load,
                                           Epi epi, Finish finish) {
  const int lane = static_cast<int>(threadIdx.x) & 31;
  const int* __restrict__ ip = S.idx + S.long_base + it.begin;
  const double* __restrict__ vp = S.val + S.long_base + it.begin;
  double ops[NR > 0 ? NR : 1];
  if (it.slot < 0 && lane == 0) load(it.row, ops);
  double acc[NP];
#pragma unroll
  for (int q = 0; q < NP; ++q) acc[q] = 0.0;
  for (int k = lane; k < it.count; k += 32 * kSliceBatch) {
    int c[kSliceBatch];
    double v[kSliceBatch];
#pragma unroll
    for (int u = 0; u < kSliceBatch; ++u) {
      const bool in = k + 32 * u < it.count;
      c[u] = in ? ld_stream(ip + k + 32 * u) : -1;
      v[u] = in ? ld_stream(vp + k + 32 * u) : 0.0;
    }
    G g[kSliceBatch];
#pragma unroll
    for (int u = 0; u < kSliceBatch; ++u) g[u] = c[u] >= 0 ? get(c[u]) : G{};
#pragma unroll
    for (int u = 0; u < kSliceBatch; ++u) mac(v[u], g[u], acc);
  }
  __syncwarp();
#pragma unroll
  for (int q = 0; q < NP; ++q) acc[q] = warp_sum(acc[q]);
  if (it.slot < 0) {
    if (lane == 0) epi(it.row, acc, ops);
    return;
  }
  if (lane == 0) {
#pragma unroll
    for (int q = 0; q < NP; ++q) chunk_part[it.slot * NP + q] = acc[q];
  }
  if (S.tickets == nullptr) return;
  const LongRow lr = S.longs[it.longs];
  int last = 0;
  if (lane == 0) {
    __threadfence();
    last = atomicAdd(S.tickets + it.longs, 1u) == static_cast<unsigned>(lr.nchunks - 1);
  }
  if (!__shfl_sync(0xffffffffu, last, 0)) return;
  __threadfence();
#pragma unroll
  for (int q = 0; q < NP; ++q) {
    acc[q] = 0.0;
    for (int c = lane; c < lr.nchunks; c += 32) acc[q] += __ldcg(chunk_part + (lr.chunk0 + c) * NP + q);
    acc[q] = warp_sum(acc[q]);
  }
  if (lane == 0) {
    S.tickets[it.longs] = 0u;
    load(it.row, ops);
    finish(it.longs, it.row, acc, ops);
  }
}

// Visit this block's rows (a multiple of 32 threads; every thread calls it):
//   fetch(c) reads element c of the gathered vector from global memory; where the layout has
//   windows they are staged from `vec`, the same vector
//   mac(v, g, acc) adds the entry's products
//   load(row, ops), epi(row, acc, ops) the row's NR operands and its epilogue
//   finish(l, row, acc, ops) the epilogue of row l of S.longs, where S.tickets is set. Which warp runs
//   it varies, so what it adds to a sum goes to a place of its own.
// WIN is false in kernels that stage no window whatever the layout has. Returns false -- in
// every thread -- if a wait gave up (only a staged window waits).
struct NoFinish {
  template <typename... Args>
  __device__ __forceinline__ void operator()(Args...) const {}
};

template <bool WIN, int NP, int NR, typename G, int P, typename Fetch, typename Mac, typename Load,
          typename Epi, typename Finish = NoFinish>
__device__ __forceinline__ bool run_slices(const SliceSet& S, SliceStart<P>& st, const G* vec,
                                           Fetch fetch, unsigned char* dsmem, double* chunk_part,
                                           Mac mac, Load load, Epi epi, Finish finish = Finish()) {
  __shared__ volatile int s_abort;
  const int W = static_cast<int>(blockDim.x) >> 5;
  const int warp = static_cast<int>(threadIdx.x) >> 5;
  uint64_t* bar = reinterpret_cast<uint64_t*>(dsmem);
  G* win = reinterpret_cast<G*>(dsmem + kSliceBarBytes);
  const bool windowed = WIN && S.wmax > 0;
  if (windowed) {
    if (threadIdx.x == 0) {
      s_abort = 0;
      mbar_init(bar, 1);
      fence_mbar_init();
    }
    __syncthreads();
  }
  bool pending = false;  // thread 0: a copy issued and not yet seen complete
  uint32_t phase = 0;
  // Without windows a block's slices are one segment.
  const int g0 = windowed ? __ldg(S.seg_start + blockIdx.x) : 0;
  const int g1 = windowed ? __ldg(S.seg_start + blockIdx.x + 1) : 1;
  bool ok = true;
  int s = st.s;
  SlicePlace p = st.place;
  PieceIndices<P> ix = st.indices;
  for (int g = g0; g < g1; ++g) {
    const SliceSeg sg = windowed ? S.segs[g] : SliceSeg{0, st.s1, 0, 0};
    if (WIN && sg.len > 0) {
      if (g != g0) __syncthreads();  // every warp is done with the window held
      if (threadIdx.x == 0) {
        const uint32_t bytes = static_cast<uint32_t>(sg.len) * static_cast<uint32_t>(sizeof(G));
        fence_proxy_async_smem();
        mbar_arrive_expect_tx(bar, bytes);
        bulk_copy_g2s(win, vec + sg.lo, bytes, bar);
        pending = true;
      }
      if (mbar_wait_or_abort(bar, phase, &s_abort)) {
        pending = false;
      } else {
        s_abort = 1;
      }
      phase ^= 1u;
      __syncthreads();
      ok = s_abort == 0;
    }
    if (!ok) break;
    const int lo = sg.lo;
    const unsigned wlen = static_cast<unsigned>(sg.len);
    auto get = [&](int c) {
      const unsigned o = static_cast<unsigned>(c - lo);
      return WIN && o < wlen ? win[o] : fetch(c);
    };
    if (g == g0) {
      for (int i = static_cast<int>(blockIdx.x) + warp * S.grid; i < S.nitems; i += W * S.grid) {
        slice_item<NP, NR, G>(S, S.items[i], chunk_part, get, mac, load, epi, finish);
      }
    }
    for (; s < sg.s1; s += W) {
      const bool has = p.m != kNoRow;
      const int row = slice_row(s, p.m);
      SlicePlace next;  // on its way while this slice is summed
      next.load(S, s + W, st.s1);
      double ops[NR > 0 ? NR : 1];
      if (has) load(row, ops);
      double acc[NP];
#pragma unroll
      for (int q = 0; q < NP; ++q) acc[q] = 0.0;
      const int width = __shfl_sync(0xffffffffu, p.len, 0);  // lane 0 holds the longest row
      slice_sum<G>(S.idx + p.at, S.val + p.at, p.len, width, ix, S.idx + next.at, next.len, get,
                   [&](double v, G gv) { mac(v, gv, acc); });
      if (has) epi(row, acc, ops);
      p = next;
    }
  }
  if (!windowed || ok) return true;
  // A window copy still in flight must land too (bounded).
  if (threadIdx.x == 0 && pending) mbar_wait_bounded(bar, phase ^ 1u);
  __syncthreads();
  return false;
}

// ---- Resident solves ----------------------------------------------------------------------
// Small problems run many steps in one RESIDENT kernel, a cluster of up to kResidentBlocks blocks.
// A block keeps in shared memory its slices' entries and its items' data and state, and a copy of
// each gathered vector, which the blocks write into one another's shared memory; they meet at the
// cluster barrier between the passes. No step touches global memory, where the other path
// launches two kernels (a step of 50 x 100 took 25 us so). The blocks of such a layout are the
// cluster's.
constexpr int kResidentBlocks = 16;
constexpr int kResidentThreads = 512;

// Blocks of the cluster for sides of `cols` and `rows` slices: four slices a block, one for each of
// an SM's FP64 units, before another SM is taken.
inline int resident_blocks(int cols, int rows) {
  int blocks = 1;
  while (blocks < kResidentBlocks && 4 * blocks < std::max(cols, rows)) blocks *= 2;
  return blocks;
}

// A block's slices of one layout in shared memory: the entries (indices as 16 bits), and per slice
// the first entry row, per slot the meta word.
struct LocalSlices {
  double* val;
  unsigned short* idx;
  unsigned short* meta;
  int* base;
  int s0, n;  // the block's first slice, its slices
};

// Bytes of a block's LocalSlices with `rows` entry rows and `slices` slices.
__host__ __device__ inline int local_slices_bytes(int rows, int slices) {
  return rows * 32 * 10 + slices * 32 * 2 + ((slices + 4) & ~3) * 4;
}

// Lays L out at `mem` and fills it; every thread calls it. Returns the first byte after it.
__device__ __forceinline__ unsigned char* fill_local(const SliceSet& S, LocalSlices& L,
                                                     unsigned char* mem) {
  L.s0 = S.block_start[blockIdx.x];
  L.n = S.block_start[blockIdx.x + 1] - L.s0;
  const unsigned first = S.base[L.s0], rows = S.base[L.s0 + L.n] - first;
  L.val = reinterpret_cast<double*>(mem);
  L.base = reinterpret_cast<int*>(L.val + rows * 32);
  L.idx = reinterpret_cast<unsigned short*>(L.base + ((L.n + 4) & ~3));
  L.meta = L.idx + rows * 32;
  const int T = static_cast<int>(blockDim.x), t = static_cast<int>(threadIdx.x);
  const size_t at = static_cast<size_t>(first) * 32;
  for (int k = t; k < static_cast<int>(rows) * 32; k += T) {
    L.val[k] = S.val[at + k];
    L.idx[k] = static_cast<unsigned short>(S.idx[at + k]);
  }
  for (int k = t; k < L.n * 32; k += T) L.meta[k] = S.meta[static_cast<size_t>(L.s0) * 32 + k];
  for (int k = t; k <= L.n; k += T) L.base[k] = static_cast<int>(S.base[L.s0 + k] - first);
  return reinterpret_cast<unsigned char*>(L.meta + L.n * 32);
}

// Last block only: the rows of several pieces, each combined from its partials in order.
template <int NP, int NR, typename Load, typename Epi>
__device__ __forceinline__ void run_slice_long_rows(const SliceSet& S, const double* chunk_part,
                                                    Load load, Epi epi) {
  for (int l = threadIdx.x; l < S.nlong; l += blockDim.x) {
    const LongRow lr = S.longs[l];
    double acc[NP];
#pragma unroll
    for (int q = 0; q < NP; ++q) acc[q] = 0.0;
    for (int c = 0; c < lr.nchunks; ++c) {
#pragma unroll
      for (int q = 0; q < NP; ++q) acc[q] += __ldcg(chunk_part + (lr.chunk0 + c) * NP + q);
    }
    double ops[NR > 0 ? NR : 1];
    load(lr.row, ops);
    epi(lr.row, acc, ops);
  }
}

}  // namespace sgb
