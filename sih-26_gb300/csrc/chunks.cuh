// chunks.cuh -- warp chunks: the sparse-product engine of the PDHG step passes.
//
// A CHUNK is a run of at most kChunkRows consecutive rows (of the CSR copy, or columns of the
// CSC copy) holding at most CH nonzeros; a row longer than CH is cut into PIECES of CH
// entries. Each warp of a block works through its own chunks, one at a time, with no
// barrier between warps:
//   1. its lanes load the chunk's indices and values straight from global memory, and the per-row
//      operands of the epilogue, lane l taking row r0 + l. Where the windows hold all entries they
//      are PACKED for this: kChunkCapF places a chunk, lane l's eight (entries l, l + 32, ...) in
//      runs of 16 bytes a lane, indices as 16 bits from the window's start, so three loads bring
//      what takes sixteen of 4 bytes, and the next chunk's entries are on their way from when this
//      one's are staged (asked for earlier they take registers that spill: 54.4 ms against 51.7 for
//      400 iterations of the block-angular LP of 1M x 2M with nine entries a column). Elsewhere the
//      loads are the sixteen, less those past the chunk's end;
//   2. they gather the vector entry of each nonzero -- from the block's staged WINDOW of the
//      vector in shared memory, or from L2 when the window does not hold it -- and stage the
//      products in the warp's shared buffer;
//   3. `L` lanes per row (the largest power of two with 32 / L >= rows) sum each row from
//      the buffer, in a fixed order (lane s takes entries s, s + L, ...; then a fixed
//      xor tree), and the row's first lane runs the epilogue with the operands shuffled to
//      it. A piece of a long row is summed by the whole warp into a piece partial; the last
//      block of the kernel combines the pieces of each long row in order.
// The stream loads of every warp in flight at once are what keep HBM busy: registers hold
// them, so shared memory is left to the window.
//
// WINDOWS. Random 4- or 8-byte gathers from L2 cost one 32-byte sector request each, and an
// SM retires about one sector request per clock: far below what the streamed matrix needs.
// So a block keeps a slice [lo, lo + len) of the gathered vector in shared memory, copied in
// by one bulk copy (cp.async.bulk) whenever its chunks move to another slice. A block owns
// a contiguous run of chunks; chunks that share a slice form a SEGMENT; the block stages each
// segment's slice in turn. Blocks are cut by a cost model (entries, plus a fixed cost per
// slice staged) so that a block that must stage two slices takes fewer entries.
//
// SPLIT LAYOUTS. A gather that misses the window stalls its whole warp on L2 latency, and in
// a chunk of 256 entries almost every warp-wide gather has a lane that misses when even 8% of
// the entries fall outside. So where a window covers most but not all of a layout's entries,
// the layout is split: the entries inside each row's window form the main matrix (gathered
// from shared memory only), the rest an OUTER matrix of their own. Each block first sums the
// outer entries of its own rows (plain L2 gathers, while its first window copy is in flight)
// into outer[row], and the main loop adds outer[row] to each row's sum before its epilogue.
//
// Every wait is bounded: a wait that gives up raises the block's abort flag, the remaining
// chunks are skipped, the copy still in flight is given a bounded time to land, and the
// caller records the error.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "tiles.cuh"

namespace sgb {

constexpr int kChunkRows = 31;     // rows per chunk (lane 31 reads the closing row pointer)
constexpr int kChunkCapF = 256;    // entries per chunk, FP32 layouts
constexpr int kChunkThreads = 1024;
// The largest window a chunk kernel stages. Shared memory and L1 share each SM's 256 KB, and
// the step passes' per-row operand and row-pointer loads go through L1: on the 1M x 2M
// block-angular LP the FP32 column pass ran in 61 us with a 128 KB window and in 84 us with
// the 160 KB that fits beside the warp buffers (the row pass: 89 us against 104 us).
constexpr int kWindowBytesMax = 128 * 1024;

// Consecutive chunks of one block that gather from the same staged slice [lo, lo + len) of
// the vector (len = 0: no slice, every gather from global memory).
struct ChunkSeg {
  int c0, c1;
  int lo, len;
};

// A chunk record is a Tile: rows [r0, r1), entries [k0, k1); r1 < 0 marks a piece of a long
// row whose partial goes to piece slot -r1 - 1.
struct ChunkSet {
  const int* ptr;        // rows + 1 (main part)
  const int* idx;        // nnz (+ kPad): the pieces' entries
  const float* val;      // nnz (+ kPad)
  int narrow;            // the windows hold every entry of the chunks of whole rows, so these are packed:
  const float* pval;     // values, kChunkCapF per chunk,
  const unsigned short* pidx;  // indices from the window's start
  const Tile* chunks;
  const ChunkSeg* segs;
  const int* seg_start;  // per block: its segments [seg_start[b], seg_start[b + 1])
  const LongRow* longs;  // long rows and their piece slots
  int nlong;
  int npieces;
  int nrows;
  int wmax;              // window capacity in gathered elements (0: the layout stages none)
  // Split layouts: the out-of-window entries as a CSR of their own. Block b sums the outer
  // entries of its rows in ROUNDS (row ranges orounds[oround_start[b] .. oround_start[b + 1]),
  // each with at most as many outer entries as the block's warp buffers hold); outer holds
  // a sum per row. A round's entries are stored by column, opos their places in the order of the
  // rows (a round's start is optr of its first row).
  const int* optr;
  const int* oidx;
  const float* oval;
  const unsigned short* opos;
  const int2* orounds;
  const int* oround_start;
  float* outer;          // nullptr: not split
};

// ---- PTX helpers ---------------------------------------------------------------------------
__device__ __forceinline__ int ld_stream(const int* p) {
  int v;
  asm volatile("ld.global.nc.L1::no_allocate.b32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float ld_stream(const float* p) {
  float v;
  asm volatile("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ double ld_stream(const double* p) {
  double v;
  asm volatile("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}

__device__ __forceinline__ float4 ld_stream(const float4* p) {
  float4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "l"(p));
  return v;
}
__device__ __forceinline__ uint4 ld_stream(const uint4* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

// Dynamic shared memory of a chunk kernel: per-warp buffers of products (half the shared-memory
// traffic of value and gathered element), the window barrier, the window.
constexpr int kChunkBufBytes = kChunkCapF * static_cast<int>(sizeof(float));
__host__ __device__ constexpr int chunk_smem(int warps, int wmax) {
  return warps * kChunkBufBytes + 128 + ((wmax * static_cast<int>(sizeof(float)) + 127) & ~127);
}

// Lanes per row for a chunk of R rows: the largest power of two L with 32 / L >= R.
__device__ __forceinline__ int chunk_lanes(int R) {
  const int p = R <= 1 ? 0 : 32 - __clz(R - 1);  // the smallest p with 2^p >= R
  return 32 >> p;
}

// A lane's eight entries of a chunk: packed, or (index -1 past the chunk's end) as the layout has them.
// With 32-bit indices packing does not pay: most chunks of real LPs' columns, two to five entries each,
// are half empty (400 iterations of a block-angular LP of 1M x 2M at two, three and five entries a
// column: 44.2, 44.2 and 46.7 ms, packed 49.4, 48.6 and 49.8).
template <bool NARROW>
struct ChunkEntries {
  static constexpr int kEach = kChunkCapF / 32;
  static_assert(kEach == 8, "two float4 and a uint4 a lane");
  float a[kEach];
  int c[kEach];
  __device__ __forceinline__ void load(const ChunkSet& cs, int, const Tile& ch) {
    const int lane = static_cast<int>(threadIdx.x) & 31, n = ch.k1 - ch.k0;
#pragma unroll
    for (int j = 0; j < kEach; ++j) {
      const int k = lane + 32 * j;
      c[j] = k < n ? ld_stream(cs.idx + ch.k0 + k) : -1;
      a[j] = k < n ? ld_stream(cs.val + ch.k0 + k) : 0.0f;
    }
  }
  __device__ __forceinline__ void unpack(float (&va)[kEach], int (&vc)[kEach]) const {
#pragma unroll
    for (int j = 0; j < kEach; ++j) {
      va[j] = a[j];
      vc[j] = c[j];
    }
  }
};

template <>
struct ChunkEntries<true> {
  static constexpr int kEach = kChunkCapF / 32;
  float4 a0, a1;
  uint4 x0;
  __device__ __forceinline__ void load(const ChunkSet& cs, int chunk, const Tile&) {
    const int lane = static_cast<int>(threadIdx.x) & 31;
    const float4* v = reinterpret_cast<const float4*>(cs.pval) + static_cast<size_t>(chunk) * 64 + lane;
    a0 = ld_stream(v);
    a1 = ld_stream(v + 32);
    x0 = ld_stream(reinterpret_cast<const uint4*>(cs.pidx) + static_cast<size_t>(chunk) * 32 + lane);
  }
  __device__ __forceinline__ void unpack(float (&a)[kEach], int (&c)[kEach]) const {
    a[0] = a0.x, a[1] = a0.y, a[2] = a0.z, a[3] = a0.w;
    a[4] = a1.x, a[5] = a1.y, a[6] = a1.z, a[7] = a1.w;
    const unsigned w[4] = {x0.x, x0.y, x0.z, x0.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      c[2 * j] = static_cast<int>(w[j] & 0xffffu);
      c[2 * j + 1] = static_cast<int>(w[j] >> 16);
    }
  }
};

// One chunk of whole rows: gather, stage, sum, epilogue (all lanes of the warp call it).
//   gather(c) -> float        the vector element of the entries' index c
//   ahead()                   once the entries are staged: their registers are free
//   load(row, ops)            the row's NR epilogue operands (lane-per-row, at chunk start)
//   epi(row, sums, ops)       once per row, on the row's first lane
template <int NR, bool NARROW, bool OUTER, typename Gather, typename Ahead, typename Load,
          typename Epi>
__device__ __forceinline__ void chunk_step(const int* __restrict__ ptr, const Tile& ch,
                                           const ChunkEntries<NARROW>& e, float* buf,
                                           const float* outer, Gather gather, Ahead ahead,
                                           Load load, Epi epi) {
  constexpr int J = kChunkCapF / 32;
  const int lane = static_cast<int>(threadIdx.x) & 31;
  const int R = ch.r1 - ch.r0;
  int pr = 0;
  float ops[NR > 0 ? NR : 1];
  float out = 0.0f;
  if (lane <= R) pr = __ldg(ptr + ch.r0 + lane);
  if (lane < R) {
    load(ch.r0 + lane, ops);
    if (OUTER) out = outer[ch.r0 + lane];
  }
  {
    float a[J];
    int c[J];
    e.unpack(a, c);
    // Past the chunk's end the entry is a zero that no row reads.
#pragma unroll
    for (int j = 0; j < J; ++j) {
      buf[lane + 32 * j] = NARROW || c[j] >= 0 ? __fmul_rn(a[j], gather(c[j])) : 0.0f;
    }
  }
  ahead();
  __syncwarp();
  const int L = chunk_lanes(R);
  const int g = lane / L, sub = lane & (L - 1);
  const int ra = __shfl_sync(0xffffffffu, pr, g & 31) - ch.k0;
  const int re = __shfl_sync(0xffffffffu, pr, (g + 1) & 31) - ch.k0;
  float s[1] = {0.0f};
  if (g < R) {
#pragma unroll 4
    for (int k = ra + sub; k < re; k += L) s[0] = s[0] + buf[k];
  }
  for (int o = L >> 1; o > 0; o >>= 1) s[0] += __shfl_xor_sync(0xffffffffu, s[0], o);
  float og[NR > 0 ? NR : 1];
#pragma unroll
  for (int q = 0; q < NR; ++q) og[q] = __shfl_sync(0xffffffffu, ops[q], g & 31);
  if (OUTER) s[0] += __shfl_sync(0xffffffffu, out, g & 31);
  if (g < R && sub == 0) epi(ch.r0 + g, s, og);
  __syncwarp();
}

// A piece of a long row: entries l, l + 32, ... per lane, products rounded before they are added.
template <typename Gather>
__device__ __forceinline__ void chunk_piece(const ChunkSet& cs, const Tile& ch, double* piece_part,
                                            Gather gather) {
  const int lane = static_cast<int>(threadIdx.x) & 31;
  float s = 0.0f;
#pragma unroll 4
  for (int k = ch.k0 + lane; k < ch.k1; k += 32) {
    s = __fadd_rn(s, __fmul_rn(ld_stream(cs.val + k), gather(ld_stream(cs.idx + k))));
  }
  const double d = warp_sum(static_cast<double>(s));
  if (lane == 0) piece_part[-ch.r1 - 1] = d;
}

// The outer sums of a split layout's rows, for this block: in each round, every thread takes
// outer entries e, e + blockDim, ... of the round's contiguous entry range (coalesced loads,
// gathers from global memory) and stages their products in the warp buffers at their places, then
// every thread sums the rows r, r + blockDim, ... of the round in entry order into outer[r].
// All threads call it; it ends with the block synchronised. An SM looks up about one line per clock,
// and 32 random columns are 32 lines: by column, a warp's gathers fall on a few (1M x 2M
// block-angular LP, 48% of the row pass's entries outside its windows: 79 us a pass in row order).
// LIVE: the running kernel writes the vector (ld_live).
template <bool LIVE>
__device__ __forceinline__ float element(const float* p) {
  return LIVE ? ld_live(p) : __ldg(p);
}

template <bool LIVE>
__device__ __forceinline__ void outer_sums(const ChunkSet& cs, const float* vec, float* stage) {
  const int B = static_cast<int>(blockDim.x);
  const int t = static_cast<int>(threadIdx.x);
  for (int q0 = cs.oround_start[blockIdx.x]; q0 < cs.oround_start[blockIdx.x + 1]; ++q0) {
    const int2 rr = cs.orounds[q0];
    const int e0 = __ldg(cs.optr + rr.x), e1 = __ldg(cs.optr + rr.y);
    const int count = e1 - e0;
    // A thread takes kOuterBatch entries at a time and issues all their index and value loads,
    // then all their gathers, so it waits for two latencies per batch, not two per entry.
    constexpr int kOuterBatch = 8;
    for (int k0 = t; k0 < count; k0 += B * kOuterBatch) {
      int ix[kOuterBatch], at[kOuterBatch];
      float av[kOuterBatch], g[kOuterBatch];
#pragma unroll
      for (int u = 0; u < kOuterBatch; ++u) {
        const int k = k0 + u * B;
        ix[u] = k < count ? ld_stream(cs.oidx + e0 + k) : -1;
        av[u] = k < count ? ld_stream(cs.oval + e0 + k) : 0.0f;
        at[u] = k < count ? __ldg(cs.opos + e0 + k) : 0;
      }
#pragma unroll
      for (int u = 0; u < kOuterBatch; ++u) g[u] = ix[u] >= 0 ? element<LIVE>(vec + ix[u]) : 0.0f;
#pragma unroll
      for (int u = 0; u < kOuterBatch; ++u) {
        const int k = k0 + u * B;
        if (k >= count) break;
        stage[at[u]] = __fmul_rn(av[u], g[u]);
      }
    }
    __syncthreads();
    for (int r = rr.x + t; r < rr.y; r += B) {
      const int a0 = __ldg(cs.optr + r) - e0, a1 = __ldg(cs.optr + r + 1) - e0;
      float s = 0.0f;
      for (int k = a0; k < a1; ++k) s = s + stage[k];
      cs.outer[r] = s;
    }
    __syncthreads();
  }
}

// Starts a window's copy (thread 0). What the block has read of the buffer, and in a LIVE kernel what
// others wrote of the vector, comes before it.
template <bool LIVE>
__device__ __forceinline__ void copy_window(float* win, const float* vec, const ChunkSeg& sg,
                                            uint64_t* bar) {
  if (LIVE) {
    asm volatile("fence.proxy.async;" ::: "memory");
  } else {
    fence_proxy_async_smem();
  }
  mbar_arrive_expect_tx(bar, static_cast<uint32_t>(sg.len) * sizeof(float));
  bulk_copy_g2s(win, vec + sg.lo, static_cast<uint32_t>(sg.len) * sizeof(float), bar);
}

template <bool LIVE, bool NARROW, bool OUTER, int NR, typename Load, typename Epi>
__device__ __forceinline__ bool run_chunks_impl(const ChunkSet& cs, const float* vec,
                                                unsigned char* dsmem, double* piece_part,
                                                Load load, Epi epi) {
  __shared__ volatile int s_abort;
  const int W = static_cast<int>(blockDim.x) >> 5;
  const int warp = static_cast<int>(threadIdx.x) >> 5;
  float* buf = reinterpret_cast<float*>(dsmem + warp * kChunkBufBytes);
  uint64_t* winbar = reinterpret_cast<uint64_t*>(dsmem + W * kChunkBufBytes);
  float* win = reinterpret_cast<float*>(dsmem + W * kChunkBufBytes + 128);
  if (threadIdx.x == 0) {
    s_abort = 0;
    mbar_init(winbar, 1);
    fence_mbar_init();
  }
  __syncthreads();
  const int s0 = cs.seg_start[blockIdx.x], s1 = cs.seg_start[blockIdx.x + 1];
  uint32_t phase = 0;
  bool pending = false;  // thread 0: a window copy issued and not yet seen complete

  // The first window copy is issued at once; a split layout sums its outer entries while it
  // is in flight.
  if (s0 < s1 && cs.segs[s0].len > 0 && threadIdx.x == 0) {
    copy_window<LIVE>(win, vec, cs.segs[s0], winbar);
    pending = true;
  }
  if (OUTER) outer_sums<LIVE>(cs, vec, reinterpret_cast<float*>(dsmem));

  for (int s = s0; s < s1; ++s) {
    const ChunkSeg sg = cs.segs[s];
    // The warp's first chunk of the segment is on its way while the window is.
    Tile ch{0, 0, 0, 0};
    ChunkEntries<NARROW> e;
    if (sg.c0 + warp < sg.c1) {
      if (NARROW) e.load(cs, sg.c0 + warp, ch);
      ch = cs.chunks[sg.c0 + warp];
    }
    if (sg.len > 0) {
      if (s != s0) {
        __syncthreads();  // every warp is done with the slice held
        if (!s_abort && threadIdx.x == 0) {
          copy_window<LIVE>(win, vec, sg, winbar);
          pending = true;
        }
      }
      if (!s_abort) {
        if (mbar_wait_or_abort(winbar, phase, &s_abort)) {
          if (threadIdx.x == 0) pending = false;
        } else {
          s_abort = 1;
        }
      }
      phase ^= 1u;
    }
    const int lo = sg.lo, len = sg.len;
    // Of column c, and of an entry's index c.
    auto gather_column = [&](int c) {
      const unsigned o = static_cast<unsigned>(c - lo);
      return o < static_cast<unsigned>(len) ? win[o] : element<LIVE>(vec + c);
    };
    auto gather = [&](int c) { return NARROW ? win[c] : gather_column(c); };
    for (int c = sg.c0 + warp; c < sg.c1; c += W) {
      if (s_abort) break;
      Tile next{0, 0, 0, 0};
      if (!NARROW && ch.r1 >= 0) e.load(cs, c, ch);
      if (c + W < sg.c1) next = cs.chunks[c + W];
      const auto ahead = [&] {
        if (NARROW && c + W < sg.c1) e.load(cs, c + W, next);
      };
      if (!LIVE && ch.r1 < 0) {
        chunk_piece(cs, ch, piece_part, gather_column);
        ahead();
      } else {
        chunk_step<NR, NARROW, OUTER>(cs.ptr, ch, e, buf, cs.outer, gather, ahead, load, epi);
      }
      ch = next;
    }
  }
  __syncthreads();
  const bool ok = s_abort == 0;
  // A window copy still in flight must land before the block exits (bounded). The next pass of the
  // kernel initialises the barrier again.
  if (threadIdx.x == 0) {
    if (!ok && pending) mbar_wait_bounded(winbar, phase ^ 1u);
    if (ok) asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_addr(winbar)) : "memory");
  }
  __syncthreads();
  return ok;
}

// Visit this block's chunks (kernel launched with a multiple of 32 threads, every thread
// calls it): NARROW as cs.narrow says, OUTER where cs.outer is not null, a kernel per form. Returns false
// -- in every thread -- if a wait gave up.
template <bool NARROW, bool OUTER, int NR, typename Load, typename Epi>
__device__ __forceinline__ bool run_chunks(const ChunkSet& cs, const float* vec,
                                           unsigned char* dsmem, double* piece_part, Load load,
                                           Epi epi) {
  return run_chunks_impl<false, NARROW, OUTER, NR>(cs, vec, dsmem, piece_part, load, epi);
}

// The same in a kernel that writes the vector itself, for layouts of narrow indices without pieces or
// outer entries.
template <int NR, typename Load, typename Epi>
__device__ __forceinline__ bool run_whole_chunks(const ChunkSet& cs, const float* vec,
                                                 unsigned char* dsmem, Load load, Epi epi) {
  return run_chunks_impl<true, true, false, NR>(cs, vec, dsmem, nullptr, load, epi);
}

// Last block only: each long row combined from its piece partials in piece order (double),
// then handed to the epilogue with its operands.
template <int NR, typename Load, typename Epi>
__device__ __forceinline__ void run_chunk_long_rows(const ChunkSet& cs, const double* piece_part,
                                                    Load load, Epi epi) {
  for (int l = threadIdx.x; l < cs.nlong; l += blockDim.x) {
    const LongRow lr = cs.longs[l];
    double acc = 0.0;
    for (int c = 0; c < lr.nchunks; ++c) acc += __ldcg(piece_part + lr.chunk0 + c);
    const float s[1] = {static_cast<float>(acc)};
    float ops[NR > 0 ? NR : 1];
    load(lr.row, ops);
    epi(lr.row, s, ops);
  }
}

}  // namespace sgb
