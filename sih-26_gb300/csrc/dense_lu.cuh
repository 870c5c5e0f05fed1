// dense_lu.cuh -- FP32 LU factors of a basis matrix, by one block, for FP64 refinement.
//
// A basis of up to kLuMost columns is factored densely in FP32 (P A = L U, partial pivoting) in the
// block's workspace in global memory, and its FP64 solves are refinement steps around the factors:
// the residual in FP64 from the sparse matrix, the correction from two triangular sweeps in FP32. A
// step divides the error by about 1 / (cond(A) 2^-24), so a well-conditioned basis takes three or
// four. FP32 has 64 times the rate of GB300's FP64 pipe, which conjugate gradients on A A' kept busy
// for thousands of iterations: 1,000 columns took 82 ms per LP so (its two solves, one SM).
//
// Right-looking in panels of kLuPanel columns:
//   panel    a thread holds two rows of the panel in registers; per column a pivot by integer maxima
//            of the magnitudes' bits, its row passed through shared memory, one rank-1 update; a
//            pivot that is tiny beside what its row and its column held at the start is rounding
//            (kLuPivotShare)
//   U block  a thread per column solves with the panel's unit lower triangle, kLuCols at a time
//   update   128 x 256 tiles, 8 x 8 a thread, L and U of the panel in shared memory
// Rows stay in place: piv[k] is the row of the k-th pivot, act the rows without one.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"

namespace sgb {

constexpr int kLuThreads = 512;
constexpr int kLuMost = 2 * kLuThreads;  // two panel rows a thread
constexpr int kLuPanel = 32;
constexpr int kLuCols = 512;
constexpr int kLuRow = kLuPanel + 4;  // floats of a row of the panel's triangle
// The factorisation is refused where the largest entry left in a column is about 2^-16 of the largest
// that the column, and of the largest that its row, held at the start, or less: 256 roundings of FP32.
// A basis that is singular to FP32 leaves such pivots. Refinement would still converge where the
// right-hand side lies in its range, to a solution with an arbitrary part from its null space, where
// the conjugate gradients find the nearest. Both shares are asked for, so that rows or columns of
// very different scale do not count as singular.
constexpr int kLuPivotShare = 16;  // its exponent, negated

__host__ __device__ inline int lu_size(int nb) { return (nb + kLuPanel - 1) / kLuPanel * kLuPanel; }

// Dynamic shared memory of a factorisation of n = lu_size() columns.
__host__ __device__ inline int lu_smem(int n) {
  return 4 * (2 * n + n / 2 + kLuPanel * kLuRow + kLuPanel * n + kLuPanel * (n < kLuCols ? n : kLuCols));
}

// The workspaces, of `each` bytes and one a block, of a launch that would have `blocks` blocks: with
// less than twice their memory free the launch has fewer blocks, so that which solves an LP gets, and
// their bits, do not depend on what else is on the device.
inline int lu_workspaces(int blocks, size_t each, size_t free_bytes) {
  const size_t fit = free_bytes / 2 / each;
  return static_cast<int>(std::max<size_t>(1, std::min<size_t>(fit, static_cast<size_t>(blocks))));
}

// The exponent field of v's size.
__device__ __forceinline__ unsigned char lu_exponent(float v) {
  return static_cast<unsigned char>(__float_as_uint(fabsf(v)) >> 23);
}

struct LuMem {
  int *piv, *act;
  float *l11, *lt, *ut;
  __device__ __forceinline__ LuMem(unsigned char* smem, int n)
      : piv(reinterpret_cast<int*>(smem)),
        act(piv + n),
        l11(reinterpret_cast<float*>(act + n + n / 2)),
        lt(l11 + kLuPanel * kLuRow),
        ut(lt + kLuPanel * n) {}
  // Exponents of the matrix's largest magnitudes by row and by column, between act and l11.
  __device__ __forceinline__ unsigned char* row_most(int n) const {
    return reinterpret_cast<unsigned char*>(act + n);
  }
  __device__ __forceinline__ unsigned char* col_most(int n) const { return row_most(n) + n; }
};

// Factors the n x n matrix at A (rows of n floats) in place; m.piv receives the pivot rows, m.row_most
// and m.col_most hold the exponents of the matrix's largest magnitudes. All threads call it; false,
// in all, where a column has no usable pivot.
static __device__ __noinline__ bool lu_factor(float* A, int n, LuMem m) {
  __shared__ unsigned s_max[2][kLuThreads / 32];
  __shared__ int s_who[2][kLuThreads / 32];
  __shared__ __align__(16) float s_row[2][kLuPanel];
  __shared__ int s_count[2][kLuThreads / 32];
  __shared__ int s_weak;
  if (threadIdx.x == 0) s_weak = 0;
  const int t = static_cast<int>(threadIdx.x), lane = t & 31, warp = t >> 5;
  constexpr int W = kLuThreads / 32;
  const int ldu = n < kLuCols ? n : kLuCols;
  for (int i = t; i < n; i += kLuThreads) m.act[i] = i;
  __syncthreads();
  int na = n;
  for (int k0 = 0; k0 < n; k0 += kLuPanel) {
    float v[2][kLuPanel];
    int row[2];
    bool live[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int a = t + q * kLuThreads;
      live[q] = a < na;
      row[q] = live[q] ? m.act[a] : -1;
#pragma unroll
      for (int j = 0; j < kLuPanel; j += 4) {
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (live[q]) x = *reinterpret_cast<const float4*>(A + static_cast<size_t>(row[q]) * n + k0 + j);
        v[q][j] = x.x;
        v[q][j + 1] = x.y;
        v[q][j + 2] = x.z;
        v[q][j + 3] = x.w;
      }
    }
#pragma unroll
    for (int c = 0; c < kLuPanel; ++c) {
      const unsigned b0 = live[0] ? __float_as_uint(fabsf(v[0][c])) : 0u;
      const unsigned b1 = live[1] ? __float_as_uint(fabsf(v[1][c])) : 0u;
      const unsigned most = __reduce_max_sync(0xffffffffu, b0 > b1 ? b0 : b1);
      const unsigned at0 = __ballot_sync(0xffffffffu, live[0] && b0 == most);
      const unsigned at1 = __ballot_sync(0xffffffffu, live[1] && b1 == most);
      if (lane == 0) {
        s_max[c & 1][warp] = most;
        s_who[c & 1][warp] = at0 != 0u   ? 2 * (warp * 32 + __ffs(at0) - 1)
                             : at1 != 0u ? 2 * (warp * 32 + __ffs(at1) - 1) + 1
                                         : -1;
      }
      __syncthreads();
      const unsigned mine = lane < W ? s_max[c & 1][lane] : 0u;
      const int whose = lane < W ? s_who[c & 1][lane] : -1;
      const unsigned top = __reduce_max_sync(0xffffffffu, mine);
      const unsigned from = __ballot_sync(0xffffffffu, whose >= 0 && mine == top);
      if (top == 0u || top >= 0x7f800000u || from == 0u) return false;
      const int who = __shfl_sync(0xffffffffu, whose, __ffs(from) - 1);
      if (t == who >> 1) {
        const bool second = (who & 1) != 0;
#pragma unroll
        for (int j = 0; j < kLuPanel; ++j) {
          const float x = second ? v[1][j] : v[0][j];
          if (j >= c) s_row[c & 1][j] = x;
          else m.l11[c * kLuRow + j] = x;
        }
        m.piv[k0 + c] = second ? row[1] : row[0];
        if (second) live[1] = false;
        else live[0] = false;
      }
      __syncthreads();
      const float inv = 1.0f / s_row[c & 1][c];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        if (!live[q]) continue;
        const float l = v[q][c] * inv;
        v[q][c] = l;
#pragma unroll
        for (int j = c + 1; j < kLuPanel; ++j) v[q][j] = fmaf(-l, s_row[c & 1][j], v[q][j]);
      }
    }
    // The panel goes back; the rows without a pivot close ranks, their multipliers in m.lt.
    unsigned stay[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      if (row[q] >= 0) {
#pragma unroll
        for (int j = 0; j < kLuPanel; j += 4) {
          *reinterpret_cast<float4*>(A + static_cast<size_t>(row[q]) * n + k0 + j) =
              make_float4(v[q][j], v[q][j + 1], v[q][j + 2], v[q][j + 3]);
        }
      }
      stay[q] = __ballot_sync(0xffffffffu, live[q]);
      if (lane == 0) s_count[q][warp] = __popc(stay[q]);
    }
    __syncthreads();
    if (t < kLuPanel) {  // the panel's pivots, kLuPivotShare
      const int at = m.piv[k0 + t];
      const int least = min(m.row_most(n)[at], m.col_most(n)[k0 + t]) - kLuPivotShare;
      if (lu_exponent(A[static_cast<size_t>(at) * n + k0 + t]) <= least) s_weak = 1;
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      if (!live[q]) continue;
      int at = __popc(stay[q] & ((1u << lane) - 1u));
      for (int w = 0; w < W; ++w) {
        if (q == 1) at += s_count[0][w];
        if (w < warp) at += s_count[q][w];
      }
      m.act[at] = row[q];
#pragma unroll
      for (int c = 0; c < kLuPanel; ++c) m.lt[c * n + at] = v[q][c];
    }
    na -= kLuPanel;
    __syncthreads();
    if (s_weak != 0) return false;
    for (int j0 = k0 + kLuPanel; j0 < n; j0 += kLuCols) {
      if (j0 + t < n) {
        float x[kLuPanel];
        float* const at = A + j0 + t;
#pragma unroll
        for (int c = 0; c < kLuPanel; ++c) x[c] = at[static_cast<size_t>(m.piv[k0 + c]) * n];
#pragma unroll
        for (int c = 0; c < kLuPanel; ++c) {
#pragma unroll
          for (int d = 0; d < c; ++d) x[c] = fmaf(-m.l11[c * kLuRow + d], x[d], x[c]);
          at[static_cast<size_t>(m.piv[k0 + c]) * n] = x[c];
          m.ut[c * ldu + t] = x[c];
        }
      }
      __syncthreads();
      const int lr = lane >> 3, lc = lane & 7;
      for (int c0 = (warp & 3) * 64; c0 < kLuCols; c0 += 256) {
        if (j0 + c0 >= n) break;
        const bool both = j0 + c0 + 32 < n;
        for (int r0 = (warp >> 2) * 32; r0 < na; r0 += 128) {
          float acc[8][8];
          float* at[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int r = r0 + lr * 4 + (i & 3) + (i >> 2) * 16;
            at[i] = r < na ? A + static_cast<size_t>(m.act[r]) * n + j0 + c0 + lc * 4 : nullptr;
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
            if (at[i] != nullptr) x = *reinterpret_cast<const float4*>(at[i]);
            if (at[i] != nullptr && both) y = *reinterpret_cast<const float4*>(at[i] + 32);
            acc[i][0] = x.x, acc[i][1] = x.y, acc[i][2] = x.z, acc[i][3] = x.w;
            acc[i][4] = y.x, acc[i][5] = y.y, acc[i][6] = y.z, acc[i][7] = y.w;
          }
          // With `both` false nothing is stored from the second group of columns.
          const float* lp = m.lt + r0 + lr * 4;
          const float* up = m.ut + c0 + lc * 4;
#pragma unroll 4
          for (int c = 0; c < kLuPanel; ++c, lp += n, up += ldu) {
            const float4 l0 = *reinterpret_cast<const float4*>(lp);
            const float4 l1 = *reinterpret_cast<const float4*>(lp + 16);
            const float4 u0 = *reinterpret_cast<const float4*>(up);
            const float4 u1 = both ? *reinterpret_cast<const float4*>(up + 32) : u0;
            const float l[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w};
            const float u[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
#pragma unroll
              for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(-l[i], u[j], acc[i][j]);
            }
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            if (at[i] == nullptr) continue;
            *reinterpret_cast<float4*>(at[i]) =
                make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
            if (both) {
              *reinterpret_cast<float4*>(at[i] + 32) =
                  make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
            }
          }
        }
      }
      __syncthreads();
    }
  }
  return true;
}

// y <- U^-1 L^-1 y (y in pivot order on entry, in column order on exit), all in shared memory but
// the factors. Blocks of 32: a warp per row takes the products with what is solved, one warp the
// triangle. All threads call it.
static __device__ __noinline__ void lu_sweeps(const float* A, int n, const int* piv, float* y) {
  __shared__ float s_part[kLuPanel];
  const int t = static_cast<int>(threadIdx.x), lane = t & 31, warp = t >> 5;
  constexpr int W = kLuThreads / 32;
  const int blocks = n / kLuPanel;
  for (int step = 0; step < 2 * blocks; ++step) {
    const bool lower = step < blocks;
    const int k0 = (lower ? step : 2 * blocks - 1 - step) * kLuPanel;
    float l[kLuPanel];
    if (warp == 0) {
      const float* row = A + static_cast<size_t>(piv[k0 + lane]) * n + k0;
#pragma unroll
      for (int j = 0; j < kLuPanel; j += 4) {
        const float4 x = *reinterpret_cast<const float4*>(row + j);
        l[j] = x.x, l[j + 1] = x.y, l[j + 2] = x.z, l[j + 3] = x.w;
      }
    }
    const int from = lower ? 0 : k0 + kLuPanel, to = lower ? k0 : n;
    for (int r = warp; r < kLuPanel; r += W) {
      const float* row = A + static_cast<size_t>(piv[k0 + r]) * n;
      float s = 0.0f;
#pragma unroll 8
      for (int j = from + lane; j < to; j += 32) s = fmaf(row[j], y[j], s);
      s = warp_sum(s);
      if (lane == 0) s_part[r] = s;
    }
    __syncthreads();
    if (warp == 0) {
      float x = y[k0 + lane] - s_part[lane];
      if (lower) {
#pragma unroll
        for (int c = 0; c < kLuPanel; ++c) {
          const float xc = __shfl_sync(0xffffffffu, x, c);
          if (lane > c) x = fmaf(-l[c], xc, x);
        }
      } else {
        float d = 1.0f;
#pragma unroll
        for (int c = 0; c < kLuPanel; ++c) d = lane == c ? l[c] : d;
        const float inv = 1.0f / d;
#pragma unroll
        for (int c = kLuPanel - 1; c >= 0; --c) {
          const float xc = __shfl_sync(0xffffffffu, x * inv, c);
          if (lane < c) x = fmaf(-l[c], xc, x);
        }
        x *= inv;
      }
      y[k0 + lane] = x;
    }
    __syncthreads();
  }
}

// y <- L'^-1 U'^-1 y (y in column order on entry, in pivot order on exit): the transposed solve. A block
// of 32 is solved by one warp, then a thread per column takes its products off the rest.
static __device__ __noinline__ void lu_sweeps_transposed(const float* A, int n, const int* piv, float* y) {
  const int t = static_cast<int>(threadIdx.x), lane = t & 31, warp = t >> 5;
  const int blocks = n / kLuPanel;
  for (int step = 0; step < 2 * blocks; ++step) {
    const bool upper = step < blocks;  // the sweep with U', from the first column on
    const int k0 = (upper ? step : 2 * blocks - 1 - step) * kLuPanel;
    if (warp == 0) {
      float l[kLuPanel], d = 1.0f;
#pragma unroll
      for (int i = 0; i < kLuPanel; ++i) {
        l[i] = A[static_cast<size_t>(piv[k0 + i]) * n + k0 + lane];
        if (upper && lane == i) d = l[i];
      }
      const float inv = 1.0f / d;
      float x = y[k0 + lane];
      if (upper) {
#pragma unroll
        for (int i = 0; i < kLuPanel; ++i) {
          const float xi = __shfl_sync(0xffffffffu, x * inv, i);
          if (lane > i) x = fmaf(-l[i], xi, x);
        }
        x *= inv;
      } else {
#pragma unroll
        for (int i = kLuPanel - 1; i >= 0; --i) {
          const float xi = __shfl_sync(0xffffffffu, x, i);
          if (lane < i) x = fmaf(-l[i], xi, x);
        }
      }
      y[k0 + lane] = x;
    }
    __syncthreads();
    const int from = upper ? k0 + kLuPanel : 0, to = upper ? n : k0;
    for (int j = from + t; j < to; j += kLuThreads) {
      float s = 0.0f;
#pragma unroll 16
      for (int i = 0; i < kLuPanel; ++i) {
        s = fmaf(A[static_cast<size_t>(piv[k0 + i]) * n + j], y[k0 + i], s);
      }
      y[j] -= s;
    }
    __syncthreads();
  }
}

}  // namespace sgb
