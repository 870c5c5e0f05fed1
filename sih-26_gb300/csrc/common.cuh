// common.cuh -- device helpers shared by every kernel of the GB300 PDHG engine.
#pragma once

#include <cuda_runtime.h>
#include <string.h>
#include <stdint.h>

#include <cmath>

namespace sgb {

constexpr int kWarp = 32;

// Absent bound: +-inf or any magnitude at or above 1e30, exactly as is_finite_bound in the
// reference (include/sankhya/types.hpp:88-96).
__host__ __device__ __forceinline__ bool finite_bound(double v) {
  return !(isinf(v) || fabs(v) >= 1e30);
}
__host__ __device__ __forceinline__ bool finite_bound(float v) {
  return !(isinf(v) || fabsf(v) >= 1e30f);
}

// Projection onto [lo, hi] tolerant of infinite sides (src/pdhg/pdhg.cpp:68-72).
template <typename T>
__host__ __device__ __forceinline__ T project(T v, T lo, T hi) {
  if (finite_bound(lo) && v < lo) return lo;
  if (finite_bound(hi) && v > hi) return hi;
  return v;
}

// Projection onto [lo, hi] when an absent side is an IEEE infinity (lo <= hi): the same
// value as project() for every non-NaN input, in two min/max instructions.
// Programmatic dependent launch: a kernel launched with programmatic stream serialization
// (launch_after, below) may have its blocks placed while the previous kernel in the stream is
// still finishing. Before it reads anything that kernel wrote, it waits here for that kernel's
// completion and the visibility of its memory. In a kernel launched the ordinary way the wait
// returns at once.
__device__ __forceinline__ void grid_dependency_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Lets the next kernel in the stream, where it was launched with launch_after, be placed as soon as
// every block of this one has called it (or left): its blocks then load what no kernel writes (the
// matrix) while this one works, and wait in grid_dependency_wait() for its end.
__device__ __forceinline__ void grid_dependency_launch() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Launches kernel<<<grid, threads, smem, s>>>(args...) with programmatic stream
// serialization: its blocks are placed on the SMs as the previous kernel's blocks leave them (or
// call grid_dependency_launch), instead of after the whole kernel and its launch; the kernel
// must call grid_dependency_wait() before its first read of anything an earlier kernel of the
// stream writes, and before its first write. Returns the launch's error.
template <typename... Params, typename... Args>
inline cudaError_t launch_after(void (*kernel)(Params...), int grid, int threads, int smem,
                                cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(grid));
  cfg.blockDim = dim3(static_cast<unsigned>(threads));
  cfg.dynamicSmemBytes = static_cast<size_t>(smem);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// All threads of the cluster meet; what each wrote before, to its own or another block's shared
// memory, is visible to the others after.
__device__ __forceinline__ void cluster_meet() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The shared-memory address of `p` in block `rank` of the cluster, and stores to such addresses.
__device__ __forceinline__ uint32_t cluster_addr(const void* p, int rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;"
      : "=r"(a)
      : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))), "r"(rank));
  return a;
}
__device__ __forceinline__ void cluster_store(uint32_t addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ void cluster_store(uint32_t addr, double2 v) {
  asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(addr), "d"(v.x), "d"(v.y)
               : "memory");
}

// Launches kernel<<<blocks, threads, smem, s>>>(args...) as one cluster of `blocks` blocks.
// Returns the launch's error.
template <typename... Params, typename... Args>
inline cudaError_t launch_cluster(void (*kernel)(Params...), int blocks, int threads, int smem,
                                  cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(blocks));
  cfg.blockDim = dim3(static_cast<unsigned>(threads));
  cfg.dynamicSmemBytes = static_cast<size_t>(smem);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(blocks);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Whether one cluster of `blocks` blocks of the kernel fits the current device.
template <typename Kernel>
inline bool cluster_fits(Kernel kernel, int blocks, int threads, int smem) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(blocks));
  cfg.blockDim = dim3(static_cast<unsigned>(threads));
  cfg.dynamicSmemBytes = static_cast<size_t>(smem);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(blocks);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return n > 0;
}

// ---- A grid whose blocks meet --------------------------------------------------------------
// What a control block's error word holds when a bounded wait gave up, and what the host says then.
constexpr int kCopyFault = 1;  // for a window or tile copy
constexpr int kMeetFault = 2;  // for the other blocks of the grid
inline const char* fault_message(int error) {
  return error == kMeetFault ? "the blocks of a step kernel did not meet in time"
                             : "a tile copy did not complete in time";
}

// A cooperative launch: all blocks run at once, so they may wait for one another. `counter` counts
// arrivals over launches of the same grid (a multiple of gridDim.x between launches, 64 bits, so it
// never wraps) and is zeroed with the control block it lives in.
struct GridMeet {
  unsigned long long* counter;
  unsigned long long target;
  // Before this block's first arrival the counter lacks at least that one of the launch's first
  // meeting, so rounding it down gives the launch's start. All threads call it (only thread 0's
  // value is used).
  __device__ __forceinline__ void start(unsigned long long* c) {
    counter = c;
    target = 0;
    if (threadIdx.x == 0) target = *reinterpret_cast<volatile unsigned long long*>(c) / gridDim.x * gridDim.x;
  }
  // All threads of all blocks meet: what each wrote before is visible to the others after (through
  // ld_live, never through the read-only path). Returns false, in every thread of the block, if
  // the others did not arrive within kMeetPolls polls (half a second or more); *error is kMeetFault then.
  // A block that gave up must not meet again, so the others give up at their next meeting.
  __device__ __forceinline__ bool meet(int* error) {
    constexpr int kMeetPolls = 1 << 21;
    __shared__ int s_met;
    __syncthreads();
    if (threadIdx.x == 0) {
      target += gridDim.x;
      asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(counter), "l"(1ull) : "memory");
      unsigned long long now = 0;
      int polls = 0;
      do {
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(now) : "l"(counter) : "memory");
      } while (now < target && ++polls < kMeetPolls);
      s_met = now >= target;
      if (now < target) *reinterpret_cast<volatile int*>(error) = kMeetFault;
    }
    __syncthreads();
    return s_met != 0;
  }
};

// A load of data that the running kernel writes: an ordinary one, as the pointer is not __restrict__
// (a volatile asm load would not be predicated but branched around).
template <typename T>
__device__ __forceinline__ T ld_live(const T* p) {
  return *p;
}

// Launches kernel<<<blocks, threads, smem, s>>>(args...) cooperatively; returns the launch's error.
template <typename... Params, typename... Args>
inline cudaError_t launch_grid(void (*kernel)(Params...), int blocks, int threads, int smem,
                               cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(blocks));
  cfg.blockDim = dim3(static_cast<unsigned>(threads));
  cfg.dynamicSmemBytes = static_cast<size_t>(smem);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Whether `blocks` blocks of the kernel run at once on the current device.
template <typename Kernel>
inline bool grid_fits(Kernel kernel, int blocks, int threads, int smem) {
  int dev = 0, sms = 0, able = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&able, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads,
                                                    static_cast<size_t>(smem)) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return able != 0 && blocks > 0 && blocks <= sms * per_sm;
}

// A key whose order as an integer is the order of the doubles (a negative zero before a positive
// one, a NaN outside both infinities). An FP64 compare holds GB300's FP64 pipe as long as an FP64
// addition does; the projections of the steps compare keys on the integer units instead.
__host__ __device__ __forceinline__ long long order_key(double v) {
#ifdef __CUDA_ARCH__
  const long long i = __double_as_longlong(v);
#else
  long long i;
  memcpy(&i, &v, sizeof(i));
#endif
  return i ^ ((i >> 63) & 0x7fffffffffffffffLL);
}
__host__ __device__ __forceinline__ bool nan_key(long long key) {
  return key > 0x7ff0000000000000LL || key < ~0x7ff0000000000000LL;
}

// min(max(v, lo), hi), for bounds that are not NaN; a NaN v gives lo as fmax would.
__host__ __device__ __forceinline__ double clamp_box(double v, double lo, double hi) {
  const long long kv = order_key(v), kl = order_key(lo);
  const bool low = kv < kl || nan_key(kv);
  const double r = low ? lo : v;
  return (low ? kl : kv) > order_key(hi) ? hi : r;
}
// The same projection with a NaN v left as it is.
__host__ __device__ __forceinline__ double clamp_box_or_nan(double v, double lo, double hi) {
  const long long kv = order_key(v);
  if (nan_key(kv)) return v;
  return kv < order_key(lo) ? lo : (kv > order_key(hi) ? hi : v);
}

// v / sigma from inv = RN(1 / sigma): Markstein's correction of the product with the correctly
// rounded reciprocal (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34(1), 1990): q = v (1/sigma), r = v - sigma q exactly by
// FMA, q + r (1/sigma) rounded once, which is the correctly rounded quotient for operands and
// results in the normal range (tests/host/qp_division_check.c holds it to IEEE division). Three FP64
// instructions where a division takes a dozen. An exact first product (r = 0) or a residual that is
// not finite (an infinite v, or a quotient past the largest number) keeps the product.
__host__ __device__ __forceinline__ double divide(double v, double sigma, double inv) {
#ifdef __CUDA_ARCH__
  const double q = __dmul_rn(v, inv);
#else
  const double q = v * inv;
#endif
  const double r = fma(-q, sigma, v);
#ifdef __CUDA_ARCH__
  const long long size = __double_as_longlong(r) & 0x7fffffffffffffffLL;
#else
  long long size;
  memcpy(&size, &r, sizeof(size));
  size &= 0x7fffffffffffffffLL;
#endif
  return size == 0 || size >= 0x7ff0000000000000LL ? q : fma(r, inv, q);
}

__device__ __forceinline__ float clamp_box(float v, float lo, float hi) {
  return fminf(fmaxf(v, lo), hi);
}

// std::max / std::min semantics (comparison order matters for NaN).
__host__ __device__ __forceinline__ double dmax(double a, double b) { return (a < b) ? b : a; }
__host__ __device__ __forceinline__ double dmin(double a, double b) { return (b < a) ? b : a; }

// ---- Deterministic reductions ------------------------------------------------------------
// Every sum in the engine goes through these: a fixed xor-butterfly inside a warp, then the
// warps of a block in index order. With a fixed grid the result is bit-identical from run to
// run, so the step-size and restart decisions are reproducible.

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = dmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Sum of `v` over a group of G consecutive lanes (G a power of two <= 32); every lane of the
// group receives the total.
template <int G, typename T>
__device__ __forceinline__ T group_sum(T v) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sums of N values (a power of two) over a warp by halves: at each level a lane hands half of its
// values to its partner and adds the partner's to the other half, so N values take N - 1 adds
// and log2(32 / N) more, not 5 N. Afterwards lane l holds the total of value warp_sums_index<N>(l)
// in v[0].
template <int N, int O = 16>
__device__ __forceinline__ void warp_sums(double* v) {
  if constexpr (O > 0) {
    constexpr int kHalf = N > 1 ? N / 2 : 1;
    const bool high = (threadIdx.x & O) != 0;
#pragma unroll
    for (int k = 0; k < kHalf; ++k) {
      if constexpr (N > 1) {
        const double give = high ? v[k] : v[k + kHalf];
        const double keep = high ? v[k + kHalf] : v[k];
        v[k] = keep + __shfl_xor_sync(0xffffffffu, give, O);
      } else {
        v[k] += __shfl_xor_sync(0xffffffffu, v[k], O);
      }
    }
    warp_sums<kHalf, O / 2>(v);
  }
}
template <int N>
__device__ __forceinline__ int warp_sums_index(int lane) {
  int at = 0;
#pragma unroll
  for (int o = 16, half = N / 2; half > 0; o >>= 1, half >>= 1) at += (lane & o) ? half : 0;
  return at;
}

// Block-wide sum of NV values per thread. `scratch` holds NV * (blockDim/32) doubles. Thread 0
// receives the totals in out[]. All threads must call it. An FP64 addition holds the pipe of its
// quarter of the SM for 64 cycles whatever its lanes add, so a warp whose values are all zero adds
// nothing, the others add by halves, and each total is taken by a warp of its own: three sums over
// 24 warps took 4.3 us as butterflies.
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double* scratch, double (&out)[NV]) {
  constexpr int kAll = NV <= 1 ? 1 : NV <= 2 ? 2 : NV <= 4 ? 4 : NV <= 8 ? 8 : 16;
  static_assert(NV <= kAll, "at most 16 sums");
  __shared__ double s_total[NV];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  long long bits = 0;
#pragma unroll
  for (int q = 0; q < NV; ++q) bits |= __double_as_longlong(v[q]);
  double w[kAll];
#pragma unroll
  for (int q = 0; q < kAll; ++q) w[q] = q < NV ? v[q] : 0.0;
  if (__any_sync(0xffffffffu, bits != 0)) warp_sums<kAll>(w);
  const int mine = warp_sums_index<kAll>(lane);
  if ((lane & (32 / kAll - 1)) == 0 && mine < NV) scratch[mine * nwarps + warp] = w[0];
  __syncthreads();
  for (int q = warp; q < NV; q += nwarps) {
    const double s = warp_sum(lane < nwarps ? scratch[q * nwarps + lane] : 0.0);
    if (lane == 0) s_total[q] = s;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NV; ++q) out[q] = s_total[q];
}

template <int NV>
__device__ __forceinline__ void block_max(double (&v)[NV], double* scratch, double (&out)[NV]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
#pragma unroll
  for (int q = 0; q < NV; ++q) v[q] = warp_max(v[q]);
  if (lane == 0) {
#pragma unroll
    for (int q = 0; q < NV; ++q) scratch[q * nwarps + warp] = v[q];
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      double s = lane < nwarps ? scratch[q * nwarps + lane] : 0.0;
      s = warp_max(s);
      out[q] = s;
    }
  }
  __syncthreads();
}

}  // namespace sgb
