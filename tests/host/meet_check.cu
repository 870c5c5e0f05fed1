// meet_check.cu -- GridMeet (common.cuh) on a GPU: a grid whose blocks all meet, and one whose last block
// never comes: the others give up within a few seconds, say so in every thread, and leave kMeetFault in
// the error word; the device stays usable and a grid that starts from a cleared counter meets again.
// Prints OK and exits 0, or the first failure.
#include <chrono>
#include <cstdio>

#include "common.cuh"

constexpr int kBlocks = 4, kThreads = 64;

__global__ void k_meet(unsigned long long* counter, int* error, int* met, int rounds, int absent) {
  sgb::GridMeet grid;
  grid.start(counter);
  if (static_cast<int>(blockIdx.x) == absent) return;
  for (int r = 0; r < rounds; ++r) {
    if (!grid.meet(error)) return;
    atomicAdd(met, 1);
  }
}

#define CHECK(x)                                                        \
  do {                                                                  \
    if (!(x)) {                                                         \
      std::printf("FAIL line %d: %s\n", __LINE__, #x);                  \
      return 1;                                                         \
    }                                                                   \
  } while (0)

int main() {
  unsigned long long* counter = nullptr;
  int* words = nullptr;  // error, met
  CHECK(cudaMalloc(&counter, sizeof(*counter)) == cudaSuccess);
  CHECK(cudaMalloc(&words, 2 * sizeof(int)) == cudaSuccess);
  CHECK(sgb::grid_fits(k_meet, kBlocks, kThreads, 0));
  for (int absent : {-1, kBlocks - 1, -1}) {
    CHECK(cudaMemset(counter, 0, sizeof(*counter)) == cudaSuccess);
    CHECK(cudaMemset(words, 0, 2 * sizeof(int)) == cudaSuccess);
    const auto t0 = std::chrono::steady_clock::now();
    CHECK(sgb::launch_grid(k_meet, kBlocks, kThreads, 0, cudaStream_t{nullptr}, counter, words, words + 1, 5,
                           absent) == cudaSuccess);
    CHECK(cudaDeviceSynchronize() == cudaSuccess);
    const double s = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    int got[2];
    CHECK(cudaMemcpy(got, words, sizeof(got), cudaMemcpyDeviceToHost) == cudaSuccess);
    std::printf("absent %d: %.3f s, error %d, %d\n", absent, s, got[0], got[1]);
    CHECK(s < 20.0);
    CHECK(got[0] == (absent < 0 ? 0 : sgb::kMeetFault));
    CHECK(got[1] == (absent < 0 ? 5 * kBlocks * kThreads : 0));
  }
  std::printf("OK\n");
  return 0;
}
