// clamp_check.cu -- the steps' projections (common.cuh, clamp_box and clamp_box_or_nan), which compare
// doubles by their bits, against floating-point comparisons on the CPU: every triple v, lo <= hi of
// edge values (zeros of both signs, denormals, the largest numbers, infinities, NaN of both signs) and
// of random bit patterns. Prints the triples that differ and exits non-zero if any does.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <limits>
#include <vector>

#include "common.cuh"

static long long bad = 0;

static bool same(double a, double b) { return (a != a && b != b) || a == b; }

static void one(double v, double lo, double hi) {
  const double want = std::fmin(std::fmax(v, lo), hi);
  const double kept = v < lo ? lo : (v > hi ? hi : v);
  if (!same(sgb::clamp_box(v, lo, hi), want) || !same(sgb::clamp_box_or_nan(v, lo, hi), kept)) {
    if (bad++ < 10) std::printf("differs: %a in [%a, %a]\n", v, lo, hi);
  }
}

int main() {
  const double inf = std::numeric_limits<double>::infinity();
  const double nan = std::numeric_limits<double>::quiet_NaN();
  std::vector<double> v = {0.0, -0.0, 4.9e-324, -4.9e-324, 2.2250738585072014e-308, 1.0, -1.0,
                           1.0 + 2.3e-16, 1e30, -1e30, 1.7976931348623157e308, -1.7976931348623157e308,
                           inf, -inf, nan, -nan};
  uint64_t state = 1;
  for (int k = 0; k < 150; ++k) {
    state = state * 6364136223846793005ull + 1442695040888963407ull;
    double d;
    memcpy(&d, &state, sizeof(d));
    v.push_back(d);
  }
  for (double a : v) {
    for (double lo : v) {
      for (double hi : v) {
        if (lo <= hi) one(a, lo, hi);
      }
    }
  }
  std::printf("%lld differ\n", bad);
  return bad != 0;
}
