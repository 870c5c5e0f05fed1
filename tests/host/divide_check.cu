// divide_check.cu -- the row prox's quotient (common.cuh, divide) against IEEE division on the CPU: every
// pair of edge values whose divisor's reciprocal is a normal number, quotients past the largest number
// and infinite numerators among them, and random pairs of the normal range, bit for bit; and the
// projection of such a quotient ends on the side that the quotient is past. Prints the pairs that
// differ and exits non-zero if any does.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <limits>
#include <vector>

#include "common.cuh"

static long long bad = 0;

static void one(double v, double sigma) {
  const double want = v / sigma, got = sgb::divide(v, sigma, 1.0 / sigma);
  const bool same = (want != want && got != got) || memcmp(&want, &got, sizeof(want)) == 0;
  const bool side = want != want ||
                    sgb::clamp_box(got, -1.0, 2.0) == std::fmin(std::fmax(want, -1.0), 2.0);
  if (!same || !side) {
    if (bad++ < 10) std::printf("differs: %a / %a = %a, %a\n", v, sigma, want, got);
  }
}

int main() {
  const double inf = std::numeric_limits<double>::infinity();
  const double most = std::numeric_limits<double>::max();
  const std::vector<double> v = {0.0, -0.0, 1.0, -1.0, 3.0, 1e-280, -1e-280, 1e30, 1e300, -1e300, most,
                                 -most, inf, -inf, std::numeric_limits<double>::quiet_NaN()};
  const std::vector<double> sigma = {1.0, 3.0, 0.1, 1e-12, 1e-20, 1e-100, 1e-300, 1e12, 1e100, 1e300};
  for (double a : v) {
    for (double b : sigma) {
      // Quotients below the normal range are outside the method's.
      if (a != 0.0 && std::fabs(a / b) < 1e-290) continue;
      one(a, b);
      one(a, -b);
    }
  }
  uint64_t state = 1;
  const auto next = [&] {
    state = state * 6364136223846793005ull + 1442695040888963407ull;
    return state >> 11;
  };
  for (int k = 0; k < 2000000; ++k) {
    const double a = std::ldexp(1.0 + static_cast<double>(next()) * 0x1p-53, static_cast<int>(next() % 400) - 200);
    const double b = std::ldexp(1.0 + static_cast<double>(next()) * 0x1p-53, static_cast<int>(next() % 200) - 100);
    one(k & 1 ? -a : a, b);
  }
  std::printf("%lld differ\n", bad);
  return bad != 0;
}
