// basis_places_check.cu -- the bound on a basis matrix's slices (batch.cuh, basis_places) on the CPU,
// against the places that the batch's rules give: random matrices, even, skewed, tall and wide, with
// lines past the sort's range, and random bases of each, dealt longest first (lines past the range in
// index order) to slices as wide as their longest line. And the bound of a wide LP with a dense row
// stays with the basis, not with the row. The workspaces of the dense factors: as many as blocks where
// half of the free memory holds them, else fewer, never none. Prints OK and exits 0, or the first failure.
#include <algorithm>
#include <cstdio>
#include <numeric>
#include <random>
#include <vector>

#include "batch.cuh"
#include "dense_lu.cuh"

using namespace sgb;

static std::mt19937 rng(7);

static long long slices_of(std::vector<int> len) {
  std::vector<int> order(len.size());
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
    return std::min(len[a], kSortLength) > std::min(len[b], kSortLength);
  });
  long long places = 0;
  for (size_t s = 0; s < order.size(); s += 32) {
    int width = 0;
    for (size_t k = s; k < std::min(s + 32, order.size()); ++k) width = std::max(width, len[order[k]]);
    places += 32LL * width;
  }
  return places;
}

// A matrix of m rows with about the given lengths over n columns; both orientations.
static bool check(const std::vector<int>& want, int n, int bases) {
  const int m = static_cast<int>(want.size());
  std::vector<std::vector<int>> rows(m), cols(n);
  for (int i = 0; i < m; ++i) {
    std::vector<char> used(n, 0);
    for (int k = 0; k < want[i]; ++k) {
      const int j = static_cast<int>(rng() % n);
      if (used[j]++) continue;
      rows[i].push_back(j);
      cols[j].push_back(i);
    }
  }
  const auto starts = [](const std::vector<std::vector<int>>& lines) {
    std::vector<int> s(1, 0);
    for (const auto& l : lines) s.push_back(s.back() + static_cast<int>(l.size()));
    return s;
  };
  const std::vector<int> rp = starts(rows), cp = starts(cols);
  const int d = std::min(m, n);
  const long long by_row = basis_places(rp.data(), m, d), by_col = basis_places(cp.data(), n, d);
  for (int b = 0; b < bases; ++b) {
    const int nb = b == 0 ? d : 1 + static_cast<int>(rng() % d);
    std::vector<int> r(m), c(n);
    std::iota(r.begin(), r.end(), 0);
    std::iota(c.begin(), c.end(), 0);
    std::shuffle(r.begin(), r.end(), rng);
    std::shuffle(c.begin(), c.end(), rng);
    // The worst bases hold the long lines.
    if (b % 2 == 0) {
      std::sort(r.begin(), r.end(), [&](int x, int y) { return rows[x].size() > rows[y].size(); });
      std::sort(c.begin(), c.end(), [&](int x, int y) { return cols[x].size() > cols[y].size(); });
    }
    std::vector<char> in_r(m, 0), in_c(n, 0);
    for (int k = 0; k < nb; ++k) in_r[r[k]] = in_c[c[k]] = 1;
    std::vector<int> lr, lc;
    for (int i = 0; i < m; ++i) {
      if (!in_r[i]) continue;
      lr.push_back(static_cast<int>(
          std::count_if(rows[i].begin(), rows[i].end(), [&](int j) { return in_c[j]; })));
    }
    for (int j = 0; j < n; ++j) {
      if (!in_c[j]) continue;
      lc.push_back(static_cast<int>(
          std::count_if(cols[j].begin(), cols[j].end(), [&](int i) { return in_r[i]; })));
    }
    if (slices_of(lr) > by_row || slices_of(lc) > by_col) {
      std::printf("FAIL %d x %d basis of %d: %lld > %lld or %lld > %lld\n", m, n, nb, slices_of(lr),
                  by_row, slices_of(lc), by_col);
      return false;
    }
  }
  return true;
}

int main() {
  for (int m : {1, 2, 31, 32, 33, 64, 65, 200}) {
    for (int n : {1, 5, 32, 100, 400}) {
      std::vector<int> even(m, std::min(n, 5)), skewed(m, 1), full(m, n);
      for (int i = 0; i < m; i += 7) skewed[i] = n;
      if (!check(even, n, 6) || !check(skewed, n, 6) || !check(full, n, 2)) return 1;
    }
  }
  std::vector<int> past(1500, 3);
  for (int i = 0; i < 70; ++i) past[20 * i] = 4000;  // some 1,400 of 1,600 columns
  if (!check(past, 1600, 4)) return 1;
  // Ten dense rows over 10,000 columns; one over 100,000.
  std::vector<int> wide(11);
  for (int i = 0; i <= 10; ++i) wide[i] = 10000 * i;
  std::vector<int> one(101, 100000);
  one[0] = 0;
  if (basis_places(wide.data(), 10, 10) > 32 * 10 || basis_places(one.data(), 100, 100) > 32 * 100 * 4) {
    std::printf("FAIL wide: %lld %lld\n", basis_places(wide.data(), 10, 10), basis_places(one.data(), 100, 100));
    return 1;
  }
  if (lu_workspaces(152, 4 << 20, size_t{200} << 30) != 152 || lu_workspaces(152, 4 << 20, 80 << 20) != 10 ||
      lu_workspaces(152, 4 << 20, 1 << 20) != 1 || lu_workspaces(1, 4096, 0) != 1) {
    std::printf("FAIL workspaces\n");
    return 1;
  }
  std::printf("OK\n");
  return 0;
}
