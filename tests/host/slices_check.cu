// slices_check.cu -- the sliced layouts (csrc/slices.cuh, plan_slices) on the CPU: every entry of
// every row is stored exactly once, at a place inside the arrays and in the row's order; the
// rows of a slice come longest first and fit the meta word; windows are aligned, within their
// capacity and inside the padded vector; the blocks' segments cover the slices in order.
// Prints OK and exits 0, or the first failure.
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "engine.hpp"

using namespace sgb;

static void fail(const char* what, long long a, long long b) {
  std::printf("FAIL %s: %lld %lld\n", what, a, b);
  std::exit(1);
}

static void check(const std::vector<int>& len, int extent, int wmax, double window_min, int sms,
                  int np, bool banded, unsigned seed) {
  const int lines = static_cast<int>(len.size());
  std::vector<int> ptr(static_cast<size_t>(lines) + 1, 0);
  for (int r = 0; r < lines; ++r) ptr[r + 1] = ptr[r] + len[r];
  std::vector<int> idx(static_cast<size_t>(ptr[lines]));
  std::mt19937 rng(seed);
  for (int r = 0; r < lines; ++r) {
    for (int k = ptr[r]; k < ptr[r + 1]; ++k) {
      const long long at = banded ? static_cast<long long>(r) * extent / lines + rng() % 64 : rng();
      idx[k] = static_cast<int>(((at % extent) + extent) % extent);
    }
  }
  const SlicePlan p = plan_slices(ptr, idx.data(), lines, extent, wmax, window_min, sms, np);
  std::vector<int> seen(static_cast<size_t>(lines), 0);
  std::vector<char> place(static_cast<size_t>(p.entries), 0);
  auto put = [&](long long at) {
    if (at < 0 || at >= p.entries) fail("entry outside the arrays", at, p.entries);
    if (place[static_cast<size_t>(at)]++) fail("two entries at one place", at, 0);
  };
  if (p.nslices % kGroupSlices != 0 || p.nslices * 32LL < lines) fail("slices", p.nslices, lines);
  if (static_cast<int>(p.base.size()) != p.nslices + 1 || p.base[p.nslices] * 32LL != p.long_base) {
    fail("bases", static_cast<long long>(p.base.size()), p.nslices);
  }
  for (int s = 0; s < p.nslices; ++s) {
    int before = kSliceLong;
    for (int l = 0; l < 32; ++l) {
      const unsigned m = p.meta[static_cast<size_t>(s) * 32 + l];
      if (m == kNoRow) {
        before = -1;
        continue;
      }
      const int row = (s / kGroupSlices) * kGroupRows + static_cast<int>(m & 127u);
      const int n = static_cast<int>(m >> 8);
      if (row >= lines) fail("row", row, lines);
      if (n != len[row]) fail("length", n, len[row]);
      if (n > before) fail("longest first", s, l);
      if (n > static_cast<int>(p.base[s + 1] - p.base[s])) fail("width", s, n);
      before = n;
      ++seen[row];
      for (int k = 0; k < n; ++k) put(static_cast<long long>(p.base[s]) * 32 + 32LL * k + l);
    }
  }
  int chunk = 0;
  for (size_t i = 0; i < p.items.size(); ++i) {
    const SliceItem& it = p.items[i];
    if (len[it.row] <= kSliceLong) fail("short row as an item", it.row, len[it.row]);
    if (it.count < 1 || it.count > kSlicePiece) fail("piece", it.count, kSlicePiece);
    if (it.slot >= 0 && it.slot != chunk++) fail("piece slot", it.slot, chunk);
    if ((it.slot < 0) != (len[it.row] <= kSlicePiece)) fail("slot of a whole row", it.row, it.slot);
    const bool first = i == 0 || p.items[i - 1].row != it.row;
    if (first) ++seen[it.row];
    if (!first && it.begin != p.items[i - 1].begin + p.items[i - 1].count) fail("piece order", it.row, it.begin);
    for (int k = 0; k < it.count; ++k) put(p.long_base + it.begin + k);
  }
  if (chunk != p.nchunks) fail("chunks", chunk, p.nchunks);
  long long stored = 0;
  for (char c : place) stored += c;
  if (stored != ptr[lines]) fail("entries stored", stored, ptr[lines]);
  for (int r = 0; r < lines; ++r) {
    if (seen[r] != 1) fail("row seen", r, seen[r]);
  }
  int total = 0;
  for (const LongRow& l : p.longs) {
    if (l.chunk0 != total || l.nchunks != (len[l.row] + kSlicePiece - 1) / kSlicePiece) fail("long row", l.row, l.nchunks);
    total += l.nchunks;
  }
  if (total != p.nchunks) fail("long rows' chunks", total, p.nchunks);
  if (p.grid < 1 || p.grid > std::max(1, sms)) fail("grid", p.grid, sms);
  if (p.threads < 128 || p.threads > kSliceThreads || p.threads % 32) fail("threads", p.threads, 0);
  if (static_cast<int>(p.seg_start.size()) != p.grid + 1 || p.seg_start[0] != 0 ||
      p.seg_start[p.grid] != static_cast<int>(p.segs.size())) {
    fail("segment starts", p.grid, static_cast<long long>(p.segs.size()));
  }
  int at = 0;
  for (int b = 0; b < p.grid; ++b) {
    if (p.seg_start[b + 1] <= p.seg_start[b]) fail("block without a segment", b, 0);
    if (p.block_start[b] != at) fail("block start", p.block_start[b], at);
    for (int g = p.seg_start[b]; g < p.seg_start[b + 1]; ++g) {
      const SliceSeg& sg = p.segs[g];
      if (sg.s1 > sg.s0) {
        if (sg.s0 != at) fail("segment start", sg.s0, at);
        at = sg.s1;
      }
      if (sg.len > 0) {
        if (sg.lo % 4 || sg.len % 4 || sg.len > p.wmax || p.wmax > wmax) fail("window", sg.lo, sg.len);
        if (sg.lo < 0 || sg.lo + sg.len > ((extent + 3) & ~3)) fail("window range", sg.lo, sg.len);
      }
    }
  }
  if (p.block_start[p.grid] != p.nslices) fail("last block", p.block_start[p.grid], p.nslices);
  if (at != p.nslices) fail("slices covered", at, p.nslices);
}

int main() {
  std::mt19937 rng(7);
  int cases = 0;
  for (int lines : {0, 1, 31, 32, 33, 127, 128, 129, 1000, 20011}) {
    for (int kind = 0; kind < 5; ++kind) {
      std::vector<int> len(static_cast<size_t>(lines));
      for (int r = 0; r < lines; ++r) {
        const int u = static_cast<int>(rng() % 100);
        switch (kind) {
          case 0: len[r] = 10; break;
          case 1: len[r] = static_cast<int>(rng() % 30); break;
          case 2: len[r] = u < 90 ? u % 5 : kSliceLong - 1 + u % 4; break;
          case 3: len[r] = u < 98 ? 0 : kSlicePiece - 1 + u % 4; break;
          default: len[r] = r == lines / 2 ? 3 * kSlicePiece + 17 : 2; break;
        }
      }
      for (int wmax : {0, 64, 16384}) {
        for (int sms : {1, 7, 152}) {
          for (int extent : {5, 3001, 100000}) {
            check(len, extent, wmax, cases % 2 ? 0.95 : 0.0, sms, 1 + cases % 2, kind % 2 == 0, 11 + cases);
            ++cases;
          }
        }
      }
    }
  }
  std::printf("OK %d layouts\n", cases);
  return 0;
}
