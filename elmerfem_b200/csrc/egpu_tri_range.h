// egpu_tri_range.h -- host plan of the row-range triangular solves (range_ilu in
// egpu_krylov.cuh): plain C++, so its arithmetic can be checked without a GPU.
//
// The rows are cut into equal contiguous ranges, one per block of the grid.  A block solves its
// range level by level (dependency levels of the rows, or of the node blocks of bs rows), its
// values in shared memory.  Every dependency lies in an earlier level of the own range or in
// another range, before it in row order (lower) or after it (upper); the values of other
// ranges a block needs (its external values) are fetched into its shared memory as they
// appear.  With all blocks resident the solve cannot deadlock.
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

#ifdef __CUDACC__
#define EGPU_HD __host__ __device__
#else
#define EGPU_HD
#endif

namespace egpu {
namespace plan {

// Entries per row are padded to G * K: G lanes a row (1, 2, 4 or 8), K entries a lane (7 or 10).
struct RangeShape {
  int g = 0, k = 0;
};
constexpr int RANGE_THREADS = 384;  // most threads of a set (two sets solve rows; the rest stage and fetch)
constexpr int RANGE_STAGES = 4;     // levels staged in shared memory at a time
constexpr int RANGE_STAGE_BYTES = 18 * 1024;  // of one level (wider levels are split)

// the smallest padding that holds `ne` entries; g = 0: too many
inline RangeShape range_shape(int ne) {
  RangeShape best;
  for (int g = 1; g <= 8; g *= 2)
    for (int k = 7; k <= 10; k += 3)
      if (g * k >= ne && (best.g == 0 || g * k < best.g * best.k)) {
        best.g = g;
        best.k = k;
      }
  return best;
}

// A level of a range is one record in device memory, staged by a single bulk copy: a 16-byte
// header (first slot, rows), the rows' numbers, the shared-memory indices (16 bits: own slots
// from 0, external values from `per`, then the zero cell) and the values of the padded entries;
// every part is padded to 16 bytes.
struct RangeLevel {
  int slot, rows;  // first slot in the range, rows
};
EGPU_HD inline int range_pad16(int b) { return (b + 15) & ~15; }
EGPU_HD inline int range_idx_at(int rows) { return 16 + range_pad16(4 * rows); }
EGPU_HD inline int range_val_at(int rows, int gk) { return range_idx_at(rows) + range_pad16(2 * rows * gk); }
EGPU_HD inline int range_record(int rows, int gk, int vsize) {
  return range_val_at(rows, gk) + range_pad16(vsize * rows * gk);
}
// where entry e of a level's row t sits in its index and value arrays
EGPU_HD inline int range_entry_at(int rows, int g, int t, int e) { return (e / g) * rows * g + t * g + e % g; }
// most rows of a level (its FP64 record fits a stage, its lanes the block)
inline int range_max_rows(RangeShape sh) {
  int r = RANGE_THREADS / sh.g;
  while (r > 1 && range_record(r, sh.g * sh.k, 8) > RANGE_STAGE_BYTES) --r;
  return r;
}

// One triangle.  Slots number the rows of a range in the order they are solved; slot s of range
// c is the global slot c * per + s.
struct RangeTriHost {
  std::vector<int> lev_ptr;          // first level of every range (nr + 1)
  std::vector<RangeLevel> lev;
  std::vector<int> slot_lev;         // level (index into lev) of every global slot
  std::vector<int> row;              // row of every global slot
  std::vector<uint16_t> slot;        // slot (in its range) of every row
  std::vector<int> ext_ptr, ext;     // external rows of every range, in the order of first use
  int max_ext = 0, max_rows = 0;     // most external rows of a range, most rows of a level
};

// first out-of-block entry of row r, and their number (bs == 1: the strictly lower / upper part)
inline void range_entries(int bs, bool lower, const std::vector<int> &rows, const std::vector<int> &diag, int r,
                          int &beg, int &ne) {
  const int r0 = r / bs * bs, e_lo = diag[r0] - rows[r0];
  const int len = rows[r0 + 1] - rows[r0];
  beg = lower ? rows[r] : rows[r] + e_lo + bs;
  ne = lower ? e_lo : len - e_lo - bs;
}

// dependency levels of the rows (bs == 1) or node blocks; returns their number
inline int range_levels(int n, int bs, bool lower, const std::vector<int> &rows, const std::vector<int> &cols,
                        std::vector<int> &lev) {
  const int nb = n / bs;
  int nl = 0;
  lev.assign(nb, 0);
  for (int q = 0; q < nb; ++q) {
    const int m = lower ? q : nb - 1 - q;
    int l = 0;
    for (int e = rows[m * bs]; e < rows[m * bs + 1]; ++e) {
      const int d = cols[e] / bs;
      if (lower ? d < m : d > m) l = std::max(l, lev[d] + 1);
    }
    lev[m] = l;
    nl = std::max(nl, l + 1);
  }
  return nl;
}

// Cycles of the plan's timing model, fitted to B200 measurements (hex 16^3 to 96^3, 3-DOF hex 24^3
// to 64^3, a randomly numbered tet mesh): a level costs the FP64 units' latency through its sums
// plus its record's way through shared memory; a value handed from one block to another a store,
// an L2 round trip and a poll, and the more external values a range has the later one comes.
inline float range_level_cycles(int bs, int bytes) { return 500.f + (bs > 1 ? 0.11f : 0.07f) * (float)bytes; }
inline float range_cross_cycles(int ext) { return 650.f + 0.45f * (float)ext; }

// modelled cycles of one triangle with ranges of `per` rows
inline double range_cycles(int n, int bs, int per, RangeShape sh, int ext, bool lower, const std::vector<int> &rows,
                           const std::vector<int> &cols, const std::vector<int> &diag, const std::vector<int> &lev) {
  const int nb = n / bs, pb = per / bs, nr = (nb + pb - 1) / pb;
  std::vector<float> done(nb, 0.f);
  std::vector<int> cnt, ids;
  const int wide = std::max(1, range_max_rows(sh) / bs);  // nodes of one (sub-)level
  const float cross = range_cross_cycles(ext);
  double cycles = 0.0;
  for (int q = 0; q < nr; ++q) {
    const int c = lower ? q : nr - 1 - q, b0 = c * pb, b1 = std::min(nb, b0 + pb);
    const auto mm = std::minmax_element(lev.begin() + b0, lev.begin() + b1);
    const int lmin = *mm.first, nl = *mm.second - lmin + 1;
    cnt.assign(nl + 1, 0);
    for (int m = b0; m < b1; ++m) cnt[lev[m] - lmin + 1]++;
    for (int l = 0; l < nl; ++l) cnt[l + 1] += cnt[l];
    ids.assign(b1 - b0, 0);
    std::vector<int> at(cnt.begin(), cnt.end() - 1);
    for (int m = b0; m < b1; ++m) ids[at[lev[m] - lmin]++] = m;
    float t = 0.f;
    for (int l = 0; l < nl; ++l) {
      if (cnt[l + 1] == cnt[l]) continue;
      for (int s = cnt[l]; s < cnt[l + 1]; ++s) {
        int beg, ne;
        range_entries(bs, lower, rows, diag, ids[s] * bs, beg, ne);
        for (int e = 0; e < ne; e += bs) {
          const int d = cols[beg + e] / bs;
          if (d < b0 || d >= b1) t = std::max(t, done[d] + cross);
        }
      }
      for (int left = cnt[l + 1] - cnt[l]; left > 0; left -= wide)
        t += range_level_cycles(bs, range_record(std::min(left, wide) * bs, sh.g * sh.k, 8));
      for (int s = cnt[l]; s < cnt[l + 1]; ++s) done[ids[s]] = t;
    }
    cycles = std::max(cycles, (double)t);
  }
  return cycles;
}

// The plan of one triangle; false when it does not fit (a row with more entries than its lanes
// hold, or more shared-memory cells than 16-bit indices reach).
inline bool range_triangle(int n, int bs, int per, RangeShape sh, bool lower, const std::vector<int> &rows,
                           const std::vector<int> &cols, const std::vector<int> &diag, const std::vector<int> &lev,
                           RangeTriHost &T) {
  const int nr = (n + per - 1) / per, maxw = range_max_rows(sh);
  T = RangeTriHost{};
  T.slot_lev.resize(n);
  T.row.resize(n);
  T.slot.resize(n);
  T.lev_ptr.assign(1, 0);
  T.ext_ptr.assign(1, 0);
  std::vector<int> cnt, mark(n, -1);
  // pass 1: slots, levels and external rows of every range
  for (int c = 0; c < nr; ++c) {
    const int r0 = c * per, r1 = std::min(n, r0 + per);
    const auto mm = std::minmax_element(lev.begin() + r0 / bs, lev.begin() + r1 / bs);
    const int lmin = *mm.first, nl = *mm.second - lmin + 1;
    cnt.assign(nl + 1, 0);
    for (int r = r0; r < r1; ++r) cnt[lev[r / bs] - lmin + 1]++;
    for (int l = 0; l < nl; ++l) cnt[l + 1] += cnt[l];
    std::vector<int> at(cnt.begin(), cnt.end() - 1);
    for (int r = r0; r < r1; ++r) {
      const int s = at[lev[r / bs] - lmin]++;
      T.row[r0 + s] = r;
      T.slot[r] = (uint16_t)s;
    }
    for (int l = 0; l < nl; ++l)
      for (int s = cnt[l]; s < cnt[l + 1]; s += maxw) {
        const RangeLevel L{s, std::min(maxw, cnt[l + 1] - s)};
        T.lev.push_back(L);
        T.max_rows = std::max(T.max_rows, L.rows);
        for (int q = 0; q < L.rows; ++q) T.slot_lev[r0 + s + q] = (int)T.lev.size() - 1;
      }
    T.lev_ptr.push_back((int)T.lev.size());
    for (int s = 0; s < r1 - r0; ++s) {
      int beg, ne;
      range_entries(bs, lower, rows, diag, T.row[r0 + s], beg, ne);
      if (ne > sh.g * sh.k) return false;
      for (int e = 0; e < ne; ++e) {
        const int d = cols[beg + e];
        if ((d < r0 || d >= r1) && mark[d] != c) {
          mark[d] = c;
          T.ext.push_back(d);
        }
      }
    }
    T.ext_ptr.push_back((int)T.ext.size());
    T.max_ext = std::max(T.max_ext, T.ext_ptr[c + 1] - T.ext_ptr[c]);
  }
  return per + T.max_ext + 1 < 65536;
}

}  // namespace plan
}  // namespace egpu
