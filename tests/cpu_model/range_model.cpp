// Replays the row-range triangular solves (range_ilu in egpu_krylov.cuh) on the CPU with the
// product's own plan (egpu_tri_range.h): the same levels, slots, shared-memory indices and
// packed entries.  Ranges advance level by level, each only when every value it reads has been
// produced, so a plan that could deadlock, or that reads a wrong or unwritten cell, is reported.
#include <cmath>
#include <vector>

#include "../../elmerfem_b200/csrc/egpu_tri_range.h"

using namespace egpu::plan;

namespace {

std::vector<int> levels(int n, int bs, bool lower, const std::vector<int> &rows, const std::vector<int> &cols) {
  const int nb = n / bs;
  std::vector<int> lev(nb, 0);
  for (int q = 0; q < nb; ++q) {
    const int m = lower ? q : nb - 1 - q;
    int l = 0;
    for (int e = rows[m * bs]; e < rows[m * bs + 1]; ++e) {
      const int d = cols[e] / bs;
      if (lower ? d < m : d > m) l = std::max(l, lev[d] + 1);
    }
    lev[m] = l;
  }
  return lev;
}

struct Tri {
  RangeTriHost T;
  bool lower;
};

}  // namespace

// 0 and z = (LU)^-1 rhs; otherwise the code of the first violation.  vals: factors on the CRS
// structure, inverted U diagonal.
extern "C" int range_replay(int n, int bs, int per, const int *rows_, const int *cols_, const int *diag_,
                            const double *vals, const double *rhs, double *z) {
  const std::vector<int> rows(rows_, rows_ + n + 1), cols(cols_, cols_ + rows_[n]), diag(diag_, diag_ + n);
  int most = 0;
  for (int r = 0; r < n; r += bs)
    for (int t = 0; t < 2; ++t) {
      int beg, ne;
      range_entries(bs, t == 0, rows, diag, r, beg, ne);
      most = std::max(most, ne);
    }
  const RangeShape sh = range_shape(most);
  if (sh.g == 0) return -1;  // too many entries: the product takes another form
  const int g = sh.g, gk = sh.g * sh.k, nr = (n + per - 1) / per;
  Tri tri[2];
  int ext = 0;
  for (int t = 0; t < 2; ++t) {
    tri[t].lower = t == 0;
    const std::vector<int> lev = levels(n, bs, tri[t].lower, rows, cols);
    if (!range_triangle(n, bs, per, sh, tri[t].lower, rows, cols, diag, lev, tri[t].T)) return 1;
    if (!(range_cycles(n, bs, per, sh, tri[t].T.max_ext, tri[t].lower, rows, cols, diag, lev) > 0.0)) return 2;
    ext = std::max(ext, tri[t].T.max_ext);
  }
  const int zero = per + ext;
  std::vector<double> work(rhs, rhs + n), x(n);
  std::vector<double> in(n);
  for (int t = 0; t < 2; ++t) {
    const bool lower = tri[t].lower;
    RangeTriHost &T = tri[t].T;
    if (T.max_rows * g > RANGE_THREADS || range_record(T.max_rows, gk, 8) > RANGE_STAGE_BYTES) return 3;
    // right-hand sides times the inverse of the node block's triangle
    for (int r0 = 0; r0 < n; r0 += bs)
      for (int q = 0; q < bs; ++q) {
        const int k = lower ? q : bs - 1 - q, r = r0 + k;
        double v = work[r];
        for (int j = 0; j < bs; ++j)
          if (lower ? j < k : j > k) v -= vals[diag[r] + j - k] * in[r0 + j];
        in[r] = lower ? v : vals[diag[r]] * v;
      }
    // level records, as k_range_index and k_range_pack fill them
    std::vector<long long> offset(T.lev.size() + 1, 0);
    for (size_t l = 0; l < T.lev.size(); ++l) offset[l + 1] = offset[l] + range_record(T.lev[l].rows, gk, 8);
    std::vector<unsigned char> rec((size_t)offset.back());
    std::vector<int> where(n, 0);
    int seen = -1;
    for (int gs = 0; gs < n; ++gs) {
      const int c = gs / per, base = c * per, s = gs - base, r = T.row[gs], kr = r % bs, r0 = r - kr;
      if (c != seen) {
        for (int q = T.ext_ptr[c]; q < T.ext_ptr[c + 1]; ++q) where[T.ext[q]] = per + q - T.ext_ptr[c];
        seen = c;
      }
      const RangeLevel L = T.lev[T.slot_lev[gs]];
      unsigned char *R = rec.data() + offset[T.slot_lev[gs]];
      if (r < base || r >= std::min(n, base + per) || T.slot[r] != s || s < L.slot || s >= L.slot + L.rows) return 4;
      const int t = s - L.slot;
      const int beg0 = rows[r0], len = rows[r0 + 1] - beg0, e_lo = diag[r0] - beg0;
      const int off = lower ? 0 : e_lo + bs, ne = lower ? e_lo : len - e_lo - bs;
      for (int e = 0; e < gk; ++e) {
        double m[4], v = 0.0;
        int x = zero;
        if (e < ne) {
          const int d = cols[rows[r] + off + e];
          x = d >= base && d < std::min(n, base + per) ? (int)T.slot[d] : where[d];
          for (int q = 0; q < bs; ++q) {
            const int j = lower ? q : bs - 1 - q;
            double w = vals[beg0 + j * len + off + e];
            for (int i = 0; i < q; ++i) w -= vals[beg0 + j * len + e_lo + (lower ? i : bs - 1 - i)] * m[i];
            m[q] = lower ? w : w * vals[beg0 + j * len + e_lo + j];
            if (j == kr) v = m[q];
          }
        }
        const int at = range_entry_at(L.rows, g, t, e);
        reinterpret_cast<uint16_t *>(R + range_idx_at(L.rows))[at] = (uint16_t)x;
        reinterpret_cast<double *>(R + range_val_at(L.rows, gk))[at] = v;
      }
      reinterpret_cast<int *>(R)[4 + t] = r;
      reinterpret_cast<int *>(R)[0] = L.slot;
      reinterpret_cast<int *>(R)[1] = L.rows;
    }
    // the solve: cells of every range, NaN until written
    const double none = std::nan("");
    std::vector<std::vector<double>> cell(nr, std::vector<double>(zero + 1, none));
    std::vector<char> done(n, 0);
    std::vector<int> at(nr), fetched(nr, 0);
    for (int c = 0; c < nr; ++c) {
      at[c] = T.lev_ptr[c];
      cell[c][zero] = 0.0;
    }
    int left = (int)T.lev.size();
    while (left > 0) {
      bool moved = false;
      for (int c = 0; c < nr; ++c) {
        // external values in list order, as far as they have appeared
        for (; T.ext_ptr[c] + fetched[c] < T.ext_ptr[c + 1]; ++fetched[c]) {
          const int r = T.ext[T.ext_ptr[c] + fetched[c]];
          if (r / per == c) return 5;
          if (lower ? r > c * per : r < c * per) return 6;
          if (!done[r]) break;
          cell[c][per + fetched[c]] = x[r];
        }
        if (at[c] >= T.lev_ptr[c + 1]) continue;
        // the lanes' reads of the staged record
        const unsigned char *R = rec.data() + offset[at[c]];
        const RangeLevel L{reinterpret_cast<const int *>(R)[0], reinterpret_cast<const int *>(R)[1]};
        const int *rw = reinterpret_cast<const int *>(R) + 4;
        const uint16_t *ix = reinterpret_cast<const uint16_t *>(R + range_idx_at(L.rows));
        const double *vv = reinterpret_cast<const double *>(R + range_val_at(L.rows, gk));
        const int wg = L.rows * g;
        std::vector<double> out(L.rows, 0.0);
        bool ready = true;
        for (int tid = 0; tid < wg; ++tid)
          for (int k = 0; k < sh.k; ++k) {
            const int i = ix[k * wg + tid];
            if (i > zero) return 7;
            const double v = cell[c][i];
            if (v != v) {
              if (i < per) return 8;  // an own value of this or a later level
              ready = false;
            }
            out[tid / g] += vv[k * wg + tid] * v;
          }
        for (int s = 0; s < L.rows; ++s) out[s] = in[rw[s]] - out[s];
        if (!ready) continue;
        for (int s = 0; s < L.rows; ++s) {
          const int r = rw[s];
          if (done[r]) return 9;
          cell[c][L.slot + s] = x[r] = out[s];
          done[r] = 1;
        }
        at[c]++;
        --left;
        moved = true;
      }
      if (!moved) return 10;  // every range waits
    }
    for (int r = 0; r < n; ++r)
      if (!done[r]) return 11;
    work = x;
  }
  for (int r = 0; r < n; ++r) z[r] = x[r];
  return 0;
}
