// egpu_tri_cta.cu -- host side of the level-synchronous single-block ILU0 solves and of the
// row-range solves (second half of the file; plan in egpu_tri_range.h).
//
// The sync-free solves (egpu_krylov.cuh) spread a level over the whole GPU and pay a
// cross-SM publish/observe round trip per dependency level.  On meshes whose levels are
// narrow (a few hundred rows) and whose dependencies reach only a few levels back, one
// block running the levels in order out of shared memory is faster: its per-level cost is
// a __syncthreads, and the factor entries stream in through cp.async ahead of use.  This
// file builds that schedule (ELL blocks per level, ring-buffer slots, staging windows),
// fills it with the factor values after every factorisation, and decides per solve which
// of the two solves to run.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <thread>

#include "egpu_krylov.cuh"
#include "egpu_solve.h"
#include "egpu_tri_plan.h"
#include "egpu_tri_range.h"

namespace egpu {

namespace {

// dynamic shared memory of the single block (227 KB per block on sm_100, less the
// kernels' static shared memory and a margin)
constexpr size_t CTA_SMEM_MAX = 200 * 1024;

int tri_mode_env() {
  // EGPU_TRI_MODE: "syncfree" never uses the single-block solve, "block" uses it whenever
  // the schedule fits, "range" uses the row-range solve whenever it fits, anything else
  // chooses by the cost estimates
  const char *m = std::getenv("EGPU_TRI_MODE");
  if (!m) return 0;
  if (!std::strcmp(m, "syncfree")) return 1;
  if (!std::strcmp(m, "block")) return 2;
  if (!std::strcmp(m, "range")) return 3;
  return 0;
}

// Estimated seconds of one M^-1 application, from B200 measurements of the solves on hex
// meshes (Poisson and 3-DOF elasticity): sync-free, about 0.9 us per dependency level (a
// cross-SM publish/observe round trip) plus 0.8 ns per row; node-block sync-free, about
// 1.7 us per block level plus 0.65 ns per row; single block, about 0.6 us per level plus
// 4 ns per row (its entries streamed and summed by one SM), plus the extra grid barrier.
double est_syncfree(int nlev_lo, int nlev_up, int n) { return 0.9e-6 * (nlev_lo + nlev_up) + 0.8e-9 * 2.0 * n; }
double est_nodeblock(int nlev_lo, int nlev_up, int n) { return 1.7e-6 * (nlev_lo + nlev_up) + 0.65e-9 * 2.0 * n; }
double est_block(int nlev_lo, int nlev_up, int n) { return 0.6e-6 * (nlev_lo + nlev_up) + 4e-9 * 2.0 * n + 3e-6; }

// rows of a range for the k-th number of ranges that is tried, largest number first; false: none
// (EGPU_TRI_RANGES sets the only one)
constexpr int RANGE_COUNTS = 10;
bool range_rows_of(const egpu_ctx *ctx, int n, int bs, int k, int &per) {
  constexpr int div[RANGE_COUNTS] = {1, 2, 3, 4, 6, 9, 12, 18, 37, 148};
  const int forced = std::getenv("EGPU_TRI_RANGES") ? std::atoi(std::getenv("EGPU_TRI_RANGES")) : 0;
  if (k >= RANGE_COUNTS || (forced && k > 0)) return false;
  const int nr = std::max(1, std::min(ctx->num_sms, forced ? forced : ctx->num_sms / div[k]));
  per = ((n + nr - 1) / nr + bs - 1) / bs * bs;
  return true;
}

}  // namespace

// node-block sync-free solve (bl / bu block levels) instead of the row schedule (nlo / nup
// row levels, sync-free or single block)?  EGPU_TRI_NODE_BLOCKS=0 never, =1 always.
bool tri_prefer_node_blocks(int nlo, int nup, int bl, int bu, int n) {
  if (const char *e = std::getenv("EGPU_TRI_NODE_BLOCKS")) {
    if (!std::strcmp(e, "0")) return false;
    if (!std::strcmp(e, "1")) return true;
  }
  const int mode = tri_mode_env();
  if (mode == 2) return false;
  const double blk = est_nodeblock(bl, bu, n);
  if (blk >= est_syncfree(nlo, nup, n)) return false;
  return mode == 1 || blk < est_block(nlo, nup, n);
}

__global__ void k_cta_fill(long long nl, long long nu, const int *__restrict__ lsrc, const int *__restrict__ usrc,
                           const double *__restrict__ lo, const double *__restrict__ up,
                           const float *__restrict__ lo32, const float *__restrict__ up32, double *clo, double *cup,
                           float *clo32, float *cup32) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < nl + nu;
       t += (long long)gridDim.x * blockDim.x) {
    if (t < nl) {
      const int s = lsrc[t];
      clo[t] = s >= 0 ? lo[s] : 0.0;
      clo32[t] = s >= 0 ? lo32[s] : 0.0f;
    } else {
      const long long k = t - nl;
      const int s = usrc[k];
      cup[k] = s >= 0 ? up[s] : 0.0;
      cup32[k] = s >= 0 ? up32[s] : 0.0f;
    }
  }
}

// Build the single-block schedule next to the sync-free one.  lo / up: slot orders;
// lp, lc / upp, uc: packed strictly-lower / strictly-upper entries per slot.
int build_cta_schedule(egpu_mat *A, const std::vector<int> &rows, const std::vector<int> &cols,
                       const std::vector<int> &diag, const std::vector<int> &lo, const std::vector<int> &up,
                       const std::vector<int> &lp, const std::vector<int> &lc, const std::vector<int> &upp,
                       const std::vector<int> &uc) {
  egpu_ctx *ctx = A->ctx;
  TriSchedule &S = A->tri;
  const int n = A->n;
  S.cta_ok[0] = S.cta_ok[1] = false;
  const int mode = tri_mode_env();
  if (mode == 1 || n == 0) return EGPU_OK;
  plan::Plan P;
  plan::make_plan(n, rows, cols, diag, lo, up, lp, lc, upp, uc, CTA_SMEM_MAX, P);
  if (!P.ok) return EGPU_OK;
  bool any = false;
  for (int v = 0; v < 2; ++v)
    if (P.fits[v] && (mode == 2 || est_block(P.lo.nlev, P.up.nlev, n) < est_syncfree(P.lo.nlev, P.up.nlev, n)))
      any = true;
  if (!any) return EGPU_OK;
  if (!plan::plan_arrays(P, n, lo, up, lp, lc, upp, uc)) {
    egpu_set_error(ctx, "internal: level-synchronous schedule dependency out of range");
    return EGPU_ERR_ARG;
  }
  auto upload = [&](const plan::TriPlan &T, CtaTriHost &H) -> int {
    std::vector<int4> lev(std::max<size_t>(1, T.lev.size()), make_int4(0, 0, 0, 0));
    for (size_t L = 0; L < T.lev.size(); ++L) lev[L] = make_int4(T.lev[L].x, T.lev[L].y, T.lev[L].z, T.lev[L].w);
    EGPU_CUDA_TRY(ctx, H.lev.alloc(lev.size()));
    EGPU_CUDA_TRY(ctx, H.ridx.alloc(T.nent));
    EGPU_CUDA_TRY(ctx, H.src.alloc(T.nent));
    EGPU_CUDA_TRY(ctx, H.map.alloc(T.map.size()));
    EGPU_CUDA_TRY(ctx, egpu_copy(ctx, H.lev.p, lev.data(), lev.size() * sizeof(int4), cudaMemcpyHostToDevice));
    EGPU_CUDA_TRY(ctx, egpu_copy(ctx, H.ridx.p, T.ridx.data(), T.nent * sizeof(uint16_t), cudaMemcpyHostToDevice));
    EGPU_CUDA_TRY(ctx, egpu_copy(ctx, H.src.p, T.src.data(), T.nent * sizeof(int), cudaMemcpyHostToDevice));
    EGPU_CUDA_TRY(ctx, egpu_copy(ctx, H.map.p, T.map.data(), T.map.size() * sizeof(int), cudaMemcpyHostToDevice));
    H.nlev = T.nlev;
    H.nent = T.nent;
    return EGPU_OK;
  };
  int rc = upload(P.lo, S.cta_lo);
  if (!rc) rc = upload(P.up, S.cta_up);
  if (rc) return rc;
  EGPU_CUDA_TRY(ctx, S.pos_lo.alloc(P.pos_lo.size()));
  EGPU_CUDA_TRY(ctx, S.pos_up.alloc(P.pos_up.size()));
  EGPU_CUDA_TRY(ctx, egpu_copy(ctx, S.pos_lo.p, P.pos_lo.data(), P.pos_lo.size() * sizeof(int), cudaMemcpyHostToDevice));
  EGPU_CUDA_TRY(ctx, egpu_copy(ctx, S.pos_up.p, P.pos_up.data(), P.pos_up.size() * sizeof(int), cudaMemcpyHostToDevice));
  S.cta_rs = P.rs;
  for (int v = 0; v < 2; ++v) {
    S.cta_ok[v] = P.fits[v];
    S.cta_pd[v] = P.pd[v];
    S.cta_sb[v] = P.sb[v];
    S.cta_sr[v] = P.sr[v];
    S.cta_smem[v] = P.smem[v];
  }
  return EGPU_OK;
}

// the factors in the ELL layout, after every factorisation
int cta_fill_values(egpu_mat *A) {
  const TriSchedule &S = A->tri;
  if (!S.cta_ok[0] && !S.cta_ok[1]) return EGPU_OK;
  egpu_ctx *ctx = A->ctx;
  const long long nl = S.cta_lo.nent, nu = S.cta_up.nent;
  EGPU_CUDA_TRY(ctx, A->cta_lo_vals.alloc(nl));
  EGPU_CUDA_TRY(ctx, A->cta_up_vals.alloc(nu));
  EGPU_CUDA_TRY(ctx, A->cta_lo_vals32.alloc(nl));
  EGPU_CUDA_TRY(ctx, A->cta_up_vals32.alloc(nu));
  const long long tot = nl + nu;
  const int grid = (int)std::max(1LL, std::min((tot + 255) / 256, (long long)ctx->num_sms * 8));
  k_cta_fill<<<grid, 256, 0, ctx->stream>>>(nl, nu, S.cta_lo.src.p, S.cta_up.src.p, A->lo_vals.p, A->up_vals.p,
                                             A->lo_vals32.p, A->up_vals32.p, A->cta_lo_vals.p, A->cta_up_vals.p,
                                             A->cta_lo_vals32.p, A->cta_up_vals32.p);
  ctx->launches++;
  EGPU_CUDA_TRY(ctx, cudaGetLastError());
  return EGPU_OK;
}

// threads of the block taking part in the level-synchronous solve: enough for the widest
// level, a multiple of 32, at most the block (EGPU_TRI_THREADS overrides)
int cta_threads(const egpu_mat *A) {
  int nt = 512;
  if (const char *e = std::getenv("EGPU_TRI_THREADS")) nt = std::atoi(e);
  nt = std::max(32, std::min(EGPU_KBLOCK, nt));
  return nt / 32 * 32;
}

// single-block solve for this precision (v = 0 FP64, 1 FP32)?
bool cta_use(const egpu_mat *A, int v) {
  const TriSchedule &S = A->tri;
  if (!S.cta_ok[v] || !A->cta_lo_vals.p) return false;
  const int mode = tri_mode_env();
  if (mode == 1) return false;
  if (mode == 2) return true;
  return est_block(S.cta_lo.nlev, S.cta_up.nlev, A->n) < est_syncfree(S.cta_lo.nlev, S.cta_up.nlev, A->n);
}

// shared-memory index of every padded entry (by global slot): the own row's slot, an external
// row's cell, or the zero cell
template <bool LOWER>
__global__ void k_range_index(int n, int bs, int per, int gk, int zero, const int *__restrict__ row,
                              const uint16_t *__restrict__ slot, const int *__restrict__ ext_ptr,
                              const int2 *__restrict__ sorted, const int *__restrict__ rows,
                              const int *__restrict__ cols, const int *__restrict__ diag, uint16_t *__restrict__ idx) {
  const long long tot = (long long)n * gk;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < tot; q += (long long)gridDim.x * blockDim.x) {
    const int gs = (int)(q / gk), e = (int)(q % gk), c = gs / per, r0 = c * per;
    const int r = row[gs], rb = r / bs * bs, e_lo = diag[rb] - rows[rb], len = rows[rb + 1] - rows[rb];
    const int beg = rows[r] + (LOWER ? 0 : e_lo + bs), ne = LOWER ? e_lo : len - e_lo - bs;
    int x = zero;
    if (e < ne) {
      const int d = cols[beg + e];
      if (d >= r0 && d < min(n, r0 + per)) {
        x = slot[d];
      } else {
        int lo = ext_ptr[c], hi = ext_ptr[c + 1] - 1;
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (sorted[mid].x < d)
            lo = mid + 1;
          else
            hi = mid;
        }
        x = per + sorted[lo].y;
      }
    }
    idx[q] = (uint16_t)x;
  }
}

constexpr size_t RANGE_SMEM = 216 * 1024;
constexpr double RANGE_PASSES = 8e-6;

namespace {

// The form is a choice: where its buffers do not fit the free device memory, the solve takes
// another form, whose buffers it has anyway.  EGPU_ERR_ALLOC for that, else EGPU_ERR_CUDA
template <typename T>
int range_buffer(egpu_ctx *ctx, DevBuf<T> &b, size_t count) {
  const cudaError_t e = b.alloc(count);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();  // not sticky
    return EGPU_ERR_ALLOC;
  }
  EGPU_CUDA_TRY(ctx, e);
  return EGPU_OK;
}

// one number of ranges: its plan and modelled time; fit 0: shared memory holds it in FP64, 1: in
// FP32 only, 2: neither
struct RangeChoice {
  int per = 0, fit = 2;
  double t = 0.0;
  plan::RangeTriHost lo, up;
};

}  // namespace

// Row-range solves when their modelled time (cycles at the 1.9 GHz the cards run at, plus the
// passes over the right-hand side) beats the estimates of the other schedules.  The number of
// ranges is the best of a few: fewer mean fewer hand-overs through L2, more mean narrower
// levels and less shared memory.  Own values, external values and right-hand sides of a range
// have to fit in shared memory (RANGE_SMEM of the 227 KB), in FP64 if any number of ranges
// allows it, else in FP32 only.
//
// The plan is host work (hex 64^3: 14 ms of counting and 9 ms of modelling a triangle and number of
// ranges), so the numbers are tried side by side, each on a thread, and one whose model without
// external values is too slow already is dropped before it is planned.  First exact solve less
// second, 16-core host: hex 32^3 12 ms, 64^3 93 ms, 96^3 240 ms, elasticity 64^3 (form not taken)
// 243 ms; one after another 100, 470, 900 and 900 ms and more.
static int build_range_schedule(egpu_mat *A, const std::vector<int> &rows, const std::vector<int> &cols,
                                const std::vector<int> &diag) {
  egpu_ctx *ctx = A->ctx;
  TriSchedule &S = A->tri;
  const int n = A->n, bs = S.bs, mode = tri_mode_env();
  int most = 0;
  for (int r = 0; r < n; r += bs) {
    int beg, ne;
    plan::range_entries(bs, true, rows, diag, r, beg, ne);
    most = std::max(most, ne);
    plan::range_entries(bs, false, rows, diag, r, beg, ne);
    most = std::max(most, ne);
  }
  const plan::RangeShape sh = plan::range_shape(most);
  if (sh.g == 0) return EGPU_OK;
  std::vector<int> lev_lo, lev_up;
  plan::range_levels(n, bs, true, rows, cols, lev_lo);
  plan::range_levels(n, bs, false, rows, cols, lev_up);
  // measured per application: sync-free 0.8 us a level + 0.24 ns a row, node blocks 1.25 us +
  // 0.4 ns (hex 32^3 372 us, 96^3 1,335 us; elasticity 24^3 440 us, 64^3 1,430 us), where the
  // row ranges take 185, 1,090, 230 and 1,600 us
  const double levels = S.lower_levels + S.upper_levels;
  const double spread = bs > 1 ? 1.25e-6 * levels + 0.4e-9 * n : 0.8e-6 * levels + 0.24e-9 * n;
  constexpr double SCATTER = 1.15;  // the model's
  auto seconds = [&](int per, int ext) {
    return (plan::range_cycles(n, bs, per, sh, ext, true, rows, cols, diag, lev_lo) +
            plan::range_cycles(n, bs, per, sh, ext, false, rows, cols, diag, lev_up)) / 1.9e9 + RANGE_PASSES;
  };
  auto evaluate = [&](RangeChoice &c) {
    if (mode != 3 && SCATTER * seconds(c.per, 0) >= spread) return;
    if (!plan::range_triangle(n, bs, c.per, sh, true, rows, cols, diag, lev_lo, c.lo) ||
        !plan::range_triangle(n, bs, c.per, sh, false, rows, cols, diag, lev_up, c.up))
      return;
    const int ext = std::max(c.lo.max_ext, c.up.max_ext), maxr = std::max(c.lo.max_rows, c.up.max_rows);
    auto bytes = [&](int vsize) { return plan::range_record(maxr, sh.g * sh.k, vsize); };
    if (range_smem_bytes<float>(c.per, ext, bytes(4)) > RANGE_SMEM) return;
    c.t = seconds(c.per, ext);
    c.fit = range_smem_bytes<double>(c.per, ext, bytes(8)) <= RANGE_SMEM ? 0 : 1;
  };
  std::vector<RangeChoice> choices(RANGE_COUNTS);
  size_t nc = 0;
  for (; nc < choices.size() && range_rows_of(ctx, n, bs, (int)nc, choices[nc].per); ++nc)
    if (range_smem_bytes<float>(choices[nc].per, 0, 0) > RANGE_SMEM || choices[nc].per > 32000) break;
  choices.resize(nc);
  {
    std::vector<std::thread> threads;
    for (RangeChoice &c : choices) {
      auto run = [&evaluate, &c] {
        try {
          evaluate(c);
        } catch (...) {  // out of host memory: not chosen
          c.fit = 2;
        }
      };
      if (&c == &choices.back()) {
        run();
        break;
      }
      try {
        threads.emplace_back(run);
      } catch (...) {  // no more threads: here
        run();
      }
    }
    for (std::thread &t : threads) t.join();
  }
  const RangeChoice *best = nullptr;
  for (const RangeChoice &c : choices)
    if (c.fit < 2 && (!best || c.fit < best->fit || (c.fit == best->fit && c.t < best->t))) best = &c;
  if (!best) return EGPU_OK;
  const plan::RangeTriHost &best_lo = best->lo, &best_up = best->up;
  const int best_per = best->per, best_fit = best->fit;
  double other = spread;
  if (S.cta_ok[best_fit]) other = std::min(other, est_block(S.cta_lo.nlev, S.cta_up.nlev, n));
  if (mode != 3 && SCATTER * best->t >= other) return EGPU_OK;
  const int ext = std::max(best_lo.max_ext, best_up.max_ext);
  const int gk = sh.g * sh.k;
  auto upload = [&](const plan::RangeTriHost &T, bool lower, RangeTriDev &D) -> int {
    static_assert(sizeof(plan::RangeLevel) == sizeof(int2), "levels are read as int2");
    auto put = [&](auto &dst, const auto &src) -> int {
      const int rc = range_buffer(ctx, dst, std::max<size_t>(1, src.size()));
      if (rc || src.empty()) return rc;
      EGPU_CUDA_TRY(ctx, egpu_copy(ctx, dst.p, src.data(), src.size() * sizeof(src[0]), cudaMemcpyHostToDevice));
      return EGPU_OK;
    };
    int rc = put(D.lev_ptr, T.lev_ptr);
    if (!rc) rc = put(D.lev, T.lev);
    if (!rc) rc = put(D.slot_lev, T.slot_lev);
    if (!rc) rc = put(D.row, T.row);
    if (!rc) rc = put(D.slot, T.slot);
    if (!rc) rc = put(D.ext_ptr, T.ext_ptr);
    if (!rc) rc = put(D.ext, T.ext);
    for (int v = 0; v < 2 && !rc; ++v) {
      std::vector<long long> off(T.lev.size() + 1, 0);
      for (size_t l = 0; l < T.lev.size(); ++l)
        off[l + 1] = off[l] + plan::range_record(T.lev[l].rows, gk, v == 0 ? 8 : 4);
      D.bytes[v] = off.back();
      rc = put(D.offset[v], off);
    }
    if (rc) return rc;
    // shared-memory indices, on the device: external rows through a sorted copy of each list
    std::vector<int2> sorted(std::max<size_t>(1, T.ext.size()));
    for (size_t c = 0; c + 1 < T.ext_ptr.size(); ++c) {
      for (int q = T.ext_ptr[c]; q < T.ext_ptr[c + 1]; ++q) sorted[q] = make_int2(T.ext[q], q - T.ext_ptr[c]);
      std::sort(sorted.begin() + T.ext_ptr[c], sorted.begin() + T.ext_ptr[c + 1],
                [](int2 x, int2 y) { return x.x < y.x; });
    }
    DevBuf<int2> ds;
    rc = put(ds, sorted);
    if (!rc) rc = range_buffer(ctx, D.idx, (size_t)n * gk);
    if (rc) return rc;
    const int grid = (int)std::max(1LL, std::min(((long long)n * gk + 255) / 256, (long long)ctx->num_sms * 32));
    if (lower)
      k_range_index<true><<<grid, 256, 0, ctx->stream>>>(n, bs, best_per, gk, best_per + ext, D.row.p, D.slot.p,
                                                         D.ext_ptr.p, ds.p, A->ilu_rows.p, A->ilu_cols.p,
                                                         A->ilu_diag.p, D.idx.p);
    else
      k_range_index<false><<<grid, 256, 0, ctx->stream>>>(n, bs, best_per, gk, best_per + ext, D.row.p, D.slot.p,
                                                          D.ext_ptr.p, ds.p, A->ilu_rows.p, A->ilu_cols.p,
                                                          A->ilu_diag.p, D.idx.p);
    ctx->launches++;
    EGPU_CUDA_TRY(ctx, cudaGetLastError());
    EGPU_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    return EGPU_OK;
  };
  int rc = upload(best_lo, true, S.rg_lo);
  if (!rc) rc = upload(best_up, false, S.rg_up);
  if (rc) return rc;
  const int maxr = std::max(best_lo.max_rows, best_up.max_rows);
  S.rg_rows = best_per;
  S.rg_ext = ext;
  S.rg_g = sh.g;
  S.rg_k = sh.k;
  S.rg_nt = (maxr * sh.g + 31) / 32 * 32;
  S.rg_stage[0] = plan::range_record(maxr, gk, 8);
  S.rg_stage[1] = plan::range_record(maxr, gk, 4);
  S.rg_ok[0] = best_fit == 0;
  S.rg_ok[1] = true;
  return EGPU_OK;
}

void range_view(TriSchedule &T, const TriSchedule &P) {
  T.rg_rows = P.rg_rows;
  T.rg_ext = P.rg_ext;
  T.rg_g = P.rg_g;
  T.rg_k = P.rg_k;
  T.rg_nt = P.rg_nt;
  for (int v = 0; v < 2; ++v) {
    T.rg_ok[v] = P.rg_ok[v];
    T.rg_stage[v] = P.rg_stage[v];
  }
  T.rg_built = P.rg_built;
  T.rg_lo.view(P.rg_lo);
  T.rg_up.view(P.rg_up);
}

// Makes the row-range plan of the ILU structure if it is not made yet; called before an exact
// triangular solve in precision v, or where one is prepared, and by nothing else, so that
// batches, Jacobi sweeps and matrices that are only factorised do not pay for it.  An ILUT factor has a new structure
// with every factorisation and is planned only where the form is asked for (EGPU_TRI_MODE=range):
// the plan costs more than one solve gains.
int ensure_range_plan(egpu_mat *A, int v) {
  TriSchedule &S = A->tri;
  const int mode = tri_mode_env();
  if (!A->tri_built || S.rg_built || mode == 1 || mode == 2) return EGPU_OK;
  if (A->ilu_order == ILU_ORDER_T && mode != 3) return EGPU_OK;
  egpu_ctx *ctx = A->ctx;
  const int n = A->n;
  int per = 0;  // of the most ranges: what FP64 cannot hold there, it can hold nowhere
  if (v == 0 && range_rows_of(ctx, n, S.bs, 0, per) && range_smem_bytes<double>(per, 0, 0) > RANGE_SMEM) return EGPU_OK;
  if (A->parent) {  // a clone shares its prototype's plan
    const int rc = ensure_range_plan(A->parent, v);
    if (rc) return rc;
    range_view(S, A->parent->tri);
    return EGPU_OK;
  }
  std::vector<int> rows(n + 1), cols(A->ilu_nnz), diag(n);
  EGPU_CUDA_TRY(ctx, egpu_copy(ctx, rows.data(), A->ilu_rows.p, (n + 1) * sizeof(int), cudaMemcpyDeviceToHost));
  EGPU_CUDA_TRY(ctx, egpu_copy(ctx, cols.data(), A->ilu_cols.p, A->ilu_nnz * sizeof(int), cudaMemcpyDeviceToHost));
  EGPU_CUDA_TRY(ctx, egpu_copy(ctx, diag.data(), A->ilu_diag.p, n * sizeof(int), cudaMemcpyDeviceToHost));
  const int rc = build_range_schedule(A, rows, cols, diag);
  if (rc == EGPU_ERR_ALLOC) {
    S.rg_lo.release();
    S.rg_up.release();
  } else if (rc) {
    return rc;
  }
  S.rg_built = true;
  return EGPU_OK;
}

bool range_use(const egpu_mat *A, int v) {
  const int mode = tri_mode_env();
  return A->tri.rg_rows > 0 && A->tri.rg_ok[v] && !A->rg_off[v] && mode != 1 && mode != 2;
}

// The level records of a triangle (plan::RangeLevel) with the factors' values.  bs > 1: row k of a
// node block takes column e of the block's out-of-block part times the inverse of the block's
// unit lower triangle, or of its upper triangle with the inverted diagonal; bs == 1: L_ij, or
// u_ii^-1 U_ij.
template <typename VT, bool LOWER>
__global__ void k_range_pack(int n, int bs, int per, int g, int gk, const int *__restrict__ row,
                             const int *__restrict__ slot_lev, const int2 *__restrict__ lev,
                             const long long *__restrict__ offset, const uint16_t *__restrict__ idx,
                             const int *__restrict__ rows, const int *__restrict__ diag,
                             const double *__restrict__ ilu, unsigned char *__restrict__ rec) {
  const long long tot = (long long)n * gk;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < tot; q += (long long)gridDim.x * blockDim.x) {
    const int gs = (int)(q / gk), e = (int)(q % gk);
    const int l = slot_lev[gs], s = gs % per;
    const int2 L = lev[l];
    unsigned char *R = rec + offset[l];
    const int r = row[gs], kr = r % bs, r0 = r - kr, t = s - L.x;
    const int beg0 = rows[r0], len = rows[r0 + 1] - beg0, e_lo = diag[r0] - beg0;
    const int off = LOWER ? 0 : e_lo + bs, ne = LOWER ? e_lo : len - e_lo - bs;
    double v = 0.0;
    if (e < ne) {
      if (bs == 1) {
        v = ilu[beg0 + off + e];
        if (!LOWER) v *= ilu[diag[r0]];
      } else {
        double m[TRI_BS_MAX];
        for (int i = 0; i < bs; ++i) {
          const int j = LOWER ? i : bs - 1 - i;  // rows in elimination order, up to this one
          double w = ilu[beg0 + j * len + off + e];
          const double *in = ilu + beg0 + j * len + e_lo;
          for (int h = 0; h < i; ++h) w -= in[LOWER ? h : bs - 1 - h] * m[h];
          if (!LOWER) w *= in[j];
          m[i] = w;
          if (j == kr) {
            v = w;
            break;
          }
        }
      }
    }
    const int at = plan::range_entry_at(L.y, g, t, e);
    reinterpret_cast<uint16_t *>(R + plan::range_idx_at(L.y))[at] = idx[q];
    reinterpret_cast<VT *>(R + plan::range_val_at(L.y, gk))[at] = (VT)v;
    if (e == 0) {
      reinterpret_cast<int *>(R)[4 + t] = r;
      if (t == 0) *reinterpret_cast<int4 *>(R) = make_int4(L.x, L.y, 0, 0);
    }
  }
}

// the record buffers of a precision, and its packing kernels loaded
int range_alloc(egpu_mat *A, int v) {
  if (!A->tri_built) return EGPU_OK;
  int rc = ensure_range_plan(A, v);
  if (rc || !range_use(A, v)) return rc;
  egpu_ctx *ctx = A->ctx;
  rc = range_buffer(ctx, A->rg_lo_rec[v], A->tri.rg_lo.bytes[v]);
  if (!rc) rc = range_buffer(ctx, A->rg_up_rec[v], A->tri.rg_up.bytes[v]);
  if (rc == EGPU_ERR_ALLOC) {
    A->rg_lo_rec[v].release();
    A->rg_up_rec[v].release();
    A->rg_off[v] = true;
    return EGPU_OK;
  }
  if (rc) return rc;
  cudaFuncAttributes fa;
  EGPU_CUDA_TRY(ctx, v == 0 ? cudaFuncGetAttributes(&fa, k_range_pack<double, true>)
                            : cudaFuncGetAttributes(&fa, k_range_pack<float, true>));
  EGPU_CUDA_TRY(ctx, v == 0 ? cudaFuncGetAttributes(&fa, k_range_pack<double, false>)
                            : cudaFuncGetAttributes(&fa, k_range_pack<float, false>));
  return EGPU_OK;
}

template <typename VT>
static int range_pack_as(egpu_mat *A, int v) {
  egpu_ctx *ctx = A->ctx;
  const TriSchedule &S = A->tri;
  const int gk = S.rg_g * S.rg_k;
  const int grid = (int)std::max(1LL, std::min(((long long)A->n * gk + 255) / 256, (long long)ctx->num_sms * 32));
  const int rc = range_alloc(A, v);
  if (rc || !range_use(A, v)) return rc;
  k_range_pack<VT, true><<<grid, 256, 0, ctx->stream>>>(
      A->n, S.bs, S.rg_rows, S.rg_g, gk, S.rg_lo.row.p, S.rg_lo.slot_lev.p, S.rg_lo.lev.p, S.rg_lo.offset[v].p,
      S.rg_lo.idx.p, A->ilu_rows.p, A->ilu_diag.p, A->ilu.p, A->rg_lo_rec[v].p);
  k_range_pack<VT, false><<<grid, 256, 0, ctx->stream>>>(
      A->n, S.bs, S.rg_rows, S.rg_g, gk, S.rg_up.row.p, S.rg_up.slot_lev.p, S.rg_up.lev.p, S.rg_up.offset[v].p,
      S.rg_up.idx.p, A->ilu_rows.p, A->ilu_diag.p, A->ilu.p, A->rg_up_rec[v].p);
  ctx->launches += 2;
  EGPU_CUDA_TRY(ctx, cudaGetLastError());
  A->rg_packed[v] = true;
  return EGPU_OK;
}

int range_pack(egpu_mat *A, int v) {
  const int rc = ensure_range_plan(A, v);
  if (rc || !range_use(A, v) || A->rg_packed[v]) return rc;
  return v == 0 ? range_pack_as<double>(A, v) : range_pack_as<float>(A, v);
}

}  // namespace egpu
