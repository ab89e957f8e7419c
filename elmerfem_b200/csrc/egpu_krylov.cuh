// egpu_krylov.cuh -- persistent Krylov kernels (CG, BiCGStab) with Jacobi / ILU0.
//
// One cooperative launch runs a whole solve.  Phases are separated by a bounded grid
// barrier; dot products are block partials reduced in a fixed order (deterministic).
//
// FP64 drop-in mode (true_residual = 1) keeps HUTI's operation sequence
// (hutiter/src/huti_cg_D.F90:158-240, huti_bicgstab_D.F90:171-267) and its stopping
// test ||A x_k - b|| / ||b|| < tol.  The A x_k product is computed in the same pass
// over the matrix as the next iteration's first SpMV (two right-hand sides per matrix
// read), so the decision for iterate k is taken one phase later; x_k is kept
// untouched until then, which returns the same iterate and HUTI_ITERS as HUTI.
//
// FP32 inner mode (true_residual = 0) is the inner solver of the mixed-precision
// refinement: x0 = 0, stopping on the recursive residual ||r_k|| <= tol * ||r_0||.  With
// resume set, a segment continues the previous one's search directions after its residual
// was replaced by the FP64 true residual (reliable updating, Sleijpen & van der Vorst 1996):
// no Krylov information is thrown away at a refinement.
#pragma once

#include "egpu_internal.cuh"
#include "egpu_tri_range.h"

namespace egpu {

enum { SLOT_BB = 0, SLOT_RHO, SLOT_PQ, SLOT_RR, SLOT_SS, SLOT_TS, SLOT_TT, SLOT_RR2, NUM_SLOTS };

// Forms of the ILU solves: sync-free (rows or node blocks; also the form of kernels without
// ILU), level-synchronous in block 0, row ranges (7 or 10 entries a lane)
enum TriForm { TRI_SYNCFREE = 0, TRI_CTA, TRI_RANGE7, TRI_RANGE10 };
constexpr bool tri_range(int form) { return form == TRI_RANGE7 || form == TRI_RANGE10; }

// One triangle of the row-range solve on the device: the level records of every range
// (laid out by plan::range_record, with values), slot of every row, external rows
struct RangeTri {
  const int *lev_ptr;
  const long long *offset;
  const unsigned char *rec;
  const uint16_t *slot;
  const int *ext_ptr, *ext;
};

// One triangle of the level-synchronous solve (layout described at CtaTriHost)
template <typename VT>
struct CtaTri {
  int nlev;
  const int4 *lev;          // {first slot, rows, entries per row, ELL offset}
  const uint16_t *ridx;     // ring slot of each ELL entry's column
  const VT *vals;           // ELL values
  const int *map;           // lower: upper-order slot of the row; upper: the row
};

template <typename VT>
struct KArgs {
  int n;
  const int *rows, *cols, *diag;  // 0-based CRS
  const int16_t *cols16;          // col - row offsets (FP32 path, optional)
  const VT *ilu;                  // ILU0 factors (inverted U diagonal)
  const VT *dvals;                // diagonal of the scaled matrix (Jacobi)
  const int *lower_order, *upper_order;
  int precond, maxit, true_residual;
  double tol;
  double divtol;                  // Linear System Divergence Tolerance (<= 0: none); GCR, BiCGStab(l)
  const VT *b;
  VT *x;
  VT *w;                          // work vectors, stride ldw
  long long ldw;
  unsigned int *bar;
  int *err;
  double *partials;               // NUM_SLOTS * gridDim.x
  int *out_i;                     // [0] info [1] iters
  double *out_d;                  // [0] residual [1] rhsnorm
  const unsigned int *skip;       // bit 1 set: zero right-hand side, return at once
  int tri_per_block;              // sub-warps per block taking part in the triangular solves
  int tri_bs;                     // rows per sync-free slot group (node blocks; 1 = row per slot)
  int unit_diag;                  // FP32 inner CG: every diagonal of the scaled matrix is 1.0f, so the
                                  // Jacobi step is the identity (Z is R, no diagonal loads)
  // ILU0 factors packed in solve order (see TriSchedule)
  const int *lo_ptr, *lo_cols, *up_ptr, *up_cols;
  const VT *lo_vals, *up_vals, *up_dinv;
  // SELL-32 copy of the scaled matrix used by every SpMV of the Krylov loop
  int nslices;
  const int *sell_ptr, *sell_w, *scols;
  const int16_t *scols16;
  const VT *svals;
  const int *sell_cptr;           // compact offsets (OFFS path): see egpu_mat::sell_cptr
  const int16_t *scolsc;
  // level-synchronous triangular solves run by block 0 out of shared memory (tri_cta != 0):
  // levels staged cta_pd ahead, ring of cta_rs slots, staging windows of cta_sb entries and
  // cta_sr rows
  int tri_cta, cta_pd, cta_rs, cta_sb, cta_sr, cta_nl, cta_nt;
  // FP32 inner solves with ILU0: M^-1 by sweeps_l / sweeps_u Jacobi sweeps on the factors
  // (0: exact triangular solves).  The factors in the matrix's SELL layout (isvals; the
  // diagonal entries unused), the inverted U diagonal in row order (idinv), and per slice
  // the k range holding its strictly-lower entries (swr.x: [0, x)) and its strictly-upper
  // ones (swr.y: [y, w)).
  int sweeps_l, sweeps_u;
  const int2 *swr;
  const VT *isvals, *idinv;
  // inner mode, reliable update: continue the previous segment's recurrences from a replaced
  // residual (B = the new true residual / its norm) instead of restarting.  carry holds
  // the previous segment's scalars (rho_{k-1}, alpha, omega; [3] = 1 when valid) and is
  // written back at a converged exit; ru_c = old residual norm / new residual norm.
  int resume;
  double ru_c;
  double *carry;
  // GCR / BiCGStab(l): restart length or polynomial degree, and extra stored vectors
  // (ext_nvec of them, stride ext_lds)
  int ext_m;
  VT *ext;
  long long ext_lds;
  const int *pos_lo, *pos_up;     // solve slot of each row, lower / upper order
  CtaTri<VT> clo, cup;
  // row-range solves (range_ilu): rows per range (0: off), external cells, log2 lanes a row,
  // threads that solve rows, bytes of a stage; the ILU structure's diagonal positions
  int rg_rows, rg_ext, rg_lg, rg_nt, rg_stage;
  RangeTri rlo, rup;
  const int *idiag;
};

// row sum step: FP64 keeps CRS_MatrixVectorProd's rounding (s = s + a*x, two roundings, row
// order); FP32 uses a fused multiply-add
__device__ __forceinline__ double row_madd(double s, double a, double x) { return __dadd_rn(s, __dmul_rn(a, x)); }
__device__ __forceinline__ float row_madd(float s, float a, float x) { return fmaf(a, x, s); }

// ---- 16-byte vector access for the element-wise phases (all work vectors are 256-byte
// aligned with a stride that is a multiple of 64 elements)
template <int W, typename VT>
__device__ __forceinline__ void vld(const VT *p, int i, VT (&v)[W]) {
  if constexpr (W == 1) {
    v[0] = p[i];
  } else if constexpr (sizeof(VT) == 8) {
    const double2 t = *reinterpret_cast<const double2 *>(p + i);
    v[0] = t.x;
    v[1] = t.y;
  } else {
    const float4 t = *reinterpret_cast<const float4 *>(p + i);
    v[0] = t.x;
    v[1] = t.y;
    v[2] = t.z;
    v[3] = t.w;
  }
}
template <int W, typename VT>
__device__ __forceinline__ void vst(VT *p, int i, const VT (&v)[W]) {
  if constexpr (W == 1) {
    p[i] = v[0];
  } else if constexpr (sizeof(VT) == 8) {
    *reinterpret_cast<double2 *>(p + i) = make_double2(v[0], v[1]);
  } else {
    *reinterpret_cast<float4 *>(p + i) = make_float4(v[0], v[1], v[2], v[3]);
  }
}
template <int W, typename VT>
__device__ __forceinline__ void vfill(VT *p, int i, VT x) {
  VT v[W];
#pragma unroll
  for (int k = 0; k < W; ++k) v[k] = x;
  vst<W>(p, i, v);
}

template <int W>
struct VW {
  static constexpr int value = W;
};

// f(i, VW<W>) over [0, n): 16-byte chunks, then a scalar tail
template <typename VT, typename F>
__device__ __forceinline__ void vec_loop(int n, F &&f) {
  constexpr int W = 16 / sizeof(VT);
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
  const int nv = n / W;
  for (int q = tid; q < nv; q += nth) f(q * W, VW<W>{});
  for (int i = nv * W + tid; i < n; i += nth) f(i, VW<1>{});
}

// Participants of the sync-free solves: the first tri_per_block sub-warps of every block,
// numbered block-fastest so consecutive slots land on different SMs.
template <int TS>
__device__ __forceinline__ bool tri_participant(int per_block, int &id, int &count) {
  const int local = threadIdx.x / TS;
  count = per_block * gridDim.x;
  id = local * gridDim.x + blockIdx.x;
  return local < per_block;
}

template <typename VT>
__device__ __forceinline__ VT ld_stream(const VT *p) {
  return __ldcs(p);
}
// Gathers of vectors written earlier in the same launch use plain cache-all loads: every
// phase starts after grid_barrier, whose acquiring poll discards stale L1 lines, and the
// stencil's reuse of x across neighbouring rows is then served from L1.
template <typename VT>
__device__ __forceinline__ VT ld_l2(const VT *p) {
  return __ldca(p);
}

// -------------------------------------------------------------------------------------
// SpMV over all rows on the SELL-32 copy: one warp per slice of 32 rows, lane = row, the
// slice's entries column-major so each step of k is one coalesced 128-byte (FP32) or
// 256-byte (FP64) warp load; each row sums in entry order.  Padding entries carry value 0
// and a valid column.  epi(row, s0, s1) runs once per row on its own lane.
//
// The loops take U entries at a time, loads first; what is left over at the end of a row goes one
// entry, two round trips, at a time, so U is the one of 9, 8 and 5 with the fewest trips: 9 for
// 27-point rows (128^3 mixed CG's inner solves: 8 34.9 ms, 9 31.8 ms, 14 44.3, 27 37.0), 5 for
// the tets' 15 entries (tet cube 40 mixed CG: 8 3.25 ms, 5 2.96 ms), 8 for 8, 16, 24 and 32.  For
// rows with offsets of their own the choice is by divisibility alone, which is as good there
// and leaves the loops cheaper.  40 CG iterations in FP32 on 10^6 rows, U = 9 or 5 only and now:
// rows that share their offsets, 7 entries 2.32 and 2.07 ms, 8 2.00 and 1.60, 15 2.85 and 2.70, 16
// 2.70 and 2.36, 24 3.21 and 2.91; own offsets, 8 1.92 and 1.71, 16 2.45 and 2.38, 24 3.31 and 3.06.
template <typename VT, int LPR, bool OFFS, bool TWO, typename F>
__device__ __forceinline__ void spmv_phase(const KArgs<VT> &a, const VT *x0, const VT *x1, F &&epi) {
  const int lane = threadIdx.x & 31;
  const int gw = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int nw = (int)(((long long)gridDim.x * blockDim.x) >> 5);
  // the values of the slice this warp takes next are prefetched into L2 (one bulk request)
  // while the current one is summed; the next slice's position is loaded a slice ahead so
  // the request never waits for it
  int nw_w = 0, nw_p = 0;
  if (gw < a.nslices) {
    nw_w = __ldg(a.sell_w + gw);
    nw_p = __ldg(a.sell_ptr + gw);
  }
  for (int s = gw; s < a.nslices; s += nw) {
    const int r = (s << 5) + lane;
    const int w = nw_w;
    const int base = nw_p + lane;
    const int s2 = s + nw;
    if (s2 < a.nslices) {
      nw_w = __ldg(a.sell_w + s2);
      nw_p = __ldg(a.sell_ptr + s2);
    }
    VT s0 = 0, s1 = 0;
    if (OFFS && a.scolsc) {
      const int cp = __ldg(a.sell_cptr + s);
      if (cp < 0) {  // one offset list for the whole slice
        // lane k holds offset k of each chunk of 32 (one coalesced load per chunk) and the
        // warp broadcasts it with a shuffle, so no gather waits on an offset load
        const int16_t *co = a.scolsc + (-cp - 1);
        for (int k0 = 0; k0 < w; k0 += 32) {
          const int kn = min(32, w - k0);
          const int offl = lane < kn ? (int)__ldg(co + k0 + lane) : 0;
          auto shared_entry = [&](int k) {
            const VT v = ld_stream(a.svals + base + ((k0 + k) << 5));
            const int c = r + __shfl_sync(0xffffffffu, offl, k);
            s0 = row_madd(s0, v, ld_l2(x0 + c));
            if (TWO) s1 = row_madd(s1, v, ld_l2(x1 + c));
          };
          const int t9 = kn / 9 + kn % 9, t8 = kn / 8 + kn % 8, t5 = kn / 5 + kn % 5;
          if (t9 <= t8 && t9 <= t5) {
#pragma unroll 9
            for (int k = 0; k < kn; ++k) shared_entry(k);
          } else if (t8 <= t5) {
#pragma unroll 8
            for (int k = 0; k < kn; ++k) shared_entry(k);
          } else {
#pragma unroll 5
            for (int k = 0; k < kn; ++k) shared_entry(k);
          }
        }
      } else {
        const int16_t *co = a.scolsc + cp + lane;
        auto own_entry = [&](int k) {
          const VT v = ld_stream(a.svals + base + (k << 5));
          const int c = r + (int)ld_stream(co + (k << 5));
          s0 = row_madd(s0, v, ld_l2(x0 + c));
          if (TWO) s1 = row_madd(s1, v, ld_l2(x1 + c));
        };
        if (w % 9 && w % 8) {
#pragma unroll 5
          for (int k = 0; k < w; ++k) own_entry(k);
        } else if (w % 9) {
#pragma unroll 8
          for (int k = 0; k < w; ++k) own_entry(k);
        } else {
#pragma unroll 9
          for (int k = 0; k < w; ++k) own_entry(k);
        }
      }
    } else {
#pragma unroll 8
      for (int k = 0; k < w; ++k) {
        const int e = base + (k << 5);
        const VT v = ld_stream(a.svals + e);
        const int c = OFFS ? r + (int)ld_stream(a.scols16 + e) : ld_stream(a.scols + e);
        s0 = row_madd(s0, v, ld_l2(x0 + c));
        if (TWO) s1 = row_madd(s1, v, ld_l2(x1 + c));
      }
    }
    if (lane == 0 && s2 < a.nslices && nw_w > 0)
      prefetch_l2_bulk(a.svals + nw_p, (unsigned)(32 * nw_w * (int)sizeof(VT)));
    if (r < a.n) epi(r, s0, s1);
  }
}

// -------------------------------------------------------------------------------------
// Sync-free triangular solves.  Rows are taken in a dependency order (lower_order /
// upper_order: ascending dependency level); slot s is handled by sub-warp s mod nsub in
// increasing s, so every dependency of a row sits in an earlier slot of a running sub-warp.
// Each produced value is published as itself; consumers poll (bounded) until the entry no
// longer holds the sentinel.
//
// lower: y_i = rhs_i - sum_{j<i} L_ij y_j            (CRS_LUSolve forward, CRSMatrix.src:3346-3352)
// upper: z_i = u_ii^-1 (y_i - sum_{j>i} U_ij z_j)     (backward, :3355-3362)
//
// Warp-collective bounded wait: every lane re-polls all of its unproduced entries (c[u] >= 0
// and x[u] still the sentinel) in one round, all loads in flight together, until no lane of
// the warp has one left.  No lane spins alone, so a warp costs one L2 round trip per round
// however its entries are spread over its lanes.  On expiry (or another block's error) the
// entries keep the sentinel and the error flag is set.  Called by all 32 lanes.
template <typename VT, int E>
__device__ __forceinline__ void warp_wait_all(VT (&xv)[E], const int (&c)[E], const VT *x, int *err) {
  bool pend = false;
#pragma unroll
  for (int u = 0; u < E; ++u) pend |= c[u] >= 0 && Sentinel<VT>::is(xv[u]);
  if (!__any_sync(0xffffffffu, pend)) return;
  const unsigned long long t0 = egpu_globaltimer();
  for (unsigned int spin = 1;; ++spin) {
    pend = false;
#pragma unroll
    for (int u = 0; u < E; ++u)
      if (c[u] >= 0 && Sentinel<VT>::is(xv[u])) xv[u] = Sentinel<VT>::peek(x + c[u]);
#pragma unroll
    for (int u = 0; u < E; ++u) pend |= c[u] >= 0 && Sentinel<VT>::is(xv[u]);
    if (!__any_sync(0xffffffffu, pend)) return;
    if ((spin & 31u) == 0) {
      int stop = 0;
      if ((threadIdx.x & 31) == 0)
        stop = egpu_globaltimer() - t0 > egpu_wait_limit(err) ? 1 : (egpu_error(err) ? 2 : 0);
      stop = __shfl_sync(0xffffffffu, stop, 0);
      if (stop) {
        if (stop == 1 && (threadIdx.x & 31) == 0) egpu_record(err, (int)EGPU_ERR_TIMEOUT);
        return;
      }
    }
  }
}

// One slot's packed entries held by a warp: lane t has entries t and t+32 (rows with more
// than 64 strictly-lower / upper entries finish the rest with a plain loop).
template <typename VT>
struct TriRow {
  int row, beg, end;
  VT v0, v1;
  int c0, c1;
};

// Self-check of the packed layout: a row or column outside [0, n) is recorded in err (as
// EGPU_ERR_ARG) and the access is skipped.
template <typename VT>
__device__ __forceinline__ void tri_fetch(TriRow<VT> &t, int s, const int *order, const int *ptr, const int *cols,
                                          const VT *vals, int lane, int n, int *err) {
  t.row = __ldg(order + s);
  t.beg = __ldg(ptr + s);
  t.end = __ldg(ptr + s + 1);
  t.c0 = t.c1 = -1;
  t.v0 = t.v1 = 0;
  if (t.row < 0 || t.row >= n || t.end < t.beg) {
    if (lane == 0) egpu_record(err, (int)EGPU_ERR_ARG);
    t.row = -1;
    t.end = t.beg;
    return;
  }
  if (t.beg + lane < t.end) {
    t.v0 = __ldg(vals + t.beg + lane);
    t.c0 = __ldg(cols + t.beg + lane);
  }
  if (t.beg + 32 + lane < t.end) {
    t.v1 = __ldg(vals + t.beg + 32 + lane);
    t.c1 = __ldg(cols + t.beg + 32 + lane);
  }
  if (t.c0 >= n || t.c1 >= n) {
    egpu_record(err, (int)EGPU_ERR_ARG);
    if (t.c0 >= n) t.c0 = -1;
    if (t.c1 >= n) t.c1 = -1;
  }
}

// sum over the slot's entries of v * x[col], waiting (bounded) for every x[col] to be produced
template <typename VT>
__device__ __forceinline__ VT tri_dot(const TriRow<VT> &t, const VT *x, const int *cols, const VT *vals, int lane,
                                      int *err) {
  // both loads in flight before either is waited on; the warp polls together
  VT acc = 0;
  const int c[2] = {t.c0, t.c1};
  VT xv[2];
  xv[0] = t.c0 >= 0 ? Sentinel<VT>::peek(x + t.c0) : (VT)0;
  xv[1] = t.c1 >= 0 ? Sentinel<VT>::peek(x + t.c1) : (VT)0;
  warp_wait_all<VT, 2>(xv, c, x, err);
  if (t.c0 >= 0) acc += t.v0 * xv[0];
  if (t.c1 >= 0) acc += t.v1 * xv[1];
  for (int j = t.beg + 64 + lane; j < t.end; j += 32) {
    const int c = __ldg(cols + j);
    if (c >= 0) acc += __ldg(vals + j) * Sentinel<VT>::wait(x + c, err);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  return acc;
}

// Node-block variant (tri_bs = bs > 1).  When the matrix is made of dense diagonal blocks of
// bs consecutive rows (the DOFs of one node, CRS_CreateMatrix with DOFs > 1), the rows of a
// block form a dependency chain, so a row-per-slot schedule has bs times the levels of the
// node graph.  Here one warp owns a whole block: slots s*bs .. s*bs+bs-1 of the orders are
// its rows (lower: ascending, upper: descending), and each row's packed entries end (lower)
// or start (upper) with its k in-block entries.  The warp sums the out-of-block entries of
// all bs rows at once (all loads in flight, polled together), then resolves the in-block
// chain in registers:
//   lower  y_k = (rhs_k - sum_ext L y) - sum_{j<k} L_kj y_j
//   upper  z_k = u_kk^-1 ((y_k - sum_ext U z) - sum_{j>k} U_kj z_j)
// The blocks are waited on and published exactly like single rows.
constexpr int TRI_BS_MAX = 4;
constexpr int TRI_BS_E = 4;  // entries per lane loaded ahead (32 * 4 per block)

template <typename VT>
__device__ __forceinline__ void blk_add(VT (&acc)[TRI_BS_MAX], int k, VT v) {
#pragma unroll
  for (int q = 0; q < TRI_BS_MAX; ++q)
    if (q == k) acc[q] += v;
}

// p[q] by a runtime q, without indexing the array (it stays in registers); p[q] = p[bs]
// for q >= bs
__device__ __forceinline__ int blk_at(const int (&p)[TRI_BS_MAX + 1], int q) {
  int r = p[0];
#pragma unroll
  for (int t = 1; t <= TRI_BS_MAX; ++t)
    if (q == t) r = p[t];
  return r;
}

// slot k of entry e, and whether e is an out-of-block entry of the block (slot k's k
// in-block entries are the last (lower) or first (upper) of its range)
template <bool LOWER>
__device__ __forceinline__ bool blk_ext(const int (&p)[TRI_BS_MAX + 1], int bs, int e, int &k) {
  k = 0;
#pragma unroll
  for (int q = 1; q < TRI_BS_MAX; ++q) k += (q < bs && e >= p[q]) ? 1 : 0;
  return e < p[TRI_BS_MAX] && (LOWER ? e < blk_at(p, k + 1) - k : e >= blk_at(p, k) + k);
}

// out-of-block sum of each of the block's rows; p[0..bs] are its packed row bounds
template <typename VT, bool LOWER>
__device__ __forceinline__ void blk_dot(VT (&acc)[TRI_BS_MAX], const int (&p)[TRI_BS_MAX + 1], int bs, const VT *x,
                                        const int *cols, const VT *vals, int lane, int n, int *err) {
#pragma unroll
  for (int q = 0; q < TRI_BS_MAX; ++q) acc[q] = 0;
  int c[TRI_BS_E];
#pragma unroll
  for (int u = 0; u < TRI_BS_E; ++u) {
    const int e = p[0] + lane + 32 * u;
    int k;
    c[u] = blk_ext<LOWER>(p, bs, e, k) ? __ldg(cols + e) : -1;
    if (c[u] >= n) {
      egpu_record(err, (int)EGPU_ERR_ARG);
      c[u] = -1;
    }
  }
  VT xv[TRI_BS_E], v[TRI_BS_E];
#pragma unroll
  for (int u = 0; u < TRI_BS_E; ++u) {
    xv[u] = c[u] >= 0 ? Sentinel<VT>::peek(x + c[u]) : (VT)0;
    v[u] = c[u] >= 0 ? __ldg(vals + p[0] + lane + 32 * u) : (VT)0;
  }
  warp_wait_all<VT, TRI_BS_E>(xv, c, x, err);
#pragma unroll
  for (int u = 0; u < TRI_BS_E; ++u) {
    if (c[u] < 0) continue;
    int k;
    blk_ext<LOWER>(p, bs, p[0] + lane + 32 * u, k);
    blk_add(acc, k, v[u] * xv[u]);
  }
  for (int e = p[0] + lane + 32 * TRI_BS_E; e < p[TRI_BS_MAX]; e += 32) {
    int k;
    if (!blk_ext<LOWER>(p, bs, e, k)) continue;
    const int cc = __ldg(cols + e);
    if (cc < 0 || cc >= n) {
      egpu_record(err, (int)EGPU_ERR_ARG);
      continue;
    }
    blk_add(acc, k, __ldg(vals + e) * Sentinel<VT>::wait(x + cc, err));
  }
#pragma unroll
  for (int q = 0; q < TRI_BS_MAX; ++q)
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], off);
}

// the block's first row and packed row bounds; false (error recorded) if out of range
__device__ __forceinline__ bool blk_fetch(int q0, int bs, const int *order, const int *ptr, int n, int lower,
                                          int &r0, int (&p)[TRI_BS_MAX + 1], int *err) {
  const int r = __ldg(order + q0);
  r0 = lower ? r : r - (bs - 1);
#pragma unroll
  for (int q = 0; q <= TRI_BS_MAX; ++q) p[q] = __ldg(ptr + q0 + (q < bs ? q : bs));
  bool ok = r0 >= 0 && r0 + bs <= n;
#pragma unroll
  for (int q = 0; q < TRI_BS_MAX; ++q)
    if (q < bs) ok = ok && p[q + 1] - p[q] >= q;
  if (!ok && (threadIdx.x & 31) == 0) egpu_record(err, (int)EGPU_ERR_ARG);
  return ok;
}

template <typename VT, typename RHS>
__device__ __forceinline__ void lower_solve_blk(const KArgs<VT> &a, VT *y, RHS &rhs) {
  const int lane = threadIdx.x & 31;
  int gsub, nsub;
  if (!tri_participant<32>(a.tri_per_block, gsub, nsub)) return;
  const int bs = a.tri_bs, nblk = a.n / bs;
  for (int sb = gsub; sb < nblk; sb += nsub) {
    int r0, p[TRI_BS_MAX + 1];
    if (!blk_fetch(sb * bs, bs, a.lower_order, a.lo_ptr, a.n, 1, r0, p, a.err)) continue;
    // lane k < bs: right-hand side of row k; lane t < bs(bs-1)/2: in-block coefficient
    // L_kj with t = k(k-1)/2 + j (the j-th of row k's last k entries)
    VT rl = 0, cl = 0;
    if (lane < bs) rl = rhs(r0 + lane);
    if (lane < bs * (bs - 1) / 2) {
      int k = 1;
      while (k * (k + 1) / 2 <= lane) ++k;
      const int j = lane - k * (k - 1) / 2;
      cl = __ldg(a.lo_vals + blk_at(p, k + 1) - k + j);
    }
    VT acc[TRI_BS_MAX];
    blk_dot<VT, true>(acc, p, bs, y, a.lo_cols, a.lo_vals, lane, a.n, a.err);
    VT yk[TRI_BS_MAX], mine = 0;
#pragma unroll
    for (int k = 0; k < TRI_BS_MAX; ++k) {
      if (k >= bs) break;
      VT t = __shfl_sync(0xffffffffu, rl, k) - acc[k];
#pragma unroll
      for (int j = 0; j < k; ++j) t -= __shfl_sync(0xffffffffu, cl, k * (k - 1) / 2 + j) * yk[j];
      yk[k] = t;
      if (lane == k) mine = t;
    }
    if (lane < bs) Sentinel<VT>::publish(y + r0 + lane, mine);
  }
}

template <typename VT, typename OUT>
__device__ __forceinline__ void upper_solve_blk(const KArgs<VT> &a, const VT *y, VT *z, OUT &out) {
  const int lane = threadIdx.x & 31;
  int gsub, nsub;
  if (!tri_participant<32>(a.tri_per_block, gsub, nsub)) return;
  const int bs = a.tri_bs, nblk = a.n / bs;
  for (int sb = gsub; sb < nblk; sb += nsub) {
    const int q0 = sb * bs;
    int r0, p[TRI_BS_MAX + 1];
    if (!blk_fetch(q0, bs, a.upper_order, a.up_ptr, a.n, 0, r0, p, a.err)) continue;
    // slot k of the block is row r0 + bs - 1 - k; its first k packed entries are the
    // in-block ones (rows of slots k-1 .. 0).  Lane t < bs(bs-1)/2: U for slot k, entry j.
    VT dl = 0, cl = 0;
    if (lane < bs) dl = __ldg(a.up_dinv + q0 + lane);
    if (lane < bs * (bs - 1) / 2) {
      int k = 1;
      while (k * (k + 1) / 2 <= lane) ++k;
      const int j = lane - k * (k - 1) / 2;
      cl = __ldg(a.up_vals + blk_at(p, k) + j);
    }
    VT acc[TRI_BS_MAX];
    blk_dot<VT, false>(acc, p, bs, z, a.up_cols, a.up_vals, lane, a.n, a.err);
    VT yl = 0;
    if (lane < bs) yl = Sentinel<VT>::wait(y + r0 + bs - 1 - lane, a.err);
    VT zk[TRI_BS_MAX], mine = 0;
#pragma unroll
    for (int k = 0; k < TRI_BS_MAX; ++k) {
      if (k >= bs) break;
      VT t = __shfl_sync(0xffffffffu, yl, k) - acc[k];
      // entry j of slot k is column r0 + bs - k + j, i.e. slot k - 1 - j
#pragma unroll
      for (int j = 0; j < k; ++j) t -= __shfl_sync(0xffffffffu, cl, k * (k - 1) / 2 + j) * zk[k - 1 - j];
      zk[k] = __shfl_sync(0xffffffffu, dl, k) * t;
      if (lane == k) mine = zk[k];
    }
    if (lane < bs) {
      Sentinel<VT>::publish(z + r0 + bs - 1 - lane, mine);
      out(r0 + bs - 1 - lane, mine);
    }
  }
}

// -------------------------------------------------------------------------------------
// Row-range triangular solves (plan: egpu_tri_range.h).
//
// What bounds a solve is the chain of dependency levels.  Spread over all SMs, as above, every
// level costs a store, an L2 round trip, a poll and a warp's sum (0.9 us; 1.7 us for a node
// block).  Here a block owns a contiguous range of rows, whose values it keeps in shared memory
// and solves level by level, one block barrier a level: G lanes a row, K entries a lane, all of
// a level's rows at once, the entries staged by one bulk copy a level.  Every value is published
// to global memory, and the ones another range's rows read are fetched from L2 into its shared
// memory by separate warps, off the chain of levels.
// (A warp per row polling shared memory was slower than no ranges at all: the polls of the
// waiting warps take the issue slots and the shared-memory pipe from the warp on the chain.)
//
// Node blocks: the packed entries are premultiplied by the inverse of the block's own
// triangle (k_range_pack), as are the right-hand sides, so the rows of a node depend on other
// nodes only and the levels are those of the node graph.
//
// Shared memory: the level stages and their mbarriers, own values (rg_rows), external values
// (rg_ext), a zero cell, right-hand sides (rg_rows).
//
// barrier among the first nt threads of the block (named barrier 1; nt a multiple of 32)
__device__ __forceinline__ void cta_bar(int nt) { asm volatile("bar.sync 1, %0;" ::"r"(nt) : "memory"); }

// mbarriers of the stages (copied; read), then the number of levels staged so far in this launch,
// then a word set when a wait for a stage ran out
constexpr int RANGE_COUNT_AT = 16 * plan::RANGE_STAGES;
constexpr int RANGE_BROKEN_AT = RANGE_COUNT_AT + 4;
constexpr int RANGE_FETCH = 8;   // warps fetching external values
constexpr int RANGE_AHEAD = 16;  // levels prefetched into L2
constexpr int RANGE_HEAD = 16 * ((RANGE_BROKEN_AT + 4 + 15) / 16);
// stage: bytes of the largest level record
template <typename VT>
__host__ __device__ constexpr size_t range_smem_bytes(int rows, int ext, int stage) {
  return RANGE_HEAD + (size_t)plan::RANGE_STAGES * stage + sizeof(VT) * (size_t)(2 * rows + ext + 1);
}

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// one bulk copy of `bytes` (a multiple of 16, both addresses 16-byte aligned), counted by bar
__device__ __forceinline__ void bulk_load(unsigned dst, const void *src, unsigned bytes, unsigned bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

// every 64th round of a wait: true when it has to end (limit passed, or an error recorded)
__device__ __forceinline__ bool range_wait_over(unsigned int spin, unsigned long long &t0, int *err) {
  if (spin & 63u) return false;
  if (egpu_error(err)) return true;
  const unsigned long long t = egpu_globaltimer();
  if (t0 == 0) t0 = t;
  if (t - t0 > egpu_wait_limit(err)) {
    egpu_record(err, (int)EGPU_ERR_TIMEOUT);
    return true;
  }
  return false;
}

// does a value loaded from a cell hold the sentinel (its high word marks it: a NaN that arithmetic
// never produces)
__device__ __forceinline__ bool range_unset(double v) { return __double2hiint(v) == (int)(EGPU_SENTINEL64 >> 32); }
__device__ __forceinline__ bool range_unset(float v) { return __float_as_uint(v) == EGPU_SENTINEL32; }

template <typename VT>
__device__ __forceinline__ VT range_lds(unsigned a) {
  VT v;
  if constexpr (sizeof(VT) == 8)
    asm volatile("ld.volatile.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
  else
    asm volatile("ld.volatile.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}
template <typename VT>
__device__ __forceinline__ void range_sts(unsigned a, VT v) {
  if constexpr (sizeof(VT) == 8)
    asm volatile("st.volatile.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
  else
    asm volatile("st.volatile.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}

// the scalars of a solve: shared-memory addresses (values, right-hand sides, stages), published
// values, lanes a row (log2), threads that solve rows
template <typename VT>
struct RangeRun {
  unsigned sx, srhs, stage, bar;
  VT *x;
  int *err;
  volatile int *broken;  // shared memory: a wait for a stage ran out in this launch
  int rows, stage_bytes, lg, nt;
  unsigned first;  // levels staged before this triangle (stage and parity go on)
};

// named barriers 1 and 2 (nt a multiple of 32; the calling warp converged)
__device__ __forceinline__ void range_sync(int id, int nt) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nt) : "memory"); }
__device__ __forceinline__ void range_arrive(int id, int nt) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(nt) : "memory"); }

// One triangle of this block's range (not inlined: the Krylov kernels keep their registers, and
// this loop its own).  Two sets of nt threads solve the levels in turn: while one set sums level
// m, the other reads the entries of level m + 1 from its stage into registers, so between two
// levels there is only a barrier, the loads of the values, the sum and a store (about 1,000
// cycles a level with one set, which read its next entries in between).  The barrier that starts
// level m: its set waits, the other arrives when level m - 1 is stored.
// The next warp stages level records, RANGE_STAGES ahead; the rest fetch external values.
//
// An error (another block's, or an external value that never comes) ends the waits for values
// only.  The waits for stages go on until the copy is there, so the sets never run ahead of the
// copies: a set more than RANGE_STAGES levels ahead would take the barrier's other phase, which
// has the same parity, for its own, and read a record while it is overwritten.  A wait for a
// stage that does run out ends every read of stages by that thread, and the block solves no
// further triangle in this launch (R.broken): its barriers' phases no longer match the levels.
// All copies have landed when this returns.
// Returns the levels staged.
template <typename VT, int K>
__device__ __noinline__ int range_triangle(const RangeTri &T, const RangeRun<VT> R) {
  constexpr int S = plan::RANGE_STAGES;
  const int b = blockIdx.x;
  const int l0 = __ldg(T.lev_ptr + b), nl = __ldg(T.lev_ptr + b + 1) - l0;
  const int nbar = 2 * R.nt;
  if ((int)threadIdx.x < 2 * R.nt) {
    const int set = (int)threadIdx.x >= R.nt ? 1 : 0, tid = (int)threadIdx.x - set * R.nt;
    const int t = tid >> R.lg, G = 1 << R.lg;
    VT v[K], r = 0;
    unsigned xa[K];  // addresses of the entries' values
    int row = -1;
    unsigned dst = 0;
    bool lost = false;  // a stage did not arrive in time: none is read any more
    // the entries of level m, from its stage into registers
    auto load = [&](int m) {
      const unsigned q = R.first + m, st = q % S, bar = R.bar + 8 * st, ph = (q / S) & 1u;
      row = -1;
      bool here = !lost && mbar_try(bar, ph);
      if (!here && !lost) {
        const unsigned long long t0 = egpu_globaltimer(), lim = egpu_wait_limit(R.err);
        while (!(here = mbar_try(bar, ph)))
          if (egpu_globaltimer() - t0 > lim) {
            egpu_record(R.err, (int)EGPU_ERR_TIMEOUT);
            *R.broken = 1;
            lost = true;
            break;
          }
      }
      const unsigned rec = R.stage + st * (unsigned)R.stage_bytes;
      int s0 = 0, w = 0;
      if (here) asm volatile("ld.shared.v2.s32 {%0, %1}, [%2];" : "=r"(s0), "=r"(w) : "r"(rec));
      if (t < w) {
        const unsigned wg = (unsigned)w << R.lg;
        const unsigned ia = rec + 16 + ((4u * w + 15) & ~15u);
        const unsigned va = ia + ((2u * K * wg + 15) & ~15u);
        asm volatile("ld.shared.s32 %0, [%1];" : "=r"(row) : "r"(rec + 16 + 4 * t));
#pragma unroll
        for (int k = 0; k < K; ++k) asm volatile("ld.shared.u16 %0, [%1];" : "=r"(xa[k]) : "r"(ia + 2 * (k * wg + tid)));
#pragma unroll
        for (int k = 0; k < K; ++k) v[k] = range_lds<VT>(va + (unsigned)sizeof(VT) * (k * wg + tid));
        r = 0;  // the row's right-hand side enters on its first lane
        if ((tid & (G - 1)) == 0) r = range_lds<VT>(R.srhs + (unsigned)sizeof(VT) * (s0 + t));
        dst = R.sx + (unsigned)sizeof(VT) * (s0 + t);
#pragma unroll
        for (int k = 0; k < K; ++k) xa[k] = R.sx + (unsigned)sizeof(VT) * xa[k];
      }
      __syncwarp();
      if ((threadIdx.x & 31) == 0) mbar_arrive(bar + 8 * S);  // this warp has read the stage
    };
    if (set < nl) load(set);
    __syncwarp();
    if (set == 1 && nl > 0) range_arrive(1, nbar);
    for (int m = set; m < nl; m += 2) {
      range_sync(1 + (m & 1), nbar);
      VT acc = 0;
      if (row >= 0) {
        VT xv[K];
        bool unset = false;
#pragma unroll
        for (int k = 0; k < K; ++k) xv[k] = range_lds<VT>(xa[k]);
#pragma unroll
        for (int k = 0; k < K; ++k) unset |= range_unset(xv[k]);
        if (unset) {  // external values that have not arrived
          unsigned long long t0 = 0;
          for (unsigned int spin = 1; unset; ++spin) {
            unset = false;
#pragma unroll
            for (int k = 0; k < K; ++k) {
              xv[k] = range_lds<VT>(xa[k]);
              unset |= range_unset(xv[k]);
            }
            if (unset && range_wait_over(spin, t0, R.err)) break;
          }
        }
        // four chains: the FP64 units' latency (about 60 cycles an operation) is the level's time
        VT p[4] = {r, VT(0), VT(0), VT(0)};
#pragma unroll
        for (int k = 0; k < K; ++k) p[k & 3] -= v[k] * xv[k];
        acc = (p[0] + p[1]) + (p[2] + p[3]);
      }
      __syncwarp();
      for (int off = G >> 1; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
      const VT z = acc;
      if (row >= 0 && (tid & (G - 1)) == 0) range_sts<VT>(dst, z);
      __syncwarp();
      if (m + 1 < nl) range_arrive(1 + ((m + 1) & 1), nbar);
      if (row >= 0 && (tid & (G - 1)) == 0) Sentinel<VT>::publish(R.x + row, z);
      if (m + 2 < nl) load(m + 2);
      __syncwarp();
    }
  } else if ((int)threadIdx.x < nbar + 32) {
    // One thread issues.  It reuses a stage when all warps of the set have read it and the copy
    // before is complete (it is, except where a thread gave up its wait for it), so at most
    // RANGE_STAGES are in flight, and it sees those end before it returns: a copy must not land in
    // the shared memory of a block that has exited.  That last wait is bounded by EGPU_WAIT_NS and
    // not by the context's limit, which may be shorter than a copy.
    if ((int)threadIdx.x == nbar) {
      auto wait = [&](unsigned bar, unsigned ph, unsigned long long lim) {
        if (mbar_try(bar, ph)) return true;
        const unsigned long long t0 = egpu_globaltimer();
        while (!mbar_try(bar, ph))
          if (egpu_globaltimer() - t0 > lim) {
            egpu_record(R.err, (int)EGPU_ERR_TIMEOUT);
            *R.broken = 1;
            return false;
          }
        return true;
      };
      const unsigned long long lim = egpu_wait_limit(R.err);
      auto bar = [&](unsigned q) { return R.bar + 8 * (q % S); };
      auto phase = [&](unsigned q) { return (q / S) & 1u; };
      int l = 0;
      long long o0 = __ldg(T.offset + l0);
      for (; l < nl; ++l) {
        const unsigned q = R.first + l;
        const long long o1 = __ldg(T.offset + l0 + l + 1);
        if (q >= S && (!wait(bar(q) + 8 * S, phase(q - S), lim) || !wait(bar(q), phase(q - S), lim))) break;
        bulk_load(R.stage + (q % S) * (unsigned)R.stage_bytes, T.rec + o0, (unsigned)(o1 - o0), bar(q));
        o0 = o1;
        // the level RANGE_AHEAD later into L2: the stages alone cover an L2 hit, not HBM
        if (l + RANGE_AHEAD < nl) {
          const long long p0 = __ldg(T.offset + l0 + l + RANGE_AHEAD), p1 = __ldg(T.offset + l0 + l + RANGE_AHEAD + 1);
          prefetch_l2_bulk(T.rec + p0, (unsigned)(p1 - p0));
        }
      }
      for (int h = max(0, l - S); h < l; ++h) wait(bar(R.first + h), phase(R.first + h), EGPU_WAIT_NS);
    }
  } else {
    // External values, in the order of their first use, 32 a warp at a time, by at most
    // RANGE_FETCH warps (twenty polling warps an SM took a third of the L2's bandwidth)
    const int f = ((int)threadIdx.x - nbar - 32) >> 5, nf = min(RANGE_FETCH, ((int)blockDim.x - nbar - 32) >> 5);
    const int e0 = __ldg(T.ext_ptr + b), e1 = __ldg(T.ext_ptr + b + 1), lane = threadIdx.x & 31;
    int e = e0 + 32 * f + lane;
    int next = f < nf && e < e1 ? __ldg(T.ext + e) : -1;
    for (int q = e0 + 32 * f; f < nf && q < e1; q += 32 * nf, e += 32 * nf) {
      const VT *p = next >= 0 ? R.x + next : nullptr;
      next = e + 32 * nf < e1 ? __ldg(T.ext + e + 32 * nf) : -1;
      bool pend = p != nullptr;
      unsigned long long t0 = 0;
      for (unsigned int spin = 1; __any_sync(0xffffffffu, pend); ++spin) {
        if (pend) {
          const VT v = Sentinel<VT>::peek(p);
          if (!Sentinel<VT>::is(v)) {
            range_sts<VT>(R.sx + (unsigned)sizeof(VT) * (R.rows + e - e0), v);
            pend = false;
          } else if (range_wait_over(spin, t0, R.err)) {
            pend = false;
          }
        }
      }
    }
  }
  return nl;
}

// Once per launch, by all threads of every block, before the first range_ilu: the stages'
// mbarriers (one object for the whole launch: their phases go on from solve to solve)
__device__ __forceinline__ void range_init(int nt) {
  extern __shared__ __align__(16) unsigned char egpu_dsm[];
  if (threadIdx.x < 2 * plan::RANGE_STAGES)
    mbar_init(smem_u32(egpu_dsm) + 8 * threadIdx.x, threadIdx.x < plan::RANGE_STAGES ? 1u : (unsigned)nt / 32);
  if (threadIdx.x == 0) {
    *reinterpret_cast<volatile unsigned *>(egpu_dsm + RANGE_COUNT_AT) = 0u;
    *reinterpret_cast<volatile int *>(egpu_dsm + RANGE_BROKEN_AT) = 0;
  }
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncthreads();
}

// z = (LU)^-1 rhs in the row-range form, called by all threads of every block: rhs(i) once for
// each of the block's own rows, out(i, z_i) for them at the end.  y and z (published values) hold
// the sentinel on entry.
template <typename VT, int TRI, typename RHS, typename OUT>
__device__ __forceinline__ void range_ilu(const KArgs<VT> &a, VT *y, VT *z, RHS &&rhs, OUT &&out) {
  constexpr int K = TRI == TRI_RANGE10 ? 10 : 7;
  extern __shared__ __align__(16) unsigned char egpu_dsm[];
  unsigned char *stage = egpu_dsm + RANGE_HEAD;
  VT *sx = reinterpret_cast<VT *>(stage + (size_t)plan::RANGE_STAGES * a.rg_stage);
  VT *srhs = sx + a.rg_rows + a.rg_ext + 1;
  volatile unsigned *count = reinterpret_cast<volatile unsigned *>(egpu_dsm + RANGE_COUNT_AT);
  const int base = blockIdx.x * a.rg_rows, cnt = min(a.rg_rows, a.n - base), bs = a.tri_bs;
  __syncthreads();  // the buffer's previous use is over
  for (int i = threadIdx.x; i <= a.rg_ext; i += blockDim.x) sx[a.rg_rows + i] = i < a.rg_ext ? Sentinel<VT>::value() : VT(0);
  // right-hand sides times the inverse of the node block's unit lower triangle
  for (int i = threadIdx.x * bs; i < cnt; i += blockDim.x * bs) {
    VT t[TRI_BS_MAX];
#pragma unroll
    for (int k = 0; k < TRI_BS_MAX; ++k)
      if (k < bs) {
        const int r = base + i + k;
        VT v = rhs(r);
        if (k > 0) {
          const int dg = __ldg(a.idiag + r);
#pragma unroll
          for (int j = 0; j < k; ++j) v -= __ldg(a.ilu + dg - k + j) * t[j];
        }
        t[k] = v;
        srhs[__ldg(a.rlo.slot + r)] = v;
      }
  }
  // read before the barrier: all threads of the block take the same way
  volatile int *broken = reinterpret_cast<volatile int *>(egpu_dsm + RANGE_BROKEN_AT);
  const bool lower = __syncthreads_or(*broken) == 0;
  RangeRun<VT> run{smem_u32(sx), smem_u32(srhs), smem_u32(stage), smem_u32(egpu_dsm), y,       a.err,
                   broken,       a.rg_rows,      a.rg_stage,      a.rg_lg,            a.rg_nt, *count};
  if (cnt > 0 && lower) run.first += (unsigned)range_triangle<VT, K>(a.rlo, run);
  __syncthreads();
  for (int i = threadIdx.x; i < a.rg_ext; i += blockDim.x) sx[a.rg_rows + i] = Sentinel<VT>::value();
  // y times the inverse of the node block's upper triangle (inverted diagonal included)
  for (int i = threadIdx.x * bs; i < cnt; i += blockDim.x * bs) {
    VT t[TRI_BS_MAX];
#pragma unroll
    for (int q = 0; q < TRI_BS_MAX; ++q) {
      const int k = TRI_BS_MAX - 1 - q;  // row of the block, last first
      if (k < bs) {
        const int r = base + i + k, dg = __ldg(a.idiag + r);
        VT v = sx[__ldg(a.rlo.slot + r)];
#pragma unroll
        for (int j = k + 1; j < TRI_BS_MAX; ++j)
          if (j < bs) v -= __ldg(a.ilu + dg + j - k) * t[j];
        t[k] = __ldg(a.ilu + dg) * v;
        srhs[__ldg(a.rup.slot + r)] = t[k];
      }
    }
  }
  const bool upper = __syncthreads_or(*broken) == 0;
  run.x = z;
  if (cnt > 0 && upper) run.first += (unsigned)range_triangle<VT, K>(a.rup, run);
  __syncthreads();
  if (threadIdx.x == 0) *count = run.first;
  for (int i = threadIdx.x; i < cnt; i += blockDim.x) out(base + i, sx[__ldg(a.rup.slot + base + i)]);
}

// lower: y_i = rhs_i - sum_{j<i} L_ij y_j (CRS_LUSolve forward, CRSMatrix.src:3346-3352).
// One warp per slot; the next slot's row and entries are fetched while this slot waits.
template <typename VT, int TS, typename RHS>
__device__ __forceinline__ void lower_solve(const KArgs<VT> &a, VT *y, RHS &&rhs) {
  static_assert(TS == 32, "one warp per row");
  if (a.tri_bs > 1) {
    lower_solve_blk<VT>(a, y, rhs);
    return;
  }
  const int lane = threadIdx.x & 31;
  int gsub, nsub;
  if (!tri_participant<TS>(a.tri_per_block, gsub, nsub)) return;
  if (gsub >= a.n) return;
  TriRow<VT> nxt;
  tri_fetch(nxt, gsub, a.lower_order, a.lo_ptr, a.lo_cols, a.lo_vals, lane, a.n, a.err);
  for (int s = gsub; s < a.n; s += nsub) {
    const TriRow<VT> cur = nxt;
    if (s + nsub < a.n) tri_fetch(nxt, s + nsub, a.lower_order, a.lo_ptr, a.lo_cols, a.lo_vals, lane, a.n, a.err);
    // the right-hand side does not depend on the solve: form it before waiting
    VT r = 0;
    if (cur.row < 0) continue;
    if (lane == 0) r = rhs(cur.row);
    const VT acc = tri_dot(cur, y, a.lo_cols, a.lo_vals, lane, a.err);
    if (lane == 0) Sentinel<VT>::publish(y + cur.row, r - acc);
  }
}

// upper: z_i = u_ii^-1 (y_i - sum_{j>i} U_ij z_j) (backward, CRSMatrix.src:3355-3362)
template <typename VT, int TS, typename OUT>
__device__ __forceinline__ void upper_solve(const KArgs<VT> &a, const VT *y, VT *z, OUT &&out) {
  static_assert(TS == 32, "one warp per row");
  if (a.tri_bs > 1) {
    upper_solve_blk<VT>(a, y, z, out);
    return;
  }
  const int lane = threadIdx.x & 31;
  int gsub, nsub;
  if (!tri_participant<TS>(a.tri_per_block, gsub, nsub)) return;
  if (gsub >= a.n) return;
  TriRow<VT> nxt;
  tri_fetch(nxt, gsub, a.upper_order, a.up_ptr, a.up_cols, a.up_vals, lane, a.n, a.err);
  VT dnext = __ldg(a.up_dinv + gsub);
  for (int s = gsub; s < a.n; s += nsub) {
    const TriRow<VT> cur = nxt;
    const VT dinv = dnext;
    if (s + nsub < a.n) {
      tri_fetch(nxt, s + nsub, a.upper_order, a.up_ptr, a.up_cols, a.up_vals, lane, a.n, a.err);
      dnext = __ldg(a.up_dinv + s + nsub);
    }
    if (cur.row < 0) continue;
    const VT acc = tri_dot(cur, z, a.up_cols, a.up_vals, lane, a.err);
    if (lane == 0) {
      const VT yi = Sentinel<VT>::wait(y + cur.row, a.err);
      const VT zi = dinv * (yi - acc);
      Sentinel<VT>::publish(z + cur.row, zi);
      out(cur.row, zi);
    }
  }
}

// -------------------------------------------------------------------------------------
// Level-synchronous triangular solves in one block.
//
// Every dependency of a row lies in an earlier level, and (for the meshes this is used on)
// only a few levels back, so block 0 runs the levels in order with one __syncthreads per
// level and keeps the values of the recent slots in a shared-memory ring (slot s at
// s mod cta_rs; the host sizes the ring so no slot is overwritten while a later row still
// reads it).  A level's ELL block of factor entries, and its rows' right-hand sides,
// inverted diagonals and output positions, are contiguous in global memory; they are
// staged into shared-memory windows with cp.async cta_pd levels ahead, so the copies of
// later levels are in flight while the current one computes.  One thread per row sums its
// entries in CRS order with the reference's operation order:
//   lower  s = b_i;  s = s - L_ij y_j ...;  y_i = s                (CRS_LUSolve :3348-3353)
//   upper  s = y_i;  s = s - U_ij z_j ...;  z_i = u_ii^-1 * s      (:3357-3363)
// so the FP64 solve rounds exactly as CRS_LUSolve does.
__device__ __forceinline__ double row_msub(double s, double a, double x) { return __dsub_rn(s, __dmul_rn(a, x)); }
__device__ __forceinline__ float row_msub(float s, float a, float x) { return fmaf(-a, x, s); }
__device__ __forceinline__ double cta_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float cta_mul(float a, float b) { return a * b; }

template <typename VT>
struct CtaSmem {
  int4 *lv;
  VT *sv;
  uint16_t *si;
  VT *ring, *rr, *rd, *ra;
  int *rm;
};

template <typename VT>
__device__ __forceinline__ CtaSmem<VT> cta_smem(const KArgs<VT> &a, unsigned char *base) {
  CtaSmem<VT> m;
  size_t o = 0;
  const int V = (int)sizeof(VT);
  m.lv = reinterpret_cast<int4 *>(base + o);
  o += (size_t)a.cta_nl * 16;
  m.sv = reinterpret_cast<VT *>(base + o);
  o += cta_align16((size_t)a.cta_sb * V);
  m.si = reinterpret_cast<uint16_t *>(base + o);
  o += cta_align16((size_t)a.cta_sb * 2);
  m.ring = reinterpret_cast<VT *>(base + o);
  o += cta_align16((size_t)(a.cta_rs + 1) * V);
  m.rr = reinterpret_cast<VT *>(base + o);
  o += cta_align16((size_t)a.cta_sr * V);
  m.rd = reinterpret_cast<VT *>(base + o);
  o += cta_align16((size_t)a.cta_sr * V);
  m.ra = reinterpret_cast<VT *>(base + o);
  o += cta_align16((size_t)a.cta_sr * V);
  m.rm = reinterpret_cast<int *>(base + o);
  return m;
}

// Positions of a level in the staging windows and the ring, advanced level by level (the
// same for every thread): sb = ELL offset mod cta_sb, rb = first slot mod cta_sr,
// qb = first slot mod cta_rs.  A level never exceeds a window, so one subtraction wraps.
struct CtaPos {
  int sb, rb, qb;
  __device__ __forceinline__ void advance(int4 lv, int SB, int SR, int RS) {
    sb += (lv.y * lv.z + 7) & ~7;
    if (sb >= SB) sb -= SB;
    rb += lv.y;
    if (rb >= SR) rb -= SR;
    qb += lv.y;
    if (qb >= RS) qb -= RS;
  }
};

__device__ __forceinline__ int cta_wrap(int i, int n) { return i >= n ? i - n : i; }


// issue the copies of level lv (window positions p) into the staging windows (threads
// 0..nt-1)
template <typename VT, bool UPPER>
__device__ __forceinline__ void cta_issue(const KArgs<VT> &a, const CtaTri<VT> &T, const CtaSmem<VT> &m, int4 lv,
                                          CtaPos p, int nt, const VT *rowv, const VT *dinv, const VT *aux) {
  constexpr int PV = 16 / sizeof(VT);
  const int SB = a.cta_sb, SR = a.cta_sr;
  const int ne = (lv.y * lv.z + 7) & ~7;
  for (int c = threadIdx.x; c < ne / PV; c += nt)
    cp_async16(m.sv + cta_wrap(p.sb + c * PV, SB), T.vals + lv.w + c * PV);
  for (int c = threadIdx.x; c < ne / 8; c += nt)
    cp_async16(m.si + cta_wrap(p.sb + c * 8, SB), T.ridx + lv.w + c * 8);
  for (int t = threadIdx.x; t < lv.y; t += nt) {
    const int d = cta_wrap(p.rb + t, SR);
    cp_async_small<sizeof(VT)>(m.rr + d, rowv + lv.x + t);
    cp_async_small<4>(m.rm + d, T.map + lv.x + t);
    if (UPPER) {
      cp_async_small<sizeof(VT)>(m.rd + d, dinv + lv.x + t);
      if (aux) cp_async_small<sizeof(VT)>(m.ra + d, aux + lv.x + t);
    }
  }
}

// One level: the solve's thread t takes the level's rows t, t + nt, ...; a row's entries
// are read four at a time (ring indices, then ring values) and subtracted in CRS order,
// s = s - L_ij y_j as CRS_LUSolve does, so the FP64 result is the reference's to the bit.
template <typename VT, bool UPPER, typename OUT>
__device__ __forceinline__ void cta_level(const KArgs<VT> &a, const CtaSmem<VT> &m, int4 lv, CtaPos p, int nt,
                                          VT *outv, OUT &&out) {
  const int SB = a.cta_sb, SR = a.cta_sr, RS = a.cta_rs;
  const int w = lv.y, nk = lv.z;
  for (int t = threadIdx.x; t < w; t += nt) {
    const int r = cta_wrap(p.rb + t, SR);
    VT s = m.rr[r];
    int e = cta_wrap(p.sb + t, SB);
    int k = 0;
    for (; k + 4 <= nk; k += 4) {
      const int e1 = cta_wrap(e + w, SB), e2 = cta_wrap(e1 + w, SB), e3 = cta_wrap(e2 + w, SB);
      const int i0 = m.si[e], i1 = m.si[e1], i2 = m.si[e2], i3 = m.si[e3];
      const VT v0 = m.sv[e], v1 = m.sv[e1], v2 = m.sv[e2], v3 = m.sv[e3];
      const VT x0 = m.ring[i0], x1 = m.ring[i1], x2 = m.ring[i2], x3 = m.ring[i3];
      s = row_msub(s, v0, x0);
      s = row_msub(s, v1, x1);
      s = row_msub(s, v2, x2);
      s = row_msub(s, v3, x3);
      e = cta_wrap(e3 + w, SB);
    }
    for (; k < nk; ++k) {
      s = row_msub(s, m.sv[e], m.ring[m.si[e]]);
      e = cta_wrap(e + w, SB);
    }
    if (UPPER) s = cta_mul(m.rd[r], s);
    m.ring[cta_wrap(p.qb + t, RS)] = s;
    const int dst = m.rm[r];
    outv[dst] = s;
    if (UPPER) out(dst, s, m.ra[r]);
  }
}

// A whole triangle, run by the block's first a.cta_nt threads (the others go straight to
// the closing __syncthreads).  rowv: right-hand side in this triangle's slot order; lower
// results go to outv[map] (the upper slot order), upper results to outv[row] and
// out(row, z, aux).
template <typename VT, bool UPPER, typename OUT>
__device__ __forceinline__ void cta_tri_solve(const KArgs<VT> &a, const CtaTri<VT> &T, const CtaSmem<VT> &m,
                                              const VT *rowv, const VT *dinv, const VT *aux, VT *outv, OUT &&out) {
  const int PD = a.cta_pd, nlev = T.nlev, nt = a.cta_nt;
  const int SB = a.cta_sb, SR = a.cta_sr, RS = a.cta_rs;
  if (threadIdx.x < nt) {
    // the level table, once per solve
    for (int L = threadIdx.x; L < nlev; L += nt) cp_async16(m.lv + L, T.lev + L);
    cp_async_commit();
    cp_async_wait(0);
    if (threadIdx.x == 0) m.ring[RS] = VT(0);
    cta_bar(nt);
    CtaPos pi{0, 0, 0}, pp{0, 0, 0};  // issue / process positions
    for (int L = 0; L < PD; ++L) {
      if (L < nlev) {
        const int4 lv = m.lv[L];
        cta_issue<VT, UPPER>(a, T, m, lv, pi, nt, rowv, dinv, aux);
        pi.advance(lv, SB, SR, RS);
      }
      cp_async_commit();
    }
    for (int L = 0; L < nlev; ++L) {
      cp_async_wait(PD - 1);
      cta_bar(nt);
      if (L + PD < nlev) {
        const int4 lv = m.lv[L + PD];
        cta_issue<VT, UPPER>(a, T, m, lv, pi, nt, rowv, dinv, aux);
        pi.advance(lv, SB, SR, RS);
      }
      cp_async_commit();
      const int4 lv = m.lv[L];
      cta_level<VT, UPPER>(a, m, lv, pp, nt, outv, out);
      pp.advance(lv, SB, SR, RS);
    }
    cp_async_wait(0);
  }
  __syncthreads();
}

// M^-1 applied by block 0: rhs in lower slot order (slo) -> y in upper slot order (yup)
// -> z (row order) with out(row, z, aux[upper slot]) per row
template <typename VT, typename OUT>
__device__ __forceinline__ void cta_ilu(const KArgs<VT> &a, const VT *slo, VT *yup, const VT *aux, VT *z, OUT &&out) {
  extern __shared__ __align__(16) unsigned char egpu_dsm[];
  const CtaSmem<VT> m = cta_smem(a, egpu_dsm);
  cta_tri_solve<VT, false>(a, a.clo, m, slo, (const VT *)nullptr, (const VT *)nullptr, yup, [](int, VT, VT) {});
  cta_tri_solve<VT, true>(a, a.cup, m, yup, a.up_dinv, aux, z, out);
}

// Jacobi: CRS_DiagPrecondition, CRSMatrix.src:1505-1509
template <typename VT>
__device__ __forceinline__ VT diag_prec(VT v, VT d) {
  return fabs((double)d) > EGPU_AEPS ? v / d : v;
}

template <typename VT>
__device__ __forceinline__ void store_partials(const KArgs<VT> &a, int slot, double v) {
  if (threadIdx.x == 0) a.partials[slot * gridDim.x + blockIdx.x] = v;
}

// -------------------------------------------------------------------------------------
// ILU0 applied by Jacobi sweeps (FP32 inner solves): instead of solving L y = v and U z = y
// exactly (one dependency level after another), iterate
//
//   y_0 = v,            y_{j+1} = v - L_s y_j                  (L unit lower triangular)
//   z_0 = D^-1 y,       z_{j+1} = D^-1 (y - U_s z_j)           (D^-1 the inverted U diagonal)
//
// a fixed number of times (E. Chow and A. Patel, "Fine-grained parallel incomplete LU
// factorization", SIAM J. Sci. Comput. 37 (2015); H. Anzt, E. Chow and J. Dongarra,
// "Iterative sparse triangular solves for preconditioning", Euro-Par 2015).  With a fixed
// count and zero start it is a fixed linear operator, a polynomial in the factors that
// tends to (LU)^-1, so BiCGStab runs with it unchanged; each sweep is one SELL pass over
// half the factor entries, fully parallel, instead of a latency-bound level sequence.  The
// inner solve's result is a correction that the FP64 refinement checks against the true
// residual, so the preconditioner need not be the reference's exact one there.
//
// One sweep over the SELL copy of the factors: lane = row; entries with col < row (LOWER)
// or col > row (UPPER) of the slice's k range; epi(row, sum of factor * zin[col]).
template <bool UPPER, bool OFFS, typename F>
__device__ __forceinline__ void sweep_phase(const KArgs<float> &a, const float *zin, F &&epi) {
  const int lane = threadIdx.x & 31;
  const int gw = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int nw = (int)(((long long)gridDim.x * blockDim.x) >> 5);
  for (int s = gw; s < a.nslices; s += nw) {
    const int r = (s << 5) + lane;
    const int w = __ldg(a.sell_w + s);
    const int2 rg = __ldg(a.swr + s);
    const int k0 = UPPER ? rg.y : 0, k1 = UPPER ? w : rg.x;
    const int base = __ldg(a.sell_ptr + s) + lane;
    float sum = 0.f;
    if (OFFS && a.scolsc) {
      const int cp = __ldg(a.sell_cptr + s);
      if (cp < 0) {  // one offset list for the slice: lane k holds offset k of each chunk of 32
        const int16_t *co = a.scolsc + (-cp - 1);
        for (int c0 = k0; c0 < k1; c0 += 32) {
          const int kn = min(32, k1 - c0);
          const int offl = lane < kn ? (int)__ldg(co + c0 + lane) : 0;
#pragma unroll 4
          for (int k = 0; k < kn; ++k) {
            const int off = __shfl_sync(0xffffffffu, offl, k);
            const float v = ld_stream(a.isvals + base + ((c0 + k) << 5));
            const bool take = UPPER ? off > 0 : off < 0;
            sum = fmaf(take ? v : 0.f, ld_l2(zin + r + off), sum);
          }
        }
      } else {
        const int16_t *co = a.scolsc + cp + lane;
#pragma unroll 4
        for (int k = k0; k < k1; ++k) {
          const int off = (int)ld_stream(co + (k << 5));
          const float v = ld_stream(a.isvals + base + (k << 5));
          const bool take = UPPER ? off > 0 : off < 0;
          sum = fmaf(take ? v : 0.f, ld_l2(zin + r + off), sum);
        }
      }
    } else {
#pragma unroll 4
      for (int k = k0; k < k1; ++k) {
        const int e = base + (k << 5);
        const int c = OFFS ? r + (int)ld_stream(a.scols16 + e) : ld_stream(a.scols + e);
        const float v = ld_stream(a.isvals + e);
        const bool take = UPPER ? c > r : c < r;
        sum = fmaf(take ? v : 0.f, ld_l2(zin + c), sum);
      }
    }
    if (r < a.n) epi(r, sum);
  }
}

// target = M^-1 vin by sweeps (vin complete in every block; ends without a closing barrier,
// which the caller's next grid barrier provides).  ya, yb, za: scratch vectors.  Returns
// false when a grid barrier failed.
template <bool OFFS>
__device__ __forceinline__ bool sweep_apply(const KArgs<float> &a, const float *vin, float *target, float *ya,
                                            float *yb, float *za, unsigned int &epoch) {
  const int ml = a.sweeps_l, mu = a.sweeps_u;
  float *z0 = (mu % 2 == 0) ? target : za;  // the U sweeps alternate so the last lands in target
  const float *yin = vin;
  for (int j = 1; j <= ml; ++j) {
    float *yout = (j & 1) ? ya : yb;
    const bool last = j == ml;
    sweep_phase<false, OFFS>(a, yin, [&](int i, float sum) {
      const float y = vin[i] - sum;
      yout[i] = y;
      if (last) z0[i] = a.idinv[i] * y;
    });
    if (!grid_barrier(a.bar, a.err, epoch)) return false;
    yin = yout;
  }
  const float *y = yin, *zin = z0;
  for (int j = 1; j <= mu; ++j) {
    float *zout = ((mu - j) % 2 == 0) ? target : za;
    sweep_phase<true, OFFS>(a, zin, [&](int i, float sum) { zout[i] = a.idinv[i] * (y[i] - sum); });
    if (j < mu && !grid_barrier(a.bar, a.err, epoch)) return false;
    zin = zout;
  }
  return true;
}

// =====================================================================================
// Every persistent Krylov kernel is instantiated per form of the ILU solves (TriForm, chosen
// per matrix), so that no form pays the registers of another.
//
// CG  (huti_dcgsolv, hutiter/src/huti_cg_D.F90:84-257)
//
// w layout: R Z P Q Y(ILU lower result)
template <typename VT, int LPR, bool OFFS, int TRI>
__global__ void __launch_bounds__(EGPU_KBLOCK, 1) cg_kernel(KArgs<VT> a) {
  if (a.skip && (*a.skip & 2u)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      a.out_i[0] = EGPU_HUTI_CONVERGENCE;
      a.out_i[1] = 0;
      a.out_d[0] = 0.0;
    }
    return;
  }
  __shared__ double sm[32 * 4];
  unsigned int epoch = 0;
  const int n = a.n;
  if constexpr (tri_range(TRI)) range_init(a.rg_nt);

  const int nb = gridDim.x;
  const bool ilu = a.precond == EGPU_PREC_ILU0;
  // FP32 inner solve with M = I (no preconditioner, or Jacobi on a unit diagonal): Z is R
  const bool zr = sizeof(VT) == 4 && !a.true_residual && !ilu && (a.precond == EGPU_PREC_NONE || a.unit_diag);
  VT *X = a.x, *R = a.w, *Z = zr ? a.w : a.w + a.ldw, *P = a.w + 2 * a.ldw, *Q = a.w + 3 * a.ldw,
     *Y = a.w + 4 * a.ldw;
  const VT *B = a.b;
  const bool cta = TRI == TRI_CTA && ilu && a.tri_cta;  // block 0 runs the ILU0 solves level-synchronously
  const VT SENT = Sentinel<VT>::value();
  // level-synchronous mode: R in lower / upper slot order, y in upper slot order
  VT *SLO = a.w + 4 * a.ldw, *YUP = a.w + 5 * a.ldw, *AUX = a.w + 6 * a.ldw;

  // ---- init: R = B - A X  (x0 = 0 in inner mode: R = B)
  {
    double acc[1] = {0.0};
    if (a.true_residual) {
      spmv_phase<VT, LPR, OFFS, false>(a, X, X, [&](int i, VT s, VT) {
        const VT r = B[i] - s;
        R[i] = r;
        if (cta) {
          SLO[a.pos_lo[i]] = r;
          AUX[a.pos_up[i]] = r;
        }
      });
    } else {
      vec_loop<VT>(n, [&](int i, auto w) {
        constexpr int W = decltype(w)::value;
        VT b[W];
        vld<W>(B, i, b);
        vst<W>(R, i, b);
        vfill<W>(X, i, VT(0));
        if (cta) {
#pragma unroll
          for (int k = 0; k < W; ++k) {
            SLO[a.pos_lo[i + k]] = b[k];
            AUX[a.pos_up[i + k]] = b[k];
          }
        }
      });
    }
    vec_loop<VT>(n, [&](int i, auto w) {
      constexpr int W = decltype(w)::value;
      VT b[W];
      vld<W>(B, i, b);
#pragma unroll
      for (int k = 0; k < W; ++k) acc[0] += (double)b[k] * (double)b[k];
      if (ilu && !cta) {
        vfill<W>(Y, i, SENT);
        vfill<W>(Z, i, SENT);
      }
    });
    block_sum<1>(acc, sm);
    store_partials(a, SLOT_BB, acc[0]);
  }
  if (!grid_barrier(a.bar, a.err, epoch)) return;
  const double rhsnorm = sqrt(reduce_partials(a.partials + SLOT_BB * nb, nb, sm));

  // ---- first preconditioning: Z = M^-1 R, partial rho = R.Z
  {
    double acc[1] = {0.0};
    if (cta) {
      if (blockIdx.x == 0)
        cta_ilu(a, SLO, YUP, AUX, Z, [&](int, VT zi, VT ri) { acc[0] += (double)ri * (double)zi; });
    } else if (ilu) {
      if constexpr (tri_range(TRI)) {
        range_ilu<VT, TRI>(a, Y, Z, [&](int i) { return R[i]; }, [&](int i, VT zi) { acc[0] += (double)R[i] * (double)zi; });
      } else {
        lower_solve<VT, LPR>(a, Y, [&](int i) { return R[i]; });
        upper_solve<VT, LPR>(a, Y, Z, [&](int i, VT zi) { acc[0] += (double)R[i] * (double)zi; });
      }
    } else {
      const bool jac = a.precond == EGPU_PREC_DIAGONAL && !zr;
      vec_loop<VT>(n, [&](int i, auto w) {
        constexpr int W = decltype(w)::value;
        VT r[W], d[W], z[W];
        vld<W>(R, i, r);
        if (jac) vld<W>(a.dvals, i, d);
#pragma unroll
        for (int k = 0; k < W; ++k) {
          z[k] = jac ? diag_prec(r[k], d[k]) : r[k];
          acc[0] += (double)r[k] * (double)z[k];
        }
        if (!zr) vst<W>(Z, i, z);
      });
    }
    block_sum<1>(acc, sm);
    store_partials(a, SLOT_RHO, acc[0]);
  }
  if (!grid_barrier(a.bar, a.err, epoch)) return;

  int k = 1, info = 0, iters = 0;
  double rho, oldrho = 1.0, residual = 0.0, rr_prev = 0.0;
  // resumed segment: p_k = z_k + (rho_k / rho_{k-1}) (sigma_new / sigma_old) p_{k-1} in the new
  // scale (rho is quadratic in the residual's scale, P linear)
  const bool resumed = a.resume && !a.true_residual;
  if (resumed) oldrho = a.carry[0] * a.ru_c;
  rho = reduce_partials(a.partials + SLOT_RHO * nb, nb, sm);
  while (true) {
    if (!a.true_residual && k > 1) {
      // inner mode: recursive residual of x_{k-1}
      residual = sqrt(rr_prev) / rhsnorm;
      if (residual <= a.tol) { info = EGPU_HUTI_CONVERGENCE; iters = k - 1; break; }
      if (k > a.maxit) { info = EGPU_HUTI_MAXITER; iters = k - 1; break; }
    }
    // ---- P = Z (first iteration) or Z + beta P
    {
      const VT beta = (VT)(rho / oldrho);
      const bool first = k == 1 && !resumed;
      vec_loop<VT>(n, [&](int i, auto w) {
        constexpr int W = decltype(w)::value;
        VT z[W], p[W];
        vld<W>(Z, i, z);
        if (!first) vld<W>(P, i, p);
#pragma unroll
        for (int q = 0; q < W; ++q) p[q] = first ? z[q] : z[q] + beta * p[q];
        vst<W>(P, i, p);
        if (ilu && !cta) {
          vfill<W>(Z, i, SENT);
          vfill<W>(Y, i, SENT);
        }
      });
    }
    if (!grid_barrier(a.bar, a.err, epoch)) return;
    // ---- Q = A P  (+ A x_{k-1} for the stopping test of iterate k-1)
    {
      double acc[2] = {0.0, 0.0};
      if (a.true_residual && k > 1) {
        spmv_phase<VT, LPR, OFFS, true>(a, P, X, [&](int i, VT s0, VT s1) {
          Q[i] = s0;
          acc[0] += (double)P[i] * (double)s0;
          const double r = (double)s1 - (double)B[i];
          acc[1] += r * r;
        });
      } else {
        spmv_phase<VT, LPR, OFFS, false>(a, P, P, [&](int i, VT s0, VT) {
          Q[i] = s0;
          acc[0] += (double)P[i] * (double)s0;
        });
      }
      block_sum<2>(acc, sm);
      store_partials(a, SLOT_PQ, acc[0]);
      store_partials(a, SLOT_RR, acc[1]);
    }
    if (!grid_barrier(a.bar, a.err, epoch)) return;
    double pqrr[2];
    reduce_partials_n<2>({a.partials + SLOT_PQ * nb, a.partials + SLOT_RR * nb}, nb, sm, pqrr);
    const double pq = pqrr[0];
    if (a.true_residual && k > 1) {
      residual = sqrt(pqrr[1]) / rhsnorm;
      if (residual < a.tol) { info = EGPU_HUTI_CONVERGENCE; iters = k - 1; break; }
      if (k > a.maxit) { info = EGPU_HUTI_MAXITER; iters = k; break; }
    }
    if (rho == 0.0) { info = EGPU_HUTI_CG_RHO; iters = k; break; }
    // ---- X += alpha P; R -= alpha Q; Z = M^-1 R; partial rho_{k+1}
    {
      const double alpha_d = rho / pq;
      const VT alpha = (VT)alpha_d;
      double acc[2] = {0.0, 0.0};
      if (cta) {
        // X, R update and the scatter of R into slot order, then block 0's solve
        vec_loop<VT>(n, [&](int i, auto w) {
          constexpr int W = decltype(w)::value;
          VT x[W], p[W], r[W], q[W];
          vld<W>(X, i, x);
          vld<W>(P, i, p);
          vld<W>(R, i, r);
          vld<W>(Q, i, q);
#pragma unroll
          for (int t = 0; t < W; ++t) {
            x[t] = x[t] + alpha * p[t];
            r[t] = r[t] - alpha * q[t];
            acc[1] += (double)r[t] * (double)r[t];
            SLO[a.pos_lo[i + t]] = r[t];
            AUX[a.pos_up[i + t]] = r[t];
          }
          vst<W>(X, i, x);
          vst<W>(R, i, r);
        });
        double rr[1] = {acc[1]};
        block_sum<1>(rr, sm);
        store_partials(a, SLOT_RR2, rr[0]);
        if (!grid_barrier(a.bar, a.err, epoch)) return;
        double rh[1] = {0.0};
        if (blockIdx.x == 0)
          cta_ilu(a, SLO, YUP, AUX, Z, [&](int, VT zi, VT ri) { rh[0] += (double)ri * (double)zi; });
        block_sum<1>(rh, sm);
        store_partials(a, SLOT_RHO, rh[0]);
      } else {
        if (ilu) {
          if constexpr (tri_range(TRI)) {
            range_ilu<VT, TRI>(a, Y, Z, [&](int i) {
              const VT r = R[i] - alpha * Q[i];
              R[i] = r;
              X[i] = X[i] + alpha * P[i];
              acc[1] += (double)r * (double)r;
              return r;
            }, [&](int i, VT zi) { acc[0] += (double)R[i] * (double)zi; });
          } else {
            lower_solve<VT, LPR>(a, Y, [&](int i) { return R[i] - alpha * Q[i]; });
            upper_solve<VT, LPR>(a, Y, Z, [&](int i, VT zi) {
              const VT r = R[i] - alpha * Q[i];
              R[i] = r;
              X[i] = X[i] + alpha * P[i];
              acc[0] += (double)r * (double)zi;
              acc[1] += (double)r * (double)r;
            });
          }
        } else {
          const bool jac = a.precond == EGPU_PREC_DIAGONAL && !zr;
          vec_loop<VT>(n, [&](int i, auto w) {
            constexpr int W = decltype(w)::value;
            VT x[W], p[W], r[W], q[W], d[W], z[W];
            vld<W>(X, i, x);
            vld<W>(P, i, p);
            vld<W>(R, i, r);
            vld<W>(Q, i, q);
            if (jac) vld<W>(a.dvals, i, d);
#pragma unroll
            for (int t = 0; t < W; ++t) {
              x[t] = x[t] + alpha * p[t];
              r[t] = r[t] - alpha * q[t];
              z[t] = jac ? diag_prec(r[t], d[t]) : r[t];
              acc[0] += (double)r[t] * (double)z[t];
              acc[1] += (double)r[t] * (double)r[t];
            }
            vst<W>(X, i, x);
            vst<W>(R, i, r);
            if (!zr) vst<W>(Z, i, z);
          });
        }
        block_sum<2>(acc, sm);
        store_partials(a, SLOT_RHO, acc[0]);
        store_partials(a, SLOT_RR2, acc[1]);
      }
    }
    if (!grid_barrier(a.bar, a.err, epoch)) return;
    oldrho = rho;
    ++k;
    double rhrr[2];
    reduce_partials_n<2>({a.partials + SLOT_RHO * nb, a.partials + SLOT_RR2 * nb}, nb, sm, rhrr);
    rho = rhrr[0];
    rr_prev = rhrr[1];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.out_i[0] = info;
    a.out_i[1] = iters;
    a.out_d[0] = residual;
    a.out_d[1] = rhsnorm;
    if (a.carry) {  // state for the next segment: P was built with oldrho
      a.carry[0] = oldrho;
      a.carry[3] = (!a.true_residual && info == EGPU_HUTI_CONVERGENCE && k > 1) ? 1.0 : 0.0;
    }
  }
}

// =====================================================================================
// BiCGStab  (huti_dbicgstabsolv, hutiter/src/huti_bicgstab_D.F90:96-284)
//
// w layout: R RTLD P V T S T1V T2V Y1 Y2
template <typename VT, int LPR, bool OFFS, int TRI, bool SW = false>
__global__ void __launch_bounds__(EGPU_KBLOCK, 1) bicgstab_kernel(KArgs<VT> a) {
  if (a.skip && (*a.skip & 2u)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      a.out_i[0] = EGPU_HUTI_CONVERGENCE;
      a.out_i[1] = 0;
      a.out_d[0] = 0.0;
    }
    return;
  }
  __shared__ double sm[32 * 4];
  unsigned int epoch = 0;
  const int n = a.n;
  if constexpr (tri_range(TRI)) range_init(a.rg_nt);

  const int nb = gridDim.x;
  VT *X = a.x;
  VT *R = a.w, *RT = a.w + a.ldw, *P = a.w + 2 * a.ldw, *V = a.w + 3 * a.ldw,
     *T = a.w + 4 * a.ldw, *S = a.w + 5 * a.ldw, *T1 = a.w + 6 * a.ldw, *T2 = a.w + 7 * a.ldw,
     *Y1 = a.w + 8 * a.ldw, *Y2 = a.w + 9 * a.ldw;
  const VT *B = a.b;
  const bool ilu = a.precond == EGPU_PREC_ILU0;
  const bool jac = a.precond == EGPU_PREC_DIAGONAL;
  const bool cta = TRI == TRI_CTA && ilu && a.tri_cta;  // block 0 runs the ILU0 solves level-synchronously
  // FP32 inner solves: ILU0 by Jacobi sweeps (Y1, Y2 and work vector 12 as scratch)
  constexpr bool sw = SW && sizeof(VT) == 4;
  const bool syncfree = ilu && !cta && !sw;
  VT *ZA = a.w + 12 * a.ldw;
  const VT SENT = Sentinel<VT>::value();
  VT *SLO = Y1, *YUP = Y2;           // level-synchronous mode: rhs / y in slot order
  // resumed segment: RTLD, P, V and rho_{k-1}, alpha, omega carry over unchanged (BiCGStab's
  // recurrences are invariant to the residual's scale)
  const bool resumed = a.resume && !a.true_residual;

  // ---- init: R = B - A X; RTLD = R; P = V = 0
  {
    double acc[2] = {0.0, 0.0};
    if (a.true_residual) {
      spmv_phase<VT, LPR, OFFS, false>(a, X, X, [&](int i, VT s, VT) {
        const VT r = B[i] - s;
        R[i] = r;
        RT[i] = r;
        acc[1] += (double)r * (double)r;
      });
    } else {
      vec_loop<VT>(n, [&](int i, auto w) {
        constexpr int W = decltype(w)::value;
        VT b[W];
        vld<W>(B, i, b);
        vfill<W>(X, i, VT(0));
        vst<W>(R, i, b);
        if (!resumed) vst<W>(RT, i, b);
#pragma unroll
        for (int k = 0; k < W; ++k) acc[1] += (double)b[k] * (double)b[k];
      });
    }
    vec_loop<VT>(n, [&](int i, auto w) {
      constexpr int W = decltype(w)::value;
      VT b[W];
      vld<W>(B, i, b);
#pragma unroll
      for (int k = 0; k < W; ++k) acc[0] += (double)b[k] * (double)b[k];
      if (!resumed) {
        vfill<W>(P, i, VT(0));
        vfill<W>(V, i, VT(0));
      }
      if (syncfree) {
        vfill<W>(Y1, i, SENT);
        vfill<W>(Y2, i, SENT);
        vfill<W>(T1, i, SENT);
        vfill<W>(T2, i, SENT);
      }
    });
    double rt[1] = {0.0};
    if (resumed)  // rho_k = RTLD . R with the kept shadow residual
      vec_loop<VT>(n, [&](int i, auto w) {
        constexpr int W = decltype(w)::value;
        VT b[W], t[W];
        vld<W>(B, i, b);
        vld<W>(RT, i, t);
#pragma unroll
        for (int k = 0; k < W; ++k) rt[0] += (double)t[k] * (double)b[k];
      });
    block_sum<2>(acc, sm);
    block_sum<1>(rt, sm);
    store_partials(a, SLOT_BB, acc[0]);
    store_partials(a, SLOT_RHO, resumed ? rt[0] : acc[1]);
    store_partials(a, SLOT_RR2, acc[1]);
  }
  if (!grid_barrier(a.bar, a.err, epoch)) return;
  const double rhsnorm = sqrt(reduce_partials(a.partials + SLOT_BB * nb, nb, sm));

  int k = 1, info = 0, iters = 0;
  double rho, oldrho = 1.0, omega = 1.0, alpha = 0.0, residual = 0.0, r0norm = 0.0;
  if (resumed) {
    oldrho = a.carry[0];
    alpha = a.carry[1];
    omega = a.carry[2];
  }
  if (!a.true_residual) r0norm = sqrt(reduce_partials(a.partials + SLOT_RR2 * nb, nb, sm));
  while (true) {
    double rhrr[2];
    reduce_partials_n<2>({a.partials + SLOT_RHO * nb, a.partials + SLOT_RR2 * nb}, nb, sm, rhrr);
    rho = rhrr[0];
    if (!a.true_residual && k > 1) {
      residual = sqrt(rhrr[1]) / r0norm;
      if (residual <= a.tol) { info = EGPU_HUTI_CONVERGENCE; iters = k - 1; break; }
      if (omega == 0.0) { info = EGPU_HUTI_BICGSTAB_OMEGA; iters = k - 1; break; }
      if (k > a.maxit) { info = EGPU_HUTI_MAXITER; iters = k - 1; break; }
    }
    const bool rho_zero = rho == 0.0;
    // ---- P = R + beta (P - omega V); T1V = M^-1 P
    {
      const VT beta = (VT)((rho * alpha) / (oldrho * omega));
      const VT om = (VT)omega;
      if (sw && ilu) {
        vec_loop<VT>(n, [&](int i, auto w) {
          constexpr int W = decltype(w)::value;
          VT r[W], p[W], v[W];
          vld<W>(R, i, r);
          vld<W>(P, i, p);
          vld<W>(V, i, v);
#pragma unroll
          for (int q = 0; q < W; ++q) p[q] = r[q] + beta * (p[q] - om * v[q]);
          vst<W>(P, i, p);
        });
        if (!grid_barrier(a.bar, a.err, epoch)) return;
        if constexpr (sw) {
          if (!sweep_apply<OFFS>(a, P, T1, Y1, Y2, ZA, epoch)) return;
        }
      } else if (cta) {
        vec_loop<VT>(n, [&](int i, auto w) {
          constexpr int W = decltype(w)::value;
          VT r[W], p[W], v[W];
          vld<W>(R, i, r);
          vld<W>(P, i, p);
          vld<W>(V, i, v);
#pragma unroll
          for (int q = 0; q < W; ++q) {
            p[q] = r[q] + beta * (p[q] - om * v[q]);
            SLO[a.pos_lo[i + q]] = p[q];
          }
          vst<W>(P, i, p);
        });
        if (!grid_barrier(a.bar, a.err, epoch)) return;
        if (blockIdx.x == 0) cta_ilu(a, SLO, YUP, (const VT *)nullptr, T1, [](int, VT, VT) {});
      } else if (ilu) {
        auto rhs = [&](int i) {
          const VT p = R[i] + beta * (P[i] - om * V[i]);
          P[i] = p;
          return p;
        };
        if constexpr (tri_range(TRI)) {
          range_ilu<VT, TRI>(a, Y1, T1, rhs, [](int, VT) {});
        } else {
          lower_solve<VT, LPR>(a, Y1, rhs);
          upper_solve<VT, LPR>(a, Y1, T1, [&](int, VT) {});
        }
      } else {
        vec_loop<VT>(n, [&](int i, auto w) {
          constexpr int W = decltype(w)::value;
          VT r[W], p[W], v[W], d[W], t[W];
          vld<W>(R, i, r);
          vld<W>(P, i, p);
          vld<W>(V, i, v);
          if (jac) vld<W>(a.dvals, i, d);
#pragma unroll
          for (int q = 0; q < W; ++q) {
            p[q] = r[q] + beta * (p[q] - om * v[q]);
            t[q] = jac ? diag_prec(p[q], d[q]) : p[q];
          }
          vst<W>(P, i, p);
          vst<W>(T1, i, t);
        });
      }
    }
    if (!grid_barrier(a.bar, a.err, epoch)) return;
    // ---- V = A T1V (+ A x_{k-1}); partials RTLD.V, ||A x_{k-1} - b||^2
    {
      double acc[2] = {0.0, 0.0};
      if (a.true_residual && k > 1) {
        spmv_phase<VT, LPR, OFFS, true>(a, T1, X, [&](int i, VT s0, VT s1) {
          V[i] = s0;
          acc[0] += (double)RT[i] * (double)s0;
          const double r = (double)s1 - (double)B[i];
          acc[1] += r * r;
        });
      } else {
        spmv_phase<VT, LPR, OFFS, false>(a, T1, T1, [&](int i, VT s0, VT) {
          V[i] = s0;
          acc[0] += (double)RT[i] * (double)s0;
        });
      }
      block_sum<2>(acc, sm);
      store_partials(a, SLOT_PQ, acc[0]);
      store_partials(a, SLOT_RR, acc[1]);
    }
    if (!grid_barrier(a.bar, a.err, epoch)) return;
    double rvrr[2];
    reduce_partials_n<2>({a.partials + SLOT_PQ * nb, a.partials + SLOT_RR * nb}, nb, sm, rvrr);
    const double rv = rvrr[0];
    if (a.true_residual && k > 1) {
      residual = sqrt(rvrr[1]) / rhsnorm;
      if (residual < a.tol) { info = EGPU_HUTI_CONVERGENCE; iters = k - 1; break; }
      if (omega == 0.0) { info = EGPU_HUTI_BICGSTAB_OMEGA; iters = k - 1; break; }
      if (k > a.maxit) { info = EGPU_HUTI_MAXITER; iters = k; break; }
    }
    if (rho_zero) { info = EGPU_HUTI_BICGSTAB_RHO; iters = k; break; }
    alpha = rho / rv;
    // ---- S = R - alpha V; T2V = M^-1 S; partial ||S||^2
    {
      const VT al = (VT)alpha;
      double acc[1] = {0.0};
      if (sw && ilu) {
        vec_loop<VT>(n, [&](int i, auto w) {
          constexpr int W = decltype(w)::value;
          VT r[W], v[W], sv[W];
          vld<W>(R, i, r);
          vld<W>(V, i, v);
#pragma unroll
          for (int q = 0; q < W; ++q) {
            sv[q] = row_msub(r[q], al, v[q]);
            acc[0] += (double)sv[q] * (double)sv[q];
          }
          vst<W>(S, i, sv);
        });
        block_sum<1>(acc, sm);
        store_partials(a, SLOT_SS, acc[0]);
        if (!grid_barrier(a.bar, a.err, epoch)) return;
        if constexpr (sw) {
          if (!sweep_apply<OFFS>(a, S, T2, Y1, Y2, ZA, epoch)) return;
        }
      } else if (cta) {
        vec_loop<VT>(n, [&](int i, auto w) {
          constexpr int W = decltype(w)::value;
          VT r[W], v[W], sv[W];
          vld<W>(R, i, r);
          vld<W>(V, i, v);
#pragma unroll
          for (int q = 0; q < W; ++q) {
            sv[q] = row_msub(r[q], al, v[q]);  // S = R - alpha V, rounded as HUTI
            acc[0] += (double)sv[q] * (double)sv[q];
            SLO[a.pos_lo[i + q]] = sv[q];
          }
          vst<W>(S, i, sv);
        });
        block_sum<1>(acc, sm);
        store_partials(a, SLOT_SS, acc[0]);
        if (!grid_barrier(a.bar, a.err, epoch)) return;
        if (blockIdx.x == 0) cta_ilu(a, SLO, YUP, (const VT *)nullptr, T2, [](int, VT, VT) {});
      } else {
        if (ilu) {
          auto rhs = [&](int i) {
            const VT s = row_msub(R[i], al, V[i]);
            S[i] = s;
            acc[0] += (double)s * (double)s;
            return s;
          };
          if constexpr (tri_range(TRI)) {
            range_ilu<VT, TRI>(a, Y2, T2, rhs, [](int, VT) {});
          } else {
            lower_solve<VT, LPR>(a, Y2, rhs);
            upper_solve<VT, LPR>(a, Y2, T2, [&](int, VT) {});
          }
        } else {
          vec_loop<VT>(n, [&](int i, auto w) {
            constexpr int W = decltype(w)::value;
            VT r[W], v[W], d[W], sv[W], t[W];
            vld<W>(R, i, r);
            vld<W>(V, i, v);
            if (jac) vld<W>(a.dvals, i, d);
#pragma unroll
            for (int q = 0; q < W; ++q) {
              sv[q] = row_msub(r[q], al, v[q]);  // S = R - alpha V, rounded as HUTI
              acc[0] += (double)sv[q] * (double)sv[q];
              t[q] = jac ? diag_prec(sv[q], d[q]) : sv[q];
            }
            vst<W>(S, i, sv);
            vst<W>(T2, i, t);
          });
        }
        block_sum<1>(acc, sm);
        store_partials(a, SLOT_SS, acc[0]);
      }
    }
    if (!grid_barrier(a.bar, a.err, epoch)) return;
    // ---- T = A T2V; partials T.S, T.T
    {
      double acc[2] = {0.0, 0.0};
      spmv_phase<VT, LPR, OFFS, false>(a, T2, T2, [&](int i, VT s0, VT) {
        T[i] = s0;
        acc[0] += (double)s0 * (double)S[i];
        acc[1] += (double)s0 * (double)s0;
      });
      block_sum<2>(acc, sm);
      store_partials(a, SLOT_TS, acc[0]);
      store_partials(a, SLOT_TT, acc[1]);
    }
    if (!grid_barrier(a.bar, a.err, epoch)) return;
    double sts[3];
    reduce_partials_n<3>({a.partials + SLOT_SS * nb, a.partials + SLOT_TS * nb, a.partials + SLOT_TT * nb}, nb, sm, sts);
    const double ss = sts[0], ts = sts[1], tt = sts[2];
    if (sqrt(ss) < EGPU_HUTI_EPSILON) {
      const VT al = (VT)alpha;
      vec_loop<VT>(n, [&](int i, auto w) {
        constexpr int W = decltype(w)::value;
        VT x[W], t[W];
        vld<W>(X, i, x);
        vld<W>(T1, i, t);
#pragma unroll
        for (int q = 0; q < W; ++q) x[q] = x[q] + al * t[q];
        vst<W>(X, i, x);
      });
      residual = sqrt(ss);
      info = EGPU_HUTI_BICGSTAB_SNORM;
      iters = k;
      break;
    }
    omega = ts / tt;
    // ---- X += alpha T1V + omega T2V; R = S - omega T; partial RTLD.R
    {
      const VT al = (VT)alpha, om = (VT)omega;
      double acc[2] = {0.0, 0.0};
      vec_loop<VT>(n, [&](int i, auto w) {
        constexpr int W = decltype(w)::value;
        VT x[W], t1[W], t2[W], sv[W], t[W], rt[W], r[W];
        vld<W>(X, i, x);
        vld<W>(T1, i, t1);
        vld<W>(T2, i, t2);
        vld<W>(S, i, sv);
        vld<W>(T, i, t);
        vld<W>(RT, i, rt);
#pragma unroll
        for (int q = 0; q < W; ++q) {
          x[q] = x[q] + al * t1[q] + om * t2[q];
          r[q] = sv[q] - om * t[q];
          acc[0] += (double)rt[q] * (double)r[q];
          acc[1] += (double)r[q] * (double)r[q];
        }
        vst<W>(X, i, x);
        vst<W>(R, i, r);
        if (syncfree) {
          vfill<W>(T1, i, SENT);
          vfill<W>(T2, i, SENT);
          vfill<W>(Y1, i, SENT);
          vfill<W>(Y2, i, SENT);
        }
      });
      block_sum<2>(acc, sm);
      store_partials(a, SLOT_RHO, acc[0]);
      store_partials(a, SLOT_RR2, acc[1]);
    }
    if (!grid_barrier(a.bar, a.err, epoch)) return;
    oldrho = rho;
    ++k;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.out_i[0] = info;
    a.out_i[1] = iters;
    a.out_d[0] = residual;
    a.out_d[1] = rhsnorm;
    if (a.carry) {  // state for the next segment: P, V were built with oldrho, alpha, omega
      a.carry[0] = oldrho;
      a.carry[1] = alpha;
      a.carry[2] = omega;
      a.carry[3] = (!a.true_residual && info == EGPU_HUTI_CONVERGENCE && k > 1) ? 1.0 : 0.0;
    }
  }
}

// =====================================================================================
// GCR with restart m (IterativeMethods.src:919-1055), FP64.
//
// Search directions T1 = M^-1 r, T2 = A T1; T2 is orthogonalised against the stored
// V_1..V_{j-1} by modified Gram-Schmidt (one dot product and one update pass each, in the
// reference's order), normalised by multiplying with 1/||T2||; x += beta T1, r -= beta T2 with
// beta = T2 . r.  The stopping test is the recursive residual ||r|| / ||b|| < tol; at every
// restart (j = 1, k > 1) r is recomputed as b - A x.
//
// w layout: R T1 T2 Y(ILU lower result) SLO YUP(level-synchronous slot order)
// stored directions: S_i = ext + i * ext_lds, V_i = ext + (m - 1 + i) * ext_lds, i < m - 1
template <int LPR, int TRI>
__global__ void __launch_bounds__(EGPU_KBLOCK, 1) gcr_kernel(KArgs<double> a) {
  using VT = double;
  struct {
    int m;
    double *S, *V;
    long long lds;
  } g{a.ext_m, a.ext, a.ext + (long long)(a.ext_m - 1) * a.ext_lds, a.ext_lds};
  if (a.skip && (*a.skip & 2u)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      a.out_i[0] = EGPU_HUTI_CONVERGENCE;
      a.out_i[1] = 0;
      a.out_d[0] = 0.0;
    }
    return;
  }
  __shared__ double sm[32 * 4];
  unsigned int epoch = 0;
  const int n = a.n, nb = gridDim.x;
  if constexpr (tri_range(TRI)) range_init(a.rg_nt);
  VT *X = a.x, *R = a.w, *T1 = a.w + a.ldw, *T2 = a.w + 2 * a.ldw, *Y = a.w + 3 * a.ldw,
     *SLO = a.w + 4 * a.ldw, *YUP = a.w + 5 * a.ldw;
  const VT *B = a.b;
  const bool ilu = a.precond == EGPU_PREC_ILU0, jac = a.precond == EGPU_PREC_DIAGONAL;
  const bool cta = TRI == TRI_CTA && ilu && a.tri_cta;
  const VT SENT = Sentinel<VT>::value();
  // per row after r changed: prepare the next M^-1 (sentinels, or r in slot order)
  auto prep = [&](int i, VT r) {
    if (cta) {
      SLO[a.pos_lo[i]] = r;
    } else if (ilu) {
      Y[i] = SENT;
      T1[i] = SENT;
    }
  };
  // ---- init: R = B - A X; ||B||, ||R||
  {
    double acc[2] = {0.0, 0.0};
    spmv_phase<VT, LPR, false, false>(a, X, X, [&](int i, VT s, VT) {
      const VT r = B[i] - s;
      R[i] = r;
      prep(i, r);
      acc[0] += (double)B[i] * (double)B[i];
      acc[1] += (double)r * (double)r;
    });
    block_sum<2>(acc, sm);
    store_partials(a, SLOT_BB, acc[0]);
    store_partials(a, SLOT_RR, acc[1]);
  }
  if (!grid_barrier(a.bar, a.err, epoch)) return;
  const double bnorm = sqrt(reduce_partials(a.partials + SLOT_BB * nb, nb, sm));
  double residual = sqrt(reduce_partials(a.partials + SLOT_RR * nb, nb, sm)) / bnorm;
  int info = 0, iters = 0;
  // IterativeMethods.src:959-961: Converged = Residual < MinTolerance; Diverged = Residual >
  // MaxTolerance (Linear System Divergence Tolerance) or NaN
  if (residual < a.tol) info = EGPU_HUTI_CONVERGENCE;
  if (residual != residual || (a.divtol > 0.0 && residual > a.divtol)) info = 3;  // HUTI_DIVERGENCE
  for (int k = 1; info == 0; ++k) {
    if (k > a.maxit) {
      info = EGPU_HUTI_MAXITER;
      break;
    }
    const int j = (k % g.m == 0) ? g.m : k % g.m;
    if (j == 1 && k > 1) {  // restart: the true residual
      spmv_phase<VT, LPR, false, false>(a, X, X, [&](int i, VT s, VT) {
        const VT r = B[i] - s;
        R[i] = r;
        prep(i, r);
      });
      if (!grid_barrier(a.bar, a.err, epoch)) return;
    }
    // ---- T1 = M^-1 R
    if (cta) {
      if (blockIdx.x == 0) cta_ilu(a, SLO, YUP, (const VT *)nullptr, T1, [](int, VT, VT) {});
    } else if (ilu) {
      if constexpr (tri_range(TRI)) {
        range_ilu<VT, TRI>(a, Y, T1, [&](int i) { return R[i]; }, [](int, VT) {});
      } else {
        lower_solve<VT, 32>(a, Y, [&](int i) { return R[i]; });
        upper_solve<VT, 32>(a, Y, T1, [&](int, VT) {});
      }
    } else {
      vec_loop<VT>(n, [&](int i, auto w) {
        constexpr int W = decltype(w)::value;
        VT r[W], d[W], t[W];
        vld<W>(R, i, r);
        if (jac) vld<W>(a.dvals, i, d);
#pragma unroll
        for (int q = 0; q < W; ++q) t[q] = jac ? diag_prec(r[q], d[q]) : r[q];
        vst<W>(T1, i, t);
      });
    }
    if (!grid_barrier(a.bar, a.err, epoch)) return;
    // ---- T2 = A T1, and the first dot of the orthogonalisation (or ||T2||^2 when j == 1)
    {
      double acc[1] = {0.0};
      const VT *V0 = g.V;
      spmv_phase<VT, LPR, false, false>(a, T1, T1, [&](int i, VT s, VT) {
        T2[i] = s;
        acc[0] += j > 1 ? (double)V0[i] * (double)s : (double)s * (double)s;
      });
      block_sum<1>(acc, sm);
      store_partials(a, j > 1 ? SLOT_PQ : SLOT_TT, acc[0]);
    }
    if (!grid_barrier(a.bar, a.err, epoch)) return;
    // ---- modified Gram-Schmidt against V_1..V_{j-1}
    for (int i = 0; i < j - 1; ++i) {
      const int rd = (i & 1) ? SLOT_SS : SLOT_PQ, wr = (i & 1) ? SLOT_PQ : SLOT_SS;
      const double beta = reduce_partials(a.partials + rd * nb, nb, sm);
      const VT *Si = g.S + (long long)i * g.lds, *Vi = g.V + (long long)i * g.lds;
      const VT *Vn = g.V + (long long)(i + 1) * g.lds;
      const bool last = i + 1 == j - 1;
      double acc[1] = {0.0};
      vec_loop<VT>(n, [&](int q0, auto w) {
        constexpr int W = decltype(w)::value;
        VT t1[W], t2[W], s[W], v[W], vn[W];
        vld<W>(T1, q0, t1);
        vld<W>(T2, q0, t2);
        vld<W>(Si, q0, s);
        vld<W>(Vi, q0, v);
        if (!last) vld<W>(Vn, q0, vn);
#pragma unroll
        for (int q = 0; q < W; ++q) {
          t1[q] = t1[q] - beta * s[q];
          t2[q] = t2[q] - beta * v[q];
          acc[0] += last ? (double)t2[q] * (double)t2[q] : (double)vn[q] * (double)t2[q];
        }
        vst<W>(T1, q0, t1);
        vst<W>(T2, q0, t2);
      });
      block_sum<1>(acc, sm);
      store_partials(a, last ? SLOT_TT : wr, acc[0]);
      if (!grid_barrier(a.bar, a.err, epoch)) return;
    }
    // ---- normalise: T1, T2 times 1/||T2||; beta = T2 . R
    {
      const double alpha = sqrt(reduce_partials(a.partials + SLOT_TT * nb, nb, sm));
      const double inv = 1.0 / alpha;
      double acc[1] = {0.0};
      vec_loop<VT>(n, [&](int q0, auto w) {
        constexpr int W = decltype(w)::value;
        VT t1[W], t2[W], r[W];
        vld<W>(T1, q0, t1);
        vld<W>(T2, q0, t2);
        vld<W>(R, q0, r);
#pragma unroll
        for (int q = 0; q < W; ++q) {
          t1[q] = inv * t1[q];
          t2[q] = inv * t2[q];
          acc[0] += (double)t2[q] * (double)r[q];
        }
        vst<W>(T1, q0, t1);
        vst<W>(T2, q0, t2);
      });
      block_sum<1>(acc, sm);
      store_partials(a, SLOT_TS, acc[0]);
    }
    if (!grid_barrier(a.bar, a.err, epoch)) return;
    // ---- x += beta T1; r -= beta T2; store the direction; ||r||
    {
      const double beta = reduce_partials(a.partials + SLOT_TS * nb, nb, sm);
      VT *Sj = g.S + (long long)(j - 1) * g.lds, *Vj = g.V + (long long)(j - 1) * g.lds;
      const bool keep = j != g.m;
      double acc[1] = {0.0};
      for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const VT t1 = T1[i], t2 = T2[i];
        X[i] = X[i] + beta * t1;
        const VT r = R[i] - beta * t2;
        R[i] = r;
        if (keep) {
          Sj[i] = t1;
          Vj[i] = t2;
        }
        acc[0] += (double)r * (double)r;
        prep(i, r);
      }
      block_sum<1>(acc, sm);
      store_partials(a, SLOT_RR, acc[0]);
    }
    if (!grid_barrier(a.bar, a.err, epoch)) return;
    residual = sqrt(reduce_partials(a.partials + SLOT_RR * nb, nb, sm)) / bnorm;
    iters = k;
    if (residual < a.tol) info = EGPU_HUTI_CONVERGENCE;
    else if (residual != residual || (a.divtol > 0.0 && residual > a.divtol)) info = 3;  // :1047-1048
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.out_i[0] = info;
    a.out_i[1] = iters;
    a.out_d[0] = residual;
    a.out_d[1] = bnorm;
  }
}

// =====================================================================================
// BiCGStab(l) (IterativeMethods.src:559-834), FP64: right-preconditioned (the iteration
// runs on A M^-1 and x = M^-1 x~ + xp at the end), l BiCG steps then the convex minimal-
// residual polynomial of degree l, reliable residual / solution updates with delta = 1e-2,
// stopping on the recursive residual.
//
// ext layout (stride ext_lds): r_0..r_l, u_0..u_l, RR(shadow) XT(x~) XP BP T
// w layout: Y(ILU lower result, w[3]) SLO YUP(level-synchronous slot order, w[4], w[5])

// small dense LU with partial pivoting (dgetrf) and solve (dgetrs 'n'), column major
__device__ inline void bl_lu(int m, double *a, int lda, int *piv) {
  for (int k = 0; k < m; ++k) {
    int p = k;
    for (int i = k + 1; i < m; ++i)
      if (fabs(a[i + k * lda]) > fabs(a[p + k * lda])) p = i;
    piv[k] = p;
    if (p != k)
      for (int j = 0; j < m; ++j) {
        const double t = a[k + j * lda];
        a[k + j * lda] = a[p + j * lda];
        a[p + j * lda] = t;
      }
    if (a[k + k * lda] != 0.0)
      for (int i = k + 1; i < m; ++i) a[i + k * lda] = a[i + k * lda] / a[k + k * lda];
    for (int j = k + 1; j < m; ++j)
      for (int i = k + 1; i < m; ++i) a[i + j * lda] = a[i + j * lda] - a[i + k * lda] * a[k + j * lda];
  }
}
__device__ inline void bl_lu_solve(int m, const double *a, int lda, const int *piv, double *b) {
  for (int k = 0; k < m; ++k)
    if (piv[k] != k) {
      const double t = b[k];
      b[k] = b[piv[k]];
      b[piv[k]] = t;
    }
  for (int k = 0; k < m; ++k)
    for (int i = k + 1; i < m; ++i) b[i] = b[i] - a[i + k * lda] * b[k];
  for (int k = m - 1; k >= 0; --k) {
    b[k] = b[k] / a[k + k * lda];
    for (int i = 0; i < k; ++i) b[i] = b[i] - a[i + k * lda] * b[k];
  }
}

constexpr int BL_MAXL = 8;

template <int LPR, int TRI>
__global__ void __launch_bounds__(EGPU_KBLOCK, 1) bicgstabl_kernel(KArgs<double> a) {
  using VT = double;
  if (a.skip && (*a.skip & 2u)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      a.out_i[0] = EGPU_HUTI_CONVERGENCE;
      a.out_i[1] = 0;
      a.out_d[0] = 0.0;
    }
    return;
  }
  __shared__ double sm[32 * 4];
  __shared__ double Zs[(BL_MAXL + 1) * (BL_MAXL + 1)], y0s[BL_MAXL + 1];
  unsigned int epoch = 0;
  const int n = a.n, nb = gridDim.x, l = a.ext_m, L1 = l + 1;
  if constexpr (tri_range(TRI)) range_init(a.rg_nt);
  const long long ld = a.ext_lds;
  auto rv = [&](int j) { return a.ext + (long long)j * ld; };
  auto uv = [&](int j) { return a.ext + (long long)(L1 + j) * ld; };
  VT *RR = a.ext + (long long)(2 * L1) * ld, *XT = RR + ld, *XP = RR + 2 * ld, *BP = RR + 3 * ld, *T = RR + 4 * ld;
  VT *X = a.x, *Y = a.w + 3 * a.ldw, *SLO = a.w + 4 * a.ldw, *YUP = a.w + 5 * a.ldw;
  const VT *B = a.b;
  const bool ilu = a.precond == EGPU_PREC_ILU0, jac = a.precond == EGPU_PREC_DIAGONAL;
  const bool cta = TRI == TRI_CTA && ilu && a.tri_cta;
  const VT SENT = Sentinel<VT>::value();
  double *gram = a.partials + 16 * nb;  // (l+1)(l+2)/2 slots of nb partials
  // dst = M^-1 src (pcondlsubr); ends after a grid barrier
  auto precond = [&](const VT *src, VT *dst) -> bool {
    if (ilu) {
      vec_loop<VT>(n, [&](int i, auto w) {
        constexpr int W = decltype(w)::value;
        if (cta) {
          VT v[W];
          vld<W>(src, i, v);
#pragma unroll
          for (int q = 0; q < W; ++q) SLO[a.pos_lo[i + q]] = v[q];
        } else {
          vfill<W>(Y, i, SENT);
          vfill<W>(dst, i, SENT);
        }
      });
      if (!grid_barrier(a.bar, a.err, epoch)) return false;
      if (cta) {
        if (blockIdx.x == 0) cta_ilu(a, SLO, YUP, (const VT *)nullptr, dst, [](int, VT, VT) {});
      } else {
        if constexpr (tri_range(TRI)) {
          range_ilu<VT, TRI>(a, Y, dst, [&](int i) { return src[i]; }, [](int, VT) {});
        } else {
          lower_solve<VT, 32>(a, Y, [&](int i) { return src[i]; });
          upper_solve<VT, 32>(a, Y, dst, [&](int, VT) {});
        }
      }
    } else {
      vec_loop<VT>(n, [&](int i, auto w) {
        constexpr int W = decltype(w)::value;
        VT v[W], d[W], t[W];
        vld<W>(src, i, v);
        if (jac) vld<W>(a.dvals, i, d);
#pragma unroll
        for (int q = 0; q < W; ++q) t[q] = jac ? diag_prec(v[q], d[q]) : v[q];
        vst<W>(dst, i, t);
      });
    }
    return grid_barrier(a.bar, a.err, epoch);
  };
  // ---- init: r_0 = B - A X; ||B||, ||r_0||; shadow, bp, xp; x~ = 0
  {
    double acc[2] = {0.0, 0.0};
    VT *R0 = rv(0);
    spmv_phase<VT, LPR, false, false>(a, X, X, [&](int i, VT s, VT) {
      const VT r = B[i] - s;
      R0[i] = r;
      RR[i] = r;
      BP[i] = r;
      XP[i] = X[i];
      XT[i] = 0.0;
      acc[0] += (double)B[i] * (double)B[i];
      acc[1] += (double)r * (double)r;
    });
    for (int j = 0; j < L1; ++j)  // u_j start at zero (RealBiCGStabl zeroes its work array)
      vec_loop<VT>(n, [&](int i, auto w) {
        constexpr int W = decltype(w)::value;
        vfill<W>(uv(j), i, VT(0));
      });
    block_sum<2>(acc, sm);
    store_partials(a, SLOT_BB, acc[0]);
    store_partials(a, SLOT_RR, acc[1]);
    store_partials(a, SLOT_RHO, acc[1]);  // rr . r_0 = ||r_0||^2
  }
  if (!grid_barrier(a.bar, a.err, epoch)) return;
  const double bnrm = sqrt(reduce_partials(a.partials + SLOT_BB * nb, nb, sm));
  const double rnrm0 = sqrt(reduce_partials(a.partials + SLOT_RR * nb, nb, sm));
  double errorind = rnrm0 / bnrm, rnrm = rnrm0, mxnrmx = rnrm0, mxnrmr = rnrm0;
  double alpha = 0.0, omega = 1.0, sigma = 1.0, rho0 = 1.0, rho1 = 0.0;
  int info = 0, round = 0, rounds = 0;
  if (errorind < a.tol) info = EGPU_HUTI_CONVERGENCE;
  else if (a.divtol > 0.0 && errorind > a.divtol) info = 3;  // IterativeMethods.src:626-629
  bool done_x = info != 0;  // converged or diverged at the initial guess: x unchanged
  for (round = 1; info == 0 && round <= a.maxit; ++round) {
    // --------------------------------------------------------------- the BiCG part
    rounds = round;
    rho0 = -omega * rho0;
    bool early = false;
    for (int k = 1; k <= l; ++k) {
      rho1 = reduce_partials(a.partials + SLOT_RHO * nb, nb, sm);
      if (rho0 == 0.0 || rho1 != rho1) {
        info = 3;  // HUTI_DIVERGENCE (the reference stops with Fatal)
        early = true;
        break;
      }
      const double beta = alpha * (rho1 / rho0);
      rho0 = rho1;
      for (int j = 0; j <= k - 1; ++j) {
        VT *U = uv(j);
        const VT *Rj = rv(j);
        vec_loop<VT>(n, [&](int i, auto w) {
          constexpr int W = decltype(w)::value;
          VT u[W], r[W];
          vld<W>(U, i, u);
          vld<W>(Rj, i, r);
#pragma unroll
          for (int q = 0; q < W; ++q) u[q] = r[q] - beta * u[q];
          vst<W>(U, i, u);
        });
      }
      if (!grid_barrier(a.bar, a.err, epoch)) return;
      if (!precond(uv(k - 1), T)) return;
      {
        double acc[1] = {0.0};
        VT *Uk = uv(k);
        spmv_phase<VT, LPR, false, false>(a, T, T, [&](int i, VT s, VT) {
          Uk[i] = s;
          acc[0] += (double)RR[i] * (double)s;
        });
        block_sum<1>(acc, sm);
        store_partials(a, SLOT_PQ, acc[0]);
      }
      if (!grid_barrier(a.bar, a.err, epoch)) return;
      sigma = reduce_partials(a.partials + SLOT_PQ * nb, nb, sm);
      if (sigma == 0.0 || sigma != sigma) {
        info = 3;
        early = true;
        break;
      }
      alpha = rho1 / sigma;
      {
        double acc[1] = {0.0};
        const VT *U0 = uv(0);
        vec_loop<VT>(n, [&](int i, auto w) {
          constexpr int W = decltype(w)::value;
          VT xt[W], u0[W];
          vld<W>(XT, i, xt);
          vld<W>(U0, i, u0);
#pragma unroll
          for (int q = 0; q < W; ++q) xt[q] = xt[q] + alpha * u0[q];
          vst<W>(XT, i, xt);
        });
        for (int j = 0; j <= k - 1; ++j) {
          VT *Rj = rv(j);
          const VT *Un = uv(j + 1);
          vec_loop<VT>(n, [&](int i, auto w) {
            constexpr int W = decltype(w)::value;
            VT r[W], u[W];
            vld<W>(Rj, i, r);
            vld<W>(Un, i, u);
#pragma unroll
            for (int q = 0; q < W; ++q) {
              r[q] = r[q] - alpha * u[q];
              if (j == 0) acc[0] += (double)r[q] * (double)r[q];
            }
            vst<W>(Rj, i, r);
          });
        }
        block_sum<1>(acc, sm);
        store_partials(a, SLOT_RR, acc[0]);
      }
      if (!grid_barrier(a.bar, a.err, epoch)) return;
      rnrm = sqrt(reduce_partials(a.partials + SLOT_RR * nb, nb, sm));
      mxnrmx = fmax(mxnrmx, rnrm);
      mxnrmr = fmax(mxnrmr, rnrm);
      errorind = rnrm / bnrm;
      if (errorind < a.tol || errorind != errorind) {
        info = errorind < a.tol ? EGPU_HUTI_CONVERGENCE : 3;
        early = true;
        break;
      }
      if (!precond(rv(k - 1), T)) return;
      {
        double acc[1] = {0.0};
        VT *Rk = rv(k);
        spmv_phase<VT, LPR, false, false>(a, T, T, [&](int i, VT s, VT) {
          Rk[i] = s;
          acc[0] += (double)RR[i] * (double)s;  // rho of the next step
        });
        block_sum<1>(acc, sm);
        store_partials(a, SLOT_RHO, acc[0]);
      }
      if (!grid_barrier(a.bar, a.err, epoch)) return;
    }
    if (early) break;
    // --------------------------------------------------------------- the polynomial part
    {
      // Gram matrix Z_ij = r_i . r_j, j <= i, one pass over the l+1 vectors per entry
      int slot = 0;
      for (int i2 = 0; i2 < L1; ++i2)
        for (int j2 = 0; j2 <= i2; ++j2, ++slot) {
          double acc[1] = {0.0};
          const VT *Ri = rv(i2), *Rj = rv(j2);
          vec_loop<VT>(n, [&](int i, auto w) {
            constexpr int W = decltype(w)::value;
            VT x1[W], x2[W];
            vld<W>(Ri, i, x1);
            vld<W>(Rj, i, x2);
#pragma unroll
            for (int q = 0; q < W; ++q) acc[0] += (double)x1[q] * (double)x2[q];
          });
          block_sum<1>(acc, sm);
          if (threadIdx.x == 0) gram[slot * nb + blockIdx.x] = acc[0];
        }
    }
    if (!grid_barrier(a.bar, a.err, epoch)) return;
    {
      int slot = 0;
      for (int i2 = 0; i2 < L1; ++i2)
        for (int j2 = 0; j2 <= i2; ++j2, ++slot) {
          const double z = reduce_partials(gram + slot * nb, nb, sm);
          if (threadIdx.x == 0) {
            Zs[i2 + j2 * L1] = z;
            Zs[j2 + i2 * L1] = z;
          }
        }
      __syncthreads();
      // every block solves the small system redundantly (identical inputs, identical result)
      if (threadIdx.x == 0) {
        double M[(BL_MAXL - 1) * (BL_MAXL - 1)], y0[BL_MAXL + 1], yl[BL_MAXL + 1], yv[BL_MAXL + 1];
        int piv[BL_MAXL];
        const int lm = l - 1;
        for (int j = 0; j < lm; ++j)
          for (int i = 0; i < lm; ++i) M[i + j * lm] = Zs[(i + 1) + (j + 1) * L1];
        if (lm > 0) bl_lu(lm, M, lm, piv);
        y0[0] = -1.0;
        for (int i = 1; i < l; ++i) y0[i] = Zs[i];
        if (lm > 0) bl_lu_solve(lm, M, lm, piv, y0 + 1);
        y0[l] = 0.0;
        yl[0] = 0.0;
        for (int i = 1; i < l; ++i) yl[i] = Zs[i + l * L1];
        if (lm > 0) bl_lu_solve(lm, M, lm, piv, yl + 1);
        yl[l] = -1.0;
        auto symv = [&](const double *v, double *o) {
          for (int i = 0; i < L1; ++i) {
            double t = 0.0;
            for (int j = 0; j < L1; ++j) t = t + Zs[i + j * L1] * v[j];
            o[i] = t;
          }
        };
        auto sdot = [&](const double *p, const double *q) {
          double t = 0.0;
          for (int i = 0; i < L1; ++i) t = t + p[i] * q[i];
          return t;
        };
        symv(y0, yv);
        const double kappa0 = sqrt(sdot(y0, yv));
        symv(yl, yv);
        const double kappal = sqrt(sdot(yl, yv));
        symv(y0, yv);
        const double varrho = sdot(yl, yv) / (kappa0 * kappal);
        const double hatgamma = varrho / fabs(varrho) * fmax(fabs(varrho), 7e-1) * kappa0 / kappal;
        for (int i = 0; i < L1; ++i) y0s[i] = y0[i] - hatgamma * yl[i];
      }
      __syncthreads();
    }
    omega = y0s[l];
    // update u_0, x~, r_0 (j = 1..l in order, per element)
    vec_loop<VT>(n, [&](int i, auto w) {
      constexpr int W = decltype(w)::value;
      VT u0[W], xt[W], r0[W], t1[W], t2[W];
      vld<W>(uv(0), i, u0);
      vld<W>(XT, i, xt);
      vld<W>(rv(0), i, r0);
      for (int j = 1; j <= l; ++j) {
        const double c = y0s[j];
        vld<W>(uv(j), i, t1);
#pragma unroll
        for (int q = 0; q < W; ++q) u0[q] = u0[q] - c * t1[q];
        vld<W>(rv(j - 1), i, t2);
#pragma unroll
        for (int q = 0; q < W; ++q) xt[q] = xt[q] + c * t2[q];
        vld<W>(rv(j), i, t1);
#pragma unroll
        for (int q = 0; q < W; ++q) r0[q] = r0[q] - c * t1[q];
      }
      vst<W>(uv(0), i, u0);
      vst<W>(XT, i, xt);
      vst<W>(rv(0), i, r0);
    });
    {
      double yv[BL_MAXL + 1];
      for (int i = 0; i < L1; ++i) {
        double t = 0.0;
        for (int j = 0; j < L1; ++j) t = t + Zs[i + j * L1] * y0s[j];
        yv[i] = t;
      }
      double t = 0.0;
      for (int i = 0; i < L1; ++i) t = t + y0s[i] * yv[i];
      rnrm = sqrt(t);
    }
    if (!grid_barrier(a.bar, a.err, epoch)) return;
    // --------------------------------------------------------------- reliable updates
    const double delta = 1.0e-2;
    mxnrmx = fmax(mxnrmx, rnrm);
    mxnrmr = fmax(mxnrmr, rnrm);
    const bool xpdt = rnrm < delta * rnrm0 && rnrm0 < mxnrmx;
    const bool rcmp = (rnrm < delta * mxnrmr && rnrm0 < mxnrmr) || xpdt;
    if (rcmp) {
      if (!precond(XT, T)) return;
      VT *R0 = rv(0);
      spmv_phase<VT, LPR, false, false>(a, T, T, [&](int i, VT s, VT) {
        const VT r = BP[i] - s;
        R0[i] = r;
        if (xpdt) {
          XP[i] = XP[i] + T[i];
          XT[i] = 0.0;
          BP[i] = r;
        }
      });
      mxnrmr = rnrm;
      if (xpdt) mxnrmx = rnrm;
      if (!grid_barrier(a.bar, a.err, epoch)) return;
    }
    // rho for the next round's first step: rr . r_0
    {
      double acc[1] = {0.0};
      const VT *R0 = rv(0);
      vec_loop<VT>(n, [&](int i, auto w) {
        constexpr int W = decltype(w)::value;
        VT x1[W], x2[W];
        vld<W>(RR, i, x1);
        vld<W>(R0, i, x2);
#pragma unroll
        for (int q = 0; q < W; ++q) acc[0] += (double)x1[q] * (double)x2[q];
      });
      block_sum<1>(acc, sm);
      store_partials(a, SLOT_RHO, acc[0]);
    }
    if (!grid_barrier(a.bar, a.err, epoch)) return;
    errorind = rnrm / bnrm;
    if (errorind < a.tol) info = EGPU_HUTI_CONVERGENCE;
    else if (errorind != errorind || (a.divtol > 0.0 && errorind > a.divtol)) info = 3;  // :817-819
  }
  if (info == 0) info = EGPU_HUTI_MAXITER;
  const int iters = rounds;
  // x = M^-1 x~ + xp
  if (!done_x) {
    if (!precond(XT, T)) return;
    vec_loop<VT>(n, [&](int i, auto w) {
      constexpr int W = decltype(w)::value;
      VT t[W], xp[W];
      vld<W>(T, i, t);
      vld<W>(XP, i, xp);
#pragma unroll
      for (int q = 0; q < W; ++q) t[q] = t[q] + xp[q];
      vst<W>(X, i, t);
    });
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.out_i[0] = info;
    a.out_i[1] = iters;
    a.out_d[0] = errorind;
    a.out_d[1] = bnrm;
  }
}

}  // namespace egpu
