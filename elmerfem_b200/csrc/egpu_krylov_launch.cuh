// egpu_krylov_launch.cuh -- launches of the persistent Krylov kernels.  Each method's kernels
// are instantiated in a translation unit of their own (egpu_kcg.cu, egpu_kbicgstab.cu,
// egpu_kext.cu).
#pragma once

#include <algorithm>

#include "egpu_krylov.cuh"
#include "egpu_solve.h"

namespace egpu {

// One warp per row in the sync-free triangular solves: rows that depend on each other
// never share a warp, so no lane spins while a diverged lane of its own warp has to
// produce the value it waits for.
constexpr int TRI_TS = 32;

// occupancy-sized cooperative launch, of at most `most` blocks (0: no limit)
template <typename K, typename Args>
int launch_coop(egpu_ctx *ctx, K kernel, Args &args, int *grid_out = nullptr, size_t smem = 0, int most = 0) {
  int bps = 0;
  if (smem > 48 * 1024) {
    const int rc = allow_shared(ctx, (const void *)kernel);
    if (rc) return rc;
  }
  EGPU_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, kernel, EGPU_KBLOCK, smem));
  if (bps < 1) {
    egpu_set_error(ctx, "persistent kernel does not fit on an SM");
    return EGPU_ERR_CUDA;
  }
  if (args.nslices == 0) return EGPU_OK;  // the query above has loaded the kernel (krylov_load)
  bps = std::min(bps, 2048 / EGPU_KBLOCK);
  int grid = ctx->num_sms * bps;
  if (most > 0) grid = std::min(grid, most);
  if (grid_out) *grid_out = grid;
  void *kargs[] = {&args};
  EGPU_CUDA_TRY(ctx, cudaLaunchCooperativeKernel((const void *)kernel, dim3(grid), dim3(EGPU_KBLOCK),
                                                 kargs, smem, ctx->stream));
  ctx->launches++;
  return EGPU_OK;
}

// Blocks of a solve without triangular solves: one for every SLICES_PER_BLOCK SELL slices.  A
// small system's iteration is barriers and reductions, which cost less among fewer blocks; with
// too few the slices of a block follow one another.  CG on hex 16^3 at 4, 8, 16, 32 and 64 slices
// a block: 683, 658, 650, 658 and 853 us (all 148 blocks: 775); from 2368 slices on every SM has one.
constexpr int SLICES_PER_BLOCK = 16;
inline int krylov_blocks(int nslices) {
  return std::max(1, (nslices + SLICES_PER_BLOCK - 1) / SLICES_PER_BLOCK);
}

// offs: 16-bit column offsets; form: a TriForm; smem: dynamic shared memory per block
int launch_cg(egpu_ctx *ctx, KArgs<double> &a, bool offs, int form, size_t smem);
int launch_cg(egpu_ctx *ctx, KArgs<float> &a, bool offs, int form, size_t smem);
int launch_bicgstab(egpu_ctx *ctx, KArgs<double> &a, bool offs, int form, size_t smem);
int launch_bicgstab(egpu_ctx *ctx, KArgs<float> &a, bool offs, int form, size_t smem);  // sweeps: a.sweeps_l > 0
int launch_ext(egpu_ctx *ctx, KArgs<double> &a, int method, int form, size_t smem);     // GCR, BiCGStab(l)

}  // namespace egpu
