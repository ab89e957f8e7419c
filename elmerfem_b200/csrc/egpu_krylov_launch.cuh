// egpu_krylov_launch.cuh -- launches of the persistent Krylov kernels.  The kernels of a method and
// a precision are instantiated in a translation unit of their own (egpu_kcg32.cu, egpu_kcg64.cu,
// egpu_kbicgstab32.cu, egpu_kbicgstab64.cu, egpu_kext.cu), so that they compile side by side.
#pragma once

#include <algorithm>
#include <type_traits>

#include "egpu_krylov.cuh"
#include "egpu_solve.h"

namespace egpu {

// One warp per row in the sync-free triangular solves: rows that depend on each other
// never share a warp, so no lane spins while a diverged lane of its own warp has to
// produce the value it waits for.
constexpr int TRI_TS = 32;

// occupancy-sized cooperative launch, of at most `most` blocks (0: no limit); load: none, the
// kernel is loaded only
template <typename K, typename Args>
int launch_coop(egpu_ctx *ctx, K kernel, Args &args, size_t smem, int most, bool load) {
  int bps = 0;
  const int rc = kernel_blocks(ctx, (const void *)kernel, smem, &bps);
  if (rc || load) return rc;
  bps = std::min(bps, 2048 / EGPU_KBLOCK);
  int grid = ctx->num_sms * bps;
  if (most > 0) grid = std::min(grid, most);
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

// pick(form as a constant): the kernel instantiated for that form; most: blocks without triangular
// solves (0: no limit)
template <typename VT, typename Pick>
int launch_form(egpu_ctx *ctx, KArgs<VT> &a, int form, size_t smem, int most, bool load, Pick pick) {
  switch (form) {
    case TRI_CTA: return launch_coop(ctx, pick(std::integral_constant<int, TRI_CTA>{}), a, smem, 0, load);
    case TRI_RANGE7: return launch_coop(ctx, pick(std::integral_constant<int, TRI_RANGE7>{}), a, smem, 0, load);
    case TRI_RANGE10: return launch_coop(ctx, pick(std::integral_constant<int, TRI_RANGE10>{}), a, smem, 0, load);
    default:
      return launch_coop(ctx, pick(std::integral_constant<int, TRI_SYNCFREE>{}), a, smem,
                         a.precond == EGPU_PREC_ILU0 ? 0 : most, load);
  }
}

// offs: 16-bit column offsets; form: a TriForm; smem: dynamic shared memory per block; load: see
// launch_coop
int launch_cg(egpu_ctx *ctx, KArgs<double> &a, bool offs, int form, size_t smem, bool load);
int launch_cg(egpu_ctx *ctx, KArgs<float> &a, bool offs, int form, size_t smem, bool load);
int launch_bicgstab(egpu_ctx *ctx, KArgs<double> &a, bool offs, int form, size_t smem, bool load);
// sweeps: a.sweeps_l > 0
int launch_bicgstab(egpu_ctx *ctx, KArgs<float> &a, bool offs, int form, size_t smem, bool load);
// GCR, BiCGStab(l)
int launch_ext(egpu_ctx *ctx, KArgs<double> &a, int method, int form, size_t smem, bool load);

}  // namespace egpu
