// egpu_kbicgstab32.cu -- the BiCGStab kernels, FP32
#include "egpu_krylov_launch.cuh"

namespace egpu {

template <typename VT, bool OFFS>
static int launch_form(egpu_ctx *ctx, KArgs<VT> &a, int form, size_t smem) {
  switch (form) {
    case TRI_CTA: return launch_coop(ctx, bicgstab_kernel<VT, TRI_TS, OFFS, TRI_CTA>, a, nullptr, smem);
    case TRI_RANGE7: return launch_coop(ctx, bicgstab_kernel<VT, TRI_TS, OFFS, TRI_RANGE7>, a, nullptr, smem);
    case TRI_RANGE10: return launch_coop(ctx, bicgstab_kernel<VT, TRI_TS, OFFS, TRI_RANGE10>, a, nullptr, smem);
    default: return launch_coop(ctx, bicgstab_kernel<VT, TRI_TS, OFFS, TRI_SYNCFREE>, a, nullptr, smem,
                                  a.precond == EGPU_PREC_ILU0 ? 0 : krylov_blocks(a.nslices));
  }
}

int launch_bicgstab(egpu_ctx *ctx, KArgs<float> &a, bool offs, int form, size_t smem) {
  if (a.sweeps_l > 0 && a.precond == EGPU_PREC_ILU0)
    return offs ? launch_coop(ctx, bicgstab_kernel<float, TRI_TS, true, TRI_SYNCFREE, true>, a, nullptr, 0, krylov_blocks(a.nslices))
                : launch_coop(ctx, bicgstab_kernel<float, TRI_TS, false, TRI_SYNCFREE, true>, a, nullptr, 0, krylov_blocks(a.nslices));
  return offs ? launch_form<float, true>(ctx, a, form, smem) : launch_form<float, false>(ctx, a, form, smem);
}

}  // namespace egpu
