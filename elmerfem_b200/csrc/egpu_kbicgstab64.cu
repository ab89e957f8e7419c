// egpu_kbicgstab64.cu -- the BiCGStab kernels, FP64
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

int launch_bicgstab(egpu_ctx *ctx, KArgs<double> &a, bool offs, int form, size_t smem) {
  return offs ? launch_form<double, true>(ctx, a, form, smem) : launch_form<double, false>(ctx, a, form, smem);
}

}  // namespace egpu
