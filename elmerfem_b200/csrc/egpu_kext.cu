// egpu_kext.cu -- the GCR and BiCGStab(l) kernels (FP64)
#include "egpu_krylov_launch.cuh"

namespace egpu {

int launch_ext(egpu_ctx *ctx, KArgs<double> &a, int method, int form, size_t smem) {
  if (method == EGPU_GCR) {
    switch (form) {
      case TRI_CTA: return launch_coop(ctx, gcr_kernel<TRI_TS, TRI_CTA>, a, nullptr, smem);
      case TRI_RANGE7: return launch_coop(ctx, gcr_kernel<TRI_TS, TRI_RANGE7>, a, nullptr, smem);
      case TRI_RANGE10: return launch_coop(ctx, gcr_kernel<TRI_TS, TRI_RANGE10>, a, nullptr, smem);
      default: return launch_coop(ctx, gcr_kernel<TRI_TS, TRI_SYNCFREE>, a, nullptr, smem);
    }
  }
  switch (form) {
    case TRI_CTA: return launch_coop(ctx, bicgstabl_kernel<TRI_TS, TRI_CTA>, a, nullptr, smem);
    case TRI_RANGE7: return launch_coop(ctx, bicgstabl_kernel<TRI_TS, TRI_RANGE7>, a, nullptr, smem);
    case TRI_RANGE10: return launch_coop(ctx, bicgstabl_kernel<TRI_TS, TRI_RANGE10>, a, nullptr, smem);
    default: return launch_coop(ctx, bicgstabl_kernel<TRI_TS, TRI_SYNCFREE>, a, nullptr, smem);
  }
}

}  // namespace egpu
