// egpu_kbicgstab32.cu -- the BiCGStab kernels, FP32
#include "egpu_krylov_launch.cuh"

namespace egpu {

template <bool OFFS>
static int launch(egpu_ctx *ctx, KArgs<float> &a, int form, size_t smem, bool load) {
  return launch_form(ctx, a, form, smem, krylov_blocks(a.nslices), load,
                     [](auto tri) { return bicgstab_kernel<float, TRI_TS, OFFS, decltype(tri)::value>; });
}

int launch_bicgstab(egpu_ctx *ctx, KArgs<float> &a, bool offs, int form, size_t smem, bool load) {
  if (a.sweeps_l > 0 && a.precond == EGPU_PREC_ILU0) {
    const int most = krylov_blocks(a.nslices);
    return offs ? launch_coop(ctx, bicgstab_kernel<float, TRI_TS, true, TRI_SYNCFREE, true>, a, 0, most, load)
                : launch_coop(ctx, bicgstab_kernel<float, TRI_TS, false, TRI_SYNCFREE, true>, a, 0, most, load);
  }
  return offs ? launch<true>(ctx, a, form, smem, load) : launch<false>(ctx, a, form, smem, load);
}

}  // namespace egpu
