// egpu_kext.cu -- the GCR and BiCGStab(l) kernels (FP64)
#include "egpu_krylov_launch.cuh"

namespace egpu {

int launch_ext(egpu_ctx *ctx, KArgs<double> &a, int method, int form, size_t smem, bool load) {
  if (method == EGPU_GCR)
    return launch_form(ctx, a, form, smem, 0, load, [](auto tri) { return gcr_kernel<TRI_TS, decltype(tri)::value>; });
  return launch_form(ctx, a, form, smem, 0, load, [](auto tri) { return bicgstabl_kernel<TRI_TS, decltype(tri)::value>; });
}

}  // namespace egpu
