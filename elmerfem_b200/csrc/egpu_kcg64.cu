// egpu_kcg64.cu -- the CG kernels, FP64
#include "egpu_krylov_launch.cuh"

namespace egpu {

template <bool OFFS>
static int launch(egpu_ctx *ctx, KArgs<double> &a, int form, size_t smem, bool load) {
  return launch_form(ctx, a, form, smem, krylov_blocks(a.nslices), load,
                     [](auto tri) { return cg_kernel<double, TRI_TS, OFFS, decltype(tri)::value>; });
}

int launch_cg(egpu_ctx *ctx, KArgs<double> &a, bool offs, int form, size_t smem, bool load) {
  return offs ? launch<true>(ctx, a, form, smem, load) : launch<false>(ctx, a, form, smem, load);
}

}  // namespace egpu
