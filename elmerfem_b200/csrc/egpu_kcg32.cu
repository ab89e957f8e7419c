// egpu_kcg32.cu -- the CG kernels, FP32
// The grid barrier out of line: the SpMV loop, which needs all 64 registers, came out up to 12%
// slower with the barrier inlined six times around it (128^3 mixed CG's inner solves, unrolled
// by 8: 39.8 and 35.3 ms).  The FP64 kernels are the other way round (57.2 and 60.9 ms).
#define EGPU_BARRIER_CALL
#include "egpu_krylov_launch.cuh"

namespace egpu {

template <bool OFFS>
static int launch(egpu_ctx *ctx, KArgs<float> &a, int form, size_t smem, bool load) {
  return launch_form(ctx, a, form, smem, krylov_blocks(a.nslices), load,
                     [](auto tri) { return cg_kernel<float, TRI_TS, OFFS, decltype(tri)::value>; });
}

int launch_cg(egpu_ctx *ctx, KArgs<float> &a, bool offs, int form, size_t smem, bool load) {
  return offs ? launch<true>(ctx, a, form, smem, load) : launch<false>(ctx, a, form, smem, load);
}

}  // namespace egpu
