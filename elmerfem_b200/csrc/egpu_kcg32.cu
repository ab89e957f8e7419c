// egpu_kcg32.cu -- the CG kernels, FP32
// The grid barrier out of line: the SpMV loop, which needs all 64 registers, came out up to 12%
// slower with the barrier inlined six times around it (128^3 mixed CG's inner solves, unrolled
// by 8: 39.8 and 35.3 ms).  The FP64 kernels are the other way round (57.2 and 60.9 ms).
#define EGPU_BARRIER_CALL
#include "egpu_krylov_launch.cuh"

namespace egpu {

template <typename VT, bool OFFS>
static int launch_form(egpu_ctx *ctx, KArgs<VT> &a, int form, size_t smem) {
  switch (form) {
    case TRI_CTA: return launch_coop(ctx, cg_kernel<VT, TRI_TS, OFFS, TRI_CTA>, a, nullptr, smem);
    case TRI_RANGE7: return launch_coop(ctx, cg_kernel<VT, TRI_TS, OFFS, TRI_RANGE7>, a, nullptr, smem);
    case TRI_RANGE10: return launch_coop(ctx, cg_kernel<VT, TRI_TS, OFFS, TRI_RANGE10>, a, nullptr, smem);
    default: return launch_coop(ctx, cg_kernel<VT, TRI_TS, OFFS, TRI_SYNCFREE>, a, nullptr, smem,
                                  a.precond == EGPU_PREC_ILU0 ? 0 : krylov_blocks(a.nslices));
  }
}

int launch_cg(egpu_ctx *ctx, KArgs<float> &a, bool offs, int form, size_t smem) {
  return offs ? launch_form<float, true>(ctx, a, form, smem) : launch_form<float, false>(ctx, a, form, smem);
}

}  // namespace egpu
