// Forward tensor-core kernels for head_dim 128 with a mask or a packed rank above 32 (both 16-bit types); the others: the
// two-stream kernels.
#include "fb_fwd_sm100.cuh"

namespace fb {

template <typename T>
static int dispatch_t(const fb_params* p, const PackPlan& plan, cudaStream_t st) {
  const bool masked = p->mask_kind != FB_MASK_NONE;
  switch (plan.RP) {
    case 0: return launch_fwd_t<T, 128, 0, 1, FWD_MASK>(p, plan, st);
    case 16: return plan.nq == 2 ? launch_fwd_t<T, 128, 16, 2, FWD_MASK>(p, plan, st)
                                 : launch_fwd_t<T, 128, 16, 1, FWD_MASK>(p, plan, st);
    case 32: return plan.nq == 2 ? launch_fwd_t<T, 128, 32, 2, FWD_MASK>(p, plan, st)
                                 : launch_fwd_t<T, 128, 32, 1, FWD_MASK>(p, plan, st);
    case 64:
      if (masked)
        return plan.nq == 2 ? launch_fwd_t<T, 128, 64, 2, FWD_MASK>(p, plan, st) : launch_fwd_t<T, 128, 64, 1, FWD_MASK>(p, plan, st);
      return plan.nq == 2 ? launch_fwd_t<T, 128, 64, 2, FWD_PLAIN>(p, plan, st) : launch_fwd_t<T, 128, 64, 1, FWD_PLAIN>(p, plan, st);
    case 128:
      if (masked)
        return plan.nq == 2 ? launch_fwd_t<T, 128, 128, 2, FWD_MASK>(p, plan, st)
                            : launch_fwd_t<T, 128, 128, 1, FWD_MASK>(p, plan, st);
      return plan.nq == 2 ? launch_fwd_t<T, 128, 128, 2, FWD_PLAIN>(p, plan, st)
                          : launch_fwd_t<T, 128, 128, 1, FWD_PLAIN>(p, plan, st);
  }
  return FB_ENOTBUILT;
}

int dispatch_fwd_d128(const fb_params* p, const PackPlan& plan, cudaStream_t st) {
  return p->dtype == FB_DTYPE_F16 ? dispatch_t<__half>(p, plan, st) : dispatch_t<__nv_bfloat16>(p, plan, st);
}

}  // namespace fb
