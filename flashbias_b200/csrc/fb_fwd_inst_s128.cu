// Two-stream forward kernels for head_dim 65 to 128 (no mask, packed rank up to 32, both 16-bit types).
#include "fb_fwd_s_sm100.cuh"

namespace fb {

template <typename T>
static int dispatch_t(const fb_params* p, const PackPlan& plan, cudaStream_t st) {
  if (p->alibi_slopes) return launch_fwd_s<T, 0, 1, FWD_ALIBI>(p, plan, st);
  switch (plan.RP) {
    case 0: return launch_fwd_s<T, 0, 1, FWD_PLAIN>(p, plan, st);
    case 16: return plan.nq == 2 ? launch_fwd_s<T, 16, 2, FWD_PLAIN>(p, plan, st) : launch_fwd_s<T, 16, 1, FWD_PLAIN>(p, plan, st);
    case 32: return plan.nq == 2 ? launch_fwd_s<T, 32, 2, FWD_PLAIN>(p, plan, st) : launch_fwd_s<T, 32, 1, FWD_PLAIN>(p, plan, st);
  }
  return FB_ENOTBUILT;
}

int dispatch_fwd_s(const fb_params* p, const PackPlan& plan, cudaStream_t st) {
  return p->dtype == FB_DTYPE_F16 ? dispatch_t<__half>(p, plan, st) : dispatch_t<__nv_bfloat16>(p, plan, st);
}

}  // namespace fb
