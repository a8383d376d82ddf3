// Two-stream backward kernels for head_dim 33 to 64 (without a mask, both 16-bit types).
#include "fb_bwd_s_sm100.cuh"

namespace fb {

template <typename T>
static int dispatch_t(const fb_params* p, const PackPlan& plan, cudaStream_t st) {
  if (p->alibi_slopes) return launch_bwd_s<T, 64, 0, 0, 1, BWD_ALIBI>(p, plan, st);
  switch (plan.RC) {
    case 0: return launch_bwd_s<T, 64, 0, 0, 1, BWD_PLAIN>(p, plan, st);
    case 16: return plan.nq == 2 ? launch_bwd_s<T, 64, 16, 16, 2, BWD_PLAIN>(p, plan, st)
                                 : launch_bwd_s<T, 64, 16, 16, 1, BWD_PLAIN>(p, plan, st);
  }
  return FB_ENOTBUILT;
}

int dispatch_bwd_s64(const fb_params* p, const PackPlan& plan, cudaStream_t st) {
  return p->dtype == FB_DTYPE_F16 ? dispatch_t<__half>(p, plan, st) : dispatch_t<__nv_bfloat16>(p, plan, st);
}

}  // namespace fb
