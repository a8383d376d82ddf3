// Backward tensor-core kernels for head_dim 128 (no factor operands, both 16-bit types).
#include "fb_bwd_t_sm100.cuh"

namespace fb {

template <typename T>
static int dispatch_bwd_t(const fb_params* p, const PackPlan& plan, cudaStream_t st) {
  if (p->alibi_slopes) return launch_bwd_t_t<T, 128, BWD_ALIBI>(p, plan, st);
  if (p->mask_kind != FB_MASK_NONE) return launch_bwd_t_t<T, 128, BWD_MASK>(p, plan, st);
  return launch_bwd_t_t<T, 128, BWD_PLAIN>(p, plan, st);
}

int dispatch_bwd_d128(const fb_params* p, const PackPlan& plan, cudaStream_t st) {
  return p->dtype == FB_DTYPE_F16 ? dispatch_bwd_t<__half>(p, plan, st) : dispatch_bwd_t<__nv_bfloat16>(p, plan, st);
}

}  // namespace fb
