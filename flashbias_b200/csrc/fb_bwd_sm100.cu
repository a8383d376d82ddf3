// Backward tensor-core path, host side: which problems the tcgen05/TMA kernels take, workspace size, and the
// dispatch to the per-head_dim translation units that hold the kernel instantiations.
#include "fb_bwd_sm100.cuh"

namespace fb {

static bool rows_16b_ok(const void* ptr, const int64_t* st) {
  if (reinterpret_cast<uintptr_t>(ptr) & 15) return false;
  for (int i = 0; i < 3; ++i)
    if (st[i] & 7) return false;
  return true;
}

// the variants launch_bwd_sm100 can dispatch to, and whether their tiles fit one SM
bool bwd_cfg_fits(int D, int RP, int nq) {
#define FB_FIT(DD, RR) \
  if (D == DD && RP == RR) return nq == 2 ? BwdCfg<DD, RR, 2>::FITS : BwdCfg<DD, RR, 1>::FITS;
  FB_FIT(32, 0) FB_FIT(32, 32) FB_FIT(32, 64)
  FB_FIT(64, 0) FB_FIT(64, 16) FB_FIT(64, 32)
#undef FB_FIT
  if (D == 128 && RP == 0) return true;  // key-major kernel only
  return false;
}

// Whether the persistent form of the query-major kernel is the better one for a problem with factors at head_dim 32.  What it
// saves is the start and the drain of a CTA per work item, so: at least two items per SM, and few query tiles per item (mean):
//  - up to rank 16, up to 20 (persistent / two-stream kernel, us: B256 H24 S256 R16 369 / 805, B1 H50 S1280 R2 80 / 88, S2304
//    causal 119 / 134, S4096 causal 319 / 336; at 32 tiles, S8192 causal 1182 / 1179; B2 H8 S16384 R5 3058 / 2789);
//  - above, where it has no staging tile to drain through, up to 4 with a split scale (B16 H16 R17 / R24 / R32, 5 tiles, 148 / 139,
//    148 / 141, 158 / 154; 8 tiles 334 / 285, 335 / 294, 361 / 325), up to 7 without (5 tiles 128 / 137, 131 / 140, 139 / 154; 6 tiles
//    178 / 184, 182 / 191, 191 / 208; 8 tiles 287 / 285, 291 / 293, 307 / 323, and causal R32 680 / 667);
//  - with a mask, where the other choice is the one-item form of the same kernel, up to 8.
static bool bwd_prefers_persistent(const fb_params* p, const PackPlan& plan) {
  int dev = 0;
  cudaGetDevice(&dev);
  const int sms = device_sm_count(dev);
  const int nq = (p->Sq + 127) / 128, nk = (p->Sk + 127) / 128;
  const int tiles_per_item = p->causal ? (nq + 1) / 2 : nq;  // mean, under causal masking
  const int most = p->mask_kind != FB_MASK_NONE ? 8 : p->R <= 16 ? 20 : plan.nq == 2 ? 4 : 7;
  return sms > 0 && tiles_per_item <= most && (int64_t)nk * p->B * p->H >= 2 * (int64_t)sms;
}

// The kernel (FB_KERNEL_BWD_*) that takes a problem with this plan.
static int bwd_kernel_for(const fb_params* p, const PackPlan& plan) {
  const bool factors = plan.RP > 0, by_query = p->flags & (factors ? FB_FLAG_BWD_ONE_ITEM : FB_FLAG_BWD_QUERY_MAJOR);
  // (the persistent form writes dK and dV with tile stores: their layout must be one a tensor map can describe)
  if (plan.TD == 32 && factors && !(p->flags & FB_FLAG_BWD_ONE_ITEM) &&
      ((p->flags & FB_FLAG_BWD_PERSISTENT) || bwd_prefers_persistent(p, plan)) &&
      (!p->dk || tma_compatible(p->dk, p->dk_stride[2], p->dk_stride[1], p->dk_stride[0], p->H, p->B)) &&
      (!p->dv || tma_compatible(p->dv, p->dv_stride[2], p->dv_stride[1], p->dv_stride[0], p->H, p->B)))
    return FB_KERNEL_BWD_PERSISTENT;
  // Every other problem without a mask at head_dim up to 64, except those that ask for another form by flag (head_dim 32), and ranks
  // 9 to 16 above head_dim 32, whose accumulators leave no room for dS^T in tensor memory.
  if (p->mask_kind == FB_MASK_NONE && plan.TD <= 64 && !(plan.TD == 32 && by_query) && !(plan.TD == 64 && plan.RP > 16))
    return FB_KERNEL_BWD_TWO_STREAM;
  // without factor operands: key-major where it is built
  if (!factors && (plan.TD == 128 || (plan.TD == 32 && !by_query))) return FB_KERNEL_BWD_KEY_MAJOR;
  return FB_KERNEL_BWD_QUERY_MAJOR;
}

bool bwd_sm100_supported(const fb_params* p, PackPlan* plan) {
  if (p->flags & FB_FLAG_FORCE_GENERAL) return false;
  if (p->alibi_slopes && p->mask_kind != FB_MASK_NONE) return false;  // both at once: shape-generic kernels
  if (p->D % 8 != 0) return false;  // other multiples of 8 run in the next wider tile, zero-filled by the loads
  if (!(p->softmax_scale > 0.f) || !isfinite(p->softmax_scale)) return false;
  if (!plan_pack(p, plan, true)) return false;
  if (!bwd_cfg_fits(plan->TD, plan->RP, plan->nq)) return false;  // shared or tensor memory of an SM exceeded
  if (!tma_compatible(p->q, p->q_stride[2], p->q_stride[1], p->q_stride[0], p->H, p->B)) return false;
  if (!tma_compatible(p->k, p->k_stride[2], p->k_stride[1], p->k_stride[0], p->H, p->B)) return false;
  if (!tma_compatible(p->v, p->v_stride[2], p->v_stride[1], p->v_stride[0], p->H, p->B)) return false;
  if (p->dout && !tma_compatible(p->dout, p->dout_stride[2], p->dout_stride[1], p->dout_stride[0], p->H, p->B))
    return false;
  if (p->dq && !rows_16b_ok(p->dq, p->dq_stride)) return false;
  if (p->dk && !rows_16b_ok(p->dk, p->dk_stride)) return false;
  if (p->dv && !rows_16b_ok(p->dv, p->dv_stride)) return false;
  if ((int64_t)p->B * p->H * ((p->Sk + 127) / 128) > 0x7fffffffLL) return false;
  plan->kernel = bwd_kernel_for(p, *plan);
  if (plan->kernel == FB_KERNEL_BWD_TWO_STREAM) plan_two_stream(p, plan);
  if (plan->kernel != FB_KERNEL_BWD_PERSISTENT) plan->qs_bytes = 0;  // k*scale is split on chip
  return true;
}

size_t bwd_sm100_workspace(const fb_params* p, const PackPlan& plan) { return bwd_layout(p, plan).total; }

int launch_bwd_sm100(const fb_params* p, const PackPlan& plan, cudaStream_t st) {
  if (plan.kernel == FB_KERNEL_BWD_TWO_STREAM)
    return plan.TD == 32 ? dispatch_bwd_s32(p, plan, st) : dispatch_bwd_s64(p, plan, st);
  if (plan.kernel == FB_KERNEL_BWD_PERSISTENT) return dispatch_bwd_d32p(p, plan, st);
  switch (plan.TD) {
    case 32: return dispatch_bwd_d32(p, plan, st);
    case 64: return dispatch_bwd_d64(p, plan, st);
    case 128: return dispatch_bwd_d128(p, plan, st);
  }
  return FB_ENOTBUILT;
}

}  // namespace fb
