// Operand preparation for the tensor-core kernels.
//
// The kernels accumulate all logit terms in ONE fp32 accumulator,  S = qs.k + qb.kb,  where the softmax
// scale has to live inside an operand:
//   * scale an exact power of two: qs = q (the caller's tensor, untouched) and qb = q_bias / scale,
//     which is exact in the 16-bit type; the exponent argument is S * scale * log2(e);
//   * otherwise: qs = q * scale as a (hi, lo) pair of 16-bit terms (contraction 2*head_dim), which the forward forms on chip,
//     and qb = q_bias as given, so that the products of the bias factors stay exact and un-scaled --
//     terms as large as an ALiBi position cancel inside one MMA instead of being rounded first.
// The backward keeps its key tile resident and streams the query tiles, so it puts the split on the key side
// instead: S = q.(k*scale), with k*scale as a (hi, lo) pair, formed on chip as well, or here for the persistent form.
// Factors are zero-padded to RP columns (16/32/64; the forward also takes 96 and 128).  The backward also gets a centred k-side copy
// (k_bias minus the k_bias of the middle key of its group of 32 keys, as a (hi, lo) pair).
#include <math.h>

#include "fb_common.cuh"
#include "fb_internal.h"

namespace fb {

static int pad_pow2_16(int x) {
  int r = 16;
  while (r < x) r <<= 1;
  return r;
}

bool plan_pack(const fb_params* p, PackPlan* plan, bool for_bwd) {
  plan->Bq = p->q_bias_stride[0] == 0 ? 1 : p->B;
  plan->Hq = p->q_bias_stride[1] == 0 ? 1 : p->H;
  plan->Bk = p->k_bias_stride[0] == 0 ? 1 : p->B;
  plan->Hk = p->k_bias_stride[1] == 0 ? 1 : p->H;
  plan->TD = p->D <= 32 ? 32 : p->D <= 64 ? 64 : 128;
  plan->kernel = FB_KERNEL_GENERAL;
  int e;
  bool pow2 = frexpf(p->softmax_scale, &e) == 0.5f;
  // fp16 factors divided by a scale below one could leave the range of the type: take the split form instead
  if (pow2 && p->dtype == FB_DTYPE_F16 && p->softmax_scale != 1.f && p->R > 0) pow2 = false;
  // without factor operands nothing shares the accumulator with q.k: the scale lives in the exponent multiplier
  if (p->R <= 0) pow2 = true;
  plan->nq = pow2 ? 1 : 2;
  plan->qb_mult = (pow2 && p->R > 0) ? (float)(1.0 / (double)p->softmax_scale) : 1.f;
  // persistent backward: scaled-key copy (the other kernels split q*scale or k*scale on chip)
  plan->qs_bytes = pow2 || !for_bwd ? 0 : round256((size_t)p->B * p->H * p->Sk * 2 * plan->TD * 2);
  plan->RC = 0;
  plan->kc_bytes = 0;
  if (p->R <= 0) {
    plan->RP = 0;
    plan->q_bytes = plan->k_bytes = 0;
    return true;
  }
  // the centred k-side copy of the backward holds a (hi, lo) pair: twice the rank
  plan->RP = pad_pow2_16(for_bwd ? 2 * p->R : p->R);
  // forward at head_dim 32: 96 packed columns fit two CTAs per SM where 128 fit one, without a mask and with an unsplit scale
  // (else one either way, with a quarter fewer columns to move and multiply)
  if (!for_bwd && plan->TD == 32 && p->R > 64 && p->R <= 96) plan->RP = 96;
  // backward at head_dim 32: factor tiles as wide as the Q/K tiles, so that [Q | Qb] and [K | Kc] are read as one
  // MMA operand each (one product instead of two per 16 query rows / keys)
  if (for_bwd && plan->TD == 32 && plan->RP < 32) plan->RP = 32;
  if (plan->RP > (for_bwd ? 64 : 128)) return false;
  plan->q_bytes = round256((size_t)plan->Bq * plan->Hq * p->Sq * plan->RP * 2);
  plan->k_bytes = round256((size_t)plan->Bk * plan->Hk * p->Sk * plan->RP * 2);
  if (for_bwd) {
    // beside a head_dim-32 K tile the centred copy is 32 columns wide: [K | Kc] then reads as one MMA operand
    plan->RC = (plan->TD == 32 && plan->RP < 32) ? 32 : plan->RP;
    plan->kc_bytes = round256((size_t)plan->Bk * plan->Hk * p->Sk * plan->RC * 2);
  }
  return true;
}

void plan_two_stream(const fb_params* p, PackPlan* plan) {
  if (p->R <= 0) return;
  plan->RP = pad_pow2_16(p->R);
  plan->RC = plan->TD == 32 ? 2 * plan->RP : pad_pow2_16(2 * p->R);
  plan->q_bytes = round256((size_t)plan->Bq * plan->Hq * p->Sq * plan->RP * 2);
  plan->k_bytes = round256((size_t)plan->Bk * plan->Hk * p->Sk * plan->RP * 2);
  plan->kc_bytes = round256((size_t)plan->Bk * plan->Hk * p->Sk * plan->RC * 2);
}

// One factor: (Bx, Hx, S, R) with strides -> rows of W packed columns.
template <typename T>
struct FactorJob {
  const T* src;
  int64_t sb, sh, ss;
  int S, W;
  float mult;
  bool vec;       // rows are whole, 16-byte aligned groups of 8 elements
  bool centered;  // the centred (hi, lo) copy instead of the factor itself
  T* dst;
  Div div_w8, div_s, div_h;  // divisions by W/8 (threads per row), S and Hx
  int64_t units;             // threads: rows x W/8
};
// One tensor scaled and split: (B, H, S, D) with strides -> (B, H, S, 2W) = [hi | lo] of x * scale, W >= D (zeros beyond).
template <typename T>
struct ScaledJob {
  const T* src;
  int64_t sb, sh, ss;
  int S, D, W;
  T* dst;
  Div div_w8, div_s, div_h;
  int64_t units;  // rows x W/8
};
// delta[bh, i] = sum_d o[i, d] * dout[i, d]: G threads per row
template <typename T>
struct DeltaJob {
  const T *o, *dout;
  int64_t o_st[3], do_st[3];
  int D, G, H;
  bool vec;
  float* delta;
  int64_t stride_bh;
  Div div_g, div_h, div_s;
  int64_t units;  // rows x G, head fastest
};

// One thread per 8 packed columns (one 16-byte store): consecutive threads write consecutive chunks of a row and read
// its elements side by side, so both sides coalesce whatever the rank (a thread per row took 26 us for the 3 x 1536 x 16
// rows of rank 32, all of it in serial, strided requests; this form 4).
template <typename T>
__device__ __forceinline__ void pack_factor_chunk(const FactorJob<T>& j, int64_t idx, int R, int* status) {
  if (idx >= j.units) return;
  const int64_t row = j.div_w8.quot(idx);
  const int c0 = (int)(idx - row * j.div_w8.d) * 8;
  const int64_t bh = j.div_s.quot(row);
  const int s = (int)(row - bh * j.S);
  const int64_t b = j.div_h.quot(bh);
  const int h = (int)(bh - b * j.div_h.d);
  const T* base = j.src + b * j.sb + h * j.sh;
  const T* in = base + (int64_t)s * j.ss;
  uint4 w = make_uint4(0u, 0u, 0u, 0u);
  T* y = reinterpret_cast<T*>(&w);
  if (!j.centered) {
    bool overflow = false;
    uint4 raw = make_uint4(0u, 0u, 0u, 0u);
    T* e = reinterpret_cast<T*>(&raw);
    if (j.vec) {
      if (c0 < R) raw = *reinterpret_cast<const uint4*>(in + c0);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (c0 + i < R) e[i] = in[c0 + i];
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (c0 + i < R) {
        const float x = to_f32(e[i]);
        y[i] = from_f32<T>(x * j.mult);  // mult is 1 or a power of two: exact unless it overflows
        overflow |= !isfinite(to_f32(y[i])) && isfinite(x);
      }
    }
    if (overflow && status) atomicExch(status, FB_DEV_FACTOR_OVERFLOW);
  } else {
    // k-side factor minus the factor of the middle key of its group of 32 keys: small-magnitude copy used
    // for dq_bias = dS.k_bias (the removed constant is re-applied in fp32 through the row sum of dS);
    // two-term split: columns [0,R) hi, [W/2, W/2 + R) lo, zero elsewhere
    const T* in0 = base + (int64_t)min((s & ~31) + 16, j.S - 1) * j.ss;
    const bool lo = c0 >= j.W / 2;
    const int cc0 = lo ? c0 - j.W / 2 : c0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int cc = cc0 + i;
      if (cc < R) {
        const float x = to_f32(in[cc]) - to_f32(in0[cc]);
        const T hi = from_f32<T>(x);
        y[i] = lo ? from_f32<T>(x - to_f32(hi)) : hi;
      }
    }
  }
  *reinterpret_cast<uint4*>(j.dst + row * j.W + c0) = w;
}

// ks[b][h][s][0:W] = T(x * scale), ks[b][h][s][W:2W] = T(x * scale - hi): the scaled key as two 16-bit terms.
// One thread converts 8 consecutive elements (16-byte load, two 16-byte stores).
template <typename T>
__device__ __forceinline__ void pack_scaled_chunk(const ScaledJob<T>& j, int64_t idx, float scale) {
  if (idx >= j.units) return;
  const int64_t row = j.div_w8.quot(idx);
  const int c = (int)(idx - row * j.div_w8.d) * 8;
  const int64_t bh = j.div_s.quot(row);
  const int s = (int)(row - bh * j.S);
  const int64_t b = j.div_h.quot(bh);
  const int h = (int)(bh - b * j.div_h.d);
  uint4 raw = make_uint4(0u, 0u, 0u, 0u);
  if (c < j.D) raw = *reinterpret_cast<const uint4*>(j.src + b * j.sb + h * j.sh + s * j.ss + c);
  const T* x = reinterpret_cast<const T*>(&raw);
  uint4 hi4, lo4;
  T* hi = reinterpret_cast<T*>(&hi4);
  T* lo = reinterpret_cast<T*>(&lo4);
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const float v = to_f32(x[e]) * scale;
    hi[e] = from_f32<T>(v);
    lo[e] = from_f32<T>(v - to_f32(hi[e]));
  }
  T* out = j.dst + row * (2 * j.W);
  *reinterpret_cast<uint4*>(out + c) = hi4;
  *reinterpret_cast<uint4*>(out + j.W + c) = lo4;
}

template <typename T>
__device__ __forceinline__ void delta_chunk(const DeltaJob<T>& j, int64_t idx) {
  const bool live = idx < j.units;
  float acc = 0.f;
  int64_t out = 0;
  int part = 0;
  if (live) {
    const int64_t row = j.div_g.quot(idx);  // (b, i, h), h fastest
    part = (int)(idx - row * j.G);
    const int64_t bi = j.div_h.quot(row);
    const int h = (int)(row - bi * j.H);
    const int64_t b = j.div_s.quot(bi);
    const int i = (int)(bi - b * j.div_s.d);
    const T* orow = j.o + b * j.o_st[0] + h * j.o_st[1] + i * j.o_st[2];
    const T* drow = j.dout + b * j.do_st[0] + h * j.do_st[1] + i * j.do_st[2];
    if (j.vec) {
      for (int d = part * 8; d < j.D; d += j.G * 8) {
        const uint4 a = *reinterpret_cast<const uint4*>(orow + d);
        const uint4 c = *reinterpret_cast<const uint4*>(drow + d);
        const T* pa = reinterpret_cast<const T*>(&a);
        const T* pc = reinterpret_cast<const T*>(&c);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc += to_f32(pa[e]) * to_f32(pc[e]);
      }
    } else {
      for (int d = part; d < j.D; d += j.G) acc += to_f32(orow[d]) * to_f32(drow[d]);
    }
    out = (b * j.H + h) * j.stride_bh + i;
  }
  for (int o = j.G >> 1; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);  // G: a power of two
  if (live && part == 0) j.delta[out] = acc;
}

// Everything a call needs before its main kernel, in one launch: block ranges pack the q-side factor, the k-side
// factor and its centred copy, split the scaled key (backward), take delta = rowsum(o * dout) and
// zero the fp32 accumulators (backward).  Three launches and a memset before; at small sizes each of them costs more in
// launch and drain than in work.
template <typename T>
struct PrepJobs {
  FactorJob<T> fq, fk, fc;
  ScaledJob<T> sc;
  DeltaJob<T> dl;
  uint4* zero;
  int64_t zero_vecs;                      // 16-byte units to clear
  unsigned end_q, end_k, end_c, end_s, end_d;  // exclusive block ranges, in this order; then the zeroing blocks
};
constexpr int kZeroPerThread = 4;

template <typename T>
__global__ void __launch_bounds__(256) prepare_operands_kernel(const __grid_constant__ PrepJobs<T> j, int R, float scale,
                                                               int* status) {
  grid_dep_launch();  // the main kernel may set itself up; it waits for this grid before it reads anything
  grid_dep_wait();    // (whatever produced the inputs)
  const unsigned blk = blockIdx.x;
  const int tid = threadIdx.x;
  if (blk < j.end_q) pack_factor_chunk<T>(j.fq, (int64_t)blk * 256 + tid, R, status);
  else if (blk < j.end_k) pack_factor_chunk<T>(j.fk, (int64_t)(blk - j.end_q) * 256 + tid, R, status);
  else if (blk < j.end_c) pack_factor_chunk<T>(j.fc, (int64_t)(blk - j.end_k) * 256 + tid, R, status);
  else if (blk < j.end_s) pack_scaled_chunk<T>(j.sc, (int64_t)(blk - j.end_c) * 256 + tid, scale);
  else if (blk < j.end_d) delta_chunk<T>(j.dl, (int64_t)(blk - j.end_s) * 256 + tid);
  else {
    const int64_t base = (int64_t)(blk - j.end_d) * (256 * kZeroPerThread) + tid;
#pragma unroll
    for (int i = 0; i < kZeroPerThread; ++i)
      if (base + i * 256 < j.zero_vecs) j.zero[base + i * 256] = make_uint4(0u, 0u, 0u, 0u);
  }
}

static unsigned blocks_for(int64_t units, int per_block = 256) { return (unsigned)((units + per_block - 1) / per_block); }

template <typename T>
static FactorJob<T> factor_job(const void* src, const int64_t* st, int Bx, int Hx, int S, int R, int W, float mult,
                               bool centered, void* dst) {
  FactorJob<T> j;
  j.src = reinterpret_cast<const T*>(src);
  j.sb = st[0]; j.sh = st[1]; j.ss = st[2];
  j.S = S; j.W = W;
  j.mult = mult;
  j.centered = centered;
  j.vec = R % 8 == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0 && !((st[0] | st[1] | st[2]) & 7);
  j.dst = reinterpret_cast<T*>(dst);
  j.div_w8 = Div(W / 8); j.div_s = Div(S); j.div_h = Div(Hx);
  j.units = (int64_t)Bx * Hx * S * (W / 8);
  return j;
}

template <typename T>
static int launch_prepare_t(const fb_params* p, const PackPlan& plan, const PrepBuffers& buf, cudaStream_t st) {
  PrepJobs<T> j{};
  unsigned n = 0;
  if (plan.RP) {
    j.fq = factor_job<T>(p->q_bias, p->q_bias_stride, plan.Bq, plan.Hq, p->Sq, p->R, plan.RP, plan.qb_mult, false, buf.qpack);
    j.fk = factor_job<T>(p->k_bias, p->k_bias_stride, plan.Bk, plan.Hk, p->Sk, p->R, plan.RP, 1.f, false, buf.kpack);
    if (buf.kcenter)
      j.fc = factor_job<T>(p->k_bias, p->k_bias_stride, plan.Bk, plan.Hk, p->Sk, p->R, plan.RC, 1.f, true, buf.kcenter);
  }
  j.end_q = n += blocks_for(j.fq.units);
  j.end_k = n += blocks_for(j.fk.units);
  j.end_c = n += blocks_for(j.fc.units);
  if (plan.nq == 2 && buf.scaled) {
    ScaledJob<T>& s = j.sc;
    s.src = reinterpret_cast<const T*>(p->k);
    s.sb = p->k_stride[0]; s.sh = p->k_stride[1]; s.ss = p->k_stride[2];
    s.S = p->Sk;
    s.D = p->D; s.W = plan.TD;
    s.dst = reinterpret_cast<T*>(buf.scaled);
    s.div_w8 = Div(plan.TD / 8); s.div_s = Div(s.S); s.div_h = Div(p->H);
    s.units = (int64_t)p->B * p->H * s.S * (plan.TD / 8);
  }
  j.end_s = n += blocks_for(j.sc.units);
  if (buf.delta) {
    DeltaJob<T>& d = j.dl;
    d.o = reinterpret_cast<const T*>(p->o);
    d.dout = reinterpret_cast<const T*>(p->dout);
    uintptr_t bits = reinterpret_cast<uintptr_t>(p->o) | reinterpret_cast<uintptr_t>(p->dout);
    for (int i = 0; i < 3; ++i) {
      d.o_st[i] = p->o_stride[i];
      d.do_st[i] = p->dout_stride[i];
      bits |= (uintptr_t)(p->o_stride[i] | p->dout_stride[i]) * 2;
    }
    d.D = p->D; d.H = p->H;
    d.vec = p->D % 8 == 0 && (bits & 15) == 0;
    // as many threads per row as it has 16-byte chunks, as far as that is a power of two (shuffle groups)
    d.G = 1;
    if (d.vec)
      while (d.G < 16 && (p->D / 8) % (2 * d.G) == 0) d.G *= 2;
    d.delta = buf.delta;
    d.stride_bh = p->lse_stride_bh;
    d.div_g = Div(d.G); d.div_h = Div(p->H); d.div_s = Div(p->Sq);
    d.units = (int64_t)p->B * p->Sq * p->H * d.G;
  }
  j.end_d = n += blocks_for(j.dl.units);
  j.zero = reinterpret_cast<uint4*>(buf.zero);
  j.zero_vecs = (int64_t)(buf.zero_bytes / 16);
  n += blocks_for(j.zero_vecs, 256 * kZeroPerThread);
  if (n == 0) return 0;
  return launch_pdl(prepare_operands_kernel<T>, n, 256, 0, st, j, (int)p->R, (float)p->softmax_scale, p->status);
}

int launch_prepare(const fb_params* p, const PackPlan& plan, const PrepBuffers& buf, cudaStream_t st) {
  return p->dtype == FB_DTYPE_F16 ? launch_prepare_t<__half>(p, plan, buf, st)
                                  : launch_prepare_t<__nv_bfloat16>(p, plan, buf, st);
}

// delta alone (the separate pre-pass of the C ABI)
int launch_bwd_preprocess(const fb_params* p, cudaStream_t st) {
  PackPlan none{};
  none.nq = 1;
  PrepBuffers buf{};
  buf.delta = p->delta;
  prof_before(KC_BWD_PREPROCESS, st);
  const int rc = launch_prepare(p, none, buf, st);
  prof_after(KC_BWD_PREPROCESS, st);
  return rc;
}

}  // namespace fb
