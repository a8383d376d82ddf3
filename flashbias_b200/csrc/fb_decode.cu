// Forward for a single query row per (batch, head): token generation against a key/value cache.
//
// Bound by reading K and V once from HBM (2 x Sk x D 16-bit values per (batch, head)); there is nothing to contract that
// a tensor-core tile of 128 query rows would not spend 127 rows of padding on, and a CTA per (batch, head) leaves most
// of the loads serial.  Here a group of G = D/8 lanes owns one head: each lane reads 16 bytes of a key's row and of its
// value's row, the group's dot product is closed with shuffles, and every lane keeps 8 columns of the output.  The lanes
// of a CTA cover neighbouring heads of the same key, so that a (B, S, H, D) cache is read as whole contiguous rows; the
// keys are split over enough CTAs to fill the GPU once, and a second small kernel merges the splits.  All arithmetic is
// fp32 on the given 16-bit values (probabilities are not rounded), and no operand is packed.
// B16 H50 Sk5001 D32 R2: 233 us with the tiled kernel (2.2 TB/s).
#include "fb_common.cuh"
#include "fb_internal.h"

namespace fb {

struct DecodeArgs {
  const void *q, *k, *v, *q_bias, *k_bias, *mask;
  int64_t q_st[2], k_st[3], v_st[3], qb_st[2], kb_st[3], mask_st[2], o_st[2];  // (batch, head[, row])
  void* o;
  float* lse;
  int64_t lse_stride_bh;
  int H, Sk, D, R;       // Sk: visible keys
  int hg, nhg, kp;       // heads per CTA, head groups, keys a CTA visits side by side
  int nsplit, per_split;  // key ranges per (batch, head group), keys in one
  float scale_log2;
  int mask_dtype, mask_batch_period;
  const float* alibi_slopes;
  float* part_acc;  // (B, H, nsplit, 8 G), when nsplit > 1
  float2* part_ml;  // (B, H, nsplit): maximum (log2 units) and sum
};

constexpr int kDecodeThreads = 256;
constexpr int kDecodeUnroll = 4;  // keys in flight per lane
constexpr float kLog2eD = 1.4426950408889634f;
constexpr float kLn2D = 0.6931471805599453f;

template <typename T>
__device__ __forceinline__ void unpack8(const uint4& raw, float (&x)[8]) {
  const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
  for (int i = 0; i < 8; ++i) x[i] = to_f32(e[i]);
}

template <typename T>
__device__ __forceinline__ void store_row8(const DecodeArgs& a, int b, int h, int d0, const float (&acc)[8], float inv) {
  uint4 w;
  w.x = Pack2<T>::pack(acc[0] * inv, acc[1] * inv);
  w.y = Pack2<T>::pack(acc[2] * inv, acc[3] * inv);
  w.z = Pack2<T>::pack(acc[4] * inv, acc[5] * inv);
  w.w = Pack2<T>::pack(acc[6] * inv, acc[7] * inv);
  *reinterpret_cast<uint4*>(reinterpret_cast<T*>(a.o) + b * a.o_st[0] + h * a.o_st[1] + d0) = w;
}

// G lanes per head, NRS bias columns per lane (rank <= G * NRS)
template <typename T, int G, int NRS>
__global__ void __launch_bounds__(kDecodeThreads, 3) decode_kernel(const DecodeArgs a) {
  __shared__ float s_acc[kDecodeThreads * 8];
  __shared__ float2 s_ml[kDecodeThreads];
  grid_dep_wait();
  const int split = blockIdx.x % a.nsplit, hgi = (blockIdx.x / a.nsplit) % a.nhg, b = blockIdx.x / (a.nsplit * a.nhg);
  const int unit = threadIdx.x / G, part = threadIdx.x % G;
  const int kl = unit / a.hg, hl = unit - kl * a.hg, h = hgi * a.hg + hl;
  const bool live = kl < a.kp && h < a.H;
  const bool cols = live && part * 8 < a.D;  // (a group is a power of two wide, a row may be shorter)
  const int k_end = min(a.Sk, (split + 1) * a.per_split);

  float qv[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, qb[NRS ? NRS : 1] = {};
  float slope2 = 0.f;
  const T *kp_ = nullptr, *vp_ = nullptr, *kbp = nullptr;
  const char* mp = nullptr;
  if (live) {
    if (cols) {
      unpack8<T>(*reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(a.q) + b * a.q_st[0] + h * a.q_st[1] + part * 8), qv);
#pragma unroll
      for (int i = 0; i < 8; ++i) qv[i] *= a.scale_log2;
    }
    kp_ = reinterpret_cast<const T*>(a.k) + b * a.k_st[0] + h * a.k_st[1] + part * 8;
    vp_ = reinterpret_cast<const T*>(a.v) + b * a.v_st[0] + h * a.v_st[1] + part * 8;
    if (NRS) {
      const T* src = reinterpret_cast<const T*>(a.q_bias) + b * a.qb_st[0] + h * a.qb_st[1];
      kbp = reinterpret_cast<const T*>(a.k_bias) + b * a.kb_st[0] + h * a.kb_st[1];
#pragma unroll
      for (int r = 0; r < NRS; ++r)
        if (part + r * G < a.R) qb[r] = to_f32(src[part + r * G]) * kLog2eD;
    }
    if (a.alibi_slopes) slope2 = a.alibi_slopes[h] * kLog2eD;
    if (a.mask) {
      const int mb = a.mask_batch_period > 0 ? b % a.mask_batch_period : b;
      mp = reinterpret_cast<const char*>(a.mask) +
           (mb * a.mask_st[0] + h * a.mask_st[1]) * (a.mask_dtype == FB_DTYPE_F32 ? 4 : 2);
    }
  }

  float m = -INFINITY, l = 0.f, acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  // every lane of a warp runs the same number of rounds (the shuffles need all of them)
  for (int k0 = split * a.per_split; k0 < k_end; k0 += a.kp * kDecodeUnroll) {
    uint4 kr[kDecodeUnroll], vr[kDecodeUnroll];
    float s[kDecodeUnroll];
#pragma unroll
    for (int u = 0; u < kDecodeUnroll; ++u) {
      const int key = k0 + u * a.kp + kl;
      kr[u] = vr[u] = make_uint4(0u, 0u, 0u, 0u);
      s[u] = 0.f;
      if (cols && key < k_end) {
        kr[u] = __ldg(reinterpret_cast<const uint4*>(kp_ + (int64_t)key * a.k_st[2]));
        vr[u] = __ldg(reinterpret_cast<const uint4*>(vp_ + (int64_t)key * a.v_st[2]));
      }
      if (NRS && live && key < k_end) {
#pragma unroll
        for (int r = 0; r < NRS; ++r)
          if (part + r * G < a.R) s[u] = fmaf(qb[r], to_f32(kbp[(int64_t)key * a.kb_st[2] + part + r * G]), s[u]);
      }
    }
    float mx = m;
#pragma unroll
    for (int u = 0; u < kDecodeUnroll; ++u) {
      const int key = k0 + u * a.kp + kl;
      float x[8];
      unpack8<T>(kr[u], x);
#pragma unroll
      for (int i = 0; i < 8; ++i) s[u] = fmaf(qv[i], x[i], s[u]);
#pragma unroll
      for (int o = G / 2; o; o >>= 1) s[u] += __shfl_xor_sync(0xffffffffu, s[u], o);
      s[u] = fmaf(slope2, (float)key, s[u]);
      if (mp && key < k_end)
        s[u] += kLog2eD * (a.mask_dtype == FB_DTYPE_F32   ? reinterpret_cast<const float*>(mp)[key]
                           : a.mask_dtype == FB_DTYPE_F16 ? __half2float(reinterpret_cast<const __half*>(mp)[key])
                                                          : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(mp)[key]));
      if (key >= k_end) s[u] = -INFINITY;
      mx = fmaxf(mx, s[u]);
    }
    const float msub = mx == -INFINITY ? 0.f : mx;
    const float alpha = fast_exp2(m - msub);  // 0 while m is still -inf
    m = mx;
    l *= alpha;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] *= alpha;
#pragma unroll
    for (int u = 0; u < kDecodeUnroll; ++u) {
      const float p = fast_exp2(s[u] - msub);
      float x[8];
      unpack8<T>(vr[u], x);
      l += p;
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = fmaf(p, x[i], acc[i]);
    }
  }

  if (a.kp > 1) {  // merge the keys visited side by side
    s_ml[threadIdx.x] = make_float2(m, l);
#pragma unroll
    for (int i = 0; i < 8; ++i) s_acc[i * kDecodeThreads + threadIdx.x] = acc[i];
    __syncthreads();
    if (!live || kl > 0) return;
    for (int j = 1; j < a.kp; ++j) {
      const int t = threadIdx.x + j * a.hg * G;
      const float2 o = s_ml[t];
      const float mn = fmaxf(m, o.x), ms = mn == -INFINITY ? 0.f : mn;
      const float fa = fast_exp2(m - ms), fb = fast_exp2(o.x - ms);
      m = mn;
      l = l * fa + o.y * fb;
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = acc[i] * fa + s_acc[i * kDecodeThreads + t] * fb;
    }
  } else if (!live) {
    return;
  }
  const int64_t bh = (int64_t)b * a.H + h;
  if (a.nsplit == 1) {
    if (cols) store_row8<T>(a, b, h, part * 8, acc, l > 0.f ? 1.f / l : 0.f);
    if (part == 0) a.lse[bh * a.lse_stride_bh] = l > 0.f ? (m + fast_log2(l)) * kLn2D : -INFINITY;
  } else {
    float4* dst = reinterpret_cast<float4*>(a.part_acc + (bh * a.nsplit + split) * (8 * G) + part * 8);
    dst[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
    dst[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
    if (part == 0) a.part_ml[bh * a.nsplit + split] = make_float2(m, l);
  }
}

// One block per (batch, head): G lanes x 8 columns, the splits spread over the other threads.
template <typename T, int G>
__global__ void __launch_bounds__(128) decode_merge_kernel(const DecodeArgs a) {
  constexpr int LANES = 128 / G;
  __shared__ float s_acc[128 * 9];
  __shared__ float s_m[4], s_l[LANES];
  grid_dep_wait();
  const int64_t bh = blockIdx.x;
  const int sl = threadIdx.x / G, part = threadIdx.x % G;
  const float2* ml = a.part_ml + bh * a.nsplit;
  float m = -INFINITY;
  for (int s = threadIdx.x; s < a.nsplit; s += 128) m = fmaxf(m, ml[s].x);
#pragma unroll
  for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) s_m[threadIdx.x >> 5] = m;
  __syncthreads();
  m = fmaxf(fmaxf(s_m[0], s_m[1]), fmaxf(s_m[2], s_m[3]));
  const float ms = m == -INFINITY ? 0.f : m;
  float l = 0.f, acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
  for (int s = sl; s < a.nsplit; s += LANES) {
    const float2 e = ml[s];
    const float f = fast_exp2(e.x - ms);
    const float4* src = reinterpret_cast<const float4*>(a.part_acc + (bh * a.nsplit + s) * (8 * G) + part * 8);
    const float4 x = src[0], y = src[1];
    l = fmaf(e.y, f, l);
    acc[0] = fmaf(x.x, f, acc[0]); acc[1] = fmaf(x.y, f, acc[1]); acc[2] = fmaf(x.z, f, acc[2]); acc[3] = fmaf(x.w, f, acc[3]);
    acc[4] = fmaf(y.x, f, acc[4]); acc[5] = fmaf(y.y, f, acc[5]); acc[6] = fmaf(y.z, f, acc[6]); acc[7] = fmaf(y.w, f, acc[7]);
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) s_acc[threadIdx.x * 9 + i] = acc[i];
  if (part == 0) s_l[sl] = l;
  __syncthreads();
  if (sl > 0) return;
  l = 0.f;
  for (int j = 0; j < LANES; ++j) l += s_l[j];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    acc[i] = 0.f;
    for (int j = 0; j < LANES; ++j) acc[i] += s_acc[(j * G + part) * 9 + i];
  }
  const int b = (int)(bh / a.H), h = (int)(bh % a.H);
  if (part * 8 < a.D) store_row8<T>(a, b, h, part * 8, acc, l > 0.f ? 1.f / l : 0.f);
  if (part == 0) a.lse[bh * a.lse_stride_bh] = l > 0.f ? (m + fast_log2(l)) * kLn2D : -INFINITY;
}

// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------
namespace {
struct DecodePlan {
  int G, NRS, hg, nhg, kp, nsplit, per_split, Sk;
  size_t acc_bytes, ml_bytes;
};

DecodePlan plan_decode(const fb_params* p) {
  DecodePlan d;
  d.G = p->D <= 8 ? 1 : p->D <= 16 ? 2 : p->D <= 32 ? 4 : p->D <= 64 ? 8 : 16;
  const int need = (p->R + d.G - 1) / d.G;
  d.NRS = need <= 1 ? need : need <= 4 ? 4 : 16;
  d.Sk = p->causal ? 1 : p->Sk;
  // all heads in one CTA if they fit, else the smallest number of equal groups
  const int fit = kDecodeThreads / d.G;
  d.nhg = (p->H + fit - 1) / fit;
  d.hg = (p->H + d.nhg - 1) / d.nhg;
  d.kp = fit / d.hg;
  // as many key ranges as fill the resident CTA slots (3 per SM) once, none shorter than 8 rounds
  int dev = 0;
  cudaGetDevice(&dev);
  const int slots = 3 * (device_sm_count(dev) > 0 ? device_sm_count(dev) : 148);
  const int64_t ctas = (int64_t)p->B * d.nhg;
  int64_t ns = slots / ctas;
  const int64_t most = (d.Sk + (int64_t)d.kp * kDecodeUnroll * 8 - 1) / ((int64_t)d.kp * kDecodeUnroll * 8);
  if (ns > most) ns = most;
  if (ns < 1) ns = 1;
  const int round = d.kp * kDecodeUnroll;
  d.per_split = (int)((d.Sk + ns - 1) / ns);
  d.per_split = (d.per_split + round - 1) / round * round;
  d.nsplit = (d.Sk + d.per_split - 1) / d.per_split;
  d.acc_bytes = d.nsplit > 1 ? round256((size_t)p->B * p->H * d.nsplit * 8 * d.G * 4) : 0;
  d.ml_bytes = d.nsplit > 1 ? round256((size_t)p->B * p->H * d.nsplit * 8) : 0;
  return d;
}

template <typename T, int G>
int launch_decode_g(const DecodeArgs& a, const DecodePlan& d, int B, cudaStream_t st) {
  const unsigned grid = (unsigned)((int64_t)B * d.nhg * d.nsplit);
  prof_before(KC_FWD_MAIN, st);
  int rc = FB_ENOTBUILT;
  switch (d.NRS) {
    case 0: rc = launch_pdl(decode_kernel<T, G, 0>, grid, kDecodeThreads, 0, st, a); break;
    case 1: rc = launch_pdl(decode_kernel<T, G, 1>, grid, kDecodeThreads, 0, st, a); break;
    case 4: rc = launch_pdl(decode_kernel<T, G, 4>, grid, kDecodeThreads, 0, st, a); break;
    case 16: rc = launch_pdl(decode_kernel<T, G, 16>, grid, kDecodeThreads, 0, st, a); break;
  }
  prof_after(KC_FWD_MAIN, st);
  if (rc || d.nsplit == 1) return rc;
  return launch_pdl(decode_merge_kernel<T, G>, (unsigned)(B * a.H), 128, 0, st, a);
}

template <typename T>
int launch_decode_t(const DecodeArgs& a, const DecodePlan& d, int B, cudaStream_t st) {
  switch (d.G) {
    case 1: return launch_decode_g<T, 1>(a, d, B, st);
    case 2: return launch_decode_g<T, 2>(a, d, B, st);
    case 4: return launch_decode_g<T, 4>(a, d, B, st);
    case 8: return launch_decode_g<T, 8>(a, d, B, st);
    case 16: return launch_decode_g<T, 16>(a, d, B, st);
  }
  return FB_ENOTBUILT;
}
}  // namespace

// One query row, rows of whole aligned 16-byte chunks, and a rank that a group of lanes can hold.  With two or more query
// rows every key would be read from L1 / L2 once per row, and the tiled kernel starts to amortise its loads.
bool decode_supported(const fb_params* p) {
  if ((p->flags & FB_FLAG_FORCE_GENERAL) || p->Sq != 1 || p->D % 8 != 0) return false;
  uintptr_t bits = reinterpret_cast<uintptr_t>(p->q) | reinterpret_cast<uintptr_t>(p->k) |
                   reinterpret_cast<uintptr_t>(p->v) | reinterpret_cast<uintptr_t>(p->o);
  for (int i = 0; i < 3; ++i) {
    bits |= (uintptr_t)(p->k_stride[i] | p->v_stride[i]) * 2;
    if (i < 2) bits |= (uintptr_t)(p->q_stride[i] | p->o_stride[i]) * 2;
  }
  if (bits & 15) return false;
  const int G = p->D <= 8 ? 1 : p->D <= 16 ? 2 : p->D <= 32 ? 4 : p->D <= 64 ? 8 : 16;
  return p->R <= 16 * G && (int64_t)p->B * p->H <= 0x7fffffffLL / 1024;
}

size_t decode_workspace(const fb_params* p) {
  const DecodePlan d = plan_decode(p);
  return d.acc_bytes + d.ml_bytes;
}

int launch_decode(const fb_params* p, cudaStream_t st) {
  const DecodePlan d = plan_decode(p);
  DecodeArgs a = {};
  a.q = p->q; a.k = p->k; a.v = p->v; a.q_bias = p->q_bias; a.k_bias = p->k_bias; a.mask = p->mask;
  for (int i = 0; i < 3; ++i) {
    a.k_st[i] = p->k_stride[i];
    a.v_st[i] = p->v_stride[i];
    a.kb_st[i] = p->k_bias_stride[i];
    if (i < 2) {
      a.q_st[i] = p->q_stride[i];
      a.qb_st[i] = p->q_bias_stride[i];
      a.mask_st[i] = p->mask_stride[i];
      a.o_st[i] = p->o_stride[i];
    }
  }
  a.o = p->o;
  a.lse = p->lse;
  a.lse_stride_bh = p->lse_stride_bh;
  a.H = p->H; a.Sk = d.Sk; a.D = p->D; a.R = p->R;
  a.hg = d.hg; a.nhg = d.nhg; a.kp = d.kp;
  a.nsplit = d.nsplit; a.per_split = d.per_split;
  a.scale_log2 = p->softmax_scale * kLog2eD;
  a.mask_dtype = p->mask_dtype;
  a.mask_batch_period = p->mask_batch_period;
  a.alibi_slopes = p->alibi_slopes;
  a.part_acc = reinterpret_cast<float*>(p->workspace);
  a.part_ml = reinterpret_cast<float2*>(reinterpret_cast<uint8_t*>(p->workspace) + d.acc_bytes);
  return p->dtype == FB_DTYPE_F16 ? launch_decode_t<__half>(a, d, p->B, st) : launch_decode_t<__nv_bfloat16>(a, d, p->B, st);
}

}  // namespace fb
