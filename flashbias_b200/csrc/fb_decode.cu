// Forward for a single query row per (batch, head): token generation against a key/value cache.
//
// Bound by reading K and V once from HBM (2 x Sk x D 16-bit values per (batch, head)); there is nothing to contract that
// a tensor-core tile of 128 query rows would not spend 127 rows of padding on, and a CTA per (batch, head) leaves most
// of the loads serial.  Here a group of G = D/8 lanes owns one head: each lane reads 16 bytes of a key's row and of its
// value's row, the group's dot product is closed with shuffles, and every lane keeps 8 columns of the output.  The lanes
// of a CTA cover neighbouring heads of the same key, so that a (B, S, H, D) cache is read as whole contiguous rows; the
// keys are split over enough CTAs to fill the GPU once, and a second small kernel merges the splits.  All arithmetic is
// fp32 on the given 16-bit values (probabilities are not rounded), and no operand is packed.
// B16 H50 Sk5001 D32 R2: 233 us a call with the tiled kernel (2.2 TB/s), 87 to 91 us here (5.6 to 5.9 TB/s; 85 us of it this
// kernel; 124 us when the rounds in flight were held in registers, 92 us with 3 CTAs and rounds of 2 keys).
#include <float.h>

#include <mutex>
#include <type_traits>

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
constexpr int kDecodeUnroll = 4;  // keys of a round
constexpr int kDecodeDepth = 3;   // rounds in the ring
constexpr int kDecodeCtas = 2;    // resident per SM
constexpr int kDecodeRing = kDecodeDepth * kDecodeUnroll * 2 * kDecodeThreads * 16;
constexpr float kLog2eD = 1.4426950408889634f;
constexpr float kLn2D = 0.6931471805599453f;

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ uint4 ld_shared_v4u(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}

// 8 consecutive 16-bit values as fp32 pairs
template <typename T>
__device__ __forceinline__ void unpack8(const uint4& raw, uint64_t (&x)[4]) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (std::is_same<T, __nv_bfloat16>::value) {
      x[i] = f2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
    } else {
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
      x[i] = f2(f.x, f.y);
    }
  }
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

// G lanes per head, NRS bias columns per lane (rank <= G * NRS); EXTRA: a mask or slopes complete the logits
template <typename T, int G, int NRS, bool EXTRA>
__global__ void __launch_bounds__(kDecodeThreads, kDecodeCtas) decode_kernel(const DecodeArgs a) {
  grid_dep_wait();
  const int split = blockIdx.x % a.nsplit, hgi = (blockIdx.x / a.nsplit) % a.nhg, b = blockIdx.x / (a.nsplit * a.nhg);
  const int unit = threadIdx.x / G, part = threadIdx.x % G;
  const int kl = unit / a.hg, hl = unit - kl * a.hg, h = hgi * a.hg + hl;
  const bool live = kl < a.kp && h < a.H;
  const bool cols = live && part * 8 < a.D;  // (a group is a power of two wide, a row may be shorter)
  const int k_end = min(a.Sk, (split + 1) * a.per_split);

  float qv[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, qb[NRS ? NRS : 1] = {};
  float slope2 = 0.f;
  const T *kp_ = reinterpret_cast<const T*>(a.k), *vp_ = reinterpret_cast<const T*>(a.v);
  const T* kbp = reinterpret_cast<const T*>(a.k_bias);
  const char* mp = nullptr;
  if (live) {
    if (cols) {
      uint64_t x[4];
      unpack8<T>(*reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(a.q) + b * a.q_st[0] + h * a.q_st[1] + part * 8), x);
#pragma unroll
      for (int i = 0; i < 4; ++i) f2_unpack(f2_mul(x[i], f2(a.scale_log2, a.scale_log2)), qv[2 * i], qv[2 * i + 1]);
    }
    kp_ += b * a.k_st[0] + h * a.k_st[1] + (cols ? part * 8 : 0);
    vp_ += b * a.v_st[0] + h * a.v_st[1] + (cols ? part * 8 : 0);
    if (NRS) {
      const T* src = reinterpret_cast<const T*>(a.q_bias) + b * a.qb_st[0] + h * a.qb_st[1];
      kbp += b * a.kb_st[0] + h * a.kb_st[1];
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

  // Each lane copies its own 16-byte chunks of K and V into its own slots of a shared-memory ring, a few rounds ahead of
  // their use: what is in flight is then bounded by shared memory (2 CTAs x 96 KB) and not by registers, and no
  // synchronisation is needed, since only the lane that copied a chunk reads it.
  extern __shared__ uint4 ring[];  // [kDecodeDepth][kDecodeUnroll][K, V][thread]
  const uint32_t slot0 = smem_u32(ring + threadIdx.x);
  constexpr uint32_t kChunk = kDecodeThreads * 16, kRound = 2 * kDecodeUnroll * kChunk;
  const int step = a.kp * kDecodeUnroll;
  const int k_begin = split * a.per_split;
  const int64_t ks = (int64_t)a.kp * a.k_st[2], vs = (int64_t)a.kp * a.v_st[2], bs = (int64_t)a.kp * a.kb_st[2];
  const T* kf = kp_ + (int64_t)(k_begin + kl) * a.k_st[2];
  const T* vf = vp_ + (int64_t)(k_begin + kl) * a.v_st[2];
  const T* bf = kbp + (NRS ? (int64_t)(k_begin + kl) * a.kb_st[2] + part : 0);
  int key_f = k_begin + kl;  // key of the first copy of the next round to fetch
  auto fetch = [&](uint32_t slot) {
#pragma unroll
    for (int u = 0; u < kDecodeUnroll; ++u) {
      const uint32_t bytes = cols && key_f + u * a.kp < k_end ? 16u : 0u;  // beyond the range: zeros, nothing is read
      cp_async16(slot + 2 * u * kChunk, bytes ? kf + u * ks : kp_, bytes);
      cp_async16(slot + (2 * u + 1) * kChunk, bytes ? vf + u * vs : vp_, bytes);
    }
    key_f += step;
    kf += kDecodeUnroll * ks;
    vf += kDecodeUnroll * vs;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  T kb[kDecodeUnroll][NRS ? NRS : 1];
  int key_b = k_begin + kl;
  auto fetch_bias = [&] {
    if constexpr (NRS > 0) {
#pragma unroll
      for (int u = 0; u < kDecodeUnroll; ++u) {
#pragma unroll
        for (int c = 0; c < NRS; ++c)
          kb[u][c] = live && key_b + u * a.kp < k_end && part + c * G < a.R ? bf[u * bs + c * G] : from_f32<T>(0.f);
      }
      key_b += step;
      bf += kDecodeUnroll * bs;
    }
  };
  float m = -INFINITY, l = 0.f;
  uint64_t acc2[4] = {0ull, 0ull, 0ull, 0ull};
  const uint64_t q2[4] = {f2(qv[0], qv[1]), f2(qv[2], qv[3]), f2(qv[4], qv[5]), f2(qv[6], qv[7])};
#pragma unroll
  for (int i = 0; i < kDecodeDepth - 1; ++i) fetch(slot0 + i * kRound);
  fetch_bias();
  uint32_t rs = 0, fs = (kDecodeDepth - 1) * kRound;  // ring offsets read and filled next
  for (int k0 = k_begin; k0 < k_end; k0 += step) {    // (the same number of rounds for every lane: the shuffles need all)
    fetch(slot0 + fs);
    fs = fs + kRound == kDecodeDepth * kRound ? 0 : fs + kRound;
    float s[kDecodeUnroll], mx = m;
    if constexpr (NRS > 0) {
#pragma unroll
      for (int u = 0; u < kDecodeUnroll; ++u) {
        s[u] = 0.f;
#pragma unroll
        for (int c = 0; c < NRS; ++c) s[u] = fmaf(qb[c], to_f32(kb[u][c]), s[u]);
      }
      fetch_bias();
    }
    asm volatile("cp.async.wait_group %0;" ::"n"(kDecodeDepth - 1) : "memory");
#pragma unroll
    for (int u = 0; u < kDecodeUnroll; ++u) {
      uint64_t x[4];
      unpack8<T>(ld_shared_v4u(slot0 + rs + 2 * u * kChunk), x);
      uint64_t t = f2_mul(q2[0], x[0]), w = f2_mul(q2[1], x[1]);
      t = f2_fma(q2[2], x[2], t);
      w = f2_fma(q2[3], x[3], w);
      float t0, t1;
      f2_unpack(f2_add(t, w), t0, t1);
      s[u] = NRS ? s[u] + (t0 + t1) : t0 + t1;
#pragma unroll
      for (int o = G / 2; o; o >>= 1) s[u] += __shfl_xor_sync(0xffffffffu, s[u], o);
      const int key = k0 + u * a.kp + kl;
      if (EXTRA) {
        s[u] = fmaf(slope2, (float)key, s[u]);
        if (mp && key < k_end)
          s[u] += kLog2eD * (a.mask_dtype == FB_DTYPE_F32   ? reinterpret_cast<const float*>(mp)[key]
                             : a.mask_dtype == FB_DTYPE_F16 ? __half2float(reinterpret_cast<const __half*>(mp)[key])
                                                            : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(mp)[key]));
      }
      if (key >= k_end) s[u] = -INFINITY;
      mx = fmaxf(mx, s[u]);
    }
    const float msub = fmaxf(mx, -FLT_MAX);  // no visible key yet: every exponential below is zero
    const float alpha = fast_exp2(m - msub);  // 0 while m is still -inf
    m = mx;
    l *= alpha;
    const uint64_t alpha2 = f2(alpha, alpha);
#pragma unroll
    for (int i = 0; i < 4; ++i) acc2[i] = f2_mul(acc2[i], alpha2);
#pragma unroll
    for (int u = 0; u < kDecodeUnroll; ++u) {
      const float p = fast_exp2(s[u] - msub);
      l += p;
      const uint64_t p2 = f2(p, p);
      uint64_t x[4];
      unpack8<T>(ld_shared_v4u(slot0 + rs + (2 * u + 1) * kChunk), x);
#pragma unroll
      for (int i = 0; i < 4; ++i) acc2[i] = f2_fma(p2, x[i], acc2[i]);
    }
    rs = rs + kRound == kDecodeDepth * kRound ? 0 : rs + kRound;
  }
  float acc[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) f2_unpack(acc2[i], acc[2 * i], acc[2 * i + 1]);

  if (a.kp > 1) {  // merge the keys visited side by side, in the ring's memory
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    float* s_acc = reinterpret_cast<float*>(ring);
    float2* s_ml = reinterpret_cast<float2*>(s_acc + 8 * kDecodeThreads);
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
#pragma unroll 4
  for (int j = 0; j < LANES; ++j) l += s_l[j];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    acc[i] = 0.f;
#pragma unroll 4
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
  d.NRS = need <= 1 ? need : 4;
  d.Sk = p->causal ? 1 : p->Sk;
  // all heads in one CTA if they fit, else the smallest number of equal groups
  const int fit = kDecodeThreads / d.G;
  d.nhg = (p->H + fit - 1) / fit;
  d.hg = (p->H + d.nhg - 1) / d.nhg;
  d.kp = fit / d.hg;
  // The largest number of key ranges with which all CTAs are resident at once, none shorter than 8 rounds.  Rounded down: where
  // it does not divide, slots stay empty, up to half of them just above one CTA per SM (rates per call, 296 slots: B37 H16
  // Sk5000 D128, 296 used, 6.6 TB/s; B25 H50 Sk5001 D128, 200 used, 5.5; B148 H16 Sk2000 D128, 296 used, 6.6; B149, 149 used,
  // 5.4; B149 H50 Sk1000 D32, 149 used, 4.1).
  int dev = 0;
  cudaGetDevice(&dev);
  const int slots = kDecodeCtas * (device_sm_count(dev) > 0 ? device_sm_count(dev) : 148);
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

template <typename T, int G, int NRS>
int launch_decode_n(const DecodeArgs& a, unsigned grid, cudaStream_t st) {
  auto kern = a.mask || a.alibi_slopes ? decode_kernel<T, G, NRS, true> : decode_kernel<T, G, NRS, false>;
  static std::mutex mu;
  static bool attr_done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  {
    std::lock_guard<std::mutex> lk(mu);
    if (!attr_done[dev & 63]) {
      cudaError_t e = cudaFuncSetAttribute(decode_kernel<T, G, NRS, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kDecodeRing);
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(decode_kernel<T, G, NRS, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kDecodeRing);
      if (e != cudaSuccess) return (int)e;
      attr_done[dev & 63] = true;
    }
  }
  return launch_pdl(kern, grid, kDecodeThreads, kDecodeRing, st, a);
}

template <typename T, int G>
int launch_decode_g(const DecodeArgs& a, const DecodePlan& d, int B, cudaStream_t st) {
  const unsigned grid = (unsigned)((int64_t)B * d.nhg * d.nsplit);
  prof_before(KC_FWD_MAIN, st);
  int rc = FB_ENOTBUILT;
  switch (d.NRS) {
    case 0: rc = launch_decode_n<T, G, 0>(a, grid, st); break;
    case 1: rc = launch_decode_n<T, G, 1>(a, grid, st); break;
    case 4: rc = launch_decode_n<T, G, 4>(a, grid, st); break;
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
  return p->R <= 4 * G && (int64_t)p->B * p->H <= 0x7fffffffLL / 1024;
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
