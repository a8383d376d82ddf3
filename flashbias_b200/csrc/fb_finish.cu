// After a backward main kernel: dq and the factor gradients leave their fp32 accumulators, in one launch.
// HBM-bound where it is large (4.8 GB for the 4096-window shape: 0.88 ms, 5.5 TB/s), launch-bound where it is small.
#include "fb_common.cuh"
#include "fb_internal.h"

namespace fb {

// dq = T(scale * acc), 8 consecutive d per thread; arrangements of the accumulator: see DQ_*.
template <typename T>
struct DqStoreJob {
  const float* acc;
  T* dq;
  int cols, H, Sq, layout;
  int64_t sb, sh, ss;
  float scale;
  Div div_d8, div_h, div_s;
  int64_t units;
};

// One factor gradient: fp32 accumulator -> 16-bit tensor with the factor's own strides.  The accumulator is
// (Bx, S, Hx, R), or -- `tiled` -- head-major in tiles of 128 rows stored rank-major, [r][row in tile] (the tensor-core
// backward stages its tiles that way: consecutive rows are consecutive floats, which keeps the threads' shared-memory
// stores free of bank conflicts); `slots` copies at distance `slot_stride` are summed.
// A block takes 128 rows x up to kRanks ranks: the tiled accumulator is read along its rows and turned in shared
// memory, so that reads and writes both coalesce (a thread per output element, rank fastest, read 4 bytes of a 32-byte
// sector: 17 us for 2 x 1536 x 16 rows of rank 32).
constexpr int kRanks = 8;
template <typename T>
struct FactorStoreJob {
  const float* acc;
  T* out;
  int Bx, S, Hx, R, tiled, slots, tiles, rchunks;
  int64_t slot_stride, sb, sh, ss;
};

template <typename T>
__device__ __forceinline__ void store_factor_block(const FactorStoreJob<T>& j, unsigned blk, float (&turn)[kRanks][132]) {
  const int rch = (int)(blk % j.rchunks);
  const int tile = (int)((blk / j.rchunks) % j.tiles);
  const int bh = (int)(blk / (j.rchunks * j.tiles));
  const int b = bh / j.Hx, h = bh % j.Hx;
  const int r0 = rch * kRanks, rc = min(kRanks, j.R - r0), s0 = tile * 128, rows = min(128, j.S - s0);
  T* out = j.out + b * j.sb + h * j.sh + r0;
  if (j.tiled) {
    const float* src = j.acc + ((int64_t)bh * j.tiles + tile) * (128 * j.R) + r0 * 128 + (threadIdx.x & 127);
    for (int r = threadIdx.x >> 7; r < rc; r += 2) {
      float v = 0.f;
#pragma unroll 8
      for (int e = 0; e < j.slots; ++e) v += src[r * 128 + e * j.slot_stride];
      turn[r][threadIdx.x & 127] = v;
    }
    __syncthreads();
  }
  for (int e = threadIdx.x; e < rows * rc; e += 256) {
    const int row = e / rc, r = e - row * rc;
    const float v = j.tiled ? turn[r][row] : j.acc[(((int64_t)b * j.S + s0 + row) * j.Hx + h) * j.R + r0 + r];
    out[(int64_t)(s0 + row) * j.ss + r] = from_f32<T>(v);
  }
}

template <typename T>
__global__ void __launch_bounds__(256) store_grads_kernel(const __grid_constant__ DqStoreJob<T> dq,
                                                          const __grid_constant__ FactorStoreJob<T> fq,
                                                          const __grid_constant__ FactorStoreJob<T> fk, unsigned end_dq,
                                                          unsigned end_q) {
  __shared__ float turn[kRanks][132];
  grid_dep_wait();
  const unsigned blk = blockIdx.x;
  if (blk >= end_q) return store_factor_block(fk, blk - end_q, turn);
  if (blk >= end_dq) return store_factor_block(fq, blk - end_dq, turn);
  const int64_t idx = (int64_t)blk * 256 + threadIdx.x;
  if (idx >= dq.units) return;
  const int64_t rowh = dq.div_d8.quot(idx);
  const int d = (int)(idx - rowh * dq.div_d8.d) * 8;
  const int64_t bs = dq.div_h.quot(rowh);
  const int h = (int)(rowh - bs * dq.H);
  const int64_t b = dq.div_s.quot(bs);
  const int s = (int)(bs - b * dq.Sq);
  float4 x, y;
  const int nq_tiles = (dq.Sq + 127) / 128;
  if (dq.layout == DQ_SWIZZLED) {
    const char* tile = reinterpret_cast<const char*>(dq.acc + ((b * dq.H + h) * nq_tiles + s / 128) * (128 * dq.cols));
    x = *reinterpret_cast<const float4*>(tile + dq_stage_off(s % 128, d / 4));
    y = *reinterpret_cast<const float4*>(tile + dq_stage_off(s % 128, d / 4 + 1));
  } else {
    const int64_t row = dq.layout == DQ_HEAD_ROWS ? (b * dq.H + h) * (nq_tiles * 128) + s : rowh;
    const float* src = dq.acc + row * dq.cols + d;
    x = *reinterpret_cast<const float4*>(src);
    y = *reinterpret_cast<const float4*>(src + 4);
  }
  uint4 w;
  w.x = Pack2<T>::pack(x.x * dq.scale, x.y * dq.scale);
  w.y = Pack2<T>::pack(x.z * dq.scale, x.w * dq.scale);
  w.z = Pack2<T>::pack(y.x * dq.scale, y.y * dq.scale);
  w.w = Pack2<T>::pack(y.z * dq.scale, y.w * dq.scale);
  *reinterpret_cast<uint4*>(dq.dq + b * dq.sb + h * dq.sh + s * dq.ss + d) = w;
}

template <typename T>
static unsigned factor_job(FactorStoreJob<T>& j, const float* acc, FactorAccLayout l, void* out, int Bx, int S, int Hx,
                           int R, const int64_t* stride) {
  j.acc = acc;
  j.out = reinterpret_cast<T*>(out);
  j.Bx = Bx; j.S = S; j.Hx = Hx; j.R = R;
  j.tiled = l.rows > 0;
  j.slots = l.slots;
  j.slot_stride = l.slot_stride;
  j.tiles = (S + 127) / 128;
  j.rchunks = (R + kRanks - 1) / kRanks;
  j.sb = stride[0]; j.sh = stride[1]; j.ss = stride[2];
  return (unsigned)((int64_t)Bx * Hx * j.tiles * j.rchunks);
}

template <typename T>
static int launch_store_t(const fb_params* p, const GradAccs& g, cudaStream_t st) {
  DqStoreJob<T> dq{};
  FactorStoreJob<T> fq{}, fk{};
  if (g.dq) {
    dq.acc = g.dq;
    dq.dq = reinterpret_cast<T*>(p->dq);
    dq.cols = g.dq_cols; dq.H = p->H; dq.Sq = p->Sq; dq.layout = g.dq_layout;
    dq.sb = p->dq_stride[0]; dq.sh = p->dq_stride[1]; dq.ss = p->dq_stride[2];
    dq.scale = p->softmax_scale;
    dq.div_d8 = Div(p->D / 8); dq.div_h = Div(p->H); dq.div_s = Div(p->Sq);
    dq.units = (int64_t)p->B * p->Sq * p->H * (p->D / 8);
  }
  const unsigned end_dq = (unsigned)((dq.units + 255) / 256);
  unsigned end_q = end_dq, n = end_dq;
  if (p->R > 0) {
    n += factor_job<T>(fq, g.dqb, g.dqb_layout, p->dq_bias, p->q_bias_stride[0] == 0 ? 1 : p->B, p->Sq,
                       p->q_bias_stride[1] == 0 ? 1 : p->H, p->R, p->dq_bias_stride);
    end_q = n;
    n += factor_job<T>(fk, g.dkb, g.dkb_layout, p->dk_bias, p->k_bias_stride[0] == 0 ? 1 : p->B, p->Sk,
                       p->k_bias_stride[1] == 0 ? 1 : p->H, p->R, p->dk_bias_stride);
  }
  if (n == 0) return 0;
  return launch_pdl(store_grads_kernel<T>, n, 256, 0, st, dq, fq, fk, end_dq, end_q);
}

int launch_store_grads(const fb_params* p, const GradAccs& g, cudaStream_t st) {
  return p->dtype == FB_DTYPE_F16 ? launch_store_t<__half>(p, g, st) : launch_store_t<__nv_bfloat16>(p, g, st);
}

}  // namespace fb
