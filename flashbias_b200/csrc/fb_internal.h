// Host-side declarations shared by the translation units of libflashbias_b200.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "flashbias_b200.h"

namespace fb {

// Division by a launch constant: multiply-high, add and shift while the dividend is below 2^31 (every index of the
// sizes that occur; four 64-bit divisions per thread cost the elementwise passes more than their memory traffic), the
// 64-bit division beyond.
struct Div {
  uint32_t d, m, s;
  Div() = default;
  explicit Div(int d_) : d((uint32_t)d_), m(0), s(0) {
    while ((1u << s) < d) ++s;  // ceil(log2 d)
    m = (uint32_t)((((uint64_t)1 << 32) * (((uint64_t)1 << s) - d)) / d + 1);
  }
#ifdef __CUDACC__
  __device__ __forceinline__ int quot32(int n) const { return (int)((__umulhi((uint32_t)n, m) + (uint32_t)n) >> s); }
  __device__ __forceinline__ int64_t quot(int64_t n) const {
    if (n < 0x80000000LL) return (int64_t)((__umulhi((uint32_t)n, m) + (uint32_t)n) >> s);
    return n / d;
  }
#endif
};

// ---- tensor maps (fb_tmap.cu) ---------------------------------------------------------------
// Tiled tensor map over a 16-bit tensor addressed (col, row, head, batch); strides in elements.
// Box = (box_cols x box_rows x 1 x 1), swizzle chosen from box_cols (32/64/128 bytes).
// Returns 0 or a negative FB_E* / positive cudaError_t.
int make_tmap_4d(CUtensorMap* out, const void* ptr, int cols, int64_t rows, int64_t heads, int64_t batch,
                 int64_t stride_row, int64_t stride_head, int64_t stride_batch, int box_cols, int box_rows);
// Tensor map over a matrix mask of any element type, box = 128 rows of 128 bytes (128-byte swizzle), extents 1 on broadcast
// dimensions; false if TMA cannot address its rows (base or a stride not a multiple of 16 bytes, a (1, Sk) mask).
bool make_tmap_mask(CUtensorMap* out, const fb_params* p);
// True if a (ptr, strides) tensor can be described by make_tmap_4d.
bool tma_compatible(const void* ptr, int64_t stride_row, int64_t stride_head, int64_t stride_batch, int64_t heads,
                    int64_t batch);

// ---- operand preparation (fb_pack.cu) ------------------------------------------------------------
// The tensor-core kernels contract over [scaled query terms | packed rank] in one fp32 accumulator.
//   nq == 1 (softmax_scale an exact power of two): the query operand is the caller's q, the q-side factor is
//           q_bias / scale (exact), logits = scale * S.
//   nq == 2: the query operand is q*scale as a (hi, lo) pair of 16-bit terms, formed on chip; factors are used as given,
//           logits = S.  (The backward splits k*scale instead: its key tile is the resident one.)
// Packed factors: (Bb, Hb, S, RP) contiguous, Bb/Hb = 1 on broadcast dims, zero-padded to RP columns.
struct PackPlan {
  int nq;          // 1 or 2 query terms
  float qb_mult;   // multiplier applied to q_bias when packing (1/scale when nq == 1)
  int TD;          // head_dim padded to the tile width: 32, 64 or 128 (missing columns are read as zero)
  int RP;          // packed factor width: 0 (no bias), 16, 32 or 64
  int RC;          // width of the centred k-side copy of the backward (>= RP; 32 beside a head_dim-32 K tile)
  int kernel;      // FB_KERNEL_* of the tensor-core kernel that takes the problem
  int Bq, Hq, Bk, Hk;
  size_t q_bytes, k_bytes, kc_bytes, qs_bytes;  // packed q factor, packed k factor, centred k factor, scaled-key
                                               // copy (each rounded to 256)
};
// false if the rank does not fit the tensor path; for_bwd reserves room for the centred (hi, lo) k-side copy
bool plan_pack(const fb_params* p, PackPlan* plan, bool for_bwd = false);
// a backward plan with factors, re-planned for the two-stream kernel: factor tiles as wide as the rank asks
void plan_two_stream(const fb_params* p, PackPlan* plan);
// What one launch prepares for a call: packed q/k factors, kcenter (optional, rows of plan.RC columns: k_bias minus the
// k_bias of the middle key of each group of 32 keys), when plan.nq == 2 the (hi, lo) split of k*scale (optional), laid out
// (B, H, Sk, 2 TD), and for the backward delta (optional) and the zeroed accumulators.
struct PrepBuffers {
  void *qpack, *kpack, *kcenter, *scaled;
  float* delta;
  void* zero;
  size_t zero_bytes;
};
int launch_prepare(const fb_params* p, const PackPlan& plan, const PrepBuffers& buf, cudaStream_t st);
// where fb_bwd takes delta itself (null: the caller has run fb_bwd_preprocess)
inline float* fused_delta(const fb_params* p) { return (p->flags & FB_FLAG_BWD_FUSED_DELTA) ? p->delta : nullptr; }

// ---- kernels ------------------------------------------------------------------------------------
int launch_fwd_general(const fb_params* p, cudaStream_t st);
int launch_bwd_preprocess(const fb_params* p, cudaStream_t st);
int launch_bwd_general(const fb_params* p, cudaStream_t st);
size_t bwd_general_workspace(const fb_params* p);

// one query row per (batch, head)
bool decode_supported(const fb_params* p);
size_t decode_workspace(const fb_params* p);
int launch_decode(const fb_params* p, cudaStream_t st);

bool fwd_sm100_supported(const fb_params* p, PackPlan* plan);
int launch_fwd_sm100(const fb_params* p, const PackPlan& plan, cudaStream_t st);

bool bwd_sm100_supported(const fb_params* p, PackPlan* plan);
size_t bwd_sm100_workspace(const fb_params* p, const PackPlan& plan);
int launch_bwd_sm100(const fb_params* p, const PackPlan& plan, cudaStream_t st);

inline size_t round256(size_t x) { return (x + 255) & ~size_t(255); }

// fp32 factor-gradient accumulators.  Default shape: the un-expanded (Bx, S, Hx, R).  The tensor-core backward
// uses `slots` copies (summed by the final store) of a head-major (Bx, Hx, rows, R) array with rows padded to
// whole 128-row tiles, so that a tile's rows are contiguous for a bulk reduction.
struct FactorAccLayout {
  int64_t rows;         // 0: default shape
  int slots;            // copies to sum
  int64_t slot_stride;  // floats between copies
};
// Arrangement of the fp32 dq accumulator: (B, Sq, H, cols); per (batch, head, tile of 128 rows) as dq_stage_off has it;
// (B, H, rows padded to 128, cols)
enum { DQ_ROWS = 0, DQ_SWIZZLED = 1, DQ_HEAD_ROWS = 2 };
// The fp32 accumulators of a backward; launch_store_grads rounds them into p->dq (unless dq is null: the main kernel
// has stored it), p->dq_bias and p->dk_bias.
struct GradAccs {
  const float* dq;
  int dq_layout;  // DQ_*
  int dq_cols;    // columns of an accumulator row (>= D)
  const float *dqb, *dkb;
  FactorAccLayout dqb_layout, dkb_layout;
};
int launch_store_grads(const fb_params* p, const GradAccs& g, cudaStream_t st);

// ---- instrumentation (fb_api.cu) ----------------------------------------------------------------
// Every kernel launch of the library is counted; while profiling is armed for a kernel class, a pair
// of CUDA events is recorded around each launch of that class on the launching stream.
enum KernelClass { KC_OTHER = 0, KC_FWD_MAIN = 1, KC_BWD_MAIN = 2, KC_BWD_PREPROCESS = 3 };
void note_launch(int n = 1);
// number of SMs of a device (cached per device); 0 if the query fails
int device_sm_count(int dev);
void prof_before(int kernel_class, cudaStream_t st);
void prof_after(int kernel_class, cudaStream_t st);

// Launch with programmatic stream serialization: the grid may be set up while the kernel before it in the stream
// drains.  Every kernel launched this way executes grid_dep_wait() before it touches global memory.
template <typename... P, typename... A>
int launch_pdl(void (*kern)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
  if (e == cudaSuccess) note_launch();
  return (int)e;
}

}  // namespace fb
