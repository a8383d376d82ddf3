// PyTorch operators on top of the C ABI: argument checks, output allocation, autograd and the calls into
// libflashbias_b200, in native code.
//
// What bounds a small call is the host: through the interpreter (a Python autograd.Function, ctypes structures and
// calls) one forward + backward of the 2 x 4 x 256 x 32 shape cost 180 us of host time around 45 us of kernels.
//
// Mirrors FlashBiasFunc / flash_bias_func of the reference (flash_bias/flash_bias_triton.py:1345-1405): same
// positional signature, layouts ((B, S, H, D) tensors, (B|1, S, H|1, R) factors, 4-D additive mask), host-side checks
// and messages (:1102-1127, :1206-1210, :1371); outputs are fresh tensors, inputs are never mutated.
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/Exceptions.h>
#include <torch/extension.h>

#include <atomic>
#include <cmath>
#include <mutex>
#include <optional>
#include <tuple>

#include "flashbias_b200.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

// Failed argument checks surface as AssertionError, as the reference's assert statements do.
struct AssertionFailure : std::exception {
  std::string msg;
  explicit AssertionFailure(const char* m) : msg(m) {}
  const char* what() const noexcept override { return msg.c_str(); }
};
#define FB_ASSERT(cond, msg) \
  do {                       \
    if (!(cond)) throw AssertionFailure(msg); \
  } while (0)

void check_rc(int rc, const char* what) {
  if (rc != 0)
    throw std::runtime_error(std::string(what) + " failed: [" + std::to_string(rc) + "] " + fb_strerror(rc));
}

// ---- status word ------------------------------------------------------------------------------------------
// One int32 in pinned (device-visible) host memory: kernels store a device-side error code there, the host reads it
// without synchronising anything.
std::mutex g_status_mu;
Tensor* g_status = nullptr;  // never freed: kernels in flight at interpreter exit may still hold its address
std::atomic<int32_t*> g_status_ptr{nullptr};

int32_t* status_ptr() {
  int32_t* p = g_status_ptr.load(std::memory_order_acquire);
  if (p) return p;
  std::lock_guard<std::mutex> lk(g_status_mu);
  if (!g_status) {
    g_status = new Tensor(at::zeros({1}, at::TensorOptions().dtype(at::kInt)).pin_memory());
    g_status_ptr.store(g_status->data_ptr<int32_t>(), std::memory_order_release);
  }
  return g_status_ptr.load(std::memory_order_acquire);
}

Tensor status_word() {
  status_ptr();
  return *g_status;
}

void check_device_status() {
  int32_t* p = g_status_ptr.load(std::memory_order_acquire);
  if (!p) return;
  const int32_t code = *reinterpret_cast<volatile int32_t*>(p);
  if (code != 0) {
    *reinterpret_cast<volatile int32_t*>(p) = 0;
    throw std::runtime_error("flashbias_b200: device-side error " + std::to_string(code) + ": " +
                             fb_status_string(code) + " [" + fb_strerror(FB_EDEVICE) + "]");
  }
}

// ---- problem description -------------------------------------------------------------------------------------
int dtype_code(at::ScalarType t) {
  return t == at::kHalf ? FB_DTYPE_F16 : t == at::kBFloat16 ? FB_DTYPE_BF16 : FB_DTYPE_F32;
}

// (batch, head, row) element strides of a (B, S, H, C) tensor
void strides_bhs(const Tensor& t, int64_t (&out)[3]) {
  const auto st = t.strides();
  out[0] = st[0];
  out[1] = st[2];
  out[2] = st[1];
}
// ... with 0 for broadcast (size-1) batch / head dimensions
void factor_strides(const Tensor& t, int64_t (&out)[3]) {
  strides_bhs(t, out);
  if (t.size(0) == 1) out[0] = 0;
  if (t.size(2) == 1) out[1] = 0;
}

void fill_common(fb_params& p, const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& q_bias,
                 const OptTensor& k_bias, const OptTensor& mask, bool causal, double scale, int flags,
                 const OptTensor& slopes) {
  p.B = (int32_t)q.size(0);
  p.Sq = (int32_t)q.size(1);
  p.H = (int32_t)q.size(2);
  p.D = (int32_t)q.size(3);
  p.Sk = (int32_t)k.size(1);
  p.R = q_bias ? (int32_t)q_bias->size(3) : 0;
  p.dtype = dtype_code(q.scalar_type());
  p.causal = causal ? 1 : 0;
  p.flags = flags;
  p.softmax_scale = (float)scale;
  p.status = status_ptr();
  p.q = q.data_ptr();
  p.k = k.data_ptr();
  p.v = v.data_ptr();
  strides_bhs(q, p.q_stride);
  strides_bhs(k, p.k_stride);
  strides_bhs(v, p.v_stride);
  if (slopes) p.alibi_slopes = slopes->data_ptr<float>();
  if (q_bias) {
    p.q_bias = q_bias->data_ptr();
    p.k_bias = k_bias->data_ptr();
    factor_strides(*q_bias, p.q_bias_stride);
    factor_strides(*k_bias, p.k_bias_stride);
  }
  if (mask) {
    p.mask = mask->data_ptr();
    p.mask_dtype = dtype_code(mask->scalar_type());
    // (1, seqlen_k) is tested first, as in the reference (:1120-1123)
    p.mask_kind = mask->size(2) == 1 ? FB_MASK_VECTOR : FB_MASK_MATRIX;
    for (int i = 0; i < 3; ++i) p.mask_stride[i] = mask->size(i) == 1 ? 0 : mask->stride(i);
    // a mask with fewer batch entries than q is read periodically (entry b % n): Swin's shift mask
    p.mask_batch_period = (mask->size(0) > 1 && mask->size(0) < q.size(0)) ? (int32_t)mask->size(0) : 0;
  }
}

void check_inputs(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& q_bias, const OptTensor& k_bias,
                  const OptTensor& mask) {
  FB_ASSERT(q.dim() == 4 && k.dim() == 4 && v.dim() == 4, "q, k and v are (batch, seqlen, nheads, headdim)");
  const int64_t batch = q.size(0), seqlen_q = q.size(1), nheads = q.size(2), d = q.size(3), seqlen_k = k.size(1);
  FB_ASSERT(k.size(0) == batch && k.size(2) == nheads && k.size(3) == d, "");
  FB_ASSERT(v.sizes() == k.sizes(), "");
  FB_ASSERT(d <= 128, "FlashAttention only support head dimensions up to 128");
  FB_ASSERT(q.scalar_type() == k.scalar_type() && k.scalar_type() == v.scalar_type(), "All tensors must have the same type");
  FB_ASSERT(q.scalar_type() == at::kHalf || q.scalar_type() == at::kBFloat16, "Only support fp16 and bf16");
  FB_ASSERT(q.is_cuda() && k.is_cuda() && v.is_cuda(), "");
  if (q_bias.has_value() != k_bias.has_value()) throw std::runtime_error("q_bias and k_bias must be given together");
  if (q_bias) {
    FB_ASSERT(q_bias->scalar_type() == q.scalar_type() && k_bias->scalar_type() == q.scalar_type(),
              "All tensors must have the same type");
    for (const Tensor& t : {*q_bias, *k_bias}) FB_ASSERT(t.is_cuda() || t.is_pinned(), "");  // pinned: read in place
    FB_ASSERT(q_bias->dim() == 4 && k_bias->dim() == 4, "");
    FB_ASSERT(k_bias->size(3) == q_bias->size(3), "");
    auto fits = [&](const Tensor& t, int64_t rows) {
      return (t.size(0) == 1 || t.size(0) == batch) && (t.size(2) == 1 || t.size(2) == nheads) && t.size(1) == rows;
    };
    FB_ASSERT(fits(*q_bias, seqlen_q), "");
    FB_ASSERT(fits(*k_bias, seqlen_k), "");
  }
  if (mask) {
    FB_ASSERT(mask->scalar_type() == q.scalar_type() || mask->scalar_type() == at::kFloat, "");
    FB_ASSERT(mask->is_cuda(), "");
    FB_ASSERT(mask->dim() == 4, "");
    if (mask->size(3) != seqlen_k || (mask->size(2) != 1 && mask->size(2) != seqlen_q))
      throw std::runtime_error("Last 2 dimensions of mask must be (1, seqlen_k) or (seqlen_q, seqlen_k)");
    // the reference expands the mask over batch and heads (:1128); a mask of n batch entries with n dividing the
    // batch is also taken and read periodically, which is what Swin's repeat() produces
    const int64_t entries = mask->size(0);  // (none: not a divisor, and an integer division by zero ends the process)
    FB_ASSERT((entries == 1 || (entries > 0 && batch % entries == 0)) && (mask->size(1) == 1 || mask->size(1) == nheads), "");
  }
}

double scale_or_default(const std::optional<double>& scale, int64_t d) {
  return (scale && *scale != 0.0) ? *scale : 1.0 / std::sqrt((double)d);
}
// at::empty_like and at::empty straight from the caching allocator.  Through the dispatcher each of a call's allocations costs
// 1.5 us of host time, which is what a small call is bound by (backward of B2 H4 S256 D32 R8: six allocations, 8.7 of the
// node's 21.7 us).  A Python dispatch mode, which may want to see them, gets the dispatcher.
Tensor empty_as(const Tensor& t) {
  if (c10::impl::dispatch_mode_enabled() || !t.is_cuda() || !t.is_non_overlapping_and_dense()) return at::empty_like(t);
  return Tensor(at::detail::empty_strided_cuda(t.sizes(), t.strides(), t.scalar_type(), t.device()));
}
Tensor empty_on(at::IntArrayRef sizes, at::ScalarType type, const Tensor& like) {
  if (c10::impl::dispatch_mode_enabled()) return at::empty(sizes, like.options().dtype(type));
  return Tensor(at::detail::empty_cuda(sizes, type, like.device(), std::nullopt));
}
// Scratch comes from torch's caching allocator: freed in stream order when the call returns, so calls from several
// threads and on several streams never share it, and it goes back to the pool.
Tensor workspace(size_t nbytes, const Tensor& like) {
  return empty_on({(int64_t)nbytes}, at::kByte, like);
}
int64_t rounded_rows(int64_t s) { return (s + 127) / 128 * 128; }

// ---- forward / backward launches ----------------------------------------------------------------------------
// The role of _flash_attn_forward (flash_bias_triton.py:1100-1194): (o, lse, softmax_scale); lse is fp32 of shape
// (B, H, ceil(Sq/128)*128).
std::tuple<Tensor, Tensor, double> forward(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& q_bias,
                                           const OptTensor& k_bias, OptTensor mask, bool causal,
                                           std::optional<double> softmax_scale, int flags, const OptTensor& slopes) {
  check_device_status();
  check_inputs(q, k, v, q_bias, k_bias, mask);
  const double scale = scale_or_default(softmax_scale, q.size(3));
  if (mask && mask->stride(3) != 1) mask = mask->contiguous();
  c10::cuda::CUDAGuard guard(q.device());
  const int64_t rows = rounded_rows(q.size(1));
  Tensor lse = empty_on({q.size(0), q.size(2), rows}, at::kFloat, q);
  Tensor o = empty_as(q);
  fb_params p{};
  fill_common(p, q, k, v, q_bias, k_bias, mask, causal, scale, flags, slopes);
  p.o = o.data_ptr();
  strides_bhs(o, p.o_stride);
  p.lse = lse.data_ptr<float>();
  p.lse_stride_bh = rows;
  Tensor ws;
  if (const size_t need = fb_fwd_workspace_bytes(&p)) {
    ws = workspace(need, q);
    p.workspace = ws.data_ptr();
    p.workspace_bytes = need;
  }
  check_rc(fb_fwd(&p, at::cuda::getCurrentCUDAStream().stream()), "fb_fwd");
  return {o, lse, scale};
}

// The role of _flash_attn_backward (flash_bias_triton.py:1197-1342): (dq, dk, dv, dq_bias, dk_bias); factor gradients
// have the shape of the factors.
std::tuple<Tensor, Tensor, Tensor, OptTensor, OptTensor> backward(
    Tensor dout, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const OptTensor& q_bias,
    const OptTensor& k_bias, const Tensor& lse, OptTensor mask, bool causal, std::optional<double> softmax_scale,
    int flags, const OptTensor& slopes) {
  check_device_status();
  check_inputs(q, k, v, q_bias, k_bias, mask);
  for (const Tensor& t : {dout, o})  // (what the kernels address with q's sizes)
    FB_ASSERT(t.sizes() == q.sizes() && t.scalar_type() == q.scalar_type() && t.is_cuda(), "");
  FB_ASSERT(!q_bias || (q_bias->is_cuda() && k_bias->is_cuda()), "");  // their gradients lie where they do
  FB_ASSERT(lse.is_cuda() && lse.scalar_type() == at::kFloat && lse.is_contiguous(), "");
  if (dout.stride(-1) != 1) dout = dout.contiguous();
  const int64_t rows = rounded_rows(q.size(1));
  FB_ASSERT(lse.dim() == 3 && lse.size(0) == q.size(0) && lse.size(1) == q.size(2) && lse.size(2) == rows, "");
  FB_ASSERT(q.stride(-1) == 1 && k.stride(-1) == 1 && v.stride(-1) == 1 && o.stride(-1) == 1, "");
  const double scale = scale_or_default(softmax_scale, q.size(3));
  if (mask && mask->stride(3) != 1) mask = mask->contiguous();
  c10::cuda::CUDAGuard guard(q.device());
  Tensor dq = empty_as(q), dk = empty_as(k), dv = empty_as(v);
  OptTensor dqb, dkb;
  fb_params p{};
  fill_common(p, q, k, v, q_bias, k_bias, mask, causal, scale, flags, slopes);
  p.o = o.data_ptr();
  strides_bhs(o, p.o_stride);
  p.lse = lse.data_ptr<float>();
  p.lse_stride_bh = rows;
  p.dout = dout.data_ptr();
  strides_bhs(dout, p.dout_stride);
  p.dq = dq.data_ptr();
  p.dk = dk.data_ptr();
  p.dv = dv.data_ptr();
  strides_bhs(dq, p.dq_stride);
  strides_bhs(dk, p.dk_stride);
  strides_bhs(dv, p.dv_stride);
  if (q_bias) {
    dqb = empty_as(*q_bias);
    dkb = empty_as(*k_bias);
    p.dq_bias = dqb->data_ptr();
    p.dk_bias = dkb->data_ptr();
    strides_bhs(*dqb, p.dq_bias_stride);
    strides_bhs(*dkb, p.dk_bias_stride);
  }
  // one scratch allocation: delta in front, the library's workspace behind it (both 256-byte aligned)
  const size_t delta_bytes = (size_t)lse.numel() * 4;  // rows are multiples of 128 floats
  Tensor ws = workspace(delta_bytes + fb_bwd_workspace_bytes(&p), q);
  p.delta = reinterpret_cast<float*>(ws.data_ptr());
  p.workspace = reinterpret_cast<uint8_t*>(ws.data_ptr()) + delta_bytes;
  p.workspace_bytes = (size_t)ws.numel() - delta_bytes;
  cudaStream_t st = at::cuda::getCurrentCUDAStream().stream();
  p.flags |= FB_FLAG_BWD_FUSED_DELTA;
  check_rc(fb_bwd(&p, st), "fb_bwd");
  return {dq, dk, dv, dqb, dkb};
}

// ---- autograd ---------------------------------------------------------------------------------------------------
Tensor unit_rows(const Tensor& t) { return t.stride(-1) == 1 ? t : t.contiguous(); }
OptTensor unit_rows(const OptTensor& t) { return t ? OptTensor(unit_rows(*t)) : t; }

// A factor passed as an expanded view (size > 1, stride 0 on batch or heads) is a broadcast factor: the library gets
// the size-1 view, so that its gradient is the fp32 sum over the broadcast dimension.
OptTensor narrow_expanded(const OptTensor& t) {
  if (!t || t->dim() != 4) return t;
  Tensor r = *t;
  for (int dim : {0, 2})
    if (r.size(dim) > 1 && r.stride(dim) == 0) r = r.narrow(dim, 0, 1);
  return r;
}
// Gradient for an input that was an expanded view: autograd sums the gradient over the expanded dimension, so the
// summed gradient goes into entry 0 and the other entries are zero.
Tensor widen_grad(const OptTensor& g, at::IntArrayRef shape) {
  if (!g) return Tensor();
  if (g->sizes() == shape) return *g;
  Tensor full = at::zeros(shape, g->options());
  Tensor view = full;
  for (int dim : {0, 2})
    if (g->size(dim) != shape[dim]) view = view.narrow(dim, 0, 1);
  view.copy_(*g);
  return full;
}

[[noreturn]] void throw_assertion_from_engine(const char* msg) {
  pybind11::gil_scoped_acquire gil;
  PyErr_SetString(PyExc_AssertionError, msg);
  python_error e;
  e.persist();
  throw e;
}

OptTensor defined_or_none(const Tensor& t) { return t.defined() ? OptTensor(t) : std::nullopt; }

struct FlashBiasNode : torch::autograd::Function<FlashBiasNode> {
  // slopes: the fused ALiBi producer (q_bias, k_bias and mask are then absent)
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& q_, const Tensor& k_, const Tensor& v_,
                        const OptTensor& q_bias_, const OptTensor& k_bias_, const OptTensor& mask,
                        const OptTensor& slopes, bool causal, std::optional<double> softmax_scale) {
    const Tensor q = unit_rows(q_), k = unit_rows(k_), v = unit_rows(v_);
    const OptTensor q_bias = narrow_expanded(unit_rows(q_bias_)), k_bias = narrow_expanded(unit_rows(k_bias_));
    auto [o, lse, scale] = ::forward(q, k, v, q_bias, k_bias, mask, causal, softmax_scale, 0, slopes);
    auto or_undef = [](const OptTensor& t) { return t ? *t : Tensor(); };
    ctx->save_for_backward({q, k, v, o, or_undef(q_bias), or_undef(k_bias), lse, or_undef(mask), or_undef(slopes)});
    ctx->saved_data["causal"] = causal;
    ctx->saved_data["scale"] = scale;
    if (q_bias_ && (q_bias->sizes() != q_bias_->sizes() || k_bias->sizes() != k_bias_->sizes())) {  // expanded views
      ctx->saved_data["qb_shape"] = q_bias_->sizes().vec();
      ctx->saved_data["kb_shape"] = k_bias_->sizes().vec();
    }
    return o;
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx,
                                                 torch::autograd::variable_list grads) {
    at::NoGradGuard no_grad;
    const auto s = ctx->get_saved_variables();
    const OptTensor q_bias = defined_or_none(s[4]), k_bias = defined_or_none(s[5]), mask = defined_or_none(s[7]),
                    slopes = defined_or_none(s[8]);
    // (edges are counted over the tensors that were given)
    if (mask && ctx->needs_input_grad(q_bias ? 5 : 3)) throw_assertion_from_engine("FlashBias does not support mask gradient yet");
    auto [dq, dk, dv, dqb, dkb] =
        ::backward(grads[0], s[0], s[1], s[2], s[3], q_bias, k_bias, s[6], mask, ctx->saved_data["causal"].toBool(),
                   ctx->saved_data["scale"].toDouble(), 0, slopes);
    Tensor gqb, gkb;
    if (q_bias) {
      gqb = *dqb;
      gkb = *dkb;
      if (ctx->saved_data.count("qb_shape")) {
        gqb = widen_grad(dqb, ctx->saved_data["qb_shape"].toIntVector());
        gkb = widen_grad(dkb, ctx->saved_data["kb_shape"].toIntVector());
      }
    }
    return {dq, dk, dv, gqb, gkb, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

bool wants_grad(const OptTensor& t) { return t && t->requires_grad(); }

// There is no forward-mode derivative: a tangent is refused, as torch.autograd.Function does without a jvp, and not
// dropped by the calls that need no node.
struct NoForwardMode : std::exception {
  const char* what() const noexcept override { return "flash_bias has no forward-mode derivative"; }
};
void refuse_tangent(const Tensor& t) {
  if (t._fw_grad(/*level=*/0).defined()) throw NoForwardMode();
}
void refuse_tangent(const OptTensor& t) {
  if (t) refuse_tangent(*t);
}
template <typename... Ts>
void refuse_tangents(const Ts&... t) {
  (refuse_tangent(t), ...);
}

Tensor flash_bias(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& q_bias, const OptTensor& k_bias,
                  const OptTensor& mask, bool causal, std::optional<double> softmax_scale) {
  refuse_tangents(q, k, v, q_bias, k_bias, mask);
  if (at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad() ||
                                     wants_grad(q_bias) || wants_grad(k_bias) || wants_grad(mask)))
    return FlashBiasNode::apply(q, k, v, q_bias, k_bias, mask, OptTensor(), causal, softmax_scale);
  return std::get<0>(forward(unit_rows(q), unit_rows(k), unit_rows(v), narrow_expanded(unit_rows(q_bias)),
                             narrow_expanded(unit_rows(k_bias)), mask, causal, softmax_scale, 0, OptTensor()));
}

// The reference's language-model call site builds the ALiBi bias as rank-2 factors from the positions and the per-head
// slopes (1_Language_Model/attention_with_alibi_bias.py:47-52); here the slopes (fp32, one per head, a constant: no
// gradient) go in directly, the positions never exist as tensors and are never rounded to 16 bits.
Tensor flash_bias_alibi(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& slopes_, bool causal,
                        std::optional<double> softmax_scale) {
  refuse_tangents(q, k, v, slopes_);
  const Tensor slopes = slopes_.detach().to(q.device(), at::kFloat).reshape({-1}).contiguous();
  FB_ASSERT(q.dim() == 4 && slopes.numel() == q.size(2), "one slope per head");
  if (at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad()))
    return FlashBiasNode::apply(q, k, v, OptTensor(), OptTensor(), OptTensor(), OptTensor(slopes), causal, softmax_scale);
  return std::get<0>(forward(unit_rows(q), unit_rows(k), unit_rows(v), OptTensor(), OptTensor(), OptTensor(), causal,
                             softmax_scale, 0, slopes));
}

// ---- caller-side layout glue (see layout.py) --------------------------------------------------------------------
Tensor prepare_bhsd(const Tensor& x, at::ScalarType dtype, bool normalize, const OptTensor& head_scale, double eps) {
  FB_ASSERT(x.dim() == 4 && x.is_cuda() && x.stride(-1) == 1, "");
  FB_ASSERT(x.scalar_type() == at::kFloat || x.scalar_type() == at::kHalf || x.scalar_type() == at::kBFloat16, "");
  FB_ASSERT(dtype == at::kHalf || dtype == at::kBFloat16, "");
  c10::cuda::CUDAGuard guard(x.device());
  Tensor y = at::empty(x.sizes(), x.options().dtype(dtype));
  OptTensor hs;
  if (head_scale) {
    hs = head_scale->detach().to(x.device(), at::kFloat).reshape({-1}).contiguous();
    FB_ASSERT(hs->numel() == x.size(1), "");
  }
  const int64_t xs[3] = {x.stride(0), x.stride(1), x.stride(2)}, ys[3] = {y.stride(0), y.stride(1), y.stride(2)};
  check_rc(fb_prepare_rows(x.data_ptr(), dtype_code(x.scalar_type()), xs, y.data_ptr(), dtype_code(dtype), ys,
                           (int32_t)x.size(0), (int32_t)x.size(1), (int32_t)x.size(2), (int32_t)x.size(3),
                           normalize ? 1 : 0, hs ? hs->data_ptr<float>() : nullptr, (float)eps,
                           at::cuda::getCurrentCUDAStream().stream()),
           "fb_prepare_rows");
  return y.permute({0, 2, 1, 3});
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  namespace py = pybind11;
  using release = py::call_guard<py::gil_scoped_release>;
  py::register_exception_translator([](std::exception_ptr e) {
    try {
      if (e) std::rethrow_exception(e);
    } catch (const AssertionFailure& x) {
      PyErr_SetString(PyExc_AssertionError, x.what());
    } catch (const NoForwardMode& x) {
      PyErr_SetString(PyExc_NotImplementedError, x.what());
    }
  });
  m.def("status_word", &status_word, release());
  m.def("check_device_status", &check_device_status, release());
  m.def("forward", &forward, release());
  m.def("backward", &backward, release());
  m.def("narrow_expanded", &narrow_expanded, release());
  m.def("widen_grad", [](const Tensor& g, const std::vector<int64_t>& shape) { return widen_grad(g, shape); }, release());
  m.def("flash_bias", &flash_bias, release(), py::arg("q"), py::arg("k"), py::arg("v"), py::arg("q_bias") = py::none(),
        py::arg("k_bias") = py::none(), py::arg("mask") = py::none(), py::arg("causal") = false,
        py::arg("softmax_scale") = py::none());
  m.def("flash_bias_alibi", &flash_bias_alibi, release(), py::arg("q"), py::arg("k"), py::arg("v"), py::arg("slopes"),
        py::arg("causal") = true, py::arg("softmax_scale") = py::none());
  m.def("prepare_bhsd", &prepare_bhsd, release());
}
