// The Python layer's frequent calls in one native step each: argument checks, allocations, stream and
// library call.  Through ctypes these cost 11 to 45 us a call (a linear 27, a quantizer 21 to 28, norm + quantize
// 30 to 38, the backward of a linear 45), more than the kernels of a few thousand rows take.
//
// Every function returns None for what is not the plain case (other types, devices, layouts or alignments,
// tensor subclasses, an active dispatch mode, an empty tensor): the Python code that called it then does what it
// always did, errors included.  Nothing is kept between calls but the address of each device's status word.
//
// The calls let go of the interpreter lock, as the ctypes calls and torch's own allocations do: a launch waits where the
// stream's queue is full and an allocation may reach the driver, and neither needs the interpreter.  Their errors are
// torch's (an allocation that does not fit raises torch.OutOfMemoryError).
#include <ATen/TensorSubclassLikeUtils.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include <atomic>
#include <optional>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/nvfp4_b200.h"

namespace {

using at::Tensor;
using Maybe = std::optional<Tensor>;

std::atomic<int*> g_status[64];           // per device; set once, before the first call there

void check(int rc, const char* what) {
  if (rc != NVFP4_OK)
    throw std::runtime_error(std::string("[s4] [nvfp4] ") + what + ": " + nvfp4_status_string(rc) + " (status " +
                             std::to_string(rc) + ")");
}

bool plain(const Tensor& t) {
  return t.defined() && t.is_cuda() && t.layout() == at::kStrided && !at::isTensorSubclassLike(t) && !t.is_conj() &&
         !t.is_neg();
}
bool modes() { return c10::impl::TorchDispatchModeTLS::any_modes_set(); }
bool aligned(const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.const_data_ptr()) & 15u) == 0; }
// absent, or contiguous of this type, size and device on a 16-byte boundary
bool fits(const Maybe& t, at::ScalarType type, int64_t numel, const Tensor& like) {
  return !t || (plain(*t) && t->scalar_type() == type && t->numel() == numel && t->device() == like.device() &&
                t->is_contiguous() && aligned(*t));
}
void* ptr(const Maybe& t) { return t ? t->data_ptr() : nullptr; }
Maybe nonempty(const Maybe& t) { return t && t->numel() > 0 ? t : Maybe(); }
int* status_of(const Tensor& t) {
  return t.get_device() < 64 ? g_status[t.get_device()].load(std::memory_order_acquire) : nullptr;
}
void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }
Tensor empty(at::IntArrayRef size, at::ScalarType type, const Tensor& like) {
  return at::empty(size, at::TensorOptions().dtype(type).device(like.device()));
}
float* f32(const Tensor& t) { return static_cast<float*>(t.data_ptr()); }
uint8_t* u8(const Tensor& t) { return static_cast<uint8_t*>(t.data_ptr()); }
uint8_t* u8(const Maybe& t) { return t ? u8(*t) : nullptr; }

void set_status(int64_t device, const Tensor& word) {
  if (device >= 0 && device < 64) g_status[device].store(static_cast<int*>(word.data_ptr()), std::memory_order_release);
}

// y = residual + gate * act(x @ w.T + bias) with the packed weight of `weight`
Maybe linear(const Tensor& x, const Tensor& weight, const Tensor& w_data, const Tensor& w_scales,
             const Tensor& w_gscale, const Maybe& bias_, const Maybe& gate, const Maybe& residual, bool gelu) {
  if (!plain(x) || !plain(weight) || modes() || x.dim() < 2 || weight.dim() != 2) return {};
  const Maybe bias = nonempty(bias_);
  const int64_t k = x.size(-1), n = weight.size(0), m = k > 0 ? x.numel() / k : 0;
  if (x.scalar_type() != at::kBFloat16 || weight.scalar_type() != at::kBFloat16 || weight.size(1) != k ||
      x.device() != weight.device() || m == 0 || n == 0 || k % 32 != 0 || n % 8 != 0 || !x.is_contiguous() ||
      !aligned(x) || !status_of(x))
    return {};
  if (!fits(bias, at::kBFloat16, n, x) || (bias && bias->dim() != 1) || !fits(gate, at::kFloat, n, x) ||
      (gate && gate->dim() != 1) || !fits(residual, at::kBFloat16, m * n, x) || (residual && residual->size(-1) != n))
    return {};
  const c10::cuda::CUDAGuard guard(x.device());
  auto size = x.sizes().vec();
  size.back() = n;
  Tensor y = empty(size, at::kBFloat16, x);
  const Tensor ws = empty({nvfp4_linear_workspace_bytes(m, k)}, at::kByte, x);
  check(nvfp4_linear_bf16(x.data_ptr(), m, k, u8(w_data), u8(w_scales), f32(w_gscale), n, ptr(bias),
                          static_cast<float*>(ptr(gate)), ptr(residual), gelu ? NVFP4_ACT_GELU_TANH : NVFP4_ACT_NONE,
                          y.data_ptr(), ws.data_ptr(), status_of(x), stream_of(x)),
        "[linear] launch");
  return y;
}

// rows, cols, data, scales, swizzled scales, amax, tensor scale
using Packed = std::tuple<int64_t, int64_t, Tensor, Maybe, Maybe, Tensor, Tensor>;

// Of a bf16 tensor of whole blocks.
std::optional<Packed> quantize(const Tensor& x, bool linear_scales, bool swizzled_scales) {
  if (!plain(x) || modes() || x.scalar_type() != at::kBFloat16 || x.dim() < 1 || x.numel() == 0 ||
      x.size(-1) % 16 != 0 || !x.is_contiguous())
    return {};
  const c10::cuda::CUDAGuard guard(x.device());
  const int64_t cols = x.size(-1), rows = x.numel() / cols;
  Tensor amax = empty({1}, at::kFloat, x), gscale = empty({1}, at::kFloat, x);
  Tensor data = empty({rows * cols / 2}, at::kByte, x);
  Maybe scales, swz;
  if (linear_scales) scales = empty({rows * cols / 16}, at::kByte, x);
  if (swizzled_scales) swz = empty({nvfp4_swizzled_scale_bytes(rows, cols)}, at::kByte, x);
  const Tensor partials = empty({NVFP4_AMAX_PARTIALS}, at::kFloat, x);
  check(nvfp4_amax_quantize_bf16(x.data_ptr(), rows, cols, f32(amax), u8(data), u8(scales), u8(swz), f32(gscale),
                                 f32(partials), stream_of(x)),
        "[tensor] amax+quantize");
  return Packed(rows, cols, data, scales, swz, amax, gscale);
}

// The same with its maximum known (amax), and into the given buffers (data, scales, swizzled scales, amax, tensor scale, row
// statistics, partial maxima).
std::optional<Packed> quantize_into(const Tensor& x, bool linear_scales, bool swizzled_scales, const Maybe& amax_,
                                    const std::optional<std::vector<Maybe>>& out) {
  if (!plain(x) || modes() || x.scalar_type() != at::kBFloat16 || x.dim() < 1 || x.numel() == 0 ||
      x.size(-1) % 16 != 0 || !x.is_contiguous())
    return {};
  if (amax_ && (!plain(*amax_) || amax_->scalar_type() != at::kFloat || amax_->numel() != 1 ||
                amax_->device() != x.device()))
    return {};
  const c10::cuda::CUDAGuard guard(x.device());
  const int64_t cols = x.size(-1), rows = x.numel() / cols;
  Tensor data, gscale, amax, partials;
  Maybe scales, swz;
  if (out) {
    const auto& o = *out;
    data = *o[0]; swz = o[2]; gscale = *o[4]; partials = *o[6];
    if (linear_scales) scales = o[1];
    amax = amax_ ? *amax_ : *o[3];
  } else {
    amax = amax_ ? *amax_ : empty({1}, at::kFloat, x);
    gscale = empty({1}, at::kFloat, x);
    data = empty({rows * cols / 2}, at::kByte, x);
    if (linear_scales) scales = empty({rows * cols / 16}, at::kByte, x);
    if (swizzled_scales) swz = empty({nvfp4_swizzled_scale_bytes(rows, cols)}, at::kByte, x);
    if (!amax_) partials = empty({NVFP4_AMAX_PARTIALS}, at::kFloat, x);
  }
  if (amax_)
    check(nvfp4_quantize_bf16(x.data_ptr(), rows, cols, f32(amax), u8(data), u8(scales), u8(swz), f32(gscale), stream_of(x)),
          "[tensor] quantize");
  else
    check(nvfp4_amax_quantize_bf16(x.data_ptr(), rows, cols, f32(amax), u8(data), u8(scales), u8(swz), f32(gscale),
                                   f32(partials), stream_of(x)),
          "[tensor] amax+quantize");
  return Packed(rows, cols, data, scales, swz, amax, gscale);
}

// The same of norm(x) * weight + bias, modulated; into the given buffers (data, scales, swizzled scales, amax,
// tensor scale, row statistics, partial maxima) or new ones.
std::optional<Packed> norm_quantize(const Tensor& x, const Maybe& weight, const Maybe& bias, const Maybe& scale,
                         const Maybe& shift, bool rms, double eps, bool linear_scales,
                         const std::optional<std::vector<Maybe>>& out) {
  if (!plain(x) || modes() || x.scalar_type() != at::kBFloat16 || x.dim() < 1 || x.numel() == 0 ||
      !x.is_contiguous() || !status_of(x))
    return {};
  const int64_t cols = x.size(-1), rows = x.numel() / cols;
  if (cols % 16 != 0 || cols > 16384) return {};
  for (const Maybe* v : {&weight, &bias, &scale, &shift})
    if (!fits(*v, at::kFloat, cols, x)) return {};
  const c10::cuda::CUDAGuard guard(x.device());
  Tensor data, amax, gscale, work;
  Maybe scales, swz;
  float *stats, *partials;
  if (out) {
    const auto& o = *out;
    data = *o[0]; swz = o[2]; amax = *o[3]; gscale = *o[4];
    if (linear_scales) scales = o[1];
    stats = f32(*o[5]);
    partials = f32(*o[6]);
  } else {
    amax = empty({1}, at::kFloat, x);
    gscale = empty({1}, at::kFloat, x);
    data = empty({rows * cols / 2}, at::kByte, x);
    if (linear_scales) scales = empty({rows * cols / 16}, at::kByte, x);
    swz = empty({nvfp4_swizzled_scale_bytes(rows, cols)}, at::kByte, x);
    work = empty({2 * rows + NVFP4_AMAX_PARTIALS}, at::kFloat, x);
    stats = f32(work);
    partials = stats + 2 * rows;
  }
  check(nvfp4_norm_mod_bf16(x.data_ptr(), rows, cols, static_cast<float*>(ptr(weight)), static_cast<float*>(ptr(bias)),
                            static_cast<float*>(ptr(scale)), static_cast<float*>(ptr(shift)), rms ? 1 : 0, (float)eps,
                            stats, f32(amax), u8(data), u8(scales), u8(swz), f32(gscale), partials, status_of(x),
                            stream_of(x)),
        "[tensor] norm+quantize");
  return Packed(rows, cols, data, scales, swz, amax, gscale);
}

Maybe dequantize(const Tensor& data, const Tensor& scales, const Tensor& amax, int64_t rows, int64_t cols,
                 const std::vector<int64_t>& shape) {
  if (!plain(data) || !plain(scales) || !plain(amax) || modes() || rows * cols == 0) return {};
  const c10::cuda::CUDAGuard guard(data.device());
  Tensor out = empty(shape, at::kBFloat16, data);
  check(nvfp4_dequantize_bf16(u8(data), u8(scales), rows, cols, f32(amax), out.data_ptr(), stream_of(data)),
        "[tensor] dequantize");
  return out;
}

// alpha * a @ b.T (+ bias, GELU, gate) + beta * c on packed [M, K] and [N, K]
Maybe gemm(const Tensor& a, const Tensor& b, const Tensor& a_scales, const Tensor& b_scales, const Tensor& a_gscale,
           const Tensor& b_gscale, int64_t M, int64_t N, int64_t K, double alpha, double beta, const Maybe& c,
           const Maybe& bias, const Maybe& gate, bool gelu, const Maybe& out, const Maybe& out_amax) {
  if (!plain(a) || !plain(b) || modes() || a.device() != b.device() || M == 0 || N == 0 || K % 32 != 0 || N % 8 != 0 ||
      !status_of(a))
    return {};
  if (!fits(c, at::kBFloat16, M * N, a) || (c && (c->dim() != 2 || c->size(0) != M)) ||
      !fits(bias, at::kBFloat16, N, a) || (bias && bias->dim() != 1) || !fits(gate, at::kFloat, N, a) ||
      (gate && gate->dim() != 1) || !fits(out, at::kBFloat16, M * N, a) ||
      (out && (out->dim() != 2 || out->size(0) != M)))
    return {};
  const c10::cuda::CUDAGuard guard(a.device());
  Tensor d = out ? *out : empty({M, N}, at::kBFloat16, a);
  check(nvfp4_gemm(u8(a), u8(b), u8(a_scales), u8(b_scales), f32(a_gscale), f32(b_gscale), M, N, K, (float)alpha,
                   (float)beta, ptr(c), ptr(bias), static_cast<float*>(ptr(gate)),
                   gelu ? NVFP4_ACT_GELU_TANH : NVFP4_ACT_NONE, d.data_ptr(), static_cast<float*>(ptr(out_amax)),
                   status_of(a), stream_of(a)),
        "[gemm] launch");
  return d;
}

// Whether something follows what is done to t: a graph being recorded, a forward-mode tangent, a trace.
bool followed(const Tensor& t) {
  return (t.requires_grad() && at::GradMode::is_enabled()) || t._fw_grad(0).defined() ||
         c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::Tracer);
}

// The gradients that are wanted of y = x @ w.T + b: dx, dw, db (not db where dy is followed: it stays torch's sum)
std::optional<std::vector<Maybe>> linear_backward(const Tensor& dy, const Tensor& x, const Tensor& w, bool want_dx,
                                                  bool want_dw, bool want_db) {
  if (!plain(dy) || !plain(x) || !plain(w) || modes() || (!want_dx && !want_dw) || dy.dim() < 1 || x.dim() < 1 ||
      w.dim() != 2 || !status_of(dy))
    return {};
  const int64_t n = w.size(0), k = w.size(1);
  if (n == 0 || k == 0 || dy.numel() == 0 || dy.size(-1) != n || x.size(-1) != k) return {};
  const int64_t m = dy.numel() / n;
  if (x.numel() != m * k || n % 32 != 0 || k % 8 != 0) return {};
  for (const Tensor* t : {&dy, &x, &w})
    if (t->scalar_type() != at::kBFloat16 || t->device() != dy.device() || !t->is_contiguous() || !aligned(*t)) return {};
  const c10::cuda::CUDAGuard guard(dy.device());
  Maybe dx, dw, db;
  if (want_dx) dx = empty(x.sizes(), at::kBFloat16, dy);
  if (want_dw) dw = empty({n, k}, at::kBFloat16, dy);
  if (want_db && !followed(dy)) db = empty({n}, at::kBFloat16, dy);
  const Tensor ws = empty({nvfp4_linear_backward_workspace_bytes(m, n, k)}, at::kByte, dy);
  check(nvfp4_linear_backward_bias_bf16(dy.data_ptr(), want_dw ? x.data_ptr() : nullptr, want_dx ? w.data_ptr() : nullptr,
                                        nullptr, m, n, k, ptr(dx), ptr(dw), ptr(db), ws.data_ptr(), status_of(dy),
                                        stream_of(dy)),
        "[linear] backward");
  return std::vector<Maybe>{dx, dw, db};
}

// RMSNorm across heads of q and k and the rotary embedding of [L, 3 * heads * head_dim]: q, k
std::optional<std::tuple<Tensor, Tensor>> qk_norm_rope(const Tensor& qkv, int64_t heads, int64_t head_dim,
                                                       const Maybe& gain_q, const Maybe& gain_k, double eps,
                                                       const Tensor& cos_sin) {
  if (!plain(qkv) || !plain(cos_sin) || modes() || heads <= 0 || head_dim <= 0 || heads > 16384 || head_dim > 16384 ||
      qkv.dim() != 2 || qkv.scalar_type() != at::kBFloat16 || !qkv.is_contiguous() ||
      qkv.get_device() != c10::cuda::current_device() || !status_of(qkv))
    return {};
  const int64_t L = qkv.size(0), dim = heads * head_dim;
  if (qkv.size(1) != 3 * dim || cos_sin.dim() != 3 || cos_sin.size(0) != L || cos_sin.size(1) != head_dim / 2 ||
      cos_sin.size(2) != 2 || !fits(cos_sin, at::kFloat, cos_sin.numel(), qkv) || !fits(gain_q, at::kFloat, dim, qkv) ||
      !fits(gain_k, at::kFloat, dim, qkv))
    return {};
  Tensor q = empty({L, heads, head_dim}, at::kBFloat16, qkv), k = empty({L, heads, head_dim}, at::kBFloat16, qkv);
  const char* base = static_cast<const char*>(qkv.data_ptr());
  check(nvfp4_qk_norm_rope_bf16(base, base + 2 * dim, nullptr, 3 * dim, L, (int)heads, (int)head_dim,
                                static_cast<float*>(ptr(gain_q)), static_cast<float*>(ptr(gain_k)), (float)eps,
                                f32(cos_sin), q.data_ptr(), k.data_ptr(), nullptr, dim, head_dim, status_of(qkv),
                                stream_of(qkv)),
        "qk_norm_rope");
  return std::make_tuple(q, k);
}

// RMSNorm of the rows of [L, heads * head_dim], which may lie apart
Maybe rms_norm(const Tensor& x, int64_t heads, int64_t head_dim, const Maybe& gain, double eps) {
  if (!plain(x) || modes() || heads <= 0 || head_dim <= 0 || heads > 16384 || head_dim > 16384 || x.dim() != 2 ||
      x.scalar_type() != at::kBFloat16 || x.get_device() != c10::cuda::current_device() || !status_of(x))
    return {};
  const int64_t L = x.size(0), dim = heads * head_dim;
  if (x.size(1) != dim || x.stride(1) != 1 || x.stride(0) % 8 != 0 || !aligned(x) || !fits(gain, at::kFloat, dim, x))
    return {};
  Tensor out = empty({L, heads, head_dim}, at::kBFloat16, x);
  check(nvfp4_qk_norm_rope_bf16(x.data_ptr(), nullptr, nullptr, x.stride(0), L, (int)heads, (int)head_dim,
                                static_cast<float*>(ptr(gain)), nullptr, (float)eps, nullptr, out.data_ptr(), nullptr,
                                nullptr, dim, head_dim, status_of(x), stream_of(x)),
        "rms_norm");
  return out;
}

Maybe attention(const Tensor& q, const Tensor& k, const Tensor& v, const Maybe& amax, const Maybe& out) {
  if (!plain(q) || !plain(k) || !plain(v) || modes() || out || q.dim() != 3 || k.dim() != 3 || v.dim() != 3 ||
      !status_of(q) || q.get_device() != c10::cuda::current_device())
    return {};
  const int64_t H = q.size(1), D = q.size(2);
  for (const Tensor* t : {&q, &k, &v})
    if (t->scalar_type() != at::kBFloat16 || t->stride(2) != 1 || t->size(1) != H || t->size(2) != D ||
        t->device() != q.device())
      return {};
  if (k.size(0) != v.size(0)) return {};
  if (amax && (!plain(*amax) || amax->scalar_type() != at::kFloat || amax->numel() < 1 || amax->device() != q.device()))
    return {};
  Tensor o = empty({q.size(0), H, D}, at::kBFloat16, q);
  check(nvfp4_attention_bf16(q.data_ptr(), q.stride(0), q.stride(1), k.data_ptr(), k.stride(0), k.stride(1),
                             v.data_ptr(), v.stride(0), v.stride(1), q.size(0), k.size(0), (int)H, (int)D,
                             (float)(1.0 / std::sqrt((double)D)), o.data_ptr(), o.stride(0), o.stride(1),
                             static_cast<float*>(ptr(amax)), status_of(q), stream_of(q)),
        "attention");
  return o;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.attr("built_for") = NVFP4_BUILT_FOR;
  m.def("set_status", &set_status);
  m.def("linear", torch::wrap_pybind_function_no_gil(linear));
  m.def("quantize", torch::wrap_pybind_function_no_gil(quantize));
  m.def("quantize_into", torch::wrap_pybind_function_no_gil(quantize_into));
  m.def("linear_backward", torch::wrap_pybind_function_no_gil(linear_backward));
  m.def("qk_norm_rope", torch::wrap_pybind_function_no_gil(qk_norm_rope));
  m.def("rms_norm", torch::wrap_pybind_function_no_gil(rms_norm));
  m.def("norm_quantize", torch::wrap_pybind_function_no_gil(norm_quantize));
  m.def("dequantize", torch::wrap_pybind_function_no_gil(dequantize));
  m.def("gemm", torch::wrap_pybind_function_no_gil(gemm));
  m.def("attention", torch::wrap_pybind_function_no_gil(attention));
}
