// The Python layer's frequent calls in one native step each: argument checks, allocations, stream and
// library call.  Through ctypes these cost 11 to 38 us a call (a linear 27, a quantizer 21 to 28, norm + quantize
// 30 to 38), more than the kernels of a few thousand rows take.
//
// Every function returns None for what is not the plain case (other types, devices, layouts or alignments,
// tensor subclasses, an active dispatch mode, an empty tensor): the Python code that called it then does what it
// always did, errors included.  Nothing is kept between calls but the address of each device's status word.
//
// The calls let go of the interpreter lock, as the ctypes calls and torch's own allocations do: a launch waits where the
// stream's queue is full and an allocation may reach the driver, and neither needs the interpreter.  Their errors are
// torch's (an allocation that does not fit raises torch.OutOfMemoryError).
#include <ATen/TensorSubclassLikeUtils.h>
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
  m.def("norm_quantize", torch::wrap_pybind_function_no_gil(norm_quantize));
  m.def("dequantize", torch::wrap_pybind_function_no_gil(dequantize));
  m.def("gemm", torch::wrap_pybind_function_no_gil(gemm));
  m.def("attention", torch::wrap_pybind_function_no_gil(attention));
}
