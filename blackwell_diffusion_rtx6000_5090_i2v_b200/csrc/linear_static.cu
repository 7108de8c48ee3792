// A whole NVFP4 linear (quantize the bf16 activation, block-scaled FP4 GEMM,
// fused bias / activation) that allocates nothing, for callers that cannot.
//
// The other entry points leave intermediate storage to the caller: the packed
// activation, its swizzled scales, the amax slot and the tensor scale are
// device buffers the caller allocates.  Some callers have no allocator to ask:
// code running inside a stream capture or another region where cudaMalloc is
// forbidden, real-time loops with a fixed memory budget, plug-ins that only
// receive input and output pointers from their host application.  For them the
// intermediates live in a fixed device array inside this library.
#include <mutex>

#include "nvfp4_common.cuh"

namespace nvfp4 {

// Largest activation the fixed scratch holds: 8 Mi elements (for example 2048 tokens of
// width 4096).  Footprint on every GPU that loads the library: 4 MiB of packed nibbles,
// 1 MiB of swizzled scales (room for row/K padding) and two fp32 slots.
constexpr int64_t kMaxElems = 8ll << 20;
constexpr int64_t kPackedBytes = kMaxElems / 2;
constexpr int64_t kScaleBytes = 2 * (kMaxElems / kBlock);
constexpr int64_t kSlotOffset = kPackedBytes + kScaleBytes;   // amax at +0, tensor scale at +4
constexpr int64_t kScratchBytes = kSlotOffset + 256;

// In host code this name is only a handle for cudaGetSymbolAddress, not a device address.
static __device__ __align__(256) uint8_t g_linear_scratch[kScratchBytes];

// Keeps the array in the module although no shipped kernel names it (never launched).
__global__ void linear_scratch_anchor(uint8_t* out) {
  if (out) *out = g_linear_scratch[0];
}

namespace {

std::mutex g_mu;
uint8_t* g_scratch_ptr[64];   // per device ordinal, resolved on first use

// Device address of the scratch array on the current device (null on failure).
uint8_t* scratch_for_current_device() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  std::lock_guard<std::mutex> lock(g_mu);
  if (!g_scratch_ptr[dev]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_linear_scratch) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    g_scratch_ptr[dev] = static_cast<uint8_t*>(p);
  }
  return g_scratch_ptr[dev];
}

// Workspace of the backward call: four packed operands, each followed by its swizzled scales, then
// scalar slots, partial maxima, and counters and partial sums for the bias.
struct BackwardLayout {
  int64_t dy, w_t, dy_t, x_t, slots, partials, counts, sums, total, k_m;
  static int64_t operand(int64_t rows, int64_t cols) {
    return (rows * cols / 2 + 255) / 256 * 256 + sf_swizzled_bytes(rows, cols);
  }
  BackwardLayout(int64_t M, int64_t N, int64_t K) : k_m((M + 31) / 32 * 32) {
    dy = 0;
    w_t = dy + operand(M, N);
    dy_t = w_t + operand(K, N);
    x_t = dy_t + operand(N, k_m);
    slots = x_t + operand(K, k_m);
    partials = slots + 256;
    counts = partials + (int64_t)sizeof(float) * NVFP4_AMAX_PARTIALS;
    sums = counts + (4 * quantize_job_col_tiles(N) + 255) / 256 * 256;
    total = sums + 4 * quantize_job_row_tiles(M) * quantize_job_col_tiles(N) * 64;
  }
};

}  // namespace
}  // namespace nvfp4

using namespace nvfp4;

extern "C" {

int64_t nvfp4_linear_bf16_static_max_elements(void) { return kMaxElems; }

int nvfp4_linear_bf16_static(const void* x_bf16, int64_t M, int64_t K, const uint8_t* w_packed,
                             const uint8_t* w_scales_swizzled, const float* w_global_scale_dev,
                             int64_t N, const void* bias_bf16, int act, void* y_bf16,
                             int* status_dev, void* stream) {
  if (M < 0 || K < 0 || N < 0 || K % 32 != 0 || N % 8 != 0) return NVFP4_ERR_BAD_ARG;
  // each extent on its own first, so that the products below cannot wrap
  if (M > kMaxElems || K > kMaxElems || N > (1 << 30)) return NVFP4_ERR_BAD_ARG;
  // The fixed scratch bounds the activation: M*K elements of nibbles, and the swizzled
  // scales, whose rows pad to 256 and K to 256 elements (so a very skinny activation can
  // exceed the scale area well below the element limit).  Larger problems must use the
  // caller-allocated path.
  if (M * K > kMaxElems || sf_swizzled_bytes(M, K) > kScaleBytes) return NVFP4_ERR_BAD_ARG;
  if (M == 0 || N == 0) return NVFP4_OK;
  if (K == 0 || !x_bf16 || !w_packed || !w_scales_swizzled || !y_bf16) return NVFP4_ERR_BAD_ARG;
  int rc = check_device_sm100();
  if (rc != NVFP4_OK) return rc;
  uint8_t* s = scratch_for_current_device();
  if (!s) return NVFP4_ERR_LAUNCH_FAILED;
  uint8_t* packed = s;
  uint8_t* scales = s + kPackedBytes;
  float* amax = reinterpret_cast<float*>(s + kSlotOffset);
  float* gscale = amax + 1;
  // amax zeroes its slot and quantize zeroes the scale padding: nothing of the previous
  // call's contents is read
  rc = nvfp4_amax_bf16(x_bf16, M * K, amax, stream);
  if (rc != NVFP4_OK) return rc;
  rc = nvfp4_quantize_bf16(x_bf16, M, K, amax, packed, nullptr, scales, gscale, stream);
  if (rc != NVFP4_OK) return rc;
  return nvfp4_gemm(packed, w_packed, scales, w_scales_swizzled, gscale, w_global_scale_dev, M, N,
                    K, 1.0f, 0.0f, nullptr, bias_bf16, nullptr, act, y_bf16, nullptr, status_dev, stream);
}

// workspace: packed activation | swizzled scales | amax and tensor scale | partial maxima
int64_t nvfp4_linear_workspace_bytes(int64_t M, int64_t K) {
  return (M * K / 2 + 255) / 256 * 256 + sf_swizzled_bytes(M, K) + 256 +
         (int64_t)sizeof(float) * NVFP4_AMAX_PARTIALS;
}

int nvfp4_linear_bf16(const void* x_bf16, int64_t M, int64_t K, const uint8_t* w_packed,
                      const uint8_t* w_scales_swizzled, const float* w_global_scale_dev, int64_t N,
                      const void* bias_bf16, const float* gate_f32, const void* residual_bf16, int act,
                      void* y_bf16, void* workspace, int* status_dev, void* stream) {
  if (M < 0 || K < 0 || N < 0 || K % 32 != 0 || N % 8 != 0) return NVFP4_ERR_BAD_ARG;
  if (M > (1 << 30) || N > (1 << 30) || K > (1 << 30)) return NVFP4_ERR_BAD_ARG;
  if (M == 0 || N == 0) return NVFP4_OK;
  if (K == 0 || !x_bf16 || !w_packed || !w_scales_swizzled || !y_bf16 || !workspace) return NVFP4_ERR_BAD_ARG;
  if (reinterpret_cast<uintptr_t>(workspace) & 255u) return NVFP4_ERR_BAD_ALIGN;
  uint8_t* packed = static_cast<uint8_t*>(workspace);
  uint8_t* scales = packed + (M * K / 2 + 255) / 256 * 256;
  float* amax = reinterpret_cast<float*>(scales + sf_swizzled_bytes(M, K));
  float* partials = amax + 64;
  const int rc = amax_quantize(x_bf16, M, K, amax, packed, nullptr, scales, amax + 1, partials, false, stream);
  if (rc != NVFP4_OK) return rc;
  return nvfp4_gemm(packed, w_packed, scales, w_scales_swizzled, amax + 1, w_global_scale_dev, M, N, K, 1.0f,
                    residual_bf16 ? 1.0f : 0.0f, residual_bf16, bias_bf16, gate_f32, act, y_bf16, nullptr,
                    status_dev, stream);
}

int64_t nvfp4_linear_backward_workspace_bytes(int64_t M, int64_t N, int64_t K) {
  return BackwardLayout(M, N, K).total;
}

// Four launches: the maxima of all operands, all operands packed (and the bias gradient), the two products.  The
// kernels of [2048, 3072] x 3072 take 60 us so, and took 89 as a launch or two per operand, memsets and torch's
// sum; the training pass, which waits for the host, 168 -> 138 us, and 110 with the native call in front.
// (dy's maximum is taken whatever is wanted, so with db alone for nothing: no caller in this package asks for that.)
int nvfp4_linear_backward_bias_bf16(const void* dy_bf16, const void* x_bf16, const void* w_bf16,
                                    const float* w_amax_dev, int64_t M, int64_t N, int64_t K, void* dx_bf16,
                                    void* dw_bf16, void* db_bf16, void* workspace, int* status_dev, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0 || N % 8 != 0 || K % 8 != 0 || (dx_bf16 && N % 32 != 0)) return NVFP4_ERR_BAD_ARG;
  if (M > (1 << 30) || N > (1 << 30) || K > (1 << 30)) return NVFP4_ERR_BAD_ARG;
  if (!dy_bf16 || !workspace || (dx_bf16 && !w_bf16) || (dw_bf16 && !x_bf16)) return NVFP4_ERR_BAD_ARG;
  const BackwardLayout at(M, N, K);
  // what the packing of the operands refuses: too many scale blocks in one of them
  const auto too_large = [](int64_t rows, int64_t cols) { return rows * cols / kBlock >= ((int64_t)1 << 31); };
  if ((dx_bf16 && (too_large(M, N) || too_large(N, K))) || (dw_bf16 && (too_large(at.k_m, N) || too_large(at.k_m, K))))
    return NVFP4_ERR_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(workspace) & 255u) || !aligned16(dy_bf16) || (dx_bf16 && !aligned16(w_bf16)) ||
      (dw_bf16 && !aligned16(x_bf16)))
    return NVFP4_ERR_BAD_ALIGN;
  int rc = check_device_sm100();
  if (rc != NVFP4_OK) return rc;
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  auto scales = [&](int64_t offset, int64_t rows, int64_t cols) {
    return ws + offset + (rows * cols / 2 + 255) / 256 * 256;
  };
  float* slot = reinterpret_cast<float*>(ws + at.slots);
  float *g_dy = slot, *g_wt = slot + 1, *g_dyt = slot + 2, *g_xt = slot + 3;
  float* partials = reinterpret_cast<float*>(ws + at.partials);
  unsigned* counts = reinterpret_cast<unsigned*>(ws + at.counts);

  QuantizeJob jobs[kQuantizeJobs] = {};
  QuantizeJob &dy = jobs[0], &x = jobs[1], &w = jobs[2];
  AmaxJob amax[3] = {};
  QuantizeJob* of[3];
  int n_amax = 0;
  auto add = [&](QuantizeJob& q, const void* data, int64_t rows, int64_t cols, const float* known) {
    q.x = data;
    q.rows = (uint32_t)rows;
    q.cols = (uint32_t)cols;
    q.amax = known;
    if (known) return;
    amax[n_amax].x = data;
    amax[n_amax].n = rows * cols;
    of[n_amax++] = &q;
  };
  auto transposed = [&](QuantizeJob& q, int64_t offset, float* gscale) {
    const int64_t k = ((int64_t)q.rows + 31) / 32 * 32;
    q.t_packed = reinterpret_cast<uint2*>(ws + offset);
    q.t_scales = scales(offset, q.cols, k);
    q.t_gscale = gscale;
    q.t_units = (uint32_t)(k / kBlock);
    q.t_k_atoms = (uint32_t)sf_k_atoms(k);
  };
  add(dy, dy_bf16, M, N, nullptr);       // its maximum does not depend on the direction
  if (dx_bf16) {
    dy.packed = reinterpret_cast<uint2*>(ws + at.dy);
    dy.scales = scales(at.dy, M, N);
    dy.gscale = g_dy;
    dy.units = (uint32_t)(N / kBlock);
    dy.k_atoms = (uint32_t)sf_k_atoms(N);
    add(w, w_bf16, N, K, w_amax_dev);
    transposed(w, at.w_t, g_wt);
  }
  if (dw_bf16) {
    transposed(dy, at.dy_t, g_dyt);
    add(x, x_bf16, M, K, nullptr);
    transposed(x, at.x_t, g_xt);
  }
  if (db_bf16) {
    dy.col_sum = static_cast<__nv_bfloat16*>(db_bf16);
    dy.col_partial = reinterpret_cast<float*>(ws + at.sums);
    dy.col_count = counts;
  }
  if (!dx_bf16 && !dw_bf16 && !db_bf16) return NVFP4_OK;
  rc = launch_amax_partials(amax, n_amax, partials, counts, db_bf16 ? (int)quantize_job_col_tiles(N) : 0, stream);
  for (int i = 0; i < n_amax; ++i) {
    of[i]->first_partial = amax[i].first;
    of[i]->n_partial = amax[i].count;
  }
  if (rc == NVFP4_OK) rc = quantize_jobs(jobs, partials, stream);
  if (rc == NVFP4_OK && dx_bf16)
    rc = nvfp4_gemm(ws + at.dy, ws + at.w_t, dy.scales, w.t_scales, g_dy, g_wt, M, K, N, 1.0f, 0.0f, nullptr, nullptr,
                    nullptr, NVFP4_ACT_NONE, dx_bf16, nullptr, status_dev, stream);
  if (rc == NVFP4_OK && dw_bf16)
    rc = nvfp4_gemm(ws + at.dy_t, ws + at.x_t, dy.t_scales, x.t_scales, g_dyt, g_xt, N, K, at.k_m, 1.0f, 0.0f, nullptr,
                    nullptr, nullptr, NVFP4_ACT_NONE, dw_bf16, nullptr, status_dev, stream);
  return rc;
}

int nvfp4_linear_backward_bf16(const void* dy_bf16, const void* x_bf16, const void* w_bf16,
                               const float* w_amax_dev, int64_t M, int64_t N, int64_t K, void* dx_bf16,
                               void* dw_bf16, void* workspace, int* status_dev, void* stream) {
  return nvfp4_linear_backward_bias_bf16(dy_bf16, x_bf16, w_bf16, w_amax_dev, M, N, K, dx_bf16, dw_bf16, nullptr,
                                         workspace, status_dev, stream);
}

}  // extern "C"
