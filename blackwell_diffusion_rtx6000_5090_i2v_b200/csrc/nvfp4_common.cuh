// Shared device/host helpers for the sm_100a NVFP4 kernels.
#pragma once

#include <cfloat>
#include <cstdint>

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>

#include "../../include/nvfp4_b200.h"

namespace nvfp4 {

constexpr int kBlock = 16;          // elements per scale block
constexpr int kSfAtomBytes = 512;   // 128 rows x 4 K-blocks
constexpr int kSfRowPad = 256;      // swizzled scale rows are padded to this
constexpr int kSfKbPad = 16;        // and K-blocks to this (= 256 elements)

// 128-row tiles and 4-block K atoms of the swizzled scale buffer.
__host__ __device__ inline int64_t sf_row_tiles(int64_t rows) {
  return (rows + kSfRowPad - 1) / kSfRowPad * (kSfRowPad / 128);
}
__host__ __device__ inline int64_t sf_k_atoms(int64_t cols) {
  return ((cols / kBlock) + kSfKbPad - 1) / kSfKbPad * (kSfKbPad / 4);
}
__host__ __device__ inline int64_t sf_swizzled_bytes(int64_t rows, int64_t cols) {
  return sf_row_tiles(rows) * sf_k_atoms(cols) * kSfAtomBytes;
}
// Byte offset of the scale of (row, K-block kb): atoms are [row tile][k atom],
// each atom is [32 rows][4 row groups][4 K-blocks].
__host__ __device__ inline int64_t sf_swizzled_offset(int64_t row, int64_t kb, int64_t k_atoms) {
  return ((row >> 7) * k_atoms + (kb >> 2)) * kSfAtomBytes + (row & 31) * 16 +
         ((row >> 5) & 3) * 4 + (kb & 3);
}

#ifdef __CUDACC__

// S_enc = min(448*6/amax, FLT_MAX); 1 when amax == 0 or the result is 0.
// IEEE division: the value must match the CPU restatement bit for bit.
__device__ __forceinline__ float global_encode_scale(float amax) {
  float s = __fdiv_rn(448.0f * 6.0f, amax);
  s = fminf(s, FLT_MAX);
  if (amax == 0.0f || s == 0.0f) return 1.0f;
  return s;
}

// x / 6, bit-identical to the IEEE quotient: one multiply by fl(1/6) and one residual
// correction (two FMAs).  The residual of a tiny quotient is itself inexact and that of an
// infinite one is NaN, so very small, very large and non-finite x take the division.  Checked
// against x / 6.0f for every bf16 x in the fast range and two million fp32 values.
__device__ __forceinline__ float div_by_6(float x) {
  const float c = 0x1.555556p-3f;
  const float q0 = __fmul_rn(x, c);
  const float q = __fmaf_rn(__fmaf_rn(-6.0f, q0, x), c, q0);
  return (x >= 1e-30f && x <= 1e37f) ? q : __fdiv_rn(x, 6.0f);
}

// E4M3 block scale: rn_satfinite( min( (amax_b / 6) * S_enc, FLT_MAX ) ).
__device__ __forceinline__ uint8_t block_scale_e4m3(float amax_b, float s_enc) {
  float d = __fmul_rn(__fdiv_rn(amax_b, 6.0f), s_enc);
  d = fminf(d, FLT_MAX);
  return (uint8_t)__nv_cvt_float_to_fp8(d, __NV_SATFINITE, __NV_E4M3);
}

__device__ __forceinline__ float e4m3_to_f32(uint8_t b) {
  __half_raw h = __nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)b, __NV_E4M3);
  return __half2float(__half(h));
}

// Element encode scale: min( 1 / (float(sf) * (1/S_enc)), FLT_MAX ).
__device__ __forceinline__ float block_encode_scale(uint8_t sf, float s_dec) {
  return fminf(__fdiv_rn(1.0f, __fmul_rn(e4m3_to_f32(sf), s_dec)), FLT_MAX);
}

// Eight floats -> eight E2M1 codes in one 32-bit word, element 0 in the low
// nibble of byte 0 (round to nearest even, saturate to +-6).
__device__ __forceinline__ uint32_t f32x8_to_e2m1x8(float v0, float v1, float v2, float v3,
                                                    float v4, float v5, float v6, float v7) {
  uint32_t out;
  asm("{\n\t"
      ".reg .b8 b0, b1, b2, b3;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n\t"
      "mov.b32 %0, {b0, b1, b2, b3};\n\t"
      "}"
      : "=r"(out)
      : "f"(v0), "f"(v1), "f"(v2), "f"(v3), "f"(v4), "f"(v5), "f"(v6), "f"(v7));
  return out;
}

__device__ __forceinline__ float bf16lo_to_f32(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16hi_to_f32(uint32_t w) {
  return __uint_as_float(w & 0xFFFF0000u);
}

// Two fp32 lanes per instruction (sm_100): each lane is rounded exactly like the scalar
// op, the pair costs one issue slot.
__device__ __forceinline__ float2 f2_add(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
      "add.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 f2_sub(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
      "sub.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 f2_mul(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
      "mul.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 f2_fma(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
      "mov.b64 rc, {%6, %7};\n\tfma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 bf16x2_to_f2(uint32_t w) {
  return make_float2(bf16lo_to_f32(w), bf16hi_to_f32(w));
}
// (lo, hi) -> packed bf16x2, round to nearest even: one instruction for the pair
__device__ __forceinline__ uint32_t f2_to_bf16x2(float2 v) {
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(v.y), "f"(v.x));
  return d;
}
// max(acc, |v|) per bf16 lane (inputs finite)
__device__ __forceinline__ uint32_t bf16x2_max_abs(uint32_t acc, uint32_t v) {
  uint32_t d;
  asm("{\n\t.reg .b32 t;\n\tabs.bf16x2 t, %2;\n\tmax.bf16x2 %0, %1, t;\n\t}"
      : "=r"(d) : "r"(acc), "r"(v));
  return d;
}

// One 16-element block, as eight bf16 pairs `h` whose packed maximum |h| is `a2`: its two words of
// E2M1 codes, and its E4M3 scale in `sf`.  `enc_tab` holds block_encode_scale() of every scale
// byte (fill_encode_table), so the reciprocal is computed 128 times per CTA and not per block.
__device__ __forceinline__ uint2 pack_block(const uint32_t (&h)[8], uint32_t a2, float s_enc,
                                            const float* enc_tab, uint32_t& sf) {
  const float amax_b = fmaxf(bf16lo_to_f32(a2), bf16hi_to_f32(a2));
  float d = __fmul_rn(div_by_6(amax_b), s_enc);
  d = fminf(d, FLT_MAX);
  sf = (uint32_t)__nv_cvt_float_to_fp8(d, __NV_SATFINITE, __NV_E4M3);
  const float enc = enc_tab[sf & 127];
  const float2 enc2 = make_float2(enc, enc);
  float2 q[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) q[e] = f2_mul(bf16x2_to_f2(h[e]), enc2);
  uint2 out;
  out.x = f32x8_to_e2m1x8(q[0].x, q[0].y, q[1].x, q[1].y, q[2].x, q[2].y, q[3].x, q[3].y);
  out.y = f32x8_to_e2m1x8(q[4].x, q[4].y, q[5].x, q[5].y, q[6].x, q[6].y, q[7].x, q[7].y);
  return out;
}
__device__ __forceinline__ void fill_encode_table(float* enc_tab, float s_dec) {
  for (int b = threadIdx.x; b < 128; b += blockDim.x) enc_tab[b] = block_encode_scale((uint8_t)b, s_dec);
}

// 4 x 4 byte transpose over a quad of lanes: lane l brings the scale bytes of rows 0..3 of K-block
// l, lane q leaves with those of K-blocks 0..3 of row q, which are adjacent in the swizzled layout.
// Whole warps only.
__device__ __forceinline__ uint32_t quad_transpose(uint32_t w) {
  const uint32_t lane = threadIdx.x;
  w = __byte_perm(w, __shfl_xor_sync(0xffffffffu, w, 1), (lane & 1) ? 0x3715u : 0x6240u);
  return __byte_perm(w, __shfl_xor_sync(0xffffffffu, w, 2), (lane & 2) ? 0x3276u : 0x5410u);
}

// A kernel launched by launch_dependent() may start while the kernel before it in its stream is still
// finishing.  This waits until everything before it has completed and is visible; what a kernel
// does ahead of it (barriers, tensor-memory allocation, index arithmetic) touches no global memory
// that another kernel writes or reads.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Loads for such a kernel.  Not __ldg and the like: those are non-coherent loads, for memory that
// stays read-only from the kernel's start to its end, which a predecessor's output is not, and nothing
// keeps them behind the wait.  These are ordinary loads, and as volatile statements they stay in
// order with it.  (`_once`: data with no second reader.)
__device__ __forceinline__ uint32_t load_u32(const void* p) {
  uint32_t v;
  asm volatile("ld.global.b32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float load_f32(const float* p) { return __uint_as_float(load_u32(p)); }
__device__ __forceinline__ float2 load_f32x2(const void* p) {
  float2 v;
  asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ float4 load_f32x4(const void* p) {
  float4 v;
  asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint4 load_u32x4(const void* p) {
  uint4 v;
  asm volatile("ld.global.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint4 load_u32x4_once(const void* p) {
  uint4 v;
  asm volatile("ld.global.cs.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// The maximum of this thread's share of a CTA's partial maxima (bits of non-negative floats): four at a time, all asked for
// before the first is needed.  One behind the other they were four trips to L2 ahead of a packing kernel's first block.
__device__ __forceinline__ unsigned max_of_partials(const unsigned* partial, int n) {
  unsigned m = 0u;
  for (int i = threadIdx.x; i < n; i += 4 * blockDim.x) {
    unsigned v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = load_u32(partial + min(i + j * (int)blockDim.x, n - 1));
    m = max(max(m, max(v[0], v[1])), max(v[2], v[3]));
  }
  return m;
}

// 32 bytes of x that are read once: one 256-bit load where the address allows, else two of 128.
__device__ __forceinline__ void load_block_once(const uint4* src, bool wide, uint32_t (&x)[8]) {
  if (wide) {
    asm volatile("ld.global.L1::no_allocate.L2::evict_first.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]), "=r"(x[4]), "=r"(x[5]), "=r"(x[6]), "=r"(x[7])
                 : "l"(src));
  } else {
    const uint4 a = load_u32x4_once(src), b = load_u32x4_once(src + 1);
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
    x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
  }
}

// Launch with programmatic stream serialization: the launch latency and the prologue of `kernel`
// overlap the tail of its predecessor, which costs a few microseconds a launch where kernels are short.
// No kernel that this may follow says before its end that the next may start.  (One does, attention's, to the
// launch of its own that shares the blocks left over, which waits for it at its end and so stands for it to
// whatever comes after.)  The kernel calls grid_dependency_wait() and loads as above.  `cluster`: CTAs per cluster along x.  Amax + pack of [27280, 3072] 67.7 -> 64.0 us, norm +
// quantize 98.0 -> 94.5 us, each called back to back; a GEMM or RoPE of that size within the spread of its
// runs.
template <typename... Params, typename... Args>
int launch_dependent(void (*kernel)(Params...), dim3 grid, unsigned threads, size_t smem, unsigned cluster,
                     cudaStream_t st, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  if (cudaLaunchKernelEx(&cfg, kernel, args...) != cudaSuccess) {
    cudaGetLastError();
    return NVFP4_ERR_LAUNCH_FAILED;
  }
  return cudaGetLastError() == cudaSuccess ? NVFP4_OK : NVFP4_ERR_LAUNCH_FAILED;
}

#endif  // __CUDACC__

// Host helpers shared by the entry points.
int check_device_sm100();                 // NVFP4_OK or NVFP4_ERR_UNSUPPORTED_ARCH (cached per device)
inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
int sm_count();                           // SMs of the current device (cached per device)

// nvfp4_amax_quantize_bf16, and whether nothing is known to follow it on the stream.
int amax_quantize(const void* x, int64_t rows, int64_t cols, float* amax_dev, uint8_t* packed, uint8_t* scales_linear,
                  uint8_t* scales_swizzled, float* global_scale_dev, float* partials, bool alone, void* stream);

// One tensor of launch_amax_partials(): n a multiple of 8, 16-byte aligned.  `first`, `count` are filled in.
struct AmaxJob {
  const void* x;
  int64_t n;
  int first, count;
};
int launch_amax_partials(AmaxJob (&jobs)[3], int n_jobs, float* partials, unsigned* zero, int n_zero, void* stream);

// One bf16 matrix of quantize_jobs() (x null: none), read once: its NVFP4 form, that of its transpose and its column
// sums, each where the pointers are given.
constexpr int kQuantizeJobs = 3;
struct QuantizeJob {
  const void* x;                 // [rows, cols], cols a multiple of 8
  uint32_t rows, cols;
  const float* amax;             // its maximum, where n_partial is 0
  int first_partial, n_partial;  // else which of the partial maxima are its own
  uint2* t_packed;               // transpose: [cols, rows padded to 32]
  uint8_t* t_scales;
  float* t_gscale;
  uint32_t t_units, t_k_atoms;   // scale blocks per row, K atoms
  uint2* packed;                 // itself: cols a multiple of 16
  uint8_t* scales;
  float* gscale;
  uint32_t units, k_atoms;
  __nv_bfloat16* col_sum;        // [cols]
  float* col_partial;            // scratch: [row tiles][column tiles * 64]
  unsigned* col_count;           // scratch: [column tiles], zeroed
  uint32_t col_tiles, row_tiles; // filled in
};
int64_t quantize_job_col_tiles(int64_t cols);
int64_t quantize_job_row_tiles(int64_t rows);
int quantize_jobs(const QuantizeJob (&jobs)[kQuantizeJobs], const float* partials, void* stream);

}  // namespace nvfp4
