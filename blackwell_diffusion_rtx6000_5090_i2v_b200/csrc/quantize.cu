// NVFP4 quantizer family for sm_100a: tensor amax, bf16 -> (E2M1 nibbles,
// E4M3 block scales, FP32 tensor scale), dequantize, scale re-layout.
//
// All kernels are HBM-bound byte movers: 128- and 256-bit loads, one 16-element scale
// block per thread so that the block amax needs no cross-lane traffic, and
// 64-bit packed stores.  Algorithmic bytes per element: 2 (bf16 in) + 0.5
// (nibbles) + 0.0625 (scale) = 2.5625.
//
// Four ways to pack, by shape (quantize_impl, nvfp4_amax_quantize_bf16):
//   small     amax and packing in one cluster of at most 8 CTAs that holds the tensor in registers
//   rows      a thread owns one scale block of every row, four rows at a time: rows that one CTA spans
//   resident  amax and packing in one cooperative launch that holds the tensor in shared memory
//   flat      blocks numbered through the tensor: everything else
#include <algorithm>
#include <atomic>

#include <cooperative_groups.h>

#include "nvfp4_common.cuh"

namespace nvfp4 {

namespace {

constexpr int kThreads = 256;
constexpr int kBlocksPerThread = 2;  // two 16-element scale blocks (64 B of input) per thread

// ---------------------------------------------------------------- amax ----

// Two forms.  For a slot: one atomic per CTA on the zeroed slot, any length.  In front of a packing kernel
// (kTensors > 0): every CTA leaves its own maximum in out[blockIdx.x] for that kernel to combine, so that no slot
// has to be zeroed first, launched by launch_dependent(); kTensors tensors share the launch, each with its own CTAs.
//
// Bound: HBM.  The second form has four 32-byte loads a thread on their way and four CTAs an SM.  kKeep: of a tensor
// that L2 does not hold it is asked to keep the last kKeptBytes, which the packing kernel reads first (and lets go).
// amax + pack, us, with 16-byte loads and eight CTAs an SM, without and with the hint: [27280, 3072] 62.4, 61.5, 60.1;
// 15000 rows 35.8, 34.8, 35.2; 4096 rows 12.1, 11.9, 11.7, but 35.1 instead of 34.6 with the GEMM behind it, whose operands
// and output want the room.
constexpr int64_t kKeptBytes = 60 << 20;
constexpr int64_t kKeepFrom = 126 << 20;      // the size of L2

template <int kTensors>
struct AmaxArgs {
  const uint4* x[kTensors];
  int64_t n_vec[kTensors];        // 16-byte pieces
  unsigned first[kTensors + 1];   // CTAs of tensor i: first[i] up to first[i + 1]
  unsigned wide;                  // bit i: tensor i starts on a 32-byte boundary
  unsigned* zero;                 // nullable: words that the next kernel wants zeroed
  int n_zero;
};

__device__ __forceinline__ uint32_t max_abs_u4(uint32_t m, const uint4& v) {
  return bf16x2_max_abs(bf16x2_max_abs(bf16x2_max_abs(bf16x2_max_abs(m, v.x), v.y), v.z), v.w);
}
// The CTA's maximum, on thread 0.  Non-negative floats order like their bit patterns.
__device__ __forceinline__ unsigned cta_max(float a) {
  __shared__ unsigned warp_max[kThreads / 32];
  unsigned bits = __reduce_max_sync(0xffffffffu, __float_as_uint(a));
  if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = bits;
  __syncthreads();
  if (threadIdx.x < 32) bits = __reduce_max_sync(0xffffffffu, threadIdx.x < kThreads / 32 ? warp_max[threadIdx.x] : 0u);
  return bits;
}

__global__ void __launch_bounds__(kThreads) amax_slot_kernel(const uint4* x, int64_t n_vec, const __nv_bfloat16* tail,
                                                             int n_tail, unsigned* out) {
  uint32_t m[4] = {0u, 0u, 0u, 0u};
  const int64_t stride = (int64_t)gridDim.x * kThreads;
  int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  // four independent 16-byte loads in flight per thread
  for (; i + 3 * stride < n_vec; i += 4 * stride) {
    uint4 v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = load_u32x4(x + i + j * stride);
#pragma unroll
    for (int j = 0; j < 4; ++j) m[j] = max_abs_u4(m[j], v[j]);
  }
  for (; i < n_vec; i += stride) m[0] = max_abs_u4(m[0], load_u32x4(x + i));
  const uint32_t h = bf16x2_max_abs(bf16x2_max_abs(bf16x2_max_abs(m[0], m[1]), m[2]), m[3]);
  float a = fmaxf(bf16lo_to_f32(h), bf16hi_to_f32(h));
  if (blockIdx.x == 0 && threadIdx.x < n_tail) a = fmaxf(a, fabsf(__bfloat162float(tail[threadIdx.x])));
  const unsigned b = cta_max(a);
  if (threadIdx.x == 0 && b != 0u) atomicMax(out, b);
}

// 32 bytes of x if they are there, else zeros, without a branch between one piece and the next.  kHint: they are there.
template <bool kHint>
__device__ __forceinline__ void load_if(const uint4* src, bool there, bool wide, uint64_t policy, uint32_t (&v)[8]) {
  if (!wide) {
    const uint4 none = make_uint4(0, 0, 0, 0), a = there ? load_u32x4(src) : none, b = there ? load_u32x4(src + 1) : none;
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else if (kHint) {
    asm volatile("ld.global.L1::no_allocate.L2::cache_hint.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8], %9;"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "l"(src), "l"(policy));
  } else {
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = 0u;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %8, 0;\n\t"
                 "@p ld.global.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%9];\n\t}"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7])
                 : "r"((int)there), "l"(src));
  }
}

template <int kTensors, bool kKeep>
__global__ void __launch_bounds__(kThreads) amax_bf16_kernel(const AmaxArgs<kTensors> p, unsigned* out) {
  const uint4* x = p.x[0];
  int64_t n_vec = p.n_vec[0];
  unsigned first = p.first[0], end = p.first[1], wide = p.wide & 1u;
#pragma unroll
  for (int k = 1; k < kTensors; ++k) {
    if (blockIdx.x >= p.first[k]) {
      x = p.x[k];
      n_vec = p.n_vec[k];
      first = p.first[k];
      end = p.first[k + 1];
      wide = p.wide >> k & 1u;
    }
  }
  uint64_t keep, drop;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(keep));
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(drop));
  grid_dependency_wait();
  if (blockIdx.x == 0)
    for (int i = threadIdx.x; i < p.n_zero; i += kThreads) p.zero[i] = 0u;
  const int64_t n = n_vec / 2, stride = (int64_t)(end - first) * kThreads, kept = n - kKeptBytes / 32;
  uint32_t m[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
  for (int64_t i = (int64_t)(blockIdx.x - first) * kThreads + threadIdx.x; i < n; i += 4 * stride) {
    uint32_t v[4][8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t at = i + j * stride;
      // past the end of a large tensor, for a few threads of all: the first piece again (predicates cost [27280, 3072] 0.2 us)
      load_if<kKeep>(x + 2 * (kKeep && at >= n ? i : at), kKeep || at < n, wide, at >= kept ? keep : drop, v[j]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int k = 0; k < 8; ++k) m[k] = bf16x2_max_abs(m[k], v[j][k]);
  }
  if ((n_vec & 1) && blockIdx.x == first && threadIdx.x == 0) m[0] = max_abs_u4(m[0], load_u32x4(x + n_vec - 1));
#pragma unroll
  for (int k = 1; k < 8; ++k) m[0] = bf16x2_max_abs(m[0], m[k]);
  const unsigned b = cta_max(fmaxf(bf16lo_to_f32(m[0]), bf16hi_to_f32(m[0])));
  if (threadIdx.x == 0) out[blockIdx.x] = b;
}

// ------------------------------------------------------------ quantize ----

// Flat form.  One thread quantizes kBlocksPerThread scale blocks.  Blocks are assigned so
// that in each of the j passes a warp reads 1 KiB of contiguous input.
__global__ void __launch_bounds__(kThreads)
quantize_bf16_kernel(const uint4* __restrict__ x, uint32_t n_blocks, uint32_t kb_per_row,
                     const float* __restrict__ amax_ptr, float amax_val,
                     uint2* __restrict__ packed, uint8_t* __restrict__ sf_lin,
                     uint8_t* __restrict__ sf_swz, uint32_t k_atoms,
                     float* __restrict__ global_scale_out) {
  const float amax_g = amax_ptr ? __ldg(amax_ptr) : amax_val;
  const float s_enc = global_encode_scale(amax_g);
  const float s_dec = __fdiv_rn(1.0f, s_enc);
  if (global_scale_out && blockIdx.x == 0 && threadIdx.x == 0) *global_scale_out = s_dec;

  // CTAs start at the END of the tensor: the amax pass that ran just before walked it
  // forwards, so its tail is what is still in L2 (126 MB) when this kernel begins
  const uint32_t base = (gridDim.x - 1u - blockIdx.x) * (kThreads * kBlocksPerThread) + threadIdx.x;
  uint4 v[kBlocksPerThread][2];
#pragma unroll
  for (int j = 0; j < kBlocksPerThread; ++j) {
    const uint32_t b = base + j * kThreads;
    if (b < n_blocks) {
      v[j][0] = __ldcs(x + 2 * (size_t)b);
      v[j][1] = __ldcs(x + 2 * (size_t)b + 1);
    } else {
      v[j][0] = make_uint4(0, 0, 0, 0);
      v[j][1] = make_uint4(0, 0, 0, 0);
    }
  }
  uint32_t row = 0, kb = 0;
  if (sf_swz) {
    row = base / kb_per_row;
    kb = base - row * kb_per_row;
  }
#pragma unroll
  for (int j = 0; j < kBlocksPerThread; ++j) {
    const uint32_t b = base + j * kThreads;
    const uint32_t w[8] = {v[j][0].x, v[j][0].y, v[j][0].z, v[j][0].w,
                           v[j][1].x, v[j][1].y, v[j][1].z, v[j][1].w};
    // block amax on the packed pairs (exact: the values are bf16), then widen once
    uint32_t a2 = 0u;
#pragma unroll
    for (int k = 0; k < 8; ++k) a2 = bf16x2_max_abs(a2, w[k]);
    const float amax_b = fmaxf(bf16lo_to_f32(a2), bf16hi_to_f32(a2));
    // (amax_b / 6) * S_enc -> E4M3; 1 / (float(sf) * S_dec): both quotients IEEE-rounded
    float d = __fmul_rn(div_by_6(amax_b), s_enc);
    d = fminf(d, FLT_MAX);
    const uint8_t sf = (uint8_t)__nv_cvt_float_to_fp8(d, __NV_SATFINITE, __NV_E4M3);
    const float enc = fminf(__frcp_rn(__fmul_rn(e4m3_to_f32(sf), s_dec)), FLT_MAX);
    const float2 enc2 = make_float2(enc, enc);
    float2 q[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) q[k] = f2_mul(bf16x2_to_f2(w[k]), enc2);
    uint2 out;
    out.x = f32x8_to_e2m1x8(q[0].x, q[0].y, q[1].x, q[1].y, q[2].x, q[2].y, q[3].x, q[3].y);
    out.y = f32x8_to_e2m1x8(q[4].x, q[4].y, q[5].x, q[5].y, q[6].x, q[6].y, q[7].x, q[7].y);
    if (b < n_blocks) {
      __stcs(packed + b, out);
      if (sf_lin) sf_lin[b] = sf;
      if (sf_swz) sf_swz[sf_swizzled_offset(row, kb, k_atoms)] = sf;
    }
    if (sf_swz) {  // advance (row, kb) by kThreads blocks
      kb += kThreads;
      while (kb >= kb_per_row) {
        kb -= kb_per_row;
        ++row;
      }
    }
  }
}

// Rows form.  Bound: HBM.  The walk is backwards over the rows (the tail of x is what the amax pass
// left in L2); the loads of kRows rows are in flight together; the scale bytes of 4 rows x 4
// K-blocks are transposed between the lanes of a quad and leave as 4-byte stores (16 single bytes
// before); the pad rows and K-blocks of the swizzled layout are written as zeros here instead of
// by a memset ahead of the kernel.
constexpr int kPackThreads = 192;
constexpr int kPackWide = 320;       // the wider of the two CTAs
constexpr int kRows = 4;

struct PackArgs {
  const uint4* x;
  int64_t rows;
  int units;                  // scale blocks per row
  const float* amax;          // device slot, or null: amax_val
  float amax_val;
  const unsigned* partial;    // per-CTA maxima (float bits) instead of a slot
  int n_partial;
  float* amax_out;            // with `partial`: receives the maximum
  uint2* packed;
  uint8_t* sf_lin;
  uint8_t* sf_swz;
  uint32_t k_atoms;
  float* gscale_out;
  int wide_x;                 // x starts on a 32-byte boundary
  int word_swz;               // sf_swz starts on a 4-byte boundary
};

// kMax: most threads of a CTA, kPackThreads or kPackWide.
constexpr int pack_ctas(int max) { return max == kPackThreads ? 4 : 3; }
template <int kMax>
__global__ void __launch_bounds__(kMax, pack_ctas(kMax)) pack_rows_kernel(const PackArgs p) {
  __shared__ float enc_tab[128];
  __shared__ unsigned warp_max[kMax / 32];
  const int u = threadIdx.x;
  const bool live = u < p.units;
  const bool in_layout = u < (int)p.k_atoms * 4;
  const bool scribe = blockIdx.x == 0 && threadIdx.x == 0;
  grid_dependency_wait();
  float amax_g;
  if (p.partial) {
    unsigned m = 0u;
    m = max_of_partials(p.partial, p.n_partial);
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = m;
    __syncthreads();
    for (int w = 0; w < (int)blockDim.x / 32; ++w) m = max(m, warp_max[w]);
    amax_g = __uint_as_float(m);
    if (scribe) *p.amax_out = amax_g;
  } else {
    amax_g = p.amax ? load_f32(p.amax) : p.amax_val;
  }
  const float s_enc = global_encode_scale(amax_g);
  const float s_dec = __fdiv_rn(1.0f, s_enc);
  if (p.gscale_out && scribe) *p.gscale_out = s_dec;
  fill_encode_table(enc_tab, s_dec);
  __syncthreads();

  const int quad = threadIdx.x & 3;
  const int64_t swz_u = (int64_t)(u >> 2) * kSfAtomBytes + quad * 16;
  const int64_t all_rows = p.sf_swz ? sf_row_tiles(p.rows) * 128 : p.rows;
  const int64_t groups = (all_rows + kRows - 1) / kRows;
  for (int64_t g = blockIdx.x; g < groups; g += gridDim.x) {
    const int64_t base = (groups - 1 - g) * kRows;
    uint32_t sf4 = 0u;
    if (base < p.rows) {
      // rows past the end and threads without a block repeat another's loads and keep quiet
      uint32_t x[kRows][8];
#pragma unroll
      for (int r = 0; r < kRows; ++r) {
        const int64_t row = base + r < p.rows ? base + r : p.rows - 1;
        load_block_once(p.x + row * p.units * 2 + 2 * (live ? u : 0), p.wide_x, x[r]);
      }
#pragma unroll
      for (int r = 0; r < kRows; ++r) {
        uint32_t a2 = 0u, sf;
#pragma unroll
        for (int e = 0; e < 8; ++e) a2 = bf16x2_max_abs(a2, x[r][e]);
        const uint2 out = pack_block(x[r], a2, s_enc, enc_tab, sf);
        if (live && base + r < p.rows) {
          const int64_t blk = (base + r) * p.units + u;
          __stcs(p.packed + blk, out);
          if (p.sf_lin) p.sf_lin[blk] = (uint8_t)sf;
          sf4 |= sf << (8 * r);
        }
      }
    }
    if (p.sf_swz) {
      sf4 = quad_transpose(sf4);      // row base + quad of the quad's four K-blocks
      if (in_layout) {
        uint8_t* dst = p.sf_swz + (base >> 7) * (int64_t)p.k_atoms * kSfAtomBytes + (base & 31) * 16 +
                       ((base >> 5) & 3) * 4 + swz_u;
        if (p.word_swz) {
          *reinterpret_cast<uint32_t*>(dst) = sf4;
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) dst[i] = (uint8_t)(sf4 >> (8 * i));
        }
      }
    }
  }
}

// Small form: amax and packing of a tensor that one cluster of CTAs holds in registers, kB blocks
// per thread.  Bound: latency -- one launch and one read of x where the other forms take a memset,
// two kernels and, for the pad of the swizzled scales, another memset.
constexpr int kSmallThreads = 512;
constexpr int kSmallCtas = 8;            // the portable cluster size
constexpr int kSmallBlocks = 8;          // most blocks per thread
constexpr int64_t kSmallMax = (int64_t)kSmallCtas * kSmallThreads * kSmallBlocks;
// Above four blocks a thread the other forms are faster where they apply: [85, 3072] 4.7 us small, 4.8 rows;
// [170, 3072] 6.8 small, 4.7 rows, 5.4 resident.
constexpr int64_t kSmallBest = kSmallMax / 2;
// Most bytes of swizzled scales, which the cluster zeroes: a few long rows are mostly pad, and a memset
// has the whole GPU for it ([1, 65536], 1 MB: 9.7 us with memsets and two kernels, 5.0 here; [1, 262144],
// 4 MB: 10.3 and 12.7; [1, 524288], 8 MB: 10.4 and 23).
constexpr int64_t kSmallPad = 2 << 20;

template <int kB>
__global__ void __launch_bounds__(kSmallThreads)
quantize_small_kernel(const uint4* x, uint32_t n_blocks, uint32_t kb_per_row, int wide_x,
                      float* __restrict__ amax_out, uint2* __restrict__ packed,
                      uint8_t* __restrict__ sf_lin, uint8_t* sf_swz, uint32_t swz_vecs,
                      uint32_t k_atoms, float* __restrict__ gscale_out) {
  __shared__ unsigned warp_max[kSmallThreads / 32];
  __shared__ unsigned cta_max;
  const uint32_t ctas = gridDim.x, rank = blockIdx.x;      // the grid is one cluster
  const uint32_t first = rank * kSmallThreads + threadIdx.x, stride = ctas * kSmallThreads;
  grid_dependency_wait();
  uint32_t v[kB][8];
  uint32_t a2[kB];
#pragma unroll
  for (int j = 0; j < kB; ++j) {
    const uint32_t b = first + j * stride;
    if (b < n_blocks) load_block_once(x + 2 * (size_t)b, wide_x, v[j]);
  }
  // the scale bytes of real blocks go over these zeros after the cluster barrier
  for (uint32_t i = first; i < swz_vecs; i += stride)
    reinterpret_cast<uint4*>(sf_swz)[i] = make_uint4(0, 0, 0, 0);
  uint32_t m2 = 0u;
#pragma unroll
  for (int j = 0; j < kB; ++j) {
    a2[j] = 0u;
    if (first + j * stride < n_blocks) {
#pragma unroll
      for (int e = 0; e < 8; ++e) a2[j] = bf16x2_max_abs(a2[j], v[j][e]);
      m2 = bf16x2_max_abs(m2, a2[j]);
    }
  }
  unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(bf16lo_to_f32(m2), bf16hi_to_f32(m2))));
  if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    m = __reduce_max_sync(0xffffffffu, threadIdx.x < kSmallThreads / 32 ? warp_max[threadIdx.x] : 0u);
    if (threadIdx.x == 0) cta_max = m;
  }
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  unsigned all = 0u;
  const uint32_t slot = (uint32_t)__cvta_generic_to_shared(&cta_max);
  for (uint32_t r = 0; r < ctas; ++r) {
    uint32_t addr;
    unsigned o;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(slot), "r"(r));
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(o) : "r"(addr) : "memory");
    all = max(all, o);
  }
  // no CTA leaves while another may still read its maximum
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  const float amax_g = __uint_as_float(all);
  const float s_enc = global_encode_scale(amax_g);
  const float s_dec = __fdiv_rn(1.0f, s_enc);
  if (first == 0) {
    *amax_out = amax_g;
    if (gscale_out) *gscale_out = s_dec;
  }
#pragma unroll
  for (int j = 0; j < kB; ++j) {
    const uint32_t b = first + j * stride;
    if (b < n_blocks) {
      const float amax_b = fmaxf(bf16lo_to_f32(a2[j]), bf16hi_to_f32(a2[j]));
      const float d = fminf(__fmul_rn(div_by_6(amax_b), s_enc), FLT_MAX);
      const uint8_t sf = (uint8_t)__nv_cvt_float_to_fp8(d, __NV_SATFINITE, __NV_E4M3);
      const float enc = block_encode_scale(sf, s_dec);
      const float2 enc2 = make_float2(enc, enc);
      float2 q[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) q[e] = f2_mul(bf16x2_to_f2(v[j][e]), enc2);
      uint2 out;
      out.x = f32x8_to_e2m1x8(q[0].x, q[0].y, q[1].x, q[1].y, q[2].x, q[2].y, q[3].x, q[3].y);
      out.y = f32x8_to_e2m1x8(q[4].x, q[4].y, q[5].x, q[5].y, q[6].x, q[6].y, q[7].x, q[7].y);
      packed[b] = out;
      if (sf_lin) sf_lin[b] = sf;
      if (sf_swz) {
        const uint32_t row = b / kb_per_row;
        sf_swz[sf_swizzled_offset(row, b - row * kb_per_row, k_atoms)] = sf;
      }
    }
  }
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

// Resident form: amax and packing of a tensor that the shared memory of the GPU holds.  Bound: HBM and the
// meeting of the grid between the two.  Every thread copies its blocks there (asynchronously, all on their way
// at once), takes their maximum, and packs them when the grid's is known: x is read once, in one launch.
constexpr int kHeldThreads = 512;
constexpr int kHeldBlocks = 6;           // most blocks per thread: two CTAs of 96 KB an SM

__global__ void __launch_bounds__(kHeldThreads, 2)
quantize_resident_kernel(const uint4* x, uint32_t n_blocks, uint32_t kb_per_row, int per, unsigned* partial,
                         float* amax_out, uint2* packed, uint8_t* sf_lin, uint8_t* sf_swz, uint32_t swz_vecs,
                         uint32_t k_atoms, float* gscale_out) {
  extern __shared__ __align__(16) uint4 held[];       // [block of the thread][half][thread]
  __shared__ unsigned warp_max[kHeldThreads / 32];
  __shared__ float enc_tab[128];
  const int t = threadIdx.x;
  const uint32_t stride = gridDim.x * kHeldThreads, first = blockIdx.x * kHeldThreads + t;
  for (int i = 0; i < per; ++i) {
    const uint32_t b = first + i * stride;
    if (b < n_blocks) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(held + (2 * i + h) * kHeldThreads + t);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(x + 2 * (size_t)b + h) : "memory");
      }
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  // the scale bytes of real blocks go over these zeros once the grid has met
  for (uint32_t i = first; i < swz_vecs; i += stride) reinterpret_cast<uint4*>(sf_swz)[i] = make_uint4(0, 0, 0, 0);
  asm volatile("cp.async.wait_all;" ::: "memory");    // a thread reads what it copied, and nothing else
  uint32_t m2 = 0u;
  for (int i = 0; i < per; ++i) {
    if (first + i * stride < n_blocks) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint4 v = held[(2 * i + h) * kHeldThreads + t];
        m2 = bf16x2_max_abs(bf16x2_max_abs(bf16x2_max_abs(bf16x2_max_abs(m2, v.x), v.y), v.z), v.w);
      }
    }
  }
  unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(bf16lo_to_f32(m2), bf16hi_to_f32(m2))));
  if ((t & 31) == 0) warp_max[t >> 5] = m;
  __syncthreads();
  if (t < 32) {
    m = __reduce_max_sync(0xffffffffu, t < kHeldThreads / 32 ? warp_max[t] : 0u);
    if (t == 0) partial[blockIdx.x] = m;
  }
  cooperative_groups::this_grid().sync();
  m = 0u;
  for (unsigned i = t; i < gridDim.x; i += kHeldThreads) m = max(m, load_u32(partial + i));
  m = __reduce_max_sync(0xffffffffu, m);
  if ((t & 31) == 0) warp_max[t >> 5] = m;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kHeldThreads / 32; ++w) m = max(m, warp_max[w]);
  const float amax_g = __uint_as_float(m);
  const float s_enc = global_encode_scale(amax_g);
  const float s_dec = __fdiv_rn(1.0f, s_enc);
  if (first == 0) {
    *amax_out = amax_g;
    if (gscale_out) *gscale_out = s_dec;
  }
  fill_encode_table(enc_tab, s_dec);
  __syncthreads();
  for (int i = 0; i < per; ++i) {
    const uint32_t b = first + i * stride;
    if (b >= n_blocks) break;
    const uint4 v0 = held[2 * i * kHeldThreads + t], v1 = held[(2 * i + 1) * kHeldThreads + t];
    const uint32_t h[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
    uint32_t a2 = 0u, sf;
#pragma unroll
    for (int e = 0; e < 8; ++e) a2 = bf16x2_max_abs(a2, h[e]);
    const uint2 out = pack_block(h, a2, s_enc, enc_tab, sf);
    __stcs(packed + b, out);
    if (sf_lin) sf_lin[b] = (uint8_t)sf;
    if (sf_swz) {
      const uint32_t row = b / kb_per_row;
      sf_swz[sf_swizzled_offset(row, b - row * kb_per_row, k_atoms)] = (uint8_t)sf;
    }
  }
}

// ---------------------------------------------------------- dequantize ----

// x = e2m1 * (float(sf) / S_enc), S_enc derived from the tensor amax (device slot or by value);
// IEEE division, so the bits match the CPU restatement of the reference formula.
//
// Bound: HBM, 2.5625 B/element.  A scale byte and a magnitude code leave only 256 x 8 possible
// results, so each CTA tabulates them once (low bytes, then high bytes, of the eight bf16 values
// of a scale byte: one 16-byte shared-memory read per block) and an element costs byte selections
// instead of a decode, a multiply and a conversion, a block no division.  [14336, 3072]: 47.1 -> 24.2 us
// through to_bfloat16() (2.4 -> 4.7 TB/s), the call's host part included.  A thread with few blocks in
// all (`direct`) makes its own entries instead, and the first loads are on their way meanwhile: small
// tensors are all latency ([64, 3072], replayed from a graph: 2.4 us with the table, 2.0 without).
constexpr int kDequantBlocks = 2;    // scale blocks in flight per thread

__device__ __forceinline__ void decode4(uint32_t codes, const uint4& t, uint32_t signs, uint32_t& o0,
                                        uint32_t& o1) {
  // four codes -> their low and high bytes -> two bf16 pairs; bit 3 of a code flips the sign
  const uint32_t sel = codes & 0x7777u;
  const uint32_t lo = __byte_perm(t.x, t.y, sel), hi = __byte_perm(t.z, t.w, sel);
  o0 = __byte_perm(lo, hi, 0x5140) ^ (((codes & 0x88u) * 0x1001000u) & signs);
  o1 = __byte_perm(lo, hi, 0x7362) ^ (((codes & 0x8800u) * 0x10010u) & signs);
}

__device__ __forceinline__ uint4 dequant_entry(uint32_t sf, float s_enc) {
  const float d = __fdiv_rn(e4m3_to_f32((uint8_t)sf), s_enc);
  const float mag[8] = {0.0f, 0.5f, 1.0f, 1.5f, 2.0f, 3.0f, 4.0f, 6.0f};
  uint32_t v[4];
#pragma unroll
  for (int k = 0; k < 4; ++k)
    v[k] = f2_to_bf16x2(make_float2(__fmul_rn(mag[2 * k], d), __fmul_rn(mag[2 * k + 1], d)));
  return make_uint4(__byte_perm(v[0], v[1], 0x6420), __byte_perm(v[2], v[3], 0x6420),
                    __byte_perm(v[0], v[1], 0x7531), __byte_perm(v[2], v[3], 0x7531));
}

__global__ void __launch_bounds__(kThreads)
dequantize_bf16_kernel(const uint32_t* __restrict__ packed, const uint8_t* __restrict__ sf_lin,
                       int64_t n_blocks, const float* __restrict__ amax_ptr, float amax_val,
                       uint4* __restrict__ out, int word2, int wide_out, int direct) {
  __shared__ uint4 table[256];
  const int64_t stride = (int64_t)gridDim.x * kThreads;
  uint2 p[kDequantBlocks];
  uint32_t sf[kDequantBlocks];
  auto load = [&](int64_t i) {
#pragma unroll
    for (int j = 0; j < kDequantBlocks; ++j) {
      const int64_t b = i + j * stride;
      if (b < n_blocks) {
        p[j] = word2 ? __ldcs(reinterpret_cast<const uint2*>(packed) + b)
                     : make_uint2(__ldcs(packed + 2 * b), __ldcs(packed + 2 * b + 1));
        sf[j] = __ldcs(sf_lin + b);
      }
    }
  };
  int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  load(i);       // on their way while the table is made: a small tensor is all latency
  const float s_enc = global_encode_scale(amax_ptr ? __ldg(amax_ptr) : amax_val);
  if (!direct) {
    for (int b = threadIdx.x; b < 256; b += kThreads) table[b] = dequant_entry(b, s_enc);
    __syncthreads();
  }
  for (; i < n_blocks; i += kDequantBlocks * stride) {
#pragma unroll
    for (int j = 0; j < kDequantBlocks; ++j) {
      const int64_t b = i + j * stride;
      if (b < n_blocks) {
        const uint4 t = direct ? dequant_entry(sf[j], s_enc) : table[sf[j]];
        const uint32_t signs = (sf[j] & 127u) == 127u ? 0u : 0x80008000u;   // a NaN scale: one NaN
        uint32_t o[8];
        decode4(p[j].x & 0xFFFFu, t, signs, o[0], o[1]);
        decode4(p[j].x >> 16, t, signs, o[2], o[3]);
        decode4(p[j].y & 0xFFFFu, t, signs, o[4], o[5]);
        decode4(p[j].y >> 16, t, signs, o[6], o[7]);
        uint4* dst = out + 2 * b;
        if (wide_out) {
          asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                       ::"l"(dst), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7])
                       : "memory");
        } else {
          dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
          dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
        }
      }
    }
    load(i + kDequantBlocks * stride);
  }
}

// -------------------------------------------------------------- swizzle ----

__global__ void __launch_bounds__(kThreads)
swizzle_scales_kernel(const uint8_t* __restrict__ lin, int64_t n_sf, uint32_t kb_per_row,
                      uint32_t k_atoms, uint8_t* __restrict__ swz) {
  const int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (i >= n_sf) return;
  const int64_t row = i / kb_per_row;
  const int64_t kb = i - row * kb_per_row;
  swz[sf_swizzled_offset(row, kb, k_atoms)] = lin[i];
}

int launch_status() {
  return cudaGetLastError() == cudaSuccess ? NVFP4_OK : NVFP4_ERR_LAUNCH_FAILED;
}

// Zero the pad region of a swizzled scale buffer so that padded rows / K-blocks
// decode to 0 (a pad byte of 0x7F would be NaN and poison the accumulators).
int zero_swizzle_padding(uint8_t* swz, int64_t rows, int64_t cols, cudaStream_t st) {
  const int64_t kb = cols / kBlock;
  const int64_t total = sf_swizzled_bytes(rows, cols);
  if (kb % kSfKbPad != 0) {
    return cudaMemsetAsync(swz, 0, (size_t)total, st) == cudaSuccess ? NVFP4_OK
                                                                      : NVFP4_ERR_LAUNCH_FAILED;
  }
  if (rows % 128 != 0 || sf_row_tiles(rows) * 128 != (rows + 127) / 128 * 128) {
    const int64_t first = (rows / 128) * sf_k_atoms(cols) * kSfAtomBytes;  // first partial tile
    return cudaMemsetAsync(swz + first, 0, (size_t)(total - first), st) == cudaSuccess
               ? NVFP4_OK
               : NVFP4_ERR_LAUNCH_FAILED;
  }
  return NVFP4_OK;
}

// The rows form takes rows that one CTA spans with at least three quarters of its threads (1152 to 5120 columns), and
// enough of them for kRows at a time: [27280, 3072] amax + pack 77.8 us flat with its two memsets, 60.1 rows.  Rows of more
// than 3072 columns have a wider CTA of their own kernel, since three of 320 threads an SM instead of four of 192 cost the
// narrower ones ([32760, 3072] 77 instead of 74): through the public call flat and rows [15000, 4096] 55.9 and 46.8, [32760,
// 4096] 108 and 97, [16000, 5120] 70.2 and 58.7.  Much wider rows are better off in the flat form, whose CTAs read one
// contiguous piece each ([27280, 14336] 291 us, 302-350 with five CTAs side by side on a row).
bool rows_form(int64_t rows, int64_t cols, bool swz, int* threads) {
  const int64_t units = swz ? sf_k_atoms(cols) * 4 : cols / kBlock;
  *threads = (int)((units + 31) / 32 * 32);
  return rows >= 32 && units <= kPackWide && *threads >= 96 && cols / kBlock * 4 >= (int64_t)*threads * 3;
}

int check_quantize(const void* x, int64_t rows, int64_t cols, const uint8_t* packed) {
  if (rows < 0 || cols < 0 || cols % kBlock != 0) return NVFP4_ERR_BAD_ARG;
  // each extent first, so that the product cannot wrap; then at most 2^31 - 1 scale blocks
  if (rows >= ((int64_t)1 << 31) || cols >= ((int64_t)1 << 31)) return NVFP4_ERR_BAD_ARG;
  const int64_t n_blocks = rows * cols / kBlock;
  if (n_blocks >= (int64_t)1 << 31) return NVFP4_ERR_BAD_ARG;
  if (n_blocks == 0) return NVFP4_OK;
  if (!x || !packed) return NVFP4_ERR_BAD_ARG;
  if (!aligned16(x) || (reinterpret_cast<uintptr_t>(packed) & 7u)) return NVFP4_ERR_BAD_ALIGN;
  return check_device_sm100();
}

template <int kMax>
int launch_rows_of(const PackArgs& a, int threads, cudaStream_t st) {
  const int64_t all_rows = a.sf_swz ? sf_row_tiles(a.rows) * 128 : a.rows;
  const int64_t groups = (all_rows + kRows - 1) / kRows;
  // CTAs per SM by the launch bound's registers, more of narrower ones
  const int64_t resident = (int64_t)sm_count() * (pack_ctas(kMax) * kMax / threads);
  return launch_dependent(pack_rows_kernel<kMax>, dim3((unsigned)(groups < resident ? groups : resident)),
                          (unsigned)threads, 0, 1, st, a);
}
int launch_rows(const PackArgs& a, int threads, cudaStream_t st) {
  return threads <= kPackThreads ? launch_rows_of<kPackThreads>(a, threads, st) : launch_rows_of<kPackWide>(a, threads, st);
}

int quantize_impl(const void* x, int64_t rows, int64_t cols, const float* amax_dev, float amax_val,
                  uint8_t* packed, uint8_t* sf_lin, uint8_t* sf_swz, float* gscale, void* stream) {
  int rc = check_quantize(x, rows, cols, packed);
  const int64_t n_blocks = rows * cols / kBlock;
  if (rc != NVFP4_OK || n_blocks == 0) return rc;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  int threads;
  // With the maximum known the flat form is one kernel where the layout has no pad, and then the rows
  // form (its table, a CTA's idle lanes) pays only for long tensors and nearly full CTAs.  Replayed from a
  // graph, us flat and rows: [256, 3072] 2.4 and 2.9, [4096, 3072] 6.1 and 6.1, [16384, 3072] 19.9 and
  // 18.8, [16384, 1280] 8.9 and 9.2; with a pad, and so a memset, [170, 3072] 3.9 and 2.8.
  // The wider CTAs pay only with a pad, and those of more than 224 threads (3584 columns) not for long tensors: flat and rows,
  // with a pad [32, 5120] 3.5 and 2.9, [1000, 4096] 4.6 and 3.4, [4095, 5120] 11.3 and 10.3, [8191, 5120] 18.8 and 17.7, [10001, 5120]
  // 22.9 and 23.1, [32760, 5120] 67.2 and 70.3, but [32760, 3280] 45.4 and 44.9; without [4096, 4096] 7.7 and 7.9, [16384, 5120]
  // 34.1 and 35.4, linear scales only [4096, 5120] 8.0 and 9.4.
  const bool pads = sf_swz && (rows % 256 != 0 || cols / kBlock % kSfKbPad != 0);
  const auto pays = [&] {
    if (threads > kPackThreads) return pads && (threads <= 224 || n_blocks <= 3 << 20);
    return pads || (n_blocks >= (1 << 20) && cols / kBlock * 8 >= (int64_t)threads * 7);
  };
  if (rows_form(rows, cols, sf_swz != nullptr, &threads) && pays()) {
    PackArgs a{};
    a.x = reinterpret_cast<const uint4*>(x);
    a.rows = rows;
    a.units = (int)(cols / kBlock);
    a.amax = amax_dev;
    a.amax_val = amax_val;
    a.packed = reinterpret_cast<uint2*>(packed);
    a.sf_lin = sf_lin;
    a.sf_swz = sf_swz;
    a.k_atoms = (uint32_t)sf_k_atoms(cols);
    a.gscale_out = gscale;
    a.wide_x = (reinterpret_cast<uintptr_t>(x) & 31u) == 0;
    a.word_swz = (reinterpret_cast<uintptr_t>(sf_swz) & 3u) == 0;
    return launch_rows(a, threads, st);
  }
  if (sf_swz) {
    rc = zero_swizzle_padding(sf_swz, rows, cols, st);
    if (rc != NVFP4_OK) return rc;
  }
  const int per_cta = kThreads * kBlocksPerThread;
  const unsigned grid = (unsigned)((n_blocks + per_cta - 1) / per_cta);
  quantize_bf16_kernel<<<grid, kThreads, 0, st>>>(
      reinterpret_cast<const uint4*>(x), (uint32_t)n_blocks, (uint32_t)(cols / kBlock), amax_dev,
      amax_val, reinterpret_cast<uint2*>(packed), sf_lin, sf_swz, (uint32_t)sf_k_atoms(cols),
      gscale);
  return launch_status();
}

unsigned amax_grid(int64_t n_vec) {
  const int64_t want = (n_vec + kThreads * 4 - 1) / (kThreads * 4);
  const int64_t most = NVFP4_AMAX_PARTIALS;
  return (unsigned)(want < 1 ? 1 : (want > most ? most : want));
}

// CTAs of amax_bf16_kernel: a thread has four pieces of 32 bytes, and four CTAs fit an SM.  (One piece a thread of a small
// tensor, and the first piece again for those past the end, amax + pack, us: [500, 3072] 5.27 -> 4.70, [2000, 1152] 6.55 -> 5.30,
// [900, 5120] with a GEMM of 5120 columns behind it 24.8 -> 24.0.)
int64_t wanted_ctas(int64_t n_vec) { return std::max<int64_t>((n_vec / 2 + 4 * kThreads - 1) / (4 * kThreads), 1); }
int64_t most_ctas() { return std::min<int64_t>(4 * (int64_t)sm_count(), NVFP4_AMAX_PARTIALS); }
unsigned partial_grid(int64_t n_vec) { return (unsigned)std::min(wanted_ctas(n_vec), most_ctas()); }
unsigned wide_bit(const void* x) { return (reinterpret_cast<uintptr_t>(x) & 31u) == 0; }

// Launches the resident form if the tensor fits; *done says whether.
int launch_resident(const void* x, int64_t rows, int64_t cols, float* amax, uint8_t* packed, uint8_t* sf_lin,
                    uint8_t* sf_swz, float* gscale, float* partials, cudaStream_t st, bool* done) {
  const int64_t n_blocks = rows * cols / kBlock, ctas_max = 2 * (int64_t)sm_count();
  const int64_t per = (n_blocks + ctas_max * kHeldThreads - 1) / (ctas_max * kHeldThreads);
  if (per > kHeldBlocks || ctas_max > NVFP4_AMAX_PARTIALS) return NVFP4_OK;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return NVFP4_ERR_BAD_ARG;
  static std::atomic<bool> allowed[64];
  if (!allowed[dev].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(quantize_resident_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kHeldBlocks * kHeldThreads * 32) != cudaSuccess)
      return NVFP4_ERR_LAUNCH_FAILED;
    allowed[dev].store(true, std::memory_order_release);
  }
  const size_t smem = (size_t)per * kHeldThreads * 32;
  const int64_t ctas = (n_blocks + per * kHeldThreads - 1) / (per * kHeldThreads);
  // CTAs that an SM holds, plus one; asked for once (a launch that is refused would invalidate a stream capture)
  static std::atomic<int> known[64][kHeldBlocks + 1];
  int an_sm = known[dev][per].load(std::memory_order_acquire);
  if (an_sm == 0) {
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&an_sm, quantize_resident_kernel, kHeldThreads, smem) != cudaSuccess) {
      cudaGetLastError();
      return NVFP4_OK;
    }
    known[dev][per].store(++an_sm, std::memory_order_release);
  }
  if (ctas > (int64_t)sm_count() * (an_sm - 1)) return NVFP4_OK;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3(kHeldThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeCooperative;
  attr.val.cooperative = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(
      &cfg, quantize_resident_kernel, reinterpret_cast<const uint4*>(x), (uint32_t)n_blocks, (uint32_t)(cols / kBlock), (int)per,
      reinterpret_cast<unsigned*>(partials), amax, reinterpret_cast<uint2*>(packed), sf_lin, sf_swz,
      (uint32_t)(sf_swz ? sf_swizzled_bytes(rows, cols) / 16 : 0), (uint32_t)sf_k_atoms(cols), gscale);
  if (e == cudaSuccess) {
    *done = true;
    return NVFP4_OK;
  }
  cudaGetLastError();
  // fewer SMs than the device has: the other forms run on any number
  return e == cudaErrorCooperativeLaunchTooLarge ? NVFP4_OK : NVFP4_ERR_LAUNCH_FAILED;
}

template <int kB>
int launch_small(const void* x, int64_t rows, int64_t cols, float* amax, uint8_t* packed, uint8_t* sf_lin,
                 uint8_t* sf_swz, float* gscale, int ctas, cudaStream_t st) {
  return launch_dependent(
      quantize_small_kernel<kB>, dim3((unsigned)ctas), kSmallThreads, 0, (unsigned)ctas, st,
      reinterpret_cast<const uint4*>(x), (uint32_t)(rows * cols / kBlock), (uint32_t)(cols / kBlock),
      (int)((reinterpret_cast<uintptr_t>(x) & 31u) == 0), amax, reinterpret_cast<uint2*>(packed), sf_lin, sf_swz,
      (uint32_t)(sf_swz ? sf_swizzled_bytes(rows, cols) / 16 : 0), (uint32_t)sf_k_atoms(cols), gscale);
}

}  // namespace

// The maxima of up to three tensors in one launch, each tensor's CTAs in proportion to its size: `job.first` and
// `job.count` say which of the partial maxima are a tensor's.
int launch_amax_partials(AmaxJob (&jobs)[3], int n_jobs, float* partials, unsigned* zero, int n_zero, void* stream) {
  const int64_t most = most_ctas();
  int64_t want = 0;
  for (int i = 0; i < n_jobs; ++i) want += wanted_ctas(jobs[i].n / 8);
  AmaxArgs<3> a{};
  unsigned next = 0;
  for (int i = 0; i < 3; ++i) {
    a.first[i] = next;
    if (i >= n_jobs) continue;
    const int64_t n_vec = jobs[i].n / 8;
    int64_t ctas = wanted_ctas(n_vec);
    // rounded down, and three single CTAs at most on top of that: no more than there is room for
    if (want > most) ctas = ctas * (most - 3) / want + 1;
    a.x[i] = static_cast<const uint4*>(jobs[i].x);
    a.n_vec[i] = n_vec;
    a.wide |= wide_bit(jobs[i].x) << i;
    jobs[i].first = (int)next;
    jobs[i].count = (int)ctas;
    next += (unsigned)ctas;
  }
  a.first[3] = next;
  a.zero = zero;
  a.n_zero = n_zero;
  return launch_dependent(amax_bf16_kernel<3, false>, dim3(next), kThreads, 0, 1, reinterpret_cast<cudaStream_t>(stream), a,
                          reinterpret_cast<unsigned*>(partials));
}

// Wide rows in up to this many blocks are packed in one launch where the caller says nothing of what follows
// (amax_quantize): the public entry cannot know, nvfp4_linear_bf16 does.
constexpr int64_t kAloneBlocks = 480 << 10;

// `alone`: nothing is known to follow on the stream (something may: a program that quantizes and multiplies in two calls).
int amax_quantize(const void* x, int64_t rows, int64_t cols, float* amax_dev, uint8_t* packed, uint8_t* scales_linear,
                  uint8_t* scales_swizzled, float* global_scale_dev, float* partials, bool alone, void* stream) {
  int rc = check_quantize(x, rows, cols, packed);
  if (rc != NVFP4_OK) return rc;
  if (!amax_dev) return NVFP4_ERR_BAD_ARG;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int64_t n_blocks = rows * cols / kBlock;
  const bool small_fits = n_blocks > 0 && n_blocks <= kSmallMax && aligned16(scales_swizzled) &&
                          (!scales_swizzled || sf_swizzled_bytes(rows, cols) <= kSmallPad);
  auto small = [&]() {
    // as few blocks per thread as the cluster allows: latency is what counts here
    int ctas = 1;
    while (ctas < kSmallCtas && n_blocks > (int64_t)ctas * kSmallThreads) ctas *= 2;
    const int64_t per = (n_blocks + (int64_t)ctas * kSmallThreads - 1) / ((int64_t)ctas * kSmallThreads);
#define NVFP4_SMALL(B) \
  launch_small<B>(x, rows, cols, amax_dev, packed, scales_linear, scales_swizzled, global_scale_dev, ctas, st)
    return per <= 1 ? NVFP4_SMALL(1) : per <= 2 ? NVFP4_SMALL(2) : per <= 4 ? NVFP4_SMALL(4) : NVFP4_SMALL(8);
#undef NVFP4_SMALL
  };
  if (small_fits && n_blocks <= kSmallBest) return small();
  int threads;
  if (n_blocks > 0 && partials && rows_form(rows, cols, scales_swizzled != nullptr, &threads) &&
      !(alone && threads > kPackThreads && n_blocks <= kAloneBlocks)) {
    const int64_t n_vec = n_blocks * 2;
    const unsigned grid = partial_grid(n_vec);
    const AmaxArgs<1> first{{reinterpret_cast<const uint4*>(x)}, {n_vec}, {0u, grid}, wide_bit(x), nullptr, 0};
    rc = n_blocks * 32 > kKeepFrom ? launch_dependent(amax_bf16_kernel<1, true>, dim3(grid), kThreads, 0, 1, st, first,
                                                      reinterpret_cast<unsigned*>(partials))
                                   : launch_dependent(amax_bf16_kernel<1, false>, dim3(grid), kThreads, 0, 1, st, first,
                                                      reinterpret_cast<unsigned*>(partials));
    if (rc != NVFP4_OK) return rc;
    PackArgs a{};
    a.x = reinterpret_cast<const uint4*>(x);
    a.rows = rows;
    a.units = (int)(cols / kBlock);
    a.partial = reinterpret_cast<const unsigned*>(partials);
    a.n_partial = (int)grid;
    a.amax_out = amax_dev;
    a.packed = reinterpret_cast<uint2*>(packed);
    a.sf_lin = scales_linear;
    a.sf_swz = scales_swizzled;
    a.k_atoms = (uint32_t)sf_k_atoms(cols);
    a.gscale_out = global_scale_dev;
    a.wide_x = (reinterpret_cast<uintptr_t>(x) & 31u) == 0;
    a.word_swz = (reinterpret_cast<uintptr_t>(scales_swizzled) & 3u) == 0;
    return launch_rows(a, threads, st);
  }
  // What the rows form does not take: the resident form where the tensor fits.  Not ahead of the rows form, whose two
  // kernels overlap what comes before and each other: us, resident and rows, [4095, 4096] 23.1 and 15.9, [4095, 5120] 23.1 and 16.6
  // (both bound by the host from there down); with a GEMM behind it 512 x 3072 x 4096 (M, N, K) 18.2 and 15.8, 900 x 5120 x 5120 29.2
  // and 26.8, 2500 x 5120 x 5120 46.7 and 42.4, 300 x 15360 x 5120 29.2 and 27.6.  But a few wide rows of a caller that says
  // nothing of a GEMM are a matter of launches: through the public call [512, 4096] 14.4 and 16.0, [1500, 5120] 14.8 and 15.8.
  // (Where that caller has a GEMM follow all the same, and no host time to save, it pays the difference above.)
  if (n_blocks > 0 && partials && aligned16(scales_swizzled) &&
      (!scales_swizzled || sf_swizzled_bytes(rows, cols) <= n_blocks * 4)) {
    bool done = false;
    rc = launch_resident(x, rows, cols, amax_dev, packed, scales_linear, scales_swizzled, global_scale_dev, partials, st,
                         &done);
    if (rc != NVFP4_OK || done) return rc;
  }
  if (small_fits) return small();
  rc = nvfp4_amax_bf16(x, rows * cols, amax_dev, stream);
  if (rc != NVFP4_OK) return rc;
  return quantize_impl(x, rows, cols, amax_dev, 0.0f, packed, scales_linear, scales_swizzled,
                       global_scale_dev, stream);
}

}  // namespace nvfp4

using namespace nvfp4;

extern "C" {

int nvfp4_amax_bf16(const void* x, int64_t n, float* amax_dev, void* stream) {
  if (n < 0 || !amax_dev) return NVFP4_ERR_BAD_ARG;
  int rc = check_device_sm100();
  if (rc != NVFP4_OK) return rc;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(amax_dev, 0, sizeof(float), st) != cudaSuccess)
    return NVFP4_ERR_LAUNCH_FAILED;
  if (n == 0) return NVFP4_OK;
  if (!x) return NVFP4_ERR_BAD_ARG;
  if (!aligned16(x)) return NVFP4_ERR_BAD_ALIGN;
  const int64_t n_vec = n / 8;
  const int n_tail = (int)(n - n_vec * 8);
  amax_slot_kernel<<<amax_grid(n_vec), kThreads, 0, st>>>(
      reinterpret_cast<const uint4*>(x), n_vec, reinterpret_cast<const __nv_bfloat16*>(x) + n_vec * 8, n_tail,
      reinterpret_cast<unsigned*>(amax_dev));
  return launch_status();
}

int64_t nvfp4_swizzled_scale_bytes(int64_t rows, int64_t cols) {
  return sf_swizzled_bytes(rows, cols);
}

int nvfp4_quantize_bf16(const void* x, int64_t rows, int64_t cols, const float* amax_dev,
                        uint8_t* packed, uint8_t* scales_linear, uint8_t* scales_swizzled,
                        float* global_scale_dev, void* stream) {
  // an empty tensor reads nothing, not even the amax slot
  if (!amax_dev && rows > 0 && cols > 0) return NVFP4_ERR_BAD_ARG;
  return quantize_impl(x, rows, cols, amax_dev, 0.0f, packed, scales_linear, scales_swizzled,
                       global_scale_dev, stream);
}

int nvfp4_amax_quantize_bf16(const void* x, int64_t rows, int64_t cols, float* amax_dev, uint8_t* packed,
                             uint8_t* scales_linear, uint8_t* scales_swizzled, float* global_scale_dev,
                             float* partials, void* stream) {
  return amax_quantize(x, rows, cols, amax_dev, packed, scales_linear, scales_swizzled, global_scale_dev, partials, true,
                       stream);
}

int nvfp4_quantize_bf16_amax(const void* x, uint8_t* packed, uint8_t* scales, int64_t n,
                             float global_amax, void* stream) {
  if (n < 0 || n % kBlock != 0) return NVFP4_ERR_BAD_ARG;
  if (n > 0 && !scales) return NVFP4_ERR_BAD_ARG;
  return quantize_impl(x, 1, n, nullptr, global_amax, packed, scales, nullptr, nullptr, stream);
}

static int dequantize_impl(const uint8_t* packed, const uint8_t* scales, int64_t n,
                           const float* amax_dev, float amax_val, void* out, void* stream) {
  if (n < 0 || n % kBlock != 0 || n / kBlock >= ((int64_t)1 << 31)) return NVFP4_ERR_BAD_ARG;
  if (n == 0) return NVFP4_OK;
  if (!packed || !scales || !out) return NVFP4_ERR_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(packed) & 3u) || !aligned16(out)) return NVFP4_ERR_BAD_ALIGN;
  int rc = check_device_sm100();
  if (rc != NVFP4_OK) return rc;
  const int64_t n_blocks = n / kBlock;
  const int direct = n_blocks <= (int64_t)sm_count() * kThreads;
  const int per_thread = direct ? 1 : kDequantBlocks;
  const int64_t want = (n_blocks + kThreads * per_thread - 1) / (kThreads * per_thread);
  const int64_t resident = (int64_t)sm_count() * 8;       // 2048 threads per SM
  dequantize_bf16_kernel<<<(unsigned)(want < resident ? want : resident), kThreads, 0,
                           reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const uint32_t*>(packed), scales, n_blocks, amax_dev, amax_val,
      reinterpret_cast<uint4*>(out), (reinterpret_cast<uintptr_t>(packed) & 7u) == 0,
      (reinterpret_cast<uintptr_t>(out) & 31u) == 0, direct);
  return launch_status();
}

int nvfp4_dequantize_bf16(const uint8_t* packed, const uint8_t* scales_linear, int64_t rows,
                          int64_t cols, const float* amax_dev, void* out_bf16, void* stream) {
  if (rows < 0 || cols < 0 || cols % kBlock != 0 || !amax_dev) return NVFP4_ERR_BAD_ARG;
  if (rows >= ((int64_t)1 << 31) || cols >= ((int64_t)1 << 31)) return NVFP4_ERR_BAD_ARG;
  return dequantize_impl(packed, scales_linear, rows * cols, amax_dev, 0.0f, out_bf16,
                         stream);
}

int nvfp4_dequantize_bf16_amax(const uint8_t* packed, const uint8_t* scales, void* out_bf16,
                               int64_t n, float global_amax, void* stream) {
  return dequantize_impl(packed, scales, n, nullptr, global_amax, out_bf16, stream);
}

int nvfp4_swizzle_scales(const uint8_t* scales_linear, int64_t rows, int64_t cols,
                         uint8_t* scales_swizzled, void* stream) {
  if (rows < 0 || cols < 0 || cols % kBlock != 0) return NVFP4_ERR_BAD_ARG;
  if (rows >= ((int64_t)1 << 31) || cols >= ((int64_t)1 << 31)) return NVFP4_ERR_BAD_ARG;
  const int64_t n_sf = rows * cols / kBlock;
  if (n_sf >= (int64_t)1 << 32) return NVFP4_ERR_BAD_ARG;      // the grid would not fit
  if (n_sf == 0) return NVFP4_OK;
  if (!scales_linear || !scales_swizzled) return NVFP4_ERR_BAD_ARG;
  int rc = check_device_sm100();
  if (rc != NVFP4_OK) return rc;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  rc = zero_swizzle_padding(scales_swizzled, rows, cols, st);
  if (rc != NVFP4_OK) return rc;
  const unsigned grid = (unsigned)((n_sf + kThreads - 1) / kThreads);
  swizzle_scales_kernel<<<grid, kThreads, 0, st>>>(scales_linear, n_sf, (uint32_t)(cols / kBlock),
                                                   (uint32_t)sf_k_atoms(cols), scales_swizzled);
  return launch_status();
}

}  // extern "C"
