// LayerNorm / RMSNorm + adaLN modulation fused with the NVFP4 quantizer.
//
//   h = bf16( ((x - mean) * rstd * w + b) * (1 + scale) + shift )      (fp32 math)
//   h -> packed E2M1 + E4M3 block scales + FP32 tensor scale
//
// replaces, for the inputs of the DiT block's QKV / Q / FFN-up linears, the
// chain norm -> modulation -> cast -> amax -> quantize
// (fx/src/s4/models/wan22/wan_transformer.py:204-206, 210, 218-220).  The
// per-tensor amax forces two sweeps; both read only x (2 B/element each) and
// recompute h, so h itself never travels: 4 + 0.5625 bytes per element moved
// against 2 + 2 + 2 + 2 + 0.5625 for the unfused chain.
//
// Work split.  A thread owns whole 16-element scale blocks: kJ of them per row
// (T * kJ * 16 >= cols for a CTA of T threads), the same columns in every row, so its slice of
// the per-column vectors (w, b, 1 + scale, shift) is loaded once into registers and costs
// nothing per row, and a block's scale needs no exchange between threads.  A CTA walks over
// many groups of kR consecutive rows.  A group is one contiguous piece of x, fetched by a
// single bulk copy into a ring of kStages shared-memory slots that completes an mbarrier;
// kStages - 1 groups are always in flight per CTA, which is what keeps HBM busy -- no register
// holds data that is still on its way.
//
// Instruction count is what limits a kernel like this once the copies are off the critical
// path (an earlier form spent 25 instructions per element and ran at a third of HBM speed), so:
// fp32 math runs two lanes per instruction (f32x2) with each lane rounded as the scalar op;
// the bf16 rounding, |h| and its maximum are packed bf16x2 ops; the row statistics take one
// pass and ONE CTA-wide reduction per group (sums of x - pivot and its square, the pivot
// being the row's first element, which keeps S2/n - (S1/n)^2 away from cancellation), whose
// warp stage folds the 2 kR values instead of reducing them one by one; the divisions of
// the quantizer are gone (x/6 by an exact three-operation form, the encode scale from a
// 128-entry table per tensor); scale offsets split into a per-row and a per-thread part.
// What is known of a call is a template parameter (kWhole), the widening of x is part of its subtraction, |h| and its
// maximum are one instruction, and the means' divisions are three operations.  Both sweeps, us, before and after:
// [27280, 3072] modulation 96.4 -> 81.7, affine 96.4 -> 80.6, all four vectors 147 -> 117, [32760, 5120] modulation 186 -> 156,
// [12000, 6384] 152 -> 122; 31 M -> 24 M and 28 M instructions.
// Sweep 1 leaves mean and rstd per row in a small stats buffer so that sweep 2, which needs
// no reduction at all, repeats exactly the same arithmetic.
//
// Sweep 1 walks the groups forwards and sweep 2 walks them backwards with an evict-first
// hint: the tail of x that sweep 1 left in L2 (126 MB) is what sweep 2 reads first.
#include <atomic>
#include <type_traits>

#include <cooperative_groups.h>

#include "nvfp4_common.cuh"

namespace nvfp4 {
namespace {

constexpr int kMaxThreads = 512;
constexpr int kMaxJ = 2;          // 2 blocks x 16 elements x 512 threads = 16384 columns
constexpr int kMaxWarps = kMaxThreads / 32;
#ifndef NVFP4_NORM_STAGES
#define NVFP4_NORM_STAGES 3
#endif
constexpr int kStages = NVFP4_NORM_STAGES;
constexpr long long kWaitCycles = 4000000000LL;   // about two seconds; then give up
constexpr int kErrCopyTimeout = 0x900;            // status code: a row group never arrived

#ifndef NVFP4_NORM_R1
#define NVFP4_NORM_R1 2
#endif
// rows per group: a slot is at most 64 KB (cols <= 8192 * kJ)
template <int kJ> struct RowsPerIter { static constexpr int value = kJ == 1 ? NVFP4_NORM_R1 : 2; };

struct NormArgs {
  const uint4* x;
  int64_t rows;
  int cols;
  const float* w;
  const float* b;
  const float* scale;
  const float* shift;
  int rms;
  float eps;
  float* stats;              // [rows][2] mean, rstd: written by sweep 1, read by sweep 2
  unsigned* amax_out;        // sweep 1
  uint4* h_out;              // sweep 1, optional
  const float* amax_in;      // sweep 2
  uint32_t* packed;          // sweep 2
  uint8_t* sf_lin;
  uint8_t* sf_swz;
  uint32_t k_atoms;
  int pad_rows;              // sweep 2: rows of the swizzled layout past `rows` that it has to zero
  float* gscale_out;
  int* status;               // nullable; receives kErrCopyTimeout
};

__device__ __forceinline__ void load16(const float* p, float2 (&d)[8]) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float4 a = load_f32x4(p + 4 * q);
    d[2 * q] = make_float2(a.x, a.y);
    d[2 * q + 1] = make_float2(a.z, a.w);
  }
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
// Contiguous global -> this CTA's shared memory, bytes reported to `bar`.  One destination,
// nothing broadcast.  Addresses 16-byte aligned, size a multiple of 16.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar,
                                          int hint) {
  if (hint != 0) {
    uint64_t policy;
    if (hint == 1) {
      asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
    } else {
      asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(policy));
    }
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint "
        "[%0], [%1], %2, [%3], %4;"
        ::"r"(dst), "l"(src), "r"(bytes), "r"(bar), "l"(policy) : "memory");
  } else {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
        ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
  }
}

// Bounded wait for a row group.  On expiry (or once any thread of the CTA has given up) the
// caller carries on without the data: every later barrier is still reached by all threads,
// the outputs of this CTA are then meaningless and the status word says so.
__device__ __forceinline__ void wait_group(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                           int* status) {
  if (mbar_try_wait(bar, parity)) return;
  const long long t0 = clock64();
  for (uint32_t it = 1;; ++it) {
    if (mbar_try_wait(bar, parity)) return;
    if ((it & 255u) == 0) {
      if (*abort_flag) return;
      if (clock64() - t0 > kWaitCycles) {
        *abort_flag = 1;
        if (status) atomicCAS(status, 0, kErrCopyTimeout);
        return;
      }
    }
  }
}

// x / n, bit-identical to the IEEE quotient, with `inv` the rounded reciprocal of n: a product and one residual
// correction (P. Markstein, IBM J. Res. Dev. 34, 1990).  Where the residual is not exact or not a number, the division.
template <bool kFast>
__device__ __forceinline__ float div_by(float x, float n, float inv) {
  if (!kFast) return __fdiv_rn(x, n);
  const float q0 = __fmul_rn(x, inv);
  const float q = __fmaf_rn(__fmaf_rn(-n, q0, x), inv, q0);
  const float a = fabsf(x);
  return (a >= 1e-25f && a <= 1e37f) ? q : __fdiv_rn(x, n);
}

// One fold step of the multi-value warp sum: a lane hands kHalf of its 2*kHalf values to the
// partner across `mask` and keeps the sums of the other kHalf.
template <int kHalf>
__device__ __forceinline__ void fold_step(float* v, bool upper, int mask) {
#pragma unroll
  for (int i = 0; i < kHalf; ++i) {
    const float keep = upper ? v[i + kHalf] : v[i];
    const float give = upper ? v[i] : v[i + kHalf];
    v[i] = keep + __shfl_xor_sync(0xffffffffu, give, mask);
  }
}

// Sum over the CTA of kV values per thread; every thread gets all kV totals, added in a
// fixed order.  Inside a warp the values are folded (kV + 2 shuffles for kV = 8 instead of
// 40).  `red` is one of two buffers used alternately, which makes one barrier per reduction
// enough: a buffer is rewritten only after the barrier of the reduction in between.
template <int kV>
__device__ __forceinline__ void cta_sum(float (&v)[kV], float (*red)[kMaxWarps], int warps) {
  static_assert(kV == 1 || kV == 2 || kV == 4 || kV == 8, "fold needs a power of two <= 8");
  constexpr int n0 = kV, n1 = n0 > 1 ? n0 / 2 : 1, n2 = n1 > 1 ? n1 / 2 : 1;
  const int lane = threadIdx.x & 31;
  int idx = 0;      // which of the kV values this lane ends up holding
  int mask = 16;
  if constexpr (n0 > 1) {
    const bool up = (lane & mask) != 0;
    fold_step<n0 / 2>(v, up, mask);
    idx += up ? n0 / 2 : 0;
    mask >>= 1;
  }
  if constexpr (n1 > 1) {
    const bool up = (lane & mask) != 0;
    fold_step<n1 / 2>(v, up, mask);
    idx += up ? n1 / 2 : 0;
    mask >>= 1;
  }
  if constexpr (n2 > 1) {
    const bool up = (lane & mask) != 0;
    fold_step<n2 / 2>(v, up, mask);
    idx += up ? n2 / 2 : 0;
    mask >>= 1;
  }
  for (int o = mask; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
  if ((lane & (2 * mask - 1)) == 0) red[idx][threadIdx.x >> 5] = v[0];
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kV; ++r) {
    float t = 0.0f;
    for (int w4 = 0; w4 < warps; w4 += 4) {
      const float4 q = *reinterpret_cast<const float4*>(&red[r][w4]);   // unused slots hold 0
      t += (q.x + q.y) + (q.z + q.w);
    }
    v[r] = t;
  }
}

// Both lanes of a bf16 pair minus m, in fp32 (exact widening, one rounding): no instruction for the widening.
__device__ __forceinline__ float2 bf16x2_sub(uint32_t w, float m) {
  float2 d;
  asm("{\n\t.reg .b16 lo, hi;\n\tmov.b32 {lo, hi}, %2;\n\tsub.rn.f32.bf16 %0, lo, %3;\n\tsub.rn.f32.bf16 %1, hi, %3;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "r"(w), "f"(m));
  return d;
}

// h for one 16-element block as 8 packed bf16 pairs, and the running bf16x2 max of |h| and a2, whose signs mean nothing.
// kMixed: widening and mean in one subtraction a lane (sweep 2 has fewer instructions the other way, but with all four vectors:
// [27280, 3072] affine 82.0 -> 80.6 us, modulation 82.1 -> 81.7, all four 116.9 -> 117.1).
template <bool kAffine, bool kMod, bool kMixed>
__device__ __forceinline__ uint32_t normalize16(uint32_t a2, const uint32_t (&xp)[8], float2 m2, float2 r2,
                                                const float2 (&cw)[8], const float2 (&cb)[8],
                                                const float2 (&cs)[8], const float2 (&ct)[8],
                                                bool has_w, bool has_b, bool has_s, bool has_t,
                                                uint32_t (&hp)[8]) {
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    float2 y = f2_mul(kMixed ? bf16x2_sub(xp[e], m2.x) : f2_sub(bf16x2_to_f2(xp[e]), m2), r2);
    if (kAffine) {
      if (has_w) y = f2_mul(y, cw[e]);
      if (has_b) y = f2_add(y, cb[e]);
    }
    if (kMod) {
      if (has_s) y = f2_mul(y, cs[e]);
      if (has_t) y = f2_add(y, ct[e]);
    }
    // the quantizer's input is the bf16 tensor the unfused model would have produced
    hp[e] = f2_to_bf16x2(y);
    asm("max.xorsign.abs.bf16x2 %0, %0, %1;" : "+r"(a2) : "r"(hp[e]));     // one instruction, where abs and max are two
  }
  return a2;
}

// The maximum of m and |h| of a block, h before its rounding to bf16: rounding keeps the order, so that the rounded
// maximum is the maximum of the rounded (NaNs are passed over by both).  One three-operand instruction a pair.
template <bool kAffine, bool kMod>
__device__ __forceinline__ float max_normed16(float m, const uint32_t (&xp)[8], float mean, float2 r2, const float2 (&cw)[8],
                                              const float2 (&cb)[8], const float2 (&cs)[8], const float2 (&ct)[8]) {
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    float2 y = f2_mul(bf16x2_sub(xp[e], mean), r2);
    if (kAffine) y = f2_add(f2_mul(y, cw[e]), cb[e]);
    if (kMod) y = f2_add(f2_mul(y, cs[e]), ct[e]);
    asm("max.abs.f32 %0, %0, %1, %2;" : "+f"(m) : "f"(y.x), "f"(y.y));
  }
  return m;
}

// kWhole: both vectors of every kind are given and every thread has blocks (T * kJ * 16 == cols), so that nothing of that
// is asked for each pair of elements or block.
template <bool kQuantize, int kJ, bool kAffine, bool kMod, bool kWhole>
__global__ void __launch_bounds__(kMaxThreads)
norm_mod_kernel(const NormArgs p) {
  constexpr int kR = RowsPerIter<kJ>::value;
  constexpr int kV = 2 * kR;                                // (sum, sum of squares) per row
  extern __shared__ __align__(128) uint8_t ring[];          // kStages slots of kR rows
  __shared__ __align__(16) float red[2][kV][kMaxWarps];
  __shared__ float red_max[kMaxWarps];
  __shared__ float enc_tab[128];                            // sweep 2: encode scale per scale byte
  __shared__ __align__(8) uint64_t full[kStages];
  __shared__ int abort_flag;
  const int T = blockDim.x;
  const int warps = T >> 5;
  const int units = p.cols >> 4;                            // 16-element blocks per row
  const uint32_t row_bytes = (uint32_t)p.cols * 2u;
  const uint32_t slot_bytes = row_bytes * kR;
  const int64_t groups = (p.rows + kR - 1) / kR;

  // group g of this CTA's walk -> first row and byte count (sweep 2 mirrors the order)
  auto group_base = [&](int64_t g) { return (kQuantize ? groups - 1 - g : g) * kR; };
  auto issue = [&](int64_t g, int slot) {
    const int64_t base = group_base(g);
    const int64_t n = p.rows - base < kR ? p.rows - base : kR;
    const uint32_t bytes = (uint32_t)n * row_bytes;
    const uint32_t bar = smem_u32(&full[slot]);
    mbar_expect_tx(bar, bytes);
#ifdef NVFP4_NORM_TAIL_MB
    const int64_t tail_rows = ((int64_t)NVFP4_NORM_TAIL_MB << 20) / row_bytes;
    const int hint = kQuantize ? 1 : (base >= p.rows - tail_rows ? 2 : 1);
#else
    const int hint = kQuantize ? 1 : 0;
#endif
    bulk_load(smem_u32(ring + (size_t)slot * slot_bytes),
              reinterpret_cast<const uint8_t*>(p.x) + base * row_bytes, bytes, bar, hint);
  };

  if (threadIdx.x == 0) {
    abort_flag = 0;
#pragma unroll
    for (int s = 0; s < kStages; ++s) mbar_init(smem_u32(&full[s]), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = threadIdx.x; i < 2 * kV * kMaxWarps; i += T) (&red[0][0][0])[i] = 0.0f;
  grid_dependency_wait();
  float s_enc = 0.0f;
  if (kQuantize) {
    s_enc = global_encode_scale(load_f32(p.amax_in));
    const float s_dec = __fdiv_rn(1.0f, s_enc);
    if (p.gscale_out && blockIdx.x == 0 && threadIdx.x == 0) *p.gscale_out = s_dec;
    // the encode scale depends on the block only through its scale byte: tabulate it
    for (int b = threadIdx.x; b < 128; b += T) enc_tab[b] = block_encode_scale((uint8_t)b, s_dec);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int s = 0; s < kStages; ++s) {
      const int64_t g = (int64_t)blockIdx.x + (int64_t)s * gridDim.x;
      if (g < groups) issue(g, s);
    }
  }

  // this thread's blocks and its slice of the per-column vectors, as pairs of fp32 lanes
  bool live[kJ];
  float2 cw[kAffine ? kJ : 1][8], cb[kAffine ? kJ : 1][8];
  float2 cs[kMod ? kJ : 1][8], ct[kMod ? kJ : 1][8];
  int64_t swz_kb[kJ];                      // K-block part of the swizzled scale offset
  bool has_w = false, has_b = false, has_s = false, has_t = false;
#pragma unroll
  for (int j = 0; j < kJ; ++j) {
    const int u = threadIdx.x + j * T;
    live[j] = kWhole || u < units;
    const int col = live[j] ? u * 16 : 0;
    swz_kb[j] = (int64_t)(u >> 2) * kSfAtomBytes + (u & 3);
    if (kAffine) {
      has_w = kWhole || p.w != nullptr; has_b = kWhole || p.b != nullptr;
      if (has_w) load16(p.w + col, cw[j]);
      if (has_b) load16(p.b + col, cb[j]);
    }
    if (kMod) {
      has_s = kWhole || p.scale != nullptr; has_t = kWhole || p.shift != nullptr;
      if (has_s) {
        load16(p.scale + col, cs[j]);
#pragma unroll
        for (int e = 0; e < 8; ++e) cs[j][e] = f2_add(make_float2(1.0f, 1.0f), cs[j][e]);
      }
      if (has_t) load16(p.shift + col, ct[j]);
    }
  }

  uint32_t amax_t = 0u;                 // bf16x2 running max of |h| (sweep 1)
  float amax_f = 0.0f;                  // the same where max_normed16 takes it
  // With one block a thread, no h wanted (with_variant): [27280, 3072] with all four vectors, both sweeps, 123.0 -> 116.9 us.
  // With two it gains or loses by the width ([32760, 5120] 157.3 -> 152.7, [27280, 3072] affine 82.2 -> 83.1).
  constexpr bool kMaxOnly = !kQuantize && kWhole && kJ == 1;
  const float cols_f = (float)p.cols, cols_inv = __fdiv_rn(1.0f, cols_f);

  // sweep 2 asks for a group's row statistics one group ahead: the load would otherwise sit
  // at the head of every group's dependency chain
  float mean_n[kR], rstd_n[kR];
  auto fetch_stats = [&](int64_t g) {
    const int64_t base = group_base(g);
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      const int64_t rr = base + r < p.rows ? base + r : base;
      const float2 st = load_f32x2(p.stats + 2 * rr);
      mean_n[r] = st.x;
      rstd_n[r] = st.y;
    }
  };
  if (kQuantize && (int64_t)blockIdx.x < groups) fetch_stats(blockIdx.x);

  // Rows that only pad the swizzled layout: whole words (4 K-blocks of a row) of zeros, written here
  // instead of by a memset launch ahead of the kernel.
  if (kQuantize && p.pad_rows > 0) {
    const int64_t words = (int64_t)p.pad_rows * p.k_atoms;
    for (int64_t i = (int64_t)blockIdx.x * T + threadIdx.x; i < words; i += (int64_t)gridDim.x * T) {
      const int64_t row = p.rows + i / p.k_atoms, atom = i % p.k_atoms;
      *reinterpret_cast<uint32_t*>(p.sf_swz + sf_swizzled_offset(row, atom * 4, p.k_atoms)) = 0u;
    }
  }

  int slot = 0;
  uint32_t phase = 0;
  int parity = 0;                        // which reduction buffer this group uses
  for (int64_t g = blockIdx.x; g < groups; g += gridDim.x, parity ^= 1) {
    const int64_t base = group_base(g);
    wait_group(smem_u32(&full[slot]), phase, &abort_flag, p.status);
    const uint8_t* slot_ptr = ring + (size_t)slot * slot_bytes;
    bool row_ok[kR];
    uint32_t xp[kR][kJ][8];             // the rows' blocks, still packed bf16 pairs
    float pivot[kR];                    // first element of the row
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      row_ok[r] = r == 0 || base + r < p.rows;
      const uint4* src = reinterpret_cast<const uint4*>(slot_ptr + (size_t)r * row_bytes);
      pivot[r] = (!kQuantize && !p.rms && row_ok[r])
                     ? bf16lo_to_f32(*reinterpret_cast<const uint32_t*>(src)) : 0.0f;
#pragma unroll
      for (int j = 0; j < kJ; ++j) {
        // (a thread without a block reads another's, a row past the end what the slot held: neither is used)
        const int u = live[j] ? threadIdx.x + j * T : 0;
        const uint4 a = src[2 * u], b = src[2 * u + 1];
        xp[r][j][0] = a.x; xp[r][j][1] = a.y; xp[r][j][2] = a.z; xp[r][j][3] = a.w;
        xp[r][j][4] = b.x; xp[r][j][5] = b.y; xp[r][j][6] = b.z; xp[r][j][7] = b.w;
      }
    }
    float mean[kR], rstd[kR];
    // once every thread holds its blocks the slot can take the group kStages ahead
    auto refill = [&]() {
      const int64_t gn = g + (int64_t)kStages * gridDim.x;
      if (threadIdx.x == 0 && gn < groups) issue(gn, slot);
    };
    if (!kQuantize) {
      // one pass: sums of d = x - pivot and of d^2 (the pivot, a sample of the row, keeps the
      // variance formula S2/n - (S1/n)^2 away from cancellation); RMSNorm needs S2 of x only
      float acc[kV];
#pragma unroll
      for (int r = 0; r < kR; ++r) {
        const float2 p2 = make_float2(pivot[r], pivot[r]);
        float2 s1 = make_float2(0.0f, 0.0f), s2 = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int j = 0; j < kJ; ++j) {
          if (live[j] && row_ok[r]) {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const float2 d = bf16x2_sub(xp[r][j][e], p2.x);
              s1 = f2_add(s1, d);
              s2 = f2_fma(d, d, s2);
            }
          }
        }
        acc[2 * r] = s1.x + s1.y;
        acc[2 * r + 1] = s2.x + s2.y;
      }
      cta_sum<kV>(acc, red[parity], warps);
      refill();
#pragma unroll
      for (int r = 0; r < kR; ++r) {
        const float m1 = div_by<kWhole>(acc[2 * r], cols_f, cols_inv), m2 = div_by<kWhole>(acc[2 * r + 1], cols_f, cols_inv);
        const float var = fmaxf(m2 - m1 * m1, 0.0f);
        mean[r] = p.rms ? 0.0f : pivot[r] + m1;
        rstd[r] = rsqrtf((p.rms ? m2 : var) + p.eps);
        if (threadIdx.x == 0 && row_ok[r])
          reinterpret_cast<float2*>(p.stats)[base + r] = make_float2(mean[r], rstd[r]);
      }
    } else {
      auto take_stats = [&]() {
#pragma unroll
        for (int r = 0; r < kR; ++r) {
          mean[r] = mean_n[r];
          rstd[r] = rstd_n[r];
        }
        if (g + gridDim.x < groups) fetch_stats(g + gridDim.x);
      };
      // The blocks were asked for above, but nothing has used them yet: where other kernels keep the SM's load units
      // busy, some are still to be read when the refill, which does not queue behind them, lands.  (In sweep 1 the
      // sums have used them.)  The fence holds every thread's reads ahead of the copy that thread 0 starts: without it
      // one call in twenty was wrong beside a quantizer on another stream.  Where there is nothing to refill, no thread
      // waits for the others.  With no vectors, or with all, the row statistics go ahead of it, so that their load is on
      // its way meanwhile.  Sweep pairs, us, without the fence, with it, as it is: [27280, 3072] no vectors 82.9, 83.8,
      // 82.5, modulation 96.2, 96.6, 96.5, all four 145.1, 150.7, 147.6; [32760, 5120] modulation 186.0, 186.8, 186.6.
      constexpr bool kStatsFirst = kAffine == kMod;
      if (kStatsFirst) take_stats();
      if (g + (int64_t)kStages * gridDim.x < groups) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        refill();
      }
      if (!kStatsFirst) take_stats();
    }

#pragma unroll
    for (int r = 0; r < kR; ++r) {
      const int64_t row = base + r;
      const float2 m2 = make_float2(mean[r], mean[r]);
      const float2 r2 = make_float2(rstd[r], rstd[r]);
      // row part of the swizzled scale offset (the K-block part is per thread)
      const int64_t swz_row = (row >> 7) * (int64_t)p.k_atoms * kSfAtomBytes + (row & 31) * 16 +
                              ((row >> 5) & 3) * 4;
#pragma unroll
      for (int j = 0; j < kJ; ++j) {
        const int u = threadIdx.x + j * T;
        const bool on = live[j] && row_ok[r];
        if constexpr (kMaxOnly) {
          if (on)
            amax_f = max_normed16<kAffine, kMod>(amax_f, xp[r][j], mean[r], r2, cw[kAffine ? j : 0], cb[kAffine ? j : 0],
                                                 cs[kMod ? j : 0], ct[kMod ? j : 0]);
          continue;
        }
        uint32_t hp[8];
        const uint32_t a2 = normalize16<kAffine, kMod, !kQuantize || (kAffine && kMod)>(
            kQuantize ? 0u : amax_t, xp[r][j], m2, r2, cw[kAffine ? j : 0], cb[kAffine ? j : 0], cs[kMod ? j : 0],
            ct[kMod ? j : 0], has_w, has_b, has_s, has_t, hp);
        if (!kQuantize) {
          if (on) {
            amax_t = a2;
            if (p.h_out) {
              uint4* dst = p.h_out + (row * units + u) * 2;
              dst[0] = make_uint4(hp[0], hp[1], hp[2], hp[3]);
              dst[1] = make_uint4(hp[4], hp[5], hp[6], hp[7]);
            }
          }
        } else if (on) {
          const float amax_b = fmaxf(fabsf(bf16lo_to_f32(a2)), fabsf(bf16hi_to_f32(a2)));
          float d = __fmul_rn(div_by_6(amax_b), s_enc);
          d = fminf(d, FLT_MAX);
          const uint8_t sf = (uint8_t)__nv_cvt_float_to_fp8(d, __NV_SATFINITE, __NV_E4M3);
          const float enc = enc_tab[sf & 127];
          const float2 enc2 = make_float2(enc, enc);
          float2 q[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) q[e] = f2_mul(bf16x2_to_f2(hp[e]), enc2);
          uint2 out;
          out.x = f32x8_to_e2m1x8(q[0].x, q[0].y, q[1].x, q[1].y, q[2].x, q[2].y, q[3].x, q[3].y);
          out.y = f32x8_to_e2m1x8(q[4].x, q[4].y, q[5].x, q[5].y, q[6].x, q[6].y, q[7].x, q[7].y);
          __stcs(reinterpret_cast<uint2*>(p.packed) + row * units + u, out);
          if (p.sf_lin) p.sf_lin[row * units + u] = sf;
          if (p.sf_swz) p.sf_swz[swz_row + swz_kb[j]] = sf;
        }
      }
    }
    if (++slot == kStages) {
      slot = 0;
      phase ^= 1u;
    }
  }

  if (!kQuantize) {
    const float amax = kMaxOnly ? __bfloat162float(__float2bfloat16(amax_f))
                              : fmaxf(fabsf(bf16lo_to_f32(amax_t)), fabsf(bf16hi_to_f32(amax_t)));
    const unsigned bits = __reduce_max_sync(0xffffffffu, __float_as_uint(amax));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red_max[threadIdx.x >> 5] = __uint_as_float(bits);
    __syncthreads();
    if (threadIdx.x == 0) {
      float m = 0.0f;
      for (int w = 0; w < warps; ++w) m = fmaxf(m, red_max[w]);
      if (m > 0.0f) atomicMax(p.amax_out, __float_as_uint(m));
    }
  }
  // Every copy this CTA issued has been waited for (each group issued is a group consumed),
  // unless a wait expired: then give copies still in flight time to land before the shared
  // memory is handed to another CTA.
  if (abort_flag) {
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL) {
    }
  }
}

// Both sweeps in one launch, for tensors that the GPU's shared memory holds: every CTA has its rows
// there from the first bulk copy on, puts h in their place, and packs h once the grid has met and the maximum
// is known.  x is read once, h computed once, and a memset and a launch go.  The arithmetic is that of the
// two sweeps, in their order.
constexpr int kMaxGroups = 16;            // row groups of a CTA

template <int kJ, bool kAffine, bool kMod, bool kWhole>
__global__ void __launch_bounds__(kMaxThreads)
norm_mod_resident_kernel(const NormArgs p, int per_cta, unsigned* partial) {
  constexpr int kR = RowsPerIter<kJ>::value;
  constexpr int kV = 2 * kR;
  extern __shared__ __align__(128) uint8_t rows_smem[];     // per_cta groups of kR rows
  __shared__ __align__(16) float red[2][kV][kMaxWarps];
  __shared__ unsigned red_max[kMaxWarps];
  __shared__ float enc_tab[128];
  __shared__ __align__(8) uint64_t full[kMaxGroups];
  __shared__ int abort_flag;
  const int T = blockDim.x;
  const int warps = T >> 5;
  const int units = p.cols >> 4;
  const uint32_t row_bytes = (uint32_t)p.cols * 2u;
  const int64_t row_first = (int64_t)blockIdx.x * per_cta * kR;
  const int my_rows = (int)(p.rows - row_first < (int64_t)per_cta * kR ? p.rows - row_first : (int64_t)per_cta * kR);
  const int my_groups = (my_rows + kR - 1) / kR;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < my_groups; ++s) mbar_init(smem_u32(&full[s]), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int s = 0; s < my_groups; ++s) {
      const int n = my_rows - s * kR < kR ? my_rows - s * kR : kR;
      const uint32_t bytes = (uint32_t)n * row_bytes, bar = smem_u32(&full[s]);
      mbar_expect_tx(bar, bytes);
      bulk_load(smem_u32(rows_smem) + (uint32_t)(s * kR) * row_bytes,
                reinterpret_cast<const uint8_t*>(p.x) + (row_first + s * kR) * row_bytes, bytes, bar, 1);
    }
  }
  for (int i = threadIdx.x; i < 2 * kV * kMaxWarps; i += T) (&red[0][0][0])[i] = 0.0f;

  bool live[kJ];
  float2 cw[kAffine ? kJ : 1][8], cb[kAffine ? kJ : 1][8];
  float2 cs[kMod ? kJ : 1][8], ct[kMod ? kJ : 1][8];
  int64_t swz_kb[kJ];
  const bool has_w = kAffine && (kWhole || p.w), has_b = kAffine && (kWhole || p.b), has_s = kMod && (kWhole || p.scale),
             has_t = kMod && (kWhole || p.shift);
#pragma unroll
  for (int j = 0; j < kJ; ++j) {
    const int u = threadIdx.x + j * T;
    live[j] = kWhole || u < units;
    const int col = live[j] ? u * 16 : 0;
    swz_kb[j] = (int64_t)(u >> 2) * kSfAtomBytes + (u & 3);
    if (has_w) load16(p.w + col, cw[j]);
    if (has_b) load16(p.b + col, cb[j]);
    if (has_s) {
      load16(p.scale + col, cs[j]);
#pragma unroll
      for (int e = 0; e < 8; ++e) cs[j][e] = f2_add(make_float2(1.0f, 1.0f), cs[j][e]);
    }
    if (has_t) load16(p.shift + col, ct[j]);
  }
  // what only pads the swizzled layout: whole rows as words, and the K-blocks past the end of every row
  if (p.sf_swz) {
    const int64_t words = (int64_t)p.pad_rows * p.k_atoms;
    for (int64_t i = (int64_t)blockIdx.x * T + threadIdx.x; i < words; i += (int64_t)gridDim.x * T) {
      const int64_t row = p.rows + i / p.k_atoms, atom = i % p.k_atoms;
      *reinterpret_cast<uint32_t*>(p.sf_swz + sf_swizzled_offset(row, atom * 4, p.k_atoms)) = 0u;
    }
    const int pad_kb = (int)p.k_atoms * 4 - units;
    for (int i = threadIdx.x; i < my_rows * pad_kb; i += T)
      p.sf_swz[sf_swizzled_offset(row_first + i / pad_kb, units + i % pad_kb, p.k_atoms)] = 0;
  }
  __syncthreads();

  uint32_t amax_t = 0u;
  const float cols_f = (float)p.cols, cols_inv = __fdiv_rn(1.0f, cols_f);
  for (int g = 0; g < my_groups; ++g) {
    wait_group(smem_u32(&full[g]), 0u, &abort_flag, p.status);
    uint8_t* group_ptr = rows_smem + (size_t)(g * kR) * row_bytes;
    bool row_ok[kR];
    uint32_t xp[kR][kJ][8];
    float pivot[kR];
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      row_ok[r] = r == 0 || g * kR + r < my_rows;
      const uint4* src = reinterpret_cast<const uint4*>(group_ptr + (size_t)r * row_bytes);
      pivot[r] = (!p.rms && row_ok[r]) ? bf16lo_to_f32(*reinterpret_cast<const uint32_t*>(src)) : 0.0f;
#pragma unroll
      for (int j = 0; j < kJ; ++j) {
        // (a thread without a block reads another's, a row past the end what the slot held: neither is used)
        const int u = live[j] ? threadIdx.x + j * T : 0;
        const uint4 a = src[2 * u], b = src[2 * u + 1];
        xp[r][j][0] = a.x; xp[r][j][1] = a.y; xp[r][j][2] = a.z; xp[r][j][3] = a.w;
        xp[r][j][4] = b.x; xp[r][j][5] = b.y; xp[r][j][6] = b.z; xp[r][j][7] = b.w;
      }
    }
    float acc[kV];
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      const float2 p2 = make_float2(pivot[r], pivot[r]);
      float2 s1 = make_float2(0.0f, 0.0f), s2 = make_float2(0.0f, 0.0f);
#pragma unroll
      for (int j = 0; j < kJ; ++j) {
        if (live[j] && row_ok[r]) {
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const float2 d = bf16x2_sub(xp[r][j][e], p2.x);
            s1 = f2_add(s1, d);
            s2 = f2_fma(d, d, s2);
          }
        }
      }
      acc[2 * r] = s1.x + s1.y;
      acc[2 * r + 1] = s2.x + s2.y;
    }
    cta_sum<kV>(acc, red[g & 1], warps);
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      const float m1 = div_by<kWhole>(acc[2 * r], cols_f, cols_inv), sq = div_by<kWhole>(acc[2 * r + 1], cols_f, cols_inv);
      const float var = fmaxf(sq - m1 * m1, 0.0f);
      const float mean = p.rms ? 0.0f : pivot[r] + m1;
      const float rstd = rsqrtf((p.rms ? sq : var) + p.eps);
      const float2 m2 = make_float2(mean, mean), r2 = make_float2(rstd, rstd);
      uint4* dst = reinterpret_cast<uint4*>(group_ptr + (size_t)r * row_bytes);
#pragma unroll
      for (int j = 0; j < kJ; ++j) {
        const int u = threadIdx.x + j * T;
        uint32_t hp[8];
        const uint32_t a2 = normalize16<kAffine, kMod, true>(
            amax_t, xp[r][j], m2, r2, cw[kAffine ? j : 0], cb[kAffine ? j : 0], cs[kMod ? j : 0], ct[kMod ? j : 0], has_w,
            has_b, has_s, has_t, hp);
        if (live[j] && row_ok[r]) {
          amax_t = a2;
          dst[2 * u] = make_uint4(hp[0], hp[1], hp[2], hp[3]);
          dst[2 * u + 1] = make_uint4(hp[4], hp[5], hp[6], hp[7]);
        }
      }
    }
  }

  // the maximum of the CTA, then of the grid
  unsigned bits = __reduce_max_sync(0xffffffffu,
                                    __float_as_uint(fmaxf(fabsf(bf16lo_to_f32(amax_t)), fabsf(bf16hi_to_f32(amax_t)))));
  if ((threadIdx.x & 31) == 0) red_max[threadIdx.x >> 5] = bits;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < warps; ++w) bits = max(bits, red_max[w]);
    partial[blockIdx.x] = bits;
  }
  cooperative_groups::this_grid().sync();
  bits = 0u;
  for (unsigned i = threadIdx.x; i < gridDim.x; i += T) bits = max(bits, load_u32(partial + i));
  bits = __reduce_max_sync(0xffffffffu, bits);
  if ((threadIdx.x & 31) == 0) red_max[threadIdx.x >> 5] = bits;
  __syncthreads();
  for (int w = 0; w < warps; ++w) bits = max(bits, red_max[w]);
  const float s_enc = global_encode_scale(__uint_as_float(bits));
  const float s_dec = __fdiv_rn(1.0f, s_enc);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *p.amax_out = bits;
    if (p.gscale_out) *p.gscale_out = s_dec;
  }
  fill_encode_table(enc_tab, s_dec);
  __syncthreads();

#pragma unroll 2
  for (int r = 0; r < my_rows; ++r) {
    const int64_t row = row_first + r;
    const uint4* src = reinterpret_cast<const uint4*>(rows_smem + (size_t)r * row_bytes);
    const int64_t swz_row = (row >> 7) * (int64_t)p.k_atoms * kSfAtomBytes + (row & 31) * 16 + ((row >> 5) & 3) * 4;
#pragma unroll
    for (int j = 0; j < kJ; ++j) {
      if (!live[j]) continue;
      const int u = threadIdx.x + j * T;
      const uint4 a = src[2 * u], b = src[2 * u + 1];     // this thread's own writes
      const uint32_t h[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
      uint32_t a2 = 0u, sf;
#pragma unroll
      for (int e = 0; e < 8; ++e) a2 = bf16x2_max_abs(a2, h[e]);
      const uint2 out = pack_block(h, a2, s_enc, enc_tab, sf);
      __stcs(reinterpret_cast<uint2*>(p.packed) + row * units + u, out);
      if (p.sf_lin) p.sf_lin[row * units + u] = (uint8_t)sf;
      if (p.sf_swz) p.sf_swz[swz_row + swz_kb[j]] = (uint8_t)sf;
    }
  }
  if (abort_flag) {
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL) {
    }
  }
}

int check_args(const void* x, int64_t rows, int64_t cols) {
  if (rows < 0 || cols <= 0 || cols % kBlock != 0 || cols > kMaxJ * 16 * kMaxThreads ||
      rows >= ((int64_t)1 << 31))
    return NVFP4_ERR_BAD_ARG;
  if (rows > 0 && !x) return NVFP4_ERR_BAD_ARG;
  if (!aligned16(x)) return NVFP4_ERR_BAD_ALIGN;
  return NVFP4_OK;     // the device is checked last: bad arguments are refused on any machine
}

bool vec_ok(const float* p) { return aligned16(p); }

// Blocks per thread (1 or 2) and threads per CTA (a multiple of 32) for a row of `units`
// 16-element blocks and this many kinds of per-column vectors (affine, modulation).
void shape_for(int units, int kinds, int* j, int* threads) {
  int J = 1;
  while (J < kMaxJ && units > J * kMaxThreads) J *= 2;
  // two blocks per thread whenever the row is long enough for two warps: the per-row
  // bookkeeping is then shared by 32 elements instead of 16 (measured 17-20 % faster).  Not with all four
  // vectors, which take 128 registers and leave none for the row (4 KB of spills in every group).
#ifndef NVFP4_NORM_FORCE_J1
  if (units % 2 == 0 && units / 2 >= 64 && kinds < 2) J = 2;
#endif
  const int per = (units + J - 1) / J;
  *j = J;
  *threads = ((per + 31) / 32) * 32;
}

template <bool kQuantize, int kJ, bool kAffine, bool kMod, bool kWhole>
int launch_variant(const NormArgs& a, int threads, cudaStream_t st) {
  auto kernel = norm_mod_kernel<kQuantize, kJ, kAffine, kMod, kWhole>;
  constexpr int kR = RowsPerIter<kJ>::value;
  const size_t smem = (size_t)kStages * kR * a.cols * 2;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return NVFP4_ERR_BAD_ARG;
  // One limit for all widths: one that followed the width could be lowered by another thread between this thread's
  // question and its launch, which is then refused.
  static std::atomic<bool> allowed[64];
  if (!allowed[dev].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kStages * kR * kJ * 16 * kMaxThreads * 2) !=
        cudaSuccess)
      return NVFP4_ERR_LAUNCH_FAILED;
    allowed[dev].store(true, std::memory_order_release);
  }
  // CTAs that an SM holds, for the last geometry of this variant in this thread: a model calls it with one row width over
  // and over
  struct Geometry { int dev, cols, threads, per_sm; };
  static thread_local Geometry last{};
  if (last.per_sm < 1 || last.dev != dev || last.cols != a.cols || last.threads != threads) {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem) != cudaSuccess || n < 1)
      return NVFP4_ERR_LAUNCH_FAILED;
    last = {dev, a.cols, threads, n};
  }
  const int per_sm = last.per_sm;
  const int64_t groups = (a.rows + kR - 1) / kR;
  const int64_t resident = (int64_t)sm_count() * per_sm;
  const unsigned grid = (unsigned)(groups < resident ? groups : resident);
  return launch_dependent(kernel, dim3(grid), (unsigned)threads, smem, 1, st, a);
}

// Row groups per CTA of the one-launch form: the least with which all CTAs are on the GPU at a time, or 0.  How many
// an SM holds is the runtime's answer for the dynamic size at hand: a sum of shared-memory constants that was 256
// bytes short gave [3800, 4096] a launch that is refused, which an eager call survives by way of the two sweeps and a
// stream capture does not.  The last answer is kept per thread, so that only a change of shape asks.
template <typename Kernel>
int groups_per_cta(Kernel kernel, int dev, int threads, int64_t groups, int64_t group_bytes) {
  constexpr int kSmemMax = 200 << 10, kSmemSm = 228 << 10;
  struct Last {
    Kernel kernel;             // all variants have the one type
    int dev, threads, per;
    int64_t groups, group_bytes;
  };
  static thread_local Last last{};
  if (last.kernel == kernel && last.dev == dev && last.threads == threads && last.groups == groups && last.group_bytes == group_bytes)
    return last.per;
  int found = 0;
  for (int per = 1; per <= kMaxGroups && per * group_bytes <= kSmemMax && !found; ++per) {
    const int64_t ctas = (groups + per - 1) / per, bytes = per * group_bytes;
    // more than the rows alone leave room for: not worth the question
    if (ctas > NVFP4_AMAX_PARTIALS || ctas > sm_count() * (kSmemSm / bytes)) continue;
    int an_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&an_sm, kernel, threads, (size_t)bytes) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    if (ctas <= (int64_t)sm_count() * an_sm) found = per;
  }
  last = {kernel, dev, threads, found, groups, group_bytes};
  return found;
}

// Launches the one-launch form if the rows fit; *done says whether.
template <int kJ, bool kAffine, bool kMod, bool kWhole>
int launch_resident(const NormArgs& a, int threads, unsigned* partial, cudaStream_t st, bool* done) {
  auto kernel = norm_mod_resident_kernel<kJ, kAffine, kMod, kWhole>;
  constexpr int kR = RowsPerIter<kJ>::value;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return NVFP4_ERR_BAD_ARG;
  static std::atomic<bool> allowed[64];
  if (!allowed[dev].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 << 10) != cudaSuccess)
      return NVFP4_ERR_LAUNCH_FAILED;
    allowed[dev].store(true, std::memory_order_release);
  }
  const int64_t groups = (a.rows + kR - 1) / kR, group_bytes = (int64_t)kR * a.cols * 2;
  const int per = groups_per_cta(kernel, dev, threads, groups, group_bytes);
  if (per == 0) return NVFP4_OK;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((groups + per - 1) / per));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = (size_t)(per * group_bytes);
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeCooperative;
  attr.val.cooperative = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, a, per, partial);
  if (e == cudaSuccess) {
    *done = true;
    return NVFP4_OK;
  }
  cudaGetLastError();
  // fewer SMs than the device has: the two sweeps run on any number
  return e == cudaErrorCooperativeLaunchTooLarge ? NVFP4_OK : NVFP4_ERR_LAUNCH_FAILED;
}

// Calls f with the variant of the kernels for these arguments: blocks per thread, affine, modulation, kWhole.
template <typename F>
int with_variant(const NormArgs& a, int* threads, F&& f) {
  int J;
  const bool affine = a.w || a.b, mod = a.scale || a.shift;
  shape_for(a.cols / 16, affine + mod, &J, threads);
  const bool whole = (!affine || (a.w && a.b)) && (!mod || (a.scale && a.shift)) && *threads * J * 16 == a.cols && (J == 2 || !a.h_out);
  auto go = [&](auto j, auto with_affine, auto with_mod) {
    return whole ? f(j, with_affine, with_mod, std::true_type()) : f(j, with_affine, with_mod, std::false_type());
  };
  auto kinds = [&](auto j) {
    if (affine) return mod ? go(j, std::true_type(), std::true_type()) : go(j, std::true_type(), std::false_type());
    return mod ? go(j, std::false_type(), std::true_type()) : go(j, std::false_type(), std::false_type());
  };
  return J == 1 ? kinds(std::integral_constant<int, 1>()) : kinds(std::integral_constant<int, 2>());
}

int try_resident(const NormArgs& a, unsigned* partial, cudaStream_t st, bool* done) {
  int threads;
  return with_variant(a, &threads, [&](auto j, auto affine, auto mod, auto whole) {
    return launch_resident<j(), affine(), mod(), whole()>(a, threads, partial, st, done);
  });
}

template <bool kQuantize>
int launch(const NormArgs& a, cudaStream_t st) {
  int threads;
  return with_variant(a, &threads, [&](auto j, auto affine, auto mod, auto whole) {
    return launch_variant<kQuantize, j(), affine(), mod(), whole()>(a, threads, st);
  });
}

}  // namespace
}  // namespace nvfp4

using namespace nvfp4;

extern "C" {

int nvfp4_norm_mod_amax_bf16(const void* x_bf16, int64_t rows, int64_t cols, const float* weight,
                             const float* bias, const float* scale, const float* shift, int rms,
                             float eps, float* row_stats, float* amax_dev, void* h_out_bf16,
                             int* status_dev, void* stream) {
  int rc = check_args(x_bf16, rows, cols);
  if (rc != NVFP4_OK) return rc;
  if (!row_stats || !amax_dev) return NVFP4_ERR_BAD_ARG;
  if (!aligned16(h_out_bf16) || !vec_ok(weight) || !vec_ok(bias) || !vec_ok(scale) || !vec_ok(shift))
    return NVFP4_ERR_BAD_ALIGN;
  rc = check_device_sm100();
  if (rc != NVFP4_OK) return rc;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(amax_dev, 0, sizeof(float), st) != cudaSuccess) return NVFP4_ERR_LAUNCH_FAILED;
  if (rows == 0) return NVFP4_OK;
  NormArgs a{};
  a.x = reinterpret_cast<const uint4*>(x_bf16);
  a.rows = rows; a.cols = (int)cols;
  a.w = weight; a.b = bias; a.scale = scale; a.shift = shift;
  a.rms = rms; a.eps = eps;
  a.stats = row_stats;
  a.amax_out = reinterpret_cast<unsigned*>(amax_dev);
  a.h_out = reinterpret_cast<uint4*>(h_out_bf16);
  a.status = status_dev;
  return launch<false>(a, st);
}

int nvfp4_norm_mod_quantize_bf16(const void* x_bf16, int64_t rows, int64_t cols,
                                 const float* weight, const float* bias, const float* scale,
                                 const float* shift, const float* row_stats,
                                 const float* amax_dev, uint8_t* packed, uint8_t* scales_linear,
                                 uint8_t* scales_swizzled, float* global_scale_dev,
                                 int* status_dev, void* stream) {
  int rc = check_args(x_bf16, rows, cols);
  if (rc != NVFP4_OK) return rc;
  if (!row_stats || !amax_dev || (rows > 0 && !packed)) return NVFP4_ERR_BAD_ARG;
  // the kernel stores 8-byte words of nibbles
  if ((reinterpret_cast<uintptr_t>(packed) & 7u) || !vec_ok(weight) || !vec_ok(bias) ||
      !vec_ok(scale) || !vec_ok(shift))
    return NVFP4_ERR_BAD_ALIGN;
  rc = check_device_sm100();
  if (rc != NVFP4_OK) return rc;
  if (rows == 0) return NVFP4_OK;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  int pad_rows = 0;
  if (scales_swizzled) {
    // pad rows / K-blocks of the swizzled buffer must decode to zero; the kernel writes the former
    const int64_t total = sf_swizzled_bytes(rows, cols);
    const bool k_pad = (cols / kBlock) % kSfKbPad != 0;
    if (!k_pad && (reinterpret_cast<uintptr_t>(scales_swizzled) & 3u) == 0) {
      pad_rows = (int)(sf_row_tiles(rows) * 128 - rows);
    } else {
      const int64_t first = k_pad ? 0 : (rows / 128) * sf_k_atoms(cols) * kSfAtomBytes;
      if (first < total &&
          cudaMemsetAsync(scales_swizzled + first, 0, (size_t)(total - first), st) != cudaSuccess)
        return NVFP4_ERR_LAUNCH_FAILED;
    }
  }
  NormArgs a{};
  a.x = reinterpret_cast<const uint4*>(x_bf16);
  a.rows = rows; a.cols = (int)cols;
  a.w = weight; a.b = bias; a.scale = scale; a.shift = shift;
  a.stats = const_cast<float*>(row_stats);
  a.amax_in = amax_dev;
  a.packed = reinterpret_cast<uint32_t*>(packed);
  a.sf_lin = scales_linear; a.sf_swz = scales_swizzled;
  a.k_atoms = (uint32_t)sf_k_atoms(cols);
  a.pad_rows = pad_rows;
  a.gscale_out = global_scale_dev;
  a.status = status_dev;
  return launch<true>(a, st);
}

int nvfp4_norm_mod_bf16(const void* x_bf16, int64_t rows, int64_t cols, const float* weight, const float* bias,
                        const float* scale, const float* shift, int rms, float eps, float* row_stats,
                        float* amax_dev, uint8_t* packed, uint8_t* scales_linear, uint8_t* scales_swizzled,
                        float* global_scale_dev, float* partials, int* status_dev, void* stream) {
  int rc = check_args(x_bf16, rows, cols);
  if (rc != NVFP4_OK) return rc;
  if (!row_stats || !amax_dev || (rows > 0 && !packed)) return NVFP4_ERR_BAD_ARG;     // whichever form it takes
  if ((reinterpret_cast<uintptr_t>(packed) & 7u) || !vec_ok(weight) || !vec_ok(bias) || !vec_ok(scale) ||
      !vec_ok(shift))
    return NVFP4_ERR_BAD_ALIGN;
  rc = check_device_sm100();
  if (rc != NVFP4_OK) return rc;
  if (rows > 0 && partials && (reinterpret_cast<uintptr_t>(scales_swizzled) & 3u) == 0) {
    NormArgs a{};
    a.x = reinterpret_cast<const uint4*>(x_bf16);
    a.rows = rows; a.cols = (int)cols;
    a.w = weight; a.b = bias; a.scale = scale; a.shift = shift;
    a.rms = rms; a.eps = eps;
    a.amax_out = reinterpret_cast<unsigned*>(amax_dev);
    a.packed = reinterpret_cast<uint32_t*>(packed);
    a.sf_lin = scales_linear; a.sf_swz = scales_swizzled;
    a.k_atoms = (uint32_t)sf_k_atoms(cols);
    a.pad_rows = (int)(sf_row_tiles(rows) * 128 - rows);
    a.gscale_out = global_scale_dev;
    a.status = status_dev;
    bool done = false;
    rc = try_resident(a, reinterpret_cast<unsigned*>(partials), reinterpret_cast<cudaStream_t>(stream), &done);
    if (rc != NVFP4_OK || done) return rc;
  }
  rc = nvfp4_norm_mod_amax_bf16(x_bf16, rows, cols, weight, bias, scale, shift, rms, eps, row_stats, amax_dev, nullptr,
                                status_dev, stream);
  if (rc != NVFP4_OK) return rc;
  return nvfp4_norm_mod_quantize_bf16(x_bf16, rows, cols, weight, bias, scale, shift, row_stats, amax_dev, packed,
                                      scales_linear, scales_swizzled, global_scale_dev, status_dev, stream);
}

}  // extern "C"
