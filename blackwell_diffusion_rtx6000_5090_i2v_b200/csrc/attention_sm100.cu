// Non-causal bf16 attention for sm_100a, head dimension 128, with the maximum |o| of the
// output folded into the kernel (the NVFP4 quantizer in front of the attention-out linear
// then needs no amax pass of its own).  Replaces the library attention at the reference's call
// sites fx/src/s4/models/wan22/wan_transformer_fast.py:47-58 (flash_attn_qkvpacked_func) and
// fx/src/s4/models/wan22/wan_transformer.py:126-129,164-167 (scaled_dot_product_attention).
//
// A pair of CTAs (one per SM) owns 256 query rows of one head, 128 each, and walks the keys 128 at a time:
//     S = Q K^T           tcgen05.mma.cta_group::2, M 256: each CTA's own Q rows, and half of the K tile from
//                         the shared memory of either CTA
//     P = exp2(S*c - m)   two threads per query row (64 keys each): tcgen05.ld, exp2, row sum, bf16 P to tensor
//                         memory of its own
//     O += P V            the same instruction with P read from tensor memory and V (keys x d, d contiguous:
//                         an MN-major operand), of which each CTA holds half of the head dimension
// Two groups of eight softmax warps take the tiles by turns.  With S and P double-buffered and apart (P used
// to lie over S, which tied S of tile j + 1 to the product of tile j) the chain S -> softmax -> P V of a tile
// runs beside that of the next: Q K^T of tile j + 2 is issued as soon as S of tile j is in registers.  A pair
// goes on from block to block (the next Q and the next tiles' S are on their way during the epilogue).
//
// Bound: the softmax of a tile, ~1100 cycles of its scheduler's issue and special-function slots against 1024 of
// tensor work, and on long sequences the board's power limit.  What was measured on the way (cycles per key
// tile of a CTA, [9472, 4, 128]): one CTA with two query tiles and P over S 1730; pairs as here 2900 with
// arrivals across the pair of release.cluster scope (a fence of about 1000 cycles each), 2000 with waits whose
// lanes polled two barriers (up to a thousand cycles of delay), 1750 with the two groups' exponentials at the
// same time; 1450 with a thread per row (half the warps, the same latencies per tile), 1330 as it is.
// Against the one CTA, us: [32760, 5, 128] back to back 2537 -> 2329; replayed from a graph [3121, 12] 94 -> 64,
// [27280 x 512 keys, 24] 257 -> 214 to 226, [512 x 512, 24] 14.4 -> 10.8; [1, 1] 5.8 -> 7.4, where the pair's hand-offs are
// latency alone.  The library kernel, in the same order, 2110, 74, 149, 10.1.
//
// Blocks that would leave pairs idle in a last wave are computed by several pairs each, which share the
// block's keys and join their results through distributed shared memory (kParts > 1, and launch()).
//
// The reference m of a row is its running maximum, raised only when a tile exceeds it by more than
// 2^8; the four threads of a row follow it by the same maxima.  (A reference that
// follows the row sums of earlier tiles needs neither the maximum nor the exchange.  But a key far above all
// before it then weighs 2^x rounded to bf16 where it should weigh exactly 1, or overflows: an error of 2.3e-3
// with q, k and v from a Student-t(4) distribution.)
// The row sum adds the probabilities as they are rounded for the product, so that numerator and
// denominator agree; adding a bf16 to an fp32 is one instruction.  Against the sum of the unrounded
// ones, relative error against 64 bits with Student-t(4) inputs 1.82e-3 -> 1.67e-3, with N(0, 1) 2.35e-3
// either way.  The partial sums are joined at the end, not at every tile.
//
// Tensor memory (512 columns): S at 0 and 128, P at 256 and 320, O at 384.
// Shared memory: two Q tiles (32 KiB each), rings of four half K and three half V tiles (16 KiB each), in the
// 128-byte swizzle that TMA writes, and a 2 KiB output slab per softmax warp.
//
// Warps 0-7: softmax + epilogue of the even tiles (warp & 3 = the 32-lane quarter of tensor memory
// it may touch, bit 2 = which 64 keys), 8-15 of the odd ones; 16 and 19: TMA loads of Q and K, and of V; 17 and
// 18, in the leader CTA: issue of the two products.  One warp for both was late for each.
// Every wait on a barrier is bounded: when one runs out the kernel records where in *status, raises a
// CTA-wide flag so that every role ends, and releases its tensor memory.
#include <cuda.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cfloat>
#include <cstdint>

#include "nvfp4_common.cuh"

namespace nvfp4 {
namespace attn {

constexpr int kD = 128;                   // head dimension
constexpr int kBQ = 128;                  // query rows per CTA (= tensor-memory lanes); a pair has 256
constexpr int kBKV = 128;                 // keys per tile: each CTA of the pair fetches half of a tile
constexpr int kHalfBytes = 128 * 128;     // 128 rows x 64 bf16
constexpr int kQBytes = 2 * kHalfBytes;
constexpr int kSlotBytes = kHalfBytes;    // a CTA's half of a K tile (64 keys) or of a V tile (64 dimensions)
constexpr int kKSlots = 4, kVSlots = 3;
constexpr int kDataBytes = 2 * kQBytes + (kKSlots + kVSlots) * kSlotBytes;
constexpr int kSlabBytes = 32 * 64;       // 32 rows x 32 output columns of a softmax warp
constexpr int kBarBytes = 384;            // barriers, abort flag, tensor-memory address
constexpr int kMaxBytes = 4 * 2 * kBQ * 4;   // row maxima of the last four tiles: [tile & 3][half][row]
constexpr int kSumBytes = 2 * 4 * kBQ * 8;   // row sums and their references: [block & 1][group, half][row]
constexpr int kSoftmaxWarps = 16;         // two groups of eight
constexpr int kSlabs = kSoftmaxWarps * kSlabBytes;
constexpr int kSmemBytes = kDataBytes + kSlabs + 1024 /*align slack*/ + kBarBytes + kMaxBytes + kSumBytes;
constexpr int kLoadKWarp = 16, kIssueSWarp = 17, kIssueOWarp = 18, kLoadVWarp = 19;
constexpr int kThreads = 640;
constexpr int kTmemCols = 512;
constexpr int kColS = 0, kColP = 256, kColO = 384;   // + 128 resp. 64 columns for the second S, P
constexpr int kPartBytes = kBQ * kD * 4;  // a split CTA's partial O, where the operands were
constexpr int kMaxParts = 4;              // pairs that share a block: eight CTAs, the portable cluster size
constexpr float kRescaleStep = 8.f;       // raise the running maximum only past 2^8
#ifndef NVFP4_ATTN_FMA_EXP_EVERY
#define NVFP4_ATTN_FMA_EXP_EVERY 11
#endif
// Every kFmaExpEvery-th element pair takes 2^x on the FMA pipe (0: none), spread evenly so that
// the special-function unit works through its pairs while the FMA pipe works through these.  [32760, 5, 128],
// us: none 2470, every 16th 2210, 11th 2157, 8th 2190, 6th 2227.
constexpr int kFmaExpEvery = NVFP4_ATTN_FMA_EXP_EVERY;
constexpr long long kWaitCycles = 4000000000LL;  // ~2 s at 2 GHz
constexpr int kErrBase = 0xA00;

static_assert(kSmemBytes <= 232448, "exceeds the 227 KiB per-CTA shared memory limit");
static_assert(kPartBytes + kBQ * 8 <= kDataBytes, "the partial result overruns the operands");

struct Params {
  int64_t q_len, kv_len;
  int64_t first, end;            // blocks of 256 query rows that this launch computes ...
  int64_t q_blocks;              // ... numbered through the heads, this many a head
  int heads, kv_tiles;
  int lets_next_start;           // a launch whose blocks are shared follows and may fill in as SMs get free
  int follows;                   // this is that launch
  float scale_log2;              // softmax scale * log2(e)
  uint8_t* o;                    // bf16 [q_len][heads][128], strided
  int64_t o_row_bytes, o_head_bytes;
  unsigned* amax;                // max |o| as float bits (atomicMax), or null
  int* status;
};

// ----------------------------------------------------------- PTX wrappers --

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t e;
  asm volatile(
      "{\n\t.reg .pred P;\n\t.reg .b32 r;\n\t"
      "elect.sync r|P, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}"
      : "=r"(e));
  return e;
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes, uint32_t on) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t"
      "@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}"
      ::"r"(bar), "r"(bytes), "r"(on)
      : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: false (after raising the abort flag and recording `where`) when the barrier
// does not flip within kWaitCycles or another role has already given up.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                          int* status, int where) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  for (uint32_t it = 1;; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 255u) == 0) {
      if (*abort_flag) return false;
      if (clock64() - t0 > kWaitCycles) {
        *abort_flag = 1;
        if (status) atomicCAS(status, 0, where);
        return false;
      }
    }
  }
}
// Arrive on a barrier given by its shared::cluster address (this CTA's or the peer's).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ uint32_t mapa_u32(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// One box of a [tokens][heads][128] tensor (64 elements wide) into this CTA's shared memory; its bytes are
// reported to a barrier that may live in the other CTA of the pair.  One destination per copy.
__device__ __forceinline__ void tma_load_3d(const CUtensorMap* map, uint32_t bar, uint32_t dst, int x,
                                            int y, int z, uint32_t on) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %6, 0;\n\t"
      "@q cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];\n\t}"
      ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z), "r"(on)
      : "memory");
}
// A slab of 32 rows x 32 elements to global memory, clipped at the tensor's edges.
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, uint32_t src, int x, int y, int z, uint32_t on) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];\n\t}"
      ::"l"(map), "r"(src), "r"(x), "r"(y), "r"(z), "r"(on)
      : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// Arrive, once this thread's earlier tcgen05 operations (in both CTAs of the pair) have completed, on the
// barrier at this offset in the CTAs of the cluster that `cta_mask` names.
__device__ __forceinline__ void tc_commit(uint32_t bar, uint16_t cta_mask, uint32_t on) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t"
      "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64"
      " [%0], %1;\n\t}"
      ::"r"(bar), "h"(cta_mask), "r"(on)
      : "memory");
}
// D[tmem] (+)= A[smem] * B[smem]
__device__ __forceinline__ void tc_mma_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                          uint32_t idesc, uint32_t accumulate, uint32_t on) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(on)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void tc_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc,
                                          uint32_t idesc, uint32_t accumulate, uint32_t on) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(on)
      : "memory");
}
// 32 lanes x 32 consecutive 32-bit columns <-> 32 registers per thread.
__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};"
      ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]),
        "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tc_ld8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tc_st8(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
               ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tc_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// 2^x for a pair, x <= 8, on the FMA pipe instead of the special-function unit (which is the
// scarcer resource here: 16 results per clock per SM against 128 FMA lanes).  x = i + f with
// f in [-0.5, 0.5] by magic-number rounding, a cubic for 2^f (relative error 7.5e-5, a fiftieth
// of a bf16 rounding step), and i added into the exponent field.  x is clamped at -126, where
// the result (1e-38) is already nothing next to the row's largest term.  A NaN stays one through the clamp, and
// its result, the sum of two NaN patterns, is the largest float: infinity as a bf16, and NaN in the row's output.
__device__ __forceinline__ float2 exp2_fma(float2 x) {
  const float kMagic = 12582912.f;   // 1.5 * 2^23: the sum's low mantissa bits hold round(x)
  asm("max.NaN.f32 %0, %0, 0fC2FC0000;" : "+f"(x.x));     // -126
  asm("max.NaN.f32 %0, %0, 0fC2FC0000;" : "+f"(x.y));
  const float2 magic = make_float2(kMagic, kMagic);
  const float2 r = f2_add(x, magic);
  const float2 f = f2_sub(x, f2_sub(r, magic));
  float2 y = f2_fma(f, make_float2(0.0551716685f, 0.0551716685f), make_float2(0.242611125f, 0.242611125f));
  y = f2_fma(y, f, make_float2(0.693260968f, 0.693260968f));
  y = f2_fma(y, f, make_float2(0.999928057f, 0.999928057f));
  y.x = __int_as_float(__float_as_int(y.x) + (__float_as_int(r.x) << 23));
  y.y = __int_as_float(__float_as_int(y.y) + (__float_as_int(r.y) << 23));
  return y;
}

// acc + the two bf16 of a word, in fp32 (mixed-precision add, sm_100)
__device__ __forceinline__ float2 add_bf16x2(uint32_t w, float2 acc) {
  asm("{\n\t.reg .b16 lo, hi;\n\tmov.b32 {lo, hi}, %2;\n\t"
      "add.f32.bf16 %0, lo, %0;\n\tadd.f32.bf16 %1, hi, %1;\n\t}"
      : "+f"(acc.x), "+f"(acc.y) : "r"(w));
  return acc;
}

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
// Shared memory of CTA `rank` of the cluster, at this CTA's address.
__device__ __forceinline__ float2 ld_cluster_f2(uint32_t addr, uint32_t rank) {
  float2 v;
  asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %2, %3;\n\t"
               "ld.shared::cluster.v2.f32 {%0, %1}, [a];\n\t}"
               : "=f"(v.x), "=f"(v.y) : "r"(addr), "r"(rank) : "memory");
  return v;
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr, uint32_t rank) {
  float4 v;
  asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %4, %5;\n\t"
               "ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [a];\n\t}"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr), "r"(rank) : "memory");
  return v;
}
// Where 16-byte chunk `c` (0..31) of a row of a partial result lies: a thread writes whole rows, so
// the chunks of eight rows are spread over the banks.
__device__ __forceinline__ uint32_t part_offset(int row, int c) {
  return (uint32_t)row * (kD * 4) + (uint32_t)((c ^ (row & 7)) << 4);
}

// Shared-memory matrix descriptor, 128-byte swizzle (layout code 2, descriptor version 1), 8-row groups
// 1024 bytes apart (stride offset); the leading offset is unused: a row is 128 bytes.  For Q and K a row
// holds 64 contraction elements (K-major), for V the 64 output dimensions of one key (MN-major).
__device__ __forceinline__ uint64_t desc_sw128(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// Instruction descriptor, kind::f16: fp32 accumulate (bit 4), A and B bf16 (code 1 at bits 7
// and 10), B MN-major when `b_mn` (bit 16), N = 128 at bits 17-22 in units of 8, M = 256 (of the pair) at
// bits 24-28 in units of 16.
__device__ __forceinline__ uint32_t make_idesc(bool b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (b_mn ? (1u << 16) : 0u) | ((uint32_t)(128 >> 3) << 17) |
         ((uint32_t)(256 >> 4) << 24);
}

// ------------------------------------------------------------------ kernel --

// kParts > 1: the cluster's pairs share one block's keys and join their results at the end; else a pair
// walks over blocks.
template <int kParts>
__global__ void __cluster_dims__(2 * kParts, 1, 1) __launch_bounds__(kThreads, 1)
attention_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                 const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_o,
                 const Params p) {
  constexpr bool kSplit = kParts > 1;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t bar_base = smem_base + kDataBytes + kSlabs;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_gen + kDataBytes + kSlabs + kBarBytes - 8);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_gen + kDataBytes + kSlabs + kBarBytes - 4);
  auto q_smem = [&](int i) { return smem_base + (uint32_t)(i & 1) * kQBytes; };
  auto k_smem = [&](int j) { return smem_base + 2 * kQBytes + (uint32_t)(j % kKSlots) * kSlotBytes; };
  auto v_smem = [&](int j) { return smem_base + 2 * kQBytes + (uint32_t)(kKSlots + j % kVSlots) * kSlotBytes; };
  // Barriers sit at the same offsets in all CTAs.  "leader": waited on in the pair's even CTA and fed by
  // both; "each": waited on in each CTA.  Of a tile by its running number j, of a block by i.
  auto q_full = [&](int i) { return bar_base + 8u * (i & 1); };                       // leader
  auto q_empty = [&](int i) { return bar_base + 8u * (2 + (i & 1)); };                // each
  auto k_full = [&](int j) { return bar_base + 8u * (4 + j % kKSlots); };              // leader
  auto k_empty = [&](int j) { return bar_base + 8u * (4 + kKSlots + j % kKSlots); };    // each
  auto v_full = [&](int j) { return bar_base + 8u * (4 + 2 * kKSlots + j % kVSlots); };     // leader
  auto v_empty = [&](int j) { return bar_base + 8u * (4 + 2 * kKSlots + kVSlots + j % kVSlots); };    // each
  constexpr int kB = 4 + 2 * (kKSlots + kVSlots);
  auto s_full = [&](int j) { return bar_base + 8u * (kB + (j & 1)); };                // each: S computed
  auto s_empty = [&](int j) { return bar_base + 8u * (kB + 2 + (j & 1)); };           // leader: S in registers
  auto p_full = [&](int j) { return bar_base + 8u * (kB + 4 + (j & 1)); };            // leader: P written
  auto pv_done = [&](int j) { return bar_base + 8u * (kB + 6 + (j & 1)); };           // each: P V added
  auto o_empty = [&]() { return bar_base + 8u * (kB + 8); };                          // leader: O read
  static_assert(kB + 9 <= 31 && 8 * (kB + 9) <= kBarBytes - 8, "a lane for every barrier, and room in their area");
  volatile float* row_max = reinterpret_cast<volatile float*>(smem_gen + kDataBytes + kSlabs + kBarBytes);
  float2* row_sum = reinterpret_cast<float2*>(smem_gen + kDataBytes + kSlabs + kBarBytes + kMaxBytes);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const uint32_t leader = rank & ~1u;           // the pair's even CTA, by its rank in the cluster
  const uint16_t both = (uint16_t)(3u << leader);
  // this pair's blocks first, first + step, ... (`blocks` of them), and its key tiles [kv0, kv0 + n)
  const int part = kSplit ? (int)rank / 2 : 0;
  const int64_t step = kSplit ? 1 : gridDim.x / 2;
  const int64_t first = p.first + (kSplit ? blockIdx.x / (2 * kParts) : blockIdx.x / 2);
  const int blocks = kSplit ? 1 : (int)((p.end - first + step - 1) / step);
  const int kv0 = kSplit ? (int)((int64_t)p.kv_tiles * part / kParts) : 0;
  const int n = kSplit ? (int)((int64_t)p.kv_tiles * (part + 1) / kParts) - kv0 : p.kv_tiles;
  const int total = (int)(blocks * n);

  if (warp == 0) {
    // arrivals: a group's eight warps of both CTAs, all softmax warps of both, or one
    if (lane < kB + 9)
      mbar_init(bar_base + 8u * lane, lane >= kB + 2 && lane < kB + 6 ? kSoftmaxWarps
                                      : lane == kB + 8                ? 2 * kSoftmaxWarps
                                                                      : 1);
    if (lane == 31) *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == kLoadKWarp && lane < 4)
    asm volatile("prefetch.tensormap [%0];" ::"l"(lane == 0 ? &map_q : lane == 1 ? &map_k : lane == 2 ? &map_v : &map_o)
                 : "memory");
  if (warp == kIssueSWarp) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  cluster_barrier();     // every CTA's barriers exist before anything is sent to them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (p.lets_next_start) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  bool ok = true;
  // Waits of the loaders and the issuers, by whole warps: with some lanes on one barrier and some on another
  // a warp went on about a thousand cycles after the last of them had flipped.
  auto wait_all = [&](uint32_t bar, uint32_t parity, int where) {
    ok = mbar_wait(bar, parity, abort_flag, p.status, kErrBase + where);
    ok = __all_sync(0xffffffffu, ok);
    return ok;
  };
  if (warp == kLoadKWarp || warp == kLoadVWarp) {
    // -------------------------------------------------------- loaders ----
    const uint32_t on = elect_one();
    const uint32_t arm = rank == leader ? on : 0u;     // the leader alone arms, for the bytes of both
    int j = 0;
    for (int i = 0; ok && i < blocks; ++i) {
      const int64_t block = first + i * step;
      const int head = (int)(block / p.q_blocks);
      if (warp == kLoadKWarp) {
        if (i >= 2 && !wait_all(q_empty(i), (uint32_t)((i >> 1) + 1) & 1u, 0x38)) break;
        const int row = (int)(block % p.q_blocks * (2 * kBQ)) + (int)(rank & 1u) * kBQ;
        mbar_expect_tx(q_full(i), 2 * kQBytes, arm);
        for (int h = 0; h < 2; ++h)
          tma_load_3d(&map_q, mapa_u32(q_full(i), leader), q_smem(i) + h * kHalfBytes, h * 64, head, row, on);
        for (int t = 0; t < n; ++t, ++j) {
          if (!wait_all(k_empty(j), (uint32_t)(j / kKSlots + 1) & 1u, 0x30)) break;
          const uint32_t bar = mapa_u32(k_full(j), leader);
          mbar_expect_tx(k_full(j), 2 * kSlotBytes, arm);
          for (int h = 0; h < 2; ++h)      // 64 of the tile's keys, the two halves of the head dimension
            tma_load_3d(&map_k, bar, k_smem(j) + h * (kSlotBytes / 2), h * 64, head,
                        (kv0 + t) * kBKV + (int)(rank & 1u) * (kBKV / 2), on);
        }
      } else {
        for (int t = 0; t < n; ++t, ++j) {
          if (!wait_all(v_empty(j), (uint32_t)(j / kVSlots + 1) & 1u, 0x34)) break;
          mbar_expect_tx(v_full(j), 2 * kSlotBytes, arm);
          tma_load_3d(&map_v, mapa_u32(v_full(j), leader), v_smem(j), (int)(rank & 1u) * 64, head, (kv0 + t) * kBKV,
                      on);
        }
      }
    }
    if (!ok) {
      // let copies already in flight land before the CTA's memory is released
      const long long t0 = clock64();
      while (clock64() - t0 < 2000000LL) {
      }
    }
  } else if (warp == kIssueSWarp) {
    // ------------------------------------------------- issuer of Q K^T ----
    if (rank == leader) {
      const uint32_t on = elect_one();
      const uint32_t idesc = make_idesc(false);
      int j = 0;
      for (int i = 0; ok && i < blocks; ++i) {
        if (!wait_all(q_full(i), (uint32_t)(i >> 1) & 1u, 0x10)) break;
        for (int t = 0; t < n; ++t, ++j) {
          // S = Q K^T: eight steps of 16 contraction elements (32 bytes inside the swizzled row,
          // the second 64 elements one half tile further)
          if (!wait_all(k_full(j), (uint32_t)(j / kKSlots) & 1u, 0x20) ||
              (j >= 2 && !wait_all(s_empty(j), (uint32_t)((j >> 1) - 1) & 1u, 0x40)))
            break;
          tc_fence_after();
          const uint64_t dq = desc_sw128(q_smem(i)), dk = desc_sw128(k_smem(j));
          const uint32_t d = tmem_base + kColS + (j & 1) * 128;
#pragma unroll
          for (int ks = 0; ks < kD / 16; ++ks)
            tc_mma_ss(d, dq + ((ks >> 2) * (kHalfBytes >> 4) + (ks & 3) * 2),
                      dk + ((ks >> 2) * (kSlotBytes >> 5) + (ks & 3) * 2), idesc, ks > 0, on);
          tc_commit(s_full(j), both, on);
          tc_commit(k_empty(j), both, on);
        }
        if (!ok) break;
        tc_commit(q_empty(i), both, on);
      }
    }
  } else if (warp == kIssueOWarp) {
    // --------------------------------------------------- issuer of P V ----
    if (rank == leader) {
      const uint32_t on = elect_one();
      const uint32_t idesc = make_idesc(true);
      int j = 0;
      for (int i = 0; ok && i < blocks; ++i) {
        if (i > 0 && !wait_all(o_empty(), (uint32_t)(i - 1) & 1u, 0x70)) break;
        for (int t = 0; t < n; ++t, ++j) {
          // O += P V: sixteen keys per step = eight 32-bit columns of P, two 8-key groups of V
          if (!wait_all(v_full(j), (uint32_t)(j / kVSlots) & 1u, 0x28) ||
              !wait_all(p_full(j), (uint32_t)(j >> 1) & 1u, 0x50))
            break;
          tc_fence_after();
          const uint64_t dv = desc_sw128(v_smem(j));
          const uint32_t a = tmem_base + kColP + (j & 1) * 64;
#pragma unroll
          for (int ks = 0; ks < kBKV / 16; ++ks)
            tc_mma_ts(tmem_base + kColO, a + ks * 8, dv + ks * (2048 >> 4), idesc, (t > 0 || ks > 0), on);
          tc_commit(pv_done(j), both, on);
          tc_commit(v_empty(j), both, on);
        }
      }
    }
  } else {
    // ------------------------------------------------------- softmax ----
    // Two groups of eight warps take the tiles by turns; two threads of a group have a row of its tile, 64 keys
    // each.  The four threads of a row follow the same maxima: their warps meet at named barriers, where a
    // warp waits at every tile of its own and arrives, without waiting, when it is through with the tile before one
    // of the other's.  A warp whose wait has run out goes through the rest of the walk without waiting, so
    // that no other is left at a barrier.
    const int group = warp >> 3;
    const int half = (warp >> 2) & 1;          // which 64 keys of the tile
    const int quarter = warp & 3;              // the lanes of tensor memory that this warp may touch
    const int r = quarter * 32 + lane;         // row in the CTA's 128
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const uint32_t s_addr = lane_addr + kColS + group * 128 + half * 64;
    const uint32_t p_addr = lane_addr + kColP + group * 64 + half * 32;
    const uint32_t o_addr = lane_addr + kColO;
    const uint32_t lead_s_empty = mapa_u32(s_empty(group), leader), lead_p_full = mapa_u32(p_full(group), leader),
                   lead_o_empty = mapa_u32(o_empty(), leader);
    const int my_bar = 1 + group * 4 + quarter, other_bar = 1 + (group ^ 1) * 4 + quarter, both_bar = 9 + quarter;
    auto wait = [&](uint32_t bar, uint32_t parity, int where) {
      if (ok) ok = mbar_wait(bar, parity, abort_flag, p.status, kErrBase + where);
      ok = __all_sync(0xffffffffu, ok);
    };
    auto max_slot = [&](int j, int h) { return row_max + ((j & 3) * 2 + h) * kBQ + r; };
    auto sum_slot = [&](int i, int gh) { return row_sum + ((i & 1) * 4 + gh) * kBQ + r; };
    const uint32_t on = elect_one();
    uint8_t* slab = smem_gen + kDataBytes + warp * kSlabBytes;
    const float c = p.scale_log2;
    uint32_t amax2 = 0u;
    // as if the tile before the first had been the second group's
    if (group == 1) asm volatile("bar.arrive %0, %1;" ::"r"(other_bar), "n"(128) : "memory");
    int j0 = 0;                                // running number of the block's first tile
    for (int i = 0; i < blocks; ++i, j0 += n) {
      float m_ref = -FLT_MAX;                  // the row's reference: no key yet, or none but keys with -inf
      float m_sum = 0.f;                       // ... and that of the sums below
      float2 sum0 = make_float2(0.f, 0.f), sum1 = make_float2(0.f, 0.f);   // this group's part of the row sum
      // The reference after a tile whose row maximum is m: the first tile's, raised where a later one exceeds it
      // by more than 2^8.  Both threads of a row apply this to the same maxima.  It is a number where every key so far
      // has -inf, so that these get no weight and any other raises it.
      auto follow = [&](float m) {
        const float m_new = m * c;
        if (m_new - m_ref > kRescaleStep) m_ref = m_new;
      };
      for (int j = j0 + ((j0 & 1) ^ group); j < j0 + n; j += 2) {
        const uint32_t parity = (uint32_t)(j >> 1) & 1u;
        wait(s_full(group), parity, 0x48 + group);
        tc_fence_after();
        uint32_t s[64];
        tc_ld32(s_addr, s);
        tc_ld32(s_addr + 32, s + 32);
        tc_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(lead_s_empty);
        // keys past the end of the sequence (their K rows were read as zeros) get no weight
        const int tile = kv0 + j - j0;
        if (tile == p.kv_tiles - 1) {
          const int valid = (int)(p.kv_len - (int64_t)tile * kBKV) - half * 64;
#pragma unroll
          for (int e = 0; e < 64; ++e)
            if (e >= valid) s[e] = 0xFF800000u;   // -inf
        }
        float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
        for (int e = 0; e < 64; e += 4) {
          mx0 = max3(mx0, __uint_as_float(s[e]), __uint_as_float(s[e + 1]));
          mx1 = max3(mx1, __uint_as_float(s[e + 2]), __uint_as_float(s[e + 3]));
        }
        float mx = fmaxf(mx0, mx1);
        *max_slot(j, half) = mx;
        asm volatile("bar.sync %0, %1;" ::"r"(my_bar), "n"(128) : "memory");
        const float before = fmaxf(*max_slot(j - 1, 0), *max_slot(j - 1, 1));     // the other group's
        mx = fmaxf(mx, *max_slot(j, half ^ 1));
        if (j > j0) follow(before);
        const float m_old = m_ref;
        follow(mx);
        if (__any_sync(0xffffffffu, m_ref != m_sum)) {
          if (__any_sync(0xffffffffu, j > j0 && m_ref != m_old)) {
            // O is at rest once the product of the tile before has been added.  (The one before that first: a
            // wait for a parity must not begin before the phase ahead of it is over.)
            if (j >= 2) wait(pv_done(group), parity ^ 1u, 0x62);
            wait(pv_done(group ^ 1), (uint32_t)((j - 1) >> 1) & 1u, 0x60);
            tc_fence_after();
            const float alpha = m_ref != m_old ? ex2(m_old - m_ref) : 1.f;
#pragma unroll 1
            for (int g = 0; g < 64 / 8; ++g) {
              uint32_t o[8];
              tc_ld8(o_addr + half * 64 + g * 8, o);
              tc_wait_ld();
#pragma unroll
              for (int e = 0; e < 8; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
              tc_st8(o_addr + half * 64 + g * 8, o);
            }
          }
          if (j > j0 + 1) {            // else the sums are still zero
            const float alpha = m_ref != m_sum ? ex2(m_sum - m_ref) : 1.f;
            sum0 = f2_mul(sum0, make_float2(alpha, alpha));
            sum1 = f2_mul(sum1, make_float2(alpha, alpha));
          }
          m_sum = m_ref;
        }
        // p = exp2(s*c - m); bf16 pairs and the row sum of what they hold
        const float2 c2 = make_float2(c, c);
        const float2 nm2 = make_float2(-m_ref, -m_ref);
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          float2 x = f2_fma(make_float2(__uint_as_float(s[2 * e]), __uint_as_float(s[2 * e + 1])), c2, nm2);
          if (kFmaExpEvery > 0 && e % (kFmaExpEvery > 0 ? kFmaExpEvery : 1) == 0) {
            x = exp2_fma(x);
          } else {
            x.x = ex2(x.x);
            x.y = ex2(x.y);
          }
          s[2 * e] = __float_as_uint(x.x);
          s[2 * e + 1] = __float_as_uint(x.y);
        }
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          const float2 x = make_float2(__uint_as_float(s[2 * e]), __uint_as_float(s[2 * e + 1]));
          float2& sum = (e & 1) ? sum1 : sum0;
          s[e] = f2_to_bf16x2(x);      // s[e] is dead by now: 2e, 2e+1 >= e
          sum = add_bf16x2(s[e], sum);
        }
        asm volatile("bar.arrive %0, %1;" ::"r"(other_bar), "n"(128) : "memory");
        // the product of this group's tile before has read the columns that P goes to
        if (j >= 2) wait(pv_done(group), parity ^ 1u, 0x62);
        tc_fence_after();
        tc_st32(p_addr, s);
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(lead_p_full);
      }
      // ---------------------------------------------------------- epilogue ----
      // The row sum of the two threads, on the reference of the one that had the last tile.
      const int last = j0 + n - 1;
      *sum_slot(i, group * 2 + half) = make_float2((sum0.x + sum0.y) + (sum1.x + sum1.y), m_sum);
      asm volatile("bar.sync %0, %1;" ::"r"(both_bar), "n"(128) : "memory");
      const int of_last = (last & 1) * 2, of_other = of_last ^ 2;
      m_ref = sum_slot(i, of_last)->y;
      float l = sum_slot(i, of_last)->x + sum_slot(i, of_last + 1)->x;
      if (n > 1) {
        const float2 a = *sum_slot(i, of_other);
        const float la = a.x + sum_slot(i, of_other + 1)->x;
        l += a.y == m_ref ? la : la * ex2(a.y - m_ref);
      }
      wait(pv_done(last), (uint32_t)(last >> 1) & 1u, 0x64);
      tc_fence_after();
      const int col = (group * 2 + half) * 32;    // this warp's columns of O
      uint32_t o[32];
      tc_ld32(o_addr + col, o);
      tc_wait_ld();
      if (kSplit) {
        // the partial result goes where the operands were: no product reads them any more
        if (group == 0 && half == 0)
          *reinterpret_cast<float2*>(smem_gen + kPartBytes + r * 8) = make_float2(m_ref > -FLT_MAX ? m_ref : -INFINITY, l);
#pragma unroll
        for (int q = 0; q < 8; ++q)
          *reinterpret_cast<uint4*>(smem_gen + part_offset(r, col / 4 + q)) =
              make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
      } else {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(lead_o_empty);
        const float inv = m_ref > -FLT_MAX ? 1.f / l : NAN;      // (no key has any weight)
#pragma unroll
        for (int e = 0; e < 16; ++e)
          o[e] = f2_to_bf16x2(make_float2(__uint_as_float(o[2 * e]) * inv, __uint_as_float(o[2 * e + 1]) * inv));
        // Through the warp's slab (64-byte swizzle, so that the lane-per-row writes spread over the banks)
        // and out with one TMA store, which clips at the last query: as 16-byte stores of 32 rows each they
        // kept the warps from the next block's tiles.
        const int64_t block = first + i * step;
        const int row0 = (int)(block % p.q_blocks * (2 * kBQ)) + (int)(rank & 1u) * kBQ + quarter * 32;
        if (row0 + lane < p.q_len) {
#pragma unroll
          for (int e = 0; e < 16; ++e) amax2 = bf16x2_max_abs(amax2, o[e]);
        }
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the store before has left the slab
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 4; ++q)
          *reinterpret_cast<uint4*>(slab + lane * 64 + ((q ^ ((lane >> 1) & 3)) << 4)) =
              make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        tma_store_3d(&map_o, smem_u32(slab), col, (int)(block / p.q_blocks), row0, row0 < p.q_len ? on : 0u);
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      }
    }
    // the shared memory must outlive the stores that read it
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    if (!kSplit && p.amax) {
      // non-negative floats order like their bit patterns: one atomic per warp
      const float a = fmaxf(bf16lo_to_f32(amax2), bf16hi_to_f32(amax2));
      const unsigned bits = __reduce_max_sync(0xffffffffu, __float_as_uint(a));
      if (lane == 0 && bits != 0u) atomicMax(p.amax, bits);
    }
    // the last tile's group has arrived once more for a tile that does not come
    if (group != ((total - 1) & 1)) asm volatile("bar.sync %0, %1;" ::"r"(my_bar), "n"(128) : "memory");
  }

  if (kSplit) {
    // ------------------------------------------- the parts of a block meet ----
    // The CTAs that hold the same 128 rows take a share of them each, eight output elements a thread at a
    // time: o = sum_k 2^(m_k - m) O_k / sum_k 2^(m_k - m) l_k over the parts k in their order.
    tc_fence_before();
    cluster_barrier();
    constexpr int kItems = kBQ * kD / 8;
    const int64_t row0 = first % p.q_blocks * (2 * kBQ) + (int64_t)(rank & 1u) * kBQ;
    uint8_t* dst = p.o + first / p.q_blocks * p.o_head_bytes;
    uint32_t amax2 = 0u;
    for (int i = kItems * part / kParts + threadIdx.x; i < kItems * (part + 1) / kParts; i += kThreads) {
      const int row = i >> 4, ch = (i & 15) * 2;
      if (row0 + row >= p.q_len) break;
      float2 ml[kParts];
      float m = -INFINITY;
#pragma unroll
      for (int k = 0; k < kParts; ++k) {
        ml[k] = ld_cluster_f2(smem_base + kPartBytes + row * 8, 2 * k + (rank & 1u));
        m = fmaxf(m, ml[k].x);
      }
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, sum = 0.f;
#pragma unroll
      for (int k = 0; k < kParts; ++k) {
        const float w = ex2(ml[k].x - m);
        const float4 a = ld_cluster_f4(smem_base + part_offset(row, ch), 2 * k + (rank & 1u));
        const float4 b = ld_cluster_f4(smem_base + part_offset(row, ch + 1), 2 * k + (rank & 1u));
        sum += w * ml[k].y;
        acc[0] += w * a.x; acc[1] += w * a.y; acc[2] += w * a.z; acc[3] += w * a.w;
        acc[4] += w * b.x; acc[5] += w * b.y; acc[6] += w * b.z; acc[7] += w * b.w;
      }
      const float inv = 1.f / sum;
      uint32_t o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        o[e] = f2_to_bf16x2(make_float2(acc[2 * e] * inv, acc[2 * e + 1] * inv));
        amax2 = bf16x2_max_abs(amax2, o[e]);
      }
      *reinterpret_cast<uint4*>(dst + (row0 + row) * p.o_row_bytes + ch * 8) = make_uint4(o[0], o[1], o[2], o[3]);
    }
    __syncwarp();
    if (p.amax) {
      const unsigned bits =
          __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(bf16lo_to_f32(amax2), bf16hi_to_f32(amax2))));
      if (lane == 0 && bits != 0u) atomicMax(p.amax, bits);
    }
    // Started while the launch before it ran (see launch()): what comes after this one in its stream waits
    // for this one alone, so this one ends after that.
    if (p.follows) grid_dependency_wait();
  }

  // No CTA of the cluster leaves while another may still use its barriers, its part or the shared
  // tensor-memory allocation.
  tc_fence_before();
  cluster_barrier();
  if (warp == kIssueSWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(kTmemCols)
                 : "memory");
  }
}

// ------------------------------------------------------------- host side ----

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                   const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &ptr, 12000, cudaEnableDefault,
                                         &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}

// Tensor map over bf16 [tokens][heads][128] with the given element strides: boxes of `box_tokens` x
// one head x 64 elements (128 bytes), 128-byte swizzle, tokens past the end read as zeros.
static bool make_map(CUtensorMap* map, const void* base, int64_t tokens, int heads, int64_t row_stride,
                     int64_t head_stride, int box_tokens, int box_width = 64) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return false;
  cuuint64_t dims[3] = {(cuuint64_t)kD, (cuuint64_t)heads, (cuuint64_t)tokens};
  cuuint64_t strides[2] = {(cuuint64_t)head_stride * 2u, (cuuint64_t)row_stride * 2u};
  cuuint32_t box[3] = {(cuuint32_t)box_width, 1u, (cuuint32_t)box_tokens};
  cuuint32_t elem[3] = {1u, 1u, 1u};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box,
            elem, CU_TENSOR_MAP_INTERLEAVE_NONE, box_width == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Per device, once: the shared memory a CTA may ask for.
template <int kParts>
int allow_smem(int dev) {
  static std::atomic<bool> done[64];
  if (done[dev].load(std::memory_order_acquire)) return NVFP4_OK;
  if (cudaFuncSetAttribute(attention_kernel<kParts>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes) !=
      cudaSuccess)
    return NVFP4_ERR_LAUNCH_FAILED;
  done[dev].store(true, std::memory_order_release);
  return NVFP4_OK;
}

// A launch whose blocks [p.first, p.end) are each computed by kParts pairs.
template <int kParts>
cudaLaunchConfig_t shared_config(const Params& p, cudaLaunchAttribute& attr, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * kParts * (p.end - p.first)));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = st;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = p.follows ? 1 : 0;
  return cfg;
}

template <int kParts>
int launch_shared(const CUtensorMap& map_q, const CUtensorMap& map_k, const CUtensorMap& map_v, const CUtensorMap& map_o,
                  const Params& p, int dev, cudaStream_t st) {
  const int rc = allow_smem<kParts>(dev);
  if (rc != NVFP4_OK) return rc;
  cudaLaunchAttribute attr;
  const cudaLaunchConfig_t cfg = shared_config<kParts>(p, attr, st);
  if (cudaLaunchKernelEx(&cfg, attention_kernel<kParts>, map_q, map_k, map_v, map_o, p) != cudaSuccess) {
    cudaGetLastError();
    return NVFP4_ERR_LAUNCH_FAILED;
  }
  return NVFP4_OK;
}

// Blocks that the GPU holds at a time when kParts pairs share each (0: it cannot be found out).
template <int kParts>
int resident_blocks(int dev) {
  static std::atomic<int> known[64];      // plus one; 0: not asked yet
  int c = known[dev].load(std::memory_order_relaxed);
  if (c == 0) {
    Params p{};
    p.end = 1;
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = shared_config<kParts>(p, attr, nullptr);
    int n = 0;
    if (allow_smem<kParts>(dev) != NVFP4_OK ||
        cudaOccupancyMaxActiveClusters(&n, attention_kernel<kParts>, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    known[dev].store(c = n + 1, std::memory_order_relaxed);
  }
  return c - 1;
}

// Pairs per block for the `rest` blocks that full waves of pairs leave over: 1 (they are a wave like the
// others), or 2 to kMaxParts where sharing their keys takes less time.  In units of a key tile (0.75 us) a wave
// of whole blocks costs its tiles and about 2 more; one of shared blocks their part of the tiles, 2, a
// meeting of 1 + parts, and 5 more behind other waves (its CTAs start as SMs get free, with empty rings).  Measured,
// us, whole and shared by 2, 3, 4 pairs: [1000, 5 heads] 13.3, 12.4, 13.5, 24.4 (more than are resident at a time);
// [300 x 512 keys, 3] 10.2, 10.6, 11.6, 11.9; behind two waves [3121, 12] 70.7, 66.0, 64.6, 64.0, [1760, 24]
// 45.0, 46.0, 46.6, 58.9; behind five [20000, 5] 911, 821, 843, 836.
int parts_for(int64_t rest, bool behind, int64_t tiles, int dev) {
  if (rest == 0 || tiles < 2) return 1;
  int best = 1;
  int64_t least = tiles + 2;
  for (int parts = 2; parts <= kMaxParts && parts <= tiles; ++parts) {
    const int64_t at_a_time = parts == 2 ? resident_blocks<2>(dev) : parts == 3 ? resident_blocks<3>(dev)
                                                                                : resident_blocks<4>(dev);
    if (at_a_time == 0) continue;
    const int64_t waves = (rest + at_a_time - 1) / at_a_time;
    const int64_t cost = waves * ((tiles + parts - 1) / parts + 3 + parts) + (behind ? 5 : 0);
    if (cost < least) {
      least = cost;
      best = parts;
    }
  }
  return best;
}

int launch(const CUtensorMap& map_q, const CUtensorMap& map_k, const CUtensorMap& map_v, const CUtensorMap& map_o,
           Params p, cudaStream_t st) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return NVFP4_ERR_BAD_ARG;
  int rc = allow_smem<1>(dev);
  if (rc != NVFP4_OK) return rc;
  p.q_blocks = (p.q_len + 2 * kBQ - 1) / (2 * kBQ);
  const int64_t blocks = p.q_blocks * p.heads;
  const int64_t pairs = sm_count() / 2, rest = blocks % pairs;
  const int parts = parts_for(rest, rest < blocks, p.kv_tiles, dev);
  const int64_t whole = parts == 1 ? blocks : blocks - rest;
  // a pair numbers its tiles in 31 bits: more than one launch only for views that overlap themselves
  const int64_t most = pairs * (((int64_t)1 << 30) / p.kv_tiles);
  while (p.first < whole) {
    Params w = p;
    w.end = whole - p.first < most ? whole : p.first + most;
    w.lets_next_start = parts > 1 && w.end == whole;
    const int64_t n = w.end - w.first < pairs ? w.end - w.first : pairs;
    attention_kernel<1><<<(unsigned)(2 * n), kThreads, kSmemBytes, st>>>(map_q, map_k, map_v, map_o, w);
    if (cudaGetLastError() != cudaSuccess) return NVFP4_ERR_LAUNCH_FAILED;
    p.first = w.end;
  }
  if (parts == 1) return NVFP4_OK;
  // Behind whole waves the shared blocks start as the first pairs get done.  They read nothing that those
  // write, and all that came before has completed when those start.
  p.follows = whole > 0;
  p.end = blocks;
  return parts == 2 ? launch_shared<2>(map_q, map_k, map_v, map_o, p, dev, st)
         : parts == 3 ? launch_shared<3>(map_q, map_k, map_v, map_o, p, dev, st)
                      : launch_shared<4>(map_q, map_k, map_v, map_o, p, dev, st);
}

}  // namespace attn
}  // namespace nvfp4

using namespace nvfp4;

extern "C" int nvfp4_attention_bf16(const void* q, int64_t q_row_stride, int64_t q_head_stride,
                                    const void* k, int64_t k_row_stride, int64_t k_head_stride,
                                    const void* v, int64_t v_row_stride, int64_t v_head_stride,
                                    int64_t q_len, int64_t kv_len, int heads, int head_dim,
                                    float softmax_scale, void* o, int64_t o_row_stride,
                                    int64_t o_head_stride, float* amax_dev, int* status_dev,
                                    void* stream) {
  if (q_len < 0 || kv_len < 1 || heads < 1 || heads > 65535 || head_dim != attn::kD ||
      q_len >= ((int64_t)1 << 31) || kv_len >= ((int64_t)1 << 31) || !(softmax_scale > 0.f))
    return NVFP4_ERR_BAD_ARG;
  if (q_len == 0) return NVFP4_OK;
  if (!q || !k || !v || !o) return NVFP4_ERR_BAD_ARG;
  const int64_t strides[8] = {q_row_stride, q_head_stride, k_row_stride, k_head_stride,
                              v_row_stride, v_head_stride, o_row_stride, o_head_stride};
  for (int64_t s : strides) {
    if (s < attn::kD || s >= ((int64_t)1 << 38)) return NVFP4_ERR_BAD_ARG;
    if (s % 8 != 0) return NVFP4_ERR_BAD_ALIGN;
  }
  if (!aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(o)) return NVFP4_ERR_BAD_ALIGN;
  int rc = check_device_sm100();
  if (rc != NVFP4_OK) return rc;

  CUtensorMap map_q, map_k, map_v, map_o;
  if (!attn::make_map(&map_q, q, q_len, heads, q_row_stride, q_head_stride, attn::kBQ) ||
      !attn::make_map(&map_k, k, kv_len, heads, k_row_stride, k_head_stride, attn::kBKV / 2) ||
      !attn::make_map(&map_v, v, kv_len, heads, v_row_stride, v_head_stride, attn::kBKV) ||
      !attn::make_map(&map_o, o, q_len, heads, o_row_stride, o_head_stride, 32, 32))
    return NVFP4_ERR_BAD_ARG;

  attn::Params p{};
  p.q_len = q_len;
  p.kv_len = kv_len;
  p.kv_tiles = (int)((kv_len + attn::kBKV - 1) / attn::kBKV);
  p.scale_log2 = softmax_scale * 1.4426950408889634f;
  p.o = static_cast<uint8_t*>(o);
  p.o_row_bytes = o_row_stride * 2;
  p.o_head_bytes = o_head_stride * 2;
  p.amax = reinterpret_cast<unsigned*>(amax_dev);
  p.status = status_dev;

  p.heads = heads;
  return attn::launch(map_q, map_k, map_v, map_o, p, reinterpret_cast<cudaStream_t>(stream));
}
