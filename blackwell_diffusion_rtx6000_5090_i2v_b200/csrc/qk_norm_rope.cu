// q/k RMSNorm across heads + rotary embedding, one pass over the QKV GEMM's output.
//
//   n = bf16( (x * rsqrt(mean(x^2) + eps)) * gain )            per token, over all heads
//   o[2i]   = bf16( n[2i] * c_i - n[2i+1] * s_i )              per head, pair i of head_dim/2
//   o[2i+1] = bf16( n[2i] * s_i + n[2i+1] * c_i )
//
// which is what the DiT block does between its QKV linear and attention
// (fx/src/s4/models/wan22/wan_transformer.py:91-92,114-115 for the norms, :61-75 for the
// rotation), there as about twenty elementwise torch kernels with fp32 round trips.  Every
// product and sum is rounded separately in fp32, as the unfused ops round them.  The value
// tensor can be carried along untouched so that q, k and v land in one packed
// [tokens, heads, 3 * head_dim] buffer ready for a head/sequence exchange.
//
// Bound: HBM, 8 B per element of q and k.  A row is reduced and then rewritten, so it has to be held.
// Two forms, neither of which stages it in shared memory:
//   CTA    a row per CTA, four 8-element chunks per thread, the next row's loads on their way while this one
//          is reduced and written
//   warp   a row per warp, a lane taking every 32nd chunk, all its loads in flight together and no barrier met
// The rotation-table entries of a thread are the same for all its chunks when a warp's (a CTA's) chunks
// are whole heads, and the gains come from L1.  The sum of squares is added in one fixed order whoever
// holds the chunks: W groups of 32 lanes (W = warps that four chunks per thread need), four chunks each,
// lanes by halving, then groups in pairs.
// [27280, 3 x 3072], L2 flushed: 160.7 us with the row staged, 125.0 a row per warp (two CTAs per SM; three
// at 80 registers: 135).  Which form when, and what each takes: warp_form().
// blockIdx.y selects the tensor: 0 = q, 1 = k, 2 = v (copy only).
#include "exchange_sync.cuh"
#include "nvfp4_common.cuh"

namespace nvfp4 {

int exchange_fill_peers(xsync::Peers& peers, void* const* sync_blocks, int world, int rank);  // exchange.cu

namespace {

constexpr int kThreads = 256;
constexpr int kMaxDim = 16384;

struct RopeArgs {
  const uint8_t* in[3];        // q, k, v: first element of row 0 (v may be null)
  int64_t in_row_bytes;        // distance between rows of an input
  int64_t rows;
  int dim;                     // heads * head_dim
  int head_dim;
  const float* gain[2];        // nullable: unit gain
  float eps;
  const float2* cos_sin;       // [rows][head_dim / 2] (cos of pair i, sin of pair i)
  uint8_t* out[3];
  int64_t out_row_bytes;
  int64_t out_head_bytes;
  // exchange form: heads are dealt out to `world` ranks, each of which receives its heads of
  // ALL tokens in a packed [tokens_total, heads_per_rank, 3 * head_dim] buffer
  uint8_t* peer[8];            // that buffer on every rank (this rank's own included)
  int heads_per_rank;          // 0: plain form
  int64_t row_offset;          // this rank's first token in the global order
  int signal;                  // exchange form: raise the peers' flags once the whole grid is done
  xsync::Peers peers;
};

// Destination of chunk c of row 0.
__device__ __forceinline__ uint8_t* chunk_dst(const RopeArgs& p, int which, int c, int per_head) {
  const int head = c / per_head, d0 = (c - head * per_head) * 8;
  uint8_t* dst = which == 0 ? p.out[0] : (which == 1 ? p.out[1] : p.out[2]);
  if (p.heads_per_rank > 0) {
    // plain stores into the owner rank's buffer (its own memory or a peer's over NVLink)
    const int owner = head / p.heads_per_rank;
#pragma unroll
    for (int r = 0; r < 8; ++r)
      if (r == owner) dst = p.peer[r];
    return dst + p.row_offset * p.out_row_bytes + (int64_t)(head - owner * p.heads_per_rank) * p.out_head_bytes +
           (int64_t)(which * p.head_dim + d0) * 2;
  }
  return dst + (int64_t)head * p.out_head_bytes + (int64_t)d0 * 2;
}

__device__ __forceinline__ void add_squares(const uint4& v, float2& s2) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 x = bf16x2_to_f2(w[e]);
    s2 = f2_fma(x, x, s2);
  }
}

__device__ __forceinline__ float warp_sum(float a) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  return a;
}

// Four pairs of a row: normalized, scaled by the gain and rounded to bf16 as the unfused model
// rounds them, then rotated.
__device__ __forceinline__ uint4 norm_rotate(const uint4& v, float2 r2, const float* gain, bool rotate,
                                             const float4 (&cs)[2]) {
  uint32_t o[4] = {v.x, v.y, v.z, v.w};
  float2 g[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) g[e] = make_float2(1.0f, 1.0f);
  if (gain) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const float4 t = load_f32x4(gain + 4 * q);
      g[2 * q] = make_float2(t.x, t.y);
      g[2 * q + 1] = make_float2(t.z, t.w);
    }
  }
  const float2 sign = make_float2(-1.0f, 1.0f);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    o[e] = f2_to_bf16x2(f2_mul(f2_mul(bf16x2_to_f2(o[e]), r2), g[e]));
    if (rotate) {
      const float2 n = bf16x2_to_f2(o[e]);
      const float4 t4 = cs[e >> 1];
      const float cc = (e & 1) ? t4.z : t4.x, ss = (e & 1) ? t4.w : t4.y;
      const float2 nc = f2_mul(n, make_float2(cc, cc));                      // (x1 c, x2 c)
      const float2 ns = f2_mul(make_float2(n.y, n.x), make_float2(ss, ss));  // (x2 s, x1 s)
      o[e] = f2_to_bf16x2(f2_fma(ns, sign, nc));   // (x1 c - x2 s, x2 c + x1 s), +-1 exact
    }
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}

// Warp form: one warp per row of at most 4 W groups of 32 chunks.
template <int W>
__global__ void __launch_bounds__(kThreads, 2) rope_warp_kernel(const RopeArgs p) {
  constexpr int kN = 4 * W, kRowsPerCta = kThreads / 32;
  extern __shared__ uint8_t* dst_tab[];
  const int which = blockIdx.y;                             // 0 q, 1 k, 2 v
  const int lane = threadIdx.x & 31;
  const int chunks = p.dim >> 3, per_head = p.head_dim >> 3;
  const uint8_t* in = which == 0 ? p.in[0] : (which == 1 ? p.in[1] : p.in[2]);
  const float* gain = which == 0 ? p.gain[0] : (which == 1 ? p.gain[1] : nullptr);
  const bool rotate = which < 2 && p.cos_sin != nullptr;
  for (int c = threadIdx.x; c < chunks; c += kThreads) dst_tab[c] = chunk_dst(p, which, c, per_head);
  __syncthreads();
  grid_dependency_wait();
  // a lane's chunks all sit at one place of their heads: one set of table entries per row
  const bool one_entry = 32 % per_head == 0;
  const int64_t half_hd = p.head_dim >> 1;
  const float dim_f = (float)p.dim;
  for (int64_t row = (int64_t)blockIdx.x * kRowsPerCta + (threadIdx.x >> 5); row < p.rows;
       row += (int64_t)gridDim.x * kRowsPerCta) {
    const uint4* src = reinterpret_cast<const uint4*>(in + row * p.in_row_bytes);
    const float4* table = reinterpret_cast<const float4*>(p.cos_sin + row * half_hd);
    uint4 v[kN];
#pragma unroll
    for (int j = 0; j < kN; ++j) {
      const int c = lane + j * 32;
      v[j] = c < chunks ? load_u32x4_once(src + c) : make_uint4(0, 0, 0, 0);
    }
    float4 cs[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
    if (rotate && one_entry) {
      cs[0] = load_f32x4(table + 2 * (lane % per_head));
      cs[1] = load_f32x4(table + 2 * (lane % per_head) + 1);
    }
    float rstd = 0.0f;
    if (which < 2) {
      float q[(W + 3) / 4 * 4] = {};
#pragma unroll
      for (int w = 0; w < W; ++w) {
        float2 s2 = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int k = 0; k < 4; ++k) add_squares(v[w + k * W], s2);    // chunks past the row hold zeros
        q[w] = warp_sum(s2.x + s2.y);
      }
      float t = 0.0f;
#pragma unroll
      for (int w = 0; w < W; w += 4) t += (q[w] + q[w + 1]) + (q[w + 2] + q[w + 3]);
      rstd = rsqrtf(t / dim_f + p.eps);
    }
    const float2 r2 = make_float2(rstd, rstd);
    const int64_t out_row = row * p.out_row_bytes;
#pragma unroll
    for (int j = 0; j < kN; ++j) {
      const int c = lane + j * 32;
      if (c >= chunks) break;
      if (which < 2) {
        if (rotate && !one_entry) {
          cs[0] = load_f32x4(table + 2 * (c % per_head));
          cs[1] = load_f32x4(table + 2 * (c % per_head) + 1);
        }
        v[j] = norm_rotate(v[j], r2, gain ? gain + 8 * c : nullptr, rotate, cs);
      }
      *reinterpret_cast<uint4*>(dst_tab[c] + out_row) = v[j];
    }
  }
  // exchange form: the CTA that finishes last tells every rank that this rank's pieces are in
  // place (flags of kind 0)
  if (p.signal) xsync::signal_when_grid_done(p.peers, 0, gridDim.x * gridDim.y, false);
}

// CTA form.  64 registers, so that 1024 threads of any CTA width fit an SM.
__global__ void __launch_bounds__(512, 2) rope_cta_kernel(const RopeArgs p) {
  extern __shared__ uint8_t* dst_tab[];
  __shared__ __align__(16) float red[2][16];
  const int which = blockIdx.y;
  const int lane = threadIdx.x & 31;
  const int T = blockDim.x;
  const int chunks = p.dim >> 3, per_head = p.head_dim >> 3;
  const uint8_t* in = which == 0 ? p.in[0] : (which == 1 ? p.in[1] : p.in[2]);
  const float* gain = which == 0 ? p.gain[0] : (which == 1 ? p.gain[1] : nullptr);
  const bool rotate = which < 2 && p.cos_sin != nullptr;
  const int64_t half_hd = p.head_dim >> 1;
  const float dim_f = (float)p.dim;
  for (int c = threadIdx.x; c < chunks; c += T) dst_tab[c] = chunk_dst(p, which, c, per_head);
  uint4 v[4], next[4];
  auto load = [&](int64_t row, uint4 (&d)[4]) {
    const uint4* src = reinterpret_cast<const uint4*>(in + row * p.in_row_bytes);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = threadIdx.x + k * T;
      d[k] = c < chunks ? load_u32x4_once(src + c) : make_uint4(0, 0, 0, 0);
    }
  };
  if (threadIdx.x < 32) (&red[0][0])[threadIdx.x] = 0.0f;
  __syncthreads();
  grid_dependency_wait();
  const bool one_entry = T % per_head == 0;      // as in the kernel above
  int parity = 0;
  if (blockIdx.x < p.rows) load(blockIdx.x, next);
  for (int64_t row = blockIdx.x; row < p.rows; row += gridDim.x, parity ^= 1) {
    const float4* table = reinterpret_cast<const float4*>(p.cos_sin + row * half_hd);
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = next[k];
    // the next row is on its way while this one is reduced and written
    if (row + gridDim.x < p.rows) load(row + gridDim.x, next);
    float4 cs[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
    if (rotate && one_entry) {
      cs[0] = load_f32x4(table + 2 * (threadIdx.x % per_head));
      cs[1] = load_f32x4(table + 2 * (threadIdx.x % per_head) + 1);
    }
    float rstd = 0.0f;
    if (which < 2) {
      float2 s2 = make_float2(0.0f, 0.0f);
#pragma unroll
      for (int k = 0; k < 4; ++k) add_squares(v[k], s2);
      const float a = warp_sum(s2.x + s2.y);
      // two buffers by turns: one is written again only after the barrier of the row in between
      if (lane == 0) red[parity][threadIdx.x >> 5] = a;
      __syncthreads();
      float t = 0.0f;
      for (int w = 0; w < T >> 5; w += 4) {
        const float4 q = *reinterpret_cast<const float4*>(&red[parity][w]);   // unused slots hold 0
        t += (q.x + q.y) + (q.z + q.w);
      }
      rstd = rsqrtf(t / dim_f + p.eps);
    }
    const float2 r2 = make_float2(rstd, rstd);
    const int64_t out_row = row * p.out_row_bytes;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = threadIdx.x + k * T;
      if (c >= chunks) break;
      if (which < 2) {
        if (rotate && !one_entry) {
          cs[0] = load_f32x4(table + 2 * (c % per_head));
          cs[1] = load_f32x4(table + 2 * (c % per_head) + 1);
        }
        v[k] = norm_rotate(v[k], r2, gain ? gain + 8 * c : nullptr, rotate, cs);
      }
      *reinterpret_cast<uint4*>(dst_tab[c] + out_row) = v[k];
    }
  }
  if (p.signal) xsync::signal_when_grid_done(p.peers, 0, gridDim.x * gridDim.y, false);
}

int64_t grid_x(int64_t rows, int rows_per_cta, int per_sm, int tensors) {
  const int64_t groups = (rows + rows_per_cta - 1) / rows_per_cta;
  const int64_t gx = ((int64_t)sm_count() * per_sm + tensors - 1) / tensors;
  return gx < groups ? gx : groups;
}

template <int W>
int launch_warp(const RopeArgs& a, int tensors, cudaStream_t st) {
  const int64_t gx = grid_x(a.rows, kThreads / 32, 2, tensors);     // the launch bound
  return launch_dependent(rope_warp_kernel<W>, dim3((unsigned)gx, (unsigned)tensors), kThreads,
                          (size_t)(a.dim / 8) * sizeof(uint8_t*), 1, st, a);
}

// The warp form wins where every warp has one row at most and the SMs are nearly full of them (its 16 warps
// per SM; for rows of one group from the first row on), and at three groups for many rows.  Replayed
// from a graph, us warp / CTA: [512, 6 heads of 128] 3.1 / 3.7, [1024, 12] 4.7 / 5.1, [1024, 24] 7.2 / 7.9,
// [32760, 24] 144 / 150, [32760, 20] 123 / 132; but [512, 24] 6.6 / 5.0, [1760, 24] 12.0 / 10.5, [8192, 12] 20.7 /
// 22.3, [32760, 12] 84 / 80, [32760, 6] 53 / 42.  Four or five groups, where a lane holds 16 or 20 chunks: [64,
// 40] 10.2 / 4.0, [1760, 40] 20.4 / 16.6, [32760, 32] 207 / 189, [32760, 40] 252 / 250.
bool warp_form(int W, int64_t rows) {
  const int64_t slots = (int64_t)sm_count() * 2 * (kThreads / 32);
  if (W > 3) return false;
  if (rows <= slots) return W == 1 || rows * 5 > slots * 4;
  return W == 3 && rows >= slots * 10;
}

int launch_rope(const RopeArgs& a, int tensors, cudaStream_t st) {
  const int W = ((a.dim / 8 + 3) / 4 + 31) / 32;
  if (warp_form(W, a.rows * tensors))
    return W == 1 ? launch_warp<1>(a, tensors, st) : W == 2 ? launch_warp<2>(a, tensors, st)
                                                            : launch_warp<3>(a, tensors, st);
  const int64_t gx = grid_x(a.rows, 1, 1024 / (32 * W), tensors);
  return launch_dependent(rope_cta_kernel, dim3((unsigned)gx, (unsigned)tensors), 32 * W,
                          (size_t)(a.dim / 8) * sizeof(uint8_t*), 1, st, a);
}

}  // namespace
}  // namespace nvfp4

using namespace nvfp4;

extern "C" NVFP4_API int nvfp4_qk_norm_rope_bf16(const void* q_in, const void* k_in, const void* v_in,
                                       int64_t in_row_stride, int64_t rows, int heads, int head_dim,
                                       const float* gain_q, const float* gain_k, float eps,
                                       const float* cos_sin, void* q_out, void* k_out, void* v_out,
                                       int64_t out_row_stride, int64_t out_head_stride,
                                       int* /*status_dev: nothing here waits*/, void* stream) {
  const int64_t dim = (int64_t)heads * head_dim;
  if (rows < 0 || heads <= 0 || head_dim <= 0 || head_dim % 16 != 0 || dim > kMaxDim ||
      in_row_stride < dim || out_head_stride < head_dim || in_row_stride % 8 != 0 ||
      out_row_stride % 8 != 0 || out_head_stride % 8 != 0)
    return NVFP4_ERR_BAD_ARG;
  if (rows > 0 && (!q_in || !q_out)) return NVFP4_ERR_BAD_ARG;
  if ((k_in == nullptr) != (k_out == nullptr) || (v_in == nullptr) != (v_out == nullptr) ||
      (v_in && !k_in))
    return NVFP4_ERR_BAD_ARG;
  if (!aligned16(q_in) || !aligned16(k_in) || !aligned16(v_in) || !aligned16(q_out) ||
      !aligned16(k_out) || !aligned16(v_out) || !aligned16(gain_q) || !aligned16(gain_k) ||
      !aligned16(cos_sin))
    return NVFP4_ERR_BAD_ALIGN;
  int rc = check_device_sm100();
  if (rc != NVFP4_OK) return rc;
  if (rows == 0) return NVFP4_OK;
  RopeArgs a{};
  a.in[0] = static_cast<const uint8_t*>(q_in);
  a.in[1] = static_cast<const uint8_t*>(k_in);
  a.in[2] = static_cast<const uint8_t*>(v_in);
  a.in_row_bytes = in_row_stride * 2;
  a.rows = rows;
  a.dim = (int)dim;
  a.head_dim = head_dim;
  a.gain[0] = gain_q;
  a.gain[1] = gain_k;
  a.eps = eps;
  a.cos_sin = reinterpret_cast<const float2*>(cos_sin);
  a.out[0] = static_cast<uint8_t*>(q_out);
  a.out[1] = static_cast<uint8_t*>(k_out);
  a.out[2] = static_cast<uint8_t*>(v_out);
  a.out_row_bytes = out_row_stride * 2;
  a.out_head_bytes = out_head_stride * 2;
  return launch_rope(a, v_in ? 3 : (k_in ? 2 : 1), reinterpret_cast<cudaStream_t>(stream));
}

extern "C" NVFP4_API int nvfp4_qk_norm_rope_exchange_bf16(
    const void* q_in, const void* k_in, const void* v_in, int64_t in_row_stride, int64_t rows,
    int heads, int head_dim, const float* gain_q, const float* gain_k, float eps,
    const float* cos_sin, void* const* rank_buffers, int world, int64_t row_offset,
    void* const* sync_blocks, int rank, int* /*status_dev: nothing here waits*/, void* stream) {
  const int64_t dim = (int64_t)heads * head_dim;
  if (rows < 0 || heads <= 0 || head_dim <= 0 || head_dim % 16 != 0 || dim > kMaxDim ||
      in_row_stride < dim || in_row_stride % 8 != 0 || world < 1 || world > 8 ||
      heads % world != 0 || row_offset < 0 || !rank_buffers)
    return NVFP4_ERR_BAD_ARG;
  if (rows > 0 && (!q_in || !k_in || !v_in)) return NVFP4_ERR_BAD_ARG;
  if (!aligned16(q_in) || !aligned16(k_in) || !aligned16(v_in) || !aligned16(gain_q) ||
      !aligned16(gain_k) || !aligned16(cos_sin))
    return NVFP4_ERR_BAD_ALIGN;
  for (int r = 0; r < world; ++r) {
    if (!rank_buffers[r]) return NVFP4_ERR_BAD_ARG;
    if (!aligned16(rank_buffers[r])) return NVFP4_ERR_BAD_ALIGN;
  }
  RopeArgs a{};
  if (sync_blocks) {
    // a rank with nothing to send would raise no flag and leave its peers waiting
    if (rows == 0) return NVFP4_ERR_BAD_ARG;
    const int prc = exchange_fill_peers(a.peers, sync_blocks, world, rank);
    if (prc != NVFP4_OK) return prc;
    a.signal = 1;
  }
  int rc = check_device_sm100();
  if (rc != NVFP4_OK) return rc;
  if (rows == 0) return NVFP4_OK;
  a.in[0] = static_cast<const uint8_t*>(q_in);
  a.in[1] = static_cast<const uint8_t*>(k_in);
  a.in[2] = static_cast<const uint8_t*>(v_in);
  a.in_row_bytes = in_row_stride * 2;
  a.rows = rows;
  a.dim = (int)dim;
  a.head_dim = head_dim;
  a.gain[0] = gain_q;
  a.gain[1] = gain_k;
  a.eps = eps;
  a.cos_sin = reinterpret_cast<const float2*>(cos_sin);
  a.heads_per_rank = heads / world;
  a.out_head_bytes = (int64_t)3 * head_dim * 2;
  a.out_row_bytes = (int64_t)a.heads_per_rank * a.out_head_bytes;
  a.row_offset = row_offset;
  for (int r = 0; r < world; ++r) a.peer[r] = static_cast<uint8_t*>(rank_buffers[r]);
  return launch_rope(a, 3, reinterpret_cast<cudaStream_t>(stream));
}
