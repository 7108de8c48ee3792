// NVFP4 quantizer of the transpose of a bf16 matrix, for the gradient GEMMs of the linear: both
// contract over an axis that is not the contiguous one of their operands
// (fx/src/s4/nvfp4/linear/nvfp4_gemm_kernel.cu:151-196), and the 16-element scale blocks run along
// the contraction.
//
// Bound: HBM, 2 B/element in and 0.5625 out.  Instead of a transposed bf16 copy that the quantizer
// then reads (4 more bytes per element and a launch), a CTA takes 128 x 64 tiles through shared
// memory: rows go in as they are, each thread reads back the 16 words of one column pair and
// one 16-row group, which are two whole scale blocks.  The words of a 16-row group are rotated by
// four banks per group, so that the eight groups x four column pairs of a warp hit 32 banks.
//
// The gradients of a linear want up to three such operands, dy also in its own direction, and dy's column
// sums: one launch makes them all (quantize_jobs), every tile read once.  The direct form of a tile is packed from
// the registers that brought it; the sums of a tile's columns are left as partial sums, which the CTA that
// finishes a column of tiles last adds in their order.  [2048, 3072] x 3072: 21 us for dy both ways, x, w and the
// sums, where five kernels took 40 (rows form 6.3, three transposes of 6.7, torch's column sum 13.2).
#include "nvfp4_common.cuh"

namespace nvfp4 {
namespace {

constexpr int kThreads = 256;
constexpr int kTileRows = 128;     // eight scale blocks of the transpose
constexpr int kTileCols = 64;      // its rows
constexpr int kTilePieces = kTileRows * kTileCols / 8 / kThreads;   // 16-byte pieces of a thread

struct TransposeArgs {
  QuantizeJob job[kQuantizeJobs];
  uint32_t first[kQuantizeJobs + 1];   // tiles of job i: first[i] up to first[i + 1]
  const unsigned* partial;
};

// E2M1 codes and the scale of a block whose two 16-byte halves are a, b
__device__ __forceinline__ uint2 pack_halves(const uint4& a, const uint4& b, float s_enc, const float* enc_tab,
                                             uint32_t& sf) {
  const uint32_t h[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  uint32_t a2 = 0u;
#pragma unroll
  for (int i = 0; i < 8; ++i) a2 = bf16x2_max_abs(a2, h[i]);
  return pack_block(h, a2, s_enc, enc_tab, sf);
}
__device__ __forceinline__ uint4 shfl_xor1(const uint4& v) {
  return make_uint4(__shfl_xor_sync(0xffffffffu, v.x, 1), __shfl_xor_sync(0xffffffffu, v.y, 1),
                    __shfl_xor_sync(0xffffffffu, v.z, 1), __shfl_xor_sync(0xffffffffu, v.w, 1));
}

// kJobs = 1: one transposed operand whose maximum is in its slot; else any of what QuantizeJob says.
template <int kJobs>
__global__ void __launch_bounds__(kThreads, kJobs == 1 ? 4 : 3) quantize_transposed_kernel(const TransposeArgs p) {
  __shared__ __align__(16) uint32_t tile[kTileRows * kTileCols / 2];
  __shared__ float enc_tab[kJobs][128];
  __shared__ float s_encs[kJobs];
  __shared__ unsigned warp_max[kThreads / 32];
  __shared__ int is_last;
  __shared__ float sums[kThreads];
  const int lane = threadIdx.x & 31;
  const int group = lane & 7;                              // 16-row group of the tile
  const int pair = (threadIdx.x >> 5) * 4 + (lane >> 3);   // column pair of the tile
  grid_dependency_wait();

  // The first tile is on its way while the scales are worked out.  (Tile numbers and coordinates fit 32 bits: a job has
  // at most 2^35 elements.  Offsets are worked out once a tile: with 64-bit divisions for every load and every use the
  // index arithmetic was two thirds of the instructions.)
  uint4 v[kTilePieces];
  struct Where {
    int job;
    uint32_t row_tile, col_tile;
  };
  auto where = [&](uint32_t t) {
    int j = 0;
#pragma unroll
    for (int k = 1; k < kJobs; ++k) j += t >= p.first[k];
    const uint32_t tt = t - p.first[j], per_row = p.job[j].col_tiles, row = tt / per_row;
    return Where{j, row, tt - row * per_row};
  };
  auto load = [&](const Where& at) {
    const QuantizeJob& q = p.job[at.job];
    const uint32_t r = at.row_tile * kTileRows + (threadIdx.x >> 3), c = at.col_tile * kTileCols + (threadIdx.x & 7) * 8;
    const uint8_t* src = static_cast<const uint8_t*>(q.x) + ((int64_t)r * q.cols + c) * 2;
    const int64_t step = (int64_t)q.cols * (2 * kThreads / 8);
    const int rows_left = c < q.cols ? (int)(q.rows - r) : 0;      // rows >= r wraps to a negative number
#pragma unroll
    for (int j = 0; j < kTilePieces; ++j)
      v[j] = rows_left > j * (kThreads / 8) ? load_u32x4(src + j * step) : make_uint4(0, 0, 0, 0);
  };
  const uint32_t tiles = p.first[kJobs];
  Where at = where(blockIdx.x);
  load(at);
#pragma unroll
  for (int k = 0; k < kJobs; ++k) {
    const QuantizeJob& q = p.job[k];
    if (kJobs > 1 && p.first[k] == p.first[k + 1]) continue;
    float amax_g;
    if (kJobs > 1 && q.n_partial > 0) {
      unsigned m = max_of_partials(p.partial + q.first_partial, q.n_partial);
      m = __reduce_max_sync(0xffffffffu, m);
      if (lane == 0) warp_max[threadIdx.x >> 5] = m;
      __syncthreads();
#pragma unroll
      for (int w = 0; w < kThreads / 32; ++w) m = max(m, warp_max[w]);
      __syncthreads();
      amax_g = __uint_as_float(m);
    } else {
      amax_g = load_f32(q.amax);
    }
    const float s_enc = global_encode_scale(amax_g);
    const float s_dec = __fdiv_rn(1.0f, s_enc);
    if (threadIdx.x == 0) {
      s_encs[k] = s_enc;
      if (blockIdx.x == 0) {
        if (q.t_gscale) *q.t_gscale = s_dec;
        if (kJobs > 1 && q.gscale) *q.gscale = s_dec;
      }
    }
    fill_encode_table(enc_tab[k], s_dec);
  }

  for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    const int ji = at.job;
    const QuantizeJob& q = p.job[ji];
    const uint32_t row_tile = at.row_tile, col_tile = at.col_tile;
    const uint32_t row0 = row_tile * kTileRows, col0 = col_tile * kTileCols;
    const bool more = t + gridDim.x < tiles;
    if (more) at = where(t + gridDim.x);
    __syncthreads();     // the previous tile has been read, the tables are there
    const float s_enc = s_encs[ji];
#pragma unroll
    for (int j = 0; j < kTilePieces; ++j) {
      const int i = threadIdx.x + j * kThreads;
      const int r = i >> 3;
      *reinterpret_cast<uint4*>(&tile[r * 32 + (((i & 7) * 4 + 4 * (r >> 4)) & 31)]) = v[j];
    }
    if (kJobs > 1 && q.packed) {
      // Direct form, from the registers: two neighbouring lanes hold the halves of a block of each of four rows;
      // after the exchange the even lane has the whole blocks of the first two rows, the odd one those of the others.
      const bool odd = lane & 1;
      const uint4 g0 = shfl_xor1(odd ? v[0] : v[2]), g1 = shfl_xor1(odd ? v[1] : v[3]);
      const uint4 k0 = odd ? v[2] : v[0], k1 = odd ? v[3] : v[1];
      const int quarter = (lane & 7) >> 1;                 // block of the tile's row
      const uint32_t kb = (col0 >> 4) + quarter, in_tile = (threadIdx.x >> 3) + (odd ? 64 : 0), r = row0 + in_tile;
      uint2* dst = q.packed + (int64_t)r * q.units + kb;
      uint32_t word[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const uint4 mine = e ? k1 : k0, got = e ? g1 : g0;
        uint32_t sf;
        const uint2 out = pack_halves(odd ? got : mine, odd ? mine : got, s_enc, enc_tab[ji], sf);
        if (r + 32 * e < q.rows && kb < q.units) dst[e ? 32 * (int64_t)q.units : 0] = out;
        word[e] = sf << (8 * quarter);
      }
      // the four scale bytes of a row meet, and leave as a word; the tile's are one atom
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        word[e] |= __shfl_xor_sync(0xffffffffu, word[e], 2);
        word[e] |= __shfl_xor_sync(0xffffffffu, word[e], 4);
      }
      if (quarter < 2)
        *reinterpret_cast<uint32_t*>(q.scales + ((int64_t)row_tile * q.k_atoms + col_tile) * kSfAtomBytes +
                                     (in_tile & 31) * 16 + (in_tile >> 5) * 4 + quarter * 4) = quarter ? word[1] : word[0];
    }
    if (kJobs == 1 || q.t_packed || q.col_sum) {
      __syncthreads();
      uint32_t w[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) w[i] = tile[(group * 16 + i) * 32 + ((pair + 4 * group) & 31)];
      if (more) load(at);
      if (kJobs == 1 || q.t_packed) {
        const uint32_t kb = (row0 >> 4) + group, n = col0 + 2 * pair;
        uint2* dst = q.t_packed + (int64_t)n * q.t_units + kb;
        uint32_t sf2 = 0u;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          uint32_t h[8], a2 = 0u, sf;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            h[i] = __byte_perm(w[2 * i], w[2 * i + 1], e ? 0x7632 : 0x5410);
            a2 = bf16x2_max_abs(a2, h[i]);
          }
          const uint2 out = pack_block(h, a2, s_enc, enc_tab[ji], sf);
          if (n + e < q.cols && kb < q.t_units) dst[e ? q.t_units : 0] = out;
          sf2 |= sf << (8 * e);
        }
        // lanes 0 and 1 of a quad leave with the four K-blocks of the pair's two columns; the tiles
        // cover the padded layout, where everything outside the matrix has scale 0
        sf2 = quad_transpose(sf2);
        if ((lane & 3) < 2) {
          const uint32_t m = n + (lane & 3);
          *reinterpret_cast<uint32_t*>(q.t_scales + ((int64_t)(m >> 7) * q.t_k_atoms + (kb >> 2)) * kSfAtomBytes +
                                       (m & 31) * 16 + ((m >> 5) & 3) * 4) = sf2;
        }
      }
      if (kJobs > 1 && q.col_sum) {
        float2 s = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int i = 0; i < 16; ++i) s = f2_add(s, bf16x2_to_f2(w[i]));
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
          s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
          s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
        }
        const uint32_t ld = q.col_tiles * kTileCols, row_tiles = q.row_tiles;
        if (group == 0) *reinterpret_cast<float2*>(q.col_partial + (int64_t)row_tile * ld + col0 + 2 * pair) = s;
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) {
          is_last = atomicAdd(q.col_count + col_tile, 1u) + 1u == row_tiles;
          __threadfence();
        }
        __syncthreads();
        if (is_last) {
          // a quarter of the row tiles each, then the quarters: the same order whoever comes last
          const int c = threadIdx.x & (kTileCols - 1);
          float a = 0.0f;
          for (uint32_t i = threadIdx.x / kTileCols; i < row_tiles; i += kThreads / kTileCols)
            a += load_f32(q.col_partial + (int64_t)i * ld + col0 + c);
          sums[threadIdx.x] = a;
          __syncthreads();
          if (threadIdx.x < kTileCols && col0 + c < q.cols)
            q.col_sum[col0 + c] = __float2bfloat16((sums[c] + sums[c + 64]) + (sums[c + 128] + sums[c + 192]));
        }
      }
    } else if (more) {
      load(at);
    }
  }
}

}  // namespace

// Both layouts are padded to whole tiles: rows and K-blocks of either to 256 elements.
int64_t quantize_job_col_tiles(int64_t cols) { return sf_row_tiles(cols) * (128 / kTileCols); }
int64_t quantize_job_row_tiles(int64_t rows) { return sf_row_tiles(rows) * (128 / kTileRows); }

namespace {

template <int kJobs>
int launch_jobs(TransposeArgs& a, const QuantizeJob* jobs, const float* partials, void* stream) {
  for (int i = 0; i < kJobs; ++i) {
    QuantizeJob& q = a.job[i];
    q = jobs[i];
    a.first[i + 1] = a.first[i];
    if (!q.x) continue;
    q.col_tiles = (uint32_t)quantize_job_col_tiles(q.cols);
    q.row_tiles = (uint32_t)quantize_job_row_tiles(q.rows);
    a.first[i + 1] += q.col_tiles * q.row_tiles;
  }
  a.partial = reinterpret_cast<const unsigned*>(partials);
  const uint32_t tiles = a.first[kJobs], resident = (uint32_t)sm_count() * (kJobs == 1 ? 4 : 3);   // the launch bound's
  return launch_dependent(quantize_transposed_kernel<kJobs>, dim3(tiles < resident ? tiles : resident),
                          kThreads, 0, 1, reinterpret_cast<cudaStream_t>(stream), a);
}

}  // namespace

int quantize_jobs(const QuantizeJob (&jobs)[kQuantizeJobs], const float* partials, void* stream) {
  TransposeArgs a{};
  return launch_jobs<kQuantizeJobs>(a, jobs, partials, stream);
}

}  // namespace nvfp4

using namespace nvfp4;

extern "C" int nvfp4_quantize_transposed_bf16(const void* x, int64_t rows, int64_t cols,
                                              const float* amax_dev, uint8_t* packed,
                                              uint8_t* scales_swizzled, float* global_scale_dev,
                                              void* stream) {
  if (rows <= 0 || cols <= 0 || cols % 8 != 0 || rows >= ((int64_t)1 << 31) || cols >= ((int64_t)1 << 31))
    return NVFP4_ERR_BAD_ARG;
  const int64_t k = (rows + 31) / 32 * 32;
  if (k * cols / kBlock >= ((int64_t)1 << 31)) return NVFP4_ERR_BAD_ARG;
  if (!x || !amax_dev || !packed || !scales_swizzled) return NVFP4_ERR_BAD_ARG;
  if (!aligned16(x) || !aligned16(scales_swizzled) || (reinterpret_cast<uintptr_t>(packed) & 7u))
    return NVFP4_ERR_BAD_ALIGN;
  int rc = check_device_sm100();
  if (rc != NVFP4_OK) return rc;
  QuantizeJob q{};
  q.x = x;
  q.rows = (uint32_t)rows;
  q.cols = (uint32_t)cols;
  q.amax = amax_dev;
  q.t_packed = reinterpret_cast<uint2*>(packed);
  q.t_scales = scales_swizzled;
  q.t_gscale = global_scale_dev;
  q.t_units = (uint32_t)(k / kBlock);
  q.t_k_atoms = (uint32_t)sf_k_atoms(k);
  TransposeArgs a{};
  return launch_jobs<1>(a, &q, nullptr, stream);
}
