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
// One training pass of a [2048, 3072] x 3072 linear, bound by the host there: 453 -> 412 us.
#include "nvfp4_common.cuh"

namespace nvfp4 {
namespace {

constexpr int kThreads = 256;
constexpr int kTileRows = 128;     // eight scale blocks of the transpose
constexpr int kTileCols = 64;      // its rows

struct TransposeArgs {
  const uint8_t* x;
  int64_t rows, cols;
  int64_t kb;                      // scale blocks per row of the transpose (rows padded to 32 elements)
  const float* amax;
  uint2* packed;
  uint8_t* sf_swz;
  int64_t k_atoms;
  float* gscale_out;
  int64_t col_tiles, tiles;
};

__global__ void __launch_bounds__(kThreads, 4) quantize_transposed_kernel(const TransposeArgs p) {
  __shared__ __align__(16) uint32_t tile[kTileRows * kTileCols / 2];
  __shared__ float enc_tab[128];
  grid_dependency_wait();
  const float s_enc = global_encode_scale(load_f32(p.amax));
  const float s_dec = __fdiv_rn(1.0f, s_enc);
  if (p.gscale_out && blockIdx.x == 0 && threadIdx.x == 0) *p.gscale_out = s_dec;
  fill_encode_table(enc_tab, s_dec);
  const int lane = threadIdx.x & 31;
  const int group = lane & 7;                              // 16-row group of the tile
  const int pair = (threadIdx.x >> 5) * 4 + (lane >> 3);   // column pair of the tile
  for (int64_t t = blockIdx.x; t < p.tiles; t += gridDim.x) {
    const int64_t row0 = t / p.col_tiles * kTileRows, col0 = t % p.col_tiles * kTileCols;
    uint4 v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = threadIdx.x + j * kThreads;            // 16-byte piece of the tile
      const int64_t r = row0 + (i >> 3), c = col0 + (i & 7) * 8;
      v[j] = r < p.rows && c < p.cols ? load_u32x4(p.x + (r * p.cols + c) * 2)
                                      : make_uint4(0, 0, 0, 0);
    }
    __syncthreads();     // the previous tile has been read
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = threadIdx.x + j * kThreads;
      const int r = i >> 3;
      *reinterpret_cast<uint4*>(&tile[r * 32 + (((i & 7) * 4 + 4 * (r >> 4)) & 31)]) = v[j];
    }
    __syncthreads();
    uint32_t w[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) w[i] = tile[(group * 16 + i) * 32 + ((pair + 4 * group) & 31)];
    const int64_t kb = (row0 >> 4) + group;
    uint32_t sf2 = 0u;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      uint32_t h[8], a2 = 0u, sf;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        h[i] = __byte_perm(w[2 * i], w[2 * i + 1], e ? 0x7632 : 0x5410);
        a2 = bf16x2_max_abs(a2, h[i]);
      }
      const uint2 out = pack_block(h, a2, s_enc, enc_tab, sf);
      const int64_t n = col0 + 2 * pair + e;
      if (n < p.cols && kb < p.kb) p.packed[n * p.kb + kb] = out;
      sf2 |= sf << (8 * e);
    }
    // lanes 0 and 1 of a quad leave with the four K-blocks of the pair's two columns; the tiles
    // cover the padded layout, where everything outside the matrix has scale 0
    sf2 = quad_transpose(sf2);
    if ((lane & 3) < 2) {
      const int64_t n = col0 + 2 * pair + (lane & 3);
      *reinterpret_cast<uint32_t*>(p.sf_swz + sf_swizzled_offset(n, kb & ~(int64_t)3, p.k_atoms)) = sf2;
    }
  }
}

}  // namespace
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
  TransposeArgs a{};
  a.x = static_cast<const uint8_t*>(x);
  a.rows = rows;
  a.cols = cols;
  a.kb = k / kBlock;
  a.amax = amax_dev;
  a.packed = reinterpret_cast<uint2*>(packed);
  a.sf_swz = scales_swizzled;
  a.k_atoms = sf_k_atoms(k);
  a.gscale_out = global_scale_dev;
  a.col_tiles = sf_row_tiles(cols) * (128 / kTileCols);
  a.tiles = a.col_tiles * (a.k_atoms * 4 / 8);
  const int64_t resident = (int64_t)sm_count() * 4;        // the launch bound's CTAs per SM
  return launch_dependent(quantize_transposed_kernel, dim3((unsigned)(a.tiles < resident ? a.tiles : resident)),
                          kThreads, 0, 1, reinterpret_cast<cudaStream_t>(stream), a);
}
