// Leaf hashing and node compression with the tensor-core permutation
// (p2_tensor.cuh); merkle.cu decides which sizes run here.
#include "kernels.h"
#include "launch.cuh"
#include "merkle_tensor.h"
#include "p2_tensor.cuh"

namespace whir {
namespace gpu {

namespace {
__device__ uint4 g_tab16[P2Mat<16>::bytes / 16];
__device__ uint4 g_tab24[P2Mat<24>::bytes / 16];

struct Tri {
  int32_t v[4];
};

// Row r of a tile is one leaf: chunks of 16 words overwrite the rate, each
// followed by a permutation; a shorter last chunk overwrites only its words.
// VEC: rows of a multiple of 4 words on 16-byte boundaries.
template <bool VEC>
__device__ __forceinline__ void load_chunk(const uint32_t *__restrict__ row, int pos, int row_len,
                                           uint32_t (&x)[16]) {
  if constexpr (VEC) {
#pragma unroll
    for (int q = 0; q < 4; q++)
      if (pos + 4 * q < row_len) {
        const uint4 v = __ldg(reinterpret_cast<const uint4 *>(row + pos) + q);
        x[4 * q] = v.x; x[4 * q + 1] = v.y; x[4 * q + 2] = v.z; x[4 * q + 3] = v.w;
      }
  } else {
#pragma unroll
    for (int j = 0; j < 16; j++)
      if (pos + j < row_len) x[j] = __ldg(row + pos + j);
  }
}

template <bool VEC>
__global__ void __launch_bounds__(p2t_threads<24>, 1)
    hash_rows_tensor_kernel(const uint32_t *__restrict__ rows, size_t n_rows, int row_len,
                            uint32_t *__restrict__ digests, const Tri tri, const WaitReport report) {
  extern __shared__ __align__(128) unsigned char sm[];
  P2Tile<24> t = p2t_begin<24>(sm, g_tab24, report);
  pdl_wait();
  const size_t tiles = (n_rows + 127) / 128, step = (size_t)gridDim.x * P2Mat<24>::TILES;
  const int lane_row = threadIdx.x & 127;
  size_t tile = (size_t)(threadIdx.x >> 7) * gridDim.x + blockIdx.x;
  uint32_t x[16];
  // rows past the end repeat the last one; only their stores are left out
  auto row_of = [&](size_t tl) {
    const size_t r = tl * 128 + lane_row;
    return rows + (r < n_rows ? r : n_rows - 1) * row_len;
  };
  const uint32_t *row = nullptr;
  if (tile < tiles) {
    row = row_of(tile);
#pragma unroll
    for (int j = 0; j < 16; j++) x[j] = 0;
    load_chunk<VEC>(row, 0, row_len, x);
  }
  while (tile < tiles) {
    const size_t at = tile * 128 + lane_row;
    uint32_t cap[8];
#pragma unroll
    for (int j = 0; j < 8; j++) cap[j] = 0;
    int pos = 0;
    for (;;) {
      {
        uint32_t u[8];
#pragma unroll
        for (int j = 0; j < 8; j++) u[j] = x[j];
        t.put_words(0, u);
#pragma unroll
        for (int j = 0; j < 8; j++) u[j] = x[8 + j];
        t.put_words(8, u);
        t.put_words(16, cap);
      }
      pos += 16;
      const bool last = pos >= row_len;
      t.permute(tri.v, [&] {
        // the next chunk of this row, or the next tile's first
        if (!last) {
          load_chunk<VEC>(row, pos, row_len, x);
        } else if (tile + step < tiles) {
          row = row_of(tile + step);
#pragma unroll
          for (int j = 0; j < 16; j++) x[j] = 0;
          load_chunk<VEC>(row, 0, row_len, x);
        }
      });
      if (last) break;
      int32_t v[8];
      t.get_words(16, v);
#pragma unroll
      for (int j = 0; j < 8; j++) cap[j] = p2t_unsigned(v[j]);
      if (row_len - pos < 16) {  // a short chunk keeps the words it does not overwrite
        t.get_words(0, v);
#pragma unroll
        for (int j = 0; j < 8; j++)
          if (pos + j >= row_len) x[j] = p2t_unsigned(v[j]);
        t.get_words(8, v);
#pragma unroll
        for (int j = 0; j < 8; j++)
          if (pos + 8 + j >= row_len) x[8 + j] = p2t_unsigned(v[j]);
      }
    }
    int32_t v[8];
    t.get_words(0, v);
    if (at < n_rows) {
      uint4 *dst = reinterpret_cast<uint4 *>(digests + at * 8);
      dst[0] = make_uint4(p2t_canonical(v[0]), p2t_canonical(v[1]), p2t_canonical(v[2]),
                          p2t_canonical(v[3]));
      dst[1] = make_uint4(p2t_canonical(v[4]), p2t_canonical(v[5]), p2t_canonical(v[6]),
                          p2t_canonical(v[7]));
    }
    tile += step;
  }
  p2t_end<24>(sm, t, report);
}

__global__ void __launch_bounds__(p2t_threads<16>, 1)
    compress_level_tensor_kernel(const uint32_t *__restrict__ src, uint32_t *__restrict__ dst,
                                 size_t half, const Tri tri, const WaitReport report) {
  extern __shared__ __align__(128) unsigned char sm[];
  P2Tile<16> t = p2t_begin<16>(sm, g_tab16, report);
  pdl_wait();
  const size_t tiles = (half + 127) / 128, step = (size_t)gridDim.x * P2Mat<16>::TILES;
  const int lane_row = threadIdx.x & 127;
  size_t tile = (size_t)(threadIdx.x >> 7) * gridDim.x + blockIdx.x;
  uint4 a0, a1, b0, b1;
  auto fetch = [&](size_t tl) {
    size_t i = tl * 128 + lane_row;
    if (i >= half) i = half - 1;
    const uint4 *a = reinterpret_cast<const uint4 *>(src + i * 8);
    const uint4 *b = reinterpret_cast<const uint4 *>(src + (i + half) * 8);
    a0 = __ldg(a); a1 = __ldg(a + 1); b0 = __ldg(b); b1 = __ldg(b + 1);
  };
  if (tile < tiles) fetch(tile);
  while (tile < tiles) {
    const size_t at = tile * 128 + lane_row;
    {
      const uint32_t l[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      t.put_words(0, l);
      const uint32_t r[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
      t.put_words(8, r);
    }
    t.permute(tri.v, [&] {
      if (tile + step < tiles) fetch(tile + step);
    });
    int32_t v[8];
    t.get_words(0, v);
    if (at < half) {
      uint4 *d = reinterpret_cast<uint4 *>(dst + at * 8);
      d[0] = make_uint4(p2t_canonical(v[0]), p2t_canonical(v[1]), p2t_canonical(v[2]),
                        p2t_canonical(v[3]));
      d[1] = make_uint4(p2t_canonical(v[4]), p2t_canonical(v[5]), p2t_canonical(v[6]),
                        p2t_canonical(v[7]));
    }
    tile += step;
  }
  p2t_end<16>(sm, t, report);
}

Tri tri_of(int width) {
  Tri t;
  for (int i = 0; i < 4; i++) t.v[i] = p2_tables(width).tri[i];
  return t;
}
unsigned grid_of(size_t n) {
  const size_t tiles = (n + 127) / 128;
  return (unsigned)(tiles < (size_t)SMS ? tiles : SMS);
}
}  // namespace

cudaError_t init_poseidon2_tensor() {
  cudaError_t e = cudaMemcpyToSymbol(g_tab16, p2_tables(16).halves.data(), P2Mat<16>::bytes);
  if (e == cudaSuccess)
    e = cudaMemcpyToSymbol(g_tab24, p2_tables(24).halves.data(), P2Mat<24>::bytes);
  const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
  if (e == cudaSuccess) e = cudaFuncSetAttribute(hash_rows_tensor_kernel<true>, a, p2t_smem<24>());
  if (e == cudaSuccess) e = cudaFuncSetAttribute(hash_rows_tensor_kernel<false>, a, p2t_smem<24>());
  if (e == cudaSuccess) e = cudaFuncSetAttribute(compress_level_tensor_kernel, a, p2t_smem<16>());
  return e;
}

void hash_rows_tensor(const uint32_t *rows, size_t n_rows, int row_len, uint32_t *digests,
                      cudaStream_t st, const WaitReport &report) {
  const bool vec = row_len % 4 == 0 && ((uintptr_t)rows & 15) == 0;
  static const Tri tri = tri_of(24);
  if (vec)
    launch(hash_rows_tensor_kernel<true>, grid_of(n_rows), p2t_threads<24>, p2t_smem<24>(), st, rows,
           n_rows, row_len, digests, tri, report);
  else
    launch(hash_rows_tensor_kernel<false>, grid_of(n_rows), p2t_threads<24>, p2t_smem<24>(), st, rows,
           n_rows, row_len, digests, tri, report);
}

void compress_level_tensor(const uint32_t *src, uint32_t *dst, size_t half, cudaStream_t st,
                           const WaitReport &report) {
  static const Tri tri = tri_of(16);
  launch(compress_level_tensor_kernel, grid_of(half), p2t_threads<16>, p2t_smem<16>(), st, src, dst,
         half, tri, report);
}

}  // namespace gpu
}  // namespace whir
