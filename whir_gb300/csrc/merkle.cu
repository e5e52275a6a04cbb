// Merkle commitment kernels: leaf hashing (width-24 sponge), tree ascent
// (width-16 truncated-permutation compression, halves pairing) and the
// opening gather.  Tree shape and hashing follow
// crates/merkle/src/poseidon_packed.rs:98-143,269-304,344-384 and
// crates/merkle/src/poseidon.rs:33-74.
#include <algorithm>
#include <atomic>

#include "kernels.h"
#include "launch.cuh"
#include "merkle_tensor.h"
#include "p2_device.cuh"
#include "p2_lanes.cuh"
#include "poseidon2_host.h"
#include "tree_plan.h"

namespace whir {
namespace gpu {

// the same tables as c_p2_16 and c_p2_24, for lanes that read different entries
__device__ uint32_t g_p2_16[8 * 16 + 20 + 16];
__device__ uint32_t g_p2_24[8 * 24 + 23 + 24];

static cudaError_t upload_p2(int width) {
  const Poseidon2Constants &c = poseidon2_constants(width);
  uint32_t buf[8 * 24 + 23 + 24];
  int n = 0;
  // round constants minus p, for the signed S-box (p2_device.cuh)
  for (int r = 0; r < 8; r++)
    for (int i = 0; i < width; i++) buf[n++] = c.ext_rc[r][i] - kb::P;
  for (int r = 0; r < c.rounds_p; r++) buf[n++] = c.int_rc[r] - kb::P;
  for (int i = 0; i < width; i++) buf[n++] = c.diag[i];
  cudaError_t e = width == 16 ? cudaMemcpyToSymbol(c_p2_16, buf, n * 4)
                              : cudaMemcpyToSymbol(c_p2_24, buf, n * 4);
  if (e == cudaSuccess)
    e = width == 16 ? cudaMemcpyToSymbol(g_p2_16, buf, n * 4)
                    : cudaMemcpyToSymbol(g_p2_24, buf, n * 4);
  return e;
}

static std::atomic<unsigned long long> g_launches{0};
unsigned long long launch_count() { return g_launches.load(); }
void count_launches(unsigned n) { g_launches.fetch_add(n, std::memory_order_relaxed); }

cudaError_t init_poseidon2_tables() {
  cudaError_t e = upload_p2(16);
  if (e == cudaSuccess) e = upload_p2(24);
  if (e == cudaSuccess) e = init_poseidon2_tensor();
  return e;
}

// Where the tensor-core kernels (merkle_tensor.cu) take over: at the break-even
// of launches alone.  Their tiles are 128 rows and 608 of them (760 of nodes)
// fill the GPU; a tile takes 9.2 us per width-24 permutation alone on its SM and
// 16.5 us among four, so launches of few tiles per SM gain nothing over one
// thread per row.  Measured, tensor against thread, us: 16-word rows 2^15
// 17.2/14.7, 2^16 22.5/25.7, 2^17 36.4/40.7, 2^18 66.4/76.0; 32-word rows 2^15
// 29.1/26.9, 2^16 38.8/48.8; 64-word rows 2^15 51.7/51.0, 2^16 70.7/94.6, 2^17
// 123/158, 2^19 442/578; nodes 2^16 17.1/17.3, 2^17 27.9/27.2, 2^18 45.6/50.0.
// (32 jobs of 2^14..2^20 evaluations on 8 streams: with either line a factor of
// two off the same within their spread of 3%.)
static bool leaves_on_tensor(size_t n_rows) { return n_rows >= (size_t)1 << 16; }
static bool nodes_on_tensor(size_t nodes) { return nodes >= (size_t)1 << 18; }
// Lanes per row of small launches (0: one thread).  A thread takes a
// permutation's latency of 8.5 us per chunk however few the rows are, a quad
// of lanes 4.2 us, a warp 2.1 us; the instructions grow the other way.  us,
// warp / quad / thread: 16-word rows 2^9 3.8/5.7/9.1, 2^11 6.1/5.7/9.1, 2^12
// 9.0/5.8/9.1, 2^13 16/7.2/9.2, 2^14 29/11.9/9.2; 64-word rows 2^9
// 10/16.7/32, 2^11 19/16.8/32, 2^12 31/16.8/33, 2^13 56/23/33, 2^14 106/41/33.
static int leaf_lanes(size_t n_rows) {
  return n_rows <= ((size_t)1 << 10) ? 32 : n_rows <= ((size_t)1 << 13) ? 4 : 0;
}
// Lanes per opened path (0: one thread): 13 to 18 permutations follow one
// another.  us, warp / quad / thread, paths of 16 words and 14 levels mixed
// with some of 64 and 12: 128 paths 34/51/111, 1024 40/52/101, 2048 62/52/102,
// 8192 184/68/102.  Quads take CTAs of 32 paths, and their time steps with the
// CTAs per SM (paths of a proof of 2^16 evaluations, quad / thread): two 73/114,
// three, up to 14592 paths, 98/114, four 122/114.
static int path_lanes(int n) { return n <= 1024 ? 32 : n <= SMS * 3 * 32 ? 4 : 0; }

// One row per thread; a row of ROW = 16·c words is c permutations
// (PaddingFreeSponge: overwrite the 16 rate lanes, permute).  Base rows are
// 2^f words and extension rows 4·2^f, so foldings 4..6 use 16..256.
// The bound of six CTAs lets a permutation use 64 registers: left at 40 (32 in
// compress_level), its S-boxes and additions follow one another, which a full
// SM hides but few rows do not (2^14 rows of 64 words 41.2 -> 32.7 us, 2^15
// 58.5 -> 50.1, 2^16 106 -> 94, 2^17 157.2 -> 156.5; 2^15 nodes 10.3 -> 9.3).
template <int ROW>
__global__ void __launch_bounds__(128, 6) hash_rows_fixed(const uint32_t *__restrict__ rows,
                                                       size_t n_rows,
                                                       uint32_t *__restrict__ digests) {
  pdl_wait();
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_rows) return;
  const uint4 *src = reinterpret_cast<const uint4 *>(rows + i * ROW);
  uint32_t s[24];
#pragma unroll
  for (int j = 16; j < 24; j++) s[j] = 0;
#pragma unroll 1
  for (int chunk = 0; chunk < ROW / 16; chunk++) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      uint4 v = __ldg(src + chunk * 4 + q);
      s[4 * q] = v.x;
      s[4 * q + 1] = v.y;
      s[4 * q + 2] = v.z;
      s[4 * q + 3] = v.w;
    }
    p2_permute<24>(s);
  }
  uint4 *dst = reinterpret_cast<uint4 *>(digests + i * 8);
  dst[0] = make_uint4(s[0], s[1], s[2], s[3]);
  dst[1] = make_uint4(s[4], s[5], s[6], s[7]);
}

// One row per warp (p2_lanes.cuh), any row length and alignment: a lane loads
// its word of the next chunk before this chunk's permutation.
__global__ void __launch_bounds__(128, 6) hash_rows_warp(const uint32_t *__restrict__ rows,
                                                      size_t n_rows, int row_len,
                                                      uint32_t *__restrict__ digests) {
  P2Warp<24> p;
  p.init(g_p2_24);
  pdl_wait();
  const size_t i = (size_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  if (i >= n_rows) return;
  const uint32_t *row = rows + i * row_len;
  const int l = p.lane;
  uint32_t x = 0;
  uint32_t next = l < 16 && l < row_len ? __ldg(row + l) : 0;
  for (int pos = 0; pos < row_len; pos += 16) {
    if (l < 16 && pos + l < row_len) x = next;
    if (l < 16 && pos + 16 + l < row_len) next = __ldg(row + pos + 16 + l);
    x = p.permute(x);
  }
  if (l < 8) digests[i * 8 + l] = x;
}

// One row per four lanes, any row length and alignment.
__global__ void __launch_bounds__(128, 6) hash_rows_quad(const uint32_t *__restrict__ rows,
                                                      size_t n_rows, int row_len,
                                                      uint32_t *__restrict__ digests) {
  __shared__ uint32_t kc[P2Quad<24>::CONSTS];
  for (int i = threadIdx.x; i < P2Quad<24>::CONSTS; i += blockDim.x) kc[i] = __ldg(g_p2_24 + i);
  P2Quad<24> p;
  p.init(g_p2_24, kc);
  __syncthreads();
  pdl_wait();
  const size_t i = (size_t)blockIdx.x * (blockDim.x / 4) + (threadIdx.x >> 2);
  const bool live = i < n_rows;  // a whole warp permutes together
  const uint32_t *row = rows + (live ? i : 0) * row_len + p.l;
  uint32_t x[6] = {0, 0, 0, 0, 0, 0}, next[4] = {0, 0, 0, 0};
#pragma unroll
  for (int j = 0; j < 4; j++)
    if (4 * j + p.l < row_len) next[j] = __ldg(row + 4 * j);
  for (int pos = 0; pos < row_len; pos += 16) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
      if (pos + 4 * j + p.l < row_len) x[j] = next[j];
      if (pos + 16 + 4 * j + p.l < row_len) next[j] = __ldg(row + pos + 16 + 4 * j);
    }
    p.permute(x);
  }
  if (live) {
    digests[i * 8 + p.l] = x[0];
    digests[i * 8 + 4 + p.l] = x[1];
  }
}

// Any row length (small foldings): the trailing partial chunk overwrites only
// its lanes and is permuted; an empty trailing chunk is not.
__global__ void __launch_bounds__(128, 6) hash_rows_generic(const uint32_t *__restrict__ rows, size_t n_rows, int row_len,
                                  uint32_t *__restrict__ digests) {
  pdl_wait();
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_rows) return;
  const uint32_t *src = rows + i * row_len;
  uint32_t s[24];
#pragma unroll
  for (int j = 0; j < 24; j++) s[j] = 0;
  int pos = 0;
  while (pos < row_len) {
    int take = row_len - pos < 16 ? row_len - pos : 16;
    for (int j = 0; j < take; j++) s[j] = src[pos + j];
    pos += take;
    p2_permute<24>(s);
  }
  for (int j = 0; j < 8; j++) digests[i * 8 + j] = s[j];
}

// One opening per thread: the leaf sponge over the row (16 rate words per
// permutation, a shorter last chunk overwriting only its words), then one
// width-16 compression per level with the sibling on the side the index's
// bit names (halves pairing: at a level of 2m nodes, index i >= m is the
// right child).
__global__ void __launch_bounds__(128, 6) verify_paths_kernel(const PathDesc *__restrict__ d,
                                                           const uint32_t *__restrict__ words,
                                                           const uint32_t *__restrict__ roots,
                                                           int n, uint8_t *__restrict__ ok) {
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const PathDesc pd = d[i];
  const uint32_t *w = words + pd.off;
  uint32_t s[24];
#pragma unroll
  for (int j = 0; j < 24; j++) s[j] = 0;
  for (int pos = 0; pos < pd.row_len; pos += 16) {
    const int take = pd.row_len - pos < 16 ? pd.row_len - pos : 16;
#pragma unroll
    for (int j = 0; j < 16; j++)
      if (j < take) s[j] = w[pos + j];
    p2_permute<24>(s);
  }
  uint32_t acc[8];
#pragma unroll
  for (int j = 0; j < 8; j++) acc[j] = s[j];
  const uint32_t *sib = w + pd.row_len;
  uint64_t idx = pd.index;
  for (int l = 0; l < pd.log_h; l++) {
    const uint64_t mid = 1ull << (pd.log_h - l - 1);
    const bool right = idx >= mid;
    uint32_t t[16];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const uint32_t a = acc[j], b = sib[8 * l + j];
      t[j] = right ? b : a;
      t[8 + j] = right ? a : b;
    }
    p2_permute<16>(t);
#pragma unroll
    for (int j = 0; j < 8; j++) acc[j] = t[j];
    idx &= mid - 1;
  }
  const uint32_t *root = roots + 8 * (size_t)i;
  bool good = true;
#pragma unroll
  for (int j = 0; j < 8; j++) good &= acc[j] == root[j];
  ok[i] = good ? 1 : 0;
}

// One opening per warp (LANES = 32, a state word per lane) or per four lanes
// (word l + 4j in lane l's j-th register): the sponge and the path one after
// the other wait for permutations only.  A warp's quads run as many
// permutations as its longest opening; the surplus is dropped.
__global__ void __launch_bounds__(128, 6) verify_paths_warp(const PathDesc *__restrict__ d,
                                                         const uint32_t *__restrict__ words,
                                                         const uint32_t *__restrict__ roots, int n,
                                                         uint8_t *__restrict__ ok) {
  P2Warp<24> leaf;
  leaf.init(g_p2_24);
  P2Warp<16> node;
  node.init(g_p2_16);
  pdl_wait();
  const int i = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  if (i >= n) return;
  const PathDesc pd = d[i];
  const uint32_t *w = words + pd.off, *sib = w + pd.row_len;
  const int lane = leaf.lane;
  uint32_t x = 0;
  for (int pos = 0; pos < pd.row_len; pos += 16) {
    if (lane < 16 && pos + lane < pd.row_len) x = w[pos + lane];
    x = leaf.permute(x);
  }
  uint64_t idx = pd.index;
  for (int l = 0; l < pd.log_h; l++) {
    const uint64_t mid = 1ull << (pd.log_h - l - 1);
    const uint32_t s = lane < 16 ? sib[8 * l + (lane & 7)] : 0;
    const uint32_t acc = __shfl_sync(0xffffffffu, x, lane & 7);
    // lanes 0..7 hold the left child: the node itself or, for a right one,
    // its sibling
    x = lane < 16 ? ((lane < 8) == (idx < mid) ? acc : s) : 0;
    x = node.permute(x);
    idx &= mid - 1;
  }
  const bool same = lane >= 8 || x == roots[8 * (size_t)i + lane];
  const bool good = __all_sync(0xffffffffu, same);
  if (lane == 0) ok[i] = good ? 1 : 0;
}

__global__ void __launch_bounds__(128, 6) verify_paths_quad(const PathDesc *__restrict__ d,
                                                         const uint32_t *__restrict__ words,
                                                         const uint32_t *__restrict__ roots, int n,
                                                         uint8_t *__restrict__ ok) {
  __shared__ uint32_t kc24[P2Quad<24>::CONSTS], kc16[P2Quad<16>::CONSTS];
  for (int i = threadIdx.x; i < P2Quad<24>::CONSTS; i += blockDim.x) kc24[i] = __ldg(g_p2_24 + i);
  for (int i = threadIdx.x; i < P2Quad<16>::CONSTS; i += blockDim.x) kc16[i] = __ldg(g_p2_16 + i);
  P2Quad<24> leaf;
  leaf.init(g_p2_24, kc24);
  P2Quad<16> node;
  node.init(g_p2_16, kc16);
  __syncthreads();
  pdl_wait();
  const int i = blockIdx.x * (blockDim.x / 4) + (threadIdx.x >> 2), lane = leaf.l;
  const bool live = i < n;  // a whole warp permutes together
  PathDesc pd = {};
  if (live) pd = d[i];
  const uint32_t *w = words + pd.off, *sib = w + pd.row_len;
  uint32_t x[6] = {0, 0, 0, 0, 0, 0};
  const int row_max = (int)__reduce_max_sync(0xffffffffu, (unsigned)pd.row_len);
  for (int pos = 0; pos < row_max; pos += 16) {
    uint32_t y[6];
#pragma unroll
    for (int j = 0; j < 6; j++) {
      y[j] = x[j];
      if (j < 4 && pos + 4 * j + lane < pd.row_len) y[j] = w[pos + 4 * j + lane];
    }
    leaf.permute(y);
#pragma unroll
    for (int j = 0; j < 6; j++)
      if (pos < pd.row_len) x[j] = y[j];
  }
  uint32_t a0 = x[0], a1 = x[1];
  uint64_t idx = pd.index;
  const int height = (int)__reduce_max_sync(0xffffffffu, (unsigned)pd.log_h);
  for (int l = 0; l < height; l++) {
    const bool on = l < pd.log_h;
    const uint64_t mid = on ? 1ull << (pd.log_h - l - 1) : 1;
    const bool right = idx >= mid;
    uint32_t s0 = 0, s1 = 0;
    if (on) {
      s0 = sib[8 * l + lane];
      s1 = sib[8 * l + 4 + lane];
    }
    uint32_t t[4] = {right ? s0 : a0, right ? s1 : a1, right ? a0 : s0, right ? a1 : s1};
    node.permute(t);
    if (on) {
      a0 = t[0];
      a1 = t[1];
      idx &= mid - 1;
    }
  }
  bool same = true;
  if (live) same = a0 == roots[8 * (size_t)i + lane] && a1 == roots[8 * (size_t)i + 4 + lane];
  const unsigned votes = __ballot_sync(0xffffffffu, same);
  if (live && lane == 0) ok[i] = (votes >> (threadIdx.x & 28) & 15u) == 15u ? 1 : 0;
}

cudaError_t verify_paths(const PathDesc *d, const uint32_t *words, const uint32_t *roots, int n,
                         uint8_t *ok, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const int T = 128;
  const int lanes = path_lanes(n);
  const unsigned per = lanes ? T / lanes : T;
  launch(lanes == 32 ? verify_paths_warp : lanes == 4 ? verify_paths_quad : verify_paths_kernel,
         ((unsigned)n + per - 1) / per, T, 0, st, d, words, roots, n, ok);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t hash_rows(const uint32_t *rows, size_t n_rows, int row_len, uint32_t *digests,
                      cudaStream_t st, const WaitReport &report) {
  if (n_rows == 0) return cudaSuccess;
  if (leaves_on_tensor(n_rows) && ((uintptr_t)digests & 15) == 0) {
    hash_rows_tensor(rows, n_rows, row_len, digests, st, report);
    count_launches(1);
    return cudaGetLastError();
  }
  const int T = 128;
  if (const int lanes = leaf_lanes(n_rows)) {
    const size_t per = T / lanes;  // rows per CTA
    const unsigned g = (unsigned)((n_rows + per - 1) / per);
    if (lanes == 32) launch(hash_rows_warp, g, T, 0, st, rows, n_rows, row_len, digests);
    else launch(hash_rows_quad, g, T, 0, st, rows, n_rows, row_len, digests);
    count_launches(1);
    return cudaGetLastError();
  }
  unsigned grid = (unsigned)((n_rows + T - 1) / T);
  // the fixed-width kernels use 16-byte vector loads and stores
  bool aligned = (((uintptr_t)rows | (uintptr_t)digests) & 15) == 0;
  switch (aligned ? row_len : 0) {
    case 16: launch(hash_rows_fixed<16>, grid, T, 0, st, rows, n_rows, digests); break;
    case 32: launch(hash_rows_fixed<32>, grid, T, 0, st, rows, n_rows, digests); break;
    case 64: launch(hash_rows_fixed<64>, grid, T, 0, st, rows, n_rows, digests); break;
    case 128: launch(hash_rows_fixed<128>, grid, T, 0, st, rows, n_rows, digests); break;
    case 256: launch(hash_rows_fixed<256>, grid, T, 0, st, rows, n_rows, digests); break;
    default: launch(hash_rows_generic, grid, T, 0, st, rows, n_rows, row_len, digests);
  }
  count_launches(1);
  return cudaGetLastError();
}

__global__ void __launch_bounds__(128, 6) compress_level(const uint32_t *__restrict__ src,
                                                      uint32_t *__restrict__ dst, size_t half) {
  pdl_wait();
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= half) return;
  const uint4 *a = reinterpret_cast<const uint4 *>(src + i * 8);
  const uint4 *b = reinterpret_cast<const uint4 *>(src + (i + half) * 8);
  uint4 a0 = __ldg(a), a1 = __ldg(a + 1), b0 = __ldg(b), b1 = __ldg(b + 1);
  uint32_t s[16] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w,
                    b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
  p2_permute<16>(s);
  uint4 *d = reinterpret_cast<uint4 *>(dst + i * 8);
  d[0] = make_uint4(s[0], s[1], s[2], s[3]);
  d[1] = make_uint4(s[4], s[5], s[6], s[7]);
}

// one level of a tree: `half` nodes from the 2 half nodes at src
static void launch_level(const uint32_t *src, uint32_t *dst, size_t half, cudaStream_t st,
                         const WaitReport &report) {
  if (nodes_on_tensor(half)) {
    compress_level_tensor(src, dst, half, st, report);
  } else {
    const int T = 128;
    launch(compress_level, (unsigned)((half + T - 1) / T), T, 0, st, src, dst, half);
  }
  count_launches(1);
}

// ---- the narrow levels of a tree ----
// With halves pairing, node i of a level with H nodes is C(i, i + H/2) of the
// level below, and i, i + H/2 agree modulo any G dividing H/2.  So the nodes
// congruent to j mod G form an independent subtree down to the level with G
// nodes: CTA j keeps its share of a level in shared memory and climbs
// log2(H/G) levels with one barrier per level, writing every level it makes
// to the tree in global memory (the openings read them).  A narrow level is
// bound by the latency of one permutation, so this replaces one launch per
// level by one to three launches per tree (G CTAs up to the level of G nodes,
// the last with G = 1 to the root).  A level of more than warp_nodes nodes per
// CTA is compressed by a quad of lanes per node, a smaller one by a warp per
// node (p2_lanes.cuh).
// A batched tree (kernels.h: batch instances' leaves interleaved) is the
// same ascent over batch 2^log_h leaves: level l holds batch 2^(log_h - l)
// nodes at batch * level_offset_words(log_h, l), and G is a multiple of
// batch, so every subtree lies inside one instance.
__global__ void __launch_bounds__(1024) tree_subtrees(uint32_t *__restrict__ nodes, int log_h,
                                                     int l0, int steps, uint32_t *host_root,
                                                     unsigned int *flag, unsigned int seq,
                                                     unsigned batch, int warp_nodes) {
  extern __shared__ uint4 sm[];  // 2 uint4 per node of this CTA's share
  __shared__ uint32_t kc[P2Quad<16>::CONSTS];
  for (int i = threadIdx.x; i < P2Quad<16>::CONSTS; i += blockDim.x) kc[i] = __ldg(g_p2_16 + i);
  P2Quad<16> pq;
  pq.init(g_p2_16, kc);
  const int l = pq.l, m = threadIdx.x >> 2;
  P2Warp<16> pw;
  pw.init(g_p2_16);
  pdl_wait();
  const size_t G = gridDim.x, j = blockIdx.x;
  int n = (int)(((size_t)batch << (log_h - l0)) / G);
  const uint4 *src = reinterpret_cast<const uint4 *>(nodes + batch * level_offset_words(log_h, l0));
  for (int q = threadIdx.x; q < 2 * n; q += blockDim.x) sm[q] = src[(j + G * (q >> 1)) * 2 + (q & 1)];
  __syncthreads();
  uint32_t *smw = reinterpret_cast<uint32_t *>(sm);
  for (int st = 0; st < steps; st++) {
    const int half = n >> 1;
    uint32_t *level = nodes + batch * level_offset_words(log_h, l0 + st + 1);
    if (half <= warp_nodes) {  // one warp per node, one word per lane
      const int wm = threadIdx.x >> 5, lane = pw.lane;
      uint32_t y = 0;
      if (wm < half) {
        // lanes 0..7: the left child, 8..15: the right child
        y = lane < 16 ? smw[lane < 8 ? 8 * wm + lane : 8 * (wm + half) + lane - 8] : 0;
        y = pw.permute(y);
        if (lane < 8) {
          level[(j + G * wm) * 8 + lane] = y;
          if (host_root && G == 1 && half == 1) host_root[lane] = y;  // the root, also to the host
        }
      }
      __syncthreads();  // every read of this level's shared copy is done
      if (wm < half && lane < 8) smw[8 * wm + lane] = y;
      __syncthreads();
      n = half;
      continue;
    }
    const bool warp_live = ((threadIdx.x & ~31) >> 2) < half;  // warp-uniform
    const bool live = m < half;
    uint32_t x[4] = {0, 0, 0, 0};
    if (warp_live) {
      if (live) {  // words l and l + 4 of the left child, then of the right one
        x[0] = smw[8 * m + l];
        x[1] = smw[8 * m + 4 + l];
        x[2] = smw[8 * (m + half) + l];
        x[3] = smw[8 * (m + half) + 4 + l];
      }
      pq.permute(x);
      if (live) {
        level[(j + G * m) * 8 + l] = x[0];
        level[(j + G * m) * 8 + 4 + l] = x[1];
      }
    }
    __syncthreads();  // every read of this level's shared copy is done
    if (live) {
      smw[8 * m + l] = x[0];
      smw[8 * m + 4 + l] = x[1];
    }
    __syncthreads();
    n = half;
  }
  if (flag && host_root && gridDim.x == 1) {  // the root is written: raise the flag
    __threadfence_system();
    __syncthreads();
    if (threadIdx.x == 0) *reinterpret_cast<volatile unsigned int *>(flag) = seq;
  }
}

// Default: levels whose step makes at least 2^15 nodes run over the whole GPU
// (launch_level); the rest (at most 2^16 nodes at the first narrow level) go
// through tree_subtrees.  Per-size overrides in tree_tune().
static std::atomic<int> g_tree_tune[41];  // 0: default, else (wide_log << 4) | (split + 2)

TreeTune tree_tune(int log_h) {
  TreeTune t;
  if (log_h < 0 || log_h > 40) return t;
  int v = g_tree_tune[log_h].load(std::memory_order_relaxed);
  if (v) {
    t.wide_log = v >> 4;
    t.split = (v & 15) - 2;
  }
  return t;
}
bool tree_tune_valid(int log_h, TreeTune t) { return tree_tune_ok(log_h, t.wide_log, t.split); }
void set_tree_tune(int log_h, TreeTune t) {
  if (log_h < 0 || log_h > 40 || !tree_tune_valid(log_h, t)) return;
  g_tree_tune[log_h].store((t.wide_log << 4) | (t.split + 2), std::memory_order_relaxed);
}

// One launch of `ctas` subtrees: levels l0 .. l0 + steps of a tree (batch
// instances).  A level of few nodes in all waits for one permutation, which
// takes a warp 2.0 us, a quad of lanes 2.8 us; a level of many is bound by
// instructions, of which a quad needs a quarter (per SM: 8 nodes 2.3 us on
// warps and 2.8 on quads, 16 nodes 3.4 and 2.8).  So warps take levels of up
// to 8 nodes per CTA and 2048 in all.
// Threads: a quad per node made at the first step, a warp per node later.
static cudaError_t launch_subtrees(uint32_t *nodes, int log_h, int l0, int steps, size_t ctas,
                                   int batch, cudaStream_t st, uint32_t *host_root = nullptr,
                                   unsigned int *flag = nullptr, unsigned int seq = 0) {
  if (steps <= 0) return cudaSuccess;
  if (steps > 9 || ctas > 0x7fffffffu) return cudaErrorInvalidValue;
  const int n = 1 << steps;  // nodes per CTA at level l0
  int warp_nodes = 0;
  for (int h = 1; h <= 8 && h <= n / 2 && ctas * h <= 2048; h *= 2) warp_nodes = h;
  const int threads = std::max({2 * n, 32, 32 * warp_nodes});
  launch(tree_subtrees, (unsigned)ctas, threads, (size_t)n * 32, st, nodes, log_h, l0, steps,
         host_root, flag, seq, (unsigned)batch, warp_nodes);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t build_tree(uint32_t *nodes, int log_h, cudaStream_t st, const WaitReport &report,
                       uint32_t *host_root, unsigned int *flag, unsigned int seq) {
  TreeTune tune = tree_tune(log_h);
  if (!tree_tune_valid(log_h, tune)) tune = TreeTune();
  int l = 0;
  for (; l < log_h && ((size_t)1 << (log_h - l)) / 2 >= ((size_t)1 << tune.wide_log); l++) {
    size_t half = ((size_t)1 << (log_h - l)) / 2;
    launch_level(nodes + level_offset_words(log_h, l), nodes + level_offset_words(log_h, l + 1),
                 half, st, report);
  }
  // the remaining S = log_h - l steps (S <= wide_log) in up to three launches
  const int S = log_h - l, g = tree_first_split(S, tune.split);
  const int g2 = g >= 6 ? g - 4 : 0;  // 16 nodes per CTA, if the top has 64 or more
  cudaError_t e;
  if (g == 0) return launch_subtrees(nodes, log_h, l, S, 1, 1, st, host_root, flag, seq);
  e = launch_subtrees(nodes, log_h, l, S - g, (size_t)1 << g, 1, st);
  if (e == cudaSuccess && g2)
    e = launch_subtrees(nodes, log_h, log_h - g, g - g2, (size_t)1 << g2, 1, st);
  if (e != cudaSuccess) return e;
  const int top = g2 ? g2 : g;  // only the last launch (one CTA) reaches the root
  return launch_subtrees(nodes, log_h, log_h - top, top, 1, 1, st, host_root, flag, seq);
}

// ---- batched trees (kernels.h) ----
// Wide levels one thread per node, as build_tree; the remaining S levels up
// to the instances' roots in two subtree launches: batch 2^g CTAs climb
// S - g levels, then batch CTAs climb g (each CTA holds at most 512 nodes).
cudaError_t build_tree_batch(uint32_t *nodes, int log_h, int batch, cudaStream_t st,
                             const WaitReport &report) {
  if (batch < 1 || log_h < 0 || log_h > 30) return cudaErrorInvalidValue;
  const size_t B = (size_t)batch;
  int l = 0;
  for (; l < log_h && (B << (log_h - l)) / 2 >= ((size_t)1 << 15); l++) {
    size_t half = (B << (log_h - l)) / 2;
    launch_level(nodes + B * level_offset_words(log_h, l),
                 nodes + B * level_offset_words(log_h, l + 1), half, st, report);
  }
  const int S = log_h - l;
  if (S == 0) return cudaGetLastError();
  int g = S / 2;
  if (S - g > 9) g = S - 9;
  if (g > 9 || (B << g) > 0x7fffffffu) return cudaErrorInvalidValue;
  const cudaError_t e = launch_subtrees(nodes, log_h, l, S - g, B << g, batch, st);
  if (e != cudaSuccess) return e;
  return launch_subtrees(nodes, log_h, log_h - g, g, B, batch, st);
}

__global__ void gather_openings_batch_kernel(const uint32_t *__restrict__ rows, int row_len,
                                             const uint32_t *__restrict__ nodes, int log_h,
                                             unsigned batch, const uint32_t *__restrict__ idx,
                                             const int *__restrict__ inst, int n,
                                             uint32_t *__restrict__ out) {
  pdl_wait();
  const int q = blockIdx.x;
  if (q >= n) return;
  const size_t b = (size_t)inst[q], r = idx[q];
  const size_t per = (size_t)row_len + 8 * (size_t)log_h;
  uint32_t *o = out + q * per;
  const uint32_t *row = rows + (r * batch + b) * row_len;
  for (int j = threadIdx.x; j < row_len; j += blockDim.x) o[j] = row[j];
  for (int t = threadIdx.x; t < 8 * log_h; t += blockDim.x) {
    const int l = t / 8, w = t % 8;
    const size_t at = r & (((size_t)1 << (log_h - l)) - 1);  // the instance's node at level l
    const size_t sib = at ^ ((size_t)1 << (log_h - l - 1));
    o[row_len + t] = nodes[batch * level_offset_words(log_h, l) + (sib * batch + b) * 8 + w];
  }
}

cudaError_t gather_openings_batch(const uint32_t *rows, int row_len, const uint32_t *nodes,
                                  int log_h, int batch, const uint32_t *idx, const int *inst,
                                  int n, uint32_t *out, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  if (batch < 1) return cudaErrorInvalidValue;
  launch(gather_openings_batch_kernel, n, 128, 0, st, rows, row_len, nodes, log_h, (unsigned)batch,
         idx, inst, n, out);
  count_launches(1);
  return cudaGetLastError();
}

// dst row r = (src row r of instance 0, of instance 1, ...): 16-byte
// pieces when the row width allows, one thread per piece of dst
template <class T>
__global__ void interleave_kernel(const T *__restrict__ src, size_t rows, size_t w, size_t batch,
                                  T *__restrict__ dst) {
  pdl_wait();
  const size_t total = rows * w * batch;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (size_t)gridDim.x * blockDim.x) {
    const size_t j = i % w, rb = i / w, b = rb % batch, r = rb / batch;
    dst[i] = src[(b * rows + r) * w + j];
  }
}

cudaError_t interleave_rows(const uint32_t *src, size_t rows, size_t w, int batch, uint32_t *dst,
                            cudaStream_t st) {
  if (batch < 1) return cudaErrorInvalidValue;
  const size_t total = rows * w * (size_t)batch;
  if (total == 0) return cudaSuccess;
  const unsigned T = 256;
  const bool vec = w % 4 == 0 && (((uintptr_t)src | (uintptr_t)dst) & 15) == 0;
  const size_t items = vec ? total / 4 : total;
  const size_t g = (items + T - 1) / T;
  const unsigned grid = (unsigned)(g < SMS * 32 ? g : SMS * 32);
  if (vec)
    launch(interleave_kernel<uint4>, grid, T, 0, st, reinterpret_cast<const uint4 *>(src), rows,
           w / 4, (size_t)batch, reinterpret_cast<uint4 *>(dst));
  else
    launch(interleave_kernel<uint32_t>, grid, T, 0, st, src, rows, w, (size_t)batch, dst);
  count_launches(1);
  return cudaGetLastError();
}

__device__ __forceinline__ void gather_one(const uint32_t *__restrict__ rows, int row_len,
                                           const uint32_t *__restrict__ nodes, int log_h,
                                           size_t index, int q, uint32_t *__restrict__ out) {
  size_t per = (size_t)row_len + 8 * (size_t)log_h;
  uint32_t *o = out + q * per;
  for (int j = threadIdx.x; j < row_len; j += blockDim.x) o[j] = rows[index * row_len + j];
  // sibling at level l is index_l ^ mid_l with mid_l = 2^(log_h - l - 1)
  for (int t = threadIdx.x; t < 8 * log_h; t += blockDim.x) {
    int l = t / 8, w = t % 8;
    size_t mask = ((size_t)1 << (log_h - l)) - 1;  // index at level l is index & mask
    size_t mid = (size_t)1 << (log_h - l - 1);
    size_t sib = (index & mask) ^ mid;
    o[row_len + t] = nodes[level_offset_words(log_h, l) + sib * 8 + w];
  }
}

__global__ void gather_openings_kernel(const uint32_t *__restrict__ rows, int row_len,
                                       const uint32_t *__restrict__ nodes, int log_h,
                                       const uint32_t *__restrict__ idx, int n,
                                       uint32_t *__restrict__ out) {
  pdl_wait();
  int q = blockIdx.x;
  if (q >= n) return;
  gather_one(rows, row_len, nodes, log_h, idx[q], q, out);
}
// the same with the indexes passed by value
__global__ void gather_openings_val_kernel(const uint32_t *__restrict__ rows, int row_len,
                                           const uint32_t *__restrict__ nodes, int log_h,
                                           const __grid_constant__ IdxArgs a,
                                           uint32_t *__restrict__ out, Publish pub) {
  pdl_wait();
  gather_one(rows, row_len, nodes, log_h, a.idx[blockIdx.x], (int)blockIdx.x, out);
  if (!pub.flag) return;
  __threadfence_system();  // the openings reach host memory before the flag
  __syncthreads();
  if (threadIdx.x == 0 && atomicAdd(pub.counter, 1u) == gridDim.x - 1) {
    atomicExch(pub.counter, 0u);
    __threadfence_system();
    *reinterpret_cast<volatile unsigned int *>(pub.flag) = pub.seq;
  }
}

cudaError_t gather_openings_val(const uint32_t *rows, int row_len, const uint32_t *nodes,
                                int log_h, const IdxArgs &a, int n, uint32_t *out,
                                cudaStream_t st, const Publish &pub) {
  if (n == 0) return cudaSuccess;
  if (n > IdxArgs::N) return cudaErrorInvalidValue;
  launch(gather_openings_val_kernel, n, 128, 0, st, rows, row_len, nodes, log_h, a, out, pub);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t gather_openings(const uint32_t *rows, int row_len, const uint32_t *nodes, int log_h,
                            const uint32_t *idx, int n, uint32_t *out, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  launch(gather_openings_kernel, n, 128, 0, st, rows, row_len, nodes, log_h, idx, n, out);
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace gpu
}  // namespace whir
