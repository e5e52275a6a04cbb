// Poseidon2 permutations spread over lanes, for the few rows or nodes whose
// permutations follow one another (small trees, the top of every tree), where
// a launch lasts as long as one permutation's dependency chain and not as its
// instructions: P2Warp on a whole warp, one state word per lane (2.0 us per
// width-16 permutation), and P2Quad on four lanes, for more of them at once.
//
// In an internal round every lane computes word 0's S-box, so nothing waits
// for a broadcast, and the lane sum is kept off its chain: with T the sum of
// words 1.. and y the S-box output, word 0 becomes T - y, and the next T is
// (W - 1)(T + y) + V, where V is the sum of d_i s_i, which needs the round
// before only.  The internal rounds are unrolled: their constants are then
// immediate operands, not loads on the chain (512 rows of 64 words, rolled
// against unrolled: warps 14.0 and 10.0 us, quads 20.0 and 17.6).
#pragma once
#include "p2_device.cuh"

namespace whir {
namespace gpu {

// x < 2^38 with x >> 31 below 128: 2^31 = 2^24 - 1 folds it below 2p, then
// one correction
__device__ __forceinline__ uint32_t fold_canonical(uint64_t x) {
  const uint32_t f = (uint32_t)(x & 0x7fffffffu) + (uint32_t)(x >> 31) * 0x00ffffffu;
  return kb::umin(f, f - kb::P);
}

// x d mod p of any word for a plain d < p, ds = floor(d 2^32 / p)
__device__ __forceinline__ uint32_t times_plain(uint32_t x, uint32_t d, uint32_t ds) {
  const uint32_t r = x * d - __umulhi(x, ds) * kb::P;
  return kb::umin(r, r - kb::P);
}

// word 0 and T through one internal round: zc is word 0 plus its constant,
// signed; next: the next round's constant minus p; V = lo + 2^16 hi
template <int W>
struct P2Internal {
  uint32_t T;   // sum of words 1.., canonical
  int32_t zc;
  uint32_t su;  // T + y, canonical: what every other word adds
  __device__ __forceinline__ void round(uint32_t next, uint64_t lo, uint32_t hi) {
    using namespace kb;
    uint32_t tr = T + next;
    tr = kb::umin(tr, tr + P);
    const uint32_t y = sbox(zc);
    zc = (int32_t)(tr - y);  // in (-p, p): as the S-box takes it
    const uint32_t s = T + y;
    su = kb::umin(s, s - P);
    T = fold_canonical((uint64_t)s * (W - 1) + lo + (uint64_t)hi * 65536u);
  }
  // word 0, canonical, after a round whose `next` was c
  __device__ __forceinline__ uint32_t word0(uint32_t c) const {
    const uint32_t u = (uint32_t)zc;
    return kb::sub(kb::umin(u, u + kb::P), c + kb::P);
  }
};

// An external round is one S-box per lane and the light MDS by shuffles (the
// other groups' words of the lane's column, then the lane's group); V is two
// hardware reductions of 16-bit halves.
template <int W>
struct P2Warp {
  static constexpr unsigned ALL = 0xffffffffu;
  static constexpr int RP = P2Shape<W>::RP;
  uint32_t rc[8];   // this lane's external constants, stored minus p
  uint32_t d, ds;   // plain diagonal entry and floor(d 2^32 / p); 0 off words 1..W-1
  int lane;

  // table: the 8 W external constants, RP internal ones and W diagonal
  // entries of p2_device.cuh in global memory (lanes read different entries)
  __device__ __forceinline__ void init(const uint32_t *__restrict__ table) {
    lane = threadIdx.x & 31;
    const int w = lane < W ? lane : 0;
#pragma unroll
    for (int r = 0; r < 8; r++) rc[r] = __ldg(table + r * W + w);
    d = lane > 0 && lane < W ? kb::to_canonical(__ldg(table + 8 * W + RP + w)) : 0;
    ds = (uint32_t)(((uint64_t)d << 32) / kb::P);
  }
  // canonical in and out; lanes >= W carry no word
  __device__ __forceinline__ uint32_t light(uint32_t x) const {
    uint64_t u = (uint64_t)x + x;
    if constexpr (W == 16) {
      u += __shfl_xor_sync(ALL, x, 4);
      u += __shfl_xor_sync(ALL, x, 8);
      u += __shfl_xor_sync(ALL, x, 12);
    } else {
#pragma unroll
      for (int q = 1; q < W / 4; q++) {
        const int l = lane + 4 * q;
        u += __shfl_sync(ALL, x, l < W ? l : l - W);
      }
    }
    const uint32_t v = (uint32_t)(u & 0x7fffffffu) + (uint32_t)(u >> 31) * 0x00ffffffu;
    const int b = lane & ~3;
    const uint32_t a1 = __shfl_sync(ALL, v, b | ((lane + 1) & 3));
    const uint32_t a2 = __shfl_sync(ALL, v, b | ((lane + 2) & 3));
    const uint32_t a3 = __shfl_sync(ALL, v, b | ((lane + 3) & 3));
    return fold_canonical(2 * (uint64_t)v + 3 * (uint64_t)a1 + a2 + a3);
  }
  // lane i < W holds word i, canonical in and out
  __device__ __forceinline__ uint32_t permute(uint32_t x) const {
    using namespace kb;
    const uint32_t *I = p2_consts<W>() + 8 * W;  // internal constants, minus p
    x = light(x);
#pragma unroll 1
    for (int h = 0; h < 2; h++) {
#pragma unroll
      for (int r = 0; r < 4; r++) x = light(sbox((int32_t)(x + (h ? rc[4 + r] : rc[r]))));
      if (h) break;
      const uint32_t s = lane > 0 && lane < W ? x : 0;
      P2Internal<W> in;
      in.T = fold_canonical((uint64_t)__reduce_add_sync(ALL, s >> 16) * 65536u +
                            __reduce_add_sync(ALL, s & 0xffffu));
      in.zc = (int32_t)(__shfl_sync(ALL, x, 0) + I[0]);
      uint32_t m = times_plain(x, d, ds);
#pragma unroll
      for (int r = 0; r < RP; r++) {
        const uint32_t vl = __reduce_add_sync(ALL, m & 0xffffu);
        const uint32_t vh = __reduce_add_sync(ALL, m >> 16);
        in.round(I[r + 1 < RP ? r + 1 : RP - 1], vl, vh);
        x = in.su + m;  // below 2p; times_plain takes any word
        m = times_plain(x, d, ds);
      }
      x = lane ? kb::umin(x, x - P) : in.word0(I[RP - 1]);
    }
    return x;
  }
};

// Four lanes of a warp per permutation: lane l of an aligned group holds words
// l, l + 4, ..: the column sums of the light MDS are its own, and the 4 x 4
// blocks take three shuffles per word.  Every lane of the warp calls permute.
template <int W>
struct P2Quad {
  static constexpr unsigned ALL = 0xffffffffu;
  static constexpr int RP = P2Shape<W>::RP, N = W / 4;
  static constexpr int CONSTS = 8 * W;  // external constants read from shared memory
  uint32_t d[N], ds[N];
  const uint32_t *kc;  // the external constants (minus p), shared memory
  int l;

  __device__ __forceinline__ void init(const uint32_t *__restrict__ table, const uint32_t *sh) {
    l = threadIdx.x & 3;
    kc = sh + l;
#pragma unroll
    for (int j = 0; j < N; j++) {
      d[j] = j + l ? kb::to_canonical(__ldg(table + 8 * W + RP + 4 * j + l)) : 0;
      ds[j] = (uint32_t)(((uint64_t)d[j] << 32) / kb::P);
    }
  }
  __device__ __forceinline__ uint32_t rot(uint32_t v, int k) const {  // lane l + k's
    return __shfl_sync(ALL, v, (l + k) & 3, 4);
  }
  __device__ __forceinline__ void light(uint32_t (&x)[N]) const {
    uint64_t c = x[0];
#pragma unroll
    for (int j = 1; j < N; j++) c += x[j];
    const uint32_t col = fold_canonical(c);
#pragma unroll
    for (int j = 0; j < N; j++) {
      const uint32_t v = x[j] + col;  // below 2p
      const uint32_t a1 = rot(v, 1), a2 = rot(v, 2), a3 = rot(v, 3);
      x[j] = fold_canonical(2 * (uint64_t)v + 3 * (uint64_t)a1 + a2 + a3);
    }
  }
  // canonical words in and out
  __device__ __forceinline__ void permute(uint32_t (&x)[N]) const {
    using namespace kb;
    const uint32_t *I = p2_consts<W>() + 8 * W;
    light(x);
#pragma unroll 1
    for (int r = 0; r < 8; r++) {
      if (r == 4) {
        uint64_t s = l ? x[0] : 0u;
#pragma unroll
        for (int j = 1; j < N; j++) s += x[j];
        uint32_t t = fold_canonical(s);
        P2Internal<W> in;
        in.T = fold_canonical((uint64_t)t + rot(t, 1) + rot(t, 2) + rot(t, 3));
        in.zc = (int32_t)(__shfl_sync(ALL, x[0], 0, 4) + I[0]);
        uint32_t m[N];
#pragma unroll
        for (int j = 0; j < N; j++) m[j] = times_plain(x[j], d[j], ds[j]);
#pragma unroll
        for (int q = 0; q < RP; q++) {
          uint64_t v = m[0];
#pragma unroll
          for (int j = 1; j < N; j++) v += m[j];
          t = fold_canonical(v);
          in.round(I[q + 1 < RP ? q + 1 : RP - 1],
                   (uint64_t)t + rot(t, 1) + rot(t, 2) + rot(t, 3), 0);
#pragma unroll
          for (int j = 0; j < N; j++) {
            x[j] = in.su + m[j];
            m[j] = times_plain(x[j], d[j], ds[j]);
          }
        }
#pragma unroll
        for (int j = 0; j < N; j++) x[j] = kb::umin(x[j], x[j] - P);
        if (l == 0) x[0] = in.word0(I[RP - 1]);
      }
#pragma unroll
      for (int j = 0; j < N; j++) x[j] = sbox((int32_t)(x[j] + kc[r * W + 4 * j]));
      light(x);
    }
  }
};

}  // namespace gpu
}  // namespace whir
