// Poseidon2 permutation on a whole warp, one state word per lane: for the few
// rows or nodes whose permutations follow one another (small trees, the top of
// every tree), where a launch lasts as long as one permutation's dependency
// chain and not as its instructions.
//
// An external round is one S-box per lane and the light MDS by shuffles (the
// other groups' words of the lane's column, then the lane's group).  In an
// internal round every lane computes word 0's S-box, so nothing waits for a
// broadcast, and the lane sum is kept off its chain: with T the sum of words
// 1.. and y the S-box output, word 0 becomes T - y, and the next T is
// (W - 1)(T + y) + V, where V is the sum of d_i s_i, which needs the round
// before only.  V is two hardware reductions of 16-bit halves.
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
  __device__ __forceinline__ uint32_t times_d(uint32_t x) const {  // any x
    const uint32_t r = x * d - __umulhi(x, ds) * kb::P;
    return kb::umin(r, r - kb::P);
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
      uint32_t z = __shfl_sync(ALL, x, 0);
      uint32_t T = fold_canonical((uint64_t)__reduce_add_sync(ALL, s >> 16) * 65536u +
                                  __reduce_add_sync(ALL, s & 0xffffu));
      uint32_t m = times_d(x);
      int32_t zc = (int32_t)(z + I[0]);
#pragma unroll 4
      for (int r = 0; r < RP; r++) {
        const uint32_t vl = __reduce_add_sync(ALL, m & 0xffffu);
        const uint32_t vh = __reduce_add_sync(ALL, m >> 16);
        uint32_t tr = T + I[r + 1 < RP ? r + 1 : RP - 1];  // T + the next constant, mod p
        tr = kb::umin(tr, tr + P);
        const uint32_t y = sbox(zc);
        zc = (int32_t)(tr - y);  // in (-p, p): as the S-box takes it
        if (r + 1 == RP) z = sub(T, y);
        const uint32_t su = T + y, sc = kb::umin(su, su - P);
        T = fold_canonical((uint64_t)su * (W - 1) + vl + (uint64_t)vh * 65536u);
        x = sc + m;  // below 2p; times_d takes any word
        m = times_d(x);
      }
      x = kb::umin(x, x - P);
      if (lane == 0) x = z;
    }
    return x;
  }
};

}  // namespace gpu
}  // namespace whir
