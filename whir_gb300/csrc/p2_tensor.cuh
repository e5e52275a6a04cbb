// Poseidon2 with its linear layers on the tensor cores (tcgen05), 128
// permutations at a time: one permutation per thread of a four-warp tile.
//
// What bounds the permutation on the integer pipes (p2_device.cuh) is not the
// S-boxes but the linear layers around them: of about 8 100 thread
// instructions of a width-24 permutation some 2 400 are S-box products, the
// rest adds, shifts and their corrections.  Here a light layer is one small
// integer matrix product, and the 20 or 23 internal rounds become blocks of
// four or (width 24) six: word 0 before each round is a linear form of earlier
// S-box outputs, one matrix product per block gives all of them up to the
// block's own outputs, and one more gives the state after the last round
// (p2_matrix.h has the tables and the proof that every sum is exact).  A thread splits a word
// into operands with two byte permutes, and takes a light layer's word from
// its two sums with three instructions and a form's from its four with six.
//
// The operands and sums of a tile live in its 128 tensor-memory columns, lane
// = row, so a thread reads and writes only its own row and no data crosses
// threads.  A CTA runs as many tiles as an SM's 512 columns hold, four of 128
// or (width 16) five of 96, which hide one another's waits: a permutation
// waits for the matrix unit 15 times (width 16: 17), 350 to 400 cycles each.  (Five
// tiles against four, 2^18 nodes 49.5 -> 45.1 us, 2^19 87.6 -> 84.4; width 24
// needs 112 columns at least.)  The tables (95 KB at width 24, 48 KB at 16) are read
// once per CTA.
#pragma once
#include "kernels.h"
#include "launch.cuh"
#include "p2_matrix.h"

namespace whir {
namespace gpu {

template <int W>
constexpr int p2t_threads = 128 * P2Mat<W>::TILES;

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// ---- tensor memory: 8, 16 or 32 columns of this thread's row ----
__device__ __forceinline__ void tm_ld8(uint32_t (&r)[8], uint32_t a) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                 "=r"(r[6]), "=r"(r[7])
               : "r"(a));
}
__device__ __forceinline__ void tm_ld16(uint32_t (&r)[16], uint32_t a) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(a));
}
__device__ __forceinline__ void tm_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// after the wait: the loaded registers are not used before it
template <int N>
__device__ __forceinline__ void tm_loaded(uint32_t (&r)[N]) {
#pragma unroll
  for (int i = 0; i < N; i++) asm volatile("" : "+r"(r[i]));
}
__device__ __forceinline__ void tm_st8(uint32_t a, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(a),
               "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
               "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tm_st2(uint32_t a, uint32_t x, uint32_t y) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1,%2};" ::"r"(a), "r"(x), "r"(y)
               : "memory");
}

// one K = 16 step: D (128 x n sums) [+]= A (tensor memory) times B (shared
// memory, K-major core matrices: the K halves n / 8 matrices apart, row
// groups adjacent; b16: its address / 16).  Issued by one elected thread of a
// converged warp with every operand the same in all its threads: then an
// n = 16 step issues every 9 cycles and n = 32 every 16, the matrix unit's own
// rate (from a lane picked by its number it took 179 cycles a step).
__device__ __forceinline__ void mma_step(uint32_t d, uint32_t a, uint32_t b16, int n,
                                         bool accumulate) {
  const uint64_t desc = (uint64_t)(b16 | ((uint32_t)n << 16)) |
                        ((uint64_t)(128 >> 4) << 32) | (1ull << 46);
  // f32 sums, f16 operands, K-major, N = n, M = 128
  const uint32_t idesc = (1u << 4) | ((uint32_t)(n >> 3) << 17) | (8u << 24);
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
      "r"(a), "l"(desc), "r"(idesc), "r"(accumulate ? 1u : 0u)
      : "memory");
}
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile(
      "{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(p));
  return p != 0;
}

// ---- words ----
// signed Montgomery reduction of a 64-bit value: v 2^-32 mod p, in
// (v / 2^32 - p / 2, v / 2^32 + p / 2]
__device__ __forceinline__ int32_t p2t_reduce(int64_t v) {
  const int32_t t = (int32_t)((uint32_t)v * kb::MU);
  return (int32_t)(v >> 32) - __mulhi(t, (int32_t)kb::P);
}
// x^3 in [-p, p] for |x| <= 0.998 2^31
__device__ __forceinline__ int32_t p2t_sbox(int32_t x) {
  const int32_t r = p2t_reduce((int64_t)x * x);
  return p2t_reduce((int64_t)r * x);
}
// N of them side by side, plus p: step by step through all, which the volatile
// statements hold the compiler to (one after the other, 2^19 rows of 64 words
// 465 us; in twos 455, fours 451, eights 449)
template <int N>
__device__ __forceinline__ void p2t_sboxes(int32_t (&x)[N]) {
  int64_t p[N];
  int32_t t[N];
#pragma unroll
  for (int i = 0; i < N; i++) asm volatile("mul.wide.s32 %0, %1, %1;" : "=l"(p[i]) : "r"(x[i]));
#pragma unroll
  for (int h = 0; h < 2; h++) {
#pragma unroll
    for (int i = 0; i < N; i++)
      asm volatile("mul.lo.s32 %0, %1, %2;" : "=r"(t[i]) : "r"((int32_t)p[i]), "r"(kb::MU));
#pragma unroll
    for (int i = 0; i < N; i++)
      asm volatile("mul.hi.s32 %0, %1, %2;" : "=r"(t[i]) : "r"(t[i]), "r"(kb::P));
#pragma unroll
    for (int i = 0; i < N; i++) {
      const uint32_t r = (uint32_t)(p[i] >> 32) - (uint32_t)t[i];
      if (h) x[i] = (int32_t)(r + kb::P);
      else asm volatile("mul.wide.s32 %0, %1, %2;" : "=l"(p[i]) : "r"(x[i]), "r"(r));
    }
  }
}
// a light layer's word from the bits of its two sums (p2_matrix.cpp chooses
// the constants so that the result is the word in a signed register)
__device__ __forceinline__ int32_t p2t_light_word(uint32_t b0, uint32_t b1) {
  return (int32_t)(b0 + (b1 << 16) - (b1 >> 15) * kb::P);
}
// a form's value times 2^32 from the bits of its four digit sums
__device__ __forceinline__ int64_t p2t_form(uint32_t b0, uint32_t b1, uint32_t b2, uint32_t b3) {
  const uint32_t lo = b0 + (b1 << 8), hi = b2 + (b3 << 8);
  return (int64_t)((uint64_t)hi * 65536u + lo);
}
// operands of a non-negative word: halves {byte 0, byte 1} and {2, 3}
__device__ __forceinline__ uint32_t p2t_low(uint32_t u) { return __byte_perm(u, 0, 0x4140); }
__device__ __forceinline__ uint32_t p2t_high(uint32_t u) { return __byte_perm(u, 0, 0x4342); }

// bounded wait for a barrier's phase: 2^18 polls, 3.8 us each while nothing
// arrives, so one second (the bound as a kernel argument costs 0.9% of 2^21
// rows of 32 words, and so does writing the host's flag in the loop)
__device__ __forceinline__ bool p2t_wait(uint32_t mbar, uint32_t parity) {
  uint32_t done = 0;
  for (int i = 0; i < (1 << 18) && !done; i++)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(mbar), "r"(parity), "r"(1000u)
        : "memory");
  return done != 0;
}
__device__ __forceinline__ void mma_commit(uint32_t mbar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
      : "memory");
}

// One tile of a CTA.  Every member is called by all 128 threads.
template <int W>
struct P2Tile {
  using L = P2Mat<W>;
  uint32_t row;    // this warp's lanes of the tile's columns
  uint32_t tile;   // the tile's columns, lane 0 (matrix operands)
  uint32_t tab;    // shared address of the tables, / 16
  uint32_t mbar;   // shared address of the tile's barrier
  uint32_t parity;
  int bar;         // named barrier of the tile
  bool issuer;     // this warp issues the tile's matrix instructions
  bool dead;       // a wait ran out: no more waiting

  // operand writes and sum reads of all rows are done; then `issue` runs on
  // one thread, and finish() waits for what it issued
  template <class F>
  __device__ __forceinline__ void start(F &&issue) {
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (!issuer) {
      asm volatile("bar.arrive %0, 128;" ::"r"(bar) : "memory");
    } else {
      asm volatile("bar.sync %0, 128;" ::"r"(bar) : "memory");
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (elect_one()) {
        issue();
        mma_commit(mbar);
      }
      __syncwarp();
    }
  }
  // The issuing warp alone polls the barrier and then releases the tile's
  // other warps.  When its wait runs out the tile goes on without waiting, its
  // results not valid; p2t_end waits for the products and tells the host.
  __device__ __forceinline__ void finish() {
    if (issuer) {
      if (!dead) dead = !p2t_wait(mbar, parity);
      __syncwarp();
      parity ^= 1u;
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    asm volatile("bar.sync %0, 128;" ::"r"(bar + L::TILES) : "memory");
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  }

  __device__ __forceinline__ void light(int l) const {
    const uint32_t d = tile + L::COL_DX;
    mma_step(d, tile + L::COL_C, tab + (L::cst_off + l * L::step_bytes(2 * L::NL)) / 16, 2 * L::NL,
             false);
#pragma unroll
    for (int s = 0; s < L::KX; s++) {
      const uint32_t b = tab + (L::ext_off + s * L::step_bytes(L::NL)) / 16;
      mma_step(d, tile + 8 * s, b, L::NL, true);
      mma_step(d + L::NL, tile + L::COL_H + 8 * s, b, L::NL, true);
    }
  }
  // a group of N columns of forms: the constant step, the external outputs,
  // ny steps of internal outputs
  template <int N>
  __device__ __forceinline__ void forms(uint32_t b, int ny) const {
    const uint32_t d = tile + L::COL_D;
    mma_step(d, tile + L::COL_C, b, N, false);
#pragma unroll
    for (int s = 0; s < 2 * L::KX; s++) {
      b += L::step_bytes(N) / 16;
      mma_step(d, tile + 8 * s, b, N, true);  // low pairs, then high ones (COL_H = W)
    }
    for (int s = 0; s < ny; s++) {
      b += L::step_bytes(N) / 16;
      mma_step(d, tile + L::COL_Y + 8 * s, b, N, true);
    }
  }

  __device__ __forceinline__ void put_words(int w0, const uint32_t (&u)[8]) const {
    uint32_t o[8];
#pragma unroll
    for (int i = 0; i < 8; i++) o[i] = p2t_low(u[i]);
    tm_st8(row + w0, o);
#pragma unroll
    for (int i = 0; i < 8; i++) o[i] = p2t_high(u[i]);
    tm_st8(row + L::COL_H + w0, o);
  }
  // words w0 .. w0 + 7 of the last light layer
  __device__ __forceinline__ void get_words(int w0, int32_t (&v)[8]) const {
    uint32_t a[8], b[8];
    tm_ld8(a, row + L::COL_DX + w0);
    tm_ld8(b, row + L::COL_DX + L::NL + w0);
    tm_ld_wait();
    tm_loaded(a);
    tm_loaded(b);
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = p2t_light_word(a[i], b[i]);
  }
  // S-boxes on a light layer's words, back into the operands
  __device__ __forceinline__ void sbox_words() const {
    uint32_t a[W / 8][8], b[W / 8][8];
#pragma unroll
    for (int g = 0; g < W / 8; g++) {
      tm_ld8(a[g], row + L::COL_DX + 8 * g);
      tm_ld8(b[g], row + L::COL_DX + L::NL + 8 * g);
    }
    tm_ld_wait();
#pragma unroll
    for (int g = 0; g < W / 8; g++) {
      int32_t x[8];
      uint32_t u[8];
      tm_loaded(a[g]);
      tm_loaded(b[g]);
#pragma unroll
      for (int i = 0; i < 8; i++) x[i] = p2t_light_word(a[g][i], b[g][i]);
      p2t_sboxes(x);
#pragma unroll
      for (int i = 0; i < 8; i++) u[i] = (uint32_t)x[i];
      put_words(8 * g, u);
    }
  }

  // Block q's outputs (two columns each; zeros behind them) as operands of the
  // blocks after it, which read whole steps of four: the columns there hold a
  // light layer's sums until an output is put.  Outputs 20.. share the
  // constants' step.
  __device__ __forceinline__ void put_outputs(int q, const uint32_t (&o)[16]) const {
    const uint32_t at = row + L::COL_Y + 2 * L::BLK * q;
    const uint32_t o0[8] = {o[0], o[1], o[2], o[3], o[4], o[5], o[6], o[7]};
    if constexpr (L::BLK == 4) {
      if (q < L::YSTEPS) tm_st8(at, o0);
    } else if (q < 3) {
      const uint32_t o1[8] = {o[8], o[9], o[10], o[11], 0, 0, 0, 0};
      tm_st8(at, o0);
      tm_st8(at + 8, o1);
    } else {
      tm_st2(at, o[0], o[1]);
      tm_st2(at + 2, o[2], o[3]);
      tm_st2(row + L::COL_C, o[4], o[5]);
      tm_st2(row + L::COL_C + 2, o[6], o[7]);
      tm_st2(row + L::COL_C + 4, o[8], o[9]);
    }
  }

  // The permutation of the words put by put_words; after it get_words reads
  // the result (signed, |v| < 2^31, congruent).  `between` runs once the
  // state needs few registers (input of the next permutation is fetched there).
  template <class F>
  __device__ __forceinline__ void permute(const int32_t (&tri)[4], F &&between) {
    start([&] { light(0); });
    finish();
#pragma unroll 1
    for (int r = 0; r < 3; r++) {
      sbox_words();
      start([&] { light(r + 1); });
      finish();
    }
    sbox_words();
#pragma unroll 1
    for (int q = 0; q < L::NBLK; q++) {
      start([&] { forms<L::NB>(tab + L::blk_off(q) / 16, L::blk_ysteps(q)); });
      finish();
      uint32_t b[16], b2[8] = {};
      tm_ld16(b, row + L::COL_D);
      if constexpr (L::BLK == 6) tm_ld8(b2, row + L::COL_D + 16);
      tm_ld_wait();
      tm_loaded(b);
      if constexpr (L::BLK == 6) tm_loaded(b2);
      uint32_t o[16] = {};
      int32_t y[L::BLK];
      uint32_t yc = 0;  // the last output, canonical
#pragma unroll
      for (int i = 0; i < L::BLK; i++) {
        const uint32_t *d = i < 4 ? b + 4 * i : b2 + 4 * (i - 4);
        int64_t x = p2t_form(d[0], d[1], d[2], d[3]);
#pragma unroll
        for (int j = 0; j + 1 < i; j++) x += (int64_t)tri[i - 2 - j] * y[j];
        int32_t z = p2t_reduce(x);
        // the output before weighs -1 (p2_matrix.cpp), so it needs no product
        if (i) z = (int32_t)(kb::umin((uint32_t)z, (uint32_t)z + kb::P) - yc);
        y[i] = p2t_sbox(z);
        yc = kb::umin((uint32_t)y[i], (uint32_t)y[i] + kb::P);
        o[2 * i] = p2t_low(yc);
        o[2 * i + 1] = p2t_high(yc);
      }
      put_outputs(q, o);
    }
    between();
    // the state after the internal rounds, FW words at a time, through round
    // 4's S-boxes; the next words' sums run meanwhile
    uint32_t u[W / 8][8];
    start([&] { forms<4 * L::FW>(tab + L::fin_off(0) / 16, L::YSTEPS); });
#pragma unroll
    for (int c = 0; c < L::NFIN; c++) {
      finish();
      uint32_t b[L::FW / 4][16];
#pragma unroll
      for (int g = 0; g < L::FW / 4; g++) tm_ld16(b[g], row + L::COL_D + 16 * g);
      tm_ld_wait();
#pragma unroll
      for (int g = 0; g < L::FW / 4; g++) tm_loaded(b[g]);
      if (c + 1 < L::NFIN)
        start([&] { forms<4 * L::FW>(tab + L::fin_off(c + 1) / 16, L::YSTEPS); });
#pragma unroll
      for (int i = 0; i < L::FW; i++) {
        const uint32_t(&d)[16] = b[i / 4];
        const int k = 4 * (i & 3), w = L::FW * c + i;
        u[w / 8][w % 8] =
            (uint32_t)p2t_sbox(p2t_reduce(p2t_form(d[k], d[k + 1], d[k + 2], d[k + 3]))) + kb::P;
      }
    }
#pragma unroll
    for (int c = 0; c < W / 8; c++) put_words(8 * c, u[c]);
    start([&] { light(4); });
    finish();
#pragma unroll 1
    for (int r = 5; r < 8; r++) {
      sbox_words();
      start([&] { light(r); });
      finish();
    }
  }
};

// canonical word of a light layer's signed one
__device__ __forceinline__ uint32_t p2t_canonical(int32_t v) {
  if (v < 0) v += (int32_t)kb::P;
  if (v < 0) v += (int32_t)kb::P;
  const uint32_t u = (uint32_t)v;
  return kb::umin(u, u - kb::P);
}
// the same residue as a non-negative word
__device__ __forceinline__ uint32_t p2t_unsigned(int32_t v) {
  return v < 0 ? (uint32_t)v + 2u * kb::P : (uint32_t)v;
}

// A CTA's start and end.  Shared memory: the tables, one barrier per tile,
// the tensor-memory address, one more barrier per tile for a wait that ran out.
template <int W>
constexpr size_t p2t_smem() {
  return P2Mat<W>::bytes + 8 * (2 * P2Mat<W>::TILES + 1);
}
template <int W>
__device__ __forceinline__ P2Tile<W> p2t_begin(unsigned char *sm, const uint4 *table,
                                               const WaitReport &report) {
  using L = P2Mat<W>;
  static_assert(L::bytes % 16 == 0, "table copy");
  uint64_t *bars = reinterpret_cast<uint64_t *>(sm + L::bytes);
  uint32_t *addr = reinterpret_cast<uint32_t *>(bars + L::TILES);
  uint4 *dst = reinterpret_cast<uint4 *>(sm);
  for (int i = threadIdx.x; i < L::bytes / 16; i += p2t_threads<W>) dst[i] = __ldg(table + i);
  if (threadIdx.x < L::TILES)
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bars + threadIdx.x))
                 : "memory");
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_addr(addr)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  // the tables and barriers are visible to the matrix unit
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  P2Tile<W> t;
  // warp numbers and addresses as warp-uniform values (see mma_step)
  const int wid = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  const int tile = wid >> 2, warp = wid & 3;
  t.tile = __shfl_sync(0xffffffffu, *addr, 0) + L::COLS * tile;
  t.row = t.tile + ((uint32_t)(32 * warp) << 16);
  t.tab = smem_addr(sm) >> 4;
  t.mbar = smem_addr(bars + tile);
  t.parity = 0;
  t.bar = 1 + tile;
  t.issuer = warp == (tile & 3);  // one issuer per scheduler
  t.dead = report.expire;
  // the constants' operands, and zeros where internal outputs 20.. will be
  const uint32_t c[8] = {0, 0, 0, 0, 0, 0, P2M_CONST0, P2M_CONST1};
  tm_st8(t.row + L::COL_C, c);
  return t;
}
template <int W>
__device__ __forceinline__ void p2t_end(unsigned char *sm, const P2Tile<W> &t,
                                        const WaitReport &report) {
  // a tile that gave up a wait: the host is told, and its products end before
  // the columns are freed (a commit covers all that the thread has issued)
  if (t.issuer && __any_sync(0xffffffffu, t.dead)) {
    *reinterpret_cast<volatile unsigned int *>(report.error) = 1u;
    __threadfence_system();
    const uint32_t bar = t.mbar + 8 * (P2Mat<W>::TILES + 1);
    if (elect_one()) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      mma_commit(bar);
    }
    __syncwarp();
    p2t_wait(bar, 0);
    __syncwarp();
  }
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t a = *reinterpret_cast<uint32_t *>(sm + P2Mat<W>::bytes + 8 * P2Mat<W>::TILES);
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(a),
                 "r"(512));
  }
}

}  // namespace gpu
}  // namespace whir
