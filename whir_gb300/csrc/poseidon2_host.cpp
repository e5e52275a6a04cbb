// Host Poseidon2 constants and permutation (see poseidon2_host.h).
#include "poseidon2_host.h"

#include <mutex>
#include <utility>

#include "kb.cuh"

#if defined(__ARM_NEON)
#include <arm_neon.h>  // vmull_u32: the compiler forms no widening product of its own vectors
#endif

namespace whir {
namespace {

// ChaCha with the original 64-bit block counter (words 12-13) and a zero
// stream id (words 14-15): the block function behind rand's StdRng.
struct ChaCha12 {
  uint32_t key[8];
  uint64_t counter = 0;
  uint32_t buf[16];
  int idx = 16;

  static uint32_t rotl(uint32_t x, int n) { return (x << n) | (x >> (32 - n)); }
  static void quarter(uint32_t &a, uint32_t &b, uint32_t &c, uint32_t &d) {
    a += b; d ^= a; d = rotl(d, 16);
    c += d; b ^= c; b = rotl(b, 12);
    a += b; d ^= a; d = rotl(d, 8);
    c += d; b ^= c; b = rotl(b, 7);
  }
  void refill() {
    uint32_t s[16] = {0x61707865, 0x3320646e, 0x79622d32, 0x6b206574};
    for (int i = 0; i < 8; i++) s[4 + i] = key[i];
    s[12] = (uint32_t)counter;
    s[13] = (uint32_t)(counter >> 32);
    s[14] = 0;
    s[15] = 0;
    uint32_t x[16];
    for (int i = 0; i < 16; i++) x[i] = s[i];
    for (int r = 0; r < 12; r += 2) {
      quarter(x[0], x[4], x[8], x[12]);
      quarter(x[1], x[5], x[9], x[13]);
      quarter(x[2], x[6], x[10], x[14]);
      quarter(x[3], x[7], x[11], x[15]);
      quarter(x[0], x[5], x[10], x[15]);
      quarter(x[1], x[6], x[11], x[12]);
      quarter(x[2], x[7], x[8], x[13]);
      quarter(x[3], x[4], x[9], x[14]);
    }
    for (int i = 0; i < 16; i++) buf[i] = x[i] + s[i];
    counter++;
    idx = 0;
  }
  explicit ChaCha12(uint64_t seed) {
    // rand_core: PCG32 output words fill the 32-byte seed little-endian.
    const uint64_t mul = 6364136223846793005ull, inc = 11634580027462260723ull;
    for (int i = 0; i < 8; i++) {
      seed = seed * mul + inc;
      uint32_t xs = (uint32_t)(((seed >> 18) ^ seed) >> 27);
      uint32_t rot = (uint32_t)(seed >> 59);
      key[i] = (xs >> rot) | (xs << ((32 - rot) & 31));
    }
  }
  uint32_t next_u32() {
    if (idx == 16) refill();
    return buf[idx++];
  }
  // StandardUniform<MontyField31>: 31 random bits, rejected at p, kept as the
  // Montgomery word.
  uint32_t next_field() {
    for (;;) {
      uint32_t v = next_u32() >> 1;
      if (v < kb::P) return v;
    }
  }
};

// Internal diagonals of p3-koala-bear's Poseidon2 (V in M_I = 1 1^T + diag(V)),
// entry i = sign * num / 2^log_den.
constexpr int v16[16][3] = {{-1, 2, 0}, {1, 1, 0},  {1, 2, 0},  {1, 1, 1},
                            {1, 3, 0},  {1, 4, 0},  {-1, 1, 1}, {-1, 3, 0},
                            {-1, 4, 0}, {1, 1, 8},  {1, 1, 3},  {1, 1, 24},
                            {-1, 1, 8}, {-1, 1, 3}, {-1, 1, 4}, {-1, 1, 24}};
constexpr int v24[24][3] = {{-1, 2, 0}, {1, 1, 0},  {1, 2, 0},  {1, 1, 1},  {1, 3, 0},
                            {1, 4, 0},  {-1, 1, 1}, {-1, 3, 0}, {-1, 4, 0}, {1, 1, 8},
                            {1, 1, 2},  {1, 1, 3},  {1, 1, 4},  {1, 1, 5},  {1, 1, 6},
                            {1, 1, 24}, {-1, 1, 8}, {-1, 1, 3}, {-1, 1, 4}, {-1, 1, 5},
                            {-1, 1, 6}, {-1, 1, 7}, {-1, 1, 9}, {-1, 1, 24}};

// diag entry sign * num / 2^log_den
uint32_t diag_value(int sign, uint32_t num, int log_den) {
  uint32_t v = kb::mul(kb::from_canonical(num), kb::inv(kb::pow(kb::from_canonical(2), log_den)));
  return sign < 0 ? kb::neg(v) : v;
}

void build(Poseidon2Constants &c, int width) {
  c.width = width;
  c.rounds_p = width == 16 ? 20 : 23;  // poseidon2_round_numbers_128 for 31-bit p, D = 3
  for (int i = 0; i < width; i++) {
    const int *v = width == 16 ? v16[i] : v24[i];
    c.diag[i] = diag_value(v[0], (uint32_t)v[1], v[2]);
  }
  ChaCha12 rng(1000);
  for (int r = 0; r < 8; r++)
    for (int i = 0; i < width; i++) c.ext_rc[r][i] = rng.next_field();
  for (int r = 0; r < c.rounds_p; r++) c.int_rc[r] = rng.next_field();
}

// x mod p for x < 2^38: 2^31 = 2^24 - 1 (mod p) folds the bits above 31,
// leaving a value below 2^32 < 3p, then two conditional subtractions.
inline uint32_t reduce38(uint64_t x) {
  uint64_t y = (x & 0x7fffffffu) + (x >> 31) * 0x00ffffffull;
  y = y >= 2ull * kb::P ? y - 2ull * kb::P : y;
  return (uint32_t)(y >= kb::P ? y - kb::P : y);
}

// The linear layers in 64-bit lanes with one reduction per output word.
inline void mat4_wide(uint64_t *x) {
  uint64_t t01 = x[0] + x[1], t23 = x[2] + x[3];
  uint64_t t0123 = t01 + t23;
  uint64_t t01123 = t0123 + x[1], t01233 = t0123 + x[3];
  uint64_t y3 = t01233 + 2 * x[0];
  uint64_t y1 = t01123 + 2 * x[2];
  uint64_t y0 = t01123 + t01;
  uint64_t y2 = t01233 + t23;
  x[0] = y0; x[1] = y1; x[2] = y2; x[3] = y3;
}
// light MDS of canonical words: every output below 49 p < 2^38 before its
// reduction
inline void mds_light(uint32_t *s) {
  constexpr int W = 24;
  uint64_t x[W];
  for (int i = 0; i < W; i++) x[i] = s[i];
  for (int i = 0; i < W; i += 4) mat4_wide(x + i);
  uint64_t sums[4] = {0, 0, 0, 0};
  for (int i = 0; i < W; i++) sums[i & 3] += x[i];
  for (int i = 0; i < W; i++) s[i] = reduce38(x[i] + sums[i & 3]);
}
// s_i <- sum + d_i s_i with the diagonal's small entries (Montgomery form is
// linear, so scaling the word scales the element): num in 1..4 as a multiple
// of x or of p - x; 2^-e as (x + m p) / 2^e with m = -x mod 2^e (exact, since
// p = 1 mod 2^24), below 2p; every lane below 2^38 before one reduction.
// Each lane's form is fixed at compile time.
template <int I>
inline void internal_lane(uint32_t *s, uint64_t sum) {
  constexpr int sign = v24[I][0], num = v24[I][1], e = v24[I][2];
  const uint64_t x = s[I];
  uint64_t t;
  if constexpr (e == 0) {
    t = sign > 0 ? (uint64_t)num * x : (uint64_t)num * (kb::P - x);
  } else {
    const uint64_t m = (0 - x) & ((1ull << e) - 1);
    const uint64_t y = (x + m * kb::P) >> e;  // < 2p
    t = sign > 0 ? y : 2ull * kb::P - y;
  }
  s[I] = reduce38(sum + t);
}
template <int... I>
inline void internal_lanes(uint32_t *s, uint64_t sum, std::integer_sequence<int, I...>) {
  (internal_lane<I>(s, sum), ...);
}
inline void internal_layer(uint32_t *s) {
  uint64_t total = 0;
  for (int i = 0; i < 24; i++) total += s[i];
  internal_lanes(s, reduce38(total), std::make_integer_sequence<int, 24>{});
}

void permute24(const Poseidon2Constants &c, uint32_t *s) {
  using namespace kb;
  mds_light(s);
  for (int r = 0; r < 4; r++) {
    for (int i = 0; i < 24; i++) s[i] = cube(add(s[i], c.ext_rc[r][i]));
    mds_light(s);
  }
  for (int r = 0; r < c.rounds_p; r++) {
    s[0] = cube(add(s[0], c.int_rc[r]));
    internal_layer(s);
  }
  for (int r = 4; r < 8; r++) {
    for (int i = 0; i < 24; i++) s[i] = cube(add(s[i], c.ext_rc[r][i]));
    mds_light(s);
  }
}

// ---- width 16 on 128-bit vectors: the challenger's permutation ----
// A proof's host work between two launches is mostly these permutations, one
// after another.  Word 4g + j of the state is lane g of vector j, so that the
// light layer's 4x4 blocks are additions of whole vectors.
// Grace (Neoverse V2): 883 ns for the form of permute24 at this width, bound by
// its 9000 instructions; 415 ns so, bound by the latency of the S-box chain
// (23.6 ns an external round, 10.8 ns an internal one).
typedef uint32_t V4 __attribute__((vector_size(16)));
typedef uint64_t D2 __attribute__((vector_size(16)));

inline V4 splat(uint32_t x) { return V4{x, x, x, x}; }
inline V4 vmin(V4 a, V4 b) { return a < b ? a : b; }
inline V4 even(D2 a, D2 b) { return __builtin_shufflevector((V4)a, (V4)b, 0, 2, 4, 6); }
inline V4 odd(D2 a, D2 b) { return __builtin_shufflevector((V4)a, (V4)b, 1, 3, 5, 7); }
// the four 64-bit products, lanes 0 and 1 in lo
inline void mul_wide(V4 a, V4 b, D2 &lo, D2 &hi) {
#if defined(__ARM_NEON)
  lo = (D2)vmull_u32(vget_low_u32((uint32x4_t)a), vget_low_u32((uint32x4_t)b));
  hi = (D2)vmull_high_u32((uint32x4_t)a, (uint32x4_t)b);
#else
  const V4 z{};
  lo = (D2)__builtin_shufflevector(a, z, 0, 4, 1, 5) * (D2)__builtin_shufflevector(b, z, 0, 4, 1, 5);
  hi = (D2)__builtin_shufflevector(a, z, 2, 6, 3, 7) * (D2)__builtin_shufflevector(b, z, 2, 6, 3, 7);
#endif
}
// a b 2^-32 mod p in (0, 2p), for a b < p 2^32; ab_mu = a b p^-1 mod 2^32
// (the low product on its own: it does not wait for the wide one)
inline V4 vmul_lazy(V4 a, V4 b, V4 ab_mu) {
  D2 l, h, tl, th;
  mul_wide(a, b, l, h);
  mul_wide(ab_mu, splat(kb::P), tl, th);
  return (odd(l, h) + kb::P) - odd(tl, th);
}
// the same in [0, p)
inline V4 vmul(V4 a, V4 b, V4 ab_mu) {
  D2 l, h, tl, th;
  mul_wide(a, b, l, h);
  mul_wide(ab_mu, splat(kb::P), tl, th);
  const V4 hi = odd(l, h), lo = odd(tl, th);
  return vmin(hi - lo, (hi + kb::P) - lo);
}
// x^3 for x < 1.4 2^31 (x^2 < p 2^32; the second factor is reduced meanwhile)
inline V4 vcube(V4 x, V4 mu) {
  const V4 xc = vmin(x, x - kb::P), xc_mu = xc * mu;
  const V4 x2 = vmul_lazy(x, x, x * x * mu);
  return vmul(x2, xc, x2 * xc_mu);
}

struct Lanes16 {
  D2 rc[8][4][2];           // external constants
  V4 rc4[4];                // those of round 4 as words
  V4 diag[4], diag_mu[4];   // the internal diagonal, lane 0 zero; times p^-1
  // p^-1 mod 2^32.  Not a constant to the compiler, which would make it shifts
  // after the product x y where (x p^-1) y leaves one multiply on the chain.
  V4 mu;
};
const Lanes16 &lanes16() {
  static const Lanes16 t = [] {
    const Poseidon2Constants &c = poseidon2_constants(16);
    Lanes16 l;
    l.mu = splat(kb::MU);
    for (int j = 0; j < 4; j++)
      for (int g = 0; g < 4; g++) {
        for (int r = 0; r < 8; r++) l.rc[r][j][g / 2][g % 2] = c.ext_rc[r][4 * g + j];
        l.rc4[j][g] = c.ext_rc[4][4 * g + j];
        l.diag[j][g] = g + j ? c.diag[4 * g + j] : 0;
        l.diag_mu[j][g] = l.diag[j][g] * kb::MU;
      }
    return l;
  }();
  return t;
}

// light layer of words below 1.02 p plus the next round's constants: 64-bit
// lanes below 37 p (rows of 2 3 1 1 in four blocks, the own one twice), folded
// once with 2^31 = 2^24 - 1 to below 2^31 + 37 2^24 < 1.4 2^31
inline void light16(V4 *x, const D2 (*rc)[2]) {
  D2 y[4][2];
  for (int h = 0; h < 2; h++) {
    D2 w[4];
    for (int j = 0; j < 4; j++)
      w[j] = h ? (D2)__builtin_shufflevector(x[j], V4{}, 2, 6, 3, 7)
               : (D2)__builtin_shufflevector(x[j], V4{}, 0, 4, 1, 5);
    const D2 t01 = w[0] + w[1], t23 = w[2] + w[3], t = t01 + t23;
    const D2 u = t + w[1], v = t + w[3];
    y[0][h] = u + t01;
    y[1][h] = u + (w[2] + w[2]);
    y[2][h] = v + t23;
    y[3][h] = v + (w[0] + w[0]);
  }
  for (int j = 0; j < 4; j++) {
    D2 sum = y[j][0] + y[j][1];
    sum += __builtin_shufflevector(sum, sum, 1, 0);
    D2 a = y[j][0], b = y[j][1];
    if (rc) {
      a += rc[j][0];
      b += rc[j][1];
    }
    a += sum;
    b += sum;
    x[j] = (even(a, b) & 0x7fffffffu) + even(a >> 31, b >> 31) * 0x00ffffffu;
  }
}
// sum of the 16 words, as an integer
inline uint64_t total16(const V4 *x) {
  const V4 a = x[0] + x[1], b = x[2] + x[3];  // below 2p < 2^32
  const D2 m = D2{0xffffffffu, 0xffffffffu};
  const D2 s = (((D2)a & m) + ((D2)a >> 32)) + (((D2)b & m) + ((D2)b >> 32));
  return s[0] + s[1];
}
// x mod p for x < 48 p, as reduce38
inline uint32_t fold48(uint64_t x) {
  const uint32_t y = (uint32_t)(x & 0x7fffffffu) + (uint32_t)(x >> 31) * 0x00ffffffu;
  return kb::umin(y, y - kb::P);
}
// z^3 for -p < z < p
inline uint32_t cube_signed(int32_t z, uint32_t mu) {
  const uint32_t zc = kb::umin((uint32_t)z, (uint32_t)z + kb::P), zc_mu = zc * mu;
  const uint32_t lo = (uint32_t)z * (uint32_t)z;
  const uint32_t z2 = (uint32_t)((uint64_t)((int64_t)z * z) >> 32) + kb::P -
                      kb::mulhi(lo * mu, kb::P);  // in (0, 2p)
  const uint32_t hi = kb::mulhi(z2, zc), th = kb::mulhi(z2 * zc_mu, kb::P);
  return hi < th ? hi + kb::P - th : hi - th;
}

// The internal rounds keep word 0 in scalar registers: with T the sum of words
// 1..15 and y the cube of word 0 (its diagonal entry is -2), the lane sum is
// S = T + y and the next word 0 is T - y, so the chain from cube to cube is one
// subtraction.  The vectors hold m = d s of words 1..15: s' = m + S, and the
// next T is sum(m) + 15 S, where sum(m) depends on the S before.
void permute16(const Poseidon2Constants &c, uint32_t *st) {
  const Lanes16 &t = lanes16();
  const uint32_t mu = t.mu[0];
  V4 x[4];
  for (int j = 0; j < 4; j++) {
    x[j] = V4{st[j], st[4 + j], st[8 + j], st[12 + j]};
    x[j] = vmin(x[j], x[j] - kb::P);  // any word is below 1.02 p now
  }
  light16(x, t.rc[0]);
  for (int r = 0; r < 4; r++) {
    for (int j = 0; j < 4; j++) x[j] = vcube(x[j], t.mu);
    light16(x, r < 3 ? t.rc[r + 1] : nullptr);
  }
  for (int j = 0; j < 4; j++) x[j] = vmin(x[j], x[j] - kb::P);
  uint32_t T = fold48(total16(x) - x[0][0]), x0 = x[0][0];
  int32_t z = (int32_t)(kb::add(x0, c.int_rc[0]));
  for (int j = 0; j < 4; j++) x[j] = vmul(x[j], t.diag[j], x[j] * t.diag_mu[j]);
  for (int r = 0; r < 20; r++) {
    const uint64_t u = total16(x);
    const uint32_t next = r < 19 ? kb::add(T, c.int_rc[r + 1]) : T;
    const uint32_t y = cube_signed(z, mu);
    const uint32_t S = kb::add(T, y);
    z = (int32_t)(next - y);
    T = fold48(u + 15ull * S);
    for (int j = 0; j < 4; j++) x[j] += splat(S);  // below 2p
    if (r < 19)
      for (int j = 0; j < 4; j++) x[j] = vmul(x[j], t.diag[j], x[j] * t.diag_mu[j]);
  }
  for (int j = 0; j < 4; j++) x[j] = vmin(x[j], x[j] - kb::P);
  x[0][0] = kb::umin((uint32_t)z, (uint32_t)z + kb::P);
  for (int j = 0; j < 4; j++) {
    x[j] += t.rc4[j];
    x[j] = vmin(x[j], x[j] - kb::P);
  }
  for (int r = 4; r < 8; r++) {
    for (int j = 0; j < 4; j++) x[j] = vcube(x[j], t.mu);
    light16(x, r < 7 ? t.rc[r + 1] : nullptr);
  }
  for (int j = 0; j < 4; j++) x[j] = vmin(x[j], x[j] - kb::P);
  for (int j = 0; j < 4; j++)
    for (int g = 0; g < 4; g++) st[4 * g + j] = x[j][g];
}

}  // namespace

const Poseidon2Constants &poseidon2_constants(int width) {
  static Poseidon2Constants c16, c24;
  static std::once_flag once;
  std::call_once(once, [] {
    build(c16, 16);
    build(c24, 24);
  });
  return width == 16 ? c16 : c24;
}

void poseidon2_permute_host(const Poseidon2Constants &c, uint32_t *s) {
  if (c.width == 16) permute16(c, s);
  else permute24(c, s);
}

void std_rng_fill_field(uint64_t seed, uint32_t *out, uint64_t n) {
  ChaCha12 rng(seed);
  for (uint64_t i = 0; i < n; i++) out[i] = rng.next_field();
}

}  // namespace whir
