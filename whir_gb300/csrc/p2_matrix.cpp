// Host construction of the tensor-core Poseidon2 tables (see p2_matrix.h).
#include "p2_matrix.h"

#include <cmath>
#include <mutex>
#include <stdexcept>

#include "poseidon2_host.h"

namespace whir {
namespace gpu {
namespace {

// an integer of at most 11 significant bits times 2^e as a half
uint16_t half_bits(int v, int e) {
  if (v == 0) return 0;
  uint16_t sign = v < 0 ? 0x8000 : 0;
  int m = v < 0 ? -v : v;
  int top = 31 - __builtin_clz((unsigned)m), exp = top + e;
  if (top > 10 || exp > 15 || exp < -14) throw std::logic_error("p2 tables: not a half");
  return (uint16_t)(sign | ((exp + 15) << 10) | ((m << (10 - top)) & 0x3ff));
}

// light MDS: mat4 on each group of 4, then every group gets the column sums
template <int W>
int light_entry(int i, int j) {
  static const int m4[4][4] = {{2, 3, 1, 1}, {1, 2, 3, 1}, {1, 1, 2, 3}, {3, 1, 1, 2}};
  return m4[i & 3][j & 3] * (i / 4 == j / 4 ? 2 : 1);
}

// a linear form of the S-box outputs: coefficients (Montgomery words) of the
// fourth external round's W outputs and the internal rounds' outputs, and an
// added residue
template <int W>
struct Form {
  uint32_t c[W + P2Mat<W>::RP] = {};
  uint32_t k = 0;
};
template <int W>
Form<W> operator+(const Form<W> &a, const Form<W> &b) {
  Form<W> r;
  for (int i = 0; i < W + P2Mat<W>::RP; i++) r.c[i] = kb::add(a.c[i], b.c[i]);
  r.k = kb::add(a.k, b.k);
  return r;
}
template <int W>
Form<W> scaled(const Form<W> &a, uint32_t d) {
  Form<W> r;
  for (int i = 0; i < W + P2Mat<W>::RP; i++) r.c[i] = kb::mul(a.c[i], d);
  r.k = kb::mul(a.k, d);
  return r;
}

template <int W>
struct Builder {
  using L = P2Mat<W>;
  P2Tables t;
  const Poseidon2Constants &pc = poseidon2_constants(W);

  void put(int off, int n, int row, int k, uint16_t h) {
    const int core = (k / 8) * (n / 8) + row / 8;
    t.halves[(off + core * 128 + (row % 8) * 16 + (k % 8) * 2) / 2] = h;
  }
  // the constant slots (K 12..14): (2^23 + v) units as three bytes
  void put_const(int off, int n, int row, uint32_t v, int e) {
    if (v >= (1u << 23)) throw std::logic_error("p2 tables: constant out of range");
    const uint32_t u = (1u << 23) + v;
    put(off, n, row, 12, half_bits((int)(u >> 16), e));
    put(off, n, row, 13, half_bits((int)((u >> 8) & 255), e));
    put(off, n, row, 14, half_bits((int)(u & 255), e));
  }

  void light_layers() {
    // unit 2^-19: a byte is 2^-24 of itself, the entry m 2^5 on the low byte
    // of a pair and m 2^13 on the high one
    int row_sum = 0;
    for (int j = 0; j < W; j++) row_sum += light_entry<W>(0, j);
    for (int s = 0; s < L::KX; s++)
      for (int i = 0; i < W; i++)
        for (int k = 0; k < 16; k++)
          put(L::ext_off + s * L::step_bytes(L::NL), L::NL, i, k,
              half_bits(light_entry<W>(i, 8 * s + k / 2), k & 1 ? 13 : 5));
    // Recombined (p2_tensor.cuh) as V = b0 + (b1 << 16) - (b1 >> 15) p of the
    // two sums' bits, V = X - q p + E - (E >> 15) - 2^32 with X the weighted
    // sum, q = (b1's integer) >> 15.  JQ 2^15 added to the high sum moves q
    // so that V fits a signed word with room on both sides.
    const int qw = (int)(((int64_t)row_sum * 65535 + 32767) >> 15) + 1;  // q - JQ <= qw
    const int64_t e = (int64_t)P2M_E_LIGHT - (P2M_E_LIGHT >> 15) - ((int64_t)1 << 32);
    const int64_t lo1 = (1ll << 24) - 1;
    // V - q lo1 lies in [e, e + 2^31 + 2^23): centre q's range
    const int64_t mid = e + (1ll << 30) + (1ll << 22);
    const int JQ = (int)((-mid - (int64_t)qw * lo1 / 2) / lo1);
    const int64_t vmin = e + JQ * lo1, vmax = e + (1ll << 31) + (1ll << 23) + (JQ + qw) * lo1;
    if (JQ < 0 || vmin < -(int64_t)(0.97 * 2147483648.) || vmax > (int64_t)(0.97 * 2147483648.))
      throw std::logic_error("p2 tables: light layer window");
    if (((int64_t)(JQ + 1) << 15) + (int64_t)row_sum * 65535 >= (1 << 23))
      throw std::logic_error("p2 tables: light layer sum");
    const int next_rc[L::NCST] = {0, 1, 2, 3, 5, 6, 7, -1};
    for (int l = 0; l < L::NCST; l++)
      for (int i = 0; i < W; i++) {
        const uint32_t rc = next_rc[l] < 0 ? 0 : pc.ext_rc[next_rc[l]][i];
        int64_t d = ((int64_t)rc - e - ((int64_t)JQ << 31)) % (int64_t)kb::P;
        if (d < 0) d += kb::P;
        const int off = L::cst_off + l * L::step_bytes(2 * L::NL);
        put_const(off, 2 * L::NL, i, (uint32_t)(d & 0xffff), -3);
        put_const(off, 2 * L::NL, L::NL + i, (uint32_t)(d >> 16) + ((uint32_t)JQ << 15), -3);
      }
  }

  // four columns (rows row..row+3 of the steps) of one form over the first
  // ny internal outputs
  void form_columns(int off, int n, int row, const Form<W> &f, int ny) {
    int64_t smin[4] = {}, smax[4] = {};
    auto place = [&](int step, int k, uint32_t coef, int byte) {
      int64_t v = kb::mul(coef, kb::from_canonical(1u << (8 * byte)));
      if (v > kb::P / 2) v -= kb::P;
      for (int d = 0; d < 4; d++) {
        int64_t digit = v;
        if (d < 3) {
          digit = ((v % 256) + 256) % 256;
          if (digit > 127) digit -= 256;
          v = (v - digit) / 256;
        }
        put(off + step * L::step_bytes(n), n, row + d, k, half_bits((int)digit, 8));
        (digit < 0 ? smin : smax)[d] += 255 * digit;
      }
    };
    for (int w = 0; w < W; w++)
      for (int b = 0; b < 4; b++)
        place(1 + (b / 2) * L::KX + w / 8, 2 * (w % 8) + (b & 1), f.c[w], b);
    for (int r = 0; r < ny; r++)
      for (int b = 0; b < 4; b++) {
        if (r < 4 * L::YSTEPS) place(1 + 2 * L::KX + r / 4, 4 * (r % 4) + b, f.c[W + r], b);
        else place(0, 4 * (r - 4 * L::YSTEPS) + b, f.c[W + r], b);
      }
    // X = E (1 + 2^16) + sum 2^(8d) (S_d + off_d), reduced by 2^-32: the
    // constant has to be k 2^32
    uint64_t have = (uint64_t)P2M_E_FORM * 65537ull % kb::P;
    for (int d = 0; d < 4; d++) have += ((uint64_t)(-smin[d]) << (8 * d)) % kb::P;
    const uint64_t want = kb::mul(f.k, kb::R2);
    const uint64_t diff = (want + 8ull * kb::P - have % kb::P) % kb::P;
    for (int d = 0; d < 4; d++) {
      const int64_t o = -smin[d] + (int64_t)((diff >> (8 * d)) & 255);
      if (o + smax[d] >= (1 << 23)) throw std::logic_error("p2 tables: form sum");
      put_const(off, n, row + d, (uint32_t)o, 0);
    }
  }

  void forms() {
    std::vector<Form<W>> s(W);
    for (int i = 0; i < W; i++)
      for (int j = 0; j < W; j++)
        s[i].c[j] = kb::from_canonical((uint32_t)light_entry<W>(i, j));
    std::vector<Form<W>> z(L::RP);
    for (int r = 0; r < L::RP; r++) {
      z[r] = s[0];
      z[r].k = kb::add(z[r].k, pc.int_rc[r]);
      s[0] = Form<W>();
      s[0].c[W + r] = kb::ONE;
      Form<W> sum;
      for (int i = 0; i < W; i++) sum = sum + s[i];
      for (int i = 0; i < W; i++) s[i] = sum + scaled(s[i], pc.diag[i]);
    }
    for (int q = 0; q < L::NBLK; q++)
      for (int i = 0; i < L::BLK && L::BLK * q + i < L::RP; i++)
        form_columns(L::blk_off(q), L::NB, 4 * i, z[L::BLK * q + i], L::BLK * q);
    for (int i = 0; i < W; i++) {
      s[i].k = kb::add(s[i].k, pc.ext_rc[4][i]);
      form_columns(L::fin_off(i / L::FW), 4 * L::FW, 4 * (i % L::FW), s[i], L::RP);
    }
    if (z[1].c[W] != kb::neg(kb::ONE)) throw std::logic_error("p2 tables: next round's weight");
    for (int d = 0; d + 2 < L::BLK; d++) {  // z_(d+2)'s weight on internal output 0
      const uint32_t c = z[d + 2].c[W];
      t.tri[d] = c > kb::P / 2 ? (int32_t)(c - kb::P) : (int32_t)c;
    }
    // The block's values stay in range (units of 2^31; a signed reduction of v
    // ends within |v| / 2^32 + p / 2).  Round i's form with the outputs up to
    // two rounds before ends within (-p, p); less the output before, both
    // canonical, the S-box's operand does too.
    const double p = kb::P / 2147483648.;
    double y[8];
    for (int i = 0; i < L::BLK; i++) {
      double v = 1e-4;  // the form itself, below 2^49
      for (int j = 0; j + 1 < i; j++) v += std::abs(t.tri[i - 2 - j] / 2147483648.) * y[j];
      const double f = v / 2 + p / 2, x = i ? p : f, r = x * x / 2 + p / 2;
      if (f > p || r > p) throw std::logic_error("p2 tables: block range");
      y[i] = r * x / 2 + p / 2;
    }
  }

  Builder() {
    t.halves.assign(L::bytes / 2, 0);
    light_layers();
    forms();
  }
};

}  // namespace

const P2Tables &p2_tables(int width) {
  static const P2Tables t16 = Builder<16>().t;
  static const P2Tables t24 = Builder<24>().t;
  return width == 16 ? t16 : t24;
}

}  // namespace gpu
}  // namespace whir
