// Launch shapes of the kernels that form their own eq tables (sumcheck.cu),
// as plain host rules.
#pragma once
#include <stddef.h>

#include "gpu_shape.h"

namespace whir {
namespace gpu {

// log2 of the rows of a block of compress_hi_point over 2^k words with 2^ks
// kept columns.  Blocks of 4096 words where the polynomial has them: the
// pipelined kernel.  Below 4 columns those would take a low table of more than
// 2^10 entries; there a thread multiplies its share of a block into one
// extension product, so blocks are as long as the table allows from 2^20 words
// on, and short before, so that a small polynomial has several CTAs (us a
// call, 2^8 rows / 2^10 / a table kernel and 2^10: one column, 2^24 words 152 /
// 65 / 69, 2^22 54 / 39 / 40, 2^20 30 / 26 / 28, 2^18 26 / 26 / 28, 2^12 20 / 27
// / 28; two columns, 2^24 113 / 54 / 56, 2^22 51 / 32 to 38 / 32, where the
// kernel alone takes 17.3 us against 3.7 + 12.9, 2^20 28 / 26 / 28).  So are
// those of 2^29 words and more with 16 columns or more (us, 4096 words / 2^10
// rows: 2^29 with 16 605 / 582, with 256 607 / 555, 2^30 with 64 1183 / 1060;
// with 8 606 / 627, 2^28 with 256 321 / 334).
inline int compress_hi_point_low(int k, int ks) {
  const int kz = k - ks, most = k >= 20 ? 10 : 8;
  if (ks >= 2 && k >= 12 && (k < 29 || ks < 4)) return 12 - ks;
  return kz < most ? kz : most;
}


// A launch of `ctas` CTAs with `smem` bytes of shared memory each.
struct PointLaunch {
  unsigned ctas;
  size_t smem;
};
// n_hi blocks over `usual` CTAs, each with `fixed` bytes and 16 for the high
// entry of each of its blocks: more CTAs where 47 KB (a kernel's own static
// words fit beside them) would not hold those.
inline PointLaunch point_launch(size_t n_hi, size_t usual, size_t fixed) {
  const size_t most = (47 * 1024 - fixed) / 16, need = (n_hi + most - 1) / most;
  const size_t cap = usual > need ? usual : need, ctas = n_hi < cap ? n_hi : cap;
  return {(unsigned)ctas, fixed + 16 * ((n_hi + ctas - 1) / ctas)};
}
// the factors of the low table (sumcheck.cu: eq_prologue)
constexpr size_t POINT_FACTORS = 64 * 16;
// compress_hi_point: about four CTAs per SM (three of the pipelined kernel, whose
// blocks are 4096 words); the low table and 2^ks columns' sums
inline PointLaunch compress_hi_point_launch(int k, int ks) {
  const int s_lo = compress_hi_point_low(k, ks);
  return point_launch((size_t)1 << (k - ks - s_lo), (size_t)SMS * (ks + s_lo == 12 ? 3 : 4),
                      ((size_t)16 << s_lo) + ((size_t)32 << ks) + POINT_FACTORS);
}
// eval_ext_point: blocks of 2^8 entries, eight CTAs per SM
inline PointLaunch eval_ext_point_launch(int k) {
  return point_launch((size_t)1 << (k < 8 ? 0 : k - 8), (size_t)SMS * 8, POINT_FACTORS);
}

}  // namespace gpu
}  // namespace whir
