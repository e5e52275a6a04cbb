// Launch shapes of the kernels that form their own eq tables (sumcheck.cu),
// as plain host rules.
#pragma once

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
// kernel alone takes 17.3 us against 3.7 + 12.9, 2^20 28 / 26 / 28).
inline int compress_hi_point_low(int k, int ks) {
  const int kz = k - ks, most = k >= 20 ? 10 : 8;
  return ks >= 2 && k >= 12 ? 12 - ks : kz < most ? kz : most;
}

}  // namespace gpu
}  // namespace whir
