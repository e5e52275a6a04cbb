// Poseidon2's linear layers as matrices of small integers for the tensor
// cores (p2_tensor.cuh runs them; this file is their shape and their host
// construction).
//
// A field word is four bytes, and a linear map of words is an integer matrix
// over those bytes.  A byte b sits in a half as the bit pattern 0x00bb, which
// is the number b 2^-24, so the operand needs no conversion.
//  - A light layer (entries 1..6 of the light MDS) is taken on the low and
//    the high 16 bits of the words apart: per output word two sums of at
//    most 49 (width 24) or 35 (width 16) times 65535.
//  - The internal rounds between two S-boxes on word 0 are linear, so word 0
//    before round r is one linear form of the S-box outputs before it (those
//    of the fourth external round, and the earlier internal ones), and so is
//    every word after the last round.  The forms' coefficients are field
//    elements; each byte of an input word gets its own coefficient (times
//    2^(8a)), taken in (-p/2, p/2) and written as four signed digits to the
//    base 256, which become four columns.
// The accumulators of all columns stay exact: every product is a multiple of
// one unit, and the sums lie between 2^23 and 2^24 units, where a float's
// low 23 bits are an integer.  The 2^23 and the column's constant (round
// constants, and offsets that keep the sums non-negative) come from three
// operand slots with fixed values.
#pragma once
#include <stdint.h>

#include <vector>

#include "kb.cuh"

namespace whir {
namespace gpu {

// Table layout and operand columns of the width-W permutation.  A step is
// one K = 16 matrix instruction: N rows of 16 halves, stored as 8-row by
// 16-byte core matrices, [K half][row group][row][8 halves].
template <int W>
struct P2Mat {
  static_assert(W == 16 || W == 24, "Poseidon2 width");
  static constexpr int RP = W == 16 ? 20 : 23;
  static constexpr int KX = W / 8;              // steps over the low (or high) byte pairs
  static constexpr int NL = W == 16 ? 16 : 32;  // columns of one half of a light layer
  static constexpr int BLK = W == 16 ? 4 : 6;   // internal rounds per block
  static constexpr int NBLK = (RP + BLK - 1) / BLK;
  static constexpr int NB = W == 16 ? 16 : 32;  // columns of a block's forms, 4 each
  static constexpr int NCST = 8;                // light layers (initial, after rounds 0-2, 4-7)
  static constexpr int TILES = W == 16 ? 5 : 4;  // 128-row tiles per CTA
  static constexpr int FW = W == 16 ? 4 : 8;    // words per final-state chunk
  static constexpr int NFIN = W / FW;
  static constexpr int YSTEPS = 5;              // steps over internal outputs 0..19
  // tables, in bytes from the start
  KB_HD static constexpr int step_bytes(int n) { return n * 32; }
  // steps over the outputs of the blocks before block q
  KB_HD static constexpr int blk_ysteps(int q) { return (BLK * q + 3) / 4; }
  static constexpr int fin_steps = 1 + 2 * KX + YSTEPS;
  static constexpr int ext_off = 0;
  static constexpr int cst_off = KX * step_bytes(NL);
  static constexpr int blk0_off = cst_off + NCST * step_bytes(2 * NL);
  KB_HD static constexpr int blk_off(int q) {
    int off = blk0_off;
    for (int i = 0; i < q; i++) off += (1 + 2 * KX + blk_ysteps(i)) * step_bytes(NB);
    return off;
  }
  KB_HD static constexpr int fin_off(int c) {
    return blk_off(NBLK) + c * fin_steps * step_bytes(4 * FW);
  }
  static constexpr int bytes = fin_off(NFIN);
  // tensor-memory columns of one 128-row tile: the W words' low
  // byte pairs, their high ones, the constant slots with the internal
  // outputs 20.. (2 columns a word, constants in the last two), the internal
  // outputs 0..19, the sums.  A light layer's 2 NL sums overlie the internal
  // outputs' columns, which are not live then.
  static constexpr int COL_H = W;
  static constexpr int COL_C = 2 * W;
  static constexpr int COL_Y = COL_C + 8;
  static constexpr int COL_D = COL_Y + 8 * YSTEPS;
  static constexpr int COLS = COL_D + (4 * FW > NB ? 4 * FW : NB);
  static constexpr int COL_DX = COLS - 2 * NL;
  static_assert(COL_DX >= COL_Y && TILES * COLS <= 512, "tile columns");
};

// exponent bits of the sums: 2^23 units of 2^-19 (light layers) or 2^-16
constexpr uint32_t P2M_E_LIGHT = 0x41800000u;  // 16.0f
constexpr uint32_t P2M_E_FORM = 0x43000000u;   // 128.0f
// fixed operand values of the constant slots: 1, 2^-8, 2^-16, 0 (halves)
constexpr uint32_t P2M_CONST0 = 0x1c003c00u;
constexpr uint32_t P2M_CONST1 = 0x00000100u;

struct P2Tables {
  std::vector<uint16_t> halves;  // P2Mat<W>::bytes / 2
  // Montgomery words, centred: weight of an internal output on word 0 two,
  // three, .. rounds later (within a block); one round later it is -1
  int32_t tri[4];
};
// Built once per width from the permutation's constants; throws if a sum
// could leave its exact range.
const P2Tables &p2_tables(int width);

}  // namespace gpu
}  // namespace whir
