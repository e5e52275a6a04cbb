// How the narrow part of a Merkle tree is cut into launches (merkle.cu), as
// plain host rules.
#pragma once
#include <algorithm>

namespace whir {
namespace gpu {

// log2 of the first launch's subtrees for a narrow part of S <= 18 levels.  Up
// to 9 levels in two launches; from 10 on three, the first with up to 128 CTAs
// (one per SM), so that all levels but the first few have at most 8 nodes per
// CTA (a launch costs 2.5 us, a level 1.9 to 2.4 us on warps and 4.2 on
// quads; 11 levels: 31.6 us in three launches, 34.7 in two).  A CTA starts
// with at most 512 nodes, so at least S - 9 and at most 9; a tuned split
// (TreeTune) moves the default by one within those.
inline int tree_first_split(int S, int split) {
  const int lo = std::max(S - 9, 0), hi = std::min(S, 9);
  const int g = S <= 5 ? 0 : S <= 9 ? S / 2 : std::min(7, S - 4);
  return std::min(std::max(std::min(std::max(g, lo), hi) + split, lo), hi);
}

// Tunings taken: a threshold of 2^10 to 2^18 nodes and a split that moves the
// default by one at most.  18 narrow levels leave no fewer than 2^9 subtrees,
// and asking for fewer is refused; elsewhere a split that cannot move is as 0.
inline bool tree_tune_ok(int log_h, int wide_log, int split) {
  return wide_log >= 10 && wide_log <= 18 && split >= -1 && split <= 1 &&
         std::min(log_h, wide_log) - split <= 18;
}

}  // namespace gpu
}  // namespace whir
