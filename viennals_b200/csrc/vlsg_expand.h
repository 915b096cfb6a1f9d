// vlsg_expand.h -- how an Expand (lsExpand.hpp:44-172) is split into band passes.
#pragma once

namespace vlsg {

// The next pass of an Expand that began at width `start` and has reached width
// `at`: one cycle or two, and whether its new values are written in place
// (kFrontierPass, vlsg_frontier.cuh).  A cycle to width w defines the undefined
// cells whose smallest neighbour + 1 is within its limit w / 2.
//
// A pass in place with limit L lets a cell see values that other cells of the
// pass have just taken.  It may take L from one of them (L - 1 next to an exact
// zero: 0, 1, 2; in FP32 also where adding 1 rounds down to L) or miss it: L is
// the largest value of the pass, and the cell has no smaller one to take, so a
// cell that misses it takes L in the next pass.  After a pass of two cycles
// (limits L - 1/2, L) such cells may therefore be one pass late, after one of a
// single cycle (limit L + 1/2, where L + 1 is too large) none is left: an
// Expand ends with a pass of one cycle, and so does the part of it whose result
// is kept (`width`).
// Starts of width 3 on may hold only the surface's cells (the rebuild for
// StencilLocalLaxFriedrichs), so that an exact zero gives 1 and 2 within the
// first cycle, which must define the 1 alone: that cycle is logged.
struct ExpandStep {
  int cycles;
  bool inPlace;
};
inline ExpandStep expandStep(int start, int at, int width) {
  if (at == start && start >= 3) return {1, false};
  return {width - at >= 3 ? 2 : 1, true};
}

} // namespace vlsg
