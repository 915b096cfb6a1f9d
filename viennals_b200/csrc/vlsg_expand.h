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
// zero; in FP32 also where adding 1 rounds down to L) or miss it: L is the largest
// value of the pass, and the cell has no smaller one to take, so a cell that
// misses it takes L in the next pass.  After a pass of two cycles (limits L - 1/2,
// L) such cells may therefore be one pass late, after one of a single cycle
// (limit L + 1/2, where L + 1 is too large) none is left: an Expand ends with a
// pass of one cycle, and so does the part of it whose result is kept (`width`).
// A value below L - 1 would serve a neighbour below L.  In a band that is complete
// up to limit l, new values are above l, so two cycles (L = l + 1) give none.  The
// bands an Expand starts from are not complete: a rebuild leaves cells undefined
// next to a value within 1e-7 of 0, one cell in ten million (1 - 1e-7 and
// 2 - 1e-7 within the limit 2).  So the first pass is one cycle.  From width 3
// on (the rebuild for StencilLocalLaxFriedrichs) that cycle itself would meet
// such values and is logged, and the band is complete after the second.
struct ExpandStep {
  int cycles;
  bool inPlace;
};
inline ExpandStep expandStep(int start, int at, int width) {
  if (at == start) return {1, start < 3};
  const int complete = start < 3 ? start + 1 : start + 2;
  return {at >= complete && width - at >= 3 ? 2 : 1, true};
}

} // namespace vlsg
