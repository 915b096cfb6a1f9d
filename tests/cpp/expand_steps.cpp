// The split of an Expand into passes (expandStep) on one line of cells away from
// a surface.  In the passes written in place a cell may see the value that its
// neighbour has just taken: none does, every cell does, or some do.  All must
// end, at the width kept on the way and at the last, with the cells and values of
// one cycle after another.  No value defined by a pass may be one that an early cell
// takes below the pass's limit (the passes repeat such an Expand cycle by cycle).
// Surfaces on the grid (value 0), values within 1e-7 of it on the other side and
// values whose sums round at the limits are among the starts.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <limits>
#include <vector>

#include "vlsg_expand.h"

template <class T> static int line(T u, int start, int width, int keep, bool full, int early) {
  const T none = std::numeric_limits<T>::max();
  std::vector<T> ref(16, none), got(16, none);
  ref[0] = got[0] = u;
  for (size_t i = 1; full && ref[i - 1] + T(1) <= T(start) * T(0.5); ++i)
    ref[i] = got[i] = ref[i - 1] + T(1);
  for (int at = start; at < width;) {
    const int stop = at < keep ? keep : width;
    const vlsg::ExpandStep s = vlsg::expandStep(start, at, stop);
    if (s.cycles < 1 || at + s.cycles > stop) return std::printf("width missed\n");
    for (int c = 1; c <= s.cycles; ++c) { // one cycle after another
      const std::vector<T> old = ref;
      for (size_t i = 1; i < ref.size(); ++i)
        if (old[i] == none && old[i - 1] + T(1) <= T(at + c) * T(0.5)) ref[i] = old[i - 1] + T(1);
    }
    const T limit = T(at + s.cycles) * T(0.5);
    const std::vector<T> old = got;
    for (size_t i = 1; i < got.size(); ++i) {
      const T from = s.inPlace && (early == 1 || (early == 2 && std::rand() % 2)) ? got[i - 1] : old[i - 1];
      if (old[i] != none || !(from + T(1) <= limit)) continue;
      got[i] = from + T(1);
      const T next = got[i] + T(1);
      if (s.inPlace && (s.cycles == 2 ? next < limit : next <= limit))
        return std::printf("start %d at %d: %.9g feeds below %g\n", start, at, (double)got[i],
                           (double)limit);
    }
    at += s.cycles;
    if (at == stop && got != ref)
      return std::printf("start %d width %d: passes differ from cycles\n", start, at);
  }
  return 0;
}

template <class T> static int all() {
  std::vector<T> starts;
  for (double base : {0.0, 0.25, 0.5, 0.75, 1.0})
    for (int k = -40; k <= 40; ++k)
      for (double e : {std::ldexp(1.0, -std::numeric_limits<T>::digits - 2), 1e-12, 1e-30}) {
        const T u = T(base + k * e);
        if (u >= T(0) && u <= T(1)) starts.push_back(u);
      }
  for (double e : {1e-7, 5e-8, 1e-9, 1e-12, 1e-15}) starts.push_back(T(-e));
  std::srand(5);
  for (int k = 0; k < 2000; ++k) starts.push_back(T(std::rand() / (double)RAND_MAX));
  for (int start = 1; start <= 4; ++start)
    for (int width = start + 1; width <= 14; ++width)
      for (int keep : {0, 3, 4, 5})
        for (T u : starts)
          for (bool full : {false, true}) // only the surface's cells, or the whole band
            for (int early : {0, 1, 2})
              if (keep < width && (full || start < 4) && line<T>(u, start, width, keep, full, early))
                return 1;
  return 0;
}

int main() { return all<float>() || all<double>(); }
