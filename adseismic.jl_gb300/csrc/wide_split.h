// wide_split.h -- where the larger FP32 acoustic plans cut a shot into its undamped
// rectangle and the damped bands around it.  Host code without CUDA.
#pragma once

#include <vector>

namespace ads {

// Damped indices 1..n of a profile x[0..n+1] (nonzero there or beside it): the leading and
// trailing runs, or all of them where there are others between.
inline void damped_runs(const std::vector<double>& x, int n, int& lead, int& trail) {
  auto near = [&](int i) { return x[i - 1] != 0.0 || x[i] != 0.0 || x[i + 1] != 0.0; };
  lead = trail = 0;
  while (lead < n && near(lead + 1)) lead++;
  while (trail < n - lead && near(n - trail)) trail++;
  for (int i = lead + 1; i <= n - trail; i++)
    if (near(i)) lead = n, trail = 0;
}

// Columns [jl, jr) of the undamped rectangle of ny columns, nl and nr of them damped at
// either end (none where jr <= jl).  jl - 1 is a multiple of 64, jr - 1 one of four.  The
// right profile's 64-column strips end at column ny; their first column moves up to the
// next such column where their undamped ones allow it, else down (the strip that is then
// left over at the end has three columns at most).
inline void wide_columns(int ny, int nl, int nr, int& jl, int& jr) {
  jl = (nl + 63) / 64 * 64 + 1;
  jr = ny - (nr + 63) / 64 * 64 + 1;
  const int over = ((jr - 1) % 4 + 4) % 4;
  if (nr > 0 && over > 0 && jr + 4 - over <= ny - nr + 1) jr += 4 - over;
  else jr -= over;
}

}  // namespace ads
