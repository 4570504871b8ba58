// When the host looks at the state of a GMRES cycle (solve.cu), host arithmetic only.
#pragma once

#include <algorithm>
#include <cmath>
#include <limits>

namespace cfd {

// Steps until a residual that falls by `rate` a step passes the threshold, at least
// one; without end where it does not fall or the threshold is zero.
inline double gmres_steps_left(double rn, double threshold, double rate) {
  if (!(rn > threshold)) return 1.0;
  if (!(threshold > 0.0) || !(rate > 0.0 && rate < 1.0)) return std::numeric_limits<double>::infinity();
  return std::max(1.0, std::ceil(std::log(threshold / rn) / std::log(rate)));
}

// The step of a cycle of m to look after next, counted from its start, for a residual
// rn after `done` of its steps; m (the cycle's own look) where nothing ends it sooner.
inline int gmres_next_look(int done, int m, double rn, double threshold, double rate) {
  return (int)std::min<double>(m, done + gmres_steps_left(rn, threshold, rate));
}

}  // namespace cfd
