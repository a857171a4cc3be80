// tune_pick.h - the autotuners' choice among measured candidates.
#pragma once
#include <cstddef>
#include <vector>

namespace csmv {

// The fastest of the candidates that were measured again (their numbers in `again`) by their
// median times `ms` (1e30 where a run failed). Equal times, which the timer's step of 32 ns makes
// now and then, go to the lowest number, not to whichever was faster in its first run.
inline size_t tune_pick(const std::vector<size_t>& again, const std::vector<double>& ms) {
  size_t best = again[0];
  for (size_t i : again)
    if (ms[i] < ms[best] || (ms[i] == ms[best] && i < best)) best = i;
  return best;
}

}  // namespace csmv
