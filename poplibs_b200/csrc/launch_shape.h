// Host-side arithmetic of launch shapes.
#pragma once

#include <algorithm>

namespace plb {

// Clusters of a persistent grid that wants `wanted` (a multiple of `multiple`) where
// `resident` fit the device at once: as many as fit in whole multiples, and one
// multiple where not even that fits.  Clusters do not wait for one another, so those
// that do not fit run after the others.
inline int clusterCount(int wanted, int resident, int multiple) {
  const int fit = std::max(1, std::min(wanted, resident));
  return std::max(multiple, fit / multiple * multiple);
}

// Pipeline stages where two threads issue the tensor-core instructions of alternate tiles
// of `steps` stages each, of the `stages` that fit; 0 where they cannot.  A thread waits for
// the parity of a stage's fill, which tells it from the fill before only if it has seen
// that one complete.  So the stages are a whole number of pairs of tiles: each thread then
// has stages of its own.  (With four stages and tiles of three, the second thread's second
// step took the first tile's stage for filled again before its first copy had arrived,
// and the pipeline went out of step; such a layer ended with a launch failure.)
inline int dualIssueStages(int stages, int steps) { return stages / (2 * steps) * (2 * steps); }

}  // namespace plb
