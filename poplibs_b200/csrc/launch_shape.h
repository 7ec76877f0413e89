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

}  // namespace plb
