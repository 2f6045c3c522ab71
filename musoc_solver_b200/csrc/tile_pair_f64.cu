// Two-column tile pass (tile_pair.cuh) on vectors of type double.
#include <algorithm>
#include <mutex>

#include "tile_pair.cuh"

namespace sevp {

template <>
int tile_pair_launch<double>(const PairLaunch<double> &L) {
  return tile_pair_launch_any<double>(L);
}

}  // namespace sevp
