// Two-column tile pass (tile_pair.cuh) on vectors of type float.
#include <algorithm>
#include <mutex>

#include "tile_pair.cuh"

namespace sevp {

template <>
int tile_pair_launch<float>(const PairLaunch<float> &L) {
  return tile_pair_launch_any<float>(L);
}

}  // namespace sevp
