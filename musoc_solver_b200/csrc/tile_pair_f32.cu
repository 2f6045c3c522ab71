// Two-column tile pass (tile_pair.cuh) on vectors of type float.
#include <algorithm>
#include <array>
#include <map>
#include <mutex>
#include <type_traits>

#include "tile_pair.cuh"

namespace sevp {

template <>
int tile_pair_launch<float>(const PairLaunch<float> &L) {
  return tile_pair_launch_any<float>(L);
}

template <>
int tile_pair_resident<float>(const TileGeom &tg, long long &warps) {
  return tile_pair_resident_any<float>(tg, warps);
}

}  // namespace sevp
