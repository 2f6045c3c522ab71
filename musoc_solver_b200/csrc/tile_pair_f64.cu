// Two-column tile pass (tile_pair.cuh) on vectors of type double.
#include <algorithm>
#include <array>
#include <map>
#include <mutex>
#include <type_traits>

#include "tile_pair.cuh"

namespace sevp {

template <>
int tile_pair_launch<double>(const PairLaunch<double> &L) {
  return tile_pair_launch_any<double>(L);
}

template <>
int tile_pair_resident<double>(const TileGeom &tg, long long &warps) {
  return tile_pair_resident_any<double>(tg, warps);
}

}  // namespace sevp
