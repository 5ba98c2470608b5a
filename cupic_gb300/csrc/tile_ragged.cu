// tile_ragged.cu -- the kRingRagged kernels of tile.cuh (one
// translation unit per mode and form, so that they compile in parallel).
#include "tile.cuh"

namespace cupic {
const void *tile_kernel_ragged(int r) {
  return reinterpret_cast<const void *>(tile::pick<tile::kRingRagged, false>(r));
}
}  // namespace cupic
