// tile_ragged_refine.cu -- the kRingRagged kernels of tile.cuh, precision form (one
// translation unit per mode and form, so that they compile in parallel).
#include "tile.cuh"

namespace cupic {
const void *tile_kernel_ragged_refine(int r) {
  return reinterpret_cast<const void *>(tile::pick<tile::kRingRagged, true>(r));
}
}  // namespace cupic
