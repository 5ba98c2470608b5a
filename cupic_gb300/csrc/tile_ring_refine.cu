// tile_ring_refine.cu -- the kRing kernels of tile.cuh, precision form (one
// translation unit per mode and form, so that they compile in parallel).
#include "tile.cuh"

namespace cupic {
const void *tile_kernel_ring_refine(int r) {
  return reinterpret_cast<const void *>(tile::pick<tile::kRing, true>(r));
}
}  // namespace cupic
