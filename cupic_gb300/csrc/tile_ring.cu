// tile_ring.cu -- the kRing kernels of tile.cuh (one
// translation unit per mode and form, so that they compile in parallel).
#include "tile.cuh"

namespace cupic {
const void *tile_kernel_ring(int r) {
  return reinterpret_cast<const void *>(tile::pick<tile::kRing, false>(r));
}
}  // namespace cupic
