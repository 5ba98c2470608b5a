// tile_halo.cu -- the kHalo kernels of tile.cuh (one
// translation unit per mode and form, so that they compile in parallel).
#include "tile.cuh"

namespace cupic {
const void *tile_kernel_halo(int r) {
  return reinterpret_cast<const void *>(tile::pick<tile::kHalo, false>(r));
}
}  // namespace cupic
