// tile_halo_refine.cu -- the kHalo kernels of tile.cuh, precision form (one
// translation unit per mode and form, so that they compile in parallel).
#include "tile.cuh"

namespace cupic {
const void *tile_kernel_halo_refine(int r) {
  return reinterpret_cast<const void *>(tile::pick<tile::kHalo, true>(r));
}
}  // namespace cupic
