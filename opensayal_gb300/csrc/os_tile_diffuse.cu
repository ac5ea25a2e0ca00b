// os_tile_diffuse.cu — the diffusion kernel of one strip height, OS_TILE_ROWS.
#include "os_tile.cuh"

namespace osg {
template <>
DiffuseKernel diffuse_kernel<OS_TILE_ROWS>(bool aligned) {
  return aligned ? k_diffuse_tiles<OS_TILE_ROWS, true> : k_diffuse_tiles<OS_TILE_ROWS, false>;
}
}  // namespace osg
