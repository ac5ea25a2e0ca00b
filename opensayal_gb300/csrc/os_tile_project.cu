// os_tile_project.cu — the projection kernels of one strip height, OS_TILE_ROWS
// (a translation unit per height, so that they compile side by side).
#include "os_tile.cuh"

namespace osg {
template <>
ProjectKernel project_kernel<OS_TILE_ROWS>(bool pressure) {
  return pressure ? k_project_tiles<OS_TILE_ROWS, true> : k_project_tiles<OS_TILE_ROWS, false>;
}
}  // namespace osg
