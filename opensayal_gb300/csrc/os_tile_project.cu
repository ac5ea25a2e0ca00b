// os_tile_project.cu — the projection kernels of one strip height, OS_TILE_ROWS
// (a translation unit per height, so that they compile side by side).
#include "os_tile.cuh"

namespace osg {
template <>
ProjectKernel project_kernel<OS_TILE_ROWS>(bool pressure, bool aligned) {
  if (aligned)
    return pressure ? k_project_tiles<OS_TILE_ROWS, true, true>
                    : k_project_tiles<OS_TILE_ROWS, false, true>;
  return pressure ? k_project_tiles<OS_TILE_ROWS, true, false>
                  : k_project_tiles<OS_TILE_ROWS, false, false>;
}
}  // namespace osg
