// os_batch_plan.cuh — the device plan of a batch (see os_batch.cuh), and the
// tile kernels that walk it.
#pragma once

#include "os_tile.cuh"

namespace osg {

constexpr int kBatchMaxPasses = 128;  // blocked passes per phase (n <= 128 * K)

struct ScenarioDesc {
  Consts c;
  int storage;       // OS_STORAGE_F32, OS_STORAGE_F16 or OS_STORAGE_BF16
  int smoke_period;
  int smoke_on;      // enable_smoke && wind_tunnel.smoke != 0
  int diff_passes;   // blocked diffusion passes per step (0 when viscosity == 0)
  int proj_passes;   // blocked projection passes per step
  int diff_tiles_x, diff_tiles_y;  // tiles under the diffusion geometry
  int proj_tiles_x, proj_tiles_y;  // tiles under the projection geometry
  const StepParams* prm;
  void *u, *v, *ub, *vb, *s, *sb;
  const uint8_t* flags;
  const uint16_t* nbr;  // fluid neighbourhoods (samplers)
};

struct TileRef {
  int slot;
  int16_t tx, ty;
};

// Head of the device plan; the arrays follow at the given byte offsets.
struct PlanHeader {
  int members;
  int admits;     // (slot, steps) pairs in the admit list
  int64_t cells;  // cells over all members
  int off_desc;                       // ScenarioDesc[slots]
  int off_slot;                       // int[members]
  int off_cell_cum;                   // int64_t[members]: cells before member k
  int off_diff_tiles, off_proj_tiles; // TileRef[tiles of pass 0]
  int off_admit;                      // int2[admits]
  int diff_items[kBatchMaxPasses];    // tiles in diffusion pass p
  int proj_items[kBatchMaxPasses];    // tiles in projection pass p
};

template <class T>
__device__ __forceinline__ const T* plan_array(const PlanHeader* P, int off) {
  return reinterpret_cast<const T*>(reinterpret_cast<const char*>(P) + off);
}

// The batch's tile kernels: clusters of CTAs of so many strips that walk the
// tiles of one pass, two CTAs to an SM (three of the diffusion's), so that one
// loads and stores while the other sweeps.
constexpr int kBatchProjectRows = 6, kBatchProjectWarps = 6;
constexpr int kBatchDiffuseRows = 8, kBatchDiffuseWarps = 4;
using BatchTileKernel = void (*)(const PlanHeader*, const int*, int, int, const RegTile,
                                 const ResidentSync);
BatchTileKernel batch_project_kernel();
BatchTileKernel batch_diffuse_kernel();

}  // namespace osg
