// os_tile_batch.cu — the tile phases of a batch: one launch per pass, whose
// clusters walk the tiles of all members with that many passes. A tile is taken
// as k_project_tiles and k_diffuse_tiles take it, one pass at a time.
//
// Bound by the sweeps' instructions and by the faces' way from strip to strip;
// the loads and stores of one tile run beside the sweeps of the other on the
// SM. 21 tunnels of 128 to 1024 cells a side (6.85 M cells in all): a step
// takes 2004 us, and took 2968 us with tiles held in shared memory; 6 tunnels
// of mixed storage 1978 us, and 3378 us.
#include "os_batch_plan.cuh"

namespace osg {
namespace {

// A tile's faces out after a pass. Which tile and whose is read anew (kept across
// the sweeps it costs registers that their faces need).
template <int R>
__device__ __forceinline__ void tile_done(float (&u)[R][8], float (&v)[R][8],
                                          const TileRef* tiles, const ScenarioDesc* descs, int it,
                                          int pass, const RegTile& g, char* smem) {
  asm volatile("" : "+r"(it));
  const TileRef t = tiles[it];
  const ScenarioDesc& d = descs[t.slot];
  const int W = d.c.W, H = d.c.H;
  const int iu = (d.diff_passes + pass) & 1, iv = pass & 1;
  const Patch P = patch_at(TilePlace{t.tx, t.ty, d.proj_tiles_x, d.proj_tiles_y}, g, R, W, H);
  float* const stage = quads_aligned(W, g.halo) ? nullptr : stage_of(smem, g);
  if (!P.idle)
    faces_out<R>(u, v, iu ? d.u : d.ub, iv ? d.v : d.vb, d.storage, P, W, H, stage,
                 pass + 1 == d.proj_passes);
}

// Two CTAs of six warps with 168 registers fill an SM's register file: three
// warps to a scheduler hide the faces' way better than two of four warps with
// 255 (2079 us against 2188 us for the 21 tunnels above).
__global__ void __launch_bounds__(32 * kBatchProjectWarps, 2)
k_batch_project_tiles(const PlanHeader* __restrict__ plan, const int* __restrict__ remaining,
                      int pass, int K, const RegTile g, const ResidentSync sync) {
  constexpr int R = kBatchProjectRows;
  extern __shared__ __align__(16) char tile_smem[];
  const ProjSmem sm = project_smem_of(tile_smem, g.warps * R, g.warps, false);
  Link<4> link = open_link<4>(tile_smem, patch_at(TilePlace{0, 0, 1, 1}, g, R, 1, 1), g);
  cluster_arrive();
  pdl_entry();
  const int items = plan->proj_items[pass];
  const TileRef* tiles = plan_array<TileRef>(plan, plan->off_proj_tiles);
  const ScenarioDesc* descs = plan_array<ScenarioDesc>(plan, plan->off_desc);
  cluster_wait();
  if (!clusters_of(g.cluster, sync)) return;
  unsigned message = 0;
#pragma unroll 1
  for (int it = blockIdx.x / g.cluster; it < items && !link.lost;
       it += gridDim.x / g.cluster) {
    const TileRef t = tiles[it];
    if (remaining[t.slot] == 0) continue;  // the same for the whole cluster
    const ScenarioDesc& d = descs[t.slot];
    const Consts c = d.c;
    const int W = c.W, H = c.H;
    const TilePlace place{t.tx, t.ty, d.proj_tiles_x, d.proj_tiles_y};
    const int sweeps = min(K, c.n - pass * K);
    const int iu = (d.diff_passes + pass) & 1, iv = pass & 1;
    float* const stage = quads_aligned(W, g.halo) ? nullptr : stage_of(tile_smem, g);
    float u[R][8], v[R][8], vt[8];
#pragma unroll
    for (int r = 0; r < R; r++)
#pragma unroll
      for (int q = 0; q < 8; q++) u[r][q] = v[r][q] = 0.0f;
#pragma unroll
    for (int q = 0; q < 8; q++) vt[q] = 0.0f;
    ProjLane L;
    int cell0;
    bool down;
    {
      const Patch P = patch_at(place, g, R, W, H);
      cell0 = P.yl * 64 + P.lane;
      down = P.down;
      flags_in<R>(d.flags, P, sm, W, H, !stage, L);
      const void* vi = iv ? d.vb : d.v;
      if (!P.idle)
        on_cells(d.storage, [&](auto io) {
          patch_in<R>(io, u, iu ? d.ub : d.u, P, W, H, stage);
          patch_in<R>(io, v, vi, P, W, H, stage);
          if (P.up) row_in(io, vt, vi, P, P.y0 + R, W, H, stage);
        });
      if (zeros_change<R>(u, v, vt, L)) {
        L.full = false;
        flags_late(d.flags, P, sm, W, H, R);
      }
    }
    tile_sweeps<false, R>(u, v, vt, L, sm, link, sync, cell0, down, c, 0.0f, sweeps, message);
    message += project_messages(sweeps);
    tile_done<R>(u, v, tiles, descs, it, pass, g, tile_smem);
  }
  cluster_arrive();  // no CTA leaves while another may still send to it
  cluster_wait();
}

__global__ void __launch_bounds__(32 * kBatchDiffuseWarps, 3)
k_batch_diffuse_tiles(const PlanHeader* __restrict__ plan, const int* __restrict__ remaining,
                      int pass, int K, const RegTile g, const ResidentSync sync) {
  constexpr int R = kBatchDiffuseRows;
  extern __shared__ __align__(16) char tile_smem[];
  Link<8> link = open_link<8>(tile_smem, patch_at(TilePlace{0, 0, 1, 1}, g, R, 1, 1), g);
  cluster_arrive();
  pdl_entry();
  const int items = plan->diff_items[pass];
  const TileRef* tiles = plan_array<TileRef>(plan, plan->off_diff_tiles);
  const ScenarioDesc* descs = plan_array<ScenarioDesc>(plan, plan->off_desc);
  cluster_wait();
  if (!clusters_of(g.cluster, sync)) return;
  unsigned message = 0;
#pragma unroll 1
  for (int it = blockIdx.x / g.cluster; it < items && !link.lost;
       it += gridDim.x / g.cluster) {
    const TileRef t = tiles[it];
    if (remaining[t.slot] == 0) continue;  // the same for the whole cluster
    const ScenarioDesc& d = descs[t.slot];
    const int W = d.c.W, H = d.c.H;
    const TilePlace place{t.tx, t.ty, d.diff_tiles_x, d.diff_tiles_y};
    const int sweeps = min(K, d.c.n - pass * K);
    float* const stage = quads_aligned(W, g.halo) ? nullptr : stage_of(tile_smem, g);
    float u[R][8];
#pragma unroll
    for (int r = 0; r < R; r++)
#pragma unroll
      for (int q = 0; q < 8; q++) u[r][q] = 0.0f;
    DiffLane L;
    {
      const Patch P = patch_at(place, g, R, W, H);
      L = diff_lane(P, R, W, H);
      if (!P.idle)
        on_cells(d.storage,
                 [&](auto io) { patch_in<R>(io, u, pass & 1 ? d.ub : d.u, P, W, H, stage); });
    }
    jacobi_sweeps<R>(u, L, link, sync, diffusion_coeff<float>(d.c, d.prm->dt), sweeps, message);
    message += sweeps;
    const Patch P = patch_at(place, g, R, W, H);
    float* const out = quads_aligned(W, g.halo) ? nullptr : stage_of(tile_smem, g);
    if (!P.idle)
      on_cells(d.storage, [&](auto io) {
        patch_out<R>(io, u, pass & 1 ? d.u : d.ub, P, rows_in(P.y0, R, P.oy0, P.oy1), W, H, out);
      });
  }
  cluster_arrive();
  cluster_wait();
}

}  // namespace

BatchTileKernel batch_project_kernel() { return k_batch_project_tiles; }
BatchTileKernel batch_diffuse_kernel() { return k_batch_diffuse_tiles; }

}  // namespace osg
