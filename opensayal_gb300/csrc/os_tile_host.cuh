// os_tile_host.cuh — which tiles a grid takes, and the launches of the phases on
// tiles in registers (os_tile.cuh).
#pragma once

#include "os_tile.cuh"

namespace osg {

template <> ProjectKernel project_kernel<2>(bool, bool);
template <> ProjectKernel project_kernel<4>(bool, bool);
template <> ProjectKernel project_kernel<6>(bool, bool);
template <> ProjectKernel project_kernel<8>(bool, bool);
template <> ProjectKernel project_kernel<10>(bool, bool);
template <> DiffuseKernel diffuse_kernel<2>(bool);
template <> DiffuseKernel diffuse_kernel<4>(bool);
template <> DiffuseKernel diffuse_kernel<6>(bool);
template <> DiffuseKernel diffuse_kernel<8>(bool);
template <> DiffuseKernel diffuse_kernel<12>(bool);

inline ProjectKernel project_kernel_of(int R, bool pressure, bool aligned) {
  switch (R) {
    case 2: return project_kernel<2>(pressure, aligned);
    case 4: return project_kernel<4>(pressure, aligned);
    case 6: return project_kernel<6>(pressure, aligned);
    case 8: return project_kernel<8>(pressure, aligned);
    default: return project_kernel<10>(pressure, aligned);
  }
}
inline DiffuseKernel diffuse_kernel_of(int R, bool aligned) {
  switch (R) {
    case 2: return diffuse_kernel<2>(aligned);
    case 4: return diffuse_kernel<4>(aligned);
    case 6: return diffuse_kernel<6>(aligned);
    case 8: return diffuse_kernel<8>(aligned);
    default: return diffuse_kernel<12>(aligned);
  }
}

inline RegTile reg_tile(int W, int H, int halo, int R, int warps, int cluster) {
  RegTile g{};
  g.R = R, g.warps = warps, g.cluster = cluster;
  g.RH = R * warps * cluster;
  const bool one = W <= kTileW && H <= g.RH;
  g.halo = one ? 0 : halo;  // a tile that is the whole grid has no halo
  g.TX = kTileW - 2 * g.halo;
  g.TY = g.RH - 2 * g.halo;
  g.tiles_x = W <= kTileW ? 1 : (W - 2 * halo + g.TX - 1) / g.TX;
  if (H <= g.RH)
    g.tiles_y = 1;
  else
    g.tiles_y = g.TY >= 2 ? (H - 2 * halo + g.TY - 1) / g.TY : 0;  // 0: does not cover the grid
  return g;
}

// CTAs per cluster that tiles are tried with. At least 2: the strips' messages
// are cluster instructions, which a launch without clusters refuses as illegal.
// More than 8 are beyond the portable size; how many clusters of a size fit
// the GPU at once depends on how its SMs are grouped (on GB300: 152 CTAs in
// clusters of 2, 144 of 4, 138 of 6, 120 of 8, 130 of 10, 96 of 12, 112 of 16).
constexpr int kClusters[] = {2, 4, 6, 8, 10, 12, 16};

// CTAs of a tile kernel that an SM holds, by the registers that its launch
// bounds allow it, its shared memory and its threads.
inline int ctas_per_sm(int R, int warps, bool projection, size_t smem) {
  const int regs = R <= 4 ? 128 : R <= (projection ? 6 : 8) ? 168 : 256;
  const int by_regs = 65536 / (regs * 32 * warps), by_smem = (int)((228 << 10) / (smem + 1024));
  return std::max(1, std::min({by_regs, by_smem, 64 / warps, 4}));
}

// Clusters of `cluster` CTAs that are resident together with `ctas` CTAs to an
// SM. An answer is kept; a query that fails is made again the next time.
inline int resident_clusters(int device, int cluster, int ctas) {
  static std::mutex mu;
  static std::map<std::tuple<int, int, int>, int> known;
  std::lock_guard<std::mutex> lock(mu);
  const auto key = std::make_tuple(device, cluster, ctas);
  auto it = known.find(key);
  if (it != known.end()) return it->second;
  const auto kernel = diffuse_kernel<2>(true);
  const size_t smem = (227 / ctas - 1) * 1024;  // as much as leaves room for no more CTAs
  int n = 0;
  cudaError_t e = allow_most(kernel);
  if (e == cudaSuccess) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cluster * sm_count(device));
    cfg.blockDim = dim3(128);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaOccupancyMaxActiveClusters(&n, kernel, &cfg);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  known[key] = n;
  return n;
}

// The tile that takes the least time by a model of n sweeps, `D` between
// exchanges or passes: issue slots on the fullest of the SM's four schedulers,
// the faces' way between CTAs of a cluster, and the region once in and out (or
// an exchange), in as many waves as the tiles take. With `resident` all tiles
// must be on the GPU together and be at least a halo wide and high (the ring
// then comes from adjacent tiles). Returns the modelled cycles, 0 when no tile
// covers the grid.
inline double choose_tile(int W, int H, int D, bool projection, bool pressure, bool resident,
                          int n, int device, RegTile* out) {
  double best = 0.0;
  const int halo = projection ? 2 * D : D;
  const int* heights = projection ? kProjectRows : kDiffuseRows;
  const int count = projection ? (int)std::size(kProjectRows) : (int)std::size(kDiffuseRows);
  for (int cluster : kClusters) {
    const int alone = resident_clusters(device, cluster, 1);
    if (alone < 1) continue;
    for (int k = 0; k < count; k++) {
      const int R = heights[k];
      const int most = projection ? project_max_warps(R) : diffuse_max_warps(R);
      for (int warps = 1; warps <= most; warps++) {
        RegTile g = reg_tile(W, H, halo, R, warps, cluster);
        if (g.tiles_y < 1) continue;
        const int64_t tiles = (int64_t)g.tiles_x * g.tiles_y;
        const bool one = tiles == 1;
        if (resident && (tiles > alone || (g.tiles_y > 1 && g.TY < halo) || g.TX < halo)) continue;
        const int rows = R * warps;
        g.smem = projection
                     ? project_tile_smem(rows, warps, pressure, g.halo, resident && !one)
                     : diffuse_tile_smem(rows, warps, g.halo, resident && !one);
        g.smem += stage_smem(W, g.halo, warps);
        if (g.smem + kStaticSmem > kMaxSmem) continue;
        // Pass by pass, several CTAs share an SM: over three waves or more they
        // drift apart, and one loads and stores beside the other's sweeps (in
        // fewer they do the same at the same time: 1920 x 1080 in passes of 8
        // sweeps took 170 us so, and 142 us with an SM to each CTA).
        int share = resident ? 1 : ctas_per_sm(R, warps, projection, g.smem);
        int fit = share > 1 ? resident_clusters(device, cluster, share) : alone;
        if (share > 1 && tiles <= 2 * fit) share = 1, fit = alone;
        if (fit < 1) continue;
        const int64_t waves = (tiles + fit - 1) / fit;
        // Cycles of a sweep: the slowest strip (one by the flags, or with kept
        // rows), the other strips of its scheduler, and the messages' way.
        const int others = (share * warps + 3) / 4 - 1;
        double sweep =
            projection ? 650.0 + (pressure ? 230.0 : 170.0) * R +
                             others * ((pressure ? 115.0 : 72.0) * R + 90.0)
                       : 450.0 + 130.0 * R + others * (50.0 * R + 60.0);
        // A round: the exchange of the rows and sides, or the region in and
        // out of memory.
        double trip = 5000.0 + share * rows * (projection ? 50.0 : 25.0);
        if (share > 1) trip *= 0.8;
        if (resident) {
          const int halo_rows = g.tiles_y > 1 ? std::min(2 * halo, rows) : 0;
          const double quads = 64.0 * halo_rows + rows * (halo / 2.0);
          // Fitted to the times of every tile that ten grids from 333 x 187 to
          // 1280 x 720 take (projection with and without the pressure,
          // diffusion; 10,000 times in all, within 5 to 7%). The choice is 1
          // to 2% behind the best of them in the mean and 9% at most; with the
          // terms of the passes above it was up to 28% (projection) and 48%
          // (diffusion) behind: four warps to a scheduler cost more than they
          // said, and the rows of an exchange less.
          sweep = !projection ? 360.0 + 140.0 * R + 280.0 * others
                  : pressure  ? 680.0 + (350.0 + 118.0 * others) * R
                              : 750.0 + (200.0 + 87.0 * others) * R;
          trip = !projection ? 3900.0 + 0.2 * quads
                 : pressure  ? 4000.0 + 0.85 * quads
                             : 4300.0 + 1.1 * quads;
        }
        const double rounds = resident ? (one ? 0 : (n + D - 1) / D - 1) : (n + D - 1) / D;
        const double cost = (double)waves * (n * sweep + rounds * trip);
        if (best == 0.0 || cost < best) {
          best = cost;
          *out = g;
        }
      }
    }
  }
  return best;
}

// A launch of all tiles: cooperative when its tiles wait on one another, else
// with programmatic stream serialisation where the handle uses it.
template <class Args>
inline cudaError_t launch_tiles(void (*kernel)(const Args), const Args& a, const RegTile& g,
                                bool cooperative, bool pdl, cudaStream_t st) {
  const cudaError_t e = allow_most(kernel);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(g.tiles_x * g.tiles_y * g.cluster);
  cfg.blockDim = dim3(32 * g.warps);
  cfg.dynamicSmemBytes = g.smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (g.cluster < 2) return cudaErrorInvalidConfiguration;
  attr[n].id = cudaLaunchAttributeClusterDimension;
  attr[n].val.clusterDim.x = g.cluster;
  attr[n].val.clusterDim.y = 1;
  attr[n++].val.clusterDim.z = 1;
  if (cooperative) {
    attr[n].id = cudaLaunchAttributeCooperative;
    attr[n++].val.cooperative = 1;
  } else if (pdl) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, a);
}

// The resident forms' tiles, all of one launch resident together, and the
// sweeps between their exchanges (n when one tile is the whole grid). block_k
// is not their depth: it says how often 16-bit fields are rounded. 0 when the
// grid does not fit.
inline int resident_tile(const os_handle* h, bool projection, RegTile* g) {
  const bool pressure = h->cfg.enable_pressure != 0;
  const int K = h->block_k, n = std::max(h->c.n, 1);
  if (K < 2 || K % (projection ? 2 : 4)) return 0;
  int depth = 0;
  double best = 0.0;
  for (int D : {2, 4, 6, 8, 12, 16, 20}) {  // halos in multiples of 4 cells
    if (!projection && D % 4) continue;
    RegTile t;
    const double cost = choose_tile(h->W, h->H, D, projection, pressure, true, n, h->cfg.device, &t);
    if (cost > 0.0 && (depth == 0 || cost < best)) {
      best = cost;
      depth = t.tiles_x * t.tiles_y == 1 ? n : D;
      *g = t;
    }
  }
  return depth;
}

// A phase's tile and the sweeps between its exchanges or passes, worked out
// once per form (the search takes some 50 us of host time). 0: none.
inline int phase_tile(os_handle* h, bool projection, int K, bool resident, RegTile* g) {
  TileChoice& t = h->tile_choice[projection ? 0 : 1];
  if (t.K != K || t.resident != resident) {
    t.K = K, t.resident = resident;
    if (resident)
      t.depth = resident_tile(h, projection, &t.tile);
    else
      t.depth = choose_tile(h->W, h->H, K, projection, projection && h->cfg.enable_pressure, false,
                            h->c.n, h->cfg.device, &t.tile) > 0.0
                    ? K
                    : 0;
  }
  *g = t.tile;
  return t.depth;
}

// The projection phase: one launch for all its passes (resident), or one per
// pass of block_k sweeps. `cur_u` / `cur_v` say which copy holds the live
// field (0: u, v; 1: ub, vb); each launch moves it to the other. `extrapolate`:
// the last pass applies the extrapolation that follows in a step. Returns the
// launches, or -1.
inline int enqueue_tiled_projection(os_handle* h, cudaStream_t st, int* cur_u, int* cur_v,
                                    bool zero_first, bool extrapolate) {
  const int K = h->block_k, n = h->c.n;
  if (n < 1) return 0;  // no sweeps, no tile to choose
  const bool pressure = h->cfg.enable_pressure != 0;
  ProjectArgs a{};
  void *const U[2] = {h->u, h->ub}, *const V[2] = {h->v, h->vb};
  a.storage = h->storage;
  a.p = h->p;
  a.flags = h->flags;
  a.c = h->c;
  a.prm = h->d_params;
  a.K = K;
  a.sync = ResidentSync{h->rflags, h->rpackets, h->rerr, h->d_host_rerr};
  const int passes = (n + K - 1) / K;
  int launches = 0;
  if (h->resident) {
    if (!(a.D = phase_tile(h, true, K, true, &a.g))) return -1;
    a.n = n;
    a.ui = U[*cur_u], a.uo = U[1 - *cur_u];
    a.vi = V[*cur_v], a.vo = V[1 - *cur_v];
    a.zero_pressure = zero_first;
    a.extrapolate = extrapolate;
    if (launch_tiles(project_kernel_of(a.g.R, pressure, quads_aligned(h->W, a.g.halo)), a, a.g,
                     n > a.D, h->pdl, st) != cudaSuccess)
      return -1;
    launches = 1;
  } else {
    if (projection_smem(2 + 4 * K, pressure) + kStaticSmem > kMaxSmem ||
        !(a.D = phase_tile(h, true, K, false, &a.g)))
      return -1;
    for (int p = 0; p < passes; p++, launches++) {
      a.n = std::min(K, n - p * K);
      const int cu = (*cur_u + p) & 1, cv = (*cur_v + p) & 1;
      a.ui = U[cu], a.uo = U[1 - cu];
      a.vi = V[cv], a.vo = V[1 - cv];
      a.zero_pressure = zero_first && p == 0;
      a.extrapolate = extrapolate && p == passes - 1;
      if (launch_tiles(project_kernel_of(a.g.R, pressure, quads_aligned(h->W, a.g.halo)), a, a.g,
                       false, h->pdl, st) != cudaSuccess)
        return -1;
    }
  }
  *cur_u = (*cur_u + launches) & 1;
  *cur_v = (*cur_v + launches) & 1;
  return launches;
}

// The diffusion phase in the same way, block_k sweeps per pass when resident,
// else diffusion_depth.
inline int enqueue_tiled_diffusion(os_handle* h, cudaStream_t st, int* cur_u) {
  const int K = h->resident_diff ? h->block_k : diffusion_depth(h), n = h->c.n;
  if (n < 1) return 0;
  DiffuseArgs a{};
  void* const U[2] = {h->u, h->ub};
  a.storage = h->storage;
  a.c = h->c;
  a.prm = h->d_params;
  a.K = K;
  a.sync = ResidentSync{h->dflags, h->dpackets, h->rerr, h->d_host_rerr};
  const int passes = (n + K - 1) / K;
  int launches = 0;
  if (h->resident_diff) {
    if (!(a.D = phase_tile(h, false, K, true, &a.g))) return -1;
    a.n = n;
    a.ui = U[*cur_u], a.uo = U[1 - *cur_u];
    if (launch_tiles(diffuse_kernel_of(a.g.R, quads_aligned(h->W, a.g.halo)), a, a.g, n > a.D,
                     h->pdl, st) != cudaSuccess)
      return -1;
    launches = 1;
  } else {
    if (!(a.D = phase_tile(h, false, K, false, &a.g))) return -1;
    for (int p = 0; p < passes; p++, launches++) {
      a.n = std::min(K, n - p * K);
      const int cu = (*cur_u + p) & 1;
      a.ui = U[cu], a.uo = U[1 - cu];
      if (launch_tiles(diffuse_kernel_of(a.g.R, quads_aligned(h->W, a.g.halo)), a, a.g, false,
                       h->pdl, st) != cudaSuccess)
        return -1;
    }
  }
  *cur_u = (*cur_u + launches) & 1;
  return launches;
}

// Device bytes of a resident phase's exchange numbers, and of its packets.
inline size_t resident_epoch_bytes(int sms) {
  return ((size_t)sms * sizeof(unsigned) + 255) / 256 * 256;
}
inline size_t resident_packet_bytes(int W, int H, int per_quad) {
  return (size_t)2 * packet_plane(W, H) * per_quad * sizeof(uint4);
}

// Failure-detection self-tests. A warp waits for a packet that nothing sends, so
// the wait must give up and report.
__global__ void k_wait_selftest(ResidentSync sync) {
  float a = 0.0f, b = 0.0f, c = 0.0f;
  bool again = true;
  for (int it = 0; again; it++) {
    const bool ok = packet_in(threadIdx.x == 0, sync.packets, a, b, c, 1u);
    again = !__all_sync(kAllLanes, ok) && poll_again(it, sync);
    again = __any_sync(kAllLanes, again);
  }
}

// The strip of the first of two CTAs takes part in `count` messages, and the
// second's sends none: the first wait must give up, and the others end with it.
// With a `cluster` that is not the launch's, it must report that and end at once.
__global__ void k_message_selftest(ResidentSync sync, int cluster, int count) {
  extern __shared__ __align__(16) char tile_smem[];
  RegTile g{};
  g.R = 2, g.warps = 1, g.cluster = 2, g.RH = 4;
  Link<4> link = open_link<4>(tile_smem, patch_at(TilePlace{0, 0, 1, 1}, g, g.R, 1, 1), g);
  cluster_arrive();
  cluster_wait();
  if (!clusters_of(cluster, sync)) return;
  if (blockIdx.x == 0) idle_messages(link, 0, count, sync);
  cluster_arrive();
  cluster_wait();
}

inline cudaError_t launch_message_selftest(const ResidentSync& sync, int cluster, int count) {
  cudaError_t e = allow_most(k_message_selftest);
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = 2;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2);
  cfg.blockDim = dim3(32);
  cfg.dynamicSmemBytes = inbox_bytes(4);
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_message_selftest, sync, cluster, count);
}

}  // namespace osg
