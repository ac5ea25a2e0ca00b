// os_blocked.cuh — the tensor-copy form of the temporally blocked diffusion (an
// option; see os_tile.cuh for the form that is used otherwise), and what the
// blocked forms share on the host.
//
// A CTA owns a TX x TY tile of cells. It stages the tile plus a halo into
// shared memory, runs `sweeps` Jacobi sweeps there (apply_diffusion_at,
// src/fluid.cu:176-183), and writes back only the cells it owns. Validity
// shrinks by one cell per sweep, so K sweeps need a halo of K cells. Every
// update is the plain kernels' (and the reference's) expression in the same
// order, so a blocked pass gives the same bits as K per-sweep launches. Passes
// read one global copy and write the other (fields <-> buffers), so no CTA
// reads a neighbour's half-updated halo.
#pragma once

#include <cuda.h>  // CUtensorMap and its enums (types only; no driver-library link)

#include <algorithm>
#include <mutex>
#include <set>
#include <type_traits>
#include <utility>

namespace osg {

constexpr int kRegionW = 256;            // region width in cells
constexpr int kQuads = kRegionW / 4;     // 4-cell groups per region row
constexpr int kBlockThreads = 1024;

struct TileGeom {
  int halo;     // halo in cells on every side
  int TX, TY;   // owned tile
  int RH;       // region rows
  int tiles_x, tiles_y;
  size_t smem;  // dynamic shared memory per CTA
};

// The shared memory a region of RH rows would take with its faces (and
// pressure) and flags staged there: it bounds the depths that are accepted.
__host__ __device__ inline size_t projection_smem(int RH, bool pressure) {
  const size_t plane = (size_t)RH * (kRegionW / 2) + 16;  // words per column parity
  return plane * (pressure ? 6 : 4) * 4 + 2 * ((size_t)RH * (kRegionW / 2) + 64);
}

__host__ __device__ inline size_t diffusion_smem(int RH) {
  return 2 * ((size_t)RH * kRegionW + 16) * 4;
}

// Four consecutive stored values as FP32 (one vector load).
__device__ __forceinline__ float4 vec4_to_f32(const float* p) {
  return __ldg(reinterpret_cast<const float4*>(p));
}
__device__ __forceinline__ float4 vec4_to_f32(const __half* p) {
  const uint2 r = __ldg(reinterpret_cast<const uint2*>(p));
  const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&r.x));
  const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&r.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ float4 vec4_to_f32(const __nv_bfloat16* p) {
  const uint2 r = __ldg(reinterpret_cast<const uint2*>(p));
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.y));
  return make_float4(a.x, a.y, b.x, b.y);
}

// One column's run of Jacobi updates, rows e0, e0 + rs, ... (n of them), from
// A into B. The buffers never overlap, so the loads of later rows may be
// issued ahead of earlier rows' stores.
__device__ __forceinline__ void diff_column(const float* __restrict__ A, float* __restrict__ B,
                                            int e0, int rs, int n, float a, float den) {
  float down = A[e0 - rs];
  float centre = A[e0];
  int e = e0;
#pragma unroll 4
  for (int t = 0; t < n; t++, e += rs) {
    const float up = A[e + rs];
    // src/fluid.cu:178-182: neighbours (i-1, j), (i+1, j), (i, j-1), (i, j+1)
    B[e] = fma_rn(a, A[e - 1] + A[e + 1] + down + up, centre) / den;
    down = centre;
    centre = up;
  }
}

// `sweeps` Jacobi sweeps on the staged region, A -> B -> A ...; on return A
// holds the result (the pointers are swapped as the sweeps go). Ends with a
// barrier. With FLIP the region's rows are stored top row first (the order
// of the global layout, as a tensor copy delivers them): region row y sits at
// row RH - 1 - y.
template <bool FLIP = false>
__device__ __forceinline__ void diff_sweeps(float*& A, float*& B, int tx, int ty, const Consts& c,
                                            const StepParams* __restrict__ prm, int sweeps,
                                            int halo, int TX, int TY) {
  const int RH = TY + 2 * halo;
  const int gx0 = tx * TX - halo, gy0 = ty * TY - halo;
  const int W = c.W, H = c.H;
  const float d_t = prm->dt;
  const float a = c.viscosity * d_t / (float)(c.h * c.h);
  // Updated cells: domain interior and not on the region's outer ring. A
  // thread owns one column and a contiguous run of rows, carrying the column
  // neighbours (j-1, j, j+1) in registers.
  const int x = threadIdx.x % kRegionW;
  const int groups = blockDim.x / kRegionW;
  const int i = gx0 + x;
  const int y_lo = max(1, 1 - gy0), y_hi = min(RH - 2, H - 2 - gy0);
  const int chunk = (y_hi - y_lo + groups) / groups;
  const int r0 = y_lo + (threadIdx.x / kRegionW) * chunk;
  const int r1 = min(y_hi + 1, r0 + chunk);
  const bool column = x > 0 && x < kRegionW - 1 && i > 0 && i < W - 1 && r0 < r1;
  const float den = fma_rn(4.0f, a, 1.0f);
  for (int t = 0; t < sweeps; t++) {
    // Only cells within `reach` (sweeps still to come) of the owned tile can
    // still influence it.
    const int reach = sweeps - 1 - t;
    const int ya = max(r0, halo - reach), yb = min(r1, RH - halo + reach);
    if (column && x >= halo - reach && x < kRegionW - halo + reach && ya < yb) {
      const int rs = FLIP ? -kRegionW : kRegionW;     // step to the next region row
      const int base = FLIP ? (RH - 1) * kRegionW : 0;
      diff_column(A, B, base + ya * rs + x, rs, yb - ya, a, den);
    }
    __syncthreads();
    float* T = A;
    A = B;
    B = T;
  }
}

// Owned cells of the region in A back to global (FLIP as in diff_sweeps).
template <bool FLIP = false>
__device__ __forceinline__ void diff_store_owned(const float* A, int tx, int ty,
                                                 float* __restrict__ u_out, const Consts& c, int halo,
                                                 int TX, int TY) {
  const int gx0 = tx * TX - halo, gy0 = ty * TY - halo;
  const int W = c.W, H = c.H;
  const int RH = TY + 2 * halo;
  const bool vec = ((W & 3) == 0) && ((gx0 & 3) == 0);
  for (int it = threadIdx.x; it < TY * kQuads; it += blockDim.x) {
    const int y = halo + it / kQuads, x = 4 * (it % kQuads);
    const int i = gx0 + x, j = gy0 + y;
    if (j >= H || i >= W) continue;
    const float* src = A + (FLIP ? RH - 1 - y : y) * kRegionW + x;
    if (vec && x >= halo && x + 3 < halo + TX) {
      *reinterpret_cast<float4*>(u_out + cell_index(W, H, i, j)) =
          *reinterpret_cast<const float4*>(src);
      continue;
    }
    for (int d = 0; d < 4; d++) {
      if (x + d < halo || x + d >= halo + TX || i + d >= W) continue;
      u_out[cell_index(W, H, i + d, j)] = src[d];
    }
  }
}

// ---------------------------------------------------------------------------
// Tensor-memory-accelerator staging of the diffusion region (FP32 fields).
// One thread issues a single 2-D bulk tensor copy of the whole 256 x RH region
// into A, completing on an mbarrier the block waits on; cells off the grid
// arrive as zero, as the vector loads stage them. The copy delivers rows in
// the global (top row first) order, so the sweeps and the write-back run with
// FLIP. Every wait is bounded: a block whose copy does not complete records
// the failure in the error words and returns.
// ---------------------------------------------------------------------------
constexpr int kTmaSpin = 1 << 22;
constexpr int kTmaAlign = 128;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
               : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}"
      : "=r"(done)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return done != 0;
}

// The box at (x, row) of `map` into dst; x * 4 bytes must be a multiple of 16.
__device__ __forceinline__ void tma_load_2d(float* dst, const CUtensorMap* map, int x, int row,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(row), "r"(smem_u32(bar))
      : "memory");
}

__global__ void __launch_bounds__(kBlockThreads, 1)
k_diffuse_blocked_tma(const __grid_constant__ CUtensorMap in_map, float* __restrict__ u_out,
                      Consts c, const StepParams* __restrict__ prm, int sweeps, int halo, int TX,
                      int TY, int tiles_x, int* __restrict__ err, int* __restrict__ host_err) {
  pdl_entry();
  extern __shared__ __align__(16) float smem_tma[];
  __shared__ __align__(8) uint64_t bar;
  const int tx = blockIdx.x % tiles_x, ty = blockIdx.x / tiles_x;
  const int RH = TY + 2 * halo;
  // Both buffers are copy destinations, 128-byte aligned (the launch adds
  // room for the alignment and a 128-byte gap between them).
  float* A = reinterpret_cast<float*>(
      (reinterpret_cast<uintptr_t>(smem_tma) + kTmaAlign - 1) & ~uintptr_t(kTmaAlign - 1));
  float* B = A + RH * kRegionW + kTmaAlign / sizeof(float);
  const int gx0 = tx * TX - halo, gy0 = ty * TY - halo;
  if (threadIdx.x == 0) mbar_init(&bar, 1);
  __syncthreads();
  if (threadIdx.x == 0) {
    // The region into both buffers (cells no sweep updates keep their value
    // in each), one copy per buffer on the same barrier.
    mbar_expect_tx(&bar, (uint32_t)(2 * RH * kRegionW * sizeof(float)));
    tma_load_2d(A, &in_map, gx0, c.H - gy0 - RH, &bar);
    tma_load_2d(B, &in_map, gx0, c.H - gy0 - RH, &bar);
  }
  bool done = false;
  for (int it = 0; it < kTmaSpin && !done; it++) done = mbar_try_wait(&bar, 0);
  if (__syncthreads_or(!done)) {
    if (threadIdx.x == 0) {
      if (err && atomicCAS(err, 0, 1) == 0 && host_err) {
        *(volatile int*)host_err = 1;
        __threadfence_system();
      }
      // The copy may still land: give it the same bound again before the
      // block's shared memory is released.
      for (int it = 0; it < kTmaSpin && !mbar_try_wait(&bar, 0); it++) {
      }
    }
    __syncthreads();
    return;
  }
  diff_sweeps<true>(A, B, tx, ty, c, prm, sweeps, halo, TX, TY);
  diff_store_owned<true>(A, tx, ty, u_out, c, halo, TX, TY);
}

// ---------------------------------------------------------------------------
// Host: tile geometry and pass enqueue.
// ---------------------------------------------------------------------------

// Whether step kernels are launched programmatically: OPENSAYAL_GB300_PDL=0 turns
// it off for the handles and batches made from then on.
inline bool programmatic_launch() {
  const char* env = std::getenv("OPENSAYAL_GB300_PDL");
  return !(env && env[0] == '0');
}

// Launch with programmatic stream serialisation when `pdl` (the kernels call
// pdl_entry() first, so the dependency on the previous kernel is kept).
template <class... KArgs, class... Args>
inline void launch_pdl(bool pdl, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                       cudaStream_t st, Args&&... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

constexpr size_t kMaxSmem = 227 * 1024;
constexpr size_t kStaticSmem = 256;

// Lets a kernel take as much dynamic shared memory as there is beside its own
// static memory, and clusters beyond the portable size. These limits belong to
// the kernel, not to a launch, and to the whole process: set to one grid's size
// before its launch, they could be lowered between the two by another thread
// with a smaller grid, and the launch was refused. So they are set once per
// kernel and device, to the most, and stay.
inline cudaError_t allow_most(const void* kernel) {
  static std::mutex mu;
  static std::set<std::pair<const void*, int>> done;
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(mu);
  if (done.count({kernel, device})) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)(kMaxSmem - kStaticSmem));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess) done.insert({kernel, device});
  return e;
}
template <class... KArgs>
inline cudaError_t allow_most(void (*kernel)(KArgs...)) {
  return allow_most(reinterpret_cast<const void*>(kernel));
}

// Owned tile height for a given halo: aim for one CTA per SM per wave
// (152 SMs), keep TY even, and fit shared memory.
inline TileGeom make_geom(int W, int H, int halo, int sms) {
  TileGeom g;
  g.halo = halo;
  g.TX = kRegionW - 2 * halo;
  g.tiles_x = (W + g.TX - 1) / g.TX;
  const int want_tiles_y = std::max(1, sms / g.tiles_x);
  int TY = (H + want_tiles_y - 1) / want_tiles_y;
  TY = std::max(2, (TY + 1) & ~1);
  // kStaticSmem: room for the kernels' own static shared memory.
  while (TY > 2 && diffusion_smem(TY + 2 * halo) + kStaticSmem > kMaxSmem) TY -= 2;
  g.TY = TY;
  g.RH = TY + 2 * halo;
  g.tiles_y = (H + TY - 1) / TY;
  g.smem = diffusion_smem(g.RH);
  return g;
}

// Sweeps per blocked pass as configured: -1 plain, K > 0 fixed, 0 = to be
// chosen by the autotuner once the handle exists.
inline int choose_block_k(const os_handle* h) {
  if (h->cfg.projection_block < 0) return -1;
  if (h->cfg.projection_block > 0) return std::min(h->cfg.projection_block, 32);
  return 0;
}

// Jacobi sweeps per blocked diffusion pass.
inline int diffusion_depth(const os_handle* h) { return h->diff_k > 0 ? h->diff_k : h->block_k; }

// FP32 arithmetic on FP32, FP16 or BF16 storage. With reduced storage a value
// is rounded to storage once per pass (the region stays FP32 in shared
// memory), not once per sweep as in the plain kernels.
template <class S, class A>
inline bool blocked_supported(const os_handle*) {
  return std::is_same<A, float>::value &&
         (std::is_same<S, float>::value || std::is_same<S, __half>::value ||
          std::is_same<S, __nv_bfloat16>::value);
}

inline int sm_count(int device) {
  int n = 0;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || n < 1)
    n = 152;
  return n;
}

// Dynamic shared memory of k_diffuse_blocked_tma: two 128-byte aligned
// buffers of RH x 256 floats and the alignment slack.
inline size_t tma_diffusion_smem(int RH) {
  return 2 * (size_t)RH * kRegionW * sizeof(float) + 2 * kTmaAlign;
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// against the driver library).
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                   const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

// Tensor maps of u and ub (FP32) with a box of one diffusion region, when the
// copy's rules hold: row pitch and region origin multiples of 16 bytes (W and
// the halo K multiples of 4), the box at most 256 rows.
inline bool prepare_tma_diffusion(os_handle* h) {
  const int K = diffusion_depth(h);
  if (h->storage != OS_STORAGE_F32 || K <= 0 || (K & 3) || (h->W & 3)) return false;
  const TileGeom g = make_geom(h->W, h->H, K, sm_count(h->cfg.device));
  if (g.RH > 256 || (g.TX & 3) || (g.halo & 3)) return false;
  if (tma_diffusion_smem(g.RH) + kStaticSmem > kMaxSmem || K > 8) return false;
  const EncodeTiledFn enc = encode_tiled();
  if (!enc) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)h->W, (cuuint64_t)h->H};
  const cuuint64_t strides[1] = {(cuuint64_t)h->W * sizeof(float)};
  const cuuint32_t box[2] = {(cuuint32_t)kRegionW, (cuuint32_t)g.RH};
  const cuuint32_t elem[2] = {1, 1};
  for (int k = 0; k < 2; k++) {
    if (enc(&h->diff_maps[k], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, k ? h->ub : h->u, dims,
            strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return false;
  }
  return true;
}

// ceil(n / K) diffusion passes staged by tensor copies.
inline int enqueue_tma_diffusion(os_handle* h, cudaStream_t st, int* cur_u) {
  const int K = diffusion_depth(h);
  const TileGeom g = make_geom(h->W, h->H, K, sm_count(h->cfg.device));
  float* U[2] = {static_cast<float*>(h->u), static_cast<float*>(h->ub)};
  const int tiles = g.tiles_x * g.tiles_y;
  const size_t smem = tma_diffusion_smem(g.RH);
  if (allow_most(k_diffuse_blocked_tma) != cudaSuccess) return -1;
  int launches = 0;
  for (int done = 0; done < h->c.n;) {
    const int sweeps = std::min(K, h->c.n - done);
    launch_pdl(h->pdl, k_diffuse_blocked_tma, tiles, kBlockThreads, smem, st,
               h->diff_maps[*cur_u], U[1 - *cur_u], h->c, (const StepParams*)h->d_params,
               sweeps, g.halo, g.TX, g.TY, g.tiles_x, h->rerr, h->d_host_rerr);
    launches++;
    *cur_u = 1 - *cur_u;
    done += sweeps;
  }
  return launches;
}

}  // namespace osg
