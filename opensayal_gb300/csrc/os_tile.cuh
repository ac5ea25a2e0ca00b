// os_tile.cuh — tiles held in registers: the red/black projection and the
// Jacobi diffusion with every face of a tile in the registers of its CTAs from
// the first sweep of a pass to the last.
//
// A tile's region is 256 columns wide and RH = R * warps * cluster rows high:
// `cluster` CTAs (a thread-block cluster) of `warps` warps each, warp by warp
// from the bottom up. A warp holds a strip of R rows, lane l its columns 8 l ..
// 8 l + 7: a patch of 8 x R cells per thread. The region of tile (tx, ty) starts
// at cell (tx * TX, ty * TY); it carries `halo` cells on each side that has a
// neighbouring tile and none at the edges of the grid, so the tiles at the
// edges own that much more and W x H takes ceil((W - 2 halo) / TX) x
// ceil((H - 2 halo) / TY) tiles.
//
// What bounds these sweeps is the FP32 pipe (128 lanes per cycle and SM, the
// packed f32x2 forms have the same rate): a red/black update is 9 operations,
// a Jacobi update 5. With the fields in shared memory the sweeps were bound by
// its 32 words per cycle instead (4 accesses per red/black update with the
// vertical faces in registers, 3 per Jacobi update). Here the only traffic
// between threads is one shuffle per row (8 cells, two rows of a colour) for
// the faces between lanes, and 4 words up and 4 down per lane and half-sweep
// between strips, by an asynchronous store into the neighbouring strip's inbox
// in shared memory, in its own CTA or the next one of the cluster, which an
// mbarrier there counts. It is on its way while the strips' inner rows are
// updated; no barrier of the CTA is in the sweeps.
//
// Updates are the plain kernels' expressions in the same order, so every
// result has the same bits.
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

#include "../../include/opensayal_gb300.h"
#include "os_common.cuh"

namespace osg {

constexpr int kTileW = 256;      // region width in cells
constexpr int kLaneCols = 8;     // columns per lane
constexpr uint32_t kAllLanes = 0xffffffffu;

// Strip heights the kernels are built for, and the warps per CTA that the
// register file holds for each: a scheduler's 16,384 registers go to whole
// warps, so 8 warps may use 255 registers a thread, 12 warps 168, 16 warps 128.
constexpr int kProjectRows[] = {2, 4, 6, 8, 10};
constexpr int kDiffuseRows[] = {2, 4, 6, 8, 12};
__host__ __device__ constexpr int project_max_warps(int R) {
  return R <= 4 ? 16 : R <= 6 ? 12 : 8;
}
// The diffusion holds one field.
__host__ __device__ constexpr int diffuse_max_warps(int R) {
  return R <= 4 ? 16 : R <= 8 ? 12 : 8;
}

struct RegTile {
  int halo;              // halo in cells, on sides that have a neighbour
  int TX, TY;            // pitch of the tiles: region minus both halos
  int RH;                // region rows, R * warps * cluster
  int R, warps, cluster;
  int tiles_x, tiles_y;
  size_t smem;           // dynamic shared memory per CTA
};

struct ResidentSync {
  unsigned* epochs;     // one per CTA: exchanges so far (monotonic)
  uint4* packets;       // two copies of the exchanged cells (see the exchange below)
  int* dev_err;         // set by a thread that gave up; polled by the others
  int* host_err;        // mapped host word the host reads after synchronising
};

// A bounded wait gave up: the host reports it (OS_ERR_TIMEOUT).
__device__ __forceinline__ void record_failure(const ResidentSync& sync) {
  if (atomicCAS(sync.dev_err, 0, 1) == 0 && sync.host_err) {
    *(volatile int*)sync.host_err = 1;
    __threadfence_system();
  }
}

// ---------------------------------------------------------------------------
// Fields in global memory: quads of 4 columns.
// ---------------------------------------------------------------------------

// Loads go through L2 only: a launch may read cells that other CTAs of it
// wrote, and a line this SM cached earlier must not be returned. Loads and
// stores are predicated instead of branched around, so that all of a patch's
// are in flight together (with a branch around each, a patch's rows came in
// one memory latency after another). The two 16-bit types share one
// instantiation (`bf` says which).
struct F32Cells {
  using Word = float;
  __device__ __forceinline__ void load4(bool on, const float* p, float* q) const {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.s32 p, %5, 0;\n @p ld.global.cg.v4.f32 {%0, %1, %2, %3}, [%4];\n}"
        : "+f"(q[0]), "+f"(q[1]), "+f"(q[2]), "+f"(q[3]) : "l"(p), "r"((int)on) : "memory");
  }
  __device__ __forceinline__ void load1(bool on, const float* p, float* q) const {
    asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %2, 0;\n @p ld.global.cg.f32 %0, [%1];\n}"
                 : "+f"(*q) : "l"(p), "r"((int)on) : "memory");
  }
  __device__ __forceinline__ float value(float q) const { return q; }
  __device__ __forceinline__ void store4(bool on, float* p, const float* q) const {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.s32 p, %5, 0;\n @p st.global.v4.f32 [%4], {%0, %1, %2, %3};\n}"
        ::"f"(q[0]), "f"(q[1]), "f"(q[2]), "f"(q[3]), "l"(p), "r"((int)on) : "memory");
  }
  __device__ __forceinline__ void store1(bool on, float* p, const float* q) const {
    asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %2, 0;\n @p st.global.f32 [%1], %0;\n}"
                 ::"f"(*q), "l"(p), "r"((int)on) : "memory");
  }
};
struct HalfCells {
  using Word = uint16_t;
  bool bf;
  __device__ __forceinline__ float from(uint32_t bits) const {
    return bf ? __uint_as_float(bits << 16) : __half2float(__ushort_as_half((uint16_t)bits));
  }
  __device__ __forceinline__ uint32_t to(float x) const {
    return bf ? (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(x))
              : (uint32_t)__half_as_ushort(__float2half_rn(x));
  }
  __device__ __forceinline__ void load4(bool on, const uint16_t* p, float* q) const {
    uint32_t a = 0u, b = 0u;
    asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %3, 0;\n @p ld.global.cg.v2.u32 {%0, %1}, [%2];\n}"
                 : "+r"(a), "+r"(b) : "l"(p), "r"((int)on) : "memory");
    q[0] = on ? from(a & 0xffffu) : q[0], q[1] = on ? from(a >> 16) : q[1];
    q[2] = on ? from(b & 0xffffu) : q[2], q[3] = on ? from(b >> 16) : q[3];
  }
  // The cell's bits, which value() turns into the cell: as it came, a patch's
  // conversions stood between its loads, and few of them were in flight.
  __device__ __forceinline__ void load1(bool on, const uint16_t* p, float* q) const {
    asm volatile("{\n .reg .pred p;\n .reg .b32 t;\n mov.b32 t, %0;\n setp.ne.s32 p, %2, 0;\n"
                 " @p ld.global.cg.u16 t, [%1];\n mov.b32 %0, t;\n}"
                 : "+f"(*q) : "l"(p), "r"((int)on) : "memory");
  }
  __device__ __forceinline__ float value(float q) const { return from(__float_as_uint(q)); }
  __device__ __forceinline__ void store4(bool on, uint16_t* p, const float* q) const {
    asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %3, 0;\n @p st.global.v2.u32 [%2], {%0, %1};\n}"
                 ::"r"(to(q[0]) | to(q[1]) << 16), "r"(to(q[2]) | to(q[3]) << 16), "l"(p),
                 "r"((int)on) : "memory");
  }
  __device__ __forceinline__ void store1(bool on, uint16_t* p, const float* q) const {
    asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %2, 0;\n @p st.global.u16 [%1], %0;\n}"
                 ::"h"((uint16_t)to(*q)), "l"(p), "r"((int)on) : "memory");
  }
};

// fn(cells) for the storage type.
template <class Fn>
__device__ __forceinline__ void on_cells(int storage, Fn&& fn) {
  if (storage == OS_STORAGE_F32)
    fn(F32Cells{});
  else
    fn(HalfCells{storage == OS_STORAGE_BF16});
}

// ---------------------------------------------------------------------------
// Where a thread's patch lies.
// ---------------------------------------------------------------------------
struct Patch {
  int gx0, gy0;    // region origin on the grid
  int lane, warp;
  int x0, y0;      // first column and row of the patch in the region
  int yl;          // its first row among the CTA's rows
  int c0, c1;      // the CTA's rows of the region
  bool left, right, below, above;  // the tile has a neighbour on that side
  int ox0, ox1, oy0, oy1;          // owned columns and rows, in the region
  bool down, up;                   // the tile has a strip below / above this one
  bool idle;                       // every row of the strip is off the grid
};

// A tile of a grid.
struct TilePlace {
  int tx, ty, tiles_x, tiles_y;
};

// Worked out anew wherever it is used outside the sweeps (the block and thread
// numbers pass through an empty asm, so that the compiler does not keep one
// copy alive): held across the sweep loops it costs registers that their faces
// need.
__device__ __forceinline__ Patch patch_at(const TilePlace& t, const RegTile& g, int R, int W,
                                          int H) {
  Patch P;
  unsigned block = blockIdx.x, thread = threadIdx.x;
  asm volatile("" : "+r"(block), "+r"(thread));
  const int rank = block % g.cluster;
  P.gx0 = t.tx * g.TX, P.gy0 = t.ty * g.TY;
  P.lane = thread & 31, P.warp = thread >> 5;
  P.yl = P.warp * R;
  P.c0 = rank * g.warps * R, P.c1 = P.c0 + g.warps * R;
  P.x0 = P.lane * kLaneCols, P.y0 = P.c0 + P.yl;
  P.left = t.tx > 0, P.right = t.tx + 1 < t.tiles_x;
  P.below = t.ty > 0, P.above = t.ty + 1 < t.tiles_y;
  P.ox0 = P.left ? g.halo : 0;
  P.oy0 = P.below ? g.halo : 0;
  P.ox1 = P.right ? kTileW - g.halo : min(kTileW, W - P.gx0);
  P.oy1 = P.above ? g.RH - g.halo : min(g.RH, H - P.gy0);
  P.down = P.warp > 0 || rank > 0;
  P.up = P.warp < g.warps - 1 || rank + 1 < g.cluster;
  P.idle = P.gy0 + P.y0 >= H;
  return P;
}
__device__ __forceinline__ Patch patch_of(const RegTile& g, int R, int W, int H) {
  unsigned tile = blockIdx.x / g.cluster;
  asm volatile("" : "+r"(tile));
  return patch_at(TilePlace{(int)tile % g.tiles_x, (int)tile / g.tiles_x, g.tiles_x, g.tiles_y}, g,
                  R, W, H);
}

// Rows of a strip of R that are in [lo, hi) of the region, as a bit mask.
__device__ __forceinline__ uint32_t rows_in(int y0, int R, int lo, int hi) {
  const int a = min(max(lo - y0, 0), R), b = min(max(hi - y0, 0), R);
  return ((1u << b) - 1u) & ~((1u << a) - 1u);
}

// ---------------------------------------------------------------------------
// Messages between neighbouring strips of a tile.
//
// Each warp has an inbox in its CTA's shared memory: for message m (buffer m %
// 2) one part from the strip below and one from the strip above, 16 or 32 bytes
// a lane, and an mbarrier that completes when both have arrived. A strip sends
// by asynchronous stores that complete bytes on the receiver's mbarrier, to a
// warp of its own CTA or of the next one in the cluster in the same way (280
// cycles from one CTA to the next; with a store, a fence and a remote arrival
// it took 540). Message m + 2 takes the buffer of message m: its sender has by
// then received the receiver's own message m + 1, which that strip sent after
// it read message m. A strip at the tile's edge sends to itself what it would
// send to the strip that is not there.
// ---------------------------------------------------------------------------
constexpr int kInboxHead = 16;      // two mbarriers
constexpr uint32_t kMessageLimit = 1000000000u;  // of a bounded wait, in ns

__host__ __device__ constexpr int inbox_bytes(int words) { return kInboxHead + 4 * words * 128; }

__device__ __forceinline__ uint32_t shared_address(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// (Of the last CTA where the cluster has none of that rank; see clusters_of.)
__device__ __forceinline__ uint32_t cluster_address(uint32_t a, uint32_t rank) {
  uint32_t r, n;
  asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(n));
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(min(rank, n - 1u)));
  return r;
}
// (Not the .aligned forms: a warp may come here with its lanes apart.)
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

// Whether the launch has the clusters that its tiles are laid out for: the strips'
// messages go to addresses that do not exist without them. A launch that has lost
// them (a profiler that makes it again may) reports a failure and does nothing.
// Asked behind the loads and before the first message: at the head of the kernels
// it took 3% of the step at 1920 x 1080 in BF16 (545 us for 526).
__device__ __forceinline__ bool clusters_of(int cluster, const ResidentSync& sync) {
  uint32_t n;
  asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(n));
  if (n == (uint32_t)cluster) return true;
  record_failure(sync);
  return false;
}

// WORDS: 32-bit words per lane in each part of a message (4 or 8).
template <int WORDS>
struct Link {
  static constexpr int kPart = WORDS * 128;  // bytes of a part, 512 per 4 words
  uint32_t mine;                 // this warp's inbox (shared address)
  uint32_t up, down;             // the neighbours' inboxes (cluster shared addresses)
  uint32_t up_part, down_part;   // where this strip's part goes in them
  bool lost;  // a wait gave up: the strip takes no further part (the same in the warp)
};

// Prepares the warp's inbox and finds the neighbours'; the caller passes a
// cluster barrier before the first message.
template <int WORDS>
__device__ __forceinline__ Link<WORDS> open_link(char* smem, const Patch& P, const RegTile& g) {
  constexpr int kBytes = kInboxHead + 4 * Link<WORDS>::kPart;
  Link<WORDS> k;
  const uint32_t base = shared_address(smem);
  const int rank = blockIdx.x % g.cluster;
  k.mine = base + P.warp * kBytes;
  k.lost = false;
  const uint32_t self = cluster_address(k.mine, rank);
  k.up = P.up ? (P.warp + 1 < g.warps ? cluster_address(k.mine + kBytes, rank)
                                      : cluster_address(base, rank + 1))
              : self;
  k.down = P.down ? (P.warp > 0 ? cluster_address(k.mine - kBytes, rank)
                                : cluster_address(base + (g.warps - 1) * kBytes, rank - 1))
                  : self;
  // Part 0 comes from below, part 1 from above.
  k.up_part = (P.up ? 0 : Link<WORDS>::kPart) + kInboxHead + P.lane * 16;
  k.down_part = (P.down ? Link<WORDS>::kPart : 0) + kInboxHead + P.lane * 16;
  if (P.lane == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(k.mine) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(k.mine + 8) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  return k;
}

// Four words (words 4 k ..) of message m to an inbox.
template <int WORDS>
__device__ __forceinline__ void post(uint32_t inbox, uint32_t part, unsigned m, int k, float4 x) {
  const uint32_t buffer = m & 1u;
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, "
      "[%5];" ::"r"(inbox + part + buffer * (2 * WORDS * 128) + k * 512),
      "f"(x.x), "f"(x.y), "f"(x.z), "f"(x.w), "r"(inbox + 8 * buffer)
      : "memory");
}

// Waits until both parts of message m are there, for kMessageLimit or until
// another wait has given up (looked at every 64 polls, each of which the hardware
// may hold for a while). A wait that gives up records the failure, and the strip
// sends and awaits nothing more: every later wait for one of its messages ends
// soon, and no mbarrier that is behind is armed again. The host reports it.
template <int WORDS>
__device__ __forceinline__ void await_message(Link<WORDS>& link, unsigned m,
                                              const ResidentSync& sync) {
  const uint32_t bar = link.mine + 8 * (m & 1u);
  if ((threadIdx.x & 31) == 0)
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                 "r"(2 * Link<WORDS>::kPart)
                 : "memory");
  uint32_t done = 0, since = 0;
#pragma unroll 1
  for (int it = 0;; it++) {
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(bar), "r"((m >> 1) & 1u)
        : "memory");
    if (done) break;
    if (it % 64 != 63) continue;
    uint32_t now;
    asm volatile("mov.u32 %0, %%globaltimer_lo;" : "=r"(now));
    if (it == 63) since = now;
    if (now - since > kMessageLimit || *(volatile int*)sync.dev_err) {
      record_failure(sync);
      break;
    }
  }
  link.lost = !__all_sync(kAllLanes, done);  // lanes may have left the loop apart
}
// Words 4 k .. of the part from below (0) or above (1) of message m.
template <int WORDS>
__device__ __forceinline__ float4 read_message(const Link<WORDS>& link, int part, unsigned m,
                                               int k) {
  float4 x;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w)
               : "r"(link.mine + kInboxHead + ((m & 1u) * 2 + part) * Link<WORDS>::kPart +
                     k * 512 + (threadIdx.x & 31) * 16)
               : "memory");
  return x;
}

// The messages of a strip off the grid, m .. m + count - 1: it takes part so
// that the strips beside it do not wait. What it sends is read by no cell of the
// grid.
template <int WORDS>
__device__ __forceinline__ void idle_messages(Link<WORDS>& link, unsigned m, int count,
                                              const ResidentSync& sync) {
#pragma unroll 1
  for (const unsigned end = m + count; m != end && !link.lost; m++) {
#pragma unroll
    for (int k = 0; k < WORDS / 4; k++) {
      post<WORDS>(link.down, link.down_part, m, k, make_float4(0.0f, 0.0f, 0.0f, 0.0f));
      post<WORDS>(link.up, link.up_part, m, k, make_float4(0.0f, 0.0f, 0.0f, 0.0f));
    }
    await_message(link, m, sync);
  }
}

// ---------------------------------------------------------------------------
// The halo exchange between tiles that stay in registers across passes.
//
// After pass q a warp sends the band of its owned cells that lie in the halos
// of neighbouring tiles, and then receives the cells of its own ring, packet by
// packet: 16 bytes that hold three values and the number of the exchange, which
// is the only synchronisation. A packet is written and read as one 128-bit
// access, so a reader that sees the number it waits for has the values; there
// is no fence, no flag and no barrier between tiles. (With the band stored to
// the fields, a fence, a flag per warp, a poll and the reload, an exchange took
// 4.2 us; the fence and the poll alone 2.3.) Within a cluster no halo is needed:
// the packets carry the sides of the tiles, and their lower and upper rows
// where tiles lie above one another.
//
// Packets lie by the cell they carry, in two copies that alternate. A copy is
// written again two exchanges later: by then the writer has received the
// exchange between from every neighbouring tile, whose CTAs sent it after their
// reads of this one: a CTA sends behind its own barrier, and the CTAs of a
// tile whose rows lie within a halo of each other have since exchanged
// messages in the sweeps between. Those reach a strip further each, and two
// exchanges lie D sweeps apart: at least D messages of the diffusion, whose halo
// of D cells is D / R strips high, and 2 D + 1 of the projection, whose halo has
// 2 D cells (R is at least 2, one strip more for the row that a strip starts in).
// ---------------------------------------------------------------------------
constexpr int kSpinLimit = 1 << 20;  // polls per wait

__device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void packet_out(bool on, uint4* p, float a, float b, float c,
                                           unsigned number) {
  asm volatile(
      "{\n .reg .pred p;\n .reg .b128 t;\n .reg .b64 x, y;\n setp.ne.s32 p, %5, 0;\n"
      " mov.b64 x, {%0, %1};\n mov.b64 y, {%2, %3};\n mov.b128 t, {x, y};\n"
      " @p st.relaxed.gpu.global.b128 [%4], t;\n}"
      ::"r"(__float_as_uint(a)), "r"(__float_as_uint(b)), "r"(__float_as_uint(c)), "r"(number),
      "l"(p), "r"((int)on) : "memory");
}

// The packet's values where `on`; returns whether its number is `number` (true
// when not `on`).
__device__ __forceinline__ bool packet_in(bool on, const uint4* p, float& a, float& b, float& c,
                                          unsigned number) {
  unsigned ua = __float_as_uint(a), ub = __float_as_uint(b), uc = __float_as_uint(c), n = number;
  asm volatile(
      "{\n .reg .pred p;\n .reg .b128 t;\n .reg .b64 x, y;\n setp.ne.s32 p, %5, 0;\n"
      " mov.b64 x, {%0, %1};\n mov.b64 y, {%2, %3};\n mov.b128 t, {x, y};\n"
      " @p ld.relaxed.gpu.global.b128 t, [%4];\n"
      " mov.b128 {x, y}, t;\n mov.b64 {%0, %1}, x;\n mov.b64 {%2, %3}, y;\n}"
      : "+r"(ua), "+r"(ub), "+r"(uc), "+r"(n) : "l"(p), "r"((int)on) : "memory");
  a = __uint_as_float(ua), b = __uint_as_float(ub), c = __uint_as_float(uc);
  return n == number;
}

// One poll of a bounded wait that did not find its packets: false when the
// wait gives up. The failure is recorded, the caller carries on with what it
// has (every later wait gives up at once), and the host reports it.
__device__ __forceinline__ bool poll_again(int it, const ResidentSync& sync) {
  if (it < kSpinLimit && (it % 64 != 63 || !*(volatile int*)sync.dev_err)) return true;
  record_failure(sync);
  return false;
}

// Where quads of the region are not aligned (W or the halo is no multiple of
// 4), a warp takes a row's cells one by one, lanes on consecutive columns, and
// turns them between that order (lane l: columns l, l + 32, ..) and the patch's
// through a row of shared memory of its own. With each lane on its own eight
// columns every access touched a sector per lane (307 x 479 in FP16, passes of
// 4 sweeps: 245 us a step, now 156; 3001 x 1500: 735 us, now 531).
constexpr int kStageBytes = kTileW * 4;  // per warp
__host__ __device__ inline bool quads_aligned(int W, int halo) { return ((W | halo) & 3) == 0; }
__host__ __device__ inline size_t stage_smem(int W, int halo, int warps) {
  return quads_aligned(W, halo) ? 0 : (size_t)warps * kStageBytes;
}
// The warp's row, at the end of the CTA's shared memory. (The kernels of a
// single grid are built for aligned quads and for others: with both ways in
// one kernel the strips of 10 rows spilled, 272 us a step at 1920 x 1080
// instead of 236.)
__device__ __forceinline__ float* stage_of(char* smem, const RegTile& g) {
  unsigned thread = threadIdx.x;
  asm volatile("" : "+r"(thread));  // worked out anew where it is used, as patch_at
  float* row = reinterpret_cast<float*>(smem + g.smem - (g.warps - (thread >> 5)) * kStageBytes);
  __builtin_assume(row != nullptr);
  return row;
}
template <class IO>
__device__ __forceinline__ void turn_in(const IO& io, float (&f)[8], float* stage, int lane) {
#pragma unroll
  for (int k = 0; k < 8; k++) stage[lane + 32 * k] = io.value(f[k]);
  __syncwarp();
  const float4 a = reinterpret_cast<const float4*>(stage)[2 * lane];
  const float4 b = reinterpret_cast<const float4*>(stage)[2 * lane + 1];
  __syncwarp();
  f[0] = a.x, f[1] = a.y, f[2] = a.z, f[3] = a.w;
  f[4] = b.x, f[5] = b.y, f[6] = b.z, f[7] = b.w;
}
__device__ __forceinline__ void turn_out(const float (&f)[8], float (&g)[8], float* stage,
                                         int lane) {
  reinterpret_cast<float4*>(stage)[2 * lane] = make_float4(f[0], f[1], f[2], f[3]);
  reinterpret_cast<float4*>(stage)[2 * lane + 1] = make_float4(f[4], f[5], f[6], f[7]);
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 8; k++) g[k] = stage[lane + 32 * k];
  __syncwarp();
}

// The whole patch from a field (row j of the grid at (H - 1 - j) W). `stage`: see
// above; null where quads are aligned: the loads then carry no condition (a
// kernel's code is fetched cold once per launch, so what it does once has to be
// short), and a cell off the grid reads the nearest quad or row of it: cells off
// the grid may hold any value, no cell of the grid depends on them.
template <int R, class IO>
__device__ __forceinline__ void patch_in(const IO& io, float (&f)[R][8], const void* field,
                                         const Patch& P, int W, int H, float* stage) {
  const int x = P.gx0 + P.x0, j0 = P.gy0 + P.y0;
  const typename IO::Word* base = static_cast<const typename IO::Word*>(field);
  if (!stage) {
    const int xa = min(x, W - 4), xb = min(x + 4, W - 4);
    const int step = H - 1 - j0;  // rows of the grid above row j0
    const typename IO::Word* row = base + (int64_t)max(step, 0) * W;
#pragma unroll
    for (int r = 0; r < R; r++) {
      io.load4(true, row + xa, &f[r][0]);
      io.load4(true, row + xb, &f[r][4]);
      if (r < step) row -= W;
    }
    return;
  }
  const int xl = P.gx0 + P.lane;
  const typename IO::Word* row = base + (int64_t)(H - 1 - j0) * W + xl;
#pragma unroll
  for (int r = 0; r < R; r++, row -= W)
#pragma unroll
    for (int k = 0; k < 8; k++) io.load1(j0 + r < H && xl + 32 * k < W, row + 32 * k, &f[r][k]);
#pragma unroll
  for (int r = 0; r < R; r++) turn_in(io, f[r], stage, P.lane);
}

// Row y of the region, the lane's eight columns, in the same way.
template <class IO>
__device__ __forceinline__ void row_in(const IO& io, float (&f)[8], const void* field,
                                       const Patch& P, int y, int W, int H, float* stage) {
  const int x = P.gx0 + P.x0, j = min(P.gy0 + y, H - 1);
  const typename IO::Word* row =
      static_cast<const typename IO::Word*>(field) + (int64_t)(H - 1 - j) * W;
  if (!stage) {
    io.load4(true, row + min(x, W - 4), &f[0]);
    io.load4(true, row + min(x + 4, W - 4), &f[4]);
  } else {
    const int xl = P.gx0 + P.lane;
#pragma unroll
    for (int k = 0; k < 8; k++) io.load1(xl + 32 * k < W, row + xl + 32 * k, &f[k]);
    turn_in(io, f, stage, P.lane);
  }
}

// The patch's rows in `rows` out to a field, the owned columns among them.
template <int R, class IO>
__device__ __forceinline__ void patch_out(const IO& io, const float (&f)[R][8], void* field,
                                          const Patch& P, uint32_t rows, int W, int H,
                                          float* stage) {
  typename IO::Word* row = static_cast<typename IO::Word*>(field) +
                           (int64_t)(H - 1 - (P.gy0 + P.y0)) * W + P.gx0 +
                           (stage ? P.lane : P.x0);
  if (!stage) {
    const int lo = P.ox0 - P.x0, hi = P.ox1 - P.x0;  // owned columns of the patch
    const bool qa = 0 >= lo && 0 < hi, qb = 4 >= lo && 4 < hi;
#pragma unroll
    for (int r = 0; r < R; r++, row -= W) {
      if (((rows >> r) & 1u) == 0u) continue;  // the same for the whole warp
      io.store4(qa, row, &f[r][0]);
      io.store4(qb, row + 4, &f[r][4]);
    }
    return;
  }
#pragma unroll
  for (int r = 0; r < R; r++, row -= W) {
    if (((rows >> r) & 1u) == 0u) continue;
    float g[8];
    turn_out(f[r], g, stage, P.lane);
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const int x = P.lane + 32 * k;
      io.store1(x >= P.ox0 && x < P.ox1, row + 32 * k, &g[k]);
    }
  }
}

// Packets of a quad of cells: three for u and v (8 values), two for u alone.
template <int FIELDS>
constexpr int kPacketsPerQuad = FIELDS == 2 ? 3 : 2;

// The cells an exchange moves, as quads: the CTA's rows of the tile's lower and
// upper halo (the ring) or of the owned rows beside them (the band), and in
// every row of the CTA halo columns on either side. The ring takes one row
// more than the CTA has, the row above its top strip, whose lower faces that
// strip holds copies of. Row quads are taken by (row, which of the lane's two
// quads, lane), side quads by (row, side, quad), both in shared memory and in
// the numbering of the items.
constexpr int kRowQuads = kTileW / 4;
struct HaloRows {
  int a0, an, b0, bn;  // rows [a0, a0 + an) and [b0, b0 + bn) of the region
  int rows, items;     // row items, all items
};
struct Exchange {
  float4* cells;  // rows: [an + bn][FIELDS][2][32], then sides: [rows][2][halo / 4][FIELDS]
  int* send;      // per item of the band: its packet's place, or -1 (not sent)
  int* take;      // per item of the ring: its packet's place, or -1 (not taken)
  HaloRows band, ring;
};
// Items of a CTA of L rows at most.
inline __host__ __device__ int exchange_items(int halo, int L) {
  const int rows = 2 * (halo < L + 1 ? halo : L + 1);
  return rows * kRowQuads + (L + 1) * (halo / 2);
}
inline __host__ __device__ size_t exchange_smem(int halo, int L, int fields) {
  return (size_t)exchange_items(halo, L) * (fields * 16 + 8);
}

__device__ __forceinline__ HaloRows halo_rows(int in, int c0, int c1, const Patch& P,
                                              const RegTile& g) {
  HaloRows s;
  const int h = g.halo;
  s.a0 = max(c0, in);
  s.an = P.below ? max(0, min(c1, in + h) - s.a0) : 0;
  s.b0 = max(c0, g.RH - h - in);
  s.bn = P.above ? max(0, min(c1, g.RH - in) - s.b0) : 0;
  s.rows = (s.an + s.bn) * kRowQuads;
  s.items = s.rows + (c1 - c0) * (h / 2);
  return s;
}

// The buffer and plan of an exchange in shared memory at `base`.
__device__ __forceinline__ Exchange exchange_view(char* base, const Patch& P, const RegTile& g,
                                                  int fields) {
  Exchange x;
  x.band = halo_rows(g.halo, P.c0, P.c1, P, g);
  x.ring = halo_rows(0, P.c0, P.c1 + 1, P, g);
  const int most = exchange_items(g.halo, P.c1 - P.c0);
  x.cells = reinterpret_cast<float4*>(base);
  x.send = reinterpret_cast<int*>(x.cells + most * fields);
  x.take = x.send + most;
  return x;
}

// The places of all items' packets, once per launch.
__device__ __forceinline__ void exchange_plan(char* base, const RegTile& g, int R, int fields,
                                              int W, int H) {
  const Patch P = patch_of(g, R, W, H);
  const Exchange x = exchange_view(base, P, g, fields);
  const int h = g.halo, hq = h / 4;
  const int half = (W + 7) / 8;  // pairs of quads in a row of the grid
#pragma unroll 1
  for (int band = 0; band < 2; band++) {
    const HaloRows s = band ? x.band : x.ring;
    const int in = band ? h : 0;
#pragma unroll 1
    for (int it = threadIdx.x; it < s.items; it += blockDim.x) {
      int y, q;
      bool on;
      if (it < s.rows) {
        const int k = it / kRowQuads;
        y = k < s.an ? s.a0 + k : s.b0 + (k - s.an);
        q = 2 * (it & 31) + ((it >> 5) & 1);
        // A row of both bands goes once.
        on = !band || k < s.an || !(P.below && y < 2 * h);
      } else {
        const int e = it - s.rows, k = e % (2 * hq);
        y = P.c0 + e / (2 * hq);
        q = k < hq ? in / 4 + k : kRowQuads - hq - in / 4 + (k - hq);
        on = (k < hq ? P.left : P.right) && y >= P.oy0 && y < P.oy1;
        // A side quad of a band row goes with its row.
        if (band)
          on = on && !(P.below && y < 2 * h) && !(P.above && y >= g.RH - 2 * h);
      }
      const int i = P.gx0 + 4 * q, j = P.gy0 + y;
      on = on && i < W && j < H && y < g.RH;
      if (band) on = on && 4 * q >= P.ox0 && 4 * q < P.ox1;  // only owned columns go
      const int Q = i / 4;
      (band ? x.send : x.take)[it] = on ? (j * 2 + (Q & 1)) * half + (Q >> 1) : -1;
    }
  }
}
// Packets of one plane (values 3 k .. 3 k + 2 of every quad of the grid).
inline __host__ __device__ int64_t packet_plane(int W, int H) {
  return (int64_t)H * 2 * ((W + 7) / 8);
}

// A lane's two quads of rows between registers and the buffer.
template <bool OUT>
__device__ __forceinline__ void move_quad(float4* p, float* q) {
  if (OUT) {
    *p = make_float4(q[0], q[1], q[2], q[3]);
  } else {
    const float4 t = *p;
    q[0] = t.x, q[1] = t.y, q[2] = t.z, q[3] = t.w;
  }
}

// The patch's share of the band out of the registers (BAND), or of the ring
// into them; with the ring also row R of the strip, the faces `f_top` of the
// last field that lie on the strip's upper edge.
template <int FIELDS, bool BAND, int R>
__device__ __forceinline__ void exchange_patch(float (&f)[R][8], float (&f2)[R][8],
                                               float (&f_top)[8], const Exchange& x,
                                               const Patch& P, const RegTile& g) {
  const int h = g.halo, hq = h / 4, in = BAND ? h : 0;
  const HaloRows s = BAND ? x.band : x.ring;
  // Side quads of the lane (halos are whole numbers of quads).
  const int l0 = 2 * P.lane - in / 4, r0 = 2 * P.lane - (kRowQuads - hq - in / 4);
  constexpr int kRows = BAND ? R : R + 1;  // row R: the strip above's first
  const uint32_t whole = rows_in(P.y0, kRows, s.a0, s.a0 + s.an) |
                         rows_in(P.y0, kRows, s.b0, s.b0 + s.bn);
  const uint32_t owned = rows_in(P.y0, kRows, P.oy0, P.oy1) & ~whole;
#pragma unroll
  for (int r = 0; r < kRows; r++) {
    if (((whole >> r) & 1u) == 0u) continue;  // the same for the warp
    const int y = P.y0 + r;
    const int k = y >= s.a0 && y < s.a0 + s.an ? y - s.a0 : s.an + y - s.b0;
    float4* row = x.cells + k * FIELDS * 64 + P.lane;
    if (r < R) {
      move_quad<BAND>(row, &f[r < R ? r : 0][0]);
      move_quad<BAND>(row + 32, &f[r < R ? r : 0][4]);
      if (FIELDS == 2) {
        move_quad<BAND>(row + 64, &f2[r < R ? r : 0][0]);
        move_quad<BAND>(row + 96, &f2[r < R ? r : 0][4]);
      }
    } else if (FIELDS == 2 && P.up) {
      move_quad<BAND>(row + 64, &f_top[0]);
      move_quad<BAND>(row + 96, &f_top[4]);
    }
  }
#pragma unroll
  for (int c = 0; c < 2; c++) {
    const bool left = P.left && l0 + c >= 0 && l0 + c < hq;
    const bool right = P.right && r0 + c >= 0 && r0 + c < hq;
    if (!left && !right) continue;
    float4* p = x.cells + s.rows * FIELDS + (P.yl * 2 * hq + (left ? l0 + c : hq + r0 + c)) * FIELDS;
#pragma unroll
    for (int r = 0; r < kRows; r++) {
      if (((owned >> r) & 1u) == 0u) continue;
      float4* at = p + r * 2 * hq * FIELDS;
      if (r < R) {
        move_quad<BAND>(at, &f[r < R ? r : 0][4 * c]);
        if (FIELDS == 2) move_quad<BAND>(at + 1, &f2[r < R ? r : 0][4 * c]);
      } else if (FIELDS == 2 && P.up) {
        move_quad<BAND>(at + 1, &f_top[4 * c]);
      }
    }
  }
}

// Place of an item's first field in the buffer, and the step to the second.
template <int FIELDS>
__device__ __forceinline__ float4* exchange_at(const Exchange& x, int rows, int it, int* step) {
  if (it < rows) {
    *step = 64;
    return x.cells + (it >> 6) * FIELDS * 64 + (it & 63);
  }
  *step = 1;
  return x.cells + it * FIELDS;
}

// One exchange of FIELDS fields f and f2 (f2 unused when FIELDS is 1). The cells
// go through shared memory, so that the packets are moved by loops of few
// instructions with every thread of the CTA on them, by places worked out
// once: as code unrolled over a patch's registers, of which only the warps and
// lanes at the edges use a part, an exchange took 14000 cycles, most of it
// instruction fetch.
template <int FIELDS, int R>
__device__ __forceinline__ void exchange(float (&f)[R][8], float (&f2)[R][8], float (&f_top)[8],
                                         char* base, const ResidentSync& sync, const RegTile& g,
                                         int W, int H, unsigned number) {
  const int64_t plane = packet_plane(W, H);
  constexpr int kPer = kPacketsPerQuad<FIELDS>;
  uint4* packets = sync.packets + (number & 1) * kPer * plane;
  // The band takes words that the last exchange's ring may still be read from:
  // a warp can be as many sweeps ahead of another as there are strips between
  // them, which may be more than lie between two exchanges.
  __syncthreads();
  {
    const Patch P = patch_of(g, R, W, H);
    exchange_patch<FIELDS, true, R>(f, f2, f_top, exchange_view(base, P, g, FIELDS), P, g);
  }
  __syncthreads();
  const Exchange x = exchange_view(base, patch_of(g, R, W, H), g, FIELDS);
#pragma unroll 1
  for (int it = threadIdx.x; it < x.band.items; it += blockDim.x) {
    const int place = x.send[it];
    if (place < 0) continue;
    int step;
    const float4* c = exchange_at<FIELDS>(x, x.band.rows, it, &step);
    uint4* p = packets + place;
    const float4 a = c[0];
    packet_out(true, p, a.x, a.y, a.z, number);
    if (FIELDS == 2) {
      const float4 b = c[step];
      packet_out(true, p + plane, a.w, b.x, b.y, number);
      packet_out(true, p + 2 * plane, b.z, b.w, 0.0f, number);
    } else {
      packet_out(true, p + plane, a.w, 0.0f, 0.0f, number);
    }
  }
  constexpr int kAtOnce = R == 4 || R == 6 ? 1 : 2;  // what those strips' registers leave
#pragma unroll 1
  for (int first = 0; first < x.ring.items; first += kAtOnce * blockDim.x) {
    float v[kAtOnce][9];
    const uint4* p[kAtOnce];
    int at[kAtOnce];
    bool on[kAtOnce], ok;
#pragma unroll
    for (int k = 0; k < kAtOnce; k++) {
      at[k] = first + k * blockDim.x + threadIdx.x;
      const int place = at[k] < x.ring.items ? x.take[at[k]] : -1;
      on[k] = place >= 0;
      p[k] = packets + max(place, 0);
    }
    int poll = 0;
    do {
      ok = true;
#pragma unroll
      for (int k = 0; k < kAtOnce; k++)
#pragma unroll
        for (int j = 0; j < kPer; j++)
          ok &= packet_in(on[k], p[k] + j * plane, v[k][3 * j], v[k][3 * j + 1], v[k][3 * j + 2],
                          number);
    } while (!ok && poll_again(poll++, sync));
    if (first == 0) __syncthreads();  // the band has been read: the buffer takes the ring
#pragma unroll
    for (int k = 0; k < kAtOnce; k++) {
      if (!on[k]) continue;
      int step;
      float4* c = exchange_at<FIELDS>(x, x.ring.rows, at[k], &step);
      c[0] = make_float4(v[k][0], v[k][1], v[k][2], v[k][3]);
      if (FIELDS == 2) c[step] = make_float4(v[k][4], v[k][5], v[k][6], v[k][7]);
    }
  }
  __syncthreads();
  const Patch P = patch_of(g, R, W, H);
  exchange_patch<FIELDS, false, R>(f, f2, f_top, exchange_view(base, P, g, FIELDS), P, g);
}

// With 16-bit storage the cells a tile keeps get the rounding that a store and
// a reload would give them, once per pass.
template <int R>
__device__ __forceinline__ void round_patch(float (&f)[R][8], int storage) {
  const HalfCells io{storage == OS_STORAGE_BF16};
#pragma unroll
  for (int r = 0; r < R; r++)
#pragma unroll
    for (int q = 0; q < 8; q++) f[r][q] = io.from(io.to(f[r][q]));
}
__device__ __forceinline__ void round_row(float (&f)[8], int storage) {
  const HalfCells io{storage == OS_STORAGE_BF16};
#pragma unroll
  for (int q = 0; q < 8; q++) f[q] = io.from(io.to(f[q]));
}

// ---------------------------------------------------------------------------
// Red/black projection.
// ---------------------------------------------------------------------------

// Flags of the region in shared memory: one word per row, column parity and
// lane, the flag bytes of columns 8 l + parity + {0, 2, 4, 6}, zero for cells
// the projection does not update.
__device__ __forceinline__ uint32_t active_flags(uint32_t w) {
  return w & (((w >> 5) & 0x01010101u) * 0xffu);  // F_ACTIVE is bit 5
}

// Flag byte of a cell with four fluid neighbours.
constexpr uint32_t kFullCell = F_FLUID | F_NBR_MASK | F_ACTIVE;
constexpr uint32_t kFullWord = kFullCell * 0x01010101u;

// What a lane of a strip knows about its cells (the same for all its rows).
struct ProjLane {
  bool wall_l;   // column 0 of the grid is the lane's first column
  bool wall_r;   // column W - 1 is the lane's last column
  bool closed_r; // and it is solid
  float rs_l, rs_r;  // reciprocal neighbour counts of the cells beside them
  bool idle;     // the strip is off the grid
  bool full;     // row_full takes every row of the strip
  bool wall;     // some lane of the warp has wall_l or wall_r
  bool own_first;  // no lane changes this lane's first face u from the left
};

// The pressure's share of an update (src/fluid.cu:225-226): one expression, so
// that the compiler rounds it the same way wherever it stands (it fuses the
// division's product with the sum; an update that is not taken is selected
// away, not masked before the sum).
__device__ __forceinline__ float add_pressure(float p, float vd, const Consts& c, float d_t) {
  return p + vd * c.density * (float)c.h / d_t;
}

// One row of a colour whose active cells have four fluid neighbours; with
// WALL, but for the columns at the grid's left and right edges (the grid's
// first or last column is not updated; the cell beside a solid one has three
// neighbours). A = first active column. A face that stays takes +0 off or -0
// on, without a branch, which leaves as it is every value but those that
// zeros_change keeps away from here. (Selected or predicated away instead: 257 and
// 246 us a step at 1920 x 1080 instead of 237.)
// The division by the count is a product with its reciprocal, which has the
// fast-math division's bits for every float input and every count (compared by
// tests/cpp/count_division.cu).
template <int A, bool PRESSURE, bool WALL>
__device__ __forceinline__ void row_full(float (&u)[8], float& ur, float (&vb)[8], float (&vt)[8],
                                         const ProjLane& L, const Consts& c, float d_t,
                                         float4* pw) {
  float4 p4 = make_float4(0.f, 0.f, 0.f, 0.f);
  if (PRESSURE) p4 = *pw;
  float* pp = &p4.x;
#pragma unroll
  for (int q = A; q < 8; q += 2) {
    float& right = (q == 7) ? ur : u[q < 7 ? q + 1 : 7];
    const float divergence = right - u[q] + vt[q] - vb[q];
    const float rs = !WALL ? 0.25f : q == 1 ? L.rs_l : q == 6 ? L.rs_r : 0.25f;
    const float vd = mul_rn(c.o, mul_rn(divergence, rs));
    const bool off = WALL && (q == 0 ? L.wall_l : q == 7 ? L.wall_r : false);
    const bool off_l = WALL && (q == 1 ? L.wall_l : off), off_r = WALL && (q == 6 ? L.closed_r : off);
    if (PRESSURE) {
      const float p = add_pressure(pp[q >> 1], vd, c, d_t);
      pp[q >> 1] = off ? pp[q >> 1] : p;
    }
    u[q] = u[q] + (off_l ? -0.0f : vd);
    right = right - (off_r ? 0.0f : vd);
    vb[q] = vb[q] + (off ? -0.0f : vd);
    vt[q] = vt[q] - (off ? 0.0f : vd);
  }
  if (PRESSURE) *pw = p4;
}

// x + y (x - y) where a bit of w is set, as a bit test and one predicated
// operation. (Masking y instead, a byte permute and a logic operation per
// face, took 1.5 times as long: those run at half the rate.)
template <uint32_t BIT>
__device__ __forceinline__ void add_if(float& x, float y, uint32_t w) {
  asm("{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n @p add.rn.ftz.f32 %0, %0, %1;\n}"
      : "+f"(x) : "f"(y), "r"(w & BIT));
}
template <uint32_t BIT>
__device__ __forceinline__ void sub_if(float& x, float y, uint32_t w) {
  asm("{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n @p sub.rn.ftz.f32 %0, %0, %1;\n}"
      : "+f"(x) : "f"(y), "r"(w & BIT));
}

// One cell of a row with any flags: byte q / 2 of the row's flag word.
template <int Q, bool PRESSURE>
__device__ __forceinline__ void cell_flags(uint32_t w, float rs, float& left, float& right,
                                           float& vb, float& vt, float& pc, const Consts& c,
                                           float d_t) {
  constexpr int sh = 8 * (Q >> 1);
  const float divergence = right - left + vt - vb;
  const float vd = mul_rn(c.o, mul_rn(divergence, rs));
  if (PRESSURE) {
    const float p = add_pressure(pc, vd, c, d_t);
    pc = w & ((uint32_t)F_FLUID << sh) ? p : pc;
  }
  add_if<(uint32_t)F_LEFT << sh>(left, vd, w);
  sub_if<(uint32_t)F_RIGHT << sh>(right, vd, w);
  add_if<(uint32_t)F_BOTTOM << sh>(vb, vd, w);
  sub_if<(uint32_t)F_TOP << sh>(vt, vd, w);
}

// One row of a colour with any flags. `w`: the row's flag word, `rs`: the
// reciprocal neighbour counts of its four cells.
template <int A, bool PRESSURE>
__device__ __forceinline__ void row_flags(uint32_t w, float4 rs, float (&u)[8], float& ur,
                                          float (&vb)[8], float (&vt)[8], const Consts& c,
                                          float d_t, float4* pw) {
  float4 p4 = make_float4(0.f, 0.f, 0.f, 0.f);
  if (PRESSURE) p4 = *pw;
  cell_flags<A, PRESSURE>(w, rs.x, u[A], u[A + 1], vb[A], vt[A], p4.x, c, d_t);
  cell_flags<A + 2, PRESSURE>(w, rs.y, u[A + 2], u[A + 3], vb[A + 2], vt[A + 2], p4.y, c, d_t);
  cell_flags<A + 4, PRESSURE>(w, rs.z, u[A + 4], u[A + 5], vb[A + 4], vt[A + 4], p4.z, c, d_t);
  cell_flags<A + 6, PRESSURE>(w, rs.w, u[A + 6], A ? ur : u[A ? 0 : 7], vb[A + 6], vt[A + 6],
                              p4.w, c, d_t);
  if (PRESSURE) *pw = p4;
}

// Shared memory of a projection tile after the warps' inboxes: the cells'
// reciprocal neighbour counts, (PRESSURE) the pressure and the flag words.
struct ProjSmem {
  float4* rs;        // [rows][2][32]
  float4* p;         // [rows][2][32]
  uint32_t* flags;   // [rows][2][32]
  char* exchange;
};

__host__ __device__ inline size_t project_tile_smem(int rows, int warps, bool pressure, int halo,
                                                    bool resident) {
  return (size_t)warps * inbox_bytes(4) +
         (size_t)rows * 64 * ((pressure ? 32 : 16) + 4) +
         (resident ? exchange_smem(halo, rows, 2) : 0);
}

__device__ __forceinline__ ProjSmem project_smem_of(char* base, int rows, int warps,
                                                    bool pressure) {
  ProjSmem s;
  s.rs = reinterpret_cast<float4*>(base + warps * inbox_bytes(4));
  s.p = s.rs + rows * 64;
  s.flags = reinterpret_cast<uint32_t*>(s.p + (pressure ? rows * 64 : 0));
  s.exchange = reinterpret_cast<char*>(s.flags + rows * 64);
  return s;
}

// 1 / s for the four cells of a flag word; 0 for a cell that is not updated.
__device__ __forceinline__ float4 reciprocal_counts(uint32_t w) {
  auto one = [](uint32_t f) {
    return f ? __fdividef(1.0f, (float)__popc(f & F_NBR_MASK)) : 0.0f;
  };
  return make_float4(one(w & 0xffu), one((w >> 8) & 0xffu), one((w >> 16) & 0xffu), one(w >> 24));
}

// The strip's flags: what row_full may take, and for a strip that it may not the
// flag words and reciprocal counts into shared memory (each lane's own).
// A lane wholly off the grid puts no condition: whatever its cells hold, no cell
// of the grid reads their faces.
template <int R>
__device__ __forceinline__ void flags_in(const uint8_t* __restrict__ flags, const Patch& P,
                                         const ProjSmem& sm, int W, int H, bool vec,
                                         ProjLane& L) {
  const int gx = P.gx0 + P.x0;
  const bool off = gx >= W;
  L.idle = P.idle;
  L.wall_l = gx == 0;
  L.wall_r = gx + 7 == W - 1;
  // What row_full takes in this lane: column 0 of the grid and its last column
  // are not updated, the cell beside column 0 has no fluid on its left, and
  // the cell beside the last column none on its right where that is solid.
  const uint32_t want_e = kFullWord & (L.wall_l ? 0xffffff00u : ~0u);
  const uint32_t want_e_closed = want_e & ~((uint32_t)F_RIGHT << 24);
  const uint32_t want_o = kFullWord & (L.wall_l ? ~(uint32_t)F_LEFT : ~0u) &
                          (L.wall_r ? 0x00ffffffu : ~0u);
  uint32_t open_e = 0u, closed_e = 0u, same_o = 0u;
  uint32_t raw[R][2];
  const uint8_t* row = flags + (int64_t)(H - 1 - (P.gy0 + P.y0)) * W + gx;
#pragma unroll
  for (int r = 0; r < R; r++, row -= W) {
    const bool on = P.gy0 + P.y0 + r < H;
    raw[r][0] = raw[r][1] = 0u;
    if (vec) {
#pragma unroll
      for (int k = 0; k < 2; k++)
        asm("{\n .reg .pred p;\n setp.ne.s32 p, %2, 0;\n @p ld.global.nc.u32 %0, [%1];\n}"
            : "+r"(raw[r][k]) : "l"(row + 4 * k), "r"((int)(on && gx + 4 * k < W)));
    } else {
#pragma unroll
      for (int d = 0; d < 8; d++) {
        uint16_t b = 0;
        asm("{\n .reg .pred p;\n setp.ne.s32 p, %2, 0;\n @p ld.global.nc.u8 %0, [%1];\n}"
            : "+h"(b) : "l"(row + d), "r"((int)(on && gx + d < W)));
        raw[r][d >> 2] |= (uint32_t)b << (8 * (d & 3));
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R; r++) {
    uint32_t lo = raw[r][0], hi = raw[r][1];
    lo = active_flags(lo), hi = active_flags(hi);
    const uint32_t ev = __byte_perm(lo, hi, 0x6420), od = __byte_perm(lo, hi, 0x7531);
    raw[r][0] = ev, raw[r][1] = od;
    const uint32_t bit = 1u << r;
    if (off || ev == want_e) open_e |= bit;
    if (off || (L.wall_r && ev == want_e_closed)) closed_e |= bit;
    if (off || od == want_o) same_o |= bit;
  }
  L.closed_r = L.wall_r && closed_e != 0u;
  L.own_first = P.lane == 0 || L.wall_l;
  L.wall = __any_sync(kAllLanes, L.wall_l || L.wall_r);
  L.rs_l = __fdividef(1.0f, L.wall_l ? 3.0f : 4.0f);
  L.rs_r = __fdividef(1.0f, L.closed_r ? 3.0f : 4.0f);
  L.full = __all_sync(kAllLanes, ((L.closed_r ? closed_e : open_e) & same_o) == (1u << R) - 1u);
  if (L.full) return;
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int e = (P.yl + r) * 64 + P.lane;
    sm.flags[e] = raw[r][0];
    sm.flags[e + 32] = raw[r][1];
    sm.rs[e] = reciprocal_counts(raw[r][0]);
    sm.rs[e + 32] = reciprocal_counts(raw[r][1]);
  }
}

// Faces that stay hold what they hold, but row_full adds zeros to those beside the
// grid's left and right edges, which flushes a value below the smallest normal
// number and makes one NaN of all. Whether it would change one of this strip,
// which then goes by its flags. (A kernel's code is fetched cold once per launch:
// an addition and a logic operation a face, where a test of its exponent took 0.5
// us of every launch at 256 x 128.)
template <int R>
__device__ __forceinline__ bool zeros_change(const float (&u)[R][8], const float (&v)[R][8],
                                             const float (&vt)[8], const ProjLane& L) {
  if (!L.full || !L.wall) return false;  // the same for the warp
  float zero = -0.0f;
  asm volatile("" : "+f"(zero));  // the compiler takes x + -0 for x
  auto changed = [&](float x) { return __float_as_uint(x + zero) ^ __float_as_uint(x); };
  uint32_t left = changed(vt[0]), right = changed(vt[7]);
#pragma unroll
  for (int r = 0; r < R; r++) {
    left |= changed(u[r][0]) | changed(u[r][1]) | changed(v[r][0]);
    right |= changed(u[r][7]) | changed(v[r][7]);
  }
  return __any_sync(kAllLanes, (L.wall_l && left) || (L.wall_r && right));
}
// The flag words and counts of a strip that flags_in took for full.
static __device__ __noinline__ void flags_late(const uint8_t* flags, const Patch P,
                                               const ProjSmem sm, int W, int H, int R) {
  const int gx = P.gx0 + P.x0;
#pragma unroll 1
  for (int r = 0; r < R; r++) {
    const uint8_t* row = flags + (int64_t)(H - 1 - (P.gy0 + P.y0 + r)) * W + gx;
#pragma unroll 1
    for (int k = 0; k < 2; k++) {
      uint32_t w = 0u;
#pragma unroll 1
      for (int d = 0; d < 4; d++)
        if (P.gy0 + P.y0 + r < H && gx + 2 * d + k < W)
          w |= active_flags((uint32_t)__ldg(row + 2 * d + k)) << (8 * d);
      const int e = (P.yl + r) * 64 + 32 * k + P.lane;
      sm.flags[e] = w;
      sm.rs[e] = reciprocal_counts(w);
    }
  }
}

// The face between two lanes that a row's update changed, to the lane that did
// not change it: with active columns 0, 2, .. the lane's own first face, with
// columns 1, 3, .. the face beyond its last column (u(0) of the grid belongs
// to no cell that is updated).
template <int A>
__device__ __forceinline__ void row_share(float (&u)[8], float& ur, const ProjLane& L) {
  if (A == 0) {
    ur = __shfl_down_sync(kAllLanes, u[0], 1);
  } else {
    const float t = __shfl_up_sync(kAllLanes, ur, 1);
    u[0] = L.own_first ? u[0] : t;
  }
}

// How a strip's cells are taken, by what its flags say: all full and away from
// the grid's left and right edges, all full, or by the flags. Each has a sweep
// loop of its own, so that no loop holds the registers of another's rows.
enum class Rows { kPlain, kWall, kFlags };

// Row r of a strip in one colour's half-sweep, and the face it shares with the
// neighbouring lane.
template <int COLOUR, bool PRESSURE, Rows ROWS, int R>
__device__ __forceinline__ void strip_row(int r, float (&u)[R][8], float (&v)[R][8],
                                          float (&ur)[R], float (&vt)[8], const ProjLane& L,
                                          const ProjSmem& sm, int cell0, const Consts& c,
                                          float d_t) {
  float(&top)[8] = r + 1 < R ? v[r + 1 < R ? r + 1 : 0] : vt;
  const int e = cell0 + r * 64 + ((r + COLOUR) & 1) * 32;
  float4* p = PRESSURE ? sm.p + e : nullptr;
  constexpr bool full = ROWS != Rows::kFlags;
  if ((r + COLOUR) & 1) {
    if (full)
      row_full<1, PRESSURE, ROWS != Rows::kPlain>(u[r], ur[r], v[r], top, L, c, d_t, p);
    else
      row_flags<1, PRESSURE>(sm.flags[e], sm.rs[e], u[r], ur[r], v[r], top, c, d_t, p);
    row_share<1>(u[r], ur[r], L);
  } else {
    if (full)
      row_full<0, PRESSURE, ROWS != Rows::kPlain>(u[r], ur[r], v[r], top, L, c, d_t, p);
    else
      row_flags<0, PRESSURE>(sm.flags[e], sm.rs[e], u[r], ur[r], v[r], top, c, d_t, p);
    row_share<0>(u[r], ur[r], L);
  }
}

// The faces on a strip's edges after a half-sweep, 4 words each way: a strip
// sends those its half-sweep changed, and receives those its neighbours
// changed.
template <int COLOUR, int R>
__device__ __forceinline__ void strip_send(const float (&v)[R][8], const float (&vt)[8],
                                           const Link<4>& link, unsigned m) {
  constexpr int cb = COLOUR, ct = (COLOUR + R - 1) & 1;  // of the bottom and the top row
  post<4>(link.up, link.up_part, m, 0, make_float4(vt[ct], vt[ct + 2], vt[ct + 4], vt[ct + 6]));
  post<4>(link.down, link.down_part, m, 0,
          make_float4(v[0][cb], v[0][cb + 2], v[0][cb + 4], v[0][cb + 6]));
}

template <int COLOUR, int R>
__device__ __forceinline__ void strip_receive(float (&v)[R][8], float (&vt)[8],
                                              Link<4>& link, unsigned m, bool down,
                                              const ResidentSync& sync) {
  constexpr int nb = 1 - COLOUR, nt = 1 - ((COLOUR + R - 1) & 1);
  await_message(link, m, sync);
  const float4 b = read_message(link, 0, m, 0), t = read_message(link, 1, m, 0);
  // Without a strip above, the top face is one that nothing owned depends on;
  // without a strip below, the bottom face stays.
  vt[nt] = t.x, vt[nt + 2] = t.y, vt[nt + 4] = t.z, vt[nt + 6] = t.w;
  v[0][nb] = down ? b.x : v[0][nb], v[0][nb + 2] = down ? b.y : v[0][nb + 2];
  v[0][nb + 4] = down ? b.z : v[0][nb + 4], v[0][nb + 6] = down ? b.w : v[0][nb + 6];
}

// A half-sweep: the strip's inner rows, then (while those ran, the last
// half-sweep's faces came in) its first and last row, whose faces go out. The
// rows of a colour share no face, so their order is free. Message m comes in,
// m + 1 goes out.
template <int COLOUR, bool PRESSURE, Rows ROWS, int R>
__device__ __forceinline__ void half_sweep(float (&u)[R][8], float (&v)[R][8], float (&ur)[R],
                                           float (&vt)[8], const ProjLane& L, const ProjSmem& sm,
                                           Link<4>& link, const ResidentSync& sync,
                                           int cell0, bool down, unsigned m, const Consts& c,
                                           float d_t) {
#pragma unroll
  for (int r = 1; r < R - 1; r++)
    strip_row<COLOUR, PRESSURE, ROWS, R>(r, u, v, ur, vt, L, sm, cell0, c, d_t);
  strip_receive<1 - COLOUR, R>(v, vt, link, m, down, sync);
  strip_row<COLOUR, PRESSURE, ROWS, R>(0, u, v, ur, vt, L, sm, cell0, c, d_t);
  strip_row<COLOUR, PRESSURE, ROWS, R>(R - 1, u, v, ur, vt, L, sm, cell0, c, d_t);
  strip_send<COLOUR, R>(v, vt, link, m + 1);
}

template <bool PRESSURE, Rows ROWS, int R>
__device__ __forceinline__ void sweep_loop(float (&u)[R][8], float (&v)[R][8], float (&ur)[R],
                                           float (&vt)[8], const ProjLane& L, const ProjSmem& sm,
                                           Link<4>& link, const ResidentSync& sync,
                                           int cell0, bool down, const Consts& c, float d_t,
                                           int sweeps, unsigned m) {
#pragma unroll 1
  for (int t = 0; t < sweeps && !link.lost; t++, m += 2) {
    half_sweep<0, PRESSURE, ROWS, R>(u, v, ur, vt, L, sm, link, sync, cell0, down, m, c, d_t);
    half_sweep<1, PRESSURE, ROWS, R>(u, v, ur, vt, L, sm, link, sync, cell0, down, m + 1, c, d_t);
  }
}

// Messages of a segment of sweeps.
__host__ __device__ inline unsigned project_messages(int sweeps) { return 2 * sweeps + 1; }

// `sweeps` red/black sweeps of the region, messages m .. m + 2 sweeps. Every
// cell of the region is updated: validity shrinks by one cell per half-sweep
// from the edges that have a halo, and a cell beyond writes faces that only
// cells beyond read from then on.
template <bool PRESSURE, int R>
__device__ __forceinline__ void tile_sweeps(float (&u)[R][8], float (&v)[R][8], float (&vt)[8],
                                            const ProjLane& L, const ProjSmem& sm,
                                            Link<4>& link, const ResidentSync& sync,
                                            int cell0, bool down, const Consts& c, float d_t,
                                            int sweeps, unsigned m) {
  static_assert(R % 2 == 0, "strips start on even rows");
  if (link.lost) return;
  if (L.idle) return idle_messages(link, m, project_messages(sweeps), sync);
  float ur[R];
#pragma unroll
  for (int r = 0; r < R; r++) ur[r] = __shfl_down_sync(kAllLanes, u[r][0], 1);
  // The faces as they are, for the first half-sweep to receive.
  strip_send<1, R>(v, vt, link, m);
  if (!L.full)
    sweep_loop<PRESSURE, Rows::kFlags, R>(u, v, ur, vt, L, sm, link, sync, cell0, down, c, d_t,
                                          sweeps, m);
  else if (L.wall)
    sweep_loop<PRESSURE, Rows::kWall, R>(u, v, ur, vt, L, sm, link, sync, cell0, down, c, d_t,
                                         sweeps, m);
  else
    sweep_loop<PRESSURE, Rows::kPlain, R>(u, v, ur, vt, L, sm, link, sync, cell0, down, c, d_t,
                                          sweeps, m);
  if (!link.lost) strip_receive<1, R>(v, vt, link, m + 2 * sweeps, down, sync);
}

// apply_extrapolation_at (src/fluid.cu:720-733) on a patch, in
// extrapolate_grid's order (the rows' rules, then the columns'): each rule
// reads a cell of the thread that holds its target or of the lane before, but
// for u(i, H - 1) = u(i, H - 2), which the thread of row H - 2 stores (the tile
// that owns one of the two rows owns both).
template <int R>
__device__ __forceinline__ void extrapolate_patch(float (&u)[R][8], float (&v)[R][8],
                                                  const Patch& P, int W) {
  if (P.gy0 + P.y0 == 0) {
#pragma unroll
    for (int q = 0; q < 8; q++) {
      u[0][q] = u[1][q];
      v[1][q] = 0.0f;
    }
  }
  const int gx = P.gx0 + P.x0;
  if (gx == 0) {
#pragma unroll
    for (int r = 0; r < R; r++) {
      v[r][0] = v[r][1];
      u[r][1] = 0.0f;
    }
  }
  const int last = W - 1 - gx;  // the last column's place in the patch
#pragma unroll
  for (int r = 0; r < R; r++) {
    const float before = __shfl_up_sync(kAllLanes, v[r][7], 1);
#pragma unroll
    for (int q = 0; q < 8; q++)
      if (last == q) v[r][q] = q ? v[r][q ? q - 1 : 0] : before;
  }
}

// The owned cells out to fields uo and vo, extrapolated where asked.
template <int R>
__device__ __forceinline__ void faces_out(float (&u)[R][8], float (&v)[R][8], void* uo, void* vo,
                                          int storage, const Patch& P, int W, int H, float* stage,
                                          bool extrapolate) {
  const uint32_t own = rows_in(P.y0, R, P.oy0, P.oy1);
  uint32_t own_u = own, top = 0u;
  if (extrapolate) {
    extrapolate_patch<R>(u, v, P, W);
    own_u &= ~rows_in(P.y0, R, H - 1 - P.gy0, H - P.gy0);
    top = own & rows_in(P.y0, R, H - 2 - P.gy0, H - 1 - P.gy0);
  }
  on_cells(storage, [&](auto io) {
    patch_out<R>(io, u, uo, P, own_u, W, H, stage);
    patch_out<R>(io, v, vo, P, own, W, H, stage);
    if (top)  // row H - 2 of u to row H - 1, which lies one row before it
      patch_out<R>(io, u, static_cast<typename decltype(io)::Word*>(uo) - W, P, top, W, H, stage);
  });
}

// The pressure of the owned cells, between its field and the tile's planes.
template <int R>
__device__ __forceinline__ void pressure_in(const ProjSmem& sm, const float* p, const Patch& P,
                                            int W, bool zero, int H, float* stage) {
  float f[R][8];
#pragma unroll
  for (int r = 0; r < R; r++)
#pragma unroll
    for (int q = 0; q < 8; q++) f[r][q] = 0.0f;
  const int lo = P.ox0 - P.x0, hi = P.ox1 - P.x0;
  const uint32_t own = zero ? 0u : rows_in(P.y0, R, P.oy0, P.oy1);
  const float* row =
      p + (int64_t)(H - 1 - (P.gy0 + P.y0)) * W + P.gx0 + (stage ? P.lane : P.x0);
  const F32Cells io;
#pragma unroll
  for (int r = 0; r < R; r++, row -= W) {
    const bool on = (own >> r) & 1u;
    if (!stage) {
      io.load4(on && 0 >= lo && 0 < hi, row, &f[r][0]);
      io.load4(on && 4 >= lo && 4 < hi, row + 4, &f[r][4]);
    } else {
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const int x = P.lane + 32 * k;
        io.load1(on && x >= P.ox0 && x < P.ox1, row + 32 * k, &f[r][k]);
      }
    }
  }
  if (stage && own) {
#pragma unroll
    for (int r = 0; r < R; r++) turn_in(io, f[r], stage, P.lane);
  }
#pragma unroll
  for (int r = 0; r < R; r++) {
    float4* out = sm.p + (P.yl + r) * 64 + P.lane;
    out[0] = make_float4(f[r][0], f[r][2], f[r][4], f[r][6]);
    out[32] = make_float4(f[r][1], f[r][3], f[r][5], f[r][7]);
  }
}

template <int R>
__device__ __forceinline__ void pressure_out(const ProjSmem& sm, float* p, const Patch& P, int W,
                                             int H, float* stage) {
  float f[R][8];
#pragma unroll
  for (int r = 0; r < R; r++) {
    const float4* in = sm.p + (P.yl + r) * 64 + P.lane;
    const float4 e = in[0], o = in[32];
    f[r][0] = e.x, f[r][2] = e.y, f[r][4] = e.z, f[r][6] = e.w;
    f[r][1] = o.x, f[r][3] = o.y, f[r][5] = o.z, f[r][7] = o.w;
  }
  patch_out<R>(F32Cells{}, f, p, P, rows_in(P.y0, R, P.oy0, P.oy1), W, H, stage);
}

// The sweeps from `done` on that run without a break, and what comes before
// them: with 16-bit storage the rounding after every K sweeps, and in a launch
// that exchanges (n > D) the ring after every D. A rounding needs no exchange: a
// tile rounds its copies of its neighbours' cells as they round theirs, and the
// halo is as wide as D sweeps need. (With an exchange at each rounding, K = 4 and
// D = 20 left 4 messages between two exchanges, and halos of 10 strips.)
struct Segment {
  int sweeps;
  bool round, exchange;
};
__host__ __device__ inline Segment segment_at(int n, int K, int D, int done, int storage) {
  const bool rounded = storage != OS_STORAGE_F32;
  Segment s;
  s.sweeps = n - done < D - done % D ? n - done : D - done % D;
  if (rounded && K - done % K < s.sweeps) s.sweeps = K - done % K;
  s.round = rounded && done > 0 && done % K == 0;
  s.exchange = n > D && done > 0 && done % D == 0;
  return s;
}

struct ProjectArgs {
  const void *ui, *vi;      // the copies of the fields that are loaded
  void *uo, *vo;            // the other copies, which take the result
  int storage;
  float* p;
  const uint8_t* flags;
  Consts c;
  const StepParams* prm;
  int n, K, D;              // sweeps in all, per pass, and between exchanges
  RegTile g;
  ResidentSync sync;        // only used when n > D
  int zero_pressure, extrapolate;
};

// n sweeps with the tile in registers throughout, and the ring exchanged after
// every D of them (the halo is 2 D cells). With n <= D no CTA waits for another,
// and the launch may hold any number of tiles; else all tiles must be resident
// together (a cooperative launch). The result is that of ceil(n / K) passes of
// K sweeps through memory: with 16-bit storage the fields are rounded after
// every K sweeps. It goes to the other copy of the fields, however many passes
// that stands for: nothing orders a tile's stores behind the loads of the halos
// of the tiles around it (they may not have started yet).
template <int R, bool PRESSURE, bool ALIGNED>
__global__ void __launch_bounds__(32 * project_max_warps(R), 1)
k_project_tiles(const __grid_constant__ ProjectArgs a) {
  extern __shared__ __align__(16) char tile_smem[];
  const Consts& c = a.c;
  const int W = c.W, H = c.H, rows = a.g.warps * R;
  const Patch P = patch_of(a.g, R, W, H);
  const ProjSmem sm = project_smem_of(tile_smem, rows, a.g.warps, PRESSURE);
  Link<4> link = open_link<4>(tile_smem, P, a.g);
  cluster_arrive();
  float* const stage = ALIGNED ? nullptr : stage_of(tile_smem, a.g);
  ProjLane L;
  // The flags do not change after creation: staged before the wait for the
  // kernel before.
  flags_in<R>(a.flags, P, sm, W, H, ALIGNED, L);
  pdl_entry();
  float u[R][8], v[R][8], vt[8];
#pragma unroll
  for (int r = 0; r < R; r++)
#pragma unroll
    for (int q = 0; q < 8; q++) u[r][q] = v[r][q] = 0.0f;
#pragma unroll
  for (int q = 0; q < 8; q++) vt[q] = 0.0f;
  const float d_t = a.prm->dt;
  on_cells(a.storage, [&](auto io) {
    patch_in<R>(io, u, a.ui, P, W, H, stage);
    patch_in<R>(io, v, a.vi, P, W, H, stage);
    if (P.up) row_in(io, vt, a.vi, P, P.y0 + R, W, H, stage);
  });
  if (zeros_change<R>(u, v, vt, L)) {
    L.full = false;
    flags_late(a.flags, patch_of(a.g, R, W, H), sm, W, H, R);
  }
  const unsigned epoch = a.n > a.D ? ld_acquire_gpu(a.sync.epochs + blockIdx.x) : 0u;
  unsigned number = epoch;
  if (a.n > a.D) exchange_plan(sm.exchange, a.g, R, 2, W, H);
  // (Behind the faces, and with its own patch: ahead of them the sweeps spilled.)
  if (PRESSURE) pressure_in<R>(sm, a.p, patch_of(a.g, R, W, H), W, a.zero_pressure, H, stage);
  cluster_wait();  // every inbox of the cluster is open
  if (!clusters_of(a.g.cluster, a.sync)) return;
  unsigned message = 0;
#pragma unroll 1
  for (int done = 0; done < a.n;) {
    const Segment s = segment_at(a.n, a.K, a.D, done, a.storage);
    if (s.round) {
      round_patch<R>(u, a.storage);
      round_patch<R>(v, a.storage);
      round_row(vt, a.storage);
    }
    if (s.exchange) {
      number++;
      exchange<2, R>(u, v, vt, sm.exchange, a.sync, a.g, W, H, number);
    }
    // (High strips have no registers to keep the patch in: 1920 x 1080 with the
    // pressure takes 320 us so, and 340 us with it kept; 640 x 448, with strips of
    // two rows, 1.4% longer with it worked out anew.)
    const Patch S = R >= 6 ? patch_of(a.g, R, W, H) : P;
    tile_sweeps<PRESSURE, R>(u, v, vt, L, sm, link, a.sync, S.yl * 64 + S.lane, S.down, c, d_t,
                             s.sweeps, message);
    message += project_messages(s.sweeps);
    done += s.sweeps;
  }
  if (number != epoch && threadIdx.x == 0) a.sync.epochs[blockIdx.x] = number;
  const Patch Q = patch_of(a.g, R, W, H);
  float* const out = ALIGNED ? nullptr : stage_of(tile_smem, a.g);
  faces_out<R>(u, v, a.uo, a.vo, a.storage, Q, W, H, out, a.extrapolate != 0);
  if (PRESSURE) pressure_out<R>(sm, a.p, Q, W, H, out);
  cluster_arrive();  // no CTA leaves while another may still send to it
  cluster_wait();
}

// ---------------------------------------------------------------------------
// Jacobi diffusion of u (apply_diffusion_at, src/fluid.cu:176-183).
// ---------------------------------------------------------------------------

// Shared memory of a diffusion tile: the warps' inboxes and the exchange.
__host__ __device__ inline size_t diffuse_tile_smem(int rows, int warps, int halo, bool resident) {
  return (size_t)warps * inbox_bytes(8) + (resident ? exchange_smem(halo, rows, 1) : 0);
}

// How a strip's cells are taken: no row or column of it kept, the columns 0, 3
// and 7 of its lanes where DiffLane says so, or any row or column, and the
// division may be one.
enum class Kept { kNone, kQuadEdges, kAny };

// What a patch holds that no sweep changes: the grid's first and last column
// (bit q of `cols`: column q of the lane) and row (bit r of `rows`, the same in
// the warp).
struct DiffLane {
  uint32_t cols, rows;
};
constexpr uint32_t kIdleRows = ~0u;  // DiffLane::rows of a strip off the grid
__device__ __forceinline__ DiffLane diff_lane(const Patch& P, int R, int W, int H) {
  DiffLane L;
  const int gx = P.gx0 + P.x0, gy = P.gy0 + P.y0;
  L.cols = (gx == 0 ? 1u : 0u) | (W - 1 - gx >= 0 && W - 1 - gx < 8 ? 1u << (W - 1 - gx) : 0u);
  L.rows = (gy == 0 ? 1u : 0u) | (H - 1 - gy >= 0 && H - 1 - gy < R ? 1u << (H - 1 - gy) : 0u);
  if (P.idle) L.rows = kIdleRows;
  return L;
}

// One row of a sweep in place: `down` holds the old row below and takes the old
// row itself, `up` is the old row above.
template <Kept KEPT>
__device__ __forceinline__ void jacobi_row(float (&u)[8], float (&down)[8], const float (&up)[8],
                                           int r, const DiffLane& L, float a, float den,
                                           float rden, bool rcp) {
  float left = __shfl_up_sync(kAllLanes, u[7], 1);
  const float right = __shfl_down_sync(kAllLanes, u[0], 1);
  uint32_t kept = L.cols;
  if (KEPT == Kept::kAny) {
    // (Worked out in each sweep: hoisted, the rows' and columns' conditions
    // are more than the seven predicates there are.)
    asm volatile("{\n .reg .s32 m;\n bfe.s32 m, %1, %2, 1;\n or.b32 %0, %0, m;\n}"
                 : "+r"(kept) : "r"(L.rows), "r"(r));
  }
#pragma unroll
  for (int q = 0; q < 8; q++) {
    const float old = u[q];
    const float rt = q < 7 ? u[q < 7 ? q + 1 : 7] : right;
    // src/fluid.cu:178-182: neighbours (i-1, j), (i+1, j), (i, j-1), (i, j+1)
    const float x = fma_rn(a, left + rt + down[q] + up[q], old);
    float y = KEPT != Kept::kAny || rcp ? mul_rn(x, rden) : x / den;
    if (KEPT == Kept::kAny || (KEPT == Kept::kQuadEdges && (q == 0 || q == 3 || q == 7)))
      y = (kept >> q) & 1u ? old : y;
    u[q] = y;
    down[q] = left = old;
  }
}

// The strip's first and last row to the strips below and above, message m.
template <int R>
__device__ __forceinline__ void rows_send(const float (&u)[R][8], const Link<8>& link,
                                          unsigned m) {
#pragma unroll
  for (int k = 0; k < 2; k++) {
    post<8>(link.down, link.down_part, m, k,
            make_float4(u[0][4 * k], u[0][4 * k + 1], u[0][4 * k + 2], u[0][4 * k + 3]));
    post<8>(link.up, link.up_part, m, k,
            make_float4(u[R - 1][4 * k], u[R - 1][4 * k + 1], u[R - 1][4 * k + 2],
                        u[R - 1][4 * k + 3]));
  }
}
__device__ __forceinline__ void row_receive(float (&f)[8], const Link<8>& link, int part,
                                            unsigned m) {
  const float4 x = read_message(link, part, m, 0), y = read_message(link, part, m, 1);
  f[0] = x.x, f[1] = x.y, f[2] = x.z, f[3] = x.w;
  f[4] = y.x, f[5] = y.y, f[6] = y.z, f[7] = y.w;
}

template <int R, Kept KEPT>
__device__ __forceinline__ void jacobi_loop(float (&u)[R][8], Link<8>& link,
                                            const ResidentSync& sync, const DiffLane& L, float a,
                                            float den, float rden, bool rcp, int sweeps,
                                            unsigned m) {
#pragma unroll 1
  for (int t = 0; t < sweeps && !link.lost; t++, m++) {
    rows_send<R>(u, link, m);
    // The inner rows first, while the neighbours' rows come in.
    float down[8], second[8], row[8];
#pragma unroll
    for (int q = 0; q < 8; q++) down[q] = u[0][q], second[q] = u[1][q];
#pragma unroll
    for (int r = 1; r < R - 1; r++)
      jacobi_row<KEPT>(u[r], down, u[r + 1], r, L, a, den, rden, rcp);
    await_message(link, m, sync);
    row_receive(row, link, 1, m);
    jacobi_row<KEPT>(u[R - 1], down, row, R - 1, L, a, den, rden, rcp);
    row_receive(row, link, 0, m);
    jacobi_row<KEPT>(u[0], row, second, 0, L, a, den, rden, rcp);
  }
}

// `sweeps` sweeps of the region, messages m .. m + sweeps - 1. A row without a
// strip beyond it is the grid's first or last, which is kept, or further than
// the sweeps reach from the owned rows.
template <int R>
__device__ __forceinline__ void jacobi_sweeps(float (&u)[R][8], const DiffLane& L,
                                              Link<8>& link, const ResidentSync& sync,
                                              float a, int sweeps, unsigned m) {
  const float den = fma_rn(4.0f, a, 1.0f);
  const float rden = __fdividef(1.0f, den);
  // The division by den as the product with its reciprocal: the same bits for
  // every float input (tests/cpp/reciprocal_product.cu), used below 2^20.
  const bool rcp = den < 1048576.0f;
  const uint32_t cols = __reduce_or_sync(kAllLanes, L.cols);
  if (L.rows == kIdleRows)
    idle_messages(link, m, sweeps, sync);
  else if (!rcp || L.rows || (cols & ~0x89u))
    jacobi_loop<R, Kept::kAny>(u, link, sync, L, a, den, rden, rcp, sweeps, m);
  else if (cols)
    jacobi_loop<R, Kept::kQuadEdges>(u, link, sync, L, a, den, rden, true, sweeps, m);
  else
    jacobi_loop<R, Kept::kNone>(u, link, sync, L, a, den, rden, true, sweeps, m);
}

struct DiffuseArgs {
  const void* ui;  // the copy of the field that is loaded
  void* uo;        // the other copy, which takes the result
  int storage;
  Consts c;
  const StepParams* prm;
  int n, K, D;    // sweeps in all, per pass, and between exchanges
  RegTile g;
  ResidentSync sync;
};

// As k_project_tiles, with a halo of D cells.
template <int R, bool ALIGNED>
__global__ void __launch_bounds__(32 * diffuse_max_warps(R), 1)
k_diffuse_tiles(const __grid_constant__ DiffuseArgs a) {
  extern __shared__ __align__(16) char tile_smem[];
  const Consts& c = a.c;
  const int W = c.W, H = c.H;
  const Patch P = patch_of(a.g, R, W, H);
  Link<8> link = open_link<8>(tile_smem, P, a.g);
  cluster_arrive();
  float* const stage = ALIGNED ? nullptr : stage_of(tile_smem, a.g);
  pdl_entry();
  float u[R][8], none[8];
#pragma unroll
  for (int r = 0; r < R; r++)
#pragma unroll
    for (int q = 0; q < 8; q++) u[r][q] = 0.0f;
  on_cells(a.storage, [&](auto io) { patch_in<R>(io, u, a.ui, P, W, H, stage); });
  const DiffLane L = diff_lane(P, R, W, H);
  const float coeff = diffusion_coeff<float>(c, a.prm->dt);
  const unsigned epoch = a.n > a.D ? ld_acquire_gpu(a.sync.epochs + blockIdx.x) : 0u;
  unsigned number = epoch;
  if (a.n > a.D) exchange_plan(tile_smem + a.g.warps * inbox_bytes(8), a.g, R, 1, W, H);
  cluster_wait();  // every inbox of the cluster is open
  if (!clusters_of(a.g.cluster, a.sync)) return;
  unsigned message = 0;
#pragma unroll 1
  for (int done = 0; done < a.n;) {
    const Segment s = segment_at(a.n, a.K, a.D, done, a.storage);
    if (s.round) round_patch<R>(u, a.storage);
    if (s.exchange) {
      number++;
      exchange<1, R>(u, u, none, tile_smem + a.g.warps * inbox_bytes(8), a.sync, a.g, W, H,
                     number);
    }
    jacobi_sweeps<R>(u, L, link, a.sync, coeff, s.sweeps, message);
    message += s.sweeps;
    done += s.sweeps;
  }
  if (number != epoch && threadIdx.x == 0) a.sync.epochs[blockIdx.x] = number;
  const Patch Q = patch_of(a.g, R, W, H);
  float* const out = ALIGNED ? nullptr : stage_of(tile_smem, a.g);
  on_cells(a.storage, [&](auto io) {
    patch_out<R>(io, u, a.uo, Q, rows_in(Q.y0, R, Q.oy0, Q.oy1), W, H, out);
  });
  cluster_arrive();  // no CTA leaves while another may still send to it
  cluster_wait();
}

using ProjectKernel = void (*)(const ProjectArgs);
using DiffuseKernel = void (*)(const DiffuseArgs);

// The kernels of one strip height, each instantiated in a translation unit of
// its own (os_tile_project.cu, os_tile_diffuse.cu).
template <int R> ProjectKernel project_kernel(bool pressure, bool aligned);
template <int R> DiffuseKernel diffuse_kernel(bool aligned);

}  // namespace osg
