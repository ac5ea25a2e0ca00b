// os_tile.cuh — tiles held in registers: the red/black projection and the
// Jacobi diffusion with every face of a tile in the registers of its CTA from
// the first sweep of a pass to the last.
//
// A tile's region is 256 columns wide and RH = R * warps rows high. Warp w
// holds the strip of rows [w R, (w + 1) R), lane l its columns 8 l .. 8 l + 7:
// a patch of 8 x R cells per thread. The region of tile (tx, ty) starts at
// cell (tx * TX, ty * TY); it carries `halo` cells on each side that has a
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
// between strips (two 16-byte stores and loads).
//
// Updates are the plain kernels' expressions in the same order, so every
// result has the same bits.
#pragma once

namespace osg {

constexpr int kTileW = 256;      // region width in cells
constexpr int kLaneCols = 8;     // columns per lane
constexpr int kMaxTileWarps = 24;
constexpr uint32_t kAllLanes = 0xffffffffu;

// Warps per CTA that the register file holds for strips of R rows.
constexpr int tile_max_warps(int R) {
  return R <= 2 ? 24 : R <= 4 ? 16 : R <= 6 ? 12 : 8;
}

// The same for the diffusion, which holds one field and two rows of neighbours.
constexpr int diffuse_max_warps(int R) {
  return R <= 2 ? 24 : R <= 4 ? 16 : R <= 8 ? 12 : 8;
}

struct RegTile {
  int halo;              // halo in cells, on sides that have a neighbour
  int TX, TY;            // pitch of the tiles: region minus both halos
  int RH;                // region rows, R * warps
  int R, warps;
  int tiles_x, tiles_y;
  size_t smem;
};

struct ResidentSync {
  unsigned* epochs;     // one per tile: passes exchanged so far (monotonic)
  uint4* packets;       // two copies of the exchanged cells (see the exchange below)
  int* dev_err;         // set by a warp that gave up; polled by the others
  int* host_err;        // mapped host word the host reads after synchronising
};

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
  __device__ __forceinline__ void load1(bool on, const uint16_t* p, float* q) const {
    uint16_t a = 0;
    asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %2, 0;\n @p ld.global.cg.u16 %0, [%1];\n}"
                 : "+h"(a) : "l"(p), "r"((int)on) : "memory");
    *q = on ? from(a) : *q;
  }
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
  int tx, ty;      // tile
  int gx0, gy0;    // region origin on the grid
  int lane, warp;
  int x0, y0;      // first column and row of the patch in the region
  bool left, right, below, above;  // the tile has a neighbour on that side
  int ox0, ox1, oy0, oy1;          // owned columns and rows, in the region
};

__device__ __forceinline__ Patch patch_of(int tx, int ty, const RegTile& g, int R, int W, int H) {
  Patch P;
  P.tx = tx, P.ty = ty;
  P.gx0 = tx * g.TX, P.gy0 = ty * g.TY;
  P.lane = threadIdx.x & 31, P.warp = threadIdx.x >> 5;
  P.x0 = P.lane * kLaneCols, P.y0 = P.warp * R;
  P.left = tx > 0, P.right = tx + 1 < g.tiles_x;
  P.below = ty > 0, P.above = ty + 1 < g.tiles_y;
  P.ox0 = P.left ? g.halo : 0;
  P.oy0 = P.below ? g.halo : 0;
  P.ox1 = P.right ? kTileW - g.halo : min(kTileW, W - P.gx0);
  P.oy1 = P.above ? g.RH - g.halo : min(g.RH, H - P.gy0);
  return P;
}

// Rows of a strip of R that are in [lo, hi) of the region, as a bit mask.
__device__ __forceinline__ uint32_t rows_in(int y0, int R, int lo, int hi) {
  const int a = min(max(lo - y0, 0), R), b = min(max(hi - y0, 0), R);
  return ((1u << b) - 1u) & ~((1u << a) - 1u);
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
// 4.2 us; the fence and the poll alone 2.3.)
//
// Packets lie by the cell they carry, in two copies that alternate. A copy is
// written again two exchanges later: by then the writer has received the
// exchange between from every neighbouring tile, whose warps sent it after the
// sweeps that follow their reads of this one (the sweeps hold barriers of the
// CTA, and a CTA receives from all its neighbours).
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
  if (atomicCAS(sync.dev_err, 0, 1) == 0) {
    *(volatile int*)sync.host_err = 1;
    __threadfence_system();
  }
  return false;
}

// The whole patch from a field (row j of the grid at (H - 1 - j) W). `vec`: W and
// the columns of the region's quads are multiples of 4; the loads then carry
// no condition (a kernel's code is fetched cold once per launch, so what it
// does once has to be short), and a cell off the grid reads the nearest quad
// or row of it: cells off the grid may hold any value, no cell of the grid
// depends on them.
template <int R, class IO>
__device__ __forceinline__ void patch_in(const IO& io, float (&f)[R][8], const void* field,
                                         const Patch& P, int W, int H, bool vec) {
  const int x = P.gx0 + P.x0, j0 = P.gy0 + P.y0;
  const typename IO::Word* base = static_cast<const typename IO::Word*>(field);
  if (vec) {
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
  const typename IO::Word* row = base + (int64_t)(H - 1 - j0) * W + x;
#pragma unroll
  for (int r = 0; r < R; r++, row -= W)
#pragma unroll
    for (int q = 0; q < 8; q++) io.load1(j0 + r < H && x + q < W, row + q, &f[r][q]);
}

// The patch's rows in `rows` out to a field, the owned columns among them.
template <int R, class IO>
__device__ __forceinline__ void patch_out(const IO& io, const float (&f)[R][8], void* field,
                                          const Patch& P, uint32_t rows, int W, int H, bool vec) {
  const int lo = P.ox0 - P.x0, hi = P.ox1 - P.x0;  // owned columns of the patch
  typename IO::Word* row = static_cast<typename IO::Word*>(field) +
                           (int64_t)(H - 1 - (P.gy0 + P.y0)) * W + P.gx0 + P.x0;
  if (vec) {
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
  for (int r = 0; r < R; r++, row -= W)
#pragma unroll
    for (int q = 0; q < 8; q++)
      io.store1(((rows >> r) & 1u) && q >= lo && q < hi, row + q, &f[r][q]);
}

// Packets of a quad of cells: three for u and v (8 values), two for u alone.
template <int FIELDS>
constexpr int kPacketsPerQuad = FIELDS == 2 ? 3 : 2;

// The cells an exchange moves, as quads: 2 halo whole rows of the region (the
// halo rows below and above as the ring; the owned rows beside them as the
// band) and, in every row, halo columns on either side. Row quads are taken by
// (row, which of the lane's two quads, lane), side quads by (row, side, quad),
// both in shared memory and in the numbering of the items.
constexpr int kRowQuads = kTileW / 4;
struct Exchange {
  float4* cells;  // rows: [2 halo][FIELDS][2][32], then sides: [RH][2][halo / 4][FIELDS]
  int* send;      // per item: its packet's place, or -1 (not sent)
  int* take;      // per item of the ring: its packet's place, or -1 (not taken)
  int rows, items;  // row items, all items
};
inline __host__ __device__ int exchange_items(int halo, int RH) {
  return 2 * halo * kRowQuads + RH * (halo / 2);
}
inline __host__ __device__ size_t exchange_smem(int halo, int RH, int fields) {
  return (size_t)exchange_items(halo, RH) * (fields * 16 + 8);
}

// Item `it` as a row and quad of the region, for the ring or the band `in`
// cells inside it.
__device__ __forceinline__ void exchange_cell(int it, int in, const RegTile& g, int rows, int* y,
                                              int* q) {
  const int h = g.halo, hq = h / 4;
  if (it < rows) {
    const int k = it / kRowQuads;
    *y = k < h ? in + k : g.RH - h - in + (k - h);
    *q = 2 * (it & 31) + ((it >> 5) & 1);
  } else {
    const int s = it - rows, k = s % (2 * hq);
    *y = s / (2 * hq);
    *q = k < hq ? in / 4 + k : kRowQuads - hq - in / 4 + (k - hq);
  }
}

// The places of all items' packets, once per launch.
__device__ __forceinline__ Exchange exchange_plan(char* base, const Patch& P, const RegTile& g,
                                                  int fields, int W, int H) {
  Exchange x;
  const int h = g.halo;
  x.rows = 2 * h * kRowQuads;
  x.items = exchange_items(h, g.RH);
  x.cells = reinterpret_cast<float4*>(base);
  x.send = reinterpret_cast<int*>(x.cells + x.items * fields);
  x.take = x.send + x.items;
  const int half = (W + 7) / 8;  // pairs of quads in a row of the grid
  for (int it = threadIdx.x; it < x.items; it += blockDim.x) {
#pragma unroll
    for (int band = 0; band < 2; band++) {
      int y, q;
      exchange_cell(it, band ? h : 0, g, x.rows, &y, &q);
      const int i = P.gx0 + 4 * q, j = P.gy0 + y;
      bool on = i < W && j < H;
      if (it < x.rows) {
        on = on && (it < x.rows / 2 ? P.below : P.above);
      } else {
        const bool left = (it - x.rows) % (h / 2) < h / 4;
        on = on && (left ? P.left : P.right) && y >= P.oy0 && y < P.oy1;
      }
      if (band) {
        // A row of both bands goes once, and a side quad of a band row with
        // its row; only owned columns go.
        const bool low = P.below && y < 2 * h, high = P.above && y >= g.RH - 2 * h;
        on = on && (it < x.rows / 2 || !low) && (it < x.rows || !high) && 4 * q >= P.ox0 &&
             4 * q < P.ox1;
      }
      const int Q = i / 4;
      (band ? x.send : x.take)[it] = on ? (j * 2 + (Q & 1)) * half + (Q >> 1) : -1;
    }
  }
  return x;
}
// Packets of one plane (values 3 k .. 3 k + 2 of every quad of the grid).
inline __host__ __device__ int64_t packet_plane(int W, int H) {
  return (int64_t)H * 2 * ((W + 7) / 8);
}

// The rows and side quads of a patch between registers and the buffer: `in` = 0
// the ring into the registers, `in` = halo the band out of them.
template <int FIELDS, bool BAND, int R>
__device__ __forceinline__ void exchange_patch(float (&f)[R][8], float (&f2)[R][8],
                                               const Exchange& x, const Patch& P,
                                               const RegTile& g) {
  const int h = g.halo, hq = h / 4, in = BAND ? h : 0;
  auto move = [&](float4* p, float* q) {
    if (BAND) {
      *p = make_float4(q[0], q[1], q[2], q[3]);
    } else {
      const float4 t = *p;
      q[0] = t.x, q[1] = t.y, q[2] = t.z, q[3] = t.w;
    }
  };
  // Side quads of the lane (halos are whole numbers of quads).
  const int l0 = 2 * P.lane - in / 4, r0 = 2 * P.lane - (kRowQuads - hq - in / 4);
  uint32_t side[2];
  float4* at[2];
#pragma unroll
  for (int c = 0; c < 2; c++) {
    const bool left = P.left && l0 + c >= 0 && l0 + c < hq;
    const bool right = P.right && r0 + c >= 0 && r0 + c < hq;
    side[c] = left || right ? rows_in(P.y0, R, P.oy0, P.oy1) : 0u;
    at[c] = x.cells + x.rows * FIELDS +
            (P.y0 * 2 * hq + (left ? l0 + c : hq + r0 + c)) * FIELDS;
  }
  uint32_t whole = (P.below ? rows_in(P.y0, R, in, in + h) : 0u) |
                   (P.above ? rows_in(P.y0, R, g.RH - h - in, g.RH - in) : 0u);
#pragma unroll
  for (int r = 0; r < R; r++) {
    if ((whole >> r) & 1u) {  // the same for the warp
      const int y = P.y0 + r;
      const int k = P.below && y < in + h ? y - in : h + y - (g.RH - h - in);
      float4* row = x.cells + k * FIELDS * 64 + P.lane;
      move(row, &f[r][0]);
      move(row + 32, &f[r][4]);
      if (FIELDS == 2) {
        move(row + 64, &f2[r][0]);
        move(row + 96, &f2[r][4]);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < 2; c++) {
    const uint32_t m = side[c] & ~whole;
    if (m == 0u) continue;
#pragma unroll
    for (int r = 0; r < R; r++) {
      if (((m >> r) & 1u) == 0u) continue;
      float4* p = at[c] + r * 2 * hq * FIELDS;
      move(p, &f[r][4 * c]);
      if (FIELDS == 2) move(p + 1, &f2[r][4 * c]);
    }
  }
}

// Place of an item's first field in the buffer, and the step to the second.
template <int FIELDS>
__device__ __forceinline__ float4* exchange_at(const Exchange& x, int it, int* step) {
  if (it < x.rows) {
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
__device__ __forceinline__ void exchange(float (&f)[R][8], float (&f2)[R][8], const Exchange& x,
                                         const ResidentSync& sync, const Patch& P,
                                         const RegTile& g, int64_t plane, unsigned number) {
  constexpr int kPer = kPacketsPerQuad<FIELDS>;
  uint4* packets = sync.packets + (number & 1) * kPer * plane;
  exchange_patch<FIELDS, true, R>(f, f2, x, P, g);
  __syncthreads();
#pragma unroll 1
  for (int it = threadIdx.x; it < x.items; it += blockDim.x) {
    const int place = x.send[it];
    if (place < 0) continue;
    int step;
    const float4* c = exchange_at<FIELDS>(x, it, &step);
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
  constexpr int kAtOnce = 2;
#pragma unroll 1
  for (int base = 0; base < x.items; base += kAtOnce * blockDim.x) {
    float v[kAtOnce][9];
    const uint4* p[kAtOnce];
    int at[kAtOnce];
    bool on[kAtOnce], ok;
#pragma unroll
    for (int k = 0; k < kAtOnce; k++) {
      at[k] = base + k * blockDim.x + threadIdx.x;
      const int place = at[k] < x.items ? x.take[at[k]] : -1;
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
    if (base == 0) __syncthreads();  // the band has been read: the buffer takes the ring
#pragma unroll
    for (int k = 0; k < kAtOnce; k++) {
      if (!on[k]) continue;
      int step;
      float4* c = exchange_at<FIELDS>(x, at[k], &step);
      c[0] = make_float4(v[k][0], v[k][1], v[k][2], v[k][3]);
      if (FIELDS == 2) c[step] = make_float4(v[k][4], v[k][5], v[k][6], v[k][7]);
    }
  }
  __syncthreads();
  exchange_patch<FIELDS, false, R>(f, f2, x, P, g);
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
// on, which leaves every value as it is, without a branch.
// The division by the count is a product with its reciprocal, which has the
// fast-math division's bits for every float input (checked for 4 and for 3 by
// tests/cpp).
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

// Shared memory of a projection tile: strip boundaries, the cells' reciprocal
// neighbour counts, (PRESSURE) the pressure and the flag words.
struct ProjSmem {
  float4* slot;      // [warps][2][32]
  float4* rs;        // [RH][2][32]
  float4* p;         // [RH][2][32]
  uint32_t* flags;   // [RH][2][32]
};

__host__ __device__ inline size_t project_tile_smem(int RH, int warps, bool pressure, int halo,
                                                    bool resident) {
  return (size_t)warps * 64 * 16 + (size_t)RH * 64 * ((pressure ? 32 : 16) + 4) +
         (resident ? exchange_smem(halo, RH, 2) : 0);
}

__device__ __forceinline__ ProjSmem project_smem_of(char* base, int RH, int warps, bool pressure) {
  ProjSmem s;
  s.slot = reinterpret_cast<float4*>(base);
  s.rs = s.slot + warps * 64;
  s.p = s.rs + RH * 64;
  s.flags = reinterpret_cast<uint32_t*>(s.p + (pressure ? RH * 64 : 0));
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
// A lane wholly off the grid puts no condition: its cells are zeros whose
// faces no cell of the grid reads.
template <int R>
__device__ __forceinline__ void flags_in(const uint8_t* __restrict__ flags, const Patch& P,
                                         const ProjSmem& sm, int W, int H, bool vec,
                                         ProjLane& L) {
  const int gx = P.gx0 + P.x0;
  const bool off = gx >= W;
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
    const int e = (P.y0 + r) * 64 + P.lane;
    sm.flags[e] = raw[r][0];
    sm.flags[e + 32] = raw[r][1];
    sm.rs[e] = reciprocal_counts(raw[r][0]);
    sm.rs[e + 32] = reciprocal_counts(raw[r][1]);
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

// One colour half-sweep over the strip. The rows between the first and the
// last come first, so that the faces that arrived from the other strips and
// lanes have time to arrive, and those that go to them leave last; the rows
// of a colour share no face, so their order is free.
template <int COLOUR, bool PRESSURE, Rows ROWS, int R>
__device__ __forceinline__ void strip_rows(float (&u)[R][8], float (&v)[R][8], float (&ur)[R],
                                           float (&vt)[8], const ProjLane& L, const ProjSmem& sm,
                                           int cell0, const Consts& c, float d_t) {
#pragma unroll
  for (int k = 0; k < R; k++) {
    const int r = k + 2 < R ? k + 1 : k + 2 == R ? 0 : R - 1;  // 1 .. R - 2, 0, R - 1
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
}

// The faces between strips after a half-sweep, through the slots, 4 words each
// way: a strip sends those its half-sweep changed, and after the barrier that
// ends the half-sweep reads those its neighbours changed. A slot is next
// written by the side that read it, so one barrier per half-sweep suffices.
template <int COLOUR, int R>
__device__ __forceinline__ void strip_send(const float (&v)[R][8], const float (&vt)[8],
                                           const Patch& P, const ProjSmem& sm, int warps) {
  constexpr int cb = COLOUR, ct = (COLOUR + R - 1) & 1;  // of the bottom and the top row
  if (P.warp + 1 < warps)
    sm.slot[(P.warp * 2 + ct) * 32 + P.lane] = make_float4(vt[ct], vt[ct + 2], vt[ct + 4], vt[ct + 6]);
  if (P.warp > 0)
    sm.slot[((P.warp - 1) * 2 + cb) * 32 + P.lane] =
        make_float4(v[0][cb], v[0][cb + 2], v[0][cb + 4], v[0][cb + 6]);
}

template <int COLOUR, int R>
__device__ __forceinline__ void strip_receive(float (&v)[R][8], float (&vt)[8], const Patch& P,
                                              const ProjSmem& sm, int warps) {
  constexpr int nb = 1 - COLOUR, nt = 1 - ((COLOUR + R - 1) & 1);
  if (P.warp + 1 < warps) {
    const float4 t = sm.slot[(P.warp * 2 + nt) * 32 + P.lane];
    vt[nt] = t.x, vt[nt + 2] = t.y, vt[nt + 4] = t.z, vt[nt + 6] = t.w;
  }
  if (P.warp > 0) {
    const float4 t = sm.slot[((P.warp - 1) * 2 + nb) * 32 + P.lane];
    v[0][nb] = t.x, v[0][nb + 2] = t.y, v[0][nb + 4] = t.z, v[0][nb + 6] = t.w;
  }
}

template <bool PRESSURE, Rows ROWS, int R>
__device__ __forceinline__ void sweep_loop(float (&u)[R][8], float (&v)[R][8], float (&ur)[R],
                                           float (&vt)[8], const Patch& P, const ProjLane& L,
                                           const ProjSmem& sm, const RegTile& g, const Consts& c,
                                           float d_t, int sweeps) {
  const int warps = g.warps, cell0 = P.y0 * 64 + P.lane;
#pragma unroll 1
  for (int t = 0; t < sweeps; t++) {
    const int reach = 2 * (sweeps - t) - 1;  // half-sweeps after the even one
    // Rows [halo - 1 - reach, RH - halo + reach) reach an owned face, on
    // sides that have a halo at all.
    const bool even = (!P.below || P.y0 + R > g.halo - 1 - reach) &&
                      (!P.above || P.y0 < g.RH - g.halo + reach);
    const bool odd = (!P.below || P.y0 + R > g.halo - reach) &&
                     (!P.above || P.y0 < g.RH - g.halo + reach - 1);
    if (even) strip_rows<0, PRESSURE, ROWS, R>(u, v, ur, vt, L, sm, cell0, c, d_t);
    strip_send<0, R>(v, vt, P, sm, warps);
    __syncthreads();
    strip_receive<0, R>(v, vt, P, sm, warps);
    if (odd) strip_rows<1, PRESSURE, ROWS, R>(u, v, ur, vt, L, sm, cell0, c, d_t);
    strip_send<1, R>(v, vt, P, sm, warps);
    __syncthreads();
    strip_receive<1, R>(v, vt, P, sm, warps);
  }
}

// `sweeps` red/black sweeps of the region. Rows that cannot reach an owned
// face any more are skipped strip by strip; within a strip every cell is
// updated: a cell off the cone of dependence writes faces that only cells off
// the cone read from then on.
template <bool PRESSURE, int R>
__device__ __forceinline__ void tile_sweeps(float (&u)[R][8], float (&v)[R][8], const Patch& P,
                                            const ProjLane& L, const ProjSmem& sm,
                                            const RegTile& g, const Consts& c, float d_t,
                                            int sweeps) {
  static_assert(R % 2 == 0, "strips start on even rows");
  const int warps = g.warps;
  float ur[R], vt[8];
  __syncthreads();  // the slots' last readers
  if (P.warp > 0) {
    float4* s = sm.slot + (P.warp - 1) * 64 + P.lane;
    s[0] = make_float4(v[0][0], v[0][2], v[0][4], v[0][6]);
    s[32] = make_float4(v[0][1], v[0][3], v[0][5], v[0][7]);
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 8; q++) vt[q] = 0.0f;
  if (P.warp + 1 < warps) {
    const float4* s = sm.slot + P.warp * 64 + P.lane;
    const float4 e = s[0], o = s[32];
    vt[0] = e.x, vt[2] = e.y, vt[4] = e.z, vt[6] = e.w;
    vt[1] = o.x, vt[3] = o.y, vt[5] = o.z, vt[7] = o.w;
  }
#pragma unroll
  for (int r = 0; r < R; r++) ur[r] = __shfl_down_sync(kAllLanes, u[r][0], 1);
  __syncthreads();  // every strip has its copies before a slot is rewritten
  if (!L.full)
    sweep_loop<PRESSURE, Rows::kFlags, R>(u, v, ur, vt, P, L, sm, g, c, d_t, sweeps);
  else if (L.wall)
    sweep_loop<PRESSURE, Rows::kWall, R>(u, v, ur, vt, P, L, sm, g, c, d_t, sweeps);
  else
    sweep_loop<PRESSURE, Rows::kPlain, R>(u, v, ur, vt, P, L, sm, g, c, d_t, sweeps);
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

// The pressure of the owned cells, between its field and the tile's planes.
template <int R>
__device__ __forceinline__ void pressure_in(const ProjSmem& sm, const float* p, const Patch& P,
                                            int W, bool zero, int H, bool vec) {
  float f[R][8];
#pragma unroll
  for (int r = 0; r < R; r++)
#pragma unroll
    for (int q = 0; q < 8; q++) f[r][q] = 0.0f;
  const int lo = P.ox0 - P.x0, hi = P.ox1 - P.x0;
  const uint32_t own = zero ? 0u : rows_in(P.y0, R, P.oy0, P.oy1);
  const float* row = p + (int64_t)(H - 1 - (P.gy0 + P.y0)) * W + P.gx0 + P.x0;
  const F32Cells io;
#pragma unroll
  for (int r = 0; r < R; r++, row -= W) {
    const bool on = (own >> r) & 1u;
    if (vec) {
      io.load4(on && 0 >= lo && 0 < hi, row, &f[r][0]);
      io.load4(on && 4 >= lo && 4 < hi, row + 4, &f[r][4]);
    } else {
#pragma unroll
      for (int q = 0; q < 8; q++) io.load1(on && q >= lo && q < hi, row + q, &f[r][q]);
    }
  }
#pragma unroll
  for (int r = 0; r < R; r++) {
    float4* out = sm.p + (P.y0 + r) * 64 + P.lane;
    out[0] = make_float4(f[r][0], f[r][2], f[r][4], f[r][6]);
    out[32] = make_float4(f[r][1], f[r][3], f[r][5], f[r][7]);
  }
}

template <int R>
__device__ __forceinline__ void pressure_out(const ProjSmem& sm, float* p, const Patch& P, int W,
                                             int H, bool vec) {
  float f[R][8];
#pragma unroll
  for (int r = 0; r < R; r++) {
    const float4* in = sm.p + (P.y0 + r) * 64 + P.lane;
    const float4 e = in[0], o = in[32];
    f[r][0] = e.x, f[r][2] = e.y, f[r][4] = e.z, f[r][6] = e.w;
    f[r][1] = o.x, f[r][3] = o.y, f[r][5] = o.z, f[r][7] = o.w;
  }
  patch_out<R>(F32Cells{}, f, p, P, rows_in(P.y0, R, P.oy0, P.oy1), W, H, vec);
}

// Sweeps from `done` to the next exchange or, with 16-bit storage, the next
// rounding.
__device__ __forceinline__ int tile_segment(int n, int K, int D, int done, int storage) {
  const int left = min(D, n - done);
  return storage == OS_STORAGE_F32 ? left : min(left, K - done % K);
}

struct ProjectArgs {
  void *U0, *U1, *V0, *V1;  // the two copies of the fields
  int cu, cv;               // which of them holds the input
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
// every K sweeps, and they end in the copy those passes would end in.
template <int R, bool PRESSURE>
__global__ void __launch_bounds__(32 * tile_max_warps(R), 1)
k_project_tiles(const __grid_constant__ ProjectArgs a) {
  extern __shared__ __align__(16) char tile_smem[];
  const Consts& c = a.c;
  const int W = c.W, H = c.H;
  const Patch P = patch_of(blockIdx.x % a.g.tiles_x, blockIdx.x / a.g.tiles_x, a.g, R, W, H);
  const ProjSmem sm = project_smem_of(tile_smem, a.g.RH, a.g.warps, PRESSURE);
  const bool vec = ((W | a.g.halo) & 3) == 0;
  ProjLane L;
  // The flags do not change after creation: staged before the wait for the
  // kernel before.
  flags_in<R>(a.flags, P, sm, W, H, vec, L);
  pdl_entry();
  float u[R][8], v[R][8];
#pragma unroll
  for (int r = 0; r < R; r++)
#pragma unroll
    for (int q = 0; q < 8; q++) u[r][q] = v[r][q] = 0.0f;
  if (PRESSURE) pressure_in<R>(sm, a.p, P, W, a.zero_pressure, H, vec);
  const float d_t = a.prm->dt;
  on_cells(a.storage, [&](auto io) {
    patch_in<R>(io, u, a.cu ? a.U1 : a.U0, P, W, H, vec);
    patch_in<R>(io, v, a.cv ? a.V1 : a.V0, P, W, H, vec);
  });
  const unsigned epoch = a.n > a.D ? ld_acquire_gpu(a.sync.epochs + blockIdx.x) : 0u;
  unsigned number = epoch;
  Exchange x;
  if (a.n > a.D)
    x = exchange_plan(reinterpret_cast<char*>(sm.flags + a.g.RH * 64), P, a.g, 2, W, H);
  const int64_t plane = packet_plane(W, H);
#pragma unroll 1
  for (int done = 0; done < a.n;) {
    if (done > 0) {
      if (a.storage != OS_STORAGE_F32 && done % a.K == 0) {
        round_patch<R>(u, a.storage);
        round_patch<R>(v, a.storage);
      }
      number++;
      exchange<2, R>(u, v, x, a.sync, P, a.g, plane, number);
    }
    const int sweeps = tile_segment(a.n, a.K, a.D, done, a.storage);
    tile_sweeps<PRESSURE, R>(u, v, P, L, sm, a.g, c, d_t, sweeps);
    done += sweeps;
  }
  if (number != epoch && threadIdx.x == 0) a.sync.epochs[blockIdx.x] = number;
  // The owned cells to the copies that ceil(n / K) passes through memory would
  // end in.
  const bool swap = ((a.n + a.K - 1) / a.K) & 1;
  void* uo = (a.cu != 0) != swap ? a.U1 : a.U0;
  void* vo = (a.cv != 0) != swap ? a.V1 : a.V0;
  const uint32_t own = rows_in(P.y0, R, P.oy0, P.oy1);
  uint32_t own_u = own, top = 0u;
  if (a.extrapolate) {
    extrapolate_patch<R>(u, v, P, W);
    own_u &= ~rows_in(P.y0, R, H - 1 - P.gy0, H - P.gy0);
    top = own & rows_in(P.y0, R, H - 2 - P.gy0, H - 1 - P.gy0);
  }
  on_cells(a.storage, [&](auto io) {
    patch_out<R>(io, u, uo, P, own_u, W, H, vec);
    patch_out<R>(io, v, vo, P, own, W, H, vec);
    if (top)  // row H - 2 of u to row H - 1, which lies one row before it
      patch_out<R>(io, u, static_cast<typename decltype(io)::Word*>(uo) - W, P, top, W, H, vec);
  });
  if (PRESSURE) pressure_out<R>(sm, a.p, P, W, H, vec);
}

// ---------------------------------------------------------------------------
// Jacobi diffusion of u (apply_diffusion_at, src/fluid.cu:176-183).
// ---------------------------------------------------------------------------

// Shared memory of a diffusion tile: each strip's bottom and top row, in two
// buffers (a sweep writes one while the other may still be read).
struct DiffSmem {
  float4* rows;   // [2][warps][bottom, top][2][32]
};
__host__ __device__ inline size_t diffuse_tile_smem(int RH, int warps, int halo, bool resident) {
  return (size_t)2 * warps * 4 * 32 * 16 + (resident ? exchange_smem(halo, RH, 1) : 0);
}

// How a strip's cells are taken: no row or column of it kept, the columns 0, 3
// and 7 of its lanes where DiffLane says so, or any row or column, and the
// division may be one (jacobi_divide).
enum class Kept { kNone, kQuadEdges, kAny };

// What a patch holds that no sweep changes: the grid's first and last column
// (bit q of `cols`: column q of the lane) and row (bit r of `rows`, the same in
// the warp).
struct DiffLane {
  uint32_t cols, rows;
};

// One sweep of the strip, row by row in place: `down` holds the old row below.
// `below` / `above`: the neighbouring strips' rows in shared memory (null: none,
// and the row beside it is off the cone or kept).
template <int R, Kept KEPT>
__device__ __forceinline__ void jacobi_strip(float (&u)[R][8], const float4* below,
                                             const float4* above, const DiffLane& L, float a,
                                             float den, float rden, bool rcp) {
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 b0 = below ? below[0] : zero, b1 = below ? below[32] : zero;
  float down[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
  for (int r = 0; r < R; r++) {
    float left = __shfl_up_sync(kAllLanes, u[r][7], 1);
    const float right = __shfl_down_sync(kAllLanes, u[r][0], 1);
    float up[8];
    if (r + 1 < R) {
#pragma unroll
      for (int q = 0; q < 8; q++) up[q] = u[r + 1 < R ? r + 1 : 0][q];
    } else {
      const float4 t0 = above ? above[0] : zero, t1 = above ? above[32] : zero;
      up[0] = t0.x, up[1] = t0.y, up[2] = t0.z, up[3] = t0.w;
      up[4] = t1.x, up[5] = t1.y, up[6] = t1.z, up[7] = t1.w;
    }
    const uint32_t kept = KEPT == Kept::kAny && ((L.rows >> r) & 1u) ? 0xffu : L.cols;
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const float old = u[r][q];
      const float rt = q < 7 ? u[r][q < 7 ? q + 1 : 7] : right;
      // src/fluid.cu:178-182: neighbours (i-1, j), (i+1, j), (i, j-1), (i, j+1)
      const float x = fma_rn(a, left + rt + down[q] + up[q], old);
      float y = KEPT != Kept::kAny || rcp ? mul_rn(x, rden) : x / den;
      if (KEPT == Kept::kAny || (KEPT == Kept::kQuadEdges && (q == 0 || q == 3 || q == 7)))
        y = (kept >> q) & 1u ? old : y;
      u[r][q] = y;
      down[q] = left = old;
    }
  }
}

template <int R, Kept KEPT>
__device__ __forceinline__ void jacobi_loop(float (&u)[R][8], const Patch& P, const DiffSmem& sm,
                                            const RegTile& g, const DiffLane& L, float a,
                                            float den, float rden, bool rcp, int sweeps) {
  const int warps = g.warps;
#pragma unroll 1
  for (int t = 0; t < sweeps; t++) {
    float4* mine = sm.rows + ((t & 1) * warps + P.warp) * 128 + P.lane;
    mine[0] = make_float4(u[0][0], u[0][1], u[0][2], u[0][3]);
    mine[32] = make_float4(u[0][4], u[0][5], u[0][6], u[0][7]);
    mine[64] = make_float4(u[R - 1][0], u[R - 1][1], u[R - 1][2], u[R - 1][3]);
    mine[96] = make_float4(u[R - 1][4], u[R - 1][5], u[R - 1][6], u[R - 1][7]);
    __syncthreads();
    const int reach = sweeps - 1 - t;  // sweeps after this one
    if ((P.below && P.y0 + R <= g.halo - reach) || (P.above && P.y0 >= g.RH - g.halo + reach))
      continue;
    jacobi_strip<R, KEPT>(u, P.warp > 0 ? mine + 64 - 128 : nullptr,
                          P.warp + 1 < warps ? mine + 128 : nullptr, L, a, den, rden, rcp);
  }
}

template <int R>
__device__ __forceinline__ void jacobi_sweeps(float (&u)[R][8], const Patch& P,
                                              const DiffSmem& sm, const RegTile& g, int W, int H,
                                              float a, int sweeps) {
  const float den = fma_rn(4.0f, a, 1.0f);
  const float rden = __fdividef(1.0f, den);
  const bool rcp = den < 1048576.0f;  // jacobi_divide
  const int gx = P.gx0 + P.x0, gy = P.gy0 + P.y0;
  DiffLane L;
  L.cols = (gx == 0 ? 1u : 0u) | (W - 1 - gx >= 0 && W - 1 - gx < 8 ? 1u << (W - 1 - gx) : 0u);
  L.rows = (gy == 0 ? 1u : 0u) | (H - 1 - gy >= 0 && H - 1 - gy < R ? 1u << (H - 1 - gy) : 0u);
  const uint32_t cols = __reduce_or_sync(kAllLanes, L.cols);
  __syncthreads();  // the rows' last readers
  if (!rcp || L.rows || (cols & ~0x89u))
    jacobi_loop<R, Kept::kAny>(u, P, sm, g, L, a, den, rden, rcp, sweeps);
  else if (cols)
    jacobi_loop<R, Kept::kQuadEdges>(u, P, sm, g, L, a, den, rden, true, sweeps);
  else
    jacobi_loop<R, Kept::kNone>(u, P, sm, g, L, a, den, rden, true, sweeps);
}

struct DiffuseArgs {
  void *U0, *U1;  // the two copies of the field
  int cu;         // which of them holds the input
  int storage;
  Consts c;
  const StepParams* prm;
  int n, K, D;    // sweeps in all, per pass, and between exchanges
  RegTile g;
  ResidentSync sync;
};

// As k_project_tiles, with a halo of D cells.
template <int R>
__global__ void __launch_bounds__(32 * diffuse_max_warps(R), 1)
k_diffuse_tiles(const __grid_constant__ DiffuseArgs a) {
  extern __shared__ __align__(16) char tile_smem[];
  const Consts& c = a.c;
  const int W = c.W, H = c.H;
  const Patch P = patch_of(blockIdx.x % a.g.tiles_x, blockIdx.x / a.g.tiles_x, a.g, R, W, H);
  float4* rows = reinterpret_cast<float4*>(tile_smem);
  const DiffSmem sm{rows};
  const bool vec = ((W | a.g.halo) & 3) == 0;
  pdl_entry();
  float u[R][8];
#pragma unroll
  for (int r = 0; r < R; r++)
#pragma unroll
    for (int q = 0; q < 8; q++) u[r][q] = 0.0f;
  const float coeff = diffusion_coeff<float>(c, a.prm->dt);
  on_cells(a.storage, [&](auto io) { patch_in<R>(io, u, a.cu ? a.U1 : a.U0, P, W, H, vec); });
  const unsigned epoch = a.n > a.D ? ld_acquire_gpu(a.sync.epochs + blockIdx.x) : 0u;
  unsigned number = epoch;
  Exchange x;
  if (a.n > a.D)
    x = exchange_plan(reinterpret_cast<char*>(rows + 2 * a.g.warps * 4 * 32), P, a.g, 1, W, H);
  const int64_t plane = packet_plane(W, H);
#pragma unroll 1
  for (int done = 0; done < a.n;) {
    if (done > 0) {
      if (a.storage != OS_STORAGE_F32 && done % a.K == 0) round_patch<R>(u, a.storage);
      number++;
      exchange<1, R>(u, u, x, a.sync, P, a.g, plane, number);
    }
    const int sweeps = tile_segment(a.n, a.K, a.D, done, a.storage);
    jacobi_sweeps<R>(u, P, sm, a.g, W, H, coeff, sweeps);
    done += sweeps;
  }
  if (number != epoch && threadIdx.x == 0) a.sync.epochs[blockIdx.x] = number;
  const bool swap = ((a.n + a.K - 1) / a.K) & 1;
  void* uo = (a.cu != 0) != swap ? a.U1 : a.U0;
  on_cells(a.storage, [&](auto io) {
    patch_out<R>(io, u, uo, P, rows_in(P.y0, R, P.oy0, P.oy1), W, H, vec);
  });
}

// ---------------------------------------------------------------------------
// Host: geometry and launches.
// ---------------------------------------------------------------------------

inline RegTile reg_tile(int W, int H, int halo, int R, int warps) {
  RegTile g{};
  g.halo = halo;
  g.R = R, g.warps = warps;
  g.RH = R * warps;
  g.TX = kTileW - 2 * halo;
  g.TY = g.RH - 2 * halo;
  g.tiles_x = W <= kTileW ? 1 : (W - 2 * halo + g.TX - 1) / g.TX;
  if (H <= g.RH)
    g.tiles_y = 1;
  else
    g.tiles_y = g.TY >= 2 ? (H - 2 * halo + g.TY - 1) / g.TY : 0;  // 0: does not cover the grid
  return g;
}

// Strip heights the kernels are built for.
constexpr int kProjectRows[] = {2, 4, 6, 8, 12};
constexpr int kDiffuseRows[] = {2, 4, 6, 8, 12};

// The tile that takes the least time by a model of n sweeps, `D` between
// exchanges or passes: issue slots on the fullest of the SM's four schedulers,
// the region once in and out (or an exchange), in as many waves as the tiles
// take. With `resident` every tile must have an SM of its own and be at least
// a halo wide and high (the ring then comes from adjacent tiles). Returns the
// modelled cycles, 0 when no tile covers the grid.
inline double choose_tile(int W, int H, int D, bool projection, bool pressure, bool resident,
                          int n, int sms, RegTile* out) {
  double best = 0.0;
  const int halo = projection ? 2 * D : D;
  const int* heights = projection ? kProjectRows : kDiffuseRows;
  const int count = projection ? (int)std::size(kProjectRows) : (int)std::size(kDiffuseRows);
  for (int k = 0; k < count; k++) {
    const int R = heights[k];
    const int most = projection ? tile_max_warps(R) : diffuse_max_warps(R);
    for (int warps = 1; warps <= most; warps++) {
      RegTile g = reg_tile(W, H, halo, R, warps);
      if (g.tiles_y < 1) continue;
      const int64_t tiles = (int64_t)g.tiles_x * g.tiles_y;
      if (resident && (tiles > sms || (g.tiles_y > 1 && g.TY < halo) || g.TX < halo)) continue;
      g.smem = projection ? project_tile_smem(g.RH, warps, pressure, halo, resident)
                          : diffuse_tile_smem(g.RH, warps, halo, resident);
      if (g.smem + kStaticSmem > kMaxSmem) continue;
      const int64_t waves = (tiles + sms - 1) / sms;
      // Cycles of a sweep: the strips on a scheduler, and a barrier and the
      // faces' way between strips for each half-sweep.
      const double strip = projection ? (pressure ? 116.0 : 78.0) * R + 40.0 : 46.0 * R + 60.0;
      const double sweep = ((warps + 3) / 4) * strip + (projection ? 350.0 : 150.0);
      const double trip = resident ? 4000.0 + 40.0 * R
                                   : 5000.0 + g.RH * (projection ? 50.0 : 25.0);
      const double rounds = (n + D - 1) / D;
      const double cost = (double)waves * (n * sweep + rounds * trip);
      if (best == 0.0 || cost < best) {
        best = cost;
        *out = g;
      }
    }
  }
  return best;
}

using ProjectKernel = void (*)(const ProjectArgs);
using DiffuseKernel = void (*)(const DiffuseArgs);

template <bool PRESSURE>
inline ProjectKernel project_kernel(int R) {
  switch (R) {
    case 2: return k_project_tiles<2, PRESSURE>;
    case 4: return k_project_tiles<4, PRESSURE>;
    case 6: return k_project_tiles<6, PRESSURE>;
    case 8: return k_project_tiles<8, PRESSURE>;
    default: return k_project_tiles<12, PRESSURE>;
  }
}
inline DiffuseKernel diffuse_kernel(int R) {
  switch (R) {
    case 2: return k_diffuse_tiles<2>;
    case 4: return k_diffuse_tiles<4>;
    case 6: return k_diffuse_tiles<6>;
    case 8: return k_diffuse_tiles<8>;
    default: return k_diffuse_tiles<12>;
  }
}

// A launch of `tiles` CTAs: cooperative when its CTAs wait on one another,
// else with programmatic stream serialisation where the handle uses it.
template <class Args>
inline cudaError_t launch_tiles(void (*kernel)(const Args), const Args& a, const RegTile& g,
                                bool cooperative, bool pdl, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)g.smem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(g.tiles_x * g.tiles_y);
  cfg.blockDim = dim3(32 * g.warps);
  cfg.dynamicSmemBytes = g.smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  if (cooperative) {
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
  } else {
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = (cooperative || pdl) ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, a);
}

// The resident forms' tiles, all of one launch resident together, and the
// sweeps between their exchanges. (block_k is not their depth: it says which
// copy the fields end in and, with 16-bit storage, how often they are rounded.)
inline int resident_tile(const os_handle* h, bool projection, RegTile* g) {
  const bool pressure = h->cfg.enable_pressure != 0;
  const int K = h->block_k;
  if (K < 2 || K % (projection ? 2 : 4)) return 0;
  int depth = 0;
  double best = 0.0;
  for (int D : {2, 4, 6, 8, 12, 16}) {  // halos in multiples of 4 cells
    if (!projection && D % 4) continue;
    RegTile t;
    const double cost = choose_tile(h->W, h->H, D, projection, pressure, true, std::max(h->c.n, 1),
                                    sm_count(h->cfg.device), &t);
    if (cost > 0.0 && (depth == 0 || cost < best)) {
      best = cost;
      depth = D;
      *g = t;
    }
  }
  return depth;
}

// The projection phase: one launch for all its passes (resident), or one per
// pass of block_k sweeps. `cur_u` / `cur_v` say which copy holds the live
// field (0: u, v; 1: ub, vb) and advance by the passes. `extrapolate`: the
// last pass applies the extrapolation that follows in a step. Returns the
// launches, or -1.
inline int enqueue_tiled_projection(os_handle* h, cudaStream_t st, int* cur_u, int* cur_v,
                                    bool zero_first, bool extrapolate) {
  const int K = h->block_k, n = h->c.n;
  const bool pressure = h->cfg.enable_pressure != 0;
  ProjectArgs a{};
  a.U0 = h->u, a.U1 = h->ub, a.V0 = h->v, a.V1 = h->vb;
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
    if (!(a.D = resident_tile(h, true, &a.g))) return -1;
    a.n = n;
    a.cu = *cur_u, a.cv = *cur_v;
    a.zero_pressure = zero_first;
    a.extrapolate = extrapolate;
    if (passes > 0 &&
        launch_tiles(pressure ? project_kernel<true>(a.g.R) : project_kernel<false>(a.g.R), a, a.g,
                     n > a.D, h->pdl, st) != cudaSuccess)
      return -1;
    launches = passes > 0;
  } else {
    a.D = K;
    if (projection_smem(2 + 4 * K, pressure) + kStaticSmem > kMaxSmem ||
        choose_tile(h->W, h->H, K, true, pressure, false, n, sm_count(h->cfg.device), &a.g) == 0.0)
      return -1;
    for (int p = 0; p < passes; p++, launches++) {
      a.n = std::min(K, n - p * K);
      a.cu = (*cur_u + p) & 1, a.cv = (*cur_v + p) & 1;
      a.zero_pressure = zero_first && p == 0;
      a.extrapolate = extrapolate && p == passes - 1;
      if (launch_tiles(pressure ? project_kernel<true>(a.g.R) : project_kernel<false>(a.g.R), a,
                       a.g, false, h->pdl, st) != cudaSuccess)
        return -1;
    }
  }
  *cur_u = (*cur_u + passes) & 1;
  *cur_v = (*cur_v + passes) & 1;
  return launches;
}

// The diffusion phase in the same way, block_k sweeps per pass when resident,
// else diffusion_depth.
inline int enqueue_tiled_diffusion(os_handle* h, cudaStream_t st, int* cur_u) {
  const int K = h->resident_diff ? h->block_k : diffusion_depth(h), n = h->c.n;
  DiffuseArgs a{};
  a.U0 = h->u, a.U1 = h->ub;
  a.storage = h->storage;
  a.c = h->c;
  a.prm = h->d_params;
  a.K = K;
  a.sync = ResidentSync{h->dflags, h->dpackets, h->rerr, h->d_host_rerr};
  const int passes = (n + K - 1) / K;
  int launches = 0;
  if (h->resident_diff) {
    if (!(a.D = resident_tile(h, false, &a.g))) return -1;
    a.n = n;
    a.cu = *cur_u;
    if (passes > 0 && launch_tiles(diffuse_kernel(a.g.R), a, a.g, n > a.D, h->pdl, st) !=
                          cudaSuccess)
      return -1;
    launches = passes > 0;
  } else {
    a.D = K;
    if (choose_tile(h->W, h->H, K, false, false, false, n, sm_count(h->cfg.device), &a.g) == 0.0)
      return -1;
    for (int p = 0; p < passes; p++, launches++) {
      a.n = std::min(K, n - p * K);
      a.cu = (*cur_u + p) & 1;
      if (launch_tiles(diffuse_kernel(a.g.R), a, a.g, false, h->pdl, st) != cudaSuccess) return -1;
    }
  }
  *cur_u = (*cur_u + passes) & 1;
  return launches;
}

// Device bytes of a resident phase's epochs, and of its packets.
inline size_t resident_epoch_bytes(int sms) { return (size_t)sms * sizeof(unsigned); }
inline size_t resident_packet_bytes(int W, int H, int per_quad) {
  return (size_t)2 * packet_plane(W, H) * per_quad * sizeof(uint4);
}

// Whether the resident forms can be launched cooperatively on this device.
template <class Args>
inline bool tiles_launchable(void (*kernel)(const Args), const RegTile& g, int sms) {
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)g.smem) !=
      cudaSuccess)
    return false;
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 32 * g.warps, g.smem) !=
      cudaSuccess)
    return false;
  return per_sm >= 1 && g.tiles_x * g.tiles_y <= per_sm * sms;
}

// Failure-detection self-test: a warp waits for a packet that nothing sends, so
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

}  // namespace osg
