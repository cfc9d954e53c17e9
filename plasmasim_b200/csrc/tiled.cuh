// Tiled particle layout and its incremental sort (the push kernel that uses
// the layout is in push_tiled.cuh).
//
// Layout. The interior cells are cut into tiles of TX x TY x 32 cells (x, y,
// z). Each (x, y) column of a tile -- 32 consecutive z cells -- is a "group"
// handled by one warp, lane L owning cell z0 + L (its "home" cell). A group's
// slots are gmax[G] rows of 32: slot goff[G] + 32 r + L is row r of lane L's
// column. A sort fills each lane's column with the particles of its cell up to
// the group's level -- its mean particles per lane, rounded up -- and puts the
// rest of the fuller cells ("strangers") into the free slots below the level
// of the group's other lanes, so that a group runs through as many rows as it
// has particles for, not as many as its fullest cell. Slots above are empty
// (cell = -1), kept for later arrivals; gtop[G] is one past the last row that
// holds a particle. A warp then reads 32 consecutive slots per step of its
// loop (one coalesced 128-byte line per array) and its 32 lanes work on 32
// cells, nearly all of them different. Rows sized for the fullest of the 32
// cells left a fifth (64 particles per cell) to 40 % (8) of the lanes idle
// once the particles had mixed. Measured, push of both species per step, such
// rows against these: 7.90 -> 7.02 ms (128^3 cells x 64 per cell), 0.413 ->
// 0.345 (64^3 x 16), 0.092 -> 0.075 (32^3 x 8), FP64 64^3 x 32 2.05 -> 1.73;
// the re-layout, which moves the strangers as well, 1.82 -> 2.01, 0.091 ->
// 0.103 and 0.0345 -> 0.035.
//
// Deposit. A lane accumulates the current of the particles that are in its
// home cell in registers (the 2x3x3 / 3x2x3 / 3x3x2 nodes such a particle can
// touch) and adds them to a shared-memory window of (TX+4) x (TY+4) x 36 nodes
// once, after its last particle. The currents of particles that have left
// their home cell since the sort are queued per warp and added to the planes
// 32 at a time; the densities of the fused push go to the window, in FP32 as
// fixed-point numbers with shared integer reductions, or, when the stencil
// leaves the window (periodic wrap, long moves), to global memory. The window is added to the global planes
// with one vector reduction per 4 nodes.
//
// Sort. Between sorts most particles stay in their cell. The sort keeps the
// order of those "stayers" within their lane column (a warp walks its columns
// row by row, so stayers are written in order without atomics, into nearly
// the same 128-byte lines they came from) and places the others -- movers,
// and particles appended by a refill -- after the stayers of their new cell
// with per-cell atomic cursors. A particle ranked past the level takes its
// group's next free slot below the level (a per-group cursor).
#pragma once

#include "common.cuh"
#include "particles.cuh"

namespace pb {

// Rows that a full sort adds to a group above its level, level / kSlackDiv +
// kSlackRows: room for a group that gains particles until the next full sort
// (empty rows above gtop cost memory only). No group takes more rows than its
// fullest cell would with a sixteenth and two rows more, which is the smaller
// of the two where the cells are evenly filled (19 rows against 21 at 16 per
// cell): a capacity that holds rows sized that way, and the refills behind
// them, always holds these.
constexpr int kSlackDiv = 8;
constexpr int kSlackRows = 3;
constexpr int kFullestDiv = 16;
constexpr int kFullestRows = 2;
// Rows of the level above the group's mean particles per lane: each spares
// some of the fuller cells' strangers and adds a partly filled row. One and
// two rows measured 9.32 and 9.34 ms per step against 9.30 at 128^3 x 64, and
// 0.682 and 0.687 against 0.682 at 64^3 x 16.
constexpr int kLevelRows = 0;

constexpr int kTileX = 2;
constexpr int kTileY = 4;
constexpr int kLanes = 32;
constexpr int kWinZ = kLanes + 4;

struct TileGeom {
  int ntx, nty, ntz;  // tiles per axis
  int ngroups;        // ntx * nty * ntz * kTileX * kTileY
};

// Group and lane of an interior cell (absolute indices), -1 outside the interior.
__device__ __forceinline__ int group_of(const Geom& g, const TileGeom& t, int i, int j, int k,
                                        int& lane) {
  i -= 2; j -= 2; k -= 2;
  if (i < 0 || j < 0 || k < 0 || i >= g.nx || j >= g.ny || k >= g.nz) return -1;
  const int tx = i / kTileX, wx = i % kTileX, ty = j / kTileY, wy = j % kTileY;
  const int tz = k >> 5;
  lane = k & 31;
  const int tile = (tx * t.nty + ty) * t.ntz + tz;
  return tile * (kTileX * kTileY) + wx * kTileY + wy;
}

// The cell that a lane of z tile tz owns. Where the interior ends inside the
// tile (nv < 32 cells), the lanes past its last cell own the tile's cells over
// again: cell z has the lanes z, z + nv, z + 2 nv, ..., n of them, and this is
// number m. (Where such lanes held nothing but strangers, the push of both
// species took 0.180, 0.464, 0.186 and 0.249 ms per step with nz = 20, 45, 70
// and 36, this way 0.137, 0.404, 0.180 and 0.244.)
struct LaneCell {
  int z, m, n;
};
__device__ __forceinline__ int tile_cells(const Geom& g, int tz) { return min(kLanes, g.nz - tz * kLanes); }
__device__ __forceinline__ int lanes_of(int nv, int z) { return nv == kLanes ? 1 : (kLanes - 1 - z) / nv + 1; }
__device__ __forceinline__ LaneCell lane_cell(int nv, int lane) {
  if (nv == kLanes) return {lane, 0, 1};
  const int z = lane % nv;
  return {z, lane / nv, lanes_of(nv, z)};
}
// This lane's part of the c particles of its cell: those ranked m, m + n, ...
__device__ __forceinline__ int lane_share(int c, const LaneCell& l) { return (c + l.n - 1 - l.m) / l.n; }

// Absolute indices of the cell that group G's lane owns; false when it owns none.
__device__ __forceinline__ bool home_cell(const Geom& g, const TileGeom& t, int G, int lane, int& i, int& j, int& k,
                                          LaneCell& l) {
  const int tile = G / (kTileX * kTileY), w = G % (kTileX * kTileY);
  const int tz = tile % t.ntz, ty = (tile / t.ntz) % t.nty, tx = tile / (t.ntz * t.nty);
  l = lane_cell(tile_cells(g, tz), lane);
  i = tx * kTileX + w / kTileY;
  j = ty * kTileY + w % kTileY;
  k = tz * kLanes + l.z;
  const bool ok = i < g.nx && j < g.ny;
  i += 2; j += 2; k += 2;
  return ok;
}

// Interior cell key of group G's lane, or -1 when the lane has no cell.
__device__ __forceinline__ int home_key(const Geom& g, const TileGeom& t, int G, int lane, LaneCell& l) {
  int i, j, k;
  return home_cell(g, t, G, lane, i, j, k, l) ? ((i - 2) * g.ny + (j - 2)) * g.nz + (k - 2) : -1;
}

__device__ __forceinline__ int cells_of_group(const Geom& g, const TileGeom& t, int G) {
  return tile_cells(g, G / (kTileX * kTileY) % t.ntz);
}

// Group and (first) lane of an interior cell key.
__device__ __forceinline__ int group_of_key(const Geom& g, const TileGeom& t, int key, int& lane) {
  const int k = key % g.nz, j = (key / g.nz) % g.ny, i = key / (g.nz * g.ny);
  return group_of(g, t, i + 2, j + 2, k + 2, lane);
}

// --------------------------------------------------------------- sort
// Counting: stayers per home cell (no atomics) over the tiled slots, movers
// and appended particles per destination cell (atomics).
template <typename real>
__global__ void tiled_count_kernel(Parts<real> P, Geom g, TileGeom t, const int* __restrict__ goff,
                                   const int* __restrict__ gmax, int* stay, int* moved) {
  const int G = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (G >= t.ngroups) return;
  LaneCell lc;
  int home = home_key(g, t, G, lane, lc);
  if (lc.n > 1) home = -1;  // the lanes of one cell have no common order: all movers
  const int base = goff[G], m = gmax[G];
  int nstay = 0;
  constexpr int U = 8;  // rows whose loads are in flight together
  for (int r0 = 0; r0 < m; r0 += U) {
    int cell[U];
#pragma unroll
    for (int u = 0; u < U; ++u) cell[u] = r0 + u < m ? P.cell[base + (r0 + u) * kLanes + lane] : -1;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int key = interior_key(g, cell[u]);
      if (key < 0) continue;
      if (key == home) ++nstay;
      else atomicAdd(moved + key, 1);
    }
  }
  if (home >= 0) stay[home] = nstay;  // cleared before: cells of several lanes keep 0
}

template <typename real>
__global__ void append_count_kernel(Parts<real> P, int first, const int* __restrict__ count, Geom g,
                                    int* moved) {
  const int n = *count;
  for (int s = first + blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
    const int key = interior_key(g, P.cell[s]);
    if (key >= 0) atomicAdd(moved + key, 1);
  }
}

// Rows a lane column keeps for the boundary refill of its cell: the refill's
// particle count plus an eighth and four, so that the refill fits into the
// column's empty slots without moving other particles.
__device__ __forceinline__ int reserve_of(int need) { return need > 0 ? need + need / 8 + 4 : 0; }
__device__ __forceinline__ int refill_need(const SourceParams& sp, const Geom& g, const TileGeom& t, int G, int lane) {
  int i, j, k;
  LaneCell l;
  return home_cell(g, t, G, lane, i, j, k, l) ? slab_need(sp, i, j, k) : 0;
}

// Inclusive sum over the lanes of a warp.
__device__ __forceinline__ int warp_scan(int v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += y;
  }
  return v;
}
__device__ __forceinline__ int warp_max(int v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ int warp_sum(int v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The level of a group of n particles: the rows that hold them when every lane
// is filled equally, plus kLevelRows.
__device__ __forceinline__ int group_level(int n) { return n > 0 ? (n + kLanes - 1) / kLanes + kLevelRows : 0; }

// One warp per group, from the (stayers + movers) counts of its 32 cells: the
// level, gmax = the level of the group with every lane's refill reserve
// counted, plus the slack, and where the group's strangers go: the slots free
// below the level, numbered lane by lane (NewLayout::free). All of it is the
// new layout's: the sort may still find that it does not fit, and the present
// layout then goes on.
__global__ void group_size_kernel(Geom g, TileGeom t, const int* __restrict__ stay,
                                  const int* __restrict__ moved, SourceParams refill, int* gmax,
                                  int* newlevel, int2* free, int* gcap) {
  const int G = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (G >= t.ngroups) return;
  LaneCell lc;
  const int home = home_key(g, t, G, lane, lc);
  const int cell = home >= 0 ? stay[home] + moved[home] : 0, need = refill_need(refill, g, t, G, lane);
  const int c = lane_share(cell, lc);
  const int level = group_level(warp_sum(c));
  const int room = group_level(warp_sum(max(c, reserve_of(lane_share(need, lc)))));
  const int fullest = warp_max(max(cell, reserve_of(need)));
  const int rows = room > 0 ? min(room + room / kSlackDiv + kSlackRows, fullest + fullest / kFullestDiv + kFullestRows) : 0;
  const int free_below = max(level - c, 0);
  free[G * kLanes + lane] = make_int2(warp_scan(free_below) - free_below, min(c, level));
  if (lane == 0) {
    gmax[G] = rows;
    newlevel[G] = level;
    gcap[G] = rows * kLanes;
  }
}

// The first pass that writes the new layout: marks the slots of every lane
// column above its own particles empty (the strangers among them are written
// afterwards) and sets the groups' levels and tops.
template <typename CellArray>
__global__ void group_pad_kernel(Geom g, TileGeom t, const int* __restrict__ stay,
                                 const int* __restrict__ moved, const int* __restrict__ goff,
                                 const int* __restrict__ gmax, const int* __restrict__ newlevel, int* glevel,
                                 int* gtop, CellArray cell) {
  const int G = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (G >= t.ngroups) return;
  LaneCell lc;
  const int home = home_key(g, t, G, lane, lc);
  const int c = min(home >= 0 ? lane_share(stay[home] + moved[home], lc) : 0, newlevel[G]);
  const int m = gmax[G], base = goff[G];
  if (lane == 0) gtop[G] = glevel[G] = newlevel[G];
  for (int r = c; r < m; ++r) cell[base + r * kLanes + lane] = -1;
}

// The new layout of a full sort, as the scatter kernels need it.
struct NewLayout {
  const int* goff;
  const int* level;   // per group (group_size_kernel)
  const int2* free;   // per lane of each group: its first stranger's number in the group, its first free row
  const int* stay;    // per cell: stayers
  int* cursor;        // per cell: movers placed so far
  int* gcursor;       // per group: strangers placed so far
};

// Slot of the particle ranked `rank` of cell z of group G, whose z tile has nv
// cells: one of its own columns below the level, else the group's next free
// slot (the slots below the level hold the whole group, so every stranger
// finds one).
__device__ __forceinline__ int layout_slot(const NewLayout& nl, int nv, int G, int z, int rank) {
  const int base = nl.goff[G];
  const int n = lanes_of(nv, z), row = rank / n;
  if (row < nl.level[G]) return base + row * kLanes + z + (rank - row * n) * nv;
  const int q = atomicAdd(nl.gcursor + G, 1);
  const int2* f = nl.free + G * kLanes;
  int b = 0;  // the last lane whose strangers start at or before number q: it has free slots
#pragma unroll
  for (int s = 16; s > 0; s >>= 1)
    if (f[b + s].x <= q) b += s;
  return base + (f[b].y + q - f[b].x) * kLanes + b;
}

template <typename real>
__device__ __forceinline__ void copy_particle(const Parts<real>& P, int s, const Parts<real>& Q, int d,
                                              int c) {
  copy_record(P, s, Q, d, c);
}

// Scatter over the tiled slots: a stayer keeps its place in its column order;
// a mover goes after the stayers of its new cell.
template <typename real>
__global__ void tiled_scatter_kernel(Parts<real> P, Geom g, TileGeom t, const int* __restrict__ goff_old,
                                     const int* __restrict__ gmax_old, NewLayout nl, Parts<real> Q) {
  const int G = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (G >= t.ngroups) return;
  LaneCell lc;
  int home = home_key(g, t, G, lane, lc);
  if (lc.n > 1) home = -1;  // as in tiled_count_kernel
  const int base = goff_old[G], m = gmax_old[G];
  int rnew = 0;
  constexpr int U = 4;  // rows whose loads are in flight together
  for (int r0 = 0; r0 < m; r0 += U) {
    int cell[U];
    real o[U][3], v[U][3];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int s = base + (r0 + u) * kLanes + lane;
      const bool in = r0 + u < m;
      cell[u] = in ? P.cell[s] : -1;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        o[u][a] = in ? P.o[a][s] : (real)0;
        v[u][a] = in ? P.v[a][s] : (real)0;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int key = interior_key(g, cell[u]);
      if (key < 0) continue;
      int d;
      if (key == home) {
        d = layout_slot(nl, kLanes, G, lane, rnew);  // a cell of one lane
        ++rnew;
      } else {
        int l2;
        const int G2 = group_of_key(g, t, key, l2);
        d = layout_slot(nl, cells_of_group(g, t, G2), G2, l2, nl.stay[key] + atomicAdd(nl.cursor + key, 1));
      }
      Q.cell[d] = cell[u];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        Q.o[a][d] = o[u][a];
        Q.v[a][d] = v[u][a];
      }
    }
  }
}

template <typename real>
__global__ void append_scatter_kernel(Parts<real> P, int first, const int* __restrict__ count, Geom g,
                                      TileGeom t, NewLayout nl, Parts<real> Q) {
  const int n = *count;
  for (int s = first + blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
    const int c = P.cell[s];
    const int key = interior_key(g, c);
    if (key < 0) continue;
    int l2;
    const int G2 = group_of_key(g, t, key, l2);
    copy_particle(P, s, Q, layout_slot(nl, cells_of_group(g, t, G2), G2, l2, nl.stay[key] + atomicAdd(nl.cursor + key, 1)),
                  c);
  }
}

__global__ void tiled_total_kernel(const int* goff, const int* gcap, int ngroups, int* count_dev) {
  *count_dev = goff[ngroups - 1] + gcap[ngroups - 1];
}

// ------------------------------------------------------------ the push
__device__ __forceinline__ void red_add_v4(float* p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};"
               :: "l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// Density deposit into the window at node s, the base of the particle's 2x2x2
// stencil (X, Y, Z hold the half-shifted weights). FP64 adds the weight. FP32
// sums in fixed point: the 2x2x2 area weights (each in [0, 1], summing to 1)
// scaled by `scale` and rounded, added with integer shared-memory reductions,
// which need no compare-and-swap loop and give a sum that does not depend on
// the order of the particles. The caller picks `scale` so that no node can
// overflow: a node collects at most one unit of weight from each particle of
// the tile, so scale = (2^32 - 1) / (slots + 1) is safe; it is also kept below
// 2^23 for the rounding below. With 64 particles per cell this resolves
// 2^-17.7 of a particle's weight, as fine as an FP32 sum of the same node.
__device__ __forceinline__ void red_shared_u32(const unsigned* p, unsigned v) {
  asm volatile("red.shared.add.u32 [%0], %1;" :: "r"((unsigned)__cvta_generic_to_shared(p)), "r"(v) : "memory");
}
template <int WY, int WZ, typename W>
__device__ __forceinline__ void add_density(float* win, float scale, const W& X, const W& Y, const W& Z) {
  // the eight node weights rounded to integers by adding 2^23 in the FMA: the
  // sum's low mantissa bits are then the rounded weight, with no
  // float-to-integer conversion; the two x planes travel as one packed pair
  const unsigned* s = reinterpret_cast<const unsigned*>(win);
  constexpr float kM = 8388608.f;       // 2^23
  constexpr unsigned kMBits = 0x4B000000u;  // its bit pattern
  const float2 M = make_float2(kM, kM);
  const float2 ax = __fmul2_rn(make_float2(X.b0, X.b1), make_float2(scale, scale));
  const float2 ay0 = __fmul2_rn(ax, make_float2(Y.b0, Y.b0));  // (a00, a10)
  const float2 ay1 = __fmul2_rn(ax, make_float2(Y.b1, Y.b1));  // (a01, a11)
  const float2 Z0 = make_float2(Z.b0, Z.b0), Z1 = make_float2(Z.b1, Z.b1);
  const float2 t00 = __ffma2_rn(ay0, Z0, M), t01 = __ffma2_rn(ay0, Z1, M);
  const float2 t10 = __ffma2_rn(ay1, Z0, M), t11 = __ffma2_rn(ay1, Z1, M);
  red_shared_u32(s, __float_as_uint(t00.x) - kMBits);
  red_shared_u32(s + 1, __float_as_uint(t01.x) - kMBits);
  red_shared_u32(s + WZ, __float_as_uint(t10.x) - kMBits);
  red_shared_u32(s + WZ + 1, __float_as_uint(t11.x) - kMBits);
  red_shared_u32(s + WY * WZ, __float_as_uint(t00.y) - kMBits);
  red_shared_u32(s + WY * WZ + 1, __float_as_uint(t01.y) - kMBits);
  red_shared_u32(s + WY * WZ + WZ, __float_as_uint(t10.y) - kMBits);
  red_shared_u32(s + WY * WZ + WZ + 1, __float_as_uint(t11.y) - kMBits);
}
template <int WY, int WZ, typename W>
__device__ __forceinline__ void add_density(double* s, double weight, const W& X, const W& Y, const W& Z) {
  const double a0 = weight * X.b0, a1 = weight * X.b1;
  const double a00 = a0 * Y.b0, a01 = a0 * Y.b1, a10 = a1 * Y.b0, a11 = a1 * Y.b1;
  atomicAdd(s, a00 * Z.b0);
  atomicAdd(s + 1, a00 * Z.b1);
  atomicAdd(s + WZ, a01 * Z.b0);
  atomicAdd(s + WZ + 1, a01 * Z.b1);
  atomicAdd(s + WY * WZ, a10 * Z.b0);
  atomicAdd(s + WY * WZ + 1, a10 * Z.b1);
  atomicAdd(s + WY * WZ + WZ, a11 * Z.b0);
  atomicAdd(s + WY * WZ + WZ + 1, a11 * Z.b1);
}

// Half-shifted weights of a particle at offset f of its home cell h (an
// interior cell) as a 3-vector over the nodes h-1, h, h+1: with g = f - 1/2
// they are (max(-g, 0), 1 - |g|, max(g, 0)).
template <typename real>
struct W3 {
  real w[3];
};
__device__ __forceinline__ W3<float> home3(float f) {
  const float g = f - 0.5f;
  W3<float> r;
  r.w[0] = fmaxf(-g, 0.f);
  r.w[1] = 1.f - fabsf(g);
  r.w[2] = fmaxf(g, 0.f);
  return r;
}
// FP64: the same from the reference's base and weights, rounded as it rounds.
__device__ __forceinline__ W3<double> home3(double f) {
  const bool up = f >= 0.5;
  const double b1 = up ? f - 0.5 : f + 0.5, b0 = 1.0 - b1;
  W3<double> r;
  r.w[0] = up ? 0.0 : b0;
  r.w[1] = up ? b0 : b1;
  r.w[2] = up ? b1 : 0.0;
  return r;
}

// cal_track4's square roots and divisions: exact in FP64, rsqrt/fast
// reciprocal in FP32 (relative error ~1e-7, below the FP32 path's tolerance).
__device__ __forceinline__ float c_over_sqrt(float c, float x) { return c * rsqrtf(x); }
__device__ __forceinline__ double c_over_sqrt(double c, double x) { return c / sqrt(x); }
__device__ __forceinline__ float quot(float a, float b) { return __fdividef(a, b); }
__device__ __forceinline__ double quot(double a, double b) { return a / b; }

template <typename real>
__device__ __forceinline__ void boris4_fast(const PushConst<real>& pc, Gathered<real> e, real& vx,
                                            real& vy, real& vz) {
  const real T = pc.T, C = pc.C;
  e.ex += pc.ex_add;
  e.ey += pc.ey_add;
  real g1 = c_over_sqrt(C, pc.C2 - vx * vx - vy * vy - vz * vz);
  if (isnan(g1)) g1 = (real)0;
  real ux = g1 * vx, uy = g1 * vy, uz = g1 * vz;
  real g2 = c_over_sqrt(C, pc.C2 + ux * ux + uy * uy + uz * uz);
  const real bux = g2 * e.bx, buy = g2 * e.by, buz = g2 * e.bz;
  const real S = quot((real)2 * T, (real)1 + T * T * (bux * bux + buy * buy + buz * buz));
  ux += e.ex * T;
  uy += e.ey * T;
  uz += e.ez * T;
  const real uox = ux + T * (uy * buz - uz * buy);
  const real uoy = uy + T * (uz * bux - ux * buz);
  const real uoz = uz + T * (ux * buy - uy * bux);
  real upx = ux + S * (uoy * buz - uoz * buy);
  real upy = uy + S * (uoz * bux - uox * buz);
  real upz = uz + S * (uox * buy - uoy * bux);
  upx += e.ex * T;
  upy += e.ey * T;
  upz += e.ez * T;
  g2 = c_over_sqrt(C, pc.C2 + upx * upx + upy * upy + upz * upz);
  vx = g2 * upx;
  vy = g2 * upy;
  vz = g2 * upz;
}


}  // namespace pb
