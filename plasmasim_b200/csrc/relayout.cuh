// In-place re-layout of the tiled particle layout (tiled.cuh).
//
// Between two sorts most particles stay in their home cell. A re-layout
// leaves those where they are and moves only the rest:
//  1. classify (one warp per group): a particle whose cell belongs to another
//     lane of its group is handed to that lane on the spot; one that has left
//     the group is copied to the append region after `count` and its slot
//     becomes a hole (cell = -1); each lane lists the rows of its holes, in row
//     order, in a scratch array laid out like the slots themselves. A warp
//     takes append slots 64 at a time from the shared counter and marks the
//     slots of its last block it does not use empty, so the counter sees one
//     atomic per 64 movers instead of one per row;
//  2. place (movers and refilled particles, all appended after `count`): the
//     particles are bucketed by their new cell -- a rank per particle from a
//     per-cell counter, an exclusive scan of the arrivals, the particle's
//     index written to its bucket slot -- and then one warp per group fills
//     the holes below the group's level (tiled.cuh), in row order: each lane
//     its own from its cell's bucket, then the lanes with holes left from the
//     buckets that did not fit (strangers). The particles of a group beyond
//     its rows are copied, compacted, into the spare buffer. Every pass
//     streams its input, so its scattered accesses are independent of one
//     another;
//  3. the particles without a hole are copied back right after the layout,
//     where the slot-order push handles them until a later re-layout finds
//     them a hole (or a full sort, when they become too many).
// Particles outside the interior are dropped, as the reference's sort drops
// them.
#pragma once

#include "common.cuh"
#include "particles.cuh"
#include "tiled.cuh"

namespace pb {

constexpr int kAppendBlock = 64;

template <typename real>
__device__ __forceinline__ void copy_slot(const Parts<real>& S, int s, const Parts<real>& D, int d, int c) {
  copy_record(S, s, D, d, c);
}

// A warp's particles on their way to another lane of their group: up to
// kPending for each lane.
constexpr int kPending = 4;
template <typename real>
struct Pending {
  real a[kPending][kLanes][4], b[kPending][kLanes][4];  // records A, B
  int n[kLanes];
};
__device__ __forceinline__ void put_record(float (&a)[4], float (&b)[4], const Rec<float>& r) {
  *reinterpret_cast<float4*>(a) = make_float4(__int_as_float(r.cell), r.o[0], r.o[1], r.o[2]);
  *reinterpret_cast<float4*>(b) = make_float4(r.v[0], r.v[1], r.v[2], 0.f);
}
__device__ __forceinline__ void put_record(double (&a)[4], double (&b)[4], const Rec<double>& r) {
  double2* pa = reinterpret_cast<double2*>(a);
  double2* pb = reinterpret_cast<double2*>(b);
  pa[0] = make_double2(__hiloint2double(0, r.cell), r.o[0]);
  pa[1] = make_double2(r.o[1], r.o[2]);
  pb[0] = make_double2(r.v[0], r.v[1]);
  pb[1] = make_double2(r.v[2], 0.0);
}
template <typename real>
__device__ __forceinline__ Rec<real> get_record(const real (&a)[4], const real (&b)[4]) {
  return Rec<real>{word_int(a[0]), {a[1], a[2], a[3]}, {b[0], b[1], b[2]}};
}

// One warp per group walks its rows, kRowsTogether at a time. A particle in
// its lane's home cell stays. One whose cell belongs to another lane of the
// group -- most of those that leave their cell do so along z, the drift's axis
// -- goes to that lane's pending list in shared memory, and after each batch
// of rows every lane copies its pending particles into its holes below the
// group's level that lie in the rows read so far; where the list is full the
// particle stays as a stranger. The others, and what is pending at the end,
// go to the append region, from where the placement takes them. Each lane
// lists the rows of its holes in order; the first hfirst of them are filled.
// With `shell` set (the re-layout after a refill), a particle of the layout
// that lies in a refill shell is deleted here, as add_*_flat's removal
// (:6015-6031) would have: one pass over the layout for both.
//
// Bound by the latency of a batch (cells, then the movers' records, then the
// pending lists) and its instructions; the next batch's cells are loaded ahead,
// and 24 warps per SM (80 registers) were faster than 16 or 32. With every
// mover in the append region the re-layout of both species took 2.00 ms per
// step at 128^3 x 64, this way 1.41; 0.092 -> 0.084 at 64^3 x 16, FP64 64^3 x 32
// 0.185 -> 0.165.
constexpr int kRowsTogether = 4;
template <typename real>
__global__ void __launch_bounds__(256, sizeof(real) == 4 ? 3 : 2) classify_kernel(Parts<real> P, Geom g, TileGeom t, const int* goff,
                                                       const int* gmax, const int* glevel, int* gtop,
                                                       int cap, int* holes, int* nholes, int* hfirst, int* append_at,
                                                       int* nonhome, int shell) {
  after_prior();
  constexpr int U = kRowsTogether;
  extern __shared__ __align__(16) unsigned char pending_raw[];
  const int G = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (G >= t.ngroups) return;  // warp-uniform
  Pending<real>& pend = reinterpret_cast<Pending<real>*>(pending_raw)[threadIdx.x >> 5];
  const unsigned below = (1u << lane) - 1u;
  int hi, hj, hk;
  LaneCell lc;
  const bool owns = home_cell(g, t, G, lane, hi, hj, hk, lc);
  const int home = owns ? pack_cell(hi, hj, hk) : -2;
  const int nv = cells_of_group(g, t, G);
  const int column = hi << (2 * kCellBits) | hj << kCellBits, z0 = hk - lc.z;  // the group's cells: column | z0 .. z0 + nv - 1
  const int base = goff[G], m = gmax[G], level = glevel[G];
  int nh = 0, hu = 0, top = 0;
  int nexth = 0;                          // row of hole hu, when hu < nh
  int blk = 0, used = kAppendBlock;       // current block of append slots (warp-uniform)
  pend.n[lane] = 0;
  __syncwarp();
  // Append slots for the lanes with `want`, -1 for the others; warp-uniform control.
  const auto append = [&](bool want) {
    const unsigned mm = __ballot_sync(0xffffffffu, want);
    const int nm = __popc(mm);
    if (nm > kAppendBlock - used) {  // close the block, take a new one
      for (int q = used + lane; q < kAppendBlock; q += kLanes)
        if (blk + q < cap) P.cell[blk + q] = -1;
      int nb = 0;
      if (lane == 0) nb = atomicAdd(append_at, kAppendBlock);
      blk = __shfl_sync(0xffffffffu, nb, 0);
      used = 0;
    }
    const int d = blk + used + __popc(mm & below);
    used += nm;
    return want ? d : -1;
  };
  const auto add_hole = [&](int r) {
    holes[base + nh * kLanes + lane] = r;
    if (nh == hu) nexth = r;
    ++nh;
  };
  int next[U];  // the next batch's cells, on their way
  const auto fetch = [&](int r0) {
#pragma unroll
    for (int u = 0; u < U; ++u) next[u] = r0 + u < m ? P.cell[base + (r0 + u) * kLanes + lane] : -1;
  };
  fetch(0);
  for (int r0 = 0; r0 < m; r0 += U) {
    int c[U], d[U], k[U], to[U];  // cell; append slot, pending entry and lane, -1 none
#pragma unroll
    for (int u = 0; u < U; ++u) c[u] = next[u];
    fetch(r0 + U);
    if (shell) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const long long tu = base + (r0 + u) * kLanes + lane;
        if (c[u] >= 0 && in_refill_shell(P, g, c[u], tu)) {
          P.cell[tu] = -1;
          c[u] = -1;
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int r = r0 + u, slot = base + r * kLanes + lane;
      d[u] = k[u] = -1;
      to[u] = 0;
      bool stays = c[u] == home, goes = false;
      if (c[u] >= 0 && !stays) {
        const int z = c[u] - (column | z0);  // below nv for the group's cells only
        if ((unsigned)z < (unsigned)nv && owns) {
          const int n = lanes_of(nv, z);
          to[u] = n == 1 ? z : z + nv * (r % n);
          k[u] = atomicAdd(&pend.n[to[u]], 1);
          if (k[u] >= kPending) {
            atomicSub(&pend.n[to[u]], 1);
            k[u] = -1;
            stays = true;
          }
        } else if (interior_key(g, c[u]) >= 0) {
          goes = true;
        } else {  // outside the interior: dropped
          P.cell[slot] = -1;
          c[u] = -1;
        }
      }
      d[u] = append(goes);
      if (goes && d[u] >= cap) {  // the append region is full: it stays where it is
        *nonhome = 1;
        d[u] = -1;
        stays = true;
      }
      if (stays) top = r + 1;
      else if (r < m) add_hole(r);
    }
    // the U rows' movers: their record loads issued together, then the copies
    Rec<real> rec[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (d[u] >= 0 || k[u] >= 0) rec[u] = load_records(P, base + (r0 + u) * kLanes + lane);
    __syncwarp();
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const Rec<real>& q = rec[u];
      if (d[u] >= 0) store_records(P, d[u], c[u], q.o[0], q.o[1], q.o[2], q.v[0], q.v[1], q.v[2]);
      if (k[u] >= 0) put_record(pend.a[k[u]][to[u]], pend.b[k[u]][to[u]], q);
      if (d[u] >= 0 || k[u] >= 0) P.cell[base + (r0 + u) * kLanes + lane] = -1;
    }
    __syncwarp();
    int np = pend.n[lane];
    while (np > 0 && hu < nh && nexth < level) {
      --np;
      const Rec<real> q = get_record(pend.a[np][lane], pend.b[np][lane]);
      store_records(P, base + nexth * kLanes + lane, q.cell, q.o[0], q.o[1], q.o[2], q.v[0], q.v[1], q.v[2]);
      top = max(top, nexth + 1);
      if (++hu < nh) nexth = holes[base + hu * kLanes + lane];
    }
    pend.n[lane] = np;
    __syncwarp();
  }
  // still pending: to the append region
  const int np = pend.n[lane];
#pragma unroll
  for (int q = 0; q < kPending; ++q) {
    const int d = append(q < np);
    const bool full = d >= cap;
    if (full) *nonhome = 1;
    if (d >= 0 && !full) {
      const Rec<real> p = get_record(pend.a[q][lane], pend.b[q][lane]);
      store_records(P, d, p.cell, p.o[0], p.o[1], p.o[2], p.v[0], p.v[1], p.v[2]);
    }
    // No room there: into the holes that are left in any lane. Every pending
    // particle left a hole in the group and every filled hole took one, so
    // there are as many holes as particles.
    for (unsigned left = __ballot_sync(0xffffffffu, full); left;) {  // warp-uniform
      const unsigned open = __ballot_sync(0xffffffffu, hu < nh);
      if (!open) break;
      int from = -1;
      for (unsigned o = open; o && left; o &= o - 1, left &= left - 1)
        if (lane == __ffs(o) - 1) from = __ffs(left) - 1;
      if (from >= 0) {
        const Rec<real> p = get_record(pend.a[q][from], pend.b[q][from]);
        store_records(P, base + nexth * kLanes + lane, p.cell, p.o[0], p.o[1], p.o[2], p.v[0], p.v[1], p.v[2]);
        top = max(top, nexth + 1);
        if (++hu < nh) nexth = holes[base + hu * kLanes + lane];
      }
    }
  }
  for (int q = used + lane; q < kAppendBlock; q += kLanes)
    if (blk + q < cap && used < kAppendBlock) P.cell[blk + q] = -1;
  nholes[G * kLanes + lane] = nh;
  hfirst[G * kLanes + lane] = hu;
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, s));
  if (lane == 0) gtop[G] = top;
}

// Before a re-layout: the append region starts at the count, and no spills, no
// particle left outside its home, no arrivals yet.
__global__ void relayout_begin_kernel(const int* count, int* append_at, int* nspill, int* nonhome, int* cursor,
                                      long long ncells) {
  after_prior();
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  for (long long c = t; c < ncells; c += (long long)gridDim.x * blockDim.x) cursor[c] = 0;
  if (t == 0) {
    *append_at = *count;
    *nspill = 0;
    *nonhome = 0;
  }
}

// Placement, pass 1: the particle's rank among the appended particles of its
// new cell (from the per-cell counter `cursor`); -1 for an empty slot or a
// particle outside the interior (dropped).
template <typename real>
__global__ void __launch_bounds__(256) place_count_kernel(Parts<real> P, int first, const int* append_at,
                                                          int cap, Geom g, int* cursor, int* rank) {
  after_prior();
  const int span = min(*append_at, cap) - first;
  const int lane = threadIdx.x & 31;
  const int stride = gridDim.x * blockDim.x;
  for (int w0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31; w0 < span; w0 += stride) {  // warp-uniform
    const int q = w0 + lane;
    const int key = q < span ? interior_key(g, P.cell[first + q]) : -1;
    const int r = warp_aggregated_inc(cursor, key < 0 ? 0 : key, key >= 0);
    if (q < span) rank[q] = key < 0 ? -1 : r;
  }
}

// Pass 2 (after an exclusive scan of the arrivals into bucket offsets): every
// particle writes its index to its bucket slot.
template <typename real>
__global__ void __launch_bounds__(256) place_bucket_kernel(Parts<real> P, int first, const int* append_at,
                                                           int cap, Geom g, const int* off,
                                                           const int* rank, int* bucket) {
  after_prior();
  const int span = min(*append_at, cap) - first;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < span; q += gridDim.x * blockDim.x) {
    const int r = rank[q];
    if (r >= 0) bucket[off[interior_key(g, P.cell[first + q])] + r] = q;
  }
}

// Pass 3, one warp per group: lane l copies the k-th particle of its home
// cell's bucket into the slot of its k-th hole below the level, U holes per
// lane in flight at once; then the particles that found no hole of their own
// lane go to the holes below the level that are left, the lowest of each lane
// first. The level counts the particles that stayed and those that arrive, so
// the holes below it hold all arrivals unless the group has outgrown its rows;
// what is left then goes to the spare buffer Q. gtop comes in as one past the
// last row that kept a particle and goes out covering the filled rows as well.
template <typename real>
__global__ void place_fill_kernel(Parts<real> P, int first, Geom g, TileGeom t, const int* goff,
                                  const int* gmax, int* glevel, int* gtop,
                                  const int* holes, const int* arrivals,
                                  const int* nholes, const int* hfirst,
                                  const int* off, const int* bucket, int* nspill,
                                  Parts<real> Q) {
  after_prior();
  constexpr int U = 4;  // holes per lane in flight together
  const int G = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (G >= t.ngroups) return;  // warp-uniform
  const unsigned below = (1u << lane) - 1u;
  LaneCell lc;
  const int home = home_key(g, t, G, lane, lc);
  // this lane's entries of its cell's bucket: o, o + lc.n, ...
  const int arr = home >= 0 ? lane_share(arrivals[home], lc) : 0;
  const int narr = warp_sum(arr);
  if (narr == 0) return;
  const int o = home >= 0 ? off[home] + lc.m : 0;
  const int hu = hfirst[G * kLanes + lane], nh = nholes[G * kLanes + lane] - hu;
  const int base = goff[G], rows = gmax[G];
  const int* hole = holes + base + hu * kLanes + lane;  // the lane's k-th hole: hole[k * kLanes]
  const int level = min(rows, group_level(rows * kLanes - warp_sum(nh) + narr));
  if (lane == 0) glevel[G] = level;
  const int n = min(arr, nh);
  int top = gtop[G];
  int used = 0;  // holes this lane has filled
  for (int k0 = 0;; k0 += U) {
    int src[U], dst[U];
    bool more = false;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = k0 + u;
      const int row = k < n ? hole[k * kLanes] : level;
      src[u] = row < level ? first + bucket[o + k * lc.n] : -1;
      dst[u] = base + row * kLanes + lane;
      if (row < level) {
        top = max(top, row + 1);
        used = k + 1;
        more = u == U - 1;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (src[u] >= 0) copy_record(P, src[u], P, dst[u], P.cell[src[u]]);
    if (!__any_sync(0xffffffffu, more)) break;
  }
  // strangers: number s of the group is entry used + (s - pre) of its lane's
  const int rest = arr - used;
  const int pre = warp_scan(rest) - rest;
  const int nrest = warp_sum(rest);
  int done = 0;
  for (int k = used; done < nrest; ++k) {
    const int row = k < nh ? hole[k * kLanes] : level;
    const unsigned m = __ballot_sync(0xffffffffu, row < level);
    if (!m) break;
    const int s = done + __popc(m & below);
    int b = 0;  // the last lane whose strangers start at or before s
#pragma unroll
    for (int q = 16; q > 0; q >>= 1)
      if (__shfl_sync(0xffffffffu, pre, b + q) <= s) b += q;
    const int e = __shfl_sync(0xffffffffu, o, b) + (__shfl_sync(0xffffffffu, used - pre, b) + s) * __shfl_sync(0xffffffffu, lc.n, b);
    if (row < level && s < nrest) {
      const int src = first + bucket[e];
      top = max(top, row + 1);
      copy_record(P, src, P, base + row * kLanes + lane, P.cell[src]);
    }
    done += __popc(m);
  }
  // a group that has outgrown its rows
  for (int s0 = done; s0 < nrest; s0 += kLanes) {
    const int s = s0 + lane;
    int b = 0;
#pragma unroll
    for (int q = 16; q > 0; q >>= 1)
      if (__shfl_sync(0xffffffffu, pre, b + q) <= s) b += q;
    const int e = __shfl_sync(0xffffffffu, o, b) + (__shfl_sync(0xffffffffu, used - pre, b) + s) * __shfl_sync(0xffffffffu, lc.n, b);
    int sb = 0;
    if (lane == 0) sb = atomicAdd(nspill, min(kLanes, nrest - s0));
    sb = __shfl_sync(0xffffffffu, sb, 0);
    if (s < nrest) {
      const int src = first + bucket[e];
      copy_record(P, src, Q, sb + lane, P.cell[src]);
    }
  }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, s));
  if (lane == 0) gtop[G] = top;
}

// The particles without a hole back to slots [first, first + n), where the
// count then ends.
template <typename real>
__global__ void unspill_kernel(Parts<real> Q, const int* nspill, Parts<real> P, int first, int* count) {
  after_prior();
  const int n = *nspill;
  if (blockIdx.x == 0 && threadIdx.x == 0) *count = first + n;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x)
    copy_slot(Q, q, P, first + q, Q.cell[q]);
}

}  // namespace pb
