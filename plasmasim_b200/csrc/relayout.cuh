// In-place re-layout of the tiled particle layout (tiled.cuh).
//
// Between two sorts most particles stay in their home cell. A re-layout
// leaves those where they are and moves only the rest:
//  1. classify (one warp per group): a particle whose cell is not its lane's
//     home cell (it moved, or sits in another lane's free slot) is copied to
//     the append region after `count` and its slot becomes a hole (cell = -1);
//     each lane lists the rows of its holes, in row order, in a scratch array
//     laid out like the slots themselves. A warp takes append slots 64 at a
//     time from the shared counter and marks the slots of its last block it
//     does not use empty, so the counter sees one atomic per 64 movers instead
//     of one per row;
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

// With `shell` set (the re-layout after a refill), a particle of the layout
// that lies in a refill shell is deleted here, as add_*_flat's removal
// (:6015-6031) would have: one pass over the layout for both.
template <typename real>
__global__ void classify_kernel(Parts<real> P, Geom g, TileGeom t, const int* __restrict__ goff,
                                const int* __restrict__ gmax, int* gtop, int cap, int* holes, int* nholes,
                                int* append_at, int* nonhome, int shell) {
  after_prior();
  constexpr int U = 4;  // rows whose loads are in flight together (8 measured no faster)
  const int G = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (G >= t.ngroups) return;  // warp-uniform
  const unsigned below = (1u << lane) - 1u;
  LaneCell lc;
  const int home = home_key(g, t, G, lane, lc);
  const int base = goff[G], m = gmax[G];
  int nh = 0, top = 0;
  int blk = 0, used = kAppendBlock;  // current block of append slots (warp-uniform)
  for (int r0 = 0; r0 < m; r0 += U) {
    int c[U], d[U];
    bool moved[U];
#pragma unroll
    for (int u = 0; u < U; ++u) c[u] = r0 + u < m ? P.cell[base + (r0 + u) * kLanes + lane] : -1;
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
      const int r = r0 + u;
      const int key = interior_key(g, c[u]);
      const bool leaves = c[u] >= 0 && (key < 0 || key != home);
      const bool mover = leaves && key >= 0;
      const unsigned mm = __ballot_sync(0xffffffffu, mover);
      const int nm = __popc(mm);
      if (nm > kAppendBlock - used) {  // close the block, take a new one
        for (int q = used + lane; q < kAppendBlock; q += kLanes)
          if (blk + q < cap) P.cell[blk + q] = -1;
        int nb = 0;
        if (lane == 0) nb = atomicAdd(append_at, kAppendBlock);
        blk = __shfl_sync(0xffffffffu, nb, 0);
        used = 0;
      }
      d[u] = blk + used + __popc(mm & below);
      used += nm;
      // a mover that finds the append region full stays where it is
      moved[u] = mover && d[u] < cap;
      if (mover && !moved[u]) *nonhome = 1;
      const bool hole = c[u] < 0 || (leaves && (moved[u] || !mover));
      if (hole && c[u] >= 0 && !moved[u]) P.cell[base + r * kLanes + lane] = -1;
      if (hole && r < m) {
        holes[base + nh * kLanes + lane] = r;
        ++nh;
      }
      if (!hole) top = r + 1;  // a particle stays in this row
    }
    // the movers of the U rows: their record loads issued together, then the copies
    Rec<real> rec[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (moved[u]) rec[u] = load_records(P, base + (r0 + u) * kLanes + lane);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (moved[u]) {
        const Rec<real>& q = rec[u];
        store_records(P, d[u], c[u], q.o[0], q.o[1], q.o[2], q.v[0], q.v[1], q.v[2]);
        P.cell[base + (r0 + u) * kLanes + lane] = -1;
      }
  }
  for (int q = used + lane; q < kAppendBlock; q += kLanes)
    if (blk + q < cap && used < kAppendBlock) P.cell[blk + q] = -1;
  nholes[G * kLanes + lane] = nh;
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
                                                           int cap, Geom g, const int* __restrict__ off,
                                                           const int* __restrict__ rank, int* bucket) {
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
__global__ void place_fill_kernel(Parts<real> P, int first, Geom g, TileGeom t, const int* __restrict__ goff,
                                  const int* __restrict__ gmax, int* gtop, const int* __restrict__ holes,
                                  const int* __restrict__ arrivals, const int* __restrict__ nholes,
                                  const int* __restrict__ off, const int* __restrict__ bucket, int* nspill,
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
  const int nh = nholes[G * kLanes + lane];
  const int base = goff[G], rows = gmax[G];
  const int level = min(rows, group_level(rows * kLanes - warp_sum(nh) + narr));
  const int n = min(arr, nh);
  int top = gtop[G];
  int used = 0;  // holes this lane has filled
  for (int k0 = 0;; k0 += U) {
    int src[U], dst[U];
    bool more = false;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = k0 + u;
      const int row = k < n ? holes[base + k * kLanes + lane] : level;
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
    const int row = k < nh ? holes[base + k * kLanes + lane] : level;
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
