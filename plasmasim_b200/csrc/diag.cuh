// FP64 diagnostics: the thrust and energy sums of thrust_f / thrust_fave and
// the Gauss-law residual. Particle and field values are read in the step's
// precision; every product and sum is formed in double.
#pragma once

#include "common.cuh"
#include "particles.cuh"
#include "push_tiled.cuh"
#include "tiled.cuh"

namespace pb {

template <int N>
__device__ __forceinline__ void block_reduce_add(double (&v)[N], double* out, const int* idx,
                                                 const double* scale) {
  __shared__ double sm[N][32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < N; ++q) {
    double x = v[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) sm[q][wid] = x;
  }
  __syncthreads();
  if (wid == 0) {
    const int nw = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int q = 0; q < N; ++q) {
      double x = lane < nw ? sm[q][lane] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
      if (lane == 0 && idx[q] >= 0) atomicAdd(out + idx[q], x * scale[q]);
    }
  }
}

// thrust_f's central box on one axis, (0.2 N dx, 0.8 N dx) open (:4984-4988),
// as cells and offsets: a particle (i, f) is above its lower face when i > cl
// or i == cl and f > fl, below its upper one when i < ch or i == ch and
// f <= fh. The host finds the offsets at which the reference's comparison of
// x = (i + f) dx in FP64 changes, so the result is the same for every (i, f).
template <typename real>
struct BoxAxis {
  int cl, ch;
  real fl, fh;
};

// One species' store as the sums walk it: the rows in use of every group of
// the tiled layout, then the slots from `tail` to the count.
template <typename real>
struct ThrustStore {
  Parts<real> P;
  const int* goff;
  const int* gtop;
  int layout;        // 0: every slot is in the tail
  int near;          // near tiles, 0 without a layout
  int tail;
  const int* count;
  double scale;      // s_p q n dx^3
  double ke;         // m n dx^3 / 2
};

struct CellBox {
  double lo[3], hi[3];   // open box on k-2, l-2, m-2 (:4965-4967)
  int ox, oy;            // myrank_x Grid_Nx, myrank_y Grid_Ny (:4971-4972)
  double e0, inv_mu0;
};

template <typename real>
struct ThrustArgs {
  ThrustStore<real> sp[2];
  Fields<real> F;
  Geom g;
  BoxAxis<real> box[3];
  CellBox cells;
  double* raw;       // 7 sums of each species (E, v x B, v^2), 2 of the fields; zero between launches
  unsigned* ticket;  // blocks done; zero between launches
  TileGeom tg;
  struct { int lo[3], n[3]; } near;  // tiles that reach into the box
  int nfar;          // blocks per species for the rest of its store
  bool vec;          // FP32 planes whose rows are multiples of 16 bytes
  double* acc;       // F[27], E[6]
  double* fave;      // when set, the running mean gains F / 500 (thrust_fave :5265-5267)
};

constexpr int kThrustRaw = 16;

template <typename real>
__device__ __forceinline__ bool in_axis(const BoxAxis<real>& b, int i, real f) {
  return (i > b.cl || (i == b.cl && f > b.fl)) && (i < b.ch || (i == b.ch && f <= b.fh));
}

// E and B at a particle: from the tile's window when its stencil lies in it.
struct ThrustWin {
  const float* fw;   // null without one
  int x0, y0, z0;
};
using ThrustPlan = PushSmem<float>;

__device__ __forceinline__ Gathered<double> thrust_gather(const ThrustWin&, const Fields<double>& F, const Geom& g,
                                                          const Rec<double>& q, int i, int j, int k) {
  return gather6(F, g, axis_weights(i, q.o[0]), axis_weights(j, q.o[1]), axis_weights(k, q.o[2]));
}
__device__ __forceinline__ Gathered<float> thrust_gather(const ThrustWin& w, const Fields<float>& F, const Geom& g,
                                                         const Rec<float>& q, int i, int j, int k) {
  using S = ThrustPlan;
  if (w.fw && i > 0 && j > 0 && k > 0 && i - 1 >= w.x0 && i + 1 < w.x0 + S::WX && j - 1 >= w.y0 &&
      j + 1 < w.y0 + S::WY && k - 1 >= w.z0 && k + 1 < w.z0 + S::WZ)
    return gather6_win<S::WY, S::WZ, S::WN>(w.fw + (((i - w.x0) * S::WY + j - w.y0) * S::WZ + k - w.z0),
                                            win_axis(q.o[0], S::WY * S::WZ), win_axis(q.o[1], S::WZ),
                                            win_axis(q.o[2], 1));
  return gather6(F, g, axis_weights(i, q.o[0]), axis_weights(j, q.o[1]), axis_weights(k, q.o[2]));
}

template <typename real>
__device__ __forceinline__ bool in_box(const ThrustArgs<real>& a, const Rec<real>& q, int& i, int& j, int& k) {
  unpack_cell(q.cell, i, j, k);
  return in_axis(a.box[0], i, q.o[0]) && in_axis(a.box[1], j, q.o[1]) && in_axis(a.box[2], k, q.o[2]);
}

// The terms of thrust_f (:4984-5101) of a particle in the box's cell (i, j, k).
template <typename real>
__device__ __forceinline__ void thrust_terms(const ThrustArgs<real>& a, const ThrustWin& win, int i, int j, int k,
                                             const Rec<real>& q, double (&s)[7]) {
  if (!stencil_ok(a.g, i, j, k)) return;
  const Gathered<real> e =
      thrust_gather(win, a.F, a.g, q, i, j, k);
  const double vx = q.v[0], vy = q.v[1], vz = q.v[2];
  const double bx = e.bx, by = e.by, bz = e.bz;
  s[0] += (double)e.ex;
  s[1] += (double)e.ey;
  s[2] += (double)e.ez;
  s[3] += vy * bz - vz * by;
  s[4] += vz * bx - vx * bz;
  s[5] += vx * by - vy * bx;
  s[6] += vx * vx + vy * vy + vz * vz;
}

template <typename real>
__device__ __forceinline__ Rec<real> empty_rec() {
  return Rec<real>{-1, {(real)0, (real)0, (real)0}, {(real)0, (real)0, (real)0}};
}
// Record A of particle t, its velocity left zero.
__device__ __forceinline__ Rec<float> load_record_a(const Parts<float>& P, int t) {
  const float4 a = reinterpret_cast<const float4*>(P.ra)[t];
  return Rec<float>{__float_as_int(a.x), {a.y, a.z, a.w}, {0.f, 0.f, 0.f}};
}
__device__ __forceinline__ Rec<double> load_record_a(const Parts<double>& P, int t) {
  const double2* a = reinterpret_cast<const double2*>(P.ra + 4 * (long long)t);
  const double2 a0 = a[0], a1 = a[1];
  return Rec<double>{__double2loint(a0.x), {a0.y, a1.x, a1.y}, {0., 0., 0.}};
}

// thrust_f (:4963-5101): E, v x B and v^2 summed over the particles of each
// species inside the central box, the field energies over its nodes (no volume
// factor, as in the reference); the last block to finish forms F and E, adds
// F / 500 to the running mean and clears the sums.
//
// A grid of three kinds of blocks, the dearest first: one per species and tile
// that reaches into the box (`near`, a box of tiles), `nfar` per species that
// walk the other tiles and the tail, the rest over the nodes. A near block
// stages E and B of its tile in shared memory as the push does (FP32); one
// warp walks a group's rows in use, U records in flight. In a far tile only
// record A is read, and B of the rare particle that has come into the box.
//
// Bound by instruction issue over the near tiles' particles (the gathers and
// FP64 sums; reading every record A, 16 bytes a particle, takes a third of the
// time). The box test is one of cells and FP32 offsets; E + v x B, which the
// reference sums beside E and v x B, is formed from the two sums; both
// species, the fields and the mean share one launch. Per step, a kernel each
// for the fields and the species with a test in FP64 per particle -> this:
// 0.162 -> 0.094 ms at 64^3 x 16, 0.063 -> 0.023 at 32^3 x 8, 0.469 ->
// 0.319 at 96 x 96 x 128 x 16. (Blocks that took tiles from an atomic
// counter: 0.099, 0.034, 0.316.)
template <typename real>
__global__ void __launch_bounds__(256, 3) thrust_kernel(const __grid_constant__ ThrustArgs<real> a) {
  after_prior();
  using S = ThrustPlan;
  constexpr int U = sizeof(real) == 4 ? 4 : 2;
  constexpr bool kWin = sizeof(real) == 4;
  extern __shared__ __align__(16) float thrust_win[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Geom& g = a.g;
  const int nnear = a.sp[0].near + a.sp[1].near;
  double s[7] = {0., 0., 0., 0., 0., 0., 0.};
  int ph;
  if ((int)blockIdx.x < nnear) {
    ph = (int)blockIdx.x >= a.sp[0].near;
    const ThrustStore<real>& st = a.sp[ph];
    const Parts<real>& P = st.P;
    int b = ph ? (int)blockIdx.x - a.sp[0].near : (int)blockIdx.x;
    const int tz = a.near.lo[2] + b % a.near.n[2];
    b /= a.near.n[2];
    const int ty = a.near.lo[1] + b % a.near.n[1], tx = a.near.lo[0] + b / a.near.n[1];
    ThrustWin win{nullptr, tx * kTileX, ty * kTileY, tz * kLanes};
    const int G = ((tx * a.tg.nty + ty) * a.tg.ntz + tz) * (kTileX * kTileY) + warp;
    const int base = st.goff[G] + lane, m = st.gtop[G];
    Rec<real> q[U];
    const auto fetch = [&](int r0) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        q[u] = r0 + u < m ? load_records(P, base + (r0 + u) * kLanes) : empty_rec<real>();
    };
    fetch(0);
    if constexpr (kWin) {
      if (a.vec) fill_win<float, S::WX, S::WY, S::WZ, true, 2>(thrust_win, a.F, g, win.x0, win.y0, win.z0);
      else fill_win<float, S::WX, S::WY, S::WZ, false, 2>(thrust_win, a.F, g, win.x0, win.y0, win.z0);
      win.fw = thrust_win;
      __syncthreads();
    }
    for (int r0 = 0; r0 < m; r0 += U) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        int i, j, k;
        if (q[u].cell >= 0 && in_box(a, q[u], i, j, k)) thrust_terms(a, win, i, j, k, q[u], s);
      }
      fetch(r0 + U);
    }
  } else if ((int)blockIdx.x < nnear + 2 * a.nfar) {
    ph = (int)blockIdx.x - nnear >= a.nfar;
    const ThrustStore<real>& st = a.sp[ph];
    const Parts<real>& P = st.P;
    const ThrustWin none{nullptr, 0, 0, 0};
    const int f = (int)blockIdx.x - nnear - ph * a.nfar;
    if (st.layout) {  // its other tiles
      const int ntiles = a.tg.ntx * a.tg.nty * a.tg.ntz;
      for (int tile = f; tile < ntiles; tile += a.nfar) {
        const int tz = tile % a.tg.ntz, ty = (tile / a.tg.ntz) % a.tg.nty, tx = tile / (a.tg.ntz * a.tg.nty);
        if ((unsigned)(tx - a.near.lo[0]) < (unsigned)a.near.n[0] && (unsigned)(ty - a.near.lo[1]) < (unsigned)a.near.n[1] &&
            (unsigned)(tz - a.near.lo[2]) < (unsigned)a.near.n[2])
          continue;
        const int G = tile * (kTileX * kTileY) + warp;
        const int base = st.goff[G] + lane, m = st.gtop[G];
        constexpr int UF = 2 * U;
        for (int r0 = 0; r0 < m; r0 += UF) {
          Rec<real> q[UF];
#pragma unroll
          for (int u = 0; u < UF; ++u)
            q[u] = r0 + u < m ? load_record_a(P, base + (r0 + u) * kLanes) : empty_rec<real>();
#pragma unroll
          for (int u = 0; u < UF; ++u) {
            int i, j, k;
            if (q[u].cell >= 0 && in_box(a, q[u], i, j, k))  // it has come in from outside
              thrust_terms(a, none, i, j, k, load_records(P, base + (r0 + u) * kLanes), s);
          }
        }
      }
    }
    const int n = *st.count;
    for (int t = st.tail + f * blockDim.x + threadIdx.x; t < n; t += a.nfar * blockDim.x) {
      const Rec<real> q = load_records(P, t);
      int i, j, k;
      if (q.cell >= 0 && in_box(a, q, i, j, k)) thrust_terms(a, none, i, j, k, q, s);
    }
  } else {
    ph = 2;
    const CellBox& b = a.cells;
    const int nint = g.nx * g.ny * g.nz, first = nnear + 2 * a.nfar;
    for (int t = ((int)blockIdx.x - first) * blockDim.x + threadIdx.x; t < nint; t += (gridDim.x - first) * blockDim.x) {
      const int m = t % g.nz, l = (t / g.nz) % g.ny, k = t / (g.nz * g.ny);
      const int kg = b.ox + k, lg = b.oy + l;
      if (!(kg < b.hi[0] && kg > b.lo[0] && lg < b.hi[1] && lg > b.lo[1] && m < b.hi[2] && m > b.lo[2])) continue;
      const int n = (k + 2) * g.sx + (l + 2) * g.gz + (m + 2);
      const double ex = a.F.f[F_EX][n], ey = a.F.f[F_EY][n], ez = a.F.f[F_EZ][n];
      const double bx = a.F.f[F_BX][n], by = a.F.f[F_BY][n], bz = a.F.f[F_BZ][n];
      s[0] += ex * ex + ey * ey + ez * ez;
      s[1] += bx * bx + by * by + bz * bz;
    }
  }
  {
    const bool part = ph < 2;
    const int idx[7] = {0, 1, part ? 2 : -1, part ? 3 : -1, part ? 4 : -1, part ? 5 : -1, part ? 6 : -1};
    const double one[7] = {1., 1., 1., 1., 1., 1., 1.};
    block_reduce_add<7>(s, a.raw + 7 * ph, idx, one);
  }
  // the last block's first warp forms the results
  if (threadIdx.x >= 32) return;
  unsigned last = 0;
  if (lane == 0) {
    __threadfence();
    last = atomicAdd(a.ticket, 1u) == gridDim.x - 1;
    __threadfence();
  }
  if (!__shfl_sync(0xffffffffu, last, 0)) return;
  const double mine = lane < kThrustRaw ? __ldcg(a.raw + lane) : 0.0;
  double raw[kThrustRaw];
#pragma unroll
  for (int q = 0; q < kThrustRaw; ++q) raw[q] = __shfl_sync(0xffffffffu, mine, q);
  double f = 0.0;  // F[lane]
#pragma unroll
  for (int q = 0; q < 3; ++q)
    if (lane == q)
      f = a.sp[0].scale * (raw[q] + raw[3 + q]) + a.sp[1].scale * (raw[7 + q] + raw[10 + q]);
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    if (lane == 3 + q) f = a.sp[0].scale * raw[q];
    if (lane == 9 + q) f = a.sp[1].scale * raw[7 + q];
  }
  if (lane < 27) a.acc[lane] = f;
  if (a.fave && lane < 27) a.fave[lane] += f * (1.0 / 500.0);
  if (lane < 6) {
    double e = 0.0;
    if (lane == 0) e = 0.5 * a.cells.e0 * raw[14];
    if (lane == 1) e = 0.5 * a.cells.inv_mu0 * raw[15];
    if (lane == 2) e = a.sp[0].ke * raw[6];
    if (lane == 3) e = a.sp[1].ke * raw[13];
    a.acc[27 + lane] = e;
  }
  if (lane < kThrustRaw) a.raw[lane] = 0.0;
  if (lane == 0) *a.ticket = 0;
}

// Gauss-law residual r = div4(E) - q (ni - ne)/e0 at cell centres; acc gets
// [sum r^2, sum (rho/e0)^2, max |r| (as ordered bits), cells].
template <typename real>
__global__ void __launch_bounds__(256) gauss_kernel(Fields<real> F, Geom g, double inv24dx, double q_e0,
                                                    double* acc, unsigned long long* maxbits) {
  double s[3] = {0.0, 0.0, 0.0};
  double mx = 0.0;
  const int nint = g.nx * g.ny * g.nz;
  const int sx = g.sx, sy = g.gz;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nint; t += gridDim.x * blockDim.x) {
    const int m = 2 + t % g.nz, l = 2 + (t / g.nz) % g.ny, k = 2 + t / (g.nz * g.ny);
    const int n = k * sx + l * sy + m;
    const real* ex = F.f[F_EX];
    const real* ey = F.f[F_EY];
    const real* ez = F.f[F_EZ];
    const double dvx = 27.0 * ((double)ex[n + sx] - (double)ex[n]) - ((double)ex[n + 2 * sx] - (double)ex[n - sx]);
    const double dvy = 27.0 * ((double)ey[n + sy] - (double)ey[n]) - ((double)ey[n + 2 * sy] - (double)ey[n - sy]);
    const double dvz = 27.0 * ((double)ez[n + 1] - (double)ez[n]) - ((double)ez[n + 2] - (double)ez[n - 1]);
    const double div = (dvx + dvy + dvz) * inv24dx;
    const double rho = q_e0 * ((double)F.f[F_NI][n] - (double)F.f[F_NE][n]);
    const double r = div - rho;
    s[0] += r * r;
    s[1] += rho * rho;
    s[2] += 1.0;
    mx = fmax(mx, fabs(r));
  }
  const int idx[3] = {0, 1, 3};
  const double scale[3] = {1.0, 1.0, 1.0};
  block_reduce_add<3>(s, acc, idx, scale);
  // max: non-negative doubles order like their bit patterns
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_down_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) atomicMax(maxbits, (unsigned long long)__double_as_longlong(mx));
}

// Fave += F / 500 (thrust_fave :5265-5267).
__global__ void fave_accumulate_kernel(const double* __restrict__ acc, double* fave, double scale) {
  const int q = threadIdx.x;
  if (q < 27) fave[q] += acc[q] * scale;
}

}  // namespace pb
