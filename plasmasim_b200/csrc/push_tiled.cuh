// The fused particle kernel over the tiled layout of tiled.cuh.
#pragma once

#include "common.cuh"
#include "particles.cuh"
#include "tiled.cuh"

namespace pb {

// Particle rows in flight per warp (with 3 to 6 rows the FP32 push of 128^3 x 64
// took 7.04, 7.02, 7.09 and 7.08 ms per step, FP64 64^3 x 32 1.690, 1.692, 1.710, 1.728).
template <typename real>
constexpr int kStages = sizeof(real) == 4 ? 4 : 3;

// Cells [lo, lo + ext) of each axis.
struct CellRange {
  int lx, ly, lz;
  unsigned ex, ey, ez;
  __device__ __forceinline__ bool has(int i, int j, int k) const {
    return (unsigned)(i - lx) < ex && (unsigned)(j - ly) < ey && (unsigned)(k - lz) < ez;
  }
};

// Shared-memory plan of one CTA (8 warps): the density window; per warp a ring
// of kStages particle rows fetched ahead with cp.async (records A and B of each
// slot: 8 reals), whose memory takes the J window after the last row; the
// tile's E and B over the window, where the gather reads them; per warp a queue
// of kQ off-home J deposits, 7 words each (cell, offsets, velocities), made 32
// at a time by the whole warp (1.7 % off the FP32 step against each particle
// depositing where it is found), and the slots left to the general path.
template <typename real>
struct PushSmem {
  static constexpr int WX = kTileX + 4, WY = kTileY + 4, WZ = kWinZ, WN = WX * WY * WZ;
  static constexpr int kWarps = kTileX * kTileY;
  static constexpr int kQ = 2 * kLanes;
  static constexpr int kRest = 8 * kLanes;
  static constexpr size_t ring_off = (WN * sizeof(real) + 15) & ~(size_t)15;
  static constexpr size_t ring_bytes = (size_t)kWarps * kStages<real> * kLanes * 8 * sizeof(real);
  static_assert(ring_bytes >= 3 * WN * sizeof(real), "the ring holds the J window");
  static constexpr size_t fwin_off = ring_off + ring_bytes;
  static constexpr size_t jq_off = fwin_off + (size_t)6 * WN * sizeof(real);
  static constexpr size_t slow_off = jq_off + (size_t)kWarps * kQ * 7 * sizeof(real);
  static constexpr size_t bytes = slow_off + (size_t)kWarps * kRest * sizeof(int);
};

// Trilinear interpolation from a window plane with compile-time strides (the
// 2x2x2 nodes from w on), the two x planes as one packed pair.
template <int WY, int WZ>
__device__ __forceinline__ float trilerp_win(const float* __restrict__ w, float x0, float x1, float2 Y0, float2 Y1,
                                             float2 Z0, float2 Z1) {
  constexpr int P = WY * WZ;  // next x plane
  const float2 n00 = make_float2(w[0], w[P]), n01 = make_float2(w[1], w[P + 1]);
  const float2 n10 = make_float2(w[WZ], w[P + WZ]), n11 = make_float2(w[WZ + 1], w[P + WZ + 1]);
  const float2 cy0 = __ffma2_rn(n01, Z1, __fmul2_rn(n00, Z0));
  const float2 cy1 = __ffma2_rn(n11, Z1, __fmul2_rn(n10, Z0));
  const float2 cx = __ffma2_rn(cy1, Y1, __fmul2_rn(cy0, Y0));
  return cx.x * x0 + cx.y * x1;
}

template <int WY, int WZ>
__device__ __forceinline__ double trilerp_win(const double* __restrict__ w, double x0, double x1, double y0, double y1,
                                              double z0, double z1) {
  constexpr int P = WY * WZ;
  const double c00 = w[0] * z0 + w[1] * z1, c01 = w[WZ] * z0 + w[WZ + 1] * z1;
  const double c10 = w[P] * z0 + w[P + 1] * z1, c11 = w[P + WZ] * z0 + w[P + WZ + 1] * z1;
  return (c00 * y0 + c01 * y1) * x0 + (c10 * y0 + c11 * y1) * x1;
}

// Weights along one axis of a particle at offset f of an interior cell (so
// never cell 0, where axis_weights' half-shifted base is the cell itself), and
// the step from the cell's node to the half-shifted base (0 or -stride).
template <typename real>
struct WinAxis {
  real a0, a1, b0, b1;
  int s;
};
template <typename real>
__device__ __forceinline__ WinAxis<real> win_axis(real f, int stride) {
  WinAxis<real> w;
  const bool up = f >= (real)0.5;
  w.a1 = f;
  w.a0 = (real)1 - f;
  w.b1 = f + (up ? (real)-0.5 : (real)0.5);
  w.b0 = (real)1 - w.b1;
  w.s = up ? 0 : -stride;
  return w;
}

// gather6 from a window of one plane per component (ex ey ez bx by bz, WN
// nodes each) at node n, the particle's cell; its stencil lies inside.
template <int WY, int WZ, int WN>
__device__ __forceinline__ Gathered<float> gather6_win(const float* __restrict__ n, const WinAxis<float>& X,
                                                       const WinAxis<float>& Y, const WinAxis<float>& Z) {
  const float2 ya0 = make_float2(Y.a0, Y.a0), ya1 = make_float2(Y.a1, Y.a1);
  const float2 yb0 = make_float2(Y.b0, Y.b0), yb1 = make_float2(Y.b1, Y.b1);
  const float2 za0 = make_float2(Z.a0, Z.a0), za1 = make_float2(Z.a1, Z.a1);
  const float2 zb0 = make_float2(Z.b0, Z.b0), zb1 = make_float2(Z.b1, Z.b1);
  Gathered<float> r;
  r.ex = trilerp_win<WY, WZ>(n + Y.s + Z.s, X.a0, X.a1, yb0, yb1, zb0, zb1);
  r.ey = trilerp_win<WY, WZ>(n + WN + X.s + Z.s, X.b0, X.b1, ya0, ya1, zb0, zb1);
  r.ez = trilerp_win<WY, WZ>(n + 2 * WN + X.s + Y.s, X.b0, X.b1, yb0, yb1, za0, za1);
  r.bx = trilerp_win<WY, WZ>(n + 3 * WN + X.s, X.b0, X.b1, ya0, ya1, za0, za1);
  r.by = trilerp_win<WY, WZ>(n + 4 * WN + Y.s, X.a0, X.a1, yb0, yb1, za0, za1);
  r.bz = trilerp_win<WY, WZ>(n + 5 * WN + Z.s, X.a0, X.a1, ya0, ya1, zb0, zb1);
  return r;
}
template <int WY, int WZ, int WN>
__device__ __forceinline__ Gathered<double> gather6_win(const double* __restrict__ n, const WinAxis<double>& X,
                                                        const WinAxis<double>& Y, const WinAxis<double>& Z) {
  Gathered<double> r;
  r.ex = trilerp_win<WY, WZ>(n + Y.s + Z.s, X.a0, X.a1, Y.b0, Y.b1, Z.b0, Z.b1);
  r.ey = trilerp_win<WY, WZ>(n + WN + X.s + Z.s, X.b0, X.b1, Y.a0, Y.a1, Z.b0, Z.b1);
  r.ez = trilerp_win<WY, WZ>(n + 2 * WN + X.s + Y.s, X.b0, X.b1, Y.b0, Y.b1, Z.a0, Z.a1);
  r.bx = trilerp_win<WY, WZ>(n + 3 * WN + X.s, X.b0, X.b1, Y.a0, Y.a1, Z.a0, Z.a1);
  r.by = trilerp_win<WY, WZ>(n + 4 * WN + Y.s, X.a0, X.a1, Y.b0, Y.b1, Z.a0, Z.a1);
  r.bz = trilerp_win<WY, WZ>(n + 5 * WN + Z.s, X.a0, X.a1, Y.a0, Y.a1, Z.b0, Z.b1);
  return r;
}

// The window's planes from F_EX .. F_BZ (16-byte loads where the row pitch
// allows; ordinary ones, which stay behind the wait for the launch before, U of
// them in flight together), zero outside the array. The compiler does not move
// an ordinary load ahead of the last one's store: with one in flight the push
// of both species took 0.298 ms per step at 64^3 x 16, 1.115 at 96 x 96 x 128 x
// 16, FP64 64^3 x 32 1.61, with four 0.292, 1.083 and 1.59. thrust_kernel, which
// holds its first records meanwhile, has registers for two (0.296 ms at 96 x 96
// x 128 x 16 against 0.314 with one and 0.321 with four).
template <typename real, int WX, int WY, int WZ, bool VEC, int U>
__device__ __forceinline__ void fill_win(real* __restrict__ fw, const Fields<real>& F, const Geom& g, int wx0, int wy0,
                                         int wz0) {
  constexpr int V = sizeof(real) == 4 ? 4 : 2, NZV = WZ / V, WN = WX * WY * WZ, N = 6 * WX * WY * NZV;
  for (int q0 = threadIdx.x; q0 < N; q0 += U * blockDim.x) {
    real v[U][V];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int q = q0 + u * blockDim.x;
      const int p = q / (WX * WY * NZV), r = q % (WX * WY * NZV);
      const int ga = wx0 + r / (WY * NZV), gb = wy0 + (r / NZV) % WY, gc = wz0 + V * (r % NZV);
#pragma unroll
      for (int e = 0; e < V; ++e) v[u][e] = (real)0;
      if (q < N && ga < g.gx && gb < g.gy) {
        const real* src = F.f[p] + (long long)ga * g.sx + gb * g.gz + gc;
        if (VEC && gc + V - 1 < g.gz) {
          if constexpr (V == 4) {
            const float4 f4 = *reinterpret_cast<const float4*>(src);
            v[u][0] = f4.x; v[u][1] = f4.y; v[u][2] = f4.z; v[u][3] = f4.w;
          } else {
            const double2 f2 = *reinterpret_cast<const double2*>(src);
            v[u][0] = f2.x; v[u][1] = f2.y;
          }
        } else {
#pragma unroll
          for (int e = 0; e < V; ++e)
            if (gc + e < g.gz) v[u][e] = src[e];
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int q = q0 + u * blockDim.x;
      if (q >= N) break;
      const int p = q / (WX * WY * NZV), r = q % (WX * WY * NZV);
      real* dst = fw + p * WN + r / NZV * WZ + V * (r % NZV);
      if constexpr (V == 4) *reinterpret_cast<float4*>(dst) = make_float4(v[u][0], v[u][1], v[u][2], v[u][3]);
      else *reinterpret_cast<double2*>(dst) = make_double2(v[u][0], v[u][1]);
    }
  }
}

// The current of the particles that are in a lane's home cell, summed in
// registers over the 2x3x3 / 3x2x3 / 3x3x2 nodes such a particle can touch:
// x(a, b, c) is the jx sum at node (h-1+a+1, h-1+b, h-1+c) of the window flush
// below, and so on for y and z.
template <typename real>
struct HomeJ {
  real jx[2][3][3], jy[3][2][3], jz[3][3][2];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          if (a < 2) jx[a][b][c] = (real)0;
          if (b < 2) jy[a][b][c] = (real)0;
          if (c < 2) jz[a][b][c] = (real)0;
        }
  }
  // the current (qx, qy, qz) of a particle at the offsets (fx, fy, fz)
  __device__ __forceinline__ void add(real qx, real qy, real qz, real fx, real fy, real fz, const W3<real>& bx,
                                      const W3<real>& by, const W3<real>& bz) {
    const real ax[2] = {(real)1 - fx, fx}, ay[2] = {(real)1 - fy, fy}, az[2] = {(real)1 - fz, fz};
#pragma unroll
    for (int b = 0; b < 3; ++b)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const real yz = by.w[b] * bz.w[c];
        jx[0][b][c] += (qx * ax[0]) * yz;
        jx[1][b][c] += (qx * ax[1]) * yz;
      }
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const real xz = bx.w[a] * bz.w[c];
        jy[a][0][c] += (qy * ay[0]) * xz;
        jy[a][1][c] += (qy * ay[1]) * xz;
      }
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        const real xy = bx.w[a] * by.w[b];
        jz[a][b][0] += (qz * az[0]) * xy;
        jz[a][b][1] += (qz * az[1]) * xy;
      }
  }
  template <typename F>
  __device__ __forceinline__ void each(F f) {
#pragma unroll
    for (int q = 0; q < 18; ++q) {
      f(jx[q / 9][q / 3 % 3][q % 3]);
      f(jy[q / 6][q / 3 % 2][q % 3]);
      f(jz[q / 6][q / 2 % 3][q % 2]);
    }
  }
  __device__ __forceinline__ real x(int a, int b, int c) const { return jx[a][b][c]; }
  __device__ __forceinline__ real y(int a, int b, int c) const { return jy[a][b][c]; }
  __device__ __forceinline__ real z(int a, int b, int c) const { return jz[a][b][c]; }
};

// The sums of the lanes that share a cell (lane z of the first nv and z + nv,
// z + 2 nv, ...) into the first of them: `each` calls its argument on every sum.
template <typename J>
__device__ __forceinline__ void merge_lanes(J& acc, int nv, int lane) {
  for (int from = lane + nv, end = kLanes; nv < end; end -= nv, from += nv) {
    const bool take = lane < nv && from < kLanes;
    acc.each([&](auto& v) {
      const auto o = __shfl_sync(0xffffffffu, v, from & (kLanes - 1));
      if (take) v += o;
    });
  }
}

// FP32: the two nodes of each component's unshifted axis as one packed pair,
// updated with the two-wide multiplies and FMAs of sm_100.
template <>
struct HomeJ<float> {
  float2 jx[3][3], jy[3][3], jz[3][3];  // jx[b][c] = (a = 0, a = 1); jy[a][c] = (b = 0, 1); jz[a][b] = (c = 0, 1)
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b) jx[a][b] = jy[a][b] = jz[a][b] = make_float2(0.f, 0.f);
  }
  __device__ __forceinline__ void add(float qx, float qy, float qz, float fx, float fy, float fz, const W3<float>& bx,
                                      const W3<float>& by, const W3<float>& bz) {
    const float2 qxa = __fmul2_rn(make_float2(qx, qx), make_float2(1.f - fx, fx));
    const float2 qya = __fmul2_rn(make_float2(qy, qy), make_float2(1.f - fy, fy));
    const float2 qza = __fmul2_rn(make_float2(qz, qz), make_float2(1.f - fz, fz));
    float2 dx[3], dy[3], dz[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      dx[q] = make_float2(bx.w[q], bx.w[q]);
      dy[q] = make_float2(by.w[q], by.w[q]);
      dz[q] = make_float2(bz.w[q], bz.w[q]);
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const float2 tx = __fmul2_rn(qxa, dy[q]);  // jx: b = q
      const float2 ty = __fmul2_rn(qya, dx[q]);  // jy: a = q
      const float2 tz = __fmul2_rn(qza, dx[q]);  // jz: a = q
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        jx[q][r] = __ffma2_rn(tx, dz[r], jx[q][r]);  // c = r
        jy[q][r] = __ffma2_rn(ty, dz[r], jy[q][r]);  // c = r
        jz[q][r] = __ffma2_rn(tz, dy[r], jz[q][r]);  // b = r
      }
    }
  }
  template <typename F>
  __device__ __forceinline__ void each(F f) {
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        f(jx[q][r].x);
        f(jx[q][r].y);
        f(jy[q][r].x);
        f(jy[q][r].y);
        f(jz[q][r].x);
        f(jz[q][r].y);
      }
  }
  __device__ __forceinline__ float x(int a, int b, int c) const { return a ? jx[b][c].y : jx[b][c].x; }
  __device__ __forceinline__ float y(int a, int b, int c) const { return b ? jy[a][c].y : jy[a][c].x; }
  __device__ __forceinline__ float z(int a, int b, int c) const { return c ? jz[a][b].y : jz[a][b].x; }
};

__device__ __forceinline__ void cp_async_16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(s), "l"(gmem) : "memory");
}

// Records A and B of particle t into 4 reals of shared memory each (16-byte copies).
template <typename real>
__device__ __forceinline__ void fetch_records(real* dst_a, real* dst_b, const Parts<real>& P, long long t) {
  constexpr int kPieces = 4 * (int)sizeof(real) / 16;  // 16-byte pieces per record
  const char* a = reinterpret_cast<const char*>(P.ra + 4 * t);
  const char* b = reinterpret_cast<const char*>(P.rb + 4 * t);
#pragma unroll
  for (int q = 0; q < kPieces; ++q) {
    cp_async_16(reinterpret_cast<char*>(dst_a) + 16 * q, a + 16 * q);
    cp_async_16(reinterpret_cast<char*>(dst_b) + 16 * q, b + 16 * q);
  }
}

// Four reals of one record from shared memory, as vector loads.
__device__ __forceinline__ void read_record(const float* p, float (&r)[4]) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  r[0] = v.x; r[1] = v.y; r[2] = v.z; r[3] = v.w;
}
__device__ __forceinline__ void read_record(const double* p, double (&r)[4]) {
  const double2 v0 = reinterpret_cast<const double2*>(p)[0], v1 = reinterpret_cast<const double2*>(p)[1];
  r[0] = v0.x; r[1] = v0.y; r[2] = v1.x; r[3] = v1.y;
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" :: "n"(N) : "memory"); }

// Moves a packed cell and its offset by less than a cell per axis: adds the
// displacement d to f and steps the cell by `unit` (the axis's field of
// pack_cell) where f leaves [0, 1). unit_fix sees to what that leaves outside:
// a sum rounded to 1, -0, NaN, and longer moves.
template <typename real>
__device__ __forceinline__ void step_axis(int& c, real& f, real d, int unit) {
  real t = f + d;
  if (t >= (real)1) {
    t -= (real)1;
    c += unit;
  }
  if (t < (real)0) {
    t += (real)1;
    c -= unit;
  }
  f = t;
}
template <typename real>
__device__ __forceinline__ void unit_fix(int& c, real& t, int unit) {
  if (!off_unit(t)) return;
  const real fl = floor(t);
  c += (int)fl * unit;
  t -= fl;
  if (t >= (real)1) {
    t = (real)0;
    c += unit;
  }
}
constexpr int kUnitX = 1 << (2 * kCellBits), kUnitY = 1 << kCellBits, kUnitZ = 1;
template <typename real>
__device__ __forceinline__ void step_cell(int& c, real& fx, real& fy, real& fz, real dx, real dy, real dz) {
  step_axis(c, fx, dx, kUnitX);
  step_axis(c, fy, dy, kUnitY);
  step_axis(c, fz, dz, kUnitZ);
}

// The scale of a tile's density window (add_density): FP32 sums fixed-point
// weights at a scale that no node of a tile of `slots` rows can overflow, below
// 2^23 as well, where the rounding by an added 2^23 is exact.
__device__ __forceinline__ double window_scale(double weight, int) { return weight; }
__device__ __forceinline__ float window_scale(float, int slots) {
  return fminf(4294967295.f / (float)(slots * kLanes + 1), 8388607.f);
}
// Four consecutive nodes of the window as densities.
template <typename real>
struct Four {
  real v[4];
};
__device__ __forceinline__ Four<double> window_density(const double* s, double, double) {
  return Four<double>{{s[0], s[1], s[2], s[3]}};
}
__device__ __forceinline__ Four<float> window_density(const float* s, float weight, float scale) {
  // in FP64: an FP32 weight / scale would be off by the same few parts in 1e8
  // for all nodes of the tile, which a Poisson step sees as a charge (median
  // error of F against FP64 over 12 seeds at 96^3 x 8 with cleaning: 8.7e-7,
  // this way 7.2e-7)
  const unsigned* u = reinterpret_cast<const unsigned*>(s);
  const double back = (double)weight / (double)scale;
  return Four<float>{{(float)(u[0] * back), (float)(u[1] * back), (float)(u[2] * back), (float)(u[3] * back)}};
}
// Adds them to a plane: one reduction where the rows allow, `left` nodes to the row's end.
template <bool VEC, typename real>
__device__ __forceinline__ void flush_nodes(real* dst, int left, const Four<real>& f) {
  if (f.v[0] == (real)0 && f.v[1] == (real)0 && f.v[2] == (real)0 && f.v[3] == (real)0) return;
  if constexpr (VEC && sizeof(real) == 4) {
    red_add_v4(dst, f.v[0], f.v[1], f.v[2], f.v[3]);
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (e < left && f.v[e] != (real)0) atomicAdd(dst + e, f.v[e]);
  }
}

// Record B's fourth word after the main loop: what is left to do for the
// particle (0 nothing, kLeftAll the whole push, kLeftEnd the density deposit
// and sr_particle).
constexpr int kLeftAll = 1, kLeftEnd = 2;
template <typename real>
__device__ __forceinline__ int left_of(const Parts<real>& P, int t) { return (int)P.rb[4 * (long long)t + 3]; }

// One species' part of a launch over the tiles: its store, with ntail CTAs for
// the slots from `tail` to *count, and a CTA for each tile.
template <typename real>
struct TileJob {
  Parts<real> P;
  PushConst<real> pc;
  const int* goff;  // first slot of each group
  const int* gtop;  // rows of each group up to the last one that holds a particle
  int ntail, tail;
  const int* count;
};
// The launch: job 0 in the first `split` CTAs, job 1 in the others.
template <typename real>
struct TileJobs {
  TileJob<real> job[2];
  int split;
  TileGeom t;
};

// The slots after the layout (particles without a hole in their group): the
// slot-order push, in a job's first blocks.
template <typename real, int MODE>
__device__ __noinline__ void push_tail(const TileJob<real>& job, int block, const Fields<real>& F, const Geom& g,
                                       unsigned long long* err) {
  push_slots<real, MODE>(job.P, job.tail + block * blockDim.x + threadIdx.x, job.ntail * blockDim.x, *job.count, F, g,
                         job.pc, err);
}

// What the main loop left of particle t to the general path.
template <typename real, int MODE>
__device__ __noinline__ void push_rest(const Parts<real>& P, int t, const Fields<real>& F, const Geom& g,
                                       const PushConst<real>& pc, unsigned long long* err) {
  const Rec<real> r = load_records(P, t);
  const int left = left_of(P, t);
  if (r.cell < 0 || left == 0) return;
  if (MODE == PUSH_J || left == kLeftAll) {
    push_one<real, MODE>(P, t, r, F, g, pc, err);
    return;
  }
  int i, j, k;
  unpack_cell(r.cell, i, j, k);
  if (in_array(g, i, j, k)) {
    if (stencil_ok(g, i, j, k))
      deposit_n(F, g, pc, axis_weights(i, r.o[0]), axis_weights(j, r.o[1]), axis_weights(k, r.o[2]));
    else
      count_err(err, ERR_DEPOSIT_OOB);
  }
  const int c = settle(g, pc.out, i, j, k, r.o[0], r.o[1], r.o[2], r.v[0], r.v[1], r.v[2], err);
  store_records(P, t, c, r.o[0], r.o[1], r.o[2], r.v[0], r.v[1], r.v[2]);
}

// The fused particle part of one step (push, J deposit at x^{n+1/2}, drift,
// n deposit at x^{n+1}, sr_particle), or with MODE = PUSH_J its first two
// parts, for one species over the tiled layout; the same arithmetic as
// push_kernel apart from the order of the sums and, in the FP32 fused push
// alone, the square roots and divisions and the fixed-point sums of the
// density window. One CTA per tile, one warp per group; a job's first ntail CTAs take
// the slots after the layout (a launch of their own, 7 to 12 us per species for
// next to no particles, before).
//
// Both species go in one launch, the second's CTAs after the first's, so that
// the first's last wave leaves no SM idle: push per step 0.044 ms at 32^3 x 8,
// 0.300 at 64^3 x 16, 0.164 at 41 x 22 x 70 x 30, 6.53 at 128^3 x 64, against
// 0.053, 0.311, 0.183 and 6.55 with a launch each, the second free to start
// while the first ran. (The constants that the species share are taken from
// the first's, so that they are operands at fixed addresses: 6.61 at 128^3 x 64
// with all of them read through the CTA's own species; the kernel's body once
// per species, 6.73.)
//
// J of a particle in its lane's home cell at x^{n+1/2} is summed in registers;
// the others add theirs to global memory with reductions (a shared J window
// taking every particle's 24 weights by FP32 shared atomics, which frees the
// registers for 3 CTAs per SM, measured 1.7x slower). The density goes to the
// window with shared reductions (every active lane at once): integer ones on
// fixed-point sums in FP32, FP64 atomics in FP64.
//
// Bound by instruction issue (16 warps per SM, 65 % of the slots issue; DRAM at
// 29 %), so the loop is written for few instructions: cells stay packed while
// they move (step_cell), one range test says that a particle needs no bounds
// checks, window addresses come from one multiply-add chain and the lanes
// without a particle run along with zero currents instead of branching. What
// the test refuses -- a particle wrapped to the other side of the domain, or
// more than a cell outside its tile -- goes to push_rest after the loop.
// Against the checks and branches per particle that this replaces, push per
// step of both species: 7.06 -> 6.55 ms at 128^3 x 64, 0.327 -> 0.309 at
// 64^3 x 16, 0.203 -> 0.183 at 41 x 22 x 70 x 30 (sides that no tile divides),
// FP64 64^3 x 32 1.72 -> 1.61. Rows loaded into registers one ahead, without
// the ring: 7.7 ms at 128^3 x 64.
// FP64 runs one CTA per SM: 254 registers and no spills, against 528 bytes of
// spill stores per thread at two (128 registers); 27.2 against 30.6 ms per step
// at 128^3 x 64. That leaves room for the field window and the J queue.
#ifndef PB_PUSH64_MIN_BLOCKS
#define PB_PUSH64_MIN_BLOCKS 1
#endif
template <typename real, bool VEC, int MODE>
__global__ void __launch_bounds__(kTileX * kTileY * 32, sizeof(real) == 4 ? 2 : PB_PUSH64_MIN_BLOCKS)
push_tiled_kernel(const __grid_constant__ TileJobs<real> jobs, const __grid_constant__ Fields<real> F,
                  const __grid_constant__ Geom g, unsigned long long* err) {
  after_prior();
  const int second = (int)blockIdx.x >= jobs.split, block = (int)blockIdx.x - (second ? jobs.split : 0);
  const TileJob<real>& job = jobs.job[second];
  const Parts<real>& P = job.P;
  // the species differ in these alone; the others stay immediate operands
  PushConst<real> pc = jobs.job[0].pc;
  pc.T = job.pc.T;
  pc.pjx = job.pc.pjx;
  pc.pjy = job.pc.pjy;
  pc.pjz = job.pc.pjz;
  pc.pn = job.pc.pn;
  pc.out = job.pc.out;
  if (block < job.ntail) {
    push_tail<real, MODE>(job, block, F, g, err);
    return;
  }
  using S = PushSmem<real>;
  constexpr int WY = S::WY, WZ = S::WZ, WN = S::WN, WX = S::WX, NS = kStages<real>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  real* wn = reinterpret_cast<real*>(smem_raw);                // [WN]: n
  real* wj = reinterpret_cast<real*>(smem_raw + S::ring_off);  // [3][WN]: jx, jy, jz, after the last row
  real* fw = reinterpret_cast<real*>(smem_raw + S::fwin_off);  // [6][WN]: E, B
  const int tile = block - job.ntail;
  const TileGeom& t = jobs.t;
  const int tz = tile % t.ntz, ty = (tile / t.ntz) % t.nty, tx = tile / (t.ntz * t.nty);
  // window origin: two nodes below the tile's first interior cell (2 + tx*TX)
  const int wx0 = tx * kTileX, wy0 = ty * kTileY, wz0 = tz * kLanes;
  for (int q = threadIdx.x; q < WN; q += blockDim.x) wn[q] = (real)0;
  fill_win<real, WX, WY, WZ, VEC, 4>(fw, F, g, wx0, wy0, wz0);
  __syncthreads();
  // the interior cells whose stencils lie in the window: a particle in one
  // needs no check of the array's bounds and none of sr_particle's
  CellRange near;
  near.lx = max(wx0 + 1, 2);
  near.ly = max(wy0 + 1, 2);
  near.lz = max(wz0 + 1, 2);
  near.ex = (unsigned)(min(wx0 + WX - 1, g.nx + 2) - near.lx);
  near.ey = (unsigned)(min(wy0 + WY - 1, g.ny + 2) - near.ly);
  near.ez = (unsigned)(min(wz0 + WZ - 1, g.nz + 2) - near.lz);
  if (pc.long_moves) near.ex = 0;  // nobody takes the short path
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = tile * (kTileX * kTileY) + warp;
  const int base = job.goff[G], jmax = job.gtop[G];
  // home cell of this lane
  const int hi = wx0 + 2 + warp / kTileY, hj = wy0 + 2 + warp % kTileY;
  const int nv = tile_cells(g, tz), hk = wz0 + 2 + lane_cell(nv, lane).z;
  const int hcell = pack_cell(hi, hj, hk);
  const int wcell0 = (wx0 * WY + wy0) * WZ + wz0;  // window node of a cell: (i WY + j) WZ + k less this
  int slots = 0;
#pragma unroll
  for (int w = 0; w < kTileX * kTileY; ++w) slots += job.gtop[tile * (kTileX * kTileY) + w];
  const real nscale = window_scale(pc.nw, slots);
  HomeJ<real> acc;
  acc.zero();
  // the warp's queue of J deposits off the home cells: entries [0, nq), 7
  // words each (7 is odd, so the lanes' entries fall on different banks).
  // They go to the planes with global reductions (into the shared J window by
  // FP32 shared atomics, where the stencil allowed, measured 0.7 ms per step
  // slower; z-adjacent pairs as 16-byte vector reductions, 0.2 ms slower)
  real* jq = reinterpret_cast<real*>(smem_raw + S::jq_off) + warp * S::kQ * 7;
  int nq = 0;
  auto deposit_queued = [&](int q) {
    const real* e = jq + q * 7;
    int qi, qj, qk;
    unpack_cell(word_int(e[0]), qi, qj, qk);
    const Axis<real> X = axis_weights(qi, e[1]), Y = axis_weights(qj, e[2]), Z = axis_weights(qk, e[3]);
    deposit_j(F, g, pc, X, Y, Z, e[4], e[5], e[6]);
  };
  // slots left to push_rest: the first kRest of them in a list
  int* rest = reinterpret_cast<int*>(smem_raw + S::slow_off) + warp * S::kRest;
  int nrest = 0;
  // ring of particle rows fetched ahead; each lane copies and reads only its
  // own slots, so the per-thread cp.async groups need no warp barrier. A
  // stage holds the row's 32 records A, then its 32 records B, so that the
  // lanes' 16-byte reads of one record fall on consecutive banks.
  real* ring = reinterpret_cast<real*>(smem_raw + S::ring_off) + warp * NS * kLanes * 8;
  auto fetch = [&](int row) {
    if (row < jmax) {
      real* stage = ring + (row % NS) * kLanes * 8;
      fetch_records(stage + lane * 4, stage + (kLanes + lane) * 4, P, base + row * kLanes + lane);
    }
    cp_async_commit();
  };
#pragma unroll
  for (int s = 0; s < NS - 1; ++s) fetch(s);
  unsigned pushed = 0, nbad = 0;
  for (int jj = 0; jj < jmax; ++jj) {
    fetch(jj + NS - 1);
    cp_async_wait<NS - 1>();
    const int slot = base + jj * kLanes + lane;
    const real* stage = ring + (jj % NS) * kLanes * 8;
    real ra[4], rb[4];
    read_record(stage + lane * 4, ra);
    read_record(stage + (kLanes + lane) * 4, rb);
    int c = word_int(ra[0]);
    real fx = ra[1], fy = ra[2], fz = ra[3];
    real vx = rb[0], vy = rb[1], vz = rb[2];
    pushed += c >= 0;
    int i, j, k;
    unpack_cell(c, i, j, k);
    bool quick = near.has(i, j, k);  // never for an empty slot
    bool push = quick;
    if (pc.bal_interior && quick && ballistic(pc, i, j, k, fx, fy, fz)) {
      push = false;
      // a velocity that Boris has not bounded by c
      quick = fabs(vx * pc.hdt) < (real)1 && fabs(vy * pc.hdt) < (real)1 && fabs(vz * pc.hdt) < (real)1;
    }
    int left = c >= 0 && !quick ? kLeftAll : 0;
    if (push) {
      const WinAxis<real> X = win_axis(fx, WY * WZ), Y = win_axis(fy, WZ), Z = win_axis(fz, 1);
      const real* n = fw + ((i * WY + j) * WZ + k - wcell0);
      const Gathered<real> eb = gather6_win<WY, WZ, WN>(n, X, Y, Z);
      if (MODE == PUSH_J) boris4(pc, eb, vx, vy, vz);
      else boris4_fast(pc, eb, vx, vy, vz);
      // one test for the three: |v| < c, so the sum of finite components is finite
      nbad += !isfinite(vx + vy + vz);
    }
    // From here to the density every lane runs, with no branch: a lane without
    // a particle, or whose particle is off its home cell, adds zero currents
    // at offsets of 1/2. Its own may be anything, and 0 times a NaN would stay
    // in the sums: an empty slot's record holds what its last particle or the
    // memory's last owner left there.
    const real dx = vx * pc.hdt, dy = vy * pc.hdt, dz = vz * pc.hdt;
    // an offset rounded to 1 or -0 deposits the same current as in the cell it
    // belongs to; the second half step puts it there
    step_cell(c, fx, fy, fz, dx, dy, dz);
    const bool home = quick && c == hcell;
    {
      const real hx = home ? fx : (real)0.5, hy = home ? fy : (real)0.5, hz = home ? fz : (real)0.5;
      const W3<real> bx = home3(hx), by = home3(hy), bz = home3(hz);
      acc.add(home ? pc.qn * vx : (real)0, home ? pc.qn * vy : (real)0, home ? pc.qn * vz : (real)0, hx, hy, hz, bx, by,
              bz);
    }
    // the others' currents go to the warp's queue: the row's queued lanes take
    // consecutive entries; a full warp's worth is deposited by all 32 lanes at
    // once (less than a cell from the interior, their stencils lie in the array)
    const bool enq = quick && !home;
    const unsigned em = __ballot_sync(0xffffffffu, enq);
    if (em) {
      if (enq) {
        real* e = jq + (nq + __popc(em & ((1u << lane) - 1u))) * 7;
        e[0] = int_word<real>(c);
        e[1] = fx; e[2] = fy; e[3] = fz;
        e[4] = vx; e[5] = vy; e[6] = vz;
      }
      nq += __popc(em);
      if (nq >= kLanes) {
        __syncwarp();
        deposit_queued(nq - kLanes + lane);
        nq -= kLanes;
        __syncwarp();
      }
    }
    if (MODE == PUSH_FUSED) step_cell(c, fx, fy, fz, dx, dy, dz);
    if (quick) {
      if (off_unit(fx) || off_unit(fy) || off_unit(fz)) {
        unit_fix(c, fx, kUnitX);
        unit_fix(c, fy, kUnitY);
        unit_fix(c, fz, kUnitZ);
      }
      unpack_cell(c, i, j, k);
      int cnew = c;
      bool dep = MODE == PUSH_FUSED && near.has(i, j, k);
      if (MODE == PUSH_FUSED && !dep) {
        // past the interior (sr_particle's business), or out of the window too
        dep = (unsigned)(i - wx0 - 1) < WX - 2 && (unsigned)(j - wy0 - 1) < WY - 2 && (unsigned)(k - wz0 - 1) < WZ - 2 &&
              stencil_ok(g, i, j, k);
        if (dep) cnew = settle(g, pc.out, i, j, k, fx, fy, fz, vx, vy, vz, err);
        else left = kLeftEnd;
      }
      if (dep) {  // n at x^{n+1}
        const int w = ((c >> (2 * kCellBits)) * WY + ((c >> kCellBits) & kCellMask)) * WZ + (c & kCellMask) - wcell0;
        const WinAxis<real> X = win_axis(fx, WY * WZ), Y = win_axis(fy, WZ), Z = win_axis(fz, 1);
        add_density<WY, WZ>(wn + w + X.s + Y.s + Z.s, nscale, X, Y, Z);
      }
      store_records(P, slot, cnew, fx, fy, fz, vx, vy, vz, (real)left);
    } else if (left) {
      P.rb[4 * (long long)slot + 3] = (real)kLeftAll;
    }
    const unsigned lm = __ballot_sync(0xffffffffu, left != 0);
    if (lm) {
      const int q = nrest + __popc(lm & ((1u << lane) - 1u));
      if (left && q < S::kRest) rest[q] = slot;
      nrest += __popc(lm);
    }
  }
  if (nbad) atomicAdd(err + ERR_NONFINITE, (unsigned long long)nbad);
  __syncwarp();
  if (lane < nq) deposit_queued(lane);
  for (int o = 16; o > 0; o >>= 1) pushed += __shfl_down_sync(0xffffffffu, pushed, o);
  if (lane == 0 && pushed) atomicAdd(err + CNT_PUSHED, (unsigned long long)pushed);
  // what the loop left: the list (particles that have crossed the periodic
  // faces of x and y since the last re-layout, mostly), or every row when the
  // list overflowed
  if (nrest > S::kRest) {
    for (int jj = 0; jj < jmax; ++jj) push_rest<real, MODE>(P, base + jj * kLanes + lane, F, g, job.pc, err);
  } else {
    for (int q = lane; q < nrest; q += kLanes) push_rest<real, MODE>(P, rest[q], F, g, job.pc, err);
  }
  // the lane's home-cell sums into the window (nodes h-1 .. h+1 around it)
  cp_async_wait<0>();
  __syncthreads();
  for (int q = threadIdx.x; q < 3 * WN; q += blockDim.x) wj[q] = (real)0;
  __syncthreads();
  if (nv < kLanes) merge_lanes(acc, nv, lane);
  if (jmax > 0 && lane < nv) {
    const int la = hi - 1 - wx0, lb = hj - 1 - wy0, lc = hk - 1 - wz0;  // window index of node h-1
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b)
#pragma unroll
        for (int cc = 0; cc < 3; ++cc) {
          const int s = ((la + a) * WY + (lb + b)) * WZ + (lc + cc);
          if (a < 2) atomicAdd(wj + s + WY * WZ, acc.x(a, b, cc));       // x nodes h, h+1
          if (b < 2) atomicAdd(wj + WN + s + WZ, acc.y(a, b, cc));       // y nodes h, h+1
          if (cc < 2) atomicAdd(wj + 2 * WN + s + 1, acc.z(a, b, cc));   // z nodes h, h+1
        }
  }
  __syncthreads();
  // flush the window: one reduction per 4 consecutive z nodes
  const int planes[4] = {pc.pjx, pc.pjy, pc.pjz, pc.pn};
  constexpr int NZ4 = WZ / 4;
  for (int q4 = threadIdx.x; q4 < (MODE == PUSH_FUSED ? 4 : 3) * WX * WY * NZ4; q4 += blockDim.x) {
    const int q = q4 / (WX * WY * NZ4);
    const int r = q4 % (WX * WY * NZ4);
    const int a = r / (WY * NZ4), b = (r / NZ4) % WY, c4 = r % NZ4;
    const int ga = wx0 + a, gb = wy0 + b, gc = wz0 + 4 * c4;
    if (ga >= g.gx || gb >= g.gy || gc >= g.gz) continue;
    Four<real> v;
    if (q == 3) {
      v = window_density(wn + (a * WY + b) * WZ + 4 * c4, pc.nw, nscale);
    } else {
      const real* src = wj + q * WN + (a * WY + b) * WZ + 4 * c4;
      v = Four<real>{{src[0], src[1], src[2], src[3]}};
    }
    flush_nodes<VEC>(F.f[planes[q]] + ga * g.sx + gb * g.gz + gc, g.gz - gc, v);
  }
}

// The density of the particles that are in a lane's home cell, summed in
// registers over the 3x3x3 nodes around it.
template <typename real>
struct HomeN {
  real n[3][3][3];
  template <typename F>
  __device__ __forceinline__ void each(F f) {
#pragma unroll
    for (int q = 0; q < 27; ++q) f(n[q / 9][q / 3 % 3][q % 3]);
  }
  __device__ __forceinline__ void zero() {
    each([](real& v) { v = (real)0; });
  }
  __device__ __forceinline__ void add(real w, const W3<real>& bx, const W3<real>& by, const W3<real>& bz) {
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        const real xy = (w * bx.w[a]) * by.w[b];
#pragma unroll
        for (int c = 0; c < 3; ++c) n[a][b][c] += xy * bz.w[c];
      }
  }
};

// The drift loop of fdtd (:818-867) over the tiled layout: each particle to
// x^{n+1} and its density, of a particle in its lane's home cell there summed in
// registers and added to the plane once per lane, of any other through the
// warp's queue, 32 at a time. The sums are of the particles' own type, as in
// slot order: in the fused push's fixed-point window a sparse cell beside a
// crowded one of its tile loses bits. One CTA per tile, one warp per group, the
// next U rows' records on their way; a job's first ntail CTAs take the slots
// after the layout.
//
// Bound by DRAM when the grid is large (128^3 x 64: 48 bytes a particle in 2.20
// ms for both species, 89 % of the copy rate), by the records' latency when it
// is small (58 us at 48^3 x 16). With the fixed-point window 1.95 ms and 47 us,
// with a thread per slot and atomics on the plane 9.67 ms and 192 us; FP64 64^3 x
// 32, where the window took FP64 shared atomics: 0.477 -> 0.300 ms. Warps per
// SM and U: 32 and 2; 24 and 2 or 4 took 2.48 and 2.25 ms, 32 and 1 or 3 2.56
// and 2.58, 40 and 1 2.77. The sums through a shared window: 2.30.
template <typename real>
__global__ void __launch_bounds__(kTileX * kTileY * 32, sizeof(real) == 4 ? 4 : 2)
drift_tiled_kernel(const __grid_constant__ TileJobs<real> jobs, const __grid_constant__ Fields<real> F,
                   const __grid_constant__ Geom g, unsigned long long* err) {
  after_prior();
  constexpr int kWarps = kTileX * kTileY, kQ = 2 * kLanes, U = 2;
  const int second = (int)blockIdx.x >= jobs.split, block = (int)blockIdx.x - (second ? jobs.split : 0);
  const TileJob<real>& job = jobs.job[second];
  const Parts<real>& P = job.P;
  const PushConst<real>& pc = job.pc;
  if (block < job.ntail) {
    drift_slots(P, job.tail + block * blockDim.x + threadIdx.x, job.ntail * blockDim.x, *job.count, F, g, pc, err);
    return;
  }
  // per warp, the densities off the home cells: cell and offsets (5 words, odd, for the banks)
  __shared__ real queue[kWarps][kQ * 5];
  const int tile = block - job.ntail;
  const TileGeom& t = jobs.t;
  const int tz = tile % t.ntz, ty = (tile / t.ntz) % t.nty, tx = tile / (t.ntz * t.nty);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = tile * kWarps + warp;
  const int base = job.goff[G] + lane, jmax = job.gtop[G];
  if (jmax == 0) return;
  const int hi = tx * kTileX + 2 + warp / kTileY, hj = ty * kTileY + 2 + warp % kTileY;
  const int nv = tile_cells(g, tz), hk = tz * kLanes + 2 + lane_cell(nv, lane).z;
  real* mine = queue[warp];
  int nq = 0;
  const auto deposit_queued = [&](int q) {
    const real* e = mine + q * 5;
    int i, j, k;
    unpack_cell(word_int(e[0]), i, j, k);
    deposit_n(F, g, pc, axis_weights(i, e[1]), axis_weights(j, e[2]), axis_weights(k, e[3]));
  };
  HomeN<real> acc;
  acc.zero();
  Rec<real> q[U];
  const auto fetch = [&](int r0) {
#pragma unroll
    for (int u = 0; u < U; ++u)
      q[u] = r0 + u < jmax ? load_records(P, base + (r0 + u) * kLanes)
                           : Rec<real>{-1, {(real)0, (real)0, (real)0}, {(real)0, (real)0, (real)0}};
  };
  fetch(0);
  for (int r0 = 0; r0 < jmax; r0 += U) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool act = q[u].cell >= 0;
      int i, j, k;
      unpack_cell(q[u].cell, i, j, k);
      real fx = q[u].o[0], fy = q[u].o[1], fz = q[u].o[2];
      if (act) {
        advance(i, fx, q[u].v[0] * pc.hdt);
        advance(j, fy, q[u].v[1] * pc.hdt);
        advance(k, fz, q[u].v[2] * pc.hdt);
        store_position(P, base + (r0 + u) * kLanes, repack(i, j, k, err), fx, fy, fz);
      }
      // a lane without a home particle adds zeros, at offsets of 1/2 whatever its own are
      const bool home = act && i == hi && j == hj && k == hk;
      acc.add(home ? pc.nw : (real)0, home3(home ? fx : (real)0.5), home3(home ? fy : (real)0.5),
              home3(home ? fz : (real)0.5));
      bool off = act && !home && in_array(g, i, j, k);
      if (off && !stencil_ok(g, i, j, k)) {
        count_err(err, ERR_DEPOSIT_OOB);
        off = false;
      }
      const unsigned em = __ballot_sync(0xffffffffu, off);
      if (off) {
        real* e = mine + (nq + __popc(em & ((1u << lane) - 1u))) * 5;
        e[0] = int_word<real>(pack_cell(i, j, k));
        e[1] = fx; e[2] = fy; e[3] = fz;
      }
      nq += __popc(em);
      if (nq >= kLanes) {
        __syncwarp();
        deposit_queued(nq - kLanes + lane);
        nq -= kLanes;
        __syncwarp();
      }
    }
    fetch(r0 + U);
  }
  __syncwarp();
  if (lane < nq) deposit_queued(lane);
  if (nv < kLanes) merge_lanes(acc, nv, lane);
  // node h + c - 1 of a lane is its neighbour's: one sum per node and column
  real* n = F.f[pc.pn] + (hi - 1) * g.sx + (hj - 1) * g.gz + hk;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const real below = __shfl_up_sync(0xffffffffu, acc.n[a][b][2], 1);
      const real above = __shfl_down_sync(0xffffffffu, acc.n[a][b][0], 1);
      real* p = n + a * g.sx + b * g.gz;
      if (lane >= nv) continue;
      atomicAdd(p, acc.n[a][b][1] + (lane > 0 ? below : (real)0) + (lane + 1 < nv ? above : (real)0));
      if (lane == 0) atomicAdd(p - 1, acc.n[a][b][0]);
      if (lane + 1 == nv) atomicAdd(p + 1, acc.n[a][b][2]);
    }
}

}  // namespace pb
