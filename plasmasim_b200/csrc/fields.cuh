// Field kernels: dipole B0 and damping profile (init_grid), the damped
// 4th-order B and E updates (renew_b4_2 / renew_e4_2), which also write the
// size-1 periodic ghost copies (sr_b / sr_e), and the fold of J and n
// (sr_current2).
//
// Each update is one thread per interior node, k (z) fastest so that a warp
// reads and writes 32 consecutive nodes of every plane it touches; the +-1/+-2
// neighbours along i and j come from L1/L2. HBM bound: per node a B half-step
// moves 12 words (E3 read, DB3 read, B0 3 read, DB3 + B3 written... see below)
// and an E step 15 words.
#pragma once

#include "common.cuh"

namespace pb {

// Damping ramp on the doubled sub-grid (init_grid, PIC/3d_pic458_domain.c:339-365);
// sigma = a (0.1 sqrt(x^4+y^4+z^4) + 0.01 sqrt(x^12+y^12+z^12)) (:366-367).
__device__ __forceinline__ double sigma_of(double a, double x, double y, double z) {
  if (x == 0.0 && y == 0.0 && z == 0.0) return 0.0;
  const double x2 = x * x, y2 = y * y, z2 = z * z;
  const double x4 = x2 * x2, y4 = y2 * y2, z4 = z2 * z2;
  return a * (0.1 * sqrt(x4 + y4 + z4) + 0.01 * sqrt(x4 * x4 * x4 + y4 * y4 * y4 + z4 * z4 * z4));
}

struct Ramps {
  const double* rx;  // 2*gx values
  const double* ry;
  const double* rz;
  double a;
};

// external_current7 (:4579-4634) at rank (0,0): analytic point dipole of
// moment I*pi*R^2 along (0, sin alpha, cos alpha), centred on node
// ((nx+4)/2, (ny+4)/2, (nz+4)/2), each component on its own stagger.
struct DipoleParams {
  double mu0, I, R, alpha, dx, cutoff, imfx, imfy, imfz;
};

template <typename real>
__global__ void init_fields_kernel(Fields<real> F, Geom g, DipoleParams d) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= g.nodes) return;
  const int k = n / g.sx, l = (n / g.gz) % g.gy, m = n % g.gz;
  const double Pi = 3.14159265358979323846;
  // k + myrank_x Grid_Nx - (PROCESS_Nx Grid_Nx + 4)/2 (:4588-4589)
  const int cx = (g.gnx + 4) / 2 - g.ox, cy = (g.gny + 4) / 2 - g.oy, cz = (g.nz + 4) / 2;
  double x = (double)(k - cx) * d.dx, y = (double)(l - cy) * d.dx, z = (double)(m - cz) * d.dx;
  double r = sqrt(x * x + y * y + z * z);
  double b0x = d.imfx, b0y = d.imfy, b0z = d.imfz;
  if (r < d.cutoff * d.dx) {
    const double mom = d.mu0 * d.I * Pi * d.R * d.R;
    const double sa = sin(d.alpha), ca = cos(d.alpha);
    x = ((double)(k - cx) + 0.5) * d.dx; y = (double)(l - cy) * d.dx; z = (double)(m - cz) * d.dx;
    r = sqrt(x * x + y * y + z * z);
    b0x = mom * (3. * x * y * sa + 3. * x * z * ca) / (4. * Pi * pow(r, 5.0)) + d.imfx;
    x = (double)(k - cx) * d.dx; y = ((double)(l - cy) + 0.5) * d.dx; z = (double)(m - cz) * d.dx;
    r = sqrt(x * x + y * y + z * z);
    b0y = mom * (3. * y * y * sa + 3. * y * z * ca - r * r * sa) / (4. * Pi * pow(r, 5.0)) + d.imfy;
    x = (double)(k - cx) * d.dx; y = (double)(l - cy) * d.dx; z = ((double)(m - cz) + 0.5) * d.dx;
    r = sqrt(x * x + y * y + z * z);
    b0z = mom * (3. * y * z * sa + 3. * z * z * ca - r * r * ca) / (4. * Pi * pow(r, 5.0)) + d.imfz;
  }
  F.f[F_B0X][n] = (real)b0x; F.f[F_B0Y][n] = (real)b0y; F.f[F_B0Z][n] = (real)b0z;
  F.f[F_BX][n] = (real)b0x; F.f[F_BY][n] = (real)b0y; F.f[F_BZ][n] = (real)b0z;
  F.f[F_DBX][n] = (real)0; F.f[F_DBY][n] = (real)0; F.f[F_DBZ][n] = (real)0;
  F.f[F_EX][n] = (real)0; F.f[F_EY][n] = (real)0; F.f[F_EZ][n] = (real)0;
#pragma unroll
  for (int q = F_JIX; q <= F_NE; ++q) F.f[q][n] = (real)0;
  F.f[F_PHI][n] = (real)0;  // :325
}

// Up to 8 planes processed by one ghost kernel.
template <typename real>
struct PlaneSet {
  real* p[8];
  int count;
};

// The periodic ghost copies of sr_b / sr_e at size 1 (x pass :1016-1101, then
// y pass :1103-1190 over every x): ghost layers 0, 1 take layers N, N+1 and
// ghosts N+2, N+3 take layers 2, 3. The layers 2, 3 and N, N+1 are disjoint
// (N >= 5), so an interior column (k, l) has at most one image in x, one in y
// and one in both; whoever updates a column writes its images as well, and no
// pass of its own is needed. (Two passes after each update, and two for the
// fold, each 4 us of launch and latency whatever the grid: with them and a
// clear of J and n the fields took 0.0637 ms per step at 32^3, 0.078 at 64^3
// and 0.190 at 128^3, now 0.0428, 0.0565 and 0.160.)
struct Images {
  int n;
  long long d[3];  // node offsets of the column's images
};
__device__ __forceinline__ int image_shift(int k, int N) { return k < 4 ? N : k >= N ? -N : 0; }
__device__ __forceinline__ Images images_of(const Geom& g, int k, int l) {
  const long long dx = (long long)image_shift(k, g.nx) * g.sx, dy = (long long)image_shift(l, g.ny) * g.gz;
  Images r;
  r.n = (dx != 0) + (dy != 0) + (dx != 0 && dy != 0);
  r.d[0] = dx != 0 ? dx : dy;
  r.d[1] = dy;
  r.d[2] = dx + dy;
  return r;
}
// Node n of plane a, just set to v, to its column's images.
template <typename real>
__device__ __forceinline__ void put_images(real* a, long long n, const Images& im, real v) {
  for (int q = 0; q < im.n; ++q) a[n + im.d[q]] = v;
}
// sr_b on the total field (:1016-1190): the ghost planes of B get the periodic
// images of B, while B0 keeps its own (non-periodic) dipole values, so the
// induced field there is B_image - B0_ghost, which the E update then sees.
template <typename real>
__device__ __forceinline__ void put_images_b(const Fields<real>& F, int c, long long n, const Images& im, real v) {
  for (int q = 0; q < im.n; ++q) {
    F.f[F_BX + c][n + im.d[q]] = v;
    F.f[F_DBX + c][n + im.d[q]] = v - F.f[F_B0X + c][n + im.d[q]];
  }
}
// The copies cover every z, the two ghost nodes at either end too: the updates
// leave those nodes of the interior columns alone, and the thread of the first
// (last) interior node of a column hands them on.
template <typename real>
__device__ __forceinline__ void z_end_images(const Fields<real>& F, const Geom& g, int first_plane, bool total_b,
                                             long long column, const Images& im, bool low) {
  const long long n = column + (low ? 0 : g.nz + 2);
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const real v = F.f[first_plane + c][n + e];
      if (total_b) put_images_b(F, c, n + e, im, v);
      else put_images(F.f[first_plane + c], n + e, im, v);
    }
}

// The interior columns of the layers 2, 3, N, N+1 (x layers over the interior
// l, then y layers over the k outside the x layers), node by node: item t is
// node m of column (k, l).
__host__ __device__ __forceinline__ long long layer_items(const Geom& g) {
  return (4LL * g.ny + 4LL * (g.nx - 4)) * g.gz;
}
__device__ __forceinline__ void layer_node(const Geom& g, long long t, int& k, int& l, int& m) {
  m = (int)(t % g.gz);
  const int col = (int)(t / g.gz), r = col & 3;
  if (col < 4 * g.ny) {
    k = r < 2 ? 2 + r : g.nx + r - 2;
    l = 2 + (col >> 2);
  } else {
    k = 4 + ((col - 4 * g.ny) >> 2);
    l = r < 2 ? 2 + r : g.ny + r - 2;
  }
}

// sr_current2 at size 1: x pass (:1815-1935), then y pass over every k
// including the x ghosts (:1937-2036); layers 2, 3 += N+2, N+3 and N, N+1 +=
// 0, 1. Both passes in one: a column in both layers works on its three ghosts
// too, in the passes' order.
template <typename real>
__device__ __forceinline__ void fold_item(real* a, const Geom& g, long long t) {
  int k, l, m;
  layer_node(g, t, k, l, m);
  const long long dx = (long long)image_shift(k, g.nx) * g.sx, dy = (long long)image_shift(l, g.ny) * g.gz;
  real* p = a + (long long)k * g.sx + (long long)l * g.gz + m;
  if (dx != 0 && dy != 0) {
    const real xy = p[dx + dy];
    const real x = p[dx], y = p[dy] + xy;  // x pass at the y ghost
    p[dy] = y;
    p[0] = (p[0] + x) + y;
    p[dx] = x + xy;                        // y pass at the x ghost
  } else {
    p[0] += p[dx + dy];
  }
}

// Work that rides in a field update's launch, in the blocks after its own:
// clearing the current and density planes for the step's deposits, or folding
// their ghosts. Neither touches what the update reads or writes.
template <typename real>
struct Rider {
  int mode;          // 0 none, 1 clear, 2 fold
  int first;         // first block of it
  float4* clear;     // 16-byte units
  long long nclear;
  PlaneSet<real> fold;
};
template <typename real>
__device__ __forceinline__ void ride(const Rider<real>& r, const Geom& g) {
  const long long t0 = (long long)(blockIdx.x - r.first) * blockDim.x + threadIdx.x;
  const long long stride = (long long)(gridDim.x - r.first) * blockDim.x;
  if (r.mode == 1) {
    for (long long t = t0; t < r.nclear; t += stride) r.clear[t] = make_float4(0.f, 0.f, 0.f, 0.f);
  } else {
    const long long per = layer_items(g);
    for (long long t = t0; t < per * r.fold.count; t += stride) fold_item(r.fold.p[t / per], g, t % per);
  }
}

// The fold on its own.
template <typename real>
__global__ void fold_kernel(Rider<real> r, Geom g) { ride(r, g); }

// sr_e / sr_phi's copies on their own: every column of the layers to its images.
template <typename real>
__global__ void wrap_kernel(PlaneSet<real> s, Geom g) {
  const long long per = layer_items(g);
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < per * s.count;
       t += (long long)gridDim.x * blockDim.x) {
    int k, l, m;
    layer_node(g, t % per, k, l, m);
    real* a = s.p[t / per];
    const long long n = (long long)k * g.sx + (long long)l * g.gz + m;
    put_images(a, n, images_of(g, k, l), a[n]);
  }
}

struct BParams {
  double temp;   // dt / (4 e0)           (renew_b4_2 :2583)
  double dth;    // dt / 2
  double inv24dx;
};

struct EParams {
  double temp;   // c^2 dt                (renew_e4_2 :2616)
  double mu0;
  double inv24dx;
};

// Damping coefficients of renew_b4_2 at sigma s: ca = (1 - s t)/(1 + s t),
// cb = (dt/2)/(1 + s t); s = 0 gives exactly (1, dt/2) without the divisions.
__device__ __forceinline__ void b_coeffs(double s, const BParams& p, double& ca, double& cb) {
  if (s == 0.0) { ca = 1.0; cb = p.dth; return; }
  ca = (1. - s * p.temp) / (1. + s * p.temp);
  cb = p.dth / (1. + s * p.temp);
}

// Damping coefficients of renew_e4_2 at sigma s: with h = mu0 s t / 2,
// ca = (1 - h)/(1 + h), cb = t/(1 + h); s = 0 gives exactly (1, t).
__device__ __forceinline__ void e_coeffs(double s, const EParams& p, double& ca, double& cb) {
  if (s == 0.0) { ca = 1.0; cb = p.temp; return; }
  const double h = 0.5 * p.mu0 * s * p.temp;
  ca = (1. - h) / (1. + h);
  cb = p.temp / (1. + h);
}

// renew_b4_2 (:2580-2611) on the induced field: DB <- ca DB - cb curl4(E),
// B = B0 + DB, with ca = (1 - s t)/(1 + s t), cb = (dt/2)/(1 + s t).
template <typename real>
__global__ void __launch_bounds__(256) renew_b_kernel(Fields<real> F, Geom g, Ramps rp, BParams p, bool ghosts,
                                                      Rider<real> rider) {
  after_prior();
  if (rider.mode && (int)blockIdx.x >= rider.first) return ride(rider, g);
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int nint = g.nx * g.ny * g.nz;
  if (t >= nint) return;
  const int m = 2 + t % g.nz, l = 2 + (t / g.nz) % g.ny, k = 2 + t / (g.nz * g.ny);
  const int n = k * g.sx + l * g.gz + m;
  const int sy = g.gz, sx = g.sx;
  const real* ex = F.f[F_EX];
  const real* ey = F.f[F_EY];
  const real* ez = F.f[F_EZ];
  const real c24 = (real)p.inv24dx;
  // x component at (k+1/2, l, m): sigma[2k+1][2l][2m]
  {
    const double s = sigma_of(rp.a, rp.rx[2 * k + 1], rp.ry[2 * l], rp.rz[2 * m]);
    double ca, cb;
    b_coeffs(s, p, ca, cb);
    const real curl = ((real)27 * (ez[n] - ez[n - sy] - ey[n] + ey[n - 1]) -
                       (ez[n + sy] - ez[n - 2 * sy] - ey[n + 1] + ey[n - 2])) * c24;
    const real db = (real)ca * F.f[F_DBX][n] - (real)cb * curl;
    F.f[F_DBX][n] = db;
    F.f[F_BX][n] = F.f[F_B0X][n] + db;
  }
  {
    const double s = sigma_of(rp.a, rp.rx[2 * k], rp.ry[2 * l + 1], rp.rz[2 * m]);
    double ca, cb;
    b_coeffs(s, p, ca, cb);
    const real curl = ((real)27 * (ex[n] - ex[n - 1] - ez[n] + ez[n - sx]) -
                       (ex[n + 1] - ex[n - 2] - ez[n + sx] + ez[n - 2 * sx])) * c24;
    const real db = (real)ca * F.f[F_DBY][n] - (real)cb * curl;
    F.f[F_DBY][n] = db;
    F.f[F_BY][n] = F.f[F_B0Y][n] + db;
  }
  {
    const double s = sigma_of(rp.a, rp.rx[2 * k], rp.ry[2 * l], rp.rz[2 * m + 1]);
    double ca, cb;
    b_coeffs(s, p, ca, cb);
    const real curl = ((real)27 * (ey[n] - ey[n - sx] - ex[n] + ex[n - sy]) -
                       (ey[n + sx] - ey[n - 2 * sx] - ex[n + sy] + ex[n - 2 * sy])) * c24;
    const real db = (real)ca * F.f[F_DBZ][n] - (real)cb * curl;
    F.f[F_DBZ][n] = db;
    F.f[F_BZ][n] = F.f[F_B0Z][n] + db;
  }
  if (!ghosts) return;
  const Images im = images_of(g, k, l);
  if (im.n == 0) return;
#pragma unroll
  for (int c = 0; c < 3; ++c) put_images_b(F, c, n, im, F.f[F_BX + c][n]);
  if (m == 2) z_end_images(F, g, F_BX, true, n - m, im, true);
  if (m == g.nz + 1) z_end_images(F, g, F_BX, true, n - m, im, false);
}

// renew_e4_2 (:2613-2652): E <- ca E + cb (curl4(DB) - mu0 (J_i - J_e)),
// ca = (1 - mu0 s t/2)/(1 + mu0 s t/2), cb = t/(1 + mu0 s t/2), t = c^2 dt.
template <typename real>
__global__ void __launch_bounds__(256) renew_e_kernel(Fields<real> F, Geom g, Ramps rp, EParams p, bool ghosts) {
  after_prior();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int nint = g.nx * g.ny * g.nz;
  if (t >= nint) return;
  const int m = 2 + t % g.nz, l = 2 + (t / g.nz) % g.ny, k = 2 + t / (g.nz * g.ny);
  const int n = k * g.sx + l * g.gz + m;
  const int sy = g.gz, sx = g.sx;
  const real* bx = F.f[F_DBX];
  const real* by = F.f[F_DBY];
  const real* bz = F.f[F_DBZ];
  const real c24 = (real)p.inv24dx;
  const real mu0 = (real)p.mu0;
  {
    const double s = sigma_of(rp.a, rp.rx[2 * k], rp.ry[2 * l + 1], rp.rz[2 * m + 1]);
    double ca, cb;
    e_coeffs(s, p, ca, cb);
    const real curl = ((real)27 * ((bz[n + sy] - bz[n]) - (by[n + 1] - by[n])) -
                       ((bz[n + 2 * sy] - bz[n - sy]) - (by[n + 2] - by[n - 1]))) * c24;
    F.f[F_EX][n] = (real)ca * F.f[F_EX][n] + (real)cb * (curl - mu0 * (F.f[F_JIX][n] - F.f[F_JEX][n]));
  }
  {
    const double s = sigma_of(rp.a, rp.rx[2 * k + 1], rp.ry[2 * l], rp.rz[2 * m + 1]);
    double ca, cb;
    e_coeffs(s, p, ca, cb);
    const real curl = ((real)27 * ((bx[n + 1] - bx[n]) - (bz[n + sx] - bz[n])) -
                       ((bx[n + 2] - bx[n - 1]) - (bz[n + 2 * sx] - bz[n - sx]))) * c24;
    F.f[F_EY][n] = (real)ca * F.f[F_EY][n] + (real)cb * (curl - mu0 * (F.f[F_JIY][n] - F.f[F_JEY][n]));
  }
  {
    const double s = sigma_of(rp.a, rp.rx[2 * k + 1], rp.ry[2 * l + 1], rp.rz[2 * m]);
    double ca, cb;
    e_coeffs(s, p, ca, cb);
    const real curl = ((real)27 * ((by[n + sx] - by[n]) - (bx[n + sy] - bx[n])) -
                       ((by[n + 2 * sx] - by[n - sx]) - (bx[n + 2 * sy] - bx[n - sy]))) * c24;
    F.f[F_EZ][n] = (real)ca * F.f[F_EZ][n] + (real)cb * (curl - mu0 * (F.f[F_JIZ][n] - F.f[F_JEZ][n]));
  }
  if (!ghosts) return;
  const Images im = images_of(g, k, l);
  if (im.n == 0) return;
#pragma unroll
  for (int c = 0; c < 3; ++c) put_images(F.f[F_EX + c], n, im, F.f[F_EX + c][n]);
  if (m == 2) z_end_images(F, g, F_EX, false, n - m, im, true);
  if (m == g.nz + 1) z_end_images(F, g, F_EX, false, n - m, im, false);
}

}  // namespace pb
