// The tile product behind the sine transforms of the 2D and 3D Poisson steps,
// which multiply small dense matrices (up to 256 or so on a side) by sine
// tables: a block of 256 threads forms a T x T tile of C = L R, (T / 16)^2
// outputs per thread.
//
// Both operands are staged k-major in shared memory, kGemmK deep, so that a
// thread reads its rows and columns with vector loads; the next stage's
// elements are on their way from global memory while this one is multiplied;
// FP32 multiplies two columns at a time. Bound by the stages' latency when the
// tiles are few (one small matrix per SM), by the FMA rate otherwise; T = 32
// gives such a small batch four times the blocks. Scalar FMAs, no prefetch and
// 64 x 64 tiles throughout (and, in 2D, sines and divisions per output in FP64)
// took 22 us a transform for 8 runs of 64 to 96 a side and 21 us for 96^3; a 3D
// step with cleaning at 96^3 x 8 went from 1.028 to 0.991 ms.
#pragma once

#include "common.cuh"

namespace pb {

constexpr int kGemmK = 32;

template <typename real, int T>
struct GemmStage {
  real l[kGemmK][T + 4];  // [k][row]
  real r[kGemmK][T + 4];  // [k][col]
};

template <int U>
__device__ __forceinline__ void load_run(const float* p, float (&v)[U]) {
  if constexpr (U == 4) {
    const float4 q = *reinterpret_cast<const float4*>(p);
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
  } else {
    const float2 q = *reinterpret_cast<const float2*>(p);
    v[0] = q.x; v[1] = q.y;
  }
}
template <int U>
__device__ __forceinline__ void load_run(const double* p, double (&v)[U]) {
#pragma unroll
  for (int u = 0; u < U; u += 2) {
    const double2 q = *reinterpret_cast<const double2*>(p + u);
    v[u] = q.x; v[u + 1] = q.y;
  }
}

// acc += sum over k < K of L(row, k) R(k, col) for the thread's rows
// U ty .. U ty + U - 1 and columns U tx .. of the tile (tx = thread % 16, ty =
// thread / 16). left(row, k) and right(k, col) give the elements of the tile's
// rows, columns and all k, zero outside the matrices. Every thread of the
// block calls it; each stage begins with a barrier, which also keeps it from the
// last one's readers of an earlier product.
template <typename real, int T, typename Left, typename Right>
__device__ __forceinline__ void gemm_tile(GemmStage<real, T>& st, int K, Left left, Right right,
                                          real (&acc)[T / 16][T / 16]) {
  constexpr int U = T / 16, N = T * kGemmK / 256;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  real lv[N], rv[N];
  // left: a warp takes 4 rows x 8 consecutive k (coalesced reads, transposed
  // stores on 32 different banks); right: consecutive columns
  const auto fetch = [&](int k0) {
#pragma unroll
    for (int e = 0; e < N; ++e) {
      const int q = threadIdx.x + 256 * e, ch = q >> 5, l = q & 31;
      lv[e] = left(4 * (ch % (T / 4)) + (l >> 3), k0 + 8 * (ch / (T / 4)) + (l & 7));
      rv[e] = right(k0 + q / T, q % T);
    }
  };
  fetch(0);
  for (int k0 = 0; k0 < K; k0 += kGemmK) {
    __syncthreads();  // the last stage's reads are done
#pragma unroll
    for (int e = 0; e < N; ++e) {
      const int q = threadIdx.x + 256 * e, ch = q >> 5, l = q & 31;
      st.l[8 * (ch / (T / 4)) + (l & 7)][4 * (ch % (T / 4)) + (l >> 3)] = lv[e];
      st.r[q / T][q % T] = rv[e];
    }
    __syncthreads();
    if (k0 + kGemmK < K) fetch(k0 + kGemmK);
#pragma unroll 8
    for (int k = 0; k < kGemmK; ++k) {
      real a[U], b[U];
      load_run<U>(&st.l[k][U * ty], a);
      load_run<U>(&st.r[k][U * tx], b);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if constexpr (sizeof(real) == 4) {
#pragma unroll
          for (int v = 0; v < U; v += 2) {
            const float2 s = __ffma2_rn(make_float2(a[u], a[u]), make_float2(b[v], b[v + 1]),
                                        make_float2(acc[u][v], acc[u][v + 1]));
            acc[u][v] = s.x;
            acc[u][v + 1] = s.y;
          }
        } else {
#pragma unroll
          for (int v = 0; v < U; ++v) acc[u][v] += a[u] * b[v];
        }
      }
    }
  }
}

}  // namespace pb
