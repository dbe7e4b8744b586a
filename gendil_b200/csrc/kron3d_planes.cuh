// Plane operations shared by the N = 4 FP64 kernels (kron3d_p3_kernel.cuh, kron3d_tma_kernel.cuh).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "kron3d_kernel.cuh"

namespace dgop {

// Y[i][j] = sum_r A(i, r) X[r][j]      (operator along the first plane index)
template <int N, typename Real, typename Mat>
__device__ __forceinline__ void apply_first(const Mat& A, const Real (&X)[N][N], Real (&Y)[N][N]) {
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int j = 0; j < N; ++j) {
      Real s = A(i, 0) * X[0][j];
#pragma unroll
      for (int r = 1; r < N; ++r) s += A(i, r) * X[r][j];
      Y[i][j] = s;
    }
}

// Y[i][j] = sum_r A(j, r) X[i][r]      (operator along the second plane index)
template <int N, typename Real, typename Mat>
__device__ __forceinline__ void apply_second(const Mat& A, const Real (&X)[N][N], Real (&Y)[N][N]) {
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int j = 0; j < N; ++j) {
      Real s = A(j, 0) * X[i][0];
#pragma unroll
      for (int r = 1; r < N; ++r) s += A(j, r) * X[i][r];
      Y[i][j] = s;
    }
}

// Layout exchange through the warp's shared tile.  z_to_y: lane t holds X[i][j] = (x=i, y=j, z=t)
// and receives X[i][k] = (x=i, y=t, z=k); otherwise the reverse.  Tile layout [y][z][x].
template <int N, typename Real>
__device__ __forceinline__ void exchange_tile_dir(Real* tile, int le, int t, bool slot, bool z_to_y, Real (&X)[N][N]) {
  using S = Kron3DShape<N, Real>;
  constexpr int V = S::V;
  Real* b = tile + le * S::TSE;
  // layout Z side: lane t = z owns (x, y = j) at j * TA + t * N + x;
  // layout Y side: lane t = y owns (x, z = k) at t * TA + k * N + x
  auto z_side = [&](int j, int i) { return b + j * S::TA + t * N + i; };
  auto y_side = [&](int k, int i) { return b + t * S::TA + k * N + i; };
  if (slot) {
#pragma unroll
    for (int j = 0; j < N; ++j)
#pragma unroll
      for (int i = 0; i < N; i += V) {
        Real v[V];
#pragma unroll
        for (int q = 0; q < V; ++q) v[q] = X[i + q][j];
        vstore<Real, V>(z_to_y ? z_side(j, i) : y_side(j, i), v);
      }
  }
  __syncwarp();
  if (slot) {
#pragma unroll
    for (int j = 0; j < N; ++j)
#pragma unroll
      for (int i = 0; i < N; i += V) {
        Real v[V];
        vload<Real, V>(z_to_y ? y_side(j, i) : z_side(j, i), v);
#pragma unroll
        for (int q = 0; q < V; ++q) X[i + q][j] = v[q];
      }
  }
  __syncwarp();  // the tile is free again
}

template <typename Real>
__device__ __forceinline__ int64_t neighbour_offset(const KronHead<Real>& P, int a, int s, uint32_t ca) {
  const int64_t n = P.sizes[a];
  const int64_t st = a == 0 ? 1 : (a == 1 ? P.sizes[0] : P.sizes[0] * P.sizes[1]);
  if (s == 0) return ca > 0 ? -st : (n - 1) * st;
  return (int64_t)ca + 1 < n ? st : -(n - 1) * st;
}

// Face word bits (5 per face f = axis * 2 + side): corner, neighbour trace, inflow value g, and the
// trace source (kron_tma.h) in bits 3-4.
enum : uint32_t { kRecCorner = 1u, kRecNb = 2u, kRecG = 4u };

}  // namespace dgop
