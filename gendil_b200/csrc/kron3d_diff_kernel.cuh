// Interior-penalty DG diffusion (the form of kronnd_diff_kernel.cuh) for 3D hexahedra, N = p + 1 <= 6,
// in registers.
//
// N consecutive lanes own one element as in kron3d_kernel.cuh: lane t holds plane z = t (layout Z,
// values [x][y]) and, after one exchange, plane y = t (layout Y, values [x][z]).  With M the 1D mass
// matrices,
//
//   y = Mz [ My (Ax u + x faces) + Mx (Ay u + y faces) ]   layout Z, one exchange, one z pass
//     + Az (My Mx u) + z faces                              layout Z, one exchange, one z pass
//
// Eight N x N passes and two exchanges.  A face's own terms are linear in the element's diffusivity
// mu_e and go into the pass: A_a = mu_e Kint_a with
//   Kint_a = Khat_a + f sum_s ( -nu/2 b d^T + kappa/2 b b^T + sigma nu/2 d b^T ),  b = l(s), d = l'(s),
// plus f kappa/2 mu_nb b b^T per interior side (on a slice for a basis with nodes on the faces).  What
// is left of a face is the neighbour line's traces (value, normal derivative) combined to two numbers
// (X, Y) per line, added as b X + d Y.  A boundary face has no neighbour; the difference of its own
// terms to those in Kint has the same form with the element's own traces.
//
// Traces of the x neighbours come from staged planes: the group is staged with the element before
// and the one after it, so only wrapped neighbours are read from global memory.  Those of the y and
// z neighbours are formed by lane t for column x = t, where the lanes of an element read consecutive
// values (all of a column's loads in flight together), and change lanes through a shared slot.  The z
// neighbours' (X, Y) pass through My and Mx like any other plane.
//
// The coefficient gradient out[e] = lam^T (dA/dmu_e) u is the same with mu_e = 1 and the neighbours'
// diffusivities 0, in a scalar product with lam on the element (its own rows), minus
//   f sum_s < -nu/2 l'(s).u + kappa/2 [u], l(1-s).lam_nb >_M    per interior face (the neighbours' rows,
// whose test function is the other side of the jump): one face array per face through the two
// tangential mass matrices.
//
// What bounds it: latency at 8 to 12 warps per SM, where two planes, a matrix and the lines in flight
// leave room for no more (p = 4: FP64 pipe 27 % busy, the neighbours' columns the longest wait).
// Measured against the shared-memory kernels (us): apply 32^3 p = 3 65.6 -> 30.7, p = 4 102 -> 64,
// 12x10x11 p = 3 14.5 -> 7.9; gradient 32^3 p = 3 138 -> 41, p = 4 225 -> 72.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "kron3d_kernel.cuh"

namespace dgop {

enum DiffMode : int { kDiffApply = 0, kDiffApplyDot = 1, kDiffGradient = 2 };

template <int N, typename Real, bool GRAD = false>
struct Kron3DDiffShape {
  using S = Kron3DShape<N, Real>;
  // per element: (X, Y) of both sides of an axis, for the gradient also the face array of both sides
  static constexpr int SLOTS = (GRAD ? 6 : 4) * S::NN;
  // shared memory per warp (Reals): staged elements with one more on either end, and one area for
  // the exchanges and, between them, the slots
  static constexpr int STAGE = ((S::EPW + 2) * S::SE + 3) / 4 * 4;
  static constexpr int AREA = (S::TILE > S::EPW * SLOTS ? S::TILE : S::EPW * SLOTS);
  static constexpr int WARP = STAGE + (AREA + 3) / 4 * 4;
};

// Y (+)= A X along the second plane index; X <- A X in place; constant matrices in parameter space.
template <int N, typename Real>
struct ConstMat {
  const Real* a;  // row stride N
  __device__ __forceinline__ Real operator()(int i, int j) const { return a[i * N + j]; }
};
template <int N, bool ACC, typename Real, typename Mat>
__device__ __forceinline__ void const_pass_z(const Mat& A, const Real (&X)[N][N], Real (&Y)[N][N]) {
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int k = 0; k < N; ++k) {
      Real s = ACC ? Y[i][k] : Real(0);
#pragma unroll
      for (int r = 0; r < N; ++r) s = (!ACC && r == 0) ? A(k, 0) * X[i][0] : s + A(k, r) * X[i][r];
      Y[i][k] = s;
    }
}
template <int N, typename Real, typename Mat>
__device__ __forceinline__ void const_line(const Mat& A, const Real (&v)[N], Real (&w)[N]) {
#pragma unroll
  for (int j = 0; j < N; ++j) {
    Real s = A(j, 0) * v[0];
#pragma unroll
    for (int i = 1; i < N; ++i) s += A(j, i) * v[i];
    w[j] = s;
  }
}

// GLL: basis with nodes on the faces (value traces are slices).
template <int N, typename Real, bool GLL, int MODE>
__global__ void __launch_bounds__(128, N <= 4 ? 3 : 2)
    kron3d_diff_kernel(const __grid_constant__ Kron3DDiffParams<Real> P) {
  using S = Kron3DShape<N, Real>;
  constexpr bool DOT = MODE == kDiffApplyDot, GRAD = MODE == kDiffGradient;
  using Sh = Kron3DDiffShape<N, Real, GRAD>;
  constexpr int NN = S::NN, NNN = S::NNN, EPW = S::EPW;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ Real rows[4][N];  // l(0), l(1), l'(0), l'(1)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int le = lane / N, t = lane - le * N;
  const bool slot = le < EPW;
  if (P.skip && *P.skip) return;  // a finished solve: nothing to do
  for (int i = threadIdx.x; i < 4 * N; i += blockDim.x) rows[i / N][i % N] = P.tv[i / N][i % N];
  __syncthreads();
  Real* buf = reinterpret_cast<Real*>(smem_raw) + (size_t)warp * Sh::WARP;
  Real* tile = buf + Sh::STAGE;
  Real* slots = tile + (slot ? le : 0) * Sh::SLOTS;
  const int64_t total = P.sizes[0] * P.sizes[1] * P.sizes[2];
  const int64_t ngroups = (P.nelem - P.e_begin + EPW - 1) / EPW;
  [[maybe_unused]] double dot_acc = 0.0;
  for (int64_t g = (int64_t)blockIdx.x * nw + warp; g < ngroups; g += (int64_t)gridDim.x * nw) {
    const int64_t e0 = P.e_begin + g * EPW;
    const int ne = group_size(EPW, P.nelem - e0);
    const int lead = e0 > 0 ? 1 : 0;  // the staged element before the group
    {
      const int nchunks = (lead + ne + (e0 + ne < total ? 1 : 0)) * NNN / S::CR;
      const Real* src = P.x + (e0 - lead) * NNN;
      for (int ch = lane; ch < nchunks; ch += 32) {
        const int d = ch * S::CR;
        const int r = d / NNN, o = d - r * NNN;
        const int z = o / NN, q = o - z * NN;
        cp_async<S::CB>(buf + r * S::SE + z * S::SP + q, src + d);
      }
      cp_async_commit();
    }
    const bool active = slot && le < ne;
    const int64_t e = e0 + (active ? le : 0);
    uint32_t c[3];
    {
      uint32_t q;
      P.fdx.divmod((uint32_t)e, q, c[0]);
      P.fdy.divmod(q, c[2], c[1]);
    }
    const Real mue = GRAD ? Real(1) : P.mu[e];
    [[maybe_unused]] Real gacc = Real(0);
    const Real* ub = buf + (lead + (slot ? le : 0)) * S::SE;
    // Face (a, s): offset of the element whose traces it takes (0: itself, on the boundary), at that
    // element's face `side`; X = ad (derivative) + ab (value), Y = gm (value); delta: own value on the
    // own slice
    struct Face {
      int64_t off;
      bool inner;
      int side;
      Real ad, ab, gm, delta;
    };
    auto face = [&](int a, int s) {
      Face F;
      const int64_t n = P.sizes[a], st = a == 0 ? 1 : (a == 1 ? P.sizes[0] : P.sizes[0] * P.sizes[1]);
      const bool edge = s ? (int64_t)c[a] + 1 == n : c[a] == 0;
      const Real f = P.f[a], nu = s ? Real(1) : Real(-1);
      F.inner = !edge || P.periodic[a];
      if (F.inner) {
        F.off = edge ? -(n - 1) * st : st;
        if (!s) F.off = -F.off;
        const Real mun = GRAD ? Real(0) : P.mu[e + F.off];
        F.side = 1 - s;
        F.ad = Real(-0.5) * f * nu * mun;
        F.ab = Real(-0.5) * f * P.kappa * (mue + mun);
        F.gm = Real(-0.5) * f * nu * P.sigma * mue;
        F.delta = Real(0.5) * f * P.kappa * mun;
      } else {
        const Real m = P.boundary ? mue : -mue;
        F.off = 0;
        F.side = s;
        F.ad = Real(-0.5) * f * nu * m;
        F.ab = Real(0.5) * f * P.kappa * m;
        F.gm = Real(0.5) * f * P.sigma * nu * m;
        F.delta = Real(0);
      }
      return F;
    };
    // column x = t of the element at src: col[i][j], i along the axis of stride so, j along that of
    // stride st.  (The gradient's interior faces need the values at the face only.)
    auto load_column = [&](const Real* src, const Face& F, int st, int so, Real(&col)[N][N]) {
#pragma unroll
      for (int i = 0; i < N; ++i)
#pragma unroll
        for (int j = 0; j < N; ++j) {
          const bool need = !(GRAD && GLL && F.inner) || j == (F.side ? N - 1 : 0);
          col[i][j] = need ? __ldg(src + st * j + so * i) : Real(0);
        }
    };
    // GRAD: the face array of face (a, s) in one value: own derivative and value, neighbour's value
    auto jump_term = [&](int a, int s, Real od, Real ov, Real vb) {
      return P.f[a] * ((s ? Real(-0.5) : Real(0.5)) * od + Real(0.5) * P.kappa * (ov - vb));
    };
    // GRAD: minus the scalar product of a row of the face array, through matrix m, with the neighbour's
    // lam trace (value r at lam(r))
    auto face_product = [&](const Real* m, const Real(&v)[N], auto lam) {
      Real w[N];
      const_line<N>(ConstMat<N, Real>{m}, v, w);
#pragma unroll
      for (int r = 0; r < N; ++r) gacc -= w[r] * lam(r);
    };
    // GRAD: lam's trace at face `side` of the element at `base`, along an axis of stride st
    auto lam_trace = [&](const Real* base, int side, int st) {
      if (GLL) return __ldg(base + (side ? (N - 1) * st : 0));
      Real v = Real(0);
#pragma unroll
      for (int i = 0; i < N; ++i) v += rows[side][i] * __ldg(base + i * st);
      return v;
    };
    if (GRAD) {
      cp_async_wait<0>();
      __syncwarp();
    }
    // (X, Y) of the y faces for column x = t, to slots [z][x]
    if (active) {
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const Face F = face(1, s);
        const Real* src = P.x + (e + F.off) * NNN + t;
        Real dr[N], col[N][N];
        [[maybe_unused]] Real fa[N];
        load_column(src, F, N, NN, col);
#pragma unroll
        for (int i = 0; i < N; ++i) dr[i] = rows[2 + F.side][i];
#pragma unroll
        for (int z = 0; z < N; ++z) {
          Real vd = Real(0), vb = Real(0);
#pragma unroll
          for (int y = 0; y < N; ++y) {
            vd += dr[y] * col[z][y];
            if (!GLL) vb += rows[F.side][y] * col[z][y];
          }
          if (GLL) vb = F.side ? col[z][N - 1] : col[z][0];
          slots[(2 * s) * NN + z * N + t] = F.ad * vd + F.ab * vb;
          slots[(2 * s + 1) * NN + z * N + t] = F.gm * vb;
          if constexpr (GRAD) {
            Real od = Real(0), ov = Real(0);
#pragma unroll
            for (int y = 0; y < N; ++y) {
              const Real v = ub[z * S::SP + N * y + t];
              od += P.tv[2 + s][y] * v;
              if (!GLL) ov += P.tv[s][y] * v;
            }
            if (GLL) ov = ub[z * S::SP + (s ? N * (N - 1) : 0) + t];
            fa[z] = jump_term(1, s, od, ov, vb);
          }
        }
        if constexpr (GRAD) {
          Real wz[N];
          const_line<N>(ConstMat<N, Real>{P.mm[2]}, fa, wz);
#pragma unroll
          for (int z = 0; z < N; ++z) slots[(4 + s) * NN + z * N + t] = wz[z];
        }
      }
    }
    if (!GRAD) cp_async_wait<0>();
    __syncwarp();
    if (GRAD && active) {
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const Face F = face(1, s);
        if (!F.inner) continue;
        const Real* lb = P.lam + (e + F.off) * NNN + NN * t;
        Real v[N];
#pragma unroll
        for (int x = 0; x < N; ++x) v[x] = slots[(4 + s) * NN + t * N + x];
        face_product(P.mm[0], v, [&](int x) { return lam_trace(lb + x, F.side, N); });
      }
    }
    if (GRAD) __syncwarp();  // the face arrays' slots are free again
    Real G[N][N];
    // ---------------------------------------------------------------- x axis
    {
      load_plane_z<N>(ub, t, active, G);
      lines_inplace<N, true>(ConstMat<N, Real>{P.kint[0]}, G);
      scale_plane<N>(mue, G);
      if (active) {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const Face F = face(0, s);
          const bool here = F.off == 0 || F.off == 1 || F.off == -1;
          const Real* src = here ? ub + (int)F.off * S::SE + t * S::SP : P.x + (e + F.off) * NNN + t * NN;
          Real dr[N];
          [[maybe_unused]] Real fa[N];
#pragma unroll
          for (int i = 0; i < N; ++i) dr[i] = rows[2 + F.side][i];
#pragma unroll
          for (int y = 0; y < N; ++y) {
            Real vd = Real(0), vb = Real(0), own = Real(0);
#pragma unroll
            for (int i = 0; i < N; ++i) {
              const Real v = src[N * y + i];
              vd += dr[i] * v;
              if (!GLL) {
                vb += rows[F.side][i] * v;
                own += P.tv[s][i] * ub[t * S::SP + N * y + i];
              }
            }
            if (GLL) {
              vb = src[N * y + (F.side ? N - 1 : 0)];
              own = ub[t * S::SP + N * y + (s ? N - 1 : 0)];
            }
            const Real X = F.ad * vd + F.ab * vb + F.delta * own, Y = F.gm * vb;
#pragma unroll
            for (int j = 0; j < N; ++j) {
              if (!GLL) G[j][y] += P.tv[s][j] * X;
              else if (j == (s ? N - 1 : 0)) G[j][y] += X;
              G[j][y] += P.tv[2 + s][j] * Y;
            }
            if constexpr (GRAD) {
              Real od = Real(0);
#pragma unroll
              for (int i = 0; i < N; ++i) od += P.tv[2 + s][i] * ub[t * S::SP + N * y + i];
              fa[y] = jump_term(0, s, od, own, vb);
            }
          }
          if constexpr (GRAD) {
            Real wy[N];
            const_line<N>(ConstMat<N, Real>{P.mm[1]}, fa, wy);
#pragma unroll
            for (int y = 0; y < N; ++y) slots[(4 + s) * NN + t * N + y] = wy[y];
          }
        }
      }
      lines_inplace<N, false>(ConstMat<N, Real>{P.mm[1]}, G);
    }
    if (GRAD) __syncwarp();
    if (GRAD && active) {
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const Face F = face(0, s);
        if (!F.inner) continue;
        const Real* lb = P.lam + (e + F.off) * NNN + N * t;
        Real v[N];
#pragma unroll
        for (int z = 0; z < N; ++z) v[z] = slots[(4 + s) * NN + z * N + t];
        face_product(P.mm[2], v, [&](int z) { return lam_trace(lb + NN * z, F.side, 1); });
      }
    }
    // ---------------------------------------------------------------- y axis
    {
      Real X2[N][N];
      load_plane_z<N>(ub, t, active, X2);
      lines_inplace<N, false>(ConstMat<N, Real>{P.kint[1]}, X2);
      scale_plane<N>(mue, X2);
      if (active) {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const Real delta = face(1, s).delta;
#pragma unroll
          for (int x = 0; x < N; ++x) {
            Real own = Real(0);
            if (GLL) {
              own = ub[t * S::SP + (s ? N * (N - 1) : 0) + x];
            } else {
#pragma unroll
              for (int y = 0; y < N; ++y) own += P.tv[s][y] * ub[t * S::SP + N * y + x];
            }
            const Real X = slots[(2 * s) * NN + t * N + x] + delta * own, Y = slots[(2 * s + 1) * NN + t * N + x];
#pragma unroll
            for (int j = 0; j < N; ++j) {
              if (!GLL) X2[x][j] += P.tv[s][j] * X;
              else if (j == (s ? N - 1 : 0)) X2[x][j] += X;
              X2[x][j] += P.tv[2 + s][j] * Y;
            }
          }
        }
      }
      lines_inplace<N, true>(ConstMat<N, Real>{P.mm[0]}, X2);
#pragma unroll
      for (int i = 0; i < N; ++i)
#pragma unroll
        for (int j = 0; j < N; ++j) G[i][j] += X2[i][j];
    }
    __syncwarp();  // the slots have been read: their area takes the exchange
    exchange_tile<N>(tile, le, t, slot, G);
    Real out[N][N];
    const_pass_z<N, false>(ConstMat<N, Real>{P.mm[2]}, G, out);
    // ---------------------------------------------------------------- z axis
    {
      Real X[N][N];
      load_plane_z<N>(ub, t, active, X);
      lines_inplace<N, true>(ConstMat<N, Real>{P.mm[0]}, X);
      lines_inplace<N, false>(ConstMat<N, Real>{P.mm[1]}, X);
      exchange_tile<N>(tile, le, t, slot, X);
      Real own[2][N];  // own traces at the two z faces
#pragma unroll
      for (int x = 0; x < N; ++x) {
        Real w[N];
        const_line<N>(ConstMat<N, Real>{P.kint[2]}, X[x], w);
#pragma unroll
        for (int z = 0; z < N; ++z) out[x][z] += mue * w[z];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          if (GLL) {
            own[s][x] = X[x][s ? N - 1 : 0];
          } else {
            own[s][x] = Real(0);
#pragma unroll
            for (int z = 0; z < N; ++z) own[s][x] += P.tv[s][z] * X[x][z];
          }
        }
      }
      // (X, Y) of the z faces for column x = t, through My, to slots [y][x]
      if (active) {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const Face F = face(2, s);
          const Real* src = P.x + (e + F.off) * NNN + t;
          Real vd[N], vb[N], w[N], col[N][N];
          load_column(src, F, NN, N, col);
#pragma unroll
          for (int y = 0; y < N; ++y) vd[y] = vb[y] = Real(0);
#pragma unroll
          for (int z = 0; z < N; ++z) {
            const Real dz = rows[2 + F.side][z], bz = rows[F.side][z];
#pragma unroll
            for (int y = 0; y < N; ++y) {
              vd[y] += dz * col[y][z];
              if (!GLL) vb[y] += bz * col[y][z];
            }
          }
          if (GLL) {
#pragma unroll
            for (int y = 0; y < N; ++y) vb[y] = F.side ? col[y][N - 1] : col[y][0];
          }
#pragma unroll
          for (int y = 0; y < N; ++y) vd[y] = F.ad * vd[y] + F.ab * vb[y];
          if constexpr (GRAD) {
            Real fa[N];
#pragma unroll
            for (int y = 0; y < N; ++y) {
              Real od = Real(0), ov = Real(0);
#pragma unroll
              for (int z = 0; z < N; ++z) {
                const Real v = ub[z * S::SP + N * y + t];
                od += P.tv[2 + s][z] * v;
                if (!GLL) ov += P.tv[s][z] * v;
              }
              if (GLL) ov = ub[(s ? N - 1 : 0) * S::SP + N * y + t];
              fa[y] = jump_term(2, s, od, ov, vb[y]);
            }
            const_line<N>(ConstMat<N, Real>{P.mm[1]}, fa, w);
#pragma unroll
            for (int y = 0; y < N; ++y) slots[(4 + s) * NN + y * N + t] = w[y];
          }
          const_line<N>(ConstMat<N, Real>{P.mm[1]}, vd, w);
#pragma unroll
          for (int y = 0; y < N; ++y) slots[(2 * s) * NN + y * N + t] = w[y];
          const_line<N>(ConstMat<N, Real>{P.mm[1]}, vb, w);
#pragma unroll
          for (int y = 0; y < N; ++y) slots[(2 * s + 1) * NN + y * N + t] = F.gm * w[y];
        }
      }
      __syncwarp();
      if (active) {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const Real delta = face(2, s).delta;
          Real v[N], X1[N], Y1[N];
#pragma unroll
          for (int x = 0; x < N; ++x) v[x] = slots[(2 * s) * NN + t * N + x];
          const_line<N>(ConstMat<N, Real>{P.mm[0]}, v, X1);
#pragma unroll
          for (int x = 0; x < N; ++x) v[x] = slots[(2 * s + 1) * NN + t * N + x];
          const_line<N>(ConstMat<N, Real>{P.mm[0]}, v, Y1);
#pragma unroll
          for (int x = 0; x < N; ++x) {
            const Real Xx = X1[x] + delta * own[s][x];
#pragma unroll
            for (int j = 0; j < N; ++j) {
              if (!GLL) out[x][j] += P.tv[s][j] * Xx;
              else if (j == (s ? N - 1 : 0)) out[x][j] += Xx;
              out[x][j] += P.tv[2 + s][j] * Y1[x];
            }
          }
        }
      }
    }
    if constexpr (GRAD) {
      if (active) {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const Face F = face(2, s);
          if (!F.inner) continue;
          const Real* lb = P.lam + (e + F.off) * NNN + N * t;
          Real v[N];
#pragma unroll
          for (int x = 0; x < N; ++x) v[x] = slots[(4 + s) * NN + t * N + x];
          face_product(P.mm[0], v, [&](int x) { return lam_trace(lb + x, F.side, NN); });
        }
        const Real* le_ = P.lam + e * NNN + N * t;
#pragma unroll
        for (int z = 0; z < N; ++z)
#pragma unroll
          for (int x = 0; x < N; ++x) gacc += out[x][z] * __ldg(le_ + NN * z + x);
      }
      // sum over the element's lanes in a fixed order
      Real sum = gacc;
#pragma unroll
      for (int i = 1; i < N; ++i) sum += __shfl_sync(0xffffffffu, gacc, (lane + i) & 31);
      if (active && t == 0) P.gout[e] = P.gscale ? P.gscale[e] * sum : sum;
      __syncwarp();
      continue;
    }
    __syncwarp();  // every lane is done reading the staged input and the slots
    if (slot) {
      Real* ob = buf + le * S::SE;
#pragma unroll
      for (int k = 0; k < N; ++k)
#pragma unroll
        for (int i = 0; i < N; i += S::V) {
          Real v[S::V];
#pragma unroll
          for (int q = 0; q < S::V; ++q) v[q] = out[i + q][k];
          vstore<Real, S::V>(ob + k * S::SP + N * t + i, v);
        }
    }
    __syncwarp();
    {
      const int nchunks = ne * NNN / S::CR;
      Real* dst = P.y + e0 * NNN;
      const Real alpha = P.alpha, by = P.beta_y;
      for (int ch = lane; ch < nchunks; ch += 32) {
        const int d = ch * S::CR;
        const int r = d / NNN, o = d - r * NNN;
        const int z = o / NN, q0 = o - z * NN;
        Real v[S::CR];
        vload<Real, S::CR>(buf + r * S::SE + z * S::SP + q0, v);
        if (by == Real(0)) {
#pragma unroll
          for (int q = 0; q < S::CR; ++q) v[q] = alpha * v[q];
        } else {
          Real y0[S::CR];
          vload<Real, S::CR>(dst + d, y0);
#pragma unroll
          for (int q = 0; q < S::CR; ++q) v[q] = alpha * v[q] + by * y0[q];
        }
        vstore<Real, S::CR>(dst + d, v);
        if constexpr (DOT) {
          Real z2[S::CR];
          vldg<Real, S::CR>(P.dot_z + e0 * NNN + d, z2);
#pragma unroll
          for (int q = 0; q < S::CR; ++q) dot_acc += (double)v[q] * (double)z2[q];
        }
      }
    }
    __syncwarp();  // the buffer is refilled
  }
  if constexpr (DOT) {
    // fixed-order sums: lanes (tree), warps (in order), one partial per CTA; entries past the grid
    // are zeroed so a reader sums a fixed count
    __shared__ double wsum[4];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dot_acc += __shfl_down_sync(0xffffffffu, dot_acc, o);
    if (lane == 0) wsum[warp] = dot_acc;
    __syncthreads();
    if (threadIdx.x == 0) {
      double s = 0.0;
      for (int w = 0; w < nw; ++w) s += wsum[w];
      P.dot_partials[blockIdx.x] = s;
    }
    for (int i = gridDim.x + blockIdx.x * blockDim.x + threadIdx.x; i < P.dot_count; i += gridDim.x * blockDim.x)
      P.dot_partials[i] = 0.0;
  }
}

}  // namespace dgop
