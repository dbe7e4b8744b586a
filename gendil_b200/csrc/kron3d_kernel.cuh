// Register-resident Kronecker-form DG operator kernel for 3D hexahedra, N = p + 1 <= 6.
//
// N consecutive lanes own one element; lane t holds an N x N plane of it in registers:
//   layout Z: plane z = t, values [x][y]      layout Y: plane y = t, values [x][z]
// Every term (x)_k A_k is a plane phase (its x and y factors, in place, in layout Z), one exchange
// to layout Y and its z factor, accumulated there:
//
//   x term: Dx, x faces, Txy                | exchange |  out  = Txz .
//   y term: Dy, y faces, Tyx                | exchange |  out += Tyz .
//   z term: Tzx, Tzy                        | exchange |  out += Dz . + z faces   (mass merged in Dz)
//   a separate mass term: Mx, My            | exchange |  out += Md .
//
// Three exchanges and one plane live beside the accumulator (the order x, z, y with the faces at
// each term's start needs four exchanges and two more planes).  The upwind neighbour trace of an
// inflow face is added to the face slice of the D-pass output, so the tangential passes that
// follow apply the face's tangential operator to it; the z faces come after the tangential
// passes, so the z neighbours' slices pass through Tzy and Tzx on their own: lane t takes column
// x = t through Tzy, then row y = t through Tzx (2 N^2 multiply-adds per lane against 9 N^3).
//
// Memory: each warp loops over groups of 32/N consecutive elements (persistent grid).  The
// group's DoFs and the neighbour traces its inflow faces need are staged into padded shared
// memory (coalesced cp.async copies; STAGES = 2: one group ahead), each term reads its plane from
// there, and results leave through the same buffer with coalesced stores.  Which traces an element
// needs is one 32-bit face word per element, built at operator creation (kron_face_words); with
// per-element velocity factors, which the caller may change between applies, the word is built
// in the kernel (N <= 4 outside the general form: kron3d_p3_kernel.cuh instead).  Constant 1D matrices
// are read from kernel-parameter space, only element-dependent ones from global memory.  For N = 2 and
// 4 the layout exchanges can be register butterflies (shfl_xor within the element's lanes); otherwise
// they go through a shared tile.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "dgop_params.h"
#include "kron.h"

namespace dgop {

template <int N, typename Real>
struct Kron3DShape {
  static constexpr int EPW = 32 / N;  // elements per warp group
  static constexpr int NN = N * N, NNN = N * N * N;
  // staging copy granule (bytes): 16 when a plane is a whole number of 16-byte chunks
  static constexpr int CB = (NN * (int)sizeof(Real)) % 16 == 0 ? 16 : ((NN * (int)sizeof(Real)) % 8 == 0 ? 8 : 4);
  static constexpr int CR = CB / (int)sizeof(Real);  // Reals per chunk
  static constexpr int pad_for(int p) { return ((NN + p) * (int)sizeof(Real)) % CB == 0 ? p : pad_for(p + 1); }
  // vector width (Reals) of shared-memory accesses along x: 16 bytes when N allows it
  static constexpr int V = kron_vec<Real>(N);
  // Shared-memory bank model: accesses of G bytes are served 128 bytes at a time (8, 16 or 32
  // lanes together); two lanes of one such phase conflict when their G-byte granules fall in the
  // same bank group.  `distinct` checks one access pattern: offset(le, t) in Reals.
  template <typename F>
  static constexpr bool distinct(int vreals, F offset) {
    const int G = vreals * (int)sizeof(Real);
    const int L = G >= 16 ? 8 : (G == 8 ? 16 : 32);
    const int CH = 128 / (G >= 16 ? 16 : G);
    for (int ph = 0; ph < 32 / L; ++ph) {
      unsigned long long seen = 0;
      for (int l = ph * L; l < ph * L + L; ++l) {
        const int le = l / N, t = l - le * N;
        if (le >= EPW) continue;
        const int c = (offset(le, t) / vreals) % CH;
        if ((seen >> c) & 1ull) return false;
        seen |= 1ull << c;
      }
    }
    return true;
  }
  // Staged element layout: (x, y, z) at z * SP + y * N + x, element stride SE.  The smallest
  // strides (keeping the copy granule's alignment) for which the layout-Z and layout-Y plane
  // accesses are conflict-free; fallback: the dense plane padded to the copy granule.
  struct Staged {
    int SP, SE;
  };
  static constexpr Staged staged_geom() {
    // a conflict-free layout more than 25 % larger than the dense one costs more shared memory
    // (warps per SM) than its conflicts cost
    const int dense = N * (NN + pad_for(1));
    for (int se = N * NN; se <= dense + dense / 4; ++se) {
      if ((se * (int)sizeof(Real)) % CB || se % V) continue;
      for (int sp = NN; N * sp <= se; ++sp) {
        if ((sp * (int)sizeof(Real)) % CB || sp % V) continue;
        if (distinct(V, [&](int le, int t) { return le * se + t * sp; }) &&
            distinct(V, [&](int le, int t) { return le * se + t * N; }))
          return {sp, se};
      }
    }
    return {NN + pad_for(1), N * (NN + pad_for(1))};
  }
  static constexpr int SP = staged_geom().SP;  // staged plane stride (Reals)
  static constexpr int SE = staged_geom().SE;  // staged element stride
  // neighbour traces (N rows of N values): slots 0 and 1 for the first x and y face that needs a
  // neighbour's trace (a second one on the same axis, rare, is read from global memory), slots 2
  // and 3 for the two z faces (their traces pass through the tangential factors in place).
  // Rows are read V-wide; the element stride TE is the smallest conflict-free one.
  static constexpr int RB = (N * (int)sizeof(Real)) % 16 == 0 ? 16 : ((N * (int)sizeof(Real)) % 8 == 0 ? 8 : 4);
  static constexpr int TR = N;                // trace row stride
  static constexpr int TS = N * TR;           // trace slot stride
  static constexpr int kTraceSlots = 4;
  static constexpr int trace_stride() {
    for (int te = kTraceSlots * TS; te <= kTraceSlots * TS + 64; ++te) {
      if ((te * (int)sizeof(Real)) % RB || te % V) continue;
      if (distinct(V, [&](int le, int t) { return le * te + t * TR; })) return te;
    }
    return kTraceSlots * TS;
  }
  static constexpr int TE = trace_stride();   // traces per element
  static constexpr int STAGE = (EPW * (SE + TE) + 3) / 4 * 4;  // one pipeline stage: DoFs, traces
  static constexpr bool BUTTERFLY = (N == 2 || N == 4);  // shuffle exchanges possible
  // Exchange tile per element, layout [y][z][x]: value (x, y, z) at y * TA + z * N + x, element
  // stride TSE.  Both sides of an exchange access V consecutive x values; TA and TSE are the
  // smallest strides for which neither side has a shared-memory bank conflict (tile_geom).
  struct Geom {
    int A, TSE;
  };
  static constexpr Geom tile_geom() {
    const int G = V * (int)sizeof(Real);  // bytes per access
    const int limit = (NNN + 1) + (NNN + 1) / 4;  // at most 25 % above the dense tile
    const int L = G == 16 ? 8 : (G == 8 ? 16 : 32);  // lanes served together
    const int CH = 128 / G;                          // access granules per 128 bytes
    for (int tse = NNN; tse <= limit; ++tse) {
      if (tse % V) continue;
      for (int a = NN; N == 1 || (N - 1) * a + NN <= tse; ++a) {
        if (a % V) continue;
        bool ok = true;
        for (int ph = 0; ph < 32 / L && ok; ++ph) {
          unsigned put = 0, get = 0;
          for (int l = ph * L; l < ph * L + L && ok; ++l) {
            const int le = l / N, t = l - le * N;
            if (le >= EPW) continue;
            const int cp = ((le * tse + t * N) / V) % CH, cg = ((le * tse + t * a) / V) % CH;
            if ((put >> cp) & 1u || (get >> cg) & 1u) ok = false;
            put |= 1u << cp;
            get |= 1u << cg;
          }
        }
        if (ok) return {a, tse};
        if (N == 1) break;
      }
    }
    return {NN, NNN};  // dense (bank conflicts accepted)
  }
  static constexpr int TA = tile_geom().A;
  static constexpr int TSE = tile_geom().TSE;
  static constexpr int TILE = EPW * TSE;
  // shared memory per warp (Reals): STAGES pipeline stages (+ the exchange tile unless shuffles)
  static constexpr int warp_smem(int stages, bool shfl) {
    return stages * STAGE + ((shfl && BUTTERFLY) ? 0 : ((TILE + 3) / 4) * 4);
  }
};

// V consecutive Reals as one shared or global access (V = 1, 2 or 4; 16-byte aligned addresses
// when V > 1), moved component-wise into register arrays.
template <typename Real, int V>
struct Vec16 {};
template <>
struct Vec16<double, 2> {
  using T = double2;
};
template <>
struct Vec16<float, 2> {
  using T = float2;
};
template <>
struct Vec16<float, 4> {
  using T = float4;
};

template <typename Real, int V>
__device__ __forceinline__ void vload(const Real* p, Real (&v)[V]) {
  if constexpr (V == 1) {
    v[0] = p[0];
  } else if constexpr (V == 2) {
    const auto w = *reinterpret_cast<const typename Vec16<Real, 2>::T*>(p);
    v[0] = w.x;
    v[1] = w.y;
  } else {
    static_assert(V == 4 && sizeof(Real) == 4, "unsupported vector width");
    const float4 w = *reinterpret_cast<const float4*>(p);
    v[0] = w.x;
    v[1] = w.y;
    v[2] = w.z;
    v[3] = w.w;
  }
}
template <typename Real, int V>
__device__ __forceinline__ void vstore(Real* p, const Real (&v)[V]) {
  if constexpr (V == 1) {
    p[0] = v[0];
  } else if constexpr (V == 2) {
    using T = typename Vec16<Real, 2>::T;
    T w;
    w.x = v[0];
    w.y = v[1];
    *reinterpret_cast<T*>(p) = w;
  } else {
    static_assert(V == 4 && sizeof(Real) == 4, "unsupported vector width");
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  }
}
template <typename Real, int V>
__device__ __forceinline__ void vldg(const Real* p, Real (&v)[V]) {
  if constexpr (V == 1) {
    v[0] = __ldg(p);
  } else if constexpr (V == 2) {
    const auto w = __ldg(reinterpret_cast<const typename Vec16<Real, 2>::T*>(p));
    v[0] = w.x;
    v[1] = w.y;
  } else {
    static_assert(V == 4 && sizeof(Real) == 4, "unsupported vector width");
    const float4 w = __ldg(reinterpret_cast<const float4*>(p));
    v[0] = w.x;
    v[1] = w.y;
    v[2] = w.z;
    v[3] = w.w;
  }
}

template <int N, typename Real>
struct RegMat {
  Real a[N][N];
  __device__ __forceinline__ Real operator()(int i, int j) const { return a[i][j]; }
};

template <int N, typename Real, int SLOT, typename Block>
struct ParamMat {
  const Block& P;
  __device__ __forceinline__ Real operator()(int i, int j) const { return P.cm[SLOT][i * N + j]; }
};

// Whether slot SLOT's matrix depends on the element: from the slot mask the kernel is compiled
// for (kron.h), or at run time.
template <int SLOT, uint32_t VM, typename Real>
__device__ __forceinline__ bool slot_varies(const KronHead<Real>& P) {
  if constexpr (VM == kVaryRuntime) return P.vary[SLOT] != 0;
  else return ((VM >> SLOT) & 1u) != 0;
}
// Slot SLOT's matrix for element coordinate `coord` along its axis (element-dependent slots).
template <int SLOT, typename Real>
__device__ __forceinline__ const Real* slot_matrix(const KronHead<Real>& P, uint32_t coord) {
  return P.mats + P.vm[SLOT].off + (int64_t)coord * P.vm[SLOT].stride;
}

// Row i of an N x N matrix at p (16-byte aligned when V > 1).
template <int N, typename Real>
__device__ __forceinline__ void matrix_row(const Real* p, int i, Real (&row)[N]) {
  constexpr int V = Kron3DShape<N, Real>::V;
#pragma unroll
  for (int j = 0; j < N; j += V) {
    Real v[V];
    vldg<Real, V>(p + i * N + j, v);
#pragma unroll
    for (int q = 0; q < V; ++q) row[j + q] = v[q];
  }
}
template <int N, typename Real>
__device__ __forceinline__ void load_matrix(const Real* p, RegMat<N, Real>& A) {
#pragma unroll
  for (int i = 0; i < N; ++i) matrix_row<N>(p, i, A.a[i]);
}

// X <- A X along the first (FIRST) or second plane index, line by line.
template <int N, bool FIRST, typename Real, typename Mat>
__device__ __forceinline__ void lines_inplace(const Mat& A, Real (&X)[N][N]) {
#pragma unroll
  for (int l = 0; l < N; ++l) {
    Real w[N];
#pragma unroll
    for (int j = 0; j < N; ++j) {
      Real s = A(j, 0) * (FIRST ? X[0][l] : X[l][0]);
#pragma unroll
      for (int i = 1; i < N; ++i) s += A(j, i) * (FIRST ? X[i][l] : X[l][i]);
      w[j] = s;
    }
#pragma unroll
    for (int j = 0; j < N; ++j) {
      if constexpr (FIRST) X[j][l] = w[j];
      else X[l][j] = w[j];
    }
  }
}

// The same for a matrix in memory that is too large to hold in registers beside the planes (N >
// 4): two lines at a time, row by row.
template <int N, bool FIRST, typename Real>
__device__ __forceinline__ void lines_inplace_rows(const Real* p, Real (&X)[N][N]) {
#pragma unroll
  for (int l = 0; l < N; l += 2) {
    constexpr int L = 2;
    Real w[L][N];
#pragma unroll
    for (int j = 0; j < N; ++j) {
      Real row[N];
      matrix_row<N>(p, j, row);
#pragma unroll
      for (int k = 0; k < L; ++k) {
        if (l + k >= N) continue;
        const int ll = l + k < N ? l + k : l;
        Real s = row[0] * (FIRST ? X[0][ll] : X[ll][0]);
#pragma unroll
        for (int i = 1; i < N; ++i) s += row[i] * (FIRST ? X[i][ll] : X[ll][i]);
        w[k][j] = s;
      }
    }
#pragma unroll
    for (int k = 0; k < L; ++k) {
      if (l + k >= N) continue;
      const int ll = l + k < N ? l + k : l;
#pragma unroll
      for (int j = 0; j < N; ++j) {
        if constexpr (FIRST) X[j][ll] = w[k][j];
        else X[ll][j] = w[k][j];
      }
    }
  }
}

// X <- A X along the first or second plane index, A in memory at p.
template <int N, bool FIRST, typename Real>
__device__ __forceinline__ void memory_pass(const Real* p, Real (&X)[N][N]) {
  if constexpr (N <= 4) {
    RegMat<N, Real> A;
    load_matrix<N>(p, A);
    lines_inplace<N, FIRST>(A, X);
  } else {
    lines_inplace_rows<N, FIRST>(p, X);
  }
}
// Y <- A X along the second plane index, or Y += with ACC, A in memory at p.  In FP64 the products accumulate
// onto Y in one multiply-add chain per value.  In FP32 a term is summed on its own and then added: the
// chain rounds every product at the size of the whole sum, which made the applies' error up to a
// quarter larger (advection against 64 bits, p = 3 / p = 5: chained 1.03e-7 / 1.19e-7, own sums 0.90e-7 /
// 0.97e-7; 48^3 p = 3 takes 26.6 us instead of 26.2).  In FP64 the two differ by less than 0.2 %.
template <int N, bool ACC, typename Real>
__device__ __forceinline__ void memory_pass_z(const Real* p, const Real (&X)[N][N], Real (&Y)[N][N]) {
  constexpr bool chain = ACC && sizeof(Real) == 8;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    Real row[N];
    matrix_row<N>(p, k, row);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      Real s = chain ? Y[i][k] : row[0] * X[i][0];
#pragma unroll
      for (int r = chain ? 0 : 1; r < N; ++r) s += row[r] * X[i][r];
      Y[i][k] = ACC && !chain ? Y[i][k] + s : s;
    }
  }
}

// X <- (slot SLOT's matrix) X along the first or second plane index.
template <int N, typename Real, int SLOT, bool FIRST, uint32_t VM, typename Block>
__device__ __forceinline__ void kron_pass(const Block& P, uint32_t coord, Real (&X)[N][N]) {
  if (slot_varies<SLOT, VM>(P)) {
    memory_pass<N, FIRST>(slot_matrix<SLOT>(P, coord), X);
  } else {
    lines_inplace<N, FIRST>(ParamMat<N, Real, SLOT, Block>{P}, X);
  }
}

// Y <- (slot SLOT's matrix) X along the second plane index, or Y += with ACC (summed as in memory_pass_z).
template <int N, typename Real, int SLOT, bool ACC, uint32_t VM, typename Block>
__device__ __forceinline__ void kron_pass_z(const Block& P, uint32_t coord, const Real (&X)[N][N],
                                            Real (&Y)[N][N]) {
  [[maybe_unused]] constexpr bool chain = ACC && sizeof(Real) == 8;
  if (slot_varies<SLOT, VM>(P)) {
    memory_pass_z<N, ACC>(slot_matrix<SLOT>(P, coord), X, Y);
  } else {
    const ParamMat<N, Real, SLOT, Block> A{P};
#pragma unroll
    for (int k = 0; k < N; ++k)
#pragma unroll
      for (int i = 0; i < N; ++i) {
        Real s = chain ? Y[i][k] : A(k, 0) * X[i][0];
#pragma unroll
        for (int r = chain ? 0 : 1; r < N; ++r) s += A(k, r) * X[i][r];
        Y[i][k] = ACC && !chain ? Y[i][k] + s : s;
      }
  }
}

// One line: w = (slot SLOT's matrix) v.
template <int N, typename Real, int SLOT, uint32_t VM, typename Block>
__device__ __forceinline__ void kron_line(const Block& P, uint32_t coord, const Real (&v)[N], Real (&w)[N]) {
  if (slot_varies<SLOT, VM>(P)) {
    const Real* p = slot_matrix<SLOT>(P, coord);
#pragma unroll
    for (int j = 0; j < N; ++j) {
      Real row[N];
      matrix_row<N>(p, j, row);
      Real s = row[0] * v[0];
#pragma unroll
      for (int i = 1; i < N; ++i) s += row[i] * v[i];
      w[j] = s;
    }
  } else {
    const ParamMat<N, Real, SLOT, Block> A{P};
#pragma unroll
    for (int j = 0; j < N; ++j) {
      Real s = A(j, 0) * v[0];
#pragma unroll
      for (int i = 1; i < N; ++i) s += A(j, i) * v[i];
      w[j] = s;
    }
  }
}

template <int N, typename Real>
__device__ __forceinline__ void copy_plane(const Real (&U)[N][N], Real (&X)[N][N]) {
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int j = 0; j < N; ++j) X[i][j] = U[i][j];
}
template <int N, typename Real>
__device__ __forceinline__ void scale_plane(Real f, Real (&X)[N][N]) {
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int j = 0; j < N; ++j) X[i][j] *= f;
}

// Layout exchange between the N lanes of an element: X[i][j] held by lane t (plane index t of
// the third axis) becomes Y[i][k] = X_k[i][t].  N = 2 and 4: shfl_xor butterflies on the lane bits;
// at the stage on bit b each lane keeps the column of each pair (j, j|m) whose bit b matches its
// own and trades the other with lane t ^ m.
template <int N, typename Real>
__device__ __forceinline__ void exchange_butterfly(int t, Real (&X)[N][N]) {
#pragma unroll
  for (int b = 0; (1 << b) < N; ++b) {
    const int m = 1 << b;
    const bool hi = (t & m) != 0;
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
      for (int j = 0; j < N; ++j) {
        if (j & m) continue;
        const Real send = hi ? X[i][j] : X[i][j | m];
        const Real recv = __shfl_xor_sync(0xffffffffu, send, m);
        if (hi) X[i][j] = recv;
        else X[i][j | m] = recv;
      }
  }
}

// Plane of an element in layout Z (values [x][y] of plane z = t) from the staged layout, where
// (x, y, z) sits at z * SP + y * N + x: V-wide loads along x.
template <int N, typename Real>
__device__ __forceinline__ void load_plane_z(const Real* ub, int t, bool active, Real (&u)[N][N]) {
  using S = Kron3DShape<N, Real>;
  constexpr int V = S::V;
#pragma unroll
  for (int j = 0; j < N; ++j)
#pragma unroll
    for (int i = 0; i < N; i += V) {
      Real v[V];
      if (active) vload<Real, V>(ub + t * S::SP + N * j + i, v);
#pragma unroll
      for (int q = 0; q < V; ++q) u[i + q][j] = active ? v[q] : Real(0);
    }
}

// Layout exchange through the warp's shared tile: lane t holds X[i][j] = (x=i, y=j, z=t) and
// receives X[i][k] = (x=i, y=t, z=k).  Tile layout [y][z][x].
template <int N, typename Real>
__device__ __forceinline__ void exchange_tile(Real* tile, int le, int t, bool slot, Real (&X)[N][N]) {
  using S = Kron3DShape<N, Real>;
  constexpr int V = S::V;
  Real* b = tile + le * S::TSE;
  if (slot) {
#pragma unroll
    for (int j = 0; j < N; ++j)
#pragma unroll
      for (int i = 0; i < N; i += V) {
        Real v[V];
#pragma unroll
        for (int q = 0; q < V; ++q) v[q] = X[i + q][j];
        vstore<Real, V>(b + j * S::TA + t * N + i, v);
      }
  }
  __syncwarp();
  if (slot) {
#pragma unroll
    for (int k = 0; k < N; ++k)
#pragma unroll
      for (int i = 0; i < N; i += V) {
        Real v[V];
        vload<Real, V>(b + t * S::TA + k * N + i, v);
#pragma unroll
        for (int q = 0; q < V; ++q) X[i + q][k] = v[q];
      }
  }
  __syncwarp();  // the tile is free again
}

// Element coordinates (x fastest).
template <typename Real>
__device__ __forceinline__ void kron_coords(const KronHead<Real>& P, uint32_t e, uint32_t (&c)[3]) {
  uint32_t q;
  P.fdx.divmod(e, q, c[0]);
  P.fdy.divmod(q, c[2], c[1]);
}

// Upwind decision for face (a, s) of element e (cartesianndmesh.hpp:109-198 for the neighbour,
// advectionoperator.hpp:379-386 / 422-428 for the flux):
//   corner: add phi * el * u[slice]              (outflow face, own trace)
//   use_nb: add coef * neighbour trace            (inflow face, or the transposed coupling)
//   use_g:  add coef * g                          (inflow boundary face with inflow value g)
struct FaceDecision {
  bool corner, use_nb, use_g;
  int64_t d;  // neighbour offset
};

template <typename Real>
__device__ __forceinline__ FaceDecision face_decide(const KronHead<Real>& P, int a, int s, const uint32_t (&c)[3],
                                                    int64_t e, Real tsign, Real el_self, Real& phi, Real& coef) {
  FaceDecision f{false, false, false, 0};
  const int64_t n = P.sizes[a];
  const int64_t st = a == 0 ? 1 : (a == 1 ? P.sizes[0] : P.sizes[0] * P.sizes[1]);
  bool interior;
  if (s == 0) {
    interior = c[a] > 0 || P.periodic[a];
    f.d = c[a] > 0 ? -st : (n - 1) * st;
  } else {
    interior = (int64_t)c[a] + 1 < n || P.periodic[a];
    f.d = (int64_t)c[a] + 1 < n ? st : -(n - 1) * st;
  }
  const bool active = interior ? (P.flags & kFaceInt) : (P.flags & kFaceBnd);
  phi = P.phi[a][c[a] * 2 + s];
  coef = Real(0);
  if (!active) return f;
  const bool outflow = phi * tsign * el_self > Real(0);
  f.corner = outflow;
  if (!(P.flags & kTranspose)) {
    if (!outflow) {
      coef = phi * el_self;
      f.use_nb = interior;
      f.use_g = !interior;
    }
  } else if (interior) {
    // transposed coupling: the neighbour's row, taken when its face (1-s) is inflow for it
    const uint32_t cn = s ? ((int64_t)c[a] + 1 == n ? 0 : c[a] + 1) : (c[a] == 0 ? (uint32_t)(n - 1) : c[a] - 1);
    const Real phin = P.phi[a][cn * 2 + (1 - s)];
    const Real eln = P.elem[a] ? P.elem[a][e + f.d] : Real(1);
    if (!(phin * tsign * eln > Real(0))) {
      coef = phin * eln;
      f.use_nb = true;
    }
  }
  return f;
}

template <typename Real>
__device__ __forceinline__ Real tan_sign(const KronHead<Real>& P, int a, const uint32_t (&c)[3]) {
  Real s = Real(1);
#pragma unroll
  for (int k = 0; k < 3; ++k)
    if (k != a) s *= (Real)P.sgn[a][k][c[k]];
  return s;
}

// Face word of an element: 3 bits per face f = 2 axis + side (own trace of an outflow face, the
// neighbour's trace, the inflow value), and bit kFaceWrap + f when that face's neighbour lies
// across a periodic boundary.
enum : uint32_t { kFaceCorner = 1u, kFaceNb = 2u, kFaceG = 4u };
constexpr int kFaceWrap = 18;

template <typename Real>
__device__ __forceinline__ uint32_t face_word(const KronHead<Real>& P, int64_t e, const uint32_t (&c)[3]) {
  uint32_t w = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const Real tsign = tan_sign(P, a, c);
    const Real el = P.elem[a] ? P.elem[a][e] : Real(1);
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      Real phi, coef;
      const FaceDecision f = face_decide(P, a, s, c, e, tsign, el, phi, coef);
      const uint32_t b = (f.corner ? kFaceCorner : 0u) | (f.use_nb ? kFaceNb : 0u) | (f.use_g ? kFaceG : 0u);
      const bool wrap = s == 0 ? c[a] == 0 : (int64_t)c[a] + 1 == P.sizes[a];
      w |= b << (3 * (2 * a + s)) | (wrap ? 1u << (kFaceWrap + 2 * a + s) : 0u);
    }
  }
  return w;
}
// With per-element velocity factors, whose values (and signs) the caller may change between
// applies: the word from the factors' current values.
template <typename Real>
__device__ __noinline__ uint32_t face_word_now(const KronHead<Real>& P, int64_t e) {
  uint32_t c[3];
  kron_coords(P, (uint32_t)e, c);
  return face_word(P, e, c);
}
template <typename Real>
__device__ __forceinline__ uint32_t load_face_word(const KronHead<Real>& P, int64_t e) {
  return P.eflags ? __ldg(P.eflags + e) : face_word_now(P, e);
}
__device__ __forceinline__ uint32_t face_bits(uint32_t w, int a, int s) { return (w >> (3 * (2 * a + s))) & 7u; }
__device__ __forceinline__ bool face_wraps(uint32_t w, int a, int s) {
  return ((w >> (kFaceWrap + 2 * a + s)) & 1u) != 0;
}

// Element offset to the neighbour across face (a, s).
template <typename Real>
__device__ __forceinline__ int64_t face_offset(const KronHead<Real>& P, uint32_t w, int a, int s) {
  const int64_t st = a == 0 ? 1 : (a == 1 ? P.sizes[0] : P.sizes[0] * P.sizes[1]);
  const int64_t d = face_wraps(w, a, s) ? -(P.sizes[a] - 1) * st : st;
  return s ? d : -d;
}
// Coefficient of the neighbour's trace on face (a, s): the element's own phi (forward) or, transposed,
// the neighbour's at its opposite face, times the per-element factor.
template <typename Real>
__device__ __forceinline__ Real face_nb_coef(const KronHead<Real>& P, uint32_t w, int a, int s, uint32_t ca, int64_t e,
                                             Real k_own) {
  if (!(P.flags & kTranspose)) return k_own;
  const uint32_t cn = face_wraps(w, a, s) ? (s ? 0u : (uint32_t)(P.sizes[a] - 1)) : (s ? ca + 1 : ca - 1);
  const Real phin = P.phi[a][cn * 2 + (1 - s)];
  return P.elem[a] ? phin * P.elem[a][e + face_offset(P, w, a, s)] : phin;
}

// One staged neighbour-trace row (N Reals), V-wide.
template <int N, typename Real>
__device__ __forceinline__ void trace_row(const Real* p, Real (&v)[N]) {
  constexpr int V = Kron3DShape<N, Real>::V;
#pragma unroll
  for (int r = 0; r < N; r += V) {
    Real w[V];
    vload<Real, V>(p + r, w);
#pragma unroll
    for (int q = 0; q < V; ++q) v[r + q] = w[q];
  }
}

// Face terms of axis a (0 or 1) added to the D-pass output X of plane z = t (the face slice is along
// the first index for a = 0, the second for a = 1).  own(i, j): the input plane's values;
// nbrow(s, v): this lane's row of the neighbour's trace on its opposite face.  The trace is the
// slice there, or with GL (a basis without nodes on the faces) the plane's lines times the basis
// values P.lf, and a face term goes to every slice with those weights.
template <int N, typename Real, int A, bool GL, typename Own, typename NbRow, typename Block>
__device__ __forceinline__ void plane_faces(const Block& P, uint32_t ca, int64_t e, uint32_t w,
                                            Real (&X)[N][N], Own own, NbRow nbrow) {
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const uint32_t f = face_bits(w, A, s);
    if (!f) continue;
    const int sl = s ? N - 1 : 0;
    Real k = P.phi[A][ca * 2 + s];
    if (P.elem[A]) k *= P.elem[A][e];
    auto add = [&](Real kk, const Real(&v)[N]) {
#pragma unroll
      for (int i = 0; i < N; ++i) {
        if (!GL && i != sl) continue;
        const Real ki = GL ? kk * P.lf[s][i] : kk;
#pragma unroll
        for (int r = 0; r < N; ++r) {
          if constexpr (A == 0) X[i][r] += ki * v[r];
          else X[r][i] += ki * v[r];
        }
      }
    };
    if (f & kFaceCorner) {
      Real v[N];
#pragma unroll
      for (int r = 0; r < N; ++r) {
        if constexpr (GL) {
          v[r] = Real(0);
#pragma unroll
          for (int i = 0; i < N; ++i) v[r] += P.lf[s][i] * (A == 0 ? own(i, r) : own(r, i));
        } else {
          v[r] = A == 0 ? own(sl, r) : own(r, sl);
        }
      }
      add(k, v);
    }
    if (f & (kFaceNb | kFaceG)) {
      Real v[N];
      if (f & kFaceNb) {
        k = face_nb_coef(P, w, A, s, ca, e, k);
        nbrow(s, v);
      } else {
#pragma unroll
        for (int r = 0; r < N; ++r) v[r] = P.g;
      }
      add(k, v);
    }
  }
}

// The z faces' neighbour traces through Tzy: col(s, v) reads column x = t (values y) of the z
// neighbour's opposite slice, put(s, w) stores the result column in place of it.
template <int N, typename Real, uint32_t VM, typename Col, typename Put, typename Block>
__device__ __forceinline__ void z_faces_prepare(const Block& P, const uint32_t (&c)[3], int64_t e,
                                                uint32_t w, Col col, Put put) {
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const uint32_t f = face_bits(w, 2, s);
    if (!(f & (kFaceNb | kFaceG))) continue;
    Real k = P.phi[2][c[2] * 2 + s];
    if (P.elem[2]) k *= P.elem[2][e];
    Real v[N], r[N];
    if (f & kFaceNb) {
      k = face_nb_coef(P, w, 2, s, c[2], e, k);
      col(s, v);
    } else {
#pragma unroll
      for (int y = 0; y < N; ++y) v[y] = P.g;
    }
    kron_line<N, Real, kSlotTZY, VM>(P, c[1], v, r);
#pragma unroll
    for (int y = 0; y < N; ++y) r[y] *= k;
    put(s, r);
  }
}
// Z-face terms added to the accumulator in layout Y: the own trace of an outflow face (X: the z
// term's lines before Dz, already scaled by the element's factor) and row y = t of the prepared
// neighbour traces (row(s, v)) through Tzx.
template <int N, typename Real, uint32_t VM, bool GL, typename Row, typename Block>
__device__ __forceinline__ void z_faces_add(const Block& P, const uint32_t (&c)[3], uint32_t w,
                                            const Real (&X)[N][N], Real (&out)[N][N], Row row) {
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const uint32_t f = face_bits(w, 2, s);
    if (!f) continue;
    const int sl = s ? N - 1 : 0;
    auto add = [&](int i, Real v) {
      if constexpr (GL) {
#pragma unroll
        for (int z = 0; z < N; ++z) out[i][z] += P.lf[s][z] * v;
      } else {
        out[i][sl] += v;
      }
    };
    if (f & kFaceCorner) {
      const Real k = P.phi[2][c[2] * 2 + s];
#pragma unroll
      for (int i = 0; i < N; ++i) {
        if constexpr (GL) {
          Real tr = Real(0);
#pragma unroll
          for (int z = 0; z < N; ++z) tr += P.lf[s][z] * X[i][z];
          add(i, k * tr);
        } else {
          out[i][sl] += k * X[i][sl];
        }
      }
    }
    if (f & (kFaceNb | kFaceG)) {
      Real v[N], r[N];
      row(s, v);
      kron_line<N, Real, kSlotTZX, VM>(P, c[0], v, r);
#pragma unroll
      for (int i = 0; i < N; ++i) add(i, r[i]);
    }
  }
}

template <int CB>
__device__ __forceinline__ void cp_async(void* smem_dst, const void* gsrc) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  if constexpr (CB == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gsrc));
  else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(d), "l"(gsrc), "n"(CB));
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int K>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(K)); }

__device__ __forceinline__ int group_size(int epw, int64_t remaining) {
  return remaining < epw ? (int)remaining : epw;
}

// Copy N contiguous Reals (a trace row) from global to shared memory.
template <int N, typename Real>
__device__ __forceinline__ void copy_row(Real* dst, const Real* src) {
  using S = Kron3DShape<N, Real>;
  constexpr int R = S::RB / (int)sizeof(Real);
#pragma unroll
  for (int i = 0; i < N; i += R) cp_async<S::RB>(dst + i, src + i);
}

// Where x face s of an element finds its neighbour's trace: the adjacent element of the same
// staged group, trace slot 0 (the first face that is not in the group), or global memory.
__device__ __forceinline__ bool x_in_group(uint32_t w, int s, int le, int ne) {
  return !face_wraps(w, 0, s) && (s ? le + 1 < ne : le > 0);
}
__device__ __forceinline__ bool x_slot_taken(uint32_t w, int le, int ne) {  // by face 0
  return (face_bits(w, 0, 0) & kFaceNb) && !x_in_group(w, 0, le, ne);
}

// Stage the DoFs of elements [e0, e0 + ne) into `buf` (padded layout, coalesced) and, for
// advection, the neighbour traces the faces in word w will read (lane t copies row t of each).
template <int N, typename Real>
__device__ __forceinline__ void stage_group(const KronHead<Real>& P, int64_t e0, int ne, Real* buf, int lane,
                                            int le, int t, uint32_t w, bool traces = true) {
  using S = Kron3DShape<N, Real>;
  const int nchunks = ne * S::NNN / S::CR;
  const Real* src = P.x + e0 * S::NNN;
  for (int ch = lane; ch < nchunks; ch += 32) {
    const int d = ch * S::CR;
    const int r = d / S::NNN, o = d - r * S::NNN;
    const int z = o / S::NN, q = o - z * S::NN;
    cp_async<S::CB>(buf + r * S::SE + z * S::SP + q, src + d);
  }
  if (!w || le >= ne || !traces) return;
  const Real* ue = P.x + (e0 + le) * S::NNN;
  Real* tb = buf + S::EPW * S::SE + le * S::TE;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      if (!(face_bits(w, a, s) & kFaceNb)) continue;
      if (a == 0 && (x_in_group(w, s, le, ne) || (s == 1 && x_slot_taken(w, le, ne)))) continue;
      if (a == 1 && s == 1 && (face_bits(w, 1, 0) & kFaceNb)) continue;
      const Real* un = ue + face_offset(P, w, a, s) * S::NNN;
      const int sl = s ? 0 : N - 1;  // the neighbour's opposite slice
      Real* dst = tb + (a == 2 ? 2 + s : a) * S::TS + t * S::TR;
      if (a == 0) {
#pragma unroll
        for (int r = 0; r < N; ++r) cp_async<(int)sizeof(Real)>(dst + r, un + sl + N * r + S::NN * t);
      } else if (a == 1) {
        copy_row<N>(dst, un + N * sl + S::NN * t);
      } else {
        copy_row<N>(dst, un + N * t + S::NN * sl);
      }
    }
}

constexpr int kron_max_warps = 4;  // warps per CTA of kron3d_kernel (128 threads)

// Kernel variants (chosen per operator by the autotuner):
//   STAGES 2: the next group is staged while this one computes; 1: no overlap inside the warp,
//   less shared memory per warp and so more warps per SM
//   SHFL:    layout exchanges by shuffle butterflies (N = 2, 4) instead of the shared tile
//   DOT:     the inner-product epilogue (P.dot_partials; FP64 solvers) is compiled in
//   VM:      the slot mask the kernel is compiled for (kVaryRuntime: read P.vary)
//   GEN:     the general form: with P.gl a basis without nodes on the faces (the neighbours' traces
//            are formed from their whole elements, read from global memory), and P.nextra mass terms
template <int N, typename Real, bool SEP, int STAGES, bool SHFL, bool DOT, uint32_t VM, bool GEN>
__device__ __forceinline__ void kron3d_body(const KronParams<Real, N, GEN>& P) {
  using S = Kron3DShape<N, Real>;
  constexpr int NN = S::NN, NNN = S::NNN, EPW = S::EPW;
  constexpr bool BFLY = SHFL && S::BUTTERFLY;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int le = lane / N, t = lane - le * N;
  Real* wbase = reinterpret_cast<Real*>(smem_raw) + (size_t)warp * S::warp_smem(STAGES, SHFL);
  [[maybe_unused]] Real* tile = wbase + STAGES * S::STAGE;
  const int64_t ngroups = (P.nelem - P.e_begin + EPW - 1) / EPW;
  const int64_t nwarps = (int64_t)gridDim.x * (blockDim.x >> 5);
  const bool adv = P.has_adv != 0;
  const bool slot = le < EPW;
  const bool gl = GEN && P.gl;
  if (P.skip && *P.skip) return;  // a finished solve: nothing to do
  [[maybe_unused]] double dot_acc = 0.0;

  auto first_of = [&](int64_t g) { return P.e_begin + g * EPW; };
  // this lane's face word in group g (0: no element, or no faces)
  auto word_of = [&](int64_t g) -> uint32_t {
    const int64_t e = first_of(g) + le;
    return (adv && slot && g < ngroups && e < P.nelem) ? load_face_word(P, e) : 0u;
  };
  auto exchange = [&](Real(&X)[N][N]) {
    if constexpr (BFLY) exchange_butterfly<N>(t, X);
    else exchange_tile<N>(tile, le, t, slot, X);
  };

  int64_t g = (int64_t)blockIdx.x * (blockDim.x >> 5) + warp;
  // face words: of this group and of the next one to be staged, loaded ahead of its copies
  uint32_t w = word_of(g), w_next = STAGES == 2 ? word_of(g + nwarps) : 0u;
  if constexpr (STAGES == 2) {
    if (g < ngroups) stage_group<N>(P, first_of(g), group_size(EPW, P.nelem - first_of(g)), wbase, lane, le, t, w, !gl);
    cp_async_commit();
  }
  for (int it = 0; g < ngroups; g += nwarps, ++it) {
    Real* buf = wbase + (STAGES == 2 ? (it & 1) * S::STAGE : 0);
    const uint32_t wc = w;
    if constexpr (STAGES == 2) {
      const int64_t gn = g + nwarps;
      if (gn < ngroups)
        stage_group<N>(P, first_of(gn), group_size(EPW, P.nelem - first_of(gn)), wbase + ((it + 1) & 1) * S::STAGE, lane,
                       le, t, w_next, !gl);
      cp_async_commit();
      w = w_next;
      w_next = word_of(gn + nwarps);
      cp_async_wait<1>();
    } else {
      stage_group<N>(P, first_of(g), group_size(EPW, P.nelem - first_of(g)), buf, lane, le, t, wc, !gl);
      cp_async_commit();
      w = word_of(g + nwarps);
      cp_async_wait<0>();
    }
    __syncwarp();
    const int64_t e0 = first_of(g);
    const int ne = group_size(EPW, P.nelem - e0);
    const int64_t e = e0 + le;
    const bool active = slot && le < ne;
    uint32_t c[3] = {0, 0, 0};
    if (active) kron_coords(P, (uint32_t)e, c);
    const Real* ub = buf + (slot ? le : 0) * S::SE;
    Real* tb = buf + EPW * S::SE + (slot ? le : 0) * S::TE;
    // the input plane: held in registers (one shared-memory read for all terms) in the forms whose
    // registers allow it, otherwise read again by each term
    constexpr bool KEEP = N <= 4 && VM != kVaryRuntime && !SEP;
    [[maybe_unused]] Real U[KEEP ? N : 1][KEEP ? N : 1];
    if constexpr (KEEP) load_plane_z<N>(ub, t, active, U);
    auto input = [&](Real(&X)[N][N]) {
      if constexpr (KEEP) copy_plane<N>(U, X);
      else load_plane_z<N>(ub, t, active, X);
    };
    auto own = [&](int i, int j) {
      if constexpr (KEEP) return U[i][j];
      else return ub[t * S::SP + N * j + i];
    };
    Real out[N][N];

    if (adv) {
      if (wc)
        z_faces_prepare<N, Real, VM>(
            P, c, e, wc,
            [&](int s, Real(&v)[N]) {
              if (GEN && gl) {
                const Real* un = P.x + (e + face_offset(P, wc, 2, s)) * NNN + t;
#pragma unroll
                for (int y = 0; y < N; ++y) v[y] = Real(0);
#pragma unroll
                for (int z = 0; z < N; ++z)
#pragma unroll
                  for (int y = 0; y < N; ++y) v[y] += P.lf[1 - s][z] * un[N * y + NN * z];
                return;
              }
#pragma unroll
              for (int y = 0; y < N; ++y) v[y] = tb[(2 + s) * S::TS + y * S::TR + t];
            },
            [&](int s, const Real(&r)[N]) {
#pragma unroll
              for (int y = 0; y < N; ++y) tb[(2 + s) * S::TS + y * S::TR + t] = r[y];
            });
      // ---------------------------------------------------------------- x term
      {
        Real X[N][N];
        input(X);
        if (P.elem[0]) scale_plane<N>(active ? P.elem[0][e] : Real(1), X);
        kron_pass<N, Real, kSlotDX, true, VM>(P, c[0], X);
        if (GEN && gl) {
          if (wc)
            plane_faces<N, Real, 0, true>(P, c[0], e, wc, X, own, [&](int s, Real(&v)[N]) {
              const Real* un = P.x + (e + face_offset(P, wc, 0, s)) * NNN + NN * t;
#pragma unroll
              for (int r = 0; r < N; ++r) {
                v[r] = Real(0);
#pragma unroll
                for (int i = 0; i < N; ++i) v[r] += P.lf[1 - s][i] * un[i + N * r];
              }
            });
        } else if (wc) {
          plane_faces<N, Real, 0, false>(P, c[0], e, wc, X, own, [&](int s, Real(&v)[N]) {
            const int sl = s ? 0 : N - 1;  // the neighbour's opposite slice
            if (x_in_group(wc, s, le, ne)) {
#pragma unroll
              for (int r = 0; r < N; ++r) v[r] = ub[(s ? S::SE : -S::SE) + t * S::SP + sl + N * r];
            } else if (s == 0 || !x_slot_taken(wc, le, ne)) {
              trace_row<N>(tb + t * S::TR, v);
            } else {
              const Real* un = P.x + (e + face_offset(P, wc, 0, s)) * NNN;
#pragma unroll
              for (int r = 0; r < N; ++r) v[r] = un[sl + N * r + NN * t];
            }
          });
        }
        kron_pass<N, Real, kSlotTXY, false, VM>(P, c[1], X);
        exchange(X);
        kron_pass_z<N, Real, kSlotTXZ, false, VM>(P, c[2], X, out);
      }
      // ---------------------------------------------------------------- y term
      {
        Real X[N][N];
        input(X);
        if (P.elem[1]) scale_plane<N>(active ? P.elem[1][e] : Real(1), X);
        kron_pass<N, Real, kSlotDY, false, VM>(P, c[1], X);
        if (GEN && gl) {
          if (wc)
            plane_faces<N, Real, 1, true>(P, c[1], e, wc, X, own, [&](int s, Real(&v)[N]) {
              const Real* un = P.x + (e + face_offset(P, wc, 1, s)) * NNN + NN * t;
#pragma unroll
              for (int r = 0; r < N; ++r) v[r] = Real(0);
#pragma unroll
              for (int y = 0; y < N; ++y)
#pragma unroll
                for (int r = 0; r < N; ++r) v[r] += P.lf[1 - s][y] * un[r + N * y];
            });
        } else if (wc) {
          plane_faces<N, Real, 1, false>(P, c[1], e, wc, X, own, [&](int s, Real(&v)[N]) {
            if (s == 0 || !(face_bits(wc, 1, 0) & kFaceNb)) {
              trace_row<N>(tb + S::TS + t * S::TR, v);
            } else {
              const Real* un = P.x + (e + face_offset(P, wc, 1, s)) * NNN;
#pragma unroll
              for (int r = 0; r < N; ++r) v[r] = un[r + N * (s ? 0 : N - 1) + NN * t];
            }
          });
        }
        kron_pass<N, Real, kSlotTYX, true, VM>(P, c[0], X);
        exchange(X);
        kron_pass_z<N, Real, kSlotTYZ, true, VM>(P, c[2], X, out);
      }
    } else {
#pragma unroll
      for (int i = 0; i < N; ++i)
#pragma unroll
        for (int k = 0; k < N; ++k) out[i][k] = Real(0);
    }
    // ------------------------------------------------ z term (with a merged mass), or the mass term
    if (!GEN || adv || P.nextra == 0) {
      Real X[N][N];
      input(X);
      const Real* ez = adv ? P.elem[2] : P.elem_mass;
      if (ez) scale_plane<N>(active ? ez[e] : Real(1), X);
      kron_pass<N, Real, kSlotTZX, true, VM>(P, c[0], X);
      kron_pass<N, Real, kSlotTZY, false, VM>(P, c[1], X);
      exchange(X);
      kron_pass_z<N, Real, kSlotDZ, true, VM>(P, c[2], X, out);
      if constexpr (BFLY) __syncwarp();  // the z traces' other columns (the tile exchange synchronizes)
      auto z_row = [&](int s, Real(&v)[N]) { trace_row<N>(tb + (2 + s) * S::TS + t * S::TR, v); };
      if (GEN && gl) {
        if (wc) z_faces_add<N, Real, VM, true>(P, c, wc, X, out, z_row);
      } else if (wc) {
        z_faces_add<N, Real, VM, false>(P, c, wc, X, out, z_row);
      }
    }
    if constexpr (GEN) {
      // the mass terms of a density that is a sum of products
      for (int m = 0; m < P.nextra; ++m) {
        auto matrix = [&](int k) { return P.mats + P.extra[m][k].off + (int64_t)c[k] * P.extra[m][k].stride; };
        Real X[N][N];
        input(X);
        if (P.elem_mass) scale_plane<N>(active ? P.elem_mass[e] : Real(1), X);
        memory_pass<N, true>(matrix(0), X);
        memory_pass<N, false>(matrix(1), X);
        exchange(X);
        memory_pass_z<N, true>(matrix(2), X, out);
      }
    }
    if constexpr (SEP) {
      Real X[N][N];
      input(X);
      if (P.elem_mass) scale_plane<N>(active ? P.elem_mass[e] : Real(1), X);
      kron_pass<N, Real, kSlotMX, true, VM>(P, c[0], X);
      kron_pass<N, Real, kSlotMY, false, VM>(P, c[1], X);
      exchange(X);
      kron_pass_z<N, Real, kSlotMD, true, VM>(P, c[2], X, out);
    }
    __syncwarp();  // every lane is done reading the staged input of this group
    if (slot) {    // output staging: the group's DoF slots, staged layout
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
      // coalesced store, in the staging granule
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
          Real o[S::CR];
          vload<Real, S::CR>(dst + d, o);
#pragma unroll
          for (int q = 0; q < S::CR; ++q) v[q] = alpha * v[q] + by * o[q];
        }
        vstore<Real, S::CR>(dst + d, v);
        if constexpr (DOT) {
          Real z[S::CR];
          vldg<Real, S::CR>(P.dot_z + e0 * NNN + d, z);
#pragma unroll
          for (int q = 0; q < S::CR; ++q) dot_acc += (double)v[q] * (double)z[q];
        }
      }
    }
    __syncwarp();  // the buffer is refilled by a later prefetch
  }
  cp_async_wait<0>();
  if constexpr (DOT) {
    // fixed-order sums: lanes (tree), warps (in order), one partial per CTA; entries past the grid
    // are zeroed so a reader sums a fixed count
    __shared__ double wsum[kron_max_warps];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dot_acc += __shfl_down_sync(0xffffffffu, dot_acc, o);
    if (lane == 0) wsum[warp] = dot_acc;
    __syncthreads();
    if (threadIdx.x == 0) {
      double s = 0.0;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += wsum[w];
      P.dot_partials[blockIdx.x] = s;
      for (int i = blockIdx.x + gridDim.x; i < P.dot_count; i += gridDim.x) P.dot_partials[i] = 0.0;
    }
  }
}

// CTAs of 128 threads per SM the register allocation aims at: planes X and out and a few lines
// live at once.
template <int N, typename Real>
constexpr int kron3d_min_ctas() {
  return sizeof(Real) == 8 ? (N <= 4 ? 4 : (N == 5 ? 3 : 2)) : (N <= 4 ? 6 : 4);
}

template <int N, typename Real, bool SEP, int STAGES, bool SHFL, bool DOT = false, uint32_t VM = kVaryRuntime,
          bool GEN = false>
__global__ void __launch_bounds__(128, kron3d_min_ctas<N, Real>())
    kron3d_kernel(const __grid_constant__ KronParams<Real, N, GEN> P) {
  kron3d_body<N, Real, SEP, STAGES, SHFL, DOT, VM, GEN>(P);
}

// Several small operators of one order in one launch (above p = 3): instance blockIdx.y's parameters are an
// entry of the launch's own parameters, so nothing has to be uploaded.  As many as a launch takes (32,764 bytes):
// 10 at N = 5, 7 at N = 6.  Same arithmetic as each operator's own launch (batch.cu says when it pays).
template <int N>
struct KronPack {
  static constexpr int MAX = 32000 / (int)sizeof(KronParams<double, N, false>);
  KronParams<double, N, false> p[MAX];
};
template <int N, bool SEP>
__global__ void __launch_bounds__(128, kron3d_min_ctas<N, double>())
    kron3d_pack_kernel(const __grid_constant__ KronPack<N> A) {
  kron3d_body<N, double, SEP, 1, false, false, kVaryRuntime, false>(A.p[blockIdx.y]);
}

// Face words of every element (P.eflags of later launches), for operators with advection terms:
// words[e] of the forward operator, words[nelem + e] of the transposed one.
template <typename Real>
__global__ void kron_face_words(const KronHead<Real> fwd, const KronHead<Real> tr, uint32_t* words) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < fwd.nelem;
       e += (int64_t)gridDim.x * blockDim.x) {
    uint32_t c[3];
    kron_coords(fwd, (uint32_t)e, c);
    words[e] = face_word(fwd, e, c);
    words[fwd.nelem + e] = face_word(tr, e, c);
  }
}

}  // namespace dgop
