// The 3D register kernel's earlier schedule, without the general features: FP64 operators at N = p + 1 =
// 4, and for N <= 4 in both precisions operators with per-element velocity factors.  Same layouts,
// variants and staging as kron3d_kernel.cuh,
//
//   Z: px = Dx u + x-faces ; qx = Txy px ; py = Dy u + y-faces             exchange qx, py -> Y
//   Y: out = Txz qx + Tyx Tyz py ; pz = Dz u + z-faces (mass merged) ; qz = Tzx pz
//                                                                           exchange qz, out -> Z
//   Z: out += Tzy qz ; y = alpha out + beta y
//
// one exchange more than there, but the z neighbours' traces need no passes of their own and the
// face decisions come with the staged record.  At N = 4 in FP64, where the planes are whole 16-byte
// vectors and 128 registers hold what either schedule keeps, this one is the faster: us per apply
// here / there 16.2 / 16.5 (37x26x31 sheared advection), 52.9 / 56.6 (47x48x48, every velocity
// component varying along its own axis), 23.1 / 24.5 (mass, 47x48x48).  In FP32 and at N = 2, 3 the other
// measured faster (FP32 48^3: 31.0 / 26.5; N = 3, 80^3: 168 / 135), but not with velocity factors: their
// values and signs may change between applies, so that the face words the other schedule reads have to
// be made in the kernel, ahead of the copies they decide on, where this one's staging decides each face
// once and keeps its coefficients (implicit system with factors, p = 1, 16x17x15 5.3 / 6.9,
// transposed 72x73x71 43.7 / 51.9; p = 0, 144x145x143 105.7 / 119.4; FP32 p = 3, 36x37x35 16.3 / 19.0).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "kron3d_kernel.cuh"
#include "kron3d_planes.cuh"

namespace dgop {

template <int N, typename Real>
struct KronP3Shape : Kron3DShape<N, Real> {
  using B = Kron3DShape<N, Real>;
  // neighbour traces: one slot per axis (N rows of N), used by the first face of that axis that
  // needs a neighbour trace; a second one on the same axis (rare) is read from global memory
  static constexpr int trace_stride() {
    for (int te = 3 * B::TS; te <= 3 * B::TS + 64; ++te) {
      if ((te * (int)sizeof(Real)) % B::RB || te % B::V) continue;
      if (B::distinct(B::V, [&](int le, int t) { return le * te + t * B::TR; })) return te;
    }
    return 3 * B::TS;
  }
  static constexpr int TE = trace_stride();
  // face record per element: 12 coefficients (axis, side, {corner, neighbour/inflow}) + flag word
  static constexpr int RE = 12 + (16 / (int)sizeof(Real));
  static constexpr int STAGE = B::EPW * (B::SE + TE + RE);  // one pipeline stage: DoFs, traces, records
  static constexpr int warp_smem(int stages, bool shfl) {
    return stages * STAGE + ((shfl && B::BUTTERFLY) ? 0 : ((B::TILE + 3) / 4 * 4));
  }
};

enum TraceSrc { kTraceLocal = 0, kTraceSlot = 1, kTraceGlobal = 2 };

// Apply slot SLOT's matrix (for element coordinate `coord` along its axis) along the first or
// second plane index: constant matrices come from kernel-parameter space.  VM: the slot mask the
// kernel is compiled for (kron.h).
template <int N, typename Real, int SLOT, bool FIRST, uint32_t VM, typename Block>
__device__ __forceinline__ void p3_apply(const Block& P, uint32_t coord, const Real (&X)[N][N],
                                           Real (&Y)[N][N]) {
  bool vary;
  if constexpr (VM == kVaryRuntime) vary = P.vary[SLOT] != 0;
  else vary = ((VM >> SLOT) & 1u) != 0;
  if (vary) {
    RegMat<N, Real> A;
    const Real* p = P.mats + P.vm[SLOT].off + (int64_t)coord * P.vm[SLOT].stride;
    // N x N blocks at offsets that are multiples of the vector width (checked at setup)
    constexpr int V = KronP3Shape<N, Real>::V;
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
      for (int j = 0; j < N; j += V) {
        Real v[V];
        vldg<Real, V>(p + i * N + j, v);
#pragma unroll
        for (int q = 0; q < V; ++q) A.a[i][j + q] = v[q];
      }
    if (FIRST) apply_first<N>(A, X, Y);
    else apply_second<N>(A, X, Y);
  } else {
    ParamMat<N, Real, SLOT, Block> A{P};
    if (FIRST) apply_first<N>(A, X, Y);
    else apply_second<N>(A, X, Y);
  }
}

// Plane of an element in layout Y (values [x][z] of plane y = t) from the staged layout.
template <int N, typename Real>
__device__ __forceinline__ void p3_load_plane_y(const Real* ub, int t, bool active, Real (&u)[N][N]) {
  using S = KronP3Shape<N, Real>;
  constexpr int V = S::V;
#pragma unroll
  for (int k = 0; k < N; ++k)
#pragma unroll
    for (int i = 0; i < N; i += V) {
      Real v[V];
      if (active) vload<Real, V>(ub + k * S::SP + N * t + i, v);
#pragma unroll
      for (int q = 0; q < V; ++q) u[i + q][k] = active ? v[q] : Real(0);
    }
}

// Is the x neighbour on side s the adjacent element of the same staged group?
__device__ __forceinline__ bool p3_x_in_group(int s, int le, int ne, uint32_t cx, int64_t nx) {
  const int rl = le + (s ? 1 : -1);
  return rl >= 0 && rl < ne && (s ? (int64_t)cx + 1 < nx : cx > 0);
}

// Face terms of axis a added to a D-pass output Pm (plane [first][second]; the face slice is along
// the first index when FIRST), from the element's face record (see p3_stage_group).  nbrow(side, src,
// e_nb, v) reads this lane's row of the neighbour trace of that side from the group's staged DoFs
// (x only), the axis' staged trace slot (V-wide), or global memory.
template <int N, typename Real, bool FIRST, typename NbRow>
__device__ __forceinline__ void p3_faces(const KronHead<Real>& P, int a, const uint32_t (&c)[3], int64_t e,
                                           uint32_t flags, const Real* rec, const Real (&U)[N][N], Real (&Pm)[N][N],
                                           NbRow nbrow) {
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const int sl = s ? N - 1 : 0;
    const uint32_t f = (flags >> (5 * (a * 2 + s))) & 31u;
    if (f & kRecCorner) {
      const Real k = rec[(a * 2 + s) * 2];
#pragma unroll
      for (int r = 0; r < N; ++r) {
        if (FIRST) Pm[sl][r] += k * U[sl][r];
        else Pm[r][sl] += k * U[r][sl];
      }
    }
    if (f & (kRecNb | kRecG)) {
      const Real k = rec[(a * 2 + s) * 2 + 1];
      if (f & kRecNb) {
        const int src = (int)(f >> 3);
        const int64_t en = src == kTraceGlobal ? e + neighbour_offset(P, a, s, c[a]) : e;
        Real v[N];
        nbrow(s, src, en, v);
#pragma unroll
        for (int r = 0; r < N; ++r) {
          if (FIRST) Pm[sl][r] += k * v[r];
          else Pm[r][sl] += k * v[r];
        }
      } else {
#pragma unroll
        for (int r = 0; r < N; ++r) {
          if (FIRST) Pm[sl][r] += k * P.g;
          else Pm[r][sl] += k * P.g;
        }
      }
    }
  }
}

// Stage the DoFs of elements [e0, e0 + ne) into `buf` (padded layout, coalesced); for advection,
// also each element's face record and the neighbour traces its faces will read (lane t copies
// row t of each trace).
template <int N, typename Real>
__device__ __forceinline__ void p3_stage_group(const KronHead<Real>& P, int64_t e0, int ne, Real* buf, int lane,
                                            int le, int t, bool adv) {
  using S = KronP3Shape<N, Real>;
  const int nchunks = ne * S::NNN / S::CR;
  const Real* src = P.x + e0 * S::NNN;
  for (int ch = lane; ch < nchunks; ch += 32) {
    const int d = ch * S::CR;
    const int r = d / S::NNN, o = d - r * S::NNN;
    const int z = o / S::NN, w = o - z * S::NN;
    cp_async<S::CB>(buf + r * S::SE + z * S::SP + w, src + d);
  }
  if (!adv || le >= ne) return;
  const int64_t e = e0 + le;
  uint32_t c[3];
  kron_coords(P, (uint32_t)e, c);
  Real* tb = buf + S::EPW * S::SE + le * S::TE;
  Real* rb = buf + S::EPW * (S::SE + S::TE) + le * S::RE;
  uint32_t flags = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const Real tsign = tan_sign(P, a, c);
    const Real el = P.elem[a] ? P.elem[a][e] : Real(1);
    bool slot_taken = false;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      Real phi, coef;
      const FaceDecision f = face_decide(P, a, s, c, e, tsign, el, phi, coef);
      uint32_t bits = 0;
      if (f.corner) bits |= kRecCorner;
      if (f.use_g) bits |= kRecG;
      int src = kTraceLocal;
      if (f.use_nb) {
        bits |= kRecNb;
        if (!(a == 0 && p3_x_in_group(s, le, ne, c[0], P.sizes[0]))) src = slot_taken ? kTraceGlobal : kTraceSlot;
      }
      bits |= (uint32_t)src << 3;
      flags |= bits << (5 * (a * 2 + s));
      if (t == 0) {
        rb[(a * 2 + s) * 2] = phi * el;
        rb[(a * 2 + s) * 2 + 1] = coef;
      }
      if (src != kTraceSlot) continue;  // staged DoFs (x neighbours in the group) or global memory
      slot_taken = true;
      const Real* un = P.x + (e + f.d) * S::NNN;
      const int sl = s ? 0 : N - 1;  // the neighbour's opposite slice
      Real* dst = tb + a * S::TS + t * S::TR;
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
  if (t == 0) *reinterpret_cast<uint32_t*>(rb + 12) = flags;
}

template <int N, typename Real, bool SEP, int STAGES, bool SHFL, bool DOT, uint32_t VM>
__device__ __forceinline__ void kron3d_p3_body(const KronParams<Real, N, false>& P) {
  using S = KronP3Shape<N, Real>;
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
  if (P.skip && *P.skip) return;  // a finished solve: nothing to do
  [[maybe_unused]] double dot_acc = 0.0;

  int64_t g = (int64_t)blockIdx.x * (blockDim.x >> 5) + warp;
  if constexpr (STAGES == 2) {
    if (g < ngroups) p3_stage_group<N>(P, P.e_begin + g * EPW, group_size(EPW, P.nelem - P.e_begin - g * EPW), wbase, lane, le, t, adv);
    cp_async_commit();
  }
  for (int it = 0; g < ngroups; g += nwarps, ++it) {
    Real* buf = wbase + (STAGES == 2 ? (it & 1) * S::STAGE : 0);
    if constexpr (STAGES == 2) {
      const int64_t gn = g + nwarps;
      if (gn < ngroups)
        p3_stage_group<N>(P, P.e_begin + gn * EPW, group_size(EPW, P.nelem - P.e_begin - gn * EPW), wbase + ((it + 1) & 1) * S::STAGE, lane, le,
                       t, adv);
      cp_async_commit();
      cp_async_wait<1>();
    } else {
      p3_stage_group<N>(P, P.e_begin + g * EPW, group_size(EPW, P.nelem - P.e_begin - g * EPW), buf, lane, le, t, adv);
      cp_async_commit();
      cp_async_wait<0>();
    }
    __syncwarp();
    const int64_t e0 = P.e_begin + g * EPW;
    const int ne = group_size(EPW, P.nelem - e0);
    const int64_t e = e0 + le;
    const bool active = slot && le < ne;
    uint32_t c[3] = {0, 0, 0};
    if (active) kron_coords(P, (uint32_t)e, c);
    const Real* ub = buf + (slot ? le : 0) * S::SE;
    const Real* tb = buf + EPW * S::SE + (slot ? le : 0) * S::TE;
    const Real* rec = buf + EPW * (S::SE + S::TE) + (slot ? le : 0) * S::RE;
    const uint32_t fflags = (adv && active) ? *reinterpret_cast<const uint32_t*>(rec + 12) : 0u;
    Real qx[N][N], py[N][N];

    // ------------------------------------------------------------ layout Z (plane z = t)
    if (adv) {
      Real u[N][N];
      load_plane_z<N>(ub, t, active, u);
      {
        Real px[N][N];
        p3_apply<N, Real, kSlotDX, true, VM>(P, c[0], u, px);
        if (P.elem[0]) {
          const Real elx = active ? P.elem[0][e] : Real(1);
#pragma unroll
          for (int i = 0; i < N; ++i)
#pragma unroll
            for (int j = 0; j < N; ++j) px[i][j] *= elx;
        }
        if (active)
          p3_faces<N, Real, true>(P, 0, c, e, fflags, rec, u, px, [&](int s, int src, int64_t en, Real(&v)[N]) {
            const int sl = s ? 0 : N - 1;  // the neighbour's opposite slice
            if (src == kTraceSlot) {
              trace_row<N>(tb + 0 * S::TS + t * S::TR, v);
            } else {
#pragma unroll
              for (int r = 0; r < N; ++r)
                v[r] = src == kTraceLocal ? ub[(s ? 1 : -1) * S::SE + t * S::SP + sl + N * r]
                                          : P.x[en * NNN + sl + N * r + NN * t];
            }
          });
        p3_apply<N, Real, kSlotTXY, false, VM>(P, c[1], px, qx);
      }
      p3_apply<N, Real, kSlotDY, false, VM>(P, c[1], u, py);
      if (P.elem[1]) {
        const Real ely = active ? P.elem[1][e] : Real(1);
#pragma unroll
        for (int i = 0; i < N; ++i)
#pragma unroll
          for (int j = 0; j < N; ++j) py[i][j] *= ely;
      }
      if (active)
        p3_faces<N, Real, false>(P, 1, c, e, fflags, rec, u, py, [&](int s, int src, int64_t en, Real(&v)[N]) {
          if (src == kTraceSlot) {
            trace_row<N>(tb + 1 * S::TS + t * S::TR, v);
          } else {
#pragma unroll
            for (int r = 0; r < N; ++r) v[r] = P.x[en * NNN + r + N * (s ? 0 : N - 1) + NN * t];
          }
        });
      if constexpr (BFLY) {
        exchange_butterfly<N>(t, qx);
        exchange_butterfly<N>(t, py);
      } else {
        exchange_tile_dir<N>(tile, le, t, slot, true, qx);
        exchange_tile_dir<N>(tile, le, t, slot, true, py);
      }
    }

    // ------------------------------------------------------------ layout Y (plane y = t)
    Real out[N][N], qz[N][N];
    [[maybe_unused]] Real qm[N][N];
    {
      // x and y terms first, so their inputs die before u is loaded
      if (adv) {
        p3_apply<N, Real, kSlotTXZ, false, VM>(P, c[2], qx, out);
        p3_apply<N, Real, kSlotTYZ, false, VM>(P, c[2], py, qx);  // qx reused as scratch
        p3_apply<N, Real, kSlotTYX, true, VM>(P, c[0], qx, py);
#pragma unroll
        for (int i = 0; i < N; ++i)
#pragma unroll
          for (int k = 0; k < N; ++k) out[i][k] += py[i][k];
      } else {
#pragma unroll
        for (int i = 0; i < N; ++i)
#pragma unroll
          for (int k = 0; k < N; ++k) out[i][k] = Real(0);
      }
      Real u[N][N], pz[N][N];
      p3_load_plane_y<N>(ub, t, active, u);
      p3_apply<N, Real, kSlotDZ, false, VM>(P, c[2], u, pz);
      if (adv) {
        if (P.elem[2]) {
          const Real elz = active ? P.elem[2][e] : Real(1);
#pragma unroll
          for (int i = 0; i < N; ++i)
#pragma unroll
            for (int k = 0; k < N; ++k) pz[i][k] *= elz;
        }
        if (active)
          p3_faces<N, Real, false>(P, 2, c, e, fflags, rec, u, pz, [&](int s, int src, int64_t en, Real(&v)[N]) {
            if (src == kTraceSlot) {
              trace_row<N>(tb + 2 * S::TS + t * S::TR, v);
            } else {
#pragma unroll
              for (int r = 0; r < N; ++r) v[r] = P.x[en * NNN + r + N * t + NN * (s ? 0 : N - 1)];
            }
          });
      } else if (P.elem_mass) {
        const Real em = active ? P.elem_mass[e] : Real(1);
#pragma unroll
        for (int i = 0; i < N; ++i)
#pragma unroll
          for (int k = 0; k < N; ++k) pz[i][k] *= em;
      }
      p3_apply<N, Real, kSlotTZX, true, VM>(P, c[0], pz, qz);
      if constexpr (SEP) {
        p3_apply<N, Real, kSlotMD, false, VM>(P, c[2], u, pz);
        if (P.elem_mass) {
          const Real em = active ? P.elem_mass[e] : Real(1);
#pragma unroll
          for (int i = 0; i < N; ++i)
#pragma unroll
            for (int k = 0; k < N; ++k) pz[i][k] *= em;
        }
        p3_apply<N, Real, kSlotMX, true, VM>(P, c[0], pz, qm);
      }
    }
    __syncwarp();  // every lane is done reading the staged input of this group
    Real* ob = buf + le * S::SE;  // output staging: the group's DoF slots, staged layout
    if constexpr (BFLY) {
      exchange_butterfly<N>(t, qz);
      exchange_butterfly<N>(t, out);
      if constexpr (SEP) exchange_butterfly<N>(t, qm);
    } else {
      // x and y terms leave in layout Y straight to the output slots; the z term crosses to
      // layout Z through the tile and is added there
      if (slot) {
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
      exchange_tile_dir<N>(tile, le, t, slot, false, qz);
      if constexpr (SEP) exchange_tile_dir<N>(tile, le, t, slot, false, qm);
    }

    // ------------------------------------------------------------ layout Z, output
    p3_apply<N, Real, kSlotTZY, false, VM>(P, c[1], qz, py);
    if constexpr (SEP) {
      p3_apply<N, Real, kSlotMY, false, VM>(P, c[1], qm, qx);
#pragma unroll
      for (int i = 0; i < N; ++i)
#pragma unroll
        for (int j = 0; j < N; ++j) py[i][j] += qx[i][j];
    }
    if (slot) {
      Real* op = ob + t * S::SP;
#pragma unroll
      for (int j = 0; j < N; ++j)
#pragma unroll
        for (int i = 0; i < N; i += S::V) {
          Real v[S::V];
          if constexpr (BFLY) {
#pragma unroll
            for (int q = 0; q < S::V; ++q) v[q] = out[i + q][j] + py[i + q][j];
          } else {
            vload<Real, S::V>(op + N * j + i, v);
#pragma unroll
            for (int q = 0; q < S::V; ++q) v[q] += py[i + q][j];
          }
          vstore<Real, S::V>(op + N * j + i, v);
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
        const int z = o / NN, w = o - z * NN;
        Real v[S::CR];
        vload<Real, S::CR>(buf + r * S::SE + z * S::SP + w, v);
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

// At N = 4 in FP64 the forms without a separate mass term are held to 128 registers, four CTAs per SM (left to itself
// the compiler takes 138 for kVarySheared), but for the double-buffered runtime-mask one, which spills
// under that cap as the forms with a separate mass term do.  Those are left to the compiler (no
// minimum: 134 to 168 registers, three CTAs per SM); a stated minimum of one CTA makes it take up to 192,
// two per SM (system with a density that varies along x, 36x37x35: 33.4 us, without it 28.3).
template <int N, typename Real, bool SEP, int STAGES, bool SHFL, bool DOT = false, uint32_t VM = kVaryRuntime>
__global__ void __launch_bounds__(128, (N == 4 && sizeof(Real) == 8 && !SEP && (VM != kVaryRuntime || STAGES == 1)) ? 4 : 0)
    kron3d_p3_kernel(const __grid_constant__ KronParams<Real, N, false> P) {
  kron3d_p3_body<N, Real, SEP, STAGES, SHFL, DOT, VM>(P);
}

}  // namespace dgop
