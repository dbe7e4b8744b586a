// Kronecker-form DG advection kernel for even dimensions (2D, 4D N <= 5, 6D N <= 3): the element's
// axes split into a fast half (the first H = D / 2) and a slow half, an element of N^D values held
// by B = N^H lanes as
//   layout F: lane = slow index, B values over the fast axes in registers
//   layout S: lane = fast index, B values over the slow axes in registers
// and a term (x)_k A_k runs the half with its own axis first, crosses to the other layout through
// shared memory once and runs the other half: one round trip per term instead of one per group of
// two axes, three of them in the paired form.  Terms of the slow axes end in layout F, are parked
// in shared memory, and the fast axes' terms end in layout S, where consecutive lanes hold
// consecutive values of y.  Face terms are added to the own axis' pass: the own trace from the
// line in registers, the neighbour's from global memory (in layout S consecutive lanes read
// consecutive values).
//
// A warp works alone on 32 / B elements (no CTA barriers).  Each pass loads its matrix with 16-byte
// loads, the same for all lanes of an element, from a table padded for them.  In 2D and 4D the matrices
// that are the same for every element are copied to shared memory once per CTA; the others, and all
// of 6D's, are read from the table through the L1 (us per apply, hybrid / all through the
// L1 / all in shared memory: 6D 8^6 p = 2 - / 5260 / 5962, p = 1 - / 362 / 400; 4D 12x10x8x8 p = 3,
// sheared velocity, 28.0 / - / 30.4, constant velocity 26.2 / 31.1 / 26.6; 2D 144x119 p = 5, velocity
// a product in both axes, 11.7 / - / 15.5; 2D 200^2 p = 7 31.2 / 37 / 31.2).  The next
// elements are copied in (cp.async) once the last term has read its input.
//
// What bounds it: in 6D (N = 3) 36 passes x 81 multiply-adds on 27 of 32 lanes, 2.0 cycles of the FP64
// pipe per DoF and SM, against 1.6 of shared-memory and L1 accesses, with 10 warps per SM (two
// planes of 27 values and a matrix in registers); the grouped kernel it replaces spends 18 round trips
// and a CTA barrier after each.  Measured (us per apply, fastest of the other variants -> this):
// 6D 8^6 p = 2: 6534 -> 5260, p = 1: 734 -> 362; 4D 12x10x8x8 p = 3: 68.7 -> 26.2, 4D 9x8x7x6 p = 4:
// 64.4 -> 37.7; 2D 144x119 p = 5: 26.0 -> 10.3, 2D 1000^2 p = 1: 175.6 -> 53.6, 2D 200^2 p = 7: 102 ->
// 31.2.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "kron_registry.h"
#include "kronnd_kernel.cuh"

namespace dgop {

template <int D, int N>
struct SplitShape {
  static constexpr int H = D / 2;
  static constexpr int B = kpow(N, H);
  static constexpr bool OK = D % 2 == 0 && N >= 2 && B <= 27;
  static constexpr int EPW = B <= 32 ? 32 / B : 1;  // elements per warp
  static constexpr int ND = B * B;
  static constexpr int BP = B | 1;    // row stride: odd, so that both layouts' accesses hit distinct banks
  static constexpr int EP = B * BP;   // element stride
  static constexpr int BUF = EPW * EP;
  static constexpr int REC = 4 * D;   // face coefficients per element
  // shared memory per warp: input, exchange and parked result, face coefficients (Reals), then
  // coordinates and face flags (ints)
  static constexpr int REALS = (3 * BUF + EPW * REC + 3) / 4 * 4;
  static constexpr int SLOTS = (D + 1) * D;  // matrix slots: D terms and the mass term
  static constexpr bool SMEM_MATS = D < 6;   // constant matrices in shared memory
  // bytes of shared memory per warp
  template <typename Real>
  static constexpr int warp_bytes() {
    return (REALS * (int)sizeof(Real) + EPW * 3 * D * 4 + 15) / 16 * 16;
  }
  // per CTA: the matrices that do not depend on the element
  template <typename Real>
  static constexpr int cta_bytes(int matp) {
    return SMEM_MATS ? SLOTS * matp * (int)sizeof(Real) : 0;
  }
};

// Matrix stride in the padded table.
template <int N, typename Real>
constexpr int split_matp() {
  constexpr int v = 16 / (int)sizeof(Real);
  return (N * N + v - 1) / v * v;
}

// CTAs per SM the register allocation aims at (two planes of B values and a matrix are live).
template <int D, int N, typename Real>
constexpr int split_min_ctas() {
  return sizeof(Real) == 4 ? 6 : (N >= 5 ? 4 : (SplitShape<D, N>::B == 27 ? 5 : 6));
}

// Shared memory of a CTA: with SMEM_MATS the constant matrices (slot by slot), then the warps' areas.
template <int D, int N, typename Real>
struct SplitArea {
  using S = SplitShape<D, N>;
  static constexpr int MATP = split_matp<N, Real>();
  const Real* cmat;
  Real *U, *X, *Y, *rec;
  int *ec, *ff;
  __device__ __forceinline__ SplitArea(unsigned char* smem, int warp) {
    cmat = reinterpret_cast<const Real*>(smem);
    unsigned char* w = smem + S::template cta_bytes<Real>(MATP) + (size_t)warp * S::template warp_bytes<Real>();
    U = reinterpret_cast<Real*>(w);
    X = U + S::BUF;
    Y = X + S::BUF;
    rec = Y + S::BUF;
    ec = reinterpret_cast<int*>(U + S::REALS);  // [EPW][D] coordinates
    ff = ec + S::EPW * D;                        // [EPW][2 D] face flags
  }
};

// Constant matrices, by the threads of a CTA (the caller synchronizes).
template <int D, int N, typename Real>
__device__ __forceinline__ void split_matrices(const KronNDParams<Real>& P, unsigned char* smem) {
  using S = SplitShape<D, N>;
  if constexpr (!S::SMEM_MATS) return;
  constexpr int MATP = split_matp<N, Real>();
  Real* cmat = reinterpret_cast<Real*>(smem);
  for (int i = threadIdx.x; i < S::SLOTS * MATP; i += blockDim.x) {
    const int sl = i / MATP, a = sl / D, k = sl - a * D;
    if (P.pvar[a][k] == 0) cmat[i] = P.pmats[(int64_t)P.pidx[a][k] * MATP + (i - sl * MATP)];
  }
}

// Input of elements [e0, e0 + ne) to U (asynchronous copies of this warp, one commit group).
template <int D, int N, typename Real>
__device__ __forceinline__ void split_stage(const KronNDParams<Real>& P, Real* U, int64_t e0, int ne) {
  using S = SplitShape<D, N>;
  const Real* src = P.x + e0 * S::ND;
  for (int i = threadIdx.x & 31; i < ne * S::ND; i += 32) {
    const int row = i / S::B;
    cp_async_value(U + row * S::BP + (i - row * S::B), src + i);  // rows of all elements in turn (EP = B BP)
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// One warp's elements [e0, e0 + ne), whose input is in U or on its way; next() is called once U has
// been read.
template <int D, int N, typename Real, typename Next>
__device__ __forceinline__ void split_elements(const KronNDParams<Real>& P, const SplitArea<D, N, Real>& M, int64_t e0,
                                               int ne, Next next) {
  using S = SplitShape<D, N>;
  constexpr int H = S::H, B = S::B, BP = S::BP, EP = S::EP, EPW = S::EPW, ND = S::ND;
  constexpr int MATP = split_matp<N, Real>(), MV = 16 / (int)sizeof(Real);
  const int lane = threadIdx.x & 31;
  Real *U = M.U, *X = M.X, *Y = M.Y, *rec = M.rec;
  int *ec = M.ec, *ff = M.ff;
  const int le0 = lane / B;
  const bool slot = le0 < EPW;
  const int le = slot ? le0 : 0, t = slot ? lane - le0 * B : 0;
  {
    for (int i = lane; i < EPW * D; i += 32) {
      const int b = i / D, k = i - b * D;
      ec[i] = b < ne ? (int)(((e0 + b) / P.estride[k]) % P.sizes[k]) : 0;
    }
    __syncwarp();
    for (int i = lane; i < EPW * 2 * D; i += 32) {
      const int b = i / (2 * D), f = i - b * (2 * D);
      uint8_t fl = 0;
      if (b < ne) nd_face_record<D>(P, e0 + b, ec + b * D, f, rec + b * S::REC, &fl);
      ff[i] = fl;
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncwarp();
    const bool act = slot && le < ne;
    const int64_t e = e0 + (act ? le : 0);
    const int* c = ec + le * D;
    const Real* r0 = rec + le * S::REC;
    const int* f0 = ff + le * 2 * D;

    Real v[B], acc[B];
    // matrix of slot (a, k) (a == D: the mass term) for this element, in registers
    struct Mat {
      Real a[MATP];
      __device__ __forceinline__ Real operator()(int j, int i) const { return a[j * N + i]; }
    };
    auto matrix = [&](int a, int k) {
      Mat m;
      auto load = [&](auto get) {
#pragma unroll
        for (int q = 0; q < MATP; q += MV) {
          const auto w = get(q);
          m.a[q] = w.x;
          m.a[q + 1] = w.y;
          if constexpr (MV == 4) {
            m.a[q + 2] = w.z;
            m.a[q + 3] = w.w;
          }
        }
      };
      using Vec = std::conditional_t<MV == 2, double2, float4>;
      const int var = P.pvar[a][k];
      if (S::SMEM_MATS && !var) {
        const Real* p = M.cmat + (a * D + k) * MATP;
        load([&](int q) { return *reinterpret_cast<const Vec*>(p + q); });
      } else {
        const Real* p = P.pmats + (int64_t)(P.pidx[a][k] + c[k] * var) * MATP;
        load([&](int q) { return __ldg(reinterpret_cast<const Vec*>(p + q)); });
      }
      return m;
    };
    // v <- A v along axis KK of the half in registers; `end(line's first position, v, w)` may add to w
    auto pass = [&](auto kc, const Mat& m, auto end) {
      constexpr int SK = kpow(N, decltype(kc)::value);
#pragma unroll
      for (int ln = 0; ln < B / N; ++ln) {
        const int p0 = (ln / SK) * SK * N + (ln % SK);
        Real w[N];
#pragma unroll
        for (int j = 0; j < N; ++j) {
          Real s = m(j, 0) * v[p0];
#pragma unroll
          for (int i = 1; i < N; ++i) s += m(j, i) * v[p0 + i * SK];
          w[j] = s;
        }
        end(p0, w);
#pragma unroll
        for (int j = 0; j < N; ++j) v[p0 + j * SK] = w[j];
      }
    };
    auto nothing = [](int, Real(&)[N]) {};

    // The terms of one half's axes: FAST: the first H axes (layout F, then S), else the others
    // (layout S, then F), accumulated in acc.
    auto half = [&](auto fc, bool with_mass) {
      constexpr bool FAST = decltype(fc)::value;
      constexpr int A0 = FAST ? 0 : H, O0 = FAST ? H : 0;  // first axis of this half, of the other
      // value r of this lane: in this half's layout, and in the other
      auto here = [&](int r) { return le * EP + (FAST ? t * BP + r : r * BP + t); };
      auto there = [&](int r) { return le * EP + (FAST ? r * BP + t : t * BP + r); };
#pragma unroll
      for (int r = 0; r < B; ++r) acc[r] = Real(0);
      const int last = with_mass ? H : H - 1;
#pragma unroll 1
      for (int j = 0; j <= last; ++j) {
        const bool mass = j == H;
        const int a = mass ? D : A0 + j;
        if (mass || P.has_adv) {
#pragma unroll
          for (int r = 0; r < B; ++r) v[r] = U[here(r)];
          // (after the last term's input has been read, the next elements may come in)
          if (FAST && j == last) {
            __syncwarp();
            next();
          }
          if (mass && P.elem_mass) {
            const Real f = P.elem_mass[e];
#pragma unroll
            for (int r = 0; r < B; ++r) v[r] *= f;
          }
          static_for<0, H>([&](auto kc) {
            constexpr int k = decltype(kc)::value;
            if (k != j) return;
            constexpr int SK = kpow(N, k), AX = A0 + k;
            const Mat m = matrix(AX, AX);
            const uint32_t fa = (uint32_t)f0[2 * AX], fb = (uint32_t)f0[2 * AX + 1];
            const Real ka = r0[4 * AX], kb = r0[4 * AX + 2];
            const bool ca = fa & 1u, cb = fb & 1u;
            const Real fe = P.elem[AX] ? P.elem[AX][e] : Real(1);
            const bool scaled = P.elem[AX] != nullptr;
            pass(kc, m, [&](int p0, Real(&w)[N]) {
              if (scaled) {
#pragma unroll
                for (int i = 0; i < N; ++i) w[i] *= fe;
              }
              if (ca) w[0] += ka * v[p0];
              if (cb) w[N - 1] += kb * v[p0 + (N - 1) * SK];
            });
            // the neighbours' traces (or the inflow value) on the two slices
#pragma unroll
            for (int s = 0; s < 2; ++s) {
              const uint32_t f = s ? fb : fa;
              if (!(f & 6u)) continue;
              const Real kn = r0[4 * AX + 2 * s + 1];
              const int sl = s ? N - 1 : 0;
              const Real* un = P.x;
              if (f & 2u) {
                const int64_t n = P.sizes[AX];
                const int64_t ca64 = c[AX];
                const int64_t cn = s ? (ca64 + 1 == n ? 0 : ca64 + 1) : (ca64 == 0 ? n - 1 : ca64 - 1);
                un += (e + (cn - ca64) * P.estride[AX]) * ND + (FAST ? t * B : t);
              }
#pragma unroll
              for (int ln = 0; ln < B / N; ++ln) {
                const int p0 = (ln / SK) * SK * N + (ln % SK);
                const int pn = p0 + (N - 1 - sl) * SK;
                const Real nb = (f & 2u) ? __ldg(un + (FAST ? pn : pn * B)) : P.g;
                v[p0 + sl * SK] += kn * nb;
              }
            }
          });
          static_for<0, H>([&](auto kc) {
            constexpr int k = decltype(kc)::value;
            if (k == j) return;
            pass(kc, matrix(a, A0 + k), nothing);
          });
#pragma unroll
          for (int r = 0; r < B; ++r)
            if (slot) X[here(r)] = v[r];
          __syncwarp();
#pragma unroll
          for (int r = 0; r < B; ++r) v[r] = X[there(r)];
          __syncwarp();
          static_for<0, H>([&](auto kc) { pass(kc, matrix(a, O0 + decltype(kc)::value), nothing); });
#pragma unroll
          for (int r = 0; r < B; ++r) acc[r] += v[r];
        }
      }
    };
    const bool sep_mass = P.has_mass && !(P.has_adv && P.mass_merged);
    half(std::integral_constant<bool, false>{}, false);
    if (slot) {
#pragma unroll
      for (int r = 0; r < B; ++r) Y[le * EP + t * BP + r] = acc[r];
    }
    half(std::integral_constant<bool, true>{}, sep_mass);
    __syncwarp();
    if (act) {
      Real* y = P.y + e * ND + t;
#pragma unroll
      for (int r = 0; r < B; ++r) {
        Real o = P.alpha * (acc[r] + Y[le * EP + r * BP + t]);
        if (P.beta_y != Real(0)) o += P.beta_y * y[r * B];
        y[r * B] = o;
      }
    }
    __syncwarp();
  }
}

template <int D, int N, typename Real>
__global__ void __launch_bounds__(kKronSplitThreads, split_min_ctas<D, N, Real>())
    kronnd_split_kernel(const __grid_constant__ KronNDParams<Real> P) {
  using S = SplitShape<D, N>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (P.skip && *P.skip) return;
  const int warp = threadIdx.x >> 5;
  const SplitArea<D, N, Real> M(smem_raw, warp);
  const int64_t ngroups = (P.nelem - P.e_begin + S::EPW - 1) / S::EPW;
  const int64_t nwarps = (int64_t)gridDim.x * (kKronSplitThreads / 32);
  auto stage = [&](int64_t g) {
    if (g >= ngroups) return;
    const int64_t e0 = P.e_begin + g * S::EPW, left = P.nelem - e0;
    split_stage<D, N>(P, M.U, e0, left < S::EPW ? (int)left : S::EPW);
  };
  int64_t g = (int64_t)blockIdx.x * (kKronSplitThreads / 32) + warp;
  stage(g);
  split_matrices<D, N>(P, smem_raw);
  __syncthreads();
  for (; g < ngroups; g += nwarps) {
    const int64_t e0 = P.e_begin + g * S::EPW, left = P.nelem - e0;
    split_elements<D, N>(P, M, e0, left < S::EPW ? (int)left : S::EPW, [&] { stage(g + nwarps); });
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// Many operators in one persistent launch (2D order 1, the smallest elements: an instance of a few
// thousand of them is a launch of a few warps per SM): table[i] holds instance i's parameters, its
// element batches (one per CTA) are the global batches [first[i], first[i + 1]).
template <int D, int N, typename Real>
__global__ void __launch_bounds__(kKronSplitThreads, split_min_ctas<D, N, Real>())
    kronnd_split_batch_kernel(const KronNDParams<Real>* __restrict__ table, const int64_t* __restrict__ first,
                              int count) {
  using S = SplitShape<D, N>;
  constexpr int W = kKronSplitThreads / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5;
  const int64_t total = first[count];
  int have = -1;  // the instance whose constant matrices are in shared memory
  for (int64_t gb = blockIdx.x; gb < total; gb += gridDim.x) {
    int lo = 0, hi = count;  // instance: the last i with first[i] <= gb
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (first[mid] <= gb) lo = mid;
      else hi = mid;
    }
    const KronNDParams<Real>& P = table[lo];
    if (lo != have) {
      __syncthreads();
      split_matrices<D, N>(P, smem_raw);
      __syncthreads();
      have = lo;
    }
    const SplitArea<D, N, Real> M(smem_raw, warp);
    const int64_t e0 = ((gb - first[lo]) * W + warp) * S::EPW, left = P.nelem - e0;
    if (left <= 0) continue;
    const int ne = left < S::EPW ? (int)left : S::EPW;
    split_stage<D, N>(P, M.U, e0, ne);
    split_elements<D, N>(P, M, e0, ne, [] {});
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

}  // namespace dgop
