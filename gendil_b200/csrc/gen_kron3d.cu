// Instantiations of the 3D Kronecker-form kernel, FP64 and FP32, every variant; compiled once per
// order with -DDGOP_GEN_N=<p + 1>, N = 1..6.
#include "kron3d_diff_kernel.cuh"
#include "kron3d_kernel.cuh"
#include "kron3d_p3_kernel.cuh"
#include "kron3d_tma_kernel.cuh"
#include "kron_registry.h"

#include <algorithm>
#include <type_traits>

#ifndef DGOP_GEN_N
#error "DGOP_GEN_N must be defined"
#endif
#define DGOP_CAT2_(a, b) a##b
#define DGOP_CAT2(a, b) DGOP_CAT2_(a, b)

namespace dgop {

#if DGOP_GEN_N == 1
const char* const kKronVariantNames[kKronVariants] = {"stage2-tile", "stage1-tile", "stage2-shfl",
                                                      "tma1-tile",   "tma2-shfl",   "tma2-tile"};
// (the any-dimension kernel's variants, kronnd_kernel.cuh, named here with the 3D kernel's)
const char* const kKronNDVariantNames[kKronNDVariants] = {"nd-passes", "nd-grouped2", "nd-grouped3", "nd-paired",
                                                          "nd-mass", "nd-split"};
#endif

namespace {
// The one-stage tile variant at N >= 4 (p >= 3) is also compiled for the masks kVaryNone and
// kVarySheared; an operator whose mask is exactly one of them runs that kernel, every other
// operator the run-time-mask kernel (same arithmetic, same results).
template <int N, int STAGES, bool SHFL>
constexpr bool masked_forms() {
  return N >= 4 && STAGES == 1 && !SHFL;
}

// The kernel of a variant: FP64 N = 4 has its own schedule (kron3d_p3_kernel.cuh), and so have (FACT)
// operators with per-element velocity factors.
template <int N, typename Real>
constexpr bool own_schedule() {
  return N == 4 && std::is_same<Real, double>::value;
}
template <int N, typename Real, int STAGES, bool SHFL, bool SEP, bool DOT, uint32_t VM, bool GEN = false, bool FACT = false>
constexpr auto kernel_entry() {
  if constexpr ((own_schedule<N, Real>() && !GEN) || FACT) return &kron3d_p3_kernel<N, Real, SEP, STAGES, SHFL, DOT, VM>;
  else return &kron3d_kernel<N, Real, SEP, STAGES, SHFL, DOT, VM, GEN>;
}

template <int N, typename Real, bool SEP, int STAGES, bool SHFL, bool DOT, bool FACT>
void launch_kron3d_block(const KronParams<Real>& p, dim3 grid, dim3 block, size_t smem, cudaStream_t s) {
  const auto b = kron_block<N, false>(p);
  if constexpr (masked_forms<N, STAGES, SHFL>()) {
    const int mi = kron_mask_index(p);
    if (mi == 0) {
      kernel_entry<N, Real, STAGES, SHFL, SEP, DOT, kVaryNone, false, FACT>()<<<grid, block, smem, s>>>(b);
      return;
    }
    if (mi == 1) {
      kernel_entry<N, Real, STAGES, SHFL, SEP, DOT, kVarySheared, false, FACT>()<<<grid, block, smem, s>>>(b);
      return;
    }
  }
  kernel_entry<N, Real, STAGES, SHFL, SEP, DOT, kVaryRuntime, false, FACT>()<<<grid, block, smem, s>>>(b);
}
// (an operator with advection terms and no face words has per-element velocity factors)
template <int N, typename Real, bool SEP, int STAGES, bool SHFL, bool DOT>
void launch_kron3d_masked(const KronParams<Real>& p, dim3 grid, dim3 block, size_t smem, cudaStream_t s) {
  if constexpr (kron_early_factors(N)) {
    if (p.has_adv && !p.eflags) {
      launch_kron3d_block<N, Real, SEP, STAGES, SHFL, DOT, true>(p, grid, block, smem, s);
      return;
    }
  }
  launch_kron3d_block<N, Real, SEP, STAGES, SHFL, DOT, false>(p, grid, block, smem, s);
}

template <int N, typename Real, int STAGES, bool SHFL>
void launch_kron3d(const KronParams<Real>& p, dim3 grid, dim3 block, size_t smem, cudaStream_t s) {
  const bool sep = p.has_adv && p.has_mass && !p.mass_merged && !p.nextra;
  if (p.general) {
    const auto b = kron_block<N, true>(p);
    if constexpr (std::is_same<Real, double>::value) {
      if (p.dot_partials) {
        if (sep) kron3d_kernel<N, Real, true, STAGES, SHFL, true, kVaryRuntime, true><<<grid, block, smem, s>>>(b);
        else kron3d_kernel<N, Real, false, STAGES, SHFL, true, kVaryRuntime, true><<<grid, block, smem, s>>>(b);
        return;
      }
    }
    if (sep) kron3d_kernel<N, Real, true, STAGES, SHFL, false, kVaryRuntime, true><<<grid, block, smem, s>>>(b);
    else kron3d_kernel<N, Real, false, STAGES, SHFL, false, kVaryRuntime, true><<<grid, block, smem, s>>>(b);
    return;
  }
  if constexpr (std::is_same<Real, double>::value) {
    if (p.dot_partials) {
      if (sep) launch_kron3d_masked<N, Real, true, STAGES, SHFL, true>(p, grid, block, smem, s);
      else launch_kron3d_masked<N, Real, false, STAGES, SHFL, true>(p, grid, block, smem, s);
      return;
    }
  }
  if (sep) launch_kron3d_masked<N, Real, true, STAGES, SHFL, false>(p, grid, block, smem, s);
  else launch_kron3d_masked<N, Real, false, STAGES, SHFL, false>(p, grid, block, smem, s);
}

template <int N, typename Real, int STAGES, bool SHFL, bool SEP, bool DOT, uint32_t VM, bool GEN = false, bool FACT = false>
const void* kernel_of() {
  return reinterpret_cast<const void*>(kernel_entry<N, Real, STAGES, SHFL, SEP, DOT, VM, GEN, FACT>());
}

// The forms for per-element velocity factors: [inner-product epilogue][separate mass term][mask index + 1].
template <int N, typename Real, int STAGES, bool SHFL, bool SEP, bool DOT>
void fill_fact(KronVariant<Real>& v) {
  v.func_fact[DOT][SEP][0] = kernel_of<N, Real, STAGES, SHFL, SEP, DOT, kVaryRuntime, false, true>();
  if constexpr (masked_forms<N, STAGES, SHFL>()) {
    v.func_fact[DOT][SEP][1] = kernel_of<N, Real, STAGES, SHFL, SEP, DOT, kVaryNone, false, true>();
    v.func_fact[DOT][SEP][2] = kernel_of<N, Real, STAGES, SHFL, SEP, DOT, kVarySheared, false, true>();
  }
}

template <int N>
void fill_pack(const KronParams<double>* const* p, int count, void* block) {
  for (int i = 0; i < count; ++i) static_cast<KronPack<N>*>(block)->p[i] = kron_block<N, false>(*p[i]);
}
template <int N>
void launch_pack(const void* block, bool sep, dim3 grid, dim3 threads, size_t smem, cudaStream_t s) {
  const KronPack<N>& a = *static_cast<const KronPack<N>*>(block);
  if (sep) kron3d_pack_kernel<N, true><<<grid, threads, smem, s>>>(a);
  else kron3d_pack_kernel<N, false><<<grid, threads, smem, s>>>(a);
}

template <int N, typename Real, int STAGES, bool SHFL>
void fill_variant(KronVariant<Real>& v) {
  v.launch = &launch_kron3d<N, Real, STAGES, SHFL>;
  v.func = kernel_of<N, Real, STAGES, SHFL, false, false, kVaryRuntime>();
  v.func_sep = kernel_of<N, Real, STAGES, SHFL, true, false, kVaryRuntime>();
  if constexpr (std::is_same<Real, double>::value) {
    v.func_dot[0] = kernel_of<N, Real, STAGES, SHFL, false, true, kVaryRuntime>();
    v.func_dot[1] = kernel_of<N, Real, STAGES, SHFL, true, true, kVaryRuntime>();
  }
  if constexpr (masked_forms<N, STAGES, SHFL>()) {
    v.func_masked[0][0][0] = kernel_of<N, Real, STAGES, SHFL, false, false, kVaryNone>();
    v.func_masked[0][0][1] = kernel_of<N, Real, STAGES, SHFL, true, false, kVaryNone>();
    v.func_masked[1][0][0] = kernel_of<N, Real, STAGES, SHFL, false, false, kVarySheared>();
    v.func_masked[1][0][1] = kernel_of<N, Real, STAGES, SHFL, true, false, kVarySheared>();
    if constexpr (std::is_same<Real, double>::value) {
      v.func_masked[0][1][0] = kernel_of<N, Real, STAGES, SHFL, false, true, kVaryNone>();
      v.func_masked[0][1][1] = kernel_of<N, Real, STAGES, SHFL, true, true, kVaryNone>();
      v.func_masked[1][1][0] = kernel_of<N, Real, STAGES, SHFL, false, true, kVarySheared>();
      v.func_masked[1][1][1] = kernel_of<N, Real, STAGES, SHFL, true, true, kVarySheared>();
    }
  }
  v.func_general[0][0] = kernel_of<N, Real, STAGES, SHFL, false, false, kVaryRuntime, true>();
  v.func_general[0][1] = kernel_of<N, Real, STAGES, SHFL, true, false, kVaryRuntime, true>();
  if constexpr (std::is_same<Real, double>::value) {
    v.func_general[1][0] = kernel_of<N, Real, STAGES, SHFL, false, true, kVaryRuntime, true>();
    v.func_general[1][1] = kernel_of<N, Real, STAGES, SHFL, true, true, kVaryRuntime, true>();
  }
  if constexpr (kron_early_factors(N)) {
    fill_fact<N, Real, STAGES, SHFL, false, false>(v);
    fill_fact<N, Real, STAGES, SHFL, true, false>(v);
    if constexpr (std::is_same<Real, double>::value) {
      fill_fact<N, Real, STAGES, SHFL, false, true>(v);
      fill_fact<N, Real, STAGES, SHFL, true, true>(v);
    }
    v.warp_smem_fact = KronP3Shape<N, Real>::warp_smem(STAGES, SHFL);
  }
  v.warp_smem_general = Kron3DShape<N, Real>::warp_smem(STAGES, SHFL);
  v.warp_smem = own_schedule<N, Real>() ? KronP3Shape<N, Real>::warp_smem(STAGES, SHFL) : v.warp_smem_general;
  v.threads = kKronThreads;
}

// (the bulk-tensor one-stage tile variant has the same compiled masks)
template <bool SEP, int STAGES, bool SHFL, bool DOT>
void launch_tma_masked(const KronTmaParams<double>& p, dim3 grid, dim3 block, size_t smem, cudaStream_t s) {
  if constexpr (STAGES == 1 && !SHFL) {
    const int mi = kron_mask_index(p.k);
    if (mi == 0) {
      kron3d_tma_kernel<SEP, STAGES, SHFL, DOT, kVaryNone><<<grid, block, smem, s>>>(p);
      return;
    }
    if (mi == 1) {
      kron3d_tma_kernel<SEP, STAGES, SHFL, DOT, kVarySheared><<<grid, block, smem, s>>>(p);
      return;
    }
  }
  kron3d_tma_kernel<SEP, STAGES, SHFL, DOT><<<grid, block, smem, s>>>(p);
}

template <int STAGES, bool SHFL>
void launch_tma(const KronTmaParams<double>& p, dim3 grid, dim3 block, size_t smem, cudaStream_t s) {
  const bool sep = p.k.has_adv && p.k.has_mass && !p.k.mass_merged;
  if (p.k.dot_partials) {
    if (sep) launch_tma_masked<true, STAGES, SHFL, true>(p, grid, block, smem, s);
    else launch_tma_masked<false, STAGES, SHFL, true>(p, grid, block, smem, s);
  } else {
    if (sep) launch_tma_masked<true, STAGES, SHFL, false>(p, grid, block, smem, s);
    else launch_tma_masked<false, STAGES, SHFL, false>(p, grid, block, smem, s);
  }
}

template <int STAGES, bool SHFL>
void fill_tma(KronVariant<double>& v) {
  v.launch_tma = &launch_tma<STAGES, SHFL>;
  v.func = reinterpret_cast<const void*>(&kron3d_tma_kernel<false, STAGES, SHFL>);
  v.func_sep = reinterpret_cast<const void*>(&kron3d_tma_kernel<true, STAGES, SHFL>);
  v.func_dot[0] = reinterpret_cast<const void*>(&kron3d_tma_kernel<false, STAGES, SHFL, true>);
  v.func_dot[1] = reinterpret_cast<const void*>(&kron3d_tma_kernel<true, STAGES, SHFL, true>);
  if constexpr (STAGES == 1 && !SHFL) {
    v.func_masked[0][0][0] = reinterpret_cast<const void*>(&kron3d_tma_kernel<false, 1, false, false, kVaryNone>);
    v.func_masked[0][0][1] = reinterpret_cast<const void*>(&kron3d_tma_kernel<true, 1, false, false, kVaryNone>);
    v.func_masked[0][1][0] = reinterpret_cast<const void*>(&kron3d_tma_kernel<false, 1, false, true, kVaryNone>);
    v.func_masked[0][1][1] = reinterpret_cast<const void*>(&kron3d_tma_kernel<true, 1, false, true, kVaryNone>);
    v.func_masked[1][0][0] = reinterpret_cast<const void*>(&kron3d_tma_kernel<false, 1, false, false, kVarySheared>);
    v.func_masked[1][0][1] = reinterpret_cast<const void*>(&kron3d_tma_kernel<true, 1, false, false, kVarySheared>);
    v.func_masked[1][1][0] = reinterpret_cast<const void*>(&kron3d_tma_kernel<false, 1, false, true, kVarySheared>);
    v.func_masked[1][1][1] = reinterpret_cast<const void*>(&kron3d_tma_kernel<true, 1, false, true, kVarySheared>);
  }
  v.warp_smem = kTmaWarps * tma_warp_bytes(STAGES, SHFL) + 1024;  // bytes per CTA, with the alignment slack
  v.threads = kTmaWarps * 32;
}

template <int N, typename Real>
void launch_diff(const Kron3DDiffParams<Real>& p, bool gll, dim3 grid, dim3 block, size_t smem, cudaStream_t s) {
  if constexpr (std::is_same<Real, double>::value) {
    if (p.gout) {
      if (gll) kron3d_diff_kernel<N, Real, true, kDiffGradient><<<grid, block, smem, s>>>(p);
      else kron3d_diff_kernel<N, Real, false, kDiffGradient><<<grid, block, smem, s>>>(p);
      return;
    }
    if (p.dot_partials) {
      if (gll) kron3d_diff_kernel<N, Real, true, kDiffApplyDot><<<grid, block, smem, s>>>(p);
      else kron3d_diff_kernel<N, Real, false, kDiffApplyDot><<<grid, block, smem, s>>>(p);
      return;
    }
  }
  if (gll) kron3d_diff_kernel<N, Real, true, kDiffApply><<<grid, block, smem, s>>>(p);
  else kron3d_diff_kernel<N, Real, false, kDiffApply><<<grid, block, smem, s>>>(p);
}

template <typename Real>
void face_words(const KronParams<Real>& fwd, const KronParams<Real>& tr, uint32_t* words, cudaStream_t s) {
  const int64_t blocks = std::min<int64_t>((fwd.nelem + 255) / 256, 4096);
  kron_face_words<Real><<<(unsigned)blocks, 256, 0, s>>>(fwd, tr, words);
}
template <typename Real>
void tma_words(const KronParams<Real>& p, uint32_t* eflags, uint32_t* gwords, cudaStream_t s) {
  const int64_t groups = (p.nelem + 7) / 8;
  const int64_t blocks = (groups * 32 + 255) / 256;
  kron_tma_words<Real><<<(unsigned)blocks, 256, 0, s>>>(p, eflags, gwords);
}

template <int N, typename Real>
void fill(KronEntry<Real>& d) {
  d.epw = Kron3DShape<N, Real>::EPW;
  // above p = 3 one staging stage: two of them and the exchange tile leave too few warps per SM
  if constexpr (N <= 4) fill_variant<N, Real, 2, false>(d.v[0]);
  fill_variant<N, Real, 1, false>(d.v[1]);
  if constexpr (N > 4 && std::is_same<Real, double>::value) {
    d.v[1].fill_pack = &fill_pack<N>;
    d.v[1].launch_pack = &launch_pack<N>;
    d.v[1].pack_bytes = sizeof(KronPack<N>);
    d.v[1].pack_stride = sizeof(KronParams<double, N, false>);
    d.v[1].func_pack[0] = reinterpret_cast<const void*>(&kron3d_pack_kernel<N, false>);
    d.v[1].func_pack[1] = reinterpret_cast<const void*>(&kron3d_pack_kernel<N, true>);
    d.v[1].pack = KronPack<N>::MAX;
  }
  if constexpr (Kron3DShape<N, Real>::BUTTERFLY) fill_variant<N, Real, 2, true>(d.v[2]);
  d.face_words = &face_words<Real>;
  if constexpr (N >= 2) {
    d.launch_diff = &launch_diff<N, Real>;
    d.func_diff[0][kDiffApply] = reinterpret_cast<const void*>(&kron3d_diff_kernel<N, Real, false, kDiffApply>);
    d.func_diff[1][kDiffApply] = reinterpret_cast<const void*>(&kron3d_diff_kernel<N, Real, true, kDiffApply>);
    if constexpr (std::is_same<Real, double>::value) {
      d.func_diff[0][kDiffApplyDot] = reinterpret_cast<const void*>(&kron3d_diff_kernel<N, Real, false, kDiffApplyDot>);
      d.func_diff[1][kDiffApplyDot] = reinterpret_cast<const void*>(&kron3d_diff_kernel<N, Real, true, kDiffApplyDot>);
      d.func_diff[0][kDiffGradient] = reinterpret_cast<const void*>(&kron3d_diff_kernel<N, Real, false, kDiffGradient>);
      d.func_diff[1][kDiffGradient] = reinterpret_cast<const void*>(&kron3d_diff_kernel<N, Real, true, kDiffGradient>);
    }
    d.diff_warp_smem[0] = Kron3DDiffShape<N, Real>::WARP;
    d.diff_warp_smem[1] = Kron3DDiffShape<N, Real, true>::WARP;
  }
#if DGOP_GEN_N == 4
  if constexpr (std::is_same<Real, double>::value) {
    fill_tma<1, false>(d.v[3]);
    fill_tma<2, true>(d.v[4]);
    fill_tma<2, false>(d.v[5]);
    d.tma_words = &tma_words<Real>;
  }
#endif
}
}  // namespace

void DGOP_CAT2(register_kron3d_n, DGOP_GEN_N)() {
  fill<DGOP_GEN_N, double>(kron3d_slot_f64(DGOP_GEN_N));
  fill<DGOP_GEN_N, float>(kron3d_slot_f32(DGOP_GEN_N));
}

}  // namespace dgop
