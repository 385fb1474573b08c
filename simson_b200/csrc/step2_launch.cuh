// Launch helpers of the step-2 kernels: transform lengths with compile-time
// plans get their own instantiations (fixed_threads threads per CTA), any
// other length the runtime plan.  Shared by the FP64 unit (simson.cu) and the
// mixed-precision unit (mixed.cu), each instantiating its own types.
#pragma once
#include <cuda_runtime.h>

#include "fft.cuh"
#include "layout.cuh"
#include "smem.h"
#include "step2.cuh"

namespace sb {

// threads per CTA of the runtime-plan FFT kernels
constexpr int SB_FFT_THREADS = 256;

// FP32 transform lengths with compile-time FFT plans (fft.cuh cfft): 3/2 of
// the even products of 2, 3 and 5 that grids are made of, up to 384; any other
// length takes the runtime plan, and so do all FP64 ones (those of
// step2_f64.cuh never come here).  Same radices, twiddles and butterflies, so
// the same results to the last bit.
#define SB_FIXED_LENGTHS(X)                                                                                          \
  X(24) X(36) X(48) X(54) X(60) X(72) X(75) X(81) X(90) X(96) X(108) X(120) X(135) X(144) X(150) X(162) X(180)       \
  X(192) X(216) X(225) X(240) X(270) X(288) X(300) X(324) X(360) X(375) X(384) X(405) X(432) X(450) X(480) X(486)    \
  X(540) X(576)

// threads per CTA for B columns, Q per work item, of an N-point compile-time
// transform: one item per thread in the widest pass (halved while above 512),
// a multiple of 32
constexpr int fixed_threads(int n, int b, int q = 1) {
  int items = cplan_max_nb(n) * b / q;
  while (items > 512) items = (items + 1) / 2;
  return ((items + 31) / 32) * 32;
}

// the runtime plan's instance serves every other length, the others one each
template <int N, class K>
inline void smem_limit(K kernel, size_t smem) {
  if constexpr (N > 0)
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  else
    smem_max(kernel);
}

template <class T, int KB, class S, int N, int NT>
inline void zinv_n(dim3 grid, size_t smem, cudaStream_t st, const typename C2<S>::type* in,
                   typename C2<T>::type* zb, const Dims& g, const FFTPlan& plan, const typename C2<T>::type* tw,
                   const double* alfa, const double* beta, int drop) {
  smem_limit<N>(k_zinv<T, KB, S, N, NT>, smem);
  k_zinv<T, KB, S, N, NT><<<grid, NT, smem, st>>>(in, zb, g, plan, tw, alfa, beta, drop);
}
template <class T, int KB, class S>
inline void launch_zinv(dim3 grid, size_t smem, cudaStream_t st, const typename C2<S>::type* in,
                        typename C2<T>::type* zb, const Dims& g, const FFTPlan& plan,
                        const typename C2<T>::type* tw, const double* alfa, const double* beta, int drop) {
  switch (sizeof(T) == 8 ? 0 : g.nzp) {
#define SB_CASE(n)                                                                                       \
  case n:                                                                                                \
    if constexpr (sizeof(T) == 4)                                                                        \
      zinv_n<T, KB, S, n, fixed_threads(n, KB)>(grid, smem, st, in, zb, g, plan, tw, alfa, beta, drop);  \
    return;
    SB_FIXED_LENGTHS(SB_CASE)
#undef SB_CASE
    default:
      zinv_n<T, KB, S, 0, SB_FFT_THREADS>(grid, smem, st, in, zb, g, plan, tw, alfa, beta, drop);
  }
}

template <class T, int KB, class S, int N, int NT>
inline void zfwd_n(dim3 grid, size_t smem, cudaStream_t st, const typename C2<T>::type* xb,
                   typename C2<S>::type* out, const Dims& g, const FFTPlan& plan, const typename C2<T>::type* tw,
                   const double* mean, double rot) {
  smem_limit<N>(k_zfwd<T, KB, S, N, NT>, smem);
  k_zfwd<T, KB, S, N, NT><<<grid, NT, smem, st>>>(xb, out, g, plan, tw, mean, rot);
}
template <class T, int KB, class S>
inline void launch_zfwd(dim3 grid, size_t smem, cudaStream_t st, const typename C2<T>::type* xb,
                        typename C2<S>::type* out, const Dims& g, const FFTPlan& plan,
                        const typename C2<T>::type* tw, const double* mean, double rot) {
  switch (sizeof(T) == 8 ? 0 : g.nzp) {
#define SB_CASE(n)                                                                                \
  case n:                                                                                         \
    if constexpr (sizeof(T) == 4)                                                                 \
      zfwd_n<T, KB, S, n, fixed_threads(n, KB)>(grid, smem, st, xb, out, g, plan, tw, mean, rot); \
    return;
    SB_FIXED_LENGTHS(SB_CASE)
#undef SB_CASE
    default:
      zfwd_n<T, KB, S, 0, SB_FFT_THREADS>(grid, smem, st, xb, out, g, plan, tw, mean, rot);
  }
}

template <class T, int RB, int N, int NT>
inline void xpass_n(dim3 grid, size_t smem, cudaStream_t st, const typename C2<T>::type* zb,
                    typename C2<T>::type* xb, const Dims& g, const FFTPlan& plan, const typename C2<T>::type* tw,
                    const double* dyi, double dxi, double dzi, double rot, unsigned long long* cfl,
                    const double* mean, Fringe fr) {
  smem_limit<N>(k_xpass<T, RB, N, NT>, smem);
#ifdef SB_XPASS_CARVEOUT
  cudaFuncSetAttribute(k_xpass<T, RB, N, NT>, cudaFuncAttributePreferredSharedMemoryCarveout, SB_XPASS_CARVEOUT);
#endif
  k_xpass<T, RB, N, NT><<<grid, NT, smem, st>>>(zb, xb, g, plan, tw, dyi, dxi, dzi, rot, cfl, mean, fr);
}
template <class T, int RB, int NT0>
inline void launch_xpass(dim3 grid, size_t smem, cudaStream_t st, const typename C2<T>::type* zb,
                         typename C2<T>::type* xb, const Dims& g, const FFTPlan& plan,
                         const typename C2<T>::type* tw, const double* dyi, double dxi, double dzi, double rot,
                         unsigned long long* cfl, const double* mean, Fringe fr) {
  switch (sizeof(T) == 8 ? 0 : g.nxp) {
#define SB_CASE(n)                                                                                                \
  case n:                                                                                                         \
    if constexpr (sizeof(T) == 4)                                                                                 \
      xpass_n<T, RB, n, fixed_threads(n, 3 * RB, fft_cols<T, 3 * RB, n>())>(grid, smem, st, zb, xb, g, plan, tw,   \
                                                                            dyi, dxi, dzi, rot, cfl, mean, fr);    \
    return;
    SB_FIXED_LENGTHS(SB_CASE)
#undef SB_CASE
    default:
      xpass_n<T, RB, 0, NT0>(grid, smem, st, zb, xb, g, plan, tw, dyi, dxi, dzi, rot, cfl, mean, fr);
  }
}

}  // namespace sb
