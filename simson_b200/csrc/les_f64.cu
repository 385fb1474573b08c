// Launchers of the two-pass transforms of the eddy-viscosity and learned
// models (les_f64.cuh).
#include "les_f64.cuh"
#include "les_f64.h"

namespace sb {

template <class K, class... A>
static void lf_launch(K kernel, dim3 grid, int nt, int sm, cudaStream_t s, A... args) {
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
  kernel<<<grid, nt, sm, s>>>(args...);
}

bool lf_zinv(cudaStream_t s, const double2* st, const float2* stf, const SgsBufs& B, const SgsGrid& G,
             const double2* tw, const double* alfa, const double* beta, int set, const double2* sf) {
  const dim3 grid((G.nx2 + LF_KB - 1) / LF_KB, G.nyp, 9);
  switch (G.nz) {
#define SB_CASE(n)                                                                                     \
  case n:                                                                                              \
    if (stf)                                                                                           \
      lf_launch(k_sgs_zinv2<n, float2>, grid, f2_threads(F2<n, LF_KB>::items), F2<n, LF_KB>::size * 16, s, stf, B, G, tw, alfa, beta, set, sf);  \
    else                                                                                               \
      lf_launch(k_sgs_zinv2<n, double2>, grid, f2_threads(F2<n, LF_KB>::items), F2<n, LF_KB>::size * 16, s, st, B, G, tw, alfa, beta, set, sf);  \
    return true;
    SB_LF_LENGTHS(SB_CASE)
#undef SB_CASE
  }
  return false;
}

bool lf_zfilt(cudaStream_t s, const SgsBufs& B, const SgsGrid& G, const double2* tw) {
  const dim3 grid((G.nx4 + LF_KB - 1) / LF_KB, G.nyp, 21);
  switch (G.nz) {
#define SB_CASE(n) \
  case n:          \
    lf_launch(k_sgs_zfilt2<n>, grid, f2_threads(F2<n, LF_KB>::items), F2<n, LF_KB>::size * 16, s, B, G, tw); \
    return true;
    SB_LF_LENGTHS(SB_CASE)
#undef SB_CASE
  }
  return false;
}

bool lf_zfwd(cudaStream_t s, const SgsBufs& B, const SgsGrid& G, const double2* tw) {
  const dim3 grid((G.nx2 + LF_KB - 1) / LF_KB, G.nyp, 6);
  switch (G.nz) {
#define SB_CASE(n) \
  case n:          \
    lf_launch(k_sgs_zfwd2<n>, grid, f2_threads(F2<n, LF_KB>::items), F2<n, LF_KB>::size * 16, s, B, G, tw); \
    return true;
    SB_LF_LENGTHS(SB_CASE)
#undef SB_CASE
  }
  return false;
}

bool lf_xpass1(cudaStream_t s, const SgsBufs& B, const SgsGrid& G, const double2* tw, const double* delta2,
               const double* s2) {
  const dim3 grid(G.nz, G.nyp);
  switch (G.nx) {
#define SB_CASE(n) \
  case n:          \
    lf_launch(k_sgs_xpass1_2<n>, grid, LF_XT, F2<n, 11, true>::size * 16, s, B, G, tw, delta2, s2); \
    return true;
    SB_LF_LENGTHS(SB_CASE)
#undef SB_CASE
  }
  return false;
}

bool lf_xpass2(cudaStream_t s, const SgsBufs& B, const SgsGrid& G, const double2* tw, const double* delta2) {
  const dim3 grid(G.nz, G.nyp);
  switch (G.nx) {
#define SB_CASE(n) \
  case n:          \
    lf_launch(k_sgs_xpass2_2<n>, grid, LF_XT, F2<n, 11, true>::size * 16, s, B, G, tw, delta2); \
    return true;
    SB_LF_LENGTHS(SB_CASE)
#undef SB_CASE
  }
  return false;
}

bool lf_xinv9(cudaStream_t s, const SgsBufs& B, const SgsGrid& G, const double2* tw, double* out, int f0) {
  const dim3 grid(G.nz, G.nyp);
  switch (G.nx) {
#define SB_CASE(n) \
  case n:          \
    lf_launch(k_sgs_xinv9_2<n>, grid, LF_XT, F2<n, 5, true>::size * 16, s, B, G, tw, out, f0); \
    return true;
    SB_LF_LENGTHS(SB_CASE)
#undef SB_CASE
  }
  return false;
}

bool lf_tau_x(cudaStream_t s, const SgsBufs& B, const SgsGrid& G, const double2* tw, const double* delta2, double re,
              int ineg, const double* tau_phys) {
  const dim3 grid(G.nz, G.nyp);
  switch (G.nx) {
#define SB_CASE(n) \
  case n:          \
    lf_launch(k_sgs_tau_x2<n>, grid, LF_XT, F2<n, 3, true>::size * 16, s, B, G, tw, delta2, re, ineg, tau_phys); \
    return true;
    SB_LF_LENGTHS(SB_CASE)
#undef SB_CASE
  }
  return false;
}

}  // namespace sb
