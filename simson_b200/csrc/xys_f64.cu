// Launchers of the xy statistics' two-pass sample (xys_f64.cuh).
#include "xys_f64.cuh"
#include "les_f64.h"

namespace sb {

static bool xys_length(int n) {
  switch (n) {
#define SB_CASE(n) case n:
    SB_XYS_LENGTHS(SB_CASE)
#undef SB_CASE
    return true;
  }
  return false;
}

template <class K>
static void xys_smem(K kernel, int bytes) {
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

bool xys_sums2(cudaStream_t s, const double2* st, const float2* stf, const double2* pr, double2* spec, double* part,
               const SgsGrid& G, const double2* twz, const double2* twx, const double* alfa, const double* beta,
               double c) {
  if (!xys_length(G.nx) || !xys_length(G.nz)) return false;
  const dim3 gz((G.nx2 + LF_KB - 1) / LF_KB, G.nyp, pr ? 9 : 8), gx(G.nz, G.nyp);
  switch (G.nz) {
#define SB_CASE(n)                                                                    \
  case n: {                                                                           \
    constexpr int nt = f2_threads(F2<n, LF_KB>::items), sm = F2<n, LF_KB>::size * 16; \
    if (stf) {                                                                        \
      xys_smem(k_xys_z8<n, float2>, sm);                                              \
      k_xys_z8<n, float2><<<gz, nt, sm, s>>>(stf, pr, spec, G, twz, beta);            \
    } else {                                                                          \
      xys_smem(k_xys_z8<n, double2>, sm);                                             \
      k_xys_z8<n, double2><<<gz, nt, sm, s>>>(st, pr, spec, G, twz, beta);            \
    }                                                                                 \
    break;                                                                            \
  }
    SB_XYS_LENGTHS(SB_CASE)
#undef SB_CASE
  }
  switch (G.nx) {
#define SB_CASE(n)                                                              \
  case n:                                                                       \
    if (pr) {                                                                   \
      xys_smem(k_xys_x15<n, true>, Xx<n, true>::smem);                          \
      k_xys_x15<n, true><<<gx, XYS_XT, Xx<n, true>::smem, s>>>(spec, G, twx, alfa);   \
    } else {                                                                    \
      xys_smem(k_xys_x15<n, false>, Xx<n, false>::smem);                        \
      k_xys_x15<n, false><<<gx, XYS_XT, Xx<n, false>::smem, s>>>(spec, G, twx, alfa); \
    }                                                                           \
    break;
    SB_XYS_LENGTHS(SB_CASE)
#undef SB_CASE
  }
  const dim3 gm((G.nx + XYS_MT - 1) / XYS_MT, XYS_GROUPS, G.nyp);
  const double* phys = reinterpret_cast<const double*>(spec);
  if (pr)
    k_xys_moments<true><<<gm, XYS_MT, 0, s>>>(phys, part, G, c);
  else
    k_xys_moments<false><<<gm, XYS_MT, 0, s>>>(phys, part, G, c);
  return true;
}

}  // namespace sb
