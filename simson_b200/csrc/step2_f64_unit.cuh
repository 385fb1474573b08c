// One unit of the two-pass FP64 kernels of step 2: the launchers for the
// lengths SB_F2_UNIT_LENGTHS, named with the suffix SB_F2_UNIT.
#include "step2_f64.cuh"
#include "step2_f64.h"

#define SB_F2_CAT_(a, b) a##b
#define SB_F2_CAT(a, b) SB_F2_CAT_(a, b)

namespace sb {

template <class K>
static void f2_smem(K kernel, int bytes) {
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}
template <int N, int C, bool NF = false>
constexpr int f2_bytes() {
  return F2<N, C, NF>::size * (int)sizeof(double2);
}

bool SB_F2_CAT(f2_zinv_, SB_F2_UNIT)(cudaStream_t s, const double2* st, const float2* stf, double2* zb, const Dims& g,
                                     const double2* tw, const double* alfa, const double* beta) {
  const dim3 grid((g.nx2 + F2_KB - 1) / F2_KB, g.y1 - g.y0);
  switch (g.nzp) {
#define SB_CASE(n)                                                                                            \
  case n: {                                                                                                   \
    constexpr int nt = f2_threads(F2<n, F2_KB>::items), sm = f2_bytes<n, F2_KB>();                            \
    if (stf) {                                                                                                \
      f2_smem(k_zinv2<n, float2>, sm);                                                                        \
      k_zinv2<n, float2><<<grid, nt, sm, s>>>(stf, zb, g, tw, alfa, beta);                                    \
    } else {                                                                                                  \
      f2_smem(k_zinv2<n, double2>, sm);                                                                       \
      k_zinv2<n, double2><<<grid, nt, sm, s>>>(st, zb, g, tw, alfa, beta);                                    \
    }                                                                                                         \
    return true;                                                                                              \
  }
    SB_F2_UNIT_LENGTHS(SB_CASE)
#undef SB_CASE
  }
  return false;
}

bool SB_F2_CAT(f2_zfwd_, SB_F2_UNIT)(cudaStream_t s, const double2* xb, double2* st, const Dims& g,
                                     const double2* tw) {
  const dim3 grid((g.nx2 + F2_KB - 1) / F2_KB, g.y1 - g.y0);
  switch (g.nzp) {
#define SB_CASE(n)                                                                 \
  case n: {                                                                        \
    constexpr int nt = f2_threads(F2<n, F2_KB>::items), sm = f2_bytes<n, F2_KB>(); \
    f2_smem(k_zfwd2<n>, sm);                                                       \
    k_zfwd2<n><<<grid, nt, sm, s>>>(xb, st, g, tw);                                \
    return true;                                                                   \
  }
    SB_F2_UNIT_LENGTHS(SB_CASE)
#undef SB_CASE
  }
  return false;
}

bool SB_F2_CAT(f2_xpass_, SB_F2_UNIT)(cudaStream_t s, const double2* zb, double2* xb, const Dims& g, const double2* tw,
                                      const double* dyi, double dxi, double dzi, double rot, unsigned long long* cfl,
                                      Fringe fr) {
  const dim3 grid((g.nzp + F2_RB - 1) / F2_RB, g.y1 - g.y0);
  switch (g.nxp) {
#define SB_CASE(n)                                                                         \
  case n: {                                                                                \
    constexpr int nt = f2_threads(F2<n, 3 * F2_RB>::items), sm = f2_bytes<n, 3 * F2_RB, true>(); \
    f2_smem(k_xpass2<n>, sm);                                                              \
    k_xpass2<n><<<grid, nt, sm, s>>>(zb, xb, g, tw, dyi, dxi, dzi, rot, cfl, fr);          \
    return true;                                                                           \
  }
    SB_F2_UNIT_LENGTHS(SB_CASE)
#undef SB_CASE
  }
  return false;
}

bool SB_F2_CAT(f2_xpass_p_, SB_F2_UNIT)(cudaStream_t s, double2* zb, const Dims& g, const double2* tw, double rot,
                                        Fringe fr) {
  const dim3 grid((g.nzp + F2_RB - 1) / F2_RB, g.nyp);
  switch (g.nxp) {
#define SB_CASE(n)                                                                         \
  case n: {                                                                                \
    constexpr int nt = f2_threads(F2<n, 3 * F2_RB>::items), sm = f2_bytes<n, 3 * F2_RB, true>(); \
    f2_smem(k_xpass_p2<n>, sm);                                                            \
    k_xpass_p2<n><<<grid, nt, sm, s>>>(zb, g, tw, rot, fr);                                \
    return true;                                                                           \
  }
    SB_F2_UNIT_LENGTHS(SB_CASE)
#undef SB_CASE
  }
  return false;
}

}  // namespace sb
