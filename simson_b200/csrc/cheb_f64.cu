// Launcher of the two-pass FP64 Chebyshev transforms (cheb_f64.cuh).
#include "cheb_f64.cuh"
#include "step2_f64.h"

namespace sb {

bool f2_cheb(cudaStream_t s, const double2* in, size_t in_fs, double2* out, size_t out_fs, const Dims& g, int nfields,
             int inverse, double scale, const double2* tw, int skip_oddball) {
  const dim3 grid((g.p1 - g.p0 + CHB2_PB - 1) / CHB2_PB, nfields);
  switch (2 * (g.nyp - 1)) {
#define SB_CASE(L)                                                                                                  \
  case L: {                                                                                                         \
    constexpr int nt = Chb2<L>::threads, sm = F2<L, CHB2_PB>::size * (int)sizeof(double2);                          \
    cudaFuncSetAttribute(k_cheb2<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);                              \
    k_cheb2<L><<<grid, nt, sm, s>>>(in, in_fs, out, out_fs, g, inverse, scale, tw, skip_oddball);                    \
    return true;                                                                                                    \
  }
    SB_CHB2_LENGTHS(SB_CASE)
#undef SB_CASE
  }
  return false;
}

}  // namespace sb
