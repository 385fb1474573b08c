// Launchers of the two-pass FP64 kernels of step 2 (step2_f64.cuh) and of the
// Chebyshev transforms (cheb_f64.cuh); false when the length has none.  The instantiations are split over four units
// (step2_f64_a.cu .. _d.cu) by length.
#pragma once
#include <cuda_runtime.h>

#include "layout.cuh"

namespace sb {

// planes y: g.y0 <= y < g.y1; tw: the length's table exp(-2 pi i m / N)
bool f2_zinv(cudaStream_t s, const double2* st, const float2* stf, double2* zb, const Dims& g, const double2* tw,
             const double* alfa, const double* beta);
bool f2_zfwd(cudaStream_t s, const double2* xb, double2* st, const Dims& g, const double2* tw);
bool f2_xpass(cudaStream_t s, const double2* zb, double2* xb, const Dims& g, const double2* tw, const double* dyi,
              double dxi, double dzi, double rot, unsigned long long* cfl, Fringe fr);
// Chebyshev transforms of nfields fields, the arguments of k_cheb; tw: length
// 2 (ny - 1)
bool f2_cheb(cudaStream_t s, const double2* in, size_t in_fs, double2* out, size_t out_fs, const Dims& g, int nfields,
             int inverse, double scale, const double2* tw, int skip_oddball);
// all planes
bool f2_xpass_p(cudaStream_t s, double2* zb, const Dims& g, const double2* tw, double rot, Fringe fr);

}  // namespace sb
