// Launchers of the two-pass transforms of the eddy-viscosity and learned
// models (les_f64.cuh); false when the length (nz for the z kernels, nx for the
// x kernels) has none.  tw: that length's table.
#pragma once
#include <cuda_runtime.h>

#include "les_dyn.cuh"

namespace sb {

// stf: the state under FP32 storage (st unused when set)
bool lf_zinv(cudaStream_t s, const double2* st, const float2* stf, const SgsBufs& B, const SgsGrid& G,
             const double2* tw, const double* alfa, const double* beta, int set, const double2* sf);
bool lf_zfilt(cudaStream_t s, const SgsBufs& B, const SgsGrid& G, const double2* tw);
bool lf_zfwd(cudaStream_t s, const SgsBufs& B, const SgsGrid& G, const double2* tw);
bool lf_xpass1(cudaStream_t s, const SgsBufs& B, const SgsGrid& G, const double2* tw, const double* delta2,
               const double* s2);
bool lf_xpass2(cudaStream_t s, const SgsBufs& B, const SgsGrid& G, const double2* tw, const double* delta2);
bool lf_xinv9(cudaStream_t s, const SgsBufs& B, const SgsGrid& G, const double2* tw, double* out, int f0);
bool lf_tau_x(cudaStream_t s, const SgsBufs& B, const SgsGrid& G, const double2* tw, const double* delta2, double re,
              int ineg, const double* tau_phys);

}  // namespace sb
