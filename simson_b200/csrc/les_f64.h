// Launchers of the two-pass transforms of the eddy-viscosity and learned
// models (les_f64.cuh) and of the xy statistics (xys_f64.cuh); false when the length (nz for the z kernels, nx for the
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

// xy statistics: the group sums of k_xys_acc (with pr, the pressure, its
// entries too); the physical fields stay in spec, [field][y][z][x] doubles, u
// the first.  false unless nx and nz both have two-pass kernels.
bool xys_sums2(cudaStream_t s, const double2* st, const float2* stf, const double2* pr, double2* spec, double* part,
               const SgsGrid& G, const double2* twz, const double2* twx, const double* alfa, const double* beta,
               double c);

}  // namespace sb
