// Launchers of the chunked pencil kernel (pencil_chunk.cu, pencil_chunk.cuh).
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "layout.cuh"
#include "press.cuh"
#include "step3.cuh"

namespace sb {

// whether ny is within the kernel's range
int pencil_chunk_fits(int ny);
// the lam-independent row factors, for the rows argument below
std::vector<double2> pencil_chunk_table(int ny);
// eliminated lower coefficients of (D^2 - (k^2 + shift)), [nyp][(nz/2 + 1) nx/2]
void pencil_tau_coef(cudaStream_t s, double* out, const Dims& g, const double* alfa, const double* beta, double shift);
// every pencil of this context's range but kx = kz = 0 and the oddball plane;
// cl, cv: pencil_tau_coef with shift 2 Re/(a_n + b_n) and 0; mean: kx = kz = 0
// in the same launch, or null
bool pencil_chunk(cudaStream_t s, const PencilBufs& B, const Dims& g, const double* alfa, const double* beta,
                  double re, RKc rk, const double* cl, const double* cv, const double2* rows, const MeanArgs* mean);

// the pressure's pencils but kx = kz = 0 (k_press_mean does that one)
bool press_chunk(cudaStream_t s, const PressArgs& P, const Dims& g, const double* cv, const double2* rows);

}  // namespace sb
