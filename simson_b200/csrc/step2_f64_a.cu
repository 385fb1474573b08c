// Two-pass FP64 kernels of step 2, lengths SB_F2_LENGTHS_A (fft2.cuh).
#define SB_F2_UNIT a
#define SB_F2_UNIT_LENGTHS SB_F2_LENGTHS_A
#include "step2_f64_unit.cuh"
