// The chunked pencil kernel of step 3 (pencil_chunk.cuh), in a unit of its own
// built with fused multiply-adds: its sums run in another order than the
// reference's in any case, and are checked against the thread-per-pencil
// kernel and at 64 bits, not bit for bit.
#include "pencil_chunk.h"

#include "pencil_chunk.cuh"

namespace sb {

int pencil_chunk_fits(int ny) { return pencil_chunk_rows(ny) > 0; }

std::vector<double2> pencil_chunk_table(int ny) {
  std::vector<double2> t;
  pc_row_table(ny, t);
  return t;
}

void pencil_tau_coef(cudaStream_t s, double* out, const Dims& g, const double* alfa, const double* beta, double shift) {
  const int items = 2 * (g.nz / 2 + 1) * g.nx2;
  k_tau_coef<<<(items + 127) / 128, 128, 0, s>>>(out, g, alfa, beta, shift);
}

bool pencil_chunk(cudaStream_t s, const PencilBufs& B, const Dims& g, const double* alfa, const double* beta,
                  double re, RKc rk, const double* cl, const double* cv, const double2* rows, const MeanArgs* mean) {
  return launch_pencil_chunk(s, B, g, alfa, beta, re, rk, cl, cv, rows, mean);
}

bool press_chunk(cudaStream_t s, const PressArgs& P, const Dims& g, const double* cv, const double2* rows) {
  return launch_press_chunk(s, P, g, cv, rows);
}

}  // namespace sb
