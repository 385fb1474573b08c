// Dispatch of the two-pass FP64 kernels of step 2 over their units.
#include "step2_f64.h"

namespace sb {

bool f2_zinv_a(cudaStream_t s, const double2* st, const float2* stf, double2* zb, const Dims& g, const double2* tw,
             const double* alfa, const double* beta);
bool f2_zinv_b(cudaStream_t s, const double2* st, const float2* stf, double2* zb, const Dims& g, const double2* tw,
             const double* alfa, const double* beta);
bool f2_zinv_c(cudaStream_t s, const double2* st, const float2* stf, double2* zb, const Dims& g, const double2* tw,
             const double* alfa, const double* beta);
bool f2_zinv_d(cudaStream_t s, const double2* st, const float2* stf, double2* zb, const Dims& g, const double2* tw,
             const double* alfa, const double* beta);
bool f2_zinv(cudaStream_t s, const double2* st, const float2* stf, double2* zb, const Dims& g, const double2* tw,
             const double* alfa, const double* beta) {
  return f2_zinv_a(s, st, stf, zb, g, tw, alfa, beta) ||
         f2_zinv_b(s, st, stf, zb, g, tw, alfa, beta) ||
         f2_zinv_c(s, st, stf, zb, g, tw, alfa, beta) ||
         f2_zinv_d(s, st, stf, zb, g, tw, alfa, beta);
}

bool f2_zfwd_a(cudaStream_t s, const double2* xb, double2* st, const Dims& g, const double2* tw);
bool f2_zfwd_b(cudaStream_t s, const double2* xb, double2* st, const Dims& g, const double2* tw);
bool f2_zfwd_c(cudaStream_t s, const double2* xb, double2* st, const Dims& g, const double2* tw);
bool f2_zfwd_d(cudaStream_t s, const double2* xb, double2* st, const Dims& g, const double2* tw);
bool f2_zfwd(cudaStream_t s, const double2* xb, double2* st, const Dims& g, const double2* tw) {
  return f2_zfwd_a(s, xb, st, g, tw) ||
         f2_zfwd_b(s, xb, st, g, tw) ||
         f2_zfwd_c(s, xb, st, g, tw) ||
         f2_zfwd_d(s, xb, st, g, tw);
}

bool f2_xpass_a(cudaStream_t s, const double2* zb, double2* xb, const Dims& g, const double2* tw, const double* dyi,
              double dxi, double dzi, double rot, unsigned long long* cfl, Fringe fr);
bool f2_xpass_b(cudaStream_t s, const double2* zb, double2* xb, const Dims& g, const double2* tw, const double* dyi,
              double dxi, double dzi, double rot, unsigned long long* cfl, Fringe fr);
bool f2_xpass_c(cudaStream_t s, const double2* zb, double2* xb, const Dims& g, const double2* tw, const double* dyi,
              double dxi, double dzi, double rot, unsigned long long* cfl, Fringe fr);
bool f2_xpass_d(cudaStream_t s, const double2* zb, double2* xb, const Dims& g, const double2* tw, const double* dyi,
              double dxi, double dzi, double rot, unsigned long long* cfl, Fringe fr);
bool f2_xpass(cudaStream_t s, const double2* zb, double2* xb, const Dims& g, const double2* tw, const double* dyi,
              double dxi, double dzi, double rot, unsigned long long* cfl, Fringe fr) {
  return f2_xpass_a(s, zb, xb, g, tw, dyi, dxi, dzi, rot, cfl, fr) ||
         f2_xpass_b(s, zb, xb, g, tw, dyi, dxi, dzi, rot, cfl, fr) ||
         f2_xpass_c(s, zb, xb, g, tw, dyi, dxi, dzi, rot, cfl, fr) ||
         f2_xpass_d(s, zb, xb, g, tw, dyi, dxi, dzi, rot, cfl, fr);
}

bool f2_xpass_p_a(cudaStream_t s, double2* zb, const Dims& g, const double2* tw, double rot, Fringe fr);
bool f2_xpass_p_b(cudaStream_t s, double2* zb, const Dims& g, const double2* tw, double rot, Fringe fr);
bool f2_xpass_p_c(cudaStream_t s, double2* zb, const Dims& g, const double2* tw, double rot, Fringe fr);
bool f2_xpass_p_d(cudaStream_t s, double2* zb, const Dims& g, const double2* tw, double rot, Fringe fr);
bool f2_xpass_p(cudaStream_t s, double2* zb, const Dims& g, const double2* tw, double rot, Fringe fr) {
  return f2_xpass_p_a(s, zb, g, tw, rot, fr) ||
         f2_xpass_p_b(s, zb, g, tw, rot, fr) ||
         f2_xpass_p_c(s, zb, g, tw, rot, fr) ||
         f2_xpass_p_d(s, zb, g, tw, rot, fr);
}

}  // namespace sb
