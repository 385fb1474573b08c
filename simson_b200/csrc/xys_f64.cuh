// The xy statistics' sample (xys.cuh) with the two-pass register transforms of
// fft2.cuh; k_xys_zinv and k_xys_acc serve the lengths without them.
//
// An x derivative commutes with the z transform, so eight fields need one (u, v,
// w, omega_x, omega_z and the z derivatives of u, v, w) instead of fifteen:
//
//   k_xys_z8       one field per CTA (grid z), inverse z
//   k_xys_x15      per z row: the fifteen rows formed from the eight spectra in
//                  shared memory, inverse x (two real rows per transform), the
//                  physical rows over the row's own place of the fields
//   k_xys_moments  one thread per x point and group of z rows: the moments in
//                  registers, streaming the physical rows
//
// A transforming thread that also kept the 41 or 57 accumulators waited for
// each row's loads in turn (1.3 TB/s); apart, all three are bound by the
// fields' way through memory, 0.25 + 0.7 + 0.48 GB at 192x129x160: 92, 221 and
// 99 us there, against 424 (k_xys_zinv) and 715 (k_xys_acc).
#pragma once
#include "les_f64.cuh"
#include "xys.cuh"

namespace sb {

// spectral field f of k_xys_z8: state slot and whether times i beta; 8: p
template <int N, class V>
__global__ void __launch_bounds__(f2_threads(F2<N, LF_KB>::items))
    k_xys_z8(const V* __restrict__ st, const double2* __restrict__ pr, double2* __restrict__ spec, SgsGrid G,
             const double2* __restrict__ tw, const double* __restrict__ beta) {
  typedef F2<N, LF_KB> P;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* E = reinterpret_cast<double2*>(smem_raw);
  const int y = blockIdx.y, f = blockIdx.z, kx0 = blockIdx.x * LF_KB, t = threadIdx.x;
  const size_t slot = (size_t)G.nyp * G.NP;
  if (t < P::items_a) {
    const int kx = min(kx0 + t % LF_KB, G.nx2 - 1);  // beyond the field: not stored
    const size_t off = (size_t)y * G.NP + kx;
    const double r = f < 5 || f == 8 ? 1.0 : 0.0, c = 1.0 - r;  // r + i c beta
    auto pass = [&](const auto* __restrict__ p) {
      f2_pass_a<N, LF_KB, LF_KB, 1, false>(
          [&](int iz, int, bool) {
            const double2 q = lf_get(p + (size_t)iz * G.nx2);
            const double b = c * __ldg(&beta[iz]);
            return iz == G.zodd ? double2{0.0, 0.0} : double2{r * q.x - b * q.y, r * q.y + b * q.x};
          },
          E, tw, t);
    };
    if (f == 8)
      pass(pr + off);
    else
      pass(st + (size_t)(f < 5 ? f : f - 5) * slot + off);
  }
  __syncthreads();
  if (t < P::items_b) {
    double2* __restrict__ out = spec + ((size_t)f * G.nyp + y) * N * G.nx2 + kx0;
    f2_pass_b<N, LF_KB, LF_KB, 1>(
        [&](int m, int, int, int b, double2 v) {
          if (kx0 + b < G.nx2) out[(size_t)m * G.nx2 + b] = v;
        },
        E, t);
  }
}

// Row f of the statistics from the eight spectra: (r0 + i c0 alpha) q_s0 + r1
// q_s1, packed as s0 + 16 s1 + 256 (r0 + 1) + 1024 (c0 + 1) + 4096 (r1 + 1).  A
// row of one spectrum names it twice: zero times another one would carry that
// one's infinities and NaN into it.
constexpr int xys_row(int s0, int r0, int c0, int s1, int r1) {
  return s0 + 16 * s1 + 256 * (r0 + 1) + 1024 * (c0 + 1) + 4096 * (r1 + 1);
}
__device__ __constant__ const int kXysRow[16] = {
    xys_row(0, 1, 0, 0, 0),    // u
    xys_row(1, 1, 0, 1, 0),    // v
    xys_row(2, 1, 0, 2, 0),    // w
    xys_row(3, 1, 0, 3, 0),    // omega_x
    xys_row(2, 0, -1, 5, 1),   // omega_y = du/dz - dw/dx
    xys_row(4, 1, 0, 4, 0),    // omega_z
    xys_row(0, 0, 1, 0, 0),    // du/dx
    xys_row(1, 0, 1, 4, -1),   // du/dy = dv/dx - omega_z
    xys_row(5, 1, 0, 5, 0),    // du/dz
    xys_row(1, 0, 1, 1, 0),    // dv/dx
    xys_row(0, 0, -1, 7, -1),  // dv/dy = -du/dx - dw/dz
    xys_row(6, 1, 0, 6, 0),    // dv/dz
    xys_row(2, 0, 1, 2, 0),    // dw/dx
    xys_row(3, 1, 0, 6, 1),    // dw/dy = omega_x + dv/dz
    xys_row(7, 1, 0, 7, 0),    // dw/dz
    xys_row(8, 1, 0, 8, 0),    // p
};

constexpr int XYS_XT = 128;  // threads of k_xys_x15

template <int N, bool PRES>
struct Xx {
  typedef F2<N, XYS_NC, true> P;
  static constexpr int ns = PRES ? 9 : 8;
  static constexpr int ld = N / 2 + 1;  // spectra in shared memory, padded
  static constexpr int smem = (P::size + ns * ld) * (int)sizeof(double2);
};

template <int N, bool PRES>
__global__ void __launch_bounds__(XYS_XT) k_xys_x15(double2* spec, SgsGrid G, const double2* __restrict__ tw,
                                                    const double* __restrict__ alfa) {
  typedef F2<N, XYS_NC, true> P;
  constexpr int NS = Xx<N, PRES>::ns, LD = Xx<N, PRES>::ld, NX2 = N / 2, NF = PRES ? 16 : 15;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* E = reinterpret_cast<double2*>(smem_raw);
  double2* S = E + P::size;  // [NS][LD]
  const int m = blockIdx.x, y = blockIdx.y, t = threadIdx.x;
  const size_t fs = (size_t)G.nyp * G.nz * NX2, row = ((size_t)y * G.nz + m) * NX2;
#pragma unroll
  for (int f = 0; f < NS; ++f)
    for (int k = t; k < NX2; k += XYS_XT) S[f * LD + k] = spec[f * fs + row + k];
  __syncthreads();
  for (int i = t; i < P::items_a; i += XYS_XT) {
    const int b = P::column(i, P::R2, XYS_NC);
    const int c0 = kXysRow[2 * b], c1 = kXysRow[2 * b + 1];
    auto value = [&](int c, int k, double al) {
      const double2 p = S[(c & 15) * LD + k], q = S[(c >> 4 & 15) * LD + k];
      const double r0 = (double)((c >> 8 & 3) - 1), a = (double)((c >> 10 & 3) - 1) * al;
      const double r1 = (double)((c >> 12) - 1);
      return double2{r0 * p.x - a * p.y + r1 * q.x, r0 * p.y + a * p.x + r1 * q.y};
    };
    f2_pass_a<N, XYS_NC, XYS_NC, 1, false, true>(
        [&](int k, int, bool) {
          const bool low = k < NX2, high = k > N - NX2;
          const int kk = low ? k : high ? N - k : 0;
          const double al = __ldg(&alfa[kk]);
          double2 p = value(c0, kk, al);
          double2 q = (PRES || b < XYS_NC - 1) ? value(c1, kk, al) : double2{0.0, 0.0};
          if (k == 0) p.y = q.y = 0.0;
          const double2 z = low ? double2{p.x - q.y, p.y + q.x} : double2{p.x + q.y, q.x - p.y};
          return (low || high) ? z : double2{0.0, 0.0};
        },
        E, tw, i);
  }
  __syncthreads();
  for (int i = t; i < P::items_b; i += XYS_XT)
    f2_pass_b<N, XYS_NC, XYS_NC, 1, true>([&](int, int k1, int k2, int b, double2 v) { E[P::at(k1, k2, b)] = v; }, E,
                                          i);
  __syncthreads();
  double* __restrict__ out = reinterpret_cast<double*>(spec) + 2 * row;
  for (int j = t; j < N; j += XYS_XT) {
    const double2* e = E + P::at(j % P::R1, j / P::R1, 0);
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      const double2 z = e[f / 2];
      out[2 * f * fs + j] = (f & 1) ? z.y : z.x;
    }
  }
}

constexpr int XYS_MT = 128;  // x points per CTA of k_xys_moments

template <bool PRES>
__global__ void __launch_bounds__(XYS_MT) k_xys_moments(const double* __restrict__ phys, double* __restrict__ part,
                                                        SgsGrid G, double c) {
  constexpr int NACC = PRES ? XYS_NACC_P : XYS_NACC, NF = PRES ? 16 : 15;
  const int j = blockIdx.x * XYS_MT + threadIdx.x, grp = blockIdx.y, y = blockIdx.z;
  if (j >= G.nx) return;
  const size_t fs = (size_t)G.nyp * G.nz * G.nx;
  const int m0 = (int)((long long)G.nz * grp / XYS_GROUPS), m1 = (int)((long long)G.nz * (grp + 1) / XYS_GROUPS);
  double acc[NACC];
#pragma unroll
  for (int k = 0; k < NACC; ++k) acc[k] = 0.0;
  const double* p = phys + ((size_t)y * G.nz + m0) * G.nx + j;
  for (int m = m0; m < m1; ++m, p += G.nx) {
    double q[16];
    q[15] = 0.0;
#pragma unroll
    for (int f = 0; f < NF; ++f) q[f] = p[f * fs];
    xys_accumulate<PRES>(q, c, acc);
  }
  const size_t plane = (size_t)G.nyp * G.nx;
#pragma unroll
  for (int k = 0; k < NACC; ++k) part[((size_t)grp * XYS_NACC_P + k) * plane + (size_t)y * G.nx + j] = acc[k];
}

// Lengths nx, nz: the multiples of four from 32 to 384 of factors 2, 3, 5.  The
// others with a split (16 to 30, 50, 54, 90, 150, 162, 250, 270) take xys.cuh's
// kernels, each length being four more to build.
#define SB_XYS_LENGTHS(X)                                                                                           \
  X(32) X(36) X(40) X(48) X(60) X(64) X(72) X(80) X(96) X(100) X(108) X(120) X(128) X(144) X(160) X(180) X(192)      \
  X(200) X(216) X(240) X(256) X(288) X(300) X(320) X(324) X(360) X(384)

}  // namespace sb
