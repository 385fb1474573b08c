// The transforms of the eddy-viscosity and learned models (les_dyn.cuh) on the
// nx x nz grid with the two-pass register transforms of fft2.cuh: the same
// fields, products and arrays as the kernels there, which serve the lengths
// without a two-pass kernel.  One field per CTA (grid z) where those loop over
// the fields: at 64x97x64 a loop of 21 transforms pairs in 388 CTAs left most
// of the chip waiting on one CTA's passes.
#pragma once
#include "fft2.cuh"
#include "les_dyn.cuh"

namespace sb {

constexpr int LF_KB = 8;  // kx columns per CTA of the z transforms

template <class V>
__device__ __forceinline__ double2 lf_get(const V* __restrict__ p) {
  const V q = *p;
  return double2{(double)q.x, (double)q.y};
}

// The spectral fields of sgs_spec_field as one form without branches,
//   (r0 + i c0) q_s0 + (r1 + i c1) q_s1,  c = ca alpha + cb beta
// (a field of one slot repeats it with zero factors): set 0 u, v, w and S_11
// S_12 S_13 S_22 S_23 S_33, set 1 the nine gradients.
struct LfField {
  int s0, s1;
  double r0, r1, a0, a1, b0, b1;  // a: ca alpha, b: cb
  __device__ __forceinline__ LfField(int f, int set, double alpha) {
    r0 = r1 = a0 = a1 = b0 = b1 = 0.0;
    s0 = 0;
    if (set == 0 && f < 3) {  // u, v, w
      s0 = s1 = f;
      r0 = 1.0;
      return;
    }
    if (set == 0 && f >= 4 && f != 6 && f != 8) {
      if (f == 4) { s0 = 1; a0 = alpha; s1 = 4; r1 = -.5; }             // S_12 = dv/dx - omega_z / 2
      if (f == 5) { s0 = 2; a0 = .5 * alpha; s1 = 0; b1 = .5; }         // S_13
      if (f == 7) { s0 = 1; b0 = 1.0; s1 = 3; r1 = .5; }                // S_23 = dv/dz + omega_x / 2
      return;
    }
    const int k = set == 0 ? (f == 3 ? 0 : f == 6 ? 4 : 8) : f;          // du_i/dx_j, i-major
    if (k == 4) { a0 = -alpha; s1 = 2; b1 = -1.0; return; }              // dv/dy = -du/dx - dw/dz
    s0 = s1 = k / 3;
    if (k % 3 == 0) a0 = alpha;
    if (k % 3 == 2) b0 = 1.0;
    if (k == 1) { s0 = 1; a0 = alpha; s1 = 4; r1 = -1.0; }               // du/dy = dv/dx - omega_z
    if (k == 7) { s0 = 1; b0 = 1.0; s1 = 3; r1 = 1.0; }                  // dw/dy = dv/dz + omega_x
  }
  __device__ __forceinline__ double2 operator()(double2 p, double2 q, double beta, bool zero) const {
    const double c0 = fma_(b0, beta, a0), c1 = fma_(b1, beta, a1);
    const double x = r0 * p.x - c0 * p.y + (r1 * q.x - c1 * q.y);
    const double y = r0 * p.y + c0 * p.x + (r1 * q.y + c1 * q.x);
    return double2{zero ? 0.0 : x, zero ? 0.0 : y};
  }
};

// field f of the set (sgs_spec_field) at every kz of eight kx columns, inverse z
template <int N, class V>
__global__ void __launch_bounds__(f2_threads(F2<N, LF_KB>::items))
    k_sgs_zinv2(const V* __restrict__ st, SgsBufs B, SgsGrid G, const double2* __restrict__ tw,
                const double* __restrict__ alfa, const double* __restrict__ beta, int set,
                const double2* __restrict__ sf) {
  typedef F2<N, LF_KB> P;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* E = reinterpret_cast<double2*>(smem_raw);
  const int y = blockIdx.y, f = blockIdx.z, kx0 = blockIdx.x * LF_KB, t = threadIdx.x;
  if (set == 0 && sgs_plane_off(B, y)) return;
  const size_t slot = (size_t)G.nyp * G.NP;
  if (t < P::items_a) {
    const int kx = min(kx0 + t % LF_KB, G.nx2 - 1);  // beyond the field: not stored
    const LfField L(f, set, __ldg(&alfa[kx]));
    const size_t off = (size_t)y * G.NP + kx;
    auto pass = [&](auto* __restrict__ p0, auto* __restrict__ p1) {
    f2_pass_a<N, LF_KB, LF_KB, 1, false>(
        [&](int iz, int, bool) {
          const size_t o = (size_t)iz * G.nx2;
          const double b = __ldg(&beta[iz]);
          return L(lf_get(p0 + o), lf_get(p1 + o), b, iz == G.zodd);
        },
        E, tw, t);
    };
    if (sf != nullptr && f >= 3)
      pass(sf + L.s0 * slot + off, sf + L.s1 * slot + off);
    else
      pass(st + L.s0 * slot + off, st + L.s1 * slot + off);
  }
  __syncthreads();
  if (t < P::items_b) {
    double2* __restrict__ out = B.spec9 + ((size_t)f * G.nyp + y) * N * G.nx2 + kx0;
    f2_pass_b<N, LF_KB, LF_KB, 1>(
        [&](int m, int, int, int b, double2 v) {
          if (kx0 + b < G.nx2) out[(size_t)m * G.nx2 + b] = v;
        },
        E, t);
  }
}

// test filter in z: forward, |kz| <= nz/4 kept, inverse, in place; a column
// q's modes q + R2 m are the inverse transform's input of the same item
template <int N>
__global__ void __launch_bounds__(f2_threads(F2<N, LF_KB>::items))
    k_sgs_zfilt2(SgsBufs B, SgsGrid G, const double2* __restrict__ tw) {
  typedef F2<N, LF_KB> P;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* E = reinterpret_cast<double2*>(smem_raw);
  const int y = blockIdx.y, kx0 = blockIdx.x * LF_KB, t = threadIdx.x;
  if (sgs_plane_off(B, y)) return;
  double2* fld = B.filt21 + ((size_t)blockIdx.z * G.nyp + y) * N * G.nx4 + kx0;
  if (t < P::items_b)
    f2_fwd_a<N, LF_KB, LF_KB, -1>(
        [&](int m, int b) { return kx0 + b < G.nx4 ? fld[(size_t)m * G.nx4 + b] : double2{0.0, 0.0}; }, E, tw, t);
  __syncthreads();
  if (t < P::items_a) {
    const int q = t / LF_KB, b = t - q * LF_KB;
    constexpr int zlo = N / 4 + 1, zhi = N - N / 4 - 1;
    double2 v[P::R1];
#pragma unroll
    for (int m = 0; m < P::R1; ++m) v[m] = E[P::at(m, q, b)];
    f2_dft<P::R1, -1>(v);
#pragma unroll
    for (int m = 0; m < P::R1; ++m) {
      const int k = q + P::R2 * m;
      if (k >= zlo && k <= zhi) v[m] = double2{0.0, 0.0};
    }
    f2_dft<P::R1, 1>(v);
    f2_twiddle<P::R1, 1>(v, tw, q);
#pragma unroll
    for (int m = 0; m < P::R1; ++m) E[P::at(m, q, b)] = v[m];
  }
  __syncthreads();
  if (t < P::items_b)
    f2_pass_b<N, LF_KB, LF_KB, 1>(
        [&](int m, int, int, int b, double2 v) {
          if (kx0 + b < G.nx4) fld[(size_t)m * G.nx4 + b] = v;
        },
        E, t);
}

// tau: forward z, oddball zeroed, into the state layout
template <int N>
__global__ void __launch_bounds__(f2_threads(F2<N, LF_KB>::items))
    k_sgs_zfwd2(SgsBufs B, SgsGrid G, const double2* __restrict__ tw) {
  typedef F2<N, LF_KB> P;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* E = reinterpret_cast<double2*>(smem_raw);
  const int y = blockIdx.y, f = blockIdx.z, kx0 = blockIdx.x * LF_KB, t = threadIdx.x;
  const double2* __restrict__ in = B.tauz6 + ((size_t)f * G.nyp + y) * N * G.nx2 + kx0;
  if (t < P::items_b)
    f2_fwd_a<N, LF_KB, LF_KB, -1>(
        [&](int m, int b) { return kx0 + b < G.nx2 ? in[(size_t)m * G.nx2 + b] : double2{0.0, 0.0}; }, E, tw, t);
  __syncthreads();
  if (t < P::items_a) {
    double2* __restrict__ dst = B.tau + (size_t)f * G.nyp * G.NP + (size_t)y * G.NP + kx0;
    f2_back_b<N, LF_KB, LF_KB, -1, false>(
        [&](int k, int, int, int b, double2 v) {
          if (kx0 + b < G.nx2) dst[(size_t)k * G.nx2 + b] = k == G.zodd ? double2{0.0, 0.0} : v;
        },
        [](int b) { return b; }, E, t);
  }
}

// sgs_pair of column c's two rows (a and a + fs; the last column may carry
// one), loads without branches: modes beyond nk read mode 0 and are zero
template <int NF>
__device__ __forceinline__ double2 lf_pair(const double2* __restrict__ a, size_t fs, int c, int k, int n, int nk) {
  const bool two = 2 * c + 1 < NF, low = k < nk, high = k > n - nk;
  const int i = low ? k : high ? n - k : 0;
  double2 p = a[i], q = a[(two ? fs : 0) + i];
  if (!two) q = double2{0.0, 0.0};
  if (k == 0) p.y = q.y = 0.0;
  const double2 z = low ? double2{p.x - q.y, p.y + q.x} : double2{p.x + q.y, q.x - p.y};
  return (low || high) ? z : double2{0.0, 0.0};
}

// inverse x of BC columns carrying NF real rows (spectra at src + f fs, nk
// modes), physical values left at (k1, k2) of the buffer
template <int N, int C, int BC, int NF>
__device__ __forceinline__ void lf_xinv(const double2* __restrict__ src, size_t fs, int nk, double2* E,
                                        const double2* __restrict__ tw, int t, int nt) {
  typedef F2<N, C, true> P;
  for (int i = t; i < P::R2 * BC; i += nt)
    f2_pass_a<N, C, BC, 1, false, true>(
        [&](int k, int c, bool) { return lf_pair<NF>(src + (size_t)(2 * c) * fs, fs, c, k, N, nk); },
        E, tw, i);
  __syncthreads();
  for (int i = t; i < P::R1 * BC; i += nt)
    f2_pass_b<N, C, BC, 1, true>([&](int, int k1, int k2, int b, double2 v) { E[P::at(k1, k2, b)] = v; }, E, i);
  __syncthreads();
}

// forward x of BC columns at (k1, k2), then the half spectra (k < nk) of the
// 2 BC real rows (NF of them kept) to dst + f fs
template <int N, int C, int BC, int NF>
__device__ __forceinline__ void lf_xfwd(double2* __restrict__ dst, size_t fs, int nk, double2* E,
                                        const double2* __restrict__ tw, int t, int nt) {
  typedef F2<N, C, true> P;
  auto col = [](int b) { return b; };
  for (int i = t; i < P::R1 * BC; i += nt) f2_back_a<N, C, BC, -1, true>(col, E, tw, i);
  __syncthreads();
  for (int i = t; i < P::R2 * BC; i += nt)
    f2_back_b<N, C, BC, -1, false, true>([&](int, int m, int q, int b, double2 v) { E[P::at(m, q, b)] = v; }, col, E, i);
  __syncthreads();
  for (int i = t; i < nk * BC; i += nt) {
    const int c = i / nk, k = i - c * nk, kk = k == 0 ? 0 : N - k;
    const double2 a = E[P::at(k / P::R2, k % P::R2, c)], b = E[P::at(kk / P::R2, kk % P::R2, c)];
    dst[(size_t)(2 * c) * fs + k] = double2{(a.x + b.x) * .5, (a.y - b.y) * .5};
    if (2 * c + 1 < NF) dst[(size_t)(2 * c + 1) * fs + k] = double2{(a.y + b.y) * .5, (b.x - a.x) * .5};
  }
}

constexpr int LF_XT = 128;  // threads of the x kernels (one z row per CTA)

template <int N>
__global__ void __launch_bounds__(LF_XT) k_sgs_xpass1_2(SgsBufs B, SgsGrid G, const double2* __restrict__ tw,
                                                        const double* __restrict__ delta2,
                                                        const double* __restrict__ s2) {
  constexpr int C = 11;
  typedef F2<N, C, true> P;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* E = reinterpret_cast<double2*>(smem_raw);
  const int m = blockIdx.x, y = blockIdx.y, t = threadIdx.x;
  if (sgs_plane_off(B, y)) return;
  const size_t fs9 = (size_t)G.nyp * G.nz * G.nx2, row = ((size_t)y * G.nz + m) * G.nx2;
  lf_xinv<N, C, 5, 9>(B.spec9 + row, fs9, G.nx2, E, tw, t, LF_XT);
  const double d2 = delta2[y];
  const size_t fs10 = (size_t)G.nyp * G.nz * G.nx, prow = ((size_t)y * G.nz + m) * G.nx;
  for (int j = t; j < N; j += LF_XT) {
    double2* e = E + P::at(j % P::R1, j / P::R1, 0);
    double q[10];
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      q[2 * c] = e[c].x;
      q[2 * c + 1] = e[c].y;
    }
    const double u = q[0], v = q[1], w = q[2];
    const double* s = q + 3;  // S11 S12 S13 S22 S23 S33
    const double sabs = sgs_sabs(s);
#pragma unroll
    for (int f = 0; f < 9; ++f) B.phys10[(size_t)f * fs10 + prow + j] = q[f];
    B.phys10[(size_t)9 * fs10 + prow + j] = sabs;
    const double dr = sabs * d2;
    double r[22];
#pragma unroll
    for (int l = 0; l < 6; ++l) r[l] = -s[l] * dr;  // M parts
    r[6] = -u * u;                                   // L parts
    r[7] = -v * u;
    r[8] = -w * u;
    r[9] = -v * v;
    r[10] = -w * v;
    r[11] = -w * w;
#pragma unroll
    for (int l = 0; l < 6; ++l) r[12 + l] = s2 ? s2[(size_t)l * fs10 + prow + j] : s[l];  // S (or S of H2 u)
    r[18] = u;
    r[19] = v;
    r[20] = w;
    r[21] = 0.0;
#pragma unroll
    for (int c = 0; c < C; ++c) e[c] = double2{r[2 * c], r[2 * c + 1]};
  }
  __syncthreads();
  const size_t fs21 = (size_t)G.nyp * G.nz * G.nx4, frow = ((size_t)y * G.nz + m) * G.nx4;
  lf_xfwd<N, C, C, 21>(B.filt21 + frow, fs21, G.nx4, E, tw, t, LF_XT);
}

template <int N>
__global__ void __launch_bounds__(LF_XT) k_sgs_xpass2_2(SgsBufs B, SgsGrid G, const double2* __restrict__ tw,
                                                        const double* __restrict__ delta2) {
  constexpr int C = 11;
  typedef F2<N, C, true> P;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* E = reinterpret_cast<double2*>(smem_raw);
  const int m = blockIdx.x, y = blockIdx.y, t = threadIdx.x;
  if (sgs_plane_off(B, y)) return;
  const size_t fs21 = (size_t)G.nyp * G.nz * G.nx4, frow = ((size_t)y * G.nz + m) * G.nx4;
  lf_xinv<N, C, C, 21>(B.filt21 + frow, fs21, G.nx4, E, tw, t, LF_XT);
  const double inv = 1.0 / (double)(G.nx * G.nz);
  const double gd2 = 2.5198420997897463295 * delta2[y];  // 4^(2/3)
  const size_t fs10 = (size_t)G.nyp * G.nz * G.nx, prow = ((size_t)y * G.nz + m) * G.nx;
  for (int j = t; j < N; j += LF_XT) {
    const double2* e = E + P::at(j % P::R1, j / P::R1, 0);
    double r[22];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      r[2 * c] = e[c].x * inv;
      r[2 * c + 1] = e[c].y * inv;
    }
    double num, den;
    sgs_germano(r, gd2, num, den);
    B.numden[prow + j] = num;
    B.numden[fs10 + prow + j] = den;
  }
}

template <int N>
__global__ void __launch_bounds__(LF_XT) k_sgs_xinv9_2(SgsBufs B, SgsGrid G, const double2* __restrict__ tw,
                                                       double* __restrict__ out, int f0) {
  constexpr int C = 5;
  typedef F2<N, C, true> P;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* E = reinterpret_cast<double2*>(smem_raw);
  const int m = blockIdx.x, y = blockIdx.y, t = threadIdx.x;
  const size_t fs9 = (size_t)G.nyp * G.nz * G.nx2, row = ((size_t)y * G.nz + m) * G.nx2;
  lf_xinv<N, C, C, 9>(B.spec9 + row, fs9, G.nx2, E, tw, t, LF_XT);
  const size_t fs10 = (size_t)G.nyp * G.nz * G.nx, prow = ((size_t)y * G.nz + m) * G.nx;
  for (int i = t; i < N * C; i += LF_XT) {
    const int c = i / N, j = i - c * N;
    const double2 z = E[P::at(j % P::R1, j / P::R1, c)];
    if (2 * c >= f0) out[(size_t)(2 * c - f0) * fs10 + prow + j] = z.x;
    if (2 * c + 1 < 9 && 2 * c + 1 >= f0) out[(size_t)(2 * c + 1 - f0) * fs10 + prow + j] = z.y;
  }
}

template <int N>
__global__ void __launch_bounds__(LF_XT) k_sgs_tau_x2(SgsBufs B, SgsGrid G, const double2* __restrict__ tw,
                                                      const double* __restrict__ delta2, double re, int ineg,
                                                      const double* __restrict__ tau_phys) {
  constexpr int C = 3;
  typedef F2<N, C, true> P;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* E = reinterpret_cast<double2*>(smem_raw);
  const int m = blockIdx.x, y = blockIdx.y, t = threadIdx.x;
  const size_t fs10 = (size_t)G.nyp * G.nz * G.nx, prow = ((size_t)y * G.nz + m) * G.nx;
  const bool learned = tau_phys != nullptr && (B.plane_on == nullptr || B.plane_on[y] == 0);
  for (int j = t; j < N; j += LF_XT) {
    double q[6];
    sgs_tau_point(B, G, delta2[y], re, ineg, learned ? tau_phys : nullptr, fs10, prow, y, j, q);
    double2* e = E + P::at(j % P::R1, j / P::R1, 0);
#pragma unroll
    for (int c = 0; c < 3; ++c) e[c] = double2{q[2 * c], q[2 * c + 1]};
  }
  __syncthreads();
  const size_t fs = (size_t)G.nyp * G.nz * G.nx2, row = ((size_t)y * G.nz + m) * G.nx2;
  lf_xfwd<N, C, C, 6>(B.tauz6 + row, fs, G.nx2, E, tw, t, LF_XT);
}

// Lengths nx, nz up to 128, the coarse grids that these models are for (and
// multiples of four, as the models ask).  20 and the 14 lengths of factors 2, 3,
// 5 from 144 to 384 split too; they take the kernels of les_dyn.cuh, each
// length being eight more kernels to build.
#define SB_LF_LENGTHS(X) X(16) X(24) X(32) X(36) X(40) X(48) X(60) X(64) X(72) X(80) X(96) X(100) X(108) X(120) X(128)

}  // namespace sb
