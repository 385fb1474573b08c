// FP64 step 2 (and the pressure's physical-space pass) with the two-pass
// transforms of fft2.cuh: the same work, arrays and normalisation as k_zinv,
// k_xpass, k_zfwd (step2.cuh) and k_xpass_p (press.cuh), which serve the lengths
// without a two-pass kernel.
//
//   k_zinv2   eight kx columns per CTA (128-byte rows of the FP64 fields)
//   k_xpass2  two z rows: six inverse columns; the products in place; three
//             forward columns (H1 + i H2 of each row, the two H3 as one)
//   k_zfwd2   eight kx columns
//   k_xpass_p2  two z rows, six inverse and four forward columns
// Three resident passes over shared memory per direction and column instead
// of six.  At 384x193x384 against the Stockham kernels: z inverse 0.96 -> 0.63
// ms, x pass 1.92 -> 1.49, z forward 0.51 -> 0.30 (moving 2.1, 3.1 and 1.5 GB;
// 192x129x160: 0.13 -> 0.09, 0.35 -> 0.20, 0.06 -> 0.04).  Bound by the shared
// memory and L1 traffic of the passes (x pass) and by HBM (z transforms).
// The x passes' work items run along a row, as the rows do in memory; with
// the columns fastest, as in the z transforms, the x pass took 1.97 ms: a warp's
// load touched eleven rows.
#pragma once
#include "fft2.cuh"
#include "layout.cuh"
#include "step2.cuh"

namespace sb {

constexpr int F2_KB = 8;  // kx columns per CTA of the z transforms
constexpr int F2_RB = 2;  // z rows per CTA of the x passes

template <int N, class SV>
__global__ void __launch_bounds__(f2_threads(F2<N, F2_KB>::items), f2_minb(f2_threads(F2<N, F2_KB>::items)))
    k_zinv2(const SV* __restrict__ st, double2* __restrict__ zb, Dims g, const double2* __restrict__ tw,
            const double* __restrict__ alfa, const double* __restrict__ beta) {
  typedef F2<N, F2_KB> P;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* E = reinterpret_cast<double2*>(smem_raw);
  const int y = g.y0 + blockIdx.y, kx0 = blockIdx.x * F2_KB;
  const size_t slot = (size_t)g.nyp * g.NP;
  const SV* __restrict__ plane = st + (size_t)y * g.NP;
  const int t = threadIdx.x;
  for (int f = 0; f < 6; ++f) {
    // fine-grid fields: u, v, w, omega_x, omega_y = i beta u - i alpha w, omega_z
    const SV* __restrict__ src = plane + (size_t)(f == 4 ? 0 : f == 5 ? 4 : f) * slot;
    // padded z index m < N/3 = nz/2: kz row m; m >= 2N/3: row m - N/3, of which
    // the first (nz/2, the oddball) is zero; kx beyond the field reads the last
    // column, whose result is not stored
    const int kxc = min(kx0 + t % F2_KB, g.nx2 - 1);
    auto row = [&](int m, bool high) { return (high ? m - N / 3 : m) * g.nx2 + kxc; };
    if (t < P::items_a && f != 4) {
      f2_pass_a<N, F2_KB, F2_KB, 1, true>(
          [&](int m, int, bool high) {
            const SV q = src[row(m, high)];
            const bool z = high && m == 2 * N / 3;
            return double2{z ? 0.0 : (double)q.x, z ? 0.0 : (double)q.y};
          },
          E, tw, t);
    } else if (t < P::items_a) {
      const double a = __ldg(&alfa[kxc]);
      f2_pass_a<N, F2_KB, F2_KB, 1, true>(
          [&](int m, int, bool high) {
            const int o = row(m, high);
            const SV u = src[o], w = src[2 * slot + o];
            const double be = __ldg(&beta[high ? m - N / 3 : m]);
            const bool z = high && m == 2 * N / 3;
            return double2{z ? 0.0 : -be * (double)u.y + a * (double)w.y,
                           z ? 0.0 : be * (double)u.x - a * (double)w.x};
          },
          E, tw, t);
    }
    __syncthreads();
    if (t < P::items_b) {
      double2* __restrict__ out = zb + ((size_t)f * g.nyp + y) * N * g.nx2 + kx0;
      f2_pass_b<N, F2_KB, F2_KB, 1>(
          [&](int m, int, int, int b, double2 v) {
            if (kx0 + b < g.nx2) out[(size_t)m * g.nx2 + b] = v;
          },
          E, t);
    }
    __syncthreads();
  }
}

// kept padded index m -> stored kz index of the forward transform, -1 dropped
template <int N>
__device__ __forceinline__ int f2_keep(int m, int nz) {
  const int nzh = nz / 2;
  return m < nzh ? m : (m >= N - nzh ? m - (N - nz) : -1);
}

template <int N>
__global__ void __launch_bounds__(f2_threads(F2<N, F2_KB>::items), f2_minb(f2_threads(F2<N, F2_KB>::items)))
    k_zfwd2(const double2* __restrict__ xb, double2* __restrict__ st, Dims g, const double2* __restrict__ tw) {
  typedef F2<N, F2_KB> P;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* E = reinterpret_cast<double2*>(smem_raw);
  const int y = g.y0 + blockIdx.y, kx0 = blockIdx.x * F2_KB;
  const size_t slot = (size_t)g.nyp * g.NP, fs = (size_t)g.nyp * N * g.nx2;
  const int t = threadIdx.x;
  for (int f = 0; f < 3; ++f) {
    const double2* __restrict__ in = xb + f * fs + (size_t)y * N * g.nx2 + kx0;
    if (t < P::items_b) {
      f2_fwd_a<N, F2_KB, F2_KB, -1>(
          [&](int m, int b) { return kx0 + b < g.nx2 ? in[(size_t)m * g.nx2 + b] : double2{0.0, 0.0}; }, E, tw, t);
    }
    __syncthreads();
    if (t < P::items_a) {
      double2* __restrict__ dst = st + f * slot + (size_t)y * g.NP + kx0;
      f2_back_b<N, F2_KB, F2_KB, -1, true>(
          [&](int k, int, int, int b, double2 v) {
            const int iz = f2_keep<N>(k, g.nz);
            if (iz >= 0 && kx0 + b < g.nx2) dst[iz * g.nx2 + b] = v;
          },
          [](int b) { return b; }, E, t);
    }
    __syncthreads();
  }
}

// element k of the Hermitian-completed spectrum of fields 2q (real part) and
// 2q + 1 (imaginary part): p0, p1 their half spectra (N/3 modes); k < N/3, or
// (high) k >= 2N/3
template <int N>
__device__ __forceinline__ double2 f2_herm(const double2* __restrict__ p0, const double2* __restrict__ p1, int k,
                                           bool high) {
  if (!high) {
    double2 a = p0[k], b = p1[k];
    if (k == 0) a.y = b.y = 0.0;
    return double2{a.x - b.y, a.y + b.x};
  }
  const bool z = k == 2 * N / 3;  // the mirror of mode N/3, which is not stored
  const int i = z ? 0 : N - k;
  const double2 a = p0[i], b = p1[i];
  return double2{z ? 0.0 : a.x + b.y, z ? 0.0 : b.x - a.y};
}

template <int N>
__global__ void __launch_bounds__(f2_threads(F2<N, 3 * F2_RB>::items), f2_minb(f2_threads(F2<N, 3 * F2_RB>::items)))
    k_xpass2(const double2* __restrict__ zb, double2* __restrict__ xb, Dims g, const double2* __restrict__ tw,
             const double* __restrict__ dyi, double dxi, double dzi, double rot,
             unsigned long long* __restrict__ cfl_bits, Fringe fr) {
  constexpr int C = 3 * F2_RB, NT = f2_threads(F2<N, C>::items);
  typedef F2<N, C, true> P;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* E = reinterpret_cast<double2*>(smem_raw);
  const int y = g.y0 + blockIdx.y, m0 = blockIdx.x * F2_RB;
  const size_t fstride = (size_t)g.nyp * g.nzp * g.nx2;
  const size_t row0 = ((size_t)y * g.nzp + m0) * g.nx2;
  const int t = threadIdx.x;
  if (t < P::items_a) {
    f2_pass_a<N, C, C, 1, true, true>(
        [&](int k, int c, bool high) {
          // (a row beyond the plane reads the last one; nothing of it is kept)
          const int q = c % 3, r = m0 + c / 3 < g.nzp ? c / 3 : 0;
          const double2* p0 = zb + row0 + (size_t)(2 * q) * fstride + r * g.nx2;
          return f2_herm<N>(p0, p0 + fstride, k, high);
        },
        E, tw, t);
  }
  __syncthreads();
  // physical values back to their own row of the buffer: x = k1 + R1 k2 at (k1, k2)
  if (t < P::items_b)
    f2_pass_b<N, C, C, 1, true>([&](int, int k1, int k2, int b, double2 v) { E[P::at(k1, k2, b)] = v; }, E, t);
  __syncthreads();
  // products of both rows of a point: H1 + i H2 of row r over column 3 r, the
  // two H3 over column 1
  const double r2 = 2.0 * rot, cy = dyi[y];
  double cmax = 0.0;
  for (int pt = t; pt < N; pt += NT) {
    const int k1 = pt / P::R2, k2 = pt - k1 * P::R2;
    double2* e = E + P::at(k1, k2, 0);
    double h3r[F2_RB];
#pragma unroll
    for (int r = 0; r < F2_RB; ++r) {
      const double2 z0 = e[3 * r], z1 = e[3 * r + 1], z2 = e[3 * r + 2];
      const double u = z0.x, v = z0.y, w = z1.x, ox = z1.y, oy = z2.x, oz = z2.y;
      double h1 = v * (oz + r2) - w * oy;
      double h2 = w * ox - u * (oz + r2);
      double h3 = u * oy - v * ox;
      if (fr.lam != nullptr) fringe_apply<double>(fr, k1 + P::R1 * k2, y, g.nyp, N, u, v, w, 0.0, 0.0, h1, h2, h3);
      e[3 * r] = double2{h1, h2};
      h3r[r] = h3;
      if (m0 + r < g.nzp) cmax = fmax(cmax, fabs(u) * dxi + fabs(v) * cy + fabs(w) * dzi);
    }
    e[1] = double2{h3r[0], h3r[1]};
  }
  __syncthreads();
  auto col = [](int b) { return b == 2 ? 3 : b; };
  if (t < P::R1 * 3) f2_back_a<N, C, 3, -1, true>(col, E, tw, t);
  __syncthreads();
  if (t < P::R2 * 3)
    f2_back_b<N, C, 3, -1, true, true>([&](int, int m, int q, int b, double2 v) { E[P::at(m, q, b)] = v; }, col, E, t);
  __syncthreads();
  for (int i = t; i < g.nx2 * F2_RB; i += NT) {
    const int r = i >= g.nx2, k = i - r * g.nx2;
    if (m0 + r >= g.nzp) continue;
    const int kk = k == 0 ? 0 : N - k;
    const double2* ek = E + P::at(k / P::R2, k % P::R2, 0);
    const double2* em = E + P::at(kk / P::R2, kk % P::R2, 0);
    const double2 a = ek[3 * r], b = em[3 * r], c = ek[1], d = em[1];
    double2* __restrict__ o = xb + row0 + r * g.nx2 + k;
    o[0] = double2{(a.x + b.x) * 0.5, (a.y - b.y) * 0.5};
    o[fstride] = double2{(a.y + b.y) * 0.5, (b.x - a.x) * 0.5};
    o[2 * fstride] = r ? double2{(c.y + d.y) * 0.5, (d.x - c.x) * 0.5} : double2{(c.x + d.x) * 0.5, (c.y - d.y) * 0.5};
  }
  for (int off = 16; off > 0; off >>= 1) cmax = fmax(cmax, __shfl_xor_sync(0xffffffffu, cmax, off));
  __shared__ double wmax[NT / 32];
  if ((t & 31) == 0) wmax[t >> 5] = cmax;
  __syncthreads();
  if (t == 0 && cfl_bits != nullptr) {
    double mx = 0.0;
    for (int i = 0; i < NT / 32; ++i) mx = fmax(mx, wmax[i]);
    atomic_max_nonneg(cfl_bits, mx);
  }
}

// k_xpass_p with two-pass transforms: H1 + i H2 in column 3 r, H3 + 2E i in
// 3 r + 1; the kept spectra over this CTA's own rows of fields 0..3, which it
// has read before the first barrier.
template <int N>
__global__ void __launch_bounds__(f2_threads(F2<N, 3 * F2_RB>::items), f2_minb(f2_threads(F2<N, 3 * F2_RB>::items)))
    k_xpass_p2(double2* zb, Dims g, const double2* __restrict__ tw, double rot, Fringe fr) {
  constexpr int C = 3 * F2_RB, NT = f2_threads(F2<N, C>::items);
  typedef F2<N, C, true> P;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* E = reinterpret_cast<double2*>(smem_raw);
  const int y = blockIdx.y, m0 = blockIdx.x * F2_RB;
  const size_t fstride = (size_t)g.nyp * g.nzp * g.nx2;
  double2* row0 = zb + ((size_t)y * g.nzp + m0) * g.nx2;
  const int t = threadIdx.x;
  if (t < P::items_a) {
    f2_pass_a<N, C, C, 1, true, true>(
        [&](int k, int c, bool high) {
          const int q = c % 3, r = m0 + c / 3 < g.nzp ? c / 3 : 0;
          const double2* p0 = row0 + (size_t)(2 * q) * fstride + r * g.nx2;
          return f2_herm<N>(p0, p0 + fstride, k, high);
        },
        E, tw, t);
  }
  __syncthreads();
  if (t < P::items_b)
    f2_pass_b<N, C, C, 1, true>([&](int, int k1, int k2, int b, double2 v) { E[P::at(k1, k2, b)] = v; }, E, t);
  __syncthreads();
  const double r2 = 2.0 * rot;
  for (int i = t; i < N * F2_RB; i += NT) {
    const int r = i / N, pt = i - r * N, k1 = pt / P::R2, k2 = pt - k1 * P::R2;
    double2* e = E + P::at(k1, k2, 3 * r);
    const double2 z0 = e[0], z1 = e[1], z2 = e[2];
    const double u = z0.x, v = z0.y, w = z1.x, ox = z1.y, oy = z2.x, oz = z2.y;
    double h1 = v * (oz + r2) - w * oy;
    double h2 = w * ox - u * (oz + r2);
    double h3 = u * oy - v * ox;
    if (fr.lam != nullptr) fringe_apply<double>(fr, k1 + P::R1 * k2, y, g.nyp, N, u, v, w, 0.0, 0.0, h1, h2, h3);
    e[0] = double2{h1, h2};
    e[1] = double2{h3, u * u + v * v + w * w};
  }
  __syncthreads();
  auto col = [](int b) { return b < 2 ? b : b + 1; };
  if (t < P::R1 * 4) f2_back_a<N, C, 4, -1, true>(col, E, tw, t);
  __syncthreads();
  if (t < P::R2 * 4)
    f2_back_b<N, C, 4, -1, true, true>([&](int, int m, int q, int b, double2 v) { E[P::at(m, q, b)] = v; }, col, E, t);
  __syncthreads();
  for (int i = t; i < g.nx2 * F2_RB; i += NT) {
    const int r = i >= g.nx2, k = i - r * g.nx2;
    if (m0 + r >= g.nzp) continue;
    const int kk = k == 0 ? 0 : N - k;
    const double2* ek = E + P::at(k / P::R2, k % P::R2, 3 * r);
    const double2* em = E + P::at(kk / P::R2, kk % P::R2, 3 * r);
    const double2 a = ek[0], b = em[0], c = ek[1], d = em[1];
    double2* o = row0 + r * g.nx2 + k;
    o[0] = double2{(a.x + b.x) * 0.5, (a.y - b.y) * 0.5};
    o[fstride] = double2{(a.y + b.y) * 0.5, (b.x - a.x) * 0.5};
    o[2 * fstride] = double2{(c.x + d.x) * 0.5, (c.y - d.y) * 0.5};
    o[3 * fstride] = double2{(c.y + d.y) * 0.5, (d.x - c.x) * 0.5};
  }
}

}  // namespace sb
