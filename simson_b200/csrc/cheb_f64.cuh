// FP64 Chebyshev transforms over pencils with two-pass register transforms
// (fft2.cuh): the DCT-I of length ny as the complex transform of the even
// extension of length L = 2 (ny - 1), the conventions and arguments of k_cheb
// (step3.cuh), which serves the other lengths.
//
// x[n] = x[L - n] halves both passes.  Pass A (DFT of R1 over n = R2 n1 + n2):
// the items n2 and R2 - n2 have reversed inputs, so one item writes both,
//   E(k1, n2) = A[k1] w^(n2 k1),  E(k1, R2 - n2) = A[R1 - k1] conj(w^(n2 k1)),
// w = exp(-2 pi i / L).  Pass B (DFT of R2): X[k] = X[L - k], so the items
// k1 <= R1/2 give every coefficient k <= L/2, the outputs above it as L - k.
#pragma once
#include "fft2.cuh"
#include "layout.cuh"

namespace sb {

constexpr int CHB2_PB = 8;  // pencils per CTA (128-byte rows)

template <int L>
struct Chb2 {
  typedef F2<L, CHB2_PB> P;
  static constexpr int items_a = (P::R2 / 2 + 1) * CHB2_PB, items_b = (P::R1 / 2 + 1) * CHB2_PB;
  static constexpr int threads = f2_threads(items_a > items_b ? items_a : items_b);
};

template <int L>
__global__ void __launch_bounds__(Chb2<L>::threads, f2_minb(Chb2<L>::threads))
    k_cheb2(const double2* __restrict__ in, size_t in_fs, double2* __restrict__ out, size_t out_fs, Dims g, int inverse,
            double scale, const double2* __restrict__ tw, int skip_oddball) {
  typedef F2<L, CHB2_PB> P;
  constexpr int PB = CHB2_PB, Ny = L / 2, R1 = P::R1, R2 = P::R2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* E = reinterpret_cast<double2*>(smem_raw);
  const int t = threadIdx.x, b = t % PB, item = t / PB;
  const int p = g.p0 + blockIdx.x * PB + b;
  const bool live = p < g.p1;
  const double2* __restrict__ src = in + blockIdx.y * in_fs + p;
  double2* __restrict__ dst = out + blockIdx.y * out_fs + p;
  if (item <= R2 / 2) {
    const int n2 = item;
    double2 v[R1];
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) {
      const int m = R2 * n1 + n2, j = m <= Ny ? m : L - m;
      double2 x{0.0, 0.0};
      if (live) x = src[(size_t)j * g.NP];
      if (inverse && j != 0 && j != Ny) x = double2{0.5 * x.x, 0.5 * x.y};
      v[n1] = x;
    }
    f2_dft<R1, -1>(v);
    // w^(n2 k): k below 4 and multiples of 4 from the table, one product each
    // for the others
    double2 lo[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) lo[k] = __ldg(&tw[k * n2]);
    const bool two = n2 > 0 && 2 * n2 < R2;
#pragma unroll
    for (int j = 0; j < R1; j += 4) {
      const double2 hi = __ldg(&tw[j * n2]);
#pragma unroll
      for (int i = 0; i < 4 && j + i < R1; ++i) {
        const int k = j + i;
        const double2 w = i == 0 ? hi : (j == 0 ? lo[i] : cmul(hi, lo[i]));
        E[P::at(k, n2, b)] = cmul(v[k], w);
        if (two) E[P::at(k, R2 - n2, b)] = cmul(v[(R1 - k) % R1], cconj(w));
      }
    }
  }
  __syncthreads();
  if (item <= R1 / 2 && live && !(skip_oddball && p / g.nx2 == g.zodd)) {
    const int k1 = item;
    double2 v[R2];
#pragma unroll
    for (int n2 = 0; n2 < R2; ++n2) v[n2] = E[P::at(k1, n2, b)];
    f2_dft<R2, -1>(v);
    const bool fold = k1 > 0 && 2 * k1 < R1;  // the item of R1 - k1 is not run
    const double fi = inverse ? scale : scale / (double)Ny, fe = inverse ? scale : 0.5 * fi;
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) {
      const int k = k1 + R1 * k2;
      if (k > Ny && !fold) continue;
      const int c = k > Ny ? L - k : k;
      const double f = (c == 0 || c == Ny) ? fe : fi;
      dst[(size_t)c * g.NP] = double2{v[k2].x * f, v[k2].y * f};
    }
  }
}

// L = 2 (ny - 1): ny = 9 and 17 to 241, ny - 1 of factors 2, 3, 5, but for ny =
// 11, 13 and 251, which split too and take k_cheb; 512 (ny = 257) has no split
#define SB_CHB2_LENGTHS(X)                                                                                       \
  X(16) X(32) X(36) X(40) X(48) X(60) X(64) X(72) X(80) X(96) X(100) X(108) X(120) X(128) X(144) X(160) X(180)    \
  X(192) X(200) X(216) X(240) X(256) X(288) X(300) X(320) X(324) X(360) X(384) X(400) X(432) X(480)

}  // namespace sb
