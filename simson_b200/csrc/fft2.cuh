// Two-pass FP64 transforms with register DFTs.
//
// A length-N transform, N = R1 R2, of C interleaved columns:
//   pass A  item (n2, b): the R1 elements n = R2 n1 + n2 of column b, a DFT of
//           R1 in registers, times w_N^(n2 k1), to the exchange buffer
//   pass B  item (k1, b): the R2 elements n2 of that k1, a DFT of R2 in
//           registers: the outputs k = k1 + R1 k2
// One exchange through shared memory instead of the two or three of the
// small-radix Stockham passes (fft.cuh): the FP64 transforms were bound by
// shared-memory bandwidth (80 % of its peak in the x pass at 192x129x160, FP64
// pipe 21 %).  The buffer holds element (k1, n2) of column b at
// k1 SR + n2 CS + b.  Eight neighbouring items of either pass touch eight
// different 16-byte bank groups, in either order of the items:
//   columns fastest (the z and Chebyshev transforms, whose columns are
//   neighbours in memory): CS = C, SR = C (mod 8)
//   elements fastest (NF; the x transforms, whose elements are): CS and SR odd
//
// Lengths are compile-time; R1 is a multiple of 3 for the 3/2-padded lengths,
// so that the zero band is whole blocks of pass A's input (the middle third of
// n1) and the dropped band whole blocks of pass B's output.
#pragma once
#include "fft.cuh"

namespace sb {

// cos, sin of 2 pi k / n at compile time (Taylor series about 0 after
// reduction to an eighth of the circle)
constexpr double f2_series(double x, bool sine) {
  double term = sine ? x : 1.0, sum = 0.0;
  double parts[14] = {};
  for (int i = 0; i < 14; ++i) {
    parts[i] = term;
    const int a = 2 * i + (sine ? 2 : 1);
    term = -term * x * x / (double)(a * (a + 1));
  }
  for (int i = 13; i >= 0; --i) sum += parts[i];  // smallest first
  return sum;
}
constexpr double F2_2PI = 6.28318530717958647692528676655900577;
constexpr double f2_cos(int k, int n) {
  k %= n;
  if (k < 0) k += n;
  if (2 * k > n) k = n - k;                       // cos is even
  if (4 * k > n) return -f2_cos(n - 2 * k, 2 * n);  // pi - x
  if (8 * k > n) return f2_series(F2_2PI * (n - 4 * k) / (4.0 * n), true);
  return f2_series(F2_2PI * k / n, false);
}
constexpr double f2_sin(int k, int n) { return f2_cos(4 * k - n, 4 * n); }  // cos(x - pi/2)

// a * exp(S 2 pi i K / R), K and R compile-time
template <int K, int R, int S>
SB_HD __forceinline__ double2 f2_rot(double2 a) {
  constexpr int k = K % R;
  if constexpr (k == 0)
    return a;
  else if constexpr (4 * k == R)
    return cmuli(a, S);
  else if constexpr (2 * k == R)
    return double2{-a.x, -a.y};
  else if constexpr (4 * k == 3 * R)
    return cmuli(a, -S);
  else {
    constexpr double c = f2_cos(k, R), s = S * f2_sin(k, R);
    return cmul(a, double2{c, s});
  }
}

// first factor of the register DFT of size r (1: a butterfly of fft.cuh)
constexpr int f2_first(int r) {
  if (r <= 6 || r == 8) return 1;
  if (r % 3 == 0) return 3;
  if (r % 4 == 0) return 4;
  if (r % 5 == 0) return 5;
  return 2;
}

template <int B, int A, int S, int N2, int K1>
SB_HD __forceinline__ void f2_twist(double2 (&t)[A]) {
  if constexpr (K1 < A) {
    t[K1] = f2_rot<N2 * K1, A * B, S>(t[K1]);
    f2_twist<B, A, S, N2, K1 + 1>(t);
  }
}

// DFT of size R in registers, natural order; ZM: the middle third of the
// inputs is zero and not read (R a multiple of 3 with first factor 3)
template <int R, int S, bool ZM = false>
SB_HD __forceinline__ void f2_dft(double2 (&v)[R]);

template <int R, int S, bool ZM, int N2>
SB_HD __forceinline__ void f2_inner(const double2 (&v)[R], double2 (&u)[R]) {
  constexpr int A = f2_first(R), B = R / A;
  if constexpr (N2 < B) {
    double2 t[A];
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) t[n1] = v[B * n1 + N2];
    if constexpr (ZM && A == 3)
      dft3_zmid<double, double2>(t[0], t[1], t[2], S);
    else
      dft_small<double, double2>(t, A, S);
    f2_twist<B, A, S, N2, 1>(t);
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) u[k1 * B + N2] = t[k1];
    f2_inner<R, S, ZM, N2 + 1>(v, u);
  }
}

template <int R, int S, bool ZM>
SB_HD __forceinline__ void f2_dft(double2 (&v)[R]) {
  constexpr int A = f2_first(R), B = R / A;
  if constexpr (R == 1) {
  } else if constexpr (A == 1) {
    if constexpr (ZM) {
#pragma unroll
      for (int n = R / 3; n < 2 * R / 3; ++n) v[n] = double2{0.0, 0.0};
    }
    dft_small<double, double2>(v, R, S);
  } else {
    double2 u[R];
    f2_inner<R, S, ZM, 0>(v, u);
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
      double2 t[B];
#pragma unroll
      for (int n2 = 0; n2 < B; ++n2) t[n2] = u[k1 * B + n2];
      f2_dft<B, S>(t);
#pragma unroll
      for (int k2 = 0; k2 < B; ++k2) v[k1 + A * k2] = t[k2];
    }
  }
}

// register DFT sizes; larger ones spill at the occupancy the kernels need
constexpr int F2_MAX_R = 25;
// R1 of length n: the factor pair closest to a square with both sides within
// F2_MAX_R, R1 a multiple of 3 where n is one (the larger side when both are);
// 0 if there is none
constexpr int f2_r1(int n) {
  int best = 0, gap = 1 << 30;
  for (int a = 2; a <= F2_MAX_R; ++a) {
    if (n % a || n / a > F2_MAX_R || n / a < 2) continue;
    if (n % 3 == 0 && a % 3) continue;
    int m = a * (n / a);
    for (int f = 2; f <= 5; ++f)
      while (m % f == 0) m /= f;
    if (m != 1) continue;
    const int d = a > n / a ? a - n / a : n / a - a;
    if (d < gap || (d == gap && a > best)) {
      gap = d;
      best = a;
    }
  }
  return best;
}

template <int N, int C, bool NF = false>
struct F2 {
  static constexpr int R1 = f2_r1(N), R2 = R1 ? N / (R1 ? R1 : 1) : 0;
  static_assert(R1 > 0, "no two-pass split of this length");
  static constexpr int CS = NF ? (C | 1) : C;           // stride of n2
  static constexpr int pad = NF ? (R2 * CS + 1) % 2 : ((C - R2 * C) % 8 + 8) % 8;
  static constexpr int SR = R2 * CS + pad;              // stride of k1
  static constexpr int size = R1 * SR;                 // exchange buffer, elements
  static constexpr int items_a = R2 * C, items_b = R1 * C;
  static constexpr int items = items_a > items_b ? items_a : items_b;
  static SB_HD __forceinline__ int at(int k1, int n2, int b) { return k1 * SR + n2 * CS + b; }
  // item t of R elements by BC columns: its element and column
  static SB_HD __forceinline__ int elem(int t, int R, int BC) { return NF ? t % R : t / BC; }
  static SB_HD __forceinline__ int column(int t, int R, int BC) { return NF ? t / R : t % BC; }
};

// v[k] *= w^k, w = exp(S 2 pi i e / N), k < R, from the table tw[m] =
// exp(-2 pi i m / N): w .. w^3 and the powers w^(4 j) are read, the others one
// product each
template <int R, int S>
__device__ __forceinline__ void f2_twiddle(double2 (&v)[R], const double2* __restrict__ tw, int e) {
  auto ld = [&](int k) {
    double2 w = __ldg(&tw[k * e]);
    if (S > 0) w.y = -w.y;
    return w;
  };
  double2 lo[4];
#pragma unroll
  for (int k = 1; k < 4 && k < R; ++k) {
    lo[k] = ld(k);
    v[k] = cmul(v[k], lo[k]);
  }
#pragma unroll
  for (int j = 4; j < R; j += 4) {
    const double2 hi = ld(j);
    v[j] = cmul(v[j], hi);
#pragma unroll
    for (int k = 1; k < 4 && j + k < R; ++k) v[j + k] = cmul(v[j + k], cmul(hi, lo[k]));
  }
}

// Pass A of item t (< items_a): ld(n, b, high) gives element n of column b,
// high (a constant once unrolled) whether n is in the upper half of the blocks
// -- with ZM the last third, n >= 2 N / 3, the others being n < N / 3 -- so
// that a load needs no branch on n and a thread's loads go out together.  BC:
// columns transformed (items t < R2 BC), C the buffer's.
template <int N, int C, int BC, int S, bool ZM, bool NF = false, class Ld>
__device__ __forceinline__ void f2_pass_a(Ld ld, double2* __restrict__ E, const double2* __restrict__ tw, int t) {
  typedef F2<N, C, NF> P;
  const int n2 = P::elem(t, P::R2, BC), b = P::column(t, P::R2, BC);
  double2 v[P::R1];
#pragma unroll
  for (int n1 = 0; n1 < P::R1; ++n1)
    if (!(ZM && 3 * n1 >= P::R1 && 3 * n1 < 2 * P::R1)) v[n1] = ld(P::R2 * n1 + n2, b, 2 * n1 >= P::R1);
  f2_dft<P::R1, S, ZM>(v);
  f2_twiddle<P::R1, S>(v, tw, n2);
#pragma unroll
  for (int k1 = 0; k1 < P::R1; ++k1) E[P::at(k1, n2, b)] = v[k1];
}

// Pass B of item t (< R1 BC): st(k, k1, k2, b, value) receives output
// k = k1 + R1 k2.
template <int N, int C, int BC, int S, bool NF = false, class St>
__device__ __forceinline__ void f2_pass_b(St st, const double2* E, int t) {
  typedef F2<N, C, NF> P;
  const int k1 = P::elem(t, P::R1, BC), b = P::column(t, P::R1, BC);
  double2 v[P::R2];
#pragma unroll
  for (int n2 = 0; n2 < P::R2; ++n2) v[n2] = E[P::at(k1, n2, b)];
  f2_dft<P::R2, S>(v);
#pragma unroll
  for (int k2 = 0; k2 < P::R2; ++k2) st(k1 + P::R1 * k2, k1, k2, b, v[k2]);
}

// The transposed pair, for a column whose element n = k1 + R1 k2 sits at
// (k1, k2), as f2_pass_b leaves it: pass A reads its own row k1 (DFT of R2,
// times w_N^(k1 q)) and writes it back in place (f2_fwd_a: reads it through
// ld); pass B, item q < R2, reads column q (DFT of R1): outputs k = q + R2 m.
// col(b): the buffer column of transform b.  DROP: the middle third of m (the
// dropped band of a forward transform) is neither computed nor stored.
template <int N, int C, int BC, int S, bool NF, class Ld, class Col>
__device__ __forceinline__ void f2_row_a(Ld ld, Col col, double2* E, const double2* __restrict__ tw,
                                         int t) {
  typedef F2<N, C, NF> P;
  const int k1 = P::elem(t, P::R1, BC), b = P::column(t, P::R1, BC);
  double2 v[P::R2];
#pragma unroll
  for (int k2 = 0; k2 < P::R2; ++k2) v[k2] = ld(k1, k2, b);
  f2_dft<P::R2, S>(v);
  f2_twiddle<P::R2, S>(v, tw, k1);
#pragma unroll
  for (int k2 = 0; k2 < P::R2; ++k2) E[P::at(k1, k2, col(b))] = v[k2];
}
template <int N, int C, int BC, int S, bool NF = false, class Col>
__device__ __forceinline__ void f2_back_a(Col col, double2* E, const double2* __restrict__ tw, int t) {
  f2_row_a<N, C, BC, S, NF>([&](int k1, int k2, int b) { return E[F2<N, C, NF>::at(k1, k2, col(b))]; }, col, E, tw, t);
}
template <int N, int C, int BC, int S, class Ld>
__device__ __forceinline__ void f2_fwd_a(Ld ld, double2* __restrict__ E, const double2* __restrict__ tw, int t) {
  f2_row_a<N, C, BC, S, false>([&](int k1, int k2, int b) { return ld(k1 + F2<N, C>::R1 * k2, b); }, [](int b) { return b; },
                        E, tw, t);
}
template <int N, int C, int BC, int S, bool DROP, bool NF = false, class St, class Col>
__device__ __forceinline__ void f2_back_b(St st, Col col, const double2* E, int t) {
  typedef F2<N, C, NF> P;
  const int q = P::elem(t, P::R2, BC), b = P::column(t, P::R2, BC);
  double2 v[P::R1];
#pragma unroll
  for (int m = 0; m < P::R1; ++m) v[m] = E[P::at(m, q, col(b))];
  f2_dft<P::R1, S>(v);
#pragma unroll
  for (int m = 0; m < P::R1; ++m)
    if (!(DROP && 3 * m >= P::R1 && 3 * m < 2 * P::R1)) st(q + P::R2 * m, m, q, col(b), v[m]);
}

// threads per CTA for items work items, a multiple of 32
constexpr int f2_threads(int items) { return (items + 31) / 32 * 32; }
// resident CTAs per SM the register budget is sized for: twelve warps of 168
// registers
constexpr int f2_minb(int threads) { return 12 * 32 / threads > 0 ? 12 * 32 / threads : 1; }

// Lengths with two-pass kernels: 3/2 of 27 grid sizes from 16 to 384.  Every
// length is five kernels to build, so not all that split are here: 27, 30, 45,
// 54, 75, 81, 162 and 375 (grid sizes 18, 20, 30, 36, 50, 54, 108, 250) split
// too and take the runtime plan.  243, 405, 486 and 540 have no split with both
// sides within F2_MAX_R.
#define SB_F2_LENGTHS_A(X) X(24) X(36) X(48) X(60) X(72) X(90) X(96) X(108) X(120)
#define SB_F2_LENGTHS_B(X) X(135) X(144) X(150) X(180) X(192) X(216) X(225)
#define SB_F2_LENGTHS_C(X) X(240) X(270) X(288) X(300) X(324) X(360)
#define SB_F2_LENGTHS_D(X) X(384) X(432) X(450) X(480) X(576)

}  // namespace sb
