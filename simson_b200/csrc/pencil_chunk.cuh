// Step 3 with a group of threads per (kx, kz) pencil: the same algebra as
// k_pencil (bla/linearbl.f:257-1860 for the channel, ibc = 0, tau method),
// each thread holding a chunk of R consecutive Chebyshev rows of its pencil.
//
// A CTA owns PC_TP neighbouring pencils times G chunks (thread = chunk * PC_TP
// + pencil), so a row of the tile is one contiguous piece of every field, all
// rows of H, p_v, p_omega are loaded at once (no serial sweep waits for
// memory) and read and written once: nothing else goes through DRAM but the
// tau coefficients.
//
// Tau solves (D^2 - lam) x = f (tau_solve in step3.cuh, 0-based rows j; the
// elimination of bla/trid.f:120-200).  With c'_j its eliminated lower
// coefficient, which depends on k^2 and lam only and is kept per RK stage
// (k_tau_coef: one real column per |kz|, shared by +-kz), the factors of a
// row cancel to
//   r_j = c'_j ((beta_j f_j - f_{j-2} - rho_j f_{j+2}) / lam - rho_j r_{j+2}),
//   x_j = r_j - c'_j x_{j-2},
// rho_j = (j-1)/(j+1), beta_j = 2j/(j+1) (1/6 and 2/3 at j = 2; zero in the
// truncated last rows): two first-order recurrences per parity class without
// a division.  A chunk solves them with zero inflow (P), keeps its response
// PM to the two rows above it and N to the two rows below it, and one warp
// walks the chunk summaries, a lane per parity, column and pencil: down for the
// inflow X from above, up for the inflow Y from below as Yp + y Yq with the
// class's first unknown y, which the boundary row (the sum over the class)
// fixes.  Then
//   x_j = P_j + PM_j X + N_j Y.
// |c'| and |c' rho| are below 1 (diagonally dominant rows), so every response
// decays -- but at the two truncated last rows, whose c' = -lam / (4 m (m + 1)),
// m = j - 1, passes 1 at large lam: they feed no row but the boundary's, and
// the reference's order has them so too.  phi_h (zero forcing, wall values 1)
// is Yq N / sum Q of the same walk; v_h is a third column of the v solve, and
// the wall slopes of v are sums of the same walk.  A Chebyshev derivative pair
// (D, D^2) is one walk of chunk sums.
//
// What bounds it (ncu at 192x129x160, R = 6): the latency of a CTA at 12 warps
// per SM.  It issues 19 % of the time; the barriers around the walks, in which
// one warp of four works, come first among the stalls (3.4 per issue), its
// loads second (2.6); FP64 pipe 14 %, DRAM 25 %.  Per
// launch, before (the better of one thread and one warp per pencil) and now:
// 48x65x48 60 -> 12 us, 64x97x64 62 -> 23, 192x129x160 591 -> 178,
// 384x193x384 1810 -> 1250, 64x257x64 1140 -> 67, 192x257x160 1320 -> 375,
// 384x257x288 1930 -> 1240.
#pragma once
#include "press.cuh"
#include "step3.cuh"

namespace sb {

constexpr int PC_TP = 4;                     // pencils per CTA
constexpr int PC_MAXG = 28;                  // chunks per pencil, a multiple of PC_WB
constexpr int PC_NT = PC_TP * PC_MAXG;       // threads per CTA at most
constexpr int PC_S = PC_NT | 1;              // stride of the exchange area: odd, so a walk's columns spread over the banks
constexpr int PC_AREA = 38;                  // exchange area, doubles per thread
constexpr int PC_WB = 4;                     // chunks a walk reads ahead of its chain
// rows per chunk: even, so that a row's class is its parity everywhere
constexpr int PC_MAX_R = 10;
// Resident CTAs per SM the register budget of k_pencil_c is sized for.  R = 4:
// four (128 registers, no spills), so that the 512 CTAs of 64x97x64 are
// resident at once (0.028 -> 0.021 ms).  R = 6, 8: three (168 registers, 20 and
// 32 bytes spilled); at four they spill more (192x129x160 0.16 -> 0.18 ms).
// R = 10: two, all that its 79 KB of shared memory a CTA leave room for; held
// to 168 registers all the same it spilled 328 bytes (384x257x288 1.46 -> 1.24
// ms, 192x257x160 0.44 -> 0.38, 64x257x64 0.077 -> 0.067).
constexpr int pc_minb(int r) { return r == 4 ? 4 : r == 10 ? 2 : 3; }
// the same of k_press_c, which spills nowhere
constexpr int pc_press_minb(int r) { return r == 4 ? 4 : 3; }

// c'_j of (D^2 - lam) for every stored kx and 0 <= |kz| <= nz/2: out[j][pa],
// pa = |kz| nx2 + kx; lam = k^2 + shift.  One thread per column and parity.
static __global__ void __launch_bounds__(128) k_tau_coef(double* __restrict__ out, Dims g,
                                                         const double* __restrict__ alfa,
                                                         const double* __restrict__ beta, double shift) {
  const int na = (g.nz / 2 + 1) * g.nx2;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int pa = t % na, par = t / na;
  if (par > 1) return;
  const int n = g.nyp;
  const double a = alfa[pa % g.nx2], b = beta[pa / g.nx2];
  const double lam = a * a + b * b + shift;
  double q = 0.0;  // c' two rows above
  // rows j = n-1 .. 2 of this parity (1-based row i = j + 1, factor row m = j - 1)
  for (int j = ((n - 1) & 1) == par ? n - 1 : n - 2; j >= 2; j -= 2) {
    const int m = j - 1, i = j + 1;
    const double c = __ldg(&kTauGlobal.c[m]) * lam;
    if (i >= n - 1) {
      q = 0.0;  // the two truncated rows (d = 1) do not enter the rows below
      out[(size_t)j * na + pa] = c;
    } else {
      const double d = 1.0 + __ldg(&kTauGlobal.d[m]) * lam;
      const double e = __ldg(&kTauGlobal.e[m]) * lam;
      q = c * (1.0 / ((i >= n - 3) ? d : d - q * e));
      out[(size_t)j * na + pa] = q;
    }
  }
  out[(size_t)par * na + pa] = 0.0;
}

// {rho_j, beta_j} of every row (zero where the truncated system has no term)
inline void pc_row_table(int n, std::vector<double2>& t) {
  t.assign((size_t)n + PC_WB * PC_MAX_R, double2{0.0, 0.0});
  for (int j = 2; j <= n - 3; ++j) {
    t[j].y = (j == 2) ? 2.0 / 3.0 : 2.0 * j / (j + 1.0);
    if (j <= n - 5) t[j].x = (j == 2) ? 1.0 / 6.0 : (j - 1.0) / (j + 1.0);
  }
}

// The exchange area: value v of chunk c and pencil q at [v][c * PC_TP + q],
// the stride a constant so that v is an immediate offset.
struct PcArea {
  double* p;
  __device__ __forceinline__ double& at(int v, int t) const { return p[v * PC_S + t]; }
};

// 8-byte asynchronous copy to shared memory (zero when !in)
__device__ __forceinline__ void pc_copy8(double* dst, const double* src, bool in) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(in ? 8 : 0) : "memory");
}
__device__ __forceinline__ void pc_copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Element of a field at a byte offset below 4 GB (one offset register serves
// every field of a row): a context holds about fifty complex fields, so one of
// 4 GB does not fit a GPU of 180 GB.
template <class T>
__device__ __forceinline__ T& pc_at(void* base, unsigned off) {
  return *reinterpret_cast<T*>(reinterpret_cast<char*>(base) + off);
}

// Chunk solve with zero inflow: f[q] becomes P, PM and N as above (N of
// chunk 0: the response to the first unknowns, rows 0 and 1).  cp: c' of row
// r at cp[r PC_NT].  The halo rows of f come from the area: values 4 q +
// {0, 1} rows 0, 1, {2, 3} rows R - 2, R - 1 of each chunk.
template <int R, int NC>
__device__ __forceinline__ void pc_local(double (&f)[NC][R], double (&PM)[R], double (&N)[R],
                                         const double* __restrict__ cp, const double2* __restrict__ tab, double il,
                                         const PcArea& A, int t, bool below, bool above) {
  double fp0[NC], fp1[NC];  // f_{r+1}, f_{r+2} before they are overwritten
#pragma unroll
  for (int q = 0; q < NC; ++q) {
    fp1[q] = above ? A.at(4 * q + 1, t + PC_TP) : 0.0;
    fp0[q] = above ? A.at(4 * q + 0, t + PC_TP) : 0.0;
  }
#pragma unroll
  for (int r = R - 1; r >= 0; --r) {
    const double2 tb = __ldg(&tab[r]);
    const double c = cp[r * PC_NT], cro = c * tb.x, cl = c * il;
    PM[r] = (r + 2 < R) ? -cro * PM[(r + 2 < R) ? r + 2 : 0] : -cro;
#pragma unroll
    for (int q = 0; q < NC; ++q) {
      const double fm = (r >= 2) ? f[q][(r >= 2) ? r - 2 : 0] : (below ? A.at(4 * q + 2 + r, t - PC_TP) : 0.0);
      const double f0 = f[q][r];
      double u = cl * fma_(-tb.x, fp1[q], fma_(tb.y, f0, -fm));
      if (r + 2 < R) u = fma_(-cro, f[q][(r + 2 < R) ? r + 2 : 0], u);
      f[q][r] = u;
      fp1[q] = fp0[q];
      fp0[q] = f0;
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const double c = -cp[r * PC_NT];
    if (r < 2) {
      N[r] = below ? c : 1.0;
    } else {
      N[r] = c * N[(r >= 2) ? r - 2 : 0];
      PM[r] = fma_(c, PM[(r >= 2) ? r - 2 : 0], PM[r]);
#pragma unroll
      for (int q = 0; q < NC; ++q) f[q][r] = fma_(c, f[q][(r >= 2) ? r - 2 : 0], f[q][r]);
    }
  }
}

// Summary of a chunk solve, class s (rows r = s, s + 2, ..) at value s VS:
// per column u (first row), P (last row), SP (sum), [KP (sum of k^2 P)]; then
// M, PM, SPM, [KPM], N, SN, [KN].
template <int NC, bool K>
struct PcSum {
  static constexpr int per = K ? 4 : 3;
  static constexpr int shared = NC * per;
  static constexpr int VS = NC * per + (K ? 7 : 5);
  static constexpr int oM = shared, oPM = shared + 1, oSPM = shared + 2, oKPM = shared + 3;
  static constexpr int oN = shared + (K ? 4 : 3), oSN = oN + 1, oKN = oN + 2;
};

template <int R, int NC, bool K>
__device__ __forceinline__ void pc_summary(const double (&f)[NC][R], const double (&PM)[R], const double (&N)[R],
                                           const PcArea& A, int t, double dj0) {
  typedef PcSum<NC, K> S;
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const int last = R - 2 + s;
    const int b = s * S::VS;
#pragma unroll
    for (int q = 0; q < NC; ++q) {
      double sp = 0.0, kp = 0.0;
#pragma unroll
      for (int r = s; r < R; r += 2) {
        sp += f[q][r];
        if (K) {
          const double k = dj0 + (double)r;
          kp = fma_(k * k, f[q][r], kp);
        }
      }
      A.at(b + q * S::per + 0, t) = f[q][s];
      A.at(b + q * S::per + 1, t) = f[q][last];
      A.at(b + q * S::per + 2, t) = sp;
      if (K) A.at(b + q * S::per + 3, t) = kp;
    }
    double sm = 0.0, sn = 0.0, km = 0.0, kn = 0.0;
#pragma unroll
    for (int r = s; r < R; r += 2) {
      sm += PM[r];
      sn += N[r];
      if (K) {
        const double k = dj0 + (double)r;
        km = fma_(k * k, PM[r], km);
        kn = fma_(k * k, N[r], kn);
      }
    }
    A.at(b + S::oM, t) = PM[s];
    A.at(b + S::oPM, t) = PM[last];
    A.at(b + S::oSPM, t) = sm;
    A.at(b + S::oN, t) = N[last];
    A.at(b + S::oSN, t) = sn;
    if (K) {
      A.at(b + S::oKPM, t) = km;
      A.at(b + S::oKN, t) = kn;
    }
  }
}

struct PcClass {
  double p, q, kp, kq;
};

// The walks of both parities (one warp: lane = (parity * 4 + column) * PC_TP +
// pencil).  Leaves X in the u slots, Yp in the P slots and Yq in the N slot of
// each chunk; the class's sums P + Q y of x (p, q) and of k^2 x (kp, kq; K),
// which fix its first unknown y, go to the caller.  The
// chains are FP64 latencies; the summaries of PC_WB chunks are read ahead.
template <int NC, bool K>
__device__ __forceinline__ PcClass pc_walk(const PcArea& A, int G, int lane) {
  typedef PcSum<NC, K> S;
  const int q = lane % PC_TP, col = (lane / PC_TP) & 3, par = lane / (4 * PC_TP);
  const bool own = col < NC;
  // this lane's column (shared values at fixed offsets from column 0)
  double* b0 = A.p + q + par * (S::VS * PC_S);
  double* bc = b0 + (own ? col : 0) * (S::per * PC_S);
  double X = 0.0;
  for (int c0 = G - PC_WB; c0 >= 0; c0 -= PC_WB) {
    const int o = c0 * PC_TP;
    double u[PC_WB], m[PC_WB], x[PC_WB];
#pragma unroll
    for (int i = PC_WB - 1; i >= 0; --i) {
      u[i] = bc[o + i * PC_TP];
      m[i] = b0[o + i * PC_TP + S::oM * PC_S];
    }
#pragma unroll
    for (int i = PC_WB - 1; i >= 0; --i) {
      x[i] = X;
      X = fma_(m[i], X, u[i]);
    }
    __syncwarp();  // the lanes beyond the columns read column 0's slots
    if (own) {
#pragma unroll
      for (int i = 0; i < PC_WB; ++i) bc[o + i * PC_TP] = x[i];
    }
  }
  __syncwarp();
  double Yp = 0.0, Yq = 1.0, Sp = 0.0, Sq = 0.0, lp = 0.0, lq = 0.0;
  for (int c0 = 0; c0 < G; c0 += PC_WB) {
    const int o = c0 * PC_TP;
    double pe[PC_WB], sp[PC_WB], kp[PC_WB], ne[PC_WB], sn[PC_WB], kn[PC_WB], yp[PC_WB], yq[PC_WB];
#pragma unroll
    for (int i = 0; i < PC_WB; ++i) {
      const double* b = bc + o + i * PC_TP;
      const double* bs = b0 + o + i * PC_TP;
      const double Xc = b[0];
      pe[i] = fma_(bs[S::oPM * PC_S], Xc, b[PC_S]);
      sp[i] = fma_(bs[S::oSPM * PC_S], Xc, b[2 * PC_S]);
      ne[i] = bs[S::oN * PC_S];
      sn[i] = bs[S::oSN * PC_S];
      if (K) {
        kp[i] = fma_(bs[S::oKPM * PC_S], Xc, b[3 * PC_S]);
        kn[i] = bs[S::oKN * PC_S];
      }
    }
#pragma unroll
    for (int i = 0; i < PC_WB; ++i) {
      yp[i] = Yp;
      yq[i] = Yq;
      Yp = fma_(ne[i], Yp, pe[i]);
      Yq = ne[i] * Yq;
    }
#pragma unroll
    for (int i = 0; i < PC_WB; ++i) {
      Sp += fma_(sn[i], yp[i], sp[i]);
      Sq = fma_(sn[i], yq[i], Sq);
      if (K) {
        lp += fma_(kn[i], yp[i], kp[i]);
        lq = fma_(kn[i], yq[i], lq);
      }
    }
    __syncwarp();
    if (own) {
#pragma unroll
      for (int i = 0; i < PC_WB; ++i) bc[o + i * PC_TP + PC_S] = yp[i];
    }
    if (col == 0) {
#pragma unroll
      for (int i = 0; i < PC_WB; ++i) b0[o + i * PC_TP + S::oN * PC_S] = yq[i];
    }
  }
  return PcClass{Sp, Sq, lp, lq};
}

// x_j = P + PM X + N Y of the chunk's rows, in f
template <int R, int NC, bool K>
__device__ __forceinline__ void pc_finish(double (&f)[NC][R], const double (&PM)[R], const double (&N)[R],
                                          const PcArea& A, const double* __restrict__ ysm, int t, int q) {
  typedef PcSum<NC, K> S;
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const int b = s * S::VS;
    const double Yq = A.at(b + S::oN, t);
    #pragma unroll
    for (int k = 0; k < NC; ++k) {
      const double X = A.at(b + k * S::per, t);
      const double Y = fma_(ysm[(s * 4 + k) * PC_TP + q], Yq, A.at(b + k * S::per + 1, t));
#pragma unroll
      for (int r = s; r < R; r += 2) f[k][r] = fma_(N[r], Y, fma_(PM[r], X, f[k][r]));
    }
  }
}

// Chunk sums of a derivative pair: a_s = sum of 2 j x_j over class s, b_s =
// sum of 2 j (D x)_j with zero inflow, at values 4 k + {a_0, a_1, b_0, b_1}
template <int R>
__device__ __forceinline__ void pc_dsum(const double (&x)[R], const PcArea& A, int k, int t, double w0) {
  double T[2] = {0.0, 0.0}, U[2] = {0.0, 0.0};
#pragma unroll
  for (int r = R - 1; r >= 0; --r) {
    const double w = w0 + (double)(2 * r);
    U[r & 1] = fma_(w, T[1 - (r & 1)], U[r & 1]);
    T[r & 1] = fma_(w, x[r], T[r & 1]);
  }
  A.at(4 * k + 0, t) = T[0];
  A.at(4 * k + 1, t) = T[1];
  A.at(4 * k + 2, t) = U[0];
  A.at(4 * k + 3, t) = U[1];
}

// Suffix walk of a derivative pair for one pencil, column and parity: the
// sums a of this parity and the sums b of the other, which a drives, become
// the inflow from the chunks above.
template <int R>
__device__ __forceinline__ void pc_dwalk(const PcArea& A, int G, int k, int par, int q) {
  double C = 0.0, E = 0.0;
  // sum of 2 j over the other parity's rows of a chunk (rows c R + 1 - par,
  // + 2, ...), from the last chunk down
  double kk = (double)(R * (G - 1) * R) + (double)((R / 2) * (R / 2 - 1) * 2 + (1 - par) * R);
  double* a = A.p + (4 * k + par) * PC_S + q;
  double* b = A.p + (4 * k + 3 - par) * PC_S + q;
  for (int c0 = G - PC_WB; c0 >= 0; c0 -= PC_WB) {
    const int o = c0 * PC_TP;
    double av[PC_WB], bv[PC_WB], ao[PC_WB], bo[PC_WB];
#pragma unroll
    for (int i = PC_WB - 1; i >= 0; --i) {
      av[i] = a[o + i * PC_TP];
      bv[i] = b[o + i * PC_TP];
    }
#pragma unroll
    for (int i = PC_WB - 1; i >= 0; --i) {
      ao[i] = C;
      bo[i] = E;
      E += fma_(kk, C, bv[i]);
      C += av[i];
      kk -= (double)(R * R);
    }
#pragma unroll
    for (int i = 0; i < PC_WB; ++i) {
      a[o + i * PC_TP] = ao[i];
      b[o + i * PC_TP] = bo[i];
    }
  }
}

// Suffix walk of one derivative's chunk sums (value v of the area)
__device__ __forceinline__ void pc_dwalk1(const PcArea& A, int G, int v, int q) {
  double C = 0.0;
  double* a = A.p + v * PC_S + q;
  for (int c0 = G - PC_WB; c0 >= 0; c0 -= PC_WB) {
    const int o = c0 * PC_TP;
    double x[PC_WB], s[PC_WB];
#pragma unroll
    for (int i = PC_WB - 1; i >= 0; --i) x[i] = a[o + i * PC_TP];
#pragma unroll
    for (int i = PC_WB - 1; i >= 0; --i) {
      s[i] = C;
      C += x[i];
    }
#pragma unroll
    for (int i = 0; i < PC_WB; ++i) a[o + i * PC_TP] = s[i];
  }
}

// kx = kz = 0 in one CTA (the algebra of k_mean, linearbl.f:1214-1470 tau
// branch, ibc = 0, and the next partial right-hand side :1712-1733): U and W
// from (D^2 - lam) U = f_u, (D^2 - lam) W = f_w with lam = 2 Re/(a_n + b_n).
// Under constant flux the reference solves for U three times (px, 2 px, the
// corrected px); the system being linear, one solve for f_u, f_w and the unit
// forcing G of row 0 gives the same three solutions as U + s G.  Pencil 0 of
// the tile works, the others carry zeros.
template <int R>
__device__ __forceinline__ void pc_mean(const MeanArgs& M, const Dims& g, double re, const RKc& rk,
                                        const double* __restrict__ CL, const double2* __restrict__ rows, int G,
                                        const PcArea& A, double* cs, double* ysm) {
  __shared__ double shift;
  const int tid = threadIdx.x, nt = G * PC_TP;
  const bool chunk = tid < nt;
  const int q = tid % PC_TP, c = chunk ? tid / PC_TP : 0, t = chunk ? tid : q;
  const int n = g.nyp, j0 = c * R;
  const size_t NP = g.NP;
  const int na = (g.nz / 2 + 1) * g.nx2;
  const double c1 = 2.0 * re / (rk.an + rk.bn) * rk.an, lam = 2.0 * re / (rk.an + rk.bn);
  const bool work = chunk && q == 0;
  double px = M.scal[0];
  double h1[R], h3[R], f[4][R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int j = j0 + r;
    h1[r] = h3[r] = f[0][r] = f[1][r] = f[2][r] = f[3][r] = 0.0;
    double cp = 0.0;
    if (chunk && j < n) {
      cp = CL[(size_t)j * na];
      if (q == 0) {
        h1[r] = M.H1[(size_t)j * NP].x;
        h3[r] = M.H3[(size_t)j * NP].x;
        f[0][r] = M.puw[j] - c1 * h1[r];
        f[1][r] = M.puw[n + j] - c1 * h3[r];
        if (j == 0) {
          f[0][r] += 2.0 * re * px;
          f[2][r] = 1.0;
        }
      }
    }
    if (chunk) cs[r * PC_NT] = cp;
  }
  if (chunk) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      A.at(4 * k + 0, t) = f[k][0];
      A.at(4 * k + 1, t) = f[k][1];
      A.at(4 * k + 2, t) = f[k][R - 2];
      A.at(4 * k + 3, t) = f[k][R - 1];
    }
  }
  __syncthreads();
  {
    double PM[R], N[R];
    pc_local<R, 4>(f, PM, N, cs, rows + j0, 1.0 / lam, A, t, c > 0, c + 1 < G);
    __syncthreads();
    if (chunk) pc_summary<R, 4, false>(f, PM, N, A, t, (double)j0);
    __syncthreads();
    if (tid < 32) {
      const PcClass w = pc_walk<4, false>(A, G, tid);
      ysm[tid] = -w.p / w.q;
    }
    __syncthreads();
    pc_finish<R, 4, false>(f, PM, N, A, ysm, t, q);
  }
  __syncthreads();
  if (M.cflux) {
    // flux m = sum over even j of -U_j 2/(j^2 - 1) of U and of G
    double mu = 0.0, mg = 0.0;
#pragma unroll
    for (int r = 0; r < R; r += 2) {
      const int j = j0 + r;
      const double wj = (j < n) ? -2.0 / ((double)j * (double)j - 1.0) : 0.0;
      mu = fma_(f[0][r], wj, mu);
      mg = fma_(f[2][r], wj, mg);
    }
    if (chunk) {
      A.at(0, t) = mu;
      A.at(1, t) = mg;
    }
    __syncthreads();
    if (tid == 0) {
      double su = 0.0, sg = 0.0;
      for (int cc = 0; cc < G; ++cc) {
        su += A.at(0, cc * PC_TP);
        sg += A.at(1, cc * PC_TP);
      }
      const double m1 = su, m2 = su + 2.0 * re * px * sg;  // U, then U with 2 Re px more in row 0
      const double pxn = px * (1.0 + (M.scal[1] - m1) / (m2 - m1));
      shift = 2.0 * re * (pxn - px);
      M.scal[0] = pxn;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r) f[0][r] = fma_(shift, f[2][r], f[0][r]);
  }
  const double w0 = 2.0 * (double)j0;
  if (chunk) {
    pc_dsum<R>(f[0], A, 0, t, w0);
    pc_dsum<R>(f[1], A, 1, t, w0);
  }
  __syncthreads();
  if (tid < 4 * PC_TP) pc_dwalk<R>(A, G, tid / (2 * PC_TP), (tid / PC_TP) & 1, tid % PC_TP);
  __syncthreads();
  double T[2][2], U[2][2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    T[k][0] = A.at(4 * k + 0, t);
    T[k][1] = A.at(4 * k + 1, t);
    U[k][0] = A.at(4 * k + 2, t);
    U[k][1] = A.at(4 * k + 3, t);
  }
  const double c1n = 2.0 * re / (rk.anp1 + rk.bnp1);
  const double c2 = 2.0 * re * rk.bnp1 / (rk.anp1 + rk.bnp1);
#pragma unroll
  for (int r = R - 1; r >= 0; --r) {
    const int j = j0 + r, s = r & 1;
    const double w = w0 + (double)(2 * r);
    double d[2], dd[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      d[k] = T[k][1 - s];
      dd[k] = U[k][1 - s];
      U[k][s] = fma_(w, d[k], U[k][s]);
      T[k][s] = fma_(w, f[k][r], T[k][s]);
      if (j == 0) {
        d[k] *= 0.5;
        dd[k] *= 0.5;
      }
    }
    if (work && j < n) {
      const size_t o = (size_t)j * NP;
      M.OU[o] = double2{f[0][r], 0.0};
      M.OW[o] = double2{f[1][r], 0.0};
      M.OV[o] = double2{0, 0.0};
      M.OX[o] = double2{d[1], 0.0};
      M.OZ[o] = double2{(-d[0]), 0.0};
      M.PV[o] = double2{0.0, 0.0};
      M.PW[o] = double2{0.0, 0.0};
      M.puw[j] = -dd[0] - c1n * f[0][r] - c2 * h1[r];
      M.puw[n + j] = -dd[1] - c1n * f[1][r] - c2 * h3[r];
    }
  }
}

// own_mean: one more CTA, the first, solves the kx = kz = 0 pencil.
template <int R>
__global__ void __launch_bounds__((PC_NT + 31) / 32 * 32, pc_minb(R))
    k_pencil_c(PencilBufs B, Dims g, const double* __restrict__ alfa, const double* __restrict__ beta, double re,
               RKc rk, const double* __restrict__ CL, const double* __restrict__ CV,
               const double2* __restrict__ rows, int G, MeanArgs M, int own_mean) {
  extern __shared__ __align__(16) unsigned char pc_smem[];
  __shared__ double ysm[2 * 4 * PC_TP];   // first unknowns by parity and column
  __shared__ double sqi[2 * PC_TP];       // 1 / sum Q of the lam solve
  __shared__ double cvs[2 * 2 * PC_TP];   // amount of v_h by parity, real and imaginary
  const int tid = threadIdx.x, nt = G * PC_TP;
  const bool chunk = tid < nt;
  const int q = tid % PC_TP, c = chunk ? tid / PC_TP : 0;
  const int t = chunk ? tid : q;
  const PcArea A{reinterpret_cast<double*>(pc_smem)};
  if (own_mean && blockIdx.x == 0) {
    pc_mean<R>(M, g, re, rk, CL, rows, G, A, A.p + PC_AREA * PC_S + t, ysm);
    return;
  }
  // the chunk's forcing rows h_v, h_omega, kept for the next right-hand sides
  double* hs = A.p + PC_AREA * PC_S + t;
  double* cs = hs + 4 * R * PC_NT;  // the chunk's c', first of the lam solve
  const int n = g.nyp;
  const size_t NP = g.NP;
  const int p = g.p0 + (blockIdx.x - own_mean) * PC_TP + q;
  const int pc = min(p, g.p1 - 1);
  const int kx = pc % g.nx2, iz = pc / g.nx2;
  const bool act = chunk && p < g.p1 && iz != g.zodd && p != 0;
  const double a = alfa[kx], be = beta[iz];
  const double k2 = (pc == 0) ? 1.0 : a * a + be * be;
  const double k2i = 1.0 / k2;
  const double lam = k2 + 2.0 * re / (rk.an + rk.bn);
  const double c1 = 2.0 * re / (rk.an + rk.bn) * rk.an;
  const int na = (g.nz / 2 + 1) * g.nx2;
  const int pa = min(iz, g.nz - iz) * g.nx2 + kx;
  const int j0 = c * R;
  const double dj0 = (double)j0, w0 = 2.0 * dj0;
  const bool below = c > 0, above = c + 1 < G;
  const bool in_last = chunk && j0 + R <= n;  // every row of the chunk is in the pencil
  auto row_in = [&](int r) { return in_last || (chunk && j0 + r < n); };
  const unsigned so = (unsigned)NP, o0 = (unsigned)j0 * so + (unsigned)pc;  // row r at element o0 + r so
  auto load_coef = [&](const double* __restrict__ C) {
    const double* src = C + (size_t)j0 * na + pa;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const bool in = row_in(r);
      if (chunk) pc_copy8(cs + r * PC_NT, in ? src + (size_t)r * na : C, in);
    }
  };
  // Up to six rows per chunk the rows of H, p_v, p_omega are asked for all at
  // once, into this thread's own slots of the exchange area and of the
  // forcing rows, which nothing else uses yet (192x129x160: 185 -> 178 us);
  // longer chunks measured slower with it (384x193x384: 1.25 -> 1.34 ms) and
  // load row by row.  Word w of field k (H1, H3, p_v, p_omega, H2) at 2 k + w.
  constexpr bool STAGE = R <= 6;
  static_assert(!STAGE || 10 * R <= PC_AREA + 4 * R, "the staged rows fit in the slots they borrow");
  auto staged = [&](int r, int w) -> double& {
    const int i = 10 * r + w;
    return i < PC_AREA ? A.at(i, t) : hs[(i - PC_AREA) * PC_NT];
  };
  double2* const field[5] = {B.H1, B.H3, B.PV, B.PW, B.H2};
  if (STAGE && chunk) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const bool in = row_in(r);
      const unsigned o = in ? (o0 + (unsigned)r * so) * 16u : 0u;
#pragma unroll
      for (int k = 0; k < 5; ++k)
#pragma unroll
        for (int w = 0; w < 2; ++w) pc_copy8(&staged(r, 2 * k + w), &pc_at<const double>(field[k], o + 8u * w), in);
    }
  }
  load_coef(CL);
  auto hv = [&](int r, int k) -> double& { return hs[(4 * r + k) * PC_NT]; };
  auto hom = [&](int r, int k) -> double& { return hs[(4 * r + 2 + k) * PC_NT]; };

  // ---- forcing (linearbl.f:303-340): g = i alpha H1 + i beta H3, h_v =
  // -(D g + k^2 H2), h_omega = i beta H1 - i alpha H3, f = p - c1 h
  double f[4][R];  // f_v re, im, f_omega re, im
  {
    double gx[R], gy[R], h2x[R], h2y[R];
    double hx_[STAGE ? R : 1], hy_[STAGE ? R : 1];
    if (STAGE) pc_copy_wait();
#pragma unroll
    for (int r = 0; r < R; ++r) {
      double2 h1{0.0, 0.0}, h2{0.0, 0.0}, h3{0.0, 0.0}, pv{0.0, 0.0}, pw{0.0, 0.0};
      if constexpr (STAGE) {
        auto get = [&](int k) { return double2{staged(r, 2 * k), staged(r, 2 * k + 1)}; };
        h1 = get(0);
        h3 = get(1);
        pv = get(2);
        pw = get(3);
        h2 = get(4);
      } else if (row_in(r)) {
        const unsigned o = (o0 + (unsigned)r * so) * 16u;
        h1 = pc_at<const double2>(B.H1, o);
        h2 = pc_at<const double2>(B.H2, o);
        h3 = pc_at<const double2>(B.H3, o);
        pv = pc_at<const double2>(B.PV, o);
        pw = pc_at<const double2>(B.PW, o);
      }
      gx[r] = -a * h1.y - be * h3.y;
      gy[r] = a * h1.x + be * h3.x;
      const double hx = -be * h1.y + a * h3.y, hy = be * h1.x - a * h3.x;
      if constexpr (STAGE) {
        hx_[r] = hx;  // into its slots once every staged row is read
        hy_[r] = hy;
      } else if (chunk) {
        hom(r, 0) = hx;
        hom(r, 1) = hy;
      }
      f[2][r] = pw.x - c1 * hx;
      f[3][r] = pw.y - c1 * hy;
      h2x[r] = k2 * h2.x;
      h2y[r] = k2 * h2.y;
      f[0][r] = pv.x;
      f[1][r] = pv.y;
    }
    if (STAGE && chunk) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        hom(r, 0) = hx_[r];
        hom(r, 1) = hy_[r];
      }
    }
    // D g: chunk sums by class, suffix walk, inflow
    double T0x = 0.0, T1x = 0.0, T0y = 0.0, T1y = 0.0;
#pragma unroll
    for (int r = R - 1; r >= 0; --r) {
      const double w = w0 + (double)(2 * r);
      double& Tx = (r & 1) ? T1x : T0x;
      double& Ty = (r & 1) ? T1y : T0y;
      Tx = fma_(w, gx[r], Tx);
      Ty = fma_(w, gy[r], Ty);
    }
    if (chunk) {
      A.at(0, t) = T0x;
      A.at(1, t) = T1x;
      A.at(2, t) = T0y;
      A.at(3, t) = T1y;
    }
    __syncthreads();
    if (tid < 4 * PC_TP) {
      // one lane per pencil, component and parity
      pc_dwalk1(A, G, tid / PC_TP, tid % PC_TP);
    }
    __syncthreads();
    double S0x = A.at(0, t), S1x = A.at(1, t), S0y = A.at(2, t), S1y = A.at(3, t);
#pragma unroll
    for (int r = R - 1; r >= 0; --r) {
      const double w = w0 + (double)(2 * r);
      double dx = (r & 1) ? S0x : S1x, dy = (r & 1) ? S0y : S1y;
      if (r & 1) {
        S1x = fma_(w, gx[r], S1x);
        S1y = fma_(w, gy[r], S1y);
      } else {
        S0x = fma_(w, gx[r], S0x);
        S0y = fma_(w, gy[r], S0y);
      }
      if (r == 0 && j0 == 0) {
        dx *= 0.5;
        dy *= 0.5;
      }
      const double vx = -(dx + h2x[r]), vy = -(dy + h2y[r]);
      if (chunk) {
        hv(r, 0) = vx;
        hv(r, 1) = vy;
      }
      const bool in = row_in(r);
      f[0][r] = in ? f[0][r] - c1 * vx : 0.0;
      f[1][r] = in ? f[1][r] - c1 * vy : 0.0;
    }
  }
  __syncthreads();  // every thread has read its inflow of D g
  double om[2][R];          // omega_y
  double vv[3][R];          // phi re, im, phi_h; then v re, im, v_h
  // ---- phi (particular), omega_y: (D^2 - lam) psi = f (linearbl.f:625-626)
  {
    double PM[R], N[R];
    if (chunk) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        A.at(4 * k + 0, t) = f[k][0];
        A.at(4 * k + 1, t) = f[k][1];
        A.at(4 * k + 2, t) = f[k][R - 2];
        A.at(4 * k + 3, t) = f[k][R - 1];
      }
    }
    pc_copy_wait();
    __syncthreads();
    pc_local<R, 4>(f, PM, N, cs, rows + j0, 1.0 / lam, A, t, below, above);
    load_coef(CV);  // under the walk
    __syncthreads();
    if (chunk) pc_summary<R, 4, false>(f, PM, N, A, t, dj0);
    __syncthreads();
    if (tid < 32) {
      const PcClass w = pc_walk<4, false>(A, G, tid);
      ysm[tid] = -w.p / w.q;  // zero wall values
      if (((tid / PC_TP) & 3) == 0) sqi[tid / (4 * PC_TP) * PC_TP + q] = 1.0 / w.q;
    }
    __syncthreads();
    pc_finish<R, 4, false>(f, PM, N, A, ysm, t, q);
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const double yh = A.at(s * PcSum<4, false>::VS + PcSum<4, false>::oN, t) * sqi[s * PC_TP + q];
#pragma unroll
      for (int r = s; r < R; r += 2) {
        vv[2][r] = N[r] * yh;
        vv[0][r] = f[0][r];
        vv[1][r] = f[1][r];
        om[0][r] = f[2][r];
        om[1][r] = f[3][r];
      }
    }
  }
  __syncthreads();
  // ---- v from phi: (D^2 - k^2) v = phi (linearbl.f:1000-1001), and v_h
  {
    double PM[R], N[R];
    if (chunk) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        A.at(4 * k + 0, t) = vv[k][0];
        A.at(4 * k + 1, t) = vv[k][1];
        A.at(4 * k + 2, t) = vv[k][R - 2];
        A.at(4 * k + 3, t) = vv[k][R - 1];
      }
    }
    pc_copy_wait();
    __syncthreads();
    pc_local<R, 3>(vv, PM, N, cs, rows + j0, k2i, A, t, below, above);
    __syncthreads();
    if (chunk) pc_summary<R, 3, true>(vv, PM, N, A, t, dj0);
    __syncthreads();
    if (tid < 32) {
      const PcClass w = pc_walk<3, true>(A, G, tid);
      const double y = -w.p / w.q, sl = fma_(y, w.kq, w.kp);
      // dv/dy = 0 at the walls (linearbl.f:1020-1085): the class sum of k^2
      // v_k is the slope, which v_h takes out
      const int col = (tid / PC_TP) & 3, par = tid / (4 * PC_TP);
      const double slh = __shfl_sync(0xffffffffu, sl, (par * 4 + 2) * PC_TP + q);
      ysm[tid] = y;
      if (col < 2) cvs[(par * 2 + col) * PC_TP + q] = -sl / slh;
    }
    __syncthreads();
    pc_finish<R, 3, true>(vv, PM, N, A, ysm, t, q);
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int par = r & 1;
    vv[0][r] = fma_(cvs[(par * 2 + 0) * PC_TP + q], vv[2][r], vv[0][r]);
    vv[1][r] = fma_(cvs[(par * 2 + 1) * PC_TP + q], vv[2][r], vv[1][r]);
  }
  __syncthreads();
  // ---- D and D^2 of v and omega_y; u, v, w, omega_x, omega_z (loop 2800,
  // :1193-1212), phi = D^2 v - k^2 v (:1160-1170) and p_omega (:1696-1800)
  if (chunk) {
    pc_dsum<R>(vv[0], A, 0, t, w0);
    pc_dsum<R>(vv[1], A, 1, t, w0);
    pc_dsum<R>(om[0], A, 2, t, w0);
    pc_dsum<R>(om[1], A, 3, t, w0);
  }
  __syncthreads();
  if (tid < 8 * PC_TP) pc_dwalk<R>(A, G, tid / (2 * PC_TP), (tid / PC_TP) & 1, tid % PC_TP);
  __syncthreads();
  const double c1n = 2.0 * re / (rk.anp1 + rk.bnp1);
  const double c2 = 2.0 * re * rk.bnp1 / (rk.anp1 + rk.bnp1);
  const double k2m = k2 - c1n;
  {
    double T[4][2], U[4][2];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      T[k][0] = A.at(4 * k + 0, t);
      T[k][1] = A.at(4 * k + 1, t);
      U[k][0] = A.at(4 * k + 2, t);
      U[k][1] = A.at(4 * k + 3, t);
    }
#pragma unroll
    for (int r = R - 1; r >= 0; --r) {
      const int s = r & 1;
      const double w = w0 + (double)(2 * r);
      const double x[4] = {vv[0][r], vv[1][r], om[0][r], om[1][r]};
      double d[4], dd[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        d[k] = T[k][1 - s];
        dd[k] = U[k][1 - s];
        U[k][s] = fma_(w, d[k], U[k][s]);
        T[k][s] = fma_(w, x[k], T[k][s]);
        if (r == 0 && j0 == 0) {
          d[k] *= 0.5;
          dd[k] *= 0.5;
        }
      }
      const double phx = dd[0] - k2 * x[0], phy = dd[1] - k2 * x[1];
      const bool in = row_in(r);
      if (act && in) {
        const unsigned o = (o0 + (unsigned)r * so) * 16u;
        pc_at<double2>(B.OU, o) = double2{((-a * d[1] + be * x[3]) * k2i), ((a * d[0] - be * x[2]) * k2i)};
        pc_at<double2>(B.OV, o) = double2{x[0], x[1]};
        pc_at<double2>(B.OW, o) = double2{((-a * x[3] - be * d[1]) * k2i), ((a * x[2] + be * d[0]) * k2i)};
        pc_at<double2>(B.OZ, o) = double2{((-be * d[3] + a * phy) * k2i), ((be * d[2] - a * phx) * k2i)};
        pc_at<double2>(B.OX, o) = double2{((-a * d[3] - be * phy) * k2i), ((a * d[2] + be * phx) * k2i)};
        pc_at<double2>(B.PW, o) = double2{-dd[2] + k2m * x[2] - c2 * hom(r, 0), -dd[3] + k2m * x[3] - c2 * hom(r, 1)};
      }
      vv[0][r] = in ? phx : 0.0;
      vv[1][r] = in ? phy : 0.0;
    }
  }
  __syncthreads();
  // ---- D^2 phi and p_v
  if (chunk) {
    pc_dsum<R>(vv[0], A, 0, t, w0);
    pc_dsum<R>(vv[1], A, 1, t, w0);
  }
  __syncthreads();
  if (tid < 4 * PC_TP) pc_dwalk<R>(A, G, tid / (2 * PC_TP), (tid / PC_TP) & 1, tid % PC_TP);
  __syncthreads();
  {
    double T[2][2], U[2][2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      T[k][0] = A.at(4 * k + 0, t);
      T[k][1] = A.at(4 * k + 1, t);
      U[k][0] = A.at(4 * k + 2, t);
      U[k][1] = A.at(4 * k + 3, t);
    }
#pragma unroll
    for (int r = R - 1; r >= 0; --r) {
      const int s = r & 1;
      const double w = w0 + (double)(2 * r);
      double dd[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        dd[k] = U[k][1 - s];
        U[k][s] = fma_(w, T[k][1 - s], U[k][s]);
        T[k][s] = fma_(w, vv[k][r], T[k][s]);
        if (r == 0 && j0 == 0) dd[k] *= 0.5;
      }
      if (act && row_in(r))
        pc_at<double2>(B.PV, (o0 + (unsigned)r * so) * 16u) = double2{-dd[0] + k2m * vv[0][r] - c2 * hv(r, 0),
                                     -dd[1] + k2m * vv[1][r] - c2 * hv(r, 1)};
    }
  }
}

// The pressure's pencils (press.cuh, k_press: the same system and Neumann data,
// bla/linearp.f:77-158) but kx = kz = 0, chunked as above: f = D H2 + (i alpha
// H1 + i beta H3), (D^2 - k^2) x = f with D x at the walls (the class sums of
// k^2 x fix the first unknowns), p = x - E.  The thread-per-pencil kernel took
// 0.58 ms at 192x129x160 for 0.25 GB, one wave of serial walks; this one
// 0.095.
template <int R, class VT>
__global__ void __launch_bounds__((PC_NT + 31) / 32 * 32, pc_press_minb(R))
    k_press_c(PressArgs P, const VT* __restrict__ V, Dims g, const double* __restrict__ CV,
              const double2* __restrict__ rows, int G) {
  extern __shared__ __align__(16) unsigned char pc_smem[];
  __shared__ double ysm[2 * 4 * PC_TP];
  __shared__ double wall[4 * PC_TP];  // D^2 v at y = +1, -1 of each pencil, real and imaginary
  const int tid = threadIdx.x, nt = G * PC_TP;
  const bool chunk = tid < nt;
  const int q = tid % PC_TP, c = chunk ? tid / PC_TP : 0;
  const int t = chunk ? tid : q;
  const PcArea A{reinterpret_cast<double*>(pc_smem)};
  double* cs = A.p + PC_AREA * PC_S + t;
  const int n = g.nyp;
  const size_t NP = g.NP;
  const int p = blockIdx.x * PC_TP + q;
  const int pc = min(p, g.NP - 1);
  const int kx = pc % g.nx2, iz = pc / g.nx2;
  const bool act = chunk && p < g.NP && iz != g.zodd && p != 0;
  const double a = P.alfa[kx], be = P.beta[iz];
  const double k2 = (pc == 0) ? 1.0 : a * a + be * be;
  const int na = (g.nz / 2 + 1) * g.nx2;
  const int pa = min(iz, g.nz - iz) * g.nx2 + kx;
  const int j0 = c * R;
  const double dj0 = (double)j0, w0 = 2.0 * dj0;
  auto row_in = [&](int r) { return chunk && j0 + r < n; };
  double f[2][R];
  // D H2 by the suffix walk, D^2 v at the walls by the quadrature weights
  {
    double hx[R], hy[R], T[4] = {0.0, 0.0, 0.0, 0.0}, S[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int r = 0; r < R; ++r) {
      double2 h{0.0, 0.0}, d{0.0, 0.0};
      if (row_in(r)) {
        const int j = j0 + r;
        const size_t o = (size_t)j * NP + pc;
        h = P.CH2[o];
        d = P.CD[o];
        const VT v = V[o];
        const double w1 = __ldg(&P.wd[j]), w2 = __ldg(&P.wd[n + j]);
        S[0] = fma_((double)v.x, w1, S[0]);
        S[1] = fma_((double)v.x, w2, S[1]);
        S[2] = fma_((double)v.y, w1, S[2]);
        S[3] = fma_((double)v.y, w2, S[3]);
        cs[r * PC_NT] = CV[(size_t)j * na + pa];
      } else if (chunk) {
        cs[r * PC_NT] = 0.0;
      }
      hx[r] = h.x;
      hy[r] = h.y;
      f[0][r] = d.x;
      f[1][r] = d.y;
    }
#pragma unroll
    for (int r = R - 1; r >= 0; --r) {
      const double w = w0 + (double)(2 * r);
      T[r & 1] = fma_(w, hx[r], T[r & 1]);
      T[2 + (r & 1)] = fma_(w, hy[r], T[2 + (r & 1)]);
    }
    if (chunk) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        A.at(i, t) = T[i];
        A.at(4 + i, t) = S[i];
      }
    }
    __syncthreads();
    if (tid < 4 * PC_TP) {
      pc_dwalk1(A, G, tid / PC_TP, q);
    } else if (tid >= 32 - 4 * PC_TP && tid < 32) {
      const int i = (tid - (32 - 4 * PC_TP)) / PC_TP;
      double s = 0.0;
      for (int cc = 0; cc < G; ++cc) s += A.at(4 + i, cc * PC_TP + q);
      wall[i * PC_TP + q] = s;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) T[i] = A.at(i, t);
#pragma unroll
    for (int r = R - 1; r >= 0; --r) {
      const double w = w0 + (double)(2 * r);
      double dx = T[1 - (r & 1)], dy = T[3 - (r & 1)];
      T[r & 1] = fma_(w, hx[r], T[r & 1]);
      T[2 + (r & 1)] = fma_(w, hy[r], T[2 + (r & 1)]);
      if (r == 0 && j0 == 0) {
        dx *= 0.5;
        dy *= 0.5;
      }
      f[0][r] = row_in(r) ? f[0][r] + dx : 0.0;
      f[1][r] = row_in(r) ? f[1][r] + dy : 0.0;
    }
  }
  __syncthreads();
  if (chunk) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      A.at(4 * k + 0, t) = f[k][0];
      A.at(4 * k + 1, t) = f[k][1];
      A.at(4 * k + 2, t) = f[k][R - 2];
      A.at(4 * k + 3, t) = f[k][R - 1];
    }
  }
  __syncthreads();
  double PM[R], N[R];
  pc_local<R, 2>(f, PM, N, cs, rows + j0, 1.0 / k2, A, t, c > 0, c + 1 < G);
  __syncthreads();
  if (chunk) pc_summary<R, 2, true>(f, PM, N, A, t, dj0);
  __syncthreads();
  if (tid < 32) {
    const PcClass w = pc_walk<2, true>(A, G, tid);
    // D x at y = +1, -1: H2 + (D^2 v - k^2 v) / Re - dv/dt (linearp.f:77-150;
    // v at the walls of the last step is zero)
    const int col = (tid / PC_TP) & 1, par = tid / (4 * PC_TP);
    double bc[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const size_t o = (e ? (size_t)(n - 1) * NP : 0) + pc;
      const double2 h = P.PH2[o];
      const double vw = col ? (double)V[o].y : (double)V[o].x;
      bc[e] = (col ? h.y : h.x) * P.cn + (wall[(2 * col + e) * PC_TP + q] - k2 * vw) / P.re - vw * P.c4t;
    }
    const double b = par ? 0.5 * (bc[0] + bc[1]) : 0.5 * (bc[0] - bc[1]);
    ysm[tid] = (b - w.kp) / w.kq;
  }
  __syncthreads();
  pc_finish<R, 2, true>(f, PM, N, A, ysm, t, q);
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (act && row_in(r)) {
      const size_t o = (size_t)(j0 + r) * NP + pc;
      const double2 ce = P.CE[o];
      P.X[o] = double2{f[0][r] - ce.x, f[1][r] - ce.y};
    }
}

// Rows per chunk for ny: 0 when ny is beyond the kernel's range
inline int pencil_chunk_rows(int ny) {
  for (int r = 4; r <= PC_MAX_R; r += 2)
    if ((ny + r - 1) / r <= PC_MAXG) return r;
  return 0;
}

template <int R>
inline void pencil_chunk_n(cudaStream_t s, const PencilBufs& B, const Dims& g, const double* alfa, const double* beta,
                           double re, RKc rk, const double* CL, const double* CV, const double2* rows,
                           const MeanArgs* M) {
  const int G = ((g.nyp + R - 1) / R + PC_WB - 1) / PC_WB * PC_WB, nt = G * PC_TP;
  constexpr int smem = (PC_S * PC_AREA + PC_NT * 5 * R) * (int)sizeof(double);
  cudaFuncSetAttribute(k_pencil_c<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  const unsigned blocks = (unsigned)((g.p1 - g.p0 + PC_TP - 1) / PC_TP) + (M ? 1u : 0u);
  k_pencil_c<R><<<blocks, (nt + 31) / 32 * 32, smem, s>>>(B, g, alfa, beta, re, rk, CL, CV, rows, G,
                                                             M ? *M : MeanArgs{}, M ? 1 : 0);
}

inline bool launch_pencil_chunk(cudaStream_t s, const PencilBufs& B, const Dims& g, const double* alfa, const double* beta,
                         double re, RKc rk, const double* CL, const double* CV, const double2* rows,
                           const MeanArgs* M) {
  switch (pencil_chunk_rows(g.nyp)) {
#define SB_PC_CASE(RR)                                                         \
  case RR:                                                                     \
    pencil_chunk_n<RR>(s, B, g, alfa, beta, re, rk, CL, CV, rows, M); \
    return true;
    SB_PC_CASE(4) SB_PC_CASE(6) SB_PC_CASE(8) SB_PC_CASE(10)
#undef SB_PC_CASE
    default:
      return false;
  }
}

template <int R>
inline void press_chunk_n(cudaStream_t s, const PressArgs& P, const Dims& g, const double* CV, const double2* rows) {
  const int G = ((g.nyp + R - 1) / R + PC_WB - 1) / PC_WB * PC_WB, nt = G * PC_TP;
  constexpr int smem = (PC_S * PC_AREA + PC_NT * R) * (int)sizeof(double);
  const unsigned blocks = (unsigned)((g.NP + PC_TP - 1) / PC_TP);
  if (P.Vf) {
    cudaFuncSetAttribute(k_press_c<R, float2>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    k_press_c<R, float2><<<blocks, (nt + 31) / 32 * 32, smem, s>>>(P, P.Vf, g, CV, rows, G);
  } else {
    cudaFuncSetAttribute(k_press_c<R, double2>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    k_press_c<R, double2><<<blocks, (nt + 31) / 32 * 32, smem, s>>>(P, P.V, g, CV, rows, G);
  }
}

inline bool launch_press_chunk(cudaStream_t s, const PressArgs& P, const Dims& g, const double* CV,
                               const double2* rows) {
  switch (pencil_chunk_rows(g.nyp)) {
#define SB_PC_CASE(RR)                        \
  case RR:                                    \
    press_chunk_n<RR>(s, P, g, CV, rows); \
    return true;
    SB_PC_CASE(4) SB_PC_CASE(6) SB_PC_CASE(8) SB_PC_CASE(10)
#undef SB_PC_CASE
    default:
      return false;
  }
}

}  // namespace sb
