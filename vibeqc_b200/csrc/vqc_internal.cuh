// Shared device-side definitions for the DF-RHF kernels (sm_100a).
//
// Integrals use Rys quadrature (Rys, Dupuis, King, J. Comput. Chem. 4, 154
// (1983)): nodes/weights come from the piecewise polynomial table generated by
// gen_rys_table.py (80-digit Golub-Welsch on Boys moments) and, for large T,
// from the Gauss-Hermite limit.  Two-dimensional integrals follow the Rys
// vertical recurrence in (e0|f0) and the horizontal transfer
// I(i, j+1) = I(i+1, j) + (A - B) I(i, j).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace vqc {

#include "rys_table.inc"
#include "sph_table.inc"

constexpr double kPi = 3.141592653589793238462643383279502884;
// Primitive pairs whose Gaussian-product factor exp(-ab/(a+b) |AB|^2) |c_a c_b|
// is below this are skipped by the 3-centre value and derivative kernels
// (tight primitives on different atoms: 56-72 % of the primitive-pair work
// of (H2O)8-16 in def2-SVP).  The Rys factors multiplying it stay far below
// 1e6 for the basis sets here, so a skipped pair changes an integral by less
// than ~1e-24; values and derivatives skip the same pairs.
constexpr double kPrimPairCut = 1e-30;
constexpr int kMaxL = 4;  // per-shell angular momentum the kernels instantiate

__host__ __device__ constexpr int ncart(int l) { return (l + 1) * (l + 2) / 2; }
__host__ __device__ constexpr int nsph(int l) { return 2 * l + 1; }

// Cartesian -> output-function transforms c_trans[mode][l][row][col] come from
// sph_table.inc: mode 0 = real spherical (PySCF order), mode 1 = normalised
// Cartesian components.

// Nodes and weights on [0, T_asym): degree-RYS_DEG polynomials on intervals of
// width RYS_H.  A warp's threads have different T, so the coefficient loads are
// a gather and the L1 takes about a cycle per thread and load: the table keeps
// the (u, w) pairs of a root together and two powers come with one 32-byte
// load (5 loads a root instead of 20 eight-byte ones).  Powers of x instead of
// a Chebyshev recurrence: one FMA per coefficient instead of an FMA and an
// addition.
__device__ __forceinline__ void rys_poly(const double* __restrict__ c, double x, double& u, double& w) {
  static_assert(RYS_LAYOUT == 2 && RYS_DEG % 2 == 1, "coefficient layout");
  double a[2 * (RYS_DEG + 1)];
#pragma unroll
  for (int k = 0; k < (RYS_DEG + 1) / 2; ++k)
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
        : "=d"(a[4 * k]), "=d"(a[4 * k + 1]), "=d"(a[4 * k + 2]), "=d"(a[4 * k + 3])
        : "l"(c + 4 * k));
  u = a[0];
  w = a[1];
#pragma unroll
  for (int k = 1; k <= RYS_DEG; ++k) {
    u = fma(u, x, a[2 * k]);
    w = fma(w, x, a[2 * k + 1]);
  }
}

template <int N>
__device__ __forceinline__ void rys_roots(double t, double (&u)[N], double (&w)[N]) {
  static_assert(N >= 1 && N <= RYS_NMAX, "root count outside the table");
  constexpr int kIntervals = RysIntervals<N>::value;
  constexpr int kOffset = RysOffset<N>::value;
  if (t < kIntervals * RYS_H) {  // false for NaN: NaN takes the closed form below
    int i = (int)(t * (1.0 / RYS_H));
    i = i < 0 ? 0 : (i >= kIntervals ? kIntervals - 1 : i);
    const double x = 2.0 * (t - i * RYS_H) * (1.0 / RYS_H) - 1.0;
    const double* c = d_rys_table + kOffset + (size_t)i * (2 * N * (RYS_DEG + 1));
#pragma unroll
    for (int s = 0; s < N; ++s) rys_poly(c + s * (2 * (RYS_DEG + 1)), x, u[s], w[s]);
  } else {
    const double inv = 1.0 / t;
    const double rs = sqrt(inv);
#pragma unroll
    for (int s = 0; s < N; ++s) {
      u[s] = d_rys_x2[N - 1][s] * inv;
      w[s] = d_rys_w[N - 1][s] * rs;
    }
  }
}

// Select G[.][kc] with a runtime kc without dynamic register indexing.
template <int M>
__device__ __forceinline__ double select_col(const double (&g)[M], int kc) {
  double v = g[0];
#pragma unroll
  for (int m = 1; m < M; ++m) v = (kc == m) ? g[m] : v;
  return v;
}

// One direction, one root: I[i][j] = <(x-A)^i (x-B)^j | (x-C)^kc> (2-D factor).
// c00, c00p, b10, b01, b00 are the Rys recurrence coefficients; ab = A - B.
template <int LA, int LB, int LC>
__device__ __forceinline__ void rys_2d(double c00, double c00p, double b10, double b01,
                                       double b00, double ab, int kc,
                                       double (&out)[LA + 1][LB + 1]) {
  constexpr int LAB = LA + LB;
  double g[LAB + 1][LC + 1];
  g[0][0] = 1.0;
  if (LAB > 0) g[1][0] = c00;
#pragma unroll
  for (int n = 1; n < LAB; ++n) g[n + 1][0] = fma(c00, g[n][0], n * b10 * g[n - 1][0]);
#pragma unroll
  for (int m = 0; m < LC; ++m) {
    g[0][m + 1] = c00p * g[0][m] + (m > 0 ? m * b01 * g[0][m > 0 ? m - 1 : 0] : 0.0);
#pragma unroll
    for (int n = 1; n <= LAB; ++n) {
      double v = fma(c00p, g[n][m], n * b00 * g[n - 1][m]);
      if (m > 0) v = fma(m * b01, g[n][m > 0 ? m - 1 : 0], v);
      g[n][m + 1] = v;
    }
  }
  double h[LAB + 1][LB + 1];
#pragma unroll
  for (int n = 0; n <= LAB; ++n) {
    double col[LC + 1];
#pragma unroll
    for (int m = 0; m <= LC; ++m) col[m] = g[n][m];
    h[n][0] = select_col<LC + 1>(col, kc);
  }
#pragma unroll
  for (int j = 0; j < LB; ++j)
#pragma unroll
    for (int i = 0; i + j < LAB; ++i) h[i][j + 1] = fma(ab, h[i][j], h[i + 1][j]);
#pragma unroll
  for (int i = 0; i <= LA; ++i)
#pragma unroll
    for (int j = 0; j <= LB; ++j) out[i][j] = h[i][j];
}

// One root of the Rys quadrature (node u_r, weight w_r) for a runtime index
// r < N.
template <int N>
__device__ __forceinline__ void rys_root_one(double t, int r, double& u, double& w) {
  static_assert(N >= 1 && N <= RYS_NMAX, "root count outside the table");
  constexpr int kIntervals = RysIntervals<N>::value;
  constexpr int kOffset = RysOffset<N>::value;
  if (t < kIntervals * RYS_H) {  // false for NaN: NaN takes the closed form below
    int i = (int)(t * (1.0 / RYS_H));
    i = i < 0 ? 0 : (i >= kIntervals ? kIntervals - 1 : i);
    const double x = 2.0 * (t - i * RYS_H) * (1.0 / RYS_H) - 1.0;
    rys_poly(d_rys_table + kOffset + (size_t)(i * N + r) * (2 * (RYS_DEG + 1)), x, u, w);
  } else {
    const double inv = 1.0 / t;
    u = d_rys_x2[N - 1][r] * inv;
    w = d_rys_w[N - 1][r] * sqrt(inv);
  }
}

// Vertical recurrence of one direction and root: G[n][m] = <(x-A)^n | (x-C)^m>
// for n <= LAB, m <= LC (the table rys_2d builds before selecting a column).
template <int LAB, int LC>
__device__ __forceinline__ void rys_vrr(double c00, double c00p, double b10, double b01,
                                        double b00, double (&g)[LAB + 1][LC + 1]) {
  g[0][0] = 1.0;
  if (LAB > 0) g[1][0] = c00;
#pragma unroll
  for (int n = 1; n < LAB; ++n) g[n + 1][0] = fma(c00, g[n][0], n * b10 * g[n - 1][0]);
#pragma unroll
  for (int m = 0; m < LC; ++m) {
    g[0][m + 1] = c00p * g[0][m] + (m > 0 ? m * b01 * g[0][m > 0 ? m - 1 : 0] : 0.0);
#pragma unroll
    for (int n = 1; n <= LAB; ++n) {
      double v = fma(c00p, g[n][m], n * b00 * g[n - 1][m]);
      if (m > 0) v = fma(m * b01, g[n][m > 0 ? m - 1 : 0], v);
      g[n][m + 1] = v;
    }
  }
}

// Horizontal transfer of column kc of a vertical table:
// I(i, j+1) = I(i+1, j) + (A - B) I(i, j).  Callers pass kc from a fully
// unrolled loop over compile-time component tables, so the column index
// folds to a constant and the tables stay in registers.
template <int LA, int LB, int LC>
__device__ __forceinline__ void rys_hrr_col(const double (&g)[LA + LB + 1][LC + 1], int kc,
                                            double ab, double (&out)[LA + 1][LB + 1]) {
  constexpr int LAB = LA + LB;
  double h[LAB + 1][LB + 1];
#pragma unroll
  for (int n = 0; n <= LAB; ++n) h[n][0] = g[n][kc];
#pragma unroll
  for (int j = 0; j < LB; ++j)
#pragma unroll
    for (int i = 0; i + j < LAB; ++i) h[i][j + 1] = fma(ab, h[i][j], h[i + 1][j]);
#pragma unroll
  for (int i = 0; i <= LA; ++i)
#pragma unroll
    for (int j = 0; j <= LB; ++j) out[i][j] = h[i][j];
}

// Cartesian component tables in CCA order.
template <int L>
struct Cart {
  int x[ncart(L)], y[ncart(L)], z[ncart(L)];
  __host__ __device__ constexpr Cart() : x(), y(), z() {
    int k = 0;
    for (int lx = L; lx >= 0; --lx)
      for (int ly = L - lx; ly >= 0; --ly) {
        x[k] = lx;
        y[k] = ly;
        z[k] = L - lx - ly;
        ++k;
      }
  }
};

struct DevBasis {
  const int* l;
  const int* atom;      // global atom index
  const int* nprim;
  const int* prim_off;
  const int* func_off;  // first function of the shell, within its molecule
  const double* exps;
  const double* coefs;  // primitive and contraction norms folded in
};

struct DevMol {
  int nao, naux, natom, atom_off;
  long long mat_off;  // N*N blocks (S, T, V, densities, Fock)
  long long met_off;  // X*X metric blocks
  long long a_off;    // packed (N(N+1)/2) * X three-centre blocks
};

// A launch chunk: a contiguous range of (pair, aux-shell) triples of one
// molecule for one angular-momentum class.
struct Chunk {
  int mol;
  int pair_begin;   // index into the class pair list
  int aux_begin;    // first aux shell of the class in this molecule
  int naux;         // aux shells of the class in this molecule
  int t0;           // first triple of this chunk (pair-major, aux fastest)
  int ntriples;     // triples of the molecule for this class
};

}  // namespace vqc
