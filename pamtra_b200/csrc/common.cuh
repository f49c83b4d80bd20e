// Shared device helpers for the B200 passive path.
//
// Arithmetic conventions: the library is compiled with --fmad=false so that
// every a*b+c written out in the restated formulas rounds twice, as the
// reference's gfortran x86-64 build does.  Hot loops (matrix products,
// Legendre and Mie series sums) call fma() explicitly.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/pamtra_b200.h"

namespace pb {

constexpr double PI = 3.141592653589793;           // constants.f90 pi
constexpr double C_LIGHT = 299792458.0;             // constants.f90 c
constexpr double R_D = 287.0596736665907;           // constants.f90 r_d
constexpr double R_V = 461.5249933083879;           // constants.f90 r_v
constexpr double RHO_WATER = 1000.0;
constexpr double RHO_ICE = 917.0;
constexpr double SKY_TEMP = 2.73;
constexpr double DELTA_D_MONO = 1.0e-8;
constexpr int MAXNLEG = PAMTRA_B200_MAXNLEG;
constexpr int MAXBIN = PAMTRA_B200_MAXBIN;

// Fortran default-REAL literal promoted to double.
__host__ __device__ __forceinline__ double F(float v) { return (double)v; }

// gfortran powi chains for constant integer exponents.
__device__ __forceinline__ double p2(double x) { return x * x; }
__device__ __forceinline__ double p3(double x) { double x2 = x * x; return x2 * x; }
__device__ __forceinline__ double p5(double x) { double x2 = x * x; double x3 = x2 * x; return x3 * x2; }

// ------------------------------------------------------------------ complex
struct cplx {
  double re, im;
};
__device__ __forceinline__ cplx cmk(double r, double i) { return cplx{r, i}; }
__device__ __forceinline__ cplx cadd(cplx a, cplx b) { return {a.re + b.re, a.im + b.im}; }
__device__ __forceinline__ cplx csub(cplx a, cplx b) { return {a.re - b.re, a.im - b.im}; }
__device__ __forceinline__ cplx cmul(cplx a, cplx b) { return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }
__device__ __forceinline__ cplx cscale(cplx a, double s) { return {a.re * s, a.im * s}; }
__device__ __forceinline__ cplx cconj(cplx a) { return {a.re, -a.im}; }
// Smith-style division as gfortran emits it (-fcx-fortran-rules).
__device__ __forceinline__ cplx cdiv(cplx a, cplx b) {
  double tr, ti, ratio, div;
  if (fabs(b.re) < fabs(b.im)) {
    ratio = b.re / b.im;
    div = (b.re * ratio) + b.im;
    tr = (a.re * ratio) + a.im;
    ti = (a.im * ratio) - a.re;
  } else {
    ratio = b.im / b.re;
    div = (b.im * ratio) + b.re;
    tr = (a.im * ratio) + a.re;
    ti = a.im - (a.re * ratio);
  }
  return {tr / div, ti / div};
}
// Principal square root: r = sqrt((|z|+x)/2), s = y/(2r) (x > 0), else the
// mirrored form; avoids cancellation in |z| - x.
__device__ __forceinline__ cplx csqrt_(cplx z) {
  double d = hypot(z.re, z.im);
  double r, s;
  if (z.re > 0) {
    r = sqrt(0.5 * (d + z.re));
    s = 0.5 * (z.im / r);
  } else {
    s = sqrt(0.5 * (d - z.re));
    r = fabs(0.5 * (z.im / s));
  }
  return {r, copysign(s, z.im)};
}
// CMPLX(x, y) without KIND: rounds both parts to REAL(4).
__device__ __forceinline__ cplx cmplx4(double x, double y) { return {(double)(float)x, (double)(float)y}; }

// ------------------------------------------------------------------ warp helpers
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// sum over the four lanes of a quad (lanes 4g .. 4g + 3)
__device__ __forceinline__ double quad_sum(double v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

// ------------------------------------------------------------------ team linear algebra
// A "team" is one CTA working on n x n FP64 matrices (n = 16, 32, 64) held in
// shared memory, column-major with leading dimension LD = n + 4 (LD = 4 mod
// 16 doubles makes the DMMA fragment loads below bank-conflict free).  The
// team has one warp per 16 x 16 output tile: T = 32 (n/16)^2 threads.
template <int n>
struct Team {
  static constexpr int T = 32 * (n / 16) * (n / 16);
  static constexpr int LD = n + 4;
  static constexpr int MAT = n * LD;  // doubles per matrix
  static constexpr int RG = T / n;    // threads per column in element-wise phases
};

__device__ __forceinline__ void team_sync() { __syncthreads(); }

// FP64 tensor-core MMA, D(8x8) += A(8x4) * B(4x8); fragments: a = A[g][q],
// b = B[q][g], d = D[g][2q], D[g][2q+1] with g = lane/4, q = lane%4.
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// C = A B, C = D + A B, C = I + A B
enum MMMode { MM_SET = 0, MM_ACC = 1, MM_IPLUS = 2 };

// ------------------------------------------------------------------ symmetric-matrix teams
// A team of n / 8 warps works on symmetric n x n matrices (and one general
// one, kept transposed): warp i owns the 8-row strip i of every result.  A
// matrix is held column by column with leading dimension n, the 16-byte
// chunks of a column (two rows) XOR-swizzled, so that the three access
// patterns below take the least number of wavefronts:
//   fragment: lane (g, q) reads rows 8u + 2q, + 1 of column 8j + g (16 bytes).
//     As the left factor of a symmetric matrix that is M[8j+g][k], as the
//     right factor M[k][8j+g], for the k pair 2q, 2q + 1 of block u: the two
//     MMAs of the block take k = 8u + 2q and k = 8u + 2q + 1, so one 16-byte
//     read serves both and a tile's accumulators (row g, columns 2q, 2q + 1) are
//     themselves the left fragment of that tile: a result strip can be the
//     left factor of the next product without leaving the registers;
//   direct store of tile (i, j): column 8i + g, rows 8j + 2q, + 1 (16 bytes;
//     the transposed tile, which for a symmetric matrix is its mirror image);
//   mirror store: column 8j + 2q + e, row 8i + g (8 bytes).
template <int n>
struct SymTeam {
  static constexpr int NB = n / 8, D = NB / 2, T = 32 * NB, MAT = n * n;
  __device__ static __forceinline__ int swz(int col) { return (((col >> 1) & 3) << 1) ^ ((col & 1) << 2); }
  // offset of element (row, col)
  __device__ static __forceinline__ int at(int row, int col) {
    return col * n + ((((row >> 1) ^ swz(col)) << 1) | (row & 1));
  }
  // offset of a lane's fragment of column block j, k block u
  __device__ static __forceinline__ int frag(int j, int u) {
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    return (8 * j + g) * n + (((4 * u + q) ^ swz(g)) << 1);
  }
  __device__ static __forceinline__ double2 ld(const double* M, int j, int u) {
    return *reinterpret_cast<const double2*>(M + frag(j, u));
  }
  __device__ static __forceinline__ void st(double* M, int i, int j, const double (&c)[2]) {
    *reinterpret_cast<double2*>(M + frag(i, j)) = make_double2(c[0], c[1]);
  }
  // both halves of a symmetric result's tile (i, j); a diagonal tile keeps its upper triangle
  __device__ static __forceinline__ void st_sym(double* M, int i, int j, const double (&c)[2]) {
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    const int row = 8 * i + g, col = 8 * j + 2 * q;
    if (i != j) {
      st(M, i, j, c);
#pragma unroll
      for (int e = 0; e < 2; e++) M[at(row, col + e)] = c[e];
    } else {
#pragma unroll
      for (int e = 0; e < 2; e++)
        if (row <= col + e) {
          M[at(row, col + e)] = c[e];
          M[at(col + e, row)] = c[e];
        }
    }
  }
  // The strip's share of a symmetric result: column blocks (i + d) mod NB for
  // d < D, and d = D for half of the strips (which half differs between the two
  // results of a pass, so every strip has NB + 1 tiles of a pair).
  __device__ static __forceinline__ int blk(int i, int d) { return (i + d) & (NB - 1); }
};

// Scratch of the inverse routines.
template <int n>
struct InvScratch {
  double f[n], fpre[n], prow[n];
  double cand_v[4];
  int cand_i[4];
  int piv[n], perm[n];
  double nrm;
  int sing;
};

// Pivot candidate of rows i >= k among the n/32 (or one) warps of a column
// group: the lanes hold rows i (value v of column k).
template <int n>
__device__ __forceinline__ void pivot_candidates(int i, int k, double v, InvScratch<n>& S) {
  constexpr int W = (n >= 32) ? 32 : n;
  S.fpre[i] = v;
  double best = (i >= k) ? fabs(v) : -1.0;
  int bi = i;
  const unsigned mask = (n >= 32) ? 0xffffffffu : (((1u << n) - 1u) << (threadIdx.x & 31 & ~(n - 1)));
#pragma unroll
  for (int o = W / 2; o > 0; o >>= 1) {
    const double ov = __shfl_xor_sync(mask, best, o);
    const int oi = __shfl_xor_sync(mask, bi, o);
    if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
  }
  if ((i & (W - 1)) == 0) {
    S.cand_v[i / W] = best;
    S.cand_i[i / W] = bi;
  }
}

// In-place Gauss-Jordan inverse with partial (row) pivoting of A (n x n).
// Thread t owns row t % n of the columns cg, cg + CG, ... (cg = t / n,
// CG = T / n), so every shared-memory sweep is bank-conflict free; the
// pivot search of the next column is fused into the elimination, leaving
// two team barriers per step.  Returns nonzero to every thread if a pivot
// was exactly zero.
template <int n, int T = Team<n>::T>
__device__ int ginv(double* A, InvScratch<n>& S) {
  constexpr int LD = Team<n>::LD, CG = T / n, NC = n / CG, NGW = (n + 31) / 32;
  const int t = threadIdx.x, i = t % n, cg = t / n;
  if (cg == 0) pivot_candidates<n>(i, 0, A[i], S);
  if (t == 0) S.sing = 0;
  team_sync();
  for (int k = 0; k < n; k++) {
    // (b) resolve the pivot, interchange rows k and p, scaled pivot row
    int p = S.cand_i[0];
    {
      double bv = S.cand_v[0];
#pragma unroll
      for (int w = 1; w < NGW; w++)
        if (S.cand_v[w] > bv) { bv = S.cand_v[w]; p = S.cand_i[w]; }
    }
    const double pv = S.fpre[p];
    const double rp = 1.0 / pv;
    if (t < n) {
      const int j = t;
      const double akj = A[j * LD + p];
      if (p != k) {
        A[j * LD + p] = A[j * LD + k];
        A[j * LD + k] = akj;
      }
      S.prow[j] = (j == k) ? rp : akj * rp;
      S.f[t] = (t == k) ? pv : ((t == p) ? S.fpre[k] : S.fpre[t]);
      if (t == 0) {
        S.piv[k] = p;
        if (pv == 0.0) S.sing = 1;
      }
    }
    team_sync();
    // (c) eliminate column k from every other row; the group that owns
    // column k+1 also finds the next pivot
    const double fi = S.f[i];
    double vnext = 0.0;
#pragma unroll
    for (int jj = 0; jj < NC; jj++) {
      const int j = cg + CG * jj;
      const double pj = S.prow[j];
      double v;
      if (i == k) v = pj;
      else if (j == k) v = -fi * rp;
      else v = fma(-fi, pj, A[j * LD + i]);
      A[j * LD + i] = v;
      if (j == k + 1) vnext = v;
    }
    if (k + 1 < n && cg == (k + 1) % CG) pivot_candidates<n>(i, k + 1, vnext, S);
    team_sync();
  }
  // undo the row interchanges as column interchanges in reverse order
  if (t == 0) {
    for (int q = 0; q < n; q++) S.perm[q] = q;
    for (int k = n - 1; k >= 0; k--) {
      const int p = S.piv[k];
      const int tmp = S.perm[k];
      S.perm[k] = S.perm[p];
      S.perm[p] = tmp;
    }
  }
  team_sync();
  double col[NC];
#pragma unroll
  for (int jj = 0; jj < NC; jj++) col[jj] = A[S.perm[cg + CG * jj] * LD + i];
  team_sync();
#pragma unroll
  for (int jj = 0; jj < NC; jj++) A[(cg + CG * jj) * LD + i] = col[jj];
  team_sync();
  return S.sing;
}

}  // namespace pb
