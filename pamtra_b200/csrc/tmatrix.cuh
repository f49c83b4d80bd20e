// T-matrix scattering of spheroids (scat_name 'tmatrix', src/tmatrix.f90 and
// the extended-precision EBCM code src/tmatrix_amplq.lp.f of the reference).
//
// Two persistent kernels in FP64, the working sets in slots of global scratch
// that stay in L1 / L2.  k_tmatrix, one particle (bin) per CTA:
//   1. the convergence of NMAX and then of the Gauss points on the m = 0
//      extinction and scattering sums (tmatrix_amplq.lp.f:386-470), each
//      step a full m = 0 solve: spheroid surface and spherical Bessel tables
//      (one node per thread, downward ratio recurrences), the EBCM surface
//      integrals (one (n1, n2) pair per thread) assembled into
//      [Q^T | -RgQ^T], and a Gauss-Jordan elimination with partial pivoting
//      that leaves T^T;
//   2. the m >= 1 blocks (TMATR, :1765-2047), each one more solve;
//   3. the T-matrix stored in single precision, as the reference stores it
//      (REAL*4 common /TMAT/), and the vectors U below.
// k_tmat_ampl, the amplitude matrices of 16 scattering azimuths (of 30, the others are mirror images) for every pair
// of Lobatto angles (calc_single_tmatrix, src/tmatrix.f90:436-684): a unit is a
// scattered angle of a canted particle, or 128 (incident, scattered) pairs of an upright
// one, so that few particles fill the chip too.
// A solve of microwave hydrometeors has order 8-40: solves one after another
// leave most threads idle and spend the time in barriers.  So two steps of the
// NMAX search and the Gauss-point step that usually follows go side by side,
// and so do all m >= 1 solves: a phase spreads the nodes, the (n1, n2) pairs
// or the decoupled systems of all of them over the CTA, a warp per system.
// Orders whose systems do not fit the slot together (NMAX above about 22) go
// one by one.  Gauss nodes come from a table of the context.
// The amplitude of an incident and a scattered direction is a sum over m of
// cos / sin(m phi) times P_m, the scattered direction's Wigner vectors (m d /
// sin, d') dotted with four vectors U of the incident angle and m (the block
// sums of CAL o T with its own Wigner vectors).  U is formed once per
// incident angle.  For an upright particle (canting 0) the scattered polar
// angle does not depend on the azimuth: P_m is formed once per scattered angle
// and the 16 azimuths weigh it; a canted particle forms P_m per scattered
// direction, 960 times fewer products than evaluating AMPL per pair.
// 1024 upright particles of NMAX 5 - 14 (1.2 - 6 mm, 89 GHz): 8.6 ms with one
// barrier chain per particle and AMPL per pair, now 0.88 ms; 96 canted ones 39 ms,
// now 0.43 ms (0.99 and 0.59 ms with all 30 azimuths).  Bound by latency (pivots,
// recurrences and phases that follow one another: FP64 pipe 19 % of the solve's active
// cycles, the largest stall at the CTA's barriers; 30 % of the amplitudes', which wait for
// loads).  With 30 azimuths, four warps per CTA and four CTAs per SM: 1.16 and
// 0.74 ms; one order after another with a warp per solve: 1.36 and 0.72 ms.
// The reference computes the solve in REAL*16; FP64 here agrees with it to
// about 1e-12 relative on microwave hydrometeors, below the single-precision
// storage of T.  The normalisation factors the reference forms in
// single-precision float() arithmetic (CONST, VIG) are formed the same way.
#pragma once
#include "common.cuh"
#include "mie.cuh"  // eps_mix_m
#include "tmatrix_limits.cuh"

namespace pb {
constexpr int TM_WARPS = TM_THREADS / 32;  // k_tmatrix
constexpr int TMA_THREADS = 128;            // k_tmat_ampl

// ---------------------------------------------------------------- scratch slot of one CTA
// Solve region of one group of threads (a warp or the CTA) for given NMAX and
// Gauss points per half: the augmented system, the Wigner tables of the
// current m, then the tables of the surface nodes and the Bessel functions.
__host__ __device__ __forceinline__ int tm_need(int nmax, int ngauss) {
  return 16 * nmax * nmax + 2 * ngauss * nmax + 7 * ngauss + 8 * ngauss * nmax;
}
// m >= 1 solves side by side: the systems and Wigner tables of every order
__host__ __device__ __forceinline__ int tm_cubes(int x) { return x * (x + 1) * (2 * x + 1) / 6; }  // 1 + 4 + ... + x^2
__host__ __device__ __forceinline__ int tm_need_all(int nmax, int ngauss) {
  return 8 * tm_cubes(nmax) + 2 * ngauss * nmax * nmax;
}
constexpr int TM_POOL = 140000 / 32 * 32;  // at least tm_need(TM_NMAX, TM_NGAUSS); all orders side by side up to NMAX 22
static_assert(TM_POOL >= 16 * TM_NMAX * TM_NMAX + 7 * TM_NGAUSS + 10 * TM_NGAUSS * TM_NMAX, "a solve of the largest order");
__device__ __forceinline__ cplx* tm_aug(double* s) { return reinterpret_cast<cplx*>(s); }
__device__ __forceinline__ double* tm_d(double* s, int k, int nmax, int ngauss) {
  return s + 16 * nmax * nmax + k * ngauss * nmax;
}
__device__ __forceinline__ double* tm_node(double* s, int k, int nmax, int ngauss) {  // s ss r dr ddr drr dri
  return s + 16 * nmax * nmax + 2 * ngauss * nmax + k * ngauss;
}
__device__ __forceinline__ double* tm_bes(double* s, int k, int nmax, int ngauss) {  // J Y JR JI DJ DY DJR DJI
  return s + 16 * nmax * nmax + 2 * ngauss * nmax + 7 * ngauss + k * ngauss * nmax;
}
// (m, n) pairs, m = 0 .. nmax, n = max(m, 1) .. nmax, and the blocks of the
// single-precision T of an order: index of the first of m
constexpr int TM_PAIRS = TM_NMAX + TM_NMAX * (TM_NMAX + 1) / 2;
constexpr int TM_T_FLOAT2 = 4 * (TM_NMAX * TM_NMAX + TM_NMAX * (TM_NMAX + 1) * (2 * TM_NMAX + 1) / 6);
__device__ __forceinline__ int tm_pair0(int nmax, int m) { return m == 0 ? 0 : nmax + (m - 1) * (2 * nmax - m + 2) / 2; }
__device__ __forceinline__ int tm_t0(int nmax, int m) {
  if (m == 0) return 0;
  return 4 * (nmax * nmax + tm_cubes(nmax) - tm_cubes(nmax - m + 1));
}
// Slot of k_tmatrix: solve pool, T, incident Wigner vectors [pair][2][nummu].
// Of the TM_NAZ azimuths 12 k degrees only k = 0 .. 15 are formed, k = 1 .. 14 with
// weight two: mirrored in the plane of the incident direction and the
// particle's axis, scattered azimuth f at incident azimuth i gives the same
// forms (F(f, i) = F(-f, -i)).  The reference's 1e-8 offset e of the incident
// azimuth makes the partner F(-f, e) = F(f, -e), and F(f, e) + F(f, -e) is 2 F(f, 0) to
// e^2: so these are formed at incident azimuth 0 (1e-14 where 0 is singular).
constexpr int TM_NAZH = TM_NAZ / 2 + 1;
static_assert(TM_NAZ % 2 == 0, "a mirrored pair of azimuths each");
constexpr int TM_DIRD = 7;  // doubles of one direction: polar cosine, cos and sin of the azimuth, rotation
struct TmSlot {
  size_t t, dvi, total;
};
__host__ __device__ inline size_t tm_geo_doubles(int nummu) {
  return (size_t)TM_DIRD * (2 * (size_t)nummu * TM_NAZH + nummu);
}
__host__ __device__ inline TmSlot tm_slot(int nummu) {
  TmSlot s;
  s.t = TM_POOL;
  s.dvi = s.t + TM_T_FLOAT2;
  s.total = (s.dvi + (size_t)TM_PAIRS * 2 * nummu + 31) / 32 * 32;
  return s;
}
// Record of a particle for k_tmat_ampl: U [pair][8][nummu], then the scattered
// Wigner vectors [pair][2][2 nummu] (upright) or its directions (canted).
__host__ __device__ inline size_t tm_record(int npair, int nummu, bool upright) {
  const size_t u = (size_t)npair * 8 * nummu;
  return (u + (upright ? (size_t)npair * 4 * nummu : tm_geo_doubles(nummu)) + 1) / 2 * 2;
}
// Scratch of a CTA of k_tmat_ampl whose working set exceeds its shared memory.
constexpr int TMA_SMEM = 9 * 8 * TMA_THREADS;  // doubles: P of an upright particle up to NMAX 8
constexpr size_t TMA_SLOT = (size_t)TM_PAIRS * 2 * TM_NAZH > (size_t)(TM_NMAX + 1) * 8 * TMA_THREADS
                                ? (size_t)TM_PAIRS * 2 * TM_NAZH : (size_t)(TM_NMAX + 1) * 8 * TMA_THREADS;

// ---------------------------------------------------------------- tables of the context
// Gauss-Legendre nodes and weights of the even orders 2 g, g = 1 .. TM_NGAUSS
// (offset g (g - 1)); |CAL|, sqrt(n^2 - m^2) and its inverse, the m-factor of
// d^m_{0m}, 1 / (2 n + 1), 2 cos and 2 sin (m phi) [m][azimuth] of an upright
// particle (m = 0: 1, 0); the directions of an upright particle for one nummu.
constexpr int TM_SQ = TM_NMAX + 2;
constexpr size_t TMT_X = 0, TMT_W = TMT_X + (size_t)TM_NGAUSS * (TM_NGAUSS + 1), TMT_CAL = TMT_W + (size_t)TM_NGAUSS * (TM_NGAUSS + 1),
                 TMT_SQ = TMT_CAL + (size_t)TM_NMAX * TM_NMAX, TMT_RQ = TMT_SQ + (size_t)TM_SQ * TM_SQ,
                 TMT_AM = TMT_RQ + (size_t)TM_SQ * TM_SQ, TMT_I2 = TMT_AM + TM_SQ, TMT_CS = TMT_I2 + TM_SQ,
                 TMT_TOTAL = TMT_CS + (size_t)(TM_NMAX + 1) * TM_NAZH * 2;

// Inputs and outputs of one launch: particle p = item * nbins + bin.
// Counters of a round (all zero at the start, but n): particles, records.  A
// round solves particles until their records fill the record pool; the rest
// waits for the next round.
struct TmRound {
  int n;                        // particles to solve
  int taken, upright, canted;   // of these: taken, with a record
  int units;                    // units of k_tmat_ampl taken
  int pad;
  unsigned long long used;      // doubles of the record pool taken
};

struct TmArgs {
  int n_items, nbins, nummu;
  const double* freq;      // [item] Hz
  const double* mrr;       // [item * nbins + bin] real part of the index used
  const double* mri;       // [item * nbins + bin] |imaginary part|
  const double* axi;       // [particle] equal-volume-sphere radius (m)
  const double* asr;       // [particle] aspect ratio
  const double* beta;      // [particle] canting angle (deg)
  const double* ndens;     // [particle] 0 = no particle
  const double* mu;        // Lobatto angles [nummu]
  const double* wq;        // Lobatto weights [nummu]
  const double* tab;       // [TMT_TOTAL]
  const double* geo;       // [tm_geo_doubles(nummu)] directions of an upright particle
  double* scat;            // [particle][2 nummu 2 nummu 2] (Fortran order of scatter_matrix)
  double* ext;             // [particle][2 2 nummu]
  double* sback;           // [particle][2 2]
  int* nmax;               // [particle] converged NMAX (0 when skipped)
  int* status;             // [particle]
  double* scratch;         // [CTAs of k_tmatrix][tm_slot(nummu).total]
  double* ascratch;        // [CTAs of k_tmat_ampl][TMA_SLOT]
  double* records;         // [rec_doubles]
  size_t rec_doubles;
  int64_t* rec;            // [particle] offset of its record
  const int* order;        // [particle] particles of this round, by decreasing size in the first
  int* again;              // [particle] particles left for the next round
  int *upright, *canted;   // [particle] particles with a record
  TmRound* round;          // this round's counters
  TmRound* next;           // the next round's
};

// first NMAX of the convergence search (tmatrix_amplq.lp.f:380) for a size parameter
__device__ __forceinline__ int tm_inm1(double xev) { return max(4, (int)(xev + 4.05 * pow(xev, 0.333333))); }

struct TmShared {
  double qe[3], qs[3];
  double piv[2];
  int ok[3], len[3][2];
  int sing[3];  // a pivot of the step vanished
  int pivrow;
  int particle;
  long long rec;
  uint16_t pm[TM_PAIRS];     // m | n << 8 of a pair
};

// Gauss-Legendre root pair k of order n (ascending nodes on [-1, 1], weights
// summing to 2) by Newton iteration on the three-term recurrence (QGAUSS,
// tmatrix_amplq.lp.f:1025-1112).
__device__ void tm_gauss_pair(int n, int k, double* x_out, double* w_out) {
  double x = cos(3.141592653589793 * ((double)k + 0.75) / ((double)n + 0.5));
  double dp = 1.0;
  for (int it = 0; it < 100; it++) {
    double p0 = 1.0, p1 = x;
    for (int j = 2; j <= n; j++) {
      const double p2 = ((double)(2 * j - 1) * x * p1 - (double)(j - 1) * p0) / (double)j;
      p0 = p1;
      p1 = p2;
    }
    dp = (double)n * (x * p1 - p0) / (x * x - 1.0);
    const double dx = p1 / dp;
    x -= dx;
    if (fabs(dx) <= 1.0e-16 * fabs(x) || fabs(dx) < 1.0e-300) break;
  }
  double p0 = 1.0, p1 = x;
  for (int j = 2; j <= n; j++) {
    const double p2 = ((double)(2 * j - 1) * x * p1 - (double)(j - 1) * p0) / (double)j;
    p0 = p1;
    p1 = p2;
  }
  dp = (double)n * (x * p1 - p0) / (x * x - 1.0);
  if ((n & 1) && k == (n - 1) / 2) x = 0.0;
  const double wk = 2.0 / ((1.0 - x * x) * dp * dp);
  x_out[n - 1 - k] = x;
  w_out[n - 1 - k] = wk;
  x_out[k] = -x;
  w_out[k] = wk;
}

// VIG (tmatrix_amplq.lp.f:2049-2105): d^n_{0m}(x) and its theta-derivative
// for n = 1..nmax, written through the callback at n - 1.  The m-factor
// prod sqrt((2i-1)/(2i)) is formed in single precision as the reference's
// float() does.
template <class F>
__device__ __forceinline__ void tm_vig(double x, int nmax, int m, F&& put) {
  const double qs = sqrt(1.0 - x * x), qs1 = 1.0 / qs;
  if (m == 0) {
    double d1 = 1.0, d2 = x;
    for (int n = 1; n <= nmax; n++) {
      const double qn = n, qn1 = n + 1, qn2 = 2 * n + 1;
      const double d3 = (qn2 * x * d2 - qn * d1) / qn1;
      const double der = qs1 * (qn1 * qn / qn2) * (-d1 + d3);
      put(n - 1, d2, der);
      d1 = d2;
      d2 = d3;
    }
    return;
  }
  for (int n = 1; n < m && n <= nmax; n++) put(n - 1, 0.0, 0.0);
  const double qmm = (double)(m * m);
  double a = 1.0;
  for (int i = 1; i <= m; i++) a = a * (double)sqrtf((float)(2 * i - 1) / (float)(2 * i)) * qs;
  double d1 = 0.0, d2 = a;
  for (int n = m; n <= nmax; n++) {
    const double qn = n, qn2 = 2 * n + 1, qn1 = n + 1;
    const double qnm = sqrt(qn * qn - qmm), qnm1 = sqrt(qn1 * qn1 - qmm);
    const double d3 = (qn2 * x * d2 - qnm * d1) / qnm1;
    const double der = qs1 * (-qn1 * qnm * d1 + qn * qnm1 * d3) / qn2;
    put(n - 1, d2, der);
    d1 = d2;
    d2 = d3;
  }
}

// The blocks that vanish by the particle's symmetry split the 2 nm unknowns
// (block b = 0, 1, order k = 0 .. nm - 1) into systems that do not couple: for
// m >= 1 two of nm unknowns (k + b even or odd), for m = 0, where the blocks do
// not couple either, four.  A quarter (a sixteenth) of the elimination's work, with the
// same arithmetic per element as in the full system, whose pivot rows come
// from the pivot column's own system.
struct TmSystems {
  int m, nm, count;
  __device__ __forceinline__ TmSystems(int m_, int nm_) : m(m_), nm(nm_), count(m_ == 0 ? 4 : 2) {}
  __device__ __forceinline__ int half(int s) const { return (nm + 1 - s) >> 1; }  // orders of parity s
  __device__ __forceinline__ int sys(int b, int k) const { return m == 0 ? 2 * b + (k & 1) : (k + b) & 1; }
  __device__ __forceinline__ int size(int s) const { return m == 0 ? half(s & 1) : nm; }
  __device__ __forceinline__ int pos(int s, int b, int k) const { return (k >> 1) + ((m != 0 && b) ? half(s) : 0); }
  __device__ __forceinline__ int base(int s) const { return s * 2 * nm * nm; }  // room for [nm][2 nm] each
};

// Constants of a particle.
struct TmPart {
  double lam, mrr, mri, rev, eps;  // wavelength, index, equal-volume radius, axial ratio
  double pi, aa, ee1;              // k, squared rotational radius, eps^2 - 1
  double ppi, pir, pii;
};

// RSP1 + VARY (tmatrix_amplq.lp.f:1194-1225, :1114-1192) for NP = -1: node t
// of one half (the other mirrors it): surface and size parameter, which it returns.
__device__ __forceinline__ double tm_surface(double* st, const double* X, int t, int nmax, int ngauss, const TmPart& A) {
  double *S = tm_node(st, 0, nmax, ngauss), *SS = tm_node(st, 1, nmax, ngauss), *R = tm_node(st, 2, nmax, ngauss),
         *DR = tm_node(st, 3, nmax, ngauss), *DDR = tm_node(st, 4, nmax, ngauss), *DRR = tm_node(st, 5, nmax, ngauss),
         *DRI = tm_node(st, 6, nmax, ngauss);
  const double v0 = 1.0 / (A.mrr * A.mrr + A.mri * A.mri);
  const double prr = A.mrr * v0, pri = -A.mri * v0;
  const double c = X[t], cc = c * c, ssv = 1.0 - cc, sv = sqrt(ssv);
  const double y = 1.0 / (1.0 - c * c);
  SS[t] = y;
  S[t] = sqrt(y);
  const double rr = 1.0 / (ssv + A.eps * A.eps * cc);
  R[t] = A.aa * rr;
  DR[t] = rr * c * sv * A.ee1;
  const double vt = sqrt(A.aa * rr) * A.pi;
  const double iv = 1.0 / vt;
  DDR[t] = iv;
  DRR[t] = prr * iv;
  DRI[t] = pri * iv;
  return vt;
}

// Recurrence lengths of BESS for the largest size parameter ta; false when the
// reference would stop (NMAX + NNMAX2 >= 1200).
__device__ __forceinline__ bool tm_lengths(double ta, int nmax, const TmPart& A, int& nnmax1, int& nnmax2) {
  double tb = ta * sqrt(A.mrr * A.mrr + A.mri * A.mri);
  tb = fmax(tb, (double)nmax);
  // bounded recurrence lengths for any input (the reference stops at 1200)
  if (!(ta > 0.0) || !(tb < (double)TM_LBES)) return false;
  nnmax1 = (int)(8.0 * sqrt(fmax(ta, (double)nmax)) + 3.0);
  nnmax2 = (int)(tb + 4.0 * pow(tb, 0.33333) + 8.0 * sqrt(tb));
  nnmax2 = nnmax2 - nmax + 5;
  return nmax + nnmax2 < TM_LBES;
}

// BESS (tmatrix_amplq.lp.f:1342-1524) of node t: j and y of the size
// parameter, or j of m times it.
__device__ void tm_bessel_real(double* st, int t, int nmax, int ngauss, int nnmax1, const TmPart& A) {
  double *J = tm_bes(st, 0, nmax, ngauss) + t * nmax, *Y = tm_bes(st, 1, nmax, ngauss) + t * nmax;
  double *DJ = tm_bes(st, 4, nmax, ngauss) + t * nmax, *DY = tm_bes(st, 5, nmax, ngauss) + t * nmax;
  const double x = sqrt(tm_node(st, 2, nmax, ngauss)[t]) * A.pi;
  // RJB: z_n = j_n / j_{n-1} downward from nmax + nnmax1; the ratios of
  // orders <= nmax wait in J until the upward pass replaces them
  {
    const int L = nmax + nnmax1;
    const double xx = 1.0 / x;
    double z = 1.0 / ((double)(2 * L + 1) * xx);
    if (L <= nmax) J[L - 1] = z;
    for (int i1 = L - 1; i1 >= 1; i1--) {
      z = 1.0 / ((double)(2 * i1 + 1) * xx - z);
      if (i1 <= nmax) J[i1 - 1] = z;
    }
    const double z0 = 1.0 / (xx - J[0]);
    const double y0 = z0 * cos(x) * xx;
    double yp = y0 * J[0];
    DJ[0] = y0 - yp * xx;
    J[0] = yp;
    for (int i = 2; i <= nmax; i++) {
      const double yi = yp * J[i - 1];
      DJ[i - 1] = yp - (double)i * yi * xx;
      J[i - 1] = yi;
      yp = yi;
    }
  }
  // RYB: y_n upward
  {
    const double c = cos(x), sn = sin(x), x1 = 1.0 / x, x2 = x1 * x1, x3 = x2 * x1;
    double ym = -c * x2 - sn * x1;
    Y[0] = ym;
    double yc = (-3.0 * x3 + x1) * c - 3.0 * x2 * sn;
    if (nmax >= 2) Y[1] = yc;
    for (int i = 2; i <= nmax - 1; i++) {
      const double yn = (double)(2 * i + 1) * x1 * yc - ym;
      Y[i] = yn;
      ym = yc;
      yc = yn;
    }
    DY[0] = -x1 * (c + Y[0]);
    for (int i = 2; i <= nmax; i++) DY[i - 1] = Y[i - 2] - (double)i * x1 * Y[i - 1];
  }
}
__device__ void tm_bessel_cplx(double* st, int t, int nmax, int ngauss, int nnmax2, const TmPart& A) {
  double *JR = tm_bes(st, 2, nmax, ngauss) + t * nmax, *JI = tm_bes(st, 3, nmax, ngauss) + t * nmax;
  double *DJR = tm_bes(st, 6, nmax, ngauss) + t * nmax, *DJI = tm_bes(st, 7, nmax, ngauss) + t * nmax;
  const double vt = sqrt(tm_node(st, 2, nmax, ngauss)[t]) * A.pi;
  const double xr = vt * A.mrr, xi = vt * A.mri;
  // CJB: RJB for the complex argument m k r
  {
    const int L = nmax + nnmax2;
    const double xrxi = 1.0 / (xr * xr + xi * xi);
    const double cxr = xr * xrxi, cxi = -xi * xrxi;
    double zr = xr / (double)(2 * L + 1), zi = xi / (double)(2 * L + 1);
    if (L <= nmax) { JR[L - 1] = zr; JI[L - 1] = zi; }
    for (int i1 = L - 1; i1 >= 1; i1--) {
      const double qf = (double)(2 * i1 + 1);
      const double ar = qf * cxr - zr, ai = qf * cxi - zi;
      const double ari = 1.0 / (ar * ar + ai * ai);
      zr = ar * ari;
      zi = -ai * ari;
      if (i1 <= nmax) { JR[i1 - 1] = zr; JI[i1 - 1] = zi; }
    }
    double ar = cxr - JR[0], ai = cxi - JI[0];
    double ari = 1.0 / (ar * ar + ai * ai);
    const double z0r = ar * ari, z0i = -ai * ari;
    const double cr = cos(xr) * cosh(xi), ci = -sin(xr) * sinh(xi);
    ar = z0r * cr - z0i * ci;
    ai = z0i * cr + z0r * ci;
    const double y0r = ar * cxr - ai * cxi, y0i = ai * cxr + ar * cxi;
    double ypr = y0r * JR[0] - y0i * JI[0], ypi = y0i * JR[0] + y0r * JI[0];
    ar = ypr * cxr - ypi * cxi;
    ai = ypi * cxr + ypr * cxi;
    DJR[0] = y0r - ar;
    DJI[0] = y0i - ai;
    JR[0] = ypr;
    JI[0] = ypi;
    for (int i = 2; i <= nmax; i++) {
      const double zr2 = JR[i - 1], zi2 = JI[i - 1];
      const double yr = ypr * zr2 - ypi * zi2, yi = ypi * zr2 + ypr * zi2;
      ar = yr * cxr - yi * cxi;
      ai = yi * cxr + yr * cxi;
      DJR[i - 1] = ypr - (double)i * ar;
      DJI[i - 1] = ypi - (double)i * ai;
      JR[i - 1] = yr;
      JI[i - 1] = yi;
      ypr = yr;
      ypi = yi;
    }
  }
}

// Wigner functions of order m at node t (and its mirror image) into D (two
// tables [node][nmax]).
__device__ __forceinline__ void tm_wnode(double* D, const double* X, int t, int m, int nmax, int ngauss) {
  double *D1 = D + (ngauss - 1 - t) * nmax, *D2 = D1 + ngauss * nmax;
  tm_vig(X[ngauss + t], nmax, m, [&](int k, double d1, double d2) {
    const double si = ((k + 1 + m) & 1) ? -1.0 : 1.0;
    D1[k] = d1 * si;
    D2[k] = -d2 * si;
  });
}

// TMATR0 / TMATR (tmatrix_amplq.lp.f:1526-2047) with NCHECK = 1: the surface
// integrals of the pair (n1, n2) of order m (the blocks of one n1 + n2 parity
// only) into [Q^T | -RgQ^T] of its systems at aug.  st: the node and Bessel
// tables, D: the Wigner tables of m, W: the Gauss weights.
__device__ void tm_pair(cplx* aug, double* st, const double* D, const double* W, int m, int n1, int n2, int nmax,
                        int ngauss, const TmPart& A) {
  const int mm1 = max(m, 1), nm = nmax - mm1 + 1;
  const TmSystems sy(m, nm);
  const double *D1 = D, *D2 = D + ngauss * nmax;
  const double *S = tm_node(st, 0, nmax, ngauss), *SS = tm_node(st, 1, nmax, ngauss), *R = tm_node(st, 2, nmax, ngauss),
               *DR = tm_node(st, 3, nmax, ngauss), *DDR = tm_node(st, 4, nmax, ngauss),
               *DRR = tm_node(st, 5, nmax, ngauss), *DRI = tm_node(st, 6, nmax, ngauss);
  const double *J = tm_bes(st, 0, nmax, ngauss), *Y = tm_bes(st, 1, nmax, ngauss), *JR = tm_bes(st, 2, nmax, ngauss),
               *JI = tm_bes(st, 3, nmax, ngauss), *DJ = tm_bes(st, 4, nmax, ngauss), *DY = tm_bes(st, 5, nmax, ngauss),
               *DJR = tm_bes(st, 6, nmax, ngauss), *DJI = tm_bes(st, 7, nmax, ngauss);
  const double ppi = A.ppi, pir = A.pir, pii = A.pii;
  const double qm = m, qmm = (double)(m * m);
  const double an1 = (double)(n1 * (n1 + 1)), an2 = (double)(n2 * (n2 + 1));
  const bool even = ((n1 + n2) & 1) == 0;
  double a11r = 0, a11i = 0, a12r = 0, a12i = 0, a21r = 0, a21i = 0, a22r = 0, a22i = 0;
  double g11r = 0, g11i = 0, g12r = 0, g12i = 0, g21r = 0, g21i = 0, g22r = 0, g22i = 0;
  if (!(m == 0 && !even)) {
    for (int i = 0; i < ngauss; i++) {
      const int o1 = i * nmax + n1 - 1, o2 = i * nmax + n2 - 1;
      const double d1n1 = D1[o1], d2n1 = D2[o1], d1n2 = D1[o2], d2n2 = D2[o2];
      const double e11 = d1n1 * d1n2, e12 = d1n1 * d2n2, e21 = d2n1 * d1n2, e22 = d2n1 * d2n2;
      const double qj1 = J[o1], qy1 = Y[o1], qdj1 = DJ[o1], qdy1 = DY[o1];
      const double qjr2 = JR[o2], qji2 = JI[o2], qdjr2 = DJR[o2], qdji2 = DJI[o2];
      const double c1r = qjr2 * qj1, c1i = qji2 * qj1, b1r = c1r - qji2 * qy1, b1i = c1i + qjr2 * qy1;
      const double c2r = qjr2 * qdj1, c2i = qji2 * qdj1, b2r = c2r - qji2 * qdy1, b2i = c2i + qjr2 * qdy1;
      const double ddri = DDR[i];
      const double c3r = ddri * c1r, c3i = ddri * c1i, b3r = ddri * b1r, b3i = ddri * b1i;
      const double c4r = qdjr2 * qj1, c4i = qdji2 * qj1, b4r = c4r - qdji2 * qy1, b4i = c4i + qdjr2 * qy1;
      const double drri = DRR[i], drii = DRI[i];
      const double c5r = c1r * drri - c1i * drii, c5i = c1i * drri + c1r * drii;
      const double b5r = b1r * drri - b1i * drii, b5i = b1i * drri + b1r * drii;
      const double uri = DR[i], wr = W[i] * R[i];
      if (m == 0 || even) {
        const double f1 = (m == 0) ? wr * e22 : wr * (e11 * (SS[i] * qmm) + e22);
        double f2 = wr * uri * an1 * e12;
        a12r = a12r + f1 * b2r + f2 * b3r;
        a12i = a12i + f1 * b2i + f2 * b3i;
        g12r = g12r + f1 * c2r + f2 * c3r;
        g12i = g12i + f1 * c2i + f2 * c3i;
        f2 = wr * uri * an2 * e21;
        a21r = a21r + f1 * b4r + f2 * b5r;
        a21i = a21i + f1 * b4i + f2 * b5i;
        g21r = g21r + f1 * c4r + f2 * c5r;
        g21i = g21i + f1 * c4i + f2 * c5i;
      } else {
        const double c6r = qdjr2 * qdj1, c6i = qdji2 * qdj1, b6r = c6r - qdji2 * qdy1, b6i = c6i + qdjr2 * qdy1;
        const double c7r = c4r * ddri, c7i = c4i * ddri, b7r = b4r * ddri, b7i = b4i * ddri;
        const double c8r = c2r * drri - c2i * drii, c8i = c2i * drri + c2r * drii;
        const double b8r = b2r * drri - b2i * drii, b8i = b2i * drri + b2r * drii;
        const double dsi = S[i] * qm * wr;
        const double e1 = dsi * (e12 + e21);
        a11r = a11r + e1 * b1r;
        a11i = a11i + e1 * b1i;
        g11r = g11r + e1 * c1r;
        g11i = g11i + e1 * c1i;
        double e2 = dsi * uri * e11;
        const double e3 = e2 * an2;
        e2 = e2 * an1;
        a22r = a22r + e1 * b6r + e2 * b7r + e3 * b8r;
        a22i = a22i + e1 * b6i + e2 * b7i + e3 * b8i;
        g22r = g22r + e1 * c6r + e2 * c7r + e3 * c8r;
        g22i = g22i + e1 * c6i + e2 * c7i + e3 * c8i;
      }
    }
  }
  // ANN(n1, n2) * 2 with the single-precision normalisation of CONST
  const double dd1 = (double)sqrtf((float)(2 * n1 + 1) / (float)(n1 * (n1 + 1)));
  const double dd2 = (double)sqrtf((float)(2 * n2 + 1) / (float)(n2 * (n2 + 1)));
  const double an12 = dd1 * dd2 * 0.5 * 2.0;
  // block phases: T11 = -X11, T12 = -i X12, T21 = i X21, T22 = -X22
  const cplx t11 = cmk(-a11r * an12, -a11i * an12), g11 = cmk(-g11r * an12, -g11i * an12);
  const cplx t12 = cmk(a12i * an12, -a12r * an12), g12 = cmk(g12i * an12, -g12r * an12);
  const cplx t21 = cmk(-a21i * an12, a21r * an12), g21 = cmk(-g21i * an12, g21r * an12);
  const cplx t22 = cmk(-a22r * an12, -a22i * an12), g22 = cmk(-g22r * an12, -g22i * an12);
  auto comb = [&](cplx x, cplx y) {
    return cmk(pir * x.re - pii * x.im + ppi * y.re, pir * x.im + pii * x.re + ppi * y.im);
  };
  const int k1 = n1 - mm1, k2 = n2 - mm1;
  // Q(r, c) goes to row c, column r of its system; -RgQ(r, c) to the right half
  auto put = [&](int b1, int b2, cplx qv, cplx gv) {
    const int sys = sy.sys(b1, k1), q = sy.size(sys);
    cplx* a = aug + sy.base(sys) + sy.pos(sys, b2, k2) * 2 * q + sy.pos(sys, b1, k1);
    a[0] = qv;
    a[q] = cmk(-gv.re, -gv.im);
  };
  if (even) {
    put(0, 0, comb(t21, t12), comb(g21, g12));
    put(1, 1, comb(t12, t21), comb(g12, g21));
  } else if (m != 0) {
    put(0, 1, comb(t11, t22), comb(g11, g22));
    put(1, 0, comb(t22, t11), comb(g22, g11));
  }
}

// A group of GS warps: one (GS = 1) or the CTA.
template <int GS>
__device__ __forceinline__ void tm_sync() {
  if (GS == 1) __syncwarp();
  else __syncthreads();
}

// T = -RgQ Q^-1 (TT, tmatrix_amplq.lp.f:2107-2153) of one system of q unknowns,
// [q][2 q] at a, by Gauss-Jordan elimination with partial pivoting: afterwards
// row j of the right half holds column j of T.  Whole group; false when a
// pivot vanishes.
template <int GS>
__device__ bool tm_eliminate(cplx* a, int q, TmShared& sh) {
  constexpr int GT = 32 * GS;
  const int lane = threadIdx.x & 31, tt = GS == 1 ? lane : (int)threadIdx.x, ldw = 2 * q;
  for (int c = 0; c < q; c++) {
    int prow = -1;
    cplx ip = cmk(0.0, 0.0);
    if (GS == 1 || threadIdx.x < 32) {
      double best = -1.0;
      int br = c;
      for (int r = c + lane; r < q; r += 32) {
        const cplx v = a[r * ldw + c];
        const double k = fabs(v.re) + fabs(v.im);
        if (k > best) { best = k; br = r; }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int orr = __shfl_xor_sync(0xffffffffu, br, o);
        if (ob > best || (ob == best && orr < br)) { best = ob; br = orr; }
      }
      if (best > 0.0) {
        prow = br;
        const cplx p = a[br * ldw + c];
        const double d = p.re * p.re + p.im * p.im;
        ip = cmk(p.re / d, -p.im / d);
      }
      if (GS > 1 && lane == 0) {
        sh.pivrow = prow;
        sh.piv[0] = ip.re;
        sh.piv[1] = ip.im;
      }
    }
    tm_sync<GS>();
    if (GS > 1) {
      prow = sh.pivrow;
      ip = cmk(sh.piv[0], sh.piv[1]);
    }
    if (prow < 0) return false;
    // swap rows c and prow and scale the pivot row (columns >= c)
    for (int j = c + tt; j < ldw; j += GT) {
      const cplx vp = a[prow * ldw + j];
      if (prow != c) a[prow * ldw + j] = a[c * ldw + j];
      a[c * ldw + j] = cmul(vp, ip);
    }
    tm_sync<GS>();
    // eliminate column c from every other row (columns > c), four rows at a
    // time with no branch between their loads; the group's warps take rows in turn
    for (int j = c + 1 + lane; j < ldw; j += 32) {
      const cplx v = a[c * ldw + j];
      for (int r = (GS == 1 ? 0 : (int)(threadIdx.x >> 5)); r < q; r += 4 * GS) {
        cplx f[4], x[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const int rk = min(r + k * GS, q - 1);
          f[k] = a[rk * ldw + c];
          x[k] = a[rk * ldw + j];
        }
#pragma unroll
        for (int k = 0; k < 4; k++) x[k] = csub(x[k], cmul(f[k], v));
#pragma unroll
        for (int k = 0; k < 4; k++)
          if (r + k * GS < q && r + k * GS != c) a[(r + k * GS) * ldw + j] = x[k];
      }
    }
    tm_sync<GS>();
  }
  return true;
}

// T of the systems at aug: row (block br, order kr), column (bc, kc), k from 0.
__device__ __forceinline__ cplx tm_tget(const cplx* aug, const TmSystems& sy, int br, int kr, int bc, int kc) {
  const int sys = sy.sys(bc, kc);
  if (sys != sy.sys(br, kr)) return cmk(0.0, 0.0);
  const int q = sy.size(sys);
  return aug[sy.base(sys) + sy.pos(sys, bc, kc) * 2 * q + q + sy.pos(sys, br, kr)];
}

// The m = 0 extinction and scattering sums of the convergence tests.
__device__ __forceinline__ void tm_sums(const cplx* aug, int nmax, double& qe, double& qs) {
  const TmSystems sy(0, nmax);
  qe = qs = 0.0;
  for (int k = 1; k <= nmax; k++) {
    const cplx a = tm_tget(aug, sy, 0, k - 1, 0, k - 1), b = tm_tget(aug, sy, 1, k - 1, 1, k - 1);
    const double dn1 = (double)(2 * k + 1);
    qs = qs + dn1 * (a.re * a.re + a.im * a.im + b.re * b.re + b.im * b.im);
    qe = qe + (a.re + b.re) * dn1;
  }
}

// Store T of order m in single precision (one of `threads` threads).
__device__ __forceinline__ void tm_store(const cplx* aug, float2* T, int m, int nmax, int tt, int threads) {
  const int nm = nmax - max(m, 1) + 1, o = tm_t0(nmax, m);
  const TmSystems sy(m, nm);
  for (int e = tt; e < 4 * nm * nm; e += threads) {
    const int b = e / (nm * nm), k = e % (nm * nm), n1 = k / nm, n2 = k % nm;
    const cplx v = tm_tget(aug, sy, b >> 1, n1, b & 1, n2);
    T[o + e] = make_float2((float)v.re, (float)v.im);
  }
}

// One step of the convergence searches: NMAX = nx with ng Gauss points per
// half, in region s.
struct TmStep {
  int nx, ng;
  double* s;
};

// The m = 0 solves of NC steps side by side: ok[c],
// qe[c], qs[c] in shared memory (ok 0: the reference would stop, or a pivot
// vanished).  Each phase spreads its tasks over all warps: nodes, then the
// Bessel and Wigner tables (a warp per step and kind), the pairs of the
// steps, the four systems of each.
template <int NC>
__device__ void tm_steps(const TmStep (&st)[NC], const TmPart& A, TmShared& sh, const double* tab) {
  constexpr int T = TM_THREADS, NW = TM_WARPS;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  __syncthreads();  // the regions and the shared results are free
#pragma unroll
  for (int c = 0; c < NC; c++)
    if (warp == c % NW) {
      const double* X = tab + TMT_X + (size_t)st[c].ng * (st[c].ng - 1);
      double ta = 0.0;
      for (int k = lane; k < st[c].ng; k += 32) ta = fmax(ta, tm_surface(st[c].s, X, k, st[c].nx, st[c].ng, A));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ta = fmax(ta, __shfl_xor_sync(0xffffffffu, ta, o));
      int l1 = 0, l2 = 0;
      const bool ok = tm_lengths(ta, st[c].nx, A, l1, l2);
      if (lane == 0) {
        sh.ok[c] = ok;
        sh.sing[c] = 0;
        sh.len[c][0] = l1;
        sh.len[c][1] = l2;
      }
    }
  __syncthreads();
  // (kind, step) tasks in chunks of 32 nodes
#pragma unroll
  for (int c = 0; c < NC; c++) {
    if (!sh.ok[c]) continue;
    const int nx = st[c].nx, ng = st[c].ng, ch = (ng + 31) / 32;
    const double* X = tab + TMT_X + (size_t)ng * (ng - 1);
    for (int w = 0; w < 3 * ch; w++) {
      if ((w + 3 * c) % NW != warp) continue;
      const int k = (w / 3) * 32 + lane, kind = w % 3;
      if (k >= ng) continue;
      if (kind == 0) tm_bessel_cplx(st[c].s, k, nx, ng, sh.len[c][1], A);
      else if (kind == 1) tm_bessel_real(st[c].s, k, nx, ng, sh.len[c][0], A);
      else tm_wnode(tm_d(st[c].s, 0, nx, ng), X, k, 0, nx, ng);
    }
  }
  __syncthreads();
  // pairs of equal parity: n1, then every second n2
  int first = 0;
#pragma unroll
  for (int c = 0; c < NC; c++) {
    if (!sh.ok[c]) continue;
    const int nx = st[c].nx, ng = st[c].ng, h = (nx + 1) / 2, np = nx * h;
    const double* W = tab + TMT_W + (size_t)ng * (ng - 1);
    for (int e = (t + T - first % T) % T; e < np; e += T) {
      const int n1 = 1 + e / h, n2 = 2 - (n1 & 1) + 2 * (e % h);
      if (n2 <= nx) tm_pair(tm_aug(st[c].s), st[c].s, tm_d(st[c].s, 0, nx, ng), W, 0, n1, n2, nx, ng, A);
    }
    first += np;
  }
  __syncthreads();
  // sh.ok stays as it is until all warps are through: a lane that read it later
  // than its neighbours would miss the shuffles they wait in
  for (int k = warp; k < 4 * NC; k += NW) {
    const int c = k >> 2;
    if (!sh.ok[c]) continue;
#pragma unroll
    for (int j = 0; j < NC; j++)
      if (j == c) {
        const TmSystems sy(0, st[j].nx);
        const int q = sy.size(k & 3);
        if (q > 0 && !tm_eliminate<1>(tm_aug(st[j].s) + sy.base(k & 3), q, sh) && lane == 0) sh.sing[c] = 1;
      }
  }
  __syncthreads();
#pragma unroll
  for (int c = 0; c < NC; c++)
    if (t == 32 * (c % NW) && sh.ok[c]) {
      if (sh.sing[c]) sh.ok[c] = 0;
      else tm_sums(tm_aug(st[c].s), st[c].nx, sh.qe[c], sh.qs[c]);
    }
  __syncthreads();
}

// VIGAMPL (tmatrix_amplq.lp.f:890-970): d^n_{0m}(x) / sin (dv1) and the
// theta-derivative (dv2) in double, with the pole values for m = 1.
template <class F>
__device__ __forceinline__ void tm_vigampl(double x, int nmax, int m, F&& put) {
  if (fabs(1.0 - fabs(x)) <= 1e-10) {
    for (int n = 1; n <= nmax; n++) {
      if (m != 1) { put(n - 1, 0.0, 0.0); continue; }
      double dn = 0.5 * sqrt((double)(n * (n + 1)));
      if (x < 0.0) dn = dn * (((n + 1) & 1) ? -1.0 : 1.0);
      const double v1 = dn;
      if (x < 0.0) dn = -dn;
      put(n - 1, v1, dn);
    }
    return;
  }
  const double qs = sqrt(1.0 - x * x), qs1 = 1.0 / qs, dsi = qs1;
  if (m == 0) {
    double d1 = 1.0, d2 = x;
    for (int n = 1; n <= nmax; n++) {
      const double qn = n, qn1 = n + 1, qn2 = 2 * n + 1;
      const double d3 = (qn2 * x * d2 - qn * d1) / qn1;
      const double der = qs1 * (qn1 * qn / qn2) * (-d1 + d3);
      put(n - 1, d2 * dsi, der);
      d1 = d2;
      d2 = d3;
    }
    return;
  }
  for (int n = 1; n < m && n <= nmax; n++) put(n - 1, 0.0, 0.0);
  const double qmm = (double)(m * m);
  double a = 1.0;
  for (int i = 1; i <= m; i++) a = a * sqrt((double)(2 * i - 1) / (double)(2 * i)) * qs;
  double d1 = 0.0, d2 = a;
  for (int n = m; n <= nmax; n++) {
    const double qn = n, qn2 = 2 * n + 1, qn1 = n + 1;
    const double qnm = sqrt(qn * qn - qmm), qnm1 = sqrt(qn1 * qn1 - qmm);
    const double d3 = (qn2 * x * d2 - qnm * d1) / qnm1;
    const double der = qs1 * (-qn1 * qnm * d1 + qn * qnm1 * d3) / qn2;
    put(n - 1, d2 * dsi, der);
    d1 = d2;
    d2 = d3;
  }
}

// Geometry of AMPL (tmatrix_amplq.lp.f:618-795) for one direction (polar tl,
// azimuth pl in degrees, with the reference's 1e-8 offsets away from the
// singular values; that of the azimuth is epsp): the particle-frame polar cosine, the particle-frame
// azimuth and the lab -> particle polarisation rotation, inverted for the
// scattered direction.  The incident and the scattered direction go through
// the same steps in the reference, so a table of each (per incident angle,
// per scattered angle and azimuth) gives the values of every AMPL call.
struct TmDir {
  double ctp, phip, M[2][2];
};
__device__ void tm_dir(double tl, double pl, double alpha, double beta, bool invert, double epsp, TmDir& d) {
  const double pin = 3.141592653589793, pin2 = pin * 0.5, pi = pin / 180.0;
  const double alph = alpha * pi;
  double bet = beta * pi, thetl = tl * pi, phil = pl * pi;
  const double eps = 1e-8;
  if (thetl < pin2) thetl = thetl + eps;
  if (thetl > pin2) thetl = thetl - eps;
  if (phil < pin) phil = phil + epsp;
  if (phil > pin) phil = phil - epsp;
  if (bet <= pin2 && pin2 - bet <= eps) bet = bet - eps;
  if (bet > pin2 && bet - pin2 <= eps) bet = bet + eps;
  const double cb = cos(bet), sb = sin(bet);
  double ct = cos(thetl), st = sin(thetl), cp = cos(phil - alph), sp = sin(phil - alph);
  const double ctp = ct * cb + st * sb * cp, thetp = acos(ctp);
  const double cpp = cb * st * cp - sb * ct, spp = st * sp;
  double phip = atan(spp / cpp);
  if (phip > 0.0 && sp < 0.0) phip = phip + pin;
  if (phip < 0.0 && sp > 0.0) phip = phip + pin;
  if (phip < 0.0) phip = phip + 2.0 * pin;
  const double ca = cos(alph), sa = sin(alph);
  const double B[3][3] = {{ca * cb, sa * cb, -sb}, {-sa, ca, 0.0}, {ca * sb, sa * sb, cb}};
  cp = cos(phil);
  sp = sin(phil);
  const double AL[3][2] = {{ct * cp, -sp}, {ct * sp, cp}, {-st, 0.0}};
  ct = ctp;
  st = sin(thetp);
  cp = cos(phip);
  sp = sin(phip);
  const double AP[2][3] = {{ct * cp, ct * sp, -st}, {-sp, cp, 0.0}};
  double C[3][2], R[2][2];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 2; j++) {
      double x = 0.0;
#pragma unroll
      for (int k = 0; k < 3; k++) x = x + B[i][k] * AL[k][j];
      C[i][j] = x;
    }
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 2; j++) {
      double x = 0.0;
#pragma unroll
      for (int k = 0; k < 3; k++) x = x + AP[i][k] * C[k][j];
      R[i][j] = x;
    }
  if (invert) {
    const double dd = 1.0 / (R[0][0] * R[1][1] - R[0][1] * R[1][0]);
    d.M[0][0] = R[1][1] * dd;
    d.M[0][1] = -R[0][1] * dd;
    d.M[1][0] = -R[1][0] * dd;
    d.M[1][1] = R[0][0] * dd;
  } else {
    d.M[0][0] = R[0][0];
    d.M[0][1] = R[0][1];
    d.M[1][0] = R[1][0];
    d.M[1][1] = R[1][1];
  }
  d.ctp = ctp;
  d.phip = phip;
}

// Tables of the context: Gauss nodes (block g - 1 < TM_NGAUSS), the constants
// (the next block).
__global__ void __launch_bounds__(TM_NGAUSS) k_tmat_tables(double* tab) {
  const int g = blockIdx.x + 1, t = threadIdx.x;
  if (g <= TM_NGAUSS) {
    if (t < g) tm_gauss_pair(2 * g, t, tab + TMT_X + (size_t)g * (g - 1), tab + TMT_W + (size_t)g * (g - 1));
    return;
  }
  for (int e = t; e < TM_NMAX * TM_NMAX; e += blockDim.x) {
    const int n = e / TM_NMAX + 1, nn = e % TM_NMAX + 1;
    tab[TMT_CAL + e] = sqrt((double)((2 * n + 1) * (2 * nn + 1)) / (double)(n * nn * (n + 1) * (nn + 1)));
  }
  for (int e = t; e < TM_SQ * TM_SQ; e += blockDim.x) {
    const int n = e / TM_SQ, m = e % TM_SQ;
    const double v = n > m ? sqrt((double)(n * n) - (double)(m * m)) : 0.0;
    tab[TMT_SQ + e] = v;
    tab[TMT_RQ + e] = n > m ? 1.0 / v : 0.0;
  }
  if (t < TM_SQ) {
    double a = 1.0;
    for (int i = 1; i <= t; i++) a = a * sqrt((double)(2 * i - 1) / (double)(2 * i));
    tab[TMT_AM + t] = a;
    tab[TMT_I2 + t] = 1.0 / (2 * t + 1);
  }
}

// Directions of a particle of canting angle beta as [TM_DIRD][azimuth][angle]
// (scattered, inverted rotations), then [TM_DIRD][incident angle]: element e
// of 2 nummu TM_NAZH + nummu.
__device__ __forceinline__ void tm_geo(double* geo, int nummu, const double* mu, double beta, int e) {
  const int na = 2 * nummu, ns = na * TM_NAZH;
  TmDir d;
  double* o;
  int stride;
  if (e < ns) {
    const int k = e / na, a = e % na, kk = a / nummu, ll = a % nummu;
    double th = acos(mu[ll] * (kk == 0 ? 1.0 : -1.0)) * 180.0 / PI;
    if (th > 179.9999) th = 180.0;
    const double phi = 360.0 / (double)TM_NAZ * ((double)(k + 1) - 1.0);
    tm_dir(th, phi, 0.0, beta, true, 1e-8, d);
    o = geo + e;
    stride = ns;
  } else {
    double th0 = acos(mu[e - ns] * 1.0) * 180.0 / PI;
    if (th0 > 179.9999) th0 = 180.0;
    tm_dir(th0, 0.0, 0.0, beta, false, beta == 0.0 ? 1e-8 : 1e-14, d);
    o = geo + TM_DIRD * ns + (e - ns);
    stride = nummu;
  }
  double sp, cp;
  sincos(d.phip, &sp, &cp);
  o[0] = d.ctp;
  o[stride] = cp;
  o[2 * stride] = sp;
  o[3 * stride] = d.M[0][0];
  o[4 * stride] = d.M[0][1];
  o[5 * stride] = d.M[1][0];
  o[6 * stride] = d.M[1][1];
}
__global__ void k_tmat_geo(double* geo, int nummu, const double* mu) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < 2 * nummu * TM_NAZH + nummu) tm_geo(geo, nummu, mu, 0.0, e);
}
// TMT_CS: the azimuth difference of an upright particle depends on neither
// polar angle; angle-addition recurrence
__global__ void k_tmat_azimuth(double* tab, const double* geo, int nummu) {
  const int t = threadIdx.x, na = 2 * nummu, ns = na * TM_NAZH;
  if (t >= TM_NAZH) return;
  const double* gin = geo + TM_DIRD * ns;
  const bool pair = t > 0 && t < TM_NAZH - 1;
  const double cs = geo[ns + t * na], ss = geo[2 * ns + t * na], ci = pair ? 1.0 : gin[nummu], si = pair ? 0.0 : gin[2 * nummu];
  const double c1 = fma(cs, ci, ss * si), s1 = fma(ss, ci, -cs * si);
  double cm = 1.0, sm = 0.0;
  for (int m = 0; m <= TM_NMAX; m++) {
    tab[TMT_CS + (m * TM_NAZH + t) * 2] = m ? 2.0 * cm : 1.0;
    tab[TMT_CS + (m * TM_NAZH + t) * 2 + 1] = 2.0 * sm;
    const double cn = cm * c1 - sm * s1;
    sm = sm * c1 + cm * s1;
    cm = cn;
  }
}

// VIGAMPL (see tm_vigampl) times m for the first vector, with the tabulated
// square roots: element n of order m at out[(n - nmin) 2 stride] (m d / sin)
// and + stride (d').
__device__ __forceinline__ void tm_wigner(double x, int nmax, int m, const double* tab, double* out, int stride) {
  const int nmin = max(m, 1);
  if (fabs(1.0 - fabs(x)) <= 1e-10) {
    tm_vigampl(x, nmax, m, [&](int k, double a, double b) {
      if (k + 1 >= nmin) {
        out[(size_t)(k + 1 - nmin) * 2 * stride] = m * a;
        out[(size_t)(k + 1 - nmin) * 2 * stride + stride] = b;
      }
    });
    return;
  }
  const double *sq = tab + TMT_SQ + m, *rq = tab + TMT_RQ + m, *i2 = tab + TMT_I2;
  const double qs = sqrt(1.0 - x * x), qs1 = 1.0 / qs;
  double d1 = 0.0, d2;
  if (m == 0) {
    d1 = 1.0;
    d2 = x;
  } else {
    double q = qs;  // qs^m
    for (int i = 1; i < m; i++) q = q * qs;
    d2 = tab[TMT_AM + m] * q;
  }
  for (int n = nmin; n <= nmax; n++, out += 2 * stride) {
    const double qnm = sq[n * TM_SQ], qnm1 = sq[(n + 1) * TM_SQ];
    const double d3 = fma((2 * n + 1) * x, d2, -qnm * d1) * rq[(n + 1) * TM_SQ];
    out[0] = m * (d2 * qs1);
    out[stride] = (qs1 * i2[n]) * fma((double)n * qnm1, d3, -(n + 1) * qnm * d1);
    d1 = d2;
    d2 = d3;
  }
}

// Lab-frame amplitudes (VV, VH, HV, HH as re, im pairs in v) by the rotations
// of the incident (R) and the scattered direction (R1)
// (tmatrix_amplq.lp.f:868-885), and their quadratic forms z11, z12, z21, z22
// (tmatrix.f90:600-640); s11 and s22 stay in v[0..1], v[6..7].
__device__ __forceinline__ void tm_forms(double (&v)[8], const double* R, int rs, const double* R1, int r1s, double f,
                                         double (&z)[4]) {
  double a[4];
#pragma unroll
  for (int c = 0; c < 4; c++) a[c] = 0.0;
#pragma unroll
  for (int e = 0; e < 2; e++) {
    const double vv = v[e], vh = v[2 + e], hv = v[4 + e], hh = v[6 + e];
    const double cvv = fma(vh, R[2 * rs], vv * R[0]), cvh = fma(vh, R[3 * rs], vv * R[rs]);
    const double chv = fma(hh, R[2 * rs], hv * R[0]), chh = fma(hh, R[3 * rs], hv * R[rs]);
    const double s11 = fma(chv, R1[r1s], cvv * R1[0]), s12 = fma(chh, R1[r1s], cvh * R1[0]);
    const double s21 = fma(chv, R1[3 * r1s], cvv * R1[2 * r1s]), s22 = fma(chh, R1[3 * r1s], cvh * R1[2 * r1s]);
    v[e] = s11;
    v[6 + e] = s22;
    a[0] = fma(s11, s11, a[0]);
    a[1] = fma(s12, s12, a[1]);
    a[2] = fma(s21, s21, a[2]);
    a[3] = fma(s22, s22, a[3]);
  }
  z[0] = f * (a[0] + a[1] + a[2] + a[3]);
  z[1] = f * (a[0] - a[1] + a[2] - a[3]);
  z[2] = f * (a[0] + a[1] - a[2] - a[3]);
  z[3] = f * (a[0] - a[1] - a[2] + a[3]);
}

// P_m of KB scattered directions for one incident angle: VV, VH, HV, HH from
// the Wigner vectors dv [pair][2][sd] and U [pair][8][nummu].
template <int KB>
__device__ __forceinline__ void tm_pm(const double* dv, int sd, const int (&k)[KB], const double* U, int nummu, int nm,
                                      double (&x)[KB][8]) {
#pragma unroll
  for (int j = 0; j < KB; j++)
#pragma unroll
    for (int c = 0; c < 8; c++) x[j][c] = 0.0;
  for (int n = 0; n < nm; n++, dv += 2 * sd, U += 8 * nummu) {
    double u[8];
#pragma unroll
    for (int c = 0; c < 8; c++) u[c] = U[c * nummu];
#pragma unroll
    for (int j = 0; j < KB; j++) {
      const double p = dv[k[j]], q = dv[sd + k[j]];
#pragma unroll
      for (int e = 0; e < 2; e++) {
        x[j][e] = fma(q, u[2 + e], fma(p, u[e], x[j][e]));               // VV = p A1 + q A2
        x[j][2 + e] = fma(q, u[6 + e], fma(p, u[4 + e], x[j][2 + e]));   // VH = p B1 + q B2
        x[j][4 + e] = fma(-p, u[2 + e], fma(-q, u[e], x[j][4 + e]));     // HV = -(q A1 + p A2)
        x[j][6 + e] = fma(p, u[6 + e], fma(q, u[4 + e], x[j][6 + e]));   // HH = q B1 + p B2
      }
    }
  }
}

// Extinction of incident angle jj from the forward amplitudes, and the
// backscattering matrix (tmatrix.f90:645-665).
__device__ __forceinline__ void tm_forward(double* ext, int jj, double fext, const double (&amp)[8]) {
  const double sp = fext * (amp[1] + amp[7]), sm = fext * (amp[1] - amp[7]);
  ext[0 + 2 * (0 + 2 * jj)] = sp;
  ext[0 + 2 * (1 + 2 * jj)] = sm;
  ext[1 + 2 * (0 + 2 * jj)] = sm;
  ext[1 + 2 * (1 + 2 * jj)] = sp;
}
__device__ __forceinline__ void tm_back(double* sback, const double (&z)[4]) {
  sback[0] = z[0];
  sback[2] = z[1];
  sback[1] = z[2];
  sback[3] = z[3];
}

// Particles of a record's kind, their outputs and factors.
struct TmUnit {
  int p, nmax;
  double fact, fext;
  double *scat, *ext, *sback;
  const double* rec;
  __device__ __forceinline__ TmUnit(const TmArgs& A, int p_) : p(p_) {
    nmax = A.nmax[p];
    const double wave_num = 2.0 * PI / (C_LIGHT / A.freq[p / A.nbins]);
    fact = 0.5 / (wave_num * wave_num);
    fext = 2.0 * PI / (wave_num * wave_num);
    scat = A.scat + (size_t)p * 8 * A.nummu * A.nummu;
    ext = A.ext + (size_t)p * 4 * A.nummu;
    sback = A.sback + (size_t)p * 4;
    rec = A.records + A.rec[p];
  }
};

// Scattered angle a of a canted particle: the Wigner vectors of its 16
// azimuths, then (incident angle, two azimuths) per thread.  buf: DV
// [pair][2][azimuth] where it fits shared memory, then the azimuth terms.
__device__ __forceinline__ void tm_canted(const TmArgs& A, const TmUnit& X, int a, double* buf, double* scratch) {
  constexpr int KB = 2;
  const int t = threadIdx.x, nummu = A.nummu, na = 2 * nummu, ns = na * TM_NAZH, nmax = X.nmax;
  const int npair = tm_pair0(nmax, nmax) + 1;
  const double *U = X.rec, *geo = U + (size_t)npair * 8 * nummu, *gin = geo + TM_DIRD * ns;
  double* const zt = buf;  // [azimuth][4][nummu]
  double* const DV = TM_NAZH * 4 * nummu + npair * 2 * TM_NAZH <= TMA_SMEM ? buf + TM_NAZH * 4 * nummu : scratch;
  const double phi_weights = 1.0 / 360.0 * (360.0 / TM_NAZ);
  for (int e = t; e < (nmax + 1) * TM_NAZH; e += TMA_THREADS) {
    const int m = e / TM_NAZH, k = e % TM_NAZH;
    tm_wigner(geo[k * na + a], nmax, m, A.tab, DV + tm_pair0(nmax, m) * 2 * TM_NAZH + k, TM_NAZH);
  }
  __syncthreads();
  const int jj = t % nummu, slot = t / nummu, nslot = TMA_THREADS / nummu;
  const double ci = gin[nummu + jj], si = gin[2 * nummu + jj];
  for (int k0 = slot * KB; k0 < TM_NAZH; k0 += nslot * KB) {
    int k[KB];
    double amp[KB][8], c1[KB], s1[KB], cm[KB], sm[KB];
#pragma unroll
    for (int j = 0; j < KB; j++) {
      k[j] = min(k0 + j, TM_NAZH - 1);
      // azimuth difference of the scattered and the incident direction
      const double cs = geo[ns + k[j] * na + a], ss = geo[2 * ns + k[j] * na + a];
      c1[j] = fma(cs, ci, ss * si);
      s1[j] = fma(ss, ci, -cs * si);
      cm[j] = 1.0;
      sm[j] = 0.0;
#pragma unroll
      for (int c = 0; c < 8; c++) amp[j][c] = 0.0;
    }
    const double *d = DV, *u = U + jj;
    for (int m = 0; m <= nmax; m++) {
      const int nm = nmax - max(m, 1) + 1;
      double x[KB][8];
      tm_pm<KB>(d, TM_NAZH, k, u, nummu, nm, x);
      d += nm * 2 * TM_NAZH;
      u += nm * 8 * nummu;
#pragma unroll
      for (int j = 0; j < KB; j++) {
        const double fc = m ? 2.0 * cm[j] : 1.0, fs = 2.0 * sm[j];
#pragma unroll
        for (int e = 0; e < 2; e++) {
          amp[j][e] = fma(fc, x[j][e], amp[j][e]);
          amp[j][2 + e] = fma(fs, x[j][2 + e], amp[j][2 + e]);
          amp[j][4 + e] = fma(fs, x[j][4 + e], amp[j][4 + e]);
          amp[j][6 + e] = fma(fc, x[j][6 + e], amp[j][6 + e]);
        }
        const double cn = cm[j] * c1[j] - sm[j] * s1[j];
        sm[j] = sm[j] * c1[j] + cm[j] * s1[j];
        cm[j] = cn;
      }
    }
#pragma unroll
    for (int j = 0; j < KB; j++) {
      if (k0 + j >= TM_NAZH) continue;
      double z[4];
      tm_forms(amp[j], gin + 3 * nummu + jj, nummu, geo + 3 * ns + k[j] * na + a, ns, X.fact, z);
      if (k[j] == 0) {
        if (a == na - 1 && jj == nummu - 1) tm_back(X.sback, z);  // 180 deg
        if (a == jj) tm_forward(X.ext, jj, X.fext, amp[j]);
      }
#pragma unroll
      for (int c = 0; c < 4; c++)
        zt[(k[j] * 4 + c) * nummu + jj] = z[c] * (k[j] == 0 || k[j] == TM_NAZH - 1 ? phi_weights : 2.0 * phi_weights);
    }
  }
  __syncthreads();
  for (int e = t; e < 4 * nummu; e += TMA_THREADS) {
    double z = 0.0;
#pragma unroll 8
    for (int k = 0; k < TM_NAZH; k++) z = z + zt[k * 4 * nummu + e];
    const int c = e / nummu, j = e % nummu, kk = a / nummu, ll = a % nummu;
    X.scat[(c >> 1) + 2 * (ll + nummu * ((c & 1) + 2 * (j + nummu * kk)))] = z;
  }
}

// 128 (incident, scattered) angle pairs of an upright particle, one per
// thread: P_m of every order into the thread's own column of buf, then the 16 azimuths, four
// at a time.  No barrier.
__device__ __forceinline__ void tm_upright(const TmArgs& A, const TmUnit& X, int part, double* buf, double* scratch) {
  constexpr int KB = 4;
  static_assert(TM_NAZH % KB == 0, "azimuths per pass");
  const int t = threadIdx.x, nummu = A.nummu, na = 2 * nummu, ns = na * TM_NAZH, nmax = X.nmax;
  const int npair = tm_pair0(nmax, nmax) + 1;
  const int a = t % na, jj = part * (TMA_THREADS / na) + t / na;
  double* const P = ((nmax + 1) * 8 * TMA_THREADS <= TMA_SMEM ? buf : scratch) + t;
  const double *u = X.rec + jj, *d = X.rec + (size_t)npair * 8 * nummu + a;
  for (int m = 0; m <= nmax; m++) {
    double x[8];
#pragma unroll
    for (int c = 0; c < 8; c++) x[c] = 0.0;
#pragma unroll 2
    for (int n = max(m, 1); n <= nmax; n++, d += 2 * na, u += 8 * nummu) {
      const double p = d[0], q = d[na];
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const double a1 = u[e * nummu], a2 = u[(2 + e) * nummu], b1 = u[(4 + e) * nummu], b2 = u[(6 + e) * nummu];
        x[e] = fma(q, a2, fma(p, a1, x[e]));
        x[2 + e] = fma(q, b2, fma(p, b1, x[2 + e]));
        x[4 + e] = fma(-p, a2, fma(-q, a1, x[4 + e]));
        x[6 + e] = fma(p, b2, fma(q, b1, x[6 + e]));
      }
    }
#pragma unroll
    for (int c = 0; c < 8; c++) P[(m * 8 + c) * TMA_THREADS] = x[c];
  }
  const double *geo = A.geo, *gin = geo + TM_DIRD * ns, *cst = A.tab + TMT_CS;
  const double phi_weights = 1.0 / 360.0 * (360.0 / TM_NAZ);
  double zs[4] = {0.0, 0.0, 0.0, 0.0};
  for (int k0 = 0; k0 < TM_NAZH; k0 += KB) {
    double amp[KB][8];
#pragma unroll
    for (int j = 0; j < KB; j++)
#pragma unroll
      for (int c = 0; c < 8; c++) amp[j][c] = 0.0;
    for (int m = 0; m <= nmax; m++) {
      double x[8];
#pragma unroll
      for (int c = 0; c < 8; c++) x[c] = P[(m * 8 + c) * TMA_THREADS];
#pragma unroll
      for (int j = 0; j < KB; j++) {
        const double2 cs = *reinterpret_cast<const double2*>(cst + (m * TM_NAZH + k0 + j) * 2);
#pragma unroll
        for (int e = 0; e < 2; e++) {
          amp[j][e] = fma(cs.x, x[e], amp[j][e]);
          amp[j][2 + e] = fma(cs.y, x[2 + e], amp[j][2 + e]);
          amp[j][4 + e] = fma(cs.y, x[4 + e], amp[j][4 + e]);
          amp[j][6 + e] = fma(cs.x, x[6 + e], amp[j][6 + e]);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < KB; j++) {
      const int k = k0 + j;
      double z[4];
      tm_forms(amp[j], gin + 3 * nummu + jj, nummu, geo + 3 * ns + k * na + a, ns, X.fact, z);
      if (k == 0) {
        if (a == na - 1 && jj == nummu - 1) tm_back(X.sback, z);  // 180 deg
        if (a == jj) tm_forward(X.ext, jj, X.fext, amp[j]);
      }
#pragma unroll
      for (int c = 0; c < 4; c++) zs[c] = zs[c] + z[c] * (k == 0 || k == TM_NAZH - 1 ? phi_weights : 2.0 * phi_weights);
    }
  }
  const int kk = a / nummu, ll = a % nummu;
#pragma unroll
  for (int c = 0; c < 4; c++) X.scat[(c >> 1) + 2 * (ll + nummu * ((c & 1) + 2 * (jj + nummu * kk)))] = zs[c];
}

// Persistent CTAs over the units of this round's particles.
__global__ void __launch_bounds__(TMA_THREADS, 3) k_tmat_ampl(TmArgs A) {
  extern __shared__ __align__(16) double smem_raw[];
  __shared__ int unit;
  double* scratch = A.ascratch + (size_t)blockIdx.x * TMA_SLOT;
  const int na = 2 * A.nummu, per = A.nummu * na / TMA_THREADS;  // units of an upright particle
  const int nu = A.round->upright * per, n = nu + A.round->canted * na;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) unit = atomicAdd(&A.round->units, 1);
    __syncthreads();
    const int k = unit;
    if (k >= n) break;
    if (k < nu) {
      const TmUnit X(A, A.upright[k / per]);
      tm_upright(A, X, k % per, smem_raw, scratch);
    } else {
      const TmUnit X(A, A.canted[(k - nu) / na]);
      tm_canted(A, X, (k - nu) % na, smem_raw, scratch);
    }
  }
}

// One particle: the converged T-matrix and its record.  Whole CTA.
__device__ void tm_particle(const TmArgs& A, double* s, const TmSlot& L, TmShared& sh, int p) {
  const int t = threadIdx.x, warp = t >> 5, nummu = A.nummu, na = 2 * nummu;
  auto none = [&](int nmax, int status) {  // no particle, or none that converges
    if (t == 0) {
      A.nmax[p] = nmax;
      if (status) A.status[p] |= status;
    }
  };
  if (A.ndens[p] == 0.0) { none(0, 0); return; }
  const int item = p / A.nbins;
  const double lam = C_LIGHT / A.freq[item];
  const double mrr = A.mrr[p], mri = A.mri[p], axi = A.axi[p], asr = A.asr[p], beta = A.beta[p];
  TmPart Q;
  Q.lam = lam;
  Q.mrr = mrr;
  Q.mri = mri;
  Q.eps = 1.0 / asr;
  Q.rev = 1.0 * axi;
  const double a0 = Q.rev * pow(Q.eps, 1.0 / 3.0);
  Q.aa = a0 * a0;
  Q.ee1 = Q.eps * Q.eps - 1.0;
  Q.pi = 2.0 * 3.141592653589793 / lam;  // k (P * 2 / LAM)
  Q.ppi = Q.pi * Q.pi;
  Q.pir = Q.ppi * mrr;
  Q.pii = Q.ppi * mri;
  const double xev = 2.0 * 3.141592653589793 * Q.rev / lam;
  const int inm1 = tm_inm1(xev);
  const double* tab = A.tab;
  int fail = 0, nmax = inm1, ngauss = 0;
  double qext1 = 0.0, qsca1 = 0.0;
  bool conv = false, gauss_done = false;
  double *sf = s, *free_s = s;  // region of the last solve, end of the regions in use
  // does a step's result stay within 0.1 % of the one before
  auto settled = [&](int c) {
    const double qext = sh.qe[c], qsca = sh.qs[c];
    const double dsca = fabs((qsca1 - qsca) / qsca), dext = fabs((qext1 - qext) / qext);
    qext1 = qext;
    qsca1 = qsca;
    return dsca <= 0.001 && dext <= 0.001;
  };
  // NMAX convergence (tmatrix_amplq.lp.f:386-431), then at least one step of
  // the Gauss points (:432-470).  NMAX and NMAX + 1 with 2 NMAX points and
  // NMAX + 1 with one point more, the usual last step, go side by side while
  // they fit the pool.
  while (!fail && !conv && nmax < TM_NMAX && 2 * (nmax + 1) + 1 <= TM_NGAUSS && 3 * tm_need(nmax + 1, 2 * nmax + 3) <= TM_POOL) {
    const int region = tm_need(nmax + 1, 2 * nmax + 3);
    const TmStep st[3] = {{nmax, 2 * nmax, s}, {nmax + 1, 2 * nmax + 2, s + region}, {nmax + 1, 2 * nmax + 3, s + 2 * region}};
    tm_steps<3>(st, Q, sh, tab);
    free_s = s + 3 * region;
    int last = -1;  // the step that settled
    for (int c = 0; c < 2 && !conv; c++) {
      if (!sh.ok[c]) { fail = 1; nmax += c; break; }
      conv = settled(c);
      last = c;
    }
    if (conv) {
      nmax += last;
      ngauss = 2 * nmax;
      if (last == 1) {  // the third step is the Gauss step of this NMAX
        ngauss++;
        sf = s + 2 * region;
        if (!sh.ok[2]) fail = 1;
        else gauss_done = settled(2);
      }
    } else if (!fail) {
      nmax += 2;
    }
  }
  auto single = [&]() {
    const TmStep st[1] = {{nmax, ngauss, s}};
    tm_steps<1>(st, Q, sh, tab);
    sf = s;
    free_s = s + tm_need(nmax, ngauss);
  };
  for (; !fail && !conv && nmax <= TM_NMAX; nmax++) {
    ngauss = 2 * nmax;
    if (ngauss > TM_NGAUSS) { fail = 1; break; }
    single();
    if (!sh.ok[0]) { fail = 1; break; }
    conv = settled(0);
    if (conv) break;
  }
  if (!conv) fail = 1;
  while (!fail && !gauss_done) {
    if (++ngauss > TM_NGAUSS) { fail = 1; break; }
    single();
    if (!sh.ok[0]) { fail = 1; break; }
    gauss_done = settled(0);
  }
  if (fail) { none(-nmax, PAMTRA_B200_FATAL | PAMTRA_B200_ST_RANGE); return; }
  // single-precision T of every order m (:472-556)
  float2* T = reinterpret_cast<float2*>(s + L.t);
  tm_store(tm_aug(sf), T, 0, nmax, t, TM_THREADS);
  const double *X = tab + TMT_X + (size_t)ngauss * (ngauss - 1), *W = tab + TMT_W + (size_t)ngauss * (ngauss - 1);
  __syncthreads();
  if (t == 0) sh.ok[0] = 1;
  const int dsz = 2 * ngauss * nmax;
  if ((free_s - s) + tm_need_all(nmax, ngauss) <= TM_POOL) {
    // all orders side by side: the system of order m at as + 4 (sum of nm^2
    // of the orders before), its Wigner tables at ds + (m - 1) dsz
    cplx* const as = reinterpret_cast<cplx*>(free_s);
    double* const ds = free_s + 8 * tm_cubes(nmax);
    for (int e = t; e < nmax * ngauss; e += TM_THREADS) {
      const int m = 1 + e / ngauss;
      tm_wnode(ds + (m - 1) * dsz, X, e % ngauss, m, nmax, ngauss);
    }
    __syncthreads();
    const int np = tm_cubes(nmax);
    for (int e = t, m = 1, o = 0; e < np; e += TM_THREADS) {
      int nm = nmax - m + 1;
      while (e - o >= nm * nm) {
        o += nm * nm;
        m++;
        nm--;
      }
      tm_pair(as + 4 * o, sf, ds + (m - 1) * dsz, W, m, m + (e - o) / nm, m + (e - o) % nm, nmax, ngauss, Q);
    }
    __syncthreads();
    for (int k = warp; k < 2 * nmax; k += TM_WARPS) {
      const int m = 1 + (k >> 1), nm = nmax - m + 1;
      const TmSystems sy(m, nm);
      if (!tm_eliminate<1>(as + 4 * (np - tm_cubes(nm)) + sy.base(k & 1), nm, sh) && (t & 31) == 0) sh.ok[0] = 0;
    }
    __syncthreads();
    for (int m = 1; m <= nmax; m++) tm_store(as + 4 * (np - tm_cubes(nmax - m + 1)), T, m, nmax, t, TM_THREADS);
  } else {
    double* const D = tm_d(sf, 0, nmax, ngauss);
    for (int m = 1; m <= nmax; m++) {
      const int nm = nmax - m + 1;
      for (int k = t; k < ngauss; k += TM_THREADS) tm_wnode(D, X, k, m, nmax, ngauss);
      __syncthreads();
      for (int e = t; e < nm * nm; e += TM_THREADS) tm_pair(tm_aug(sf), sf, D, W, m, m + e / nm, m + e % nm, nmax, ngauss, Q);
      __syncthreads();
      const TmSystems sy(m, nm);
      bool ok = true;
      for (int k = 0; k < 2 && ok; k++) ok = tm_eliminate<TM_WARPS>(tm_aug(sf) + sy.base(k), nm, sh);
      if (!ok) {
        if (t == 0) sh.ok[0] = 0;
        break;
      }
      tm_store(tm_aug(sf), T, m, nmax, t, TM_THREADS);
      __syncthreads();
    }
  }
  // (m, n) of a pair
  for (int m = t; m <= nmax; m += TM_THREADS) {
    int o = tm_pair0(nmax, m);
    for (int n = max(m, 1); n <= nmax; n++) sh.pm[o++] = (uint16_t)(m | (n << 8));
  }
  const bool upright = (beta == 0.0);
  const int npair = tm_pair0(nmax, nmax) + 1;
  if (t == 0) {
    const size_t need = tm_record(npair, nummu, upright);
    const unsigned long long o = atomicAdd(&A.round->used, (unsigned long long)need);
    sh.rec = o + need <= A.rec_doubles ? (long long)o : -1;
  }
  __syncthreads();
  if (!sh.ok[0]) { none(-nmax, PAMTRA_B200_FATAL | PAMTRA_B200_ST_RANGE); return; }
  if (sh.rec < 0) {
    if (t == 0) A.again[atomicAdd(&A.next->n, 1)] = p;
    return;
  }
  // ---------------- what the amplitudes take from T (tmatrix.f90:560-600)
  double* const U = A.records + sh.rec;
  double* const rest = U + (size_t)npair * 8 * nummu;  // scattered Wigner vectors or directions
  double* const DVI = s + L.dvi;
  const int ns = na * TM_NAZH;
  const double* geo = A.geo;
  if (!upright) {
    for (int e = t; e < ns + nummu; e += TM_THREADS) tm_geo(rest, nummu, A.mu, beta, e);
    geo = rest;
    __syncthreads();
  }
  const double* gin = geo + TM_DIRD * ns;
  // Wigner vectors of the incident angles, and of the scattered ones of an upright particle
  const int nd = nummu + (upright ? na : 0);
  for (int e = t; e < (nmax + 1) * nd; e += TM_THREADS) {
    const int m = e / nd, d = e % nd, pr = tm_pair0(nmax, m);
    if (d < nummu) tm_wigner(gin[d], nmax, m, tab, DVI + (size_t)pr * 2 * nummu + d, nummu);
    else tm_wigner(geo[d - nummu], nmax, m, tab, rest + (size_t)pr * 2 * na + d - nummu, na);
  }
  __syncthreads();
  // U = sum over nn of CAL(n, nn) T(m, n, nn) with the incident vectors p0, q0:
  // A1 = T11 p0 + T12 q0, A2 = T21 p0 + T22 q0, B1 = T11 q0 + T12 p0, B2 = T21 q0 + T22 p0
  for (int e = t; e < npair * nummu; e += TM_THREADS) {
    const int pr = e / nummu, jj = e % nummu, m = sh.pm[pr] & 255, n = sh.pm[pr] >> 8;
    const int nmin = max(m, 1), nm = nmax - nmin + 1;
    const float2* tp = T + tm_t0(nmax, m) + (n - nmin) * nm;
    const double* dv = DVI + (size_t)tm_pair0(nmax, m) * 2 * nummu + jj;
    const double* cal = tab + TMT_CAL + (size_t)(n - 1) * TM_NMAX + nmin - 1;
    double u[8];
#pragma unroll
    for (int c = 0; c < 8; c++) u[c] = 0.0;
    for (int k = 0; k < nm; k++) {
      const double p0 = dv[(size_t)k * 2 * nummu], q0 = dv[(size_t)k * 2 * nummu + nummu], rn = cal[k];
      const int ph = (nmin + k - n - 1) & 3;  // CAL = rn i^ph
      double c[4][2];
#pragma unroll
      for (int b = 0; b < 4; b++) {
        const float2 f = tp[b * nm * nm + k];
        const double x = rn * f.x, y = rn * f.y;
        c[b][0] = (ph & 1) ? ((ph & 2) ? y : -y) : ((ph & 2) ? -x : x);
        c[b][1] = (ph & 1) ? ((ph & 2) ? -x : x) : ((ph & 2) ? -y : y);
      }
#pragma unroll
      for (int i = 0; i < 2; i++) {
        u[i] = fma(c[1][i], q0, fma(c[0][i], p0, u[i]));
        u[2 + i] = fma(c[3][i], q0, fma(c[2][i], p0, u[2 + i]));
        u[4 + i] = fma(c[1][i], p0, fma(c[0][i], q0, u[4 + i]));
        u[6 + i] = fma(c[3][i], p0, fma(c[2][i], q0, u[6 + i]));
      }
    }
#pragma unroll
    for (int c = 0; c < 8; c++) U[((size_t)pr * 8 + c) * nummu + jj] = u[c];
  }
  if (t == 0) {
    A.nmax[p] = nmax;
    A.rec[p] = sh.rec;
    if (upright) A.upright[atomicAdd(&A.round->upright, 1)] = p;
    else A.canted[atomicAdd(&A.round->canted, 1)] = p;
  }
}

// Persistent CTAs of eight warps over the particles of a round, one scratch slot
// each.
__global__ void __launch_bounds__(TM_THREADS, 2) k_tmatrix(TmArgs A) {
  __shared__ TmShared sh;
  const TmSlot L = tm_slot(A.nummu);
  double* s = A.scratch + (size_t)blockIdx.x * L.total;
  const int np = A.round->n;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) {
      const int k = atomicAdd(&A.round->taken, 1);
      sh.particle = k < np ? A.order[k] : -1;
      // a full record pool: the rest waits
      if (k < np && *reinterpret_cast<volatile unsigned long long*>(&A.round->used) >= A.rec_doubles) {
        A.again[atomicAdd(&A.next->n, 1)] = sh.particle;
        sh.particle = -2;
      }
    }
    __syncthreads();
    const int p = sh.particle;
    if (p == -1) break;
    if (p >= 0) tm_particle(A, s, L, sh, p);
  }
}

// Per-bin set-up of calc_tmatrix (src/tmatrix.f90:124-183): input checks,
// the soft-spheroid index of ice bins (eps_mix with air), the equal-volume
// radius from the maximum dimension and the aspect ratio.  A bin that fails
// a check gets FATAL | ST_RANGE and no particle.
__global__ void k_tmat_prep(int n_items, int nbins, const double* freq, const double* ref_re, const double* ref_im, const int* phase,
                            const double* dmax, const double* del_d, const double* ndens, const double* density,
                            const double* asr, const double* canting, double* mrr, double* mri, double* axi,
                            double* nd_eff, int* status, int* key) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n_items * nbins) return;
  const int item = p / nbins;
  const double nd = ndens[p];
  status[p] = 0;
  nd_eff[p] = 0.0;
  key[p] = 0;
  mrr[p] = mri[p] = axi[p] = 0.0;
  if (nd == 0.0) return;
  const bool bad = !(nd > 0.0) || !(del_d[p] > 0.0) || !(density[p] > 0.0) || !(asr[p] > 0.0) ||
                   !(dmax[p] > 0.0) || !(canting[p] >= 0.0) || canting[p] > 180.0 ||
                   (phase[item] != 1 && phase[item] != -1) || !(freq[item] > 0.0) || !isfinite(freq[item]) ||
                   !isfinite(ref_re[item]) || !isfinite(ref_im[item]) || !isfinite(dmax[p]) || !isfinite(asr[p]);
  if (bad) {
    status[p] = PAMTRA_B200_FATAL | PAMTRA_B200_ST_RANGE;
    return;
  }
  cplx m = cmk(ref_re[item], ref_im[item]);
  if (phase[item] == -1 && density[p] != 917.0) m = eps_mix_m(m, density[p]);
  mrr[p] = m.re;
  mri[p] = fabs(-m.im);  // mindex = conjg(mMix); the solve takes |Im|
  const double a = asr[p];
  axi[p] = (a <= 1.0) ? 0.5 * dmax[p] * pow(a, 1.0 / 3.0) : 0.5 * dmax[p] / pow(a, 2.0 / 3.0);
  nd_eff[p] = nd;
  key[p] = min(63, tm_inm1(2.0 * 3.141592653589793 * axi[p] * freq[item] / C_LIGHT));
}


// Particles by decreasing first NMAX (key, 0 .. 63; 0: no particle): a particle
// of NMAX 13 takes five times one of NMAX 5, and the last ones to start decide
// when the launch ends.  One block; the order within a key is immaterial, since
// particles do not depend on one another.
__global__ void __launch_bounds__(1024) k_tmat_order(int n, const int* key, int* order, TmRound* first) {
  __shared__ int start[64];
  if (threadIdx.x < 64) start[threadIdx.x] = 0;
  if (threadIdx.x == 0) first->n = n;
  __syncthreads();
  for (int p = threadIdx.x; p < n; p += blockDim.x) atomicAdd(&start[key[p]], 1);
  __syncthreads();
  if (threadIdx.x == 0) {
    int acc = 0;
    for (int k = 63; k >= 0; k--) { const int v = start[k]; start[k] = acc; acc += v; }
  }
  __syncthreads();
  for (int p = threadIdx.x; p < n; p += blockDim.x) order[atomicAdd(&start[key[p]], 1)] = p;
}

// Species sums of calc_tmatrix (src/tmatrix.f90:413-416) in bin order, and
// the per-bin "NN" backscattering 4 pi ndens Sback(1,1) (:383).  Thread per
// (item, element): block y takes 256 elements of item x, block 0 the per-bin
// values too.
__global__ void __launch_bounds__(256) k_tmat_sum(int n_items, int nbins, int nummu, const double* ndens, const double* del_d,
                                                  const double* pscat, const double* pext, const double* psback,
                                                  const int* pstatus, double* scat, double* ext, double* sback,
                                                  double* back_spec, int* status) {
  const int item = blockIdx.x;
  const size_t NS = (size_t)2 * nummu * 2 * nummu * 2, NE = 4 * (size_t)nummu;
  const size_t tot = NS + NE + 4, e = (size_t)blockIdx.y * 256 + threadIdx.x;
  if (e < tot) {
    // this element's array, its length per particle and place in it
    const double* src = pscat;
    double* dst = scat;
    size_t len = NS, o = e;
    if (e >= NS + NE) { src = psback; dst = sback; len = 4; o = e - NS - NE; }
    else if (e >= NS) { src = pext; dst = ext; len = NE; o = e - NS; }
    src += (size_t)item * nbins * len + o;
    double acc = 0.0;
#pragma unroll 8
    for (int b = 0; b < nbins; b++) {
      const size_t p = (size_t)item * nbins + b;
      const double nd = ndens[p], v = src[(size_t)b * len];
      if (nd == 0.0 || pstatus[p]) continue;
      acc = acc + v * nd * del_d[p];
    }
    dst[(size_t)item * len + o] = acc;
  }
  if (blockIdx.y) return;
  for (int b = threadIdx.x; b < nbins; b += blockDim.x) {
    const size_t p = (size_t)item * nbins + b;
    back_spec[p] = (ndens[p] == 0.0 || pstatus[p]) ? 0.0 : 4.0 * PI * ndens[p] * psback[p * 4];
  }
  if (threadIdx.x == 0) {
    int st = 0;
    for (int b = 0; b < nbins; b++) st |= pstatus[(size_t)item * nbins + b];
    status[item] = st;
  }
}

// Emission vector of an item: extinction minus the scattering integrated over
// the sphere (tmatrix.f90:670-680), linear in the bins and so taken from the
// sums.
__global__ void k_tmat_emis(int n_items, int nummu, const double* wq, const double* scat, const double* ext, double* emis) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n_items * 2 * nummu) return;
  const int item = e / (2 * nummu), jj = (e >> 1) % nummu, i1 = e & 1;
  const double* s = scat + (size_t)item * 8 * nummu * nummu;
  double v = 0.0;
#pragma unroll 8
  for (int k = 0; k < 2 * nummu; k++)
    v = v + s[2 * (k % nummu + nummu * (i1 + 2 * (jj + nummu * (k / nummu))))] * wq[k % nummu] * 2.0 * PI;
  emis[e] = ext[(size_t)item * 4 * nummu + 2 * (i1 + 2 * jj)] - v;
}

}  // namespace pb
