// RT4 on the GPU.
//   k_layer<N>: per (present layer, frequency) item -- scatcnv (Legendre
//     series -> quadrature phase matrices), check_norm4, INITIALIZE4 /
//     INITIAL_SOURCE4 and DOUBLING_INTEGRATION4; writes the layer's R, T and
//     S+/S- to the scratch arena.
// The adding of a column's layers is in adding.cuh.  Both are persistent
// kernels: one CTA ("team", see common.cuh) per item, items taken from a
// device-side counter.
#pragma once
#include "common.cuh"
#include "work.cuh"

namespace pb {

constexpr double TWO_PI = 2.0 * 3.1415926535897932384;
constexpr double LN2_F32 = 0.693147182464599609375;  // log(2.) in REAL(4) (radtran4.f90:325)
constexpr int KMAX = 104;                             // azimuth points: numpts/2+1 for nlegen <= 199

// Legendre upward-recurrence coefficients P_l = a_l x P_{l-1} - b_l P_{l-2},
// a_l = (2l-1)/l, b_l = (l-1)/l (filled at context creation).
__constant__ double c_leg_a[MAXNLEG], c_leg_b[MAXNLEG];

// src/rt_utilities.f90:69-90 PLANCK_FUNCTION, UNITS='r'
__device__ __forceinline__ double planck(double T, double wl) {
  return (T > 0.0) ? 1.1911e8 / p5(wl) / (exp(1.4388e4 / (wl * T)) - 1) : 0.0;
}

// src/rt_utilities.f90:687-735 CONVERT_OUTPUT (UNITS='T', FLUXCODE=0)
__device__ __forceinline__ double rad_to_tb(double rad, double wl) {
  if (rad > 0.0) return 1.4388e4 / (wl * log(1.0 + 1.1911e8 / (rad * p5(wl))));
  if (rad == 0.0) return 0.0;
  return -1.4388e4 / (wl * log(1.0 + 1.1911e8 / (-rad * p5(wl))));
}

template <int N>
struct RTCfg {
  static constexpr int n = 2 * N;
  static constexpr int T = Team<n>::T;
  static constexpr int LD = Team<n>::LD;
  static constexpr int MAT = Team<n>::MAT;
};

__host__ __device__ __forceinline__ size_t lay_stride_n(int N) {
  const int n = 2 * N;
  return 2 * (size_t)n * (n + 4) + 2 * n;
}

// ============================================================== layer kernel
// With M = diag(mu_j w_j) the layer matrices of Mie spheres are symmetric in
// the scaled form M^(1/2) R M^(-1/2) (reciprocity: the azimuth-mean phase
// matrix of (I, Q) obeys P(mu1, mu2) = P(mu2, mu1)^T, and likewise for
// (-mu1, mu2)), and doubling keeps them so.  k_layer carries R and T scaled.
template <int N>
struct LayerSmem {
  static constexpr int n = 2 * N, LMAT = RTCfg<N>::MAT;
  static constexpr int COEF = 3 * MAXNLEG;
  // R, T, X and Y^T of the doubling (SymTeam layout); before it the set-up's R
  // and T (column-major, leading dimension n + 4), coefficients and azimuth
  // table; the elimination's I - X takes X and Y
  static constexpr int M = (4 * SymTeam<n>::MAT > 2 * LMAT + COEF + 2 * KMAX) ? 4 * SymTeam<n>::MAT : 2 * LMAT + COEF + 2 * KMAX;
  static_assert(LMAT <= 2 * SymTeam<n>::MAT, "the elimination's matrix fits X and Y");
  alignas(16) double m[M];
  alignas(16) double C[n], E[n];    // constant source C and e = o - f C / 2
  alignas(16) double UC[n], UE[n];  // C + R C, e - R e
  double o[n];                    // odd part of the linear source
  double lin[2 * n], cst[2 * n];  // thin-layer sources of layer_setup
  double mu[N], wq[N], nrm[N];
  double sc[n], is[n];            // sqrt(mu w) per row and its inverse
  double fro[n / 8];              // sums of squares of the scaled R, per warp
  InvScratch<n> inv;
  int item;
  // set-up buffers (layer_setup): 0 R, 1 T, 2 coefficients, 4 azimuth table
  __device__ __forceinline__ double* mat(int k) {
    return m + (k < 2 ? k * LMAT : 2 * LMAT + (k == 4 ? COEF : 0));
  }
};

// Azimuth weights of scatcnv (src/scatcnv.f90:103-192 with SUM_LEGENDRE,
// ROTATE_PHASE_MATRIX, MATRIX_SYMMETRY and FOURIER_BASIS order 0 of
// src/rt_utilities.f90:242-493).  For NSTOKES = 2 the m = 0 phase-matrix
// entries of one (mu1, mu2) pair are linear in the Legendre coefficients
// c0, c1, c2 of an item:
//   P11 = sum_l c0_l A_l,  P12 = sum_l c1_l B_l,  P21 = sum_l c1_l C_l,
//   P22 = sum_l (c0_l D_l + c2_l E_l),
// where A..E are the azimuth sums over k = 0..numpts/2 (weight 1 at the two
// ends, 2 inside, / numpts) of P_l(cos Theta_k) times 1, cos 2i1, cos 2i2,
// cos 2i1 cos 2i2 and -sin 2i1 sin 2i2.  Exchanging mu1 and mu2 exchanges i1 and
// i2: A, D and E stay, B and C change places.  Turning mu1 over, with k from
// the other end, turns cos Theta over and sin 2i2 too: A .. D gain (-1)^l, E
// loses it.  So the table holds the pairs 0 < mu1 <= mu2 (index j2 (j2 + 1) / 2 + j1)
// and an item's sums over even and over odd l give both signs and both
// orders: 136 of 512 pairs for N = 16.  Layer stage (latency of these L2 reads
// before the doubling): 13.4 -> 13.0 ms for 1024 columns of the split form, 20.0 ->
// 19.7 ms for 40 columns of mixed NUMMU, 3.18 -> 3.12 ms for 40 Mie-heavy ones.
// The tables depend only on NUMMU and numpts, so one kernel fills every
// numpts a batch has met (wt_need) that is not filled yet (wt_ready); one thread
// per (numpts, mu1, mu2).
__device__ __forceinline__ int scat_pair_row(int pair) {  // j2 of a pair
  int j = (int)((sqrtf(8.0f * pair + 1.0f) - 1.0f) * 0.5f);
  while (j * (j + 1) / 2 > pair) j--;
  while ((j + 1) * (j + 2) / 2 <= pair) j++;
  return j;
}
template <int N>
__global__ void __launch_bounds__(128) k_scat_weights(double* __restrict__ tab, const int* __restrict__ need,
                                                      const int* __restrict__ ready, const double* lob_mu) {
  constexpr int C2 = scat_pairs(N);
  constexpr int NB = (C2 + 127) / 128;
  const int pi = blockIdx.x / NB;
  const int combo = (blockIdx.x % NB) * 128 + threadIdx.x;
  const int ni = nmu_index(N);
  if (pi >= SCAT_NPI || combo >= C2 || !need[ni * SCAT_NPI + pi] || ready[ni * SCAT_NPI + pi]) return;
  const int numpts = 2 * pi + 4, K = numpts / 2 + 1, nl = numpts - 3;
  const int j2 = scat_pair_row(combo), j1 = combo - j2 * (j2 + 1) / 2;
  const double mu1 = lob_mu[lob_off(N) + j1], mu2 = lob_mu[lob_off(N) + j2];
  const double st1 = sqrt(1. - mu1 * mu1), st2 = sqrt(1. - mu2 * mu2);
  const double sqm = sqrt((1. - mu1 * mu1) * (1. - mu2 * mu2));
  double* T = tab + scat_weight_offset(N, pi) + combo;
  for (int e = 0; e < nl * 5; e++) T[(size_t)e * C2] = 0.0;
  for (int k = 0; k < K; k++) {
    const double delphi = (TWO_PI * k) / numpts;
    const double cosphi = cos(delphi), sinphi = sin(delphi);
    const double cs = mu1 * mu2 + sqm * cosphi;
    const double ss = sqrt(fmax(0.0, 1. - cs * cs));
    double sin1, sin2, cos1, cos2;
    if (ss == 0.0) {
      sin1 = 0; sin2 = 0; cos1 = 1; cos2 = -1;
    } else {
      const double r = 1.0 / ss;
      sin1 = st2 * sinphi * r;
      sin2 = st1 * sinphi * r;
      cos1 = (st1 * mu2 - st2 * mu1 * cosphi) * r;
      cos2 = (st2 * mu1 - st1 * mu2 * cosphi) * r;
    }
    const double sin21 = 2.0 * sin1 * cos1, cos21 = 1.0 - 2.0 * (sin1 * sin1);
    const double sin22 = 2.0 * sin2 * cos2, cos22 = 1.0 - 2.0 * (sin2 * sin2);
    const double wk = (k > 0 && k < K - 1) ? 2.0 : 1.0;
    const double f[5] = {wk, wk * cos21, wk * cos22, wk * (cos21 * cos22), -wk * (sin21 * sin22)};
    double pl1 = 1.0, pl2 = 0.0;
    for (int l = 0; l < nl; l++) {
      double pl = 1.0;
      if (l > 0) {
        pl = fma(c_leg_a[l] * cs, pl1, -c_leg_b[l] * pl2);
        pl2 = pl1;
        pl1 = pl;
      }
      double* Tl = T + (size_t)l * 5 * C2;
#pragma unroll
      for (int e = 0; e < 5; e++) Tl[(size_t)e * C2] = fma(pl, f[e], Tl[(size_t)e * C2]);
    }
  }
  const double inv = 1.0 / numpts;
  for (int e = 0; e < nl * 5; e++) T[(size_t)e * C2] *= inv;
}

// Mark the numpts tables of N filled by k_scat_weights (run by one block of
// the kernel that follows it on the stream).  Without a table (its allocation
// failed) nothing was filled: a later call that gets one fills it.
template <int N>
__device__ __forceinline__ void scat_weights_mark_ready(const Work& w) {
  const int ni = nmu_index(N);
  if (blockIdx.x == 0 && w.wt_need && w.wtab[ni])
    for (int i = threadIdx.x; i < SCAT_NPI; i += blockDim.x)
      if (w.wt_need[ni * SCAT_NPI + i]) w.wt_ready[ni * SCAT_NPI + i] = 1;
}

// Per-item state of the layer stage after the thin-layer initialisation.
struct LayerItem {
  int c, z, fi, nd, status;
  double linfac;
};

// scatcnv, CHECK_NORM4, number of doublings, INITIALIZE4 and
// INITIAL_SOURCE4 of one (present layer, frequency) item: leaves the
// thin-layer R (S.m[0]) and T (S.m[1]) and the sources S.lin / S.cst in
// shared memory.  Returns false when the item is not for this N.
// Latency of one CTA, while its neighbours double: the table rows of several
// orders travel at once, the Planck functions run in the last warp beside the
// coefficients, norms eight lanes to a row.
// Layer stage, 1500 columns (N = 16) 22.0 -> 21.8 ms, mixed NUMMU 19.7 -> 19.4 (split
// form 14.2 -> 13.7), split form 13.0 -> 12.85: the set-up halved, but the doubling of the
// CTAs beside it takes up most of that.
template <int N, class SM, int T = RTCfg<N>::T>
__device__ __forceinline__ bool layer_setup(const Batch& b, const Work& w, const pamtra_b200_settings& st,
                                            double* __restrict__ ssp_scat, SM& S, int item,
                                            LayerItem& it) {
  constexpr int n = RTCfg<N>::n, LD = RTCfg<N>::LD, MAT = RTCfg<N>::MAT;
  static_assert(T == 8 * N, "eight threads per angle");
  const int t = threadIdx.x;
  const int Lm = b.max_nlyrs, Fm = b.max_nfreq;
    const int p = item / Fm, fi = item % Fm;
    const int cz = w.plist[p];
    const int c = cz / Lm, z = cz % Lm;
    if (fi >= b.col_nfreq(c) || b.col_nummu(c) != N) return false;
    const double freq = b.freq(c, fi);
    const double wl = C_LIGHT / (freq * 1.e3);
    const double* hl = w.hgt_lev + (size_t)c * (Lm + 1);
    const double* tl = w.temp_lev + (size_t)c * (Lm + 1);
    const double zdiff = fabs(hl[z + 1] - hl[z]);
    const double gas = fmax(w.kgas[((size_t)c * Fm + fi) * Lm + z], 0.0);
    // Planck functions at the layer's upper and lower boundary, for now in S.lin
    if (t >= T - 2) S.lin[T - 1 - t] = planck(tl[z + (T - 1 - t)], wl);
    const int nleg = w.m_nleg[item];
    const double kext = w.m_kext[item], salb = w.m_salb[item];
    double* Rb = S.mat(0);
    double* Tb = S.mat(1);
    double* Gb = S.mat(2);
    double* Yb = S.mat(4);
    double ext = 0.0, emis = 0.0;
    int status = 0;
    // ---------------- scatcnv (src/scatcnv.f90) into P1 (Tb) and P2 (Rb)
    if (nleg > 0) {
      ext = kext;
      emis = (1.0 - salb) * kext;
      const double cst = kext * salb / (4.0 * 3.1415926535897932384);
      const double* lg = w.m_legen ? w.m_legen + (size_t)item * 3 * MAXNLEG : nullptr;
      const float* lg32 = w.m_legen32 ? w.m_legen32 + (size_t)item * 3 * MAXNLEG : nullptr;
      double* coef = Gb;          // [3][MAXNLEG] (S.mat(2) provides that many; for n = 16 the next matrix)
      double* cphi = Yb;          // [KMAX]
      double* sphi = Yb + KMAX;   // [KMAX]
      const int numpts = 2 * ((nleg + 1) / 2) + 4;
      const int K = numpts / 2 + 1;
      for (int l = t; l <= nleg; l += T) {
#pragma unroll
        for (int k = 0; k < 3; k++)
          coef[k * MAXNLEG + l] = cst * (lg ? lg[k * MAXNLEG + l] : (double)lg32[k * MAXNLEG + l]);
      }
      const double* W = w.wtab[nmu_index(N)];
      if (W) {
        // phase matrices from the azimuth weight tables (k_scat_weights)
        team_sync();
        // thread per angle pair in rounds of T; a remainder of up to T / 16 pairs
        // takes sixteen threads each, over the orders
        constexpr int C2 = scat_pairs(N), REST = C2 % T;
        constexpr bool SPREAD = REST > 0 && REST * 16 <= T;
        constexpr int CPT = C2 / T + (REST > 0 && !SPREAD ? 1 : 0), LS = CPT > 1 ? 2 : 4;
        const double* Wp = W + scat_weight_offset(N, (numpts - 4) / 2);
        auto store = [&](int pair, const double (&ev)[5], const double (&od)[5]) {
          const int j2 = scat_pair_row(pair), j1 = pair - j2 * (j2 + 1) / 2;
#pragma unroll
          for (int q = 0; q < 2; q++) {
            double* Qm = (q == 0) ? Tb : Rb;
            double p[5];
#pragma unroll
            for (int e = 0; e < 5; e++) p[e] = q == 0 ? ev[e] + od[e] : ev[e] - od[e];
            const double p22 = q == 0 ? p[3] + p[4] : p[3] - p[4];
            const int a = 2 * j1, b2 = 2 * j2;
            Qm[a * LD + b2] = p[0];
            Qm[(a + 1) * LD + b2] = p[1];
            Qm[a * LD + b2 + 1] = p[2];
            Qm[(a + 1) * LD + b2 + 1] = p22;
            if (j1 != j2) {
              Qm[b2 * LD + a] = p[0];
              Qm[b2 * LD + a + 1] = p[1];
              Qm[(b2 + 1) * LD + a] = p[2];
              Qm[(b2 + 1) * LD + a + 1] = p22;
            }
          }
        };
        const int r = t & 15, rest = C2 - REST + min(t >> 4, REST - 1);
        double x[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
        if (SPREAD && r <= nleg) {
#pragma unroll
          for (int e = 0; e < 5; e++) x[e] = Wp[((size_t)r * 5 + e) * C2 + rest];
        }
        double acc[CPT > 0 ? CPT : 1][2][5];  // sums of the five weights over even and odd l
#pragma unroll
        for (int u = 0; u < CPT; u++)
#pragma unroll
          for (int e = 0; e < 10; e++) (&acc[u][0][0])[e] = 0.0;
        for (int l0 = 0; l0 <= nleg; l0 += LS) {
          double v[LS][CPT][5];
#pragma unroll
          for (int k = 0; k < LS; k++) {
            const double* Wl = Wp + (size_t)min(l0 + k, nleg) * 5 * C2;
#pragma unroll
            for (int u = 0; u < CPT; u++)
#pragma unroll
              for (int e = 0; e < 5; e++) v[k][u][e] = Wl[e * C2 + min(t + u * T, C2 - 1)];
          }
#pragma unroll
          for (int k = 0; k < LS; k++) {
            const int l = l0 + k;
            if (l > nleg) break;
            const double c0 = coef[l], c1 = coef[MAXNLEG + l], c2 = coef[2 * MAXNLEG + l];
#pragma unroll
            for (int u = 0; u < CPT; u++) {
              double(&a)[5] = acc[u][k & 1];
              a[0] = fma(c0, v[k][u][0], a[0]);
              a[1] = fma(c1, v[k][u][1], a[1]);
              a[2] = fma(c1, v[k][u][2], a[2]);
              a[3] = fma(c0, v[k][u][3], a[3]);
              a[4] = fma(c2, v[k][u][4], a[4]);
            }
          }
        }
#pragma unroll
        for (int u = 0; u < CPT; u++)
          if (t + u * T < C2) store(t + u * T, acc[u][0], acc[u][1]);
        if (SPREAD) {
          double sum[5] = {0.0, 0.0, 0.0, 0.0, 0.0}, other[5];
          for (int l = r; l <= nleg; l += 16) {
            if (l > r) {
#pragma unroll
              for (int e = 0; e < 5; e++) x[e] = Wp[((size_t)l * 5 + e) * C2 + rest];
            }
            const double c0 = coef[l], c1 = coef[MAXNLEG + l], c2 = coef[2 * MAXNLEG + l];
            sum[0] = fma(c0, x[0], sum[0]);
            sum[1] = fma(c1, x[1], sum[1]);
            sum[2] = fma(c1, x[2], sum[2]);
            sum[3] = fma(c0, x[3], sum[3]);
            sum[4] = fma(c2, x[4], sum[4]);
          }
#pragma unroll
          for (int e = 0; e < 5; e++) {
#pragma unroll
            for (int o = 2; o < 16; o <<= 1) sum[e] += __shfl_xor_sync(0xffffffffu, sum[e], o);
            other[e] = __shfl_xor_sync(0xffffffffu, sum[e], 1);
          }
          if (r == 0 && (t >> 4) < REST) store(rest, sum, other);
        }
      } else {
        for (int k = t; k < K; k += T) {
          const double delphi = (TWO_PI * k) / numpts;
          cphi[k] = cos(delphi);
          sphi[k] = sin(delphi);
        }
        team_sync();
        for (int it = t; it < 2 * N * N; it += T) {
          const int q = it / (N * N), j1 = (it / N) % N, j2 = it % N;
          const double mu1 = (q == 0) ? S.mu[j1] : -S.mu[j1];
          const double mu2 = S.mu[j2];
          const double st1 = sqrt(1. - mu1 * mu1), st2 = sqrt(1. - mu2 * mu2);
          const double sqm = sqrt((1. - mu1 * mu1) * (1. - mu2 * mu2));
          double a11 = 0, a12 = 0, a21 = 0, a22 = 0, m11 = 0, m12 = 0, m21 = 0, m22 = 0;
          for (int k = 0; k < K; k++) {
            const double cosphi = cphi[k], sinphi = sphi[k];
            const double cs = mu1 * mu2 + sqm * cosphi;
            // SUM_LEGENDRE, DOSUM = (1,1,1,0,0,0)
            double s0 = coef[0], s1 = coef[MAXNLEG], s2 = coef[2 * MAXNLEG];
            double pl1 = 1.0, pl2 = 0.0;
            for (int L = 1; L <= nleg; L++) {
              const double pl = fma(c_leg_a[L] * cs, pl1, -c_leg_b[L] * pl2);
              s0 = fma(coef[L], pl, s0);
              s1 = fma(coef[MAXNLEG + L], pl, s1);
              s2 = fma(coef[2 * MAXNLEG + L], pl, s2);
              pl2 = pl1;
              pl1 = pl;
            }
            // ROTATE_PHASE_MATRIX (NSTOKES=2)
            const double ss = sqrt(fmax(0.0, 1. - cs * cs));
            double sin1, sin2, cos1, cos2;
            if (ss == 0.0) {
              sin1 = 0; sin2 = 0; cos1 = 1; cos2 = -1;
            } else {
              const double r = 1.0 / ss;
              sin1 = st2 * sinphi * r;
              sin2 = st1 * sinphi * r;
              cos1 = (st1 * mu2 - st2 * mu1 * cosphi) * r;
              cos2 = (st2 * mu1 - st1 * mu2 * cosphi) * r;
            }
            const double sin21 = 2.0 * sin1 * cos1, cos21 = 1.0 - 2.0 * (sin1 * sin1);
            const double sin22 = 2.0 * sin2 * cos2, cos22 = 1.0 - 2.0 * (sin2 * sin2);
            const double e11 = s0, e12 = s1 * cos21, e21 = s1 * cos22, e22 = s0 * cos21 * cos22 - s2 * sin21 * sin22;
            // FOURIER_BASIS order 0: points k and numpts-k coincide (MATRIX_SYMMETRY)
            a11 += e11; a12 += e12; a21 += e21; a22 += e22;
            if (k > 0 && k < K - 1) { m11 += e11; m12 += e12; m21 += e21; m22 += e22; }
          }
          double* Q = (q == 0) ? Tb : Rb;
          const int row0 = 2 * j2, col0 = 2 * j1;
          Q[(col0 + 0) * LD + row0 + 0] = (a11 + m11) / numpts;
          Q[(col0 + 1) * LD + row0 + 0] = (a12 + m12) / numpts;
          Q[(col0 + 0) * LD + row0 + 1] = (a21 + m21) / numpts;
          Q[(col0 + 1) * LD + row0 + 1] = (a22 + m22) / numpts;
        }
      }
      team_sync();
      if (!st.lhyd_scattering) {
        for (int e = t; e < MAT; e += T) { Tb[e] = 0.0; Rb[e] = 0.0; }
        team_sync();
      }
      if (!st.lhyd_emission) emis = 0.0;
    } else {
      for (int e = t; e < MAT; e += T) { Tb[e] = 0.0; Rb[e] = 0.0; }
      team_sync();
    }
    // optional save_ssp output of the 4 quadrants (l=1,4 equal; l=2,3 equal)
    if (ssp_scat) {
      const int nn = 2 * b.max_nummu;
      const size_t o = (((size_t)c * Fm + fi) * Lm + z) * 4 * (size_t)nn * nn;
      for (int e = t; e < n * n; e += T) {
        const int row = e / n, col = e % n;
        const double p1 = Tb[col * LD + row], p2 = Rb[col * LD + row];
        ssp_scat[o + 0 * (size_t)nn * nn + (size_t)row * nn + col] = p1;
        ssp_scat[o + 1 * (size_t)nn * nn + (size_t)row * nn + col] = p2;
        ssp_scat[o + 2 * (size_t)nn * nn + (size_t)row * nn + col] = p2;
        ssp_scat[o + 3 * (size_t)nn * nn + (size_t)row * nn + col] = p1;
      }
    }
    const double planck0 = S.lin[1], planck1 = S.lin[0];
    // ---------------- number of doublings (src/radtran4.f90:319-329): INT(LOG(tau /
    // 1e-6) / LN2) + 1.  The logarithm in single precision is good to 1e-4 here; only
    // next to a whole number does the double-precision one decide.
    const double extinct = ext + gas;
    const double tau = fmax(extinct * zdiff, 1.0e-7);
    int nd = 0;
    {
      const float flf = log2f((float)(tau * 1.0e6));
      if (fabsf(flf - rintf(flf)) > 1.0e-3f && flf < 100.0f) {
        if (flf > 0.0f) nd = (int)flf + 1;
      } else {
        const double fl = log(tau / 1.0e-6) / LN2_F32;
        if (fl > 0.0) nd = (int)fl + 1;
      }
    }
    const double inv_sub = ldexp(1.0, -nd);
    const double delta_z = zdiff * inv_sub;
    // ---------------- CHECK_NORM4 (src/radscat4.f90:87-136), eight lanes per angle
    bool bad;
    {
      const int j = t >> 3;
      double sum = 0.0;
#pragma unroll
      for (int j2 = t & 7; j2 < N; j2 += 8)
        sum = sum + 2.0 * 3.1415926535897932384 * S.wq[j2] * (Tb[(2 * j) * LD + 2 * j2] + Rb[(2 * j) * LD + 2 * j2]);
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      bad = fabs(emis - ext + sum) > 5.0e-4;
      if ((t & 7) == 0) S.nrm[j] = delta_z / S.mu[j];
    }
    if (__syncthreads_or(bad)) status |= PAMTRA_B200_FATAL | PAMTRA_B200_ST_NORM;
    // ---------------- INITIALIZE4 (src/radintg4.f90:1-45), in place over P1/P2
    {
      const double C = 2.0 * 3.1415926535897932384;
#pragma unroll 4
      for (int e = t; e < n * n; e += T) {
        const int col = e / n, row = e % n;
        const int i1 = col & 1, j1 = col >> 1, i2 = row & 1, j2 = row >> 1;
        const double wj1 = S.wq[j1];
        const double tmp = S.nrm[j2];
        const double gext = (i1 == i2) ? gas : 0.0;
        const double diag = (row == col) ? 1.0 : 0.0;
        double ex = 0.0;
        if (j1 == j2) ex = ((i1 == i2) ? ext : 0.0) + gext;
        Rb[col * LD + row] = C * tmp * wj1 * Rb[col * LD + row];
        Tb[col * LD + row] = diag - tmp * (ex - C * wj1 * Tb[col * LD + row]);
      }
    }
    // INITIAL_SOURCE4 (src/radintg4.f90:51-73)
    if (t < n) {
      const int i = t & 1, jj = t >> 1;
      const double tmp = planck0 * delta_z / S.mu[jj];
      const double v = (i == 0) ? tmp * (emis + gas) : tmp * (0.0 + 0.0);
      S.lin[t] = v;
      S.lin[n + t] = v;
      S.cst[t] = v;
      S.cst[n + t] = v;
    }
    double linfac = (planck0 == 0.0) ? 0.0 : (planck1 / planck0 - 1.0) * inv_sub;
    team_sync();
  it.c = c;
  it.z = z;
  it.fi = fi;
  it.nd = nd;
  it.status = status;
  it.linfac = linfac;
  return true;
}

// Write the layer R, T and S+/S- of an item (FP64, unscaled, column-major with
// leading dimension n + 4: what k_adding<N, false> reads).
template <int N, int T = RTCfg<N>::T>
__device__ __forceinline__ void layer_store(const Work& w, int item, const double* Rb, const double* Tb,
                                            const double* lin) {
  constexpr int n = RTCfg<N>::n, MAT = RTCfg<N>::MAT;
  const int t = threadIdx.x;
  double* out = w.lay + (size_t)item * w.lay_stride;
  for (int e = t; e < MAT; e += T) { out[e] = Rb[e]; out[MAT + e] = Tb[e]; }
  for (int e = t; e < 2 * n; e += T) out[2 * MAT + e] = lin[e];
}

// DOUBLING_INTEGRATION4, SYMMETRIC (src/radintg4.f90:174-309):
//   R' = R + T G R T, T' = T G T with G = (I - R R)^-1,
// as X = R R, Y = R T, W = T G, then R' = R + W Y and T' = W T; the source
// chains use W u for T G u.  In the scaled form R, T, X, R' and T' are
// symmetric, so three of the five products compute NB (NB + 1) / 2 of NB^2
// tiles (10 of 16 for n = 32, 36 of 64 for n = 64).
// The sources: the constant parts C+ and C- start equal and stay so; the
// linear ones are S+- = (1 + a) C +- o, where the even part follows C (a grows by
// f / 2 per step) and the odd part obeys
//   o' = o + f C / 2 + W (I - R) e,  e = o - f C / 2,
// so two mat-vec pairs carry the four chains of the reference:
// C' = C + W (C + R C) and o'.  They take the fragments the passes hold anyway.
// Three barriers per step:
//   pass 1  X, Y^T = T R and the vectors C + R C, e - R e into shared memory;
//   pass 2  the warp's strip of W, in registers: W = T + T X + ..., one product
//           per term (W <- T + W X) with no barrier between them, since a strip
//           of W is the left factor of its own next term; for thick layers
//           W <- W + W X^(2^k) with X squared in place;
//   pass 3  R', T' and the sources from the W strip (left factor, still in
//           registers) with Y, T and those vectors, written after a barrier.
// The trace of X = R R bounds its norm (X is positive semidefinite) and is
// the sum of squares of R, known before X.
// What bounds it: the FP64 tensor pipe, 77 % busy (66 % with five full products
// in 16 x 16 tiles, 8-byte fragments and five barriers per step), then the
// data path of shared memory (58 %).  1500 columns x 50 layers x 4 frequencies, NUMMU 16:
// 30.6 -> 22.3 ms; 40 columns of mixed NUMMU: 27.3 -> 20.0 ms for the three kernels.
template <int N>
struct LayerCfg {
  static constexpr int n = 2 * N, T = SymTeam<n>::T;
  // resident CTAs the registers are bounded for.  N = 16: five (96 registers);
  // six would fit shared memory but spill more and measure the same (22.2 ms).
  static constexpr int CTAS = (N == 8) ? 8 : (N == 16) ? 5 : 1;
};

template <int N>
__global__ void __launch_bounds__(LayerCfg<N>::T, LayerCfg<N>::CTAS) k_layer(Batch b, Work w, pamtra_b200_settings st,
                                                                            double* __restrict__ ssp_scat) {
  using TM = SymTeam<2 * N>;
  constexpr int n = 2 * N, T = TM::T, NB = TM::NB, D = TM::D;
  constexpr int LD = RTCfg<N>::LD;  // leading dimension of layer_setup's matrices and the elimination
  extern __shared__ double smem_raw[];
  LayerSmem<N>& S = *reinterpret_cast<LayerSmem<N>*>(smem_raw);
  const int t = threadIdx.x, lane = t & 31, i = t >> 5;  // i: this warp's strip
  const int g = lane >> 2, q = lane & 3;
  const bool low = i < D;
  const int Fm = b.max_nfreq;
  const int P = min(w.counters[0], w.pmax);
  const int nitems = P * Fm;
  scat_weights_mark_ready<N>(w);
  if (t < N) { S.mu[t] = w.lob_mu[lob_off(N) + t]; S.wq[t] = w.lob_w[lob_off(N) + t]; }
  if (t < n) {
    const double v = sqrt(w.lob_mu[lob_off(N) + (t >> 1)] * w.lob_w[lob_off(N) + (t >> 1)]);
    S.sc[t] = v;
    S.is[t] = 1.0 / v;
  }
  double *const R = S.m, *const Tm = S.m + TM::MAT, *const X = S.m + 2 * TM::MAT, *const Y = S.m + 3 * TM::MAT;
  for (;;) {
    team_sync();
    if (t == 0) S.item = atomicAdd(&w.counters[2 + (N == 8 ? 0 : (N == 16 ? 1 : 2))], 1);
    team_sync();
    const int item = S.item;
    if (item >= nitems) break;
    LayerItem it;
    if (!layer_setup<N, LayerSmem<N>, T>(b, w, st, ssp_scat, S, item, it)) continue;
    const int nd = it.nd, c = it.c, fi = it.fi;
    int status = it.status;
    double f = it.linfac;
    // scaled, symmetric R and T from the set-up's layout (through registers:
    // the two layouts overlap); scaled sources
    double fro = 0.0;
    {
      constexpr int E = (n * n + T - 1) / T;
      double r[E], v[E];
#pragma unroll
      for (int k = 0; k < E; k++) {
        const int e = t + k * T, col = e / n, row = e % n;
        // exactly 1 on the diagonal: T is near the identity, whose rounding counts most
        const double s1 = (row == col) ? 1.0 : S.sc[row] * S.is[col], s2 = (row == col) ? 1.0 : S.sc[col] * S.is[row];
        const double *Rs = S.mat(0), *Ts = S.mat(1);
        r[k] = 0.5 * (Rs[col * LD + row] * s1 + Rs[row * LD + col] * s2);
        v[k] = 0.5 * (Ts[col * LD + row] * s1 + Ts[row * LD + col] * s2);
        fro += r[k] * r[k];
      }
      team_sync();
#pragma unroll
      for (int k = 0; k < E; k++) {
        const int e = t + k * T, col = e / n, row = e % n;
        R[TM::at(row, col)] = r[k];
        Tm[TM::at(row, col)] = v[k];
      }
    }
    fro = warp_sum(fro);
    if (lane == 0) S.fro[i] = fro;
    double even = 1.0;  // 1 + a
    if (t < n) {  // INITIAL_SOURCE4 leaves all four sources equal
      const double c0 = S.cst[t] * S.sc[t];
      S.C[t] = c0;
      S.o[t] = 0.0;
      S.E[t] = -(0.5 * f) * c0;
    }
    int tiles = 0;  // 8 x 8 tiles of products issued for this item (counted by thread 0)
    const int row = 8 * i + g;
    for (int itd = 0; itd < nd; itd++) {
      team_sync();
      double nrm = 0.0;  // trace of X
#pragma unroll
      for (int k = 0; k < NB; k++) nrm += S.fro[k];
      // ---- pass 1
      {
        double x[D + 1][2], y[NB][2], zc = 0.0, ze = 0.0;
#pragma unroll
        for (int e = 0; e < 2; e++) {
#pragma unroll
          for (int d = 0; d <= D; d++) x[d][e] = 0.0;
#pragma unroll
          for (int d = 0; d < NB; d++) y[d][e] = 0.0;
        }
#pragma unroll 2
        for (int u = 0; u < NB; u++) {
          const double2 a = TM::ld(R, i, u), at = TM::ld(Tm, i, u);
#pragma unroll
          for (int d = 0; d < NB; d++) {
            const double2 bb = (d == 0) ? a : TM::ld(R, TM::blk(i, d), u);
            if (d < D || (d == D && low)) {
              dmma(x[d < D ? d : D], a.x, bb.x);
              dmma(x[d < D ? d : D], a.y, bb.y);
            }
            dmma(y[d], at.x, bb.x);
            dmma(y[d], at.y, bb.y);
          }
          const double2 vc = *reinterpret_cast<const double2*>(S.C + 8 * u + 2 * q);
          const double2 ve = *reinterpret_cast<const double2*>(S.E + 8 * u + 2 * q);
          zc = fma(a.y, vc.y, fma(a.x, vc.x, zc));
          ze = fma(a.y, ve.y, fma(a.x, ve.x, ze));
        }
#pragma unroll
        for (int d = 0; d < D; d++) TM::st_sym(X, i, TM::blk(i, d), x[d]);
        if (low) TM::st_sym(X, i, TM::blk(i, D), x[D]);
#pragma unroll
        for (int d = 0; d < NB; d++) TM::st(Y, i, TM::blk(i, d), y[d]);
        zc = quad_sum(zc);
        ze = quad_sum(ze);
        if (q == 0) S.UC[row] = S.C[row] + zc;
        else if (q == 1) S.UE[row] = S.E[row] - ze;
      }
      team_sync();
      // ---- pass 2
      double W[NB][2];
#pragma unroll
      for (int u = 0; u < NB; u++) {
        const double2 a = TM::ld(Tm, i, u);
        W[u][0] = a.x;
        W[u][1] = a.y;
      }
      // W <- (T or W) + W X
      auto term = [&](bool add_t) {
        double h[NB][2];
#pragma unroll
        for (int j = 0; j < NB; j++) {
          h[j][0] = W[j][0];
          h[j][1] = W[j][1];
          if (add_t) {
            const double2 a = TM::ld(Tm, i, j);
            h[j][0] = a.x;
            h[j][1] = a.y;
          }
        }
#pragma unroll
        for (int u = 0; u < NB; u++)
#pragma unroll
          for (int j = 0; j < NB; j++) {
            const double2 bb = TM::ld(X, j, u);
            dmma(h[j], W[u][0], bb.x);
            dmma(h[j], W[u][1], bb.y);
          }
#pragma unroll
        for (int j = 0; j < NB; j++) { W[j][0] = h[j][0]; W[j][1] = h[j][1]; }
      };
      int kh = 0, m = 1;
      if (nrm * nrm > 5.0e-17) {
        if (nrm > 0.5) {
          // the trace is a loose bound for thick layers: the row-sum norm of
          // the unscaled X decides between the series and the elimination
          if (t < n) {
            double r = 0.0;
            for (int j = 0; j < n; j++) r += fabs(X[TM::at(j, t)]) * S.sc[j];
            r *= S.is[t];
            const unsigned mask = (n >= 32) ? 0xffffffffu : ((1u << n) - 1u);
#pragma unroll
            for (int o = ((n >= 32) ? 16 : n / 2); o > 0; o >>= 1) r = fmax(r, __shfl_xor_sync(mask, r, o));
            if ((t & 31) == 0) S.inv.cand_v[t >> 5] = r;
          }
          team_sync();
          double rs = S.inv.cand_v[0];
#pragma unroll
          for (int k = 1; k < (n + 31) / 32; k++) rs = fmax(rs, S.inv.cand_v[k]);
          nrm = fmin(nrm, rs);
        }
        // further terms: kh by Horner (remainder nrm^(kh + 2) below 5e-17) or m - 1 squarings
        // (remainder nrm^(2^m), m the first with nrm^(2^(m-1)) below 5e-17: one factor to spare)
        for (double pw = nrm; pw > 5.0e-17 && m < 8; m++) pw = pw * pw;
        for (double ph = nrm * nrm; ph > 5.0e-17 && kh < 2 * (m - 1); kh++) ph = ph * nrm;
      }
      if (m >= 8) {
        // Gauss-Jordan on I - X in the column-major layout, over X and Y (Y waits in registers)
        constexpr int E = n * n / T;
        double x[E], y[E];
#pragma unroll
        for (int k = 0; k < E; k++) {
          const int e = t + k * T, col = e / n, r = e % n;
          x[k] = ((r == col) ? 1.0 : 0.0) - X[TM::at(r, col)];
          y[k] = Y[e];
        }
        team_sync();
#pragma unroll
        for (int k = 0; k < E; k++) { const int e = t + k * T; X[(e / n) * LD + e % n] = x[k]; }
        team_sync();
        if (ginv<n, T>(X, S.inv)) status |= PAMTRA_B200_FATAL | PAMTRA_B200_ST_PIVOT;
#pragma unroll
        for (int k = 0; k < E; k++) {  // G - I
          const int e = t + k * T, col = e / n, r = e % n;
          x[k] = X[col * LD + r] - ((r == col) ? 1.0 : 0.0);
        }
        team_sync();
#pragma unroll
        for (int k = 0; k < E; k++) {
          const int e = t + k * T;
          X[TM::at(e % n, e / n)] = x[k];
          Y[e] = y[k];
        }
        team_sync();
        term(false);  // W = T + T (G - I)
        tiles += 2 * NB * NB;
      } else if (kh <= 7 * (m - 1) / 4) {
        term(false);
        for (int k = 0; k < kh; k++) term(true);
        tiles += (kh + 1) * NB * NB;
      } else {
        // W = T (I + X)(I + X^2)(I + X^4)..., m factors (the remainder would allow m - 1)
        term(false);
        for (int k = 1; k < m; k++) {
          double x[D + 1][2];
#pragma unroll
          for (int d = 0; d <= D; d++) x[d][0] = x[d][1] = 0.0;
          for (int u = 0; u < NB; u++) {
            const double2 a = TM::ld(X, i, u);
#pragma unroll
            for (int d = 0; d <= D; d++)
              if (d < D || low) {
                const double2 bb = (d == 0) ? a : TM::ld(X, TM::blk(i, d), u);
                dmma(x[d], a.x, bb.x);
                dmma(x[d], a.y, bb.y);
              }
          }
          team_sync();
#pragma unroll
          for (int d = 0; d < D; d++) TM::st_sym(X, i, TM::blk(i, d), x[d]);
          if (low) TM::st_sym(X, i, TM::blk(i, D), x[D]);
          team_sync();
          term(false);
        }
        tiles += m * NB * NB + (m - 1) * (NB * (NB + 1) / 2);
      }
      // ---- pass 3
      {
        double r[D][2], v[D][2], x[2], zc = 0.0, ze = 0.0;
        // the extra tile: of R' for the low strips, of T' for the others
        const int jx = TM::blk(i, D);
        const double* const Bx = low ? Y : Tm;
#pragma unroll
        for (int d = 0; d < D; d++) {
          const double2 a = TM::ld(R, i, TM::blk(i, d));
          r[d][0] = a.x;
          r[d][1] = a.y;
          v[d][0] = v[d][1] = 0.0;
        }
        x[0] = x[1] = 0.0;
        if (low) {
          const double2 a = TM::ld(R, i, jx);
          x[0] = a.x;
          x[1] = a.y;
        }
#pragma unroll
        for (int u = 0; u < NB; u++) {
#pragma unroll
          for (int d = 0; d < D; d++) {
            const double2 by = TM::ld(Y, TM::blk(i, d), u), bt = TM::ld(Tm, TM::blk(i, d), u);
            dmma(r[d], W[u][0], by.x);
            dmma(v[d], W[u][0], bt.x);
            dmma(r[d], W[u][1], by.y);
            dmma(v[d], W[u][1], bt.y);
          }
          const double2 bx = TM::ld(Bx, jx, u);
          dmma(x, W[u][0], bx.x);
          dmma(x, W[u][1], bx.y);
          const double2 vc = *reinterpret_cast<const double2*>(S.UC + 8 * u + 2 * q);
          const double2 ve = *reinterpret_cast<const double2*>(S.UE + 8 * u + 2 * q);
          zc = fma(W[u][1], vc.y, fma(W[u][0], vc.x, zc));
          ze = fma(W[u][1], ve.y, fma(W[u][0], ve.x, ze));
        }
        zc = quad_sum(zc);
        ze = quad_sum(ze);
        team_sync();
        fro = 0.0;
#pragma unroll
        for (int d = 0; d < D; d++) {
          TM::st_sym(R, i, TM::blk(i, d), r[d]);
          TM::st_sym(Tm, i, TM::blk(i, d), v[d]);
          fro += (d == 0 ? 1.0 : 2.0) * (r[d][0] * r[d][0] + r[d][1] * r[d][1]);
        }
        TM::st_sym(low ? R : Tm, i, jx, x);
        if (low) fro += 2.0 * (x[0] * x[0] + x[1] * x[1]);
        if (q == 0) {
          const double cc = S.C[row], cn = cc + zc, on = S.o[row] + (0.5 * f) * cc + ze;
          S.C[row] = cn;
          S.o[row] = on;
          S.E[row] = on - f * cn;  // the next step's f is twice this one's
        }
        fro = warp_sum(fro);
        if (lane == 0) S.fro[i] = fro;
      }
      tiles += 3 * (NB * (NB + 1) / 2) + NB * NB;
      even = even + 0.5 * f;
      f = 2.0 * f;
    }
    team_sync();
    // the layer record k_adding<N, true> reads: the scaled R and T as they lie, S+ and S-
    {
      double* out = w.lay + (size_t)item * w.lay_stride;
      const double2 *r2 = reinterpret_cast<const double2*>(R), *t2 = reinterpret_cast<const double2*>(Tm);
      double2* o2 = reinterpret_cast<double2*>(out);
      for (int e = t; e < n * n / 2; e += T) {
        o2[e] = r2[e];
        o2[n * n / 2 + e] = t2[e];
      }
      for (int e = t; e < n; e += T) {
        const double m = even * S.C[e], o = S.o[e];
        out[2 * n * n + e] = m + o;
        out[2 * n * n + n + e] = m - o;
      }
    }
    if (t == 0) {
      w.lay_nd[item] = nd;
      if (status) atomicOr(&w.status[(size_t)c * Fm + fi], status);
      // products of n x n matrices by the multiply-adds issued (a symmetric one counts its computed tiles)
      const int nprod = (tiles + NB * NB / 2) / (NB * NB);
      if (nprod) atomicAdd(reinterpret_cast<unsigned long long*>(w.counters + COUNTER_PRODUCTS),
                           (unsigned long long)nprod);
    }
  }
}

}  // namespace pb
