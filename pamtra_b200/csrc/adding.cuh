// k_adding<N, SYM>: adding of all layers of a (column, frequency) unit from the
// top down (COMBINE_LAYERS4, src/radintg4.f90:447-513), the surface, the
// radiances at the output levels and their conversion to brightness
// temperature.  With Gp = (I - R1p R2m)^-1 the combine of a stack 1 on top of
// a stack or layer 2 takes one inverse,
//   R+' = R2p + A R1p T2m,  T+' = A T1p,             A = T2p Gp
//   R-' = R1m + B T1p,      T-' = (T1m + B R1p) T2m, B = T1m R2m Gp
//   S+' = S2+ + A (S1+ + R1p S2-)
//   S-' = S1- + T1m w + B (R1p w),  w = S2- + R2m S1+
// since Gm = (I - R2m R1p)^-1 = I + R2m Gp R1p.
//
// SYM: layers of k_layer, in its scaled symmetric form (see there).  Then
// R+ and R- are symmetric and T- = T+^T for any stack: T- is not formed, and
// R+', R-' compute their upper tiles only.  Otherwise (layers of the
// split-precision doubling, symmetric to FP32 rounding only): unscaled and in full.
//
// Layout and roles are those of SymTeam: n / 8 warps, warp i owns the strip of
// rows 8i .. 8i + 7 of every result; the strip of a product is the left factor
// of the next without an exchange, and R- (and T-), which their owner alone reads,
// have no place in shared memory.  That holds the registers full: 128 at four CTAs per
// SM for n = 32, 255 for n = 64, and the rest spills to local memory (bytes of
// stores / loads per thread: <16, true> 390 / 432, <16, false> 634 / 608, <32, true>
// 946 / 984, <32, false> 2222 / 2236; NUMMU 8 none).  Shared memory holds R+, T+,
// the layer's R and T and two work matrices (R1p R2m and its powers): 49 KB
// for n = 32; n = 64 fits without the global scratch it took.
//
// A unit's layers go in segments of about sqrt(M) of its M scattering layers
// (adding is associative), each a work item of its own; the CTA that finishes
// a unit's last segment combines the segments and ends the unit.  The work is
// the same, and a column's chain of M dependent combines becomes one of about
// 2 sqrt(M).  Segments follow from the column alone, so results do not
// depend on the batch.  What bounds it: the chain of dependent products of a
// combine at 16 warps per SM (8 for n = 64): FP64 tensor pipe 48 %, 65 % for n = 64, with
// the barriers and spills between.  Adding stage, before (one chain per unit,
// twelve or ten full products, two CTAs per SM) and now: one column 0.43 ->
// 0.16 ms, 1500 columns x 50 layers x 4 frequencies 6.4 -> 4.4 ms (three
// CTAs per SM 4.6), 64 columns of 150 layers 1.65 -> 1.02 ms, 40 columns of
// mixed NUMMU 11.3 -> 4.4 ms, with the split doubling 11.6 -> 6.4 ms.
#pragma once
#include "common.cuh"
#include "work.cuh"
#include "rt.cuh"

namespace pb {

// Segments of a unit with M scattering layers, of about max(4, sqrt(M)) layers each
// and at least three (M = 9: 3, 3, 3); a segment's stack needs the first two of its
// layer records.
__host__ __device__ __forceinline__ int add_segments(int M) {
  if (M < 8) return 1;
  int len = 4;
  while (len * len < M) len++;
  return (M + len - 1) / len;
}
// most segments of any unit of at most L layers
inline int add_max_segments(int L) {
  int m = 1;
  for (int M = 8; M <= L; M++) m = m > add_segments(M) ? m : add_segments(M);
  return m;
}

template <int N>
struct AddSmem {
  static constexpr int n = 2 * N;
  alignas(16) double m[6][n * n];  // R+, T+, R and T of the layer, two work matrices
  alignas(16) double sp[n], sm[n], s2p[n], s2m[n], wp[n], wm[n], v[n], cm[n], cp[n], sky[n], gnd[n], dn[n], up[n];
  double tc[n], upt[n];
  double sc[n], is[n], mu[N], wq[N], nw[n / 8];
  InvScratch<n> inv;
  int unit, last;
};

// Register-resident parts of a stack: this warp's strip of R- and T-.
template <int N, bool SYM>
struct AddRegs {
  static constexpr int NB = SymTeam<2 * N>::NB, D = SymTeam<2 * N>::D;
  double rm[SYM ? D + 1 : NB][2];  // SYM: tiles (i, i + d), d = 0 .. D (the last for i < D)
  double tm[SYM ? 1 : NB][2];
};

template <int N, bool SYM>
struct Adder {
  using TM = SymTeam<2 * N>;
  using SM = AddSmem<N>;
  using RG = AddRegs<N, SYM>;
  static constexpr int n = 2 * N, T = TM::T, NB = TM::NB, D = TM::D, LD = n + 4;
  static constexpr int RECORD_BYTES = 8 * (SYM ? 2 * n * n + 2 * n : 2 * n * LD + 2 * n);

  // left-factor fragment of rows 8i + g of a general matrix held column-major
  __device__ static __forceinline__ double2 ldrow(const double* M, int i, int u) {
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    return make_double2(M[TM::at(8 * i + g, 8 * u + 2 * q)], M[TM::at(8 * i + g, 8 * u + 2 * q + 1)]);
  }
  // ... of a matrix that is symmetric in the SYM form
  __device__ static __forceinline__ double2 ldsym(const double* M, int i, int u) {
    return SYM ? TM::ld(M, i, u) : ldrow(M, i, u);
  }
  __device__ static __forceinline__ void strow(double* M, int i, int j, const double (&c)[2]) {
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    M[TM::at(8 * i + g, 8 * j + 2 * q)] = c[0];
    M[TM::at(8 * i + g, 8 * j + 2 * q + 1)] = c[1];
  }
  __device__ static __forceinline__ double2 vec(const double* x, int u) {
    return *reinterpret_cast<const double2*>(x + 8 * u + 2 * (threadIdx.x & 3));
  }
  // c (+)= strip a times B, all column blocks (c starts at `init`, null: zero)
  __device__ static __forceinline__ void mul(const double (&a)[NB][2], const double* B, double (&c)[NB][2],
                                             const double (*init)[2]) {
#pragma unroll
    for (int j = 0; j < NB; j++) {
      c[j][0] = init ? init[j][0] : 0.0;
      c[j][1] = init ? init[j][1] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < NB; u++)
#pragma unroll
      for (int j = 0; j < NB; j++) {
        const double2 bb = TM::ld(B, j, u);
        dmma(c[j], a[u][0], bb.x);
        dmma(c[j], a[u][1], bb.y);
      }
  }
  // this warp's tiles of a result of kind R (symmetric in the SYM form): c += strip a times B
  template <int NT>
  __device__ static __forceinline__ void mulsym(const double (&a)[NB][2], const double* B, double (&c)[NT][2], int i) {
#pragma unroll
    for (int u = 0; u < NB; u++)
#pragma unroll
      for (int d = 0; d < NT; d++) {
        if (SYM && d == D && i >= D) continue;
        const double2 bb = TM::ld(B, SYM ? TM::blk(i, d) : d, u);
        dmma(c[d], a[u][0], bb.x);
        dmma(c[d], a[u][1], bb.y);
      }
  }
  // store this warp's tiles of a result of kind R
  template <int NT>
  __device__ static __forceinline__ void stres(double* M, const double (&c)[NT][2], int i) {
#pragma unroll
    for (int d = 0; d < NT; d++) {
      if (SYM) {
        if (d < D || i < D) TM::st_sym(M, i, TM::blk(i, d), c[d]);
      } else {
        strow(M, i, d, c[d]);
      }
    }
  }
  // row 8i + g of strip a times x, in every lane of the quad
  __device__ static __forceinline__ double mv(const double (&a)[NB][2], const double* x) {
    double s = 0.0;
#pragma unroll
    for (int u = 0; u < NB; u++) {
      const double2 v = vec(x, u);
      s = fma(a[u][1], v.y, fma(a[u][0], v.x, s));
    }
    return quad_sum(s);
  }
  __device__ static __forceinline__ double mvsym(const double* M, int i, const double* x) {
    double s = 0.0;
#pragma unroll 4
    for (int u = 0; u < NB; u++) {
      const double2 a = ldsym(M, i, u), v = vec(x, u);
      s = fma(a.y, v.y, fma(a.x, v.x, s));
    }
    return quad_sum(s);
  }
  // T- times x
  __device__ static __forceinline__ double mvtm(const SM& S, const RG& G, int i, const double* x) {
    if constexpr (SYM) {
      double s = 0.0;
#pragma unroll 4
      for (int u = 0; u < NB; u++) {
        const double2 a = TM::ld(S.m[1], i, u), v = vec(x, u);
        s = fma(a.y, v.y, fma(a.x, v.x, s));
      }
      return quad_sum(s);
    } else {
      return mv(G.tm, x);
    }
  }

  // H = (I - X)^-1 - I for X = R1p R2m in S.m[4] (SYM: X as the right factor
  // there and X^T in S.m[5]), `x` this warp's strip of X (SYM: of X^T), nrm a
  // norm of X: returns the matrix holding H as a right factor.  Series of degree d
  // with remainder nrm^(d + 1) below FP64 rounding: d = 1 is X itself; up to
  // 3 by Horner, up to 17 by Horner in X^3 over I + X + X^2 (2 + j products
  // for degree 2 + 3j, against d - 1 by plain Horner), then by squaring, all
  // on the strip (in the SYM form on that of the transposed matrices) with a
  // barrier only where a new power is shared; from 0.556 on by elimination.
  __device__ static __forceinline__ double* series(SM& S, double (&x)[NB][2], double nrm, int i, int& status) {
    const int t = threadIdx.x;
    int deg = 1;
    for (double p = nrm * nrm; p > 5.0e-17 && deg < 64; deg++) p = p * nrm;
    if (deg == 1) return S.m[4];
    double *P = SYM ? S.m[5] : S.m[4], *Q = SYM ? S.m[4] : S.m[5];  // powers to multiply with, and the other
    double h[NB][2];
    if (deg >= 64) {
      double* const M = S.m[4];  // column-major, leading dimension n + 4, over both work matrices
      team_sync();
#pragma unroll
      for (int j = 0; j < NB; j++)
#pragma unroll
        for (int e = 0; e < 2; e++) {
          const int r = 8 * i + ((t & 31) >> 2), c = 8 * j + 2 * (t & 3) + e;
          M[SYM ? r * LD + c : c * LD + r] = ((r == c) ? 1.0 : 0.0) - x[j][e];
        }
      team_sync();
      if (ginv<n, T>(M, S.inv)) status |= PAMTRA_B200_FATAL | PAMTRA_B200_ST_PIVOT;
#pragma unroll
      for (int j = 0; j < NB; j++)
#pragma unroll
        for (int e = 0; e < 2; e++) {
          const int r = 8 * i + ((t & 31) >> 2), c = 8 * j + 2 * (t & 3) + e;
          h[j][e] = M[SYM ? r * LD + c : c * LD + r] - ((r == c) ? 1.0 : 0.0);
        }
      team_sync();
    } else if (deg <= 3) {
      mul(x, P, h, x);  // X + X X
      if (deg == 3) {
        double k[NB][2];
        mul(h, P, k, x);  // X + (X + X X) X
#pragma unroll
        for (int j = 0; j < NB; j++) { h[j][0] = k[j][0]; h[j][1] = k[j][1]; }
      }
    } else if (deg <= 17) {
      double y[NB][2], z[NB][2];
      mul(x, P, y, nullptr);  // X^2
      mul(y, P, z, nullptr);  // X^3
#pragma unroll
      for (int j = 0; j < NB; j++) { strow(Q, i, j, z[j]); x[j][0] += y[j][0]; x[j][1] += y[j][1]; }  // x = X + X^2
      team_sync();
      { double* s = P; P = Q; Q = s; }
      // F = I + H: F <- (I + X + X^2) + F X^3, first H = x + X^3 + x X^3
#pragma unroll
      for (int j = 0; j < NB; j++) { y[j][0] = x[j][0] + z[j][0]; y[j][1] = x[j][1] + z[j][1]; }
      mul(x, P, h, y);
      for (int d = 5; d < deg; d += 3) {
        mul(h, P, z, y);
#pragma unroll
        for (int j = 0; j < NB; j++) { h[j][0] = z[j][0]; h[j][1] = z[j][1]; }
      }
    } else {
      // (I + X)(I + X^2)(I + X^4)...: H <- (H + X^(2^k)) + H X^(2^k)
#pragma unroll
      for (int j = 0; j < NB; j++) { h[j][0] = x[j][0]; h[j][1] = x[j][1]; }
      for (int d = 1; d < deg; d = 2 * d + 1) {
        double y[NB][2], z[NB][2];
        mul(x, P, y, nullptr);
#pragma unroll
        for (int j = 0; j < NB; j++) {
          strow(Q, i, j, y[j]);
          x[j][0] = y[j][0];
          x[j][1] = y[j][1];
          y[j][0] += h[j][0];
          y[j][1] += h[j][1];
        }
        team_sync();
        { double* s = P; P = Q; Q = s; }
        mul(h, P, z, y);
#pragma unroll
        for (int j = 0; j < NB; j++) { h[j][0] = z[j][0]; h[j][1] = z[j][1]; }
      }
    }
    // Q was last read before a barrier all warps have passed
#pragma unroll
    for (int j = 0; j < NB; j++) {
      if (SYM) TM::st(Q, i, j, h[j]);
      else strow(Q, i, j, h[j]);
    }
    return Q;
  }

  // Stack (R+ S.m[0], T+ S.m[1], S.sp, S.sm, G) on top of R2m S.m[2], T2m
  // S.m[3], sources S.s2p / S.s2m; a layer (rec0 null) has R2p = R2m, T2p = T2m,
  // a segment its own in rec0.  Complete before the call.  Ends with a
  // barrier after the last read of the second operand and writes the stack; the
  // caller synchronises before the next read.
  __device__ static __forceinline__ void combine(SM& S, RG& G, const double* rec0, int i, int& status) {
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3, row = 8 * i + g;
    double *Rp = S.m[0], *Tp = S.m[1], *R2 = S.m[2], *T2 = S.m[3];
    double x[NB][2];
    // ---- X = R1p R2m (SYM: X^T = R2m R1p), w+ = S1+ + R1p S2-, w = S2- + R2m S1+
    {
      double zp = 0.0, zm = 0.0, rs = 0.0;
#pragma unroll
      for (int j = 0; j < NB; j++) x[j][0] = x[j][1] = 0.0;
      const double *L = SYM ? R2 : Rp, *B = SYM ? Rp : R2;
#pragma unroll 2
      for (int u = 0; u < NB; u++) {
        const double2 a = ldsym(L, i, u), o = ldsym(B, i, u);
#pragma unroll
        for (int j = 0; j < NB; j++) {
          const double2 bb = TM::ld(B, j, u);
          dmma(x[j], a.x, bb.x);
          dmma(x[j], a.y, bb.y);
        }
        const double2 r1 = SYM ? o : a, r2 = SYM ? a : o, vm = vec(S.s2m, u), vp = vec(S.sp, u);
        zp = fma(r1.y, vm.y, fma(r1.x, vm.x, zp));
        zm = fma(r2.y, vp.y, fma(r2.x, vp.x, zm));
      }
      // row-sum norm in the unscaled (flux) weights
#pragma unroll
      for (int j = 0; j < NB; j++) {
        rs += fabs(x[j][0]) * S.sc[8 * j + 2 * q] + fabs(x[j][1]) * S.sc[8 * j + 2 * q + 1];
        if (SYM) {
          TM::st(S.m[4], i, j, x[j]);
          strow(S.m[5], i, j, x[j]);
        } else {
          strow(S.m[4], i, j, x[j]);
        }
      }
      rs = quad_sum(rs) * S.is[row];
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) rs = fmax(rs, __shfl_xor_sync(0xffffffffu, rs, o));
      if (lane == 0) S.nw[i] = rs;
      zp = quad_sum(zp);
      zm = quad_sum(zm);
      if (q == 0) {
        S.wp[row] = S.sp[row] + zp;
        S.wm[row] = S.s2m[row] + zm;
      }
    }
    team_sync();
    double nrm = S.nw[0];
#pragma unroll
    for (int k = 1; k < NB; k++) nrm = fmax(nrm, S.nw[k]);
    {
      const double z = mvsym(Rp, i, S.wm);  // R1p w
      if (q == 0) S.v[row] = z;
    }
    const double* const H = series(S, x, nrm, i, status);
    team_sync();
    // ---- A = T2p G and what it gives
    double tp[NB][2], rp[SYM ? D + 1 : NB][2], sp, sm;
    {
      double a[NB][2], ta[NB][2];
#pragma unroll
      for (int u = 0; u < NB; u++) {  // T2p
        double2 f;
        if (SYM) f = TM::ld(T2, i, u);  // row of T2p = column of T2m
        else if (!rec0) f = ldrow(T2, i, u);
        else f = make_double2(__ldcg(rec0 + n * n + TM::at(row, 8 * u + 2 * q)), __ldcg(rec0 + n * n + TM::at(row, 8 * u + 2 * q + 1)));
        ta[u][0] = f.x;
        ta[u][1] = f.y;
      }
      mul(ta, H, a, ta);
      sp = S.s2p[row] + mv(a, S.wp);
      mul(a, Tp, tp, nullptr);
      double ar[NB][2];
      mul(a, Rp, ar, nullptr);
#pragma unroll
      for (int d = 0; d < (SYM ? D + 1 : NB); d++) {  // R2p
        const int j = SYM ? TM::blk(i, d) : d;
        double2 f;
        if (!rec0) f = ldsym(R2, i, j);
        else f = make_double2(__ldcg(rec0 + TM::at(row, 8 * j + 2 * q)), __ldcg(rec0 + TM::at(row, 8 * j + 2 * q + 1)));
        rp[d][0] = f.x;
        rp[d][1] = f.y;
      }
      mulsym(ar, T2, rp, i);
    }
    // ---- B = T1m R2m G and what it gives
    {
      double b0[NB][2], bb[NB][2];
      if constexpr (SYM) {
        double a[NB][2];
#pragma unroll
        for (int u = 0; u < NB; u++) {
          const double2 f = TM::ld(Tp, i, u);
          a[u][0] = f.x;
          a[u][1] = f.y;
        }
        sm = S.sm[row] + mv(a, S.wm);
        mul(a, R2, b0, nullptr);
      } else {
        sm = S.sm[row] + mv(G.tm, S.wm);
        mul(G.tm, R2, b0, nullptr);
      }
      mul(b0, H, bb, b0);
      sm = sm + mv(bb, S.v);
      mulsym(bb, Tp, G.rm, i);
      if constexpr (!SYM) {
        double c1[NB][2];
        mul(bb, Rp, c1, G.tm);
        mul(c1, T2, G.tm, nullptr);
      }
    }
    team_sync();
    stres(Rp, rp, i);
#pragma unroll
    for (int j = 0; j < NB; j++) strow(Tp, i, j, tp[j]);
    if (q == 0) {
      S.sp[row] = sp;
      S.sm[row] = sm;
    }
  }

  // Layer record -> S.m[2], S.m[3], S.s2p, S.s2m.  SYM: the scaled swizzled images k_layer writes.
  __device__ static __forceinline__ void load_layer(SM& S, const double* src) {
    const int t = threadIdx.x;
    if (SYM) {
      const double2* s = reinterpret_cast<const double2*>(src);
      double2* d = reinterpret_cast<double2*>(S.m[2]);
#pragma unroll 8
      for (int e = t; e < n * n; e += T) d[e] = s[e];  // R and T: 2 n^2 doubles
      if (t < 2 * n) (t < n ? S.s2p : S.s2m)[t < n ? t : t - n] = src[2 * n * n + t];
    } else {
#pragma unroll 4
      for (int e = t; e < n * n; e += T) {
        const int col = e / n, row = e % n;
        S.m[2][TM::at(row, col)] = src[col * LD + row];
        S.m[3][TM::at(row, col)] = src[n * LD + col * LD + row];
      }
      if (t < 2 * n) (t < n ? S.s2p : S.s2m)[t < n ? t : t - n] = src[2 * n * LD + t];
    }
  }

  // The clear run (S.tc, S.cp, S.cm: transmission and sources of consecutive
  // NONSCATTER_LAYER4 layers) below the stack.  Complete before the call; the
  // caller synchronises before the next read.
  __device__ static __forceinline__ void add_clear(SM& S, RG& G, int i) {
    const int t = threadIdx.x, lane = t & 31, g = lane >> 2, q = lane & 3, row = 8 * i + g;
    const double zp = mvsym(S.m[0], i, S.cm), zm = mvtm(S, G, i, S.cm);
    const double sp = S.cp[row] + S.tc[row] * (S.sp[row] + zp), sm = S.sm[row] + zm;
    team_sync();
    for (int e = t; e < n * n; e += T) {
      const int col = e / n, r = e % n, a = TM::at(r, col);
      S.m[0][a] = S.tc[r] * (S.m[0][a] * S.tc[col]);
      S.m[1][a] = S.tc[r] * S.m[1][a];
    }
    if constexpr (!SYM) {
#pragma unroll
      for (int j = 0; j < NB; j++)
#pragma unroll
        for (int e = 0; e < 2; e++) G.tm[j][e] = G.tm[j][e] * S.tc[8 * j + 2 * q + e];
    }
    if (q == 0) {
      S.sp[row] = sp;
      S.sm[row] = sm;
    }
  }

  // The first scattering layer (S.m[2], S.m[3], S.s2p, S.s2m) below a clear
  // run (none: tc = 1, cp = cm = 0) starts the stack.
  __device__ static __forceinline__ void start(SM& S, RG& G, int i) {
    const int t = threadIdx.x, lane = t & 31, g = lane >> 2, q = lane & 3, row = 8 * i + g;
    for (int e = t; e < n * n; e += T) {
      const int col = e / n, r = e % n, a = TM::at(r, col);
      S.m[0][a] = S.m[2][a];
      S.m[1][a] = S.m[3][a] * S.tc[col];
    }
    const double tr = S.tc[row];
#pragma unroll
    for (int d = 0; d < (SYM ? D + 1 : NB); d++) {
      const int j = SYM ? TM::blk(i, d) : d;
      const double2 r2 = ldsym(S.m[2], i, j);
      G.rm[d][0] = tr * (r2.x * S.tc[8 * j + 2 * q]);
      G.rm[d][1] = tr * (r2.y * S.tc[8 * j + 2 * q + 1]);
    }
    if constexpr (!SYM) {
#pragma unroll
      for (int j = 0; j < NB; j++) {
        const double2 t2 = ldrow(S.m[3], i, j);
        G.tm[j][0] = tr * t2.x;
        G.tm[j][1] = tr * t2.y;
      }
    }
    const double zp = mvsym(S.m[3], i, S.cp), zm = mvsym(S.m[2], i, S.cp);
    if (q == 0) {
      S.sp[row] = S.s2p[row] + zp;
      S.sm[row] = S.cm[row] + tr * (S.s2m[row] + zm);
    }
  }

  // A segment's stack into (rec0: R+, T+, S+, S-; rec1: R-, T-) as images of
  // right factors.  SYM: segments below the top store T+^T (their T2m) for T+.
  __device__ static __forceinline__ void save(SM& S, const RG& G, int i, bool top, double* rec0, double* rec1) {
    const int t = threadIdx.x;
    stres(S.m[4], G.rm, i);
    if constexpr (!SYM) {
#pragma unroll
      for (int j = 0; j < NB; j++) strow(S.m[5], i, j, G.tm[j]);
    }
    team_sync();
    for (int e = t; e < n * n; e += T) {
      const int col = e / n, r = e % n, a = TM::at(r, col);
      rec0[a] = S.m[0][a];
      rec0[n * n + a] = (SYM && !top) ? S.m[1][TM::at(col, r)] : S.m[1][a];
      rec1[a] = S.m[4][a];
      if (!SYM) rec1[n * n + a] = S.m[5][a];
    }
    if (t < 2 * n) rec0[2 * n * n + t] = t < n ? S.sp[t] : S.sm[t - n];
  }

  // The top segment's stack back.
  __device__ static __forceinline__ void load_top(SM& S, RG& G, int i, const double* rec0, const double* rec1) {
    const int t = threadIdx.x, lane = t & 31, g = lane >> 2, q = lane & 3, row = 8 * i + g;
    for (int e = t; e < n * n; e += T) {
      S.m[0][e] = __ldcg(rec0 + e);
      S.m[1][e] = __ldcg(rec0 + n * n + e);
    }
#pragma unroll
    for (int d = 0; d < (SYM ? D + 1 : NB); d++)
#pragma unroll
      for (int e = 0; e < 2; e++)
        G.rm[d][e] = __ldcg(rec1 + TM::at(row, 8 * (SYM ? TM::blk(i, d) : d) + 2 * q + e));
    if constexpr (!SYM) {
#pragma unroll
      for (int j = 0; j < NB; j++)
#pragma unroll
        for (int e = 0; e < 2; e++) G.tm[j][e] = __ldcg(rec1 + n * n + TM::at(row, 8 * j + 2 * q + e));
    }
    if (t < 2 * n) (t < n ? S.sp : S.sm)[t < n ? t : t - n] = __ldcg(rec0 + 2 * n * n + t);
  }

  // A lower segment's stack as second operand: R2m, T2m and the sources.
  __device__ static __forceinline__ void load_lower(SM& S, const double* rec0, const double* rec1) {
    const int t = threadIdx.x;
    const double* t2m = SYM ? rec0 + n * n : rec1 + n * n;
    for (int e = t; e < n * n; e += T) {
      S.m[2][e] = __ldcg(rec1 + e);
      S.m[3][e] = __ldcg(t2m + e);
    }
    if (t < 2 * n) (t < n ? S.s2p : S.s2m)[t < n ? t : t - n] = __ldcg(rec0 + 2 * n * n + t);
  }

  // End of a unit: the stack on the surface (src/sfc_matrices.f90; default
  // emissivity sfc_optics.f90:79-81) under the sky (src/surface.f90:169-195).
  // INTERNAL_RADIANCE4 (src/radintg4.f90:119-172) at the surface is the solution of
  //   dn = R+ up + T+ sky + S+,  up = Rs dn + gnd,
  // that is (I - R+ Rs) dn = T+ sky + S+ + R+ gnd; at the top dn = sky and
  //   up = R- sky + T- up(surface) + S-,
  // the same radiances as the stack combined with the surface: one elimination
  // per unit instead of three inverses and fourteen products.  `scat`: the stack
  // has matrices, else it is the clear run.  Complete before the call.
  __device__ static __forceinline__ void finish(const Batch& b, const Work& w, const pamtra_b200_settings& st,
                                                const pamtra_b200_outputs& out, SM& S, const RG& G, int i, int c,
                                                int fi, bool scat, int status) {
    const int t = threadIdx.x, lane = t & 31, g = lane >> 2, q = lane & 3, row = 8 * i + g;
    const int Fm = b.max_nfreq, L = b.nlyrs[c];
    const double wl = C_LIGHT / (b.freq(c, fi) * 1.e3);
    const char refl = (char)b.sfc_refl[c];
    const double e = st.emissivity, rr = 1.0 - e;
    const bool spec = refl == 'S' || refl == 'F', lamb = refl == 'L';
    if (!spec && !lamb) status |= PAMTRA_B200_WARNING;
    const double r1 = spec ? (rr + rr) / 2.0 : 0.0;
    if (t < n) {
      const double pg = planck(w.gtemp[c], wl), psky = planck(SKY_TEMP, wl);
      const bool I = (t & 1) == 0;
      S.gnd[t] = I ? (spec ? (1.0 - r1) * pg : lamb ? e * pg : 0.0) * S.sc[t] : 0.0;
      S.sky[t] = I ? psky * S.sc[t] : 0.0;
    }
    team_sync();
    // Rs x for component t: specular r1 x; Lambert 2 rr sum over I of mu w x, on I (scaled: both sides)
    auto surface = [&](const double* x) -> double {
      if (spec) return r1 * x[t];
      if (!lamb || (t & 1)) return 0.0;
      double s = 0.0;
      for (int j = 0; j < N; j++) s += 2.0 * rr * S.mu[j] * S.wq[j] * (x[2 * j] * S.is[2 * j]);
      return s * S.sc[t];
    };
    if (scat) {
      double s = mvsym(S.m[0], i, S.gnd), z = 0.0;
#pragma unroll 4
      for (int u = 0; u < NB; u++) {
        const double2 a = ldrow(S.m[1], i, u), v = vec(S.sky, u);
        z = fma(a.y, v.y, fma(a.x, v.x, z));
      }
      z = quad_sum(z);
      if (q == 0) S.v[row] = s + z + S.sp[row];
      // I - R+ Rs, column-major with leading dimension n + 4
      double* const M = S.m[4];
      for (int k = t; k < n * n; k += T) {
        const int col = k / n, r = k % n;
        double v = 0.0;
        if (spec) {
          v = r1 * S.m[0][TM::at(r, col)];
        } else if (lamb && (col & 1) == 0) {
          for (int j = 0; j < N; j++) v += S.m[0][TM::at(r, 2 * j)] * S.sc[2 * j];
          v = v * (2.0 * rr * S.mu[col >> 1] * S.wq[col >> 1] * S.is[col]);
        }
        M[col * LD + r] = ((r == col) ? 1.0 : 0.0) - v;
      }
      team_sync();
      if (ginv<n, T>(M, S.inv)) status |= PAMTRA_B200_FATAL | PAMTRA_B200_ST_PIVOT;
      if (t < n) {
        double d = 0.0;
        for (int k = 0; k < n; k++) d = fma(M[k * LD + t], S.v[k], d);
        S.dn[t] = d;
      }
      team_sync();
      if (t < n) S.up[t] = surface(S.dn) + S.gnd[t];
      stres(S.m[4], G.rm, i);
      team_sync();
      const double zr = mvsym(S.m[4], i, S.sky), zt = mvtm(S, G, i, S.up);
      if (q == 0) S.upt[row] = zr + zt + S.sm[row];
    } else {
      if (t < n) S.dn[t] = S.tc[t] * S.sky[t] + S.cp[t];
      team_sync();
      if (t < n) {
        S.up[t] = surface(S.dn) + S.gnd[t];
        S.upt[t] = S.cm[t] + S.tc[t] * S.up[t];
      }
    }
    team_sync();
    // output levels: L + 1 the surface, 1 the top (a later output of the same level takes it)
    int io_sfc = -1, io_top = -1;
    for (int io = 0; io < b.noutlevels; io++) {
      const int lev = w.outlev[(size_t)c * b.noutlevels + io];
      if (lev == L + 1) io_sfc = io;
      else if (lev == 1) io_top = io;
      else status |= PAMTRA_B200_FATAL | PAMTRA_B200_ST_SIZE;  // intermediate levels not supported
    }
    // collect_output + CONVERT_OUTPUT
    if (t < 2 * N) {
      const int jj = t % N, io = t < N ? io_sfc : io_top;
      if (io >= 0) {
        const double *U = t < N ? S.up : S.upt, *Dn = t < N ? S.dn : S.sky;
        const double f = S.is[2 * jj];
        double u0 = U[2 * jj] * f, u1 = U[2 * jj + 1] * f, d0 = Dn[2 * jj] * f, d1 = Dn[2 * jj + 1] * f;
        if (st.outpol_vh) {
          double iv = 0.5 * (u0 + u1), ih = 0.5 * (u0 - u1);
          u0 = iv; u1 = ih;
          iv = 0.5 * (d0 + d1); ih = 0.5 * (d0 - d1);
          d0 = iv; d1 = ih;
          u0 = 2.0 * u0; u1 = 2.0 * u1; d0 = 2.0 * d0; d1 = 2.0 * d1;
        }
        const int NA = 2 * b.max_nummu;
        double* tbo = out.tb + ((size_t)c * b.noutlevels + io) * NA * Fm * 2;
        const size_t up_i = ((size_t)(N - 1 - jj) * Fm + fi) * 2, dn_i = ((size_t)(N + jj) * Fm + fi) * 2;
        tbo[up_i + 0] = rad_to_tb(u0, wl);
        tbo[up_i + 1] = rad_to_tb(u1, wl);
        tbo[dn_i + 0] = rad_to_tb(d0, wl);
        tbo[dn_i + 1] = rad_to_tb(d1, wl);
      }
    }
    if (out.emissivity)
      for (int k = t; k < 2 * N; k += T)
        out.emissivity[(((size_t)c * 2 + k / N) * Fm + fi) * b.max_nummu + k % N] = e;
    if (t == 0 && status) atomicOr(&w.status[(size_t)c * Fm + fi], status);
  }

  // quadrature nodes and the scaling of the stack's rows (1 when not SYM)
  __device__ static __forceinline__ void init(SM& S, const Work& w) {
    const int t = threadIdx.x;
    if (t < N) { S.mu[t] = w.lob_mu[lob_off(N) + t]; S.wq[t] = w.lob_w[lob_off(N) + t]; }
    if (t < n) {
      const double v = SYM ? sqrt(w.lob_mu[lob_off(N) + (t >> 1)] * w.lob_w[lob_off(N) + (t >> 1)]) : 1.0;
      S.sc[t] = v;
      S.is[t] = SYM ? 1.0 / v : 1.0;
    }
  }
};

template <int N, bool SYM>
__global__ void __launch_bounds__(SymTeam<2 * N>::T, (N == 32 ? 1 : 4)) k_adding(Batch b, Work w, pamtra_b200_settings st,
                                                                                pamtra_b200_outputs out, int maxseg) {
  using A = Adder<N, SYM>;
  using TM = SymTeam<2 * N>;
  constexpr int n = 2 * N;
  extern __shared__ double smem_raw[];
  AddSmem<N>& S = *reinterpret_cast<AddSmem<N>*>(smem_raw);
  const int t = threadIdx.x, lane = t & 31, i = t >> 5;
  const int Lm = b.max_nlyrs, Fm = b.max_nfreq;
  const int nitems = b.ncol * Fm * maxseg;
  A::init(S, w);
  for (;;) {
    team_sync();
    if (t == 0) S.unit = atomicAdd(&w.counters[5 + (N == 8 ? 0 : (N == 16 ? 1 : 2))], 1);
    team_sync();
    const int item = S.unit;
    if (item >= nitems) break;
    const int unit = item / maxseg, seg = item % maxseg, c = unit / Fm, fi = unit % Fm;
    if (fi >= b.col_nfreq(c) || w.col_nmu[c] != N) continue;
    const int L = b.nlyrs[c];
    const int* pres = w.pres_idx + (size_t)c * Lm;
    // scattering layers of the unit, and of this segment: top-down layers k0 .. k1 - 1
    int M = 0;
    for (int k = 0; k < L; k += 32) M += __popc(__ballot_sync(0xffffffffu, k + lane < L && pres[L - 1 - min(k + lane, L - 1)] >= 0));
    const int nseg = add_segments(M);
    if (seg >= nseg) continue;
    const int s0 = (int)((long long)M * seg / nseg), s1 = (int)((long long)M * (seg + 1) / nseg);
    int k0 = 0, k1 = L;
    auto layer_of = [&](int s) {  // top-down index of the s-th scattering layer
      int seen = 0;
      for (int k = 0; k < L; k += 32) {
        const unsigned m = __ballot_sync(0xffffffffu, k + lane < L && pres[L - 1 - min(k + lane, L - 1)] >= 0);
        if (seen + __popc(m) > s) {
          unsigned r = m;
          for (; seen < s; seen++) r &= r - 1;
          return k + __ffs((int)r) - 1;
        }
        seen += __popc(m);
      }
      return L;
    };
    if (seg > 0) k0 = layer_of(s0);
    if (seg + 1 < nseg) k1 = layer_of(s1);
    const double wl = C_LIGHT / (b.freq(c, fi) * 1.e3);
    const double* hl = w.hgt_lev + (size_t)c * (Lm + 1);
    const double* tl = w.temp_lev + (size_t)c * (Lm + 1);
    const double* kg = w.kgas + ((size_t)c * Fm + fi) * Lm;
    int status = 0;
    typename A::RG G;
    auto record = [&](int k) { return w.lay + ((size_t)pres[L - 1 - k] * Fm + fi) * w.lay_stride; };
    // consecutive clear layers, per angle (threads t < n)
    double ct = 1.0, cp = 0.0, cm = 0.0;
    bool run = false, scat = false;
    int k = k0;      // top-down layer index
    int next = 0;    // segment to combine next (0: this segment's layers are not done)
    bool mine = true;
    for (;;) {
      const double* rec0 = nullptr;
      if (next == 0) {
        for (; k < k1 && pres[L - 1 - k] < 0; k++) {
          // NONSCATTER_LAYER4 (src/radintg4.f90:79-117) below the run
          const int z = L - 1 - k;
          if (t < n) {
            const double zdiff = fabs(hl[z + 1] - hl[z]);
            const double dtau = zdiff * fmax(kg[z], 0.0);
            const double p0 = planck(tl[z + 1], wl), p1 = planck(tl[z], wl);
            const double path = dtau / S.mu[t >> 1], tr = exp(-path);
            double a = 0.0, bq = 0.0;
            if (dtau > 0.0 && (t & 1) == 0) {
              const double slope = (p1 - p0) / path;
              a = (p1 - slope - (p1 - slope * (1.0 + path)) * tr) * S.sc[t];
              bq = (p0 + slope - (p0 + slope * (1.0 + path)) * tr) * S.sc[t];
            }
            cp = a + tr * cp;
            cm = cm + ct * bq;
            ct = tr * ct;
          }
          run = true;
        }
        const bool end = k >= k1, first = !scat && !end;
        if (!end) {
          A::load_layer(S, record(k));
          k++;
          if (t == 0) {  // the next scattering layer's record on its way to L2
            int kk = k;
            while (kk < k1 && pres[L - 1 - kk] < 0) kk++;
            if (kk < k1)
              asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(record(kk)), "r"(A::RECORD_BYTES) : "memory");
          }
        }
        if (run || !scat) {
          if (t < n) { S.tc[t] = ct; S.cp[t] = cp; S.cm[t] = cm; }
          ct = 1.0;
          cp = cm = 0.0;
          run = false;
          team_sync();
          if (first) A::start(S, G, i);
          else if (scat) A::add_clear(S, G, i);
        }
        team_sync();
        if (first) {
          scat = true;
          continue;
        }
        if (end) {
          if (nseg == 1) break;
          // the stack into the segment's first two layer records; the CTA of the unit's last segment goes on
          A::save(S, G, i, seg == 0, record(layer_of(s0)), record(layer_of(s0 + 1)));
          __threadfence();
          team_sync();
          if (t == 0) S.last = atomicAdd(&w.seg_cnt[unit], 1) == nseg - 1;
          team_sync();
          mine = S.last;
          if (!mine) break;
          __threadfence();
          A::load_top(S, G, i, record(layer_of(0)), record(layer_of(1)));
          next = 1;
        }
      }
      if (next > 0) {
        if (next == nseg) break;
        const int f0 = (int)((long long)M * next / nseg);
        rec0 = record(layer_of(f0));
        A::load_lower(S, rec0, record(layer_of(f0 + 1)));
        team_sync();
        next++;
      }
      A::combine(S, G, rec0, i, status);
      team_sync();
    }
    if (!mine) {
      if (t == 0 && status) atomicOr(&w.status[(size_t)c * Fm + fi], status);
      continue;
    }
    A::finish(b, w, st, out, S, G, i, c, fi, scat, status | w.col_status[c]);
  }
}

}  // namespace pb
