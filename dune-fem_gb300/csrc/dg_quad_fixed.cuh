// FP64 apply with kappa a DG field, at the Gauss points, in block fixed point on
// the integer pipes (fixed_point.cuh).  The same integrals and the same order of
// contractions as dg_apply_kernel (dg_kernel.cuh), which is bound by the FP64
// pipe (270 multiply-adds per dof at Q3, 0.5 clocks each on an SM).
//
// What bounds it: integer issue and the barriers between the contractions (2.3
// instructions a clock and SM), about 3500 instructions per dof at Q3 in place of 135
// clocks of FP64 pipe.  Measured (GB300), dg_apply_kernel before, this after:
// 45 x 38 x 33 Q3 2152 -> 571 us.
//
// Numbers.  All of a cell's values are integers v 2^(s-(E-1022)) of its exponent E
// (its largest dof's), |integer| <= 2^60; a contraction with a matrix c of row sums
// L1 <= 2.5 S, held as round(c / S 2^62), gives (sum X C) / 2^64, so s drops by
// 2 + log2 S while the bound holds.  What the bound leaves unused is taken back
// before the next contraction, which shifts its input left by the room above the
// largest magnitude in the cell (on the face).  So every rounding is relative to
// the values it contracts, as in FP64, at 2^-56 to 2^-58 of the largest one.  kappa is
// held per cell in 62 bits of its largest point value.  The exponent of a face is
// the larger of its two cells'; a neighbour's line is converted with its own
// exponent and aligned.
//
//  volume  U = B B B u;  along each axis d and line: G = Dc U, f = kappa G,
//          V += Dt_d f with Dt = diag(1/w) Dc^T diag(w) eps |K| / h_d^2 (so that the
//          weights sit in the last three contractions);  r = (B^T diag w)^3 V
//  faces   J = v- - v+ and D = r dv/dn of both sides (r = 1 / (2 penalty)) as
//          coefficients, to the points;  Val = kbar J - k- D- - k+ D+, Grad = k- J;
//          back with B^T diag w;  r_i += cv L_i (Val_1 +- Val_0) + cg L_i' (Grad_1 +- Grad_0)
// Weak u = 0 is J = 2 v, D+ = v + D-, k+ = k-.
//
// Each line is one thread's; every output is a fixed-order sum of integers.  A CTA
// that meets values or kappas it cannot hold (infinities, NaN, magnitudes beyond
// 2^-622 .. 2^577) recomputes its cells with dg_apply_cells.
#pragma once
#include <cuda_runtime.h>
#include <type_traits>

#include "dg_kernel.cuh"
#include "dg_quad_tables.hpp"

namespace gbfem {

// X = v 2^(60-(E-1022)), truncated
__device__ __forceinline__ long long qx_from_double(double v, int E) { return fx_from_double(v, E) >> 1; }

__device__ __forceinline__ uint32_t qx_mag(long long v) {
  const int hi = int(uint64_t(v) >> 32);
  return uint32_t(hi ^ (hi >> 31)) + 1u;  // |v| <= qx_mag 2^32
}
// The traces keep kQxUp more bits than a contraction's result: all coefficients of
// a face share the unit that the largest needs, and the interpolation to the points
// adds their roundings up.  They stay below 2^61, J and D+ below 2^62.
constexpr int kQxUp = 3;

// left shift that brings magnitudes below m 2^32 under 2^60
__device__ __forceinline__ int qx_room(uint32_t m) {
  return __clz(int(m)) - 4;
}
// (negative only for J and D, which may need up to two bits more)
__device__ __forceinline__ long long qx_shift(long long v, int k) {
  return k >= 0 ? (long long)(uint64_t(v) << (k & 63)) : v >> -k;
}

// NC groups of arrays (cell stride ics / ocs) of dims [I0][I1][I2], contracted along
// AX with M (OUT x IN, entry M[o LDM + i]).  The input is shifted left as far as its
// largest magnitude room[c] allows (null: not at all); mag[c] takes the output's
// (null: not kept).  SUB groups per cell, ISUB / OSUB apart, counted by c.  BOTH: the
// shift may be to the right.
template <int AX, int I0, int I1, int I2, int OUT, int LDM, int NC, int T, int SUB = 1, int ISUB = 0, int OSUB = 0,
          bool BOTH = false>
__device__ __forceinline__ void qx_contract(const long long* __restrict__ in, int ics, long long* __restrict__ out,
                                            int ocs, const FxCoef* __restrict__ M, const uint32_t* room, uint32_t* mag) {
  constexpr int IN = AX == 0 ? I0 : (AX == 1 ? I1 : I2);
  constexpr int O1 = AX == 1 ? OUT : I1, O2 = AX == 2 ? OUT : I2;
  constexpr int NB = AX == 2 ? I1 : I2, NA = AX == 0 ? I1 : I0;
  constexpr int SIA = AX == 0 ? I2 : I1 * I2, SIB = AX == 2 ? I2 : 1, SI = AX == 0 ? I1 * I2 : (AX == 1 ? I2 : 1);
  constexpr int SOA = AX == 0 ? O2 : O1 * O2, SOB = AX == 2 ? O2 : 1, SO = AX == 0 ? O1 * O2 : (AX == 1 ? O2 : 1);
  constexpr int LINES = NA * NB;
  for (int item = threadIdx.x; item < NC * LINES; item += T) {
    const int c = item / LINES, ln = item - c * LINES;
    const int xa = ln / NB, xb = ln - xa * NB;
    const long long* src = in + (c / SUB) * ics + (c % SUB) * ISUB + xa * SIA + xb * SIB;
    long long* dst = out + (c / SUB) * ocs + (c % SUB) * OSUB + xa * SOA + xb * SOB;
    const int k = room ? qx_room(room[c]) : 0;
    FxLimbs x[IN];
#pragma unroll
    for (int i = 0; i < IN; ++i) x[i] = fx_split(BOTH ? qx_shift(src[i * SI], k) : (long long)(uint64_t(src[i * SI]) << (k & 63)));
    uint32_t m = 0;
#pragma unroll
    for (int o = 0; o < OUT; ++o) {
      FxAcc acc = FxAcc::rounded();
#pragma unroll
      for (int i = 0; i < IN; ++i) acc.add(x[i], M[o * LDM + i]);
      const long long v = acc.value();
      dst[o * SO] = v;
      if (mag) m = max(m, qx_mag(v));
    }
    if (mag) atomicMax(mag + c, m);
  }
}

template <int N, int Q, int CPB>
struct QxSmem {
  static constexpr int N2 = N * N, N3 = N2 * N, Q2 = Q * Q, Q3 = Q2 * Q;
  static constexpr int VOL = Q * N2 + Q2 * N + 2 * Q3;                 // T1, T2, U, V
  static constexpr int FACE = 6 * (N2 + Q * N + Q2) + 4 * Q2;          // per direction: both faces
  static constexpr int WORK = VOL > FACE ? VOL : FACE;
  static constexpr size_t FIXED = size_t(CPB) * (2 * N3 + WORK) * 8;   // X, r, work
  static constexpr size_t SLOW = size_t(DgSmem<N, Q, true, 1>::TOTAL) * 8;
  static constexpr size_t BYTES = FIXED > SLOW ? FIXED : SLOW;
};

// One cell by the FP64 formulas (not inlined: its registers are not the fast path's).
template <int N, int Q>
__device__ __noinline__ void qx_cell_f64(const DgArgsT<double>& args, const DgTablesT<double>& tabs, double* sm,
                                         long long cell) {
  DgArgsT<double> one = args;
  one.cell_begin = cell;
  one.cell_count = 1;
  dg_apply_cells<double, N, Q, true, 1>(one, tabs, sm, cell);
}

// Cells and threads per CTA.  32 warps per SM in four CTAs hide each other's barriers:
// 45 x 38 x 33 Q3 takes 571 us, 621 with three CTAs (80 registers), 567 with five,
// 648 with half the cells and threads in eight, 634 with 320 threads in three; Q1, Q2
// and Q4 1056, 742 and 596 us at 101 x 77 x 64, 61 x 52 x 47 and 33 x 30 x 31, against
// 1243, 820 and 781 with five CTAs of 128 threads.
template <int N, int Q>
struct QxShape {
  static constexpr int CPB = N == 2 ? 32 : (N == 3 ? 16 : (N == 4 ? 8 : 6));
  static constexpr int T = 256, MINB = 4;
};

template <int N, int Q>
__global__ void __launch_bounds__(QxShape<N, Q>::T, QxShape<N, Q>::MINB) dg_quad_fixed_kernel(const __grid_constant__ DgArgsT<double> args,
                                                                         const __grid_constant__ DgTablesT<double> tabs,
                                                                         const __grid_constant__ QxTables qx,
                                                                         const QxArgs kx) {
  constexpr int CPB = QxShape<N, Q>::CPB, T = QxShape<N, Q>::T;
  using S = QxSmem<N, Q, CPB>;
  constexpr int N2 = S::N2, N3 = S::N3, Q2 = S::Q2, Q3 = S::Q3, WS = S::WORK;
  extern __shared__ __align__(16) unsigned char qx_smem[];
  long long* const sX = reinterpret_cast<long long*>(qx_smem);   // [CPB][N3]
  double* const sr = reinterpret_cast<double*>(sX + CPB * N3);   // [CPB][N3]
  long long* const work = reinterpret_cast<long long*>(sr + CPB * N3);  // [CPB][WORK]
  __shared__ int sE[CPB], sKe[CPB], slow;
  // largest magnitudes after each contraction: of the cell's values (t1, t2, U; V,
  // t2, t1), and on each face (coefficients, after B, at the points; fluxes, after
  // one and both B^T)
  __shared__ uint32_t magV[6][CPB], magF[6][2 * CPB];
  __shared__ int eF[2 * CPB], xF[2 * CPB];
  const int tid = threadIdx.x;
  const long long cend = args.cell_begin + (args.cell_count > 0 ? args.cell_count : args.ncells);
  const long long c0 = args.cell_begin + (long long)blockIdx.x * CPB;
  if (c0 >= cend) return;
  const int ncell = int(cend - c0 < CPB ? cend - c0 : CPB);
  if (tid == 0) slow = 0;
  for (int c = tid; c < CPB; c += T) {
    sE[c] = kQxMinExp;
    for (int k = 0; k < 6; ++k) magV[k][c] = 0;
    const int ke = c < ncell ? int(kx.ke[c0 + c]) : 1023;
    sKe[c] = ke;
  }
  __syncthreads();
  // ---- own dofs, the cells' exponents -----------------------------------------
  const double* ug = args.u + c0 * N3;
  for (int e = tid; e < CPB * N3; e += T) {
    const int c = e / N3;
    const double v = c < ncell ? __ldg(ug + e) : 0.0;
    sr[e] = v;
    const uint32_t hi = fx_abs_hi(v);
    const int ex = int(hi >> 20);
    // (a value below the range counts as the smallest exponent: it only has to
    // be zero or negligible, which the check of the cell's largest one decides)
    if (ex > kQxMinExp) atomicMax(&sE[c], ex);
    else if ((fx_bits(v) << 1) != 0 && ex <= kQxMinExp) atomicMax(&sE[c], kQxMinExp + 1);
  }
  __syncthreads();
  for (int e = tid; e < CPB * N3; e += T) sX[e] = qx_from_double(sr[e], sE[e / N3]);
  for (int c = tid; c < ncell; c += T)
    if (sE[c] >= kQxMaxExp || sE[c] == kQxMinExp + 1 || sKe[c] == kQxSlow) slow = 1;
  __syncthreads();
  // ---- volume -------------------------------------------------------------------
  {
    long long* t1 = work;
    long long* t2 = t1 + Q * N2;
    long long* U = t2 + Q2 * N;
    long long* V = U + Q3;
    qx_contract<0, N, N, N, Q, N, CPB, T>(sX, N3, t1, WS, qx.B, nullptr, magV[0]);
    __syncthreads();
    qx_contract<1, Q, N, N, Q, N, CPB, T>(t1, WS, t2, WS, qx.B, magV[0], magV[1]);
    __syncthreads();
    qx_contract<2, Q, Q, N, Q, N, CPB, T>(t2, WS, U, WS, qx.B, magV[1], magV[2]);
    __syncthreads();
    // (one copy of the code for the three axes, and for the three directions below:
    // unrolled, the kernel does not fit the instruction cache)
#pragma unroll 1
    for (int D = 0; D < 3; ++D) {
      const int STR = D == 0 ? Q2 : (D == 1 ? Q : 1);
      for (int item = tid; item < CPB * Q2; item += T) {
        const int c = item / Q2, ln = item - c * Q2, a = ln / Q, b = ln - a * Q;
        const int base = D == 0 ? ln : (D == 1 ? a * Q2 + b : ln * Q);
        const long long* src = U + c * WS + base;
        long long* dst = V + c * WS + base;
        const long long* kp = kx.kq + (c0 + (c < ncell ? c : 0)) * Q3 + base;
        const int k = qx_room(magV[2][c]);
        FxLimbs x[Q], f[Q];
#pragma unroll
        for (int i = 0; i < Q; ++i) x[i] = fx_split((long long)(uint64_t(src[i * STR]) << (k & 63)));
#pragma unroll
        for (int o = 0; o < Q; ++o) {
          const FxLimbs kl = fx_split(__ldg(kp + o * STR));
          FxAcc g = FxAcc::rounded();
#pragma unroll
          for (int i = 0; i < Q; ++i) g.add(x[i], qx.D[o * Q + i]);
          FxAcc fl = FxAcc::rounded();
          fl.add(fx_split(g.value()), FxCoef{kl.h, kl.l});
          f[o] = fx_split(fl.value() * 4);
        }
        uint32_t m = 0;
#pragma unroll
        for (int o = 0; o < Q; ++o) {
          FxAcc acc = FxAcc::rounded();
#pragma unroll
          for (int i = 0; i < Q; ++i) acc.add(f[i], qx.Dt[D][o * Q + i]);
          long long v = acc.value();
          if (D != 0) v += dst[o * STR];
          dst[o * STR] = v;
          if (D == 2) m = max(m, qx_mag(v));
        }
        if (D == 2) atomicMax(magV[3] + c, m);
      }
      __syncthreads();
    }
    qx_contract<2, Q, Q, Q, N, Q, CPB, T>(V, WS, t2, WS, qx.BT, magV[3], magV[4]);
    __syncthreads();
    qx_contract<1, Q, Q, N, N, Q, CPB, T>(t2, WS, t1, WS, qx.BT, magV[4], magV[5]);
    __syncthreads();
    // the last one straight into FP64
    for (int item = tid; item < CPB * N2; item += T) {
      const int c = item / N2, jk = item - c * N2;
      const long long* src = t1 + c * WS + jk;
      int s = 0;
#pragma unroll
      for (int k = 0; k < 6; ++k) s += qx_room(magV[k][c]);
      const int k = qx_room(magV[5][c]);
      FxLimbs x[Q];
#pragma unroll
      for (int a = 0; a < Q; ++a) x[a] = fx_split((long long)(uint64_t(src[a * N2]) << k));
      // three B; G; f (shifted back by two); V; three B^T
      s += 60 - 3 * (2 + qx.lB) - (2 + qx.lD) - (sKe[c] - 1022) - (2 + qx.lDt) - 6;
      const double scale = fx_pow2((sE[c] + 1 - s) << 20);
#pragma unroll
      for (int i = 0; i < N; ++i) {
        FxAcc acc = FxAcc::rounded();
#pragma unroll
        for (int a = 0; a < Q; ++a) acc.add(x[a], qx.BT[i * Q + a]);
        sr[c * N3 + i * N2 + jk] = double(acc.value()) * scale;
      }
    }
    __syncthreads();
  }
  // ---- faces, one direction at a time ----------------------------------------------
#pragma unroll 1
  for (int D = 0; D < 3; ++D) {
    const int STR = D == 0 ? N2 : (D == 1 ? N : 1);
    long long* FC = work;              // [2 sides][J, D-, D+][N][N]
    long long* FT = FC + 6 * N2;       // [2][3][Q][N]
    long long* FQ = FT + 6 * Q * N;    // [2][3][Q][Q]
    long long* FV = FQ + 6 * Q2;       // [2][Val, Grad][Q][Q]
    // the cell across face (D, s), -1 at a domain boundary
    auto neighbour = [&](int c, int s) -> long long {
      const long long cell = c0 + (c < ncell ? c : 0);
      const long long nxy = (long long)args.nc[0] * args.nc[1];
      const long long cz = cell / nxy, rem = cell - cz * nxy, cy = rem / args.nc[0], cx = rem - cy * args.nc[0];
      const long long cd = D == 0 ? cx : (D == 1 ? cy : cz), st = D == 0 ? 1 : (D == 1 ? (long long)args.nc[0] : nxy);
      long long nb = cd + (s ? 1 : -1);
      if (nb < 0 || nb >= args.nc[D]) {
        if (!args.periodic[D]) return -1;
        nb = nb < 0 ? nb + args.nc[D] : nb - args.nc[D];
      }
      return cell + (nb - cd) * st;
    };
    for (int e = tid; e < 2 * CPB; e += T) {
      eF[e] = sE[e >> 1];
      for (int k = 0; k < 6; ++k) magF[k][e] = 0;
    }
    __syncthreads();
    // traces: v and D of the own cell (aligned below) and of the neighbour's line
    constexpr int ITEMS = CPB * 2 * N2, R = (ITEMS + T - 1) / T;
    long long tv[R], td[R];
    int te[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int item = tid + r * T;
      tv[r] = td[r] = 0;
      te[r] = -1;  // no neighbour
      if (item < ITEMS) {
        const int c = item / (2 * N2), f = item - c * 2 * N2, s = f / N2, jk = f - s * N2;
        const int j = jk / N, k = jk - j * N;
        const int base = D == 0 ? jk : (D == 1 ? j * N2 + k : jk * N);
        const long long nb = neighbour(c, s);
        if (nb >= 0) {
          const double* xs = args.u + nb * N3 + base;
          double x[N];
          uint32_t m = 0;
          uint64_t any = 0;
#pragma unroll
          for (int i = 0; i < N; ++i) {
            x[i] = __ldg(xs + i * STR);
            m = max(m, fx_abs_hi(x[i]));
            any |= fx_bits(x[i]) << 1;
          }
          int ex = int(m >> 20);
          if (ex <= kQxMinExp && any) slow = 1;
          if (ex >= kQxMaxExp) slow = 1;
          ex = max(ex, kQxMinExp);
          FxAcc ev, od, de, dd;  // even and odd parts of v and of L'
#pragma unroll
          for (int i = 0; i < N; ++i) {
            const FxLimbs l = fx_split(qx_from_double(x[i], ex));
            if (i & 1) {
              od.add(l, qx.tv[i]);
              dd.add(l, qx.td[i]);
            } else {
              ev.add(l, qx.tv[i]);
              if (i) de.add(l, qx.td[i]);
            }
          }
          // the neighbour's face 1 - s; D along this cell's outward normal:
          // s L'(1-s) with L_i'(0) = (-1)^(i+1) L_i'(1)
          const long long e = ev.value_up<kQxUp>(), o = od.value_up<kQxUp>();
          const long long g = de.value_up<kQxUp>(), q = dd.value_up<kQxUp>();
          tv[r] = s ? e - o : e + o;
          td[r] = s ? q - g : -(q + g);
          te[r] = ex;
          atomicMax(&eF[2 * c + s], ex);
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int item = tid + r * T;
      if (item < ITEMS) {
        const int c = item / (2 * N2), f = item - c * 2 * N2, s = f / N2, jk = f - s * N2;
        const int j = jk / N, k = jk - j * N;
        const int base = D == 0 ? jk : (D == 1 ? j * N2 + k : jk * N);
        const int E = eF[2 * c + s];
        const long long* xs = sX + c * N3 + base;
        FxAcc ev, od, de, dd;
#pragma unroll
        for (int i = 0; i < N; ++i) {
          const FxLimbs l = fx_split(xs[i * STR]);
          if (i & 1) {
            od.add(l, qx.tv[i]);
            dd.add(l, qx.td[i]);
          } else {
            ev.add(l, qx.tv[i]);
            if (i) de.add(l, qx.td[i]);
          }
        }
        const int so = min(E - sE[c], 63);
        const long long e = ev.value_up<kQxUp>(), o = od.value_up<kQxUp>();
        const long long g = de.value_up<kQxUp>(), q = dd.value_up<kQxUp>();
        const long long v = fx_shr(s ? e + o : e - o, so), dm = fx_shr(s ? q + g : g - q, so);
        long long J, dp;
        if (te[r] >= 0) {
          const int sn = min(E - te[r], 63);
          J = v - fx_shr(tv[r], sn);
          dp = fx_shr(td[r], sn);
        } else {
          J = args.weak_dirichlet ? 2 * v : 0;
          dp = args.weak_dirichlet ? v + dm : 0;
        }
        const long long dmm = te[r] >= 0 || args.weak_dirichlet ? dm : 0;
        long long* fc = FC + c * WS + s * 3 * N2 + jk;
        fc[0] = J;
        fc[N2] = dmm;
        fc[2 * N2] = dp;
        atomicMax(&magF[0][2 * c + s], max(qx_mag(J), max(qx_mag(dmm), qx_mag(dp))));
      }
    }
    __syncthreads();
    // to the points
    qx_contract<1, 3, N, N, Q, N, 2 * CPB, T, 2, 3 * N2, 3 * Q * N, true>(FC, WS, FT, WS, qx.B, magF[0], magF[1]);
    __syncthreads();
    qx_contract<2, 3, Q, N, Q, N, 2 * CPB, T, 2, 3 * Q * N, 3 * Q2>(FT, WS, FQ, WS, qx.B, magF[1], magF[2]);
    __syncthreads();
    // fluxes
    for (int item = tid; item < CPB * 2 * Q2; item += T) {
      const int c = item / (2 * Q2), f = item - c * 2 * Q2, s = f / Q2, ab = f - s * Q2;
      const long long cell = c0 + (c < ncell ? c : 0), nb = neighbour(c, s);
      const long long* fq = FQ + c * WS + s * 3 * Q2 + ab;
      const int kem = sKe[c];
      long long km = __ldg(kx.kf + (cell * 6 + 2 * D + s) * Q2 + ab), kp = km;
      int kef = kem;
      if (nb >= 0) {
        const int kep = int(__ldg(kx.ke + nb));
        if (kep == kQxSlow) slow = 1;
        kp = __ldg(kx.kf + (nb * 6 + 2 * D + 1 - s) * Q2 + ab);
        kef = kep == kQxSlow ? kem : max(kem, kep);
        km = fx_shr(km, min(kef - kem, 63));
        kp = fx_shr(kp, min(max(kef - kep, 0), 63));
      }
      const int fe = 2 * c + s, shQ = qx_room(magF[2][fe]);
      const FxLimbs J = fx_split((long long)(uint64_t(fq[0]) << shQ));
      const FxLimbs dm = fx_split(-(long long)(uint64_t(fq[Q2]) << shQ));
      const FxLimbs dp = fx_split(-(long long)(uint64_t(fq[2 * Q2]) << shQ));
      const FxLimbs a = fx_split(km), b = fx_split(kp), m = fx_split((km + kp) >> 1);
      FxAcc val = FxAcc::rounded(), grad = FxAcc::rounded();
      val.add(J, FxCoef{m.h, m.l});
      val.add(dm, FxCoef{a.h, a.l});
      val.add(dp, FxCoef{b.h, b.l});
      grad.add(J, FxCoef{a.h, a.l});
      long long* fv = FV + c * WS + s * 2 * Q2 + ab;
      const long long vv = val.value(), gg = grad.value();
      fv[0] = vv;
      fv[Q2] = gg;
      atomicMax(&magF[3][fe], max(qx_mag(vv), qx_mag(gg)));
      if (ab == 0) xF[fe] = kef;
    }
    __syncthreads();
    qx_contract<2, 2, Q, Q, N, Q, 2 * CPB, T, 2, 2 * Q2, 2 * Q * N>(FV, WS, FT, WS, qx.BT, magF[3], magF[4]);
    __syncthreads();
    qx_contract<1, 2, Q, N, N, Q, 2 * CPB, T, 2, 2 * Q * N, 2 * N2>(FT, WS, FC, WS, qx.BT, magF[4], magF[5]);
    __syncthreads();
    // the faces' scales: value = (integer << room) 2^xF, after the traces, two B,
    // kappa and two B^T
    for (int e = tid; e < 2 * CPB; e += T) {
      int sc = 60 - (2 + qx.lT) + kQxUp - 2 * (2 + qx.lB) - 2 - (xF[e] - 1022) - 4;
      for (int k = 0; k < 6; ++k) sc += qx_room(magF[k][e]);
      xF[e] = eF[e] - 1022 - sc;
    }
    __syncthreads();
    // expansion along the normal, both faces
    for (int item = tid; item < CPB * N2; item += T) {
      const int c = item / N2, jk = item - c * N2;
      const int j = jk / N, k = jk - j * N;
      const int base = D == 0 ? jk : (D == 1 ? j * N2 + k : jk * N);
      const long long* fc = FC + c * WS + jk;
      const int x0 = xF[2 * c], x1 = xF[2 * c + 1], xm = max(x0, x1);
      const int s0 = min(xm - x0, 63), s1 = min(xm - x1, 63);
      const int r0 = qx_room(magF[5][2 * c]), r1 = qx_room(magF[5][2 * c + 1]);
      auto at = [&](int q, int room, int sh) { return fx_shr((long long)(uint64_t(fc[q * N2]) << room), sh); };
      const long long v0 = at(0, r0, s0), g0 = at(1, r0, s0), v1 = at(2, r1, s1), g1 = at(3, r1, s1);
      const FxLimbs vs = fx_split(v1 + v0), vd = fx_split(v1 - v0), gs = fx_split(g1 + g0), gd = fx_split(g1 - g0);
      double* rc = sr + c * N3 + base;
#pragma unroll
      for (int i = 0; i < N; ++i) {
        FxAcc acc = FxAcc::rounded();
        acc.add((i & 1) ? vd : vs, qx.fv[D][i]);
        if (i) acc.add((i & 1) ? gd : gs, qx.fg[D][i]);
        // / 2^64 with CB = 62: 2^2, and the row's S
        rc[i * STR] = fma(double(acc.value()), fx_pow2((xm + 2 + qx.lF[D][i] + 1023) << 20), rc[i * STR]);
      }
    }
    __syncthreads();
  }
  if (slow) {
    __syncthreads();
    for (int c = 0; c < ncell; ++c) {
      qx_cell_f64<N, Q>(args, tabs, reinterpret_cast<double*>(qx_smem), c0 + c);
      __syncthreads();
    }
    return;
  }
  for (int e = tid; e < ncell * N3; e += T) __stcs(args.w + c0 * N3 + e, sr[e]);
}

}  // namespace gbfem
