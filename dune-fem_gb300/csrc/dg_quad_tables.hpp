// Coefficient tables of the integer-pipe FP64 apply at the Gauss points
// (dg_quad_fixed.cuh).
#pragma once
#include <cmath>

#include "dg_kernel.cuh"
#include "fixed_point.cuh"

namespace gbfem {

constexpr int kQxMinExp = 400, kQxMaxExp = 1600;  // biased exponents of u
constexpr int kQxKappaSpan = 100;                 // kappa within 2^+-100
constexpr int kQxSlow = 0xFFFF;
// smallest log2 of a scale of the operator.  A result's scale 2^x, built as an exponent
// field, is smallest where a cell and its neighbours are zero: x = 400 - 1022 (u), - 209
// (47 bits of the contractions, 6 27 shifts of zero magnitudes), - 99 (kappa) and this:
// at -93 the field is 1.
constexpr int kQxRowExpMin = -90;

struct QxTables {
  FxCoef B[kDgMaxQ * kDgMaxN];        // B[a n + i], S = 2^lB
  FxCoef D[kDgMaxQ * kDgMaxQ];        // Dc[a q + b], S = 2^lD
  FxCoef Dt[3][kDgMaxQ * kDgMaxQ];    // Dt_d[o q + a], S = 2^lDt
  FxCoef BT[kDgMaxN * kDgMaxQ];       // w_a L_i(x_a), [i q + a], S = 1
  FxCoef tv[kDgMaxN], td[kDgMaxN];    // L_i(1), r L_i'(1), S = 2^lT
  FxCoef fv[3][kDgMaxN], fg[3][kDgMaxN];  // cv L_i(1), cg L_i'(1), S = 2^lF[d][i]
  int lB, lD, lDt, lT;
  int lF[3][kDgMaxN];
};

struct QxArgs {
  const long long *kq, *kf;    // kappa 2^(62-(ke-1022)) at the points
  const unsigned short* ke;    // [cell] kappa's exponent, kQxSlow: not representable
};

inline FxCoef qx_coef(long double c, int lS) {
  const long long v = llroundl(ldexpl(c, 62 - lS));
  const FxLimbs s = fx_split(v);
  return FxCoef{s.h, s.l};
}
// log2 of the smallest power of two >= big, and >= sum / ratio
inline int qx_scale(long double big, long double sum, long double ratio) {
  int e = 0;
  const long double need = fmaxl(big, sum / ratio);
  if (need > 0.0L) frexpl(need, &e);
  return e;
}

}  // namespace gbfem
