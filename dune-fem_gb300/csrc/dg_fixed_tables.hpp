// Coefficient tables of the integer-pipe FP64 apply (dg_fixed_kernel.cuh).
#pragma once
#include "dg_kernel.cuh"
#include "fixed_point.cuh"

namespace gbfem {

// Integer coefficients of one axis (n <= 5).
struct FxAxis {
  FxCoef v[kDgMaxN], P[kDgMaxN];  // traces on the upper face, / 8, CB = 62
  FxCoef O[kDgMaxN * kDgMaxN];    // line operator
  FxCoef nv[kDgMaxN], np[kDgMaxN], a[kDgMaxN];  // face part
  int ex[kDgMaxN];                // row i: y_i = Y 2^(E + (ex[i] >> 20) - 1023)
};
struct FxTables {
  FxAxis ax[3];
  int inflow_upper[3];  // the neighbour a_i couples is the upper one
  int couple[3][2];     // the lower / upper neighbour enters the line at all
  int slope;            // no penalty: the second trace is fx_slope_scale times minus the outward slope
};

// Traces are T = v 2^(56-(E-1022)), 1/32 of the scale of X, so that with
// coefficients of at most kFxClassSum in each parity class a difference of two
// summed over two faces stays below 2^61.7, and a row of at most 2 s in sum
// below 2^63 in its middle sum: CB = 62 without advection, 61 with its longer
// rows.
constexpr double kFxClassSum = 6.3;
constexpr int kFxTraceExp = 56;
// scale of the slope trace: its largest class sum over 2 <= n <= 5 is 3.5, 3.4,
// 4.4 and 4.6 with it
GBFEM_HD constexpr double fx_slope_scale(int n) { return n == 2 ? 1.0 : (n == 3 ? 0.25 : (n == 4 ? 0.125 : 0.0625)); }
constexpr int fx_coef_bits(bool adv) { return adv ? 61 : 62; }

// y = u + sum_j a[j] w_j, j < earlier from memory and j = earlier the apply's result
struct FxStage {
  const double* u;
  const double* w[2];
  double a[3];
  int earlier;  // results before this one
  double* y;
};

}  // namespace gbfem
