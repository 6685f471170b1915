// The integer-pipe FP64 apply of the closed form: its coefficient tables and
// launches (dg_fixed_kernel.cuh).
#include <cmath>
#include <type_traits>

#include "dg_fixed_kernel.cuh"
#include "gbfem_internal.cuh"
#include "operator_impl.hpp"
#include "tables.hpp"

namespace gbfem {

static FxCoef fx_coef(long double c, int bits) {
  const long long v = llroundl(ldexpl(c, bits));
  const FxLimbs s = fx_split(v);
  return FxCoef{s.h, s.l};
}

// 1-D tables of the basis, made once per process (extended precision is slow
// on hosts that emulate it).
struct FxBasis {
  ConstTables1D ct;
  long double L[kDgMaxN], dL[kDgMaxN];  // at 1
  explicit FxBasis(int n) : ct(make_const_tables(n)) {
    for (int i = 0; i < n; ++i) legendre01(i, 1.0L, &L[i], &dL[i]);
  }
};

// The tables of a constant-kappa operator, from the descriptor in long double
// and rounded once; false where its coefficients do not fit the fixed-point
// ranges (a penalty so small that the trace P = v - r dv outgrows v, scales
// beyond 2^+-kFxRowExpMax) or where a line would hold fewer bits than in FP64: a row
// is formed at the largest exponent of its line and its neighbours', so every line that
// takes part has to weigh in it.  With V = sum L_j(1), a penalty alone weighs between
// V / 64 and V / 32 of the row's scale 2^e (which covers the face's 32 L_i); the least
// accepted is 0.009 (1 + V).  Error against 128 bits, entry by entry over all ratios of
// the neighbours' sizes, root mean square relative to FP64's: above that line 0.3-1.3
// (up to 1.6 where a line's own coefficients differ by 2^40, with p = 1; there also
// 1.4 far above it); below, at velocity 1 and h = 1/8: p = 1 3 (diffusion 1e-3), p = 2 6
// and 860 (1e-4 and 1e-6).
bool fx_make_tables(const gbfem_dg_desc& d, int n, FxTables* out) {
  *out = FxTables{};
  if (d.kappa || d.kappa_cell) return false;
  // (a NaN would be lost in the integers; fmaxl drops it too)
  if (!std::isfinite(d.mass) || !std::isfinite(d.velocity[0]) || !std::isfinite(d.velocity[1]) ||
      !std::isfinite(d.velocity[2]))
    return false;
  static const FxBasis bases[4] = {FxBasis(2), FxBasis(3), FxBasis(4), FxBasis(5)};
  const ConstTables1D& ct = bases[n - 2].ct;
  const long double *L = bases[n - 2].L, *dL = bases[n - 2].dL;
  long double h[3], vol = 1.0L;
  for (int k = 0; k < 3; ++k) {
    h[k] = ((long double)d.grid.upper[k] - d.grid.lower[k]) / d.grid.cells[k];
    vol *= h[k];
  }
  const bool adv = d.velocity[0] != 0.0 || d.velocity[1] != 0.0 || d.velocity[2] != 0.0;
  const bool sipg = d.diffusion * d.penalty != 0.0;
  const int bits = fx_coef_bits(adv);
  out->slope = sipg ? 0 : 1;
  for (int k = 0; k < 3; ++k) {
    FxAxis& ax = out->ax[k];
    const long double area = vol / h[k], eps = d.diffusion, b = d.velocity[k];
    const long double A2 = area * eps * 0.5L / h[k];
    const long double C = sipg ? area * eps * d.penalty / h[k] : 1.0L, r = A2 / C;
    if (!std::isfinite(double(r)) || !std::isfinite(double(C))) return false;
    long double cls[2] = {0.0L, 0.0L}, slope = 0.0L, vsum = 0.0L;
    for (int i = 0; i < n; ++i) {
      // without penalty (C = 1) P - v = -r dv is what the flux takes, and it is
      // held as such: P itself would carry it below the digits of v
      const long double p = sipg ? L[i] - r * dL[i] : -dL[i] * (long double)fx_slope_scale(n);
      cls[i & 1] += fabsl(p);
      slope += sipg ? fabsl(r * dL[i]) : 0.0L;
      if (!(fabsl(p) <= 8.0L)) return false;
      ax.v[i] = fx_coef(L[i] / 8.0L, 62);
      ax.P[i] = fx_coef(p / 8.0L, 62);
    }
    if (!(cls[0] <= kFxClassSum && cls[1] <= kFxClassSum && slope <= 2 * kFxClassSum)) return false;
    for (int i = 0; i < n; ++i) vsum += fabsl(L[i]);
    // a line without any face term
    if (d.grid.cells[k] == 1 && !d.weak_dirichlet && (eps != 0.0L || b != 0.0L || (k == 0 && d.mass != 0.0))) return false;
    // inflow and outflow faces: b.n < 0 and > 0
    const int out_side = b > 0.0L ? 1 : 0, in_side = 1 - out_side;
    out->inflow_upper[k] = in_side;
    for (int side = 0; side < 2; ++side) out->couple[k][side] = eps != 0.0L || (b != 0.0L && side == in_side);
    auto sgn = [](int side, int i) { return side == 0 && (i & 1) ? -1.0L : 1.0L; };
    for (int i = 0; i < n; ++i) {
      long double O[kDgMaxN], own = 0.0L, big = 0.0L;
      for (int j = 0; j < n; ++j) {
        O[j] = eps * vol / (h[k] * h[k]) * ct.K1[i][j] - b * vol / h[k] * ct.D1[i][j];
        if (k == 0 && i == j) O[j] += d.mass * vol;
        O[j] += area * fabsl(b) * sgn(out_side, i) * sgn(out_side, j) * L[i] * L[j];
        if (!adv && ((i + j) & 1)) O[j] = 0.0L;
        own += fabsl(O[j]);
        big = fmaxl(big, fabsl(O[j]));
      }
      const long double np = 32.0L * (sipg ? C : A2 / (long double)fx_slope_scale(n)) * L[i], nv = -32.0L * A2 * dL[i];
      const long double a = -32.0L * area * fabsl(b) * sgn(in_side, i) * L[i];
      const long double face = fabsl(np) + fabsl(nv) + fabsl(a);
      big = fmaxl(fmaxl(big, fmaxl(fabsl(np), fabsl(nv))), fmaxl(fabsl(a), fmaxl(own, face) / 2));
      int e = 0;
      if (!std::isfinite(double(big))) return false;
      if (big > 0.0L) frexpl(big, &e);  // big < 2^e
      if (e > kFxRowExpMax || e < -kFxRowExpMax) return false;
      for (int side = 0; side < 2 && big > 0.0L; ++side) {
        const long double w = fabsl(np) * (cls[0] + cls[1]) + (fabsl(nv) + (side == in_side ? fabsl(a) : 0.0L)) * vsum;
        if (out->couple[k][side] && !(w >= 32.0L * 0.009L * (1.0L + vsum) * ldexpl(1.0L, e))) return false;
      }
      // nothing but the mass: an entry has no part in the others of its line
      if (big > 0.0L && !out->couple[k][0] && !out->couple[k][1]) return false;
      for (int j = 0; j < n; ++j) ax.O[i * n + j] = fx_coef(ldexpl(O[j], -e), bits);
      ax.np[i] = fx_coef(ldexpl(np, -e), bits);
      ax.nv[i] = fx_coef(ldexpl(nv, -e), bits);
      ax.a[i] = fx_coef(ldexpl(a, -e), bits);
      ax.ex[i] = (e + 4 - bits) * (1 << 20);
    }
  }
  return true;
}

template <int N, bool ADV, bool SMALL, bool STAGE>
static int fx_launch_brick(const DgArgsT<double>& a, const DgConstTablesT<double>& ct, const FxTables& fx, int z0, int z1,
                           cudaStream_t s, const FxStage& st) {
  using B = FxBrick<N, SMALL>;
  auto kern = dg_fixed_kernel<N, ADV, SMALL, STAGE>;
  constexpr size_t smem = FxSmem<N, B>::BYTES;
  GBFEM_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  const long long nb = (long long)((a.nc[0] + B::X - 1) / B::X) * ((a.nc[1] + B::Y - 1) / B::Y) *
                       ((z1 - z0 + B::Z - 1) / B::Z);
  if (nb <= 0) return GBFEM_OK;
  if (nb > 2147483647LL) return set_error(GBFEM_ERR_INVALID, "dg apply: grid too large");
  kern<<<unsigned(nb), fx_threads<N, B>(), smem, s>>>(a, ct, fx, z0, z1, st);
  GBFEM_CUDA_TRY(cudaGetLastError());
  return GBFEM_OK;
}

template <int N, bool ADV>
static int fx_launch_one(const DgArgsT<double>& a, const DgConstTablesT<double>& ct, const FxTables& fx, int z0, int z1,
                         cudaStream_t s, const FxStage* st) {
  const long long cells = (long long)a.nc[0] * a.nc[1] * (z1 - z0);
  using B = FxBrick<N, false>;
  const bool small = cells < 152LL * B::X * B::Y * B::Z;
  if (st)
    return small ? fx_launch_brick<N, ADV, true, true>(a, ct, fx, z0, z1, s, *st)
                 : fx_launch_brick<N, ADV, false, true>(a, ct, fx, z0, z1, s, *st);
  return small ? fx_launch_brick<N, ADV, true, false>(a, ct, fx, z0, z1, s, FxStage{})
               : fx_launch_brick<N, ADV, false, false>(a, ct, fx, z0, z1, s, FxStage{});
}

// w = A u on the z-planes [z0, z1), with the stage st where one is given.
int dg_fixed_launch(const DgArgsT<double>& a, const DgConstTablesT<double>& ct, const FxTables& fx, int n, int z0,
                    int z1, cudaStream_t s, const FxStage* st) {
#define GBFEM_FX_CASE(NN)                                               \
  if (n == NN)                                                          \
    return a.advect ? fx_launch_one<NN, true>(a, ct, fx, z0, z1, s, st) \
                    : fx_launch_one<NN, false>(a, ct, fx, z0, z1, s, st);
  GBFEM_FX_CASE(2)
  GBFEM_FX_CASE(3)
  GBFEM_FX_CASE(4)
  GBFEM_FX_CASE(5)
#undef GBFEM_FX_CASE
  return set_error(GBFEM_ERR_NOT_IMPLEMENTED, "dg apply: unsupported order");
}

}  // namespace gbfem
