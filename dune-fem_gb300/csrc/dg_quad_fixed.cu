// The integer-pipe FP64 apply with kappa a DG field: tables, kappa's fixed-point
// point values, launches (dg_quad_fixed.cuh).
#include <cmath>

#include "dg_quad_fixed.cuh"
#include "gbfem_internal.cuh"
#include "operator_impl.hpp"
#include "tables.hpp"

namespace gbfem {

// false: the form or its coefficients are not for the fixed-point kernel
bool qx_make_tables(const gbfem_dg_desc& d, int n, int q, QxTables* out) {
  *out = QxTables{};
  if (!d.kappa || d.mass != 0.0 || !(d.penalty > 0.0) || d.diffusion == 0.0) return false;
  for (int k = 0; k < 3; ++k)
    if (d.velocity[k] != 0.0) return false;
  const Tables1D t = make_tables(n, q);
  long double h[3], vol = 1.0L;
  for (int k = 0; k < 3; ++k) {
    h[k] = ((long double)d.grid.upper[k] - d.grid.lower[k]) / d.grid.cells[k];
    vol *= h[k];
  }
  // B
  long double big = 0.0L, sum = 0.0L;
  for (int a = 0; a < q; ++a) {
    long double r = 0.0L;
    for (int i = 0; i < n; ++i) {
      r += fabsl(t.B[a][i]);
      big = fmaxl(big, fabsl(t.B[a][i]));
    }
    sum = fmaxl(sum, r);
  }
  out->lB = qx_scale(big, sum, 2.5L);
  for (int a = 0; a < q; ++a)
    for (int i = 0; i < n; ++i) {
      out->B[a * n + i] = qx_coef(t.B[a][i], out->lB);
      out->BT[i * q + a] = qx_coef(t.wts[a] * t.B[a][i], 0);
    }
  // Dc and its transposes
  big = sum = 0.0L;
  for (int a = 0; a < q; ++a) {
    long double r = 0.0L;
    for (int b = 0; b < q; ++b) {
      r += fabsl(t.Dc[a][b]);
      big = fmaxl(big, fabsl(t.Dc[a][b]));
    }
    sum = fmaxl(sum, r);
  }
  out->lD = qx_scale(big, sum, 2.5L);
  for (int a = 0; a < q; ++a)
    for (int b = 0; b < q; ++b) out->D[a * q + b] = qx_coef(t.Dc[a][b], out->lD);
  big = sum = 0.0L;
  long double Dt[3][kMaxQ][kMaxQ];
  for (int k = 0; k < 3; ++k) {
    long double most = 0.0L;
    for (int o = 0; o < q; ++o) {
      long double r = 0.0L;
      for (int a = 0; a < q; ++a) {
        Dt[k][o][a] = t.wts[a] * t.Dc[a][o] / t.wts[o] * d.diffusion * vol / (h[k] * h[k]);
        r += fabsl(Dt[k][o][a]);
        big = fmaxl(big, fabsl(Dt[k][o][a]));
      }
      most = fmaxl(most, r);
    }
    sum += most;  // the three axes add up
  }
  if (!std::isfinite(double(sum)) || !(sum > 0.0L)) return false;
  out->lDt = qx_scale(big, sum, 2.5L);
  if (out->lDt > kFxRowExpMax || out->lDt < kQxRowExpMin) return false;
  for (int k = 0; k < 3; ++k)
    for (int o = 0; o < q; ++o)
      for (int a = 0; a < q; ++a) out->Dt[k][o * q + a] = qx_coef(Dt[k][o][a], out->lDt);
  // traces
  const long double r = 1.0L / (2.0L * d.penalty);
  long double sv = 0.0L, sd = 0.0L;
  for (int i = 0; i < n; ++i) {
    sv += fabsl(t.tr[1][i]);
    sd += fabsl(r * t.dtr[1][i]);
  }
  if (!(sd <= sv)) return false;
  out->lT = qx_scale(sv, sv, 2.0L);
  for (int i = 0; i < n; ++i) {
    out->tv[i] = qx_coef(t.tr[1][i], out->lT);
    out->td[i] = qx_coef(r * t.dtr[1][i], out->lT);
  }
  for (int k = 0; k < 3; ++k) {
    const long double area = vol / h[k];
    const long double cv = area * d.diffusion * d.penalty / h[k], cg = -0.5L * area * d.diffusion / h[k];
    for (int i = 0; i < n; ++i) {
      const long double a = cv * t.tr[1][i], b = cg * t.dtr[1][i];
      if (!std::isfinite(double(a)) || !std::isfinite(double(b))) return false;
      const int e = qx_scale(fmaxl(fabsl(a), fabsl(b)), fabsl(a) + fabsl(b), 2.0L);
      if (e > kFxRowExpMax || e < kQxRowExpMin) return false;
      out->lF[k][i] = e;
      out->fv[k][i] = qx_coef(a, e);
      out->fg[k][i] = qx_coef(b, e);
    }
  }
  return true;
}

// One warp per cell: the exponent of kappa's largest point value, then the values.
__global__ void qx_kappa_kernel(const double* __restrict__ kq, const double* __restrict__ kf, long long ncells, int q3,
                                int f6, long long* __restrict__ xq, long long* __restrict__ xf,
                                unsigned short* __restrict__ ke) {
  const int lane = threadIdx.x & 31;
  const long long w0 = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  for (long long c = w0; c < ncells; c += ((long long)gridDim.x * blockDim.x) >> 5) {
    uint32_t m = 0;
    for (int i = lane; i < q3; i += 32) m = max(m, fx_abs_hi(kq[c * q3 + i]));
    for (int i = lane; i < f6; i += 32) m = max(m, fx_abs_hi(kf[c * f6 + i]));
    m = __reduce_max_sync(0xffffffffu, m);
    const int ex = int(m >> 20);
    const bool zero = m == 0;  // (values below 2^-1042 count as zero)
    const bool ok = zero || (ex > 1022 - kQxKappaSpan && ex < 1022 + kQxKappaSpan);
    const int E = zero ? 1022 : ex;
    for (int i = lane; i < q3; i += 32) xq[c * q3 + i] = ok ? fx_from_double(kq[c * q3 + i], E) * 2 : 0;
    for (int i = lane; i < f6; i += 32) xf[c * f6 + i] = ok ? fx_from_double(kf[c * f6 + i], E) * 2 : 0;
    if (lane == 0) ke[c] = (unsigned short)(ok ? E : kQxSlow);
  }
}

static thread_local bool qx_no_memory = false;  // self test

// kappa's fixed-point values from the operator's FP64 point caches.  They take as much
// memory as those (Q3 2.2 KB per cell, Q4 3.5); where there is none left for them the
// operator stays on the FP64 kernel, which needs the FP64 values only.
int qx_kappa(gbfem_operator_s* op) {
  const int q2 = op->q * op->q, q3 = q2 * op->q;
  if (!op->kq_fixed) {
    void* t[3] = {nullptr, nullptr, nullptr};
    const size_t bytes[3] = {size_t(op->ncells) * q3 * 8, size_t(op->ncells) * 6 * q2 * 8, size_t(op->ncells) * 2};
    bool ok = !qx_no_memory;
    for (int i = 0; i < 3 && ok; ++i) ok = cudaMalloc(&t[i], bytes[i]) == cudaSuccess;
    if (!ok) {
      (void)cudaGetLastError();
      for (void* p : t)
        if (p) cudaFree(p);
      op->quad_fixed = false;
      return GBFEM_OK;
    }
    op->kq_fixed = t[0];
    op->kf_fixed = t[1];
    op->ke_fixed = t[2];
  }
  long long blocks = (op->ncells + 7) / 8;
  if (blocks > 152LL * 32) blocks = 152LL * 32;
  qx_kappa_kernel<<<unsigned(blocks), 256>>>(static_cast<const double*>(op->kq_cache),
                                             static_cast<const double*>(op->kf_cache), op->ncells, q3, 6 * q2,
                                             static_cast<long long*>(op->kq_fixed),
                                             static_cast<long long*>(op->kf_fixed),
                                             static_cast<unsigned short*>(op->ke_fixed));
  GBFEM_CUDA_TRY(cudaGetLastError());
  return GBFEM_OK;
}

template <int N, int Q>
static int qx_launch_one(const DgArgsT<double>& a, const DgTablesT<double>& t, const QxTables& qx, const QxArgs& kx,
                         cudaStream_t s) {
  using Sh = QxShape<N, Q>;
  using S = QxSmem<N, Q, Sh::CPB>;
  auto kern = dg_quad_fixed_kernel<N, Q>;
  GBFEM_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(S::BYTES)));
  const long long count = a.cell_count > 0 ? a.cell_count : a.ncells;
  const long long blocks = (count + Sh::CPB - 1) / Sh::CPB;
  if (blocks <= 0) return GBFEM_OK;
  if (blocks > 2147483647LL) return set_error(GBFEM_ERR_INVALID, "dg apply: grid too large");
  kern<<<unsigned(blocks), Sh::T, S::BYTES, s>>>(a, t, qx, kx);
  GBFEM_CUDA_TRY(cudaGetLastError());
  return GBFEM_OK;
}

int dg_quad_fixed_launch(const gbfem_operator_s* op, const DgArgsT<double>& a, cudaStream_t s) {
  QxArgs kx;
  kx.kq = static_cast<const long long*>(op->kq_fixed);
  kx.kf = static_cast<const long long*>(op->kf_fixed);
  kx.ke = static_cast<const unsigned short*>(op->ke_fixed);
#define GBFEM_QX_CASE(NN, QQ) \
  if (op->n == NN && op->q == QQ) return qx_launch_one<NN, QQ>(a, op->tab64, op->qx, kx, s);
  GBFEM_QX_CASE(2, 2)
  GBFEM_QX_CASE(2, 3)
  GBFEM_QX_CASE(3, 3)
  GBFEM_QX_CASE(3, 4)
  GBFEM_QX_CASE(4, 4)
  GBFEM_QX_CASE(4, 5)
  GBFEM_QX_CASE(5, 5)
  GBFEM_QX_CASE(5, 6)
#undef GBFEM_QX_CASE
  return set_error(GBFEM_ERR_NOT_IMPLEMENTED, "dg apply: unsupported (p, q)");
}

}  // namespace gbfem

extern "C" int gbfem_selftest_no_fixed_memory(int on) {
  gbfem::qx_no_memory = on != 0;
  return GBFEM_OK;
}
