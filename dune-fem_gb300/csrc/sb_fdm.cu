// Scaled shared-block Jacobi by fast diagonalisation.
//
// The preconditioner z_c = H_t(c)^-1 r_c / kappa_c of a cellwise-kappa DG
// operator (solver.cu): H_t, the diagonal block of the kappa = 1 operator for a
// cell of boundary type t, is a Kronecker sum over the axes,
//     H_t = A_x (+) A_y (+) A_z,   A_d = |K|/h_d^2 eps K1 + the cell's own part of
//                                  its two faces normal to d,
// because the tangential face mass matrices of the orthonormal basis are the
// identity.  With A_d = V_d L_d V_d^T (n x n, symmetric),
//     H_t^-1 = (V_x x V_y x V_z) (L_x + L_y + L_z)^-1 (V_x x V_y x V_z)^T
// (Lynch, Rice & Thomas, Numer. Math. 6 (1964)): 6 n multiply-adds per dof and
// one division instead of the n^3 of the dense inverse.  Only V_d and L_d of the
// at most four boundary types per axis are kept.
//
// What bounds it: 8 bytes per dof of traffic (HBM), then shared-memory passes.
// Per cell n threads; thread i owns the plane i0 = i (contiguous dofs) for the y
// and z contractions in registers, and the plane i1 = i for the x contraction,
// the division and the x contraction back, so the cell goes through shared
// memory twice, besides the staging of r and z that makes their accesses
// coalesced.  Interior cells, in warps that hold nothing else, take V_d from
// the kernel parameters (uniform operands); other warps read each cell's own
// from shared memory.  Measured (GB300), tcgen05 3xTF32 tiles of the dense
// inverse before, this kernel after: 48^3 Q4 94 -> 44 us, 64^3 Q3 116 -> 41; error
// against 64 bits 9.1e-7 -> 1.4e-7 and 3.8e-7 -> 1.4e-7.
//
// For p = 3 and 4 only: with p <= 2 the dense products are FP32 sums of 27 terms at
// most, error 8e-8 where six rounded contractions have 2.7e-7 (61 x 50 x 58 Q2: 80 us
// against 16).
#include <cuda_runtime.h>
#include <cmath>
#include <new>

#include "gbfem_internal.cuh"
#include "operator_impl.hpp"
#include "solver_impl.hpp"
#include "tables.hpp"

namespace gbfem {

// Boundary types of an axis: bit 0 a domain boundary below the cell, bit 1 above.
struct SbFdmTables {
  float V[3][4][kDgMaxN * kDgMaxN];  // V[d][type][i n + k]: component i of eigenvector k
  float L[3][4][kDgMaxN];
};

struct SbFdmArgs {
  const float *kcell, *r;
  float* z;
  long long ncells;
  int nc[3], periodic[3];
};

template <int N>
struct SbFdm {
  static constexpr int N2 = N * N, N3 = N2 * N;
  // cells per CTA (64^3 Q3: 41.3 us with 40 cells, 43.1 with 32, 47.1 with 64; 48^3
  // Q4: 43.6 with 32, 52.7 with 64)
  static constexpr int CPB = N == 4 ? 40 : 32;
  static constexpr int T = CPB * N;
  // plane stride in shared memory: 16-byte rows that spread over the banks for
  // n = 4, the odd stride of n = 5 as it is
  static constexpr int PL = N == 4 ? 20 : N2;
  static constexpr int CS = N * PL;
  static_assert(T % 32 == 0, "whole warps");
};

// y[.., k, ..] = sum_i M[i][k] x[.., i, ..] (FWD, M = V) or sum_i M[k][i] x (back)
// along the first (AX 0) or second axis of an n x n plane; M from `m`
template <int N, int AX, bool FWD>
__device__ __forceinline__ void sb_plane(float (&x)[N * N], const float* __restrict__ m) {
#pragma unroll
  for (int l = 0; l < N; ++l) {
    float v[N];
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = x[AX == 0 ? i * N + l : l * N + i];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      float a = 0.f;
#pragma unroll
      for (int i = 0; i < N; ++i) a = fmaf(FWD ? m[i * N + k] : m[k * N + i], v[i], a);
      x[AX == 0 ? k * N + l : l * N + k] = a;
    }
  }
}

template <int N>
__global__ void __launch_bounds__(SbFdm<N>::T) k_sb_fdm(const __grid_constant__ SbFdmArgs g,
                                                        const __grid_constant__ SbFdmTables tabs) {
  using S = SbFdm<N>;
  constexpr int N2 = S::N2, N3 = S::N3, PL = S::PL, CS = S::CS, T = S::T;
  __shared__ __align__(16) float buf[S::CPB * CS];
  __shared__ float sV[3 * 4 * N2];
  __shared__ float sL[3 * 4 * N];
  __shared__ float sInv[N3];  // 1 / (Lx + Ly + Lz) of an interior cell, [i0][i1][i2]
  const int tid = threadIdx.x;
  const long long c0 = (long long)blockIdx.x * S::CPB;
  const int ncell = int(g.ncells - c0 < S::CPB ? g.ncells - c0 : S::CPB);
  for (int e = tid; e < 12 * N2; e += T) sV[e] = tabs.V[e / (4 * N2)][(e / N2) % 4][e % N2];
  for (int e = tid; e < 12 * N; e += T) sL[e] = tabs.L[e / (4 * N)][(e / N) % 4][e % N];
  for (int e = tid; e < N3; e += T)
    sInv[e] = 1.0f / (tabs.L[0][0][e / N2] + tabs.L[1][0][(e / N) % N] + tabs.L[2][0][e % N]);
  // r in, coalesced, into planes of stride PL: 16 bytes at a time where the
  // vectors and the chunk allow it (a plane is a multiple of 16 bytes, or the
  // planes are contiguous)
  const float* rg = g.r + c0 * N3;
  float* zg = g.z + c0 * N3;
  const int total = ncell * N3;
  const bool wide =
      ((reinterpret_cast<uintptr_t>(rg) | reinterpret_cast<uintptr_t>(zg)) & 15) == 0 && total % 4 == 0;
  auto place = [](int e) { return N2 == PL ? e : (e / N2) * PL + e % N2; };
  constexpr int K4 = (N2 + 3) / 4;
  if (wide) {
    float4 t[K4];
#pragma unroll
    for (int j = 0; j < K4; ++j)
      if (4 * (tid + j * T) < total) t[j] = __ldg(reinterpret_cast<const float4*>(rg) + tid + j * T);
#pragma unroll
    for (int j = 0; j < K4; ++j)
      if (4 * (tid + j * T) < total) *reinterpret_cast<float4*>(buf + place(4 * (tid + j * T))) = t[j];
  } else {
    for (int e = tid; e < total; e += T) buf[place(e)] = __ldg(rg + e);
  }
  // this thread's cell and its type on each axis
  const int lc = tid / N, i = tid - lc * N;
  const bool on = lc < ncell;
  const long long cell = c0 + (on ? lc : 0);
  const int nxy = g.nc[0] * g.nc[1];
  const int cz = int(cell / nxy), rem = int(cell - (long long)cz * nxy), cy = rem / g.nc[0];
  const int pos[3] = {rem - cy * g.nc[0], cy, cz};
  int type[3];
  bool inner[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    type[d] = g.periodic[d] ? 0 : (pos[d] == 0 ? 1 : 0) | (pos[d] == g.nc[d] - 1 ? 2 : 0);
    inner[d] = __all_sync(0xffffffffu, type[d] == 0);
  }
  const float scale = 1.0f / __ldg(g.kcell + cell);
  __syncthreads();
  float x[N2];
  float* const mine = buf + lc * CS + i * PL;  // plane i0 = i
  auto read_plane = [&]() {
    if constexpr (N2 % 4 == 0) {
#pragma unroll
      for (int q = 0; q < N2 / 4; ++q) {
        const float4 t = *reinterpret_cast<const float4*>(mine + 4 * q);
        x[4 * q] = t.x;
        x[4 * q + 1] = t.y;
        x[4 * q + 2] = t.z;
        x[4 * q + 3] = t.w;
      }
    } else {
#pragma unroll
      for (int q = 0; q < N2; ++q) x[q] = mine[q];
    }
  };
  auto write_plane = [&]() {
    if constexpr (N2 % 4 == 0) {
#pragma unroll
      for (int q = 0; q < N2 / 4; ++q)
        *reinterpret_cast<float4*>(mine + 4 * q) = make_float4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
    } else {
#pragma unroll
      for (int q = 0; q < N2; ++q) mine[q] = x[q];
    }
  };
  // [i1][i2] of plane i0: z, then y
  read_plane();
  if (inner[2]) sb_plane<N, 1, true>(x, tabs.V[2][0]);
  else sb_plane<N, 1, true>(x, sV + (8 + type[2]) * N2);
  if (inner[1]) sb_plane<N, 0, true>(x, tabs.V[1][0]);
  else sb_plane<N, 0, true>(x, sV + (4 + type[1]) * N2);
  write_plane();
  __syncthreads();
  // [i0][i2] of plane i1 = i: x, the division, x back
  float* const across = buf + lc * CS + i * N;
#pragma unroll
  for (int q = 0; q < N2; ++q) x[q] = across[(q / N) * PL + q % N];
  if (inner[0]) sb_plane<N, 0, true>(x, tabs.V[0][0]);
  else sb_plane<N, 0, true>(x, sV + type[0] * N2);
  if (inner[0] && inner[1] && inner[2]) {
#pragma unroll
    for (int q = 0; q < N2; ++q) x[q] *= scale * sInv[(q / N) * N2 + i * N + q % N];
  } else {
    const float ly = sL[(4 + type[1]) * N + i];
#pragma unroll
    for (int a = 0; a < N; ++a) {
      const float lxy = sL[type[0] * N + a] + ly;
#pragma unroll
      for (int b = 0; b < N; ++b) x[a * N + b] *= scale / (lxy + sL[(8 + type[2]) * N + b]);
    }
  }
  if (inner[0]) sb_plane<N, 0, false>(x, tabs.V[0][0]);
  else sb_plane<N, 0, false>(x, sV + type[0] * N2);
#pragma unroll
  for (int q = 0; q < N2; ++q) across[(q / N) * PL + q % N] = x[q];
  __syncthreads();
  read_plane();
  if (inner[1]) sb_plane<N, 0, false>(x, tabs.V[1][0]);
  else sb_plane<N, 0, false>(x, sV + (4 + type[1]) * N2);
  if (inner[2]) sb_plane<N, 1, false>(x, tabs.V[2][0]);
  else sb_plane<N, 1, false>(x, sV + (8 + type[2]) * N2);
  write_plane();
  __syncthreads();
  if (wide) {
#pragma unroll
    for (int j = 0; j < K4; ++j)
      if (4 * (tid + j * T) < total)
        reinterpret_cast<float4*>(zg)[tid + j * T] = *reinterpret_cast<const float4*>(buf + place(4 * (tid + j * T)));
  } else {
    for (int e = tid; e < total; e += T) zg[e] = buf[place(e)];
  }
}

// Eigenvectors (columns of V) and values of the symmetric n x n matrix a, by
// cyclic Jacobi rotations (Golub & Van Loan, section 8.5).  In double: the tables are
// FP32, and extended precision is slow on hosts that emulate it.
static void sb_eigen(int n, double (&a)[kDgMaxN][kDgMaxN], double (&V)[kDgMaxN][kDgMaxN]) {
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < n; ++j) V[i][j] = i == j ? 1.0 : 0.0;
  for (int sweep = 0; sweep < 30; ++sweep) {
    double off = 0.0, dia = 0.0;
    for (int i = 0; i < n; ++i)
      for (int j = 0; j < n; ++j) (i == j ? dia : off) += a[i][j] * a[i][j];
    if (!(off > 1e-30 * dia)) break;
    for (int p = 0; p < n; ++p)
      for (int q = p + 1; q < n; ++q) {
        if (a[p][q] == 0.0) continue;
        const double tau = (a[q][q] - a[p][p]) / (2.0 * a[p][q]);
        const double t = (tau >= 0.0 ? 1.0 : -1.0) / (std::fabs(tau) + std::sqrt(1.0 + tau * tau));
        const double c = 1.0 / std::sqrt(1.0 + t * t), s = t * c;
        for (int k = 0; k < n; ++k) {
          const double x = a[k][p], y = a[k][q];
          a[k][p] = c * x - s * y;
          a[k][q] = s * x + c * y;
        }
        for (int k = 0; k < n; ++k) {
          const double x = a[p][k], y = a[q][k];
          a[p][k] = c * x - s * y;
          a[q][k] = s * x + c * y;
        }
        for (int k = 0; k < n; ++k) {
          const double x = V[k][p], y = V[k][q];
          V[k][p] = c * x - s * y;
          V[k][q] = s * x + c * y;
        }
      }
  }
}

// The tables, in pc->sb_fdm; left null for p <= 2 (above) and where a block is not
// positive definite: a penalty too small, whose eigenvalues' sums cancel (penalty 0,
// Q3: error 1e-5), or one cell without a boundary term, where the division gives
// infinities and the dense inverse of the rounded block does not.  Positive definite
// blocks keep 2e-7 up to condition numbers of 1e6.
int sb_fdm_setup(gbfem_preconditioner_s* pc) {
  const gbfem_operator_s* op = pc->sor_op;
  const gbfem_dg_desc& d = op->dg;
  const int n = op->n;
  if (n < 4) return GBFEM_OK;
  const ConstTables1D ct = make_const_tables(n);
  auto* t = new (std::nothrow) SbFdmTables{};
  if (!t) return set_error(GBFEM_ERR_INVALID, "out of host memory");
  long double h[3], vol = 1.0L, v[2][kDgMaxN], g[2][kDgMaxN];
  for (int k = 0; k < 3; ++k) {
    h[k] = ((long double)d.grid.upper[k] - d.grid.lower[k]) / d.grid.cells[k];
    vol *= h[k];
  }
  for (int s = 0; s < 2; ++s)
    for (int i = 0; i < n; ++i) legendre01(i, (long double)s, &v[s][i], &g[s][i]);
  for (int k = 0; k < 3; ++k)
    for (int type = 0; type < 4; ++type) {
      const long double eps = d.diffusion, area = vol / h[k], sigma = d.penalty / h[k];
      double a[kDgMaxN][kDgMaxN], V[kDgMaxN][kDgMaxN];
      for (int i = 0; i < n; ++i)
        for (int j = 0; j < n; ++j) {
          long double m = eps * vol / (h[k] * h[k]) * ct.K1[i][j];
          for (int s = 0; s < 2; ++s) {
            const bool edge = (type >> s) & 1;
            if (edge && !d.weak_dirichlet) continue;
            // sigma u v - w (dn u v + u dn v), w = 1/2 of the average, 1 on the boundary
            const long double w = edge ? 1.0L : 0.5L, sg = s ? 1.0L / h[k] : -1.0L / h[k];
            m += eps * area * (sigma * v[s][i] * v[s][j] - w * sg * (g[s][i] * v[s][j] + v[s][i] * g[s][j]));
          }
          a[i][j] = double(m);
        }
      sb_eigen(n, a, V);
      for (int i = 0; i < n; ++i) {
        t->L[k][type][i] = float(a[i][i]);
        for (int j = 0; j < n; ++j) t->V[k][type][i * n + j] = float(V[i][j]);
      }
    }
  // the boundary types that occur on an axis
  auto occurs = [&](int k, int type) {
    const int nc = d.grid.cells[k];
    if (d.grid.periodic[k]) return type == 0;
    return nc == 1 ? type == 3 : (type == 1 || type == 2 || (type == 0 && nc > 2));
  };
  bool regular = true;
  for (int e = 0; e < 64; ++e) {
    const int ty[3] = {e & 3, (e >> 2) & 3, e >> 4};
    if (!occurs(0, ty[0]) || !occurs(1, ty[1]) || !occurs(2, ty[2])) continue;
    float least = INFINITY, most = 0.f;
    for (int l = 0; l < n * n * n; ++l) {
      const float v = t->L[0][ty[0]][l / (n * n)] + t->L[1][ty[1]][(l / n) % n] + t->L[2][ty[2]][l % n];
      least = fminf(least, v);
      most = fmaxf(most, v);
    }
    regular = regular && least > 1e-7f * most;
  }
  if (regular) pc->sb_fdm = t;
  else delete t;
  return GBFEM_OK;
}

void sb_fdm_destroy(void* t) { delete static_cast<SbFdmTables*>(t); }

template <int N>
static int sb_fdm_launch(const SbFdmArgs& a, const SbFdmTables& t, cudaStream_t s) {
  using S = SbFdm<N>;
  const long long grid = (a.ncells + S::CPB - 1) / S::CPB;
  if (grid <= 0) return GBFEM_OK;
  if (grid > 2147483647LL) return set_error(GBFEM_ERR_INVALID, "scaled block Jacobi: grid too large");
  k_sb_fdm<N><<<unsigned(grid), S::T, 0, s>>>(a, t);
  GBFEM_CUDA_TRY(cudaGetLastError());
  return GBFEM_OK;
}

int sb_fdm_apply(const gbfem_preconditioner_s* pc, const float* r, float* z, cudaStream_t s) {
  const gbfem_operator_s* op = pc->sor_op;
  SbFdmArgs a{};
  a.r = r;
  a.z = z;
  a.kcell = static_cast<const float*>(op->dg.kappa_cell);
  a.ncells = op->ncells;
  for (int d = 0; d < 3; ++d) {
    a.nc[d] = op->dg.grid.cells[d];
    a.periodic[d] = op->dg.grid.periodic[d];
  }
  const SbFdmTables& t = *static_cast<const SbFdmTables*>(pc->sb_fdm);
  switch (op->n) {
    case 4: return sb_fdm_launch<4>(a, t, s);
    case 5: return sb_fdm_launch<5>(a, t, s);
  }
  return set_error(GBFEM_ERR_NOT_IMPLEMENTED, "scaled block Jacobi: unsupported order");
}

}  // namespace gbfem
