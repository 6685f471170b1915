// The FP64 reaction term of reaction_kernel.cuh for the built-in family, with its
// contractions and exp on the integer pipes (fixed_point.cuh, fx_exp.cuh).
//
// What bounds it: integer issue and barriers; the FP64 kernel it replaces takes
// about 900 FP64 operations per Q2 cell for the contractions and 20 per point for
// exp, one output per thread and step.  Per point three to seven FP64 operations
// remain (to FP64, the function, the weight).  Measured (GB300): 32^3 Q2 (r = -5
// e^u), one mode 130 -> 44 us.
//
// Numbers as in dg_quad_fixed.cuh: a cell's dofs in 60 bits of its largest, every
// contraction renormalised by the cell's largest magnitude; the values at the
// points become FP64, the weighted results again 60-bit integers of the cell's
// largest.  The three contractions along the third axis, the function and the
// first contraction back are one thread's line.  A CTA that meets values it cannot
// hold recomputes its cells with dg_reaction_cells.
#pragma once
#include "dg_quad_fixed.cuh"
#include "fx_exp.cuh"
#include "reaction_kernel.cuh"

namespace gbfem {

struct RxTables {
  FxCoef B[kDgMaxQ * kDgMaxN];   // B[a n + i], S = 2^lB
  FxCoef BT[kDgMaxN * kDgMaxQ];  // L_i(x_a), [i q + a], S = 2^lBT
  int lB, lBT;
  FxExpTables exp;
};

template <int N, int Q>
struct RxShape {
  // Newton's three calls on 32^3 Q2 and 30 x 29 x 30 Q3: 170 and 304 us; with 16 cells
  // at Q2 174, without the register bound (MINB) 331 at Q3, with 256 threads 176 and
  // 305; 9 x 10 x 11 Q2 41 us, 50 with 16 cells.
  static constexpr int CPB = N == 2 ? 32 : (N == 3 || N == 4 ? 8 : 4);
  static constexpr int T = 128, MINB = N == 5 ? 1 : 8;
  static constexpr int N2 = N * N, N3 = N2 * N, Q2 = Q * Q, Q3 = Q2 * Q;
  static constexpr int WS = Q * N2 + Q2 * N;  // t1, t2
  static constexpr size_t BYTES = size_t(CPB) * (N3 + WS) * 8 + size_t(Q3) * 8 + 32 * 8;
};

template <int N, int Q>
__device__ __noinline__ void rx_cell_f64(int mode, const double* u, double* w, double* pts, long long cell,
                                         const ReactTabsT<double>& tb) {
  dg_reaction_cells<double, N, Q, 1, BuiltinReaction>(mode, u, w, pts, cell, cell + 1, tb);
}

// modes as dg_reaction_body
template <int N, int Q, int MODE>
__global__ void __launch_bounds__(RxShape<N, Q>::T, RxShape<N, Q>::MINB) dg_reaction_fixed_kernel(
    const double* __restrict__ u, double* __restrict__ w, double* __restrict__ pts, long long cell_begin,
    long long count, const __grid_constant__ ReactTabsT<double> tb, const __grid_constant__ RxTables rx) {
  using S = RxShape<N, Q>;
  constexpr int CPB = S::CPB, T = S::T, N2 = S::N2, N3 = S::N3, Q2 = S::Q2, Q3 = S::Q3, WS = S::WS;
  extern __shared__ __align__(16) unsigned char rx_smem[];
  long long* const sX = reinterpret_cast<long long*>(rx_smem);
  long long* const work = sX + CPB * N3;
  double* const sW = reinterpret_cast<double*>(work + CPB * WS);
  uint64_t* const sPow = reinterpret_cast<uint64_t*>(sW + Q3);
  __shared__ int sE[CPB], sEv[CPB], slow;
  __shared__ uint32_t mag[4][CPB];
  __shared__ double sScale[CPB];
  const int tid = threadIdx.x;
  const long long c0 = cell_begin + (long long)blockIdx.x * CPB, cend = cell_begin + count;
  if (c0 >= cend) return;
  const int ncell = int(cend - c0 < CPB ? cend - c0 : CPB);
  if (tid == 0) slow = 0;
  for (int c = tid; c < CPB; c += T) {
    sE[c] = sEv[c] = kQxMinExp;
    for (int k = 0; k < 4; ++k) mag[k][c] = 0;
  }
  if (MODE != 2) {
    for (int e = tid; e < Q3; e += T) sW[e] = tb.w[e / Q2] * tb.w[(e / Q) % Q] * tb.w[e % Q] * tb.detK;
    if (tid < 32) sPow[tid] = rx.exp.pow[tid];
  }
  __syncthreads();
  const double* ug = u + c0 * N3;
  constexpr int RX = (CPB * N3 + T - 1) / T;
  double x[RX];
#pragma unroll
  for (int r = 0; r < RX; ++r) {
    const int e = tid + r * T, c = e / N3;
    x[r] = c < ncell ? __ldg(ug + e) : 0.0;
    if (e < CPB * N3) {
      const int ex = int(fx_abs_hi(x[r]) >> 20);
      if (ex > kQxMinExp) atomicMax(&sE[c], ex);
      else if ((fx_bits(x[r]) << 1) != 0) atomicMax(&sE[c], kQxMinExp + 1);
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < RX; ++r) {
    const int e = tid + r * T;
    if (e < CPB * N3) sX[e] = qx_from_double(x[r], sE[e / N3]);
  }
  for (int c = tid; c < ncell; c += T)
    if (sE[c] >= kQxMaxExp || sE[c] == kQxMinExp + 1) slow = 1;
  __syncthreads();
  long long* t1 = work;
  long long* t2 = t1 + Q * N2;
  qx_contract<0, N, N, N, Q, N, CPB, T>(sX, N3, t1, WS, rx.B, nullptr, mag[0]);
  __syncthreads();
  qx_contract<1, Q, N, N, Q, N, CPB, T>(t1, WS, t2, WS, rx.B, mag[0], mag[1]);
  __syncthreads();
  for (int c = tid; c < CPB; c += T) {
    const int s = 60 - 3 * (2 + rx.lB) + qx_room(mag[0][c]) + qx_room(mag[1][c]);
    sScale[c] = fx_pow2((sE[c] + 1 - s) << 20);
  }
  __syncthreads();
  // lines of Q points along the third axis
  constexpr int LINES = CPB * Q2, R = (LINES + T - 1) / T;
  double v[R][Q];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int item = tid + r * T, c = item / Q2, ab = item - c * Q2;
    if (item < LINES) {
      const long long* src = t2 + c * WS + ab * N;
      const int k = qx_room(mag[1][c]);
      FxLimbs l[N];
#pragma unroll
      for (int i = 0; i < N; ++i) l[i] = fx_split((long long)(uint64_t(src[i]) << (k & 63)));
      double* pg = pts + (c0 + (c < ncell ? c : 0)) * Q3 + ab * Q;
      uint32_t m = 0;
      uint64_t any = 0;
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        FxAcc acc = FxAcc::rounded();
#pragma unroll
        for (int i = 0; i < N; ++i) acc.add(l[i], rx.B[q * N + i]);
        const double uq = double(acc.value()) * sScale[c];
        double f;
        if (MODE == 2) {
          f = pg[q] * uq;
        } else {
          const double ex = tb.ce != 0.0 ? fx_exp(uq, rx.exp, sPow) : 0.0;
          if (MODE == 0) {
            f = tb.ce != 0.0 ? tb.ce * ex : 0.0;
            if (tb.c1 != 0.0 || tb.c3 != 0.0) f = tb.c1 * uq + tb.c3 * uq * uq * uq + f;
          } else {
            f = tb.c1 + 3.0 * tb.c3 * uq * uq + (tb.ce != 0.0 ? tb.ce * ex : 0.0);
          }
          f *= sW[ab * Q + q];
        }
        if (MODE == 1) {
          if (c < ncell) pg[q] = f;
        } else {
          v[r][q] = f;
          m = max(m, fx_abs_hi(f));
          any |= fx_bits(f) << 1;
        }
      }
      if (MODE != 1) {
        int ex = int(m >> 20);
        if (ex >= kQxMaxExp || (ex <= kQxMinExp && any)) slow = 1;
        if (ex > kQxMinExp) atomicMax(&sEv[c], ex);
      }
    }
  }
  __syncthreads();
  if (slow) {
    for (int c = 0; c < ncell; ++c) {
      rx_cell_f64<N, Q>(MODE, u, w, pts, c0 + c, tb);
      __syncthreads();
    }
    return;
  }
  if (MODE == 1) return;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int item = tid + r * T, c = item / Q2, ab = item - c * Q2;
    if (item < LINES) {
      FxLimbs l[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) l[q] = fx_split(qx_from_double(v[r][q], sEv[c]));
      long long* dst = t2 + c * WS + ab * N;
      uint32_t m = 0;
#pragma unroll
      for (int i = 0; i < N; ++i) {
        FxAcc acc = FxAcc::rounded();
#pragma unroll
        for (int q = 0; q < Q; ++q) acc.add(l[q], rx.BT[i * Q + q]);
        const long long t = acc.value();
        dst[i] = t;
        m = max(m, qx_mag(t));
      }
      atomicMax(&mag[2][c], m);
    }
  }
  __syncthreads();
  qx_contract<1, Q, Q, N, N, Q, CPB, T>(t2, WS, t1, WS, rx.BT, mag[2], mag[3]);
  __syncthreads();
  for (int item = tid; item < ncell * N2; item += T) {
    const int c = item / N2, jk = item - c * N2;
    const long long* src = t1 + c * WS + jk;
    const int k = qx_room(mag[3][c]);
    FxLimbs l[Q];
#pragma unroll
    for (int a = 0; a < Q; ++a) l[a] = fx_split((long long)(uint64_t(src[a * N2]) << (k & 63)));
    const int s = 60 - 3 * (2 + rx.lBT) + qx_room(mag[2][c]) + k;
    const double scale = fx_pow2((sEv[c] + 1 - s) << 20);
    double* wc = w + (c0 + c) * N3 + jk;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      FxAcc acc = FxAcc::rounded();
#pragma unroll
      for (int a = 0; a < Q; ++a) acc.add(l[a], rx.BT[i * Q + a]);
      wc[i * N2] = fma(double(acc.value()), scale, wc[i * N2]);
    }
  }
}

}  // namespace gbfem
