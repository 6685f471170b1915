// One-kernel FP64 apply of the constant-coefficient closed form, computed in
// block fixed point on the integer pipes (fixed_point.cuh; the algebra is
// that of dg_const_kernel.cuh, whose two FP64-pipe kernels this replaces
// where the coefficients allow it).
//
// What bounds it: integer issue and its latencies.  Per dof and axis about 150
// instructions (conversions in and out, alignment, 15-18 products of three
// multiply-adds) take the place of 7.5 FP64 ones, which at 2 per clock and SM
// cost 3.75 clocks; two FP64 instructions remain, the conversion of the result
// and its addition (the FP64 pipe is half busy).  The traces never leave the
// SM.  Measured (GB300, two-kernel form before, this kernel after): 64^3 Q3
// 822 -> 295 us, 80^3 Q2 with advection 1050 -> 315 us.
//
// A line is the n coefficients of a cell along one axis.  With the line's own
// coefficients x, its face traces (v, P) and those of its two neighbours on
// the shared faces, the operator along the axis is
//     y_i = sum_j O_ij x_j + np_i (dP1 + s_i dP0) + nv_i (J1 + s_i J0) + a_i v_in,
// s_i = (-1)^i, dP = P - P_neighbour and J = v - v_neighbour on the upper (1)
// and lower (0) face: O is M_d plus the upwind flux through the outflow face
// (without advection its entries with i+j odd vanish), a_i couples the inflow
// neighbour.  The differences keep what they are for: a constant gives exactly
// zero.  At a domain boundary with weak u = 0, J = 2 v and dP = 2 P - v (2 P
// where am1 = -1) turn the interior flux into the boundary flux; without a
// boundary term both are zero, and there is no inflow.  Without a penalty
// (am1 = -1) the second trace is P - v, the scaled slope, itself.
//
// Exponents: each line has its own (its largest coefficient), its traces carry
// it, and the line's result is formed at the largest of its own and its two
// neighbours', the lines that enter it with weight (fx_make_tables refuses the
// operators where one hardly does).  So an entry is as exact relative to these lines
// as an FP64 sum is, whatever the rest of the cell holds: one unit of a trace is
// 2^-56 of the line's binade, where an FP64 trace rounds at 2^-53 of its value.
// Lines that fixed point cannot hold (infinities, NaN, magnitudes outside
// 2^-822 .. 2^777) are computed by the FP64 formulas instead, line by line.
//
// Layout of the work: a CTA owns a brick of cells and goes through the axes.
// A. every thread takes its lines of the brick (one lane per line: n loads),
//    converts them, computes the own part O x and the four traces, and stores
//    the traces and the line's exponent in shared memory; the lines of the
//    brick's face neighbours outside it get the one face's traces the same
//    way.
// B. every thread reads the neighbours' traces of its lines, adds their part
//    and converts the n results to FP64.  Results accumulate over the axes
//    in shared memory (x starts, y adds, z adds and stores w).
// Every output is one thread's fixed-order sum of its own line's data:
// deterministic, and the same whatever brick or slab a cell lands in.
#pragma once
#include <cuda_runtime.h>
#include <type_traits>

#include "dg_const_kernel.cuh"
#include "dg_fixed_tables.hpp"

namespace gbfem {

// Cells per brick and cell layers per pass of the CTA: the threads cover all
// lines of L layers of the brick (X Y L n^2 threads, in whole warps) and take
// Z / L of them each, so that a thread's lines differ in z only.  Small CTAs
// hide each other's barriers and loads better than large ones, whose halo is
// smaller: 64^3 Q3 takes 295 us with 4 x 4 x 2 cells and 5 CTAs per SM, 306 with 4,
// 326 with 4 x 4 x 1, 382 with 4 x 4 x 4, 317 with 4 x 2 x 2 in one pass.  SMALL: grids of less than one
// full brick per SM, where the time is that of one CTA (6 x 5 x 7 Q2: 11.3 us a
// call against 20.4 with full bricks).
template <int N, bool SMALL>
struct FxBrick;
template <>
struct FxBrick<2, false> { static constexpr int X = 8, Y = 4, Z = 4, L = 2, MINB = 4; };
template <>
struct FxBrick<3, false> { static constexpr int X = 4, Y = 4, Z = 4, L = 2, MINB = 3; };
template <>
struct FxBrick<4, false> { static constexpr int X = 4, Y = 4, Z = 2, L = 1, MINB = 5; };
template <>
struct FxBrick<5, false> { static constexpr int X = 4, Y = 2, Z = 2, L = 1, MINB = 4; };
template <>
struct FxBrick<2, true> { static constexpr int X = 4, Y = 4, Z = 2, L = 2, MINB = 2; };
template <>
struct FxBrick<3, true> { static constexpr int X = 4, Y = 2, Z = 2, L = 2, MINB = 2; };
template <>
struct FxBrick<4, true> { static constexpr int X = 2, Y = 2, Z = 2, L = 2, MINB = 2; };
template <>
struct FxBrick<5, true> { static constexpr int X = 2, Y = 2, Z = 2, L = 2, MINB = 2; };
template <int N, class B>
constexpr int fx_threads() { return (B::X * B::Y * B::L * N * N + 31) / 32 * 32; }

struct FxPair {
  long long v, p;
};

template <int N, class B>
struct FxSmem {
  static constexpr int N2 = N * N, N3 = N2 * N, CELLS = B::X * B::Y * B::Z;
  static constexpr int SX = (B::X + 1) * B::Y * B::Z, SY = B::X * (B::Y + 1) * B::Z, SZ = B::X * B::Y * (B::Z + 1);
  static constexpr int SLOTS = SX > SY ? (SX > SZ ? SX : SZ) : (SY > SZ ? SY : SZ);
  static constexpr int LINES = SLOTS * N2;
  // [2 sides][slot][line] trace pairs and exponents, results
  static constexpr size_t BYTES = size_t(2) * LINES * 16 + size_t(CELLS) * N3 * 8 + size_t(2) * LINES * 2;
};

// Place of result i of line jk along axis D in the cell's block of shared
// memory: the local index, XOR-swizzled for n = 4 so that the y lines of a
// warp fall into distinct banks.
template <int N, int D>
__device__ __forceinline__ int fx_res_off(int jk, int i) {
  const int j = jk / N, k = jk - j * N;
  const int i0 = D == 0 ? i : j, i1 = D == 0 ? j : (D == 1 ? i : k), i2 = D == 2 ? i : k;
  if (N == 4) return i0 * 16 + ((i1 * 4 + i2) ^ (i0 * 4));
  return (i0 * N + i1) * N + i2;
}
// The n coefficients of a line; a z line is contiguous and goes out in 16-byte
// loads where the vector allows it.
template <int N, int D>
__device__ __forceinline__ void fx_load_line(const double* __restrict__ xs, bool wide, double (&x)[N]) {
  constexpr int STR = D == 0 ? N * N : (D == 1 ? N : 1);
  if (D == 2 && N % 2 == 0 && wide) {
#pragma unroll
    for (int i = 0; i < N; i += 2) {
      const double2 t = __ldg(reinterpret_cast<const double2*>(xs + i));
      x[i] = t.x;
      x[i + 1 < N ? i + 1 : i] = t.y;
    }
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = __ldg(xs + i * STR);
  }
}
template <int N, int D>
__device__ __forceinline__ int fx_line_base(int jk) {
  const int j = jk / N, k = jk - j * N;
  return D == 0 ? jk : (D == 1 ? j * N * N + k : j * N * N + k * N);
}

constexpr int kFxSlow = 0xFFFF;  // exponent mark: the traces are FP64 values

// Exponent of a line, or kFxSlow.
template <int N>
__device__ __forceinline__ int fx_line_exp(const double (&x)[N]) {
  uint32_t m = 0;
#pragma unroll
  for (int i = 0; i < N; ++i) m = max(m, fx_abs_hi(x[i]));
  if (m - (uint32_t(kFxMinExp) << 20) < (uint32_t(kFxMaxExp - kFxMinExp) << 20)) return int(m >> 20);
  uint64_t any = 0;
#pragma unroll
  for (int i = 0; i < N; ++i) any |= fx_bits(x[i]) << 1;
  return any ? kFxSlow : kFxMinExp;  // an all-zero line has X = 0 at any exponent
}

// both faces' traces (v, P) by dg_trace_kernel's FP64 formulas
template <int N, int D>
__device__ __forceinline__ void fx_traces_f64(const double (&x)[N], const DgConstTablesT<double>& ct, double (&t)[4]) {
  double ev = x[0], od = 0.0, pe = x[0], po = 0.0;
#pragma unroll
  for (int i = 1; i < N; ++i) {
    if (i & 1) {
      od = fma(ct.tr[N + i], x[i], od);
      po = fma(ct.pc[D][i], x[i], po);
    } else {
      ev = fma(ct.tr[N + i], x[i], ev);
      pe = fma(ct.pc[D][i], x[i], pe);
    }
  }
  t[0] = ev - od;
  t[1] = pe - po;
  t[2] = ev + od;
  t[3] = pe + po;
}

// A line's even and odd partial sums of both traces in fixed point: the
// traces are (ev + od, pe + po) on the upper face, (ev - od, pe - po) on the
// lower one.
struct FxSums {
  long long ev, od, pe, po;
};
template <int N>
__device__ __forceinline__ FxSums fx_trace_sums(const FxLimbs (&x)[N], const FxAxis& ax) {
  FxAcc ev, od, pe, po;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    if (i & 1) {
      od.add(x[i], ax.v[i]);
      po.add(x[i], ax.P[i]);
    } else {
      ev.add(x[i], ax.v[i]);
      pe.add(x[i], ax.P[i]);
    }
  }
  return FxSums{ev.value(), od.value(), pe.value(), po.value()};
}

// The line by the FP64 formulas of dg_const_kernel: for the lines that fixed
// point cannot hold.  eu, el: the exponents of the neighbours' traces.
template <int N, bool ADV, int D>
__device__ __noinline__ void fx_line_f64(const DgArgsT<double>& args, const DgConstTablesT<double>& ct,
                                         const double* xs, bool has_up, bool has_lo, FxPair up, int eu, FxPair lo,
                                         int el, bool slope, double* y) {
  constexpr int STR = D == 0 ? N * N : (D == 1 ? N : 1);
  double x[N], own[4];
#pragma unroll
  for (int i = 0; i < N; ++i) x[i] = __ldg(xs + i * STR);
  fx_traces_f64<N, D>(x, ct, own);
  double Val[2], G[2];
  for (int s = 0; s < 2; ++s) {
    const double vm = own[2 * s], pm = own[2 * s + 1];
    const bool nb = s ? has_up : has_lo;
    const int e = s ? eu : el;
    const long long tv = s ? up.v : lo.v, tp = s ? up.p : lo.p;
    double val = 0.0, grad = 0.0;
    const double bn = s ? args.b[D] : -args.b[D];
    if (nb) {
      const double vp = e == kFxSlow ? __longlong_as_double(tv) : ldexp(double(tv), e - 1022 - kFxTraceExp);
      double pp = e == kFxSlow ? __longlong_as_double(tp) : ldexp(double(tp), e - 1022 - kFxTraceExp);
      if (e != kFxSlow && slope) pp = fma(ct.A2[D] / fx_slope_scale(N), pp, vp);
      const double J = vm - vp;
      val = pm - pp;
      if (ct.am1 != 0.0) val = fma(ct.am1, J, val);
      grad = J;
      if (ADV) val = fma(ct.adv[2 * D + s], bn >= 0.0 ? vm : vp, val);
    } else {
      if (args.weak_dirichlet) {
        val = fma(ct.am2, vm, pm + pm);
        grad = vm + vm;
      }
      if (ADV && bn > 0.0) val = fma(ct.adv[2 * D + s], vm, val);
    }
    Val[s] = val;
    G[s] = grad;
  }
  const double vs = Val[1] + Val[0], vd = Val[1] - Val[0], gs = G[1] + G[0], gd = G[1] - G[0];
  const bool has_mass = ct.M[0][0] != 0.0;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    double acc = 0.0;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const bool k1 = i != 0 && j != 0 && !((i + j) & 1);
      const bool d1 = j < i && ((i + j) & 1);
      if (k1 || (D == 0 && i == 0 && j == 0 && has_mass) || (ADV && d1)) acc = fma(ct.M[D][i * N + j], x[j], acc);
    }
    acc = fma(ct.etr[D][i], (i & 1) ? vd : vs, acc);
    if (i > 0) acc = fma(ct.edtr[D][i], (i & 1) ? gd : gs, acc);
    y[i] = acc;
  }
}

// STAGE: a Runge-Kutta stage goes with the apply, st.y = st.u + sum_j st.a[j] w_j over
// the earlier results st.w[j] and, last, this one, which is stored only if args.w is
// given (st.y may be st.u, not args.u).  The FP64 pipe has room for its one to three
// multiply-adds per dof and the memory system for its vectors: three applies and three
// passes over the vectors, 1158 us at 80^3 Q2, become 1090.
template <int N, bool ADV, bool SMALL, bool STAGE>
__global__ void __launch_bounds__(fx_threads<N, FxBrick<N, SMALL>>(), FxBrick<N, SMALL>::MINB)
    dg_fixed_kernel(const __grid_constant__ DgArgsT<double> args, const __grid_constant__ DgConstTablesT<double> ct,
                    const __grid_constant__ FxTables fx, int z0, int z1, const __grid_constant__ FxStage st) {
  using B = FxBrick<N, SMALL>;
  using S = FxSmem<N, B>;
  constexpr int N2 = N * N, N3 = N2 * N;
  constexpr int T = fx_threads<N, B>(), CELLS = S::CELLS, R = B::Z / B::L;
  extern __shared__ __align__(16) unsigned char fx_smem[];
  FxPair* const tr = reinterpret_cast<FxPair*>(fx_smem);  // [side][slot][line]
  double* const res = reinterpret_cast<double*>(tr + 2 * S::LINES);
  unsigned short* const exps = reinterpret_cast<unsigned short*>(res + CELLS * N3);  // [side][slot][line]
  const int tid = threadIdx.x;
  const int nbx = (args.nc[0] + B::X - 1) / B::X, nby = (args.nc[1] + B::Y - 1) / B::Y;
  int o[3], e[3];
  {
    const int b = blockIdx.x, bz = b / (nbx * nby), rem = b - bz * nbx * nby, by = rem / nbx;
    o[0] = (rem - by * nbx) * B::X;
    o[1] = by * B::Y;
    o[2] = z0 + bz * B::Z;
    e[0] = min(B::X, args.nc[0] - o[0]);
    e[1] = min(B::Y, args.nc[1] - o[1]);
    e[2] = min(B::Z, z1 - o[2]);
  }
  const int nx = args.nc[0];
  const long long nxy = (long long)nx * args.nc[1];
  // this thread's lines: cells (lx, ly, lz + r L) of the brick, line jk
  const int c0 = tid / N2, jk = tid - c0 * N2;
  const int lx = c0 % B::X, ly = (c0 / B::X) % B::Y, lz = c0 / (B::X * B::Y);
  const int rows = lz < B::L && lx < e[0] && ly < e[1] ? (e[2] - lz + B::L - 1) / B::L : 0;  // r < rows
  const long long first = ((o[0] + lx) + (long long)nx * (o[1] + ly) + nxy * (o[2] + lz)) * N3;
  const long long zstep = nxy * (B::L * N3);
  const bool wide = ((reinterpret_cast<uintptr_t>(args.u) | reinterpret_cast<uintptr_t>(args.w)) & 15) == 0;

  auto axis = [&](auto dc) {
    constexpr int D = decltype(dc)::value;
    constexpr int A = D == 0 ? 1 : 0, C = D == 2 ? 1 : 2;  // the other axes
    constexpr int BD = D == 0 ? B::X : (D == 1 ? B::Y : B::Z);
    constexpr int BA = A == 0 ? B::X : B::Y, BC = C == 1 ? B::Y : B::Z;
    constexpr int ZSLOT = (D == 2 ? 1 : (BD + 1) * BA) * B::L * N2;  // slot step of r
    const FxAxis& ax = fx.ax[D];
    const double* const xs = args.u + first + fx_line_base<N, D>(jk);
    auto slot = [&](int f, int la, int lc) { return (f + (BD + 1) * (la + BA * lc)) * N2; };
    const int l[3] = {lx, ly, lz};
    const int own_slot = slot(l[D], l[A], l[C]) + jk;
    long long yo[R][N];
    int eo[R];
    // ---- A: own lines -------------------------------------------------------
#pragma unroll
    for (int r = 0; r < R; ++r) {
      eo[r] = 0;
      if (r < rows) {
        double x[N];
        fx_load_line<N, D>(xs + r * zstep, wide, x);
        const int ex = fx_line_exp<N>(x);
        const int at = own_slot + r * ZSLOT;
        if (ex != kFxSlow) {
          FxLimbs xl[N];
#pragma unroll
          for (int i = 0; i < N; ++i) xl[i] = fx_split(fx_from_double(x[i], ex));
          const FxSums t = fx_trace_sums<N>(xl, ax);
          tr[at] = FxPair{t.ev - t.od, t.pe - t.po};
          tr[S::LINES + at + N2] = FxPair{t.ev + t.od, t.pe + t.po};
#pragma unroll
          for (int i = 0; i < N; ++i) {
            FxAcc acc;
#pragma unroll
            for (int j = 0; j < N; ++j) {
              // without advection O has the zeros of K1, but for the mass at (0, 0)
              if (ADV || (i && j && !((i + j) & 1)) || (D == 0 && !i && !j)) acc.add(xl[j], ax.O[i * N + j]);
            }
            yo[r][i] = acc.value();
          }
        } else {
          double t[4];
          fx_traces_f64<N, D>(x, ct, t);
          tr[at] = FxPair{__double_as_longlong(t[0]), __double_as_longlong(t[1])};
          tr[S::LINES + at + N2] = FxPair{__double_as_longlong(t[2]), __double_as_longlong(t[3])};
        }
        eo[r] = ex;
        exps[at] = (unsigned short)ex;
        exps[S::LINES + at + N2] = (unsigned short)ex;
      }
    }
    // ---- A: the face neighbours outside the brick ---------------------------
    for (int item = tid; item < 2 * BA * BC * N2; item += T) {
      const int h = item / N2, hjk = item - h * N2;
      const int up = h >= BA * BC, q = up ? h - BA * BC : h, lc = q / BA, la = q - lc * BA;
      int g = up ? o[D] + e[D] : o[D] - 1;
      bool there = la < e[A] && lc < e[C];
      if (g < 0 || g >= args.nc[D]) {
        if (args.periodic[D]) g = g < 0 ? g + args.nc[D] : g - args.nc[D];
        else there = false;
      }
      if (!there) continue;
      int p[3];
      p[D] = g;
      p[A] = o[A] + la;
      p[C] = o[C] + lc;
      double x[N];
      fx_load_line<N, D>(args.u + (p[0] + (long long)nx * p[1] + nxy * p[2]) * N3 + fx_line_base<N, D>(hjk), wide, x);
      const int ex = fx_line_exp<N>(x);
      // an upper neighbour's lower face, a lower neighbour's upper face
      const int at = (up ? slot(e[D], la, lc) : S::LINES + slot(0, la, lc)) + hjk;
      if (ex != kFxSlow) {
        FxLimbs xl[N];
#pragma unroll
        for (int i = 0; i < N; ++i) xl[i] = fx_split(fx_from_double(x[i], ex));
        const FxSums t = fx_trace_sums<N>(xl, ax);
        tr[at] = FxPair{t.ev + (up ? -t.od : t.od), t.pe + (up ? -t.po : t.po)};
      } else {
        double t[4];
        fx_traces_f64<N, D>(x, ct, t);
        tr[at] = FxPair{__double_as_longlong(up ? t[0] : t[2]), __double_as_longlong(up ? t[1] : t[3])};
      }
      exps[at] = (unsigned short)ex;
    }
    __syncthreads();
    // ---- B: face part and results -------------------------------------------
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (r < rows) {
        const int g = o[D] + l[D] + (D == 2 ? r * B::L : 0);
        const bool has_up = g + 1 < args.nc[D] || args.periodic[D];
        const bool has_lo = g > 0 || args.periodic[D];
        // side 1 of a face's slot holds the traces of the cell below it, side 0
        // those of the cell above
        const int s0 = own_slot + r * ZSLOT, s1 = s0 + N2;
        FxPair own1 = tr[S::LINES + s1], own0 = tr[s0], up, lo;
        int eu = eo[r], el = eo[r];
        if (has_up) {
          up = tr[s1];
          eu = exps[s1];
        } else {
          up = own1;
          if (args.weak_dirichlet) up = FxPair{-own1.v, (fx.slope ? 0 : own1.v) - own1.p};
        }
        if (has_lo) {
          lo = tr[S::LINES + s0];
          el = exps[S::LINES + s0];
        } else {
          lo = own0;
          if (args.weak_dirichlet) lo = FxPair{-own0.v, (fx.slope ? 0 : own0.v) - own0.p};
        }
        // without diffusion the outflow neighbour has no part in the line, and its
        // magnitude must not either (au, al: the exponents to align at; eu, el stay what
        // the neighbours' traces are held in)
        int au = eu, al = el;
        if (ADV) {
          if (!fx.couple[D][1] && eu != kFxSlow) au = eo[r];
          if (!fx.couple[D][0] && el != kFxSlow) al = eo[r];
        }
        const int ef = max(eo[r], max(au, al));
        double* const rc = res + (c0 + r * (B::X * B::Y * B::L)) * N3;
        double y[N];
        if (D == 0) {
#pragma unroll
          for (int i = 0; i < N; ++i) y[i] = 0.0;
        } else {
#pragma unroll
          for (int i = 0; i < N; ++i) y[i] = rc[fx_res_off<N, D>(jk, i)];
        }
        if (ef != kFxSlow) {
          const int so = min(ef - eo[r], 63), su = min(ef - au, 63), sl = min(ef - al, 63);
          const long long vu = fx_shr(up.v, su), vl = fx_shr(lo.v, sl);
          const long long J1 = fx_shr(own1.v, so) - vu, P1 = fx_shr(own1.p, so) - fx_shr(up.p, su);
          const long long J0 = fx_shr(own0.v, so) - vl, P0 = fx_shr(own0.p, so) - fx_shr(lo.p, sl);
          const FxLimbs vs = fx_split(J1 + J0), vd = fx_split(J1 - J0);
          const FxLimbs ps = fx_split(P1 + P0), pd = fx_split(P1 - P0);
          FxLimbs in{0, 0};
          if (ADV) in = fx_split(fx.inflow_upper[D] ? (has_up ? vu : 0) : (has_lo ? vl : 0));
#pragma unroll
          for (int i = 0; i < N; ++i) {
            FxAcc acc(fx_shr(yo[r][i], so), 1ll << 31);
            acc.add((i & 1) ? pd : ps, ax.np[i]);
            if (i) acc.add((i & 1) ? vd : vs, ax.nv[i]);  // L_0' = 0
            if (ADV) acc.add(in, ax.a[i]);
            y[i] = fma(double(acc.value()), fx_pow2((ef << 20) + ax.ex[i]), y[i]);
          }
        } else {
          double ys[N];  // (the call takes an address: y itself stays in registers)
          fx_line_f64<N, ADV, D>(args, ct, xs + r * zstep, has_up, has_lo, up, eu, lo, el, fx.slope != 0, ys);
#pragma unroll
          for (int i = 0; i < N; ++i) y[i] += ys[i];
        }
        if (D == 2) {
          const long long at = first + r * zstep + jk * N;
          if (STAGE) {
#pragma unroll
            for (int i = 0; i < N; ++i) {
              double v = st.u[at + i];
              if (st.earlier > 0) v = fma(st.a[0], __ldg(st.w[0] + at + i), v);
              if (st.earlier > 1) v = fma(st.a[1], __ldg(st.w[1] + at + i), v);
              __stcs(st.y + at + i, fma(st.a[st.earlier], y[i], v));
            }
            if (!args.w) continue;
          }
          double* wc = args.w + at;
          if (N % 2 == 0 && wide) {
#pragma unroll
            for (int i = 0; i < N; i += 2)
              __stcs(reinterpret_cast<double2*>(wc + i), make_double2(y[i], y[i + 1 < N ? i + 1 : i]));
          } else {
#pragma unroll
            for (int i = 0; i < N; ++i) __stcs(wc + i, y[i]);
          }
        } else {
#pragma unroll
          for (int i = 0; i < N; ++i) rc[fx_res_off<N, D>(jk, i)] = y[i];
        }
      }
    }
    if (D < 2) __syncthreads();
  };
  axis(std::integral_constant<int, 0>());
  axis(std::integral_constant<int, 1>());
  axis(std::integral_constant<int, 2>());
}

}  // namespace gbfem
