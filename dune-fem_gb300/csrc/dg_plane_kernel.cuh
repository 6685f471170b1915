// One-kernel FP32 apply of the constant-coefficient closed form, p >= 2 (the same
// operator as dg_trace_kernel + dg_const_kernel; the algebra is described in
// dg_const_kernel.cuh), without the trace buffer in HBM.
//
// What bounds it: the issue of instructions (2.7 a clock and SM, 90 per dof, of which
// 37 are the arithmetic, 1.5 halo rows per own row included) and, next, the latency of
// the three phases; DRAM runs at 18 %.  Three quarters of a brick's reads are its
// halo's, through L2.  Measured (GB300, cold L2, launch included), the form with one
// thread per cell (64 dofs and 64 results in registers, 12 warps per SM; p = 4: the
// two-kernel form) before, this one after, constant kappa / kappa per cell:
//   Q2 64^3  70 / 75 -> 52 / 55 us      Q3 64^3  92 / 102 -> 65 / 69
//   Q3 32^3  22.5 / 24.4 -> 18.0 / 18.5  Q4 64^3  424 / 441 -> 193 / 206
// Bricks (Q3): 4x4x4 with 4 CTAs per SM 69 us, with 3 74; 8x4x4 70; 4x4x8 76;
// 4x4x2 72.  Own planes loaded and stored directly, n^2 dofs apart between
// neighbouring threads: L1 wavefronts bound it, 76 (Q4: 301 instead of 193).
//
// Layout of the work: a CTA owns a brick of cells, n threads per cell.  Thread i
// of a cell owns its plane i0 = i (n^2 contiguous dofs) for the y and z lines and
// the plane i1 = i for the x lines; the planes are exchanged through shared memory
// within the warp (a cell's threads sit in one warp).  A row is the n values of
// one trace that a thread's n lines of an axis give: row i of the face's n x n
// coefficients, the same i for the two cells of a face.  A face's numerical flux is
// computed once and exchanged through shared memory, which holds one slot per face
// of the brick and one per face on its lower boundary (2 n^2 values each).
//  0. the brick's cells go to the exchange buffer by coalesced rows; rows of the face
//     neighbours outside the brick (their traces on the face that touches it) go into
//     the slots, one row per thread and item;
//  1. every thread writes its rows of the traces (v, P) of the cell's lower faces
//     into the faces' slots, or, on the brick's lower boundary, the boundary slots;
//  2. every thread computes its row of the flux through the cell's upper faces
//     from its own traces and the slot (the upper neighbour's) and overwrites the
//     row with (Val, G) as seen from the lower cell; spare threads do the rows of
//     the brick's lower faces.  The upper cell of a face reads the numbers
//     negated: the interior fluxes are odd in the two sides' traces, which holds
//     exactly in floating point; a domain-boundary face's terms are stored negated
//     where the cell is the upper one;
//  3. the 1-D line operators and the face expansion, x lines first, then y and z
//     on top, with dg_const_kernel's formulas and order; store.
// Every output is one thread's fixed-order sum: deterministic, independent of
// the launch.
#pragma once
#include <cuda_runtime.h>

#include "cg_device.cuh"
#include "dg_const_kernel.cuh"

namespace gbfem {

// Cells of a brick (a multiple of the cells a warp holds, so that every warp is full).
template <int N>
struct PlaneBrick;
template <>
struct PlaneBrick<3> { static constexpr int X = 5, Y = 4, Z = 4, MINB = 4; };
template <>
struct PlaneBrick<4> { static constexpr int X = 4, Y = 4, Z = 4, MINB = 4; };
template <>
struct PlaneBrick<5> { static constexpr int X = 3, Y = 4, Z = 4, MINB = 3; };

template <int N>
struct PlaneShape {
  using B = PlaneBrick<N>;
  static constexpr int N2 = N * N, N3 = N2 * N, CELLS = B::X * B::Y * B::Z;
  static constexpr int CW = 32 / N;  // cells per warp
  static constexpr int WARPS = CELLS / CW, T = WARPS * 32;
  static constexpr int NX = (B::X + 1) * B::Y * B::Z, NY = B::X * (B::Y + 1) * B::Z, NZ = B::X * B::Y * (B::Z + 1);
  static constexpr int NFACE = NX + NY + NZ, NBND = B::Y * B::Z + B::X * B::Z + B::X * B::Y;
  static constexpr int SLOT = 2 * N2;  // floats
  static constexpr int EXCHANGE = ((NFACE + NBND) * SLOT * 4 + 255) / 256 * 256;
  static constexpr size_t BYTES = EXCHANGE + CELLS * N3 * 4 + 240;  // 240: room to align the start
  static_assert(CELLS % CW == 0, "full warps");
};

// Slot of the face at position f (0..B_d) along axis d; la, lb are the brick-local
// coordinates along the other two axes (in increasing axis order).
template <int N>
__device__ __forceinline__ int plane_slot(int d, int f, int la, int lb) {
  using S = PlaneShape<N>;
  using B = PlaneBrick<N>;
  if (d == 0) return f + (B::X + 1) * (la + B::Y * lb);
  if (d == 1) return S::NX + la + B::X * (f + (B::Y + 1) * lb);
  return S::NX + S::NY + la + B::X * (lb + B::Y * f);
}
// Boundary slot of the brick cell's lower face along d.
template <int N>
__device__ __forceinline__ int plane_bnd_slot(int d, int la, int lb) {
  using S = PlaneShape<N>;
  using B = PlaneBrick<N>;
  if (d == 0) return S::NFACE + la + B::Y * lb;
  if (d == 1) return S::NFACE + B::Y * B::Z + la + B::X * lb;
  return S::NFACE + B::Y * B::Z + B::X * B::Z + la + B::X * lb;
}

// Shared-memory addresses are 32-bit window addresses: the generic ones cost an
// address conversion at each use.
// Row i of half 0 (v or Val) and of half 1 (P or G) of a slot.  n = 4: 16-byte rows,
// the halves swapped where `odd` (the parity of x), so that the rows of two cells
// next to one another along x fall into distinct banks.
struct PlaneRow {
  unsigned v, g;
};
template <int N>
__device__ __forceinline__ PlaneRow plane_row(unsigned slots, int s, int odd, int i) {
  PlaneRow r;
  if (N == 4) {
    r.v = slots + s * 128 + ((i ^ ((odd & 1) << 2)) << 4);
    r.g = r.v ^ 64;
  } else {
    r.v = slots + (s * 2 * N + i) * (4 * N);
    r.g = r.v + 4 * N * N;
  }
  return r;
}
__device__ __forceinline__ void plane_st(unsigned at, float a) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(at), "f"(a) : "memory");
}
__device__ __forceinline__ float plane_ld(unsigned at) {
  float a;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(a) : "r"(at) : "memory");
  return a;
}
template <int N>
__device__ __forceinline__ void plane_put(unsigned at, const float (&a)[N]) {
  if constexpr (N == 4)
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(at), "f"(a[0]), "f"(a[1]), "f"(a[2]), "f"(a[3])
                 : "memory");
  else {
#pragma unroll
    for (int k = 0; k < N; ++k) plane_st(at + 4 * k, a[k]);
  }
}
template <int N>
__device__ __forceinline__ void plane_get(unsigned at, float (&a)[N]) {
  if constexpr (N == 4)
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(a[0]), "=f"(a[1]), "=f"(a[2]), "=f"(a[3])
                 : "r"(at)
                 : "memory");
  else {
#pragma unroll
    for (int k = 0; k < N; ++k) a[k] = plane_ld(at + 4 * k);
  }
}

// Byte offset of (i0, i1, .) of brick cell c in the exchange buffer.  n = 4: 16-byte
// chunks, XOR-ed so that both the plane and the x-line accesses of two cells'
// threads fall into distinct banks.
template <int N>
__device__ __forceinline__ int plane_at(int c, int i0, int i1) {
  if (N == 4) return c * 256 + (((i0 * 4 + (i1 ^ i0)) ^ ((c & 1) << 2)) << 4);
  return (c * N * N + i0 * N + i1) * (4 * N);
}

// Both traces of the lower or upper face for the n lines of a plane x: line k is
// x[k][.] (LAST: along the plane's second index) or x[.][k].
template <int N, bool KC, int D, bool LAST>
__device__ __forceinline__ void plane_traces(const float (&x)[N * N], bool upper, const DgConstTablesT<float>& tabs,
                                             float (&v)[N], float (&p)[N]) {
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const float x0 = LAST ? x[k * N] : x[k];
    float ev = x0, od = 0.f, pe = KC ? 0.f : x0, po = 0.f;
#pragma unroll
    for (int i = 1; i < N; ++i) {
      const float xi = LAST ? x[k * N + i] : x[i * N + k];
      if (i & 1) {
        od = fmaf(tabs.tr[N + i], xi, od);
        po = fmaf(tabs.pc[D][i], xi, po);
      } else {
        ev = fmaf(tabs.tr[N + i], xi, ev);
        pe = fmaf(tabs.pc[D][i], xi, pe);
      }
    }
    v[k] = upper ? ev + od : ev - od;
    p[k] = upper ? pe + po : pe - po;
  }
}

// The flux through an interior face normal to D as seen from its lower cell m,
// from m's upper-face traces and the upper cell p's lower-face traces.
template <int N, bool ADV, bool KC, int D>
__device__ __forceinline__ void plane_interior(const float (&vm)[N], const float (&pm)[N], const float (&vp)[N],
                                               const float (&pp)[N], float km, float kp, const DgArgsT<float>& args,
                                               const DgConstTablesT<float>& tabs, float (&val)[N], float (&G)[N]) {
  const bool fold_alpha = tabs.am1 != 0.f;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const float J = vm[k] - vp[k];
    float vv;
    if (KC) {
      vv = fmaf(tabs.A1[D] * (0.5f * (km + kp)), J, -tabs.A2[D] * (km * pm[k] - kp * pp[k]));
    } else {
      vv = pm[k] - pp[k];
      if (fold_alpha) vv = fmaf(tabs.am1, J, vv);
      if (ADV) vv = fmaf(tabs.adv[2 * D + 1], args.b[D] >= 0.f ? vm[k] : vp[k], vv);
    }
    val[k] = vv;
    G[k] = J;
  }
}

// A domain-boundary face normal to D from the cell's own traces on it; stored
// negated when it is the cell's lower face.
template <int N, bool ADV, bool KC, int D>
__device__ __forceinline__ void plane_boundary(bool upper, const float (&vo)[N], const float (&po)[N], float kc,
                                               const DgArgsT<float>& args, const DgConstTablesT<float>& tabs,
                                               float (&val)[N], float (&G)[N]) {
  const float bn = upper ? args.b[D] : -args.b[D];
#pragma unroll
  for (int k = 0; k < N; ++k) {
    float vv = 0.f, gg = 0.f;
    if (args.weak_dirichlet) {
      if (KC) vv = fmaf(tabs.A1[D] * kc, vo[k], -2.f * tabs.A2[D] * kc * po[k]);
      else vv = fmaf(tabs.am2, vo[k], po[k] + po[k]);
      gg = vo[k] + vo[k];
    }
    if (ADV && bn > 0.f) vv = fmaf(tabs.adv[2 * D + (upper ? 1 : 0)], vo[k], vv);
    val[k] = upper ? vv : -vv;
    G[k] = upper ? gg : -gg;
  }
}

template <int N, bool WIDE>
__device__ __forceinline__ void plane_load_row(const float* __restrict__ src, float (&x)[N]) {
  if constexpr (N == 4 && WIDE) {
    const float4 t = __ldg(reinterpret_cast<const float4*>(src));
    x[0] = t.x;
    x[1] = t.y;
    x[2] = t.z;
    x[3] = t.w;
  } else {
#pragma unroll
    for (int k = 0; k < N; ++k) x[k] = __ldg(src + k);
  }
}
// n^2 dofs: plane i0 of the cell at src (x lines: the plane i1 = i, rows n^2 apart)
template <int N, bool WIDE>
__device__ __forceinline__ void plane_load(const float* __restrict__ src, int step, float (&x)[N * N]) {
#pragma unroll
  for (int r = 0; r < N; ++r) {
    float t[N];
    plane_load_row<N, WIDE>(src + r * step, t);
#pragma unroll
    for (int k = 0; k < N; ++k) x[r * N + k] = t[k];
  }
}

// Brick geometry shared by the phases.
struct PlaneGeometry {
  int nc[3];
  int o[3];  // first cell of the brick
  int e[3];  // the brick's extent inside the grid
  long long stride[3];
};

// The warp's cells between global memory and the exchange buffer, whole rows of
// cells along x by consecutive lanes: a thread's own plane is n^2 dofs apart from its
// neighbour's, which as direct loads and stores costs n times the L1 wavefronts.
template <int N, bool IN, bool WIDE>
__device__ __forceinline__ void plane_stage(unsigned ex, const float* __restrict__ src, float* __restrict__ dst, int warp,
                                            int lane, const PlaneGeometry& B) {
  using S = PlaneShape<N>;
  using Br = PlaneBrick<N>;
#pragma unroll
  for (int r = 0; r < S::CW / Br::X; ++r) {
    const int c = warp * S::CW + r * Br::X, l1 = (c / Br::X) % Br::Y, l2 = c / (Br::X * Br::Y);
    if (l1 >= B.e[1] || l2 >= B.e[2]) continue;
    const long long at = (B.o[0] + B.stride[1] * (B.o[1] + l1) + B.stride[2] * (B.o[2] + l2)) * S::N3;
    if constexpr (N == 4) {
#pragma unroll
      for (int q0 = 0; q0 < Br::X * 16; q0 += 32) {
        const int q = q0 + lane;
        if (q >= B.e[0] * 16) continue;
        const unsigned e = ex + plane_at<N>(c + (q >> 4), (q >> 2) & 3, q & 3);
        if (IN) {
          float t[4];
          plane_load_row<N, WIDE>(src + at + 4 * q, t);
          plane_put<4>(e, t);
        } else {
          float t[4];
          plane_get<4>(e, t);
          float* const g = dst + at + 4 * q;
          if (WIDE) {
            __stcs(reinterpret_cast<float4*>(g), make_float4(t[0], t[1], t[2], t[3]));
          } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) __stcs(g + k, t[k]);
          }
        }
      }
    } else {
#pragma unroll
      for (int q0 = 0; q0 < Br::X * S::N3; q0 += 32) {
        const int q = q0 + lane;
        if (q >= B.e[0] * S::N3) continue;
        const unsigned e = ex + 4 * (c * S::N3 + q);
        if (IN) plane_st(e, __ldg(src + at + q));
        else __stcs(dst + at + q, plane_ld(e));
      }
    }
  }
}

// The face neighbour of brick-boundary position (D, la, lb) below (upper = false)
// or above the brick; false where the domain ends there.
template <int D>
__device__ __forceinline__ bool plane_halo(bool upper, int la, int lb, const PlaneGeometry& B,
                                           const DgArgsT<float>& args, long long* hcell, long long* bcell) {
  constexpr int A = D == 0 ? 1 : 0, C = D == 2 ? 1 : 2;  // the other axes, increasing
  const long long tang = (long long)(B.o[A] + la) * B.stride[A] + (long long)(B.o[C] + lb) * B.stride[C];
  *bcell = tang + (long long)(upper ? B.o[D] + B.e[D] - 1 : B.o[D]) * B.stride[D];
  int g = upper ? B.o[D] + B.e[D] : B.o[D] - 1;
  if (g < 0 || g >= B.nc[D]) {
    if (!args.periodic[D]) return false;
    g = g < 0 ? B.nc[D] - 1 : 0;
  }
  *hcell = tang + (long long)g * B.stride[D];
  return true;
}

// The r-th face on the brick's lower (or upper) boundary, counted over the whole
// brick: its axis and brick-local coordinates.  false: outside the grid.
template <int N>
__device__ __forceinline__ bool plane_boundary_face(int r, const PlaneGeometry& B, int* d, int* la, int* lb) {
  using Br = PlaneBrick<N>;
  constexpr int C0 = Br::Y * Br::Z, C1 = Br::X * Br::Z;
  if (r < C0) {
    *d = 0;
    *lb = r / Br::Y;
    *la = r - *lb * Br::Y;
    return *la < B.e[1] && *lb < B.e[2];
  }
  if (r < C0 + C1) {
    r -= C0;
    *d = 1;
    *lb = r / Br::X;
    *la = r - *lb * Br::X;
    return *la < B.e[0] && *lb < B.e[2];
  }
  r -= C0 + C1;
  *d = 2;
  *lb = r / Br::X;
  *la = r - *lb * Br::X;
  return *la < B.e[0] && *lb < B.e[1];
}

// Phase 0 item: row i of the trace of the halo cell's face towards the brick.  The
// loads of all of a thread's items are issued before the first is used.
struct PlaneHalo {
  int D;  // -1: none
  bool upper;
  PlaneRow r;
};
template <int N, bool WIDE>
__device__ __forceinline__ PlaneHalo plane_halo_load(int item, const PlaneGeometry& B, const DgArgsT<float>& args,
                                                     unsigned slots, float (&x)[N * N]) {
  constexpr int N2 = N * N, N3 = N2 * N;
  PlaneHalo h;
  h.D = -1;
  h.upper = (item / N) & 1;
  const int i = item % N;
  int D, la, lb;
  if (item >= 2 * PlaneShape<N>::NBND * N || !plane_boundary_face<N>(item / (2 * N), B, &D, &la, &lb)) return h;
  long long hcell, bcell;
  if (!(D == 0   ? plane_halo<0>(h.upper, la, lb, B, args, &hcell, &bcell)
        : D == 1 ? plane_halo<1>(h.upper, la, lb, B, args, &hcell, &bcell)
                 : plane_halo<2>(h.upper, la, lb, B, args, &hcell, &bcell)))
    return h;
  h.D = D;
  const int f = h.upper ? (D == 0 ? B.e[0] : D == 1 ? B.e[1] : B.e[2]) : 0;
  h.r = plane_row<N>(slots, plane_slot<N>(D, f, la, lb), D == 0 ? f : la, i);
  plane_load<N, WIDE>(args.u + hcell * N3 + i * (D == 0 ? N : N2), D == 0 ? N2 : N, x);
  return h;
}
template <int N, bool KC>
__device__ __forceinline__ void plane_halo_row(const PlaneHalo& h, const float (&x)[N * N],
                                               const DgConstTablesT<float>& tabs) {
  if (h.D < 0) return;
  float v[N], p[N];
  if (h.D == 0) plane_traces<N, KC, 0, false>(x, !h.upper, tabs, v, p);
  else if (h.D == 1) plane_traces<N, KC, 1, false>(x, !h.upper, tabs, v, p);
  else plane_traces<N, KC, 2, true>(x, !h.upper, tabs, v, p);
  plane_put<N>(h.r.v, v);
  plane_put<N>(h.r.g, p);
}

// kappa of the brick's cell and of the halo cell at the brick's lower face (D, la, lb)
template <int D>
__device__ __forceinline__ void plane_lower_kappa(int la, int lb, const PlaneGeometry& B, const DgArgsT<float>& args,
                                                  float* kb, float* kh) {
  long long hcell, bcell;
  const bool has_nb = plane_halo<D>(false, la, lb, B, args, &hcell, &bcell);
  *kb = __ldg(args.kcell + bcell);
  if (has_nb) *kh = __ldg(args.kcell + hcell);
}

// Phase 2 item: row i of the flux through the brick's lower face at (D, la, lb).
template <int N, bool ADV, bool KC, int D>
__device__ __forceinline__ void plane_lower_row(int la, int lb, int i, float kb, float kh,
                                                const PlaneGeometry& B, const DgArgsT<float>& args,
                                                const DgConstTablesT<float>& tabs, unsigned slots) {
  long long hcell, bcell;
  const bool has_nb = plane_halo<D>(false, la, lb, B, args, &hcell, &bcell);
  const int odd = D == 0 ? 0 : la;
  const PlaneRow r0 = plane_row<N>(slots, plane_slot<N>(D, 0, la, lb), odd, i);
  const PlaneRow rb = plane_row<N>(slots, plane_bnd_slot<N>(D, la, lb), odd, i);
  float vo[N], po[N], a[N], b[N];
  plane_get<N>(rb.v, vo);
  plane_get<N>(rb.g, po);
  if (has_nb) {
    float vh[N], ph[N];
    plane_get<N>(r0.v, vh);
    plane_get<N>(r0.g, ph);
    plane_interior<N, ADV, KC, D>(vh, ph, vo, po, kh, kb, args, tabs, a, b);
  } else {
    plane_boundary<N, ADV, KC, D>(false, vo, po, kb, args, tabs, a, b);
  }
  plane_put<N>(r0.v, a);
  plane_put<N>(r0.g, b);
}

// Phase 1: the n rows a thread's plane x gives of the cell's lower face along D.
template <int N, bool KC, int D, bool LAST>
__device__ __forceinline__ void plane_own_lower(const float (&x)[N * N], const int (&l)[3], int i,
                                                const DgConstTablesT<float>& tabs, unsigned slots) {
  const int la = l[D == 0 ? 1 : 0], lb = l[D == 2 ? 1 : 2];
  const int s = l[D] > 0 ? plane_slot<N>(D, l[D], la, lb) : plane_bnd_slot<N>(D, la, lb);
  float v[N], p[N];
  plane_traces<N, KC, D, LAST>(x, false, tabs, v, p);
  const PlaneRow r = plane_row<N>(slots, s, l[0], i);
  plane_put<N>(r.v, v);
  plane_put<N>(r.g, p);
}

// Phase 2: row i of the flux through the cell's upper face along D.
template <int N, bool ADV, bool KC, int D, bool LAST>
__device__ __forceinline__ void plane_own_upper(const float (&x)[N * N], const int (&l)[3], int i, float kc,
                                                float kn, const PlaneGeometry& B, const DgArgsT<float>& args,
                                                const DgConstTablesT<float>& tabs, unsigned slots) {
  const int sl = plane_slot<N>(D, l[D] + 1, l[D == 0 ? 1 : 0], l[D == 2 ? 1 : 2]);
  const bool has_nb = B.o[D] + l[D] + 1 < B.nc[D] || args.periodic[D];
  float vo[N], po[N], a[N], b[N];
  plane_traces<N, KC, D, LAST>(x, true, tabs, vo, po);
  const PlaneRow r = plane_row<N>(slots, sl, l[0] + (D == 0), i);
  if (has_nb) {
    float vn[N], pn[N];
    plane_get<N>(r.v, vn);
    plane_get<N>(r.g, pn);
    plane_interior<N, ADV, KC, D>(vo, po, vn, pn, kc, kn, args, tabs, a, b);
  } else {
    plane_boundary<N, ADV, KC, D>(true, vo, po, kc, args, tabs, a, b);
  }
  plane_put<N>(r.v, a);
  plane_put<N>(r.g, b);
}

// Line operators and face expansion of the n lines of a plane (x: dofs, w: results),
// D == 0 starts the results, the others add.
template <int N, bool ADV, bool KC, int D, bool LAST>
__device__ __forceinline__ void plane_lines(const float (&x)[N * N], float (&w)[N * N], unsigned slots, const int (&l)[3],
                                            int row, float kc, bool has_mass, bool has_massK,
                                            const DgConstTablesT<float>& tabs) {
  float V0[N], G0[N], V1[N], G1[N];
  const int la = l[D == 0 ? 1 : 0], lb = l[D == 2 ? 1 : 2];
  const PlaneRow r0 = plane_row<N>(slots, plane_slot<N>(D, l[D], la, lb), l[0], row);
  const PlaneRow r1 = plane_row<N>(slots, plane_slot<N>(D, l[D] + 1, la, lb), l[0] + (D == 0), row);
  plane_get<N>(r0.v, V0);
  plane_get<N>(r0.g, G0);
  plane_get<N>(r1.v, V1);
  plane_get<N>(r1.g, G1);
  const float gscale = KC ? -tabs.A2[D] * kc : 1.f;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    // own view: Val_0 = -slot0, Val_1 = slot1 (G likewise)
    const float vs = V1[k] - V0[k], vd = V1[k] + V0[k];
    float gs = G1[k] - G0[k], gd = G1[k] + G0[k];
    if (KC) {
      gs *= gscale;
      gd *= gscale;
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
      float& out = w[LAST ? k * N + i : i * N + k];
      float acc = D == 0 ? 0.f : out;
      if (KC) {
        float tt = 0.f;
#pragma unroll
        for (int j = 0; j < N; ++j)
          if (i != 0 && j != 0 && !((i + j) & 1)) tt = fmaf(tabs.M[D][i * N + j], x[LAST ? k * N + j : j * N + k], tt);
        acc = fmaf(kc, tt, acc);
        if (D == 0 && has_massK) acc = fmaf(tabs.massK, x[LAST ? k * N + i : i * N + k], acc);
        acc = fmaf(tabs.tr[N + i], (i & 1) ? vd : vs, acc);
        if (i > 0) acc = fmaf(tabs.dtr[N + i], (i & 1) ? gd : gs, acc);
      } else {
#pragma unroll
        for (int j = 0; j < N; ++j) {
          const bool mass00 = D == 0 && i == 0 && j == 0 && has_mass;
          const bool k1 = i != 0 && j != 0 && !((i + j) & 1);
          const bool d1 = j < i && ((i + j) & 1);
          if (k1 || mass00 || (ADV && d1)) acc = fmaf(tabs.M[D][i * N + j], x[LAST ? k * N + j : j * N + k], acc);
        }
        acc = fmaf(tabs.etr[D][i], (i & 1) ? vd : vs, acc);
        if (i > 0) acc = fmaf(tabs.edtr[D][i], (i & 1) ? gd : gs, acc);
      }
      out = acc;
    }
  }
}

// DOT: the operator of a device-resident CG iteration (cg_device.cuh): nothing
// once it has converged; otherwise also <u, w>, and alpha by the last CTA.
template <int N, bool ADV, bool KC, bool DOT, bool WIDE>
__global__ void __launch_bounds__(PlaneShape<N>::T, PlaneBrick<N>::MINB)
    dg_plane_kernel(const __grid_constant__ DgArgsT<float> args, const __grid_constant__ DgConstTablesT<float> tabs,
                    double* __restrict__ partial, CgScalars* sc) {
  if (DOT && !sc->active) return;
  using S = PlaneShape<N>;
  using Br = PlaneBrick<N>;
  constexpr int N2 = S::N2, T = S::T;
  static_assert(!(KC && ADV), "cellwise kappa without advection");
  extern __shared__ __align__(16) float plane_smem[];
  // 256-byte aligned: the rows' places are XOR-ed into the addresses
  const unsigned slots = (unsigned(__cvta_generic_to_shared(plane_smem)) + 255u) & ~255u;
  const unsigned ex = slots + S::EXCHANGE;  // planes <-> x lines
  const int tid = threadIdx.x, lane = tid & 31;
  PlaneGeometry B;
  B.nc[0] = args.nc[0];
  B.nc[1] = args.nc[1];
  B.nc[2] = args.nc[2];
  const unsigned nbx = unsigned(B.nc[0] + Br::X - 1) / Br::X, nby = unsigned(B.nc[1] + Br::Y - 1) / Br::Y;
  const unsigned bxy = blockIdx.x / nbx, bz = bxy / nby, by = bxy - bz * nby;
  B.o[0] = (blockIdx.x - bxy * nbx) * Br::X;
  B.o[1] = by * Br::Y;
  B.o[2] = bz * Br::Z;
  B.e[0] = min(Br::X, B.nc[0] - B.o[0]);
  B.e[1] = min(Br::Y, B.nc[1] - B.o[1]);
  B.e[2] = min(Br::Z, B.nc[2] - B.o[2]);
  B.stride[0] = 1;
  B.stride[1] = B.nc[0];
  B.stride[2] = (long long)B.nc[0] * B.nc[1];
  const int lc = lane / N, i = lane - lc * N;
  const int c = (tid >> 5) * S::CW + lc;  // the brick's cell
  const int l[3] = {c % Br::X, (c / Br::X) % Br::Y, c / (Br::X * Br::Y)};
  const bool valid = lc < S::CW && l[0] < B.e[0] && l[1] < B.e[1] && l[2] < B.e[2];
  const long long cell = (B.o[0] + l[0]) + B.stride[1] * (B.o[1] + l[1]) + B.stride[2] * (B.o[2] + l[2]);

  // ---- 0. own plane, halo rows ----------------------------------------------------
  constexpr int HITEMS = 2 * S::NBND * N, HB = N < 5 ? (HITEMS + T - 1) / T : 1;  // items, in flight per thread
  {
    float x[HB][N2];
    PlaneHalo h[HB];
#pragma unroll
    for (int k = 0; k < HB; ++k) h[k] = plane_halo_load<N, WIDE>(tid + k * T, B, args, slots, x[k]);
    plane_stage<N, true, WIDE>(ex, args.u, nullptr, tid >> 5, lane, B);
#pragma unroll
    for (int k = 0; k < HB; ++k) plane_halo_row<N, KC>(h[k], x[k], tabs);
#pragma unroll 1
    for (int item = tid + HB * T; item < HITEMS; item += T) {
      const PlaneHalo g = plane_halo_load<N, WIDE>(item, B, args, slots, x[0]);
      plane_halo_row<N, KC>(g, x[0], tabs);
    }
  }
  // rows [r][.] of the plane i0 = i, and rows [i0 = r][i][.] of the x lines
  const unsigned at_plane = ex + plane_at<N>(c, i, 0), at_x = ex + plane_at<N>(c, 0, i);
  auto row_at = [&](int r, bool plane) {
    if (N == 4) return plane ? at_plane ^ (r << 4) : at_x ^ (r * 80);
    return plane ? at_plane + r * 4 * N : at_x + r * 4 * N2;
  };
  auto put_rows = [&](const float (&x)[N2], bool plane) {
#pragma unroll
    for (int r = 0; r < N; ++r) {
      float t[N];
#pragma unroll
      for (int k = 0; k < N; ++k) t[k] = x[r * N + k];
      plane_put<N>(row_at(r, plane), t);
    }
  };
  auto get_rows = [&](float (&x)[N2], bool plane) {
#pragma unroll
    for (int r = 0; r < N; ++r) {
      float t[N];
      plane_get<N>(row_at(r, plane), t);
#pragma unroll
      for (int k = 0; k < N; ++k) x[r * N + k] = t[k];
    }
  };
  __syncwarp();
  float u[N2];
  if (valid) get_rows(u, true);

  // ---- 1. own lower-face traces -----------------------------------------------------
  if (valid) {
    float x[N2];
    get_rows(x, false);
    plane_own_lower<N, KC, 0, false>(x, l, i, tabs, slots);
    plane_own_lower<N, KC, 1, false>(u, l, i, tabs, slots);
    plane_own_lower<N, KC, 2, true>(u, l, i, tabs, slots);
  }
  // kappa for phase 2, in flight over the barrier
  float kc = 0.f, kn[3] = {0.f, 0.f, 0.f}, kb = 0.f, kh = 0.f;
  if (KC) {
    if (valid) {
      kc = __ldg(args.kcell + cell);
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const int cd = B.o[d] + l[d];
        if (cd + 1 < B.nc[d]) kn[d] = __ldg(args.kcell + cell + B.stride[d]);
        else if (args.periodic[d]) kn[d] = __ldg(args.kcell + cell - cd * B.stride[d]);
      }
    }
    int D, la, lb;
    if (tid < S::NBND * N && plane_boundary_face<N>(tid / N, B, &D, &la, &lb)) {
      if (D == 0) plane_lower_kappa<0>(la, lb, B, args, &kb, &kh);
      else if (D == 1) plane_lower_kappa<1>(la, lb, B, args, &kb, &kh);
      else plane_lower_kappa<2>(la, lb, B, args, &kb, &kh);
    }
  }
  __syncthreads();

  // ---- 2. fluxes of the upper faces, and of the brick's lower faces -------------------
  if (valid) {
    float x[N2];
    get_rows(x, false);
    plane_own_upper<N, ADV, KC, 0, false>(x, l, i, kc, kn[0], B, args, tabs, slots);
    plane_own_upper<N, ADV, KC, 1, false>(u, l, i, kc, kn[1], B, args, tabs, slots);
    plane_own_upper<N, ADV, KC, 2, true>(u, l, i, kc, kn[2], B, args, tabs, slots);
  }
#pragma unroll 1
  for (int item = tid; item < S::NBND * N; item += T) {
    const int row = item % N;
    int D, la, lb;
    if (!plane_boundary_face<N>(item / N, B, &D, &la, &lb)) continue;
    if (KC && item >= T) {
      if (D == 0) plane_lower_kappa<0>(la, lb, B, args, &kb, &kh);
      else if (D == 1) plane_lower_kappa<1>(la, lb, B, args, &kb, &kh);
      else plane_lower_kappa<2>(la, lb, B, args, &kb, &kh);
    }
    if (D == 0) plane_lower_row<N, ADV, KC, 0>(la, lb, row, kb, kh, B, args, tabs, slots);
    else if (D == 1) plane_lower_row<N, ADV, KC, 1>(la, lb, row, kb, kh, B, args, tabs, slots);
    else plane_lower_row<N, ADV, KC, 2>(la, lb, row, kb, kh, B, args, tabs, slots);
  }
  __syncthreads();

  // ---- 3. line operators and face expansion, x then y then z ----------------------------
  const bool has_massK = KC && tabs.massK != 0.f, has_mass = tabs.M[0][0] != 0.f;
  float w[N2];
  if (valid) {
    float x[N2];
    get_rows(x, false);
    plane_lines<N, ADV, KC, 0, false>(x, w, slots, l, i, kc, has_mass, has_massK, tabs);
    put_rows(w, false);
  }
  __syncwarp();
  DotAcc<float> acc;
  if (valid) {
    get_rows(w, true);
    plane_lines<N, ADV, KC, 1, false>(u, w, slots, l, i, kc, has_mass, has_massK, tabs);
    plane_lines<N, ADV, KC, 2, true>(u, w, slots, l, i, kc, has_mass, has_massK, tabs);
    put_rows(w, true);
    if (DOT) {
#pragma unroll
      for (int q = 0; q < N2; ++q) acc.add(u[q], w[q]);
    }
  }
  __syncwarp();
  plane_stage<N, false, WIDE>(ex, nullptr, args.w, tid >> 5, lane, B);
  if constexpr (DOT) {
    if (!cg_deliver(cg_block_part(acc), partial, sc, 0)) return;
    const double t = cg_sum_parts(partial, int(gridDim.x));
    if (tid == 0) cg_set_alpha(sc, t);
  }
}

}  // namespace gbfem
