// FP32 instantiations of the DG apply kernel (the inner-solve precision of
// the mixed-precision path).
#include <type_traits>

#include "dg_cell_kernel.cuh"
#include "dg_plane_kernel.cuh"
#include "dg_launch.cuh"

namespace gbfem {
int dg_launch_f32(const DgArgsT<float>& a, const DgTablesT<float>& t, int n, int q, bool kappa,
                  cudaStream_t s) {
  return dg_launch<float>(a, t, n, q, kappa, s);
}
int dg_const_launch_f32(const DgArgsT<float>& a, const DgConstTablesT<float>& t, int n, float* traces, int phase,
                        cudaStream_t s, float* ucopy) {
  return dg_const_launch<float>(a, t, n, traces, phase, s, ucopy);
}
// One-kernel closed form over the whole grid.  p = 1 keeps one thread per cell
// (dg_cell_kernel.cuh; 64^3: 21 us, with n threads per cell 24: planes of four dofs
// are too little work per thread); p >= 2 has n threads per cell
// (dg_plane_kernel.cuh; 64^3 Q2 70 -> 52, Q3 92 -> 65, Q4 from two kernels' 424 to 193).
template <int N>
static long long plane_blocks(const int* nc) {
  using B = PlaneBrick<N>;
  return (long long)((nc[0] + B::X - 1) / B::X) * ((nc[1] + B::Y - 1) / B::Y) * ((nc[2] + B::Z - 1) / B::Z);
}
static long long cell_blocks(const int* nc) {
  return (long long)((nc[0] + kCellBX - 1) / kCellBX) * ((nc[1] + kCellBY - 1) / kCellBY) *
         ((nc[2] + kCellBZ - 1) / kCellBZ);
}
long long dg_one_kernel_blocks(int n, const int* nc) {
  return n == 2 ? cell_blocks(nc) : (n == 3 ? plane_blocks<3>(nc) : (n == 4 ? plane_blocks<4>(nc) : plane_blocks<5>(nc)));
}

template <int N, bool ADV, bool KC, bool DOT>
static int dg_cell_launch_one(const DgArgsT<float>& a, const DgConstTablesT<float>& t, cudaStream_t s, double* partial,
                              CgScalars* sc) {
  // whole cells move as 16-byte accesses
  if ((reinterpret_cast<uintptr_t>(a.u) | reinterpret_cast<uintptr_t>(a.w)) & 15)
    return set_error(GBFEM_ERR_INVALID, "dg apply: FP32 vectors of order 1 have to be 16-byte aligned");
  auto kern = dg_cell_kernel<N, ADV, KC, DOT>;
  constexpr size_t smem = CellSlots<N>::BYTES;
  GBFEM_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  const long long blocks = cell_blocks(a.nc);
  if (blocks <= 0) return GBFEM_OK;
  if (blocks > 2147483647LL) return set_error(GBFEM_ERR_INVALID, "dg apply: grid too large");
  kern<<<unsigned(blocks), kCellThreads, smem, s>>>(a, t, partial, sc);
  GBFEM_CUDA_TRY(cudaGetLastError());
  return GBFEM_OK;
}
template <int N, bool ADV, bool KC>
static int dg_cell_launch_form(const DgArgsT<float>& a, const DgConstTablesT<float>& t, cudaStream_t s, double* partial,
                               CgScalars* sc) {
  return sc ? dg_cell_launch_one<N, ADV, KC, true>(a, t, s, partial, sc)
            : dg_cell_launch_one<N, ADV, KC, false>(a, t, s, partial, sc);
}

template <int N, bool ADV, bool KC, bool DOT, bool WIDE>
static int dg_plane_launch_one(const DgArgsT<float>& a, const DgConstTablesT<float>& t, cudaStream_t s, double* partial,
                               CgScalars* sc) {
  auto kern = dg_plane_kernel<N, ADV, KC, DOT, WIDE>;
  constexpr size_t smem = PlaneShape<N>::BYTES;
  GBFEM_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  const long long blocks = plane_blocks<N>(a.nc);
  if (blocks <= 0) return GBFEM_OK;
  if (blocks > 2147483647LL) return set_error(GBFEM_ERR_INVALID, "dg apply: grid too large");
  kern<<<unsigned(blocks), PlaneShape<N>::T, smem, s>>>(a, t, partial, sc);
  GBFEM_CUDA_TRY(cudaGetLastError());
  return GBFEM_OK;
}

template <int N, bool ADV, bool KC>
static int dg_plane_launch_form(const DgArgsT<float>& a, const DgConstTablesT<float>& t, cudaStream_t s,
                                double* partial, CgScalars* sc) {
  // rows of four dofs move as one 16-byte access where both vectors allow it
  const bool wide = ((reinterpret_cast<uintptr_t>(a.u) | reinterpret_cast<uintptr_t>(a.w)) & 15) == 0;
  if constexpr (N == 4)
    if (wide)
      return sc ? dg_plane_launch_one<N, ADV, KC, true, true>(a, t, s, partial, sc)
                : dg_plane_launch_one<N, ADV, KC, false, true>(a, t, s, partial, sc);
  return sc ? dg_plane_launch_one<N, ADV, KC, true, false>(a, t, s, partial, sc)
            : dg_plane_launch_one<N, ADV, KC, false, false>(a, t, s, partial, sc);
}

// sc (and partial): the apply of a device-resident CG iteration, with <u, w>
int dg_one_kernel_launch_f32(const DgArgsT<float>& a, const DgConstTablesT<float>& t, int n, cudaStream_t s,
                             double* partial, CgScalars* sc) {
  const bool kc = a.kcell != nullptr, adv = a.advect != 0;
#define GBFEM_ONE_KERNEL(FORM, NN)                                  \
  if (n == NN) {                                                    \
    if (kc) return FORM<NN, false, true>(a, t, s, partial, sc);     \
    if (adv) return FORM<NN, true, false>(a, t, s, partial, sc);    \
    return FORM<NN, false, false>(a, t, s, partial, sc);            \
  }
  GBFEM_ONE_KERNEL(dg_cell_launch_form, 2)
  GBFEM_ONE_KERNEL(dg_plane_launch_form, 3)
  GBFEM_ONE_KERNEL(dg_plane_launch_form, 4)
  GBFEM_ONE_KERNEL(dg_plane_launch_form, 5)
#undef GBFEM_ONE_KERNEL
  return set_error(GBFEM_ERR_NOT_IMPLEMENTED, "dg apply: unsupported order");
}

int dg_kappa_points_f32(const float* kappa, float* kq, float* kf, long long ncells, const DgTablesT<float>& t, int n,
                         int q, cudaStream_t s) {
  return dg_kappa_points<float>(kappa, kq, kf, ncells, t, n, q, s);
}
}  // namespace gbfem
