// FP32 instantiations of the DG apply kernel (the inner-solve precision of
// the mixed-precision path).
#include <type_traits>

#include "dg_cell_kernel.cuh"
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
// One-kernel closed form (dg_cell_kernel.cuh) for n <= 4 over the whole grid.
long long dg_cell_blocks(const int* nc) {
  return (long long)((nc[0] + kCellBX - 1) / kCellBX) * ((nc[1] + kCellBY - 1) / kCellBY) *
         ((nc[2] + kCellBZ - 1) / kCellBZ);
}

template <int N, bool ADV, bool KC, bool DOT>
static int dg_cell_launch_one(const DgArgsT<float>& a, const DgConstTablesT<float>& t, cudaStream_t s, double* partial,
                              CgScalars* sc) {
  auto kern = dg_cell_kernel<N, ADV, KC, DOT>;
  constexpr size_t smem = CellSlots<N>::BYTES;
  GBFEM_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  const long long blocks = dg_cell_blocks(a.nc);
  if (blocks <= 0) return GBFEM_OK;
  if (blocks > 2147483647LL) return set_error(GBFEM_ERR_INVALID, "dg apply: grid too large");
  kern<<<unsigned(blocks), kCellThreads, smem, s>>>(a, t, partial, sc);
  GBFEM_CUDA_TRY(cudaGetLastError());
  return GBFEM_OK;
}

bool dg_cell_supported(int n) { return n >= 2 && n <= 4; }

int dg_cell_launch_f32(const DgArgsT<float>& a, const DgConstTablesT<float>& t, int n, cudaStream_t s, double* partial,
                       CgScalars* sc) {
  const bool kc = a.kcell != nullptr, adv = a.advect != 0;
#define GBFEM_CELL_KIND(NN, ADV, KC)                                                      \
  return sc ? dg_cell_launch_one<NN, ADV, KC, true>(a, t, s, partial, sc)                \
            : dg_cell_launch_one<NN, ADV, KC, false>(a, t, s, partial, sc);
#define GBFEM_CELL_CASE(NN)                          \
  if (n == NN) {                                     \
    if (kc) GBFEM_CELL_KIND(NN, false, true)         \
    if (adv) GBFEM_CELL_KIND(NN, true, false)        \
    GBFEM_CELL_KIND(NN, false, false)                \
  }
  GBFEM_CELL_CASE(2)
  GBFEM_CELL_CASE(3)
  GBFEM_CELL_CASE(4)
#undef GBFEM_CELL_CASE
#undef GBFEM_CELL_KIND
  return set_error(GBFEM_ERR_NOT_IMPLEMENTED, "dg apply: one-kernel closed form needs p <= 3");
}

int dg_kappa_points_f32(const float* kappa, float* kq, float* kf, long long ncells, const DgTablesT<float>& t, int n,
                         int q, cudaStream_t s) {
  return dg_kappa_points<float>(kappa, kq, kf, ncells, t, n, q, s);
}
}  // namespace gbfem
