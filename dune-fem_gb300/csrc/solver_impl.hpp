// Definition of the opaque preconditioner handle.
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "../../include/gbfem.h"

namespace gbfem {

enum class PcKind { Diagonal = 1, BlockJacobi = 2, External = 3, Sor = 4, ScaledBlock = 5 };

int precond_apply(const struct ::gbfem_preconditioner_s* pc, const void* r, void* z, cudaStream_t s);
// Jacobi / Gauss-Seidel / SOR / SSOR sweeps over an assembled operator (sor.cu)
int sor_apply(const struct ::gbfem_preconditioner_s* pc, const void* r, void* z, cudaStream_t s);
// scaled block Jacobi on the tensor cores (sb_tc.cu), the solves' form: set-up from
// the (type, start, count) tiles, and the apply
int sb_tc_setup(struct ::gbfem_preconditioner_s* pc, const std::vector<int>& tiles3, int nb, cudaStream_t s);
int sb_tc_apply(const struct ::gbfem_preconditioner_s* pc, const float* kcell, const float* r, float* z,
                cudaStream_t s);
// the same by fast diagonalisation (sb_fdm.cu), the direct apply's form
int sb_fdm_setup(struct ::gbfem_preconditioner_s* pc);
int sb_fdm_apply(const struct ::gbfem_preconditioner_s* pc, const float* r, float* z, cudaStream_t s);
void sb_fdm_destroy(void* tables);
struct CgScalars;
// h = A q, <q, h> and alpha; 0 parts where the operator has no such kernel
long long cg_apply_dot_parts(const struct ::gbfem_operator_s* op);
int cg_apply_dot(const struct ::gbfem_operator_s* op, const void* q, void* h, double* partial, CgScalars* sc,
                 cudaStream_t s);
int dg_mixed_form(struct ::gbfem_operator_s* op, struct ::gbfem_operator_s* keep, struct ::gbfem_operator_s** out);
// the Q1 operator's CG in one kernel (q1_cg.cu), for the solves it takes
struct Q1Trial {     // self test
  int late_cta;      // a CTA whose waits all run out, -1: none
  int no_cluster;    // as if no cluster could be placed
  int no_grid;       // as if the device held fewer blocks than the other form has
};
bool q1_cg_takes(gbfem_operator op, gbfem_preconditioner pc, const gbfem_solver_params& prm);
int q1_cg(gbfem_operator op, gbfem_preconditioner pc, const gbfem_solver_params& prm, const void* b, void* x,
          cudaStream_t s, gbfem_solver_info* info, bool* taken, const Q1Trial* trial);

}  // namespace gbfem

struct gbfem_preconditioner_s {
  gbfem::PcKind kind = gbfem::PcKind::Diagonal;
  int precision = GBFEM_F64;
  long long n = 0;
  int nloc = 1;
  void* data = nullptr;  // diagonal inverse or block inverses
  bool owns_data = true;
  int storage = GBFEM_F64;   // block Jacobi: GBFEM_F64, GBFEM_F32 or GBFEM_F16 (scaled) blocks
  float* scales = nullptr;   // GBFEM_F16 storage: one scale per block
  // External (e.g. the learned preconditioner): z = P(r)
  int (*ext_apply)(void* ctx, const void* r, void* z, cudaStream_t s) = nullptr;
  void (*ext_destroy)(void* ctx) = nullptr;
  void* ext_ctx = nullptr;
  // Flexible solvers switch to this preconditioner when the iteration with
  // this one stagnates (the learned preconditioner's block-Jacobi fallback).
  struct gbfem_preconditioner_s* fallback = nullptr;
  // Sor (and ScaledBlock: the cellwise-kappa operator): the operator (not owned), method (GBFEM_SMOOTHER_*),
  // sweeps, relaxation, cells grouped by level x+y+z with the level offsets,
  // and the previous iterate of Jacobi; data holds 1/diag
  const struct gbfem_operator_s* sor_op = nullptr;
  int sor_method = 0, sor_sweeps = 1;
  double sor_relax = 1.0;
  int* sor_cells = nullptr;
  void* sor_tmp = nullptr;
  std::vector<long long> sor_level_offsets;
  // ScaledBlock: sor_cells holds the cells sorted by boundary type; tiles of
  // (type, start, count) into it
  int* sb_tiles = nullptr;
  long long sb_ntiles = 0;
  // ScaledBlock on the tensor cores: tiles without padding, A_hi | A_lo
  // images per type, the kernel's status word (1 = a wait timed out)
  int* sb_tc_tiles = nullptr;
  int sb_tc_ntiles = 0;
  int sb_tc_wide = 0;  // 64-cell tiles with K = 64 (blocks of up to 64 dofs)
  void* sb_tc_img = nullptr;
  int* sb_tc_status = nullptr;
  void* sb_fdm = nullptr;  // ScaledBlock by fast diagonalisation: its tables (host), null without
};
