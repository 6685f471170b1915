// Scalars of the device-resident CG loop and the pieces its kernels share.
#pragma once
#include <cuda_runtime.h>

#include "blas.cuh"

namespace gbfem {

// In device memory.  Written by the last CTA of the two scalar products of an
// iteration (cg_set_alpha, cg_set_end); every other kernel only reads it.  alpha
// and beta are kept in FP32 too: a conversion in every thread of an FP32 vector
// kernel would go through the FP64 pipe.
struct CgScalars {
  double res, alpha, beta, tol;  // <p, s>, step, direction factor, squared tolerance
  float alpha_f, beta_f;
  int active, dir;               // this iteration is done at all / has a direction update
  int conv, it, max_it, status;
  unsigned done[2];              // CTAs that have delivered their part
};

template <typename T> __device__ __forceinline__ T cg_alpha(const CgScalars* s);
template <> __device__ __forceinline__ double cg_alpha<double>(const CgScalars* s) { return s->alpha; }
template <> __device__ __forceinline__ float cg_alpha<float>(const CgScalars* s) { return s->alpha_f; }
template <typename T> __device__ __forceinline__ T cg_beta(const CgScalars* s);
template <> __device__ __forceinline__ double cg_beta<double>(const CgScalars* s) { return s->beta; }
template <> __device__ __forceinline__ float cg_beta<float>(const CgScalars* s) { return s->beta_f; }

// alpha = rho / <q, h>
__device__ __forceinline__ void cg_set_alpha(CgScalars* s, double qh) {
  if (!s->active) return;
  const double alpha = s->res / qh;
  if (!isfinite(alpha)) {
    s->status = 1;
    s->conv = 1;
    s->active = 0;
    return;
  }
  s->alpha = alpha;
  s->alpha_f = float(alpha);
}

// the new rho: the end of the iteration, and the next one's beta
__device__ __forceinline__ void cg_set_end(CgScalars* s, double rho) {
  if (!s->active) return;
  const double beta = rho / s->res;
  s->beta = beta;
  s->beta_f = float(beta);
  s->dir = 1;
  s->res = rho;
  s->it += 1;
  if (!(rho > s->tol) || s->it >= s->max_it) s->conv = 1;
  if (!isfinite(rho)) {
    s->status = 1;
    s->conv = 1;
  }
  if (s->conv) s->active = 0;
}

// Thread 0 of every CTA hands in its part of scalar product `which`; true in the
// CTA that came last, for which all parts are visible.  (Called by all threads.)
__device__ __forceinline__ bool cg_deliver(double part, double* partial, CgScalars* s, int which) {
  __shared__ int cg_last;
  if (threadIdx.x == 0) {
    partial[blockIdx.x] = part;
    __threadfence();
    cg_last = atomicInc(&s->done[which], gridDim.x - 1) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  return cg_last != 0;
}

// Sum of a float-float value (s + c) over the warp, in float-float.
__device__ __forceinline__ void cg_ff_warp_sum(float& s, float& c) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float b = __shfl_down_sync(0xffffffffu, s, o), d = __shfl_down_sync(0xffffffffu, c, o);
    const float t = s + b, bp = t - s;
    c += d + ((s - (t - bp)) + (b - bp));
    s = t;
  }
}

// The CTA's part of an FP32 scalar product from its threads' accumulators, valid
// in thread 0 (whole warps; up to 32).  Float-float down to one value per warp,
// FP64 above.
__device__ __forceinline__ double cg_block_part(DotAcc<float> a) {
  __shared__ float cg_part[2][32];
  cg_ff_warp_sum(a.s, a.c);
  if ((threadIdx.x & 31) == 0) {
    cg_part[0][threadIdx.x >> 5] = a.s;
    cg_part[1][threadIdx.x >> 5] = a.c;
  }
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (unsigned w = 0; w < blockDim.x / 32; ++w) t += f32_to_f64(cg_part[0][w]) + f32_to_f64(cg_part[1][w]);
  return t;
}

// Sum of the CTAs' parts by the last CTA, valid in thread 0.
__device__ __forceinline__ double cg_sum_parts(const double* partial, int np) {
  __shared__ double cg_sum[32];
  double s = 0.0;
  for (int i = threadIdx.x; i < np; i += blockDim.x) s += __ldcg(partial + i);
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) cg_sum[threadIdx.x >> 5] = s;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (unsigned w = 0; w < blockDim.x / 32; ++w) t += cg_sum[w];
  return t;
}

}  // namespace gbfem
