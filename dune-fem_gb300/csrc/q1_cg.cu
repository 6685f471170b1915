// CG of the continuous Q1 operator (2-D, strong Dirichlet rows) with the
// diagonal preconditioner or none, whole solve in one cooperative kernel.
//
// What bounds it: latency.  The problem is small (65^2 vertices at 64 x 64
// cells; 34 KB a vector), so an iteration of the general loop is its six or more
// launches: 28 us of kernels that each run a few microseconds for microseconds
// of work spread over one or two CTAs.  Here every CTA keeps a contiguous range
// of vertices for the whole solve, x, p and the search direction in registers
// and shared memory, and an iteration costs two grid-wide sums, which are also
// its only synchronisations: chains of dependent FP64 additions (65 clocks each)
// and one division (600).  Measured, general loop (graph chunks of 32) -> this
// kernel: 64 x 64 (154 iterations) 4.28 -> 0.88 ms, 150 x 150 13.3 -> 4.0 ms,
// 500 x 400 58.9 -> 22.0 ms.
//
//  1. q = s + beta q on the CTA's range and a halo of one grid row and a vertex on
//     either side (the halo from the s its owners published), h = A q, sum q.h;
//  2. alpha;  x += alpha q, p -= alpha h, s = P p (published), sum p.s; beta.
//
// A grid-wide sum: each CTA stores its part together with the number of the
// sum (both halves of the value tagged, so a reader needs no other flag), every
// warp of every CTA polls all parts and adds them in the same order.  All CTAs
// so take the same decisions on the same bits.  Two sets of slots alternate: a
// CTA that writes sum k+2 has seen every part of sum k+1, hence every CTA is done
// reading sum k.  The polls of a wait are bounded; a CTA that gives up sets a word that
// the host checks and leaves.  The statements are those of LinearSolver::cg (solver/linear/cg.hh:
// 18-117) on p = b - A x; without a preconditioner s = p.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <climits>
#include <cmath>
#include <cstring>

#include "blas.cuh"
#include "gbfem_internal.cuh"
#include "operator_impl.hpp"
#include "solver_impl.hpp"

namespace gbfem {

constexpr int kQ1Threads = 256;
constexpr int kQ1MaxPer = 8;           // vertices per thread
constexpr int kQ1MaxCluster = 16;
constexpr int kQ1MaxGrid = 160;        // CTAs (one per SM)
constexpr int kQ1PollLimit = 1 << 20;  // polls of one wait, a sum or a halo (about a second)

struct Q1CgArgs {
  const void *b, *dinv;
  void *x, *p, *q;            // p, q: kept between launches
  unsigned long long* slots;  // [2][grid][2]: tagged parts of the grid-wide sums
  unsigned long long* s;      // [n][2]: tagged s, for the neighbours' halos
  double* out;                // residual, iterations, status, tolerance, beta
  int* late;                  // set by a CTA that gave up
  int late_cta;               // this CTA's waits all run out (self test; -1: none)
  int resume;
  int n, vxn, vyn, per_cta;
  double c[9];                // stencil, row by row from the lower left vertex
  double tol;                 // squared tolerance factor
  int measure, max_it;
};

enum { Q1_OK = 0, Q1_NONFINITE = 1, Q1_TIMEOUT = 2 };
enum { Q1_RES = 0, Q1_IT, Q1_STATUS, Q1_TOL, Q1_BETA, Q1_OUT };
// iterations of one launch (tens of milliseconds): a solve that cannot reach its
// tolerance must not occupy the GPU without end
constexpr int kQ1Chunk = 8192;

__device__ __forceinline__ double q1_warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

struct Q1Shared {
  double part[kQ1Threads];
  double parts[2][kQ1MaxCluster];  // cluster: the CTAs' parts of a sum
  double sum, quotient;
  int ok;
  int late;  // a poll of this CTA ran out
};

// A value and its tag in two words, each of which carries the tag: a reader that
// finds both has the value, without a fence on either side.
__device__ __forceinline__ void q1_put(unsigned long long* at, double v, unsigned tag) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(v), t = (unsigned long long)tag << 32;
  volatile unsigned long long* w = at;
  w[0] = t | (bits & 0xffffffffull);
  w[1] = t | (bits >> 32);
}
__device__ __forceinline__ double q1_get(const unsigned long long* at, unsigned tag, int limit, int& polls) {
  const volatile unsigned long long* w = at;
  unsigned long long a = 0, b = 0;
  do {
    a = w[0];
    b = w[1];
  } while (((unsigned)(a >> 32) != tag || (unsigned)(b >> 32) != tag) && ++polls < limit);
  return __longlong_as_double((long long)((a & 0xffffffffull) | (b << 32)));
}

// Sum of v over the grid into sh.sum, and other / sum (inverse: sum / other)
// into sh.quotient; the same bits in every CTA.  Warp 0 does all of it: a
// warp's FP64 instruction holds the SM's FP64 pipe for 16 clocks, so eight warps
// doing the same would take eight times as long.  false: parts did not arrive.
// (No barrier reductions here: their aligned form must not meet a warp that
// comes out of a divergent loop.)
template <bool CLUSTER>
__device__ __forceinline__ bool q1_grid_sum(double v, double other, bool inverse, unsigned epoch,
                                            unsigned long long* slots, Q1Shared& sh, int limit) {
  const int tid = threadIdx.x, grid = gridDim.x;
  sh.part[tid] = v;
  __syncthreads();
  double t = 0.0;
  if (tid < 32) {
    double w[kQ1Threads / 32];
#pragma unroll
    for (int k = 0; k < kQ1Threads / 32; ++k) w[k] = sh.part[tid + 32 * k];
#pragma unroll
    for (int o = kQ1Threads / 64; o > 0; o >>= 1)
#pragma unroll
      for (int k = 0; k < o; ++k) w[k] += w[k + o];
    t = q1_warp_sum(w[0]);
  }
  if constexpr (CLUSTER) {
    auto cl = cooperative_groups::this_cluster();
    // every CTA gets every part
    if (tid < grid) cl.map_shared_rank(&sh, unsigned(tid))->parts[epoch & 1u][blockIdx.x] = t;
    __syncwarp();
    cl.sync();
    if (tid < 32) {
      t = q1_warp_sum(tid < grid ? sh.parts[epoch & 1u][tid] : 0.0);
      const double q = inverse ? t / other : other / t;
      if (tid == 0) {
        sh.sum = t;
        sh.quotient = q;
        sh.ok = 1;
      }
    }
  } else {
    if (tid < 32) {
      unsigned long long* set = slots + (size_t)(epoch & 1u) * grid * 2;
      if (tid == 0) q1_put(set + 2 * blockIdx.x, t, epoch);
      t = 0.0;
      int polls = 0;
      for (int c = tid; c < grid; c += 32) t += q1_get(set + 2 * c, epoch, limit, polls);
      __syncwarp();
      t = q1_warp_sum(t);
      const bool late = __any_sync(0xffffffffu, polls >= limit) || sh.late;
      const double q = inverse ? t / other : other / t;
      if (tid == 0) {
        sh.sum = t;
        sh.quotient = q;
        sh.ok = late ? 0 : 1;
      }
    }
  }
  __syncthreads();
  return sh.ok != 0;
}

template <typename T, int PER, bool CLUSTER>
__global__ void __launch_bounds__(kQ1Threads) q1_cg_kernel(const __grid_constant__ Q1CgArgs g) {
  extern __shared__ __align__(16) unsigned char q1_smem[];
  __shared__ Q1Shared sh;
  T* const sq = reinterpret_cast<T*>(q1_smem);  // q on [v0 - halo, v1 + halo)
  T* const ss = sq + (g.per_cta + 2 * (g.vxn + 1));  // cluster: s on [v0, v1)
  // s of this CTA's vertex v, where the neighbours can read it
  auto publish = [&](int v, T sv, unsigned tag) {
    if (CLUSTER) ss[v - blockIdx.x * g.per_cta] = sv;
    else q1_put(g.s + 2ll * v, double(sv), tag);
  };
  const int tid = threadIdx.x, halo = g.vxn + 1;
  const int v0 = min(int(blockIdx.x) * g.per_cta, g.n), v1 = min(v0 + g.per_cta, g.n);
  const int h0 = max(v0 - halo, 0), h1 = min(v1 + halo, g.n);
  const T* b = static_cast<const T*>(g.b);
  const T* dinv = static_cast<const T*>(g.dinv);
  T* xg = static_cast<T*>(g.x);
  T x[PER], p[PER], s[PER], di[PER], h[PER];
  bool in[PER];  // interior vertex
  auto each = [&](auto f) {
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const int v = v0 + tid + k * kQ1Threads;
      if (v < v1) f(k, v);
    }
  };
  // A on the vector in sq at vertex v (in double, rounded once)
  auto apply = [&](int k, int v) -> T {
    const T* q = sq + (v - h0);
    if (!in[k]) return q[0];
    double a[3];  // one chain per row: the FP64 latency is what counts
#pragma unroll
    for (int dy = -1; dy <= 1; ++dy) {
      const T* r = q + dy * g.vxn;
      const double* c = g.c + (dy + 1) * 3;
      a[dy + 1] = fma(c[2], double(r[1]), fma(c[1], double(r[0]), c[0] * double(r[-1])));
    }
    return T(a[0] + a[1] + a[2]);
  };
  if (tid == 0) sh.late = 0;
  if constexpr (CLUSTER) cooperative_groups::this_cluster().sync();  // every CTA runs before its memory is written
  unsigned epoch = 0, tag = 0;
  const int limit = int(blockIdx.x) == g.late_cta ? 0 : kQ1PollLimit;
  auto total = [&](double v, double other, bool inverse) {
    ++epoch;
    return q1_grid_sum<CLUSTER>(v, other, inverse, epoch, g.slots, sh, limit);
  };

  // p = b - A x, s = P p, q = s (or the state the last launch left)
  T* pg = static_cast<T*>(g.p);
  T* qg = static_cast<T*>(g.q);
  const T* first = g.resume ? qg : xg;
  for (int v = h0 + tid; v < h1; v += kQ1Threads) sq[v - h0] = first[v];
  each([&](int k, int v) {
    const int vy = v / g.vxn, vx = v - vy * g.vxn;
    in[k] = vx > 0 && vy > 0 && vx < g.vxn - 1 && vy < g.vyn - 1;
    x[k] = xg[v];
    di[k] = dinv ? dinv[v] : T(1);
  });
  double before[Q1_OUT];
  for (int k = 0; k < Q1_OUT; ++k) before[k] = g.resume ? g.out[k] : 0.0;
  __syncthreads();
  DotAcc<T> acc, accb;
  ++tag;
  each([&](int k, int v) {
    const T bv = b[v];
    p[k] = g.resume ? pg[v] : bv - apply(k, v);
    s[k] = dinv ? p[k] * di[k] : p[k];
    publish(v, s[k], tag);
    acc.add(p[k], s[k]);
    accb.add(bv, bv);
  });
  bool ok = total(acc.value(), 1.0, true);
  double residual = sh.sum, bb = 1.0;
  if (!g.resume && g.measure == GBFEM_TOL_RELATIVE) {
    ok = ok && total(accb.value(), 1.0, true);
    bb = sh.sum;
  }
  double tolerance =
      g.tol * (g.measure == GBFEM_TOL_RELATIVE ? bb : (g.measure == GBFEM_TOL_RESIDUAL_REDUCTION ? residual : 1.0));
  int it = 0;
  T beta = T(0);
  if (g.resume) {
    residual = before[Q1_RES];
    tolerance = before[Q1_TOL];
    it = int(before[Q1_IT]);
    beta = T(before[Q1_BETA]);
  }
  int status = ok ? Q1_OK : Q1_TIMEOUT;
  if (ok && !(isfinite(residual) && isfinite(tolerance))) status = Q1_NONFINITE;
  const int last = g.max_it - it > kQ1Chunk ? it + kQ1Chunk : g.max_it;
  for (; status == Q1_OK && residual > tolerance && it < last; ++it) {
    const T bt = beta;
    each([&](int k, int v) { sq[v - h0] = it > 0 ? s[k] + bt * sq[v - h0] : s[k]; });
    int polls = 0;
    for (int j = tid; j < (v0 - h0) + (h1 - v1); j += kQ1Threads) {
      const int v = j < v0 - h0 ? h0 + j : v1 + (j - (v0 - h0));
      T sv;
      if constexpr (CLUSTER) {
        const int c = v / g.per_cta;
        sv = cooperative_groups::this_cluster().map_shared_rank(ss, unsigned(c))[v - c * g.per_cta];
      } else {
        sv = T(q1_get(g.s + 2ll * v, tag, limit, polls));
      }
      sq[v - h0] = it > 0 ? sv + bt * sq[v - h0] : sv;
    }
    if (!CLUSTER && polls >= limit) sh.late = 1;
    __syncthreads();
    DotAcc<T> qh;
    each([&](int k, int v) {
      h[k] = apply(k, v);
      qh.add(sq[v - h0], h[k]);
    });
    if (!total(qh.value(), residual, false)) { status = Q1_TIMEOUT; break; }
    const double alpha = sh.quotient;  // residual / q.h
    if (!isfinite(alpha)) { status = Q1_NONFINITE; break; }
    const T a = T(alpha);
    DotAcc<T> ps;
    ++tag;
    each([&](int k, int v) {
      x[k] = a * sq[v - h0] + x[k];
      p[k] = -a * h[k] + p[k];
      s[k] = dinv ? p[k] * di[k] : p[k];
      publish(v, s[k], tag);
      ps.add(p[k], s[k]);
    });
    if (!total(ps.value(), residual, true)) { status = Q1_TIMEOUT; break; }
    beta = T(sh.quotient);  // new / old residual
    residual = sh.sum;
  }
  if (status == Q1_OK && !isfinite(residual)) status = Q1_NONFINITE;
  if (status != Q1_TIMEOUT)
    each([&](int k, int v) {
      xg[v] = x[k];
      pg[v] = p[k];
      qg[v] = sq[v - h0];
    });
  if (status == Q1_TIMEOUT && tid == 0) atomicExch(g.late, 1);
  if (blockIdx.x == 0 && tid == 0) {
    g.out[Q1_RES] = residual;
    g.out[Q1_IT] = double(it);
    g.out[Q1_STATUS] = double(status);
    g.out[Q1_TOL] = tolerance;
    g.out[Q1_BETA] = double(beta);
  }
  if constexpr (CLUSTER) {
    __syncwarp();
    cooperative_groups::this_cluster().sync();  // no CTA leaves while its memory may be read
  }
}

// fits: ask only whether the device can hold the launch
template <typename T, int PER>
static cudaError_t q1_launch(const Q1CgArgs& a, int grid, bool cluster, cudaStream_t s, bool* fits) {
  const size_t smem = size_t(2 * a.per_cta + 2 * (a.vxn + 1)) * sizeof(T);
  auto kern = cluster ? q1_cg_kernel<T, PER, true> : q1_cg_kernel<T, PER, false>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(grid));
  cfg.blockDim = dim3(kQ1Threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at{};
  if (cluster) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = unsigned(grid);
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
  } else {
    at.id = cudaLaunchAttributeCooperative;
    at.val.cooperative = 1;
  }
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  if (fits) {
    int dev = 0, sms = 0, held = 0;
    if (cluster) {
      e = cudaOccupancyMaxActiveClusters(&held, kern, &cfg);
      *fits = e == cudaSuccess && held > 0;
    } else {
      e = cudaGetDevice(&dev);
      if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&held, kern, kQ1Threads, smem);
      *fits = e == cudaSuccess && (long long)held * sms >= grid;
    }
    return e;
  }
  return cudaLaunchKernelEx(&cfg, kern, a);
}

template <typename T>
static cudaError_t q1_launch_per(const Q1CgArgs& a, int grid, bool cluster, cudaStream_t s, bool* fits) {
  const int per = (a.per_cta + kQ1Threads - 1) / kQ1Threads;
  if (per <= 1) return q1_launch<T, 1>(a, grid, cluster, s, fits);
  if (per <= 2) return q1_launch<T, 2>(a, grid, cluster, s, fits);
  if (per <= 4) return q1_launch<T, 4>(a, grid, cluster, s, fits);
  return q1_launch<T, kQ1MaxPer>(a, grid, cluster, s, fits);
}
static cudaError_t q1_launch_any(int precision, const Q1CgArgs& a, int grid, bool cluster, cudaStream_t s, bool* fits) {
  return precision == GBFEM_F64 ? q1_launch_per<double>(a, grid, cluster, s, fits)
                                : q1_launch_per<float>(a, grid, cluster, s, fits);
}

// Whether q1_cg takes the solve: no per-iteration output, the stops of the CG
// loop on <p, s>, and a size whose state fits one CTA per SM.
bool q1_cg_takes(gbfem_operator op, gbfem_preconditioner pc, const gbfem_solver_params& prm) {
  if (op->kind != OpKind::Q1 || prm.verbose) return false;
  if (pc && (pc->kind != PcKind::Diagonal || pc->precision != op->precision || pc->n != op->ndofs)) return false;
  if (prm.error_measure == GBFEM_TOL_RELATIVE_RESIDUAL) return false;
  int dev = 0, sms = 0, coop = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess)
    return false;
  if (sms > kQ1MaxGrid) sms = kQ1MaxGrid;
  // shared memory: a CTA's range and halo
  const long long halo = 2LL * (op->grid.cells[0] + 2);
  return coop && op->ndofs <= (long long)sms * kQ1Threads * kQ1MaxPer &&
         (2LL * kQ1Threads * kQ1MaxPer + halo) * 8 <= 200 * 1024;
}

// *taken false: nothing is done, the device cannot hold the kernel.
int q1_cg(gbfem_operator op, gbfem_preconditioner pc, const gbfem_solver_params& prm, const void* b, void* x,
          cudaStream_t s, gbfem_solver_info* info, bool* taken, const Q1Trial* trial) {
  int dev = 0, sms = 0;
  GBFEM_CUDA_TRY(cudaGetDevice(&dev));
  GBFEM_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  if (sms > kQ1MaxGrid) sms = kQ1MaxGrid;
  Q1CgArgs a{};
  a.n = int(op->ndofs);
  a.vxn = op->grid.cells[0] + 1;
  a.vyn = op->grid.cells[1] + 1;
  // Up to 16384 vertices: one cluster of at most 16 CTAs, whose sums and halos go
  // through distributed shared memory (65^2: 5.0 us an iteration, 7.2 with the
  // sums through L2); beyond, where 16 SMs' FP64 work outweighs that, the whole GPU
  // (121^2: 8.4 us with one cluster; 151^2: 11.1 us over 90 SMs), and where the device
  // cannot place such a cluster; the general loop where it can hold neither.
  bool cluster = a.n <= kQ1MaxCluster * 1024, fits = false;
  int grid = 0;
  for (;; cluster = false) {
    grid = (a.n + kQ1Threads - 1) / kQ1Threads;
    if (cluster) {
      const int want = (a.n + 63) / 64;
      for (grid = 1; grid < want && grid < kQ1MaxCluster;) grid *= 2;
    }
    if (grid > sms) grid = sms;
    a.per_cta = (a.n + grid - 1) / grid;
    if (!cluster) grid = (a.n + a.per_cta - 1) / a.per_cta;  // (a cluster's last CTAs may be empty)
    if (q1_launch_any(op->precision, a, grid, cluster, s, &fits) != cudaSuccess) {
      (void)cudaGetLastError();
      fits = false;
    }
    if (trial && (cluster ? trial->no_cluster : trial->no_grid)) fits = false;
    if (fits || !cluster) break;
  }
  *taken = fits;
  if (!fits) return GBFEM_OK;
  // the four elements around a vertex: element (cx, cy) has it as its corner
  // (1 - cx) + 2 (1 - cy)
  for (int cy = 0; cy < 2; ++cy)
    for (int cx = 0; cx < 2; ++cx)
      for (int k = 0; k < 4; ++k)
        a.c[(cy + (k >> 1)) * 3 + cx + (k & 1)] += op->q1.K[((1 - cx) + 2 * (1 - cy)) * 4 + k];
  a.tol = prm.tolerance * prm.tolerance;
  a.measure = prm.error_measure;
  a.max_it = prm.max_iterations;
  a.b = b;
  a.x = x;
  a.dinv = pc ? pc->data : nullptr;
  a.late_cta = trial ? trial->late_cta : -1;
  const size_t es = op->precision == GBFEM_F64 ? 8 : 4;
  const size_t vec = (size_t(a.n) * es + 15) / 16 * 16, slots = size_t(2) * grid * 16 + size_t(a.n) * 16;
  struct Buffer {
    char* p = nullptr;
    ~Buffer() { if (p) cudaFree(p); }
  } buf;
  constexpr int kOut = Q1_OUT + 1;  // out, and the late word in a double's place
  GBFEM_CUDA_TRY(cudaMalloc(&buf.p, 2 * vec + slots + kOut * sizeof(double)));
  a.p = buf.p;
  a.q = buf.p + vec;
  a.slots = reinterpret_cast<unsigned long long*>(buf.p + 2 * vec);
  a.s = a.slots + size_t(4) * grid;
  a.out = reinterpret_cast<double*>(buf.p + 2 * vec + slots);
  a.late = reinterpret_cast<int*>(a.out + Q1_OUT);
  double out[kOut];
  GBFEM_CUDA_TRY(cudaMemsetAsync(a.late, 0, sizeof(double), s));
  for (;;) {
    GBFEM_CUDA_TRY(cudaMemsetAsync(a.slots, 0, slots, s));
    const cudaError_t e = q1_launch_any(op->precision, a, grid, cluster, s, nullptr);
    if (e != cudaSuccess) return set_cuda_error(e, "q1 cg");
    GBFEM_CUDA_TRY(cudaMemcpyAsync(out, a.out, sizeof(out), cudaMemcpyDeviceToHost, s));
    GBFEM_CUDA_TRY(cudaStreamSynchronize(s));
    int late;
    std::memcpy(&late, out + Q1_OUT, sizeof(late));
    if (late) return set_error(GBFEM_ERR_CUDA, "q1 cg: a grid-wide sum did not complete");
    if (int(out[Q1_STATUS]) != Q1_OK || !(out[Q1_RES] > out[Q1_TOL]) || int(out[Q1_IT]) >= a.max_it) break;
    a.resume = 1;
  }
  const int it = int(out[Q1_IT]);
  if (int(out[Q1_STATUS]) == Q1_NONFINITE) info->status = GBFEM_ERR_NONFINITE;
  info->residual = std::sqrt(std::fabs(out[Q1_RES]));
  info->iterations = it < prm.max_iterations ? it : -it;
  info->converged = (it < prm.max_iterations && info->status == GBFEM_OK) ? 1 : 0;
  info->operator_applies = it + 1;
  info->preconditioner_applies = pc ? it + 1 : 0;
  return GBFEM_OK;
}

}  // namespace gbfem
