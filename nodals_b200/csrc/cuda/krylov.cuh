// Kernels of the mixed-precision pressure solve (precision NDS_MIXED, no
// reference counterpart; the reference solves the pressure correction with
// FP64 or FP32 PCG / Richardson / outer Chebyshev, h8_main_base.cu:569-726):
//
//  * FP64 defect correction: r = b - A x in FP64 on the FP64 fine operator,
//    the inner solve of A d = r / ||r|| in FP32 (PCG, or FGMRES whose
//    Gram-Schmidt dot products and Hessenberg least squares are FP64), then
//    x += ||r|| d in FP64;
//  * FGMRES(m) with right preconditioning run on the device: the iteration
//    index j, the Hessenberg matrix, the Givens rotations and the residual
//    estimate live in device memory, so one loop body (a conditional while
//    node of a CUDA graph) serves every j;
//  * the Galerkin initial guess over earlier pressure corrections.
//
// Every reduction goes through fixed-order block partials (deterministic).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "common.cuh"
#include "kernels.cuh"

namespace nds {
namespace k {

// x += s y (y in FP32, x in FP64)
__global__ void axpy_from_float(int n, double s, const float* y, double* x) {
  pdl_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] += s * (double)y[i];
}

// ---------------------------------------------------------------------------
// FGMRES(m) device loop.  Layout of the FP64 work array fg (m = restart):
//   H  [(m+1) x m], column j at fg + j (m+1)   (rotated in place: becomes R)
//   cs [m], sn [m], g [m+1], y [m]
// ctl: [0] j = basis vectors built in this pass, [1] converged, [2] -,
//      [3] iteration cap of this pass.   flags bit 16: breakdown / non-finite.
// sc[slot_wn]: ||w||^2 of the current Arnoldi vector (block partial sum).
// ---------------------------------------------------------------------------
struct FgLayout {
  int m;
  __host__ __device__ int H(int i, int j) const { return j * (m + 1) + i; }
  __host__ __device__ int cs(int j) const { return (m + 1) * m + j; }
  __host__ __device__ int sn(int j) const { return (m + 1) * m + m + j; }
  __host__ __device__ int g(int j) const { return (m + 1) * m + 2 * m + j; }
  __host__ __device__ int y(int j) const { return (m + 1) * m + 3 * m + 1 + j; }
  __host__ __device__ int size() const { return (m + 1) * m + 4 * m + 1; }
};

// Z[ctl[0]] = z
__global__ void fg_store(int n, const float* z, const int* ctl, float* __restrict__ Z) {
  pdl_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) Z[(size_t)ctl[0] * n + i] = z[i];
}
// Hessenberg column j: H[j+1][j] = ||w||, the earlier rotations, a new one;
// g and the residual estimate |g[j+1]| (relative: the pass starts from a
// unit vector, g[0] = 1).  Counts the vector, stores ||w|| for fg_normalize,
// and stops the loop on convergence (|g[j+1]| <= tol), at the cap, on a
// happy breakdown (||w|| = 0) or on a non-finite value.
struct FgScalars {
  double* sc;
  int wn2_slot, wn_slot, tol_slot;
  int* ctl;
  int* flags;
  cudaGraphConditionalHandle loop;
  int in_graph;
  HostWords host;
};
__device__ __forceinline__ void fg_givens(double* __restrict__ fg, const FgLayout& L, const FgScalars& p) {
  double* const sc = p.sc;
  int* const ctl = p.ctl;
  int* const flags = p.flags;
  const int wn2_slot = p.wn2_slot, wn_slot = p.wn_slot, tol_slot = p.tol_slot, in_graph = p.in_graph;
  const cudaGraphConditionalHandle loop = p.loop;
  const double tol = sc[tol_slot];
  const int j = ctl[0];
  const double wn = sqrt(sc[wn2_slot]);
  sc[wn_slot] = wn;
  double* col = fg + L.H(0, j);
  col[j + 1] = wn;
  for (int i = 0; i < j; ++i) {
    const double c = fg[L.cs(i)], s = fg[L.sn(i)];
    const double a = col[i], b = col[i + 1];
    col[i] = c * a + s * b;
    col[i + 1] = -s * a + c * b;
  }
  const double a = col[j], b = col[j + 1];
  const double r = hypot(a, b);
  bool bad = !isfinite(r) || !isfinite(wn);
  double c = 1.0, s = 0.0;
  if (r > 0.0) {
    c = a / r;
    s = b / r;
  } else {
    bad = true;  // a zero column: the preconditioned operator is singular on this vector
  }
  fg[L.cs(j)] = c;
  fg[L.sn(j)] = s;
  col[j] = r;
  col[j + 1] = 0.0;
  const double gj = fg[L.g(j)];
  fg[L.g(j)] = c * gj;
  fg[L.g(j + 1)] = -s * gj;
  const double res = fabs(fg[L.g(j + 1)]);
  if (bad) *flags |= 16;
  ctl[0] = j + 1;
  const int conv = !bad && (res <= tol || wn == 0.0);
  ctl[1] = conv;
  const bool stop = conv || bad || j + 1 >= ctl[3];
  if (in_graph) cudaGraphSetConditional(loop, stop ? 0u : 1u);
  if (stop || !in_graph) p.host.put(j + 1, conv, ctl[3], *flags, sc[wn2_slot]);
}
// H[i][j] = V_i . w for i <= j = ctl[0]: blockIdx.y takes the vectors y, y +
// gridDim.y, ...; each vector's block partials (part[i gridDim.x + block]) are
// added in order by the vector's last block (tickets, zero between launches)
constexpr int kDotRows = 8;
__global__ void __launch_bounds__(kBlock) fg_dots(int n, const float* V, const float* w,
                                                  const int* ctl, double* part,
                                                  unsigned* tickets, FgLayout L, double* __restrict__ fg) {
  pdl_begin();
  __shared__ bool last;
  const int j = ctl[0];
  for (int vi = blockIdx.y; vi <= j; vi += gridDim.y) {
    const float* v = V + (size_t)vi * n;
    double acc[1] = {0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
      acc[0] += (double)v[i] * (double)w[i];
    block_sum<1>(acc);
    if (threadIdx.x == 0) {
      part[(size_t)vi * gridDim.x + blockIdx.x] = acc[0];
      __threadfence();
      last = atomicAdd(tickets + vi, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (last) {
      __threadfence();
      acc[0] = 0.0;
      for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x) acc[0] += __ldcg(part + (size_t)vi * gridDim.x + b);
      block_sum<1>(acc);
      if (threadIdx.x == 0) {
        tickets[vi] = 0u;
        fg[L.H(vi, j)] = acc[0];
      }
    }
    __syncthreads();
  }
}
// w -= sum_{i <= j} H[i][j] V_i (FP64 sums, FP32 storage) and ||w||^2, whose
// last block then takes the Givens step
__global__ void __launch_bounds__(kBlock) fg_orth(int n, const float* V, double* fg,
                                                  FgLayout L, float* w, double* part,
                                                  unsigned* ticket, FgScalars a) {
  pdl_begin();
  __shared__ bool last;
  const int j = a.ctl[0];
  const double* h = fg + L.H(0, j);
  double acc[1] = {0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double s = (double)w[i];
    for (int q = 0; q <= j; ++q) s -= h[q] * (double)V[(size_t)q * n + i];
    const float f = (float)s;
    w[i] = f;
    acc[0] += (double)f * (double)f;
  }
  block_sum<1>(acc);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = acc[0];
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  acc[0] = 0.0;
  for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x) acc[0] += __ldcg(part + b);
  block_sum<1>(acc);
  if (threadIdx.x == 0) {
    *ticket = 0u;
    a.sc[a.wn2_slot] = acc[0];
    fg_givens(fg, L, a);
  }
}
// v = w / ||w|| (zero when ||w|| = 0) into V[ctl[0]] and into the next
// preconditioner input; with x1 also the first step of its fine pre-smoother
__global__ void fg_normalize(int n, const float* w, const double* sc, int wn_slot,
                             const int* ctl, float* __restrict__ V, float* __restrict__ in,
                             const float* __restrict__ den0, float w0, float* __restrict__ x1) {
  pdl_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double wn = sc[wn_slot];
  const float v = wn > 0.0 ? (float)((double)w[i] / wn) : 0.0f;
  V[(size_t)ctl[0] * n + i] = v;
  in[i] = v;
  if (x1) x1[i] = w0 * v / den0[i];
}
// start of a pass: g = (1, 0, ...) (the loop's scalars: loop_start)
__global__ void fg_start(double* __restrict__ fg, FgLayout L) {
  for (int q = 0; q <= L.m; ++q) fg[L.g(q)] = q == 0 ? 1.0 : 0.0;
}
// y = R^-1 g over the k = ctl[0] columns built (back substitution, FP64)
__global__ void fg_backsolve(double* __restrict__ fg, FgLayout L, const int* __restrict__ ctl) {
  const int k = ctl[0];
  for (int i = k - 1; i >= 0; --i) {
    double s = fg[L.g(i)];
    for (int q = i + 1; q < k; ++q) s -= fg[L.H(i, q)] * fg[L.y(q)];
    const double d = fg[L.H(i, i)];
    fg[L.y(i)] = d != 0.0 ? s / d : 0.0;
  }
}
// x += scale sum_{i < k} y_i Z_i  (FP64 sums into the FP64 iterate)
__global__ void fg_combine(int n, const float* __restrict__ Z, const double* __restrict__ fg, FgLayout L,
                           const int* __restrict__ ctl, double scale, double* __restrict__ x) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int k = ctl[0];
  double s = 0.0;
  for (int q = 0; q < k; ++q) s += fg[L.y(q)] * (double)Z[(size_t)q * n + i];
  x[i] += scale * s;
}

// ---------------------------------------------------------------------------
// Galerkin initial guess over K earlier corrections y_0..y_{K-1} (FP64),
// with w_a = A_a y_a kept from the solve that made y_a (A_a: the pressure
// operator of that SIMPLE iteration; w = b - r of its last FP64 defect, so
// it costs nothing): solve G c = f with G_ab = y_a . w_b (a <= b, mirrored)
// and f_a = y_a . b, then x = sum c_a y_a.  The operator changes slowly from
// one SIMPLE iteration to the next, so G is close to the Galerkin matrix of
// the current operator; the residual of x is then evaluated exactly, so the
// guess only changes the starting point, never the FP64 stopping test.
// ---------------------------------------------------------------------------
constexpr int kMaxGuess = 8;
// partials, per block: G (upper triangle, row-major a <= b) then f
template <int K>
__global__ void __launch_bounds__(kBlock) guess_dots(int n, const double* Y, const double* W,
                                                     const double* b, double* __restrict__ part) {
  pdl_begin();
  constexpr int NG = K * (K + 1) / 2 + K;
  double acc[NG];
#pragma unroll
  for (int q = 0; q < NG; ++q) acc[q] = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double y[K], w[K];
#pragma unroll
    for (int a = 0; a < K; ++a) {
      y[a] = Y[(size_t)a * n + i];
      w[a] = W[(size_t)a * n + i];
    }
    const double bi = b[i];
    int q = 0;
#pragma unroll
    for (int a = 0; a < K; ++a)
#pragma unroll
      for (int c = a; c < K; ++c) acc[q++] += y[a] * w[c];
#pragma unroll
    for (int a = 0; a < K; ++a) acc[q++] += y[a] * bi;
  }
  write_partials<NG>(acc, part);
}
// x = sum c_a y_a
template <int K>
struct GuessCoef {
  double c[K];
};
template <int K>
__global__ void guess_combine(int n, const double* Y, GuessCoef<K> coef, double* __restrict__ x) {
  pdl_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double xs = 0.0;
#pragma unroll
  for (int a = 0; a < K; ++a) xs += coef.c[a] * Y[(size_t)a * n + i];
  x[i] = xs;
}
// the stored product of a new correction: w = b - r (= A x for r = b - A x)
__global__ void guess_store(int n, const double* x, const double* b,
                            const double* r, double* __restrict__ y, double* __restrict__ w) {
  pdl_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  y[i] = x[i];
  w[i] = b[i] - r[i];
}

}  // namespace k
}  // namespace nds
