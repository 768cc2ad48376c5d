// sm_100a kernels of the SIMPLE hot path.  All kernels are deterministic:
// every output element is owned by one thread, group or warp, and every
// reduction goes through fixed-order block partials (no floating atomics).
//
// T is the storage/arithmetic type of states, operators and AMG data
// (double for the FP64 path, float for FP32); reductions and Krylov scalars
// are double in both, as in the reference (gpu/serial_cuda/precision.hpp:7-36).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "../host/fem.hpp"
#include "common.cuh"

namespace nds {
namespace k {

// ---------------------------------------------------------------------------
// block partial reductions -> out[NV] (single block, fixed order)
// ---------------------------------------------------------------------------
template <int NV>
__global__ void reduce_partials(const double* part, int nblocks, double* __restrict__ out) {
  pdl_begin();
  double v[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = 0.0;
  for (int b = threadIdx.x; b < nblocks; b += blockDim.x)
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] += part[(size_t)b * NV + k];
  block_sum<NV>(v);
  if (threadIdx.x == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) out[k] = v[k];
}

template <int NV>
__device__ __forceinline__ void write_partials(double (&v)[NV], double* part) {
  block_sum<NV>(v);
  if (threadIdx.x == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) part[(size_t)blockIdx.x * NV + k] = v[k];
}

// The velocity state is stored interleaved, component d of dof g at
// u[kVel g + d]: the momentum sweep, the cell pass and the continuity
// residual gather all three components of a dof, which then share a sector.
// Kernels take the three component pointers u, u + 1, u + 2.
constexpr int kVel = 3;

// u[3 i + d] = a_d[i] for the components given (null: left as is)
template <class T>
__global__ void interleave3(int n, const T* __restrict__ a0, const T* __restrict__ a1, const T* __restrict__ a2,
                            T* __restrict__ u) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (a0) u[kVel * (size_t)i] = a0[i];
  if (a1) u[kVel * (size_t)i + 1] = a1[i];
  if (a2) u[kVel * (size_t)i + 2] = a2[i];
}
template <class T>
__global__ void deinterleave3(int n, const T* __restrict__ u, T* __restrict__ a0, T* __restrict__ a1,
                              T* __restrict__ a2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  a0[i] = u[kVel * (size_t)i];
  a1[i] = u[kVel * (size_t)i + 1];
  a2[i] = u[kVel * (size_t)i + 2];
}

// ---------------------------------------------------------------------------
// Momentum assembly (a9 + a10 + a11 + a12) in two passes
//
//   A[i,:]  = K[i,:] + sum_{(c,a) incident to i} C_c[a,:]           (convection, lagged u)
//   conv_i  = - sum C_c[a,b] u_fixed(b)                              (Dirichlet columns)
//   delta_i = (1/alpha_u - 1) sum_k |A[i,k]|, A[i,i] += delta_i     (row-L1 relaxation)
//   diag_i  = A[i,i], rau_i = rau_scale / A[i,i]
//   b_d[i]  = s_d[i] + conv_d[i] + (B^T p)_d[i] + delta_i u_d[i]
// with C_c[a,b] = det_c sum_m sum_j ur[m][j] T[a][m][b][j],
//      ur[m][j] = sum_d u_d(m) invJ_c[j][d].
// Reference: h7_momentum_assembly.cuh:16-85, h4_kernels.cuh:10-56,
// g5e_fp32_kernels.cuh:78-85 and :97-105, h8_precomputed_b.cuh:93-114.
//
// Pass 1 (mom_cell_conv, cell-owned) evaluates each cell's 8x8 convection
// block once.  Pass 2 (mom_assemble, row-owned) builds every velocity row in
// shared memory from K and the blocks of its incident cells, visited in
// ascending cell order, so every A entry is summed in a fixed order (K
// first) with no atomics; relaxation, diag, rAU, B^T p and the RHS follow in
// the same pass.
// ---------------------------------------------------------------------------

// Cell pass: each cell's 8x8 convection block, row a of it written to C[8 z + b],
// z the incidence (c, a) in the velocity rows' incidence lists, so that a
// row's blocks lie contiguous; the cell's pressure goes to pz[z] for the B^T p
// terms of the row pass.
//
// Four lanes a cell, lane i with the columns of
// vertex i and of the bubble opposite to it.  With the velocity in
// barycentric components s_k(m) = u_m . grad lambda_k (s_0 = -(s_1 + s_2 +
// s_3)), a vertex column needs one mass matrix, C[a][i] = det sum_m M[a][m]
// s_i(m), and a bubble column three tensors, C[a][4+i] = det sum_(k != i)
// sum_m N_ik[a][m] s_k(m) with N_ik[a][m] = int phi_a phi_m dphi_(4+i)/dlambda_k;
// M and N are symmetric in (a, m).  So a cell takes 1024 multiply-adds instead
// of 1536, and a lane reads each of the 36 symmetric table records (its three
// N and M, two 16-byte loads) once for both (a, m) and (m, a): 9 loads of a
// warp per cell where the 8-lane form takes 48, which bound it (shared-memory
// stalls).  Bound by the L1 / shared-memory pipe (80 % busy at 383k cells: the
// records, then the scattered 8-value rows), with 16 warps of 128 registers an
// SM; the FP64 pipe is 22 % busy, DRAM 23 %.  Assembly at 1.23M cells 1.55 ->
// 1.31 ms, at 404k 0.50 -> 0.43, at 40k 0.079 -> 0.070.
template <class T>
__device__ __forceinline__ void conv_record(const T* __restrict__ t, T& n0, T& n1, T& n2, T& mm) {
  if constexpr (sizeof(T) == 8) {
    const double2 a = reinterpret_cast<const double2*>(t)[0], b = reinterpret_cast<const double2*>(t)[1];
    n0 = a.x; n1 = a.y; n2 = b.x; mm = b.y;
  } else {
    const float4 a = reinterpret_cast<const float4*>(t)[0];
    n0 = a.x; n1 = a.y; n2 = a.z; mm = a.w;
  }
}
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
// the records (three N and M of column pair i) of the pairs a <= m in shared memory
template <class T>
__device__ __forceinline__ void conv_load(T* __restrict__ sN, const T* __restrict__ table) {
  for (int e = threadIdx.x; e < kConvTable; e += blockDim.x) sN[e] = table[e];
}
template <class T>
__global__ void __launch_bounds__(kBlock, 2) mom_cell_conv(int nc, const int32_t* __restrict__ ref,
                                                            const T* __restrict__ fixed, const T* __restrict__ u0,
                                                            const T* __restrict__ u1, const T* __restrict__ u2,
                                                            const T* __restrict__ invJ, const T* __restrict__ det,
                                                            const T* __restrict__ table,
                                                            const int32_t* __restrict__ zpos, T* __restrict__ C,
                                                            const T* __restrict__ p, T* __restrict__ pz) {
  __shared__ __align__(16) T sN[kConvTable];
  conv_load(sN, table);
  __syncthreads();
  const int i = threadIdx.x & 3;
  const unsigned mask = 0xFu << (threadIdx.x & 28);
  const int groups = blockDim.x >> 2;
  for (int c = blockIdx.x * groups + (threadIdx.x >> 2); c < nc; c += gridDim.x * groups) {
    int g[2];
    T r[2][3];
#pragma unroll
    for (int h = 0; h < 2; ++h) g[h] = ref[8 * (size_t)c + 4 * h + i];
    T I[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) I[k] = invJ[9 * (size_t)c + k];
    const T dc = det[c], pc = p[c];
    int zl[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) zl[h] = zpos[8 * (size_t)c + 4 * h + i];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      T q0, q1, q2;
      if (g[h] >= 0) {
        q0 = u0[kVel * (size_t)g[h]];
        q1 = u1[kVel * (size_t)g[h]];
        q2 = u2[kVel * (size_t)g[h]];
      } else {
        const T* f = fixed + 3 * (size_t)(-g[h] - 1);
        q0 = f[0];
        q1 = f[1];
        q2 = f[2];
      }
#pragma unroll
      for (int j = 0; j < 3; ++j) r[h][j] = fma(q2, I[3 * j + 2], fma(q1, I[3 * j + 1], q0 * I[3 * j]));
      if (zl[h] >= 0) pz[zl[h]] = pc;
    }
    // A0..A2: s_k of the three k != i (ascending), D: s_i
    T A0[8], A1[8], A2[8], D[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      const T s1 = __shfl_sync(mask, r[m >> 2][0], m & 3, 4), s2 = __shfl_sync(mask, r[m >> 2][1], m & 3, 4),
              s3 = __shfl_sync(mask, r[m >> 2][2], m & 3, 4);
      const T s0 = -(s1 + s2 + s3);
      A0[m] = i == 0 ? s1 : s0;
      A1[m] = i <= 1 ? s2 : s1;
      A2[m] = i <= 2 ? s3 : s2;
      D[m] = i == 0 ? s0 : i == 1 ? s1 : i == 2 ? s2 : s3;
    }
    T cb[8], cv[8];
#pragma unroll
    for (int a = 0; a < 8; ++a) cb[a] = cv[a] = T(0);
    int e = 0;
#pragma unroll
    for (int a = 0; a < 8; ++a) {
#pragma unroll
      for (int m = a; m < 8; ++m, ++e) {
        T n0, n1, n2, mm;
        conv_record(sN + 16 * e + 4 * i, n0, n1, n2, mm);
        cb[a] = fma(n2, A2[m], fma(n1, A1[m], fma(n0, A0[m], cb[a])));
        cv[a] = fma(mm, D[m], cv[a]);
        if (m > a) {
          cb[m] = fma(n2, A2[a], fma(n1, A1[a], fma(n0, A0[a], cb[m])));
          cv[m] = fma(mm, D[a], cv[m]);
        }
      }
    }
#pragma unroll
    for (int a = 0; a < 8; ++a) {
      const int za = __shfl_sync(mask, zl[a >> 2], a & 3, 4);
      if (za >= 0) {
        C[8 * (size_t)za + i] = cv[a] * dc;
        C[8 * (size_t)za + 4 + i] = cb[a] * dc;
      }
    }
  }
}

// Laminar SUPG terms, implicit form (h7_momentum_assembly.cuh:100-226; host
// twin g4_host.hpp:324-419), added to the rows the cell pass wrote:
//   S[a][b] = sum_q tau_q w_q det (adv_q . grad phi_a) strong_b(q),
//   strong_b = adv . grad phi_b (- nu lap phi_b for the bubbles),
//   tau_q = tau_scale / sqrt(max(4 |adv_q|^2 / h^2 + magic (4 nu / h^2)^2, 1e-30)),
// over the 64-point collapsed rule (rule: 64 x (lambda0..3, weight)).
// With sigma_k = adv . grad lambda_k every adv . grad phi_a is a few products
// of sigma and lambda, so a point is given by sigma_1..3 and its weight: of
// the four lanes of a cell each prepares every fourth point (velocity from
// shared memory, square root and division), the lanes exchange the four
// values, and lane i adds the columns of vertex i and of the bubble opposite
// to it.  The FP64 pipe is 47 % busy at 35k cells, the rest is the latency of
// its chains (16 warps of 124 registers an SM): assembly with these terms takes
// 0.132 ms there, 0.288 when every lane of eight evaluated the basis gradients
// at every point.
struct SupgArgs {
  double nu, tau_scale, magic;
};
template <class T>
__global__ void __launch_bounds__(kBlock, 2) mom_cell_supg(int nc, const int32_t* __restrict__ ref,
                                                           const T* __restrict__ fixed, const T* __restrict__ u0,
                                                           const T* __restrict__ u1, const T* __restrict__ u2,
                                                           const T* __restrict__ invJ, const T* __restrict__ det,
                                                           const int32_t* __restrict__ zpos, T* __restrict__ C,
                                                           const T* __restrict__ rule, const T* __restrict__ h2,
                                                           SupgArgs sa) {
  constexpr int kCells = kBlock / 4;
  __shared__ T sr[64][13];          // lambda0..3, weight, phi_0..7
  __shared__ T su[kCells][8][3];    // velocities of the block's cells
  for (int q = threadIdx.x; q < 64; q += blockDim.x) {
    T l[4];
    for (int k = 0; k < 4; ++k) sr[q][k] = l[k] = rule[5 * q + k];
    sr[q][4] = rule[5 * q + 4];
    for (int k = 0; k < 4; ++k) {
      sr[q][5 + k] = l[k];
      const T a = k == 0 ? l[1] : l[0], b = k <= 1 ? l[2] : l[1], c = k <= 2 ? l[3] : l[2];
      sr[q][9 + k] = T(27) * a * b * c;
    }
  }
  __syncthreads();
  const int i = threadIdx.x & 3, slot = threadIdx.x >> 2;
  const unsigned mask = 0xFu << (threadIdx.x & 28);
  const int j0 = i == 0 ? 1 : 0, j1 = i <= 1 ? 2 : 1, j2 = i <= 2 ? 3 : 2;  // the vertices of face i
  const T nu = T(sa.nu);
  for (int c = blockIdx.x * kCells + slot; c < nc; c += gridDim.x * kCells) {
    int zl[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int m = 4 * h + i, g = ref[8 * (size_t)c + m];
      zl[h] = zpos[8 * (size_t)c + m];
      if (g >= 0) {
        su[slot][m][0] = u0[kVel * (size_t)g];
        su[slot][m][1] = u1[kVel * (size_t)g];
        su[slot][m][2] = u2[kVel * (size_t)g];
      } else {
        const T* f = fixed + 3 * (size_t)(-g - 1);
        su[slot][m][0] = f[0];
        su[slot][m][1] = f[1];
        su[slot][m][2] = f[2];
      }
    }
    T I[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) I[k] = invJ[9 * (size_t)c + k];
    const T dc = det[c], h = h2[c], diff = T(4) * nu / h, base = T(sa.magic) * diff * diff;
    // products of the gradients of face i's vertices (grad lambda_0 = -(sum of the others))
    auto grad = [&](int k, int d) { return k == 0 ? -(I[d] + I[3 + d] + I[6 + d]) : I[3 * (k - 1) + d]; };
    T g01 = 0, g02 = 0, g12 = 0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const T a = grad(j0, d), b = grad(j1, d), e = grad(j2, d);
      g01 += a * b;
      g02 += a * e;
      g12 += b * e;
    }
    __syncwarp(mask);
    T cv[8], cb[8];
#pragma unroll
    for (int a = 0; a < 8; ++a) cv[a] = cb[a] = T(0);
    for (int q4 = 0; q4 < 64; q4 += 4) {
      // this lane's point
      T a0 = 0, a1 = 0, a2 = 0;
#pragma unroll
      for (int m = 0; m < 8; ++m) {
        const T ph = sr[q4 + i][5 + m];
        a0 += su[slot][m][0] * ph;
        a1 += su[slot][m][1] * ph;
        a2 += su[slot][m][2] * ph;
      }
      const T den = fmax(T(4) * (a0 * a0 + a1 * a1 + a2 * a2) / h + base, T(1e-30));
      const T wq = T(sa.tau_scale) / sqrt(den) * sr[q4 + i][4] * dc;
      const T p1 = a0 * I[0] + a1 * I[1] + a2 * I[2], p2 = a0 * I[3] + a1 * I[4] + a2 * I[5],
              p3 = a0 * I[6] + a1 * I[7] + a2 * I[8];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const T w = __shfl_sync(mask, wq, t, 4), s1 = __shfl_sync(mask, p1, t, 4), s2 = __shfl_sync(mask, p2, t, 4),
                s3 = __shfl_sync(mask, p3, t, 4), s0 = -(s1 + s2 + s3);
        const T* l = sr[q4 + t];
        const T l0 = l[0], l1 = l[1], l2 = l[2], l3 = l[3];
        T st[8];
        st[0] = s0;
        st[1] = s1;
        st[2] = s2;
        st[3] = s3;
        st[4] = T(27) * (l2 * l3 * s1 + l1 * l3 * s2 + l1 * l2 * s3);
        st[5] = T(27) * (l2 * l3 * s0 + l0 * l3 * s2 + l0 * l2 * s3);
        st[6] = T(27) * (l1 * l3 * s0 + l0 * l3 * s1 + l0 * l1 * s3);
        st[7] = T(27) * (l1 * l2 * s0 + l0 * l2 * s1 + l0 * l1 * s2);
        const T lap = T(54) * (l[j2] * g01 + l[j1] * g02 + l[j0] * g12);
        const T sv = i == 0 ? st[0] : i == 1 ? st[1] : i == 2 ? st[2] : st[3];
        const T sb = (i == 0 ? st[4] : i == 1 ? st[5] : i == 2 ? st[6] : st[7]) - nu * lap;
#pragma unroll
        for (int a = 0; a < 8; ++a) {
          const T ta = w * st[a];
          cv[a] += ta * sv;
          cb[a] += ta * sb;
        }
      }
    }
#pragma unroll
    for (int a = 0; a < 8; ++a) {
      const int za = __shfl_sync(mask, zl[a >> 2], a & 3, 4);
      if (za >= 0) {
        C[8 * (size_t)za + i] += cv[a];
        C[8 * (size_t)za + 4 + i] += cb[a];
      }
    }
    __syncwarp(mask);  // the slot's velocities are read no more
  }
}

template <class T>
struct MomArgs {
  int nrows;
  const int2* __restrict__ span;        // row i's (begin, end) in the colour-ordered storage
  const int32_t* __restrict__ dpos;     // diagonal position (absolute)
  const T* __restrict__ K;              // persistent diffusion values
  const int32_t* __restrict__ inc_off;  // row -> incident (cell,a)
  const uint32_t* __restrict__ inc;     // (cell << 3) | a
  const int32_t* __restrict__ ref;      // 8 per cell
  const uint8_t* __restrict__ slot;     // 64 per cell
  const T* C;              // 8 per incidence: convection rows from mom_cell_conv
  const uint8_t* __restrict__ slotz;    // 8 per incidence: slot[c][a][b] of incidence (c, a)
  const T* __restrict__ Bz;             // 3 per incidence: B[c][a]
  const T* pz;             // per incidence: p_c (written by the cell pass)
  const uint8_t* __restrict__ fixz;     // per incidence: bit b set when dof b of the cell is fixed
  const T* __restrict__ bco;            // 24 per cell
  const T* __restrict__ fixed;          // 3 per fixed slot
  const T* __restrict__ u0;
  const T* __restrict__ u1;
  const T* __restrict__ u2;
  const T* __restrict__ p;
  const T* __restrict__ s0;
  const T* __restrict__ s1;
  const T* __restrict__ s2;
  // fused form (no cell pass): C rows are evaluated per incidence
  const T* __restrict__ invJ;           // 9 per cell
  const T* __restrict__ det;            // 1 per cell
  const T* __restrict__ table;          // convection records (conv_table)
  T alpha_u, rau_scale;
  int row_cap;                          // shared row buffer length per group
  T* __restrict__ A;
  T* __restrict__ delta;
  T* __restrict__ diag;
  T* __restrict__ rau;
  T* __restrict__ b0;
  T* __restrict__ b1;
  T* __restrict__ b2;
};

// 8 lanes per velocity row; lane b adds column b of each incident block.
// Convection entries C_c[a][lane8] of one incidence (cell c, basis a), the
// same expressions and order as mom_cell_conv: lane m maps the velocity of
// basis m by J^-1, the group shares the eight mapped velocities, lane b sums
// over m.  ga: this lane's DOF of cell c (ref[8 c + lane8]).
template <class T>
__device__ __forceinline__ T conv_entry(const MomArgs<T>& g, const T* __restrict__ sN, int c, int a, int ga,
                                        int lane8, unsigned gmask) {
  T q0, q1, q2;
  if (ga >= 0) {
    q0 = g.u0[kVel * (size_t)ga];
    q1 = g.u1[kVel * (size_t)ga];
    q2 = g.u2[kVel * (size_t)ga];
  } else {
    const T* f = g.fixed + 3 * (size_t)(-ga - 1);
    q0 = f[0];
    q1 = f[1];
    q2 = f[2];
  }
  const T* I = g.invJ + 9 * (size_t)c;
  T r[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) r[j] = fma(q2, I[3 * j + 2], fma(q1, I[3 * j + 1], q0 * I[3 * j]));
  const int i = lane8 & 3;
  T cb = 0, cv = 0;
#pragma unroll
  for (int m = 0; m < 8; ++m) {
    const T s1 = __shfl_sync(gmask, r[0], m, 8), s2 = __shfl_sync(gmask, r[1], m, 8), s3 = __shfl_sync(gmask, r[2], m, 8);
    const T s0 = -(s1 + s2 + s3);
    const T A0 = i == 0 ? s1 : s0, A1 = i <= 1 ? s2 : s1, A2 = i <= 2 ? s3 : s2;
    const T D = i == 0 ? s0 : i == 1 ? s1 : i == 2 ? s2 : s3;
    const int lo = a < m ? a : m, hi = a < m ? m : a;
    T n0, n1, n2, mm;
    conv_record(sN + 16 * (lo * 8 - lo * (lo - 1) / 2 + hi - lo) + 4 * i, n0, n1, n2, mm);
    cb = fma(n2, A2, fma(n1, A1, fma(n0, A0, cb)));
    cv = fma(mm, D, cv);
  }
  const T dc = g.det[c];
  return mul_rn(lane8 < 4 ? cv : cb, dc);  // rounded here: the cell pass stores the product
}

// FUSED 0: the row pass of the two-pass assembly; each velocity row reads
// its incident cells' convection rows, which the cell pass wrote contiguous
// in incidence order, kAsmAhead at a time.  FUSED 1: C rows evaluated per
// incidence (conv_entry) instead, with the reference tensor staged in shared
// memory after the row buffers (no cell pass).  Both add the same values in
// the same order.
constexpr int kAsmAhead = 4;
template <class T, int FUSED = 0>
__global__ void __launch_bounds__(kBlock) mom_assemble(MomArgs<T> g) {
  pdl_begin();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* sRow = reinterpret_cast<T*>(smem_raw);  // groups * row_cap
  const int tid = threadIdx.x;
  const int lane8 = tid & 7;
  const int grp = tid >> 3;
  const int groups = blockDim.x >> 3;
  T* buf = sRow + (size_t)grp * g.row_cap;
  T* sT = sRow + (size_t)groups * g.row_cap;
  if (FUSED) {
    conv_load(sT, g.table);
    __syncthreads();
  }
  const unsigned gmask = group8_mask();
  for (int i = blockIdx.x * groups + grp; i < g.nrows; i += gridDim.x * groups) {
    const int2 sp = g.span[i];
    const int rb = sp.x, len = sp.y - sp.x;
    for (int k = lane8; k < len; k += 8) buf[k] = g.K[rb + k];
    __syncwarp(gmask);
    T conv0 = 0, conv1 = 0, conv2 = 0, bt0 = 0, bt1 = 0, bt2 = 0;
    const int z0 = g.inc_off[i], z1 = g.inc_off[i + 1];
    if (FUSED == 1) {
      for (int z = z0; z < z1; ++z) {
        const uint32_t pa = g.inc[z];
        const int ca = (int)(pa >> 3), aa = (int)(pa & 7u);
        const int ga = g.ref[8 * (size_t)ca + lane8];
        const int sa = g.slot[64 * (size_t)ca + 8 * aa + lane8];
        const T va = conv_entry<T>(g, sT, ca, aa, ga, lane8, gmask);
        if (ga >= 0) {
          buf[sa] += va;
        } else {
          const T* f = g.fixed + 3 * (size_t)(-ga - 1);
          conv0 -= va * f[0];
          conv1 -= va * f[1];
          conv2 -= va * f[2];
        }
        if (lane8 == 0) {
          const T pv = g.p[ca];
          const T* B = g.bco + 24 * (size_t)ca + 3 * aa;
          bt0 += B[0] * pv;
          bt1 += B[1] * pv;
          bt2 += B[2] * pv;
        }
        __syncwarp(gmask);
      }
    }
    if (FUSED == 0) {
      // B^T p: lane d < 3 sums component d over the row's incidences in
      // incidence order (B and p contiguous per row); lane 0 then takes the
      // other two components
      {
        T btd = 0;
        if (lane8 < 3)
          for (int z = z0; z < z1; ++z) btd += g.Bz[3 * (size_t)z + lane8] * g.pz[z];
        const T t1 = __shfl_sync(gmask, btd, 1, 8), t2 = __shfl_sync(gmask, btd, 2, 8);
        if (lane8 == 0) {
          bt0 = btd;
          bt1 = t1;
          bt2 = t2;
        }
      }
      // the row's convection rows, contiguous in incidence order, kAsmAhead
      // at a time; added in incidence order
      for (int zb = z0; zb < z1; zb += kAsmAhead) {
        T cz[kAsmAhead];
        int sz[kAsmAhead];
        uint32_t fm[kAsmAhead];
#pragma unroll
        for (int u = 0; u < kAsmAhead; ++u) {
          const int z = zb + u;
          const bool ok = z < z1;
          cz[u] = ok ? g.C[8 * (size_t)z + lane8] : T(0);
          sz[u] = ok ? g.slotz[8 * (size_t)z + lane8] : 0;
          fm[u] = ok ? g.fixz[z] : 0u;
        }
#pragma unroll
        for (int u = 0; u < kAsmAhead; ++u) {
          if (zb + u < z1) {
            if ((fm[u] >> lane8) & 1u) {
              const uint32_t pa = g.inc[zb + u];
              const int ga = g.ref[8 * (size_t)(pa >> 3) + lane8];
              const T* f = g.fixed + 3 * (size_t)(-ga - 1);
              conv0 -= cz[u] * f[0];
              conv1 -= cz[u] * f[1];
              conv2 -= cz[u] * f[2];
            } else {
              buf[sz[u]] += cz[u];
            }
          }
          __syncwarp(gmask);
        }
      }
    }
    conv0 = group_sum<8>(conv0, gmask);
    conv1 = group_sum<8>(conv1, gmask);
    conv2 = group_sum<8>(conv2, gmask);
    T l1 = 0;
    for (int k = lane8; k < len; k += 8) l1 += fabs(buf[k]);
    l1 = group_sum<8>(l1, gmask);
    const int dl = g.dpos[i] - rb;
    const T de = (T(1) / g.alpha_u - T(1)) * l1;
    __syncwarp(gmask);
    if (lane8 == 0) buf[dl] += de;
    __syncwarp(gmask);
    for (int k = lane8; k < len; k += 8) g.A[rb + k] = buf[k];
    if (lane8 == 0) {
      const T d = buf[dl];
      g.delta[i] = de;
      g.diag[i] = d;
      g.rau[i] = (T(1) / d) * g.rau_scale;
      g.b0[i] = g.s0[i] + conv0 + bt0 + de * g.u0[kVel * (size_t)i];
      g.b1[i] = g.s1[i] + conv1 + bt1 + de * g.u1[kVel * (size_t)i];
      g.b2[i] = g.s2[i] + conv2 + bt2 + de * g.u2[kVel * (size_t)i];
    }
    __syncwarp(gmask);
  }
}

// One multicolour Gauss-Seidel colour pass on the shared momentum matrix,
// three right-hand sides (g5e_fp32_kernels.cuh:106-116).  8 lanes per row.
// The matrix is stored colour by colour (the rows of one colour contiguous,
// each colour's rows in ascending order), so one pass streams one block of
// the matrix; span: the storage range of each of the colour's rows (pad
// entries have the row's own column), rows: their natural indices (their
// right-hand sides, diagonals and unknowns).
// Each lane takes its entries kGsAhead at a time: it loads their columns and
// values, then gathers their unknowns, so a batch's loads are in flight
// together; the diagonal entry and the padding of a batch contribute 0.
// Per lane the entries are summed in the order of the storage, then over
// the 8 lanes.
constexpr int kGsAhead = 2;
template <class T>
__global__ void __launch_bounds__(kBlock, 6) mom_gs_color(int count, const int32_t* __restrict__ rows,
                                                       const int2* __restrict__ span, const int32_t* __restrict__ ci,
                                                       const T* av, const T* diag, const T* b0, const T* b1,
                                                       const T* b2, T* x0, T* x1, T* x2, T omega) {
  pdl_begin();
  const int lane8 = threadIdx.x & 7;
  const int q = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  if (q >= count) return;
  const unsigned gmask = group8_mask();
  const int i = rows[q];
  const int2 sp = span[q];
  const int kb = sp.x, ke = sp.y;
  T d = 0, c0 = 0, c1 = 0, c2 = 0, y0 = 0, y1 = 0, y2 = 0;
  const size_t vi = kVel * (size_t)i;
  if (lane8 == 0) {
    d = diag[i];
    c0 = b0[i];
    c1 = b1[i];
    c2 = b2[i];
    y0 = x0[vi];
    y1 = x1[vi];
    y2 = x2[vi];
  }
  T s0 = 0, s1 = 0, s2 = 0;
  for (int k0 = kb + lane8; k0 < ke; k0 += 8 * kGsAhead) {
    int jj[kGsAhead];
    T aa[kGsAhead];
#pragma unroll
    for (int u = 0; u < kGsAhead; ++u) {
      const int k = k0 + 8 * u;
      jj[u] = k < ke ? ci[k] : i;
      aa[u] = k < ke ? av[k] : T(0);
    }
#pragma unroll
    for (int u = 0; u < kGsAhead; ++u) {
      const T a = jj[u] == i ? T(0) : aa[u];
      const size_t vj = kVel * (size_t)jj[u];
      s0 += a * x0[vj];
      s1 += a * x1[vj];
      s2 += a * x2[vj];
    }
  }
  s0 = group_sum<8>(s0, gmask);
  s1 = group_sum<8>(s1, gmask);
  s2 = group_sum<8>(s2, gmask);
  if (lane8 == 0) {
    const T iv = T(1) / d;
    x0[vi] = (T(1) - omega) * y0 + omega * ((c0 - s0) * iv);
    x1[vi] = (T(1) - omega) * y1 + omega * ((c1 - s1) * iv);
    x2[vi] = (T(1) - omega) * y2 + omega * ((c2 - s2) * iv);
  }
}

// ||b_d||^2 and ||b_d - A u_d||^2 (g5e_fp32_kernels.cuh:117-126); 6 partials per block.
template <class T>
__global__ void __launch_bounds__(kBlock) mom_audit(int n, const int2* __restrict__ span, const int32_t* __restrict__ ci,
                                                    const T* __restrict__ av, const T* __restrict__ b0,
                                                    const T* __restrict__ b1, const T* __restrict__ b2,
                                                    const T* __restrict__ x0, const T* __restrict__ x1,
                                                    const T* __restrict__ x2, double* __restrict__ part) {
  const int lane8 = threadIdx.x & 7;
  const unsigned gmask = group8_mask();
  double acc[6] = {0, 0, 0, 0, 0, 0};
  const int groups_total = (gridDim.x * blockDim.x) >> 3;
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 3; i < n; i += groups_total) {
    T a0 = 0, a1 = 0, a2 = 0;
    const int2 sp = span[i];
    for (int k = sp.x + lane8; k < sp.y; k += 8) {
      const size_t vj = kVel * (size_t)ci[k];
      const T a = av[k];
      a0 += a * x0[vj];
      a1 += a * x1[vj];
      a2 += a * x2[vj];
    }
    a0 = group_sum<8>(a0, gmask);
    a1 = group_sum<8>(a1, gmask);
    a2 = group_sum<8>(a2, gmask);
    if (lane8 == 0) {
      const double db0 = (double)b0[i], db1 = (double)b1[i], db2 = (double)b2[i];
      const double r0 = (double)(b0[i] - a0), r1 = (double)(b1[i] - a1), r2 = (double)(b2[i] - a2);
      acc[0] += db0 * db0;
      acc[1] += db1 * db1;
      acc[2] += db2 * db2;
      acc[3] += r0 * r0;
      acc[4] += r1 * r1;
      acc[5] += r2 * r2;
    }
  }
  write_partials<6>(acc, part);
}

// ---------------------------------------------------------------------------
// Continuity r_c = fixedDiv_c + sum_a B[c][a] . u(ref a)  (h8_precomputed_b.cuh:140-163),
// stored negated as the pressure right-hand side, with sum r^2 partials.
// Component d of velocity dof g is ud[VS g]: VS = kVel for the solver's
// interleaved state, 1 for three separate arrays.
// ---------------------------------------------------------------------------
template <class T, int VS = kVel>
__global__ void __launch_bounds__(kBlock) continuity(int nc, const int32_t* __restrict__ ref, const T* __restrict__ bco,
                                                     const T* __restrict__ fixed_div, const T* u0,
                                                     const T* u1, const T* u2,
                                                     T* __restrict__ rhs, double* __restrict__ part) {
  pdl_begin();
  double acc[1] = {0.0};
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < nc; c += gridDim.x * blockDim.x) {
    T s = fixed_div[c];
    // the cell's 8 dofs and 24 coefficients in 16-byte loads (the records
    // are 32 and 24 * sizeof(T) bytes, so 16-byte aligned)
    int rf[8];
    T B[24];
    {
      const int4* r4 = reinterpret_cast<const int4*>(ref + 8 * (size_t)c);
      const int4 q0 = r4[0], q1 = r4[1];
      rf[0] = q0.x; rf[1] = q0.y; rf[2] = q0.z; rf[3] = q0.w;
      rf[4] = q1.x; rf[5] = q1.y; rf[6] = q1.z; rf[7] = q1.w;
      if constexpr (sizeof(T) == 8) {
        const double2* b2 = reinterpret_cast<const double2*>(bco + 24 * (size_t)c);
#pragma unroll
        for (int k = 0; k < 12; ++k) {
          const double2 v = b2[k];
          B[2 * k] = v.x;
          B[2 * k + 1] = v.y;
        }
      } else {
#pragma unroll
        for (int k = 0; k < 24; ++k) B[k] = bco[24 * (size_t)c + k];
      }
    }
#pragma unroll
    for (int a = 0; a < 8; ++a) {
      const int g = rf[a];
      if (g < 0) continue;
      const size_t vg = (size_t)VS * g;
      s += B[3 * a] * u0[vg] + B[3 * a + 1] * u1[vg] + B[3 * a + 2] * u2[vg];
    }
    const T sr = s;
    acc[0] += (double)sr * (double)sr;
    rhs[c] = -s;
  }
  write_partials<1>(acc, part);
}

// ---------------------------------------------------------------------------
// CSR SpMV family, warp per row (h2b_fine_csr.cuh:579-596, h6_coarse_spmv.cuh:10-32)
// ---------------------------------------------------------------------------
// Lane l of a G-lane group sums entries rb+l, rb+l+G, ... in that order;
// the loads of eight entries are issued before their products are added
// (same order, an eighth of the dependent memory round trips).
// Coarse-level CSR rows (one to a few hundred entries) go to a warp each
// (G = 32), or to 16 lanes on the FP16 copies of the mixed path.  Lane l
// takes entries rb + l + G u; one round of predicated loads (eight per lane:
// columns and values, then the x gathers) covers a row of up to 8 G entries,
// so a row costs three dependent round trips (row bounds, columns and
// values, gathers).  Longer rows take further rounds.
// MT: the stored value type (T, or __half for an FP16 copy of a level whose
// values are scaled by a power of two; the caller multiplies the row sum back).
// CT: the column type (int32 absolute, or int16 deltas to the row).
template <class T, class MT>
__device__ __forceinline__ T load_val(const MT* __restrict__ v, int k) {
  if constexpr (std::is_same<MT, __half>::value) return (T)__half2float(v[k]);
  else return v[k];
}
// column of entry k of row i: absolute (int32) or a 16-bit delta to the row
__device__ __forceinline__ int col_at(const int32_t* __restrict__ ci, int k, int) { return ci[k]; }
__device__ __forceinline__ int col_at(const int16_t* __restrict__ ci, int k, int i) { return i + ci[k]; }
// The entries are constant during a solve: WAIT loads the first round of them
// before pdl_wait().
template <int G, class T, class MT = T, class CT = int32_t, bool WAIT = false>
__device__ __forceinline__ T lane_batched_dot(int rb, int re, const CT* __restrict__ ci, const MT* __restrict__ v,
                                              const T* x, int lane, int i = 0) {
  T s = 0;
  int c[8];
  T a[8];
  auto entries = [&](int k0) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = k0 + u * G;
      c[u] = k < re ? col_at(ci, k, i) : -1;
      a[u] = k < re ? load_val<T, MT>(v, k) : T(0);
    }
  };
  entries(rb + lane);
  if (WAIT) pdl_wait();
  for (int k0 = rb + lane; k0 < re; k0 += 8 * G) {
    T xv[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) xv[u] = c[u] >= 0 ? x[c[u]] : T(0);
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (c[u] >= 0) s += a[u] * xv[u];
    entries(k0 + 8 * G);
  }
  return s;
}
constexpr int kRowLanes = 32;
// live: the group has a row; every thread of the block calls it (it waits for
// the previous kernel after loading the first entries)
template <class T, class MT = T, class CT = int32_t, int GL = kRowLanes>
__device__ __forceinline__ T group_row_dot(const int32_t* __restrict__ rp, const CT* __restrict__ ci,
                                           const MT* __restrict__ v, const T* x, int i, int lane,
                                           unsigned mask, bool live, T vinv = T(1)) {
  const int rb = live ? rp[i] : 0, re = live ? rp[i + 1] : 0;
  T s = group_sum<GL>(lane_batched_dot<GL, T, MT, CT, true>(rb, re, ci, v, x, lane, i), mask);
  if constexpr (!std::is_same<MT, T>::value) s *= vinv;
  return s;
}

// y = A x (GL lanes per row)
template <class T, class MT = T, class CT = int32_t, int GL = kRowLanes>
__global__ void __launch_bounds__(kBlock) spmv(int n, const int32_t* __restrict__ rp, const CT* __restrict__ ci,
                                               const MT* __restrict__ v, const T* x, T* __restrict__ y,
                                               T vinv = T(1)) {
  pdl_trigger();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = t / GL, lane = t % GL;
  const T s = group_row_dot<T, MT, CT, GL>(rp, ci, v, x, i, lane, group_mask<GL>(), i < n, vinv);
  if (i < n && lane == 0) y[i] = s;
}

// r = b - A x  (optionally also r2 = r)
template <class T, class MT = T, class CT = int32_t, int GL = kRowLanes>
__global__ void __launch_bounds__(kBlock) spmv_resid(int n, const int32_t* __restrict__ rp, const CT* __restrict__ ci,
                                                     const MT* __restrict__ v, const T* x,
                                                     const T* b, T* __restrict__ r, T* __restrict__ r2,
                                                     const T* __restrict__ den, T w, T vinv = T(1)) {
  pdl_trigger();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = t / GL, lane = t % GL;
  const T s = group_row_dot<T, MT, CT, GL>(rp, ci, v, x, i, lane, group_mask<GL>(), i < n, vinv);
  if (i < n && lane == 0) {
    // r; r2 = r (den null) or the first Jacobi step w r / den
    const T q = b[i] - s;
    r[i] = q;
    if (den) r2[i] = w * q / den[i];
    else if (r2) r2[i] = q;
  }
}

// Jacobi-type smoothing step: x_out = x_in + w (b - A x_in) / den
template <class T, class MT = T, class CT = int32_t, int GL = kRowLanes>
__global__ void __launch_bounds__(kBlock) spmv_smooth(int n, const int32_t* __restrict__ rp,
                                                      const CT* __restrict__ ci, const MT* __restrict__ v,
                                                      const T* xin, const T* b,
                                                      const T* __restrict__ den, T w, T* __restrict__ xout,
                                                      T* add_to, T vinv = T(1)) {
  pdl_trigger();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = t / GL, lane = t % GL;
  const T s = group_row_dot<T, MT, CT, GL>(rp, ci, v, xin, i, lane, group_mask<GL>(), i < n, vinv);
  if (i < n && lane == 0) {
    // with add_to the step is added to add_to instead of stored in xout
    const T r = b[i] - s;
    const T val = xin[i] + w * r / den[i];
    if (add_to) add_to[i] += val;
    else xout[i] = val;
  }
}

// The same three products on FP64 levels of many rows, with x staged in shared
// memory: a level's numbering keeps a row's columns near the row (at most
// 4,544 away on the 74,540-row level of the 1.23M-cell pipe), so the rows of a
// block read one window of x, which the block copies once, and gather from
// shared memory.  Persistent blocks, 16 lanes a row, ten entries in flight per
// lane, row bounds one row ahead.  win: first and one-past-last column of each
// block's rows.  The explicit levels of that mesh's FP64 V-cycle take 20 us a
// product on average, 25 with the kernel of a lane group per row, which waits
// for the scattered reads of x.  FP16 levels keep that one: windows of packed entries
// gained 1 us a product by themselves but nothing to 26 us were lost an
// iteration, as their shared memory keeps the next launch from starting early.
enum { LEV_Y = 0, LEV_RESID = 1, LEV_SMOOTH = 2 };
// x[lo, hi) into shared memory at the offset lo - lo4, lo4 = lo rounded down to
// a 16-byte boundary: vector loads, eight in flight (x from cudaMalloc, padded
// reads stay inside [lo4, hi))
template <int BLOCK, class T>
__device__ __forceinline__ void stage_window(T* __restrict__ sx, const T* x, int lo4, int hi) {
  constexpr int W = 16 / sizeof(T);
  using V = typename std::conditional<std::is_same<T, float>::value, float4, double2>::type;
  const int nv = (hi - lo4) / W;
  const V* src = reinterpret_cast<const V*>(x + lo4);
  V* dst = reinterpret_cast<V*>(sx);
#pragma unroll 8
  for (int i = threadIdx.x; i < nv; i += BLOCK) dst[i] = src[i];
  for (int i = lo4 + nv * W + threadIdx.x; i < hi; i += BLOCK) sx[i - lo4] = x[i];
}
constexpr int kWinBlock = 512, kWinPerSm = 2, kWinAhead = 10;
template <int MODE, class CT>
__global__ void __launch_bounds__(kWinBlock, kWinPerSm)
    level_window(int n, int rows, const int2* __restrict__ win, const int32_t* __restrict__ rp,
                 const CT* __restrict__ ci, const double* __restrict__ v, const double* x,
                 const double* b, const double* __restrict__ den, double w, double* __restrict__ y,
                 double* y2) {
  using T = double;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* sx = reinterpret_cast<T*>(smem_raw);
  pdl_trigger();
  const int r0 = blockIdx.x * rows, r1 = min(n, r0 + rows);
  constexpr int groups = kWinBlock / 16;
  const int lane = threadIdx.x & 15;
  const unsigned mask = group_mask<16>();
  int r = r0 + (threadIdx.x >> 4);
  int rb = 0, re = 0;
  if (r < r1) {
    rb = rp[r];
    re = rp[r + 1];
  }
  const int2 wn = win[blockIdx.x];
  pdl_wait();
  const int lo4 = wn.x & ~(16 / (int)sizeof(T) - 1);
  stage_window<kWinBlock>(sx, x, lo4, wn.y);
  __syncthreads();
  const T* xs = sx - lo4;
  for (; r < r1; r += groups) {
    int nb = 0, ne = 0;
    if (r + groups < r1) {
      nb = rp[r + groups];
      ne = rp[r + groups + 1];
    }
    T bi = 0, di = 1;
    if (MODE != LEV_Y && lane == 0) {
      bi = b[r];
      if (MODE == LEV_SMOOTH || den) di = den[r];
    }
    T s = 0;
    for (int k0 = rb + lane; k0 < re; k0 += 16 * kWinAhead) {
      int c[kWinAhead];
      T a[kWinAhead];
#pragma unroll
      for (int u = 0; u < kWinAhead; ++u) {
        const int k = k0 + 16 * u;
        c[u] = k < re ? col_at(ci, k, r) : -1;
        a[u] = k < re ? v[k] : T(0);
      }
#pragma unroll
      for (int u = 0; u < kWinAhead; ++u)
        if (c[u] >= 0) s += a[u] * xs[c[u]];
    }
    s = group_sum<16>(s, mask);
    if (lane == 0) {
      if (MODE == LEV_Y) {
        y[r] = s;
      } else if (MODE == LEV_RESID) {
        const T q = bi - s;
        y[r] = q;
        if (den) y2[r] = w * q / di;
        else if (y2) y2[r] = q;
      } else {
        const T val = xs[r] + w * (bi - s) / di;
        if (y2) y2[r] += val;
        else y[r] = val;
      }
    }
    rb = nb;
    re = ne;
  }
}

// ---------------------------------------------------------------------------
// vector kernels (g5e_fp32_kernels.cuh:132-150, vector_kernels.cuh)
// ---------------------------------------------------------------------------
template <class T>
__global__ void jacobi_zero(int n, T w, const T* b, const T* __restrict__ d, T* __restrict__ x) {
  pdl_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] = w * b[i] / d[i];
}
template <class T>
__global__ void axpy(int n, T a, const T* x, T* y) {
  pdl_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] += a * x[i];
}
template <class T>
__global__ void copy(int n, const T* __restrict__ a, T* __restrict__ b) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) b[i] = a[i];
}
template <class T>
__global__ void scale(int n, T s, T* __restrict__ x) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] *= s;
}
template <class T>
__global__ void div_sqrt(int n, const T* __restrict__ x, const T* __restrict__ d, T* __restrict__ y) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = x[i] / sqrt(d[i]);
}
template <class T>
__global__ void power_init(int n, T* __restrict__ v) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    const T g = T(i + 1);
    v[i] = sin(T(0.731) * g) + T(0.27) * cos(T(1.117) * g);
  }
}

// partial sums of x.y
template <class T, class U = T>
__global__ void __launch_bounds__(kBlock) dot(int n, const T* x, const U* y,
                                              double* __restrict__ part) {
  pdl_begin();
  double acc[1] = {0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    acc[0] += (double)x[i] * (double)y[i];
  write_partials<1>(acc, part);
}
// PCG scalar steps on device.  flags bit 1: pAp <= 0 or non-finite; bit 2: rho <= 0 or non-finite.
// sc layout: [0] rho  [1] pq  [2] alpha  [3] rn2  [4] rhon  [5] beta
__device__ __forceinline__ void pcg_alpha_step(double* __restrict__ sc, int* __restrict__ flags) {
  const double pq = sc[1];
  if (!(pq > 0.0) || !isfinite(pq)) {
    *flags |= 1;
    sc[2] = 0.0;
    return;
  }
  sc[2] = sc[0] / pq;
}
// Device-resident PCG loop (one CUDA graph with a conditional while node).
// ctl: [0] iterations done, [1] converged, [2] first iteration pending.
// flags bit 8: initial rho <= 0 or non-finite; bit 4: residual non-finite.
//
// rho step of the loop body: on the first iteration rho = r.z (p = z follows),
// afterwards beta = rho_new / rho.
__device__ __forceinline__ void pcg_rho_step(double* __restrict__ sc, int* __restrict__ flags,
                                             const int* __restrict__ ctl) {
  const double rhon = sc[4];
  if (ctl[2]) {
    if (!(rhon > 0.0) || !isfinite(rhon)) *flags |= 8;
    sc[0] = rhon;
    sc[5] = 0.0;
    return;
  }
  if (!(rhon > 0.0) || !isfinite(rhon)) {
    *flags |= 2;
    sc[5] = 0.0;
    return;
  }
  sc[5] = rhon / sc[0];
  sc[0] = rhon;
}
// p = z on the first iteration, else p = z + beta p
template <class T, class Z = T>
__global__ void p_update_dev(int n, const double* beta_dev, const int* ctl,
                             const Z* z, T* p) {
  pdl_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  p[i] = ctl[2] ? T(z[i]) : T(z[i]) + T(*beta_dev) * p[i];
}
// A loop's end state written straight to page-locked host memory (the host
// reads it after it has waited for the stream), instead of three copies of a
// few bytes behind the loop.
struct HostWords {
  double* rn2;  // ||r||^2
  int* words;   // [0] flags, [4] iterations, [5] converged, [7] cap
  __device__ __forceinline__ void put(int it, int conv, int cap, int flags, double v) const {
    words[0] = flags;
    words[4] = it;
    words[5] = conv;
    words[7] = cap;
    *rn2 = v;
    __threadfence_system();
  }
};
// the scalars a solve starts from, set by its first kernel
struct SolveInit {
  double* sc;
  int* ctl;
  int* flags;
  int r0_slot, target_slot, first, cap;
  double r0, target;
  __device__ __forceinline__ void set() const {
    sc[r0_slot] = r0;
    sc[target_slot] = target;
    ctl[0] = 0;
    ctl[1] = 0;
    ctl[2] = first;
    ctl[3] = cap;
    *flags = 0;
  }
};
// End of the loop body: count the iteration and test ||r|| <= target the way
// the host loop does (sqrt, then compare); stop on convergence, on any flag
// or at the cap ctl[3], set per solve.  The loop always ends: every body pass
// takes this step and the count reaches the cap.  in_graph = 0: launched
// outside a graph (host-driven loop), no condition to set.
__device__ __forceinline__ void pcg_check_step(const double* __restrict__ sc, int rn2_slot, int r0_slot,
                                               int target_slot, int* __restrict__ flags, int* __restrict__ ctl,
                                               cudaGraphConditionalHandle loop, int in_graph, const HostWords& host) {
  const int it = ++ctl[0];
  ctl[2] = 0;
  const double rn = sqrt(sc[rn2_slot]);
  if (!isfinite(rn / fmax(sc[r0_slot], 1e-300))) *flags |= 4;
  const int conv = rn <= sc[target_slot];
  ctl[1] = conv;
  const bool stop = conv || *flags != 0 || it >= ctl[3];
  if (in_graph) cudaGraphSetConditional(loop, stop ? 0u : 1u);
  if (stop || !in_graph) host.put(it, conv, ctl[3], *flags, sc[rn2_slot]);
}
// The scalar step taken with a reduction: rho and beta of PCG (PCG_RHO), alpha
// (PCG_ALPHA), the stopping test (PCG_CHECK) or none (SUM_ONLY).
enum { PCG_RHO = 1, PCG_ALPHA = 2, PCG_CHECK = 3, SUM_ONLY = 4 };
struct PcgScalars {
  double* sc;
  int* flags;
  int* ctl;
  int rn2_slot, r0_slot, target_slot;
  cudaGraphConditionalHandle loop;
  int in_graph;
  HostWords host;
};
// p.q from the block partials of a product that does not reduce them itself
// (as reduce_partials<1>), and the step alpha
__global__ void reduce_alpha(const double* part, int nblocks, double* sc, int* flags) {
  pdl_begin();
  double v[1] = {0.0};
  for (int b = threadIdx.x; b < nblocks; b += blockDim.x) v[0] += part[b];
  block_sum<1>(v);
  if (threadIdx.x == 0) {
    sc[1] = v[0];
    pcg_alpha_step(sc, flags);
  }
}

// The same reduction taken by the kernel that produced the values: every
// block leaves its partial sum, and the block that finishes last (a ticket
// counter) adds the partials in the fixed order of reduce_partials and takes the
// scalar step.  The order of the sums does not depend on which block that
// is.  It saves a launch of 3 to 6 microseconds, a tenth of a PCG iteration
// on small meshes.  blockDim.x = kBlock; every thread of the block calls it.
struct ReduceTail {
  double* part;      // one value per block of the launch
  unsigned* ticket;  // zero between launches
  double* out;
  PcgScalars ps;
};
template <int STEP>
__device__ __forceinline__ void reduce_tail(double value, const ReduceTail& t) {
  __shared__ bool last;
  double v[1] = {value};
  block_sum<1>(v);
  if (threadIdx.x == 0) {
    t.part[blockIdx.x] = v[0];
    __threadfence();
    last = atomicAdd(t.ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  v[0] = 0.0;
  for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x) v[0] += __ldcg(t.part + b);
  block_sum<1>(v);
  if (threadIdx.x == 0) {
    *t.ticket = 0u;
    t.out[0] = v[0];
    if (STEP == PCG_RHO) pcg_rho_step(t.ps.sc, t.ps.flags, t.ps.ctl);
    else if (STEP == PCG_ALPHA) pcg_alpha_step(t.ps.sc, t.ps.flags);
    else if (STEP == PCG_CHECK)
      pcg_check_step(t.ps.sc, t.ps.rn2_slot, t.ps.r0_slot, t.ps.target_slot, t.ps.flags, t.ps.ctl,
                     t.ps.loop, t.ps.in_graph, t.ps.host);
  }
}

// x.y with the reduction tail STEP
template <class T, class U, int STEP>
__global__ void __launch_bounds__(kBlock) dot_step(int n, const T* x, const U* y,
                                                   ReduceTail tail) {
  pdl_begin();
  double acc = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    acc += (double)x[i] * (double)y[i];
  reduce_tail<STEP>(acc, tail);
}

// Start of a pressure solve: r = b, x = 0, and ||b||^2 (SUM_ONLY tail)
template <class T>
__global__ void __launch_bounds__(kBlock) solve_start(int n, const T* b, T* __restrict__ r,
                                                      T* __restrict__ x, ReduceTail tail) {
  pdl_begin();
  double acc = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const T v = b[i];
    r[i] = v;
    x[i] = T(0);
    acc += (double)v * (double)v;
  }
  reduce_tail<SUM_ONLY>(acc, tail);
}
// Start of a Krylov loop from the residual r: the loop's scalars; with rs the
// scaled residual rs = s r in precision S (and rs2 = rs), with x zero = 0;
// with rA the residual in the preconditioner's precision, and with x1 the
// first (diagonal) step of its fine pre-smoother on it, x1 = w0 r / den0.
template <class R, class S, class TA>
__global__ void loop_start(int n, const R* r, double s, S* __restrict__ rs, S* __restrict__ rs2,
                           S* __restrict__ x, TA* __restrict__ rA, const TA* __restrict__ den0, TA w0,
                           TA* __restrict__ x1, SolveInit init) {
  pdl_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) init.set();
  if (i >= n) return;
  const S v = rs ? (S)(s * (double)r[i]) : (S)r[i];
  if (rs) rs[i] = v;
  if (rs2) rs2[i] = v;
  if (x) x[i] = S(0);
  const TA a = TA(v);
  if (rA) rA[i] = a;
  if (x1) x1[i] = w0 * a / den0[i];
}

// x += a p; r -= a q; partial r.r.  a = alpha_dev ? *alpha_dev : alpha.
// With x1: also the first (diagonal) step of the next preconditioner
// application's fine pre-smoother on the new r, x1 = w0 r / den0 (the
// expression of jacobi_zero), and with rA the new r in the preconditioner's
// precision (x1 from it).  STEP PCG_CHECK: the reduction and the stopping
// test by the last block; 0: partials only (to tail.part).
template <class T, class TA, int STEP>
__global__ void __launch_bounds__(kBlock) xr_update(int n, double alpha, const double* alpha_dev,
                                                    const T* p, const T* q,
                                                    T* x, T* r,
                                                    ReduceTail tail, const TA* __restrict__ den0, TA w0,
                                                    TA* __restrict__ x1, TA* __restrict__ rA) {
  pdl_begin();
  const T a = T(alpha_dev ? *alpha_dev : alpha);
  double acc[1] = {0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const T pi = p[i], qi = q[i], xi = x[i], ri = r[i];
    x[i] = xi + a * pi;
    const T rr = ri - a * qi;
    r[i] = rr;
    if (x1) {
      const TA ra = TA(rr);
      if (rA) rA[i] = ra;
      x1[i] = w0 * ra / den0[i];
    }
    acc[0] += (double)rr * (double)rr;
  }
  if (STEP != 0) reduce_tail<STEP>(acc[0], tail);
  else write_partials<1>(acc, tail.part);
}

// ---------------------------------------------------------------------------
// transfers and terminal solve (g5e_fp32_kernels.cuh:140-150)
// ---------------------------------------------------------------------------
// f += P c (one thread per fine row; P in ELL with entry k of row i at
// k nf + i, so a warp's loads of P are coalesced).  Sequential sum over k
// with the loads of eight entries issued ahead (a row of the SA transfers has
// about eight); padding adds 0 c[0].  18.6 us at 1.23M cells in FP32, 22.4
// with four entries ahead.
template <class T>
__global__ void prolong_add(int nf, int pw, const int32_t* __restrict__ pc, const T* __restrict__ pv,
                            const T* c, T* f) {
  pdl_trigger();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const size_t n = (size_t)nf;
  int j[8];
  T a[8];
  auto entries = [&](int k0) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const bool ok = i < nf && k0 + u < pw;
      const size_t o = (size_t)(k0 + u) * n + i;
      j[u] = ok ? pc[o] : -1;
      a[u] = ok ? pv[o] : T(0);
    }
  };
  entries(0);
  pdl_wait();
  if (i >= nf) return;
  const T fi = f[i];
  T s = 0;
  for (int k0 = 0; k0 < pw; k0 += 8) {
    if (k0) entries(k0);
    T x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = j[u] >= 0 ? c[j[u]] : T(0);
#pragma unroll
    for (int u = 0; u < 8; ++u) s += a[u] * x[u];
  }
  f[i] = fi + s;
}

// ---------------------------------------------------------------------------
// Dense form of the V-cycle from a level down: the explicit levels never
// change after setup, so the cycle from level l on is one constant matrix
// M_l.  Its columns are the cycle applied to the unit vectors, all at once on
// row-major n x m blocks (column j of the block is the vector of unit vector
// j): a row of the level matrix is read once for all columns, and the columns
// lie contiguous for the threads.
// ---------------------------------------------------------------------------
// epilogues of block_spmm: the modes of spmv / spmv_resid / spmv_smooth
enum { BLK_Y = 0, BLK_RESID = 1, BLK_SMOOTH = 2 };
template <class T, class MT, class CT, int MODE>
__global__ void __launch_bounds__(kBlock) block_spmm(int n, int m, const int32_t* __restrict__ rp,
                                                     const CT* __restrict__ ci, const MT* __restrict__ v, T vinv,
                                                     const T* __restrict__ x, const T* __restrict__ b,
                                                     const T* __restrict__ den, T w, T* __restrict__ y) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m) return;
  for (int i = blockIdx.y; i < n; i += gridDim.y) {
    T s = 0;
    for (int k = rp[i]; k < rp[i + 1]; ++k) s += load_val<T, MT>(v, k) * x[(size_t)col_at(ci, k, i) * m + j];
    if constexpr (!std::is_same<MT, T>::value) s *= vinv;
    const size_t o = (size_t)i * m + j;
    if (MODE == BLK_Y) y[o] = s;
    else if (MODE == BLK_RESID) y[o] = b[o] - s;
    else y[o] = x[o] + w * (b[o] - s) / den[i];
  }
}
// y += P x, P in ELL (entry k of row i at k n + i)
template <class T>
__global__ void __launch_bounds__(kBlock) block_prolong_add(int n, int m, int pw, const int32_t* __restrict__ pc,
                                                            const T* __restrict__ pv, const T* __restrict__ x,
                                                            T* __restrict__ y) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m) return;
  for (int i = blockIdx.y; i < n; i += gridDim.y) {
    T s = 0;
    for (int k = 0; k < pw; ++k) s += pv[(size_t)k * n + i] * x[(size_t)pc[(size_t)k * n + i] * m + j];
    y[(size_t)i * m + j] += s;
  }
}
// y = A x with a dense n x n A (row stride ld)
template <class T>
__global__ void __launch_bounds__(kBlock) block_dense(int n, int ld, int m, const T* __restrict__ A, const T* __restrict__ x,
                                                      T* __restrict__ y) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m) return;
  for (int i = blockIdx.y; i < n; i += gridDim.y) {
    T s = 0;
    for (int k = 0; k < n; ++k) s += A[(size_t)i * ld + k] * x[(size_t)k * m + j];
    y[(size_t)i * m + j] = s;
  }
}
// y = w b / den by rows; unit blocks; y += x
template <class T>
__global__ void block_jacobi(size_t total, int m, T w, const T* __restrict__ b, const T* __restrict__ den,
                             T* __restrict__ y) {
  const size_t o = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (o < total) y[o] = w * b[o] / den[o / m];
}
template <class T>
__global__ void block_unit(size_t total, int m, T* __restrict__ y) {
  const size_t o = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (o < total) y[o] = T(o / m == o % m ? 1 : 0);
}
template <class T>
__global__ void block_add(size_t total, const T* __restrict__ x, T* __restrict__ y) {
  const size_t o = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (o < total) y[o] += x[o];
}

// y = A x with a dense row-major n x ld A (ld a multiple of 4, rows padded
// with zeros, x readable up to ld): a block of kDenseWarps warps per row, so
// that a few thousand rows of 10 to 40 KB keep every SM's loads in flight;
// 16-byte loads.  Fixed order: lanes, then warps.
// The first entries of a row are loaded before the previous kernel is waited
// for.
constexpr int kDenseWarps = 4;
template <class T>
__global__ void __launch_bounds__(32 * kDenseWarps) dense_rows(int n, int ld, const T* __restrict__ A,
                                                               const T* b, T* __restrict__ x) {
  pdl_trigger();
  constexpr int W = 16 / sizeof(T), step = 32 * kDenseWarps, ahead = 4;
  using V = typename std::conditional<std::is_same<T, float>::value, float4, double2>::type;
  __shared__ T part[kDenseWarps];
  const int i = blockIdx.x;
  const V* a = reinterpret_cast<const V*>(A + (size_t)i * ld);
  const V* bb = reinterpret_cast<const V*>(b);
  T s = 0;
  const int nv = ld / W;
  V p[ahead];
  auto entries = [&](int k0) {
#pragma unroll
    for (int u = 0; u < ahead; ++u) p[u] = k0 + u * step < nv ? a[k0 + u * step] : V{};
  };
  entries(threadIdx.x);
  pdl_wait();
  for (int k0 = threadIdx.x; k0 < nv; k0 += ahead * step) {
    V q[ahead];
#pragma unroll
    for (int u = 0; u < ahead; ++u) q[u] = k0 + u * step < nv ? bb[k0 + u * step] : V{};
#pragma unroll
    for (int u = 0; u < ahead; ++u) {
      if constexpr (W == 4) s += p[u].x * q[u].x + p[u].y * q[u].y + p[u].z * q[u].z + p[u].w * q[u].w;
      else s += p[u].x * q[u].x + p[u].y * q[u].y;
    }
    entries(k0 + ahead * step);
  }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    T r = part[0];
#pragma unroll
    for (int q = 1; q < kDenseWarps; ++q) r += part[q];
    x[i] = r;
  }
}

// multicolour GS colour pass on an AMG level (h8_main_base.cu:205-223)
template <class T>
__global__ void amg_gs_color(int count, const int32_t* __restrict__ rows, const int32_t* __restrict__ rp,
                             const int32_t* __restrict__ ci, const T* __restrict__ v, const T* __restrict__ diag,
                             const T* __restrict__ b, T* __restrict__ x, T omega) {
  const int q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (q >= count) return;
  const int i = rows[q];
  T off = 0;
  for (int k = rp[i] + lane; k < rp[i + 1]; k += 32) {
    const int j = ci[k];
    if (j != i) off += v[k] * x[j];
  }
  off = warp_sum(off);
  if (lane == 0) {
    const T old = x[i];
    const T gs = (b[i] - off) / diag[i];
    x[i] = old + omega * (gs - old);
  }
}

}  // namespace k
}  // namespace nds

namespace nds {
namespace k {

// ---------------------------------------------------------------------------
// Fine Schur operator in sliced ELL with 4-wide lanes (SELL-32x4): rows are
// grouped in slices of 32 (one warp); each row's entries are padded to a
// multiple of 4 and entry k of row i (slice s = i/32, lane l = i%32) lives at
//   base[s] + 128 (k/4) + 4 l + (k%4),
// so every thread reads four consecutive entries of its own row with one
// vector load while the warp's loads stay fully coalesced (512 B of FP32
// values per instruction).  width[s] is the slice's longest row; padding
// entries carry value 0 and the row's own column.  One thread owns a row.
// ---------------------------------------------------------------------------
struct Sell {
  int n;
  const int32_t* __restrict__ base;
  const int32_t* __restrict__ width;
  const int32_t* __restrict__ col;   // absolute columns (used when dcol is null)
  const int16_t* __restrict__ dcol;  // column - row, when every |column - row| < 2^15
};

__device__ __forceinline__ int sell_offset(int base, int lane, int k) { return base + 128 * (k >> 2) + 4 * lane + (k & 3); }

// the four column indices of entries o..o+3 of row i (o a multiple of 4)
template <bool D16>
__device__ __forceinline__ void sell_col4(const Sell& A, int o, int i, int j[4]) {
  if (D16) {
    const short4 d = *reinterpret_cast<const short4*>(A.dcol + o);
    j[0] = i + d.x;
    j[1] = i + d.y;
    j[2] = i + d.z;
    j[3] = i + d.w;
  } else {
    const int4 c = *reinterpret_cast<const int4*>(A.col + o);
    j[0] = c.x;
    j[1] = c.y;
    j[2] = c.z;
    j[3] = c.w;
  }
}
template <class T>
__device__ __forceinline__ void sell_val4(const T* __restrict__ v, int o, T a[4]);
template <>
__device__ __forceinline__ void sell_val4<float>(const float* __restrict__ v, int o, float a[4]) {
  const float4 q = *reinterpret_cast<const float4*>(v + o);
  a[0] = q.x;
  a[1] = q.y;
  a[2] = q.z;
  a[3] = q.w;
}
template <>
__device__ __forceinline__ void sell_val4<double>(const double* __restrict__ v, int o, double a[4]) {
  const double2 p = *reinterpret_cast<const double2*>(v + o);
  const double2 q = *reinterpret_cast<const double2*>(v + o + 2);
  a[0] = p.x;
  a[1] = p.y;
  a[2] = q.x;
  a[3] = q.y;
}
// FP16 operator copy (values scaled by a power of two into FP16 range): four
// values of one 8-byte load, widened
__device__ __forceinline__ void sell_val4h(const __half* __restrict__ v, int o, float a[4]) {
  const uint2 q = *reinterpret_cast<const uint2*>(v + o);
  const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&q.x));
  const float2 hi = __half22float2(*reinterpret_cast<const __half2*>(&q.y));
  a[0] = lo.x;
  a[1] = lo.y;
  a[2] = hi.x;
  a[3] = hi.y;
}
template <class T, class MT>
__device__ __forceinline__ void sell_vals4(const MT* __restrict__ v, int o, T a[4]) {
  if constexpr (std::is_same<MT, __half>::value) sell_val4h(v, o, a);
  else sell_val4<T>(v, o, a);
}
template <bool D16>
__device__ __forceinline__ int sell_col(const Sell& A, int o, int i) {
  if (D16) return i + (int)A.dcol[o];
  return A.col[o];
}

enum SellMode { SELL_Y = 0, SELL_RESID = 1, SELL_SMOOTH = 2, SELL_DOT = 3 };

// Row dot product: entries in batches of 8 (two vector loads of values and
// of columns, then the 8 x gathers), even entries into s0 and odd ones into
// s1; the last w mod 8 entries (and the zero padding) go to s0 in order.
// Fixed order -> deterministic.
template <class T, bool D16, class MT = T>
__device__ __forceinline__ T sell_row(const Sell& A, const MT* __restrict__ v, const T* x, int i) {
  const int s = i >> 5, lane = i & 31;
  const int b = A.base[s];
  const int w = A.width[s];
  const int w8 = w & ~7, wp = (w + 3) & ~3;
  T s0 = 0, s1 = 0;
  int k = 0;
  if constexpr (std::is_same<MT, __half>::value) {
    // the FP16 copy moves 4 B per entry: 16 entries in flight per thread
    // keep as many bytes in flight as 8 entries of the wider formats
    const int w16 = w & ~15;
    for (; k < w16; k += 16) {
      int j[16];
      T a[16];
#pragma unroll
      for (int g4 = 0; g4 < 4; ++g4) {
        const int o = sell_offset(b, lane, k + 4 * g4);
        sell_col4<D16>(A, o, i, j + 4 * g4);
        sell_vals4<T, MT>(v, o, a + 4 * g4);
      }
      T xv[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) xv[u] = x[j[u]];
#pragma unroll
      for (int u = 0; u < 16; u += 2) {
        s0 += a[u] * xv[u];
        s1 += a[u + 1] * xv[u + 1];
      }
    }
  }
  for (; k < w8; k += 8) {
    int j[8];
    T a[8];
    const int o0 = sell_offset(b, lane, k), o1 = o0 + 128;
    sell_col4<D16>(A, o0, i, j);
    sell_col4<D16>(A, o1, i, j + 4);
    sell_vals4<T, MT>(v, o0, a);
    sell_vals4<T, MT>(v, o1, a + 4);
    T xv[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) xv[u] = x[j[u]];
#pragma unroll
    for (int u = 0; u < 8; u += 2) {
      s0 += a[u] * xv[u];
      s1 += a[u + 1] * xv[u + 1];
    }
  }
  for (; k < wp; k += 4) {
    int j[4];
    T a[4];
    const int o = sell_offset(b, lane, k);
    sell_col4<D16>(A, o, i, j);
    sell_vals4<T, MT>(v, o, a);
#pragma unroll
    for (int u = 0; u < 4; ++u) s0 += a[u] * x[j[u]];
  }
  return s0 + s1;
}

// MODE SELL_Y:      y = A x
// MODE SELL_RESID:  y = b - A x (and y2 = y when y2 != null)
// MODE SELL_SMOOTH: y = x + w (b - A x) / den
// MODE SELL_DOT:    y = A x, partials of x.y (grid-stride; blockDim = kBlock)
// MT: the operator's value type (T, or __half for the FP16 copy whose values
// are a s, with vinv = 1 / s: a power of two, so the product is exact)
template <class T, int MODE, bool D16, class MT = T>
__global__ void __launch_bounds__(kBlock, 8) sell_spmv(Sell A, const MT* __restrict__ v, const T* x,
                                                    const T* b, const T* __restrict__ den, T w,
                                                    T* __restrict__ y, T* y2, double* __restrict__ part,
                                                    T vinv = T(1)) {
  pdl_begin();
  if (MODE == SELL_DOT) {
    double acc[1] = {0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < A.n; i += gridDim.x * blockDim.x) {
      T s = sell_row<T, D16, MT>(A, v, x, i);
      if constexpr (!std::is_same<MT, T>::value) s *= vinv;
      y[i] = s;
      acc[0] += (double)x[i] * (double)s;
    }
    write_partials<1>(acc, part);
    return;
  }
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= A.n) return;
  T s = sell_row<T, D16, MT>(A, v, x, i);
  if constexpr (!std::is_same<MT, T>::value) s *= vinv;
  if (MODE == SELL_Y) {
    y[i] = s;
  } else if (MODE == SELL_RESID) {
    // y = r; y2 = r (den null) or the first Jacobi step w r / den
    const T q = b[i] - s;
    y[i] = q;
    if (den) y2[i] = w * q / den[i];
    else if (y2) y2[i] = q;
  } else {
    // smoothing step; with y2 the step is added to y2 instead of stored
    const T val = x[i] + w * (b[i] - s) / den[i];
    if (y2) y2[i] += val;
    else y[i] = val;
  }
}

// Static part of the fine Schur refresh: for every directed contribution q of
// row c (basis a of c, incidence (c2, b) of the shared velocity dof), the
// geometric factor G_q = B[c][a] . B[c2][b].  Evaluated once at setup.
// cs[q]: basis a in bits 0-2 (0xFFFF: pad entry, G = 0); cpk[q] = c2 << 3 | b.
template <class T>
__global__ void refresh_geometry(int nc, const int32_t* __restrict__ coff, const uint32_t* __restrict__ cpk,
                                 const uint16_t* __restrict__ cs, const T* __restrict__ bco, T* __restrict__ G) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nc) return;
  const T* Bc = bco + 24 * (size_t)c;
  for (int q = coff[c]; q < coff[c + 1]; ++q) {
    if (cs[q] == 0xFFFFu) {
      G[q] = T(0);
      continue;
    }
    const int a = cs[q] & 7;
    const uint32_t pk = cpk[q];
    const T* bb = bco + 24 * (size_t)(pk >> 3) + 3 * (pk & 7u);
    G[q] = Bc[3 * a] * bb[0] + Bc[3 * a + 1] * bb[1] + Bc[3 * a + 2] * bb[2];
  }
}

// Fine Schur numeric refresh A_p = B diag(rau) B^T (h8_precomputed_b.cuh:37-91)
// into the SELL layout.  Each value is sum_q rau_{g(c,a_q)} G_q over the
// row's contributions to that entry, in the reference's (basis, incidence)
// order (h2b_fine_csr.cuh:480-520), each product rounded on its own.  The
// contributions of a row are stored as runs, one per fine entry (the row's
// longest runs first), that never straddle a 32-entry chunk; the code word
// cs gives the basis a (bits 0-2), the position in the run (bits 3-5), the
// run's last entry (bit 6) and the entry's slot (bits 7-15); pads are
// 0xFFFF.  The next chunk's code words and factors are loaded before the
// current chunk is summed.
//
// One block of 32 warps per SELL slice, a warp per row, a lane per
// contribution: a shuffle chain sums every run sequentially (the lane at
// position j adds its product to the finished sum of position j-1), so each
// value is the reference's serial sum; no atomics.  The run's last lane
// puts the value into the slice's shared-memory image ([entry][row], row
// stride 33 against bank conflicts), which the block then writes out
// contiguously in SELL order (padding as zeros).  Values go to val
// (operator precision T) and, in the mixed modes, also to valA (AMG precision
// TA) and valH (FP16, scaled by hscale and saturated); the diagonal and L1
// row sums feed the AMG smoothers.
// Launch: blockDim 1024; dynamic shared memory 33 * padded max width * sizeof(T).
constexpr int kRefreshBlock = 1024;
template <class T>
__device__ __forceinline__ T mul_rn(T a, T b);
template <>
__device__ __forceinline__ double mul_rn<double>(double a, double b) { return __dmul_rn(a, b); }
template <>
__device__ __forceinline__ float mul_rn<float>(float a, float b) { return __fmul_rn(a, b); }
template <class T, class TA>
__global__ void __launch_bounds__(kRefreshBlock) sell_refresh(int nc, const int32_t* __restrict__ coff,
                                                              const uint16_t* __restrict__ cs, const T* __restrict__ G,
                                                              const int32_t* __restrict__ ref, const T* __restrict__ rau,
                                                              const int32_t* __restrict__ dslot,
                                                              const int32_t* __restrict__ sbase,
                                                              const int32_t* __restrict__ swidth, T* __restrict__ val,
                                                              TA* __restrict__ valA, TA* __restrict__ diag,
                                                              TA* __restrict__ l1, __half* __restrict__ valH = nullptr,
                                                              float hscale = 1.f) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* sv = reinterpret_cast<T*>(smem_raw);
  __shared__ T sR[32][8];
  const int slice = blockIdx.x;
  const int width = (swidth[slice] + 3) & ~3;  // padded to the 4-wide lanes
  for (int t = threadIdx.x; t < 33 * width; t += blockDim.x) sv[t] = T(0);
  const int lane = threadIdx.x & 31, r = threadIdx.x >> 5;
  const int c = slice * 32 + r;
  const bool live_row = c < nc;
  int qb = 0, qe = 0, ds = -1;
  // the code word and factor of this lane's contribution in the next chunk,
  // loaded one chunk ahead (the first chunk's loads overlap the rAU staging)
  unsigned vn = 0xFFFFu;
  T gn = 0;
  if (live_row) {
    if (lane < 8) {
      const int g = ref[8 * (size_t)c + lane];
      sR[r][lane] = g >= 0 ? rau[g] : T(0);
    }
    qb = coff[c];
    qe = coff[c + 1];
    ds = dslot[c];
    if (qb + lane < qe) {
      vn = cs[qb + lane];
      gn = G[qb + lane];
    }
  }
  __syncthreads();  // image zeroed, rAU of every row staged
  T asum = 0;
  for (int q0 = qb; q0 < qe; q0 += 32) {  // warp-uniform bounds
    const unsigned v = vn;
    const T gq = gn;
    vn = 0xFFFFu;
    gn = 0;
    if (q0 + 32 + lane < qe) {
      vn = cs[q0 + 32 + lane];
      gn = G[q0 + 32 + lane];
    }
    // each product rounded on its own, then summed serially along the run
    const T p = v != 0xFFFFu ? mul_rn<T>(sR[r][v & 7u], gq) : T(0);
    const bool real = v != 0xFFFFu;
    const int pos = real ? (int)((v >> 3) & 7u) : 0;
    const int maxpos = __reduce_max_sync(0xffffffffu, pos);
    T acc = p;
    for (int j = 1; j <= maxpos; ++j) {
      const T up = __shfl_up_sync(0xffffffffu, acc, 1);
      if (pos == j) acc = up + p;
    }
    if (real && (v & 64u)) {
      const int sl = (int)(v >> 7);
      sv[sl * 33 + r] = acc;
      if (sl == ds) diag[c] = TA(acc);
      asum += fabs(acc);
    }
  }
  if (l1 && live_row) {
    asum = warp_sum(asum);
    if (lane == 0) l1[c] = TA(asum);
  }
  __syncthreads();
  const size_t base = (size_t)sbase[slice];
  for (int t = threadIdx.x; t < 32 * width; t += blockDim.x) {
    // element t of the slice is entry 4 (t/128) + t%4 of row (t/4)%32
    const T v = sv[(4 * (t >> 7) + (t & 3)) * 33 + ((t >> 2) & 31)];
    val[base + t] = v;
    if (valA) valA[base + t] = TA(v);
    if (valH) valH[base + t] = __float2half_rn(fminf(fmaxf((float)v * hscale, -65504.f), 65504.f));
  }
}

template <class Tin, class Tout>
__global__ void cast_copy(int n, const Tin* a, Tout* __restrict__ b) {
  pdl_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) b[i] = Tout(a[i]);
}
// b = a in the other precision, and the fine pre-smoother's diagonal step
// x1 = w0 b / den0
template <class Tin, class Tout>
__global__ void cast_jacobi(int n, const Tin* a, Tout* __restrict__ b, Tout w0,
                            const Tout* __restrict__ den0, Tout* __restrict__ x1) {
  pdl_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const Tout v = Tout(a[i]);
  b[i] = v;
  x1[i] = w0 * v / den0[i];
}

// multicolour GS colour pass on the SELL fine operator (thread per row)
template <class T, bool D16>
__global__ void sell_gs_color(int count, const int32_t* __restrict__ rows, Sell A, const T* __restrict__ v,
                              const T* __restrict__ diag, const T* __restrict__ b, T* __restrict__ x, T omega) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= count) return;
  const int i = rows[q];
  const int s = i >> 5;
  const int base = A.base[s];
  T off = 0;
  for (int k = 0; k < A.width[s]; ++k) {
    const int o = sell_offset(base, i & 31, k);
    const int j = sell_col<D16>(A, o, i);
    if (j != i) off += v[o] * x[j];
  }
  const T old = x[i];
  const T gs = (b[i] - off) / diag[i];
  x[i] = old + omega * (gs - old);
}

// The restriction to a level of many rows: a warp a row, persistent, the next
// row's entries (160 in one round; a row of the SA transfers has about 130)
// loaded before the current row's gathers and sum.  At 1.23M cells in FP32 the
// transfers of a V-cycle average 15.7 us, 17.8 with a lane group per row and
// four entries of the prolongation ahead.
constexpr int kRestAhead = 5;
template <class T>
constexpr int rest_blocks() { return sizeof(T) == 8 ? 4 : 6; }  // per SM
template <class T>
__global__ void __launch_bounds__(kBlock, rest_blocks<T>()) restrict_stream(int nc, const int32_t* __restrict__ rr,
                                                             const int32_t* __restrict__ rc, const T* __restrict__ rv,
                                                             const T* f, T* __restrict__ c,
                                                             const T* __restrict__ den0, T w0, T* __restrict__ x1) {
  pdl_trigger();
  const int lane = threadIdx.x & 31, stride = gridDim.x * kWarps;
  int I = blockIdx.x * kWarps + (threadIdx.x >> 5);
  auto bounds = [&](int i) { return i < nc ? make_int2(rr[i], rr[i + 1]) : make_int2(0, 0); };
  auto entries = [&](int (&j)[kRestAhead], T (&v)[kRestAhead], int2 o) {
#pragma unroll
    for (int u = 0; u < kRestAhead; ++u) {
      const int k = o.x + lane + 32 * u;
      j[u] = k < o.y ? rc[k] : -1;
      v[u] = k < o.y ? rv[k] : T(0);
    }
  };
  int2 cur = bounds(I), nxt = bounds(I + stride);
  int j[kRestAhead];
  T v[kRestAhead];
  entries(j, v, cur);
  pdl_wait();
  for (; I < nc; I += stride) {
    const int2 nn = bounds(I + 2 * stride);
    T x[kRestAhead];
#pragma unroll
    for (int u = 0; u < kRestAhead; ++u) x[u] = j[u] >= 0 ? f[j[u]] : T(0);
    int jn[kRestAhead];
    T vn[kRestAhead];
    entries(jn, vn, nxt);
    T di = 1;
    if (x1 && lane == 0) di = den0[I];
    T s = 0;
#pragma unroll
    for (int u = 0; u < kRestAhead; ++u) s += v[u] * x[u];
    for (int k = cur.x + lane + 32 * kRestAhead; k < cur.y; k += 32) s += rv[k] * f[rc[k]];
    s = warp_sum(s);
    if (lane == 0) {
      c[I] = s;
      // with x1: the coarse pre-smoother's diagonal step w0 c / den0
      if (x1) x1[I] = w0 * s / di;
    }
    cur = nxt;
    nxt = nn;
#pragma unroll
    for (int u = 0; u < kRestAhead; ++u) {
      j[u] = jn[u];
      v[u] = vn[u];
    }
  }
}
// c = P^T f, a kRowLanes group per coarse row over R = P^T (deterministic
// tree per row)
template <class T, int GL = kRowLanes>
__global__ void __launch_bounds__(kBlock) restrict_rows(int nc, const int32_t* __restrict__ rr,
                                                        const int32_t* __restrict__ rc, const T* __restrict__ rv,
                                                        const T* f, T* __restrict__ c,
                                                        const T* __restrict__ den0, T w0, T* __restrict__ x1) {
  pdl_trigger();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int I = t / GL, lane = t % GL;
  const T s = group_row_dot<T, T, int32_t, GL>(rr, rc, rv, f, I, lane, group_mask<GL>(), I < nc);
  if (I < nc && lane == 0) {
    c[I] = s;
    // with x1: the coarse pre-smoother's diagonal step w0 c / den0
    if (x1) x1[I] = w0 * s / den0[I];
  }
}

}  // namespace k
}  // namespace nds
