// The fine Schur operator A = B diag(rAU) B^T in split form.
//
// A pressure cell reaches its neighbours through two kinds of velocity
// unknowns (B[c][a][d], gpu/serial_cuda/g2_host.hpp:67-76):
//  * a face bubble belongs to the two cells of its face and to nothing else,
//    and the two rows of B are opposite (the face's area vector), so the
//    bubbles give a face Laplacian with tau_f = rAU_f |B[c][f]|^2:
//    sum_f tau_f (x_c - x_neighbour), or tau_f x_c on an outlet face;
//  * a vertex function's rows are V grad(lambda_a): w_v = rAU_v sum_(c,a at v)
//    B[c][a] x_c per free vertex, then sum_a B[c][a] . w_v(a) per cell.
// The product is taken in these two steps (split_vertex, split_cell) instead
// of from assembled rows.  An assembled row of the pipe meshes has 69.5
// entries (nearly all through the vertices: 24 cells around each), that is
// 278 bytes a cell in FP16 with 16-bit column deltas, 417 in FP32 and 695 in
// FP64; the two steps read 32 + 56, 64 + 76 and 112 + 128 bytes a cell, and
// the refresh writes 4 tau a cell where the assembled form rewrites every
// entry.  Smoothers that need the entries of a row (multicolour Gauss-Seidel,
// L1-Jacobi) keep the assembled SELL form.
//
// Both steps are bound by HBM on large meshes and by their two dependent
// memory round trips on small ones: every load of a step that does not
// depend on another is issued first.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"

namespace nds {
namespace k {

// |B of a face bubble|^2 / |B of the opposite vertex|^2
constexpr double kBubble2 = (27.0 / 20.0) * (27.0 / 20.0);

// Incidences of the free vertices, CSR by vertex (off), ascending cell; per
// incidence the vector B[c][a] and the cell.
//  double: component arrays bx, by, bz and the cells
//  float:  one 16-byte record (x, y, z, cell)
//  __half: one 8-byte record of three scaled halves and the cell's 16-bit
//          offset from the vertex's first cell (base); meshes whose
//          numbering does not allow that keep the halves' values in the
//          16-byte records (rec8 null)
struct SplitVerts {
  int n = 0;
  const int32_t* off = nullptr;
  const double* bx = nullptr;
  const double* by = nullptr;
  const double* bz = nullptr;
  const int32_t* cell = nullptr;
  const float4* rec16 = nullptr;
  const uint2* rec8 = nullptr;
  const int32_t* base = nullptr;
};
enum SplitRec { REC_SOA = 0, REC_16 = 1, REC_8 = 2 };

// one incidence as stored
template <int REC>
struct SplitRaw;
template <>
struct SplitRaw<REC_SOA> {
  double x, y, z;
  int c;
  __device__ __forceinline__ void load(const SplitVerts& a, int k) {
    x = a.bx[k];
    y = a.by[k];
    z = a.bz[k];
    c = a.cell[k];
  }
  __device__ __forceinline__ int cell(int) const { return c; }
  __device__ __forceinline__ void vec(double (&b)[3]) const { b[0] = x; b[1] = y; b[2] = z; }
};
template <>
struct SplitRaw<REC_16> {
  float4 q;
  __device__ __forceinline__ void load(const SplitVerts& a, int k) { q = a.rec16[k]; }
  __device__ __forceinline__ int cell(int) const { return __float_as_int(q.w); }
  __device__ __forceinline__ void vec(float (&b)[3]) const { b[0] = q.x; b[1] = q.y; b[2] = q.z; }
};
template <>
struct SplitRaw<REC_8> {
  uint2 q;
  __device__ __forceinline__ void load(const SplitVerts& a, int k) { q = a.rec8[k]; }
  __device__ __forceinline__ int cell(int base) const { return base + (int)(q.y >> 16); }
  __device__ __forceinline__ void vec(float (&b)[3]) const {
    const float2 xy = __half22float2(*reinterpret_cast<const __half2*>(&q.x));
    b[0] = xy.x;
    b[1] = xy.y;
    b[2] = __half2float(__ushort_as_half((unsigned short)(q.y & 0xFFFFu)));
  }
};

// w_v = scale rAU_v sum B x over the vertex's cells, eight lanes a vertex
// (24 incidences on average: four records per lane cover 32 in one round).  w
// holds 4 values a vertex; entry n stays zero (fixed vertices).
//
// Three dependent loads a vertex (offsets, records, x) and little else: bound
// by their latency when each group does one vertex (21 us at 1.23M cells in
// FP16, 46 MB).  So the groups are persistent and pipelined: the offsets are
// loaded two vertices ahead and the records one ahead, and a vertex waits
// only for its gathers: 13.3 us so.  FP64 records keep one vertex's in
// registers: with the next one's only two blocks fit an SM and the next kernel
// cannot start early (40k cells: 62 us an iteration of the pressure loop
// instead of 56).  The first records, constant during a solve, are loaded
// before the wait for the kernel that writes x.
constexpr int kSplitAhead = 4;
template <int REC>
constexpr int split_vertex_blocks() { return REC == REC_SOA ? 3 : REC == REC_16 ? 4 : 5; }  // per SM
template <class V, int REC>
__global__ void __launch_bounds__(kBlock, split_vertex_blocks<REC>())
    split_vertex(SplitVerts a, const V* __restrict__ rau, const V* x, V* __restrict__ w, V scale) {
  pdl_trigger();
  constexpr bool PIPE = REC != REC_SOA;  // the next vertex's records in registers
  const int t = blockIdx.x * blockDim.x + threadIdx.x, stride = (gridDim.x * blockDim.x) >> 3;
  const int lane = t & 7;
  const unsigned mask = group8_mask();
  int g = t >> 3;
  struct Off {
    int b, e, base;
  };
  auto offsets = [&](int v) {
    Off o{0, 0, 0};
    if (v < a.n) {
      o.b = a.off[v];
      o.e = a.off[v + 1];
      if (REC == REC_8) o.base = a.base[v];
    }
    return o;
  };
  auto records = [&](SplitRaw<REC> (&raw)[kSplitAhead], const Off& o) {
#pragma unroll
    for (int u = 0; u < kSplitAhead; ++u) {
      const int z = o.b + lane + 8 * u;
      if (z < o.e) raw[u].load(a, z);
    }
  };
  Off cur = offsets(g), nxt = offsets(g + stride);
  SplitRaw<REC> raw[kSplitAhead] = {};
  records(raw, cur);
  pdl_wait();
  while (g < a.n) {
    const Off nn = offsets(g + 2 * stride);
    SplitRaw<REC> rawn[kSplitAhead] = {};
    V xv[kSplitAhead];
#pragma unroll
    for (int u = 0; u < kSplitAhead; ++u)
      xv[u] = cur.b + lane + 8 * u < cur.e ? x[raw[u].cell(cur.base)] : V(0);
    if (PIPE) records(rawn, nxt);
    V r = 0;
    if (lane == 0) r = scale * rau[g];
    V s0 = 0, s1 = 0, s2 = 0;
#pragma unroll
    for (int u = 0; u < kSplitAhead; ++u) {
      V b[3];
      raw[u].vec(b);
      s0 += b[0] * xv[u];
      s1 += b[1] * xv[u];
      s2 += b[2] * xv[u];
    }
    for (int z = cur.b + lane + 8 * kSplitAhead; z < cur.e; z += 8) {
      SplitRaw<REC> q;
      q.load(a, z);
      V b[3];
      q.vec(b);
      const V xz = x[q.cell(cur.base)];
      s0 += b[0] * xz;
      s1 += b[1] * xz;
      s2 += b[2] * xz;
    }
    s0 = group_sum<8>(s0, mask);
    s1 = group_sum<8>(s1, mask);
    s2 = group_sum<8>(s2, mask);
    if (lane == 0) {
      if constexpr (std::is_same<V, float>::value) {
        reinterpret_cast<float4*>(w)[g] = make_float4(r * s0, r * s1, r * s2, 0.f);
      } else {
        reinterpret_cast<double2*>(w)[2 * (size_t)g] = make_double2(r * s0, r * s1);
        w[4 * (size_t)g + 2] = r * s2;
      }
    }
    g += stride;
    cur = nxt;
    nxt = nn;
    if (PIPE) {
#pragma unroll
      for (int u = 0; u < kSplitAhead; ++u) raw[u] = rawn[u];
    } else if (g < a.n) {
      records(raw, cur);
    }
  }
}

// Cell data of the second step, structure of arrays of vector loads:
//  vid: the four vertices (n_vertices for a fixed one); nid / nd16: the four
//  face neighbours, absolute (-1: none) or as 16-bit deltas to the cell (0:
//  none) when they all fit; tau: the four face couplings (0 on a fixed face).
//  geo: B of the vertices 1, 2, 3 (the four sum to zero): float 4 + 4 + 1,
//  double 2 + 2 + 2 + 2 + 1; __half: all four, scaled, in 8 + 4 values, each
//  rounded as in the vertex records, so that the FP16 operator is symmetric
//  (zero for a fixed vertex).
//  A free face without a neighbour (outlet) couples as tau x_c.
struct SplitCells {
  int n = 0;
  const int4* vid = nullptr;
  const int4* nid = nullptr;
  const short4* nd16 = nullptr;
  const void* g0 = nullptr;
  const void* g1 = nullptr;
  const void* g2 = nullptr;
  const void* tau = nullptr;
};

// a vector read as it is
template <class V>
struct PlainVector {
  const V* x;
  __device__ __forceinline__ V operator()(int c) const { return x[c]; }
};

// the vertex sums of split_vertex
template <class V>
struct PlainVertices {
  const V* w;
  __device__ __forceinline__ void operator()(int v, V (&o)[3]) const {
    if constexpr (std::is_same<V, float>::value) {
      const float4 u = reinterpret_cast<const float4*>(w)[v];
      o[0] = u.x; o[1] = u.y; o[2] = u.z;
    } else {
      const double2 u = reinterpret_cast<const double2*>(w)[2 * (size_t)v];
      o[0] = u.x; o[1] = u.y;
      o[2] = w[4 * (size_t)v + 2];
    }
  }
};

// A cell's data (constant during a solve) and its row's product
template <class V, class MT>
struct SplitGeo;
template <class V>
struct SplitGeo<V, __half> {
  uint4 p;
  uint2 q, th;
  __device__ __forceinline__ void load(const SplitCells& a, int c) {
    p = static_cast<const uint4*>(a.g0)[c];
    q = static_cast<const uint2*>(a.g1)[c];
    th = static_cast<const uint2*>(a.tau)[c];
  }
  static __device__ __forceinline__ float2 h2(unsigned u) { return __half22float2(*reinterpret_cast<const __half2*>(&u)); }
  __device__ __forceinline__ void tau(V (&t)[4]) const {
    const float2 t01 = h2(th.x), t23 = h2(th.y);
    t[0] = t01.x; t[1] = t01.y; t[2] = t23.x; t[3] = t23.y;
  }
  __device__ __forceinline__ V vertices(const V (&wv)[4][3]) const {
    const float2 b01 = h2(p.x), b23 = h2(p.y), b45 = h2(p.z), b67 = h2(p.w), b89 = h2(q.x), bab = h2(q.y);
    V s = b01.x * wv[0][0] + b01.y * wv[0][1] + b23.x * wv[0][2];
    s += b23.y * wv[1][0] + b45.x * wv[1][1] + b45.y * wv[1][2];
    s += b67.x * wv[2][0] + b67.y * wv[2][1] + b89.x * wv[2][2];
    s += b89.y * wv[3][0] + bab.x * wv[3][1] + bab.y * wv[3][2];
    return s;
  }
};
// the vertices enter by the gradients of 1, 2, 3: sum_j S_j . (w_j - w_0)
template <class V>
__device__ __forceinline__ V split_gradients(const V (&b)[9], const V (&wv)[4][3]) {
  V s = 0;
#pragma unroll
  for (int j = 0; j < 3; ++j)
#pragma unroll
    for (int d = 0; d < 3; ++d) s += b[3 * j + d] * (wv[j + 1][d] - wv[0][d]);
  return s;
}
template <>
struct SplitGeo<float, float> {
  float4 p, q, tt;
  float l;
  __device__ __forceinline__ void load(const SplitCells& a, int c) {
    p = static_cast<const float4*>(a.g0)[c];
    q = static_cast<const float4*>(a.g1)[c];
    l = static_cast<const float*>(a.g2)[c];
    tt = static_cast<const float4*>(a.tau)[c];
  }
  __device__ __forceinline__ void tau(float (&t)[4]) const {
    t[0] = tt.x; t[1] = tt.y; t[2] = tt.z; t[3] = tt.w;
  }
  __device__ __forceinline__ float vertices(const float (&wv)[4][3]) const {
    const float b[9] = {p.x, p.y, p.z, p.w, q.x, q.y, q.z, q.w, l};
    return split_gradients(b, wv);
  }
};
template <>
struct SplitGeo<double, double> {
  double2 g[4], ta, tb;
  double l;
  __device__ __forceinline__ void load(const SplitCells& a, int c) {
    const double2* gp = static_cast<const double2*>(a.g0);
    const ptrdiff_t n = a.n;
#pragma unroll
    for (int k = 0; k < 4; ++k) g[k] = gp[k * n + c];
    l = static_cast<const double*>(a.g2)[c];
    const double2* tp = static_cast<const double2*>(a.tau) + 2 * (ptrdiff_t)c;
    ta = tp[0];
    tb = tp[1];
  }
  __device__ __forceinline__ void tau(double (&t)[4]) const {
    t[0] = ta.x; t[1] = ta.y; t[2] = tb.x; t[3] = tb.y;
  }
  __device__ __forceinline__ double vertices(const double (&wv)[4][3]) const {
    const double b[9] = {g[0].x, g[0].y, g[1].x, g[1].y, g[2].x, g[2].y, g[3].x, g[3].y, l};
    return split_gradients(b, wv);
  }
};
template <class V, class MT, bool D16>
struct SplitRow {
  int4 vi;
  int nb[4];
  SplitGeo<V, MT> geo;
  __device__ __forceinline__ void load(const SplitCells& a, int c) {
    vi = a.vid[c];
    if (D16) {
      const short4 d = a.nd16[c];
      nb[0] = d.x ? c + d.x : -1;
      nb[1] = d.y ? c + d.y : -1;
      nb[2] = d.z ? c + d.z : -1;
      nb[3] = d.w ? c + d.w : -1;
    } else {
      const int4 d = a.nid[c];
      nb[0] = d.x; nb[1] = d.y; nb[2] = d.z; nb[3] = d.w;
    }
    geo.load(a, c);
  }
  // vertices from w, faces from x (xc = x(c))
  template <class X, class W>
  __device__ __forceinline__ V product(const X& x, const W& w, V xc, V tinv) const {
    V wv[4][3], xn[4], t[4];
    w(vi.x, wv[0]);
    w(vi.y, wv[1]);
    w(vi.z, wv[2]);
    w(vi.w, wv[3]);
#pragma unroll
    for (int f = 0; f < 4; ++f) xn[f] = nb[f] >= 0 ? x(nb[f]) : V(0);
    const V s = geo.vertices(wv);
    geo.tau(t);
    V f = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) f += t[k] * (xc - xn[k]);
    if constexpr (std::is_same<MT, __half>::value) return s + tinv * f;
    else return s + f;
  }
};
template <class V, class MT, bool D16, class X, class W>
__device__ __forceinline__ V split_row(const SplitCells& a, const X& x, const W& w, int c, V xc, V tinv) {
  SplitRow<V, MT, D16> r;
  r.load(a, c);
  return r.product(x, w, xc, tinv);
}

// The modes Y, RESID and SMOOTH of sell_spmv on the split form (w from
// split_vertex on the same x).  STEP SUM_ONLY (RESID): also ||r||^2.  Y with y2: also x into vector at[0] of y2.
// STEP PCG_RHO (SMOOTH with y2, the last step
// of the V-cycle): also r.z of the new z = y2 with the reduction tail.
template <class V, int MODE, bool D16, class MT, int STEP = 0, class R = V>
__global__ void __launch_bounds__(kBlock) split_cell(SplitCells a, const V* w, const V* x,
                                                     const V* b, const V* __restrict__ den, V wt,
                                                     V* __restrict__ y, V* y2, V tinv,
                                                     const R* rr, ReduceTail tail,
                                                     const int* at) {
  pdl_trigger();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  double acc = 0.0;
  SplitRow<V, MT, D16> row;
  V dc = 1;
  if (c < a.n) {
    row.load(a, c);
    if (MODE == SELL_SMOOTH || (MODE == SELL_RESID && den)) dc = den[c];
  }
  pdl_wait();
  if (c < a.n) {
    const V xc = x[c];
    const V bc = MODE != SELL_Y ? b[c] : V(0);
    const V s = row.product(PlainVector<V>{x}, PlainVertices<V>{w}, xc, tinv);
    if (MODE == SELL_Y) {
      y[c] = s;
      if (y2) y2[(size_t)at[0] * a.n + c] = xc;
    } else if (MODE == SELL_RESID) {
      const V q = bc - s;
      y[c] = q;
      if (den) y2[c] = wt * q / dc;
      else if (y2) y2[c] = q;
      if (STEP != 0) acc = (double)q * (double)q;
    } else {
      V val = xc + wt * (bc - s) / dc;
      if (y2) {
        val += y2[c];
        y2[c] = val;
      } else {
        y[c] = val;
      }
      if (STEP != 0) acc = (double)rr[c] * (double)val;
    }
  }
  if (STEP != 0) reduce_tail<STEP>(acc, tail);
}
// q = A p with p.q and the step alpha of PCG (grid-stride; the data type of
// the operator is that of the vectors)
template <class V, bool D16>
__global__ void __launch_bounds__(kBlock) split_cell_dot(SplitCells a, const V* w,
                                                         const V* p, V* __restrict__ q, V tinv,
                                                         ReduceTail tail) {
  pdl_trigger();
  double acc = 0.0;
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  SplitRow<V, V, D16> row;
  if (c < a.n) row.load(a, c);
  pdl_wait();
  while (c < a.n) {
    const V pc = p[c];
    const V s = row.product(PlainVector<V>{p}, PlainVertices<V>{w}, pc, tinv);
    q[c] = s;
    acc += (double)pc * (double)s;
    c += gridDim.x * blockDim.x;
    if (c < a.n) row.load(a, c);
  }
  reduce_tail<PCG_ALPHA>(acc, tail);
}

// Refresh of the split form from rAU: thread c writes cell c's face couplings
// in the precisions in use (g4: |B|^2 of the four vertices, static) and the
// diagonal A_cc = sum_i |B_i|^2 (rAU_vertex + kBubble2 rAU_face); threads
// below nvert also copy the vertices' rAU.  rv and tau in the operator's
// precision T; rvA and tauA (FP32, the mixed modes) and tauH (FP16, scaled
// and saturated) may be null.
template <class T, class TA>
__global__ void __launch_bounds__(kBlock) split_refresh(int nc, int nvert, const int32_t* __restrict__ ref,
                                                        const T* __restrict__ g4, const T* __restrict__ rau,
                                                        T* __restrict__ rv, TA* __restrict__ rvA,
                                                        T* __restrict__ tau, TA* __restrict__ tauA,
                                                        __half* __restrict__ tauH, float hscale,
                                                        TA* __restrict__ diag) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < nvert) {
    const T r = rau[c];
    rv[c] = r;
    if (rvA) rvA[c] = TA(r);
  }
  if (c >= nc) return;
  const int4* r4 = reinterpret_cast<const int4*>(ref + 8 * (size_t)c);
  const int4 v = r4[0], f = r4[1];
  const int vi[4] = {v.x, v.y, v.z, v.w}, fi[4] = {f.x, f.y, f.z, f.w};
  T g[4], rvv[4], rf[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    g[i] = g4[(size_t)i * nc + c];
    rvv[i] = vi[i] >= 0 ? rau[vi[i]] : T(0);
    rf[i] = fi[i] >= 0 ? rau[fi[i]] : T(0);
  }
  T d = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const T t = T(kBubble2) * g[i] * rf[i];
    d += rvv[i] * g[i] + t;
    tau[4 * (size_t)c + i] = t;
    if (tauA) tauA[4 * (size_t)c + i] = TA(t);
    if (tauH) tauH[4 * (size_t)c + i] = __float2half_rn(fminf((float)t * hscale, 65504.f));
  }
  diag[c] = TA(d);
}

// a_ij of the face neighbours of each cell, off[4 i + k] = face k's position
// in the cell (its opposite vertex): the face coupling plus the shared
// vertices' part, from the operator's own data in its precision
template <class T>
__global__ void split_edges(int n, const int32_t* __restrict__ nbr, const uint8_t* __restrict__ face,
                            const int32_t* __restrict__ ref, const T* __restrict__ bco, const T* __restrict__ rv,
                            const T* __restrict__ tau, const float* __restrict__ dscale, float* __restrict__ ew) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 4 * n) return;
  const int i = t >> 2, j = nbr[t];
  if (j < 0) {
    ew[t] = 0.f;
    return;
  }
  T s = -tau[4 * (size_t)i + face[t]];
  for (int a = 0; a < 4; ++a) {
    const int g = ref[8 * (size_t)i + a];
    if (g < 0) continue;
    for (int b = 0; b < 4; ++b)
      if (ref[8 * (size_t)j + b] == g) {
        const T* p = bco + 24 * (size_t)i + 3 * a;
        const T* q = bco + 24 * (size_t)j + 3 * b;
        s += rv[g] * (p[0] * q[0] + p[1] * q[1] + p[2] * q[2]);
      }
  }
  ew[t] = (float)s * dscale[i] * dscale[j];
}

}  // namespace k
}  // namespace nds
