// PCG with its V-cycle as one kernel of one cluster, for small meshes.
//
// A PCG iteration of the split operator with a dense coarse level is fourteen
// dependent steps.  On a few thousand cells each has well under a microsecond
// of work, and as kernels (or as phases of a grid that meets at barriers in
// global memory) a step costs two to three microseconds of launch, cold loads
// and round trips to L2.  Here one cluster of eight blocks keeps every vector
// of the solve in its shared memory: block k owns the cells, free vertices
// and coarse rows of the k-th eighth, neighbours are read through distributed
// shared memory, and the steps are separated by the cluster's hardware
// barrier.  The barrier's acquire empties L1, so constant data read from
// global memory costs an L2 round trip in every step: the operators' data is
// copied to shared memory too, as far as it fits (the V-cycle's first: four
// of five products).  Bound by the chain of latencies in a step (shared
// memory, FP64 arithmetic and shuffles, barrier), about 1.5 us each.  512
// threads of 128 registers: the FP64 forms spill 72 to 76 bytes there.
// Microseconds of an iteration, loop of kernels / this: 720 cells FP64 35.5 /
// 20, FP32 37 / 20; 2,400 cells FP64 38 / 24, mixed FP16 45 / 30; 4,608 cells
// FP32 35 / 35.  One block instead of eight was tried: 34 at 720 cells, 93 at
// 2,400 (FP64); one block per SM meeting at barriers in global memory: 44 at
// 720 cells, 57 to 65 at 48,000, no better than the kernels.
//
// Every block forms the scalars from the same eight partial sums in the same
// order, so all take the same decisions and a run is reproducible.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"
#include "split.cuh"

namespace nds {
namespace k {

constexpr int kResBlock = 512;
constexpr int kResWarps = kResBlock / 32;
constexpr int kResCluster = 8;
constexpr int kResSteps = 16;  // smoother degrees up to 16
constexpr int kResParts = 4;   // warps that share a row of the dense level

template <class S, class TA>
struct Resident {
  int nc, chunk;             // cells, cells per block
  unsigned inv_chunk;        // cell / chunk = umulhi(cell, inv_chunk)
  int vchunk;                // vertices per block
  unsigned inv_vchunk;
  // operator of the Krylov method (precision S) and of the V-cycle (TA)
  SplitVerts vs, va;
  SplitCells cs, ca;
  const S* rvs;
  const TA* rva;
  TA wscale, tinv;
  const TA* den;
  int m;                     // smoothing steps after the diagonal one
  TA w[kResSteps];           // weights: diagonal step, then the steps
  // coarse level: R in CSR, its V-cycle matrix (row stride ld), P in ELL
  int nk, kchunk, ld, pw;
  const int32_t* rr;
  const int32_t* rc;
  const TA* rv;
  const TA* dense;
  const int32_t* pc;
  const TA* pv;
  // largest number of vertex incidences of a block, and whether the V-cycle's
  // and the Krylov method's operator are copied to shared memory (with the
  // same data, both are when the first is)
  int zmax, copy_a, copy_s;
  const S* r;                // in: the residual
  S* x;                      // out: the solution (from zero)
  double* sc;                // [3] ||r||^2 out
  int r0_slot, target_slot;
  int* flags;
  int* ctl;                  // [0] iterations, [1] converged out; [3] cap in
  HostWords host;
};
// floor(2^32 / chunk) + 1: umulhi(i, .) = i / chunk for i chunk < 2^32
inline unsigned res_inverse(int chunk) { return (unsigned)(0x100000000ull / (unsigned)chunk + 1); }
// bytes of dynamic shared memory per block
template <class S, class TA>
inline size_t res_smem(int chunk, int vchunk, int ld) {
  const bool same = std::is_same<S, TA>::value;
  return (size_t)chunk * (5 * sizeof(S) + (same ? 5 : 6) * sizeof(TA)) + 4 * (size_t)vchunk * sizeof(S) +
         2 * (size_t)ld * sizeof(TA) + 16 * 16;
}
// bytes of an operator's copy (V: arithmetic type; MT: its data)
template <class V, class MT>
inline size_t res_copy_bytes(int chunk, int vchunk, int zmax, bool d16, bool rec8) {
  const bool half = std::is_same<MT, __half>::value;
  const size_t cell = 16 + (d16 ? 8 : 16) + (half ? 32 : 13 * sizeof(V)) + sizeof(V);  // with den
  const size_t inc = std::is_same<V, double>::value ? 28 : rec8 ? 8 : 16;
  return (size_t)chunk * cell + (size_t)zmax * inc + (size_t)(vchunk + 1) * (4 + 4 + sizeof(V)) + 16 * 16;
}

__device__ __forceinline__ uint32_t dsm_addr(const void* p, unsigned cta) {
  uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(p)), o;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(o) : "r"(a), "r"(cta));
  return o;
}
__device__ __forceinline__ void dsm_load(uint32_t a, float& v) {
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
}
__device__ __forceinline__ void dsm_load(uint32_t a, double& v) {
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
}
__device__ __forceinline__ void dsm_load3(uint32_t a, float (&v)[3]) {
  float pad;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(pad)
               : "r"(a)
               : "memory");
}
__device__ __forceinline__ void dsm_load3(uint32_t a, double (&v)[3]) {
  asm volatile("ld.shared::cluster.v2.f64 {%0,%1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "r"(a) : "memory");
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v[2]) : "r"(a + 16) : "memory");
}
__device__ __forceinline__ void dsm_store(uint32_t a, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void dsm_store(uint32_t a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

// a distributed vector (its part in every block at the same place)
template <class V>
struct DsmVector {
  const V* x;
  int chunk;
  unsigned inv;
  __device__ __forceinline__ V operator()(int c) const {
    const unsigned k = __umulhi((unsigned)c, inv);
    V v;
    dsm_load(dsm_addr(x + (c - (int)k * chunk), k), v);
    return v;
  }
};
// the search direction p = z + beta p_old (p = z at the first iteration),
// formed where it is read
template <class S, class TA>
struct DsmDirection {
  DsmVector<TA> z;
  DsmVector<S> old;
  S beta;
  bool first;
  __device__ __forceinline__ S operator()(int c) const {
    const S zc = S(z(c));
    return first ? zc : zc + beta * old(c);
  }
};
// the vertex sums (four values a vertex)
template <class V>
struct DsmVertices {
  const V* w;
  int n, chunk;
  unsigned inv;
  __device__ __forceinline__ void operator()(int v, V (&o)[3]) const {
    if (v >= n) {  // fixed
      o[0] = o[1] = o[2] = V(0);
      return;
    }
    const unsigned k = __umulhi((unsigned)v, inv);
    dsm_load3(dsm_addr(w + 4 * (v - (int)k * chunk), k), o);
  }
};

// products of one vertex's incidences with x, by a group of eight lanes; the
// sums are valid in every lane
template <class V, class X>
__device__ __forceinline__ void resident_vertex(const SplitVerts& a, int g, int lane, unsigned mask, const X& x,
                                                V (&s)[3]) {
  const int zb = a.off[g], ze = a.off[g + 1];
  V s0 = 0, s1 = 0, s2 = 0;
  for (int z0 = zb + lane; z0 < ze; z0 += 8 * kSplitAhead) {
    V b0[kSplitAhead], b1[kSplitAhead], b2[kSplitAhead], xv[kSplitAhead];
    int c[kSplitAhead];
#pragma unroll
    for (int u = 0; u < kSplitAhead; ++u) {
      const int z = z0 + 8 * u;
      c[u] = -1;
      b0[u] = b1[u] = b2[u] = V(0);
      if (z < ze) {
        if constexpr (std::is_same<V, double>::value) {
          b0[u] = a.bx[z];
          b1[u] = a.by[z];
          b2[u] = a.bz[z];
          c[u] = a.cell[z];
        } else if (a.rec8) {
          const uint2 q = a.rec8[z];
          const float2 xy = __half22float2(*reinterpret_cast<const __half2*>(&q.x));
          b0[u] = xy.x;
          b1[u] = xy.y;
          b2[u] = __half2float(__ushort_as_half((unsigned short)(q.y & 0xFFFFu)));
          c[u] = a.base[g] + (int)(q.y >> 16);
        } else {
          const float4 q = a.rec16[z];
          b0[u] = q.x;
          b1[u] = q.y;
          b2[u] = q.z;
          c[u] = __float_as_int(q.w);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < kSplitAhead; ++u) xv[u] = c[u] >= 0 ? x(c[u]) : V(0);
#pragma unroll
    for (int u = 0; u < kSplitAhead; ++u) {
      s0 += b0[u] * xv[u];
      s1 += b1[u] * xv[u];
      s2 += b2[u] * xv[u];
    }
  }
  s[0] = group_sum<8>(s0, mask);
  s[1] = group_sum<8>(s1, mask);
  s[2] = group_sum<8>(s2, mask);
}

template <class S, class TA, class MT>
__global__ void __launch_bounds__(kResBlock, 1) __cluster_dims__(kResCluster, 1, 1)
    pcg_resident(const Resident<S, TA> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ TA srow[kResWarps];
  __shared__ double sred[kResWarps];
  __shared__ double spart[3][kResCluster];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned me = blockIdx.x;  // one cluster: the block's rank
  const int n = a.chunk, lo = (int)me * n, cnt = max(0, min(n, a.nc - lo));
  const int vlo = (int)me * a.vchunk, vcnt = max(0, min(a.vchunk, a.vs.n - vlo));
  const int klo = (int)me * a.kchunk, kcnt = max(0, min(a.kchunk, a.nk - klo));
  // shared arrays, 16-byte aligned, at the same place in every block
  unsigned char* top = smem_raw;
  auto take = [&](auto tag, size_t len) {
    using V = decltype(tag);
    V* p = reinterpret_cast<V*>(top);
    top += (len * sizeof(V) + 15) / 16 * 16;
    return p;
  };
  S* const w = take(S{}, 4 * (size_t)a.vchunk);
  TA* const wa = reinterpret_cast<TA*>(w);
  TA* const cb = take(TA{}, (size_t)a.ld);
  TA* const cx = take(TA{}, (size_t)a.ld);
  S* const x = take(S{}, (size_t)n);
  S* const r = take(S{}, (size_t)n);
  S* const q = take(S{}, (size_t)n);
  S* const p0 = take(S{}, (size_t)n);
  S* const p1 = take(S{}, (size_t)n);
  TA* const z = take(TA{}, (size_t)n);
  TA* const v0 = take(TA{}, (size_t)n);
  TA* const v1 = take(TA{}, (size_t)n);
  TA* const res = take(TA{}, (size_t)n);
  TA* const ex = take(TA{}, (size_t)n);
  TA* rA;
  if constexpr (std::is_same<S, TA>::value) rA = r;
  else rA = take(TA{}, (size_t)n);

  // the operators, from shared memory where copied (their pointers shifted so
  // that global indices address the block's part)
  SplitCells ca = a.ca, cs = a.cs;
  SplitVerts va = a.va, vs = a.vs;
  const TA* rva = a.rva;
  const S* rvs = a.rvs;
  const TA* den = a.den + lo;
  auto fetch = [&](auto*& src, ptrdiff_t from, ptrdiff_t len, size_t room) {
    using V = std::remove_const_t<std::remove_pointer_t<std::remove_reference_t<decltype(src)>>>;
    V* d = take(V{}, room);
    for (ptrdiff_t k = tid; k < len; k += kResBlock) d[k] = src[from + k];
    src = d - from;
  };
  auto copy_op = [&](auto tag, auto mt, SplitCells& cc, SplitVerts& vv, auto*& rau) {
    using V = decltype(tag);
    using M = decltype(mt);
    const int zlo = vcnt > 0 ? vv.off[vlo] : 0, zn = vcnt > 0 ? vv.off[vlo + vcnt] - zlo : 0;
    fetch(cc.vid, lo, cnt, n);
    if (cc.nd16) fetch(cc.nd16, lo, cnt, n);
    else fetch(cc.nid, lo, cnt, n);
    auto part = [&](const void*& p, auto t, ptrdiff_t per) {
      using U = decltype(t);
      const U* q = static_cast<const U*>(p);
      fetch(q, per * lo, per * cnt, (size_t)per * n);
      p = q;
    };
    if constexpr (std::is_same<M, __half>::value) {
      part(cc.g0, uint4{}, 1);
      part(cc.g1, uint2{}, 1);
      part(cc.tau, uint2{}, 1);
    } else if constexpr (std::is_same<V, float>::value) {
      part(cc.g0, float4{}, 1);
      part(cc.g1, float4{}, 1);
      part(cc.g2, float{}, 1);
      part(cc.tau, float4{}, 1);
    } else {
      double2* d = take(double2{}, 4 * (size_t)n);
      const double2* g = static_cast<const double2*>(cc.g0);
      for (int k = tid; k < 4 * cnt; k += kResBlock) {
        const int q4 = k / cnt, l = k - q4 * cnt;
        d[q4 * n + l] = g[(size_t)q4 * cc.n + lo + l];
      }
      cc.g0 = d - lo;
      cc.n = n;  // stride of the four parts
      part(cc.g2, double{}, 1);
      part(cc.tau, double2{}, 2);
    }
    if constexpr (std::is_same<V, double>::value) {
      fetch(vv.bx, zlo, zn, a.zmax);
      fetch(vv.by, zlo, zn, a.zmax);
      fetch(vv.bz, zlo, zn, a.zmax);
      fetch(vv.cell, zlo, zn, a.zmax);
    } else if (vv.rec8) {
      fetch(vv.rec8, zlo, zn, a.zmax);
      fetch(vv.base, vlo, vcnt, a.vchunk);
    } else {
      fetch(vv.rec16, zlo, zn, a.zmax);
    }
    fetch(vv.off, vlo, vcnt > 0 ? vcnt + 1 : 0, a.vchunk + 1);
    fetch(rau, vlo, vcnt, a.vchunk);
  };
  if (a.copy_a) {
    copy_op(TA{}, MT{}, ca, va, rva);
    const TA* d = a.den;
    fetch(d, lo, cnt, n);
    den = d + lo;
    if constexpr (std::is_same<S, TA>::value && std::is_same<MT, TA>::value) {
      cs = ca;
      vs = va;
      rvs = rva;
    }
  }
  if constexpr (!(std::is_same<S, TA>::value && std::is_same<MT, TA>::value)) {
    if (a.copy_s) copy_op(S{}, S{}, cs, vs, rvs);
  }
  __syncthreads();

  auto vec = [&](const auto* y) {
    using V = std::remove_const_t<std::remove_pointer_t<decltype(y)>>;
    return DsmVector<V>{y, n, a.inv_chunk};
  };
  const unsigned mask8 = group8_mask();
  auto vertices = [&](auto* ww, const SplitVerts& v, const auto* rau, const auto& xx, auto scale) {
    using V = std::remove_pointer_t<decltype(ww)>;
    for (int l = tid >> 3; l < vcnt; l += kResBlock / 8) {
      V s[3];
      const V rr = scale * rau[vlo + l];
      resident_vertex<V>(v, vlo + l, tid & 7, mask8, xx, s);
      if ((tid & 7) == 0) {
        ww[4 * l] = rr * s[0];
        ww[4 * l + 1] = rr * s[1];
        ww[4 * l + 2] = rr * s[2];
      }
    }
  };
  auto vert_a = [&](const TA* y) { vertices(wa, va, rva, vec(y), a.wscale); };
  const DsmVertices<TA> wva{wa, a.va.n, a.vchunk, a.inv_vchunk};
  const DsmVertices<S> wvs{w, a.vs.n, a.vchunk, a.inv_vchunk};
  auto row_a = [&](const TA* y, int l, TA yc) {
    return ca.nd16 ? split_row<TA, MT, true>(ca, vec(y), wva, lo + l, yc, a.tinv)
                     : split_row<TA, MT, false>(ca, vec(y), wva, lo + l, yc, a.tinv);
  };
  // sum over all threads of the cluster, the same value everywhere; a barrier
  auto reduce = [&](double v, int slot) {
    v = warp_sum(v);
    if (lane == 0) sred[warp] = v;
    __syncthreads();
    if (warp == 0) {
      double s = lane < kResWarps ? sred[lane] : 0.0;
      s = warp_sum(s);
      if (lane < kResCluster) dsm_store(dsm_addr(&spart[slot][me], (unsigned)lane), s);
    }
    cluster_sync();
    double s = 0;
#pragma unroll
    for (int k = 0; k < kResCluster; ++k) s += spart[slot][k];
    return s;
  };
  // r in the V-cycle's precision and the first smoothing step
  auto first_step = [&](int l, S rr) {
    const TA ra = TA(rr);
    if constexpr (!std::is_same<S, TA>::value) rA[l] = ra;
    v0[l] = a.w[0] * ra / den[l];
  };

  for (int l = tid; l < cnt; l += kResBlock) {
    const S rr = a.r[lo + l];
    r[l] = rr;
    x[l] = S(0);
    first_step(l, rr);
  }
  for (int k = tid; k < a.ld; k += kResBlock) cb[k] = cx[k] = TA(0);
  const double target = a.sc[a.target_slot], r0 = a.sc[a.r0_slot];
  const int cap = a.ctl[3];
  double rho = 0, rn2 = 0;
  int its = 0, flags = 0, conv = 0;
  bool first = true;
  cluster_sync();

  for (;;) {
    // ---- z = M r
    TA* cur = v0;
    TA* nxt = v1;
    for (int st = 1; st <= a.m; ++st) {
      vert_a(cur);
      cluster_sync();
      for (int l = tid; l < cnt; l += kResBlock) {
        const TA xc = cur[l];
        nxt[l] = xc + a.w[st] * (rA[l] - row_a(cur, l, xc)) / den[l];
      }
      cluster_sync();
      TA* t = cur;
      cur = nxt;
      nxt = t;
    }
    vert_a(cur);
    cluster_sync();
    for (int l = tid; l < cnt; l += kResBlock) res[l] = rA[l] - row_a(cur, l, cur[l]);
    cluster_sync();
    // restriction, 16 lanes a coarse row; the result goes to every block
    {
      const int l16 = tid & 15;
      const unsigned m16 = group_mask<16>();
      const auto f = vec(res);
      for (int l = tid >> 4; l < kcnt; l += kResBlock / 16) {
        const int i = klo + l, re = a.rr[i + 1];
        TA s = 0;
        for (int k0 = a.rr[i] + l16; k0 < re; k0 += 128) {
          int j[8];
          TA v[8], fv[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const int k = k0 + 16 * u;
            j[u] = k < re ? a.rc[k] : -1;
            v[u] = k < re ? a.rv[k] : TA(0);
          }
#pragma unroll
          for (int u = 0; u < 8; ++u) fv[u] = j[u] >= 0 ? f(j[u]) : TA(0);
#pragma unroll
          for (int u = 0; u < 8; ++u) s += v[u] * fv[u];
        }
        s = group_sum<16>(s, m16);
        if (l16 < kResCluster) dsm_store(dsm_addr(cb + i, (unsigned)l16), s);
      }
    }
    cluster_sync();
    // dense coarse level, four warps a row
    {
      constexpr int W = 16 / sizeof(TA);
      using V4 = typename std::conditional<std::is_same<TA, float>::value, float4, double2>::type;
      const V4* s4 = reinterpret_cast<const V4*>(cb);
      const int nv = a.ld / W, per = (nv + kResParts - 1) / kResParts;
      const int pt = warp % kResParts, row0 = warp / kResParts;
      constexpr int rows = kResWarps / kResParts;  // at a time
      for (int base = 0; base < kcnt; base += rows) {
        const int l = base + row0;
        if (l < kcnt) {
          const V4* A4 = reinterpret_cast<const V4*>(a.dense + (size_t)(klo + l) * a.ld);
          const int e = min(nv, (pt + 1) * per);
          TA s = 0;
#pragma unroll 4
          for (int k = pt * per + lane; k < e; k += 32) {
            const V4 p = A4[k], y = s4[k];
            if constexpr (W == 4) s += p.x * y.x + p.y * y.y + p.z * y.z + p.w * y.w;
            else s += p.x * y.x + p.y * y.y;
          }
          s = warp_sum(s);
          if (lane == 0) srow[warp] = s;
        }
        __syncthreads();
        if (l < kcnt && pt == 0 && lane < kResCluster) {
          TA s = srow[warp];
#pragma unroll
          for (int k = 1; k < kResParts; ++k) s += srow[warp + k];
          dsm_store(dsm_addr(cx + klo + l, (unsigned)lane), s);
        }
        __syncthreads();
      }
    }
    cluster_sync();
    // cur += P x_c
    for (int l = tid; l < cnt; l += kResBlock) {
      TA s = 0;
      for (int k = 0; k < a.pw; ++k) {
        const size_t o = (size_t)k * a.nc + lo + l;
        s += a.pv[o] * cx[a.pc[o]];
      }
      cur[l] += s;
    }
    cluster_sync();
    // post-smoothing (res now its right-hand side); the last step forms z and r.z
    vert_a(cur);
    cluster_sync();
    double acc = 0;
    TA* g = nxt;
    TA* gn = ex;
    for (int l = tid; l < cnt; l += kResBlock) {
      const TA xc = cur[l];
      const TA e = rA[l] - row_a(cur, l, xc);
      if (a.m == 0) {
        const TA zc = xc + a.w[0] * e / den[l];
        z[l] = zc;
        acc += (double)r[l] * (double)zc;
      } else {
        res[l] = e;
        g[l] = a.w[0] * e / den[l];
      }
    }
    for (int st = 1; st <= a.m; ++st) {
      cluster_sync();
      vert_a(g);
      cluster_sync();
      for (int l = tid; l < cnt; l += kResBlock) {
        const TA xc = g[l];
        const TA val = xc + a.w[st] * (res[l] - row_a(g, l, xc)) / den[l];
        if (st < a.m) {
          gn[l] = val;
        } else {
          const TA zc = val + cur[l];
          z[l] = zc;
          acc += (double)r[l] * (double)zc;
        }
      }
      TA* t = g;
      g = gn;
      gn = t;
    }
    // ---- rho, beta
    const double rhon = reduce(acc, 0);
    double beta = 0;
    if (!(rhon > 0.0) || !isfinite(rhon)) flags |= first ? 8 : 2;
    if (first) {
      rho = rhon;
    } else if (!(flags & 2)) {
      beta = rhon / rho;
      rho = rhon;
    }
    // ---- q = A p, p.q
    const DsmDirection<S, TA> dir{vec(z), vec((its & 1) ? p1 : p0), S(beta), first};
    S* const pn = (its & 1) ? p0 : p1;
    vertices(w, vs, rvs, dir, S(1));
    cluster_sync();
    acc = 0;
    for (int l = tid; l < cnt; l += kResBlock) {
      const S pc = dir(lo + l);
      const S s = cs.nd16 ? split_row<S, S, true>(cs, dir, wvs, lo + l, pc, S(1))
                            : split_row<S, S, false>(cs, dir, wvs, lo + l, pc, S(1));
      pn[l] = pc;
      q[l] = s;
      acc += (double)pc * (double)s;
    }
    const double pq = reduce(acc, 1);
    double alpha = 0;
    if (!(pq > 0.0) || !isfinite(pq)) flags |= 1;
    else alpha = rho / pq;
    // ---- x, r, ||r||^2, the next first step
    const S al = S(alpha);
    acc = 0;
    for (int l = tid; l < cnt; l += kResBlock) {
      x[l] += al * pn[l];
      const S rr = r[l] - al * q[l];
      r[l] = rr;
      first_step(l, rr);
      acc += (double)rr * (double)rr;
    }
    rn2 = reduce(acc, 2);
    ++its;
    first = false;
    const double rn = sqrt(rn2);
    if (!isfinite(rn / fmax(r0, 1e-300))) flags |= 4;
    conv = rn <= target;
    if (conv || flags != 0 || its >= cap) break;
  }
  for (int l = tid; l < cnt; l += kResBlock) a.x[lo + l] = x[l];
  if (me == 0 && tid == 0) {
    a.sc[3] = rn2;
    a.ctl[0] = its;
    a.ctl[1] = conv;
    a.ctl[2] = 0;
    *a.flags = flags;
    a.host.put(its, conv, cap, flags, rn2);
  }
  cluster_sync();  // no block leaves while another may still read its memory
}

}  // namespace k
}  // namespace nds
