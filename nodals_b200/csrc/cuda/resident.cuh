// PCG with its V-cycle as one kernel, for meshes that leave the chip idle.
//
// A PCG iteration of the split operator with a dense coarse level is fifteen
// kernels of one to three microseconds of work each; below about a hundred
// thousand cells their launches and their cold first loads are most of the
// time.  Here one block per SM (or one cluster of eight blocks on the
// smallest meshes) stays resident for the whole solve: the steps are
// separated by barriers, the operator's constant data stays in the L1 caches
// (a cell is always visited by the same thread), and only the vectors that
// other blocks read go through L2 (loads that bypass L1).
//
// The scalars are formed by every block from the same per-block partial sums
// in the same order, so all blocks take the same decisions and a run is
// reproducible.  Barriers between the blocks of a grid wait on a counter for
// at most kResidentSpins polls; when one runs out the kernel sets flag 32,
// and every block leaves.  The launch is cooperative (or one cluster), so all
// blocks run at the same time.
#pragma once
#include <cooperative_groups.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"
#include "split.cuh"

namespace nds {
namespace k {

constexpr int kResidentBlock = 512;
constexpr int kResidentWarps = kResidentBlock / 32;
constexpr int kResidentCluster = 8;
constexpr int kResidentSteps = 16;        // smoother degrees up to 16
constexpr unsigned kResidentSpins = 1u << 22;  // about a second
constexpr int kResidentRows = 64;         // rows of the dense level a block takes at a time
constexpr int kResidentParts = 4;         // warps that share such a row

template <class S, class TA>
struct Resident {
  int nc;
  // operator of the Krylov method (precision S) and of the V-cycle (TA)
  SplitVerts vs, va;
  SplitCells cs, ca;
  const S* rvs;
  const TA* rva;
  S* ws;
  TA* wa;
  TA wscale, tinv;
  const TA* den;
  int m;                     // smoothing steps after the diagonal one
  TA w[kResidentSteps];      // weights: diagonal step, then the steps
  // coarse level: R in CSR, its V-cycle matrix (row stride ld), P in ELL
  int nk, ld, pw;
  const int32_t* rr;
  const int32_t* rc;
  const TA* rv;
  const TA* dense;
  const int32_t* pc;
  const TA* pv;
  // vectors
  S *x, *r, *q, *p0, *p1;
  TA *z, *rA;                // rA: r in TA (r itself when S = TA)
  TA *b0, *b1, *g0, *g1, *res, *rhs2;
  TA *cb, *cx;               // coarse right-hand side (padded to ld) and result
  double* part;              // 3 x gridDim.x
  unsigned* bar;             // zero at launch
  double* sc;                // [3] ||r||^2 out
  int r0_slot, target_slot;
  int* flags;
  int* ctl;                  // [0] iterations, [1] converged out; [3] cap in
};

template <class T>
__device__ __forceinline__ T ld_l2(const T* p) {
  return __ldcg(p);
}

// a barrier of all blocks; false when it ran out
template <bool CLUSTER>
__device__ __forceinline__ bool resident_sync(unsigned* bar, unsigned& seq, int* flags) {
  if constexpr (CLUSTER) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    return true;
  } else {
    __shared__ int ok;
    ++seq;
    __syncthreads();
    if (threadIdx.x == 0) {
      const unsigned goal = seq * gridDim.x;
      unsigned now;
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
      unsigned n = 0;
      do {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(now) : "l"(bar) : "memory");
      } while ((int)(now - goal) < 0 && ++n < kResidentSpins);
      ok = (int)(now - goal) >= 0;
      if (!ok) atomicOr(flags, 32);
    }
    __syncthreads();
    return ok != 0;
  }
}

// products of one vertex's incidences with x (read through L2), group of
// eight lanes; the sums are valid in every lane
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

template <class V>
struct L2Vector {
  const V* x;
  __device__ __forceinline__ V operator()(int c) const { return ld_l2(x + c); }
};
// the search direction p = z + beta p_old, formed where it is read (p = z at
// the first iteration): two gathers, but one step between barriers less
template <class S, class TA>
struct L2Direction {
  const TA* z;
  const S* old;
  S beta;
  bool first;
  __device__ __forceinline__ S operator()(int c) const {
    const S zc = S(ld_l2(z + c));
    return first ? zc : zc + beta * ld_l2(old + c);
  }
};

template <class S, class TA, class MT, bool CLUSTER>
__global__ void __launch_bounds__(kResidentBlock, 1) pcg_resident(const Resident<S, TA> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TA* sv = reinterpret_cast<TA*>(smem_raw);  // a coarse vector (ld values)
  __shared__ TA srow[kResidentRows][kResidentParts];
  __shared__ double sred[kResidentWarps];
  __shared__ double stot;
  const int tid = threadIdx.x, nt = gridDim.x * kResidentBlock, gt = blockIdx.x * kResidentBlock + tid;
  const int lane = tid & 31, warp = tid >> 5;
  unsigned seq = 0;
  bool alive = true;

  auto sync = [&] { alive = alive && resident_sync<CLUSTER>(a.bar, seq, a.flags); };
  // sum over all threads of all blocks, the same value everywhere; also a barrier
  auto reduce = [&](double v, int slot) {
    v = warp_sum(v);
    if (lane == 0) sred[warp] = v;
    __syncthreads();
    if (tid == 0) {
      double s = 0;
      for (int q = 0; q < kResidentWarps; ++q) s += sred[q];
      a.part[slot * gridDim.x + blockIdx.x] = s;
      __threadfence();
    }
    sync();
    if (warp == 0) {
      double s = 0;
      for (int b = lane; b < (int)gridDim.x; b += 32) s += ld_l2(a.part + slot * gridDim.x + b);
      s = warp_sum(s);
      if (lane == 0) stot = s;
    }
    __syncthreads();
    return stot;
  };
  const unsigned mask8 = group8_mask();
  auto vertices = [&](auto tag, const SplitVerts& v, const auto* rau, const auto& x, auto* w, auto scale) {
    using V = decltype(tag);
    for (int g = gt >> 3; g < v.n; g += nt >> 3) {
      V s[3];
      const V r = scale * rau[g];
      resident_vertex<V>(v, g, tid & 7, mask8, x, s);
      if ((tid & 7) == 0) {
        if constexpr (std::is_same<V, float>::value) {
          reinterpret_cast<float4*>(w)[g] = make_float4(r * s[0], r * s[1], r * s[2], 0.f);
        } else {
          reinterpret_cast<double2*>(w)[2 * (size_t)g] = make_double2(r * s[0], r * s[1]);
          w[4 * (size_t)g + 2] = r * s[2];
        }
      }
    }
  };
  auto row_a = [&](const TA* x, int c, TA xc) {
    return a.ca.nd16 ? split_row<TA, MT, true, true>(a.ca, L2Vector<TA>{x}, a.wa, c, xc, a.tinv)
                     : split_row<TA, MT, false, true>(a.ca, L2Vector<TA>{x}, a.wa, c, xc, a.tinv);
  };
  auto vert_a = [&](const TA* x) { vertices(TA{}, a.va, a.rva, L2Vector<TA>{x}, a.wa, a.wscale); };

  // r in the V-cycle's precision and the first smoothing step
  auto first_step = [&](int c, S r) {
    TA ra;
    if constexpr (std::is_same<S, TA>::value) {
      ra = r;
    } else {
      ra = TA(r);
      a.rA[c] = ra;
    }
    a.b0[c] = a.w[0] * ra / a.den[c];
  };
  for (int c = gt; c < a.nc; c += nt) first_step(c, a.r[c]);
  const double target = a.sc[a.target_slot], r0 = a.sc[a.r0_slot];
  const int cap = a.ctl[3];
  double rho = 0, rn2 = 0;
  int its = 0, flags = 0, conv = 0;
  bool first = true;
  sync();

  while (alive) {
    // ---- z = M r
    TA* cur = a.b0;
    TA* nxt = a.b1;
    for (int st = 1; st <= a.m; ++st) {
      vert_a(cur);
      sync();
      for (int c = gt; c < a.nc; c += nt) {
        const TA xc = cur[c];
        nxt[c] = xc + a.w[st] * (a.rA[c] - row_a(cur, c, xc)) / a.den[c];
      }
      sync();
      TA* t = cur;
      cur = nxt;
      nxt = t;
    }
    vert_a(cur);
    sync();
    for (int c = gt; c < a.nc; c += nt) a.res[c] = a.rA[c] - row_a(cur, c, cur[c]);
    sync();
    // restriction: 16 lanes a coarse row
    {
      const int l16 = tid & 15;
      const unsigned m16 = group_mask<16>();
      for (int i = gt >> 4; i < a.nk; i += nt >> 4) {
        TA s = 0;
        const int re = a.rr[i + 1];
        for (int k0 = a.rr[i] + l16; k0 < re; k0 += 128) {
          int j[8];
          TA v[8], f[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const int k = k0 + 16 * u;
            j[u] = k < re ? a.rc[k] : -1;
            v[u] = k < re ? a.rv[k] : TA(0);
          }
#pragma unroll
          for (int u = 0; u < 8; ++u) f[u] = j[u] >= 0 ? ld_l2(a.res + j[u]) : TA(0);
#pragma unroll
          for (int u = 0; u < 8; ++u) s += v[u] * f[u];
        }
        s = group_sum<16>(s, m16);
        if (l16 == 0) a.cb[i] = s;
      }
    }
    sync();
    // dense coarse level: each block takes the rows blockIdx.x + k gridDim.x,
    // four warps a row (a few dozen rows of 10 to 40 KB per block)
    {
      constexpr int W = 16 / sizeof(TA);
      using V4 = typename std::conditional<std::is_same<TA, float>::value, float4, double2>::type;
      V4* s4 = reinterpret_cast<V4*>(sv);
      const int nv = a.ld / W;
      for (int k = tid; k < nv; k += kResidentBlock) s4[k] = ld_l2(reinterpret_cast<const V4*>(a.cb) + k);
      __syncthreads();
      const int per = (nv + kResidentParts - 1) / kResidentParts;
      const int rows = blockIdx.x < (unsigned)a.nk ? (a.nk - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
      for (int base = 0; base < rows; base += kResidentRows) {
        const int cnt = rows - base < kResidentRows ? rows - base : kResidentRows;
        for (int t = warp; t < cnt * kResidentParts; t += kResidentWarps) {
          const int rI = t / kResidentParts, pt = t % kResidentParts;
          const size_t i = blockIdx.x + (size_t)(base + rI) * gridDim.x;
          const V4* A4 = reinterpret_cast<const V4*>(a.dense + i * a.ld);
          const int e = min(nv, (pt + 1) * per);
          TA s = 0;
#pragma unroll 4
          for (int k = pt * per + lane; k < e; k += 32) {
            const V4 p = __ldcs(A4 + k), q = s4[k];
            if constexpr (W == 4) s += p.x * q.x + p.y * q.y + p.z * q.z + p.w * q.w;
            else s += p.x * q.x + p.y * q.y;
          }
          s = warp_sum(s);
          if (lane == 0) srow[rI][pt] = s;
        }
        __syncthreads();
        if (tid < cnt) {
          TA s = srow[tid][0];
#pragma unroll
          for (int q = 1; q < kResidentParts; ++q) s += srow[tid][q];
          a.cx[blockIdx.x + (size_t)(base + tid) * gridDim.x] = s;
        }
        __syncthreads();
      }
    }
    sync();
    // x += P x_c
    for (int k = tid; k < a.nk; k += kResidentBlock) sv[k] = ld_l2(a.cx + k);
    __syncthreads();
    for (int c = gt; c < a.nc; c += nt) {
      TA s = 0;
      for (int k = 0; k < a.pw; ++k) {
        const size_t o = (size_t)k * a.nc + c;
        s += a.pv[o] * sv[a.pc[o]];
      }
      cur[c] += s;
    }
    sync();
    // post-smoothing; the last step forms z and r.z
    vert_a(cur);
    sync();
    double acc = 0;
    TA* g = a.g0;
    TA* gn = a.g1;
    for (int c = gt; c < a.nc; c += nt) {
      const TA xc = cur[c];
      const TA q = a.rA[c] - row_a(cur, c, xc);
      if (a.m == 0) {
        const TA zc = xc + a.w[0] * q / a.den[c];
        a.z[c] = zc;
        acc += (double)a.r[c] * (double)zc;
      } else {
        a.rhs2[c] = q;
        g[c] = a.w[0] * q / a.den[c];
      }
    }
    for (int st = 1; st <= a.m; ++st) {
      sync();
      vert_a(g);
      sync();
      for (int c = gt; c < a.nc; c += nt) {
        const TA xc = g[c];
        const TA val = xc + a.w[st] * (a.rhs2[c] - row_a(g, c, xc)) / a.den[c];
        if (st < a.m) {
          gn[c] = val;
        } else {
          const TA zc = val + cur[c];
          a.z[c] = zc;
          acc += (double)a.r[c] * (double)zc;
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
    if (first) rho = rhon;
    else if (!(flags & 2)) {
      beta = rhon / rho;
      rho = rhon;
    }
    // ---- q = A p, p.q
    const L2Direction<S, TA> dir{a.z, (its & 1) ? a.p1 : a.p0, S(beta), first};
    S* pn = (its & 1) ? a.p0 : a.p1;
    vertices(S{}, a.vs, a.rvs, dir, a.ws, S(1));
    sync();
    acc = 0;
    for (int c = gt; c < a.nc; c += nt) {
      const S pc = dir(c);
      const S s = a.cs.nd16 ? split_row<S, S, true, true>(a.cs, dir, a.ws, c, pc, S(1))
                            : split_row<S, S, false, true>(a.cs, dir, a.ws, c, pc, S(1));
      pn[c] = pc;
      a.q[c] = s;
      acc += (double)pc * (double)s;
    }
    const double pq = reduce(acc, 1);
    double alpha = 0;
    if (!(pq > 0.0) || !isfinite(pq)) flags |= 1;
    else alpha = rho / pq;
    // ---- x, r, ||r||^2, the next first step
    const S al = S(alpha);
    acc = 0;
    for (int c = gt; c < a.nc; c += nt) {
      a.x[c] += al * pn[c];
      const S rr = a.r[c] - al * a.q[c];
      a.r[c] = rr;
      first_step(c, rr);
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
  if (gt == 0) {
    a.sc[3] = rn2;
    a.ctl[0] = its;
    a.ctl[1] = conv;
    a.ctl[2] = 0;
    if (flags) atomicOr(a.flags, flags);
  }
}

}  // namespace k
}  // namespace nds
