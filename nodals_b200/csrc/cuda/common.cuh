// Shared device helpers for the sm_100a kernels.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <stdexcept>
#include <string>

namespace nds {

struct CudaError : std::runtime_error {
  using std::runtime_error::runtime_error;
};

inline void cuda_check(cudaError_t e, const char* what, const char* file, int line) {
  if (e != cudaSuccess)
    throw CudaError(std::string("CUDA failure ") + what + " at " + file + ":" + std::to_string(line) + ": " +
                    cudaGetErrorString(e));
}
#define NDS_CUDA(call) ::nds::cuda_check((call), #call, __FILE__, __LINE__)
// every kernel launch of the library goes through NDS_LAUNCH, which also
// counts launches (nds_launch_count)
extern unsigned long long g_launches;
#define NDS_LAUNCH() (++::nds::g_launches, ::nds::cuda_check(cudaGetLastError(), "kernel launch", __FILE__, __LINE__))

// Launch of a kernel that begins with pdl_begin(): the grid may be set up
// while the kernel before it in the stream still runs (programmatic dependent
// launch), which takes about a microsecond off every step of a chain of short
// kernels.  pdl_trigger() lets the next kernel be set up, pdl_wait() waits for
// the whole of the previous one (and so for all before it).  Every kernel
// launched this way calls both; before pdl_wait() it may read only what no
// kernel of the stream writes between a full dependency (host
// synchronisation, event wait, graph boundary) and itself: the kernels of the
// pressure solve load their matrix entries there, constant during a solve, so
// that these round trips overlap the previous kernel's end.  For the same
// reason a pointer to memory that a kernel of such a chain writes is no
// __restrict__ parameter where it is read: const __restrict__ lets the compiler
// take its loads as invariant for the whole kernel, which begins before the
// writer has ended, and move them above pdl_wait().  Constant data and outputs
// that are only stored to keep the qualifier.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_begin() {
  pdl_trigger();
  pdl_wait();
}
template <class... P, class... A>
inline void pdl_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  NDS_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
}

constexpr int kBlock = 256;
constexpr int kWarps = kBlock / 32;

inline int grid_for(long long n, int per_block = kBlock) {
  long long g = (n + per_block - 1) / per_block;
  return (int)(g < 1 ? 1 : g);
}

template <class T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// sum over an aligned group of G lanes (G a power of two <= 32); mask names
// exactly the lanes of the calling group, which may have diverged from the
// other groups of its warp
template <int G, class T>
__device__ __forceinline__ T group_sum(T v, unsigned mask) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o, G);
  return v;
}
// lanes of the aligned 8-lane group of the calling thread
__device__ __forceinline__ unsigned group8_mask() { return 0xffu << (threadIdx.x & 24); }
// lanes of the aligned G-lane group of the calling thread (G = 8, 16 or 32)
template <int G>
__device__ __forceinline__ unsigned group_mask() {
  return G == 32 ? 0xffffffffu : (((1u << G) - 1u) << (threadIdx.x & (32 - G)));
}

// Deterministic block reduction of NV doubles; thread 0 holds the sums.
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV]) {
  __shared__ double red[kWarps][NV];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = warp_sum(v[k]);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) red[w][k] = v[k];
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      double s = 0;
      for (int q = 0; q < kWarps; ++q) s += red[q][k];
      v[k] = s;
    }
  }
  __syncthreads();
}

}  // namespace nds
