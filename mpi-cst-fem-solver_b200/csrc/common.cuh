// Shared device helpers for the CST / Jacobi-PCG kernels (sm_100a).
#pragma once

#include <utility>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/cstfem_b200.h"

namespace cstg {

// Launch geometry. 148 SMs on a B200; the fixed grids below are multiples of it so that the
// deterministic reductions see the same partial-sum layout on every run.
constexpr int kSMs = 148;
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
// Largest grid of the reduction kernels (their partial-sum buffers hold 4 x kMaxGrid doubles).
// The actual grid is one full wave: SMs x resident blocks per SM (occupancy calculator).
constexpr int kMaxGrid = 2048;

// Largest node neighbourhood (self included) the pattern builder accepts.
constexpr int kMaxNeighbours = 64;

// Bounded spin limit for grid barriers (iterations of a ~100 ns poll): about 2 s.
constexpr long long kSpinLimit = 20000000LL;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Deterministic block sum: fixed shuffle tree, then warp 0 sums the warp totals in order.
// Every thread must call it; the result is valid in all threads.
template <int NT>
__device__ __forceinline__ double block_sum(double v, double* smem /* >= NT/32 */) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) smem[w] = v;
  __syncthreads();
  double t = 0.0;
  if (w == 0) {
    t = lane < NT / 32 ? smem[lane] : 0.0;
    t = warp_sum(t);
    if (lane == 0) smem[0] = t;
  }
  __syncthreads();
  t = smem[0];
  __syncthreads();
  return t;
}

// Loads that bypass L1 (data written by other blocks of the same grid).
__device__ __forceinline__ double ld_cg(const double* p) { return __ldcg(p); }
__device__ __forceinline__ int ld_cg(const int* p) { return __ldcg(p); }

// ---- launches that overlap their predecessor's end ------------------------------------------------
// A kernel launched by launch_next may start while the kernel before it on the stream is still running;
// it calls wait_previous() before anything that depends on that kernel (or on what it overwrites), which
// returns when that kernel has finished and its writes are visible. A kernel calls start_next() after that,
// if at all, so whatever came before a kernel's predecessor has finished too. Worth it where a kernel has
// a prologue and the next one the same shared-memory split: encoder and layers of the network, 353 -> 341
// us for 1,000,122 nodes. Not between the multigrid cycle's kernels: overlapping kernels keep the SM's
// split of shared memory and L1 (after a layer: hardly any L1 for the sweeps' gathers), and the learned
// solve of that plate took 82 to 109 ms instead of 78.
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void start_next() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

// A load of what the kernel before wrote: this kernel was alive then, so the data is not read-only for its
// lifetime, which __ldg (ld.global.nc) asks for. After wait_previous().
__device__ __forceinline__ uint4 ld_chained(const uint4* p) {
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

template <class... P, class... A>
cudaError_t launch_next(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

}  // namespace cstg
