// Largest of value(0 .. n-1) (none negative) over a block of T threads, in every thread. `word` is shared
// memory that nothing else uses. Names of CUDA's device language only, so that host threads can run it too.
#pragma once

namespace cstg {

template <int T, class Value>
__device__ __forceinline__ int block_max(int* word, int n, Value value) {
  if (threadIdx.x == 0) *word = 0;
  __syncthreads();  // (a maximum taken before this store would be lost in it)
  for (int i = threadIdx.x; i < n; i += T) atomicMax(word, value(i));
  __syncthreads();
  return *word;
}

}  // namespace cstg
