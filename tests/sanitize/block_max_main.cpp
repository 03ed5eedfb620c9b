// csrc/block_max.cuh run by host threads in place of a block's: thread 0 reaches the function last.
#include <algorithm>
#include <barrier>
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>

constexpr int kT = 8;
static thread_local struct {
  int x;
} threadIdx;
static std::barrier<> block(kT);
static void __syncthreads() { block.arrive_and_wait(); }
static int atomicMax(int* p, int v) {
  int old = __atomic_load_n(p, __ATOMIC_RELAXED);
  while (old < v && !__atomic_compare_exchange_n(p, &old, v, false, __ATOMIC_RELAXED, __ATOMIC_RELAXED)) {
  }
  return old;
}
#define __device__
#define __forceinline__ inline
#include "../../mpi-cst-fem-solver_b200/csrc/block_max.cuh"

int main() {
  int wrong = 0;
  for (int n : {0, 1, 5, kT, 3 * kT + 2}) {
    int word = -1;
    std::vector<int> got(kT, -1);
    std::vector<std::thread> threads;
    for (int t = 0; t < kT; ++t)
      threads.emplace_back([&, t] {
        threadIdx.x = t;
        if (t == 0) std::this_thread::sleep_for(std::chrono::milliseconds(50));
        got[t] = cstg::block_max<kT>(&word, n, [&](int i) { return 7 + (i * 5) % 11; });
      });
    for (std::thread& t : threads) t.join();
    int most = 0;
    for (int i = 0; i < n; ++i) most = std::max(most, 7 + (i * 5) % 11);
    for (int g : got) wrong += g != most;
  }
  std::printf("%s\n", wrong ? "wrong" : "ok");
  return wrong != 0;
}
