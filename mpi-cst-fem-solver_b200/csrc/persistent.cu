// Persistent Jacobi-PCG: one launch runs every iteration of a solve, on the mesh (2x2-block) matrix
// in FP64 or mixed precision, or on a caller's CSR matrix in FP64.
//
// Per iteration, two phases and two reductions over the team of blocks:
//   1  x += alpha p of the iteration before, p = z + beta p, Ap = A p, p'Ap   -> alpha
//   2  r -= alpha Ap, z = D^-1 r, r'r, r'z                                    -> convergence test, beta
//   R  (mixed, when due) r = b - A64 x                                        -> reliable update / switch
// The recurrence and every operation on a vector element are those of the per-phase kernels
// (solver.cpp:35-105); only the order of the sums differs.
//
// Each block owns a contiguous range of nodes (rows). It keeps p at its own nodes and at its halo (the
// other blocks' nodes that its rows read) in shared memory and updates both itself, so z at the halo
// is all that passes between blocks: 16 bytes of payload per halo node instead of a vector gather
// per matrix block. The halo, the rows' 16-bit numbering of their neighbours in [own | halo] and
// the list of nodes that others need are built at the start of the launch. r, Ap, x and D^-1 at own
// nodes live in shared memory as far as they fit, and so does the matrix when all of it fits (33 MB
// over 148 SMs: O-grids of up to about 200k DOFs in FP64, 290k mixed). A larger matrix is streamed: every
// warp has a ring of stages that bulk copies fill with its next groups of rows, also while the block
// waits in a reduction, so the copies never stop for one. What no block can hold, O-grids above about 2.1M DOFs
// and, from about 400k, numberings without locality, whose halos do not fit, is left to the grid kernel
// (persistent_grid.cu), or for a caller's CSR to the captured kernels.
//
// Nothing between blocks needs a memory fence: a word of z or of a partial sum carries the number of
// its reduction in its upper half (32 bits of payload per 64-bit word), so a reader polls the data
// itself. Both are double-buffered by that number's parity. Polls are bounded (spin_limit): a
// block that gives up sets bar_err and returns, and so do all others; the host reports the timeout.
//
// What bounds it: at small sizes two reductions of 1 to 2.5 us and the chain of shared-memory reads of
// a row; at large ones the bytes that do not fit on the chip. Against three passes with a grid barrier
// of the last-block kind after each (us an iteration, before and now): 3,321 nodes FP64 20 -> 3.9;
// 65,341 nodes FP64 21 -> 7.9; 15,006 CSR rows 25 -> 5.9 (three kernels an iteration in a graph before);
// 501,651 nodes mixed 47 -> 22 (120 MB that cannot be avoided: 18 at the measured 6.5 TB/s), FP64 54 ->
// 28; 1,000,122 nodes FP64 96 -> 61, mixed 77 -> 49.
//
// Reductions. A block adds its threads' values in a fixed order and hands the sums to every block;
// every block adds all blocks' sums in index order and takes the same decisions, so no last block
// does serial work for the others and nothing is released.
//  * Grid team (cooperative launch, one block per SM): a block writes its sums to every block's own
//    inbox in global memory, so each inbox is polled by one warp alone.
//  * Cluster team (one cluster of up to 16 blocks, small systems): sums go to every block's shared
//    memory before the cluster barrier, a hardware barrier that needs no polling.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "block_max.cuh"
#include "common.cuh"
#include "kernels.h"

namespace cg = cooperative_groups;

namespace cstg {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kClusterTeam = 16;
constexpr int kMaxTeam = 160;  // blocks of a grid team (five slots per polling lane)
constexpr int kCopies = 16;     // copies of the published sums: block b polls copy b % kCopies

enum Op { kBlock64 = 0, kMixed = 1, kCsr = 2 };

// ---- element types: a node's two DOFs, or one row of a CSR matrix ---------------------------------
__device__ __forceinline__ double2 vzero(double2) { return make_double2(0.0, 0.0); }
__device__ __forceinline__ double vzero(double) { return 0.0; }
__device__ __forceinline__ double2 axpy(double s, double2 a, double2 b) {
  return make_double2(fma(s, a.x, b.x), fma(s, a.y, b.y));
}
__device__ __forceinline__ double axpy(double s, double a, double b) { return fma(s, a, b); }
__device__ __forceinline__ double2 mul(double2 a, double2 b) { return make_double2(a.x * b.x, a.y * b.y); }
__device__ __forceinline__ double mul(double a, double b) { return a * b; }
__device__ __forceinline__ double dot(double2 a, double2 b, double c) { return fma(a.x, b.x, fma(a.y, b.y, c)); }
__device__ __forceinline__ double dot(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ double2 sub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }

template <class V>
__device__ __forceinline__ V ld(const V* p) {  // written by other blocks: always from L2
  return __ldcg(p);
}

struct SolveArgs {
  int n = 0;  // nodes, or rows of a CSR matrix
  BlockMatrix A64;
  MixedMatrix A32;
  CsrMatrixDev csr;
  double *x = nullptr, *r = nullptr, *Ap = nullptr;
  double* p = nullptr;        // out, after a precision switch: the next direction
  ulonglong2* z = nullptr;           // [2][n] tagged z (a node: two pairs of words, a row: one), zero at launch
  // neighbours in the block's own numbering: of the streamed matrix's entries, or (mixed, resident)
  // of the FP64 blocks that a precision switch goes on with
  unsigned short* lcol = nullptr;
  const double* invd = nullptr;
  const double* b = nullptr;
  double* history = nullptr;
  PcgState* st = nullptr;
  unsigned char* wanted = nullptr;   // nodes that other blocks need, zero at launch
  ulonglong2* sums = nullptr;        // grid team: [2][kCopies][kMaxTeam][2], zero at launch
  int max_final_checks = 0;
  long long spin_limit = 0;
  unsigned smem = 0;  // dynamic shared memory of a block
};

// One of the block's own vectors: the first `lim` entries in shared memory (ALL: every one).
template <class V, bool ALL>
struct Own {
  V *s, *g;
  int lim;
  __device__ __forceinline__ V& operator[](int i) const { return ALL || i < lim ? s[i] : g[i]; }
};

constexpr int kHash = 16384;  // slots of the halo's hash set; a halo holds at most half as many

constexpr int kStages = 2;  // of a warp's ring

// What only the mixed method's reliable updates need (thread 0 writes, see phase R).
struct Reliable {
  double best_true, true_rel;
  int replaced, final_checks, switch_iter, stall;
};

template <int T>
struct Shared {
  double red[2][T / 32];
  double tot[2];
  double inbox[2][16][2];  // cluster team: every block's sums, double-buffered
  unsigned long long full[T / 32][kStages];  // mbarriers of the warps' rings
  Reliable rel;
  int scan[T / 32];
  int ok;
  int halo;     // nodes of the halo
  int widest;   // entries of the widest group of rows
};

// ---- reductions ----------------------------------------------------------------------------------

__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ void st_tagged(ulonglong2* p, double v, unsigned tag) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(v), e = (unsigned long long)tag << 32;
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(e | (u & 0xffffffffull)),
               "l"(e | (u >> 32))
               : "memory");
}
__device__ __forceinline__ bool ld_tagged(const ulonglong2* p, unsigned tag, double& v) {
  unsigned long long lo, hi;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(lo), "=l"(hi) : "l"(p) : "memory");
  v = __longlong_as_double((long long)((lo & 0xffffffffull) | (hi << 32)));
  return (unsigned)(lo >> 32) == tag && (unsigned)(hi >> 32) == tag;
}
__device__ __forceinline__ void st_z(ulonglong2* z, int i, double2 v, unsigned tag) {
  st_tagged(z + 2L * i, v.x, tag);
  st_tagged(z + 2L * i + 1, v.y, tag);
}
__device__ __forceinline__ void st_z(ulonglong2* z, int i, double v, unsigned tag) { st_tagged(z + i, v, tag); }
__device__ __forceinline__ bool ld_z(const ulonglong2* z, int i, unsigned tag, double2& v) {
  const bool a = ld_tagged(z + 2L * i, tag, v.x), b = ld_tagged(z + 2L * i + 1, tag, v.y);
  return a && b;
}
__device__ __forceinline__ bool ld_z(const ulonglong2* z, int i, unsigned tag, double& v) {
  return ld_tagged(z + i, tag, v);
}
// A poll reads a line from L2 (about 0.7 us with its loop), so it counts for 16 of the limit's polls (40 ns).
constexpr long long kPollWeight = 16;
// One more poll of a wait: false when it has to give up (its limit, or another block's timeout).
__device__ __forceinline__ bool poll_again(const SolveArgs& a, long long& spins) {
  spins += kPollWeight;
  return spins <= a.spin_limit && ((spins & (64 * kPollWeight - 1)) != 0 || !__ldcg(&a.st->bar_err));
}
__device__ __forceinline__ void give_up(const SolveArgs& a) {
  atomicExch(&a.st->bar_err, 1);
  a.st->done = CSTG_SOLVE_TIMEOUT + 1;
}

// Sum over the first N lanes of a warp (the others hold zero), in every lane.
template <int N>
__device__ __forceinline__ double first_lanes_sum(double v) {
  constexpr int P = N > 8 ? 8 : N > 4 ? 4 : N > 2 ? 2 : 1;
#pragma unroll
  for (int o = P; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return __shfl_sync(kFull, v, 0);
}

// Sums NV values per thread over the team; every thread of every block gets the totals. FENCE: data
// written before it with plain stores is visible to the other blocks after it. False: a wait of
// this block ran out, here or since the last reduction (sh.ok).
template <int NV, bool FENCE, bool CLUSTER, int T>
__device__ __forceinline__ bool team_sum(const SolveArgs& a, Shared<T>& sh, unsigned& tag, double (&v)[NV]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    v[q] = warp_sum(v[q]);
    if (lane == 0) sh.red[q][w] = v[q];
  }
  ++tag;
  __syncthreads();
  if constexpr (CLUSTER) {
    const cg::cluster_group cl = cg::this_cluster();
    const int C = (int)cl.num_blocks();
    double(*box)[2] = sh.inbox[tag & 1u];
    if (w == 0) {
      double s[NV];
#pragma unroll
      for (int q = 0; q < NV; ++q) s[q] = first_lanes_sum<T / 32>(lane < T / 32 ? sh.red[q][lane] : 0.0);
      if (lane < C) {
        double* to = cl.map_shared_rank(&box[cl.block_rank()][0], lane);
#pragma unroll
        for (int q = 0; q < NV; ++q) to[q] = s[q];
      }
    }
    cl.sync();  // release / acquire at cluster scope
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      double s = 0.0;
      for (int i = 0; i < C; ++i) s += box[i][q];
      v[q] = s;
    }
    return sh.ok != 0;
  } else {
    if (w == 0) {
      const int G = gridDim.x;
      ulonglong2* box = a.sums + (tag & 1u) * (2L * kCopies * kMaxTeam);
      double s[NV];
#pragma unroll
      for (int q = 0; q < NV; ++q) s[q] = first_lanes_sum<T / 32>(lane < T / 32 ? sh.red[q][lane] : 0.0);
      if (FENCE) fence_gpu();
      if (lane < kCopies) {
#pragma unroll
        for (int q = 0; q < NV; ++q) st_tagged(box + 2L * (lane * kMaxTeam + (int)blockIdx.x) + q, s[q], tag);
      }
      box += 2L * kMaxTeam * (blockIdx.x % kCopies);
      long long spins = 0;
      bool ok = true;
      while (true) {
        bool all = true;
#pragma unroll
        for (int q = 0; q < NV; ++q) s[q] = 0.0;
#pragma unroll
        for (int k = 0; k < kMaxTeam / 32; ++k) {
          const int i = lane + 32 * k;
          if (i < G) {
#pragma unroll
            for (int q = 0; q < NV; ++q) {
              double t;
              all &= ld_tagged(box + 2 * i + q, tag, t);
              s[q] += t;
            }
          }
        }
        if (__all_sync(kFull, all)) break;
        if (!(ok = __all_sync(kFull, poll_again(a, spins)))) break;
      }
      if (FENCE) fence_gpu();
#pragma unroll
      for (int q = 0; q < NV; ++q) s[q] = warp_sum(s[q]);
      if (lane == 0) {
#pragma unroll
        for (int q = 0; q < NV; ++q) sh.tot[q] = s[q];
        if (!ok) {
          sh.ok = 0;
          give_up(a);
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NV; ++q) v[q] = sh.tot[q];
    return sh.ok != 0;
  }
}

// ---- rows of Ap = A p, L lanes per node (row); p by local slot --------------------------------------
// U steps of L neighbours have their matrix loads in flight together.

template <int L>
__device__ __forceinline__ double lane_sum(double v) {
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

// The loops have no branch per neighbour: past a row's end the last entry is read again and multiplied by
// an exact zero.

// IDX: unsigned short (a slot of p) or int (a node of a vector in global memory)
template <int L, class IDX>
__device__ __forceinline__ double2 row_block64(const int* ptr, const IDX* nbr, const double2* v2, int i, bool ok,
                                               const double2* p) {
  constexpr int U = L >= 8 ? 1 : L >= 4 ? 2 : 4;
  const int l = threadIdx.x & (L - 1);
  double ya = 0.0, yb = 0.0;
  if (ok) {
    const int b0 = ptr[i], deg = ptr[i + 1] - b0;
    const double2 *ra = v2 + 2L * b0, *rb = ra + deg;
    for (int k0 = l; k0 < deg; k0 += U * L) {
      double2 pv[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int k = k0 + u * L;
        const int m = nbr[b0 + min(k, deg - 1)];
        pv[u] = sizeof(IDX) == 2 ? p[m] : ld(p + m);
        if (k >= deg) pv[u] = make_double2(0.0, 0.0);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int k = min(k0 + u * L, deg - 1);
        ya = dot(ra[k], pv[u], ya);
        yb = dot(rb[k], pv[u], yb);
      }
    }
  }
  return make_double2(lane_sum<L>(ya), lane_sum<L>(yb));
}

// FP32 difference form (mixed_kernels.cu): sum K_nm (p_m - p_n) + S_n p_n
template <int L>
__device__ __forceinline__ double2 row_mixed(const int* ptr, int self, const unsigned short* nbr, const float4* val,
                                             const double2* S, int i, bool ok, const double2* p, double2 pn) {
  constexpr int U = L >= 8 ? 1 : L >= 4 ? 2 : 3;
  const int l = threadIdx.x & (L - 1);
  double ya = 0.0, yb = 0.0;
  if (ok) {
    // node i's off-diagonal blocks start at ptr[i] less the self blocks before it (self + i)
    const int b = ptr[i], o = b - (self + i), c = ptr[i + 1] - b - 1;
    for (int k0 = l; k0 < c; k0 += U * L) {
      double2 d[U];
      float4 f[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int k = k0 + u * L, kk = min(k, c - 1);
        d[u] = sub(p[nbr[o + kk]], pn);
        f[u] = val[o + kk];
        if (k >= c) d[u] = make_double2(0.0, 0.0);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        ya = fma((double)f[u].x, d[u].x, fma((double)f[u].y, d[u].y, ya));
        yb = fma((double)f[u].z, d[u].x, fma((double)f[u].w, d[u].y, yb));
      }
    }
  }
  ya = lane_sum<L>(ya);
  yb = lane_sum<L>(yb);
  if (ok) {
    ya = dot(S[2 * i], pn, ya);
    yb = dot(S[2 * i + 1], pn, yb);
  }
  return make_double2(ya, yb);
}

template <int L>
__device__ __forceinline__ double row_csr(const int* rp, const unsigned short* cols, const double* vals, int i,
                                          bool ok, const double* p) {
  constexpr int U = L >= 8 ? 2 : 4;
  const int l = threadIdx.x & (L - 1);
  double s = 0.0;
  if (ok) {
    const int hi = rp[i + 1];
    for (int k0 = rp[i] + l; k0 < hi; k0 += U * L) {
      double pv[U], f[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int k = k0 + u * L, kk = min(k, hi - 1);
        pv[u] = p[cols[kk]];
        f[u] = vals[kk];
        if (k >= hi) pv[u] = 0.0;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) s = fma(f[u], pv[u], s);
    }
  }
  return lane_sum<L>(s);
}

// Rows read from global memory: the mixed method's residuals and its iterations after a precision
// switch. Rare, so a call, which keeps its registers out of the main loop.
template <int L, class IDX>
__device__ __noinline__ double2 row_block64_call(const int* ptr, const IDX* nbr, const double2* v2, int i, bool ok,
                                                 const double2* p) {
  return row_block64<L, IDX>(ptr, nbr, v2, i, ok, p);
}

// ---- streaming: a warp's ring of stages -------------------------------------------------------------

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes, uint32_t bar, uint64_t policy) {
  if (bytes)
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;\n" ::"r"(
            smem_addr(dst)),
        "l"(src), "r"(bytes), "r"(bar), "l"(policy)
        : "memory");
}
// Bounded wait for a phase of an mbarrier (try_wait suspends the thread a while by itself, so a poll
// here is long and a million of them are enough).
__device__ __forceinline__ bool stage_wait(uint32_t bar, uint32_t parity, long long limit) {
  limit = min(limit, 1LL << 20);
  for (long long i = 0; i <= limit; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// One group of rows in a stage: matrix values, then (mixed) the row-block sums, then the neighbours'
// slots. Slots start on the 16-byte boundary at or before the group's first one.
template <int OP>
struct Group {
  int i0, i1;      // rows of the group in the block
  int first, ne;   // its entries in the global arrays
  __device__ __forceinline__ Group(const int* ptr, int n0, int cnt, int g, int rows) {
    i0 = g * rows;
    i1 = min(cnt, i0 + rows);
    first = ptr[i0] - (OP == kMixed ? n0 + i0 : 0);
    ne = ptr[i1] - (OP == kMixed ? n0 + i1 : 0) - first;
  }
  __device__ __forceinline__ int slot0() const { return first & ~7; }
};
template <int OP>
constexpr int kEntryBytes = OP == kMixed ? 16 : 32;

// ---- the halo -------------------------------------------------------------------------------------

// Exclusive prefix sum of c over the block; `total` gets the sum.
template <int T>
__device__ __forceinline__ int block_scan(int c, Shared<T>& sh, int& total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int s = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(kFull, s, o);
    if (lane >= o) s += t;
  }
  if (lane == 31) sh.scan[w] = s;
  __syncthreads();
  int before = 0;
  total = 0;
  for (int q = 0; q < T / 32; ++q) {
    if (q < w) before += sh.scan[q];
    total += sh.scan[q];
  }
  __syncthreads();
  return before + s - c;
}

// Collects the nodes outside [n0, n1) among cols[e0 .. e1) in a hash set keyed by the node's low bits
// (so the compacted list keeps runs of consecutive nodes together), lists them in hid[] and gives
// every one a slot from n1 - n0 on. Returns their number, or -1 when there are more than cap (or an
// entry that is no node at all).
template <int T>
__device__ __forceinline__ int build_halo(const int* cols, int e0, int e1, int n, int n0, int n1, int cap, int* keys,
                                          unsigned short* slot, int* hid, Shared<T>& sh) {
  for (int i = threadIdx.x; i < kHash; i += T) keys[i] = -1;
  if (threadIdx.x == 0) sh.halo = 0;
  __syncthreads();
  volatile int* count = &sh.halo;
  for (int e = e0 + (int)threadIdx.x; e < e1 && *count <= cap; e += T) {
    const int m = cols[e];
    if (m >= n0 && m < n1) continue;
    if (m < 0 || m >= n) {
      atomicAdd(&sh.halo, 2 * kHash);
      break;
    }
    // at most cap + T <= kHash / 2 + T keys are ever inserted, so a probe always ends
    for (int h = m & (kHash - 1);; h = (h + 1) & (kHash - 1)) {
      const int k = atomicCAS(&keys[h], -1, m);
      if (k == -1) atomicAdd(&sh.halo, 1);
      if (k == -1 || k == m) break;
    }
  }
  __syncthreads();
  if (sh.halo > cap) return -1;
  constexpr int per = (kHash + T - 1) / T;
  const int h0 = min((int)threadIdx.x * per, kHash), h1 = min(h0 + per, kHash);
  int mine = 0, total;
  for (int h = h0; h < h1; ++h) mine += keys[h] >= 0;
  int at = block_scan<T>(mine, sh, total);
  for (int h = h0; h < h1; ++h) {
    const int k = keys[h];
    if (k >= 0) {
      hid[at] = k;
      slot[h] = (unsigned short)(n1 - n0 + at);
      ++at;
    }
  }
  __syncthreads();
  return total;
}

__device__ __forceinline__ unsigned short local_slot(int m, int n0, int n1, const int* keys,
                                                     const unsigned short* slot) {
  if (m >= n0 && m < n1) return (unsigned short)(m - n0);
  int h = m & (kHash - 1);
  while (keys[h] != m) h = (h + 1) & (kHash - 1);  // (every such m is in the set)
  return slot[h];
}

// ---- the solve -------------------------------------------------------------------------------------

template <int OP>
struct Elem {
  using V = double2;
};
template <>
struct Elem<kCsr> {
  using V = double;
};

template <int OP, bool CLUSTER, bool RES, int L, int T>
__global__ void __launch_bounds__(T, 1) k_pcg_persistent(const SolveArgs a) {
  using V = typename Elem<OP>::V;
  constexpr int kGroup = 32 / L, kWarpsT = T / 32;  // rows of a warp's group
  constexpr int kZ = sizeof(V) / 8;
  constexpr int kU = RES ? 2 : 4;  // elements of a vector loop whose loads are in flight together
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ Shared<T> sh;
  PcgState* st = a.st;
  if (__ldcg(&st->done)) return;
  const int G = gridDim.x;
  const int n0 = (int)((long long)a.n * blockIdx.x / G), n1 = (int)((long long)a.n * (blockIdx.x + 1) / G);
  const int cnt = n1 - n0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned tag = 0;
  if (threadIdx.x == 0) sh.ok = 1;
  if constexpr (CLUSTER) cg::this_cluster().sync();  // every block runs before its inbox is written

  // -- the halo and the rows' local numbering
  const int* gptr = (OP == kCsr ? a.csr.row_ptr : OP == kMixed ? a.A32.node_ptr : a.A64.node_ptr) + n0;
  const int* gcol = OP == kCsr ? a.csr.cols : OP == kMixed ? a.A32.nbr32 : a.A64.bnbr;
  const int e0 = cnt > 0 ? gptr[0] : 0, e1 = cnt > 0 ? gptr[cnt] : 0;
  const int first = OP == kMixed ? e0 - n0 : e0;  // first entry of the block in gcol
  const int last = OP == kMixed ? e1 - n1 : e1;
  int* hid = reinterpret_cast<int*>(dyn);
  int nh;
  const int groups = (cnt + kGroup - 1) / kGroup;
  unsigned stage_S = 0, stage_col = 0, stage_bytes = 0;  // a stage: offsets of the sums and slots, size
  if constexpr (!RES) {
    const unsigned widest =
        (unsigned)block_max<T>(&sh.widest, groups, [&](int g) { return Group<OP>(gptr, n0, cnt, g, kGroup).ne; });
    stage_S = (widest * kEntryBytes<OP> + 15u) & ~15u;
    stage_col = stage_S + (OP == kMixed ? 32u * kGroup : 0u);
    stage_bytes = stage_col + ((widest * 2u + 14u + 15u) & ~15u);
  }
  {
    // p at own nodes and halo, the halo's list, the row starts and the wanted bits must fit, and
    // with them the own vectors and the matrix (RES) or the rings
    long long room = (long long)a.smem - (long long)cnt * ((int)sizeof(V) + 4) - cnt / 8 - 256;
    if (RES)
      room -= (long long)cnt * (4 * (int)sizeof(V) + (OP == kMixed ? 32 : 0)) +
              (long long)(last - first) * (2 + (OP == kCsr ? 8 : OP == kMixed ? 16 : 32));
    else
      room -= (long long)stage_bytes * (kStages * kWarpsT);
    const int cap = (int)max(0LL, min((long long)min(kHash / 2, 65535 - min(cnt, 65535)), room / ((int)sizeof(V) + 4)));
    int* keys = reinterpret_cast<int*>(dyn + a.smem) - kHash;
    unsigned short* slot = reinterpret_cast<unsigned short*>(keys) - kHash;
    nh = cnt > 65535 || room < 0 ? -1 : build_halo<T>(gcol, first, last, a.n, n0, n1, cap, keys, slot, hid, sh);
    if (nh >= 0) {
      for (int j = threadIdx.x; j < nh; j += T) a.wanted[hid[j]] = 1;
      // (resident: straight to their place after the halo's list, which is below the hash set: 4 nh + 2 ne
      // bytes are at most 80 KB when all fits)
      unsigned short* c = RES ? reinterpret_cast<unsigned short*>(dyn + (((unsigned)nh * 4u + 15u) & ~15u)) - first : a.lcol;
      for (int e = first + (int)threadIdx.x; e < last; e += T) c[e] = local_slot(gcol[e], n0, n1, keys, slot);
      if (OP == kMixed && RES)
        for (int e = e0 + (int)threadIdx.x; e < e1; e += T)
          a.lcol[e] = local_slot(a.A64.bnbr[e], n0, n1, keys, slot);
    }
    asm volatile("fence.proxy.async;" ::: "memory");  // (bulk copies read lcol)
    double unfit[1] = {threadIdx.x == 0 && nh < 0 ? 1.0 : 0.0};
    if (!team_sum<1, true, CLUSTER, T>(a, sh, tag, unfit)) return;
    if (unfit[0] > 0.0) {
      if (blockIdx.x == 0 && threadIdx.x == 0) st->no_halo = 1;
      if constexpr (CLUSTER) cg::this_cluster().sync();
      return;
    }
  }

  // -- shared memory: halo list, p, row starts, wanted flags; the matrix or the rings; own vectors
  unsigned used = 0;
  auto take = [&](unsigned bytes) {
    unsigned char* at = dyn + used;
    used += (bytes + 15u) & ~15u;
    return at;
  };
  const int ne = last - first;
  take((unsigned)nh * 4u);
  const unsigned short* scol = nullptr;  // (indexed with the global entry number, like the values)
  if (RES) scol = reinterpret_cast<unsigned short*>(take(2u * (unsigned)ne)) - first;
  V* p = reinterpret_cast<V*>(take((unsigned)(cnt + nh) * (unsigned)sizeof(V)));
  int* sptr = reinterpret_cast<int*>(take((unsigned)(cnt + 1) * 4u));
  unsigned* want = reinterpret_cast<unsigned*>(take((unsigned)(cnt + 31) / 32 * 4u));  // a bit per node
  {
    // at entry (a start or a restart) the direction is D^-1 r
    const V *rg = reinterpret_cast<const V*>(a.r), *dg = reinterpret_cast<const V*>(a.invd);
    for (int j = threadIdx.x; j < cnt + nh; j += T) {
      const int m = j < cnt ? n0 + j : hid[j - cnt];
      p[j] = mul(dg[m], rg[m]);
    }
  }
  for (int i = threadIdx.x; i <= cnt; i += T) sptr[i] = cnt > 0 ? gptr[i] : 0;
  for (int i0 = warp * 32; i0 < cnt; i0 += T) {
    const unsigned m = __ballot_sync(kFull, i0 + lane < cnt && __ldcg(a.wanted + n0 + i0 + lane));
    if (lane == 0) want[i0 / 32] = m;
  }
  auto wanted = [&](int i) { return (want[i >> 5] >> (i & 31) & 1u) != 0; };
  __syncthreads();
  double2 *s64 = nullptr, *sS = nullptr;
  float4* s32 = nullptr;
  double* scv = nullptr;
  unsigned char* ring = nullptr;
  if constexpr (RES) {
    if constexpr (OP == kBlock64) {
      double2* v = reinterpret_cast<double2*>(take(32u * (unsigned)ne));
      const double2* g = reinterpret_cast<const double2*>(a.A64.vals) + 2L * e0;
      for (int i = threadIdx.x; i < 2 * ne; i += T) v[i] = __ldcs(g + i);
      s64 = v - 2L * e0;
    } else if constexpr (OP == kMixed) {
      float4* v = reinterpret_cast<float4*>(take(16u * (unsigned)ne));
      for (int i = threadIdx.x; i < ne; i += T) v[i] = __ldcs(a.A32.val32 + first + i);
      s32 = v - first;
      sS = reinterpret_cast<double2*>(take(32u * (unsigned)cnt));
      for (int i = threadIdx.x; i < 2 * cnt; i += T) sS[i] = __ldcs(a.A32.S64 + 2L * n0 + i);
    } else {
      double* v = reinterpret_cast<double*>(take(8u * (unsigned)ne));
      for (int i = threadIdx.x; i < ne; i += T) v[i] = __ldcs(a.csr.vals + e0 + i);
      scv = v - e0;
    }
  } else {
    ring = take(stage_bytes * (kStages * kWarpsT)) + (size_t)warp * kStages * stage_bytes;
  }
  auto own = [&](const double* g) {
    Own<V, RES> v;
    v.g = reinterpret_cast<V*>(const_cast<double*>(g)) + n0;
    v.lim = RES ? cnt : (int)min((unsigned)cnt, (a.smem - min(used, a.smem)) / (unsigned)sizeof(V));
    v.s = reinterpret_cast<V*>(take((unsigned)v.lim * (unsigned)sizeof(V)));
    return v;
  };
  const Own<V, RES> r = own(a.r), invd = own(a.invd), Ap = own(a.Ap), x = own(a.x);
  for (int i = threadIdx.x; i < cnt; i += T) {
    if (i < r.lim) r.s[i] = r.g[i];
    if (i < x.lim) x.s[i] = x.g[i];
    if (i < invd.lim) invd.s[i] = invd.g[i];
  }

  // -- the warp's ring: groups warp, warp + kWarpsT, ... over and over, kStages copies ahead. Copies are
  // marked evict-first: the matrix does not fit L2 and would push the vectors out of it.
  unsigned issued = 0, taken = 0;  // stages filled and consumed so far
  int next = warp;                 // the group of the next copy
  bool lost = false;               // a copy's wait ran out
  const uint32_t full0 = smem_addr(&sh.full[warp][0]);
  uint64_t policy = 0;
  auto issue = [&]() {  // one lane
    if constexpr (!RES) {
      const Group<OP> q(sptr, n0, cnt, next, kGroup);
      const unsigned k = issued % kStages;
      unsigned char* at = ring + (size_t)k * stage_bytes;
      const uint32_t vb = (uint32_t)q.ne * kEntryBytes<OP>, sb = OP == kMixed ? 32u * (uint32_t)(q.i1 - q.i0) : 0u;
      const uint32_t cb = ((uint32_t)(q.first + q.ne - q.slot0()) * 2u + 15u) & ~15u;
      const uint32_t bar = full0 + 8u * k;
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(vb + sb + cb) : "memory");
      const char* vals = OP == kMixed ? reinterpret_cast<const char*>(a.A32.val32) : reinterpret_cast<const char*>(a.A64.vals);
      bulk_copy(at, vals + (size_t)q.first * kEntryBytes<OP>, vb, bar, policy);
      if (OP == kMixed) bulk_copy(at + stage_S, a.A32.S64 + 2L * (n0 + q.i0), sb, bar, policy);
      bulk_copy(at + stage_col, a.lcol + q.slot0(), cb, bar, policy);
    }
  };
  auto advance = [&]() {
    ++issued;
    next = next + kWarpsT < groups ? next + kWarpsT : warp;
  };
  if constexpr (!RES) {
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
    if (lane == 0) {
      for (int k = 0; k < kStages; ++k)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(full0 + 8u * k), "r"(1));
      asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    asm volatile("fence.proxy.async;" ::: "memory");  // (the halo's hash set was written where the ring is)
    __syncthreads();
    for (int k = 0; k < kStages && warp < groups; ++k) {
      if (lane == 0) issue();
      advance();
    }
  }

  // -- scalars: the same in every thread of every block
  const double bnorm = __ldcg(&st->bnorm), rtol = __ldcg(&st->rtol), delta = __ldcg(&st->delta);
  const int max_iter = __ldcg(&st->max_iter), cycle_limit = __ldcg(&st->cycle_limit);
  const bool hist = __ldcg(&st->hist_on) != 0 && blockIdx.x == 0 && threadIdx.x == 0;
  double rz = __ldcg(&st->rz), rz_prev = 0.0, rel = __ldcg(&st->rel), rr = __ldcg(&st->rr), pAp = 0.0;
  double rmax = __ldcg(&st->rmax), alpha = 0.0, beta = 0.0;
  int it = __ldcg(&st->iter), done = 0;
  int last_replace = __ldcg(&st->last_replace), fp64_mode = OP == kMixed ? __ldcg(&st->fp64_mode) : 0;
  if (threadIdx.x == 0) {
    sh.rel.best_true = __ldcg(&st->best_true);
    sh.rel.true_rel = __ldcg(&st->true_rel);
    sh.rel.replaced = __ldcg(&st->replace_count);
    sh.rel.final_checks = __ldcg(&st->final_checks);
    sh.rel.switch_iter = __ldcg(&st->fp64_switch_iter);
    sh.rel.stall = __ldcg(&st->stall_cycles);
  }
  __syncthreads();

  unsigned zt = 0;  // tag of the z that the next phase 1 reads; z of iteration k is in buffer k & 1
  for (unsigned k = 1;; ++k) {
    // ---- phase 1: the step of x of the iteration before; p at own nodes and halo
    if (k > 1) {
      const ulonglong2* zr = a.z + (size_t)((k - 1) & 1u) * a.n * kZ;
      for (int j0 = cnt + (int)threadIdx.x; j0 < cnt + nh; j0 += kU * T) {
        V zj[kU];
        bool got[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          const int j = j0 + u * T;
          got[u] = j >= cnt + nh || ld_z(zr, hid[j - cnt], zt, zj[u]);
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          const int j = j0 + u * T;
          if (j >= cnt + nh) break;
          if (!got[u] && !CLUSTER) {  // (the cluster's barrier has made it visible)
            long long spins = 0;
            while (!ld_z(zr, hid[j - cnt], zt, zj[u]))
              if (!poll_again(a, spins)) {
                sh.ok = 0;
                give_up(a);
                break;
              }
          }
          p[j] = axpy(beta, p[j], zj[u]);
        }
      }
      for (int i0 = threadIdx.x; i0 < cnt; i0 += kU * T) {
        V xi[kU], zi[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          const int i = min(i0 + u * T, cnt - 1);
          xi[u] = x[i];
          zi[u] = mul(invd[i], r[i]);
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          const int i = i0 + u * T;
          if (i >= cnt) break;
          const V pi = p[i];
          x[i] = axpy(alpha, pi, xi[u]);
          p[i] = axpy(beta, pi, zi[u]);
        }
      }
      __syncthreads();
    }
    double d[1] = {0.0};
    for (int g = warp; g < groups; g += kWarpsT) {
      const int i = g * kGroup + lane / L;
      const bool ok = i < cnt;
      const V pn = ok ? p[i] : vzero(V());
      V y;
      if constexpr (!RES) {
        const unsigned slot = taken % kStages;
        const bool got = !lost && stage_wait(full0 + 8u * slot, (taken / kStages) & 1u, a.spin_limit);
        if (!__all_sync(kFull, got)) {  // (nothing of the stage may be read: leave at the next reduction)
          lost = true;
          sh.ok = 0;
          give_up(a);
          continue;
        }
        const Group<OP> q(sptr, n0, cnt, g, kGroup);
        const unsigned char* at = ring + (size_t)slot * stage_bytes;
        const unsigned short* c = reinterpret_cast<const unsigned short*>(at + stage_col) - q.slot0();
        if constexpr (OP == kBlock64)
          y = row_block64<L>(sptr, c, reinterpret_cast<const double2*>(at) - 2L * q.first, i, ok, p);
        else
          y = row_mixed<L>(sptr, n0, c, reinterpret_cast<const float4*>(at) - q.first,
                           reinterpret_cast<const double2*>(at + stage_S) - 2L * q.i0, i, ok, p, pn);
        __syncwarp();  // every lane has read the stage
        if (lane == 0) issue();
        advance();
        ++taken;
      } else if constexpr (OP == kBlock64) {
        y = row_block64<L>(sptr, scol, s64, i, ok, p);
      } else if constexpr (OP == kMixed) {
        y = fp64_mode ? row_block64_call<L>(gptr, a.lcol, reinterpret_cast<const double2*>(a.A64.vals), i, ok, p)
                      : row_mixed<L>(sptr, n0, scol, s32, sS, i, ok, p, pn);
      } else {
        y = row_csr<L>(sptr, scol, scv, i, ok, p);
      }
      if (ok && (lane & (L - 1)) == 0) {
        Ap[i] = y;
        d[0] = dot(pn, y, d[0]);
      }
    }
    if (!team_sum<1, false, CLUSTER, T>(a, sh, tag, d)) break;
    pAp = d[0];
    if (!(pAp > 0.0)) {
      alpha = 0.0;
      done = CSTG_SOLVE_BREAKDOWN + 1;
      break;
    }
    alpha = rz / pAp;

    // ---- phase 2
    ulonglong2* zw = a.z + (size_t)(k & 1u) * a.n * kZ;
    zt = 2u * k;
    double v[2] = {0.0, 0.0};
    for (int i0 = threadIdx.x; i0 < cnt; i0 += kU * T) {
      V ri[kU], di[kU];
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int i = min(i0 + u * T, cnt - 1);
        ri[u] = axpy(-alpha, Ap[i], r[i]);
        di[u] = invd[i];
      }
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int i = i0 + u * T;
        if (i >= cnt) break;
        const V zi = mul(di[u], ri[u]);
        if (wanted(i)) st_z(zw, n0 + i, zi, zt);
        r[i] = ri[u];
        v[0] = dot(ri[u], ri[u], v[0]);
        v[1] = dot(ri[u], zi, v[1]);
      }
    }
    if (!team_sum<2, false, CLUSTER, T>(a, sh, tag, v)) break;
    ++it;
    const double rn = sqrt(v[0]);
    rel = rn / bnorm;
    rr = v[0];
    if (hist) a.history[it] = rel;
    int pending = 0;
    if (OP != kMixed) {
      if (rel < rtol)
        done = CSTG_SOLVE_CONVERGED + 1;
      else if (it >= max_iter)
        done = CSTG_SOLVE_MAX_ITER + 1;
    } else {
      rmax = fmax(rmax, rn);
      if (rel < rtol)
        pending = 2;
      else if (!fp64_mode && rn < delta * rmax)
        pending = 1;
      else if (!fp64_mode && it - last_replace >= cycle_limit)
        pending = 3;  // (plain FP64 CG after the switch, as in mixed_kernels.cu)
      else if (it >= max_iter)
        done = CSTG_SOLVE_MAX_ITER + 1;
    }
    rz_prev = rz;
    beta = v[1] / rz;
    rz = v[1];
    if (done) break;

    // ---- R (mixed): reliable update with the FP64 residual
    if constexpr (OP == kMixed) {
      if (pending) {
        for (int i = threadIdx.x; i < cnt; i += T) {
          const V xi = axpy(alpha, p[i], x[i]);
          x[i] = xi;
          __stcg(x.g + i, xi);
        }
        alpha = 0.0;  // (x is up to date)
        double none[1] = {0.0};
        if (!team_sum<1, true, CLUSTER, T>(a, sh, tag, none)) break;
        zt = 2u * k + 1u;
        double q[2] = {0.0, 0.0};
        for (int g = warp; g < groups; g += kWarpsT) {
          const int i = g * kGroup + lane / L;
          const bool ok = i < cnt;
          const V y = row_block64_call<L>(gptr, a.A64.bnbr, reinterpret_cast<const double2*>(a.A64.vals), i, ok,
                                          reinterpret_cast<const V*>(a.x));
          if (ok && (lane & (L - 1)) == 0) {
            const V ri = sub(reinterpret_cast<const V*>(a.b)[n0 + i], y);
            const V zi = mul(invd[i], ri);
            if (wanted(i)) st_z(zw, n0 + i, zi, zt);
            r[i] = ri;
            q[0] = dot(ri, ri, q[0]);
            q[1] = dot(ri, zi, q[1]);
          }
        }
        if (!team_sum<2, false, CLUSTER, T>(a, sh, tag, q)) break;
        const double tn = sqrt(q[0]), tr = tn / bnorm;
        const double rec = rel;  // the recursive residual this replacement corrects
        Reliable m = sh.rel;
        __syncthreads();
        m.true_rel = tr;
        m.replaced += 1;
        rel = tr;
        rr = q[0];
        rmax = tn;
        last_replace = it;
        if (hist) a.history[it] = tr;
        beta = rz_prev > 0.0 ? q[1] / rz_prev : 0.0;
        rz = q[1];
        if (tr < rtol) {
          done = CSTG_SOLVE_CONVERGED + 1;
        } else {
          // (the precision switch of mixed_kernels.cu's k_replace_mixed, same rule)
          if (pending == 3)
            m.stall =
                ((tr > 0.9 * m.best_true || tr > kGapRatio * rec) && m.best_true < kStallGate) ? m.stall + 1 : 0;
          if (!fp64_mode &&
              (pending == 2 || (pending == 1 && tr > 0.5 * m.best_true) || (pending == 3 && m.stall >= 2))) {
            fp64_mode = 1;
            m.switch_iter = it;
            beta = 0.0;
          } else if (fp64_mode) {
            beta = 0.0;
          }
          if (pending == 2 && ++m.final_checks > a.max_final_checks) done = CSTG_SOLVE_CONVERGED + 1;
          if (it >= max_iter) done = CSTG_SOLVE_MAX_ITER + 1;
        }
        m.best_true = fmin(m.best_true, tr);
        if (threadIdx.x == 0) sh.rel = m;
        if (done || (!RES && fp64_mode)) break;
      }
    }
  }

  // ---- end: copies in flight land (bounded), the last step of x, the state. A streamed mixed solve
  // that switched precision (done = 0) leaves its iteration to the grid kernel: r and the
  // next direction go back to global memory.
  if (!RES && lane == 0)
    for (; taken != issued; ++taken)
      stage_wait(full0 + 8u * (taken % kStages), (taken / kStages) & 1u, kBarrierSpinDefault);
  if (sh.ok) {
    for (int i = threadIdx.x; i < cnt; i += T) {
      x.g[i] = alpha != 0.0 ? axpy(alpha, p[i], x[i]) : x[i];
      if (OP == kMixed && !RES && !done) {
        const V ri = r[i];
        r.g[i] = ri;
        reinterpret_cast<V*>(a.p)[n0 + i] = axpy(beta, p[i], mul(invd[i], ri));
      }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      st->rz = rz;
      st->rz_prev = rz_prev;
      st->alpha = alpha;
      st->beta = beta;
      st->rel = rel;
      st->rr = rr;
      st->pAp = pAp;
      st->iter = it;
      if (OP == kMixed) {
        st->rmax = rmax;
        st->last_replace = last_replace;
        st->fp64_mode = fp64_mode;
        st->best_true = sh.rel.best_true;
        st->true_rel = sh.rel.true_rel;
        st->replace_count = sh.rel.replaced;
        st->final_checks = sh.rel.final_checks;
        st->fp64_switch_iter = sh.rel.switch_iter;
        st->stall_cycles = sh.rel.stall;
      }
      atomicCAS(&st->done, 0, done);  // (a block that timed out in the last wait has set it)
    }
  }
  if constexpr (CLUSTER) cg::this_cluster().sync();  // no block leaves while another may write its inbox
}

template <int OP, bool CLUSTER, bool RES, int L, int T>
cudaError_t launch_team(SolveArgs& a, int blocks, cudaStream_t s) {
  auto kern = k_pcg_persistent<OP, CLUSTER, RES, L, T>;
  // all of the shared memory that a block may have
  int dev = 0, most = 0;
  cudaGetDevice(&dev);
  cudaError_t e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e != cudaSuccess) return e;
  a.smem = (unsigned)(most - (int)sizeof(Shared<T>)) / 1024u * 1024u;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)a.smem);
  if (e == cudaSuccess && CLUSTER && blocks > 8)
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  if (CLUSTER) {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)blocks;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
  } else {
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
  }
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3(T);
  cfg.dynamicSmemBytes = a.smem;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (CLUSTER) {  // (a cooperative launch that does not fit is refused by itself)
    int room = 0;
    e = cudaOccupancyMaxActiveClusters(&room, kern, &cfg);
    if (e != cudaSuccess) return e;
    if (room < 1) return cudaErrorInvalidClusterSize;
  }
  e = cudaLaunchKernelEx(&cfg, kern, a);
  if (e == cudaSuccess) count_launches(1);
  return e;
}

// Blocks of a grid team: one per SM, but at least 64 nodes (rows) each, so that small systems wait for
// fewer partners.
int team_blocks(int n) {
  int dev = 0, sms = kSMs;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return std::min(std::min(sms, kMaxTeam), std::max(1, (n + 63) / 64));
}

template <int OP>
cudaError_t launch_op(SolveArgs& a, PcgTeam team, cudaStream_t s) {
  const int blocks = team_blocks(a.n);
  // Lanes per node: one, or two where a block's nodes outnumber its threads and FP64 rows (or CSR
  // rows) read enough shared memory for the split to pay (180 x 360 plate, FP64: 8.5 against 8.3 us
  // an iteration; mixed: 6.9 against 7.6, so never there).
  const bool two = OP != kMixed && a.n > 256 * (team == PcgTeam::kCluster ? kClusterTeam : blocks);
  switch (team) {
    case PcgTeam::kCluster:
      return two ? launch_team<OP, true, true, 2, 256>(a, kClusterTeam, s)
                 : launch_team<OP, true, true, 1, 256>(a, kClusterTeam, s);
    case PcgTeam::kResident:
      return two ? launch_team<OP, false, true, 2, 256>(a, blocks, s)
                 : launch_team<OP, false, true, 1, 256>(a, blocks, s);
    case PcgTeam::kStream:
      if constexpr (OP == kBlock64) return launch_team<OP, false, false, 2, 384>(a, blocks, s);
      if constexpr (OP == kMixed) return launch_team<OP, false, false, 1, 384>(a, blocks, s);
      break;
    case PcgTeam::kStreamNarrow:
      if constexpr (OP == kBlock64) return launch_team<OP, false, false, 2, 256>(a, blocks, s);
      if constexpr (OP == kMixed) return launch_team<OP, false, false, 2, 384>(a, blocks, s);
      break;
    default: break;
  }
  return cudaErrorInvalidValue;
}

}  // namespace

size_t pcg_persistent_work(int n) {
  return 32 * (size_t)n + (size_t)n + 256 + sizeof(ulonglong2) * 4 * kCopies * kMaxTeam;
}

// The first team whose shared memory holds a system of n nodes (rows) with `entries` matrix blocks
// (entries) in all, by the average block and without its halo: the kernel checks what it finds and
// declines (PcgState::no_halo), and the caller goes on with the next team.
PcgTeam pcg_persistent_team(int n, long long entries, bool mixed, bool csr, bool small_ok, PcgTeam after) {
  int dev = 0, most = 0;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return PcgTeam::kNone;
  const double room = most - 4096.0;
  const double v = csr ? 8.0 : 16.0, e = csr ? 10.0 : mixed ? 18.0 : 34.0, s = mixed ? 32.0 : 0.0;
  const double per = n > 0 ? (double)entries / n - (mixed ? 1.0 : 0.0) : 0.0;  // entries of a row
  const auto resident = [&](int blocks) { return (double)n / blocks * (5.0 * v + 4.125 + s + per * e) < room; };
  const auto stream = [&](int rows, int warps) {
    return !csr && (double)n / team_blocks(n) * (v + 4.125) + 2.0 * warps * rows * (per * e + s) < room;
  };
  const auto fits = [&](PcgTeam t) {
    switch (t) {
      // A cluster's barrier is hardware (1.0 us a reduction against 1.5 to 2.5 us of a grid team), but it
      // has 16 SMs: at 3,321 nodes 3.9 against 4.7 us an iteration, at 15,006 CSR rows 6.4 both.
      case PcgTeam::kCluster: return small_ok && n <= (csr ? 12000 : 6000) && resident(kClusterTeam);
      case PcgTeam::kResident: return resident(team_blocks(n));
      case PcgTeam::kStream: return stream(mixed ? 32 : 16, 12);
      case PcgTeam::kStreamNarrow: return stream(16, mixed ? 12 : 8);
      case PcgTeam::kGrid: return !csr;
      default: return true;
    }
  };
  for (int t = (int)after + 1; t < (int)PcgTeam::kNone; ++t)
    if (fits((PcgTeam)t)) return (PcgTeam)t;
  return PcgTeam::kNone;
}

cudaError_t launch_pcg_persistent(PcgTeam team, const PcgBuffers& w, const BlockMatrix* A64, const MixedMatrix* A32,
                                  const CsrMatrixDev* csr, void* work, unsigned short* slots, int max_final_checks,
                                  long long spin_limit, cudaStream_t s) {
  if (team == PcgTeam::kGrid) return launch_pcg_grid(w, *A64, A32, max_final_checks, spin_limit, s);
  SolveArgs a;
  const size_t n = (size_t)w.n;
  a.n = csr ? w.n : w.n / 2;
  if (A64) a.A64 = *A64;
  if (A32) a.A32 = *A32;
  if (csr) a.csr = *csr;
  a.x = w.x;
  a.r = w.r;
  a.Ap = w.Ap;
  a.p = w.p;
  // work: z, wanted, sums, all zero at launch (tags start at 1)
  const size_t zb = 32 * n, wb = ((size_t)a.n + 255) & ~(size_t)255, sb = sizeof(ulonglong2) * 4 * kCopies * kMaxTeam;
  unsigned char* wk = static_cast<unsigned char*>(work);
  a.z = reinterpret_cast<ulonglong2*>(wk);
  a.wanted = wk + zb;
  a.sums = reinterpret_cast<ulonglong2*>(wk + zb + wb);
  a.lcol = slots;
  a.invd = w.inv_diag;
  a.b = w.b;
  a.history = w.history;
  a.st = w.st;
  a.max_final_checks = max_final_checks;
  a.spin_limit = spin_limit;
  cudaError_t e = cudaMemsetAsync(work, 0, zb + wb + sb, s);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(&w.st->no_halo, 0, 2 * sizeof(int), s);  // (and bar_err)
  if (e != cudaSuccess) return e;
  return csr ? launch_op<kCsr>(a, team, s) : A32 ? launch_op<kMixed>(a, team, s) : launch_op<kBlock64>(a, team, s);
}

}  // namespace cstg
