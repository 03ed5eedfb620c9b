// Smoothed-aggregation algebraic multigrid (a preconditioner for the same Jacobi-PCG path; no
// reference counterpart). Setup and V-cycle kernels; host orchestration in amg_api.cu.
//
// Levels hold block-sparse matrices (BSR, row-major B x B blocks, B = 2 on the finest level,
// 3 = the rigid-body modes on coarser levels) and a near-nullspace basis per node (B x 3: the
// 2D rigid-body modes on the finest level). One coarsening step:
//   1. aggregation: roots = a distance-2 maximal independent set of the block graph (Luby rounds
//      with fixed hash priorities), aggregate = root + its neighbours, leftovers join the
//      aggregated neighbour with the strongest block (Frobenius norm), isolated leftovers become
//      singletons;
//   2. tentative prolongator: per aggregate, Gram-Schmidt QR of the stacked nullspace blocks:
//      P0 = Q (one B x 3 block per node), coarse nullspace = R;
//   3. smoothed prolongator P = (I - w D^-1 A) P0, w = 4 / (3 lambda_max(D^-1 A));
//   4. Galerkin coarse operator A_c = P' (A P) (3 x 3 blocks).
// Every kernel adds in a fixed order (thread-per-row kernels, or warp-per-row kernels whose lanes
// own output blocks): the hierarchy and the cycle are deterministic. Rows are built in two passes
// (count, then fill after a prefix sum); row widths are bounded by kAmgMaxRow (checked: the error
// word records the first overflow).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <mutex>
#include <utility>
#include <vector>

#include "common.cuh"
#include "kernels.h"

namespace cstg {

namespace cg = cooperative_groups;

namespace {

constexpr int kU = 0, kRoot = 1, kOut = 2;  // aggregation states

__device__ __forceinline__ unsigned long long node_key(int i) {
  unsigned long long h = (unsigned long long)(unsigned)i * 0x9E3779B97F4A7C15ull;
  h ^= h >> 29;
  h *= 0xBF58476D1CE4E5B9ull;
  h ^= h >> 32;
  return (h & 0xFFFFFFFF00000000ull) | (unsigned)i;  // unique: low bits are the index
}

// sorted small set insert; returns position or -1 on overflow
__device__ __forceinline__ int set_insert(int* s, int& n, int v, int cap) {
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (s[mid] < v)
      lo = mid + 1;
    else
      hi = mid;
  }
  if (lo < n && s[lo] == v) return lo;
  if (n >= cap) return -1;
  for (int k = n; k > lo; --k) s[k] = s[k - 1];
  s[lo] = v;
  ++n;
  return lo;
}

__device__ __forceinline__ int row_find(const int* cols, int lo, int hi, int v) {
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (cols[mid] < v)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

// ---- fine-level conversion: the node-run layout -> BSR 2x2 --------------------------------------

// Eight lanes per node, 16 bytes each, so that reads and writes are runs (a thread per node: 122 us for
// 1,003,302 DOFs; 39 so).
__global__ void k_amg_bsr2(int N, const int* __restrict__ node_ptr, const double* __restrict__ vals,
                           double* __restrict__ out) {
  const int n = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 3);
  if (n >= N) return;
  const int b0 = node_ptr[n], deg = node_ptr[n + 1] - b0;
  const double2* in = reinterpret_cast<const double2*>(vals) + 2 * (size_t)b0;
  double2* o = reinterpret_cast<double2*>(out) + 2 * (size_t)b0;
  for (int u = threadIdx.x & 7; u < 2 * deg; u += 8) o[u] = in[(u & 1) * deg + (u >> 1)];
}

template <int B>
__global__ void k_amg_dinv(int n, AmgBsr A, double* __restrict__ dinv, int* err) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int k = row_find(A.col, A.ptr[i], A.ptr[i + 1], i);
  if (k >= A.ptr[i + 1] || A.col[k] != i) {
    atomicMin(&err[kErrDiag], i);
    return;
  }
  const double* blk = A.val + (size_t)k * B * B;
  for (int c = 0; c < B; ++c) {
    const double d = blk[c * B + c];
    if (!(d > 0.0)) atomicMin(&err[kErrDiag], i);
    dinv[(size_t)i * B + c] = d > 0.0 ? 1.0 / d : 0.0;
  }
}

// ---- aggregation ----------------------------------------------------------------------------------

// Strength of connection (the graph the aggregation walks): block (i, j) is strong when
// ||A_ij||_F >= theta sqrt(||A_ii||_F ||A_jj||_F); diagonal blocks always are. strong == nullptr
// (theta 0) keeps every block of the pattern.
template <int B>
__global__ void k_amg_diag_norm(int n, AmgBsr A, double* __restrict__ dn) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double s = 0.0;
  for (int k = A.ptr[i]; k < A.ptr[i + 1]; ++k)
    if (A.col[k] == i) {
      const double* blk = A.val + (size_t)k * B * B;
      for (int q = 0; q < B * B; ++q) s += blk[q] * blk[q];
    }
  dn[i] = sqrt(s);
}

template <int B>
__global__ void k_amg_strength(int n, AmgBsr A, const double* __restrict__ dn, double theta,
                               unsigned char* __restrict__ strong) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double t2 = theta * theta * dn[i];
  for (int k = A.ptr[i]; k < A.ptr[i + 1]; ++k) {
    const int j = A.col[k];
    const double* blk = A.val + (size_t)k * B * B;
    double s = 0.0;
    for (int q = 0; q < B * B; ++q) s += blk[q] * blk[q];
    strong[k] = (j == i || s >= t2 * dn[j]) ? 1 : 0;
  }
}

__device__ __forceinline__ bool is_strong(const unsigned char* strong, int k) { return !strong || strong[k]; }

__global__ void k_mis_m1(int n, AmgBsr A, const unsigned char* __restrict__ strong, const int* __restrict__ state,
                         unsigned long long* __restrict__ m1) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  unsigned long long m = 0;
  for (int k = A.ptr[i]; k < A.ptr[i + 1]; ++k) {
    const int j = A.col[k];
    if (is_strong(strong, k) && state[j] == kU) m = max(m, node_key(j) + 1);
  }
  m1[i] = m;
}

__global__ void k_mis_root(int n, AmgBsr A, const unsigned char* __restrict__ strong, int* __restrict__ state,
                           const unsigned long long* __restrict__ m1, int* __restrict__ newroot) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  newroot[i] = 0;
  if (state[i] != kU) return;
  unsigned long long m = 0;
  for (int k = A.ptr[i]; k < A.ptr[i + 1]; ++k)
    if (is_strong(strong, k)) m = max(m, m1[A.col[k]]);
  if (m == node_key(i) + 1) newroot[i] = 1;
}

// near[i] = 1 if a new root is in N(i) (incl. i)
__global__ void k_mis_near(int n, AmgBsr A, const unsigned char* __restrict__ strong,
                           const int* __restrict__ newroot, int* __restrict__ near) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int f = 0;
  for (int k = A.ptr[i]; k < A.ptr[i + 1] && !f; ++k) f = is_strong(strong, k) && newroot[A.col[k]];
  near[i] = f;
}

__global__ void k_mis_out(int n, AmgBsr A, const unsigned char* __restrict__ strong, int* __restrict__ state,
                          const int* __restrict__ newroot, const int* __restrict__ near, int* __restrict__ undecided) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (newroot[i]) {
    state[i] = kRoot;
    return;
  }
  if (state[i] != kU) return;
  int f = 0;
  for (int k = A.ptr[i]; k < A.ptr[i + 1] && !f; ++k) f = is_strong(strong, k) && near[A.col[k]];
  if (f)
    state[i] = kOut;
  else
    atomicAdd(undecided, 1);
}

// phase 1: roots (ids from the prefix sum of root flags) and their strong neighbours
__global__ void k_agg_phase1(int n, AmgBsr A, const unsigned char* __restrict__ strong,
                             const int* __restrict__ state, const int* __restrict__ root_id, int* __restrict__ agg) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int a = -1;
  if (state[i] == kRoot) {
    a = root_id[i];
  } else {
    for (int k = A.ptr[i]; k < A.ptr[i + 1]; ++k) {
      const int j = A.col[k];
      if (is_strong(strong, k) && state[j] == kRoot) {
        a = root_id[j];
        break;
      }
    }
  }
  agg[i] = a;
}

// phase 2: join the aggregated neighbour (phase-1 assignment) with the strongest block
template <int B>
__global__ void k_agg_phase2(int n, AmgBsr A, const int* __restrict__ agg1, int* __restrict__ agg2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int a = agg1[i];
  if (a < 0) {
    double best = -1.0;
    for (int k = A.ptr[i]; k < A.ptr[i + 1]; ++k) {
      const int j = A.col[k];
      if (j == i || agg1[j] < 0) continue;
      const double* blk = A.val + (size_t)k * B * B;
      double s = 0.0;
      for (int q = 0; q < B * B; ++q) s += blk[q] * blk[q];
      if (s > best) {
        best = s;
        a = agg1[j];
      }
    }
  }
  agg2[i] = a;
}

// phase 3: leftovers become singleton aggregates numbered after the others
__global__ void k_agg_phase3(int n, int n_agg, const int* __restrict__ left_id, int* __restrict__ agg) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (agg[i] < 0) agg[i] = n_agg + left_id[i];
}

__global__ void k_flag_negative(int n, const int* __restrict__ a, int* __restrict__ f) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) f[i] = a[i] < 0 ? 1 : 0;
}

__global__ void k_flag_eq(int n, const int* __restrict__ a, int v, int* __restrict__ f) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) f[i] = a[i] == v ? 1 : 0;
}

// members of each aggregate (count / fill / sort by node)
__global__ void k_count_by(int n, const int* __restrict__ key, int* __restrict__ cnt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) atomicAdd(&cnt[key[i]], 1);
}

__global__ void k_fill_by(int n, const int* __restrict__ key, const int* __restrict__ ptr, int* __restrict__ cur,
                          int* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[ptr[key[i]] + atomicAdd(&cur[key[i]], 1)] = i;
}

__global__ void k_sort_segments(int m, const int* __restrict__ ptr, int* __restrict__ v) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= m) return;
  for (int i = ptr[s] + 1; i < ptr[s + 1]; ++i) {
    const int x = v[i];
    int j = i - 1;
    while (j >= ptr[s] && v[j] > x) {
      v[j + 1] = v[j];
      --j;
    }
    v[j + 1] = x;
  }
}

// ---- tentative prolongator: per aggregate, QR (modified Gram-Schmidt) of the stacked B x 3 blocks ----

// Eight lanes per aggregate, its stacked blocks in shared memory: the lanes take the rows' updates, and
// each lane runs the sums over the rows (in order) for itself. A chain of dependent FP64 operations per
// aggregate bounds it (a thread per aggregate in global memory: 306 us for 48,233 aggregates of ten
// nodes; the coarse levels, with few aggregates, 80 to 95 us; 74 and 18 so).
constexpr int kTentLanes = 8, kTentWarps = 2;

template <int B>
__global__ void __launch_bounds__(32 * kTentWarps) k_amg_tentative(int n_agg, const int* __restrict__ agg_ptr,
                                                                   const int* __restrict__ members,
                                                                   const double* __restrict__ Bf,
                                                                   double* __restrict__ P0, double* __restrict__ Bc,
                                                                   int* err) {
  constexpr int kGroups = 32 * kTentWarps / kTentLanes;
  __shared__ double sm[kGroups][kAmgMaxAgg * B * 3];  // Q in place: row r of the stacked matrix at 3 r
  const int g = threadIdx.x / kTentLanes, l = threadIdx.x % kTentLanes;
  const unsigned mask = 0xffu << ((threadIdx.x & 31) / kTentLanes * kTentLanes);
  const int a = blockIdx.x * kGroups + g;
  if (a >= n_agg) return;  // (uniform over a group; groups synchronise alone)
  const int lo = agg_ptr[a], hi = agg_ptr[a + 1], m = hi - lo;
  if (m > kAmgMaxAgg) {
    if (l == 0) atomicMin(&err[kErrAmg], a);
    return;
  }
  const int rows = m * B;
  double* q = sm[g];
  double scale = 0.0;
  for (int e = l; e < rows * 3; e += kTentLanes) {
    const double v = Bf[(size_t)members[lo + e / (B * 3)] * B * 3 + e % (B * 3)];
    q[e] = v;
    scale = fmax(scale, fabs(v));
  }
#pragma unroll
  for (int o = kTentLanes / 2; o > 0; o >>= 1) scale = fmax(scale, __shfl_xor_sync(mask, scale, o));
  __syncwarp(mask);
  double R[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
#pragma unroll
    for (int p = 0; p < c; ++p) {
      double d = 0.0;
      for (int r = 0; r < rows; ++r) d = fma(q[3 * r + p], q[3 * r + c], d);
      R[p * 3 + c] = d;
      __syncwarp(mask);
      for (int r = l; r < rows; r += kTentLanes) q[3 * r + c] = fma(-d, q[3 * r + p], q[3 * r + c]);
      __syncwarp(mask);
    }
    double nrm = 0.0;
    for (int r = 0; r < rows; ++r) nrm = fma(q[3 * r + c], q[3 * r + c], nrm);
    nrm = sqrt(nrm);
    const bool drop = nrm <= 1e-10 * (scale > 0.0 ? scale : 1.0);  // dependent column (tiny aggregate)
    R[c * 3 + c] = drop ? 0.0 : nrm;
    __syncwarp(mask);
    for (int r = l; r < rows; r += kTentLanes) q[3 * r + c] = drop ? 0.0 : q[3 * r + c] / nrm;
    __syncwarp(mask);
  }
  for (int e = l; e < rows * 3; e += kTentLanes)
    P0[(size_t)members[lo + e / (B * 3)] * B * 3 + e % (B * 3)] = q[e];
  for (int k = l; k < 9; k += kTentLanes) {
    double v = R[0];
#pragma unroll
    for (int u = 1; u < 9; ++u) v = k == u ? R[u] : v;
    Bc[(size_t)a * 9 + k] = v;
  }
}

// ---- lambda_max(D^-1 A) by power iteration ----------------------------------------------------------
// Each step y = s D^-1 A x with s = 1 / ||x|| from the previous step (1 on the first) writes
// per-block partial sums of ||y||^2 on a fixed grid (k_amg_dinva_fine / _coarse, after the cycle
// kernels); the last block by ticket adds them in block order (a launch of its own took 3 us a step).
constexpr int kLamGrid = 148 * 8;

// t: the block's sum (thread 0). The last block: lam = sqrt(sum of the partials), sc = 1 / lam.
__device__ __forceinline__ void amg_norm_epilogue(double t, double* part, double* lam, double* sc, unsigned* ticket,
                                                  double* sm) {
  __shared__ bool am_last;
  if (threadIdx.x == 0) {
    part[blockIdx.x] = t;
    __threadfence();
    am_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!am_last) return;
  __threadfence();
  double s = 0.0;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) s += __ldcg(&part[b]);
  const double sum = block_sum<kThreads>(s, sm);
  if (threadIdx.x == 0) {
    const double nrm = sqrt(sum);
    *lam = nrm;
    *sc = nrm > 0.0 ? 1.0 / nrm : 0.0;
    *ticket = 0u;
  }
}

__global__ void k_amg_init_vec(int n, double* __restrict__ x) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    x[i] = 1.0 + 0.5 * (double)((node_key(i) >> 40) & 0xff) / 255.0;
}

// ---- smoothed prolongator P = P0 - w D^-1 A P0 --------------------------------------------------------

template <int B>
__global__ void k_amg_p_count(int n, AmgBsr A, const int* __restrict__ agg, int* __restrict__ cnt, int* err) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int s[kAmgMaxRow];
  int m = 0;
  for (int k = A.ptr[i]; k < A.ptr[i + 1]; ++k)
    if (set_insert(s, m, agg[A.col[k]], kAmgMaxRow) < 0) {
      atomicMin(&err[kErrAmg], i);
      break;
    }
  if (set_insert(s, m, agg[i], kAmgMaxRow) < 0) atomicMin(&err[kErrAmg], i);
  cnt[i] = m;
}

// P's column sets (sorted aggregates of the row's neighbours, the node's own included)
template <int B>
__global__ void k_amg_p_cols(int n, AmgBsr A, const int* __restrict__ agg, AmgBsr P) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int s[kAmgMaxRow];
  int m = 0;
  for (int k = A.ptr[i]; k < A.ptr[i + 1]; ++k) set_insert(s, m, agg[A.col[k]], kAmgMaxRow);
  set_insert(s, m, agg[i], kAmgMaxRow);
  int* cols = const_cast<int*>(P.col) + P.ptr[i];
  for (int q = 0; q < m; ++q) cols[q] = s[q];
}

// ---- AP = A P (rows: B x 3 blocks) --------------------------------------------------------------------

template <int B>
__global__ void k_amg_ap_count(int n, AmgBsr A, AmgBsr P, int* __restrict__ cnt, int* err) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int s[kAmgMaxRow];
  int m = 0;
  bool over = false;
  for (int k = A.ptr[i]; k < A.ptr[i + 1] && !over; ++k) {
    const int j = A.col[k];
    for (int q = P.ptr[j]; q < P.ptr[j + 1]; ++q)
      if (set_insert(s, m, P.col[q], kAmgMaxRow) < 0) {
        over = true;
        break;
      }
  }
  if (over) atomicMin(&err[kErrAmg], i);
  cnt[i] = m;
}

// The fill of a Galerkin factor runs in two kernels: one writes the rows' sorted column sets (as the
// count kernel found them), then G lanes per row sum the row's block products. Each lane owns the output
// blocks lane, lane + G, ... (a pass per G blocks) and goes through the row's candidate products (one per
// pair of input blocks) in their fixed order, computing those that fall on its block: every output block
// sees the same additions in the same order on every run, and nothing goes through shared memory (a warp
// per row that left the products there for their owners took 719 us for AP, 561 for P and 317 for A_c of
// 1,003,302 DOFs, most lanes idle in the additions; these take 204, 100 and 197). Latency of the chain of
// indices bounds them; G fits the rows' usual number of output blocks.
constexpr int kGalWarps = 8;

// The largest value over the warp.
__device__ __forceinline__ int warp_max(int v) { return __reduce_max_sync(0xffffffffu, v); }

// Prolongator smoothing weight w = kProlongOmega / lambda_max(D^-1 A). 1.6 rather than the usual
// 4/3: on the plates it gives 3-4 % fewer cycle iterations and slightly smaller coarse levels.
constexpr double kProlongOmega = 1.6;

// P = P0 - w D^-1 A P0: values, warp per row i. Candidates: the blocks k of A's row i in order,
// each the B x 3 product -w D_i^-1 A_k P0_{A.col[k]}; then P0_i is added to the node's own
// aggregate's block.
template <int B, int G>
__global__ void __launch_bounds__(32 * kGalWarps) k_amg_p_vals(int n, AmgBsr A, const int* __restrict__ agg,
                                                               const double* __restrict__ P0,
                                                               const double* __restrict__ dinv,
                                                               const double* __restrict__ wp, AmgBsr P) {
  constexpr int NV = B * 3, R = 32 / G;
  const int lane = threadIdx.x & 31, gl = lane % G;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  const double om = kProlongOmega / *wp;
  for (int base = warp * R; base < n; base += nw * R) {
    const int i = base + lane / G;
    const bool on = i < n;
    const int c0 = on ? P.ptr[i] : 0, m = on ? P.ptr[i + 1] - c0 : 0;
    const int k0 = on ? A.ptr[i] : 0, k1 = on ? A.ptr[i + 1] : 0;
    const int own = on ? agg[i] : -1;
    double f[B];
#pragma unroll
    for (int r = 0; r < B; ++r) f[r] = on ? -om * dinv[(size_t)i * B + r] : 0.0;
    const int passes = warp_max(m), span = warp_max(k1 - k0);
    for (int p = 0; p < passes; p += G) {
      const int mine = p + gl < m ? P.col[c0 + p + gl] : -1;
      double acc[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) acc[v] = 0.0;
      for (int kb = 0; kb < span; kb += G) {
        int j = 0, to = -2;  // the candidates' nodes and aggregates, one per lane
        if (k0 + kb + gl < k1) {
          j = A.col[k0 + kb + gl];
          to = agg[j];
        }
        const int us = min(G, span - kb);
        for (int u = 0; u < us; ++u) {
          const int ju = __shfl_sync(0xffffffffu, j, u, G);
          if (__shfl_sync(0xffffffffu, to, u, G) != mine) continue;
          const double* blk = A.val + (size_t)(k0 + kb + u) * B * B;
          const double* p0 = P0 + (size_t)ju * NV;
#pragma unroll
          for (int r = 0; r < B; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              double t = 0.0;
#pragma unroll
              for (int q = 0; q < B; ++q) t = fma(blk[r * B + q], p0[q * 3 + c], t);
              acc[r * 3 + c] = __dadd_rn(acc[r * 3 + c], __dmul_rn(f[r], t));
            }
        }
      }
      if (p + gl < m) {
        double* out = const_cast<double*>(P.val) + (size_t)(c0 + p + gl) * NV;
#pragma unroll
        for (int v = 0; v < NV; ++v) out[v] = own == mine ? acc[v] + P0[(size_t)i * NV + v] : acc[v];
      }
    }
  }
}

// AP = A P: column sets
template <int B>
__global__ void k_amg_ap_cols(int n, AmgBsr A, AmgBsr P, AmgBsr AP) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int s[kAmgMaxRow];
  int m = 0;
  for (int k = A.ptr[i]; k < A.ptr[i + 1]; ++k) {
    const int j = A.col[k];
    for (int q = P.ptr[j]; q < P.ptr[j + 1]; ++q) set_insert(s, m, P.col[q], kAmgMaxRow);
  }
  int* cols = const_cast<int*>(AP.col) + AP.ptr[i];
  for (int q = 0; q < m; ++q) cols[q] = s[q];
}

// The block of a sorted row (columns col[beg .. beg + len)) whose column is `mine`, or -1: the lanes of a
// group share the row and load its columns together.
template <int G>
__device__ __forceinline__ int gal_hit(const int* __restrict__ col, int beg, int len, int mine, int gl) {
  int hit = -1;
  const int most = warp_max(len);
  for (int x0 = 0; x0 < most; x0 += G) {
    const int c = x0 + gl < len ? col[beg + x0 + gl] : -2;
    const int xs = min(G, most - x0);
    for (int x = 0; x < xs; ++x)
      if (__shfl_sync(0xffffffffu, c, x, G) == mine) hit = beg + x0 + x;
  }
  return hit;
}

// AP = A P: values. Row i's candidates: for each block k of A's row i (ascending), for each block
// q of P's row A.col[k] (ascending), the B x 3 product A_k P_q.
template <int B, int G>
__global__ void __launch_bounds__(32 * kGalWarps) k_amg_ap_vals(int n, AmgBsr A, AmgBsr P, AmgBsr AP) {
  constexpr int NV = B * 3, R = 32 / G;
  const int lane = threadIdx.x & 31, gl = lane % G;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  for (int base = warp * R; base < n; base += nw * R) {
    const int i = base + lane / G;
    const bool on = i < n;
    const int c0 = on ? AP.ptr[i] : 0, m = on ? AP.ptr[i + 1] - c0 : 0;
    const int k0 = on ? A.ptr[i] : 0, k1 = on ? A.ptr[i + 1] : 0;
    const int passes = warp_max(m), span = warp_max(k1 - k0);
    for (int p = 0; p < passes; p += G) {
      const int mine = p + gl < m ? AP.col[c0 + p + gl] : -1;
      double acc[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) acc[v] = 0.0;
      for (int kb = 0; kb < span; kb += G) {
        int pbeg = 0, len = 0;
        if (k0 + kb + gl < k1) {
          const int j = A.col[k0 + kb + gl];
          pbeg = P.ptr[j];
          len = P.ptr[j + 1] - pbeg;
        }
        const int us = min(G, span - kb);
        for (int u = 0; u < us; ++u) {
          const int hit = gal_hit<G>(P.col, __shfl_sync(0xffffffffu, pbeg, u, G), __shfl_sync(0xffffffffu, len, u, G),
                                     mine, gl);
          if (hit < 0) continue;
          const double* a = A.val + (size_t)(k0 + kb + u) * B * B;
          const double* pb = P.val + (size_t)hit * NV;
#pragma unroll
          for (int r = 0; r < B; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              double x = 0.0;
#pragma unroll
              for (int z = 0; z < B; ++z) x = fma(a[r * B + z], pb[z * 3 + c], x);
              acc[r * 3 + c] = __dadd_rn(acc[r * 3 + c], x);
            }
        }
      }
      if (p + gl < m) {
        double* out = const_cast<double*>(AP.val) + (size_t)(c0 + p + gl) * NV;
#pragma unroll
        for (int v = 0; v < NV; ++v) out[v] = acc[v];
      }
    }
  }
}

// P' structure: for each coarse node J the P blocks (fine row, block index) in ascending fine row
__global__ void k_pt_count(int n, AmgBsr P, int* __restrict__ cnt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int q = P.ptr[i]; q < P.ptr[i + 1]; ++q) atomicAdd(&cnt[P.col[q]], 1);
}

__global__ void k_pt_fill(int n, AmgBsr P, const int* __restrict__ ptr, int* __restrict__ cur, int* __restrict__ idx) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int q = P.ptr[i]; q < P.ptr[i + 1]; ++q) {
    const int J = P.col[q];
    idx[ptr[J] + atomicAdd(&cur[J], 1)] = q;  // P block index (its fine row is found by search)
  }
}

// A_c = P' (AP): the column set of coarse row J, one warp per row. The lanes take the fine rows i
// of column J of P (the P' list) and insert the columns of AP's row i into a per-warp open-
// addressing set in shared memory (kAcSet slots, twice the row bound, so a row within the bound
// never fills it). FILL = false: cnt[J] = the number of distinct columns (error word if above
// kAmgMaxRow); FILL = true: the columns in ascending order, each written at its rank in the set.
// Insertion order (and so the set's layout) varies between runs; the counts and sorted columns
// do not.
constexpr int kAcSet = 2 * kAmgMaxRow;
constexpr int kAcWarps = 8;
constexpr int ilog2(int v) { return v <= 1 ? 0 : 1 + ilog2(v >> 1); }
constexpr int kAcShift = 32 - ilog2(kAcSet);
static_assert((kAcSet & (kAcSet - 1)) == 0 && kAcSet % 32 == 0, "set size: a power of two, whole warps");

__device__ __forceinline__ unsigned ac_slot(int c) {
  return ((unsigned)c * 2654435761u) >> kAcShift;  // multiplicative hash, top bits
}

template <bool FILL>
__global__ void __launch_bounds__(32 * kAcWarps) k_amg_ac_pattern(int nc, const int* __restrict__ pt_ptr,
                                                                  const int* __restrict__ pt_idx,
                                                                  const int* __restrict__ p_row /* null: rows pt_idx */,
                                                                  AmgBsr AP,
                                                                  int* __restrict__ cnt, AmgBsr Ac, int* err) {
  __shared__ int set[kAcWarps][kAcSet];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int J = blockIdx.x * kAcWarps + w; J < nc; J += gridDim.x * kAcWarps) {
    for (int h = lane; h < kAcSet; h += 32) set[w][h] = -1;
    __syncwarp();
    int full = 0;
    const int t1 = pt_ptr[J + 1];
    for (int t = pt_ptr[J] + lane; t < t1; t += 32) {
      const int i = p_row ? p_row[pt_idx[t]] : pt_idx[t];
      for (int q = AP.ptr[i]; q < AP.ptr[i + 1]; ++q) {
        const int c = AP.col[q];
        unsigned h = ac_slot(c);
        int probe = 0;
        for (; probe < kAcSet; ++probe) {
          const int old = atomicCAS(&set[w][h], -1, c);
          if (old == -1 || old == c) break;
          h = (h + 1) & (kAcSet - 1);
        }
        if (probe == kAcSet) full = 1;
      }
    }
    __syncwarp();
    // the distinct columns, packed to the front of the set
    int v[kAcSet / 32], at[kAcSet / 32];
    int m = 0;
#pragma unroll
    for (int u = 0; u < kAcSet / 32; ++u) {
      v[u] = set[w][lane + 32 * u];
      const unsigned on = __ballot_sync(0xffffffffu, v[u] >= 0);
      at[u] = m + __popc(on & ((1u << lane) - 1u));
      m += __popc(on);
    }
    full = __any_sync(0xffffffffu, full);
    if (!FILL) {
      if (lane == 0) {
        if (full || m > kAmgMaxRow) atomicMin(&err[kErrAmg], J);
        cnt[J] = m;
      }
    } else {
#pragma unroll
      for (int u = 0; u < kAcSet / 32; ++u)
        if (v[u] >= 0) set[w][at[u]] = v[u];
      __syncwarp();
      int* cols = const_cast<int*>(Ac.col) + Ac.ptr[J];
      for (int e = lane; e < m; e += 32) {  // each at its rank among them
        const int c = set[w][e];
        int r = 0;
        for (int h = 0; h < m; ++h) r += set[w][h] < c ? 1 : 0;
        cols[r] = c;
      }
    }
    __syncwarp();
  }
}

// A_c = P' (AP): values. Coarse row J's candidates: for each P block (i, J) in ascending fine row
// i, for each block q of AP's row i (ascending), the 3 x 3 product P_iJ' (AP)_q.
template <int B, int G>
__global__ void __launch_bounds__(32 * kGalWarps) k_amg_ac_vals(int nc, const int* __restrict__ pt_ptr,
                                                                const int* __restrict__ pt_idx,
                                                                const int* __restrict__ p_row, AmgBsr P, AmgBsr AP,
                                                                AmgBsr Ac) {
  constexpr int NV = B * 3, R = 32 / G;
  const int lane = threadIdx.x & 31, gl = lane % G;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  for (int base = warp * R; base < nc; base += nw * R) {
    const int J = base + lane / G;
    const bool on = J < nc;
    const int c0 = on ? Ac.ptr[J] : 0, m = on ? Ac.ptr[J + 1] - c0 : 0;
    const int t0 = on ? pt_ptr[J] : 0, t1 = on ? pt_ptr[J + 1] : 0;
    const int passes = warp_max(m), span = warp_max(t1 - t0);
    for (int p = 0; p < passes; p += G) {
      const int mine = p + gl < m ? Ac.col[c0 + p + gl] : -1;
      double acc[9];
#pragma unroll
      for (int v = 0; v < 9; ++v) acc[v] = 0.0;
      for (int tb = 0; tb < span; tb += G) {
        int pq = 0, abeg = 0, len = 0;
        if (t0 + tb + gl < t1) {
          pq = pt_idx[t0 + tb + gl];
          const int i = p_row[pq];
          abeg = AP.ptr[i];
          len = AP.ptr[i + 1] - abeg;
        }
        const int us = min(G, span - tb);
        for (int u = 0; u < us; ++u) {
          const int pu = __shfl_sync(0xffffffffu, pq, u, G);
          const int hit = gal_hit<G>(AP.col, __shfl_sync(0xffffffffu, abeg, u, G),
                                     __shfl_sync(0xffffffffu, len, u, G), mine, gl);
          if (hit < 0) continue;
          const double* pb = P.val + (size_t)pu * NV;    // P_iJ (B x 3)
          const double* ab = AP.val + (size_t)hit * NV;  // (AP)_iK (B x 3)
#pragma unroll
          for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              double x = 0.0;
#pragma unroll
              for (int z = 0; z < B; ++z) x = fma(pb[z * 3 + r], ab[z * 3 + c], x);
              acc[r * 3 + c] = __dadd_rn(acc[r * 3 + c], x);
            }
        }
      }
      if (p + gl < m) {
        double* out = const_cast<double*>(Ac.val) + (size_t)(c0 + p + gl) * 9;
#pragma unroll
        for (int v = 0; v < 9; ++v) out[v] = acc[v];
      }
    }
  }
}

// fine row of every P block (for P' traversal)
__global__ void k_p_rows(int n, AmgBsr P, int* __restrict__ p_row) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int q = P.ptr[i]; q < P.ptr[i + 1]; ++q) p_row[q] = i;
}

// sort the P' lists by fine row (so that A_c's additions follow a fixed order)
// P' lists in ascending block index (= ascending fine row): one warp per coarse node J; each
// entry of the unsorted list `in` goes to its rank among the list's entries (all distinct).
__global__ void __launch_bounds__(256) k_rank_pt(int nc, const int* __restrict__ ptr, const int* __restrict__ in,
                                                 int* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  for (int J = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; J < nc; J += (gridDim.x * blockDim.x) >> 5) {
    const int lo = ptr[J], hi = ptr[J + 1];
    for (int a = lo + lane; a < hi; a += 32) {
      const int x = in[a];
      int r = 0;
      for (int b = lo; b < hi; ++b) r += in[b] < x ? 1 : 0;
      out[lo + r] = x;
    }
  }
}

// ---- coarsest level: dense inverse (Gauss-Jordan without pivoting: A is SPD) ---------------------------

template <int B>
__global__ void k_amg_dense(int nb, AmgBsr A, double* __restrict__ M) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nb) return;
  const int n = nb * B;
  for (int k = A.ptr[i]; k < A.ptr[i + 1]; ++k) {
    const int j = A.col[k];
    for (int r = 0; r < B; ++r)
      for (int c = 0; c < B; ++c) M[(size_t)(B * i + r) * n + B * j + c] = A.val[(size_t)k * B * B + r * B + c];
  }
}

// One CTA. M (n x n) is replaced by its inverse; a zero pivot (a dropped nullspace direction
// leaves an exactly singular coarse row) is skipped: that row and column of the inverse are 0.
__global__ void __launch_bounds__(1024) k_amg_gauss_jordan(int n, double* __restrict__ M, double* __restrict__ piv) {
  for (int k = 0; k < n; ++k) {
    __syncthreads();
    const double d = M[(size_t)k * n + k];
    const double scale = fabs(d) > 0.0 ? 1.0 / d : 0.0;
    if (threadIdx.x == 0) piv[k] = scale;
    __syncthreads();
    // column k of the other rows (kept before the row update)
    for (int i = threadIdx.x; i < n; i += blockDim.x) piv[n + i] = i == k ? 0.0 : M[(size_t)i * n + k];
    __syncthreads();
    for (int j = threadIdx.x; j < n; j += blockDim.x) M[(size_t)k * n + j] = j == k ? scale : M[(size_t)k * n + j] * scale;
    __syncthreads();
    for (int t = threadIdx.x; t < n * n; t += blockDim.x) {
      const int i = t / n, j = t - i * n;
      if (i == k) continue;
      const double f = piv[n + i];
      if (j == k)
        M[(size_t)i * n + j] = -f * scale;
      else
        M[(size_t)i * n + j] -= f * M[(size_t)k * n + j];
    }
  }
}

// The same for n <= 128, the matrix in the threads' registers (16 entries each, rows ti + 32 a, columns
// tj + 32 b); a step publishes the pivot's row, column and reciprocal through shared memory (two sets,
// one barrier a step). Latency: the kernel above meets five barriers and the caches at each step, 367 us
// for 102 unknowns; this takes 152.
constexpr int kGjMax = 128;

__global__ void __launch_bounds__(1024) k_amg_gauss_jordan_regs(int n, double* __restrict__ M) {
  constexpr int T = kGjMax / 32;
  __shared__ double row[2][kGjMax], col[2][kGjMax], scale[2];
  const int ti = threadIdx.x >> 5, tj = threadIdx.x & 31;
  double m[T][T];
#pragma unroll
  for (int a = 0; a < T; ++a)
#pragma unroll
    for (int b = 0; b < T; ++b) {
      const int i = ti + 32 * a, j = tj + 32 * b;
      m[a][b] = i < n && j < n ? M[(size_t)i * n + j] : 0.0;
    }
  for (int k = 0; k < n; ++k) {
    const int h = k & 1, ka = k >> 5, kt = k & 31;
#pragma unroll
    for (int a = 0; a < T; ++a)
#pragma unroll
      for (int b = 0; b < T; ++b) {
        if (tj == kt && b == ka) col[h][ti + 32 * a] = m[a][b];
        if (ti == kt && a == ka) row[h][tj + 32 * b] = m[a][b];
        if (ti == kt && tj == kt && a == ka && b == ka) scale[h] = fabs(m[a][b]) > 0.0 ? 1.0 / m[a][b] : 0.0;
      }
    __syncthreads();
    const double s = scale[h];
    double f[T], r[T];
#pragma unroll
    for (int a = 0; a < T; ++a) f[a] = col[h][ti + 32 * a];
#pragma unroll
    for (int b = 0; b < T; ++b) r[b] = row[h][tj + 32 * b] * s;
#pragma unroll
    for (int a = 0; a < T; ++a)
#pragma unroll
      for (int b = 0; b < T; ++b) {
        const bool ik = ti == kt && a == ka, jk = tj == kt && b == ka;
        m[a][b] = ik ? (jk ? s : r[b]) : jk ? -f[a] * s : fma(-f[a], r[b], m[a][b]);
      }
  }
#pragma unroll
  for (int a = 0; a < T; ++a)
#pragma unroll
    for (int b = 0; b < T; ++b) {
      const int i = ti + 32 * a, j = tj + 32 * b;
      if (i < n && j < n) M[(size_t)i * n + j] = m[a][b];
    }
}

// ---- cycle kernels ----------------------------------------------------------------------------------

// A cycle launched inside the flexible-CG graph carries the solver's done flag: once the solve
// has converged, the rest of the captured chunk's cycles return at once.
__device__ __forceinline__ bool skipped(const int* skip) { return skip && *(volatile const int*)skip != 0; }

// Smoother steps. With r(x) = D^-1 (b - A x):
//   kSweepFirst     xo = beta x0 + gamma r(x0), x0 = a0 D^-1 b (finest level: formed on the fly, x not
//                   read; below: x, written with b by the restriction)
//   kSweepSmooth    xo = x + gamma r(x)
//   kSweepSecond    xo = x + cd (x - xp) + gamma r(x)   (xp: the iterate before x)
//   kSweepResidual  xo = b - A x
// Damped Jacobi (weight w = 4 / (3 lam)): a0 = gamma = w, beta = 1, every post step kSweepSmooth.
// Chebyshev of degree 2 on [hi / kChebRatio, hi], hi = kChebHi lam (the three-term recurrence:
// theta = (hi + lo) / 2, delta = (hi - lo) / 2, sigma = theta / delta, rho1 = 1 / sigma,
// rho2 = 1 / (2 sigma - rho1)): the two pre-smoothing steps from x = 0 are one kSweepFirst with
// a0 = 1 / theta, beta = 1 + rho2 rho1, gamma = 2 rho2 / delta; the two post-smoothing steps are
// kSweepSmooth with gamma = 1 / theta, then kSweepSecond with cd = rho2 rho1, gamma = 2 rho2 / delta.
constexpr double kChebHi = 1.1, kChebRatio = 20.0;

struct SweepCoef {
  double a0, beta, gamma, cd;
};

__device__ SweepCoef sweep_coef_of(int mode, double l, int cheb) {
  SweepCoef c{0.0, 1.0, 0.0, 0.0};
  if (mode == kSweepResidual) return c;
  if (!cheb) {
    const double w = 4.0 / (3.0 * l);
    c.a0 = w;
    c.gamma = w;
    return c;
  }
  const double hi = kChebHi * l, lo = hi / kChebRatio;
  const double theta = 0.5 * (hi + lo), delta = 0.5 * (hi - lo), sigma = theta / delta;
  const double rho1 = 1.0 / sigma, rho2 = 1.0 / (2.0 * sigma - rho1);
  if (mode == kSweepFirst) {
    c.a0 = 1.0 / theta;
    c.beta = 1.0 + rho2 * rho1;
    c.gamma = 2.0 * rho2 / delta;
  } else if (mode == kSweepSmooth) {
    c.gamma = 1.0 / theta;
  } else {
    c.cd = rho2 * rho1;
    c.gamma = 2.0 * rho2 / delta;
  }
  return c;
}

// The coefficients of every step follow lambda_max in its buffer (kAmgLamDoubles), computed once per
// setup: in the sweeps every thread spent five dependent FP64 divisions on them, more than on its node.
__global__ void k_amg_sweep_coef(double* lam) {
  const int t = threadIdx.x;  // 4 steps x (Jacobi, Chebyshev)
  const SweepCoef c = sweep_coef_of(t & 3, lam[0], t >> 2);
  double* o = lam + 1 + 4 * t;
  o[0] = c.a0;
  o[1] = c.beta;
  o[2] = c.gamma;
  o[3] = c.cd;
}

template <int MODE>
__device__ __forceinline__ SweepCoef sweep_coef(const double* lam, int cheb) {
  if (MODE == kSweepResidual) return SweepCoef{0.0, 1.0, 0.0, 0.0};
  const double* o = lam + 1 + 4 * (MODE + (cheb ? 4 : 0));
  return SweepCoef{__ldg(&o[0]), __ldg(&o[1]), __ldg(&o[2]), __ldg(&o[3])};
}

// the update of component i given its current value xi (and previous value xpi for kSweepSecond)
template <int MODE>
__device__ __forceinline__ double sweep_out(const SweepCoef& c, double dinv_i, double res, double xi, double xpi) {
  if (MODE == kSweepResidual) return res;
  if (MODE == kSweepFirst) return fma(c.gamma * dinv_i, res, c.beta == 1.0 ? xi : c.beta * xi);
  if (MODE == kSweepSecond) return fma(c.gamma * dinv_i, res, fma(c.cd, xi - xpi, xi));
  return fma(c.gamma * dinv_i, res, xi);
}

// x0 = a0 D^-1 b, component i (the first step's iterate)
__device__ __forceinline__ double first_x(double a0, const double* __restrict__ dinv, const double* __restrict__ b,
                                          size_t i) {
  return a0 * dinv[i] * b[i];
}

// The flexible-CG scalars that follow a cycle (k_fcg_dots of fcg.cu), taken in the cycle's last
// finest-level sweep, which already holds z (its output) and r (its right-hand side): z'r and
// z'q reduced on the sweep's fixed grid (per-block partials, the last block by ticket adds them
// in block order), then beta = -alpha z'q / (z'r)_old (Polak-Ribiere; a restart or a non-descent
// z gives beta = 0). The cycle is symmetric positive, so the Jacobi fallback of the learned
// network is not needed here.
__device__ __forceinline__ void fcg_dots_epilogue(double zr, double zq, const FcgDotSink& d) {
  __shared__ double sm[kWarps];
  __shared__ bool am_last;
  const double a = block_sum<kThreads>(zr, sm);
  const double c = block_sum<kThreads>(zq, sm);
  if (threadIdx.x == 0) {
    d.partials[blockIdx.x] = a;
    d.partials[gridDim.x + blockIdx.x] = c;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) am_last = atomicAdd(&d.st->ticket[6], 1u) == gridDim.x - 1;
  __syncthreads();
  if (!am_last) return;
  __threadfence();
  double s0 = 0.0, s1 = 0.0;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) {
    s0 += __ldcg(&d.partials[i]);
    s1 += __ldcg(&d.partials[gridDim.x + i]);
  }
  const double t0 = block_sum<kThreads>(s0, sm);
  const double t1 = block_sum<kThreads>(s1, sm);
  if (threadIdx.x == 0) {
    PcgState* st = d.st;
    const bool restart = st->restart_pending != 0 || !(t0 > 0.0);
    st->beta = (!restart && st->rz > 0.0) ? -st->alpha * t1 / st->rz : 0.0;
    st->rz = t0;
    st->use_jacobi = 0;
    st->restart_pending = 0;
    st->ticket[6] = 0u;
  }
}

// Finest-level sweep on the FP32 difference-form operator of mixed_kernels.cu (the smoother is a
// preconditioner: FP32 matrix values, FP64 vectors and accumulation). Thread per node; four
// neighbours' index and value loads are in flight at once, their gathers next, and the additions
// follow in neighbour order. DOTS: the cycle's last sweep inside flexible CG also takes z'r and
// z'q (fcg_dots_epilogue).
template <int MODE, bool DOTS = false>
__global__ void __launch_bounds__(256) k_amg_sweep_f32(const int* skip, MixedMatrix M, const double* __restrict__ dinv,
                                                       const double* __restrict__ lam, int cheb,
                                                       const double* __restrict__ b, const double* __restrict__ x,
                                                       const double* xp, double* xo, FcgDotSink dots) {
  if (skipped(skip)) return;
  double zr = 0.0, zq = 0.0;
  const SweepCoef cf = sweep_coef<MODE>(lam, cheb);
  const double2* x2 = reinterpret_cast<const double2*>(x);
  auto xnode = [&](int m) -> double2 {
    if (MODE == kSweepFirst)
      return make_double2(first_x(cf.a0, dinv, b, 2 * (size_t)m), first_x(cf.a0, dinv, b, 2 * (size_t)m + 1));
    return x2[m];
  };
  for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < M.n_nodes; n += gridDim.x * blockDim.x) {
    const int bb = __ldg(&M.node_ptr[n]);
    const int o = bb - n, c = __ldg(&M.node_ptr[n + 1]) - bb - 1;
    const double2 xs = xnode(n);
    double ya = 0.0, yb = 0.0;
    int k = 0;
    for (; k + 4 <= c; k += 4) {
      int m[4];
      float4 a[4];
      double2 xm[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        m[u] = __ldg(&M.nbr32[o + k + u]);
        a[u] = __ldg(&M.val32[o + k + u]);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) xm[u] = xnode(m[u]);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const double dx = xm[u].x - xs.x, dy = xm[u].y - xs.y;
        ya = fma((double)a[u].x, dx, fma((double)a[u].y, dy, ya));
        yb = fma((double)a[u].z, dx, fma((double)a[u].w, dy, yb));
      }
    }
    for (; k < c; ++k) {
      const int m = __ldg(&M.nbr32[o + k]);
      const float4 a = __ldg(&M.val32[o + k]);
      const double2 xm = xnode(m);
      const double dx = xm.x - xs.x, dy = xm.y - xs.y;
      ya = fma((double)a.x, dx, fma((double)a.y, dy, ya));
      yb = fma((double)a.z, dx, fma((double)a.w, dy, yb));
    }
    const double2 sa = __ldg(&M.S64[2 * n]), sb = __ldg(&M.S64[2 * n + 1]);
    ya = fma(sa.x, xs.x, fma(sa.y, xs.y, ya));
    yb = fma(sb.x, xs.x, fma(sb.y, xs.y, yb));
    const double2 bv = reinterpret_cast<const double2*>(b)[n];
    const double ra = bv.x - ya, rbv = bv.y - yb;
    double2 out;
    if (MODE == kSweepResidual) {
      out = make_double2(ra, rbv);
    } else {
      const double2 dv = reinterpret_cast<const double2*>(dinv)[n];
      const double2 pv = MODE == kSweepSecond ? reinterpret_cast<const double2*>(xp)[n] : make_double2(0.0, 0.0);
      out = make_double2(sweep_out<MODE>(cf, dv.x, ra, xs.x, pv.x), sweep_out<MODE>(cf, dv.y, rbv, xs.y, pv.y));
    }
    reinterpret_cast<double2*>(xo)[n] = out;
    if (DOTS) {
      const double2 qv = reinterpret_cast<const double2*>(dots.q)[n];
      zr = fma(out.x, bv.x, fma(out.y, bv.y, zr));
      zq = fma(out.x, qv.x, fma(out.y, qv.y, zq));
    }
  }
  if (DOTS) fcg_dots_epilogue(zr, zq, dots);
}

// Loads of vectors: COH = false for standalone launches (the vector was written by an earlier
// launch), true inside the coarse-tail kernel, where another CTA of the cluster wrote it in an
// earlier phase: those loads go to L2 (ld.global.cg), never through the non-coherent path.
template <bool COH>
__device__ __forceinline__ double ldv(const double* p) {
  if (COH) return __ldcg(p);
  return *p;
}

// Coarse-level sweep on the FP32 copy of a 3 x 3 block operator (FP64 vectors and accumulation).
// The copy is stored entry-major (val[e * nnzb + k], e = 0..8). 8 lanes per row (4 rows per
// warp): the lanes of a row take consecutive blocks, so each entry load of the 8 lanes is one
// contiguous 32-byte run; a fixed 3-step shuffle tree adds the lanes. Row groups are strided over
// `nw` warps (warp index `warp`): rows of any length keep 8 lanes busy, and small levels still
// spread over the whole grid.
template <int MODE, bool COH>
__device__ __forceinline__ void sweep3_rows(const AmgBsr32& A, const double* dinv, const SweepCoef& cf,
                                            const double* b, const double* x, const double* xp, double* xo, int warp,
                                            int nw, int lane) {
  auto xval = [&](size_t d) -> double { return ldv<COH>(&x[d]); };  // (kSweepFirst: x0, from the restriction)
  const size_t nb = (size_t)A.nnzb;
  const int l8 = lane & 7, sub = lane >> 3;
  for (int base = warp * 4; base < A.n; base += nw * 4) {
    const int i = base + sub;
    double a0 = 0.0, a1 = 0.0, a2 = 0.0;
    if (i < A.n) {
      const int k1 = __ldg(&A.ptr[i + 1]);
      for (int k = __ldg(&A.ptr[i]) + l8; k < k1; k += 8) {
        const int c = __ldg(&A.col[k]);
        float v[9];
#pragma unroll
        for (int e = 0; e < 9; ++e) v[e] = __ldg(&A.val[(size_t)e * nb + k]);
        const double x0 = xval(3 * (size_t)c), x1 = xval(3 * (size_t)c + 1), x2v = xval(3 * (size_t)c + 2);
        a0 = fma((double)v[0], x0, fma((double)v[1], x1, fma((double)v[2], x2v, a0)));
        a1 = fma((double)v[3], x0, fma((double)v[4], x1, fma((double)v[5], x2v, a1)));
        a2 = fma((double)v[6], x0, fma((double)v[7], x1, fma((double)v[8], x2v, a2)));
      }
    }
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) {
      a0 += __shfl_xor_sync(0xffffffffu, a0, off);
      a1 += __shfl_xor_sync(0xffffffffu, a1, off);
      a2 += __shfl_xor_sync(0xffffffffu, a2, off);
    }
    if (i < A.n && l8 < 3) {
      const size_t d = 3 * (size_t)i + l8;
      const double acc = l8 == 0 ? a0 : l8 == 1 ? a1 : a2;
      const double res = ldv<COH>(&b[d]) - acc;
      xo[d] = MODE == kSweepResidual
                  ? res
                  : sweep_out<MODE>(cf, __ldg(&dinv[d]), res, xval(d), MODE == kSweepSecond ? ldv<COH>(&xp[d]) : 0.0);
    }
  }
}

template <int MODE>
__global__ void __launch_bounds__(256, 8) k_amg_sweep3_f32(const int* skip, AmgBsr32 A,
                                                        const double* __restrict__ dinv,
                                                        const double* __restrict__ lam, int cheb, const double* b,
                                                        const double* x, const double* xp, double* xo) {
  if (skipped(skip)) return;
  const SweepCoef cf = sweep_coef<MODE>(lam, cheb);
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  sweep3_rows<MODE, false>(A, dinv, cf, b, x, xp, xo, warp, nw, threadIdx.x & 31);
}

// The B x 3 entries of FP32 transfer block t (the finest level's as 8-byte loads: its blocks are 24 bytes,
// and a load of a scattered word costs the load units as much as one of two).
template <int B>
__device__ __forceinline__ void load_transfer(const float* p32, size_t t, float (&v)[B * 3]) {
  if (B == 2) {
    const float2* q = reinterpret_cast<const float2*>(p32 + t * 6);
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      const float2 w = __ldg(&q[e]);
      v[2 * e] = w.x;
      v[2 * e + 1] = w.y;
    }
  } else {
#pragma unroll
    for (int e = 0; e < B * 3; ++e) v[e] = __ldg(&p32[t * B * 3 + e]);
  }
}

// bc_J = sum over the P blocks of column J of P_iJ' r_i, from the FP32 copy of P stored by coarse
// row (pt32, pt_row): one warp per coarse row, lanes over the row's blocks, fixed shuffle tree. The next
// row's extent is loaded a row ahead.
// bc's level starts from x0 = a0 D^-1 bc, written here (x0 null: the dense coarsest level): its first
// sweep formed it at every neighbour from dinv and b, 18.5 us on 287,703 DOFs where it now takes 13.8.
template <int B, bool COH>
__device__ __forceinline__ void restrict_rows(int nc, const int* pt_ptr, const int* pt_row, const float* pt32,
                                              const double* r, double* bc, const RestrictStart& st, int warp, int nw,
                                              int lane) {
  const double first = st.x0 ? sweep_coef<kSweepFirst>(st.lam, st.cheb).a0 : 0.0;
  int t0 = 0, t1 = 0;
  if (warp < nc) {
    t0 = __ldg(&pt_ptr[warp]);
    t1 = __ldg(&pt_ptr[warp + 1]);
  }
  for (int J = warp; J < nc; J += nw) {
    int n0 = 0, n1 = 0;
    if (J + nw < nc) {
      n0 = __ldg(&pt_ptr[J + nw]);
      n1 = __ldg(&pt_ptr[J + nw + 1]);
    }
    const double dv = st.x0 && lane < 3 ? __ldg(&st.dinv[3 * (size_t)J + lane]) : 0.0;
    double a0 = 0.0, a1 = 0.0, a2 = 0.0;
    for (int t = t0 + lane; t < t1; t += 32) {
      const int i = __ldg(&pt_row[t]);
      float v[B * 3];
      load_transfer<B>(pt32, (size_t)t, v);
      double rv[B];
      if (B == 2 && !COH) {
        const double2 w = reinterpret_cast<const double2*>(r)[i];
        rv[0] = w.x;
        rv[1] = w.y;
      } else {
#pragma unroll
        for (int z = 0; z < B; ++z) rv[z] = ldv<COH>(&r[(size_t)i * B + z]);
      }
#pragma unroll
      for (int z = 0; z < B; ++z) {
        a0 = fma((double)v[z * 3 + 0], rv[z], a0);
        a1 = fma((double)v[z * 3 + 1], rv[z], a1);
        a2 = fma((double)v[z * 3 + 2], rv[z], a2);
      }
    }
    a0 = warp_sum(a0);
    a1 = warp_sum(a1);
    a2 = warp_sum(a2);
    if (lane < 3) {
      const size_t d = 3 * (size_t)J + lane;
      const double v = lane == 0 ? a0 : lane == 1 ? a1 : a2;
      bc[d] = v;
      if (st.x0) st.x0[d] = first * dv * v;
    }
    t0 = n0;
    t1 = n1;
  }
}

template <int B>
__global__ void __launch_bounds__(256) k_amg_restrict_f32(const int* skip, int nc, const int* __restrict__ pt_ptr,
                                                          const int* __restrict__ pt_row,
                                                          const float* __restrict__ pt32, const double* r,
                                                          double* bc, RestrictStart st) {
  if (skipped(skip)) return;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  restrict_rows<B, false>(nc, pt_ptr, pt_row, pt32, r, bc, st, warp, nw, threadIdx.x & 31);
}

// x += P xc with the FP32 copy of P (thread per fine row). The loads of several blocks are in flight at
// once; the additions follow in block order. Bound by the load units (scattered rows); 2,000,244 DOFs: 34
// -> 25 us with 8-byte loads, three blocks at a time (15 at the measured HBM bandwidth).
template <int B, bool COH>
__device__ __forceinline__ void prolong_rows(int n, const int* p_ptr, const int* p_col, const float* p32,
                                             const double* xc, double* x, int tid, int nt) {
  constexpr int U = B == 2 ? 3 : 2;
  for (int i = tid; i < n; i += nt) {
    double acc[B];
    if (B == 2 && !COH) {
      const double2 w = reinterpret_cast<const double2*>(x)[i];
      acc[0] = w.x;
      acc[1] = w.y;
    } else {
#pragma unroll
      for (int r = 0; r < B; ++r) acc[r] = ldv<COH>(&x[(size_t)i * B + r]);
    }
    const int q1 = __ldg(&p_ptr[i + 1]);
    for (int q = __ldg(&p_ptr[i]); q < q1; q += U) {
      float v[U][B * 3];
      double c[U][3];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int k = min(q + u, q1 - 1);
        const double* xj = xc + 3 * (size_t)__ldg(&p_col[k]);
        load_transfer<B>(p32, (size_t)k, v[u]);
#pragma unroll
        for (int e = 0; e < 3; ++e) c[u][e] = ldv<COH>(&xj[e]);
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (q + u < q1) {
#pragma unroll
          for (int r = 0; r < B; ++r)
            acc[r] = fma((double)v[u][r * 3 + 2], c[u][2],
                         fma((double)v[u][r * 3 + 1], c[u][1], fma((double)v[u][r * 3], c[u][0], acc[r])));
        }
    }
    if (B == 2) {
      reinterpret_cast<double2*>(x)[i] = make_double2(acc[0], acc[1]);
    } else {
#pragma unroll
      for (int r = 0; r < B; ++r) x[(size_t)i * B + r] = acc[r];
    }
  }
}

template <int B>
__global__ void __launch_bounds__(256) k_amg_prolong_f32(const int* skip, int n, const int* __restrict__ p_ptr,
                                                         const int* __restrict__ p_col, const float* __restrict__ p32,
                                                         const double* xc, double* x) {
  if (skipped(skip)) return;
  prolong_rows<B, false>(n, p_ptr, p_col, p32, xc, x, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

// x = M b (dense, n x n): one warp per row
template <bool COH>
__device__ __forceinline__ void gemv_rows(int n, const double* M, const double* b, double* x, int warp, int nw,
                                          int lane) {
  for (int i = warp; i < n; i += nw) {
    double s = 0.0;
    for (int j = lane; j < n; j += 32) s = fma(__ldg(&M[(size_t)i * n + j]), ldv<COH>(&b[j]), s);
    s = warp_sum(s);
    if (lane == 0) x[i] = s;
  }
}

__global__ void k_amg_gemv(const int* skip, int n, const double* __restrict__ M, const double* b, double* x) {
  if (skipped(skip)) return;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  gemv_rows<false>(n, M, b, x, warp, nw, threadIdx.x & 31);
}

// The bottom of the V-cycle (the small coarse levels and the dense coarsest solve) in ONE launch
// of one thread-block cluster: every phase (sweep, residual, restriction, coarsest product,
// prolongation) is spread over all threads of the cluster and the phases are separated by
// cluster barriers (release/acquire at cluster scope; vectors written in a phase are read in the
// next through L2). The same row functions and orders of addition as the per-level launches, so
// the result is bit-identical to them; only the ~13 launch latencies of these small levels go.
__device__ __forceinline__ void prefetch_l2(const void* p, size_t bytes, int tid, int nt) {
  const char* c = static_cast<const char*>(p);
  for (size_t o = (size_t)tid * 128; o < bytes; o += (size_t)nt * 128)
    asm volatile("prefetch.global.L2 [%0];\n" ::"l"(c + o));
}

__global__ void __launch_bounds__(kAmgTailThreads, 1) k_amg_tail(const int* skip, const __grid_constant__ AmgTail T) {
  if (skipped(skip)) return;  // (uniform over the cluster: every CTA leaves before any barrier)
  const cg::cluster_group cl = cg::this_cluster();
  const int tid = (int)cl.block_rank() * blockDim.x + threadIdx.x;
  const int nt = (int)cl.num_blocks() * blockDim.x;
  const int lane = threadIdx.x & 31, warp = tid >> 5, nw = nt >> 5;
  // the rest of the cycle has pushed the levels' operators out of L2: their DRAM latencies all at once
  for (int l = 0; l + 1 < T.nl; ++l) {
    const AmgTailLevel& v = T.L[l];
    prefetch_l2(v.A.ptr, sizeof(int) * (size_t)(v.A.n + 1), tid, nt);
    prefetch_l2(v.A.col, sizeof(int) * (size_t)v.A.nnzb, tid, nt);
    prefetch_l2(v.A.val, sizeof(float) * 9 * (size_t)v.A.nnzb, tid, nt);
    prefetch_l2(v.dinv, sizeof(double) * 3 * (size_t)v.A.n, tid, nt);
    prefetch_l2(v.pt_ptr, sizeof(int) * (size_t)(v.nc + 1), tid, nt);
    prefetch_l2(v.p_ptr, sizeof(int) * (size_t)(v.A.n + 1), tid, nt);
    prefetch_l2(v.pt_row, sizeof(int) * (size_t)v.nnz_p, tid, nt);
    prefetch_l2(v.p_col, sizeof(int) * (size_t)v.nnz_p, tid, nt);
    prefetch_l2(v.pt32, sizeof(float) * 9 * (size_t)v.nnz_p, tid, nt);
    prefetch_l2(v.p32, sizeof(float) * 9 * (size_t)v.nnz_p, tid, nt);
  }
  prefetch_l2(T.Minv, sizeof(double) * (size_t)T.n_coarse * T.n_coarse, tid, nt);
  for (int l = 0; l + 1 < T.nl; ++l) {
    const AmgTailLevel& v = T.L[l];
    sweep3_rows<kSweepFirst, true>(v.A, v.dinv, sweep_coef<kSweepFirst>(v.lam, T.cheb), v.b, v.xa, nullptr, v.x,
                                   warp, nw, lane);
    cl.sync();
    sweep3_rows<kSweepResidual, true>(v.A, v.dinv, SweepCoef{0.0, 1.0, 0.0, 0.0}, v.b, v.x, nullptr, v.r, warp, nw,
                                      lane);
    cl.sync();
    const AmgTailLevel& w = T.L[l + 1];
    restrict_rows<3, true>(v.nc, v.pt_ptr, v.pt_row, v.pt32, v.r, w.b,
                           RestrictStart{l + 2 < T.nl ? w.xa : nullptr, w.dinv, w.lam, T.cheb}, warp, nw, lane);
    cl.sync();
  }
  gemv_rows<true>(T.n_coarse, T.Minv, T.L[T.nl - 1].b, T.L[T.nl - 1].x, warp, nw, lane);
  for (int l = T.nl - 2; l >= 0; --l) {
    const AmgTailLevel& v = T.L[l];
    cl.sync();
    prolong_rows<3, true>(v.A.n, v.p_ptr, v.p_col, v.p32, T.L[l + 1].x, v.x, tid, nt);
    cl.sync();
    sweep3_rows<kSweepSmooth, true>(v.A, v.dinv, sweep_coef<kSweepSmooth>(v.lam, T.cheb), v.b, v.x, nullptr, v.xa,
                                    warp, nw, lane);
    cl.sync();
    if (T.cheb)
      sweep3_rows<kSweepSecond, true>(v.A, v.dinv, sweep_coef<kSweepSecond>(v.lam, T.cheb), v.b, v.xa, v.x, v.x,
                                      warp, nw, lane);
    else
      sweep3_rows<kSweepSmooth, true>(v.A, v.dinv, sweep_coef<kSweepSmooth>(v.lam, T.cheb), v.b, v.xa, nullptr, v.x,
                                      warp, nw, lane);
  }
}

// FP32 copy of a coarse operator that is exactly symmetric: block (I, J) with J < I is the
// transpose of the rounded block (J, I) (the FP64 Galerkin product is symmetric only to rounding).
// Stored entry-major: entry e of block k at val32[e * nnzb + k].
__global__ void k_amg_coarse_f32(AmgBsr A, float* __restrict__ val32) {
  const int I = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;  // eight lanes per row
  if (I >= A.n) return;
  const size_t nb = (size_t)A.ptr[A.n];
  for (int k = A.ptr[I] + (threadIdx.x & 7); k < A.ptr[I + 1]; k += 8) {
    const int J = A.col[k];
    int src = k;
    bool tr = false;
    if (J < I) {
      const int m = row_find(A.col, A.ptr[J], A.ptr[J + 1], I);
      if (m < A.ptr[J + 1] && A.col[m] == I) {
        src = m;
        tr = true;
      }
    }
    const double* sv = A.val + (size_t)src * 9;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) val32[(size_t)(r * 3 + c) * nb + k] = (float)(tr ? sv[c * 3 + r] : sv[r * 3 + c]);
  }
}

// FP32 copies of P: by fine row (p32, P's own layout) and by coarse row (pt32 with the fine row
// of each block in pt_row, in the order of the P' lists)
template <int B>
__global__ void k_amg_transfer_f32(int nnz_p, const double* __restrict__ pval, const int* __restrict__ pt_idx,
                                   const int* __restrict__ p_row, float* __restrict__ p32, int* __restrict__ pt_row,
                                   float* __restrict__ pt32) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nnz_p) return;
  const int q = pt_idx[t];
  pt_row[t] = p_row[q];
#pragma unroll
  for (int v = 0; v < B * 3; ++v) {
    p32[(size_t)t * B * 3 + v] = (float)pval[(size_t)t * B * 3 + v];
    pt32[(size_t)t * B * 3 + v] = (float)pval[(size_t)q * B * 3 + v];
  }
}

// 2D rigid-body modes per node: [[1, 0, -y], [0, 1, x]]
__global__ void k_amg_rigid(int N, const double* __restrict__ xy, double* __restrict__ Bf) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  double* b = Bf + 6 * (size_t)n;
  b[0] = 1.0;
  b[1] = 0.0;
  b[2] = -xy[2 * n + 1];
  b[3] = 0.0;
  b[4] = 1.0;
  b[5] = xy[2 * n];
}

// ---- lambda_max(D^-1 A) on the cycle's FP32 operators ---------------------------------------------------
// The power-iteration step (y = s D^-1 A x, per-block partial sums of ||y||^2 on the fixed
// kLamGrid grid) with the operators the smoother applies: the finest level's FP32 difference
// form (thread per node) and a coarse level's entry-major FP32 copy (8 lanes per row).

__global__ void __launch_bounds__(kThreads) k_amg_dinva_fine(MixedMatrix M, const double* __restrict__ dinv,
                                                             double* sc, int first, const double* __restrict__ x,
                                                             double* __restrict__ y, double* part,
                                                             double* lam, unsigned* ticket) {
  const double s = first ? 1.0 : *sc;
  const double2* x2 = reinterpret_cast<const double2*>(x);
  double ss = 0.0;
  for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < M.n_nodes; n += gridDim.x * blockDim.x) {
    const int bb = __ldg(&M.node_ptr[n]);
    const int o = bb - n, c = __ldg(&M.node_ptr[n + 1]) - bb - 1;
    const double2 xs = x2[n];
    double ya = 0.0, yb = 0.0;
    for (int k = 0; k < c; ++k) {
      const int m = __ldg(&M.nbr32[o + k]);
      const float4 a = __ldg(&M.val32[o + k]);
      const double2 xm = x2[m];
      const double dx = xm.x - xs.x, dy = xm.y - xs.y;
      ya = fma((double)a.x, dx, fma((double)a.y, dy, ya));
      yb = fma((double)a.z, dx, fma((double)a.w, dy, yb));
    }
    const double2 sa = __ldg(&M.S64[2 * n]), sb = __ldg(&M.S64[2 * n + 1]);
    ya = fma(sa.x, xs.x, fma(sa.y, xs.y, ya));
    yb = fma(sb.x, xs.x, fma(sb.y, xs.y, yb));
    const double2 dv = reinterpret_cast<const double2*>(dinv)[n];
    const double va = s * (dv.x * ya), vb = s * (dv.y * yb);
    reinterpret_cast<double2*>(y)[n] = make_double2(va, vb);
    ss = fma(va, va, fma(vb, vb, ss));
  }
  __shared__ double sm[kWarps];
  const double t = block_sum<kThreads>(ss, sm);
  amg_norm_epilogue(t, part, lam, sc, ticket, sm);
}

__global__ void __launch_bounds__(kThreads) k_amg_dinva_coarse(AmgBsr32 A, const double* __restrict__ dinv,
                                                               double* sc, int first, const double* __restrict__ x,
                                                               double* __restrict__ y, double* part,
                                                             double* lam, unsigned* ticket) {
  const double s = first ? 1.0 : *sc;
  const size_t nb = (size_t)A.nnzb;
  const int lane = threadIdx.x & 31, l8 = lane & 7, sub = lane >> 3;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  double ss = 0.0;
  for (int base = warp * 4; base < A.n; base += nw * 4) {
    const int i = base + sub;
    double a0 = 0.0, a1 = 0.0, a2 = 0.0;
    if (i < A.n) {
      const int k1 = __ldg(&A.ptr[i + 1]);
      for (int k = __ldg(&A.ptr[i]) + l8; k < k1; k += 8) {
        const int c = __ldg(&A.col[k]);
        float v[9];
#pragma unroll
        for (int e = 0; e < 9; ++e) v[e] = __ldg(&A.val[(size_t)e * nb + k]);
        const double x0 = x[3 * (size_t)c], x1 = x[3 * (size_t)c + 1], x2v = x[3 * (size_t)c + 2];
        a0 = fma((double)v[0], x0, fma((double)v[1], x1, fma((double)v[2], x2v, a0)));
        a1 = fma((double)v[3], x0, fma((double)v[4], x1, fma((double)v[5], x2v, a1)));
        a2 = fma((double)v[6], x0, fma((double)v[7], x1, fma((double)v[8], x2v, a2)));
      }
    }
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) {
      a0 += __shfl_xor_sync(0xffffffffu, a0, off);
      a1 += __shfl_xor_sync(0xffffffffu, a1, off);
      a2 += __shfl_xor_sync(0xffffffffu, a2, off);
    }
    if (i < A.n && l8 < 3) {
      const size_t d = 3 * (size_t)i + l8;
      const double v = s * (dinv[d] * (l8 == 0 ? a0 : l8 == 1 ? a1 : a2));
      y[d] = v;
      ss = fma(v, v, ss);
    }
  }
  __shared__ double sm[kWarps];
  const double t = block_sum<kThreads>(ss, sm);
  amg_norm_epilogue(t, part, lam, sc, ticket, sm);
}

// One full wave of a grid-stride kernel: every SM gets as many blocks as it can hold at once
// (capped by the work), so no partial second wave idles part of the GPU. The occupancy of each
// kernel (256 threads, no dynamic shared memory) is queried once and cached.
int one_wave(const void* kern, long long n_threads) {
  static std::mutex mu;
  static std::vector<std::pair<const void*, int>> cache;
  static int sms = 0;
  int per_sm = 0;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (!sms) {
      int dev = 0;
      cudaGetDevice(&dev);
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      sms = std::max(sms, 1);
    }
    for (const auto& e : cache)
      if (e.first == kern) per_sm = e.second;
    if (!per_sm) {
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 256, 0) != cudaSuccess || per_sm < 1) {
        cudaGetLastError();
        per_sm = 1;
      }
      cache.emplace_back(kern, per_sm);
    }
  }
  const long long need = (n_threads + 255) / 256;
  return (int)std::max<long long>(1, std::min<long long>(need, (long long)per_sm * sms));
}

inline int g1(long long n, int t = 256) { return (int)std::max<long long>(1, std::min<long long>((n + t - 1) / t, 1LL << 30)); }
inline int ac_grid(long long nc) {
  return (int)std::max<long long>(1, std::min<long long>((nc + kAcWarps - 1) / kAcWarps, 148LL * 16));
}
inline int gw(long long n) { return (int)std::max<long long>(1, std::min<long long>((n + 255) / 256, 148LL * 8)); }

}  // namespace

// ---- launchers ---------------------------------------------------------------------------------------

// blocks of the Galerkin value kernels: `lanes` lanes per row, at most 16 blocks per SM
inline int gal_grid(long long rows, int lanes) {
  const long long b = (rows * lanes + 32 * kGalWarps - 1) / (32 * kGalWarps);
  return (int)std::max<long long>(1, std::min<long long>(b, 148LL * 16));
}

cudaError_t amg_fine_bsr(int N, const int* node_ptr, const double* vals, double* out, cudaStream_t s) {
  k_amg_bsr2<<<g1((long long)N * 8), 256, 0, s>>>(N, node_ptr, vals, out);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t amg_dinv(int B, const AmgBsr& A, double* dinv, int* err, cudaStream_t s) {
  if (B == 2)
    k_amg_dinv<2><<<g1(A.n), 256, 0, s>>>(A.n, A, dinv, err);
  else
    k_amg_dinv<3><<<g1(A.n), 256, 0, s>>>(A.n, A, dinv, err);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t amg_strength(int B, const AmgBsr& A, double theta, double* dn, unsigned char* strong, cudaStream_t s) {
  if (B == 2) {
    k_amg_diag_norm<2><<<g1(A.n), 256, 0, s>>>(A.n, A, dn);
    k_amg_strength<2><<<g1(A.n), 256, 0, s>>>(A.n, A, dn, theta, strong);
  } else {
    k_amg_diag_norm<3><<<g1(A.n), 256, 0, s>>>(A.n, A, dn);
    k_amg_strength<3><<<g1(A.n), 256, 0, s>>>(A.n, A, dn, theta, strong);
  }
  count_launches(2);
  return cudaGetLastError();
}

cudaError_t amg_mis_round(const AmgBsr& A, const unsigned char* strong, int* state, unsigned long long* m1,
                          int* newroot, int* near, int* undecided, cudaStream_t s) {
  const int n = A.n;
  cudaMemsetAsync(undecided, 0, sizeof(int), s);
  k_mis_m1<<<g1(n), 256, 0, s>>>(n, A, strong, state, m1);
  k_mis_root<<<g1(n), 256, 0, s>>>(n, A, strong, state, m1, newroot);
  k_mis_near<<<g1(n), 256, 0, s>>>(n, A, strong, newroot, near);
  k_mis_out<<<g1(n), 256, 0, s>>>(n, A, strong, state, newroot, near, undecided);
  count_launches(4);
  return cudaGetLastError();
}

cudaError_t amg_flag_eq(int n, const int* a, int v, int* f, cudaStream_t s) {
  k_flag_eq<<<g1(n), 256, 0, s>>>(n, a, v, f);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t amg_aggregate(int B, const AmgBsr& A, const unsigned char* strong, const int* state, const int* root_id,
                          int* agg1, int* agg2, cudaStream_t s) {
  const int n = A.n;
  k_agg_phase1<<<g1(n), 256, 0, s>>>(n, A, strong, state, root_id, agg1);
  if (B == 2)
    k_agg_phase2<2><<<g1(n), 256, 0, s>>>(n, A, agg1, agg2);
  else
    k_agg_phase2<3><<<g1(n), 256, 0, s>>>(n, A, agg1, agg2);
  count_launches(2);
  return cudaGetLastError();
}

cudaError_t amg_flag_negative(int n, const int* a, int* f, cudaStream_t s) {
  k_flag_negative<<<g1(n), 256, 0, s>>>(n, a, f);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t amg_phase3(int n, int n_agg, const int* left_id, int* agg, cudaStream_t s) {
  k_agg_phase3<<<g1(n), 256, 0, s>>>(n, n_agg, left_id, agg);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t amg_group(int n, const int* key, int m, int* ptr, int* cnt, int* cur, int* out, int* scan_tmp,
                      cudaStream_t s) {
  cudaMemsetAsync(cnt, 0, sizeof(int) * (size_t)m, s);
  cudaMemsetAsync(cur, 0, sizeof(int) * (size_t)m, s);
  k_count_by<<<g1(n), 256, 0, s>>>(n, key, cnt);
  cudaError_t e = scan_exclusive(cnt, m, ptr, scan_tmp, s);
  if (e != cudaSuccess) return e;
  k_fill_by<<<g1(n), 256, 0, s>>>(n, key, ptr, cur, out);
  k_sort_segments<<<g1(m), 256, 0, s>>>(m, ptr, out);
  count_launches(3);
  return cudaGetLastError();
}

cudaError_t amg_tentative(int B, int n_agg, const int* agg_ptr, const int* members, const double* Bf, double* P0,
                          double* Bc, int* err, cudaStream_t s) {
  if (B == 2)
    k_amg_tentative<2><<<g1((long long)n_agg * kTentLanes, 32 * kTentWarps), 32 * kTentWarps, 0, s>>>(n_agg, agg_ptr, members, Bf, P0, Bc, err);
  else
    k_amg_tentative<3><<<g1((long long)n_agg * kTentLanes, 32 * kTentWarps), 32 * kTentWarps, 0, s>>>(n_agg, agg_ptr, members, Bf, P0, Bc, err);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t amg_lambda_f32(const MixedMatrix* fine, const AmgBsr32* coarse, const double* dinv, double* x, double* y,
                           double* part, double* lam, int iters, cudaStream_t s) {
  const int n = fine ? 2 * fine->n_nodes : 3 * coarse->n;
  double* sc = part + kLamGrid;  // the scale of the next step
  unsigned* ticket = reinterpret_cast<unsigned*>(part + kLamGrid + 1);
  const cudaError_t e = cudaMemsetAsync(ticket, 0, sizeof(unsigned), s);
  if (e != cudaSuccess) return e;
  k_amg_init_vec<<<gw(n), 256, 0, s>>>(n, x);
  // (a block without rows adds an exact zero: small levels leave those out)
  const int grid = std::min(kLamGrid, fine ? g1(fine->n_nodes, kThreads) : g1(coarse->n * 8LL, kThreads));
  for (int t = 0; t < iters; ++t) {
    if (fine)
      k_amg_dinva_fine<<<grid, kThreads, 0, s>>>(*fine, dinv, sc, t == 0, x, y, part, lam, ticket);
    else
      k_amg_dinva_coarse<<<grid, kThreads, 0, s>>>(*coarse, dinv, sc, t == 0, x, y, part, lam, ticket);
    std::swap(x, y);
  }
  k_amg_sweep_coef<<<1, 8, 0, s>>>(lam);
  count_launches(2LL + iters);
  return cudaGetLastError();
}

size_t amg_lambda_scratch() { return sizeof(double) * (kLamGrid + 8); }

cudaError_t amg_p_count(int B, const AmgBsr& A, const int* agg, int* cnt, int* err, cudaStream_t s) {
  if (B == 2)
    k_amg_p_count<2><<<g1(A.n, 128), 128, 0, s>>>(A.n, A, agg, cnt, err);
  else
    k_amg_p_count<3><<<g1(A.n, 128), 128, 0, s>>>(A.n, A, agg, cnt, err);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t amg_p_fill(int B, const AmgBsr& A, const int* agg, const double* P0, const double* dinv, const double* lam,
                       const AmgBsr& P, cudaStream_t s) {
  if (B == 2) {
    k_amg_p_cols<2><<<g1(A.n, 128), 128, 0, s>>>(A.n, A, agg, P);
    k_amg_p_vals<2, 4><<<gal_grid(A.n, 4), 32 * kGalWarps, 0, s>>>(A.n, A, agg, P0, dinv, lam, P);
  } else {
    k_amg_p_cols<3><<<g1(A.n, 128), 128, 0, s>>>(A.n, A, agg, P);
    k_amg_p_vals<3, 8><<<gal_grid(A.n, 8), 32 * kGalWarps, 0, s>>>(A.n, A, agg, P0, dinv, lam, P);
  }
  count_launches(2);
  return cudaGetLastError();
}

cudaError_t amg_ap_count(int B, const AmgBsr& A, const AmgBsr& P, int* cnt, int* err, cudaStream_t s) {
  if (B == 2)
    k_amg_ap_count<2><<<g1(A.n, 128), 128, 0, s>>>(A.n, A, P, cnt, err);
  else
    k_amg_ac_pattern<false><<<ac_grid(A.n), 32 * kAcWarps, 0, s>>>(A.n, A.ptr, A.col, nullptr, P, cnt, AmgBsr{}, err);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t amg_ap_fill(int B, const AmgBsr& A, const AmgBsr& P, const AmgBsr& AP, cudaStream_t s) {
  if (B == 2) {
    k_amg_ap_cols<2><<<g1(A.n, 128), 128, 0, s>>>(A.n, A, P, AP);
    k_amg_ap_vals<2, 8><<<gal_grid(A.n, 8), 32 * kGalWarps, 0, s>>>(A.n, A, P, AP);
  } else {
    k_amg_ac_pattern<true><<<ac_grid(A.n), 32 * kAcWarps, 0, s>>>(A.n, A.ptr, A.col, nullptr, P, nullptr, AP, nullptr);
    k_amg_ap_vals<3, 16><<<gal_grid(A.n, 16), 32 * kGalWarps, 0, s>>>(A.n, A, P, AP);
  }
  count_launches(2);
  return cudaGetLastError();
}

cudaError_t amg_pt(int n, int nc, const AmgBsr& P, int* p_row, int* pt_ptr, int* cnt, int* cur, int* pt_tmp,
                   int* pt_idx, int* scan_tmp, cudaStream_t s) {
  cudaMemsetAsync(cnt, 0, sizeof(int) * (size_t)nc, s);
  cudaMemsetAsync(cur, 0, sizeof(int) * (size_t)nc, s);
  k_p_rows<<<g1(n), 256, 0, s>>>(n, P, p_row);
  k_pt_count<<<g1(n), 256, 0, s>>>(n, P, cnt);
  cudaError_t e = scan_exclusive(cnt, nc, pt_ptr, scan_tmp, s);
  if (e != cudaSuccess) return e;
  k_pt_fill<<<g1(n), 256, 0, s>>>(n, P, pt_ptr, cur, pt_tmp);
  k_rank_pt<<<gw((long long)nc * 32), 256, 0, s>>>(nc, pt_ptr, pt_tmp, pt_idx);
  count_launches(4);
  return cudaGetLastError();
}

cudaError_t amg_ac_count(int B, int nc, const int* pt_ptr, const int* pt_idx, const int* p_row, const AmgBsr& AP,
                         int* cnt, int* err, cudaStream_t s) {
  (void)B;
  k_amg_ac_pattern<false><<<ac_grid(nc), 32 * kAcWarps, 0, s>>>(nc, pt_ptr, pt_idx, p_row, AP, cnt, AmgBsr{}, err);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t amg_ac_fill(int B, int nc, const int* pt_ptr, const int* pt_idx, const int* p_row, const AmgBsr& P,
                        const AmgBsr& AP, const AmgBsr& Ac, cudaStream_t s) {
  k_amg_ac_pattern<true><<<ac_grid(nc), 32 * kAcWarps, 0, s>>>(nc, pt_ptr, pt_idx, p_row, AP, nullptr, Ac, nullptr);
  if (B == 2)
    k_amg_ac_vals<2, 16><<<gal_grid(nc, 16), 32 * kGalWarps, 0, s>>>(nc, pt_ptr, pt_idx, p_row, P, AP, Ac);
  else
    k_amg_ac_vals<3, 32><<<gal_grid(nc, 32), 32 * kGalWarps, 0, s>>>(nc, pt_ptr, pt_idx, p_row, P, AP, Ac);
  count_launches(2);
  return cudaGetLastError();
}

cudaError_t amg_coarsest(int B, const AmgBsr& A, double* M, double* piv, cudaStream_t s) {
  const int n = A.n * B;
  cudaMemsetAsync(M, 0, sizeof(double) * (size_t)n * n, s);
  if (B == 2)
    k_amg_dense<2><<<g1(A.n), 256, 0, s>>>(A.n, A, M);
  else
    k_amg_dense<3><<<g1(A.n), 256, 0, s>>>(A.n, A, M);
  if (n <= kGjMax)
    k_amg_gauss_jordan_regs<<<1, 1024, 0, s>>>(n, M);
  else
    k_amg_gauss_jordan<<<1, 1024, 0, s>>>(n, M, piv);
  count_launches(2);
  return cudaGetLastError();
}

void amg_prepare_launch_shapes() {
  // (the occupancy queries run here, outside any stream capture)
  one_wave((const void*)k_amg_sweep_f32<kSweepResidual>, 1);
  one_wave((const void*)k_amg_sweep_f32<kSweepFirst>, 1);
  one_wave((const void*)k_amg_sweep_f32<kSweepSecond>, 1);
  one_wave((const void*)k_amg_sweep_f32<kSweepSmooth>, 1);
  one_wave((const void*)k_amg_sweep_f32<kSweepSecond, true>, 1);
  one_wave((const void*)k_amg_sweep_f32<kSweepSmooth, true>, 1);
  one_wave((const void*)k_amg_restrict_f32<2>, 1);
  one_wave((const void*)k_amg_prolong_f32<2>, 1);
}

cudaError_t amg_sweep_f32(const int* skip, int mode, int cheb, const MixedMatrix& M, const double* dinv,
                          const double* lam, const double* b, const double* x, const double* xp, double* xo,
                          cudaStream_t s, const FcgDotSink* dots) {
  const long long t = M.n_nodes;
  const FcgDotSink d = dots ? *dots : FcgDotSink{};
  auto go = [&](auto kern) {
    kern<<<one_wave((const void*)kern, t), 256, 0, s>>>(skip, M, dinv, lam, cheb, b, x, xp, xo, d);
  };
  if (dots && mode == kSweepSecond)
    go(k_amg_sweep_f32<kSweepSecond, true>);
  else if (dots && mode == kSweepSmooth)
    go(k_amg_sweep_f32<kSweepSmooth, true>);
  else if (dots)
    return cudaErrorInvalidValue;  // the dots ride on a cycle's last (smoothing) sweep only
  else if (mode == kSweepResidual)
    go(k_amg_sweep_f32<kSweepResidual>);
  else if (mode == kSweepFirst)
    go(k_amg_sweep_f32<kSweepFirst>);
  else if (mode == kSweepSecond)
    go(k_amg_sweep_f32<kSweepSecond>);
  else
    go(k_amg_sweep_f32<kSweepSmooth>);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t amg_sweep3_f32(const int* skip, int mode, int cheb, const AmgBsr32& A, const double* dinv,
                           const double* lam, const double* b, const double* x, const double* xp, double* xo,
                           cudaStream_t s) {
  const int g = gw((long long)A.n * 8);
  switch (mode) {
    case kSweepResidual:
      k_amg_sweep3_f32<kSweepResidual><<<g, 256, 0, s>>>(skip, A, dinv, lam, cheb, b, x, xp, xo);
      break;
    case kSweepFirst: k_amg_sweep3_f32<kSweepFirst><<<g, 256, 0, s>>>(skip, A, dinv, lam, cheb, b, x, xp, xo); break;
    case kSweepSecond: k_amg_sweep3_f32<kSweepSecond><<<g, 256, 0, s>>>(skip, A, dinv, lam, cheb, b, x, xp, xo); break;
    default: k_amg_sweep3_f32<kSweepSmooth><<<g, 256, 0, s>>>(skip, A, dinv, lam, cheb, b, x, xp, xo); break;
  }
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t amg_restrict_f32(const int* skip, int B, int nc, const int* pt_ptr, const int* pt_row, const float* pt32,
                             const double* r, double* bc, const RestrictStart& st, cudaStream_t s) {
  if (B == 2)
    k_amg_restrict_f32<2><<<one_wave((const void*)k_amg_restrict_f32<2>, (long long)nc * 32), 256, 0, s>>>(skip, nc, pt_ptr, pt_row,
                                                                                            pt32, r, bc, st);
  else
    k_amg_restrict_f32<3><<<gw((long long)nc * 32), 256, 0, s>>>(skip, nc, pt_ptr, pt_row, pt32, r, bc, st);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t amg_prolong_f32(const int* skip, int B, int n, const int* p_ptr, const int* p_col, const float* p32,
                            const double* xc, double* x, cudaStream_t s) {
  if (B == 2)
    k_amg_prolong_f32<2><<<one_wave((const void*)k_amg_prolong_f32<2>, n), 256, 0, s>>>(skip, n, p_ptr, p_col, p32, xc, x);
  else
    k_amg_prolong_f32<3><<<gw(n), 256, 0, s>>>(skip, n, p_ptr, p_col, p32, xc, x);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t amg_coarse_f32(const AmgBsr& A, float* val32, cudaStream_t s) {
  k_amg_coarse_f32<<<g1((long long)A.n * 8), 256, 0, s>>>(A, val32);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t amg_transfer_f32(int B, const AmgBsr& P, int nnz_p, const int* pt_idx, const int* p_row, float* p32,
                             int* pt_row, float* pt32, cudaStream_t s) {
  if (nnz_p <= 0) return cudaSuccess;
  if (B == 2)
    k_amg_transfer_f32<2><<<g1(nnz_p), 256, 0, s>>>(nnz_p, P.val, pt_idx, p_row, p32, pt_row, pt32);
  else
    k_amg_transfer_f32<3><<<g1(nnz_p), 256, 0, s>>>(nnz_p, P.val, pt_idx, p_row, p32, pt_row, pt32);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t amg_tail(const int* skip, const AmgTail& t, int cluster, int* max_clusters, cudaStream_t s) {
  if (cluster < 1 || cluster > 16) return cudaErrorInvalidValue;
  if (cluster > 8 && max_clusters) {  // the shape query precedes any launch (never in a capture)
    const cudaError_t e = cudaFuncSetAttribute(k_amg_tail, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)cluster;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)cluster);
  cfg.blockDim = dim3(kAmgTailThreads);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (max_clusters) {
    *max_clusters = 0;
    return cudaOccupancyMaxActiveClusters(max_clusters, (void*)k_amg_tail, &cfg);
  }
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k_amg_tail, skip, t);
  count_launches(1);
  return e;
}

cudaError_t amg_rigid_modes(int N, const double* xy, double* Bf, cudaStream_t s) {
  k_amg_rigid<<<g1(N), 256, 0, s>>>(N, xy, Bf);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t amg_gemv(const int* skip, int n, const double* M, const double* b, double* x, cudaStream_t s) {
  k_amg_gemv<<<gw((long long)n * 32), 256, 0, s>>>(skip, n, M, b, x);
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace cstg
