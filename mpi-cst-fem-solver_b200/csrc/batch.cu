// Batched Jacobi-PCG: many disjoint systems (plates of uneven size) x up to four right-hand
// sides (load cases) in ONE persistent launch of thread-block clusters.
//
// The batch is one block-diagonal matrix (the plates' meshes concatenated, assembled and
// eliminated by the single-system kernels). Each cluster takes the next plate from a queue
// (largest first), solves all of its load cases together, and takes another plate until the
// queue is empty. Inside a plate the cluster's CTAs split the plate's nodes; the reductions of
// a CG iteration (p'Ap; r'z and r'r; the true-residual norms) are summed per CTA, exchanged
// through distributed shared memory after a cluster barrier, and added in CTA-rank order by
// every CTA, so all CTAs take identical decisions and the results are deterministic for a given
// launch shape. No grid-wide barrier and no global-memory spin: clusters never wait on each
// other.
//
// Per load case the recurrence is pcg_iterate's (solver.cpp:35-105) with the FP32
// difference-form operator of mixed_kernels.cu; x, r, p, Ap and every scalar are FP64. Reliable
// updates replace r by the FP64 true residual b - A x once per decade of residual reduction
// (p is kept); when the recursive residual meets rtol the true residual is checked the same way,
// and a load case stops only when the FP64 true residual meets rtol. A plate whose FP32
// operator stops improving the true residual (or fails more checks than max_refinements)
// switches to the FP64 operator with one restart.
//
// Vectors are interleaved per node: [node][load case][2] doubles, so every matrix block is read once
// per iteration for all load cases.
//
// Two kernels. k_batch_halo keeps p of a block's own nodes and of its halo (the neighbours' nodes that
// its rows read) in shared memory for all load cases, forms p = z + beta p there itself, and so needs
// two reductions an iteration and passes only z between blocks; r, Ap and x follow as far as they fit.
// It is bound by the L2 traffic of what does not (x, the matrix) and the shared-memory gathers of p:
// about 35 us an iteration for 20,301 nodes x 4 cases on 8 SMs, against about 100 us for k_batch_pcg, which
// gathers p through L2 and runs three phases (64 plates of n_r 20 .. 100: 166 against 382 ms). The FP32
// blocks are regrouped at a plate's start, the k-th blocks of a warp's 32 rows side by side, so that a load
// is one run of 512 bytes instead of 32 sectors that the small L1 beside the vectors drops before their
// second half is read (177 -> 166 ms). Larger
// plates, whose p does not fit, run faster with all cases on k_batch_pcg than with a case or two
// at a time here (n_r 20 .. 200: 2.1 against 3.6 s), so a batch that holds one goes there as a whole; a
// single plate whose numbering makes its halo too large is put on a list for it.
#include <cooperative_groups.h>

#include "../../include/cstfem_b200.h"
#include "batch_rule.h"
#include "common.cuh"
#include "kernels.h"

#include <algorithm>
#include <cmath>

namespace cg = cooperative_groups;

namespace cstg {

namespace {

// Cluster-wide deterministic sum of V values per thread; the totals land in `tot` (all CTAs).
// wsum holds max(T/32, 16) * V doubles.
template <int V, int T>
__device__ __forceinline__ void cluster_sum(const cg::cluster_group& cl, const double (&v)[V],
                                            double* wsum, double* red, int& buf, double* tot) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const double s = warp_sum(v[i]);
    if (lane == 0) wsum[w * V + i] = s;
  }
  __syncthreads();
  double* mine = red + buf * V;
  if (threadIdx.x < V) {
    double s = 0.0;
#pragma unroll 4
    for (int q = 0; q < T / 32; ++q) s += wsum[q * V + threadIdx.x];
    mine[threadIdx.x] = s;
  }
  cl.sync();  // release/acquire at cluster scope: every CTA's partials (and prior writes) visible
  // Fetch all ranks' partials at once (one remote load per thread), then add them in rank order.
  const unsigned nb = cl.num_blocks();
  if (threadIdx.x < nb * V) wsum[threadIdx.x] = cl.map_shared_rank(mine, threadIdx.x / V)[threadIdx.x % V];
  __syncthreads();
  if (threadIdx.x < V) {
    double s = 0.0;
    for (unsigned q = 0; q < nb; ++q) s += wsum[q * V + threadIdx.x];
    tot[threadIdx.x] = s;
  }
  __syncthreads();
  buf ^= 1;  // the other buffer is next; a cluster barrier separates any two uses of one buffer
}

// Reliable updates: replace r by the FP64 true residual when the recursive r'r has fallen to
// this fraction (0.1^2: one decade of ||r||) of its largest value since the last replacement,
// or after this many iterations without one.
constexpr double kBatchDelta2 = 1e-2;
constexpr int kBatchCycle = 1000;

__device__ __forceinline__ double dot2(double2 a, double2 b, double acc) {
  return fma(a.x, b.x, fma(a.y, b.y, acc));
}

template <int R, int T>
__global__ void __launch_bounds__(T, (T >= 512 ? 1 : 512 / T)) k_batch_pcg(const BatchArgs a) {
  const cg::cluster_group cl = cg::this_cluster();
  const int crank = (int)cl.block_rank(), C = (int)cl.num_blocks();
  constexpr int V = 2 * R;
  __shared__ double wsum[(T / 32 > 16 ? T / 32 : 16) * V];  // warp partials, then <= 16 ranks' partials
  __shared__ double red[2 * V];
  __shared__ double tot[V];
  __shared__ int s_plate, s_limit;
  int buf = 0;
  const double2* __restrict__ invd2 = reinterpret_cast<const double2*>(a.inv_diag);
  const double2* __restrict__ b2 = reinterpret_cast<const double2*>(a.b);
  double2* __restrict__ x2 = reinterpret_cast<double2*>(a.x);
  double2* __restrict__ r2 = reinterpret_cast<double2*>(a.r);
  double2* p2 = reinterpret_cast<double2*>(a.p);  // read by neighbours: always through L2
  double2* __restrict__ Ap2 = reinterpret_cast<double2*>(a.Ap);
  const double2* __restrict__ v64 = reinterpret_cast<const double2*>(a.A64.vals);
  const double rtol2 = a.rtol * a.rtol;

  for (;;) {
    if (crank == 0 && threadIdx.x == 0) {
      const int q = atomicAdd(a.queue + 1, 1);
      s_plate = q < (a.n_rest ? *a.n_rest : a.n_sys) ? (a.n_rest ? a.rest[q] : a.order[q]) : -1;
    }
    cl.sync();
    const int plate = *cl.map_shared_rank(&s_plate, 0);
    if (plate < 0) break;
    const int n0 = a.sys_node[plate], n1 = a.sys_node[plate + 1];
    if (threadIdx.x == 0) s_limit = a.limit[plate];  // (read after the first sums)
    const int first = n0 + crank * T + (int)threadIdx.x, stride = C * T;

    // x = 0, r = b, p = D^-1 b; r'z and b'b per load case (solver.cpp:42-58)
    double v[V];
#pragma unroll
    for (int i = 0; i < V; ++i) v[i] = 0.0;
    for (int n = first; n < n1; n += stride) {
      const double2 d = invd2[n];
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const size_t k = (size_t)n * R + q;
        const double2 bk = b2[k];
        const double2 z = make_double2(d.x * bk.x, d.y * bk.y);
        x2[k] = make_double2(0.0, 0.0);
        r2[k] = bk;
        __stcg(&p2[k], z);
        v[q] = dot2(bk, z, v[q]);
        v[R + q] = dot2(bk, bk, v[R + q]);
      }
    }
    cluster_sum<V, T>(cl, v, wsum, red, buf, tot);

    double rz[R], bn2[R], alpha[R], beta[R], rel[R], true_rel[R], prev_true[R], rmax[R];
    int it[R], nref[R], nfail[R], last_rep[R], status[R];
    unsigned active = 0;
    bool fp64 = a.start_fp64 != 0;
#pragma unroll
    for (int q = 0; q < R; ++q) {
      rz[q] = tot[q];
      bn2[q] = tot[R + q];
      rmax[q] = bn2[q];
      alpha[q] = beta[q] = 0.0;
      it[q] = nref[q] = nfail[q] = last_rep[q] = 0;
      prev_true[q] = INFINITY;
      true_rel[q] = 0.0;
      rel[q] = bn2[q] > 0.0 ? 1.0 : 0.0;
      status[q] = CSTG_SOLVE_CONVERGED;
      if (bn2[q] > 0.0)
        active |= 1u << q;
      else
        status[q] = CSTG_SOLVE_ZERO_RHS;  // x = 0 is exact
    }

    while (active) {
      // ---- Phase A: Ap = A p and p'Ap (all load cases share the matrix read). Neighbours are
      // taken two at a time so both index loads, then all their p loads, are in flight at once.
#pragma unroll
      for (int i = 0; i < V; ++i) v[i] = 0.0;
      for (int n = first; n < n1; n += stride) {
        double2 pn[R], y[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
          pn[q] = __ldcg(&p2[(size_t)n * R + q]);
          y[q] = make_double2(0.0, 0.0);
        }
        if (fp64) {
          const int b0 = __ldg(&a.A64.node_ptr[n]), deg = __ldg(&a.A64.node_ptr[n + 1]) - b0;
          const double2* ra = v64 + 2L * b0;
          const double2* rb = ra + deg;
          for (int k = 0; k < deg; k += 2) {
            const bool two = k + 1 < deg;
            const int m0 = __ldg(&a.A64.bnbr[b0 + k]);
            const int m1 = two ? __ldg(&a.A64.bnbr[b0 + k + 1]) : m0;
            const double2 ka0 = __ldg(ra + k), kb0 = __ldg(rb + k);
            const double2 ka1 = two ? __ldg(ra + k + 1) : make_double2(0.0, 0.0);
            const double2 kb1 = two ? __ldg(rb + k + 1) : make_double2(0.0, 0.0);
            double2 p0[R], p1[R];
#pragma unroll
            for (int q = 0; q < R; ++q) {
              p0[q] = __ldcg(&p2[(size_t)m0 * R + q]);
              p1[q] = __ldcg(&p2[(size_t)m1 * R + q]);
            }
#pragma unroll
            for (int q = 0; q < R; ++q) {
              y[q].x = dot2(ka1, p1[q], dot2(ka0, p0[q], y[q].x));
              y[q].y = dot2(kb1, p1[q], dot2(kb0, p0[q], y[q].y));
            }
          }
        } else {
          const int bb = __ldg(&a.A32.node_ptr[n]);
          const int o = bb - n, c = __ldg(&a.A32.node_ptr[n + 1]) - bb - 1;
          for (int k = 0; k < c; k += 2) {
            const bool two = k + 1 < c;
            const int m0 = __ldg(&a.A32.nbr32[o + k]);
            const int m1 = two ? __ldg(&a.A32.nbr32[o + k + 1]) : n;
            const float4 f0 = __ldg(&a.A32.val32[o + k]);
            const float4 f1 = two ? __ldg(&a.A32.val32[o + k + 1]) : make_float4(0.f, 0.f, 0.f, 0.f);
            double2 p0[R], p1[R];
#pragma unroll
            for (int q = 0; q < R; ++q) {
              p0[q] = __ldcg(&p2[(size_t)m0 * R + q]);
              p1[q] = __ldcg(&p2[(size_t)m1 * R + q]);
            }
#pragma unroll
            for (int q = 0; q < R; ++q) {
              const double dx0 = p0[q].x - pn[q].x, dy0 = p0[q].y - pn[q].y;
              const double dx1 = p1[q].x - pn[q].x, dy1 = p1[q].y - pn[q].y;
              y[q].x = fma((double)f0.x, dx0, fma((double)f0.y, dy0, y[q].x));
              y[q].y = fma((double)f0.z, dx0, fma((double)f0.w, dy0, y[q].y));
              y[q].x = fma((double)f1.x, dx1, fma((double)f1.y, dy1, y[q].x));
              y[q].y = fma((double)f1.z, dx1, fma((double)f1.w, dy1, y[q].y));
            }
          }
          const double2 sa = __ldg(&a.A32.S64[2 * n]), sb = __ldg(&a.A32.S64[2 * n + 1]);
#pragma unroll
          for (int q = 0; q < R; ++q) {
            y[q].x = dot2(sa, pn[q], y[q].x);
            y[q].y = dot2(sb, pn[q], y[q].y);
          }
        }
#pragma unroll
        for (int q = 0; q < R; ++q) {
          Ap2[(size_t)n * R + q] = y[q];
          v[q] = dot2(pn[q], y[q], v[q]);
        }
      }
      cluster_sum<V, T>(cl, v, wsum, red, buf, tot);
#pragma unroll
      for (int q = 0; q < R; ++q) {
        if (!((active >> q) & 1u)) continue;
        const double pAp = tot[q];
        if (!(pAp > 0.0)) {  // solver.cpp:64-68
          status[q] = CSTG_SOLVE_BREAKDOWN;
          active &= ~(1u << q);
          alpha[q] = 0.0;
        } else {
          alpha[q] = rz[q] / pAp;
        }
      }
      if (!active) break;

      // ---- Phase B: x += alpha p, r -= alpha Ap; r'z and r'r. All loads of a node are issued
      // before any store (stores of finished cases are skipped), so its 4R loads fly together.
#pragma unroll
      for (int i = 0; i < V; ++i) v[i] = 0.0;
#pragma unroll 2
      for (int n = first; n < n1; n += stride) {
        const double2 d = invd2[n];
        double2 pk[R], apk[R], xk[R], rk[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
          const size_t k = (size_t)n * R + q;
          pk[q] = __ldcg(&p2[k]);
          apk[q] = Ap2[k];
          xk[q] = x2[k];
          rk[q] = r2[k];
        }
#pragma unroll
        for (int q = 0; q < R; ++q) {
          xk[q].x = fma(alpha[q], pk[q].x, xk[q].x);
          xk[q].y = fma(alpha[q], pk[q].y, xk[q].y);
          rk[q].x = fma(-alpha[q], apk[q].x, rk[q].x);
          rk[q].y = fma(-alpha[q], apk[q].y, rk[q].y);
          if ((active >> q) & 1u) {
            const size_t k = (size_t)n * R + q;
            x2[k] = xk[q];
            r2[k] = rk[q];
          }
          v[q] = fma(rk[q].x, d.x * rk[q].x, fma(rk[q].y, d.y * rk[q].y, v[q]));
          v[R + q] = dot2(rk[q], rk[q], v[R + q]);
        }
      }
      cluster_sum<V, T>(cl, v, wsum, red, buf, tot);
      // Which load cases need the FP64 true residual now: a convergence check (the recursive
      // residual met rtol, or max_iter), or a reliable update (the recursive residual fell by
      // kBatchDelta2 since the largest one after the last update, or kBatchCycle iterations
      // passed). A reliable update replaces r and keeps p (van der Vorst and Ye's scheme).
      unsigned check = 0, repl = 0;
#pragma unroll
      for (int q = 0; q < R; ++q) {
        if (!((active >> q) & 1u)) continue;
        ++it[q];
        const double rr = tot[R + q];
        rel[q] = sqrt(rr / bn2[q]);
        rmax[q] = fmax(rmax[q], rr);
        if (rr <= rtol2 * bn2[q] || it[q] >= s_limit) {
          check |= 1u << q;
        } else if (rr <= kBatchDelta2 * rmax[q] || it[q] - last_rep[q] >= kBatchCycle) {
          repl |= 1u << q;
        } else {
          beta[q] = tot[q] / rz[q];
          rz[q] = tot[q];
        }
      }
      repl |= check;

      if (repl) {
        // ---- Phase R: FP64 true residual r = b - A x for the replaced load cases
#pragma unroll
        for (int i = 0; i < V; ++i) v[i] = 0.0;
        for (int n = first; n < n1; n += stride) {
          const double2 d = invd2[n];
          const int b0 = __ldg(&a.A64.node_ptr[n]), deg = __ldg(&a.A64.node_ptr[n + 1]) - b0;
          const double2* ra = v64 + 2L * b0;
          const double2* rb = ra + deg;
          double2 t[R];
#pragma unroll
          for (int q = 0; q < R; ++q) t[q] = make_double2(0.0, 0.0);
          for (int k = 0; k < deg; ++k) {
            const int m = __ldg(&a.A64.bnbr[b0 + k]);
            const double2 ka = __ldg(ra + k), kb = __ldg(rb + k);
#pragma unroll
            for (int q = 0; q < R; ++q) {
              if (!((repl >> q) & 1u)) continue;
              const double2 xm = __ldcg(&x2[(size_t)m * R + q]);
              t[q].x = dot2(ka, xm, t[q].x);
              t[q].y = dot2(kb, xm, t[q].y);
            }
          }
#pragma unroll
          for (int q = 0; q < R; ++q) {
            if (!((repl >> q) & 1u)) continue;
            const size_t k = (size_t)n * R + q;
            const double2 bk = b2[k];
            const double2 rk = make_double2(bk.x - t[q].x, bk.y - t[q].y);
            r2[k] = rk;
            v[q] = dot2(rk, rk, v[q]);
            v[R + q] = fma(rk.x, d.x * rk.x, fma(rk.y, d.y * rk.y, v[R + q]));
          }
        }
        cluster_sum<V, T>(cl, v, wsum, red, buf, tot);
        bool restart = false;
#pragma unroll
        for (int q = 0; q < R; ++q) {
          if (!((repl >> q) & 1u)) continue;
          const double rr = tot[q], tr = sqrt(rr / bn2[q]);
          true_rel[q] = tr;
          const bool is_check = (check >> q) & 1u;
          if (is_check && rr <= rtol2 * bn2[q]) {
            status[q] = CSTG_SOLVE_CONVERGED;
            active &= ~(1u << q);
            continue;
          }
          if (it[q] >= s_limit) {
            status[q] = CSTG_SOLVE_MAX_ITER;
            active &= ~(1u << q);
            continue;
          }
          ++nref[q];
          last_rep[q] = it[q];
          rmax[q] = rr;
          rel[q] = tr;
          if (is_check) {  // the recursive residual met rtol but the true one did not
            ++nfail[q];
            if (!fp64 && (nfail[q] > a.max_refine || tr > 0.5 * prev_true[q])) {
              fp64 = true;  // the FP32 operator's accuracy floor: FP64 from here, restarted
              restart = true;
            }
            prev_true[q] = tr;
          }
          beta[q] = tot[R + q] / rz[q];
          rz[q] = tot[R + q];
        }
        if (restart)
#pragma unroll
          for (int q = 0; q < R; ++q) beta[q] = 0.0;
      }

      // ---- Phase C: p = D^-1 r + beta p
      if (active) {
#pragma unroll 2
        for (int n = first; n < n1; n += stride) {
          const double2 d = invd2[n];
          double2 rk[R], pk[R];
#pragma unroll
          for (int q = 0; q < R; ++q) {
            const size_t k = (size_t)n * R + q;
            rk[q] = r2[k];
            pk[q] = __ldcg(&p2[k]);
          }
#pragma unroll
          for (int q = 0; q < R; ++q)
            if ((active >> q) & 1u)
              __stcg(&p2[(size_t)n * R + q], make_double2(fma(beta[q], pk[q].x, d.x * rk[q].x),
                                                          fma(beta[q], pk[q].y, d.y * rk[q].y)));
        }
      }
      cl.sync();  // Phase C's p visible to the neighbours' CTAs before the next SpMV
    }

    if (crank == 0 && threadIdx.x == 0) {
#pragma unroll
      for (int q = 0; q < R; ++q) {
        BatchResultDev o;
        o.iterations = it[q];
        o.status = status[q];
        o.refinements = nref[q];
        o.fp64 = fp64 ? 1 : 0;
        o.rel = rel[q];
        o.true_rel = true_rel[q];
        a.res[(size_t)plate * a.res_stride + a.res_offset + q] = o;
      }
    }
  }
  cl.sync();  // no CTA leaves while another may still read its shared memory
}

// ---- plates whose p fits in shared memory ----------------------------------------------------------

constexpr int kHaloHash = 8192;  // slots of the halo's hash set; a halo holds at most half as many

template <int R, int T>
struct HaloShared {
  double wsum[T / 32][2 * R];
  double inbox[2][16][2 * R];  // every block's sums, double-buffered
  double alpha[R], beta[R], xalpha[R];  // xalpha: step of x not yet taken
  // per load case, kept by lane q of warp 0 (the same values in every block)
  double rz[R], bn2[R], rel[R], true_rel[R], prev_true[R], rmax[R];
  int it[R], nref[R], nfail[R], last_rep[R], status[R];
  unsigned active, repl;
  int fp64, plate, halo;
  int scan[T / 32];
};

// Cluster-wide sums of V values per thread: lane i < V of warp 0 gets sum i (the others nothing). The
// values are halved over the lanes on the way down, so a warp adds 7 + 2 numbers instead of 8 x 5.
template <int V, int R, int T>
__device__ __forceinline__ double cluster_totals(const cg::cluster_group& cl, HaloShared<R, T>& sh, unsigned& seq,
                                                 const double (&v)[V]) {
  constexpr int P = V <= 2 ? 2 : V <= 4 ? 4 : 8, kPart = 32 / P;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int idx = lane / kPart, part = lane % kPart;
  double a[P];
#pragma unroll
  for (int j = 0; j < P; ++j) a[j] = j < V ? v[j] : 0.0;
  int o = 16;
#pragma unroll
  for (int h = P / 2; h > 0; h >>= 1, o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int j = 0; j < h; ++j) {
      const double give = up ? a[j] : a[j + h];
      a[j] = (up ? a[j + h] : a[j]) + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
#pragma unroll
  for (int k = kPart / 2; k > 0; k >>= 1) a[0] += __shfl_xor_sync(0xffffffffu, a[0], k);
  if (part == 0 && idx < V) sh.wsum[w][idx] = a[0];
  ++seq;
  __syncthreads();
  const int C = (int)cl.num_blocks();
  double(*box)[2 * R] = sh.inbox[seq & 1u];
  if (w == 0) {
    double s = 0.0;
    if (idx < V)
      for (int k = part; k < T / 32; k += kPart) s += sh.wsum[k][idx];
#pragma unroll
    for (int k = kPart / 2; k > 0; k >>= 1) s += __shfl_xor_sync(0xffffffffu, s, k);
    if (idx < V)
      for (int c = part; c < C; c += kPart) *cl.map_shared_rank(&box[cl.block_rank()][idx], c) = s;
  }
  cl.sync();  // release / acquire at cluster scope: sums and vectors
  double s = 0.0;
  if (w == 0) {
    if (idx < V)
      for (int c = part; c < C; c += kPart) s += box[c][idx];
#pragma unroll
    for (int k = kPart / 2; k > 0; k >>= 1) s += __shfl_xor_sync(0xffffffffu, s, k);
    s = __shfl_sync(0xffffffffu, s, (lane * kPart) & 31);
  }
  return s;
}

// A block's own vector of G load cases: [node][case] (IT) or [case][node], the first `lim` nodes in
// shared memory, the others in the interleaved global array.
template <int G, bool IT>
struct OwnCases {
  double2* s;
  double2* g;      // at the block's first node
  int lim, pitch;  // (pitch of a case in shared memory)
  __device__ __forceinline__ double2& at(int i, int q) const {
    return i < lim ? s[IT ? i * G + q : q * pitch + i] : g[(size_t)i * G + q];
  }
};

// Slots of a case's array: a multiple of 8 plus 8 / G, so that the 8 lanes of a shared-memory phase
// that hold consecutive (node, case) items hit different banks.
template <int G>
__device__ __forceinline__ int case_pitch(int n) {
  return (n + 7) / 8 * 8 + (G == 1 ? 0 : 8 / G);
}

// The place of the k-th off-diagonal block of each lane's row among the regrouped blocks of a warp's 32
// nodes (all first blocks, all second blocks, ...): `run` is the next free place, c the row's blocks (0: no
// row). A lane without a k-th block gets a valid place.
__device__ __forceinline__ int lane_place(int& run, int k, int c, int lane) {
  const unsigned on = __ballot_sync(0xffffffffu, k < c);
  const int at = run + __popc(on & ((1u << lane) - 1u));
  run += __popc(on);
  return k < c ? at : run - 1;
}

// All load cases of a plate; dyn: shared memory from the end of the halo's list on.
template <int R, int T>
__device__ __forceinline__ void solve_cases(const BatchArgs& a, const cg::cluster_group& cl, HaloShared<R, T>& sh,
                                            unsigned& seq, unsigned char* dyn, unsigned smem, int n0,
                                            int cnt, int nh, const int* hid, const unsigned* want, int plate) {
  constexpr int G = R, V = 2 * G;
  constexpr int kItems = T / G * G;  // threads of the item loops: a thread keeps its load case
  const int tid = threadIdx.x, lane = tid & 31;
  const int tq = tid % G, tn = tid < kItems ? tid / G : 1 << 30;
  constexpr int kStep = T / G;
  const double2* __restrict__ invd2 = reinterpret_cast<const double2*>(a.inv_diag) + n0;
  const double2* __restrict__ v64 = reinterpret_cast<const double2*>(a.A64.vals);
  const double rtol2 = a.rtol * a.rtol;
  const int limit = __ldg(&a.limit[plate]);
  const size_t base = (size_t)n0 * R;
  double2* zg = reinterpret_cast<double2*>(a.p);  // z of wanted nodes, in p's array
  const double2* bg = reinterpret_cast<const double2*>(a.b) + base;

  unsigned used = 0;
  const int pitch = case_pitch<G>(cnt + nh);
  double2* p = reinterpret_cast<double2*>(dyn);
  used += (unsigned)pitch * G * 16u;
  auto room = [&]() { return smem > used ? (int)min((smem - used) / (16u * G), (unsigned)cnt) : 0; };
  OwnCases<G, true> r, x;
  OwnCases<G, false> Ap;
  r.g = reinterpret_cast<double2*>(a.r) + base;
  x.g = reinterpret_cast<double2*>(a.x) + base;
  Ap.g = reinterpret_cast<double2*>(a.Ap) + base;
  r.pitch = x.pitch = 0;
  r.lim = room();
  r.s = reinterpret_cast<double2*>(dyn + used);
  used += (unsigned)r.lim * G * 16u;
  Ap.lim = max(0, room() - 16);
  Ap.pitch = case_pitch<G>(Ap.lim);
  Ap.s = reinterpret_cast<double2*>(dyn + used);
  if (Ap.lim > 0) used += (unsigned)Ap.pitch * G * 16u;
  x.lim = room();
  x.s = reinterpret_cast<double2*>(dyn + used);

  // x = 0, r = b, p = D^-1 b; r'z and b'b per load case (solver.cpp:42-58)
  double v[V];
#pragma unroll
  for (int i = 0; i < V; ++i) v[i] = 0.0;
  double s0 = 0.0, s1 = 0.0;
  for (int i = tn; i < cnt; i += kStep) {
    const double2 d = invd2[i], bk = bg[(size_t)i * R + tq];
    const double2 z = make_double2(d.x * bk.x, d.y * bk.y);
    x.at(i, tq) = make_double2(0.0, 0.0);
    r.at(i, tq) = bk;
    p[tq * pitch + i] = z;
    s0 = dot2(bk, z, s0);
    s1 = dot2(bk, bk, s1);
  }
  for (int j = tn; j < nh; j += kStep) {
    const int m = hid[j];
    const double2 d = reinterpret_cast<const double2*>(a.inv_diag)[m];
    const double2 bk = reinterpret_cast<const double2*>(a.b)[(size_t)m * R + tq];
    p[tq * pitch + cnt + j] = make_double2(d.x * bk.x, d.y * bk.y);
  }
#pragma unroll
  for (int q = 0; q < G; ++q) {
    v[q] = q == tq ? s0 : 0.0;
    v[G + q] = q == tq ? s1 : 0.0;
  }
  {
    const double t = cluster_totals<V>(cl, sh, seq, v);
    const double t2 = __shfl_sync(0xffffffffu, t, (lane + G) & 31);
    if (tid < 32) {
      const bool mine = lane < G;
      if (mine) {
        sh.rz[lane] = t;
        sh.bn2[lane] = sh.rmax[lane] = t2;
        sh.alpha[lane] = sh.beta[lane] = sh.xalpha[lane] = 0.0;
        sh.it[lane] = sh.nref[lane] = sh.nfail[lane] = sh.last_rep[lane] = 0;
        sh.prev_true[lane] = INFINITY;
        sh.true_rel[lane] = 0.0;
        sh.rel[lane] = t2 > 0.0 ? 1.0 : 0.0;
        sh.status[lane] = t2 > 0.0 ? CSTG_SOLVE_CONVERGED : CSTG_SOLVE_ZERO_RHS;  // x = 0 is exact
      }
      const unsigned act = __ballot_sync(0xffffffffu, mine && t2 > 0.0);
      if (lane == 0) {
        sh.active = act;
        sh.fp64 = a.start_fp64 != 0;
      }
    }
    __syncthreads();
  }

  for (bool begun = false; sh.active; begun = true) {
    // ---- Phase 1: the step of x of the iteration before, p = z + beta p at own nodes and halo
    if (begun) {
      const double beta = sh.beta[tq], xa = sh.xalpha[tq];
      if ((sh.active >> tq) & 1u) {
        constexpr int kU = 4;
        for (int j0 = tn; j0 < nh; j0 += kU * kStep) {
          double2 z[kU];
#pragma unroll
          for (int u = 0; u < kU; ++u)
            z[u] = __ldcg(&zg[(size_t)hid[min(j0 + u * kStep, nh - 1)] * R + tq]);
#pragma unroll
          for (int u = 0; u < kU; ++u) {
            const int j = j0 + u * kStep;
            if (j >= nh) break;
            double2& pj = p[tq * pitch + cnt + j];
            pj = make_double2(fma(beta, pj.x, z[u].x), fma(beta, pj.y, z[u].y));
          }
        }
        for (int i0 = tn; i0 < cnt; i0 += kU * kStep) {
          double2 xi[kU], ri[kU], di[kU];
#pragma unroll
          for (int u = 0; u < kU; ++u) {
            const int i = min(i0 + u * kStep, cnt - 1);
            xi[u] = x.at(i, tq);
            ri[u] = r.at(i, tq);
            di[u] = __ldg(&invd2[i]);
          }
#pragma unroll
          for (int u = 0; u < kU; ++u) {
            const int i = i0 + u * kStep;
            if (i >= cnt) break;
            double2& pi = p[tq * pitch + i];
            x.at(i, tq) = make_double2(fma(xa, pi.x, xi[u].x), fma(xa, pi.y, xi[u].y));
            pi = make_double2(fma(beta, pi.x, di[u].x * ri[u].x), fma(beta, pi.y, di[u].y * ri[u].y));
          }
        }
      }
      __syncthreads();
    }
    // Ap = A p and p'Ap: a thread per node, all load cases (the matrix row is read once)
#pragma unroll
    for (int i = 0; i < V; ++i) v[i] = 0.0;
    double pap[G];
#pragma unroll
    for (int q = 0; q < G; ++q) pap[q] = 0.0;
    const bool fp64 = sh.fp64 != 0;
    for (int i0 = tid - lane; i0 < cnt; i0 += T) {
      const bool on = i0 + lane < cnt;  // (a lane past the end repeats the last row, and adds nothing)
      const int i = on ? i0 + lane : cnt - 1;
      const int n = n0 + i;
      const int b0 = __ldg(&a.A64.node_ptr[n]), deg = __ldg(&a.A64.node_ptr[n + 1]) - b0;
      const unsigned short* sl = a.slots + (b0 - n);
      double2 y[G], pn[G];
#pragma unroll
      for (int q = 0; q < G; ++q) {
        y[q] = make_double2(0.0, 0.0);
        pn[q] = p[q * pitch + i];
      }
      if (fp64) {
        const double2 *ra = v64 + 2L * b0, *rb = ra + deg;
        int off = 0;  // slots are of the off-diagonal blocks only
        for (int k = 0; k < deg; ++k) {
          const int slot = __ldg(&a.A64.bnbr[b0 + k]) == n ? i : (int)sl[off++];
          const double2 ka = __ldg(ra + k), kb = __ldg(rb + k);
#pragma unroll
          for (int q = 0; q < G; ++q) {
            const double2 pm = p[q * pitch + slot];
            y[q].x = dot2(ka, pm, y[q].x);
            y[q].y = dot2(kb, pm, y[q].y);
          }
        }
      } else {
        const int c = on ? deg - 1 : 0;
        const int longest = __reduce_max_sync(0xffffffffu, c);
        int run = __shfl_sync(0xffffffffu, b0 - n, 0);
        constexpr int kN = 3;  // neighbours whose matrix loads are in flight together
        for (int k0 = 0; k0 < longest; k0 += kN) {
          int slot[kN];
          float4 f[kN];
#pragma unroll
          for (int u = 0; u < kN; ++u) {
            const int at = lane_place(run, k0 + u, c, lane);
            const int to = (int)__ldcg(&a.lane_slots[at]);
            f[u] = __ldcg(&a.lane_vals[at]);
            slot[u] = k0 + u < c ? to : i;  // (the node itself: a zero difference)
          }
#pragma unroll
          for (int u = 0; u < kN; ++u) {
#pragma unroll
            for (int q = 0; q < G; ++q) {
              const double2 pm = p[q * pitch + slot[u]];
              const double dx = pm.x - pn[q].x, dy = pm.y - pn[q].y;
              y[q].x = fma((double)f[u].x, dx, fma((double)f[u].y, dy, y[q].x));
              y[q].y = fma((double)f[u].z, dx, fma((double)f[u].w, dy, y[q].y));
            }
          }
        }
        const double2 sa = __ldg(&a.A32.S64[2 * n]), sb = __ldg(&a.A32.S64[2 * n + 1]);
#pragma unroll
        for (int q = 0; q < G; ++q) {
          y[q].x = dot2(sa, pn[q], y[q].x);
          y[q].y = dot2(sb, pn[q], y[q].y);
        }
      }
#pragma unroll
      for (int q = 0; q < G; ++q) {
        if (!on) break;
        Ap.at(i, q) = y[q];
        pap[q] = dot2(pn[q], y[q], pap[q]);
      }
    }
    {
      const double t = cluster_totals<G>(cl, sh, seq, pap);
      if (tid < 32) {
        bool on = false;
        if (lane < G) {
          on = (sh.active >> lane) & 1u;
          if (on && !(t > 0.0)) {  // solver.cpp:64-68
            sh.status[lane] = CSTG_SOLVE_BREAKDOWN;
            on = false;
          }
          sh.alpha[lane] = sh.xalpha[lane] = on ? sh.rz[lane] / t : 0.0;
        }
        const unsigned act = __ballot_sync(0xffffffffu, on);
        if (lane == 0) sh.active = act;
      }
      __syncthreads();
    }
    if (!sh.active) break;

    // ---- Phase 2: r -= alpha Ap, z = D^-1 r; r'z and r'r
    {
      const double alpha = sh.alpha[tq];
      s0 = s1 = 0.0;
      constexpr int kU = 4;
      if ((sh.active >> tq) & 1u)
        for (int i0 = tn; i0 < cnt; i0 += kU * kStep) {
          double2 ri[kU], di[kU];
#pragma unroll
          for (int u = 0; u < kU; ++u) {
            const int i = min(i0 + u * kStep, cnt - 1);
            const double2 ai = Ap.at(i, tq);
            ri[u] = r.at(i, tq);
            ri[u] = make_double2(fma(-alpha, ai.x, ri[u].x), fma(-alpha, ai.y, ri[u].y));
            di[u] = __ldg(&invd2[i]);
          }
#pragma unroll
          for (int u = 0; u < kU; ++u) {
            const int i = i0 + u * kStep;
            if (i >= cnt) break;
            const double2 z = make_double2(di[u].x * ri[u].x, di[u].y * ri[u].y);
            r.at(i, tq) = ri[u];
            if ((want[i >> 5] >> (i & 31)) & 1u) __stcg(&zg[(size_t)(n0 + i) * R + tq], z);
            s0 = dot2(ri[u], z, s0);
            s1 = dot2(ri[u], ri[u], s1);
          }
        }
#pragma unroll
      for (int q = 0; q < G; ++q) {
        v[q] = q == tq ? s0 : 0.0;
        v[G + q] = q == tq ? s1 : 0.0;
      }
      const double t = cluster_totals<V>(cl, sh, seq, v);
      const double rr = __shfl_sync(0xffffffffu, t, (lane + G) & 31);
      if (tid < 32) {
        // Which load cases need the FP64 true residual now (see k_batch_pcg): a convergence check or
        // a reliable update; the others go on with beta.
        bool chk = false, rep = false;
        if (lane < G && ((sh.active >> lane) & 1u)) {
          const int it = ++sh.it[lane];
          sh.rel[lane] = sqrt(rr / sh.bn2[lane]);
          const double rm = fmax(sh.rmax[lane], rr);
          sh.rmax[lane] = rm;
          if (rr <= rtol2 * sh.bn2[lane] || it >= limit) {
            chk = true;
          } else if (rr <= kBatchDelta2 * rm || it - sh.last_rep[lane] >= kBatchCycle) {
            rep = true;
          } else {
            sh.beta[lane] = t / sh.rz[lane];
            sh.rz[lane] = t;
          }
        }
        const unsigned c = __ballot_sync(0xffffffffu, chk), m = __ballot_sync(0xffffffffu, rep);
        if (lane == 0) sh.repl = (c | m) | c << 16;
      }
      __syncthreads();
    }
    const unsigned repl = sh.repl & 0xffffu, check = sh.repl >> 16;
    if (repl) {
      // ---- Phase R: FP64 true residual r = b - A x for the replaced load cases
      if ((repl >> tq) & 1u) {
        const double xa = sh.xalpha[tq];
        for (int i = tn; i < cnt; i += kStep) {
          const double2 pi = p[tq * pitch + i];
          double2 xi = x.at(i, tq);
          xi = make_double2(fma(xa, pi.x, xi.x), fma(xa, pi.y, xi.y));
          x.at(i, tq) = xi;
          __stcg(&x.g[(size_t)i * R + tq], xi);
        }
      }
      cl.sync();  // x visible to the other blocks
      if (tid < G && ((repl >> tid) & 1u)) sh.xalpha[tid] = 0.0;
#pragma unroll
      for (int i = 0; i < V; ++i) v[i] = 0.0;
      for (int i = tid; i < cnt; i += T) {
        const int n = n0 + i;
        const double2 d = invd2[i];
        const int b0 = __ldg(&a.A64.node_ptr[n]), deg = __ldg(&a.A64.node_ptr[n + 1]) - b0;
        const double2 *ra = v64 + 2L * b0, *rb = ra + deg;
        double2 t[G];
#pragma unroll
        for (int q = 0; q < G; ++q) t[q] = make_double2(0.0, 0.0);
        for (int k = 0; k < deg; ++k) {
          const int m = __ldg(&a.A64.bnbr[b0 + k]);
          const double2 ka = __ldg(ra + k), kb = __ldg(rb + k);
#pragma unroll
          for (int q = 0; q < G; ++q) {
            if (!((repl >> q) & 1u)) continue;
            const double2 xm = __ldcg(reinterpret_cast<const double2*>(a.x) + (size_t)m * R + q);
            t[q].x = dot2(ka, xm, t[q].x);
            t[q].y = dot2(kb, xm, t[q].y);
          }
        }
#pragma unroll
        for (int q = 0; q < G; ++q) {
          if (!((repl >> q) & 1u)) continue;
          const double2 bk = bg[(size_t)i * R + q];
          const double2 rk = make_double2(bk.x - t[q].x, bk.y - t[q].y);
          const double2 z = make_double2(d.x * rk.x, d.y * rk.y);
          r.at(i, q) = rk;
          if ((want[i >> 5] >> (i & 31)) & 1u) __stcg(&zg[(size_t)n * R + q], z);
          v[q] = dot2(rk, rk, v[q]);
          v[G + q] = dot2(rk, z, v[G + q]);
        }
      }
      const double rr = cluster_totals<V>(cl, sh, seq, v);
      const double rzn = __shfl_sync(0xffffffffu, rr, (lane + G) & 31);
      if (tid < 32) {
        bool off = false, restart = false;
        if (lane < G && ((repl >> lane) & 1u)) {
          const bool is_check = (check >> lane) & 1u;
          const double tr = sqrt(rr / sh.bn2[lane]);
          sh.true_rel[lane] = tr;
          if (is_check && rr <= rtol2 * sh.bn2[lane]) {
            sh.status[lane] = CSTG_SOLVE_CONVERGED;
            off = true;
          } else if (sh.it[lane] >= limit) {
            sh.status[lane] = CSTG_SOLVE_MAX_ITER;
            off = true;
          } else {
            ++sh.nref[lane];
            sh.last_rep[lane] = sh.it[lane];
            sh.rmax[lane] = rr;
            sh.rel[lane] = tr;
            if (is_check) {  // the recursive residual met rtol but the true one did not
              ++sh.nfail[lane];
              // the FP32 operator's accuracy floor: FP64 from here, restarted
              restart = !fp64 && (sh.nfail[lane] > a.max_refine || tr > 0.5 * sh.prev_true[lane]);
              sh.prev_true[lane] = tr;
            }
            sh.beta[lane] = rzn / sh.rz[lane];
            sh.rz[lane] = rzn;
          }
        }
        const unsigned gone = __ballot_sync(0xffffffffu, off), again = __ballot_sync(0xffffffffu, restart);
        if (again && lane < G) sh.beta[lane] = 0.0;
        if (lane == 0) {
          sh.active &= ~gone;
          if (again) sh.fp64 = 1;
        }
      }
      __syncthreads();
    }
  }

  // x of the load cases that did not end in a check (breakdown: the step before is already in)
  for (int i = tn; i < cnt; i += kStep)
    if (i < x.lim) x.g[(size_t)i * R + tq] = x.s[i * G + tq];
  if (cl.block_rank() == 0 && tid < G) {
    BatchResultDev o;
    o.iterations = sh.it[tid];
    o.status = sh.status[tid];
    o.refinements = sh.nref[tid];
    o.fp64 = sh.fp64 != 0;
    o.rel = sh.rel[tid];
    o.true_rel = sh.true_rel[tid];
    a.res[(size_t)plate * a.res_stride + a.res_offset + tid] = o;
  }
  __syncthreads();
}

template <int R, int T>
__global__ void __launch_bounds__(T, 1) k_batch_halo(const BatchArgs a) {
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ HaloShared<R, T> sh;
  const cg::cluster_group cl = cg::this_cluster();
  const int crank = (int)cl.block_rank(), C = (int)cl.num_blocks();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned seq = 0;
  for (;;) {
    if (crank == 0 && tid == 0) {
      const int q = atomicAdd(a.queue, 1);
      sh.plate = q < a.n_sys ? a.order[q] : -1;
    }
    cl.sync();
    const int plate = *cl.map_shared_rank(&sh.plate, 0);
    if (plate < 0) break;
    const int p0 = a.sys_node[plate], np = a.sys_node[plate + 1] - p0;
    const int n0 = p0 + (int)((long long)np * crank / C), n1 = p0 + (int)((long long)np * (crank + 1) / C);
    const int cnt = n1 - n0;

    // -- the halo: nodes outside [n0, n1) among the rows' neighbours, in a hash set keyed by their low
    // bits (so the compacted list keeps runs of consecutive nodes together)
    int* hid = reinterpret_cast<int*>(dyn);
    int* keys = reinterpret_cast<int*>(dyn + a.smem) - kHaloHash;
    unsigned short* slot = reinterpret_cast<unsigned short*>(keys) - kHaloHash;
    const int e0 = cnt > 0 ? a.A64.node_ptr[n0] : 0, e1 = cnt > 0 ? a.A64.node_ptr[n1] : 0;
    const int want_words = (cnt + 31) / 32;
    for (int i = tid; i < kHaloHash; i += T) keys[i] = -1;
    if (tid == 0) sh.halo = 0;
    __syncthreads();
    volatile int* count = &sh.halo;
    for (int e = e0 + tid; e < e1 && *count <= kHaloHash / 2; e += T) {
      const int m = a.A64.bnbr[e];
      if (m >= n0 && m < n1) continue;
      for (int h = m & (kHaloHash - 1);; h = (h + 1) & (kHaloHash - 1)) {
        const int k = atomicCAS(&keys[h], -1, m);
        if (k == -1) atomicAdd(&sh.halo, 1);
        if (k == -1 || k == m) break;
      }
    }
    __syncthreads();
    const int nh = sh.halo;
    // p of all load cases must fit beside the halo's list and the wanted bits, in every block
    const unsigned head = (((unsigned)nh + (unsigned)want_words) * 4u + 15u) & ~15u;
    const bool fits = nh <= kHaloHash / 2 && cnt + nh <= 65535 &&
                      (long long)head + 16LL * R * case_pitch<R>(cnt + nh) <= (long long)a.smem;
    bool all = true;
    ++seq;
    if (tid < C) *cl.map_shared_rank(&sh.inbox[seq & 1u][crank][0], tid) = fits ? 1.0 : 0.0;
    cl.sync();
    for (int c = 0; c < C; ++c) all &= sh.inbox[seq & 1u][c][0] != 0.0;
    if (!all) {
      if (crank == 0 && tid == 0) a.rest[atomicAdd(a.n_rest, 1)] = plate;
      continue;
    }
    {
      constexpr int per = kHaloHash / T;
      int mine = 0;
      for (int k = 0; k < per; ++k) mine += keys[tid * per + k] >= 0;
      int s = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += t;
      }
      if (lane == 31) sh.scan[warp] = s;
      __syncthreads();
      int at = s - mine;
      for (int k = 0; k < warp; ++k) at += sh.scan[k];
      for (int k = 0; k < per; ++k) {
        const int h = tid * per + k, m = keys[h];
        if (m >= 0) {
          hid[at] = m;
          a.wanted[m] = 1;
          slot[h] = (unsigned short)(cnt + at);
          ++at;
        }
      }
      __syncthreads();
      // slots of the off-diagonal blocks, numbered as the FP32 operator's
      for (int i = tid; i < cnt; i += T) {
        const int n = n0 + i, b0 = a.A64.node_ptr[n], b1 = a.A64.node_ptr[n + 1];
        int o = b0 - n;
        for (int e = b0; e < b1; ++e) {
          const int m = a.A64.bnbr[e];
          if (m == n) continue;
          unsigned short s16;
          if (m >= n0 && m < n1) {
            s16 = (unsigned short)(m - n0);
          } else {
            int h = m & (kHaloHash - 1);
            while (keys[h] != m) h = (h + 1) & (kHaloHash - 1);
            s16 = slot[h];
          }
          a.slots[o++] = s16;
        }
      }
      // the rows of each warp's 32 nodes regrouped, by the lanes that will read them (and wrote the slots)
      if (a.A32.val32)
        for (int i0 = tid - lane; i0 < cnt; i0 += T) {
          const bool on = i0 + lane < cnt;
          const int n = n0 + (on ? i0 + lane : cnt - 1), b0 = a.A64.node_ptr[n], from = b0 - n;
          const int c = on ? a.A64.node_ptr[n + 1] - b0 - 1 : 0;
          const int longest = __reduce_max_sync(0xffffffffu, c);
          int run = __shfl_sync(0xffffffffu, from, 0);
          for (int k = 0; k < longest; ++k) {
            const int at = lane_place(run, k, c, lane);
            if (k >= c) continue;
            a.lane_slots[at] = a.slots[from + k];
            a.lane_vals[at] = a.A32.val32[from + k];
          }
        }
    }
    cl.sync();  // the wanted marks of all blocks
    unsigned* want = reinterpret_cast<unsigned*>(hid + nh);
    for (int i0 = warp * 32; i0 < cnt; i0 += T) {
      const unsigned m = __ballot_sync(0xffffffffu, i0 + lane < cnt && __ldcg(a.wanted + n0 + i0 + lane));
      if (lane == 0) want[i0 / 32] = m;
    }
    __syncthreads();
    solve_cases<R, T>(a, cl, sh, seq, dyn + head, a.smem - head, n0, cnt, nh, hid, want, plate);
  }
  cl.sync();  // no block leaves while another may still read or write its shared memory
}

// [rhs][2N] (ld doubles apart) <-> [node][R][2] for load cases q0 .. q0 + R - 1
__global__ void k_batch_pack(int N, int R, int q0, long long ld, const double* __restrict__ src,
                             double2* __restrict__ dst) {
  const long long total = (long long)N * R;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int n = (int)(i / R), q = (int)(i - (long long)n * R);
    const double* s = src + (q0 + q) * ld + 2LL * n;
    dst[i] = make_double2(s[0], s[1]);
  }
}

__global__ void k_batch_unpack(int N, int R, int q0, long long ld, const double2* __restrict__ src,
                               double* __restrict__ dst) {
  const long long total = (long long)N * R;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int n = (int)(i / R), q = (int)(i - (long long)n * R);
    const double2 v = src[i];
    double* d = dst + (q0 + q) * ld + 2LL * n;
    d[0] = v.x;
    d[1] = v.y;
  }
}

// Every node's neighbours must lie in the node's own plate: the smallest offending node is
// recorded (a coupled batch would be solved wrongly, since plates never synchronise).
__global__ void k_batch_check(int N, int n_sys, const int* __restrict__ sys_node,
                              const int* __restrict__ node_ptr, const int* __restrict__ bnbr, int* err) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  int lo = 0, hi = n_sys;  // plate s with sys_node[s] <= n < sys_node[s + 1]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (sys_node[mid] <= n)
      lo = mid;
    else
      hi = mid;
  }
  const int a = sys_node[lo], b = sys_node[lo + 1];
  for (int k = node_ptr[n]; k < node_ptr[n + 1]; ++k) {
    const int m = bnbr[k];
    if (m < a || m >= b) {
      atomicMin(&err[kErrBatch], n);
      return;
    }
  }
}

int grid_for(long long work) {
  const long long g = (work + 255) / 256;
  return (int)std::min<long long>(std::max<long long>(g, 1), 148LL * 8);
}

template <int R, int T>
cudaError_t launch_shape(const BatchArgs* a, int cluster, const int* n_clusters, int* max_clusters,
                         cudaStream_t s) {
  auto kern = k_batch_pcg<R, T>;
  if (cluster > 8 && max_clusters) {  // the shape query always precedes a launch (never in a capture)
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
  }
  auto halo = k_batch_halo<R, T>;
  unsigned smem = 0;
  bool halo_ok = true;
  {
    int dev = 0, most = 0;
    cudaGetDevice(&dev);
    cudaError_t e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    smem = (unsigned)(most - (int)sizeof(HaloShared<R, T>)) / 1024u * 1024u;
    if (max_clusters) {
      e = cudaFuncSetAttribute(halo, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e == cudaSuccess && cluster > 8) e = cudaFuncSetAttribute(halo, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
      halo_ok = e == cudaSuccess;
      if (!halo_ok) cudaGetLastError();
    }
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)cluster;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.blockDim = dim3(T);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (max_clusters) {
    cfg.gridDim = dim3((unsigned)cluster);
    int n = 0;
    max_clusters[0] = max_clusters[1] = 0;
    cudaError_t e = cudaOccupancyMaxActiveClusters(&n, (void*)kern, &cfg);
    if (e != cudaSuccess) return e;
    max_clusters[0] = n;
    if (!halo_ok) return cudaSuccess;
    cfg.dynamicSmemBytes = smem;
    if (cudaOccupancyMaxActiveClusters(&n, (void*)halo, &cfg) == cudaSuccess)
      max_clusters[1] = n;
    else
      cudaGetLastError();
    return cudaSuccess;
  }
  BatchArgs b = *a;
  b.smem = smem;
  if (batch_halo_runs({n_clusters[0], n_clusters[1]}, a->largest, cluster, R, smem)) {
    cfg.dynamicSmemBytes = smem;
    cfg.gridDim = dim3((unsigned)(std::min(n_clusters[1], a->n_sys) * cluster));
    const cudaError_t e = cudaLaunchKernelEx(&cfg, halo, b);
    if (e != cudaSuccess) return e;
    count_launches(1);
    cfg.dynamicSmemBytes = 0;
  } else {
    b.n_rest = nullptr;
  }
  cfg.gridDim = dim3((unsigned)(std::min(n_clusters[0], a->n_sys) * cluster));
  count_launches(1);
  return cudaLaunchKernelEx(&cfg, kern, b);
}

template <int R>
cudaError_t launch_r(const BatchArgs* a, int cluster, int threads, const int* n_clusters, int* max_clusters,
                     cudaStream_t s) {
  switch (threads) {
    case 256: return launch_shape<R, 256>(a, cluster, n_clusters, max_clusters, s);
    case 512: return launch_shape<R, 512>(a, cluster, n_clusters, max_clusters, s);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t dispatch(const BatchArgs* a, int R, int cluster, int threads, const int* n_clusters, int* max_clusters,
                     cudaStream_t s) {
  if (cluster < 1 || cluster > 16) return cudaErrorInvalidValue;
  switch (R) {
    case 1: return launch_r<1>(a, cluster, threads, n_clusters, max_clusters, s);
    case 2: return launch_r<2>(a, cluster, threads, n_clusters, max_clusters, s);
    case 3: return launch_r<3>(a, cluster, threads, n_clusters, max_clusters, s);
    case 4: return launch_r<4>(a, cluster, threads, n_clusters, max_clusters, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

cudaError_t batch_max_clusters(int R, int cluster, int threads, int* n) {
  return dispatch(nullptr, R, cluster, threads, nullptr, n, nullptr);
}

cudaError_t launch_batch_pcg(const BatchArgs& a, int R, int cluster, int threads, const int* n_clusters,
                             cudaStream_t s) {
  return dispatch(&a, R, cluster, threads, n_clusters, nullptr, s);
}

cudaError_t launch_batch_pack(int N, int R, int q0, long long ld, const double* src, double* dst,
                              cudaStream_t s) {
  if (N <= 0) return cudaSuccess;
  k_batch_pack<<<grid_for((long long)N * R), 256, 0, s>>>(N, R, q0, ld, src, reinterpret_cast<double2*>(dst));
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_batch_unpack(int N, int R, int q0, long long ld, const double* src, double* dst,
                                cudaStream_t s) {
  if (N <= 0) return cudaSuccess;
  k_batch_unpack<<<grid_for((long long)N * R), 256, 0, s>>>(N, R, q0, ld, reinterpret_cast<const double2*>(src),
                                                             dst);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_batch_check(int N, int n_sys, const int* sys_node, const int* node_ptr, const int* bnbr,
                               int* err, cudaStream_t s) {
  if (N <= 0) return cudaSuccess;
  k_batch_check<<<(N + 255) / 256, 256, 0, s>>>(N, n_sys, sys_node, node_ptr, bnbr, err);
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace cstg
