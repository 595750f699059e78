// Batching form: many independent 7-point upwind convection-diffusion systems
// (the operator of a constant velocity v and D = 1 on an n0 x n1 x n2 grid,
// unit spacing, zero Dirichlet values outside) solved by Jacobi-BiCGStab in
// ONE persistent launch.
//
// What bounds it: the FP64 pipe (2 FMAs per SM and cycle) and how the systems'
// rows are spread over the SMs.  One CTA per system left the batch at the
// largest system's own time on one SM: 192 systems of 12^3 to 48^3 rows took
// 163 ms, of which the pipe needs about 25 for all of them.  The launch
// therefore runs clusters of CTAs.  A system of more than the batch's fair share
// of rows per CTA (between one and two times kBatchSplitRows) is solved by a
// whole cluster, its rows in contiguous slices; when the clusters have taken all
// of those, every CTA takes the remaining systems by itself.  Both queues are
// largest first.  Measured (to 1e-11 but the last, to 1e-8): 192 systems of 12^3
// to 48^3 rows 163 -> 37 ms, one of 48^3 and eight of 40^3 to 48^3 (clusters of
// 16) 6.2 and 8.5 ms (clusters of 8: 10.4, 13.8), 64 of 12^3 to 20^3 2.3 ms, 1024
// of 12^3 to 48^3 230 -> 172 ms.
//
// A solver (cluster or CTA) runs the whole BiCGStab iteration of
// bicgstab/solver.hpp:73-151 for its system: the operator is matrix-free, its
// phases are separated by cluster (CTA) barriers, the dot products are
// fixed-shape reductions (deterministic; every CTA of a cluster adds the same
// partial sums in the same order, so all take the same decisions), and the
// termination test (||r|| <= rtol ||r0||, maxit, rho == 0, as
// run_iterative_solver) is taken on the device.  No host round trip and no
// further launch happens until every system is done.  A system that the alpha
// step solves exactly (r = 0, where the reference's omega = 0 / 0 would give
// NaN) ends as converged.
//
// The diagonal is constant, so the Jacobi step is a scalar: with
// s = relax / diag the product A J(p) is the operator with its coefficients
// scaled by s (s * diag = relax), and x gains (alpha s) p + (omega s) r once
// per iteration.  Per row and iteration that leaves 23 FP64 operations (30
// with the step as a vector of its own) and 19 vector passes.
#include <cuda_runtime.h>

#include <algorithm>
#include <numeric>
#include <vector>

#include "lgx_internal.cuh"
#include "lgx_rows.cuh"

namespace lgx {

int sm_count();

constexpr int kBatchThreads = 512;
// CTAs per cluster: 8, the portable size, or 16 when the systems for clusters are
// so few that clusters of 16 take them all at once
constexpr int kBatchMaxCluster = 16;
// doubles of a CTA's shared memory for its rows (two CTAs per SM)
constexpr int kBatchOwn = 12 * 1024;
// A CTA's rows from which a system goes to a cluster: below 4096 a cluster's
// barriers cost more than its rows; above 8192 splitting pays even where the
// queue would balance (its rows' vectors stay in shared memory): 190 systems of
// 24^3 to 48^3 65 ms split from the fair share of 34k rows, 56 from 16k, 51 from 8k.
constexpr int64_t kBatchSplitRows = 4096;

struct BatchSys {
  int32_t n0, n1, n2;
  int64_t off;      // first row in the concatenated vectors
  double c[6];      // |a_ij| toward -d0, +d0, -d1, +d1, -d2, +d2
  double diag;
  double s, sc[6];  // relax / diag and the coefficients times it
};

namespace {

constexpr int kT = kBatchThreads;

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cluster_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// all threads of the cluster; global and shared memory written before it is
// visible to the cluster after it
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;"
               ::: "memory");
}
// stores to the same shared-memory variable of CTA `rank` of the cluster
__device__ __forceinline__ unsigned cluster_addr(const void *p, unsigned rank) {
  unsigned a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
               : "=r"(a)
               : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ void cluster_store(double *p, unsigned rank, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(cluster_addr(p, rank)), "d"(v) : "memory");
}
__device__ __forceinline__ void cluster_store(int *p, unsigned rank, int v) {
  asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(cluster_addr(p, rank)), "r"(v) : "memory");
}

// A solver's scalars: one thread per CTA computes them at the end of a reduction
// (all CTAs of a cluster from the same sums), the others read them.  Computed by
// every thread, the divisions, square roots and tests of an iteration took 60
// FP64 instructions of each of 16 warps, 7 us.
struct BatchState {
  double res2, r0n, rho, alpha, omega, beta, as, os;  // as, os: alpha s, omega s
  int64_t it;
  int status, go, exact, rere;
};

struct BatchShared {
  double tree[2][kT];
  double part[2][2][kBatchMaxCluster];  // [parity][value][rank]
  int flag[2][kBatchMaxCluster];
  BatchSys sys;  // the system at hand
  BatchState st;
  int item;
};

// v^2 rounds to more than 0 for |v| above 2^-537.5, whose square is half the smallest
// double: the largest double below it, and the magnitude's upper half to compare with
// its upper half first
constexpr long long kZeroSquare = 0x1e56a09e667f3bccll;
__device__ __forceinline__ int upper_magnitude(double v) {
  return __double2hiint(v) & 0x7fffffff;
}

// in-grid neighbours of row i: bits 0..5 for -d0, +d0, -d1, +d1, -d2, +d2
__device__ __forceinline__ unsigned row_mask(const BatchSys &S, unsigned i) {
  const unsigned n2 = (unsigned)S.n2, n1 = (unsigned)S.n1, q = i / n2;
  const unsigned p0 = q / n1, p1 = q - p0 * n1, p2 = i - q * n2;
  return (p0 > 0 ? 1u : 0u) | (p0 + 1 < (unsigned)S.n0 ? 2u : 0u) | (p1 > 0 ? 4u : 0u) |
         (p1 + 1 < n1 ? 8u : 0u) | (p2 > 0 ? 16u : 0u) | (p2 + 1 < n2 ? 32u : 0u);
}

// d x_i - sum c_j x_j over the in-grid neighbours, from acc = d x_i; the six
// loads leave together (a missing neighbour reads as 0, which leaves the sum)
__device__ __forceinline__ double apply_row(const BatchSys &S, const double (&c)[6], unsigned m,
                                            const double *x, unsigned i, double acc) {
  const int s1 = S.n2, s0 = S.n1 * S.n2;
  double v[6];
  ld_if(v[0], x + i - s0, (m & 1u) != 0u);
  ld_if(v[1], x + i - s1, (m & 4u) != 0u);
  ld_if(v[2], x + i - 1, (m & 16u) != 0u);
  ld_if(v[3], x + i + 1, (m & 32u) != 0u);
  ld_if(v[4], x + i + s1, (m & 8u) != 0u);
  ld_if(v[5], x + i + s0, (m & 2u) != 0u);
  acc = fma(-c[0], v[0], acc);
  acc = fma(-c[2], v[1], acc);
  acc = fma(-c[4], v[2], acc);
  acc = fma(-c[5], v[3], acc);
  acc = fma(-c[3], v[4], acc);
  return fma(-c[1], v[5], acc);
}

// The threads working on one system: a CTA, or all CTAs of a cluster.
template <bool CLUSTER>
struct Team {
  BatchShared &sh;
  unsigned rank, size;
  int parity;
  __device__ explicit Team(BatchShared &s)
    : sh(s), rank(CLUSTER ? cluster_rank() : 0u), size(CLUSTER ? cluster_size() : 1u),
      parity(0) {}
  __device__ __forceinline__ void sync() {
    if constexpr (CLUSTER) cluster_sync();
    else __syncthreads();
  }
  // sums of N values over the team's threads in a fixed order, and whether any
  // thread raised `flag`, handed to post(sums, any) in one thread of each CTA; a
  // barrier of the team: what was written before, and what post stored in shared
  // memory, is visible after.
  template <int N, class Post>
  __device__ __forceinline__ void reduce(const double (&v)[N], bool flag, Post post) {
    static_assert(N <= 2, "BatchShared");
    const int t = threadIdx.x;
    int any = __syncthreads_or(flag);
#pragma unroll
    for (int k = 0; k < N; ++k) sh.tree[k][t] = v[k];
    __syncthreads();
#pragma unroll
    for (int w = kT / 2; w >= 32; w >>= 1) {
      if (t < w) {
#pragma unroll
        for (int k = 0; k < N; ++k) sh.tree[k][t] += sh.tree[k][t + w];
      }
      __syncthreads();
    }
    double r[N];
    if (t < 32) {
#pragma unroll
      for (int k = 0; k < N; ++k) {
        r[k] = sh.tree[k][t];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) r[k] += __shfl_xor_sync(0xffffffffu, r[k], o);
      }
    }
    if constexpr (CLUSTER) {
      if ((unsigned)t < size) {
#pragma unroll
        for (int k = 0; k < N; ++k) cluster_store(&sh.part[parity][k][rank], (unsigned)t, r[k]);
        cluster_store(&sh.flag[parity][rank], (unsigned)t, any);
      }
      cluster_sync();
      if (t < 32) {
        const unsigned l = (unsigned)t & (size - 1);
#pragma unroll
        for (int k = 0; k < N; ++k) {
          r[k] = sh.part[parity][k][l];
          for (unsigned o = size / 2; o > 0; o >>= 1)
            r[k] += __shfl_xor_sync(0xffffffffu, r[k], o);
        }
        any = __any_sync(0xffffffffu, sh.flag[parity][l]);
      }
      parity ^= 1;
    }
    if (t == 0) post(r, any != 0);
    __syncthreads();
  }
};

struct BatchArgs {
  const BatchSys *sys;
  const double *b;
  double *x, *ws;
  uint8_t *mask;
  int64_t total;
  double rtol;
  int64_t maxit, rere;
  double relax;
  int64_t *iters;
  double *rel;
  int *status;
};

// status: 0 converged, 1 breakdown, 2 non-finite, 3 maxit reached
template <bool CLUSTER>
__device__ void solve_system(const BatchArgs &A, int id, BatchShared &shm) {
  Team<CLUSTER> team(shm);
  if (threadIdx.x == 0) shm.sys = A.sys[id];
  __syncthreads();
  const BatchSys &S = shm.sys;
  const unsigned n = (unsigned)S.n0 * S.n1 * S.n2;
  // this CTA's rows
  const unsigned chunk = CLUSTER ? ((n + team.size - 1) / team.size + 31) / 32 * 32 : n;
  const unsigned lo = min(team.rank * chunk, n), hi = min(lo + chunk, n);
  const unsigned first = lo + threadIdx.x;
  // v, t and r0 are read on this CTA's own rows only: as many of them as fit
  // stay in its shared memory (index i - lo)
  extern __shared__ double own[];
  const unsigned fit = kBatchOwn / (hi > lo ? hi - lo : 1u);
  const bool relax_one = A.relax == 1.0;
  const double *b = A.b + S.off;
  double *x = A.x + S.off;
  uint8_t *mask = A.mask + S.off;
  double *r = A.ws + S.off, *p = r + A.total;
  double *v = fit >= 1 ? own - lo : p + A.total;
  double *t = fit >= 2 ? own + (hi - lo) - lo : p + 2 * A.total;
  double *r0 = fit >= 3 ? own + 2 * (hi - lo) - lo : p + 3 * A.total;

  BatchState &st = shm.st;
  // whether run_iterative_solver goes on
  auto go_on = [&]() {
    st.go = st.status == 0 && st.it < A.maxit && sqrt(st.res2) > A.rtol * st.r0n && st.rho != 0.0;
  };

  // r = b - A x, r0 = p = r, rho = ||r||^2 (bicgstab/solver.hpp:51-71)
  double one[1] = {0.0}, two[2];
  for (unsigned i = first; i < hi; i += kT) {
    const unsigned m = row_mask(S, i);
    mask[i] = (uint8_t)m;
    const double rv = b[i] - apply_row(S, S.c, m, x, i, S.diag * x[i]);
    r[i] = rv;
    r0[i] = rv;
    p[i] = rv;
    one[0] = fma(rv, rv, one[0]);
  }
  team.reduce(one, false, [&](const double (&sum)[1], bool) {
    st.res2 = st.rho = sum[0];
    st.r0n = sqrt(sum[0]);
    st.it = 0;
    st.exact = 0;
    st.status = isfinite(sum[0]) ? 0 : 2;
    go_on();
  });
  while (st.go) {
    // v = A J(p) ; den = r0.v ; alpha = rho / den
    one[0] = 0.0;
#pragma unroll 2
    for (unsigned i = first; i < hi; i += kT) {
      const double pv = p[i];
      const double vv = apply_row(S, S.sc, mask[i], p, i, relax_one ? pv : A.relax * pv);
      v[i] = vv;
      one[0] = fma(r0[i], vv, one[0]);
    }
    team.reduce(one, false, [&](const double (&sum)[1], bool) {
      const double den = sum[0];
      if (den == 0.0) st.status = 1;
      if (!isfinite(st.rho) || !isfinite(den)) st.status = 2;
      st.alpha = st.rho / den;
      st.as = st.alpha * S.s;
    });
    if (st.status) break;
    const double alpha = st.alpha;
    // r -= alpha v; whether ||r||^2 is 0 (no entry's square rounds to more) by the
    // largest magnitude's bits, off the FP64 pipe
    int top = 0;
#pragma unroll 2
    for (unsigned i = first; i < hi; i += kT) {
      const double rv = fma(-alpha, v[i], r[i]);
      r[i] = rv;
      top = max(top, upper_magnitude(rv));
    }
    bool live = top > (int)(kZeroSquare >> 32);
    if (top == (int)(kZeroSquare >> 32))
      for (unsigned i = first; i < hi; i += kT)
        live |= (__double_as_longlong(r[i]) & 0x7fffffffffffffffll) > kZeroSquare;
    team.sync();
    // t = A J(r) ; omega = t.r / t.t
    two[0] = two[1] = 0.0;
#pragma unroll 2
    for (unsigned i = first; i < hi; i += kT) {
      const double rv = r[i];
      const double tv = apply_row(S, S.sc, mask[i], r, i, relax_one ? rv : A.relax * rv);
      t[i] = tv;
      two[0] = fma(tv, rv, two[0]);
      two[1] = fma(tv, tv, two[1]);
    }
    team.reduce(two, live, [&](const double (&sum)[2], bool any) {
      // the alpha step solved the system exactly (omega would be 0 / 0)
      st.exact = !any;
      if (any) {
        if (sum[1] == 0.0) st.status = 1;
        if (!isfinite(sum[0]) || !isfinite(sum[1])) st.status = 2;
      }
      if (st.status == 0) ++st.it;
      st.omega = sum[0] / sum[1];
      st.os = st.omega * S.s;
      st.rere = A.rere > 0 && st.it % A.rere == 0;
      if (st.exact) st.res2 = 0.0;
    });
    const double as = st.as;
    if (st.exact || st.status) {  // the iteration ends with the alpha step
      for (unsigned i = first; i < hi; i += kT) x[i] = fma(p[i], as, x[i]);
      break;
    }
    // x += alpha J(p) + omega J(r) ; r -= omega t (or r = b - A x) ;
    // rho_new = r.r0, res2 = r.r
    const double omega = st.omega, os = st.os;
    two[0] = two[1] = 0.0;
    if (st.rere) {
      for (unsigned i = first; i < hi; i += kT) x[i] = fma(r[i], os, fma(p[i], as, x[i]));
      team.sync();
      for (unsigned i = first; i < hi; i += kT) {
        const double rv = b[i] - apply_row(S, S.c, mask[i], x, i, S.diag * x[i]);
        r[i] = rv;
        two[0] = fma(rv, r0[i], two[0]);
        two[1] = fma(rv, rv, two[1]);
      }
    } else {
#pragma unroll 2
      for (unsigned i = first; i < hi; i += kT) {
        const double ro = r[i];
        x[i] = fma(ro, os, fma(p[i], as, x[i]));
        const double rv = fma(-omega, t[i], ro);
        r[i] = rv;
        two[0] = fma(rv, r0[i], two[0]);
        two[1] = fma(rv, rv, two[1]);
      }
    }
    team.reduce(two, false, [&](const double (&sum)[2], bool) {
      const double rho_new = sum[0];
      st.res2 = sum[1];
      if (st.omega == 0.0) st.status = 1;
      if (!isfinite(rho_new) || !isfinite(st.omega) || !isfinite(sum[1])) st.status = 2;
      st.beta = (rho_new / st.rho) * (st.alpha / st.omega);
      if (st.status == 0) st.rho = rho_new;
      go_on();
    });
    if (!st.go) break;
    const double beta = st.beta;
    // p = r + beta (p - omega v)
#pragma unroll 2
    for (unsigned i = first; i < hi; i += kT) p[i] = fma(fma(-omega, v[i], p[i]), beta, r[i]);
    team.sync();
  }
  if (threadIdx.x == 0 && team.rank == 0) {
    int status = st.status;
    if (status == 0 && sqrt(st.res2) > A.rtol * st.r0n && st.rho != 0.0) status = 3;
    A.iters[id] = st.it;
    A.rel[id] = st.r0n > 0.0 ? sqrt(st.res2) / st.r0n : 0.0;
    A.status[id] = status;
  }
  team.sync();
}

}  // namespace

// order: the systems, largest first; the first nsplit are solved by clusters
__global__ void __launch_bounds__(kBatchThreads, 2)
  k_batch_bicgstab(int32_t nsys, int32_t nsplit, const int32_t *__restrict__ order,
                   unsigned *queue, BatchArgs A) {
  __shared__ BatchShared sh;
  const unsigned rank = cluster_rank();
  while (nsplit > 0) {
    if (rank == 0 && threadIdx.x == 0) {
      const int q = (int)min(atomicAdd(&queue[0], 1u), (unsigned)nsplit);
      for (unsigned k = 0; k < cluster_size(); ++k) cluster_store(&sh.item, k, q);
    }
    cluster_sync();
    const int q = sh.item;
    cluster_sync();
    if (q >= nsplit) break;
    solve_system<true>(A, order[q], sh);
  }
  for (;;) {
    if (threadIdx.x == 0) sh.item = nsplit + (int)min(atomicAdd(&queue[1], 1u), (unsigned)nsys);
    __syncthreads();
    const int q = sh.item;
    __syncthreads();
    if (q >= nsys) return;
    solve_system<false>(A, order[q], sh);
  }
}

}  // namespace lgx

using namespace lgx;

extern "C" {

lgx_status lgx_batch_convdiff_bicgstab(int32_t nsys, const lgx_convdiff_system *h_systems,
                                       const double *d_b, double *d_x, double rtol, int64_t maxit,
                                       int64_t rere_period, double relax, lgx_stream stream,
                                       int64_t *h_iterations, double *h_rel_residual,
                                       int32_t *h_status) {
  if (nsys < 0 || (nsys > 0 && !h_systems)) return fail(LGX_ERR_INVALID, "bad system list");
  if (nsys == 0) return LGX_OK;
  std::vector<BatchSys> sys(nsys);
  std::vector<int64_t> rows(nsys);
  int64_t total = 0;
  for (int32_t s = 0; s < nsys; ++s) {
    const lgx_convdiff_system &in = h_systems[s];
    if (in.dims[0] < 1 || in.dims[1] < 1 || in.dims[2] < 1)
      return fail(LGX_ERR_INVALID, "system with an empty grid");
    const int64_t n = in.dims[0] * in.dims[1] * in.dims[2];
    if (n > INT32_MAX) return fail(LGX_ERR_INVALID, "system too large");
    BatchSys &S = sys[s];
    S.n0 = (int32_t)in.dims[0];
    S.n1 = (int32_t)in.dims[1];
    S.n2 = (int32_t)in.dims[2];
    S.off = total;
    double diag = 0.0;
    for (int d = 0; d < 3; ++d) {
      const double up_minus = in.v[d] > 0.0 ? in.v[d] : 0.0;
      const double up_plus = in.v[d] < 0.0 ? -in.v[d] : 0.0;
      S.c[2 * d] = 1.0 + up_minus;
      S.c[2 * d + 1] = 1.0 + up_plus;
    }
    for (int e = 0; e < 6; ++e) diag = diag + S.c[e];
    S.diag = diag;
    S.s = relax / diag;
    for (int e = 0; e < 6; ++e) S.sc[e] = S.s * S.c[e];
    rows[s] = n;
    total += n;
  }
  if (!d_b || !d_x) return fail(LGX_ERR_INVALID, "null vector");
  // largest systems first
  std::vector<int32_t> order(nsys);
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(),
                   [&](int32_t a, int32_t b) { return rows[a] > rows[b]; });
  DBuf<BatchSys> d_sys;
  DBuf<int32_t> d_order, d_status;
  DBuf<unsigned> d_queue;
  DBuf<uint8_t> d_mask;
  DBuf<double> ws, d_rel;
  DBuf<int64_t> d_iters;
  LGX_CHECK(d_sys.alloc(nsys));
  LGX_CHECK(d_order.alloc(nsys));
  LGX_CHECK(d_status.alloc(nsys));
  LGX_CHECK(d_queue.alloc(2));
  LGX_CHECK(ws.alloc(5 * total));
  LGX_CHECK(d_mask.alloc(total));
  LGX_CHECK(d_rel.alloc(nsys));
  LGX_CHECK(d_iters.alloc(nsys));
  LGX_CUDA(cudaMemcpyAsync(d_sys.p, sys.data(), sizeof(BatchSys) * nsys, cudaMemcpyHostToDevice,
                           stream));
  LGX_CUDA(cudaMemcpyAsync(d_order.p, order.data(), sizeof(int32_t) * nsys,
                           cudaMemcpyHostToDevice, stream));
  LGX_CUDA(cudaMemsetAsync(d_queue.p, 0, 2 * sizeof(unsigned), stream));
  constexpr size_t smem = sizeof(double) * kBatchOwn;
  LGX_CUDA(cudaFuncSetAttribute(k_batch_bicgstab, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)smem));
  LGX_CUDA(cudaFuncSetAttribute(k_batch_bicgstab, cudaFuncAttributeNonPortableClusterSizeAllowed,
                                1));
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  cfg.blockDim = dim3(kBatchThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  // clusters of `size` CTAs resident at a time (at least one)
  auto resident = [&](int size, int *count) -> lgx_status {
    cfg.gridDim = dim3((unsigned)size);
    attr[0].val.clusterDim = {(unsigned)size, 1, 1};
    LGX_CUDA(cudaOccupancyMaxActiveClusters(count, k_batch_bicgstab, &cfg));
    *count = std::max(*count, 1);
    return LGX_OK;
  };
  int size = 8, clusters = 0;
  LGX_CHECK(resident(size, &clusters));
  // systems beyond a CTA's fair share of the rows go to clusters
  const int64_t fair = total / ((int64_t)clusters * size);
  const int64_t share = std::min(std::max(fair, kBatchSplitRows), 2 * kBatchSplitRows);
  int32_t nsplit = 0;
  while (nsplit < nsys && rows[order[nsplit]] > share) ++nsplit;
  if (nsplit > 0) {
    int wide = 0;
    LGX_CHECK(resident(kBatchMaxCluster, &wide));
    if (nsplit <= wide) {
      size = kBatchMaxCluster;
      clusters = wide;
    }
  }
  if (nsplit == 0) {
    // no clusters to form: single CTAs, which the SMs get one by one (the CTAs of a
    // cluster share SMs while others idle: 152 systems of 16^3 3.1 ms instead of 2.0)
    size = 1;
    LGX_CHECK(resident(size, &clusters));
  }
  const int64_t want = nsplit + (nsys - nsplit + size - 1) / size;
  attr[0].val.clusterDim = {(unsigned)size, 1, 1};
  cfg.gridDim = dim3((unsigned)(std::min<int64_t>(clusters, want) * size));
  const BatchArgs args{d_sys.p, d_b,   d_x,         ws.p,  d_mask.p,  total,   rtol,
                       maxit,   rere_period, relax, d_iters.p, d_rel.p, d_status.p};
  LGX_CUDA(cudaLaunchKernelEx(&cfg, k_batch_bicgstab, nsys, nsplit, (const int32_t *)d_order.p,
                              d_queue.p, args));
  LGX_LAUNCH_CHECK();
  std::vector<int64_t> it(nsys);
  std::vector<double> rel(nsys);
  std::vector<int32_t> st(nsys);
  LGX_CUDA(cudaMemcpyAsync(it.data(), d_iters.p, sizeof(int64_t) * nsys, cudaMemcpyDeviceToHost,
                           stream));
  LGX_CUDA(cudaMemcpyAsync(rel.data(), d_rel.p, sizeof(double) * nsys, cudaMemcpyDeviceToHost,
                           stream));
  LGX_CUDA(cudaMemcpyAsync(st.data(), d_status.p, sizeof(int32_t) * nsys, cudaMemcpyDeviceToHost,
                           stream));
  LGX_CUDA(cudaStreamSynchronize(stream));
  if (h_iterations) std::copy(it.begin(), it.end(), h_iterations);
  if (h_rel_residual) std::copy(rel.begin(), rel.end(), h_rel_residual);
  if (h_status) std::copy(st.begin(), st.end(), h_status);
  for (int32_t s = 0; s < nsys; ++s)
    if (st[s] == 1 || st[s] == 2)
      return fail(st[s] == 1 ? LGX_ERR_BREAKDOWN : LGX_ERR_NONFINITE,
                  "system " + std::to_string(s) + (st[s] == 1 ? ": breakdown" : ": non-finite"));
  return LGX_OK;
}

}  // extern "C"
