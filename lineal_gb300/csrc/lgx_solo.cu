// CG and BiCGStab without a preconditioner or with Jacobi, a whole solve in one
// cooperative launch.
//
// On systems that fit the L2 an iteration is a few microseconds of work behind
// five to eight launches and a host round trip: 52 us per Jacobi-CG iteration on
// the 64^3 lookup stencil, of which its FP64 operations take 7.  Here one CTA
// per SM or two own a slice of the rows each (their vectors stay in a workspace in
// global memory, which the L2 holds), the phases of
// conjugate-gradients/solver.hpp:75-115 and bicgstab/solver.hpp:73-151 are
// separated by grid barriers, every CTA adds the same partial sums in the same
// order (so all take the same decisions) and the stopping rule of
// run_iterative_solver is evaluated on the device: 21 us per iteration (about 2.7
// for each of its three barriers).
//
// The rows have the arithmetic of the products they replace (csr_spmv,
// k_st_apply) and the Jacobi step that of k_jacobi_diag_zero, its quotient
// through a reciprocal (div_by_recip: the same bits); only the grouping of the
// dot products' sums differs.
//
// Every wait at the grid barrier is bounded (about one second of SM clock): on
// timeout the CTA records the device error flag and leaves, and the others
// follow when their own waits run out.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "lgx_internal.cuh"
#include "lgx_rows.cuh"
#include "lgx_stencil.cuh"

namespace lgx {

namespace {

constexpr int kST = 512;              // threads per CTA
constexpr int kSoloMaxCtas = 32 * 10;  // a lane adds up to 10 CTAs' sums
// rows from which two CTAs per SM are worth their barriers: Jacobi-BiCGStab on
// CSR rows at 96^3, 50 iterations, one CTA per SM 7.8 ms, two 5.9; at 64^3 2.5, 2.5
constexpr int64_t kSoloTwoRows = 600000;
// rows of a CTA below which the grid shrinks: fewer CTAs, cheaper barriers
constexpr int64_t kSoloMinRows = 512;

enum SoloOp { S_CSR64, S_CSR32, S_LOOKUP, S_VALUE };

struct SoloArgs {
  int n, chunk;  // rows, rows per CTA
  const int64_t *rowptr;
  const int32_t *col;
  const double *v64;
  const float *v32;
  StencilDev st;
  const double *diag;  // null: no preconditioner
  const double *b;
  double *x;
  double *ws;          // vectors of n entries
  double relax, rtol;
  int64_t maxit, rere;
  double *hist;        // squared residual norms
  double *part;        // [2 parities][2 values][CTAs]
  unsigned *arrived;
  int *err;
  struct SoloResult *out;
};

struct SoloResult {
  double res2, r0;
  int64_t it;
  int flag;   // bit 0: breakdown, bit 1: non-finite
  int start;  // 1: the initial residual is not finite
};

struct SoloShared {
  double tree[2][kST];
  double conn[48];
  double alpha, beta, omega, rho, res2, r0, stop2;
  int64_t it;
  int flag, go, rere, lost;
  int huge;  // some CTA met an entry of 2^501 or more
};

// Up to kSoloMaxRows entries below 2^501 have a finite sum of squares.  BiCGStab
// takes the norm of its half residual only where there are larger ones (for its
// error on overflow); that there are travels as the top bit of the barriers'
// counter, which counts to less than 2^31: at most seven barriers an iteration, of
// kSoloMaxCtas CTAs, in kSoloMaxIterations (beyond them, the launches).
constexpr int kSoloHuge = 1023 + 501;
constexpr unsigned kSoloHugeBit = 0x80000000u;
constexpr int64_t kSoloMaxIterations = 900000;
static_assert(7 * (kSoloMaxIterations + 1) * kSoloMaxCtas < (int64_t)kSoloHugeBit, "counter");

__device__ __forceinline__ bool finite_bits(double v) { return exponent_field(v) != 0x7ff; }

// What ||r||^2 has to exceed for ||r|| > limit (a square root is a chain of its own
// in every iteration): the limit's square rounded down, so that neither a tiny nor
// a huge one changes the answer; nothing is at or below a negative limit, and
// nothing beyond one that is not a number.
__device__ __forceinline__ double stop_square(double limit) {
  return limit < 0.0 ? -1.0 : __dmul_rd(limit, limit);
}

// The barrier of the whole grid and the reductions that end in it.  A reduction
// leaves its CTA's sums in the barrier's parity of A.part, arrives on one counter
// and, when all have arrived, adds the sums of all CTAs.  (Polling every CTA's
// sums directly, marked with the barrier's number, saves the counter's round trip
// and loses more to 152 warps reading 600 words that are being written: Jacobi-CG
// at 64^3 36 us per iteration instead of 21.)
// HUGE: the counter may carry kSoloHugeBit.  It is raised and looked at in one kind
// of barrier only, sync_huge; a CTA that is still in the barrier before it when
// another one raises the bit ignores it there and finds it here.
template <bool HUGE>
struct SoloGrid {
  const SoloArgs &A;
  SoloShared &sh;
  unsigned epoch;
  __device__ SoloGrid(const SoloArgs &a, SoloShared &s) : A(a), sh(s), epoch(0) {}
  // one thread, after a CTA barrier: arrive, wait for all
  __device__ __forceinline__ unsigned arrive_and_wait() {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(A.arrived) : "memory");
    const unsigned target = epoch * gridDim.x;
    const long long start = clock64();
    unsigned seen;
    for (;;) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(A.arrived) : "memory");
      if ((HUGE ? seen & ~kSoloHugeBit : seen) >= target) break;
      if (clock64() - start > (1ll << 31)) {
        sh.lost = 1;
        atomicExch(A.err, 1);
        break;
      }
    }
    return seen;
  }
  // warp 0, after a CTA barrier: every CTA's r (of lane 0) summed (lane-strided,
  // then a tree) in all lanes
  template <int N>
  __device__ __forceinline__ void exchange(double (&r)[N]) {
    const int lane = threadIdx.x;
    ++epoch;
    double *part = A.part + (size_t)(epoch & 1u) * 2 * gridDim.x;
    if (lane == 0) {
#pragma unroll
      for (int k = 0; k < N; ++k) __stcg(part + k * gridDim.x + blockIdx.x, r[k]);
      arrive_and_wait();
    }
    __syncwarp();
    double v[N][kSoloMaxCtas / 32];
#pragma unroll
    for (int j = 0; j < kSoloMaxCtas / 32; ++j) {
      const unsigned c = lane + 32 * j;
#pragma unroll
      for (int k = 0; k < N; ++k) v[k][j] = c < gridDim.x ? __ldcg(part + k * gridDim.x + c) : 0.0;
    }
#pragma unroll
    for (int k = 0; k < N; ++k) {
      r[k] = 0.0;
#pragma unroll
      for (int j = 0; j < kSoloMaxCtas / 32; ++j)
        if (32u * j < gridDim.x) r[k] += v[k][j];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) r[k] += __shfl_xor_sync(0xffffffffu, r[k], o);
    }
  }
  // false: a wait ran out
  __device__ __forceinline__ bool sync() {
    __syncthreads();
    if (gridDim.x > 1) {
      ++epoch;
      if (threadIdx.x == 0) arrive_and_wait();
      __syncthreads();
    }
    return !sh.lost;
  }
  // sync, after which sh.huge says whether any thread of the grid has set it
  __device__ __forceinline__ bool sync_huge() {
    __syncthreads();
    if (gridDim.x > 1) {
      ++epoch;
      if (threadIdx.x == 0) {
        if (sh.huge) atomicOr(A.arrived, kSoloHugeBit);
        if (arrive_and_wait() & kSoloHugeBit) sh.huge = 1;
      }
      __syncthreads();
    }
    return !sh.lost;
  }
  // sums of N values over the grid in a fixed order, handed to post(sums) in one
  // thread of each CTA; what was written before is visible after
  template <int N, class Post>
  __device__ __forceinline__ bool reduce(const double (&v)[N], Post post) {
    const int t = threadIdx.x;
#pragma unroll
    for (int k = 0; k < N; ++k) sh.tree[k][t] = v[k];
    __syncthreads();
#pragma unroll
    for (int w = kST / 2; w >= 32; w >>= 1) {
      if (t < w) {
#pragma unroll
        for (int k = 0; k < N; ++k) sh.tree[k][t] += sh.tree[k][t + w];
      }
      __syncthreads();
    }
    if (t < 32) {
      double r[N];
#pragma unroll
      for (int k = 0; k < N; ++k) {
        r[k] = sh.tree[k][t];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) r[k] += __shfl_xor_sync(0xffffffffu, r[k], o);
      }
      if (gridDim.x > 1) exchange(r);
      if (t == 0) post(r);
    } else {
      ++epoch;
    }
    __syncthreads();
    return !sh.lost;
  }
};

// (A x)_i; x is written by other CTAs between barriers, so its loads are plain
template <int OP>
__device__ __forceinline__ double solo_apply(const SoloArgs &A, const double *conn,
                                             const double *x, int i) {
  if constexpr (OP == S_CSR64 || OP == S_CSR32) {
    const int64_t b = A.rowptr[i];
    const int len = (int)(A.rowptr[i + 1] - b);
    if constexpr (OP == S_CSR64)
      return row_dot<8, true, double, double>(A.col + b, A.v64 + b, len, x, 0.0);
    else
      return row_dot<8, true, float, double>(A.col + b, A.v32 + b, len, x, 0.0);
  } else {
    const unsigned n2 = (unsigned)A.st.n2, n1 = (unsigned)A.st.n1, q = (unsigned)i / n2;
    const int p0 = (int)(q / n1), p1 = (int)(q - (unsigned)p0 * n1), p2 = (int)((unsigned)i - q * n2);
    double cv[6];
    int64_t cj[6];
    bool has[6];
    st_row<OP == S_LOOKUP>(A.st, conn, p0, p1, p2, i, cv, cj, has);
    double xv[6];
#pragma unroll
    for (int e = 0; e < 6; ++e) ld_if(xv[e], x + cj[e], has[e]);
    double sum = 0.0;
#pragma unroll
    for (int e = 0; e < 6; ++e)
      if (has[e]) sum = fma(-cv[e], xv[e], sum);
    return fma(A.st.diag[i], x[i], sum);
  }
}

// Jacobi from zero: fma(relax, r / d, (1 - relax) 0); y = 1 / d, or 0: divide
__device__ __forceinline__ double solo_jacobi(const SoloArgs &A, double r, double y, int i) {
  const double q = nonzero_bits(y) && exponent_within_400(r) ? div_by_recip(r, A.diag[i], y)
                                                             : r / A.diag[i];
  return A.relax == 1.0 ? q : fma(A.relax, q, (1.0 - A.relax) * 0.0);
}

template <int OP>
__global__ void __launch_bounds__(kST, 2) k_solo_cg(SoloArgs A) {
  __shared__ SoloShared sh;
  SoloGrid<false> grid(A, sh);
  if (threadIdx.x == 0) sh.lost = 0;
  if (threadIdx.x < 48) sh.conn[threadIdx.x] = A.st.conn[threadIdx.x];
  __syncthreads();
  const size_t n = (size_t)A.n;
  const bool precon = A.diag != nullptr;
  double *r = A.ws, *p = r + n, *q = p + n, *rd = q + n;
  const int lo = min((int)blockIdx.x * A.chunk, A.n), hi = min(lo + A.chunk, A.n);
  const int first = lo + (int)threadIdx.x;
  double one[1], two[2] = {0.0, 0.0};
  auto go_on = [&]() {
    sh.go = sh.flag == 0 && sh.it < A.maxit && sh.res2 > sh.stop2 && sh.rho != 0.0;
  };
  // r = b - A x, p = z = M r, rho = r.z
  for (int i = first; i < hi; i += kST) {
    const double rv = A.b[i] - solo_apply<OP>(A, sh.conn, A.x, i);
    r[i] = rv;
    double z = rv;
    if (precon) {
      const double y = exponent_within_400(A.diag[i]) ? 1.0 / A.diag[i] : 0.0;
      rd[i] = y;
      z = solo_jacobi(A, rv, y, i);
    }
    p[i] = z;
    two[0] = fma(rv, rv, two[0]);
    two[1] = fma(z, rv, two[1]);
  }
  if (!grid.reduce(two, [&](const double (&s)[2]) {
        sh.res2 = s[0];
        sh.rho = precon ? s[1] : s[0];
        sh.r0 = sqrt(s[0]);
        sh.stop2 = stop_square(A.rtol * sh.r0);
        sh.it = 0;
        sh.flag = finite_bits(s[0]) && finite_bits(sh.rho) ? 0 : 4;
        go_on();
        if (A.hist && blockIdx.x == 0) A.hist[0] = s[0];
      }))
    return;
  while (sh.go) {
    // q = A p ; alpha = rho / p.q
    one[0] = 0.0;
    for (int i = first; i < hi; i += kST) {
      const double qv = solo_apply<OP>(A, sh.conn, p, i);
      q[i] = qv;
      one[0] = fma(p[i], qv, one[0]);
    }
    if (!grid.reduce(one, [&](const double (&s)[1]) {
          if (!finite_bits(sh.rho) || !finite_bits(s[0])) sh.flag |= 2;
          if (s[0] == 0.0) sh.flag |= 1;
          sh.alpha = sh.rho / s[0];
          sh.rere = A.rere > 0 && sh.it > 0 && sh.it % A.rere == 0;
        }))
      return;
    // x += alpha p ; r -= alpha q, or b - A x ; z = M r (kept in q)
    const double alpha = sh.alpha;
    const bool rere = sh.rere;
    two[0] = two[1] = 0.0;
    if (rere) {
      for (int i = first; i < hi; i += kST) A.x[i] = fma(p[i], alpha, A.x[i]);
      if (!grid.sync()) return;
    }
    for (int i = first; i < hi; i += kST) {
      double rv;
      if (rere) {
        rv = A.b[i] - solo_apply<OP>(A, sh.conn, A.x, i);
      } else {
        A.x[i] = fma(p[i], alpha, A.x[i]);
        rv = fma(-alpha, q[i], r[i]);
      }
      r[i] = rv;
      two[0] = fma(rv, rv, two[0]);
      if (precon) {
        const double z = solo_jacobi(A, rv, rd[i], i);
        q[i] = z;
        two[1] = fma(rv, z, two[1]);
      }
    }
    if (!grid.reduce(two, [&](const double (&s)[2]) {
          const double rho = precon ? s[1] : s[0];
          sh.res2 = s[0];
          // (a recomputed residual's norm is looked at as the next iteration's rho)
          if (!finite_bits(s[0]) || !finite_bits(rho)) {
            if (!sh.rere || (precon && !finite_bits(rho))) sh.flag |= 2;
          }
          sh.beta = rho / sh.rho;
          sh.rho = rho;
          ++sh.it;
          go_on();
          if (A.hist && blockIdx.x == 0) A.hist[sh.it] = s[0];
        }))
      return;
    if (!sh.go) break;
    // p = z + beta p
    const double beta = sh.beta;
    const double *z = precon ? q : r;
    for (int i = first; i < hi; i += kST) p[i] = fma(p[i], beta, z[i]);
    if (!grid.sync()) return;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0)
    *A.out = SoloResult{sh.res2, sh.r0, sh.it, sh.flag & 3, sh.flag >> 2};
}

template <int OP>
__global__ void __launch_bounds__(kST, 2) k_solo_bicgstab(SoloArgs A) {
  __shared__ SoloShared sh;
  SoloGrid<true> grid(A, sh);
  if (threadIdx.x == 0) sh.lost = sh.huge = 0;
  if (threadIdx.x < 48) sh.conn[threadIdx.x] = A.st.conn[threadIdx.x];
  __syncthreads();
  const size_t n = (size_t)A.n;
  const bool precon = A.diag != nullptr;
  double *r = A.ws, *r0 = r + n, *p = r0 + n, *v = p + n, *t = v + n;
  // the preconditioned p and r (themselves without a preconditioner)
  double *zp = precon ? t + n : p, *zr = precon ? zp + n : r;
  double *rd = t + 3 * n;
  const int lo = min((int)blockIdx.x * A.chunk, A.n), hi = min(lo + A.chunk, A.n);
  const int first = lo + (int)threadIdx.x;
  double one[1] = {0.0}, two[2];
  auto go_on = [&]() {
    sh.go = sh.flag == 0 && sh.it < A.maxit && sh.res2 > sh.stop2 && sh.rho != 0.0;
  };
  // r = b - A x, r0 = p = r, rho = ||r||^2
  for (int i = first; i < hi; i += kST) {
    const double rv = A.b[i] - solo_apply<OP>(A, sh.conn, A.x, i);
    r[i] = rv;
    r0[i] = rv;
    p[i] = rv;
    if (precon) {
      const double y = exponent_within_400(A.diag[i]) ? 1.0 / A.diag[i] : 0.0;
      rd[i] = y;
      zp[i] = solo_jacobi(A, rv, y, i);
    }
    one[0] = fma(rv, rv, one[0]);
  }
  if (!grid.reduce(one, [&](const double (&s)[1]) {
        sh.res2 = sh.rho = s[0];
        sh.r0 = sqrt(s[0]);
        sh.stop2 = stop_square(A.rtol * sh.r0);
        sh.it = 0;
        sh.flag = finite_bits(s[0]) ? 0 : 4;
        go_on();
        if (A.hist && blockIdx.x == 0) A.hist[0] = s[0];
      }))
    return;
  while (sh.go) {
    // v = A M p ; alpha = rho / r0.v
    one[0] = 0.0;
    for (int i = first; i < hi; i += kST) {
      const double vv = solo_apply<OP>(A, sh.conn, zp, i);
      v[i] = vv;
      one[0] = fma(r0[i], vv, one[0]);
    }
    if (!grid.reduce(one, [&](const double (&s)[1]) {
          if (!finite_bits(sh.rho) || !finite_bits(s[0])) sh.flag |= 2;
          if (s[0] == 0.0) sh.flag |= 1;
          sh.alpha = sh.rho / s[0];
        }))
      return;
    // x += alpha M p ; r -= alpha v ; M r
    const double alpha = sh.alpha;
    bool huge = false;
    for (int i = first; i < hi; i += kST) {
      A.x[i] = fma(zp[i], alpha, A.x[i]);
      const double rv = fma(-alpha, v[i], r[i]);
      r[i] = rv;
      huge |= exponent_field(rv) >= kSoloHuge;
      if (precon) zr[i] = solo_jacobi(A, rv, rd[i], i);
    }
    if (huge) sh.huge = 1;
    if (!grid.sync_huge()) return;
    if (sh.huge) {  // whether ||r||^2 overflows
      one[0] = 0.0;
      for (int i = first; i < hi; i += kST) one[0] = fma(r[i], r[i], one[0]);
      if (!grid.reduce(one, [&](const double (&s)[1]) {
            if (!finite_bits(s[0])) sh.flag |= 2;
          }))
        return;
    }
    // t = A M r ; omega = t.r / t.t
    two[0] = two[1] = 0.0;
    for (int i = first; i < hi; i += kST) {
      const double tv = solo_apply<OP>(A, sh.conn, zr, i);
      t[i] = tv;
      two[0] = fma(tv, r[i], two[0]);
      two[1] = fma(tv, tv, two[1]);
    }
    if (!grid.reduce(two, [&](const double (&s)[2]) {
          if (!finite_bits(s[0]) || !finite_bits(s[1])) sh.flag |= 2;
          if (s[1] == 0.0) sh.flag |= 1;
          sh.omega = s[0] / s[1];
          sh.rere = A.rere > 0 && sh.it > 0 && sh.it % A.rere == 0;
        }))
      return;
    // x += omega M r ; r -= omega t, or b - A x ; rho = r.r0
    const double omega = sh.omega;
    const bool rere = sh.rere;
    two[0] = two[1] = 0.0;
    if (rere) {
      for (int i = first; i < hi; i += kST) A.x[i] = fma(zr[i], omega, A.x[i]);
      if (!grid.sync()) return;
    }
    for (int i = first; i < hi; i += kST) {
      double rv;
      if (rere) {
        rv = A.b[i] - solo_apply<OP>(A, sh.conn, A.x, i);
      } else {
        A.x[i] = fma(zr[i], omega, A.x[i]);
        rv = fma(-omega, t[i], r[i]);
      }
      r[i] = rv;
      two[0] = fma(rv, r0[i], two[0]);
      two[1] = fma(rv, rv, two[1]);
    }
    if (!grid.reduce(two, [&](const double (&s)[2]) {
          if (!finite_bits(s[0]) || !finite_bits(sh.omega)) sh.flag |= 2;
          if (sh.omega == 0.0 || sh.rho == 0.0) sh.flag |= 1;
          sh.beta = (s[0] / sh.rho) * (sh.alpha / sh.omega);
          sh.rho = s[0];
          sh.res2 = s[1];
          ++sh.it;
          go_on();
          if (A.hist && blockIdx.x == 0) A.hist[sh.it] = s[1];
        }))
      return;
    if (!sh.go) break;
    // p = r + beta (p - omega v) ; M p
    const double beta = sh.beta;
    for (int i = first; i < hi; i += kST) {
      const double pv = fma(fma(-omega, v[i], p[i]), beta, r[i]);
      p[i] = pv;
      if (precon) zp[i] = solo_jacobi(A, pv, rd[i], i);
    }
    if (!grid.sync()) return;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0)
    *A.out = SoloResult{sh.res2, sh.r0, sh.it, sh.flag & 3, sh.flag >> 2};
}

// the kernel and the grid's upper bound (all CTAs resident)
template <int OP>
lgx_status solo_kernel(bool cg, int64_t n, void **fn, int *most) {
  *fn = cg ? (void *)k_solo_cg<OP> : (void *)k_solo_bicgstab<OP>;
  int per_sm = 0;
  LGX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, *fn, kST, 0));
  *most = std::min(std::min(per_sm, n > kSoloTwoRows ? 2 : 1) * sm_count(), kSoloMaxCtas);
  return LGX_OK;
}

}  // namespace

// Runs the solve when the system is one for this path (*done), else leaves it.
// Where the line lies: beyond kSoloMaxRows rows or kSoloMaxEntries entries an
// iteration is bound by bandwidth, and the launches' own kernels stream better than
// this one's plain loops.  50 Jacobi-CG iterations, setup included, launches / one
// launch, ms: lookup stencil 24^3 2.2 / 0.8, 64^3 3.3 / 1.4, 96^3 4.9 / 2.8, 112^3
// 6.6 / 4.2, 128^3 8.2 / 8.5; 7-point CSR 64^3 3.3 / 1.5, 112^3 7.2 / 5.0, 128^3 9.2
// / 9.1; 27-point CSR 64^3 4.1 / 2.7, 96^3 7.9 / 7.2, 104^3 (30M entries) 9.3 / 8.8,
// 108^3 (33M) 10.0 / 9.8, 112^3 (37M) 10.7 / 10.7 (BiCGStab 16.5 / 16.2, 17.8 /
// 18.0, 19.4 / 19.7).
constexpr int64_t kSoloMaxRows = 1500000, kSoloMaxEntries = 32000000;
// A thread works its rows entry by entry, about 0.18 us each, and all CTAs wait for
// the slowest: a chain of up to kSoloChain entries per product, and one more for
// every kSoloChainStep entries of the matrix (which the launches have to stream),
// beats the launches.  The chain is bounded by the longest row, so a few long rows
// leave the system to the launches, and no barrier waits for more than 0.4 ms of
// work.  50 Jacobi-CG iterations, launches / one launch, ms, even rows: 2000 rows
// of 30 entries 2.7 / 1.3, of 100 2.8 / 2.7, of 400 3.7 / 8.0; 5000 of 200 3.0 /
// 4.5; 20000 of 60 2.8 / 1.9, of 200 3.8 / 4.5; 100000 of 100 6.2 / 3.9, of 200
// 10.7 / 6.8; 300000 of 80 10.4 / 6.8.
constexpr int64_t kSoloChain = 192, kSoloChainStep = 20000;

lgx_status solo_solve(bool cg, const lgx_matrix *a, const double *d_b, double *d_x,
                      const lgx_solve_params *p, cudaStream_t s, int64_t *iterations,
                      double *final_rel, double *history, bool *done) {
  *done = false;
  const int64_t n = a->n;
  if ((p->precon != LGX_PRECON_NONE && p->precon != LGX_PRECON_JACOBI) || !p->use_graphs ||
      (cg && p->flexible && p->precon != LGX_PRECON_NONE) || n < 1 || n > kSoloMaxRows ||
      p->maxit < 0 || p->maxit > kSoloMaxIterations || overlap(d_b, d_x, sizeof(double) * (size_t)n))
    return LGX_OK;
  int dev = 0, coop = 0;
  LGX_CUDA(cudaGetDevice(&dev));
  LGX_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
  if (!coop) return LGX_OK;
  SoloArgs A{};
  void *fn = nullptr;
  int most = 0;
  if (a->kind == LGX_MATRIX_CSR) {
    const Csr &c = a->csr;
    A.rowptr = c.rowptr.p;
    A.col = c.col.p;
    A.v64 = c.v64.p;
    A.v32 = c.v32.p;
    if (c.storage == LGX_F64) LGX_CHECK(solo_kernel<S_CSR64>(cg, n, &fn, &most));
    else LGX_CHECK(solo_kernel<S_CSR32>(cg, n, &fn, &most));
  } else {
    LGX_CHECK(stencil_ensure(const_cast<lgx_matrix *>(a), s));
    A.st = dev_of(a);
    if (a->st.lookup) LGX_CHECK(solo_kernel<S_LOOKUP>(cg, n, &fn, &most));
    else LGX_CHECK(solo_kernel<S_VALUE>(cg, n, &fn, &most));
  }
  if (most < 1) return LGX_OK;
  const int64_t ctas = std::min<int64_t>(most, std::max<int64_t>(1, n / kSoloMinRows));
  A.n = (int)n;
  A.chunk = (int)(((n + ctas - 1) / ctas + 31) / 32 * 32);
  if (a->kind == LGX_MATRIX_CSR &&
      (a->csr.nnz > kSoloMaxEntries ||
       (A.chunk + kST - 1) / kST * a->csr.max_row > kSoloChain + a->csr.nnz / kSoloChainStep))
    return LGX_OK;
  if (p->precon == LGX_PRECON_JACOBI)
    LGX_CHECK(matrix_diagonal(const_cast<lgx_matrix *>(a), s, &A.diag));
  const unsigned grid = (unsigned)((n + A.chunk - 1) / A.chunk);
  DBuf<double> ws, hist;
  DBuf<double> part;
  DBuf<unsigned> arrived;
  DBuf<SoloResult> out;
  LGX_CHECK(ws.alloc((cg ? 4 : 8) * n));
  LGX_CHECK(part.alloc(4 * (int64_t)grid));
  LGX_CHECK(arrived.alloc(1));
  LGX_CHECK(out.alloc(1));
  if (history) LGX_CHECK(hist.alloc(p->maxit + 1));
  LGX_CUDA(cudaMemsetAsync(arrived.p, 0, sizeof(unsigned), s));
  A.b = d_b;
  A.x = d_x;
  A.ws = ws.p;
  A.relax = p->relax;
  A.rtol = p->rtol;
  A.maxit = p->maxit;
  A.rere = p->rere_period;
  A.hist = history ? hist.p : nullptr;
  A.part = part.p;
  A.arrived = arrived.p;
  A.err = device_error_flag();
  A.out = out.p;
  void *args[] = {&A};
  const cudaError_t launched = cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kST), args, 0, s);
  if (launched == cudaErrorCooperativeLaunchTooLarge) {
    // less of the device than its properties say (a shared or divided one): the
    // launches take the solve, x is as it was
    cudaGetLastError();
    return LGX_OK;
  }
  LGX_CUDA(launched);
  count_launch();
  SoloResult h{};
  LGX_CUDA(cudaMemcpyAsync(&h, out.p, sizeof(h), cudaMemcpyDeviceToHost, s));
  LGX_CUDA(cudaStreamSynchronize(s));
  LGX_CHECK(check_device_error(s));
  *done = true;
  if (h.start)
    return fail(LGX_ERR_NONFINITE, "non-finite initial residual or preconditioned residual");
  if (history) {
    LGX_CUDA(cudaMemcpyAsync(history, hist.p, sizeof(double) * (size_t)(h.it + 1),
                             cudaMemcpyDeviceToHost, s));
    LGX_CUDA(cudaStreamSynchronize(s));
    for (int64_t k = 0; k <= h.it; ++k) history[k] = std::sqrt(history[k]);
  }
  if (iterations) *iterations = h.it;
  if (final_rel) *final_rel = h.r0 > 0 ? std::sqrt(h.res2) / h.r0 : 0.0;
  if (h.flag & 2)
    return fail(LGX_ERR_NONFINITE, "non-finite value in iteration " + std::to_string(h.it));
  if (h.flag & 1)
    return fail(LGX_ERR_BREAKDOWN, "zero denominator in iteration " + std::to_string(h.it));
  return LGX_OK;
}

}  // namespace lgx
