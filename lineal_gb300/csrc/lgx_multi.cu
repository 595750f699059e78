// Multi-right-hand-side (blocked) AMG-PCG: up to 32 right-hand sides share
// every pass over the matrices.  Vectors are row-major blocks, X[i * K + k].  In
// the row kernels a group of lanes shares a row, a few columns per lane (MLane),
// and a row's column indices and values are read once by the group (a lane an
// entry, then broadcast by shuffles) and applied to all K columns, whose gathers
// x[c * K + k] are contiguous; in the dots and the dense solve lane k of a warp
// handles column k.  Per column the arithmetic is the
// single-vector one (products in storage order, SOR row formula, aggregate
// sums in list order), so each column follows its own CG recurrence; the CG
// scalars are per column and a converged column is frozen.
//
// The outer iteration is FP64 (the finest matrix in FP64, FP64 dots); the
// preconditioner is the hierarchy's V-cycle in the hierarchy's cycle type
// (float for cycle_f32 hierarchies), with the coarsest solve through the
// FP64 dense inverse.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "lgx_amg.cuh"
#include "lgx_internal.cuh"
#include "lgx_rows.cuh"

namespace lgx {

constexpr int kMaxRhs = 32;
constexpr int kMThreads = 256;  // 8 warps per CTA

__device__ __forceinline__ int64_t warp_id_global() {
  return ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
}
__device__ __forceinline__ int64_t warps_global() { return ((int64_t)gridDim.x * blockDim.x) >> 5; }

inline unsigned mgrid(int64_t rows) {
  const int64_t warps_per_block = kMThreads / 32;
  const int64_t g = (rows + warps_per_block - 1) / warps_per_block;
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>(g, 65535));
}

// ---- a group of lanes per row ----------------------------------------------
// The K columns of a row are spread over G lanes (a power of two) of V columns
// each, one 16-byte vector for float columns in fours and FP64 columns in
// pairs, so that a warp works on 32 / G rows at once.  A warp per row with a
// column per lane spends two shuffles, a load and an FMA on each entry of one
// row and is bound by issuing them: the red-black colours of 128^3 rows, 32
// float columns, took 390 us against 85 for their bytes; 8 lanes of 4 columns
// spend the same instructions on four rows: 190 us a colour, the residual 645
// -> 146 (the first colour's rows; the second's are 0, m_zero_from), the FP64
// product 973 -> 890 us (its FP64 FMAs alone take 750).
template <typename T, int V>
struct alignas(sizeof(T) * V) MVec {
  T v[V];
};
template <typename T, int V>
__device__ __forceinline__ MVec<T, V> m_load(const T *p, bool on) {
  MVec<T, V> r;
#pragma unroll
  for (int j = 0; j < V; ++j) r.v[j] = T(0);
  if (on) r = *reinterpret_cast<const MVec<T, V> *>(p);
  return r;
}
template <typename T, int V>
__device__ __forceinline__ void m_store(T *p, const MVec<T, V> &r) {
  *reinterpret_cast<MVec<T, V> *>(p) = r;
}

// lanes: the lane's place in its row's group, its first column, the row
template <int V>
struct MLane {
  int g, g0, k0;  // place in the group, the group's first lane, first column
  int64_t r;      // row of this lane's group among all groups of the grid
  __device__ __forceinline__ explicit MLane(int G) {
    const int lane = threadIdx.x & 31;
    g = lane & (G - 1);
    g0 = lane - g;
    k0 = g * V;
    r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
  }
};
// how many columns a lane takes, and the lanes of a row
template <typename XT>
inline int m_vec(int K) {
  return K % 4 == 0 && sizeof(XT) == 4 ? 4 : K % 2 == 0 ? 2 : 1;
}
inline int m_group(int K, int V) {
  int G = 4;
  while (G * V < K) G *= 2;
  return G;
}
inline unsigned m_ctas(int64_t rows, int G) {
  const int64_t per_cta = kMThreads / G;
  return (unsigned)std::max<int64_t>(1, (rows + per_cta - 1) / per_cta);
}

// Rows [rb, re) of a CSR matrix on K columns.
//  M_MUL: y = A x, b - A x with b, -A x with neg;
//  M_SOR: the row formula of gauss-seidel-variant/sweep.hpp:134-200 in place on
//    x (from_zero: a forward sweep from x = 0, rows at or after visit_end read
//    as 0); M_LO: such a sweep on a natural-order level's earlier-colour
//    halves, the diagonals in pdiag.
// Matrix row r is vector row rows[r] (natural-order levels), or r itself.  The
// entries go in chunks of G, a lane loading one, and in batches of B <= G gathers.
//
// Launches of so few rows that a column per lane, at least eight lanes (so entries
// of a chunk) and eight gathers at once take no more than a quarter of the chip last
// as long as one row's chain, which is shorter so.  Blocked FP64 solves of 7 points,
// vectors per lane throughout / so, and a warp per row before either, ms: 336 rows, 32
// columns 2.60 / 2.24 / 2.42, 27 rows, 8 columns 0.78 / 0.70 / 0.71.  With the line at
// 320000 lanes 64000 rows of 27 points and 32 columns take 25.2 instead of 24.2, and
// with it at 80000 columns 64000 rows of 7 points and one column 10.63 instead of
// 10.44.
constexpr int64_t kMFewLanes = 80000;
constexpr int kMFewBatch = 8;
enum MRowMode { M_MUL, M_SOR, M_LO };

template <typename VT, typename XT, int MODE, int V, int B>
__global__ void __launch_bounds__(kMThreads)
  k_mrows(int64_t rb, int64_t re, const int64_t *__restrict__ rowptr,
          const int32_t *__restrict__ col, const VT *__restrict__ val,
          const int32_t *__restrict__ rows, const double *__restrict__ pdiag, int K, int G,
          const XT *__restrict__ b, const XT *x, XT *y, XT relax, XT m1, int neg, int ultra,
          int from_zero, int64_t visit_end) {
  constexpr unsigned kAll = 0xffffffffu;
  const MLane<V> L(G);
  const int64_t r = rb + L.r;
  const bool in = r < re, on = in && L.k0 < K;
  const int64_t rr = in ? r : re - 1;
  const int64_t e0 = rowptr[rr];
  const int len = in ? (int)(rowptr[rr + 1] - e0) : 0;
  const int64_t i = rows ? (int64_t)rows[rr] : rr;
  const int64_t at = i * K + L.k0;
  MVec<XT, V> bv, xi, acc;
  bv = m_load<XT, V>(b + at, on && (MODE != M_MUL || b));
  xi = m_load<XT, V>(x + at, on && MODE == M_SOR && !from_zero);
  XT diag = MODE == M_LO ? (XT)pdiag[rr] : XT(0);
#pragma unroll
  for (int j = 0; j < V; ++j) acc.v[j] = MODE == M_MUL ? XT(0) : bv.v[j];
  const int longest = __reduce_max_sync(kAll, len);
  for (int base = 0; base < longest; base += G) {
    int32_t c_l = 0;
    VT a_l = VT(0);
    if (base + L.g < len) {
      c_l = col[e0 + base + L.g];
      a_l = val[e0 + base + L.g];
    }
    const int m = longest - base < G ? longest - base : G;
    for (int u0 = 0; u0 < m; u0 += B) {
      MVec<XT, V> xv[B];
      XT av[B];
      bool own[B];
#pragma unroll
      for (int u = 0; u < B; ++u) {
        const int src = L.g0 + ((u0 + u) & (G - 1));
        const int32_t c = __shfl_sync(kAll, c_l, src);
        av[u] = (XT)__shfl_sync(kAll, a_l, src);
        own[u] = MODE == M_SOR && c == i;
        xv[u] = m_load<XT, V>(x + (int64_t)c * K + L.k0,
                              on && base + u0 + u < len && !own[u] &&
                                !(MODE == M_SOR && from_zero && c >= visit_end));
      }
#pragma unroll
      for (int u = 0; u < B; ++u) {
        if (base + u0 + u < len) {
          if (own[u]) {
            diag = av[u];
            if (ultra) {
#pragma unroll
              for (int j = 0; j < V; ++j) acc.v[j] = fma(-av[u], xi.v[j], acc.v[j]);
            }
          } else {
#pragma unroll
            for (int j = 0; j < V; ++j)
              acc.v[j] = fma(MODE == M_MUL ? av[u] : -av[u], xv[u].v[j], acc.v[j]);
          }
        }
      }
    }
  }
  if (!on) return;
#pragma unroll
  for (int j = 0; j < V; ++j) {
    if (MODE == M_MUL) acc.v[j] = b ? bv.v[j] - acc.v[j] : neg ? -acc.v[j] : acc.v[j];
    else if (ultra) acc.v[j] = xi.v[j] + relax * acc.v[j] / fabs(diag);
    else acc.v[j] = fma(relax, acc.v[j] / diag, m1 * xi.v[j]);
  }
  m_store<XT, V>(y + at, acc);
}

// The first colour of a forward sweep from zero: x = relax b / d (every
// neighbour reads 0).
template <typename XT, int V>
__global__ void __launch_bounds__(kMThreads)
  k_mfirst(int64_t rb, int64_t re, const double *__restrict__ pdiag,
           const int32_t *__restrict__ rows, int K, int G, const XT *__restrict__ b,
           XT *__restrict__ x, XT relax, XT m1, int ultra) {
  const MLane<V> L(G);
  const int64_t r = rb + L.r;
  if (r >= re || L.k0 >= K) return;
  const int64_t at = (rows ? (int64_t)rows[r] : r) * K + L.k0;
  const XT d = (XT)pdiag[r];
  MVec<XT, V> v = m_load<XT, V>(b + at, true);
#pragma unroll
  for (int j = 0; j < V; ++j)
    v.v[j] = ultra ? relax * v.v[j] / fabs(d) : fma(relax, v.v[j] / d, m1 * XT(0));
  m_store<XT, V>(x + at, v);
}

// b_c[c] = sum over the aggregate's fine rows (list order) of r; fine rows at
// or after zero_from hold 0 and are not read
template <typename XT, int V>
__global__ void __launch_bounds__(kMThreads)
  k_mrestrict(int64_t nc, const int64_t *__restrict__ rptr, const int32_t *__restrict__ rlist,
              int K, int G, int64_t zero_from, const XT *__restrict__ r, XT *__restrict__ bc) {
  constexpr int B = 4;
  const MLane<V> L(G);
  if (L.r >= nc || L.k0 >= K) return;
  MVec<XT, V> s;
#pragma unroll
  for (int j = 0; j < V; ++j) s.v[j] = XT(0);
  const int64_t p0 = rptr[L.r];
  const int len = (int)(rptr[L.r + 1] - p0);
  for (int k = 0; k < len; k += B) {
    MVec<XT, V> v[B];
#pragma unroll
    for (int u = 0; u < B; ++u) {
      const int64_t i = rlist[p0 + min(k + u, len - 1)];
      v[u] = m_load<XT, V>(r + i * K + L.k0, k + u < len && i < zero_from);
    }
#pragma unroll
    for (int u = 0; u < B; ++u)
      if (k + u < len) {
#pragma unroll
        for (int j = 0; j < V; ++j) s.v[j] = s.v[j] + v[u].v[j];
      }
  }
  m_store<XT, V>(bc + L.r * K + L.k0, s);
}

// x_f += inv_relax * refine(x_c)
template <typename XT, int V>
__global__ void __launch_bounds__(kMThreads)
  k_mprolong(int64_t n, const uint32_t *__restrict__ agg_p, int K, int G,
             const XT *__restrict__ xc, XT inv_relax, XT *__restrict__ x) {
  const MLane<V> L(G);
  if (L.r >= n || L.k0 >= K) return;
  const uint32_t a = agg_p[L.r];
  const MVec<XT, V> ref = m_load<XT, V>(xc + (int64_t)a * K + L.k0, a < kIsolated);
  MVec<XT, V> v = m_load<XT, V>(x + L.r * K + L.k0, true);
#pragma unroll
  for (int j = 0; j < V; ++j) v.v[j] = v.v[j] + ref.v[j] * inv_relax;
  m_store<XT, V>(x + L.r * K + L.k0, v);
}

// X = A^-1 B with the FP64 dense inverse: a CTA takes kMDenseRows rows, its
// warps a share of the columns each, the shares summed in warp order.  (A warp
// per row read B once per row and kept one chain of loads in flight: 450 us
// for 1588 rows and 32 columns, whose FMAs take 130; now 215.)
constexpr int kMDenseRows = 4, kMBatch = 8;
template <typename XT>
__global__ void __launch_bounds__(kMThreads)
  k_mdense(int64_t n, const double *__restrict__ ainv, int K, const XT *__restrict__ b,
           XT *__restrict__ x) {
  constexpr int W = kMThreads / 32, R = kMDenseRows;
  __shared__ double sh[W][R][32];
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  const int64_t i0 = (int64_t)blockIdx.x * R;
  double acc[R];
#pragma unroll
  for (int q = 0; q < R; ++q) acc[q] = 0.0;
  // 32 columns of the inverse at a time: lane l loads column j0 + l of each row
  for (int64_t j0 = (int64_t)wl * 32; j0 < n; j0 += 32 * W) {
    double a_l[R];
#pragma unroll
    for (int q = 0; q < R; ++q)
      a_l[q] = (j0 + lane < n && i0 + q < n) ? ainv[(i0 + q) * n + j0 + lane] : 0.0;
    const int m = n - j0 < 32 ? (int)(n - j0) : 32;
    for (int u0 = 0; u0 < m; u0 += kMBatch) {
      XT v[kMBatch];
#pragma unroll
      for (int u = 0; u < kMBatch; ++u)
        ld_if(v[u], b + (j0 + u0 + u) * K + lane, u0 + u < m && lane < K);
#pragma unroll
      for (int u = 0; u < kMBatch; ++u) {
        if (u0 + u < m) {
#pragma unroll
          for (int q = 0; q < R; ++q)
            acc[q] = fma(__shfl_sync(0xffffffffu, a_l[q], (u0 + u) & 31), (double)v[u], acc[q]);
        }
      }
    }
  }
#pragma unroll
  for (int q = 0; q < R; ++q) sh[wl][q][lane] = acc[q];
  __syncthreads();
  if (wl < R && lane < K && i0 + wl < n) {
    double t = 0.0;
    for (int w = 0; w < W; ++w) t += sh[w][wl][lane];
    x[(i0 + wl) * K + lane] = (XT)t;
  }
}

template <typename T, typename U>
__global__ void k_mconvert(int64_t total, const T *__restrict__ src, U *__restrict__ dst) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x)
    dst[t] = (U)src[t];
}

// row blocks between natural and permuted order: dst[r] = src[perm[r]]
// (gather) or dst[perm[r]] = src[r] (scatter)
__global__ void k_mpermute(int64_t n, const int32_t *__restrict__ perm, int K, int scatter,
                           const double *__restrict__ src, double *__restrict__ dst) {
  const int64_t total = n * K;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = t / K;
    const int k = (int)(t - r * K);
    const int64_t p = perm[r];
    if (scatter) {
      dst[p * K + k] = src[t];
    } else {
      dst[t] = src[p * K + k];
    }
  }
}

// float to double by integer operations (exact, as the conversion is): the FP64
// pipe converts at its own rate, 2 per SM and cycle, and bounds a dot whose
// FMAs already fill it.
__device__ __forceinline__ double m_wide(double v) { return v; }
__device__ __forceinline__ double m_wide(float v) {
  const unsigned u = __float_as_uint(v);
  unsigned e = (u >> 23) & 0xffu, m = u & 0x7fffffu;
  if (e == 0u) {  // zero, or a subnormal m 2^-149
    if (m != 0u) {
      const int p = 31 - __clz((int)m);
      m = (m << (23 - p)) & 0x7fffffu;
      e = (unsigned)(p + 874);
    }
  } else {
    e = e == 0xffu ? 0x7ffu : e + 896u;
  }
  return __hiloint2double((int)((u & 0x80000000u) | (e << 20) | (m >> 3)), (int)(m << 29));
}

// Per-column dots: out[k] = sum_i u[i,k] v[i,k] and (SQ) out[K + k] =
// sum_i u[i,k]^2.  Each block reduces a fixed strided set of rows per column
// in a fixed tree; the scalar kernels add the block partials in a fixed order.
template <typename ZT, bool SQ>
__global__ void __launch_bounds__(kMThreads)
  k_mdot(int64_t n, int K, const double *__restrict__ u, const ZT *__restrict__ v,
         double *__restrict__ partials) {
  __shared__ double sh[2][kMThreads / 32][kMaxRhs];
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  double s1 = 0.0, s2 = 0.0;
  if (lane < K) {
    const int64_t step = warps_global();
    int64_t i = warp_id_global();
    // four rows' loads together
    for (; i + 3 * step < n; i += 4 * step) {
      double a[4];
      ZT z[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int64_t t = (i + q * step) * K + lane;
        a[q] = u[t];
        z[q] = v[t];
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        s1 = fma(a[q], m_wide(z[q]), s1);
        if (SQ) s2 = fma(a[q], a[q], s2);
      }
    }
    for (; i < n; i += step) {
      const double a = u[i * K + lane];
      s1 = fma(a, m_wide(v[i * K + lane]), s1);
      if (SQ) s2 = fma(a, a, s2);
    }
  }
  sh[0][wl][lane] = s1;
  sh[1][wl][lane] = s2;
  __syncthreads();
  if (threadIdx.x < 2 * kMaxRhs) {
    const int which = threadIdx.x / kMaxRhs, k = threadIdx.x % kMaxRhs;
    double t = 0.0;
    for (int q = 0; q < kMThreads / 32; ++q) t += sh[which][q][k];
    partials[((int64_t)blockIdx.x * 2 + which) * kMaxRhs + k] = t;
  }
}

// The threads of an elementwise kernel stride by a multiple of K, so that each
// stays on one column (no division per element).
__device__ __forceinline__ int64_t m_stride(int K) {
  const int64_t t = (int64_t)gridDim.x * blockDim.x;
  return t - t % K;
}

// X += alpha P, R -= alpha Q (alpha per column); rf != null: R as float too (a
// float cycle's input)
__global__ void k_mupdate(int64_t n, int K, const double *__restrict__ alpha,
                          const double *__restrict__ p, const double *__restrict__ q,
                          double *__restrict__ x, double *__restrict__ r,
                          float *__restrict__ rf) {
  const int64_t total = n * K, stride = m_stride(K);
  int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= stride) return;
  const double a = alpha[t % K];
#pragma unroll 2
  for (; t < total; t += stride) {
    x[t] = fma(p[t], a, x[t]);
    const double rv = fma(-a, q[t], r[t]);
    r[t] = rv;
    if (rf) rf[t] = (float)rv;
  }
}

// P = Z + beta P for active columns (beta NaN marks a frozen column)
template <typename ZT>
__global__ void k_mxpby(int64_t n, int K, const double *__restrict__ beta,
                        const ZT *__restrict__ z, double *__restrict__ p) {
  const int64_t total = n * K, stride = m_stride(K);
  int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= stride) return;
  const double bk = beta[t % K];
  if (bk != bk) return;
#pragma unroll 4
  for (; t < total; t += stride) p[t] = fma(p[t], bk, m_wide(z[t]));
}

inline unsigned egrid(int64_t total) {
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>((total + 255) / 256, 16384));
}

// ---- multi-column V-cycle (permuted spaces) -------------------------------
template <typename XT>
struct MWork {
  std::vector<DBuf<XT>> b, x, r;
};

// f(V as a constant) with the columns per lane for K columns of type XT
template <typename XT, typename F>
static lgx_status m_with_vec(int K, F f) {
  const int V = m_vec<XT>(K);
  const int G = m_group(K, V);
  if constexpr (sizeof(XT) == 4)
    if (V == 4) return f(std::integral_constant<int, 4>{}, G);
  if (V == 2) return f(std::integral_constant<int, 2>{}, G);
  return f(std::integral_constant<int, 1>{}, G);
}

template <typename VT, typename XT, int MODE>
static lgx_status m_rows(int64_t rb, int64_t re, const Csr &p, const VT *val, const int32_t *rows,
                         const double *pdiag, int K, const XT *b, const XT *x, XT *y, XT relax,
                         int neg, int ultra, int from_zero, cudaStream_t s) {
  if (re <= rb) return LGX_OK;
  auto launch = [&](auto v, auto batch, int G) -> lgx_status {
    k_mrows<VT, XT, MODE, v, batch><<<m_ctas(re - rb, G), kMThreads, 0, s>>>(
      rb, re, p.rowptr.p, p.col.p, val, rows, pdiag, K, G, b, x, y, relax, XT(1) - relax, neg,
      ultra, from_zero, rb);
    LGX_LAUNCH_CHECK();
    return LGX_OK;
  };
  const int few = std::max(kMFewBatch, m_group(K, 1));
  if ((re - rb) * few <= kMFewLanes)
    return launch(std::integral_constant<int, 1>{}, std::integral_constant<int, kMFewBatch>{},
                  few);
  return m_with_vec<XT>(K, [&](auto v, int G) {
    return launch(v, std::integral_constant<int, sizeof(XT) == 8 ? 2 : 4>{}, G);
  });
}

template <typename VT, typename XT>
static lgx_status m_sor(const lgx_colouring &c, const VT *val, const VT *lo_val, int K, int forward,
                        int from_zero, const XT *b, XT *x, XT relax, int ultra, cudaStream_t s) {
  const int fz = from_zero && forward;
  const int32_t *rows = c.natural ? c.perm.p : nullptr;
  for (int32_t k = 0; k < c.ncolours; ++k) {
    const int32_t cid = forward ? k : c.ncolours - 1 - k;
    const int64_t rb = c.offsets[cid], re = c.offsets[cid + 1];
    if (re <= rb) continue;
    if (fz && k == 0) {
      LGX_CHECK(m_with_vec<XT>(K, [&](auto v, int G) -> lgx_status {
        k_mfirst<XT, v><<<m_ctas(re - rb, G), kMThreads, 0, s>>>(rb, re, c.pdiag.p, rows, K, G, b,
                                                                 x, relax, XT(1) - relax, ultra);
        LGX_LAUNCH_CHECK();
        return LGX_OK;
      }));
    } else if (fz && c.natural) {
      LGX_CHECK((m_rows<VT, XT, M_LO>(rb, re, c.lo, lo_val, rows, c.pdiag.p, K, b, x, x, relax, 0,
                                      ultra, 1, s)));
    } else {
      LGX_CHECK((m_rows<VT, XT, M_SOR>(rb, re, c.pcsr, val, rows, nullptr, K, b, x, x, relax, 0,
                                       ultra, fz, s)));
    }
  }
  return LGX_OK;
}

template <typename XT>
static lgx_status m_level_sor(const lgx_amg &h, const lgx_amg_level &lv, int K, int forward,
                              int from_zero, const XT *b, XT *x, cudaStream_t s) {
  const lgx_colouring &c = *lv.col;
  const XT relax = (XT)h.p.smoother_relax;
  const int ultra = h.p.smoother_ultra;
  if constexpr (sizeof(XT) == 8)
    if (c.pcsr.storage == LGX_F64)
      return m_sor<double, XT>(c, c.pcsr.v64.p, c.lo.v64.p, K, forward, from_zero, b, x, relax,
                               ultra, s);
  const float *v = c.pcsr.storage == LGX_F32 ? c.pcsr.v32.p : c.pv32.p;
  return m_sor<float, XT>(c, v, c.lo.v32.p, K, forward, from_zero, b, x, relax, ultra, s);
}

// With relax 1 the residual that follows a forward sweep from zero is 0 in the
// rows of the last colour (mc_up_residual): permuted levels compute the rows
// before m_zero_from only, and the restriction does not read the others.
static int64_t m_zero_from(const lgx_amg &h, const lgx_amg_level &lv) {
  const lgx_colouring &c = *lv.col;
  if (c.natural || h.p.smoother_relax != 1.0 || h.p.smoother_ultra || c.ncolours < 1)
    return INT64_MAX;
  return c.offsets[c.ncolours - 1];
}

template <typename XT>
static lgx_status m_level_residual(const lgx_amg &h, const lgx_amg_level &lv, int K, const XT *b,
                                   const XT *x, XT *r, cudaStream_t s) {
  const lgx_colouring &c = *lv.col;
  // natural-order levels after such a sweep: the later-colour halves
  const bool up = c.natural && h.p.smoother_relax == 1.0 && !h.p.smoother_ultra;
  const Csr &p = up ? c.up : c.pcsr;
  const int32_t *rows = c.natural && !up ? c.perm.p : nullptr;
  const int64_t re = std::min(p.n, m_zero_from(h, lv));
  auto run = [&](auto *v) {
    using VT = std::remove_const_t<std::remove_pointer_t<decltype(v)>>;
    return m_rows<VT, XT, M_MUL>(0, re, p, v, rows, nullptr, K, up ? nullptr : b, x, r, XT(1), up, 0,
                                 0, s);
  };
  if constexpr (sizeof(XT) == 8)
    if (p.storage == LGX_F64) return run((const double *)p.v64.p);
  return run((const float *)(p.storage == LGX_F32 ? p.v32.p : c.pv32.p));
}

template <typename XT>
static lgx_status m_vcycle(const lgx_amg &h, int K, MWork<XT> &w, const XT *b0, XT *x0,
                           cudaStream_t s) {
  const int64_t L = (int64_t)h.lv.size();
  auto bv = [&](int64_t l) { return l == 0 ? b0 : (const XT *)w.b[l].p; };
  auto xv = [&](int64_t l) { return l == 0 ? x0 : w.x[l].p; };
  for (int64_t l = 0; l + 1 < L; ++l) {
    const lgx_amg_level &lv = *h.lv[l];
    if (lv.a->n == 0) continue;
    LGX_CHECK(m_level_sor<XT>(h, lv, K, 1, 1, bv(l), xv(l), s));
    LGX_CHECK(m_level_residual<XT>(h, lv, K, bv(l), xv(l), w.r[l].p, s));
    const int64_t nc = h.lv[l + 1]->a->n;
    if (nc) {
      LGX_CHECK(m_with_vec<XT>(K, [&](auto v, int G) -> lgx_status {
        k_mrestrict<XT, v><<<m_ctas(nc, G), kMThreads, 0, s>>>(
          nc, lv.rptr.p, lv.rlist.p, K, G, m_zero_from(h, lv), w.r[l].p, w.b[l + 1].p);
        LGX_LAUNCH_CHECK();
        return LGX_OK;
      }));
    }
  }
  {
    const int64_t nc = h.lv[L - 1]->a->n;
    if (nc) {
      k_mdense<XT><<<(unsigned)((nc + kMDenseRows - 1) / kMDenseRows), kMThreads, 0, s>>>(
        nc, h.inv.p, K, bv(L - 1), xv(L - 1));
      LGX_LAUNCH_CHECK();
    }
  }
  const XT inv_relax = (XT)(1.0 / h.p.relax);
  for (int64_t l = L - 2; l >= 0; --l) {
    const lgx_amg_level &lv = *h.lv[l];
    const int64_t n = lv.a->n;
    if (n == 0) continue;
    LGX_CHECK(m_with_vec<XT>(K, [&](auto v, int G) -> lgx_status {
      k_mprolong<XT, v><<<m_ctas(n, G), kMThreads, 0, s>>>(n, lv.agg_p.p, K, G, xv(l + 1),
                                                           inv_relax, xv(l));
      LGX_LAUNCH_CHECK();
      return LGX_OK;
    }));
    LGX_CHECK(m_level_sor<XT>(h, lv, K, 0, 0, bv(l), xv(l), s));
  }
  return LGX_OK;
}

// Per-column CG scalars of the blocked solver.  They stay on the device, so
// that an iteration needs no host round trip and is captured once as a
// CUDA graph; the host reads the block once per iteration for the stopping
// test.
struct MState {
  double rho[kMaxRhs], r0[kMaxRhs], res2[kMaxRhs];
  int64_t it_done[kMaxRhs];  // last iteration each column took part in
  int active[kMaxRhs];
  int64_t it;                // iterations completed
  int n_active;
  int flags;                 // 1: p.Ap = 0 (breakdown), 2: non-finite
  int bad_col;               // lowest column that raised `flags`
};

// The k_mdot block partials (`which` 0: u.v, 1: w.w) of column k in lane k of
// warp 0: up to 32 warps (as many as partials, m_scalar_threads) sum strided shares,
// warp 0 adds them in warp order.  All threads call it.  (One thread per column
// summing 1024 partials in turn took 95 us, and 186 for both; now 15 and 27 cold.)
inline unsigned m_scalar_threads(unsigned g) { return 32 * std::min(g, 32u); }
__device__ double m_column_sum(const double *partials, unsigned g, int which) {
  __shared__ double sh[32][kMaxRhs];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, warps = blockDim.x >> 5;
  double a = 0.0;
#pragma unroll 4
  for (unsigned q = w; q < g; q += 32) a += partials[((size_t)q * 2 + which) * kMaxRhs + lane];
  __syncthreads();
  sh[w][lane] = a;
  __syncthreads();
  double t = 0.0;
  if (w == 0)
    for (int v = 0; v < warps; ++v) t += sh[v][lane];
  return t;
}

__device__ void m_raise(MState *st, unsigned mask, int flag) {
  if (mask && threadIdx.x == 0) {
    st->flags |= flag;
    st->bad_col = __ffs(mask) - 1;
  }
}

// rho = R.Z, r0 = ||R||, active = r0 > 0 and rho != 0 
__global__ void k_minit(unsigned g, int K, const double *__restrict__ partials, int64_t maxit,
                        MState *st) {
  const int k = threadIdx.x;
  const double rho = m_column_sum(partials, g, 0);
  const double res2 = m_column_sum(partials, g, 1);
  if (k >= 32) return;
  int act = 0, bad = 0;
  if (k < K) {
    bad = !isfinite(res2) || !isfinite(rho);
    st->rho[k] = rho;
    st->res2[k] = res2;
    st->r0[k] = sqrt(res2);
    act = !bad && st->r0[k] > 0.0 && rho != 0.0 && maxit > 0;
    st->active[k] = act;
    st->it_done[k] = 0;
  }
  const unsigned am = __ballot_sync(~0u, act), bm = __ballot_sync(~0u, bad);
  if (k == 0) {
    st->n_active = __popc(am);
    st->it = 0;
    st->flags = 0;
    st->bad_col = -1;
  }
  __syncwarp();
  m_raise(st, bm, 2);
}

// alpha = rho / P.Q for active columns, 0 for the others
__global__ void k_malpha(unsigned g, int K, const double *__restrict__ partials, MState *st,
                         double *__restrict__ alpha) {
  const int k = threadIdx.x;
  const double den = m_column_sum(partials, g, 0);
  if (k >= 32) return;
  double a = 0.0;
  int zero = 0, bad = 0;
  if (k < K && st->active[k]) {
    bad = !isfinite(den);
    zero = den == 0.0;
    if (!bad && !zero) a = st->rho[k] / den;
  }
  if (k < K) alpha[k] = a;
  const unsigned zm = __ballot_sync(~0u, zero), bm = __ballot_sync(~0u, bad);
  m_raise(st, zm, 1);
  __syncwarp();
  m_raise(st, bm, 2);
}

// stopping test and beta = rho_new / rho; converged and inactive columns get
// a NaN beta (k_mxpby leaves their P frozen)
__global__ void k_mbeta(unsigned g, int K, const double *__restrict__ partials, double rtol,
                        MState *st, double *__restrict__ beta) {
  const int k = threadIdx.x;
  const double rho_new = m_column_sum(partials, g, 0);
  const double res2 = m_column_sum(partials, g, 1);
  if (k >= 32) return;
  const int64_t it = st->it + 1;
  double b = __longlong_as_double(0x7ff8000000000000ll);
  int act = 0;
  if (k < K) {
    st->res2[k] = res2;
    if (st->active[k]) {
      st->it_done[k] = it;
      if (sqrt(res2) <= rtol * st->r0[k] || rho_new == 0.0) {
        st->active[k] = 0;
      } else {
        b = rho_new / st->rho[k];
        st->rho[k] = rho_new;
        act = 1;
      }
    }
    beta[k] = b;
  }
  const unsigned am = __ballot_sync(~0u, act);
  if (k == 0) {
    st->n_active = __popc(am);
    st->it = it;
  }
}

// owns the captured iterations and the stream they are recorded on
struct MGraphs {
  cudaStream_t capture = nullptr;
  cudaGraphExec_t exec[2] = {nullptr, nullptr};
  ~MGraphs() {
    for (auto &e : exec)
      if (e) cudaGraphExecDestroy(e);
    if (capture) cudaStreamDestroy(capture);
  }
};

template <typename XT>
static lgx_status pcg_multi(const lgx_matrix *a, lgx_amg &h, int K, const double *d_b,
                            double *d_x, double rtol, int64_t maxit, int use_graphs,
                            cudaStream_t user_stream, int64_t *h_it, double *h_rel) {
  const int64_t n = a->n;
  const int64_t L = (int64_t)h.lv.size();
  const bool permuted = L > 1;
  const int32_t *perm = permuted ? h.lv[0]->perm() : nullptr;
  const Csr &A = perm ? h.lv[0]->col->pcsr : a->csr;  // (the hierarchy's own, checked)
  const int64_t nk = n * K;
  // the stream every launch below goes to: the caller's, or the capture
  // stream while an iteration is recorded
  cudaStream_t s = user_stream;
  // outer vectors (permuted order): B, X, R, P, Q, Z
  DBuf<double> B, X, R, P, Q, Z, alpha_d, beta_d, partials;
  DBuf<MState> state;
  for (DBuf<double> *v : {&B, &X, &R, &P, &Q}) LGX_CHECK(v->alloc(std::max<int64_t>(nk, 1)));
  LGX_CHECK(alpha_d.alloc(kMaxRhs));
  LGX_CHECK(beta_d.alloc(kMaxRhs));
  LGX_CHECK(partials.alloc(1024 * 2 * kMaxRhs));
  LGX_CHECK(state.alloc(1));
  const unsigned gdot = std::min<unsigned>(mgrid(n), 1024);
  if (perm) {
    k_mpermute<<<egrid(nk), 256, 0, s>>>(n, perm, K, 0, d_b, B.p);
    k_mpermute<<<egrid(nk), 256, 0, s>>>(n, perm, K, 0, d_x, X.p);
    LGX_LAUNCH_CHECK();
  } else {
    LGX_CUDA(cudaMemcpyAsync(B.p, d_b, sizeof(double) * nk, cudaMemcpyDeviceToDevice, s));
    LGX_CUDA(cudaMemcpyAsync(X.p, d_x, sizeof(double) * nk, cudaMemcpyDeviceToDevice, s));
  }
  // V-cycle workspace (cycle type XT); level 0 of a float cycle has its own b/x
  MWork<XT> w;
  w.b.resize(L);
  w.x.resize(L);
  w.r.resize(L);
  for (int64_t l = 0; l < L; ++l) {
    const int64_t nl = std::max<int64_t>(h.lv[l]->a->n * K, 1);
    LGX_CHECK(w.r[l].alloc(nl));
    if (l > 0 || sizeof(XT) == 4) {
      LGX_CHECK(w.b[l].alloc(nl));
      LGX_CHECK(w.x[l].alloc(nl));
    }
  }
  // A float cycle reads R as float (w.b[0], written by k_mupdate or converted)
  // and leaves Z as float in w.x[0], which the dots and the direction read.
  constexpr bool kFloat = sizeof(XT) == 4;
  float *rf = nullptr;
  const XT *z = nullptr;
  if constexpr (kFloat) {
    rf = w.b[0].p;
    z = w.x[0].p;
  } else {
    LGX_CHECK(Z.alloc(std::max<int64_t>(nk, 1)));
    z = Z.p;
  }
  auto to_float = [&]() -> lgx_status {
    if constexpr (kFloat) {
      k_mconvert<double, float><<<egrid(nk), 256, 0, s>>>(nk, R.p, rf);
      LGX_LAUNCH_CHECK();
    }
    return LGX_OK;
  };
  auto precondition = [&]() -> lgx_status {
    if constexpr (kFloat) return m_vcycle<float>(h, K, w, rf, w.x[0].p, s);
    else return m_vcycle<double>(h, K, w, R.p, Z.p, s);
  };
  // y = A x, or b - A x
  auto apply = [&](const double *bb, const double *x, double *y) -> lgx_status {
    auto run = [&](auto *v) {
      using VT = std::remove_const_t<std::remove_pointer_t<decltype(v)>>;
      return m_rows<VT, double, M_MUL>(0, n, A, v, nullptr, nullptr, K, bb, x, y, 1.0, 0, 0, 0, s);
    };
    return A.storage == LGX_F64 ? run((const double *)A.v64.p) : run((const float *)A.v32.p);
  };
  // partials of R.Z and R.R
  auto dots_rz = [&]() -> lgx_status {
    k_mdot<XT, true><<<gdot, kMThreads, 0, s>>>(n, K, R.p, z, partials.p);
    LGX_LAUNCH_CHECK();
    return LGX_OK;
  };
  // one iteration (conjugate-gradients/solver.hpp:75-117 per column); with
  // `rere` the residual is recomputed as B - A X (every 8th iteration)
  auto iteration = [&](int rere) -> lgx_status {
    // Q = A P ; alpha = rho / P.Q ; X += alpha P ; R -= alpha Q
    LGX_CHECK(apply(nullptr, P.p, Q.p));
    k_mdot<double, false><<<gdot, kMThreads, 0, s>>>(n, K, P.p, Q.p, partials.p);
    LGX_LAUNCH_CHECK();
    k_malpha<<<1, m_scalar_threads(gdot), 0, s>>>(gdot, K, partials.p, state.p, alpha_d.p);
    k_mupdate<<<egrid(nk), 256, 0, s>>>(n, K, alpha_d.p, P.p, Q.p, X.p, R.p, rere ? nullptr : rf);
    LGX_LAUNCH_CHECK();
    if (rere) {
      LGX_CHECK(apply(B.p, X.p, R.p));
      LGX_CHECK(to_float());
    }
    // Z = M R ; beta = R.Z / rho ; P = Z + beta P
    LGX_CHECK(precondition());
    LGX_CHECK(dots_rz());
    k_mbeta<<<1, m_scalar_threads(gdot), 0, s>>>(gdot, K, partials.p, rtol, state.p, beta_d.p);
    k_mxpby<XT><<<egrid(nk), 256, 0, s>>>(n, K, beta_d.p, z, P.p);
    LGX_LAUNCH_CHECK();
    return LGX_OK;
  };
  MGraphs graphs;
  auto capture = [&](int rere) -> lgx_status {
    if (!graphs.capture)
      LGX_CUDA(cudaStreamCreateWithFlags(&graphs.capture, cudaStreamNonBlocking));
    s = graphs.capture;
    cudaGraph_t gr = nullptr;
    cudaError_t e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
    lgx_status st = e == cudaSuccess ? iteration(rere) : cuda_fail(e, "cudaStreamBeginCapture");
    const cudaError_t e2 = cudaStreamEndCapture(s, &gr);
    s = user_stream;
    if (st != LGX_OK) {
      if (gr) cudaGraphDestroy(gr);
      return st;
    }
    if (e2 != cudaSuccess) return cuda_fail(e2, "cudaStreamEndCapture");
    e = cudaGraphInstantiate(&graphs.exec[rere], gr, 0);
    cudaGraphDestroy(gr);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGraphInstantiate");
    return LGX_OK;
  };
  MState hs{};
  auto read_state = [&]() -> lgx_status {
    LGX_CUDA(cudaMemcpyAsync(&hs, state.p, sizeof(MState), cudaMemcpyDeviceToHost, s));
    LGX_CUDA(cudaStreamSynchronize(s));
    return LGX_OK;
  };
  // R = B - A X ; Z = M R ; rho = R.Z ; P = Z (conjugate-gradients/solver.hpp:50-73)
  LGX_CHECK(apply(B.p, X.p, R.p));
  LGX_CHECK(to_float());
  LGX_CHECK(precondition());
  LGX_CHECK(dots_rz());
  k_minit<<<1, m_scalar_threads(gdot), 0, s>>>(gdot, K, partials.p, maxit, state.p);
  LGX_LAUNCH_CHECK();
  if constexpr (kFloat) {
    k_mconvert<float, double><<<egrid(nk), 256, 0, s>>>(nk, z, P.p);
    LGX_LAUNCH_CHECK();
  } else {
    LGX_CUDA(cudaMemcpyAsync(P.p, z, sizeof(double) * nk, cudaMemcpyDeviceToDevice, s));
  }
  LGX_CHECK(read_state());
  if (hs.flags & 2)
    return fail(LGX_ERR_NONFINITE,
                "non-finite initial residual in column " + std::to_string(hs.bad_col));
  int64_t it = 0;
  while (hs.n_active > 0 && it < maxit) {
    const int rere = (it + 1) % 8 == 0;
    if (use_graphs && it > 0) {
      // the first iteration ran eagerly; later ones replay the recording
      if (!graphs.exec[rere]) LGX_CHECK(capture(rere));
      LGX_CUDA(cudaGraphLaunch(graphs.exec[rere], s));
    } else {
      LGX_CHECK(iteration(rere));
    }
    ++it;
    LGX_CHECK(read_state());
    if (hs.flags)
      return fail(hs.flags & 2 ? LGX_ERR_NONFINITE : LGX_ERR_BREAKDOWN,
                  "column " + std::to_string(hs.bad_col) + ": p.Ap is zero or non-finite");
  }
  for (int k = 0; k < K; ++k) {
    h_it[k] = hs.it_done[k];
    h_rel[k] = hs.r0[k] > 0.0 ? std::sqrt(hs.res2[k]) / hs.r0[k] : 0.0;
  }
  if (perm) {
    k_mpermute<<<egrid(nk), 256, 0, s>>>(n, perm, K, 1, X.p, d_x);
    LGX_LAUNCH_CHECK();
  } else {
    LGX_CUDA(cudaMemcpyAsync(d_x, X.p, sizeof(double) * nk, cudaMemcpyDeviceToDevice, s));
  }
  LGX_CUDA(cudaStreamSynchronize(s));
  if (hs.n_active > 0)
    return fail(LGX_ERR_NOT_CONVERGED, "maxit reached before every column converged");
  return LGX_OK;
}

}  // namespace lgx

using namespace lgx;

extern "C" {

lgx_status lgx_pcg_multi(const lgx_matrix *a, lgx_amg *amg, int32_t nrhs, const double *d_b,
                         double *d_x, double rtol, int64_t maxit, int use_graphs,
                         lgx_stream stream, int64_t *h_iterations, double *h_rel_residual) {
  if (!a || !amg) return fail(LGX_ERR_INVALID, "null matrix or hierarchy");
  if (nrhs < 1 || nrhs > kMaxRhs) return fail(LGX_ERR_INVALID, "nrhs must be in [1, 32]");
  if (a->kind != LGX_MATRIX_CSR || amg->lv.empty() || amg->lv[0]->a != &a->csr)
    return fail(LGX_ERR_INVALID, "the hierarchy was not built from this CSR matrix");
  if (a->n > 0 && (!d_b || !d_x)) return fail(LGX_ERR_INVALID, "null vector");
  std::vector<int64_t> it(nrhs, 0);
  std::vector<double> rel(nrhs, 0.0);
  lgx_status st = amg->f32 ? pcg_multi<float>(a, *amg, nrhs, d_b, d_x, rtol, maxit, use_graphs,
                                               stream, it.data(), rel.data())
                           : pcg_multi<double>(a, *amg, nrhs, d_b, d_x, rtol, maxit, use_graphs,
                                                stream, it.data(), rel.data());
  if (h_iterations) std::copy(it.begin(), it.end(), h_iterations);
  if (h_rel_residual) std::copy(rel.begin(), rel.end(), h_rel_residual);
  return st;
}

}  // extern "C"
