// Stationary smoothers: Jacobi (jacobi/sweep.hpp:66-87) and multicolour SOR,
// the GB300 replacement of the thread-block-hybrid SOR of
// gauss-seidel-variant/sweep.hpp:134-200, plus graph colouring.
//
// A multicolour sweep works on a copy of the matrix with its rows in colour order:
// colour c occupies the contiguous rows [offsets[c], offsets[c+1]), so every colour
// pass is a coalesced row-block kernel.  In the colour-permuted form (a colouring
// by itself, a hierarchy's finest level with a given colouring) the columns and the
// vectors are in that order too; in the natural-order form (the other levels of a
// hierarchy, lgx_colouring::natural) columns and vectors stay as they are, a list
// names the vector row of each matrix row, and sweeps from zero and the residuals
// after them run on halves of the rows.  Either way rows keep their original column
// order, hence each row sum is formed in exactly the order of the
// reference's scalar CSR path; the sweep equals the reference SOR run in the
// order "rows sorted by (colour, index)".
#include <cuda_runtime.h>

#include <algorithm>
#include <memory>
#include <cmath>
#include <vector>

#include "lgx_internal.cuh"
#include "lgx_rows.cuh"

namespace lgx {

// ---- Jacobi ----------------------------------------------------------------
template <typename VT>
struct JacobiOp {
  const double *x_in;  // nullptr: zero input vector
  double *x_out;
  const double *b;
  double relax, m1;
  using X = double;
  static constexpr bool kReduce = false;
  static constexpr bool kRounds = false;
  double *partials = nullptr;
  unsigned *counter = nullptr;
  template <int W, bool FLAT>
  __device__ __forceinline__ double row(int64_t i, const int32_t *c, const VT *v, int len) const {
    double accum = b[i], diag = 0.0;
    for (int k = 0; k < len; ++k) {
      const int32_t j = c[k];
      const double a = (double)v[k];
      if (j == i) {
        diag = a;
      } else {
        accum = fma(-a, x_in ? __ldg(x_in + j) : 0.0, accum);
      }
    }
    const double quot = accum / diag;
    x_out[i] = fma(relax, quot, m1 * (x_in ? x_in[i] : 0.0));
    return 0.0;
  }
  __device__ __forceinline__ void finish(double) const {}
};

// Jacobi from a zero start with a cached diagonal (stencil matrices):
// x = fma(relax, b / d, m1 * 0) -- the reference's arithmetic with x_in = 0.
__global__ void k_jacobi_diag_zero(int64_t n, const double *__restrict__ d, double relax,
                                   const double *__restrict__ b, double *__restrict__ x) {
  const double m1 = 1.0 - relax;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    x[i] = fma(relax, b[i] / d[i], m1 * 0.0);
}

// Stencil Jacobi with a general input: accum = b - sum_{j != i} a_ij x_j via
// y = A x (off-diagonal part: A x - d x would reorder the sum), so it is
// computed from the assembled rows; used through the CSR path instead.

// ---- graph colouring -----------------------------------------------------
__device__ __forceinline__ uint64_t splitmix(uint64_t seed, uint64_t i) {
  uint64_t z = seed * 0x9E3779B97F4A7C15ull + i + 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// Jones-Plassmann colouring (see the oracle's lo_colour_jp): in a round a vertex
// that beats all its uncoloured neighbours on (priority, index) takes the smallest
// colour its coloured neighbours leave, as they stood before the round.
//
// Bound by the rounds (64 for 27 entries a row): a colour is kept with its round, so
// that one launch a round can tell what the round wrote; a round's list holds the
// vertices still without a colour, each with a neighbour that beat it, and most look
// at that one alone.  G lanes share a row, 8 of them while many vertices are left and
// 32 below kJpWide, where a round is as long as one row's chain of loads.  With all
// rows in every round and the colours committed by a second launch, a setup and solve
// of 998400 rows of 27 entries took 110.8 ms, now 108.8 (rounds of the finest level
// 2.8 ms, of 6k to 170k rows 0.3 to 0.65).
constexpr int kJpRounds = 8;  // rounds between two looks of the host at what remains
constexpr int kJpWide = 32768;

// the colour of a vertex before `round`, negative while it had none (low half:
// colour, high half: its round; past L1, other vertices of the launch write)
__device__ __forceinline__ int32_t jp_colour(const int64_t *p, int32_t round) {
  int64_t v;
  asm volatile("ld.relaxed.gpu.global.s64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return (int32_t)(v >> 32) == round ? -1 : (int32_t)v;
}

template <int G, bool FIRST>
__global__ void __launch_bounds__(256) k_jp_round(
  int64_t n, const int64_t *__restrict__ rowptr, const int32_t *__restrict__ col, uint64_t seed,
  int64_t *state, int32_t round, unsigned long long *count, const int2 *__restrict__ list,
  int2 *__restrict__ rest) {
  __shared__ int2 kept[256 / G];
  __shared__ int nkept;
  __shared__ unsigned long long base;
  if (threadIdx.x == 0) nkept = 0;
  __syncthreads();
  const int64_t t = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
  const int lane = threadIdx.x % G;
  const unsigned group = G == 32 ? 0xffffffffu
                                 : ((1u << (G % 32)) - 1) << (threadIdx.x / G * G % 32);
  if (t < (FIRST ? n : (int64_t)count[0])) {
    int2 v = FIRST ? make_int2((int)t, -1) : list[t];
    const int64_t i = v.x;
    if (FIRST || jp_colour(state + v.y, round) >= 0) {
      v.y = -1;
      const int64_t b = rowptr[i], e = rowptr[i + 1];
      const uint64_t pi = splitmix(seed, (uint64_t)i);
      uint64_t used = 0;  // colours below 64
      for (int64_t k0 = b; k0 < e && v.y < 0; k0 += G) {
        const int64_t k = k0 + lane, j = k < e ? (int64_t)col[k] : i;
        bool beaten = false;
        if (j != i) {
          const int32_t cj = FIRST ? -1 : jp_colour(state + j, round);
          const uint64_t pj = splitmix(seed, (uint64_t)j);
          if (cj < 0) beaten = pj > pi || (pj == pi && j > i);
          else if (cj < 64) used |= 1ull << cj;
        }
        const unsigned m = __ballot_sync(group, beaten) & group;
        if (m) v.y = (int)__shfl_sync(group, (int)j, __ffs(m) - 1);
      }
      if (v.y < 0) {
        int32_t c = 0;
        for (int32_t c0 = 0;; c0 += 64) {
          if (c0) {
            used = 0;
            for (int64_t k = b + lane; k < e; k += G) {
              if (col[k] == i) continue;
              const int32_t cj = jp_colour(state + col[k], round) - c0;
              if (cj >= 0 && cj < 64) used |= 1ull << cj;
            }
          }
          const uint64_t lo = __reduce_or_sync(group, (unsigned)used);
          const uint64_t all = (uint64_t)__reduce_or_sync(group, (unsigned)(used >> 32)) << 32 | lo;
          c = c0 + __ffsll((long long)~all) - 1;
          if (~all) break;
        }
        if (lane == 0) {
          const int64_t w = (int64_t)round << 32 | c;
          asm volatile("st.relaxed.gpu.global.s64 [%0], %1;" ::"l"(state + i), "l"(w) : "memory");
        }
      }
    }
    if (v.y >= 0 && lane == 0) kept[atomicAdd(&nkept, 1)] = v;
  }
  __syncthreads();
  if (nkept == 0) return;
  if (threadIdx.x == 0) base = atomicAdd(count + 1, (unsigned long long)nkept);
  __syncthreads();
  if ((int)threadIdx.x < nkept) rest[base + threadIdx.x] = kept[threadIdx.x];
}

__global__ void __launch_bounds__(256) k_jp_colours(int64_t n, const int64_t *__restrict__ state,
                                                    int32_t *__restrict__ colour, int *maxc) {
  int top = -1;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    colour[i] = (int32_t)state[i];
    top = max(top, colour[i]);
  }
  top = __reduce_max_sync(0xffffffffu, top);
  if ((threadIdx.x & 31) == 0 && top >= 0) atomicMax(maxc, top);
}

lgx_status colouring_jp(const Csr &a, uint64_t seed, cudaStream_t s, DBuf<int32_t> &colour,
                        int32_t &ncolours) {
  const int64_t n = a.n;
  LGX_CHECK(colour.alloc(n));
  // states, two lists, the rounds' list lengths and the highest colour
  DBuf<int64_t> work;
  LGX_CHECK(work.alloc(3 * n + kJpRounds + 2));
  int64_t *state = work.p;
  int2 *list[2] = {reinterpret_cast<int2 *>(work.p + n), reinterpret_cast<int2 *>(work.p + 2 * n)};
  unsigned long long *count = reinterpret_cast<unsigned long long *>(work.p + 3 * n);
  int *maxc = reinterpret_cast<int *>(count + kJpRounds + 1);
  LGX_CUDA(cudaMemsetAsync(state, 0xFF, sizeof(int64_t) * n, s));
  LGX_CUDA(cudaMemsetAsync(maxc, 0xFF, sizeof(int), s));
  unsigned long long h_rem = (unsigned long long)n;
  int32_t round = 0;
  while (h_rem > 0) {
    // a round colours at least the first of the remaining vertices
    if (round > n) return fail(LGX_ERR_INVALID, "colouring did not terminate");
    LGX_CUDA(cudaMemcpyAsync(count, &h_rem, sizeof(h_rem), cudaMemcpyHostToDevice, s));
    LGX_CUDA(cudaMemsetAsync(count + 1, 0, sizeof(unsigned long long) * kJpRounds, s));
    const bool wide = h_rem < kJpWide;
    const unsigned g = (unsigned)((h_rem * (wide ? 32 : 8) + 255) / 256);
    for (int q = 0; q < kJpRounds; ++q, ++round) {
      auto *kern = round == 0 ? (wide ? k_jp_round<32, true> : k_jp_round<8, true>)
                              : (wide ? k_jp_round<32, false> : k_jp_round<8, false>);
      kern<<<g, 256, 0, s>>>(n, a.rowptr.p, a.col.p, seed, state, round, count + q,
                             list[round & 1], list[(round + 1) & 1]);
      LGX_LAUNCH_CHECK();
    }
    LGX_CUDA(cudaMemcpyAsync(&h_rem, count + kJpRounds, sizeof(h_rem), cudaMemcpyDeviceToHost, s));
    LGX_CUDA(cudaStreamSynchronize(s));
  }
  if (n > 0) {
    k_jp_colours<<<(unsigned)std::min<int64_t>(grid_for(n, 256), 16384), 256, 0, s>>>(
        n, state, colour.p, maxc);
    LGX_LAUNCH_CHECK();
  }
  int h_max = -1;
  LGX_CUDA(cudaMemcpyAsync(&h_max, maxc, sizeof(int), cudaMemcpyDeviceToHost, s));
  LGX_CUDA(cudaStreamSynchronize(s));
  ncolours = h_max + 1;
  return LGX_OK;
}

__global__ void k_colour_flag(int64_t n, const int32_t *colour, int32_t c, int64_t *flag,
                              int *bad, int32_t ncolours) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t ci = colour[i];
    if (c == 0 && (ci < 0 || ci >= ncolours)) atomicOr(bad, 1);
    flag[i] = ci == c;
  }
}

__global__ void k_colour_place(int64_t n, const int32_t *colour, int32_t c, const int64_t *pos,
                               int64_t base, int32_t *perm, int32_t *iperm) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    if (colour[i] != c) continue;
    const int64_t p = base + pos[i];
    perm[p] = (int32_t)i;
    iperm[i] = (int32_t)p;
  }
}

// The row order of up to kSortColours colours as one stable counting sort: rows
// in blocks of kSortRows, counts per colour and block (table[c * blocks + block]),
// their prefix sums, placement.  Bound by latency (three launches and a prefix sum);
// a flag, a scan and a placement per colour with a host round trip each took, with
// the rounds of the colouring before it, 2.4 ms on a level of 32k rows and 16
// colours, now 1.65.  More colours than a block's counters hold keep the passes.
constexpr int kSortColours = 64, kSortRows = 1024;

__global__ void __launch_bounds__(256) k_colour_count(int64_t n, const int32_t *__restrict__ colour,
                                                      int32_t ncolours, int64_t blocks,
                                                      int64_t *__restrict__ table, int *bad) {
  __shared__ int count[kSortColours];
  if (threadIdx.x < kSortColours) count[threadIdx.x] = 0;
  __syncthreads();
  const int64_t i0 = (int64_t)blockIdx.x * kSortRows;
  for (int64_t i = i0 + threadIdx.x; i < i0 + kSortRows && i < n; i += 256) {
    const int32_t c = colour[i];
    if (c < 0 || c >= ncolours) atomicOr(bad, 1);
    else atomicAdd(&count[c], 1);
  }
  __syncthreads();
  if ((int)threadIdx.x < ncolours) table[threadIdx.x * blocks + blockIdx.x] = count[threadIdx.x];
}

__global__ void __launch_bounds__(256) k_colour_sort(int64_t n, const int32_t *__restrict__ colour,
                                                     int32_t ncolours, int64_t blocks,
                                                     const int64_t *__restrict__ start,
                                                     int32_t *__restrict__ perm,
                                                     int32_t *__restrict__ iperm) {
  __shared__ int64_t at[kSortColours];
  __shared__ int count[8][kSortColours];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if ((int)threadIdx.x < ncolours) at[threadIdx.x] = start[threadIdx.x * blocks + blockIdx.x];
  const int64_t i0 = (int64_t)blockIdx.x * kSortRows;
  for (int64_t base = i0; base < i0 + kSortRows && base < n; base += 256) {
    for (int k = threadIdx.x; k < 8 * kSortColours; k += 256) (&count[0][0])[k] = 0;
    __syncthreads();
    const int64_t i = base + threadIdx.x;
    int32_t c = i < n ? colour[i] : -1;
    if (c >= ncolours) c = -1;
    const unsigned same = __match_any_sync(0xffffffffu, c);
    const int rank = __popc(same & ((1u << lane) - 1));
    if (c >= 0 && rank == 0) count[w][c] = __popc(same);
    __syncthreads();
    if (c >= 0) {
      int64_t p = at[c] + rank;
      for (int v = 0; v < w; ++v) p += count[v][c];
      perm[p] = (int32_t)i;
      iperm[i] = (int32_t)p;
    }
    __syncthreads();
    if ((int)threadIdx.x < ncolours)
      for (int v = 0; v < 8; ++v) at[threadIdx.x] += count[v][threadIdx.x];
    __syncthreads();
  }
}

// adjacent rows must not share a colour
__global__ void k_colour_validate(int64_t n, const int64_t *rowptr, const int32_t *col,
                                  const int32_t *colour, int *bad) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    for (int64_t k = rowptr[i]; k < rowptr[i + 1]; ++k)
      if (col[k] != i && colour[col[k]] == colour[i]) atomicOr(bad, 2);
}

__global__ void k_perm_rowlen(int64_t n, const int64_t *rowptr, const int32_t *perm,
                              int64_t *len) {
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n;
       r += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = perm[r];
    len[r] = rowptr[i + 1] - rowptr[i];
  }
}

// one warp per permuted row: the row's entries copy coalesced (a thread
// per row walked 32 scattered rows per warp instruction: 216 GB/s at 256^3)
template <typename VT>
__global__ void k_perm_fill(int64_t n, const int64_t *rowptr, const int32_t *col, const VT *val,
                            const int32_t *perm, const int32_t *iperm, const int64_t *prowptr,
                            int32_t *pcol, VT *pval) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; r < n; r += nw) {
    const int64_t i = perm[r];
    const int64_t b = rowptr[i], len = rowptr[i + 1] - b, o = prowptr[r];
    for (int64_t k = lane; k < len; k += 32) {
      pcol[o + k] = iperm[col[b + k]];
      pval[o + k] = val[b + k];
    }
  }
}

// Reciprocal of every permuted row's diagonal, rounded once by the IEEE
// division; 0 marks rows whose diagonal lies outside [2^-400, 2^400] in
// magnitude (or is not finite), where the sweep divides directly.
template <typename VT>
__global__ void k_colour_rdiag(int64_t n, const int64_t *rowptr, const int32_t *col,
                               const VT *val, double *rdiag, double *pdiag) {
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n;
       r += (int64_t)gridDim.x * blockDim.x) {
    double d = 0.0;
    for (int64_t k = rowptr[r]; k < rowptr[r + 1]; ++k)
      if (col[k] == r) d = (double)val[k];
    pdiag[r] = d;
    if (rdiag) {
      const int e = (int)((__double_as_longlong(d) >> 52) & 0x7ff);
      rdiag[r] = (e > 1023 - 400 && e < 1023 + 400) ? 1.0 / d : 0.0;
    }
  }
}

__global__ void k_to_f32(int64_t n, const double *src, float *dst) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    dst[i] = (float)src[i];
}

// the colours checked and the row order they give (perm, iperm, offsets);
// `flag` holds n int64 of scratch for the caller afterwards
static lgx_status colouring_order(const Csr &a, const int32_t *d_colour, int32_t ncolours,
                                  cudaStream_t s, lgx_colouring &out, DBuf<int64_t> &flag) {
  const int64_t n = a.n;
  if (ncolours < 1 && n > 0) return fail(LGX_ERR_INVALID, "colouring needs at least one colour");
  out.n = n;
  out.ncolours = ncolours;
  if (out.colour.p != d_colour) {
    LGX_CHECK(out.colour.alloc(n));
    LGX_CUDA(cudaMemcpyAsync(out.colour.p, d_colour, sizeof(int32_t) * n,
                             cudaMemcpyDeviceToDevice, s));
  }
  LGX_CHECK(out.perm.alloc(n));
  LGX_CHECK(out.iperm.alloc(n));
  DBuf<int64_t> pos;
  DBuf<int> bad;
  LGX_CHECK(flag.alloc(n));
  LGX_CHECK(bad.alloc(1));
  LGX_CUDA(cudaMemsetAsync(bad.p, 0, sizeof(int), s));
  const unsigned g = (unsigned)std::min<int64_t>(grid_for(n, 256), 16384);
  out.offsets.assign((size_t)ncolours + 1, 0);
  int64_t base = 0;
  if (n > 0 && ncolours <= kSortColours) {
    const int64_t blocks = (n + kSortRows - 1) / kSortRows, entries = ncolours * blocks;
    DBuf<int64_t> table;
    LGX_CHECK(table.alloc(entries));
    LGX_CHECK(pos.alloc(entries + 1));
    k_colour_count<<<(unsigned)blocks, 256, 0, s>>>(n, out.colour.p, ncolours, blocks, table.p,
                                                    bad.p);
    LGX_LAUNCH_CHECK();
    LGX_CHECK(inclusive_offsets(entries, table.p, pos.p, s));
    k_colour_sort<<<(unsigned)blocks, 256, 0, s>>>(n, out.colour.p, ncolours, blocks, pos.p,
                                                   out.perm.p, out.iperm.p);
    LGX_LAUNCH_CHECK();
    // the colours' first entries of the prefix sums, and the total
    LGX_CUDA(cudaMemcpy2DAsync(out.offsets.data(), sizeof(int64_t), pos.p,
                               sizeof(int64_t) * (size_t)blocks, sizeof(int64_t),
                               (size_t)ncolours, cudaMemcpyDeviceToHost, s));
    LGX_CUDA(cudaMemcpyAsync(&base, pos.p + entries, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    LGX_CUDA(cudaStreamSynchronize(s));
  } else {
    LGX_CHECK(pos.alloc(n + 1));
    for (int32_t c = 0; c < ncolours; ++c) {
      k_colour_flag<<<g, 256, 0, s>>>(n, out.colour.p, c, flag.p, bad.p, ncolours);
      LGX_LAUNCH_CHECK();
      LGX_CHECK(inclusive_offsets(n, flag.p, pos.p, s));
      k_colour_place<<<g, 256, 0, s>>>(n, out.colour.p, c, pos.p, base, out.perm.p, out.iperm.p);
      LGX_LAUNCH_CHECK();
      int64_t cnt = 0;
      LGX_CUDA(cudaMemcpyAsync(&cnt, pos.p + n, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
      LGX_CUDA(cudaStreamSynchronize(s));
      out.offsets[c] = base;
      base += cnt;
    }
  }
  out.offsets[ncolours] = base;
  k_colour_validate<<<g, 256, 0, s>>>(n, a.rowptr.p, a.col.p, out.colour.p, bad.p);
  LGX_LAUNCH_CHECK();
  int h_bad = 0;
  LGX_CUDA(cudaMemcpyAsync(&h_bad, bad.p, sizeof(int), cudaMemcpyDeviceToHost, s));
  LGX_CUDA(cudaStreamSynchronize(s));
  if (h_bad & 1) return fail(LGX_ERR_INVALID, "colour index out of range");
  if (h_bad & 2) return fail(LGX_ERR_INVALID, "adjacent rows share a colour");
  if (base != n) return fail(LGX_ERR_INVALID, "colouring does not cover every row");
  return LGX_OK;
}

lgx_status colouring_build(const Csr &a, const int32_t *d_colour, int32_t ncolours,
                           cudaStream_t s, lgx_colouring &out) {
  DBuf<int64_t> flag;
  LGX_CHECK(colouring_order(a, d_colour, ncolours, s, out, flag));
  const int64_t n = a.n;
  const unsigned g = (unsigned)std::min<int64_t>(grid_for(n, 256), 16384);
  // permuted CSR
  Csr &p = out.pcsr;
  p.n = n;
  p.nnz = a.nnz;
  p.symmetric = a.symmetric;
  p.storage = a.storage;
  p.max_row = a.max_row;
  LGX_CHECK(p.rowptr.alloc(n + 3));  // +2: staged row-offset spans
  LGX_CHECK(csr_alloc_arrays(p, a.nnz, a.storage));
  k_perm_rowlen<<<g, 256, 0, s>>>(n, a.rowptr.p, out.perm.p, flag.p);
  LGX_LAUNCH_CHECK();
  LGX_CHECK(inclusive_offsets(n, flag.p, p.rowptr.p, s));
  if (a.storage == LGX_F64) {
    k_perm_fill<double><<<g, 256, 0, s>>>(n, a.rowptr.p, a.col.p, a.v64.p, out.perm.p,
                                          out.iperm.p, p.rowptr.p, p.col.p, p.v64.p);
  } else {
    k_perm_fill<float><<<g, 256, 0, s>>>(n, a.rowptr.p, a.col.p, a.v32.p, out.perm.p, out.iperm.p,
                                         p.rowptr.p, p.col.p, p.v32.p);
  }
  LGX_LAUNCH_CHECK();
  if (n > 0) {
    LGX_CHECK(out.pdiag.alloc(n));
    if (a.storage == LGX_F64) {
      LGX_CHECK(out.rdiag.alloc(n));
      k_colour_rdiag<double><<<g, 256, 0, s>>>(n, p.rowptr.p, p.col.p, p.v64.p, out.rdiag.p,
                                               out.pdiag.p);
    } else {
      k_colour_rdiag<float><<<g, 256, 0, s>>>(n, p.rowptr.p, p.col.p, p.v32.p, nullptr,
                                              out.pdiag.p);
    }
    LGX_LAUNCH_CHECK();
  }
  return csr_compute_max_window(p, s);
}

// entries of each row in earlier (lo, by colour order) and later (up, by
// natural order) colours, and the whole row's length (by colour order)
__global__ void k_half_count(int64_t n, const int64_t *__restrict__ rowptr,
                             const int32_t *__restrict__ col, const int32_t *__restrict__ perm,
                             const int32_t *__restrict__ colour, int64_t *len, int64_t *lo_len,
                             int64_t *up_len) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; r < n; r += nw) {
    const int64_t i = perm[r];
    const int64_t b = rowptr[i], m = rowptr[i + 1] - b;
    const int32_t ci = colour[i];
    int lo = 0, up = 0;
    for (int64_t k = lane; k < m; k += 32) {
      const int32_t cj = colour[col[b + k]];
      lo += cj < ci;
      up += cj > ci;
    }
    lo = __reduce_add_sync(0xffffffffu, lo);
    up = __reduce_add_sync(0xffffffffu, up);
    if (lane == 0) {
      len[r] = m;
      lo_len[r] = lo;
      up_len[i] = up;
    }
  }
}

template <typename T>
struct RowsOut {
  const int64_t *ptr;
  int32_t *col;
  T *val;
};

// the rows and their halves, a warp per row, entries in row order; the
// diagonal and (FP64 values) its reciprocal as k_colour_rdiag gives them
template <typename VT, typename OT>
__global__ void k_half_fill(int64_t n, const int64_t *__restrict__ rowptr,
                            const int32_t *__restrict__ col, const VT *__restrict__ val,
                            const int32_t *__restrict__ perm, const int32_t *__restrict__ colour,
                            RowsOut<OT> full, RowsOut<OT> lo, RowsOut<OT> up, double *pdiag,
                            double *rdiag) {
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; r < n; r += nw) {
    const int64_t i = perm[r];
    const int64_t b = rowptr[i], m = rowptr[i + 1] - b;
    const int32_t ci = colour[i];
    int64_t o = full.ptr[r], ol = lo.ptr[r], ou = up.ptr[i];
    for (int64_t k0 = 0; k0 < m; k0 += 32) {
      const int64_t k = k0 + lane;
      const bool in = k < m;
      const int32_t c = in ? col[b + k] : 0;
      const VT v = in ? val[b + k] : VT(0);
      const int32_t cj = in ? colour[c] : ci;
      const bool is_lo = cj < ci, is_up = cj > ci;
      const unsigned ml = __ballot_sync(0xffffffffu, is_lo), mu = __ballot_sync(0xffffffffu, is_up);
      if (in) {
        full.col[o + k] = c;
        full.val[o + k] = (OT)v;
        if (c == i) {
          const double d = (double)v;
          pdiag[r] = d;
          if (rdiag) {
            const int e = (int)((__double_as_longlong(d) >> 52) & 0x7ff);
            rdiag[r] = (e > 1023 - 400 && e < 1023 + 400) ? 1.0 / d : 0.0;
          }
        }
      }
      if (is_lo) {
        const int64_t at = ol + __popc(ml & below);
        lo.col[at] = c;
        lo.val[at] = (OT)v;
      }
      if (is_up) {
        const int64_t at = ou + __popc(mu & below);
        up.col[at] = c;
        up.val[at] = (OT)v;
      }
      ol += __popc(ml);
      ou += __popc(mu);
    }
  }
}

template <typename OT>
static RowsOut<OT> rows_out(Csr &a) {
  if constexpr (sizeof(OT) == 8) return {a.rowptr.p, a.col.p, a.v64.p};
  else return {a.rowptr.p, a.col.p, a.v32.p};
}

lgx_status colouring_build_natural(const Csr &a, const int32_t *d_colour, int32_t ncolours,
                                   bool f32, cudaStream_t s, lgx_colouring &out) {
  DBuf<int64_t> len, lo_len, up_len;
  LGX_CHECK(colouring_order(a, d_colour, ncolours, s, out, len));
  const int64_t n = a.n;
  const lgx_dtype storage = f32 ? LGX_F32 : a.storage;
  out.natural = true;
  LGX_CHECK(lo_len.alloc(n));
  LGX_CHECK(up_len.alloc(n));
  // a warp per row
  const unsigned g = (unsigned)std::min<int64_t>(grid_for(std::max<int64_t>(n, 1) * 32, 256), 16384);
  if (n > 0) {
    k_half_count<<<g, 256, 0, s>>>(n, a.rowptr.p, a.col.p, out.perm.p, out.colour.p, len.p,
                                   lo_len.p, up_len.p);
    LGX_LAUNCH_CHECK();
  }
  Csr *list[3] = {&out.pcsr, &out.lo, &out.up};
  const int64_t *lens[3] = {len.p, lo_len.p, up_len.p};
  int64_t nnz[3] = {0, 0, 0};
  for (int k = 0; k < 3; ++k) {
    list[k]->n = n;
    list[k]->symmetric = k == 0 ? a.symmetric : 0;
    list[k]->storage = storage;
    LGX_CHECK(list[k]->rowptr.alloc(n + 3));  // +2: staged row-offset spans
    LGX_CHECK(inclusive_offsets(n, lens[k], list[k]->rowptr.p, s));
    LGX_CUDA(cudaMemcpyAsync(&nnz[k], list[k]->rowptr.p + n, sizeof(int64_t),
                             cudaMemcpyDeviceToHost, s));
  }
  LGX_CHECK(csr_compute_extents(list, 3, s));  // synchronises: nnz has arrived
  for (int k = 0; k < 3; ++k) {
    list[k]->nnz = nnz[k];
    LGX_CHECK(csr_alloc_arrays(*list[k], nnz[k], storage));
  }
  if (n == 0) return LGX_OK;
  // (0 stands where a row stored no diagonal, as k_colour_rdiag has it: such a row
  // divides by 0.  Matrices without one are refused where they are created.)
  LGX_CHECK(out.pdiag.alloc(n));
  LGX_CUDA(cudaMemsetAsync(out.pdiag.p, 0, sizeof(double) * (size_t)n, s));
  if (storage == LGX_F64) {
    LGX_CHECK(out.rdiag.alloc(n));
    LGX_CUDA(cudaMemsetAsync(out.rdiag.p, 0, sizeof(double) * (size_t)n, s));
    k_half_fill<double, double><<<g, 256, 0, s>>>(
      n, a.rowptr.p, a.col.p, a.v64.p, out.perm.p, out.colour.p, rows_out<double>(out.pcsr),
      rows_out<double>(out.lo), rows_out<double>(out.up), out.pdiag.p, out.rdiag.p);
  } else if (a.storage == LGX_F64) {
    k_half_fill<double, float><<<g, 256, 0, s>>>(
      n, a.rowptr.p, a.col.p, a.v64.p, out.perm.p, out.colour.p, rows_out<float>(out.pcsr),
      rows_out<float>(out.lo), rows_out<float>(out.up), out.pdiag.p, nullptr);
  } else {
    k_half_fill<float, float><<<g, 256, 0, s>>>(
      n, a.rowptr.p, a.col.p, a.v32.p, out.perm.p, out.colour.p, rows_out<float>(out.pcsr),
      rows_out<float>(out.lo), rows_out<float>(out.up), out.pdiag.p, nullptr);
  }
  LGX_LAUNCH_CHECK();
  return LGX_OK;
}

lgx_status colouring_make_f32(lgx_colouring &c, cudaStream_t s) {
  if (c.pcsr.storage == LGX_F32 || c.pv32.p) return LGX_OK;
  LGX_CHECK(c.pv32.alloc(c.pcsr.nnz + kCsrPad));
  k_to_f32<<<std::min<int64_t>(grid_for(c.pcsr.nnz, 256), 16384), 256, 0, s>>>(
    c.pcsr.nnz, c.pcsr.v64.p, c.pv32.p);
  LGX_LAUNCH_CHECK();
  return LGX_OK;
}

// bfloat16 copy of the permuted values scaled by the row's diagonal:
// pv16 = bf16(a_ij / a_ii) (the diagonal becomes exactly 1), pscale = a_ii.
// Rows without a nonzero diagonal keep scale 1 and bf16(a_ij).
template <typename VT>
__global__ void k_to_bf16_scaled(int64_t n, const int64_t *rowptr, const int32_t *col,
                                 const VT *val, bf16 *out, float *scale) {
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n;
       r += (int64_t)gridDim.x * blockDim.x) {
    double d = 0.0;
    for (int64_t k = rowptr[r]; k < rowptr[r + 1]; ++k)
      if (col[k] == r) d = (double)val[k];
    const bool use = d != 0.0 && isfinite(d);
    for (int64_t k = rowptr[r]; k < rowptr[r + 1]; ++k)
      out[k] = __float2bfloat16_rn((float)(use ? (double)val[k] / d : (double)val[k]));
    scale[r] = use ? (float)d : 1.0f;
  }
}

lgx_status colouring_make_bf16(lgx_colouring &c, cudaStream_t s) {
  if (c.pv16.p) return LGX_OK;
  const Csr &p = c.pcsr;
  LGX_CHECK(c.pv16.alloc(p.nnz + kCsrPad));
  LGX_CHECK(c.pscale.alloc(std::max<int64_t>(p.n, 1)));
  if (p.n == 0) return LGX_OK;
  const unsigned g = (unsigned)std::min<int64_t>(grid_for(p.n, 256), 16384);
  if (p.storage == LGX_F64)
    k_to_bf16_scaled<double><<<g, 256, 0, s>>>(p.n, p.rowptr.p, p.col.p, p.v64.p, c.pv16.p,
                                               c.pscale.p);
  else
    k_to_bf16_scaled<float><<<g, 256, 0, s>>>(p.n, p.rowptr.p, p.col.p, p.v32.p, c.pv16.p,
                                              c.pscale.p);
  LGX_LAUNCH_CHECK();
  return LGX_OK;
}

// ---- multicolour SOR -------------------------------------------------------
// One row of gauss-seidel-variant/sweep.hpp:134-200 in place: rows of other
// colours already visited in this sweep hold their new values in x, the rest
// their input values; rows of the same colour are never adjacent.
// With rdiag (FP64 values and vectors) the regular row divides through the
// reciprocal table (same quotient), and relax == 1 skips the (1 - relax) x_i
// term where it cannot change the result (q nonzero, x_i finite).
// accum / diag by the row's formula, the sweep's last step: x_i from the
// accumulated sum, with y the reciprocal table's entry (0: divide)
template <typename XT>
__device__ __forceinline__ XT sor_value(XT accum, XT diag, XT xi, double y, XT relax, XT m1,
                                        int ultra, int relax_one) {
  if (ultra) return xi + relax * accum / fabs(diag);
  XT quot;
  if constexpr (sizeof(XT) == 8) {
    quot = (nonzero_bits(y) && exponent_within_400(accum)) ? div_by_recip(accum, diag, y)
                                                           : accum / diag;
    // fma(1, q, 0 * x_i) == q for nonzero q and finite x_i
    if (relax_one && nonzero_bits(quot) && exponent_field(xi) != 0x7ff) return quot;
  } else {
    quot = accum / diag;
  }
  return fma(relax, quot, m1 * xi);
}

template <typename VT, typename XT>
struct SorOp {
  const XT *b;
  XT *x;
  XT relax, m1;
  int ultra;
  const double *rdiag = nullptr;
  int relax_one = 0;
  // forward sweep from x = 0 without clearing x first: rows of colours not
  // yet visited in this sweep (index >= visit_end) read as 0, this row too
  int from_zero = 0;
  int64_t visit_end = 0;
  const float *scale = nullptr;  // bfloat16 values: row factor (the diagonal)
  const int32_t *rows = nullptr;  // natural-order levels: vector row of each matrix row
  using X = XT;
  static constexpr bool kReduce = false;
  static constexpr bool kList = true;
  static constexpr bool kBranchForm = !kIsBf16<VT>;
  static constexpr int kTuneClass = 1;
  double *partials = nullptr;
  unsigned *counter = nullptr;
  template <int W, bool FLAT>
  __device__ __forceinline__ double row(int64_t r, int32_t i, const int32_t *c, const VT *v,
                                        int len) const {
    if constexpr (kIsBf16<VT>) {
      return row_scaled<W>(i, c, v, len);
    }
    XT accum = b[i], diag = XT(0);
    const XT xi = from_zero ? XT(0) : x[i];
    const int64_t end = from_zero ? visit_end : INT64_MAX;
    // constant, so it loads with the row's first loads
    const double y = sizeof(XT) == 8 && rdiag ? rdiag[r] : 0.0;
    for (int k = 0; k < len; k += W) {
      const int m = len - k;
      int32_t cc[W];
      XT xv[W];
      if constexpr (FLAT) {
        row_columns<W>(c, k, len, cc);
#pragma unroll
        for (int u = 0; u < W; ++u) ld_if(xv[u], x + cc[u], u < m && cc[u] != i && cc[u] < end);
      } else {
#pragma unroll
        for (int u = 0; u < W; ++u)
          if (u < m) {
            cc[u] = c[k + u];
            xv[u] = cc[u] < end ? x[cc[u]] : XT(0);
          }
      }
#pragma unroll
      for (int u = 0; u < W; ++u) {
        if (u < m) {
          const XT a = cvt<XT>(v[k + u]);
          if (cc[u] == i) {
            diag = a;
            if (ultra) accum = fma(-a, xi, accum);
          } else {
            accum = fma(-a, xv[u], accum);
          }
        }
      }
    }
    x[i] = sor_value<XT>(accum, diag, xi, y, relax, m1, ultra, relax_one);
    return 0.0;
  }
  // the row from gathered entries (natural-order rows, xs[k] = x[c[k]])
  static constexpr int kLongRow = 16;  // entries on average (launch_rows)
  bool spread() const { return rows && !from_zero; }
  struct Pre {
    XT b, xi;
    double y;
  };
  __device__ __forceinline__ Pre begin(int64_t r, int32_t i) const {
    return {b[i], x[i], sizeof(XT) == 8 && rdiag ? rdiag[r] : 0.0};
  }
  __device__ __forceinline__ void staged(const Pre &p, int32_t i, const int32_t *c, const VT *v,
                                         const XT *xs, int len) const {
    XT accum = p.b, diag = XT(0);
#pragma unroll 4
    for (int k = 0; k < len; ++k) {
      const XT a = cvt<XT>(v[k]);
      const bool own = c[k] == i;
      if (own) diag = a;
      if (!own || ultra) accum = fma(-a, xs[k], accum);
    }
    x[i] = sor_value<XT>(accum, diag, p.xi, p.y, relax, m1, ultra, relax_one);
  }
  // bfloat16 values v with a_ij = s_i v_ij: accum = b_i - s_i sum_{j != i} v_ij x_j,
  // a_ii = s_i v_ii (float arithmetic; a precision-form smoother, not the
  // reference's bits)
  template <int W>
  __device__ __forceinline__ double row_scaled(int64_t i, const int32_t *c, const VT *v,
                                               int len) const {
    const XT si = scale[i];
    const XT xi = from_zero ? XT(0) : x[i];
    XT t = XT(0), vd = XT(0);
    const int64_t end = from_zero ? visit_end : INT64_MAX;
    for (int k = 0; k < len; k += W) {
      const int m = len - k;
      int32_t cc[W];
      XT xv[W];
      row_columns<W>(c, k, len, cc);
#pragma unroll
      for (int u = 0; u < W; ++u) ld_if(xv[u], x + cc[u], u < m && cc[u] != i && cc[u] < end);
#pragma unroll
      for (int u = 0; u < W; ++u) {
        if (u < m) {
          const XT a = cvt<XT>(v[k + u]);
          if (cc[u] == i) {
            vd = a;
          } else {
            t = fma(a, xv[u], t);
          }
        }
      }
    }
    const XT diag = si * vd;
    XT accum = fma(-si, t, b[i]);
    if (ultra) {
      accum = fma(-diag, xi, accum);
      x[i] = xi + relax * accum / fabs(diag);
    } else {
      x[i] = fma(relax, accum / diag, m1 * xi);
    }
    return 0.0;
  }
  __device__ __forceinline__ void finish(double) const {}
};

// One colour of a forward sweep from x = 0 on the rows' earlier-colour halves
// (lgx_colouring::lo): what SorOp does with the entries of colours not yet
// visited reading 0, whose products leave the sum as it is.
template <typename VT, typename XT>
struct SorLoOp {
  const XT *b;
  XT *x;
  XT relax, m1;
  int ultra, relax_one;
  const double *pdiag, *rdiag;
  const int32_t *rows;
  using X = XT;
  static constexpr bool kReduce = false;
  static constexpr bool kList = true;
  static constexpr int kTuneClass = 1;
  double *partials = nullptr;
  unsigned *counter = nullptr;
  template <int W, bool FLAT>
  __device__ __forceinline__ double row(int64_t r, int32_t i, const int32_t *c, const VT *v,
                                        int len) const {
    const double y = sizeof(XT) == 8 && rdiag ? rdiag[r] : 0.0;
    const XT diag = (XT)pdiag[r];
    XT accum = b[i];
    for (int k = 0; k < len; k += W) {
      const int m = len - k;
      int32_t cc[W];
      XT xv[W];
      row_columns<W>(c, k, len, cc);
#pragma unroll
      for (int u = 0; u < W; ++u) ld_if(xv[u], x + cc[u], u < m);
#pragma unroll
      for (int u = 0; u < W; ++u)
        if (u < m) accum = fma(-cvt<XT>(v[k + u]), xv[u], accum);
    }
    x[i] = sor_value<XT>(accum, diag, XT(0), y, relax, m1, ultra, relax_one);
    return 0.0;
  }
  static constexpr int kLongRow = 8;  // half rows
  bool spread() const { return rows != nullptr; }
  struct Pre {
    XT b, diag;
    double y;
  };
  __device__ __forceinline__ Pre begin(int64_t r, int32_t i) const {
    return {b[i], (XT)pdiag[r], sizeof(XT) == 8 && rdiag ? rdiag[r] : 0.0};
  }
  __device__ __forceinline__ void staged(const Pre &p, int32_t i, const int32_t *, const VT *v,
                                         const XT *xs, int len) const {
    XT accum = p.b;
#pragma unroll 4
    for (int k = 0; k < len; ++k) accum = fma(-cvt<XT>(v[k]), xs[k], accum);
    x[i] = sor_value<XT>(accum, p.diag, XT(0), p.y, relax, m1, ultra, relax_one);
  }
  __device__ __forceinline__ void finish(double) const {}
};

// r = -U x (mc_up_residual) / r = b - A x on listed rows (mc_residual)
template <typename VT, typename XT, bool UP>
struct ListResidualOp {
  const XT *b, *x;
  XT *r;
  const int32_t *rows;
  using X = XT;
  static constexpr bool kReduce = false;
  static constexpr bool kList = true;
  double *partials = nullptr;
  unsigned *counter = nullptr;
  template <int W, bool FLAT>
  __device__ __forceinline__ double row(int64_t, int32_t i, const int32_t *c, const VT *v,
                                        int len) const {
    const XT ax = row_dot<W, FLAT, VT, XT>(c, v, len, x, XT(0));
    r[i] = UP ? -ax : b[i] - ax;
    return 0.0;
  }
  bool spread() const { return rows != nullptr; }
  struct Pre {
    XT b;
  };
  __device__ __forceinline__ Pre begin(int64_t, int32_t i) const { return {UP ? XT(0) : b[i]}; }
  __device__ __forceinline__ void staged(const Pre &p, int32_t i, const int32_t *, const VT *v,
                                         const XT *xs, int len) const {
    XT ax = XT(0);
#pragma unroll 4
    for (int k = 0; k < len; ++k) ax = fma(cvt<XT>(v[k]), xs[k], ax);
    r[i] = UP ? -ax : p.b - ax;
  }
  __device__ __forceinline__ void finish(double) const {}
};

// r = -U x on whole rows in colour order: row i's entries of later colours are
// those right of i (no two rows of a colour are neighbours)
template <typename VT, typename XT>
struct LaterResidualOp {
  const XT *x;
  XT *r;
  using X = XT;
  static constexpr bool kReduce = false;
  double *partials = nullptr;
  unsigned *counter = nullptr;
  template <int W, bool FLAT>
  __device__ __forceinline__ double row(int64_t i, const int32_t *c, const VT *v, int len) const {
    XT ax = XT(0);
    for (int k = 0; k < len; k += W) {
      int32_t cc[W];
      XT xv[W];
      row_columns<W>(c, k, len, cc);
#pragma unroll
      for (int u = 0; u < W; ++u) ld_if(xv[u], x + cc[u], k + u < len && cc[u] > i);
#pragma unroll
      for (int u = 0; u < W; ++u)
        if (k + u < len && cc[u] > i) ax = fma(cvt<XT>(v[k + u]), xv[u], ax);
    }
    r[i] = -ax;
    return 0.0;
  }
  __device__ __forceinline__ void finish(double) const {}
};

// First colour of a forward sweep from x = 0: every neighbour still reads 0,
// so the row's products with them leave accum = b_i (an fma with a zero
// product; where only the sign of a zero could differ, the row's result is
// +0 either way) and the row needs only b_i and its diagonal: 32 bytes per
// row instead of the whole row.  Same quotient and update as SorOp.
template <typename VT, typename XT>
__global__ void k_sor_first_colour(int64_t rb, int64_t re, const double *__restrict__ pdiag,
                                   const double *__restrict__ rdiag,
                                   const float *__restrict__ scale,
                                   const int32_t *__restrict__ rows, const XT *__restrict__ b,
                                   XT *__restrict__ x, XT relax, XT m1, int ultra,
                                   int relax_one) {
  pdl_trigger();
  pdl_wait();
  for (int64_t r = rb + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < re;
       r += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = rows ? rows[r] : r;
    const XT accum = b[i];
    XT diag;
    if constexpr (kIsBf16<VT>) {
      diag = scale[i];  // s_i * v_ii with v_ii = 1 (scaled by the diagonal)
    } else {
      diag = (XT)pdiag[r];
    }
    const double y = sizeof(XT) == 8 && !kIsBf16<VT> && rdiag ? rdiag[r] : 0.0;
    x[i] = sor_value<XT>(accum, diag, XT(0), y, relax, m1, ultra, relax_one);
  }
}

template <typename VT, typename XT>
lgx_status mc_sor_sweep(const lgx_colouring &c, const VT *val, double relax, int forward,
                        int ultra, const XT *b, XT *x, cudaStream_t s, int from_zero,
                        const float *scale, XT *r_last, int64_t *res_from) {
  if (res_from) *res_from = c.n;
  const Csr &p = c.pcsr;
  SorOp<VT, XT> op{b, x, (XT)relax, XT(1) - (XT)relax, ultra};
  op.scale = scale;
  op.rows = c.natural ? c.perm.p : nullptr;
  if (kIsBf16<VT> && c.natural)
    return fail(LGX_ERR_UNSUPPORTED, "natural-order levels have no bfloat16 values");
  if (kIsBf16<VT> && !scale) return fail(LGX_ERR_INVALID, "bfloat16 values need row scales");
  if constexpr (sizeof(VT) == 8 && sizeof(XT) == 8) {
    op.rdiag = c.rdiag.p;
    op.relax_one = relax == 1.0;
  }
  op.from_zero = from_zero && forward;
  if (from_zero && !forward && c.n > 0)
    LGX_CUDA(cudaMemsetAsync(x, 0, sizeof(XT) * c.n, s));
  for (int32_t k = 0; k < c.ncolours; ++k) {
    const int32_t col_id = forward ? k : c.ncolours - 1 - k;
    const int64_t rb = c.offsets[col_id], re = c.offsets[col_id + 1];
    if (op.from_zero && k == 0 && c.pdiag.p) {
      if (re > rb) {
        const unsigned g = (unsigned)std::min<int64_t>(grid_for(re - rb, 256), 16384);
        LGX_CUDA(launch_pdl(sizeof(XT) == 4 || re - rb <= pdl_fp64_rows(),
                            k_sor_first_colour<VT, XT>, dim3(g), dim3(256), 0,
                            s, rb, re, (const double *)c.pdiag.p, (const double *)op.rdiag,
                            scale, op.rows, b, x, op.relax, op.m1, ultra, op.relax_one));
        count_launch();
      }
      continue;
    }
    if constexpr (!kIsBf16<VT>) {
      if (op.from_zero && c.lo.n > 0) {
        // half the entries of the row
        const VT *lv;
        if constexpr (sizeof(VT) == 8) lv = c.lo.v64.p;
        else lv = c.lo.v32.p;
        LGX_CHECK(launch_rows<VT>(rb, re, c.lo, lv,
                                  SorLoOp<VT, XT>{b, x, op.relax, op.m1, ultra, op.relax_one,
                                                  c.pdiag.p, op.rdiag, op.rows},
                                  s));
        continue;
      }
    }
    // forward: exactly the rows before this colour are visited (a natural-order
    // level has its halves for sweeps from zero)
    op.visit_end = rb;
    // the last colour of a forward sweep on grid rows can also leave its
    // rows' residuals in r_last
    const bool with_res = r_last && res_from && forward && k == c.ncolours - 1 && re > rb &&
                          !kIsBf16<VT> && sizeof(XT) == 4 && grid_sweep_residual(p);
    bool done = false;
    LGX_CHECK((grid_sor_rows<VT, XT>(p, val, rb, re, b, x, relax, ultra, op.rdiag, op.relax_one,
                                     op.from_zero, op.visit_end, scale, s, &done,
                                     with_res ? r_last : nullptr)));
    if (done) {
      if (with_res) *res_from = rb;
      continue;
    }
    LGX_CHECK(launch_rows<VT>(rb, re, p, val, op, s));
  }
  return LGX_OK;
}

template <typename VT, typename XT>
lgx_status mc_residual(const lgx_colouring &c, const VT *val, const XT *b, const XT *x, XT *r,
                       cudaStream_t s) {
  return launch_rows<VT>(0, c.n, c.pcsr, val, ListResidualOp<VT, XT, false>{b, x, r, c.perm.p}, s);
}

template <typename VT, typename XT>
lgx_status mc_up_residual(const lgx_colouring &c, const VT *val, const XT *x, XT *r,
                          cudaStream_t s) {
  if (!c.natural) {
    bool done = false;
    LGX_CHECK((grid_up_residual<VT, XT>(c.pcsr, val, x, r, s, &done)));
    if (done || c.ncolours < 1) return LGX_OK;
    return launch_rows<VT>(0, c.offsets[c.ncolours - 1], c.pcsr, val,
                           LaterResidualOp<VT, XT>{x, r}, s);
  }
  const VT *v;
  if constexpr (sizeof(VT) == 8) v = c.up.v64.p;
  else v = c.up.v32.p;
  return launch_rows<VT>(0, c.n, c.up, v, ListResidualOp<VT, XT, true>{nullptr, x, r, nullptr}, s);
}

#define LGX_MC_RESIDUAL(VT, XT)                                                              \
  template lgx_status mc_residual<VT, XT>(const lgx_colouring &, const VT *, const XT *,     \
                                          const XT *, XT *, cudaStream_t);                   \
  template lgx_status mc_up_residual<VT, XT>(const lgx_colouring &, const VT *, const XT *,  \
                                             XT *, cudaStream_t);
LGX_MC_RESIDUAL(double, double)
LGX_MC_RESIDUAL(float, double)
LGX_MC_RESIDUAL(float, float)
#undef LGX_MC_RESIDUAL

template lgx_status mc_sor_sweep<double, double>(const lgx_colouring &, const double *, double,
                                                 int, int, const double *, double *,
                                                 cudaStream_t, int, const float *, double *,
                                                 int64_t *);
template lgx_status mc_sor_sweep<float, double>(const lgx_colouring &, const float *, double, int,
                                                int, const double *, double *, cudaStream_t, int,
                                                const float *, double *, int64_t *);
template lgx_status mc_sor_sweep<float, float>(const lgx_colouring &, const float *, double, int,
                                               int, const float *, float *, cudaStream_t, int,
                                               const float *, float *, int64_t *);
template lgx_status mc_sor_sweep<bf16, float>(const lgx_colouring &, const bf16 *, double, int,
                                              int, const float *, float *, cudaStream_t, int,
                                              const float *, float *, int64_t *);

lgx_status jacobi_csr(const Csr &a, double relax, const double *x_in, double *x_out,
                      const double *b, cudaStream_t s) {
  if (a.n == 0) return LGX_OK;
  if (a.storage == LGX_F64)
    return launch_rows<double>(0, a.n, a, a.v64.p,
                               JacobiOp<double>{x_in, x_out, b, relax, 1.0 - relax}, s);
  return launch_rows<float>(0, a.n, a, a.v32.p,
                            JacobiOp<float>{x_in, x_out, b, relax, 1.0 - relax}, s);
}

lgx_status jacobi_diag_zero(int64_t n, const double *d, double relax, const double *b, double *x,
                            cudaStream_t s) {
  if (n == 0) return LGX_OK;
  k_jacobi_diag_zero<<<std::min<int64_t>(grid_for(n, 256), 16384), 256, 0, s>>>(n, d, relax, b,
                                                                                 x);
  LGX_LAUNCH_CHECK();
  return LGX_OK;
}

// Public sweep on natural-order vectors: gather into the permuted order,
// sweep in place, scatter back.
lgx_status colouring_sweep_natural(lgx_colouring &c, double relax, int forward, int ultra,
                                   const double *x_in, double *x_out, const double *b,
                                   cudaStream_t s) {
  const int64_t n = c.n;
  if (!c.work_b.p) {
    LGX_CHECK(c.work_b.alloc(n));
    LGX_CHECK(c.work_x.alloc(n));
  }
  LGX_CHECK(gather<double, double>(n, c.perm.p, b, c.work_b.p, s));
  if (x_in) LGX_CHECK(gather<double, double>(n, c.perm.p, x_in, c.work_x.p, s));
  const int from_zero = x_in == nullptr;
  if (c.pcsr.storage == LGX_F64) {
    LGX_CHECK(mc_sor_sweep<double, double>(c, c.pcsr.v64.p, relax, forward, ultra, c.work_b.p,
                                           c.work_x.p, s, from_zero));
  } else {
    LGX_CHECK(mc_sor_sweep<float, double>(c, c.pcsr.v32.p, relax, forward, ultra, c.work_b.p,
                                          c.work_x.p, s, from_zero));
  }
  return scatter<double, double>(n, c.perm.p, c.work_x.p, x_out, s);
}

}  // namespace lgx

using namespace lgx;

extern "C" {

lgx_status lgx_jacobi_sweep(const lgx_matrix *a, double relax, const double *d_x_in,
                            double *d_x_out, const double *d_b, lgx_stream stream) {
  if (!a || (a->n > 0 && (!d_x_out || !d_b))) return fail(LGX_ERR_INVALID, "null argument");
  if (a->kind == LGX_MATRIX_CSR) return jacobi_csr(a->csr, relax, d_x_in, d_x_out, d_b, stream);
  if (d_x_in) return fail(LGX_ERR_UNSUPPORTED,
                          "stencil Jacobi sweeps start from zero; assemble the matrix for a "
                          "general input vector");
  const double *d = nullptr;
  LGX_CHECK(matrix_diagonal(const_cast<lgx_matrix *>(a), stream, &d));
  return jacobi_diag_zero(a->n, d, relax, d_b, d_x_out, stream);
}

lgx_status lgx_colouring_create_jp(const lgx_matrix *a, uint64_t seed, lgx_stream stream,
                                   lgx_colouring **out) {
  if (!a || !out) return fail(LGX_ERR_INVALID, "null argument");
  if (a->kind != LGX_MATRIX_CSR) return fail(LGX_ERR_UNSUPPORTED, "colouring needs a CSR matrix");
  auto *c = new lgx_colouring();
  int32_t nc = 0;
  lgx_status st = colouring_jp(a->csr, seed, stream, c->colour, nc);
  if (st == LGX_OK) st = colouring_build(a->csr, c->colour.p, nc, stream, *c);
  if (st != LGX_OK) {
    delete c;
    return st;
  }
  *out = c;
  return LGX_OK;
}

// Smallest-last greedy colouring on the host.  Ordering: vertices sit in
// buckets by their degree among the vertices not yet removed (off-diagonal
// pattern entries), each bucket a list with the most recently inserted vertex
// at its head; the initial insertion runs in index order; each step removes
// the head of the lowest non-empty bucket and moves each remaining neighbour
// (in CSR order) to the head of the bucket below.  Colouring: in the reverse
// of the removal order, each vertex takes the smallest colour none of its
// coloured neighbours has.  O(nnz); every step is fixed, so the colouring is
// deterministic.
// The pattern's adjacency as the colouring sees it: the rows themselves when
// the off-diagonal pattern is structurally symmetric, else every row's sorted
// union with the matching column of the transpose (the pattern of A + A^T),
// so that a colouring is proper for both directions of every edge.  Returns
// false when the rows are used as given.
static bool symmetrised_pattern(int64_t n, const int64_t *rowptr, const int32_t *col,
                                std::vector<int64_t> &sptr, std::vector<int32_t> &scol) {
  std::vector<int64_t> tptr((size_t)n + 1, 0);
  for (int64_t i = 0; i < n; ++i)
    for (int64_t e = rowptr[i]; e < rowptr[i + 1]; ++e)
      if (col[e] != i) ++tptr[(size_t)col[e] + 1];
  for (int64_t i = 0; i < n; ++i) tptr[(size_t)i + 1] += tptr[(size_t)i];
  std::vector<int32_t> tcol((size_t)tptr[(size_t)n]);
  std::vector<int64_t> fill(tptr.begin(), tptr.end() - 1);
  for (int64_t i = 0; i < n; ++i)
    for (int64_t e = rowptr[i]; e < rowptr[i + 1]; ++e)
      if (col[e] != i) tcol[(size_t)fill[(size_t)col[e]]++] = (int32_t)i;
  bool symmetric = true;
  std::vector<int32_t> row;
  for (int64_t i = 0; i < n && symmetric; ++i) {
    row.clear();
    for (int64_t e = rowptr[i]; e < rowptr[i + 1]; ++e)
      if (col[e] != i) row.push_back(col[e]);
    std::sort(row.begin(), row.end());
    symmetric = std::equal(row.begin(), row.end(), tcol.begin() + tptr[(size_t)i],
                           tcol.begin() + tptr[(size_t)i + 1]) &&
                (int64_t)row.size() == tptr[(size_t)i + 1] - tptr[(size_t)i];
  }
  if (symmetric) return false;
  sptr.assign((size_t)n + 1, 0);
  scol.clear();
  for (int64_t i = 0; i < n; ++i) {
    row.clear();
    for (int64_t e = rowptr[i]; e < rowptr[i + 1]; ++e)
      if (col[e] != i) row.push_back(col[e]);
    row.insert(row.end(), tcol.begin() + tptr[(size_t)i], tcol.begin() + tptr[(size_t)i + 1]);
    std::sort(row.begin(), row.end());
    row.erase(std::unique(row.begin(), row.end()), row.end());
    scol.insert(scol.end(), row.begin(), row.end());
    sptr[(size_t)i + 1] = (int64_t)scol.size();
  }
  return true;
}

}  // extern "C"

namespace lgx {
lgx_status colour_smallest_last(int64_t n, const int64_t *rowptr, const int32_t *col,
                                int32_t *colour, int32_t *ncolours, bool known_symmetric);
}  // namespace lgx

extern "C" lgx_status lgx_colour_smallest_last(int64_t n, const int64_t *rowptr,
                                               const int32_t *col, int32_t *colour,
                                               int32_t *ncolours) {
  return lgx::colour_smallest_last(n, rowptr, col, colour, ncolours, false);
}

// known_symmetric: the caller's matrix is symmetric (the AMG levels of a
// symmetric matrix), so its pattern needs no symmetrisation check
lgx_status lgx::colour_smallest_last(int64_t n, const int64_t *rowptr, const int32_t *col,
                                     int32_t *colour, int32_t *ncolours, bool known_symmetric) {
  if (n < 0 || n > INT32_MAX || (n > 0 && (!rowptr || !col || !colour)) || !ncolours)
    return fail(LGX_ERR_INVALID, "bad argument");
  *ncolours = 0;
  if (n == 0) return LGX_OK;
  if (rowptr[0] != 0) return fail(LGX_ERR_INVALID, "row offsets must start at 0");
  for (int64_t i = 0; i < n; ++i)
    if (rowptr[i + 1] < rowptr[i]) return fail(LGX_ERR_INVALID, "decreasing row offsets");
  for (int64_t e = 0; e < rowptr[n]; ++e)
    if (col[e] < 0 || col[e] >= n) return fail(LGX_ERR_INVALID, "column index out of range");
  std::vector<int64_t> sptr;
  std::vector<int32_t> scol;
  if (!known_symmetric && symmetrised_pattern(n, rowptr, col, sptr, scol)) {
    rowptr = sptr.data();
    col = scol.data();
  }
  std::vector<int64_t> deg((size_t)n), next((size_t)n, -1), prev((size_t)n, -1);
  int64_t maxdeg = 0;
  for (int64_t i = 0; i < n; ++i) {
    int64_t d = 0;
    for (int64_t e = rowptr[i]; e < rowptr[i + 1]; ++e) d += col[e] != i;
    deg[(size_t)i] = d;
    maxdeg = std::max(maxdeg, d);
  }
  std::vector<int64_t> head((size_t)maxdeg + 1, -1);
  auto unlink = [&](int64_t v) {
    const int64_t p = prev[(size_t)v], q = next[(size_t)v];
    if (p >= 0) next[(size_t)p] = q; else head[(size_t)deg[(size_t)v]] = q;
    if (q >= 0) prev[(size_t)q] = p;
  };
  auto push = [&](int64_t v) {
    const int64_t h = head[(size_t)deg[(size_t)v]];
    prev[(size_t)v] = -1;
    next[(size_t)v] = h;
    if (h >= 0) prev[(size_t)h] = v;
    head[(size_t)deg[(size_t)v]] = v;
  };
  for (int64_t i = 0; i < n; ++i) push(i);
  std::vector<uint8_t> removed((size_t)n, 0);
  std::vector<int32_t> order;
  order.reserve((size_t)n);
  int64_t low = 0;
  for (int64_t step = 0; step < n; ++step) {
    while (head[(size_t)low] < 0) ++low;
    const int64_t v = head[(size_t)low];
    unlink(v);
    removed[(size_t)v] = 1;
    order.push_back((int32_t)v);
    for (int64_t e = rowptr[v]; e < rowptr[v + 1]; ++e) {
      const int64_t u = col[e];
      if (u == v || removed[(size_t)u]) continue;
      unlink(u);
      --deg[(size_t)u];
      push(u);
    }
    if (low > 0) --low;  // a neighbour may now sit one bucket lower
  }
  std::vector<int64_t> stamp((size_t)maxdeg + 2, -1);
  for (int64_t i = 0; i < n; ++i) colour[i] = -1;
  int32_t used = 0;
  for (int64_t k = n - 1; k >= 0; --k) {
    const int64_t v = order[(size_t)k];
    for (int64_t e = rowptr[v]; e < rowptr[v + 1]; ++e) {
      const int32_t c = colour[col[e]];
      if (col[e] != v && c >= 0 && c <= maxdeg) stamp[(size_t)c] = v;
    }
    int32_t c = 0;
    while (stamp[(size_t)c] == v) ++c;
    colour[v] = c;
    used = std::max(used, c + 1);
  }
  *ncolours = used;
  return LGX_OK;
}

extern "C" {

lgx_status lgx_colouring_create(const lgx_matrix *a, const int32_t *d_colour, int32_t ncolours,
                                lgx_stream stream, lgx_colouring **out) {
  if (!a || !out || (a->n > 0 && !d_colour)) return fail(LGX_ERR_INVALID, "null argument");
  if (a->kind != LGX_MATRIX_CSR) return fail(LGX_ERR_UNSUPPORTED, "colouring needs a CSR matrix");
  auto *c = new lgx_colouring();
  lgx_status st = colouring_build(a->csr, d_colour, ncolours, stream, *c);
  if (st != LGX_OK) {
    delete c;
    return st;
  }
  *out = c;
  return LGX_OK;
}

lgx_status lgx_colouring_grid27(lgx_colouring *c, const int64_t dims[3], int with_float,
                                lgx_stream stream, int *attached) {
  if (!c || !dims) return fail(LGX_ERR_INVALID, "null argument");
  if (c->stencil_rb) {
    if (attached) *attached = 0;
    return LGX_OK;
  }
  if (with_float && c->pcsr.storage == LGX_F64) LGX_CHECK(colouring_make_f32(*c, stream));
  bool att = false;
  LGX_CHECK(grid27_attach(*c, dims, 27, stream, &att));
  if (attached) *attached = att ? 1 : 0;
  return LGX_OK;
}

}  // extern "C"

namespace lgx {
// The failure path of the kernels' bounded waits, exercised on purpose: one
// thread initialises an mbarrier that expects one arrival, issues nothing,
// and waits on it with the same bounded wait the row engine uses (about
// one second of SM clock); the wait gives up, the kernel records it in the
// device error flag and returns.  No copy is ever in flight.
__global__ void k_wait_selftest(int *err) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x != 0) return;
  mbar_init(&bar, 1);
  fence_mbar_init();
  if (!mbar_wait_bounded(&bar, 0)) atomicOr(err, 1);
}

__global__ void k_red_black_colour(int64_t n, int64_t n1, int64_t n2, int32_t *colour) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    colour[i] = (int32_t)(((i / (n1 * n2)) + ((i / n2) % n1) + (i % n2)) & 1);
}
}  // namespace lgx

extern "C" {

lgx_status lgx_wait_selftest(lgx_stream stream) {
  int *err = device_error_flag();
  if (!err) return fail(LGX_ERR_NOMEM, "device error flag not allocated");
  k_wait_selftest<<<1, 32, 0, stream>>>(err);
  LGX_LAUNCH_CHECK();
  return check_device_error(stream);
}

lgx_status lgx_colouring_create_red_black(const lgx_matrix *a, lgx_stream stream,
                                          lgx_colouring **out) {
  if (!a || !out) return fail(LGX_ERR_INVALID, "null argument");
  if (a->kind == LGX_MATRIX_CSR)
    return fail(LGX_ERR_UNSUPPORTED,
                "red-black colouring is for stencil matrices (CSR: lgx_colouring_create)");
  auto c = std::make_unique<lgx_colouring>();
  const int64_t n0 = a->st.dims[0], n1 = a->st.dims[1], n2 = a->st.dims[2];
  c->n = a->n;
  c->ncolours = 2;
  c->stencil_rb = true;
  LGX_CHECK(c->colour.alloc(a->n));
  if (a->n) {
    k_red_black_colour<<<std::min<int64_t>(grid_for(a->n, 256), 16384), 256, 0, stream>>>(
      a->n, n1, n2, c->colour.p);
    LGX_LAUNCH_CHECK();
  }
  // colour 0 holds the cells with even p0 + p1 + p2
  int64_t even = 0;
  for (int64_t p0 = 0; p0 < n0; ++p0)
    for (int64_t p1 = 0; p1 < n1; ++p1) even += (n2 + 1 - ((p0 + p1) & 1)) / 2;
  c->offsets = {0, even, a->n};
  LGX_CUDA(cudaStreamSynchronize(stream));
  *out = c.release();
  return LGX_OK;
}

lgx_status lgx_colouring_destroy(lgx_colouring *c) {
  delete c;
  return LGX_OK;
}

lgx_status lgx_colouring_export(const lgx_colouring *c, int32_t *d_colour, int32_t *ncolours,
                                lgx_stream stream) {
  if (!c) return fail(LGX_ERR_INVALID, "null colouring");
  if (d_colour && c->n)
    LGX_CUDA(cudaMemcpyAsync(d_colour, c->colour.p, sizeof(int32_t) * c->n,
                             cudaMemcpyDeviceToDevice, stream));
  if (ncolours) *ncolours = c->ncolours;
  LGX_CUDA(cudaStreamSynchronize(stream));
  return LGX_OK;
}

lgx_status lgx_sor_sweep(const lgx_matrix *a, const lgx_colouring *c, double relax, int forward,
                         int ultra, const double *d_x_in, double *d_x_out, const double *d_b,
                         lgx_stream stream) {
  if (!a || !c || (a->n > 0 && (!d_x_out || !d_b))) return fail(LGX_ERR_INVALID, "null argument");
  if (c->n != a->n) return fail(LGX_ERR_INVALID, "colouring does not match the matrix");
  if (c->stencil_rb != (a->kind != LGX_MATRIX_CSR))
    return fail(LGX_ERR_UNSUPPORTED, a->kind == LGX_MATRIX_CSR
                                       ? "a stencil's red-black colouring on a CSR matrix"
                                       : "a stencil matrix sweeps with its red-black colouring");
  if (c->stencil_rb)
    return stencil_sor_sweep(a, relax, forward, ultra, d_x_in, d_x_out, d_b, stream);
  return colouring_sweep_natural(*const_cast<lgx_colouring *>(c), relax, forward, ultra, d_x_in,
                                 d_x_out, d_b, stream);
}

lgx_status lgx_colouring_permute(const lgx_colouring *c, const double *d_src, double *d_dst,
                                 lgx_stream stream) {
  if (!c || (c->n > 0 && (!d_src || !d_dst))) return fail(LGX_ERR_INVALID, "null argument");
  if (c->stencil_rb)
    return fail(LGX_ERR_UNSUPPORTED, "a stencil colouring sweeps in natural order (lgx_sor_sweep)");
  return gather<double, double>(c->n, c->perm.p, d_src, d_dst, stream);
}

lgx_status lgx_colouring_unpermute(const lgx_colouring *c, const double *d_src, double *d_dst,
                                   lgx_stream stream) {
  if (!c || (c->n > 0 && (!d_src || !d_dst))) return fail(LGX_ERR_INVALID, "null argument");
  if (c->stencil_rb)
    return fail(LGX_ERR_UNSUPPORTED, "a stencil colouring sweeps in natural order (lgx_sor_sweep)");
  return scatter<double, double>(c->n, c->perm.p, d_src, d_dst, stream);
}

lgx_status lgx_sor_sweep_permuted(const lgx_colouring *c, double relax, int forward, int ultra,
                                  double *d_x, const double *d_b, lgx_stream stream) {
  if (!c || (c->n > 0 && (!d_x || !d_b))) return fail(LGX_ERR_INVALID, "null argument");
  if (c->stencil_rb)
    return fail(LGX_ERR_UNSUPPORTED, "a stencil colouring sweeps in natural order (lgx_sor_sweep)");
  if (c->pcsr.storage == LGX_F64)
    return mc_sor_sweep<double, double>(*c, c->pcsr.v64.p, relax, forward, ultra, d_b, d_x,
                                        stream);
  return mc_sor_sweep<float, double>(*c, c->pcsr.v32.p, relax, forward, ultra, d_b, d_x, stream);
}

lgx_status lgx_sor_sweep_permuted_f32(lgx_colouring *c, float relax, int forward, int ultra,
                                      float *d_x, const float *d_b, lgx_stream stream) {
  if (!c || (c->n > 0 && (!d_x || !d_b))) return fail(LGX_ERR_INVALID, "null argument");
  if (c->stencil_rb)
    return fail(LGX_ERR_UNSUPPORTED, "a stencil colouring sweeps in natural order (lgx_sor_sweep)");
  const float *v = c->pcsr.v32.p;
  if (c->pcsr.storage == LGX_F64) {
    LGX_CHECK(colouring_make_f32(*c, stream));
    v = c->pv32.p;
  }
  return mc_sor_sweep<float, float>(*c, v, relax, forward, ultra, d_b, d_x, stream);
}

}  // extern "C"
