// Kernel view of a matrix-free 7-point diffusion stencil and its row (see
// lgx_spmv.cu for the row's semantics).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "lgx_internal.cuh"

namespace lgx {

struct StencilDev {
  int n0, n1, n2;
  int lookup;
  double conn[48];  // lookup tables, staged into shared memory by each block
  const uint8_t *mat;
  const double *face0, *face1, *face2;  // value valuator: face d of cell i joins i and i+stride_d
  const double *diag;
};

// Copies the lookup tables of S into shared memory (all threads of the block
// must call it).
__device__ __forceinline__ const double *stage_conn(const StencilDev &S, double *sh) {
  const unsigned t = threadIdx.x + blockDim.x * threadIdx.y;
  if (S.lookup && t < 48) sh[t] = S.conn[t];
  __syncthreads();
  return sh;
}

__device__ __forceinline__ double st_conn_lookup(const double *conn, const uint8_t *mat, int d,
                                                 int64_t i, int64_t j) {
  return conn[d * 16 + mat[i] * 4 + mat[j]];
}

// off-diagonal connection values of cell (p0,p1,p2) = i, in visiting order
template <bool LOOKUP>
__device__ __forceinline__ void st_row(const StencilDev &S, const double *conn, int p0, int p1,
                                       int p2, int64_t i, double cv[6], int64_t cj[6],
                                       bool has[6]) {
  const int64_t s0 = (int64_t)S.n1 * S.n2, s1 = S.n2;
  // before: d = 0, 1, 2 ; after: d = 2, 1, 0
  has[0] = p0 > 0;
  has[1] = p1 > 0;
  has[2] = p2 > 0;
  has[3] = p2 + 1 < S.n2;
  has[4] = p1 + 1 < S.n1;
  has[5] = p0 + 1 < S.n0;
  cj[0] = i - s0;
  cj[1] = i - s1;
  cj[2] = i - 1;
  cj[3] = i + 1;
  cj[4] = i + s1;
  cj[5] = i + s0;
  if constexpr (LOOKUP) {
    cv[0] = has[0] ? st_conn_lookup(conn, S.mat, 0, i, cj[0]) : 0.0;
    cv[1] = has[1] ? st_conn_lookup(conn, S.mat, 1, i, cj[1]) : 0.0;
    cv[2] = has[2] ? st_conn_lookup(conn, S.mat, 2, i, cj[2]) : 0.0;
    cv[3] = has[3] ? st_conn_lookup(conn, S.mat, 2, i, cj[3]) : 0.0;
    cv[4] = has[4] ? st_conn_lookup(conn, S.mat, 1, i, cj[4]) : 0.0;
    cv[5] = has[5] ? st_conn_lookup(conn, S.mat, 0, i, cj[5]) : 0.0;
  } else {
    cv[0] = has[0] ? S.face0[cj[0]] : 0.0;
    cv[1] = has[1] ? S.face1[cj[1]] : 0.0;
    cv[2] = has[2] ? S.face2[cj[2]] : 0.0;
    cv[3] = has[3] ? S.face2[i] : 0.0;
    cv[4] = has[4] ? S.face1[i] : 0.0;
    cv[5] = has[5] ? S.face0[i] : 0.0;
  }
}

// the view of a stencil matrix whose diagonal and faces exist (stencil_ensure)
StencilDev dev_of(const lgx_matrix *a);

}  // namespace lgx
