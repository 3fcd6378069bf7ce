// Device helpers shared by the row-filter kernels: fused pre-operations on
// load.
#pragma once

#include "fbp_internal.h"

namespace fbp {

// The pending pre-operations (log normalisation, then FDK weight) on the raw
// sample x of row r, column i.
__device__ __forceinline__ float pre_op(const RowSet& rs, long long r, int i, float x) {
  if (rs.log_norm) {
    float y = fmaxf(x, 1e-30f * rs.log_base);
    x = -logf(y / rs.log_base);
  }
  if (rs.weight) {
    int iv = rs.sinogram ? (int)(r / rs.n_views) : (int)(r % rs.n_v);
    float u = (i + 0.5f - 0.5f * rs.m) * rs.w_du;
    float v = (iv + 0.5f - 0.5f * rs.n_v + rs.w_voff) * rs.w_dv;
    x *= rs.w_sdd * rsqrtf(rs.w_sdd * rs.w_sdd + u * u + v * v);
  }
  return x;
}

__device__ __forceinline__ float load_pre(const RowSet& rs, long long r, int i) {
  return pre_op(rs, r, i, rs.data[r * rs.pitch + i]);
}

__device__ __forceinline__ int row_view(const RowSet& rs, long long r) {
  return rs.sinogram ? (int)(r % rs.n_views) : (int)(r / rs.n_v);
}

}  // namespace fbp
