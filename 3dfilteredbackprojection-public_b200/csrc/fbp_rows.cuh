// Device helpers shared by the row-filter kernels: fused pre-operations on
// load.
#pragma once

#include "fbp_internal.h"

namespace fbp {

// The pending pre-operations (log normalisation, then FDK weight) on the raw
// sample x of column i. dist2: squared distance from the source to the row's
// centre (pre_row).
__device__ __forceinline__ float pre_row(const RowSet& rs, long long r) {
  int iv;
  if (r >> 32) {
    iv = (int)(rs.sinogram ? r / rs.n_views : r % rs.n_v);
  } else {  // a 32-bit division is a fifth of a 64-bit one
    const unsigned row = (unsigned)r;
    iv = (int)(rs.sinogram ? row / (unsigned)rs.n_views : row % (unsigned)rs.n_v);
  }
  const float v = (iv + 0.5f - 0.5f * rs.n_v + rs.w_voff) * rs.w_dv;
  return fmaf(v, v, rs.w_sdd * rs.w_sdd);
}

__device__ __forceinline__ float pre_log(const RowSet& rs, float x) {
  float y = fmaxf(x, 1e-30f * rs.log_base);
  return -logf(y / rs.log_base);
}

// sdd / distance for a detector column u off the centre
__device__ __forceinline__ float pre_weight(const RowSet& rs, float dist2, float u) {
  return rs.w_sdd * rsqrtf(fmaf(u, u, dist2));
}

__device__ __forceinline__ float pre_op(const RowSet& rs, long long r, int i, float x) {
  if (rs.log_norm) x = pre_log(rs, x);
  if (rs.weight) x *= pre_weight(rs, pre_row(rs, r), (i + 0.5f - 0.5f * rs.m) * rs.w_du);
  return x;
}

__device__ __forceinline__ float load_pre(const RowSet& rs, long long r, int i) {
  return pre_op(rs, r, i, rs.data[r * rs.pitch + i]);
}

__device__ __forceinline__ int row_view(const RowSet& rs, long long r) {
  if (r >> 32) return rs.sinogram ? (int)(r % rs.n_views) : (int)(r / rs.n_v);
  const unsigned row = (unsigned)r;
  return (int)(rs.sinogram ? row % (unsigned)rs.n_views : row / (unsigned)rs.n_v);
}

}  // namespace fbp
