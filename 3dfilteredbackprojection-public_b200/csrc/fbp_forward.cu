// Ray-driven forward projection of the volume:
// FBP3D::project_forward_cone_to_projections / _to_sinogram and
// project_forward_parallel_to_projections / _to_sinogram
// (Source/FilteredBackProjection/FBP3D.cpp:212-330), FBP2D::project_forward
// (FBP2D.cpp:54-94). The reference's radon shaders are absent; the transform
// is defined in the backprojector's conventions (same angles, source, detector
// axes and pixel centres): the ray of detector pixel (iu, iv) at view k is
// clipped to the volume box, its length L cut into n = ceil(L / (vox / 2))
// equal steps, and the trilinearly interpolated volume (zero outside) summed
// at the step midpoints times the step.
//
// One thread per ray. The per-ray setup (ray-box clipping, n) is FP64, so the
// sample count matches the FP64 restatement; the march is FP32 (position by
// FMA from the step index, eight trilinear taps).
//
// What bounds the march is the eight gathers of a sample: a warp instruction
// costs L1 one pass per 128-byte line its lanes touch. Rays of one detector
// column (same u, neighbouring v) share their path in the x-z plane and differ
// in y alone, so forward_columns_kernel gives a warp 32 detector rows of one
// column and reads a copy of the volume whose fastest axis is y: the lanes of
// a gather fall on one or two lines at every view angle. In the volume's own
// layout (x fastest) a warp's rays touch up to 32 lines when they run along x.
// 256^3, 360 views of 256 x 256: 140.6 ms with 8 x 4 rays a warp in the
// volume's layout, 19.8 ms here, the copy included (1.1e10 samples x 32 bytes
// = 18 TB/s through L1, half its rate: two lines for 32 unaligned lanes).
// The copy has a border of one zero voxel on every side, so samples near the
// faces need neither clamps nor masked weights.

#include "fbp_internal.h"

#include <algorithm>

namespace fbp {
namespace {

struct FPArgs {
  const float* vol;
  int nx, ny, nz;
  double vox;
  int cone;
  double sod, sdd, du, dv, span, offset;
  int nu, nv, nviews;
  float* out;
  long long pitch;  // floats per detector row
  bool sinogram;    // rows ordered [v][view]
};

// Ray of detector pixel (iu, iv) at the view (c, s), clipped to the volume box:
// n samples of length step, the first at voxel-index position f0 (voxel centres
// at integers), each next one by d (FP32). n = 0: the ray misses
// the box.
struct RayMarch {
  long long n;
  float step, fx0, fy0, fz0, dx, dy, dz;
};

__device__ __forceinline__ RayMarch ray_march(const FPArgs& a, double c, double s, int iu, int iv) {
  const double u = (iu + 0.5 - 0.5 * a.nu) * a.du, v = (iv + 0.5 - 0.5 * a.nv) * a.dv;
  const double hx = 0.5 * a.nx * a.vox, hy = 0.5 * a.ny * a.vox, hz = 0.5 * a.nz * a.vox;
  double S[3], D[3];
  if (a.cone) {
    S[0] = -a.sod * c;
    S[1] = 0.0;
    S[2] = -a.sod * s;
    D[0] = (a.sdd - a.sod) * c - u * s - S[0];
    D[1] = v;
    D[2] = (a.sdd - a.sod) * s + u * c - S[2];
  } else {
    const double R = 2.0 * (hx + hy + hz);
    S[0] = -R * c - u * s;
    S[1] = v;
    S[2] = -R * s + u * c;
    D[0] = c;
    D[1] = 0.0;
    D[2] = s;
  }
  const double len = sqrt(D[0] * D[0] + D[1] * D[1] + D[2] * D[2]);
  const double h[3] = {hx, hy, hz};
  double t0 = -1e300, t1 = 1e300;
  bool miss = false;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    D[q] /= len;
    if (fabs(D[q]) < 1e-300) {
      if (S[q] <= -h[q] || S[q] >= h[q]) miss = true;
      continue;
    }
    double ta = (-h[q] - S[q]) / D[q], tb = (h[q] - S[q]) / D[q];
    if (ta > tb) {
      const double tt = ta;
      ta = tb;
      tb = tt;
    }
    t0 = fmax(t0, ta);
    t1 = fmin(t1, tb);
  }
  RayMarch r{};
  if (!miss && t1 > t0) {
    r.n = (long long)ceil((t1 - t0) / (0.5 * a.vox));
    const double step = (t1 - t0) / r.n;
    const double tm = t0 + 0.5 * step;
    r.step = (float)step;
    r.fx0 = (float)((S[0] + tm * D[0]) / a.vox + 0.5 * a.nx - 0.5);
    r.fy0 = (float)((S[1] + tm * D[1]) / a.vox + 0.5 * a.ny - 0.5);
    r.fz0 = (float)((S[2] + tm * D[2]) / a.vox + 0.5 * a.nz - 0.5);
    r.dx = (float)(step * D[0] / a.vox);
    r.dy = (float)(step * D[1] / a.vox);
    r.dz = (float)(step * D[2] / a.vox);
  }
  return r;
}

// Detectors of a few rows (a 2D image has one): the volume in its own layout,
// lanes along the detector row.
__global__ void __launch_bounds__(128) forward_rows_kernel(const FPArgs a) {
  const int iu = blockIdx.x * 128 + threadIdx.x, k = blockIdx.z;
  if (iu >= a.nu) return;
  double s, c;
  sincos(a.offset + a.span * k / a.nviews, &s, &c);
  const long long sx = 1, sy = a.nx, sz = (long long)a.nx * a.ny;
  for (int iv = blockIdx.y; iv < a.nv; iv += gridDim.y) {
    const RayMarch r = ray_march(a, c, s, iu, iv);
    float acc = 0.f;
    for (long long q = 0; q < r.n; ++q) {
      const float fq = (float)q;
      const float fx = fmaf(fq, r.dx, r.fx0), fy = fmaf(fq, r.dy, r.fy0), fz = fmaf(fq, r.dz, r.fz0);
      const float flx = floorf(fx), fly = floorf(fy), flz = floorf(fz);
      const int i0 = (int)flx, j0 = (int)fly, l0 = (int)flz;
      const float wx = fx - flx, wy = fy - fly, wz = fz - flz;
      // corners clamped into the volume, with zero weight where they fall outside
      const float ax0 = (unsigned)i0 < (unsigned)a.nx ? 1.f - wx : 0.f;
      const float ax1 = (unsigned)(i0 + 1) < (unsigned)a.nx ? wx : 0.f;
      const float ay0 = (unsigned)j0 < (unsigned)a.ny ? 1.f - wy : 0.f;
      const float ay1 = (unsigned)(j0 + 1) < (unsigned)a.ny ? wy : 0.f;
      const float az0 = (unsigned)l0 < (unsigned)a.nz ? 1.f - wz : 0.f;
      const float az1 = (unsigned)(l0 + 1) < (unsigned)a.nz ? wz : 0.f;
      const long long x0 = min(max(i0, 0), a.nx - 1) * sx, x1 = min(max(i0 + 1, 0), a.nx - 1) * sx;
      const long long y0 = min(max(j0, 0), a.ny - 1) * sy, y1 = min(max(j0 + 1, 0), a.ny - 1) * sy;
      const long long z0 = min(max(l0, 0), a.nz - 1) * sz, z1 = min(max(l0 + 1, 0), a.nz - 1) * sz;
      const float* p = a.vol;
      const float c00 = fmaf(ax1, __ldg(p + z0 + y0 + x1), ax0 * __ldg(p + z0 + y0 + x0));
      const float c01 = fmaf(ax1, __ldg(p + z0 + y1 + x1), ax0 * __ldg(p + z0 + y1 + x0));
      const float c10 = fmaf(ax1, __ldg(p + z1 + y0 + x1), ax0 * __ldg(p + z1 + y0 + x0));
      const float c11 = fmaf(ax1, __ldg(p + z1 + y1 + x1), ax0 * __ldg(p + z1 + y1 + x0));
      acc += fmaf(az1, fmaf(ay1, c11, ay0 * c10), az0 * fmaf(ay1, c01, ay0 * c00));
    }
    acc *= r.step;
    const long long row = a.sinogram ? (long long)iv * a.nviews + k : (long long)k * a.nv + iv;
    a.out[row * a.pitch + iu] = acc;
  }
}

// vol [z][y][x] -> out [z + 1][x + 1][y + 1] of (nz + 2) x (nx + 2) x py, zero
// border (and zero padding of y up to py). One 32 x 32 (x, y) tile a block.
__global__ void __launch_bounds__(256) volume_columns_kernel(const float* __restrict__ vol, int nx, int ny, int nz,
                                                             int py, float* __restrict__ out) {
  __shared__ float tile[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int x0 = blockIdx.x * 32 - 1, y0 = blockIdx.y * 32 - 1, z = (int)blockIdx.z - 1;
#pragma unroll
  for (int j = ty; j < 32; j += 8) {
    const int x = x0 + tx, y = y0 + j;
    const bool in = (unsigned)x < (unsigned)nx && (unsigned)y < (unsigned)ny && (unsigned)z < (unsigned)nz;
    tile[j][tx] = in ? __ldg(vol + ((size_t)z * ny + y) * nx + x) : 0.f;
  }
  __syncthreads();
#pragma unroll
  for (int j = ty; j < 32; j += 8) {
    const int x = x0 + 1 + j, y = y0 + 1 + tx;  // indices in the bordered copy
    if (x < nx + 2 && y < py) out[((size_t)blockIdx.z * (nx + 2) + x) * py + y] = tile[tx][j];
  }
}

__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long r) {
  float2 d;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(r));
  return d;
}
// packed FP32 pairs (sm_100): a b + c, a b, a + b toward zero, a - b
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long add2_rz(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("add.rz.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23: x + kMagic toward zero is kMagic + floor(x) for |x| < 2^22
constexpr uint32_t kMagicBits = 0x4B400000u;
// Detector rows from which the column march is the faster one although it
// leaves lanes idle below 32 (256 x ny x 256, 180 views, ms: rows 1.21, 1.91,
// 3.65 and columns 1.25, 1.25, 1.25 at ny = 4, 8, 16).
constexpr int kMinColumnRows = 6;
constexpr int kColWarps = 4;  // neighbouring detector columns per block (their rays share lines in L1)

__global__ void __launch_bounds__(32 * kColWarps) forward_columns_kernel(const FPArgs a, const float* __restrict__ cols,
                                                                         int py, uint32_t last) {
  const int iu = blockIdx.x * kColWarps + (threadIdx.x >> 5), iv = blockIdx.y * 32 + (threadIdx.x & 31);
  const int k = blockIdx.z;
  if (iu >= a.nu || iv >= a.nv) return;
  double s, c;
  sincos(a.offset + a.span * k / a.nviews, &s, &c);
  const RayMarch r = ray_march(a, c, s, iu, iv);
  const uint32_t px = (uint32_t)py, pz = (uint32_t)py * (uint32_t)(a.nx + 2);
  // element of the cell (i, j, l), which the bordered copy has at i + 1, j + 1,
  // l + 1; the position's bit patterns minus kMagicBits are i, j, l
  const uint32_t base = (1u - kMagicBits) * (px + pz + 1u);
  const unsigned long long dxz = pack2(r.dx, r.dz), fxz0 = pack2(r.fx0, r.fz0);
  const unsigned long long magic2 = pack2(kMagic, kMagic);
  float acc = 0.f, fq = 0.f;
  const int n = (int)r.n;
#pragma unroll 2
  for (int q = 0; q < n; ++q) {
    const unsigned long long xz = fma2(pack2(fq, fq), dxz, fxz0);
    const float y = fmaf(fq, r.dy, r.fy0);
    fq += 1.f;
    const unsigned long long txz = add2_rz(xz, magic2);
    const float ty = __fadd_rz(y, kMagic);
    const float2 w = unpack2(sub2(xz, sub2(txz, magic2)));
    const float wy = y - (ty - kMagic);
    const float2 t = unpack2(txz);
    uint32_t e = __float_as_uint(t.x) * px + __float_as_uint(t.y) * pz + (__float_as_uint(ty) + base);
    e = min(e, last);  // samples lie inside the box, so this never moves one: it bounds the reads
    const float* p00 = cols + e;
    const float* p10 = p00 + px;
    const float* p01 = p00 + pz;
    const float* p11 = p01 + px;
    // pairs over z; weighted sums along y, x, z (a + w (b - a) would turn an
    // infinite voxel into NaN, and rounds the difference as well)
    const unsigned long long a0 = pack2(__ldg(p00), __ldg(p01)), a1 = pack2(__ldg(p00 + 1), __ldg(p01 + 1));
    const unsigned long long b0 = pack2(__ldg(p10), __ldg(p11)), b1 = pack2(__ldg(p10 + 1), __ldg(p11 + 1));
    const float vx = 1.f - w.x, vy = 1.f - wy;
    const unsigned long long wy2 = pack2(wy, wy), vy2 = pack2(vy, vy);
    const unsigned long long ax = fma2(wy2, a1, mul2(vy2, a0)), bx = fma2(wy2, b1, mul2(vy2, b0));
    const float2 z = unpack2(fma2(pack2(w.x, w.x), bx, mul2(pack2(vx, vx), ax)));
    acc += fmaf(w.y, z.y, (1.f - w.y) * z.x);
  }
  const long long row = a.sinogram ? (long long)iv * a.nviews + k : (long long)k * a.nv + iv;
  a.out[row * a.pitch + iu] = acc * r.step;
}

}  // namespace

int launch_forward(fbp_context* ctx, const float* vol, int nx, int ny, int nz, double vox, bool cone, double sod,
                   double sdd, double du, double dv, double span, double offset, int nu, int nv, int nviews,
                   float* out, long long pitch, bool sinogram) {
  if (nu <= 0 || nv <= 0 || nviews <= 0 || nviews > 65535)
    return set_error(ctx, FBP_ERR_INVALID_ARGUMENT, "forward projection: bad detector size or view count");
  FPArgs a;
  a.vol = vol;
  a.nx = nx;
  a.ny = ny;
  a.nz = nz;
  a.vox = vox;
  a.cone = cone ? 1 : 0;
  a.sod = sod;
  a.sdd = sdd;
  a.du = du;
  a.dv = dv;
  a.span = span;
  a.offset = offset;
  a.nu = nu;
  a.nv = nv;
  a.nviews = nviews;
  a.out = out;
  a.pitch = pitch;
  a.sinogram = sinogram;
  // The column march needs detector rows to fill its warps, a bordered copy
  // that 32-bit element indices reach, and room for it. A copy of up to
  // kKeptCopy stays with the context (its scratch); a larger one, up to 16 GB,
  // belongs to the call: allocated and freed in stream order, it is the
  // device's again at the next wait.
  constexpr size_t kKeptCopy = 256u << 20;
  const int py = (ny + 2 + 3) / 4 * 4;
  const size_t elems = (size_t)(nz + 2) * (nx + 2) * py, bytes = elems * sizeof(float);
  if (nv >= kMinColumnRows && ny > 1 && elems < (1ull << 32) - 1 && nz + 2 <= 65535 && (ny + 33) / 32 <= 65535) {
    const bool keep = bytes <= kKeptCopy;
    void* cols = nullptr;
    if (keep) {
      cols = scratch(ctx, bytes);
    } else if (cudaMallocAsync(&cols, bytes, ctx->stream) != cudaSuccess) {
      cudaGetLastError();
      cols = nullptr;
    }
    if (cols) {
      float* const copy = static_cast<float*>(cols);
      volume_columns_kernel<<<dim3((nx + 2 + 31) / 32, (py + 31) / 32, nz + 2), 256, 0, ctx->stream>>>(vol, nx, ny, nz,
                                                                                                      py, copy);
      int rc = launched(ctx, "volume_columns_kernel");
      if (!rc) {
        // the last element that a cell may start at (its far corner is the copy's last element)
        const uint32_t last = (uint32_t)(elems - 2 - (size_t)py * (nx + 2) - py);
        const dim3 grid((nu + kColWarps - 1) / kColWarps, (nv + 31) / 32, nviews);
        forward_columns_kernel<<<grid, 32 * kColWarps, 0, ctx->stream>>>(a, copy, py, last);
        rc = launched(ctx, "forward_columns_kernel");
      }
      if (!keep) {
        const cudaError_t e = cudaFreeAsync(cols, ctx->stream);
        if (!rc) rc = cuda_check(ctx, e, "cudaFreeAsync(volume copy)");
      }
      return rc;
    }
    ctx->last_error.clear();  // no room for the copy: march through the volume itself
  }
  const dim3 grid((nu + 127) / 128, std::min(nv, 65535), nviews);
  forward_rows_kernel<<<grid, 128, 0, ctx->stream>>>(a);
  return launched(ctx, "forward_rows_kernel");
}

}  // namespace fbp
