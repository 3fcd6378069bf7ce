// Voxel-driven, distance-weighted backprojection with bilinear detector
// interpolation, for flat-panel cone beam (FDK) and parallel beam, in 3D and
// 2D (a 2D image is a volume with one y-slice and a one-row detector).
//
// Replaces the reference's per-view dispatch loop
// FBP3D::project_backward_cone_fdk_from_projections (Source/FilteredBackProjection/
// FBP3D.cpp:524-559, one full read-modify-write of the volume per view) and the
// 3D / 2D parallel variants (FBP3D.cpp:460-522, FBP2D.cpp:96-122). The GLSL
// bodies are not in the reference; the arithmetic is the textbook FDK one.
//
// Design (one launch for all views):
//   * A CTA owns a TX x TZ tile of voxel columns and NY voxels along the
//     rotation axis (y); each consumer thread owns one column segment of NY
//     voxels and keeps its NY sums in registers across every view, so the
//     volume is written exactly once (clip epilogue fused into the store).
//   * Warp specialisation (generic kernel): one producer warp computes, in FP64, the tile's
//     detector footprint and tile-local projective coefficients for 32 views
//     at a time (one view per lane), re-based on the tile corner and on the
//     staged window so that the FP32 coordinates the consumers form stay small
//     and accurate, and copies each view's footprint window (box_u x box_v
//     elements) into a ring of shared-memory stages with TMA
//     (cp.async.bulk.tensor, no multicast). Samples outside the detector
//     arrive as zeros from the TMA out-of-bounds fill. Full / empty mbarriers
//     per stage replace block barriers; consumer warps never wait for one
//     another.
//   * Per view a consumer thread forms 1/D, its detector column u (constant
//     along the column), the distance weight and the v step once; per voxel it
//     forms v and takes floor / fraction with the 1.5 * 2^23 rounding constant
//     (no conversion instructions). FP16 views are staged as row pairs
//     (element (v, u) holds rows v and v + 1), FP32 views as plain rows along
//     which the taps march.
//   * Every mbarrier wait is bounded; on expiry the CTA records an error and
//     leaves, and every CTA checks the error word before starting.

#include "fbp_internal.h"

#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstdio>
#include <type_traits>
#include <vector>

namespace fbp {
namespace {

constexpr int kMaxStages = 8;                // shared-memory ring stages (one view each)
constexpr uint32_t kWaitLimit = 1u << 22;  // mbarrier polls before giving up

struct ViewCoef {
  float Dx, Dz, D0;  // D = L / SOD (cone) or 1 (parallel), affine in (x', z')
  float Nx, Nz, N0;  // u_local * D
  float Vx, Vz, V0;  // v_local * D at the tile's first y
  float wscale;      // extra per-view weight (FP16 views: 1 / scale)
  int skip;          // bit 0: tile footprint misses the detector; bit 1: rows advance by less than one per voxel
  int box;           // staged window: width (elements) | rows << 16
};

// Per-view window boxes: a grid of tensor maps over the same filtered stack,
// 8 widths x 8 heights chosen per geometry from the histogram of window sizes
// that the footprint pass collects (the largest of each = the largest
// window); the producer stages each (tile, view) window with the smallest box
// that holds it, so a copy moves little more than what the view needs.
constexpr int kNW = kBoxGrid, kNH = kBoxGrid;
struct BoxMaps {
  CUtensorMap map[kNW * kNH];  // [width index][height index]
  int w[kNW];                  // box widths in elements of the layout
  int h[kNH];                  // box heights in element rows
};

struct BPArgs {
  float* vol;
  int nx, ny, nz;
  int nu, nv, nviews;
  int kind;
  double sod, sdd, du, dv, vox;
  double cu, cv;          // (nu - 1) / 2, (nv - 1) / 2
  float dvn;              // v step per voxel times D
  float scale;            // pi / K * filter spacing factor
  const double2* trig;    // (cos, sin) per view
  const float* inv_scale; // FP16 per-view 1/scale or nullptr
  int box_u, box_v, align;  // largest window (elements, element rows)
  int box_bytes;            // smem bytes reserved per staged window (multiple of 128)
  int chunk;              // ring stages
  int ntx, ntz;           // tiles along x and z
  int sino_layout;        // tensor coordinates (u, view, v) instead of (u, v, view)
  int pair_rows;          // 1: an element carries rows v and v + 1 (pair layouts)
  int clip_ylimit;        // clip negatives where iy < clip_ylimit
  int* err;
  // interleaved layout in global memory, for windows too large to stage:
  // 16-byte entries, [group][element row][plane][element column]
  const uint4* qg;
  int qg_pitch, qg_rows;  // element columns per plane row, element rows per group
  // orbits of the interleaved layouts (struct Orbits) and their representative
  // tiles; wrap: slots past one that the sums move by from the last phase to the first
  int groups, mirror, wrap;
  int nbx, nbz;
  int resident;           // CTAs resident on the GPU at once (view-group skew of the interleaved walk)
  int band;               // tile orbits along z in one band of the symmetric kernel's tile order
  int* minmax;            // fold the stored values' min / max into this pair (or nullptr)
  int y_off, ny_total;    // the volume is y-slices [y_off, y_off + ny) of ny_total
  int vol_ystride;        // y-slices between z planes of the output buffer
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait: returns false (and records kDevTimeout) after kWaitLimit polls.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* err) {
  for (uint32_t i = 0; i < kWaitLimit; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  atomicCAS(err, 0, kDevTimeout);
  return false;
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
      "[%5];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
      "[%6];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ int floor_div(int a, int b) {  // b > 0
  int q = a / b;
  return (a % b != 0 && a < 0) ? q - 1 : q;
}

// Tile geometry for view k in FP64: the affine coefficients of D (= L/SOD
// for cone beam, 1 for parallel beam), of u*D and of v*D in tile-local voxel
// offsets (x', z', y'), and the detector extremes over the tile's corner
// voxels. A projective map attains its extremes over a box at the corners.
struct TileGeo {
  double Dx, Dz, D0, Ux, Uz, U0, G, Yc;
  double umin, umax, vmin, vmax, dmin;
};

__device__ void tile_geo(const BPArgs& a, int k, int ix0, int iy0, int iz0, int ex, int ey, int ez, TileGeo& t) {
  const double c = a.trig[k].x, s = a.trig[k].y;
  const double Xc = (ix0 + 0.5 - 0.5 * a.nx) * a.vox;
  const double Zc = (iz0 + 0.5 - 0.5 * a.nz) * a.vox;
  t.Yc = (a.y_off + iy0 + 0.5 - 0.5 * a.ny_total) * a.vox;
  if (a.kind == FBP_GEOMETRY_CONE) {
    const double K = a.sdd / (a.sod * a.du);
    t.Dx = a.vox * c / a.sod;
    t.Dz = a.vox * s / a.sod;
    t.D0 = (a.sod + Xc * c + Zc * s) / a.sod;
    t.Ux = -a.vox * s * K;
    t.Uz = a.vox * c * K;
    t.U0 = (-Xc * s + Zc * c) * K;
    t.G = a.sdd / (a.sod * a.dv);
  } else {
    t.Dx = 0.0;
    t.Dz = 0.0;
    t.D0 = 1.0;
    t.Ux = -a.vox * s / a.du;
    t.Uz = a.vox * c / a.du;
    t.U0 = (-Xc * s + Zc * c) / a.du;
    t.G = 1.0 / a.dv;
  }
  t.umin = 1e300;
  t.umax = -1e300;
  t.vmin = 1e300;
  t.vmax = -1e300;
  t.dmin = 1e300;
#pragma unroll
  for (int cx = 0; cx < 2; ++cx)
#pragma unroll
    for (int cz = 0; cz < 2; ++cz) {
      const double x = cx ? ex : 0, z = cz ? ez : 0;
      const double D = t.Dx * x + t.Dz * z + t.D0;
      t.dmin = fmin(t.dmin, D);
      // one FP64 reciprocal per corner column instead of three divisions (the
      // producer computes this for every quad, skipped ones included)
      const double rD = 1.0 / D;
      const double u = (t.Ux * x + t.Uz * z + t.U0) * rD + a.cu;
      t.umin = fmin(t.umin, u);
      t.umax = fmax(t.umax, u);
#pragma unroll
      for (int cy = 0; cy < 2; ++cy) {
        const double y = cy ? ey : 0;
        const double v = t.G * (t.Yc + a.vox * y) * rD + a.cv;
        t.vmin = fmin(t.vmin, v);
        t.vmax = fmax(t.vmax, v);
      }
    }
}

constexpr double kSlack = 1.0 / 64;  // detector samples of margin around the footprint

__device__ __forceinline__ bool tile_skip(const BPArgs& a, const TileGeo& t) {
  return t.dmin <= 1e-6 || t.umax <= -1.0 || t.umin >= (double)a.nu || t.vmax <= -1.0 || t.vmin >= (double)a.nv;
}

// Window origin (u0 aligned down for TMA) and the samples the tile needs.
__device__ __forceinline__ void tile_window(const BPArgs& a, const TileGeo& t, int& u0, int& v0, int& need_u,
                                            int& need_v) {
  u0 = floor_div((int)floor(t.umin - kSlack), a.align) * a.align;
  v0 = (int)floor(t.vmin - kSlack);
  need_u = (int)floor(t.umax + kSlack) + 2 - u0;
  need_v = (int)floor(t.vmax + kSlack) + 2 - v0;
}

// Coefficients for view k of this tile; returns skip.
__device__ bool tile_view_coef(const BPArgs& a, int k, int ix0, int iy0, int iz0, int ex, int ey, int ez,
                               ViewCoef& vc, int& u0, int& v0, int& need_u, int& need_v, bool& overflow,
                               bool& behind) {
  TileGeo t;
  tile_geo(a, k, ix0, iy0, iz0, ex, ey, ez, t);
  behind = t.dmin <= 1e-6;
  const bool skip = tile_skip(a, t);
  tile_window(a, t, u0, v0, need_u, need_v);
  overflow = !skip && (need_u > a.box_u || need_v - a.pair_rows > a.box_v);
  const double du0 = a.cu - u0, dv0 = a.cv - v0;
  vc.Dx = (float)t.Dx;
  vc.Dz = (float)t.Dz;
  vc.D0 = (float)t.D0;
  vc.Nx = (float)(t.Ux + du0 * t.Dx);
  vc.Nz = (float)(t.Uz + du0 * t.Dz);
  vc.N0 = (float)(t.U0 + du0 * t.D0);
  vc.Vx = (float)(dv0 * t.Dx);
  vc.Vz = (float)(dv0 * t.Dz);
  vc.V0 = (float)(t.G * t.Yc + dv0 * t.D0);
  vc.wscale = a.inv_scale ? a.inv_scale[k] : 1.0f;
  // largest row step of the tile (FP32 rounding of the walk stays far below the margin)
  vc.skip = (skip ? 1 : 0) | (a.dvn < 0.999 * t.dmin ? 2 : 0);
  return skip;
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ float lds_f32(uint32_t addr) {
  float v;
  asm("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ float2 lds_f32x2(uint32_t addr) {
  float2 v;
  asm("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr));
  return v;
}
__device__ __forceinline__ __half2 lds_h2(uint32_t addr) {
  uint32_t v;
  asm("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr));
  return *reinterpret_cast<__half2*>(&v);
}

// Two FP32 FMAs in one instruction (sm_100 packed f32x2), d = a * b + c per lane.
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) {
  unsigned long long ra, rb, rc, rd;
  asm("mov.b64 %0, {%1, %2};" : "=l"(ra) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(rb) : "f"(b.x), "f"(b.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(rc) : "f"(c.x), "f"(c.y));
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(rd) : "l"(ra), "l"(rb), "l"(rc));
  float2 d;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(rd));
  return d;
}

__device__ __forceinline__ unsigned long long pack2(float2 a) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long r) {
  float2 d;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(r));
  return d;
}
// a + b per lane rounded toward zero or to nearest, and a - b rounded to nearest (packed f32x2)
__device__ __forceinline__ float2 fadd2_rz(float2 a, float2 b) {
  unsigned long long d;
  asm("add.rz.f32x2 %0, %1, %2;" : "=l"(d) : "l"(pack2(a)), "l"(pack2(b)));
  return unpack2(d);
}
__device__ __forceinline__ float2 fadd2(float2 a, float2 b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(pack2(a)), "l"(pack2(b)));
  return unpack2(d);
}
__device__ __forceinline__ float2 fsub2(float2 a, float2 b) {
  unsigned long long d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(pack2(a)), "l"(pack2(b)));
  return unpack2(d);
}

__device__ __forceinline__ float2 fmul2(float2 a, float2 b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(pack2(a)), "l"(pack2(b)));
  return unpack2(d);
}

// Value I (0..15) of a kLayoutQuadG24 element held in 12 words: its three
// bytes sit at byte 3 I, and the float is rebuilt as (bytes << 8) | low byte.
template <int I>
__device__ __forceinline__ float dec24(const uint32_t (&w)[12]) {
  constexpr int B = 3 * I, W = B >> 2, O = B & 3;
  constexpr int W1 = W + 1 < 12 ? W + 1 : W;  // the last value needs no second word
  constexpr unsigned sel = O | (O << 4) | ((O + 1) << 8) | ((O + 2) << 12);
  return __uint_as_float(__byte_perm(w[W], w[W1], sel));
}

__device__ __forceinline__ uint4 lds_u4(uint32_t addr) {
  uint4 v;
  asm("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}

// Hardware approximate reciprocal (max 1 ulp error; D is a distance ratio near 1).
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// The same after one Newton-Raphson step, r + r (1 - x r): as good as a rounded
// division here (error against FP64 to three digits), at a third of its cost.
__device__ __forceinline__ float rcp_newton(float x) {
  const float r = rcp_approx(x);
  return fmaf(r, fmaf(-x, r, 1.f), r);
}

// FP16 x FP16 + FP32 with one rounding to FP32.
__device__ __forceinline__ float fma_f16_f32(__half a, __half b, float c) {
  float d;
  asm("fma.rn.f32.f16 %0, %1, %2, %3;" : "=f"(d) : "h"(__half_as_ushort(a)), "h"(__half_as_ushort(b)), "f"(c));
  return d;
}

constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23
constexpr uint32_t kMagicBits = 0x4B400000u;

template <int LAYOUT, int TX, int TZ, int NY>
__global__ void __launch_bounds__(TX* TZ + 32, 2) bp_kernel(const __grid_constant__ BoxMaps maps, const BPArgs a) {
  static_assert(TX % 8 == 0 && TZ % 4 == 0, "warp tile is 8 x 4 columns");
  constexpr int NCW = TX * TZ / 32;  // consumer warps
  extern __shared__ __align__(1024) unsigned char smem[];
  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  const int S = a.chunk;  // ring stages (one view each)
  const int bx = blockIdx.x % a.ntx, bz = blockIdx.x / a.ntx;
  const int ix0 = bx * TX, iz0 = bz * TZ, iy0 = blockIdx.y * NY;

  ViewCoef* coef = reinterpret_cast<ViewCoef*>(smem + (size_t)S * a.box_bytes);
  uint64_t* full = reinterpret_cast<uint64_t*>(coef + S);
  uint64_t* empty = full + S;
  volatile int* s_abort = reinterpret_cast<volatile int*>(empty + S);

  if (tid == 0) {
    *s_abort = *(volatile int*)a.err != 0;
    for (int s = 0; s < S; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], NCW);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  if (*s_abort) return;

  if (warp == NCW) {
    // ---------------------------------------------------------------- producer
    // Lane l computes view kb + l of each batch of 32; then the views are
    // staged in order, each with the smallest box of the grid that holds it.
    int issued = 0;
    for (int kb = 0; kb < a.nviews && !*s_abort; kb += 32) {
      const int k = kb + lane;
      ViewCoef vc;
      int u0 = 0, v0 = 0, wi = 0, hi = 0;
      bool skip = true;
      vc.skip = 1;
      if (k < a.nviews) {
        bool overflow = false, behind = false;
        int need_u = 0, need_v = 0;
        // full tile extents: every consumer thread's samples lie in the window
        skip = tile_view_coef(a, k, ix0, iy0, iz0, TX - 1, NY - 1, TZ - 1, vc, u0, v0, need_u, need_v, overflow,
                              behind);
        if (overflow) atomicCAS(a.err, 0, kDevFootprint);
        if (behind) atomicCAS(a.err, 0, kDevGeometry);
        if (overflow || behind) skip = true, vc.skip = 1;
        const int rows = need_v - a.pair_rows;  // element rows to stage
        while (wi < kNW - 1 && maps.w[wi] < need_u) ++wi;
        while (hi < kNH - 1 && maps.h[hi] < rows) ++hi;
        vc.box = maps.w[wi] | (maps.h[hi] << 16);
      }
      const int nb = min(32, a.nviews - kb);
      for (int i = 0; i < nb; ++i) {
        const int kk = kb + i;
        const int s = kk % S;
        if (kk >= S && !mbar_wait(&empty[s], ((kk / S) & 1) ^ 1, a.err)) {
          *s_abort = 1;
          break;
        }
        if (lane == i) coef[s] = vc;
        const int sk = __shfl_sync(0xffffffffu, (int)skip, i);
        const int cu0 = __shfl_sync(0xffffffffu, u0, i), cv0 = __shfl_sync(0xffffffffu, v0, i);
        const int mi = __shfl_sync(0xffffffffu, wi * kNH + hi, i);
        __syncwarp();
        if (lane == 0) {
          if (sk) {
            mbar_arrive(&full[s]);
          } else {
            const CUtensorMap* m = &maps.map[mi];
            mbar_arrive_expect_tx(&full[s], (uint32_t)(maps.w[mi / kNH] * maps.h[mi % kNH] * 4));
            const int e0 = cv0 + a.pair_rows;  // pair layout: row v is element row v + 1
            void* dst = smem + (size_t)s * a.box_bytes;
            if (a.sino_layout)
              tma_load_3d(dst, m, cu0, kk, e0, &full[s]);
            else
              tma_load_3d(dst, m, cu0, e0, kk, &full[s]);
          }
        }
        __syncwarp();
        issued = kk + 1;
      }
    }
    // leave only when every copy issued into this CTA's memory has landed
    for (int kk = max(0, issued - S); kk < issued; ++kk) mbar_wait(&full[kk % S], (kk / S) & 1, a.err);
    return;
  }

  // ------------------------------------------------------------------ consumers
  constexpr int WX = TX / 8;
  const int tx = (warp % WX) * 8 + (lane & 7);
  const int tz = (warp / WX) * 4 + (lane >> 3);
  const float fx = (float)tx, fz = (float)tz;
  constexpr int ESZ = 4;
  // rows of a window usable as floor(v): all for the pair layout, all but the
  // last for the raw layout (it also reads row v + 1)
  constexpr int kRowTail = LAYOUT == kLayoutRaw32 ? 1 : 0;

  float acc[NY];
#pragma unroll
  for (int j = 0; j < NY; ++j) acc[j] = 0.f;

  int s = 0;
  uint32_t ph = 0;
  bool bad = false;
  for (int k = 0; k < a.nviews; ++k) {
    if (!mbar_wait(&full[s], ph, a.err)) {
      *s_abort = 1;
      break;
    }
    const ViewCoef g = coef[s];
    if (!(g.skip & 1)) {
      const float D = fmaf(g.Dx, fx, fmaf(g.Dz, fz, g.D0));
      const float rD = rcp_newton(D);
      const float ul = fmaf(g.Nx, fx, fmaf(g.Nz, fz, g.N0)) * rD;
      const float vl = fmaf(g.Vx, fx, fmaf(g.Vz, fz, g.V0)) * rD;
      const float dvv = a.dvn * rD;
      const float W = rD * rD * g.wscale;
      const float fuf = floorf(ul);
      const int iu = (int)fuf;
      const float fu = ul - fuf;
      const float vlast = fmaf((float)(NY - 1), dvv, vl);
      const int BU = g.box & 0xffff, BV = g.box >> 16;
      const uint32_t RB = (uint32_t)(BU * ESZ);
      // exclusive bound on v, kSlack / 2 inside the window: the footprint pass
      // leaves kSlack, so the guard never trips for a voxel of the tile, and
      // the rounded row index can never pass the last staged row
      const float vmax_ok = (float)(BV - kRowTail) - (float)(kSlack / 2);
      if (iu >= 0 && iu <= BU - 2 && vl >= 0.f && vlast < vmax_ok) {
        const uint32_t c0 = smem_u32(smem + (size_t)s * a.box_bytes) + (uint32_t)(iu * ESZ) - kMagicBits * RB;
        // floor and fraction of v with the rounding constant: v + kMagic toward
        // zero is kMagic + floor(v), whose bit pattern times RB plus c0 is the
        // element's address; two voxels at a time in packed FP32. v is formed anew
        // for each voxel: stepped from the one before, its rounding adds up
        const float2 magic2 = make_float2(kMagic, kMagic);
        auto v_at = [&](int j) { return make_float2(fmaf((float)j, dvv, vl), fmaf((float)(j + 1), dvv, vl)); };
        if constexpr (LAYOUT == kLayoutRaw32) {
          // where the rows advance by less than one per voxel, march along the
          // column: a voxel's upper row, interpolated in u (the distance weight
          // folded in), is the next voxel's lower row or its upper one again,
          // so a voxel reads one new row (8 bytes) instead of two
          const float wb = W * fu, wa = W - wb;
          auto load = [&](uint32_t at) { return fmaf(wb, lds_f32(at + 4), wa * lds_f32(at)); };
          auto march = [&](auto shortc) {
            constexpr bool SHORT = decltype(shortc)::value;
            float lo = 0.f, hi = 0.f;
            uint32_t before = 0;
#pragma unroll
            for (int j = 0; j < NY; j += 2) {
              const float2 v2 = v_at(j), t2 = fadd2_rz(v2, magic2);
              const float2 fv2 = fsub2(v2, fsub2(t2, magic2));
#pragma unroll
              for (int p = 0; p < 2 && j + p < NY; ++p) {
                const uint32_t bits = __float_as_uint(p ? t2.y : t2.x);
                const uint32_t at = bits * RB + c0;
                if (j + p == 0 || !SHORT) lo = load(at);
                else lo = bits == before ? lo : hi;
                hi = load(at + RB);
                acc[j + p] += fmaf(p ? fv2.y : fv2.x, hi - lo, lo);
                before = bits;
              }
            }
          };
          if (g.skip & 2) march(std::true_type{});
          else march(std::false_type{});
        } else {
          // element = (row v, row v + 1 minus row v); the u-lerp of both in FP32
#pragma unroll
          for (int j = 0; j < NY; j += 2) {
            const float2 v2 = v_at(j), t2 = fadd2_rz(v2, magic2);
            const float2 fv2 = fsub2(v2, fsub2(t2, magic2));
#pragma unroll
            for (int p = 0; p < 2 && j + p < NY; ++p) {
              const uint32_t at = __float_as_uint(p ? t2.y : t2.x) * RB + c0;
              const float2 x = __half22float2(lds_h2(at)), y = __half22float2(lds_h2(at + 4));
              const float2 ag = ffma2(make_float2(fu, fu), fsub2(y, x), x);
              acc[j + p] = fmaf(W, fmaf(p ? fv2.y : fv2.x, ag.y, ag.x), acc[j + p]);
            }
          }
        }
      } else {
        bad = true;  // cannot happen when the footprint pass is right; recorded below
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[s]);
    if (++s == S) {
      s = 0;
      ph ^= 1;
    }
  }
  if (bad) atomicCAS(a.err, 0, kDevFootprint);
  if (*s_abort) return;

  const int ix = ix0 + tx, iz = iz0 + tz;
  float lo = __int_as_float(0x7f800000), hi = -lo;
  if (ix < a.nx && iz < a.nz) {
    float* out = a.vol + ((size_t)iz * a.vol_ystride) * a.nx + ix;
#pragma unroll
    for (int j = 0; j < NY; ++j) {
      const int iy = iy0 + j;
      if (iy < a.ny) {
        float r = acc[j] * a.scale;
        if (iy < a.clip_ylimit) r = fmaxf(r, 0.f);
        out[(size_t)iy * a.nx] = r;
        lo = fminf(lo, r);
        hi = fmaxf(hi, r);
      }
    }
  }
  if (a.minmax) fold_minmax(a.minmax, lo, hi);
}

// ---------------------------------------------------------------------------
// Four-fold symmetric backprojector.
//
// On a circular orbit with K views over one turn (K % 4 == 0) and a square
// volume (nx == nz), voxel P = (X, Z) at view k and the voxel rotated by 90
// degrees, (-Z, X), at view k + K/4 project to the same detector coordinate
// (t = X cos + Z sin and s = -X sin + Z cos are unchanged). A CTA therefore
// owns an orbit of four 16 x 16 x NY tiles (a tile of the lower-left quadrant
// and its three rotations) and walks all K views of the representative tile:
// one warp computes the tile footprint and coefficients once per view k, a
// second one stages one window of the interleaved stack, whose element holds the
// samples of the views g + s K/4 (g = k mod K/4) in slots s = 0 .. 3; each
// consumer thread forms its detector column, weights and v steps once per view
// and applies every floor / fraction / address to four accumulator sets.
// Rotation r of the tile reads slot (m + r) mod 4 at view k = g + m K/4: the
// sums stay in slot order and are turned by one slot whenever the walk passes
// from one quarter turn to the next, so one copy of the tap code serves all
// quarters. Windows live in a byte ring (entries of variable size, freed in
// order), so typical small windows keep several views in flight while the
// largest still fits.
//
// Layouts: FP16 and 24-bit gradient quads (MIXED, MIXED24), whose element
// carries everything a tap needs, and plain FP32 quads (FP32 form), where a
// tap needs two rows of two columns. A column's voxels share u, so the FP32
// taps march along it: the row above the previous voxel's becomes this
// voxel's lower row, already interpolated in u, and each voxel reads one new
// row (two 16-byte loads, 8 bytes an update, against 16 for the four samples)
// as long as the rows advance by at most one per voxel, and a second one where
// they advance by more.
//
// Bound (counters at 256^3): FP32, the shared-memory wavefronts of the load /
// store unit (81% of its rate; issue slots 61%, heavy FMA pipe 60%); MIXED, the
// FMA pipes' dependent chains (heavy pipe 70%, issue 65%, wavefronts 68%);
// 24-bit, wavefronts 78% and issue 70% (12 bytes and four half-rate byte
// permutes an update, which the FP32 form does without: it is the faster one);
// FP16 row pairs on orbits, the heavy FMA pipe (76%).
// Measured, backprojection with its packing, before = four row-pair windows
// (FP32) or the quarters unrolled (MIXED), 8 consumer warps, one producer warp:
//            256^3 x 360     512^3 x 720     480^3 x 480*    768^3 x 1024
//   FP32     3.59 -> 2.51    55.6 -> 37.4    23.8 -> 17.3    264.6 -> 175.9 ms
//   MIXED    2.66 -> 2.45    39.4 -> 36.2    15.9 -> 14.7    185.5 -> 163.6 ms
//   24-bit   3.63 -> 3.11    52.8 -> 44.7    20.9 -> 19.1    247.5 -> 208.7 ms
// (* the 1440^3 geometry at a third). Tried and slower: fetching a view's record
// and projection before the previous view's taps (and two windows held at once
// can need more than the ring), 16 voxels a thread for FP32.

constexpr int kQuadEntries = 8;  // outstanding view-quads per CTA

// Quad record flags.
constexpr int kQSkip = 1;    // the tile footprint misses the detector (or failed a check): no taps
constexpr int kQDirect = 2;  // window not staged, consumers gather it from global memory
constexpr int kQFirst = 4;   // first quad of a work item (a tile orbit and y-slab of one job)
constexpr int kQLast = 8;    // last quad of a work item: the consumers store its voxels next
constexpr int kQExit = 16;   // multi-job launch: the queue is empty, the CTA leaves
constexpr int kQTurn = 32;   // last view of a quarter turn: the sums move on by one slot
constexpr int kQShort = 64;  // rows advance by less than one per voxel everywhere in the tile

// 16-byte aligned so that consumers read a record with vector loads: four for
// every layout, the fifth (weights) for the FP16 views, the last for windows
// that are not staged and for the next item
struct alignas(16) QuadCoef {
  float Dx, Dz, D0, Nx;
  float Nz, N0, Vx, Vz;
  float V0;
  float dvn;       // the job's v step per voxel times D
  float vmax;      // exclusive bound on the window-local v of a tap
  int flags;       // kQ* bits
  // consumer constants of the window, formed once by the producer
  uint32_t cbase;  // ring address of element column 0 minus kMagicBits element rows
  uint32_t rb;     // bytes per staged element row
  int bu2;         // last element column a tap may start at (box width - 2)
  uint32_t plane;  // bytes between the 16-byte planes of an element row
  float ws[4];     // per-view extra weight of the four slots (FP16 views: 1 / scale)
  int grp;         // view group
  int u0, e0;      // direct: element column / element row of the window origin
  int item;        // work item of this quad
};
static_assert(sizeof(QuadCoef) == 96, "six 16-byte loads per record");

// A quad from the geometry warp to the issuing warp: the consumers' record
// (its ring address still open) and its copy.
struct alignas(16) QuadStage {
  QuadCoef qc;
  int need, tx_bytes;  // ring bytes, bytes of the copy (0, -: nothing to copy)
  int x, y, grp, mi;   // tensor coordinates and box
  int pad[2];
};
constexpr int kGeoQuads = 32;  // quads per block between the two (one a lane)
static_assert(sizeof(QuadStage) == 128, "stage records");

__device__ __forceinline__ void named_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void named_arrive(int id, int threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Multi-job launch (several reconstructions in one persistent launch): one
// entry per job in global memory; work item item0 + i of job j is the job's
// tile t0 + i (tiles ordered y-slab, then z, then x), so a launch can carry
// a whole job or a range of its tiles.
struct QuadJob {
  BPArgs a;
  long long item0;  // first work item of the job in this launch
  long long t0;     // its tile
};
struct QuadQueue {
  const QuadJob* jobs;    // sorted by item0
  const BoxMaps* maps;    // one grid of tensor maps per job
  int njobs;
  long long nitems;
  unsigned long long* next;  // work-item counter (zero before the launch)
  int* err;                  // device error word of the launch
  int ring;                  // ring bytes of every CTA
};

__device__ __forceinline__ int find_job(const QuadQueue& qq, long long item) {
  int lo = 0, hi = qq.njobs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (qq.jobs[mid].item0 <= item) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

template <bool MULTI>
__device__ __forceinline__ const BPArgs& job_args(const BPArgs& a, const QuadQueue& qq, int jb) {
  if constexpr (MULTI) return qq.jobs[jb].a;
  else return a;
}
template <bool MULTI>
__device__ __forceinline__ const BoxMaps& job_maps(const BoxMaps& m, const QuadQueue& qq, int jb) {
  if constexpr (MULTI) return qq.maps[jb];
  else return m;
}

// Tile of a work item and the first view of its walk. The walk starts at an
// offset advanced by about K views per `resident` CTAs in tile order: tiles
// that run at the same time then read the same views (their windows share L2)
// instead of all starting at view 0. The offset depends only on the tile, so
// results are the same whichever CTA, launch or batch computes it.
//
// Tile order within a y-slab: bands of `band` orbit rows along z, walked
// column by column along x, so the ~`resident` tiles that run at once form a
// near-square patch of the slab (band ~ sqrt(resident)); their windows of one
// view group then span about half the detector columns a slab-wide row of
// tiles would, and DRAM reads of the filtered views fall in proportion.
struct ItemTile {
  int ix0, iy0, iz0;
  int k0;
};
template <int NY>
__device__ __forceinline__ ItemTile item_tile(const BPArgs& ja, long long t) {
  ItemTile it;
  const long long per = (long long)ja.nbx * ja.nbz;
  const int by = (int)(t / per);
  const int rem = (int)(t - (long long)by * per);
  const int H = min(max(1, ja.band), ja.nbz);
  const int b = rem / (H * ja.nbx);
  const int hb = min(H, ja.nbz - b * H);  // orbit rows in this band (the last may be short)
  const int r2 = rem - b * H * ja.nbx;
  const int bx = r2 / hb, bz = b * H + (r2 - bx * hb);
  it.ix0 = bx * 16;
  it.iz0 = bz * 16;
  it.iy0 = by * NY;
  const int K = ja.nviews;
  it.k0 = (int)((t * K / max(1, ja.resident)) % K);
  return it;
}

// Shapes. A CTA's representative tile is 16 x 16 columns x TY = NY YW voxels:
// eight consumer warps, or two times eight one above the other (YW = 2), of 32
// columns x NY voxels (4 NY sums a thread), then the issuing warp and the
// geometry warp. What separates the shapes is how many consumer warps a
// scheduler has to hide the taps' chains behind one another (8 of NY = 16: two;
// 16 of NY = 8 or 12: four) against the registers they leave (168, 96 .. 112)
// and the work per view and thread, which is the same for any NY (about a fifth
// of the instructions at NY = 16, a third at 8). Launches give every warp the
// same registers; the shapes that need more for their consumers get whole
// warpgroups (four warps, two of them idle) of producers and move the
// producers' surplus with setmaxnreg: 640 x 96 = 512 x 112 + 128 x 32, 384 x 80
// = 256 x 104 + 128 x 32.
constexpr bool quad_moves_regs(int layout, int NY, int YW) { return YW == 2 || (layout == kLayoutQuad32 && NY == 12); }
constexpr int quad_threads(int layout, int NY, int YW) {
  return 256 * YW + (quad_moves_regs(layout, NY, YW) ? 128 : 64);
}

// MULTI = false: one job, one work item (tile orbit and y-slab) per CTA, from
// the block index. MULTI = true: a persistent launch of OCC CTAs per SM over
// the work items of several jobs (uneven sizes, each with its own geometry,
// views and tensor maps, all of one staged layout); the producer takes the
// next item from the queue's counter and streams its quads into the ring
// without a pause between items, the consumers reset their sums at an item's
// first quad and store its voxels after its last. An item's arithmetic and
// view order do not depend on the launch, so a job's volume is the same bits
// alone or batched with others.
// EDGES: volumes that are not whole tiles to the half, and walks whose last
// phase does not lead back by one slot (the epilogue's conditions cost the
// 24-bit and the 12-high FP32 shapes 2 to 3% through their registers).
template <int LAYOUT, int NY, int YW, int OCC, bool MULTI, bool EDGES>
__global__ void __launch_bounds__(quad_threads(LAYOUT, NY, YW), OCC)
    bp_quad_kernel(const __grid_constant__ BoxMaps maps, const __grid_constant__ BPArgs a,
                   const __grid_constant__ QuadQueue qq) {
  constexpr int TX = 16, TZ = 16, TY = NY * YW, NCW = 8 * YW, E = kQuadEntries;
  constexpr bool Q24 = LAYOUT == kLayoutQuadG24;
  constexpr bool Q32 = LAYOUT == kLayoutQuad32 || LAYOUT == kLayoutDuo32;
  constexpr bool P16 = is_p16_layout(LAYOUT);
  constexpr bool GRAD = is_grad_layout(LAYOUT);
  constexpr int S = slots_of(LAYOUT);
  // whether a step tells the end of a phase, or the walk counts (512^3, 24-bit
  // 46.5 / 46.4 ms, 960-wide FP32 273.8 / 266.4, 768^3 FP16 163.7 / 165.6: what
  // ptxas keeps in registers)
  constexpr bool FLAGGED = MULTI || LAYOUT == kLayoutQuadG16;
  constexpr int NPL = Q24 ? 3 : GRAD ? 2 : 1;  // planes per element row
  constexpr int CB = S == 4 ? 16 : 8;          // bytes per column of a plane
  constexpr int ESZ = CB * NPL;
  constexpr int kRowTail = Q32 ? 1 : 0;  // a tap also reads the next element row
  constexpr int kCol0 = GRAD ? 1 : 0;    // element column of detector column 0 (gradient elements start at -1)
  extern __shared__ __align__(1024) unsigned char smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int R = MULTI ? qq.ring : a.box_bytes;  // ring bytes
  int* const err = MULTI ? qq.err : a.err;

  QuadCoef* coef = reinterpret_cast<QuadCoef*>(smem + R);
  QuadStage* stage = reinterpret_cast<QuadStage*>(coef + E);  // two blocks
  uint64_t* full = reinterpret_cast<uint64_t*>(stage + 2 * kGeoQuads);
  uint64_t* empty = full + E;
  // end_pos: ring byte position (64-bit: a persistent CTA allocates far more
  // than 2^31 bytes over its items) where each entry's windows end
  long long* end_pos = reinterpret_cast<long long*>(empty + E);
  volatile int* s_abort = reinterpret_cast<volatile int*>(end_pos + E);
  volatile int* hdr = s_abort + 1;  // per block: quads (-1: no more), job

  if (tid == 0) {
    *s_abort = *(volatile int*)err != 0;
    for (int e = 0; e < E; ++e) {
      mbar_init(&full[e], 1);
      mbar_init(&empty[e], NCW);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  if (*s_abort) return;

  // Named barriers between the two producer warps: block b full, block b free
  constexpr int kBarFull = 1, kBarFree = 3;
  if (warp >= NCW) {
    if constexpr (quad_moves_regs(LAYOUT, NY, YW)) asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
    if (warp > NCW + 1) return;
  }
  if (warp == NCW + 1) {
    // ---------------------------------------------------------------- geometry
    // one quad a lane, a block ahead of the issuing warp: its FP64 chains and
    // (at 32 registers) spills stay off the ring's path
    int b = 0, blocks = 0;
    bool first = true;
    while (!*s_abort) {
      // the next work item: this CTA's tile, or the queue's next item
      long long item;
      if constexpr (MULTI) {
        unsigned long long t = 0;
        if (lane == 0) t = atomicAdd(qq.next, 1ull);
        item = (long long)__shfl_sync(0xffffffffu, t, 0);
        if (item >= qq.nitems) break;
      } else {
        if (!first) break;
        item = (long long)blockIdx.y * gridDim.x + blockIdx.x;
      }
      first = false;
      const int jb = MULTI ? find_job(qq, item) : 0;
      const BPArgs& ja = job_args<MULTI>(a, qq, jb);
      const BoxMaps& jm = job_maps<MULTI>(maps, qq, jb);
      const long long t_local = MULTI ? item - qq.jobs[jb].item0 + qq.jobs[jb].t0 : item;
      const ItemTile til = item_tile<TY>(ja, t_local);
      const int K = ja.nviews, Q = ja.groups;
      for (int kb = 0; kb < K && !*s_abort; kb += kGeoQuads) {
        if (blocks >= 2) named_sync(kBarFree + b, 64);
        const int it = kb + lane;         // quad of the item (ring entry order)
        const int k = (it + til.k0) % K;  // view of the representative tile
        if (it < K) {
          QuadStage& st = stage[b * kGeoQuads + lane];
          ViewCoef vc;
          bool overflow = false, behind = false;
          int u0, v0, need_u = 0, need_v = 0;
          bool skip = tile_view_coef(ja, k, til.ix0, til.iy0, til.iz0, TX - 1, TY - 1, TZ - 1, vc, u0, v0, need_u,
                                     need_v, overflow, behind);
          // checks of the job's geometry go to the job's error word
          if (overflow) atomicCAS(ja.err, 0, kDevFootprint);
          if (behind) atomicCAS(ja.err, 0, kDevGeometry);
          if (overflow || behind) skip = true;
          int wi = 0, hi = 0;
          const int rows = need_v - ja.pair_rows;
          while (wi < kNW - 1 && jm.w[wi] < need_u) ++wi;
          while (hi < kNH - 1 && jm.h[hi] < rows) ++hi;
          const int tx_bytes = jm.w[wi] * jm.h[hi] * ESZ;
          const int bytes = (tx_bytes + 127) & ~127;
          // a window wider than the widest box or larger than the ring (rare
          // near-source tiles) is read from global memory instead
          const bool direct = !skip && (need_u > jm.w[kNW - 1] || rows > jm.h[kNH - 1] || bytes > R);
          st.need = (skip || direct) ? 0 : bytes;
          st.tx_bytes = tx_bytes;
          st.x = CB / 8 * (u0 + kCol0);
          st.y = v0 + ja.pair_rows;
          st.grp = k % Q;
          st.mi = wi * kNH + hi;
          QuadCoef& qc = st.qc;
          qc.Dx = vc.Dx; qc.Dz = vc.Dz; qc.D0 = vc.D0;
          qc.Nx = vc.Nx; qc.Nz = vc.Nz; qc.N0 = vc.N0;
          qc.Vx = vc.Vx; qc.Vz = vc.Vz; qc.V0 = vc.V0;
#pragma unroll
          for (int r = 0; r < S; ++r)
            qc.ws[r] = ja.inv_scale ? ja.inv_scale[k % Q + (r < ja.mirror ? r : r - ja.mirror) * Q] : 1.0f;
          qc.flags = (skip ? kQSkip : 0) | (direct ? kQDirect : 0) | (it == 0 ? kQFirst : 0) |
                     (it == K - 1 ? kQLast : 0) | ((k + 1) % Q == 0 ? kQTurn : 0) | (vc.skip & 2 ? kQShort : 0);
          // window: width (elements) and rows
          const int BU = direct ? need_u : jm.w[wi], BV = direct ? rows : jm.h[hi];
          qc.grp = k % Q;
          qc.u0 = u0 + kCol0;
          qc.e0 = v0 + ja.pair_rows;
          qc.rb = (uint32_t)(BU * ESZ);
          qc.plane = (uint32_t)(BU * CB);
          qc.bu2 = BU - 2;
          qc.vmax = (float)(BV - kRowTail) - (float)(kSlack / 2);
          qc.dvn = ja.dvn;
          qc.item = (int)item;
        }
        if (lane == 0) {
          hdr[2 * b] = min(kGeoQuads, K - kb);
          hdr[2 * b + 1] = jb;
        }
        __syncwarp();
        named_arrive(kBarFull + b, 64);
        b ^= 1;
        ++blocks;
      }
    }
    if (blocks >= 2) named_sync(kBarFree + b, 64);
    if (lane == 0) hdr[2 * b] = -1;
    __syncwarp();
    named_arrive(kBarFull + b, 64);
    if (blocks >= 1) named_sync(kBarFree + (b ^ 1), 64);  // the last block's release: no arrival is left pending
    return;
  }
  if (warp == NCW) {
    // ----------------------------------------------------------------- issuing
    // head / tail: ring bytes allocated / freed; hpos = head mod R; oldest:
    // first quad not yet known to be released; seq: quads issued since the
    // launch (all items)
    long long head = 0, tail = 0;
    int hpos = 0, oldest = 0, seq = 0;
    for (int b = 0;; b ^= 1) {
      named_sync(kBarFull + b, 64);
      const int nb = hdr[2 * b];
      if (nb < 0) break;
      const BoxMaps& jm = job_maps<MULTI>(maps, qq, MULTI ? hdr[2 * b + 1] : 0);
      for (int i = 0; i < nb && !*s_abort; ++i) {  // after an abort the blocks are only handed back
        const QuadStage& st = stage[b * kGeoQuads + i];
        const int q = seq, e = q % E;  // ring sequence number and entry
        const int qneed = st.need;
        // allocate qneed contiguous ring bytes: wrap to 0 when the tail end is too short
        const bool wrap = hpos + qneed > R;
        const long long start = wrap ? head + (R - hpos) : head;
        bool ok = true;
        while (oldest < q && (oldest <= q - E || start + qneed - tail > R)) {
          if (!mbar_wait(&empty[oldest % E], (oldest / E) & 1, err)) {
            ok = false;
            break;
          }
          tail = end_pos[oldest % E];
          ++oldest;
        }
        if (!ok) {
          *s_abort = 1;
          break;
        }
        if (oldest == q) tail = start;    // nothing outstanding: the whole ring is free
        const int off = wrap ? 0 : hpos;  // start mod R
        // the record, one word a lane, its ring address filled in
        constexpr int kWords = sizeof(QuadCoef) / 4, kBaseWord = offsetof(QuadCoef, cbase) / 4;
        if (lane < kWords) {
          uint32_t w = reinterpret_cast<const uint32_t*>(&st.qc)[lane];
          if (lane == kBaseWord) w = smem_u32(smem) + (uint32_t)off - kMagicBits * st.qc.rb;
          reinterpret_cast<uint32_t*>(&coef[e])[lane] = w;
        }
        if (lane == 0) end_pos[e] = start + qneed;
        head = start + qneed;
        hpos = off + qneed == R ? 0 : off + qneed;
        __syncwarp();
        if (lane == 0) {
          if (qneed == 0) {
            mbar_arrive(&full[e]);
          } else {
            mbar_arrive_expect_tx(&full[e], (uint32_t)st.tx_bytes);
            tma_load_4d(smem + off, &jm.map[st.mi], st.x, 0, st.y, st.grp, &full[e]);
          }
        }
        __syncwarp();
        ++seq;
      }
      named_arrive(kBarFree + b, 64);
    }
    if (MULTI && !*s_abort) {
      // queue empty: one record that tells the consumers to leave
      const int q = seq, e = q % E;
      bool ok = true;
      while (oldest < q && oldest <= q - E) {
        if (!mbar_wait(&empty[oldest % E], (oldest / E) & 1, err)) {
          ok = false;
          break;
        }
        ++oldest;
      }
      if (ok) {
        if (lane == 0) {
          coef[e].flags = kQExit | kQSkip;
          mbar_arrive(&full[e]);
        }
        __syncwarp();
        ++seq;
      } else {
        *s_abort = 1;
      }
    }
    // leave only when every copy issued into this CTA's memory has landed
    for (int q = max(0, seq - E); q < seq; ++q) mbar_wait(&full[q % E], (q / E) & 1, err);
    return;
  }

  if constexpr (YW == 2) asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
  else if constexpr (quad_moves_regs(LAYOUT, NY, YW)) asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
  // ------------------------------------------------------------------ consumers
  // a warp owns 8 x 4 columns; each quarter-warp (one shared-memory phase of
  // 16-byte loads) is a compact 4 x 2 patch, whose detector columns stay
  // within 8 elements (no bank conflicts)
  const int tx = (warp & 1) * 8 + ((lane >> 3) & 1) * 4 + (lane & 3);
  const int tz = ((warp >> 1) & 3) * 4 + (lane >> 4) * 2 + ((lane >> 2) & 1);
  const int ty = (warp >> 3) * NY;  // first of this warp's voxels along y
  const float fx = (float)tx, fz = (float)tz;
  // plain FP32 sums: four slots x NY voxels in registers (a compensated sum
  // was measured to change no digit of the MIXED form's error, which the
  // FP16 views set, and cost 5% at C4)
  float acc[S][NY];
  // the next phase: its slot s belongs to the rotation of slot s - 1
  auto turn = [&]() {
#pragma unroll
    for (int j = 0; j < NY; ++j) {
      const float t = acc[S - 1][j];
#pragma unroll
      for (int s = S - 1; s > 0; --s) acc[s][j] = acc[s - 1][j];
      acc[0][j] = t;
    }
  };
  // a new work item: zero every sum of this thread
  auto reset = [&]() {
#pragma unroll
    for (int r = 0; r < S; ++r)
#pragma unroll
      for (int j = 0; j < NY; ++j) acc[r][j] = 0.f;
  };
  reset();
  int e = 0;
  uint32_t ph = 0;
  bool bad = false, stop = false, last = false, leave = false, turned = false;
  long long item = -1;  // work item being accumulated
  int jb = 0;         // its job
  // one quad: wait for its window, apply it to the 4 x NY voxels, release it
  auto step = [&]() {
    if (!mbar_wait(&full[e], ph, err)) {
      *s_abort = 1;
      stop = true;
      return;
    }
    const QuadCoef g = coef[e];  // all of it at once: one latency
    const int flags = g.flags;
    if constexpr (MULTI) {  // one job's single item: set up before the loop, the loop counts its quads
      if (flags & (kQExit | kQFirst)) {
        if (flags & kQExit) {  // no more items
          leave = true;
        } else {
          item = g.item;
          jb = find_job(qq, item);
        }
      }
      last = (flags & kQLast) != 0;
    }
    if (!(flags & kQSkip)) {
      // explicit roundings (no contraction): the same bits in every instantiation
      const float D = fmaf(g.Dx, fx, fmaf(g.Dz, fz, g.D0));
      const float rD = EDGES ? rcp_newton(D) : rcp_approx(D);
      const float ul = __fmul_rn(fmaf(g.Nx, fx, fmaf(g.Nz, fz, g.N0)), rD);
      const float dvv = __fmul_rn(g.dvn, rD);
      const float vl0 = __fmul_rn(fmaf(g.Vx, fx, fmaf(g.Vz, fz, g.V0)), rD);
      const float vl = YW == 1 ? vl0 : fmaf((float)ty, dvv, vl0);
      const float W = __fmul_rn(rD, rD);
      const float fuf = floorf(ul);
      const int iu = (int)fuf;
      const float fu = ul - fuf;
      const float vlast = fmaf((float)(NY - 1), dvv, vl);
      const uint32_t RB = g.rb;
      if (iu >= 0 && iu <= g.bu2 && vl >= 0.f && vlast < g.vmax) {
        const uint32_t c0 = g.cbase + (uint32_t)(iu * CB);
        // v of voxels j and j + 1, stepped by 2 dvv from (vl, vl + dvv): no
        // per-pair constants (a few ulps of v from the repeated additions, which
        // the orbits of the plain kernel's geometries do without as that does);
        // floor and fraction of the pair with packed FP32 ops
        static_assert(NY % 2 == 0, "voxels stepped in pairs");
        const float2 magic2 = make_float2(kMagic, kMagic);
        const float dv2 = 2.f * dvv;
        const float2 step2 = make_float2(dv2, dv2);
        float2 v2 = make_float2(vl, vl + dvv);
        auto advance = [&](int j) {
          if constexpr (EDGES)
            v2 = ffma2(make_float2((float)j, (float)(j + 1)), make_float2(dvv, dvv), make_float2(vl, vl));
          else if (j)
            v2 = fadd2(v2, step2);
        };
        if constexpr (Q32) {
          // weights of the two columns, the distance weight folded in
          const float wbs = __fmul_rn(W, fu), was = __fsub_rn(W, wbs);
          const float2 wa = make_float2(was, was), wb = make_float2(wbs, wbs);
          // an element row at this thread's detector position: the slots' pairs, interpolated in u
          auto blend = [&](const float2& A, const float2& B) { return ffma2(wb, B, fmul2(wa, A)); };
          // One rounding into a sum: the two products added to it one after the
          // other cost an operation less and a fifth more error (256^3 x 360 4.0
          // -> 4.8e-7 against FP64; 2.76 and 2.82 ms). Two forms of the
          // interpolation, by what ptxas makes of them (12 high 42.3 and 43.4 ms
          // at a drawn 420^3; 8 high 2.84 and 2.82 ms).
          auto add = [&](const float2 (&lo)[S / 2], const float2 (&hi)[S / 2], float fv, int j) {
            const float2 fv2 = make_float2(fv, fv), fl2 = make_float2(1.f - fv, 1.f - fv);
#pragma unroll
            for (int p = 0; p < S / 2; ++p) {
              const float2 t = NY == 12 ? ffma2(fv2, hi[p], fmul2(fl2, lo[p])) : ffma2(fv2, fsub2(hi[p], lo[p]), lo[p]);
              const float2 d = fadd2(make_float2(acc[2 * p][j], acc[2 * p + 1][j]), t);
              acc[2 * p][j] = d.x;
              acc[2 * p + 1][j] = d.y;
            }
          };
          if (!(flags & kQDirect)) {
            auto load = [&](uint32_t at, float2 (&q)[S / 2]) {
              if constexpr (S == 4) {
                const uint4 A = lds_u4(at), B = lds_u4(at + CB);
                q[0] = blend(make_float2(__uint_as_float(A.x), __uint_as_float(A.y)),
                             make_float2(__uint_as_float(B.x), __uint_as_float(B.y)));
                q[S / 2 - 1] = blend(make_float2(__uint_as_float(A.z), __uint_as_float(A.w)),
                                     make_float2(__uint_as_float(B.z), __uint_as_float(B.w)));
              } else {
                q[0] = blend(lds_f32x2(at), lds_f32x2(at + CB));
              }
            };
            auto march = [&](auto shortc) {
              constexpr bool SHORT = decltype(shortc)::value;
              float2 lo[S / 2], hi[S / 2];
              uint32_t before = 0;  // bit pattern of the previous voxel's row
#pragma unroll
              for (int j = 0; j < NY; j += 2) {
                advance(j);
                const float2 t2 = fadd2_rz(v2, magic2);
                const float2 fv2 = fsub2(v2, fsub2(t2, magic2));
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                  const uint32_t bits = __float_as_uint(p ? t2.y : t2.x);
                  const uint32_t at = bits * RB + c0;
                  if (j + p == 0) {
                    load(at, lo);
                  } else {
                    const bool same = bits == before;
#pragma unroll
                    for (int i = 0; i < S / 2; ++i) {
                      lo[i].x = same ? lo[i].x : hi[i].x;
                      lo[i].y = same ? lo[i].y : hi[i].y;
                    }
                    if (!SHORT && bits - before > 1u) load(at, lo);
                  }
                  load(at + RB, hi);
                  add(lo, hi, p ? fv2.y : fv2.x, j + p);
                  before = bits;
                }
              }
            };
            if (flags & kQShort) march(std::true_type{});
            else march(std::false_type{});
          } else {
            // window not staged: read the elements from global memory (zero
            // outside the stored extent, as the TMA fill would give)
            const BPArgs& ja = job_args<MULTI>(a, qq, jb);
            const int col = g.u0 + iu;
            auto load = [&](int row, float2 (&q)[S / 2]) {
              const float2* p = reinterpret_cast<const float2*>(ja.qg) +
                                (((size_t)g.grp * ja.qg_rows + row) * ja.qg_pitch + col) * (S / 2);
              const bool in = row >= 0 && row < ja.qg_rows;
              const bool inA = in && col >= 0 && col < ja.qg_pitch, inB = in && col + 1 >= 0 && col + 1 < ja.qg_pitch;
#pragma unroll
              for (int i = 0; i < S / 2; ++i)
                q[i] = blend(inA ? __ldg(p + i) : make_float2(0.f, 0.f), inB ? __ldg(p + S / 2 + i) : make_float2(0.f, 0.f));
            };
#pragma unroll
            for (int j = 0; j < NY; ++j) {
              const float v = fmaf((float)j, dvv, vl);
              const float t = __fadd_rz(v, kMagic);
              const int row = g.e0 + (int)(__float_as_uint(t) - kMagicBits);
              float2 lo[S / 2], hi[S / 2];
              load(row, lo);
              load(row + 1, hi);
              add(lo, hi, v - (t - kMagic), j);
            }
          }
        } else if constexpr (P16) {
          // slots' (row v, row v + 1 minus row v): the u-lerp of both in FP32
          float Wr[S];
#pragma unroll
          for (int r = 0; r < S; ++r) Wr[r] = __fmul_rn(W, g.ws[r]);
          auto tap = [&](const uint32_t (&X)[S], const uint32_t (&Y)[S], float fv, int j) {
#pragma unroll
            for (int r = 0; r < S; ++r) {
              const float2 x = __half22float2(*reinterpret_cast<const __half2*>(&X[r]));
              const float2 y = __half22float2(*reinterpret_cast<const __half2*>(&Y[r]));
              const float2 ag = ffma2(make_float2(fu, fu), fsub2(y, x), x);
              acc[r][j] = fmaf(Wr[r], fmaf(fv, ag.y, ag.x), acc[r][j]);
            }
          };
          if (!(flags & kQDirect)) {
            auto load = [&](uint32_t at, uint32_t (&X)[S]) {
              if constexpr (S == 4) {
                const uint4 q = lds_u4(at);
                X[0] = q.x, X[1] = q.y, X[S - 2] = q.z, X[S - 1] = q.w;
              } else {
                const float2 q = lds_f32x2(at);
                X[0] = __float_as_uint(q.x), X[1] = __float_as_uint(q.y);
              }
            };
#pragma unroll
            for (int j = 0; j < NY; j += 2) {
              advance(j);
              const float2 t2 = fadd2_rz(v2, magic2);
              const float2 fv2 = fsub2(v2, fsub2(t2, magic2));
#pragma unroll
              for (int p = 0; p < 2; ++p) {
                const uint32_t at = __float_as_uint(p ? t2.y : t2.x) * RB + c0;
                uint32_t X[S], Y[S];
                load(at, X);
                load(at + CB, Y);
                tap(X, Y, p ? fv2.y : fv2.x, j + p);
              }
            }
          } else {
            const BPArgs& ja = job_args<MULTI>(a, qq, jb);
            const int col = g.u0 + iu;
#pragma unroll
            for (int j = 0; j < NY; ++j) {
              const float v = fmaf((float)j, dvv, vl);
              const float t = __fadd_rz(v, kMagic);
              const int row = g.e0 + (int)(__float_as_uint(t) - kMagicBits);
              const uint32_t* p = reinterpret_cast<const uint32_t*>(ja.qg) +
                                  (((size_t)g.grp * ja.qg_rows + row) * ja.qg_pitch + col) * S;
              const bool in = row >= 0 && row < ja.qg_rows;
              const bool inA = in && col >= 0 && col < ja.qg_pitch, inB = in && col + 1 >= 0 && col + 1 < ja.qg_pitch;
              uint32_t X[S], Y[S];
#pragma unroll
              for (int r = 0; r < S; ++r) X[r] = inA ? __ldg(p + r) : 0u, Y[r] = inB ? __ldg(p + S + r) : 0u;
              tap(X, Y, v - (t - kMagic), j);
            }
          }
        } else {
          const __half2 fu2 = __float2half2_rn(fu);
          float Wr[4];
#pragma unroll
          for (int r = 0; r < 4; ++r) Wr[r] = __fmul_rn(W, g.ws[r]);
          // (A, G) of the four slots at one voxel from the 16-byte planes of
          // its element: A = u-lerp of row e - 1, G = u-lerp of the row difference
          auto decode = [&](const uint4& L0, const uint4& L1, const uint4& L2, float (&A)[4], float (&G)[4]) {
            if constexpr (Q24) {
              const uint32_t wv[12] = {L0.x, L0.y, L0.z, L0.w, L1.x, L1.y, L1.z, L1.w, L2.x, L2.y, L2.z, L2.w};
              // (A, G) = (a, b - a) + fu (c' - a, d - c' - b + a) of slot SL
              auto slot = [&](auto slc) {
                constexpr int SL = decltype(slc)::value;
                const float2 ag = ffma2(make_float2(fu, fu), make_float2(dec24<4 * SL + 2>(wv), dec24<4 * SL + 3>(wv)),
                                        make_float2(dec24<4 * SL>(wv), dec24<4 * SL + 1>(wv)));
                A[SL] = ag.x;
                G[SL] = ag.y;
              };
              slot(std::integral_constant<int, 0>{});
              slot(std::integral_constant<int, 1>{});
              slot(std::integral_constant<int, 2>{});
              slot(std::integral_constant<int, 3>{});
            } else {
              const uint32_t wv[8] = {L0.x, L0.y, L0.z, L0.w, L1.x, L1.y, L1.z, L1.w};
#pragma unroll
              for (int sl = 0; sl < 4; ++sl) {
                const __half2 X1 = *reinterpret_cast<const __half2*>(&wv[2 * sl]);      // (a, b - a)
                const __half2 X2 = *reinterpret_cast<const __half2*>(&wv[2 * sl + 1]);  // (c' - a, d - c' - b + a)
                const float2 P = __half22float2(X1);
                A[sl] = fma_f16_f32(__low2half(fu2), __low2half(X2), P.x);
                G[sl] = fma_f16_f32(__low2half(fu2), __high2half(X2), P.y);
              }
            }
          };
          // slot pairs (0, 1), (2, 3) of one voxel: v-lerp and weighted sum as packed pairs
          auto slot_pairs = [&](const float (&A)[4], const float (&G)[4], float fv, int j) {
#pragma unroll
            for (int pr = 0; pr < 2; ++pr) {
              float& d0 = acc[2 * pr][j];
              float& d1 = acc[2 * pr + 1][j];
              const float2 t = ffma2(make_float2(fv, fv), make_float2(G[2 * pr], G[2 * pr + 1]),
                                     make_float2(A[2 * pr], A[2 * pr + 1]));
              const float2 d = ffma2(make_float2(Wr[2 * pr], Wr[2 * pr + 1]), t, make_float2(d0, d1));
              d0 = d.x;
              d1 = d.y;
            }
          };
          if (!(flags & kQDirect)) {
            const uint32_t plane = g.plane;
#pragma unroll
            for (int j = 0; j < NY; j += 2) {
              advance(j);
              const float2 t2 = fadd2_rz(v2, magic2);
              const float2 fv2 = fsub2(v2, fsub2(t2, magic2));
              const uint32_t a0 = __float_as_uint(t2.x) * RB + c0, a1 = __float_as_uint(t2.y) * RB + c0;
              // slots 0, 1 | slots 2, 3 (24-bit: the 48 bytes of the element)
              const uint4 z4 = make_uint4(0u, 0u, 0u, 0u);
              float A0[4], G0[4];
              decode(lds_u4(a0), lds_u4(a0 + plane), Q24 ? lds_u4(a0 + 2 * plane) : z4, A0, G0);
              slot_pairs(A0, G0, fv2.x, j);
              decode(lds_u4(a1), lds_u4(a1 + plane), Q24 ? lds_u4(a1 + 2 * plane) : z4, A0, G0);
              slot_pairs(A0, G0, fv2.y, j + 1);
            }
          } else {
            // window not staged: read the elements from global memory (zero
            // outside the stored extent, as the TMA fill would give)
            const BPArgs& ja = job_args<MULTI>(a, qq, jb);
            const int col = g.u0 + iu;
            const bool col_ok = col >= 0 && col < ja.qg_pitch;
            const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
            for (int j = 0; j < NY; ++j) {
              const float v = fmaf((float)j, dvv, vl);
              const float t = __fadd_rz(v, kMagic);
              const float fv = v - (t - kMagic);
              const int row = g.e0 + (int)(__float_as_uint(t) - kMagicBits);
              uint4 L0 = zero, L1 = zero, L2 = zero;
              if (col_ok && row >= 0 && row < ja.qg_rows) {
                const uint4* p = ja.qg + ((size_t)g.grp * ja.qg_rows + row) * NPL * ja.qg_pitch + col;
                L0 = __ldg(p);
                L1 = __ldg(p + ja.qg_pitch);
                if (Q24) L2 = __ldg(p + 2 * ja.qg_pitch);
              }
              float A[4], G[4];
              decode(L0, L1, L2, A, G);
              slot_pairs(A, G, fv, j);
            }
          }
        }
      } else {
        bad = true;
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[e]);
    if (++e == E) {
      e = 0;
      ph ^= 1;
    }
    if (FLAGGED) turned = (flags & kQTurn) != 0;
  };
  // the item's sums into its voxels: the rotated columns, (x, z) ->
  // (n-1-z, x) -> (n-1-x, n-1-z) -> (z, n-1-x), or (x, z) -> (n-1-x, n-1-z)
  auto store = [&]() {
    const BPArgs& ja = job_args<MULTI>(a, qq, jb);
    const ItemTile til = item_tile<TY>(ja, MULTI ? item - qq.jobs[jb].item0 + qq.jobs[jb].t0 : item);
    // a whole walk brings the sums back to the first view's slots, where
    // rotation r sits in slot r + its phase: move it to slot r
    for (int i = (S - til.k0 / ja.groups % S) % S; i > 0; --i) turn();
    // representative columns: four slots, x < n - h and z < h (h = n / 2) and
    // the centre of an odd size; two slots, z < h and an odd size's middle
    // row; columns that are their own image are rotation 0's alone
    const int n = ja.nx, h = n >> 1;
    const int ix = til.ix0 + tx, iz = til.iz0 + tz;
    const bool mid = EDGES && (n & 1) && iz == h && (S == 2 || ix == h);
    const bool own = !EDGES || ((S == 4 ? ix < n - h : ix < n) && (iz < h || mid));
    const int cx[4] = {ix, S == 4 ? n - 1 - iz : n - 1 - ix, n - 1 - ix, iz};
    const int cz[4] = {iz, S == 4 ? ix : n - 1 - iz, n - 1 - iz, n - 1 - ix};
    float* const vol = ja.vol;
    const int ystride = ja.vol_ystride, ny = ja.ny, ylim = ja.clip_ylimit;
    const float scale = ja.scale;
    float lo = __int_as_float(0x7f800000), hi = -lo;
#pragma unroll
    for (int r = 0; r < S; ++r) {
      if (!own || (mid && r > 0)) continue;
      float* out = vol + ((size_t)cz[r] * ystride) * n + cx[r];
#pragma unroll
      for (int j = 0; j < NY; ++j) {
        const int iy = til.iy0 + ty + j;
        if (iy < ny) {
          float val = acc[r][j] * scale;
          if (iy < ylim) val = fmaxf(val, 0.f);
          out[(size_t)iy * n] = val;
          lo = fminf(lo, val);
          hi = fmaxf(hi, val);
        }
      }
    }
    if (ja.minmax) fold_minmax(ja.minmax, lo, hi);
  };
  if constexpr (!MULTI) {
    // one work item, K quads (as many as views): a loop of known length
    item = (long long)blockIdx.y * gridDim.x + blockIdx.x;
    const int K = a.nviews;
    // the phases, the first one entered at its view k0 mod Q and finished at
    // the end (the turns stay out of the inner loop)
    const int Q = a.groups, k0 = item_tile<TY>(a, item).k0, first = Q - k0 % Q;
    int left = K;
    for (int n = first; left > 0 && !stop; n = min(Q, left)) {
      left -= n;
#pragma unroll 2
      for (int q = 0; q < n; ++q) { step(); if (stop) break; }
      if (FLAGGED ? turned : (k0 - left) % Q == 0) turn();
      if (EDGES && k0 == left)  // from the last phase back to the first
        for (int i = 0; i < a.wrap; ++i) turn();
    }
    if (bad) atomicCAS(a.err, 0, kDevFootprint);
    if (stop || *s_abort) return;
    store();
    return;
  }
  for (;;) {
    do step();
    while (!(stop || leave || turned || last));
    if (stop || leave) break;
    if (turned) turn();
    if (last) {
      if (bad) atomicCAS(job_args<MULTI>(a, qq, jb).err, 0, kDevFootprint);
      bad = false;
      if (*s_abort) break;
      store();
      reset();
      last = false;
    }
  }
  if (bad) atomicCAS(err, 0, kDevFootprint);
}

// Footprint pre-pass: one warp per tile (lanes over views) finds the
// largest window any (tile, view) needs; same FP64 code as the
// backprojector's producer, so the largest box always fits. With `hist`, it
// also counts the windows by (width, height), clamped to kBoxHist - 1, in a
// shared-memory histogram (kBoxHist^2 counters) added to `hist` at the end.
template <int TX, int TZ, int NY>
__global__ void footprint_kernel(BPArgs a, int nty, int* spans, unsigned* hist) {
  extern __shared__ unsigned sh_hist[];
  if (hist)
    for (int i = threadIdx.x; i < kBoxHist * kBoxHist; i += blockDim.x) sh_hist[i] = 0u;
  __syncthreads();
  const long long ntiles = (long long)a.ntx * a.ntz * nty;
  const int lane = threadIdx.x & 31;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  int gu = 0, gv = 0;
  for (long long T = blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5); T < ntiles; T += warps) {
    const int by = (int)(T / ((long long)a.ntx * a.ntz));
    const int rr = (int)(T - (long long)by * a.ntx * a.ntz);
    const int bz = rr / a.ntx, bx = rr - bz * a.ntx;
    const int ix0 = bx * TX, iz0 = bz * TZ, iy0 = by * NY;
    for (int k = lane; k < a.nviews; k += 32) {
      TileGeo g;
      // full tile extents, as the backprojector's producer uses them
      tile_geo(a, k, ix0, iy0, iz0, TX - 1, NY - 1, TZ - 1, g);
      if (g.dmin <= 1e-6) atomicCAS(a.err, 0, kDevGeometry);
      if (tile_skip(a, g)) continue;
      int u0, v0, nu_, nv_;
      tile_window(a, g, u0, v0, nu_, nv_);
      gu = max(gu, nu_);
      gv = max(gv, nv_);
      if (hist)
        atomicAdd(&sh_hist[min(max(nu_, 0), kBoxHist - 1) * kBoxHist + min(max(nv_, 0), kBoxHist - 1)], 1u);
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    gu = max(gu, __shfl_xor_sync(0xffffffffu, gu, o));
    gv = max(gv, __shfl_xor_sync(0xffffffffu, gv, o));
  }
  if (lane == 0) {
    atomicMax(spans, gu);
    atomicMax(spans + 1, gv);
  }
  __syncthreads();
  if (hist)
    for (int i = threadIdx.x; i < kBoxHist * kBoxHist; i += blockDim.x)
      if (sh_hist[i]) atomicAdd(&hist[i], sh_hist[i]);
}

__global__ void clip_kernel(float* vol, int nx, int ny, int nz, int ylim) {
  const long long total = (long long)nx * ny * nz;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    long long iy = (e / nx) % ny;
    if (iy < ylim) vol[e] = fmaxf(vol[e], 0.f);
  }
}

// Fan (flat detector) -> parallel rebinning; see the C ABI comment.
__global__ void rebin_fan_kernel(const float* fan, int bins, int views, double sod, double sdd, double du,
                                 double span, double offset, float* par, int out_bins, double du_out) {
  const long long total = (long long)views * out_bins;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    int k = (int)(e / out_bins), j = (int)(e % out_bins);
    double th = offset + span * k / views;
    double s = (j + 0.5 - out_bins / 2.0) * du_out;
    float val = 0.f;
    if (fabs(s) < sod) {
      double gam = asin(s / sod);
      double beta = th - gam;
      double ui = sdd * tan(gam) / du + bins / 2.0 - 0.5;
      double bi = (beta - offset) / (span / views);
      double bf = floor(bi), ab = bi - bf;
      long long b0 = (long long)bf;
      double fu = floor(ui), au = ui - fu;
      long long iu = (long long)fu;
      double acc = 0.0;
      for (int t = 0; t < 2; ++t) {
        long long bb = (((b0 + t) % views) + views) % views;
        const float* row = fan + bb * bins;
        double p0 = (iu >= 0 && iu < bins) ? row[iu] : 0.0;
        double p1 = (iu + 1 >= 0 && iu + 1 < bins) ? row[iu + 1] : 0.0;
        double r = p0 * (1 - au) + p1 * au;
        acc += t ? r * ab : r * (1 - ab);
      }
      val = (float)acc;
    }
    par[e] = val;
  }
}

template <int LAYOUT, int TX, int TZ, int NY>
cudaError_t launch_cfg(const BoxMaps& maps, const BPArgs& a, size_t smem, cudaStream_t stream) {
  auto kern = bp_kernel<LAYOUT, TX, TZ, NY>;
  // The attribute is process-wide: contexts on other threads launch this kernel
  // with other sizes, so it is always raised to the device maximum (a launch
  // still uses only its own dynamic size).
  (void)smem;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynamicSmem);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return e;
  dim3 grid(a.ntx * a.ntz, (a.ny + NY - 1) / NY);
  kern<<<grid, TX * TZ + 32, smem, stream>>>(maps, a);
  return cudaGetLastError();
}

template <int LAYOUT, int NY, int YW, int OCC, bool EDGES>
cudaError_t launch_quad_cfg(const BoxMaps& maps, const BPArgs& a, size_t smem, cudaStream_t stream) {
  auto kern = bp_quad_kernel<LAYOUT, NY, YW, OCC, false, EDGES>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynamicSmem);
  if (e != cudaSuccess) return e;
  // all of L1 as shared memory, so that two CTAs of up to 113 KB share an SM
  e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return e;
  dim3 grid(a.nbx * a.nbz, (a.ny + NY * YW - 1) / (NY * YW));
  kern<<<grid, quad_threads(LAYOUT, NY, YW), smem, stream>>>(maps, a, QuadQueue{});
  return cudaGetLastError();
}

// The kernel shape of a staged layout and tile height (quad_tile_ny's values).
#define FBP_SYMMETRIC_SHAPES(LAUNCH)                                                         \
  case kLayoutQuadG16:                                                                       \
    return ny_tile == 8    ? LAUNCH(kLayoutQuadG16, 8, 1, 2)                                 \
           : ny_tile == 16 ? LAUNCH(kLayoutQuadG16, 8, 2, 1)                                 \
                           : LAUNCH(kLayoutQuadG16, 12, 2, 1);                               \
  case kLayoutQuadG24:                                                                       \
    return ny_tile == 8    ? LAUNCH(kLayoutQuadG24, 8, 1, 2)                                 \
           : ny_tile == 12 ? LAUNCH(kLayoutQuadG24, 12, 1, 2)                                \
                           : LAUNCH(kLayoutQuadG24, 16, 1, 1);                               \
  default:                                                                                   \
    return ny_tile == 8    ? LAUNCH(kLayoutQuad32, 8, 1, 2)                                  \
           : ny_tile == 12 ? LAUNCH(kLayoutQuad32, 12, 1, 2)                                 \
                           : LAUNCH(kLayoutQuad32, 16, 1, 1);

cudaError_t launch_quad(int layout, int ny_tile, const BoxMaps& maps, const BPArgs& a, size_t smem,
                        cudaStream_t stream) {
#define FBP_LAUNCH(L, NY, YW, OCC) launch_quad_cfg<L, NY, YW, OCC, false>(maps, a, smem, stream)
#define FBP_EDGES(L, NY, YW, OCC) launch_quad_cfg<L, NY, YW, OCC, true>(maps, a, smem, stream)
  if (layout == kLayoutDuo32) return FBP_EDGES(kLayoutDuo32, 16, 1, 2);
  if (layout == kLayoutQuadP16) return FBP_EDGES(kLayoutQuadP16, 8, 1, 2);
  if (layout == kLayoutDuoP16) return FBP_EDGES(kLayoutDuoP16, 16, 1, 2);
  if (layout == kLayoutQuad32 && (a.nx % 32 || a.wrap))
    return ny_tile == 12 ? FBP_EDGES(kLayoutQuad32, 12, 1, 2) : FBP_EDGES(kLayoutQuad32, 8, 1, 2);
  switch (layout) { FBP_SYMMETRIC_SHAPES(FBP_LAUNCH) }
#undef FBP_EDGES
#undef FBP_LAUNCH
}

int quad_occ(int layout, int ny_tile) {
  return ny_tile == 8 || ny_tile == 12 || layout == kLayoutDuo32 || layout == kLayoutDuoP16 ? 2 : 1;
}

// Tile height of a symmetric backprojection: the caller's (8 or 16), or the one
// with the least time by a fit to volumes of 96^3 to 384^3 (ms for 360 views;
// shapes with two CTAs a SM against the waves of tiles W = tiles / (2 SMs),
// those with one against the tiles on the fullest SM). At 96^3, 128^3, 192^3,
// 384^3: MIXED 8 high 0.29, 0.45, 1.18, 8.1; 16 high 0.42, 0.44, 1.16, 8.1; 24
// high 0.56, 0.59, 1.11, 7.6. FP32 and 24-bit take 12 from 36 waves on
// (about 440^3): 8 and 12 high 0.31 and 0.47, 0.50 and 0.77, 1.40 and 1.48, 9.8
// and 10.1 at those sizes, then 18.8 and 17.3 at 480 x 490 x 480 (480 views),
// 38.1 and 37.4 at 512^3 (720 views; 24-bit 46.8 and 44.7); and where it makes
// one wave of more than 1.2 (160 x 128 x 160: 0.87 and 0.72, 24-bit 0.90 and
// 0.86; 128 x 153 x 128, 1.08 waves, 0.59 and 0.81).
int quad_tile_height(int asked, int layout, int orbits, int ny, int num_sms) {
  if (asked) return asked;
  if (layout == kLayoutDuo32 || layout == kLayoutDuoP16) return 16;
  if (layout == kLayoutQuadP16) return 8;
  auto tiles = [&](int h) { return (long long)orbits * ((ny + h - 1) / h); };
  auto waves = [&](int h) { return (double)tiles(h) / (2.0 * num_sms); };
  auto fullest = [&](int h) { return (double)((tiles(h) + num_sms - 1) / num_sms); };
  if (layout == kLayoutQuadG16) {
    const double c8 = 0.345 * (std::max(0.5, waves(8)) + 0.45);
    const double c16 = 0.36 * (fullest(16) + 0.15), c24 = 0.47 * (fullest(24) + 0.2);
    return c8 < c16 && c8 < c24 ? 8 : c16 < c24 ? 16 : 24;
  }
  return waves(8) >= 36.0 || (waves(8) > 1.2 && waves(12) <= 1.0) ? 12 : 8;
}

template <int TX, int TZ, int NY>
cudaError_t launch_layout(int layout, const BoxMaps& maps, const BPArgs& a, size_t smem, cudaStream_t stream) {
  switch (layout) {
    case kLayoutPair16:
      return launch_cfg<kLayoutPair16, TX, TZ, NY>(maps, a, smem, stream);
    default:
      return launch_cfg<kLayoutRaw32, TX, TZ, NY>(maps, a, smem, stream);
  }
}

}  // namespace

// A box width whose shared-memory row stride (planes x width sixteen-byte
// units) is 3, 4 or 5 mod 8.
static bool bank_friendly(int planes, int w) {
  const int r = (planes * w) % 8;
  return r >= 3 && r <= 5;
}

// Per-view (cos, sin) of theta_k = offset + span k / K in FP64, computed on
// the device (no host staging, so a new view set needs no stream sync) and
// kept while the view set stays the same.
__global__ void trig_kernel(double2* trig, int n, double offset, double span) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  double sn, cs;
  sincos(offset + span * k / n, &sn, &cs);
  trig[k] = make_double2(cs, sn);
}

int ensure_trig(fbp_context* ctx, const BPGeom& g) {
  if (ctx->trig_cap < g.nviews) {
    cudaFree(ctx->d_trig);
    ctx->d_trig = nullptr;
    ctx->trig_cap = 0;
    ctx->trig_key[0] = -1;
    if (cuda_check(ctx, cudaMalloc(&ctx->d_trig, sizeof(double2) * g.nviews), "cudaMalloc(trig)"))
      return FBP_ERR_OUT_OF_MEMORY;
    ctx->trig_cap = g.nviews;
  }
  if (ctx->trig_key[0] == g.nviews && ctx->trig_key[1] == g.span && ctx->trig_key[2] == g.offset) return FBP_OK;
  trig_kernel<<<(g.nviews + 127) / 128, 128, 0, ctx->stream>>>(ctx->d_trig, g.nviews,
                                                                g.offset, g.span);
  if (int rc = launched(ctx, "trig_kernel")) return rc;
  ctx->trig_key[0] = g.nviews;
  ctx->trig_key[1] = g.span;
  ctx->trig_key[2] = g.offset;
  return FBP_OK;
}

// Thresholds t_0 < ... < t_{n-1} = the last candidate, taken from `cand`
// (ascending), minimising sum_v weight[v] * (smallest t_i >= v) over the
// values v = 0 .. weight.size() - 1 (weights of values above the last
// candidate are ignored): dynamic program over the candidates. Fewer
// candidates than n repeat the last threshold.
static void best_thresholds(const std::vector<double>& weight, const std::vector<int>& cand, int n, int* out) {
  const int C = (int)cand.size();
  // W[j] = total weight of the values <= cand[j]
  std::vector<double> W(C, 0.0);
  for (int j = 0; j < C; ++j) {
    double acc = 0.0;
    for (int v = 0; v < (int)weight.size() && v <= cand[j]; ++v) acc += weight[v];
    W[j] = acc;
  }
  const double inf = 1e300;
  std::vector<double> dp((size_t)(n + 1) * C, inf);
  std::vector<int> from((size_t)(n + 1) * C, -1);
  for (int j = 0; j < C; ++j) dp[(size_t)1 * C + j] = cand[j] * W[j];
  for (int m = 2; m <= n; ++m)
    for (int j = 0; j < C; ++j)
      for (int i = 0; i < j; ++i) {
        const double c = dp[(size_t)(m - 1) * C + i] + cand[j] * (W[j] - W[i]);
        if (c < dp[(size_t)m * C + j]) {
          dp[(size_t)m * C + j] = c;
          from[(size_t)m * C + j] = i;
        }
      }
  // the most thresholds that the candidates allow, ending at the last one
  int m = std::min(n, C);
  int j = C - 1;
  std::vector<int> t;
  for (; m >= 1 && j >= 0; --m) {
    t.push_back(cand[j]);
    j = from[(size_t)m * C + j];
  }
  std::sort(t.begin(), t.end());
  for (int i = 0; i < n; ++i) out[i] = t[std::min(i, (int)t.size() - 1)];
}

// The backprojector's box grid for one plan: kBoxGrid widths (multiples of
// align, the largest = mbu) and kBoxGrid heights (the largest = mbv) that
// minimise the staged window area summed over the footprint histogram, by
// alternating the width and the height programs (each exact for the other
// fixed). Windows larger than the largest box are left out (they take the
// direct path or fail the footprint check). Without a histogram: a linear
// grid, each of the quarters 1/4 .. 4/4 of the largest window in each
// dimension taken twice.
static void choose_boxes(const std::vector<unsigned>& hist, int mbu, int mbv, int align, int pair_rows, int planes,
                         int* w, int* h) {
  const int n = kBoxGrid, B = kBoxHist;
  for (int i = 0; i < n; ++i) {
    const int quarter = i / 2 + 1;
    const int wi = (mbu * quarter + 3) / 4;
    w[i] = std::max(align, (wi + align - 1) / align * align);
    h[i] = std::max(1, (mbv * quarter + 3) / 4);
  }
  w[n - 1] = mbu;
  h[n - 1] = mbv;
  if ((int)hist.size() != B * B) return;
  // counts over (width rounded up to align, rows staged)
  const int U = std::max(mbu, 1) + 1, V = std::max(mbv, 1) + 1;
  std::vector<double> cnt((size_t)U * V, 0.0);
  double total = 0.0;
  for (int nu = 0; nu < B; ++nu)
    for (int nv = 0; nv < B; ++nv) {
      const unsigned c = hist[(size_t)nu * B + nv];
      if (!c) continue;
      const int u = std::max(align, (nu + align - 1) / align * align);
      const int r = std::max(1, nv - pair_rows);
      if (u > mbu || r > mbv) continue;
      cnt[(size_t)u * V + r] += c;
      total += c;
    }
  if (total <= 0.0) return;
  // widths: multiples of align; with planes > 0 (interleaved layouts, 16-byte
  // planes) only those whose row stride is 3 to 5 mod 8 sixteen-byte units,
  // so that the quarter-warp's two voxel rows (same detector column, next
  // element row) fall in different bank groups (a simulation of the C4
  // access pattern: 1.22 wavefronts per 16-byte load phase at 4 mod 8, 1.23
  // at 3 or 5, against 1.31 at 2 or 6 and 1.44 at 0)
  std::vector<int> cu, cv;
  for (int u = align; u <= mbu; u += align)
    if (planes <= 0 || bank_friendly(planes, u)) cu.push_back(u);
  if (cu.empty() || cu.back() != mbu) cu.push_back(mbu);
  for (int r = 1; r <= mbv; ++r) cv.push_back(r);
  auto pick = [](const int* t, int n, int x) {
    for (int i = 0; i < n; ++i)
      if (t[i] >= x) return t[i];
    return t[n - 1];
  };
  for (int it = 0; it < 3; ++it) {
    std::vector<double> wu(U, 0.0), wv(V, 0.0);
    for (int u = 0; u < U; ++u)
      for (int r = 0; r < V; ++r) {
        const double c = cnt[(size_t)u * V + r];
        if (c) wu[u] += c * pick(h, n, r);
      }
    best_thresholds(wu, cu, n, w);
    for (int u = 0; u < U; ++u)
      for (int r = 0; r < V; ++r) {
        const double c = cnt[(size_t)u * V + r];
        if (c) wv[r] += c * pick(w, n, u);
      }
    best_thresholds(wv, cv, n, h);
  }
}

// The orbits of a view set; four slots only where the volume is square.
static Orbits find_orbits(bool cone, double turns, int K, bool square) {
  const long long whole = llround(turns), halves = llround(2.0 * turns);
  const bool full_turn = fabs(turns - (double)whole) < 1e-9;
  const bool half_turn = !full_turn && fabs(2.0 * turns - (double)halves) < 1e-9;  // an odd number of halves
  if (square && full_turn && whole % 4 == 1 && K % 4 == 0) return {4, K / 4, 4, 4};
  if (square && !cone && half_turn && halves % 4 == 1 && K % 2 == 0) return {4, K / 2, 2, 2};
  if (full_turn && (whole % 2 == 1 || whole % 2 == -1) && K % 2 == 0) return {2, K / 2, 2, 2};
  if (!cone) return {2, K, 1, 1};
  return {1, K, 1, 1};
}

// Whether a volume off the symmetric kernel runs on rotational orbits, and on
// which: the least of (tiles on the fullest SM + 0.4) x the cost of a tile,
// with the costs measured in units of the plain kernel's 16 x 16 x 16 tile
// (300 x 251 x 300, 450 to 452 views; 256^3 parallel; the 0.4 is what a SM's
// last tiles lose by running alone, 100 x 80 x 100). FP32: four slots 1.13 (8
// high) or 1.76 (12 high), two slots 1.42; FP16 pairs: 1.36 and 1.44.
static bool choose_orbits(const BPGeom& g, int ny, double turns, bool p16, int num_sms, Orbits* orb) {
  const bool cone = g.kind == FBP_GEOMETRY_CONE;
  const int t16 = (g.nx + 15) / 16, half = ((g.nx + 1) / 2 + 15) / 16;
  auto cost = [&](long long columns, int height, double rel) {
    const long long tiles = columns * ((ny + height - 1) / height);
    return rel * ((double)((tiles + num_sms - 1) / num_sms) + 0.4);
  };
  double best = cost((long long)t16 * t16, 16, 1.0);
  bool any = false;
  const Orbits four = find_orbits(cone, turns, g.nviews, true), two = find_orbits(cone, turns, g.nviews, false);
  if (four.slots == 4) {
    const double c = p16 ? cost((long long)half * half, 8, 1.36)
                         : std::min(cost((long long)half * half, 8, 1.13), cost((long long)half * half, 12, 1.76));
    if (c < best) best = c, *orb = four, any = true;
  }
  if (two.slots == 2 && cost((long long)t16 * half, 16, p16 ? 1.44 : 1.42) < best) *orb = two, any = true;
  if (!any) *orb = Orbits{1, g.nviews, 1, 1};
  return any;
}

// A planned backprojection: everything a launch needs (arguments, tensor
// maps, shared memory) after the footprint pass and the packing.
struct BPLaunchPlan {
  BPArgs a;
  BoxMaps maps;
  size_t smem = 0;
  int layout = 0, ny_tile = 0, occ = 2;
  bool use_quad = false;
  bool orbit = false;  // the quad kernel on an orbit of the generic backprojector's geometries
};

BPLaunchPlan* new_bp_plan() { return new BPLaunchPlan(); }
void free_bp_plan(BPLaunchPlan* p) { delete p; }

int plan_backproject(fbp_context* ctx, const BPGeom& g, Stack& st, float* vol, int clip_ylimit, bool mixed,
                     BPLaunchPlan* plan_out, const PlanLimits& lim) {
  const double pi = 3.14159265358979323846;
  // MIXED24: 24-bit views for the symmetric kernel (FP32 rows otherwise)
  const bool c24 = mixed && ctx->precision == FBP_PRECISION_MIXED24;
  // Four-fold symmetric path: square volume, views over one turn (or
  // 4m + 1 turns) with K % 4 == 0, an even number of 16-wide tiles per axis.
  const bool is2d = g.ny == 1;
  const double turns = g.span / (2.0 * pi);
  const long long iturns = llround(turns);
  const bool symmetric = !is2d && g.nx == g.nz && g.nx % 32 == 0 && g.nviews % 4 == 0 &&
                         fabs(turns - (double)iturns) < 1e-9 && iturns % 4 == 1;
  const bool quad = symmetric && lim.symmetric &&
                    (ctx->bp_variant == FBP_BACKPROJECTOR_AUTO || ctx->bp_variant == FBP_BACKPROJECTOR_SYMMETRIC);
  if (ctx->bp_variant == FBP_BACKPROJECTOR_SYMMETRIC && !symmetric)
    return set_error(ctx, FBP_ERR_UNSUPPORTED,
                     "the four-fold symmetric backprojector needs nx == nz (a multiple of 32), views % 4 == 0 and "
                     "views over one full turn");
  // Square volumes off those sizes that still have rotational orbits (half
  // turns, parallel beam) run on the same kernel, four or two voxels to a tap
  // position, where that is faster; an explicit view ring is the plain kernel's.
  const bool p16 = mixed && !c24;
  Orbits orb = find_orbits(g.kind == FBP_GEOMETRY_CONE, turns, g.nviews, g.nx == g.nz);
  const int rule_ny = g.rule_ny > 0 ? g.rule_ny : g.ny;
  const bool tuned_orbits = ctx->bp_variant == FBP_BACKPROJECTOR_ORBITS;  // the tuner's shape, never a caller's
  const bool orbit = !quad && !is2d && lim.orbits && g.nx == g.nz && ctx->bp_stages == 0 &&
                     (ctx->bp_variant == FBP_BACKPROJECTOR_AUTO || (tuned_orbits && !symmetric)) &&
                     choose_orbits(g, rule_ny, turns, p16, ctx->num_sms, &orb);
  if (tuned_orbits && lim.orbits && !orbit)
    return set_error(ctx, FBP_ERR_UNSUPPORTED, "rotational orbits are not this volume's faster form");
  // what the selected kernel reads: interleaved views (symmetric, orbits), FP16
  // pairs (MIXED) or the FP32 rows themselves
  const bool packed = quad || orbit || p16;
  const int layout = quad    ? (!mixed ? kLayoutQuad32 : c24 ? kLayoutQuadG24 : kLayoutQuadG16)
                     : orbit ? (orb.slots == 4 ? (p16 ? kLayoutQuadP16 : kLayoutQuad32) : p16 ? kLayoutDuoP16 : kLayoutDuo32)
                     : p16   ? kLayoutPair16
                             : kLayoutRaw32;
  const int esize = Stack::elem_bytes(layout);
  BPArgs a{};
  a.vol = vol;
  a.nx = g.nx;
  a.ny = g.ny;
  a.nz = g.nz;
  a.nu = g.nu;
  a.nv = g.nv;
  a.nviews = g.nviews;
  a.kind = g.kind;
  a.sod = g.sod;
  a.sdd = g.sdd;
  a.du = g.du;
  a.dv = g.dv;
  a.vox = g.vox;
  a.cu = 0.5 * g.nu - 0.5;
  // row band of a taller detector / y-slab of a taller volume (sharding)
  a.cv = 0.5 * (g.nv_total > 0 ? g.nv_total : g.nv) - 0.5 - g.row_off;
  a.y_off = g.y_off;
  a.vol_ystride = g.vol_ystride > 0 ? g.vol_ystride : g.ny;
  a.ny_total = g.ny_total > 0 ? g.ny_total : g.ny;
  if (g.kind == FBP_GEOMETRY_CONE) {
    a.dvn = (float)(g.sdd / (g.sod * g.dv) * g.vox);
    a.scale = (float)(pi / g.nviews * g.sdd / (g.sod * g.du));
  } else {
    a.dvn = (float)(g.vox / g.dv);
    a.scale = (float)(pi / g.nviews / g.du);
  }
  a.groups = orb.groups;
  a.mirror = orb.mirror;
  a.wrap = (orb.slots - orb.phases) % orb.slots;
  const int half = ((g.nx + 1) / 2 + 15) / 16;
  a.nbx = orb.slots == 4 ? half : (g.nx + 15) / 16;
  a.nbz = orb.slots == 1 ? (g.nx + 15) / 16 : half;
  // TMA: x * element size must be a multiple of 16 bytes (the interleaved
  // layouts' x counts 8-byte words, two per 16-byte plane element: always even)
  a.align = !is_quad_layout(layout) ? 4 : esize == 8 ? 2 : 1;
  a.sino_layout = st.sinogram ? 1 : 0;
  a.pair_rows = is_pair_layout(layout) ? 1 : 0;
  a.clip_ylimit = clip_ylimit;
  a.err = ctx->d_err;

  // per-view trig in FP64 (cached per view set)
  if (int rc = ensure_trig(ctx, g)) return rc;
  a.trig = ctx->d_trig;

  // tile configuration: 16 x 16 columns, NY voxels along y (1 for 2D)
  const int TX = 16, TZ = 16;
  const int NY = is2d    ? 1
                 : quad  ? quad_tile_height(ctx->quad_tile_ny, layout, a.nbx * a.nbz, rule_ny, ctx->num_sms)
                 : orbit ? quad_tile_height(0, layout, a.nbx * a.nbz, rule_ny, ctx->num_sms)
                         : std::min(lim.max_height, ctx->bp_variant == FBP_BACKPROJECTOR_GENERIC_Y8 ? 8 : 16);
  a.ntx = (g.nx + TX - 1) / TX;
  a.ntz = (g.nz + TZ - 1) / TZ;
  const int nty = (g.ny + NY - 1) / NY;

  // footprint pre-pass (cached per geometry and layout)
  double key[20] = {(double)g.kind, g.sod, g.sdd, g.du, g.dv, g.vox, g.span, g.offset, (double)g.nu,
                    (double)g.nv, (double)g.nviews, (double)g.nx, (double)g.ny, (double)g.nz,
                    (double)a.align, (double)NY, (double)g.row_off, (double)g.nv_total, (double)g.y_off,
                    (double)g.ny_total};
  fbp_context::BPPlan* found = nullptr;
  for (auto& p : ctx->plans) {
    bool same = p.valid;
    for (int i = 0; i < 20 && same; ++i) same = p.key[i] == key[i];
    if (same) {
      found = &p;
      break;
    }
  }
  // a plan made without the histogram (not a symmetric candidate then) is
  // redone in place when the symmetric kernel may now run
  const bool redo = found && (quad || orbit) && found->hist.empty();
  const bool hit = found != nullptr && !redo;
  fbp_context::BPPlan& plan = found ? *found : ctx->plans[ctx->plan_next];
  if (!hit) {
    if (!found) ctx->plan_next = (ctx->plan_next + 1) % (int)(sizeof(ctx->plans) / sizeof(ctx->plans[0]));
    plan.valid = false;
    // 4 span words, then the (width, height) histogram
    constexpr int kSpanWords = 4 + kBoxHist * kBoxHist;
    if (ctx->span_cap < kSpanWords) {
      cudaFree(ctx->d_span);
      ctx->d_span = nullptr;
      ctx->span_cap = 0;
      if (cuda_check(ctx, cudaMalloc(&ctx->d_span, sizeof(int) * kSpanWords), "cudaMalloc(footprint spans)"))
        return FBP_ERR_OUT_OF_MEMORY;
      ctx->span_cap = kSpanWords;
    }
    // the window histogram only for the symmetric kernel (its interleaved
    // layouts fit their boxes to it); the other plans take quarter steps
    unsigned* d_hist = quad || orbit ? reinterpret_cast<unsigned*>(ctx->d_span + 4) : nullptr;
    cudaMemsetAsync(ctx->d_span, 0, (d_hist ? kSpanWords : 4) * sizeof(int), ctx->stream);
    const long long ntiles = (long long)a.ntx * a.ntz * nty;
    // few blocks: each adds its whole shared histogram to the global one
    const int blocks = (int)std::max(1LL, std::min<long long>((ntiles + 7) / 8, (long long)ctx->num_sms * 2));
    const size_t hist_smem = sizeof(unsigned) * kBoxHist * kBoxHist;
    auto fk = NY == 1    ? footprint_kernel<16, 16, 1>
              : NY == 8  ? footprint_kernel<16, 16, 8>
              : NY == 12 ? footprint_kernel<16, 16, 12>
              : NY == 16 ? footprint_kernel<16, 16, 16>
                         : footprint_kernel<16, 16, 24>;
    if (cuda_check(ctx, cudaFuncSetAttribute(fk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)hist_smem),
                   "footprint_kernel shared memory"))
      return FBP_ERR_CUDA;
    fk<<<blocks, 256, hist_smem, ctx->stream>>>(a, nty, ctx->d_span, d_hist);
    if (int rc = launched(ctx, "footprint_kernel")) return rc;
    const int words = d_hist ? kSpanWords : 4;
    std::vector<int> hs(words);
    if (cuda_check(ctx, cudaMemcpyAsync(hs.data(), ctx->d_span, sizeof(int) * words, cudaMemcpyDeviceToHost,
                                        ctx->stream),
                   "spans") ||
        cuda_check(ctx, cudaStreamSynchronize(ctx->stream), "footprint sync"))
      return FBP_ERR_CUDA;
    plan.box_u = std::max(hs[0], 2);
    plan.box_v = std::max(hs[1], 2);
    if (d_hist)
      plan.hist.assign(reinterpret_cast<const unsigned*>(hs.data() + 4),
                       reinterpret_cast<const unsigned*>(hs.data() + kSpanWords));
    else
      plan.hist.clear();
    plan.sel_layout = -1;
    plan.valid = true;
    for (int i = 0; i < 20; ++i) plan.key[i] = key[i];
  }
  const int bu = (plan.box_u + a.align - 1) / a.align * a.align;
  // a pair element carries row v + 1 with it: one row less to stage
  const int bv = a.pair_rows ? std::max(1, plan.box_v - 1) : plan.box_v;
  // Limits of the FP32 form: windows of filtered rows up to 128 x 257 samples,
  // of other rows up to 256 x 256 (what a staged box of them holds), the
  // symmetric kernel's four together at most the ring
  const bool fp32 = layout == kLayoutRaw32 || layout == kLayoutQuad32 || layout == kLayoutDuo32;
  const int fu = st.filtered ? (plan.box_u + 1) / 2 * 2 : (plan.box_u + 3) / 4 * 4;
  const int fv = st.filtered ? std::max(1, plan.box_v - 1) : plan.box_v;
  if ((fp32 && ((st.filtered ? 2 * fu : fu) > 256 || fv > 256)) ||
      (is_p16_layout(layout) && ((plan.box_u + 3) / 4 * 4 > 256 || bv > 256)))
    return set_error(ctx, FBP_ERR_UNSUPPORTED,
                     "detector footprint of a voxel tile exceeds the 256-element TMA box; geometry magnification "
                     "too large for the staged backprojector");
  // A box holds 256 rows. FP32 rows take one more than the pairs of rows that
  // the limit above is about (parallel beam, 17 detector rows a voxel: 257 for
  // 16 voxels): lower tiles, down to one slice.
  if (layout == kLayoutRaw32 && bv > 256 && NY > 1)
    return plan_backproject(ctx, g, st, vol, clip_ylimit, mixed, plan_out, PlanLimits{false, false, NY > 8 ? 8 : 1});
  a.box_u = bu;
  a.box_v = bv;
  // two CTAs per SM: each gets half of the 228 KB shared memory
  const int occ = quad || orbit ? quad_occ(layout, NY) : 2;
  const size_t smem_cap = occ == 1 ? (size_t)kMaxDynamicSmem : 113 * 1024;
  const size_t max_box = (size_t)(bu * bv * esize + 127) / 128 * 128;
  size_t smem = 0;
  bool use_quad = quad || orbit;
  if (orbit) {
    // Windows of a size at which two in half an SM (the plain kernel's least
    // ring; rows, or pairs of filtered FP32 rows) are in doubt, by these tiles'
    // windows taken to 16 voxels: the plain kernel, whose own windows decide.
    // They are smaller than that where the rows spread with the distance too.
    const int rows16 = ((p16 ? bv : fv) - 2) * 16 / NY + 2;
    const size_t box = ((size_t)(p16 ? (plan.box_u + 3) / 4 * 4 : fu) * rows16 * (fp32 && st.filtered ? 8 : 4) + 127) / 128 * 128;
    if ((113 * 1024 - 64) / (box + sizeof(ViewCoef) + 2 * sizeof(uint64_t)) < 2)
      return plan_backproject(ctx, g, st, vol, clip_ylimit, mixed, plan_out, PlanLimits{false, false});
  }
  if (use_quad) {
    // byte ring for the windows + entry records
    const size_t fixed = kQuadEntries * (sizeof(QuadCoef) + 2 * sizeof(uint64_t) + sizeof(long long)) +
                         2 * kGeoQuads * sizeof(QuadStage) + 64;
    const size_t ring = (smem_cap - fixed) / 128 * 128;
    // Windows that do not fit are gathered from global memory; the FP32 form
    // keeps to the generic kernel where four separate windows of its rows
    // (pairs of rows when filtered) would not fit an SM (half, tile height 8)
    const size_t entry = fp32 ? 4 * (((size_t)fu * fv * (st.filtered ? 8 : 4) + 127) / 128 * 128) : 0;
    const size_t limit = ((ctx->quad_tile_ny == 8 ? 113 * 1024 : (size_t)kMaxDynamicSmem) - 1024) / 128 * 128;
    if (quad && entry > limit) {
      use_quad = false;  // the largest quad does not fit: generic path
      if (ctx->bp_variant == FBP_BACKPROJECTOR_SYMMETRIC)
        return set_error(ctx, FBP_ERR_UNSUPPORTED, "detector windows too large for the symmetric backprojector");
    } else {
      a.box_bytes = (int)ring;
      smem = ring + fixed;
    }
  }
  if (!use_quad) {
    if (quad) return plan_backproject(ctx, g, st, vol, clip_ylimit, mixed, plan_out, PlanLimits{false, lim.orbits});
    a.box_bytes = (int)max_box;
    const size_t per_stage = a.box_bytes + sizeof(ViewCoef) + 2 * sizeof(uint64_t);
    int stages = (int)std::min<size_t>(kMaxStages, (smem_cap - 64) / per_stage);
    if (ctx->bp_stages > 0) stages = std::min(stages, ctx->bp_stages);
    if (stages < 2)
      return set_error(ctx, FBP_ERR_UNSUPPORTED, "staged detector window does not fit in shared memory");
    a.chunk = stages;
    smem = (size_t)stages * per_stage + 64;
  }

  if (packed && !(st.pack_ready && st.filt_layout == layout))
    if (int rc = prepare_packed(ctx, st, layout, orb)) {
      // no room for the interleaved copy, or more view groups than its packer
      // takes: the plain kernel reads the rows themselves, or pairs of at most
      // the orbits' bytes
      if ((rc == FBP_ERR_OUT_OF_MEMORY || rc == FBP_ERR_UNSUPPORTED) && (orbit || layout == kLayoutQuad32))
        return plan_backproject(ctx, g, st, vol, clip_ylimit, mixed, plan_out, PlanLimits{false, false});
      return rc;
    }
  a.inv_scale = is_p16_layout(layout) || layout == kLayoutQuadG16 ? st.inv_scale : nullptr;  // set by the pack
  a.resident = occ * ctx->num_sms;  // CTAs resident at once (view-group skew of the symmetric kernel)
  a.band = std::max(1, (int)std::lround(std::sqrt((double)a.resident)));
  if (is_quad_layout(layout)) {
    a.qg = static_cast<const uint4*>(st.filt);
    a.qg_pitch = st.filt_pitch;
    a.qg_rows = st.v + a.pair_rows;
  }
  // the grid of boxes over the staged views (4-byte elements, or 16-byte planes)
  const void* base = packed ? st.filt : (const void*)st.f32;
  const int pitch_el = packed ? st.filt_pitch : st.pitch;
  const uint64_t pitch_bytes = (uint64_t)pitch_el * esize;
  const uint64_t ux = (uint64_t)st.u;
  const uint64_t rows_v = (uint64_t)st.v + a.pair_rows;  // element rows per view
  BoxMaps maps;
  // interleaved layout: boxes of at most 128 x 256 elements (TMA: 256 words per
  // box row) and at most the ring; larger windows are gathered directly
  // (the widest box of the interleaved layouts is widened, within 128, to a
  // bank-friendly row stride, as choose_boxes picks the narrower ones)
  const int planes = is_quad_layout(layout) ? esize / 16 : 0;  // 0: 8-byte elements
  int mbu = is_quad_layout(layout) ? std::min(bu, 128) : bu;
  if (planes > 0)
    for (int wider = mbu; wider <= 128 && wider < mbu + 8; ++wider)
      if (bank_friendly(planes, wider)) {
        mbu = wider;
        break;
      }
  const int mbv = is_quad_layout(layout) ? std::min({bv, 256, std::max(1, (int)(a.box_bytes / (esize * mbu)))}) : bv;
  if (!(plan.sel_layout == layout && plan.sel_u == mbu && plan.sel_v == mbv)) {
    // the interleaved layouts take the boxes fitted to the histogram (C4: the
    // MIXED backprojection 1405 -> 1289 ms); the others keep the quarter steps
    // of the largest window
    static const std::vector<unsigned> no_hist;
    choose_boxes(is_quad_layout(layout) ? plan.hist : no_hist, mbu, mbv, a.align, a.pair_rows, planes, plan.sel_w,
                 plan.sel_h);
    // 4-byte rows: a warp's lanes fall on two or three neighbouring rows, ten
    // to twenty columns wide; widths of 12 to 20 mod 32 keep those off one
    // another's banks (FP32 rows, 300 x 251 x 300, 451 views: 8.58 -> 7.40 ms)
    if (!is_quad_layout(layout))
      for (int i = 0; i < kNW; ++i) {
        int w = plan.sel_w[i];
        while (w < mbu && !(w % 32 >= 12 && w % 32 <= 20)) w += 4;
        plan.sel_w[i] = w;
      }
    plan.sel_layout = layout;
    plan.sel_u = mbu;
    plan.sel_v = mbv;
  }
  for (int i = 0; i < kNW; ++i) maps.w[i] = plan.sel_w[i];
  for (int j = 0; j < kNH; ++j) maps.h[j] = plan.sel_h[j];
  for (int i = 0; i < kNW; ++i)
    for (int j = 0; j < kNH; ++j) {
      if (is_quad_layout(layout)) {  // [group][element row][plane][element column][2 x 8 bytes]
        const uint32_t words = esize == 8 ? 1 : 2;  // 8-byte words per column of a plane
        const uint32_t np = (uint32_t)std::max(1, planes);
        const uint64_t d4[4] = {(uint64_t)words * pitch_el, np, rows_v, (uint64_t)orb.groups};
        const uint64_t s4[3] = {8ull * words * pitch_el, (uint64_t)esize * pitch_el, (uint64_t)esize * pitch_el * rows_v};
        const uint32_t b4[4] = {words * maps.w[i], np, (uint32_t)maps.h[j], 1};
        if (int rc = make_tensor_map_4d(ctx, &maps.map[i * kNH + j], CU_TENSOR_MAP_DATA_TYPE_UINT64,
                                        const_cast<void*>(base), d4, s4, b4))
          return rc;
        continue;
      }
      const uint32_t box_x = maps.w[i];
      uint64_t dims[3], strides[2];
      uint32_t box[3];
      if (st.sinogram) {  // [v][view][u]
        dims[0] = ux;
        dims[1] = st.n;
        dims[2] = rows_v;
        strides[0] = pitch_bytes;
        strides[1] = pitch_bytes * st.n;
        box[0] = box_x;
        box[1] = 1;
        box[2] = maps.h[j];
      } else {  // [view][v][u]
        dims[0] = ux;
        dims[1] = rows_v;
        dims[2] = st.n;
        strides[0] = pitch_bytes;
        strides[1] = pitch_bytes * rows_v;
        box[0] = box_x;
        box[1] = maps.h[j];
        box[2] = 1;
      }
      if (int rc = make_tensor_map_3d(ctx, &maps.map[i * kNH + j], CU_TENSOR_MAP_DATA_TYPE_FLOAT32,
                                      const_cast<void*>(base), dims, strides, box))
        return rc;
    }
  // the stored values' extremes feed histogram normalisation of the context's volume
  if (vol == ctx->vol && ctx->d_minmax) {
    if (int rc = launch_minmax_init(ctx, ctx->d_minmax)) return rc;
    a.minmax = ctx->d_minmax;
  }
  BPLaunchPlan& p = *plan_out;
  p.a = a;
  p.maps = maps;
  p.smem = smem;
  p.layout = layout;
  p.ny_tile = NY;
  p.occ = occ;
  p.use_quad = use_quad;
  p.orbit = orbit;
  return FBP_OK;
}

int launch_bp_plan(fbp_context* ctx, const BPLaunchPlan& p) {
  const int NY = p.ny_tile;
  ctx->last_bp[0] = p.orbit      ? FBP_BACKPROJECTOR_ORBITS
                    : p.use_quad ? FBP_BACKPROJECTOR_SYMMETRIC
                    : NY == 8    ? FBP_BACKPROJECTOR_GENERIC_Y8
                                 : FBP_BACKPROJECTOR_GENERIC;
  ctx->last_bp[1] = p.layout;
  ctx->last_bp[2] = p.a.box_u;
  ctx->last_bp[3] = p.a.box_v;
  ctx->last_bp[4] = NY;
  cudaError_t e = p.use_quad ? launch_quad(p.layout, NY, p.maps, p.a, p.smem, ctx->stream)
                  : NY == 1  ? launch_layout<16, 16, 1>(p.layout, p.maps, p.a, p.smem, ctx->stream)
                  : NY == 8  ? launch_layout<16, 16, 8>(p.layout, p.maps, p.a, p.smem, ctx->stream)
                             : launch_layout<16, 16, 16>(p.layout, p.maps, p.a, p.smem, ctx->stream);
  if (e == cudaSuccess) ctx->launches++;
  ctx->minmax_valid = e == cudaSuccess && p.a.minmax != nullptr;
  return cuda_check(ctx, e, "bp_kernel");
}

int launch_backproject(fbp_context* ctx, const BPGeom& g, Stack& st, float* vol, int clip_ylimit, bool mixed) {
  BPLaunchPlan p;
  if (int rc = plan_backproject(ctx, g, st, vol, clip_ylimit, mixed, &p)) return rc;
  return launch_bp_plan(ctx, p);
}

long long bp_plan_batch_key(const BPLaunchPlan& p) {
  if (!p.use_quad || p.orbit) return 0;  // the persistent launch runs the four-fold symmetric kernel
  return 1 + p.layout + 16LL * p.ny_tile + 4096LL * p.occ + 65536LL * p.a.box_bytes;
}

namespace {

template <int LAYOUT, int NY, int YW, int OCC>
cudaError_t launch_quad_multi_cfg(const QuadQueue& qq, size_t smem, int grid, cudaStream_t stream) {
  auto kern = bp_quad_kernel<LAYOUT, NY, YW, OCC, true, false>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynamicSmem);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return e;
  static const BoxMaps no_maps{};
  static const BPArgs no_args{};
  kern<<<grid, quad_threads(LAYOUT, NY, YW), smem, stream>>>(no_maps, no_args, qq);
  return cudaGetLastError();
}

cudaError_t launch_quad_multi(int layout, int ny_tile, const QuadQueue& qq, size_t smem, int grid,
                              cudaStream_t stream) {
#define FBP_LAUNCH(L, NY, YW, OCC) launch_quad_multi_cfg<L, NY, YW, OCC>(qq, smem, grid, stream)
  switch (layout) { FBP_SYMMETRIC_SHAPES(FBP_LAUNCH) }
#undef FBP_LAUNCH
}

}  // namespace

// Several jobs' symmetric backprojections (plans with one batch key) in one
// persistent launch on the launcher's stream: OCC CTAs per SM walk a queue
// of (job, tile orbit, y-slab) work items, largest jobs first in the order
// given. The job table goes up through the launcher's pinned staging.
long long bp_plan_tiles(const BPLaunchPlan& p) {
  return (long long)p.a.nbx * p.a.nbz * ((p.a.ny + p.ny_tile - 1) / p.ny_tile);
}

int launch_bp_batch(fbp_context* L, BPLaunchPlan* const* plans, int n, const long long* tile_begin,
                    const long long* tile_end) {
  if (n <= 0) return FBP_OK;
  const BPLaunchPlan& p0 = *plans[0];
  const long long key = bp_plan_batch_key(p0);
  if (key == 0) return set_error(L, FBP_ERR_INVALID_ARGUMENT, "backprojection plan cannot run in a batch");
  const size_t jobs_bytes = (sizeof(QuadJob) * n + 63) / 64 * 64;
  const size_t maps_bytes = sizeof(BoxMaps) * n;
  const size_t bytes = jobs_bytes + maps_bytes + 64;
  if (L->batch_cap < bytes) {
    cudaFree(L->d_batch);
    L->d_batch = nullptr;
    L->batch_cap = 0;
    if (cuda_check(L, cudaMalloc(&L->d_batch, bytes), "cudaMalloc(batch table)")) return FBP_ERR_OUT_OF_MEMORY;
    L->batch_cap = bytes;
  }
  if (L->h_batch_cap < bytes) {
    // the previous table may still be on its way up
    if (L->h_batch && cuda_check(L, cudaStreamSynchronize(L->stream), "batch staging sync")) return FBP_ERR_CUDA;
    cudaFreeHost(L->h_batch);
    L->h_batch = nullptr;
    L->h_batch_cap = 0;
    if (cuda_check(L, cudaMallocHost(&L->h_batch, bytes), "cudaMallocHost(batch table)")) return FBP_ERR_OUT_OF_MEMORY;
    L->h_batch_cap = bytes;
  } else if (L->ev_batch_copy) {
    if (cuda_check(L, cudaEventSynchronize(L->ev_batch_copy), "batch staging reuse")) return FBP_ERR_CUDA;
  }
  unsigned char* h = static_cast<unsigned char*>(L->h_batch);
  QuadJob* hj = reinterpret_cast<QuadJob*>(h);
  BoxMaps* hm = reinterpret_cast<BoxMaps*>(h + jobs_bytes);
  long long items = 0;
  for (int i = 0; i < n; ++i) {
    const BPLaunchPlan& p = *plans[i];
    if (bp_plan_batch_key(p) != key)
      return set_error(L, FBP_ERR_INVALID_ARGUMENT, "a batch needs one staged layout, tile height and ring size");
    hj[i] = QuadJob{};
    hj[i].a = p.a;
    hj[i].a.minmax = nullptr;  // no histogram range for batched jobs
    hj[i].item0 = items;
    const long long all = bp_plan_tiles(p);
    const long long t0 = tile_begin ? std::max(0LL, tile_begin[i]) : 0;
    const long long t1 = tile_end ? std::min(all, tile_end[i]) : all;
    if (t1 <= t0) return set_error(L, FBP_ERR_INVALID_ARGUMENT, "empty tile range in a batch");
    hj[i].t0 = t0;
    hm[i] = p.maps;
    items += t1 - t0;
  }
  *reinterpret_cast<unsigned long long*>(h + jobs_bytes + maps_bytes) = 0ull;
  unsigned char* d = static_cast<unsigned char*>(L->d_batch);
  if (cuda_check(L, cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, L->stream), "batch table upload"))
    return FBP_ERR_CUDA;
  if (!L->ev_batch_copy && cuda_check(L, cudaEventCreateWithFlags(&L->ev_batch_copy, cudaEventDisableTiming),
                                      "batch event"))
    return FBP_ERR_CUDA;
  if (cuda_check(L, cudaEventRecord(L->ev_batch_copy, L->stream), "batch event record")) return FBP_ERR_CUDA;
  QuadQueue qq;
  qq.jobs = reinterpret_cast<const QuadJob*>(d);
  qq.maps = reinterpret_cast<const BoxMaps*>(d + jobs_bytes);
  qq.njobs = n;
  qq.nitems = items;
  qq.next = reinterpret_cast<unsigned long long*>(d + jobs_bytes + maps_bytes);
  qq.err = L->d_err;
  qq.ring = p0.a.box_bytes;
  const int grid = (int)std::min<long long>(items, (long long)p0.occ * L->num_sms);
  cudaError_t e = launch_quad_multi(p0.layout, p0.ny_tile, qq, p0.smem, grid, L->stream);
  if (e == cudaSuccess) L->launches++;
  return cuda_check(L, e, "bp_quad_kernel (batch)");
}

// ---------------------------------------------------------------------------
// 2D backprojection (parallel beam and flat-detector fan beam, FBP2D.cpp:96-122
// and FBP2D.cpp:31-52 with FBP3D's FDK weight restricted to v = 0).
//
// What bounds it is shared memory: a linear tap reads two FP32 samples, 8
// bytes an update. Everything else of a tap - the projected position, its
// floor and fraction, the distance weight - is shared by the pixels of a
// rotational orbit: on a circular orbit the pixel (X, Z) at view k and its
// image under the rotation that takes view k to view k + j Q project to the
// same detector position. The filtered rows are packed so that one element
// holds the samples of the SLOTS rows that such an orbit reads at one detector
// position:
//   SLOTS 4  one turn, K % 4 == 0, square image: rows g + j K/4
//   SLOTS 4  half a turn of parallel beam, K even, square image: rows g,
//            g + K/2 and the same two mirrored (the view half a turn on)
//   SLOTS 2  one turn, K even: rows g, g + K/2; any other parallel-beam view
//            set: row g and its mirror image (the half-turned pixel, same view)
//   SLOTS 1  any other fan-beam view set
// In phase m (rows g + m Q of the representative pixel, m < PHASES) the
// pixel's rotation r reads slot (m + r) mod SLOTS. The phases are the outer
// loop and the sums stay in slot order, turned by one slot between phases.
//
// A CTA owns a 32 x 32 tile of representative pixels, four pixels of one
// column a thread. A producer warp computes each step's tile-local projective
// coefficients and window origin in FP64 (one step a lane, re-based to the
// window so FP32 stays accurate) and copies the windows into a ring of
// shared-memory entries of kSteps2D steps with cp.async.bulk; the packed rows
// carry `pad` zero columns on either side, so a window that leaves the
// detector is an ordinary copy. The views are split over the CTAs of a cluster
// when the tiles alone would leave SMs idle; the partial sums are added in
// rank order through distributed shared memory, so results do not depend on
// timing.
//
// Measured (the packing included), before = one 32 x 32 tile of plain pixels
// a CTA with its setup and staging between block barriers: fan 1024^2, 1440
// views 2297 -> 537 us (82% of the shared-memory rate while a SM has work),
// 1441 views 2301 -> 1132 us; fan 512^2, 720 views 467 -> 83 us; parallel
// 256^2, 360 views 132 -> 21 us (about 12 us of it two launches and a CTA's
// start).
constexpr int kTile2D = 32;     // representative pixels per tile side
constexpr int kPix2D = 4;       // pixels per thread along z
constexpr int kSteps2D = 4;     // views per ring entry
constexpr int kWin2DMax = 516;  // widest staged window (columns)
constexpr int kMaxRing2D = 6;   // ring entries
constexpr int kMaxSplit2D = 4;  // CTAs that share a tile's views (one cluster)
constexpr int kPart2D = kTile2D + 1;  // row pitch of the partial sums (no bank conflicts across rows)

struct alignas(16) Coef2D {
  float Nx, Nz, N0;  // (u - u0) D, affine in the tile-local pixel
  float Dx, Dz, D0;
  float pad[2];
};

struct BP2DArgs {
  const float* rows;  // [groups][pitch][SLOTS]: column c is detector column c - pad
  long long pitch;
  float* image;       // [nz][nx]
  const double2* trig;
  double vox, cu;
  double du_per_mm;   // detector columns per unit of u D (cone: sdd / (sod du); parallel: 1 / du)
  double inv_sod;     // cone: D = 1 + (X cos + Z sin) inv_sod
  int nu, nx, nz;
  int groups, phases;
  int pad, win;       // zero columns either side, staged columns of a window
  int ring;           // ring entries
  float scale;
  int* err;
};

// rows [view][pitch] -> [g][column][SLOTS] with zero columns outside the detector
template <int SLOTS>
__global__ void pack2d_kernel(const float* __restrict__ src, long long spitch, int nu, int groups, int pad, int mirror,
                              long long pitch, float* __restrict__ out) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x, u = c - pad;
  if (c >= pitch) return;
  const bool in = u >= 0 && u < nu;
  for (int g = blockIdx.y; g < groups; g += gridDim.y) {
    float v[SLOTS];
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
      // slots past `mirror` rows are the first ones' mirror images
      const int row = s < mirror ? s : s - mirror, at = s < mirror ? u : nu - 1 - u;
      v[s] = in ? __ldg(src + (long long)(g + row * groups) * spitch + at) : 0.f;
    }
    float* o = out + ((long long)g * pitch + c) * SLOTS;
    if constexpr (SLOTS == 4) *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
    else if constexpr (SLOTS == 2) *reinterpret_cast<float2*>(o) = make_float2(v[0], v[1]);
    else o[0] = v[0];
  }
}

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

template <bool CONE, int SLOTS>
__global__ void __launch_bounds__(256 + 32, 2) bp2d_kernel(const BP2DArgs a) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(128) unsigned char smem2d[];
  constexpr int NCW = 8;
  constexpr int ALIGN = 4 / SLOTS;  // columns per 16 bytes
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), nsplit = (int)cluster.num_blocks();
  const int E = a.ring;
  const uint32_t win_bytes = (uint32_t)(a.win * SLOTS * 4);
  float* part = reinterpret_cast<float*>(smem2d);  // [SLOTS][32][kPart2D]
  unsigned char* wins = smem2d + sizeof(float) * SLOTS * kTile2D * kPart2D;  // a multiple of 128 bytes
  Coef2D* coef = reinterpret_cast<Coef2D*>(wins + (size_t)E * kSteps2D * win_bytes);
  uint64_t* full = reinterpret_cast<uint64_t*>(coef + E * kSteps2D);
  uint64_t* empty = full + E;
  volatile int* s_abort = reinterpret_cast<volatile int*>(empty + E);
  if (tid == 0) {
    *s_abort = *(volatile int*)a.err != 0;
    for (int e = 0; e < E; ++e) {
      mbar_init(&full[e], 1);
      mbar_init(&empty[e], NCW);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  const int ix0 = blockIdx.x * kTile2D, iz0 = blockIdx.y * kTile2D;
  // this CTA's row groups, in every phase
  const int g0 = (int)((long long)a.groups * rank / nsplit), g1 = (int)((long long)a.groups * (rank + 1) / nsplit);
  const int ng = g1 - g0, entries = (ng + kSteps2D - 1) / kSteps2D;
  const bool run = *s_abort == 0;  // an error already recorded: nothing is computed, the cluster still meets below

  float acc[SLOTS][kPix2D];
#pragma unroll
  for (int s = 0; s < SLOTS; ++s)
#pragma unroll
    for (int j = 0; j < kPix2D; ++j) acc[s][j] = 0.f;

  if (run && warp == NCW) {
    // ---------------------------------------------------------------- producer
    // the packed rows (and whatever ran before them) are complete from here on
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const double Xc = (ix0 + 0.5 - 0.5 * a.nx) * a.vox, Zc = (iz0 + 0.5 - 0.5 * a.nz) * a.vox;
    int seq = 0;  // entries filled
    bool ok = true;
    for (int m = 0; m < a.phases && ok; ++m)
      for (int gb = 0; gb < ng && ok; gb += 32) {
        Coef2D cf{};
        int start = 0;
        if (gb + lane < ng) {
          const int k = g0 + gb + lane + m * a.groups;
          const double c = a.trig[k].x, s = a.trig[k].y;
          double Dx = 0.0, Dz = 0.0, D0 = 1.0;
          if (CONE) {
            Dx = a.vox * a.inv_sod * c;
            Dz = a.vox * a.inv_sod * s;
            D0 = 1.0 + (Xc * c + Zc * s) * a.inv_sod;
          }
          const double Ux = -a.vox * s * a.du_per_mm, Uz = a.vox * c * a.du_per_mm;
          const double U0 = (-Xc * s + Zc * c) * a.du_per_mm;
          // Detector window over the tile's four corners (u is monotonic along
          // each edge, so the corners bound it). The FP64 chain of a lane is what
          // delays a CTA's first steps, so it holds no division: a Newton step on
          // the FP32 reciprocal leaves 1e-13 of a column's distance.
          double umin = 1e300, umax = -1e300, dmin = 1e300;
#pragma unroll
          for (int cc = 0; cc < 4; ++cc) {
            const double x = (cc & 1) ? kTile2D - 1 : 0, z = (cc & 2) ? kTile2D - 1 : 0;
            double u = Ux * x + (Uz * z + U0);
            if (CONE) {
              const double D = Dx * x + (Dz * z + D0), r = (double)rcp_approx((float)D);
              dmin = fmin(dmin, D);
              u *= r * (2.0 - D * r);
            }
            umin = fmin(umin, u);
            umax = fmax(umax, u);
          }
          // one column of margin on each side for the FP32 rounding of the taps'
          // positions; a window that starts left of the padding or past the
          // detector holds zeros only, whatever its origin
          const double cap = 1 << 30;
          const int u0 = (int)floor(fmin(fmax(umin + a.cu - 1.0, -cap), cap)) & ~(ALIGN - 1);
          const bool fits = floor(umax + a.cu) + 3.0 - u0 <= (double)a.win;
          if (!(dmin > 1e-6) || !fits) atomicCAS(a.err, 0, kDevFootprint);
          start = min(max(u0 + a.pad, 0), a.pad + (a.nu + ALIGN - 1) / ALIGN * ALIGN);
          const double du0 = a.cu - u0;  // u - u0 = (N . (x, z, 1)) / D with N re-based
          cf.Nx = (float)(Ux + du0 * Dx);
          cf.Nz = (float)(Uz + du0 * Dz);
          cf.N0 = (float)(U0 + du0 * D0);
          cf.Dx = (float)Dx;
          cf.Dz = (float)Dz;
          cf.D0 = (float)D0;
        }
        const int left = min(32, ng - gb);
        for (int i = 0; i < left; i += kSteps2D) {
          const int e = seq % E, n = min(kSteps2D, left - i);
          if (seq >= E && !mbar_wait(&empty[e], ((seq / E) & 1) ^ 1, a.err)) {
            ok = false;
            *s_abort = 1;
            break;
          }
          if (lane >= i && lane < i + n) coef[e * kSteps2D + lane - i] = cf;
          __syncwarp();
          if (lane == 0) mbar_arrive_expect_tx(&full[e], (uint32_t)n * win_bytes);
          __syncwarp();
          if (lane >= i && lane < i + n)
            bulk_load(wins + (size_t)(e * kSteps2D + lane - i) * win_bytes,
                      a.rows + ((long long)(g0 + gb + lane) * a.pitch + start) * SLOTS, win_bytes, &full[e]);
          __syncwarp();
          ++seq;
        }
      }
    // leave only when every copy issued into this CTA's memory has landed
    for (int q = max(0, seq - E); q < seq; ++q) mbar_wait(&full[q % E], (q / E) & 1, a.err);
  } else if (run) {
    // --------------------------------------------------------------- consumers
    const float fx = (float)lane, fz = (float)(warp * kPix2D);
    const uint32_t wbase = smem_u32(wins);
    // a tap's column is in [0, win - 2]: bounds the reads. worst: the largest
    // one that a tap asked for (negative ones are larger than any)
    const uint32_t last = (uint32_t)(a.win - 2);
    uint32_t worst = 0;
    const float2 magic2 = make_float2(kMagic, kMagic);
    int e = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int m = 0; m < a.phases && ok; ++m) {
      for (int q = 0; q < entries; ++q) {
        if (!mbar_wait(&full[e], ph, a.err)) {
          ok = false;
          *s_abort = 1;
          break;
        }
        const int n = min(kSteps2D, ng - q * kSteps2D);
        for (int i = 0; i < n; ++i) {
          const float4 N = *reinterpret_cast<const float4*>(&coef[e * kSteps2D + i]);
          const float2 D = *reinterpret_cast<const float2*>(&coef[e * kSteps2D + i].Dz);
          const uint32_t c0 = wbase + (uint32_t)(e * kSteps2D + i) * win_bytes;
          // pixels j, j + 1 as packed pairs, each from its own z (stepped from pixel
          // to pixel, the rounding adds up)
          const float n0 = fmaf(N.x, fx, N.z), d0 = fmaf(N.w, fx, D.y);
#pragma unroll
          for (int j = 0; j < kPix2D; j += 2) {
            const float2 z2 = make_float2(fz + (float)j, fz + (float)(j + 1));
            float2 u = ffma2(make_float2(N.y, N.y), z2, make_float2(n0, n0)), W = make_float2(1.f, 1.f);
            if (CONE) {
              const float2 den = ffma2(make_float2(D.x, D.x), z2, make_float2(d0, d0));
              float2 rD = make_float2(rcp_approx(den.x), rcp_approx(den.y));  // and a Newton step, as rcp_newton
              rD = ffma2(rD, ffma2(make_float2(-den.x, -den.y), rD, make_float2(1.f, 1.f)), rD);
              u = fmul2(u, rD);
              W = fmul2(rD, rD);
            }
            const float2 t = fadd2_rz(u, magic2);
            const float2 fu = fsub2(u, fsub2(t, magic2));
            const uint32_t col[2] = {__float_as_uint(t.x) - kMagicBits, __float_as_uint(t.y) - kMagicBits};
            worst = max(worst, max(col[0], col[1]));
#pragma unroll
            for (int p = 0; p < 2; ++p) {
              const uint32_t at = min(col[p], last) * (4u * SLOTS) + c0;
              // one rounding into a sum: two weighted products added to it in turn cost
              // an operation less and up to a third more error (3.0 -> 4.2e-7 at a
              // drawn rebinned slice; fan 1024^2, 1440 views 645 and 661 us the call)
              const float fp = p ? fu.y : fu.x, Wp = p ? W.y : W.x;
              auto add = [&](int s, float2 A, float2 B) {
                const float2 x = ffma2(make_float2(fp, fp), fsub2(B, A), A);
                const float2 c = make_float2(acc[s][j + p], acc[s + 1][j + p]);
                const float2 d = CONE ? ffma2(make_float2(Wp, Wp), x, c) : fadd2(c, x);
                acc[s][j + p] = d.x, acc[s + 1][j + p] = d.y;
              };
              if constexpr (SLOTS == 4) {
                const uint4 A = lds_u4(at), B = lds_u4(at + 16);
                add(0, make_float2(__uint_as_float(A.x), __uint_as_float(A.y)),
                    make_float2(__uint_as_float(B.x), __uint_as_float(B.y)));
                add(2, make_float2(__uint_as_float(A.z), __uint_as_float(A.w)),
                    make_float2(__uint_as_float(B.z), __uint_as_float(B.w)));
              } else if constexpr (SLOTS == 2) {
                add(0, lds_f32x2(at), lds_f32x2(at + 8));
              } else {
                const float A = lds_f32(at), x = fmaf(fp, lds_f32(at + 4) - A, A);
                acc[0][j + p] = CONE ? fmaf(Wp, x, acc[0][j + p]) : acc[0][j + p] + x;
              }
            }
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[e]);
        if (++e == E) {
          e = 0;
          ph ^= 1;
        }
      }
      // the next phase's slot s belongs to the rotation of this phase's slot s - 1
#pragma unroll
      for (int j = 0; j < kPix2D; ++j) {
        const float t = acc[SLOTS - 1][j];
#pragma unroll
        for (int s = SLOTS - 1; s > 0; --s) acc[s][j] = acc[s - 1][j];
        acc[0][j] = t;
      }
    }
    // cannot happen when the window above is right (a NaN angle's taps are NaN)
    if (worst > last && worst != 0x7fffffffu - kMagicBits) atomicCAS(a.err, 0, kDevFootprint);
  }
  if (warp < NCW) {
    // after `phases` turns rotation r sits in slot (r + phases) mod SLOTS
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
      const int r = (s + SLOTS - a.phases % SLOTS) % SLOTS;
#pragma unroll
      for (int j = 0; j < kPix2D; ++j) part[(r * kTile2D + warp * kPix2D + j) * kPart2D + lane] = acc[s][j];
    }
  }
  __syncwarp();
  if (nsplit > 1) cluster.sync();
  else __syncthreads();
  // The tile's SLOTS rotated images, a 32-pixel line of image x a warp: for
  // the quarter turns (x, z) -> (n-1-z, x) -> (n-1-x, n-1-z) -> (z, n-1-x)
  // image x runs along the tile's z. Pixels that are their own image (the
  // middle row / the centre of an odd size) are written by rotation 0 alone.
  const bool skip = *s_abort != 0;
  for (int l = rank + nsplit * warp; l < SLOTS * kTile2D && !skip && warp < NCW; l += nsplit * NCW) {
    const int r = l / kTile2D, i = l - r * kTile2D;
    const bool turned = SLOTS == 4 && (r & 1);
    const int x = turned ? i : lane, z = turned ? lane : i;
    const float* own = part + (r * kTile2D + z) * kPart2D + x;
    float sum;
    if (nsplit == 1) {
      sum = *own;
    } else {  // all ranks' loads in flight, added in rank order
      float v[kMaxSplit2D];
#pragma unroll
      for (int q = 0; q < kMaxSplit2D; ++q) v[q] = q < nsplit ? *cluster.map_shared_rank(own, q) : 0.f;
      sum = v[0];
#pragma unroll
      for (int q = 1; q < kMaxSplit2D; ++q) sum += v[q];
    }
    const int ix = ix0 + x, iz = iz0 + z;
    bool in = ix < a.nx && iz < a.nz;
    int ox = ix, oz = iz;
    if (SLOTS == 4) {
      const int n = a.nx, h = n / 2;  // representatives: x < n - h, z < h, and the centre of an odd size
      in = ix < n - h && (iz < h || (r == 0 && iz == h && ix == h && (n & 1)));
      if (r == 1) ox = n - 1 - iz, oz = ix;
      if (r == 2) ox = n - 1 - ix, oz = n - 1 - iz;
      if (r == 3) ox = iz, oz = n - 1 - ix;
    } else if (SLOTS == 2) {
      in = ix < a.nx && (iz < a.nz / 2 || (r == 0 && iz == a.nz / 2 && (a.nz & 1)));
      if (r == 1) ox = a.nx - 1 - ix, oz = a.nz - 1 - iz;
    }
    if (in) a.image[(size_t)oz * a.nx + ox] = sum * a.scale;
  }
  __syncwarp();
  if (nsplit > 1) cluster.sync();  // no CTA leaves while another reads its sums
}

// The rows where they are, a pixel a thread, positions in FP64: for a device
// without room for the packed rows.
__global__ void __launch_bounds__(256) bp2d_rows_kernel(const BP2DArgs a, int nviews) {
  const int ix = blockIdx.x * 32 + threadIdx.x % 32;
  for (int iz = blockIdx.y * 8 + threadIdx.x / 32; iz < a.nz && ix < a.nx; iz += gridDim.y * 8) {
    const double X = (ix + 0.5 - 0.5 * a.nx) * a.vox, Z = (iz + 0.5 - 0.5 * a.nz) * a.vox;
    float acc = 0.f;
    for (int k = 0; k < nviews; ++k) {
      const double c = a.trig[k].x, s = a.trig[k].y;
      const double rD = 1.0 / (1.0 + (X * c + Z * s) * a.inv_sod);
      const double u = (Z * c - X * s) * a.du_per_mm * rD + a.cu, fl = floor(u);
      if (!(fl >= -1.0 && fl < (double)a.nu)) continue;
      const int iu = (int)fl;
      const float* p = a.rows + (long long)k * a.pitch + iu;
      const float lo = iu >= 0 ? __ldg(p) : 0.f, hi = iu + 1 < a.nu ? __ldg(p + 1) : 0.f;
      acc = fmaf((float)(rD * rD), fmaf((float)(u - fl), hi - lo, lo), acc);
    }
    a.image[(size_t)iz * a.nx + ix] = acc * a.scale;
  }
}

template <bool CONE, int SLOTS>
cudaError_t launch_bp2d_cfg(const BP2DArgs& a, dim3 grid, size_t smem, cudaStream_t stream) {
  auto kern = bp2d_kernel<CONE, SLOTS>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynamicSmem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(256 + 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 1;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = grid.z;
  // the CTAs start (barriers, cluster) while the packing kernel drains
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kern, a);
}

int launch_bp2d(fbp_context* ctx, const BPGeom& g, const float* sino, long long pitch, float* image) {
  const double pi = 3.14159265358979323846;
  const bool cone = g.kind == FBP_GEOMETRY_CONE;
  // widest window of a tile over all views: the tile diagonal magnified at the
  // image point nearest the source
  const double diag = (kTile2D - 1) * std::sqrt(2.0) * g.vox;
  double width = diag / g.du;
  if (cone) {
    const double r = 0.5 * std::sqrt((double)g.nx * g.nx + (double)g.nz * g.nz) * g.vox + diag;
    const double dmin = (g.sod - r) / g.sod;
    if (dmin < 0.05) return FBP_ERR_UNSUPPORTED;  // the source inside or near the image: general path
    width *= g.sdd / (g.sod * dmin);
  }
  if (!(width < kWin2DMax)) return FBP_ERR_UNSUPPORTED;
  const int win = ((int)std::ceil(width) + 8 + 3) / 4 * 4;
  if (win > kWin2DMax) return FBP_ERR_UNSUPPORTED;
  // rotational orbits of the view set
  // Four slots halve the work of two, but also the tiles: below one CTA a SM
  // (the cluster split included) two are faster (parallel 256^2, 360 views,
  // half a turn: 27.1 us with four slots, 21.0 with two)
  const int K = g.nviews;
  const int half = ((g.nx + 1) / 2 + kTile2D - 1) / kTile2D;
  const Orbits orb = find_orbits(cone, g.span / (2.0 * pi), K,
                                 g.nx == g.nz && half * half * kMaxSplit2D >= ctx->num_sms);
  const int slots = orb.slots, groups = orb.groups, phases = orb.phases, mirror = orb.mirror;
  const int rx = slots == 4 ? (g.nx + 1) / 2 : g.nx, rz = slots == 1 ? g.nz : (g.nz + 1) / 2;
  const int tiles_x = (rx + kTile2D - 1) / kTile2D, tiles_z = (rz + kTile2D - 1) / kTile2D;
  const long long tiles = (long long)tiles_x * tiles_z;
  if (int rc = ensure_trig(ctx, g)) return rc;
  BP2DArgs a{};
  a.image = image;
  a.trig = ctx->d_trig;
  a.vox = g.vox;
  a.cu = 0.5 * g.nu - 0.5;
  a.du_per_mm = cone ? g.sdd / (g.sod * g.du) : 1.0 / g.du;
  a.inv_sod = cone ? 1.0 / g.sod : 0.0;
  a.nu = g.nu;
  a.nx = g.nx;
  a.nz = g.nz;
  a.groups = groups;
  a.phases = phases;
  a.scale = cone ? (float)(pi / K * g.sdd / (g.sod * g.du)) : (float)(pi / K / g.du);
  a.err = ctx->d_err;
  a.pad = win;
  a.win = win;
  a.pitch = (g.nu + 3) / 4 * 4 + 2LL * win;
  const size_t bytes = sizeof(float) * (size_t)a.pitch * groups * slots;
  float* rows = static_cast<float*>(scratch(ctx, bytes));
  if (!rows) {
    ctx->last_error.clear();
    a.rows = sino;
    a.pitch = pitch;
    bp2d_rows_kernel<<<dim3((g.nx + 31) / 32, std::min((g.nz + 7) / 8, 65535)), 256, 0, ctx->stream>>>(a, K);
    return launched(ctx, "bp2d_rows_kernel");
  }
  const dim3 pgrid((unsigned)((a.pitch + 255) / 256), std::min(groups, 65535));
  if (slots == 4)
    pack2d_kernel<4><<<pgrid, 256, 0, ctx->stream>>>(sino, pitch, g.nu, groups, a.pad, mirror, a.pitch, rows);
  else if (slots == 2)
    pack2d_kernel<2><<<pgrid, 256, 0, ctx->stream>>>(sino, pitch, g.nu, groups, a.pad, mirror, a.pitch, rows);
  else
    pack2d_kernel<1><<<pgrid, 256, 0, ctx->stream>>>(sino, pitch, g.nu, groups, a.pad, mirror, a.pitch, rows);
  if (int rc = launched(ctx, "pack2d_kernel")) return rc;
  a.rows = rows;
  const size_t entry = (size_t)kSteps2D * (win * slots * 4 + sizeof(Coef2D)) + 2 * sizeof(uint64_t);
  const size_t fixed = sizeof(float) * slots * kTile2D * kPart2D + 16;
  a.ring = (int)std::max<size_t>(2, std::min<size_t>(kMaxRing2D, (48 * 1024) / entry));
  size_t smem = fixed + a.ring * entry;
  // Split the views over a cluster until one and a half tiles a SM are in
  // flight (fan 512^2, 720 views, 64 tiles: 164.0, 91.9, 83.0, 93.6 us split
  // 1, 2, 4, 8 ways; 1024^2, 1440 views, 256 tiles: 537.3, 536.3, 532.3,
  // 569.2 us). Clusters of 8 leave SMs of a GPC over.
  int split = 1;
  while (split < kMaxSplit2D && 2 * tiles * split < 3LL * ctx->num_sms && groups >= 16 * split) split *= 2;
  // CTAs that all find an SM of their own must not share one (the tap's
  // shared-memory rate is per SM): ask for more than half an SM's memory
  if (tiles * split <= ctx->num_sms) smem = std::max<size_t>(smem, 116 * 1024);
  const dim3 grid(tiles_x, tiles_z, split);
  cudaError_t e;
  if (slots == 4) e = cone ? launch_bp2d_cfg<true, 4>(a, grid, smem, ctx->stream) : launch_bp2d_cfg<false, 4>(a, grid, smem, ctx->stream);
  else if (slots == 2) e = cone ? launch_bp2d_cfg<true, 2>(a, grid, smem, ctx->stream) : launch_bp2d_cfg<false, 2>(a, grid, smem, ctx->stream);
  else e = cone ? launch_bp2d_cfg<true, 1>(a, grid, smem, ctx->stream) : launch_bp2d_cfg<false, 1>(a, grid, smem, ctx->stream);
  if (e == cudaSuccess) ctx->launches++;
  return cuda_check(ctx, e, "bp2d_kernel");
}

int launch_clip(fbp_context* ctx, float* vol, int nx, int ny, int nz, int y_limit) {
  long long total = (long long)nx * ny * nz;
  int blocks = (int)std::min<long long>((total + 255) / 256, (long long)ctx->num_sms * 16);
  if (total == 0) return FBP_OK;
  clip_kernel<<<blocks, 256, 0, ctx->stream>>>(vol, nx, ny, nz, y_limit);
  return launched(ctx, "clip_kernel");
}

int launch_rebin_fan(fbp_context* ctx, const float* fan, int bins, int views, const BPGeom& g, float* par,
                     int out_bins, double du_out) {
  long long total = (long long)views * out_bins;
  if (total == 0) return FBP_OK;
  int blocks = (int)std::min<long long>((total + 255) / 256, (long long)ctx->num_sms * 16);
  rebin_fan_kernel<<<blocks, 256, 0, ctx->stream>>>(fan, bins, views, g.sod, g.sdd, g.du, g.span, g.offset, par,
                                                    out_bins, du_out);
  return launched(ctx, "rebin_fan_kernel");
}

}  // namespace fbp
