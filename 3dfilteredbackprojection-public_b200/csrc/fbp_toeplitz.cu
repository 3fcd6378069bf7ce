// Row filtering as a dense product on the tensor cores (tcgen05).
//
// Filtering every detector row with the circular kernel g of the padded
// length n is Y = X T with T[k][i] = g[(i - k) mod n] (k, i < m): a dense,
// symmetric Toeplitz matrix (g is even). It replaces the per-view FFT chain of
// FBP3D::apply_filter_to_projections (Source/FilteredBackProjection/
// FBP3D.cpp:389-414) for the MIXED form. Precision: X and T are split into
// BF16 hi + lo parts (hi = bf16(x), lo = bf16(x - hi)), and
// Y = Xh Th + Xh Tl + Xl Th is accumulated in FP32 in tensor memory (the
// dropped Xl Tl term and the split residuals are ~2^-17 of |x|). Each row's
// smooth baseline b = sum_j c_j P_j (a degree-8 Chebyshev fit of the row, 9
// coefficients) is taken out before the split and its filtered contribution
// T b = sum_j c_j (T P_j) added back by the same tensor-core product: the K
// extent is extended by one 64-wide block whose first 9 columns hold the
// coefficients c_j (X side, split hi / lo) and the columns T P_j (T side,
// summed in FP64, split hi / lo). Detector rows sit on large, slowly varying
// values (line integrals of ~10, plateaus of opaque rays) against a high-pass
// output ten to a hundred times smaller, and the split's error follows
// |x - b| instead of |x|. On the noisy 2D fan case (768 bins, Poisson I0 =
// 1e5) the image error against the FP64 oracle is 3.2e-4 with the row mean
// alone and 4.1e-5 with the degree-8 baseline (numpy emulation of the same
// split); any baseline is exact in principle, since the same coefficients are
// subtracted and added back (to the split's 16 bits).
//
// Kernel: persistent, one CTA per SM, over 128 x 256 output tiles. One warp
// streams 32-wide K blocks of Xh, Xl, Th, Tl into a ring of four or more
// stages with TMA (64-byte swizzle), one issues
// tcgen05.mma.cta_group::1.kind::f16 (M 128, N up to 256, K 16: 6 per K block)
// into one of two accumulators in tensor memory and frees stages with
// tcgen05.commit, and four load the other accumulator with tcgen05.ld and
// write it in place, 32 columns at a time, by TMA stores that clip at the row's
// end. What bounds it: at long rows the tensor cores, then the operands' way
// from L2 (48 KB per 768 tensor cycles of a K block); at short ones the rows'
// bytes. All waits are bounded and TMEM is always released.

#include "fbp_internal.h"
#include "fbp_rows.cuh"

#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <utility>

namespace fbp {
namespace {

constexpr int BM = 128, BN = 256, BK = 32;
constexpr int A_BYTES = BM * BK * 2;  // 8 KB
constexpr int kMaxStages = 8;
constexpr int TMEM_COLS = 512;                // two accumulators
constexpr int kOutCols = 32;                  // columns of one output store: 128-byte rows
constexpr int OUT_BYTES = 32 * kOutCols * 4;  // 32 rows of a warp
constexpr int kGemmThreads = 192;
constexpr uint32_t kWait = 1u << 22;
constexpr int kBasis = 9;       // Chebyshev polynomials P_0 .. P_8 of the row baseline

// Inverse Gram matrix of the baseline basis on the row's samples (FP64 on the
// host, rounded to FP32): coefficients c = Ginv * (moments <x, P_j>).
struct BasisGram {
  float ginv[kBasis * kBasis];
};

__device__ __forceinline__ uint32_t su32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void bar_init(uint64_t* b, uint32_t n) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(b)), "r"(n) : "memory");
}
__device__ __forceinline__ void bar_expect_tx(uint64_t* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(su32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_wait(uint64_t* b, uint32_t parity, int* err) {
  for (uint32_t i = 0; i < kWait; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(su32(b)), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  atomicCAS(err, 0, kDevTimeout);
  return false;
}
__device__ __forceinline__ void tma_2d(void* dst, const CUtensorMap* m, int x, int y, uint64_t* b) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
          "r"(su32(dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(x), "r"(y), "r"(su32(b))
      : "memory");
}

__device__ __forceinline__ void tma_store_2d(const CUtensorMap* m, const void* src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(
                   reinterpret_cast<uint64_t>(m)),
               "r"(x), "r"(y), "r"(su32(src))
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

// Shared-memory matrix descriptor, K-major operand with 64-byte swizzle:
// start address >> 4 (bits 0-13), stride between 8-row groups 512 B >> 4
// (bits 32-45), descriptor version 1 (bits 46-47), swizzle mode 4 = 64B
// (bits 61-63). The leading-dimension offset is unused for swizzled K-major.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFF);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(512 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)4 << 61;
  return d;
}

// Instruction descriptor, kind::f16: D FP32 (bits 4-5 = 1), A and B BF16
// (bits 7-9 = 1, 10-12 = 1), both K-major, N >> 3 in bits 17-22, M >> 4 in
// bits 24-28.
__device__ __forceinline__ uint32_t instr_desc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}

__device__ __forceinline__ void mma(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(
          d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc));
}
__device__ __forceinline__ void mma_commit(uint64_t* b) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(su32(b)) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(su32(b)) : "memory");
}

struct GemmArgs {
  long long row0;  // first stack row of this chunk
  int nrows;       // rows in this chunk
  int m;           // samples per row (N and K extent)
  int ntile_n;     // tiles along N
  int bn;          // their width
  int tiles;       // tiles of the chunk
  int kblocks;     // 32-wide K blocks: the padded row and the baseline block
  int stages;
  int* err;
};

__host__ __device__ constexpr int stage_bytes(int bn) { return 2 * A_BYTES + 2 * bn * BK * 2; }

// Persistent, against one CTA per tile with the epilogue behind the last MMA,
// a two-stage ring of 64-wide K blocks and row-contiguous stores from padded
// shared memory:
// 18944 rows of 1152 161 -> 112 us (1.39 PFLOP/s), of 768 86 -> 52 us, 69120
// rows of 192 84 -> 33 us.
__global__ void __launch_bounds__(kGemmThreads, 1) toeplitz_gemm_kernel(const __grid_constant__ CUtensorMap mah,
                                                                       const __grid_constant__ CUtensorMap mal,
                                                                       const __grid_constant__ CUtensorMap mbh,
                                                                       const __grid_constant__ CUtensorMap mbl,
                                                                       const __grid_constant__ CUtensorMap mout,
                                                                       const GemmArgs g) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // the swizzle patterns repeat every 1024 bytes at most
  unsigned char* smem = smem_raw + ((1024 - (su32(smem_raw) & 1023)) & 1023);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int b_bytes = g.bn * BK * 2, sbytes = stage_bytes(g.bn), S = g.stages;
  unsigned char* out = smem + (size_t)S * sbytes;  // two output buffers per epilogue warp
  uint64_t* full = reinterpret_cast<uint64_t*>(out + 8 * OUT_BYTES);
  uint64_t* empty = full + kMaxStages;
  uint64_t* acc_full = empty + kMaxStages;
  uint64_t* acc_empty = acc_full + 2;
  uint64_t* done = acc_empty + 2;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(done + 1);
  const int KB = g.kblocks;

  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      bar_init(&full[s], 1);
      bar_init(&empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      bar_init(&acc_full[i], 1);
      bar_init(&acc_empty[i], 4);
    }
    bar_init(done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(tmem_holder)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_holder;

  if (warp == 0) {
    if (lane == 0) {  // TMA producer
      int it = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < g.tiles && ok; t += gridDim.x) {
        const int rowt = t / g.ntile_n * BM, col0 = t % g.ntile_n * g.bn;
        for (int kb = 0; kb < KB; ++kb, ++it) {
          const int s = it % S;
          if (it >= S && !bar_wait(&empty[s], ((it / S) & 1) ^ 1, g.err)) {
            ok = false;
            break;
          }
          unsigned char* st = smem + (size_t)s * sbytes;
          bar_expect_tx(&full[s], (uint32_t)sbytes);
          tma_2d(st, &mah, kb * BK, rowt, &full[s]);
          tma_2d(st + 2 * A_BYTES, &mbh, kb * BK, col0, &full[s]);
          tma_2d(st + 2 * A_BYTES + b_bytes, &mbl, kb * BK, col0, &full[s]);
          tma_2d(st + A_BYTES, &mal, kb * BK, rowt, &full[s]);
        }
      }
      if (!ok)  // drain: the last copy into each stage must land before the CTA exits
        for (int s = 0; s < S && s < it; ++s) bar_wait(&full[s], ((it - s + S - 1) / S - 1) & 1, g.err);
    }
  } else if (warp == 1) {
    if (lane == 0) {  // MMA issuer: D += Ah Bh + Ah Bl + Al Bh per K block
      int it = 0, i = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < g.tiles && ok; t += gridDim.x, ++i) {
        const int col0 = t % g.ntile_n * g.bn;
        const uint32_t idesc = instr_desc(min(g.bn, (g.m - col0 + 31) / 32 * 32));
        const uint32_t d = tmem + (uint32_t)(i & 1) * 256u;
        if (i >= 2 && !bar_wait(&acc_empty[i & 1], ((i >> 1) & 1) ^ 1, g.err)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int kb = 0; kb < KB; ++kb, ++it) {
          const int s = it % S;
          if (!bar_wait(&full[s], (it / S) & 1, g.err)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t st = su32(smem + (size_t)s * sbytes);
          const uint32_t ah = st, al = st + A_BYTES, bh = st + 2 * A_BYTES, bl = bh + b_bytes;
#pragma unroll
          for (int term = 0; term < 3; ++term) {
            const uint32_t a = term == 2 ? al : ah;
            const uint32_t b = term == 1 ? bl : bh;
#pragma unroll
            for (int ks = 0; ks < BK / 16; ++ks)  // 16 BF16 = 32 bytes along K inside the swizzled row
              mma(d, smem_desc(a + ks * 32), smem_desc(b + ks * 32), idesc, (kb | term | ks) ? 1u : 0u);
          }
          mma_commit(&empty[s]);  // stage free once these MMAs have read it
        }
        if (ok) mma_commit(&acc_full[i & 1]);
      }
      mma_commit(done);  // no MMA in flight past this, after a time-out either
      bar_wait(done, 0, g.err);
    }
  } else {
    // epilogue: a warp reads the TMEM lanes 32 (warp % 4) .. + 31, one row each
    const int quarter = warp & 3;
    unsigned char* buf = out + (warp - 2) * 2 * OUT_BYTES;
    int i = 0, stores = 0;
    for (int t = blockIdx.x; t < g.tiles; t += gridDim.x, ++i) {
      const int row = t / g.ntile_n * BM + 32 * quarter, col0 = t % g.ntile_n * g.bn;
      const int cols = min(g.bn, g.m - col0);
      if (!bar_wait(&acc_full[i & 1], (i >> 1) & 1, g.err)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int c = 0; c < cols; c += kOutCols) {
        uint32_t v[32];
        const uint32_t addr = tmem + ((uint32_t)(32 * quarter) << 16) + (uint32_t)((i & 1) * 256 + c);
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%"
            "19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
              "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
              "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
              "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
            : "r"(addr));
        unsigned char* b = buf + (stores & 1) * OUT_BYTES;
        // the store before the last has left this buffer
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        __syncwarp();
        // 128-byte swizzle: eight rows' 16-byte pieces in different banks
#pragma unroll
        for (int j = 0; j < 8; ++j)
          *reinterpret_cast<uint4*>(b + lane * 128 + ((j ^ (lane & 7)) << 4)) =
              make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0 && row < g.nrows) tma_store_2d(&mout, b, col0 + c, (int)(g.row0 + row));
        ++stores;
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive(&acc_empty[i & 1]);
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}

// Chebyshev polynomials P_0 .. P_8 at t in [-1, 1]: P_{j+1} = 2 t P_j - P_{j-1}.
__device__ __forceinline__ void cheb9(float t, float (&p)[kBasis]) {
  const float t2 = t + t;
  p[0] = 1.f;
  p[1] = t;
#pragma unroll
  for (int j = 1; j + 1 < kBasis; ++j) p[j + 1] = fmaf(t2, p[j], -p[j - 1]);
}

// Sums v[0 .. 31] over the warp: lane l returns the sum of v[l]. Each exchange
// halves what a lane still carries (31 shuffles for 32 sums).
__device__ __forceinline__ float warp_sums32(float (&v)[32], int lane) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const float give = up ? v[i] : v[i + o], keep = up ? v[i + o] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  return v[0];
}

__device__ __forceinline__ void split2(float x, float y, uint32_t& h, uint32_t& l) {
  const __nv_bfloat162 hh = __floats2bfloat162_rn(x, y);
  h = *reinterpret_cast<const uint32_t*>(&hh);
  const __nv_bfloat162 ll = __floats2bfloat162_rn(x - __uint_as_float(h << 16), y - __uint_as_float(h & 0xffff0000u));
  l = *reinterpret_cast<const uint32_t*>(&ll);
}

constexpr int kSplitWarps = 4;
constexpr int kCoef = 12;  // floats per row of the moments and coefficients in shared memory

__host__ __device__ constexpr size_t split_smem(int R, int kp, bool stage) {
  return sizeof(float) * (84 + kSplitWarps * (2 * R * kCoef + (stage ? (size_t)R * kp : 0)));
}

// X rows (fused log / weight) -> BF16 hi and lo rows of x - b,
// b = the row's degree-8 Chebyshev fit, whose coefficients (split the same
// way) fill the first columns of the row's baseline block [kp, kx). A warp
// takes R rows at once, four samples of each per lane step (16-byte loads,
// 8-byte stores): bound by the arithmetic of the fit, of which the polynomials
// are formed once for R rows and the nine moments of all of them summed
// together. One row at a time took 82 us for 65536 rows of 192 samples and
// 274 us for as many of 1152;
// now 48 and 192 us.
// STAGE: the rows' pre-processed samples wait in shared memory between the fit
// and the split instead of being read and pre-processed twice.
template <int R, bool STAGE>
__global__ void __launch_bounds__(32 * kSplitWarps) split_rows_kernel(RowSet rs, long long row0, int nrows, int kp,
                                                                      int kx, __nv_bfloat16* xh, __nv_bfloat16* xl,
                                                                      const BasisGram gram) {
  extern __shared__ __align__(16) float sm[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  float* ginv = sm;  // 81 of 84 floats
  float* mom = sm + 84 + wib * 2 * R * kCoef;
  float* coef = mom + R * kCoef;
  float4* buf = reinterpret_cast<float4*>(sm + 84 + kSplitWarps * 2 * R * kCoef + (size_t)wib * R * kp);
  for (int i = threadIdx.x; i < kBasis * kBasis; i += blockDim.x) ginv[i] = gram.ginv[i];
  __syncthreads();
  const int step = gridDim.x * kSplitWarps * R;
  const float half_span = rs.m > 1 ? 0.5f * (float)(rs.m - 1) : 1.f;
  const float inv_half = 1.f / half_span;
  const int nq4 = kp >> 2;  // float4 groups of the padded row
  for (int r = (blockIdx.x * kSplitWarps + wib) * R; r < nrows; r += step) {
    const float* src[R];
    float dist2[R];
#pragma unroll
    for (int k = 0; k < R; ++k) {  // rows past the chunk: its last one again
      const long long gr = row0 + min(r + k, nrows - 1);
      src[k] = rs.data + gr * rs.pitch;
      dist2[k] = rs.weight ? pre_row(rs, gr) : 0.f;
    }
    auto load = [&](int q, float (&x)[R][4]) {
#pragma unroll
      for (int k = 0; k < R; ++k) {
        // the row pitch is a multiple of 4: the 16-byte load stays in the row
        const float4 v = 4 * q < rs.m ? reinterpret_cast<const float4*>(src[k])[q] : make_float4(0.f, 0.f, 0.f, 0.f);
        x[k][0] = v.x, x[k][1] = v.y, x[k][2] = v.z, x[k][3] = v.w;
      }
      if (rs.log_norm) {
#pragma unroll
        for (int k = 0; k < R; ++k)
#pragma unroll
          for (int t = 0; t < 4; ++t) x[k][t] = pre_log(rs, x[k][t]);
      }
      if (rs.weight) {
        const float u = (4 * q + 0.5f - 0.5f * rs.m) * rs.w_du;
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
          for (int k = 0; k < R; ++k) x[k][t] *= pre_weight(rs, dist2[k], fmaf((float)t, rs.w_du, u));
      }
      if (4 * q + 3 >= rs.m) {
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
          for (int k = 0; k < R; ++k)
            if (4 * q + t >= rs.m) x[k][t] = 0.f;
      }
    };
    // moments <x, P_j> of the pre-processed rows (zero past m)
    float acc[R][kBasis];
#pragma unroll
    for (int k = 0; k < R; ++k)
#pragma unroll
      for (int j = 0; j < kBasis; ++j) acc[k][j] = 0.f;
    for (int q = lane; q < nq4; q += 32) {
      float x[R][4];
      load(q, x);
      const float t0 = ((float)(4 * q) - half_span) * inv_half;
      if (STAGE) {
#pragma unroll
        for (int k = 0; k < R; ++k) buf[k * nq4 + q] = make_float4(x[k][0], x[k][1], x[k][2], x[k][3]);
      }
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        float p[kBasis];
        cheb9(fmaf((float)t, inv_half, t0), p);
#pragma unroll
        for (int k = 0; k < R; ++k)
#pragma unroll
          for (int j = 0; j < kBasis; ++j) acc[k][j] = fmaf(x[k][t], p[j], acc[k][j]);
      }
    }
    // sums of the R x 8 first moments together, the ninths one by one
    {
      float v[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = i < 8 * R ? acc[i / 8][i % 8] : 0.f;
      const float s = warp_sums32(v, lane);
      if (lane < 8 * R) mom[lane / 8 * kCoef + lane % 8] = s;
    }
#pragma unroll
    for (int k = 0; k < R; ++k) {
      float s = acc[k][8];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) mom[k * kCoef + 8] = s;
    }
    __syncwarp();
    for (int e = lane; e < R * kBasis; e += 32) {
      const int k = e / kBasis, a = e - k * kBasis;
      float sum = 0.f;
#pragma unroll
      for (int b = 0; b < kBasis; ++b) sum = fmaf(ginv[a * kBasis + b], mom[k * kCoef + b], sum);
      coef[k * kCoef + a] = sum;
    }
    __syncwarp();
    float c[R][kBasis];
#pragma unroll
    for (int k = 0; k < R; ++k)
#pragma unroll
      for (int j = 0; j < kBasis; ++j) c[k][j] = coef[k * kCoef + j];  // wide broadcast reads
    // the baseline blocks (columns kp .. kp + 31): c_0 .. c_8, then zeros
#pragma unroll
    for (int k = 0; k < R; ++k) {
      if (lane < (kx - kp) / 4 && r + k < nrows) {
        float v[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) v[t] = 4 * lane + t < kBasis ? coef[k * kCoef + 4 * lane + t] : 0.f;
        uint2 h, l;
        split2(v[0], v[1], h.x, l.x);
        split2(v[2], v[3], h.y, l.y);
        reinterpret_cast<uint2*>(xh + (size_t)(r + k) * kx)[(kp >> 2) + lane] = h;
        reinterpret_cast<uint2*>(xl + (size_t)(r + k) * kx)[(kp >> 2) + lane] = l;
      }
    }
    // x - b, split into BF16 hi and lo (each lane reads back what it wrote);
    // past m that is the fit's own value, which meets zeros on the T side
    for (int q = lane; q < nq4; q += 32) {
      float x[R][4];
      if (STAGE) {
#pragma unroll
        for (int k = 0; k < R; ++k) {
          const float4 v = buf[k * nq4 + q];
          x[k][0] = v.x, x[k][1] = v.y, x[k][2] = v.z, x[k][3] = v.w;
        }
      } else {
        load(q, x);
      }
      const float t0 = ((float)(4 * q) - half_span) * inv_half;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        float p[kBasis];
        cheb9(fmaf((float)t, inv_half, t0), p);
#pragma unroll
        for (int k = 0; k < R; ++k) {
          float b = c[k][0];
#pragma unroll
          for (int j = 1; j < kBasis; ++j) b = fmaf(c[k][j], p[j], b);
          x[k][t] -= b;
        }
      }
#pragma unroll
      for (int k = 0; k < R; ++k) {
        uint2 h, l;
        split2(x[k][0], x[k][1], h.x, l.x);
        split2(x[k][2], x[k][3], h.y, l.y);
        if (r + k < nrows) {
          reinterpret_cast<uint2*>(xh + (size_t)(r + k) * kx)[q] = h;
          reinterpret_cast<uint2*>(xl + (size_t)(r + k) * kx)[q] = l;
        }
      }
    }
    __syncwarp();  // the moments and coefficients are written again
  }
}

// tp[j][i] = sum over k < m of P_j(t_k) T[k][i] = P_j(t_k) g[(i - k) mod n], in
// FP64, one warp per i (a thread per i left most SMs idle: 377 us at m = 1536,
// now 23 us).
__global__ void toeplitz_basis_kernel(const float* g, int n, int m, float* tp) {
  const double half = m > 1 ? 0.5 * (m - 1) : 1.0;
  const int lane = threadIdx.x & 31, i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i >= m) return;
  double acc[kBasis];
#pragma unroll
  for (int j = 0; j < kBasis; ++j) acc[j] = 0.0;
  for (int k = lane; k < m; k += 32) {
    const double t = (k - half) / half, gk = (double)g[(((i - k) % n) + n) % n];
    double pm = 1.0, pj = t;
    acc[0] += gk;
    acc[1] += t * gk;
#pragma unroll
    for (int j = 1; j + 1 < kBasis; ++j) {
      const double pn = 2.0 * t * pj - pm;
      acc[j + 1] += pn * gk;
      pm = pj;
      pj = pn;
    }
  }
#pragma unroll
  for (int j = 0; j < kBasis; ++j) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
    if (lane == 0) tp[(size_t)j * m + i] = (float)acc[j];
  }
}

// Bt[i][k] = T[k][i] = g[(i - k) mod n] for k < m, (T P_j)[i] for k = kp + j
// (the baseline block), zero otherwise; split into BF16 hi and lo (k < kx).
__global__ void build_toeplitz_kernel(const float* g, int n, int m, int kp, int kx, const float* tp,
                                      __nv_bfloat16* th, __nv_bfloat16* tl) {
  const long long total = (long long)m * kx;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e / kx), k = (int)(e - (long long)i * kx);
    float t = 0.f;
    if (k < m)
      t = g[(((i - k) % n) + n) % n];
    else if (k >= kp && k < kp + kBasis)
      t = tp[(size_t)(k - kp) * m + i];
    const __nv_bfloat16 h = __float2bfloat16_rn(t);
    th[e] = h;
    tl[e] = __float2bfloat16_rn(t - __bfloat162float(h));
  }
}


}  // namespace

bool toeplitz_supported(int m) { return m >= 64 && m <= 8192; }

namespace {
// Inverse Gram matrix of the Chebyshev P_0 .. P_8 at t_k = (k - (m - 1) / 2) / ((m - 1) / 2),
// k < m, in FP64 (Gauss-Jordan with partial pivoting; the matrix is nearly
// diagonal), rounded to FP32.
BasisGram basis_gram(int m) {
  double G[kBasis][2 * kBasis] = {};
  const double half = m > 1 ? 0.5 * (m - 1) : 1.0;
  for (int k = 0; k < m; ++k) {
    const double t = (k - half) / half;
    double p[kBasis];
    p[0] = 1.0;
    p[1] = t;
    for (int j = 1; j + 1 < kBasis; ++j) p[j + 1] = 2.0 * t * p[j] - p[j - 1];
    for (int a = 0; a < kBasis; ++a)
      for (int b = 0; b < kBasis; ++b) G[a][b] += p[a] * p[b];
  }
  for (int a = 0; a < kBasis; ++a) G[a][kBasis + a] = 1.0;
  for (int col = 0; col < kBasis; ++col) {
    int piv = col;
    for (int r = col + 1; r < kBasis; ++r)
      if (std::fabs(G[r][col]) > std::fabs(G[piv][col])) piv = r;
    for (int c = 0; c < 2 * kBasis; ++c) std::swap(G[col][c], G[piv][c]);
    const double d = G[col][col];
    for (int c = 0; c < 2 * kBasis; ++c) G[col][c] /= d;
    for (int r = 0; r < kBasis; ++r) {
      if (r == col) continue;
      const double f = G[r][col];
      for (int c = 0; c < 2 * kBasis; ++c) G[r][c] -= f * G[col][c];
    }
  }
  BasisGram out;
  for (int a = 0; a < kBasis; ++a)
    for (int b = 0; b < kBasis; ++b) out.ginv[a * kBasis + b] = (float)G[a][kBasis + b];
  return out;
}
}  // namespace

int launch_filter_toeplitz(fbp_context* ctx, const RowSet& rs, int n, int filter) {
  const int m = rs.m;
  if (!toeplitz_supported(m)) return set_error(ctx, FBP_ERR_UNSUPPORTED, "Toeplitz filter needs 64 <= width <= 8192");
  if (rs.rows == 0) return FBP_OK;
  const int kp = (m + BK - 1) / BK * BK;  // K padded to whole blocks (16-byte pitch too)
  const int kx = kp + BK;                  // and one block for the row baseline
  ToeplitzTables& t = ctx->ttab;
  if (!(t.m == m && t.n == n && t.filter == filter)) {
    t.m = 0;
    const size_t bytes = sizeof(__nv_bfloat16) * (size_t)m * kx;
    const size_t need = 2 * bytes + sizeof(float) * kBasis * m;
    if (need > t.cap) {  // grow only
      cudaFree(t.th);
      t.th = nullptr;
      t.cap = 0;
      if (cuda_check(ctx, device_alloc(ctx, &t.th, need), "cudaMalloc(Toeplitz operands)")) return FBP_ERR_OUT_OF_MEMORY;
      t.cap = need;
    }
    if (int rc = ensure_filter_tables(ctx, n, filter)) return rc;
    float* tp = reinterpret_cast<float*>(static_cast<unsigned char*>(t.th) + 2 * bytes);
    toeplitz_basis_kernel<<<(m + 3) / 4, 128, 0, ctx->stream>>>(ctx->ftab.kernel, n, m, tp);
    if (int rc = launched(ctx, "toeplitz_basis_kernel")) return rc;
    build_toeplitz_kernel<<<ctx->num_sms * 8, 256, 0, ctx->stream>>>(ctx->ftab.kernel, n, m, kp, kx, tp,
                                                                     (__nv_bfloat16*)t.th,
                                                                     (__nv_bfloat16*)t.th + (size_t)m * kx);
    if (int rc = launched(ctx, "build_toeplitz_kernel")) return rc;
    t.m = m;
    t.n = n;
    t.filter = filter;
  }
  // Rows in chunks of whole waves of tiles whose split operands (at most 96 MB,
  // and 256 KB per padded sample) stay in the L2 cache between the two kernels
  const long long wave = (long long)ctx->num_sms * BM;
  const long long cap = std::min((96LL << 20), 65536LL * 4 * (kp + 64)) / (4LL * kx);
  long long rows = cap / wave * wave;
  if (rows == 0) {  // long rows: the row tiles of whole waves of 256-wide tiles
    const long long nt = (m + BN - 1) / BN, w = cap / BM * nt / ctx->num_sms;
    rows = std::max(w > 0 ? w * ctx->num_sms / nt : cap / BM, 1LL) * BM;
  }
  const long long chunk = std::min<long long>(rs.rows, rows);
  const size_t sbytes = sizeof(__nv_bfloat16) * (size_t)chunk * kx;
  unsigned char* sp = static_cast<unsigned char*>(scratch(ctx, 2 * sbytes + 1024));
  if (!sp) return FBP_ERR_OUT_OF_MEMORY;
  __nv_bfloat16* xh = reinterpret_cast<__nv_bfloat16*>(sp);
  __nv_bfloat16* xl = reinterpret_cast<__nv_bfloat16*>(sp + sbytes);
  BasisGram gram;
  if (t.gm != m) {
    gram = basis_gram(m);
    std::copy(gram.ginv, gram.ginv + kBasis * kBasis, t.ginv);
    t.gm = m;
  } else {
    std::copy(t.ginv, t.ginv + kBasis * kBasis, gram.ginv);
  }
  // Four rows a warp up to 640 samples, where the staged rows leave 20 warps a
  // SM, two beyond, fewer where that leaves SMs without 16 warps; past 2048
  // samples the rows are read twice instead.
  const bool stage = kp <= 2048;
  const long long per_sm = chunk / (16LL * ctx->num_sms);
  const int R = kp <= 640 && per_sm >= 4 ? 4 : per_sm >= 2 ? 2 : 1;
  auto* split = R == 4   ? split_rows_kernel<4, true>
                : R == 2 ? (stage ? split_rows_kernel<2, true> : split_rows_kernel<2, false>)
                         : (stage ? split_rows_kernel<1, true> : split_rows_kernel<1, false>);
  // the attribute is process-wide and other contexts launch with other row
  // lengths: always the largest staged size
  const size_t split_cap = R == 4 ? split_smem(4, 640, true) : split_smem(R, 2048, true);
  if (cudaError_t ea = cudaFuncSetAttribute(split, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)split_cap))
    return cuda_check(ctx, ea, "split smem attribute");
  const size_t split_bytes = split_smem(R, kp, stage);
  const int split_rows = kSplitWarps * R;
  const int split_occ = (int)std::max<size_t>(1, std::min<size_t>(8, (size_t)kMaxDynamicSmem / (split_bytes + 1024)));
  // Tile width: the least time of the fullest SM, where a tile takes as long as
  // its operands take from L2 (128 rows of X and its width of T): 256 except
  // where narrower tiles reach more SMs or waste less of the last one
  int bn = BN;
  double best = 1e300;
  for (int w = BN; w >= 128; w -= 64) {
    const int width = std::min(w, (m + 31) / 32 * 32);
    const long long nt = (m + width - 1) / width, tiles = (chunk + BM - 1) / BM * nt;
    const double cost = (double)((tiles + ctx->num_sms - 1) / ctx->num_sms) * (BM + (double)m / nt);
    if (cost < best) best = cost, bn = width;
  }
  const int ntn = (m + bn - 1) / bn;
  CUtensorMap mah, mal, mbh, mbl, mout;
  const uint64_t pitch_b = (uint64_t)kx * 2;
  if (int rc = make_tensor_map_2d_bf16_sw64(ctx, &mah, xh, kx, chunk, pitch_b, BK, BM)) return rc;
  if (int rc = make_tensor_map_2d_bf16_sw64(ctx, &mal, xl, kx, chunk, pitch_b, BK, BM)) return rc;
  __nv_bfloat16* th = (__nv_bfloat16*)t.th;
  if (int rc = make_tensor_map_2d_bf16_sw64(ctx, &mbh, th, kx, m, pitch_b, BK, bn)) return rc;
  if (int rc = make_tensor_map_2d_bf16_sw64(ctx, &mbl, th + (size_t)m * kx, kx, m, pitch_b, BK, bn)) return rc;
  if (int rc = make_tensor_map_2d_f32_sw128(ctx, &mout, rs.data, m, rs.rows, (uint64_t)rs.pitch * 4, kOutCols, 32))
    return rc;
  constexpr int kFixed = 1024 + 8 * OUT_BYTES + (2 * kMaxStages + 5) * 8 + 64;
  GemmArgs ga;
  ga.m = m;
  ga.ntile_n = ntn;
  ga.bn = bn;
  ga.kblocks = kx / BK;
  ga.stages = std::min(kMaxStages, (kMaxDynamicSmem - kFixed) / stage_bytes(bn));
  ga.err = ctx->d_err;
  // no second CTA on the SM: each takes all of its tensor memory
  cudaError_t e = cudaFuncSetAttribute(toeplitz_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynamicSmem);
  if (e != cudaSuccess) return cuda_check(ctx, e, "toeplitz smem attribute");
  for (long long r0 = 0; r0 < rs.rows; r0 += chunk) {
    const int nr = (int)std::min<long long>(chunk, rs.rows - r0);
    const int sgrid = std::min((nr + split_rows - 1) / split_rows, ctx->num_sms * split_occ);
    split<<<sgrid, 32 * kSplitWarps, split_bytes, ctx->stream>>>(rs, r0, nr, kp, kx, xh, xl, gram);
    if (int rc = launched(ctx, "split_rows_kernel")) return rc;
    ga.row0 = r0;
    ga.nrows = nr;
    ga.tiles = (nr + BM - 1) / BM * ntn;
    toeplitz_gemm_kernel<<<std::min(ga.tiles, ctx->num_sms), kGemmThreads, kMaxDynamicSmem, ctx->stream>>>(
        mah, mal, mbh, mbl, mout, ga);
    if (int rc = launched(ctx, "toeplitz_gemm_kernel")) return rc;
  }
  return FBP_OK;
}

}  // namespace fbp
