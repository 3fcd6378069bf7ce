// Detector-row filtering: FDK cosine weight + ramp-type filter.
//
// Replaces the reference's per-view chain (FBP3D::apply_filter_to_projections,
// Source/FilteredBackProjection/FBP3D.cpp:389-414): load, real->complex blit,
// pad, FFFT::fft (radix-2 over texture rows, FastFourierTransformGPU.cpp:3-52),
// fft_shift, FBP2D::apply_filter (FBP2D.cpp:124-144), inverse shift, inverse
// FFT (conj-FFT-conj-divide, FastFourierTransformGPU.cpp:30-36), blit, store:
// ~45 full-texture passes per view. Here one kernel reads each row once and
// writes it once.
//
// Algorithm: two real rows are packed as the real and imaginary parts of one
// complex row (the filter response H is real and even, so the filtered rows
// come back as the real and imaginary parts). The forward transform is a
// decimation-in-frequency FFT (natural order in, bit-reversed out), the
// spectrum is multiplied by H[bitrev(k)]/n, and the inverse is a
// decimation-in-time FFT (bit-reversed in, natural order out), so no
// bit-reversal permutation is ever executed. Row padding to n samples is the
// reference's (next power of two >= width, FastFourierTransformGPU.cpp:258-262).
//
// The transforms run in registers: a thread holds E = 8 or 16 samples whose
// indices differ in log2(E) index bits and does those radix-2 stages at once
// (constant twiddles inside, one table twiddle per sample after them); the
// row is exchanged through shared memory between such phases only. n = 512 is
// three phases of three bits (two exchanges each way), n = 1024 .. 4096 three
// phases of up to four bits. The samples a thread holds in the last forward
// phase are those of the first inverse phase, and those of the last inverse
// phase are the ones it loaded, so the row is read from and written to memory
// from registers.
//
// The filter response and the spatial kernel are generated on the GPU in
// FP64 from the band-limited ramp kernel (h(0) = 1/4, h(odd k) = -1/(pi k)^2,
// Kak & Slaney eq. 3.61) wrapped onto the n-point circle, times the window.

#include "fbp_internal.h"
#include "fbp_rows.cuh"

#include <cmath>
#include <cstdio>

namespace fbp {
namespace {

__device__ __forceinline__ double ramp_tap(long long k) {
  if (k == 0) return 0.25;
  if ((k & 1) == 0) return 0.0;
  const double pi = 3.14159265358979323846;
  double kk = (double)k;
  return -1.0 / (pi * pi * kk * kk);
}

__device__ __forceinline__ double filter_window(int filter, double f) {
  const double pi = 3.14159265358979323846;
  switch (filter) {
    case FBP_FILTER_SHEPP_LOGAN:
      return f == 0.0 ? 1.0 : sin(pi * f) / (pi * f);
    case FBP_FILTER_COSINE:
      return cospi(f);
    case FBP_FILTER_HANN:
      return 0.5 * (1.0 + cospi(2.0 * f));
    default:
      return 1.0;
  }
}

// Register phases of the n = 2^L transform: E = 2^fft_ebits(L) samples a
// thread; phase k covers the E index bits below the first k E, the last phase
// what is left. E keeps the number of phases (the exchanges) lowest with the
// fewest registers.
__host__ __device__ constexpr int fft_ebits(int L) { return L <= 4 ? L : (L == 7 || L == 12) ? 4 : 3; }
__host__ __device__ constexpr int fft_phases(int L) { return L == 0 ? 1 : (L + fft_ebits(L) - 1) / fft_ebits(L); }
// Lowest index bit of phase k (not the last one) and its first entry in the
// twiddle table: phase k's table is [slot 1 .. E - 1][d < 2^lo].
__host__ __device__ constexpr int fft_lo(int L, int k) { return L - (k + 1) * fft_ebits(L); }
__host__ __device__ constexpr int fft_tw_offset(int L, int k) {
  int o = 0;
  for (int i = 0; i < k; ++i) o += ((1 << fft_ebits(L)) - 1) << fft_lo(L, i);
  return o;
}

// The filter tables are O(n^2) sums of FP64 cosines. One block takes one
// entry; the cosines cos(2 pi p / n) come from a table that the block fills
// (n / 4 + 1 values, the other quadrants by symmetry) instead of one FP64
// cosine and one 64-bit remainder per term: at n = 2048, 1.39 ms before.
constexpr int kTableThreads = 128;

__device__ __forceinline__ void fill_quarter_cos(int n, double* q) {
  for (int i = threadIdx.x; i <= n / 4; i += blockDim.x) q[i] = cospi(2.0 * (double)i / n);
}
__device__ __forceinline__ double quarter_cos(const double* q, int n, unsigned p) {  // cos(2 pi p / n), p taken mod n
  p &= (unsigned)(n - 1);
  if (n < 4) return n == 1 || p == 0 ? 1.0 : -1.0;
  const unsigned h = p <= (unsigned)n / 2 ? p : n - p;  // cos is even about n / 2
  return h <= (unsigned)n / 4 ? q[h] : -q[n / 2 - h];
}
__device__ __forceinline__ double block_sum(double v) {
  __shared__ double part[kTableThreads / 32];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  v = 0.0;
  for (int i = 0; i < kTableThreads / 32; ++i) v += part[i];
  return v;
}

// H[k], FP64: the transform of the wrapped band-limited ramp times the window.
__global__ void __launch_bounds__(kTableThreads) response_kernel(int n, int filter, double* H) {
  extern __shared__ double quarter[];
  if (filter != FBP_FILTER_RAMP_SAMPLED) fill_quarter_cos(n, quarter);
  __syncthreads();
  for (int k = blockIdx.x; k <= n / 2; k += gridDim.x) {
    const double f = (double)k / n;
    double h = f;
    if (filter != FBP_FILTER_RAMP_SAMPLED) {
      // odd taps j and n - j are equal and share their cosine
      double s = 0.0;
      for (int j = 1 + 2 * (int)threadIdx.x; j < n; j += 2 * kTableThreads)
        s += ramp_tap(j <= n / 2 ? j : n - j) * quarter_cos(quarter, n, (unsigned)j * (unsigned)k);
      h = (0.25 + block_sum(s)) * filter_window(filter, f);  // j = 0 term 1/4 (cos 0 = 1)
    }
    if (threadIdx.x == 0) {
      H[k] = h;
      if (k > 0 && k < n - k) H[n - k] = h;  // even
    }
  }
}

// From H: hbr (bit-reversed, divided by n), the phases' twiddles and (kernel
// != nullptr) the spatial kernel g.
__global__ void __launch_bounds__(kTableThreads) tables_kernel(int n, int log2n, const double* H, float* hbr,
                                                               float2* tws, float* g) {
  extern __shared__ double quarter[];
  if (g) fill_quarter_cos(n, quarter);
  __syncthreads();
  const int stride = gridDim.x * blockDim.x;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += stride) {
    const unsigned r = log2n > 0 ? __brev((unsigned)k) >> (32 - log2n) : 0u;  // n = 1: the one sample
    hbr[k] = (float)(H[r] / n);
  }
  const int e = fft_ebits(log2n);
  for (int k = 0; k + 1 < fft_phases(log2n); ++k) {
    const int lo = fft_lo(log2n, k), off = fft_tw_offset(log2n, k);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ((1 << e) - 1) << lo; i += stride) {
      const int slot = (i >> lo) + 1, d = i & ((1 << lo) - 1);
      double s, c;  // exp(-2 pi i bitrev(slot) d / 2^(lo + e))
      sincospi(-2.0 * (double)((__brev((unsigned)slot) >> (32 - e)) * (unsigned)d) / (double)(1 << (lo + e)), &s, &c);
      tws[off + i] = make_float2((float)c, (float)s);
    }
  }
  if (!g) return;
  for (int k = blockIdx.x; k <= n / 2; k += gridDim.x) {
    double acc = 0.0;
    for (int j = threadIdx.x; j < n; j += kTableThreads)
      acc += H[j] * quarter_cos(quarter, n, (unsigned)j * (unsigned)k);
    acc = block_sum(acc);
    if (threadIdx.x == 0) {
      g[k] = (float)(acc / n);
      if (k > 0 && k < n - k) g[n - k] = (float)(acc / n);  // even
    }
  }
}

__global__ void twiddle_kernel(int n, float2* tw) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n / 2) return;
  double s, c;
  sincospi(-2.0 * (double)k / n, &s, &c);
  tw[k] = make_float2((float)c, (float)s);
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cmulc(float2 a, float2 b) {  // a * conj(b)
  return make_float2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}

struct FilterKArgs {
  RowSet rs;
  long long npairs;
  const float2* tws;
  const float* hbr;
};

__device__ __forceinline__ float2 cadd(float2 a, float2 b) {
  float2 d;
  asm("{\n .reg .b64 x, y, z;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n add.rn.f32x2 z, x, y;\n mov.b64 {%0, %1}, z;\n}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 csub(float2 a, float2 b) {
  float2 d;
  asm("{\n .reg .b64 x, y, z;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n sub.rn.f32x2 z, x, y;\n mov.b64 {%0, %1}, z;\n}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}

// a exp(-2 pi i j / 16) (CONJ: its conjugate), j < 8 a constant after unrolling
template <bool CONJ>
__device__ __forceinline__ float2 rot16(float2 a, int j) {
  constexpr float c1 = 0.92387953251128675613f, c2 = 0.70710678118654752440f, c3 = 0.38268343236508977173f;
  if (j == 0) return a;
  if (j == 4) return CONJ ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
  const float c[8] = {1.f, c1, c2, c3, 0.f, -c3, -c2, -c1};
  const float s[8] = {0.f, c3, c2, c1, 1.f, c1, c2, c3};
  const float2 w = make_float2(c[j], -s[j]);
  return CONJ ? cmulc(a, w) : cmul(a, w);
}

// Radix-2 stages over the low Q bits of the register index, decimation in
// frequency (highest bit first) and its inverse.
template <int E, int Q>
__device__ __forceinline__ void dif_regs(float2 (&x)[E]) {
#pragma unroll
  for (int b = Q - 1; b >= 0; --b)
#pragma unroll
    for (int i = 0; i < E; ++i)
      if (!(i >> b & 1)) {
        const float2 u = x[i], v = x[i + (1 << b)];
        x[i] = cadd(u, v);
        x[i + (1 << b)] = rot16<false>(csub(u, v), (i & ((1 << b) - 1)) << (3 - b));
      }
}
template <int E, int Q>
__device__ __forceinline__ void dit_regs(float2 (&x)[E]) {
#pragma unroll
  for (int b = 0; b < Q; ++b)
#pragma unroll
    for (int i = 0; i < E; ++i)
      if (!(i >> b & 1)) {
        const float2 u = x[i], v = rot16<true>(x[i + (1 << b)], (i & ((1 << b) - 1)) << (3 - b));
        x[i] = cadd(u, v);
        x[i + (1 << b)] = csub(u, v);
      }
}

// Place of sample p in the exchange buffer (linear over XOR). Half a warp of
// 8-byte accesses is free of bank conflicts when its places differ in the low
// four bits. A phase's threads step through its low lo index bits and then
// from bit lo + log2 E on, the last phase's from bit log2 E on; XORing bits
// 4, 5, 6 (E = 8) or 4 .. 7 (E = 16) into the low four as below makes every
// one of these patterns a permutation of the 16 bank pairs.
template <int L>
__host__ __device__ constexpr int fft_place(int p) {
  return fft_ebits(L) == 3 ? p ^ ((p >> 3) & 14) ^ ((p >> 6) & 1) : p ^ ((p >> 4) & 15);
}

// Element I of the phase's twiddles at w0: volatile, so that the table stays
// in L1 and out of the registers between pairs.
template <int I>
__device__ __forceinline__ float2 load_twiddle(const float2* w0) {
  float2 w;
  asm volatile("ld.global.nc.v2.f32 {%0, %1}, [%2 + %3];" : "=f"(w.x), "=f"(w.y) : "l"(w0), "n"(I * (int)sizeof(float2)));
  return w;
}
// x[i] *= twiddle i (CONJ: its conjugate) for i = 1 .. E - 1
template <int E, int LO, bool CONJ, int I = 1>
__device__ __forceinline__ void twiddle_regs(float2 (&x)[E], const float2* w0) {
  if constexpr (I < E) {
    const float2 w = load_twiddle<((I - 1) << LO)>(w0);
    x[I] = CONJ ? cmulc(x[I], w) : cmul(x[I], w);
    twiddle_regs<E, LO, CONJ, I + 1>(x, w0);
  }
}

// Forward phases K .. and inverse phases K .. 0 around the last one: the
// phase's radix-2 stages and twiddles in registers, then the exchange. Every
// place is written and read by the same thread within a phase, so one barrier
// between the write and the next phase's read orders an exchange.
template <int L, int K, int E, class At, class Sync>
__device__ __forceinline__ void fft_forward(float2 (&x)[E], const float2* tws, int t, At& at, Sync& sync) {
  if constexpr (K + 1 < fft_phases(L)) {
    constexpr int LO = fft_lo(L, K);
    dif_regs<E, fft_ebits(L)>(x);
    twiddle_regs<E, LO, false>(x, tws + fft_tw_offset(L, K) + (t & ((1 << LO) - 1)));
#pragma unroll
    for (int i = 0; i < E; ++i) at(K, i) = x[i];
    sync();
#pragma unroll
    for (int i = 0; i < E; ++i) x[i] = at(K + 1, i);
    fft_forward<L, K + 1>(x, tws, t, at, sync);
  }
}
template <int L, int K, int E, class At, class Sync>
__device__ __forceinline__ void fft_inverse(float2 (&x)[E], const float2* tws, int t, At& at, Sync& sync) {
  if constexpr (K >= 0) {
    constexpr int LO = fft_lo(L, K);
#pragma unroll
    for (int i = 0; i < E; ++i) at(K + 1, i) = x[i];
    sync();
#pragma unroll
    for (int i = 0; i < E; ++i) x[i] = at(K, i);
    twiddle_regs<E, LO, true>(x, tws + fft_tw_offset(L, K) + (t & ((1 << LO) - 1)));
    dit_regs<E, fft_ebits(L)>(x);
    fft_inverse<L, K - 1>(x, tws, t, at, sync);
  }
}

// One group of n / E threads filters a pair of rows at a time, grid-stride
// over the pairs; a block holds as many groups as its size allows. Groups of
// up to a warp synchronise by warp, larger ones through a named barrier each.
//
// Bound: the load / store unit (78-83% busy: exchanges and twiddles). Measured
// with the rows in place, before = radix-4 passes through shared memory with
// block barriers into pairs of rows: 138240 rows of 384 (n = 512) 819 -> 183 us
// (425 MB: 2.3 TB/s), 138240 rows of 768 (n = 1024) 1628 -> 424 us, 92160 rows
// of 1536 (n = 2048) 2288 -> 518 us. Four blocks a SM at 64
// registers spill and are 1-14% slower, E = 16 for n = 1024, 2048 1.4 times
// slower, the twiddles held in registers (one block a SM) 2 times.
template <int L>
__global__ void __launch_bounds__(256, fft_ebits(L) == 4 ? 2 : 3) filter_fft_kernel(const FilterKArgs a) {
  constexpr int EB = fft_ebits(L), E = 1 << EB, N = 1 << L, T = N / E, NP = fft_phases(L);
  constexpr int REM = L - (NP - 1) * EB;  // index bits of the last phase
  extern __shared__ __align__(16) float2 fft_buf[];
  const int grp = threadIdx.x / T, t = threadIdx.x % T;
  const RowSet& rs = a.rs;
  const unsigned mask = T >= 32 ? 0xffffffffu : ((1u << (T & 31)) - 1u) << ((threadIdx.x & 31) / T * T);
  auto sync = [&]() {
    if constexpr (T <= 32) __syncwarp(mask);
    else asm volatile("bar.sync %0, %1;" ::"r"(grp + 1), "r"(T) : "memory");
  };
  float h[E];  // response at this thread's samples of the last phase: E t .. E t + E - 1
#pragma unroll
  for (int i = 0; i < E; ++i) h[i] = a.hbr[E * t + i];
  // Slot i of phase k holds sample (t >> lo << (lo + EB)) | (i << lo) | (t mod
  // 2^lo), of the last phase E t + i; off[k] is slot 0's place in bytes, and
  // the place being linear, slot i's is off[k] ^ place(i << lo).
  uint32_t off[NP];
#pragma unroll
  for (int k = 0; k < NP; ++k) {
    const int lo = k == NP - 1 ? 0 : fft_lo(L, k);
    off[k] = ((uint32_t)grp << (L + 3)) | (uint32_t)(fft_place<L>((t >> lo << (lo + EB)) | (t & ((1 << lo) - 1))) * 8);
  }
  auto at = [&](int k, int i) -> float2& {
    const int lo = k == NP - 1 ? 0 : fft_lo(L, k);
    return *reinterpret_cast<float2*>(reinterpret_cast<char*>(fft_buf) + (off[k] ^ (uint32_t)(fft_place<L>(i << lo) * 8)));
  };
  const int groups = blockDim.x / T;
  for (long long pr = (long long)blockIdx.x * groups + grp; pr < a.npairs; pr += (long long)gridDim.x * groups) {
    const long long r0 = 2 * pr;
    const bool two = r0 + 1 < rs.rows;
    const float* s0 = rs.data + r0 * rs.pitch + t;
    const float* s1 = two ? s0 + rs.pitch : s0;
    const int left = rs.m - t;  // sample t + i T exists for i T < left
    float2 x[E];
#pragma unroll
    for (int i = 0; i < E; ++i) {  // real part row r0, imaginary part row r0 + 1, zero padded
      x[i] = make_float2(0.f, 0.f);
      if (i * T < left) x[i] = make_float2(s0[i * T], two ? s1[i * T] : 0.f);
    }
    if (rs.log_norm) {
#pragma unroll
      for (int i = 0; i < E; ++i)
        if (i * T < left) {
          x[i].x = -logf(fmaxf(x[i].x, 1e-30f * rs.log_base) / rs.log_base);
          if (two) x[i].y = -logf(fmaxf(x[i].y, 1e-30f * rs.log_base) / rs.log_base);
        }
    }
    if (rs.weight) {
      const long long rb = two ? r0 + 1 : r0;
      const int iv0 = rs.sinogram ? (int)(r0 / rs.n_views) : (int)(r0 % rs.n_v);
      const int iv1 = rs.sinogram ? (int)(rb / rs.n_views) : (int)(rb % rs.n_v);
      const float v0 = (iv0 + 0.5f - 0.5f * rs.n_v + rs.w_voff) * rs.w_dv;
      const float v1 = (iv1 + 0.5f - 0.5f * rs.n_v + rs.w_voff) * rs.w_dv;
#pragma unroll
      for (int i = 0; i < E; ++i) {
        const float u = (t + i * T + 0.5f - 0.5f * rs.m) * rs.w_du;
        const float uu = rs.w_sdd * rs.w_sdd + u * u;
        x[i].x *= rs.w_sdd * rsqrtf(uu + v0 * v0);
        x[i].y *= rs.w_sdd * rsqrtf(uu + v1 * v1);
      }
    }
    fft_forward<L, 0>(x, a.tws, t, at, sync);
    dif_regs<E, REM>(x);
#pragma unroll
    for (int i = 0; i < E; ++i) x[i] = make_float2(x[i].x * h[i], x[i].y * h[i]);
    dit_regs<E, REM>(x);
    fft_inverse<L, NP - 2>(x, a.tws, t, at, sync);
    float* d0 = rs.data + r0 * rs.pitch + t;
#pragma unroll
    for (int i = 0; i < E; ++i) {
      if (i * T >= left) continue;
      d0[i * T] = x[i].x;
      if (two) d0[rs.pitch + i * T] = x[i].y;
    }
  }
}

template <int L>
cudaError_t launch_fft_cfg(const FilterKArgs& a, int num_sms, cudaStream_t stream) {
  constexpr int T = (1 << L) >> fft_ebits(L), MAXG = 256 / T;
  // few pairs: a group a block, so that they spread over the SMs
  int groups = (int)std::max<long long>(1, std::min<long long>(MAXG, a.npairs / num_sms));
  if (T * groups < 32) groups = std::min(MAXG, 32 / T);
  const size_t smem = fft_phases(L) > 1 ? sizeof(float2) * ((size_t)groups << L) : 0;
  const int per_sm = (fft_ebits(L) == 4 ? 2 : 3) * 256 / (T * groups);  // blocks resident (the launch bounds)
  const long long blocks = (a.npairs + groups - 1) / groups;
  filter_fft_kernel<L><<<(unsigned)std::min<long long>(blocks, (long long)num_sms * per_sm), T * groups, smem, stream>>>(a);
  return cudaGetLastError();
}

// The filter kernel of padded length n = 2^log2n, n <= 4096.
cudaError_t launch_fft(const FilterKArgs& a, int log2n, int num_sms, cudaStream_t stream) {
  switch (log2n) {
    case 0: return launch_fft_cfg<0>(a, num_sms, stream);
    case 1: return launch_fft_cfg<1>(a, num_sms, stream);
    case 2: return launch_fft_cfg<2>(a, num_sms, stream);
    case 3: return launch_fft_cfg<3>(a, num_sms, stream);
    case 4: return launch_fft_cfg<4>(a, num_sms, stream);
    case 5: return launch_fft_cfg<5>(a, num_sms, stream);
    case 6: return launch_fft_cfg<6>(a, num_sms, stream);
    case 7: return launch_fft_cfg<7>(a, num_sms, stream);
    case 8: return launch_fft_cfg<8>(a, num_sms, stream);
    case 9: return launch_fft_cfg<9>(a, num_sms, stream);
    case 10: return launch_fft_cfg<10>(a, num_sms, stream);
    case 11: return launch_fft_cfg<11>(a, num_sms, stream);
    case 12: return launch_fft_cfg<12>(a, num_sms, stream);
    default: return cudaErrorInvalidValue;
  }
}

// The filter tables for n: the response and the tables that follow from it
// (g may be nullptr).
cudaError_t launch_tables(int n, int log2n, int filter, double* H, float* hbr, float2* tws, float* g,
                          cudaStream_t stream) {
  const size_t smem = sizeof(double) * (n / 4 + 1);
  const int blocks = std::min(n / 2 + 1, 1024);
  response_kernel<<<blocks, kTableThreads, smem, stream>>>(n, filter, H);
  tables_kernel<<<blocks, kTableThreads, smem, stream>>>(n, log2n, H, hbr, tws, g);
  return cudaGetLastError();
}

__global__ void elementwise_pre_kernel(RowSet rs) {
  long long total = rs.rows * (long long)rs.m;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    long long r = e / rs.m;
    int i = (int)(e - r * rs.m);
    rs.data[r * rs.pitch + i] = load_pre(rs, r, i);
  }
}

// Per-view max |pre-processed sample| (as float bits: non-negative floats
// order like integers). A warp reduces four neighbouring rows at once with
// 16-byte loads, lane 0 folds them into a shared per-view table, and each block
// flushes its table once. Bound by the rows' bytes:
// 360 views of 192 x 192 32 -> 17 us, of 367 x 256 (sinograms) 42 -> 29 us,
// against one row at a time with 4-byte loads and 64-bit divisions.
__global__ void __launch_bounds__(256) view_absmax_kernel(RowSet rs, unsigned* vmax) {
  extern __shared__ unsigned smax[];
  for (int i = threadIdx.x; i < rs.n_views; i += blockDim.x) smax[i] = 0u;
  __syncthreads();
  constexpr int R = 4;
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const bool pre = rs.log_norm || rs.weight;
  for (long long r0 = (blockIdx.x * (long long)warps + (threadIdx.x >> 5)) * R; r0 < rs.rows;
       r0 += (long long)gridDim.x * warps * R) {
    float mx[R];
#pragma unroll
    for (int k = 0; k < R; ++k) mx[k] = 0.f;
    if (pre) {
      for (int k = 0; k < R && r0 + k < rs.rows; ++k) {
        float m = 0.f;
        for (int i = lane; i < rs.m; i += 32) m = fmaxf(m, fabsf(load_pre(rs, r0 + k, i)));
#pragma unroll
        for (int j = 0; j < R; ++j)
          if (j == k) mx[j] = m;
      }
    } else {
      // the row pitch is a multiple of 4: the 16-byte loads stay in the row
      for (int q = lane; 4 * q < rs.m; q += 32) {
        float4 v[R];
#pragma unroll
        for (int k = 0; k < R; ++k)
          v[k] = r0 + k < rs.rows ? reinterpret_cast<const float4*>(rs.data + (r0 + k) * rs.pitch)[q]
                                  : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < R; ++k) {
          if (4 * q + 1 >= rs.m) v[k].y = 0.f;
          if (4 * q + 2 >= rs.m) v[k].z = 0.f;
          if (4 * q + 3 >= rs.m) v[k].w = 0.f;
          mx[k] = fmaxf(fmaxf(mx[k], fmaxf(fabsf(v[k].x), fabsf(v[k].y))), fmaxf(fabsf(v[k].z), fabsf(v[k].w)));
        }
      }
    }
#pragma unroll
    for (int k = 0; k < R; ++k) {
      for (int o = 16; o > 0; o >>= 1) mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], o));
      if (lane == 0 && mx[k] > 0.f) atomicMax(smax + row_view(rs, r0 + k), __float_as_uint(mx[k]));
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < rs.n_views; i += blockDim.x)
    if (smax[i]) atomicMax(vmax + i, smax[i]);
}

// scale = largest power of two with scale * max|value| <= limit (so FP16,
// max 65504, holds every stored value and its neighbour differences).
__global__ void view_scale_kernel(const unsigned* vmax, int nviews, float limit, float* scale, float* inv) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nviews) return;
  const float bound = __uint_as_float(vmax[k]);
  float s = 1.f;
  if (bound > 0.f && isfinite(bound)) {
    int e = (int)floorf(log2f(limit / bound));
    e = max(-100, min(100, e));
    s = ldexpf(1.f, e);
  }
  scale[k] = s;
  inv[k] = 1.f / s;
}

constexpr int kPackRows = 8;  // element rows per block of the quad packers

// f32 rows -> pair16: element (view, e, c) = (row e - 1, row e - row e - 1) * scale.
__global__ void pack_pair16_kernel(const float* src, long long spitch, int m, int n_views, int n_v, bool sinogram,
                                   const float* scale, __half2* out, long long opitch) {
  // grid: x over columns, y over element rows e, z over views
  const int e = blockIdx.y, view = blockIdx.z;
  const long long er = sinogram ? (long long)e * n_views + view : (long long)view * (n_v + 1) + e;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < m; c += gridDim.x * blockDim.x) {
    auto row = [&](int iv) -> long long { return sinogram ? (long long)iv * n_views + view : (long long)view * n_v + iv; };
    const float lo = e >= 1 ? src[row(e - 1) * spitch + c] : 0.f;
    const float hi = e < n_v ? src[row(e) * spitch + c] : 0.f;
    const float sc = scale[view];
    // (row e - 1, row e minus row e - 1 as read back): the second value's
    // rounding does not add to the first's (error feedback, as the quads)
    const __half hl = __float2half_rn(lo * sc);
    const __half hd = __float2half_rn(fmaf(hi, sc, -__half2float(hl)));
    out[er * opitch + c] = __halves2half2(hl, hd);
  }
}

// f32 rows -> quad-interleaved gradient layout: one thread per (group g,
// element row e, element column s), writing the 32 bytes of the four slots
// as two 16-byte plane entries.
//
// Each slot holds a 2x2 neighbourhood (a, b: rows e - 1, e of column c; c',
// d: the same rows of column c + 1) as four FP16 values that the
// backprojector reads back as a_r, a_r + c1, a_r + g0 and a_r + c1 + g0 + g1.
// The differences are taken against the values as they will be read back
// (error feedback): a_r = fp16(a), c1 = fp16(c' - a_r), g0 = fp16(b - a_r),
// g1 = fp16(d - (a_r + c1 + g0)). Only a carries a's own rounding error, and
// a bilinear tap weights it by (1 - fu)(1 - fv); the other three corners err
// by the rounding of a difference. On ramp-filtered noisy C4-class views
// this halves the per-tap error of independently rounded differences
// (2.4e-4 -> 1.2e-4 relative).
__global__ void pack_quadg16_kernel(const float* src, long long spitch, int m, int n_views, int n_v, bool sinogram,
                                    const float* scale, uint4* out) {
  // grid: x over element columns, y over runs of kPackRows element rows (each
  // row's samples are loaded once and carried to the next row), z over view
  // groups g
  const int Q = n_views >> 2, P = m + 1;
  const int g = blockIdx.z, e0 = blockIdx.y * kPackRows, e1 = min(e0 + kPackRows, n_v + 1);
  float k[4];
#pragma unroll
  for (int slot = 0; slot < 4; ++slot) k[slot] = scale[g + slot * Q];
  for (int sc = blockIdx.x * blockDim.x + threadIdx.x; sc < P; sc += gridDim.x * blockDim.x) {
    const int c = sc - 1;  // element column sc covers columns c, c + 1
    // samples of row iv at columns c, c + 1 for the four slots (zero outside)
    auto load = [&](int iv, float (&lo)[4], float (&hi)[4]) {
#pragma unroll
      for (int slot = 0; slot < 4; ++slot) {
        const int view = g + slot * Q;
        const bool ok = iv >= 0 && iv < n_v;
        const long long r = sinogram ? (long long)iv * n_views + view : (long long)view * n_v + iv;
        lo[slot] = ok && c >= 0 ? src[r * spitch + c] : 0.f;
        hi[slot] = ok && c + 1 < m ? src[r * spitch + c + 1] : 0.f;
      }
    };
    float pa[4], pc[4], pb[4], pd[4];
    load(e0 - 1, pa, pc);
    for (int e = e0; e < e1; ++e) {
      load(e, pb, pd);
      uint32_t w[8];
#pragma unroll
      for (int slot = 0; slot < 4; ++slot) {
        const float kk = k[slot];
        const __half ha = __float2half_rn(pa[slot] * kk);
        const float ar = __half2float(ha);
        const __half hc1 = __float2half_rn(fmaf(pc[slot], kk, -ar));
        const __half hg0 = __float2half_rn(fmaf(pb[slot], kk, -ar));
        const float c1 = __half2float(hc1), g0 = __half2float(hg0);
        const __half hg1 = __float2half_rn(fmaf(pd[slot], kk, -((ar + c1) + g0)));
        const __half2 x1 = __halves2half2(ha, hg0);   // (a_r, g0): the row e - 1 value and the row step
        const __half2 x2 = __halves2half2(hc1, hg1);  // (c1, g1): their steps along u
        w[2 * slot] = *reinterpret_cast<const uint32_t*>(&x1);
        w[2 * slot + 1] = *reinterpret_cast<const uint32_t*>(&x2);
        pa[slot] = pb[slot];
        pc[slot] = pd[slot];
      }
      // two planes per element row: slots 0, 1 then slots 2, 3, 16 bytes per column each
      const long long ge = (long long)g * (n_v + 1) + e;
      out[(2 * ge) * P + sc] = make_uint4(w[0], w[1], w[2], w[3]);
      out[(2 * ge + 1) * P + sc] = make_uint4(w[4], w[5], w[6], w[7]);
    }
  }
}

// 24-bit store of an FP32 value for kLayoutQuadG24: the top three bytes S of
// a stored value are read back as the float with bits (S << 8) | (S & 0xff).
// That map is monotonic in S; with D the last byte of x less the one before it,
// the truncation x >> 8 reads back D below x, the next S 257 - D above and the
// one before 257 + D below: the nearest is one further where |D| > 128. The
// sign is carried along (bits past 24 are dropped by the packing).
__device__ __forceinline__ uint32_t store24(float x) {
  const uint32_t b = __float_as_uint(x), t = b >> 8;
  const int D = (int)(b & 0xffu) - (int)(t & 0xffu);
  return t + (D > 128 ? 1u : 0u) - (D < -128 ? 1u : 0u);
}

// f32 rows -> kLayoutQuadG24: one thread per (group g, element row e, element
// column s); the 16 values (slot-major: a, b - a, c' - a, d - c' - b + a) are
// stored as 3-byte little-endian fields of 12 words, written as three
// 16-byte plane entries. 4 bytes read and 12 written per sample;
// with the nearest of three candidates searched for and the fields shifted into
// place it was bound by its instructions (720 views of 768 x 768: 2.92 ms, now
// 1.31; the bytes take 1.04).
__global__ void pack_quadg24_kernel(const float* src, long long spitch, int m, int n_views, int n_v, bool sinogram,
                                    uint4* out) {
  // grid: x over element columns, y over runs of kPackRows element rows, z
  // over view groups g (as pack_quadg16_kernel)
  const int Q = n_views >> 2, P = m + 1;
  const int g = blockIdx.z, e0 = blockIdx.y * kPackRows, e1 = min(e0 + kPackRows, n_v + 1);
  for (int sc = blockIdx.x * blockDim.x + threadIdx.x; sc < P; sc += gridDim.x * blockDim.x) {
    const int c = sc - 1;
    auto load = [&](int iv, float (&lo)[4], float (&hi)[4]) {
#pragma unroll
      for (int slot = 0; slot < 4; ++slot) {
        const int view = g + slot * Q;
        const bool ok = iv >= 0 && iv < n_v;
        const long long r = sinogram ? (long long)iv * n_views + view : (long long)view * n_v + iv;
        lo[slot] = ok && c >= 0 ? src[r * spitch + c] : 0.f;
        hi[slot] = ok && c + 1 < m ? src[r * spitch + c + 1] : 0.f;
      }
    };
    float pa[4], pc[4], pb[4], pd[4];
    load(e0 - 1, pa, pc);
    for (int e = e0; e < e1; ++e) {
      load(e, pb, pd);
      uint32_t w[12];
#pragma unroll
      for (int slot = 0; slot < 4; ++slot) {
        const uint32_t v0 = store24(pa[slot]), v1 = store24(pb[slot] - pa[slot]), v2 = store24(pc[slot] - pa[slot]),
                       v3 = store24((pd[slot] - pc[slot]) - (pb[slot] - pa[slot]));
        w[3 * slot] = __byte_perm(v0, v1, 0x4210);
        w[3 * slot + 1] = __byte_perm(v1, v2, 0x5421);
        w[3 * slot + 2] = __byte_perm(v2, v3, 0x6542);
        pa[slot] = pb[slot];
        pc[slot] = pd[slot];
      }
      const long long ge = (long long)g * (n_v + 1) + e;
      out[(3 * ge) * P + sc] = make_uint4(w[0], w[1], w[2], w[3]);
      out[(3 * ge + 1) * P + sc] = make_uint4(w[4], w[5], w[6], w[7]);
      out[(3 * ge + 2) * P + sc] = make_uint4(w[8], w[9], w[10], w[11]);
    }
  }
}

// f32 rows -> the orbits' layouts: the slots' samples of one detector pixel
// (FP32), or its FP16 row pair (row e - 1, row e minus it as read back: the
// values of pack_pair16_kernel), as one element. Grid: x over element columns,
// y over runs of kPackRows element rows, z over groups. Bound by its bytes
// (FP32: 4 read and 4 written per sample and slot): with a row a thread, and each
// row of the pairs read twice, 178 us for 360 views of 367 x 256 as FP16 row
// pairs and their mirror images; eight rows in flight, 78 us (the bytes: 62).
template <int SLOTS, bool P16>
__global__ void __launch_bounds__(256) pack_orbit_kernel(const float* __restrict__ src, long long spitch, int m,
                                                         int n_views, int n_v, bool sinogram, int groups, int mirror,
                                                         const float* __restrict__ scale, long long pitch,
                                                         float* __restrict__ out) {
  const int g = blockIdx.z, c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= pitch) return;
  const int rows = n_v + (P16 ? 1 : 0);
  const long long step = sinogram ? (long long)n_views * spitch : spitch;
  const float* base[SLOTS];  // row 0 of the slot's view, at its column
  float sc[SLOTS];
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) {
    // slots past `mirror` views are the first ones' mirror images
    const int view = g + (s < mirror ? s : s - mirror) * groups, col = s < mirror ? c : m - 1 - c;
    base[s] = src + (sinogram ? (long long)view : (long long)view * n_v) * spitch + col;
    sc[s] = P16 ? scale[view] : 1.f;
  }
  for (int e0 = blockIdx.y * kPackRows; e0 < rows; e0 += gridDim.y * kPackRows) {
    // the run's rows, the one before it first where a row pair wants it
    constexpr int N = kPackRows + (P16 ? 1 : 0);
    float x[SLOTS][N];
#pragma unroll
    for (int s = 0; s < SLOTS; ++s)
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const int iv = e0 + i - (P16 ? 1 : 0);
        x[s][i] = c < m && iv >= 0 && iv < n_v ? __ldg(base[s] + iv * step) : 0.f;
      }
    float* o = out + (((long long)g * rows + e0) * pitch + c) * SLOTS;
#pragma unroll
    for (int i = 0; i < kPackRows; ++i) {
      if (e0 + i < rows) {
        float v[SLOTS];
#pragma unroll
        for (int s = 0; s < SLOTS; ++s) {
          if constexpr (P16) {
            const __half hl = __float2half_rn(x[s][i] * sc[s]);
            const __half2 h = __halves2half2(hl, __float2half_rn(fmaf(x[s][i + 1], sc[s], -__half2float(hl))));
            v[s] = *reinterpret_cast<const float*>(&h);
          } else {
            v[s] = x[s][i];
          }
        }
        if constexpr (SLOTS == 4) *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
        else *reinterpret_cast<float2*>(o) = make_float2(v[0], v[1]);
      }
      o += pitch * SLOTS;
    }
  }
}

// Natural-order complex FFT of rows (FFFT::fft_radix2 / inverse_fft_radix2,
// FastFourierTransformGPU.cpp:3-36): inverse = conj, FFT, conj, divide by n.
__global__ void __launch_bounds__(256) fft_rows_kernel(float2* data, int n, int log2n, int rows,
                                                       int inverse, const float2* twg) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int half = n >> 1;
  float2* tw = reinterpret_cast<float2*>(smem_raw);
  float2* buf = tw + half;
  for (int i = threadIdx.x; i < half; i += blockDim.x) tw[i] = twg[i];
  for (int r = blockIdx.x; r < rows; r += gridDim.x) {
    __syncthreads();
    float2* row = data + (long long)r * n;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      float2 x = row[i];
      if (inverse) x.y = -x.y;
      buf[i] = x;
    }
    __syncthreads();
    for (int lh = log2n - 1; lh >= 0; --lh) {
      const int h = 1 << lh, tsh = log2n - 1 - lh;
      for (int q = threadIdx.x; q < half; q += blockDim.x) {
        int j = q & (h - 1), blk = q >> lh;
        float2* d = buf + (blk << (lh + 1)) + j;
        float2 x0 = d[0], x1 = d[h];
        d[0] = make_float2(x0.x + x1.x, x0.y + x1.y);
        d[h] = cmul(make_float2(x0.x - x1.x, x0.y - x1.y), tw[j << tsh]);
      }
      __syncthreads();
    }
    const float sc = inverse ? 1.f / n : 1.f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      unsigned br = __brev((unsigned)i) >> (32 - log2n);
      float2 x = buf[br];
      if (inverse) x = make_float2(x.x * sc, -x.y * sc);
      row[i] = x;
    }
  }
}

// out[(i + s) mod n] = in[i] per row (FFFT::fft_shift, FastFourierTransformGPU.cpp:93-142).
__global__ void fft_shift_kernel(float2* data, int n, int rows, int shift) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* buf = reinterpret_cast<float2*>(smem_raw);
  for (int r = blockIdx.x; r < rows; r += gridDim.x) {
    __syncthreads();
    float2* row = data + (long long)r * n;
    for (int i = threadIdx.x; i < n; i += blockDim.x) buf[i] = row[i];
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      int j = (int)((((long long)i + shift) % n + n) % n);
      row[j] = buf[i];
    }
  }
}

int ilog2(int n) {
  int l = 0;
  while ((1 << l) < n) l++;
  return l;
}

int grid_for(fbp_context* ctx, long long work, int per_block) {
  long long b = (work + per_block - 1) / per_block;
  long long cap = (long long)ctx->num_sms * 16;
  return (int)std::max(1LL, std::min(b, cap));
}

}  // namespace

int ensure_filter_tables(fbp_context* ctx, int n, int filter) {
  FilterTables& t = ctx->ftab;
  if (t.n == n && t.filter == filter) return FBP_OK;
  if (n < 1 || (n & (n - 1)) || n > 8192)
    return set_error(ctx, FBP_ERR_INVALID_ARGUMENT, "filter length must be a power of two in [1, 8192]");
  if (filter < 0 || filter > FBP_FILTER_RAMP_SAMPLED)
    return set_error(ctx, FBP_ERR_INVALID_ARGUMENT, "unknown filter type");
  if (n > t.cap) {  // grow only: a context serving many row lengths stops allocating
    cudaFree(t.tws);
    cudaFree(t.hbr);
    cudaFree(t.kernel);
    t.tws = nullptr;
    t.hbr = nullptr;
    t.kernel = nullptr;
    t.n = 0;
    t.cap = 0;
    // at most (E - 1) / E n entries for the first phase and 1 / E of that for each further one
    if (cuda_check(ctx, cudaMalloc(&t.tws, sizeof(float2) * (n + 8)), "cudaMalloc(twiddles)") ||
        cuda_check(ctx, cudaMalloc(&t.hbr, sizeof(float) * n), "cudaMalloc(hbr)") ||
        cuda_check(ctx, cudaMalloc(&t.kernel, sizeof(float) * n), "cudaMalloc(kernel)"))
      return FBP_ERR_OUT_OF_MEMORY;
    t.cap = n;
  }
  double* H = static_cast<double*>(scratch(ctx, sizeof(double) * n));
  if (!H) return FBP_ERR_OUT_OF_MEMORY;
  if (int rc = cuda_check(ctx, launch_tables(n, ilog2(n), filter, H, t.hbr, t.tws, t.kernel, ctx->stream),
                          "filter tables"))
    return rc;
  ctx->launches += 2;
  t.n = n;
  t.filter = filter;
  return FBP_OK;
}

int launch_filter_fft(fbp_context* ctx, const RowSet& rs, int n) {
  if (n < rs.m) return set_error(ctx, FBP_ERR_INVALID_ARGUMENT, "padded length smaller than the row");
  if (n > 4096) return set_error(ctx, FBP_ERR_UNSUPPORTED, "FFT filter supports padded lengths up to 4096");
  if (rs.rows == 0) return FBP_OK;
  FilterKArgs a;
  a.rs = rs;
  a.npairs = (rs.rows + 1) / 2;
  a.tws = ctx->ftab.tws;
  a.hbr = ctx->ftab.hbr;
  if (int rc = cuda_check(ctx, launch_fft(a, ilog2(n), ctx->num_sms, ctx->stream), "filter_fft_kernel")) return rc;
  ctx->launches++;
  return FBP_OK;
}

int launch_elementwise_pre(fbp_context* ctx, const RowSet& rs) {
  if (rs.rows == 0) return FBP_OK;
  elementwise_pre_kernel<<<grid_for(ctx, rs.rows * rs.m, 256), 256, 0, ctx->stream>>>(rs);
  return launched(ctx, "elementwise_pre_kernel");
}

int launch_view_scales(fbp_context* ctx, const RowSet& rs, float limit, float* view_scale, float* inv_scale) {
  if (rs.n_views > 16384) return set_error(ctx, FBP_ERR_UNSUPPORTED, "at most 16384 views in MIXED precision");
  unsigned* vmax = static_cast<unsigned*>(scratch(ctx, sizeof(unsigned) * rs.n_views + 64));
  if (!vmax) return FBP_ERR_OUT_OF_MEMORY;
  if (int rc = cuda_check(ctx, cudaMemsetAsync(vmax, 0, sizeof(unsigned) * rs.n_views, ctx->stream), "memset"))
    return rc;
  const int blocks = (int)std::max(1LL, std::min<long long>((rs.rows + 31) / 32, (long long)ctx->num_sms * 4));
  const size_t sm = sizeof(unsigned) * rs.n_views;
  cudaFuncSetAttribute(view_absmax_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
  view_absmax_kernel<<<blocks, 256, sm, ctx->stream>>>(rs, vmax);
  view_scale_kernel<<<(rs.n_views + 127) / 128, 128, 0, ctx->stream>>>(vmax, rs.n_views, limit, view_scale, inv_scale);
  ctx->launches += 1;  // two launches above
  return launched(ctx, "view scale kernels");
}

int launch_pack(fbp_context* ctx, const Stack& s, int layout, const Orbits& o, void* out, long long pitch,
                const float* view_scale) {
  if (layout == kLayoutPair16) {
    if (s.v + 1 > 65535 || s.n > 65535)
      return set_error(ctx, FBP_ERR_UNSUPPORTED, "the pair layout takes up to 65534 rows and 65535 views");
    const dim3 grid((s.u + 255) / 256, s.v + 1, s.n);
    pack_pair16_kernel<<<grid, 256, 0, ctx->stream>>>(s.f32, s.pitch, s.u, s.n, s.v, s.sinogram, view_scale,
                                                      static_cast<__half2*>(out), pitch);
    return launched(ctx, "pack_pair16_kernel");
  }
  if (layout == kLayoutQuadG16) {
    if (s.n % 4) return set_error(ctx, FBP_ERR_UNSUPPORTED, "the interleaved layout needs a multiple of 4 views");
    if (s.v + 1 > 65535 || s.n / 4 > 65535)
      return set_error(ctx, FBP_ERR_UNSUPPORTED, "the interleaved layout takes up to 65534 rows and 262140 views");
    const dim3 grid((s.u + 1 + 255) / 256, (s.v + 1 + kPackRows - 1) / kPackRows, s.n / 4);
    pack_quadg16_kernel<<<grid, 256, 0, ctx->stream>>>(s.f32, s.pitch, s.u, s.n, s.v, s.sinogram, view_scale,
                                                       static_cast<uint4*>(out));
    return launched(ctx, "pack_quadg16_kernel");
  }
  if (layout == kLayoutQuadG24) {
    if (s.n % 4) return set_error(ctx, FBP_ERR_UNSUPPORTED, "the interleaved layout needs a multiple of 4 views");
    if (s.v + 1 > 65535 || s.n / 4 > 65535)
      return set_error(ctx, FBP_ERR_UNSUPPORTED, "the interleaved layout takes up to 65534 rows and 262140 views");
    const dim3 grid((s.u + 1 + 255) / 256, (s.v + 1 + kPackRows - 1) / kPackRows, s.n / 4);
    pack_quadg24_kernel<<<grid, 256, 0, ctx->stream>>>(s.f32, s.pitch, s.u, s.n, s.v, s.sinogram,
                                                       static_cast<uint4*>(out));
    return launched(ctx, "pack_quadg24_kernel");
  }
  if (is_quad_layout(layout) && !is_grad_layout(layout)) {
    if (o.groups > 65535) return set_error(ctx, FBP_ERR_UNSUPPORTED, "interleaved views take up to 65535 view groups");
    const int rows = s.v + (is_pair_layout(layout) ? 1 : 0);
    const dim3 grid((unsigned)((pitch + 255) / 256), std::min((rows + kPackRows - 1) / kPackRows, 65535), o.groups);
    auto kern = layout == kLayoutQuad32    ? pack_orbit_kernel<4, false>
                : layout == kLayoutDuo32   ? pack_orbit_kernel<2, false>
                : layout == kLayoutQuadP16 ? pack_orbit_kernel<4, true>
                                           : pack_orbit_kernel<2, true>;
    kern<<<grid, 256, 0, ctx->stream>>>(s.f32, s.pitch, s.u, s.n, s.v, s.sinogram, o.groups, o.mirror, view_scale, pitch,
                                        static_cast<float*>(out));
    return launched(ctx, "pack_orbit_kernel");
  }
  return set_error(ctx, FBP_ERR_INVALID_ARGUMENT, "unknown packed layout");
}

int launch_fft_rows(fbp_context* ctx, float2* data, int n, int rows, int inverse) {
  if (n < 2 || (n & (n - 1)) || n > 8192)
    return set_error(ctx, FBP_ERR_INVALID_ARGUMENT, "FFT length must be a power of two in [2, 8192]");
  if (rows <= 0) return FBP_OK;
  // twiddles for n (independent of the filter tables' n)
  float2* tw = static_cast<float2*>(scratch(ctx, sizeof(float2) * (n / 2)));
  if (!tw) return FBP_ERR_OUT_OF_MEMORY;
  twiddle_kernel<<<(n / 2 + 127) / 128, 128, 0, ctx->stream>>>(n, tw);
  size_t smem = sizeof(float2) * (n / 2 + n);
  cudaFuncSetAttribute(fft_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);
  fft_rows_kernel<<<std::min(rows, ctx->num_sms * 4), 256, smem, ctx->stream>>>(data, n, ilog2(n), rows, inverse,
                                                                                 tw);
  ctx->launches += 1;  // twiddle_kernel
  return launched(ctx, "fft_rows_kernel");
}

int launch_fft_shift_rows(fbp_context* ctx, float2* data, int n, int rows, int shift) {
  if (n <= 0 || n > 8192) return set_error(ctx, FBP_ERR_INVALID_ARGUMENT, "row length must be in [1, 8192]");
  if (rows <= 0) return FBP_OK;
  cudaFuncSetAttribute(fft_shift_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);
  fft_shift_kernel<<<std::min(rows, ctx->num_sms * 4), 256, sizeof(float2) * n, ctx->stream>>>(data, n, rows,
                                                                                                shift);
  return launched(ctx, "fft_shift_kernel");
}

}  // namespace fbp

// ---------------------------------------------------------------------------
// Allocation-free variant of fbp2d_filter_sinogram.
//
// Some callers cannot allocate device memory while they run: hosts that hand
// out all GPU memory from their own pool at start-up, real-time acquisition
// loops where a cudaMalloc / cudaFree would synchronise the device and stall
// the detector read-out, and plugins whose host forbids allocations after
// initialisation. This entry point needs no context and allocates nothing:
// the filter tables it generates (FP64 response, twiddles, bit-reversed
// response) live in the file-scope array below, which every GPU that loads
// the library holds until the process exits.
//
// Capacity: padded row lengths up to kNoAllocMaxN = 4096 samples (rows up to
// 4096 bins with the default padding). The array is shared by all calls on a
// device and keeps the last call's tables; each call rewrites every table
// entry it reads before reading it, so nothing needs clearing. Calls whose
// work overlaps on the GPU (other streams, other host threads) race on the
// array and must be serialised by the caller.

namespace {
constexpr int kNoAllocMaxN = 4096;
constexpr size_t kNoAllocH = 0;                                           // double[4096]
constexpr size_t kNoAllocTw = kNoAllocH + sizeof(double) * kNoAllocMaxN;  // float2[4096]
constexpr size_t kNoAllocHbr = kNoAllocTw + sizeof(float2) * kNoAllocMaxN;  // float[4096]
constexpr size_t kNoAllocBytes = kNoAllocHbr + sizeof(float) * kNoAllocMaxN;  // 80 KiB
}  // namespace

static __device__ __align__(256) unsigned char fbp_noalloc_filter_scratch[kNoAllocBytes];

extern "C" int fbp2d_filter_sinogram_noalloc(float* sinogram, int bins, int views, int filter_type, float fan_sdd,
                                              float detector_width, int padded_length, void* cuda_stream) {
  using namespace fbp;
  if (!sinogram || bins <= 0 || views <= 0)
    return set_error(nullptr, FBP_ERR_INVALID_ARGUMENT, "bad sinogram");
  if (filter_type < 0 || filter_type > FBP_FILTER_RAMP_SAMPLED)
    return set_error(nullptr, FBP_ERR_INVALID_ARGUMENT, "unknown filter type");
  if (fan_sdd > 0.f && !(detector_width > 0.f))
    return set_error(nullptr, FBP_ERR_INVALID_ARGUMENT, "detector width must be positive");
  int n = padded_length;
  if (n <= 0) {  // the reference's rule: next power of two >= bins (1 for one bin)
    int l = 0;
    for (long t = 2L * bins - 1; t > 1; t >>= 1) l++;
    n = l < 31 ? 1 << l : 0;
  }
  if (n < bins || n < 1 || (n & (n - 1)))
    return set_error(nullptr, FBP_ERR_INVALID_ARGUMENT, "padded length must be a power of two >= the row width");
  if (n > kNoAllocMaxN)
    return set_error(nullptr, FBP_ERR_UNSUPPORTED,
                     "padded row length " + std::to_string(n) +
                         " exceeds the 4096-sample maximum of fbp2d_filter_sinogram_noalloc");
  // an error left by the caller's own earlier work would otherwise be read
  // back below and reported as this call's
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess)
    return set_error(nullptr, FBP_ERR_CUDA,
                     std::string("a CUDA error was pending before fbp2d_filter_sinogram_noalloc: ") +
                         cudaGetErrorString(e));
  // Device address of the scratch array in the current device's context (the
  // array's host-side name is not a device address). Looked up on every
  // call: a context torn down and made again (cudaDeviceReset) may load the
  // module elsewhere. The first call on a device loads the module's device
  // code, which is why that call should come before any stream capture.
  void* base = nullptr;
  e = cudaGetSymbolAddress(&base, fbp_noalloc_filter_scratch);
  if (e != cudaSuccess) return cuda_check(nullptr, e, "cudaGetSymbolAddress(filter scratch)");
  unsigned char* b = static_cast<unsigned char*>(base);
  double* H = reinterpret_cast<double*>(b + kNoAllocH);
  float2* tws = reinterpret_cast<float2*>(b + kNoAllocTw);
  float* hbr = reinterpret_cast<float*>(b + kNoAllocHbr);
  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  int dev = 0, sms = 148;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return cuda_check(nullptr, e, "cudaGetDevice");
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
    return cuda_check(nullptr, e, "cudaDeviceGetAttribute(multiprocessor count)");

  if ((e = launch_tables(n, ilog2(n), filter_type, H, hbr, tws, nullptr, stream)) != cudaSuccess)
    return cuda_check(nullptr, e, "fbp2d_filter_sinogram_noalloc: filter tables");

  RowSet rs{};
  rs.data = sinogram;
  rs.pitch = bins;
  rs.rows = views;
  rs.m = bins;
  rs.n_views = views;
  rs.n_v = 1;
  rs.sinogram = false;
  if (fan_sdd > 0.f) {
    rs.weight = true;
    rs.w_sdd = fan_sdd;
    rs.w_du = detector_width / bins;
    rs.w_dv = 0.f;
  }
  FilterKArgs a;
  a.rs = rs;
  a.npairs = (rs.rows + 1) / 2;
  a.tws = tws;
  a.hbr = hbr;
  return cuda_check(nullptr, launch_fft(a, ilog2(n), sms, stream), "fbp2d_filter_sinogram_noalloc: filter_fft_kernel");
}
