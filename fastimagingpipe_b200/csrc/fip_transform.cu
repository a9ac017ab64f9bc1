// The imager's transforms: band-pruned inverse FFT (fip_fft.cuh), its
// crop-and-correction epilogue, and the crop of cuFFT's output for the
// remaining grid sides.  Compiled with --use_fast_math like the other stages
// of the plain form (fip_plain.cu).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "fip_common.cuh"
#include "fip_fft.cuh"
#include "fip_fft_any.cuh"
#include "fip_kernels.h"
#include "fip_tma.cuh"

namespace {

constexpr int kThreads = 256;
constexpr int kAnyThreads = 256;
// Run-time lengths: the largest M (image sides up to 4,800), and the largest
// prime factor of M they take.  Up to that M two CTAs fit an SM and the passes
// win whatever the coverage (plain snapshots at 4800^2, baselines up to a fifth,
// half and nine tenths of the grid's half side: 484, 640 and 952 us, with cuFFT
// 952, 957 and 983); beyond it one does, and full coverage loses (5000^2 609, 841
// and 1,346 against 1,116, 1,135 and 1,156; 6000^2 927, 1,293 and 2,030 against
// 1,417, 1,427 and 1,458).
// A prime's pass costs in proportion to it, cuFFT's convolution transform of the
// whole grid does not: the lines are where the passes still win at half of the half
// side (us, own and cuFFT, at a fifth / half / nine tenths): p = 199 at 1592^2 173,
// 200, 250 and 239, p = 251 at 2008^2 250, 300, 382 and 325, at 3012^2 490, 644, 840
// and 880, p = 379 at 3032^2 636, 844, 1,111 and 884, p = 467 at 3736^2 1,034, 1,387,
// 1,896 and 1,780, p = 509 at 4072^2 1,242, 1,646, 2,211 and 1,765; p = 359 at 1436^2
// both passes alone 152 against 120.
constexpr int kAnyMax = 2400;
constexpr int kAnyPrime = 509;
static int any_prime_limit(int m) { return m >= 1500 ? kAnyPrime : (m >= 500 ? 251 : 199); }

inline int sm_count() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

// Block-wide maximum of non-negative v, folded into *out (float bits) with
// one atomic per CTA.  All threads of the CTA must call it.
__device__ __forceinline__ void block_max_to(float v, unsigned* out) {
  __shared__ float s_m[32];
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) s_m[warp] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    float m = 0.f;
    for (int w = 0; w < (int)((blockDim.x + 31) >> 5); ++w) m = fmaxf(m, s_m[w]);
    atomicMax(out, __float_as_uint(m));
  }
}

// ---------------------------------------------------------------------------
// Band-pruned inverse FFT (power-of-two images), instantiated per
// M = 2^LM = G / 3 and E = 2^LE values per thread (3 M / E threads).
// Column pass: P[c][yy] = sum_r1 H[c][r1 mod G] e^{+2 pi i y r1 / G},
// y = yy - N/2, for the occupied half-plane columns c <= bbox[1] and rows
// |r1| <= bbox[0].
// ---------------------------------------------------------------------------
template <int LM, int LE>
__host__ __device__ constexpr int fft_threads() { return 3 << (LM - LE); }
// CTAs per SM the register budget allows: the staged forms hold two
// buffers of shared memory (two CTAs of 768 or 384 threads); the direct form
// holds one, so three CTAs of 384 threads fit.
template <int LM, int LE, bool DIRECT>
__host__ __device__ constexpr int fft_min_blocks() {
  return fft_threads<LM, LE>() >= 768 && LE == 4 ? 1 : (DIRECT && LE == 4 ? 3 : 2);
}

template <int LM, int LE, bool DIRECT>
__global__ void __launch_bounds__(fft_threads<LM, LE>(), (fft_min_blocks<LM, LE, DIRECT>()))
    k_fft_cols(const float2* __restrict__ H, const unsigned* __restrict__ bbox,
               float2* __restrict__ P, const float2* __restrict__ tw, size_t grid_stride,
               size_t col_stride) {
  constexpr int M = 1 << LM, g = 3 * M, half = g / 2, n = 2 * M, NT = fft_threads<LM, LE>();
  extern __shared__ float2 s_fft[];
  // Batched launches: snapshot blockIdx.y.
  H += blockIdx.y * grid_stride;
  P += blockIdx.y * col_stride;
  bbox += 4 * blockIdx.y;
  const int k2 = (int)bbox[1];
  const int k1 = min((int)bbox[0], half);
  // Row band [lo, hi]; row -G/2 is row +G/2 (counted once).
  const int lo = (k1 == half) ? 1 - k1 : -k1, hi = k1;
  // Stage the band densely (coalesced): st[r - lo] = H[c][r mod G]; or
  // (DIRECT) read it from global memory in the first pass.
  // A band no wider than M is staged pre-twiddled for the three
  // sub-transforms (fipfft::stage_pre).
  float2* st = s_fft + fipfft::stage_offset(g);
  const bool fold = !DIRECT && hi - lo + 1 <= M;
  auto band = [&](int c, int r) -> float2 { return H[(size_t)c * g + (r < 0 ? r + g : r)]; };
  // The staged form is persistent over columns (blockIdx.x + k gridDim.x):
  // a thread's first staged element of the next column is loaded while the
  // current column is transformed.
  const int r0 = lo + (int)threadIdx.x;
  float2 pf = make_float2(0.f, 0.f);
  if (!DIRECT && (int)blockIdx.x <= k2 && r0 <= hi) pf = band(blockIdx.x, r0);
  for (int c = blockIdx.x; c <= k2; c += gridDim.x) {
    // Pass twiddles (registers): loaded after the staging loop, so their
    // latency overlaps the staging barrier without holding registers through
    // the loop (measured faster here than loading them up front).
    fipfft::PassTw<LM, LE> pt;
    if (DIRECT) pt.load(tw + g, fipfft::sub_lane<LM, LE>(threadIdx.x));
    if (fold) {
      fipfft::StageTw w(tw, g, r0, NT);
      if (r0 <= hi) fipfft::stage_pre<M>(st, r0, pf, w.w1, w.w2);
      w.next();
      for (int i = threadIdx.x + NT; i <= hi - lo; i += NT, w.next()) {
        const int r = i + lo;
        fipfft::stage_pre<M>(st, r, band(c, r), w.w1, w.w2);
      }
    } else if (!DIRECT) {
      if (r0 <= hi) st[threadIdx.x] = pf;
      for (int i = threadIdx.x + NT; i <= hi - lo; i += NT) st[i] = band(c, i + lo);
    }
    if (!DIRECT) {
      pt.load(tw + g, fipfft::sub_lane<LM, LE>(threadIdx.x));
      if (fold) fipfft::zero_pre<M>(st, lo, hi, threadIdx.x, NT);
      __syncthreads();
      // The next column's first element, in flight during this transform.
      const int nx = c + gridDim.x;
      if (nx <= k2 && r0 <= hi) pf = band(nx, r0);
    }
    if (fold) {
      fipfft::run_pre<LM, LE>(s_fft, pt);
    } else {
      auto load = [&](int r) -> float2 { return DIRECT ? band(c, r) : st[r - lo]; };
      fipfft::run<LM, LE, DIRECT>(s_fft, tw, pt, lo, hi, load);
    }
    float4* out = reinterpret_cast<float4*>(P + (size_t)c * n);
    for (int o2 = threadIdx.x; o2 < n / 2; o2 += NT) {
      float2 ab[2];
      fipfft::fetch_run<LM, LE, 2, DIRECT>(s_fft, 2 * o2, ab);
      out[o2] = make_float4(ab[0].x, ab[0].y, ab[1].x, ab[1].y);
    }
    // The next staging writes the second buffer: when the last pass left
    // its outputs there, every thread must be done reading them.
    if constexpr (!DIRECT && ((fipfft::pass_count<LM, LE>() - 1) & 1)) __syncthreads();
  }
}

// The row pass's band copy: columns 0 .. K2 (at most kBandCap; wider bands
// read global memory) of a row pair, kBandBox columns per bulk copy, 16
// bytes (rows yy1, yy1 + 1 of one column) each.
constexpr int kBandCap = 1024;
constexpr int kBandBox = 256;
// The copy's buffer follows the direct form's pass buffer; a bulk tensor
// copy's shared-memory destination must be 128-byte aligned, and dynamic
// shared memory starts after the kernel's static shared memory (not on a
// 128-byte boundary), so the buffer is aligned at run time within 128 bytes
// of slack.
template <int LM>
__host__ __device__ constexpr size_t band_offset() {  // bytes
  return (size_t)fipfft::direct_smem_elems(3 << LM) * sizeof(float2);
}
template <int LM>
__host__ __device__ constexpr size_t band_smem_bytes() {
  return band_offset<LM>() + 128 + (size_t)kBandCap * 16;
}

// Row pass for image rows yy1 = 2b, yy2 = 2b+1: their Hermitian spectra
// X1, X2 (the column-pass output, extended by X(-c) = conj X(c)) are packed as
// Z = X1 + i X2 so one complex transform yields both real rows.  The epilogue
// is the reference's crop/correction (FIPkernels.cu:256-287): the image pixel
// is |out| / (taper|x| taper|y| norm^2) (the checkerboard signs cancel
// against the centred grid origin), applied as a product of the reciprocal
// table rck[t] = 1 / (taper[t] norm).
// BAND (with DIRECT, persistent over row pairs): the first pass reads the
// row pair's band from a shared-memory copy that bulk tensor copies bring in
// one row pair ahead (band_map: the column-pass output as floats [batch][G/2
// + 1][2 N]); a copy that does not arrive within the wait limit switches the
// CTA to global reads (same results).
template <int LM, int LE, bool DIRECT, bool BAND = false>
__global__ void __launch_bounds__(fft_threads<LM, LE>(), (fft_min_blocks<LM, LE, DIRECT>()))
    k_fft_rows(const float2* __restrict__ P, unsigned* bbox,
               const float* __restrict__ rck, float* __restrict__ pre,
               const float2* __restrict__ tw, size_t col_stride, size_t pre_stride,
               const __grid_constant__ CUtensorMap band_map) {
  static_assert(!BAND || DIRECT, "the band copy replaces the direct form's global reads");
  constexpr int M = 1 << LM, g = 3 * M, half = g / 2, n = 2 * M, h = M, NT = fft_threads<LM, LE>();
  extern __shared__ float2 s_fft[];
  // Batched launches: snapshot blockIdx.y.
  P += blockIdx.y * col_stride;
  pre += blockIdx.y * pre_stride;
  bbox += 4 * blockIdx.y;
  const int k2 = min((int)bbox[1], half);
  // Column band [lo, hi]; column -G/2 is column +G/2 (counted once).
  const int lo = (k2 == half) ? 1 - k2 : -k2, hi = k2;
  // Stage Z[c] = X1[c] + i X2[c] at st[c - lo], with X(-c) = conj X(c):
  // one 16-byte load per occupied column c (the column pass stores
  // P[c][yy]), written at c and -c.
  float2* st = s_fft + fipfft::stage_offset(g);
  // Pass twiddles first: their loads overlap the staging loads.
  fipfft::PassTw<LM, LE> pt;
  pt.load(tw + g, fipfft::sub_lane<LM, LE>(threadIdx.x));
  // A band no wider than M is staged pre-twiddled (fipfft::stage_pre).
  const bool fold = !DIRECT && hi - lo + 1 <= M;
  // The staged form is persistent over row pairs (blockIdx.x + k gridDim.x):
  // a thread's first staged column of the next row pair is loaded into
  // registers while the current pair is transformed, so its latency leaves
  // the staging step (two columns measured slower: more spills).
  constexpr int kPf = 1;
  float4 pf[kPf];
  auto col_load = [&](int c, int yy) -> float4 {
    return *reinterpret_cast<const float4*>(P + (size_t)c * n + yy);
  };
#pragma unroll
  for (int m = 0; m < kPf; ++m) {
    const int c = threadIdx.x + m * NT;
    if (!DIRECT && c <= k2) pf[m] = col_load(c, 2 * blockIdx.x);
  }
  // BAND: the copy's buffer, its mbarrier, and the parity of a copy issued
  // but not yet consumed (-1: none).
  char* band_raw = reinterpret_cast<char*>(s_fft) + band_offset<LM>();
  float4* sband =
      reinterpret_cast<float4*>(band_raw + ((128u - (smem_u32(band_raw) & 127u)) & 127u));
  __shared__ uint64_t s_bandbar;
  // Uniform over the CTA; a misaligned buffer (not expected) reads global
  // memory instead.
  bool band = BAND && k2 + 1 <= kBandCap && (smem_u32(sband) & 127u) == 0;
  int pend = -1;
  const int nbox = (k2 + kBandBox) / kBandBox;  // boxes covering columns 0 .. k2
  auto issue = [&](int rpair) {  // one thread
    mbar_expect_tx(&s_bandbar, (unsigned)(nbox * kBandBox * 16));
    for (int b = 0; b < nbox; ++b)
      tma_load_3d(sband + b * kBandBox, &band_map, 4 * rpair, b * kBandBox, (int)blockIdx.y,
                  &s_bandbar);
  };
  if (BAND && band) {
    if (threadIdx.x == 0) {
      mbar_init(&s_bandbar, 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    if (blockIdx.x < n / 2) {
      if (threadIdx.x == 0) issue(blockIdx.x);
      pend = 0;
    }
  }
  float vmax = 0.f;
  int it = 0;
  for (int rp = blockIdx.x; rp < n / 2; rp += gridDim.x, ++it) {
    const int yy1 = 2 * rp;
    if (BAND && band) {
      const bool got = mbar_wait(&s_bandbar, (unsigned)(it & 1));
      band = __syncthreads_and(got) != 0;
      if (band) pend = -1;  // else the copy stays pending: drained at the end
    }
    if (!DIRECT) {
      fipfft::StageTw w(tw, g, threadIdx.x, NT);
      auto stage = [&](int c, const float4& ab) {
        float ay = ab.y, by = ab.w;
        if (c == 0 || c == half) {  // self-conjugate bins are real
          ay = 0.f;
          by = 0.f;
        }
        const float2 zp = make_float2(ab.x - by, ay + ab.z);
        const float2 zm = make_float2(ab.x + by, ab.z - ay);  // conj X1 + i conj X2
        if (fold) {
          // w^{-c} = conj w^c
          fipfft::stage_pre<M>(st, c, zp, w.w1, w.w2);
          if (c > 0 && -c >= lo)
            fipfft::stage_pre<M>(st, -c, zm, make_float2(w.w1.x, -w.w1.y),
                                 make_float2(w.w2.x, -w.w2.y));
        } else {
          st[c - lo] = zp;
          if (c > 0 && -c >= lo) st[-c - lo] = zm;
        }
      };
#pragma unroll
      for (int m = 0; m < kPf; ++m, w.next()) {
        const int c = threadIdx.x + m * NT;
        if (c <= k2) stage(c, pf[m]);
      }
      for (int c = threadIdx.x + kPf * NT; c <= k2; c += NT, w.next()) stage(c, col_load(c, yy1));
      if (fold) fipfft::zero_pre<M>(st, lo, hi, threadIdx.x, NT);
      __syncthreads();
      // The next row pair's first columns, in flight during this transform.
      const int nx = rp + gridDim.x;
#pragma unroll
      for (int m = 0; m < kPf; ++m) {
        const int c = threadIdx.x + m * NT;
        if (nx < n / 2 && c <= k2) pf[m] = col_load(c, 2 * nx);
      }
    }
    // DIRECT: Z[c] straight from the column-pass output (L2-resident).
    auto zval = [&](int c) -> float2 {
      const int a = c < 0 ? -c : c;
      const float4 ab = (BAND && band) ? sband[a] : col_load(a, yy1);
      float ay = ab.y, by = ab.w;
      if (a == 0 || a == half) {
        ay = 0.f;
        by = 0.f;
      }
      return c >= 0 ? make_float2(ab.x - by, ay + ab.z) : make_float2(ab.x + by, ab.z - ay);
    };
    auto load = [&](int c) -> float2 { return DIRECT ? zval(c) : st[c - lo]; };
    if (fold) {
      fipfft::run_pre<LM, LE>(s_fft, pt);
    } else if constexpr (BAND) {
      // Once every thread holds its band values, the next row pair's copy
      // goes into the buffer (it lands during this pair's passes).
      auto loaded = [&]() {
        if (!band) return;
        __syncthreads();
        const int nx = rp + (int)gridDim.x;
        if (nx < n / 2) {
          if (threadIdx.x == 0) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            issue(nx);
          }
          pend = (it + 1) & 1;
        }
      };
      fipfft::run<LM, LE, DIRECT>(s_fft, tw, pt, lo, hi, load, loaded);
    } else {
      fipfft::run<LM, LE, DIRECT>(s_fft, tw, pt, lo, hi, load);
    }
    const float ry1 = rck[abs(yy1 - h)], ry2 = rck[abs(yy1 + 1 - h)];
    float4* row1 = reinterpret_cast<float4*>(pre + (size_t)yy1 * n);
    float4* row2 = reinterpret_cast<float4*>(pre + (size_t)(yy1 + 1) * n);
    // The epilogue's correction factors, all loads issued before the first
    // output is formed.
    constexpr int KQ = (n / 4 + NT - 1) / NT;
    float rxs[KQ][4];
#pragma unroll
    for (int q = 0; q < KQ; ++q) {
      const int o4 = threadIdx.x + q * NT;
#pragma unroll
      for (int e = 0; e < 4; ++e)
        rxs[q][e] = o4 < n / 4 ? __ldg(&rck[abs(4 * o4 + e - h)]) : 0.f;
    }
#pragma unroll
    for (int q = 0; q < KQ; ++q) {
      const int o4 = threadIdx.x + q * NT;
      if (o4 < n / 4) {
        float a[4], b[4];
        float2 v[4];
        fipfft::fetch_run<LM, LE, 4, DIRECT>(s_fft, 4 * o4, v);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float rx = rxs[q][e];
          a[e] = fabsf(v[e].x * (rx * ry1));
          b[e] = fabsf(v[e].y * (rx * ry2));
          vmax = fmaxf(vmax, fmaxf(a[e], b[e]));
        }
        row1[o4] = make_float4(a[0], a[1], a[2], a[3]);
        row2[o4] = make_float4(b[0], b[1], b[2], b[3]);
      }
    }
    // The next staging writes the second buffer: when the last pass left
    // its outputs there, every thread must be done reading them.
    if constexpr (!DIRECT && ((fipfft::pass_count<LM, LE>() - 1) & 1)) __syncthreads();
  }
  // A copy still pending (its wait ran out) lands before the CTA's shared
  // memory goes away (bounded, like every wait here).
  if (BAND && pend >= 0 && threadIdx.x == 0) mbar_wait(&s_bandbar, (unsigned)pend);
  // Image maximum (bbox[3], float bits; zeroed by the binning), which
  // scales the reprojection's fixed-point sums.
  block_max_to(vmax, &bbox[3]);
}

// Split forms of the two passes: one CTA of M / E threads per (column or row
// pair, sub-transform s), grid.y = s, grid.z = snapshot of a batch.  Three
// times the CTAs of a quarter of the size: each CTA's barriers hold four
// warps instead of twelve, and CTAs at different phases share an SM.  Each
// CTA stages the band itself (in its second buffer when it fits, else reads
// it from global memory) and writes its outputs X[3 q + s] directly.
template <int LM, int LE>
__host__ __device__ constexpr int split_threads() { return 1 << (LM - LE); }

template <int LM, int LE>
__global__ void __launch_bounds__(split_threads<LM, LE>(), (LE == 4 ? 6 : 4))
    k_fft_cols_split(const float2* __restrict__ H, const unsigned* __restrict__ bbox,
                     float2* __restrict__ P, const float2* __restrict__ tw, size_t grid_stride,
                     size_t col_stride) {
  constexpr int M = 1 << LM, g = 3 * M, half = g / 2, n = 2 * M, NT = split_threads<LM, LE>();
  constexpr int kCap = fipfft::sub_stride(M);  // staging capacity (the second buffer)
  extern __shared__ float2 s_fft[];
  H += blockIdx.z * grid_stride;
  P += blockIdx.z * col_stride;
  bbox += 4 * blockIdx.z;
  const int c = blockIdx.x, s = blockIdx.y;
  const int k2 = (int)bbox[1];
  if (c > k2) return;
  const int k1 = min((int)bbox[0], half);
  const int lo = (k1 == half) ? 1 - k1 : -k1, hi = k1;
  const float2* col = H + (size_t)c * g;
  float2* st = s_fft + kCap;
  const bool staged = hi - lo + 1 <= kCap;
  if (staged)
    for (int i = threadIdx.x; i <= hi - lo; i += NT) {
      const int r = i + lo;
      st[i] = col[r < 0 ? r + g : r];
    }
  __syncthreads();
  auto load = [&](int r) -> float2 { return staged ? st[r - lo] : col[r < 0 ? r + g : r]; };
  fipfft::PassTw<LM, LE> pt;
  pt.load(tw + g, threadIdx.x);
  fipfft::run_single<LM, LE>(s_fft, s, tw, pt, lo, hi, load);
  float2* out = P + (size_t)c * n;
  for (int q = threadIdx.x; q < M; q += NT) {
    const int pp = 3 * q + s;  // output p = pp (mod G), kept when |p| <= M
    const int o = pp < M ? pp + M : (pp >= 2 * M ? pp - 2 * M : -1);
    if (o >= 0) out[o] = fipfft::single_out<LM, LE>(s_fft, q);
  }
}

template <int LM, int LE>
__global__ void __launch_bounds__(split_threads<LM, LE>(), (LE == 4 ? 6 : 4))
    k_fft_rows_split(const float2* __restrict__ P, unsigned* bbox, const float* __restrict__ rck,
                     float* __restrict__ pre, const float2* __restrict__ tw, size_t col_stride,
                     size_t pre_stride) {
  constexpr int M = 1 << LM, g = 3 * M, half = g / 2, n = 2 * M, h = M;
  constexpr int NT = split_threads<LM, LE>(), kCap = fipfft::sub_stride(M);
  extern __shared__ float2 s_fft[];
  P += blockIdx.z * col_stride;
  pre += blockIdx.z * pre_stride;
  bbox += 4 * blockIdx.z;
  const int yy1 = 2 * blockIdx.x, s = blockIdx.y;
  const int k2 = min((int)bbox[1], half);
  const int lo = (k2 == half) ? 1 - k2 : -k2, hi = k2;
  // Z[c] = X1[c] + i X2[c], X(-c) = conj X(c), from the column-pass output.
  auto zval = [&](int c) -> float2 {
    const int a = c < 0 ? -c : c;
    const float4 ab = *reinterpret_cast<const float4*>(P + (size_t)a * n + yy1);
    float ay = ab.y, by = ab.w;
    if (a == 0 || a == half) {  // self-conjugate bins are real
      ay = 0.f;
      by = 0.f;
    }
    return c >= 0 ? make_float2(ab.x - by, ay + ab.z) : make_float2(ab.x + by, ab.z - ay);
  };
  float2* st = s_fft + kCap;
  const bool staged = hi - lo + 1 <= kCap;
  if (staged)
    for (int c = threadIdx.x; c <= k2; c += NT) {
      const float4 ab = *reinterpret_cast<const float4*>(P + (size_t)c * n + yy1);
      float ay = ab.y, by = ab.w;
      if (c == 0 || c == half) {
        ay = 0.f;
        by = 0.f;
      }
      st[c - lo] = make_float2(ab.x - by, ay + ab.z);
      if (c > 0 && -c >= lo) st[-c - lo] = make_float2(ab.x + by, ab.z - ay);
    }
  __syncthreads();
  auto load = [&](int c) -> float2 { return staged ? st[c - lo] : zval(c); };
  fipfft::PassTw<LM, LE> pt;
  pt.load(tw + g, threadIdx.x);
  fipfft::run_single<LM, LE>(s_fft, s, tw, pt, lo, hi, load);
  const float ry1 = rck[abs(yy1 - h)], ry2 = rck[abs(yy1 + 1 - h)];
  float* row1 = pre + (size_t)yy1 * n;
  float* row2 = row1 + n;
  float vmax = 0.f;
  for (int q = threadIdx.x; q < M; q += NT) {
    const int pp = 3 * q + s;
    const int o = pp < M ? pp + M : (pp >= 2 * M ? pp - 2 * M : -1);
    if (o >= 0) {
      const float2 v = fipfft::single_out<LM, LE>(s_fft, q);
      const float rx = rck[abs(o - h)];
      const float a = fabsf(v.x * (rx * ry1)), b = fabsf(v.y * (rx * ry2));
      row1[o] = a;
      row2[o] = b;
      vmax = fmaxf(vmax, fmaxf(a, b));
    }
  }
  block_max_to(vmax, &bbox[3]);
}

// The two passes for run-time lengths (fip_fft_any.cuh): a CTA per column or row
// pair in turn, several CTAs per SM hiding one another's barriers; inputs,
// outputs and epilogue as the power-of-two passes'.  Bound: shared-memory
// round trips and barriers (44 % of issue slots, three CTAs per SM at 3000^2).
// Both passes against cuFFT's transform of the whole grid and the crop, us:
// 1000^2 15 and 39, 1500^2 24 and 55, 1484^2 (factor 53) 60 and 120, 3000^2 93 and
// 236 with baselines up to three tenths of the grid's half side, 198 and 237 up to
// nine tenths; the band layout they allow also spares the gridder the rest of the
// grid (3000^2 66 -> 45 us).
__global__ void __launch_bounds__(kAnyThreads) k_fft_any_cols(const float2* __restrict__ H,
                                                              const unsigned* __restrict__ bbox,
                                                              float2* __restrict__ P,
                                                              const float2* __restrict__ tw,
                                                              const __grid_constant__ fipfft::Plan p,
                                                              size_t grid_stride,
                                                              size_t col_stride) {
  extern __shared__ float2 s_fft[];
  const int g = p.g, n = 2 * p.m, half = g / 2;
  H += blockIdx.y * grid_stride;
  P += blockIdx.y * col_stride;
  bbox += 4 * blockIdx.y;
  const int k2 = (int)bbox[1], k1 = min((int)bbox[0], half);
  // Row -G/2 is row +G/2 (counted once).
  const int lo = (k1 == half) ? 1 - k1 : -k1, hi = k1;
  fipfft::any_load_roots(s_fft, p, tw);
  for (int c = blockIdx.x; c <= k2; c += gridDim.x) {
    const float2* col = H + (size_t)c * g;
    fipfft::any_stage(s_fft, p, lo, hi, tw, [&](int r) { return col[r < 0 ? r + g : r]; });
    __syncthreads();
    const float2* y = fipfft::any_run(s_fft, p, tw);
    float2* out = P + (size_t)c * n;
    for (int o = threadIdx.x; o < n; o += blockDim.x) out[o] = fipfft::any_fetch(y, p.m, o);
    __syncthreads();  // the next staging may write the buffer just read
  }
}

__global__ void __launch_bounds__(kAnyThreads) k_fft_any_rows(const float2* __restrict__ P,
                                                              unsigned* bbox,
                                                              const float* __restrict__ rck,
                                                              float* __restrict__ pre,
                                                              const float2* __restrict__ tw,
                                                              const __grid_constant__ fipfft::Plan p,
                                                              size_t col_stride,
                                                              size_t pre_stride) {
  extern __shared__ float2 s_fft[];
  const int n = 2 * p.m, half = p.g / 2, h = p.m;
  P += blockIdx.y * col_stride;
  pre += blockIdx.y * pre_stride;
  bbox += 4 * blockIdx.y;
  const int k2 = min((int)bbox[1], half);
  const int lo = (k2 == half) ? 1 - k2 : -k2, hi = k2;
  float vmax = 0.f;
  fipfft::any_load_roots(s_fft, p, tw);
  for (int rp = blockIdx.x; rp < n / 2; rp += gridDim.x) {
    const int yy1 = 2 * rp;
    // Z[c] = X1[c] + i X2[c], X(-c) = conj X(c); self-conjugate bins are real.
    fipfft::any_stage(s_fft, p, lo, hi, tw, [&](int c) {
      const int a = c < 0 ? -c : c;
      const float4 ab = *reinterpret_cast<const float4*>(P + (size_t)a * n + yy1);
      const bool self = a == 0 || a == half;
      const float ay = self ? 0.f : ab.y, by = self ? 0.f : ab.w;
      return c >= 0 ? make_float2(ab.x - by, ay + ab.z) : make_float2(ab.x + by, ab.z - ay);
    });
    __syncthreads();
    const float2* y = fipfft::any_run(s_fft, p, tw);
    const float ry1 = rck[abs(yy1 - h)], ry2 = rck[abs(yy1 + 1 - h)];
    float* row1 = pre + (size_t)yy1 * n;
    float* row2 = row1 + n;
    for (int o = threadIdx.x; o < n; o += blockDim.x) {
      const float2 v = fipfft::any_fetch(y, p.m, o);
      const float rx = rck[abs(o - h)];
      const float a = fabsf(v.x * (rx * ry1)), b = fabsf(v.y * (rx * ry2));
      row1[o] = a;
      row2[o] = b;
      vmax = fmaxf(vmax, fmaxf(a, b));
    }
    __syncthreads();
  }
  block_max_to(vmax, &bbox[3]);
}

// Crop + correction of the cuFFT C2R output (images whose grid side the
// transforms above do not cover): row (y mod G), column (x mod G), row stride G + 2 floats.
__global__ void k_correct_c2r(const float* __restrict__ fft_out, const float* __restrict__ ck,
                              int n, int g, float* __restrict__ pre, unsigned* pre_max) {
  const int xx = blockIdx.x * blockDim.x + threadIdx.x, yy = blockIdx.y;
  float v = 0.f;
  if (xx < n) {
    const int h = n / 2;
    const long x = (long)xx - h, y = (long)yy - h;
    const int row = (int)(y < 0 ? y + g : y), col = (int)(x < 0 ? x + g : x);
    float px = fft_out[(size_t)row * (size_t)(g + 2) + col];
    const float norm = FIP_CONV_NORM;
    px *= 1 / (ck[labs(x)] * ck[labs(y)] * norm * norm);
    v = fabs(px);
    pre[(size_t)yy * n + xx] = v;
  }
  block_max_to(v, pre_max);
}

}  // namespace

// Run-time passes for M = G / 3: the largest prime factors first (one pass
// each above 7), then 7s, and the 2, 3, 5 part in the fewest passes, odd radices
// first (their first-pass stores fall on distinct banks).
static bool plan_any(int g, fipfft::Plan& p) {
  const int m = g / 3;
  p = fipfft::Plan{};
  if (m < 8 || m % 2 != 0 || m > kAnyMax) return false;
  int r = m, big[fipfft::kMaxPasses], nbig = 0, e2 = 0, e3 = 0, e5 = 0;
  while (r % 2 == 0) r /= 2, ++e2;
  while (r % 3 == 0) r /= 3, ++e3;
  while (r % 5 == 0) r /= 5, ++e5;
  for (int f = 7; r > 1; f += 2)
    while (r % f == 0) {
      if (f > any_prime_limit(m) || nbig >= 4) return false;
      big[nbig++] = f;
      r /= f;
    }
  int n = 0;
  for (int k = nbig - 1; k >= 0; --k) p.radix[n++] = big[k];
  // Pair the factors into codelets: 15, 9, 10, 12, 6, then powers of two.
  while (e3 && e5) p.radix[n++] = 15, --e3, --e5;
  while (e3 >= 2) p.radix[n++] = 9, e3 -= 2;
  int tail[fipfft::kMaxPasses], nt = 0;
  while (e5 && n + nt < 10) {
    if (e2 > 0) tail[nt++] = 10, --e2; else tail[nt++] = 5;
    --e5;
  }
  while (e3 && n + nt < 10) {
    if (e2 > 1) tail[nt++] = 12, e2 -= 2;
    else if (e2 == 1) tail[nt++] = 6, --e2;
    else tail[nt++] = 3;
    --e3;
  }
  while (e2 > 0 && n + nt < fipfft::kMaxPasses) {
    const int t = e2 >= 4 && e2 != 5 && e2 != 6 ? 4 : (e2 >= 3 ? 3 : e2);
    tail[nt++] = 1 << t;
    e2 -= t;
  }
  if (e2 || e3 || e5 || n + nt > fipfft::kMaxPasses) return false;
  for (int k = 0; k < nt; ++k) p.radix[n++] = tail[k];
  p.g = g;
  p.m = m;
  p.any = 1;
  p.passes = n;
  p.nt = std::max(64, std::min(kAnyThreads, (3 * m / 8 + 31) / 32 * 32));
  return true;
}

bool fip_fft_plan(int g, fipfft::Plan& p, int values_per_thread) {
  if (g < 24 || g % 3 != 0) return false;
  const int m = g / 3;
  if ((m & (m - 1)) || g < 48) return values_per_thread == 0 && plan_any(g, p);
  int lm = 0;
  while ((1 << lm) < m) ++lm;
  // Instantiated: 8 values per thread for M = 2^4..2^11, 16 for 2^5..2^12
  // (<= 768 threads).  Default: 8 up to M = 1024 (N = 2048), 16 beyond -- at
  // M = 2048 the 16-value row pass takes about two thirds of the 8-value one's
  // time on B200, and the autotuner picks it there.
  int le = (lm <= 10) ? 3 : 4;
  if (values_per_thread == 8) le = 3;
  if (values_per_thread == 16) le = 4;
  if (le == 3 && (lm < 4 || lm > 11)) return false;
  if (le == 4 && (lm < 5 || lm > 12)) return false;
  p = fipfft::Plan{};
  p.g = g;
  p.m = m;
  p.lm = lm;
  p.le = le;
  p.e = 1 << le;
  p.nt = 3 * (m >> le);
  p.split = 0;
  p.direct = 0;
  return true;
}

// The transforms' dynamic shared memory depends on the grid side.  Their
// limit is raised to the most the device allows next to the kernel's static
// shared memory, the same value for every caller, so imagers of different
// sizes launching from concurrent host threads never lower it under one
// another's launch.
static cudaError_t fft_smem_attr(const void* fn, size_t smem) {
  int dev = 0, optin = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess)
    e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e != cudaSuccess) return e;
  cudaFuncAttributes fa{};
  e = cudaFuncGetAttributes(&fa, fn);
  if (e != cudaSuccess) return e;
  const int most = optin - (int)fa.sharedSizeBytes;  // static + dynamic <= opt-in maximum
  if (smem > (size_t)most) return cudaErrorInvalidConfiguration;
  return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
}

template <int LM, int LE>
static cudaError_t launch_cols(const FipGeom& geo, const float2* grid, const unsigned* bbox,
                               float2* colbuf, const float2* tw, cudaStream_t s, int batch,
                               size_t grid_stride, size_t col_stride, int split, int direct) {
  size_t smem;
  cudaError_t e;
  if (split) {
    smem = 2 * (size_t)fipfft::sub_stride(1 << LM) * sizeof(float2);
    if ((e = fft_smem_attr((const void*)k_fft_cols_split<LM, LE>, smem)) != cudaSuccess)
      return e;
    k_fft_cols_split<LM, LE><<<dim3(geo.hp, 3, batch), split_threads<LM, LE>(), smem, s>>>(
        grid, bbox, colbuf, tw, grid_stride, col_stride);
    return cudaGetLastError();
  }
  if (direct == 1) {  // (2: the row pass's band copy; the column pass stays staged)
    smem = (size_t)fipfft::direct_smem_elems(geo.g) * sizeof(float2);
    e = fft_smem_attr((const void*)k_fft_cols<LM, LE, true>, smem);
    if (e != cudaSuccess) return e;
    k_fft_cols<LM, LE, true><<<dim3(geo.hp, batch), fft_threads<LM, LE>(), smem, s>>>(
        grid, bbox, colbuf, tw, grid_stride, col_stride);
    return cudaGetLastError();
  }
  smem = (size_t)fipfft::smem_elems(geo.g) * sizeof(float2);
  e = fft_smem_attr((const void*)k_fft_cols<LM, LE, false>, smem);
  if (e != cudaSuccess) return e;
  // Persistent over columns: the CTAs that fit at once.
  // (Queried once per instantiation: the shape and shared memory are fixed by it.)
  static const int per_sm = [&] {
    int v = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_fft_cols<LM, LE, false>,
                                                      fft_threads<LM, LE>(), smem) != cudaSuccess)
      v = 1;
    return std::max(v, 1);
  }();
  const int ctas = std::max(1, std::min(geo.hp, per_sm * sm_count()));
  k_fft_cols<LM, LE, false><<<dim3(ctas, batch), fft_threads<LM, LE>(), smem, s>>>(
      grid, bbox, colbuf, tw, grid_stride, col_stride);
  return cudaGetLastError();
}

// The column-pass output of a batch as floats [batch][G/2 + 1][2 N], in boxes
// of 4 floats (rows yy1, yy1 + 1 of a column) x kBandBox columns.
static bool encode_band_map(CUtensorMap* m, const float2* colbuf, const FipGeom& geo, int batch,
                            size_t col_stride) {
  const PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
  if (!enc || ((uintptr_t)colbuf & 15) != 0 || batch < 1) return false;
  const cuuint64_t dims[3] = {2 * (cuuint64_t)geo.n, (cuuint64_t)geo.hp, (cuuint64_t)batch};
  const cuuint64_t strides[2] = {2 * (cuuint64_t)geo.n * 4,
                                 (cuuint64_t)(batch > 1 ? col_stride : (size_t)geo.hp * geo.n) * 8};
  const cuuint32_t box[3] = {4, (cuuint32_t)kBandBox, 1};
  const cuuint32_t es[3] = {1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float2*>(colbuf), dims, strides,
             box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
         CUDA_SUCCESS;
}

template <int LM, int LE>
static cudaError_t launch_rows(const FipGeom& geo, const float2* colbuf, unsigned* bbox,
                               const float* taper, const float2* tw, float* pre,
                               cudaStream_t s, int batch, size_t col_stride,
                               size_t pre_stride, int split, int direct) {
  size_t smem;
  cudaError_t e;
  const CUtensorMap no_map{};
  if (split) {
    smem = 2 * (size_t)fipfft::sub_stride(1 << LM) * sizeof(float2);
    if ((e = fft_smem_attr((const void*)k_fft_rows_split<LM, LE>, smem)) != cudaSuccess)
      return e;
    k_fft_rows_split<LM, LE><<<dim3(geo.n / 2, 3, batch), split_threads<LM, LE>(), smem, s>>>(
        colbuf, bbox, taper + geo.n / 2 + 1, pre, tw, col_stride, pre_stride);
    return cudaGetLastError();
  }
  CUtensorMap band_map{};
  if (direct == 2 && encode_band_map(&band_map, colbuf, geo, batch, col_stride)) {
    // Persistent over row pairs (the CTAs that fit at once), the band copy
    // one row pair ahead.
    smem = band_smem_bytes<LM>();
    e = fft_smem_attr((const void*)k_fft_rows<LM, LE, true, true>, smem);
    if (e != cudaSuccess) return e;
    static const int per_sm = [&] {
      int v = 0;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_fft_rows<LM, LE, true, true>,
                                                        fft_threads<LM, LE>(), smem) !=
          cudaSuccess)
        v = 1;
      return std::max(v, 1);
    }();
    const int ctas = std::max(1, std::min(geo.n / 2, per_sm * sm_count()));
    k_fft_rows<LM, LE, true, true><<<dim3(ctas, batch), fft_threads<LM, LE>(), smem, s>>>(
        colbuf, bbox, taper + geo.n / 2 + 1, pre, tw, col_stride, pre_stride, band_map);
    return cudaGetLastError();
  }
  if (direct) {
    smem = (size_t)fipfft::direct_smem_elems(geo.g) * sizeof(float2);
    e = fft_smem_attr((const void*)k_fft_rows<LM, LE, true>, smem);
    if (e != cudaSuccess) return e;
    k_fft_rows<LM, LE, true><<<dim3(geo.n / 2, batch), fft_threads<LM, LE>(), smem, s>>>(
        colbuf, bbox, taper + geo.n / 2 + 1, pre, tw, col_stride, pre_stride, no_map);
    return cudaGetLastError();
  }
  smem = (size_t)fipfft::smem_elems(geo.g) * sizeof(float2);
  e = fft_smem_attr((const void*)k_fft_rows<LM, LE, false>, smem);
  if (e != cudaSuccess) return e;
  // Persistent over row pairs: the CTAs that fit at once.
  // (Queried once per instantiation: the shape and shared memory are fixed by it.)
  static const int per_sm = [&] {
    int v = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_fft_rows<LM, LE, false>,
                                                      fft_threads<LM, LE>(), smem) != cudaSuccess)
      v = 1;
    return std::max(v, 1);
  }();
  const int ctas = std::max(1, std::min(geo.n / 2, per_sm * sm_count()));
  k_fft_rows<LM, LE, false><<<dim3(ctas, batch), fft_threads<LM, LE>(), smem, s>>>(
      colbuf, bbox, taper + geo.n / 2 + 1, pre, tw, col_stride, pre_stride, no_map);
  return cudaGetLastError();
}

// CTAs of a run-time pass over `items` columns or row pairs.
static int any_ctas(const void* fn, const fipfft::Plan& plan, size_t smem, int items,
                    cudaError_t& e) {
  e = fft_smem_attr(fn, smem);
  if (e != cudaSuccess) return 0;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, plan.nt, smem);
  return std::max(1, std::min(items, std::max(1, per_sm) * sm_count()));
}

static cudaError_t launch_any_cols(const FipGeom& geo, const float2* grid, const unsigned* bbox,
                                   float2* colbuf, const float2* tw, const fipfft::Plan& plan,
                                   cudaStream_t s, int batch, size_t grid_stride,
                                   size_t col_stride) {
  const size_t smem = (size_t)fipfft::any_smem_elems(plan) * sizeof(float2);
  cudaError_t e;
  const int ctas = any_ctas((const void*)k_fft_any_cols, plan, smem, geo.hp, e);
  if (e != cudaSuccess) return e;
  k_fft_any_cols<<<dim3(ctas, batch), plan.nt, smem, s>>>(grid, bbox, colbuf, tw, plan,
                                                          grid_stride, col_stride);
  return cudaGetLastError();
}

static cudaError_t launch_any_rows(const FipGeom& geo, const float2* colbuf, unsigned* bbox,
                                   const float* taper, const float2* tw,
                                   const fipfft::Plan& plan, float* pre, cudaStream_t s,
                                   int batch, size_t col_stride, size_t pre_stride) {
  const size_t smem = (size_t)fipfft::any_smem_elems(plan) * sizeof(float2);
  cudaError_t e;
  const int ctas = any_ctas((const void*)k_fft_any_rows, plan, smem, geo.n / 2, e);
  if (e != cudaSuccess) return e;
  k_fft_any_rows<<<dim3(ctas, batch), plan.nt, smem, s>>>(
      colbuf, bbox, taper + geo.n / 2 + 1, pre, tw, plan, col_stride, pre_stride);
  return cudaGetLastError();
}

// Calls F<LM, LE> for the plan's instantiation.
#define FIP_FFT_SWITCH(PLAN, CALL)                                      \
  do {                                                                  \
    const int key_ = (PLAN).lm * 8 + (PLAN).le;                         \
    switch (key_) {                                                     \
      case 4 * 8 + 3: { constexpr int LM_ = 4, LE_ = 3; return CALL; }  \
      case 5 * 8 + 3: { constexpr int LM_ = 5, LE_ = 3; return CALL; }  \
      case 6 * 8 + 3: { constexpr int LM_ = 6, LE_ = 3; return CALL; }  \
      case 7 * 8 + 3: { constexpr int LM_ = 7, LE_ = 3; return CALL; }  \
      case 8 * 8 + 3: { constexpr int LM_ = 8, LE_ = 3; return CALL; }  \
      case 9 * 8 + 3: { constexpr int LM_ = 9, LE_ = 3; return CALL; }  \
      case 10 * 8 + 3: { constexpr int LM_ = 10, LE_ = 3; return CALL; } \
      case 11 * 8 + 3: { constexpr int LM_ = 11, LE_ = 3; return CALL; } \
      case 5 * 8 + 4: { constexpr int LM_ = 5, LE_ = 4; return CALL; }  \
      case 6 * 8 + 4: { constexpr int LM_ = 6, LE_ = 4; return CALL; }  \
      case 7 * 8 + 4: { constexpr int LM_ = 7, LE_ = 4; return CALL; }  \
      case 8 * 8 + 4: { constexpr int LM_ = 8, LE_ = 4; return CALL; }  \
      case 9 * 8 + 4: { constexpr int LM_ = 9, LE_ = 4; return CALL; }  \
      case 10 * 8 + 4: { constexpr int LM_ = 10, LE_ = 4; return CALL; } \
      case 11 * 8 + 4: { constexpr int LM_ = 11, LE_ = 4; return CALL; } \
      case 12 * 8 + 4: { constexpr int LM_ = 12, LE_ = 4; return CALL; } \
      default: return cudaErrorInvalidValue;                             \
    }                                                                   \
  } while (0)

cudaError_t fip_launch_fft_cols(const FipGeom& geo, const float2* grid, const unsigned* bbox,
                                float2* colbuf, const float2* twiddles, const fipfft::Plan& plan,
                                cudaStream_t s, int batch, size_t grid_stride,
                                size_t col_stride) {
  if (plan.g != geo.g || batch < 1 || batch > 65535) return cudaErrorInvalidValue;
  if (plan.any)
    return launch_any_cols(geo, grid, bbox, colbuf, twiddles, plan, s, batch, grid_stride,
                           col_stride);
  FIP_FFT_SWITCH(plan, (launch_cols<LM_, LE_>(geo, grid, bbox, colbuf, twiddles, s, batch,
                                              grid_stride, col_stride, plan.split,
                                              plan.direct)));
}

cudaError_t fip_launch_fft_rows(const FipGeom& geo, const float2* colbuf, unsigned* bbox,
                                const float* taper, const float2* twiddles,
                                const fipfft::Plan& plan, float* pre, cudaStream_t s, int batch,
                                size_t col_stride, size_t pre_stride) {
  if (plan.g != geo.g || batch < 1 || batch > 65535) return cudaErrorInvalidValue;
  if (plan.any)
    return launch_any_rows(geo, colbuf, bbox, taper, twiddles, plan, pre, s, batch, col_stride,
                           pre_stride);
  FIP_FFT_SWITCH(plan, (launch_rows<LM_, LE_>(geo, colbuf, bbox, taper, twiddles, pre, s, batch,
                                              col_stride, pre_stride, plan.split,
                                              plan.direct)));
}

cudaError_t fip_launch_correct_c2r(const FipGeom& geo, const float* fft_out, const float* taper,
                                   float* pre, unsigned* pre_max, cudaStream_t s) {
  dim3 bl((geo.n + kThreads - 1) / kThreads, geo.n);
  k_correct_c2r<<<bl, kThreads, 0, s>>>(fft_out, taper, geo.n, geo.g, pre, pre_max);
  return cudaGetLastError();
}
