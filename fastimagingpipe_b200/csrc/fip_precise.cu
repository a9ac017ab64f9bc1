// IEEE-arithmetic stages (compiled without fast math): plane projection of
// baseline uvw, Stokes-I collapse, and the reduced-precision visibility
// storage of the precision form.
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include <cooperative_groups.h>
#include <stdint.h>

#include <algorithm>

#include "fip_common.cuh"
#include "fip_kernels.h"

namespace {

constexpr int kThreads = 256;
constexpr double kLight = 299792458.0;
constexpr int kSms = 148;  // of a B200, the one device this is built for

// ---------------------------------------------------------------------------
// Plane fit of a snapshot's uvw (SVDPreprocessKernels.cu:41-206).  Sample
// s = row + chan * rows (SVDPreprocessMain.cpp:36-38) lies at uvw[row] f / c
// wavelengths (SVDPreprocessKernels.cu:41-61), so every moment factors into
// one over the rows and one over the channels: with u = uvw[row], S the
// centred scatter of the rows, m their mean, and k = f / c over `chans`
// channels,
//   sum_s (x - mean)(x - mean)^T = (sum k^2) S + (sum (k - mean k)^2) R m m^T
// and one pass over the rows (not over the samples) suffices.  S is formed
// from sums shifted by the first row, FP64, both terms positive: no
// cancellation beyond the rows' own spread.
// The fit needs no device memory of its own: up to kPlaneOneCluster samples
// take one launch of one eight-CTA cluster, whose partial sums meet in
// distributed shared memory; larger ones keep the partial sums and the basis
// in the head of B itself, whose first samples are projected last.  The
// bound is latency: three FP64 reductions and ~15 dependent rotations.
// 130,816 rows of an Earth-rotating array: 17.8 us of kernels against 136 us
// for the six launches this replaces (a single-thread FP64 Jacobi iteration
// to 1e-300 out of local memory, 99 us, and two serial reductions, 22 us),
// whose stream-ordered scratch was also mapped anew after every
// synchronisation (a first pass on a new snapshot: + 0.4 ms).
// Few rows of many channels are projected by sample, and more than kWarpChans
// channels summed by every thread (left to one thread per row and one warp, 1 row
// of 65,536 channels took 2,345 us and 5 rows of 52,500 455; now 29 and 19).
// ---------------------------------------------------------------------------
constexpr int kMom = 9;  // sum u' (3), sum u' u'^T (6: 00 01 02 11 12 22), u' = u - uvw[0]
constexpr int kChan = 2;  // sum k', sum k'^2, k' = k - k of channel 0
// Channels that one warp sums; more are summed by all threads.
constexpr size_t kWarpChans = 256;

// Adds the moments of rows first, first + step, ... to acc.
__device__ __forceinline__ void row_moments(const float* __restrict__ uvw, size_t rows,
                                            size_t first, size_t step, double (&acc)[kMom]) {
  const double a0 = uvw[0], a1 = uvw[1], a2 = uvw[2];
#pragma unroll
  for (int k = 0; k < kMom; ++k) acc[k] = 0.0;
#pragma unroll 4
  for (size_t r = first; r < rows; r += step) {
    const double x = uvw[3 * r] - a0, y = uvw[3 * r + 1] - a1, z = uvw[3 * r + 2] - a2;
    acc[0] += x; acc[1] += y; acc[2] += z;
    acc[3] += x * x; acc[4] += x * y; acc[5] += x * z;
    acc[6] += y * y; acc[7] += y * z; acc[8] += z * z;
  }
}

// Adds the moments of channels first, first + step, ... to acc.
__device__ __forceinline__ void channel_moments(const float* __restrict__ freqs, size_t chans,
                                                size_t first, size_t step, double (&acc)[kChan]) {
  const double k0 = (double)freqs[0] / kLight;
  acc[0] = acc[1] = 0.0;
  for (size_t c = first; c < chans; c += step) {
    const double d = (double)freqs[c] / kLight - k0;
    acc[0] += d;
    acc[1] += d * d;
  }
}

// sum k^2 and sum (k - mean k)^2 from the channels' moments.
__device__ __forceinline__ void channel_sums(const double* mom, const float* __restrict__ freqs,
                                             size_t chans, double& k2, double& var) {
  const double k0 = (double)freqs[0] / kLight, n = (double)chans;
  k2 = n * k0 * k0 + 2.0 * k0 * mom[0] + mom[1];
  var = fmax(0.0, mom[1] - mom[0] * mom[0] / n);
}

// Sums the CTA's accumulators into out[K] (shared memory, ends with a barrier).
template <int NT, int K>
__device__ __forceinline__ void block_moments(double (&acc)[K], double (*sh)[K], double* out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
    if (lane == 0) sh[warp][k] = acc[k];
  }
  __syncthreads();
  if (threadIdx.x < K) {
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < NT / 32; ++w) t += sh[w][threadIdx.x];
    out[threadIdx.x] = t;
  }
  __syncthreads();
}

// The sums of up to kWarpChans channels by one warp: sum k^2 and sum (k - mean k)^2.
__device__ __forceinline__ void warp_channel_sums(const float* __restrict__ freqs, size_t chans,
                                                  double& k2, double& var) {
  const int lane = threadIdx.x & 31;
  double s = 0.0;
  for (size_t c = lane; c < chans; c += 32) s += (double)freqs[c] / kLight;
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  const double mean = s / (double)chans;
  k2 = 0.0;
  var = 0.0;
  for (size_t c = lane; c < chans; c += 32) {
    const double k = (double)freqs[c] / kLight, d = k - mean;
    k2 += k * k;
    var += d * d;
  }
  for (int o = 16; o > 0; o >>= 1) {
    k2 += __shfl_xor_sync(0xffffffffu, k2, o);
    var += __shfl_xor_sync(0xffffffffu, var, o);
  }
}

// One Jacobi rotation in the plane (P, Q) of a symmetric 3 x 3 matrix a
// (row-major, both triangles kept) with its accumulated rotations q.  The
// angle's tangent t is FP32 (it only decides how far the off-diagonal entry
// shrinks: seven digits a rotation); the rotation itself is orthogonal to
// FP64: c = 1 / sqrt(1 + t^2) by two Newton steps on an FP32 estimate, s = t c.
template <int P, int Q>
__device__ __forceinline__ void jacobi_rotate(double (&a)[9], double (&q)[9]) {
  const double apq = a[P * 3 + Q];
  if (apq == 0.0) return;
  const float tau = (float)((a[Q * 3 + Q] - a[P * 3 + P]) / (2.0 * apq));
  const float at = fabsf(tau);
  // |tau| beyond FP32's squares: the tangent is 1 / (2 tau).
  const float tf = at > 1e18f ? 0.5f / at : 1.0f / (at + sqrtf(1.0f + at * at));
  const double t = (double)(tau >= 0.f ? tf : -tf);
  const double u = 1.0 + t * t;
  double c = (double)rsqrtf((float)u);
  c = c * (1.5 - 0.5 * u * c * c);
  c = c * (1.5 - 0.5 * u * c * c);
  const double s = t * c;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double x = a[k * 3 + P], y = a[k * 3 + Q];
    a[k * 3 + P] = c * x - s * y;
    a[k * 3 + Q] = s * x + c * y;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double x = a[P * 3 + k], y = a[Q * 3 + k];
    a[P * 3 + k] = c * x - s * y;
    a[Q * 3 + k] = s * x + c * y;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double x = q[k * 3 + P], y = q[k * 3 + Q];
    q[k * 3 + P] = c * x - s * y;
    q[k * 3 + Q] = s * x + c * y;
  }
}

// The basis from the moments (one thread): cyclic Jacobi of the covariance
// over its trace, until the off-diagonal part is 1e-16 of it (its rounding; a handful of
// sweeps, all in registers), then the principal axes in descending order,
// each signed so its largest-magnitude component is positive
// (SVDPreprocessKernels.cu:115-206).
__device__ __forceinline__ void plane_basis(const double* mom, const float* __restrict__ uvw,
                                            size_t rows, size_t chans, double k2, double kvar,
                                            double (&b)[6]) {
  const double inv = 1.0 / (double)rows;
  const double m0 = mom[0] * inv, m1 = mom[1] * inv, m2 = mom[2] * inv;  // of u'
  const double g0 = m0 + uvw[0], g1 = m1 + uvw[1], g2 = m2 + uvw[2];     // of u
  const double vr = kvar * (double)rows;
  double a[9];
  a[0] = k2 * (mom[3] - mom[0] * m0) + vr * g0 * g0;
  a[1] = k2 * (mom[4] - mom[0] * m1) + vr * g0 * g1;
  a[2] = k2 * (mom[5] - mom[0] * m2) + vr * g0 * g2;
  a[4] = k2 * (mom[6] - mom[1] * m1) + vr * g1 * g1;
  a[5] = k2 * (mom[7] - mom[1] * m2) + vr * g1 * g2;
  a[8] = k2 * (mom[8] - mom[2] * m2) + vr * g2 * g2;
  const double tr = a[0] + a[4] + a[8];
  const double sc = tr > 0.0 ? 1.0 / tr : 1.0;
  a[0] *= sc; a[1] *= sc; a[2] *= sc; a[4] *= sc; a[5] *= sc; a[8] *= sc;
  a[3] = a[1]; a[6] = a[2]; a[7] = a[5];
  double q[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
  for (int sweep = 0; sweep < 16; ++sweep) {
    if (a[1] * a[1] + a[2] * a[2] + a[5] * a[5] <= 1e-32) break;
    jacobi_rotate<0, 1>(a, q);
    jacobi_rotate<0, 2>(a, q);
    jacobi_rotate<1, 2>(a, q);
  }
  const double d0 = a[0], d1 = a[4], d2 = a[8];
  // Largest, then the larger of the other two (ties to the lower index).
  const int big = d1 > d0 ? (d2 > d1 ? 2 : 1) : (d2 > d0 ? 2 : 0);
  const int lo = big == 0 ? 1 : 0, hi = big == 2 ? 1 : 2;
  const double dl = lo == 0 ? d0 : d1, dh = hi == 1 ? d1 : d2;
  const int mid = dh > dl ? hi : lo;
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    b[r] = big == 0 ? q[3 * r] : (big == 1 ? q[3 * r + 1] : q[3 * r + 2]);
    b[3 + r] = mid == 0 ? q[3 * r] : (mid == 1 ? q[3 * r + 1] : q[3 * r + 2]);
  }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const double x = b[3 * r], y = b[3 * r + 1], z = b[3 * r + 2];
    double l = x;
    if (fabs(y) > fabs(l)) l = y;
    if (fabs(z) > fabs(l)) l = z;
    if (l < 0.0) {
      b[3 * r] = -x;
      b[3 * r + 1] = -y;
      b[3 * r + 2] = -z;
    }
  }
}

// V: the two axes and their cross product.
__device__ __forceinline__ void write_basis(const double* b, float* V) {
  for (int k = 0; k < 6; ++k) V[k] = (float)b[k];
  V[6] = (float)(b[1] * b[5] - b[2] * b[4]);
  V[7] = (float)(b[2] * b[3] - b[0] * b[5]);
  V[8] = (float)(b[0] * b[4] - b[1] * b[3]);
}

// B[s] = x_s . basis^T, uncentred (SVDPreprocessKernels.cu:142-165), of rows
// r0, r0 + step, ... and channels [c0, c1), samples >= skip: a row's two
// projections once, scaled per channel.  ksc: k of channel c0 + i (shared).
__device__ __forceinline__ void project_rows(const float* __restrict__ uvw, size_t rows,
                                             size_t r0, size_t step, size_t c0, size_t c1,
                                             const double* ksc, const double* b, size_t skip,
                                             float* B) {
  const bool pair = (reinterpret_cast<uintptr_t>(B) & 7) == 0;
  const double b0 = b[0], b1 = b[1], b2 = b[2], b3 = b[3], b4 = b[4], b5 = b[5];
  for (size_t r = r0; r < rows; r += step) {
    const double x = uvw[3 * r], y = uvw[3 * r + 1], z = uvw[3 * r + 2];
    const double p = x * b0 + y * b1 + z * b2, w = x * b3 + y * b4 + z * b5;
    for (size_t c = c0; c < c1; ++c) {
      const size_t s = r + c * rows;
      const double k = ksc[c - c0];
      if (s < skip) continue;
      if (pair) {
        reinterpret_cast<float2*>(B)[s] = make_float2((float)(p * k), (float)(w * k));
      } else {
        B[2 * s] = (float)(p * k);
        B[2 * s + 1] = (float)(w * k);
      }
    }
  }
}

// The same of samples s0, s0 + step, ... >= skip, one at a time: for few rows.
__device__ __forceinline__ void project_samples(const float* __restrict__ uvw,
                                                const float* __restrict__ freqs, size_t rows,
                                                size_t ns, size_t s0, size_t step,
                                                const double* b, size_t skip, float* B) {
  const bool pair = (reinterpret_cast<uintptr_t>(B) & 7) == 0;
  const double b0 = b[0], b1 = b[1], b2 = b[2], b3 = b[3], b4 = b[4], b5 = b[5];
  for (size_t s = s0; s < ns; s += step) {
    if (s < skip) continue;
    const size_t c = s / rows, r = s - c * rows;
    const double x = uvw[3 * r], y = uvw[3 * r + 1], z = uvw[3 * r + 2];
    const double p = x * b0 + y * b1 + z * b2, w = x * b3 + y * b4 + z * b5;
    const double k = (double)freqs[c] / kLight;
    if (pair) {
      reinterpret_cast<float2*>(B)[s] = make_float2((float)(p * k), (float)(w * k));
    } else {
      B[2 * s] = (float)(p * k);
      B[2 * s + 1] = (float)(w * k);
    }
  }
}

constexpr int kPlaneCluster = 8, kPlaneThreads = 1024;
constexpr int kPlaneChans = 256;  // channels staged at a time
// Rows below which the projection goes by sample, one cluster's and the spread
// form's: a quarter of the cluster's threads, one CTA's threads.
constexpr size_t kFewRowsOne = 2048, kFewRows = kThreads;

// The whole fit in one cluster: moments of an eighth of the rows per CTA,
// summed through distributed shared memory (the same order in every CTA), the
// basis by one thread of each CTA, the projection of the CTA's rows.
__global__ void __cluster_dims__(kPlaneCluster, 1, 1) __launch_bounds__(kPlaneThreads)
    k_plane_fit(const float* __restrict__ uvw, const float* __restrict__ freqs, size_t rows,
                size_t chans, float* B, float* V) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ double s_warp[kPlaneThreads / 32][kMom];
  __shared__ double s_chan[kPlaneThreads / 32][kChan];
  __shared__ double s_mom[kMom], s_all[kMom], s_b[6], s_k[kPlaneChans], s_ch[kChan];
  const size_t first = blockIdx.x * (size_t)kPlaneThreads + threadIdx.x;
  const size_t step = (size_t)kPlaneCluster * kPlaneThreads;
  double acc[kMom];
  row_moments(uvw, rows, first, step, acc);
  block_moments<kPlaneThreads>(acc, s_warp, s_mom);
  if (chans <= kWarpChans) {
    if (threadIdx.x >= kPlaneThreads - 32) {
      double k2, var;
      warp_channel_sums(freqs, chans, k2, var);
      if (threadIdx.x == kPlaneThreads - 1) {
        s_ch[0] = k2;
        s_ch[1] = var;
      }
    }
  } else {  // by every CTA for itself
    double ch[kChan], k2, var;
    channel_moments(freqs, chans, threadIdx.x, kPlaneThreads, ch);
    block_moments<kPlaneThreads>(ch, s_chan, s_ch);
    channel_sums(s_ch, freqs, chans, k2, var);
    __syncthreads();
    if (threadIdx.x == 0) {
      s_ch[0] = k2;
      s_ch[1] = var;
    }
  }
  cluster.sync();
  if (threadIdx.x < kMom) {
    double t = 0.0;
    for (int c = 0; c < kPlaneCluster; ++c) t += cluster.map_shared_rank(s_mom, c)[threadIdx.x];
    s_all[threadIdx.x] = t;
  }
  cluster.sync();  // every CTA has read the others' sums
  if (threadIdx.x == 0) {
    double b[6];
    plane_basis(s_all, uvw, rows, chans, s_ch[0], s_ch[1], b);
    for (int k = 0; k < 6; ++k) s_b[k] = b[k];
    if (blockIdx.x == 0) write_basis(b, V);
  }
  if (rows < kFewRowsOne && chans > 1) {
    __syncthreads();
    project_samples(uvw, freqs, rows, rows * chans, first, step, s_b, 0, B);
    return;
  }
  for (size_t c0 = 0; c0 < chans; c0 += kPlaneChans) {
    const size_t c1 = c0 + kPlaneChans < chans ? c0 + kPlaneChans : chans;
    __syncthreads();
    if (c0 + threadIdx.x < c1) s_k[threadIdx.x] = (double)freqs[c0 + threadIdx.x] / kLight;
    __syncthreads();
    project_rows(uvw, rows, first, step, c0, c1, s_k, s_b, 0, B);
  }
}

// The large form.  A double as two 4-byte words at p (B need not be 8-byte
// aligned).
__device__ __forceinline__ void put_words(float* p, double v) {
  p[0] = __int_as_float(__double2loint(v));
  p[1] = __int_as_float(__double2hiint(v));
}
__device__ __forceinline__ double get_words(const float* p) {
  return __hiloint2double(__float_as_int(p[1]), __float_as_int(p[0]));
}
constexpr int kSums = kMom + kChan;
constexpr int kPlaneParts = kSms;  // moment CTAs; their sums fill 22 floats of B each
constexpr size_t kPlaneStash = 6;  // samples whose B slots hold the basis until the end

__global__ void __launch_bounds__(kThreads) k_plane_moments(const float* __restrict__ uvw,
                                                            const float* __restrict__ freqs,
                                                            size_t rows, size_t chans, float* B) {
  __shared__ double s_warp[kThreads / 32][kMom], s_chan[kThreads / 32][kChan], s_mom[kSums];
  const size_t first = blockIdx.x * (size_t)kThreads + threadIdx.x;
  const size_t step = (size_t)gridDim.x * kThreads;
  double acc[kMom];
  row_moments(uvw, rows, first, step, acc);
  block_moments<kThreads>(acc, s_warp, s_mom);
  const bool many = chans > kWarpChans;
  if (many) {
    double ch[kChan];
    channel_moments(freqs, chans, first, step, ch);
    block_moments<kThreads>(ch, s_chan, s_mom + kMom);
  }
  if (threadIdx.x < (many ? kSums : kMom))
    put_words(B + 2 * ((size_t)blockIdx.x * kSums + threadIdx.x), s_mom[threadIdx.x]);
}

// One CTA: the partial sums (one moment per warp, ascending within a lane),
// the basis into V and, as FP64, the head of B.
__global__ void __launch_bounds__(kSums * 32) k_plane_basis(const float* __restrict__ uvw,
                                                           const float* __restrict__ freqs,
                                                           size_t rows, size_t chans, int parts,
                                                           float* B, float* V) {
  __shared__ double s_mom[kSums];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool many = chans > kWarpChans;
  if (warp < kMom || many) {
    double t = 0.0;
    for (int p = lane; p < parts; p += 32) t += get_words(B + 2 * ((size_t)p * kSums + warp));
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) s_mom[warp] = t;
  }
  double k2 = 0.0, var = 0.0;
  if (warp == 0 && !many) warp_channel_sums(freqs, chans, k2, var);
  __syncthreads();
  if (threadIdx.x == 0) {
    if (many) channel_sums(s_mom + kMom, freqs, chans, k2, var);
    double b[6];
    plane_basis(s_mom, uvw, rows, chans, k2, var, b);
    for (int k = 0; k < 6; ++k) put_words(B + 2 * k, b[k]);
    write_basis(b, V);
  }
}

// Samples kPlaneStash .. ns - 1: CTA (x, y) takes row blocks x, x + gridDim.x,
// ... of channel blocks y, y + gridDim.y, ... of per_y channels (at most
// kPlaneChans).
__global__ void __launch_bounds__(kThreads) k_plane_project(const float* __restrict__ uvw,
                                                            const float* __restrict__ freqs,
                                                            size_t rows, size_t chans,
                                                            size_t per_y, float* B) {
  __shared__ double s_k[kPlaneChans];
  double b[6];
  for (int k = 0; k < 6; ++k) b[k] = get_words(B + 2 * k);
  for (size_t c0 = blockIdx.y * per_y; c0 < chans; c0 += gridDim.y * per_y) {
    const size_t c1 = c0 + per_y < chans ? c0 + per_y : chans;
    for (size_t c = c0 + threadIdx.x; c < c1; c += kThreads)
      s_k[c - c0] = (double)freqs[c] / kLight;
    __syncthreads();
    project_rows(uvw, rows, blockIdx.x * (size_t)kThreads + threadIdx.x,
                 (size_t)gridDim.x * kThreads, c0, c1, s_k, b, kPlaneStash, B);
    __syncthreads();
  }
}

// The same of fewer than kFewRows rows.
__global__ void __launch_bounds__(kThreads) k_plane_project_few(const float* __restrict__ uvw,
                                                                const float* __restrict__ freqs,
                                                                size_t rows, size_t chans,
                                                                float* B) {
  double b[6];
  for (int k = 0; k < 6; ++k) b[k] = get_words(B + 2 * k);
  project_samples(uvw, freqs, rows, rows * chans, blockIdx.x * (size_t)kThreads + threadIdx.x,
                  (size_t)gridDim.x * kThreads, b, kPlaneStash, B);
}

// The samples whose slots held the basis (one warp).
__global__ void k_plane_tail(const float* __restrict__ uvw, const float* __restrict__ freqs,
                             size_t rows, float* B) {
  double b[6];
  for (int k = 0; k < 6; ++k) b[k] = get_words(B + 2 * k);
  __syncthreads();
  const size_t s = threadIdx.x;
  if (s < kPlaneStash) {
    const size_t r = s % rows, c = s / rows;
    const double k = (double)freqs[c] / kLight;
    const double x = uvw[3 * r], y = uvw[3 * r + 1], z = uvw[3 * r + 2];
    B[2 * s] = (float)((x * b[0] + y * b[1] + z * b[2]) * k);
    B[2 * s + 1] = (float)((x * b[3] + y * b[4] + z * b[5]) * k);
  }
}

// SVDPreprocessKernels.cu:208-237.
__global__ void k_collapse(const float* v0r, const float* v0i, const float* v3r, const float* v3i,
                           const unsigned char* f0, const unsigned char* f3, const float* w0,
                           const float* w3, float* out_re, float* out_im, size_t ns) {
  const FipRawVis r{v0r, v0i, v3r, v3i, f0, f3, w0, w3};
  for (size_t s = blockIdx.x * (size_t)kThreads + threadIdx.x; s < ns;
       s += (size_t)gridDim.x * kThreads)
    fip_collapse_sample(r, s, out_re[s], out_im[s]);
}

// Sample k of the visibilities: FP32 arrays, or raw polarisations collapsed
// to Stokes I on load.
struct F32Vis {
  const float* vr;
  const float* vi;
  __device__ __forceinline__ void operator()(size_t k, float& re, float& im) const {
    re = vr[k];
    im = vi[k];
  }
  __device__ __forceinline__ F32Vis at(size_t off) const { return F32Vis{vr + off, vi + off}; }
};
struct RawVis {
  FipRawVis r;
  __device__ __forceinline__ void operator()(size_t k, float& re, float& im) const {
    fip_collapse_sample(r, k, re, im);
  }
  __device__ __forceinline__ RawVis at(size_t) const { return *this; }  // one snapshot per launch
};

// One block of FIP_QBLOCK samples per CTA (kThreads threads, four samples
// each): the block's max-abs, its power-of-two scale 2^(e - 14) for a max-abs
// in [2^e, 2^(e+1)) (so the max lands in [2^14, 2^15), inside FP16's range,
// and the division by the scale is exact), then the values divided by it.
// Batched launches: snapshot blockIdx.y, counts.nb[blockIdx.y] samples.
template <int VT, class L>
__global__ void __launch_bounds__(kThreads) k_quantize(const L load0,
                                                       const __grid_constant__ FipCounts counts,
                                                       void* qr, void* qi, float* scales,
                                                       size_t in_stride, size_t out_stride) {
  const size_t nb = counts.nb[blockIdx.y];
  const L load = load0.at(blockIdx.y * in_stride);
  qr = static_cast<uint16_t*>(qr) + blockIdx.y * out_stride;
  qi = static_cast<uint16_t*>(qi) + blockIdx.y * out_stride;
  scales += blockIdx.y * fip_qblocks(out_stride);
  static_assert(FIP_QBLOCK == 4 * kThreads, "four samples per thread");
  __shared__ float s_max[kThreads / 32];
  const size_t base = (size_t)blockIdx.x * FIP_QBLOCK;
  if (base >= nb) return;  // a shorter snapshot than the launch's longest
  float re[4], im[4];
  float m = 0.f;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const size_t i = base + (size_t)k * kThreads + threadIdx.x;
    re[k] = 0.f;
    im[k] = 0.f;
    if (i < nb) load(i, re[k], im[k]);
    m = fmaxf(m, fmaxf(fabsf(re[k]), fabsf(im[k])));
  }
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = m;
  __syncthreads();
  m = s_max[0];
#pragma unroll
  for (int w = 1; w < kThreads / 32; ++w) m = fmaxf(m, s_max[w]);
  // The max's biased exponent E gives scale 2^(E - 141) (bits E - 14) and
  // inverse 2^(141 - E) (bits 268 - E).  E is held >= 15 so both are normal:
  // a block whose max is below 2^-112 (zero included) takes scale 2^-126.
  const int eb = max((int)((__float_as_uint(m) >> 23) & 0xffu), 15);
  const float scale = __uint_as_float((unsigned)(eb - 14) << 23);
  const float inv = __uint_as_float((unsigned)(268 - eb) << 23);
  if (threadIdx.x == 0) scales[blockIdx.x] = scale;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const size_t i = base + (size_t)k * kThreads + threadIdx.x;
    if (i >= nb) continue;
    if (VT == FIP_VIS_F16) {
      reinterpret_cast<__half*>(qr)[i] = __float2half_rn(re[k] * inv);
      reinterpret_cast<__half*>(qi)[i] = __float2half_rn(im[k] * inv);
    } else {
      reinterpret_cast<__nv_bfloat16*>(qr)[i] = __float2bfloat16_rn(re[k] * inv);
      reinterpret_cast<__nv_bfloat16*>(qi)[i] = __float2bfloat16_rn(im[k] * inv);
    }
  }
}

}  // namespace

// One cluster while its eight SMs keep up; beyond it the moments and the
// projection spread over the device (a call, launches included: 32,640 rows
// 14.4 us in one cluster against 20.5 us spread, 130,816 rows 22.6 against
// 21.5 us).
constexpr size_t kPlaneOneCluster = (size_t)1 << 16;

cudaError_t fip_launch_plane_project(const float* uvw, const float* freqs, size_t rows,
                                     size_t chans, float* B, float* V, cudaStream_t s) {
  const size_t ns = rows * chans;
  if (ns <= kPlaneOneCluster) {
    k_plane_fit<<<kPlaneCluster, kPlaneThreads, 0, s>>>(uvw, freqs, rows, chans, B, V);
    return cudaGetLastError();
  }
  const size_t most = chans > kWarpChans ? std::max(rows, chans) : rows;
  const int parts = (int)std::min<size_t>(kPlaneParts, (most + kThreads - 1) / kThreads);
  k_plane_moments<<<parts, kThreads, 0, s>>>(uvw, freqs, rows, chans, B);
  k_plane_basis<<<1, kSums * 32, 0, s>>>(uvw, freqs, rows, chans, parts, B, V);
  if (rows < kFewRows) {
    const unsigned blocks = (unsigned)std::min<size_t>(8 * kSms, (ns + kThreads - 1) / kThreads);
    k_plane_project_few<<<blocks, kThreads, 0, s>>>(uvw, freqs, rows, chans, B);
    k_plane_tail<<<1, 32, 0, s>>>(uvw, freqs, rows, B);
    return cudaGetLastError();
  }
  // About four CTAs per SM: rows first, channels where the rows are few.
  const size_t bx = std::min<size_t>(4 * kSms, (rows + kThreads - 1) / kThreads);
  const size_t want_y = (4 * kSms + bx - 1) / bx;
  size_t per_y = std::max<size_t>(1, (chans + want_y - 1) / want_y);
  per_y = std::min<size_t>(per_y, kPlaneChans);
  const size_t by = std::min<size_t>(65535, (chans + per_y - 1) / per_y);
  k_plane_project<<<dim3((unsigned)bx, (unsigned)by), kThreads, 0, s>>>(uvw, freqs, rows, chans,
                                                                        per_y, B);
  k_plane_tail<<<1, 32, 0, s>>>(uvw, freqs, rows, B);
  return cudaGetLastError();
}

cudaError_t fip_launch_collapse(const float* v0r, const float* v0i, const float* v3r,
                                const float* v3i, const unsigned char* f0,
                                const unsigned char* f3, const float* w0, const float* w3,
                                float* out_re, float* out_im, size_t ns, cudaStream_t s) {
  const int blocks = (int)std::min<size_t>(4 * kSms, (ns + kThreads - 1) / kThreads + 1);
  k_collapse<<<blocks, kThreads, 0, s>>>(v0r, v0i, v3r, v3i, f0, f3, w0, w3, out_re, out_im, ns);
  return cudaGetLastError();
}

template <class L>
static cudaError_t launch_quantize(const L& load, const size_t* nb, int vis_type, void* out_re,
                                  void* out_im, float* scales, cudaStream_t s, int batch = 1,
                                  size_t in_stride = 0, size_t out_stride = 0) {
  if (batch < 1 || batch > FIP_MAX_BATCH) return cudaErrorInvalidValue;
  FipCounts counts{};
  size_t blocks = 0;
  for (int k = 0; k < batch; ++k) {
    counts.nb[k] = (unsigned)nb[k];
    if (counts.nb[k] != nb[k]) return cudaErrorInvalidValue;
    blocks = std::max(blocks, fip_qblocks(nb[k]));
  }
  if (blocks == 0) return cudaSuccess;
  if (vis_type == FIP_VIS_F16)
    k_quantize<FIP_VIS_F16><<<dim3((unsigned)blocks, batch), kThreads, 0, s>>>(
        load, counts, out_re, out_im, scales, in_stride, out_stride);
  else
    k_quantize<FIP_VIS_BF16><<<dim3((unsigned)blocks, batch), kThreads, 0, s>>>(
        load, counts, out_re, out_im, scales, in_stride, out_stride);
  return cudaGetLastError();
}

cudaError_t fip_launch_quantize(const float* vr, const float* vi, const size_t* nb, int vis_type,
                                void* out_re, void* out_im, float* scales, cudaStream_t s,
                                int batch, size_t in_stride, size_t out_stride) {
  return launch_quantize(F32Vis{vr, vi}, nb, vis_type, out_re, out_im, scales, s, batch,
                         in_stride, out_stride);
}

cudaError_t fip_launch_quantize_raw(const FipRawVis& raw, size_t nb, int vis_type, void* out_re,
                                    void* out_im, float* scales, cudaStream_t s) {
  return launch_quantize(RawVis{raw}, &nb, vis_type, out_re, out_im, scales, s);
}
