// Device stages of the snapshot imaging + tLISI trigger path.
//
// This translation unit is compiled with --use_fast_math, the flags of the
// reference's CUDA build (reference Makefile:13), because the plain FP32 form
// reproduces the reference's FP32 arithmetic (fip_refmath.cuh).  Data
// movement is B200-native:
//   * gridding bins every visibility by 64x64 tile of the Hermitian half-plane
//     uv grid; a thread per visibility of a work item takes its footprint
//     and kernel values into registers and adds its in-tile taps into the
//     tile in shared memory (int32 fixed point), which is committed once
//     (plain stores for tiles owned by one work item, vector reductions for
//     the few dense tiles split over several); only tiles inside the
//     occupied uv band are written;
//   * the 2-D inverse FFT is band-pruned: column transforms run only over the
//     occupied half-plane columns and keep only the N needed outputs; row
//     transforms pack two real image rows into one complex transform and
//     apply the grid correction in their epilogue (fip_fft.cuh);
//   * the reference's pixel mapping (compute-bound) runs on a side stream
//     while gridding and the FFT run, and reprojection is destination-tile
//     major: each 64x64 output tile gathers its candidate source pixels,
//     splats them in shared memory, stores the tile once and reports its
//     maximum -- no global atomics, no memsets;
//   * the trigger reads the three images once, in 128-bit loads, with
//     warp-shuffle tile reductions; a batch's sliding window streams each
//     tile's slices through registers, every image read once for all the
//     triples it is in.
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>

#include "fip_common.cuh"
#include "fip_fft.cuh"
#include "fip_kernels.h"
#include "fip_map.cuh"
#include "fip_refmath.cuh"

namespace {

constexpr int kThreads = 256;

// Grid row of signed row index v in [-G, G): v mod G without a division.
__device__ __forceinline__ int wrap_row(int v, int g) { return v < 0 ? v + g : (v >= g ? v - g : v); }

// ---------------------------------------------------------------------------
// Taper (FIPkernels.cu:173-186)
// ---------------------------------------------------------------------------
// taper[t] for t <= N/2, then the reciprocal correction
// taper[N/2 + 1 + t] = 1 / (taper[t] norm) that the row transform applies.
__global__ void k_taper(float* taper, size_t n, size_t g) {
  size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (t < n / 2 + 1) {
    const float c = fipref::taper(t, g);
    taper[t] = c;
    taper[n / 2 + 1 + t] = (float)(1.0 / ((double)c * (double)FIP_CONV_NORM));
  }
}

// ---------------------------------------------------------------------------
// Visibility footprint (FIPkernels.cu:211-219): taps [a0,a1] x [b0,b1],
// clamped to the grid.  Returns false when empty.
// ---------------------------------------------------------------------------
struct Footprint {
  float p1, p2;
  int a0, a1, b0, b1;
};

// Positions beyond 1e9 cells (and NaN) have no footprint; the rest convert
// exactly to 32-bit integers.
__device__ __forceinline__ bool footprint(float b0, float b1, float scale, int g, Footprint& f) {
  const float hs = (float)(FIP_SUPPORT / 2);
  const int gmin = -(g / 2), gmax = (g - 1) / 2;
  f.p1 = __fmul_rn(b0, scale);
  f.p2 = __fmul_rn(b1, scale);
  if (!(fabsf(f.p1) < 1e9f && fabsf(f.p2) < 1e9f)) {
    f.a0 = f.b0 = 0;
    f.a1 = f.b1 = -1;
    return false;
  }
  f.a0 = max((int)ceilf(f.p1 - hs), gmin);
  f.a1 = min((int)floorf(f.p1 + hs), gmax);
  f.b0 = max((int)ceilf(f.p2 - hs), gmin);
  f.b1 = min((int)floorf(f.p2 + hs), gmax);
  return f.a0 <= f.a1 && f.b0 <= f.b1;
}

// Half-plane image of a virtual visibility.  The grid holds the Hermitian
// part h(r) = (g(r) + conj g(-r)) / 2 of the reference's grid g, whose real
// transform is the real part the reference keeps (FIPkernels.cu:266): the
// direct copy keeps taps with r2 >= 0 at (r1 mod G, r2), the mirrored copy
// (conjugated) keeps taps with r2 <= 0 at (-r1 mod G, -r2).  Columns are
// taken modulo G, so for even G a tap at r2 = -G/2 (the reference's first
// grid column, FIPkernels.cu:202) lies on the Nyquist column G/2 of the
// direct copy as well as of the mirrored one; a footprint spans 9 columns at
// most, so for G > 18 that column is then the direct copy's only one.
__device__ __forceinline__ bool half_cols(const Footprint& f, int mir, int g, int& c0, int& c1) {
  if (!mir) {
    if (f.b1 < 0) {
      if ((g & 1) == 0 && f.b0 == -(g / 2)) {
        c0 = c1 = g / 2;
        return true;
      }
      return false;
    }
    c0 = max(f.b0, 0); c1 = f.b1;
  } else {
    if (f.b0 > 0) return false;
    c0 = max(-f.b1, 0); c1 = -f.b0;
  }
  return true;
}

// Distinct tile rows touched by rows r1 in [a0,a1] (direct) or -r1
// (mirrored), modulo G.  At most 3.
__device__ __forceinline__ int tile_rows(const Footprint& f, int mir, int g, int* out) {
  // Signed row range [lo, hi] (<= 9 rows) wraps into at most two segments.
  const int lo = mir ? -f.a1 : f.a0, hi = mir ? -f.a0 : f.a1;
  int n = 0;
  auto add_segment = [&](int a, int b) {  // rows a..b within [0, g)
    for (int tr = a / FIP_GTILE; tr <= b / FIP_GTILE && n < 3; ++tr) {
      bool seen = false;
      for (int k = 0; k < n; ++k) seen |= (out[k] == tr);
      if (!seen) out[n++] = tr;
    }
  };
  if (lo < 0 && hi >= 0) {
    add_segment(lo + g, g - 1);
    add_segment(0, hi);
  } else if (hi >= g) {
    add_segment(lo, g - 1);
    add_segment(0, hi - g);
  } else {
    add_segment(wrap_row(lo, g), wrap_row(hi, g));
  }
  return n;
}

// Warp-aggregated increment of cnt[key]; returns this lane's slot.
__device__ __forceinline__ unsigned agg_inc(unsigned* cnt, unsigned key, unsigned active) {
  unsigned peers = __match_any_sync(active, key);
  int leader = __ffs(peers) - 1;
  unsigned rank = __popc(peers & ((1u << (threadIdx.x & 31)) - 1));
  unsigned base = 0;
  if ((int)(threadIdx.x & 31) == leader) base = atomicAdd(&cnt[key], (unsigned)__popc(peers));
  base = __shfl_sync(peers, base, leader);
  return base + rank;
}

// pass 0: count entries per tile and record the occupied band
// (bbox[0] = max |r1|, bbox[1] = max half-plane column); pass 1: scatter.
template <int PASS>
__global__ void k_bin(const float* __restrict__ B, int nb, float scale, int g, int tiles_c,
                      unsigned* cnt, const unsigned* __restrict__ offset, unsigned* entries,
                      unsigned* bbox) {
  int v = blockIdx.x * blockDim.x + threadIdx.x;
  Footprint f;
  bool ok = v < nb && footprint(B[2 * v], B[2 * v + 1], scale, g, f);
  unsigned k1 = 0, k2 = 0;
  if (ok) k1 = (unsigned)max(abs(f.a0), abs(f.a1));
  for (int mir = 0; mir < 2; ++mir) {
    int c0 = 0, c1 = -1, trs[3], ntr = 0;
    bool on = ok && half_cols(f, mir, g, c0, c1);
    if (on) {
      ntr = tile_rows(f, mir, g, trs);
      k2 = max(k2, (unsigned)c1);
    }
    int tc0 = on ? c0 / FIP_GTILE : 0, tc1 = on ? c1 / FIP_GTILE : -1;
    // Up to 3 x 2 (tile-row, tile-col) pairs; every lane walks the same
    // 6 slots so the warp-aggregated atomics stay converged.
    for (int s = 0; s < 6; ++s) {
      int kr = s >> 1, kc = s & 1;
      bool act = on && kr < ntr && tc0 + kc <= tc1;
      unsigned mask = __ballot_sync(0xffffffffu, act);
      if (act) {
        unsigned tile = (unsigned)(trs[kr] * tiles_c + tc0 + kc);
        unsigned slot = agg_inc(cnt, tile, mask);
        if (PASS == 1) entries[offset[tile] + slot] = ((unsigned)v << 1) | (unsigned)mir;
      }
    }
  }
  if (PASS == 0) {
    for (int o = 16; o > 0; o >>= 1) {
      k1 = max(k1, __shfl_xor_sync(0xffffffffu, k1, o));
      k2 = max(k2, __shfl_xor_sync(0xffffffffu, k2, o));
    }
    if ((threadIdx.x & 31) == 0) {
      atomicMax(&bbox[0], k1);
      atomicMax(&bbox[1], k2);
    }
  }
}

// Is grid tile t inside the band that the transform reads?
__device__ __forceinline__ bool in_band(int t, int tiles_c, int g, int layout,
                                        const unsigned* bbox) {
  if (layout == 0) return true;
  const int tr = t / tiles_c, tc = t % tiles_c;
  const int k1 = (int)bbox[0], k2 = (int)bbox[1];
  if (tc * FIP_GTILE > k2) return false;
  const int r0 = tr * FIP_GTILE, r1 = min(r0 + FIP_GTILE, g) - 1;
  return r0 <= k1 || r1 >= g - k1;
}

// Exclusive scans of tile counts, construction of the work list (every band
// tile gets >= 1 item, so the band is fully written), and the list of tiles
// split over several items (zeroed before their reductions).  One CTA of
// kScanThreads walks the tiles in coalesced chunks.
constexpr int kScanThreads = 1024;

__device__ __forceinline__ uint3 block_exclusive_scan(uint3 v, uint3& total) {
  __shared__ uint3 s_w[kScanThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint3 inc = v;
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned a = __shfl_up_sync(0xffffffffu, inc.x, o);
    const unsigned b = __shfl_up_sync(0xffffffffu, inc.y, o);
    const unsigned c = __shfl_up_sync(0xffffffffu, inc.z, o);
    if (lane >= o) {
      inc.x += a;
      inc.y += b;
      inc.z += c;
    }
  }
  if (lane == 31) s_w[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    uint3 w = lane < kScanThreads / 32 ? s_w[lane] : make_uint3(0, 0, 0);
    uint3 wi = w;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned a = __shfl_up_sync(0xffffffffu, wi.x, o);
      const unsigned b = __shfl_up_sync(0xffffffffu, wi.y, o);
      const unsigned c = __shfl_up_sync(0xffffffffu, wi.z, o);
      if (lane >= o) {
        wi.x += a;
        wi.y += b;
        wi.z += c;
      }
    }
    if (lane < kScanThreads / 32) s_w[lane] = make_uint3(wi.x - w.x, wi.y - w.y, wi.z - w.z);
  }
  __syncthreads();
  const uint3 base = s_w[warp];
  uint3 ex = make_uint3(base.x + inc.x - v.x, base.y + inc.y - v.y, base.z + inc.z - v.z);
  __shared__ uint3 s_total;
  if (threadIdx.x == kScanThreads - 1) s_total = make_uint3(ex.x + v.x, ex.y + v.y, ex.z + v.z);
  __syncthreads();
  total = s_total;
  __syncthreads();
  return ex;
}

__global__ void __launch_bounds__(kScanThreads) k_bin_scan(
    const unsigned* __restrict__ cnt, const unsigned* __restrict__ bbox, int ntiles, int tiles_c,
    int g, int layout, unsigned* offset, unsigned* cursor, int4* work, unsigned* nwork, int wcap,
    unsigned* multi, unsigned* nmulti) {
  uint3 carry = make_uint3(0, 0, 0);
  for (int base = 0; base < ntiles; base += kScanThreads) {
    const int t = base + threadIdx.x;
    unsigned c = 0, nch = 0;
    if (t < ntiles) {
      c = cnt[t];
      nch = in_band(t, tiles_c, g, layout, bbox) ? max(1u, (c + FIP_GCHUNK - 1) / FIP_GCHUNK)
                                                 : 0u;
    }
    uint3 total;
    const uint3 ex = block_exclusive_scan(make_uint3(c, nch, nch > 1 ? 1u : 0u), total);
    if (t < ntiles) {
      const unsigned run = carry.x + ex.x, wrun = carry.y + ex.y;
      offset[t] = run;
      cursor[t] = 0;
      for (unsigned k = 0; k < nch; ++k)
        if ((int)(wrun + k) < wcap)
          work[wrun + k] = make_int4(t, (int)(run + min(k * FIP_GCHUNK, c)),
                                     (int)(run + min((k + 1) * FIP_GCHUNK, c)), nch == 1);
      if (nch > 1) multi[carry.z + ex.z] = (unsigned)t;
    }
    carry.x += total.x;
    carry.y += total.y;
    carry.z += total.z;
  }
  if (threadIdx.x == 0) {
    offset[ntiles] = carry.x;
    *nwork = min(carry.y, (unsigned)wcap);
    *nmulti = carry.z;
  }
}

// ---------------------------------------------------------------------------
// Binning with per-CTA shared-memory histograms (grids of up to
// kMaxSmemTiles tiles), the snapshots of a call side by side (blockIdx.y).
// Each CTA takes a contiguous range of visibilities, counts their tile
// entries in shared memory (native integer atomics, one per entry: the
// hardware serialises lanes that hit one counter, cheaper than matching the
// lanes first), and adds its non-zero counts to the global ones, which
// returns where its entries start within each tile's list; one CTA per
// snapshot then scans the tiles; the scatter pass starts its shared-memory
// cursors from the two and fills the lists in one sweep.  A few CTAs per SM
// over the whole launch (fip_bin_ctas): more of them multiply the histograms'
// fixed cost (zeroing and merging every tile's counter), fewer leave the
// loads' latency exposed.
// Bound: the entries' integer arithmetic, then latency (three dependent
// launches).  1.05 M visibilities at 2048^2: 25 + 11 + 50 us (count, scan,
// scatter) with a recount in the scatter pass, 1,184 small CTAs and 64-bit
// footprint arithmetic, 16 + 8 + 19 us (the split tiles' zeroing included,
// a launch of its own before) in this form; eight snapshots of 0.45 M at
// 2048^2 435 -> 108 us of kernels.
// ---------------------------------------------------------------------------
constexpr int kBinThreads = 512;
constexpr int kBinUnroll = 4;         // visibilities in flight per thread
constexpr int kMaxSmemTiles = 12288;  // 48 KB of counters

// Visits the tile of every entry of a visibility at (b0, b1): f(tile, mir).
// A footprint's nine rows and columns touch two tile rows and columns at
// most, or the rows of both grid ends where it wraps.
template <class F>
__device__ __forceinline__ void for_each_entry(float b0, float b1, float scale, int g,
                                               int tiles_c, unsigned& k1, unsigned& k2, F&& f) {
  Footprint fp;
  if (!footprint(b0, b1, scale, g, fp)) return;
  k1 = max(k1, (unsigned)max(abs(fp.a0), abs(fp.a1)));
#pragma unroll
  for (int mir = 0; mir < 2; ++mir) {
    int c0, c1;
    if (!half_cols(fp, mir, g, c0, c1)) continue;
    k2 = max(k2, (unsigned)c1);
    const int rl = wrap_row(mir ? -fp.a1 : fp.a0, g), rh = wrap_row(mir ? -fp.a0 : fp.a1, g);
    const int t0 = rl / FIP_GTILE, t1 = (rl <= rh ? rh : g - 1) / FIP_GTILE;
    const int tc0 = c0 / FIP_GTILE, tc1 = c1 / FIP_GTILE;
    for (int tr = t0; tr <= t1; ++tr)
      for (int tc = tc0; tc <= tc1; ++tc) f((unsigned)(tr * tiles_c + tc), mir);
    if (rl > rh && t0 > 0)  // wrapped: the rows from 0 (a one-tile grid has them already)
      for (int tc = tc0; tc <= tc1; ++tc) f((unsigned)tc, mir);
  }
}

// Runs body(b0, b1, v) over the CTA's visibilities, kBinUnroll loads in
// flight per thread.
template <class F>
__device__ __forceinline__ void for_each_vis(const float* __restrict__ B, int v0, int v1,
                                             F&& body) {
  const bool pair = (reinterpret_cast<uintptr_t>(B) & 7) == 0;
  for (int base = v0; base < v1; base += kBinThreads * kBinUnroll) {
    float2 b[kBinUnroll];
#pragma unroll
    for (int q = 0; q < kBinUnroll; ++q) {
      const int v = base + q * kBinThreads + threadIdx.x;
      if (v < v1)
        b[q] = pair ? reinterpret_cast<const float2*>(B)[v] : make_float2(B[2 * v], B[2 * v + 1]);
    }
#pragma unroll
    for (int q = 0; q < kBinUnroll; ++q) {
      const int v = base + q * kBinThreads + threadIdx.x;
      if (v < v1) body(b[q].x, b[q].y, v);
    }
  }
}

template <int NT>
__device__ __forceinline__ uint3 block_scan3(uint3 v, uint3& total) {
  __shared__ uint3 s_w[NT / 32];
  __shared__ uint3 s_total;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint3 inc = v;
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned a = __shfl_up_sync(0xffffffffu, inc.x, o);
    const unsigned b = __shfl_up_sync(0xffffffffu, inc.y, o);
    const unsigned c = __shfl_up_sync(0xffffffffu, inc.z, o);
    if (lane >= o) {
      inc.x += a;
      inc.y += b;
      inc.z += c;
    }
  }
  if (lane == 31) s_w[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    const uint3 w = lane < NT / 32 ? s_w[lane] : make_uint3(0, 0, 0);
    uint3 wi = w;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned a = __shfl_up_sync(0xffffffffu, wi.x, o);
      const unsigned b = __shfl_up_sync(0xffffffffu, wi.y, o);
      const unsigned c = __shfl_up_sync(0xffffffffu, wi.z, o);
      if (lane >= o) {
        wi.x += a;
        wi.y += b;
        wi.z += c;
      }
    }
    if (lane < NT / 32) s_w[lane] = make_uint3(wi.x - w.x, wi.y - w.y, wi.z - w.z);
    if (lane == NT / 32 - 1) s_total = wi;
  }
  __syncthreads();
  const uint3 base = s_w[warp];
  total = s_total;
  __syncthreads();
  return make_uint3(base.x + inc.x - v.x, base.y + inc.y - v.y, base.z + inc.z - v.z);
}

// Count pass: per-CTA shared-memory counts added to count[] (base: the CTA's
// start within each tile's list), and the occupied band (bbox[0], bbox[1]).
// count and bbox are zero on entry.
__global__ void __launch_bounds__(kBinThreads) k_bin_count(
    const __grid_constant__ FipBinBatch in) {
  extern __shared__ unsigned s_hist[];
  __shared__ unsigned s_k[2];
  const FipBinSnap& sn = in.s[blockIdx.y];
  const int ntiles = sn.ntiles, g = sn.g, tiles_c = sn.tiles_c;
  const float scale = sn.scale;
  for (int t = threadIdx.x; t < ntiles; t += kBinThreads) s_hist[t] = 0;
  if (threadIdx.x < 2) s_k[threadIdx.x] = 0;
  __syncthreads();
  const int per_cta = (sn.nb + gridDim.x - 1) / gridDim.x;
  const int v0 = min(sn.nb, (int)blockIdx.x * per_cta), v1 = min(sn.nb, v0 + per_cta);
  unsigned k1 = 0, k2 = 0;
  for_each_vis(sn.B, v0, v1, [&](float b0, float b1, int) {
    for_each_entry(b0, b1, scale, g, tiles_c, k1, k2,
                   [&](unsigned tile, int) { atomicAdd(&s_hist[tile], 1u); });
  });
  k1 = __reduce_max_sync(0xffffffffu, k1);
  k2 = __reduce_max_sync(0xffffffffu, k2);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&s_k[0], k1);
    atomicMax(&s_k[1], k2);
  }
  __syncthreads();
  if (sn.base) {
    unsigned* base = sn.base + (size_t)blockIdx.x * ntiles;
    for (int t = threadIdx.x; t < ntiles; t += kBinThreads)
      if (s_hist[t]) base[t] = atomicAdd(&sn.count[t], s_hist[t]);
  } else {
    for (int t = threadIdx.x; t < ntiles; t += kBinThreads)
      if (s_hist[t]) atomicAdd(&sn.count[t], s_hist[t]);
  }
  if (threadIdx.x == 0) {
    atomicMax(&sn.bbox[0], s_k[0]);
    atomicMax(&sn.bbox[1], s_k[1]);
  }
}

// Tile scan over the final counts, one CTA of kScanThreads per snapshot:
// offsets, cursors, the work list (every band tile gets >= 1 item) and the
// list of tiles split over several items.  A thread scans kScanPer
// consecutive tiles and writes their first work items; the split tiles'
// further items are written by a warp per tile in a second sweep, so a tile
// with thousands of entries does not serialise on one thread.
constexpr int kScanPer = 8;
__global__ void __launch_bounds__(kScanThreads) k_bin_scan_tiles(
    const __grid_constant__ FipBinBatch in) {
  extern __shared__ unsigned s_wp[];  // [ntiles] first work item of each split tile
  const FipBinSnap& sn = in.s[blockIdx.x];
  const int ntiles = sn.ntiles, tiles_c = sn.tiles_c, g = sn.g;
  const unsigned wcap = sn.wcap, chunk = sn.chunk;
  const int k1 = (int)sn.bbox[0], k2 = (int)sn.bbox[1];
  const bool full = sn.layout == 0;
  uint3 carry = make_uint3(0, 0, 0);
  for (int base = 0; base < ntiles; base += kScanThreads * kScanPer) {
    const int t0 = base + threadIdx.x * kScanPer;
    unsigned c[kScanPer], nch[kScanPer];
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) c[k] = t0 + k < ntiles ? sn.count[t0 + k] : 0u;
    uint3 sum = make_uint3(0, 0, 0);
    int tr = t0 / tiles_c, tc = t0 - tr * tiles_c;
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) {
      const int r0 = tr * FIP_GTILE, r1 = min(r0 + FIP_GTILE, g) - 1;
      const bool band = full || (tc * FIP_GTILE <= k2 && (r0 <= k1 || r1 >= g - k1));
      nch[k] = t0 + k < ntiles && band ? max(1u, (c[k] + chunk - 1) / chunk) : 0u;
      if (++tc == tiles_c) {
        tc = 0;
        ++tr;
      }
      sum.x += c[k];
      sum.y += nch[k];
      sum.z += nch[k] > 1 ? 1u : 0u;
    }
    uint3 total;
    const uint3 ex = block_scan3<kScanThreads>(sum, total);
    unsigned run = carry.x + ex.x, wrun = carry.y + ex.y, mrun = carry.z + ex.z;
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) {
      const int t = t0 + k;
      if (t < ntiles) {
        sn.offset[t] = run;
        if (!sn.base) sn.cursor[t] = 0;
        if (nch[k] > 0 && wrun < wcap)
          sn.work[wrun] = make_int4(t, (int)run, (int)(run + min(chunk, c[k])),
                                    nch[k] == 1);
        if (nch[k] > 1) {
          sn.multi[mrun++] = (unsigned)t;
          s_wp[t] = wrun;
        }
        run += c[k];
        wrun += nch[k];
      }
    }
    carry.x += total.x;
    carry.y += total.y;
    carry.z += total.z;
  }
  if (threadIdx.x == 0) {
    if (sn.clear) *sn.clear = 0;
    sn.offset[ntiles] = carry.x;
    *sn.nwork = min(carry.y, wcap);
    *sn.nmulti = carry.z;
  }
  __syncthreads();
  for (unsigned m = threadIdx.x >> 5; m < carry.z; m += kScanThreads / 32) {
    const unsigned t = sn.multi[m], run = sn.offset[t], c = sn.count[t], w0 = s_wp[t];
    const unsigned n = (c + chunk - 1) / chunk;
    for (unsigned q = 1 + (threadIdx.x & 31); q < n; q += 32)
      if (w0 + q < wcap)
        sn.work[w0 + q] = make_int4((int)t, (int)(run + q * chunk),
                                    (int)(run + min((q + 1) * chunk, c)), 0);
  }
}

__device__ __forceinline__ size_t cell_index(int row, int col, int g, int hp, int layout) {
  return layout ? (size_t)col * g + row : (size_t)row * hp + col;
}

// Zeroes grid tile t (the CTA's threads together).
__device__ __forceinline__ void zero_tile(int t, int tiles_c, int g, int hp, int layout,
                                          float2* __restrict__ grid, int threads) {
  const int row0 = (t / tiles_c) * FIP_GTILE, col0 = (t % tiles_c) * FIP_GTILE;
  for (int k = threadIdx.x; k < FIP_GTILE * FIP_GTILE; k += threads) {
    const int lr = layout ? k % FIP_GTILE : k / FIP_GTILE;
    const int lc = layout ? k / FIP_GTILE : k % FIP_GTILE;
    const int row = row0 + lr, col = col0 + lc;
    if (row < g && col < hp) grid[cell_index(row, col, g, hp, layout)] = make_float2(0.f, 0.f);
  }
}

// Scatter pass: entries of the CTA's visibility range into the tile lists,
// and the split tiles of the grid zeroed (their work items reduce into them).
// Without the count pass's list positions (base) the range is recounted and
// reserves its slices from the cursors.
__global__ void __launch_bounds__(kBinThreads) k_bin_scatter(
    const __grid_constant__ FipBinBatch in) {
  extern __shared__ unsigned s_hist[];
  const FipBinSnap& sn = in.s[blockIdx.y];
  const int ntiles = sn.ntiles, g = sn.g, tiles_c = sn.tiles_c;
  const float scale = sn.scale;
  const int per_cta = (sn.nb + gridDim.x - 1) / gridDim.x;
  const int v0 = min(sn.nb, (int)blockIdx.x * per_cta), v1 = min(sn.nb, v0 + per_cta);
  unsigned k1 = 0, k2 = 0;
  if (sn.base) {
    const unsigned* base = sn.base + (size_t)blockIdx.x * ntiles;
    for (int t = threadIdx.x; t < ntiles; t += kBinThreads) s_hist[t] = sn.offset[t] + base[t];
  } else {
    for (int t = threadIdx.x; t < ntiles; t += kBinThreads) s_hist[t] = 0;
    __syncthreads();
    for_each_vis(sn.B, v0, v1, [&](float b0, float b1, int) {
      for_each_entry(b0, b1, scale, g, tiles_c, k1, k2,
                     [&](unsigned tile, int) { atomicAdd(&s_hist[tile], 1u); });
    });
    __syncthreads();
    for (int t = threadIdx.x; t < ntiles; t += kBinThreads) {
      const unsigned c = s_hist[t];
      if (c) s_hist[t] = sn.offset[t] + atomicAdd(&sn.cursor[t], c);
    }
  }
  __syncthreads();
  for_each_vis(sn.B, v0, v1, [&](float b0, float b1, int v) {
    for_each_entry(b0, b1, scale, g, tiles_c, k1, k2, [&](unsigned tile, int mir) {
      sn.entries[atomicAdd(&s_hist[tile], 1u)] = ((unsigned)v << 1) | (unsigned)mir;
    });
  });
  if (sn.grid) {
    const unsigned nm = *sn.nmulti;
    for (unsigned m = blockIdx.x; m < nm; m += gridDim.x)
      zero_tile((int)sn.multi[m], tiles_c, g, sn.hp, sn.layout, sn.grid, kBinThreads);
  }
}

// The split tiles of a snapshot whose grid has too many tiles for the
// binning above.
__global__ void k_zero_tiles(const unsigned* __restrict__ multi, const unsigned* __restrict__ nmulti,
                             int tiles_c, int g, int hp, int layout, float2* __restrict__ grid) {
  const unsigned nm = *nmulti;
  for (unsigned w = blockIdx.x; w < nm; w += gridDim.x)
    zero_tile((int)multi[w], tiles_c, g, hp, layout, grid, kThreads);
}

template <int VT>
__device__ __forceinline__ float load_vis(const void* p, int v) {
  if (VT == FIP_VIS_F32) return reinterpret_cast<const float*>(p)[v];
  if (VT == FIP_VIS_F16) return __half2float(reinterpret_cast<const __half*>(p)[v]);
  return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[v]);
}

// Shared-memory layout of one gridding work item: the tile (int32 fixed
// point) and the bound reduction; the precision form adds the tile's low
// limbs.
// Row stride: odd, so that the commit's walk down a column (the band layout's
// contiguous direction) reads 32 banks.  (With a stride of 72 that walk hit
// four banks, 38 % of the gridder's shared-memory wavefronts.)
constexpr int kTS = FIP_GTILE + 1;
static_assert(FIP_GTILE * kTS % 4 == 0, "the tile is zeroed in 16-byte stores");
struct GridSmem {
  float bound[kThreads / 32];
  // Real and imaginary sums (plain form, or the high limbs), then the
  // precision form's low limbs.
  float tile[2 * FIP_GTILE * kTS];
};
// Dynamic shared memory of a gridding CTA.
__host__ __device__ constexpr size_t grid_smem_bytes(bool comp) {
  return sizeof(GridSmem) + (comp ? 2 * FIP_GTILE * kTS * sizeof(float) : 0);
}

// Weights of one entry: the visibility (FIPkernels.cu:188-195), halved for the
// Hermitian split, conjugated for the mirrored copy.
template <int VT>
__device__ __forceinline__ void entry_weights(const void* vr, const void* vi,
                                              const float* vis_scale, float inten, unsigned ent,
                                              const FipRawVis& raw, float& owr, float& owi) {
  const int v = (int)(ent >> 1), mir = (int)(ent & 1);
  float wr, wi;
  if constexpr (VT == FIP_VIS_RAW) {
    // Stokes-I collapse fused into the load: no collapsed copy in memory.
    float cr, ci;
    fip_collapse_sample(raw, (size_t)v, cr, ci);
    wr = cr / inten;
    wi = ci / inten;
  } else if constexpr (VT == FIP_VIS_F32) {
    wr = load_vis<VT>(vr, v) / inten;
    wi = load_vis<VT>(vi, v) / inten;
  } else {
    // Reduced storage: the value over its block's power-of-two scale.
    const float sc = vis_scale[v >> FIP_QBLOCK_SHIFT];
    wr = (load_vis<VT>(vr, v) * sc) / inten;
    wi = (load_vis<VT>(vi, v) * sc) / inten;
  }
  owr = 0.5f * wr;
  owi = mir ? -0.5f * wi : 0.5f * wi;
}

// One entry's taps inside a tile: its in-tile rows ia in [ia_lo, ia_hi) and
// columns ib in [ib_lo, ib_hi) of the footprint, the tile cell cell0 of tap
// (ia_lo, ib_lo), the row direction and the separable kernel values.
struct EntryTaps {
  int ia_lo, ia_hi, ib_lo, ib_hi, cell0, r1, mir;
  float k1[9], k2[9];
  __device__ bool empty() const { return ia_lo >= ia_hi || ib_lo >= ib_hi; }
};

// EXACT: a tap's distance r - b scale is one rounding of the exact difference, by
// explicit multiply-adds (precision form); else it is taken from the position
// rounded to FP32, the order of operations that the plain form keeps
// (FIPkernels.cu:199-219; half an ulp of hundreds of cells: the grid 1.3e-5 off in
// relative RMS at 1400^2 with baselines up to the grid's edge, against 5e-7).
template <bool EXACT>
__device__ __forceinline__ void entry_taps(const float* __restrict__ B, float scale, int g,
                                           unsigned ent, int trow0, int tcol0, EntryTaps& e) {
  const int v = (int)(ent >> 1), mir = (int)(ent & 1);
  const float b0 = B[2 * v], b1 = B[2 * v + 1];
  Footprint f;
  footprint(b0, b1, scale, g, f);
  int c0, c1;
  half_cols(f, mir, g, c0, c1);
  e.mir = mir;
  const int nr = f.a1 - f.a0 + 1, nc = c1 - c0 + 1;
  // Tap row ia is grid row wrap(r1), r1 = a0 + ia (mirrored: -(a0 + ia)).
  // Unless the grid is little more than one tile high (fewer than nine rows
  // beyond it), no tile holds rows of a footprint from both grid ends, so a
  // tile's rows of the footprint are one run of ia along which the tile row
  // moves by +1 (mirrored: -1).
  int ia_lo = 9, ia_hi = 0, lr_first = 0;
  if (g >= FIP_GTILE + 9) {
    // Tile row of ia = 0 before wrapping, or from the other grid end where
    // that reaches the tile.
    const int rows = min(FIP_GTILE, g - trow0);  // of the tile
    const int first = (mir ? -f.a0 : f.a0) - trow0;
    if (!mir) {
      const int off = first > -9 && first < rows ? first : first + g;
      ia_lo = max(0, -off);
      ia_hi = min(nr, rows - off);
      lr_first = off + ia_lo;
    } else {
      const int off = first >= 0 && first < rows + 9 ? first : first + g;
      ia_lo = max(0, off - rows + 1);
      ia_hi = min(nr, off + 1);
      lr_first = off - ia_lo;
    }
  } else {
#pragma unroll
    for (int a = 0; a < 9; ++a)
      if (a < nr) {
        const int lr = wrap_row(mir ? -(f.a0 + a) : f.a0 + a, g) - trow0;
        if ((unsigned)lr < (unsigned)FIP_GTILE) {
          if (a < ia_lo) {
            ia_lo = a;
            lr_first = lr;
          }
          ia_hi = a + 1;
        }
      }
  }
  e.ia_lo = ia_lo;
  e.ia_hi = ia_hi;
  e.ib_lo = max(0, tcol0 - c0);
  e.ib_hi = min(nc, tcol0 + FIP_GTILE - c0);
  e.cell0 = lr_first * kTS + (c0 + e.ib_lo - tcol0);
  e.r1 = mir ? -(f.a0 + ia_lo) : f.a0 + ia_lo;
  const float ihs = 1 / static_cast<float>(FIP_SUPPORT / 2);
  // Row taps r1 = a0 + ia; column taps in half-plane order c0 .. c1: original
  // r2 = c (direct) or -c (mirrored); on the Nyquist column, always a direct
  // footprint's only one, r2 = -G/2 (r2 never reaches +G/2,
  // FIPkernels.cu:203).  Integers below 2^24: exact in FP32.  The ninth tap
  // exists only for a position exactly on a cell.
  const bool down = mir || 2 * c0 == g;
  const float r0 = (float)f.a0, q0 = (float)(down ? -c0 : c0), qs = down ? -1.0f : 1.0f;
  const auto away = [&](float r, float b, float p) {
    return EXACT ? __fmaf_rn(-b, scale, r) : __fadd_rn(r, -p);
  };
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    e.k1[k] = fipref::es(away(r0 + (float)k, b0, f.p1) * ihs);
    e.k2[k] = fipref::es(away(q0 + qs * (float)k, b1, f.p2) * ihs);
  }
  e.k1[8] = e.k2[8] = 0.f;
  if (nr > 8) e.k1[8] = fipref::es(away(r0 + 8.0f, b0, f.p1) * ihs);
  if (nc > 8) e.k2[8] = fipref::es(away(q0 + qs * 8.0f, b1, f.p2) * ihs);
}

// One gridding work item (tile, entry range) of one snapshot, one or two
// entries per thread.  Phase 1 loads their weights and reduces the item's
// bound, phase 2 takes an entry's footprint and kernel values into registers
// and walks its in-tile taps into the shared tile, phase 3 commits.  The tile sums are fixed point, so the shared-memory
// sums are native integer atomics: exact and independent of their order.
// Plain form: q = round(tap * 2^31 / bound) in one int32, `bound` (the
// item's summed weights) bounding every cell sum.
// Precision form with FP32 visibilities (COMP; with FP16/BF16 storage the
// precision form sums as the plain form does): t = tap * 2^e, 2^e = the power of two with
// bound * 2^e < 2^45, is exact in FP32 and is split exactly into
// hi * 2^23 + lo (hi < 2^22 in magnitude, 0 <= lo <= 2^23), two int32 limbs
// summed separately (FIP_GCHUNK_MAX taps per cell per item at most: no overflow), so a
// cell holds the exact sum of its FP32 taps to 2^-45 of the bound and is
// rounded once at the commit.
template <int VT, bool COMP>
__device__ __forceinline__ void grid_item(GridSmem& S, float* s_cre, float* s_cim,
                                          const float* __restrict__ B,
                                          const void* vr, const void* vi,
                                          const float* vis_scale, float inten, float scale,
                                          int g, int hp, int tiles_c,
                                          int layout, const unsigned* __restrict__ entries,
                                          int4 item, float2* __restrict__ grid,
                                          const FipRawVis& raw = FipRawVis{}) {
  static_assert(FIP_GCHUNK_MAX <= 2 * kThreads, "two entries per thread at most");
  // The precision form: compensated, or with reduced storage.
  constexpr bool kExact = COMP || VT == FIP_VIS_F16 || VT == FIP_VIS_BF16;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tile = item.x, cnt = item.z - item.y;
  const int trow0 = (tile / tiles_c) * FIP_GTILE, tcol0 = (tile % tiles_c) * FIP_GTILE;
  // The tile (and, behind it, its low limbs) zeroed in 16-byte stores.
  {
    constexpr int kWords = (2 + (COMP ? 2 : 0)) * FIP_GTILE * kTS / 4;
    for (int k = threadIdx.x; k < kWords; k += kThreads)
      reinterpret_cast<float4*>(S.tile)[k] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  // Phase 1: the weights of this thread's entries (one, or two in items of
  // more than kThreads).
  const bool have = (int)threadIdx.x < cnt, more = (int)threadIdx.x + kThreads < cnt;
  unsigned ent = 0, ent2 = 0;
  float wr = 0.f, wi = 0.f, wr2 = 0.f, wi2 = 0.f;
  if (have) {
    ent = entries[item.y + threadIdx.x];
    if (more) ent2 = entries[item.y + threadIdx.x + kThreads];
    entry_weights<VT>(vr, vi, vis_scale, inten, ent, raw, wr, wi);
    if (more) entry_weights<VT>(vr, vi, vis_scale, inten, ent2, raw, wr2, wi2);
  }
  // Sum over the item of max(|wr|, |wi|): bounds every cell sum.
  float bound = fmaxf(fabsf(wr), fabsf(wi)) + fmaxf(fabsf(wr2), fabsf(wi2));
  for (int o = 16; o > 0; o >>= 1) bound += __shfl_xor_sync(0xffffffffu, bound, o);
  if (lane == 0) S.bound[warp] = bound;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) tot += S.bound[w];
  tot *= 1.0001f;  // margin for the rounding of the weights and their sum
  float fx = 0.f, fx_inv = 0.f;
  if (!COMP) {
    fx = tot > 0.f ? 2147483648.0f / tot : 0.f;
    fx_inv = tot * (1.0f / 2147483648.0f);
  } else if (tot > 0.f) {
    int ex = 0;
    frexpf(tot, &ex);  // tot < 2^ex
    fx = ldexpf(1.0f, 45 - ex);
    fx_inv = ldexpf(1.0f, ex - 45);
  }
  int* s_qre = reinterpret_cast<int*>(S.tile);
  int* s_qim = s_qre + FIP_GTILE * kTS;
  unsigned* s_lre = reinterpret_cast<unsigned*>(s_cre);
  unsigned* s_lim = reinterpret_cast<unsigned*>(s_cim);
  // Exact limbs of t = x * 2^e (precision form, see above).
  auto limbs = [&](float x, int& hi, unsigned& lo) {
    const float t = x * fx;
    const float hf = floorf(t * (1.0f / 8388608.0f));
    const float lf = fmaf(hf, -8388608.0f, t);  // exact: t - hi 2^23 in [0, 2^23]
    hi = __float_as_int(hf + 12582912.0f) - 0x4B400000;  // |hf| < 2^22: exact
    lo = __float_as_uint(lf + 8388608.0f) - 0x4B000000u;  // round to integer
  };
  // Phase 2: the thread walks its entries' in-tile taps.
#pragma unroll 1
  for (int left = have ? (more ? 2 : 1) : 0; left > 0; --left, ent = ent2, wr = wr2, wi = wi2) {
    EntryTaps et;
    entry_taps<kExact>(B, scale, g, ent, trow0, tcol0, et);
    if (et.empty()) continue;
    const float wrf = COMP ? wr : wr * fx, wif = COMP ? wi : wi * fx;
    const int dstep = et.mir ? -kTS : kTS;
    const unsigned rn = et.ia_hi - et.ia_lo, cn = et.ib_hi - et.ib_lo;
    const int cell = et.cell0 - et.ib_lo;  // of tap (ia_lo, 0)
    auto add = [&](int c, float x, float y) {
      if (!COMP) {
        atomicAdd(&s_qre[c], __float2int_rn(x));
        atomicAdd(&s_qim[c], __float2int_rn(y));
      } else {
        int hr, hi;
        unsigned lr2, li2;
        limbs(x, hr, lr2);
        limbs(y, hi, li2);
        atomicAdd(&s_qre[c], hr);
        atomicAdd(&s_lre[c], lr2);
        atomicAdd(&s_qim[c], hi);
        atomicAdd(&s_lim[c], li2);
      }
    };
    if (g >= FIP_GTILE + 9) {
      int rc = cell - et.ia_lo * dstep;
#pragma unroll
      for (int a = 0; a < 8; ++a, rc += dstep) {
        if ((unsigned)(a - et.ia_lo) >= rn) continue;
        const float ra = wrf * et.k1[a], rb = wif * et.k1[a];
#pragma unroll
        for (int b = 0; b < 8; ++b)
          if ((unsigned)(b - et.ib_lo) < cn) add(rc + b, ra * et.k2[b], rb * et.k2[b]);
        if (et.ib_hi > 8) add(rc + 8, ra * et.k2[8], rb * et.k2[8]);
      }
      if (et.ia_hi > 8) {
        const float ra = wrf * et.k1[8], rb = wif * et.k1[8];
#pragma unroll
        for (int b = 0; b < 9; ++b)
          if ((unsigned)(b - et.ib_lo) < cn) add(rc + b, ra * et.k2[b], rb * et.k2[b]);
      }
    } else {
      // Grids of little more than one tile: a tile may hold rows from both
      // grid ends, with the rows between them in another tile or none, so
      // each tap row is wrapped and checked on its own.
      const int lc0 = cell - (wrap_row(et.r1, g) - trow0) * kTS;
#pragma unroll
      for (int a = 0; a < 9; ++a) {
        if ((unsigned)(a - et.ia_lo) >= rn) continue;
        const int lr = wrap_row(et.r1 + (et.mir ? et.ia_lo - a : a - et.ia_lo), g) - trow0;
        if ((unsigned)lr >= (unsigned)FIP_GTILE) continue;
        const float ra = wrf * et.k1[a], rb = wif * et.k1[a];
#pragma unroll
        for (int b = 0; b < 9; ++b)
          if ((unsigned)(b - et.ib_lo) < cn)
            add(lr * kTS + lc0 + b, ra * et.k2[b], rb * et.k2[b]);
      }
    }
  }
  __syncthreads();
  // Phase 3: commit in the layout's contiguous direction: each thread keeps its
  // place along it and steps across.
  const bool single = item.w != 0;
  const int along = threadIdx.x % FIP_GTILE, across0 = threadIdx.x / FIP_GTILE;
  constexpr int kStep = kThreads / FIP_GTILE;
  const int na = layout ? g - trow0 : hp - tcol0, nx = layout ? hp - tcol0 : g - trow0;
  const int sa = layout ? kTS : 1, sx = layout ? 1 : kTS;  // shared strides along, across
  float2* dst = grid + cell_index(trow0, tcol0, g, hp, layout) + along +
                (size_t)across0 * (layout ? g : hp);
  const size_t dstep = (size_t)kStep * (layout ? g : hp);
  int at = along * sa + across0 * sx;
  if (along < na) {
#pragma unroll 4
    for (int k = 0; k < FIP_GTILE / kStep; ++k, at += kStep * sx, dst += dstep) {
      if (across0 + k * kStep >= nx) break;
      float2 val;
      if (COMP) {
        val = make_float2((float)(((double)s_qre[at] * 8388608.0 + (double)s_lre[at]) * fx_inv),
                          (float)(((double)s_qim[at] * 8388608.0 + (double)s_lim[at]) * fx_inv));
      } else {
        val = make_float2((float)s_qre[at] * fx_inv, (float)s_qim[at] * fx_inv);
      }
      if (single) {
        *dst = val;
      } else if (val.x != 0.f || val.y != 0.f) {
        atomicAdd(dst, val);
      }
    }
  }
  __syncthreads();
}

__device__ __forceinline__ float plane_intensity(const float* V) {
  return fabs(V[0 * 3 + 0] * V[1 * 3 + 1] - V[0 * 3 + 1] * V[1 * 3 + 0]);
}

// Persistent gridder over the work items of one snapshot.
template <int VT, bool COMP>
__global__ void __launch_bounds__(kThreads) k_grid(const float* __restrict__ B, const void* vr,
                                                   const void* vi,
                                                   const float* __restrict__ vis_scale_p,
                                                   const float* __restrict__ V, float scale,
                                                   int g, int hp, int tiles_c, int layout,
                                                   const unsigned* __restrict__ entries,
                                                   const int4* __restrict__ work,
                                                   const unsigned* __restrict__ nwork,
                                                   float2* __restrict__ grid,
                                                   const FipRawVis raw) {
  extern __shared__ float4 s_raw[];
  GridSmem& S = *reinterpret_cast<GridSmem*>(s_raw);
  float* s_cre = reinterpret_cast<float*>(reinterpret_cast<char*>(s_raw) + sizeof(GridSmem));
  float* s_cim = s_cre + FIP_GTILE * kTS;
  const float inten = plane_intensity(V);
  const unsigned nw = *nwork;
  __syncthreads();
  for (unsigned w = blockIdx.x; w < nw; w += gridDim.x)
    grid_item<VT, COMP>(S, s_cre, s_cim, B, vr, vi, vis_scale_p, inten, scale, g, hp, tiles_c,
                        layout, entries, work[w], grid, raw);
}

// Persistent gridder over the work items of a batch of snapshots (one launch
// for the batch, whatever their image sizes): snapshot k's inputs, bins,
// grid and geometry are in.s[k].
template <int VT, bool COMP>
__global__ void __launch_bounds__(kThreads) k_grid_batch(const __grid_constant__ FipGridBatch in) {
  extern __shared__ float4 s_raw[];
  __shared__ unsigned s_first[FIP_MAX_BATCH + 1];  // prefix of the snapshots' item counts
  GridSmem& S = *reinterpret_cast<GridSmem*>(s_raw);
  float* s_cre = reinterpret_cast<float*>(reinterpret_cast<char*>(s_raw) + sizeof(GridSmem));
  float* s_cim = s_cre + FIP_GTILE * kTS;
  // (Two snapshots per lane of the first warp.)
  if (threadIdx.x < 32) {
    const int k = 2 * threadIdx.x;
    const unsigned a = k < in.count ? *in.s[k].nwork : 0u;
    const unsigned b = k + 1 < in.count ? *in.s[k + 1].nwork : 0u;
    unsigned inc = a + b;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, inc, o);
      if ((int)threadIdx.x >= o) inc += y;
    }
    if (k <= in.count) s_first[k] = inc - a - b;
    if (k + 1 <= in.count) s_first[k + 1] = inc - b;
    if (k + 2 == FIP_MAX_BATCH && in.count == FIP_MAX_BATCH) s_first[FIP_MAX_BATCH] = inc;
  }
  __syncthreads();
  const unsigned total = s_first[in.count];
  int k = 0;
  for (unsigned w = blockIdx.x; w < total; w += gridDim.x) {
    while (s_first[k + 1] <= w) ++k;  // items are visited in increasing order
    const FipGridSnap& sn = in.s[k];
    const float inten = plane_intensity(sn.V);
    grid_item<VT, COMP>(S, s_cre, s_cim, sn.B, sn.vr, sn.vi, sn.vis_scale, inten, sn.scale, sn.g,
                        sn.hp, sn.tiles_c, sn.layout, sn.entries, sn.work[w - s_first[k]],
                        sn.grid);
  }
}

// ---------------------------------------------------------------------------
// Reprojection (FIPkernels.cu:289-413).
// ---------------------------------------------------------------------------

// The reference's pixel mapping for every source pixel: targets[j*N + i] =
// (LL, MM) of source column i, row j.  Overlapped with the gridding and the FFT
// on a side stream.  Bound by instruction issue (most of it
// inside atan2f and acosf; 134 MB written at 4096^2, 21 us): FP32 degree
// conversions in place of FP64 ones took 4096^2 from 124 to 97 us (239 to 187
// instructions a pixel), one test for the special cases and no branch for planes
// without a tilt to 91 (172).  Four pixels
// per thread share the loads of V and the row's terms (two: 101, eight: 103).
constexpr int kTargetsPerThread = 4;
// ttab: the theta-terms table (fipref::kThetaTabSize entries) or null.
// MANY: launches over several snapshots (blockIdx.z).
template <bool MANY>
__global__ void k_targets(const float* __restrict__ V, int n, float dc,
                          const float2* __restrict__ ttab, float2* __restrict__ tg,
                          size_t stride) {
  if (MANY) {
    V += 9 * blockIdx.z;
    tg += blockIdx.z * stride;
  }
  const int j = blockIdx.y;
  const fipref::Frame fr{V[0], V[1], V[3], V[4], V[8], V[6], V[7], dc};
#pragma unroll
  for (int q = 0; q < kTargetsPerThread; ++q) {
    const int i = (blockIdx.x * kTargetsPerThread + q) * blockDim.x + threadIdx.x;
    if (i < n) {
      float LL, MM;
      fipref::pixel_target(fr, i, j, n, LL, MM, ttab);
      tg[(size_t)j * n + i] = make_float2(LL, MM);
    }
  }
}

__global__ void k_theta_table(float2* __restrict__ tab) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= fipref::kThetaTabSize) return;
  float r, zr0;
  fipref::theta_terms(__uint_as_float(fipref::kThetaTabLo + (unsigned)k), r, zr0);
  tab[k] = make_float2(r, zr0);
}

// Source-major reprojection, the reference's own scheme (FIPkernels.cu:378-413):
// one thread per source pixel, four atomics into a zeroed destination.
__global__ void k_reproject_scatter(const float* __restrict__ pre, const float* __restrict__ V,
                                    int n, int nb, float dc, float* __restrict__ dst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= n || j >= n) return;
  fipref::Frame fr{V[0], V[1], V[3], V[4], V[8], V[6], V[7], dc};
  const float inv_nb = 1.0f / static_cast<float>(nb);
  const float value = pre[(size_t)j * n + i] * inv_nb;
  float LL, MM;
  fipref::pixel_target(fr, i, j, n, LL, MM);
  const size_t half = n / 2;
  const long c = (long)(half * n + half);
  if (fabs(LL) < half - 1 && fabs(MM) < half - 1) {
    const long fl = fipref::floor_l(LL), cl = fipref::ceil_l(LL);
    const long fm = fipref::floor_l(MM), cm = fipref::ceil_l(MM);
    atomicAdd(&dst[c + fm * (long)n + fl], (1 - LL + fl) * (1 - MM + fm) * value);
    atomicAdd(&dst[c + cm * (long)n + fl], (1 - LL + fl) * (MM - fm) * value);
    atomicAdd(&dst[c + fm * (long)n + cl], (LL - fl) * (1 - MM + fm) * value);
    atomicAdd(&dst[c + cm * (long)n + cl], (LL - fl) * (MM - fm) * value);
  }
}

struct Acc {
  float s, sc, r, rc, m;
};

template <bool PRECISE>
__device__ __forceinline__ void acc_add(Acc& a, float d, float q) {
  if (!PRECISE) {
    a.s += d;
    a.r += q;
  } else {
    float t = a.s + d;
    a.sc += (fabsf(a.s) >= fabsf(d)) ? (a.s - t) + d : (d - t) + a.s;
    a.s = t;
    t = a.r + q;
    a.rc += (fabsf(a.r) >= fabsf(q)) ? (a.r - t) + q : (q - t) + a.r;
    a.r = t;
  }
  a.m = fmaxf(a.m, d);
}

template <bool PRECISE>
__device__ __forceinline__ void acc_pixel(Acc& a, float i1, float i2, float i3) {
  const float d = fabs(fabs(i1 - i2) - fabs(i2 - i3));
  const float s2 = (i2 <= 0) ? FIP_TRIGGER_FLOOR : i2;
  const float q = d / s2;
  acc_add<PRECISE>(a, d, fminf(q, 1.0f));  // NaN counts 1, as (q < 1) ? q : 1
}

// The warp's reduction of its lanes' tile statistics (valid in lane 0).
template <bool PRECISE>
__device__ __forceinline__ void warp_stats(Acc a, double& S, double& R, float& M) {
  if (!PRECISE) {
    for (int o = 16; o > 0; o >>= 1) {
      a.s += __shfl_xor_sync(0xffffffffu, a.s, o);
      a.r += __shfl_xor_sync(0xffffffffu, a.r, o);
      a.m = fmaxf(a.m, __shfl_xor_sync(0xffffffffu, a.m, o));
    }
    S = (double)a.s;
    R = (double)a.r;
  } else {
    double s = (double)a.s + (double)a.sc, r = (double)a.r + (double)a.rc;
    for (int o = 16; o > 0; o >>= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, o);
      r += __shfl_xor_sync(0xffffffffu, r, o);
      a.m = fmaxf(a.m, __shfl_xor_sync(0xffffffffu, a.m, o));
    }
    S = s;
    R = r;
  }
  M = a.m;
}

// Statistics of one trigger tile (FIPkernels.cu:499-552 before the combine),
// one warp per T x T tile at base: S = sum d, R = sum min(d / I2', 1) (NaN
// counts as 1), M = max(0, max d), in the lanes' and shuffles' order (valid
// in lane 0).  Plain form: FP32 sums; precise form: Neumaier-compensated FP32
// sums combined in FP64.  L2: load through L2 only (data other SMs wrote in
// the same kernel).
template <bool PRECISE, bool L2>
__device__ __forceinline__ void tile_stats(const float* __restrict__ I1,
                                           const float* __restrict__ I2,
                                           const float* __restrict__ I3, size_t base, int n,
                                           int t, int vec, int lane, double& S, double& R,
                                           float& M) {
  auto ld4 = [](const float* p) {
    return L2 ? __ldcg(reinterpret_cast<const float4*>(p)) : *reinterpret_cast<const float4*>(p);
  };
  auto ld1 = [](const float* p) { return L2 ? __ldcg(p) : *p; };
  Acc a{0.f, 0.f, 0.f, 0.f, 0.f};
  if (vec) {
    const int q = t / 4;  // float4 per tile row
    for (int k = lane; k < t * q; k += 32) {
      const int r = k / q, c = (k % q) * 4;
      const size_t o = base + (size_t)r * n + c;
      const float4 x1 = ld4(I1 + o);
      const float4 x2 = ld4(I2 + o);
      const float4 x3 = ld4(I3 + o);
      acc_pixel<PRECISE>(a, x1.x, x2.x, x3.x);
      acc_pixel<PRECISE>(a, x1.y, x2.y, x3.y);
      acc_pixel<PRECISE>(a, x1.z, x2.z, x3.z);
      acc_pixel<PRECISE>(a, x1.w, x2.w, x3.w);
    }
  } else {
    for (int k = lane; k < t * t; k += 32) {
      const size_t o = base + (size_t)(k / t) * n + (k % t);
      acc_pixel<PRECISE>(a, ld1(I1 + o), ld1(I2 + o), ld1(I3 + o));
    }
  }
  warp_stats<PRECISE>(a, S, R, M);
}

// The tLISI of one tile from its statistics and the three image maxima
// (FIPkernels.cu:550): the plain form's FP32 expression, the precise form's
// FP64 one.
template <bool PRECISE>
__device__ __forceinline__ float tlisi_of(double S, double R, float M, const float max3[3], int t) {
  if (!PRECISE) {
    const float maxallval = max(max3[0], max(max3[1], max3[2]));
    const size_t us = (size_t)t;
    return 1 - ((float)S / us / us) * M * ((float)R / us / us) / maxallval / maxallval;
  }
  const double mx = fmax(fmax((double)max3[0], (double)max3[1]), (double)max3[2]);
  const double tt = (double)t;
  return (float)(1.0 - (S / tt / tt) * (double)M * (R / tt / tt) / mx / mx);
}

// The trigger fused into the reprojections of a three-snapshot call: the
// gather CTA that writes the last of the three images of its 64 x 64 region
// (a per-region count) computes the region's trigger-tile statistics, and a
// final one-pass kernel applies the maxima.
struct FipTriggerFuse {
  const float* img[3];  // I1, I2, I3
  unsigned* count;      // [gather tiles], zero at the call's start
  double* stats;        // [U*U][3]: S, R, M
  int t, u;
};

constexpr int kMaxRows = 256;    // candidate source rows per tile (one per thread)
static_assert(kMaxRows == kThreads, "the gather numbers rows one per thread");

// The exact map around a per-tile origin (a0, b0) of source offsets, for the
// precision form's splats.  With Q = P - 1 the vector whose squared length,
// times cell^2, is rho, and Q0 its value at the origin, a source d = M (a -
// a0, b - b0) away has
//   rho - rho0 = cell^2 g,   g = 2 Q0.d + d.d,
//   z(rho) - z(rho0) = cell g / (sqrt(1 - rho0) + sqrt(1 - rho))
// (z = slant over cell), so its target relative to the destination tile is
//   L = l0 + d1 - xi dz,  M = m0 + d2 + eta dz,
// with l0, m0 the origin's target in tile coordinates (FP64).  Every FP32
// quantity is then a tile-sized offset or a relative correction: rsqrtf and
// __fdividef (a few ulp) move a target by ~1e-5 pixel, well inside the
// FP64 tolerance, where the slant term in absolute form rounds at its own
// magnitude (hundreds of pixels on wide fields).  Beyond the horizon
// (rho > 1) the slant term is 0, as in the closed form; the relative form
// needs the origin inside it, which every tile in the gather's domain has.
struct TileMap {
  float m00, m01, m10, m11;  // M / |V22|
  float xi, eta, cell, c2;   // c2 = cell^2
  float q1, q2;              // 2 Q0
  float u0, s0, z0;          // 1 - rho0, its square root, the slant term at the origin
  float l0, m0;              // the origin's target relative to the tile's corner
  int a0, b0;
};

__device__ __forceinline__ TileMap tile_map(const ExactMap<double>& md, const float (*q)[2],
                                            int seg, int cl, int rl) {
  TileMap t;
  // Origin: the rounded mean of the preimage polygon's four corners.
  t.a0 = (int)rintf(0.25f * (q[0][0] + q[seg][0] + q[2 * seg][0] + q[3 * seg][0]));
  t.b0 = (int)rintf(0.25f * (q[0][1] + q[seg][1] + q[2 * seg][1] + q[3 * seg][1]));
  const double P1 = md.m00 * t.a0 + md.m01 * t.b0, P2 = md.m10 * t.a0 + md.m11 * t.b0;
  const double Q1 = P1 - 1.0, Q2 = P2 - 1.0;
  const double rho = md.cell * md.cell * (Q1 * Q1 + Q2 * Q2);
  const double u0 = 1.0 - rho;
  const double s0 = u0 > 0.0 ? sqrt(u0) : 0.0;
  const double z0 = rho <= 1.0 ? (rho / (1.0 + s0)) / md.cell : 0.0;
  t.m00 = (float)md.m00; t.m01 = (float)md.m01; t.m10 = (float)md.m10; t.m11 = (float)md.m11;
  t.xi = (float)md.xi; t.eta = (float)md.eta;
  t.cell = (float)md.cell; t.c2 = (float)(md.cell * md.cell);
  t.q1 = (float)(2.0 * Q1); t.q2 = (float)(2.0 * Q2);
  t.u0 = (float)u0; t.s0 = (float)s0; t.z0 = (float)z0;
  t.l0 = (float)(P1 - md.xi * z0 - (double)cl);
  t.m0 = (float)(P2 + md.eta * z0 - (double)rl);
  return t;
}

// Target (L, M), relative to the tile's corner, of the source at offsets
// (a, b) from the image centre.
__device__ __forceinline__ void tile_target(const TileMap& t, int a, int b, float& L, float& M) {
  const float da = (float)(a - t.a0), db = (float)(b - t.b0);
  const float d1 = t.m00 * da + t.m01 * db, d2 = t.m10 * da + t.m11 * db;
  const float g = d1 * (t.q1 + d1) + d2 * (t.q2 + d2);
  const float u = t.u0 - t.c2 * g;
  float dz = -t.z0;
  if (u >= 0.f) {
    const float s = u > 0.f ? u * rsqrtf(u) : 0.f;
    dz = __fdividef(t.cell * g, t.s0 + s);
  }
  L = t.l0 + d1 - t.xi * dz;
  M = t.m0 + d2 + t.eta * dz;
}

// Destination-tile-major reprojection.  The candidate source pixels of a
// 64x64 destination tile are the integer points of the preimage of the tile
// widened by the splat reach (1 pixel) and delta (the FP32 chain's deviation
// from the exact map): per source row, one column interval.  Each candidate
// is splatted (bilinear weights of FIPkernels.cu:394-410) into shared memory;
// the tile is stored once and its maximum folded into *img_max.
// EXACT: targets from the closed form (precision form), in FP32 relative to
// a per-tile origin whose terms are FP64 (TileMap), instead of the
// precomputed reference-chain targets.
// The shared tile carries an apron of kAp pixels on every side, so the four
// pixels of any candidate's splat land inside it without per-pixel checks
// (apron pixels belong to the neighbouring tiles, which splat them
// themselves, and are dropped at the commit).  Its row stride is odd, so the
// lanes of a warp (neighbouring sources, mapped along an arbitrary
// direction) fall on distinct banks down a column as well as along a row.
constexpr int kAp = 4;
constexpr int kTW = kDT + 2 * kAp;  // tile side with the apron
constexpr int kTR = kTW + 1;        // row stride
// MANY: a launch over several snapshots (blockIdx.y); launches of one keep
// every pointer in the constant bank (with MANY's register pairs for the
// per-snapshot pointers the splats spill more: a 4096^2 plain call 969
// against 949 us).
template <bool EXACT, bool MANY>
__device__ __forceinline__ void gather_tile(const FipGatherBatch& in,
                                            const float* __restrict__ pre,
                                            const float2* __restrict__ tg, int n, float cell,
                                            float delta, const unsigned* __restrict__ pre_max,
                                            unsigned* err, const FipTriggerFuse& fuse, int tile) {
  const int snap = MANY ? (int)blockIdx.y : 0;
  const float* __restrict__ V = in.V[snap];
  if (MANY) {
    pre += snap * (size_t)n * n;
    if (!EXACT) tg += snap * (size_t)n * n;
  }
  __shared__ __align__(16) unsigned s_tile[kTW * kTR];
  __shared__ int s_base[kMaxRows];  // pixel index of row r's first candidate minus its number
  __shared__ int s_off[kMaxRows + 1];
  __shared__ int s_wsum[kThreads / 32];
  __shared__ float s_q[kPoly][2];
  __shared__ float s_wmax[kThreads / 32];

  const int tiles = (n + kDT - 1) / kDT;
  const int tr = tile / tiles, tc = tile % tiles;
  const int r0 = tr * kDT, c0 = tc * kDT;
  const int h = n / 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

  static_assert((kTW * kTR) % 4 == 0, "the tile is zeroed in 16-byte stores");
  for (int k = threadIdx.x; k < kTW * kTR / 4; k += kThreads)
    reinterpret_cast<uint4*>(s_tile)[k] = make_uint4(0u, 0u, 0u, 0u);
  // Precision form: the FP64 map, formed once per CTA by a lane of warp 1
  // while warp 0 traces the preimage, and turned into the tile's FP32
  // constants (TileMap) by one thread after the barrier.
  __shared__ ExactMap<double> s_md;
  __shared__ TileMap s_tm;
  if (EXACT && threadIdx.x == 32) s_md = make_map<double>(V, cell);
  // Preimage of the tile's boundary, widened by the splat reach and delta:
  // kPoly points, kSeg per edge, in order around it (lanes of warp 0), the
  // tile's domain check and its curvature margin.
  __shared__ float s_sag, s_bmin, s_bmax, s_parea;
  if (warp == 0) {
    float a, b;
    const TilePreimage pr =
        trace_preimage(make_map_f32(V, cell), r0, c0, h, delta, cell, lane, a, b);
    if (lane < kPoly) {
      s_q[lane][0] = a;
      s_q[lane][1] = b;
    }
    if (lane == 0) {
      // A tile outside the domain is reported, not skipped.
      if (err && !pr.ok) atomicOr(err, 1u);
      s_sag = pr.sag;
      s_bmin = pr.bmin;
      s_bmax = pr.bmax;
      s_parea = pr.area;
    }
  }
  __syncthreads();
  const float bmin = s_bmin, bmax = s_bmax;
  const float sag = s_sag + 1e-3f;
  const int jlo = (int)fmaxf(0.f, ceilf(fmaxf(bmin + h - sag, -1.f)));
  const int jhi = (int)fminf((float)(n - 1), floorf(fminf(bmax + h + sag, (float)n)));
  const size_t half = n / 2;
  const float lim = half - 1;  // the reference compares |LL| with size_t (N/2 - 1)
  // A candidate that reaches the tile has LL in [c0 - h - 1, c0 - h + kDT)
  // (MM likewise): for tiles at least two pixels inside that range check on
  // both axes, every such candidate passes it, and a candidate that would fail
  // it lands beyond the tile, so the check is left out there.
  const bool inner = c0 >= 4 && c0 + kDT + 4 <= 2 * h && r0 >= 4 && r0 + kDT + 4 <= 2 * h;
  // Fixed-point tile sums: a source's splat value v / nb is carried as
  // v * 2^(28 - sh) / max(pre).  Every contribution is <= 2^(28 - sh), and
  // the bilinear weights landing on one pixel sum to about the density of
  // sources per destination pixel (four times it at most), so the sums stay
  // below 2^32 while that density is <= 2^(2 + sh): the shared-memory sums
  // are native integer atomics, exact and independent of their order, and
  // the tile is converted back once.  sh is 0 (resolution 2^-28 of the image
  // maximum) unless the preimage of the tile, with its margins, covers more
  // than twice the tile's area -- a map that contracts, which only very wide
  // fields with a tilted plane reach -- and then grows by one per doubling.
  const float parea = s_parea;  // preimage polygon's area (shoelace)
  int sh = 0;
  while (sh < 12 && parea > (float)(2 * kDT * kDT) * (float)(1 << sh)) ++sh;
  const float pmax = __uint_as_float(pre_max[4 * snap]);
  const float qk = pmax > 0.f ? 268435456.0f / (pmax * (float)(1 << sh)) : 0.f;
  // Precision form: the tile's constants, from FP64 by a thread of the last
  // warp (idle in the row-interval step unless a chunk has 256 rows); every
  // thread reads them after the chunk's barriers, before its first splat.
  if (EXACT && threadIdx.x == kThreads - 1) s_tm = tile_map(s_md, s_q, kSeg, c0 - h, r0 - h);
  TileMap tm;
  auto splat = [&](int i, int j, float vq, float2 t) {
    int fl, fm;
    float wl1, wm1, wl0, wm0;
    if (!EXACT) {
      const float LL = t.x, MM = t.y;
      if (!inner && !(fabsf(LL) < lim && fabsf(MM) < lim)) return;
      const float flf = floorf(LL), fmf = floorf(MM);
      // The reference's weight expressions (FIPkernels.cu:397-409).  Its far
      // pixel is ceil(LL), equal to floor(LL) + 1 except on exact integers,
      // where the far weight LL - floor(LL) is 0: splatting the far weight at
      // floor + 1 adds the same sums.
      wl0 = 1 - LL + flf; wl1 = LL - flf;
      wm0 = 1 - MM + fmf; wm1 = MM - fmf;
      fl = (int)flf + (h - c0);
      fm = (int)fmf + (h - r0);
    } else {
      float Lr, Mr;
      tile_target(tm, i - h, j - h, Lr, Mr);
      if (!inner && !(fabsf(Lr + (float)(c0 - h)) < lim && fabsf(Mr + (float)(r0 - h)) < lim))
        return;
      const float flr = floorf(Lr), fmr = floorf(Mr);
      fl = (int)flr;
      fm = (int)fmr;
      wl1 = Lr - flr; wm1 = Mr - fmr;
      wl0 = 1.0f - wl1; wm0 = 1.0f - wm1;
    }
    // Pixels (fm|fm+1, fl|fl+1), local to the tile with its apron.  A splat
    // that reaches the tile lies inside the apron (fl, fm >= -1); one that
    // does not touches no pixel of the tile and is skipped.
    fl += kAp;
    fm += kAp;
    if ((unsigned)fl > (unsigned)(kTW - 2) || (unsigned)fm > (unsigned)(kTW - 2)) return;
    const float a = wl0 * vq, b = wl1 * vq;
    unsigned* px = &s_tile[fm * kTR + fl];
    atomicAdd(px, __float2uint_rn(a * wm0));
    atomicAdd(px + 1, __float2uint_rn(b * wm0));
    atomicAdd(px + kTR, __float2uint_rn(a * wm1));
    atomicAdd(px + kTR + 1, __float2uint_rn(b * wm1));
  };
  // Candidate rows in chunks of kMaxRows (one row per thread): a single
  // chunk unless the preimage spans more than kMaxRows source rows.
  for (int cj = jlo; cj <= jhi; cj += kMaxRows) {
    const int nrows = min(kMaxRows, jhi - cj + 1);
    // Column interval of every candidate row (the preimage quadrilateral
    // intersected with the row), one row per thread, and the exclusive prefix
    // of the interval lengths: candidates are then numbered 0 .. total-1 row by
    // row, so every warp step splats 32 candidates whatever the row lengths.
    int cnt = 0, ilo = 0;
    {
      const int r = threadIdx.x;
      if (r < nrows) {
        // Rows in the margin beyond the quadrilateral's extreme corners take
        // the interval at that corner (then widened like every interval).
        const float b = fminf(fmaxf((float)(cj + r - h), bmin), bmax);
        float alo = 3e38f, ahi = -3e38f;
#pragma unroll
        for (int k = 0; k < kPoly; ++k) {
          const float ax = s_q[k][0], bx = s_q[k][1];
          const float ay = s_q[(k + 1) % kPoly][0], by = s_q[(k + 1) % kPoly][1];
          if ((bx <= b && b <= by) || (by <= b && b <= bx)) {
            if (by == bx) {
              alo = fminf(alo, fminf(ax, ay));
              ahi = fmaxf(ahi, fmaxf(ax, ay));
            } else {
              const float a = ax + (ay - ax) * ((b - bx) / (by - bx));
              alo = fminf(alo, a);
              ahi = fmaxf(ahi, a);
            }
          }
        }
        int ihi = -1;
        if (alo <= ahi) {
          ilo = (int)fmaxf(0.f, ceilf(fmaxf(alo + h - sag, -1.f)));
          ihi = (int)fminf((float)(n - 1), floorf(fminf(ahi + h + sag, (float)n)));
        }
        cnt = ihi >= ilo ? ihi - ilo + 1 : 0;
      }
      int inc = cnt;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
      }
      if (lane == 31) s_wsum[warp] = inc;
      __syncthreads();
      int wbase = 0;
      for (int w = 0; w < warp; ++w) wbase += s_wsum[w];
      if (r < kMaxRows) {
        s_off[r] = wbase + inc - cnt;
        // Candidate f of row r is pixel (cj + r) n + ilo + (f - off): s_base + f
        // (< N^2 <= 2^30 for image_size <= 32768).
        s_base[r] = (cj + r) * n + ilo - (wbase + inc - cnt);
      }
      if (r == kThreads - 1) s_off[kMaxRows] = wbase + inc;
    }
    __syncthreads();
    const int total = s_off[kMaxRows];
    if (EXACT) tm = s_tm;
    // Rows past nrows have no candidates: their offsets equal total.
    // Each warp takes a contiguous eighth of the candidates, so a lane's row
    // cursor moves about half a row per candidate; its start is found by
    // bisection of the row offsets.  Warp step: candidates f0 + lane + 32 e,
    // e < 4, all loads issued first; the cursor only moves forward.
    constexpr int kPer = 4, kWarps = kThreads / 32;
    const int per = (total + kWarps - 1) / kWarps;
    const int wb = min(total, warp * per), we = min(total, wb + per);
    int row = 0;
    for (int step = kMaxRows / 2; step > 0; step >>= 1)
      if (s_off[row + step] <= wb) row += step;  // last row whose offset is <= wb
    for (int f0 = wb; f0 < we; f0 += 32 * kPer) {
      int at[kPer], rw[kPer];
      float p[kPer];
      float2 tt[kPer];
#pragma unroll
      for (int e = 0; e < kPer; ++e) {
        const int f = f0 + lane + 32 * e;
        rw[e] = -1;
        if (f < we) {
          while (s_off[row + 1] <= f) ++row;
          rw[e] = row;
          at[e] = s_base[row] + f;
          p[e] = pre[at[e]];
          if (!EXACT) tt[e] = tg[at[e]];
        }
      }
#pragma unroll
      for (int e = 0; e < kPer; ++e) {
        if (rw[e] < 0) continue;
        const int j = cj + rw[e];
        splat(at[e] - j * n, j, p[e] * qk, EXACT ? make_float2(0.f, 0.f) : tt[e]);
      }
    }
    __syncthreads();  // the next chunk rewrites the row offsets
  }
  // (Per-snapshot values are read from the parameters only here, so that none
  // of them holds a register through the splats.)
  const float deq = __uint_as_float(pre_max[4 * snap]) *
                    (1.0f / static_cast<float>(in.nb[snap])) *
                    ((float)(1 << sh) / 268435456.0f);
  float* __restrict__ dst = in.dst[snap];
  unsigned* img_max = in.img_max[snap];
  float vmax = 0.f;
  for (int k = threadIdx.x; k < kDT * kDT / 4; k += kThreads) {
    const int lr = (4 * k) / kDT, g4 = ((4 * k) % kDT) >> 2;
    const int rr = r0 + lr, cc = c0 + 4 * g4;
    const unsigned* src = &s_tile[(lr + kAp) * kTR + kAp + 4 * g4];
    const uint4 q = make_uint4(src[0], src[1], src[2], src[3]);
    const float4 val = make_float4((float)q.x * deq, (float)q.y * deq, (float)q.z * deq,
                                   (float)q.w * deq);
    if (rr < n) {
      if (cc + 3 < n && (n & 3) == 0) {
        *reinterpret_cast<float4*>(&dst[(size_t)rr * n + cc]) = val;
        vmax = fmaxf(vmax, fmaxf(fmaxf(val.x, val.y), fmaxf(val.z, val.w)));
      } else {
        const float vv[4] = {val.x, val.y, val.z, val.w};
        for (int e = 0; e < 4; ++e)
          if (cc + e < n) {
            dst[(size_t)rr * n + cc + e] = vv[e];
            vmax = fmaxf(vmax, vv[e]);
          }
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
  if (lane == 0) s_wmax[warp] = vmax;
  __syncthreads();
  if (threadIdx.x == 0 && img_max) {
    float b = 0.f;
    for (int w = 0; w < kThreads / 32; ++w) b = fmaxf(b, s_wmax[w]);
    atomicMax(img_max, __float_as_uint(b));
  }
  if (fuse.count) {
    // Fused trigger: every thread's stores made visible device-wide, then one
    // count per region; the CTA that completes the region's third image
    // reads all three through L2 and reduces each trigger tile in it.
    __shared__ unsigned s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      const unsigned old = atomicAdd(&fuse.count[tile], 1u);
      s_last = old == 2u;
      __threadfence();
    }
    __syncthreads();
    if (s_last) {
      const int per = kDT / fuse.t;
      const int vec = (fuse.t % 4 == 0) && (n % 4 == 0);
      for (int k = warp; k < per * per; k += kThreads / 32) {
        const int ti = r0 / fuse.t + k / per, tj = c0 / fuse.t + k % per;
        const size_t base = (size_t)ti * fuse.t * n + (size_t)tj * fuse.t;
        double S, R;
        float M;
        tile_stats<EXACT, true>(fuse.img[0], fuse.img[1], fuse.img[2], base, n, fuse.t, vec,
                                lane, S, R, M);
        if (lane == 0) {
          double* o = fuse.stats + 3 * ((size_t)ti * fuse.u + tj);
          o[0] = S;
          o[1] = R;
          o[2] = (double)M;
        }
      }
    }
  }
}

template <bool EXACT, bool MANY>
__global__ void __launch_bounds__(kThreads, EXACT ? 5 : 8) k_reproject_gather(
    const __grid_constant__ FipGatherBatch in, const float* __restrict__ pre,
    const float2* __restrict__ tg, int n, float cell, float delta,
    const unsigned* __restrict__ pre_max, unsigned* err,
    const __grid_constant__ FipTriggerFuse fuse) {
  gather_tile<EXACT, MANY>(in, pre, tg, n, cell, delta, pre_max, err, fuse, (int)blockIdx.x);
}

// The splat over the tiles that the pull left out (word 2 of a tile's plan, of
// `words` words, is 0): persistent over the tiles, usually none.
__global__ void __launch_bounds__(kThreads, 5) k_reproject_rest(
    const __grid_constant__ FipGatherBatch in, const float* __restrict__ pre, int n, float cell,
    float delta, const unsigned* __restrict__ pre_max, unsigned* err,
    const unsigned* __restrict__ plans, int words) {
  const int tiles = (n + kDT - 1) / kDT, total = tiles * tiles;
  plans += (size_t)blockIdx.y * total * words;
  // Which of the CTA's tiles are left out: kThreads tiles a look.
  for (int base = blockIdx.x; base < total; base += gridDim.x * kThreads) {
    const int mine = base + (int)gridDim.x * threadIdx.x;
    const bool rest = mine < total && plans[(size_t)mine * words + 2] == 0;
    if (!__syncthreads_or(rest)) continue;
    for (int k = 0; k < kThreads; ++k) {
      const int tile = base + (int)gridDim.x * k;
      if (tile >= total) break;
      if (plans[(size_t)tile * words + 2] != 0) continue;
      __syncthreads();  // the previous tile's shared memory is free
      gather_tile<true, true>(in, pre, nullptr, n, cell, delta, pre_max, err, FipTriggerFuse{},
                              tile);
    }
    __syncthreads();
  }
}

// mode 0: the FP32 chain with the theta table (null: evaluated), 2: the
// chain evaluated, 1: the exact closed form.
__global__ void k_pixel_targets(const float* __restrict__ V, int n, float dc, float cell,
                                int mode, const float2* __restrict__ ttab,
                                float* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y;
  if (i >= n) return;
  float LL, MM;
  if (mode != 1) {
    fipref::Frame fr{V[0], V[1], V[3], V[4], V[8], V[6], V[7], dc};
    fipref::pixel_target(fr, i, j, n, LL, MM, mode == 0 ? ttab : nullptr);
  } else {
    const ExactMap<double> m = make_map<double>(V, cell);
    double Ld, Md;
    exact_forward(m, (double)(i - n / 2), (double)(j - n / 2), Ld, Md);
    LL = (float)Ld;
    MM = (float)Md;
  }
  out[2 * ((size_t)j * n + i)] = LL;
  out[2 * ((size_t)j * n + i) + 1] = MM;
}

// Maximum of non-negative floats (bit-pattern order), NaN ignored.
__global__ void k_image_max(const float* __restrict__ img, size_t count, unsigned* out) {
  float m = 0.f;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < count;
       k += (size_t)gridDim.x * blockDim.x)
    m = fmaxf(m, img[k]);
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, __float_as_uint(m));
}

// ---------------------------------------------------------------------------
// Trigger (FIPkernels.cu:415-552, 831-840).  One warp per T x T tile:
// D = | |I1-I2| - |I2-I3| |, I2 clamped to C after D, S = sum D,
// M = max(0, max D), R = sum min(D/I2c, 1) (NaN counts 1).
// PRECISE: Neumaier-compensated S and R, FP64 combine.
// ---------------------------------------------------------------------------
// RING: the triples of a ring of images (fip_launch_trigger_ring).
template <bool PRECISE, bool RING>
__global__ void __launch_bounds__(kThreads) k_trigger(const float* __restrict__ I1,
                                                      const float* __restrict__ I2,
                                                      const float* __restrict__ I3,
                                                      const float* __restrict__ m1,
                                                      const float* __restrict__ m2,
                                                      const float* __restrict__ m3, int n,
                                                      int t, int u, int vec,
                                                      float* __restrict__ result,
                                                      size_t img_stride, size_t res_stride,
                                                      int ring, int first) {
  float max3[3];
  if (RING) {
    // Triple blockIdx.y is images k, k + 1, k + 2 (k = first + y, modulo
    // ring) of the ring at I1 with maxima m1[ring].
    const float* base = I1;
    const int k0 = (first + (int)blockIdx.y) % ring, k1 = (k0 + 1) % ring, k2 = (k0 + 2) % ring;
    I1 = base + k0 * img_stride;
    I2 = base + k1 * img_stride;
    I3 = base + k2 * img_stride;
    max3[0] = m1[k0];
    max3[1] = m1[k1];
    max3[2] = m1[k2];
  } else {
    // Batched launches: triple blockIdx.y is images y, y+1, y+2 of a linear
    // ring (stride img_stride) with maxima m1[y], m2[y], m3[y].
    I1 += blockIdx.y * img_stride;
    I2 += blockIdx.y * img_stride;
    I3 += blockIdx.y * img_stride;
    max3[0] = m1[blockIdx.y];
    max3[1] = m2[blockIdx.y];
    max3[2] = m3[blockIdx.y];
  }
  result += blockIdx.y * res_stride;
  const int lane = threadIdx.x & 31;
  const int b = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
  if (b >= u * u) return;
  const int ti = b / u, tj = b % u;
  const size_t base = (size_t)ti * t * n + (size_t)tj * t;
  double S, R;
  float M;
  tile_stats<PRECISE, false>(I1, I2, I3, base, n, t, vec, lane, S, R, M);
  if (lane == 0) result[b] = tlisi_of<PRECISE>(S, R, M, max3, t);
}

// ---------------------------------------------------------------------------
// Sliding-window trigger streamed through registers: tLISI of triples
// (k, k+1, k+2) over a linear ring of images.  A warp owns one trigger tile
// and a chunk of consecutive triples; each lane keeps its float4s of the
// last three slices in registers and loads the next slice's while it
// reduces the current triple, so every image of the chunk is read from HBM
// once instead of once per triple it is in.  Lane k's float4s and the
// accumulation and shuffle order are k_trigger's (bit-identical results).
// NV: float4s per lane, >= T*T/128.
// ---------------------------------------------------------------------------
constexpr int kStreamThreads = 128;

template <bool PRECISE, int NV>
__global__ void __launch_bounds__(kStreamThreads) k_trigger_stream(
    const float* __restrict__ images, size_t img_stride, int count, int chunk,
    const float* __restrict__ maxima, int n, int t, int u, float* __restrict__ result) {
  const int lane = threadIdx.x & 31;
  const int b = blockIdx.x * (kStreamThreads / 32) + (threadIdx.x >> 5);
  if (b >= u * u) return;
  const int y0 = blockIdx.y * chunk, y1 = min(count, y0 + chunk);
  const int q = t / 4, nv = t * q;  // float4s per tile row, per tile
  const float* base = images + (size_t)(b / u) * t * n + (size_t)(b % u) * t;
  unsigned off[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int k = lane + 32 * i;
    off[i] = (unsigned)((k / q) * n + (k % q) * 4);
  }
  auto load = [&](float4(&v)[NV], int sl) {
    const float* img = base + (size_t)sl * img_stride;
#pragma unroll
    for (int i = 0; i < NV; ++i)
      if (lane + 32 * i < nv) v[i] = __ldcs(reinterpret_cast<const float4*>(img + off[i]));
  };
  // Triple y from slices (P0, P1, P2); slice y + 3 is loaded into NX first
  // so that its latency hides behind the reduction.
  auto step = [&](float4(&P0)[NV], float4(&P1)[NV], float4(&P2)[NV], float4(&NX)[NV], int y) {
    if (y + 1 < y1) load(NX, y + 3);
    Acc a{0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < NV; ++i)
      if (lane + 32 * i < nv) {
        acc_pixel<PRECISE>(a, P0[i].x, P1[i].x, P2[i].x);
        acc_pixel<PRECISE>(a, P0[i].y, P1[i].y, P2[i].y);
        acc_pixel<PRECISE>(a, P0[i].z, P1[i].z, P2[i].z);
        acc_pixel<PRECISE>(a, P0[i].w, P1[i].w, P2[i].w);
      }
    double S, R;
    float M;
    warp_stats<PRECISE>(a, S, R, M);
    if (lane == 0) {
      const float max3[3] = {maxima[y], maxima[y + 1], maxima[y + 2]};
      result[(size_t)y * u * u + b] = tlisi_of<PRECISE>(S, R, M, max3, t);
    }
  };
  // Four slice buffers whose roles rotate with the triple (no copies).
  float4 s0[NV], s1[NV], s2[NV], s3[NV];
  load(s0, y0);
  load(s1, y0 + 1);
  load(s2, y0 + 2);
  for (int y = y0; y < y1; y += 4) {
    step(s0, s1, s2, s3, y);
    if (y + 1 >= y1) break;
    step(s1, s2, s3, s0, y + 1);
    if (y + 2 >= y1) break;
    step(s2, s3, s0, s1, y + 2);
    if (y + 3 >= y1) break;
    step(s3, s0, s1, s2, y + 3);
  }
}

// Final pass of the fused trigger: tLISI from the statistics and the maxima.
template <bool PRECISE>
__global__ void k_trigger_combine(const double* __restrict__ stats, const float* __restrict__ max3p,
                                  int u, int t, float* __restrict__ result) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= u * u) return;
  const float max3[3] = {max3p[0], max3p[1], max3p[2]};
  result[b] = tlisi_of<PRECISE>(stats[3 * b], stats[3 * b + 1], (float)stats[3 * b + 2], max3, t);
}

inline float cell_degrees(float cell) { return (float)((double)cell / FIP_M_PI * 180); }

inline int sm_count() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

}  // namespace

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------

cudaError_t fip_launch_taper(float* taper, const FipGeom& geo, cudaStream_t s) {
  const int cnt = geo.n / 2 + 1;
  k_taper<<<(cnt + kThreads - 1) / kThreads, kThreads, 0, s>>>(taper, (size_t)geo.n,
                                                                (size_t)geo.g);
  return cudaGetLastError();
}

bool fip_bin_batchable(const FipGeom& geo) {
  return (size_t)geo.tiles_r * geo.tiles_c <= (size_t)kMaxSmemTiles;
}

int fip_bin_launches(const FipGeom& geo) { return fip_bin_batchable(geo) ? 3 : 4; }

// An item's fixed cost (zeroing and committing its tile) asks for large chunks,
// a launch with few items for enough of them to fill the device: two per SM,
// about 1.4 entries per visibility.  Two, four and eight items per SM wanted,
// us: three-snapshot calls at 4096^2 929 / 940 / 951 (plain), 568 / 578 / 590
// (FP16), at 512^2 72 / 76 / 76.  The 148 is a B200's SMs, fixed so that the
// bound of the work list (FIP_GITEMS_SPARE) holds whatever the device reports.
unsigned fip_grid_chunk(size_t nb) {
  const size_t want = (size_t)(1.4 * (double)nb) / (2 * 148);
  return (unsigned)std::max<size_t>(64, std::min<size_t>(FIP_GCHUNK_MAX, want / 32 * 32));
}

int fip_bin_ctas(int count, size_t nbmax) {
  // Two CTAs per SM for one snapshot, four for several (eight snapshots of
  // 0.45 M visibilities: 109 -> 102 us of the three kernels; one of 1.05 M: 43
  // -> 46).
  const size_t per = (size_t)kBinThreads;
  const int most = count > 1 ? kFipBinCtas / count : kFipBinCtas / 2;
  return std::max(1, (int)std::min<size_t>(most, (nbmax + per - 1) / per));
}

FipBinSnap fip_bin_snap(const FipGeom& geo, const float* B, int nb, const FipBins& bins,
                        float2* grid, unsigned* clear) {
  FipBinSnap q{};
  q.B = B;
  q.nb = nb;
  q.scale = geo.cell * (float)(size_t)geo.g;  // r1r2_scale (FIPkernels.cu:584)
  q.g = geo.g;
  q.hp = geo.hp;
  q.tiles_c = geo.tiles_c;
  q.ntiles = geo.tiles_r * geo.tiles_c;
  q.layout = geo.layout;
  q.wcap = (unsigned)bins.wcap;
  q.count = bins.count;
  q.offset = bins.offset;
  q.cursor = bins.cursor;
  q.entries = bins.entries;
  q.work = bins.work;
  q.nwork = bins.nwork;
  q.bbox = bins.bbox;
  q.multi = bins.multi;
  q.nmulti = bins.nmulti;
  q.grid = grid;
  q.clear = clear;
  return q;
}

cudaError_t fip_launch_bin_batch(FipBinBatch& in, unsigned* base, cudaStream_t s) {
  if (in.count < 1 || in.count > FIP_MAX_BATCH) return cudaErrorInvalidValue;
  int ntiles = 0, nb = 0;
  size_t total = 0;
  for (int k = 0; k < in.count; ++k) {
    ntiles = std::max(ntiles, in.s[k].ntiles);
    nb = std::max(nb, in.s[k].nb);
    total += (size_t)in.s[k].nb;
  }
  if (ntiles > kMaxSmemTiles) return cudaErrorInvalidValue;
  const int ctas = fip_bin_ctas(in.count, (size_t)nb);
  const unsigned chunk = fip_grid_chunk(total);
  for (int k = 0; k < in.count; ++k) {
    in.s[k].chunk = chunk;
    in.s[k].base = base ? base + (size_t)k * ctas * ntiles : nullptr;
  }
  const size_t smem = (size_t)ntiles * sizeof(unsigned);
  const dim3 grid(ctas, in.count);
  k_bin_count<<<grid, kBinThreads, smem, s>>>(in);
  k_bin_scan_tiles<<<in.count, kScanThreads, smem, s>>>(in);
  k_bin_scatter<<<grid, kBinThreads, smem, s>>>(in);
  return cudaGetLastError();
}

cudaError_t fip_launch_bin(const FipGeom& geo, const float* B, int nb, FipBins& bins,
                           float2* grid, cudaStream_t s) {
  const int ntiles = geo.tiles_r * geo.tiles_c;
  const float scale = geo.cell * (float)(size_t)geo.g;  // r1r2_scale (FIPkernels.cu:584)
  cudaError_t e = cudaMemsetAsync(bins.count, 0, ntiles * sizeof(unsigned), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(bins.bbox, 0, 4 * sizeof(unsigned), s);
  if (e != cudaSuccess) return e;
  if (fip_bin_batchable(geo)) {
    FipBinBatch in;
    in.count = 1;
    in.s[0] = fip_bin_snap(geo, B, nb, bins, grid);
    return fip_launch_bin_batch(in, bins.base, s);
  }
  const int blocks = (nb + kThreads - 1) / kThreads;
  if (nb > 0)
    k_bin<0><<<blocks, kThreads, 0, s>>>(B, nb, scale, geo.g, geo.tiles_c, bins.count, nullptr,
                                         nullptr, bins.bbox);
  k_bin_scan<<<1, kScanThreads, 0, s>>>(bins.count, bins.bbox, ntiles, geo.tiles_c, geo.g,
                                    geo.layout, bins.offset, bins.cursor, bins.work, bins.nwork,
                                    (int)bins.wcap, bins.multi, bins.nmulti);
  if (nb > 0)
    k_bin<1><<<blocks, kThreads, 0, s>>>(B, nb, scale, geo.g, geo.tiles_c, bins.cursor,
                                         bins.offset, bins.entries, nullptr);
  if (grid)
    k_zero_tiles<<<sm_count(), kThreads, 0, s>>>(bins.multi, bins.nmulti, geo.tiles_c, geo.g,
                                                 geo.hp, geo.layout, grid);
  return cudaGetLastError();
}

// CTAs per SM that fit: the precision form's shared memory (the tile and its
// low limbs) allows three, the plain form's registers four.
int fip_grid_max_ctas_per_sm(int compensated) { return compensated ? 3 : 4; }

cudaError_t fip_launch_grid(const FipGeom& geo, const float* B, const void* vr, const void* vi,
                            int vis_type, const float* vis_scale, const float* V, int nb,
                            const FipBins& bins, float2* grid, int compensated, cudaStream_t s,
                            int ctas_per_sm, const FipRawVis* raw) {
  if (vis_type == FIP_VIS_RAW && !raw) return cudaErrorInvalidValue;
  const FipRawVis rv = raw ? *raw : FipRawVis{};
  const float scale = geo.cell * (float)(size_t)geo.g;
  const int sms = sm_count();
  const size_t smem = grid_smem_bytes(compensated != 0);
  const int most = fip_grid_max_ctas_per_sm(compensated);
  const int blocks = sms * (ctas_per_sm > 0 ? min(ctas_per_sm, most) : most);
#define FIP_GRID_CASE(VT, C)                                                                    \
  do {                                                                                          \
    auto kern = k_grid<VT, C>;                                                                  \
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);         \
    kern<<<blocks, kThreads, smem, s>>>(B, vr, vi, vis_scale, V, scale, geo.g, geo.hp,          \
                                        geo.tiles_c, geo.layout, bins.entries, bins.work,       \
                                        bins.nwork, grid, rv);                                  \
  } while (0)
  if (vis_type == FIP_VIS_RAW) {
    if (compensated) FIP_GRID_CASE(FIP_VIS_RAW, true); else FIP_GRID_CASE(FIP_VIS_RAW, false);
  } else if (vis_type == FIP_VIS_F32) {
    if (compensated) FIP_GRID_CASE(FIP_VIS_F32, true); else FIP_GRID_CASE(FIP_VIS_F32, false);
  } else if (vis_type == FIP_VIS_F16) {
    if (compensated) FIP_GRID_CASE(FIP_VIS_F16, true); else FIP_GRID_CASE(FIP_VIS_F16, false);
  } else {
    if (compensated) FIP_GRID_CASE(FIP_VIS_BF16, true); else FIP_GRID_CASE(FIP_VIS_BF16, false);
  }
#undef FIP_GRID_CASE
  (void)nb;
  return cudaGetLastError();
}

cudaError_t fip_launch_grid_batch(const FipGridBatch& in, int vis_type, int compensated,
                                  cudaStream_t s, int ctas_per_sm) {
  if (in.count < 1 || in.count > FIP_MAX_BATCH) return cudaErrorInvalidValue;
  const int sms = sm_count();
  const size_t smem = grid_smem_bytes(compensated != 0);
  const int most = fip_grid_max_ctas_per_sm(compensated);
  const int blocks = sms * (ctas_per_sm > 0 ? min(ctas_per_sm, most) : most);
#define FIP_GRID_CASE(VT, C)                                                                   \
  do {                                                                                         \
    auto kern = k_grid_batch<VT, C>;                                                           \
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);        \
    kern<<<blocks, kThreads, smem, s>>>(in);                                                   \
  } while (0)
  if (vis_type == FIP_VIS_F32) {
    if (compensated) FIP_GRID_CASE(FIP_VIS_F32, true); else FIP_GRID_CASE(FIP_VIS_F32, false);
  } else if (vis_type == FIP_VIS_F16) {
    if (compensated) FIP_GRID_CASE(FIP_VIS_F16, true); else FIP_GRID_CASE(FIP_VIS_F16, false);
  } else {
    if (compensated) FIP_GRID_CASE(FIP_VIS_BF16, true); else FIP_GRID_CASE(FIP_VIS_BF16, false);
  }
#undef FIP_GRID_CASE
  return cudaGetLastError();
}

const void* fip_targets_kernel() { return reinterpret_cast<const void*>(&k_targets<false>); }

cudaError_t fip_launch_targets(const FipGeom& geo, const float* V, const float2* theta_tab,
                               float2* targets, cudaStream_t s, int batch, size_t stride) {
  if (batch < 1 || batch > 65535) return cudaErrorInvalidValue;
  const int per = kThreads * kTargetsPerThread;
  dim3 bl((geo.n + per - 1) / per, geo.n, batch);
  auto kern = batch > 1 ? k_targets<true> : k_targets<false>;
  kern<<<bl, kThreads, 0, s>>>(V, geo.n, cell_degrees(geo.cell), theta_tab, targets, stride);
  return cudaGetLastError();
}

cudaError_t fip_launch_reproject_scatter(const FipGeom& geo, const float* pre, const float* V,
                                         int nb, float* dst, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(dst, 0, (size_t)geo.n * geo.n * sizeof(float), s);
  if (e != cudaSuccess) return e;
  dim3 th(32, 8), bl((geo.n + 31) / 32, (geo.n + 7) / 8);
  k_reproject_scatter<<<bl, th, 0, s>>>(pre, V, geo.n, nb, cell_degrees(geo.cell), dst);
  return cudaGetLastError();
}

// Target deviation allowance of the FP32 chain from the exact map, in
// destination pixels: half a pixel plus eight ulps of a unit-scale cosine
// expressed in pixels (the chain evaluates cos(theta) ~ R in degrees).
static float chain_delta(float cell) { return 0.5f + 8.0f * 4.76837158e-7f / cell; }

bool fip_gather_supported(const FipGeom& geo, int exact_targets) {
  return exact_targets || chain_delta(geo.cell) <= 40.f;
}

bool fip_trigger_fusable(const FipGeom& geo) {
  return geo.t > 0 && kDT % geo.t == 0 && geo.n % kDT == 0;
}

size_t fip_trigger_fuse_counts(const FipGeom& geo) {
  const size_t tiles = (geo.n + kDT - 1) / kDT;
  return tiles * tiles;
}

cudaError_t fip_launch_reproject_gather(const FipGeom& geo, const FipGatherBatch& in,
                                        const float* pre, const float2* targets,
                                        const unsigned* pre_max, int exact_targets,
                                        cudaStream_t s, unsigned* err, const FipFuse* fuse) {
  const int tiles = (geo.n + kDT - 1) / kDT;
  const float delta = exact_targets ? 0.25f : chain_delta(geo.cell);
  if (in.count < 1 || in.count > FIP_MAX_BATCH) return cudaErrorInvalidValue;
  if (!fip_gather_supported(geo, exact_targets)) return cudaErrorInvalidValue;
  FipTriggerFuse tf{};
  if (fuse) {
    if (!fip_trigger_fusable(geo)) return cudaErrorInvalidValue;
    for (int k = 0; k < 3; ++k) tf.img[k] = fuse->img[k];
    tf.count = fuse->count;
    tf.stats = fuse->stats;
    tf.t = geo.t;
    tf.u = geo.u;
  }
  const dim3 blocks(tiles * tiles, in.count);
  const float2* tg = exact_targets ? nullptr : targets;
  auto kern = exact_targets
                  ? (in.count > 1 ? k_reproject_gather<true, true> : k_reproject_gather<true, false>)
                  : (in.count > 1 ? k_reproject_gather<false, true>
                                  : k_reproject_gather<false, false>);
  kern<<<blocks, kThreads, 0, s>>>(in, pre, tg, geo.n, geo.cell, delta, pre_max, err, tf);
  return cudaGetLastError();
}

cudaError_t fip_launch_reproject_rest(const FipGeom& geo, const FipGatherBatch& in,
                                      const float* pre, const unsigned* plans,
                                      const unsigned* pre_max, cudaStream_t s, unsigned* err) {
  if (in.count < 1 || in.count > FIP_MAX_BATCH) return cudaErrorInvalidValue;
  const int tiles = (geo.n + kDT - 1) / kDT;
  const dim3 blocks(std::min(tiles * tiles, 5 * sm_count()), in.count);
  k_reproject_rest<<<blocks, kThreads, 0, s>>>(in, pre, geo.n, geo.cell, 0.25f, pre_max, err,
                                               plans,
                                               (int)(fip_pull_plan_words(geo) / (tiles * tiles)));
  return cudaGetLastError();
}

cudaError_t fip_launch_trigger_combine(const FipGeom& geo, const double* stats,
                                       const float* max3, float* result, int precise,
                                       cudaStream_t s) {
  const int tiles = geo.u * geo.u;
  if (tiles == 0) return cudaSuccess;
  const int blocks = (tiles + kThreads - 1) / kThreads;
  if (precise)
    k_trigger_combine<true><<<blocks, kThreads, 0, s>>>(stats, max3, geo.u, geo.t, result);
  else
    k_trigger_combine<false><<<blocks, kThreads, 0, s>>>(stats, max3, geo.u, geo.t, result);
  return cudaGetLastError();
}

bool fip_gather_domain_ok(const float* V, int n, float cell) {
  // The exact map on a 65 x 65 lattice over the source image (and one pixel
  // beyond): inside the horizon with room (r2 < 0.98) and no fold of the
  // slant part (its Jacobian determinant above 1/4), the conditions the
  // gather checks per tile.  V is row-major 3 x 3 on the host.
  const double a22 = fabs((double)V[8]);
  if (!(a22 > 0.0)) return false;
  const double m00 = -(double)V[0] / a22, m01 = (double)V[3] / a22;
  const double m10 = -(double)V[1] / a22, m11 = (double)V[4] / a22;
  const double xi = (double)V[6] / (double)V[8], eta = (double)V[7] / (double)V[8];
  const double h = n / 2, lo = -h - 2.0, span = (double)n + 4.0;
  for (int q = 0; q <= 64; ++q)
    for (int p = 0; p <= 64; ++p) {
      const double a = lo + span * p / 64.0, b = lo + span * q / 64.0;
      const double X = cell * (m00 * a + m01 * b - 1.0), Y = cell * (m10 * a + m11 * b - 1.0);
      const double r2 = X * X + Y * Y;
      if (!(r2 < 0.98)) return false;
      const double nn = sqrt(1.0 - r2);
      if (!(1.0 - xi * X / nn + eta * Y / nn > 0.25)) return false;
    }
  return true;
}

cudaError_t fip_launch_image_max(const float* img, size_t count, unsigned* out, cudaStream_t s) {
  k_image_max<<<1184, kThreads, 0, s>>>(img, count, out);
  return cudaGetLastError();
}

// ---- The streamed sliding-window trigger ----------------------------------
static std::atomic<int> g_trigger_stream{1};

void fip_trigger_stream_enable(int on) { g_trigger_stream.store(on ? 1 : 0); }
int fip_trigger_stream_enabled() { return g_trigger_stream.load(); }

template <bool PRECISE>
static cudaError_t launch_stream_window(const FipGeom& geo, const float* images, int count,
                                        const float* maxima, float* results, cudaStream_t s) {
  const int tiles = geo.u * geo.u;
  const int bx = (tiles + kStreamThreads / 32 - 1) / (kStreamThreads / 32);
  // Chunks of triples: enough warps to fill the device (about eight waves
  // of 12 warps per SM), each chunk re-reading only its first two slices.
  const int want = 8 * 12 * sm_count();
  int chunks = std::max(1, std::min(count, want / std::max(1, tiles)));
  const int chunk = (count + chunks - 1) / chunks;
  chunks = (count + chunk - 1) / chunk;
  if (chunks > 65535) return cudaErrorInvalidValue;
  const dim3 grid(bx, chunks);
  const size_t n2 = (size_t)geo.n * geo.n;
  const int nv = (geo.t * geo.t / 4 + 31) / 32;
#define FIP_STREAM(NV)                                                                         \
  k_trigger_stream<PRECISE, NV><<<grid, kStreamThreads, 0, s>>>(                               \
      images, n2, count, chunk, maxima, geo.n, geo.t, geo.u, results)
  if (nv <= 1)
    FIP_STREAM(1);
  else if (nv <= 2)
    FIP_STREAM(2);
  else if (nv <= 4)
    FIP_STREAM(4);
  else
    FIP_STREAM(8);
#undef FIP_STREAM
  return cudaGetLastError();
}

cudaError_t fip_launch_trigger(const FipGeom& geo, const float* I1, const float* I2,
                               const float* I3, const float* max3, float* stats, float* result,
                               int precise, cudaStream_t s) {
  (void)stats;
  return fip_launch_trigger3(geo, I1, I2, I3, max3, max3 + 1, max3 + 2, result, precise, s);
}

cudaError_t fip_launch_trigger3(const FipGeom& geo, const float* I1, const float* I2,
                                const float* I3, const float* m1, const float* m2,
                                const float* m3, float* result, int precise, cudaStream_t s) {
  const int tiles = geo.u * geo.u;
  const int blocks = (tiles + kThreads / 32 - 1) / (kThreads / 32);
  if (tiles == 0) return cudaSuccess;
  const int vec = (geo.t % 4 == 0) && (geo.n % 4 == 0) &&
                  ((((uintptr_t)I1) | ((uintptr_t)I2) | ((uintptr_t)I3)) & 15) == 0;
  if (precise)
    k_trigger<true, false><<<blocks, kThreads, 0, s>>>(I1, I2, I3, m1, m2, m3, geo.n, geo.t, geo.u, vec,
                                                result, 0, 0, 0, 0);
  else
    k_trigger<false, false><<<blocks, kThreads, 0, s>>>(I1, I2, I3, m1, m2, m3, geo.n, geo.t, geo.u,
                                                 vec, result, 0, 0, 0, 0);
  return cudaGetLastError();
}

cudaError_t fip_launch_trigger_ring(const FipGeom& geo, const float* images, const float* maxima,
                                    int ring, int first, int count, float* results, int precise,
                                    cudaStream_t s) {
  const int tiles = geo.u * geo.u;
  if (tiles == 0 || count <= 0) return cudaSuccess;
  if (count > 65535 || ring < 3) return cudaErrorInvalidValue;
  const size_t n2 = (size_t)geo.n * geo.n;
  const dim3 blocks((tiles + kThreads / 32 - 1) / (kThreads / 32), count);
  const int vec = (geo.t % 4 == 0) && (geo.n % 4 == 0) && ((uintptr_t)images & 15) == 0;
  auto kern = precise ? k_trigger<true, true> : k_trigger<false, true>;
  kern<<<blocks, kThreads, 0, s>>>(images, images, images, maxima, maxima, maxima, geo.n, geo.t,
                                   geo.u, vec, results, n2, (size_t)tiles, ring, first);
  return cudaGetLastError();
}

cudaError_t fip_launch_trigger_batch(const FipGeom& geo, const float* images, const float* maxima,
                                     int count, float* results, int precise, cudaStream_t s) {
  const int tiles = geo.u * geo.u;
  if (tiles == 0 || count <= 0) return cudaSuccess;
  if (count > 65535) return cudaErrorInvalidValue;
  // Plain form, three or more triples: the register stream (each image read
  // once).  The precision form's compensated sums make it issue-bound; its
  // triples keep the plain loads, which hide latency with more warps.
  if (g_trigger_stream.load() && !precise && count >= 3 && geo.t % 4 == 0 && geo.t <= 32 &&
      geo.n % 4 == 0 && ((uintptr_t)images & 15) == 0)
    return launch_stream_window<false>(geo, images, count, maxima, results, s);
  const size_t n2 = (size_t)geo.n * geo.n;
  const dim3 blocks((tiles + kThreads / 32 - 1) / (kThreads / 32), count);
  const int vec = (geo.t % 4 == 0) && (geo.n % 4 == 0) && ((uintptr_t)images & 15) == 0;
  if (precise)
    k_trigger<true, false><<<blocks, kThreads, 0, s>>>(images, images + n2, images + 2 * n2, maxima,
                                                maxima + 1, maxima + 2, geo.n, geo.t, geo.u, vec,
                                                results, n2, (size_t)tiles, 0, 0);
  else
    k_trigger<false, false><<<blocks, kThreads, 0, s>>>(images, images + n2, images + 2 * n2, maxima,
                                                 maxima + 1, maxima + 2, geo.n, geo.t, geo.u,
                                                 vec, results, n2, (size_t)tiles, 0, 0);
  return cudaGetLastError();
}

cudaError_t fip_launch_pixel_targets(const FipGeom& geo, const float* V, float* out,
                                     int mode, const float2* theta_tab, cudaStream_t s) {
  if (mode < 0 || mode > 2) return cudaErrorInvalidValue;
  dim3 bl((geo.n + kThreads - 1) / kThreads, geo.n);
  k_pixel_targets<<<bl, kThreads, 0, s>>>(V, geo.n, cell_degrees(geo.cell), geo.cell, mode,
                                          theta_tab, out);
  return cudaGetLastError();
}

size_t fip_theta_table_elems() { return (size_t)fipref::kThetaTabSize; }

cudaError_t fip_launch_theta_table(float2* tab, cudaStream_t s) {
  k_theta_table<<<(fipref::kThetaTabSize + kThreads - 1) / kThreads, kThreads, 0, s>>>(tab);
  return cudaGetLastError();
}
