// The precision form's reprojection by destination pixel.
//
// Every destination pixel sums the sources whose exact targets lie within one
// pixel of it, with the bilinear weights of the forward splat
// (FIPkernels.cu:394-410): out(x, y) = sum_s pre_s (1 - |L_s - x|)+ (1 - |M_s - y|)+ / nb,
// the same sum the splat accumulates source by source.  While the map is
// nearly a rotation with a stretch of at least one (every image plane that is
// not folded; the plan below checks it tile by tile), those sources lie among
// the 3 x 3 around the pixel's preimage, so a pixel costs nine shared-memory
// reads and no atomics, conversions or candidate lists.
//
// Two kernels: k_pull_plan, a few lanes per tile, depends on the plane only:
// the tile's domain and extent, the map and its inverse expanded to second
// order about the tile's centre in FP64.  k_pull, a CTA per 64 x 64 tile,
// brings the tile's source patch into shared memory with bulk tensor copies
// (zeros outside the image) and evaluates its pixels from the expansion.
// Tiles outside the expansion's range (wide cells, odd planes) keep the splat
// (fip_launch_reproject_gather's rest list).
//
// Accuracy: targets within 1.1e-6 pixel RMS of the exact map over most planes and
// 1.3e-6 where the coarser form ends (7.5e-6 at most), against the splat's 1.5e-6
// (9e-6): the FP32 arithmetic of both emulated on the host over 16 geometries.
// The expansion's origin is the source pixel nearest to the tile centre's source,
// so that positions round as offsets within a tile.
//
// Bound: instruction issue (18 tents, 24 additions, 22 multiply-adds and 13
// products among 102 instructions a pixel, 74 % of the issue slots) with the
// shared-memory loads (2.3 wavefronts a read at a 20 degree turn, 64 % of their
// rate) beside it.  4096^2: 68 us (and 6 us of plan beside the binning, 3 us for
// the empty rest list) against 86 us for the splat's 122 instructions a pixel;
// three-snapshot FP16 calls 632 -> 590 us, FP32 674 -> 629; images' error against
// FP64 2.3e-6 -> 1.2e-6 at 1024^2 (no fixed-point sums).  The finer form of curved
// tiles adds 13 us.  All-scalar arithmetic: 118 instructions, 70.5 us.  Five CTAs
// per SM (48 registers): 71.5 us.  Patch rows of 108 floats: the same.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "fip_common.cuh"
#include "fip_kernels.h"
#include "fip_map.cuh"
#include "fip_tma.cuh"

namespace {

constexpr int kThreads = 256;
// Source patch: rows of kPW floats (26 16-byte units: an 8 x 4 block of pixels
// reads distinct banks whether the map turns it by 0 or by 90 degrees), in
// kChunk-row copies.
constexpr int kPW = 104, kPH = 100, kChunk = 20;
constexpr int kPatchBytes = kPW * kPH * 4;
static_assert(kPH % kChunk == 0 && (kPW * 4) % 16 == 0 && (kPW * kChunk * 4) % 128 == 0,
              "TMA box and destination alignment");

// What one tile needs.
struct Plan {
  int a_lo, b_lo;  // patch origin (source pixel; a_lo a multiple of 4)
  int rows;        // patch rows, 0: the tile keeps the splat
  int flags;       // kInner, kFine
  int at;          // patch index of the corner of the 3 x 3 around the origin, the
                   // source pixel nearest to the tile centre's source
  float ac, bc;    // the centre's source, relative to the origin (within half a pixel)
  float a00, a01, a10, a11;            // d source / d destination
  float ka, kb, h11, h12, h22;         // second order: source += (ka, kb) quad(dx, dy),
  float lx, ly;                        // third: (ka, kb) quad (lx dx + ly dy)
  float j0[4], jx[4], jy[4];           // d(L, M)/da, d(L, M)/db at the centre, per dx, per dy
  float ea[2], eb[2], eab[2];          // second order of unit source steps along a, b, both
};
constexpr int kPlanWords = sizeof(Plan) / 4;
// kInner: no target of the tile's sources can leave the image.  kFine: the
// nearest source's target is taken to second order in its offset, the Jacobian
// at the source rather than at the pixel, and a diagonal step's cross term is
// kept.
constexpr int kInner = 1, kFine = 2;

// Curvature of the map (pixels per pixel^2) above which a tile is kFine, and
// above which it keeps the splat; and the bound, in pixels, on the orders left
// out over the tile (see k_pull_plan).
constexpr double kCurvFine = 6e-6, kCurvMax = 4.5e-5, kPullSlack = 3e-6;

// kPoly lanes per tile; snapshot blockIdx.y.
__global__ void __launch_bounds__(kThreads) k_pull_plan(const __grid_constant__ FipGatherBatch in,
                                                        int n, float cell, int tiles,
                                                        Plan* __restrict__ plans) {
  const int lane = threadIdx.x & 31;
  const int tile = (int)((blockIdx.x * kThreads + threadIdx.x) / kPoly);
  const bool on = tile < tiles * tiles;
  const int tt = on ? tile : 0;
  const int r0 = (tt / tiles) * kDT, c0 = (tt % tiles) * kDT, h = n / 2;
  const float* V = in.V[blockIdx.y];
  float va, vb;
  const TilePreimage pr =
      trace_preimage(make_map_f32(V, cell), r0, c0, h, 0.25f, cell, lane, va, vb);
  if (!on || (lane % kPoly) != 0) return;
  Plan p{};
  const ExactMap<double> m = make_map<double>(V, cell);
  // The centre's source: (P1, P2) = (L + xi z, M - eta z), z the slant term at P
  // (a contraction in the domain; Newton on z).
  const double Lc = (double)(c0 - h) + 0.5 * (kDT - 1), Mc = (double)(r0 - h) + 0.5 * (kDT - 1);
  const double w0 = -m.xi, w1 = m.eta;
  double z = 0.0, Q1 = 0.0, Q2 = 0.0, s = 1.0, det = 1.0;
  bool ok = pr.ok;
  for (int it = 0; it < 6 && ok; ++it) {
    Q1 = Lc - w0 * z - 1.0;
    Q2 = Mc - w1 * z - 1.0;
    const double rho = m.cell * m.cell * (Q1 * Q1 + Q2 * Q2);
    ok = rho < 0.98;
    if (!ok) break;
    s = sqrt(1.0 - rho);
    det = 1.0 + m.cell / s * (Q1 * w0 + Q2 * w1);
    const double step = ((rho / (1.0 + s)) / m.cell - z) / det;
    z += step;
    if (fabs(step) < 1e-10) break;
  }
  if (ok) {
    const double P1 = Lc - w0 * z, P2 = Mc - w1 * z;
    const double as = m.i00 * P1 + m.i01 * P2, bs = m.i10 * P1 + m.i11 * P2;
    // Gradient and Hessian of z in P, K = d P / d (L, M).
    const double G0 = m.cell * Q1 / s, G1 = m.cell * Q2 / s, is = m.cell / s;
    const double H00 = is * (1.0 + G0 * G0), H01 = is * G0 * G1, H11 = is * (1.0 + G1 * G1);
    const double K00 = 1.0 - w0 * G0 / det, K01 = -w0 * G1 / det;
    const double K10 = -w1 * G0 / det, K11 = 1.0 - w1 * G1 / det;
    p.a00 = (float)(m.i00 * K00 + m.i01 * K10);
    p.a01 = (float)(m.i00 * K01 + m.i01 * K11);
    p.a10 = (float)(m.i10 * K00 + m.i11 * K10);
    p.a11 = (float)(m.i10 * K01 + m.i11 * K11);
    const double N00 = H00 * K00 + H01 * K10, N01 = H00 * K01 + H01 * K11;
    const double N10 = H01 * K00 + H11 * K10, N11 = H01 * K01 + H11 * K11;
    p.h11 = (float)(0.5 / det * (K00 * N00 + K10 * N10));
    p.h12 = (float)(1.0 / det * (K00 * N01 + K10 * N11));
    p.h22 = (float)(0.5 / det * (K01 * N01 + K11 * N11));
    p.ka = (float)-(m.i00 * w0 + m.i01 * w1);
    p.kb = (float)-(m.i10 * w0 + m.i11 * w1);
    // d(L, M)/d(a, b) = m + w (G . m_column), G linear over the tile.
    const double mc[2][2] = {{m.m00, m.m10}, {m.m01, m.m11}};
    for (int q = 0; q < 2; ++q) {
      const double g = G0 * mc[q][0] + G1 * mc[q][1];
      const double gx = N00 * mc[q][0] + N10 * mc[q][1], gy = N01 * mc[q][0] + N11 * mc[q][1];
      p.j0[2 * q] = (float)(mc[q][0] + w0 * g);
      p.j0[2 * q + 1] = (float)(mc[q][1] + w1 * g);
      p.jx[2 * q] = (float)(w0 * gx);
      p.jx[2 * q + 1] = (float)(w1 * gx);
      p.jy[2 * q] = (float)(w0 * gy);
      p.jy[2 * q + 1] = (float)(w1 * gy);
      const double e = 0.5 * (H00 * mc[q][0] * mc[q][0] + 2.0 * H01 * mc[q][0] * mc[q][1] +
                              H11 * mc[q][1] * mc[q][1]);
      float* ev = q ? p.eb : p.ea;
      ev[0] = (float)(w0 * e);
      ev[1] = (float)(w1 * e);
    }
    const double eab = H00 * m.m00 * m.m01 + H01 * (m.m00 * m.m11 + m.m10 * m.m01) +
                       H11 * m.m10 * m.m11;
    p.eab[0] = (float)(w0 * eab);
    p.eab[1] = (float)(w1 * eab);
    p.lx = (float)(-(N00 * w0 + N10 * w1) / det);
    p.ly = (float)(-(N01 * w0 + N11 * w1) / det);
    // Left out over the tile: the fourth order of the curvature and the slant
    // term's own third derivative, at the half diagonal; and, without kFine, per
    // source the curvature over the steps of a pixel or less (three quarters of
    // it, and the cross term).
    const double wn = fabs(w0) + fabs(w1), curv = wn * is / (s * s * det), R = 46.0;
    const double left = curv * curv * curv * R * R * R * R +
                        0.5 * wn * is * is * sqrt(G0 * G0 + G1 * G1) / (s * s) * R * R * R;
    ok = left < kPullSlack && curv < kCurvMax;
    const bool fine = curv > kCurvFine || wn * fabs(eab) > 0.5 * kCurvFine;
    // A pixel's sources within one of its nearest: a unit square of
    // destinations spans less than 1.5 sources either way, across the tile.
    const double grow = 1.0 + 46.0 * 4.0 * curv;
    ok = ok && (fabs(p.a00) + fabs(p.a01)) * grow < 1.49 &&
         (fabs(p.a10) + fabs(p.a11)) * grow < 1.49;
    // Patch: the polygon's extent, the window and rounding
    // (the polygon reaches 1.25 destinations past the outermost pixels, the
    // window 1.5 sources past theirs).
    const int amin = (int)floorf(pr.amin - pr.sag) + h - 1, amax = (int)ceilf(pr.amax + pr.sag) + h + 1;
    const int bmin = (int)floorf(pr.bmin - pr.sag) + h - 1, bmax = (int)ceilf(pr.bmax + pr.sag) + h + 1;
    const int alo = amin & ~3;
    ok = ok && amax - alo < kPW && bmax - bmin < kPH;
    p.a_lo = alo;
    p.b_lo = bmin;
    const double ao = rint(as), bo = rint(bs);
    p.at = ((int)bo + h - bmin - 1) * kPW + (int)ao + h - alo - 1;
    p.ac = (float)(as - ao);
    p.bc = (float)(bs - bo);
    p.rows = ok ? bmax - bmin + 1 : 0;
    const bool inner = c0 >= 4 && c0 + kDT + 4 <= 2 * h && r0 >= 4 && r0 + kDT + 4 <= 2 * h;
    p.flags = (inner ? kInner : 0) | (fine ? kFine : 0);
  }
  plans[(size_t)blockIdx.y * tiles * tiles + tile] = p;
}

// (1 - |x|)+ in one instruction.
__device__ __forceinline__ float tent(float x) {
  float r;
  asm("{\n .reg .f32 t;\n abs.f32 t, %1;\n sub.ftz.sat.f32 %0, 0f3F800000, t;\n}"
      : "=f"(r)
      : "f"(x));
  return r;
}

// Pairs of FP32 values in one 64-bit register: one instruction for two
// additions or multiply-adds.  The products with the source values stay
// scalar (their pairs' moves cost more than they save: 145 against 126
// instructions a pixel).
typedef unsigned long long f2;
__device__ __forceinline__ f2 pk(float x, float y) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void upk(f2 v, float& x, float& y) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// One warp: 8 columns x 4 rows of pixels at a time, 16 times down the tile.
template <bool INNER, bool FINE>
__device__ __forceinline__ float pull_tile(const Plan& p, const float* __restrict__ patch, int r0,
                                           int c0, int n, float scale, float* __restrict__ dst) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int x = 8 * warp + (lane & 7), y0 = lane >> 3;
  const float dx = (float)x - 0.5f * (kDT - 1);
  // Horner coefficients in dy of the source position and the Jacobian:
  // quad (1 + l) with quad = q0 + q1 dy + q2 dy^2, l = l0 + ly dy.
  const float q0 = p.h11 * dx * dx, q1 = p.h12 * dx, q2 = p.h22, l0 = fmaf(p.lx, dx, 1.0f);
  const float k0 = q0 * l0, k1 = fmaf(q0, p.ly, q1 * l0), k2 = fmaf(q1, p.ly, q2 * l0);
  const float k3 = q2 * p.ly;
  const f2 s0 = pk(fmaf(p.ka, k0, fmaf(p.a00, dx, p.ac)), fmaf(p.kb, k0, fmaf(p.a10, dx, p.bc)));
  const f2 s1 = pk(fmaf(p.ka, k1, p.a01), fmaf(p.kb, k1, p.a11));
  const f2 s2 = pk(p.ka * k2, p.kb * k2), s3 = pk(p.ka * k3, p.kb * k3);
  const f2 ja0 = pk(fmaf(p.jx[0], dx, p.j0[0]), fmaf(p.jx[1], dx, p.j0[1]));
  const f2 jb0 = pk(fmaf(p.jx[2], dx, p.j0[2]), fmaf(p.jx[3], dx, p.j0[3]));
  const f2 jay = pk(p.jy[0], p.jy[1]), jby = pk(p.jy[2], p.jy[3]);
  const f2 ea = pk(p.ea[0], p.ea[1]), eb = pk(p.eb[0], p.eb[1]), eab = pk(p.eab[0], p.eab[1]);
  const f2 neg = pk(-1.0f, -1.0f);
  const float kMagic = 12582912.0f;  // 1.5 2^23: adding it rounds to an integer
  const int kBias = 0x4B400000;      // its bits
  const f2 magic = pk(kMagic, kMagic), nmagic = pk(-kMagic, -kMagic);
  const int h = n / 2;
  const float lim = (float)(n / 2 - 1);  // the reference compares |LL| with N/2 - 1
  const int count = c0 + x < n ? min(kDT / 4, (n - r0 - y0 + 3) / 4) : 0;
  float vmax = 0.f;
  float* out = dst + (size_t)(r0 + y0) * n + c0 + x;
  f2 dy2 = pk((float)y0 - 0.5f * (kDT - 1), (float)y0 - 0.5f * (kDT - 1));
  const f2 four = pk(4.0f, 4.0f);
#pragma unroll 2
  for (int i = 0; i < count; ++i, dy2 = add2(dy2, four), out += 4 * (size_t)n) {
    const f2 src = fma2(fma2(fma2(s3, dy2, s2), dy2, s1), dy2, s0);
    const f2 t = add2(src, magic);
    float ta, tb, fa, fb;
    upk(t, ta, tb);
    // The nearest source's offset from the pixel's preimage, and the corner
    // of its 3 x 3 (the plan keeps it inside the patch; the bound holds for
    // any plan).
    upk(fma2(src, neg, add2(t, nmagic)), fa, fb);
    const unsigned idx =
        (unsigned)((__float_as_int(tb) - kBias) * kPW + (__float_as_int(ta) - kBias) + p.at);
    const float* q = patch + min(idx, (unsigned)(kPW * (kPH - 2) - 3));
    f2 ja = fma2(jay, dy2, ja0), jb = fma2(jby, dy2, jb0);
    // Targets of the nearest source and its neighbours relative to the pixel.
    float au, av, bu, bv;
    upk(ja, au, av);
    upk(jb, bu, bv);
    float cu = fmaf(fa, au, fb * bu), cv = fmaf(fa, av, fb * bv);
    f2 c = pk(cu, cv);
    if (FINE) {
      const float aa = fa * fa, bb = fb * fb, ab = fa * fb;
      c = fma2(pk(aa, aa), ea, fma2(pk(bb, bb), eb, fma2(pk(ab, ab), eab, c)));
      upk(c, cu, cv);
      ja = pk(fmaf(p.jx[0], cu, fmaf(p.jy[0], cv, au)), fmaf(p.jx[1], cu, fmaf(p.jy[1], cv, av)));
      jb = pk(fmaf(p.jx[2], cu, fmaf(p.jy[2], cv, bu)), fmaf(p.jx[3], cu, fmaf(p.jy[3], cv, bv)));
    }
    const f2 ce = add2(c, ea), cf = add2(c, eb);
    const f2 ap = add2(ce, ja), am = fma2(ja, neg, ce);
    const f2 ape = add2(ap, eb), ame = add2(am, eb);
    // Diagonal steps: + eab where both steps have the same sign, - eab else.
    const f2 jq = FINE ? add2(jb, eab) : jb, jr = FINE ? fma2(eab, neg, jb) : jb;
    const f2 uv[9] = {fma2(jr, neg, ame), fma2(jb, neg, cf), fma2(jq, neg, ape), am, c, ap,
                      add2(ame, jr),      add2(cf, jb),      add2(ape, jq)};
    float wu[9], wv[9];
#pragma unroll
    for (int e = 0; e < 9; ++e) {
      float u, v;
      upk(uv[e], u, v);
      wu[e] = tent(u);
      wv[e] = tent(v);
      if (!INNER) {
        // A source whose target leaves the image is dropped altogether.
        const bool in =
            fabsf(u + (float)(c0 - h + x)) < lim && fabsf(v + (float)(r0 - h + y0 + 4 * i)) < lim;
        wu[e] = in ? wu[e] : 0.f;
      }
    }
    float sum = 0.f;
#pragma unroll
    for (int e = 0; e < 9; ++e) sum = fmaf(wu[e] * wv[e], q[(e / 3) * kPW + e % 3], sum);
    // Sources are magnitudes, so this only turns a NaN (an image whose
    // visibilities hold an infinity) into 0, as the splat's integer sums do.
    const float val = fmaxf(sum * scale, 0.f);
    *out = val;
    vmax = fmaxf(vmax, val);
  }
  return vmax;
}

// pre_map: the images before reprojection as floats [count][N][N], boxes of
// kPW x kChunk.
__global__ void __launch_bounds__(kThreads, 4) k_pull(const __grid_constant__ FipGatherBatch in,
                                                      const __grid_constant__ CUtensorMap pre_map,
                                                      const Plan* __restrict__ plans, int n,
                                                      int tiles, unsigned* err) {
  extern __shared__ char s_raw[];
  __shared__ uint64_t s_bar;
  __shared__ Plan s_plan;
  __shared__ float s_max[kThreads / 32];
  // The copies' destination, 128-byte aligned within the slack.
  float* patch = reinterpret_cast<float*>(s_raw + ((128u - (smem_u32(s_raw) & 127u)) & 127u));
  const Plan* plan = plans + (size_t)blockIdx.y * tiles * tiles + blockIdx.x;
  const int rows = __ldg(&plan->rows);
  if (rows == 0) return;  // uniform: the tile keeps the splat
  if (threadIdx.x == 0) {
    mbar_init(&s_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    const int chunks = (rows + kChunk - 1) / kChunk;
    mbar_expect_tx(&s_bar, (unsigned)(chunks * kChunk * kPW * 4));
    const int a_lo = __ldg(&plan->a_lo), b_lo = __ldg(&plan->b_lo);
    for (int k = 0; k < chunks; ++k)
      tma_load_3d(patch + k * kChunk * kPW, &pre_map, a_lo, b_lo + k * kChunk, (int)blockIdx.y,
                  &s_bar);
  }
  if (threadIdx.x < kPlanWords)
    reinterpret_cast<float*>(&s_plan)[threadIdx.x] =
        __ldg(reinterpret_cast<const float*>(plan) + threadIdx.x);
  __syncthreads();
  const int r0 = (int)(blockIdx.x / tiles) * kDT, c0 = (int)(blockIdx.x % tiles) * kDT;
  const float scale = 1.0f / (float)in.nb[blockIdx.y];
  float* dst = in.dst[blockIdx.y];
  const bool got = mbar_wait(&s_bar, 0);
  if (!__syncthreads_and(got)) {
    // The copy did not arrive within the wait's limit: report the image as
    // unusable rather than hang.
    if (threadIdx.x == 0) {
      if (err) atomicOr(err, 1u);
      mbar_wait(&s_bar, 0);
    }
    return;
  }
  float vmax;
  if (s_plan.flags == kInner)
    vmax = pull_tile<true, false>(s_plan, patch, r0, c0, n, scale, dst);
  else if (s_plan.flags == (kInner | kFine))
    vmax = pull_tile<true, true>(s_plan, patch, r0, c0, n, scale, dst);
  else
    vmax = pull_tile<false, true>(s_plan, patch, r0, c0, n, scale, dst);
  unsigned* img_max = in.img_max[blockIdx.y];
  for (int o = 16; o > 0; o >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
  if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = vmax;
  __syncthreads();
  if (threadIdx.x == 0 && img_max) {
    float b = 0.f;
    for (int w = 0; w < kThreads / 32; ++w) b = fmaxf(b, s_max[w]);
    atomicMax(img_max, __float_as_uint(b));
  }
}

bool encode_pre_map(CUtensorMap* m, const float* pre, int n, int count) {
  const PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
  if (!enc || ((uintptr_t)pre & 15) != 0) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)n, (cuuint64_t)n, (cuuint64_t)count};
  const cuuint64_t strides[2] = {(cuuint64_t)n * 4, (cuuint64_t)n * n * 4};
  const cuuint32_t box[3] = {(cuuint32_t)kPW, (cuuint32_t)kChunk, 1};
  const cuuint32_t es[3] = {1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(pre), dims, strides, box,
             es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
         CUDA_SUCCESS;
}

}  // namespace

size_t fip_pull_plan_words(const FipGeom& geo) {
  const size_t tiles = (geo.n + kDT - 1) / kDT;
  return tiles * tiles * (sizeof(Plan) / 4);
}

bool fip_pull_supported(const FipGeom& geo) {
  return geo.n >= kPullMin && geo.cell <= kPullCell && geo.n % 4 == 0 && tensor_map_encoder();
}

cudaError_t fip_launch_pull_plan(const FipGeom& geo, const FipGatherBatch& in, unsigned* plans,
                                 cudaStream_t s) {
  const int tiles = (geo.n + kDT - 1) / kDT;
  const dim3 blocks((tiles * tiles * kPoly + kThreads - 1) / kThreads, in.count);
  k_pull_plan<<<blocks, kThreads, 0, s>>>(in, geo.n, geo.cell, tiles,
                                          reinterpret_cast<Plan*>(plans));
  return cudaGetLastError();
}

cudaError_t fip_launch_pull(const FipGeom& geo, const FipGatherBatch& in, const float* pre,
                            const unsigned* plans, const unsigned* pre_max, cudaStream_t s,
                            unsigned* err) {
  if (in.count < 1 || in.count > FIP_MAX_BATCH) return cudaErrorInvalidValue;
  CUtensorMap map{};
  if (!encode_pre_map(&map, pre, geo.n, in.count)) return cudaErrorInvalidValue;
  const int tiles = (geo.n + kDT - 1) / kDT;
  const size_t smem = kPatchBytes + 128;
  cudaError_t e =
      cudaFuncSetAttribute(k_pull, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k_pull<<<dim3(tiles * tiles, in.count), kThreads, smem, s>>>(
      in, map, reinterpret_cast<const Plan*>(plans), geo.n, tiles, err);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return fip_launch_reproject_rest(geo, in, pre, plans, pre_max, s, err);
}
