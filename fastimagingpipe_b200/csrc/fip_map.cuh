// The exact plane-to-sky map of the reprojections, and the preimage of a
// destination tile under it.  Included by translation units compiled with
// --use_fast_math (the FP32 parts serve bounds whose margins dwarf it).
#pragma once

#include "fip_common.cuh"

constexpr int kDT = 64;  // destination tile side of the reprojections

namespace {

// Exact map: LL = P1 - xi z / cell, MM = P2 + eta z / cell with
// z = 1 - sqrt(1 - rho), rho = cell^2 ((P1 - 1)^2 + (P2 - 1)^2),
// P = M (a, b) / |V22| -- the closed form of coordschange + p2p.
template <typename T>
struct ExactMap {
  T m00, m01, m10, m11;  // M / |V22|
  T i00, i01, i10, i11;  // its inverse
  T xi, eta, cell;
};

template <typename T>
__device__ __forceinline__ ExactMap<T> make_map(const float* V, float cell) {
  ExactMap<T> m;
  const double a22 = fabs((double)V[8]);
  const double m00 = -(double)V[0] / a22, m01 = (double)V[3] / a22;
  const double m10 = -(double)V[1] / a22, m11 = (double)V[4] / a22;
  const double det = m00 * m11 - m01 * m10;
  m.m00 = (T)m00; m.m01 = (T)m01; m.m10 = (T)m10; m.m11 = (T)m11;
  m.i00 = (T)(m11 / det); m.i01 = (T)(-m01 / det);
  m.i10 = (T)(-m10 / det); m.i11 = (T)(m00 / det);
  m.xi = (T)((double)V[6] / (double)V[8]);
  m.eta = (T)((double)V[7] / (double)V[8]);
  m.cell = (T)cell;
  return m;
}

// The same map in FP32 arithmetic throughout (three reciprocals): for the
// gather's candidate bounds, whose margins (a quarter pixel at least) dwarf
// its rounding (~1e-4 pixel at 4096^2).
__device__ __forceinline__ ExactMap<float> make_map_f32(const float* V, float cell) {
  ExactMap<float> m;
  const float ia = 1.0f / fabsf(V[8]), iv = 1.0f / V[8];
  m.m00 = -V[0] * ia;
  m.m01 = V[3] * ia;
  m.m10 = -V[1] * ia;
  m.m11 = V[4] * ia;
  const float idet = 1.0f / (m.m00 * m.m11 - m.m01 * m.m10);
  m.i00 = m.m11 * idet;
  m.i01 = -m.m01 * idet;
  m.i10 = -m.m10 * idet;
  m.i11 = m.m00 * idet;
  m.xi = V[6] * iv;
  m.eta = V[7] * iv;
  m.cell = cell;
  return m;
}

template <typename T>
__device__ __forceinline__ T slant_over_cell(const ExactMap<T>& m, T P1, T P2) {
  const T rho = m.cell * m.cell * ((P1 - 1) * (P1 - 1) + (P2 - 1) * (P2 - 1));
  return rho <= 1 ? (rho / (1 + sqrt(1 - rho))) / m.cell : (T)0;
}

// FP32, for the gather's candidate bounds only: rsqrtf and __fdividef (a few
// ulp), whose rounding the bounds' margins dwarf.
__device__ __forceinline__ float slant_over_cell(const ExactMap<float>& m, float P1, float P2) {
  const float rho = m.cell * m.cell * ((P1 - 1) * (P1 - 1) + (P2 - 1) * (P2 - 1));
  if (!(rho <= 1.f)) return 0.f;
  const float u = 1.f - rho;
  const float s = u > 0.f ? u * rsqrtf(u) : 0.f;
  return __fdividef(rho, m.cell * (1.f + s));
}

template <typename T>
__device__ __forceinline__ void exact_forward(const ExactMap<T>& m, T a, T b, T& LL, T& MM) {
  const T P1 = m.m00 * a + m.m01 * b, P2 = m.m10 * a + m.m11 * b;
  const T zc = slant_over_cell(m, P1, P2);
  LL = P1 - m.xi * zc;
  MM = P2 + m.eta * zc;
}

// Source (a, b), relative to the centre, of an exact target (LL, MM):
// fixed-point iteration on the slant term, a contraction wherever the map
// does not fold (the slant part's Jacobian determinant stays positive); it
// runs until the step is below 1e-3 pixel (or 128 steps).  Returns how far
// the forward map of the result lands from (LL, MM), in pixels.
template <typename T>
__device__ __forceinline__ T exact_inverse(const ExactMap<T>& m, T LL, T MM, T& a, T& b) {
  T P1 = LL, P2 = MM;
  for (int it = 0; it < 128; ++it) {
    const T zc = slant_over_cell(m, P1, P2);
    const T q1 = LL + m.xi * zc, q2 = MM - m.eta * zc;
    const T step = fmax(fabs(q1 - P1), fabs(q2 - P2));
    P1 = q1;
    P2 = q2;
    if (step <= (T)1e-3) break;
  }
  a = m.i00 * P1 + m.i01 * P2;
  b = m.i10 * P1 + m.i11 * P2;
  T L2, M2;
  exact_forward(m, a, b, L2, M2);
  return fmax(fabs(L2 - LL), fabs(M2 - MM));
}

// The preimage of a tile's boundary is sampled at kSeg points per edge: a
// polygon of kPoly vertices, whose chords stay within a small curvature
// margin of the true preimage even for strongly tilted wide fields.
constexpr int kSeg = 2;
constexpr int kPoly = 4 * kSeg;
static_assert(kPoly <= 32 && (kPoly & (kPoly - 1)) == 0, "one warp's lanes, a power of two");

// The preimage of a destination tile's boundary, widened by the splat reach
// and delta, as its polygon's extent, area and curvature margin; ok: the tile
// lies in the gather's domain.
struct TilePreimage {
  float amin, amax, bmin, bmax, sag, area;
  bool ok;
};

// Traced by kPoly consecutive lanes of a warp (every lane of the warp calls
// it): lane k returns vertex k (a, b), the other values are the same in every
// lane of the group.  (r0, c0): the tile's corner, h = N / 2.
__device__ __forceinline__ TilePreimage trace_preimage(const ExactMap<float>& mf, int r0, int c0,
                                                       int h, float delta, float cell, int lane,
                                                       float& a, float& b) {
  const int v = lane % kPoly;
  const float Llo = (float)(c0 - h) - 1.0f - delta, Lhi = (float)(c0 + kDT - h) + delta;
  const float Mlo = (float)(r0 - h) - 1.0f - delta, Mhi = (float)(r0 + kDT - h) + delta;
  // Corners (Llo, Mlo), (Lhi, Mlo), (Lhi, Mhi), (Llo, Mhi); point s of
  // edge e lies s / kSeg of the way from corner e to corner e + 1.
  const int e = v / kSeg, sg = v % kSeg;
  const float Le = (e == 0 || e == 3) ? Llo : Lhi, Me = (e < 2) ? Mlo : Mhi;
  const int e1 = (e + 1) & 3;
  const float Ln = (e1 == 0 || e1 == 3) ? Llo : Lhi, Mn = (e1 < 2) ? Mlo : Mhi;
  const float w = (float)sg * (1.0f / (float)kSeg);
  const float L = Le + (Ln - Le) * w, M = Me + (Mn - Me) * w;
  float res = exact_inverse(mf, L, M, a, b);
  // Sky offset (X, Y) in radians of the source point, held inside the
  // source image (the candidates are, too), and the slant part's Jacobian
  // determinant there: 1 - xi X / n + eta Y / n, n = sqrt(1 - r2).
  const float lim = (float)h + 2.0f;
  const float ac = fminf(fmaxf(a, -lim), lim), bc = fminf(fmaxf(b, -lim), lim);
  const float X = cell * (mf.m00 * ac + mf.m01 * bc - 1.0f);
  const float Y = cell * (mf.m10 * ac + mf.m11 * bc - 1.0f);
  float r2 = X * X + Y * Y;
  const float n1 = sqrtf(fmaxf(1.0f - r2, 1e-6f));
  float det = 1.0f - mf.xi * X / n1 + mf.eta * Y / n1;
  // Extent and shoelace area of the polygon, reduced over its lanes.
  float amn = a, amx = a, bmn = b, bmx = b;
  const int nxt = lane - v + (v + 1) % kPoly;
  const float an = __shfl_sync(0xffffffffu, a, nxt), bn = __shfl_sync(0xffffffffu, b, nxt);
  float area = a * bn - an * b;
#pragma unroll
  for (int o = 1; o < kPoly; o <<= 1) {
    res = fmaxf(res, __shfl_xor_sync(0xffffffffu, res, o));
    r2 = fmaxf(r2, __shfl_xor_sync(0xffffffffu, r2, o));
    det = fminf(det, __shfl_xor_sync(0xffffffffu, det, o));
    amn = fminf(amn, __shfl_xor_sync(0xffffffffu, amn, o));
    amx = fmaxf(amx, __shfl_xor_sync(0xffffffffu, amx, o));
    bmn = fminf(bmn, __shfl_xor_sync(0xffffffffu, bmn, o));
    bmx = fmaxf(bmx, __shfl_xor_sync(0xffffffffu, bmx, o));
    area += __shfl_xor_sync(0xffffffffu, area, o);
  }
  TilePreimage p;
  p.amin = amn;
  p.amax = amx;
  p.bmin = bmn;
  p.bmax = bmx;
  p.area = fabsf(0.5f * area);
  // The candidate bounds hold while the inverse converged, the tile lies
  // well inside the horizon (r2 < 0.98) and the map does not fold
  // (det > 1/4).
  p.ok = res < 0.05f && r2 < 0.98f && det > 0.25f;
  // The preimage's edges bow away from the chords between its points
  // by at most ell^2 / 8 times the slant term's second derivative
  // (|(xi, eta)| cell / n^3, divided by det for the inverse), ell the
  // length of one segment: widen the candidate intervals by that (with a
  // 20 % allowance).
  const float nn = sqrtf(fmaxf(1.0f - r2, 0.02f));
  const float ell = ((float)kDT + 2.0f + 2.0f * delta) * (1.0f / (float)kSeg);
  p.sag = 0.15f * hypotf(mf.xi, mf.eta) * cell * ell * ell /
          (nn * nn * nn * fmaxf(det, 0.25f));
  return p;
}

}  // namespace
