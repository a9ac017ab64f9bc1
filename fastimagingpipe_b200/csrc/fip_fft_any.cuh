// Shared-memory FFT for lengths G = 3 M with any even M (the grid sides of
// images whose side is a multiple of four but not a power of two), beside the
// power-of-two transform of fip_fft.cuh and with its conventions: exponent +i,
// inputs z[c] on a band lo <= c <= hi around 0, decimation in frequency by 3
// into three length-M transforms Y_s, the 2 M outputs X[p], -M <= p < M.
//
// The length is a run-time value: Stockham passes between two shared-memory
// buffers, one radix a pass, each thread taking whole butterflies (all in
// registers) in turn.  Radices up to 16 have compile-time codelets built from
// 2, 3, 4, 5 and 7; a larger prime factor p takes a pass of its own in two
// steps, the sums and differences of its inputs' conjugate pairs and then
// (p - 1)^2 / 4 products per output pair, p multiply-adds an element.  The pass
// twiddles of butterfly j, W_M^{step k}, are products of table entries at the
// powers of two of k (a few ulps).
#pragma once

#include "fip_fft.cuh"

namespace fipfft {

// Compile-time cosine and sine of 2 pi k / r (Taylor series after reduction to
// an eighth of a turn).
constexpr double kPi = 3.14159265358979323846;
constexpr double taylor_cos(double x) {
  double t = 1, s = 1;
  for (int n = 1; n < 14; ++n) {
    t *= -x * x / ((2 * n - 1) * (2 * n));
    s += t;
  }
  return s;
}
constexpr double taylor_sin(double x) {
  double t = x, s = x;
  for (int n = 1; n < 14; ++n) {
    t *= -x * x / ((2 * n) * (2 * n + 1));
    s += t;
  }
  return s;
}
// The angle 2 pi k / r for 0 <= k < r, by octants.
constexpr double turn_cos(int k, int r) {
  k %= r;
  if (2 * k > r) k = r - k;                                   // [0, r/2]
  if (4 * k > r) return -turn_cos(r - 2 * k, 2 * r);          // pi - x
  if (8 * k > r) return taylor_sin(kPi / 2 - 2 * kPi * k / r);
  return taylor_cos(2 * kPi * k / r);
}
constexpr double turn_sin(int k, int r) {
  k %= r;
  if (2 * k > r) return -turn_sin(r - k, r);
  if (4 * k > r) return turn_sin(r - 2 * k, 2 * r);
  if (8 * k > r) return taylor_cos(kPi / 2 - 2 * kPi * k / r);
  return taylor_sin(2 * kPi * k / r);
}

// cos and sin of 2 pi k / R, k < R, evaluated by the compiler.
template <int R>
struct Turns {
  float c[R], s[R];
  constexpr Turns() : c(), s() {
    for (int k = 0; k < R; ++k) {
      c[k] = (float)turn_cos(k, R);
      s[k] = (float)turn_sin(k, R);
    }
  }
};

// DFT of odd prime length R (exponent +i) by conjugate pairs.
template <int R>
__device__ __forceinline__ void dft_pairs(float2* x) {
  constexpr int H = (R - 1) / 2;
  constexpr Turns<R> w;
  float2 a[H], b[H];
#pragma unroll
  for (int k = 0; k < H; ++k) {
    a[k] = cadd(x[k + 1], x[R - 1 - k]);
    b[k] = csub(x[k + 1], x[R - 1 - k]);
  }
  const float2 x0 = x[0];
  float2 sum = x0;
#pragma unroll
  for (int k = 0; k < H; ++k) sum = cadd(sum, a[k]);
  x[0] = sum;
#pragma unroll
  for (int m = 1; m <= H; ++m) {
    float2 u = x0, v = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < H; ++k) {
      const float c = w.c[((k + 1) * m) % R], s = w.s[((k + 1) * m) % R];
      u.x += c * a[k].x;
      u.y += c * a[k].y;
      v.x += s * b[k].x;
      v.y += s * b[k].y;
    }
    x[m] = make_float2(u.x - v.y, u.y + v.x);      // u + i v
    x[R - m] = make_float2(u.x + v.y, u.y - v.x);  // u - i v
  }
}
template <>
__device__ __forceinline__ void dft<3>(float2* x) { dft_pairs<3>(x); }
template <>
__device__ __forceinline__ void dft<5>(float2* x) { dft_pairs<5>(x); }
template <>
__device__ __forceinline__ void dft<7>(float2* x) { dft_pairs<7>(x); }

// R = P Q: n = n1 + P n2, k = k2 + Q k1.
template <int P, int Q>
__device__ __forceinline__ void dft_split(float2* x) {
  constexpr int R = P * Q;
  constexpr Turns<R> w;
  float2 a[R];
#pragma unroll
  for (int n1 = 0; n1 < P; ++n1) {
    float2 t[Q];
#pragma unroll
    for (int n2 = 0; n2 < Q; ++n2) t[n2] = x[n1 + P * n2];
    dft<Q>(t);
#pragma unroll
    for (int k2 = 0; k2 < Q; ++k2)
      a[n1 * Q + k2] =
          n1 * k2 == 0 ? t[k2] : cmul(t[k2], make_float2(w.c[n1 * k2], w.s[n1 * k2]));
  }
#pragma unroll
  for (int k2 = 0; k2 < Q; ++k2) {
    float2 t[P];
#pragma unroll
    for (int n1 = 0; n1 < P; ++n1) t[n1] = a[n1 * Q + k2];
    dft<P>(t);
#pragma unroll
    for (int k1 = 0; k1 < P; ++k1) x[k2 + Q * k1] = t[k1];
  }
}
template <>
__device__ __forceinline__ void dft<6>(float2* x) { dft_split<2, 3>(x); }
template <>
__device__ __forceinline__ void dft<9>(float2* x) { dft_split<3, 3>(x); }
template <>
__device__ __forceinline__ void dft<10>(float2* x) { dft_split<2, 5>(x); }
template <>
__device__ __forceinline__ void dft<12>(float2* x) { dft_split<3, 4>(x); }
template <>
__device__ __forceinline__ void dft<15>(float2* x) { dft_split<3, 5>(x); }

// Distance between the sub-transforms' buffers (a few elements apart modulo
// the banks, so that outputs interleaved by 3 spread over them).
__host__ __device__ __forceinline__ int any_stride(int m) { return m + 3; }
// Shared memory: two buffers, then the roots of unity of a first radix above 16.
__host__ __device__ __forceinline__ int any_roots(int m) { return 6 * any_stride(m); }
__host__ __device__ __forceinline__ int any_smem_elems(const Plan& p) {
  return any_roots(p.m) + (p.radix[0] > 16 ? p.radix[0] : 0);
}
// Fills the roots (before a barrier).
__device__ __forceinline__ void any_load_roots(float2* sm, const Plan& p,
                                               const float2* __restrict__ tw) {
  if (p.radix[0] > 16)
    for (int k = threadIdx.x; k < p.radix[0]; k += blockDim.x)
      sm[any_roots(p.m) + k] = __ldg(&tw[k * (p.g / p.radix[0])]);
}

// Exact i / d for 0 <= i < 2^20, inv = 1 / d.
__device__ __forceinline__ int fdiv(int i, float inv) { return (int)(((float)i + 0.5f) * inv); }

// One pass of radix R over the three sub-transforms: src -> dst (base of the
// first sub-transform, any_stride apart), ns outputs of the previous passes.
template <int R>
__device__ __forceinline__ void any_pass(const float2* src, float2* dst, int m, int ns, int g,
                                         const float2* __restrict__ tw) {
  const int per = m / R, total = 3 * per, stride = any_stride(m);
  const float iper = 1.0f / (float)per, ins = 1.0f / (float)ns;
  const int tstep = 3 * (m / (ns * R));  // of W_G
  for (int b = threadIdx.x; b < total; b += blockDim.x) {
    const int s = fdiv(b, iper), j = b - s * per;
    const float2* in = src + s * stride + j;
    float2 x[R];
#pragma unroll
    for (int k = 0; k < R; ++k) x[k] = in[k * per];
    int q = j, lo = 0;
    if (ns > 1) {
      q = fdiv(j, ins);
      lo = j - q * ns;
      const int step = lo * tstep;
      float2 w[R];
#pragma unroll
      for (int k = 1; k < R; k <<= 1) w[k] = __ldg(&tw[step * k]);
#pragma unroll
      for (int k = 3; k < R; ++k) {
        const int top = k >= 8 ? 8 : (k >= 4 ? 4 : 2);
        if (k != top) w[k] = cmul(w[k - top], w[top]);
      }
#pragma unroll
      for (int k = 1; k < R; ++k) x[k] = cmul(x[k], w[k]);
    }
    dft<R>(x);
    float2* out = dst + s * stride + q * ns * R + lo;
#pragma unroll
    for (int k = 0; k < R; ++k) out[k * ns] = x[k];
  }
  __syncthreads();
  (void)g;
}

// One pass of odd prime radix p: the inputs' pair sums and differences in
// place, then the outputs (pairs m, p - m).
constexpr int kPrimeOut = 4;
template <bool SHARED>
__device__ __forceinline__ void any_pass_prime(float2* src, float2* dst, int m, int p, int ns,
                                               int g, const float2* __restrict__ tw,
                                               const float2* roots) {
  const int per = m / p, stride = any_stride(m), hp = (p - 1) / 2;
  const float iper = 1.0f / (float)per, ins = 1.0f / (float)ns;
  const int tstep = 3 * (m / (ns * p));
  for (int b = threadIdx.x; b < 3 * per * hp; b += blockDim.x) {
    const int r = fdiv(b, iper), j = b - r * per;  // r = s * hp + (k - 1)
    const int s = r >= 2 * hp ? 2 : (r >= hp ? 1 : 0), k = r - s * hp + 1;
    float2* u = src + s * stride + j + k * per;
    float2* v = src + s * stride + j + (p - k) * per;
    float2 x = *u, y = *v;
    if (ns > 1) {
      const int step = (j - fdiv(j, ins) * ns) * tstep;
      x = cmul(x, __ldg(&tw[step * k]));
      y = cmul(y, __ldg(&tw[step * (p - k)]));
    }
    *u = cadd(x, y);
    *v = csub(x, y);
  }
  __syncthreads();
  // kPrimeOut pairs of outputs per item, so that an input pair is read once for
  // them; the roots of unity come from the shared table of the plan's first
  // radix, or the global one.
  const int wstep = g / p, groups = (hp + kPrimeOut) / kPrimeOut;  // pairs 0 .. hp
  for (int b = threadIdx.x; b < 3 * per * groups; b += blockDim.x) {
    const int r = fdiv(b, iper), j = b - r * per;  // r = s * groups + group
    const int s = r >= 2 * groups ? 2 : (r >= groups ? 1 : 0), m0 = r - s * groups;
    const float2* in = src + s * stride + j;
    float2 u[kPrimeOut], v[kPrimeOut];
    int e[kPrimeOut], mm[kPrimeOut];  // e: k mm mod p
#pragma unroll
    for (int o = 0; o < kPrimeOut; ++o) {
      mm[o] = min(m0 + o * groups, hp);  // the last item may repeat pair hp
      u[o] = in[0];
      v[o] = make_float2(0.f, 0.f);
      e[o] = 0;
    }
    const float2* pa = in;
    const float2* pd = in + (p - 1) * per;
    for (int k = 1; k <= hp; ++k, pd -= per) {
      pa += per;
      const float2 a = *pa, d = *pd;
#pragma unroll
      for (int o = 0; o < kPrimeOut; ++o) {
        e[o] += mm[o];
        if (e[o] >= p) e[o] -= p;
        const float2 w = SHARED ? roots[e[o]] : __ldg(&tw[e[o] * wstep]);
        u[o].x = fmaf(w.x, a.x, u[o].x);
        u[o].y = fmaf(w.x, a.y, u[o].y);
        v[o].x = fmaf(w.y, d.x, v[o].x);
        v[o].y = fmaf(w.y, d.y, v[o].y);
      }
    }
    const int q = ns > 1 ? fdiv(j, ins) : j;
    float2* out = dst + s * stride + q * ns * p + (ns > 1 ? j - q * ns : 0);
#pragma unroll
    for (int o = 0; o < kPrimeOut; ++o) {
      out[mm[o] * ns] = make_float2(u[o].x - v[o].y, u[o].y + v[o].x);
      if (mm[o] > 0) out[(p - mm[o]) * ns] = make_float2(u[o].x + v[o].y, u[o].y - v[o].x);
    }
  }
  __syncthreads();
}

// The passes of plan p over the staged inputs (second buffer, written before a
// barrier) -> the buffer that holds Y_s in natural order.
__device__ __forceinline__ const float2* any_run(float2* sm, const Plan& p,
                                                 const float2* __restrict__ tw) {
  float2* src = sm + 3 * any_stride(p.m);
  float2* dst = sm;
  int ns = 1;
  for (int k = 0; k < p.passes; ++k) {
    const int r = p.radix[k];
    switch (r) {
      case 2: any_pass<2>(src, dst, p.m, ns, p.g, tw); break;
      case 3: any_pass<3>(src, dst, p.m, ns, p.g, tw); break;
      case 4: any_pass<4>(src, dst, p.m, ns, p.g, tw); break;
      case 5: any_pass<5>(src, dst, p.m, ns, p.g, tw); break;
      case 6: any_pass<6>(src, dst, p.m, ns, p.g, tw); break;
      case 7: any_pass<7>(src, dst, p.m, ns, p.g, tw); break;
      case 8: any_pass<8>(src, dst, p.m, ns, p.g, tw); break;
      case 9: any_pass<9>(src, dst, p.m, ns, p.g, tw); break;
      case 10: any_pass<10>(src, dst, p.m, ns, p.g, tw); break;
      case 12: any_pass<12>(src, dst, p.m, ns, p.g, tw); break;
      case 15: any_pass<15>(src, dst, p.m, ns, p.g, tw); break;
      case 16: any_pass<16>(src, dst, p.m, ns, p.g, tw); break;
      default:
        if (k == 0 && r > 16)
          any_pass_prime<true>(src, dst, p.m, r, ns, p.g, tw, sm + any_roots(p.m));
        else
          any_pass_prime<false>(src, dst, p.m, r, ns, p.g, tw, nullptr);
        break;
    }
    ns *= r;
    float2* t = src;
    src = dst;
    dst = t;
  }
  return src;
}

// Stages z (zero outside lo .. hi, at most G wide) folded and pre-twiddled:
// y_s[n] = sum over c = n + t M of z[c] w^{c s}; load(c) returns z[c].
template <class Load>
__device__ __forceinline__ void any_stage(float2* sm, const Plan& p, int lo, int hi,
                                          const float2* __restrict__ tw, Load&& load) {
  float2* st = sm + 3 * any_stride(p.m);
  const int stride = any_stride(p.m);
  const float h3 = 0.86602540378443864676f;  // sqrt(3) / 2
  const bool wide = hi >= p.m || lo < -p.m;
  for (int n = threadIdx.x; n < p.m; n += blockDim.x) {
    float2 y0 = make_float2(0.f, 0.f), y1 = y0, y2 = y0;
    // w^n and w^{2 n}; c = n + t M turns them by e^{2 pi i t s / 3}.
    const float2 w1 = __ldg(&tw[n]), w2 = __ldg(&tw[2 * n]);
    const float2 r1 = make_float2(-0.5f, h3), r2 = make_float2(-0.5f, -h3);
    for (int t = wide ? -2 : -1; t <= (wide ? 1 : 0); ++t) {
      const int c = n + t * p.m;
      if (c < lo || c > hi) continue;
      const float2 z = load(c);
      y0 = cadd(y0, z);
      float2 a = cmul(z, w1), b = cmul(z, w2);
      if (t == -1 || t == -2 || t == 1) {  // e^{2 pi i t / 3}: t = 1, -2 -> r1; t = -1 -> r2
        a = cmul(a, t == -1 ? r2 : r1);
        b = cmul(b, t == -1 ? r1 : r2);
      }
      y1 = cadd(y1, a);
      y2 = cadd(y2, b);
    }
    st[n] = y0;
    st[stride + n] = y1;
    st[2 * stride + n] = y2;
  }
}

// Output o in [0, 2 M): X[o - M] from the result buffer.
__device__ __forceinline__ float2 any_fetch(const float2* y, int m, int o) {
  int pp = o - m;
  if (pp < 0) pp += 3 * m;
  const int q = pp / 3, s = pp - 3 * q;
  return y[s * any_stride(m) + q];
}

}  // namespace fipfft
