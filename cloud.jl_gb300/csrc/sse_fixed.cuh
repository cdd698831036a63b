// sse_fixed.cuh -- 64-bit block fixed-point arithmetic of the FP64 form.
//
// GB300 issues 2 FP64 FMAs per cycle per SM (1.7 for a separate add or
// multiply), but 64 integer multiply-adds 32 x 32 + 64 -> 64 bits and 64
// 64-bit additions (measured).  The two-point fluxes of one element are sums
// and products of node values of similar size, so they are evaluated on
// integers scaled by powers of two that the element's own extremes choose
// (block fixed point, 60 fraction bits).  A product keeps the three upper of
// its four partial products, i.e. 60 bits below the element's scale, where
// FP64 keeps 53 below the operand; sums are exact, and, being integers, do
// not depend on their order.  Elements whose densities or enthalpies span
// more than 2^4, or are not positive and finite, take the FP64 algebra.
#pragma once

#include "sse_device.cuh"

namespace sse {

// value (hi 2^30 + lo) 2^-60 of its unit; sums of two are formed part by part,
// without a carry
struct Fx {
  int lo, hi;
};

constexpr int kFxLow = 30;
constexpr int kFxMask = (1 << kFxLow) - 1;

SSE_HD long long fx_wide(int a, int b, long long c) { return (long long)a * b + c; }

// sum of products: h counts 2^-60, x counts 2^-90 (the low x low products,
// below 2^-60, are left out)
struct FxDot {
  // cross products first: h continues from x >> 30.  x starts at half of what the
  // shift drops, so that results are rounded to nearest: dropped bits pull every
  // flux the same way, and a mean over the mesh shows it (the drift of the
  // domain integrals was 1.4 times that of the FP64 kernels)
  long long x = 1LL << (kFxLow - 1);
  SSE_HD void cross(Fx a, Fx b) { x = fx_wide(a.hi, b.lo, fx_wide(a.lo, b.hi, x)); }
};

SSE_HD Fx fx_split(long long v) { return Fx{(int)v & kFxMask, (int)(v >> kFxLow)}; }
// the same with lo in [-2^29, 2^29): the form of stored values, which leaves
// room in the low part for sums and corrections
SSE_HD Fx fx_split_near(long long v) {
  return Fx{(int)((unsigned)v << 2) >> 2, (int)((v + (1 << (kFxLow - 1))) >> kFxLow)};
}
SSE_HD long long fx_join(Fx a) { return fx_wide(a.hi, 1 << kFxLow, a.lo); }
SSE_HD Fx fx_add(Fx a, Fx b) { return Fx{a.lo + b.lo, a.hi + b.hi}; }

// a b in 2^-60
SSE_HD long long fx_mul(Fx a, Fx b) {
  FxDot s;
  s.cross(a, b);
  return fx_wide(a.hi, b.hi, s.x >> kFxLow);
}

// sum over n of a[n] b[n] in 2^-60
template <int N>
SSE_HD long long fx_dot(const Fx *a, const Fx *b) {
  FxDot s;
#pragma unroll
  for (int n = 0; n < N; ++n) s.cross(a[n], b[n]);
  long long h = s.x >> kFxLow;
#pragma unroll
  for (int n = 0; n < N; ++n) h = fx_wide(a[n].hi, b[n].hi, h);
  return h;
}

// x 2^(60 - e) for |x| < 2^(e + 3), truncated toward zero in magnitude (exact
// when x's last bit is at least 2^(e - 60)); integer operations only
SSE_HD long long fx_from_double(double x, int e) {
  const long long b = sse_bits(x);
  const int ex = (int)((b >> 52) & 0x7ff);
  if (ex == 0) return 0;  // zero or subnormal
  const unsigned long long m = ((unsigned long long)b & 0x000fffffffffffffULL) | 0x0010000000000000ULL;
  const int sh = ex - 1075 + 60 - e;
  const unsigned long long v = sh >= 0 ? m << (sh < 10 ? sh : 10) : (sh > -64 ? m >> -sh : 0ULL);
  const long long s = b >> 63;
  return ((long long)v ^ s) - s;
}

// 2^e for |e| < 1000
SSE_HD double fx_pow2(int e) { return sse_from_bits((long long)(e + 1023) << 52); }

// exponent e with x < 2^e of a positive normal x, from its upper 32 bits
SSE_HD int fx_exponent(unsigned hi) { return (int)(hi >> 20) - 1022; }

// A node's density and enthalpy rounded to two floats each (48 bits), for
// the small corrections of their means
struct FxPair {
  float rh, rl, hh, hl;
};

SSE_HD void fx_two_floats(Fx v, float *h, float *l) {
  // hi 2^-30 rounded to 24 bits, and what is left with the low part
  const float a = (float)v.hi;
  const float r = (float)(v.hi - (int)a) + (float)v.lo * 0x1p-30f;
  *h = a * 0x1p-30f;
  *l = r * 0x1p-30f;
}

// FP32 operations that must not be contracted or reassociated
SSE_HD float f_add(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fadd_rn(a, b);
#else
  volatile float s = a + b;
  return s;
#endif
}
SSE_HD float f_sub(float a, float b) { return f_add(a, -b); }
SSE_HD float f_mul(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fmul_rn(a, b);
#else
  volatile float s = a * b;
  return s;
#endif
}
SSE_HD float f_fma(float a, float b, float c) {
#ifdef __CUDA_ARCH__
  return __fmaf_rn(a, b, c);
#else
  return std::fmaf(a, b, c);
#endif
}
SSE_HD float f_rcp(float s) {
#ifdef __CUDA_ARCH__
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(s));
  return y;
#else
  return 1.0f / s;
#endif
}
SSE_HD int f_bits(float x) {
#ifdef __CUDA_ARCH__
  return __float_as_int(x);
#else
  int b;
  std::memcpy(&b, &x, 4);
  return b;
#endif
}
SSE_HD int f_rint(float x) {
#ifdef __CUDA_ARCH__
  return __float2int_rn(x);
#else
  return (int)std::nearbyintf(x);
#endif
}

// Means of two positive values as (x + y)(1 - c): twice the logarithmic mean
// L (kind 0, the density) or twice x y / L (kind 1: for the enthalpies h =
// theta/(gamma - 1) of the two states, the inverse logarithmic mean of beta =
// 1/theta over gamma - 1).  With f = (x - y)/(x + y) and z = f^2
//   L       = (x + y)/2 (1 - z/3 - 4 z^2/45 - 44 z^3/945 - ...)
//   x y / L = (x + y)/2 (1 - 2 z/3 - 2 z^2/15 - 2 z^3/35 - ...)
// so below z = 1e-4 the correction (x + y) c = (x - y) f (1/3 + ...) is at
// most 6.7e-5 (x + y), and 2^-40 of it is 2^-54 of the mean: pairs of FP32
// numbers (48 bits) carry it.  corr: the correction in units 2^-30 (hi) and
// 2^-60 (lo); returns z.
template <int KIND>
SSE_HD float fx_mean_correction(float xh, float xl, float yh, float yl, Fx *corr) {
  constexpr float T = (KIND == 0 ? (float)(1.0 / 3.0) : (float)(2.0 / 3.0)) * 0x1p30f;
  constexpr float Tl = (KIND == 0 ? (float)(1.0 / 3.0 - (double)(float)(1.0 / 3.0))
                                  : (float)(2.0 / 3.0 - (double)(float)(2.0 / 3.0))) * 0x1p30f;
  constexpr float K1 = (KIND == 0 ? (float)(4.0 / 45.0) : (float)(2.0 / 15.0)) * 0x1p30f;
  constexpr float K2 = (KIND == 0 ? (float)(44.0 / 945.0) : (float)(2.0 / 35.0)) * 0x1p30f;
  // difference and sum as pairs (the leading difference is exact for values
  // within a factor of two)
  const float dh = f_sub(xh, yh), dl = f_sub(xl, yl);
  const float d0 = f_add(dh, dl), d1 = f_sub(dl, f_sub(d0, dh));
  const float sh = f_add(xh, yh);
  const float sl = f_add(f_add(f_sub(fmaxf(xh, yh), sh), fminf(xh, yh)), f_add(xl, yl));
  // f = d / s: FP32 quotient and one correction
  const float r = f_rcp(sh);
  const float q0 = f_mul(d0, r);
  const float q1 = f_mul(f_add(f_fma(-q0, sh, d0), f_fma(-q0, sl, d1)), r);
  // w = d f; z = f^2 and its rest
  const float w0 = f_mul(d0, q0);
  const float w1 = f_fma(d1, q0, f_fma(d0, q1, f_fma(d0, q0, -w0)));
  const float z = f_mul(q0, q0);
  const float zl = f_fma(f_add(q0, q0), q1, f_fma(q0, q0, -z));
  // corr = w (T + z (K1 + z K2)) in units of 2^-30
  const float t1 = f_fma(zl, K1, f_fma(z, f_fma(z, K2, K1), Tl));
  const float t = f_add(T, t1), tl = f_add(f_sub(T, t), t1);
  const float a0 = f_mul(w0, t);
  const float a1 = f_fma(w1, t, f_fma(w0, tl, f_fma(w0, t, -a0)));
  // hi: nearest integer of a0 (below 2^22); lo: the rest and a1
  const float magic = 12582912.0f;  // 1.5 2^23
  const float m = f_add(a0, magic);
  corr->hi = f_bits(m) - 0x4b400000;
  const float rem = f_sub(a0, f_sub(m, magic));
  corr->lo = f_rint(f_mul(rem, 0x1p30f)) + f_rint(f_mul(a1, 0x1p30f));
  return z;
}

// the same means off the series branch, in FP64 (scaled values): atanh(f)/f by
// its series up to z = 0.02 (the first term left out is below 2^-56), the
// logarithm beyond
SSE_HD double fx_mean_wide(double x, double y, int kind) {
  const double s = x + y;
  const double f = (x - y) * sse_rcp(s);
  const double z = f * f;
  if (z < 0.02) {
    double q = 1.0 / 19.0;
    q = fma(q, z, 1.0 / 17.0);
    q = fma(q, z, 1.0 / 15.0);
    q = fma(q, z, 1.0 / 13.0);
    q = fma(q, z, 1.0 / 11.0);
    q = fma(q, z, 1.0 / 9.0);
    q = fma(q, z, 1.0 / 7.0);
    q = fma(q, z, 1.0 / 5.0);
    q = fma(q, z, 1.0 / 3.0);
    // s (1 - z) q = s - s (z - (1 - z)(q - 1)) with q - 1 = z (...)
    const double qm1 = q * z;
    if (kind == 0) return s - s * (qm1 * sse_rcp(1.0 + qm1));
    return s - s * (z - (1.0 - z) * qm1);
  }
  const double L = (x - y) / log(x / y);
  return kind == 0 ? 2.0 * L : 2.0 * x * y / L;
}

SSE_HD double fx_to_unit_double(Fx a) { return fma((double)a.hi, 0x1p-30, (double)a.lo * 0x1p-60); }

#ifdef __CUDA_ARCH__
static __device__ __noinline__
#else
static inline
#endif
Fx fx_mean_slow(Fx x, Fx y, int kind) {
  const double v = fx_mean_wide(fx_to_unit_double(x), fx_to_unit_double(y), kind);
  return fx_split((long long)(v * 0x1p60));
}

// Node values in an element's units: rho / 2^eR <= 1/2, p / 2^(eR + eH - 2),
// h = p / ((gamma - 1) rho) / 2^eH <= 1/2, |V_m| / 2^eV <= 1/2, kept as
// [rho, p, h, V_1..V_D]; kappa = eH - 2 eV >= 0.
template <int D>
constexpr int kFxNode = 3 + D;
// words (8 bytes) per node of the shared-memory array: odd, so that the nodes
// of a warp's pairs meet distinct banks
template <int D>
constexpr int kFxStride = (3 + D) % 2 ? 3 + D : 4 + D;

// Ranocha's flux contracted with a halved metric vector G (see
// ec_flux_dot_half), in an element's units: with g = sum over the pairs of a
// node of |G|_1 <= 1,
//   out[0]     2^-62 of 2^(eR + eG + eV - 1)    |sum| <= 1
//   out[1 + m] 2^-61 of 2^(eR + eH - 2 + eG)    |sum| <= 1 + 2 (gamma - 1) < 4
//   out[D + 1] 2^-61 of 2^(eR + eH - 2 + eG + eV)
// Every partial sum stays below 2^63 for gamma <= 1.7 (sums of cross products:
// 7.2 2^60 in the energy, the largest).
template <int D>
SSE_HD void fx_ec_flux(const Fx *Pi, const Fx *Pj, const FxPair &fi, const FxPair &fj, const Fx *G, int kappa,
                       long long *out) {
  // (x + y)(1 - c) of density and enthalpy
  Fx cr, ch;
  const float zr = fx_mean_correction<0>(fi.rh, fi.rl, fj.rh, fj.rl, &cr);
  const float zh = fx_mean_correction<1>(fi.hh, fi.hl, fj.hh, fj.hl, &ch);
  Fx rm{Pi[0].lo + Pj[0].lo - cr.lo, Pi[0].hi + Pj[0].hi - cr.hi};
  Fx hm{Pi[2].lo + Pj[2].lo - ch.lo, Pi[2].hi + Pj[2].hi - ch.hi};
  if (!(fmaxf(zr, zh) < 1.0e-4f)) {
    if (!(zr < 1.0e-4f)) rm = fx_mean_slow(Pi[0], Pj[0], 0);
    if (!(zh < 1.0e-4f)) hm = fx_mean_slow(Pi[2], Pj[2], 1);
  }
  Fx vi[D], vj[D], vs[D];
#pragma unroll
  for (int m = 0; m < D; ++m) {
    vi[m] = Pi[3 + m];
    vj[m] = Pj[3 + m];
    vs[m] = fx_add(vi[m], vj[m]);
  }
  const Fx gi = fx_split(fx_dot<D>(G, vi)), gj = fx_split(fx_dot<D>(G, vj));
  const Fx vv = fx_split(fx_dot<D>(vi, vj));
  // f0 = rm (gi + gj)
  const Fx gs = fx_add(gi, gj);
  FxDot c;
  c.cross(rm, gs);
  const long long f0 = fx_wide(rm.hi, gs.hi, c.x >> kFxLow);
  out[0] = ((long long)rm.hi * gs.hi << 2) + ((c.x - (3LL << (kFxLow - 3))) >> (kFxLow - 2));
  const Fx f = fx_split(f0), t = fx_split((f0 + ((1LL << kappa) >> 1)) >> kappa);
  const Fx ps = fx_add(Pi[1], Pj[1]);
#pragma unroll
  for (int m = 0; m < D; ++m) {
    FxDot s{1LL << (kFxLow - 2)};
    s.cross(t, vs[m]);
    s.cross(ps, G[m]);
    out[1 + m] = (fx_wide(t.hi, vs[m].hi, (long long)ps.hi * G[m].hi) << 1) + (s.x >> (kFxLow - 1));
  }
  FxDot s{1LL << (kFxLow - 2)};
  s.cross(f, hm);
  s.cross(t, vv);
  s.cross(Pi[1], gj);
  s.cross(Pj[1], gi);
  out[D + 1] = (fx_wide(f.hi, hm.hi, fx_wide(t.hi, vv.hi, fx_wide(Pi[1].hi, gj.hi, (long long)Pj[1].hi * gi.hi))) << 1) +
               (s.x >> (kFxLow - 1));
}

}  // namespace sse
