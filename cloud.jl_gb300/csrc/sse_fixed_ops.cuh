// sse_fixed_ops.cuh -- team-parallel operator applications in block fixed
// point (sse_fixed.cuh), the counterparts of sse_ops.cuh for the FP64 form.
//
// A product with an operator entry is three integer multiply-adds, a tenth of
// one FP64 FMA's issue time, so the contractions of an element leave the FP64
// pipe altogether.
//
// Values here have 62 fraction bits, hi 2^31 + lo with lo in [-2^30, 2^30).
// The entries of V's factors are scaled to at most 1/4 per mode vector (the
// headroom that the sums of up to 8 cross products need; products are moved up
// by 2 bits again) and per node: row i of V is taken times 2^K_i, K_i <= 0, about
// the square root of the node's quadrature weight, because the orthonormal
// basis grows like its inverse toward the collapsed vertex; without it the
// modes' scales 2^T_l would cost the leading modes 5 to 8 bits.  With modal
// values in a unit that bounds sum_l 2^T_l |x_l| no partial sum of the sum
// factorisation exceeds the unit, and the unit is that tight for the values at
// hand.
#pragma once

#include <cmath>

#include "sse_kernels.cuh"

namespace sse {

// v 2^-s to the nearest integer, 0 <= s < 63
struct FxShift {
  int s;
  long long half;
  __device__ __forceinline__ explicit FxShift(int s_) : s(s_), half((1LL << s_) >> 1) {}
  __device__ __forceinline__ long long operator()(long long v) const { return (v + half) >> s; }
};

// v 2^e to the nearest double, |e| <= 900, by integer operations (two FP64 FMAs
// would take the place of a hundred of them)
__device__ __forceinline__ double fx_to_double(long long v, int e) {
  const long long s = v >> 63;
  const unsigned long long a = (unsigned long long)((v ^ s) - s);
  const int z = __clzll((long long)a);
  const unsigned long long m = a << z;  // [2^63, 2^64), and v 2^e = m 2^(e - z)
  const unsigned long long b = ((unsigned long long)(1085 + e - z) << 52) + (m >> 11) + ((m >> 10) & 1);
  return a == 0 ? 0.0 : __longlong_as_double((long long)(b | ((unsigned long long)s & 0x8000000000000000ULL)));
}

constexpr int kFoLow = 31;       // bits of the low part
constexpr int kFoUp = 2;         // operator entries are at most 2^-2
__host__ __device__ __forceinline__ Fx fo_split(long long v) {
  return Fx{(int)((unsigned)v << 1) >> 1, (int)((v + (1LL << (kFoLow - 1))) >> kFoLow)};
}
__device__ __forceinline__ long long fo_join(Fx a) { return ((long long)a.hi << kFoLow) + a.lo; }
// x 2^(62 - e)
__host__ __device__ __forceinline__ Fx fo_from_double(double x, int e) { return fo_split(fx_from_double(x, e - 2)); }
// Exponent e of an operator row with absolute sum `row` (positive and finite):
// its entries stay below (1 - 2^-20) 2^e.  An entry of (1 - 2^-32) 2^e or more
// would round to a high part of 2^31, beyond an int.
inline int fo_row_exponent(double row) { return std::ilogb(row * (1.0 + 1e-6)) + 1; }

// NC sums of products with one operator entry each
template <int NC>
struct FxSums {
  long long h[NC], x[NC];
  __device__ __forceinline__ FxSums() {
#pragma unroll
    for (int e = 0; e < NC; ++e) { h[e] = 0; x[e] = 0; }
  }
  // += a v[e stride]
  __device__ __forceinline__ void add(Fx a, const Fx *v, int stride) {
#pragma unroll
    for (int e = 0; e < NC; ++e) {
      const Fx b = v[e * stride];
      x[e] = fx_wide(a.hi, b.lo, fx_wide(a.lo, b.hi, x[e]));
      h[e] = fx_wide(a.hi, b.hi, h[e]);
    }
  }
  // what the cross products have above 2^-62, moved to the others
  __device__ __forceinline__ void fold() {
#pragma unroll
    for (int e = 0; e < NC; ++e) {
      h[e] += x[e] >> kFoLow;
      x[e] &= (1LL << kFoLow) - 1;
    }
  }
  // the sum, up by UP bits, rounded to nearest (FxDot)
  template <int UP>
  __device__ __forceinline__ long long value(int e) const {
    return (long long)((unsigned long long)h[e] << UP) + ((x[e] + (1LL << (kFoLow - UP - 1))) >> (kFoLow - UP));
  }
  template <int UP>
  __device__ __forceinline__ void store(Fx *v, int stride) const {
#pragma unroll
    for (int e = 0; e < NC; ++e) v[e * stride] = fo_split(value<UP>(e));
  }
};

// Sizes of an element with P1 nodes a direction (and, with a modal tensor-
// product V, P1 modes): constants of the compiled kernel, so that loops unroll
// and addresses are offsets; P1 = 0 takes them from the operators.
template <int D, int P1>
struct FxSize {
  static __device__ __forceinline__ int nq(const DevOps &op) { return P1 ? (D == 2 ? P1 * P1 : P1 * P1 * P1) : op.nq; }
  static __device__ __forceinline__ int npf(const DevOps &op) { return P1 ? (D == 2 ? P1 : P1 * P1) : op.npf; }
  static __device__ __forceinline__ int nfac(const DevOps &op) { return P1 ? D + 1 : op.nfac; }
  static __device__ __forceinline__ int nf(const DevOps &op) { return P1 ? nfac(op) * npf(op) : op.nf; }
  static __device__ __forceinline__ int p1(const DevOps &op) { return P1 ? P1 : op.p1; }
  static __device__ __forceinline__ int M1(const DevOps &op) { return P1 ? P1 : op.M1; }
  static __device__ __forceinline__ int M2(const DevOps &op) { return P1 ? P1 : op.M2; }
  static __device__ __forceinline__ int M3(const DevOps &op) { return P1 ? P1 : op.M3; }
  static __device__ __forceinline__ int nb12(const DevOps &op) { return P1 ? P1 * (P1 + 1) / 2 : op.nb12; }
  // s / n for 0 <= s < 2^21
  static __device__ __forceinline__ int div(int s, int n) { return P1 ? s / n : qdiv(s, qrcp(n)); }
  static __device__ __forceinline__ int np(const DevOps &op) {
    return P1 ? (D == 2 ? P1 * (P1 + 1) / 2 : P1 * (P1 + 1) * (P1 + 2) / 6) : op.np;
  }
};

// sum over k < n of entry(k) times the vectors at v + k step: P1 steps unrolled
// where it is given (n <= P1), so that their loads are in flight together
template <int NC, int P1, typename Entry>
__device__ __forceinline__ FxSums<NC> fx_line(int n, Entry entry, const Fx *v, int step, int stride) {
  FxSums<NC> acc;
  if constexpr (P1 > 0) {
#pragma unroll
    for (int k = 0; k < P1; ++k)
      if (k < n) acc.add(entry(k), v + k * step, stride);
  } else {
    for (int k = 0; k < n; ++k) acc.add(entry(k), v + k * step, stride);
  }
  return acc;
}

// y (NC x nq, times 2^K_i) = V x (NC x np, times 2^T_l).  Modal vectors are in
// the order of the sum factorisation (FxTables::order), the modes of one (b1)
// or (b1, b2) contiguous from FxTables::base.
template <int D, int NC, int P1>
__device__ void fx_vdm_mul(const DevOps &op, const FxTables &fx, const Fx *x, Fx *y, Fx *Z, Fx *W, int lane, int tpe) {
  using N = FxSize<D, P1>;
  const int np = N::np(op), nq = N::nq(op), p1 = N::p1(op), M1 = N::M1(op), M2 = N::M2(op);
  if constexpr (D == 2) {
    for (int s = lane; s < p1 * M2; s += tpe) {
      const int b1 = N::div(s, M2), a2 = s - b1 * M2;
      fx_line<NC, P1>(p1 - b1, [&](int k) { return fx.B[a2 + M2 * (b1 + p1 * k)]; }, x + fx.base[b1], 1, np)
          .template store<kFoUp>(Z + s, p1 * M2);
    }
    __syncthreads();
    for (int s = lane; s < M1 * M2; s += tpe) {
      const int a1 = N::div(s, M2), a2 = s - a1 * M2;
      fx_line<NC, P1>(p1, [&](int k) { return fx.A[a1 + M1 * k]; }, Z + a2, M2, p1 * M2).template store<kFoUp>(y + s, nq);
    }
    __syncthreads();
  } else {
    const int M3 = N::M3(op), nb12 = N::nb12(op);
    for (int s = lane; s < nb12 * M3; s += tpe) {
      const int q = N::div(s, M3), a3 = s - q * M3;
      const int b1 = op.b12[q] & 0xff, b2 = op.b12[q] >> 8;
      fx_line<NC, P1>(p1 - b1 - b2, [&](int k) { return fx.C[a3 + M3 * (b1 + p1 * (b2 + p1 * k))]; }, x + fx.base[q], 1, np)
          .template store<kFoUp>(Z + s, nb12 * M3);
    }
    __syncthreads();
    for (int s = lane; s < p1 * M2 * M3; s += tpe) {
      const int r = N::div(s, M3), a3 = s - r * M3, b1 = N::div(r, M2), a2 = r - b1 * M2;
      // the (b1, b2) are listed by b1
      fx_line<NC, P1>(p1 - b1, [&](int k) { return fx.B[a2 + M2 * (b1 + p1 * k)]; }, Z + op.b12_index[b1] * M3 + a3, M3,
                      nb12 * M3)
          .template store<kFoUp>(W + s, p1 * M2 * M3);
    }
    __syncthreads();
    for (int s = lane; s < M1 * M2 * M3; s += tpe) {
      const int r = N::div(s, M3), a3 = s - r * M3, a1 = N::div(r, M2), a2 = r - a1 * M2;
      fx_line<NC, P1>(p1, [&](int k) { return fx.A[a1 + M1 * k]; }, W + a2 * M3 + a3, M2 * M3, p1 * M2 * M3)
          .template store<kFoUp>(y + s, nq);
    }
    __syncthreads();
  }
}

// x (NC x np, without the factors 2^T_l) = V^T y (NC x nq, times 2^-K_i)
template <int D, int NC, int P1>
__device__ void fx_vdm_tmul(const DevOps &op, const FxTables &fx, const Fx *y, Fx *x, Fx *Z, Fx *W, int lane, int tpe) {
  using N = FxSize<D, P1>;
  const int np = N::np(op), nq = N::nq(op), p1 = N::p1(op), M1 = N::M1(op), M2 = N::M2(op);
  if constexpr (D == 2) {
    for (int s = lane; s < p1 * M2; s += tpe) {
      const int b1 = N::div(s, M2), a2 = s - b1 * M2;
      fx_line<NC, P1>(M1, [&](int k) { return fx.A[k + M1 * b1]; }, y + a2, M2, nq).template store<kFoUp>(Z + s, p1 * M2);
    }
    __syncthreads();
    for (int l = lane; l < np; l += tpe) {
      const int m = fx.modes[l], b1 = m & 0xff, b2 = (m >> 8) & 0xff;
      fx_line<NC, P1>(M2, [&](int k) { return fx.B[k + M2 * (b1 + p1 * b2)]; }, Z + b1 * M2, 1, p1 * M2)
          .template store<kFoUp>(x + l, np);
    }
    __syncthreads();
  } else {
    const int M3 = N::M3(op), nb12 = N::nb12(op);
    for (int s = lane; s < p1 * M2 * M3; s += tpe) {
      const int r = N::div(s, M3), a3 = s - r * M3, b1 = N::div(r, M2), a2 = r - b1 * M2;
      fx_line<NC, P1>(M1, [&](int k) { return fx.A[k + M1 * b1]; }, y + a2 * M3 + a3, M2 * M3, nq)
          .template store<kFoUp>(W + s, p1 * M2 * M3);
    }
    __syncthreads();
    for (int s = lane; s < nb12 * M3; s += tpe) {
      const int q = N::div(s, M3), a3 = s - q * M3;
      const int b1 = op.b12[q] & 0xff, b2 = op.b12[q] >> 8;
      fx_line<NC, P1>(M2, [&](int k) { return fx.B[k + M2 * (b1 + p1 * b2)]; }, W + b1 * M2 * M3 + a3, M3, p1 * M2 * M3)
          .template store<kFoUp>(Z + s, nb12 * M3);
    }
    __syncthreads();
    for (int l = lane; l < np; l += tpe) {
      const int m = fx.modes[l], b1 = m & 0xff, b2 = (m >> 8) & 0xff, b3 = (m >> 16) & 0xff;
      fx_line<NC, P1>(M3, [&](int k) { return fx.C[k + M3 * (b1 + p1 * (b2 + p1 * b3))]; }, Z + op.b12_index[b1 + p1 * b2] * M3,
                      1, nb12 * M3)
          .template store<kFoUp>(x + l, np);
    }
    __syncthreads();
  }
}

// entry (e, a) of A x (NC x np) for the element's mass operator A (column-major,
// the absolute sums of its rows at most 1)
template <int MAXU>
__device__ __forceinline__ long long fx_mass_row(const Fx *A, const Fx *xe, int np, int a) {
  FxSums<1> acc;
#pragma unroll MAXU
  for (int b = 0; b < np; ++b) acc.add(A[b * np + a], xe + b, 0);
  return acc.template value<0>(0);
}

// *m = max(*m, v) over the team (m in shared memory)
__device__ __forceinline__ void fx_team_max(unsigned *m, unsigned v, int lane, int tpe) {
  if (tpe >= 32) {
    v = __reduce_max_sync(0xffffffffu, v);
    if ((lane & 31) == 0) atomicMax(m, v);
  } else {
    for (int o = tpe >> 1; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (lane == 0) atomicMax(m, v);
  }
}

// fetch the lines of `bytes` bytes at p into L2
__device__ __forceinline__ void fx_prefetch(const void *p, size_t bytes, int lane, int tpe) {
  const char *c = static_cast<const char *>(p);
  for (size_t o = (size_t)lane * 128; o < bytes; o += (size_t)tpe * 128)
    asm volatile("prefetch.global.L2 [%0];" ::"l"(c + o));
}

// Unit exponents of the NC vectors of modal values: unit[e] with
// sum_l 2^T_l |x_l| < 2^unit[e]; each group of `width` lanes takes whole
// components.  kFxBad: not finite (or beyond 2^900).
constexpr int kFxBad = 100000;

// x in FP64; place l is taken from order[l] (null: l), without factors where T is
// null
template <int NC>
__device__ __forceinline__ void fx_modal_units(const double *x, const signed char *T, const int *order, int np, int *unit, int lane,
                                               int tpe) {
  const int width = tpe < 32 ? tpe : 32, groups = tpe / width, g = lane / width, w = lane - g * width;
  for (int e0 = 0; e0 < NC; e0 += groups) {
    const int e = e0 + g;
    int m = -2000;
    if (e < NC)
      for (int l = w; l < np; l += width) {
        const int ex = (__double2hiint(x[e * np + (order ? order[l] : l)]) >> 20) & 0x7ff;
        if (ex > 0) m = max(m, ex == 0x7ff ? kFxBad : ex - 1023 + (T ? T[l] : 0));
      }
    for (int o = width >> 1; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    float s = 0.f;
    if (e < NC)
      for (int l = w; l < np; l += width) {
        const double v = x[e * np + (order ? order[l] : l)];
        const int ex = (__double2hiint(v) >> 20) & 0x7ff, d = m - (ex - 1023 + (T ? T[l] : 0));
        // the mantissa, rounded up, times 2^-d
        const float f = __int_as_float(0x3f800000 + ((__double2hiint(v) & 0xfffff) << 3) + 8);
        if (ex > 0 && d < 100) s += f * __int_as_float((127 - d) << 23);
      }
    for (int o = width >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (e < NC && w == 0)
      unit[e] = m > 900 ? kFxBad : max(-800, m + (__float_as_int(s * 1.0001f) >> 23) - 126);
  }
}

// x in fixed point, unit 2^0, times 2^T_l where scaled
template <int NC>
__device__ __forceinline__ void fx_modal_units(const Fx *x, const signed char *T, int np, int *unit, int lane, int tpe) {
  const int width = tpe < 32 ? tpe : 32, groups = tpe / width, g = lane / width, w = lane - g * width;
  for (int e0 = 0; e0 < NC; e0 += groups) {
    const int e = e0 + g;
    float s = 0.f;
    if (e < NC)
      for (int l = w; l < np; l += width)
        s += ((float)abs((float)x[e * np + l].hi) + 1.f) * __int_as_float((127 - kFoLow + T[l]) << 23);
    for (int o = width >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (e < NC && w == 0) unit[e] = (__float_as_int(s * 1.0001f) >> 23) - 126;
  }
}

// FP64 value of v in unit 2^(unit + more); NaN for kFxBad
__device__ __forceinline__ double fx_value(long long v, int unit, int more = 0) {
  const int e = unit + more - 2 * kFoLow;
  if (e > 900) return __longlong_as_double(0x7ff8000000000000LL);
  return e < -900 ? 0.0 : fx_to_double(v, e);
}
__device__ __forceinline__ double fx_value(Fx v, int unit, int more = 0) { return fx_value(fo_join(v), unit, more); }

// x 2^s, |s| < 60, the result at most 1
__device__ __forceinline__ Fx fx_scale(Fx a, int s) {
  const long long v = fo_join(a);
  return fo_split(s >= 0 ? (long long)((unsigned long long)v << s) : FxShift(-s)(v));
}

}  // namespace sse
