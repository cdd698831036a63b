// sse_device.cuh -- device-side data layout and pointwise physics of the
// GB300 residual library.
//
// Pointwise physics restates src/ConservationLaws/ConservationLaws.jl:75-156,
// src/ConservationLaws/euler_navierstokes.jl:58-225 and
// src/ConservationLaws/linear_advection_diffusion.jl:54-128 in FP64.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>
#include <cuda_runtime.h>

namespace sse {

constexpr int kMaxC = 5;
constexpr int kMaxD = 3;

// Reference-element operators on the device, preprocessed from the caller's
// CSC matrices and warped-product factors (all indices 0-based, int32).
struct DevOps {
  int d, nc, np, nq, nf, nfac, npf;
  // warped tensor-product Vandermonde (has_vdm == 0: V = I)
  int has_vdm, p1, M1, M2, M3;
  const double *A;    // M1 x p1      (Julia column-major)
  const double *B;    // M2 x p1 x p1
  const double *C;    // M3 x p1^3
  int nb12;           // number of (b1, b2) with b1 + b2 < p1 (3-D)
  const int *b12;     // packed b1 | b2 << 8, 3-D stage list
  const int *b12_index;  // p1 x p1 -> position in b12 list or -1
  const int *modes;   // np packed b1 | b2 << 8 | b3 << 16 in modal order
  const int *sigma;   // p1^d: modal index of (b1, b2[, b3]) or -1
  // R (facet x volume) as CSR rows, and R^T as CSR rows
  const int *R_ptr, *R_idx; const double *R_val;
  const int *Rt_ptr, *Rt_idx; const double *Rt_val;
  // StandardForm D_m and D_m^T as CSR rows
  const int *D_ptr[kMaxD], *D_idx[kMaxD]; const double *D_val[kMaxD];
  const int *Dt_ptr[kMaxD], *Dt_idx[kMaxD]; const double *Dt_val[kMaxD];
  // FluxDifferencingForm volume pairs: unique (i < j) in the union of the
  // S_m patterns; S values per direction (0 where S_m has no entry)
  int nvp;
  const int *vp_ij;      // i | j << 16
  const double *vp_S;    // nvp x d (pair-major)
  const double *vp_Sh;   // the same halved (exact), for ec_flux_dot_half
  const int *vp_inc_ptr; // nq + 1
  const int *vp_inc;     // (pair << 1) | (node is i ? 1 : 0)
  // facet-correction pairs: nonzeros of C (volume node i, facet node j)
  int nfp;
  const int *fp_ij;      // i | j << 16
  const double *fp_C;
  const double *fp_Ch;   // fp_C halved (exact)
  const int *fp_q_ptr, *fp_q;  // per volume node: incident pair ids
  const int *fp_f_ptr, *fp_f;  // per facet node: incident pair ids
  // FP32 copies of the operator values for the mixed form (rounded from FP64)
  const float *Af, *Bf, *Cf, *R_valf, *Rt_valf, *vp_Sf, *fp_Cf;
  // the mixed phase B's pair tables, one vector load per pair: volume pairs
  // as float4 (S_1..S_D in FP32, zero-padded, and vp_ij's bits in w), facet
  // pairs as float2 (C in FP32, fp_ij's bits in y)
  const float *vp_pkf, *fp_pkf;
  // dense V (nq x np, column-major) of a multidimensional modal basis:
  // has_vdm == 1 and dense_v == 1, the warped factors unused
  int dense_v;
  const double *Vd;
  const float *Vdf;
  // tables of sse_log / sse_exp (3 kLogTab + 2 kExpTab doubles)
  const double *math_tab;
};

// Operator values of scalar type T (FP64 form: the caller's values; mixed
// form: their FP32 roundings).
template <typename T> struct OpVals;
template <> struct OpVals<double> {
  __device__ static const double *A(const DevOps &o) { return o.A; }
  __device__ static const double *B(const DevOps &o) { return o.B; }
  __device__ static const double *C(const DevOps &o) { return o.C; }
  __device__ static const double *Rt(const DevOps &o) { return o.Rt_val; }
  __device__ static const double *Vd(const DevOps &o) { return o.Vd; }
};
template <> struct OpVals<float> {
  __device__ static const float *A(const DevOps &o) { return o.Af; }
  __device__ static const float *B(const DevOps &o) { return o.Bf; }
  __device__ static const float *C(const DevOps &o) { return o.Cf; }
  __device__ static const float *Rt(const DevOps &o) { return o.Rt_valf; }
  __device__ static const float *Vd(const DevOps &o) { return o.Vdf; }
};

__device__ __forceinline__ int modes_index2(const DevOps &op, int b1, int b2) {
  return op.sigma[b1 + op.p1 * b2];
}
__device__ __forceinline__ int modes_index3(const DevOps &op, int b1, int b2, int b3) {
  return op.sigma[b1 + op.p1 * (b2 + op.p1 * b3)];
}

struct DevGeo {
  const double *BJf;          // nf x ne
  const double *n_f;          // d x nf x ne
  const int *mapP;            // nf x ne, 0-based linear index into (nf, ne)
  const double *halfWLambda;  // nq x d x d x ne
  const double *WJ;           // nq x ne
  const double *Lambda_q;     // nq x d x d x ne
  const double *halfnJf;      // d x nf x ne
  const double *halfnJq;      // d x nfac x nq x ne
  const double *JinvW;        // nq x ne
  const double *WJinv;        // nq x ne
  // FP32 roundings of the FP64 metric terms for the mixed form; halfnJqt:
  // halfnJq transposed to (f D + m) n_q + i per element, so that the lanes
  // of a warp (different volume nodes i) read different banks; Lambda_qn:
  // Lambda_q node-major, value v = m + D n of node i at lambda_stride(D) i +
  // v (an odd stride: distinct nodes of a warp meet distinct banks)
  const float *BJff, *n_ff, *Lambda_qn, *halfnJff, *halfnJqf, *halfnJqt, *JinvWf, *WJinvf;
  // mixed form: the entropy projection of the constant function 1 at the
  // volume nodes (V M^-1 V^T (W J), nq x ne) and its facet values (R P1, nf x ne)
  const double *P1, *RP1;
  // their FP32 roundings less one (P(1) - 1, R P(1) - 1) and of W J, for the
  // FP32 phase A (the FP64 difference and conversion made once on the device)
  const float *P1m1f, *RP1m1f, *WJf;
  // mixed form: the FP64 phase-B residual of the constant reference state
  // (np x nc x ne), i.e. the reference-pressure terms the FP32 fluxes leave
  // out; zero to round-off on free-stream-preserving metrics, O(1) on curved
  // tets with the exact metrics.  Added back in the mixed phase B's FP64
  // epilogue; null until the reference state is chosen.
  const double *Rref;
};

// floats per node of the node-major FP32 metric terms Lambda_qn
__host__ __device__ constexpr int lambda_stride(int D) { return (D * D) % 2 ? D * D : D * D + 1; }

// Constants of the FP32 perturbation entropy maps, rounded once from the FP64
// reference state (w_ref: its entropy variables).
struct EntropyRefF {
  float gamma, gm1, igm1, rho_ref, p_ref, ip_ref, irho_ref, a_ref, ia_ref, rhoe_ref;
  float w_ref[5];
};

struct Physics {
  int law;       // 0 advection, 1 Euler
  int nflux;     // 0 LF, 1 central, 2 EC numerical flux
  int ec;        // two-point flux: 1 entropy-conservative (Ranocha), 0 otherwise
  int chandrashekar;  // 1: Chandrashekar's EC flux (taken when ec == 0)
  double half_lambda;
  double gamma, gm1, igm1, log_gm1;
  double ilm_q[4];   // igm1 (2, 2/3, 2/5, 2/7): the scaled inverse-logmean series
  double a[3];
  // mixed form: constant reference state (rho_ref, 0, ..., 0, E_ref) that the
  // FP32 nodal states are stored relative to, and p_ref = (gamma-1) E_ref
  double rho_ref, E_ref, p_ref;
  double theta_ref;  // p_ref / rho_ref
  double H_ref;      // gamma/(gamma-1) theta_ref: enthalpy removed from the energy fluxes
  double w_ref[5];   // entropy variables of the reference state
  // mixed-form phase A: the reference state's modal coefficient (mode0) and
  // the constants of the entropy-variable maps around it
  int mode0;         // modal index of the constant basis function
  double u_ref_modal[5];
  double ip_ref, irho_ref;  // 1 / p_ref, 1 / rho_ref
  double a_ref, ia_ref;     // a_ref and 1 / a_ref with a = -(gamma-1) w_E
  double rhoe_ref;          // (rho e) of the reference state: p_ref / (gamma-1)
  // FP32 roundings of the constants the mixed-form kernels use, made once on
  // the host when the reference state is chosen (a conversion in every
  // thread would run on the FP64 pipe, 1/64 of the FP32 rate)
  float f_gamma, f_gm1, f_igm1, f_half_lambda, f_rho_ref, f_p_ref, f_theta_ref, f_H_ref, f_E_ref;
  EntropyRefF cref;
};

// Integer quotient a / b for 0 <= a < 2^21 and b >= 1 through the
// correctly rounded FP32 reciprocal rb = 1/b (qrcp): the exact value
// (a + 1/2)/b lies at least 1/(2b) from the nearest integer, and the two
// roundings of the product move it by at most (a + 1/2) 2^-23 / b < 1/(4b),
// so truncation gives floor(a / b) exactly -- a few instructions instead of
// an integer division by a value known only at run time.
__device__ __forceinline__ float qrcp(int b) { return __frcp_rn((float)b); }
__device__ __forceinline__ int qdiv(int a, float rb) { return __float2int_rz(__fmul_rn((float)a + 0.5f, rb)); }

// ---------------------------------------------------------------------------
// logmean / inverse logmean (ConservationLaws.jl:132-156)
// ---------------------------------------------------------------------------
__device__ __forceinline__ double logmean(double x, double y) {
  double f2 = (x * (x - 2 * y) + y * y) / (x * (x + 2 * y) + y * y);
  if (f2 < 1.0e-4) return (x + y) * 105 / (210 + f2 * (70 + f2 * (42 + f2 * 30)));
  return (y - x) / log(y / x);
}

__device__ __forceinline__ double inv_logmean(double x, double y) {
  double f2 = (x * (x - 2 * y) + y * y) / (x * (x + 2 * y) + y * y);
  if (f2 < 1.0e-4) return (210 + f2 * (70 + f2 * (42 + f2 * 30))) / ((x + y) * 105);
  return log(y / x) / (y - x);
}

// ---------------------------------------------------------------------------
// FP64 fast path.  GB300 issues FP64 at 1/62 of its FP32 rate, so the
// residual's cost is its FP64 instruction count.  The functions below compute
// the reference's quantities with fewer FP64 instructions: one reciprocal
// shared by the logarithmic mean's series branch, the two-point flux
// contracted with its metric vector before the flux tensor is formed, and
// logarithms/exponentials instead of pow.  They agree with the reference's
// formulas to a few ulps (checked on the host in tests/test_device_math.py
// and against the oracle on the GPU).
// ---------------------------------------------------------------------------
#define SSE_HD __host__ __device__ __forceinline__

// 1/s for the positive, normal arguments of the flux and entropy algebra
// (sums of densities, pressures, temperatures, entropy variables): the
// hardware reciprocal approximation (PTX rcp.approx.ftz.f64) refined by two
// Newton-Raphson steps y <- y + y (1 - s y), each of which squares the
// relative error, which leaves the result within about an ulp of 1/s -- four
// FMAs, where a correctly rounded reciprocal needs a longer sequence on the
// FP64 pipe.  Zero, infinite and subnormal arguments (never physical here)
// give NaN or flush, which the non-physical flag reports.
SSE_HD double sse_rcp(double s) {
#ifdef __CUDA_ARCH__
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(s));
  double e = fma(-s, y, 1.0);
  y = fma(y, e, y);
  e = fma(-s, y, 1.0);
  return fma(y, e, y);
#else
  return 1.0 / s;
#endif
}

// 1/s to about 2^-38 relative: one Newton-Raphson step on the hardware
// approximation, for a quotient that only enters through the square of a
// ratio below 1e-2 (the logarithmic mean's f = (x - y)/(x + y) on its
// series branch), where that error moves the result by about 1e-16.
SSE_HD double sse_rcp_coarse(double s) {
#ifdef __CUDA_ARCH__
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(s));
  return fma(y, fma(-s, y, 1.0), y);
#else
  return 1.0 / s;
#endif
}

// ---------------------------------------------------------------------------
// Table-driven FP64 logarithm and exponential (P. T. P. Tang, "Table-driven
// implementation of the logarithm function in IEEE floating-point
// arithmetic", ACM TOMS 16(4), 1990, and "... of the exponential function",
// ACM TOMS 15(2), 1989), for the entropy-variable maps: about half the FP64
// instructions of a general log on this pipe (measured 9.4 against 17.5 ms
// for 2.7e8 calls), within ~2 ulp.
//
// log: x = 2^e m, m in [1, 2), F = m truncated to 7 fractional bits,
//   log x = e ln2 + log F + log(1 + r), r = (m - F) / F in [0, 2^-7),
//   log F in two parts from the table, log(1 + r) by its Taylor series to r^7.
// exp: x = (32 k + j) ln2/32 + r, |r| <= ln2/64,
//   exp x = 2^k 2^(j/32) exp(r), 2^(j/32) in two parts from the table,
//   exp(r) - 1 by its Taylor series to r^6.
// Zero, negative, subnormal, infinite or NaN arguments of log and |x| >= 700
// or NaN arguments of exp take the library functions (a non-physical state
// then still yields its NaN).
// ---------------------------------------------------------------------------
constexpr int kLogTab = 128, kExpTab = 32;  // log table: invF, logF hi, logF lo; exp: 2^(j/32) hi, lo

SSE_HD long long sse_bits(double x) {
#ifdef __CUDA_ARCH__
  return __double_as_longlong(x);
#else
  long long b;
  std::memcpy(&b, &x, 8);
  return b;
#endif
}
SSE_HD double sse_from_bits(long long b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double(b);
#else
  double x;
  std::memcpy(&x, &b, 8);
  return x;
#endif
}

// the tables (3 kLogTab + 2 kExpTab doubles), built on the host in extended precision
inline void sse_build_math_tables(double *t) {
  for (int j = 0; j < kLogTab; ++j) {
    const long double F = 1.0L + j / (long double)kLogTab;
    const long double l = logl(F);
    t[j] = (double)(1.0L / F);
    t[kLogTab + j] = (double)l;
    t[2 * kLogTab + j] = (double)(l - (long double)t[kLogTab + j]);
  }
  double *e = t + 3 * kLogTab;
  for (int j = 0; j < kExpTab; ++j) {
    const long double v = exp2l(j / (long double)kExpTab);
    e[j] = (double)v;
    e[kExpTab + j] = (double)(v - (long double)e[j]);
  }
}

SSE_HD double sse_log(double x, const double *tab) {
  const long long b = sse_bits(x);
  // positive normal finite x: 0x0010... <= b < 0x7ff0...
  if (!tab || (unsigned long long)(b - 0x0010000000000000LL) >= 0x7fe0000000000000ULL) return log(x);
  const int e = (int)(b >> 52) - 1023;
  const long long mb = (b & 0x000fffffffffffffLL) | 0x3ff0000000000000LL;
  const int j = (int)((mb >> 45) & (kLogTab - 1));
  const double m = sse_from_bits(mb), F = sse_from_bits(mb & ~0x00001fffffffffffLL);
#ifdef __CUDA_ARCH__
  const double invF = __ldg(tab + j), lF = __ldg(tab + kLogTab + j), lFlo = __ldg(tab + 2 * kLogTab + j);
#else
  const double invF = tab[j], lF = tab[kLogTab + j], lFlo = tab[2 * kLogTab + j];
#endif
  const double r = (m - F) * invF;
  const double p = fma(r * r,
                       fma(r, fma(r, fma(r, fma(r, fma(r, 1.0 / 7.0, -1.0 / 6.0), 0.2), -0.25), 1.0 / 3.0), -0.5),
                       r);
  const double ed = (double)e;
  // ln 2 in two parts, the first with trailing zeros (e ln2_hi exact)
  const double hi = fma(ed, 0x1.62e42fefa3800p-1, lF);
  const double lo = fma(ed, 0x1.ef35793c76730p-45, lFlo);
  return hi + (lo + p);
}

SSE_HD double sse_exp(double x, const double *tab) {
  const long long b = sse_bits(x);
  // |x| < 700 and not NaN
  if (!tab || (b & 0x7fffffffffffffffLL) >= 0x4085e00000000000LL) return exp(x);
  const double *e = tab + 3 * kLogTab;
  const double shift = 0x1.8p52;                          // round-to-integer shift
  const double t = fma(x, 0x1.71547652b82fep5, shift);    // x 32 / ln2
  const double nd = t - shift;
  const int n = (int)(sse_bits(t) & 0xffffffffLL);
  const int j = n & (kExpTab - 1), k = n >> 5;
  double r = fma(-nd, 0x1.62e42fefa0000p-6, x);           // ln2/32 in two parts
  r = fma(-nd, 0x1.cf79abc9e3b3ap-45, r);
  const double p =
      r * fma(r, fma(r, fma(r, fma(r, fma(r, 1.0 / 720.0, 1.0 / 120.0), 1.0 / 24.0), 1.0 / 6.0), 0.5), 1.0);
#ifdef __CUDA_ARCH__
  const double sh = __ldg(e + j), sl = __ldg(e + kExpTab + j);
#else
  const double sh = e[j], sl = e[kExpTab + j];
#endif
  const double v = sh + fma(sh, p, sl);
  return sse_from_bits(sse_bits(v) + ((long long)k << 52));
}

// 1/q(z) for q(z) = 1 + z/3 + z^2/5 + z^3/7 by its power series; for
// z < 1e-4 the first omitted term is below 1e-17 relative.
constexpr double kInvQ1 = -1.0 / 3.0;
constexpr double kInvQ2 = -4.0 / 45.0;
constexpr double kInvQ3 = -44.0 / 945.0;

// logmean(x, y) of ConservationLaws.jl:132-145: (x + y) / (2 q(f^2)) with
// f = (x - y)/(x + y) on the series branch, (y - x)/log(y/x) otherwise.
SSE_HD double logmean_fast(double x, double y) {
  const double s = x + y;
  const double f = (x - y) * sse_rcp_coarse(s);
  const double z = f * f;
  // (s / 2) (1/q) with the 1/2 taken by the coefficients: the same bits
  // (halving is exact), one multiplication fewer
  if (z < 1.0e-4) return s * fma(z, fma(z, fma(z, 0.5 * kInvQ3, 0.5 * kInvQ2), 0.5 * kInvQ1), 0.5);
  return (y - x) / log(y / x);
}

// inv_logmean(x, y) of ConservationLaws.jl:147-156: 2 q(f^2) / (x + y).
SSE_HD double inv_logmean_fast(double x, double y) {
  const double s = x + y;
  const double r = sse_rcp(s);
  const double f = (x - y) * r;
  const double z = f * f;
  // (2 r) q with the 2 taken by the coefficients: the same bits
  if (z < 1.0e-4) return r * fma(z, fma(z, fma(z, 2.0 * (1.0 / 7.0), 2.0 * 0.2), 2.0 * (1.0 / 3.0)), 2.0);
  return log(y / x) / (y - x);
}

// Per-node primitives in the layout [rho, p, beta = rho/p, V_1..V_D].
template <int D>
SSE_HD void euler_prim_fast(double gm1, const double *u, double *P) {
  const double rr = sse_rcp(u[0]);
  double s = 0.0;
#pragma unroll
  for (int m = 0; m < D; ++m) {
    P[3 + m] = u[m + 1] * rr;
    s = fma(P[3 + m], P[3 + m], s);
  }
  const double p = gm1 * (u[D + 1] - 0.5 * u[0] * s);
  P[0] = u[0];
  P[1] = p;
  P[2] = u[0] * sse_rcp(p);
}

// out[e] = sum_n G[n] F_ec(i, j)[e][n] for Ranocha's flux tensor
// (euler_navierstokes.jl:171-195) without forming the tensor:
//   out[0]     = rho_hat (Vbar . G)
//   out[1 + m] = rho_hat Vbar_m (Vbar . G) + pbar G_m
//   out[D + 1] = C rho_hat (Vbar . G) + (p_i (G . V_j) + p_j (G . V_i)) / 2
template <int D>
SSE_HD void ec_flux_dot(double igm1, const double *Pi, const double *Pj, const double *G,
                        double *out) {
  const double rho_hat = logmean_fast(Pi[0], Pj[0]);
  const double ilm = inv_logmean_fast(Pi[2], Pj[2]);
  double vs[D];
  double vv = 0.0, gvs = 0.0, gvi = 0.0, gvj = 0.0;
#pragma unroll
  for (int m = 0; m < D; ++m) {
    vs[m] = Pi[3 + m] + Pj[3 + m];
    vv = fma(Pi[3 + m], Pj[3 + m], vv);
    gvs = fma(G[m], vs[m], gvs);
    gvi = fma(G[m], Pi[3 + m], gvi);
    gvj = fma(G[m], Pj[3 + m], gvj);
  }
  const double f0 = 0.5 * rho_hat * gvs;
  const double pbar = 0.5 * (Pi[1] + Pj[1]);
  const double C = fma(igm1, ilm, 0.5 * vv);
  const double t = 0.5 * f0;
  out[0] = f0;
#pragma unroll
  for (int m = 0; m < D; ++m) out[1 + m] = fma(t, vs[m], pbar * G[m]);
  out[D + 1] = fma(C, f0, 0.5 * fma(Pi[1], gvj, Pj[1] * gvi));
}

// c inv_logmean(x, y) with c folded into the series coefficients
// q = c (2, 2/3, 2/5, 2/7) (on the series branch, one multiplication fewer
// than scaling the mean afterwards)
SSE_HD double inv_logmean_scaled(double x, double y, double c, const double *q) {
  const double s = x + y;
  const double r = sse_rcp(s);
  const double f = (x - y) * r;
  const double z = f * f;
  if (z < 1.0e-4) return r * fma(z, fma(z, fma(z, q[3], q[2]), q[1]), q[0]);
  return c * log(y / x) / (y - x);
}

// ec_flux_dot for a metric vector given halved (Gh = G / 2, exact): the
// factors 1/2 of the average pressure, of rho_hat Vbar . G and of the energy's
// pressure-velocity term are taken by the halved vector, which saves three
// multiplications, and the energy's C f0 = igm1 ilm f0 + (vv/2) f0 is formed
// as fma(f0/2, vv, f0 (igm1 ilm)) with igm1 in the inverse logmean's series
// coefficients (ilm_q = igm1 (2, 2/3, 2/5, 2/7)), two operations fewer.  The
// mass and momentum fluxes are bitwise those of ec_flux_dot(G) (scaling by
// 1/2 is exact away from underflow); the energy flux agrees to rounding.
template <int D>
SSE_HD void ec_flux_dot_half(double igm1, const double *ilm_q, const double *Pi, const double *Pj,
                             const double *Gh, double *out) {
  const double rho_hat = logmean_fast(Pi[0], Pj[0]);
  const double ilmc = inv_logmean_scaled(Pi[2], Pj[2], igm1, ilm_q);
  double vs[D];
  double vv = 0.0, gvs = 0.0, gvi = 0.0, gvj = 0.0;
#pragma unroll
  for (int m = 0; m < D; ++m) {
    vs[m] = Pi[3 + m] + Pj[3 + m];
    vv = fma(Pi[3 + m], Pj[3 + m], vv);
    gvs = fma(Gh[m], vs[m], gvs);
    gvi = fma(Gh[m], Pi[3 + m], gvi);
    gvj = fma(Gh[m], Pj[3 + m], gvj);
  }
  const double f0 = rho_hat * gvs;
  const double psum = Pi[1] + Pj[1];
  const double t = 0.5 * f0;
  out[0] = f0;
#pragma unroll
  for (int m = 0; m < D; ++m) out[1 + m] = fma(t, vs[m], psum * Gh[m]);
  out[D + 1] = fma(t, vv, fma(f0, ilmc, fma(Pi[1], gvj, Pj[1] * gvi)));
}

// conservative_to_entropy! (euler_navierstokes.jl:100-113) with
// log(p / rho^gamma) = log(p) - gamma log(rho).
// mt: the tables of sse_log / sse_exp (null: the library functions)
template <int D>
SSE_HD void cons_to_entropy_fast(double gamma, double gm1, double igm1, const double *u, double *w,
                                 const double *mt = nullptr) {
  double s = 0.0;
#pragma unroll
  for (int m = 0; m < D; ++m) s = fma(u[m + 1], u[m + 1], s);
  const double k = 0.5 * s * sse_rcp(u[0]);
  const double p = gm1 * (u[D + 1] - k);
  const double ip = sse_rcp(p);
  w[0] = fma(igm1, gamma - (sse_log(p, mt) - gamma * sse_log(u[0], mt)), -k * ip);
#pragma unroll
  for (int m = 0; m < D; ++m) w[m + 1] = u[m + 1] * ip;
  w[D + 1] = -u[0] * ip;
}

// entropy_to_conservative! (euler_navierstokes.jl:115-131) with
// (gm1/(-w_E)^gamma)^(1/gm1) exp(-s/gm1) = exp((log gm1 - gamma log(-w_E) - s)/gm1).
template <int D>
SSE_HD void entropy_to_cons_fast(double gamma, double gm1, double igm1, double log_gm1,
                                 const double *w_in, double *u, const double *mt = nullptr) {
  double w[D + 2];
#pragma unroll
  for (int e = 0; e < D + 2; ++e) w[e] = w_in[e] * gm1;
  double s = 0.0;
#pragma unroll
  for (int m = 0; m < D; ++m) s = fma(w[m + 1], w[m + 1], s);
  const double k = 0.5 * s * sse_rcp(w[D + 1]);
  const double sv = gamma - w[0] + k;
  const double rhoe = sse_exp(igm1 * (log_gm1 - gamma * sse_log(-w[D + 1], mt) - sv), mt);
  u[0] = -w[D + 1] * rhoe;
#pragma unroll
  for (int m = 0; m < D; ++m) u[m + 1] = w[m + 1] * rhoe;
  u[D + 1] = rhoe * (1 - k);
}

// The same map with fewer operations: in the formula above the factors of
// gamma - 1 cancel, so that with k = |w_m|^2 / (2 w_E) and p the pressure
//   log p = w_0 - k - gamma/(gamma - 1) (1 + log(-w_E)),
//   rho = -w_E p, m = w_m p, E = p (1/(gamma - 1) - k).
// On a par in accuracy (residual errors within 5 % of the other's either way).
template <int D>
SSE_HD void entropy_to_cons_pressure(double gamma, double igm1, const double *w, double *u, const double *mt) {
  double s = 0.0;
#pragma unroll
  for (int m = 0; m < D; ++m) s = fma(w[m + 1], w[m + 1], s);
  const double k = 0.5 * s * sse_rcp(w[D + 1]);
  const double g = gamma * igm1;
  const double p = sse_exp(fma(-g, sse_log(-w[D + 1], mt), (w[0] - k) - g), mt);
  u[0] = -w[D + 1] * p;
#pragma unroll
  for (int m = 0; m < D; ++m) u[m + 1] = w[m + 1] * p;
  u[D + 1] = p * (igm1 - k);
}

// ---------------------------------------------------------------------------
// Reverse-mode derivatives (discrete adjoint of the FP64 residual).  Each
// function below is the hand-written transpose of the forward function of
// the same name above; tests/device_math_check.cu checks them against
// central differences.
// ---------------------------------------------------------------------------

// logmean_fast(x, y) and its partial derivatives, sharing one reciprocal
SSE_HD double logmean_fast_vgrad(double x, double y, double *dx, double *dy) {
  const double s = x + y;
  const double r = sse_rcp(s);
  const double f = (x - y) * r;
  const double z = f * f;
  if (z < 1.0e-4) {
    const double P = fma(z, fma(z, fma(z, kInvQ3, kInvQ2), kInvQ1), 1.0);
    const double dP = fma(z, fma(z, 3.0 * kInvQ3, 2.0 * kInvQ2), kInvQ1);
    const double c = 2.0 * s * dP * f * r * r;  // (s/2) P'(z) dz/dx with dz/dx = 4 f y / s^2
    *dx = fma(c, y, 0.5 * P);
    *dy = fma(-c, x, 0.5 * P);
    return 0.5 * s * P;
  }
  const double N = y - x, Dl = log(y / x);
  const double iD = 1.0 / Dl;
  const double iD2 = iD * iD;
  *dx = (-Dl + N / x) * iD2;
  *dy = (Dl - N / y) * iD2;
  return N * iD;
}

// inv_logmean_fast(x, y) and its partial derivatives
SSE_HD double inv_logmean_fast_vgrad(double x, double y, double *dx, double *dy) {
  const double s = x + y;
  const double r = sse_rcp(s);
  const double f = (x - y) * r;
  const double z = f * f;
  if (z < 1.0e-4) {
    const double Q = fma(z, fma(z, fma(z, 1.0 / 7.0, 0.2), 1.0 / 3.0), 1.0);
    const double dQ = fma(z, fma(z, 3.0 / 7.0, 0.4), 1.0 / 3.0);
    const double r2 = r * r;
    const double base = -2.0 * r2 * Q;
    const double c = 8.0 * r * dQ * f * r2;  // 2 r Q'(z) dz/dx with dz/dx = 4 f y / s^2
    *dx = fma(c, y, base);
    *dy = fma(-c, x, base);
    return 2.0 * r * Q;
  }
  const double N = y - x, Dl = log(y / x);
  const double iN = 1.0 / N;
  const double iN2 = iN * iN;
  *dx = (Dl - N / x) * iN2;
  *dy = (N / y - Dl) * iN2;
  return Dl * iN;
}

// Transpose of ec_flux_dot with respect to the two primitive vectors:
// given ob = d(objective)/d(out), returns Pbi, Pbj (layout [rho, p, beta, V]).
template <int D>
SSE_HD void ec_flux_dot_bwd(double igm1, const double *Pi, const double *Pj, const double *G,
                            const double *ob, double *Pbi, double *Pbj) {
  double dlx, dly, dix, diy;
  const double rho_hat = logmean_fast_vgrad(Pi[0], Pj[0], &dlx, &dly);
  const double ilm = inv_logmean_fast_vgrad(Pi[2], Pj[2], &dix, &diy);
  double vs[D];
  double vv = 0.0, gvs = 0.0, gvi = 0.0, gvj = 0.0;
#pragma unroll
  for (int m = 0; m < D; ++m) {
    vs[m] = Pi[3 + m] + Pj[3 + m];
    vv = fma(Pi[3 + m], Pj[3 + m], vv);
    gvs = fma(G[m], vs[m], gvs);
    gvi = fma(G[m], Pi[3 + m], gvi);
    gvj = fma(G[m], Pj[3 + m], gvj);
  }
  const double f0 = 0.5 * rho_hat * gvs;
  const double C = fma(igm1, ilm, 0.5 * vv);
  const double t = 0.5 * f0;
  const double oE = ob[D + 1];
  // reverse sweep
  double ovs_dot = 0.0, pbar_b = 0.0;
#pragma unroll
  for (int m = 0; m < D; ++m) {
    ovs_dot = fma(ob[1 + m], vs[m], ovs_dot);
    pbar_b = fma(ob[1 + m], G[m], pbar_b);
  }
  const double f0b = ob[0] + C * oE + 0.5 * ovs_dot;
  const double Cb = oE * f0;
  const double gvjb = 0.5 * oE * Pi[1];
  const double gvib = 0.5 * oE * Pj[1];
  const double gvsb = 0.5 * rho_hat * f0b;
  const double rhob = 0.5 * gvs * f0b;
  const double ilmb = igm1 * Cb;
  const double vvb = 0.5 * Cb;
  Pbi[0] = rhob * dlx;
  Pbj[0] = rhob * dly;
  Pbi[1] = 0.5 * pbar_b + 0.5 * oE * gvj;
  Pbj[1] = 0.5 * pbar_b + 0.5 * oE * gvi;
  Pbi[2] = ilmb * dix;
  Pbj[2] = ilmb * diy;
#pragma unroll
  for (int m = 0; m < D; ++m) {
    const double vsb = fma(t, ob[1 + m], G[m] * gvsb);
    Pbi[3 + m] = vsb + Pj[3 + m] * vvb + G[m] * gvib;
    Pbj[3 + m] = vsb + Pi[3 + m] * vvb + G[m] * gvjb;
  }
}

// Transpose of euler_prim_fast: accumulate ub += (dP/du)^T Pb.
template <int D>
SSE_HD void euler_prim_bwd(double gm1, const double *u, const double *P, const double *Pb, double *ub) {
  const double rho = P[0], p = P[1];
  const double rr = sse_rcp(rho);
  const double pb = Pb[1] - Pb[2] * rho / (p * p);
  double v2 = 0.0, vvb = 0.0;
#pragma unroll
  for (int m = 0; m < D; ++m) {
    v2 = fma(P[3 + m], P[3 + m], v2);
    vvb = fma(Pb[3 + m], P[3 + m], vvb);
  }
  ub[0] += Pb[0] + Pb[2] / p + 0.5 * gm1 * pb * v2 - vvb * rr;
#pragma unroll
  for (int m = 0; m < D; ++m) ub[m + 1] += fma(-gm1 * pb, P[3 + m], Pb[3 + m] * rr);
  ub[D + 1] += gm1 * pb;
  (void)u;
}

// Directional derivative of cons_to_entropy_fast at u along du.  The map is
// the gradient of the entropy function, so its Jacobian is symmetric and
// this is also the transpose product.
template <int D>
SSE_HD void cons_to_entropy_jvp(double gamma, double gm1, double igm1, const double *u,
                                const double *du, double *dw) {
  const double rho = u[0], rr = sse_rcp(rho);
  double s = 0.0, vdm = 0.0;
#pragma unroll
  for (int m = 0; m < D; ++m) {
    s = fma(u[m + 1], u[m + 1], s);
    vdm = fma(u[m + 1] * rr, du[m + 1], vdm);
  }
  const double k = 0.5 * s * rr;
  const double dk = vdm - 0.5 * s * rr * rr * du[0];
  const double p = gm1 * (u[D + 1] - k);
  const double dp = gm1 * (du[D + 1] - dk);
  const double ip = sse_rcp(p);
  dw[0] = -igm1 * (dp * ip - gamma * du[0] * rr) - (dk * ip - k * dp * ip * ip);
#pragma unroll
  for (int m = 0; m < D; ++m) dw[m + 1] = du[m + 1] * ip - u[m + 1] * dp * ip * ip;
  dw[D + 1] = -du[0] * ip + rho * dp * ip * ip;
}

// Directional derivative of entropy_to_cons_fast at w along dw (symmetric
// Jacobian: the inverse of the entropy Hessian).
template <int D>
SSE_HD void entropy_to_cons_jvp(double gamma, double gm1, double igm1, double log_gm1,
                                const double *w_in, const double *dw_in, double *du,
                                const double *mt = nullptr) {
  double w[D + 2], dw[D + 2];
#pragma unroll
  for (int e = 0; e < D + 2; ++e) {
    w[e] = w_in[e] * gm1;
    dw[e] = dw_in[e] * gm1;
  }
  double s = 0.0, ds = 0.0;
#pragma unroll
  for (int m = 0; m < D; ++m) {
    s = fma(w[m + 1], w[m + 1], s);
    ds = fma(w[m + 1], dw[m + 1], ds);
  }
  const double iwE = sse_rcp(w[D + 1]);
  const double k = 0.5 * s * iwE;
  const double dk = ds * iwE - k * dw[D + 1] * iwE;
  const double sv = gamma - w[0] + k;
  const double dsv = -dw[0] + dk;
  const double rhoe = sse_exp(igm1 * (log_gm1 - gamma * sse_log(-w[D + 1], mt) - sv), mt);
  const double drhoe = rhoe * igm1 * (-gamma * dw[D + 1] * iwE - dsv);
  du[0] = -dw[D + 1] * rhoe - w[D + 1] * drhoe;
#pragma unroll
  for (int m = 0; m < D; ++m) du[m + 1] = dw[m + 1] * rhoe + w[m + 1] * drhoe;
  du[D + 1] = drhoe * (1 - k) - rhoe * dk;
}

// ---------------------------------------------------------------------------
// Mixed form: FP32 arithmetic on perturbations u' = u - u_ref from a constant
// reference state u_ref = (rho_ref, 0, ..., 0, E_ref) with p_ref =
// (gamma - 1) E_ref.  At Mach 0.1 the pressure (~71) exceeds its fluctuations
// by three orders of magnitude; an FP32 state would lose them, a perturbation
// keeps them.  The reference pressure is dropped from every momentum flux
// (volume pairs, facet correction, interface flux): for the constant state
// u_ref all fluxes reduce to that isotropic pressure term, so the dropped
// terms are, together, the FP64 residual of u_ref evaluated at its nodal
// states -- a constant of the mesh (DevGeo::Rref).  It vanishes to round-off
// where the metric terms preserve a free stream (conservative-curl metrics,
// straight or 2-D elements) and is O(p_ref) on curved tets with the exact
// metrics (the reference's default); phase B adds it back in FP64, so the
// mixed residual equals the FP64 one on both.  Being constant in u, it
// changes no Jacobian: the mixed-form VJP needs no counterpart.
// ---------------------------------------------------------------------------

// FP32 quotient for the mixed form: the fast reciprocal-based division
// (2 ulp) on the device, where the form's error budget is set by the FP32
// rounding of the perturbations anyway; exact division on the host.
SSE_HD float sse_fdiv(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fdividef(a, b);
#else
  return a / b;
#endif
}

// 1 + z/3 + z^2/5 + z^3/7 + z^4/9 + z^5/11 (= atanh(f)/f, z = f^2)
SSE_HD float q_series_f(float z) {
  return fmaf(z, fmaf(z, fmaf(z, fmaf(z, fmaf(z, 1.f / 11.f, 1.f / 9.f), 1.f / 7.f), 0.2f), 1.f / 3.f), 1.f);
}

// logmean in FP32 with the series branch widened to z < 0.05 (truncation
// below 2e-9 relative), so the log branch -- relative error ~ eps/|f| -- is
// only taken for |f| > 0.22.
SSE_HD float logmean_mixed(float x, float y) {
  const float s = x + y;
  const float f = (x - y) / s;
  const float z = f * f;
  if (z < 0.05f) return 0.5f * s / q_series_f(z);
  return (y - x) / logf(y / x);
}

SSE_HD float inv_logmean_mixed(float x, float y) {
  const float s = x + y;
  const float f = (x - y) / s;
  const float z = f * f;
  if (z < 0.05f) return 2.f * q_series_f(z) / s;
  return logf(y / x) / (y - x);
}

// The energy flux carries a large enthalpy part: Ranocha's energy flux is
// f_E = f_rho C + (p_i V_j + p_j V_i)/2 with C ~ theta/(gamma-1), theta =
// p/rho.  With H_ref = gamma/(gamma-1) theta_ref (theta_ref = p_ref/rho_ref)
// the reduced flux f_E - H_ref f_rho is, exactly,
//   f_rho (C - C_ref) + (Vbar . G)(rho_ref - rho_hat) theta_ref
//   + (p'_i V_j + p'_j V_i)/2,          C_ref = theta_ref/(gamma-1),
// a sum of products of fluctuations.  Every energy flux (volume pairs, facet
// correction, interface flux including its dissipation) is reduced the same
// way, so the energy residual equals H_ref times the density residual plus
// the residual of the reduced fluxes; that sum is formed in FP64 at the end.


SSE_HD EntropyRefF entropy_ref_f(const Physics &ph) {
  EntropyRefF c;
  c.gamma = (float)ph.gamma;
  c.gm1 = (float)ph.gm1;
  c.igm1 = (float)ph.igm1;
  c.rho_ref = (float)ph.rho_ref;
  c.p_ref = (float)ph.p_ref;
  c.ip_ref = (float)ph.ip_ref;
  c.irho_ref = (float)ph.irho_ref;
  c.a_ref = (float)ph.a_ref;
  c.ia_ref = (float)ph.ia_ref;
  c.rhoe_ref = (float)ph.rhoe_ref;
  for (int e = 0; e < 5; ++e) c.w_ref[e] = (float)ph.w_ref[e];
  return c;
}

// Entropy variables as perturbations, in FP32: dw = w(u_ref + du) - w_ref for
// du = u - u_ref (cons_to_entropy, euler_navierstokes.jl:100-115).  Every term
// is formed from perturbations -- s - s_ref = log1p(dp/p_ref) - gamma
// log1p(drho/rho_ref), rho/p - rho_ref/p_ref = (drho - rho_ref dp/p_ref)/p --
// so FP32 keeps its relative accuracy on dw, which is small where the flow is
// near the reference state (no difference of two O(1) entropy variables).
template <int D>
SSE_HD void cons_to_entropy_pert(const EntropyRefF &c, const float *du, float *dw) {
  float s2 = 0.f;
#pragma unroll
  for (int m = 0; m < D; ++m) s2 = fmaf(du[m + 1], du[m + 1], s2);
  const float k = 0.5f * sse_fdiv(s2, c.rho_ref + du[0]);   // kinetic energy
  const float dp = c.gm1 * (du[D + 1] - k);                   // p - p_ref
  const float ip = sse_fdiv(1.f, c.p_ref + dp);
  const float dpr = dp * c.ip_ref;
  const float ds = log1pf(dpr) - c.gamma * log1pf(du[0] * c.irho_ref);  // s - s_ref
  dw[0] = -fmaf(c.igm1, ds, k * ip);
#pragma unroll
  for (int m = 0; m < D; ++m) dw[m + 1] = du[m + 1] * ip;
  dw[D + 1] = -fmaf(-c.rho_ref, dpr, du[0]) * ip;
}

// Conservative perturbations from entropy-variable perturbations, in FP32:
// du = u(w_ref + dw) - u_ref (entropy_to_cons, euler_navierstokes.jl:117-131).
// With a = -(gamma-1) w_E = a_ref (1 + alpha), k = |(gamma-1) w_m|^2 / (2 (gamma-1)
// w_E) and (rho e) = (rho e)_ref (1 + beta):  drho = rho_ref (alpha + beta +
// alpha beta), m = (gamma-1) w_m (rho e), dE = (rho e)_ref (beta - k (1 + beta)).
template <int D>
SSE_HD void entropy_pert_core(const EntropyRefF &c, const float *dw, float &alpha, float &beta, float &k) {
  float s2 = 0.f;
#pragma unroll
  for (int m = 0; m < D; ++m) {
    const float g = c.gm1 * dw[m + 1];
    s2 = fmaf(g, g, s2);
  }
  const float gw = c.gm1 * dw[D + 1];
  alpha = -gw * c.ia_ref;                                      // a / a_ref - 1
  k = -0.5f * sse_fdiv(s2, c.a_ref - gw);
  const float dX = dw[0] - c.igm1 * fmaf(c.gamma, log1pf(alpha), k);
  beta = expm1f(dX);                                           // (rho e) / (rho e)_ref - 1
}

template <int D>
SSE_HD void entropy_to_cons_pert(const EntropyRefF &c, const float *dw, float *du) {
  float alpha, beta, k;
  entropy_pert_core<D>(c, dw, alpha, beta, k);
  const float rhoe = c.rhoe_ref * (1.f + beta);
  du[0] = c.rho_ref * fmaf(alpha, beta, alpha + beta);
#pragma unroll
  for (int m = 0; m < D; ++m) du[m + 1] = c.gm1 * dw[m + 1] * rhoe;
  du[D + 1] = c.rhoe_ref * fmaf(-k, 1.f + beta, beta);
}

// FP32 JVPs of the entropy-variable maps for the mixed-form VJP (both
// Jacobians are symmetric, so the transposes are these JVPs), at absolute
// FP32 states: the Jacobian entries are O(1) functions of the state, which
// FP32 resolves to its own relative accuracy.  Same formulas as
// cons_to_entropy_jvp and entropy_to_cons_jvp, the latter given rho e.
template <int D>
SSE_HD void cons_to_entropy_jvp_f(float gamma, float gm1, float igm1, const float *u, const float *du,
                                  float *dw) {
  const float rho = u[0], rr = sse_fdiv(1.f, rho);
  float s = 0.f, vdm = 0.f;
#pragma unroll
  for (int m = 0; m < D; ++m) {
    s = fmaf(u[m + 1], u[m + 1], s);
    vdm = fmaf(u[m + 1] * rr, du[m + 1], vdm);
  }
  const float k = 0.5f * s * rr;
  const float dk = vdm - 0.5f * s * rr * rr * du[0];
  const float p = gm1 * (u[D + 1] - k);
  const float dp = gm1 * (du[D + 1] - dk);
  const float ip = sse_fdiv(1.f, p);
  dw[0] = -igm1 * (dp * ip - gamma * du[0] * rr) - (dk * ip - k * dp * ip * ip);
#pragma unroll
  for (int m = 0; m < D; ++m) dw[m + 1] = du[m + 1] * ip - u[m + 1] * dp * ip * ip;
  dw[D + 1] = -du[0] * ip + rho * dp * ip * ip;
}

template <int D>
SSE_HD void entropy_to_cons_jvp_rhoe_f(float gm1, float igm1, float gamma, const float *w_in, float rhoe,
                                       const float *dw_in, float *du) {
  float w[D + 2], dw[D + 2];
#pragma unroll
  for (int e = 0; e < D + 2; ++e) {
    w[e] = w_in[e] * gm1;
    dw[e] = dw_in[e] * gm1;
  }
  float s = 0.f, ds = 0.f;
#pragma unroll
  for (int m = 0; m < D; ++m) {
    s = fmaf(w[m + 1], w[m + 1], s);
    ds = fmaf(w[m + 1], dw[m + 1], ds);
  }
  const float iwE = sse_fdiv(1.f, w[D + 1]);
  const float k = 0.5f * s * iwE;
  const float dk = ds * iwE - k * dw[D + 1] * iwE;
  const float dsv = -dw[0] + dk;
  const float drhoe = rhoe * igm1 * (-gamma * dw[D + 1] * iwE - dsv);
  du[0] = -dw[D + 1] * rhoe - w[D + 1] * drhoe;
#pragma unroll
  for (int m = 0; m < D; ++m) du[m + 1] = dw[m + 1] * rhoe + w[m + 1] * drhoe;
  du[D + 1] = drhoe * (1.f - k) - rhoe * dk;
}

// FP32 primitives from a perturbation du = u - u_ref, layout
// [rho, rho - rho_ref, theta - theta_ref, V_1..V_D, p - p_ref].
template <int D>
SSE_HD void euler_prim_mixed(float gm1, float rho_ref, float p_ref, const float *du, float *P) {
  const float rho = rho_ref + du[0];
  const float rr = sse_fdiv(1.f, rho);
  float s = 0.f;
#pragma unroll
  for (int m = 0; m < D; ++m) {
    P[3 + m] = du[m + 1] * rr;
    s = fmaf(P[3 + m], P[3 + m], s);
  }
  const float pp = gm1 * (du[D + 1] - 0.5f * rho * s);
  P[0] = rho;
  P[1] = du[0];
  P[2] = sse_fdiv((pp * rho_ref - p_ref * du[0]) * rr, rho_ref);  // p/rho - p_ref/rho_ref
  P[3 + D] = pp;
}

// q(z) - 1 = z/3 + z^2/5 + ... (series of the FP32 branch)
SSE_HD float q_minus_one_f(float z) {
  return z * fmaf(z, fmaf(z, fmaf(z, fmaf(z, 1.f / 11.f, 1.f / 9.f), 1.f / 7.f), 0.2f), 1.f / 3.f);
}

// logmean(rho_i, rho_j) - rho_ref from density perturbations
SSE_HD float logmean_minus_ref(float rho_ref, float ri, float rj, float dri, float drj) {
  const float s = 2.f * rho_ref + (dri + drj);
  const float f = sse_fdiv(dri - drj, s);
  const float z = f * f;
  if (z < 0.05f) {
    const float qm1 = q_minus_one_f(z);
    return sse_fdiv(0.5f * (dri + drj) - rho_ref * qm1, 1.f + qm1);
  }
  return sse_fdiv(rj - ri, logf(sse_fdiv(rj, ri))) - rho_ref;
}

// inv_logmean(beta_i, beta_j) - theta_ref with beta = 1/theta, from
// temperature perturbations dti = theta_i - theta_ref
SSE_HD float inv_logmean_beta_minus_ref(float theta_ref, float dti, float dtj) {
  const float ti = theta_ref + dti, tj = theta_ref + dtj;
  const float sig = dti + dtj;
  const float den = 2.f * theta_ref + sig;
  const float rden = sse_fdiv(1.f, den);
  const float f = (dtj - dti) * rden;
  const float z = f * f;
  if (z < 0.05f) {
    const float hm_minus = (theta_ref * sig + 2.f * dti * dtj) * rden;  // 2 ti tj/(ti+tj) - theta_ref
    const float hm = theta_ref + hm_minus;
    return fmaf(q_minus_one_f(z), hm, hm_minus);
  }
  return sse_fdiv(ti * tj * logf(sse_fdiv(ti, tj)), ti - tj) - theta_ref;
}

// ec_flux_dot in FP32: momentum with pbar - p_ref, energy reduced by H_ref f_rho.
template <int D>
SSE_HD void ec_flux_dot_mixed(float igm1, float rho_ref, float theta_ref, const float *Pi,
                              const float *Pj, const float *G, float *out) {
  // both means by their series when both pairs of arguments are close (one
  // branch per flux; the same expressions as logmean_minus_ref and
  // inv_logmean_beta_minus_ref, which take the other cases)
  float drho_hat, dilm;
  {
    const float dri = Pi[1], drj = Pj[1], dti = Pi[2], dtj = Pj[2];
    const float fr = sse_fdiv(dri - drj, 2.f * rho_ref + (dri + drj));
    const float zr = fr * fr;
    const float sig = dti + dtj;
    const float rden = sse_fdiv(1.f, 2.f * theta_ref + sig);
    const float ft = (dtj - dti) * rden;
    const float zt = ft * ft;
    if (zr < 0.05f && zt < 0.05f) {
      const float qm1 = q_minus_one_f(zr);
      drho_hat = sse_fdiv(0.5f * (dri + drj) - rho_ref * qm1, 1.f + qm1);
      const float hm_minus = (theta_ref * sig + 2.f * dti * dtj) * rden;
      const float hm = theta_ref + hm_minus;
      dilm = fmaf(q_minus_one_f(zt), hm, hm_minus);
    } else {
      drho_hat = logmean_minus_ref(rho_ref, rho_ref + dri, rho_ref + drj, dri, drj);  // = P[0] (no load)
      dilm = inv_logmean_beta_minus_ref(theta_ref, dti, dtj);
    }
  }
  float vs[D];
  float vv = 0.f, gvs = 0.f, gvi = 0.f, gvj = 0.f;
#pragma unroll
  for (int m = 0; m < D; ++m) {
    vs[m] = Pi[3 + m] + Pj[3 + m];
    vv = fmaf(Pi[3 + m], Pj[3 + m], vv);
    gvs = fmaf(G[m], vs[m], gvs);
    gvi = fmaf(G[m], Pi[3 + m], gvi);
    gvj = fmaf(G[m], Pj[3 + m], gvj);
  }
  const float rho_hat = rho_ref + drho_hat;
  const float f0 = 0.5f * rho_hat * gvs;
  const float pbar_pert = 0.5f * (Pi[3 + D] + Pj[3 + D]);
  const float dC = fmaf(igm1, dilm, 0.5f * vv);  // C - C_ref
  const float t = 0.5f * f0;
  out[0] = f0;
#pragma unroll
  for (int m = 0; m < D; ++m) out[1 + m] = fmaf(t, vs[m], pbar_pert * G[m]);
  out[D + 1] = fmaf(dC, f0, fmaf(-0.5f * gvs * theta_ref, drho_hat,
                                 0.5f * fmaf(Pi[3 + D], gvj, Pj[3 + D] * gvi)));
}

// ---------------------------------------------------------------------------
// Reverse mode of the mixed form (FP32): transposes of euler_prim_mixed and
// ec_flux_dot_mixed.  The residual's energy component is H_ref times the
// density residual plus the reduced-flux residual, so for a cotangent lam of
// the residual the reduced fluxes see lam~ = (lam_rho + H_ref lam_E, lam_m,
// lam_E); their Jacobians carry no enthalpy-sized terms, which keeps FP32
// accurate at low Mach.  Checked against the FP64 transposes in
// tests/device_math_check.cu.
// ---------------------------------------------------------------------------

// q'(z) for q = 1 + z/3 + z^2/5 + ... (the FP32 series)
SSE_HD float q_series_f_deriv(float z) {
  return fmaf(z, fmaf(z, fmaf(z, fmaf(z, 5.f / 11.f, 4.f / 9.f), 3.f / 7.f), 0.4f), 1.f / 3.f);
}

// partial derivatives of logmean(x, y) (the value of the mixed form comes
// from logmean_minus_ref)
SSE_HD void logmean_f_grad(float x, float y, float *dx, float *dy) {
  const float s = x + y;
  const float is = sse_fdiv(1.f, s);
  const float f = (x - y) * is;
  const float z = f * f;
  if (z < 0.05f) {
    const float iq = sse_fdiv(1.f, q_series_f(z));
    const float c = 2.f * q_series_f_deriv(z) * f * iq * iq * is;
    *dx = fmaf(-c, y, 0.5f * iq);
    *dy = fmaf(c, x, 0.5f * iq);
    return;
  }
  const float L = logf(sse_fdiv(y, x)), iL = sse_fdiv(1.f, L), N = y - x;
  *dx = (sse_fdiv(N, x) - L) * iL * iL;
  *dy = (L - sse_fdiv(N, y)) * iL * iL;
}

// partial derivatives of inv_logmean(1/theta_i, 1/theta_j) w.r.t. the
// temperatures theta_i, theta_j: q(z) hm with hm = 2 ti tj/(ti + tj),
// f = (tj - ti)/(ti + tj) on the series branch
SSE_HD void inv_logmean_theta_grad(float ti, float tj, float *di, float *dj) {
  const float sg = ti + tj;
  const float isg = sse_fdiv(1.f, sg);
  const float f = (tj - ti) * isg;
  const float z = f * f;
  if (z < 0.05f) {
    const float q = q_series_f(z), qp = q_series_f_deriv(z);
    const float is2 = isg * isg;
    const float hm = 2.f * ti * tj * isg;
    *di = fmaf(qp * hm, -4.f * f * tj * is2, q * 2.f * tj * tj * is2);
    *dj = fmaf(qp * hm, 4.f * f * ti * is2, q * 2.f * ti * ti * is2);
    return;
  }
  const float L = logf(sse_fdiv(ti, tj)), N = ti - tj, iN = sse_fdiv(1.f, N);
  const float w = ti * tj * L * iN * iN;
  *di = fmaf(tj, (L + 1.f) * iN, -w);
  *dj = fmaf(ti, (L - 1.f) * iN, w);
}

// Transpose of ec_flux_dot_mixed w.r.t. the two primitive vectors (layout
// [rho, rho', theta', V_1..V_D, p']); the density cotangent is returned in
// slot 1 (rho' and rho are the same variable), slot 0 is zero.
template <int D>
SSE_HD void ec_flux_dot_mixed_bwd(float igm1, float rho_ref, float theta_ref, const float *Pi,
                                  const float *Pj, const float *G, const float *ob, float *Pbi,
                                  float *Pbj) {
  const float drho_hat = logmean_minus_ref(rho_ref, Pi[0], Pj[0], Pi[1], Pj[1]);
  const float dilm = inv_logmean_beta_minus_ref(theta_ref, Pi[2], Pj[2]);
  float vs[D];
  float vv = 0.f, gvs = 0.f, gvi = 0.f, gvj = 0.f;
#pragma unroll
  for (int m = 0; m < D; ++m) {
    vs[m] = Pi[3 + m] + Pj[3 + m];
    vv = fmaf(Pi[3 + m], Pj[3 + m], vv);
    gvs = fmaf(G[m], vs[m], gvs);
    gvi = fmaf(G[m], Pi[3 + m], gvi);
    gvj = fmaf(G[m], Pj[3 + m], gvj);
  }
  const float rho_hat = rho_ref + drho_hat;
  const float f0 = 0.5f * rho_hat * gvs;
  const float dC = fmaf(igm1, dilm, 0.5f * vv);
  const float t = 0.5f * f0;
  const float oE = ob[D + 1];
  float ovs = 0.f, pbar_b = 0.f;
#pragma unroll
  for (int m = 0; m < D; ++m) {
    ovs = fmaf(ob[1 + m], vs[m], ovs);
    pbar_b = fmaf(ob[1 + m], G[m], pbar_b);
  }
  const float f0b = fmaf(0.5f, ovs, fmaf(dC, oE, ob[0]));
  const float gvsb = fmaf(0.5f * rho_hat, f0b, -0.5f * theta_ref * drho_hat * oE);
  const float drb = fmaf(0.5f * gvs, f0b, -0.5f * gvs * theta_ref * oE);
  const float dCb = f0 * oE;
  const float vvb = 0.5f * dCb;
  const float gvjb = 0.5f * oE * Pi[3 + D];
  const float gvib = 0.5f * oE * Pj[3 + D];
  float lx, ly, ti, tj;
  logmean_f_grad(Pi[0], Pj[0], &lx, &ly);
  inv_logmean_theta_grad(theta_ref + Pi[2], theta_ref + Pj[2], &ti, &tj);
  Pbi[0] = 0.f;
  Pbj[0] = 0.f;
  Pbi[1] = drb * lx;
  Pbj[1] = drb * ly;
  Pbi[2] = igm1 * dCb * ti;
  Pbj[2] = igm1 * dCb * tj;
  Pbi[3 + D] = fmaf(0.5f * oE, gvj, 0.5f * pbar_b);
  Pbj[3 + D] = fmaf(0.5f * oE, gvi, 0.5f * pbar_b);
#pragma unroll
  for (int m = 0; m < D; ++m) {
    const float vsb = fmaf(t, ob[1 + m], G[m] * gvsb);
    Pbi[3 + m] = fmaf(G[m], gvib, fmaf(Pj[3 + m], vvb, vsb));
    Pbj[3 + m] = fmaf(G[m], gvjb, fmaf(Pi[3 + m], vvb, vsb));
  }
}

// Transpose of euler_prim_mixed: accumulate ub += (dP/du')^T Pb.
template <int D>
SSE_HD void euler_prim_mixed_bwd(float gm1, float theta_ref, const float *P, const float *Pb, float *ub) {
  const float rho = P[0], rr = sse_fdiv(1.f, rho);
  const float theta = theta_ref + P[2];
  const float pb = fmaf(Pb[2], rr, Pb[3 + D]);  // p' cotangent, including theta' = (p_ref + p')/rho - theta_ref
  float v2 = 0.f, vvb = 0.f;
#pragma unroll
  for (int m = 0; m < D; ++m) {
    v2 = fmaf(P[3 + m], P[3 + m], v2);
    vvb = fmaf(Pb[3 + m], P[3 + m], vvb);
  }
  ub[0] += Pb[0] + Pb[1] - Pb[2] * theta * rr + 0.5f * gm1 * pb * v2 - vvb * rr;
#pragma unroll
  for (int m = 0; m < D; ++m) ub[m + 1] += fmaf(-gm1 * pb, P[3 + m], Pb[3 + m] * rr);
  ub[D + 1] += gm1 * pb;
}


// Primitive quantities of one Euler state, computed once per node so that
// the pairwise loops do no per-pair divisions for them.
template <int D>
struct Prim {
  double rho, p, beta;  // beta = rho / p
  double V[D];
};

template <int D>
__device__ __forceinline__ Prim<D> euler_prim(const Physics &ph, const double *u) {
  Prim<D> q;
  q.rho = u[0];
  double s = 0.0;
#pragma unroll
  for (int m = 0; m < D; ++m) q.V[m] = u[m + 1] / u[0];
#pragma unroll
  for (int m = 0; m < D; ++m) s += q.V[m] * q.V[m];
  q.p = ph.gm1 * (u[D + 1] - 0.5 * u[0] * s);
  q.beta = u[0] / q.p;
  return q;
}

// Ranocha's entropy-conservative flux tensor F[e][n] (euler_navierstokes.jl:171-195).
template <int D>
__device__ __forceinline__ void ec_flux(const Physics &ph, const Prim<D> &L, const Prim<D> &R,
                                        double F[D + 2][D]) {
  double rho_avg = logmean(L.rho, R.rho);
  double Vavg[D];
  double vv = 0.0;
#pragma unroll
  for (int m = 0; m < D; ++m) Vavg[m] = 0.5 * (L.V[m] + R.V[m]);
#pragma unroll
  for (int m = 0; m < D; ++m) vv += L.V[m] * R.V[m];
  double pavg = 0.5 * (L.p + R.p);
  double C = 0.5 * vv + ph.igm1 * inv_logmean(L.beta, R.beta);
#pragma unroll
  for (int n = 0; n < D; ++n) {
    double frho = rho_avg * Vavg[n];
    F[0][n] = frho;
#pragma unroll
    for (int m = 0; m < D; ++m) F[m + 1][n] = rho_avg * Vavg[m] * Vavg[n] + (m == n ? pavg : 0.0);
    F[D + 1][n] = frho * C + 0.5 * (L.p * R.V[n] + R.p * L.V[n]);
  }
}

// Euler physical flux tensor (euler_navierstokes.jl:58-68).
template <int D>
__device__ __forceinline__ void euler_flux(const Physics &ph, const double *u, double F[D + 2][D]) {
  double V[D], s = 0.0;
#pragma unroll
  for (int m = 0; m < D; ++m) V[m] = u[m + 1] / u[0];
#pragma unroll
  for (int m = 0; m < D; ++m) s += u[m + 1] * V[m];
  double p = ph.gm1 * (u[D + 1] - 0.5 * s);
  double ht = u[D + 1] + p;
#pragma unroll
  for (int n = 0; n < D; ++n) {
    F[0][n] = u[n + 1];
#pragma unroll
    for (int m = 0; m < D; ++m) F[m + 1][n] = u[m + 1] * V[n] + (m == n ? p : 0.0);
    F[D + 1][n] = ht * V[n];
  }
}

// Chandrashekar (2013), entropy conservative and kinetic-energy preserving:
// with beta = rho / (2 p) and logarithmic means rho_hat, beta_hat,
//   F_rho = rho_hat Vbar_n,  F_m = F_rho Vbar_m + p_hat delta_mn,
//   p_hat = avg(rho) / (2 avg(beta)),
//   F_E = F_rho (1 / (2 (gamma - 1) beta_hat) - avg(|V|^2) / 2) + F_m . Vbar.
template <int D>
__device__ __forceinline__ void chandrashekar_flux(const Physics &ph, const double *uL, const double *uR,
                                                   double F[D + 2][D]) {
  double VL[D], VR[D], sL = 0.0, sR = 0.0;
#pragma unroll
  for (int m = 0; m < D; ++m) {
    VL[m] = uL[m + 1] / uL[0];
    VR[m] = uR[m + 1] / uR[0];
    sL += VL[m] * VL[m];
    sR += VR[m] * VR[m];
  }
  const double pL = ph.gm1 * (uL[D + 1] - 0.5 * uL[0] * sL);
  const double pR = ph.gm1 * (uR[D + 1] - 0.5 * uR[0] * sR);
  const double bL = uL[0] / (2.0 * pL), bR = uR[0] / (2.0 * pR);
  const double rho_hat = logmean(uL[0], uR[0]);
  const double beta_hat = logmean(bL, bR);
  const double p_hat = 0.5 * (uL[0] + uR[0]) / (bL + bR);
  const double v2avg = 0.5 * (sL + sR);
  const double h = 1.0 / (2.0 * ph.gm1 * beta_hat) - 0.5 * v2avg;
  double Vb[D];
#pragma unroll
  for (int m = 0; m < D; ++m) Vb[m] = 0.5 * (VL[m] + VR[m]);
#pragma unroll
  for (int n = 0; n < D; ++n) {
    const double frho = rho_hat * Vb[n];
    F[0][n] = frho;
    double fe = frho * h;
#pragma unroll
    for (int m = 0; m < D; ++m) {
      const double fm = frho * Vb[m] + (m == n ? p_hat : 0.0);
      F[m + 1][n] = fm;
      fe += fm * Vb[m];
    }
    F[D + 1][n] = fe;
  }
}

// Two-point flux tensor for a pair of states: Euler EC (Ranocha),
// Chandrashekar or conservative average, or advection a_m (u_L + u_R)/2.
template <int D, int NC>
__device__ __forceinline__ void two_point(const Physics &ph, const double *uL, const double *uR,
                                          double F[NC][D]) {
  if constexpr (NC == 1) {
    double f1 = 0.5 * (uL[0] + uR[0]);
#pragma unroll
    for (int m = 0; m < D; ++m) F[0][m] = ph.a[m] * f1;
  } else {
    if (ph.ec) {
      Prim<D> L = euler_prim<D>(ph, uL), R = euler_prim<D>(ph, uR);
      ec_flux<D>(ph, L, R, F);
    } else if (ph.chandrashekar) {
      chandrashekar_flux<D>(ph, uL, uR, F);
    } else {
      double FL[D + 2][D], FR[D + 2][D];
      euler_flux<D>(ph, uL, FL);
      euler_flux<D>(ph, uR, FR);
#pragma unroll
      for (int e = 0; e < D + 2; ++e)
#pragma unroll
        for (int n = 0; n < D; ++n) F[e][n] = 0.5 * (FL[e][n] + FR[e][n]);
    }
  }
}

// wave_speed (euler_navierstokes.jl:133-150; linear_advection_diffusion.jl:106-111)
template <int D, int NC>
__device__ __forceinline__ double wave_speed(const Physics &ph, const double *ui, const double *uo,
                                             const double *n) {
  if constexpr (NC == 1) {
    double s = 0.0;
#pragma unroll
    for (int m = 0; m < D; ++m) s += ph.a[m] * n[m];
    return fabs(s);
  } else {
    double si = 0.0, so = 0.0, vni = 0.0, vno = 0.0;
#pragma unroll
    for (int m = 0; m < D; ++m) { si += ui[m + 1] * ui[m + 1]; so += uo[m + 1] * uo[m + 1]; }
    double pin = ph.gm1 * (ui[D + 1] - (0.5 / ui[0]) * si);
    double pout = ph.gm1 * (uo[D + 1] - (0.5 / uo[0]) * so);
#pragma unroll
    for (int m = 0; m < D; ++m) { vni += (ui[m + 1] / ui[0]) * n[m]; vno += (uo[m + 1] / uo[0]) * n[m]; }
    double ci = sqrt(ph.gamma * pin / ui[0]);
    double co = sqrt(ph.gamma * pout / uo[0]);
    return fmax(fabs(vni), fabs(vno)) + fmax(ci, co);
  }
}

// conservative_to_entropy! (euler_navierstokes.jl:100-113)
template <int D>
__device__ __forceinline__ void cons_to_entropy(const Physics &ph, const double *u, double *w) {
  double s = 0.0;
#pragma unroll
  for (int m = 0; m < D; ++m) s += u[m + 1] * u[m + 1];
  double k = (0.5 / u[0]) * s;
  double p = ph.gm1 * (u[D + 1] - k);
  double ip = 1.0 / p;
  w[0] = ph.igm1 * (ph.gamma - log(p / pow(u[0], ph.gamma))) - k * ip;
#pragma unroll
  for (int m = 0; m < D; ++m) w[m + 1] = u[m + 1] * ip;
  w[D + 1] = -u[0] * ip;
}

// entropy_to_conservative! (euler_navierstokes.jl:115-131)
template <int D>
__device__ __forceinline__ void entropy_to_cons(const Physics &ph, const double *w_in, double *u) {
  double w[D + 2];
#pragma unroll
  for (int e = 0; e < D + 2; ++e) w[e] = w_in[e] * ph.gm1;
  double s = 0.0;
#pragma unroll
  for (int m = 0; m < D; ++m) s += w[m + 1] * w[m + 1];
  double k = s / (2 * w[D + 1]);
  double sv = ph.gamma - w[0] + k;
  double rhoe = pow(ph.gm1 / pow(-w[D + 1], ph.gamma), ph.igm1) * exp(-sv * ph.igm1);
  u[0] = -w[D + 1] * rhoe;
#pragma unroll
  for (int m = 0; m < D; ++m) u[m + 1] = w[m + 1] * rhoe;
  u[D + 1] = rhoe * (1 - k);
}

}  // namespace sse
