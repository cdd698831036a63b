// Host-side check of the block fixed-point arithmetic (sse_fixed.cuh) against
// long double: the two means near and far from their branch points, the
// entropy-conservative flux over Mach numbers and jumps, and conversions.
// Built and run by tests/test_fixed_point.py with nvcc; needs no GPU.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>

#include "../cloud.jl_gb300/csrc/sse_fixed.cuh"

using namespace sse;
typedef long double LD;

static LD ref_logmean(LD x, LD y) {
  const LD f = (x - y) / (x + y), z = f * f;
  if (z < 1e-3L) {
    LD s = 0;
    for (int k = 14; k >= 1; --k) s = (s + 1.0L / (2 * k + 1)) * z;
    return (x + y) / 2 / (1 + s);
  }
  return (x - y) / logl(x / y);
}

// P: rho, p, V; G halved (ec_flux_dot_half)
template <int D>
static void ref_flux(LD gamma, const double *Pi, const double *Pj, const double *G, LD *out) {
  const LD rh = ref_logmean(Pi[0], Pj[0]);
  const LD lb = ref_logmean((LD)Pi[0] / Pi[1], (LD)Pj[0] / Pj[1]);
  LD vv = 0, gi = 0, gj = 0;
  for (int m = 0; m < D; ++m) {
    vv += (LD)Pi[2 + m] * Pj[2 + m];
    gi += (LD)G[m] * Pi[2 + m];
    gj += (LD)G[m] * Pj[2 + m];
  }
  const LD f0 = rh * (gi + gj);
  out[0] = f0;
  for (int m = 0; m < D; ++m) out[1 + m] = f0 / 2 * ((LD)Pi[2 + m] + Pj[2 + m]) + ((LD)Pi[1] + Pj[1]) * G[m];
  out[D + 1] = f0 / 2 * vv + f0 / lb / (gamma - 1) + Pi[1] * gj + Pj[1] * gi;
}

// worst ratio, over components, of the fixed-point to the FP64 rms error, and
// the fixed-point rms error relative to the rms flux
template <int D>
static void flux_errors(double gamma, double mach, double amp, double *worst_ratio, double *worst_rel) {
  std::mt19937_64 r(17);
  std::uniform_real_distribution<double> U(-1, 1);
  double ef[D + 2] = {}, ed[D + 2] = {}, mag[D + 2] = {};
  for (int it = 0; it < 20000; ++it) {
    double P[2][2 + D], Q[2][3 + D], G[D], rho = 0, h = 0, v = 0;
    for (int s = 0; s < 2; ++s) {
      P[s][0] = 1 + amp * U(r);
      P[s][1] = (1 + amp * U(r)) / (gamma * mach * mach);
      for (int m = 0; m < D; ++m) P[s][2 + m] = U(r);
      rho = std::max(rho, P[s][0]);
      h = std::max(h, P[s][1] / P[s][0] / (gamma - 1));
      for (int m = 0; m < D; ++m) v = std::max(v, std::fabs(P[s][2 + m]));
    }
    const int eR = std::ilogb(rho) + 2;
    int eV = std::ilogb(v) + 2;
    const int eH = std::max(std::ilogb(h) + 2, 2 * eV);
    eV = std::max(eV, (eH - 40) >> 1);
    const int eP = eR + eH - 2;
    Fx Gx[D], N[2][3 + D];
    FxPair F[2];
    for (int m = 0; m < D; ++m) {
      G[m] = 0.3 * U(r);
      Gx[m] = fx_split(fx_from_double(G[m], 0));
    }
    for (int s = 0; s < 2; ++s) {
      N[s][0] = fx_split_near(fx_from_double(P[s][0], eR));
      N[s][1] = fx_split_near(fx_from_double(P[s][1], eP));
      N[s][2] = fx_split_near(fx_from_double(P[s][1] / P[s][0] / (gamma - 1), eH));
      fx_two_floats(N[s][0], &F[s].rh, &F[s].rl);
      fx_two_floats(N[s][2], &F[s].hh, &F[s].hl);
      Q[s][0] = P[s][0];
      Q[s][1] = P[s][1];
      Q[s][2] = P[s][0] / P[s][1];
      for (int m = 0; m < D; ++m) {
        N[s][3 + m] = fx_split_near(fx_from_double(P[s][2 + m], eV));
        Q[s][3 + m] = P[s][2 + m];
      }
    }
    long long o[D + 2];
    fx_ec_flux<D>(N[0], N[1], F[0], F[1], Gx, eH - 2 * eV, o);
    LD want[D + 2];
    ref_flux<D>(gamma, P[0], P[1], G, want);
    const double ig = 1 / (gamma - 1), q[4] = {ig * 2, ig * 2 / 3, ig * 0.4, ig * 2 / 7};
    double d[D + 2];
    ec_flux_dot_half<D>(ig, q, Q[0], Q[1], G, d);
    for (int e = 0; e < D + 2; ++e) {
      const int unit = e == 0 ? eR + eV - 63 : (e <= D ? eP - 61 : eP + eV - 61);
      const LD a = (LD)o[e] * ldexpl(1, unit) - want[e], b = (LD)d[e] - want[e];
      ef[e] += (double)(a * a);
      ed[e] += (double)(b * b);
      mag[e] += (double)(want[e] * want[e]);
    }
  }
  for (int e = 0; e < D + 2; ++e) {
    *worst_ratio = std::max(*worst_ratio, std::sqrt(ef[e] / ed[e]));
    *worst_rel = std::max(*worst_rel, std::sqrt(ef[e] / mag[e]));
  }
}

template <int KIND>
static double mean_error(double amp) {
  std::mt19937_64 r(3);
  std::uniform_real_distribution<double> U(-1, 1);
  double worst = 0;
  for (int it = 0; it < 200000; ++it) {
    // around a power of two, where a sum changes its exponent
    const double x = 0.25 * (1 + amp * U(r)), y = 0.25 * (1 + amp * U(r));
    const Fx X = fx_split_near(fx_from_double(x, 0)), Y = fx_split_near(fx_from_double(y, 0));
    FxPair a, b;
    fx_two_floats(X, &a.rh, &a.rl);
    fx_two_floats(Y, &b.rh, &b.rl);
    Fx c;
    const float z = fx_mean_correction<KIND>(a.rh, a.rl, b.rh, b.rl, &c);
    LD got = (LD)x + y - (c.hi * 0x1p-30L + c.lo * 0x1p-60L);
    if (!(z < 1.0e-4f)) got = fx_join(fx_mean_slow(X, Y, KIND)) * 0x1p-60L;
    const LD L = ref_logmean(x, y), want = KIND == 0 ? 2 * L : 2 * (LD)x * y / L;
    worst = std::max(worst, (double)(fabsl(got - want) / want));
  }
  return worst;
}

int main() {
  double ratio = 0, rel = 0;
  for (double gamma : {1.4, 5.0 / 3.0})
    for (double mach : {1e-3, 0.1, 0.8, 3.0})
      for (double amp : {1e-5, 3e-3, 1.2e-2, 0.1, 0.4}) {
        flux_errors<2>(gamma, mach, amp, &ratio, &rel);
        flux_errors<3>(gamma, mach, amp, &ratio, &rel);
      }
  double mean = 0;
  for (double amp : {1e-6, 1e-3, 1.2e-2, 0.1, 0.25, 0.6})
    mean = std::max({mean, mean_error<0>(amp), mean_error<1>(amp)});
  // conversions: exact for values within 2^7 of the unit, zero and signs kept
  long long bad = 0;
  std::mt19937_64 r(9);
  std::uniform_real_distribution<double> U(-1, 1);
  for (int it = 0; it < 100000; ++it) {
    const double x = U(r);
    const long long v = fx_from_double(x, 1);
    const Fx a = fx_split(v), b = fx_split_near(v);
    bad += std::fabs(x) > 0x1p-7 && (LD)v != (LD)x * 0x1p59L;
    bad += fx_join(a) != v || fx_join(b) != v || a.lo < 0 || b.lo < -(1 << 29) || b.lo >= (1 << 29);
    bad += fx_from_double(-x, 1) != -v;
  }
  bad += fx_from_double(0.0, 0) != 0 || fx_from_double(-0.0, 3) != 0 || fx_from_double(1e-300, 0) != 0;
  printf("{\"flux_error_ratio\": %.3f, \"flux_relative\": %.3e, \"mean\": %.3e, \"conversion_mismatches\": %lld}\n", ratio,
         rel, mean, bad);
  return 0;
}
