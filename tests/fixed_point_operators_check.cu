// Host-side check of the scaling of fixed-point operator rows
// (sse_fixed_ops.cuh): entries next to a power of two, alone in their row or
// not, must come back from their integers as they went in.  Built and run by
// tests/test_fixed_point_operators.py with nvcc; needs no GPU.
#include <cmath>
#include <cstdio>
#include <initializer_list>

#include "../cloud.jl_gb300/csrc/sse_fixed_ops.cuh"

using namespace sse;

int main() {
  long long bad = 0;
  for (int e = -30; e <= 30; ++e)
    for (double x : {1.0, 0.75, 0.5, std::nextafter(1.0, 0.0), std::nextafter(1.0, 2.0), 1.0 - 0x1p-40, 1.0 - 0x1p-33,
                     1.0 - 0x1p-32, 1.0 - 0x1p-31, 1.0 - 0x1p-20})
      for (double other : {0.0, 0x1p-45, 0x1p-33})
        for (double sign : {1.0, -1.0}) {
          const double v = std::ldexp(sign * x, e), row = std::ldexp(x + other, e);
          const int unit = fo_row_exponent(row);
          const Fx a = fo_from_double(v, unit);
          // 62 fraction bits hold every bit of an entry within 2^-8 of the unit
          bad += std::ldexp((double)a.hi * 0x1p31 + a.lo, unit - 62) != v;
          bad += std::fabs(v) > std::ldexp(1.0, unit) || row < std::ldexp(0.49, unit);
        }
  printf("{\"mismatches\": %lld}\n", bad);
  return 0;
}
