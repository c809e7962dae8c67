// Host check of sinf_cr, logf_cr and powf_cr where their results lie next to a
// power of two (the floats below it are twice as dense, which the rounding
// test must know) and of the sine's float-float series over (2^-30, 1.6]:
// correctly rounded, and within 1e-13 of the series' exact value.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include "../../wrf_gb300/csrc/ffmath.h"

using namespace wrfgpu_ff;

int main() {
  long n = 0, bad = 0;
  double maxe = 0.0;
  for (int which = 0; which < 3; ++which)
    for (int e = -20; e <= 1; ++e) {
      const double p = std::ldexp(1.0, e);
      if (which == 0 && e > 0) continue;
      const double x0 = which == 0 ? std::asin(p) : which == 1 ? std::exp(p) : std::pow(p, 1.0 / 1.4);
      const uint32_t u0 = f2u((float)x0);
      for (int d = -40000; d <= 40000; ++d) {
        const float x = u2f(u0 + (uint32_t)d);
        if (which == 0 && !(x > 0.f && x <= 1.5707964f)) continue;
        const float r = which == 0 ? sinf_cr(x) : which == 1 ? logf_cr(x) : powf_cr(x, 1.4f);
        const long double ex = which == 0 ? sinl((long double)x)
                               : which == 1 ? logl((long double)x) : powl((long double)x, (long double)1.4f);
        ++n;
        bad += r != (float)ex;
      }
    }
  for (uint32_t u = f2u(0x1p-30f); u <= f2u(1.6f); u += 101) {
    const float x = u2f(u);
    const ff v = ff_sin_t(x);
    const long double ex = sinl((long double)x);
    const double err = (double)fabsl(((long double)v.hi + (long double)v.lo - ex) / ex);
    maxe = err > maxe ? err : maxe;
    ++n;
    bad += sinf_cr(x) != (float)ex;
  }
  std::printf("%ld points, %ld mismatches, series error %.2e\n", n, bad, maxe);
  return bad || maxe > 1e-13;
}
