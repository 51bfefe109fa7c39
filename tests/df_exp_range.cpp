// Host harness of tests/test_df_range.py: the shading exponential of st_df.cuh
// over every optical depth.  Prints x, exp_(x) as hi and lo, and the blend of one
// sample of unit radiance: its emission and the transmittance behind it.
#include <cstdio>
#include <cstdlib>
#include "../spacetime_gb300/csrc/st_df.cuh"

using namespace st;
namespace S = st::dfm::sh;

int main(int argc, char** argv) {
  for (int i = 1; i < argc; ++i) {
    const double x = std::atof(argv[i]);
    const float h = (float)x;
    const df2 e = S::exp_(df2{h, std::isfinite(x) ? (float)(x - (double)h) : 0.f});
    const df2 w = S::addf(dfm::neg(e), 1.f);
    printf("%.17g %.17g %.17g %.17g %.17g\n", x, e.hi, e.lo, w.hi + w.lo, e.hi + e.lo);
  }
  return 0;
}
