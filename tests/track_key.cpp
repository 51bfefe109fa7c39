// Host harness of tests/test_track_key.py: the launch block of a camera track for
// cameras at different places.  Prints whether the two blocks are equal and the
// flag of the pair kernel's range, a line for each pair of radii.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "../spacetime_gb300/csrc/st_internal.h"

static st::TraceParams block(const st::TraceParams& rules, double r, int n) {
  st::TraceParams p = rules;
  st::FrameCam fc[8] = {};
  for (int f = 0; f < n; ++f) {
    fc[f].r_escape = r * (1.0 + 0.01 * f);
    fc[f].nmax = rules.nmax;
  }
  // the first camera's own fields, as the render call fills them
  p.pos[0] = -r / 2;
  p.pos[2] = r / 7;
  for (int k = 0; k < 4; ++k) { p.Ef[k] = 1 / r; p.Er[k] = k / r; p.Eu[k] = -1 / r; p.U[k] = 1 + 1 / r; }
  p.r_escape = fc[0].r_escape;
  st::use_frame_table(&p, fc, n);
  return p;
}

int main(int argc, char** argv) {
  st::TraceParams rules;
  std::memset(&rules, 0, sizeof rules);
  rules.M = 1.0;
  rules.dt = 0.02;
  rules.nmax = 4000;
  for (int i = 1; i + 1 < argc; i += 2) {
    const st::TraceParams a = block(rules, std::atof(argv[i]), 4), b = block(rules, std::atof(argv[i + 1]), 4);
    printf("%d %d %d\n", std::memcmp(&a, &b, sizeof a) == 0, a.pair_range, b.pair_range);
  }
  return 0;
}
