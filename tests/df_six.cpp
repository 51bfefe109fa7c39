// Host harness of tests/test_df_guard.py: the guard step component by component
// (rk4_six) against the packed form (rk4), bit for bit, along rays of a camera at 15 M.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "../spacetime_gb300/csrc/st_df.cuh"

using namespace st;
namespace D = st::dfm;

static double U() { return (rand() + rand() / (RAND_MAX + 1.0)) / (RAND_MAX + 1.0); }

template <int KERR>
static void run(double a, int n) {
  long differ = 0, steps = 0;
  for (int it = 0; it < n; ++it) {
    const double th = 80 * M_PI / 180, r0 = 15;
    df2 y[6] = {D::pair_of(std::sqrt(r0 * r0 + a * a) * std::sin(th)), D::q(0.f), D::pair_of(r0 * std::cos(th))};
    double d[3] = {-1, 1.95 * (U() - 0.5), 1.12 * (U() - 0.5)};
    const double dn = std::sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
    for (int k = 0; k < 3; ++k) y[3 + k] = D::pair_of(d[k] / dn);
    const df2 pt = D::q(-0.93f);
    const D::Hole H{D::q(1.f), D::pair_of(a), D::pair_of(a * a)};
    for (int k = 0; k < 2000; ++k) {
      const float r = std::sqrt(y[0].hi * y[0].hi + y[1].hi * y[1].hi + y[2].hi * y[2].hi);
      if (!(r < 30.f && r > 1.2f)) break;
      const df2 h = D::q(0.02f * std::fmin(std::fmax(0.16f * r, 1.f), 8.f));
      df2 inc[6];
      D::rk4_six<KERR>(y, pt, H, h, inc);
      const v2 zero = D::mkv(0.f, 0.f);
      const D::t3 P{D::mkv(y[0].hi, y[1].hi), D::mkv(y[0].lo, y[1].lo), zero};
      const D::t3 M{D::mkv(y[3].hi, y[4].hi), D::mkv(y[3].lo, y[4].lo), zero};
      const D::t3 W{D::mkv(y[2].hi, y[5].hi), D::mkv(y[2].lo, y[5].lo), zero};
      dd iP, iQ, iW;
      df2 hh;
      D::rk4<KERR>(
          P, M, W, pt, H, [&](const D::Geo&, df2* o) { *o = h; return false; }, [](const dd&, const dd&) {}, &hh, &iP,
          &iQ, &iW);
      const df2 packed[6] = {D::fst(iP), D::snd(iP), D::fst(iW), D::fst(iQ), D::snd(iQ), D::snd(iW)};
      differ += std::memcmp(packed, inc, sizeof inc) != 0;
      ++steps;
      for (int c = 0; c < 6; ++c) y[c] = D::add(y[c], inc[c]);
    }
  }
  printf("%g %ld %ld\n", a, steps, differ);
}

int main() {
  srand(3);
  run<1>(0.9, 40);
  run<1>(-0.99, 40);
  run<1>(1e-6, 40);
  run<0>(0.0, 40);
  return 0;
}
