// Host harness of tests/test_df_guard.py: the guarded path's step (rk4_six, add_rn)
// on its state of two floats a component, and the same step formed in double on
// that state, both measured from 128-bit arithmetic.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>
#if defined(__x86_64__)
#include <quadmath.h>
typedef __float128 Q;
static Q sqrt_(Q x) { return sqrtq(x); }
#else
typedef long double Q;  // IEEE quad on aarch64
static Q sqrt_(Q x) { return sqrtl(x); }
#endif
static double sqrt_(double x) { return std::sqrt(x); }
#include "../spacetime_gb300/csrc/st_df.cuh"

using namespace st;
namespace D = st::dfm;

static df2 pair(Q v) {
  const float h = (float)v;
  return df2{h, (float)(v - (Q)h)};
}
static double U() { return (rand() + rand() / (RAND_MAX + 1.0)) / (RAND_MAX + 1.0); }

// Kerr slopes term by term, M = 1.
template <class T>
static void slopes(const T* s, T pt, T a, T* d) {
  const T x = s[0], y = s[1], z = s[2], px = s[3], py = s[4], pz = s[5], a2 = a * a, z2 = z * z;
  const T w = x * x + y * y + z2 - a2, r2 = T(0.5) * (w + sqrt_(w * w + T(4) * a2 * z2)), r = sqrt_(r2);
  const T ir = T(1) / r, r3 = r2 * r, is = T(1) / (r2 * r2 + a2 * z2), r2a = r2 + a2, ira = T(1) / r2a;
  const T Lx = (r * x + a * y) * ira, Ly = (r * y - a * x) * ira, Lz = z * ir;
  const T l = -pt + Lx * px + Ly * py + Lz * pz, f = T(2) * r3 * is, fl = f * l;
  const T drx = x * r3 * is, dry = y * r3 * is, drz = z * r * r2a * is;
  const T dfdr = T(2) * r2 * (T(3) * a2 * z2 - r2 * r2) * is * is, dfz = T(-4) * r3 * a2 * z * is * is;
  const T dlx = (r * px - a * py) * ira, dly = (a * px + r * py) * ira, dlz = pz * ir;
  const T dl = (px * (x * r2a - T(2) * r * (r * x + a * y)) + py * (y * r2a - T(2) * r * (r * y - a * x))) * ira * ira -
               z * pz * ir * ir;
  const T h = T(0.5) * l * l;
  d[0] = px - fl * Lx; d[1] = py - fl * Ly; d[2] = pz - fl * Lz;
  d[3] = h * (dfdr * drx) + fl * (dl * drx + dlx);
  d[4] = h * (dfdr * dry) + fl * (dl * dry + dly);
  d[5] = h * (dfdr * drz + dfz) + fl * (dl * drz + dlz);
}
template <class T>
static void step(T* y, T pt, T a, T h) {
  T k[4][6], t[6];
  slopes(y, pt, a, k[0]);
  for (int s = 1; s < 4; ++s) {
    for (int i = 0; i < 6; ++i) t[i] = y[i] + (s < 3 ? h / 2 : h) * k[s - 1][i];
    slopes(t, pt, a, k[s]);
  }
  for (int i = 0; i < 6; ++i) y[i] += h / 6 * (k[0][i] + 2 * k[1][i] + 2 * k[2][i] + k[3][i]);
}

static void ray(double a, double* s, double* pt) {
  const double th = 80 * M_PI / 180, r0 = 15;
  s[0] = std::sqrt(r0 * r0 + a * a) * std::sin(th); s[1] = 0; s[2] = r0 * std::cos(th);
  const double m = std::sqrt(s[0] * s[0] + s[2] * s[2]), f[3] = {-s[0] / m, 0, -s[2] / m};
  const double u = 1.95 * (U() - 0.5), v = 1.12 * (U() - 0.5);
  const double d[3] = {f[0] - v * f[2], u, f[2] + v * f[0]};
  const double dn = std::sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
  for (int k = 0; k < 3; ++k) s[3 + k] = d[k] / dn;
  const Q x = s[0], z = s[2], A = a, w = x * x + z * z - A * A, r2 = (w + sqrt_(w * w + 4 * A * A * z * z)) / 2,
          r = sqrt_(r2);
  const Q l[3] = {r * x / (r2 + A * A), -A * x / (r2 + A * A), z / r}, ff = 2 * r2 * r / (r2 * r2 + A * A * z * z);
  const Q lp = l[0] * s[3] + l[1] * s[4] + l[2] * s[5], p2 = (Q)s[3] * s[3] + (Q)s[4] * s[4] + (Q)s[5] * s[5];
  const Q b = -2 * ff * lp, c = ff * lp * lp - p2;
  *pt = (double)(float)((-b - sqrt_(b * b - 4 * (1 + ff) * c)) / (2 * (1 + ff)));  // a float, as the kernel's
}

template <int KERR>
static void run(double a, int n) {
  std::vector<double> ed, ep;
  for (int it = 0; it < n; ++it) {
    double s[6], pt;
    ray(a, s, &pt);
    const D::Hole H{pair((Q)1), pair((Q)a), pair((Q)a * a)};
    Q yq[6];
    df2 yd[6], yp[6];
    for (int k = 0; k < 6; ++k) { yd[k] = yp[k] = pair((Q)s[k]); yq[k] = (Q)yp[k].hi + (Q)yp[k].lo; }
    bool out = false;
    for (int k = 0; k < 4800; ++k) {
      const double rr = (double)sqrt_(yq[0] * yq[0] + yq[1] * yq[1] + yq[2] * yq[2]);
      if (rr > 30) { out = true; break; }
      if (rr < (KERR ? 1.6 : 2.9)) break;
      const float h = 0.02f * (float)std::min(std::max(0.16 * rr, 1.0), 8.0);
      step<Q>(yq, (Q)pt, (Q)a, (Q)h);
      // in double, rounded to the state's two floats
      double t[6];
      for (int c = 0; c < 6; ++c) t[c] = (double)yd[c].hi + (double)yd[c].lo;
      step<double>(t, pt, a, (double)h);
      for (int c = 0; c < 6; ++c) yd[c] = pair((Q)t[c]);
      // in pairs
      df2 inc[6];
      D::rk4_six<KERR>(yp, pair((Q)pt), H, D::q(h), inc);
      for (int c = 0; c < 6; ++c) yp[c] = D::add_rn(yp[c], inc[c]);
    }
    if (!out) continue;
    auto err = [&](const df2* y) {
      Q np = 0, nq = 0, e = 0;
      for (int k = 3; k < 6; ++k) { const Q v = (Q)y[k].hi + (Q)y[k].lo; np += v * v; nq += yq[k] * yq[k]; }
      np = sqrt_(np); nq = sqrt_(nq);
      for (int k = 3; k < 6; ++k) { const Q t = ((Q)y[k].hi + (Q)y[k].lo) / np - yq[k] / nq; e += t * t; }
      return (double)sqrt_(e);
    };
    ed.push_back(err(yd));
    ep.push_back(err(yp));
  }
  std::sort(ed.begin(), ed.end());
  std::sort(ep.begin(), ep.end());
  const size_t c = ed.size();
  printf("%g %zu %g %g\n", a, c, ed[c / 2], ep[c / 2]);
}

int main() {
  srand(3);
  run<1>(0.9, 300);
  run<1>(0.99, 300);
  run<1>(0.3, 300);
  run<0>(0.0, 300);
  return 0;
}
