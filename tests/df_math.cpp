// Host harness of tests/test_df_math.py: the float-pair code of st_df.cuh
// against 128-bit arithmetic.  Prints one line of numbers per quantity.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>
#if defined(__x86_64__)
#include <quadmath.h>
typedef __float128 Q;
static Q sqrt_(Q x) { return sqrtq(x); }
static Q exp_(Q x) { return expq(x); }
static Q log_(Q x) { return logq(x); }
static Q atan2_(Q y, Q x) { return atan2q(y, x); }
#else
typedef long double Q;  // IEEE quad on aarch64
static Q sqrt_(Q x) { return sqrtl(x); }
static Q exp_(Q x) { return expl(x); }
static Q log_(Q x) { return logl(x); }
static Q atan2_(Q y, Q x) { return atan2l(y, x); }
#endif
static double sqrt_(double x) { return std::sqrt(x); }
#include "../spacetime_gb300/csrc/st_df.cuh"

using namespace st;
namespace D = st::dfm;

static df2 pair(Q v) {
  const float h = (float)v;
  return df2{h, (float)(v - (Q)h)};
}
static Q val(df2 x) { return (Q)x.hi + (Q)x.lo; }
static Q val(D::f3 x) { return (Q)x.h + (Q)x.m + (Q)x.l; }
static D::f3 limbs(double v) {
  const float h = (float)v, m = (float)(v - (double)h);
  return D::f3{h, m, (float)(v - (double)h - (double)m)};
}

// The Kerr slopes term by term, M = 1.
template <class T>
static void slopes(const T* s, T pt, T a, T* d) {
  const T x = s[0], y = s[1], z = s[2], px = s[3], py = s[4], pz = s[5], a2 = a * a, z2 = z * z;
  const T w = x * x + y * y + z * z - a2, r2 = T(0.5) * (w + sqrt_(w * w + T(4) * a2 * z2)), r = sqrt_(r2);
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
static void step(T* y, T pt, T a) {
  T c = T(0.16) * sqrt_(y[0] * y[0] + y[1] * y[1] + y[2] * y[2]);
  c = c < T(1) ? T(1) : (c > T(8) ? T(8) : c);
  const T h = T(0.02) * c;
  T k[4][6], t[6];
  slopes(y, pt, a, k[0]);
  for (int s = 1; s < 4; ++s) {
    for (int i = 0; i < 6; ++i) t[i] = y[i] + (s < 3 ? h / 2 : h) * k[s - 1][i];
    slopes(t, pt, a, k[s]);
  }
  for (int i = 0; i < 6; ++i) y[i] += h / 6 * (k[0][i] + 2 * k[1][i] + 2 * k[2][i] + k[3][i]);
}

template <int KERR>
static void step_pairs(D::t3* P, D::t3* Qm, D::t3* W, df2 pt, const D::Hole& H) {
  dd iP, iQ, iW;
  df2 h;
  D::rk4<KERR>(
      *P, *Qm, *W, pt, H,
      [](const D::Geo& g, df2* hh) {
        const df2 c = D::mul(pair((Q)0.16), D::sqrt_(g.flat2));
        *hh = D::mul(pair((Q)0.02), D::min_(D::max_(c, D::q(1)), D::q(8)));
        return false;
      },
      [](const dd&, const dd&) {}, &h, &iP, &iQ, &iW);
  *P = D::add3(*P, iP); *Qm = D::add3(*Qm, iQ); *W = D::add3(*W, iW);
}

static double U() { return (rand() + rand() / (RAND_MAX + 1.0)) / (RAND_MAX + 1.0); }

// Exit errors (direction, and position across the ray over the escape radius)
// of rays from a camera at 15 M, 80 degrees, spin a.
template <int KERR>
static void rays(double a, int n) {
  std::vector<double> ed, ep;
  for (int it = 0; it < n; ++it) {
    const double th = 80 * M_PI / 180, r0 = 15;
    double s[6] = {std::sqrt(r0 * r0 + a * a) * std::sin(th), 0, r0 * std::cos(th)};
    const double m = std::sqrt(s[0] * s[0] + s[2] * s[2]), f[3] = {-s[0] / m, 0, -s[2] / m};
    const double u = 1.95 * (U() - 0.5), v = 1.12 * (U() - 0.5);
    double d[3] = {f[0] - v * f[2], u, f[2] + v * f[0]};
    const double dn = std::sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
    for (int k = 0; k < 3; ++k) s[3 + k] = d[k] / dn;
    // p_t of the null ray
    Q x = s[0], z = s[2], A = a, w = x * x + z * z - A * A, r2 = (w + sqrt_(w * w + 4 * A * A * z * z)) / 2, r = sqrt_(r2);
    const Q l[3] = {r * x / (r2 + A * A), -A * x / (r2 + A * A), z / r}, ff = 2 * r2 * r / (r2 * r2 + A * A * z * z);
    const Q lp = l[0] * s[3] + l[1] * s[4] + l[2] * s[5], p2 = (Q)s[3] * s[3] + (Q)s[4] * s[4] + (Q)s[5] * s[5];
    const Q b = -2 * ff * lp, c = ff * lp * lp - p2;
    const double pt = (double)((-b - sqrt_(b * b - 4 * (1 + ff) * c)) / (2 * (1 + ff)));
    Q yq[6];
    double yd[6];
    for (int k = 0; k < 6; ++k) { yq[k] = s[k]; yd[k] = s[k]; }
    D::t3 P = D::two(limbs(s[0]), limbs(s[1])), M = D::two(limbs(s[3]), limbs(s[4])), W = D::two(limbs(s[2]), limbs(s[5]));
    const D::Hole H{pair((Q)1), pair((Q)a), pair((Q)a * a)};
    bool out = false;
    for (int k = 0; k < 4800; ++k) {
      const double rr = (double)sqrt_(yq[0] * yq[0] + yq[1] * yq[1] + yq[2] * yq[2]);
      if (rr > 30) { out = true; break; }
      if (rr < (KERR ? 1.6 : 2.9)) break;
      step<Q>(yq, (Q)pt, (Q)a);
      step<double>(yd, pt, a);
      step_pairs<KERR>(&P, &M, &W, pair((Q)pt), H);
    }
    if (!out) continue;
    const Q yp[6] = {val(D::fst(P)), val(D::snd(P)), val(D::fst(W)), val(D::fst(M)), val(D::snd(M)), val(D::snd(W))};
    auto err = [&](auto get) {
      Q np = 0, nq = 0, e = 0, al = 0, dd_ = 0;
      for (int k = 3; k < 6; ++k) { np += get(k) * get(k); nq += yq[k] * yq[k]; }
      np = sqrt_(np); nq = sqrt_(nq);
      for (int k = 0; k < 3; ++k) {
        const Q t = get(3 + k) / np - yq[3 + k] / nq, dx = get(k) - yq[k];
        e += t * t; al += dx * yq[3 + k] / nq; dd_ += dx * dx;
      }
      const Q across = dd_ - al * al;
      return (double)sqrt_(e) + (across > 0 ? (double)sqrt_(across) / 30 : 0.0);
    };
    ed.push_back(err([&](int k) { return (Q)yd[k]; }));
    ep.push_back(err([&](int k) { return yp[k]; }));
  }
  std::sort(ed.begin(), ed.end());
  std::sort(ep.begin(), ep.end());
  const size_t c = ed.size();
  printf("rays %g %zu %g %g %g %g\n", a, c, ed[c / 2], ep[c / 2], ed[c * 9 / 10], ep[c * 9 / 10]);
}

int main() {
  srand(1);
  rays<1>(0.9, 250);
  rays<1>(0.99, 250);
  rays<1>(0.3, 250);
  rays<0>(0.0, 250);
  double e[3] = {0, 0, 0};
  for (int i = 0; i < 200000; ++i) {
    df2 x = pair((Q)(U() * 120 - 40));
    e[0] = std::max(e[0], std::fabs((double)(val(D::sh::exp_(x)) / exp_(val(x)) - 1)));
    x = pair((Q)std::exp(U() * 40 - 20));
    e[1] = std::max(e[1], std::fabs((double)(val(D::sh::log_(x)) - log_(val(x)))));
    df2 y = pair((Q)(U() * 40 - 20));
    x = pair((Q)(U() * 40 - 20));
    if (i % 4 == 0) y = pair(val(y) * 1e-6);
    if (i % 4 == 1) x = pair(val(x) * 1e-4);
    e[2] = std::max(e[2], std::fabs((double)(val(D::sh::atan2_(y, x)) - atan2_(val(y), val(x)))));
  }
  printf("exp %g log %g atan2 %g\n", e[0], e[1], e[2]);
  return 0;
}
