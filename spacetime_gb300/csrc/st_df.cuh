// st_df.cuh -- float-pair ("double-float") arithmetic on the FP32 pipe, and
// the geodesic right-hand sides, state and shading functions built on it.
//
// Why: a GB300 SM issues a warp's double operation every 19 cycles (measured:
// dependent chains of fma on 4 and 16 warps per SM, whatever the number of
// active lanes), a float operation four times a cycle.  A pair operation of 8
// to 19 float instructions is therefore 4 to 9 times cheaper than the double
// operation it stands for.
//
// Precision: a value is hi + lo with |lo| <= ulp(hi) (about 48 bits).  An
// integration that forms its slopes in pairs and keeps its state in three
// floats (72 bits) is closer to the exact RK4 sequence than one all in double:
// the step h ~ 0.02-0.16 takes the slopes' 2^-48 below the 2^-53 with which a
// double state is rounded at every step.  tests/test_df_math.py measures both
// against 128-bit arithmetic over cameras and spins.
//
// The file compiles on the host too (no CUDA header), for that test; there
// the hardware's reciprocal seeds are plain divisions, and the file wants
// -ffp-contract=off.  On the device every operation is a rounded intrinsic, so
// no contraction and no fast-math flag of the unit touches it.
#pragma once

#include <math.h>

#ifdef __CUDACC__
#define ST_DF __device__ __forceinline__
#else
#define ST_DF inline
#endif

namespace st {

struct df2 {
  float hi, lo;
};

#ifdef __CUDACC__
typedef float2 v2;
#else
struct v2 {
  float x, y;
};
#endif
// two pairs: (h.x, l.x) and (h.y, l.y)
struct dd {
  v2 h, l;
};

namespace dfm {

#ifdef __CUDA_ARCH__
ST_DF float fadd(float a, float b) { return __fadd_rn(a, b); }
ST_DF float fsub(float a, float b) { return __fsub_rn(a, b); }
ST_DF float fmul(float a, float b) { return __fmul_rn(a, b); }
ST_DF float ffma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
// seeds (a few ulp): MUFU reciprocal, reciprocal square root, 2^x, log2
ST_DF float rcp_seed(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
ST_DF float rsqrt_seed(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
ST_DF int f2i_bits(float x) { return __float_as_int(x); }
ST_DF float i2f_bits(int x) { return __int_as_float(x); }
#else
ST_DF float fadd(float a, float b) { return a + b; }
ST_DF float fsub(float a, float b) { return a - b; }
ST_DF float fmul(float a, float b) { return a * b; }
ST_DF float ffma(float a, float b, float c) { return fmaf(a, b, c); }
ST_DF float rcp_seed(float x) { return 1.f / x; }
ST_DF float rsqrt_seed(float x) { return 1.f / sqrtf(x); }
ST_DF int f2i_bits(float x) { union { float f; int i; } u; u.f = x; return u.i; }
ST_DF float i2f_bits(int x) { union { float f; int i; } u; u.i = x; return u.f; }
#endif

ST_DF df2 q(float a) { return df2{a, 0.f}; }
ST_DF df2 neg(df2 x) { return df2{-x.hi, -x.lo}; }
// Knuth's TwoSum and Dekker's FastTwoSum (|a| >= |b| or a = 0): exact
ST_DF df2 two_sum(float a, float b) {
  const float s = fadd(a, b);
  const float bb = fsub(s, a);
  return df2{s, fadd(fsub(a, fsub(s, bb)), fsub(b, bb))};
}
ST_DF df2 fast(float a, float b) {
  const float s = fadd(a, b);
  return df2{s, fsub(b, fsub(s, a))};
}
// x + y: one TwoSum on the high parts, the low parts added in float
ST_DF df2 add(df2 x, df2 y) {
  const df2 s = two_sum(x.hi, y.hi);
  return fast(s.hi, fadd(s.lo, fadd(x.lo, y.lo)));
}
ST_DF df2 sub(df2 x, df2 y) { return add(x, neg(y)); }
ST_DF df2 addf(df2 x, float f) {
  const df2 s = two_sum(x.hi, f);
  return fast(s.hi, fadd(s.lo, x.lo));
}
// x y without the final renormalisation: |lo| up to 2 ulp(hi), for operands of
// a sum
ST_DF df2 mulu(df2 x, df2 y) {
  const float p = fmul(x.hi, y.hi);
  const float e = ffma(x.hi, y.hi, -p);
  return df2{p, fadd(e, ffma(x.hi, y.lo, ffma(x.lo, y.hi, fmul(x.lo, y.lo))))};
}
ST_DF df2 mul(df2 x, df2 y) {
  const df2 p = mulu(x, y);
  return fast(p.hi, p.lo);
}
ST_DF df2 mulf(df2 x, float f) {
  const float p = fmul(x.hi, f);
  return fast(p, ffma(x.lo, f, ffma(x.hi, f, -p)));
}
// x times a power of two
ST_DF df2 scale(df2 x, float p2) { return df2{fmul(x.hi, p2), fmul(x.lo, p2)}; }
// a b + c d, a b - c d and a b + c d + e f with one renormalisation
ST_DF df2 dot2(df2 a, df2 b, df2 c, df2 d) {
  const df2 u = mulu(a, b), v = mulu(c, d);
  const df2 s = two_sum(u.hi, v.hi);
  return fast(s.hi, fadd(s.lo, fadd(u.lo, v.lo)));
}
ST_DF df2 dot3(df2 a, df2 b, df2 c, df2 d, df2 e, df2 f) {
  const df2 u = mulu(a, b), v = mulu(c, d), w = mulu(e, f);
  const df2 s = two_sum(u.hi, v.hi), t = two_sum(s.hi, w.hi);
  return fast(t.hi, fadd(fadd(s.lo, t.lo), fadd(fadd(u.lo, v.lo), w.lo)));
}
// x + a b, and x + a b + c d
ST_DF df2 fma1(df2 a, df2 b, df2 x) {
  const df2 u = mulu(a, b);
  const df2 s = two_sum(x.hi, u.hi);
  return fast(s.hi, fadd(s.lo, fadd(x.lo, u.lo)));
}
ST_DF df2 fma2(df2 a, df2 b, df2 c, df2 d, df2 x) {
  const df2 u = mulu(a, b), v = mulu(c, d);
  const df2 s = two_sum(x.hi, u.hi), t = two_sum(s.hi, v.hi);
  return fast(t.hi, fadd(fadd(s.lo, t.lo), fadd(fadd(u.lo, v.lo), x.lo)));
}
// 1 / x and 1 / sqrt(x).  The seed (1-2 ulp) first takes a Newton-Raphson step
// in float, so that r is within about half an ulp and the correction below it
// small: an error of two ulp there would cost the pair two bits.  Then the
// residual e (1 - x r, or 1 - x r^2) to second order, r (1 + e + e^2) and
// r (1 + e/2 + 3 e^2/8).
ST_DF df2 rcp(df2 x) {
  float r = rcp_seed(x.hi);
  r = ffma(r, ffma(-x.hi, r, 1.f), r);
  float e = ffma(-x.hi, r, 1.f);
  e = ffma(-x.lo, r, e);
  return fast(r, fmul(r, ffma(e, e, e)));
}
ST_DF df2 rsq(df2 x) {
  float r = rsqrt_seed(x.hi);
  r = ffma(fmul(0.5f, r), ffma(-fmul(x.hi, r), r, 1.f), r);
  const float p = fmul(r, r), pl = ffma(r, r, -p);
  float e = ffma(-x.hi, p, 1.f);
  e = ffma(-x.hi, pl, e);
  e = ffma(-x.lo, p, e);
  return fast(r, fmul(r, fmul(e, ffma(0.375f, e, 0.5f))));
}
// sqrt(x), 0 for x <= 0
ST_DF df2 sqrt_(df2 x) { return x.hi > 0.f ? mul(x, rsq(x)) : q(0.f); }
ST_DF df2 div(df2 x, df2 y) { return mul(x, rcp(y)); }

// comparisons of normalised pairs
ST_DF bool lt(df2 x, df2 y) { return x.hi < y.hi || (x.hi == y.hi && x.lo < y.lo); }
ST_DF df2 min_(df2 x, df2 y) { return lt(y, x) ? y : x; }
ST_DF df2 max_(df2 x, df2 y) { return lt(x, y) ? y : x; }

// x^2 + y^2 + z^2 + w as one sum: exact squares of the high parts, exact sums
// of those, everything below added in float.  (x^2 + y^2 + z^2 - a^2 is what
// the Kerr-Schild radius, and with it every term of the right-hand side, comes
// from: by separate products and sums it alone made the error of a ray three
// times as large.)
ST_DF df2 sumsq(df2 x, df2 y, df2 z, df2 w) {
  const float p1 = fmul(x.hi, x.hi), p2 = fmul(y.hi, y.hi), p3 = fmul(z.hi, z.hi);
  const float l1 = fadd(ffma(x.hi, x.hi, -p1), ffma(fadd(x.hi, x.hi), x.lo, fmul(x.lo, x.lo)));
  const float l2 = fadd(ffma(y.hi, y.hi, -p2), ffma(fadd(y.hi, y.hi), y.lo, fmul(y.lo, y.lo)));
  const float l3 = fadd(ffma(z.hi, z.hi, -p3), ffma(fadd(z.hi, z.hi), z.lo, fmul(z.lo, z.lo)));
  const df2 a = two_sum(p1, p2), b = two_sum(a.hi, p3), c = two_sum(b.hi, w.hi);
  return fast(c.hi, fadd(fadd(fadd(a.lo, b.lo), c.lo), fadd(fadd(fadd(l1, l2), l3), w.lo)));
}

// ---------------------------------------------------------------------------
// Two pairs at once, on Blackwell's packed FP32 instructions: one issued
// instruction does both halves, and negated, swapped and repeated operands cost
// nothing.  The functions are those above, half by half.
// ---------------------------------------------------------------------------
ST_DF v2 mkv(float x, float y) {
  v2 r;
  r.x = x;
  r.y = y;
  return r;
}
#ifdef __CUDA_ARCH__
ST_DF v2 vadd(v2 a, v2 b) { return __fadd2_rn(a, b); }
ST_DF v2 vmul(v2 a, v2 b) { return __fmul2_rn(a, b); }
ST_DF v2 vfma(v2 a, v2 b, v2 c) { return __ffma2_rn(a, b, c); }
#else
ST_DF v2 vadd(v2 a, v2 b) { return mkv(fadd(a.x, b.x), fadd(a.y, b.y)); }
ST_DF v2 vmul(v2 a, v2 b) { return mkv(fmul(a.x, b.x), fmul(a.y, b.y)); }
ST_DF v2 vfma(v2 a, v2 b, v2 c) { return mkv(ffma(a.x, b.x, c.x), ffma(a.y, b.y, c.y)); }
#endif
ST_DF v2 vneg(v2 a) { return mkv(-a.x, -a.y); }
ST_DF v2 vsub(v2 a, v2 b) { return vadd(a, vneg(b)); }

ST_DF dd two(df2 a, df2 b) { return dd{mkv(a.hi, b.hi), mkv(a.lo, b.lo)}; }
ST_DF dd both(df2 a) { return two(a, a); }
ST_DF df2 fst(dd a) { return df2{a.h.x, a.l.x}; }
ST_DF df2 snd(dd a) { return df2{a.h.y, a.l.y}; }
ST_DF dd neg(dd a) { return dd{vneg(a.h), vneg(a.l)}; }
// (a, b) -> (b, -a)
ST_DF dd turn(dd a) { return dd{mkv(a.h.y, -a.h.x), mkv(a.l.y, -a.l.x)}; }
ST_DF dd two_sum(v2 a, v2 b) {
  const v2 s = vadd(a, b);
  const v2 bb = vsub(s, a);
  return dd{s, vadd(vsub(a, vsub(s, bb)), vsub(b, bb))};
}
ST_DF dd fast(v2 a, v2 b) {
  const v2 s = vadd(a, b);
  return dd{s, vsub(b, vsub(s, a))};
}
ST_DF dd add(dd x, dd y) {
  const dd s = two_sum(x.h, y.h);
  return fast(s.h, vadd(s.l, vadd(x.l, y.l)));
}
ST_DF dd mulu(dd x, dd y) {
  const v2 p = vmul(x.h, y.h);
  const v2 e = vfma(x.h, y.h, vneg(p));
  return dd{p, vadd(e, vfma(x.h, y.l, vfma(x.l, y.h, vmul(x.l, y.l))))};
}
ST_DF dd mul(dd x, dd y) {
  const dd p = mulu(x, y);
  return fast(p.h, p.l);
}
ST_DF dd scale(dd x, float p2) { return dd{vmul(x.h, mkv(p2, p2)), vmul(x.l, mkv(p2, p2))}; }
ST_DF dd dot2(dd a, dd b, dd c, dd d) {
  const dd u = mulu(a, b), v = mulu(c, d);
  const dd s = two_sum(u.h, v.h);
  return fast(s.h, vadd(s.l, vadd(u.l, v.l)));
}
ST_DF dd dot3(dd a, dd b, dd c, dd d, dd e, dd f) {
  const dd u = mulu(a, b), v = mulu(c, d), w = mulu(e, f);
  const dd s = two_sum(u.h, v.h), t = two_sum(s.h, w.h);
  return fast(t.h, vadd(vadd(s.l, t.l), vadd(vadd(u.l, v.l), w.l)));
}
ST_DF dd fma1(dd a, dd b, dd x) {
  const dd u = mulu(a, b);
  const dd s = two_sum(x.h, u.h);
  return fast(s.h, vadd(s.l, vadd(x.l, u.l)));
}
ST_DF dd fma2(dd a, dd b, dd c, dd d, dd x) {
  const dd u = mulu(a, b), v = mulu(c, d);
  const dd s = two_sum(x.h, u.h), t = two_sum(s.h, v.h);
  return fast(t.h, vadd(vadd(s.l, t.l), vadd(vadd(u.l, v.l), x.l)));
}

// ---------------------------------------------------------------------------
// Three-float state: h + m + l, about 72 bits.
// ---------------------------------------------------------------------------
struct f3 {
  float h, m, l;
};
// two of them: a ray's state is (x, y), (p_x, p_y), (z, p_z)
struct t3 {
  v2 h, m, l;
};
ST_DF t3 two(f3 a, f3 b) { return t3{mkv(a.h, b.h), mkv(a.m, b.m), mkv(a.l, b.l)}; }
ST_DF f3 fst(t3 a) { return f3{a.h.x, a.m.x, a.l.x}; }
ST_DF f3 snd(t3 a) { return f3{a.h.y, a.m.y, a.l.y}; }
ST_DF dd top(t3 y) { return dd{y.h, y.m}; }
// y += c: TwoSums down the limbs, then one pass to keep them apart
ST_DF t3 add3(t3 y, dd c) {
  const dd s = two_sum(y.h, c.h), t = two_sum(y.m, c.l), u = two_sum(t.h, s.l);
  const v2 l = vadd(y.l, vadd(t.l, u.l));
  const dd v = fast(s.h, u.h), w = fast(v.l, l);
  const dd v2_ = fast(v.h, w.h), w2 = fast(v2_.l, w.l);
  return t3{v2_.h, w2.h, w2.l};
}

// to and from double
ST_DF df2 pair_of(double v) {
  const float h = (float)v;
  return df2{h, (float)(v - (double)h)};
}
ST_DF f3 f3_of(double v) {
  const float h = (float)v;
  const double r = v - (double)h;
  const float m = (float)r;
  return f3{h, m, (float)(r - (double)m)};
}
ST_DF double dbl(df2 x) { return (double)x.hi + (double)x.lo; }
ST_DF double dbl(f3 x) { return (double)x.h + ((double)x.m + (double)x.l); }
// (x, y, z, p_x, p_y, p_z) of a ray's state, and back
ST_DF void doubles(const t3& P, const t3& Q, const t3& W, double* y) {
  y[0] = dbl(fst(P)); y[1] = dbl(snd(P)); y[2] = dbl(fst(W));
  y[3] = dbl(fst(Q)); y[4] = dbl(snd(Q)); y[5] = dbl(snd(W));
}
ST_DF void set_state(const double* y, t3* P, t3* Q, t3* W) {
  *P = two(f3_of(y[0]), f3_of(y[1]));
  *Q = two(f3_of(y[3]), f3_of(y[4]));
  *W = two(f3_of(y[2]), f3_of(y[5]));
}

// ---------------------------------------------------------------------------
// Geodesic right-hand sides (the regrouped forms of st_trace.cuh).
// ---------------------------------------------------------------------------
struct Hole {
  df2 M, a, a2;  // a2 = a^2
};

// Scene constants as pairs, from the doubles of the launch block.
struct Scene {
  Hole H;
  df2 dt, hcoef, inv_rkill2;  // step rule: dt, hcoef / M, 1 / max(rkill2, 1e-6)
  df2 r32, r295;              // 3.2 M and 2.95 M
  df2 ds, ds_span;            // gas sample spacing, opacity x spacing
  df2 ln_in, ln_out;          // radial extent of the grid
  df2 kr, kphi, kz, klut;     // grid and colour-table index scales
  df2 tmin, tmax;             // colour table's range
  df2 emis100, T0;            // 100 x emission scale, exp(10.034259)
  df2 isco, inv_isco, E, L;   // ISCO radius, its inverse, E and L there
  df2 sqM, inv_2m;            // sqrt(M), 1 / (2M)
  df2 rb2;                    // squared radius that holds the gas
  df2 tspan;
};

// What a position fixes: |x|^2 for a = 0; for Kerr the Kerr-Schild radius and
// S = sqrt(w^2/4 + a^2 z^2), the quartic's root term, through which
// Sigma = r^4 + a^2 z^2 = 2 r^2 S needs no reciprocal of its own.
struct Geo {
  df2 flat2;       // x^2 + y^2 + z^2
  df2 r2, r, ir;   // Kerr-Schild r^2, r, 1/r (Kerr); |x|^2, |x|, 1/|x| (a = 0)
  df2 iS, qz;      // 1/S and a^2 z^2 (Kerr)
};

// P = (x, y), z
template <int KERR>
ST_DF Geo geometry(dd P, df2 z, const Hole& H) {
  Geo g;
  if (KERR) {
    const df2 w = sumsq(fst(P), snd(P), z, neg(H.a2));
    const df2 az = mul(H.a, z);
    g.flat2 = add(w, H.a2);
    g.qz = mul(az, az);
    const df2 wh = scale(w, 0.5f);
    const df2 S2 = fma1(wh, wh, g.qz);
    g.iS = rsq(S2);
    g.r2 = fma1(S2, g.iS, wh);
    if (!(g.r2.hi > 1e-12f)) g.r2 = q(1e-12f);
  } else {
    g.flat2 = g.r2 = sumsq(fst(P), snd(P), z, q(0.f));
    g.iS = g.qz = q(0.f);
  }
  g.ir = rsq(g.r2);
  g.r = mul(g.r2, g.ir);
  return g;
}

// The slopes of (x, y), (p_x, p_y), (z, p_z) = P, Q, W.
template <int KERR>
ST_DF void rhs(dd P, dd Q, dd W, const Geo& g, df2 pt, const Hole& H, dd* dP, dd* dQ, dd* dW) {
  const df2 z = fst(W), pz = snd(W), ir = g.ir;
  if (KERR) {
    const df2 r = g.r;
    const df2 r2a = add(g.r2, H.a2);
    const df2 ira = rcp(r2a);
    const dd ra = two(r, H.a);
    // A = p_x x + p_y y, B = p_x y - p_y x
    const dd AB = dot2(both(fst(Q)), P, both(snd(Q)), turn(P));
    const df2 A = fst(AB);
    const dd rab = mulu(ra, AB);
    const df2 T = mul(add(fst(rab), snd(rab)), ira);
    const dd m1 = mul(two(z, r), two(pz, g.iS));  // z p_z, 2 r^3 / Sigma
    const dd m2 = mul(m1, two(ir, H.M));
    const df2 Z = fst(m2), riS = snd(m1);
    const df2 ell = sub(add(T, Z), pt);
    const df2 fl = mul(snd(m2), ell);             // f l
    const dd ff = mul(both(fl), two(ira, ir));
    const df2 flir = snd(ff);
    const dd F = mul(both(fst(ff)), ra);          // f l r, f l a over r^2 + a^2
    *dP = fma2(neg(both(fst(F))), P, neg(both(snd(F))), turn(P), Q);
    const df2 rT2 = scale(mul(r, T), -2.f);
    const df2 dldr = dot2(add(A, rT2), ira, neg(Z), ir);
    const dd e = mul(two(ir, ell), both(ir));
    const df2 is2 = mul(g.iS, fst(e));            // 2 / Sigma
    const dd c = mul(two(g.qz, z), both(is2));
    const df2 inner = fma1(snd(e), addf(fst(c), -0.5f), dldr);
    const df2 G = mul(fl, inner);
    const dd Gs = mul(both(G), two(riS, r));
    *dQ = dot3(both(scale(fst(Gs), 0.5f)), P, both(fst(F)), Q, neg(both(snd(F))), turn(Q));
    const df2 zt = dot2(snd(Gs), r2a, mul(neg(H.a2), ell), fl);
    *dW = two(fma1(neg(flir), z, pz), dot2(scale(snd(c), 0.5f), zt, flir, pz));
  } else {
    const dd u = mulu(P, Q);
    const df2 v = mulu(z, pz);
    const df2 s = two_sum(u.h.x, u.h.y), t = two_sum(s.hi, v.hi);
    const df2 xp = fast(t.hi, fadd(fadd(s.lo, t.lo), fadd(fadd(u.l.x, u.l.y), v.lo)));
    const dd m = mul(two(xp, scale(H.M, 2.f)), both(ir));
    const df2 kap = fst(m);
    const df2 ell = sub(kap, pt);
    const df2 c1 = mul(mul(snd(m), ell), ir);
    const df2 c2 = mul(mul(c1, add(scale(ell, 0.5f), kap)), ir);
    const dd C1 = both(c1), n2 = neg(both(c2));
    *dP = fma1(neg(C1), P, Q);
    *dQ = dot2(C1, Q, n2, P);
    *dW = two(fma1(neg(c1), z, pz), dot2(c1, pz, neg(c2), z));
  }
}

// Classical RK4: the increments of one step of size *h from (P, Q, W).  begin(g, h)
// sees the geometry of the state, sets the step's size and may end the ray;
// first(dP, dW) sees the slopes at the state.  The four stages share one copy
// of the right-hand side.
template <int KERR, class Begin, class First>
ST_DF bool rk4(const t3& P, const t3& Q, const t3& W, df2 pt, const Hole& H, const Begin& begin, const First& first,
               df2* h, dd* iP, dd* iQ, dd* iW) {
  dd tP = top(P), tQ = top(Q), tW = top(W);
  dd sP = two(q(0.f), q(0.f)), sQ = sP, sW = sP;
#ifdef __CUDACC__
#pragma unroll 1
#endif
  for (int s = 0; s < 4; ++s) {
    const Geo g = geometry<KERR>(tP, fst(tW), H);
    if (s == 0 && begin(g, h)) return true;
    dd kP, kQ, kW;
    rhs<KERR>(tP, tQ, tW, g, pt, H, &kP, &kQ, &kW);
    if (s == 0) first(kP, kW);
    const float w = (s == 1 || s == 2) ? 2.f : 1.f;
    sP = add(sP, scale(kP, w));
    sQ = add(sQ, scale(kQ, w));
    sW = add(sW, scale(kW, w));
    const dd hs = both(scale(*h, s < 2 ? 0.5f : 1.f));
    tP = fma1(hs, kP, top(P));
    tQ = fma1(hs, kQ, top(Q));
    tW = fma1(hs, kW, top(W));
  }
  const dd h6 = both(mul(*h, df2{0.166666672f, -4.96705388e-9f}));
  *iP = mul(h6, sP);
  *iQ = mul(h6, sQ);
  *iW = mul(h6, sW);
  return false;
}

// rhs and rk4 component by component, y = (x, y, z, p_x, p_y, p_z): the same
// sums and products, so the same bits, in plain instructions.  For a step that a
// few lanes of a warp take beside others' work (the guard steps; the reason and
// the figures are at guard_step in st_trace.cuh).
template <int KERR>
ST_DF void rhs6(const df2* y, const Geo& g, df2 pt, const Hole& H, df2* d) {
  const df2 ir = g.ir;
  if (KERR) {
    const df2 r = g.r, a = H.a;
    const df2 r2a = add(g.r2, H.a2);
    const df2 ira = rcp(r2a);
    const df2 A = dot2(y[3], y[0], y[4], y[1]), B = dot2(y[3], y[1], y[4], neg(y[0]));
    const df2 T = mul(add(mulu(r, A), mulu(a, B)), ira);
    const df2 Z = mul(mul(y[2], y[5]), ir), riS = mul(r, g.iS);
    const df2 ell = sub(add(T, Z), pt);
    const df2 fl = mul(mul(riS, H.M), ell);
    const df2 fi = mul(fl, ira), flir = mul(fl, ir);
    const df2 Fr = mul(fi, r), Fa = mul(fi, a);
    d[0] = fma2(neg(Fr), y[0], neg(Fa), y[1], y[3]);
    d[1] = fma2(neg(Fr), y[1], neg(Fa), neg(y[0]), y[4]);
    const df2 dldr = dot2(add(A, scale(mul(r, T), -2.f)), ira, neg(Z), ir);
    const df2 is2 = mul(g.iS, mul(ir, ir));
    const df2 inner = fma1(mul(ell, ir), addf(mul(g.qz, is2), -0.5f), dldr);
    const df2 G = mul(fl, inner);
    const df2 s = scale(mul(G, riS), 0.5f);
    d[3] = dot3(s, y[0], Fr, y[3], neg(Fa), y[4]);
    d[4] = dot3(s, y[1], Fr, y[4], neg(Fa), neg(y[3]));
    const df2 zt = dot2(mul(G, r), r2a, mul(neg(H.a2), ell), fl);
    d[2] = fma1(neg(flir), y[2], y[5]);
    d[5] = dot2(scale(mul(y[2], is2), 0.5f), zt, flir, y[5]);
  } else {
    const df2 kap = mul(dot3(y[0], y[3], y[1], y[4], y[2], y[5]), ir);
    const df2 ell = sub(kap, pt);
    const df2 c1 = mul(mul(mul(scale(H.M, 2.f), ir), ell), ir);
    const df2 c2 = mul(mul(c1, add(scale(ell, 0.5f), kap)), ir);
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int k = 0; k < 3; ++k) {
      d[k] = fma1(neg(c1), y[k], y[k + 3]);
      d[k + 3] = dot2(c1, y[k + 3], neg(c2), y[k]);
    }
  }
}

// The increments of one step of size h from y.
template <int KERR>
ST_DF void rk4_six(const df2* y, df2 pt, const Hole& H, df2 h, df2* inc) {
  df2 t[6], s[6];
#ifdef __CUDACC__
#pragma unroll
#endif
  for (int k = 0; k < 6; ++k) { t[k] = y[k]; s[k] = q(0.f); }
#ifdef __CUDACC__
#pragma unroll 1
#endif
  for (int st = 0; st < 4; ++st) {
    df2 d[6];
    rhs6<KERR>(t, geometry<KERR>(two(t[0], t[1]), t[2], H), pt, H, d);
    const float w = (st == 1 || st == 2) ? 2.f : 1.f;
    const df2 hs = scale(h, st < 2 ? 0.5f : 1.f);
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int k = 0; k < 6; ++k) {
      s[k] = add(s[k], scale(d[k], w));
      t[k] = fma1(hs, d[k], y[k]);
    }
  }
  const df2 h6 = mul(h, df2{0.166666672f, -4.96705388e-9f});
#ifdef __CUDACC__
#pragma unroll
#endif
  for (int k = 0; k < 6; ++k) inc[k] = mul(h6, s[k]);
}

// x + y with one rounding of x's low part, for |y| < |x|: half an ulp of it where
// add is off by one or two.  For a state that is added to at every step, whose
// rounding is then all that a guarded ray is off by.
ST_DF df2 add_rn(df2 x, df2 y) {
  const df2 s = two_sum(x.hi, y.hi), u = two_sum(s.lo, x.lo), v = fast(s.hi, u.hi);
  return fast(v.hi, fadd(v.lo, fadd(u.lo, y.lo)));
}

// ---------------------------------------------------------------------------
// Shading.  Its results go into a float image, so its pairs are kept to about
// 2^-40: products and sums without the last renormalisation (half the
// instructions, and half the code: the step and a sample together have to stay
// near the instruction cache's size).  Comparisons and floors renormalise.
// ---------------------------------------------------------------------------
namespace sh {

ST_DF df2 add(df2 x, df2 y) {
  const df2 s = two_sum(x.hi, y.hi);
  return df2{s.hi, fadd(s.lo, fadd(x.lo, y.lo))};
}
ST_DF df2 sub(df2 x, df2 y) { return add(x, neg(y)); }
ST_DF df2 addf(df2 x, float f) {
  const df2 s = two_sum(x.hi, f);
  return df2{s.hi, fadd(s.lo, x.lo)};
}
ST_DF df2 mul(df2 x, df2 y) {
  const float p = fmul(x.hi, y.hi);
  return df2{p, ffma(x.lo, y.hi, ffma(x.hi, y.lo, ffma(x.hi, y.hi, -p)))};
}
ST_DF df2 mulf(df2 x, float f) {
  const float p = fmul(x.hi, f);
  return df2{p, ffma(x.lo, f, ffma(x.hi, f, -p))};
}
ST_DF df2 fma1(df2 a, df2 b, df2 x) { return add(x, mul(a, b)); }
ST_DF df2 dot2(df2 a, df2 b, df2 c, df2 d) { return add(mul(a, b), mul(c, d)); }
ST_DF df2 norm(df2 x) { return fast(x.hi, x.lo); }
ST_DF df2 rcp(df2 x) {
  const float r = rcp_seed(x.hi);
  const float e = ffma(-x.lo, r, ffma(-x.hi, r, 1.f));
  return df2{r, fmul(r, ffma(e, e, e))};
}
ST_DF df2 rsq(df2 x) {
  const float r = rsqrt_seed(x.hi);
  const float p = fmul(r, r), pl = ffma(r, r, -p);
  const float e = ffma(-x.lo, p, ffma(-x.hi, pl, ffma(-x.hi, p, 1.f)));
  return df2{r, fmul(r, fmul(e, ffma(0.375f, e, 0.5f)))};
}
ST_DF df2 sqrt_(df2 x) { return x.hi > 0.f ? mul(x, rsq(x)) : q(0.f); }
ST_DF df2 div(df2 x, df2 y) { return mul(x, rcp(y)); }
// the same for two at once
ST_DF dd add(dd x, dd y) {
  const dd s = two_sum(x.h, y.h);
  return dd{s.h, vadd(s.l, vadd(x.l, y.l))};
}
ST_DF dd mul(dd x, dd y) {
  const v2 p = vmul(x.h, y.h);
  return dd{p, vfma(x.l, y.h, vfma(x.h, y.l, vfma(x.h, y.h, vneg(p))))};
}
ST_DF dd fma1(dd a, dd b, dd x) { return add(x, mul(a, b)); }

// exp, log and atan2 from their series, the argument reduced until the terms
// below the pair terms fit a float.

// e^x, x <= 80: x = n ln 2 + r, e^(r/16) - 1 by Taylor's series, and four times
// (1 + s)^2 - 1 = 2 s + s^2.  Below -87.3, where 2^n would leave a float's normal
// exponents, it is e^-87.3 (the argument may be -infinity: an optical depth is as large
// as the user's opacity, spacing and density make it).
ST_DF df2 exp_(df2 x) {
  if (x.hi < -87.3f) x = q(-87.3f);
  const float n = rintf(fmul(x.hi, 1.44269504f));
  // ln 2 in three floats
  const float p = fmul(n, 0.693147182f), pe = ffma(n, 0.693147182f, -p);
  const df2 d = two_sum(x.hi, -p);
  const float t = ffma(-n, -1.90465421e-9f, x.lo), te = ffma(-n, -8.78318374e-17f, 0.f);
  df2 r = add(d, two_sum(t, fsub(te, pe)));
  r = scale(r, 0.0625f);
  const df2 r2 = mul(r, r);
  const float h = r.hi;
  const float tail = fmul(fmul(r2.hi, r2.hi), ffma(h, ffma(h, ffma(h, 1.98412698e-4f, 1.38888889e-3f), 8.33333333e-3f),
                                                  4.16666667e-2f));
  // r + r^2/2 + r^3/6 + tail
  df2 s = fma1(mul(r2, r), df2{0.166666672f, -4.96705388e-9f}, addf(scale(r2, 0.5f), tail));
  s = add(r, s);
#pragma unroll
  for (int k = 0; k < 4; ++k) s = fma1(s, s, scale(s, 2.f));
  return scale(norm(addf(s, 1.f)), i2f_bits(((int)n + 127) << 23));
}

// ln x, x > 0 and normal: x = 2^e m with m in [3/4, 3/2), ln m = 2 atanh((m - 1)/(m + 1)).
ST_DF df2 log_(df2 x) {
  const int e = (f2i_bits(x.hi) - 0x3f400000) >> 23;
  const df2 m = scale(x, i2f_bits((127 - e) << 23));
  const df2 z = div(addf(m, -1.f), addf(m, 1.f));
  const df2 z2 = mul(z, z);
  const float v = z2.hi;
  const float tail = fmul(fmul(fmul(v, v), v), ffma(v, ffma(v, ffma(v, ffma(v, ffma(v, 0.117647059f, 0.133333333f),
                     0.153846154f), 0.181818182f), 0.222222222f), 0.285714286f));
  // 2 z (1 + z^2/3 + z^4/5) + z tail
  const df2 c = fma1(z2, fma1(z2, df2{0.400000006f, -5.96046457e-9f}, df2{0.666666687f, -1.98682155e-8f}), addf(q(tail), 2.f));
  const float n = (float)e;
  const float p = fmul(n, 0.693147182f);
  const df2 l = two_sum(p, ffma(n, 0.693147182f, -p));
  return fma1(z, c, addf(l, fmul(n, -1.90465421e-9f)));
}

// atan(k / 8), k = 0..8
#ifdef __CUDACC__
__device__ const
#else
static const
#endif
    float kAtan8[9][2] = {
        {0.f, 0.f},
        {0.124354996f, -1.24038224e-09f},
        {0.244978666f, -3.17867777e-09f},
        {0.358770669f, 1.76394988e-09f},
        {0.463647604f, 5.01215869e-09f},
        {0.558599293f, 2.21115979e-08f},
        {0.643501103f, 5.86893734e-09f},
        {0.718829989f, 1.01883355e-08f},
        {0.785398185f, -2.18556941e-08f}};

// atan2(y, x): the smaller over the larger magnitude, turned back by the
// nearest atan(k / 8) (one division), and atan's series below 1/15.
ST_DF df2 atan2_(df2 y, df2 x) {
  const df2 ay = y.hi < 0.f ? neg(y) : y, ax = x.hi < 0.f ? neg(x) : x;
  const bool steep = lt(ax, ay);  // normalised inputs
  const df2 mn = steep ? ax : ay, mx = steep ? ay : ax;
  const int k = (int)rintf(fmul(8.f, fmul(mn.hi, rcp_seed(mx.hi))));
  const float c = fmul((float)k, 0.125f);
  const df2 z = div(add(mn, mulf(mx, -c)), add(mx, mulf(mn, c)));
  const df2 z2 = mul(z, z);
  const float v = z2.hi;
  const float tail = fmul(fmul(v, v), ffma(v, ffma(v, 0.111111111f, -0.142857143f), 0.2f));
  const df2 u = fma1(z2, df2{-0.333333343f, 9.93410776e-9f}, q(tail));
  df2 t = add(df2{kAtan8[k][0], kAtan8[k][1]}, fma1(z, u, z));
  if (steep) t = sub(df2{1.57079637f, -4.37113883e-8f}, t);
  if (x.hi < 0.f) t = sub(df2{3.14159274f, -8.74227766e-8f}, t);
  return y.hi < 0.f ? neg(t) : t;
}

// ---------------------------------------------------------------------------
// The gas (the double code of march_gas, sample_volume and emitter_opz in
// st_trace.cuh, term for term).
// ---------------------------------------------------------------------------

// 1 + z of the emitter at (x, y); iE = 1 / E of the ray.
ST_DF df2 emitter(df2 x, df2 y, df2 px, df2 py, df2 s2, df2 iE, const Scene& C) {
  const df2 a = C.H.a, a2 = C.H.a2, M = C.H.M;
  const df2 r2 = max_(norm(sub(s2, a2)), q(1e-6f));
  const df2 r = norm(sqrt_(r2));
  df2 ut, ux, uy;
  if (!lt(r, C.isco)) {
    const df2 sr = sqrt_(r);
    const df2 r32 = mul(r, sr);
    const df2 asm_ = mul(a, C.sqM);
    const df2 den = max_(norm(add(fma1(scale(M, -3.f), sr, r32), scale(asm_, 2.f))), df2{0.00999999978f, 2.23517413e-10f});
    const df2 inv = rsq(mul(r32, den));
    ut = mul(add(r32, asm_), inv);
    const df2 up = mul(C.sqM, inv);
    ux = neg(mul(y, up));
    uy = mul(x, up);
  } else {
    const df2 M2 = scale(M, 2.f), ir = rcp(r), rr = mul(r, r), rr2 = add(rr, a2);
    const df2 delta = fma1(neg(M2), r, rr2);
    const df2 id = rcp(max_(norm(delta), df2{0.00100000005f, -4.74974504e-11f}));
    const df2 mr = mul(M2, ir), maL = mul(mul(mr, a), C.L);
    const df2 t1 = dot2(C.E, rr2, neg(a), C.L), t2 = fma1(neg(a), C.E, C.L);
    const df2 R = max_(norm(dot2(t1, t1, neg(delta), fma1(t2, t2, rr))), q(0.f));
    const df2 ur = neg(mul(sqrt_(R), mul(ir, ir)));
    ut = fma1(mul(mul(M2, r), id), ur, mul(sub(mul(fma1(mr, a2, rr2), C.E), maL), id));
    const df2 up0 = mul(dot2(mul(mr, a), C.E, sub(q(1.f), mr), C.L), id);
    const df2 up = fma1(mul(a, id), ur, up0);
    const df2 is2 = rcp(max_(norm(s2), q(1e-6f)));
    ux = dot2(mul(ur, is2), dot2(r, x, a, y), neg(y), up);
    uy = dot2(mul(ur, is2), dot2(r, y, neg(a), x), x, up);
  }
  const df2 z = norm(fma1(neg(dot2(px, ux, py, uy)), iE, ut));
  return min_(max_(z, df2{0.100000001f, -1.49011614e-9f}), q(20.f));
}

// floor of a normalised pair, and the remainder
ST_DF int floor_(df2 x, df2* rest) {
  float f = floorf(x.hi);
  if (f == x.hi && x.lo < 0.f) f = fsub(f, 1.f);
  *rest = fast(fsub(x.hi, f), x.lo);
  return (int)f;
}

// a + t (b - a)
ST_DF df2 lerp(df2 t, df2 a, df2 b) { return fma1(t, sub(b, a), a); }

// Trilinear density at squared cylinder radius s2 (> 0), azimuth direction
// (x, y) and height z, |z| < zmax; v(offset) reads the grid.
template <class Load>
ST_DF df2 density(const Load& v, int nr, int nphi, int nz, float zmax, df2 s2, df2 x, df2 y, df2 z, const Scene& C) {
  const df2 ls = norm(scale(log_(s2), 0.5f));
  if (!lt(C.ln_in, ls) || !lt(ls, C.ln_out)) return q(0.f);
  df2 phi = atan2_(y, x);
  if (phi.hi < 0.f) phi = add(phi, df2{6.28318548f, -1.74845553e-7f});
  df2 tr, tp, tz;
  const int i = floor_(norm(mul(sub(ls, C.ln_in), C.kr)), &tr);
  const int j = floor_(norm(mul(phi, C.kphi)), &tp);
  const int k = floor_(norm(mul(addf(z, zmax), C.kz)), &tz);
  // the double code's clamps: to the first and last cell, the fraction from there
  const int i0 = i < 0 ? 0 : (i > nr - 2 ? nr - 2 : i), k0 = k < 0 ? 0 : (k > nz - 2 ? nz - 2 : k);
  if (i0 != i) tr = addf(tr, (float)(i - i0));
  if (k0 != k) tz = addf(tz, (float)(k - k0));
  const int ja = j >= nphi ? j - nphi : (j < 0 ? j + nphi : j);
  const int jb = ja + 1 >= nphi ? ja + 1 - nphi : ja + 1;
  const int sk = nr * nphi, b0 = i0 + sk * k0 + nr * ja, b1 = i0 + sk * k0 + nr * jb;
  const v2 zero = mkv(0.f, 0.f);
  const v2 la = mkv(v(b0), v(b1)), lb = mkv(v(b0 + 1), v(b1 + 1));
  const v2 ua = mkv(v(b0 + sk), v(b1 + sk)), ub = mkv(v(b0 + sk + 1), v(b1 + sk + 1));
  const dd l = fma1(both(tr), two_sum(lb, vneg(la)), dd{la, zero});  // lower cell, at j and j + 1
  const dd u = fma1(both(tr), two_sum(ub, vneg(ua)), dd{ua, zero});
  const dd c0 = two(fst(l), fst(u)), c1 = two(snd(l), snd(u));
  const dd c = fma1(both(tp), add(c1, neg(c0)), c0);
  return norm(lerp(tz, fst(c), snd(c)));
}

}  // namespace sh
}  // namespace dfm
}  // namespace st
