// st_trace_pairs.cu -- ST_PREC_FP64 frames with the integration on the FP32
// pipe: slopes in float pairs, state in three floats (st_df.cuh).
//
// The all-double kernels are bound by the FP64 pipe (86-89 % busy; one warp
// operation every 19 cycles of an SM), so this one keeps double for what a ray
// does once -- its launch, its landing on the escape sphere, its sky -- and for
// the few disc crossings, and runs the ~1,000 steps between on the FP32 pipe.
// The state it carries is wider than double's, and the exit directions are
// closer to the exact RK4 sequence than the double kernel's
// (tests/test_df_math.py).  Bound by the FP32 issue and pipe (58-67 % of the FMA
// pipe) and, on small frames, by the longest ray's own chain of steps.  Measured
// per frame, all-double before: 320x180 Schwarzschild disc by the CPU renderer's
// rules 53.8 -> 8.9 ms, 320x180 Kerr gas 130 -> 17.6 ms.
#include "st_kernels.cuh"

namespace st {
namespace {

using dfm::dbl;
using dfm::doubles;
using dfm::fst;
using dfm::pair_of;
using dfm::snd;
using dfm::t3;
using dfm::two;

struct PairRay {
  t3 P, Q, W;  // (x, y), (p_x, p_y), (z, p_z)
  df2 pt, iE, scam;
  df2 acc[3], alpha, march, lambda;
  df2 r_prev;
  df2 r_esc, r_floor;
  df2 land_h;  // > 0: the ray ended on a sphere inside a step of this size from y
  int nmax, steps, gas, flags;
  bool inside0;
  float r_cross, g_cross;
  // gas: samples waiting in the queue, the step being sampled (distance of the
  // next sample and length), and the step at which a ray found opaque ends
  int queued, stop;
  int marching;  // samples the step may still take
  df2 t, seg;
};

// The gas samples of a warp's rays wait in shared memory, up to GAS_Q a ray, and
// are shaded together.  Sampled as they come, a step in two has a sample, the
// rays of a warp at different steps: the shading ran for 14 of 32 lanes after
// nearly every step, and its code and the integrator's drove each other out of
// the instruction cache.  With eight a ray the lanes hold nearly equal numbers.
// With this, packed pairs and the short shading arithmetic of st_df.cuh the Kerr
// gas frame went from 25.2 to 18.0 ms at 320x180 and from 142 to 109 ms at
// 960x540 (all in double: 130 ms and about 1,000 ms).
constexpr int GAS_Q = 8;
struct GasWarp {
  dd P[GAS_Q][32], Q[GAS_Q][32];  // (x, y), (p_x, p_y) at the sample
  float2 z[GAS_Q][32];
  int step[GAS_Q][32];            // the step it belongs to
  // the step being sampled: the state before it and its increment
  dd sP[32], sQ[32], iP[32], iQ[32];
  float2 sz[32], iz[32];
  // the ray as the last shading left it, from where a ray that turns out to
  // have become opaque meanwhile goes again to the step that ended it
  t3 P0[32], Q0[32], W0[32];
  df2 r_prev0[32];
  int steps0[32], flags0[32];
};

__device__ __forceinline__ float2 f2(df2 x) { return make_float2(x.hi, x.lo); }
__device__ __forceinline__ df2 d2(float2 x) { return df2{x.x, x.y}; }

// Starts march_gas's walk along one step: the state before it and its increment.
__device__ __forceinline__ void start_gas(const TraceParams& p, const t3& P, const t3& Q, const t3& W, dd iP, dd iQ,
                                          dd iW, df2 r2p, df2 r2n, df2 seg, PairRay& st, GasWarp& g, int lane) {
  using namespace dfm;
  if (!lt(min_(r2p, r2n), p.d.rb2) || !(seg.hi < 64.f)) return;
  const df2 t = sub(p.d.ds, st.march);
  if (lt(seg, t)) { st.march = add(st.march, seg); return; }
  st.t = t;
  st.seg = seg;
  st.marching = 8192;
  g.sP[lane] = top(P);
  g.sQ[lane] = top(Q);
  g.sz[lane] = make_float2(W.h.x, W.m.x);
  g.iP[lane] = iP;
  g.iQ[lane] = iQ;
  g.iz[lane] = f2(fst(iW));
}

// The samples of the step being walked into the queue, until it ends or the
// queue is full; samples outside the slab count for nothing and are not kept.
__device__ __forceinline__ void queue_gas(const TraceParams& p, PairRay& st, GasWarp& g, int lane) {
  using namespace dfm;
  const df2 ds = p.d.ds, inv_seg = rcp(st.seg);
#pragma unroll 1
  while (st.queued < GAS_Q) {
    const df2 fs = mul(st.t, inv_seg);
    const df2 z = fma1(fs, d2(g.iz[lane]), d2(g.sz[lane]));
    if (lt(z.hi < 0.f ? neg(z) : z, q(p.f.zmax))) {
      g.z[st.queued][lane] = f2(z);
      g.P[st.queued][lane] = fma1(both(fs), g.iP[lane], g.sP[lane]);
      g.Q[st.queued][lane] = fma1(both(fs), g.iQ[lane], g.sQ[lane]);
      g.step[st.queued][lane] = st.steps;
      ++st.queued;
    }
    st.t = add(st.t, ds);
    if (--st.marching == 0 || lt(st.seg, st.t)) {
      st.march = sub(st.seg, sub(st.t, ds));
      st.marching = 0;
      break;
    }
  }
}

// Shades one sample (the body of march_gas).
__device__ __forceinline__ void shade_gas(const TraceParams& p, df2 sx, df2 sy, df2 sz, df2 px, df2 py, PairRay& st) {
  using namespace dfm::sh;
  using dfm::f2i_bits;
  using dfm::lt;
  using dfm::max_;
  using dfm::min_;
  using dfm::neg;
  using dfm::q;
  const dfm::Scene& C = p.d;
  const df2 s2 = dot2(sx, sx, sy, sy);
  if (!(s2.hi > 1e-12f)) return;
  df2 rho = density([&](int o) { return __ldg(p.vol + o); }, p.nr, p.nphi, p.nz, p.f.zmax, s2, sx, sy, sz, C);
  ++st.gas;
  if (!lt(df2{9.99999975e-5f, 2.52621613e-12f}, rho)) return;  // 1e-4
  const df2 s = norm(sqrt_(s2));
  // T = exp(10.034259) (s / 2M)^(-3/4) outside the ISCO, its value there inside
  const bool in = lt(s, C.isco);
  const df2 u = rsq(mul(in ? C.isco : s, C.inv_2m));
  const df2 T = mul(C.T0, mul(u, sqrt_(u)));
  if (in) { const df2 t3 = mul(s, C.inv_isco); rho = mul(rho, mul(t3, mul(t3, t3))); }
  const df2 opz = emitter(sx, sy, px, py, s2, st.iE, C);
  const df2 obs = norm(div(mul(T, st.scam), opz));
  df2 rest;
  const df2 tc = min_(max_(obs, C.tmin), C.tmax);
  const int idx = floor_(norm(addf(mul(sub(tc, C.tmin), C.klut), 0.5f)), &rest);
  const float4 col = __ldg(p.lut + min(max(idx, 0), p.lut_size - 1));
  // e^(-tau) and the Planck factor's e^(29622.4 / T) by one copy of exp; beyond
  // e^80 the radiance is below 1e-32
  const df2 x = div(df2{29622.4004f, -3.90625006e-4f}, max_(obs, q(1.f)));
  const bool faint = x.hi > 80.f;
  df2 e, ex = faint ? q(80.f) : x;
#pragma unroll 1
  for (int n = 0; n < 2; ++n) {
    e = exp_(ex);
    if (n == 0) { ex = neg(mul(C.ds_span, rho)); rho = e; }
  }
  const df2 inten = faint ? q(0.f) : mul(C.emis100, rcp(addf(rho, -1.f)));
  const df2 w = mul(mul(st.alpha, addf(neg(e), 1.f)), inten);
  // the sums over a ray's samples keep the full pair
  st.acc[0] = dfm::add(st.acc[0], mulf(w, col.x));
  st.acc[1] = dfm::add(st.acc[1], mulf(w, col.y));
  st.acc[2] = dfm::add(st.acc[2], mulf(w, col.z));
  st.alpha = dfm::mul(st.alpha, e);
}

// Shades the queue.  A ray that becomes opaque ends with the state of that
// sample's step: at once if that is the ray's last step, else it starts again
// from where the queue was last empty and stops there.  Returns whether the ray
// has steps to take.
__device__ __forceinline__ bool shade_queue(const TraceParams& p, bool run, PairRay& st, GasWarp& g, int lane) {
  const df2 amin{0.00300000003f, -2.60770321e-11f};  // 0.003
#pragma unroll 1
  for (int n = 0; n < st.queued; ++n) {
    const dd P = g.P[n][lane], Q = g.Q[n][lane];
    shade_gas(p, fst(P), snd(P), d2(g.z[n][lane]), fst(Q), snd(Q), st);
    if (!dfm::lt(amin, st.alpha)) {
      st.marching = 0;
      st.stop = g.step[n][lane];
      // the state is that step's unless the ray went on, or ended (its flags tell)
      run = false;
      if (st.stop != st.steps || st.flags != g.flags0[lane]) {
        st.P = g.P0[lane];
        st.Q = g.Q0[lane];
        st.W = g.W0[lane];
        st.r_prev = g.r_prev0[lane];
        st.steps = g.steps0[lane];
        st.land_h = dfm::q(0.f);
        run = st.steps != st.stop;
      }
      st.flags = g.flags0[lane];
      break;
    }
  }
  st.queued = 0;
  return run;
}

__device__ __forceinline__ void mark_ray(const PairRay& st, GasWarp& g, int lane) {
  g.P0[lane] = st.P;
  g.Q0[lane] = st.Q;
  g.W0[lane] = st.W;
  g.r_prev0[lane] = st.r_prev;
  g.steps0[lane] = st.steps;
  g.flags0[lane] = st.flags;
}

__device__ __forceinline__ void set_state(const double* y, PairRay& st) { dfm::set_state(y, &st.P, &st.Q, &st.W); }

// The disc where a step crosses z = 0, in double as in step_ray; P, Q, W the
// state before the step, st the state after it.
__device__ __forceinline__ void cross_pairs(const TraceParams& p, const t3& P, const t3& Q, const t3& W, bool kepler,
                                            PairRay& st) {
  double s[6], yn[6];
  doubles(P, Q, W, s);
  doubles(st.P, st.Q, st.W, yn);
  const double c = s[2] / (s[2] - yn[2]);
#pragma unroll
  for (int k = 0; k < 6; ++k) s[k] += c * (yn[k] - s[k]);
  double acc[3] = {dbl(st.acc[0]), dbl(st.acc[1]), dbl(st.acc[2])}, alpha = dbl(st.alpha);
  const double pt = dbl(st.pt), scam = dbl(st.scam);
  const double g = kepler ? disc_kepler(p, s[0], s[1], s + 3, pt, scam, acc, &alpha)
                          : disc_exact(p, s[0], s[1], s[3], s[4], pt, scam, acc, &alpha);
#pragma unroll
  for (int k = 0; k < 3; ++k) st.acc[k] = pair_of(acc[k]);
  st.alpha = pair_of(alpha);
  if (g > 0.0 && st.r_cross < 0.f) {
    st.r_cross = (float)sqrt(s[0] * s[0] + s[1] * s[1]);
    st.g_cross = (float)g;
    st.flags |= ST_RAY_CROSSED;
  }
}

// The tests of step_ray before a step (capture, escape, budget) and the step's
// size; true when the ray is done.
template <int KERR, int VOL, int SEM>
__device__ __forceinline__ bool begin_pairs(const TraceParams& p, const dfm::Geo& g, PairRay& st, df2* h) {
  using namespace dfm;
  const Scene& C = p.d;
  const df2 r = KERR ? sqrt_(g.flat2) : g.r;
  if constexpr (SEM == ST_SEM_DRAFT) {
    if constexpr (KERR) {
      if (lt(g.r2, q(p.f.rkill2))) { st.flags |= ST_RAY_CAPTURED; return true; }
    } else if (lt(r, C.r32)) {
      const float back = fadd(fsub(r.hi, st.r_prev.hi), fsub(r.lo, st.r_prev.lo));
      if (lt(r, st.r_floor) || (lt(r, C.r295) && st.r_prev.hi > 0.f && back < -1e-4f * p.f.M)) {
        st.flags |= ST_RAY_CAPTURED;
        return true;
      }
      st.r_prev = r;
    }
    if (lt(st.r_esc, r)) { st.flags |= ST_RAY_ESCAPED; return true; }
  } else {
    if (!lt(r, st.r_esc)) { st.flags |= ST_RAY_ESCAPED; return true; }
    if (!lt(st.lambda, C.tspan)) { st.flags |= ST_RAY_BUDGET; return true; }
    const float back = fadd(fsub(r.hi, st.r_prev.hi), fsub(r.lo, st.r_prev.lo));
    if (lt(r, C.r295) && st.r_prev.hi > 0.f && back < -1e-4f * p.f.M) {
      st.flags |= ST_RAY_CAPTURED;
      return true;
    }
    st.r_prev = r;
  }
  const float cap = (VOL && lt(g.flat2, C.rb2)) ? 2.f : p.f.hcap;
  *h = mul(C.dt, min_(max_(mul(C.hcoef, r), q(1.f)), q(cap)));
  if constexpr (KERR && SEM == ST_SEM_DRAFT) {
    const df2 fr = min_(max_(mul(addf(g.r2, -p.f.rkill2), C.inv_rkill2), q(0.f)), q(1.f));
    // 0.12 + 0.88 fr
    *h = mul(*h, fma1(df2{0.879999995f, 4.76837159e-9f}, fr, df2{0.119999997f, 2.68220901e-9f}));
  }
  if constexpr (SEM == ST_SEM_RENDER) *h = min_(*h, sub(C.tspan, st.lambda));
  return false;
}

// One step of step_ray's rules (RK4); true when the ray is done.  The four
// stages share one copy of the right-hand side (dfm::rk4): unrolled, the step and the gas
// sample outgrow the instruction caches (4.8 of 7 stall cycles an instruction
// were fetches, and the 320x180 gas frame took 34.7 ms, rolled 25.2).
template <int KERR, int VOL, int SEM>
__device__ __forceinline__ bool step_pairs(const TraceParams& p, PairRay& st, GasWarp* gas, int lane) {
  using namespace dfm;
  const Scene& C = p.d;
  if (st.steps >= st.nmax) { st.flags |= ST_RAY_BUDGET; return true; }
  df2 h, r2, v2;
  dd iP, iQ, iW;
  const bool done = rk4<KERR>(
      st.P, st.Q, st.W, st.pt, C.H,
      [&](const Geo& g, df2* hh) { r2 = g.flat2; return begin_pairs<KERR, VOL, SEM>(p, g, st, hh); },
      [&](const dd& kP, const dd& kW) { if (VOL) v2 = sumsq(fst(kP), snd(kP), fst(kW), q(0.f)); },
      &h, &iP, &iQ, &iW);
  if (done) return true;
  const t3 P = st.P, Q = st.Q, W = st.W;
  st.P = add3(P, iP);
  st.Q = add3(Q, iQ);
  st.W = add3(W, iW);
  ++st.steps;
  const float2 n = st.P.h;
  const float nz = st.W.h.x;
  if (!(n.x == n.x) || !(nz == nz) || !(st.Q.h.x == st.Q.h.x)) {
    st.flags |= ST_RAY_CAPTURED;
    return true;
  }
  const float pz0 = W.h.x;
  const bool through = (pz0 < 0.f && nz > 0.f) || (pz0 > 0.f && nz < 0.f);
  if constexpr (SEM == ST_SEM_DRAFT) {
    // |x|^2 to a float's precision; as a pair where the gas or the escape sphere asks
    const float r2f = fmaf(n.x, n.x, fmaf(n.y, n.y, nz * nz));
    const bool far = r2f > 0.9999f * st.r_esc.hi * st.r_esc.hi;
    const df2 r2n = (VOL || far) ? sumsq(fst(top(st.P)), snd(top(st.P)), fst(top(st.W)), q(0.f)) : q(r2f);
    if constexpr (VOL) {
      if (st.steps == st.stop) return true;
      if (st.stop < 0) start_gas(p, P, Q, W, iP, iQ, iW, r2, r2n, mul(h, max_(sqrt_(v2), q(1e-20f))), st, *gas, lane);
    } else {
      if (p.disc_on && through && lt(df2{0.00100000005f, -4.74974504e-11f}, st.alpha))
        cross_pairs(p, P, Q, W, p.emitter == ST_EMIT_KEPLER, st);
    }
    if (p.exit_landing && far && lt(mul(st.r_esc, st.r_esc), r2n)) {
      st.P = P;
      st.Q = Q;
      st.W = W;
      st.land_h = h;
      st.flags |= ST_RAY_ESCAPED;
      return true;
    }
  } else {
    if (p.disc_on && through) cross_pairs(p, P, Q, W, p.emitter == ST_EMIT_KEPLER, st);
    st.lambda = add(st.lambda, h);
    const df2 rn = sqrt_(sumsq(fst(top(st.P)), snd(top(st.P)), fst(top(st.W)), q(0.f)));
    const df2 cb{2.00001001f, -1.34506226e-8f};  // 2.00001
    const bool in = !st.inside0 && !lt(cb, rn), out = !in && !lt(rn, st.inside0 ? cb : st.r_esc);
    if (in || out) {
      st.P = P;
      st.Q = Q;
      st.W = W;
      st.land_h = h;
      st.flags |= out && !st.inside0 ? ST_RAY_ESCAPED : ST_RAY_CAPTURED;
      return true;
    }
  }
  return false;
}

// Blocks of one warp: a quarter of a tile of trace_pixel_kernel's grid, so a
// frame of a few hundred tiles still spreads over all SMs and an SM takes the
// next warp as soon as one ends.  12 warps an SM leave 168 registers a thread.
constexpr int PAIR_BLOCK = 32;
#ifndef ST_PAIR_MINB
#define ST_PAIR_MINB 12
#endif

// One thread per pixel, as trace_pixel_kernel (RK4, no layer, no buckets).
template <int KERR, int VOL, int SEM>
__global__ void __launch_bounds__(PAIR_BLOCK, ST_PAIR_MINB) trace_pairs_kernel(const __grid_constant__ TraceParams p, int bx, int by) {
  constexpr int PREC = ST_PREC_FP64;
  int t = blockIdx.y * (gridDim.x >> 2) + (blockIdx.x >> 2);  // tile of the grid
  const int gx = gridDim.x >> 2;
  if (p.tile_order) t = __ldg(p.tile_order + t);
  const int in_tile = (blockIdx.x & 3) * 32 + threadIdx.x;
  int i = (t % gx) * bx + in_tile % bx, j = (t / gx) * by + in_tile / bx;
  if (p.box_cols > 0) {
    if (i >= p.box_cols || j >= p.box_rows) i = p.width;  // idle
    i += p.box_col0;
    j += p.box_row0;
  }
  if (p.pix_list) {
    const int k = blockIdx.x * 32 + threadIdx.x;
    const int pix = k < *p.n_list ? p.pix_list[k] : -1;
    i = pix >= 0 ? pix % p.width : p.width;
    j = pix >= 0 ? pix / p.width : 0;
  }
  const bool live = i < p.width && j < p.height;
  int base = 0;
  PairRay st;
  bool run = false;
  if (live) {
    CamView cam{p.pos, p.Ef, p.Er, p.Eu, p.U, p.r_escape, p.nmax};
    if (p.frames) {
      const FrameCam& fc = p.frames[blockIdx.z];
      cam = CamView{fc.pos, fc.Ef, fc.Er, fc.Eu, fc.U, fc.r_escape, fc.nmax};
      base = blockIdx.z * p.frame_stride;
    }
    RayState<double> s0;
    init_ray<PREC, KERR, SEM>(p, cam, i, j, s0);
    set_state(s0.y, st);
    st.pt = pair_of(s0.pt);
    const double E = -s0.pt;
    st.iE = pair_of(1.0 / (fabs(E) > 1e-6 ? E : 1e-6));
    st.scam = pair_of(s0.scam);
    st.flags = s0.flags;
    st.r_floor = pair_of(s0.r_floor);
    st.inside0 = s0.inside0;
    st.r_esc = pair_of(cam.r_escape);
    st.nmax = cam.nmax;
    run = !final_at_launch<SEM>(p, st.flags);
    if (!run) st.flags |= ST_RAY_CAPTURED;
  }
  st.acc[0] = st.acc[1] = st.acc[2] = st.march = st.lambda = dfm::q(0.f);
  st.alpha = dfm::q(1.f);
  st.land_h = dfm::q(0.f);
  st.r_prev = dfm::q(-1.f);
  st.steps = st.gas = st.queued = 0;
  st.stop = -1;
  st.marching = 0;
  st.r_cross = -1.f;
  st.g_cross = 0.f;
  if constexpr (VOL) {
    __shared__ GasWarp g;
    const int lane = threadIdx.x;
    if (run) mark_ray(st, g, lane);
    for (;;) {
      if (run && !st.marching && step_pairs<KERR, VOL, SEM>(p, st, &g, lane)) run = false;
      if (st.marching) queue_gas(p, st, g, lane);
      const bool more = __any_sync(0xffffffffu, run || st.marching);
      if (__any_sync(0xffffffffu, st.queued == GAS_Q) || !more) {
        run = shade_queue(p, run, st, g, lane);
        if (run && st.stop < 0) mark_ray(st, g, lane);
        if (!__any_sync(0xffffffffu, run || st.marching)) break;
      }
    }
  } else {
    while (run && !step_pairs<KERR, VOL, SEM>(p, st, nullptr, 0)) {
    }
  }
  unsigned long long steps = 0, gas = 0, rays = 0;
  if (live) {
    RayState<double> s1;
    doubles(st.P, st.Q, st.W, s1.y);
    // after the loop, for all rays of the warp together: inside it each ray lands
    // at a step of its own, and that double code took a third of the kernel's time
    if (st.land_h.hi > 0.f)
      land_in_step<KERR>(s1.y, dbl(st.pt), p.M, p.a, dbl(st.land_h),
                         SEM == ST_SEM_RENDER && (st.flags & ST_RAY_CAPTURED) ? 2.00001 : dbl(st.r_esc));
    s1.pt = dbl(st.pt);
    s1.scam = dbl(st.scam);
#pragma unroll
    for (int k = 0; k < 3; ++k) s1.acc[k] = dbl(st.acc[k]);
    s1.alpha = dbl(st.alpha);
    s1.flags = st.flags;
    s1.guard_ray = KERR && SEM == ST_SEM_DRAFT && (st.flags & ST_RAY_GRAZE) && p.crit_band > 0.0;
    s1.r_cross = st.r_cross;
    s1.g_cross = st.g_cross;
    s1.steps = st.steps;
    s1.fp64_steps = 0;
    s1.lambda = dbl(st.lambda);
    const int pix = base + j * p.width + i;
    finish_ray<PREC, KERR, SEM, 0>(p, s1, pix, p.frames ? pix : j * p.width + i);
    steps = st.steps; gas = st.gas; rays = 1;
  }
  flush_counters(p, steps, 0, gas, rays);
}

template <int KERR, int VOL, int SEM>
cudaError_t launch_pairs(const TraceParams& p, int bx, int by, cudaStream_t s) {
  if (bx <= 0 || by <= 0 || bx * by != 128) { bx = 16; by = 8; }
  const int w = p.box_cols > 0 ? p.box_cols : p.width, h = p.box_cols > 0 ? p.box_rows : p.height;
  dim3 grid(4 * ((w + bx - 1) / bx), (h + by - 1) / by);
  if (p.pix_list) grid = dim3((unsigned)(((long long)p.width * p.height + 127) / 128 * 4), 1);
  else if (p.frames) grid.z = (unsigned)(p.n_frames > 0 ? p.n_frames : 1);
  trace_pairs_kernel<KERR, VOL, SEM><<<grid, PAIR_BLOCK, 0, s>>>(p, bx, by);
  return cudaGetLastError();
}

}  // namespace

// The rule: RK4 frames of the pixel schedule whose lengths and times keep every
// intermediate of the right-hand side (up to r^4 and 1 / r^2, with 48 bits
// below) far inside a float's exponent, and whose gas absorbs (with a negative
// opacity e^-tau grows beyond a float's range).  Everything else -- the adaptive
// integrators, the layered engine's layer, depth buckets, the persistent queue
// and scenes in other units -- stays on the all-double kernels.
bool pairs_take(const Variant& v, const TraceParams& p) {
  return v.prec == ST_PREC_FP64 && v.sched == ST_SCHED_PIXEL && p.order == 4 && p.nb == 0 && !p.layer &&
         p.M >= 1.0 / 64 && p.M <= 64.0 && p.pair_range && p.dt >= 1e-5 && p.dt <= 100.0 &&
         p.tspan <= 1e7 && (!p.vol_on || p.opac >= 0.0);
}

cudaError_t launch_trace_pairs(const Variant& v, const TraceParams& p, int bx, int by, cudaStream_t s) {
  if (v.sem == ST_SEM_RENDER) return launch_pairs<0, 0, ST_SEM_RENDER>(p, bx, by, s);
  if (v.kerr) return v.vol ? launch_pairs<1, 1, ST_SEM_DRAFT>(p, bx, by, s) : launch_pairs<1, 0, ST_SEM_DRAFT>(p, bx, by, s);
  return v.vol ? launch_pairs<0, 1, ST_SEM_DRAFT>(p, bx, by, s) : launch_pairs<0, 0, ST_SEM_DRAFT>(p, bx, by, s);
}

}  // namespace st
