// st_trace_split.cuh -- small FP32 gas frames: a warp that integrates and three
// that shade, for the same 32 rays.
//
// A frame of fewer rays than the GPU holds is as slow as its longest ray, and a
// ray that crosses gas was a chain of integration (711 cycles a step at 64x36)
// and gas samples (another 970: arctangent, eight gathers from L2, the emitter,
// the Planck factor).  The geodesic does not depend on the gas, so here one warp
// integrates SPLIT_K steps of its rays into one half of a buffer in shared
// memory while three others shade the half before: they walk the sampled points
// along the steps, evaluate the samples (their absorption, radiance and colour,
// which do not depend on what lies in front) in parallel, and one of them blends
// each ray's samples in order.  A ray found opaque ends with the state of that
// sample's step, from the buffer; the steps that the integrator took beyond are
// dropped.  The arithmetic of steps and samples is the pixel kernel's: 120 random
// gas frames had the same bits as that kernel gave them.
// 64x36 Kerr gas: 2.05 -> 1.07 ms (an earlier build 1.01; there 1.16 with 8 steps a
// batch, 1.10 with seven shading warps).
#pragma once

#include "st_kernels.cuh"

namespace st {

constexpr int SPLIT_K = 16;       // steps of a batch
constexpr int SPLIT_SHADERS = 3;  // warps that shade
constexpr int SPLIT_SLOTS = 18;   // samples of a ray that are evaluated together

struct SplitBlock {
  float y[2][SPLIT_K + 1][6][32];  // the states before and after a batch's steps
  float seg[2][SPLIT_K][32];       // a step's arc length where the gas is sampled, else -1
  int cnt[2][32], stop[2][32];     // a batch's steps; the one that left the ray opaque, or -1
  int have[2];                     // a batch has steps
  float2 samp[SPLIT_SLOTS][32];    // a sample's fraction of its step, and the step
  float aa[SPLIT_SLOTS][32], inte[SPLIT_SLOTS][32], col[SPLIT_SLOTS][3][32];
  float pt[32], scam[32], acc[4][32];
  int dead[32], gas[32];
};
// a sample's aa when it blends nothing: counted as taken, or on the axis and not
constexpr float SPLIT_NONE = -2.f, SPLIT_SKIP = -1.f;

// step_ray's gas: leaves the step for the shading warps.
struct RecordStep {
  float (*y)[6][32];
  float (*seg)[32];
  int* n;
  int lane;
  __device__ __forceinline__ bool operator()(const TraceParams& p, const float*, const float* yn, float r2p, float h,
                                             float vlen, RayState<float>&) const {
    const float r2n = yn[0] * yn[0] + yn[1] * yn[1] + yn[2] * yn[2];
    const float len = h * vlen;
    seg[*n][lane] = min_(r2p, r2n) < p.f.vol_rb2 && len < 64.f ? len : -1.f;
    ++*n;
#pragma unroll
    for (int c = 0; c < 6; ++c) y[*n][c][lane] = yn[c];
    return false;
  }
};

// MarchGas's walk over a batch's steps, for the samples of one ray (lane), and
// their shading.  All shading warps walk alike; warp w evaluates every third
// sample; warp 0 blends.
struct SplitShade {
  float march = 0.f;
  bool dead = false;
  float acc[3] = {0.f, 0.f, 0.f}, alpha = 1.f;
  int gas = 0;

  __device__ __forceinline__ static void sync() { asm volatile("bar.sync 1, %0;" ::"n"(32 * SPLIT_SHADERS) : "memory"); }

  __device__ __forceinline__ void batch(const TraceParams& p, SplitBlock& s, int c, int w, int lane) {
    const int n = s.cnt[c][lane];
    const float pt = s.pt[lane], scam = s.scam[lane], ds = p.f.ds_gas, zmax = p.f.zmax;
    int k = 0, stop = -1, guard = 0;
    bool in = false;  // within step k
    float t = 0.f, seg = 0.f, inv_seg = 0.f;
    while (true) {
      int m = 0;
      while (m < SPLIT_SLOTS && k < n && !dead) {
        if (!in) {
          seg = s.seg[c][k][lane];
          t = ds - march;
          if (seg < 0.f) { ++k; continue; }
          if (t > seg) { march += seg; ++k; continue; }
          inv_seg = 1.f / seg;
          guard = 0;
          in = true;
        }
        const float fs = t * inv_seg;
        const float z0 = s.y[c][k][2][lane], z1 = s.y[c][k + 1][2][lane];
        if (fabsf(z0 + fs * (z1 - z0)) < zmax) {
          if (m % SPLIT_SHADERS == w) s.samp[m][lane] = make_float2(fs, __int_as_float(k));
          ++m;
        }
        t += ds;
        ++guard;
        if (!(guard < 8192 && t <= seg)) {
          march = seg - (t - ds);
          in = false;
          ++k;
        }
      }
#pragma unroll 1
      for (int q = w; q < m; q += SPLIT_SHADERS) {
        const float2 a = s.samp[q][lane];
        const float fs = a.x;
        const int j = __float_as_int(a.y);
        float yp[6], yn[6];
#pragma unroll
        for (int e = 0; e < 5; ++e) { yp[e] = s.y[c][j][e][lane]; yn[e] = s.y[c][j + 1][e][lane]; }
        const float sx = yp[0] + fs * (yn[0] - yp[0]);
        const float sy = yp[1] + fs * (yn[1] - yp[1]);
        const float sz = yp[2] + fs * (yn[2] - yp[2]);
        const float scyl = sqrt_(sx * sx + sy * sy);
        float aa = SPLIT_SKIP;
        if (scyl > 1e-6f) {
          GasSample<float> o;
          aa = SPLIT_NONE;
          if (gas_sample(p, yp, yn, fs, sx, sy, sz, scyl, pt, scam, &o)) {
            aa = o.aa;
            s.inte[q][lane] = o.inte;
            s.col[q][0][lane] = o.col.x; s.col[q][1][lane] = o.col.y; s.col[q][2][lane] = o.col.z;
          }
        }
        s.aa[q][lane] = aa;
      }
      sync();
      if (w == 0) {
        for (int q = 0; q < m && !dead; ++q) {
          const float aa = s.aa[q][lane];
          if (aa != SPLIT_SKIP) ++gas;
          if (!(aa == SPLIT_SKIP || aa == SPLIT_NONE))
            blend_sample(p, GasSample<float>{aa, s.inte[q][lane], make_float4(s.col[q][0][lane], s.col[q][1][lane],
                                                                              s.col[q][2][lane], 0.f)},
                         acc, &alpha);
          if (!(alpha > 0.003f)) {
            dead = true;
            if (alpha < 0.003f) stop = __float_as_int(s.samp[q][lane].y);
          }
        }
        s.dead[lane] = dead;
        s.stop[c][lane] = stop;
      }
      sync();
      dead = s.dead[lane] != 0;
      if (!__any_sync(0xffffffffu, !dead && k < n)) break;
    }
  }
};

// One 8 x 4 tile of pixels a block.
template <int KERR>
__global__ void __launch_bounds__(32 * (1 + SPLIT_SHADERS)) trace_split_kernel(const __grid_constant__ TraceParams p) {
  constexpr int PREC = ST_PREC_FP32, SEM = ST_SEM_DRAFT;
  __shared__ SplitBlock s;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = blockIdx.x * 8 + (lane & 7), j = blockIdx.y * 4 + (lane >> 3);
  const bool live = i < p.width && j < p.height;
  RayState<float> st;
  SplitShade shade;
  bool run = false, ended = false;
  int flags0 = 0, steps0 = 0, before = 0;  // steps at the start of this batch and of the one before
  if (warp == 0) {
    st.flags = st.steps = 0;
    st.pt = st.scam = 0.f;
#pragma unroll
    for (int c = 0; c < 6; ++c) st.y[c] = 0.f;
    if (live) {
      const CamView cam{p.pos, p.Ef, p.Er, p.Eu, p.U, p.r_escape, p.nmax};
      init_ray<PREC, KERR, SEM>(p, cam, i, j, st);
      st.pix = j * p.width + i;
      run = !final_at_launch<SEM>(p, st.flags);
      if (!run) st.flags |= ST_RAY_CAPTURED;
      flags0 = st.flags;
    }
    s.pt[lane] = st.pt;
    s.scam[lane] = st.scam;
  }
  __syncthreads();
  for (int it = 0;; ++it) {
    const int b = it & 1;
    if (warp == 0) {
      const bool any = __any_sync(0xffffffffu, run);
      int n = 0;
      if (any) {
        steps0 = st.steps;
#pragma unroll
        for (int c = 0; c < 6; ++c) s.y[b][0][c][lane] = st.y[c];
        const RecordStep rec{s.y[b], s.seg[b], &n, lane};
#pragma unroll 1
        for (int k = 0; k < SPLIT_K && run; ++k)
          if (step_ray<PREC, KERR, 1, SEM, 4, 0, 0, RecordStep>(p, st, rec)) run = false;
      }
      s.cnt[b][lane] = n;
      if (lane == 0) s.have[b] = any;
    } else if (it > 0 && s.have[b ^ 1]) {
      shade.batch(p, s, b ^ 1, warp - 1, lane);
    }
    __syncthreads();
    if (warp == 0) {
      if (it > 0 && s.have[b ^ 1] && !ended && s.stop[b ^ 1][lane] >= 0) {
        const int k = s.stop[b ^ 1][lane] + 1;
#pragma unroll
        for (int c = 0; c < 6; ++c) st.y[c] = s.y[b ^ 1][k][c][lane];
        st.steps = before + k;
        st.flags = flags0;
        run = false;
        ended = true;
      }
      before = steps0;
    }
    if (!s.have[b]) break;
  }
  if (warp == 1) {
#pragma unroll
    for (int c = 0; c < 3; ++c) s.acc[c][lane] = shade.acc[c];
    s.acc[3][lane] = shade.alpha;
    s.gas[lane] = shade.gas;
  }
  __syncthreads();
  if (warp != 0) return;
  unsigned long long steps = 0, gas = 0, rays = 0;
  if (live) {
#pragma unroll
    for (int c = 0; c < 3; ++c) st.acc[c] = s.acc[c][lane];
    st.alpha = s.acc[3][lane];
    st.gas = s.gas[lane];
    finish_ray<PREC, KERR, SEM, 0>(p, st, st.pix, st.pix);
    steps = st.steps; gas = st.gas; rays = 1;
  }
  flush_counters(p, steps, 0, gas, rays);
}

// The rule: whole FP32 gas frames of the pixel schedule with so few rays in flight
// that a step's latency and not its instructions are the frame's time.  Where the
// line lies depends on how many of a ray's steps have samples, so it was set by
// random scenes (spins, radii from 1.3 to 90 M, slabs, opacities to 3,000, strides to
// 16, steps to 0.2; 10 to 49 a size).  Times against the pixel kernel's, geometric
// mean, and how many frames of 0.1 ms or more were slower:
//   64x36 0.79, none; 128x72 0.65, none; 160x90 0.69, none; 200x113 (22,600 rays)
//   0.86, none, shorter ones by up to 28 us; 240x135 (32,400) 0.84, 3, by up to 117 us;
//   280x158 1.01, 3; 300x169 1.14, 6; 256x256 1.10, 10, by up to 0.5 ms.
// Near the horizon of a fast hole a step's samples run to hundreds, most of them
// below the slab's inner edge, and all shading warps walk past all of them: 120x90
// from 55 M with samples every step or two, spin 0.95 0.71 to 0.80 of the pixel
// kernel's time, 0.99 0.94 to 1.24, 0.998 1.15 to 1.34 (every fourth step: 0.96).
constexpr long long SPLIT_RAYS = 24576;
inline bool split_takes(const Variant& v, const TraceParams& p) {
  return v.vol && v.sem == ST_SEM_DRAFT && v.sched == ST_SCHED_PIXEL && p.order == 4 && p.nb == 0 && !p.layer &&
         !p.pix_list && !p.frames && p.box_cols <= 0 && (p.a <= 0.96 * p.M || p.ds_gas >= 3.5 * p.dt) &&
         (long long)p.width * p.height * (p.beside > 1 ? p.beside : 1) <= SPLIT_RAYS;
}
inline cudaError_t launch_split(const Variant& v, const TraceParams& p, cudaStream_t s) {
  const dim3 grid((p.width + 7) / 8, (p.height + 3) / 4);
  if (v.kerr) trace_split_kernel<1><<<grid, 32 * (1 + SPLIT_SHADERS), 0, s>>>(p);
  else trace_split_kernel<0><<<grid, 32 * (1 + SPLIT_SHADERS), 0, s>>>(p);
  return cudaGetLastError();
}

}  // namespace st
