// st_fluid.cu -- the live fluid-simulated accretion disc (DiscFluidSim /
// step_sim!, src/disc_sim.jl): a 2-D stable-fluids solver on the gas volume's
// own (log s, phi) grid whose surface density is extruded through the
// vertical envelope into the context's density texture, which the trace
// kernels then sample unchanged.
//
// One step of the reference is ~20 dispatches (src/disc_sim.jl:287-320):
// velocity advection, forcing, divergence, 2 ceil(jacobi / 2) Jacobi sweeps,
// gradient subtraction, forward and backward density advection, the
// MacCormack combine and the extrusion.  Here the steps of a call are one
// cooperative launch (fluid_steps_kernel) of two phases a step:
//
//   pressure   a tile and a halo as wide as its sweeps in shared memory: the
//              divergence, every sweep on the shrinking valid region, and the
//              gradient subtraction (in passes where the sweeps are many);
//              blocks without a tile meanwhile evaluate the noise that the
//              next phase needs, which depends on the clock alone;
//   advection  MacCormack advection and relaxation of the surface density, and
//              the next step's velocity advection and forcing, both of which
//              need the projected velocity of all cells and nothing more.
//              The forward density at the four corners of a cell's backward
//              point is recomputed in registers, so the forward and backward
//              fields never go through memory.
//
// The extrusion of the density through the nz envelope cells follows the last
// step of a launch: the texture is read by later work of the stream only.
//
// What bounds it: a grid is some ten thousand cells, so a step is latency, not
// work.  As four launches (velocity, divergence, pressure, density) a step
// was 21 us, most of it launch and drain; the two grid barriers that are left
// cost about 1.5 us each.  256 x 64 cells, 8 sweeps: 20.5 -> 8.9 us a step of
// 100 in a call, 21.4 -> 16.3 us a single one.  Grids that fill the GPU several
// times over take the same phases as launches of their own.
//
// Each cell's arithmetic is the reference's, in the same order, in float;
// this unit is compiled without multiply-add contraction so every operation
// rounds as written.  Index arithmetic is 1-based in the formulas, as in the
// reference; field (i, j) lives at (i - 1) + nr (j - 1).
//
// The simulation clock lives on the device (a step of parity q reads t[q] and
// leaves t[1 - q] = t[q] + dt) and the density ping-pongs between two buffers
// by the same parity.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "st_internal.h"

namespace st {
namespace fluid {

// ---- device helpers (src/disc_sim.jl:80-134) ---------------------------------

__device__ __forceinline__ float hash01(int x, int y, int z) {
  uint32_t h = ((uint32_t)x * 0x8da6b343u) ^ ((uint32_t)y * 0xd8163841u) ^ ((uint32_t)z * 0xcb1ab31fu);
  h ^= h >> 13;
  h *= 0x9e3779b9u;
  h ^= h >> 16;
  return (float)(h & 0x00ffffffu) * 5.9604645e-8f;
}

// Value noise on the hashed lattice, smoothstep-weighted trilinear.
__device__ __forceinline__ float noise3(float x, float y, float z) {
  const float flx = floorf(x), fly = floorf(y), flz = floorf(z);
  const int ix = (int)flx, iy = (int)fly, iz = (int)flz;
  float fx = x - flx, fy = y - fly, fz = z - flz;
  fx = fx * fx * (3.0f - 2.0f * fx);
  fy = fy * fy * (3.0f - 2.0f * fy);
  fz = fz * fz * (3.0f - 2.0f * fz);
  const int i1 = ix + 1, j1 = iy + 1, k1 = iz + 1;
  const float h000 = hash01(ix, iy, iz), h100 = hash01(i1, iy, iz);
  const float h010 = hash01(ix, j1, iz), h110 = hash01(i1, j1, iz);
  const float h001 = hash01(ix, iy, k1), h101 = hash01(i1, iy, k1);
  const float h011 = hash01(ix, j1, k1), h111 = hash01(i1, j1, k1);
  const float c00 = h000 + fx * (h100 - h000);
  const float c10 = h010 + fx * (h110 - h010);
  const float c01 = h001 + fx * (h101 - h001);
  const float c11 = h011 + fx * (h111 - h011);
  const float c0 = c00 + fy * (c10 - c00);
  const float c1 = c01 + fy * (c11 - c01);
  return c0 + fz * (c1 - c0);
}

__device__ __forceinline__ int jmod(int a, int n) {
  const int r = a % n;
  return r < 0 ? r + n : r;
}

// jmod for a in [-n, 2n) by compare (the footprints and halos stay there);
// anything else falls back to the division.
__device__ __forceinline__ int jwrap(int a, int n) {
  const int b = a < 0 ? a + n : (a >= n ? a - n : a);
  return (b >= 0 && b < n) ? b : jmod(a, n);
}

// Corners of the bilinear footprint of (x, y): radius clamped, phi periodic.
struct Foot {
  int o00, o10, o01, o11;  // storage offsets of (i0, j0a), (i0+1, j0a), (i0, j1a), (i0+1, j1a)
  int i0, j0a, j1a;        // the corners' 1-based indices
  float tx, ty;
};

__device__ __forceinline__ Foot footprint(float x, float y, int nr, int nphi) {
  x = fminf(fmaxf(x, 1.0f), (float)nr);
  const int i0 = min(max((int)floorf(x), 1), nr - 1);
  Foot f;
  f.tx = x - (float)i0;
  const float yw = y - (float)nphi * floorf((y - 1.0f) / (float)nphi);
  const int j0 = (int)floorf(yw);
  f.ty = yw - (float)j0;
  const int j0a = jwrap(j0 - 1, nphi) + 1;
  const int j1a = jwrap(j0, nphi) + 1;
  f.i0 = i0; f.j0a = j0a; f.j1a = j1a;
  f.o00 = (i0 - 1) + nr * (j0a - 1);
  f.o10 = f.o00 + 1;
  f.o01 = (i0 - 1) + nr * (j1a - 1);
  f.o11 = f.o01 + 1;
  return f;
}

// (plain pointers: the fields change within a launch, and the read-only path
// could return what it held before a barrier)
__device__ __forceinline__ float bilerp(const float* f, const Foot& q) {
  const float a = f[q.o00] + q.tx * (f[q.o10] - f[q.o00]);
  const float b = f[q.o01] + q.tx * (f[q.o11] - f[q.o01]);
  return a + q.ty * (b - a);
}

// ---- kernels -------------------------------------------------------------------

struct Fields {
  int nr, nphi, nz;
  float* vu; float* vv;         // velocity after projection (cells / M-time)
  float* vu2; float* vv2;       // advected + forced velocity
  float* dens[2];               // surface density, ping-pong by parity
  const float* base;            // radial profile (relaxation target)
  const float* shear;           // [nr] Keplerian shear, phi cells / M-time
  const float* env;             // [nr][nz] vertical envelope, (nr, nz) column-major
  float* prs[2];                // pressure ping-pong and
  float* div;                   //   divergence, where the sweeps take several passes
  float* fu; float* fv;         // the forcing's curl noise for the next velocity phase
  float* tgt;                   // the relaxation target of the next density phase
  float* t;                     // [2] simulation clock by parity
  unsigned* count;              // arrivals at the grid barrier, never reset
  int* status;                  // set when a barrier's wait ran out
  int* fault;                   // and with it this word of the context, in host memory
  float* vol;                   // (nr, nphi, nz) density texture of the context
};

constexpr int THREADS = 512, WARPS = THREADS / 32;
constexpr int TI = 32;             // tile of the pressure phase along i (fastest)
constexpr int LOW = 8, TALL = 32;  // and along j: in the one launch, in launches by phase
// Sweeps per pass; halo = sweeps (+1 on the last pass).  The widest staged block
// is then 64 cells along i: a thread owns one column of it, every eighth row.
constexpr int MAX_SWEEPS = 15;
constexpr int COLS = TI + 2 * (MAX_SWEEPS + 1), ROWS = THREADS / COLS;
// Polls of a barrier, some seconds.  A constant of the kernel: as a parameter it
// made the polling loop, and with it a step of 256 x 64 cells, 1.3 % slower.
constexpr unsigned WAIT_LIMIT = 1u << 22;

// Floats of shared memory of a pass: p twice.
constexpr size_t tile_floats(int tj, int H) { return 2 * (size_t)(TI + 2 * H) * (tj + 2 * H); }
static_assert(tile_floats(TALL, MAX_SWEEPS + 1) * sizeof(float) <= 48 * 1024, "no opt-in needed");

// Tells the host, without a copy or a wait on its side: the next step of a solver
// and the next render of the context look at this word.
__device__ __forceinline__ void report_fault(const Fields& F) {
  *static_cast<volatile int*>(F.fault) = 1;
  __threadfence_system();
}

// All blocks of the (cooperative) launch; `target` counts their arrivals since
// the counter's creation, modulo 2^32.  False, for the whole block, when the
// wait ran out; the fields are then not to be used.  (A word a block that every
// block polls instead of one counter took 30,000 cycles: 152 x 152 polls.)
template <unsigned LIMIT>
__device__ __forceinline__ bool grid_barrier(const Fields& F, unsigned target) {
  int out = 0;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned v;
    asm volatile("atom.add.release.gpu.global.u32 %0, [%1], 1;" : "=r"(v) : "l"(F.count) : "memory");
    unsigned polls = 0;
    while (true) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(F.count) : "memory");
      if ((int)(v - target) >= 0) break;
      if (++polls >= LIMIT) {
        out = 1;
        atomicExch(F.status, 1);
        report_fault(F);
        break;
      }
    }
  }
  return !__syncthreads_or(out);
}

// psi on a coarse lattice (~12-cell eddies) drifting in time; F = curl(psi z)
// (k_force!, src/disc_sim.jl:150-172).
constexpr float FORCE_SC = 0.085f, FORCE_E = 0.35f;
__device__ __forceinline__ float force_u(int i, int j, float t) {
  const float px = (float)i * FORCE_SC, py = (float)j * FORCE_SC, pz = t * 0.35f;
  const float dpy = noise3(px, py + FORCE_E, pz) - noise3(px, py - FORCE_E, pz);
  return dpy / (2.0f * FORCE_E);
}
__device__ __forceinline__ float force_v(int i, int j, float t) {
  const float px = (float)i * FORCE_SC, py = (float)j * FORCE_SC, pz = t * 0.35f;
  const float dpx = noise3(px + FORCE_E, py, pz) - noise3(px - FORCE_E, py, pz);
  return -dpx / (2.0f * FORCE_E);
}
__device__ __forceinline__ float target(const Fields& F, int idx, int i, int j, float t) {
  const float n = noise3((float)i * 0.11f, (float)j * 0.11f, t * 0.25f);
  return F.base[idx] * expf(1.2f * (2.0f * n - 1.0f));
}

// Semi-Lagrangian velocity advection, then forcing + drag + edge taper
// (k_advect_vel!, k_force!: src/disc_sim.jl:136-172).
__device__ __forceinline__ void velocity_cell(const Fields& F, int idx, int i, int j, float fu, float fv, float dt,
                                              float amp, float drag) {
  const int nr = F.nr, nphi = F.nphi;
  const float x = (float)i - dt * F.vu[idx];
  const float y = (float)j - dt * (F.vv[idx] + F.shear[i - 1]);
  const Foot q = footprint(x, y, nr, nphi);
  float u = bilerp(F.vu, q);
  float v = bilerp(F.vv, q);
  float edge = fminf((float)i - 1.0f, (float)(nr - i)) * 0.125f;
  edge = fminf(fmaxf(edge, 0.0f), 1.0f);
  const float damp = expf(-drag * dt);
  u = (u + dt * amp * fu * edge) * damp * edge;
  v = (v + dt * amp * fv * edge) * damp;
  F.vu2[idx] = u;
  F.vv2[idx] = v;
}

// One tile's `sweeps` Jacobi sweeps (k_jacobi!, src/disc_sim.jl:184-192).  The
// first pass forms the divergence (k_div!) and starts from the sweep from p = 0
// (0.25 ((((0 + 0) + 0) + 0) - dv) = 0.25 (-dv)) or, with no sweeps at all, from
// p = 0; later ones read p from prs[src].  The last pass subtracts the gradient
// (k_subgrad!, src/disc_sim.jl:194-203): (vu, vv) = (vu2, vv2) - grad p / 2; the
// others write p to prs[1 - src].  A thread keeps its cells' divergence in
// registers over the sweeps, and no cell's place needs a division.
template <int TJ>
__device__ __forceinline__ void pressure_tile(const Fields& F, int bi, int bj, bool first, bool any, int src,
                                              int sweeps, bool last, float* sm) {
  const int nr = F.nr, nphi = F.nphi;
  const int H = sweeps + (last ? 1 : 0);
  const int RI = TI + 2 * H, RJ = TJ + 2 * H;
  float* cur = sm;
  float* nxt = sm + RI * RJ;
  constexpr int MAX_CELLS = (TJ + 2 * (MAX_SWEEPS + 1) + ROWS - 1) / ROWS;
  const int li = threadIdx.x % COLS, row = threadIdx.x / COLS;
  const int gi = bi * TI + 1 - H + li;  // global i of the thread's column
  const int j0 = bj * TJ - H;           // global (unwrapped, 0-based) j of local row 0
  const bool in = li < RI && gi >= 1 && gi <= nr;
  // clamped radial neighbours
  const int up = gi + 1 <= nr ? 1 : 0, dn = gi - 1 >= 1 ? -1 : 0;
  const int edge = in ? min(li, RI - 1 - li) : -1;
  const bool mine = in && li >= H && li < H + TI;
  const float* pin = src ? F.prs[1] : F.prs[0];
  float* pout = src ? F.prs[0] : F.prs[1];
  float D[MAX_CELLS], pv[MAX_CELLS];
#pragma unroll
  for (int c = 0; c < MAX_CELLS; ++c) {
    const int lj = row + c * ROWS;
    D[c] = pv[c] = 0.0f;
    if (lj >= RJ || !in) continue;
    const int j = jwrap(j0 + lj, nphi), o = (gi - 1) + nr * j;
    if (first) {
      const int jp = j + 1 < nphi ? o + nr : gi - 1, jm = j > 0 ? o - nr : (gi - 1) + nr * (nphi - 1);
      D[c] = 0.5f * (F.vu2[o + up] - F.vu2[o + dn] + F.vv2[jp] - F.vv2[jm]);
      if (any) pv[c] = 0.25f * (0.0f - D[c]);
    } else {
      D[c] = F.div[o];
      pv[c] = pin[o];
    }
  }
  float* at = cur + li + RI * row;  // the thread's cells lie ROWS rows apart
#pragma unroll
  for (int c = 0; c < MAX_CELLS; ++c)
    if (li < RI && row + c * ROWS < RJ) at[c * ROWS * RI] = pv[c];
  __syncthreads();
  for (int k = 1; k <= sweeps; ++k) {
    // valid region after this sweep: margin k from every side of the staged block
    if (edge >= k) {
      const float* a = cur + li + RI * row;
      float* b = nxt + li + RI * row;
#pragma unroll
      for (int c = 0; c < MAX_CELLS; ++c) {
        const int lj = row + c * ROWS;
        if (lj < k || lj >= RJ - k) continue;
        const float* p = a + c * ROWS * RI;
        b[c * ROWS * RI] = 0.25f * (p[up] + p[dn] + p[RI] + p[-RI] - D[c]);
      }
    }
    __syncthreads();
    float* tmp = cur; cur = nxt; nxt = tmp;
  }
  // the tile's own cells
#pragma unroll
  for (int c = 0; c < MAX_CELLS; ++c) {
    const int lj = row + c * ROWS;
    if (!mine || lj < H || lj >= H + TJ || j0 + lj >= nphi) continue;
    const int o = (gi - 1) + nr * (j0 + lj);
    const float* p = cur + li + RI * lj;
    if (!last) {
      pout[o] = p[0];
      if (first) F.div[o] = D[c];
      continue;
    }
    F.vu[o] = F.vu2[o] - 0.5f * (p[up] - p[dn]);
    F.vv[o] = F.vv2[o] - 0.5f * (p[RI] - p[-RI]);
  }
  __syncthreads();
}

// Forward semi-Lagrangian density sample at cell (ci, cj) (k_adv_scalar!).
__device__ __forceinline__ float advect_at(const Fields& F, const float* d, int ci, int cj, float dt) {
  const int o = (ci - 1) + F.nr * (cj - 1);
  const float x = (float)ci - dt * F.vu[o];
  const float y = (float)cj - dt * (F.vv[o] + F.shear[ci - 1]);
  return bilerp(d, footprint(x, y, F.nr, F.nphi));
}

// MacCormack density step + relaxation (k_adv_scalar! forward and backward,
// k_maccormack!: src/disc_sim.jl:205-251); returns the new value.
__device__ __forceinline__ float density_cell(const Fields& F, int parity, int idx, int i, int j, float tgt, float dt,
                                              float relax) {
  const int nr = F.nr, nphi = F.nphi;
  const float* d = parity ? F.dens[1] : F.dens[0];
  float* dout = parity ? F.dens[0] : F.dens[1];
  // forward: d1 = d at the backtraced point; its corners bound the limiter
  const float x = (float)i - dt * F.vu[idx];
  const float y = (float)j - dt * (F.vv[idx] + F.shear[i - 1]);
  const Foot q = footprint(x, y, nr, nphi);
  const float d1 = bilerp(d, q);
  const float lo = fminf(fminf(d[q.o00], d[q.o10]), fminf(d[q.o01], d[q.o11]));
  const float hi = fmaxf(fmaxf(d[q.o00], d[q.o10]), fmaxf(d[q.o01], d[q.o11]));
  // backward: the forward field re-advected by -dt, sampled at the cell
  const float ndt = -dt;
  const float xb = (float)i - ndt * F.vu[idx];
  const float yb = (float)j - ndt * (F.vv[idx] + F.shear[i - 1]);
  const Foot qb = footprint(xb, yb, nr, nphi);
  const float c00 = advect_at(F, d, qb.i0, qb.j0a, dt), c10 = advect_at(F, d, qb.i0 + 1, qb.j0a, dt);
  const float c01 = advect_at(F, d, qb.i0, qb.j1a, dt), c11 = advect_at(F, d, qb.i0 + 1, qb.j1a, dt);
  const float ea = c00 + qb.tx * (c10 - c00);
  const float eb = c01 + qb.tx * (c11 - c01);
  const float d2 = ea + qb.ty * (eb - ea);
  const float a = fminf(fmaxf(d1 + 0.5f * (d[idx] - d2), lo), hi);
  const float dn = fmaxf(a + relax * dt * (tgt - a), 0.0f);
  dout[idx] = dn;
  return dn;
}

// The envelope loads of a batch are issued before its stores, so the column's
// latency is paid once per eight cells rather than per cell (k_extrude!,
// src/disc_sim.jl:253-266).
__device__ __forceinline__ void extrude(const Fields& F, int idx, int i, float dn) {
  const size_t plane = (size_t)F.nr * F.nphi;
  const float* __restrict__ env = F.env + (i - 1);
  float* __restrict__ vol = F.vol + idx;
  int k = 0;
  for (; k + 8 <= F.nz; k += 8) {
    float e[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) e[q] = __ldg(env + (size_t)F.nr * (k + q));
#pragma unroll
    for (int q = 0; q < 8; ++q) vol[plane * (k + q)] = dn * e[q];
  }
  for (; k < F.nz; ++k) vol[plane * k] = dn * __ldg(env + (size_t)F.nr * k);
}

// `nsteps` steps from the state of `parity`; `sweeps` Jacobi sweeps each
// (even, or 0); `base` barrier arrivals before this launch.  Work of a phase is
// dealt in whole warps, round the blocks, so that a few hundred warps of work
// occupy every SM.
template <int BLOCKS_SM, unsigned LIMIT>
__global__ void __launch_bounds__(THREADS, BLOCKS_SM)
    fluid_steps_kernel(Fields F, int parity, int nsteps, float dt, int sweeps, float amp, float drag, float relax,
                       unsigned base) {
  extern __shared__ float sm[];
  const unsigned nr = F.nr, n = nr * (unsigned)F.nphi;
  const unsigned warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (*static_cast<volatile int*>(F.status)) {  // an earlier launch's wait ran out
    if (blockIdx.x == 0 && threadIdx.x == 0) report_fault(F);
    return;
  }
  unsigned bars = base;
  // f(kind, idx, i, j) for `kinds` kinds of work on every cell, by blocks b of nb
  auto cells = [&](unsigned kinds, unsigned b, unsigned nb, auto f) {
    const unsigned per = (n + 31) / 32, jobs = kinds * per;
    for (unsigned w = warp * nb + b; w < jobs; w += WARPS * nb) {
      const unsigned kind = w / per, idx = (w - kind * per) * 32 + lane;
      if (idx >= n) continue;
      const unsigned j = idx / nr;
      f((int)kind, (int)idx, (int)(idx - j * nr) + 1, (int)j + 1);
    }
  };
  const int gx = (F.nr + TI - 1) / TI, tiles = gx * ((F.nphi + LOW - 1) / LOW);
  // blocks that have no tile evaluate the noise, if they are a fair share of the
  // grid; else the advection does as it goes
  const int spare = (int)gridDim.x - tiles;
  const bool apart = spare * 4 >= (int)gridDim.x;
  float t = parity ? F.t[1] : F.t[0];
  cells(1, blockIdx.x, gridDim.x, [&](int, int idx, int i, int j) {
    velocity_cell(F, idx, i, j, force_u(i, j, t), force_v(i, j, t), dt, amp, drag);
  });
  if (!grid_barrier<LIMIT>(F, bars += gridDim.x)) return;
  for (int k = 0; k < nsteps; ++k) {
    const float tn = t + dt;
    const bool end = k + 1 == nsteps;
    if (blockIdx.x == 0 && threadIdx.x == 0) F.t[1 - parity] = tn;
    int left = sweeps > 0 ? sweeps - 1 : 0, src = 0;
    bool first = true;
    while (true) {
      const int m = min(left, MAX_SWEEPS);
      left -= m;
      for (int b = blockIdx.x; b < tiles; b += gridDim.x)
        pressure_tile<LOW>(F, b % gx, b / gx, first, sweeps > 0, src, m, left == 0, sm);
      if (left == 0) break;
      if (!grid_barrier<LIMIT>(F, bars += gridDim.x)) return;
      src = 1 - src;
      first = false;
    }
    if (apart && (int)blockIdx.x >= tiles)
      cells(end ? 1 : 3, blockIdx.x - tiles, spare, [&](int kind, int idx, int i, int j) {
        if (kind == 0) F.tgt[idx] = target(F, idx, i, j, t);
        else if (kind == 1) F.fu[idx] = force_u(i, j, tn);
        else F.fv[idx] = force_v(i, j, tn);
      });
    if (!grid_barrier<LIMIT>(F, bars += gridDim.x)) return;
    cells(end ? 1 : 2, blockIdx.x, gridDim.x, [&](int kind, int idx, int i, int j) {
      if (kind == 0) {
        const float dn =
            density_cell(F, parity, idx, i, j, apart ? F.tgt[idx] : target(F, idx, i, j, t), dt, relax);
        if (end) extrude(F, idx, i, dn);
      } else {
        velocity_cell(F, idx, i, j, apart ? F.fu[idx] : force_u(i, j, tn), apart ? F.fv[idx] : force_v(i, j, tn), dt,
                      amp, drag);
      }
    });
    if (!end && !grid_barrier<LIMIT>(F, bars += gridDim.x)) return;
    parity ^= 1;
    t = tn;
  }
}

// The phases as launches of their own, for grids that fill the GPU several times
// over: a barrier's microsecond is nothing there, and blocks that come and go
// keep the SMs fuller than a fixed few.  Blocks of the advection are 64 cells of
// a phi row; its z is 0 for the density (`end`: and extrusion), 1 for the next
// step's velocity.
__global__ void __launch_bounds__(THREADS) fluid_pressure_kernel(Fields F, int parity, float dt, bool first, bool any,
                                                                 int src, int sweeps, bool last) {
  extern __shared__ float sm[];
  if (first && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0)
    F.t[1 - parity] = (parity ? F.t[1] : F.t[0]) + dt;
  pressure_tile<TALL>(F, blockIdx.x, blockIdx.y, first, any, src, sweeps, last, sm);
}
__global__ void __launch_bounds__(64) fluid_advect_kernel(Fields F, int parity, int kind0, bool end, float dt,
                                                          float amp, float drag, float relax) {
  const int i = blockIdx.x * 64 + threadIdx.x + 1, j = blockIdx.y + 1;
  if (i > F.nr) return;
  const int idx = (i - 1) + F.nr * (j - 1);
  if (blockIdx.z + kind0 == 0) {
    const float dn = density_cell(F, parity, idx, i, j, target(F, idx, i, j, parity ? F.t[1] : F.t[0]), dt, relax);
    if (end) extrude(F, idx, i, dn);
  } else {
    // the clock of the step to come: after a density phase's, or the call's first
    const float t = (parity ^ (kind0 == 0 ? 1 : 0)) ? F.t[1] : F.t[0];
    velocity_cell(F, idx, i, j, force_u(i, j, t), force_v(i, j, t), dt, amp, drag);
  }
}

}  // namespace fluid
}  // namespace st

// ---- host side --------------------------------------------------------------

using namespace st::fluid;

struct st_fluid {
  st_context* ctx = nullptr;
  int device = 0;
  cudaStream_t stream = nullptr;
  int nr = 0, nphi = 0, nz = 0;
  float* block = nullptr;  // every field in one allocation
  Fields F{};
  int parity = 0;
  double forcing = 6.0, drag = 0.15, relax = 0.05;
  unsigned arrivals = 0;  // at the grid barrier, as the device counts them
  int num_sms = 0;
  long long steps = 0;
};

namespace {

constexpr int DENSE = 3;  // blocks an SM of the larger grids
constexpr int LAUNCH_STEPS = 1024;  // steps of one launch, some milliseconds

// The one-launch kernel for `blocks` blocks.  SPACETIME_GB300_FLUID_WAIT=1 in the
// environment takes the kernels whose barriers give up after one poll, so a test can
// make a wait run out (the blocks then leave the launch one by one, the fields are
// not to be used, and the solver and the context report it).
const void* steps_kernel(bool dense) {
  const char* e = std::getenv("SPACETIME_GB300_FLUID_WAIT");
  if (e && std::strcmp(e, "1") == 0)
    return dense ? (const void*)fluid_steps_kernel<DENSE, 1> : (const void*)fluid_steps_kernel<1, 1>;
  return dense ? (const void*)fluid_steps_kernel<DENSE, WAIT_LIMIT> : (const void*)fluid_steps_kernel<1, WAIT_LIMIT>;
}

// `nsteps` (<= LAUNCH_STEPS) steps from the current parity on stream s.
int launch_steps(st_fluid* f, float* vol, int nsteps, float dt, int jacobi, cudaStream_t s) {
  Fields F = f->F;
  F.vol = vol;
  // 2 ceil(jacobi / 2) sweeps (src/disc_sim.jl:305-308)
  int sweeps = jacobi > 0 ? 2 * ((jacobi + 1) / 2) : 0;
  // the first sweep needs no neighbours; the rest run in passes of at most MAX_SWEEPS
  const int rest = sweeps > 0 ? sweeps - 1 : 0;
  const int passes = std::max(1, (rest + MAX_SWEEPS - 1) / MAX_SWEEPS);
  // a block an SM, and no more than have two warps of cells, since the barriers'
  // cost grows with the blocks; where there are more tiles, blocks for each and
  // half as many for the noise; where the SMs do not hold those, launches by
  // phase with taller tiles, which stage 2.3 cells for each of their own (8
  // sweeps) and not 4.5.  us a step of 100: 192 x 256 cells 12.0 in one launch
  // (22.0 as four launches a step), 1024 x 512 cells 62.8 in one, 46.6 by phase
  // (61.5 as four)
  const size_t cells = (size_t)f->nr * f->nphi;
  const size_t gx = (f->nr + TI - 1) / TI, tiles = gx * ((f->nphi + LOW - 1) / LOW);
  const size_t most = (size_t)f->num_sms * DENSE;
  const int widest = std::min(rest, MAX_SWEEPS) + 1;
  if (tiles > most) {
    const dim3 ga((f->nr + 63) / 64, f->nphi, 1), gp(gx, (f->nphi + TALL - 1) / TALL);
    const float amp = (float)f->forcing, drag = (float)f->drag, relax = (float)f->relax;
    fluid_advect_kernel<<<ga, 64, 0, s>>>(F, f->parity, 1, false, dt, amp, drag, relax);
    for (int k = 0; k < nsteps; ++k) {
      const bool end = k + 1 == nsteps;
      int left = rest;
      for (int pass = 0; pass < passes; ++pass) {
        const int m = std::min(left, MAX_SWEEPS);
        left -= m;
        fluid_pressure_kernel<<<gp, THREADS, tile_floats(TALL, widest) * sizeof(float), s>>>(
            F, f->parity, dt, pass == 0, sweeps > 0, pass & 1, m, left == 0);
      }
      fluid_advect_kernel<<<dim3(ga.x, ga.y, end ? 1 : 2), 64, 0, s>>>(F, f->parity, 0, end, dt, amp, drag, relax);
      f->parity ^= 1;
    }
    f->steps += nsteps;
    return cudaGetLastError() == cudaSuccess ? ST_OK : ST_ECUDA;
  }
  const unsigned blocks = (unsigned)std::min(
      most, std::max(std::min<size_t>(f->num_sms, (cells + 63) / 64), tiles + tiles / 2));
  const void* kernel = steps_kernel(blocks > (unsigned)f->num_sms);
  const size_t smem = tile_floats(LOW, widest) * sizeof(float);
  int parity = f->parity;
  float amp = (float)f->forcing, drag = (float)f->drag, relax = (float)f->relax;
  unsigned base = f->arrivals;
  void* args[] = {&F, &parity, &nsteps, &dt, &sweeps, &amp, &drag, &relax, &base};
  if (cudaLaunchCooperativeKernel(kernel, dim3(blocks), dim3(THREADS), args, smem, s) !=
      cudaSuccess) {
    (void)cudaGetLastError();
    return ST_ECUDA;
  }
  f->arrivals = base + blocks * (unsigned)nsteps * (unsigned)(passes + 1);
  f->parity ^= nsteps & 1;
  f->steps += nsteps;
  return ST_OK;
}

}  // namespace

extern "C" {

void st_fluid_params_default(st_fluid_params* p) {
  if (!p) return;
  std::memset(p, 0, sizeof(*p));
  p->M = 1.0;
  p->forcing = 6.0;
  p->drag = 0.15;
  p->relax = 0.05;
  p->scale_height = 0.08;
}

int st_fluid_create(st_fluid** out, st_context* ctx, const st_disc* disc, const st_fluid_params* fp) {
  if (!out || !ctx || !disc || !fp) return ST_EINVAL;
  *out = nullptr;
  if (!(fp->M > 0.0) || !(fp->scale_height > 0.0) || !(disc->outer > disc->inner) || !(disc->inner > 0.0))
    return ST_EINVAL;
  st::CtxVolume cv;
  if (st::context_volume(ctx, &cv) != ST_OK || !cv.on || !cv.d_vol) return ST_ESTATE;
  const int nr = cv.meta.nr, nphi = cv.meta.nphi, nz = cv.meta.nz;
  if (nr < 2 || nphi < 1 || nz < 2) return ST_ESTATE;
  if (nphi > 65535) return ST_EUNSUPPORTED;  // one grid row per phi row
  if (cudaSetDevice(cv.device) != cudaSuccess) return ST_ECUDA;
  const size_t n = (size_t)nr * nphi;
  // initial density: the volume's midplane slice k = (nz + 1) / 2 (1-based),
  // normalised to a peak of 1 (src/disc_sim.jl:45-91)
  std::vector<float> dens0(n);
  const size_t kmid = (size_t)((nz + 1) / 2 - 1);
  if (cudaMemcpyAsync(dens0.data(), cv.d_vol + kmid * n, n * sizeof(float), cudaMemcpyDeviceToHost, cv.stream) !=
          cudaSuccess ||
      cudaStreamSynchronize(cv.stream) != cudaSuccess)
    return ST_ECUDA;
  float peak = dens0[0];
  for (float v : dens0) peak = std::max(peak, v);
  if (peak > 0.0f)
    for (float& v : dens0) v /= peak;
  std::vector<float> base(n), env((size_t)nr * nz), shear(nr);
  const double M = fp->M;
  const float log_in = cv.meta.log_s_in, log_out = cv.meta.log_s_out, zmax = cv.meta.z_max;
  const float hsc = (float)fp->scale_height;
  const float dlog = log_out - log_in;  // a Float32 difference, as the reference forms it
  for (int i = 1; i <= nr; ++i) {
    const double s = std::exp((double)log_in + (double)(i - 1) / (double)(nr - 1) * (double)dlog);
    // _disc_radial_profile, src/disc_volume.jl:274-283
    const double R = s / (2.0 * M), R_in = disc->inner / (2.0 * M), R_out = disc->outer / (2.0 * M);
    const double iscotaper = std::min(std::max((R * R - R_in * R_in) * 0.3, 0.0), 1.0);
    const double T_emit = std::exp(10.034259 - 0.375 * std::log(R * R));
    const double outertaper = std::min(std::max(T_emit / 1000.0, 0.0), 1.0);
    const double dens = std::min(std::max((R_out - R) / (R_out - R_in), 0.0), 1.0);
    const float b = (float)(iscotaper * outertaper * std::pow(dens, disc->falloff));
    for (int j = 0; j < nphi; ++j) base[(size_t)(i - 1) + (size_t)nr * j] = b;
    const double H = (double)hsc * s;
    for (int k = 1; k <= nz; ++k) {
      const double z = -(double)zmax + (double)(k - 1) / (double)(nz - 1) * 2.0 * (double)zmax;
      env[(size_t)(i - 1) + (size_t)nr * (k - 1)] = (float)std::exp(-z * z / (2.0 * H * H));
    }
    shear[i - 1] = (float)(std::sqrt(M / (s * s * s)) * nphi / (2.0 * 3.141592653589793));
  }
  int* fault = nullptr;
  const int frc = st::context_gas_fault(ctx, &fault);
  if (frc != ST_OK) return frc;
  st_fluid* f = new st_fluid;
  f->ctx = ctx;
  f->device = cv.device;
  f->nr = nr; f->nphi = nphi; f->nz = nz;
  f->forcing = fp->forcing; f->drag = fp->drag; f->relax = fp->relax;
  // layout: vu vv vu2 vv2 dens0 dens1 base prs0 prs1 div fu fv tgt (n each), env (nr nz), shear (nr), t (2),
  // count, status
  bool up = cudaDeviceGetAttribute(&f->num_sms, cudaDevAttrMultiProcessorCount, f->device) == cudaSuccess;
  if (!up) { delete f; return ST_ECUDA; }
  const size_t total = 13 * n + (size_t)nr * nz + nr + 4;
  if (cudaStreamCreateWithFlags(&f->stream, cudaStreamNonBlocking) != cudaSuccess) { delete f; return ST_ECUDA; }
  if (cudaMalloc(&f->block, total * sizeof(float)) != cudaSuccess) {
    cudaStreamDestroy(f->stream);
    delete f;
    return ST_ENOMEM;
  }
  float* b = f->block;
  Fields& F = f->F;
  F.nr = nr; F.nphi = nphi; F.nz = nz;
  F.vu = b; F.vv = b + n; F.vu2 = b + 2 * n; F.vv2 = b + 3 * n;
  F.dens[0] = b + 4 * n; F.dens[1] = b + 5 * n;
  float* base_d = b + 6 * n;
  F.prs[0] = b + 7 * n; F.prs[1] = b + 8 * n; F.div = b + 9 * n;
  F.fu = b + 10 * n; F.fv = b + 11 * n; F.tgt = b + 12 * n;
  float* env_d = b + 13 * n;
  float* shear_d = env_d + (size_t)nr * nz;
  F.t = shear_d + nr;
  F.count = reinterpret_cast<unsigned*>(F.t + 2);
  F.status = reinterpret_cast<int*>(F.t + 3);
  F.base = base_d; F.env = env_d; F.shear = shear_d;
  F.fault = fault;
  bool ok = cudaMemsetAsync(b, 0, total * sizeof(float), f->stream) == cudaSuccess;
  ok = ok && cudaMemcpyAsync(F.dens[0], dens0.data(), n * sizeof(float), cudaMemcpyHostToDevice, f->stream) ==
                 cudaSuccess;
  ok = ok && cudaMemcpyAsync(base_d, base.data(), n * sizeof(float), cudaMemcpyHostToDevice, f->stream) ==
                 cudaSuccess;
  ok = ok && cudaMemcpyAsync(env_d, env.data(), env.size() * sizeof(float), cudaMemcpyHostToDevice, f->stream) ==
                 cudaSuccess;
  ok = ok && cudaMemcpyAsync(shear_d, shear.data(), nr * sizeof(float), cudaMemcpyHostToDevice, f->stream) ==
                 cudaSuccess;
  ok = ok && cudaStreamSynchronize(f->stream) == cudaSuccess;
  if (!ok) {
    cudaFree(f->block);
    cudaStreamDestroy(f->stream);
    delete f;
    return ST_ECUDA;
  }
  *out = f;
  return ST_OK;
}

int st_fluid_step(st_fluid* f, double dt, int jacobi, int nsteps, int, float* ms) {
  if (!f || !(std::isfinite(dt)) || jacobi < 0 || jacobi > 4096 || nsteps < 0) return ST_EINVAL;
  if (ms) *ms = 0.f;
  if (cudaSetDevice(f->device) != cudaSuccess) return ST_ECUDA;
  st::CtxVolume cv;
  if (st::context_volume(f->ctx, &cv) != ST_OK || !cv.on || cv.meta.nr != f->nr || cv.meta.nphi != f->nphi ||
      cv.meta.nz != f->nz)
    return ST_ESTATE;
  if (st::context_gas_failed(f->ctx)) return ST_ECUDA;
  // the steps run on the context's stream, so the next render sees the field
  cudaStream_t s = cv.stream;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (ms && (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess)) return ST_ECUDA;
  if (e0 && cudaEventRecord(e0, s) != cudaSuccess) return ST_ECUDA;
  int rc = ST_OK;
  for (int left = nsteps; left > 0 && rc == ST_OK; left -= LAUNCH_STEPS)
    rc = launch_steps(f, cv.d_vol, std::min(left, LAUNCH_STEPS), (float)dt, jacobi, s);
  if (e1) {
    int status = 0;
    if (cudaEventRecord(e1, s) != cudaSuccess || cudaEventSynchronize(e1) != cudaSuccess) rc = ST_ECUDA;
    else if (cudaEventElapsedTime(ms, e0, e1) != cudaSuccess) { (void)cudaGetLastError(); *ms = 0.f; }
    if (cudaMemcpy(&status, f->F.status, sizeof status, cudaMemcpyDeviceToHost) != cudaSuccess || status != 0)
      rc = ST_ECUDA;
  }
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  return rc;
}

int st_fluid_state(st_fluid* f, float* vu, float* vv, float* dens, float* volume, double* t) {
  if (!f) return ST_EINVAL;
  if (cudaSetDevice(f->device) != cudaSuccess) return ST_ECUDA;
  st::CtxVolume cv;
  if (st::context_volume(f->ctx, &cv) != ST_OK) return ST_ESTATE;
  cudaStream_t s = cv.stream;
  const size_t n = (size_t)f->nr * f->nphi;
  struct { float t[2]; unsigned count; int status; } tail{};  // as they lie
  bool ok = true;
  if (vu) ok = ok && cudaMemcpyAsync(vu, f->F.vu, n * sizeof(float), cudaMemcpyDeviceToHost, s) == cudaSuccess;
  if (vv) ok = ok && cudaMemcpyAsync(vv, f->F.vv, n * sizeof(float), cudaMemcpyDeviceToHost, s) == cudaSuccess;
  if (dens)
    ok = ok && cudaMemcpyAsync(dens, f->F.dens[f->parity], n * sizeof(float), cudaMemcpyDeviceToHost, s) ==
                   cudaSuccess;
  if (volume) {
    if (!cv.on || cv.meta.nr != f->nr || cv.meta.nphi != f->nphi || cv.meta.nz != f->nz) return ST_ESTATE;
    ok = ok && cudaMemcpyAsync(volume, cv.d_vol, n * f->nz * sizeof(float), cudaMemcpyDeviceToHost, s) ==
                   cudaSuccess;
  }
  ok = ok && cudaMemcpyAsync(&tail, f->F.t, sizeof tail, cudaMemcpyDeviceToHost, s) == cudaSuccess;
  ok = ok && cudaStreamSynchronize(s) == cudaSuccess;
  if (!ok || tail.status != 0) return ST_ECUDA;
  if (t) *t = (double)tail.t[f->parity];
  return ST_OK;
}

void st_fluid_destroy(st_fluid* f) {
  if (!f) return;
  cudaSetDevice(f->device);
  if (f->stream) cudaStreamSynchronize(f->stream);
  cudaFree(f->block);
  if (f->stream) cudaStreamDestroy(f->stream);
  delete f;
}

}  // extern "C"
