// st_train.cuh -- a training step of the surrogate in three kernels: forward
// and backward of 128-row tiles (train_tile_kernel), the hidden layers' weight
// gradients (train_dw_kernel), and their sums with AdamW (train_update_kernel).
//
// What bounds a step: its products are 19 GFLOP at a batch of 16,384 (10 us of
// the tensor cores), its inputs a megabyte.  As one launch for each layer's
// product it was 25 kernels that passed every activation and pre-activation, and
// transposed copies of most, through L2: 320 us.  Here a CTA takes its rows
// through all layers forward and back with the activations in shared memory;
// what leaves the SM is two layers' SiLU derivatives (FP32, read back by the same
// thread) and the two operands of each weight gradient, as the swizzled bf16
// tiles that the next kernel's copies and matrix descriptors take unchanged.  A
// tile is a chain of six products and eight element-wise passes; 128 tiles fill 128
// of the 152 SMs once.  SiLU costs two MUFU operations a value (4,100 cycles a
// pass over a tile at 16 a clock), so each forward pass takes the derivative
// from the same exponential and reciprocal and keeps it: for two layers in
// tensor memory in the place of the pre-activations, for two in global memory.
// Batch 16,384: 0.324 -> 0.082 ms a step.
//
// The arithmetic of a row is that of the layer-by-layer path: FP32 edge layers
// in the same order, bf16 operands, FP32 accumulation over K in the same order,
// the same rounding of activations and of their gradients, and the sums over the
// batch in its order where that is fixed; what it added by atomics is in order here.
#pragma once

namespace st {
namespace sur {

constexpr int TR_THREADS = 512;
constexpr uint32_t TR_IMG = TC_ROWS * NH * 2;  // one 128 x 256 bf16 tile, 64 KB
// columns of the edge partials: dW0, db0, db1..db3, dW4, db4
constexpr int TR_B1 = NH * NIN + NH, TR_W4 = TR_B1 + 3 * NH, TR_B4 = TR_W4 + NOUT * NH, TR_EDGE = TR_B4 + NOUT;
constexpr int TR_ROW = 4104;  // their row stride
static_assert(TR_EDGE <= TR_ROW, "edge partials");
// shares of the batch in the hidden weight gradients, at most this many
constexpr int TR_SPLITS = 64;
inline int train_splits(int ntiles) { return std::max(1, std::min(TR_SPLITS, ntiles / 8)); }

struct TrainSmall {
  // rows of eight, read as two 16-byte words: a unit's layer-0 weights and bias, a
  // row's inputs, its targets and then its output gradient
  float w0[NH][8], X[TC_ROWS][8];
  float dout[TC_ROWS][8];
  float w4t[NOUT][NH], bh[3][NH], b4[8];
  uint64_t bar_w, bar_mma;
  uint32_t tmem;
  int fail;
};
constexpr size_t TR_SMEM = 1024 + TC_A_BYTES + TC_B_BYTES + sizeof(TrainSmall);
static_assert(TR_SMEM <= 227 * 1024, "training tile exceeds shared memory");

struct TrainParams {
  const float* P;
  const unsigned char* WF;  // [3] hidden weights, K-major swizzled images
  const unsigned char* WT;  // [3] their transposes
  const float* X;
  const float* T;
  int n;                    // rows that count (the rest of the last tile carries no gradient)
  int ntiles;
  float inv_batch;
  unsigned char* H;         // [3][ntiles] activations H0..H2
  unsigned char* D;         // [3][ntiles] gradients dZ1..dZ3
  float* Z;                 // [grid][2][256][128] SiLU derivatives of layers 0 and 1
  float* part;              // [4 ntiles][TR_ROW] edge partials, one row of them for 32 of the batch
  float* loss;              // 4 sums, added to
  int* status;
};

// Programmatic dependent launch.  A step's three kernels take 12 to 52 us, and
// between two of them the last block's end, the launch and the next one's
// barriers and tensor memory took two more.  Each kernel now lets the next start
// when its own blocks are nearly done (let_next_start), and waits for the end of
// the one before (wait_for_previous) ahead of its first access to global memory,
// reads of inputs and writes alike.  The one before has waited in the same way, so
// no kernel touches memory while the one two before it runs.  20 steps of 16,384
// in a call: 1,767 -> 1,657 us, when the 25-launch step took 6,579 and 6,471.
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("fence.proxy.async.global;" ::: "memory");  // before bulk copies of what its plain stores wrote
}

// shared -> global bulk copy (TMA), in the thread's bulk group
__device__ __forceinline__ void bulk_s2g(void* dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\ncp.async.bulk.commit_group;" ::"l"(dst),
               "r"(tc::smem_u32(src)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// 32 values as bf16 pairs, and the pairs into row `row`, columns col.. of the tile.
__device__ __forceinline__ void pack32(const float* v, uint32_t* pk) {
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
    pk[e] = *reinterpret_cast<const uint32_t*>(&h);
  }
}
__device__ __forceinline__ void put32(unsigned char* As, int row, int col, const uint32_t* pk) {
#pragma unroll
  for (int e = 0; e < 4; ++e)
    *reinterpret_cast<uint4*>(As + tc::sw128_off(row, col + 8 * e, TC_ROWS)) =
        make_uint4(pk[4 * e], pk[4 * e + 1], pk[4 * e + 2], pk[4 * e + 3]);
}
// SiLU and its derivative from one exponential and one reciprocal: mlp::dsilu, and
// mlp::silu's quotient z / (1 + e^-z) as the product with the reciprocal that it is
__device__ __forceinline__ void silu_both(float& z, float& g) {
  const float s = __fdividef(1.f, 1.f + __expf(-z));
  g = s * (1.f + z * (1.f - s));
  z = z * s;
}
__device__ __forceinline__ float get1(const unsigned char* As, int row, int col) {
  return __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(As + tc::sw128_off(row, col, TC_ROWS)));
}
// columns col (even) and col + 1
__device__ __forceinline__ float2 get2(const unsigned char* As, int row, int col) {
  return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(As + tc::sw128_off(row, col, TC_ROWS)));
}
__device__ __forceinline__ void row8(const float* r, float* v) {
  const float4 a = *reinterpret_cast<const float4*>(r), b = *reinterpret_cast<const float4*>(r + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

// RUN_OUT: the first copy is left out, so that each CTA's first wait runs out (the
// failure path under test).
template <bool RUN_OUT>
__global__ void __launch_bounds__(TR_THREADS, 1) train_tile_kernel(const TrainParams tp) {
  extern __shared__ unsigned char tr_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(tr_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  unsigned char* As = base;               // activations, then their gradients
  unsigned char* Bs = base + TC_A_BYTES;  // the current product's weights
  TrainSmall& S = *reinterpret_cast<TrainSmall*>(Bs + TC_B_BYTES);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float* P = tp.P;
  if (tid == 0) {
    tc::mbar_init(&S.bar_w, 1);
    tc::mbar_init(&S.bar_mma, 1);
    S.fail = 0;
    tc::mbar_fence_init();
  }
  if (warp == 0) tc::tmem_alloc(&S.tmem, 512);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = S.tmem;
  const uint32_t a_addr = tc::smem_u32(As), b_addr = tc::smem_u32(Bs);
  // warp w: rows 32 (w mod 4).., columns 64 (w div 4)..
  const uint32_t q = warp & 3, cq = warp >> 2;
  const int row = (int)(q * 32 + lane), col0 = (int)cq * 64;
  const uint32_t t_lane = tmem + ((q * 32u) << 16);
  // product m's weights: forward 1, 2, 3, then back 3, 2, 1
  auto load_w = [&](int m) {
    const unsigned char* src = m < 3 ? tp.WF + (size_t)m * TC_B_BYTES : tp.WT + (size_t)(5 - m) * TC_B_BYTES;
    tc::mbar_expect_tx(&S.bar_w, TC_B_BYTES);
#pragma unroll
    for (int c = 0; c < 4; ++c) tc::bulk_g2s(Bs + c * 32768, src + c * 32768, 32768, &S.bar_w);
  };
  uint32_t pw = 0, pm = 0;
  bool w_out = false, m_out = false;  // thread 0: a copy or a product is in flight
  wait_for_previous();
  if (tid == 0 && !RUN_OUT) {
    load_w(0);
    w_out = true;
  }
  {
    // all loads before the first store
    constexpr int N0 = NH * NIN / TR_THREADS, N4 = NH * NOUT / TR_THREADS;
    static_assert(NH * NIN % TR_THREADS == 0 && NH * NOUT % TR_THREADS == 0 && TR_THREADS == 2 * NH, "parameter loads");
    float a[N0], c[N4];
#pragma unroll
    for (int e = 0; e < N0; ++e) a[e] = __ldcg(P + OW0 + tid + e * TR_THREADS);
#pragma unroll
    for (int e = 0; e < N4; ++e) c[e] = __ldcg(P + OW4 + tid + e * TR_THREADS);
    const int u = tid & (NH - 1);
    const float b0 = __ldcg(P + (tid < NH ? OB0 : OB1) + u), b1 = __ldcg(P + (tid < NH ? OB2 : OB3) + u);
    const float b4 = tid < NOUT ? __ldcg(P + OB4 + tid) : 0.f;
#pragma unroll
    for (int e = 0; e < N0; ++e) {
      const int k = tid + e * TR_THREADS;
      S.w0[k / NIN][k % NIN] = a[e];
    }
#pragma unroll
    for (int e = 0; e < N4; ++e) {
      const int k = tid + e * TR_THREADS;
      S.w4t[k / NH][k % NH] = c[e];
    }
    if (tid < NH) S.w0[u][NIN] = b0;
    else S.bh[0][u] = b0;
    S.bh[tid < NH ? 1 : 2][u] = b1;
    if (tid < NOUT) S.b4[tid] = b4;
  }
  // kept derivatives: four columns of a row together, rows along a warp
  float4* Z0 = reinterpret_cast<float4*>(tp.Z) + (size_t)blockIdx.x * 2 * (NH / 4) * TC_ROWS;
  float4* Z1 = Z0 + (NH / 4) * TC_ROWS;
  auto z_at = [&](int col, int r) { return (col >> 2) * (int)TC_ROWS + r; };
  auto z_load = [&](const float4* Z, int col, float* g) {
#pragma unroll
    for (int e = 0; e < 32; e += 4) {
      const float4 z = Z[z_at(col + e, row)];
      g[e] = z.x; g[e + 1] = z.y; g[e + 2] = z.z; g[e + 3] = z.w;
    }
  };
  // sums over a tile's rows: two columns and a quarter of the rows a thread, each
  // quarter in a row of partials of its own.  Small batches depend on the order of
  // these sums: AdamW steps by g / |g| at first, a rounding more or less moves a
  // bf16 weight, and ten steps later the loss differs in its fourth digit.
  // train_update_kernel keeps reduce_parts' order.  (Their loops over rows are
  // unrolled by four: by eight they spill, and there is next to no L1 beside the
  // shared memory, 59.0 -> 51.9 us.)
  const int n2 = (tid & 127) * 2, quart = tid >> 7, r0 = quart * 32;
  for (int t = blockIdx.x; t < tp.ntiles; t += gridDim.x) {
    float* part = tp.part + ((size_t)t * 4 + quart) * TR_ROW;
    for (int k = tid; k < (int)TC_ROWS * NIN; k += TR_THREADS)
      S.X[k / NIN][k % NIN] = tp.X[(size_t)t * TC_ROWS * NIN + k];
    // the targets wait where each row's output gradient will be
    for (int k = tid; k < (int)TC_ROWS * NT; k += TR_THREADS)
      if ((long long)t * TC_ROWS + k / NT < tp.n) S.dout[k / NT][k % NT] = tp.T[(size_t)t * TC_ROWS * NT + k];
    __syncthreads();
    {
      // layer 0 in l0_fwd's order: a thread takes two rows and 32 units, so a
      // unit's weights are read once for both
      const int ra = (warp & 1) * 64 + lane, c0 = (warp >> 1) * 32;
      float xa[8], xb[8];
      row8(S.X[ra], xa);
      row8(S.X[ra + 32], xb);
      uint32_t pa[16], pb[16];
#pragma unroll
      for (int c = 0; c < 32; c += 4) {
        float za[4], zb[4], ga[4], gb[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float w[8];
          row8(S.w0[c0 + c + e], w);
          za[e] = zb[e] = w[NIN];
#pragma unroll
          for (int i = 0; i < NIN; ++i) {
            za[e] += xa[i] * w[i];
            zb[e] += xb[i] * w[i];
          }
          silu_both(za[e], ga[e]);
          silu_both(zb[e], gb[e]);
        }
        Z0[z_at(c0 + c, ra)] = make_float4(ga[0], ga[1], ga[2], ga[3]);
        Z0[z_at(c0 + c, ra + 32)] = make_float4(gb[0], gb[1], gb[2], gb[3]);
#pragma unroll
        for (int e = 0; e < 4; e += 2) {
          const __nv_bfloat162 ha = __floats2bfloat162_rn(za[e], za[e + 1]), hb = __floats2bfloat162_rn(zb[e], zb[e + 1]);
          pa[(c + e) / 2] = *reinterpret_cast<const uint32_t*>(&ha);
          pb[(c + e) / 2] = *reinterpret_cast<const uint32_t*>(&hb);
        }
      }
      put32(As, ra, c0, pa);
      put32(As, ra + 32, c0, pb);
    }
    tc::fence_proxy_async();
    __syncthreads();
#pragma unroll 1
    for (int m = 0; m < 6; ++m) {
      if (m == 5 && t + (int)gridDim.x >= tp.ntiles) let_next_start();
      if (tid == 0) {
        tc::fence_after_sync();
        if (!tc::mbar_wait(&S.bar_w, pw, RUN_OUT ? 1024u : TC_WAIT_LIMIT)) {
          S.fail = 1;
        } else {
          w_out = false;
          const uint32_t d = tmem + (m == 1 ? 256u : 0u);
#pragma unroll
          for (int s = 0; s < NH / 16; ++s)
            tc::mma_bf16(d, tc::sw128_desc(a_addr + (s >> 2) * (TC_ROWS * 128) + (s & 3) * 32),
                         tc::sw128_desc(b_addr + (s >> 2) * (NH * 128) + (s & 3) * 32), TC_IDESC, s > 0 ? 1u : 0u);
          tc::mma_commit(&S.bar_mma);
          m_out = true;
          // the tile is also an operand of a weight gradient
          bulk_s2g((m < 3 ? tp.H + (size_t)m * tp.ntiles * TR_IMG : tp.D + (size_t)(5 - m) * tp.ntiles * TR_IMG) +
                       (size_t)t * TR_IMG,
                   As, TR_IMG);
        }
      }
      pw ^= 1u;
      // beside the product: the derivatives the pass after it needs from global
      // memory (threads of layer 0 wrote other elements than they read: a barrier
      // has passed since), and the tile's column sums
      float g[32];
      if (m >= 4) z_load(m == 4 ? Z1 : Z0, col0, g);
      if (m >= 3) {
        float2 s = make_float2(0.f, 0.f);
#pragma unroll 8
        for (int b = 0; b < 32; ++b) s = __fadd2_rn(s, get2(As, r0 + b, n2));
        *reinterpret_cast<float2*>(part + TR_B1 + (5 - m) * NH + n2) = s;
      }
      if (tid == 0 && !S.fail) {
        if (!tc::mbar_wait(&S.bar_mma, pm, TC_WAIT_LIMIT)) S.fail = 1;
        else m_out = false;
      }
      pm ^= 1u;
      __syncthreads();
      if (S.fail) break;
      tc::fence_after_sync();
      if (tid == 0 && (m < 5 || t + (int)gridDim.x < tp.ntiles)) {
        load_w(m < 5 ? m + 1 : 0);
        w_out = true;
      }
      // the pass after product m, 32 columns at a time; the first are computed
      // while the bulk store may still be reading the tile
#pragma unroll 1
      for (int c = 0; c < 64; c += 32) {
        const int k0 = col0 + c;
        float v[32];
        uint32_t pk[16];
        tc::tmem_ld32(t_lane + (m == 1 ? 256u : 0u) + (uint32_t)k0, v);
        if (m < 3) {
          // forward: bias, SiLU; its derivative kept
#pragma unroll
          for (int e = 0; e < 32; e += 4) {
            const float4 b = *reinterpret_cast<const float4*>(S.bh[m] + k0 + e);
            v[e] += b.x; v[e + 1] += b.y; v[e + 2] += b.z; v[e + 3] += b.w;
          }
#pragma unroll
          for (int e = 0; e < 32; ++e) silu_both(v[e], g[e]);
          if (m == 0) {
#pragma unroll
            for (int e = 0; e < 32; e += 4) Z1[z_at(k0 + e, row)] = make_float4(g[e], g[e + 1], g[e + 2], g[e + 3]);
          } else {
            tc::tmem_st32(t_lane + (m == 1 ? 256u : 0u) + (uint32_t)k0, g);
          }
        } else {
          // back: times the derivative of the layer below
          if (m == 3) tc::tmem_ld32(t_lane + 256u + (uint32_t)k0, g);
#pragma unroll
          for (int e = 0; e < 32; ++e) v[e] *= g[e];
          if (m >= 4 && c == 0) z_load(m == 4 ? Z1 : Z0, k0 + 32, g);
        }
        pack32(v, pk);
        if (c == 0) {
          if (tid == 0) bulk_wait_read();
          __syncthreads();
        }
        put32(As, row, k0, pk);
      }
      if (m == 2) {
        __syncthreads();
        // layer 4 and the loss (l4_fwd's order of sums): a warp takes its eight
        // rows four at a time; the exchanges halve the number of rows a lane holds
        float o[NOUT] = {0, 0, 0, 0, 0, 0};
#pragma unroll 1
        for (int r = 0; r < 8; r += 4) {
          float h[4][NH / 32];
#pragma unroll
          for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int i = 0; i < NH / 32; ++i) h[k][i] = get1(As, warp * 8 + r + k, lane + 32 * i);
#pragma unroll
          for (int j = 0; j < NOUT; ++j) {
            float a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int i = 0; i < NH / 32; ++i) {
              const float w = S.w4t[j][lane + 32 * i];
#pragma unroll
              for (int k = 0; k < 4; ++k) a[k] += h[k][i] * w;
            }
            // lanes with bit 4 set keep rows 2 and 3, with bit 3 set the odd one
            const bool hi = lane & 16, odd = lane & 8;
            const float b0 = (hi ? a[2] : a[0]) + __shfl_xor_sync(0xffffffffu, hi ? a[0] : a[2], 16);
            const float b1 = (hi ? a[3] : a[1]) + __shfl_xor_sync(0xffffffffu, hi ? a[1] : a[3], 16);
            float s = (odd ? b1 : b0) + __shfl_xor_sync(0xffffffffu, odd ? b0 : b1, 8);
#pragma unroll
            for (int x = 4; x > 0; x >>= 1) s += __shfl_xor_sync(0xffffffffu, s, x);
            // row r + k is in lanes 8 k ..; lane r + k keeps it
            s = __shfl_sync(0xffffffffu, s, (lane & 3) * 8);
            if ((lane & ~3) == r) o[j] = s + S.b4[j];
          }
        }
        float l[4] = {0.f, 0.f, 0.f, 0.f};
        if (lane < 8) {
          const int b = warp * 8 + lane;
          const long long gb = (long long)t * TC_ROWS + b;
          float gr[NOUT] = {0, 0, 0, 0, 0, 0};
          float tg[8];
          row8(S.dout[b], tg);
          if (gb < tp.n) row_loss(o, tg, gr, l);
#pragma unroll
          for (int k = 0; k < NOUT; ++k) S.dout[b][k] = gr[k] * tp.inv_batch;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
#pragma unroll
          for (int s = 4; s > 0; s >>= 1) l[k] += __shfl_xor_sync(0xffffffffu, l[k], s);
          if (lane == 0) atomicAdd(tp.loss + k, l[k] * tp.inv_batch);
        }
        __syncthreads();
        {
          // dW4 of the tile, and db4
          float2 a[NOUT];
#pragma unroll
          for (int j = 0; j < NOUT; ++j) a[j] = make_float2(0.f, 0.f);
#pragma unroll 4
          for (int b = r0; b < r0 + 32; ++b) {
            const float2 h = get2(As, b, n2);
            float d[8];
            row8(S.dout[b], d);
#pragma unroll
            for (int j = 0; j < NOUT; ++j) a[j] = __ffma2_rn(make_float2(d[j], d[j]), h, a[j]);
          }
          if ((tid & 127) < NOUT) {
            float s = 0.f;
#pragma unroll 8
            for (int b = r0; b < r0 + 32; ++b) s += S.dout[b][tid & 127];
            part[TR_B4 + (tid & 127)] = s;
          }
#pragma unroll
          for (int j = 0; j < NOUT; ++j) *reinterpret_cast<float2*>(part + TR_W4 + j * NH + n2) = a[j];
          __syncthreads();  // the tile is read
        }
        // dZ3 = (dout W4) times the derivative of layer 3, from tensor memory
        float d[8];
        row8(S.dout[row], d);
#pragma unroll 1
        for (int c = 0; c < 64; c += 32) {
          float v[32];
          uint32_t pk[16];
          tc::tmem_ld32(t_lane + (uint32_t)(col0 + c), v);
#pragma unroll
          for (int e = 0; e < 32; e += 4) {
            float2 s0 = make_float2(0.f, 0.f), s1 = s0;
#pragma unroll
            for (int j = 0; j < NOUT; ++j) {
              const float4 w = *reinterpret_cast<const float4*>(&S.w4t[j][col0 + c + e]);
              const float2 dj = make_float2(d[j], d[j]);
              s0 = __ffma2_rn(dj, make_float2(w.x, w.y), s0);
              s1 = __ffma2_rn(dj, make_float2(w.z, w.w), s1);
            }
            v[e] *= s0.x; v[e + 1] *= s0.y; v[e + 2] *= s1.x; v[e + 3] *= s1.y;
          }
          pack32(v, pk);
          put32(As, row, col0 + c, pk);
        }
      }
      tc::fence_proxy_async();
      tc::fence_before_sync();
      __syncthreads();
    }
    if (S.fail) break;
    {
      // dW0 and db0 of the tile
      float2 a[NIN + 1];
#pragma unroll
      for (int i = 0; i <= NIN; ++i) a[i] = make_float2(0.f, 0.f);
#pragma unroll 4
      for (int b = r0; b < r0 + 32; ++b) {
        const float2 d = get2(As, b, n2);
        float xr[8];
        row8(S.X[b], xr);
#pragma unroll
        for (int i = 0; i < NIN; ++i) a[i] = __ffma2_rn(make_float2(xr[i], xr[i]), d, a[i]);
        a[NIN] = __fadd2_rn(a[NIN], d);
      }
      static_assert(NIN == 6, "two columns of dW0 in three words");
      float4* w = reinterpret_cast<float4*>(part + n2 * NIN);
      w[0] = make_float4(a[0].x, a[1].x, a[2].x, a[3].x);
      w[1] = make_float4(a[4].x, a[5].x, a[0].y, a[1].y);
      w[2] = make_float4(a[2].y, a[3].y, a[4].y, a[5].y);
      *reinterpret_cast<float2*>(part + NH * NIN + n2) = a[NIN];
      __syncthreads();  // the tile is read
    }
  }
  const bool failed = S.fail != 0;
  if (tid == 0) {
    if (failed) {
      // drain what is in flight before shared and tensor memory are given up
      if (w_out) (void)tc::mbar_wait(&S.bar_w, pw ^ 1u, TC_WAIT_LIMIT);
      if (m_out) (void)tc::mbar_wait(&S.bar_mma, pm ^ 1u, TC_WAIT_LIMIT);
      atomicExch(tp.status, 1);
    }
    bulk_wait_all();
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, 512);
  }
}

// Shared-memory descriptor of a bf16 tile of `rows` rows x 256 columns (the
// layout of sw128_off) read along its columns: the operand's M or N runs along
// the contiguous direction ("MN-major"), K down the rows.  Atoms of 64 columns x
// 8 rows; LBO is the distance of 64-column blocks, SBO that of 8-row groups.
__device__ __forceinline__ uint64_t sw128_mn_desc(uint32_t saddr, uint32_t rows) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)((rows * 128u) >> 4) << 16;
  d |= (uint64_t)(1024u >> 4) << 32;
  d |= (uint64_t)1u << 46;
  d |= (uint64_t)2u << 61;
  return d;
}
constexpr uint32_t TR_IDESC_MN = TC_IDESC | (1u << 15) | (1u << 16);  // A and B MN-major

// Weight gradients of the hidden layers: dW_l = dZ_l^T H_{l-1}, as D[i][o] over
// half of the inputs i, all outputs o and one share of the batch's tiles.  Both
// operands are the tiles that train_tile_kernel left, copied as they are into two
// stages of 96 KB; K is the batch.  The accumulator goes to a partial of its own
// (in the parameters' order, coalesced along i), summed by train_update_kernel in
// order.  A share is 1,024 rows, in blocks of 64: 96 CTAs at a batch of 16,384, 13.0
// us.  Tiles dealt to 150 CTAs took 11.7 us, but made a batch under 2,048 rows 25
// sums of the one it is (see train_tile_kernel).
constexpr uint32_t DW_STAGE = TR_IMG / 2 + TR_IMG;
constexpr size_t DW_SMEM = 1024 + 2 * (size_t)DW_STAGE + 64;
__global__ void __launch_bounds__(256, 1) train_dw_kernel(const unsigned char* __restrict__ H,
                                                          const unsigned char* __restrict__ D, int ntiles, float* pw,
                                                          int* status) {
  extern __shared__ unsigned char dw_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(dw_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(base + 2 * DW_STAGE);
  uint64_t* done = full + 2;
  uint32_t* slot = reinterpret_cast<uint32_t*>(done + 2);
  int* fail = reinterpret_cast<int*>(slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int s0 = blockIdx.x, half = blockIdx.y, layer = blockIdx.z;
  if (tid == 0) {
    for (int k = 0; k < 2; ++k) { tc::mbar_init(full + k, 1); tc::mbar_init(done + k, 1); }
    *fail = 0;
    tc::mbar_fence_init();
  }
  if (warp == 0) tc::tmem_alloc(slot, 256);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *slot;
  wait_for_previous();
  if (tid == 0) {
    const unsigned char* Hl = H + (size_t)layer * ntiles * TR_IMG + half * (TR_IMG / 2);
    const unsigned char* Dl = D + (size_t)layer * ntiles * TR_IMG;
    auto load = [&](int t, int st) {
      unsigned char* a = base + st * DW_STAGE;
      tc::mbar_expect_tx(full + st, DW_STAGE);
      tc::bulk_g2s(a, Hl + (size_t)t * TR_IMG, TR_IMG / 2, full + st);
      tc::bulk_g2s(a + TR_IMG / 2, Dl + (size_t)t * TR_IMG, TR_IMG / 2, full + st);
      tc::bulk_g2s(a + TR_IMG, Dl + (size_t)t * TR_IMG + TR_IMG / 2, TR_IMG / 2, full + st);
    };
    // blocks kb0.. of 64 rows, in tiles t0.. (the first and last perhaps by half)
    const int per = (2 * ntiles + (int)gridDim.x - 1) / (int)gridDim.x;
    const int kb0 = s0 * per, kb1 = min(2 * ntiles, kb0 + per), t0 = kb0 >> 1, nt = ((kb1 + 1) >> 1) - t0;
    bool ok = true;
    int loaded = 0, issued = 0;
    for (; loaded < 2 && loaded < nt; ++loaded) load(t0 + loaded, loaded);
    for (int k = 0; k < nt && ok; ++k) {
      const int st = k & 1;
      ok = tc::mbar_wait(full + st, (uint32_t)(k >> 1) & 1u, TC_WAIT_LIMIT);
      if (!ok) break;
      tc::fence_after_sync();
      const uint32_t a = tc::smem_u32(base + st * DW_STAGE), b = a + TR_IMG / 2;
      const int s1 = (k == 0 && (kb0 & 1)) ? 4 : 0, s2 = (k == nt - 1 && (kb1 & 1)) ? 4 : 8;
      for (int s = s1; s < s2; ++s)
        tc::mma_bf16(tmem, sw128_mn_desc(a + s * 2048, TC_ROWS), sw128_mn_desc(b + s * 2048, TC_ROWS), TR_IDESC_MN,
                     (k > 0 || s > s1) ? 1u : 0u);
      tc::mma_commit(done + st);
      ++issued;
      if (loaded < nt) {
        // the stage is free once its products are done; the other one's copy is on its way
        ok = tc::mbar_wait(done + st, (uint32_t)(k >> 1) & 1u, TC_WAIT_LIMIT);
        if (ok) { load(t0 + loaded, st); ++loaded; }
      }
    }
    // the last products; after a wait that ran out, whatever is still in flight
    for (int k = issued > 2 ? issued - 2 : 0; k < issued; ++k)
      ok = tc::mbar_wait(done + (k & 1), (uint32_t)(k >> 1) & 1u, TC_WAIT_LIMIT) && ok;
    for (int k = issued; k < loaded; ++k) (void)tc::mbar_wait(full + (k & 1), (uint32_t)(k >> 1) & 1u, TC_WAIT_LIMIT);
    if (!ok) { *fail = 1; atomicExch(status, 1); }
  }
  __syncthreads();
  tc::fence_after_sync();
  let_next_start();
  if (!*fail) {
    // warp w: inputs 32 (w mod 4).. of the half, outputs 128 (w div 4)..
    const uint32_t q = warp & 3;
    const int i = half * 128 + (int)q * 32 + lane, o0 = (warp >> 2) * 128;
    float* out = pw + ((size_t)s0 * 3 + layer) * NH * NH + i;
#pragma unroll 1
    for (int c = 0; c < 128; c += 32) {
      float v[32];
      tc::tmem_ld32(tmem + ((q * 32u) << 16) + (uint32_t)(o0 + c), v);
#pragma unroll
      for (int e = 0; e < 32; ++e) out[(size_t)(o0 + c + e) * NH] = v[e];
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, 256);
  }
}

struct AdamParams {
  float *P, *M, *V;
  float lr, b1, b2, eps, wd, bc1, bc2;
};
// One parameter's AdamW update (decoupled weight decay on weight matrices only);
// returns its new value.
__device__ __forceinline__ float adam_one(const AdamParams& a, size_t i, float g, bool is_bias) {
  const float m = a.b1 * a.M[i] + (1.f - a.b1) * g;
  const float v = a.b2 * a.V[i] + (1.f - a.b2) * g * g;
  a.M[i] = m;
  a.V[i] = v;
  float p = a.P[i];
  if (!is_bias) p -= a.lr * a.wd * p;
  p = p - a.lr * (m / a.bc1) / (sqrtf(v / a.bc2) + a.eps);
  a.P[i] = p;
  return p;
}

// Sums the partials of every gradient in a fixed order and either writes the
// gradient (G) or takes the AdamW step, refreshing the hidden layers' bf16
// images.  Blocks 0..191: 16 outputs x 64 inputs of a hidden layer, four inputs a
// thread, the partials of five shares in flight at once (their latency is the
// kernel's time); the rest: 32 edge parameters, their partial rows over 8 warps.
constexpr int UPD_HIDDEN = 3 * (NH / 16) * (NH / 64), UPD_EDGE = (TR_EDGE + 31) / 32;
__global__ void __launch_bounds__(256) train_update_kernel(const float* pw, int splits, const float* part,
                                                           int nparts, float* G,
                                                           AdamParams a, unsigned char* WF, unsigned char* WT) {
  wait_for_previous();
  let_next_start();
  if (blockIdx.x < UPD_HIDDEN) {
    __shared__ __nv_bfloat16 tr[64][24];  // [input][output], rows of 48 bytes
    const int layer = blockIdx.x / 64, b = blockIdx.x % 64;
    const int o0 = (b >> 2) * 16, i0 = (b & 3) * 64;
    const int o = o0 + (threadIdx.x >> 4), i = i0 + (threadIdx.x & 15) * 4;
    const float4* src = reinterpret_cast<const float4*>(pw + (size_t)layer * NH * NH + (size_t)o * NH + i);
    constexpr size_t SHARE = 3 * (size_t)NH * NH / 4;
    float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
    int s = 0;
    for (; s + 5 <= splits; s += 5) {
      float4 t[5];
#pragma unroll
      for (int k = 0; k < 5; ++k) t[k] = __ldcg(src + (s + k) * SHARE);
#pragma unroll
      for (int k = 0; k < 5; ++k) { g.x += t[k].x; g.y += t[k].y; g.z += t[k].z; g.w += t[k].w; }
    }
    for (; s < splits; ++s) {
      const float4 t = __ldcg(src + s * SHARE);
      g.x += t.x; g.y += t.y; g.z += t.z; g.w += t.w;
    }
    const size_t off = (layer == 0 ? OW1 : layer == 1 ? OW2 : OW3) + (size_t)o * NH + i;
    const float gv[4] = {g.x, g.y, g.z, g.w};
    if (G) {
#pragma unroll
      for (int k = 0; k < 4; ++k) G[off + k] = gv[k];
      return;
    }
    uint32_t pk[2];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const __nv_bfloat16 h = __float2bfloat16_rn(adam_one(a, off + k, gv[k], false));
      const uint32_t u = __bfloat16_as_ushort(h);
      pk[k >> 1] = (k & 1) ? pk[k >> 1] | (u << 16) : u;
      tr[i - i0 + k][o - o0] = h;
    }
    *reinterpret_cast<uint2*>(WF + (size_t)layer * TC_B_BYTES + tc::sw128_off(o, i, NH)) = make_uint2(pk[0], pk[1]);
    __syncthreads();
    if (threadIdx.x < 128) {
      // an input's 16 outputs: two 16-byte chunks of the transposed image
      const int r = threadIdx.x >> 1, c = (threadIdx.x & 1) * 8;
      *reinterpret_cast<uint4*>(WT + (size_t)layer * TC_B_BYTES + tc::sw128_off(i0 + r, o0 + c, NH)) =
          *reinterpret_cast<const uint4*>(&tr[r][c]);
    }
    return;
  }
  // the partials of every 32nd row, then those 32 sums, in order; a warp takes four
  __shared__ float red[32][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int c = (blockIdx.x - UPD_HIDDEN) * 32 + lane;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  if (c < TR_EDGE) {
#pragma unroll 4
    for (int p = w; p < nparts; p += 32)
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (p + 8 * k < nparts) acc[k] += __ldcg(part + (size_t)(p + 8 * k) * TR_ROW + c);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) red[w + 8 * k][lane] = acc[k];
  __syncthreads();
  if (w != 0 || c >= TR_EDGE) return;
  float g = red[0][lane];
#pragma unroll
  for (int k = 1; k < 32; ++k) g += red[k][lane];
  // the parameter of column c
  size_t i;
  bool is_bias = true;
  if (c < NH * NIN + NH) { i = OW0 + c; is_bias = c >= NH * NIN; }
  else if (c < TR_W4) { const int l = (c - TR_B1) / NH; i = (l == 0 ? OB1 : l == 1 ? OB2 : OB3) + (c - TR_B1) % NH; }
  else { i = OW4 + (c - TR_W4); is_bias = c >= TR_B4; }
  if (G) G[i] = g;
  else adam_one(a, i, g, is_bias);
}

// P -> the hidden layers' bf16 images, plain and transposed.
__global__ void pack_train(const float* __restrict__ P, unsigned char* WF, unsigned char* WT) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= 3 * NH * NH) return;
  const int l = idx / (NH * NH), o = (idx / NH) % NH, i = idx % NH;
  const __nv_bfloat16 h = __float2bfloat16_rn(P[(l == 0 ? OW1 : l == 1 ? OW2 : OW3) + (size_t)o * NH + i]);
  *reinterpret_cast<__nv_bfloat16*>(WF + (size_t)l * TC_B_BYTES + tc::sw128_off(o, i, NH)) = h;
  *reinterpret_cast<__nv_bfloat16*>(WT + (size_t)l * TC_B_BYTES + tc::sw128_off(i, o, NH)) = h;
}

}  // namespace sur
}  // namespace st
