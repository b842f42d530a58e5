// Fused forward / backward kernels of the surrogate's networks of width W =
// 64 and 128 (other widths: one GEMM per layer, mlp.cu).
//
// One CTA takes 128 rows of one network through all four layers: the weights
// sit in shared memory, the accumulators in tensor memory, and between layers
// only the BF16 activations pass through shared memory as the next layer's
// operand.  Everything the layer-by-layer form wrote to and read from global
// memory in between (FP32 pre-activations, activations, their gradients: 24
// bytes per row, unit and layer) stays on the SM.
//
// One layout serves every product.  A matrix lies in shared memory as 8 x 8
// core matrices of 128 bytes, block row by block row (core_index).  Read as a
// K-major operand its rows are M / N; read as an MN-major operand its rows are
// K.  So the same bytes are the operand of X W and of dZ W^T (the weights), or
// of A W and of A^T dZ (the activations), and tiles move between global and
// shared memory as one bulk copy, with no gather and no transposition.  The
// products accumulate over K in the same order as the layer-by-layer form.
#include "mlp_fused.h"

#include <algorithm>
#include <atomic>

#include "umma.cuh"

namespace chaos {
namespace mlp {
namespace {

using bf16 = __nv_bfloat16;
using namespace umma;

constexpr int kThreads = 256;  // 2 warps per TMEM lane quarter, half the columns each
constexpr int kRows = 128;     // rows per tile (M of the forward MMAs)

// Shared memory of the forward / training kernel.
template <int W> struct Smem {
  static constexpr int w1 = 0, w2 = w1 + kFeat * W * 2, w3 = w2 + W * W * 2, w4 = w3 + W * W * 2,
                       x = w4 + W * kOutPad * 2, act = x + kRows * kFeat * 2,
                       bias = act + kRows * W * 2, bars = bias + (3 * W + kOutPad) * 4,
                       bytes = bars + 32;
};

__device__ __forceinline__ uint32_t pack2(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t *>(&h);
}

// K-major / MN-major descriptor of a matrix of C columns at `addr`, and the
// bytes from one K = 16 slice to the next.
__device__ __forceinline__ uint64_t desc_k(uint32_t addr, int C) {
  return smem_desc(addr, 128, C * 16);
}
__device__ __forceinline__ uint64_t desc_mn(uint32_t addr, int C) {
  return smem_desc(addr, C * 16, 128);
}
constexpr uint32_t kStepK = 256;
__host__ __device__ constexpr uint32_t step_mn(int C) { return C * 32; }

// D (+)= the product of `slices` K = 16 slices; the descriptors' start
// addresses advance by sa / sb bytes per slice.
__device__ __forceinline__ void mma_slices(uint32_t d, uint64_t a, uint32_t sa, uint64_t b,
                                           uint32_t sb, uint32_t idesc, int slices,
                                           bool accumulate) {
  for (int j = 0; j < slices; j++)
    mma_bf16(d, a + (uint64_t)(j * (sa >> 4)), b + (uint64_t)(j * (sb >> 4)), idesc,
             accumulate || j > 0);
}

// kChunk accumulator columns from column c of this warp's lanes.
constexpr int kChunk = 16;
__device__ __forceinline__ void load_columns(uint32_t tmem, int quarter, int c,
                                             float (&v)[kChunk]) {
  uint32_t a[kChunk / 16][16];
#pragma unroll
  for (int i = 0; i < kChunk / 16; i++)
    tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(c + 16 * i), a[i]);
  tmem_wait_ld();
#pragma unroll
  for (int j = 0; j < kChunk; j++) v[j] = __uint_as_float(a[j / 16][j % 16]);
}

struct FwdArgs {
  Params P;
  FeatureMap f;
  const double *xy;
  int64_t rows;
  // prediction
  float *Y;
  int ys;
  // training
  const double *T;
  const int *idx;
  const float *tmean, *tinv;
  TrainBuffers b;
  float *loss;
};

template <int W>
__device__ __forceinline__ void load_weights(const FwdArgs &g, int z, uint32_t base,
                                             uint32_t wbar) {
  using S = Smem<W>;
  const bf16 *pb = g.P.pb + z * g.P.np;
  mbar_expect_tx(wbar, (kFeat * W + 2 * W * W + W * kOutPad) * 2);
  bulk_load(base + S::w1, pb + g.P.off_w[0], kFeat * W * 2, wbar);
  bulk_load(base + S::w2, pb + g.P.off_w[1], W * W * 2, wbar);
  bulk_load(base + S::w3, pb + g.P.off_w[2], W * W * 2, wbar);
  bulk_load(base + S::w4, pb + g.P.off_w[3], W * kOutPad * 2, wbar);
}
template <int W>
__device__ __forceinline__ void load_biases(const FwdArgs &g, int z, float *bias) {
  const float *p = g.P.p + z * g.P.np;
  for (int i = threadIdx.x; i < 3 * W + kOutPad; i += blockDim.x)
    bias[i] = __ldcg(p + (i < 3 * W ? g.P.off_b[i / W] + i % W : g.P.off_b[3] + i - 3 * W));
}

// One product of a tile: thread 0 issues its MMAs once every thread's operand
// stores are done, then every thread waits for them.
struct Product {
  uint32_t mbar, phase;
  bool ok;
  __device__ __forceinline__ void operator()(uint32_t d, uint64_t a, uint32_t sa, uint64_t b,
                                             uint32_t sb, uint32_t idesc, int slices) {
    fence_proxy_async();
    fence_before_sync();
    __syncthreads();
    if (threadIdx.x == 0) {
      fence_after_sync();
      mma_slices(d, a, sa, b, sb, idesc, slices, false);
      mma_commit(mbar);
    }
    if (ok) ok = mbar_wait(mbar, phase);
    phase ^= 1;
    fence_after_sync();
  }
};

// Prediction.  Grid (CTAs per network, networks): one CTA per SM with its
// network's weights resident and kPredictTiles tiles of 128 rows in flight, each
// with its own 256 threads (a thread takes one row's half of the columns), act
// buffer, accumulator and barriers, striding over the rows: while one tile waits
// for its MMAs the others are in their SiLU epilogues, which bound the kernel
// (two special-function operations per unit and row at 16 per cycle and SM: 0.69
// ms for 2^20 rows of 4 networks of width 128).  2^20 rows: 1.12 ms (two CTAs
// per SM with one tile each: 1.31 ms; layer by layer: 17.7 ms).  Rolled loops:
// unrolled over the layers, the epilogues waited on instruction fetch.
constexpr int kPredictTiles = 4;
template <int W> struct PredictSmem {
  using S = Smem<W>;
  static constexpr int x = S::x, tile = kRows * (kFeat + W) * 2,  // features, activations
                       bias = x + kPredictTiles * tile, bars = bias + (3 * W + kOutPad) * 4,
                       bytes = bars + 8 * (1 + kPredictTiles) + 16;
};

template <int W>
__global__ void __launch_bounds__(kThreads *kPredictTiles, 1)
    predict_kernel(const __grid_constant__ FwdArgs g) {
  using S = Smem<W>;
  using Q = PredictSmem<W>;
  constexpr int HC = W / 2;  // columns per thread and layer
  constexpr uint32_t kCols = kPredictTiles * W <= 256 ? 256 : 512;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t base = smem_u32(smem);
  float *bias = reinterpret_cast<float *>(smem + Q::bias);
  const int group = threadIdx.x / kThreads, tid = threadIdx.x % kThreads;
  const uint32_t wbar = base + Q::bars, mbar = wbar + 8 * (1 + group);
  uint32_t *slot = reinterpret_cast<uint32_t *>(smem + Q::bars + 8 * (1 + kPredictTiles));
  const int warp = tid >> 5, lane = tid & 31;
  const int quarter = warp & 3, half = warp >> 2;
  const int row = quarter * 32 + lane;  // this thread's row in the epilogues
  const int z = blockIdx.y;
  const uint32_t x = base + Q::x + group * Q::tile, act = x + kRows * kFeat * 2;
  uint8_t *const xs = smem + Q::x + group * Q::tile, *const as = xs + kRows * kFeat * 2;
  if (threadIdx.x == 0) {
    for (int i = 0; i <= kPredictTiles; i++) mbar_init(wbar + 8 * i, 1);
    mbar_init_fence();
    load_weights<W>(g, z, base, wbar);
  }
  if (threadIdx.x < 32) tmem_alloc(smem_u32(slot), kCols);
  load_biases<W>(g, z, bias);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = *slot + group * W;
  bool ok = mbar_wait(wbar, 0);
  uint32_t phase = 0;
  // Product, for the threads of one tile
  auto product = [&](uint64_t a, uint64_t b, uint32_t sb, uint32_t idesc, int slices) {
    fence_proxy_async();
    fence_before_sync();
    asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(kThreads) : "memory");
    if (tid == 0) {
      fence_after_sync();
      mma_slices(tmem, a, kStepK, b, sb, idesc, slices, false);
      mma_commit(mbar);
    }
    if (ok) ok = mbar_wait(mbar, phase);
    phase ^= 1;
    fence_after_sync();
  };

  const int64_t tiles = (g.rows + kRows - 1) / kRows;
  for (int64_t tile = (int64_t)blockIdx.x * kPredictTiles + group; tile < tiles;
       tile += (int64_t)gridDim.x * kPredictTiles) {
    {  // features: two threads per row, four frequency vectors each
      const int r = tid >> 1, h = tid & 1;
      const int64_t i = tile * kRows + r;
      uint4 q = make_uint4(0, 0, 0, 0);
      if (i < g.rows) {
        float u, v, sn[4], cs[4];
        normalised(g.f, g.xy, i, u, v);
#pragma unroll
        for (int f = 0; f < 4; f++) feature_pair(g.f, u, v, 4 * h + f, sn[f], cs[f]);
        q = make_uint4(pack2(sn[0], cs[0]), pack2(sn[1], cs[1]), pack2(sn[2], cs[2]),
                       pack2(sn[3], cs[3]));
      }
      *reinterpret_cast<uint4 *>(xs + ((r >> 3) * 2 + h) * 128 + (r & 7) * 16) = q;
    }
    // hidden layers: Z = A W; A' = SiLU(Z + b)
#pragma unroll 1
    for (int l = 0; l < 3; l++) {
      const uint64_t a = l == 0 ? desc_k(x, kFeat) : desc_k(act, W);
      const uint32_t w = base + (l == 0 ? S::w1 : l == 1 ? S::w2 : S::w3);
      product(a, desc_mn(w, W), step_mn(W), instr_desc(kRows, W, false, true),
              l == 0 ? 1 : W / 16);
#pragma unroll 1
      for (int c0 = half * HC; c0 < (half + 1) * HC; c0 += kChunk) {
        float v[kChunk];
        load_columns(tmem, quarter, c0, v);
#pragma unroll
        for (int c = 0; c < kChunk; c++) v[c] += bias[l * W + c0 + c];
        silu_chunk(v);
#pragma unroll
        for (int c = 0; c < kChunk; c += 8)
          *reinterpret_cast<uint4 *>(as + ((row >> 3) * (W / 8) + ((c0 + c) >> 3)) * 128 +
                                     (row & 7) * 16) =
              make_uint4(pack2(v[c], v[c + 1]), pack2(v[c + 2], v[c + 3]),
                         pack2(v[c + 4], v[c + 5]), pack2(v[c + 6], v[c + 7]));
      }
    }
    product(desc_k(act, W), desc_mn(base + S::w4, kOutPad), step_mn(kOutPad),
            instr_desc(kRows, kOutPad, false, true), W / 16);
    const int64_t i = tile * kRows + row;
    if (half == 0) {
      uint32_t a[16];
      tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16), a);
      tmem_wait_ld();
      if (i < g.rows) {
        float *y = g.Y + (z * g.rows + i) * g.ys;
#pragma unroll
        for (int c = 0; c < kOutPad; c += 4)
          if (c < g.ys)
            *reinterpret_cast<float4 *>(y + c) = make_float4(
                __uint_as_float(a[c]) + bias[3 * W + c],
                __uint_as_float(a[c + 1]) + bias[3 * W + c + 1],
                __uint_as_float(a[c + 2]) + bias[3 * W + c + 2],
                __uint_as_float(a[c + 3]) + bias[3 * W + c + 3]);
      }
    }
  }
  if (!ok && lane == 0) atomicExch(g.P.err, 1);
  fence_before_sync();
  __syncthreads();
  if (threadIdx.x < 32) tmem_dealloc(*slot, kCols);
}

// Training: the forward pass of kTrainRows = 64 rows of one network, the loss
// gradient, and the backward pass down to dZ1; activations and their gradients
// go out in core-matrix order for gradient_kernel.  A minibatch is a few
// thousand rows at most, so the chain of seven products and epilogues of one
// tile is the kernel's time: 64 rows, sixteen in each quarter of the MMA's 128
// (the other lanes are not read), so that all four schedulers share a tile's
// epilogue and a 1024-row batch of 4 networks spreads over 64 SMs.  The
// pre-activations of the hidden layers stay in tensor memory (columns 0 .. 3 W)
// for the backward pass.  A step of 1024 rows and 4 networks of width 128, this
// kernel and gradient_kernel: 22 us (24 launches, layer by layer: 530 us).
constexpr int kTrainRows = 64, kTrainThreads = 512;

template <int W>
__global__ void __launch_bounds__(kTrainThreads, 1) train_kernel(const __grid_constant__ FwdArgs g) {
  using S = Smem<W>;
  constexpr int HC = W / 4;  // columns per thread and layer
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t base = smem_u32(smem);
  float *bias = reinterpret_cast<float *>(smem + S::bias);
  const uint32_t wbar = base + S::bars, mbar = wbar + 8;
  uint32_t *slot = reinterpret_cast<uint32_t *>(smem + S::bars + 16);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int quarter = warp & 3, part = warp >> 2;
  const int z = blockIdx.y;
  const int64_t tile = blockIdx.x;
  const int64_t padded = (g.rows + kRows - 1) / kRows * kRows;  // rows of a buffer per network
  const int outs = g.P.outs;

  // Preamble: nothing here depends on the previous step.  (The rows are the
  // caller's, ordered before this kernel by the copy of the indices or the
  // clearing of the losses that precedes a call's first step.)
  if (tid == 0) {
    mbar_init(wbar, 1);
    mbar_init(mbar, 1);
    mbar_init_fence();
  }
  if (warp == 0) tmem_alloc(smem_u32(slot), 4 * W);
  // features: eight threads per row, one frequency vector each
  const int fr = tid >> 3, fh = tid & 7;
  const int64_t fi = tile * kTrainRows + fr;
  uint32_t fq = 0;
  if (fi < g.rows) {
    float u, v, sn, cs;
    normalised(g.f, g.xy, g.idx ? (int64_t)g.idx[fi] : fi, u, v);
    feature_pair(g.f, u, v, fh, sn, cs);
    fq = pack2(sn, cs);
  }
  const int fin = (fr & 7) * 16 + (fh & 3) * 4;
  {  // row r of the tile is row (r / 16) * 32 + r % 16 of the MMA
    const int mg = (fr >> 4) * 4 + ((fr >> 3) & 1);
    *reinterpret_cast<uint32_t *>(smem + S::x + (mg * 2 + (fh >> 2)) * 128 + fin) = fq;
  }
  // this thread's rows in the epilogues, r0 and r0 + 8, and their targets
  const int r0 = quarter * 16 + (lane >> 2), cp = (lane & 3) * 2;
  // (target - mean, and 1 / std: standardised where it is used)
  float tc[2][4], ti[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const int c = (j >> 1) * 8 + cp + (j & 1);
    ti[j] = part == 0 && c < outs ? g.tinv[c] : 0.f;
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int64_t i = tile * kTrainRows + r0 + 8 * q;
      tc[q][j] = 0.f;
      if (part == 0 && c < outs && i < g.rows) {
        const int64_t k = g.idx ? (int64_t)g.idx[i] : i;
        tc[q][j] = (float)g.T[k * outs + c] - g.tmean[c];
      }
    }
  }
  // (launch_dependents only once this CTA holds its tensor memory: umma.cuh)
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = *slot;
  wait_previous();
  launch_dependents();
  if (tid == 0) load_weights<W>(g, z, base, wbar);
  load_biases<W>(g, z, bias);  // read after the first product's barrier
  if (z == 0)
    *reinterpret_cast<uint32_t *>(reinterpret_cast<uint8_t *>(g.b.X) +
                                  ((fi >> 3) * 2 + (fh >> 2)) * 128 + fin) = fq;
  const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
  Product product{mbar, 0, mbar_wait(wbar, 0)};
  const int64_t row0 = z * padded + tile * kTrainRows;  // the tile's first row in the buffers

  // this thread's columns from c0: the next operand, and the same core matrices
  // outside
  auto store = [&](int c0, const float (&v)[HC / 2], bf16 *out) {
#pragma unroll
    for (int i = 0; i < HC / 8; i++)
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const uint32_t x = pack2(v[4 * i + 2 * q], v[4 * i + 2 * q + 1]);
        const int in = (lane >> 2) * 16 + cp * 2, cg = (c0 >> 3) + i;
        *reinterpret_cast<uint32_t *>(smem + S::act + ((quarter * 4 + q) * (W / 8) + cg) * 128 +
                                      in) = x;
        *reinterpret_cast<uint32_t *>(reinterpret_cast<uint8_t *>(out) +
                                      (((row0 >> 3) + quarter * 2 + q) * (W / 8) + cg) * 128 +
                                      in) = x;
      }
  };
  auto load = [&](uint32_t col, float (&v)[HC / 2]) {
    uint32_t a[HC / 2];
    if constexpr (HC == 32) tmem_ld_16x32(tmem + lanes + col, a);
    else tmem_ld_16x16(tmem + lanes + col, a);
    tmem_wait_ld();
#pragma unroll
    for (int j = 0; j < HC / 2; j++) v[j] = __uint_as_float(a[j]);
  };
  auto add_bias = [&](int c, float (&v)[HC / 2]) {
#pragma unroll
    for (int i = 0; i < HC / 8; i++) {
      const float2 b = *reinterpret_cast<const float2 *>(bias + c + 8 * i + cp);
      v[4 * i] += b.x;
      v[4 * i + 1] += b.y;
      v[4 * i + 2] += b.x;
      v[4 * i + 3] += b.y;
    }
  };
  const int c0 = part * HC;

  // hidden layers: Z = A W; A' = SiLU(Z + b)
#pragma unroll 1
  for (int l = 0; l < 3; l++) {
    const uint64_t a = l == 0 ? desc_k(base + S::x, kFeat) : desc_k(base + S::act, W);
    const uint32_t w = base + (l == 0 ? S::w1 : l == 1 ? S::w2 : S::w3);
    product(tmem + l * W, a, kStepK, desc_mn(w, W), step_mn(W), instr_desc(kRows, W, false, true),
            l == 0 ? 1 : W / 16);
    bf16 *out = l == 0 ? g.b.A[0] : l == 1 ? g.b.A[1] : g.b.A[2];
    float v[HC / 2];
    load(l * W + c0, v);
    add_bias(l * W + c0, v);
    silu_chunk(v);
    store(c0, v, out);
  }
  // output layer, loss and its gradient dY = 2 (Y - T) / (rows outs), zero on
  // the padding and past the rows
  const uint32_t dy = tmem + 3 * W;
  product(dy, desc_k(base + S::act, W), kStepK, desc_mn(base + S::w4, kOutPad), step_mn(kOutPad),
          instr_desc(kRows, kOutPad, false, true), W / 16);
  if (part == 0) {
    uint32_t a[8];
    tmem_ld_16x16(dy + lanes, a);
    tmem_wait_ld();
    float l = 0.f;
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int64_t i = tile * kTrainRows + r0 + 8 * q;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        float dv[2];
#pragma unroll
        for (int e = 0; e < 2; e++) {
          const int c = 8 * h + cp + e;
          dv[e] = 0.f;
          if (c < outs && i < g.rows) {
            const float y = __uint_as_float(a[4 * h + 2 * q + e]) + bias[3 * W + c];
            const float d = fmaf(-tc[q][2 * h + e], ti[2 * h + e], y);
            l += d * d;
            dv[e] = 2.f * d / (float)(g.rows * outs);
          }
        }
        const uint32_t x = pack2(dv[0], dv[1]);
        const int in = (lane >> 2) * 16 + cp * 2;
        // over the features, which only the first layer's MMA read
        *reinterpret_cast<uint32_t *>(smem + S::x + ((quarter * 4 + q) * 2 + h) * 128 + in) = x;
        *reinterpret_cast<uint32_t *>(reinterpret_cast<uint8_t *>(g.b.dY) +
                                      (((row0 >> 3) + quarter * 2 + q) * 2 + h) * 128 + in) = x;
      }
    }
    if (g.loss) {
      float s = l / (float)(g.rows * outs);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) atomicAdd(&g.loss[z], s);
    }
  }
  // dA = dZ' W^T; dZ = dA SiLU'(Z + b)
#pragma unroll 1
  for (int l = 2; l >= 0; l--) {
    const uint64_t a = l == 2 ? desc_k(base + S::x, kOutPad) : desc_k(base + S::act, W);
    const uint64_t w = l == 2 ? desc_k(base + S::w4, kOutPad)
                              : desc_k(base + (l == 1 ? S::w3 : S::w2), W);
    product(dy, a, kStepK, w, kStepK, instr_desc(kRows, W), l == 2 ? 1 : W / 16);
    bf16 *out = l == 0 ? g.b.dZ[0] : l == 1 ? g.b.dZ[1] : g.b.dZ[2];
    float da[HC / 2], v[HC / 2];
    load(3 * W + c0, da);
    load(l * W + c0, v);
    add_bias(l * W + c0, v);
    dsilu_chunk(da, v);
    store(c0, v, out);
  }
  if (!product.ok && lane == 0) atomicExch(g.P.err, 1);
  fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 4 * W);
}

// ------------------------------------------------------- weight gradients
struct GradArgs {
  Params P;
  TrainBuffers b;
  int64_t rows;
  int adam;
  AdamStep a;
};

__device__ __forceinline__ void apply(const GradArgs &g, int64_t i, float grad) {
  if (g.adam) {
    float m = g.P.m[i], v = g.P.v[i];
    g.P.p[i] = adam_update(g.P.p[i], grad, m, v, g.a.lr, g.a.b1, g.a.b2, g.a.eps, g.a.c1, g.a.c2);
    g.P.m[i] = m;
    g.P.v[i] = v;
  } else {
    g.P.g[i] = grad;
  }
}

constexpr int kSlice = 32;   // columns of a W x W gradient per CTA
constexpr int kStages = 5;
template <int W> struct GradSmem {
  static constexpr int mat = kRows * W * 2, stage = mat + kRows * kSlice * 2,
                       bars = kStages * stage, bytes = bars + 16 * kStages + 16;
};

// Weight matrix l of network z, columns n0 .. n0 + kSlice of the square ones:
// dW = A^T dZ over all rows, 128 at a time, in row order, accumulated in tensor
// memory (both operands MN-major: K runs over the rows); the first layer's
// gradient transposed (dZ^T X), so that M is the network's width.  Tiles arrive
// by bulk copies, kStages of them in flight, one copy per lane of a warp; the
// kernel's time is a CTA's reads of A from L2 (40 KB per tile) and the chain of
// its epilogue, which is why the square matrices are cut into slices.  The
// epilogue applies Adam through shared memory, consecutive threads on consecutive
// parameters (a lane per row of the accumulator, 32 lines per access, took four
// times as long), the first parameters and moments read ahead: the step before
// the previous kernel wrote them, and they come from L2, past any older line of
// this SM's first-level cache.
template <int W>
__device__ void weight_gradient(const GradArgs &g, int l, int n0, int z, uint8_t *smem) {
  using S = GradSmem<W>;
  const uint32_t base = smem_u32(smem);
  const uint32_t full = base + S::bars, done = full + 8 * kStages;
  uint32_t *slot = reinterpret_cast<uint32_t *>(smem + S::bars + 16 * kStages);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int quarter = warp & 3, half = warp >> 2;
  const int64_t tiles = (g.rows + kRows - 1) / kRows;
  const bool square = l == 1 || l == 2;
  const int N = square ? kSlice : 16;
  const bf16 *a = (l == 0 ? g.b.dZ[0] : g.b.A[l - 1]) + z * tiles * kRows * W;
  const bf16 *b = l == 0 ? g.b.X
                         : (l == 3 ? g.b.dY + z * tiles * kRows * kOutPad
                                   : g.b.dZ[l] + z * tiles * kRows * W);
  const uint32_t bytes_a = kRows * W * 2, bytes_b = kRows * N * 2;
  if (tid == 0) {
    for (int i = 0; i < 2 * kStages; i++) mbar_init(full + 8 * i, 1);
    mbar_init_fence();
  }
  if (warp == 0) tmem_alloc(smem_u32(slot), 32);
  // The epilogue's elements, four consecutive ones of a gradient row at a time:
  // quad q is row r, columns c .. c + 3 of a matrix of `cols` columns.  Quads of
  // consecutive threads are consecutive in memory.  The first quad's parameter
  // and moments are read ahead.
  const int64_t w0 = z * g.P.np + g.P.off_w[l];
  const int cols = square || l == 0 ? W : kOutPad;
  const int per_row = (l == 0 ? W : N) / 4, quads = W * N / 4;
  auto row_of = [&](int q) { return q / per_row; };
  auto col_of = [&](int q) { return (square ? n0 : 0) + q % per_row * 4; };
  auto at = [&](int q) { return w0 + (int64_t)row_of(q) * cols + col_of(q); };
  auto read = [&](const float *src, int q) {
    return __ldcg(reinterpret_cast<const float4 *>(src + at(q)));
  };
  float4 p, mo, ve;
  if (g.adam && tid < quads) {
    p = read(g.P.p, tid);
    mo = read(g.P.m, tid);
    ve = read(g.P.v, tid);
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = *slot;
  wait_previous();
  launch_dependents();
  int *flag = reinterpret_cast<int *>(slot + 1);
  if (warp == 1) {  // loads, one copy per lane
    bool ok = true;
    for (int64_t t = 0; t < tiles; t++) {
      const int st = (int)(t % kStages);
      const uint32_t bar = full + 8 * st, sa = base + st * S::stage;
      // the MMAs of the stage's last tile
      if (t >= kStages && ok) ok = mbar_wait(done + 8 * st, (uint32_t)((t / kStages - 1) & 1));
      if (lane == 0) mbar_expect_tx(bar, bytes_a + bytes_b);
      __syncwarp();
      if (lane == 16) bulk_load(sa, a + t * kRows * W, bytes_a, bar);
      if (square && lane < kRows / 8)  // the slice's core matrices, row group by row group
        bulk_load(sa + S::mat + lane * kSlice * 16,
                  b + (t * (kRows / 8) + lane) * W * 8 + n0 * 8, kSlice * 16, bar);
      if (!square && lane == 0) bulk_load(sa + S::mat, b + t * kRows * N, bytes_b, bar);
    }
    if (!ok && lane == 0) atomicExch(g.P.err, 1);
  }
  if (tid == 0) {
    bool ok = true;
    const uint32_t idesc = instr_desc(kRows, N, true, true);
    for (int64_t t = 0; t < tiles; t++) {
      const int st = (int)(t % kStages);
      if (ok) ok = mbar_wait(full + 8 * st, (uint32_t)((t / kStages) & 1));
      const uint32_t sa = base + st * S::stage;
      mma_slices(tmem, desc_mn(sa, W), step_mn(W), desc_mn(sa + S::mat, N), step_mn(N), idesc,
                 kRows / 16, t > 0);
      mma_commit(done + 8 * st);
    }
    // thread 0 waits for the last tile's MMAs (its commit covers all before
    // it); the barrier after that releases the others, who have not followed
    // the stages' phases
    const int64_t last = tiles - 1;
    if (ok) ok = mbar_wait(done + 8 * (int)(last % kStages), (uint32_t)((last / kStages) & 1));
    *flag = ok;
    if (!ok) atomicExch(g.P.err, 1);
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  // accumulator -> shared memory (over the first stage), lane = row m; rows
  // beyond W are the next rows' bytes read as features
  constexpr int pitch = kSlice + 4;
  float *const acc = reinterpret_cast<float *>(smem);
  const bool ready = *flag != 0;
  if (quarter * 32 < W && half * 16 < N) {
    uint32_t v[16];
    tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * 16), v);
    tmem_wait_ld();
    float4 *d = reinterpret_cast<float4 *>(acc + (quarter * 32 + lane) * pitch + half * 16);
#pragma unroll
    for (int c = 0; c < 4; c++)
      d[c] = make_float4(__uint_as_float(v[4 * c]), __uint_as_float(v[4 * c + 1]),
                         __uint_as_float(v[4 * c + 2]), __uint_as_float(v[4 * c + 3]));
  }
  __syncthreads();
  // Rolled: it runs once per launch, so its instructions are fetched cold.
  if (ready) {
#pragma unroll 1
    for (int q = tid; q < quads; q += kThreads) {
      float4 pn = p, mn = mo, vn = ve;
      if (g.adam && q + kThreads < quads) {
        pn = read(g.P.p, q + kThreads);
        mn = read(g.P.m, q + kThreads);
        vn = read(g.P.v, q + kThreads);
      }
      const int r = row_of(q), c = q % per_row * 4;
      const float4 d = l == 0 ? make_float4(acc[c * pitch + r], acc[(c + 1) * pitch + r],
                                            acc[(c + 2) * pitch + r], acc[(c + 3) * pitch + r])
                              : *reinterpret_cast<const float4 *>(acc + r * pitch + c);
      if (!g.adam) {
        *reinterpret_cast<float4 *>(g.P.g + at(q)) = d;
        continue;
      }
      const AdamStep &s = g.a;
      p.x = adam_update(p.x, d.x, mo.x, ve.x, s.lr, s.b1, s.b2, s.eps, s.c1, s.c2);
      p.y = adam_update(p.y, d.y, mo.y, ve.y, s.lr, s.b1, s.b2, s.eps, s.c1, s.c2);
      p.z = adam_update(p.z, d.z, mo.z, ve.z, s.lr, s.b1, s.b2, s.eps, s.c1, s.c2);
      p.w = adam_update(p.w, d.w, mo.w, ve.w, s.lr, s.b1, s.b2, s.eps, s.c1, s.c2);
      *reinterpret_cast<float4 *>(g.P.p + at(q)) = p;
      *reinterpret_cast<float4 *>(g.P.m + at(q)) = mo;
      *reinterpret_cast<float4 *>(g.P.v + at(q)) = ve;
      *reinterpret_cast<uint2 *>(g.P.pb + w0 + core_index(r, col_of(q), cols)) =
          make_uint2(pack2(p.x, p.y), pack2(p.z, p.w));
      p = pn, mo = mn, ve = vn;
    }
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 32);
}

// Columns n0 .. n0 + 31 (of the output layer: all 16) of bias vector l of
// network z: db[c] = the sum of dZ's column c over the rows, in row order -- one
// chain of additions per column, a lane each, straight from the tiles' core
// matrices in shared memory (the copies of kBiasTiles tiles in flight).
constexpr int kBiasTiles = 8;
template <int C, int NC>
__device__ void bias_gradient(const GradArgs &g, const bf16 *src, int n0, int64_t i0,
                              uint8_t *smem) {
  constexpr int kTile = kRows * NC * 2, kBars = kBiasTiles * kTile;
  const uint32_t base = smem_u32(smem), full = base + kBars;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t tiles = (g.rows + kRows - 1) / kRows;
  if (tid == 0) {
    for (int i = 0; i < kBiasTiles; i++) mbar_init(full + 8 * i, 1);
    mbar_init_fence();
  }
  wait_previous();
  launch_dependents();
  __syncthreads();
  float s = 0.f;
  bool ok = true;
  for (int64_t t0 = 0; t0 < tiles; t0 += kBiasTiles) {
    const uint32_t parity = (uint32_t)((t0 / kBiasTiles) & 1);
    const int nt = (int)min((int64_t)kBiasTiles, tiles - t0);
    if (warp == 1) {
      for (int t = 0; t < nt; t++) {
        const uint32_t bar = full + 8 * t, dst = base + t * kTile;
        if (lane == 0) mbar_expect_tx(bar, kTile);
        __syncwarp();
        if (lane < kRows / 8)  // the columns' core matrices, row group by row group
          bulk_load(dst + lane * NC * 16, src + ((t0 + t) * (kRows / 8) + lane) * C * 8 + n0 * 8,
                    NC * 16, bar);
      }
    } else if (warp == 0) {
      for (int t = 0; t < nt; t++) {
        if (ok) ok = mbar_wait(full + 8 * t, parity);
        const int n = (int)min((int64_t)kRows, g.rows - (t0 + t) * kRows);
        const uint8_t *col = smem + t * kTile + (lane >> 3) * 128 + (lane & 7) * 2;
        auto at = [&](int j) {  // row j of 16 at col
          return __bfloat162float(
              *reinterpret_cast<const bf16 *>(col + (j >> 3) * NC * 16 + (j & 7) * 16));
        };
        if (lane < NC) {
          int left = n;
          if (left >= 16) {  // 16 rows read ahead of the 16 being added
            float x[16], y[16];
#pragma unroll
            for (int j = 0; j < 16; j++) x[j] = at(j);
            col += 2 * NC * 16;
#pragma unroll 1
            for (left -= 16; left >= 16; left -= 16, col += 2 * NC * 16) {
#pragma unroll
              for (int j = 0; j < 16; j++) y[j] = at(j);
#pragma unroll
              for (int j = 0; j < 16; j++) s += x[j];
#pragma unroll
              for (int j = 0; j < 16; j++) x[j] = y[j];
            }
#pragma unroll
            for (int j = 0; j < 16; j++) s += x[j];
          }
          for (int j = 0; j < left; j++) s += at(j);
        }
      }
    }
    if (t0 + kBiasTiles < tiles) __syncthreads();  // the buffers are free again
  }
  if (warp == 0) {
    if (!ok && lane == 0) atomicExch(g.P.err, 1);
    if (ok && lane < NC) {
      apply(g, i0 + n0 + lane, s);
      if (g.adam) g.P.pb[i0 + n0 + lane] = __float2bfloat16(g.P.p[i0 + n0 + lane]);
    }
  }
}

// blockIdx.y: network; blockIdx.x: the slices of the two square weight matrices,
// the first and last one, then the bias vectors in pieces of 32 columns.
template <int W> struct GradGrid {
  static constexpr int slices = W / kSlice, weights = 2 + 2 * slices, pieces = W / 32,
                       blocks = weights + 3 * pieces + 1;
};
template <int W>
__global__ void __launch_bounds__(kThreads, 1) gradient_kernel(const __grid_constant__ GradArgs g) {
  extern __shared__ __align__(1024) uint8_t smem[];
  using B = GradGrid<W>;
  const int z = blockIdx.y, x = blockIdx.x;
  const int64_t tiles = (g.rows + kRows - 1) / kRows;
  if (x < 2 * B::slices) {
    weight_gradient<W>(g, 1 + x / B::slices, x % B::slices * kSlice, z, smem);
  } else if (x < B::weights) {
    weight_gradient<W>(g, x == 2 * B::slices ? 0 : 3, 0, z, smem);
  } else if (x < B::blocks - 1) {
    const int l = (x - B::weights) / B::pieces, n0 = (x - B::weights) % B::pieces * 32;
    bias_gradient<W, 32>(g, g.b.dZ[l] + z * tiles * kRows * W, n0, z * g.P.np + g.P.off_b[l], smem);
  } else {
    bias_gradient<kOutPad, kOutPad>(g, g.b.dY + z * tiles * kRows * kOutPad, 0,
                                    z * g.P.np + g.P.off_b[3], smem);
  }
}

// Raises a kernel's dynamic shared memory limit once per device.
template <class K> int allow_smem(K kern, int bytes, std::atomic<uint64_t> &seen) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 64 && (seen.load() >> dev & 1)) return 0;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess && dev < 64) seen.fetch_or(1ull << dev);
  return (int)e;
}

template <int W> int launch_predict(const FwdArgs &a, unsigned gx, cudaStream_t s) {
  static std::atomic<uint64_t> seen{0};
  if (int rc = allow_smem(predict_kernel<W>, PredictSmem<W>::bytes, seen)) return rc;
  predict_kernel<W><<<dim3(gx, a.P.E), kThreads * kPredictTiles, PredictSmem<W>::bytes, s>>>(a);
  return (int)cudaGetLastError();
}

// The training kernels alternate on one stream, each waiting for the one
// before it (wait_previous) after a preamble that does not need it: launched
// with the programmatic-dependency attribute, the preamble and the launch
// itself overlap the previous kernel's end.
template <class Args>
int launch_dependent(void (*kern)(Args), dim3 grid, int threads, int smem, cudaStream_t s,
                     const Args &args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return (int)cudaLaunchKernelEx(&cfg, kern, args);
}
template <int W> int launch_train(const FwdArgs &a, cudaStream_t s) {
  static std::atomic<uint64_t> seen{0};
  if (int rc = allow_smem(train_kernel<W>, Smem<W>::bytes, seen)) return rc;
  // whole 128-row tiles: gradient_kernel reads the padding rows (zeros)
  const dim3 grid((unsigned)(train_tiles(a.rows) * (kRows / kTrainRows)), a.P.E);
  return launch_dependent<FwdArgs>(train_kernel<W>, grid, kTrainThreads, Smem<W>::bytes, s, a);
}
template <int W> int launch_gradient(const GradArgs &a, cudaStream_t s) {
  static std::atomic<uint64_t> seen{0};
  if (int rc = allow_smem(gradient_kernel<W>, GradSmem<W>::bytes, seen)) return rc;
  return launch_dependent<GradArgs>(gradient_kernel<W>, dim3(GradGrid<W>::blocks, a.P.E),
                                    kThreads, GradSmem<W>::bytes, s, a);
}

}  // namespace

int fused_predict(const Params &P, const FeatureMap &f, const double *xy, int64_t rows, float *Y,
                  cudaStream_t s) {
  if (rows <= 0) return 0;
  FwdArgs a{};
  a.P = P;
  a.f = f;
  a.xy = xy;
  a.rows = rows;
  a.Y = Y;
  a.ys = (P.outs + 3) / 4 * 4;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t per_net = std::max(1, sms / P.E);
  const int64_t need = (rows + kRows * kPredictTiles - 1) / (kRows * kPredictTiles);
  const unsigned gx = (unsigned)std::min<int64_t>(per_net, need);
  return P.W == 128 ? launch_predict<128>(a, gx, s) : launch_predict<64>(a, gx, s);
}

int fused_gradient(const Params &P, const FeatureMap &f, const double *xy, const double *T,
                   const int *idx, int64_t rows, const float *tmean, const float *tinv,
                   const TrainBuffers &b, const AdamStep *adam, float *loss, cudaStream_t s) {
  FwdArgs a{};
  a.P = P;
  a.f = f;
  a.xy = xy;
  a.rows = rows;
  a.T = T;
  a.idx = idx;
  a.tmean = tmean;
  a.tinv = tinv;
  a.b = b;
  a.loss = loss;
  int rc = P.W == 128 ? launch_train<128>(a, s) : launch_train<64>(a, s);
  if (rc) return rc;
  GradArgs g{};
  g.P = P;
  g.b = b;
  g.rows = rows;
  g.adam = adam != nullptr;
  if (adam) g.a = *adam;
  return P.W == 128 ? launch_gradient<128>(g, s) : launch_gradient<64>(g, s);
}

}  // namespace mlp
}  // namespace chaos
