// Fused kernels of the surrogate's networks of width 64 and 128 (mlp_fused.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace chaos {
namespace mlp {

constexpr int kFeat = 16;    // input features
constexpr int kOutPad = 16;  // output width padded for the tensor-core tiles

// sin / cos feature frequencies (cycles over the unit box).
struct Freqs {
  float w[8][2];
};

// The domain box and feature frequencies: parameter point -> 16 features.
struct FeatureMap {
  double u0, us, v0, vs;
  Freqs fr;
};

// Parameters of E networks (layout: mlp.cu), as the kernels read them.  The
// BF16 weight matrices are stored in the tensor core's core-matrix order
// (weight_index).
struct Params {
  int E, W, outs;
  int64_t np;
  int64_t off_w[4], off_b[4];
  float *p;
  __nv_bfloat16 *pb;
  float *g, *m, *v;  // gradients (may be null), Adam moments
  int *err;          // set to 1 if a bounded wait gave up
};

inline bool fused_width(int W) { return W == 64 || W == 128; }

// Element (r, c) of a rows x C matrix (C a multiple of 8) in core-matrix
// order: 8 x 8 blocks of 128 bytes, blocks row-major, rows of 16 bytes inside.
__host__ __device__ inline int64_t core_index(int64_t r, int64_t c, int64_t C) {
  return ((r >> 3) * (C >> 3) + (c >> 3)) * 64 + ((r & 7) << 3) + (c & 7);
}

// Where parameter i of a network lies in its BF16 copy: weight matrices of
// the fused widths in core-matrix order, everything else (and other widths)
// in place.
struct BfOrder {
  int W;
  int64_t off_w[4], size_w[4];
  int cols[4];
  __host__ __device__ int64_t at(int64_t i) const {
    if (W != 64 && W != 128) return i;
#pragma unroll
    for (int l = 0; l < 4; l++)
      if (i >= off_w[l] && i < off_w[l] + size_w[l]) {
        const int64_t e = i - off_w[l];
        return off_w[l] + core_index(e / cols[l], e % cols[l], cols[l]);
      }
    return i;
  }
};

// Activations and their gradients of one minibatch in tiles of 128 rows, each
// tile a 128 x W (X, dY: 128 x 16) matrix in core-matrix order.
struct TrainBuffers {
  __nv_bfloat16 *X;         // tiles x (128 x 16), shared by the networks
  __nv_bfloat16 *A[3];      // E x tiles x (128 x W): activations of layers 1..3
  __nv_bfloat16 *dZ[3];     // E x tiles x (128 x W)
  __nv_bfloat16 *dY;        // E x tiles x (128 x 16)
};

// Adam step of the weight-gradient kernel; null: gradients go to Params::g.
struct AdamStep {
  float lr, b1, b2, eps, c1, c2;
};

inline int64_t train_tiles(int64_t rows) { return (rows + 127) / 128; }

// Y[z][row][ys] = outputs (still standardised) of every network on `rows`
// points; ys = outs rounded up to 4.
int fused_predict(const Params &P, const FeatureMap &f, const double *xy, int64_t rows, float *Y,
                  cudaStream_t s);
// Forward and backward pass of every network on `rows` rows (idx null: rows 0
// .. rows - 1 of xy / T, else rows idx[0] ..), then the weight gradients: into
// P.g, or applied by `adam`.  loss (may be null): per-network sums, added to.
int fused_gradient(const Params &P, const FeatureMap &f, const double *xy, const double *T,
                   const int *idx, int64_t rows, const float *tmean, const float *tinv,
                   const TrainBuffers &b, const AdamStep *adam, float *loss, cudaStream_t s);

// One Adam update of a parameter; returns the new value.  The multiply-adds
// are explicit, so that every kernel that applies it rounds alike.
__device__ __forceinline__ float adam_update(float p, float g, float &m, float &v, float lr,
                                             float b1, float b2, float eps, float c1, float c2) {
  const float mi = fmaf(1.f - b1, g, b1 * m);
  const float vi = fmaf((1.f - b2) * g, g, b2 * v);
  m = mi;
  v = vi;
  const float upd = lr * (mi * c1) / (sqrtf(vi * c2) + eps);
  return p - upd;
}

__device__ __forceinline__ float silu(float z) { return z / (1.f + __expf(-z)); }
__device__ __forceinline__ float dsilu(float z) {
  const float sg = 1.f / (1.f + __expf(-z));
  return sg * (1.f + z * (1.f - sg));
}

// z / d for finite z and 1 <= d < kFastDivLimit: an approximate reciprocal
// refined by one step of Newton's method, then Markstein's quotient correction
// (IBM J. Res. Dev. 34, 1990, 111-119).  Equal to the `/` operator, signed zeros
// included, for every z with d = 1 + e^-z and for z = 1 with every d of the range
// (tests/test_gpu_silu.py runs all of them).  The fused epilogues are bound by
// the special-function pipe (71 % busy in predict_kernel), which this uses once
// per quotient.  The callers send a chunk with a larger d (SiLU at z < -85), a
// NaN or an infinite z through the plain functions.
constexpr float kFastDivLimit = 1e37f;
__device__ __forceinline__ float divide_above_one(float z, float d) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  r = fmaf(fmaf(-d, r, 1.f), r, r);
  const float q = z * r;
  return fmaf(-fmaf(q, d, -z), r, q);  // (the remainder negated twice keeps -0)
}
// 1 + e^-z as 1 + 2^(-z log2 e).  Denormal powers may flush to zero: the sum is
// 1 either way.
__device__ __forceinline__ float one_plus_exp_neg(float z) {
  float e;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(-z * 1.44269504088896341f));
  return 1.f + e;
}
// v[i] = SiLU(v[i]), and v[i] = u[i] SiLU'(v[i]): the values of silu / dsilu.
template <int N> __device__ __forceinline__ void silu_chunk(float (&v)[N]) {
  float q[N];
  bool fast = true;
#pragma unroll
  for (int i = 0; i < N; i++) {
    const float d = one_plus_exp_neg(v[i]);
    // false for NaN; at z = +inf the quotient's remainder would be inf - inf.  (A
    // second comparison per unit: 2^20 rows of 4 networks of width 128 take 1.119
    // ms instead of 1.116; a maximum over the chunk, or z x 0 added to d, 1.143 and
    // 1.160.)
    fast = fast && d < kFastDivLimit && v[i] < INFINITY;
    q[i] = divide_above_one(v[i], d);
  }
  if (fast) {
#pragma unroll
    for (int i = 0; i < N; i++) v[i] = q[i];
  } else {
#pragma unroll 1
    for (int i = 0; i < N; i++) {
      float x = 0.f;
#pragma unroll
      for (int j = 0; j < N; j++) x = j == i ? v[j] : x;
      x = silu(x);
#pragma unroll
      for (int j = 0; j < N; j++) v[j] = j == i ? x : v[j];
    }
  }
}
template <int N>
__device__ __forceinline__ void dsilu_chunk(const float (&u)[N], float (&v)[N]) {
  float q[N];
  bool fast = true;
#pragma unroll
  for (int i = 0; i < N; i++) {
    const float d = one_plus_exp_neg(v[i]);
    fast = fast && d < kFastDivLimit;
    const float sg = divide_above_one(1.f, d);
    q[i] = u[i] * (sg * (1.f + v[i] * (1.f - sg)));
  }
  if (fast) {
#pragma unroll
    for (int i = 0; i < N; i++) v[i] = q[i];
  } else {
#pragma unroll 1
    for (int i = 0; i < N; i++) {
      float x = 0.f, y = 0.f;
#pragma unroll
      for (int j = 0; j < N; j++) x = j == i ? v[j] : x, y = j == i ? u[j] : y;
      x = y * dsilu(x);
#pragma unroll
      for (int j = 0; j < N; j++) v[j] = j == i ? x : v[j];
    }
  }
}

// Two of a point's 16 features: sin and cos of 2 pi (w_f . (u, v)).
__device__ __forceinline__ void feature_pair(const FeatureMap &m, float u, float v, int f,
                                             float &sn, float &cs) {
  sincospif(2.f * (m.fr.w[f][0] * u + m.fr.w[f][1] * v), &sn, &cs);
}
__device__ __forceinline__ void normalised(const FeatureMap &m, const double *xy, int64_t i,
                                           float &u, float &v) {
  u = (float)((xy[2 * i] - m.u0) * m.us);
  v = (float)((xy[2 * i + 1] - m.v0) * m.vs);
}

}  // namespace mlp
}  // namespace chaos
