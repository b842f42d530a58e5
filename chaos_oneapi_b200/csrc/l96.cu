// Warp-per-point sweep for the 40-dimensional Lorenz-96 model
//   x_i' = (x_{i+1} - x_{i-2}) x_{i-1} - gamma x_i + F   (cyclic)
// with its k <= 40 tangent vectors: Dormand-Prince 5(4) in FP32, modified
// Gram-Schmidt QR in FP64, log-norms in FP64.
//
// Layout.  One warp owns one point.  Its 32 lanes form 4 groups of 8; a group
// holds one 40-vector, 5 consecutive components per lane, so the stencil's
// neighbours i-2, i-1, i+1 are in the lane except at its edges, where 3
// shuffles per stage fetch them from the adjacent lanes (cyclically within
// the group).  A step runs the state first (every group computes it, so each
// lane has the stage points it needs for J without any exchange), then the k
// tangent vectors four at a time.  Per-step registers: the lane's 5
// components of the 7 stage points as Jacobian coefficients, plus one
// vector's Dopri5 stages.  Between steps the tangent vectors live in shared
// memory, double-buffered (accepted / candidate, swapped on acceptance):
// 2 x k x 40 floats per warp.  Their first-stage derivatives are not stored:
// J(x) v at the step's start costs one stencil pass with the stage-0
// Jacobian coefficients the state pass computes anyway (the same floats an
// FSAL copy would hold), and leaving them out halves the shared memory per
// point, so twice as many points fit on an SM.  Gram-Schmidt works on
// FP64 copies in registers, two lanes per vector, and keeps the finished ones
// over both halves (k x 40 doubles); see mgs_qr.
//
// The phase and renormalisation logic follows adaptive.cuh (transient /
// alignment / averaging with clamped landings, the renormalisation interval
// of renorm.cuh from the Gram-Schmidt cancellation and the shrinking of the
// norms, norm products flushed into Kahan sums, escape radius, step budget);
// every decision is warp-uniform.
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.h"
#include "renorm.cuh"

namespace chaos {
namespace l96 {

constexpr int N = 40;        // model dimension
constexpr int G = 4;         // vectors processed at once per warp (lane groups)
constexpr int C = 5;         // components per lane
constexpr int WARPS = 4;     // warps (points) per block
constexpr unsigned FULL = 0xffffffffu;

struct DPc {  // Dormand-Prince 5(4), cuda/tools/dopri.dp.cpp:14-44
  static constexpr float a21 = 0.2f;
  static constexpr float a31 = 3.f / 40.f, a32 = 9.f / 40.f;
  static constexpr float a41 = 44.f / 45.f, a42 = -56.f / 15.f, a43 = 32.f / 9.f;
  static constexpr float a51 = 19372.f / 6561.f, a52 = -25360.f / 2187.f, a53 = 64448.f / 6561.f,
                         a54 = -212.f / 729.f;
  static constexpr float a61 = 9017.f / 3168.f, a62 = -355.f / 33.f, a63 = 46732.f / 5247.f,
                         a64 = 49.f / 176.f, a65 = -5103.f / 18656.f;
  static constexpr float b1 = 35.f / 384.f, b3 = 500.f / 1113.f, b4 = 125.f / 192.f,
                         b5 = -2187.f / 6784.f, b6 = 11.f / 84.f;
  static constexpr float e1 = 71.f / 57600.f, e3 = -71.f / 16695.f, e4 = 71.f / 1920.f,
                         e5 = -17253.f / 339200.f, e6 = 22.f / 525.f, e7 = -1.f / 40.f;
};

// Neighbour fetch within the lane's group: left lane's components 3, 4 and
// the right lane's component 0.
struct Nb {
  float l3, l4, r0;
};
__device__ __forceinline__ Nb neighbours(const float (&v)[C], int left, int right) {
  Nb n;
  n.l3 = __shfl_sync(FULL, v[3], left);
  n.l4 = __shfl_sync(FULL, v[4], left);
  n.r0 = __shfl_sync(FULL, v[0], right);
  return n;
}
// Extended window w[-2..5] of the lane's components: at(j) = w[j] for j in -2..5.
struct Win {
  float w[C + 3];
  __device__ __forceinline__ float at(int j) const { return w[j + 2]; }
};
__device__ __forceinline__ Win window(const float (&v)[C], const Nb &n) {
  Win e;
  e.w[0] = n.l3;
  e.w[1] = n.l4;
#pragma unroll
  for (int j = 0; j < C; j++) e.w[j + 2] = v[j];
  e.w[C + 2] = n.r0;
  return e;
}

// Jacobian coefficients of one stage point for the lane's components:
// (J v)_i = (v_{i+1} - v_{i-2}) A_i + B_i v_{i-1} - gamma v_i,
// A_i = x_{i-1}, B_i = x_{i+1} - x_{i-2}.
struct Jc {
  float A[C], B[C];
};

// a b + c d and the longer sums of the passes below, left to right, with their
// multiply-adds explicit: the compiler may fuse either product, and a sweep's
// step sequence must not depend on its choice.
__device__ __forceinline__ float lin(float a, float b, float c, float d) {
  return fmaf(a, b, __fmul_rn(c, d));
}
__device__ __forceinline__ float lin_on(float acc) { return acc; }
template <class... R>
__device__ __forceinline__ float lin_on(float acc, float c, float k, R... r) {
  return lin_on(fmaf(c, k, acc), r...);
}
template <class... R>
__device__ __forceinline__ float lin(float c1, float k1, float c2, float k2, float c3, float k3,
                                     R... r) {
  return lin_on(lin(c1, k1, c2, k2), c3, k3, r...);
}

__device__ __forceinline__ void rhs_state(const float (&x)[C], float (&dx)[C], Jc &jc, float F,
                                          float gam, int left, int right) {
  const Win e = window(x, neighbours(x, left, right));
#pragma unroll
  for (int j = 0; j < C; j++) {
    jc.A[j] = e.at(j - 1);
    jc.B[j] = e.at(j + 1) - e.at(j - 2);
    dx[j] = lin(jc.B[j], jc.A[j], -gam, e.at(j)) + F;
  }
}

__device__ __forceinline__ void rhs_tangent(const float (&v)[C], float (&dv)[C], const Jc &jc,
                                            float gam, int left, int right) {
  const Win e = window(v, neighbours(v, left, right));
#pragma unroll
  for (int j = 0; j < C; j++)
    dv[j] = fmaf(-gam, e.at(j), lin(e.at(j + 1) - e.at(j - 2), jc.A[j], jc.B[j], e.at(j - 1)));
}

__device__ __forceinline__ float err_term(float y0, float y1, float e, float rtol, float atol,
                                          float acc) {
  const float m = fmaxf(fabsf(y0), fabsf(y1));
  const float r = __fdividef(e, fmaf(rtol, m, atol));
  return fmaf(r, r, acc);
}

// One Dopri5 pass over the lane's 5 components.  rhs(s, arg, out) evaluates
// stage s (1..6; stage 0 = k1 is given) at arg.
template <class RHS>
__device__ __forceinline__ void dopri_pass(const float (&y)[C], const float (&k1)[C], float h,
                                           const RHS &rhs, float (&y1)[C], float (&k7)[C],
                                           float &err2, float rtol, float atol) {
  using T = DPc;
  float k2[C], k3[C], k4[C], k5[C], arg[C], e[C];
#pragma unroll
  for (int j = 0; j < C; j++) arg[j] = fmaf(h, __fmul_rn(T::a21, k1[j]), y[j]);
  rhs(1, arg, k2);
#pragma unroll
  for (int j = 0; j < C; j++) arg[j] = fmaf(h, lin(T::a31, k1[j], T::a32, k2[j]), y[j]);
  rhs(2, arg, k3);
#pragma unroll
  for (int j = 0; j < C; j++)
    arg[j] = fmaf(h, lin(T::a41, k1[j], T::a42, k2[j], T::a43, k3[j]), y[j]);
  rhs(3, arg, k4);
#pragma unroll
  for (int j = 0; j < C; j++)
    arg[j] = fmaf(h, lin(T::a51, k1[j], T::a52, k2[j], T::a53, k3[j], T::a54, k4[j]), y[j]);
  rhs(4, arg, k5);
#pragma unroll
  for (int j = 0; j < C; j++) {
    arg[j] = fmaf(h, lin(T::a61, k1[j], T::a62, k2[j], T::a63, k3[j], T::a64, k4[j], T::a65, k5[j]),
                  y[j]);
    e[j] = lin(T::e1, k1[j], T::e3, k3[j], T::e4, k4[j], T::e5, k5[j]);
    y1[j] = lin(T::b1, k1[j], T::b3, k3[j], T::b4, k4[j], T::b5, k5[j]);
  }
  {
    float k6[C];
    rhs(5, arg, k6);
#pragma unroll
    for (int j = 0; j < C; j++) {
      y1[j] = fmaf(h, fmaf(T::b6, k6[j], y1[j]), y[j]);
      e[j] = fmaf(T::e6, k6[j], e[j]);
    }
  }
  rhs(6, y1, k7);
#pragma unroll
  for (int j = 0; j < C; j++) {
    e[j] = fmaf(T::e7, k7[j], e[j]);
    err2 = err_term(y[j], y1[j], h * e[j], rtol, atol, err2);
  }
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  return v;
}
enum Phase : int { kTransient = 0, kAlign = 1, kAverage = 2 };

struct Warp {
  // per lane
  float x[C], kx[C];
  double sum[2], comp[2], prod[2];  // exponents lane and lane + 32
  // warp-uniform
  float F, gam, h, fac_old;
  bool reject;
  int phase;
  double t_phase, phase_len, t_gs, L, rate_max, t_avg;
  long long steps;
  long long pt;
};

__device__ __forceinline__ void flush_logs(Warp &w) {
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const double y = log(w.prod[i]) - w.comp[i];
    const double s = w.sum[i] + y;
    w.comp[i] = (s - w.sum[i]) - y;
    w.sum[i] = s;
    w.prod[i] = 1.0;
  }
}

// Gram-Schmidt layout.  Two lanes hold one vector in registers, 20 components
// each, so a warp orthogonalises a block of 16 vectors at once; the finished
// vectors lie in shared memory in FP64.  The 40 components are eight runs of
// five; lane 0 of a pair takes runs 0, 4, 2, 6, lane 1 runs 1, 5, 3, 7, each
// lane's 20 contiguous in shared memory (gs_pos).  A dot product is a chain of
// five multiply-adds per run, the runs added as ((0 + 4) + (2 + 6)) + ((1 + 5) +
// (3 + 7)): two additions in the lane and one exchange in the pair.  (With one
// run per lane, the layout of the steps, the same sum was three shuffle levels
// per dot product, and each vector was read and rewritten in shared memory for
// every earlier one.)
constexpr int kPairVecs = 16;
__device__ __forceinline__ int gs_run(int half, int i) {  // run i of a lane's four
  return half + ((i & 1) << 2) + (i & 2);
}
__device__ __forceinline__ int gs_pos(int run) {  // first double of a run in a stored vector
  return (run & 1) * 20 + (((run >> 2) & 1) + (run & 2)) * 5;
}

// The lane's half of a dot product with the stored half vector q (16-byte
// aligned; both lanes of every pair read the same two addresses: broadcasts).
__device__ __forceinline__ double pair_sum(const double (&p)[4]) {
  const double h = (p[0] + p[1]) + (p[2] + p[3]);
  return h + __shfl_xor_sync(FULL, h, 1);
}
__device__ __forceinline__ double dot_stored(const double2 *q, const double (&w)[20]) {
  double p[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int i = 0; i < 10; i++) {
    const double2 t = q[i];
    p[(2 * i) / 5] = fma(t.x, w[2 * i], p[(2 * i) / 5]);
    p[(2 * i + 1) / 5] = fma(t.y, w[2 * i + 1], p[(2 * i + 1) / 5]);
  }
  return pair_sum(p);
}
__device__ __forceinline__ double dot_self(const double (&w)[20]) {
  double p[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int i = 0; i < 20; i++) p[i / 5] = fma(w[i], w[i], p[i / 5]);
  return pair_sum(p);
}
__device__ __forceinline__ void subtract_stored(const double2 *q, double c, double (&w)[20]) {
#pragma unroll
  for (int i = 0; i < 10; i++) {
    const double2 t = q[i];
    w[2 * i] = fma(-c, t.x, w[2 * i]);
    w[2 * i + 1] = fma(-c, t.y, w[2 * i + 1]);
  }
}

// Modified Gram-Schmidt in FP64 on the k vectors of V (k x 40, FP32, in the
// lower or upper half of the warp's area `base`, 2 k x 40 floats); the
// orthonormal vectors end in the lower half.
//
// Left-looking: a block of 16 vectors is loaded into registers, the finished
// vectors before it are projected out one by one, then the block's own, each
// normalised and stored as its turn comes.  Every vector meets its predecessors
// in the same order as in the right-looking form, with the same operations.
// The area holds the finished vectors in FP64 (vector q over floats 80 q ..
// 80 q + 79) while the later ones wait in the upper half (vector j at floats
// 40 k + 40 j): storing the vectors of block b, the last at 80 (16 b + 15) + 79,
// never reaches the first one not yet loaded, at 40 k + 640 (b + 1), since
// that one exists only if 16 (b + 1) < k.
// A pass of 40 vectors is a chain of 40 normalisations (dot product, reciprocal
// root, store, dot product) and about 6,000 FP64 instructions; beside three
// other warps on the scheduler it takes 91,000 cycles (right-looking, with one
// run per lane: 135,000, 71 % of the sweep's time).  64^2 points, T 5 + 50:
// 135.8 -> 115.9 ms.
struct GsResult {
  double cancel;  // max |v_q|^2 / r_q^2, the cancellation factor
  double rmin;    // the smallest r_q
  double r[2];    // r_q of the exponents this lane owns (lane, lane + 32); else 1
  bool ok;
};
// (not inlined: its registers are the vectors', the step's are saved around the
// call, once per pass)
__device__ __noinline__ GsResult mgs_qr(const float *V, float *base, int k, int lane) {
  double *W = reinterpret_cast<double *>(base);
  float *U = base + k * N;
  if (V == base) {  // to the upper half
    for (int i = lane; i < k * N / 4; i += 32)
      reinterpret_cast<float4 *>(U)[i] = reinterpret_cast<const float4 *>(V)[i];
    __syncwarp();
  }
  const int pair = lane >> 1, half = lane & 1;
  double cancel = 1.0, rmin = 1e300;
  GsResult res;
  res.r[0] = res.r[1] = 1.0;
  res.ok = true;
  for (int v0 = 0; v0 < k; v0 += kPairVecs) {
    const int vec = v0 + pair;
    double x[20];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < C; j++)
        x[i * C + j] = vec < k ? (double)U[vec * N + gs_run(half, i) * C + j] : 0.0;
    const double nb = dot_self(x);  // squared norm before the projections
    __syncwarp();                   // the whole block is in registers
    for (int q = 0; q < v0; q++) {
      const double2 *wq = reinterpret_cast<const double2 *>(W + q * N + half * 20);
      const double c = dot_stored(wq, x);
      subtract_stored(wq, c, x);
    }
    const int nv = min(kPairVecs, k - v0);
    double s = 1.0, r = 1.0;
    for (int i = 0; i < nv; i++) {
      const double t = dot_self(x);  // every pair's; vector i's counts
      double2 *wq = reinterpret_cast<double2 *>(W + (v0 + i) * N + half * 20);
      if (pair == i) {
        s = t;
        const double inv = rsqrt(t);
        r = t * inv;
#pragma unroll
        for (int j = 0; j < 20; j++) x[j] *= inv;
#pragma unroll
        for (int j = 0; j < 10; j++) wq[j] = make_double2(x[2 * j], x[2 * j + 1]);
      }
      __syncwarp();
      if (i + 1 < nv) {
        const double c = dot_stored(wq, x);
        if (pair > i) subtract_stored(wq, c, x);
      }
    }
    const bool mine = vec < k;
    res.ok = __all_sync(FULL, !mine || ((r > 0.0) && (r < 1e300))) && res.ok;
    if (mine) {
      rmin = fmin(rmin, r);
      // norm before any projection vs r (the first vector has none)
      if (vec > 0) cancel = fmax(cancel, nb / s);
    }
    // the norms to the lanes that own their exponents: q in lane q % 32, slot q / 32
    const double rq = __shfl_sync(FULL, r, 2 * (lane & (kPairVecs - 1)));
    const int q = v0 + (lane & (kPairVecs - 1));
    if (q < k && (q & 31) == lane) {
      if (q >> 5) res.r[1] = rq;
      else res.r[0] = rq;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    cancel = fmax(cancel, __shfl_xor_sync(FULL, cancel, o));
    rmin = fmin(rmin, __shfl_xor_sync(FULL, rmin, o));
  }
  // FP64 -> FP32 into the lower half, four vectors at a time, each chunk read
  // whole before it is written: vector q's floats end below 160 (q + 1) bytes,
  // its unread doubles start at 320 q.
  for (int v0 = 0; v0 < k; v0 += G) {
    const int vec = v0 + (lane >> 3), run = lane & 7;
    double d[C];
#pragma unroll
    for (int j = 0; j < C; j++) d[j] = vec < k ? W[vec * N + gs_pos(run) + j] : 0.0;
    __syncwarp();
    if (vec < k) {
#pragma unroll
      for (int j = 0; j < C; j++) base[vec * N + run * C + j] = (float)d[j];
    }
    __syncwarp();
  }
  res.cancel = cancel;
  res.rmin = rmin;
  return res;
}

__device__ void finish(Warp &w, const AdaptiveArgs &a, int k, int lane, int status) {
  flush_logs(w);
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const int q = lane + 32 * i;
    if (q < k) {
      const double lam = status ? __longlong_as_double(0x7ff8000000000000ULL) : w.sum[i] / w.t_avg;
      a.spectrum.base[w.pt * a.spectrum.ps + q * a.spectrum.cs] = lam;
    }
  }
  if (lane == 0) {
    if (a.status) a.status[w.pt] = status;
    if (a.steps) a.steps[w.pt] = w.steps;
  }
}

// What a launch runs of its points: everything, their transients only (end
// states into a.resume), or their averaging phases from there.
enum Mode : int { kWhole = 0, kTransients = 1, kAveraging = 2 };

template <int MODE>
__device__ __forceinline__ long long fetch(const AdaptiveArgs &a, int lane, long long direct) {
  if (!a.queue) return direct;
  for (;;) {
    unsigned long long q = 0;
    if (lane == 0) q = atomicAdd(a.queue, 1ULL);
    q = __shfl_sync(FULL, q, 0);
    if (q >= (unsigned long long)a.P) return a.P;
    const long long pt =
        MODE == kAveraging
            ? (long long)a.order[q]
            : (long long)((q * (unsigned long long)a.queue_stride) % (unsigned long long)a.P);
    if (MODE != kAveraging || a.resume.steps[pt] >= 0) return pt;  // else ended in its transient
  }
}

template <int MODE>
__global__ void __launch_bounds__(WARPS * 32, 4) l96_kernel(const AdaptiveArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int g = lane >> 3, li = lane & 7;
  const int left = g * 8 + ((li + 7) & 7), right = g * 8 + ((li + 1) & 7);
  const int k = a.k;
  const size_t per_warp = (size_t)2 * k * N;  // floats: accepted and candidate vectors
  float *base = reinterpret_cast<float *>(smem) + wid * per_warp;
  float *V = base, *V1 = base + k * N;

  const float rtol = (float)a.rtol, atol = (float)a.atol;
  const float tau = 0.3f * logf(1.0f / fmaxf(rtol, 5.96e-8f));
  const double hmax = a.hmax > 0 ? a.hmax : 1e300, hmin = fmax(a.hmin, 1e-12);
  const float esc = (float)(a.escape > 0 ? a.escape : 1e4);
  constexpr float safe = 0.9f, beta = 0.04f, facc1 = 5.0f, facc2 = 0.1f;
  constexpr float expo1 = 0.2f - beta * 0.75f;

  Warp w;
  long long direct = (long long)blockIdx.x * WARPS + wid;
  w.pt = fetch<MODE>(a, lane, direct);

  auto start_tangent = [&]() {
    for (int idx = lane; idx < k * N; idx += 32) V[idx] = (idx / N == idx % N) ? 1.f : 0.f;
    __syncwarp();
    w.fac_old = 1e-4f;
    w.t_phase = 0.0;
    w.t_gs = 0.0;
    if (a.t_align > 0) {
      w.phase = kAlign;
      w.phase_len = a.t_align;
    } else {
      w.phase = kAverage;
      w.phase_len = w.t_avg;
    }
  };
  auto start_point = [&]() {
    w.F = (float)a.params.base[w.pt * a.params.ps + 0 * a.params.cs];
    w.gam = (float)a.params.base[w.pt * a.params.ps + 1 * a.params.cs];
    if constexpr (MODE == kAveraging) {
      const float *st = static_cast<const float *>(a.resume.state) + w.pt;
#pragma unroll
      for (int j = 0; j < C; j++) {
        w.x[j] = st[(li * C + j) * a.P];
        w.kx[j] = st[(N + li * C + j) * a.P];
      }
      w.h = st[2 * N * a.P];
      const long long steps = a.resume.steps[w.pt];
      w.reject = (steps & kResumeReject) != 0;
      w.steps = steps & ~kResumeReject;
    } else {
#pragma unroll
      for (int j = 0; j < C; j++)
        w.x[j] = (float)a.inits.base[w.pt * a.inits.ps + (li * C + j) * a.inits.cs];
      w.h = (float)a.h0;
      w.reject = false;
      w.steps = 0;
    }
    w.fac_old = 1e-4f;
    w.t_avg = a.t_avg_per_point ? a.t_avg_per_point[w.pt] : a.t_avg;
    w.L = a.dt_renorm / adaptive::kRenormSplitInit;
    w.rate_max = adaptive::initial_renorm_rate(tau, (float)a.dt_renorm);
#pragma unroll
    for (int i = 0; i < 2; i++) w.sum[i] = w.comp[i] = 0.0, w.prod[i] = 1.0;
    if constexpr (MODE != kAveraging) {
      Jc jc;
      rhs_state(w.x, w.kx, jc, w.F, w.gam, left, right);
    }
    if (MODE != kAveraging && a.t_transient > 0) {
      w.phase = kTransient;
      w.phase_len = a.t_transient;
      w.t_phase = 0.0;
      w.t_gs = 0.0;
    } else {
      start_tangent();
    }
  };
  // The transient's end state, and the expected cost of the averaging phase.
  auto save_point = [&]() {
    float *st = static_cast<float *>(a.resume.state) + w.pt;
    if (g == 0) {
#pragma unroll
      for (int j = 0; j < C; j++) {
        st[(li * C + j) * a.P] = w.x[j];
        st[(N + li * C + j) * a.P] = w.kx[j];
      }
    }
    if (lane == 0) {
      st[2 * N * a.P] = w.h;
      a.resume.steps[w.pt] = w.steps | (w.reject ? kResumeReject : 0);
      a.resume.cost[w.pt] = (double)w.steps * (w.t_avg / a.t_transient);
    }
  };
  // Gram-Schmidt of the warp's point; false on a degenerate basis.
  auto gram_schmidt = [&]() -> bool {
    const GsResult gs = mgs_qr(V, base, k, lane);
    V = base;  // the orthonormal vectors are in the lower half now
    V1 = base + k * N;
    if (!gs.ok) return false;
    if (w.phase == kAverage) {
      bool fl = false;
#pragma unroll
      for (int i = 0; i < 2; i++) {
        w.prod[i] *= gs.r[i];
        fl = fl || !(w.prod[i] < 1e150 && w.prod[i] > 1e-150);
      }
      if (__any_sync(FULL, fl)) flush_logs(w);
    }
    if (w.t_gs > 0.0)  // the policy of every adaptive form (renorm.cuh)
      adaptive::next_renorm_interval(w.L, w.rate_max, (float)gs.cancel, gs.rmin, w.t_gs, tau,
                                     a.dt_renorm);
    w.t_gs = 0.0;
    return true;
  };

  if (w.pt < a.P) start_point();
  while (w.pt < a.P) {
    constexpr int kSaved = 5;
    int status = -1;  // -1: running; kSaved: the transient is done
    if (w.steps == 0) {  // an initial state outside the escape radius (adaptive.cuh: state_inside)
      bool inside = true;
#pragma unroll
      for (int j = 0; j < C; j++) inside = inside && (fabsf(w.x[j]) <= esc);
      if (!__all_sync(FULL, inside)) status = 4;
    }
    if (status < 0 && w.steps >= a.max_steps) status = 3;
    if (status < 0 && !((double)w.h >= hmin)) status = 2;
    if (status < 0) {
      const double remaining = w.phase_len - w.t_phase;
      const bool clamped = (double)w.h >= remaining;
      const float h = clamped ? (float)remaining : w.h;
      const bool joint = MODE == kAveraging || (MODE == kWhole && w.phase != kTransient);
      w.steps++;
      // state pass: every group computes it; the stage points become J coefficients
      Jc jcs[7];
      float x1[C], kx1[C], err_state = 0.f;
      {
        auto rhs = [&](int s, const float (&arg)[C], float (&out)[C]) {
          rhs_state(arg, out, jcs[s], w.F, w.gam, left, right);
        };
        // stage 0 coefficients at the current state
        float dummy[C];
        rhs_state(w.x, dummy, jcs[0], w.F, w.gam, left, right);
        dopri_pass(w.x, w.kx, h, rhs, x1, kx1, err_state, rtol, atol);
      }
      float err2 = (g == 0) ? err_state : 0.f;
      if (joint) {
        for (int r = 0; r < (k + G - 1) / G; r++) {
          const int vec = r * G + g;
          const bool valid = vec < k;
          float v[C], kv[C], v1[C], kv1[C];
#pragma unroll
          for (int j = 0; j < C; j++) v[j] = valid ? V[vec * N + li * C + j] : 0.f;
          // first stage: J(x) v with the state pass's stage-0 coefficients
          rhs_tangent(v, kv, jcs[0], w.gam, left, right);
          float e2 = 0.f;
          auto rhs = [&](int s, const float (&arg)[C], float (&out)[C]) {
            rhs_tangent(arg, out, jcs[s], w.gam, left, right);
          };
          dopri_pass(v, kv, h, rhs, v1, kv1, e2, rtol, atol);
          if (valid) {
            err2 += e2;
#pragma unroll
            for (int j = 0; j < C; j++) V1[vec * N + li * C + j] = v1[j];
          }
        }
      }
      const float nc = joint ? (float)(N * (1 + k)) : (float)N;
      const float err = sqrtf(warp_sum(err2) / nc);
      if (!(err == err) || err > 3.0e38f) {  // the other forms' rule (adaptive.cuh: point_finite)
        bool fin = (w.F - w.F == 0.f) && (w.gam - w.gam == 0.f);
#pragma unroll
        for (int j = 0; j < C; j++) fin = fin && (w.x[j] - w.x[j] == 0.f);
        if (!__all_sync(FULL, fin)) {
          status = 1;
        } else {
          w.h = h / 5.0f;  // the controller's largest reduction
          w.reject = true;
        }
      } else {
        const float fac11 = exp2f(expo1 * __log2f(fmaxf(err, 1e-30f)));
        if (err <= 1.0f) {
          float fac = fac11 * exp2f(-beta * __log2f(w.fac_old));
          fac = fmaxf(facc2, fminf(facc1, fac * (1.0f / safe)));
          float hnew = h * __fdividef(1.0f, fac);
          w.fac_old = fmaxf(err, 1e-4f);
#pragma unroll
          for (int j = 0; j < C; j++) {
            w.x[j] = x1[j];
            w.kx[j] = kx1[j];
          }
          __syncwarp();
          if (joint) {  // accept the candidate: swap buffers
            float *t0 = V;
            V = V1;
            V1 = t0;
          }
          if ((double)hnew > hmax) hnew = (float)hmax;
          if (w.reject && hnew > h) hnew = h;
          w.reject = false;
          if (!clamped || hnew < h) w.h = hnew;
          w.t_phase = clamped ? w.phase_len : w.t_phase + (double)h;
          w.t_gs += (double)h;
          bool inside = true;
#pragma unroll
          for (int j = 0; j < C; j++) inside = inside && (fabsf(w.x[j]) <= esc);
          if (!__all_sync(FULL, inside)) {
            status = 4;
          } else if (clamped) {
            if (MODE == kTransients) {
              save_point();
              status = kSaved;
            } else if (w.phase == kTransient) {
              start_tangent();
            } else if (w.phase == kAlign) {
              if (!gram_schmidt()) status = 1;
              w.phase = kAverage;
              w.phase_len = w.t_avg;
              w.t_phase = 0.0;
            } else {
              status = gram_schmidt() ? 0 : 1;
            }
          } else if (joint && w.t_gs >= w.L) {
            if (!gram_schmidt()) status = 1;
          }
        } else {
          w.h = h * __fdividef(1.0f, fminf(facc1, fac11 * (1.0f / safe)));
          w.reject = true;
        }
      }
    }
    if (status >= 0) {
      if (MODE != kTransients || status != kSaved) finish(w, a, k, lane, status);
      if (MODE == kTransients && status != kSaved && lane == 0) {
        a.resume.steps[w.pt] = -1;
        a.resume.cost[w.pt] = 0.0;
      }
      w.pt = fetch<MODE>(a, lane, a.P);
      if (w.pt < a.P) start_point();
    }
  }
}

}  // namespace l96

namespace {
template <int MODE> int64_t l96_blocks(const AdaptiveArgs &a, size_t smem) {
  using namespace l96;
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, l96_kernel<MODE>, WARPS * 32, smem);
  return std::min<int64_t>((int64_t)std::max(1, per_sm) * sms, (a.P + WARPS - 1) / WARPS);
}
size_t l96_smem(int k) { return (size_t)l96::WARPS * 2 * k * l96::N * sizeof(float); }
template <int MODE> int launch_l96_mode(const AdaptiveArgs &a, cudaStream_t s) {
  using namespace l96;
  const size_t smem = MODE == kTransients ? 0 : l96_smem(a.k);
  if (smem) {
    const cudaError_t e = cudaFuncSetAttribute(
        l96_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  const int64_t grid = a.queue ? l96_blocks<MODE>(a, smem) : (a.P + WARPS - 1) / WARPS;
  l96_kernel<MODE><<<(unsigned)grid, WARPS * 32, smem, s>>>(a);
  return (int)cudaGetLastError();
}
bool l96_supported(int integrator, int precision, int k) {
  return integrator == kDopri5 && precision == kFP32 && k >= 1 && k <= l96::N;
}
}  // namespace

int launch_l96_warp(int integrator, int precision, const AdaptiveArgs &a, int, cudaStream_t s) {
  if (!l96_supported(integrator, precision, a.k)) return kErrUnsupported;
  return launch_l96_mode<l96::kWhole>(a, s);
}

int64_t l96_resident(int integrator, int precision, int k) {
  if (!l96_supported(integrator, precision, k)) return 0;
  const size_t smem = l96_smem(k);
  if (cudaFuncSetAttribute(l96::l96_kernel<l96::kWhole>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)smem) != cudaSuccess)
    return 0;
  AdaptiveArgs all{};
  all.P = INT64_MAX / 2;
  return l96_blocks<l96::kWhole>(all, smem) * l96::WARPS;
}

int launch_l96_two_phase(int integrator, int precision, const AdaptiveArgs &a, void *order_scratch,
                         cudaStream_t s) {
  if (!l96_supported(integrator, precision, a.k)) return kErrUnsupported;
  int rc = launch_l96_mode<l96::kTransients>(a, s);
  if (!rc) rc = (int)cudaMemsetAsync(a.queue, 0, sizeof(unsigned long long), s);
  if (!rc)
    rc = launch_order_longest_first(a.resume.cost, a.P, const_cast<int32_t *>(a.order),
                                    order_scratch, s);
  return rc ? rc : launch_l96_mode<l96::kAveraging>(a, s);
}

}  // namespace chaos
