// Adaptive sweep kernels for the 3-4-dimensional flows (see adaptive.cuh for
// the numerics).  One thread per point.  Two launch forms share one kernel:
//  * direct: thread i integrates point i;
//  * persistent work queue: a grid sized to the machine (a multiple of the
//    SM count) whose threads pull point indices from a device counter, so a
//    thread whose point needed fewer adaptive steps (or a shorter averaging
//    time) starts the next point at once instead of idling until the
//    slowest lane of its warp is done.  A sweep of a few waves runs as two
//    such launches, every point's transient, then the averaging phases
//    longest first (launch_adaptive_two_phase).
#include <algorithm>

#include "adaptive.cuh"

namespace chaos {
namespace adaptive {

// The queue hands out points in the order q -> (q * stride) mod P (stride
// coprime to P, so a permutation): neighbouring grid points cost alike, and
// spreading them over the run keeps a cluster of expensive points (a chaotic
// band, escaping orbits) from forming the tail of the launch.
// With an explicit order (longest averaging time first, order.cu) the queue
// hands out order[q] instead.
__device__ __forceinline__ int64_t next_point(const AdaptiveArgs &a) {
  const unsigned long long q = atomicAdd(a.queue, 1ULL);
  if (q >= (unsigned long long)a.P) return a.P;
  if (a.order) return (int64_t)a.order[q];
  return (int64_t)((q * (unsigned long long)a.queue_stride) % (unsigned long long)a.P);
}

// RESUME: the next point that has an averaging phase left (points that ended in
// their transient are in the order too).
template <bool RESUME> __device__ __forceinline__ int64_t next_open_point(const AdaptiveArgs &a) {
  int64_t pt = next_point(a);
  if (RESUME)
    while (pt < a.P && a.resume.steps[pt] < 0) pt = next_point(a);
  return pt;
}
template <bool RESUME, class M, int K, class R, int INTEG>
__device__ __forceinline__ void lane_begin(Lane<M, K, R, INTEG> &L, const AdaptiveArgs &a,
                                           int64_t pt) {
  if constexpr (RESUME) lane_resume(L, a, pt);
  else lane_start(L, a, pt);
}

// Each lane owns one point at a time and runs it as a state machine (one
// step attempt per loop iteration), so a lane never waits for another lane's
// phase or renormalisation interval to end: when its point is done it takes
// the next one from the queue (persistent form) and carries on.  Gram-Schmidt
// is voted per warp: when any lane is due, every lane past its transient
// renormalises in the same pass.
// MINB: resident 128-thread blocks per SM the kernel is compiled for (a
// register cap: 3 -> at most 168 registers, 4 -> 128, 5 -> 96 with a few spills); the
// autotuner picks the variant, except in batches (kBatchVariant).
// RESUME: the averaging phases of points whose transients have run.
template <class M, int K, class R, int INTEG, int MINB, bool RESUME = false>
__global__ void __launch_bounds__(128, MINB) sweep_kernel(const AdaptiveArgs a) {
  const Ctl &c = a.ctl;
  Lane<M, K, R, INTEG> L;
  int64_t pt = a.queue ? next_open_point<RESUME>(a) : (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  bool active = pt < a.P;
  if (active) lane_begin<RESUME>(L, a, pt);
  while (__any_sync(0xffffffffu, active)) {
    if (active && lane_step(L, a, c) == kFinished) {
      pt = a.queue ? next_open_point<RESUME>(a) : a.P;
      active = pt < a.P;
      if (active) lane_begin<RESUME>(L, a, pt);
    }
    const bool due = active && L.phase != kTransient && L.t_gs >= L.L;
    if (__any_sync(0xffffffffu, due)) {
      if (active && L.phase != kTransient && L.t_gs > 0.f && !lane_gram_schmidt(L, a, c)) {
        lane_finish(L, a, 1);
        pt = a.queue ? next_open_point<RESUME>(a) : a.P;
        active = pt < a.P;
        if (active) lane_begin<RESUME>(L, a, pt);
      }
    }
  }
}

// The transients of all points, one thread each (neighbouring points cost
// alike), the state alone.
template <class M, class R, int INTEG>
__global__ void __launch_bounds__(128) transient_kernel(const AdaptiveArgs a) {
  const int64_t pt = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (pt < a.P) run_transient<M, R, INTEG>(a, a.ctl, pt);
}

template <class M, class R, int INTEG, bool RESUME> auto sweep_kernel_of(int variant) {
  if constexpr (sizeof(R) == 4) {
    if constexpr (!RESUME)  // (batches have no launch of averaging phases alone)
      if (variant == kBatchVariant) return sweep_kernel<M, M::N, R, INTEG, 3>;
    return variant == 1 ? sweep_kernel<M, M::N, R, INTEG, 5, RESUME>
                        : sweep_kernel<M, M::N, R, INTEG, 4, RESUME>;
  } else {
    return sweep_kernel<M, M::N, R, INTEG, 1, RESUME>;
  }
}

// What a launch of one (model, precision, integrator) does.
struct Launch {
  enum Kind { kRun, kTransients, kAveraging, kResident } kind;
  int block, variant;
  cudaStream_t s;
  int64_t resident;   // result of kResident: points
  int lanes_per_sm;   // kRun: at most so many (0: all that fit)
};

// One full wave of blocks: resident blocks per SM x SM count.
template <class K> int64_t full_wave(K kern, int block, int lanes_per_sm = 0) {
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, block, 0);
  if (lanes_per_sm > 0) per_sm = std::min(per_sm, lanes_per_sm / block);
  return (int64_t)std::max(1, per_sm) * std::max(1, sms);
}

template <class M, class R, int INTEG> int launch_mri(const AdaptiveArgs &a, Launch &l) {
  const auto kern = sweep_kernel_of<M, R, INTEG, false>(l.variant);
  if (l.kind == Launch::kResident) {
    l.resident = full_wave(kern, l.block) * l.block;
    return 0;
  }
  if (a.k != M::N) return kErrUnsupported;
  AdaptiveArgs ka = a;
  ka.ctl = make_ctl<R>(a);
  const int64_t need = (a.P + l.block - 1) / l.block;  // never more blocks than points need
  if (l.kind == Launch::kTransients) {
    transient_kernel<M, R, INTEG><<<(unsigned)((a.P + 127) / 128), 128, 0, l.s>>>(ka);
  } else if (l.kind == Launch::kAveraging) {
    // Few waves: no more blocks than the one-launch form holds (a longest
    // point's chain of steps, slower the more warps share its scheduler, is
    // the run); many: every block that fits.
    const auto resume = sweep_kernel_of<M, R, INTEG, true>(l.variant);
    const int64_t most = full_wave(resume, l.block), base = full_wave(kern, l.block);
    const int64_t wave = a.P < 3 * most * l.block ? std::min(most, base) : most;
    resume<<<(unsigned)std::min(wave, need), l.block, 0, l.s>>>(ka);
  } else {
    const int64_t grid =
        a.queue ? std::min(full_wave(kern, l.block, l.lanes_per_sm), need) : need;
    kern<<<(unsigned)grid, l.block, 0, l.s>>>(ka);
  }
  return (int)cudaGetLastError();
}

template <class M> int launch_m(int integ, int prec, const AdaptiveArgs &a, Launch &l) {
  if (integ == kDverk65) {
    if (prec == kFP64) return launch_mri<M, double, kDverk65>(a, l);
    if (prec == kFP32) return launch_mri<M, float, kDverk65>(a, l);
  } else if (integ == kDopri5) {
    if (prec == kFP64) return launch_mri<M, double, kDopri5>(a, l);
    if (prec == kFP32) return launch_mri<M, float, kDopri5>(a, l);
  }
  return kErrUnsupported;
}

int launch_model(int model, int integ, int prec, const AdaptiveArgs &a, Launch &l) {
  if (l.block <= 0 || l.block > 128 || l.block % 32) l.block = 128;
  switch (model) {
    case kShimizu: return launch_m<Shimizu>(integ, prec, a, l);
    case kLorenz: return launch_m<Lorenz>(integ, prec, a, l);
    case kRossler: return launch_m<Rossler>(integ, prec, a, l);
    case kChua: return launch_m<Chua>(integ, prec, a, l);
    case kHyperRossler: return launch_m<HyperRossler>(integ, prec, a, l);
    default: return kErrUnsupported;
  }
}

// ----------------------------------------------------------- mixed batch
// One persistent launch over segments of different models (3- and
// 4-dimensional) and per-point averaging times.  Every warp works on one
// segment at a time (warps start on segments round robin); while it does, it
// runs that segment's model-specific loop -- the sweep kernel's loop with the
// segment's queue -- so the step code is specialised to the model, with no
// per-step dispatch, and a lane that finishes a point takes the next point of
// the segment: lanes refill independently, so uneven point lengths do not
// strand warps, and all lanes of a warp run one model's instruction stream.
// When all lanes of the warp are idle (the segment's queue is empty) the warp
// moves on to the next segment with points left.  (Letting lanes move on
// individually mixes models inside warps, which runs every model's step code
// for the warp and measured slower than three separate launches.)

// Next point of segment `seg` for this lane, if any is left.
__device__ __forceinline__ bool batch_take(const BatchArgs &b, int seg, int64_t &pt) {
  const int64_t P = b.seg[seg].P;
  const unsigned long long q = atomicAdd(&b.queues[seg], 1ULL);
  if (q >= (unsigned long long)P) return false;
  pt = b.seg[seg].order
           ? (int64_t)b.seg[seg].order[q]
           : (int64_t)((q * (unsigned long long)b.seg[seg].queue_stride) % (unsigned long long)P);
  return true;
}

template <class M, class R, int INTEG>
__device__ __noinline__ void lane_segment(const BatchArgs &b, int seg, bool active, int64_t pt) {
  const AdaptiveArgs &a = b.seg[seg];
  const Ctl &c = a.ctl;
  Lane<M, M::N, R, INTEG> L;
  if (active) lane_start(L, a, pt);
  while (__any_sync(0xffffffffu, active)) {
    if (active && lane_step(L, a, c) == kFinished) {
      active = batch_take(b, seg, pt);
      if (active) lane_start(L, a, pt);
    }
    const bool due = active && L.phase != kTransient && L.t_gs >= L.L;
    if (__any_sync(0xffffffffu, due)) {
      if (active && L.phase != kTransient && L.t_gs > 0.f && !lane_gram_schmidt(L, a, c)) {
        lane_finish(L, a, 1);
        active = batch_take(b, seg, pt);
        if (active) lane_start(L, a, pt);
      }
    }
  }
}

template <class R, int INTEG>
__global__ void __launch_bounds__(128, sizeof(R) == 4 ? 3 : 1)
    batch_kernel(const __grid_constant__ BatchArgs b) {
  const int warp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  int wseg = warp % b.nseg;
  for (int tried = 0; tried < b.nseg; wseg = (wseg + 1) % b.nseg) {
    int64_t pt = 0;
    const bool active = batch_take(b, wseg, pt);
    if (!__any_sync(0xffffffffu, active)) {  // nothing left here for this warp
      ++tried;
      continue;
    }
    tried = 0;
    switch (b.model[wseg]) {
      case kShimizu: lane_segment<Shimizu, R, INTEG>(b, wseg, active, pt); break;
      case kLorenz: lane_segment<Lorenz, R, INTEG>(b, wseg, active, pt); break;
      case kRossler: lane_segment<Rossler, R, INTEG>(b, wseg, active, pt); break;
      case kChua: lane_segment<Chua, R, INTEG>(b, wseg, active, pt); break;
      default: lane_segment<HyperRossler, R, INTEG>(b, wseg, active, pt); break;
    }
  }
}

}  // namespace adaptive

int launch_batch(int integ, int prec, const BatchArgs &b, int block, cudaStream_t s) {
  using namespace adaptive;
  if (b.nseg <= 0 || b.nseg > kMaxSegments) return kErrUnsupported;
  int64_t total = 0;
  for (int i = 0; i < b.nseg; i++) {
    if (b.model[i] < 0 || b.model[i] >= kLorenz96) return kErrUnsupported;
    const int dim = b.model[i] == kHyperRossler ? 4 : 3;
    if (b.seg[i].k != dim) return kErrUnsupported;
    total += b.seg[i].P;
  }
  if (total <= 0) return 0;
  if (block <= 0 || block > 128 || block % 32) block = 128;
  void (*kern)(BatchArgs) = nullptr;
  if (integ == kDopri5 && prec == kFP32) kern = batch_kernel<float, kDopri5>;
  else if (integ == kDopri5 && prec == kFP64) kern = batch_kernel<double, kDopri5>;
  else if (integ == kDverk65 && prec == kFP32) kern = batch_kernel<float, kDverk65>;
  else if (integ == kDverk65 && prec == kFP64) kern = batch_kernel<double, kDverk65>;
  else return kErrUnsupported;
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, block, 0);
  const int64_t full = (int64_t)std::max(1, per_sm) * sms;
  const int64_t grid = std::min<int64_t>(full, (total + block - 1) / block);
  kern<<<(unsigned)grid, (unsigned)block, 0, s>>>(with_ctl(b, prec));
  return (int)cudaGetLastError();
}

int launch_adaptive(int model, int integ, int prec, const AdaptiveArgs &a, int block, int variant,
                    cudaStream_t s, int lanes_per_sm) {
  using namespace adaptive;
  if (a.P <= 0) return 0;
  Launch l{Launch::kRun, block, variant, s, 0, lanes_per_sm};
  return launch_model(model, integ, prec, a, l);
}

int64_t adaptive_resident(int model, int integ, int prec, int block, int variant) {
  using namespace adaptive;
  Launch l{Launch::kResident, block, variant, nullptr, 0, 0};
  return launch_model(model, integ, prec, AdaptiveArgs{}, l) ? 0 : l.resident;
}

int launch_adaptive_two_phase(int model, int integ, int prec, const AdaptiveArgs &a, int block,
                              int variant, void *order_scratch, cudaStream_t s) {
  using namespace adaptive;
  if (a.P <= 0) return 0;
  Launch l{Launch::kTransients, block, variant, s, 0, 0};
  int rc = launch_model(model, integ, prec, a, l);
  if (!rc)
    rc = launch_order_longest_first(a.resume.cost, a.P, const_cast<int32_t *>(a.order),
                                    order_scratch, s);
  l.kind = Launch::kAveraging;
  return rc ? rc : launch_model(model, integ, prec, a, l);
}

}  // namespace chaos
