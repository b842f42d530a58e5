// Kernel of the split form (split.cuh): a sweep over one model with one parameter
// point per group of four lanes.
#include <algorithm>
#include <type_traits>

#include "split.cuh"

namespace chaos {
namespace adaptive {

// Next point for the group: its first lane takes it from the queue (in the
// queue's order) and hands it to the other three.
__device__ __forceinline__ int64_t group_next_point(const AdaptiveArgs &a, const Group &g) {
  int64_t pt = 0;
  if (g.r == 0) {
    const unsigned long long q = atomicAdd(a.queue, 1ULL);
    if (q >= (unsigned long long)a.P) pt = a.P;
    else if (a.order) pt = (int64_t)a.order[q];
    else pt = (int64_t)((q * (unsigned long long)a.queue_stride) % (unsigned long long)a.P);
  }
  return __shfl_sync(g.mask, pt, g.base);
}

// Direct form: group i integrates point i.  Persistent form: groups pull
// points from the queue until it is empty.  Gram-Schmidt is voted per warp,
// as in the one-lane form.
template <class M, class R, int INTEG, bool XCH>
__global__ void __launch_bounds__(128) split_kernel(const AdaptiveArgs a) {
  const Group g = group_of();
  const Ctl &c = a.ctl;
  SplitLane<M, R, INTEG, XCH> L;
  int64_t pt = a.queue ? group_next_point(a, g)
                       : ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kSplitLanes;
  bool active = pt < a.P;
  if (active) split_start(L, a, pt, g);
  while (__any_sync(0xffffffffu, active)) {
    if (active && split_step(L, a, c, g) == kFinished) {
      pt = a.queue ? group_next_point(a, g) : a.P;
      active = pt < a.P;
      if (active) split_start(L, a, pt, g);
    }
    const bool due = active && L.phase != kTransient && L.t_gs >= L.L;
    if (__any_sync(0xffffffffu, due)) {
      if (active && L.phase != kTransient && L.t_gs > 0.f && !split_gram_schmidt(L, a, c, g)) {
        split_finish(L, a, g, 1);
        pt = a.queue ? group_next_point(a, g) : a.P;
        active = pt < a.P;
        if (active) split_start(L, a, pt, g);
      }
    }
  }
}

// variant 1: the exchange layout (split.cuh: XCH), FP64 and 3-dimensional
// models only; otherwise the default layout.
template <class M, class R, int INTEG>
int launch_split_mri(const AdaptiveArgs &a, int block, int variant, cudaStream_t s,
                     bool high_priority) {
  if (a.k != M::N) return kErrUnsupported;
  constexpr bool xch_ok = std::is_same<R, double>::value && M::N == 3;
  void (*kern)(AdaptiveArgs) = split_kernel<M, R, INTEG, false>;
  if constexpr (xch_ok) {
    if (variant == 1) kern = split_kernel<M, R, INTEG, true>;
  }
  unsigned grid;
  const int64_t groups_per_block = block / kSplitLanes;
  const int64_t need = (a.P + groups_per_block - 1) / groups_per_block;
  if (a.queue) {
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, block, 0);
    grid = (unsigned)std::min<int64_t>((int64_t)std::max(1, per_sm) * sms, need);
  } else {
    grid = (unsigned)need;
  }
  AdaptiveArgs ka = a;
  ka.ctl = make_ctl<R>(a);
  return (int)launch_with_priority(kern, grid, (unsigned)block, s, high_priority, ka);
}

template <class M>
int launch_split_m(int integ, int prec, const AdaptiveArgs &a, int block, int variant,
                   cudaStream_t s, bool hp) {
  if (integ == kDverk65) {
    if (prec == kFP64) return launch_split_mri<M, double, kDverk65>(a, block, variant, s, hp);
    if (prec == kFP32) return launch_split_mri<M, float, kDverk65>(a, block, variant, s, hp);
  } else if (integ == kDopri5) {
    if (prec == kFP64) return launch_split_mri<M, double, kDopri5>(a, block, variant, s, hp);
    if (prec == kFP32) return launch_split_mri<M, float, kDopri5>(a, block, variant, s, hp);
  }
  return kErrUnsupported;
}

}  // namespace adaptive

int launch_split(int model, int integ, int prec, const AdaptiveArgs &a, int block, int variant,
                 cudaStream_t s, bool hp) {
  using namespace adaptive;
  if (a.P <= 0) return 0;
  if (block <= 0 || block > kMaxLaneBlock || block % 32) block = 64;
  switch (model) {
    case kShimizu: return launch_split_m<Shimizu>(integ, prec, a, block, variant, s, hp);
    case kLorenz: return launch_split_m<Lorenz>(integ, prec, a, block, variant, s, hp);
    case kRossler: return launch_split_m<Rossler>(integ, prec, a, block, variant, s, hp);
    case kChua: return launch_split_m<Chua>(integ, prec, a, block, variant, s, hp);
    case kHyperRossler: return launch_split_m<HyperRossler>(integ, prec, a, block, variant, s, hp);
    default: return kErrUnsupported;
  }
}

}  // namespace chaos
