// C ABI of the sweep (include/chaos_lyap.h): model registry, handles,
// argument checking, launch dispatch, host-buffer path, autotuner and the
// drop-in for the reference launcher cudaLyapunov.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>

#include "../../include/chaos_lyap.h"
#include "kernels.h"
#include "models.cuh"
#include "trajectory.cuh"

namespace {

thread_local std::string g_err;

int fail(int code, const char *fmt, ...) __attribute__((format(printf, 2, 3)));
int fail(int code, const char *fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  g_err = buf;
  return code;
}

int cuda_fail(cudaError_t e, const char *what) {
  return fail(CHAOS_LYAP_ECUDA, "%s: %s", what, cudaGetErrorString(e));
}

struct ModelInfo {
  const char *name;
  int id, dim, nparams, type;
  const char *pnames, *phase, *eq;
};

// The registry the reference fills at static-initialisation time
// (model_factory.h:36-39, shimizu.dp.cpp:203-204); here the device code is
// compiled in (models.cuh) and the table only carries the descriptions.
const ModelInfo kModels[] = {
    {"chua", chaos::kChua, 3, 4, 0, "alpha, beta, m0, m1", "x, y, z",
     "x' = alpha * (y - x - f(x));y' = x - y + z;z' = - beta * y;"
     "f(x) = m1 * x + 0.5 * (m0 - m1) * (|x + 1| - |x - 1|)"},
    {"henon", chaos::kHenon, 2, 2, 1, "a, b", "x, y", "x -> 1 - a * x^2 + y;y -> b * x"},
    {"hyper_rossler", chaos::kHyperRossler, 4, 2, 0, "c, d", "x, y, z, w",
     "x' = - y - z;y' = x + 0.25 * y + w;z' = 3 + x * z;w' = - c * z + d * w"},
    {"lorenz", chaos::kLorenz, 3, 3, 0, "sigma, rho, beta", "x, y, z",
     "x' = sigma * (y - x);y' = x * (rho - z) - y;z' = x * y - beta * z"},
    {"lorenz96", chaos::kLorenz96, 40, 2, 0, "F, gamma", "x0..x39",
     "x_i' = (x_{i+1} - x_{i-2}) * x_{i-1} - gamma * x_i + F (cyclic, N = 40)"},
    {"rossler", chaos::kRossler, 3, 3, 0, "a, b, c", "x, y, z",
     "x' = - y - z;y' = x + a * y;z' = b + z * (x - c)"},
    {"shimizu", chaos::kShimizu, 3, 2, 0, "alpha, lamda", "x, y, z",
     "x' = y;y' = - alpha * y - x * z + x;z' = - lamda * z + x ** 2.0"},
};
constexpr int kModelCount = sizeof(kModels) / sizeof(kModels[0]);

const ModelInfo *find_model(const char *name) {
  if (!name) return nullptr;
  for (const auto &m : kModels)
    if (std::strcmp(m.name, name) == 0) return &m;
  return nullptr;
}

// Keeps the caller's current device across a call.
struct DeviceGuard {
  int prev = -1;
  bool ok = false;
  explicit DeviceGuard(int dev) {
    if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
    ok = (prev == dev) || cudaSetDevice(dev) == cudaSuccess;
  }
  ~DeviceGuard() {
    int cur = -1;
    if (prev >= 0 && cudaGetDevice(&cur) == cudaSuccess && cur != prev) cudaSetDevice(prev);
  }
};

chaos::View view(double *p, int64_t P, int C, int layout) {
  return layout == CHAOS_LAYOUT_COMP_MAJOR ? chaos::View{p, 1, P} : chaos::View{p, C, 1};
}
chaos::CView cview(const double *p, int64_t P, int C, int layout) {
  return layout == CHAOS_LAYOUT_COMP_MAJOR ? chaos::CView{p, 1, P} : chaos::CView{p, C, 1};
}

}  // namespace

namespace chaos {
int model_id_of(const char *name, int *dim, int *nparams) {
  const ModelInfo *m = find_model(name);
  if (!m) return -1;
  if (dim) *dim = m->dim;
  if (nparams) *nparams = m->nparams;
  return m->id;
}
}  // namespace chaos

// Memory of the two-launch sweeps (see TwoPhase): one pool per device, made with
// the device's first adaptive handle and destroyed with its last, shared by all
// of them in stream order.  It keeps at most kPoolKeepBytes between runs (the
// rest goes back at the next synchronisation).  cudaMalloc inside a new
// handle's first run took 0.5-16 ms on a shared host.
struct ResumePool {
  cudaMemPool_t pool = nullptr;
  int handles = 0;
};
constexpr uint64_t kPoolKeepBytes = 256ull << 20;
static std::mutex g_pool_mutex;
constexpr int kPoolDevices = 64;
static ResumePool g_pools[kPoolDevices];

// nullptr if the device has no memory pools: its sweeps run as one launch.
static cudaMemPool_t pool_acquire(int device) {
  if (device >= kPoolDevices) return nullptr;
  std::lock_guard<std::mutex> lock(g_pool_mutex);
  ResumePool &p = g_pools[device];
  if (!p.pool) {
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    if (cudaMemPoolCreate(&p.pool, &props) != cudaSuccess) {
      cudaGetLastError();
      p.pool = nullptr;
      return nullptr;
    }
    uint64_t keep = kPoolKeepBytes;
    int off = 0;  // another stream's block only once its work is done: sweeps on two streams overlap
    cudaMemPoolSetAttribute(p.pool, cudaMemPoolAttrReleaseThreshold, &keep);
    cudaMemPoolSetAttribute(p.pool, cudaMemPoolReuseAllowInternalDependencies, &off);
  }
  ++p.handles;
  return p.pool;
}

static void pool_release(int device) {
  std::lock_guard<std::mutex> lock(g_pool_mutex);
  ResumePool &p = g_pools[device];
  if (--p.handles > 0) return;
  cudaMemPoolDestroy(p.pool);
  p.pool = nullptr;
}

struct chaos_lyap_handle {
  chaos_lyap_desc d;
  const ModelInfo *model;
  int sm_count = 0;
  int block = 0;
  int schedule = CHAOS_SCHED_PERSISTENT;
  int variant = 0;  // kernel variant (chaos_lyap_desc.variant; autotuned)
  int32_t launches = 0;  // kernels of the last run (chaos_lyap_get_launches)
  cudaStream_t own_stream = nullptr;
  cudaStream_t last_stream = nullptr;
  unsigned long long *queue = nullptr;  // point counters: persistent sweep / batch segments
  // longest-first hand-out order of points with their own averaging times
  int32_t *order = nullptr;
  void *order_scratch = nullptr;
  int64_t order_cap = 0;
  cudaMemPool_t pool = nullptr;  // the device's ResumePool, if this handle holds it
  // further streams and fork / join events of a batch, one per segment after the
  // first
  cudaStream_t aux_stream[chaos::kMaxSegments - 1] = {};
  cudaEvent_t ev_fork = nullptr, ev_join[chaos::kMaxSegments - 1] = {};
  // host-path staging
  double *s_params = nullptr, *s_inits = nullptr, *s_spec = nullptr, *s_tavg = nullptr;
  int32_t *s_status = nullptr;
  int64_t *s_steps = nullptr;
  int64_t s_cap = 0;
};

extern "C" {

int chaos_lyap_abi_version(void) { return CHAOS_LYAP_ABI_VERSION; }

const char *chaos_lyap_last_error(void) { return g_err.c_str(); }

int chaos_lyap_desc_init(chaos_lyap_desc *d) {
  if (!d) return fail(CHAOS_LYAP_EINVAL, "desc is null");
  std::memset(d, 0, sizeof *d);
  d->struct_size = (int32_t)sizeof *d;
  std::strcpy(d->model, "lorenz");
  d->method = CHAOS_METHOD_VAR;
  d->integrator = CHAOS_INTEG_DVERK65;
  d->precision = CHAOS_PREC_FP64;
  d->gs = CHAOS_GS_CLASSICAL;
  d->layout = CHAOS_LAYOUT_POINT_MAJOR;
  d->eps = 1e-7;
  d->h = 1e-3;
  d->rtol = d->atol = 1e-10;
  d->max_steps = 100000000LL;
  d->escape = 1e4;
  d->schedule = CHAOS_SCHED_AUTO;
  return CHAOS_LYAP_OK;
}

int chaos_lyap_model_count(void) { return kModelCount; }

int chaos_lyap_model_name(int index, char *buf, int buflen) {
  if (index < 0 || index >= kModelCount || !buf || buflen <= 0)
    return fail(CHAOS_LYAP_EINVAL, "model index %d out of range", index);
  std::snprintf(buf, (size_t)buflen, "%s", kModels[index].name);
  return CHAOS_LYAP_OK;
}

int chaos_lyap_query_model(const char *name, int32_t *dim, int32_t *nparams, int32_t *type) {
  const ModelInfo *m = find_model(name);
  if (!m) return fail(CHAOS_LYAP_ENOMODEL, "unknown model '%s'", name ? name : "(null)");
  if (dim) *dim = m->dim;
  if (nparams) *nparams = m->nparams;
  if (type) *type = m->type;
  return CHAOS_LYAP_OK;
}

int chaos_lyap_model_text(const char *name, int which, char *buf, int buflen) {
  const ModelInfo *m = find_model(name);
  if (!m) return fail(CHAOS_LYAP_ENOMODEL, "unknown model '%s'", name ? name : "(null)");
  if (!buf || buflen <= 0 || which < 0 || which > 2) return fail(CHAOS_LYAP_EINVAL, "bad buffer");
  const char *s = which == 0 ? m->pnames : which == 1 ? m->phase : m->eq;
  std::snprintf(buf, (size_t)buflen, "%s", s);
  return (int)std::strlen(s) < buflen ? CHAOS_LYAP_OK
                                      : fail(CHAOS_LYAP_EINVAL, "buffer too small");
}

}  // extern "C"

namespace chaos {
static int msg_fail(char *msg, size_t len, int code, const char *fmt, ...)
    __attribute__((format(printf, 4, 5)));
static int msg_fail(char *msg, size_t len, int code, const char *fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(msg, len, fmt, ap);
  va_end(ap);
  return code;
}

// Descriptor validation shared by the handle path (chaos_lyap_create) and
// the no-allocation batch entry: CHAOS_LYAP_OK, or an error code with the
// reason in msg.  k must already be resolved (k == 0 means "dim" only at
// create time).
int validate_desc(const chaos_lyap_desc *d, char *msg, size_t len) {
  if (!d) return msg_fail(msg, len, CHAOS_LYAP_EINVAL, "desc is null");
  if (d->struct_size != (int32_t)sizeof(chaos_lyap_desc))
    return msg_fail(msg, len, CHAOS_LYAP_EINVAL, "desc.struct_size %d != %d", d->struct_size,
                (int)sizeof(chaos_lyap_desc));
  char name[33];
  std::memcpy(name, d->model, 32);
  name[32] = 0;
  const ModelInfo *m = find_model(name);
  if (!m) return msg_fail(msg, len, CHAOS_LYAP_ENOMODEL, "unknown model '%s'", name);
  if (d->k < 1 || d->k > m->dim)
    return msg_fail(msg, len, CHAOS_LYAP_EINVAL,
        "k = %d outside 1..%d for model %s", d->k, m->dim, m->name);
  if (d->layout != CHAOS_LAYOUT_POINT_MAJOR && d->layout != CHAOS_LAYOUT_COMP_MAJOR)
    return msg_fail(msg, len, CHAOS_LYAP_EINVAL, "bad layout %d", d->layout);
  if (d->method < CHAOS_METHOD_FD || d->method > CHAOS_METHOD_QR)
    return msg_fail(msg, len, CHAOS_LYAP_EINVAL, "bad method %d", d->method);
  if (!(d->h > 0) || !std::isfinite(d->h)) return msg_fail(msg, len, CHAOS_LYAP_EINVAL,
      "h must be > 0");
  if (d->precision == CHAOS_PREC_COMPAT_FP64) {
    if (d->integrator != CHAOS_INTEG_DVERK_FIXED)
      return msg_fail(msg, len, CHAOS_LYAP_EINVAL,
          "compat precision needs the fixed-step DVERK integrator");
    if (d->method == CHAOS_METHOD_QR && d->k != m->dim)
      return msg_fail(msg, len, CHAOS_LYAP_EUNSUPPORTED,
                  "QR method needs k == dim (the reference's QR assumes a square matrix)");
    if (!(d->t_avg > 0)) return msg_fail(msg, len, CHAOS_LYAP_EINVAL, "t_avg must be > 0");
  } else if (d->precision == CHAOS_PREC_FP64 || d->precision == CHAOS_PREC_FP32) {
    if (d->integrator != CHAOS_INTEG_DVERK65 && d->integrator != CHAOS_INTEG_DOPRI5)
      return msg_fail(msg, len, CHAOS_LYAP_EINVAL,
          "adaptive precision forms need DVERK65 or DOPRI5");
    if (d->method != CHAOS_METHOD_VAR)
      return msg_fail(msg, len, CHAOS_LYAP_EUNSUPPORTED,
          "adaptive forms integrate the variational equations (VAR)");
    if (d->k != m->dim && m->dim <= 4)
      return msg_fail(msg, len, CHAOS_LYAP_EUNSUPPORTED,
          "adaptive forms compute the full spectrum (k == dim)");
    if (!(d->rtol > 0) || !(d->atol > 0)) return msg_fail(msg, len, CHAOS_LYAP_EINVAL,
        "rtol/atol must be > 0");
    if (!(d->dt_renorm > 0) || !(d->t_avg > 0) || d->t_transient < 0 || d->t_align < 0)
      return msg_fail(msg, len, CHAOS_LYAP_EINVAL,
          "times: dt_renorm, t_avg > 0; t_transient, t_align >= 0");
    if (d->max_steps <= 0) return msg_fail(msg, len, CHAOS_LYAP_EINVAL, "max_steps must be > 0");
    if (d->gs != CHAOS_GS_CLASSICAL && d->gs != CHAOS_GS_MODIFIED)
      return msg_fail(msg, len, CHAOS_LYAP_EINVAL, "bad gs %d", d->gs);
  } else {
    return msg_fail(msg, len, CHAOS_LYAP_EINVAL, "bad precision %d", d->precision);
  }
  if (m->type != 0) {  // maps: the reference's FD / VAR map branches, in compat precision
    if (d->precision != CHAOS_PREC_COMPAT_FP64)
      return msg_fail(msg, len, CHAOS_LYAP_EUNSUPPORTED,
                  "map model %s: maps are iterated, not integrated; use compat precision", m->name);
    if (d->method == CHAOS_METHOD_QR)
      return msg_fail(msg, len, CHAOS_LYAP_EUNSUPPORTED,
          "map model %s: the QR method has no map branch",
                  m->name);
  }
  return CHAOS_LYAP_OK;
}
}  // namespace chaos

static int check_desc(const chaos_lyap_desc *d, const ModelInfo **mout) {
  char msg[512];
  const int rc = chaos::validate_desc(d, msg, sizeof msg);
  if (rc) return fail(rc, "%s", msg);
  char name[33];
  std::memcpy(name, d->model, 32);
  name[32] = 0;
  *mout = find_model(name);
  return CHAOS_LYAP_OK;
}

extern "C" {

int chaos_lyap_create(const chaos_lyap_desc *desc, chaos_lyap_handle **out) {
  if (!out) return fail(CHAOS_LYAP_EINVAL, "out is null");
  *out = nullptr;
  chaos_lyap_desc d;
  if (!desc) return fail(CHAOS_LYAP_EINVAL, "desc is null");
  d = *desc;
  const ModelInfo *m0 = find_model(d.model);
  if (d.k == 0 && m0) d.k = m0->dim;
  const ModelInfo *m = nullptr;
  int rc = check_desc(&d, &m);
  if (rc) return rc;
  int ndev = 0;
  cudaError_t e = cudaGetDeviceCount(&ndev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetDeviceCount");
  if (d.device < 0 || d.device >= ndev)
    return fail(CHAOS_LYAP_EINVAL, "device %d not present (%d devices)", d.device, ndev);
  DeviceGuard g(d.device);
  if (!g.ok) return fail(CHAOS_LYAP_ECUDA, "cannot select device %d", d.device);
  auto *h = new chaos_lyap_handle();
  h->d = d;
  h->model = m;
  cudaDeviceGetAttribute(&h->sm_count, cudaDevAttrMultiProcessorCount, d.device);
  h->block = d.block > 0 ? d.block : (d.precision == CHAOS_PREC_COMPAT_FP64 ? 64 : 128);
  h->schedule = (d.schedule >= CHAOS_SCHED_DIRECT && d.schedule <= CHAOS_SCHED_SPLIT_PERSISTENT)
                    ? d.schedule
                    : CHAOS_SCHED_PERSISTENT;
  h->variant = d.variant == 1 ? 1 : 0;
  if ((e = cudaStreamCreateWithFlags(&h->own_stream, cudaStreamNonBlocking)) != cudaSuccess) {
    delete h;
    return cuda_fail(e, "cudaStreamCreate");
  }
  if ((e = cudaMalloc(&h->queue, sizeof(unsigned long long) * chaos::kMaxSegments)) != cudaSuccess) {
    cudaStreamDestroy(h->own_stream);
    delete h;
    return fail(CHAOS_LYAP_ENOMEM, "cudaMalloc(queue): %s", cudaGetErrorString(e));
  }
  if (d.precision != CHAOS_PREC_COMPAT_FP64) h->pool = pool_acquire(d.device);
  *out = h;
  return CHAOS_LYAP_OK;
}

static void free_staging(chaos_lyap_handle *h) {
  cudaFree(h->s_params);
  cudaFree(h->s_inits);
  cudaFree(h->s_spec);
  cudaFree(h->s_tavg);
  cudaFree(h->s_status);
  cudaFree(h->s_steps);
  h->s_params = h->s_inits = h->s_spec = h->s_tavg = nullptr;
  h->s_status = nullptr;
  h->s_steps = nullptr;
  h->s_cap = 0;
}

int chaos_lyap_destroy(chaos_lyap_handle *h) {
  if (!h) return CHAOS_LYAP_OK;
  DeviceGuard g(h->d.device);
  cudaStreamSynchronize(h->own_stream);
  free_staging(h);
  cudaFree(h->queue);
  cudaFree(h->order);
  cudaFree(h->order_scratch);
  if (h->pool) pool_release(h->d.device);
  for (cudaStream_t s : h->aux_stream)
    if (s) {
      cudaStreamSynchronize(s);
      cudaStreamDestroy(s);
    }
  if (h->ev_fork) cudaEventDestroy(h->ev_fork);
  for (cudaEvent_t e : h->ev_join)
    if (e) cudaEventDestroy(e);
  cudaStreamDestroy(h->own_stream);
  delete h;
  return CHAOS_LYAP_OK;
}

// Device buffers for the longest-first order of P points (grown on demand;
// allocated outside any stream capture: before a run or a graph capture).
static int ensure_order(chaos_lyap_handle *h, int64_t P) {
  if (P <= h->order_cap) return CHAOS_LYAP_OK;
  DeviceGuard g(h->d.device);
  cudaFree(h->order);
  h->order = nullptr;
  h->order_cap = 0;
  cudaError_t e = cudaMalloc(&h->order, sizeof(int32_t) * P);
  if (e == cudaSuccess && !h->order_scratch) e = cudaMalloc(&h->order_scratch, chaos::kOrderScratchBytes);
  if (e != cudaSuccess) {
    cudaFree(h->order);
    h->order = nullptr;
    return fail(CHAOS_LYAP_ENOMEM, "cudaMalloc(order): %s", cudaGetErrorString(e));
  }
  h->order_cap = P;
  return CHAOS_LYAP_OK;
}

// A persistent sweep (one lane or one warp per point) runs as two launches -- all
// transients, then the averaging phases, those expected to take longest first --
// when its points are more than the GPU holds at once (otherwise every point starts
// at once and the order cannot matter).  Needs a transient, which is what predicts
// the cost, of any length: t_transient / t_avg 0.1 to 60, points in the map's order
// or shuffled, 1.55 to 31 waves: 0.99 (hyper-Rossler, 0.1, which gains nothing) to
// 2.7 times as fast as one launch, the longer the transient the more.  The buffers
// take 48-92 bytes per point (Lorenz-96: 344-668).  One launch -> two, B200: 256^2
// Lorenz points in FP64 (1.7 waves) 245 -> 195 ms; FP32 Lorenz, 152k points (2 waves)
// 62 -> 47 ms, 300k 103 -> 85 ms, 1024^2 (14 waves) 309 -> 279 ms; FP32 Rossler, whose
// longest points take twice the mean, 152k points 82 -> 77 ms.
//
// From 1.5 waves on, because a lane renormalises with its warp, so that results
// move with the grouping of the points, by less than the method's own error but
// far on chaotic cells.  Just above one wave nearly every warp of a one-launch
// sweep holds the same points in every run and the results repeat; two launches
// would group all of them anew (FP32 Rossler, 1.1 waves: 55 -> 52 ms, and four times
// the difference of two runs of one launch).  At 1.55 waves that is 1.26 times (root
// mean square 0.044 against 0.035), with the same errors against the exact exponents
// (tests/test_gpu_two_phase_models.py).
constexpr double kTwoPhaseMinWaves = 1.5;
// The warp-per-point form renormalises each point by itself, so its results do
// not depend on the order at all: from the first point that has to wait.
// Lorenz-96, 64^2 points (1.7 waves): 116 -> 94 ms.
constexpr double kTwoPhaseMinWavesWarp = 1.0;
// Up to here the buffers stay below 120 MB, within what the pool keeps; the gain of
// a short transient is down to 1.06 (FP32) and 1.03 (FP64) at 31 waves.
constexpr int64_t kTwoPhaseMaxWaves = 32;

// Buffers of one two-launch sweep of P points, from the pool and back to it in
// the order of stream s.  Empty (the sweep runs as one launch) during a stream
// capture, where the allocation would be the graph's, and when memory is short.
struct TwoPhase {
  // An allocation from the pool is refused, and ends the capture, while a capture
  // of another stream is open (this thread's, or a global one of any thread's),
  // unless the calling thread's mode is relaxed.  Nothing below depends on what a
  // capture of another stream records, so it is.  (Restored last: the block goes
  // back to the pool under it.)
  struct Relaxed {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
  } relaxed;
  char *base = nullptr;
  cudaStream_t s;
  void *scratch = nullptr;
  int32_t *order = nullptr;
  chaos::Resume resume{};
  TwoPhase(const chaos_lyap_handle *h, int prec, int64_t P, cudaStream_t stream) : s(stream) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (!h->pool || cudaStreamIsCapturing(s, &cap) != cudaSuccess ||
        cap != cudaStreamCaptureStatusNone) {
      cudaGetLastError();
      return;
    }
    const size_t head = (chaos::kOrderScratchBytes + 255) / 256 * 256;
    const size_t state = (size_t)chaos::resume_state_bytes(h->model->dim, prec) * P;
    void *b = nullptr;
    if (cudaMallocFromPoolAsync(&b, head + 16 * P + state + sizeof(int32_t) * P, h->pool, s) !=
        cudaSuccess) {
      cudaGetLastError();
      return;
    }
    base = static_cast<char *>(b);
    scratch = base;
    resume.cost = reinterpret_cast<double *>(base + head);
    resume.steps = reinterpret_cast<int64_t *>(resume.cost + P);
    resume.state = resume.steps + P;
    order = reinterpret_cast<int32_t *>(base + head + 16 * P + state);
  }
  ~TwoPhase() {
    if (base) cudaFreeAsync(base, s);
  }
  TwoPhase(const TwoPhase &) = delete;
  TwoPhase &operator=(const TwoPhase &) = delete;
};

// P points of params / inits are read at every `stride`-th point of arrays
// that hold P_full points (stride 1, P_full = 0: the arrays themselves); the
// spectrum, status and steps arrays hold P points.
static int enqueue(chaos_lyap_handle *h, int64_t P, const double *params, double *inits,
                   double *spectrum, int32_t *status, int64_t *steps, const double *tavg,
                   cudaStream_t s, int block, int schedule, int variant, double t_avg_override,
                   double t_transient_override, int64_t P_full = 0, int64_t stride = 1) {
  const chaos_lyap_desc &d = h->d;
  const ModelInfo *m = h->model;
  int rc, launches = 1;
  if (d.precision == CHAOS_PREC_COMPAT_FP64) {
    chaos::CompatArgs a{};
    a.P = P;
    a.k = d.k;
    a.method = d.method;
    a.eps = d.eps;
    a.step = d.h;
    a.t_skip = d.t_transient;
    a.t_skip_clp = d.t_align;
    a.calc_time = d.t_avg;
    a.add_skip = d.dt_renorm / d.h;  // tasklyapunov.cpp:65
    a.params = cview(params, P, m->nparams, d.layout);
    a.inits = view(inits, P, m->dim, d.layout);
    a.close = nullptr;
    a.lyap = view(spectrum, P, d.k, d.layout);
    a.accumulate = 0;
    a.status = status;
    rc = chaos::launch_compat(m->id, a, block, s);
  } else {
    chaos::AdaptiveArgs a{};
    a.P = P;
    a.k = d.k;
    a.gs = d.gs;
    a.rtol = d.rtol;
    a.atol = d.atol;
    a.h0 = d.h;
    a.hmax = d.h_max;
    a.hmin = d.h_min;
    a.t_transient = t_transient_override >= 0 ? t_transient_override : d.t_transient;
    a.t_align = d.t_align;
    a.t_avg = t_avg_override > 0 ? t_avg_override : d.t_avg;
    a.dt_renorm = d.dt_renorm;
    a.max_steps = d.max_steps;
    a.escape = d.escape > 0 ? d.escape : 1e4;
    a.params = cview(params, P_full > 0 ? P_full : P, m->nparams, d.layout);
    a.inits = cview(inits, P_full > 0 ? P_full : P, m->dim, d.layout);
    a.params.ps *= stride;
    a.inits.ps *= stride;
    a.t_avg_per_point = t_avg_override > 0 ? nullptr : tavg;
    a.spectrum = view(spectrum, P, d.k, d.layout);
    a.status = status;
    a.steps = steps;
    const int integ = d.integrator == CHAOS_INTEG_DOPRI5 ? chaos::kDopri5 : chaos::kDverk65;
    const int prec = d.precision == CHAOS_PREC_FP32 ? chaos::kFP32 : chaos::kFP64;
    const bool split = schedule == CHAOS_SCHED_SPLIT_DIRECT || schedule == CHAOS_SCHED_SPLIT_PERSISTENT;
    if (schedule == CHAOS_SCHED_PERSISTENT || schedule == CHAOS_SCHED_SPLIT_PERSISTENT) {
      cudaError_t e = cudaMemsetAsync(h->queue, 0, sizeof(unsigned long long), s);
      if (e != cudaSuccess) return cuda_fail(e, "cudaMemsetAsync(queue)");
      a.queue = h->queue;
      a.queue_stride = chaos::queue_stride_for(P);
      const bool warp = m->dim > 4;
      // (also where this run takes two launches: a capture of the same call takes one
      // and cannot allocate)
      if (a.t_avg_per_point && !warp && (rc = ensure_order(h, P))) return rc;
      if (!split && a.t_transient > 0) {
        const int64_t held = warp ? chaos::l96_resident(integ, prec, d.k)
                                  : chaos::adaptive_resident(m->id, integ, prec, block, variant);
        const double least = warp ? kTwoPhaseMinWavesWarp : kTwoPhaseMinWaves;
        if (held > 0 && P > (int64_t)(least * held) && P <= kTwoPhaseMaxWaves * held) {
          TwoPhase t(h, prec, P, s);
          if (t.base) {
            a.order = t.order;
            a.resume = t.resume;
            rc = warp ? chaos::launch_l96_two_phase(integ, prec, a, t.scratch, s)
                      : chaos::launch_adaptive_two_phase(m->id, integ, prec, a, block, variant,
                                                         t.scratch, s);
            if (rc && rc != chaos::kErrUnsupported)
              return cuda_fail((cudaError_t)rc, "kernel launch");
            if (!rc) {
              h->last_stream = s;
              h->launches = 2 + chaos::kOrderKernels;
              return CHAOS_LYAP_OK;
            }
            a.resume = chaos::Resume{};
            a.order = nullptr;
          }
        }
      }
      if (a.t_avg_per_point && !warp) {  // longest averaging time first
        rc = chaos::launch_order_longest_first(a.t_avg_per_point, P, h->order, h->order_scratch, s);
        if (rc) return cuda_fail((cudaError_t)rc, "order launch");
        a.order = h->order;
        launches += chaos::kOrderKernels;
      }
    }
    if (m->dim > 4) rc = chaos::launch_l96_warp(integ, prec, a, 0, s);
    else if (split) rc = chaos::launch_split(m->id, integ, prec, a, block, variant, s);
    else rc = chaos::launch_adaptive(m->id, integ, prec, a, block, variant, s);
  }
  if (rc == chaos::kErrUnsupported)
    return fail(CHAOS_LYAP_EUNSUPPORTED, "no kernel for model %s with this integrator/precision/k",
                m->name);
  if (rc != 0) return cuda_fail((cudaError_t)rc, "kernel launch");
  h->last_stream = s;
  h->launches = launches;
  return CHAOS_LYAP_OK;
}

int chaos_lyap_run(chaos_lyap_handle *h, int64_t P, const double *params, double *inits,
                   double *spectrum, int32_t *status, int64_t *steps, const double *tavg,
                   void *stream) {
  if (!h) return fail(CHAOS_LYAP_EINVAL, "handle is null");
  if (P < 0) return fail(CHAOS_LYAP_EINVAL, "P < 0");
  if (P == 0) return CHAOS_LYAP_OK;
  if (!params || !inits || !spectrum) return fail(CHAOS_LYAP_EINVAL, "null array");
  DeviceGuard g(h->d.device);
  if (!g.ok) return fail(CHAOS_LYAP_ECUDA, "cannot select device %d", h->d.device);
  return enqueue(h, P, params, inits, spectrum, status, steps, tavg, (cudaStream_t)stream, h->block,
                 h->schedule, h->variant, -1.0, -1.0);
}

int chaos_lyap_sync(chaos_lyap_handle *h) {
  if (!h) return fail(CHAOS_LYAP_EINVAL, "handle is null");
  DeviceGuard g(h->d.device);
  cudaError_t e = h->last_stream ? cudaStreamSynchronize(h->last_stream) : cudaDeviceSynchronize();
  if (e != cudaSuccess) return cuda_fail(e, "synchronize");
  e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "sweep");
  return CHAOS_LYAP_OK;
}

int chaos_lyap_run_host(chaos_lyap_handle *h, int64_t P, const double *params, double *inits,
                        double *spectrum, int32_t *status, int64_t *steps, const double *tavg) {
  if (!h) return fail(CHAOS_LYAP_EINVAL, "handle is null");
  if (P < 0) return fail(CHAOS_LYAP_EINVAL, "P < 0");
  if (P == 0) return CHAOS_LYAP_OK;
  if (!params || !inits || !spectrum) return fail(CHAOS_LYAP_EINVAL, "null array");
  DeviceGuard g(h->d.device);
  if (!g.ok) return fail(CHAOS_LYAP_ECUDA, "cannot select device %d", h->d.device);
  const ModelInfo *m = h->model;
  const int k = h->d.k;
  cudaError_t e;
  if (P > h->s_cap) {
    free_staging(h);
    if ((e = cudaMalloc(&h->s_params, sizeof(double) * P * m->nparams)) != cudaSuccess ||
        (e = cudaMalloc(&h->s_inits, sizeof(double) * P * m->dim)) != cudaSuccess ||
        (e = cudaMalloc(&h->s_spec, sizeof(double) * P * k)) != cudaSuccess ||
        (e = cudaMalloc(&h->s_tavg, sizeof(double) * P)) != cudaSuccess ||
        (e = cudaMalloc(&h->s_status, sizeof(int32_t) * P)) != cudaSuccess ||
        (e = cudaMalloc(&h->s_steps, sizeof(int64_t) * P)) != cudaSuccess) {
      free_staging(h);
      return fail(CHAOS_LYAP_ENOMEM, "staging for %lld points: %s", (long long)P,
                  cudaGetErrorString(e));
    }
    h->s_cap = P;
  }
  cudaStream_t s = h->own_stream;
  const size_t bp = sizeof(double) * P * m->nparams, bx = sizeof(double) * P * m->dim,
               bs = sizeof(double) * P * k;
  if ((e = cudaMemcpyAsync(h->s_params, params, bp, cudaMemcpyHostToDevice, s)) != cudaSuccess ||
      (e = cudaMemcpyAsync(h->s_inits, inits, bx, cudaMemcpyHostToDevice, s)) != cudaSuccess)
    return cuda_fail(e, "copy in");
  if (tavg && (e = cudaMemcpyAsync(h->s_tavg, tavg, sizeof(double) * P, cudaMemcpyHostToDevice,
                                   s)) != cudaSuccess)
    return cuda_fail(e, "copy in");
  int rc = enqueue(h, P, h->s_params, h->s_inits, h->s_spec, status ? h->s_status : nullptr,
                   steps ? h->s_steps : nullptr, tavg ? h->s_tavg : nullptr, s, h->block,
                   h->schedule, h->variant, -1.0, -1.0);
  if (rc) return rc;
  if ((e = cudaMemcpyAsync(spectrum, h->s_spec, bs, cudaMemcpyDeviceToHost, s)) != cudaSuccess)
    return cuda_fail(e, "copy out");
  if (h->d.precision == CHAOS_PREC_COMPAT_FP64 &&
      (e = cudaMemcpyAsync(inits, h->s_inits, bx, cudaMemcpyDeviceToHost, s)) != cudaSuccess)
    return cuda_fail(e, "copy out");
  if (status && (e = cudaMemcpyAsync(status, h->s_status, sizeof(int32_t) * P,
                                     cudaMemcpyDeviceToHost, s)) != cudaSuccess)
    return cuda_fail(e, "copy out");
  if (steps && (e = cudaMemcpyAsync(steps, h->s_steps, sizeof(int64_t) * P,
                                    cudaMemcpyDeviceToHost, s)) != cudaSuccess)
    return cuda_fail(e, "copy out");
  if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return cuda_fail(e, "synchronize");
  return CHAOS_LYAP_OK;
}

// Times short runs of `sample` points -- every `stride`-th of the P_full
// points of the arrays -- in every launch shape and keeps the fastest.
static int autotune(chaos_lyap_handle *h, int64_t P_full, int64_t sample, int64_t stride,
                    const double *params, const double *inits, int32_t *block_out,
                    int32_t *schedule_out) {
  if (!h) return fail(CHAOS_LYAP_EINVAL, "handle is null");
  if (sample <= 0 || !params || !inits) return fail(CHAOS_LYAP_EINVAL, "bad sample");
  if (h->d.precision == CHAOS_PREC_COMPAT_FP64 || h->model->dim > 4) {
    if (block_out) *block_out = h->block;
    if (schedule_out) *schedule_out = h->schedule;
    return CHAOS_LYAP_OK;
  }
  DeviceGuard g(h->d.device);
  const int k = h->d.k;
  double *spec = nullptr;
  cudaError_t e;
  if ((e = cudaMalloc(&spec, sizeof(double) * sample * k)) != cudaSuccess)
    return fail(CHAOS_LYAP_ENOMEM, "autotune buffer: %s", cudaGetErrorString(e));
  // Short horizons: the launch-shape ranking does not need the full run.
  // Stage 1 times every shape on a horizon of 20 renormalisation intervals;
  // stage 2 re-times the shapes within 15 % of the fastest on a horizon four
  // times longer, where the few points whose chains set a small map's
  // length weigh as they do in the full run (on a 64^2 map the short
  // horizon alone ranked two split layouts 10 % apart the wrong way round).
  const double t_avg1 = std::min(h->d.t_avg, 20.0 * h->d.dt_renorm);
  const double t_tr1 = std::min(h->d.t_transient, 5.0 * h->d.dt_renorm);
  const double t_avg2 = std::min(h->d.t_avg, 80.0 * h->d.dt_renorm);
  const double t_tr2 = std::min(h->d.t_transient, 20.0 * h->d.dt_renorm);
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  const int blocks[] = {64, 128};
  const int scheds[] = {CHAOS_SCHED_DIRECT, CHAOS_SCHED_PERSISTENT, CHAOS_SCHED_SPLIT_DIRECT,
                        CHAOS_SCHED_SPLIT_PERSISTENT};
  const bool fp32 = h->d.precision == CHAOS_PREC_FP32;
  struct Shape {
    int b, sc, v;
    float ms;
  };
  Shape shapes[16];
  int n = 0, rc = CHAOS_LYAP_OK;
  cudaStream_t s = h->own_stream;
  auto time_shape = [&](Shape &x, double t_avg, double t_tr) {
    for (int rep = 0; rep < 2 && rc == CHAOS_LYAP_OK; ++rep) {
      cudaEventRecord(e0, s);
      rc = enqueue(h, sample, params, const_cast<double *>(inits), spec, nullptr, nullptr,
                   nullptr, s, x.b, x.sc, x.v, t_avg, t_tr, P_full, stride);
      cudaEventRecord(e1, s);
      cudaEventSynchronize(e1);
      cudaEventElapsedTime(&x.ms, e0, e1);  // second repetition is the warm one
    }
  };
  for (int v = 0; v < 2 && rc == CHAOS_LYAP_OK; v++)
    for (int b : blocks)
      for (int sc : scheds) {
        // variant 1: the register cap of the FP32 one-lane forms, the
        // exchange layout of the FP64 split forms of 3-dimensional models
        const bool split = sc == CHAOS_SCHED_SPLIT_DIRECT || sc == CHAOS_SCHED_SPLIT_PERSISTENT;
        if (v > 0 && (split ? (fp32 || h->model->dim != 3) : !fp32)) continue;
        if (rc != CHAOS_LYAP_OK || n >= 16) break;
        shapes[n] = Shape{b, sc, v, 0.f};
        time_shape(shapes[n], t_avg1, t_tr1);
        ++n;
      }
  float best1 = 1e30f;
  for (int i = 0; i < n; i++) best1 = std::min(best1, shapes[i].ms);
  Shape best{h->block, h->schedule, h->variant, 1e30f};
  const bool longer = t_avg2 > t_avg1 || t_tr2 > t_tr1;
  for (int i = 0; i < n && rc == CHAOS_LYAP_OK; i++) {
    Shape x = shapes[i];
    if (x.ms > 1.15f * best1) continue;
    if (longer) time_shape(x, t_avg2, t_tr2);
    if (rc == CHAOS_LYAP_OK && x.ms < best.ms) best = x;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(spec);
  if (rc) return rc;
  const int best_b = best.b, best_s = best.sc, best_v = best.v;
  h->block = best_b;
  h->schedule = best_s;
  h->variant = best_v;
  if (block_out) *block_out = best_b;
  if (schedule_out) *schedule_out = best_s;
  return CHAOS_LYAP_OK;
}

int chaos_lyap_autotune(chaos_lyap_handle *h, int64_t sample, const double *params,
                        const double *inits, int32_t *block_out, int32_t *schedule_out) {
  return autotune(h, sample, sample, 1, params, inits, block_out, schedule_out);
}

int chaos_lyap_autotune_map(chaos_lyap_handle *h, int64_t P, int64_t sample,
                            const double *params, const double *inits, int32_t *block_out,
                            int32_t *schedule_out) {
  if (P <= 0 || sample <= 0) return fail(CHAOS_LYAP_EINVAL, "P and sample must be > 0");
  const int64_t n = std::min(P, sample);
  return autotune(h, P, n, P / n, params, inits, block_out, schedule_out);
}

// A batch runs each segment in the form of its handle's schedule, one persistent
// launch per segment, side by side: forked onto the first handle's further
// streams, joined before the batch ends (branches of one graph when captured).
// Each launch is its model's own sweep kernel, and where the segments fit beside
// one another they share the SMs from the start.  Segments with a split
// schedule -- the form chosen for segments whose longest points set the run's
// length -- are launched first and at the device's greatest priority; the others'
// blocks take the slots that are left or that theirs free as their queues run
// dry.  (One kernel per form that moved its warps from segment to segment, with
// the registers of the largest model, ran the two forms one after the other and
// each model slower.)
//
// An FP32 batch of few waves whose points have averaging times of their own is as
// long as its longest points' chains of steps, and a step takes longer the more
// warps share its scheduler: its one-lane segments run in the build of up to 168
// registers, three blocks per SM instead of four for the models that use more than
// 128 (hyper-Rossler 164, Shimizu 143, Lorenz 137; Rossler and Chua still fit four
// times).  Averaging times T to 4 T, one kernel for all / 128 registers / 168:
// 65,536 hyper-Rossler and as many Lorenz points 307 / 371 / 305 ms, with as many
// Chua points 383 / 391 / 298 ms; 150,000 Lorenz points (2 waves) 8.0 / 6.8 / 6.8 ms.
// From kBatchFewWaves waves on throughput counts: 300,000 Lorenz points (4 waves)
// 15.2 / 12.3 / 12.9 ms.  Segments that lie apart gain nothing: 19,891 Lorenz and as
// many Rossler points (0.5 waves) 4.1 / 3.0-3.3 / 3.3 ms, eight segments of 4,096
// 3.6 / 1.4 / 1.5 ms; beside a split segment they meet sooner (3 x 128^2 points, 0.4
// waves of them: 36.1 / 27.6 / 26.4 ms).
constexpr double kBatchFewWaves = 3.0, kBatchApartWaves = 0.6, kBatchApartWavesSplit = 0.25;
// Such a batch of one segment takes two blocks per SM while its points come out
// even over them, up to kBatchSoloPoints.  One kernel / 128 registers / 168 / two
// blocks: hyper-Rossler, 39,782 points 252 / 278 / 294 / 223 ms, 65,546 points 280 /
// 384 / 297 / 221, 77,670 points 291 / 387 / 299 / 227; Lorenz, 39,782 points 3.5 / 4.0 /
// 3.9 / 3.0, 77,670 points 4.6 / 5.2 / 4.1 / 4.1, 100,000 points 5.6 / 5.4 / 4.7 / 5.2 ms.
constexpr int kBatchSoloLanes = 256, kBatchSoloPoints = 576;  // per SM
// Among the one-lane segments those of fewer points are launched first: they
// start whole beside a part of the larger ones, whose other points follow as
// lanes become free.  If they do not all fit, the orders are made before the
// fork, so that the sweep kernels themselves start in that order: 120,000 Lorenz
// and 3,000 hyper-Rossler points, either way round, 42 ms as one kernel, 27 ms
// this way, 35 ms with the Lorenz points first; 20,000 points each of three
// models and 5,000 of a fourth 51 ms, 27 ms, and 28-45 ms where the order was
// left to the streams.
struct BatchPlan {
  int nseg;
  // the segments in launch order: split ones first
  struct Part {
    chaos::AdaptiveArgs a;
    chaos_lyap_handle *h;
    void *scratch;  // of the longest-first ordering, with per-point times
    bool split;
  } part[chaos::kMaxSegments];
  int integ, prec;
  bool few_waves;    // FP32: kBatchVariant for one-lane segments of uneven points
  bool solo;         // FP32, one such segment: kBatchSoloLanes
  bool order_first;  // all hand-out orders before the fork
};

static int part_variant(const BatchPlan &p, const BatchPlan::Part &q) {
  return p.few_waves && q.a.order ? chaos::kBatchVariant : q.h->variant;
}

// Points of the one-lane segments in waves of the points the GPU holds (FP32: of
// kBatchVariant, or of the handles' builds).
static double lane_waves(const BatchPlan &p, bool batch_build) {
  double waves = 0;
  for (int i = 0; i < p.nseg; i++) {
    const BatchPlan::Part &q = p.part[i];
    if (q.split) continue;
    const int64_t held =
        chaos::adaptive_resident(q.h->model->id, p.integ, p.prec, q.h->block,
                                 batch_build ? chaos::kBatchVariant : q.h->variant);
    waves += (double)q.a.P / (double)std::max<int64_t>(1, held);
  }
  return waves;
}

// Device buffers of one segment's longest-first hand-out order.
struct OrderBuf {
  int32_t *order;
  void *scratch;
};

static bool is_split(const chaos_lyap_handle *h) {
  return h->schedule == CHAOS_SCHED_SPLIT_DIRECT || h->schedule == CHAOS_SCHED_SPLIT_PERSISTENT;
}

// Checks the segments and lays out the launch.  Each segment's longest-first
// order goes into `own[i]` when given (buffers a graph owns, sized for the
// segment), else into the segment handle's own buffers (grown on demand).
// Every segment has its own handle: two segments of one handle would share
// that handle's order buffer.
static int check_segments(const chaos_lyap_segment *segs, int nseg) {
  if (!segs || nseg <= 0 || nseg > chaos::kMaxSegments)
    return fail(CHAOS_LYAP_EINVAL, "nseg must be 1..%d", chaos::kMaxSegments);
  for (int i = 0; i < nseg; i++) {
    if (!segs[i].handle) return fail(CHAOS_LYAP_EINVAL, "segment %d: null handle", i);
    for (int j = 0; j < i; j++)
      if (segs[j].handle == segs[i].handle)
        return fail(CHAOS_LYAP_EINVAL,
                    "segments %d and %d share a handle: every segment needs its own", j, i);
  }
  return CHAOS_LYAP_OK;
}

static int build_batch(const chaos_lyap_segment *segs, int nseg, BatchPlan *plan,
                       const OrderBuf *own) {
  int rc0 = check_segments(segs, nseg);
  if (rc0) return rc0;
  std::memset(plan, 0, sizeof *plan);
  plan->nseg = nseg;
  int nsplit = 0, next_split = 0;
  for (int i = 0; i < nseg; i++) nsplit += is_split(segs[i].handle);
  int next_lane = nsplit;
  chaos_lyap_handle *h0 = segs[0].handle;
  for (int i = 0; i < nseg; i++) {
    const chaos_lyap_segment &sg = segs[i];
    const chaos_lyap_desc &d = sg.handle->d;
    if (d.precision == CHAOS_PREC_COMPAT_FP64 || sg.handle->model->dim > 4)
      return fail(CHAOS_LYAP_EUNSUPPORTED,
                  "segment %d: batches take the adaptive forms of 3-4 dimensional models", i);
    if (i > 0 && (d.precision != segs[0].handle->d.precision ||
                  d.integrator != segs[0].handle->d.integrator ||
                  d.device != segs[0].handle->d.device))
      return fail(CHAOS_LYAP_EINVAL, "segment %d: integrator / precision / device differ", i);
    if (sg.P < 0 || (sg.P > 0 && (!sg.params || !sg.inits || !sg.spectrum)))
      return fail(CHAOS_LYAP_EINVAL, "segment %d: bad arrays", i);
    const bool sp = is_split(sg.handle);
    BatchPlan::Part &part = plan->part[sp ? next_split++ : next_lane++];
    part.h = sg.handle;
    part.split = sp;
    chaos::AdaptiveArgs &a = part.a;
    a.P = sg.P;
    a.k = d.k;
    a.gs = d.gs;
    a.rtol = d.rtol;
    a.atol = d.atol;
    a.h0 = d.h;
    a.hmax = d.h_max;
    a.hmin = d.h_min;
    a.t_transient = d.t_transient;
    a.t_align = d.t_align;
    a.t_avg = d.t_avg;
    a.dt_renorm = d.dt_renorm;
    a.max_steps = d.max_steps;
    a.escape = d.escape > 0 ? d.escape : 1e4;
    const ModelInfo *m = sg.handle->model;
    a.params = cview(sg.params, sg.P, m->nparams, d.layout);
    a.inits = cview(sg.inits, sg.P, m->dim, d.layout);
    a.t_avg_per_point = sg.t_avg_per_point;
    a.spectrum = view(sg.spectrum, sg.P, d.k, d.layout);
    a.status = sg.status;
    a.steps = sg.steps;
    a.queue_stride = chaos::queue_stride_for(sg.P);
    a.queue = h0->queue + i;  // the first handle's counters
    if (sg.t_avg_per_point && sg.P > 0) {  // longest averaging time first
      if (own) {
        a.order = own[i].order;
        part.scratch = own[i].scratch;
      } else {
        int rc = ensure_order(sg.handle, sg.P);
        if (rc) return rc;
        a.order = sg.handle->order;
        part.scratch = sg.handle->order_scratch;
      }
    }
  }
  const chaos_lyap_desc &d0 = h0->d;
  plan->integ = d0.integrator == CHAOS_INTEG_DOPRI5 ? chaos::kDopri5 : chaos::kDverk65;
  plan->prec = d0.precision == CHAOS_PREC_FP32 ? chaos::kFP32 : chaos::kFP64;
  std::stable_sort(plan->part + nsplit, plan->part + nseg,
                   [](const BatchPlan::Part &x, const BatchPlan::Part &y) { return x.a.P < y.a.P; });
  DeviceGuard g(d0.device);
  const double waves = lane_waves(*plan, false);
  plan->few_waves =
      plan->prec == chaos::kFP32 && waves < kBatchFewWaves &&
      (nseg == 1 || waves > (nsplit ? kBatchApartWavesSplit : kBatchApartWaves));
  plan->solo = plan->few_waves && nseg == 1 && nsplit == 0 && plan->part[0].a.order &&
               plan->part[0].a.P <= (int64_t)kBatchSoloPoints * h0->sm_count;
  plan->order_first = nseg > 1 && nsplit == 0 && lane_waves(*plan, plan->few_waves) > 1.0;
  if (nseg > 1) {  // fork / join resources
    cudaError_t e = cudaSuccess;
    if (!h0->ev_fork) e = cudaEventCreateWithFlags(&h0->ev_fork, cudaEventDisableTiming);
    for (int i = 0; i + 1 < nseg && e == cudaSuccess; i++) {
      if (!h0->aux_stream[i])
        e = cudaStreamCreateWithFlags(&h0->aux_stream[i], cudaStreamNonBlocking);
      if (e == cudaSuccess && !h0->ev_join[i])
        e = cudaEventCreateWithFlags(&h0->ev_join[i], cudaEventDisableTiming);
    }
    if (e != cudaSuccess) return cuda_fail(e, "batch fork streams / events");
  }
  return CHAOS_LYAP_OK;
}

static int batch_rc(int rc) {
  if (rc == chaos::kErrUnsupported) return fail(CHAOS_LYAP_EUNSUPPORTED, "no batch kernel for this mix");
  if (rc) return cuda_fail((cudaError_t)rc, "batch launch");
  return CHAOS_LYAP_OK;
}

static int launch_part(const BatchPlan &p, const BatchPlan::Part &q, cudaStream_t s) {
  const chaos_lyap_handle *h = q.h;
  if (q.split)
    return batch_rc(chaos::launch_split(h->model->id, p.integ, p.prec, q.a, h->block, h->variant, s,
                                        p.nseg > 1));
  return batch_rc(chaos::launch_adaptive(h->model->id, p.integ, p.prec, q.a, h->block,
                                         part_variant(p, q), s, p.solo ? kBatchSoloLanes : 0));
}

static int launch_order(const BatchPlan::Part &q, cudaStream_t s) {
  if (!q.a.order) return CHAOS_LYAP_OK;
  const int rc = chaos::launch_order_longest_first(q.a.t_avg_per_point, q.a.P,
                                                   const_cast<int32_t *>(q.a.order), q.scratch, s);
  return rc ? cuda_fail((cudaError_t)rc, "order launch") : CHAOS_LYAP_OK;
}

static int enqueue_batch(const BatchPlan &p, chaos_lyap_handle *h0, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(h0->queue, 0, sizeof(unsigned long long) * p.nseg, s);
  if (e != cudaSuccess) return cuda_fail(e, "cudaMemsetAsync(queues)");
  int rc = CHAOS_LYAP_OK;
  for (int i = 0; i < p.nseg && p.order_first && !rc; i++) rc = launch_order(p.part[i], s);
  if (p.nseg > 1 && (e = cudaEventRecord(h0->ev_fork, s)) != cudaSuccess)
    return cuda_fail(e, "batch fork");
  for (int i = 0; i < p.nseg; i++) {
    const BatchPlan::Part &q = p.part[i];
    const cudaStream_t t = i ? h0->aux_stream[i - 1] : s;
    if (i && (e = cudaStreamWaitEvent(t, h0->ev_fork, 0)) != cudaSuccess)
      return cuda_fail(e, "batch fork");
    if (!rc && !p.order_first) rc = launch_order(q, t);
    if (!rc) rc = launch_part(p, q, t);
    // join even after a failed launch, so that a capture still ends cleanly
    if (i && ((e = cudaEventRecord(h0->ev_join[i - 1], t)) != cudaSuccess ||
              (e = cudaStreamWaitEvent(s, h0->ev_join[i - 1], 0)) != cudaSuccess))
      return cuda_fail(e, "batch join");
  }
  h0->launches = 0;
  for (int i = 0; i < p.nseg && !rc; i++)
    if (p.part[i].a.P > 0) h0->launches += 1 + (p.part[i].a.order ? chaos::kOrderKernels : 0);
  return rc;
}

int chaos_lyap_run_batch(const chaos_lyap_segment *segs, int nseg, void *stream) {
  BatchPlan plan;
  int rc = build_batch(segs, nseg, &plan, nullptr);
  if (rc) return rc;
  DeviceGuard g(segs[0].handle->d.device);
  rc = enqueue_batch(plan, segs[0].handle, (cudaStream_t)stream);
  if (!rc) segs[0].handle->last_stream = (cudaStream_t)stream;
  return rc;
}

// A captured batch.  The graph owns the longest-first order buffers of its
// segments, so a later run on one of its handles (which may regrow that
// handle's own buffer) cannot leave the graph reading freed memory.
struct chaos_lyap_graph {
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  int device = 0;
  OrderBuf order[chaos::kMaxSegments] = {};
};

static void free_graph(chaos_lyap_graph *gr) {
  if (gr->exec) cudaGraphExecDestroy(gr->exec);
  if (gr->graph) cudaGraphDestroy(gr->graph);
  for (auto &o : gr->order) {
    cudaFree(o.order);
    cudaFree(o.scratch);
  }
  delete gr;
}

int chaos_lyap_batch_graph_create(const chaos_lyap_segment *segs, int nseg, chaos_lyap_graph **out) {
  if (!out) return fail(CHAOS_LYAP_EINVAL, "out is null");
  *out = nullptr;
  int rc = check_segments(segs, nseg);
  if (rc) return rc;
  DeviceGuard g(segs[0].handle->d.device);
  auto *gr = new chaos_lyap_graph();
  gr->device = segs[0].handle->d.device;
  for (int i = 0; i < nseg; i++) {
    if (!segs[i].t_avg_per_point || segs[i].P <= 0) continue;
    cudaError_t e = cudaMalloc(&gr->order[i].order, sizeof(int32_t) * segs[i].P);
    if (e == cudaSuccess) e = cudaMalloc(&gr->order[i].scratch, chaos::kOrderScratchBytes);
    if (e != cudaSuccess) {
      free_graph(gr);
      return fail(CHAOS_LYAP_ENOMEM, "cudaMalloc(graph order): %s", cudaGetErrorString(e));
    }
  }
  BatchPlan plan;
  rc = build_batch(segs, nseg, &plan, gr->order);
  if (rc) {
    free_graph(gr);
    return rc;
  }
  cudaStream_t cs;
  cudaError_t e = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking);
  if (e != cudaSuccess) {
    free_graph(gr);
    return cuda_fail(e, "cudaStreamCreate");
  }
  e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
  if (e == cudaSuccess) {
    rc = enqueue_batch(plan, segs[0].handle, cs);
    cudaError_t e2 = cudaStreamEndCapture(cs, &gr->graph);
    if (!rc && e2 != cudaSuccess) rc = cuda_fail(e2, "cudaStreamEndCapture");
  } else {
    rc = cuda_fail(e, "cudaStreamBeginCapture");
  }
  // per-node priorities: the split kernel's blocks are dispatched first
  if (!rc && (e = cudaGraphInstantiate(&gr->exec, gr->graph, cudaGraphInstantiateFlagUseNodePriority)) !=
                 cudaSuccess)
    rc = cuda_fail(e, "cudaGraphInstantiate");
  cudaStreamDestroy(cs);
  if (rc) {
    free_graph(gr);
    return rc;
  }
  *out = gr;
  return CHAOS_LYAP_OK;
}

int chaos_lyap_graph_launch(chaos_lyap_graph *g, void *stream) {
  if (!g) return fail(CHAOS_LYAP_EINVAL, "graph is null");
  DeviceGuard dg(g->device);
  cudaError_t e = cudaGraphLaunch(g->exec, (cudaStream_t)stream);
  return e == cudaSuccess ? CHAOS_LYAP_OK : cuda_fail(e, "cudaGraphLaunch");
}

int chaos_lyap_graph_destroy(chaos_lyap_graph *g) {
  if (!g) return CHAOS_LYAP_OK;
  DeviceGuard dg(g->device);
  free_graph(g);
  return CHAOS_LYAP_OK;
}

int chaos_lyap_trajectory(chaos_lyap_handle *h, int64_t P, const double *params,
                          const double *inits, int32_t nsteps, double *t_out, double *h_out,
                          double *x_out, int32_t *status, void *stream) {
  if (!h) return fail(CHAOS_LYAP_EINVAL, "handle is null");
  const chaos_lyap_desc &d = h->d;
  const ModelInfo *m = h->model;
  if (d.precision == CHAOS_PREC_COMPAT_FP64)
    return fail(CHAOS_LYAP_EUNSUPPORTED, "trajectories take the adaptive forms (FP64 or FP32)");
  if (m->type != 0 || m->dim > 4)
    return fail(CHAOS_LYAP_EUNSUPPORTED, "trajectories of flows of dimension <= 4 (model %s)",
                m->name);
  if (P < 0 || nsteps < 0) return fail(CHAOS_LYAP_EINVAL, "P and nsteps must be >= 0");
  if (P == 0 || nsteps == 0) return CHAOS_LYAP_OK;
  if (!params || !inits || !t_out || !h_out || !x_out) return fail(CHAOS_LYAP_EINVAL, "null array");
  DeviceGuard g(d.device);
  if (!g.ok) return fail(CHAOS_LYAP_ECUDA, "cannot select device %d", d.device);
  chaos::adaptive::TrajectoryArgs ta{};
  chaos::AdaptiveArgs &a = ta.a;
  a.P = P;
  a.k = m->dim;
  a.rtol = d.rtol;
  a.atol = d.atol;
  a.h0 = d.h;
  a.hmax = d.h_max;
  a.hmin = d.h_min;
  a.max_steps = d.max_steps;
  a.escape = d.escape > 0 ? d.escape : 1e4;
  a.params = cview(params, P, m->nparams, d.layout);
  a.inits = cview(inits, P, m->dim, d.layout);
  ta.nsteps = nsteps;
  ta.t_out = t_out;
  ta.h_out = h_out;
  ta.x_out = x_out;
  ta.status = status;
  const int integ = d.integrator == CHAOS_INTEG_DOPRI5 ? chaos::kDopri5 : chaos::kDverk65;
  const int prec = d.precision == CHAOS_PREC_FP32 ? chaos::kFP32 : chaos::kFP64;
  const int rc = chaos::launch_trajectory(m->id, integ, prec, ta, (cudaStream_t)stream);
  if (rc == chaos::kErrUnsupported)
    return fail(CHAOS_LYAP_EUNSUPPORTED, "no trajectory kernel for model %s", m->name);
  if (rc) return cuda_fail((cudaError_t)rc, "trajectory launch");
  h->last_stream = (cudaStream_t)stream;
  h->launches = 1;
  return CHAOS_LYAP_OK;
}

int chaos_lyap_get_variant(chaos_lyap_handle *h, int32_t *variant) {
  if (!h || !variant) return fail(CHAOS_LYAP_EINVAL, "null argument");
  *variant = h->variant;
  return CHAOS_LYAP_OK;
}

int chaos_lyap_get_launches(chaos_lyap_handle *h, int32_t *kernels) {
  if (!h || !kernels) return fail(CHAOS_LYAP_EINVAL, "null argument");
  *kernels = h->launches;
  return CHAOS_LYAP_OK;
}

int chaos_lyap_cudaLyapunov(int bn, int bs, size_t taskNum, int isQr, int isVar, int modelType,
                            double *inits, double *closePoints, int32_t dimension,
                            const char *model, double *params, int32_t paramsDim, double eps,
                            double integrationStep, double *lyapExps, int32_t expsNum,
                            double timeSkip, double timeSkipClP, double calcTime,
                            double addSkipSteps, void *stream) {
  (void)bn;
  (void)bs;
  const ModelInfo *m = find_model(model);
  if (!m) return fail(CHAOS_LYAP_ENOMODEL, "unknown model '%s'", model ? model : "(null)");
  if (modelType != m->type)
    return fail(CHAOS_LYAP_EINVAL, "model %s is a %s, modelType %d", m->name,
                m->type ? "map" : "flow", modelType);
  if (m->type != 0 && isQr)
    return fail(CHAOS_LYAP_EUNSUPPORTED, "map model %s: the QR method has no map branch", m->name);
  if (dimension != m->dim || paramsDim != m->nparams)
    return fail(CHAOS_LYAP_EINVAL, "model %s has dim %d and %d params (got %d, %d)", m->name,
                m->dim, m->nparams, dimension, paramsDim);
  if (expsNum < 1 || expsNum > m->dim) return fail(CHAOS_LYAP_EINVAL, "expsNum out of range");
  if (isQr && expsNum != m->dim)
    return fail(CHAOS_LYAP_EUNSUPPORTED, "QR method needs expsNum == dimension");
  if (!(integrationStep > 0)) return fail(CHAOS_LYAP_EINVAL, "integrationStep must be > 0");
  if (taskNum == 0) return CHAOS_LYAP_OK;
  if (!inits || !params || !lyapExps) return fail(CHAOS_LYAP_EINVAL, "null array");
  chaos::CompatArgs a{};
  a.P = (int64_t)taskNum;
  a.k = expsNum;
  a.method = isQr ? 2 : (isVar ? 1 : 0);
  a.eps = eps;
  a.step = integrationStep;
  a.t_skip = timeSkip;
  a.t_skip_clp = timeSkipClP;
  a.calc_time = calcTime;
  a.add_skip = addSkipSteps;
  a.params = chaos::CView{params, paramsDim, 1};
  a.inits = chaos::View{inits, dimension, 1};
  a.close = closePoints;
  a.lyap = chaos::View{lyapExps, expsNum, 1};
  a.accumulate = 1;
  a.status = nullptr;
  int rc = chaos::launch_compat(m->id, a, 64, (cudaStream_t)stream);
  if (rc == chaos::kErrUnsupported) return fail(CHAOS_LYAP_EUNSUPPORTED, "no kernel for this k");
  if (rc) return cuda_fail((cudaError_t)rc, "cudaLyapunov launch");
  return CHAOS_LYAP_OK;
}

}  // extern "C"
