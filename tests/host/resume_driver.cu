// Test infrastructure only: a point run as two pieces -- its transient
// (chaos_oneapi_b200/csrc/adaptive.cuh: run_transient), then the averaging phase
// from what that left (lane_resume) -- against the same point run start to finish
// (run_point), on the CPU.  Built by tests/test_host_resume.py with nvcc; never
// linked into the library.
//
//   resume_driver POINTS
// Prints per model, precision, integrator and scenario: the points, how many of
// them ended with status 0 .. 4, how many ended in their transient, and how many
// differ in any bit of status, steps or spectrum.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "../../chaos_oneapi_b200/csrc/adaptive.cuh"

using namespace chaos;
using namespace chaos::adaptive;

struct Model {
  const char *name;
  int n, np;
  double p[4], x[4];
};
static const Model kModels[] = {{"shimizu", 3, 2, {0.8, 0.5}, {0.1, 0.05, 0.02}},
                                {"lorenz", 3, 3, {10.0, 28.0, 8.0 / 3.0}, {1.0, 1.0, 1.0}},
                                {"rossler", 3, 3, {0.2, 0.2, 5.7}, {1.0, 1.0, 0.0}},
                                {"chua", 3, 4, {9.0, 14.3, -8.0 / 7.0, -5.0 / 7.0}, {0.1, 0.0, 0.0}},
                                {"hyper_rossler", 4, 2, {0.25, 0.05}, {-10.0, -6.0, 0.0, 10.0}}};

static const char *kScenarios[] = {"plain", "align", "mgs", "own_times", "max_steps", "hmin",
                                   "escape", "nonfinite"};

template <class M, class R, int INTEG>
static void run(const Model &m, int P, const char *prec, const char *integ, int scenario) {
  constexpr int N = M::N;
  std::mt19937_64 rng(scenario * 7 + N);
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  std::vector<double> params(P * m.np), inits(P * N), spec(2 * P * N, 7.0), t_avg(P), cost(P);
  for (int i = 0; i < P * m.np; i++) params[i] = m.p[i % m.np] * (1 + 0.05 * u(rng));
  for (int i = 0; i < P * N; i++) inits[i] = m.x[i % N] + 1e-3 * u(rng);
  for (double &t : t_avg) t = 3.0 + 2.0 * u(rng);
  std::vector<int32_t> status(2 * P, -1);
  std::vector<int64_t> steps(2 * P, -1), left(P);
  std::vector<R> state((2 * N + 1) * P);
  AdaptiveArgs a{};
  a.P = P;
  a.k = N;
  a.rtol = a.atol = sizeof(R) == 4 ? 1e-6 : 1e-8;
  a.h0 = 1e-2;
  a.t_transient = 4.0;
  a.t_avg = 5.0;
  a.dt_renorm = 1.0;
  a.max_steps = 1000000;
  a.escape = 1e4;
  a.params = CView{params.data(), m.np, 1};
  a.inits = CView{inits.data(), N, 1};
  if (!std::strcmp(kScenarios[scenario], "align")) a.t_align = 1.5;
  if (!std::strcmp(kScenarios[scenario], "mgs")) a.gs = 1;
  if (!std::strcmp(kScenarios[scenario], "own_times")) a.t_avg_per_point = t_avg.data();
  if (!std::strcmp(kScenarios[scenario], "nonfinite"))
    for (int i = 0; i < P; i++) params[i * m.np + i % m.np] = i % 3 ? NAN : 1e300 * (1 + i % 2);
  a.resume.state = state.data();
  a.resume.steps = left.data();
  a.resume.cost = cost.data();
  int counts[5] = {}, ended = 0, differ = 0;
  for (int pt = 0; pt < P; pt++) {
    if (!std::strcmp(kScenarios[scenario], "max_steps")) a.max_steps = 1 + 3 * pt;
    if (!std::strcmp(kScenarios[scenario], "hmin")) a.hmin = 1e-4 * std::pow(1.15, pt % 40);
    if (!std::strcmp(kScenarios[scenario], "escape")) a.escape = 0.05 * std::pow(1.2, pt % 40);
    a.spectrum = View{spec.data(), N, 1};
    a.status = status.data();
    a.steps = steps.data();
    run_point<M, N, R, INTEG>(a, pt);
    a.spectrum = View{spec.data() + P * N, N, 1};
    a.status = status.data() + P;
    a.steps = steps.data() + P;
    const Ctl c = make_ctl<R>(a);
    run_transient<M, R, INTEG>(a, c, pt);
    if (left[pt] < 0) {
      ended++;
    } else {
      Lane<M, N, R, INTEG> L;
      lane_resume(L, a, pt);
      for (;;) {
        if (lane_step(L, a, c) == kFinished) break;
        if (L.phase != kTransient && L.t_gs >= L.L && !lane_gram_schmidt(L, a, c)) {
          lane_finish(L, a, 1);
          break;
        }
      }
    }
    if (status[pt] >= 0 && status[pt] <= 4) counts[status[pt]]++;
    bool same = status[pt] == status[P + pt] && steps[pt] == steps[P + pt];
    for (int i = 0; i < N; i++) {
      const double s = spec[pt * N + i], t = spec[(P + pt) * N + i];
      same = same && (std::memcmp(&s, &t, sizeof s) == 0 || (s != s && t != t));
    }
    differ += !same;
  }
  std::printf("%s %s %s %s %d %d %d %d %d %d %d %d\n", m.name, prec, integ, kScenarios[scenario], P,
              counts[0], counts[1], counts[2], counts[3], counts[4], ended, differ);
}

template <class M> static void model(const Model &m, int P) {
  for (int s = 0; s < (int)(sizeof kScenarios / sizeof *kScenarios); s++) {
    run<M, double, kDopri5>(m, P, "fp64", "dopri5", s);
    run<M, double, kDverk65>(m, P, "fp64", "dverk65", s);
    run<M, float, kDopri5>(m, P, "fp32", "dopri5", s);
    run<M, float, kDverk65>(m, P, "fp32", "dverk65", s);
  }
}

int main(int argc, char **argv) {
  const int P = argc > 1 ? std::atoi(argv[1]) : 0;
  if (P < 1 || P > 10000) return 2;
  model<Shimizu>(kModels[0], P);
  model<Lorenz>(kModels[1], P);
  model<Rossler>(kModels[2], P);
  model<Chua>(kModels[3], P);
  model<HyperRossler>(kModels[4], P);
  return 0;
}
