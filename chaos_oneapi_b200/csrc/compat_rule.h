// Which of the fixed-step sweep's two launch forms is faster: a group of lanes
// per point (compat_rows_kernel) or a thread per point (compat_kernel).
#pragma once
#include <cstdint>

namespace chaos {

// Lanes of a group: the state and k rows, rounded up to a power of two.
constexpr int compat_row_lanes(int k) { return k + 1 <= 2 ? 2 : k + 1 <= 4 ? 4 : 8; }

// A run's steps: of the state alone; of the state and its k rows; and how many of
// the latter end with a Gram-Schmidt pass.
struct CompatSteps {
  double state, rows, passes;
};
inline CompatSteps compat_steps(int method, double step, double t_skip, double t_skip_clp,
                                double calc_time, double add_skip) {
  auto steps = [&](double t) { return t > 0 ? t / step : 0.0; };
  const double calc = steps(calc_time);
  if (method == 2) return {steps(t_skip), calc, calc};  // QR: a pass after every step
  const double clp = steps(t_skip_clp);
  // (a period that is no whole number of steps is never reached)
  const bool whole = add_skip >= 1 && add_skip <= INT32_MAX && add_skip == (double)(int32_t)add_skip;
  return {steps(t_skip), clp + calc, clp + (whole ? calc / add_skip : 0.0)};
}

// Cost model, in steps of the state alone on a thread of its own (0.25-0.33 us).
//  Threads: up to kMaxLanePointsPerSm a scheduler has one warp, so a step lasts
//    its 1 + k rows one after the other, then their pass.
//  Groups: a step lasts one row and its pass; w warps of a scheduler share its FP64
//    pipe.  Every lane of a group repeats the steps of the state alone, which is
//    what the form loses where they are many.
// Fitted to 2,220 runs on a B200 (five models, FD / VAR / QR, k = 1 .. 4, 1 .. 87
// points per SM, six divisions of about 320 steps into the phases): the choice
// costs at most 6 % over the better form, where groups throughout cost up to 190 %
// (hyper-Rossler, k = 4, 87 points per SM, nine tenths of the steps of the state
// alone: 707 us against 244).  Lorenz FD, k = 3, 52 points per SM, thread / group:
// with nearly all steps of the rows 538 / 278 us, of the state alone 113 / 180 us.
struct CompatCost {
  double t_row, t_pass;          // thread: per row of a step, per row of a pass
  double state, row, pass;       // group: per step or pass, one warp per scheduler
  double state_w, row_w, pass_w; // and more for each further warp
};
// chua: a right-hand side of few operations, whose rows overlap on a thread.
inline CompatCost compat_cost(int method, int k, bool chua) {
  static constexpr CompatCost general[] = {{1.20, .58, 1.08, 1.65, 1.30, 1.00, .93, .07},
                                           {1.34, .97, 1.04, 1.41, 2.30, .98, .99, .22},
                                           {1.20, .54, 1.06, 2.15, 1.15, 1.00, .80, .10},
                                           {1.37, .97, 1.03, 1.70, 2.30, .99, 1.11, .10},
                                           {2.60, .00, .98, 4.30, .00, .97, 1.45, .00}},
                              short_f[] = {{.92, .48, 1.27, 1.74, .90, .67, .58, .02},
                                           {1.19, .74, 1.09, 1.45, 1.78, .81, .75, .05},
                                           {.91, .41, 1.29, 1.82, .92, .65, .46, .00},
                                           {1.09, .71, 1.10, 1.67, 1.75, .82, .74, .00},
                                           {1.98, .00, .96, 3.41, .00, .80, .93, .00}};
  const int i = method == 2 ? 4 : (method == 1 ? 2 : 0) + (k > 1);
  return chua ? short_f[i] : general[i];
}

inline bool compat_rows_faster(int method, int k, bool chua, int64_t P, int sms,
                               const CompatSteps &n) {
  // From here on one thread per point fills its schedulers (16,384 points: one
  // warp each); 800 steps of 16,384 points, k = 3, thread / group: Shimizu FD 976 /
  // 958 us, Lorenz VAR 1028 / 1120, Lorenz QR 1391 / 1474.
  constexpr int64_t kMaxLanePointsPerSm = 88;
  if (P > kMaxLanePointsPerSm * sms) return false;
  const int64_t warps = (P * compat_row_lanes(k) + 31) / 32;
  const double w = (double)((warps + 4LL * sms - 1) / (4LL * sms)) - 1.0;
  const CompatCost c = compat_cost(method, k, chua);
  const double threads = n.state + (1 + k) * (n.rows * c.t_row + n.passes * c.t_pass);
  const double groups = n.state * (c.state + c.state_w * w) + n.rows * (c.row + c.row_w * w) +
                        n.passes * (c.pass + c.pass_w * w);
  return groups < threads;
}

}  // namespace chaos
