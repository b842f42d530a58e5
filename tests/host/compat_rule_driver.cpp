// Test infrastructure only: evaluates the fixed-step sweep's choice of a launch
// form (chaos_oneapi_b200/csrc/compat_rule.h).  Built by tests/test_compat_rule.py.
// One line of standard input per question: method k chua P sms step t_skip
// t_skip_clp calc_time add_skip; prints 1 (groups) or 0 (threads) for each.
#include <cstdio>

#include "../../chaos_oneapi_b200/csrc/compat_rule.h"

int main() {
  int method, k, chua, sms;
  long long P;
  double step, skip, clp, calc, add;
  while (std::scanf("%d %d %d %lld %d %lf %lf %lf %lf %lf", &method, &k, &chua, &P, &sms, &step,
                    &skip, &clp, &calc, &add) == 10)
    std::printf("%d\n", (int)chaos::compat_rows_faster(
                            method, k, chua != 0, P, sms,
                            chaos::compat_steps(method, step, skip, clp, calc, add)));
}
