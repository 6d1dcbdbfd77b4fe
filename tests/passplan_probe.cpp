// The host rules of the stage kernels (csrc/passplan.h) behind plain C
// functions, so that tests/test_passplan_rules.py can call the code itself.
#include "passplan.h"

extern "C" {
// the radix sequence of L and its tables; 0 if L has none
int probe_plan(int L, int maxr, int line, SfPlan* out) { return sf_plan(L, *out, maxr, line != 0); }
int probe_plan_bytes() { return (int)sizeof(SfPlan); }
double probe_mid_cost(const SfPlan* S, long long count, int e) {
    double c;
    sf_mid_rows(*S, count, (size_t)e, sf_budget((size_t)e), &c);
    return c;
}
int probe_cols_pays(long long n, long long count, int e) { return sf_cols_pays(n, count, (size_t)e); }
int probe_tile(const SfPlan* S, long long count, int e, int row, long long nb) {
    return sf_tile(*S, count, (size_t)e, row != 0, sf_pass_budget((size_t)e), nullptr, nb);
}
}
