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
// twiddle table entry i is w_N^e
void probe_tw(const SfPlan* S, int i, long long* e, int* N) { sf_tw_entry(*S, i, e, N); }
// pitches of a row tile of V rows: out = run pitch, row pitch, shared memory
void probe_row(const SfPlan* S, int V, int e, int mid, int* out) {
    out[0] = sf_qp(*S, V, (size_t)e, mid != 0);
    out[1] = sf_qw(*S, V, (size_t)e, mid != 0);
    out[2] = (int)sf_row_smem(*S, V, (size_t)e, mid != 0);
}
// LINE: run pitch, row pitch, first digit's extra pitch, shared memory
void probe_line(const SfPlan* S, int V, int e, int* out) {
    out[0] = sf_qp(*S, 1, (size_t)e, true);
    out[1] = sf_line_qw(*S);
    out[2] = sf_line_q0(*S);
    out[3] = (int)sf_line_smem(*S, V, (size_t)e);
}
long long probe_clus_smem(const SfPlan* a, const SfPlan* c, int C, int e) { return (long long)sf_clus_smem(*a, *c, C, (size_t)e); }
unsigned probe_magic(int d) { return sf_magic(d); }
}
