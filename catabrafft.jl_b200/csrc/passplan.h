// passplan.h -- host rules of the HBM-pass kernels (passes.cuh), shared by the
// planner and the no-allocation entry point: radix sequence of a
// sub-transform, its twiddle table, tile widths and shared memory.
#pragma once
#include <algorithm>
#include <cmath>

#include "engine_types.h"

// Radix sequence of L (7-smooth, L >= 2): the fewest stages first (a stage is
// a shared-memory round trip and a barrier), then the least arithmetic, in
// ascending order -- the last radix is the largest, so the runs that the row
// layout keeps contiguous span a half-warp.  One stage becomes two (L, 1), as
// the kernels always run a first and a last one.
inline double sf_radix_cost(int r) {
    // real additions and multiplications per point of the codelets
    switch (r) {
        case 2: return 2.0; case 3: return 5.3; case 4: return 4.0; case 5: return 8.0; case 6: return 7.3;
        case 7: return 12.9; case 8: return 6.5; case 9: return 11.1; case 10: return 10.0; case 12: return 9.3;
        case 14: return 14.9; case 15: return 13.6; case 16: return 9.8;
    }
    return 1e9;
}
inline void sf_search(int rem, int maxr, int depth, double cost, int* cur, int* best, int* nbest, double* cbest) {
    static const int rad[] = {16, 15, 14, 12, 10, 9, 8, 7, 6, 5, 4, 3, 2};
    if (rem == 1) {
        if (depth < *nbest || (depth == *nbest && cost < *cbest)) {
            *nbest = depth;
            *cbest = cost;
            for (int i = 0; i < depth; i++) best[i] = cur[i];
        }
        return;
    }
    if (depth == SF_MAXS || depth >= *nbest) return;
    for (int r : rad) {
        if (r > maxr || rem % r) continue;
        cur[depth] = r;
        sf_search(rem / r, r, depth + 1, cost + sf_radix_cost(r) + 0.05 * r, cur, best, nbest, cbest);
    }
}
// fills L, np, r and the table layout; false if L has no sequence
inline bool sf_plan(int L, SfPlan& S) {
    S = SfPlan();
    S.L = L;
    if (L < 2) return false;
    int cur[SF_MAXS], best[SF_MAXS], n = SF_MAXS + 1;
    double c = 1e30;
    sf_search(L, 16, 0, 0.0, cur, best, &n, &c);
    if (n > SF_MAXS) return false;
    S.np = n < 2 ? 2 : n;
    if (n == 1) {
        S.r[0] = best[0];
        S.r[1] = 1;
    } else {
        for (int i = 0; i < n; i++) S.r[i] = best[n - 1 - i];
    }
    int off = 0, Ls = L;
    for (int s = 0; s < S.np - 1; s++) {
        S.off[s] = off;
        off += (S.r[s] - 1) * (Ls / S.r[s]);
        Ls /= S.r[s];
    }
    S.twlen = off;
    int pre = 1;
    for (int s = 1; s < S.np; s++) {
        pre *= S.r[s - 1];
        S.boff[s] = off;
        off += (S.r[s] - 1) * pre;
    }
    S.twall = off;
    return true;
}
// entry i of the twiddle table is w_N^e
inline __host__ __device__ void sf_tw_entry(const SfPlan& S, int i, long long* e, int* N) {
    if (i < S.twlen) {
        int s = 0, Ls = S.L;
        while (s + 1 < S.np - 1 && S.off[s + 1] <= i) Ls /= S.r[s++];
        const int nb = Ls / S.r[s], k = i - S.off[s];
        *e = (long long)(k / nb + 1) * (k % nb);
        *N = Ls;
        return;
    }
    int s = 1, pre = S.r[0];
    while (s + 1 < S.np && S.boff[s + 1] <= i) pre *= S.r[s++];
    const int n = (i - S.boff[s]) / pre + 1;
    int b = (i - S.boff[s]) % pre, K = 0;
    for (int j = s - 1; j >= 1; j--) {
        K = (K + b % S.r[j]) * S.r[j - 1];
        b /= S.r[j];
    }
    *e = (long long)n * (K + b);
    *N = pre * S.r[s];
}

// shared memory per CTA: three ComplexF32 or two ComplexF64 CTAs per SM (the
// register budgets of the kernels)
inline size_t sf_budget(size_t e) { return (e == 8 ? 74 : 112) * (size_t)1024; }
inline int sf_lg(int v) {
    int l = 0;
    while ((2 << l) <= v) l++;
    return l;
}
// rows: pitch of a last-radix run (odd) and of a row (odd, for ROWPASS)
inline int sf_qp(const SfPlan& S) { return S.r[S.np - 1] | 1; }
inline int sf_qw(const SfPlan& S) { return (S.L / S.r[S.np - 1] * sf_qp(S)) | 1; }
inline size_t sf_col_smem(const SfPlan& S, int V, size_t e) { return (size_t)S.L * V * e; }
inline size_t sf_row_smem(const SfPlan& S, int V, size_t e) { return (size_t)sf_qw(S) * V * e; }
// tile width (a power of two) of a pass over `count` columns / rows of `per`
// shared elements: about 4096 (ComplexF32) or 2048 (ComplexF64) elements a
// tile, wider until a segment of the strided side is 128 bytes as long as the
// budget holds it, and no wider than the count needs
inline int sf_tile(long long count, long long per, size_t e) {
    const long long want = e == 8 ? 4096 : 2048;
    long long V = 1;
    while (2 * V <= 64 && 2 * V * per * (long long)e <= (long long)sf_budget(e) && V < count &&
           (2 * V * per <= want || 2 * V * (long long)e <= 128))
        V *= 2;
    return (int)V;
}
// how a pass of sub-length L over `count` neighbours scores (lower is better):
// stages, short segments on the strided side, idle columns of a partial tile
inline double sf_pass_cost(const SfPlan& S, long long count, long long per, size_t e) {
    const int V = sf_tile(count, per, e);
    if ((size_t)V * per * e > sf_budget(e)) return 1e9;
    double c = 2.0 + S.np;
    for (int s = 0; s < S.np; s++) c += 0.06 * (S.r[s] > 1 ? sf_radix_cost(S.r[s]) : 0.0);
    const long long seg = V * (long long)e;
    if (seg < 32) c += 6.0;
    else if (seg < 64) c += 2.5;
    else if (seg < 128) c += 0.7;
    const long long tiles = (count + V - 1) / V;
    return c * (double)(tiles * V) / (double)count;
}
// MIDPASS: whole rows, contiguous on both sides; about 4096 (2048) elements
inline int sf_mid_rows(const SfPlan& S, long long count, size_t e) {
    const long long want = e == 8 ? 4096 : 2048;
    return (int)std::max<long long>(1, std::min<long long>(count, want / sf_qw(S)));
}
inline double sf_mid_cost(const SfPlan& S, long long count, size_t e) {
    const int V = sf_mid_rows(S, count, e);
    if (sf_row_smem(S, V, e) > sf_budget(e)) return 1e9;
    double c = 2.0 + 1.6 * S.np;
    for (int s = 0; s < S.np; s++) c += 0.12 * (S.r[s] > 1 ? sf_radix_cost(S.r[s]) : 0.0);
    const long long tiles = (count + V - 1) / V;
    return c * (double)(tiles * V) / (double)count;
}
