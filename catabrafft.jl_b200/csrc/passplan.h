// passplan.h -- host rules of the HBM-pass kernels (passes.cuh), shared by the
// planner and the no-allocation entry point: radix sequence of a
// sub-transform, its twiddle table, tile widths and shared memory.
#pragma once
#include <algorithm>
#include <cmath>

#include "engine_types.h"

static const int SF_THREADS = 256;    // CTA size of the pass kernels
static const int SF_SMS = 148;        // a B200's SMs, the only device this is built for

// Radix sequence of L (7-smooth, L >= 2): the fewest stages first (a stage is
// a shared-memory round trip and a barrier), then the least arithmetic, in
// ascending order -- the last radix is the largest, so the runs that the row
// layout keeps contiguous span a half-warp (the other way round a 24000-point
// two-pass plan took 225 us against 212).  One stage becomes two (L, 1), as
// the kernels always run a first and a last one.  Radices go up to maxr: 20 for
// ComplexF32 in LINE, at 8 bytes of spill (50000 x 360 as 18 x 20 63 us, as 6 x 6
// x 10 86; of 28 lengths from 162 to 8000 all are 2 - 38 % faster with them at
// full batches but 3600, 13 % slower), and so in COLS, which repeats LINE's
// arithmetic (884 bytes of spill stores, 260 without; from 24 % faster, 400 x
// 3000, to 6 % slower, 6000 x 1000); 16 elsewhere: in LCONV 18 and 20 spill 816
// bytes (144 without) and are slower throughout, 181 x 1 13.6 us (6.2 without),
// 3001 x 1 33.1 (23.2), x 4000 437 (376); in the HBM passes they measured from 5 %
// faster to 10 % slower, and 21 to 27 spill at 80 registers and lose 15 - 25 %
inline double sf_radix_cost(int r) {
    // real additions and multiplications per point of the codelets
    switch (r) {
        case 2: return 2.0; case 3: return 5.3; case 4: return 4.0; case 5: return 8.0; case 6: return 7.3;
        case 7: return 12.9; case 8: return 6.5; case 9: return 11.1; case 10: return 10.0; case 12: return 9.3;
        case 14: return 14.9; case 15: return 13.6; case 16: return 9.8; case 18: return 14.5; case 20: return 13.0;
    }
    return 1e9;
}
inline void sf_search(int rem, int maxr, int depth, double cost, int* cur, int* best, int* nbest, double* cbest) {
    static const int rad[] = {20, 18, 16, 15, 14, 12, 10, 9, 8, 7, 6, 5, 4, 3, 2};
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
// x / d = (x m) >> 32 with m = ceil(2^32 / d), exact for x < 2^20 and d <= 2^12;
// 0 stands for d = 1
inline unsigned sf_magic(int d) { return d == 1 ? 0u : (unsigned)(((1ULL << 32) + d - 1) / d); }
// fills L, np, r and the table layout; false if L has no sequence
inline bool sf_plan(int L, SfPlan& S, int maxr = 16, bool line = false) {
    S = SfPlan();
    S.L = L;
    if (L < 1) return false;
    if (L == 1) {                      // the identity (LINE)
        S.np = 2;
        S.r[0] = S.r[1] = 1;
        return true;
    }
    int cur[SF_MAXS], best[SF_MAXS], n = SF_MAXS + 1;
    double c = 1e30;
    sf_search(L, maxr, 0, 0.0, cur, best, &n, &c);
    if (n > SF_MAXS) return false;
    if (line && n == 1) {
        // a row of one butterfly is read a row per lane: two stages where L
        // factors, whose lanes read adjacent elements
        for (int a = 4; a >= 2 && n == 1; a--)
            if (L % a == 0 && L / a >= a) {
                best[0] = L / a;
                best[1] = a;
                n = 2;
            }
    }
    S.np = n < 2 ? 2 : n;
    if (n == 1) {
        S.r[0] = (unsigned char)best[0];
        S.r[1] = 1;
    } else {
        for (int i = 0; i < n; i++) S.r[i] = (unsigned char)best[n - 1 - i];
    }
    int off = 0, Ls = L;
    for (int s = 0; s < S.np - 1; s++) {
        S.off[s] = (unsigned short)off;      // at most 2 x 9216 entries
        off += (S.r[s] - 1) * (Ls / S.r[s]);
        Ls /= S.r[s];
    }
    S.twlen = off;
    int pre = 1;
    for (int s = 1; s < S.np; s++) {
        pre *= S.r[s - 1];
        S.boff[s] = (unsigned short)off;
        off += (S.r[s] - 1) * pre;
    }
    S.twall = off;
    int sub = L;
    for (int s = 0; s < S.np; s++) {
        sub /= S.r[s];
        S.mnb[s] = sf_magic(sub);
        S.mper[s] = sf_magic(L / S.r[s]);
        S.mr[s] = sf_magic(S.r[s]);
    }
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
// ... and of a pass's tile in a launch of its own: ComplexF64 tiles above 76 KB
// leave too little of an SM's L1 to the loads in flight (10^6 x 64 1422 us at
// 112 KB, 1212 at 76, 1283 at 64; 999983 x 32 2246 / 2182 / 2219).  The work
// queue's items keep the larger tiles: each pays the queue's overhead (1000
// mixed lengths 5785 us against 6580)
inline size_t sf_pass_budget(size_t e) { return (e == 8 ? 74 : 76) * (size_t)1024; }
// Pitches of a row tile, in elements: of a last-radix run, and of a row.
// ROWPASS's later stages take V adjacent rows in adjacent lanes: B lanes (16
// ComplexF32, 8 ComplexF64) share a wavefront, so from V = B rows an odd row
// pitch alone is conflict-free; below, the rows step by B / V and the B / V
// butterflies between them by an odd run pitch.  MIDPASS's lanes walk one row,
// whose last stage reads runs at an odd pitch.
inline int sf_qp(const SfPlan& S, int V, size_t e, bool mid) {
    const int rl = S.r[S.np - 1], B = e == 8 ? 16 : 8;
    return !mid && V >= B ? rl : rl | 1;
}
inline int sf_qw(const SfPlan& S, int V, size_t e, bool mid) {
    const int len = S.L / S.r[S.np - 1] * sf_qp(S, V, e, mid), B = e == 8 ? 16 : 8;
    if (mid) return len;
    const int step = V >= B || B % V ? 1 : B / V;
    return len + ((step - len) % B + B) % B;
}
inline size_t sf_col_smem(const SfPlan& S, int V, size_t e) { return (size_t)S.L * V * e; }
inline size_t sf_row_smem(const SfPlan& S, int V, size_t e, bool mid) { return (size_t)sf_qw(S, V, e, mid) * V * e; }
// Cost model of a tile, in SM cycles of one of its CTAs.  In the HBM passes a
// round of butterflies of radix R (each thread runs at most one) takes about
// 1340 + 171 R cycles at three CTAs per SM -- fitted to B200 timings of COLPASS
// at radix 10 (268 instructions a butterfly, one every 12 cycles) -- whether or
// not every thread has one, and a tile costs about one more such latency to
// start.  So widths are picked to fill the rounds, not for a target size.
inline double sf_round(int R, int dfts) { return 1340.0 + 171.0 * R * dfts; }
inline double sf_start() { return 2500.0; }
// LINE and LCONV, whole launches of equal CTAs: a round with idle threads costs
// its share less, a CTA a third of a round to start.  400000 x 120 ComplexF32
// (radices 10, 12) by rows per CTA: 10 224 us, 21 (one full round a stage) 160,
// 32 168, 42 (two) 148, 64 (three) 168: beyond about 130 KB of shared memory
// per SM the L1 left for the loads in flight shrinks.
inline double sf_rounds(long long items, int threads, int R, int dfts) {
    const double full = (double)(items / threads), rest = (double)(items % threads) / threads;
    return sf_round(R, dfts) * (full + (rest > 0 ? 0.4 + 0.6 * rest : 0.0));
}
inline double sf_line_start() { return 1100.0; }
inline double sf_crowd(size_t smem, size_t e) {
    const double total = (double)smem * (e == 8 ? 3 : 2) / 1024.0;
    return total > 130.0 ? 1.0 + 0.12 * (total - 130.0) / 68.0 : 1.0;
}
// A pass of nb transforms (0: many) of `tiles` tiles each costs its tiles, or as
// much as 200 (ComplexF64: 148) of them: fewer leave SMs idle, and then narrower
// tiles, each with fewer rounds, are faster however many they are.  ComplexF32 on
// B200, without this bound / with 148 / 200 / 296: 117649 x 1 22.4 / 10.4 / 10.3 /
// 10.4 us (15.4 before the stage kernels), 100000 x 8 17.0 / 15.3 / 13.8 / 13.8;
// ComplexF64 59049 x 4 17.3 / 13.7 / 13.3 / 13.2, 177147 x 4 23.1 / 23.2 / 25.1 /
// 27.0, 40009 x 1 27.0 / 19.1 / 19.3 / 19.2
inline double sf_launch(long long tiles, long long nb, size_t e) {
    const double least = e == 8 ? 200.0 : SF_SMS;
    return nb > 0 && (double)(tiles * nb) < least ? least / (double)nb : (double)tiles;
}
// cycles per useful element of a COLPASS / ROWPASS tile of width V
inline double sf_tile_cost(const SfPlan& S, int V, long long count, size_t e, bool row, size_t budget,
                           long long nb = 0) {
    const size_t smem = row ? sf_row_smem(S, V, e, false) : sf_col_smem(S, V, e);
    if (smem > budget) return 1e9 + (double)smem;
    const int ks = SF_THREADS / V;
    double c = sf_start();
    for (int s = 0; s < S.np; s++) {
        const int nb = S.L / S.r[s];
        // the column mapping keeps ks V threads
        c += sf_round(S.r[s], 1) * (row && s == 0 ? (V * nb + SF_THREADS - 1) / SF_THREADS : (nb + ks - 1) / ks);
    }
    // the strided side moves 32-byte sectors: whole ones if V and the row
    // length allow, else one more per segment
    const long long seg = V * (long long)e;
    const bool whole = seg % 32 == 0 && count * (long long)e % 32 == 0;
    const double sectors = (double)((seg + 31) / 32 + (whole ? 0 : 1)) * 32.0 / (double)seg;
    c *= 1.0 + 0.25 * (sectors - 1.0) + (seg < 64 ? 0.3 : seg < 128 ? 0.1 : 0.0);
    const long long tiles = (count + V - 1) / V;
    return c / (double)S.L * sf_launch(tiles, nb, e) / (double)count;
}
// the width with the least cost (at most 64)
inline int sf_tile(const SfPlan& S, long long count, size_t e, bool row, size_t budget, double* cost = nullptr,
                   long long nb = 0) {
    int best = 1;
    double bc = 1e300;
    for (int V = 1; V <= 64 && V <= count; V++) {
        const double c = sf_tile_cost(S, V, count, e, row, budget, nb);
        if (c < bc) {
            bc = c;
            best = V;
        }
    }
    if (cost) *cost = bc;
    return best;
}
inline double sf_pass_cost(const SfPlan& S, long long count, size_t e, bool row) {
    double c;
    sf_tile(S, count, e, row, sf_budget(e), &c);
    return c;
}
// MIDPASS and LCONV fuse the last stage with the second transform's first one
// (mid_center), which has no radix-1 form: a length of one radix, whose
// sequence is (L, 1), is no row of a convolution
inline bool sf_mid_fits(const SfPlan& S) { return S.r[S.np - 1] >= 2; }
// MIDPASS: whole rows, contiguous on both sides, the second transform's first
// stage fused with the first one's last
inline double sf_mid_tile_cost(const SfPlan& S, int V, long long count, size_t e, size_t budget, long long nb = 0) {
    if (!sf_mid_fits(S)) return 1e300;
    const size_t smem = sf_row_smem(S, V, e, true);
    if (smem > budget) return 1e9 + (double)smem;
    double c = sf_start();
    for (int s = 0; s < S.np; s++) {
        const int rounds = (V * (S.L / S.r[s]) + SF_THREADS - 1) / SF_THREADS;
        c += rounds * (s == S.np - 1 ? sf_round(S.r[s], 2) : 2.0 * sf_round(S.r[s], 1));
    }
    const long long tiles = (count + V - 1) / V;
    return c / (double)S.L * sf_launch(tiles, nb, e) / (double)count;
}
inline int sf_mid_rows(const SfPlan& S, long long count, size_t e, size_t budget, double* cost = nullptr,
                       long long nb = 0) {
    int best = 1;
    double bc = 1e300;
    for (int V = 1; V <= 32 && V <= count; V++) {
        const double c = sf_mid_tile_cost(S, V, count, e, budget, nb);
        if (c < bc) {
            bc = c;
            best = V;
        }
    }
    if (cost) *cost = bc;
    return best;
}
// LINE: V whole rows; lanes of the first and middle stages walk a row, those
// of the last one step by the first digit's pitch (odd)
inline int sf_line_q0(const SfPlan& S) {
    const int rl = S.r[S.np - 1];
    if (S.np < 3) return 0;
    return ((S.L / S.r[0] / rl) * (rl | 1)) % 2 ? 0 : 1;
}
inline int sf_line_qw(const SfPlan& S) {
    const int rl = S.r[S.np - 1];
    return S.L / rl * (rl | 1) + S.r[0] * sf_line_q0(S);
}
inline size_t sf_line_smem(const SfPlan& S, int V, size_t e) { return (size_t)sf_line_qw(S) * V * e; }
// transforms per CTA: the model's cost of the whole batch, waves of CTAs on
// 148 SMs x (three ComplexF32 or two ComplexF64)
inline int sf_line_rows(const SfPlan& S, long long batch, size_t e) {
    const long long slots = SF_SMS * (e == 8 ? 3 : 2);
    int best = 1;
    double bc = 1e300;
    for (int V = 1; V <= 1024 && V <= batch; V++) {
        if (V > 1 && sf_line_smem(S, V, e) > sf_budget(e)) break;
        double c = sf_line_start();
        for (int s = 0; s < S.np; s++) c += sf_rounds((long long)V * (S.L / S.r[s]), SF_THREADS, S.r[s], 1);
        c *= sf_crowd(sf_line_smem(S, V, e), e);
        // whole waves while there are few; their tails matter less and less
        const double waves = (double)((batch + V - 1) / V) / (double)slots;
        c *= waves < 4.0 ? std::ceil(waves) : waves + 0.5;
        if (c < bc) {
            bc = c;
            best = V;
        }
    }
    return best;
}
// LCONV: V rows of M points, and two FP64 values a row (Rader)
inline size_t sf_lconv_smem(const SfPlan& S, int V, size_t e) {
    return ((size_t)sf_qw(S, V, e, true) * V * e + 15) / 16 * 16 + (size_t)V * 32;
}
inline int sf_lconv_rows(const SfPlan& S, long long batch, size_t e, double* cost = nullptr) {
    const long long slots = SF_SMS * (e == 8 ? 3 : 2);
    int best = 1;
    double bc = 1e300;
    for (int V = 1; V <= 256 && V <= batch; V++) {
        if (V > 1 && sf_lconv_smem(S, V, e) > sf_budget(e)) break;
        double c = sf_line_start();
        for (int s = 0; s < S.np; s++) {
            const long long items = (long long)V * (S.L / S.r[s]);
            c += s == S.np - 1 ? sf_rounds(items, SF_THREADS, S.r[s], 2) : 2.0 * sf_rounds(items, SF_THREADS, S.r[s], 1);
        }
        c *= sf_crowd(sf_lconv_smem(S, V, e), e);
        const double waves = (double)((batch + V - 1) / V) / (double)slots;
        c *= waves < 4.0 ? std::ceil(waves) : waves + 0.5;
        if (c < bc) {
            bc = c;
            best = V;
        }
    }
    if (cost) *cost = bc;
    return best;
}
// Strided plans whose transforms lie side by side: as columns of tiles (COLS)
// only from 4.5 MB on, else as LINE's strided rows.  Whole segments save more
// with size, but a 2D transform that runs its other axis in LINE then runs two
// large kernels in turn, each finding the instruction caches without it: 2.5 to
// 4.5 us a pair.  Both axes of a ComplexF32 image on B200, with COLS / with LINE
// alone: 128 x 128 8.2 / 5.3 us, 256 x 256 11.3 / 6.8, 512 x 512 (2 MB) 11.0 /
// 9.3, 640 x 640 (3.1) 13.4 / 13.0, 768 x 768 (4.5) 13.5 / 15.2, 1000 x 1000 18.7
// / 23.0; ComplexF64 512 x 512 (4) 12.2 / 10.5, 640 x 640 (6.3) 15.8 / 16.4
inline bool sf_cols_pays(long long n, long long count, size_t e) {
    return (double)n * (double)count * (double)e >= 4.5 * (1 << 20);
}
// tile, pitches and shared memory of a pass (mode, N1, N2, sa, sc set)
// (own: in a launch of its own, of nb transforms; 0: many)
inline void sf_stage(KParams& k, size_t e, size_t* smem, bool own, long long nb = 0) {
    const size_t budget = own ? sf_pass_budget(e) : sf_budget(e);
    const bool mid = k.mode == MODE_MIDPASS;
    if (k.mode == MODE_COLPASS) k.V = sf_tile(k.sa, k.N2, e, false, budget, nullptr, nb);
    else if (mid) k.V = sf_mid_rows(k.sc, k.N1, e, budget, nullptr, nb);
    else k.V = sf_tile(k.sc, k.N1, e, true, budget, nullptr, nb);
    k.mv = sf_magic(k.V);
    k.ks = SF_THREADS / k.V;
    k.qp = sf_qp(k.sc, k.V, e, mid);
    k.qw = sf_qw(k.sc, k.V, e, mid);
    *smem = k.mode == MODE_COLPASS ? sf_col_smem(k.sa, k.V, e) : sf_row_smem(k.sc, k.V, e, mid);
}
// CLUS: shared memory of an N1 x N2 split on C CTAs
inline size_t sf_clus_smem(const SfPlan& a, const SfPlan& c, int C, size_t e) {
    return ((size_t)a.L * (c.L / C) + (size_t)(a.L / C) * sf_qw(c, a.L / C, e, false)) * e;
}
// cycles of a CTA of CLUS, with its segments' sectors and its barriers
inline double sf_clus_cycles(const SfPlan& a, const SfPlan& c, int C, size_t e, int threads) {
    const int W = c.L / C, R1 = a.L / C, kc = threads / W, kr = threads / R1;
    double t = sf_start() + 2000.0;
    for (int s = 0; s < a.np; s++) t += sf_round(a.r[s], 1) * ((a.L / a.r[s] + kc - 1) / kc);
    for (int s = 0; s < c.np; s++) {
        const int nb = c.L / c.r[s];
        t += sf_round(c.r[s], 1) * (s == c.np - 1 ? (nb + kr - 1) / kr : (R1 * nb + threads - 1) / threads);
    }
    for (long long seg : {W * (long long)e, R1 * (long long)e})
        t *= seg < 32 ? 1.6 : seg < 64 ? 1.2 : seg < 128 ? 1.05 : 1.0;
    if (W < 32) t *= 1.2;          // the exchange writes runs of W elements
    return t * (1.0 + 0.02 * C + (C > 8 ? 0.3 : 0.0));
}
// ... per element, of many transforms
inline double sf_clus_cost(const SfPlan& a, const SfPlan& c, int C, size_t e, int threads) {
    if (c.L / C > threads || a.L / C > threads) return 1e9;
    const double t = sf_clus_cycles(a, c, C, e, threads);
    return (sf_clus_smem(a, c, C, e) > 112 * 1024 ? 1.6 * t : t) / ((double)a.L * (c.L / C));
}
// Time of `batch` transforms in cycles.  Up to 148 CTAs take a CTA's own time
// however few they are, so that a few transforms take as many CTAs as shorten
// them; more share SMs (at least 1.35 times as long, 2.1 times at 296, two to an
// SM) and then run in waves.  By cost per element 8 x 19683 ComplexF64 took
// clusters of 3 (18.4 us; 10.3 on clusters of 9, 14.7 before the stage kernels).
// Above 148 CTAs fewer are as good: 40 x 9000 10.7 us on clusters of 3, 11.7 on 5;
// 40 x 9604 12.6 on 2, 17.2 on 7; 40 x 10000 11.7 on 4, 12.3 on 2
inline double sf_clus_time(const SfPlan& a, const SfPlan& c, int C, size_t e, int threads, long long batch) {
    const double t = sf_clus_cycles(a, c, C, e, threads);
    if (batch * C <= SF_SMS) return t;
    const bool one = sf_clus_smem(a, c, C, e) > 112 * 1024;
    const double w = (double)batch * C / (one ? 148.0 : 296.0);
    return t * std::max(1.35, (one ? 1.68 : 2.1) * (w < 1.0 ? w : w < 4.0 ? std::ceil(w) : w + 0.5));
}
