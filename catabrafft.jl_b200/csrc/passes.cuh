// passes.cuh -- the HBM passes of lengths that exceed a CTA (or cluster):
//
//   COLPASS  a tile of V adjacent columns of the N1 x N2 view of a transform:
//            N1-point DFTs down the columns, then either the four-step
//            twiddle w_M^(c k1) into the intermediate (POST_TWIDDLE) or the
//            Bluestein chirp into the caller's output (POST_CHIRP)
//   ROWPASS  a tile of V adjacent rows of the intermediate: N2-point DFTs,
//            X[k1 + N1 k2] into the caller's output
//   MIDPASS  the middle of a convolution, in place on V rows of the
//            intermediate: N2-point DFT, product with the FP64 spectrum,
//            conjugation, N2-point DFT that takes the digits in reverse
//            order, four-step twiddle w_M^(k1 j2)
//   LCONV    V whole convolutions (Rader or Bluestein) that fit a CTA, one row
//            of M points each: MIDPASS's stages between a prologue that reads
//            the caller's input (through the generator permutation, or times
//            the chirp) and an epilogue that writes the caller's output
//   CLUS     one transform on a cluster of C CTAs: COLPASS's stages over N2 / C
//            columns in each CTA, whose last stage writes the twiddled values
//            through distributed shared memory into the rows of the CTA that
//            owns them, then ROWPASS's stages over N1 / C rows
//   LINE     V whole transforms that fit a CTA, one row each: one kernel from
//            the caller's input to the caller's output
//
// A smooth length is COLPASS + ROWPASS; a Bluestein convolution is COLPASS
// (chirp) + MIDPASS + COLPASS (chirp): three passes over its M points, the
// four-step of the second FFT being the first one's run backwards.  (The
// reference runs the layered Stockham passes over the whole vector in memory,
// src/radix_exec.jl, and splits mixed lengths four-step style,
// src/mixed_radix.jl:44-78.)
//
// Sub-transforms (SfPlan, engine_types.h) are two to six stages.  The first
// stage's butterflies read global memory straight into registers and the last
// stage's write it straight from registers; between them every stage reads
// and writes its own positions of one shared-memory tile, so a stage costs
// one shared read and one write per element, one barrier, and no second
// buffer, and a thread's butterfly never has to be held across a barrier.  An
// earlier form staged the tile by cp.async and ran all stages from shared
// memory with runtime divisions per wave: it spent twice the instructions
// (issue slots are what bounds these kernels: 40 % ALU at 12 % of DRAM).
// Measured on B200, before it and now, per launch of the whole plan: ComplexF32
// 10^6 x 64 1321 -> 659 us, 3^10 x 512 510 -> 309, prime 999983 x 32 (a four-pass
// convolution before) 3822 -> 1329, 100003 x 128 1981 -> 494; ComplexF64 10^6 x 64
// 2475 -> 1202, 999983 x 32 8172 -> 2267.
// What a stage does per butterfly of radix R: R loads and R stores at a fixed
// stride, one DFT_R codelet, R - 1 table twiddles (exactly rounded, read
// through L1), and one or two small integer quotients.
//
// COLPASS tiles are stored position-major (position, column), the column
// fastest: adjacent lanes touch adjacent slots, and twiddle reads are
// broadcasts.  ROWPASS
// and MIDPASS tiles are row-major with every run of r[np - 1] positions
// padded to an odd pitch qp (position t at (t / r) qp + t % r), which keeps
// the last stage's stride-r reads off one bank, and rows at an odd pitch qw
// for ROWPASS, whose later stages take adjacent rows in adjacent lanes.
#pragma once
#include "engine.cuh"

// R as a compile-time constant for each radix the planner uses (sf_search in
// passplan.h); SF_SWITCH_LINE adds 18 and 20 for ComplexF32 (V of the enclosing
// template) in LINE and COLS, and radix 1.  (SF_SWITCH_CONV, LCONV's, has that
// case too: it is never reached, but without it the compiler spills twice as much)
#define SF_CASES(CALL)              \
    case 2: CALL(2); break;         \
    case 3: CALL(3); break;         \
    case 4: CALL(4); break;         \
    case 5: CALL(5); break;         \
    case 6: CALL(6); break;         \
    case 7: CALL(7); break;         \
    case 8: CALL(8); break;         \
    case 9: CALL(9); break;         \
    case 10: CALL(10); break;       \
    case 12: CALL(12); break;       \
    case 14: CALL(14); break;       \
    case 15: CALL(15); break;
#define SF_SWITCH(r, CALL)          \
    switch (r) {                    \
        SF_CASES(CALL)              \
        default: CALL(16); break;   \
    }
#define SF_SWITCH_LINE(r, CALL)                                   \
    switch (r) {                                                  \
        SF_CASES(CALL)                                            \
        case 1: CALL(1); break;                                   \
        case 18: if constexpr (sizeof(V) == 8) { CALL(18); } break; \
        case 20: if constexpr (sizeof(V) == 8) { CALL(20); } break; \
        default: CALL(16); break;                                 \
    }
// ComplexF64 takes LINE's switch, where 18 and 20 are empty cases: with the same
// registers and spills the compiler's code without them measured slower (97 x 1
// 7.2 us, 6.3 with; 2018 x 128 16.7, 16.2; 2503 x 8 the other way, 32.1, 32.7)
#define SF_SWITCH_CONV(r, CALL)     \
    if constexpr (sizeof(V) == 16) { SF_SWITCH_LINE(r, CALL) } \
    else switch (r) {               \
        SF_CASES(CALL)              \
        case 1: CALL(1); break;     \
        default: CALL(16); break;   \
    }
#define SF_SWITCH_LAST(r, CALL)     \
    if ((r) == 1) { CALL(1); }      \
    else SF_SWITCH(r, CALL)

template <int R, typename V> __device__ __forceinline__ void sf_dft(V (&v)[R]) {
    if constexpr (R > 1) dft<R>(v);
}
// v[k] *= t[(k - 1) step], k = 1 .. R - 1
template <int R, typename V> __device__ __forceinline__ void sf_twiddle(V (&v)[R], const V* t, int step) {
#pragma unroll
    for (int k = 1; k < R; k++) v[k] = cmul(v[k], __ldg(t + (k - 1) * step));
}
// x / d by the host's multiplier (sf_magic): x < 2^20, d <= 2^12
__device__ __forceinline__ int sf_div(int x, unsigned m) { return m ? (int)__umulhi((unsigned)x, m) : x; }
// output index of position b in digits 0 .. s - 1 (b < r[0] .. r[s - 1])
__device__ __forceinline__ int sf_index(const SfPlan& S, int s, int b) {
    int k = 0;
    for (int i = s - 1; i >= 1; i--) {
        const int q = sf_div(b, S.mr[i]);
        k = (k + (b - q * S.r[i])) * S.r[i - 1];
        b = q;
    }
    return k + b;
}

// ---------------------------------------------------------------- COLPASS
// thread -> column w = tid % V of the tile and butterflies k0, k0 + ks, ...
// (k0 = tid / V, ks = floor(T / V); the T - ks V threads left over idle)
struct ColThread {
    int w, k0, col;
    bool ok;
};
template <typename V, int R>
__device__ __forceinline__ void col_first(const KParams& p, V* buf, int t, const ColThread& c) {
    const SfPlan& S = p.sa;
    const int nb = S.L / R, N2 = p.N2, W = p.V, step = nb * N2;
    const V* tw = (const V*)S.tw + S.off[0];
    for (int b = c.k0; b < nb; b += p.ks) {
        V v[R];
        const int j0 = b * N2 + c.col;
        if (p.pre == PRE_CHIRP) {
            // rows past the input's end are zero; their reads go to the
            // butterfly's first row, so that no branch keeps the loads apart
            const int j1 = min(j0, p.nx - 1);
            if (p.in_fmt == IO_PLAIN) {
                const V* src = (const V*)p.in + (long long)t * p.in_dist;
#pragma unroll
                for (int m = 0; m < R; m++) v[m] = ldg_stream(src + (j0 + m * step < p.nx ? j0 + m * step : j1));
            } else {
#pragma unroll
                for (int m = 0; m < R; m++) v[m] = user_ld<V>(p, t, j0 + m * step < p.nx ? j0 + m * step : j1);
            }
            if (p.dir) {
#pragma unroll
                for (int m = 0; m < R; m++) v[m] = conjv(v[m]);
            }
#pragma unroll
            for (int m = 0; m < R; m++) {
                const int j = j0 + m * step;
                const V x = fromd<V>(cmul(tod(v[m]), __ldg(p.chirp + (j < p.nx ? j : j1))));
                v[m] = j < p.nx ? x : zero<V>();
            }
        } else if (p.post == POST_STORE) {
            const V* src = (const V*)p.in + (long long)b * p.in_stride + c.col;
            const long long rs = (long long)nb * p.in_stride;
#pragma unroll
            for (int m = 0; m < R; m++) v[m] = load_in(p, ldg_stream(src + m * rs));
        } else if (p.pre == PRE_NONE && p.in_fmt != IO_PLAIN) {
#pragma unroll
            for (int m = 0; m < R; m++) v[m] = load_in(p, user_ld<V>(p, t, (long long)j0 + (long long)m * step));
        } else {
            const V* src = (const V*)p.in + (long long)t * p.in_dist + j0;
#pragma unroll
            for (int m = 0; m < R; m++) v[m] = p.pre == PRE_RAW ? __ldcg(src + m * step) : ldg_stream(src + m * step);
            if (p.pre == PRE_NONE && p.dir) {
#pragma unroll
                for (int m = 0; m < R; m++) v[m] = conjv(v[m]);
            }
        }
        sf_dft<R>(v);
        sf_twiddle<R>(v, tw + b, nb);
        V* dst = buf + b * W + c.w;
        const int ds = nb * W;
#pragma unroll
        for (int m = 0; m < R; m++) dst[m * ds] = v[m];
    }
}
template <typename V, int R>
__device__ __forceinline__ void col_mid(const KParams& p, V* buf, int s, int Ls, const ColThread& c) {
    const SfPlan& S = p.sa;
    const int nb = Ls / R, total = S.L / R, W = p.V;
    const V* tw = (const V*)S.tw + S.off[s];
    for (int b = c.k0; b < total; b += p.ks) {
        const int K = sf_div(b, S.mnb[s]), tp = b - K * nb;
        V* e = buf + (K * Ls + tp) * W + c.w;
        const int ds = nb * W;
        V v[R];
#pragma unroll
        for (int m = 0; m < R; m++) v[m] = e[m * ds];
        sf_dft<R>(v);
        sf_twiddle<R>(v, tw + tp, nb);
#pragma unroll
        for (int m = 0; m < R; m++) e[m * ds] = v[m];
    }
}
template <typename V, int R>
__device__ __forceinline__ void col_last(const KParams& p, const V* buf, int t, const ColThread& c) {
    const SfPlan& S = p.sa;
    const int total = S.L / R, N2 = p.N2, W = p.V, col = c.col;
    // outputs k = K + total j of column c take w_M^(c K) (w_M^(c total))^j:
    // FP64 products of two table values, at most 15 of them (relative error a
    // few 1e-15), rounded once to the data type
    double2 st = make_double2(1, 0);
    if (p.post == POST_TWIDDLE) st = tw_two(p.t4, (unsigned)(col * total));
    for (int b = c.k0; b < total; b += p.ks) {
        const V* e = buf + b * R * W + c.w;
        V v[R];
#pragma unroll
        for (int m = 0; m < R; m++) v[m] = e[m * W];
        sf_dft<R>(v);
        const int K = sf_index(S, S.np - 1, b);
        if (p.post == POST_TWIDDLE) {
            V* o = (V*)p.out + (long long)t * p.out_dist + (K * N2 + col);
            const int step = total * N2;
            double2 wk = tw_two(p.t4, (unsigned)(col * K));
#pragma unroll
            for (int j = 0; j < R; j++) {
                o[j * step] = cmul(v[j], fromd<V>(wk));
                if (j < R - 1) wk = cmul(wk, st);
            }
        } else if (p.post == POST_STORE) {
            V* o = (V*)p.out + (long long)K * p.out_stride + col;
            const long long step = (long long)total * p.out_stride;
#pragma unroll
            for (int j = 0; j < R; j++) stg_stream(o + j * step, store_out(p, v[j]));
        } else {
            // outputs past the transform's end are dropped
            const int j0 = K * N2 + col, step = total * N2, j1 = min(j0, p.nx - 1);
#pragma unroll
            for (int j = 0; j < R; j++) {
                const int jj = j0 + j * step;
                v[j] = store_out(p, fromd<V>(cmul(tod(conjv(v[j])), __ldg(p.chirp + (jj < p.nx ? jj : j1)))));
            }
            if (p.out_fmt == IO_PLAIN) {
                V* o = (V*)p.out + (long long)t * p.out_dist + j0;
#pragma unroll
                for (int j = 0; j < R; j++)
                    if (j0 + j * step < p.nx) stg_stream(o + j * step, v[j]);
            } else {
#pragma unroll
                for (int j = 0; j < R; j++)
                    if (j0 + j * step < p.nx) user_st(p, t, j0 + j * step, v[j]);
            }
        }
    }
}
// LINE: whole transforms in columns, with LINE's radices (the same arithmetic)
template <typename V, bool LINE = false> __device__ __forceinline__ void colpass_body(const KParams& p, unsigned char* smem) {
    V* buf = (V*)smem;
    const SfPlan& S = p.sa;
    const int tile = block_id(p), tiles = (p.N2 + p.V - 1) / p.V;
    const int t = tile / tiles;
    if (t >= p.batch) return;                   // uniform across the CTA
    ColThread c;
    {
        const int tid = opaque_tid();
        c.k0 = sf_div(tid, p.mv);
        c.w = tid - c.k0 * p.V;
        c.col = (tile - t * tiles) * p.V + c.w;
        c.ok = c.k0 < p.ks && c.col < p.N2;     // the last tile may be partial
    }
#define SF_CALL(R) col_first<V, R>(p, buf, t, c)
    if (c.ok) {
        if constexpr (LINE) { SF_SWITCH_LINE(S.r[0], SF_CALL) }
        else { SF_SWITCH(S.r[0], SF_CALL) }
    }
#undef SF_CALL
    __syncthreads();
    int Ls = S.L / S.r[0];
    for (int s = 1; s < S.np - 1; s++) {
#define SF_CALL(R) col_mid<V, R>(p, buf, s, Ls, c)
        if (c.ok) {
            if constexpr (LINE) { SF_SWITCH_LINE(S.r[s], SF_CALL) }
            else { SF_SWITCH(S.r[s], SF_CALL) }
        }
#undef SF_CALL
        __syncthreads();
        Ls /= S.r[s];
    }
#define SF_CALL(R) col_last<V, R>(p, buf, t, c)
    if (c.ok) {
        if constexpr (LINE) { SF_SWITCH_LINE(S.r[S.np - 1], SF_CALL) }
        else { SF_SWITCH_LAST(S.r[S.np - 1], SF_CALL) }
    }
#undef SF_CALL
}

// ------------------------------------------------------- rows of a tile
// position t of a row sits at (t / rl) qp + t % rl, rl = r[np - 1]; strides of
// every stage but the last are multiples of rl positions
__device__ __forceinline__ int row_at(const SfPlan& S, int t, int qp) {
    const int q = sf_div(t, S.mr[S.np - 1]);
    return q * qp + (t - q * S.r[S.np - 1]);
}
// first stage: lanes take adjacent butterflies of a row (contiguous reads, of
// an intermediate that other SMs may have written in the same launch: through
// L2)
template <typename V, int R>
__device__ __forceinline__ void row_first(const KParams& p, V* buf, const V* src, int rows) {
    const SfPlan& S = p.sc;
    const int nb = S.L / R, qp = p.qp, total = rows * nb;
    const int ds = sf_div(nb, S.mr[S.np - 1]) * qp;
    const V* tw = (const V*)S.tw + S.off[0];
    for (int i = opaque_tid(); i < total; i += CFFT_THREADS) {
        const int r = sf_div(i, S.mnb[0]), b = i - r * nb;
        const V* x = src + (r * S.L + b);
        V v[R];
#pragma unroll
        for (int m = 0; m < R; m++) v[m] = __ldcg(x + m * nb);
        sf_dft<R>(v);
        sf_twiddle<R>(v, tw + b, nb);
        V* e = buf + r * p.qw + row_at(S, b, qp);
#pragma unroll
        for (int m = 0; m < R; m++) e[m * ds] = v[m];
    }
}
// a middle stage; LANES_W: adjacent lanes take adjacent rows (as COLPASS's
// adjacent columns), else adjacent butterflies of a row.  BACK: the second
// transform's stage on the same digit
template <typename V, int R, bool LANES_W, bool BACK, int T = CFFT_THREADS>
__device__ __forceinline__ void row_mid(const KParams& p, V* buf, int s, int Ls, int rows) {
    const SfPlan& S = p.sc;
    const int nb = Ls / R, per = S.L / R, qp = p.qp;
    const int ds = sf_div(nb, S.mr[S.np - 1]) * qp, pre = BACK ? S.L / Ls : 0;
    const V* tw = (const V*)S.tw + (BACK ? S.boff[s] : S.off[s]);
    const int tid = opaque_tid(), k0 = LANES_W ? sf_div(tid, p.mv) : 0;
    const int total = LANES_W ? (k0 < p.ks ? per : 0) : rows * per;
    for (int i = LANES_W ? k0 : tid; i < total; i += LANES_W ? p.ks : T) {
        int r, b;
        if (LANES_W) {
            r = tid - k0 * p.V;
            b = i;
        } else {
            r = sf_div(i, S.mper[s]);
            b = i - r * per;
        }
        const int K = sf_div(b, S.mnb[s]), tp = b - K * nb;
        V* e = buf + r * p.qw + row_at(S, K * Ls + tp, qp);
        V v[R];
#pragma unroll
        for (int m = 0; m < R; m++) v[m] = e[m * ds];
        sf_dft<R>(v);
        if (BACK) sf_twiddle<R>(v, tw + K, pre);
        else sf_twiddle<R>(v, tw + tp, nb);
#pragma unroll
        for (int m = 0; m < R; m++) e[m * ds] = v[m];
    }
}

// ---------------------------------------------------------------- ROWPASS
// thread -> row r of the tile and butterflies k0, k0 + ks, ... (adjacent lanes
// take adjacent rows: adjacent outputs)
template <typename V, int R>
__device__ __forceinline__ void row_last(const KParams& p, const V* buf, int t, int r0, int r, int k0, int ks) {
    const SfPlan& S = p.sc;
    const int per = S.L / R, N1 = p.N1;
    for (int b = k0; b < per; b += ks) {
        const V* e = buf + r * p.qw + b * p.qp;
        V v[R];
#pragma unroll
        for (int m = 0; m < R; m++) v[m] = e[m];
        sf_dft<R>(v);
        const int k0 = (r0 + r) + N1 * sf_index(S, S.np - 1, b), step = N1 * per;
        if (p.out_fmt == IO_PLAIN) {
            V* o = (V*)p.out + (long long)t * p.out_dist + k0;
#pragma unroll
            for (int j = 0; j < R; j++) stg_stream(o + j * step, store_out(p, v[j]));
        } else {
#pragma unroll
            for (int j = 0; j < R; j++) user_st(p, t, (long long)k0 + (long long)step * j, store_out(p, v[j]));
        }
    }
}
template <typename V> __device__ __forceinline__ void rowpass_body(const KParams& p, unsigned char* smem) {
    V* buf = (V*)smem;
    const SfPlan& S = p.sc;
    const int tile = block_id(p), tiles = (p.N1 + p.V - 1) / p.V;
    const int t = tile / tiles;
    if (t >= p.batch) return;                   // uniform across the CTA
    const int r0 = (tile - t * tiles) * p.V, rows = min(p.V, p.N1 - r0);
    const V* src = (const V*)p.in + (long long)t * p.in_dist + (long long)r0 * p.N2;
#define SF_CALL(R) row_first<V, R>(p, buf, src, rows)
    SF_SWITCH(S.r[0], SF_CALL)
#undef SF_CALL
    __syncthreads();
    int Ls = S.L / S.r[0];
    for (int s = 1; s < S.np - 1; s++) {
        // rows past the tile's last are padding: transformed, never stored
#define SF_CALL(R) row_mid<V, R, true, false>(p, buf, s, Ls, rows)
        SF_SWITCH(S.r[s], SF_CALL)
#undef SF_CALL
        __syncthreads();
        Ls /= S.r[s];
    }
    const int tid = opaque_tid(), k0 = sf_div(tid, p.mv), r = tid - k0 * p.V;
    if (k0 >= p.ks || r >= rows) return;
#define SF_CALL(R) row_last<V, R>(p, buf, t, r0, r, k0, p.ks)
    SF_SWITCH_LAST(S.r[S.np - 1], SF_CALL)
#undef SF_CALL
}

// ---------------------------------------------------------------- MIDPASS
// The last stage of the first transform leaves X[row][K + per j] of position
// b = the butterfly's in its registers: times the spectrum (stored in this
// order: entry row L + j per + b; ONE: one spectrum for every row), conjugated, it is the input of the second
// transform's first stage over the same digit.
template <typename V, int R, bool ONE>
__device__ __forceinline__ void mid_center(const KParams& p, V* buf, int r0, int rows) {
    const SfPlan& S = p.sc;
    const int per = S.L / R, total = rows * per;
    const V* tw = (const V*)S.tw + S.boff[S.np - 1];
    for (int i = opaque_tid(); i < total; i += CFFT_THREADS) {
        const int r = sf_div(i, S.mper[S.np - 1]), b = i - r * per;
        V* e = buf + r * p.qw + b * p.qp;
        const double2* sp = p.spec + (ONE ? (long long)b : (long long)(r0 + r) * S.L + b);
        V v[R];
#pragma unroll
        for (int m = 0; m < R; m++) v[m] = e[m];
        sf_dft<R>(v);
#pragma unroll
        for (int j = 0; j < R; j++) v[j] = conjv(fromd<V>(cmul(tod(v[j]), __ldg(sp + j * per))));
        sf_dft<R>(v);
        sf_twiddle<R>(v, tw + b, per);
#pragma unroll
        for (int m = 0; m < R; m++) e[m] = v[m];
    }
}
// the second transform's last stage (digit 0): outputs j2 = b + nb m of the
// row, times w_M^(k1 j2), back in the row's place in the intermediate
template <typename V, int R>
__device__ __forceinline__ void mid_last(const KParams& p, const V* buf, V* dst, int r0, int rows) {
    const SfPlan& S = p.sc;
    const int nb = S.L / R, qp = p.qp, total = rows * nb;
    const int ds = sf_div(nb, S.mr[S.np - 1]) * qp;
    for (int i = opaque_tid(); i < total; i += CFFT_THREADS) {
        const int r = sf_div(i, S.mnb[0]), b = i - r * nb;
        const V* e = buf + r * p.qw + row_at(S, b, qp);
        V v[R];
#pragma unroll
        for (int m = 0; m < R; m++) v[m] = e[m * ds];
        sf_dft<R>(v);
        // FP64 products as in col_last
        const unsigned k1 = (unsigned)(r0 + r);
        const double2 st = tw_two(p.t4, k1 * (unsigned)nb);
        double2 wk = tw_two(p.t4, k1 * (unsigned)b);
        V* o = dst + (r * S.L + b);
#pragma unroll
        for (int m = 0; m < R; m++) {
            o[m * nb] = cmul(v[m], fromd<V>(wk));
            if (m < R - 1) wk = cmul(wk, st);
        }
    }
}
template <typename V> __device__ __forceinline__ void midpass_body(const KParams& p, unsigned char* smem) {
    V* buf = (V*)smem;
    const SfPlan& S = p.sc;
    const int tile = block_id(p), tiles = (p.N1 + p.V - 1) / p.V;
    const int t = tile / tiles;
    if (t >= p.batch) return;                   // uniform across the CTA
    const int r0 = (tile - t * tiles) * p.V, rows = min(p.V, p.N1 - r0);
    const V* src = (const V*)p.in + (long long)t * p.in_dist + (long long)r0 * p.N2;
    V* dst = (V*)p.out + (long long)t * p.out_dist + (long long)r0 * p.N2;
#define SF_CALL(R) row_first<V, R>(p, buf, src, rows)
    SF_SWITCH(S.r[0], SF_CALL)
#undef SF_CALL
    __syncthreads();
    int Ls = S.L / S.r[0];
    for (int s = 1; s < S.np - 1; s++) {
#define SF_CALL(R) row_mid<V, R, false, false>(p, buf, s, Ls, rows)
        SF_SWITCH(S.r[s], SF_CALL)
#undef SF_CALL
        __syncthreads();
        Ls /= S.r[s];
    }
#define SF_CALL(R) mid_center<V, R, false>(p, buf, r0, rows)
    SF_SWITCH(S.r[S.np - 1], SF_CALL)
#undef SF_CALL
    __syncthreads();
    for (int s = S.np - 2; s >= 1; s--) {
        Ls *= S.r[s];
#define SF_CALL(R) row_mid<V, R, false, true>(p, buf, s, Ls, rows)
        SF_SWITCH(S.r[s], SF_CALL)
#undef SF_CALL
        __syncthreads();
    }
#define SF_CALL(R) mid_last<V, R>(p, buf, dst, r0, rows)
    SF_SWITCH(S.r[0], SF_CALL)
#undef SF_CALL
}

// ------------------------------------------------------------------- LINE
// Row layout as above, plus the first digit's blocks q0 further apart, so that
// the last stage's lanes, which take adjacent outputs (adjacent first digits),
// step by an odd pitch too.
__device__ __forceinline__ int line_at(const KParams& p, int t) {
    return row_at(p.sc, t, p.qp) + sf_div(t, p.sc.mnb[0]) * p.q0;
}
template <typename V, int R>
__device__ __forceinline__ void line_first(const KParams& p, V* buf, int t0, int rows) {
    const SfPlan& S = p.sc;
    const int nb = S.L / R, total = rows * nb;
    const int ds = sf_div(nb, S.mr[S.np - 1]) * p.qp + p.q0;
    const V* tw = (const V*)S.tw + S.off[0];
    for (int i = opaque_tid(); i < total; i += CFFT_THREADS) {
        const int r = sf_div(i, S.mnb[0]), b = i - r * nb;
        V v[R];
        if (p.in_fmt == IO_PLAIN) {
            const V* x = (const V*)p.in + (long long)(t0 + r) * p.in_dist + b;
#pragma unroll
            for (int m = 0; m < R; m++) v[m] = ldg_stream(x + m * nb);
        } else {
#pragma unroll
            for (int m = 0; m < R; m++) v[m] = user_ld<V>(p, t0 + r, b + m * nb);
        }
        if (p.dir) {
#pragma unroll
            for (int m = 0; m < R; m++) v[m] = conjv(v[m]);
        }
        sf_dft<R>(v);
        sf_twiddle<R>(v, tw + b, nb);
        V* e = buf + r * p.qw + row_at(S, b, p.qp);
#pragma unroll
        for (int m = 0; m < R; m++) e[m * ds] = v[m];
    }
}
template <typename V, int R>
__device__ __forceinline__ void line_mid(const KParams& p, V* buf, int s, int Ls, int rows) {
    const SfPlan& S = p.sc;
    const int nb = Ls / R, per = S.L / R, total = rows * per;
    const int ds = sf_div(nb, S.mr[S.np - 1]) * p.qp;
    const V* tw = (const V*)S.tw + S.off[s];
    for (int i = opaque_tid(); i < total; i += CFFT_THREADS) {
        const int r = sf_div(i, S.mper[s]), b = i - r * per;
        const int K = sf_div(b, S.mnb[s]), tp = b - K * nb;
        V* e = buf + r * p.qw + line_at(p, K * Ls + tp);
        V v[R];
#pragma unroll
        for (int m = 0; m < R; m++) v[m] = e[m * ds];
        sf_dft<R>(v);
        sf_twiddle<R>(v, tw + tp, nb);
#pragma unroll
        for (int m = 0; m < R; m++) e[m * ds] = v[m];
    }
}
// lanes take adjacent outputs K (stores are whole segments); the butterfly's
// position is K's digits in position order
template <typename V, int R>
__device__ __forceinline__ void line_last(const KParams& p, const V* buf, int t0, int rows) {
    const SfPlan& S = p.sc;
    const int per = S.L / R, total = rows * per;
    for (int i = opaque_tid(); i < total; i += CFFT_THREADS) {
        const int r = sf_div(i, S.mper[S.np - 1]), K = i - r * per;
        int k = K, d0 = K, b = K;
        if (S.np > 2) {
            k = sf_div(K, S.mr[0]);
            d0 = b = K - k * S.r[0];
            for (int s = 1; s < S.np - 2; s++) {
                const int q = sf_div(k, S.mr[s]);
                b = b * S.r[s] + (k - q * S.r[s]);
                k = q;
            }
            b = b * S.r[S.np - 2] + k;
        }
        const V* e = buf + r * p.qw + b * p.qp + d0 * p.q0;
        V v[R];
#pragma unroll
        for (int m = 0; m < R; m++) v[m] = e[m];
        sf_dft<R>(v);
        if (p.out_fmt == IO_PLAIN) {
            V* o = (V*)p.out + (long long)(t0 + r) * p.out_dist + K;
#pragma unroll
            for (int j = 0; j < R; j++) stg_stream(o + j * per, store_out(p, v[j]));
        } else {
#pragma unroll
            for (int j = 0; j < R; j++) user_st(p, t0 + r, K + j * per, store_out(p, v[j]));
        }
    }
}
template <typename V> __device__ __forceinline__ void line_body(const KParams& p, unsigned char* smem) {
    V* buf = (V*)smem;
    const SfPlan& S = p.sc;
    const int t0 = block_id(p) * p.V, rows = min(p.V, p.batch - t0);
    if (rows <= 0) return;                      // uniform across the CTA
#define SF_CALL(R) line_first<V, R>(p, buf, t0, rows)
    SF_SWITCH_LINE(S.r[0], SF_CALL)
#undef SF_CALL
    __syncthreads();
    int Ls = S.L / S.r[0];
    for (int s = 1; s < S.np - 1; s++) {
#define SF_CALL(R) line_mid<V, R>(p, buf, s, Ls, rows)
        SF_SWITCH_LINE(S.r[s], SF_CALL)
#undef SF_CALL
        __syncthreads();
        Ls /= S.r[s];
    }
#define SF_CALL(R) line_last<V, R>(p, buf, t0, rows)
    SF_SWITCH_LINE(S.r[S.np - 1], SF_CALL)
#undef SF_CALL
}

// ------------------------------------------------------------------ LCONV
// prologue + first stage: row r holds the zero-padded convolution input
//   Rader      x[g^j], j < n - 1 (src/prime.jl:66-74)
//   Bluestein  x[j] chirp[j], j < n
// reads past the end go to the butterfly's first entry (or the last one), so
// that no branch keeps the loads apart
template <typename V, int R>
__device__ __forceinline__ void lconv_first(const KParams& p, V* buf, int t0, int rows) {
    const SfPlan& S = p.sc;
    const int nb = S.L / R, total = rows * nb, len = p.conv == CONV_RADER ? p.nx - 1 : p.nx;
    const int ds = sf_div(nb, S.mr[S.np - 1]) * p.qp;
    const V* tw = (const V*)S.tw + S.off[0];
    for (int i = opaque_tid(); i < total; i += CFFT_THREADS) {
        const int r = sf_div(i, S.mnb[0]), b = i - r * nb, b1 = min(b, len - 1);
        V v[R];
        if (p.conv == CONV_RADER) {
            int g[R];
#pragma unroll
            for (int m = 0; m < R; m++) g[m] = __ldg(p.perm + (b + nb * m < len ? b + nb * m : b1));
            if (p.in_fmt == IO_PLAIN) {
                const V* x = (const V*)p.in + (long long)(t0 + r) * p.in_dist;
#pragma unroll
                for (int m = 0; m < R; m++) v[m] = x[g[m]];
            } else {
#pragma unroll
                for (int m = 0; m < R; m++) v[m] = user_ld<V>(p, t0 + r, g[m]);
            }
        } else if (p.in_fmt == IO_PLAIN) {
            const V* x = (const V*)p.in + (long long)(t0 + r) * p.in_dist;
#pragma unroll
            for (int m = 0; m < R; m++) v[m] = ldg_stream(x + (b + nb * m < len ? b + nb * m : b1));
        } else {
#pragma unroll
            for (int m = 0; m < R; m++) v[m] = user_ld<V>(p, t0 + r, b + nb * m < len ? b + nb * m : b1);
        }
        if (p.dir) {
#pragma unroll
            for (int m = 0; m < R; m++) v[m] = conjv(v[m]);
        }
#pragma unroll
        for (int m = 0; m < R; m++) {
            const int j = b + nb * m;
            if (p.conv == CONV_BLUE) v[m] = fromd<V>(cmul(tod(v[m]), __ldg(p.chirp + (j < len ? j : b1))));
            if (j >= len) v[m] = zero<V>();
        }
        sf_dft<R>(v);
        sf_twiddle<R>(v, tw + b, nb);
        V* e = buf + r * p.qw + row_at(S, b, p.qp);
#pragma unroll
        for (int m = 0; m < R; m++) e[m * ds] = v[m];
    }
}
// last stage + epilogue: c[j] = the conjugated outputs j = b + nb m
//   Rader      y[g^-j] = x[0] + c[j]  (x0: this row's, already conjugated)
//   Bluestein  y[j] = c[j] chirp[j]
template <typename V, int R>
__device__ __forceinline__ void lconv_last(const KParams& p, const V* buf, const double2* x0, int t0, int rows) {
    const SfPlan& S = p.sc;
    const int nb = S.L / R, total = rows * nb, len = p.conv == CONV_RADER ? p.nx - 1 : p.nx;
    const int ds = sf_div(nb, S.mr[S.np - 1]) * p.qp;
    for (int i = opaque_tid(); i < total; i += CFFT_THREADS) {
        const int r = sf_div(i, S.mnb[0]), b = i - r * nb, b1 = min(b, len - 1);
        const V* e = buf + r * p.qw + row_at(S, b, p.qp);
        V v[R];
#pragma unroll
        for (int m = 0; m < R; m++) v[m] = e[m * ds];
        sf_dft<R>(v);
        int k[R];
        if (p.conv == CONV_RADER) {
            const V z = fromd<V>(x0[2 * r]);
#pragma unroll
            for (int m = 0; m < R; m++) {
                k[m] = __ldg(p.iperm + (b + nb * m < len ? b + nb * m : b1));
                const V c = conjv(v[m]);
                v[m] = store_out(p, mk<V>(z.x + c.x, z.y + c.y));
            }
        } else {
#pragma unroll
            for (int m = 0; m < R; m++) {
                k[m] = b + nb * m;
                v[m] = store_out(p, fromd<V>(cmul(tod(conjv(v[m])), __ldg(p.chirp + (k[m] < len ? k[m] : b1)))));
            }
        }
        if (p.out_fmt == IO_PLAIN) {
            V* o = (V*)p.out + (long long)(t0 + r) * p.out_dist;
#pragma unroll
            for (int m = 0; m < R; m++)
                if (b + nb * m < len) o[k[m]] = v[m];
        } else {
#pragma unroll
            for (int m = 0; m < R; m++)
                if (b + nb * m < len) user_st(p, t0 + r, k[m], v[m]);
        }
    }
}
template <typename V> __device__ __forceinline__ void lconv_body(const KParams& p, unsigned char* smem) {
    V* buf = (V*)smem;
    const SfPlan& S = p.sc;
    const int t0 = block_id(p) * p.V, rows = min(p.V, p.batch - t0);
    if (rows <= 0) return;                      // uniform across the CTA
    double2* x0 = after16(buf + p.V * p.qw);    // per row: x[0], x[0] + the sum of the others
    if (p.conv == CONV_RADER) {
        // y[0] = x[0] + sum(x[1:]), summed in FP64 by one warp per row
        // (src/prime.jl:63-65); the input may be overwritten later (in place)
        const int lane = opaque_tid() & 31;
        for (int r = opaque_tid() >> 5; r < rows; r += CFFT_THREADS / 32) {
            double2 s = make_double2(0, 0);
            for (int j = 1 + lane; j < p.nx; j += 32) {
                const double2 d = tod(load_in(p, user_ld<V>(p, t0 + r, j)));
                s.x += d.x;
                s.y += d.y;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
                s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
            }
            if (lane == 0) {
                const double2 z = tod(load_in(p, user_ld<V>(p, t0 + r, 0)));
                x0[2 * r] = z;
                x0[2 * r + 1] = make_double2(z.x + s.x, z.y + s.y);
            }
        }
    }
#define SF_CALL(R) lconv_first<V, R>(p, buf, t0, rows)
    SF_SWITCH_CONV(S.r[0], SF_CALL)
#undef SF_CALL
    __syncthreads();
    int Ls = S.L / S.r[0];
    for (int s = 1; s < S.np - 1; s++) {
#define SF_CALL(R) row_mid<V, R, false, false>(p, buf, s, Ls, rows)
        SF_SWITCH_CONV(S.r[s], SF_CALL)
#undef SF_CALL
        __syncthreads();
        Ls /= S.r[s];
    }
#define SF_CALL(R) mid_center<V, R, true>(p, buf, 0, rows)
    SF_SWITCH_CONV(S.r[S.np - 1], SF_CALL)
#undef SF_CALL
    __syncthreads();
    for (int s = S.np - 2; s >= 1; s--) {
        Ls *= S.r[s];
#define SF_CALL(R) row_mid<V, R, false, true>(p, buf, s, Ls, rows)
        SF_SWITCH_CONV(S.r[s], SF_CALL)
#undef SF_CALL
        __syncthreads();
    }
#define SF_CALL(R) lconv_last<V, R>(p, buf, x0, t0, rows)
    SF_SWITCH_CONV(S.r[0], SF_CALL)
#undef SF_CALL
    if (p.conv == CONV_RADER)
        for (int r = opaque_tid(); r < rows; r += CFFT_THREADS)
            user_st(p, t0 + r, 0, store_out(p, fromd<V>(x0[2 * r + 1])));
}

// ------------------------------------------------------------------- CLUS
// the last column stage: output k1 = K + total j of column i2 goes, twiddled,
// to row k1 % R1 of CTA k1 / R1, whose row buffer nobody reads before the
// cluster barrier that follows
template <typename V, int R>
__device__ __forceinline__ void clus_exchange(const KParams& p, const V* buf, V* rowbuf, const ColThread& c) {
    cg::cluster_group cl = cg::this_cluster();
    const SfPlan& S = p.sa;
    const int total = S.L / R, W = p.V, R1 = p.N1 / p.C, at = row_at(p.sc, c.col, p.qp);
    const double2 st = tw_two(p.t4, (unsigned)(c.col * total));
    for (int b = c.k0; b < total; b += p.ks) {
        const V* e = buf + b * R * W + c.w;
        V v[R];
#pragma unroll
        for (int m = 0; m < R; m++) v[m] = e[m * W];
        sf_dft<R>(v);
        const int K = sf_index(S, S.np - 1, b);
        double2 wk = tw_two(p.t4, (unsigned)(c.col * K));
#pragma unroll
        for (int j = 0; j < R; j++) {
            const int k1 = K + total * j, d = sf_div(k1, p.mr1);
            V* dst = cl.map_shared_rank(rowbuf, d);
            dst[(k1 - d * R1) * p.qw + at] = cmul(v[j], fromd<V>(wk));
            if (j < R - 1) wk = cmul(wk, st);
        }
    }
}
template <typename V, int T> __device__ __forceinline__ void clus_body(const KParams& p, unsigned char* smem) {
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank(), t = block_id(p) / p.C;
    if (t >= p.batch) return;                   // uniform across the cluster
    V* buf = (V*)smem;                          // N1 x W columns
    V* rowbuf = buf + p.N1 * p.V;               // R1 rows
    {
        const SfPlan& S = p.sa;
        ColThread c;
        const int tid = opaque_tid();
        c.k0 = sf_div(tid, p.mv);
        c.w = tid - c.k0 * p.V;
        c.col = rank * p.V + c.w;
        c.ok = c.k0 < p.ks;
#define SF_CALL(R) col_first<V, R>(p, buf, t, c)
        if (c.ok) { SF_SWITCH(S.r[0], SF_CALL) }
#undef SF_CALL
        __syncthreads();
        int Ls = S.L / S.r[0];
        for (int s = 1; s < S.np - 1; s++) {
#define SF_CALL(R) col_mid<V, R>(p, buf, s, Ls, c)
            if (c.ok) { SF_SWITCH(S.r[s], SF_CALL) }
#undef SF_CALL
            __syncthreads();
            Ls /= S.r[s];
        }
        cl.sync();                              // every CTA of the cluster has started
#define SF_CALL(R) clus_exchange<V, R>(p, buf, rowbuf, c)
        if (c.ok) { SF_SWITCH_LAST(S.r[S.np - 1], SF_CALL) }
#undef SF_CALL
    }
    cl.sync();                                  // rows complete; no remote access after this
    const SfPlan& S = p.sc;
    const int R1 = p.N1 / p.C;
    int Ls = S.L;
    for (int s = 0; s < S.np - 1; s++) {
#define SF_CALL(R) row_mid<V, R, false, false, T>(p, rowbuf, s, Ls, R1)
        SF_SWITCH(S.r[s], SF_CALL)
#undef SF_CALL
        __syncthreads();
        Ls /= S.r[s];
    }
    const int tid = opaque_tid(), k0 = sf_div(tid, p.mr1), r = tid - k0 * R1;
    if (k0 >= p.ks2) return;
#define SF_CALL(R) row_last<V, R>(p, rowbuf, t, rank * R1, r, k0, p.ks2)
    SF_SWITCH_LAST(S.r[S.np - 1], SF_CALL)
#undef SF_CALL
}
