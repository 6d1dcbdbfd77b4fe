// engine_types.h -- parameter blocks shared by the kernels and the planner.
#pragma once
#include <vector_types.h>

#define CFFT_MAXP 24

// Radix passes run in this order: odd radices first, so that the first
// pass's stride-R writes never hit a multiple of 8 elements (which would
// put a quarter-warp of 16-byte stores on one bank group).
#define CFFT_EXEC_ORDER {9, 7, 5, 3, 16, 8, 4, 2}

struct SubPlan {
    int L;                        // sub-transform length
    int np;                       // number of radix passes
    int G;                        // sub-transforms per block-wide wave (fits EMAX regs/thread)
    int Gwarp;                    // sub-transforms per warp group (0: block mode)
    unsigned char radix[CFFT_MAXP];  // pass radices in execution order
    unsigned char cnt[8];         // multiplicities of 9, 7, 5, 3, 16, 8, 4, 2 (CFFT_EXEC_ORDER)
    int twlen;                    // entries of tw
    // per-pass twiddle blocks in execution order: pass p (stride s, n1 =
    // L/(s r)) owns (r-1)*n1 entries, tw[off + (j-1)*n1 + q] = w_L^(j*q*s),
    // so adjacent lanes (adjacent q) read adjacent entries
    const void* tw;
};

// A sub-transform of the HBM-pass kernels (passes.cuh): L = r[0] r[1] ...
// r[np - 1], one stage per radix, every stage in place.  Before any stage,
// element t sits at position t; a position is the mixed-radix number of its
// digits d[0] .. d[np - 1] (d[0] most significant, d[s] < r[s]).  Stage s
// transforms digit s, so afterwards output index
//   k = d[0] + r[0] d[1] + r[0] r[1] d[2] + ...
// sits at the position of its digits.
#define SF_MAXS 6
struct SfPlan {
    int L, np;
    unsigned char r[SF_MAXS + 2];
    // forward twiddles of stage s < np - 1 (Ls = r[s] r[s+1] ..., nb = Ls / r[s]):
    //   tw[off[s] + (k - 1) nb + t] = w_Ls^(t k), 1 <= k < r[s], t < nb
    unsigned short off[SF_MAXS];
    // twiddles of stage s >= 1 of a second transform that takes the digits
    // last to first (pre = r[0] .. r[s - 1], K = the index of digits 0 .. s - 1):
    //   tw[boff[s] + (n - 1) pre + b] = w_(pre r[s])^(K(b) n), 1 <= n < r[s], b < pre
    unsigned short boff[SF_MAXS];
    int twlen;                    // entries of the forward blocks
    int twall;                    // entries of all blocks
    // ceil(2^32 / d) for quotients by d = nb of stage s, L / r[s] and r[s] (sf_div)
    unsigned mnb[SF_MAXS], mper[SF_MAXS], mr[SF_MAXS];
    const void* tw;
};

struct TwoLevel {                 // w_N^e = lo[e & mask] * hi[e >> bits]  (FP64)
    const double2* lo;
    const double2* hi;
    int bits;
    int N;
};

// w^e of the real transforms' sweeps in FP64, rounded once but for its last
// step: hi (1 + lo1), hi's rounding error kept in hr and lo1 = w^l - 1 small
struct RootTable {
    const double2* lo1;           // w^l - 1, l < 2^bits
    const double2* hi;            // w^(h 2^bits)
    const double2* hr;            // ... minus its rounded value
    int bits;
};

enum { MODE_ROWS = 0, MODE_FOUR = 1, MODE_COLPASS = 2, MODE_ROWPASS = 3, MODE_P2COL = 4, MODE_P2ROW = 5,
       MODE_CONVC = 6, MODE_MIXC = 7, MODE_P2CL = 8, MODE_MIDPASS = 9, MODE_LINE = 10,
       MODE_CLUS = 11, MODE_LCONV = 12 };
// kernel selector only (KParams.mode stays MODE_COLPASS): whole transforms in
// columns
enum { MODE_COLS = 17 };
// kernel selector only (KParams.mode stays MODE_FOUR): the generic four-step
// kernel instantiated with warp-synchronous sub-transforms
enum { MODE_FOUR_WARP = 16 };
enum { CONV_NONE = 0, CONV_RADER = 1, CONV_BLUE = 2 };
enum { PRE_NONE = 0, PRE_CHIRP = 1, PRE_RAW = 2 };       // COLPASS: the caller's input, times the chirp, an intermediate
// COLPASS: to the intermediate; times the chirp to the caller's output; to the
// caller's output as it is (whole transforms in columns)
enum { POST_TWIDDLE = 0, POST_CHIRP = 1, POST_STORE = 2 };

struct KParams {
    int mode, conv;
    int nx;                       // user transform length
    int M;                        // working FFT length (nx unless conv)
    int N1, N2, C;                // FOUR / pass split
    int V;                        // LINE / LCONV: transforms per CTA; passes: tile width
    int PA, PC;                   // smem pitches (column layout / row layout)
    int XP;                       // Rader x staging: chunk (FOUR)
    int pre, post;                // pass prologue / epilogue
    union {                       // FOUR: column (N1) / row (N2) plans; passes.cuh: sub-transforms
        struct { SubPlan pa, pc; };
        struct { SfPlan sa, sc; };
    };
    unsigned mv;                  // passes: multiplier of V (V = tile width of COLPASS / ROWPASS, rows of MIDPASS)
    int ks;                       // passes: floor(threads / V)
    int qp, qw;                   // ROWPASS / MIDPASS / LINE: pitches of a last-radix run and of a row
    int q0;                       // LINE: extra pitch of the first digit
    unsigned mr1;                 // CLUS: multiplier of R1 = N1 / C (rows per CTA)
    int ks2;                      // CLUS: floor(threads / R1)
    TwoLevel t4;                  // four-step twiddles w_M^(i2 k1)
    const int* perm;              // Rader: g^j mod nx, j < nx-1
    const int* iperm;             // Rader: g^-j mod nx
    const double2* chirp;         // Bluestein: exp(-i pi j^2 / nx), j < nx
    const double2* spec;          // conv spectrum / M (FP64)
    const void* in;
    void* out;
    long long in_dist, out_dist;  // elements between consecutive transforms
    int batch;                    // transforms in this launch
    int dir;                      // 0 forward, 1 inverse (scaled), 2 backward
    double scale;                 // 1/nx for dir 1, else 1
    // multiply-shift reciprocals (see fdiv) of the layout's divisors
    unsigned long long mW, mN2, mR1;
    int blk0;                     // first block of this parameter block in its launch
    unsigned char in_user, out_user;  // batched launches: in/out relative to the caller's buffers
    unsigned char in_fmt, out_fmt;    // IO_*: how in / out hold the caller's elements
    long long in_off, out_off;    // batched launches: element offsets added to the bases
    // power-of-two passes: the four-step table of w_n (row pass) and the
    // single-level table w_N1^e, e < N1 (column pass)
    TwoLevel t4n;
    const double2* twN1;
    // element strides of in / out (IO_STRIDED, IO_HALF; unused for IO_PLAIN)
    long long in_stride, out_stride;
};
// The caller's buffers as a plan's first and last stage address them:
// contiguous elements of the data type (IO_PLAIN), elements of the data type
// at a stride (IO_STRIDED), or ComplexF16 elements at a stride (IO_HALF, the
// arithmetic in ComplexF32).  Element i of transform t sits at
// t * dist + i * stride.
enum { IO_PLAIN = 0, IO_STRIDED = 1, IO_HALF = 2 };

// One launch of the batched executor: parameter blocks in device memory and,
// per block of the grid, the index of its parameter block.
struct BatchLaunch {
    const KParams* desc;
    const int* block_desc;
    const void* in_base;
    void* out_base;
    int dir;                      // direction of every block, or -1: each block's own
    int pad_;
};


// The batched form's single persistent launch: CTAs claim work items in
// ticket order; an item is one block of a parameter block (a whole
// single-CTA transform, or one tile of a two-pass stage).  An item may wait
// for a counter to reach `need` (the previous stage of its transform, or the
// release of the scratch half its chunk reuses) and adds one to counter
// `done` when finished.  Every wait is on items with smaller tickets, so the
// queue drains whatever the residency.
enum { QK_COLPASS = 0, QK_ROWPASS = 1, QK_MIDPASS = 2, QK_LINE = 3, QK_LCONV = 4 };
struct QItem {
    int desc;                     // parameter block
    int blk;                      // block within the parameter block
    int kind;                     // QK_*
    int wait, need;               // counter (-1: none) and the count to wait for
    int done;                     // counter to add one to (-1: none)
};
struct QueueLaunch {
    const KParams* desc;
    const QItem* items;
    const void* in_base;
    void* out_base;
    int* ctl;                     // [0] ticket, [1] abort flag, [2 ...] counters; zero before each launch
    int nitems;
    int dir;                      // direction of every item, or -1: each parameter block's own
};
