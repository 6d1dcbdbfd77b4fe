// noalloc.cu -- cfft_fft_twopass_noalloc: the two-HBM-pass FFT with no
// device allocation.
//
// Some callers cannot allocate device memory at the moment they need a
// transform: code running inside a memory pool that forbids cudaMalloc, or
// inside a framework that owns every allocation through its own allocator
// and may not see the library allocate behind its back.  This entry point
// serves them: its scratch (the intermediate between the column pass and the
// row pass) and its twiddle tables live in one file-scope __device__ array of
// fixed size that every GPU loading the library holds until the process
// exits.  The caller passes the
// input and output; nothing else is allocated -- no cudaMalloc / cudaFree,
// no allocating library call, no host heap.
//
// Limits and behaviour:
//   * n must be 7-smooth and split as n = N1 * N2 with N1, N2 <= 4096, and
//     n <= kScratchBytes / element size (2^21 ComplexF64 or 2^22 ComplexF32
//     elements); larger or non-smooth n are rejected with CFFT_ERR_UNSUPPORTED.
//   * The batch is processed in chunks that fit the scratch.
//   * The first call on a device looks up the array's device address
//     (cudaGetSymbolAddress) and sets kernel attributes, once per device,
//     with that device current; make that first call before any stream
//     capture begins.
//   * Every call shares the array, and each call overwrites the tables and
//     scratch it uses (nothing is assumed to start at zero): calls that
//     overlap on the GPU -- on different streams, or from different host
//     threads -- race and corrupt each other's results.  Serialise them.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>

#include "../../include/catabra_b200.h"
#include "engine_types.h"
#include "kernels.h"
#include "passplan.h"

static constexpr size_t kScratchBytes = 32u << 20;   // intermediate between the passes
static constexpr size_t kTableBytes = 256u << 10;    // sub-transform + four-step twiddles
static constexpr int kMaxDevices = 64;

// the whole working set of the entry point, 256-byte aligned; in host code
// this name is a host-side stand-in, never a device address
static __device__ __align__(256) unsigned char g_noalloc_arena[kScratchBytes + kTableBytes];

namespace {

std::mutex g_setup_mu;
unsigned char* g_arena_ptr[kMaxDevices] = {};

// errors go to the library's thread-local cfft_last_error() text (a fixed
// buffer, no heap)
int noalloc_fail(int code, const char* what, cudaError_t e = cudaSuccess) {
    char msg[256];
    if (e != cudaSuccess)
        snprintf(msg, sizeof msg, "cfft_fft_twopass_noalloc: %s: %s", what, cudaGetErrorString(e));
    else
        snprintf(msg, sizeof msg, "cfft_fft_twopass_noalloc: %s", what);
    cfft_set_last_error(msg);
    return code;
}

// w_L^m = exp(-2 pi i m / L) in FP64 (sincospi), rounded once to the data type
template <typename V> __device__ V round_to(double c, double s);
template <> __device__ double2 round_to<double2>(double c, double s) { return make_double2(c, s); }
template <> __device__ float2 round_to<float2>(double c, double s) {
    return make_float2((float)c, (float)s);
}
__device__ double2 omega_dev(long long m, long long L) {
    m %= L;
    double s, c;
    sincospi(-2.0 * (double)m / (double)L, &s, &c);
    return make_double2(c, s);
}
// forward twiddle blocks of both sub-transforms (SfPlan.off) and the two-level table of w_M
template <typename V>
__global__ void k_noalloc_tables(V* twA, SfPlan A, V* twC, SfPlan Cc, double2* lo, int nlo, double2* hi, int nhi,
                                 int M) {
    const int stride = gridDim.x * blockDim.x;
    const int total = max(max(A.twlen, Cc.twlen), max(nlo, nhi));
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        for (int w = 0; w < 2; w++) {
            const SfPlan& T = w ? Cc : A;
            V* dst = w ? twC : twA;
            if (i >= T.twlen) continue;
            long long e;
            int N;
            sf_tw_entry(T, i, &e, &N);
            const double2 v = omega_dev(e, N);
            dst[i] = round_to<V>(v.x, v.y);
        }
        if (i < nlo) lo[i] = omega_dev(i, M);
        if (i < nhi) hi[i] = omega_dev((long long)i * nlo, M);
    }
}
// split of n, tiles and shared memory of its two passes (parameter blocks
// without pointers, direction or batch)
struct Split {
    long long n = 0;
    size_t e = 0;
    KParams col, row;
    size_t smem_col = 0, smem_row = 0;
};
// by the planner's rule: factors <= 4096 and 7-smooth, the least cost of the two
// passes.  Pricing every divisor pair takes up to 0.4 ms of host time (30240:
// 87 pairs), several times the transform, so the last lengths keep theirs in a
// fixed table, a slot by length
bool find_split(long long n, size_t e, Split& sp) {
    static std::mutex mu;
    static Split kept[32];
    Split& slot = kept[(size_t)(n * 2 + (e == 8)) * 2654435761u % 32];
    {
        std::lock_guard<std::mutex> lk(mu);
        if (slot.n == n && slot.e == e) {
            sp = slot;
            return true;
        }
    }
    long long N1 = -1;
    double best = 1e8;
    SfPlan pa, pc;
    for (long long a = 2; a <= 4096; a++) {
        if (n % a) continue;
        const long long b = n / a;
        if (b < 2 || b > 4096) continue;
        SfPlan ta, tc;
        if (!sf_plan((int)a, ta) || !sf_plan((int)b, tc)) continue;
        const double sc = sf_pass_cost(ta, b, e, false) + sf_pass_cost(tc, a, e, true);
        if (sc < best) { best = sc; N1 = a; pa = ta; pc = tc; }
    }
    if (N1 < 0) return false;
    sp.n = n;
    sp.e = e;
    KParams kp;
    memset(&kp, 0, sizeof kp);
    kp.conv = CONV_NONE;
    kp.nx = (int)n;
    kp.M = (int)n;
    kp.N1 = (int)N1;
    kp.N2 = (int)(n / N1);
    kp.C = 1;
    kp.sa = pa;
    kp.sc = pc;
    sp.col = sp.row = kp;
    sp.col.mode = MODE_COLPASS;
    sp.col.pre = PRE_NONE;
    sp.col.post = POST_TWIDDLE;
    sf_stage(sp.col, e, &sp.smem_col, true);
    sp.row.mode = MODE_ROWPASS;
    sf_stage(sp.row, e, &sp.smem_row, true);
    std::lock_guard<std::mutex> lk(mu);
    slot = sp;
    return true;
}
}  // namespace

extern "C" int cfft_fft_twopass_noalloc(int64_t n, int64_t batch, int dtype, const void* d_in,
                                        void* d_out, int direction, void* stream) {
    cfft_set_last_error("");
    if (n < 4 || batch < 1 || !d_in || !d_out || direction < 0 || direction > 2)
        return noalloc_fail(CFFT_ERR_INVALID, "bad argument (n >= 4, batch >= 1, buffers, direction)");
    if (dtype != CFFT_C128 && dtype != CFFT_C64)
        return noalloc_fail(CFFT_ERR_INVALID, "dtype must be CFFT_C128 or CFFT_C64");
    const size_t e = (dtype == CFFT_C128) ? 16 : 8;
    if ((size_t)n * e > kScratchBytes)
        return noalloc_fail(CFFT_ERR_UNSUPPORTED,
                            "n exceeds the fixed scratch (2^21 ComplexF64 / 2^22 ComplexF32 elements)");
    if (((uintptr_t)d_in % e) || ((uintptr_t)d_out % e))
        return noalloc_fail(CFFT_ERR_INVALID, "buffers must be aligned to the element size");
    Split sp;
    if (!find_split(n, e, sp))
        return noalloc_fail(CFFT_ERR_UNSUPPORTED,
                            "n must be 7-smooth with a split n = N1*N2, N1, N2 <= 4096");
    const SfPlan &pa = sp.col.sa, &pc = sp.col.sc;

    int dev = 0;
    cudaError_t ce = cudaGetDevice(&dev);
    if (ce != cudaSuccess) return noalloc_fail(CFFT_ERR_CUDA, "cudaGetDevice", ce);
    if (dev < 0 || dev >= kMaxDevices) return noalloc_fail(CFFT_ERR_UNSUPPORTED, "device index");
    const void* fcol = cfft_kernel_for(MODE_COLPASS, dtype);
    const void* frow = cfft_kernel_for(MODE_ROWPASS, dtype);
    unsigned char* arena;
    {
        std::lock_guard<std::mutex> lk(g_setup_mu);
        if (!g_arena_ptr[dev]) {
            // host code must not use g_noalloc_arena's name as an address: ask
            // the runtime for this device's copy, with this device current
            void* ptr = nullptr;
            ce = cudaGetSymbolAddress(&ptr, g_noalloc_arena);
            if (ce != cudaSuccess || !ptr)
                return noalloc_fail(CFFT_ERR_CUDA, "cudaGetSymbolAddress", ce);
            // shared-memory attributes for both element types' pass kernels
            for (int dt = 0; dt < 2 && ce == cudaSuccess; dt++) {
                ce = cfft_prepare_fn(cfft_kernel_for(MODE_COLPASS, dt), 128 * 1024, 1);
                if (ce == cudaSuccess) ce = cfft_prepare_fn(cfft_kernel_for(MODE_ROWPASS, dt), 128 * 1024, 1);
            }
            if (ce != cudaSuccess) return noalloc_fail(CFFT_ERR_CUDA, "kernel attributes", ce);
            g_arena_ptr[dev] = (unsigned char*)ptr;
        }
        arena = g_arena_ptr[dev];
    }
    cudaStream_t st = (cudaStream_t)stream;

    // carve the table region: twA[N1] twC[N2] (data type), then FP64 lo/hi
    int bits = 0;
    while ((1LL << (2 * bits)) < n) bits++;
    const int nlo = 1 << bits, nhi = (int)((n + nlo - 1) / nlo + 1);
    unsigned char* tab = arena + kScratchBytes;
    void* twA = tab;
    void* twC = tab + (size_t)pa.twlen * e;
    size_t off = (size_t)((pa.twlen + pc.twlen) * e + 255) & ~(size_t)255;
    double2* lo = (double2*)(tab + off);
    double2* hi = lo + nlo;
    if (off + (size_t)(nlo + nhi) * sizeof(double2) > kTableBytes)
        return noalloc_fail(CFFT_ERR_UNSUPPORTED, "twiddle tables exceed the fixed table region");
    if (dtype == CFFT_C128)
        k_noalloc_tables<double2><<<32, 256, 0, st>>>((double2*)twA, pa, (double2*)twC, pc, lo, nlo, hi,
                                                        nhi, (int)n);
    else
        k_noalloc_tables<float2><<<32, 256, 0, st>>>((float2*)twA, pa, (float2*)twC, pc, lo, nlo, hi,
                                                       nhi, (int)n);
    ce = cudaGetLastError();
    if (ce != cudaSuccess) return noalloc_fail(CFFT_ERR_CUDA, "table kernel launch", ce);

    KParams &col = sp.col, &row = sp.row;
    for (KParams* kp : {&col, &row}) {
        kp->dir = direction;
        kp->scale = (direction == CFFT_INVERSE) ? 1.0 / (double)n : 1.0;
        kp->t4.lo = lo;
        kp->t4.hi = hi;
        kp->t4.bits = bits;
        kp->t4.N = (int)n;
        kp->sa.tw = twA;
        kp->sc.tw = twC;
    }

    const long long chunk = std::max<long long>(1, (long long)(kScratchBytes / ((size_t)n * e)));
    for (long long b0 = 0; b0 < batch; b0 += chunk) {
        const long long nb = std::min(chunk, batch - b0);
        col.batch = row.batch = (int)nb;
        col.in = (const char*)d_in + (size_t)b0 * n * e;
        col.out = arena;
        col.in_dist = n;
        col.out_dist = n;
        row.in = arena;
        row.out = (char*)d_out + (size_t)b0 * n * e;
        row.in_dist = n;
        row.out_dist = n;
        ce = cfft_launch_fn(fcol, col, (unsigned)(nb * ((col.N2 + col.V - 1) / col.V)), CFFT_THREADS, sp.smem_col, 1, st);
        if (ce == cudaSuccess)
            ce = cfft_launch_fn(frow, row, (unsigned)(nb * ((row.N1 + row.V - 1) / row.V)), CFFT_THREADS, sp.smem_row, 1, st);
        if (ce != cudaSuccess) return noalloc_fail(CFFT_ERR_CUDA, "kernel launch", ce);
    }
    return CFFT_OK;
}
