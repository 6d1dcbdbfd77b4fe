// passes_kernels.cuh -- the HBM-pass kernels of one data type (passes.cuh),
// instantiated by passes32.cu and passes64.cu: three ComplexF32 CTAs per SM
// (80 registers) or two ComplexF64 ones (128).
#pragma once
#include "kernels.h"
#include "passes.cuh"

template <typename V> struct PassBlocks { static constexpr int value = 3; };
template <> struct PassBlocks<double2> { static constexpr int value = 2; };

template <typename V, int MODE> __device__ __forceinline__ void pass_body(const KParams& p, unsigned char* smem) {
    if constexpr (MODE == MODE_COLPASS) colpass_body<V>(p, smem);
    else if constexpr (MODE == MODE_COLS) colpass_body<V, true>(p, smem);
    else if constexpr (MODE == MODE_ROWPASS) rowpass_body<V>(p, smem);
    else if constexpr (MODE == MODE_MIDPASS) midpass_body<V>(p, smem);
    else if constexpr (MODE == MODE_LINE) line_body<V>(p, smem);
    else lconv_body<V>(p, smem);
}
template <typename V, int MODE>
__global__ void __launch_bounds__(CFFT_THREADS, PassBlocks<V>::value) k_pass(const __grid_constant__ KParams p) {
    extern __shared__ __align__(128) unsigned char smem[];
    pass_body<V, MODE>(p, smem);
}
template <typename V, int MODE>
__global__ void __launch_bounds__(CFFT_THREADS, PassBlocks<V>::value) kb_pass(BatchLaunch L) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ KParams sp;
    pass_body<V, MODE>(stage_params<V>(L, &sp), smem);
}
// cluster kernels: 384 ComplexF32 threads (two CTAs per SM at 80 registers, as
// many warps as three of 256) or 256 ComplexF64 ones
template <typename V> struct ClusThreads { static constexpr int value = CFFT_CLUS32; };
template <> struct ClusThreads<double2> { static constexpr int value = CFFT_CLUS64; };
template <typename V>
__global__ void __launch_bounds__(ClusThreads<V>::value, 2) k_clus(const __grid_constant__ KParams p) {
    extern __shared__ __align__(128) unsigned char smem[];
    clus_body<V, ClusThreads<V>::value>(p, smem);
}
template <typename V> __global__ void __launch_bounds__(ClusThreads<V>::value, 2) kb_clus(BatchLaunch L) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ KParams sp;
    clus_body<V, ClusThreads<V>::value>(stage_params<V>(L, &sp), smem);
}
template <typename V> const void* pass_kernel(int mode, bool batched) {
    switch (mode) {
        case MODE_COLPASS: return batched ? (const void*)kb_pass<V, MODE_COLPASS> : (const void*)k_pass<V, MODE_COLPASS>;
        case MODE_ROWPASS: return batched ? (const void*)kb_pass<V, MODE_ROWPASS> : (const void*)k_pass<V, MODE_ROWPASS>;
        case MODE_MIDPASS: return batched ? (const void*)kb_pass<V, MODE_MIDPASS> : (const void*)k_pass<V, MODE_MIDPASS>;
        case MODE_LINE: return batched ? (const void*)kb_pass<V, MODE_LINE> : (const void*)k_pass<V, MODE_LINE>;
        case MODE_LCONV: return batched ? (const void*)kb_pass<V, MODE_LCONV> : (const void*)k_pass<V, MODE_LCONV>;
        case MODE_COLS: return batched ? nullptr : (const void*)k_pass<V, MODE_COLS>;
        case MODE_CLUS: return batched ? (const void*)kb_clus<V> : (const void*)k_clus<V>;
    }
    return nullptr;
}
