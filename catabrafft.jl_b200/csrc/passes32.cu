// passes32.cu -- the HBM-pass kernels for ComplexF32.
#include "passes_kernels.cuh"

const void* cfft_pass_kernel32(int mode, bool batched) { return pass_kernel<float2>(mode, batched); }
