// passes64.cu -- the HBM-pass kernels for ComplexF64.
#include "passes_kernels.cuh"

const void* cfft_pass_kernel64(int mode, bool batched) { return pass_kernel<double2>(mode, batched); }
