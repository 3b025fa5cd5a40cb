// Mixed-radix line kernels, float.
#define FZ_MR_T float
#define FZ_MR_GET fftz_mr_kernel_f32
#include "fft_mr_kernels.cuh"
