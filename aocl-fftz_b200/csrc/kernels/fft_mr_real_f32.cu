// Mixed-radix line kernels for real lines, float.
#define FZ_MR_T float
#define FZ_MR_REAL
#define FZ_MR_GET fftz_mr_real_kernel_f32
#include "fft_mr_kernels.cuh"
