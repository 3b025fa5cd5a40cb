// Mixed-radix line kernels, double.
#define FZ_MR_T double
#define FZ_MR_GET fftz_mr_kernel_f64
#include "fft_mr_kernels.cuh"
