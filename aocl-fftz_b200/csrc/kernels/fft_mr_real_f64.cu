// Mixed-radix line kernels for real lines, double.
#define FZ_MR_T double
#define FZ_MR_REAL
#define FZ_MR_GET fftz_mr_real_kernel_f64
#include "fft_mr_kernels.cuh"
