// Ragged executor, double.
#include "fft_ragged.cuh"

extern "C" const void *fftz_ragged_kernel_f64(void) { return (const void *)&fftz::fft_ragged_kernel<double>; }
