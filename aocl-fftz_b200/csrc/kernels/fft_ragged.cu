// Ragged executor: float instance and the launch side.
#include "fft_ragged.cuh"

extern "C" const void *fftz_ragged_kernel_f64(void);

static const void *ragged_kernel(int dtype) {
  return dtype == 0 ? (const void *)&fftz::fft_ragged_kernel<float> : fftz_ragged_kernel_f64();
}

extern "C" int fftz_ragged_grid(int dtype, int smem_bytes) {
  const void *fn = ragged_kernel(dtype);
  cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes > 48 * 1024 ? smem_bytes : 48 * 1024);
  // all of the unified L1 / shared array as shared memory: several CTAs per SM
  cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  int occ = 0, dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, 256, (size_t)smem_bytes) != cudaSuccess || occ < 1) {
    cudaGetLastError();
    occ = 1;
  }
  return occ * (nsm > 0 ? nsm : 148);
}

extern "C" int fftz_launch_ragged(const fftz_ragged_t *r, int grid, void *stream) {
  const void *fn = ragged_kernel(r->dtype);
  void *args[1] = {(void *)r};
  return (int)cudaLaunchKernel(fn, dim3((unsigned)grid), dim3(256), args, (size_t)r->smem_bytes, (cudaStream_t)stream);
}
