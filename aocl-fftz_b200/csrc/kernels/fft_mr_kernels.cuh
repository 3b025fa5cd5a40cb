// Instances of the mixed-radix line kernel for one dtype (FZ_MR_T): plain
// lines and four-step column passes for every radix, chirp passes (tables,
// two sweeps) for radices without 11 and 13, which no convolution length has.
#include "fft_mr.cuh"

namespace fftz {

// float: at most 1024 threads = 64 registers; double: 512 threads = 128
// registers (a radix-16 butterfly holds 32 / 64 registers of data); the
// radix-11 / 13 instances get 768 / 384 threads for their longer live ranges.
template <typename T, bool BIG> __host__ __device__ constexpr int mr_lb() {
  return sizeof(T) == 4 ? (BIG ? 768 : 1024) : (BIG ? 384 : 512);
}

// Measured on B200 against the ping-pong tiles this replaced (two buffers, one
// prime radix a stage, 153 thread instructions a point at n = 1000; now 86):
// n = 1000 x 32768 float 242 -> 130 us (2.16 -> 4.04 TB/s read + written),
// four 1920 x 1080 images (rows, then columns) 181 -> 94 us, 120000 = 375 x 320 in
// double x 64 (two passes) 307 -> 160 us, 77 x 100000 float 45 us. ncu at n = 1000:
// issue 64%, shared-memory wavefronts 70%, DRAM 45% of peak -- issue and the
// shared-memory pipe together, not HBM, bound it. Lines per CTA at n = 1000, at 94
// instructions: 2 166, 3 136, 4 146, 5 135 (fz_mr_shape's choice), 6 142 us.
// Real lines, against the kernels that loaded, transformed and recombined in
// separate sweeps of shared memory (r2c / c2r us, before -> after): 2048 x 8192
// float 56 / 54 -> 41 / 42, 512 x 262144 double 730 / 642 -> 521 / 460, 1024 x 65536
// double 329 / 351 -> 247 / 273, 256 x 65536 float 133 / 133 -> 42 / 40, 1000 x 16000
// float 203 / 204 -> 43 / 41, 44100 x 200 float (four passes before) 311 / 309 -> 51 / 47.
template <typename T, int FEAT, bool BIG>
__global__ void __launch_bounds__(mr_lb<T, BIG>()) fft_mr_kernel(const __grid_constant__ fftz_pass_t P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  mr_tile<T, FEAT, BIG ? MR_ALL : MR_SMOOTH>(P, (int64_t)blockIdx.x, smem_raw);
}

}  // namespace fftz

/* The mixed-radix kernel for a feature set (FEAT_MR_*), or NULL. */
#ifdef FZ_MR_REAL
extern "C" const void *FZ_MR_GET(int feat, int big) {
  using namespace fftz;
#define FZ_MR_K(F) \
  case (F): return big ? (const void *)&fft_mr_kernel<FZ_MR_T, (F), true> : (const void *)&fft_mr_kernel<FZ_MR_T, (F), false>;
  switch (feat) { FZ_MR_K(FEAT_MR_R2C) FZ_MR_K(FEAT_MR_C2R) FZ_MR_K(FEAT_MR_RFULL) FZ_MR_K(FEAT_MR_CFULL) }
  return 0;
}
#else
extern "C" const void *FZ_MR_GET(int feat, int big) {
  using namespace fftz;
#define FZ_MR_K(F, BIG) \
  case (F): return (const void *)&fft_mr_kernel<FZ_MR_T, (F), BIG>;
  if (big) switch (feat) { FZ_MR_K(0, true) FZ_MR_K(FEAT_MR_TW4, true) }
  else switch (feat) {
      FZ_MR_K(0, false)
      FZ_MR_K(FEAT_MR_TW4, false)
      FZ_MR_K(FEAT_MR_PRE | FEAT_MR_TW4, false)                   // three-pass chirp: columns,
      FZ_MR_K(FEAT_MR_BLUE | FEAT_MR_TW4, false)                  // rows,
      FZ_MR_K(FEAT_MR_POST, false)                                // columns of the second FFT
      FZ_MR_K(FEAT_MR_PRE | FEAT_MR_POST | FEAT_MR_BLUE, false)   // one-kernel chirp
    }
  return 0;
}
#endif
