#pragma once
// Shared-memory FFT kernel for sm_100a (runtime radix list, every element kind).
//
// One CTA holds tf_per_cta whole transforms of length n in shared memory. The
// transform is a sequence of Stockham radix-R stages (R in {2,3,4,5,7,8,11,13,16},
// butterflies from codelets.cuh): each thread pulls its butterflies' R inputs
// at stride n/R, multiplies by the stage twiddles W_{Ns*R}^{k*r}, runs the
// register DFT and writes the R outputs at stride Ns into the auto-sorted
// position, so the result lands in natural order without a bit-reversal pass.
//
// Every element kind goes through a load and a store phase with a thread map of
// its own: lanes along elements (mode 0) or along neighbouring transforms (mode 1),
// coalesced for rows (unit element stride) and columns (unit batch stride).
//
// The backward transform is conj(FFT(conj(x))): conjugation is fused into the
// load and the store, so only forward codelets and forward twiddles exist.
// The reference counterpart of this kernel is the pow2 iterative solver
// (core/solvers/complex/pow2_iterative_solver_dft.c:275-380) together with the
// radix and twiddle codelets it calls (core/kernels/dft/c2c, tw_c2c_fwd/bwd).
#include <cuda_runtime.h>
#include <stdint.h>

#include "fft_common.cuh"

namespace fftz {

// One Stockham stage of radix R, in shared memory, over the transform this thread
// is mapped to.
template <typename T, int R>
__device__ __noinline__ void run_stage(const fftz_pass_t &P, typename Cplx<T>::type *sdata, int s, int Ns) {
  typedef typename Cplx<T>::type T2;
  constexpr int NB = kMaxE / R;
  constexpr int SH = Cplx<T>::PADSH;
  const int n = P.n;
  const int nb = n / R;
  const int p = threadIdx.x / P.tpt, j = threadIdx.x - p * P.tpt;
  T2 *sd = sdata + (size_t)p * P.sstride;
  T2 v[NB][R];
#pragma unroll
  for (int q = 0; q < NB; q++) {
    const int b = j + q * P.tpt;
    if (b < nb) {
#pragma unroll
      for (int r = 0; r < R; r++) v[q][r] = sd[phys<SH>(b + r * nb)];
    }
  }
  __syncthreads();
  const T2 *tw = (const T2 *)P.tw + P.tw_off[s];
#pragma unroll
  for (int q = 0; q < NB; q++) {
    const int b = j + q * P.tpt;
    if (b < nb) {
      const int k = (int)((unsigned)b % (unsigned)Ns);
      if (Ns > 1) {
#pragma unroll
        for (int r = 1; r < R; r++) v[q][r] = cmul(v[q][r], __ldg(tw + (r - 1) * Ns + k));
      }
      Dft<R>::template apply<T, T2>(v[q]);
      const int d0 = (b - k) * R + k;
#pragma unroll
      for (int r = 0; r < R; r++) sd[phys<SH>(d0 + r * Ns)] = v[q][r];
    }
  }
  __syncthreads();
}

template <typename T>
__device__ __forceinline__ void stage_dispatch(const fftz_pass_t &P, typename Cplx<T>::type *sdata, int s, int Ns) {
  switch (P.radix[s]) {
    case 2: run_stage<T, 2>(P, sdata, s, Ns); break;
    case 3: run_stage<T, 3>(P, sdata, s, Ns); break;
    case 4: run_stage<T, 4>(P, sdata, s, Ns); break;
    case 5: run_stage<T, 5>(P, sdata, s, Ns); break;
    case 7: run_stage<T, 7>(P, sdata, s, Ns); break;
    case 8: run_stage<T, 8>(P, sdata, s, Ns); break;
    case 11: run_stage<T, 11>(P, sdata, s, Ns); break;
    case 13: run_stage<T, 13>(P, sdata, s, Ns); break;
    default: run_stage<T, 16>(P, sdata, s, Ns); break;
  }
}

// Global -> shared load phase for every element kind.
template <typename T>
__device__ void load_phase(const fftz_pass_t &P, typename Cplx<T>::type *sdata, const int64_t *s_in,
                           const int64_t *s_col) {
  typedef typename Cplx<T>::type T2;
  constexpr int SH = Cplx<T>::PADSH;
  const int total = P.tpc * P.nload;
  const int f = P.flags;
  for (int i = threadIdx.x; i < total; i += blockDim.x) {
    int p, e;
    if (P.in_mode == 0) {
      p = i / P.nload;
      e = i - p * P.nload;
    } else {
      e = i / P.tpc;
      p = i - e * P.tpc;
    }
    const int64_t col = s_col[p];
    T2 x = zero2<T2>();
    if (col >= 0) {
      switch (P.in_kind) {
        case FFTZ_IN_COMPLEX: {
          x = ((const T2 *)P.in)[s_in[p] + (int64_t)e * P.ies];
          if (f & FFTZ_F_CONJ_IN) x.y = -x.y;
          break;
        }
        case FFTZ_IN_REAL_PAIRS: {
          const T *g = (const T *)P.in + s_in[p];
          x.x = g[(int64_t)(2 * e) * P.ies];
          x.y = g[(int64_t)(2 * e + 1) * P.ies];
          if (f & FFTZ_F_CONJ_IN) x.y = -x.y;
          break;
        }
        case FFTZ_IN_REAL: {
          const T *g = (const T *)P.in + s_in[p];
          x.x = g[(int64_t)e * P.ies];
          break;
        }
        case FFTZ_IN_HERM_FULL: {
          const int half = P.n / 2;
          const int idx = (e <= half) ? e : P.n - e;
          x = ((const T2 *)P.in)[s_in[p] + (int64_t)idx * P.ies];
          if (e > half) x.y = -x.y;
          if (f & FFTZ_F_CONJ_IN) x.y = -x.y;
          break;
        }
        default: {  // FFTZ_IN_HERM_SEPARATE: raw X[e], e <= M
          x = ((const T2 *)P.in)[s_in[p] + (int64_t)e * P.ies];
          break;
        }
      }
    }
    sdata[(size_t)p * P.sstride + phys<SH>(e)] = x;
  }
  __syncthreads();
  if (P.in_kind == FFTZ_IN_HERM_SEPARATE) {
    // 2 Z[k] = (X_k + conj X_{M-k}) + i e^{+2 pi i k/2M} (X_k - conj X_{M-k}); the
    // conjugation of the backward transform is applied here as well.
    const int M = P.n;
    const int npairs = M / 2 + 1;
    const T2 *rtw = (const T2 *)P.rtw;
    for (int i = threadIdx.x; i < P.tpc * npairs; i += blockDim.x) {
      const int p = i / npairs;
      const int k = i - p * npairs;
      T2 *sd = sdata + (size_t)p * P.sstride;
      const int km = (k == 0) ? M : M - k;
      const T2 xk = sd[phys<SH>(k)];
      const T2 xm = sd[phys<SH>(km)];
      const T2 w = __ldg(rtw + k);  // e^{-2 pi i k / 2M}
      // E = conj(w) applied to D = X_k - conj(X_m)
      const T dr = xk.x - xm.x, di = xk.y + xm.y;
      const T er = w.x * dr + w.y * di, ei = w.x * di - w.y * dr;  // conj(w) * D
      T2 zk;
      zk.x = (xk.x + xm.x) - ei;
      zk.y = -((xk.y - xm.y) + er);  // conjugated
      if (k != 0 && km != k) {
        // Z[M-k]: S' = X_m + conj X_k, D' = X_m - conj X_k, twiddle conj(w_{M-k}) = -w
        const T dr2 = xm.x - xk.x, di2 = xm.y + xk.y;
        const T er2 = -(w.x * dr2 - w.y * di2), ei2 = -(w.x * di2 + w.y * dr2);  // -w * D'
        T2 zm;
        zm.x = (xm.x + xk.x) - ei2;
        zm.y = -((xm.y - xk.y) + er2);
        sd[phys<SH>(km)] = zm;
      }
      sd[phys<SH>(k)] = zk;
    }
    __syncthreads();
  }
}

// Shared -> global store phase for every element kind.
template <typename T>
__device__ void store_phase(const fftz_pass_t &P, typename Cplx<T>::type *sdata, const int64_t *s_out,
                            const int64_t *s_col) {
  typedef typename Cplx<T>::type T2;
  constexpr int SH = Cplx<T>::PADSH;
  const int total = P.tpc * P.nstore;
  for (int i = threadIdx.x; i < total; i += blockDim.x) {
    int p, k;
    if (P.out_mode == 0) {
      p = i / P.nstore;
      k = i - p * P.nstore;
    } else {
      k = i / P.tpc;
      p = i - k * P.tpc;
    }
    const int64_t col = s_col[p];
    if (col < 0) continue;
    const T2 *sd = sdata + (size_t)p * P.sstride;
    switch (P.out_kind) {
      case FFTZ_OUT_COMPLEX:
      case FFTZ_OUT_HALF:
        store_complex<T>(P, sd[phys<SH>(k)], k, col, s_out[p]);
        break;
      case FFTZ_OUT_HALF_RECOMBINE: {
        // X_k = (Z_k + conj Z_{M-k})/2 - (i/2) W^k (Z_k - conj Z_{M-k}), Z_M = Z_0
        const int M = P.n;
        const T2 zk = sd[phys<SH>(k == M ? 0 : k)];
        const T2 zm = sd[phys<SH>(k == 0 ? 0 : M - k)];
        const T2 w = __ldg((const T2 *)P.rtw + k);
        const T er = (T)0.5 * (zk.x + zm.x), ei = (T)0.5 * (zk.y - zm.y);
        const T orr = (T)0.5 * (zk.y + zm.y), oi = (T)0.5 * (zm.x - zk.x);
        T2 x;
        x.x = er + (w.x * orr - w.y * oi);
        x.y = ei + (w.x * oi + w.y * orr);
        store_complex<T>(P, x, k, col, s_out[p]);
        break;
      }
      case FFTZ_OUT_REAL_PAIRS: {
        T2 v = sd[phys<SH>(k)];
        if (P.flags & FFTZ_F_CONJ_OUT) v.y = -v.y;
        T *g = (T *)P.out + s_out[p];
        g[(int64_t)(2 * k) * P.oes] = v.x;
        g[(int64_t)(2 * k + 1) * P.oes] = v.y;
        break;
      }
      default: {  // FFTZ_OUT_REAL
        T *g = (T *)P.out + s_out[p];
        g[(int64_t)k * P.oes] = sd[phys<SH>(k)].x;
        break;
      }
    }
  }
}

// One CTA-worth of a pass: transforms [blk * tpc, (blk + 1) * tpc).
template <typename T>
__device__ __forceinline__ void generic_tile(const fftz_pass_t &P, int64_t blk, unsigned char *smem_raw) {
  typedef typename Cplx<T>::type T2;
  T2 *sdata = (T2 *)smem_raw;
  int64_t *s_in = (int64_t *)(sdata + (size_t)P.tpc * P.sstride);
  int64_t *s_out = s_in + P.tpc;
  int64_t *s_col = s_out + P.tpc;
  const int64_t tf0 = blk * P.tpc;
  for (int p = threadIdx.x; p < P.tpc; p += blockDim.x) batch_offsets(P, tf0 + p, s_in + p, s_out + p, s_col + p);
  pdl_begin();
  __syncthreads();

  load_phase<T>(P, sdata, s_in, s_col);
  int Ns = 1;
  for (int s = 0; s < P.nstages; s++) {
    stage_dispatch<T>(P, sdata, s, Ns);
    Ns *= P.radix[s];
  }
  store_phase<T>(P, sdata, s_out, s_col);
}

// float: at most 80 registers (3 CTAs of 256 threads per SM) -- measured on
// B200 1.6-2.8x faster than the unbounded build for mixed-radix lines
// (n = 1000 ... 44100); double keeps the plain thread bound (a minimum-blocks
// bound of 1 measured 1.7x slower for it)
template <typename T>
__global__ void __launch_bounds__(256, 3) fft_smem_kernel_occ3(const __grid_constant__ fftz_pass_t P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  generic_tile<T>(P, (int64_t)blockIdx.x, smem_raw);
}

template <typename T>
__global__ void __launch_bounds__(256) fft_smem_kernel(const __grid_constant__ fftz_pass_t P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  generic_tile<T>(P, (int64_t)blockIdx.x, smem_raw);
}

}  // namespace fftz

