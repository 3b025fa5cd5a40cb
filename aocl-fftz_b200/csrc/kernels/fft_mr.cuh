// Mixed-radix lines in one shared-memory buffer (runtime radix list, radices
// 2..16 composites included).
//
// A line of n = R_0 R_1 ... R_{S-1} points sits in shared memory in its natural
// digit order, position sum_s d_s M_s with M_s = R_{s+1} ... R_{S-1} (plus
// mr_pad slots per step of digit 0). Stage s transforms digit s in place
// (decimation in frequency): a butterfly reads its R_s values M_s apart,
// transforms them, multiplies by W_{R_s M_s}^{k r} (r = position below digit s)
// and writes them back to the same slots, so one buffer and one barrier a
// stage are enough and the address arithmetic is paid once per butterfly. The
// first stage reads HBM, the last one writes it: output k = k_0 + R_0 (k_1 +
// R_1 (...)), so the last stage's butterflies are taken with k_0 fastest and
// every store run is contiguous. Two-sweep passes (FEAT_MR_BLUE: FFT, product with
// mid_tab, FFT) fuse the last stage, the product and the second sweep's first
// stage in registers: the second sweep runs the stages backwards (decimation
// in time), from digit-reversed to natural order, with the same twiddles.
//
// What bounds it: HBM for long batches, instruction issue otherwise; see the
// measurements beside fft_mr_kernel.
#pragma once
#include "codelets_mr.cuh"
#include "fft_common.cuh"

namespace fftz {

enum { FEAT_MR_TW4 = 1, FEAT_MR_TABS = 2, FEAT_MR_BLUE = 4 };

// x / d by the host's m = ceil(2^32 / d) (0 for d = 1); exact while x d < 2^32
__device__ __forceinline__ int mr_div(int x, uint32_t m) { return m ? (int)__umulhi((uint32_t)x, m) : x; }

// Per-tile view shared by the stages.
template <typename T> struct MrTile {
  typename Cplx<T>::type *sd;   // tpc lines, P.sstride apart
  typename Cplx<T>::type *stp;  // four-step factors W^{col nb r}: 16 per line
  const int64_t *s_in, *s_out, *s_col;
  int nl;                       // lines of the tile that exist (the last tile may be short)
};

// Four-step factor of output K of column col: col * K < tw4_n, both below
// 2^28 elements, so no reduction and 32 bits are enough.
template <typename T>
__device__ __forceinline__ typename Cplx<T>::type mr_tw4(const fftz_pass_t &P, uint32_t r) {
  typedef typename Cplx<T>::type T2;
  const int sh = 31 - __clz((int)P.tw4_l);
  return cmul(__ldg((const T2 *)P.tw4_hi + (r >> sh)), __ldg((const T2 *)P.tw4_lo + (r & ((1u << sh) - 1u))));
}

// Outputs K + r nb (r < R) of line p.
template <typename T, int R, int FEAT>
__device__ __forceinline__ void mr_store(const fftz_pass_t &P, const MrTile<T> &t, const typename Cplx<T>::type (&v)[R],
                                         int p, int K, int nb) {
  typedef typename Cplx<T>::type T2;
  const int64_t col = t.s_col[p];
  const int64_t oes = P.oes;
  T2 *g = (T2 *)P.out + t.s_out[p] + (int64_t)K * oes;
  const int64_t st = (int64_t)nb * oes;
  const bool cj = (P.flags & FFTZ_F_CONJ_OUT) != 0;
  const bool tw4 = (FEAT & FEAT_MR_TW4) || ((FEAT & FEAT_MR_TABS) && (P.flags & FFTZ_F_TW4));
  T2 w = zero2<T2>();
  if (tw4) w = mr_tw4<T>(P, (uint32_t)col * (uint32_t)K);
  const T2 *stp = t.stp + p * 16;
  if constexpr ((FEAT & FEAT_MR_TABS) != 0) {
    const int pes = (int)P.post_es, pn = P.post_n > 0 ? (int)P.post_n : 0x7fffffff;
    const int l0 = (int)(col * P.post_cs) + K * pes, ls = nb * pes;
    const bool post = (P.flags & FFTZ_F_POST_TAB) != 0, sc = (P.flags & FFTZ_F_SCALE) != 0;
#pragma unroll
    for (int r = 0; r < R; r++) {
      T2 y = v[r];
      if (tw4) y = cmul(y, r ? cmul(w, stp[r]) : w);
      if (cj) y.y = -y.y;
      const int li = l0 + r * ls;
      if (li < pn) {
        if (post) y = cmul(y, __ldg((const T2 *)P.post_tab + li));
        if (sc) {
          y.x = (T)(y.x * P.scale);
          y.y = (T)(y.y * P.scale);
        }
        g[r * st] = y;
      }
    }
  } else {
#pragma unroll
    for (int r = 0; r < R; r++) {
      T2 y = v[r];
      if (tw4) y = cmul(y, r ? cmul(w, stp[r]) : w);
      if (cj) y.y = -y.y;
      g[r * st] = y;
    }
  }
}

// Inputs e = rest + r nb (r < R) of line p.
template <typename T, int R, int FEAT>
__device__ __forceinline__ void mr_load(const fftz_pass_t &P, const MrTile<T> &t, typename Cplx<T>::type (&v)[R], int p,
                                        int rest, int nb) {
  typedef typename Cplx<T>::type T2;
  const int64_t col = t.s_col[p];
  const T2 *g = (const T2 *)P.in + t.s_in[p] + (int64_t)rest * P.ies;
  const int64_t st = (int64_t)nb * P.ies;
  const bool cj = (P.flags & FFTZ_F_CONJ_IN) != 0;
  if constexpr ((FEAT & FEAT_MR_TABS) != 0) {
    const int pes = (int)P.pre_es, pn = P.pre_n > 0 ? (int)P.pre_n : 0x7fffffff;
    const int l0 = (int)(col * P.pre_cs) + rest * pes, ls = nb * pes;
    const bool pre = (P.flags & FFTZ_F_PRE_TAB) != 0;
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int li = l0 + r * ls;
      T2 x = zero2<T2>();
      if (li < pn) {
        x = g[r * st];
        if (cj) x.y = -x.y;
        if (pre) x = cmul(x, __ldg((const T2 *)P.pre_tab + li));
      }
      v[r] = x;
    }
  } else {
#pragma unroll
    for (int r = 0; r < R; r++) {
      v[r] = g[r * st];
      if (cj) v[r].y = -v[r].y;
    }
  }
}

// item i of a boundary stage (nb butterflies a line) -> line p, position x
__device__ __forceinline__ void mr_item(const fftz_pass_t &P, int mode, int i, int nb, uint32_t mnb, int &p, int &x) {
  if (mode == 1) {
    x = mr_div(i, P.mr.mg_tpc);  // the caller skips p >= nl
    p = i - x * P.tpc;
  } else {
    p = mr_div(i, mnb);
    x = i - p * nb;
  }
}

template <typename T, int R>
__device__ __forceinline__ void mr_twiddle(const typename Cplx<T>::type *tw, typename Cplx<T>::type (&v)[R], int M,
                                           int rest) {
  // uniform row pointers plus one 32-bit lane offset
  const uint32_t o = (uint32_t)rest * (uint32_t)sizeof(*tw);
#pragma unroll
  for (int r = 1; r < R; r++) {
    const char *row = (const char *)(tw + (r - 1) * M);
    v[r] = cmul(v[r], __ldg((const typename Cplx<T>::type *)(row + o)));
  }
}

// Stage 0: HBM -> shared memory (S > 1), or HBM -> HBM (S == 1).
template <typename T, int R, int FEAT>
__device__ __forceinline__ void mr_first(const fftz_pass_t &P, const MrTile<T> &t) {
  typedef typename Cplx<T>::type T2;
  const int M = P.n / R, S0 = M + P.mr.pad;
  const T2 *tw = (const T2 *)P.tw + P.tw_off[0];
  const int total = (P.in_mode == 1 ? P.tpc : t.nl) * M;
  for (int i = threadIdx.x; i < total; i += blockDim.x) {
    int p, rest;
    mr_item(P, P.in_mode, i, M, P.mr.mg_nb[0], p, rest);
    if (p >= t.nl) continue;
    T2 v[R];
    mr_load<T, R, FEAT>(P, t, v, p, rest, M);
    Dft<R>::template apply<T, T2>(v);
    mr_twiddle<T, R>(tw, v, M, rest);
    T2 *d = t.sd + p * P.sstride + rest;
#pragma unroll
    for (int r = 0; r < R; r++) d[r * S0] = v[r];
  }
}
template <typename T, int R, int FEAT>
__device__ __forceinline__ void mr_single(const fftz_pass_t &P, const MrTile<T> &t) {
  typedef typename Cplx<T>::type T2;
  for (int p = threadIdx.x; p < t.nl; p += blockDim.x) {
    T2 v[R];
    mr_load<T, R, FEAT>(P, t, v, p, 0, 1);
    Dft<R>::template apply<T, T2>(v);
    mr_store<T, R, FEAT>(P, t, v, p, 0, 1);
  }
}

// Stage 0 < s < S - 1 in place; DIT: twiddles before the butterfly (second sweep).
template <typename T, int R, bool DIT>
__device__ __forceinline__ void mr_mid(const fftz_pass_t &P, const MrTile<T> &t, int s, int M) {
  typedef typename Cplx<T>::type T2;
  const int nb = P.n / R, total = t.nl * nb, step = M * (R - 1), pad = P.mr.pad;
  const uint32_t mnb = P.mr.mg_nb[s], mM = P.mr.mg_m[s], mB = P.mr.mg_b[s];
  const T2 *tw = (const T2 *)P.tw + P.tw_off[s];
  for (int i = threadIdx.x; i < total; i += blockDim.x) {
    const int p = mr_div(i, mnb);
    const int j = i - p * nb;
    const int b = mr_div(j, mM);
    const int rest = j - b * M;
    T2 *d = t.sd + p * P.sstride + j + b * step + mr_div(b, mB) * pad;
    T2 v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = d[r * M];
    if (DIT) mr_twiddle<T, R>(tw, v, M, rest);
    Dft<R>::template apply<T, T2>(v);
    if (!DIT) mr_twiddle<T, R>(tw, v, M, rest);
#pragma unroll
    for (int r = 0; r < R; r++) d[r * M] = v[r];
  }
}

// Slot of the last stage's butterfly K = k_0 + R_0 (k_1 + R_1 (...)).
__device__ __forceinline__ int mr_slot(const fftz_pass_t &P, int K) {
  const int S0 = P.mr.m[0] + P.mr.pad, S = P.nstages;
  if (S == 2) return K * S0;
  int q = mr_div(K, P.mr.mg_r[0]);
  int o = (K - q * P.radix[0]) * S0;
  for (int s = 1; s < S - 2; s++) {
    const int x = mr_div(q, P.mr.mg_r[s]);
    o += (q - x * P.radix[s]) * P.mr.m[s];
    q = x;
  }
  return o + q * P.mr.m[S - 2];
}

// Last stage: shared memory -> HBM, butterflies in output order.
template <typename T, int R, int FEAT>
__device__ __forceinline__ void mr_last(const fftz_pass_t &P, const MrTile<T> &t, int s) {
  typedef typename Cplx<T>::type T2;
  const int nb = P.n / R, total = (P.out_mode == 1 ? P.tpc : t.nl) * nb;
  for (int i = threadIdx.x; i < total; i += blockDim.x) {
    int p, K;
    mr_item(P, P.out_mode, i, nb, P.mr.mg_nb[s], p, K);
    if (p >= t.nl) continue;
    const T2 *d = t.sd + p * P.sstride + mr_slot(P, K);
    T2 v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = d[r];
    Dft<R>::template apply<T, T2>(v);
    mr_store<T, R, FEAT>(P, t, v, p, K, nb);
  }
}

// Two-sweep passes: last stage of the first FFT, v = conj(v) * mid_tab, first
// stage of the second FFT, in place.
template <typename T, int R>
__device__ __forceinline__ void mr_product(const fftz_pass_t &P, const MrTile<T> &t, int s) {
  typedef typename Cplx<T>::type T2;
  const int nb = P.n / R, total = t.nl * nb;
  for (int i = threadIdx.x; i < total; i += blockDim.x) {
    const int p = mr_div(i, P.mr.mg_nb[s]);
    const int K = i - p * nb;
    T2 *d = t.sd + p * P.sstride + mr_slot(P, K);
    T2 v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = d[r];
    Dft<R>::template apply<T, T2>(v);
    const T2 *mt = (const T2 *)P.mid_tab + t.s_col[p] * P.mid_cs + K;
#pragma unroll
    for (int r = 0; r < R; r++) {
      T2 x = v[r];
      x.y = -x.y;
      v[r] = cmul(x, __ldg(mt + r * nb));
    }
    Dft<R>::template apply<T, T2>(v);
#pragma unroll
    for (int r = 0; r < R; r++) d[r] = v[r];
  }
}

// Second sweep's last stage (digit 0): shared memory -> HBM, natural order.
template <typename T, int R, int FEAT>
__device__ __forceinline__ void mr_dit_last(const fftz_pass_t &P, const MrTile<T> &t) {
  typedef typename Cplx<T>::type T2;
  const int M = P.n / R, S0 = M + P.mr.pad;
  const T2 *tw = (const T2 *)P.tw + P.tw_off[0];
  const int total = (P.out_mode == 1 ? P.tpc : t.nl) * M;
  for (int i = threadIdx.x; i < total; i += blockDim.x) {
    int p, rest;
    mr_item(P, P.out_mode, i, M, P.mr.mg_nb[0], p, rest);
    if (p >= t.nl) continue;
    const T2 *d = t.sd + p * P.sstride + rest;
    T2 v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = d[r * S0];
    mr_twiddle<T, R>(tw, v, M, rest);
    Dft<R>::template apply<T, T2>(v);
    mr_store<T, R, FEAT>(P, t, v, p, rest, M);
  }
}

// BIG: radices 11 and 13 too (their butterflies hold more live values).
#define FZ_MR_SWITCH(R_, BIG, CALL)                       \
  switch (R_) {                                           \
    case 2: { constexpr int R = 2; CALL; } break;         \
    case 3: { constexpr int R = 3; CALL; } break;         \
    case 4: { constexpr int R = 4; CALL; } break;         \
    case 5: { constexpr int R = 5; CALL; } break;         \
    case 6: { constexpr int R = 6; CALL; } break;         \
    case 7: { constexpr int R = 7; CALL; } break;         \
    case 8: { constexpr int R = 8; CALL; } break;         \
    case 9: { constexpr int R = 9; CALL; } break;         \
    case 10: { constexpr int R = 10; CALL; } break;       \
    case 11: if constexpr (BIG) { constexpr int R = 11; CALL; } break; \
    case 12: { constexpr int R = 12; CALL; } break;       \
    case 13: if constexpr (BIG) { constexpr int R = 13; CALL; } break; \
    case 14: { constexpr int R = 14; CALL; } break;       \
    case 15: { constexpr int R = 15; CALL; } break;       \
    case 16: { constexpr int R = 16; CALL; } break;       \
  }

// One CTA-worth of a pass: transforms [blk * tpc, (blk + 1) * tpc).
template <typename T, int FEAT, bool BIG>
__device__ __forceinline__ void mr_tile(const fftz_pass_t &P, int64_t blk, unsigned char *smem_raw) {
  typedef typename Cplx<T>::type T2;
  constexpr bool TW4 = (FEAT & (FEAT_MR_TW4 | FEAT_MR_TABS)) != 0;
  MrTile<T> t;
  t.sd = (T2 *)smem_raw;
  t.stp = t.sd + (size_t)P.tpc * P.sstride;
  int64_t *s_in = (int64_t *)(t.stp + ((P.flags & FFTZ_F_TW4) ? 16 * P.tpc : 0));
  int64_t *s_out = s_in + P.tpc, *s_col = s_out + P.tpc;
  t.s_in = s_in;
  t.s_out = s_out;
  t.s_col = s_col;
  t.nl = P.ntf - blk * P.tpc < P.tpc ? (int)(P.ntf - blk * P.tpc) : P.tpc;
  for (int p = threadIdx.x; p < P.tpc; p += blockDim.x)
    batch_offsets(P, blk * P.tpc + p, s_in + p, s_out + p, s_col + p);
  __syncthreads();
  const int S = P.nstages;
  if (TW4 && (P.flags & FFTZ_F_TW4)) {
    // W^{col nb r} of the final butterflies (outputs nb apart), formed per line
    const int Rl = (FEAT & FEAT_MR_BLUE) ? P.radix[0] : P.radix[S - 1];
    const int nb = P.n / Rl;
    for (int i = threadIdx.x; i < 16 * P.tpc; i += blockDim.x) {
      const int p = i >> 4, r = i & 15;
      const int64_t col = s_col[p];
      if (col >= 0 && r < Rl) t.stp[i] = mr_tw4<T>(P, (uint32_t)col * (uint32_t)(nb * r));
    }
    if (S == 1) __syncthreads();
  }
  if (S == 1) {
    if constexpr ((FEAT & FEAT_MR_BLUE) == 0) FZ_MR_SWITCH(P.radix[0], BIG, (mr_single<T, R, FEAT>(P, t)));
    return;
  }
  FZ_MR_SWITCH(P.radix[0], BIG, (mr_first<T, R, FEAT>(P, t)));
  __syncthreads();
  for (int s = 1; s < S - 1; s++) {
    const int M = P.mr.m[s];
    FZ_MR_SWITCH(P.radix[s], BIG, (mr_mid<T, R, false>(P, t, s, M)));
    __syncthreads();
  }
  if constexpr ((FEAT & FEAT_MR_BLUE) != 0) {
    FZ_MR_SWITCH(P.radix[S - 1], BIG, (mr_product<T, R>(P, t, S - 1)));
    __syncthreads();
    for (int s = S - 2; s > 0; s--) {
      const int M = P.mr.m[s];
      FZ_MR_SWITCH(P.radix[s], BIG, (mr_mid<T, R, true>(P, t, s, M)));
      __syncthreads();
    }
    FZ_MR_SWITCH(P.radix[0], BIG, (mr_dit_last<T, R, FEAT>(P, t)));
  } else {
    FZ_MR_SWITCH(P.radix[S - 1], BIG, (mr_last<T, R, FEAT>(P, t, S - 1)));
  }
}

}  // namespace fftz
