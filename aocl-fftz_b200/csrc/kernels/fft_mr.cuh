// Mixed-radix lines in one shared-memory buffer (runtime radix list, radices
// 2..16 composites included).
//
// A line of n = R_0 R_1 ... R_{S-1} points sits in shared memory in its natural
// digit order, position sum_s d_s M_s with M_s = R_{s+1} ... R_{S-1} (plus
// mr.pad slots per step of digit 0). Stage s transforms digit s in place
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
// What a stage reads of its pass is copied to locals before its loop: in the
// ragged executor the pass lies in shared memory, where the loop's own stores
// would force every field to be read again for each butterfly.
//
// What bounds it: HBM for long batches, instruction issue otherwise; see the
// measurements beside fft_mr_kernel.
#pragma once
#include "codelets_mr.cuh"
#include "fft_common.cuh"

namespace fftz {

// Features of a pass, all compile-time: a form for every combination the planner
// makes. (One form with run-time flags for the table passes spent most of its time
// waiting for instructions: 11 of 19 stall cycles an instruction in a 256-point
// chirp pass.) TW4: output k of column c times W_{tw4_n}^{c k}. PRE / POST: bound
// and table product on the load / store side. BLUE: two sweeps around mid_tab.
// R2C / C2R: real lines of 2 n points packed as n complex ones, with the Hermitian
// recombination in the last stage's registers / the separation in the first
// stage's. RFULL / CFULL: real lines of n points as n complex ones (odd lengths).
enum {
  FEAT_MR_TW4 = 1, FEAT_MR_PRE = 2, FEAT_MR_POST = 4, FEAT_MR_BLUE = 8,
  FEAT_MR_R2C = 16, FEAT_MR_C2R = 32, FEAT_MR_RFULL = 64, FEAT_MR_CFULL = 128
};

// x / d by the host's m = ceil(2^32 / d) (0 for d = 1); exact while x d < 2^32
__device__ __forceinline__ int mr_div(int x, uint32_t m) { return m ? (int)__umulhi((uint32_t)x, m) : x; }

// Offset of a line on one HBM side, and its column.
struct __align__(16) MrLine {
  int64_t off, col;
};

// A tile's shared memory: tpc lines P.sstride apart, the four-step factors
// W^{col nb r} (16 per line), the lines' places on the input and output side, a
// copy of the stage twiddles in the executor (otherwise they are read through L1);
// nl of the lines exist (the last tile of a pass may be short).
template <typename T> struct MrTile {
  typename Cplx<T>::type *sd, *stp;
  const MrLine *in, *out;
  int nl;
  bool has_tw;                       // tw holds the stage twiddles
  const typename Cplx<T>::type *tw;  // (a shared-memory array: never NULL, since the
                                     // compiler's shared-memory address of NULL is not)
};

// One component of a complex product of factors held as sums of two doubles
// (hi, then what the rounding to it left): a.x b.x + a.y b.y, rounded once.
__device__ __forceinline__ double mr_dot2(double ax, double bx, double ay, double by, double low) {
  const double p = __dmul_rn(ax, bx), q = __dmul_rn(ay, by), s = __dadd_rn(p, q), z = __dsub_rn(s, p);
  const double left = __dadd_rn(__dsub_rn(p, __dsub_rn(s, z)), __dsub_rn(q, z));  // p + q - s
  return s + (left + (fma(ax, bx, -p) + fma(ay, by, -q) + low));
}

// W_{tw4_n}^r from the two factor tables. A final factor is the product of two of
// these (mr_store, mr_steps), so each is rounded to T once: float passes hold the
// tables in double, double passes each entry as a sum of two. (From tables and
// products in T the error of a 500000-point float line was 4%, of a 117649-point
// double line 3% above that of one table product an output.) r = column * output <
// tw4_n < 2^32 (fz_tw4_tables refuses more): no reduction.
template <typename T2> struct MrTw4 {
  const double2 *hi, *lo;
  int sh;
  __device__ __forceinline__ T2 operator()(uint32_t r) const {
    T2 f;
    if constexpr (sizeof(T2) == sizeof(double2)) {
      const double2 *a = hi + 2 * (r >> sh), *b = lo + 2 * (r & ((1u << sh) - 1u));
      const double2 ah = __ldg(a), al = __ldg(a + 1), bh = __ldg(b), bl = __ldg(b + 1);
      f.x = mr_dot2(ah.x, bh.x, -ah.y, bh.y, ah.x * bl.x - ah.y * bl.y + (al.x * bh.x - al.y * bh.y));
      f.y = mr_dot2(ah.x, bh.y, ah.y, bh.x, ah.x * bl.y + ah.y * bl.x + (al.x * bh.y + al.y * bh.x));
    } else {
      const double2 w = cmul(__ldg(hi + (r >> sh)), __ldg(lo + (r & ((1u << sh) - 1u))));
      f.x = (float)w.x;
      f.y = (float)w.y;
    }
    return f;
  }
};

template <typename T2> __device__ __forceinline__ MrTw4<T2> mr_tw4(const fftz_pass_t &P) {
  return MrTw4<T2>{(const double2 *)P.tw4_hi, (const double2 *)P.tw4_lo, 31 - __clz((int)P.tw4_l)};
}

// Table factors in flight beside R values: as many as the registers hold (float
// 64, double 128).
template <int R> __host__ __device__ constexpr int mr_chunk() { return R <= 8 ? R : R <= 12 ? 6 : 4; }

// v[r] *= tab[min(l0 + r ls, last)], C factors in flight
template <typename T2, int R>
__device__ __forceinline__ void mr_table(T2 (&v)[R], const T2 *tab, int l0, int ls, int last) {
  constexpr int C = mr_chunk<R>();
#pragma unroll
  for (int q = 0; q < R; q += C) {
    T2 w[C];
#pragma unroll
    for (int r = q; r < R && r < q + C; r++) w[r - q] = __ldg(tab + min(l0 + r * ls, last));
#pragma unroll
    for (int r = q; r < R && r < q + C; r++) v[r] = cmul(v[r], w[r - q]);
  }
}

// Outputs K + r nb (r < R) of line p (v is used up).
template <typename T, int R, int FEAT>
__device__ __forceinline__ void mr_store(const fftz_pass_t &P, const MrTile<T> &t, typename Cplx<T>::type (&v)[R], int p,
                                         int K, int nb) {
  typedef typename Cplx<T>::type T2;
  const MrLine L = t.out[p];
  const int64_t oes = P.oes;
  if constexpr ((FEAT & FEAT_MR_C2R) != 0) {
    // value k is the pair (out[2k], out[2k + 1]), conjugated
    T *x = (T *)P.out + L.off;
    if (oes == 1 && ((uintptr_t)x & (sizeof(T2) - 1)) == 0) {
      T2 *g = (T2 *)x + K;
#pragma unroll
      for (int r = 0; r < R; r++) {
        v[r].y = -v[r].y;
        g[r * nb] = v[r];
      }
    } else {
#pragma unroll
      for (int r = 0; r < R; r++) {
        T *g = x + 2 * (int64_t)(K + r * nb) * oes;
        g[0] = v[r].x;
        g[oes] = -v[r].y;
      }
    }
    return;
  }
  if constexpr ((FEAT & FEAT_MR_CFULL) != 0) {
    T *g = (T *)P.out + L.off + (int64_t)K * oes;
#pragma unroll
    for (int r = 0; r < R; r++) g[(int64_t)r * nb * oes] = v[r].x;
    return;
  }
  T2 *g = (T2 *)P.out + L.off + (int64_t)K * oes;
  const int64_t st = (int64_t)nb * oes;
  if constexpr ((FEAT & FEAT_MR_RFULL) != 0) {
    const int half = P.n / 2;
#pragma unroll
    for (int r = 0; r < R; r++)
      if (K + r * nb <= half) g[r * st] = v[r];
    return;
  }
  if constexpr ((FEAT & FEAT_MR_TW4) != 0) {
    const T2 w = mr_tw4<T2>(P)((uint32_t)L.col * (uint32_t)K);
    const T2 *stp = t.stp + p * 16;
    v[0] = cmul(v[0], w);
#pragma unroll
    for (int r = 1; r < R; r++) v[r] = cmul(v[r], cmul(w, stp[r]));
  }
  if (P.flags & FFTZ_F_CONJ_OUT) {
#pragma unroll
    for (int r = 0; r < R; r++) v[r].y = -v[r].y;
  }
  if constexpr ((FEAT & FEAT_MR_POST) != 0) {
    const int pes = (int)P.post_es, pn = (int)P.post_n;
    const int l0 = (int)(L.col * P.post_cs) + K * pes, ls = nb * pes;
    mr_table<T2, R>(v, (const T2 *)P.post_tab, l0, ls, pn - 1);
#pragma unroll
    for (int r = 0; r < R; r++)
      if (l0 + r * ls < pn) g[r * st] = v[r];
  } else {
#pragma unroll
    for (int r = 0; r < R; r++) g[r * st] = v[r];
  }
}

// Inputs e = rest + r nb (r < R) of line p.
template <typename T, int R, int FEAT>
__device__ __forceinline__ void mr_load(const fftz_pass_t &P, const MrTile<T> &t, typename Cplx<T>::type (&v)[R], int p,
                                        int rest, int nb) {
  typedef typename Cplx<T>::type T2;
  const MrLine L = t.in[p];
  const int64_t ies = P.ies;
  if constexpr ((FEAT & FEAT_MR_R2C) != 0) {
    // value e is the pair (in[2e], in[2e + 1])
    const T *x = (const T *)P.in + L.off;
    if (ies == 1 && ((uintptr_t)x & (sizeof(T2) - 1)) == 0) {
      const T2 *g = (const T2 *)x + rest;
#pragma unroll
      for (int r = 0; r < R; r++) v[r] = g[r * nb];
    } else {
#pragma unroll
      for (int r = 0; r < R; r++) {
        const T *g = x + 2 * (int64_t)(rest + r * nb) * ies;
        v[r].x = g[0];
        v[r].y = g[ies];
      }
    }
    return;
  }
  if constexpr ((FEAT & FEAT_MR_RFULL) != 0) {
    const T *g = (const T *)P.in + L.off + (int64_t)rest * ies;
#pragma unroll
    for (int r = 0; r < R; r++) {
      v[r].x = g[(int64_t)r * nb * ies];
      v[r].y = 0;
    }
    return;
  }
  if constexpr ((FEAT & FEAT_MR_CFULL) != 0) {
    // bins above n / 2 are the conjugates of those below; the backward
    // transform's conjugation included
    const T2 *g = (const T2 *)P.in + L.off;
    const int n = P.n;
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int e = rest + r * nb;
      const bool up = 2 * e > n;
      v[r] = g[(int64_t)(up ? n - e : e) * ies];
      if (!up) v[r].y = -v[r].y;
    }
    return;
  }
  const T2 *g = (const T2 *)P.in + L.off + (int64_t)rest * ies;
  const int64_t st = (int64_t)nb * ies;
  const bool cj = (P.flags & FFTZ_F_CONJ_IN) != 0;
  if constexpr ((FEAT & FEAT_MR_PRE) != 0) {
    const int pes = (int)P.pre_es, pn = (int)P.pre_n;
    const int l0 = (int)(L.col * P.pre_cs) + rest * pes, ls = nb * pes;
    // every load first, then the table factors, at an index clamped to the table
#pragma unroll
    for (int r = 0; r < R; r++) {
      v[r] = zero2<T2>();
      if (l0 + r * ls < pn) v[r] = g[r * st];
    }
    if (cj) {
#pragma unroll
      for (int r = 0; r < R; r++) v[r].y = -v[r].y;
    }
    mr_table<T2, R>(v, (const T2 *)P.pre_tab, l0, ls, pn - 1);
  } else {
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = g[r * st];
    if (cj) {
#pragma unroll
      for (int r = 0; r < R; r++) v[r].y = -v[r].y;
    }
  }
}

// item i of a boundary stage (nb butterflies a line) -> line p, position x;
// with lanes along lines (mode 1) items of lines p >= nl are skipped
struct MrItems {
  int mode, tpc, nb, total;
  uint32_t mg;
  __device__ __forceinline__ MrItems(const fftz_pass_t &P, int mode_, int nb_, uint32_t mnb, int nl)
      : mode(mode_), tpc(P.tpc), nb(nb_) {
    total = (mode == 1 ? tpc : nl) * nb;
    mg = mode == 1 ? P.mr.mg_tpc : mnb;
  }
  __device__ __forceinline__ void at(int i, int &p, int &x) const {
    const int q = mr_div(i, mg);
    if (mode == 1) {
      x = q;
      p = i - q * tpc;
    } else {
      p = q;
      x = i - q * nb;
    }
  }
};

// v[r] *= tw[(r - 1) M + rest], from the table's shared-memory copy sh where the
// tile has one.
template <typename T, int R>
__device__ __forceinline__ void mr_twiddle(const typename Cplx<T>::type *tw, const typename Cplx<T>::type *sh, bool has,
                                           typename Cplx<T>::type (&v)[R], int M, int rest) {
  typedef typename Cplx<T>::type T2;
  if (has) {
#pragma unroll
    for (int r = 1; r < R; r++) v[r] = cmul(v[r], sh[(r - 1) * M + rest]);
    return;
  }
  // uniform row pointers plus one 32-bit lane offset
  const uint32_t o = (uint32_t)rest * (uint32_t)sizeof(T2);
#pragma unroll
  for (int r = 1; r < R; r++) {
    const char *row = (const char *)(tw + (r - 1) * M);
    v[r] = cmul(v[r], __ldg((const T2 *)(row + o)));
  }
}

// Stage 0: HBM -> shared memory (S > 1), or HBM -> HBM (S == 1).
template <typename T, int R, int FEAT>
__device__ __forceinline__ void mr_first(const fftz_pass_t &P, const MrTile<T> &t, const fftz_mr_stage_t &st) {
  typedef typename Cplx<T>::type T2;
  const int M = st.m, S0 = M + P.mr.pad, sst = P.sstride;
  const T2 *tw = (const T2 *)P.tw + st.tw, *sh = t.tw + st.tw;
  const MrItems it(P, P.in_mode, M, st.mg_nb, t.nl);
  for (int i = threadIdx.x; i < it.total; i += blockDim.x) {
    int p, rest;
    it.at(i, p, rest);
    if (p >= t.nl) continue;
    T2 v[R];
    mr_load<T, R, FEAT>(P, t, v, p, rest, M);
    Dft<R>::template apply<T, T2>(v);
    mr_twiddle<T, R>(tw, sh, t.has_tw, v, M, rest);
    T2 *d = t.sd + p * sst + rest;
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
__device__ __forceinline__ void mr_mid(const fftz_pass_t &P, const MrTile<T> &t, const fftz_mr_stage_t &st) {
  typedef typename Cplx<T>::type T2;
  const int M = st.m, nb = st.nb, total = t.nl * nb, step = M * (R - 1), pad = P.mr.pad, sst = P.sstride;
  const uint32_t mnb = st.mg_nb, mM = st.mg_m, mB = st.mg_b;
  const T2 *tw = (const T2 *)P.tw + st.tw, *sh = t.tw + st.tw;
  for (int i = threadIdx.x; i < total; i += blockDim.x) {
    const int p = mr_div(i, mnb);
    const int j = i - p * nb;
    const int b = mr_div(j, mM);
    const int rest = j - b * M;
    T2 *d = t.sd + p * sst + j + b * step + mr_div(b, mB) * pad;
    T2 v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = d[r * M];
    if (DIT) mr_twiddle<T, R>(tw, sh, t.has_tw, v, M, rest);
    Dft<R>::template apply<T, T2>(v);
    if (!DIT) mr_twiddle<T, R>(tw, sh, t.has_tw, v, M, rest);
#pragma unroll
    for (int r = 0; r < R; r++) d[r * M] = v[r];
  }
}

// Slot of the last stage's butterfly K = k_0 + R_0 (k_1 + R_1 (...)).
__device__ __forceinline__ int mr_slot(const fftz_pass_t &P, int S, int S0, int K) {
  if (S == 2) return K * S0;
  int q = mr_div(K, P.mr.st[0].mg_r);
  int o = (K - q * P.mr.st[0].r) * S0;
  for (int s = 1; s < S - 2; s++) {
    const int x = mr_div(q, P.mr.st[s].mg_r);
    o += (q - x * P.mr.st[s].r) * P.mr.st[s].m;
    q = x;
  }
  return o + q * P.mr.st[S - 2].m;
}

// Last stage: shared memory -> HBM, butterflies in output order.
template <typename T, int R, int FEAT>
__device__ __forceinline__ void mr_last(const fftz_pass_t &P, const MrTile<T> &t, const fftz_mr_stage_t &st) {
  typedef typename Cplx<T>::type T2;
  const int nb = st.nb, S = P.nstages, S0 = P.mr.st[0].m + P.mr.pad, sst = P.sstride;
  const MrItems it(P, P.out_mode, nb, st.mg_nb, t.nl);
  for (int i = threadIdx.x; i < it.total; i += blockDim.x) {
    int p, K;
    it.at(i, p, K);
    if (p >= t.nl) continue;
    const T2 *d = t.sd + p * sst + mr_slot(P, S, S0, K);
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
__device__ __forceinline__ void mr_product(const fftz_pass_t &P, const MrTile<T> &t, const fftz_mr_stage_t &st) {
  typedef typename Cplx<T>::type T2;
  const int nb = st.nb, total = t.nl * nb, S = P.nstages, S0 = P.mr.st[0].m + P.mr.pad, sst = P.sstride;
  const uint32_t mnb = st.mg_nb;
  const T2 *mid = (const T2 *)P.mid_tab;
  const int64_t mid_cs = P.mid_cs;
  for (int i = threadIdx.x; i < total; i += blockDim.x) {
    const int p = mr_div(i, mnb);
    const int K = i - p * nb;
    T2 *d = t.sd + p * sst + mr_slot(P, S, S0, K);
    T2 v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = d[r];
    Dft<R>::template apply<T, T2>(v);
    const T2 *mt = mid + t.in[p].col * mid_cs + K;
#pragma unroll
    for (int r = 0; r < R; r++) v[r].y = -v[r].y;
    mr_table<T2, R>(v, mt, 0, nb, 0x7fffffff);
    Dft<R>::template apply<T, T2>(v);
#pragma unroll
    for (int r = 0; r < R; r++) d[r] = v[r];
  }
}

// Second sweep's last stage (digit 0): shared memory -> HBM, natural order.
template <typename T, int R, int FEAT>
__device__ __forceinline__ void mr_dit_last(const fftz_pass_t &P, const MrTile<T> &t, const fftz_mr_stage_t &st) {
  typedef typename Cplx<T>::type T2;
  const int M = st.m, S0 = M + P.mr.pad, sst = P.sstride;
  const T2 *tw = (const T2 *)P.tw + st.tw, *sh = t.tw + st.tw;
  const MrItems it(P, P.out_mode, M, st.mg_nb, t.nl);
  for (int i = threadIdx.x; i < it.total; i += blockDim.x) {
    int p, rest;
    it.at(i, p, rest);
    if (p >= t.nl) continue;
    const T2 *d = t.sd + p * sst + rest;
    T2 v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = d[r * S0];
    mr_twiddle<T, R>(tw, sh, t.has_tw, v, M, rest);
    Dft<R>::template apply<T, T2>(v);
    mr_store<T, R, FEAT>(P, t, v, p, rest, M);
  }
}

// Real lines pair bin k with bin n - k. Butterfly A of a boundary stage (nb of
// them, values A + r nb) mirrors butterfly nb - A, value r against value R - 1 -
// r, so a thread that holds both recombines in registers. Item 0 holds the two
// butterflies that mirror themselves: 0 (value r against R - r) and, for even nb,
// nb / 2 (r against R - 1 - r).
__device__ __forceinline__ int mr_mirror(int q, int nb) { return q ? nb - q : (nb & 1 ? 0 : nb >> 1); }

// X_k and X_{n-k} from Z_k, Z_{n-k} and w = W_{2n}^k: with E = (Z_k + conj
// Z_{n-k}) / 2, O = -i (Z_k - conj Z_{n-k}) / 2, X_k = E + w O, X_{n-k} = conj(E - w O).
template <typename T2> __device__ __forceinline__ void mr_recombine(T2 &zk, T2 &zm, T2 w) {
  typedef decltype(zk.x) T;
  const T er = T(0.5) * (zk.x + zm.x), ei = T(0.5) * (zk.y - zm.y);
  const T orr = T(0.5) * (zk.y + zm.y), oi = T(0.5) * (zm.x - zk.x);
  const T tr = w.x * orr - w.y * oi, ti = w.x * oi + w.y * orr;
  zk.x = er + tr;
  zk.y = ei + ti;
  zm.x = er - tr;
  zm.y = ti - ei;
}
// 2 conj Z_k and 2 conj Z_{n-k} from X_k, X_{n-k}.
template <typename T2> __device__ __forceinline__ void mr_separate(T2 &xk, T2 &xm, T2 w) {
  typedef decltype(xk.x) T;
  const T dr = xk.x - xm.x, di = xk.y + xm.y, s = xk.x + xm.x, d = xk.y - xm.y;
  const T er = w.x * dr + w.y * di, ei = w.x * di - w.y * dr;  // conj(w) (X_k - conj X_{n-k})
  xk.x = s - ei;
  xk.y = -(d + er);
  xm.x = s + ei;
  xm.y = d - er;
}

// Bins of butterflies A (a) and B = mr_mirror(q, nb) (b) to HBM.
template <typename T, int R>
__device__ __forceinline__ void mr_store_half(const fftz_pass_t &P, const MrTile<T> &t, typename Cplx<T>::type (&a)[R],
                                              typename Cplx<T>::type (&b)[R], int p, int q, int nb) {
  typedef typename Cplx<T>::type T2;
  const int64_t oes = P.oes;
  const int n = P.n;
  T2 *g = (T2 *)P.out + t.out[p].off;
  const T2 *rtw = (const T2 *)P.rtw;
  if (q) {
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int k = q + r * nb;
      mr_recombine(a[r], b[R - 1 - r], __ldg(rtw + k));
      g[k * oes] = a[r];
      g[(n - k) * oes] = b[R - 1 - r];
    }
    return;
  }
#pragma unroll
  for (int r = 0; r <= R / 2; r++) {
    const int k = r * nb;
    T2 zk = a[r], zm = a[(R - r) % R];
    mr_recombine(zk, zm, __ldg(rtw + k));
    g[k * oes] = zk;
    if (2 * r != R) g[(n - k) * oes] = zm;
  }
  if (nb & 1) return;
#pragma unroll
  for (int r = 0; r <= (R - 1) / 2; r++) {
    const int k = (nb >> 1) + r * nb;
    T2 zk = b[r], zm = b[R - 1 - r];
    mr_recombine(zk, zm, __ldg(rtw + k));
    g[k * oes] = zk;
    if (r != R - 1 - r) g[(n - k) * oes] = zm;
  }
}

// The same two butterflies' inputs from the half spectrum in HBM.
template <typename T, int R>
__device__ __forceinline__ void mr_load_half(const fftz_pass_t &P, const MrTile<T> &t, typename Cplx<T>::type (&a)[R],
                                             typename Cplx<T>::type (&b)[R], int p, int q, int nb) {
  typedef typename Cplx<T>::type T2;
  const int64_t ies = P.ies;
  const int n = P.n;
  const T2 *g = (const T2 *)P.in + t.in[p].off;
  const T2 *rtw = (const T2 *)P.rtw;
  if (q) {
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int k = q + r * nb;
      a[r] = g[k * ies];
      b[R - 1 - r] = g[(n - k) * ies];
    }
#pragma unroll
    for (int r = 0; r < R; r++) mr_separate(a[r], b[R - 1 - r], __ldg(rtw + q + r * nb));
    return;
  }
#pragma unroll
  for (int r = 0; r <= R / 2; r++) {
    const int k = r * nb;
    T2 xk = g[k * ies], xm = g[(n - k) * ies];
    mr_separate(xk, xm, __ldg(rtw + k));
    a[r] = xk;
    if (r > 0 && 2 * r != R) a[R - r] = xm;
  }
  if (nb & 1) {
#pragma unroll
    for (int r = 0; r < R; r++) b[r] = zero2<T2>();
    return;
  }
#pragma unroll
  for (int r = 0; r <= (R - 1) / 2; r++) {
    const int k = (nb >> 1) + r * nb;
    T2 xk = g[k * ies], xm = g[(n - k) * ies];
    mr_separate(xk, xm, __ldg(rtw + k));
    b[r] = xk;
    if (r != R - 1 - r) b[R - 1 - r] = xm;
  }
}

// Last stage of a packed r2c line: shared memory -> half spectrum in HBM.
template <typename T, int R>
__device__ __forceinline__ void mr_last_r2c(const fftz_pass_t &P, const MrTile<T> &t, const fftz_mr_stage_t &st) {
  typedef typename Cplx<T>::type T2;
  const int nb = st.nb, S = P.nstages, S0 = P.mr.st[0].m + P.mr.pad, sst = P.sstride;
  const MrItems it(P, P.out_mode, (nb + 1) >> 1, P.mr.mg_pair, t.nl);
  for (int i = threadIdx.x; i < it.total; i += blockDim.x) {
    int p, q;
    it.at(i, p, q);
    if (p >= t.nl) continue;
    const T2 *da = t.sd + p * sst + mr_slot(P, S, S0, q), *db = t.sd + p * sst + mr_slot(P, S, S0, mr_mirror(q, nb));
    T2 a[R], b[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
      a[r] = da[r];
      b[r] = db[r];
    }
    Dft<R>::template apply<T, T2>(a);
    Dft<R>::template apply<T, T2>(b);
    mr_store_half<T, R>(P, t, a, b, p, q, nb);
  }
}

// Stage 0 of a packed c2r line: half spectrum in HBM -> shared memory.
template <typename T, int R>
__device__ __forceinline__ void mr_first_c2r(const fftz_pass_t &P, const MrTile<T> &t, const fftz_mr_stage_t &st) {
  typedef typename Cplx<T>::type T2;
  const int M = st.m, S0 = M + P.mr.pad, sst = P.sstride;
  const T2 *tw = (const T2 *)P.tw + st.tw, *sh = t.tw + st.tw;
  const MrItems it(P, P.in_mode, (M + 1) >> 1, P.mr.mg_pair, t.nl);
  for (int i = threadIdx.x; i < it.total; i += blockDim.x) {
    int p, q;
    it.at(i, p, q);
    if (p >= t.nl) continue;
    const int B = mr_mirror(q, M);
    T2 a[R], b[R];
    mr_load_half<T, R>(P, t, a, b, p, q, M);
    T2 *d = t.sd + p * sst;
    Dft<R>::template apply<T, T2>(a);
    mr_twiddle<T, R>(tw, sh, t.has_tw, a, M, q);
#pragma unroll
    for (int r = 0; r < R; r++) d[q + r * S0] = a[r];
    if (B == q) continue;  // odd M: butterfly 0 alone
    Dft<R>::template apply<T, T2>(b);
    mr_twiddle<T, R>(tw, sh, t.has_tw, b, M, B);
#pragma unroll
    for (int r = 0; r < R; r++) d[B + r * S0] = b[r];
  }
}

// Packed lines of one stage (n <= 16): a thread a line.
template <typename T, int R, int FEAT>
__device__ __forceinline__ void mr_single_real(const fftz_pass_t &P, const MrTile<T> &t) {
  typedef typename Cplx<T>::type T2;
  for (int p = threadIdx.x; p < t.nl; p += blockDim.x) {
    T2 a[R], b[R];
    if constexpr ((FEAT & FEAT_MR_C2R) != 0)
      mr_load_half<T, R>(P, t, a, b, p, 0, 1);
    else
      mr_load<T, R, FEAT>(P, t, a, p, 0, 1);
    Dft<R>::template apply<T, T2>(a);
    if constexpr ((FEAT & FEAT_MR_C2R) != 0)
      mr_store<T, R, FEAT>(P, t, a, p, 0, 1);
    else
      mr_store_half<T, R>(P, t, a, b, p, 0, 1);
  }
}

// Radix sets: MR_SMOOTH without 11 and 13 (whose butterflies hold more live
// values), MR_ALL, and those of the stage that holds mirrored butterflies (two
// of them in a thread: at most 8, or 11 and 13 where a line has nothing else).
enum { MR_SMOOTH = 0, MR_ALL = 1, MR_PAIR = 2 };
__host__ __device__ constexpr bool mr_has(int set, int R) {
  return set == MR_ALL || (set == MR_PAIR ? R <= 8 || R == 11 || R == 13 : R != 11 && R != 13);
}
#define FZ_MR_CASE(SET, R_, CALL) \
  case R_:                        \
    if constexpr (mr_has(SET, R_)) { constexpr int R = R_; CALL; } \
    break;
#define FZ_MR_SWITCH(R_, SET, CALL)                                                                             \
  switch (R_) {                                                                                                 \
    FZ_MR_CASE(SET, 2, CALL) FZ_MR_CASE(SET, 3, CALL) FZ_MR_CASE(SET, 4, CALL) FZ_MR_CASE(SET, 5, CALL)         \
    FZ_MR_CASE(SET, 6, CALL) FZ_MR_CASE(SET, 7, CALL) FZ_MR_CASE(SET, 8, CALL) FZ_MR_CASE(SET, 9, CALL)         \
    FZ_MR_CASE(SET, 10, CALL) FZ_MR_CASE(SET, 11, CALL) FZ_MR_CASE(SET, 12, CALL) FZ_MR_CASE(SET, 13, CALL)     \
    FZ_MR_CASE(SET, 14, CALL) FZ_MR_CASE(SET, 15, CALL) FZ_MR_CASE(SET, 16, CALL)                               \
  }

// Four-step factors W^{col nb r} of the final butterflies of radix Rl (outputs
// nb apart), formed per line; read after the caller's next barrier.
template <typename T> __device__ __forceinline__ void mr_steps(const fftz_pass_t &P, const MrTile<T> &t, int Rl) {
  typedef typename Cplx<T>::type T2;
  const uint32_t nb = (uint32_t)(P.n / Rl);
  const MrTw4<T2> w = mr_tw4<T2>(P);
  for (int i = threadIdx.x; i < 16 * t.nl; i += blockDim.x) {
    const int p = i >> 4, r = i & 15;
    if (r < Rl) t.stp[i] = w((uint32_t)t.out[p].col * (nb * (uint32_t)r));
  }
}

// One CTA-worth of a pass: transforms [blk * tpc, (blk + 1) * tpc).
template <typename T, int FEAT, int SET>
__device__ __forceinline__ void mr_tile(const fftz_pass_t &P, int64_t blk, unsigned char *smem_raw) {
  typedef typename Cplx<T>::type T2;
  const int S = P.nstages, tpc = P.tpc;
  MrTile<T> t;
  t.sd = (T2 *)smem_raw;
  t.stp = (T2 *)(smem_raw + (((size_t)tpc * P.sstride * sizeof(T2) + 15) & ~(size_t)15));
  MrLine *in = (MrLine *)(t.stp + ((FEAT & FEAT_MR_TW4) ? 16 * tpc : 0)), *out = in + tpc;
  t.has_tw = false;
  t.tw = t.sd;
  t.in = in;
  t.out = out;
  t.nl = P.ntf - blk * tpc < tpc ? (int)(P.ntf - blk * tpc) : tpc;
  for (int p = threadIdx.x; p < t.nl; p += blockDim.x) {
    batch_offsets(P, blk * tpc + p, &in[p].off, &out[p].off, &in[p].col);
    out[p].col = in[p].col;
  }
  pdl_begin();
  __syncthreads();
  if constexpr ((FEAT & FEAT_MR_TW4) != 0) {
    mr_steps<T>(P, t, (FEAT & FEAT_MR_BLUE) ? P.mr.st[0].r : P.mr.st[S - 1].r);
    if (S == 1) __syncthreads();
  }
  if (S == 1) {
    if constexpr ((FEAT & (FEAT_MR_R2C | FEAT_MR_C2R)) != 0) {
      if (P.n == 1) mr_single_real<T, 1, FEAT>(P, t);
      FZ_MR_SWITCH(P.mr.st[0].r, SET, (mr_single_real<T, R, FEAT>(P, t)));
    } else if constexpr ((FEAT & FEAT_MR_BLUE) == 0) {
      if (P.n == 1) mr_single<T, 1, FEAT>(P, t);
      FZ_MR_SWITCH(P.mr.st[0].r, SET, (mr_single<T, R, FEAT>(P, t)));
    }
    return;
  }
  if constexpr ((FEAT & FEAT_MR_C2R) != 0) {
    FZ_MR_SWITCH(P.mr.st[0].r, MR_PAIR, (mr_first_c2r<T, R>(P, t, P.mr.st[0])));
  } else {
    FZ_MR_SWITCH(P.mr.st[0].r, SET, (mr_first<T, R, FEAT>(P, t, P.mr.st[0])));
  }
  __syncthreads();
  for (int s = 1; s < S - 1; s++) {
    FZ_MR_SWITCH(P.mr.st[s].r, SET, (mr_mid<T, R, false>(P, t, P.mr.st[s])));
    __syncthreads();
  }
  if constexpr ((FEAT & FEAT_MR_BLUE) != 0) {
    FZ_MR_SWITCH(P.mr.st[S - 1].r, SET, (mr_product<T, R>(P, t, P.mr.st[S - 1])));
    __syncthreads();
    for (int s = S - 2; s > 0; s--) {
      FZ_MR_SWITCH(P.mr.st[s].r, SET, (mr_mid<T, R, true>(P, t, P.mr.st[s])));
      __syncthreads();
    }
    FZ_MR_SWITCH(P.mr.st[0].r, SET, (mr_dit_last<T, R, FEAT>(P, t, P.mr.st[0])));
  } else if constexpr ((FEAT & FEAT_MR_R2C) != 0) {
    FZ_MR_SWITCH(P.mr.st[S - 1].r, MR_PAIR, (mr_last_r2c<T, R>(P, t, P.mr.st[S - 1])));
  } else {
    FZ_MR_SWITCH(P.mr.st[S - 1].r, SET, (mr_last<T, R, FEAT>(P, t, P.mr.st[S - 1])));
  }
}

}  // namespace fftz
