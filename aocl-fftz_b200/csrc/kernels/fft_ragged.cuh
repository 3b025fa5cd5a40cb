// Persistent DAG executor for ragged batches: transforms of different lengths
// and algorithms run in ONE launch (captured in a CUDA graph by the host).
//
// The host groups the transforms by length, plans each group as one batched
// plan whose transform dimension is indirect (every transform keeps its own
// offset in the packed buffers), and flattens the passes into a table of CTA
// tiles ("items"), ordered so that all tiles of pass depth d precede those of
// depth d+1. Each CTA repeatedly takes the next item with an atomic counter,
// copies the item's pass descriptor into shared memory (resolving buffer
// offsets against the launch's in / out / scratch bases), waits -- with a
// bounded spin -- until every tile of the item's predecessor pass is done,
// runs the tile and counts itself done with release semantics. Every tile is a
// mixed-radix tile (fft_mr.cuh) of the CTA's 256 threads. One warp takes the
// next item, copies its pass, forms its lines' offsets and looks at its
// predecessor during the current tile, so a tile starts with its first loads
// unless it has to wait. An item is
// held only by a running CTA, and every predecessor item was taken before its
// successors: the lowest unfinished item is always running (its CTA takes items
// in order), so the waits end; the spin limit turns a broken invariant into an
// error flag instead of a hang.
#include "fft_mr.cuh"

namespace fftz {

__device__ __forceinline__ int ld_acquire(const int *p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// What a CTA holds of one tile: the item, its pass with the buffers resolved, its
// lines' places, and whether its predecessor was seen complete.
struct RgSlot {
  fftz_pass_t P;
  MrLine in[FFTZ_RG_LINES], out[FFTZ_RG_LINES];
  fftz_ritem_t item;
  long long next;  // the item's index (>= nitems: no more)
  int ready;
};

// The slots' copies of their passes' stage twiddles. A pass of the batch shares
// its table with few tiles, so reading it where it is used costs an L2 access each
// time; copied with the pass, one tile ahead, it costs none.
template <typename T> __device__ __forceinline__ typename Cplx<T>::type *rg_tw(int b) {
  __shared__ __align__(16) typename Cplx<T>::type tw[2][FFTZ_RG_TW];
  return tw[b];
}

// The CTA's two slots (its only other static shared memory, so that out-of-line stages
// address them as shared memory).
__device__ __forceinline__ RgSlot *rg_slot(int b) {
  __shared__ __align__(16) RgSlot slot[2];
  return &slot[b];
}

// One warp: item `it` (drawn by lane 0) into *s.
__device__ __forceinline__ long long rg_draw(const fftz_ragged_t &R) {
  return (threadIdx.x & 31) == 0 ? (long long)atomicAdd(R.queue, 1ULL) : 0;
}
template <typename T> __device__ __forceinline__ void rg_fetch(const fftz_ragged_t &R, int b, long long it) {
  typedef typename Cplx<T>::type T2;
  RgSlot *s = rg_slot(b);
  const int lane = threadIdx.x & 31;
  it = __shfl_sync(0xffffffffu, it, 0);
  if (lane == 0) s->next = it;
  if (it >= R.nitems) return;
  const fftz_ritem_t x = R.items[it];
  const int4 *src = (const int4 *)(R.passes + x.pass);
  static_assert(sizeof(fftz_pass_t) % 16 == 0, "16-byte words");
  for (int i = lane; i < (int)(sizeof(fftz_pass_t) / 16); i += 32) ((int4 *)&s->P)[i] = __ldg(src + i);
  __syncwarp();
  const fftz_pass_t &P = s->P;
  if (P.ntw <= FFTZ_RG_TW) {
    constexpr int Q = 16 / sizeof(T2);  // entries of a 16-byte copy; tables are 256-byte aligned and padded
    T2 *d = rg_tw<T>(b);
    for (int i = lane * Q; i < P.ntw; i += 32 * Q)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(d + i)),
                   "l"((const T2 *)P.tw + i)
                   : "memory");
  }
  for (int p = lane; p < P.tpc; p += 32) {
    batch_offsets(P, x.blk * P.tpc + p, &s->in[p].off, &s->out[p].off, &s->in[p].col);
    s->out[p].col = s->in[p].col;
  }
  if (lane == 0) {
    s->item = x;
    s->ready = x.dep < 0 || ld_acquire(R.done + x.dep) >= x.dep_count;
    const unsigned char *ib = (const unsigned char *)(P.src_buf == FFTZ_RBUF_IN    ? R.in
                                                      : P.src_buf == FFTZ_RBUF_OUT ? (const void *)R.out
                                                                                   : (const void *)R.scratch);
    unsigned char *ob = (unsigned char *)(P.dst_buf == FFTZ_RBUF_IN    ? (void *)R.in
                                          : P.dst_buf == FFTZ_RBUF_OUT ? R.out
                                                                       : R.scratch);
    s->P.in = ib + (size_t)P.in;
    s->P.out = ob + (size_t)P.out;
  }
}

// The fetching warp, before the barrier that opens the fetched slot: its copies
// have landed.
__device__ __forceinline__ void rg_landed() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// One stage (radix R, form FORM) of slot s out of line: each has its own register
// allocation within the kernel's bound (inlined together they spilled 4.5 KB).
enum {
  RG_FIRST, RG_FIRST_PRE, RG_MID, RG_LAST, RG_LAST_TW4, RG_LAST_POST, RG_PRODUCT, RG_MID2, RG_LAST2_TW4, RG_LAST2_POST,
  RG_SINGLE
};

template <typename T> __device__ __forceinline__ MrTile<T> rg_view(int b, unsigned char *smem_raw) {
  const RgSlot *s = rg_slot(b);
  typedef typename Cplx<T>::type T2;
  MrTile<T> t;
  t.sd = (T2 *)smem_raw;
  t.stp = (T2 *)(smem_raw + (((size_t)s->P.tpc * s->P.sstride * sizeof(T2) + 15) & ~(size_t)15));
  t.has_tw = s->P.ntw <= FFTZ_RG_TW;
  t.tw = rg_tw<T>(b);
  t.in = s->in;
  t.out = s->out;
  const int64_t left = s->P.ntf - s->item.blk * s->P.tpc;
  t.nl = left < s->P.tpc ? (int)left : s->P.tpc;
  return t;
}

template <typename T, int R, int FORM> __device__ __noinline__ void rg_stage(int b, int j) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const MrTile<T> t = rg_view<T>(b, smem_raw);
  const fftz_pass_t &P = rg_slot(b)->P;
  const fftz_mr_stage_t &st = P.mr.st[j];
  if constexpr (FORM == RG_FIRST) mr_first<T, R, 0>(P, t, st);
  if constexpr (FORM == RG_FIRST_PRE) mr_first<T, R, FEAT_MR_PRE>(P, t, st);
  if constexpr (FORM == RG_MID) mr_mid<T, R, false>(P, t, st);
  if constexpr (FORM == RG_LAST) mr_last<T, R, 0>(P, t, st);
  if constexpr (FORM == RG_LAST_TW4) mr_last<T, R, FEAT_MR_TW4>(P, t, st);
  if constexpr (FORM == RG_LAST_POST) mr_last<T, R, FEAT_MR_POST>(P, t, st);
  if constexpr (FORM == RG_PRODUCT) mr_product<T, R>(P, t, st);
  if constexpr (FORM == RG_MID2) mr_mid<T, R, true>(P, t, st);
  if constexpr (FORM == RG_LAST2_TW4) mr_dit_last<T, R, FEAT_MR_TW4>(P, t, st);
  if constexpr (FORM == RG_LAST2_POST) mr_dit_last<T, R, FEAT_MR_POST>(P, t, st);
  if constexpr (FORM == RG_SINGLE) mr_single<T, R, 0>(P, t);
}

// One tile of slot b. The last warp draws the CTA's next item before stage 0 and
// fetches it into the other slot after that stage's barrier.
template <typename T> __device__ __forceinline__ void rg_tile(const fftz_ragged_t &R_, int b, unsigned char *smem_raw) {
  const fftz_pass_t &P = rg_slot(b)->P;
  const int S = P.nstages, flags = P.flags, r0 = P.mr.st[0].r, rl = P.mr.st[S - 1].r;
  const bool two = (flags & FFTZ_F_MID_TAB) != 0, tw4 = (flags & FFTZ_F_TW4) != 0;
  const bool fetcher = threadIdx.x >= 224;
  long long it = 0;
  if (fetcher) it = rg_draw(R_);
  if (tw4) mr_steps<T>(P, rg_view<T>(b, smem_raw), two ? r0 : rl);
  if (S > 1) {
    if (flags & FFTZ_F_PRE_TAB) {
      FZ_MR_SWITCH(r0, MR_SMOOTH, (rg_stage<T, R, RG_FIRST_PRE>(b, 0)));
    } else {
      FZ_MR_SWITCH(r0, MR_ALL, (rg_stage<T, R, RG_FIRST>(b, 0)));
    }
  }
  __syncthreads();
  if (fetcher) rg_fetch<T>(R_, b ^ 1, it);
  if (S == 1) {
    if (P.n == 1) rg_stage<T, 1, RG_SINGLE>(b, 0);
    FZ_MR_SWITCH(r0, MR_ALL, (rg_stage<T, R, RG_SINGLE>(b, 0)));
    return;
  }
  for (int j = 1; j < S - 1; j++) {
    FZ_MR_SWITCH(P.mr.st[j].r, MR_ALL, (rg_stage<T, R, RG_MID>(b, j)));
    __syncthreads();
  }
  if (!two) {
    if (flags & FFTZ_F_POST_TAB) {
      FZ_MR_SWITCH(rl, MR_SMOOTH, (rg_stage<T, R, RG_LAST_POST>(b, S - 1)));
    } else if (tw4) {
      FZ_MR_SWITCH(rl, MR_ALL, (rg_stage<T, R, RG_LAST_TW4>(b, S - 1)));
    } else {
      FZ_MR_SWITCH(rl, MR_ALL, (rg_stage<T, R, RG_LAST>(b, S - 1)));
    }
    return;
  }
  FZ_MR_SWITCH(rl, MR_SMOOTH, (rg_stage<T, R, RG_PRODUCT>(b, S - 1)));
  __syncthreads();
  for (int j = S - 2; j > 0; j--) {
    FZ_MR_SWITCH(P.mr.st[j].r, MR_SMOOTH, (rg_stage<T, R, RG_MID2>(b, j)));
    __syncthreads();
  }
  if (tw4) {
    FZ_MR_SWITCH(r0, MR_SMOOTH, (rg_stage<T, R, RG_LAST2_TW4>(b, 0)));
  } else {
    FZ_MR_SWITCH(r0, MR_SMOOTH, (rg_stage<T, R, RG_LAST2_POST>(b, 0)));
  }
}

// float 64 registers (4 CTAs per SM), double 128 (2): the bounds at which the
// radix-16 butterflies keep their values in registers.
template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 4 : 2) fft_ragged_kernel(const __grid_constant__ fftz_ragged_t R) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (threadIdx.x >= 224) {
    rg_fetch<T>(R, 0, rg_draw(R));
    rg_landed();
  }
  __syncthreads();
  for (int b = 0; rg_slot(b)->next < R.nitems; b ^= 1) {
    RgSlot *s = rg_slot(b);
    if (!s->ready) {  // uniform: every thread reads the same word
      __syncthreads();
      if (threadIdx.x == 0) {
        int ok = 1;
        long long spins = 0;
        while (ld_acquire(R.done + s->item.dep) < s->item.dep_count) {
          if (++spins > R.spin_limit) {
            atomicExch(R.err, 1);
            ok = -1;
            break;
          }
          __nanosleep(100);
        }
        __threadfence();
        s->ready = ok;
      }
      __syncthreads();
    }
    if (s->ready > 0)
      rg_tile<T>(R, b, smem_raw);
    else if (threadIdx.x >= 224)
      rg_fetch<T>(R, b ^ 1, rg_draw(R));
    if (threadIdx.x >= 224) rg_landed();
    __syncthreads();
    // only passes that another pass waits for publish their tiles (the fence
    // waits for the tile's stores, which nothing else needs to do)
    if (s->item.signal && threadIdx.x == 0) {
      __threadfence();
      atomicAdd(R.done + s->item.pass, 1);
    }
  }
}

}  // namespace fftz
