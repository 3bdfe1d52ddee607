// The order of tie_order.cuh for lists that fit shared memory (11 bytes an entry), by one thread block.
//
// Same steps with four barriers a level instead of five, and without a trip to L2 behind each of them: a thread keeps
// the ranges of its positions in registers, the prefix counts are kept at the ends of a range only (a range has 16
// positions or more, so that position / 16 numbers it), and the two position lists are stored by their counts over all
// ranges, not from the start of the range, so that nobody waits for a range's first count before storing.
#pragma once

#include "tie_order.cuh"

namespace orca {
namespace tie {

constexpr int SHARED_MAX = 20480;   // entries: 220 KB, and positions and counts fit 16 bits

// The lists lie at the start of the kernel's dynamic shared memory (named here, so that every access is known to be to
// shared memory), `cap` entries each, a multiple of 16.
extern __shared__ __align__(16) char smem[];
struct Shared {
  int cap;
  static constexpr int BYTES = 11;
  __device__ int32_t &key(int i) const { return ((int32_t *)smem)[i]; }                    // keys in sort order
  __device__ uint16_t &idx(int i) const { return ((uint16_t *)(smem + 4 * cap))[i]; }      // the entries' numbers
  __device__ uint16_t &left(int i) const { return ((uint16_t *)(smem + 6 * cap))[i]; }     // positions, key >= pivot
  __device__ uint16_t &right(int i) const { return ((uint16_t *)(smem + 8 * cap))[i]; }    // positions, key <= pivot
  // of the range that starts at lo: counts (left | right << 16) before its ends, pivot, the pivot's place
  __device__ uint32_t &before_lo(int lo) const { return ((uint32_t *)(smem + 10 * cap))[lo >> 4]; }
  __device__ uint32_t &before_hi(int lo) const { return ((uint32_t *)(smem + 10 * cap))[(cap >> 4) + (lo >> 4)]; }
  __device__ int32_t &pivot(int lo) const { return ((int32_t *)(smem + 10 * cap))[2 * (cap >> 4) + (lo >> 4)]; }
  __device__ int32_t &place(int lo) const { return ((int32_t *)(smem + 10 * cap))[3 * (cap >> 4) + (lo >> 4)]; }
};

__device__ __forceinline__ uint32_t range(int lo, int hi) { return (uint32_t)lo | (uint32_t)hi << 16; }
__device__ __forceinline__ int lo_of(uint32_t r) { return (int)(r & 0xffff); }
__device__ __forceinline__ int hi_of(uint32_t r) { return (int)(r >> 16); }
constexpr uint32_t NO_RANGE = 0xffffu;   // lo 65535, hi 0: of no position

__device__ __forceinline__ void park_pivot(const Shared w, int lo, int hi) {
  const int mid = (lo + hi) >> 1;
  int32_t a = w.key(lo), c = w.key(mid), d = w.key(hi), t;
  uint16_t ia = w.idx(lo), ic = w.idx(mid), id = w.idx(hi), it;
  if (c < a) { t = a; a = c; c = t; it = ia; ia = ic; ic = it; }
  if (d < c) { t = d; d = c; c = t; it = id; id = ic; ic = it; }
  if (c < a) { t = a; a = c; c = t; it = ia; ia = ic; ic = it; }
  w.key(lo) = a; w.idx(lo) = ia;
  w.key(mid) = d; w.idx(mid) = id;
  w.key(hi) = c; w.idx(hi) = ic;
  w.pivot(lo) = c;
}
__device__ __forceinline__ void swap_entries(const Shared w, int l, int r) {
  const int32_t k = w.key(l), kr = w.key(r);
  const uint16_t i = w.idx(l), ir = w.idx(r);
  w.key(l) = kr; w.idx(l) = ir;
  w.key(r) = k; w.idx(r) = i;
}

// All T threads call this.  Thread t owns positions first + 32 * i, first = (t / 32) * 32 * items + t % 32, i < items
// <= ITEMS; r[i] is the range of such a position (NO_RANGE past the end), and every live range has its pivot parked.
// Partitions until no live range is longer than `stop` (>= 15).  tot: NW words of shared memory.  Every level takes the
// pivot out of each live range, so that it ends.
template <int ITEMS>
__device__ __forceinline__ void partition_levels(const Shared w, uint32_t *tot, int items, int keep, int stop,
                                                 uint32_t (&r)[ITEMS]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  const int first = warp * 32 * items + lane;
  bool more = false;
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) more |= i < items && live(lo_of(r[i]), hi_of(r[i]), keep) && hi_of(r[i]) - lo_of(r[i]) >= stop;
  while (__syncthreads_or(more)) {
    uint32_t fl = 0, fr = 0, at = 0;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      if (i < items) {
        const int pos = first + 32 * i, lo = lo_of(r[i]), hi = hi_of(r[i]);
        const bool in = live(lo, hi, keep) && pos < hi;
        const int32_t k = in ? w.key(pos) : 0, p = in ? w.pivot(lo) : 0;
        const bool l = in && k >= p, g = in && k <= p;
        fl |= (l ? 1u : 0u) << i;
        fr |= (g ? 1u : 0u) << i;
        at += __popc(__ballot_sync(0xffffffffu, l)) | __popc(__ballot_sync(0xffffffffu, g)) << 16;
      }
    }
    if (lane == 0) tot[warp] = at;
    __syncthreads();
    uint32_t incl = tot[lane];
    const uint32_t mine = incl;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    at = __shfl_sync(0xffffffffu, incl - mine, warp);
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      if (i < items) {
        const int pos = first + 32 * i, lo = lo_of(r[i]), hi = hi_of(r[i]);
        const bool l = (fl >> i) & 1u, g = (fr >> i) & 1u;
        const uint32_t ml = __ballot_sync(0xffffffffu, l), mr = __ballot_sync(0xffffffffu, g);
        const uint32_t me = at + (__popc(ml & lt) | __popc(mr & lt) << 16);
        if (l) w.left(me & 0xffff) = (uint16_t)pos;
        if (g) w.right(me >> 16) = (uint16_t)pos;
        if (live(lo, hi, keep)) {
          if (pos == lo) w.before_lo(lo) = me;
          if (pos == hi) w.before_hi(lo) = me;
        }
        at += __popc(ml) | __popc(mr) << 16;
      }
    }
    __syncthreads();
    // pair m (its thread: position lo + m) swaps while its left position is left of its right position
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      if (i < items) {
        const int pos = first + 32 * i, lo = lo_of(r[i]), hi = hi_of(r[i]);
        if (live(lo, hi, keep) && pos < hi) {
          const uint32_t a = w.before_lo(lo), z = w.before_hi(lo);
          const int al = (int)(a & 0xffff), nl = (int)(z & 0xffff) - al, nr = (int)(z >> 16) - (int)(a >> 16);
          const int pairs = min(nl, nr), m = pos - lo, last_r = (int)(z >> 16) - 1;
          if (m < pairs) {
            const int pl = w.left(al + m), pr = w.right(last_r - m);
            const int next_l = m + 1 < nl ? (int)w.left(al + m + 1) : hi;
            if (pl < pr) {
              swap_entries(w, pl, pr);
              if (m + 1 >= pairs || next_l >= (int)w.right(last_r - m - 1)) w.place(lo) = min(next_l, pr);
            } else if (m == 0) {
              w.place(lo) = pl;
            }
          } else if (m == 0) {
            w.place(lo) = nl > 0 ? (int)w.left(al) : hi;
          }
        }
      }
    }
    __syncthreads();
    // pivots into place, ranges split, next pivots parked
    more = false;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      if (i < items) {
        const int pos = first + 32 * i;
        int lo = lo_of(r[i]), hi = hi_of(r[i]);
        if (live(lo, hi, keep)) {
          const int p = w.place(lo);
          if (pos == p + 1) swap_entries(w, p, hi);   // (the thread that parks the pivot of the right part)
          if (pos < p) hi = p - 1;
          else if (pos > p) lo = p + 1;
          else lo = hi = p;
          r[i] = range(lo, hi);
          if (live(lo, hi, keep)) {
            more |= hi - lo >= stop;
            if (pos == lo) park_pivot(w, lo, hi);
          }
        }
      }
    }
  }
}

// where the entry at `pos` ends up in its range of fewer than 16
__device__ __forceinline__ int place_of(const Shared w, int pos, int lo, int hi) {
  const int32_t k = w.key(pos);
  int place = lo;
  for (int q = lo; q <= hi; ++q) {
    const int32_t ko = w.key(q);
    place += (ko < k || (ko == k && q < pos)) ? 1 : 0;
  }
  return place;
}

// All T threads call this with key and idx filled (n <= 1024 * ITEMS): calls
// f(place, entry) for the first `keep` places of the argsort.
template <int ITEMS, class F>
__device__ __forceinline__ void sort_first_shared(const Shared w, uint32_t *tot, int n, int keep, F f) {
  const int items = (n + T - 1) / T;
  const int first = (threadIdx.x >> 5) * 32 * items + (threadIdx.x & 31);
  uint32_t r[ITEMS];
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) r[i] = i < items && first + 32 * i < n ? range(0, n - 1) : NO_RANGE;
  __syncthreads();
  if (threadIdx.x == 0 && live(0, n - 1, keep)) park_pivot(w, 0, n - 1);
  partition_levels<ITEMS>(w, tot, items, keep, 15, r);
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    if (i < items && hi_of(r[i]) - lo_of(r[i]) >= 0 && lo_of(r[i]) < keep) {
      const int pos = first + 32 * i, place = place_of(w, pos, lo_of(r[i]), hi_of(r[i]));
      if (place < keep) f(place, (int)w.idx(pos));
    }
  }
  __syncthreads();
}

}  // namespace tie
}  // namespace orca
