// The order of tie_order.cuh for lists that fit shared memory (15 bytes an entry), by one thread block.
//
// Same steps with four barriers a level instead of five, and without a trip to L2 behind each of them.  A level is bound
// by the instructions of its one block: a thread owns consecutive positions (an odd number of them, so that the threads
// of a warp fall on different banks), looks a range up once instead of once a position, and the prefix counts take one
// warp scan a level instead of votes for every 32 positions (30,000 cycles a level of 10,500 entries with those,
// 14,000 now).  The counts are kept at the ends of a range only (a range has 16 positions or more, so that position / 16
// numbers it), and the two position lists are stored by their counts over all ranges, not from the start of the range, so
// that nobody waits for a range's first count before storing.
#pragma once

#include "tie_order.cuh"

namespace orca {
namespace tie {

constexpr int SHARED_MAX = 14848;   // entries: 218 KB, and positions and counts fit 16 bits

// The lists lie at the start of the kernel's dynamic shared memory (named here, so that every access is known to be to
// shared memory), `cap` entries each, a multiple of 16.
extern __shared__ __align__(16) char smem[];
struct Shared {
  int cap;
  static constexpr int BYTES = 15;
  __device__ int32_t &key(int i) const { return ((int32_t *)smem)[i]; }                    // keys in sort order
  __device__ uint16_t &idx(int i) const { return ((uint16_t *)(smem + 4 * cap))[i]; }      // the entries' numbers
  __device__ uint16_t &left(int i) const { return ((uint16_t *)(smem + 6 * cap))[i]; }     // positions, key >= pivot
  __device__ uint16_t &right(int i) const { return ((uint16_t *)(smem + 8 * cap))[i]; }    // positions, key <= pivot
  __device__ uint32_t &ranges(int i) const { return ((uint32_t *)(smem + 10 * cap))[i]; }  // range of a position
  // of the range that starts at lo: counts (left | right << 16) before its ends, pivot, the pivot's place
  __device__ uint32_t &before_lo(int lo) const { return ((uint32_t *)(smem + 14 * cap))[lo >> 4]; }
  __device__ uint32_t &before_hi(int lo) const { return ((uint32_t *)(smem + 14 * cap))[(cap >> 4) + (lo >> 4)]; }
  __device__ int32_t &pivot(int lo) const { return ((int32_t *)(smem + 14 * cap))[2 * (cap >> 4) + (lo >> 4)]; }
  __device__ int32_t &place(int lo) const { return ((int32_t *)(smem + 14 * cap))[3 * (cap >> 4) + (lo >> 4)]; }
};

__device__ __forceinline__ uint32_t range(int lo, int hi) { return (uint32_t)lo | (uint32_t)hi << 16; }
__device__ __forceinline__ int lo_of(uint32_t r) { return (int)(r & 0xffff); }
__device__ __forceinline__ int hi_of(uint32_t r) { return (int)(r >> 16); }

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

// All T threads call this, behind a barrier after the entries and their ranges were stored and the pivot of every live
// range was parked.  Partitions all live ranges, a level at a time, until none is longer than `stop` (>= 15) or `levels`
// are done; returns whether one is (the same in every thread).  tot: NW words of shared memory.  n <= 31 * T.  Every
// level takes the pivot out of each live range, so that it ends.
static __device__ __noinline__ bool partition_many(const Shared w, uint32_t *tot, int n, int keep, int stop, int levels) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int items = ((n + T - 1) / T) | 1, first = min(n, (int)threadIdx.x * items), end = min(n, first + items);
  bool more = false;
  for (int pos = first; pos < end;) {
    const uint32_t r = w.ranges(pos);
    more |= live(lo_of(r), hi_of(r), keep) && hi_of(r) - lo_of(r) >= stop;
    pos = hi_of(r) + 1;
  }
  // f(lo, hi, from, to) for the part [from, to) of each live range that this thread owns
  const auto live_parts = [&](auto f) {
    for (int pos = first; pos < end;) {
      const uint32_t r = w.ranges(pos);
      const int lo = lo_of(r), hi = hi_of(r), to = min(end, hi + 1);
      if (live(lo, hi, keep)) f(lo, hi, pos, to);
      pos = to;
    }
  };
  while (true) {
    const bool any = __syncthreads_or(more);
    if (!any || levels-- == 0) return any;
    // counts of the left list (key >= pivot) and the right list (key <= pivot)
    uint32_t fl = 0, fr = 0, cnt = 0;
    live_parts([&](int lo, int hi, int pos, int to) {
      const int32_t p = w.pivot(lo);
      to = min(to, hi);
#pragma unroll 4
      for (; pos < to; ++pos) {
        const int32_t k = w.key(pos);
        const uint32_t at = 1u << (pos - first);
        fl |= k >= p ? at : 0u;
        fr |= k <= p ? at : 0u;
      }
    });
    cnt = __popc(fl) | __popc(fr) << 16;
    uint32_t incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    if (lane == 31) tot[warp] = incl;
    __syncthreads();
    uint32_t at = tot[lane];
    at = lane < warp ? at : 0u;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) at += __shfl_xor_sync(0xffffffffu, at, o);
    at += incl - cnt;
    const auto before = [&](int pos) {
      const uint32_t upto = (1u << (pos - first)) - 1u;
      return at + (__popc(fl & upto) | __popc(fr & upto) << 16);
    };
    live_parts([&](int lo, int hi, int pos, int to) {
      if (pos == lo) w.before_lo(lo) = before(lo);
      if (to > hi) w.before_hi(lo) = before(hi);
    });
    {
      int l = at & 0xffff, g = at >> 16;
      for (uint32_t m = fl; m != 0; m &= m - 1) w.left(l++) = (uint16_t)(first + __ffs(m) - 1);
      for (uint32_t m = fr; m != 0; m &= m - 1) w.right(g++) = (uint16_t)(first + __ffs(m) - 1);
    }
    __syncthreads();
    // pair m (its thread: position lo + m) swaps while its left position is left of its right position
    live_parts([&](int lo, int hi, int pos, int to) {
      const uint32_t a = w.before_lo(lo), z = w.before_hi(lo);
      const int al = (int)(a & 0xffff), nl = (int)(z & 0xffff) - al, last_r = (int)(z >> 16) - 1;
      const int pairs = min(nl, last_r + 1 - (int)(a >> 16));
      if (pos == lo && pairs == 0) w.place(lo) = nl > 0 ? (int)w.left(al) : hi;
      to = min(to, lo + pairs);
      int pl = pos < to ? (int)w.left(al + pos - lo) : 0, pr = pos < to ? (int)w.right(last_r - (pos - lo)) : 0;
      if (pos == lo && pos < to && pl >= pr) w.place(lo) = pl;
      for (; pos < to && pl < pr; ++pos) {   // (behind a pair that does not swap, none does)
        const int m = pos - lo;
        const int next_l = m + 1 < nl ? (int)w.left(al + m + 1) : hi;
        const int next_r = m + 1 < pairs ? (int)w.right(last_r - m - 1) : -1;
        swap_entries(w, pl, pr);
        if (next_l >= next_r) w.place(lo) = min(next_l, pr);
        pl = next_l;
        pr = next_r;
      }
    });
    __syncthreads();
    // pivots into place, ranges split, next pivots parked
    more = false;
    live_parts([&](int lo, int hi, int pos, int to) {
      const int p = w.place(lo);
#pragma unroll 4
      for (int i = pos; i < to; ++i)
        w.ranges(i) = i < p ? range(lo, p - 1) : i == p ? range(p, p) : range(p + 1, hi);
      const auto next = [&](int l, int h) {   // (one thread per part: the one that owns its first position)
        if (live(l, h, keep)) {
          more |= h - l >= stop;
          park_pivot(w, l, h);
        }
      };
      if (pos <= lo) next(lo, p - 1);
      if (pos <= p + 1 && p + 1 < to) {
        swap_entries(w, p, hi);   // the pivot to its place
        next(p + 1, hi);
      }
    });
  }
}

// The same for lists of up to FEW * T entries: a thread keeps the ranges of its positions, 32 apart, in registers and the
// loops are unrolled, since here the latency of a level is what counts (250 sorts of 2000 one after the other in a plan:
// 2.7 ms less than with the loops above; at 15 positions a thread they spill, and a level of 10,500 entries takes 42,000 cycles).
// r[i]: the range of position first + 32 * i, NO_RANGE past the end.
constexpr int FEW = 4;
constexpr uint32_t NO_RANGE = 0xffffu;   // lo 65535, hi 0: of no position
__device__ __forceinline__ int few_first(int items) { return (threadIdx.x >> 5) * 32 * items + (threadIdx.x & 31); }
__device__ __forceinline__ bool partition_few(const Shared w, uint32_t *tot, int items, int keep, int stop, int levels,
                                              uint32_t (&r)[FEW]) {
  constexpr int ITEMS = FEW;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  const int first = few_first(items);
  bool more = false;
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) more |= i < items && live(lo_of(r[i]), hi_of(r[i]), keep) && hi_of(r[i]) - lo_of(r[i]) >= stop;
  bool any;
  while ((any = __syncthreads_or(more)) && levels-- > 0) {
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
  return any;
}

__device__ __forceinline__ bool partition(const Shared w, uint32_t *tot, int n, int keep, int stop, int levels) {
  if (n > FEW * T) return partition_many(w, tot, n, keep, stop, levels);
  const int items = (n + T - 1) / T, first = few_first(items);
  uint32_t r[FEW];
#pragma unroll
  for (int i = 0; i < FEW; ++i) r[i] = i < items && first + 32 * i < n ? w.ranges(first + 32 * i) : NO_RANGE;
  const bool any = partition_few(w, tot, items, keep, stop, levels, r);
#pragma unroll
  for (int i = 0; i < FEW; ++i)
    if (i < items && first + 32 * i < n) w.ranges(first + 32 * i) = r[i];
  __syncthreads();
  return any;
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

// All T threads call this with key and idx filled (n <= SHARED_MAX): calls f(place, entry) for the first `keep` places
// of the argsort.
template <class F>
__device__ __forceinline__ void sort_first_shared(const Shared w, uint32_t *tot, int n, int keep, F f) {
  const auto place = [&](int pos, uint32_t r) {
    if (lo_of(r) >= keep) return;
    const int at = place_of(w, pos, lo_of(r), hi_of(r));
    if (at < keep) f(at, (int)w.idx(pos));
  };
  if (n > FEW * T) {
    for (int pos = threadIdx.x; pos < n; pos += T) w.ranges(pos) = range(0, n - 1);
    __syncthreads();
    if (threadIdx.x == 0 && live(0, n - 1, keep)) park_pivot(w, 0, n - 1);
    __syncthreads();
    partition_many(w, tot, n, keep, 15, n);
    for (int pos = threadIdx.x; pos < n; pos += T) place(pos, w.ranges(pos));
  } else {
    const int items = (n + T - 1) / T, first = few_first(items);
    uint32_t r[FEW];
#pragma unroll
    for (int i = 0; i < FEW; ++i) r[i] = i < items && first + 32 * i < n ? range(0, n - 1) : NO_RANGE;
    __syncthreads();
    if (threadIdx.x == 0 && live(0, n - 1, keep)) park_pivot(w, 0, n - 1);
    partition_few(w, tot, items, keep, 15, n, r);
#pragma unroll
    for (int i = 0; i < FEW; ++i)
      if (i < items && first + 32 * i < n) place(first + 32 * i, r[i]);
  }
  __syncthreads();
}

}  // namespace tie
}  // namespace orca
