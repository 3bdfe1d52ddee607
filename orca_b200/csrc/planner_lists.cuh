// What the cache planners share when they walk lists of distinct nodes instead of neighbour tables (planner_lists.cu).
#pragma once

#include "tie_shared.cuh"

namespace orca {
namespace lists {

constexpr int T = tie::T, NW = tie::NW;
constexpr int CAP = 13696;      // entries of a list that is selected from: 17 bytes of shared memory each, whole words of bits

// The distinct nodes of a batch in ascending order: its endpoints (TARGET set) and the out-of-batch neighbours of its table.
// A batch can have as many as its table has entries and has a tenth of them or less as a rule (1,450 of 44,000 on the largest
// graph), so the lists of a whole plan lie one behind the other as they get ready, in as much memory as the caller gives
// (with a stride of the most there can be, the lists of 7.8 M edges took 2.1 GB, 0.07 of it in use); those of a part of a
// plan have a stride.
constexpr int32_t TARGET = (int32_t)0x80000000u;
struct __align__(16) Span {
  int64_t at;        // of the batch's first entry
  int32_t n;
};
struct Lists {
  int32_t *id;       // node | TARGET
  int32_t *mult;     // out-of-batch neighbours: entries of the table that hold the node
  Span *span;        // [batches]
  int64_t stride;    // 0: one behind the other, and
  unsigned long long *used;     // entries taken,
  int64_t room;      // entries there are,
  int32_t *failed;   // set when a list has more than CAP of them, or there is no room
};
inline int64_t stride_of(int32_t bs, int32_t k, int64_t n_nodes) {
  const int64_t most = 2ll * bs * (k + 1);
  return most < n_nodes ? most : n_nodes;
}
// bytes of bitmaps and prefix counts for the blocks that make the lists, and their number
constexpr int64_t SCRATCH = 64 << 20;
inline int64_t block_bytes(int64_t n_nodes) { return (n_nodes + 31) / 32 * 12; }
inline int blocks_for(int64_t n_batches, int64_t n_nodes, int sms) {
  int64_t n = SCRATCH / block_bytes(n_nodes);
  n = n < 1 ? 1 : n > sms ? sms : n;
  return (int)(n < n_batches ? n : n_batches);
}
constexpr int MOST_BLOCKS = 256;     // what a workspace has room for (devices have fewer SMs)
inline int64_t scratch_bytes(int64_t n_batches, int64_t n_nodes) {
  return blocks_for(n_batches, n_nodes, MOST_BLOCKS) * block_bytes(n_nodes);
}
// The lists of batches [b0, b1) (l.span[0] is b0's).  code (optional): set to `code_init` for every node on the way
int launch_batch_lists(const int32_t *d_nodes, const int32_t *d_nbr, int64_t n_edges, int32_t bs, int32_t k, int64_t n_nodes,
                       int64_t b0, int64_t b1, const Lists &l, void *d_scratch, int32_t *d_code, int32_t code_init,
                       cudaStream_t s);

// An entry of a selection: key and place in its list.
constexpr int KEY_BITS = 16, IDX_BITS = 14;
constexpr uint32_t FAR = (1u << KEY_BITS) - 1, IDX = (1u << IDX_BITS) - 1;    // FAR: the largest key
static_assert(CAP <= 1 << IDX_BITS && KEY_BITS + IDX_BITS <= 32, "an entry is a word");

// Bitmaps over places of a list, with the number of bits before each word.
struct Word {
  uint32_t bits;
  int32_t before;
};
// Fills `before` in; returns the number of bits.  All T threads, n <= T words, behind a barrier; ends with one.
__device__ __forceinline__ int count_words(Word *w, int n, int32_t *s_w) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int c = tid < n ? __popc(w[tid].bits) : 0;
  int incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += up;
  }
  if (lane == 31) s_w[warp] = incl;
  __syncthreads();
  const int x = s_w[lane];
  const int before = __reduce_add_sync(0xffffffffu, lane < warp ? x : 0), all = __reduce_add_sync(0xffffffffu, x);
  if (tid < n) w[tid].before = before + incl - c;
  __syncthreads();
  return all;
}
__device__ __forceinline__ bool bit_of(Word w, int i) { return (w.bits >> (i & 31)) & 1u; }
__device__ __forceinline__ int bits_before(Word w, int i) { return w.before + __popc(w.bits & ((1u << (i & 31)) - 1u)); }
// the place of bit number m (there are more than m)
__device__ __forceinline__ int bit_number(const Word *w, int n, int m) {
  int lo = 0, hi = n;      // the last word with no more than m bits before it
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (w[mid].before <= m) lo = mid;
    else hi = mid;
  }
  uint32_t bits = w[lo].bits;
  m -= w[lo].before;
  int at = 0;
#pragma unroll
  for (int half = 16; half > 0; half >>= 1) {
    const int c = __popc(bits & ((1u << half) - 1u));
    if (m >= c) m -= c, at += half, bits >>= half;
  }
  return 32 * lo + at;
}

// Numba's quicksort on a range [lo, hi] of equal keys: the place of the entry that ends up at place y.  A step parks the
// middle entry at the end, turns the others round and puts it back in the middle; ranges of fewer than 16 stay as they
// are.  So: down to the range in which y stays, and back through the steps.
__device__ __forceinline__ int source_of_equal(int y, int lo, int hi) {
  constexpr int DEPTH = 11;      // (the range is halved: no longer than 2^DEPTH * 15)
  static_assert(CAP <= 15 << DEPTH, "");
  int l[DEPTH], h[DEPTH], d = 0;
  bool there = false;
#pragma unroll
  for (int i = 0; i < DEPTH; ++i) {
    l[i] = lo, h[i] = hi;
    const int mid = (lo + hi) >> 1;
    there |= hi - lo < 15 || y == mid;
    if (!there) {
      d = i + 1;
      if (y < mid) hi = mid - 1;
      else lo = mid + 1;
    }
  }
  int q = y;
#pragma unroll
  for (int i = DEPTH - 1; i >= 0; --i)
    if (i < d) {
      const int mid = (l[i] + h[i]) >> 1;
      if (q == h[i]) q = mid;
      q = l[i] + h[i] - 1 - q;
      if (q == mid) q = h[i];
    }
  return q;
}

// A range of at most WARP_RANGE entries is partitioned by one warp, without the block's barriers: a level of 130 entries
// takes it 1,900 cycles, the block 2,300 to 2,800 (plans of 250 batches: 3.8 -> 3.5 ms).  Moves [lo, hi] (the pivot parked
// at hi) to the range that the line falls into, until it is short, its keys are equal, or the line lies between ranges.
constexpr int WARP_RANGE = 512;
struct Line {
  int lo, hi;
  bool in, equal;     // the line falls into [lo, hi]; all its keys are equal
};
struct Entries {      // of a selection: key << IDX_BITS | index
  uint32_t *e;
  __device__ uint32_t key(int i) const { return e[i] >> IDX_BITS; }
  __device__ void swap(int i, int j) const { const uint32_t x = e[i]; e[i] = e[j]; e[j] = x; }
  // median of three, the pivot at the end (the head of numba's partition step)
  __device__ void park(int lo, int hi) const {
    const int mid = (lo + hi) >> 1;
    uint32_t a = e[lo], c = e[mid], d = e[hi], t;
    if (c >> IDX_BITS < a >> IDX_BITS) t = a, a = c, c = t;
    if (d >> IDX_BITS < c >> IDX_BITS) t = d, d = c, c = t;
    if (c >> IDX_BITS < a >> IDX_BITS) t = a, a = c, c = t;
    e[lo] = a, e[mid] = d, e[hi] = c;
  }
};
// the part of the line's range behind a step whose pivot came to place m
__device__ __forceinline__ Line next_range(Line r, int m, int keep) {
  if (keep <= m) {
    r.in = keep < m;        // (keep == m: the left part stays, the rest goes; keep > lo, for the line is in the range)
    r.hi = m - 1;
    if (!r.in) r.lo = keep, r.hi = keep - 1;
  } else {
    r.in = keep > m + 1;
    r.lo = m + 1;
    if (!r.in) r.hi = r.lo - 1;
  }
  return r;
}
__device__ __forceinline__ Line partition_warp(Entries e, Line r, int keep, uint16_t *left, uint16_t *right) {
  const int lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  while (r.in && !r.equal && r.hi - r.lo >= 15) {
    const int lo = r.lo, hi = r.hi, len = hi - lo;
    const uint32_t p = e.key(hi);
    int nl = 0, nr = 0;
#pragma unroll 4
    for (int i0 = lo; i0 < hi; i0 += 32) {
      const int pos = i0 + lane;
      const uint32_t k = pos < hi ? e.key(pos) : 0;
      const uint32_t ml = __ballot_sync(0xffffffffu, pos < hi && k >= p), mr = __ballot_sync(0xffffffffu, pos < hi && k <= p);
      if (ml >> lane & 1u) left[nl + __popc(ml & lt)] = (uint16_t)pos;
      if (mr >> lane & 1u) right[nr + __popc(mr & lt)] = (uint16_t)pos;
      nl += __popc(ml);
      nr += __popc(mr);
    }
    __syncwarp();
    if (nl == len && nr == len) {
      if (lane == 0) e.swap((lo + hi) >> 1, hi);     // as before the step: source_of_equal counts from there
      r.equal = true;
      break;
    }
    const int pairs = min(nl, nr);
    int swaps = 0;
    for (int m0 = 0; m0 < pairs; m0 += 32) {
      const int m = m0 + lane, pl = m < pairs ? (int)left[m] : 0, pr = m < pairs ? (int)right[nr - 1 - m] : 0;
      if (pl < pr) e.swap(pl, pr);
      const int c = __popc(__ballot_sync(0xffffffffu, pl < pr));
      swaps += c;
      if (c < 32) break;                             // (behind a pair that does not swap, none does)
    }
    const int next_l = swaps < nl ? (int)left[swaps] : hi;
    const int m = swaps > 0 ? min(next_l, (int)right[nr - swaps]) : next_l;     // the pivot's place
    r = next_range(r, m, keep);
    __syncwarp();
    if (lane == 0) {
      e.swap(m, hi);
      if (r.in && r.hi - r.lo >= 15) e.park(r.lo, r.hi);
    }
    __syncwarp();
  }
  return r;
}

// Calls f(index) for the entries of e[0 .. n) (key << IDX_BITS | index, in list order) that numba's argsort leaves at
// `keep` or behind, 0 < keep < n (FIRST: for those before `keep`): its steps on the range that contains the line, until
// that range is short or its keys are equal.  left, right: [n].  All T threads, behind a barrier; no barrier at the end.
// aside(): work of one warp that may be done beside the first one's partition steps; returns whether it was (the same in
// every thread).
struct Nothing {
  __device__ void operator()() const {}
};
template <bool FIRST, class F, class Aside = Nothing>
__device__ __forceinline__ bool select_by_order(uint32_t *ents, int n, int keep, uint16_t *left, uint16_t *right,
                                                uint32_t *s_tot, Line *s_line, F f, Aside aside = Aside()) {
  bool done = false;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  const Entries e{ents};
  if (tid == 0) {
    *s_line = Line{0, n - 1, true, false};
    if (n - 1 >= 15) e.park(0, n - 1);
  }
  __syncthreads();
  while (true) {
    const Line r = *s_line;
    const int lo = r.lo, hi = r.hi, len = hi - lo;
    if (!r.in || r.equal || len < 15) break;
    if (len < WARP_RANGE) {
      __syncthreads();      // (everybody has read the range)
      if (warp == 0) {
        const Line z = partition_warp(e, r, keep, left, right);
        if (lane == 0) *s_line = z;
      } else if (warp == 1) {
        aside();
      }
      done = true;
      __syncthreads();
      break;
    }
    const uint32_t p = e.key(hi);
    const int items = (len + T - 1) / T, first = lo + warp * 32 * items + lane;
    uint32_t fl = 0, fr = 0, at = 0;
#pragma unroll 4
    for (int i = 0; i < items; ++i) {
      const int pos = first + 32 * i;
      const uint32_t kv = pos < hi ? e.key(pos) : 0;
      const bool l = pos < hi && kv >= p, r = pos < hi && kv <= p;
      fl |= (l ? 1u : 0u) << i;
      fr |= (r ? 1u : 0u) << i;
      at += __popc(__ballot_sync(0xffffffffu, l)) | __popc(__ballot_sync(0xffffffffu, r)) << 16;
    }
    if (lane == 0) s_tot[warp] = at;
    __syncthreads();
    const uint32_t t = s_tot[lane], all = __reduce_add_sync(0xffffffffu, t);
    at = __reduce_add_sync(0xffffffffu, lane < warp ? t : 0u);
    const int nl = all & 0xffff, nr = all >> 16;
    if (nl == len && nr == len) {       // (uniform over the block)
      if (tid == 0) {
        e.swap((lo + hi) >> 1, hi);     // as before the step: source_of_equal counts from there
        s_line->equal = true;
      }
      __syncthreads();
      break;
    }
#pragma unroll 4
    for (int i = 0; i < items; ++i) {
      const int pos = first + 32 * i;
      const bool l = (fl >> i) & 1u, r = (fr >> i) & 1u;
      const uint32_t ml = __ballot_sync(0xffffffffu, l), mr = __ballot_sync(0xffffffffu, r);
      if (l) left[(at & 0xffff) + __popc(ml & lt)] = (uint16_t)pos;
      if (r) right[(at >> 16) + __popc(mr & lt)] = (uint16_t)pos;
      at += __popc(ml) | __popc(mr) << 16;
    }
    __syncthreads();
    // the m-th of the left list swaps with the m-th from the end of the right list while it lies left of it; s_tot[0]:
    // the pivot's place
    const int pairs = min(nl, nr);
    for (int m = tid; m < pairs; m += T) {
      const int pl = left[m], pr = right[nr - 1 - m];
      if (pl >= pr) {
        if (m == 0) s_tot[0] = (uint32_t)pl;
        break;                          // (behind a pair that does not swap, none does)
      }
      const int next_l = m + 1 < nl ? (int)left[m + 1] : hi;
      if (m + 1 >= pairs || next_l >= (int)right[nr - 2 - m]) s_tot[0] = (uint32_t)min(next_l, pr);
      e.swap(pl, pr);
    }
    if (tid == 0 && pairs == 0) s_tot[0] = (uint32_t)(nl > 0 ? (int)left[0] : hi);
    __syncthreads();
    if (tid == 0) {
      const int m = (int)s_tot[0];
      const Line z = next_range(r, m, keep);
      e.swap(m, hi);
      if (z.in && z.hi - z.lo >= 15) e.park(z.lo, z.hi);
      *s_line = z;
    }
    __syncthreads();
  }
  const Line r = *s_line;
  const int lo = r.lo, hi = r.hi;
  if (r.equal) {
    for (int y = (FIRST ? lo : keep) + tid; y < (FIRST ? keep : hi + 1); y += T) f((int)(ents[source_of_equal(y, lo, hi)] & IDX));
  } else if (lo + tid <= hi) {          // (fewer than 16)
    const int pos = lo + tid;
    const uint32_t k = e.key(pos);
    int place = lo;
    for (int q = lo; q <= hi; ++q) place += e.key(q) < k || (e.key(q) == k && q < pos) ? 1 : 0;
    if ((place < keep) == FIRST) f((int)(ents[pos] & IDX));
  }
  for (int pos = (FIRST ? 0 : hi + 1) + tid; pos < (FIRST ? lo : n); pos += T) f((int)(ents[pos] & IDX));
  return done;
}

// The usual first step of a selection over a list whose keys are given by key(i): its pivot is the largest key there is,
// FAR, the right part contains the line, and nothing needs to be moved.  The step's left list is the FAR entries, its right list
// everything, so that the m-th FAR entry from the left goes to place n - 2 - m for as long as it lies left of that, and
// these places are the right part, all of one key.  Calls f(i) for the entries left at `keep` or behind and returns
// true, or returns false if the step is another one.  words: [(n + 31) / 32].  All T threads, behind a barrier.
template <class Key, class F>
__device__ __forceinline__ bool select_by_far_step(Key key, int n, int keep, Word *words, uint32_t *s_tot, F f) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int hi = n - 1, mid = hi >> 1;
  if (hi < 15) return false;
  // the parked three: a at place 0, d in the middle, the pivot c at the end
  int a = 0, c = mid, d = hi, t;
  if (key(c) < key(a)) t = a, a = c, c = t;
  if (key(d) < key(c)) t = d, d = c, c = t;
  if (key(c) < key(a)) t = a, a = c, c = t;
  if (key(c) != FAR) return false;
  const auto entry = [&](int i) { return i == 0 ? a : i == mid ? d : i; };      // i < hi
  const int n_words = (hi + 31) / 32;
#pragma unroll 4
  for (int i0 = warp * 32; i0 < hi; i0 += T) {
    const uint32_t w = __ballot_sync(0xffffffffu, i0 + lane < hi && key(entry(min(i0 + lane, hi - 1))) == FAR);
    if (lane == 0) words[i0 >> 5].bits = w;
  }
  __syncthreads();
  count_words(words, n_words, (int32_t *)s_tot);
  if (tid == 0) s_tot[0] = 0;
  __syncthreads();
  // swaps of the step: entry m at i swaps while i + m < hi - 1, which grows from entry to entry
  if (tid < n_words) {
    uint32_t w = words[tid].bits;
    const int first = 32 * tid + words[tid].before;
    int count = __popc(w);
    if (w != 0 && first + 31 - __clz(w) + count - 1 >= hi - 1) {     // (the word's last one does not)
      count = 0;
      for (; w != 0 && first + __ffs(w) - 1 + count < hi - 1; w &= w - 1) ++count;
    }
    if (count != 0) atomicAdd(&s_tot[0], (uint32_t)count);
  }
  __syncthreads();
  const int swaps = (int)s_tot[0], at = hi - 1 - swaps;
  // the pivot's place: a FAR entry that need not swap, if it lies in the middle, else where the right part begins
  bool stays = false;
  if (at >= 0 && at < hi) {
    const Word w = words[at >> 5];
    stays = bit_of(w, at) && bits_before(w, at) == swaps;
  }
  const int m = stays ? at : hi - swaps;
  if (keep <= m + 1) return false;
  // the right part: its places hi - 1, hi - 2, ... hold the first FAR entries, place hi the one after them
  for (int y = keep + tid; y <= hi; y += T) {
    const int q = source_of_equal(y, m + 1, hi);
    f(entry(bit_number(words, n_words, q == hi ? hi - m - 1 : hi - 1 - q)));
  }
  return true;
}

// MRD over lists.  Lists or candidates of more than CAP entries, or more lists than there is room for, set
// *State::failed: the kernels of planner_mrd.cu do the plan then.
bool mrd_takes(int64_t n_edges, int32_t bs);
bool mrd_always(int64_t n_edges, int32_t bs, int32_t k, int64_t n_nodes, int32_t budget);      // (it cannot fail)
int64_t mrd_workspace_bytes(int64_t n_edges, int32_t bs, int32_t k, int64_t n_nodes, int32_t budget);
int launch_mrd(const int32_t *d_nodes, const int32_t *d_nbr, int64_t n_edges, int32_t bs, int32_t k, int64_t n_nodes,
               int32_t budget, int32_t *d_plan, int64_t plan_cap, int64_t *d_plan_off, int64_t *d_stats, int32_t *d_status,
               void *d_workspace, const int32_t **d_failed, cudaStream_t s);

}  // namespace lists
}  // namespace orca
