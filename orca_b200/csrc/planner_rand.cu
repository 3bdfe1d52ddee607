// LRU and 2Q cache planning on the device (utils/cache.py:338-403 and 175-333, with read_batches :19-89).
//
// Both policies walk the batches in order and evict at random: numba's np.random.choice(..., replace=False)
// is a Fisher-Yates shuffle driven by its private Mersenne Twister, first entries kept.  How many numbers a swap
// consumes depends on the numbers (rejection sampling), but not on what is shuffled: one warp takes the generator's
// numbers 32 at a time and finds by votes which of them are accepted and for which swap.  The swaps themselves are one
// serial chain, in shared memory, and are left out where the whole list is taken whatever its order.
// The out-of-batch neighbours of all batches, without duplicates, are listed before (planner_lists.cu).  The rest is data
// parallel over the block: the reuse statistics, sets as bitmaps that list their members in ascending order by a popcount
// scan (np.where of the reference), and the LRU evictions, which are the first entries of numba's argsort of the
// last-use times: only which they are matters, so only the range that the line falls into is partitioned
// (planner_lists.cuh; tie_order.cuh for lists that do not fit shared memory).
// One CTA of 1024 threads per plan; its bound is latency, of the barriers and of the scattered loads in between.
// 250 batches of 600 edges with 20 neighbours, LRU, ms of the kernel: 19.2 with draws, swaps, bitmaps and sort in global
// memory, 9.9 with those in shared memory, 3.4 with lists in place of the tables' 24,000 entries a batch and without the
// levels of the sort that do not decide, 3.0 with the generator beside the selection and members listed by half words.
#include <algorithm>

#include "common.cuh"
#include "planner_lists.cuh"
#include "tie_shared.cuh"

namespace orca {
namespace rnd {

constexpr int T = tie::T;
constexpr int NW = tie::NW;

// numba's generator (MT19937) and its bounded draw: the low bits that cover n - 1, redrawn while >= n
struct Twister {
  static constexpr int N = 624, M = 397;
  uint32_t s[N];
  int pos;
  __device__ void seed(uint32_t x) {
    s[0] = x;
    for (int i = 1; i < N; ++i) s[i] = 1812433253u * (s[i - 1] ^ (s[i - 1] >> 30)) + (uint32_t)i;
    pos = N;
  }
  // The rest by one warp.  A chunk of 32 words needs words of later chunks (still old) and words 227 places back.
  __device__ void refill() {
    const int lane = threadIdx.x & 31;
    for (int i0 = 0; i0 < N; i0 += 32) {
      const int i = i0 + lane;
      uint32_t v = 0;
      if (i < N) {
        const uint32_t y = (s[i] & 0x80000000u) | (s[(i + 1) % N] & 0x7fffffffu);
        v = s[(i + M) % N] ^ (y >> 1) ^ ((y & 1u) ? 0x9908b0dfu : 0u);
      }
      __syncwarp();
      if (i < N) s[i] = v;
      __syncwarp();
    }
  }
  // The draws of a shuffle of n entries, from the back: entry i swaps with draw[i] (draw may be null: the generator
  // moves on all the same).  Number l of a group of 32 is accepted iff it lies below its bound, which falls by one for
  // every number accepted before it: the votes settle from the left, in two or three rounds as a rule, 33 at most.
  __device__ __noinline__ void draws(int n, int32_t *draw) {
    const int lane = threadIdx.x & 31;
    int at = pos;
    while (n > 1) {
      if (at >= N) {
        refill();
        at = 0;
      }
      const bool have = lane < N - at;
      uint32_t y = have ? s[at + lane] : 0;
      y ^= y >> 11;
      y ^= (y << 7) & 0x9d2c5680u;
      y ^= (y << 15) & 0xefc60000u;
      y ^= y >> 18;
      uint32_t accepted = 0, r = 0;
      int bound = 0;
      for (int round = 0; round <= 33; ++round) {
        bound = n - __popc(accepted & ((1u << lane) - 1u));
        r = bound > 1 ? y & (0xffffffffu >> __clz(bound - 1)) : 0;
        const uint32_t a = __ballot_sync(0xffffffffu, have && bound > 1 && r < (uint32_t)bound);
        if (a == accepted) break;
        accepted = a;
      }
      if (draw != nullptr && ((accepted >> lane) & 1u)) draw[bound - 1] = (int32_t)r;
      at += __popc(__ballot_sync(0xffffffffu, have && bound > 1));
      n -= __popc(accepted);
    }
    __syncwarp();
    if (lane == 0) pos = at;
    __syncwarp();
  }
};

// Of a plan, between the launches for its chunks of batches.
struct State {
  uint32_t rng[Twister::N];
  int32_t rng_pos, failed, n[2];      // n: LRU: cached; 2Q: fifo, lru
  int64_t used;
};

struct Work {
  State *st;
  lists::Lists lists;             // of the launch's batches
  int32_t *t0, *t1, *t2;          // [n_nodes] LRU: last use, arrival; 2Q: LRU last use, LRU arrival, FIFO arrival
  uint32_t *bm[2];                // [words] LRU: cached; 2Q: fifo, lru
  int32_t *list[4];               // [cap] member lists
  tie::Buf sort;
  int64_t cap;
  int cap_shared;                 // entries of a list in shared memory
  bool bm_shared;                 // the bitmaps lie behind them
  bool keys_fit;                  // a batch's number is a key of a selection (planner_lists.cuh)
};

// (bitmaps lie in shared memory where they fit, else in global memory, where their words are changed by atomics, which
// act in L2: they are read from there, not through L1)
__device__ __forceinline__ uint32_t word(const uint32_t *bm, int64_t i) { return *(const volatile uint32_t *)&bm[i]; }
__device__ __forceinline__ bool bit(const uint32_t *bm, int32_t v) { return (word(bm, v >> 5) >> (v & 31)) & 1u; }
__device__ __forceinline__ void set_bit(uint32_t *bm, int32_t v) { atomicOr(&bm[v >> 5], 1u << (v & 31)); }
__device__ __forceinline__ void clear_bit(uint32_t *bm, int32_t v) { atomicAnd(&bm[v >> 5], ~(1u << (v & 31))); }

// Members of a bitmap in ascending order -> out; returns their number (the same in every thread).  All T
// threads call it.  s_cnt: NW ints of shared memory.
// Bitmaps of a few words a thread are dealt out by half words, neighbouring ones to a thread: a thread then lists a handful
// of members (343 words, a word a lane of eleven warps: 5,600 cycles a batch with the copy out; half words over all of them: 3,400).
// Up to two words a thread, that is 65,536 nodes.  100 batches, words / half words, ms a plan: LRU 600 edges, budget 10,000,
// 11 k nodes 1.64 / 1.47, 33 k 1.79 / 1.64, 65 k 1.80 / 1.72; 2Q 200 edges, budget 500, 3.51 / 2.99, 3.69 / 3.26, 3.74 / 3.39; LRU
// 200 edges, budget 500, 1.57 / 1.60, 1.58 / 1.64, 1.62 / 1.72.  The kernels are made for either (FEW): with both forms in one
// kernel plans of larger graphs took 1 to 12 % longer (LRU, 200 k nodes, 600 edges, budget 10,000 2.22 for 2.18 ms, 200 edges, budget 500
// 2.05 for 1.83).
constexpr int FEW_WORDS = 2 * T;
template <bool FEW>
__device__ __forceinline__ int list_members(uint32_t *bm, int64_t words, int32_t *out, int *s_cnt) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (FEW) {
    constexpr int MOST = 2 * FEW_WORDS / T;
    const int halves = 2 * (int)words, per = (halves + T - 1) / T;
    __syncthreads();   // (earlier writes to the bitmap; earlier readers of s_cnt)
    uint32_t bits[MOST];
    int cnt = 0;
#pragma unroll
    for (int i = 0; i < MOST; ++i) {
      const int at = tid * per + i;
      bits[i] = i < per && at < halves ? word(bm, at >> 1) >> 16 * (at & 1) & 0xffffu : 0u;
      cnt += __popc(bits[i]);
    }
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    if (lane == 31) s_cnt[warp] = incl;
    __syncthreads();
    const int x = s_cnt[lane];
    int pos = __reduce_add_sync(0xffffffffu, lane < warp ? x : 0) + incl - cnt;
    const int n = __reduce_add_sync(0xffffffffu, x);
#pragma unroll
    for (int i = 0; i < MOST; ++i)
      for (uint32_t b = bits[i]; b != 0; b &= b - 1) out[pos++] = 16 * (tid * per + i) + __ffs(b) - 1;
    __syncthreads();
    return n;
  }
  const int wchunk = (int)(((words + NW - 1) / NW + 31) & ~31ll);
  __syncthreads();   // (earlier writes to the bitmap; earlier readers of s_cnt)
  int cnt = 0;
  for (int j = lane; j < wchunk; j += 32) {
    const int64_t wi = (int64_t)warp * wchunk + j;
    if (wi < words) cnt += __popc(word(bm, wi));
  }
  for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
  if (lane == 0) s_cnt[warp] = cnt;
  __syncthreads();
  int n = 0, base = 0;
  for (int i = 0; i < NW; ++i) {
    const int c = s_cnt[i];
    if (i < warp) base += c;
    n += c;
  }
  for (int j = 0; j < wchunk; j += 32) {
    const int64_t wi = (int64_t)warp * wchunk + j + lane;
    uint32_t bits = 0;
    if (wi < words) bits = word(bm, wi);
    const int c = __popc(bits);
    int incl = c;
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    int pos = base + incl - c;
    base += __shfl_sync(0xffffffffu, incl, 31);
    while (bits) {
      out[pos++] = (int32_t)(wi * 32 + (__ffs(bits) - 1));
      bits &= bits - 1;
    }
  }
  __syncthreads();
  return n;
}

// Fisher-Yates of x[0 .. n) from the back, as numba shuffles; the caller keeps the first entries.  `any_order`: the
// caller keeps all of them, so that only the generator has to move.  All T threads call it.
__device__ void shuffle(const Work &w, Twister &rng, int32_t *x, int n, bool any_order) {
  __syncthreads();
  if (any_order) {
    if (threadIdx.x < 32) rng.draws(n, nullptr);
    __syncthreads();
    return;
  }
  const bool fits = 8ll * n <= (int64_t)tie::Shared::BYTES * w.cap_shared;
  int32_t *at = fits ? (int32_t *)tie::smem : x, *draw = fits ? at + n : w.sort.lpos;
  if (threadIdx.x < 32) rng.draws(n, draw);
  if (fits)
    for (int i = threadIdx.x; i < n; i += T) at[i] = x[i];
  __syncthreads();
  if (threadIdx.x == 0)
    for (int i = n - 1; i > 0; --i) {
      const int j = draw[i];
      const int32_t a = at[i];
      at[i] = at[j];
      at[j] = a;
    }
  __syncthreads();
  if (fits)
    for (int i = threadIdx.x; i < n; i += T) x[i] = at[i];
  __syncthreads();
}

// the first `count` entries, fewer than n, of numba's argsort of key[ids[i]] (i < n): calls f(id) for each of them.
// aside: select_by_order's; `beside` is set if it was done
template <class F, class Aside>
__device__ bool for_first_by_key(const Work &w, const int32_t *ids, int n, int count, const int32_t *key, int *s_a,
                                 int *s_b, F f, Aside aside, bool &beside) {
  if (count >= n) {
    for (int i = threadIdx.x; i < n; i += T) f(ids[i]);
    __syncthreads();
    return true;
  }
  if (n <= w.cap_shared && w.keys_fit) {
    uint32_t *e = (uint32_t *)tie::smem;
    uint16_t *left = (uint16_t *)(e + w.cap_shared), *right = left + w.cap_shared;
    for (int i = threadIdx.x; i < n; i += T) e[i] = (uint32_t)key[ids[i]] << lists::IDX_BITS | (uint32_t)i;
    __syncthreads();
    __shared__ lists::Line s_line;
    beside = lists::select_by_order<true>(e, n, count, left, right, (uint32_t *)s_a, &s_line, [&](int i) { f(ids[i]); }, aside);
    __syncthreads();
    return true;
  }
  for (int i = threadIdx.x; i < n; i += T) w.sort.e[i] = ((uint64_t)(uint32_t)key[ids[i]] << 32) | (uint32_t)i;
  __syncthreads();
  if (!tie::sort_first(w.sort, n, count, s_a, s_b)) return false;
  for (int pos = threadIdx.x; pos < n; pos += T)
    if (tie::place_of(w.sort, pos, count) >= 0) f(ids[(uint32_t)w.sort.e[pos]]);
  __syncthreads();
  return true;
}

// The bitmaps of a plan (SH: in shared memory, behind the lists).
constexpr int N_BM = 2;
template <bool SH>
__device__ __forceinline__ uint32_t *bitmap(const Work &w, int i, int64_t words) {
  return SH ? (uint32_t *)(tie::smem + tie::Shared::BYTES * w.cap_shared) + i * words : w.bm[i];
}
// at the start of a launch: the first one's are empty, the others' as the one before left them (LOAD: false: that)
template <bool SH, bool LOAD>
__device__ void move_bitmaps(const Work &w, int64_t words, bool first) {
  for (int64_t i = threadIdx.x; i < N_BM * words; i += T) {
    const int m = (int)(i / words);
    const int64_t j = i % words;
    if (LOAD && first) bitmap<SH>(w, m, words)[j] = 0;
    else if (SH && LOAD) bitmap<SH>(w, m, words)[j] = w.bm[m][j];
    else if (SH) w.bm[m][j] = bitmap<SH>(w, m, words)[j];
  }
}

// Deals the out-of-batch neighbours of list a out to three lists: kind(v, entries of the table) says which (0 .. 2, else
// none).  The lists stay in ascending order; n: their lengths, the same in every thread.  s_cnt: NW words.  All T threads;
// ends behind a barrier.
template <class Kind>
__device__ __forceinline__ void deal_neighbors(const lists::Lists &l, lists::Span a, int32_t *const (&out)[3], int (&n)[3],
                                               uint32_t *s_cnt, Kind kind) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  const int n_list = a.n;
  const int32_t *id = l.id + a.at, *mult = l.mult + a.at;
  n[0] = n[1] = n[2] = 0;
  for (int i0 = 0; i0 < n_list; i0 += T) {
    const int i = i0 + tid;
    const int32_t v = i < n_list ? id[i] : lists::TARGET;
    const int k = v >= 0 ? kind(v, mult[i]) : 3;
    uint32_t m[3], c = 0;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      m[j] = __ballot_sync(0xffffffffu, k == j);
      c |= __popc(m[j]) << 10 * j;       // (32 at most)
    }
    __syncthreads();      // (s_cnt of the turn before)
    if (lane == 0) s_cnt[warp] = c;
    __syncthreads();
    const uint32_t x = s_cnt[lane];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const int mine = (x >> 10 * j) & 1023u;
      const int before = __reduce_add_sync(0xffffffffu, lane < warp ? mine : 0);
      if (k == j) out[j][n[j] + before + __popc(m[j] & lt)] = v;
      n[j] += __reduce_add_sync(0xffffffffu, mine);
    }
  }
  __syncthreads();
}

struct Totals {
  long long reuse = 0, recompute = 0, dist = 0;
};
__device__ void write_totals(const Totals &t, int64_t *stats) {
  long long a = t.reuse, b = t.recompute, c = t.dist;
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
    c += __shfl_xor_sync(0xffffffffu, c, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd((unsigned long long *)&stats[0], (unsigned long long)a);
    atomicAdd((unsigned long long *)&stats[1], (unsigned long long)b);
    atomicAdd((unsigned long long *)&stats[2], (unsigned long long)c);
  }
}

// The state of a plan at the start and at the end of a launch; false: an earlier launch has failed.
__device__ __forceinline__ bool resume(const Work &w, Twister &rng, uint32_t seed, bool first) {
  if (first) {
    if (threadIdx.x == 0) rng.seed(seed);
    return true;
  }
  if (w.st->failed) return false;
  for (int i = threadIdx.x; i < Twister::N; i += T) rng.s[i] = w.st->rng[i];
  if (threadIdx.x == 0) rng.pos = w.st->rng_pos;
  return true;
}
__device__ __forceinline__ void suspend(const Work &w, const Twister &rng, bool failed, int n0, int n1, int64_t used) {
  for (int i = threadIdx.x; i < Twister::N; i += T) w.st->rng[i] = rng.s[i];
  if (threadIdx.x == 0) {
    w.st->rng_pos = rng.pos, w.st->failed = failed;
    w.st->n[0] = n0, w.st->n[1] = n1, w.st->used = used;
  }
}

// ------------------------------------------------------------------------------ LRU (utils/cache.py:338-403)
template <bool SH, bool FEW>
__global__ void __launch_bounds__(T, 1) lru_kernel(int64_t b0, int64_t b1, int64_t nb, int64_t n_nodes, int32_t budget,
                                                uint32_t seed, Work w, int32_t *plan, int64_t plan_cap, int64_t *plan_off,
                                                int64_t *stats, int32_t *status) {
  __shared__ Twister rng;
  __shared__ int s_a[NW], s_b[NW];
  const int tid = threadIdx.x;
  const int64_t words = (n_nodes + 31) / 32;
  if (!resume(w, rng, seed, b0 == 0)) return;
  move_bitmaps<SH, true>(w, words, b0 == 0);
  uint32_t *cached = bitmap<SH>(w, 0, words);
  int32_t *used_at = w.t0, *arrived = w.t1;
  int32_t *cand = w.list[0];
  for (int64_t v = tid; b0 == 0 && v < n_nodes; v += T) {
    used_at[v] = 0;
    arrived[v] = 0;
  }
  __syncthreads();
  Totals tot;
  int64_t used = b0 == 0 ? 0 : w.st->used;
  int n_held = b0 == 0 ? 0 : w.st->n[0];      // members of `cached`, listed in `held`
  // (no more than the budget; a plan that would not fit is listed elsewhere)
  const auto listed_at = [&](int64_t at) { return at + min((int64_t)budget, n_nodes) <= plan_cap ? plan + at : w.list[1]; };
  int32_t *held = listed_at(used - n_held);
  bool failed = false;
  lists::Span span_next = w.lists.span[0];
  for (int64_t b = b0; b < b1; ++b) {
    const lists::Span span = span_next;
    if (b + 1 < b1) span_next = w.lists.span[b + 1 - b0];
    int32_t *const out[3] = {cand, nullptr, nullptr};
    int n[3];
    deal_neighbors(w.lists, span, out, n, (uint32_t *)s_a, [&](int32_t v, int m) {
      if (!bit(cached, v)) {
        tot.recompute += m;
        return 0;
      }
      tot.reuse += m;
      tot.dist += (b - arrived[v]) * m;
      used_at[v] = (int32_t)b;
      return 3;
    });
    const int n_cand = n[0];
    const int room = budget - n_held;
    const int evict = room >= n_cand ? 0 : min(n_cand - room, n_held);
    const int take = (evict + room >= n_cand) ? n_cand : budget;
    // (where all candidates are taken only the generator moves: beside the selection, 3,600 of 27,500 cycles a batch)
    bool drawn = false;
    if (evict != 0) {
      if (!for_first_by_key(w, held, n_held, evict, used_at, s_a, s_b, [&](int32_t v) { clear_bit(cached, v); },
                            [&]() { if (take == n_cand) rng.draws(n_cand, nullptr); }, drawn)) {
        if (tid == 0) report(status, ORCA_E_TIMEOUT, (int)b);
        failed = true;
        break;
      }
    }
    if (!drawn || take != n_cand) shuffle(w, rng, cand, n_cand, take == n_cand);
    for (int i = tid; i < take; i += T) {
      const int32_t v = cand[i];
      set_bit(cached, v);
      used_at[v] = arrived[v] = (int32_t)b;
    }
    held = listed_at(used);
    n_held = list_members<FEW>(cached, words, held, s_a);
    if (used + n_held > plan_cap) {
      if (tid == 0) report(status, ORCA_E_CAPACITY, (int)b);
      failed = true;
      break;
    }
    if (held != plan + used)
      for (int i = tid; i < n_held; i += T) plan[used + i] = held[i];
    if (tid == 0) plan_off[b] = used;
    used += n_held;
    __syncthreads();
  }
  write_totals(tot, stats);
  if (b1 < nb) {
    suspend(w, rng, failed, n_held, 0, used);
    move_bitmaps<SH, false>(w, words, false);
  }
  if (tid == 0 && (failed || b1 == nb)) plan_off[nb] = used;
}

// ------------------------------------------------------------------------------ 2Q (utils/cache.py:175-333)
// a FIFO half and an LRU half of budget / 2 entries each
template <bool SH, bool FEW>
__global__ void __launch_bounds__(T, 1) twoq_kernel(int64_t b0, int64_t b1, int64_t nb, int64_t n_nodes, int32_t budget,
                                                 uint32_t seed, Work w, int32_t *plan, int64_t plan_cap, int64_t *plan_off,
                                                 int64_t *stats, int32_t *status) {
  __shared__ Twister rng;
  __shared__ int s_a[NW], s_b[NW];
  const int tid = threadIdx.x;
  const int64_t words = (n_nodes + 31) / 32;
  const int half = budget / 2;
  if (!resume(w, rng, seed, b0 == 0)) return;
  move_bitmaps<SH, true>(w, words, b0 == 0);
  uint32_t *fifo = bitmap<SH>(w, 0, words), *lru = bitmap<SH>(w, 1, words);
  int32_t *lru_used = w.t0, *lru_arr = w.t1, *fifo_arr = w.t2;
  int32_t *promote = w.list[0], *fresh = w.list[1], *touched = w.list[2], *ids = w.list[3];
  for (int64_t v = tid; b0 == 0 && v < n_nodes; v += T) {
    lru_used[v] = lru_arr[v] = fifo_arr[v] = 0;
  }
  __syncthreads();
  Totals tot;
  int64_t used = b0 == 0 ? 0 : w.st->used;
  int n_fifo = b0 == 0 ? 0 : w.st->n[0], n_lru = b0 == 0 ? 0 : w.st->n[1];
  bool failed = false;
  lists::Span span_next = w.lists.span[0];
  for (int64_t b = b0; b < b1 && !failed; ++b) {
    const lists::Span span = span_next;
    if (b + 1 < b1) span_next = w.lists.span[b + 1 - b0];
    const int32_t now = (int32_t)b;
    int32_t *const out[3] = {promote, fresh, touched};
    int n_out[3];
    deal_neighbors(w.lists, span, out, n_out, (uint32_t *)s_a, [&](int32_t v, int m) {
      if (bit(fifo, v)) {
        tot.reuse += m;
        tot.dist += (long long)(now - fifo_arr[v]) * m;
        return 0;
      }
      if (bit(lru, v)) {
        tot.reuse += m;
        tot.dist += (long long)(now - lru_arr[v]) * m;
        return 2;
      }
      tot.recompute += m;
      return 1;
    });
    const int n_promote = n_out[0], n_fresh = n_out[1], n_touched = n_out[2];
    // ---- FIFO half
    const int fifo_kept = n_fifo - n_promote, fifo_room = half - fifo_kept;
    for (int i = tid; i < n_promote; i += T) clear_bit(fifo, promote[i]);
    __syncthreads();
    if (n_fresh <= fifo_room) {
      for (int i = tid; i < n_fresh; i += T) {
        set_bit(fifo, fresh[i]);
        fifo_arr[fresh[i]] = now;
      }
      n_fifo = fifo_kept + n_fresh;
    } else if (n_fresh >= half) {
      for (int i = tid; i < n_fresh; i += T) ids[i] = fresh[i];
      for (int64_t i = tid; i < words; i += T) fifo[i] = 0;
      for (int64_t v = tid; v < n_nodes; v += T) fifo_arr[v] = 0;
      __syncthreads();
      shuffle(w, rng, ids, n_fresh, n_fresh == half);
      for (int i = tid; i < half; i += T) {
        set_bit(fifo, ids[i]);
        fifo_arr[ids[i]] = now;
      }
      n_fifo = half;
    } else {
      const int n_ids = list_members<FEW>(fifo, words, ids, s_a);
      shuffle(w, rng, ids, n_ids, false);
      for (int i = tid; i < n_fresh - fifo_room; i += T) clear_bit(fifo, ids[i]);
      __syncthreads();
      for (int i = tid; i < n_fresh; i += T) {
        set_bit(fifo, fresh[i]);
        fifo_arr[fresh[i]] = now;
      }
      n_fifo = half;
    }
    __syncthreads();
    // ---- LRU half
    for (int i = tid; i < n_touched; i += T) lru_used[touched[i]] = now;
    __syncthreads();
    const int lru_room = half - n_lru, lru_evictable = n_lru - n_touched;
    auto admit = [&](int32_t v) {
      set_bit(lru, v);
      lru_used[v] = now;
      lru_arr[v] = fifo_arr[v];
    };
    if (n_promote <= lru_room) {
      for (int i = tid; i < n_promote; i += T) admit(promote[i]);
      n_lru += n_promote;
    } else if (n_promote <= lru_room + lru_evictable) {
      const int n_ids = list_members<FEW>(lru, words, ids, s_a);
      bool beside = false;
      if (!for_first_by_key(w, ids, n_ids, n_promote - lru_room, lru_used, s_a, s_b,
                            [&](int32_t v) { clear_bit(lru, v); }, lists::Nothing(), beside)) {
        if (tid == 0) report(status, ORCA_E_TIMEOUT, (int)b);
        failed = true;
        continue;
      }
      for (int i = tid; i < n_promote; i += T) admit(promote[i]);
      n_lru = half;
    } else {
      const int n_ids = list_members<FEW>(lru, words, ids, s_a);
      for (int i = tid; i < n_ids; i += T)
        if (lru_used[ids[i]] < now) clear_bit(lru, ids[i]);
      __syncthreads();
      for (int i = tid; i < n_promote; i += T) ids[i] = promote[i];
      __syncthreads();
      shuffle(w, rng, ids, n_promote, false);
      for (int i = tid; i < half - n_touched; i += T) admit(ids[i]);
      n_lru = half;
    }
    // ---- plan = FIFO ids ascending, then LRU ids ascending
    n_fifo = list_members<FEW>(fifo, words, ids, s_a);
    if (used + n_fifo > plan_cap) {
      if (tid == 0) report(status, ORCA_E_CAPACITY, (int)b);
      failed = true;
      continue;
    }
    for (int i = tid; i < n_fifo; i += T) plan[used + i] = ids[i];
    n_lru = list_members<FEW>(lru, words, ids, s_a);
    if (used + n_fifo + n_lru > plan_cap) {
      if (tid == 0) report(status, ORCA_E_CAPACITY, (int)b);
      failed = true;
      continue;
    }
    for (int i = tid; i < n_lru; i += T) plan[used + n_fifo + i] = ids[i];
    if (tid == 0) plan_off[b] = used;
    used += n_fifo + n_lru;
    __syncthreads();
  }
  write_totals(tot, stats);
  if (b1 < nb) {
    suspend(w, rng, failed, n_fifo, n_lru, used);
    move_bitmaps<SH, false>(w, words, false);
  }
  if (tid == 0 && (failed || b1 == nb)) plan_off[nb] = used;
}

// Batches whose lists lie in memory at a time: as many as fit 128 MB (670,000 edges with 20 neighbours, 600 a batch, are one
// launch of 16.1 ms; with 64 MB they are two, which take 16.3: lists that nothing runs beside, and state and bitmaps).
constexpr int64_t LISTS = 128 << 20;
static int64_t chunk_of(int64_t nb, int32_t bs, int32_t k, int64_t n_nodes) {
  return std::min(nb, std::max<int64_t>(1, LISTS / (8 * lists::stride_of(bs, k, n_nodes))));
}

struct Layout {
  int64_t st, id, mult, span, scratch, t[3], bm[N_BM], list[4], sort, total, cap;
};
static Layout layout(int64_t n_edges, int32_t bs, int32_t k, int64_t n_nodes, int32_t budget) {
  Layout L;
  const int64_t words = (n_nodes + 31) / 32;
  L.cap = std::max<int64_t>(2ll * bs * k, budget) + 64;
  int64_t at = 0;
  auto take = [&](int64_t bytes) {
    const int64_t o = at;
    at += (bytes + 255) & ~255ll;
    return o;
  };
  const int64_t stride = lists::stride_of(bs, k, n_nodes), chunk = chunk_of((n_edges + bs - 1) / bs, bs, k, n_nodes);
  L.st = take(sizeof(State));
  L.id = take(chunk * stride * 4);
  L.mult = take(chunk * stride * 4);
  L.span = take(chunk * sizeof(lists::Span));
  L.scratch = take(lists::scratch_bytes(chunk, n_nodes));
  for (int i = 0; i < 3; ++i) L.t[i] = take(n_nodes * 4);
  for (int i = 0; i < N_BM; ++i) L.bm[i] = take(words * 4);
  for (int i = 0; i < 4; ++i) L.list[i] = take(L.cap * 4);
  L.sort = take(tie::buf_bytes(L.cap) + 7 * 256);
  L.total = at;
  return L;
}

}  // namespace rnd
}  // namespace orca

using namespace orca;

extern "C" int64_t orca_plan_mrd_workspace_bytes(int64_t n_edges, int32_t bs, int32_t k, int64_t n_nodes, int32_t budget);
extern "C" int orca_plan_mrd(const int32_t *d_nodes, int64_t n_edges, int32_t bs, int32_t k, const int32_t *d_nbr,
                             int64_t n_nodes, int32_t budget, int32_t *d_plan_flat, int64_t plan_cap,
                             int64_t *d_plan_off, int64_t *d_stats, int32_t *d_status, void *d_workspace,
                             int64_t workspace_bytes, void *stream);

extern "C" int64_t orca_plan_device_workspace_bytes(int32_t strategy, int64_t n_edges, int32_t bs, int32_t k,
                                                    int64_t n_nodes, int32_t budget) {
  if (strategy == 0) return orca_plan_mrd_workspace_bytes(n_edges, bs, k, n_nodes, budget);
  if (strategy < 0 || strategy > 2 || n_edges < 0 || bs <= 0 || k < 1 || n_nodes <= 0 || budget <= 0) return -1;
  return rnd::layout(n_edges, bs, k, n_nodes, budget).total;
}

extern "C" int orca_plan_device(int32_t strategy, const int32_t *d_nodes, int64_t n_edges, int32_t bs, int32_t k,
                                const int32_t *d_nbr, int64_t n_nodes, int32_t budget, uint32_t seed,
                                int32_t *d_plan_flat, int64_t plan_cap, int64_t *d_plan_off, int64_t *d_stats,
                                int32_t *d_status, void *d_workspace, int64_t workspace_bytes, void *stream) {
  if (strategy == 0)
    return orca_plan_mrd(d_nodes, n_edges, bs, k, d_nbr, n_nodes, budget, d_plan_flat, plan_cap, d_plan_off, d_stats,
                         d_status, d_workspace, workspace_bytes, stream);
  ORCA_CHECK_ARG(strategy == 1 || strategy == 2);
  ORCA_CHECK_ARG(d_nodes && d_nbr && d_plan_flat && d_plan_off && d_stats && d_status && d_workspace);
  ORCA_CHECK_ARG(n_edges >= 0 && bs > 0 && k >= 1 && k <= ORCA_MAX_K && n_nodes > 0 && budget > 0);
  ORCA_CHECK_ARG(n_nodes < (1ll << 31) && (n_edges + bs - 1) / bs < (1ll << 30) && 2ll * bs * k < (1ll << 30));
  ORCA_CHECK_ARG(((uintptr_t)d_workspace & 255) == 0);
  const rnd::Layout L = rnd::layout(n_edges, bs, k, n_nodes, budget);
  if (workspace_bytes < L.total)
    return set_error(ORCA_E_CAPACITY, "orca_plan_device: workspace of %lld bytes, %lld needed",
                     (long long)workspace_bytes, (long long)L.total);
  char *base = (char *)d_workspace;
  rnd::Work w;
  const int64_t nb = (n_edges + bs - 1) / bs;
  w.st = (rnd::State *)(base + L.st);
  w.lists = lists::Lists{(int32_t *)(base + L.id), (int32_t *)(base + L.mult), (lists::Span *)(base + L.span),
                         lists::stride_of(bs, k, n_nodes), nullptr, 0, nullptr};
  w.keys_fit = nb < (int64_t)lists::FAR;
  w.t0 = (int32_t *)(base + L.t[0]);
  w.t1 = (int32_t *)(base + L.t[1]);
  w.t2 = (int32_t *)(base + L.t[2]);
  for (int i = 0; i < rnd::N_BM; ++i) w.bm[i] = (uint32_t *)(base + L.bm[i]);
  for (int i = 0; i < 4; ++i) w.list[i] = (int32_t *)(base + L.list[i]);
  w.cap = L.cap;
  {
    char *p = base + L.sort;
    auto take = [&](int64_t bytes) {
      char *o = p;
      p += (bytes + 255) & ~255ll;
      return o;
    };
    w.sort.e = (uint64_t *)take(L.cap * 8);
    w.sort.seg = (int2 *)take(L.cap * 8);
    w.sort.pre = (int2 *)take(L.cap * 8);
    w.sort.lpos = (int32_t *)take(L.cap * 4);
    w.sort.rpos = (int32_t *)take(L.cap * 4);
    w.sort.pivot = (int32_t *)take(L.cap * 4);
    w.sort.swaps = (int32_t *)take(2 * L.cap * 4);
    w.sort.cap = L.cap;
  }
  // Shared memory: lists first, then two bitmaps where they fit (up to some 600,000 nodes: each of their scattered reads
  // costs a trip to L2 otherwise).  The lists that are selected from are no longer than the budget; there is room for
  // those, and for the shuffles of 7000 entries.
  constexpr int64_t per = tie::Shared::BYTES, most = per * tie::SHARED_MAX;
  const int64_t bitmaps = rnd::N_BM * ((n_nodes + 31) / 32) * 4;
  w.cap_shared = (int)((std::min({L.cap, n_nodes, std::max<int64_t>(budget, 4096), (int64_t)tie::SHARED_MAX}) + 15) & ~15ll);
  if (per * w.cap_shared + bitmaps > most && per * (budget + 16ll) + bitmaps <= most)
    w.cap_shared = (int)(((most - bitmaps) / per) & ~15ll);
  w.bm_shared = per * w.cap_shared + bitmaps <= most;
  const int smem = (int)(per * w.cap_shared + (w.bm_shared ? bitmaps : 0));
  cudaStream_t s = (cudaStream_t)stream;
  ORCA_CUDA(cudaMemsetAsync(d_stats, 0, 3 * sizeof(int64_t), s));
  if (n_edges == 0) {
    ORCA_CUDA(cudaMemsetAsync(d_plan_off, 0, sizeof(int64_t), s));
    return ORCA_OK;
  }
  const bool few = (n_nodes + 31) / 32 <= rnd::FEW_WORDS;
  auto kernel = strategy == 1 ? (w.bm_shared ? (few ? rnd::lru_kernel<true, true> : rnd::lru_kernel<true, false>)
                                             : (few ? rnd::lru_kernel<false, true> : rnd::lru_kernel<false, false>))
                              : (w.bm_shared ? (few ? rnd::twoq_kernel<true, true> : rnd::twoq_kernel<true, false>)
                                             : (few ? rnd::twoq_kernel<false, true> : rnd::twoq_kernel<false, false>));
  ORCA_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const int64_t chunk = rnd::chunk_of(nb, bs, k, n_nodes);
  for (int64_t b0 = 0; b0 < nb; b0 += chunk) {
    const int64_t b1 = std::min(nb, b0 + chunk);
    const int rc = lists::launch_batch_lists(d_nodes, d_nbr, n_edges, bs, k, n_nodes, b0, b1, w.lists, base + L.scratch,
                                             nullptr, 0, s);
    if (rc != ORCA_OK) return rc;
    kernel<<<1, rnd::T, smem, s>>>(b0, b1, nb, n_nodes, budget, seed, w, d_plan_flat, plan_cap, d_plan_off, d_stats, d_status);
    ORCA_COUNT_LAUNCH();
    ORCA_LAUNCH_CHECK();
  }
  return ORCA_OK;
}
