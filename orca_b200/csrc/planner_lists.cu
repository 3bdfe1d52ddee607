// Cache plans from lists of distinct nodes (utils/cache.py:19-166, MRD).
//
// The policy is sequential over batches, so a plan takes as long as one batch's step times their number.  Most of what a
// step used to do needs no earlier batch, and is done for all batches at once, a block per batch:
//   batch_lists_kernel   the distinct nodes of a batch in ascending order, with their number of table entries: 40,000
//                        table entries of a batch of 2000 edges are 900 endpoints and 550 out-of-batch neighbours
//   sort_plan_kernel     the order of a plan: the first `budget` places of numba's argsort of a batch's candidates
// What is left to one block, batch after batch (mrd_lists_kernel): candidates = cached | distinct nodes, and WHICH of
// them the sort leaves in its first `budget` places.  For that, of numba's quicksort (tie_order.cuh) only the steps on
// the range that the budget line falls into are needed, one or two as a rule: two candidates in three share the largest
// key, which is the first pivot then, and where the equal keys of a range end up follows from its length alone.
// 200 batches of 2000 edges, 10,700 candidates each, ms of kernels: 24.4 with the kernels of planner_mrd.cu, which walk
// tables and sort whole lists batch after batch on a cluster of 16 SMs, 3.64 here: lists 0.14, next uses 0.34, the serial
// step 2.88 (14 us a batch: the block's instructions and barriers), orders 0.29.
#include <algorithm>

#include "common.cuh"
#include "context.cuh"
#include "host_threads.cuh"
#include "planner_lists.cuh"

namespace orca {
namespace lists {

// ------------------------------------------------------------------------------ queries
// [times][sources][destinations] of the edges -> the query list and its times
__global__ void __launch_bounds__(256) queries_kernel(const double *ts, const int32_t *src, const int32_t *dst, int64_t n_edges,
                                                      int32_t bs, int32_t *nodes, double *out_ts) {
  for (int64_t i = blockIdx.x * 256ll + threadIdx.x; i < n_edges; i += gridDim.x * 256ll) {
    const int64_t b = i / bs, lo = b * bs, n = min((int64_t)bs, n_edges - lo), at = 2 * lo + (i - lo);
    nodes[at] = src[i];
    nodes[at + n] = dst[i];
    out_ts[at] = out_ts[at + n] = ts[i];
  }
}

// ------------------------------------------------------------------------------ lists
// One block a batch, blocks walk the batches.  Two bitmaps over the nodes (the batch's nodes, its endpoints) and the
// prefix counts of the first, in global memory, left empty.  Bound by the latency of the table entries' lookups.
__global__ void __launch_bounds__(T) batch_lists_kernel(const int32_t *nodes, const int32_t *nbr, int64_t n_edges, int32_t bs,
                                                        int32_t k, int64_t n_nodes, int64_t b0, int64_t b1, Lists l,
                                                        uint32_t *bitmaps, int32_t *code, int32_t code_init) {
  __shared__ int s_cnt[NW];
  __shared__ int64_t s_at;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t words = (n_nodes + 31) / 32;
  uint32_t *all = bitmaps + blockIdx.x * 3 * words, *target = all + words;
  int32_t *before = (int32_t *)(target + words);
  for (int64_t i = tid; i < 2 * words; i += T) all[i] = 0;
  if (code != nullptr)
    for (int64_t v = blockIdx.x * T + tid; v < n_nodes; v += (int64_t)gridDim.x * T) code[v] = code_init;
  __syncthreads();
  const int64_t chunk = ((words + NW - 1) / NW + 31) & ~31ll;     // words of a warp
  constexpr int STEP = 8;
  for (int64_t b = b0 + blockIdx.x; b < b1; b += gridDim.x) {
    const int64_t s = b * bs;
    const int m2 = 2 * (int)(min(n_edges, s + bs) - s);
    const int32_t *q = nodes + 2 * s, *tab = nbr + 2 * s * k;
    for (int i = tid; i < m2; i += T) {
      const int32_t v = q[i];
      const uint32_t bit = 1u << (v & 31);
      if (!(__ldcg(&target[v >> 5]) & bit)) {
        atomicOr(&target[v >> 5], bit);
        atomicOr(&all[v >> 5], bit);
      }
    }
    __syncthreads();
    // f(v) for the out-of-batch entries of the table, several at a time: their lookups overlap
    const auto neighbors = [&](auto f) {
      for (int64_t i0 = tid; i0 < (int64_t)m2 * k; i0 += STEP * T) {
        int32_t v[STEP];
        uint32_t w[STEP];
#pragma unroll
        for (int u = 0; u < STEP; ++u) v[u] = i0 + u * T < (int64_t)m2 * k ? tab[i0 + u * T] : 0;
#pragma unroll
        for (int u = 0; u < STEP; ++u) w[u] = v[u] != 0 ? __ldcg(&target[v[u] >> 5]) : 0;
#pragma unroll
        for (int u = 0; u < STEP; ++u)
          if (v[u] != 0 && !((w[u] >> (v[u] & 31)) & 1u)) f(v[u]);
      }
    };
    neighbors([&](int32_t v) {
      const uint32_t bit = 1u << (v & 31);
      if (!(__ldcg(&all[v >> 5]) & bit)) atomicOr(&all[v >> 5], bit);
    });
    __syncthreads();
    int cnt = 0;
    for (int64_t j = lane; j < chunk; j += 32) {
      const int64_t wi = warp * chunk + j;
      if (wi < words) cnt += __popc(__ldcg(&all[wi]));
    }
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (lane == 0) s_cnt[warp] = cnt;
    __syncthreads();
    const int c_lane = s_cnt[lane];
    int base = __reduce_add_sync(0xffffffffu, lane < warp ? c_lane : 0);
    const int n = __reduce_add_sync(0xffffffffu, c_lane);
    if (tid == 0) {
      int64_t at = (b - b0) * l.stride;
      if (l.stride == 0) {
        at = n <= CAP ? (int64_t)atomicAdd(l.used, (unsigned long long)n) : l.room;
        if (at + n > l.room) {
          at = -1;
          *l.failed = 1;
        }
      }
      s_at = at;
      l.span[b - b0] = Span{max(at, (int64_t)0), at < 0 ? 0 : n};
    }
    __syncthreads();
    if (s_at < 0) {      // (nobody looks at these lists)
      for (int64_t i = tid; i < 2 * words; i += T) all[i] = 0;
      __syncthreads();
      continue;
    }
    int32_t *id = l.id + s_at, *mult = l.mult + s_at;
    for (int64_t j = 0; j < chunk; j += 32) {
      const int64_t wi = warp * chunk + j + lane;
      uint32_t bits = wi < words ? __ldcg(&all[wi]) : 0;
      const int c = __popc(bits);
      if (!__any_sync(0xffffffffu, c != 0)) continue;
      int incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
      }
      int pos = base + incl - c;
      base += __shfl_sync(0xffffffffu, incl, 31);
      if (bits != 0) {
        before[wi] = pos;
        const uint32_t t = __ldcg(&target[wi]);
        for (; bits != 0; bits &= bits - 1, ++pos) {
          const int bit = __ffs(bits) - 1;
          id[pos] = (int32_t)(wi * 32 + bit) | ((t >> bit) & 1u ? TARGET : 0);
          mult[pos] = 0;
        }
      }
    }
    __syncthreads();
    neighbors([&](int32_t v) {
      atomicAdd(&mult[__ldcg(&before[v >> 5]) + __popc(__ldcg(&all[v >> 5]) & ((1u << (v & 31)) - 1u))], 1);
    });
    __syncthreads();
    for (int i = tid; i < n; i += T) {
      const int32_t v = __ldcg(&id[i]) & ~TARGET;
      all[v >> 5] = 0;
      target[v >> 5] = 0;
    }
    __syncthreads();
  }
}

int launch_batch_lists(const int32_t *d_nodes, const int32_t *d_nbr, int64_t n_edges, int32_t bs, int32_t k, int64_t n_nodes,
                       int64_t b0, int64_t b1, const Lists &l, void *d_scratch, int32_t *d_code, int32_t code_init,
                       cudaStream_t s) {
  const Ctx *c = cur();
  if (c == nullptr) return set_error(ORCA_E_CUDA, "launch_batch_lists: no context for the current device");
  const int grid = blocks_for(b1 - b0, n_nodes, std::min(c->sm_count, MOST_BLOCKS));
  batch_lists_kernel<<<grid, T, 0, s>>>(d_nodes, d_nbr, n_edges, bs, k, n_nodes, b0, b1, l, (uint32_t *)d_scratch, d_code,
                                        code_init);
  ORCA_COUNT_LAUNCH();
  ORCA_LAUNCH_CHECK();
  return ORCA_OK;
}

// ------------------------------------------------------------------------------ MRD
// A node's state is a word: key << 16 | the batch its embedding was computed in.

// The key of every listed node at its batch: the batch of its next use if that is as an out-of-batch neighbour, else
// FAR.  (The reference sorts by the distance to it, or 1e8 + 1: the same order.)  One block, backwards: a batch waits for
// one trip to L2, what the next one needs is under way before.
__global__ void __launch_bounds__(T) next_use_lists_kernel(Lists l, int64_t nb, int32_t *next, int32_t *key) {
  const int tid = threadIdx.x;
  constexpr int AHEAD = 2;
  if (*l.failed) return;
  const auto load = [&](Span a, int i) { return i < a.n ? l.id[a.at + i] : 0; };
  Span a = l.span[nb - 1], a_next = nb > 1 ? l.span[nb - 2] : Span{0, 0};
  int32_t x[AHEAD], y[AHEAD];
#pragma unroll
  for (int u = 0; u < AHEAD; ++u) x[u] = load(a, tid + u * T);
  for (int64_t b = nb - 1; b >= 0; --b) {
    const auto node = [&](int i, int32_t e) {
      const int32_t v = e & ~TARGET;
      key[a.at + i] = __ldcg(&next[v]);
      next[v] = e < 0 ? (int32_t)FAR : (int32_t)b;     // (distinct nodes: nobody else reads or writes it in this batch)
    };
#pragma unroll
    for (int u = 0; u < AHEAD; ++u)
      if (tid + u * T < a.n) node(tid + u * T, x[u]);
    for (int i = tid + AHEAD * T; i < a.n; i += T) node(i, l.id[a.at + i]);
    const Span a_after = b > 1 ? l.span[b - 2] : Span{0, 0};
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) y[u] = load(a_next, tid + u * T);
    __syncthreads();
    a = a_next;
    a_next = a_after;
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) x[u] = y[u];
  }
}

__device__ __forceinline__ void bulk_s2g(void *dst, const void *src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
               "r"((uint32_t)__cvta_generic_to_shared(src)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

struct State {           // of a plan, between the launches for its chunks of batches
  int32_t n_cached, failed;
  int64_t used;
  unsigned long long reuse, recompute, dist, listed;
};
struct MrdArgs {
  Lists l;
  const int32_t *key;           // of the listed nodes
  int64_t b0, b1, nb;           // batches of this launch, of the plan
  int32_t budget, cap;
  State *st;
  int32_t *cached;              // [cap] cached ids, ascending (between launches)
  uint32_t *cached_state;       // [cap] their states (between launches)
  int32_t *place;               // [cap] of the listed nodes: cached ids before it
  int32_t *cand;                // [batches of a launch][2][cap] candidates, and their states
  int32_t *cand_n;              // [batches of a launch]
  int64_t plan_cap;
  int64_t *plan_off;
  int32_t *status;
};

// Forward sweep over batches b0 .. b1, one block.  Shared memory: cached ids and their states, later entries and lists of
// a selection; candidates and their states; four words each, then bitmaps.  What a batch costs is the walk over all of
// its candidates, twice (into the list and back into the cached ids), a warp for a word of the bitmaps at a time, and the
// selection.  (With the states in global memory the two walks took 17,000 of a batch's 34,000 cycles: an SM's own loads
// and stores get some 15 bytes a cycle out of L2.)  Candidates leave by bulk copies that nobody waits for.
__global__ void __launch_bounds__(T, 1) mrd_lists_kernel(const __grid_constant__ MrdArgs g) {
  extern __shared__ __align__(16) char raw[];
  __shared__ uint32_t s_tot[NW];
  __shared__ Line s_line;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, cap = g.cap, n_words = cap / 32;
  int32_t *s_cached = (int32_t *)raw;
  uint32_t *s_state = (uint32_t *)(s_cached + cap);
  int32_t *s_cand = (int32_t *)(s_state + cap);
  uint32_t *s_cand_state = (uint32_t *)(s_cand + cap);
  uint32_t *s_ent = (uint32_t *)s_cached;
  uint16_t *left = (uint16_t *)s_state, *right = left + cap;
  Word *s_list = (Word *)(s_cand_state + cap), *s_new = s_list + n_words, *s_kept = s_new + n_words;
  uint32_t *s_known = (uint32_t *)(s_kept + n_words);
  if (g.st->failed) return;
  int n_cached = g.st->n_cached;
  int64_t used = g.st->used;
  unsigned long long reuse = 0, recompute = 0, dist = 0;
  for (int i = tid; i < n_cached; i += T) s_cached[i] = g.cached[i], s_state[i] = g.cached_state[i];
  bool failed = false;
  // the first nodes of the next batch's list, loaded ahead
  constexpr int AHEAD = 2;
  int32_t x_next[AHEAD], mult_next[AHEAD];
  Span next = g.l.span[g.b0];
  const auto load_ahead = [&]() {
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      const int64_t i = tid + u * T;
      x_next[u] = i < next.n ? g.l.id[next.at + i] : 0;
      mult_next[u] = i < next.n ? g.l.mult[next.at + i] : 0;
    }
  };
  load_ahead();
  for (int64_t b = g.b0; b < g.b1; ++b) {
    const int64_t at = next.at;
    const int n_list = next.n;      // (no more than cap)
    int32_t *cand = g.cand + (b - g.b0) * 2 * cap;
    for (int i = tid; i < n_words; i += T) s_new[i].bits = s_known[i] = s_list[i].bits = 0;
    if (tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");      // (the candidates of the batch before)
    __syncthreads();         // (and the cached ids are there)
    // which of the batch's nodes are cached: a bit in s_list; statistics of the reuse
    const auto look_up = [&](int i, int32_t x, int m) {
      bool cached = false;
      if (i < n_list) {
        const int32_t v = x & ~TARGET;
        int lo = 0, hi = n_cached;
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (s_cached[mid] < v) lo = mid + 1;
          else hi = mid;
        }
        cached = lo < n_cached && s_cached[lo] == v;
        g.place[i] = lo;
        if (x >= 0) {
          if (cached) {
            reuse += m;
            dist += (unsigned long long)m * (unsigned long long)(b - (s_state[lo] & 0xffffu));
          } else {
            recompute += m;
          }
        }
      }
      const uint32_t w = __ballot_sync(0xffffffffu, cached);
      if (lane == 0) s_list[i >> 5].bits = w;
    };
#pragma unroll
    for (int u = 0; u < AHEAD; ++u)
      if (u * T + warp * 32 < n_list) look_up(tid + u * T, x_next[u], mult_next[u]);
    for (int i0 = AHEAD * T + warp * 32; i0 < n_list; i0 += T) {
      const int i = i0 + lane;
      look_up(i, i < n_list ? g.l.id[at + i] : 0, i < n_list ? g.l.mult[at + i] : 0);
    }
    __syncthreads();
    const int n = n_cached + n_list - count_words(s_list, n_words, (int32_t *)s_tot);
    if (n > cap) {
      failed = true;
      break;
    }
    // candidates in ascending order: first the batch's nodes, then the other cached ones around them
    const auto place = [&](int i, int32_t x) {
      if (i >= n_list) return;
      const uint32_t key = (uint32_t)g.key[at + i];
      const Word w = s_list[i >> 5];
      const int c = g.place[i], pos = c + i - bits_before(w, i);
      const bool cached = bit_of(w, i);
      s_cand[pos] = x & ~TARGET;
      s_cand_state[pos] = key << 16 | (x < 0 || !cached ? (uint32_t)b : s_state[c] & 0xffffu);
      atomicOr(cached ? &s_known[pos >> 5] : &s_new[pos >> 5].bits, 1u << (pos & 31));
    };
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) place(tid + u * T, x_next[u]);
    for (int i = tid + AHEAD * T; i < n_list; i += T) place(i, g.l.id[at + i]);
    if (b + 1 < g.b1) {
      next = g.l.span[b + 1];
      load_ahead();
    }
    __syncthreads();
    count_words(s_new, n_words, (int32_t *)s_tot);
#pragma unroll 4
    for (int w = warp; w < n_words; w += NW) {
      const Word add = s_new[w];
      const int pos = 32 * w + lane;
      if (pos < n && !(((add.bits | s_known[w]) >> lane) & 1u)) {
        const int c = pos - bits_before(add, lane);
        s_cand[pos] = s_cached[c];
        s_cand_state[pos] = s_state[c];
      }
      if (lane == 0) s_kept[w].bits = n >= 32 * w + 32 ? 0xffffffffu : n > 32 * w ? (1u << (n - 32 * w)) - 1u : 0u;
    }
    const int keep = min(n, g.budget);
    if (used + keep > g.plan_cap) {      // (uniform over the block)
      if (tid == 0) report(g.status, ORCA_E_CAPACITY, (int)b);
      failed = true;
      break;
    }
    fence_async();           // (what the bulk copies read)
    __syncthreads();
    if (tid == 0) {
      const uint32_t bytes = (uint32_t)(n + 3) / 4 * 16;
      bulk_s2g(cand, s_cand, bytes);
      bulk_s2g(cand + cap, s_cand_state, bytes);
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
    if (keep < n) {
      const auto drop = [&](int i) { atomicAnd(&s_kept[i >> 5].bits, ~(1u << (i & 31))); };
      if (!select_by_far_step([&](int i) { return s_cand_state[i] >> 16; }, n, keep, s_list, s_tot, drop)) {
        for (int i = tid; i < n; i += T) s_ent[i] = s_cand_state[i] >> 16 << IDX_BITS | (uint32_t)i;
        __syncthreads();
        select_by_order<false>(s_ent, n, keep, left, right, s_tot, &s_line, drop);
      }
    }
    __syncthreads();
    count_words(s_kept, n_words, (int32_t *)s_tot);
#pragma unroll 4
    for (int w = warp; w < n_words; w += NW) {
      const Word kept = s_kept[w];
      if (!bit_of(kept, lane)) continue;
      const int c = bits_before(kept, lane);
      s_cached[c] = s_cand[32 * w + lane];
      s_state[c] = s_cand_state[32 * w + lane];
    }
    if (tid == 0) {
      g.plan_off[b] = used;
      g.cand_n[b - g.b0] = n;
    }
    n_cached = keep;
    used += keep;
  }
  __syncthreads();
  for (int i = tid; i < n_cached && !failed; i += T) g.cached[i] = s_cached[i], g.cached_state[i] = s_state[i];
  if (tid == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");      // (shared memory is read until then)
  for (int o = 16; o > 0; o >>= 1) {
    reuse += __shfl_xor_sync(0xffffffffu, reuse, o);
    recompute += __shfl_xor_sync(0xffffffffu, recompute, o);
    dist += __shfl_xor_sync(0xffffffffu, dist, o);
  }
  if (lane == 0) {
    atomicAdd(&g.st->reuse, reuse);
    atomicAdd(&g.st->recompute, recompute);
    atomicAdd(&g.st->dist, dist);
  }
  if (tid == 0) {
    g.st->n_cached = n_cached;
    g.st->used = used;
    g.st->failed = failed;
    if (g.b1 == g.nb) g.plan_off[g.nb] = used;
  }
}

// The order of the plans of a launch's batches, a block each; the last one's totals.
__global__ void __launch_bounds__(T, 1) sort_plan_kernel(const __grid_constant__ MrdArgs g, int32_t *plan, int64_t *stats) {
  __shared__ uint32_t s_tot[NW];
  if (g.st->failed) return;
  if (g.b1 == g.nb && blockIdx.x == 0 && threadIdx.x == 0)
    stats[0] = g.st->reuse, stats[1] = g.st->recompute, stats[2] = g.st->dist;
  const tie::Shared w{g.cap};
  for (int64_t b = g.b0 + blockIdx.x; b < g.b1; b += gridDim.x) {
    const int n = g.cand_n[b - g.b0], keep = min(n, g.budget);
    const int32_t *cand = g.cand + (b - g.b0) * 2 * g.cap;
    int32_t *out = plan + g.plan_off[b];
    for (int i = threadIdx.x; i < n; i += T) {
      w.key(i) = (int32_t)((uint32_t)cand[g.cap + i] >> 16);
      w.idx(i) = (uint16_t)i;
    }
    tie::sort_first_shared(w, s_tot, n, keep, [&](int place, int i) { out[place] = cand[i]; });
  }
}

constexpr int64_t CHUNK = 512;      // batches of a launch: bounds the candidates that wait for their order (2 x 4 * CAP bytes each)

// Entries that the lists of a plan have room for: all that there can be, up to 16 M (12 bytes each; 400,000 edges with 20
// neighbours), and beyond that a third, which is what the tables of the kernels of planner_mrd.cu take, in whose workspace
// these lists lie.  (Lists of the largest graph's stream fill a thirtieth, those of streams with few repetitions a third.)
constexpr int64_t ROOM = 16 << 20;
static int64_t room_for(int64_t n_edges, int32_t bs, int32_t k, int64_t n_nodes) {
  const int64_t most = (n_edges + bs - 1) / bs * std::min<int64_t>(stride_of(bs, k, n_nodes), CAP);
  return std::min(most, std::max(ROOM, 2 * n_edges * (k + 1) / 3));
}

struct MrdLayout {
  int64_t state, id, mult, span, key, next, scratch, cached, cached_state, place, cand, cand_n, total;
  int64_t room;
  int32_t cap;
};
static MrdLayout mrd_layout(int64_t n_edges, int32_t bs, int32_t k, int64_t n_nodes, int32_t budget) {
  MrdLayout L;
  const int64_t nb = (n_edges + bs - 1) / bs, chunk = std::min(nb, CHUNK);
  L.room = room_for(n_edges, bs, k, n_nodes);
  L.cap = (int32_t)((std::min<int64_t>({(int64_t)budget + 2ll * bs * (k + 1), n_nodes, (int64_t)CAP}) + 31) & ~31ll);
  int64_t at = 0;
  auto take = [&](int64_t bytes) {
    const int64_t o = at;
    at += (bytes + 255) & ~255ll;
    return o;
  };
  L.state = take(sizeof(State));
  L.id = take(L.room * 4);
  L.mult = take(L.room * 4);
  L.span = take(nb * sizeof(Span));
  L.key = take(L.room * 4);
  L.next = take(n_nodes * 4);
  L.scratch = take(scratch_bytes(nb, n_nodes));
  L.cached = take(L.cap * 4);
  L.cached_state = take(L.cap * 4);
  L.place = take(L.cap * 4);
  L.cand = take(chunk * L.cap * 8);
  L.cand_n = take(chunk * 4);
  L.total = at;
  return L;
}

// (a key has to name every batch)
bool mrd_takes(int64_t n_edges, int32_t bs) { return (n_edges + bs - 1) / bs < (int64_t)FAR; }
bool mrd_always(int64_t n_edges, int32_t bs, int32_t k, int64_t n_nodes, int32_t budget) {
  const int64_t list = stride_of(bs, k, n_nodes);
  return std::min(budget + list, n_nodes) <= CAP && room_for(n_edges, bs, k, n_nodes) == (n_edges + bs - 1) / bs * list;
}
int64_t mrd_workspace_bytes(int64_t n_edges, int32_t bs, int32_t k, int64_t n_nodes, int32_t budget) {
  return mrd_layout(n_edges, bs, k, n_nodes, budget).total;
}

int launch_mrd(const int32_t *d_nodes, const int32_t *d_nbr, int64_t n_edges, int32_t bs, int32_t k, int64_t n_nodes,
               int32_t budget, int32_t *d_plan, int64_t plan_cap, int64_t *d_plan_off, int64_t *d_stats, int32_t *d_status,
               void *d_workspace, const int32_t **d_failed, cudaStream_t s) {
  const Ctx *c = cur();
  if (c == nullptr) return set_error(ORCA_E_CUDA, "orca_plan_mrd: no context for the current device");
  const MrdLayout L = mrd_layout(n_edges, bs, k, n_nodes, budget);
  char *base = (char *)d_workspace;
  MrdArgs g{};
  g.l.id = (int32_t *)(base + L.id), g.l.mult = (int32_t *)(base + L.mult), g.l.span = (Span *)(base + L.span);
  g.key = (int32_t *)(base + L.key);
  g.nb = (n_edges + bs - 1) / bs;
  g.budget = budget, g.cap = L.cap;
  g.st = (State *)(base + L.state);
  g.l.stride = 0, g.l.used = &g.st->listed, g.l.room = L.room, g.l.failed = &g.st->failed;
  g.cached = (int32_t *)(base + L.cached), g.cached_state = (uint32_t *)(base + L.cached_state);
  g.place = (int32_t *)(base + L.place);
  g.cand = (int32_t *)(base + L.cand);
  g.cand_n = (int32_t *)(base + L.cand_n);
  g.plan_cap = plan_cap, g.plan_off = d_plan_off, g.status = d_status;
  ORCA_CUDA(cudaMemsetAsync(g.st, 0, sizeof(State), s));
  int rc = launch_batch_lists(d_nodes, d_nbr, n_edges, bs, k, n_nodes, 0, g.nb, g.l, base + L.scratch,
                              (int32_t *)(base + L.next), (int32_t)FAR, s);
  if (rc != ORCA_OK) return rc;
  next_use_lists_kernel<<<1, T, 0, s>>>(g.l, g.nb, (int32_t *)(base + L.next), (int32_t *)(base + L.key));
  ORCA_COUNT_LAUNCH();
  ORCA_LAUNCH_CHECK();
  const int smem = 16 * L.cap + 7 * (L.cap / 32) * 4, smem_sort = tie::Shared::BYTES * L.cap;
  ORCA_CUDA(cudaFuncSetAttribute(mrd_lists_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  ORCA_CUDA(cudaFuncSetAttribute(sort_plan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_sort));
  for (g.b0 = 0; g.b0 < g.nb; g.b0 = g.b1) {
    g.b1 = std::min(g.nb, g.b0 + CHUNK);
    mrd_lists_kernel<<<1, T, smem, s>>>(g);
    ORCA_COUNT_LAUNCH();
    ORCA_LAUNCH_CHECK();
    sort_plan_kernel<<<(int)std::min<int64_t>(g.b1 - g.b0, c->sm_count), T, smem_sort, s>>>(g, d_plan, d_stats);
    ORCA_COUNT_LAUNCH();
    ORCA_LAUNCH_CHECK();
  }
  *d_failed = &g.st->failed;
  return ORCA_OK;
}

}  // namespace lists
}  // namespace orca

using namespace orca;

extern "C" int orca_plan_queries(const int64_t *h_src, const int64_t *h_dst, const double *h_ts, int64_t n_edges, int32_t bs,
                                 void *h_pinned, void *d_buffer, int32_t *d_nodes, double *d_ts, void *stream) {
  ORCA_CHECK_ARG(n_edges >= 0 && bs > 0);
  if (n_edges == 0) return ORCA_OK;
  ORCA_CHECK_ARG(h_src && h_dst && h_ts && h_pinned && d_buffer && d_nodes && d_ts && ((uintptr_t)d_buffer & 7) == 0);
  double *ts = (double *)h_pinned;
  int32_t *src = (int32_t *)(ts + n_edges), *dst = src + n_edges;
  // (a thread is worth starting for 50,000 edges: 400,000 take 0.9 ms on one, 0.2 on eight)
  const int threads = (int)std::max<int64_t>(1, std::min<int64_t>({8, n_edges / 50000, (int64_t)std::thread::hardware_concurrency()}));
  const int rc = on_threads(threads, [&](int t) {
    const int64_t lo = n_edges * t / threads, hi = n_edges * (t + 1) / threads;
    for (int64_t i = lo; i < hi; ++i) {
      ts[i] = h_ts[i];
      src[i] = (int32_t)h_src[i];
      dst[i] = (int32_t)h_dst[i];
    }
  }, "orca_plan_queries");
  if (rc != ORCA_OK) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  ORCA_CUDA(cudaMemcpyAsync(d_buffer, h_pinned, (size_t)n_edges * 16, cudaMemcpyHostToDevice, s));
  const double *dt = (const double *)d_buffer;
  const int32_t *ds = (const int32_t *)(dt + n_edges);
  lists::queries_kernel<<<(int)std::min<int64_t>((n_edges + 255) / 256, 1184), 256, 0, s>>>(dt, ds, ds + n_edges, n_edges, bs,
                                                                                             d_nodes, d_ts);
  ORCA_COUNT_LAUNCH();
  ORCA_LAUNCH_CHECK();
  return ORCA_OK;
}
