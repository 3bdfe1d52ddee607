// Scores a group of consecutive batches of a stream as one unit of work.
//
// Batch by batch, a batch is a chain of small dependent launches that leaves most of the chip idle (0.12 to 0.17 ms
// for 200 to 2000 edges).  But little of that chain is real: batch n + 1 depends on batch n only through the memory
// rows that n rewrites and through the historical embeddings that n's layer 1 pushes, and where either row comes
// from is known from the ids alone.  So a group keeps the rewritten memory rows of all its batches in a log and the
// layer-1 output of all its batches in one array, and the index kernels turn every neighbour id into the row that
// holds its value at that point of the stream: (memory table | log) for layer 1, (history table | layer-1 output)
// for layer 2.  What stays serial is the memory update, batch after batch (raw messages, GRU); everything else is
// one launch over the rows of all batches.  Every row is computed from the same operands in the same order as batch
// by batch, so results are the same bits.
//
//   index stream   neighbour tables of all batch rows; bit sets per node (cached / in batch / positive / recomputed,
//                  one bit per batch) and a (node, batch) hash table; recomputed rows; resolution of the ids; the
//                  cache flags of the group's last plan
//   chain stream   raw messages and GRU of batch 0, 1, ... into the log, of large groups only those that a later batch
//                  reads; the others behind it, at once.  Runs a group ahead of the main stream: rows of the group
//                  before are read from that group's log
//   main stream    layer 1, layer 2, scores of all batches; then the last version of every rewritten row goes to
//                  the memory and history tables
// Buffers of the index and chain streams exist twice (group parity).
#include <algorithm>
#include <climits>

#include "attn_out.cuh"
#include "chain.cuh"
#include "common.cuh"
#include "context.cuh"
#include "group.cuh"
#include "gru_rows.cuh"
#include "index_ops.cuh"
#include "sampling.cuh"
#include "tc_gemm.cuh"

namespace orca {
namespace grp {

// ------------------------------------------------------------------------------------------------ index kernels
__device__ __forceinline__ void set_bit(uint32_t *word, uint32_t bit) {
  if ((__ldcg(word) & bit) == 0) atomicOr(word, bit);    // (hub nodes: the bit is set nearly always)
}

__device__ __forceinline__ KnownIds known_ids(const Args &a) {
  return {(uint32_t)(a.n_nodes - 1), (uint32_t)a.n_edge_rows - 1};
}

// neighbour tables of the batch rows; membership bits; last positions; cache bits of the plans inside the group
template <int G>
__global__ void __launch_bounds__(256) head_kernel(const __grid_constant__ Args a) {
  dep_trigger();
  dep_wait();
  const int n_rows = 3 * a.edges();
  const int lane = threadIdx.x % G;
  const int gshift = (threadIdx.x % 32) / G * G;
  const unsigned gmask = (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << gshift);
  const int per = blockDim.x / G;
  for (int q = blockIdx.x * per + threadIdx.x / G; q < n_rows; q += gridDim.x * per) {
    const int n = q / (3 * a.bs), r = q - n * 3 * a.bs, b = a.b_of(n);
    const int node = a.img[a.off[n] + r];
    const double t = a.ts[n * a.bs + r % b];
    sample_query<G>(a.indptr, a.adj_nbr, a.adj_eid, a.adj_ts, a.n_nodes, known_ids(a), node, t, q, a.k, lane, gmask, gshift,
                    a.nbr1, a.eid1, nullptr, a.dt1, a.status, nullptr, nullptr, nullptr, nullptr);
  }
  // Membership, a thread per row.  A batch holds its hub nodes hundreds of times over: rows of one node that meet in a
  // warp make one entry (the last of them), else every one of them queues at the same words.
  const int step = gridDim.x * blockDim.x;
  for (int q0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31); q0 < n_rows; q0 += step) {
    const int q = q0 + (threadIdx.x & 31);
    int n = 0, r = 0, b = 1, node = -1;
    if (q < n_rows) {
      n = q / (3 * a.bs), r = q - n * 3 * a.bs, b = a.b_of(n);
      node = a.img[a.off[n] + r];
      if (node >= a.n_nodes || (r >= 2 * b && !a.keeps_history())) node = -1;
    }
    const unsigned long long key = node >= 0 ? key_of(node, n) : 0;
    const unsigned group = __match_any_sync(0xffffffffu, key);
    const unsigned positive = group & __ballot_sync(0xffffffffu, r < 2 * b);
    const int from = positive ? 31 - __clz(positive) : 0;
    const int r_pos = __shfl_sync(0xffffffffu, r, from), last_pos = positive ? r_pos : -1;
    if (node < 0 || (group >> (threadIdx.x & 31)) != 1u) continue;     // the highest lane speaks for the group
    const uint32_t bit = 1u << n;
    set_bit(&a.bits[node].in_rows, bit);
    if (last_pos >= 0) set_bit(&a.bits[node].positive, bit);
    uint32_t h = hash_of(key) & a.table_mask;
    for (;;) {    // (at most half of the table is ever used)
      Entry *e = a.table + h;
      unsigned long long k = __ldcg(&e->key);
      if (k == 0) k = atomicCAS(&e->key, 0ull, key);
      if (k == 0 || k == key) {
        if (__ldcg(&e->row) < r + 1) atomicMax(&e->row, r + 1);
        if (last_pos >= 0 && __ldcg(&e->pos) < last_pos + 1) atomicMax(&e->pos, last_pos + 1);
        break;
      }
      h = (h + 1) & a.table_mask;
    }
  }
  if (a.budget())
    for (int n = 0; n + 1 < a.nb; ++n) {
      const int32_t *plan = a.img + a.off[n] + 4 * a.b_of(n);
      for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n_plan[n]; i += step) {
        const int v = plan[i];
        if (v >= 0 && v < a.n_nodes) atomicOr(&a.bits[v].cached, 1u << (n + 1));
      }
    }
}

// next place in batch n's list: one atomic for the lanes of a warp that ask for the same batch
__device__ __forceinline__ int place(int32_t *counter, int n) {
  const unsigned group = __match_any_sync(__activemask(), n), lane = threadIdx.x & 31;
  const int leader = __ffs(group) - 1;
  int at = 0;
  if (lane == leader) at = atomicAdd(counter, __popc(group));
  return __shfl_sync(group, at, leader) + __popc(group & ((1u << lane) - 1u));
}

// candidates of the recomputed set, and the memory updates: the last position of every node among [src | dst]
__global__ void __launch_bounds__(256) mark_kernel(const __grid_constant__ Args a) {
  dep_trigger();
  dep_wait();
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  if (a.budget()) {
    // Node 0 pads the tables: it is in thousands of slots and a candidate of nearly every batch.  One thread a block
    // and batch asks for it (all of them queued at its word: 62 us for eight batches of 2000 edges, 11 so).
    __shared__ uint32_t padded;
    if (threadIdx.x == 0) padded = 0;
    __syncthreads();
    const int n_slots = 3 * a.edges() * a.k, per = 3 * a.bs * a.k;
    for (int i = tid; i < n_slots; i += step) {
      const int n = i / per, v = a.nbr1[i];
      const uint32_t bit = 1u << n;
      if (v == 0 && ((*(volatile uint32_t *)&padded & bit) || (atomicOr(&padded, bit) & bit))) continue;
      // (through L1: hub nodes are sampled thousands of times, and a stale word only costs the atomic below)
      const uint4 b = *reinterpret_cast<const uint4 *>(&a.bits[v]);
      if ((b.y & bit) || (b.w & bit) || (n > 0 ? (b.x & bit) != 0 : a.cache_flag[v] != 0)) continue;
      if (__ldcg(&a.bits[v].fetched) & bit) continue;
      if (atomicOr(&a.bits[v].fetched, bit) & bit) continue;
      const int p = place(&a.cnt->n_cand[n], n);
      if (p < a.u_cap1) a.cand[(size_t)n * a.u_cap1 + p] = v;
      atomicMax(&a.cnt->low_cand[n], INT_MAX - v);
    }
  }
  // (a warp stays together here, for one atomic a warp and batch)
  const int n_pos = 2 * a.edges(), per = 2 * a.bs;
  for (int i0 = tid & ~31; i0 < n_pos; i0 += step) {
    const int i = i0 + (threadIdx.x & 31), n = min(i, n_pos - 1) / per, r = i - n * per, b = a.b_of(n);
    const int32_t *batch = a.img + a.off[n];
    const int v = i < n_pos ? batch[r] : -1;
    // (node ids outside the table are reported by the sampling and are no updates; edge ids here)
    const int eid = i < n_pos ? batch[3 * b + r % b] : 0;
    const bool known = eid >= 0 && eid < a.n_edge_rows;
    if (!known) report(a.status, ORCA_E_BOUNDS, eid);
    Entry *e = nullptr;
    if (v >= 0 && v < a.n_nodes) {
      e = a.table + find_entry(a.table, a.table_mask, v, n);
      if (e->pos != r + 1) e = nullptr;
    }
    const bool back = e != nullptr && a.split && !a.again(v, n);
    __syncwarp();
    const unsigned group = __match_any_sync(0xffffffffu, e != nullptr ? 2 * n + (back ? 1 : 0) : -1);
    const int leader = __ffs(group) - 1, lane = threadIdx.x & 31;
    int w = 0;
    if (e != nullptr && lane == leader) w = atomicAdd(back ? &a.cnt->n_back[n] : &a.cnt->n_win[n], __popc(group));
    w = __shfl_sync(0xffffffffu, w, leader) + __popc(group & ((1u << lane) - 1u));
    if (e == nullptr) continue;
    if (back) w = per - 1 - w;
    e->pos = IN_LOG | w;     // (no other position of the node equals it)
    const int at = n * per + w, other = r < b ? batch[b + r] : batch[r - b];
    a.win_node[at] = v;
    a.win_other[at] = other >= 0 && other < a.n_nodes ? other : 0;
    a.win_eid[at] = known ? eid : 0;
    a.win_t[at] = (float)a.ts[n * a.bs + r % b];
  }
}

// one block: query times of the recomputed rows, the candidate that every batch drops (the smallest id,
// modules/embedding_module.py:212), places of the recomputed rows, row counts
__global__ void __launch_bounds__(1024) count_kernel(const __grid_constant__ Args a) {
  __shared__ int s_cand[MAX_BATCHES];
  const int n = threadIdx.x >> 5, lane = threadIdx.x & 31;
  dep_trigger();
  dep_wait();
  if (n < a.nb) {
    const int b = a.b_of(n);
    double t = -1.0e300;
    for (int i0 = lane; i0 < b; i0 += 32 * 8) {
      double x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = i0 + 32 * u < b ? a.ts[n * a.bs + i0 + 32 * u] : -1.0e300;
#pragma unroll
      for (int u = 0; u < 8; ++u) t = fmax(t, x[u]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t = fmax(t, __shfl_xor_sync(0xffffffffu, t, o));
    if (lane == 0) {
      const int c = min(a.cnt->n_cand[n], a.u_cap1);
      const int low = c > 0 ? INT_MAX - a.cnt->low_cand[n] : -1;
      s_cand[n] = c;
      a.cnt->dropped[n] = low;
      a.cnt->t_max[n] = t;
      if (low >= 0) atomicAnd(&a.bits[low].fetched, ~(1u << n));
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int sum = 0;
    for (int i = 0; i < a.nb; ++i) {
      a.cnt->app_off[i] = sum;
      sum += s_cand[i];
    }
    a.cnt->app_off[a.nb] = sum;
    const int batch_rows = 3 * a.edges();
    if (a.layers == 2 && a.mode == ORCA_MODE_NO_REUSE) sum = batch_rows * a.k;
    const int rows = batch_rows + sum;
    a.cnt->n_rows = rows;
    if (a.status != nullptr) {     // counts of the last batch (status word layout, common.cuh)
      const int rows_last = 3 * a.b_last;
      a.status[1] = a.budget() ? rows_last + max(0, s_cand[a.nb - 1] - 1)
                    : a.layers == 2 && a.mode == ORCA_MODE_NO_REUSE ? rows_last * (1 + a.k) : rows_last;
      a.status[2] = a.cnt->n_win[a.nb - 1] + a.cnt->n_back[a.nb - 1];
    }
  }
}

__device__ __forceinline__ int batch_of_app(const Args &a, int p) {
  int n = 0;
  while (n + 1 < a.nb && p >= a.cnt->app_off[n + 1]) ++n;
  return n;
}

// neighbour tables of the rows behind the batch rows: the recomputed nodes at their batch's latest time or, without
// reuse, every sampled neighbour at the time of the row that sampled it
template <int G>
__global__ void __launch_bounds__(256) append_kernel(const __grid_constant__ Args a) {
  dep_trigger();
  dep_wait();
  const int batch_rows = 3 * a.edges(), n_app = a.cnt->n_rows - batch_rows;
  const int lane = threadIdx.x % G;
  const int gshift = (threadIdx.x % 32) / G * G;
  const unsigned gmask = (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << gshift);
  const int per = blockDim.x / G;
  for (int p = blockIdx.x * per + threadIdx.x / G; p < n_app; p += gridDim.x * per) {
    int v;
    double t;
    if (a.mode == ORCA_MODE_NO_REUSE) {
      const int q = p / a.k, n = q / (3 * a.bs);
      v = a.nbr1[p];
      t = a.ts[n * a.bs + (q - n * 3 * a.bs) % a.b_of(n)];
    } else {
      const int n = batch_of_app(a, p);
      v = a.cand[(size_t)n * a.u_cap1 + (p - a.cnt->app_off[n])];
      t = a.cnt->t_max[n];
      if (lane == 0 && v != a.cnt->dropped[n]) {
        const unsigned long long key = key_of(v, n), word = key << APP_ROW_BITS | (unsigned long long)(p + 1);
        uint32_t h = hash_of(key) & a.app_mask;
        while (atomicCAS(&a.app_table[h], 0ull, word) != 0ull) h = (h + 1) & a.app_mask;   // (keys are distinct)
      }
    }
    if (lane == 0) a.app_node[p] = v;
    sample_query<G>(a.indptr, a.adj_nbr, a.adj_eid, a.adj_ts, a.n_nodes, known_ids(a), v, t, batch_rows + p, a.k, lane, gmask,
                    gshift, a.nbr1, a.eid1, nullptr, a.dt1, a.status, nullptr, nullptr, nullptr, nullptr);
  }
}

// ids -> rows of the two-part tables
__global__ void __launch_bounds__(256) resolve_kernel(const __grid_constant__ Args a, const float *last_update) {
  dep_trigger();
  dep_wait();
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  const int batch_rows = 3 * a.edges(), n_slots = a.cnt->n_rows * a.k;
  for (int i = tid; i < n_slots; i += step) {
    const int row = i / a.k;
    int n;
    if (row < batch_rows) {
      n = row / (3 * a.bs);
    } else {
      const int p = row - batch_rows;
      n = a.mode == ORCA_MODE_NO_REUSE ? p / a.k / (3 * a.bs) : batch_of_app(a, p);
    }
    const int v = a.nbr1[i];
    if (row < batch_rows && a.layers == 2)
      a.nbr2[i] = v == 0 ? 0 : a.mode == ORCA_MODE_NO_REUSE ? (int)a.n_nodes + batch_rows + i : history_row(a, v, n);
    if (v != 0) a.nbr1[i] = memory_row(a, v, n);
  }
  // The rows' own nodes.  Rows that share their own features share what layer 1 makes of them (the query, the merger's
  // part): 0.18 to 0.48 of a group's rows are distinct (hub nodes fill a batch, and most nodes have not changed since the
  // batch before).  A thread a row: one atomic a warp on the list's counter.
  for (int row = tid; row < a.cnt->n_rows; row += step) {
    int n, node;
    if (row < batch_rows) {
      n = row / (3 * a.bs);
      node = a.img[a.off[n] + row - n * 3 * a.bs];
    } else {
      const int p = row - batch_rows;
      n = a.mode == ORCA_MODE_NO_REUSE ? p / a.k / (3 * a.bs) : batch_of_app(a, p);
      node = a.app_node[p];
    }
    const int own = node > 0 && node < a.n_nodes ? memory_row(a, node, n) : 0;
    a.own1[row] = own;
    if (__ldcg(&a.own_seen[own]) == 0 && atomicCAS(&a.own_seen[own], 0, -1) == 0) {
      const int l = place(&a.cnt->n_own, 0);
      a.own_list[l] = own;
      a.own_seen[own] = l + 1;
    }
  }
  const int per = 2 * a.bs;
  for (int i = tid; i < a.nb * per; i += step) {
    const int n = i / per;
    if (!a.is_update(n, i - n * per)) continue;
    const int v = a.win_node[i], row = memory_row_early(a, v, n);
    if (!a.again(v, n)) {
      const int l = place(&a.cnt->n_last, 0);
      a.last_at[l] = i;
      a.last_node[l] = v;
    }
    a.win_mem[i] = row;
    a.win_gap[i] = a.win_t[i] - last_update_of(a, last_update, v, row);
    a.win_other[i] = memory_row_early(a, a.win_other[i], n);
  }
}

// the layer-1 rows' places in own_list
__global__ void __launch_bounds__(256) own_kernel(const __grid_constant__ Args a) {
  dep_trigger();
  dep_wait();
  const int n = a.cnt->n_rows;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) a.own_at[i] = a.own_seen[a.own1[i]] - 1;
}

// ------------------------------------------------------------------------------------------------ last versions
// A warp takes up to eight items, memory rows first and then layer-1 rows: its lanes look them up side by side, and what is
// to be copied goes four rows at a time.  (64 threads an item, one chain of lookups after the other: 20 us for 50 k rows,
// 10 so.)  Where there are fewer items than eight a warp, they are spread over all warps.
__global__ void __launch_bounds__(256)
write_back_kernel(const __grid_constant__ Args a, const float *log, const float *emb1, float *memory, float *history,
                  int32_t *h_status) {
  dep_trigger();
  dep_wait();
  // the last kernel of the group: what the others have reported goes straight to the host
  if (h_status != nullptr && blockIdx.x == 0 && threadIdx.x < 4) h_status[threadIdx.x] = __ldcg(a.status + threadIdx.x);
  constexpr int MOST = 8, ROWS = 4, PIECES = D / 4;
  const int lane = threadIdx.x & 31, warps = gridDim.x * (blockDim.x >> 5);
  const int n_upd = a.cnt->n_last, batch_rows = 3 * a.edges();
  const int n_items = n_upd + (a.keeps_history() ? a.cnt->n_rows : 0);
  const int items = min(MOST, (n_items + warps - 1) / warps);
  for (int i0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * items; i0 < n_items; i0 += warps * items) {
    const int i = i0 + lane;
    int to = -1, from = 0;      // this lane's row: where it goes (history: behind the memory rows), where it lies
    if (lane < items && i < n_items) {
      if (i < n_upd) {
        to = a.last_node[i];
        from = a.log_base + a.last_at[i];
      } else {
        const int row = i - n_upd;
        int n, v;
        bool wins;
        if (row < batch_rows) {
          n = row / (3 * a.bs);
          const int r = row - n * 3 * a.bs;
          v = a.img[a.off[n] + r];
          wins = v >= 0 && v < a.n_nodes && a.table[find_entry(a.table, a.table_mask, v, n)].row == r + 1;
        } else {
          n = batch_of_app(a, row - batch_rows);
          v = a.app_node[row - batch_rows];
          wins = v != a.cnt->dropped[n];
        }
        // (unless a later batch pushes the node's)
        if (wins && !((unsigned long long)(a.bits[v].in_rows | a.bits[v].fetched) >> (n + 1))) to = v, from = row;
      }
    }
    for (uint32_t todo = __ballot_sync(0xffffffffu, to >= 0); todo != 0;) {
      float4 x[ROWS][2];
      float4 *dst[ROWS];
      int n = 0;
#pragma unroll
      for (int k = 0; k < ROWS; ++k) {
        const int l = todo != 0 ? __ffs(todo) - 1 : 0;
        const int v = __shfl_sync(0xffffffffu, to, l), f = __shfl_sync(0xffffffffu, from, l);
        dst[k] = nullptr;
        if (todo == 0) continue;
        todo &= todo - 1;
        const bool mem = i0 + l < n_upd;
        const float4 *src = reinterpret_cast<const float4 *>((mem ? log : emb1) + (size_t)f * D);
        dst[k] = reinterpret_cast<float4 *>((mem ? memory : history) + (size_t)v * D);
        x[k][0] = src[lane];
        if (lane + 32 < PIECES) x[k][1] = src[lane + 32];
        ++n;
      }
#pragma unroll
      for (int k = 0; k < ROWS; ++k)
        if (k < n) {
          dst[k][lane] = x[k][0];
          if (lane + 32 < PIECES) dst[k][lane + 32] = x[k][1];
        }
    }
  }
}

// ------------------------------------------------------------------------------------------------ host side
static inline size_t align_up(size_t x) { return (x + 255) & ~(size_t)255; }
static inline uint32_t pow2_at_least(uint64_t x) {
  uint32_t p = 64;
  while (p < x) p <<= 1;
  return p;
}

// Batches per group: at most four row blocks of 128 per SM, at most a bit each.  A larger group has fewer partly empty last
// rounds of row blocks.  What the first group costs before its layers start, index kernels and the memory chain (8 us a
// batch), is not hidden by anything, so that group is half as large (two blocks per SM; where the chain matters, that is not
// without reuse), and the rest is dealt out evenly.  us for a stream of 600 x K 20 / 1000 / 2000 edges a batch / without
// reuse / 40 x 200, by rows of a group and of the first, 148 SMs:
//   57 k, one after the other  2280 / 2403 / 4587 / 1634 / 1566      76 k so           2274 / 2295 / 4538 / 1584 / 1552
//   57 k and 38 k              2260 / 2341 / 4491 / 1634 / 1560      76 k and 19 k     2255 / 2368 / 4522 / 1589 / 1550
//   76 k and 38 k              2260 / 2338 / 4517 / 1591 / 1547      76 k and 57 k     2277 / 2417 / 4540 / 1595 / 1553
//   95 k and 38 k              2267 / 2347 / 4472 / 1594 / 1554
// (the forms lie within 3 % of one another; before the layers' kernels were faster the first row was 6 to 14 % slower than the third)
// (Device memory of a group's buffers at 2000 edges a batch, K 10: 2.5 GB, half of it queries and attention sums.)
static int group_rows() {
  int device = 0, sms = 0;      // (asked of the device itself: no context is made for it)
  if (cudaGetDevice(&device) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
    (void)cudaGetLastError();
    sms = 148;
  }
  return 4 * 128 * sms;
}
static int64_t batch_rows(int bs, int k, int layers, int mode) {
  return 3ll * bs * (layers == 2 && mode == ORCA_MODE_NO_REUSE ? 1 + k : 1);
}
static int group_size(int bs, int k, int layers, int mode) {
  return (int)std::max<int64_t>(1, std::min<int64_t>(MAX_BATCHES, group_rows() / batch_rows(bs, k, layers, mode)));
}
// sizes of the groups of a stream of n batches -> sizes (n entries); their number
static int group_sizes(int n, int bs, int k, int layers, int mode, int32_t *sizes) {
  const int most = group_size(bs, k, layers, mode), first_rows = group_rows() / 2;
  const int64_t rows = batch_rows(bs, k, layers, mode);
  int groups = 0, left = n;
  if (!(layers == 2 && mode == ORCA_MODE_NO_REUSE) && n * rows > 2ll * first_rows) {
    sizes[groups++] = (int)std::max<int64_t>(1, std::min<int64_t>(most, first_rows / rows));
    left -= sizes[0];
  }
  for (int rest = ceil_div(left, most); rest > 0; --rest) {
    sizes[groups] = left / rest;
    left -= sizes[groups++];
  }
  return groups;
}

// The memory chain is serial, so only what a later batch of the group reads belongs there: in a group of 2000-edge
// batches on the largest graph 125 of a batch's 890 updates.  The others, every node's last update in the group, wait for
// nobody, and one launch (gru_rows.cu) does them behind the chain (chain 208 -> 74 us a group on half of the
// SMs).  That launch and the message rows it reads are some 20 us of latency, of which a group with few updates wins back
// nothing, while the largest graph's wins at every size.  us for a stream of one group, without / with, by its positions:
//            8 k      12 k     16 k     20 k     24 k     32 k        40 k
//   2000     441/414  539/491  700/632  806/716  883/775  1124/985    1352/1183      edges a batch, largest graph
//   1000     448/450  508/507  631/629  719/721  828/815  1027/1028   1279/1265
//   600      528/537  693/696  838/837  975/967  1102/1101  1419/1412                 (K 20)
//   200      607/606  779/798
constexpr int SPLIT_FROM = 16384;      // positions [src | dst] of a group

// Index buffers (two of each) and main-stream buffers.  The layer-1 rows that exist at all are few more than the
// batches' own, but a batch with a cold cache can recompute every sampled neighbour: the projected queries and
// attention sums (9 KB a row) are sized for `chunk` rows, and layer 1 runs over as many chunks as there are: the
// index kernels' row count comes back to the host while the group before is still being worked on.
struct Parity {
  NodeBits *bits;
  Entry *table;
  unsigned long long *app_table;
  Counters *cnt;
  size_t zero_bytes;       // bits, tables and counters are zeroed together, from `bits`
  int32_t *cand, *app_node, *nbr1, *eid1, *nbr2, *own1, *own_seen, *own_list, *own_at;
  float *dt1;
  int32_t *win_node, *win_eid, *win_mem, *win_other;
  float *win_t, *win_gap;
  int32_t *last_at, *last_node;
  char *stage;
  void *upd_image;         // split inputs of the memory updates (chain.cu)
};
struct Buffers {
  Parity par[2];
  float *log;              // two parities, one after the other
  char *msg_image;         // of the messages of every node's last update (groups whose last updates leave the chain)
  float *qt, *own, *emb1;
  // operand images (attn_out.cuh): attention sums, own features, layer 2's own features, pairs that are scored
  char *ctx, *feat, *feat2, *pairs;
  uint8_t *valid;
  uint32_t table_size, app_size;
  int64_t rows_max;        // layer-1 rows a group can have
  int chunk;
  size_t stage_bytes, total;
};

static Buffers carve(void *base, int bs, int nb, int k, int u_cap, int plan_cap, int64_t n_nodes, int layers, int mode) {
  Buffers w{};
  size_t off = 0;
  char *p = (char *)base;
  auto take = [&](size_t bytes) { void *r = p ? p + off : nullptr; off += align_up(bytes); return r; };
  const int64_t E = (int64_t)nb * bs, batch_rows = 3 * E;
  const bool budget = layers == 2 && mode == ORCA_MODE_BUDGET, no_reuse = layers == 2 && mode == ORCA_MODE_NO_REUSE;
  const int64_t apps = budget ? (int64_t)nb * (u_cap + 1) : no_reuse ? batch_rows * k : 0;
  w.rows_max = batch_rows + apps;
  w.chunk = (int)(no_reuse ? w.rows_max : std::min<int64_t>(w.rows_max, batch_rows + std::max<int64_t>(u_cap + 1, batch_rows / 4)));
  w.table_size = pow2_at_least(2 * batch_rows);
  w.app_size = pow2_at_least(budget ? 2 * apps : 1);
  w.stage_bytes = align_up((size_t)(4 * E + (int64_t)nb * plan_cap) * 4) + align_up((size_t)E * 8);
  for (Parity &x : w.par) {
    const size_t first = off;
    x.bits = (NodeBits *)take((size_t)n_nodes * sizeof(NodeBits));
    x.table = (Entry *)take((size_t)w.table_size * sizeof(Entry));
    x.app_table = (unsigned long long *)take((size_t)w.app_size * 8);
    x.own_seen = (int32_t *)take((size_t)(n_nodes + 4 * E) * 4);
    x.cnt = (Counters *)take(sizeof(Counters));
    x.zero_bytes = off - first;
    x.cand = (int32_t *)take(budget ? (size_t)apps * 4 : 4);
    x.app_node = (int32_t *)take((size_t)std::max<int64_t>(apps, 1) * 4);
    x.nbr1 = (int32_t *)take((size_t)w.rows_max * k * 4);
    x.eid1 = (int32_t *)take((size_t)w.rows_max * k * 4);
    x.dt1 = (float *)take((size_t)w.rows_max * k * 4);
    x.nbr2 = (int32_t *)take((size_t)batch_rows * k * 4);
    x.own1 = (int32_t *)take((size_t)w.rows_max * 4);
    x.own_list = (int32_t *)take((size_t)w.rows_max * 4);
    x.own_at = (int32_t *)take((size_t)w.rows_max * 4);
    x.win_node = (int32_t *)take((size_t)2 * E * 4);
    x.win_eid = (int32_t *)take((size_t)2 * E * 4);
    x.win_mem = (int32_t *)take((size_t)2 * E * 4);
    x.win_other = (int32_t *)take((size_t)2 * E * 4);
    x.win_t = (float *)take((size_t)2 * E * 4);
    x.win_gap = (float *)take((size_t)2 * E * 4);
    x.last_at = (int32_t *)take((size_t)2 * E * 4);
    x.last_node = (int32_t *)take((size_t)2 * E * 4);
    x.stage = (char *)take(w.stage_bytes);
    x.upd_image = take(update_image_bytes(2 * E));
  }
  w.log = (float *)take((size_t)2 * 2 * E * D * 4);
  w.msg_image = (char *)take(2 * E > SPLIT_FROM ? gru_image_bytes(std::min(2 * E, n_nodes)) : 4);
  w.qt = (float *)take((size_t)w.chunk * QT_LD * 4);
  w.own = (float *)take((size_t)w.chunk * OWN_LD * 4);
  w.ctx = (char *)take(img::bytes(w.chunk, img::CTX_STAGES));
  w.feat = (char *)take(img::bytes(w.chunk, img::FEAT_STAGES));
  w.feat2 = (char *)take(layers == 2 ? img::bytes(batch_rows, img::FEAT_STAGES) : 4);
  w.valid = (uint8_t *)take((size_t)w.chunk);
  w.emb1 = (float *)take(layers == 2 ? (size_t)w.rows_max * D * 4 : 4);     // (one layer leaves pairs)
  w.pairs = (char *)take(img::bytes(2 * E, img::PAIR_STAGES));
  w.total = off;
  return w;
}

static int launch_index(const Args &a, const float *last_update, size_t zero_bytes, int32_t *h_rows, cudaEvent_t counted,
                        cudaStream_t s, int sms) {
  ORCA_CUDA(cudaMemsetAsync(a.bits, 0, zero_bytes, s));
  const int E = a.edges(), rows = 3 * E;
  const bool wide = a.k > 16;
  const int grid_rows = std::min(ceil_div(rows, wide ? 8 : 16), sms * 16);
  const int grid_slots = std::min(ceil_div(rows * a.k, 256), sms * 8);
  if (wide) ORCA_CUDA(launch_dep(head_kernel<32>, grid_rows, 256, 0, s, a));
  else ORCA_CUDA(launch_dep(head_kernel<16>, grid_rows, 256, 0, s, a));
  ORCA_CUDA(launch_dep(mark_kernel, grid_slots, 256, 0, s, a));
  ORCA_CUDA(launch_dep(count_kernel, 1, 1024, 0, s, a));
  ORCA_CUDA(cudaMemcpyAsync(h_rows, &a.cnt->n_rows, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
  ORCA_CUDA(cudaEventRecord(counted, s));
  if (a.layers == 2 && a.mode != ORCA_MODE_REUSE_ALL) {
    const int grid = a.mode == ORCA_MODE_NO_REUSE ? sms * 16 : sms * 2;
    if (wide) ORCA_CUDA(launch_dep(append_kernel<32>, grid, 256, 0, s, a));
    else ORCA_CUDA(launch_dep(append_kernel<16>, grid, 256, 0, s, a));
    ORCA_COUNT_LAUNCH();
  }
  ORCA_CUDA(launch_dep(resolve_kernel, grid_slots, 256, 0, s, a, last_update));
  ORCA_CUDA(launch_dep(own_kernel, std::min(ceil_div(rows, 256), sms * 8), 256, 0, s, a));
  for (int i = 0; i < 5; ++i) ORCA_COUNT_LAUNCH();
  return ORCA_OK;
}

}  // namespace grp
}  // namespace orca

using namespace orca;

#define ORCA_TRY(call)        \
  do {                        \
    int rc_ = (call);         \
    if (rc_ != ORCA_OK) return rc_; \
  } while (0)

extern "C" {

int32_t orca_group_size(int32_t bs, int32_t k, int32_t n_layers, int32_t mode) {
  if (bs <= 0 || k < 1 || k > ORCA_MAX_K) return -1;
  return grp::group_size(bs, k, n_layers, mode);
}

int32_t orca_group_sizes(int32_t n_batches, int32_t bs, int32_t k, int32_t n_layers, int32_t mode, int32_t *h_sizes) {
  if (n_batches <= 0 || bs <= 0 || k < 1 || k > ORCA_MAX_K || h_sizes == nullptr) return -1;
  return grp::group_sizes(n_batches, bs, k, n_layers, mode, h_sizes);
}

int64_t orca_group_workspace_bytes(int32_t bs, int32_t nb, int32_t k, int32_t u_cap, int32_t plan_cap, int64_t n_nodes,
                                   int32_t n_layers, int32_t mode) {
  if (bs <= 0 || nb <= 0 || nb > grp::MAX_BATCHES || k < 1 || k > ORCA_MAX_K || u_cap < 0 || plan_cap < 0 || n_nodes <= 0)
    return -1;
  return (int64_t)grp::carve(nullptr, bs, nb, k, u_cap, plan_cap, n_nodes, n_layers, mode).total;
}

int orca_tgn_eval_group(const orca_tgn_t *m, const orca_group_t *g, void *d_workspace, int64_t workspace_bytes,
                        float *d_prob, float *h_prob, int32_t *d_status, void *stream) {
  ORCA_CHECK_ARG(m && g && d_workspace && d_prob && d_status && g->h_i32 && g->h_ts && g->off_i32 && g->n_plan);
  ORCA_CHECK_ARG(g->nb > 0 && g->nb <= g->nb_max && g->nb_max <= grp::MAX_BATCHES && g->bs > 0 && g->b_last > 0 &&
                 g->b_last <= g->bs && g->u_cap >= 0 && g->h_rows && g->seq >= 0);
  ORCA_CHECK_ARG(g->d_metrics == nullptr || (g->h_metrics && orca_link_metric_parts(g->bs) > 0));
  ORCA_CHECK_ARG((m->n_layers == 1 || m->n_layers == 2) && m->k >= 1 && m->k <= ORCA_MAX_K && m->world <= 1);
  const int layers = m->n_layers, k = m->k, mode = layers == 2 ? m->mode : ORCA_MODE_BUDGET;
  ORCA_CHECK_ARG(mode == ORCA_MODE_BUDGET || mode == ORCA_MODE_REUSE_ALL || mode == ORCA_MODE_NO_REUSE);
  const bool budget = layers == 2 && mode == ORCA_MODE_BUDGET, history = layers == 2 && mode != ORCA_MODE_NO_REUSE;
  if (history) ORCA_CHECK_ARG(m->hist_emb != nullptr);
  if (budget) ORCA_CHECK_ARG(m->cache_flag && m->n_prev_plan && m->prev_plan);
  Ctx *c = m->ctx != nullptr ? reinterpret_cast<Ctx *>(m->ctx) : default_ctx();
  if (c == nullptr) return set_error(ORCA_E_CUDA, "orca_tgn_eval_group: no context for the current device");
  CtxScope scope(c);
  if (!projections_on_tensor_cores())
    return set_error(ORCA_E_UNSUPPORTED, "orca_tgn_eval_group: only with the tensor-core projections");
  const grp::Buffers w = grp::carve(d_workspace, g->bs, g->nb_max, k, g->u_cap, g->plan_cap, m->n_nodes, layers, mode);
  if ((int64_t)w.total > workspace_bytes)
    return set_error(ORCA_E_CAPACITY, "orca_tgn_eval_group: workspace of %lld bytes, %lld needed", (long long)workspace_bytes,
                     (long long)w.total);
  ORCA_CHECK_ARG(w.rows_max < (1 << grp::APP_ROW_BITS) &&
                 m->n_nodes + w.rows_max < INT_MAX);
  const int p = (int)(g->seq & 1);
  const grp::Parity &x = w.par[p], &prev = w.par[p ^ 1];
  const int E_max = g->nb_max * g->bs;
  grp::Args a{};
  a.indptr = m->indptr, a.adj_nbr = m->adj_nbr, a.adj_eid = m->adj_eid, a.adj_ts = m->adj_ts, a.n_nodes = m->n_nodes;
  a.nb = g->nb, a.bs = g->bs, a.b_last = g->b_last, a.k = k, a.mode = mode, a.layers = layers;
  a.u_cap1 = g->u_cap + 1;
  a.n_edge_rows = m->n_edge_rows > 0 ? (int)std::min<int64_t>(m->n_edge_rows, INT_MAX) : INT_MAX;
  const int64_t base_i32 = g->off_i32[0];
  int64_t n_i32 = 0;
  for (int n = 0; n < g->nb; ++n) {
    const int plan = std::max(g->n_plan[n], 0);
    ORCA_CHECK_ARG(g->off_i32[n] == base_i32 + n_i32 && plan <= g->plan_cap && (!budget || g->n_plan[n] >= 0));
    a.off[n] = (int)n_i32, a.n_plan[n] = plan;
    n_i32 += 4ll * a.b_of(n) + plan;
  }
  if (budget) ORCA_CHECK_ARG(a.n_plan[g->nb - 1] <= m->plan_cap);
  const int E = a.edges();
  a.img = (const int32_t *)x.stage;
  const size_t ts_off = grp::align_up((size_t)(4ll * E_max + (int64_t)g->nb_max * g->plan_cap) * 4);
  a.ts = (const double *)(x.stage + ts_off);
  a.cache_flag = m->cache_flag, a.status = d_status;
  a.bits = x.bits, a.table = x.table, a.app_table = x.app_table, a.cnt = x.cnt;
  a.table_mask = w.table_size - 1, a.app_mask = w.app_size - 1;
  if (g->seq > 0) a.prev_bits = prev.bits, a.prev_table = prev.table, a.prev_mask = w.table_size - 1;
  a.cand = x.cand, a.app_node = x.app_node, a.nbr1 = x.nbr1, a.eid1 = x.eid1, a.dt1 = x.dt1, a.nbr2 = x.nbr2;
  a.own1 = x.own1, a.own_seen = x.own_seen, a.own_list = x.own_list, a.own_at = x.own_at;
  a.win_node = x.win_node, a.win_eid = x.win_eid, a.win_mem = x.win_mem, a.win_other = x.win_other, a.win_t = x.win_t, a.win_gap = x.win_gap;
  a.last_at = x.last_at, a.last_node = x.last_node;
  a.split = 2 * E > grp::SPLIT_FROM;
  a.prev_win_t = prev.win_t;
  a.log_base = (int)m->n_nodes + p * 2 * E_max, a.prev_log_base = (int)m->n_nodes + (p ^ 1) * 2 * E_max;
  // second parts of the two-part tables, moved back by the first part's rows
  const float *log = w.log - (size_t)m->n_nodes * D;
  const float *emb = w.emb1 - (size_t)m->n_nodes * D;

  int32_t *saved_status = c->status_word;
  c->status_word = d_status;
  if (g->phase & 1) launch_counter() = 0;
  cudaStream_t s = (cudaStream_t)stream, si = c->overlap ? c->idx : s, sx = c->overlap ? c->aux : s;
  auto prepare = [&]() -> int {
    // ---- inputs and index stream
    cudaStream_t sc = c->overlap ? c->copy : s;
    if (g->seq == 0) {
      ORCA_CUDA(cudaEventRecord(c->ev_gin, s));
      if (sc != s) ORCA_CUDA(cudaStreamWaitEvent(sc, c->ev_gin, 0));
      c->gdone_recorded[0] = c->gdone_recorded[1] = false;
    }
    if (c->gdone_recorded[p] && sc != s) ORCA_CUDA(cudaStreamWaitEvent(sc, c->ev_gdone[p], 0));
    ORCA_CUDA(cudaMemcpyAsync(x.stage, g->h_i32 + base_i32, (size_t)n_i32 * 4, cudaMemcpyHostToDevice, sc));
    ORCA_CUDA(cudaMemcpyAsync(x.stage + ts_off, g->h_ts, (size_t)E * 8, cudaMemcpyHostToDevice, sc));
    if (si != sc) {     // (in order behind the copies: the parity's buffers are free, too)
      ORCA_CUDA(cudaEventRecord(c->ev_gin, sc));
      ORCA_CUDA(cudaStreamWaitEvent(si, c->ev_gin, 0));
    }
    ORCA_TRY(grp::launch_index(a, m->mem.last_update, x.zero_bytes, g->h_rows + p, c->ev_gcount[p], si, c->sm_count));
    if (si != sx) {
      ORCA_CUDA(cudaEventRecord(c->ev_gidx[p], si));
      ORCA_CUDA(cudaStreamWaitEvent(sx, c->ev_gidx[p], 0));
    }
    if (budget) {
      const int last = g->nb - 1;
      ORCA_TRY(launch_plan_flags(m, a.img + a.off[last] + 4 * g->b_last, a.n_plan[last], si));
    }
    if (si != s) ORCA_CUDA(cudaEventRecord(c->ev_gidx[p], si));     // (from here on: index work and flags)
    // ---- memory chain
    grp::ChainArgs ch{a, m->mem, log, w.log + (size_t)p * 2 * E_max * D, m->edge_table, m->time_w, m->gru.Wg_chain, m->gru.bg,
                      x.upd_image, a.split ? w.msg_image : nullptr, nullptr, 0};
    ORCA_TRY(grp::launch_gru_chain(ch, sx));
    if (a.split)
      ORCA_TRY(gru_rows(&m->gru, m->mem, w.msg_image, x.last_node, x.last_at, (int)std::min<int64_t>(2 * E, m->n_nodes), &x.cnt->n_last,
                        ch.log_out, sx));
    if (sx != s) ORCA_CUDA(cudaEventRecord(c->ev_gchain[p], sx));
    return ORCA_OK;
  };
  auto finish = [&]() -> int {
    ORCA_CUDA(cudaEventSynchronize(c->ev_gcount[p]));
    const int n_rows = g->h_rows[p];
    ORCA_CHECK_ARG(n_rows >= 3 * E && n_rows <= w.rows_max);
    if (sx != s) {
      ORCA_CUDA(cudaStreamWaitEvent(s, c->ev_gchain[p], 0));
      ORCA_CUDA(cudaStreamWaitEvent(s, c->ev_gidx[p], 0));
    }
    int32_t *tk = c->d_words + CTX_TICKET_MAIN;
    auto output = [&](int layer, int rows, const int32_t *own_row, float *out) {
      OutArgs o{};
      o.w = m->attn[layer], o.ctx = w.ctx, o.own = w.own, o.own_row = own_row, o.valid = w.valid, o.n_cap = rows, o.out = out;
      if (layer == layers - 1) o.pair_image = w.pairs, o.pair_bs = g->bs, o.pair_nb = g->nb, o.pair_last = g->b_last;
      return o;
    };
    // (a group with a cold cache, whose rows take several chunks, goes without sharing)
    const bool shared = n_rows <= w.chunk;
    for (int r0 = 0; r0 < n_rows; r0 += w.chunk) {
      const int rows = std::min(w.chunk, n_rows - r0);
      const size_t slot = (size_t)r0 * k;
      const tc::RowSrc own{m->mem.memory, shared ? x.own_list : x.own1 + r0, D, 0, 0, log, (int)m->n_nodes};
      const int32_t *d_own = shared ? &x.cnt->n_own : nullptr, *own_at = shared ? x.own_at : nullptr;
      ORCA_TRY(feat_image(own, rows, d_own, w.feat, s));
      ORCA_TRY(attn_query_image(&m->attn[0], w.feat, rows, d_own, w.qt, w.own, s));
      ORCA_TRY(launch_attn_gather(w.qt, m->mem.memory, m->edge_table, m->time_w, x.nbr1 + slot, x.eid1 + slot, x.dt1 + slot, k,
                                  rows, nullptr, 0, nullptr, w.ctx, true, w.valid, tk, s, log, (int)m->n_nodes, own_at));
      OutArgs o = output(0, rows, own_at, layers == 2 ? w.emb1 + (size_t)r0 * D : nullptr);
      // (the batch rows are layer 2's rows; they all lie in the first chunk)
      if (layers == 2 && r0 == 0) o.out_image = w.feat2, o.out_image_rows = 3 * E;
      ORCA_TRY(attn_output_rows(o, s));
    }
    if (layers == 2) {
      ORCA_TRY(attn_query_image(&m->attn[1], w.feat2, 3 * E, nullptr, w.qt, w.own, s));
      // (without reuse every row lies in the layer-1 output: the first part is never read)
      ORCA_TRY(launch_attn_gather(w.qt, history ? m->hist_emb : m->mem.memory, m->edge_table, m->time_w, x.nbr2, x.eid1,
                                  x.dt1, k, 3 * E, nullptr, 0, nullptr, w.ctx, true, w.valid, tk, s, emb, (int)m->n_nodes));
      ORCA_TRY(attn_output_rows(output(1, 3 * E, nullptr, nullptr), s));
    }
    ORCA_TRY(score_rows(&m->score, w.pairs, 2 * E, d_prob, s));
    ORCA_CUDA(launch_dep(grp::write_back_kernel, c->sm_count * 8, 256, 0, s, a, log, (const float *)w.emb1, m->mem.memory,
                         m->hist_emb, g->h_status));
    ORCA_COUNT_LAUNCH();
    if (g->d_metrics != nullptr) {
      ORCA_TRY(launch_link_metrics(d_prob, g->nb, g->bs, g->b_last, g->d_metrics, s));
      ORCA_CUDA(cudaMemcpyAsync(g->h_metrics, g->d_metrics, (size_t)g->nb * orca_link_metric_parts(g->bs) * 4 * sizeof(double),
                                cudaMemcpyDeviceToHost, s));
    }
    if (h_prob != nullptr) ORCA_CUDA(cudaMemcpyAsync(h_prob, d_prob, (size_t)2 * E * 4, cudaMemcpyDeviceToHost, s));
    ORCA_CUDA(cudaEventRecord(c->ev_gdone[p], s));
    c->gdone_recorded[p] = true;
    return ORCA_OK;
  };
  auto body = [&]() -> int {
    if (g->phase & 1) ORCA_TRY(prepare());
    return g->phase & 2 ? finish() : ORCA_OK;
  };
  const int rc = body();
  c->status_word = saved_status;
  c->last_batch_launches = launch_counter();
  return settled(rc, c, s);
}

}  // extern "C"
