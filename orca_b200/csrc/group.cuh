// A group of consecutive batches as one unit of work (group.cu): device-side description shared by its kernels.
#pragma once

#include "common.cuh"

namespace orca {
namespace grp {

constexpr int MAX_BATCHES = ORCA_GROUP_MAX;   // (a batch is a bit of a 32-bit word)
static_assert(MAX_BATCHES <= 32, "a batch of the group is a bit of a 32-bit word");

// What the batches of the group do with a node: bit n belongs to batch n.
struct NodeBits {
  uint32_t cached;    // its historical embedding is cached when batch n samples
  uint32_t in_rows;   // it is a row of batch n (source, destination or negative)
  uint32_t positive;  // it is a source or destination of batch n: batch n updates its memory
  uint32_t fetched;   // it was sampled by batch n, is neither cached nor a row of it: batch n recomputes it
};
// (node, batch) -> its last row in the batch, and the place of its new memory row in the log
struct Entry {
  unsigned long long key;   // 0: free
  int32_t row;              // last row of the node in the batch, + 1
  int32_t pos;              // last position among [src | dst], + 1; later IN_LOG | place in the batch's log
};
constexpr int32_t IN_LOG = 1 << 30;

struct Counters {
  int32_t n_cand[MAX_BATCHES], low_cand[MAX_BATCHES] /* INT_MAX - smallest candidate */;
  // Memory updates of the batch: the memory chain's lie at the front of the batch's places, those that are left to one
  // launch behind the chain (Args::split) at the back.
  int32_t n_win[MAX_BATCHES], n_back[MAX_BATCHES];
  int32_t n_last;                          // entries of last_at
  int32_t n_own;                           // entries of own_list
  int32_t dropped[MAX_BATCHES];            // smallest candidate of the batch (-1: none): it is not recomputed
  int32_t app_off[MAX_BATCHES + 1];        // first recomputed row of the batch, counted from the group's first
  int32_t n_rows;                          // layer-1 rows of the group
  double t_max[MAX_BATCHES];               // latest query time of the batch
  int32_t arrived[MAX_BATCHES];            // CTAs of the memory chain that have finished the batch
};

struct Args {
  // graph, batches
  const int64_t *indptr;
  const int32_t *adj_nbr, *adj_eid;
  const double *adj_ts;
  int64_t n_nodes;
  int n_edge_rows;
  const int32_t *img;               // [src | dst | neg | eidx | plan] of batch n at off[n]
  const double *ts;                 // times of batch n at n * bs
  int nb, bs, b_last, k, mode, layers;
  int u_cap1;                       // candidates a batch can have (list capacity)
  int off[MAX_BATCHES], n_plan[MAX_BATCHES];
  const uint8_t *cache_flag;        // flags before the group's first batch
  int32_t *status;
  // index structures of this group and of the one before it (prev_bits == nullptr: its rows are in the tables)
  NodeBits *bits;
  Entry *table;
  unsigned long long *app_table;
  uint32_t table_mask, app_mask;
  const NodeBits *prev_bits;
  const Entry *prev_table;
  uint32_t prev_mask;
  Counters *cnt;
  int32_t *cand;                    // [nb][u_cap1]
  // layer-1 rows: the batches' rows, then the recomputed ones
  int32_t *app_node;
  int32_t *nbr1, *eid1;             // neighbours: sampled ids, then rows of (memory table | log)
  float *dt1;
  int32_t *nbr2;                    // batch rows: rows of (history table | layer-1 output)
  int32_t *own1;                    // row of (memory table | log) of the row's own node
  int32_t *own_seen;                // by row of (memory table | log): 1 + its place in own_list, 0: not there
  int32_t *own_list, *own_at;       // the distinct rows of own1, and own1's places in the list
  // memory updates: batch n's at n * 2 * bs (Counters says which of these places are taken)
  int32_t *win_node, *win_eid, *win_mem, *win_other;
  float *win_t, *win_gap;           // time of the update, and since the node's update before it
  int32_t *last_at, *last_node;     // the last update of every node that the group updates: place, node
  int split;                        // whether last updates are left out of the memory chain (group.cu)
  const float *prev_win_t;
  int log_base, prev_log_base;      // row of (memory table | log) where this / the previous group's log starts

  __host__ __device__ int b_of(int n) const { return n == nb - 1 ? b_last : bs; }
  __host__ __device__ int edges() const { return (nb - 1) * bs + b_last; }
  __device__ bool budget() const { return layers == 2 && mode == ORCA_MODE_BUDGET; }
  // whether place w of batch n holds an update
  __device__ bool is_update(int n, int w) const { return w < cnt->n_win[n] || w >= 2 * bs - cnt->n_back[n]; }
  // whether a later batch of the group updates node v (and reads what batch n's update leaves)
  __device__ bool again(int v, int n) const { return (unsigned long long)__ldcg(&bits[v].positive) >> (n + 1) != 0; }
  __device__ bool keeps_history() const { return layers == 2 && mode != ORCA_MODE_NO_REUSE; }
};

// ---- (node, batch) tables: open addressing, capacity at least twice the entries
__device__ __forceinline__ unsigned long long key_of(int v, int n) { return ((unsigned long long)(uint32_t)v << 5 | (unsigned)n) + 1; }
__device__ __forceinline__ uint32_t hash_of(unsigned long long key) {
  return (uint32_t)((key * 0x9e3779b97f4a7c15ull) >> 32);
}
__device__ __forceinline__ int find_entry(const Entry *t, uint32_t mask, int v, int n) {
  const unsigned long long key = key_of(v, n);
  uint32_t h = hash_of(key) & mask;
  for (uint32_t i = 0; i <= mask; ++i, h = (h + 1) & mask)   // (the entry is there: found after a step or two)
    if (t[h].key == key) break;
  return (int)h;
}
// recomputed rows: one word per entry, key << 27 | (row + 1)
constexpr int APP_ROW_BITS = 27;

// row of (memory table | log) that holds node v's memory when batch n of the group reads it
__device__ __forceinline__ int memory_row(const Args &a, int v, int n) {
  const uint32_t m = a.bits[v].positive & ((1u << n) - 1u);
  if (m == 0) return v;
  const int last = 31 - __clz(m);
  return a.log_base + last * 2 * a.bs + (a.table[find_entry(a.table, a.table_mask, v, last)].pos & ~IN_LOG);
}
// the same while the previous group's rows may not have reached the table yet
__device__ __forceinline__ int memory_row_early(const Args &a, int v, int n) {
  const int r = memory_row(a, v, n);
  if (r != v || a.prev_bits == nullptr) return r;
  const uint32_t m = a.prev_bits[v].positive;
  if (m == 0) return v;
  const int last = 31 - __clz(m);
  return a.prev_log_base + last * 2 * a.bs + (a.prev_table[find_entry(a.prev_table, a.prev_mask, v, last)].pos & ~IN_LOG);
}
// time of the node's last update before batch n; `row`: its memory row (memory_row_early)
__device__ __forceinline__ float last_update_of(const Args &a, const float *last_update, int v, int row) {
  if (row < a.n_nodes) return last_update[v];
  const int mine = row - a.log_base;
  return mine >= 0 && mine < a.nb * 2 * a.bs ? a.win_t[mine] : a.prev_win_t[row - a.prev_log_base];
}
// row of (history table | layer-1 output) that holds node v's embedding when batch n's top layer reads it: the
// latest push up to and including batch n's own
__device__ __forceinline__ int history_row(const Args &a, int v, int n) {
  const NodeBits b = a.bits[v];
  const uint32_t m = (b.in_rows | b.fetched) & (0xffffffffu >> (31 - n));
  if (m == 0) return v;
  const int last = 31 - __clz(m);
  if (b.in_rows >> last & 1u)
    return (int)a.n_nodes + 3 * last * a.bs + a.table[find_entry(a.table, a.table_mask, v, last)].row - 1;
  const unsigned long long key = key_of(v, last);
  uint32_t h = hash_of(key) & a.app_mask;
  unsigned long long e = 0;
  for (uint32_t i = 0; i <= a.app_mask; ++i, h = (h + 1) & a.app_mask) {
    e = a.app_table[h];
    if ((e >> APP_ROW_BITS) == key) break;
  }
  return (int)a.n_nodes + 3 * a.edges() + (int)(e & ((1ull << APP_ROW_BITS) - 1)) - 1;
}

}  // namespace grp

// metrics.cu: records of a group's scores ([pos | neg] of batch n from n * 2 * bs)
int launch_link_metrics(const float *d_prob, int nb, int bs, int b_last, double *d_out, cudaStream_t s);
}  // namespace orca
