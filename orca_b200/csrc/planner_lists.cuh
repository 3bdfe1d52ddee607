// What the cache planners share when they walk lists of distinct nodes instead of neighbour tables (planner_lists.cu).
#pragma once

#include "tie_shared.cuh"

namespace orca {
namespace lists {

constexpr int T = tie::T, NW = tie::NW;

// The distinct nodes of every batch in ascending order, batch b's from b * stride: its endpoints (TARGET set) and the
// out-of-batch neighbours of its table.
constexpr int32_t TARGET = (int32_t)0x80000000u;
struct Lists {
  int32_t *id;       // node | TARGET
  int32_t *mult;     // out-of-batch neighbours: entries of the table that hold the node
  int32_t *count;    // [batches]
  int64_t stride;
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
// code (optional): set to `code_init` for every node on the way
int launch_batch_lists(const int32_t *d_nodes, const int32_t *d_nbr, int64_t n_edges, int32_t bs, int32_t k, int64_t n_nodes,
                       const Lists &l, void *d_scratch, int32_t *d_code, int32_t code_init, cudaStream_t s);

// MRD over lists.  Candidate lists longer than CAP set *State::failed: the kernels of planner_mrd.cu do the plan then.
constexpr int CAP = tie::SHARED_MAX;
bool mrd_takes(int64_t n_edges, int32_t bs);
int64_t mrd_workspace_bytes(int64_t n_edges, int32_t bs, int32_t k, int64_t n_nodes, int32_t budget);
int launch_mrd(const int32_t *d_nodes, const int32_t *d_nbr, int64_t n_edges, int32_t bs, int32_t k, int64_t n_nodes,
               int32_t budget, int32_t *d_plan, int64_t plan_cap, int64_t *d_plan_off, int64_t *d_stats, int32_t *d_status,
               void *d_workspace, const int32_t **d_failed, cudaStream_t s);

}  // namespace lists
}  // namespace orca
