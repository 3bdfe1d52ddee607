// Interface of the memory-update chain of a group of batches (chain.cu).
#pragma once

#include <algorithm>

#include "group.cuh"

namespace orca {
namespace grp {

struct ChainArgs {
  Args a;
  orca_memory_t mem;
  const float *log;         // second part of (memory table | log), moved back by the table's rows
  float *log_out;           // the group's log rows: update w of batch n at row n * 2 * bs + w
  const float *edge_table, *time_w;
  const void *w;            // weights.prepare_gru: one image per column tile
  const float *bias;
  void *image;              // update_image_bytes(nb * 2 * bs)
  char *msg_image;          // optional: operand image of the messages of every node's last update (gru_rows.cuh)
  int32_t *status;          // set by launch_gru_chain
  long long wait_limit;
};
// split edge features and time encodings of the updates: 44 chunks of 32 bytes each
inline size_t update_image_bytes(int64_t updates) { return (size_t)updates * 44 * 32; }
// all memory updates of the group, then message table, times and flags
int launch_gru_chain(const ChainArgs &g, cudaStream_t s);
// The updates of one batch on its own (batch by batch): d_cnt->n_win[0] of them at the list's pointers, new rows to
// d_rows; d_image: update_image_bytes(2 * b).  The memory table is written by scatter_updates.
int launch_gru_single(const orca_memory_t &mem, const orca_gru_weights_t &w, const float *edge_table, const float *time_w,
                      int b, const int32_t *d_node, const int32_t *d_other, const int32_t *d_eid, const float *d_t,
                      Counters *d_cnt, void *d_image, float *d_rows, cudaStream_t s);
int scatter_updates(const orca_memory_t &mem, const int32_t *d_node, const Counters *d_cnt, int cap, const float *d_rows,
                    cudaStream_t s);

}  // namespace grp
}  // namespace orca
