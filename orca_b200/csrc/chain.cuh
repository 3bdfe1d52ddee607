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

}  // namespace grp
}  // namespace orca
