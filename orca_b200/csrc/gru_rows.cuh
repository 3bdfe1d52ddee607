// Operand image of messages, and the memory updates that read it (gru_rows.cu).
#pragma once

#include "attn_out.cuh"

namespace orca {

// The message's four parts of 172 columns, padded to 176, in the order of the packed GRU weights: edge features, time
// encoding, own memory, other memory.  The memory row's own product (the weights' fifth part) reads the own part again.
constexpr int GRU_IMG_STAGES = 4 * tc::GRU_PART / 32, GRU_IMG_OWN = 2 * tc::GRU_PART;
static_assert(4 * tc::GRU_PART % 32 == 0, "");
inline size_t gru_image_bytes(int64_t rows) { return img::bytes(rows, GRU_IMG_STAGES); }

// piece c (columns 4 c .. 4 c + 3) of a part of message number `row`; parts as the message table has them: own memory, other
// memory, edge features, time encoding.  The last piece brings the padding behind it.
__device__ __forceinline__ void put_message(char *image, int row, int part, int c, float4 x) {
  const int col = ((part + 2) & 3) * tc::GRU_PART + 4 * c;
  img::put4<GRU_IMG_STAGES>(image, row, col, x);
  if (c == D / 4 - 1) img::put4<GRU_IMG_STAGES>(image, row, col + 4, make_float4(0.f, 0.f, 0.f, 0.f));
}

// orca_message_store, which also writes the image of the messages (d_image: optional), in the order of the winners
int message_store(const orca_memory_t *mem, const float *d_edge_table, const float *d_time_w, const int32_t *d_cat_src,
                  const int32_t *d_cat_dst, const double *d_ts, const int32_t *d_eidx, int32_t b, const int32_t *d_win_pos,
                  int32_t n_win_cap, const int32_t *d_n_win, int32_t *d_win_nodes, char *d_image, cudaStream_t s);
// row m of the image: the message of node d_node[m], whose new memory goes to row d_out_row[m] (nullptr: m) of d_out; the old
// memory is the own part of the message table's row
int gru_rows(const orca_gru_weights_t *w, const orca_memory_t &mem, const char *d_image, const int32_t *d_node,
             const int32_t *d_out_row, int cap, const int32_t *d_n, float *d_out, cudaStream_t s);

}  // namespace orca
