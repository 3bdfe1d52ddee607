// The operand image between the gather kernel and the output kernel of an attention layer, and the output kernel.
#pragma once

#include "common.cuh"
#include "tc_gemm.cuh"
#include "tc_ptx.cuh"

namespace orca {
namespace img {

// Operand images.  The products of an attention layer read their rows as bf16 heads and tails.  They are written once,
// by the kernels that compute them, in the form the tensor core reads from shared memory: blocks of 128 rows, K in
// stages of 32 columns, a stage = [128 rows x 64 bytes of heads | the same of tails] with the 16-byte chunks of a row
// swizzled by bits 1 and 2 of the row (64-byte swizzle), so that a stage is one contiguous copy and a row's piece of
// it one 64-byte write.  Two images per layer: the rows' own features (172 columns, padded to 192; attn_query.cu) and the
// attention sums (1032 columns, padded to 1056; attn_out.cu).  Padding is zero.
constexpr int ROWS = 128;
constexpr int STAGE_K = 32;
constexpr int STAGE_BYTES = 2 * ROWS * STAGE_K * 2;
constexpr int FEAT_STAGES = 6, CTX_STAGES = 33;
constexpr int PAIR_STAGES = 11;     // two embeddings one after the other, 344 columns, padded to 352 (score_rows.cu)
inline size_t bytes(int64_t rows, int stages) { return (size_t)((rows + ROWS - 1) / ROWS) * stages * STAGE_BYTES; }

// columns c .. c + 3 of row r: heads, and tails half a stage further
template <int STAGES>
__device__ __forceinline__ char *at(char *image, int r, int c) {
  return image + ((size_t)(r / ROWS) * STAGES + (c >> 5)) * STAGE_BYTES + (r % ROWS) * 64 +
         ((((c >> 3) & 3) ^ ((r >> 1) & 3)) << 4) + 2 * (c & 7);
}
template <int STAGES>
__device__ __forceinline__ void put4(char *image, int r, int c, float4 x) {
  uint2 hi, lo;
  hi.x = tc::pack_split(x.x, x.y, lo.x);
  hi.y = tc::pack_split(x.z, x.w, lo.y);
  char *p = at<STAGES>(image, r, c);
  *reinterpret_cast<uint2 *>(p) = hi;
  *reinterpret_cast<uint2 *>(p + STAGE_BYTES / 2) = lo;
}
__device__ __forceinline__ uint64_t desc_sw64(uint32_t addr) {   // K-major, 64-byte swizzle: 8 rows = 512 bytes
  return (uint64_t)((addr >> 4) & 0x3fff) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 |
         (uint64_t)4 << 61;
}

}  // namespace img

struct OutArgs {
  orca_attn_weights_t w;
  const char *ctx;            // operand image of the rows' attention sums
  const float *own;           // [., OWN_LD] what the rows' own features add to the hidden layer (attn_query.cu)
  const int32_t *own_row;     // row m's place in it (nullptr: m)
  const uint8_t *valid;       // rows whose slots are all padding have no attention term
  int n_cap;
  const int32_t *d_n;
  float *out;                 // [rows, 172]; may be nullptr where pair_image is not
  char *out_image;            // optional: operand image of the first out_image_rows rows (the next layer's features)
  int out_image_rows;
  // optional: operand image of the pairs that are scored.  The rows are [src | dst | neg] of pair_nb batches of pair_bs edges
  // (the last one: pair_last), the pairs [positive | negative] of batch n from n * 2 * pair_bs on.
  char *pair_image;
  int pair_bs, pair_nb, pair_last;
  // optional history push: winners by flag, or (push_win == nullptr) by record: row m wins if m >= push_all_from or
  // push_last_pos[push_ids[m]] == push_base + m
  float *push_table;
  const int32_t *push_ids;
  const uint8_t *push_win;
  const unsigned long long *push_last_pos;
  long long push_base;
  int push_all_from;
  tc::PeerOut peer;           // peer.world == 0: no delivery
  int32_t *status;            // set by attn_output_rows from the context
  long long wait_limit;
};
// operand image of rows of a (two-part) table
int feat_image(const tc::RowSrc &feat, int n_cap, const int32_t *d_n, char *d_image, cudaStream_t s);
// qt = feat . Mq + cq and (optional) own = feat . G[1032:], [., OWN_LD], from the rows' image
int attn_query_image(const orca_attn_weights_t *w, const char *d_image, int n_cap, const int32_t *d_n, float *d_qt,
                     float *d_own, cudaStream_t s);
int attn_output_rows(const OutArgs &g, cudaStream_t s);
// scores of pairs that lie in an operand image
int score_rows(const orca_score_weights_t *w, const char *d_pairs, int pairs, float *d_prob, cudaStream_t s);

}  // namespace orca
