// Memory updates whose inputs are all there: gates = [message | memory] . Wg + bg and the new memory row, for rows that come
// as an operand image (attn_out.cuh) of the message's four parts.
//
// The update of a single call and the last updates of a group.  A tile of the general projection
// kernel, whose producer warps fetch fp32 rows, convert and store them k-block by k-block, four times over (once per tile of
// 44 units), takes 30 us; here the kernels that store the messages (state.cu, chain.cu) write the parts' heads and tails as
// well, and the main loop is bulk copies and MMAs: 28 stages of 32 columns (16 KB of rows, 22 KB of weights) through a ring of
// five, the memory row's product from the image of the message's own part.  A unit of work is a row block of 128 and a tile of
// 176 gate columns; its gates are worked out while the next unit's stages land.
// 8 k rows (a group of eleven batches of 2000 edges): 60 -> 32 us; 900 rows (one batch): 34 -> 20.
// Every unit's products are the ones of the general kernel and of the memory chain, k-step by k-step: the same bits.
// Warp 0: copies.  Warp 1: tensor memory, MMA issue.  Warps 2-9: gates (thread = row, half of the tile's units).
#include <algorithm>

#include "attn_out.cuh"
#include "context.cuh"
#include "gru_rows.cuh"
#include "tc_ptx.cuh"

namespace orca {
namespace gr {

constexpr int BM = img::ROWS, BN = 176, TILES = 4, UNITS = BN / 4;
constexpr int A_STAGE = img::STAGE_BYTES, W_LBO = BN * 16, W_HALF = 4 * W_LBO, STAGE = A_STAGE + 2 * W_HALF;
constexpr int K_STAGES = (tc::GRU_K + 31) / 32;                       // 28, the last one half
constexpr int OWN_STAGE = GRU_IMG_OWN / 32;                           // where the own part starts: also the memory row's operand
constexpr int KB_BYTES = 4 * W_HALF, KBS = (tc::GRU_K + 63) / 64;     // the packed weights are blocks of 64 rows
static_assert(GRU_IMG_OWN % 32 == 0 && tc::GRU_K == GRU_IMG_STAGES * 32 + tc::GRU_PART && tc::BN == BN, "");
constexpr int SLOTS = 5;
constexpr int SMEM = SLOTS * STAGE + 1024;
constexpr int EPI_WARPS = 8, THREADS = 64 + 32 * EPI_WARPS;
constexpr int TMEM_COLS = 512, SMALL = 256;

struct Args {
  const char *image;
  const void *w;
  const float *bias, *messages;
  const int32_t *nodes, *out_rows, *d_n;
  float *out;
  int n_cap;
  int32_t *status;
  long long wait_limit;
};

__global__ void __launch_bounds__(THREADS, 1) gru_rows_kernel(const __grid_constant__ Args g) {
  using namespace tc;
  extern __shared__ unsigned char raw[];
  __shared__ __align__(16) float s_bias[TILES * BN];
  __shared__ __align__(8) unsigned long long s_bar[2 * SLOTS + 2];
  __shared__ uint32_t s_tmem;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const uint32_t base = (smem_addr(raw) + 1023u) & ~1023u;
  auto full = [&](int s) { return smem_addr(&s_bar[s]); };
  auto empty = [&](int s) { return smem_addr(&s_bar[SLOTS + s]); };
  const uint32_t accfull = smem_addr(&s_bar[2 * SLOTS]), accfree = smem_addr(&s_bar[2 * SLOTS + 1]);
  dep_trigger();
  if (tid == 0) {
    for (int s = 0; s < SLOTS; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), 1);
    }
    mbar_init(accfull, 1);
    mbar_init(accfree, EPI_WARPS);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&s_tmem)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  for (int i = tid; i < TILES * BN; i += THREADS) s_bias[i] = g.bias[i];
  dep_wait();
  const int M = rows_of(g.n_cap, g.d_n), units = (M + BM - 1) / BM * TILES;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *(volatile uint32_t *)&s_tmem, 0);
  bool alive = true;

  if (warp == 0) {
    if (lane == 0) {
      int it = 0;
      for (int u = blockIdx.x; alive && u < units; u += gridDim.x) {
        const char *rows = g.image + (size_t)(u / TILES) * GRU_IMG_STAGES * A_STAGE;
        const char *w = reinterpret_cast<const char *>(g.w) + (size_t)(u % TILES) * KBS * KB_BYTES;
        for (int st = 0; st < K_STAGES; ++st, ++it) {
          const int s = it % SLOTS;
          const uint32_t at = base + s * STAGE;
          mbar_wait(empty(s), ((it / SLOTS) & 1) ^ 1, g.status, 900, alive, g.wait_limit);
          if (!alive) break;
          mbar_expect_tx(full(s), STAGE);
          bulk_g2s(at, rows + (size_t)(st < GRU_IMG_STAGES ? st : st - GRU_IMG_STAGES + OWN_STAGE) * A_STAGE, A_STAGE, full(s));
          const char *kb = w + (size_t)(st / 2) * KB_BYTES + (st & 1) * W_HALF;     // (heads of 64 rows, then their tails)
          bulk_g2s(at + A_STAGE, kb, W_HALF, full(s));
          bulk_g2s(at + A_STAGE + W_HALF, kb + 2 * W_HALF, W_HALF, full(s));
        }
      }
      for (int q = max(0, it - SLOTS); q < it; ++q) mbar_settle(full(q % SLOTS), (q / SLOTS) & 1);
    }
    __syncwarp();
  } else if (warp == 1) {
    constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
    int it = 0, t = 0;
    for (int u = blockIdx.x; u < units; u += gridDim.x, ++t) {
      if (t > 0) mbar_wait(accfree, (t - 1) & 1, g.status, 910, alive, g.wait_limit);
      tc_fence_after();
      for (int st = 0; st < K_STAGES; ++st, ++it) {
        const int s = it % SLOTS;
        const uint32_t a = base + s * STAGE, w = a + A_STAGE;
        mbar_wait(full(s), (it / SLOTS) & 1, g.status, 911, alive, g.wait_limit);
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < 2; ++ks) {
            if (!alive || (ks == 1 && st == K_STAGES - 1)) break;      // (the last half is nothing but padding)
            const uint64_t ah = img::desc_sw64(a + ks * 32), al = img::desc_sw64(a + A_STAGE / 2 + ks * 32);
            const uint64_t bh = make_desc(w + ks * 2 * W_LBO, W_LBO, 128), bl = make_desc(w + W_HALF + ks * 2 * W_LBO, W_LBO, 128);
            const uint32_t more = st > 0 || ks > 0 ? 1u : 0u;
            mma_bf16(tmem, ah, bh, idesc, more);
            mma_bf16(tmem + SMALL, al, bh, idesc, more);
            mma_bf16(tmem + SMALL, ah, bl, idesc, 1u);
          }
          if (alive) mma_commit(empty(s));
          if (st == K_STAGES - 1) mma_commit(accfull);
        }
        __syncwarp();
      }
    }
    if (t > 0) mbar_settle(accfull, (t - 1) & 1);
  } else {
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const int row = quarter * 32 + lane, ch0 = half ? 6 : 0, nc = half ? 5 : 6;     // chunks of 16 columns: four units
    const uint32_t trow = tmem + ((uint32_t)(quarter * 32) << 16) + ch0 * 16;
    int t = 0;
    for (int u = blockIdx.x; u < units; u += gridDim.x, ++t) {
      const int m = u / TILES * BM + row, nt = u % TILES, unit0 = nt * UNITS + 4 * ch0;
      const bool live = m < M;
      const int to = live ? (g.out_rows != nullptr ? g.out_rows[m] : m) : 0;
      float4 h[6];      // old memory: the message's own part
#pragma unroll
      for (int c = 0; c < 6; ++c) h[c] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (live) {
        const float4 *src = reinterpret_cast<const float4 *>(g.messages + (size_t)g.nodes[m] * MSG + unit0);
#pragma unroll
        for (int c = 0; c < 6; ++c)
          if (c < nc && unit0 + 4 * c < D) h[c] = __ldg(src + c);
      }
      mbar_wait(accfull, t & 1, g.status, 920, alive, g.wait_limit);
      tc_fence_after();
      float v[6][16];
#pragma unroll
      for (int c = 0; c < 6; ++c)
        if (c < nc) tmem_ld16_sum(trow + c * 16, SMALL, v[c]);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(accfree);      // (the next unit's products may start)
      const float *bias = s_bias + nt * BN + 16 * ch0;
      float4 *out = reinterpret_cast<float4 *>(g.out + (size_t)to * D + unit0);
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        if (c >= nc || unit0 + 4 * c >= D) break;
        const float ho[4] = {h[c].x, h[c].y, h[c].z, h[c].w};
        float o[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 b = *reinterpret_cast<const float4 *>(bias + 16 * c + 4 * i);
          o[i] = gru_gates(make_float4(v[c][4 * i] + b.x, v[c][4 * i + 1] + b.y, v[c][4 * i + 2] + b.z, v[c][4 * i + 3] + b.w), ho[i]);
        }
        if (live) out[c] = make_float4(o[0], o[1], o[2], o[3]);
      }
    }
    __syncwarp();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}

}  // namespace gr

int gru_rows(const orca_gru_weights_t *w, const orca_memory_t &mem, const char *d_image, const int32_t *d_node,
             const int32_t *d_out_row, int cap, const int32_t *d_n, float *d_out, cudaStream_t s) {
  if (cap <= 0) return ORCA_OK;
  Ctx *c = cur();
  if (c == nullptr) return set_error(ORCA_E_CUDA, "gru_rows: no context for the current device");
  ORCA_CHECK_ARG(w->Wg_tc != nullptr && w->bg != nullptr && mem.messages != nullptr && d_image && d_node && d_out);
  static thread_local int configured_device = -1;
  if (configured_device != c->device) {
    ORCA_CUDA(cudaFuncSetAttribute(gr::gru_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, gr::SMEM));
    configured_device = c->device;
  }
  const gr::Args g{d_image, w->Wg_tc, w->bg, mem.messages, d_node, d_out_row, d_n, d_out, cap, c->status_word, c->wait_limit};
  const int units = ceil_div(cap, gr::BM) * gr::TILES;
  ORCA_CUDA(launch_dep(gr::gru_rows_kernel, std::min(units, c->sm_count), gr::THREADS, gr::SMEM, s, g));
  ORCA_COUNT_LAUNCH();
  ORCA_LAUNCH_CHECK();
  return ORCA_OK;
}

}  // namespace orca
