// Link scores from the operand image of the pairs: p = sigmoid(relu([a | b] . W1t + b1) . w2 + b2).
//
// The output kernel of the top layer (attn_out.cu) writes a row's heads and tails where the pairs that it is part of want
// them, so that a pair's two embeddings lie side by side and nobody fetches or converts them again; its 344 columns are 11
// stages of bulk copies and MMAs against 22 KB of weights each, the hidden layer's dot product is taken from the accumulators
// while the next block's stages land.  The general projection kernel, with two gathered fp32 rows a pair and a k-block after the
// other, took 13.4 us for one block and 36 for 44 k pairs; 10.6 and 24.5 here.
// The products are that kernel's, k-step by k-step, and so is the order of the sums: the same bits as orca_score.
// Warp 0: copies.  Warp 1: tensor memory, MMA issue.  Warps 2-9: dot products (thread = pair, half of the columns).
#include <algorithm>

#include "attn_out.cuh"
#include "context.cuh"
#include "tc_ptx.cuh"

namespace orca {
namespace sr {

constexpr int BM = img::ROWS, BN = 176;
constexpr int A_STAGE = img::STAGE_BYTES, W_LBO = BN * 16, W_HALF = 4 * W_LBO, STAGE = A_STAGE + 2 * W_HALF;
constexpr int K_STAGES = img::PAIR_STAGES;
constexpr int KB_BYTES = 4 * W_HALF;              // the packed weights are blocks of 64 rows: heads, then tails
static_assert(tc::BN == BN && tc::BK == 64 && 2 * D <= K_STAGES * img::STAGE_K, "");
constexpr int SLOTS = 5;
constexpr int SMEM = SLOTS * STAGE + 1024;
constexpr int EPI_WARPS = 8, THREADS = 64 + 32 * EPI_WARPS;
constexpr int TMEM_COLS = 512, SMALL = 256;

struct Args {
  const char *image;
  const void *w;
  const float *b1, *w2;
  float b2;
  float *prob;
  int n;
  int32_t *status;
  long long wait_limit;
};

__global__ void __launch_bounds__(THREADS, 1) score_rows_kernel(const __grid_constant__ Args g) {
  using namespace tc;
  extern __shared__ unsigned char raw[];
  __shared__ __align__(16) float s_b1[BN], s_w2[BN];
  __shared__ float s_dot[2][BM];
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
  for (int i = tid; i < BN; i += THREADS) {
    s_b1[i] = i < D ? g.b1[i] : 0.f;
    s_w2[i] = i < D ? g.w2[i] : 0.f;
  }
  dep_wait();
  const int blocks = (g.n + BM - 1) / BM;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *(volatile uint32_t *)&s_tmem, 0);
  bool alive = true;

  if (warp == 0) {
    if (lane == 0) {
      const uint64_t once = policy_evict_first();
      int it = 0;
      for (int blk = blockIdx.x; alive && blk < blocks; blk += gridDim.x) {
        const char *rows = g.image + (size_t)blk * K_STAGES * A_STAGE;
        for (int st = 0; st < K_STAGES; ++st, ++it) {
          const int s = it % SLOTS;
          const uint32_t at = base + s * STAGE;
          mbar_wait(empty(s), ((it / SLOTS) & 1) ^ 1, g.status, 1000, alive, g.wait_limit);
          if (!alive) break;
          mbar_expect_tx(full(s), STAGE);
          bulk_g2s_hint(at, rows + (size_t)st * A_STAGE, A_STAGE, full(s), once);
          const char *kb = reinterpret_cast<const char *>(g.w) + (size_t)(st / 2) * KB_BYTES + (st & 1) * W_HALF;
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
    for (int blk = blockIdx.x; blk < blocks; blk += gridDim.x, ++t) {
      if (t > 0) mbar_wait(accfree, (t - 1) & 1, g.status, 1010, alive, g.wait_limit);
      tc_fence_after();
      for (int st = 0; st < K_STAGES; ++st, ++it) {
        const int s = it % SLOTS;
        const uint32_t a = base + s * STAGE, w = a + A_STAGE;
        mbar_wait(full(s), (it / SLOTS) & 1, g.status, 1011, alive, g.wait_limit);
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < 2; ++ks) {
            if (!alive) break;
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
    const int row = quarter * 32 + lane, ch0 = half ? 6 : 0, ch1 = half ? BN / 16 : 6;     // chunks of 16 columns
    const uint32_t trow = tmem + ((uint32_t)(quarter * 32) << 16);
    int t = 0;
    for (int blk = blockIdx.x; blk < blocks; blk += gridDim.x, ++t) {
      mbar_wait(accfull, t & 1, g.status, 1020, alive, g.wait_limit);
      tc_fence_after();
      float dot = 0.f;
#pragma unroll 1
      for (int ch = ch0; ch < ch1; ++ch) {
        float v[16];
        tmem_ld16_sum(trow + ch * 16, SMALL, v);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const int c = ch * 16 + i;
          if (c < D) dot += relu(v[i] + s_b1[c]) * s_w2[c];
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(accfree);      // (the next block's products may start)
      // (two buffers: a warp writes one again only when its partner has read it, behind the barrier in between)
      if (half) s_dot[t & 1][row] = dot;
      asm volatile("bar.sync %0, 64;" ::"r"(1 + quarter) : "memory");
      const int m = blk * BM + row;
      if (!half && m < g.n) g.prob[m] = 1.f / (1.f + expf(-(dot + s_dot[t & 1][row] + g.b2)));
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

}  // namespace sr

int score_rows(const orca_score_weights_t *w, const char *d_pairs, int pairs, float *d_prob, cudaStream_t s) {
  if (pairs <= 0) return ORCA_OK;
  Ctx *c = cur();
  if (c == nullptr) return set_error(ORCA_E_CUDA, "score_rows: no context for the current device");
  ORCA_CHECK_ARG(w->W1t_tc != nullptr && w->b1 != nullptr && w->w2 != nullptr && d_pairs && d_prob);
  static thread_local int configured_device = -1;
  if (configured_device != c->device) {
    ORCA_CUDA(cudaFuncSetAttribute(sr::score_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sr::SMEM));
    configured_device = c->device;
  }
  const sr::Args g{d_pairs, w->W1t_tc, w->b1, w->w2, w->b2, d_prob, pairs, c->status_word, c->wait_limit};
  ORCA_CUDA(launch_dep(sr::score_rows_kernel, std::min(ceil_div(pairs, sr::BM), c->sm_count), sr::THREADS, sr::SMEM, s, g));
  ORCA_COUNT_LAUNCH();
  ORCA_LAUNCH_CHECK();
  return ORCA_OK;
}

}  // namespace orca
