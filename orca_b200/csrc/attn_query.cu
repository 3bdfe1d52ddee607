// What an attention layer makes of its rows' own features, on the tensor cores: qt[r] = feat[row of r] . Mq + cq, [rows, 1056]
// floats, and own[r] = feat[row of r] . G[1032:], [rows, 192], the features' part of the merger's hidden layer (attn_out.cu
// adds it).
//
// A launch writes 5 KB per row and reads 0.7 six times over (once per weight tile).  A CTA keeps its weight
// tile (heads and tails of 208 columns) for the whole launch and walks row blocks of 128, which come as an operand image
// (attn_out.cuh): one thread streams 16 KB stages through a ring, one multiplies, eight warps carry the accumulators from
// tensor memory to the outputs, in whole lines through shared memory.  6 / 31 / 66 k rows: 16 / 55 / 106 us (qt alone,
// tiles of 176 columns: 14 / 50 / 92).  A group's layer 1, where 0.18 to 0.48 of the rows are distinct, asks for those
// only (66 k rows of the largest graph: 92 -> 51 us, 57 k of 600-edge batches 75 -> 20), and the output kernel leaves six of
// its 39 stages out.  What bounds it: 4.8 us a block and CTA against 2 of products; without the stores 66 us, stores alone 48.
// Measured instead, 6 / 31 / 66 k rows: pairs of CTAs with half of a tile of 224 columns each and six stages 22 / 71 / 141;
// stores of fragments without the boxes, five stages, 18 / 53 / 95; stores of the boxes by tensor map 16 / 53 / 104.
// orca_attn_query, whose rows come as floats and which wants qt alone (tiles of 176 columns), writes the image to scratch memory
// first: 14.7 / 20.8 / 84.4 us for 600 / 6000 / 51,000 rows, against 12.3 / 24.6 / 129 for a kernel of its own that split the rows eleven times over.
#include <algorithm>

#include "attn_out.cuh"
#include "context.cuh"
#include "tc_gemm.cuh"
#include "tc_ptx.cuh"

namespace orca {
namespace aqi {

constexpr int BM = 128;
constexpr int CHUNKS = 22, STEPS = CHUNKS / 2;                // K = 172, padded to 176
constexpr int TILES = 6;
// weights: per eight columns [head | tail][K / 8][8 columns][8], so that any whole number of them is one piece
constexpr int W_HALF = CHUNKS * 128, W_GROUP = 2 * W_HALF;
constexpr int STAGE = img::STAGE_BYTES;
constexpr int EPI_WARPS = 8, THREADS = 64 + 32 * EPI_WARPS;
constexpr int BOX = 32 * 128;                                 // of a warp: 32 rows x 32 columns on their way out
// OWN: the features' part of the hidden layer as well, in tiles of 208 columns; without it tiles of 176 and a stage more
// (orca_attn_query, 6 / 18 / 36 / 51 / 66 k rows, caches flushed: 20.8 / 37.2 / 63.8 / 84.4 / 106.8 us; with tiles of 208, whose
// last columns nobody asked for, 20.8 / 39.3 / 67.9 / 92.4 / 115.1)
template <bool OWN>
struct Tile {
  static constexpr int BN = OWN ? 208 : 176, CHUNKS_16 = BN / 16, MOST = (CHUNKS_16 + 1) / 2;   // MOST: 16-column chunks of a warp
  static constexpr int W_BYTES = BN / 8 * W_GROUP;
  static constexpr int STAGES = OWN ? 3 : 4;
  static constexpr int RING = (W_BYTES + 1023) / 1024 * 1024;      // (the swizzle wants aligned stages)
  static constexpr int SMEM = RING + STAGES * STAGE + EPI_WARPS * BOX + 1024;
  static_assert(TILES * BN >= QT_LD + (OWN ? D : 0) && QT_LD % 32 == 0 && OWN_LD % 32 == 0, "whole lines belong to one of the two outputs");
};
constexpr int TMEM_COLS = 512, SMALL = 256;                   // one buffer of main + cross-term accumulators

struct Args {
  const char *image;
  int n_cap;
  const int32_t *d_n;
  const void *w;
  const float *bias;
  float *qt, *own;
  int32_t *status;
  long long wait_limit;
};

template <bool OWN>
__global__ void __launch_bounds__(THREADS, 1) attn_query_image_kernel(const __grid_constant__ Args g) {
  using namespace tc;
  constexpr int BN = Tile<OWN>::BN, STAGES = Tile<OWN>::STAGES, W_BYTES = Tile<OWN>::W_BYTES, RING = Tile<OWN>::RING;
  extern __shared__ unsigned char raw[];
  __shared__ __align__(16) float s_bias[BN];
  __shared__ __align__(8) unsigned long long s_bar[2 * STAGES + 3];
  __shared__ uint32_t s_tmem;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int nt = blockIdx.x;
  const uint32_t base = (smem_addr(raw) + 1023u) & ~1023u, ring = base + RING;
  auto full = [&](int s) { return smem_addr(&s_bar[s]); };
  auto empty = [&](int s) { return smem_addr(&s_bar[STAGES + s]); };
  const uint32_t wbar = smem_addr(&s_bar[2 * STAGES]);
  const uint32_t accfull = smem_addr(&s_bar[2 * STAGES + 1]), accfree = smem_addr(&s_bar[2 * STAGES + 2]);
  dep_trigger();
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), 1);
    }
    mbar_init(wbar, 1);
    mbar_init(accfull, 1);
    mbar_init(accfree, EPI_WARPS);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_expect_tx(wbar, W_BYTES);       // (weights: written by nobody but the host, long ago)
    bulk_g2s(base, reinterpret_cast<const char *>(g.w) + (size_t)nt * W_BYTES, W_BYTES, wbar);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&s_tmem)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid >= 64 && tid < 64 + BN) s_bias[tid - 64] = nt * BN + tid - 64 < QT_LD ? g.bias[nt * BN + tid - 64] : 0.f;
  dep_wait();
  const int M = rows_of(g.n_cap, g.d_n);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *(volatile uint32_t *)&s_tmem, 0);
  bool alive = true;

  if (warp == 0) {
    if (lane == 0) {
      int it = 0;
      for (int blk = blockIdx.y; alive && blk * BM < M; blk += gridDim.y) {
        const char *rows = g.image + (size_t)blk * img::FEAT_STAGES * STAGE;
        for (int st = 0; st < img::FEAT_STAGES; ++st, ++it) {
          const int s = it % STAGES;
          mbar_wait(empty(s), ((it / STAGES) & 1) ^ 1, g.status, 540, alive, g.wait_limit);
          if (!alive) break;
          mbar_expect_tx(full(s), STAGE);
          bulk_g2s(ring + s * STAGE, rows + (size_t)st * STAGE, STAGE, full(s));
        }
      }
      mbar_settle(wbar, 0);
      for (int q = max(0, it - STAGES); q < it; ++q) mbar_settle(full(q % STAGES), (q / STAGES) & 1);
    }
    __syncwarp();
  } else if (warp == 1) {
    constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
    mbar_wait(wbar, 0, g.status, 550, alive, g.wait_limit);
    int it = 0, t = 0;
    for (int blk = blockIdx.y; blk * BM < M; blk += gridDim.y, ++t) {
      if (t > 0) mbar_wait(accfree, (t - 1) & 1, g.status, 551, alive, g.wait_limit);
#pragma unroll
      for (int st = 0; st < img::FEAT_STAGES; ++st, ++it) {
        const int s = it % STAGES;
        const uint32_t a = ring + s * STAGE;
        mbar_wait(full(s), (it / STAGES) & 1, g.status, 552, alive, g.wait_limit);
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < 2; ++ks) {
            if (2 * st + ks >= STEPS || !alive) continue;
            const uint32_t w = base + (2 * st + ks) * 2 * 128;
            const uint64_t ah = img::desc_sw64(a + ks * 32), al = img::desc_sw64(a + STAGE / 2 + ks * 32);
            const uint64_t bh = make_desc(w, 128, W_GROUP), bl = make_desc(w + W_HALF, 128, W_GROUP);
            const uint32_t more = st > 0 || ks > 0 ? 1u : 0u;
            mma_bf16(tmem, ah, bh, idesc, more);
            mma_bf16(tmem + SMALL, al, bh, idesc, more);
            mma_bf16(tmem + SMALL, ah, bl, idesc, 1u);
          }
          if (alive) mma_commit(empty(s));
          if (st == img::FEAT_STAGES - 1) mma_commit(accfull);
        }
        __syncwarp();
      }
    }
    if (t > 0) mbar_settle(accfull, (t - 1) & 1);
  } else {
    // A tile of 13 chunks of 16 columns: every other one starts in the middle of a 128-byte line.  The warps' parts are six
    // chunks from a line's start (even tiles: 0 and 6, odd ones: 1 and 7) and, for the first (odd) or last (even) four warps,
    // the half line that is left.  A tile of 11: six chunks and five, from its start.
    constexpr int MOST = Tile<OWN>::MOST;
    const int quarter = warp & 3, half = (warp - 2) >> 2, odd = OWN ? nt & 1 : 0;
    const int c0 = half * 6 + odd, single = odd ? 0 : 12;
    const bool last = OWN ? half != odd : half == 0;      // whether these warps have a last, the MOST-th, chunk
    const uint32_t box = ring + STAGES * STAGE + (warp - 2) * BOX;
    int t = 0;
    for (int blk = blockIdx.y; blk * BM < M; blk += gridDim.y, ++t) {
      const int m0 = blk * BM + quarter * 32;
      mbar_wait(accfull, t & 1, g.status, 560, alive, g.wait_limit);
      tc_fence_after();
      const uint32_t acc = tmem + ((uint32_t)(quarter * 32) << 16);
      float v[MOST][16];
#pragma unroll
      for (int ch = 0; ch < MOST; ++ch)
        if (ch < MOST - 1 || last) tmem_ld16_sum(acc + (ch < 6 ? c0 + ch : single) * 16, SMALL, v[ch]);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(accfree);      // (the next block's products may start before this one is stored)
      // 32 columns at a time through shared memory (16-byte pieces of a row exchanged by its number's low bits: no bank
      // conflicts either way), out in whole lines of a row
#pragma unroll
      for (int b = 0; b < (MOST + 1) / 2; ++b) {
        if (b == 3 && !last) break;
        const int at = b < 3 ? (c0 + 2 * b) * 16 : single * 16;      // first column of the box in the tile
        const bool whole = OWN || b < 2 ? b < 3 : last;
#pragma unroll
        for (int p = 0; p < 8; ++p) {
          const int ch = 2 * b + (p >> 2), c = 4 * (p & 3);
          if (ch >= MOST || (!OWN && ch == MOST - 1 && !last)) continue;
          const float4 y = *reinterpret_cast<const float4 *>(s_bias + at + 16 * (p >> 2) + c);
          st_shared_f4(box + lane * 128 + ((p ^ (lane & 7)) << 4),
                       make_float4(v[ch][c] + y.x, v[ch][c + 1] + y.y, v[ch][c + 2] + y.z, v[ch][c + 3] + y.w));
        }
        __syncwarp();
        const int p = whole ? lane & 7 : lane & 3, col = nt * BN + at + 4 * p;
        const bool query = !OWN || col < QT_LD;
        float *out = query ? g.qt + col : g.own + (col - QT_LD);
        const int ld = query ? QT_LD : OWN_LD;
        const bool on = query || (g.own != nullptr && col < QT_LD + OWN_LD);
#pragma unroll
        for (int i = 0; i < (b < 3 ? 8 : 4); ++i) {
          const int r = whole ? 4 * i + (lane >> 3) : 8 * i + (lane >> 2);
          if (on && (OWN || whole || i < 4) && m0 + r < M)
            *reinterpret_cast<float4 *>(out + (size_t)(m0 + r) * ld) = ld_shared_f4(box + r * 128 + ((p ^ (r & 7)) << 4));
        }
        __syncwarp();
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}

// rows -> operand image: a thread per 16-byte chunk (eight columns)
__global__ void __launch_bounds__(256) feat_image_kernel(tc::RowSrc feat, int n_cap, const int32_t *d_n, char *image) {
  dep_trigger();
  dep_wait();
  constexpr int CH = img::FEAT_STAGES * img::STAGE_K / 8;
  const int n = rows_of(n_cap, d_n);
  for (long long u = (long long)blockIdx.x * blockDim.x + threadIdx.x; u < (long long)n * CH; u += (long long)gridDim.x * blockDim.x) {
    const int m = (int)(u / CH), c = (int)(u - (long long)m * CH);
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
    if (c < CHUNKS) {
      const int r = feat.idx ? feat.idx[m] : m + feat.add;
      const float4 *p = reinterpret_cast<const float4 *>(feat.base(r) + (size_t)r * D) + 2 * c;
      x = *p;
      if (c < CHUNKS - 1) y = p[1];
    }
    uint4 hi, lo;
    tc::split_chunk(x, y, hi, lo);
    char *o = img::at<img::FEAT_STAGES>(image, m, 8 * c);
    *reinterpret_cast<uint4 *>(o) = hi;
    *reinterpret_cast<uint4 *>(o + img::STAGE_BYTES / 2) = lo;
  }
}

}  // namespace aqi

int feat_image(const tc::RowSrc &feat, int n_cap, const int32_t *d_n, char *d_image, cudaStream_t s) {
  if (n_cap <= 0) return ORCA_OK;
  Ctx *c = cur();
  const int sms = c != nullptr ? c->sm_count : 148;
  const long long units = (long long)n_cap * (img::FEAT_STAGES * 4);
  const int grid = (int)std::min<long long>((units + 255) / 256, sms * 8);
  ORCA_CUDA(launch_dep(aqi::feat_image_kernel, grid, 256, 0, s, feat, n_cap, d_n, d_image));
  ORCA_COUNT_LAUNCH();
  ORCA_LAUNCH_CHECK();
  return ORCA_OK;
}

int attn_query_image(const orca_attn_weights_t *w, const char *d_image, int n_cap, const int32_t *d_n, float *d_qt,
                     float *d_own, cudaStream_t s) {
  if (n_cap <= 0) return ORCA_OK;
  Ctx *c = cur();
  if (c == nullptr) return set_error(ORCA_E_CUDA, "attn_query_image: no context for the current device");
  ORCA_CHECK_ARG(w && w->Mq_img && w->cq && d_image && d_qt && (((uintptr_t)d_qt | (uintptr_t)d_own) & 15) == 0);
  static thread_local int configured_device = -1;
  if (configured_device != c->device) {
    ORCA_CUDA(cudaFuncSetAttribute(aqi::attn_query_image_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, aqi::Tile<false>::SMEM));
    ORCA_CUDA(cudaFuncSetAttribute(aqi::attn_query_image_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, aqi::Tile<true>::SMEM));
    configured_device = c->device;
  }
  const aqi::Args g{d_image, n_cap, d_n, w->Mq_img, w->cq, d_qt, d_own, c->status_word, c->wait_limit};
  const dim3 grid(aqi::TILES, std::min(ceil_div(n_cap, aqi::BM), std::max(1, c->sm_count / aqi::TILES)));
  if (d_own != nullptr) ORCA_CUDA(launch_dep(aqi::attn_query_image_kernel<true>, grid, aqi::THREADS, aqi::Tile<true>::SMEM, s, g));
  else ORCA_CUDA(launch_dep(aqi::attn_query_image_kernel<false>, grid, aqi::THREADS, aqi::Tile<false>::SMEM, s, g));
  ORCA_COUNT_LAUNCH();
  ORCA_LAUNCH_CHECK();
  return ORCA_OK;
}

}  // namespace orca
