// Output side of an attention layer on the tensor cores:
//   out[r] = LayerNorm(relu(ctx . G[:1032] + own + b1 + valid * g) . W2t + b2), optional history push and peer delivery
// where own = feat . G[1032:] comes from the kernel that computes the queries from the same features (attn_query.cu): of rows
// that share their features (a group's layer 1) it is computed once, and a block's chain here is six stages shorter.
// The rows come as an operand image (attn_out.cuh): bf16 heads and tails, split once by the kernels that computed them,
// in the form the tensor core reads.  So the main loop is nothing but bulk copies and MMAs: one thread streams stages
// of 32 K columns (16 KB of rows + 22 KB of weights) through a ring of three (of five for the first product of a CTA's
// first block, while the room of the hidden tile is still unused: a launch of few blocks waits for these loads), one
// thread multiplies, eight warps do the two epilogues -- of one row block while the stages of the next are already
// landing.  A block of 128 rows takes 33 + 6 stages of 6 MMAs and 1.4 MB.  The general projection kernel, whose producer
// warps load fp32 rows, convert and store them stage by stage, takes 49 us per block whatever the number of blocks.
// 66 k rows, 104 us: the first block's stages come at the pace of their MMAs (0.32 us), which read their operands from
// shared memory, later ones at 0.6 us, since all SMs read their rows from DRAM at once (rows from L2: 12 % less; without
// the weights' copies: the same).  A block is 20 us of that, 1 for the hidden tile, 2 for the second product, 0.5 for the
// accumulators' way out; LayerNorm and stores run beside the next block's stages.
// Measured instead: five slots with a LayerNorm in registers, 98 us alone, but streams 3 to 4 % slower and a single call's
// launch 5 us longer (an unrolled epilogue runs once, from a cold instruction cache); pairs of CTAs with half of the weights
// each (cta_group::2), which wait for two free SMs side by side: 50 batches of 2000 1.2 % faster, single calls of 3000 and
// 4000 edges with 20 neighbours 13 and 8 % slower; a row block on a cluster of two or four CTAs that share the columns:
// one block 27 -> 33 us, 36 blocks 29 -> 34 and 58 (a block waits for its chain of dependent stages, not for their width).
// Between the two products the hidden tile stays on the SM (bias + ReLU, split, A image of the second product), and
// the second product's accumulators reuse the first one's columns.
// Warp 0: copies.  Warp 1: tensor memory, MMA issue.  Warps 2-9: epilogues (thread = row, then warp = row).
#include <algorithm>

#include "attn_out.cuh"
#include "context.cuh"
#include "tc_ptx.cuh"

namespace orca {
namespace ao {

constexpr int BM = img::ROWS, BN = 176;
constexpr int STAGES = 3;
constexpr int A_STAGE = img::STAGE_BYTES, W_LBO = BN * 16, W_STAGE = 2 * 4 * W_LBO, STAGE = A_STAGE + W_STAGE;
constexpr int K_STAGES = img::CTX_STAGES;                                        // 33
constexpr int K2_CHUNKS = BN / 8, K2_STAGES = (K2_CHUNKS + 3) / 4;               // 22, 6
constexpr int A2_LBO = BM * 16 + 16, A2_BYTES = K2_CHUNKS * A2_LBO;
constexpr int TILE_LD = 180;                       // floats per row of the output tile (conflict-free 16-byte stores)
constexpr int FRONT = 90 * 1024;                   // hidden image, then output tile
static_assert(2 * A2_BYTES <= FRONT && BM * TILE_LD * 4 <= FRONT && STAGE % 1024 == 0, "");
constexpr int FIRST = 5;                           // stages of the first product of a CTA's first block
static_assert((FIRST - STAGES) * STAGE <= FRONT && K_STAGES % FIRST >= STAGES, "");
constexpr int FIRST_USES = K_STAGES / FIRST + 1;   // of each of the first STAGES slots
constexpr int SMEM = FRONT + STAGES * STAGE + 1024;
constexpr int EPI_WARPS = 8, THREADS = 64 + 32 * EPI_WARPS;
constexpr int TMEM_COLS = 512, SMALL = 256;

using img::desc_sw64;

// PAIRS: the top layer, whose rows go where the pairs that are scored want them (and to g.out, if given)
template <bool PAIRS>
__global__ void __launch_bounds__(THREADS, 1) attn_output_image_kernel(const __grid_constant__ OutArgs g) {
  using namespace tc;
  extern __shared__ unsigned char raw[];
  __shared__ __align__(16) float s_b1[BN], s_g[BN], s_b2[BN], s_lw[BN], s_lb[BN];
  __shared__ __align__(8) unsigned long long s_bar[2 * FIRST + 4];
  __shared__ float2 s_sum[2][BM];                  // of a row's two halves: sum and sum of squares
  __shared__ uint32_t s_tmem;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const uint32_t base = (smem_addr(raw) + 1023u) & ~1023u, ring = base + FRONT;
  auto full = [&](int s) { return smem_addr(&s_bar[s]); };
  auto empty = [&](int s) { return smem_addr(&s_bar[FIRST + s]); };
  const uint32_t acc1 = smem_addr(&s_bar[2 * FIRST]), a2bar = smem_addr(&s_bar[2 * FIRST + 1]),
                 acc2 = smem_addr(&s_bar[2 * FIRST + 2]), tfree = smem_addr(&s_bar[2 * FIRST + 3]);
  // stage number `it` of this CTA: its slot, how often the slot was used before, and where it lies
  auto slot_of = [&](int it) { return it < K_STAGES ? it % FIRST : (it - K_STAGES) % STAGES; };
  auto use_of = [&](int it) { return it < K_STAGES ? it / FIRST : FIRST_USES + (it - K_STAGES) / STAGES; };
  auto place = [&](int s) { return s < STAGES ? ring + s * STAGE : base + (s - STAGES) * STAGE; };
  dep_trigger();
  if (tid == 0) {
    for (int s = 0; s < FIRST; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), 1);
    }
    mbar_init(acc1, 1);
    mbar_init(a2bar, EPI_WARPS);
    mbar_init(acc2, 1);
    mbar_init(tfree, EPI_WARPS);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&s_tmem)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  for (int i = tid; i < BN; i += THREADS) {
    const bool in = i < D;
    s_b1[i] = in ? g.w.b1[i] : 0.f;
    s_g[i] = in ? g.w.g[i] : 0.f;
    s_b2[i] = in ? g.w.b2[i] : 0.f;
    s_lw[i] = in ? g.w.ln_w[i] : 0.f;
    s_lb[i] = in ? g.w.ln_b[i] : 0.f;
  }
  dep_wait();
  const int M = rows_of(g.n_cap, g.d_n);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *(volatile uint32_t *)&s_tmem, 0);
  bool alive = true;

  if (warp == 0) {
    // ------------------------------------------------------------------ stages
    if (lane == 0) {
      const char *w1 = reinterpret_cast<const char *>(g.w.G_img), *w2 = reinterpret_cast<const char *>(g.w.W2_img);
      const uint64_t once = policy_evict_first();      // (the rows are not read again: 1 % of a stream)
      int it = 0;
      for (int blk = blockIdx.x; alive && blk * BM < M; blk += gridDim.x) {
        const char *ctx = g.ctx + (size_t)blk * img::CTX_STAGES * A_STAGE;
        for (int st = 0; st < K_STAGES + K2_STAGES; ++st, ++it) {
          const int s = slot_of(it);
          const uint32_t at = place(s);
          mbar_wait(empty(s), (use_of(it) & 1) ^ 1, g.status, 700, alive, g.wait_limit);
          if (!alive) break;
          if (st < K_STAGES) {
            mbar_expect_tx(full(s), STAGE);
            bulk_g2s_hint(at, ctx + (size_t)st * A_STAGE, A_STAGE, full(s), once);
            bulk_g2s(at + A_STAGE, w1 + (size_t)st * W_STAGE, W_STAGE, full(s));
          } else {
            mbar_expect_tx(full(s), W_STAGE);
            bulk_g2s(at + A_STAGE, w2 + (size_t)(st - K_STAGES) * W_STAGE, W_STAGE, full(s));
          }
        }
      }
      for (int q = it - 1, seen = 0; q >= max(0, it - FIRST); --q) {      // (the last use of every slot)
        const int s = slot_of(q);
        if (!(seen >> s & 1)) mbar_settle(full(s), use_of(q) & 1);
        seen |= 1 << s;
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issue
    constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
    int it = 0, t = 0;
    for (int blk = blockIdx.x; blk * BM < M; blk += gridDim.x, ++t) {
      if (t > 0) mbar_wait(tfree, (t - 1) & 1, g.status, 710, alive, g.wait_limit);
      tc_fence_after();
      for (int st = 0; st < K_STAGES; ++st, ++it) {
        const int s = slot_of(it);
        const uint32_t a = place(s), w = a + A_STAGE;
        const bool half = st == K_STAGES - 1;     // (the second step is nothing but padding)
        mbar_wait(full(s), use_of(it) & 1, g.status, 711, alive, g.wait_limit);
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < 2; ++ks) {
            if (!alive || (ks == 1 && half)) break;
            const uint64_t ah = desc_sw64(a + ks * 32), al = desc_sw64(a + A_STAGE / 2 + ks * 32);
            const uint64_t bh = make_desc(w + ks * 2 * W_LBO, W_LBO, 128), bl = make_desc(w + W_STAGE / 2 + ks * 2 * W_LBO, W_LBO, 128);
            const uint32_t more = (st > 0 || ks > 0) ? 1u : 0u;
            mma_bf16(tmem, ah, bh, idesc, more);
            mma_bf16(tmem + SMALL, al, bh, idesc, more);
            mma_bf16(tmem + SMALL, ah, bl, idesc, 1u);
          }
          if (alive) mma_commit(empty(s));
          if (st == K_STAGES - 1) mma_commit(acc1);
        }
        __syncwarp();
      }
      mbar_wait(a2bar, t & 1, g.status, 712, alive, g.wait_limit);
      tc_fence_after();
      for (int st = 0; st < K2_STAGES; ++st, ++it) {
        const int s = slot_of(it);
        const uint32_t w = place(s) + A_STAGE, a = base + st * 4 * A2_LBO;
        mbar_wait(full(s), use_of(it) & 1, g.status, 713, alive, g.wait_limit);
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < 2; ++ks) {
            if (!alive || 2 * st + ks >= K2_CHUNKS / 2) break;
            const uint64_t ah = make_desc(a + ks * 2 * A2_LBO, A2_LBO, 128);
            const uint64_t al = make_desc(a + A2_BYTES + ks * 2 * A2_LBO, A2_LBO, 128);
            const uint64_t bh = make_desc(w + ks * 2 * W_LBO, W_LBO, 128), bl = make_desc(w + W_STAGE / 2 + ks * 2 * W_LBO, W_LBO, 128);
            const uint32_t more = (st > 0 || ks > 0) ? 1u : 0u;
            mma_bf16(tmem, ah, bh, idesc, more);
            mma_bf16(tmem + SMALL, al, bh, idesc, more);
            mma_bf16(tmem + SMALL, ah, bl, idesc, 1u);
          }
          if (alive) mma_commit(empty(s));
          if (st == K2_STAGES - 1) mma_commit(acc2);
        }
        __syncwarp();
      }
    }
    if (t > 0) mbar_settle(acc2, (t - 1) & 1);
  } else {
    // ------------------------------------------------------------------ epilogues
    const int ew = warp - 2, quarter = warp & 3, half = ew >> 2;
    const int row = quarter * 32 + lane;
    const uint32_t trow = tmem + ((uint32_t)(quarter * 32) << 16);
    const int ch0 = half ? 6 : 0, ch1 = half ? BN / 16 : 6;     // accumulator chunks of 16 columns of this warp
    const bool has1 = lane + 32 < D / 4;
    const float4 f4z = make_float4(0.f, 0.f, 0.f, 0.f);
    auto vec = [&](const float *s, int j, bool on) { return on ? *reinterpret_cast<const float4 *>(s + 4 * j) : f4z; };
    int t = 0;
    for (int blk = blockIdx.x; blk * BM < M; blk += gridDim.x, ++t) {
      const int m0 = blk * BM, m_rows = min(BM, M - m0);
      const float on = (row < m_rows && (g.valid == nullptr || g.valid[m0 + row] != 0)) ? 1.f : 0.f;
      // lane i holds what row ew + 8 * i of the output pass needs: history push; or the row's (first) pair, and how much
      // further its second one is (0: it is a destination or negative, the second of one pair)
      int push_id = 0, push = 0;
      if (PAIRS) {
        const int m = m0 + ew + EPI_WARPS * (lane & 15), n = m / (3 * g.pair_bs), i = m - n * 3 * g.pair_bs;
        const int b = n == g.pair_nb - 1 ? g.pair_last : g.pair_bs;
        push_id = n * 2 * g.pair_bs + (i < b ? i : i - b), push = i < b ? b : 0;
      } else if (g.push_table != nullptr && lane < BM / EPI_WARPS && ew + EPI_WARPS * lane < m_rows) {
        const int m = m0 + ew + EPI_WARPS * lane;
        push_id = g.push_ids[m];
        push = g.push_win != nullptr ? g.push_win[m]
               : (m >= g.push_all_from || g.push_last_pos[push_id] == (unsigned long long)(g.push_base + m)) ? 1 : 0;
      }
      // what the row's own features add: asked for while the product is still running
      float4 own[6][4];
      {
        const int m = m0 + min(row, m_rows - 1);
        const float4 *src = reinterpret_cast<const float4 *>(g.own + (size_t)(g.own_row != nullptr ? g.own_row[m] : m) * OWN_LD) + 4 * ch0;
#pragma unroll
        for (int ch = 0; ch < 6; ++ch)
#pragma unroll
          for (int q = 0; q < 4; ++q) own[ch][q] = ch < ch1 - ch0 ? __ldg(src + 4 * ch + q) : f4z;
      }
      // first: hidden = relu(acc + own + b1 + valid * g), split, A image of the second product
      mbar_wait(acc1, t & 1, g.status, 720, alive, g.wait_limit);
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        const int ch = ch0 + c;
        if (ch >= ch1) break;
        float v[16];
        tmem_ld16_sum(trow + ch * 16, SMALL, v);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          v[4 * q] += own[c][q].x, v[4 * q + 1] += own[c][q].y;
          v[4 * q + 2] += own[c][q].z, v[4 * q + 3] += own[c][q].w;
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = relu(v[i] + s_b1[ch * 16 + i] + on * s_g[ch * 16 + i]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint4 hi, lo;
          split_chunk(make_float4(v[8 * h], v[8 * h + 1], v[8 * h + 2], v[8 * h + 3]),
                      make_float4(v[8 * h + 4], v[8 * h + 5], v[8 * h + 6], v[8 * h + 7]), hi, lo);
          st_shared_v4(base + (uint32_t)(2 * ch + h) * A2_LBO + row * 16, hi);
          st_shared_v4(base + A2_BYTES + (uint32_t)(2 * ch + h) * A2_LBO + row * 16, lo);
        }
      }
      fence_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(a2bar);
      // second: accumulators -> row-major tile (over the hidden image, which has been read) with the bias added; this thread's
      // half of its row gives both moments in one sweep (the row is O(1) after the merger, so E[y^2] - mean^2 loses nothing
      // that matters at the 1e-5 epsilon; columns from 172 on are zero, bias included)
      mbar_wait(acc2, t & 1, g.status, 721, alive, g.wait_limit);
      tc_fence_after();
      float sum = 0.f, sq = 0.f;
#pragma unroll 1
      for (int ch = ch0; ch < ch1; ++ch) {
        float v[16];
        tmem_ld16_sum(trow + ch * 16, SMALL, v);
        float4 a = f4z, b = f4z;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float4 y = *reinterpret_cast<const float4 *>(s_b2 + ch * 16 + q * 4);
          const float4 z = make_float4(v[q * 4] + y.x, v[q * 4 + 1] + y.y, v[q * 4 + 2] + y.z, v[q * 4 + 3] + y.w);
          a.x += z.x, a.y += z.y, a.z += z.z, a.w += z.w;
          b.x += z.x * z.x, b.y += z.y * z.y, b.z += z.z * z.z, b.w += z.w * z.w;
          st_shared_f4(base + (uint32_t)(row * TILE_LD + ch * 16 + q * 4) * 4u, z);
        }
        sum += (a.x + a.y) + (a.z + a.w);
        sq += (b.x + b.y) + (b.z + b.w);
      }
      tc_fence_before();
      s_sum[half][row] = make_float2(sum, sq);
      __syncwarp();
      if (lane == 0) mbar_arrive(tfree);
      asm volatile("bar.sync 1, 256;" ::: "memory");
      // then whole rows, a warp each
      const float4 wA = vec(s_lw, lane, true), wB = vec(s_lw, lane + 32, has1);
      const float4 lA = vec(s_lb, lane, true), lB = vec(s_lb, lane + 32, has1);
      constexpr int RB = 4;     // rows in flight per warp
#pragma unroll 1
      for (int i0 = 0; i0 < BM / EPI_WARPS; i0 += RB) {
        if (ew + EPI_WARPS * i0 >= m_rows) break;
        float4 a[RB], b[RB];
        float mean[RB], inv[RB];
#pragma unroll
        for (int k = 0; k < RB; ++k) {
          const int r = ew + EPI_WARPS * (i0 + k);
          const uint32_t ra = base + (uint32_t)(r * TILE_LD + 4 * lane) * 4u;
          a[k] = ld_shared_f4(ra);
          b[k] = has1 ? ld_shared_f4(ra + 512u) : f4z;
          const float2 x = s_sum[0][r], y = s_sum[1][r];
          const float total = x.x + y.x;
          mean[k] = total * (1.f / D);
          inv[k] = 1.f / sqrtf(fmaxf(x.y + y.y - total * mean[k], 0.f) * (1.f / D) + 1e-5f);
        }
#pragma unroll
        for (int k = 0; k < RB; ++k) {
          const int r = ew + EPI_WARPS * (i0 + k);
          const int to = __shfl_sync(0xffffffffu, push_id, i0 + k), win = __shfl_sync(0xffffffffu, push, i0 + k);
          if (r >= m_rows) continue;
          const float4 ya = make_float4((a[k].x - mean[k]) * inv[k] * wA.x + lA.x, (a[k].y - mean[k]) * inv[k] * wA.y + lA.y,
                                        (a[k].z - mean[k]) * inv[k] * wA.z + lA.z, (a[k].w - mean[k]) * inv[k] * wA.w + lA.w);
          const float4 yb = make_float4((b[k].x - mean[k]) * inv[k] * wB.x + lB.x, (b[k].y - mean[k]) * inv[k] * wB.y + lB.y,
                                        (b[k].z - mean[k]) * inv[k] * wB.z + lB.z, (b[k].w - mean[k]) * inv[k] * wB.w + lB.w);
          auto store = [&](float *o) {
            *reinterpret_cast<float4 *>(o + 4 * lane) = ya;
            if (has1) *reinterpret_cast<float4 *>(o + 4 * lane + 128) = yb;
          };
          // heads and tails of the lane's columns; behind the row, the padding
          uint2 hiA, loA, hiB, loB;
          auto pack = [](float4 x, uint2 &hi, uint2 &lo) {
            hi.x = pack_split(x.x, x.y, lo.x);
            hi.y = pack_split(x.z, x.w, lo.y);
          };
          // (img::at, with the row's part taken out)
          auto put = [&](char *row, int sw, int c, bool second) {
            auto at = [&](int x) { return row + (((x >> 5) * A_STAGE + (x >> 3 & 3) * 16 + 2 * (x & 7)) ^ sw); };
            char *p = at(c), *q = at(c + 128);
            *reinterpret_cast<uint2 *>(p) = hiA;
            *reinterpret_cast<uint2 *>(p + A_STAGE / 2) = loA;
            if (second) {
              *reinterpret_cast<uint2 *>(q) = hiB;
              *reinterpret_cast<uint2 *>(q + A_STAGE / 2) = loB;
            }
          };
          if (PAIRS || m0 + r < g.out_image_rows) pack(ya, hiA, loA), pack(has1 ? yb : f4z, hiB, loB);
          if (PAIRS) {
            if (g.out != nullptr) store(g.out + (size_t)(m0 + r) * D);
            const int second = win == 0;
            auto to_pair = [&](int pair) {
              put(g.pair_image + (size_t)(pair / img::ROWS) * (img::PAIR_STAGES * A_STAGE) + (pair % img::ROWS) * 64, (pair << 3) & 0x30,
                  4 * lane + second * D, lane < D / 4 - 32 + 2 * second);
            };
            to_pair(to);
            if (!second) to_pair(to + win);
            continue;
          }
          store(g.out + (size_t)(m0 + r) * D);
          if (g.push_table != nullptr && win != 0) store(g.push_table + (size_t)to * D);
          if (m0 + r < g.out_image_rows)     // (columns 172 .. 191 are padding)
            put(g.out_image + (size_t)blk * (img::FEAT_STAGES * A_STAGE) + r * 64, (r << 3) & 0x30, 4 * lane, lane < 16);
          // multi-GPU exchange: the row also goes to every rank's exchange buffer (peer stores)
          for (int q = 0; q < g.peer.world; ++q) store(g.peer.rows[q] + g.peer.off + (size_t)(m0 + r) * D);
        }
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");     // the tile has been read: the next hidden image may land
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
  if (!PAIRS && g.peer.world > 0) {
    // every CTA (with or without rows) checks out; the last one posts the batch's sequence number to all ranks, after
    // every CTA's peer stores have been fenced system-wide
    __threadfence_system();
    __syncthreads();
    if (tid == 0 && atomicAdd(g.peer.counter, 1) == (int)gridDim.x - 1) {
      *g.peer.counter = 0;
      __threadfence_system();
      for (int q = 0; q < g.peer.world; ++q)
        asm volatile("st.release.sys.global.s32 [%0], %1;" ::"l"(g.peer.flags[q] + g.peer.rank), "r"(g.peer.seq)
                     : "memory");
    }
  }
}

}  // namespace ao

int attn_output_rows(const OutArgs &args, cudaStream_t s) {
  if (args.n_cap <= 0) return ORCA_OK;
  Ctx *c = cur();
  if (c == nullptr) return set_error(ORCA_E_CUDA, "attn_output_rows: no context for the current device");
  ORCA_CHECK_ARG(args.w.G_img && args.w.W2_img && args.ctx && args.own && (args.out || args.pair_image));
  // (the top layer of one GPU: no push, no image of its own, no delivery)
  ORCA_CHECK_ARG(args.pair_image == nullptr || (args.push_table == nullptr && args.out_image_rows == 0 && args.peer.world == 0));
  ORCA_CHECK_ARG(args.pair_image == nullptr || (args.pair_bs > 0 && args.pair_nb > 0 && args.pair_last > 0 && args.pair_last <= args.pair_bs));
  static thread_local int configured_device = -1;
  if (configured_device != c->device) {
    ORCA_CUDA(cudaFuncSetAttribute(ao::attn_output_image_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, ao::SMEM));
    ORCA_CUDA(cudaFuncSetAttribute(ao::attn_output_image_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, ao::SMEM));
    configured_device = c->device;
  }
  OutArgs g = args;
  g.status = c->status_word;
  g.wait_limit = c->wait_limit;
  const int grid = std::min(ceil_div(g.n_cap, ao::BM), c->sm_count);
  ORCA_CUDA(launch_dep(g.pair_image != nullptr ? ao::attn_output_image_kernel<true> : ao::attn_output_image_kernel<false>, grid,
                       ao::THREADS, ao::SMEM, s, g));
  ORCA_COUNT_LAUNCH();
  ORCA_LAUNCH_CHECK();
  return ORCA_OK;
}

}  // namespace orca
