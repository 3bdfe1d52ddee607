// The memory updates of a group of batches in one launch: raw message + GRU of batch 0, 1, ..., each reading the memory
// rows that the batches before it wrote.
//
// As launches of the general projection kernel this chain costs 43 us a batch (message rows written and read back,
// a pipeline filled and drained, two launches) whatever the batch size, and it is the only part of a group that is
// serial: with small batches it is what a stream waits for.  What a batch really waits for is its memory rows.  So
// one cooperative grid walks the batches:
//   - 22 column tiles of 32 gate columns (eight units) times row blocks of 64 updates, one CTA each, up to five (launch).
//     A CTA keeps its weight columns (880 x 32, bf16 head and tail, 113 KB) in shared memory for the whole launch.
//   - K is laid out so that what does not depend on the batch before comes first: edge features and time encoding
//     (352 columns).  A launch of its own splits them for all updates of the group (computed in the chain, the cosines
//     alone were half of a turn), and they are multiplied for batch n + 1 while batch n is still being finished.
//   - Then the grid meets at a counter, and only the node's own and the other endpoint's memory rows (2 x 688 bytes
//     an update) are gathered, split and multiplied; the GRU's hidden operand is the own row's image again.
//   - The result goes to the log row of the update; message table, times and flags follow in one launch at the end.
// MMAs of 64 rows: an MMA of 32 columns is bound by its reads of the row operand.  Row r of the tile sits in tensor
// memory lane 32 * (r / 16) + r % 16.
// A step's products are the ones of the projection kernel, k-step by k-step, so the results are the same bits.
// Warps 0-3: epilogue (16 rows each, a lane for four of a row's units).  Warps 4-11: gather and split.  Warp 12: MMA
// issue, tensor memory.
// Every wait is bounded; one that gives up reports ORCA_E_TIMEOUT and the kernel runs to its end.
#include "chain.cuh"
#include "context.cuh"
#include "gru_rows.cuh"
#include "tc_gemm.cuh"
#include "tc_ptx.cuh"

namespace orca {
namespace grp {

constexpr int ROWS = 64;                       // updates per row block
constexpr int COLS = 32, UNITS = COLS / 4;     // gate columns / units per CTA
constexpr int COL_TILES = (4 * D + COLS - 1) / COLS;   // 22
constexpr int PART_CHUNKS = tc::GRU_PART / 8;  // 22 chunks of 8 K elements per part
constexpr int PART_STEPS = tc::GRU_PART / 16;  // 11 MMA steps per part
constexpr int W_LBO = COLS * 16, W_BYTES = 5 * PART_CHUNKS * W_LBO;
// two parts of K at a time: first edge features and time encoding, then, once those have been read, the memory rows
constexpr int A_CHUNKS = 2 * PART_CHUNKS, A_LBO = ROWS * 16 + 16, A_BYTES = A_CHUNKS * A_LBO;   // (+16: conflict-free stores)
constexpr int SMEM = 2 * W_BYTES + 2 * A_BYTES + 1024;
constexpr int EPI_WARPS = 4, PRODUCERS = 256, THREADS = 32 * EPI_WARPS + PRODUCERS + 32;
constexpr int TMEM_COLS = 128, BUF_COLS = 64, SMALL = 32;   // two accumulator buffers of main + cross terms
// Updates that a row block takes before there is another one, in groups whose last updates leave the chain.  A CTA holds an SM
// beside layers that want every one, and 64 rows take hardly longer than 32.  32 / 64, us a stream: 48 batches of 1000
// 2527 / 2473, 50 of 2000 and 51 of 600 within 1 %; 30 of 400 970 / 978, 30 of 600 1213 / 1233; 20 to 2000 edges a batch, one and two
// layers, 10 and 20 neighbours otherwise within 1 %.  (96 and 128 cost batches of 600 and 2000 2 and 3 %.)
constexpr int BLOCK_ROWS = 64;
constexpr int META = 4;                        // steps whose memory rows are kept
constexpr int PER = 6;                         // chunks a producer thread has in flight: 34 rows at a time

// Edge features and time encoding of every update, split: 44 chunks of [heads 16 bytes | tails 16 bytes].  The memory
// rows that the chain will read from the table start on their way into L2.
__global__ void __launch_bounds__(256) update_image_kernel(const __grid_constant__ ChainArgs g) {
  const Args &a = g.a;
  dep_trigger();
  dep_wait();
  const int lane = threadIdx.x & 31;
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < a.nb * 2 * a.bs; i += (gridDim.x * blockDim.x) >> 5) {
    const int n = i / (2 * a.bs), w = i - n * 2 * a.bs;
    if (w >= a.cnt->n_win[n]) continue;
    const float gap = a.win_gap[i];
    if (lane < 12) {
      const int r = lane < 6 ? a.win_mem[i] : a.win_other[i];
      if (r < a.n_nodes)
        asm volatile("prefetch.global.L2 [%0];" ::"l"((const char *)(g.mem.memory + (size_t)r * D) + min((lane % 6) * 128, ROW_BYTES - 4)));
    }
    const float4 *e = reinterpret_cast<const float4 *>(g.edge_table + (size_t)a.win_eid[i] * D);
    for (int c = lane; c < A_CHUNKS; c += 32) {
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
      if (c < PART_CHUNKS) {
        x = __ldg(e + 2 * c);
        if (c < PART_CHUNKS - 1) y = __ldg(e + 2 * c + 1);
      } else {
        const int d = (c - PART_CHUNKS) * 8;
        const float4 w0 = __ldg(reinterpret_cast<const float4 *>(g.time_w + d));
        x = make_float4(cos_any(gap * w0.x), cos_any(gap * w0.y), cos_any(gap * w0.z), cos_any(gap * w0.w));
        if (d + 4 < D) {
          const float4 w1 = __ldg(reinterpret_cast<const float4 *>(g.time_w + d + 4));
          y = make_float4(cos_any(gap * w1.x), cos_any(gap * w1.y), cos_any(gap * w1.z), cos_any(gap * w1.w));
        }
      }
      uint4 hi, lo;
      tc::split_chunk(x, y, hi, lo);
      uint4 *o = reinterpret_cast<uint4 *>(g.image) + ((size_t)i * A_CHUNKS + c) * 2;
      o[0] = hi;
      o[1] = lo;
    }
  }
}

__global__ void __launch_bounds__(THREADS, 1) gru_chain_kernel(const __grid_constant__ ChainArgs g) {
  using namespace tc;
  extern __shared__ unsigned char raw[];
  __shared__ int s_win[MAX_BATCHES];
  __shared__ int s_self[META][ROWS], s_other[META][ROWS];
  __shared__ __align__(16) float s_bias[COLS];
  __shared__ __align__(8) unsigned long long s_bar[8];
  __shared__ uint32_t s_tmem;
  const Args &a = g.a;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int ct = blockIdx.x, rb = blockIdx.y;
  const uint32_t base = (smem_addr(raw) + 1023u) & ~1023u;
  const uint32_t w_hi = base, w_lo = base + W_BYTES, a_hi = base + 2 * W_BYTES, a_lo = a_hi + A_BYTES;
  const uint32_t wbar = smem_addr(&s_bar[0]), ebar = smem_addr(&s_bar[1]), mbar = smem_addr(&s_bar[2]),
                 edone = smem_addr(&s_bar[3]), accbar = smem_addr(&s_bar[4]);
  auto tfree = [&](int b) { return smem_addr(&s_bar[5 + b]); };
  if (tid == 0) {
    mbar_init(wbar, 1);
    mbar_init(ebar, PRODUCERS / 32);
    mbar_init(mbar, PRODUCERS / 32);
    mbar_init(edone, 1);
    mbar_init(accbar, 1);
    mbar_init(tfree(0), EPI_WARPS);
    mbar_init(tfree(1), EPI_WARPS);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_expect_tx(wbar, 2 * W_BYTES);
    bulk_g2s(w_hi, reinterpret_cast<const char *>(g.w) + (size_t)ct * 2 * W_BYTES, 2 * W_BYTES, wbar);
  }
  if (warp == 12) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&s_tmem)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid < MAX_BATCHES) s_win[tid] = tid < a.nb ? a.cnt->n_win[tid] : 0;
  if (tid >= 32 && tid < 64) s_bias[tid - 32] = ct * COLS + tid - 32 < 4 * D ? g.bias[ct * COLS + tid - 32] : 0.f;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *(volatile uint32_t *)&s_tmem, 0);
  bool alive = true;
  // row blocks of a group whose last updates are done elsewhere: as many as the batch with the most updates asks for; the
  // others have nothing to do
  int most = 0;
  for (int n = 0; n < a.nb; ++n) most = max(most, s_win[n]);
  const int n_rb = a.split ? max(1, min((int)gridDim.y, (most + BLOCK_ROWS - 1) / BLOCK_ROWS)) : (int)gridDim.y;
  const int n_cta = gridDim.x * n_rb, nb = rb < n_rb ? a.nb : 0;
  // rows of a row block in a batch: the updates spread over the blocks, in steps of eight, at most a tile's
  auto rows_per = [&](int win) { return min(ROWS, ((win + n_rb - 1) / n_rb + 7) & ~7); };
  auto mem_row = [&](int r) { return (r >= a.n_nodes ? g.log : g.mem.memory) + (size_t)r * D; };

  int s = 0;    // steps of this CTA so far: the rows of one turn of one batch each
  if (warp < EPI_WARPS) {
    // ------------------------------------------------------------------ gates
    const int row = warp * 16 + (lane & 15), hi = lane >> 4;     // this lane: units 4 * hi .. 4 * hi + 3 of the row
    const int u0 = ct * UNITS + 4 * hi;
    for (int n = 0; n < nb; ++n) {
      const int rows = rows_per(s_win[n]);
      for (int r0 = rb * rows; r0 < s_win[n]; r0 += n_rb * rows, ++s) {
        const bool live = row < rows && r0 + row < s_win[n] && u0 < D;      // (the last tile has four units)
        mbar_wait(mbar, s & 1, g.status, 610, alive, g.wait_limit);         // (the batches before are complete then)
        float4 h = make_float4(0.f, 0.f, 0.f, 0.f);
        if (live) h = __ldcg(reinterpret_cast<const float4 *>(mem_row(s_self[s & (META - 1)][row]) + u0));
        mbar_wait(accbar, s & 1, g.status, 611, alive, g.wait_limit);
        tc_fence_after();
        float x[16], y[16];
        const uint32_t t = tmem + ((uint32_t)(warp * 32) << 16) + (s & 1) * BUF_COLS;
        tmem_ld16_sum(t, SMALL, x);
        tmem_ld16_sum(t + 16, SMALL, y);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(tfree(s & 1));
        // (rows live in the lower 16 lanes: the upper ones take over the second half of their columns)
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float z = __shfl_sync(0xffffffffu, y[i], lane & 15);
          if (hi) x[i] = z;
        }
        const float *b = s_bias + 16 * hi;
        const float ho[4] = {h.x, h.y, h.z, h.w};
        float o[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          o[u] = gru_gates(make_float4(x[4 * u] + b[4 * u], x[4 * u + 1] + b[4 * u + 1], x[4 * u + 2] + b[4 * u + 2],
                                       x[4 * u + 3] + b[4 * u + 3]), ho[u]);
        if (live)
          *reinterpret_cast<float4 *>(g.log_out + (size_t)(n * 2 * a.bs + r0 + row) * D + u0) = make_float4(o[0], o[1], o[2], o[3]);
      }
      __syncwarp();      // (the release below covers the warp's stores)
      if (lane == 0) asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(&a.cnt->arrived[n]) : "memory");
    }
  } else if (warp < 12) {
    // ------------------------------------------------------------------ gather and split
    const int pt = tid - 32 * EPI_WARPS;
    auto put = [&](int chunk, int row, uint4 hi, uint4 lo) {
      st_shared_v4(a_hi + chunk * A_LBO + row * 16, hi);
      st_shared_v4(a_lo + chunk * A_LBO + row * 16, lo);
    };
    for (int n = 0; n < nb; ++n) {
      bool met = n == 0;
      const int full_rows = rows_per(s_win[n]);
      for (int r0 = rb * full_rows; r0 < s_win[n]; r0 += n_rb * full_rows, ++s) {
        const int q = s & (META - 1), rows = min(full_rows, s_win[n] - r0), n_units = rows * A_CHUNKS;
        const int at = n * 2 * a.bs + r0;
        if (pt < rows) {
          s_self[q][pt] = a.win_mem[at + pt];
          s_other[q][pt] = a.win_other[at + pt];
        }
        // edge features and time encoding
        const uint4 *im = reinterpret_cast<const uint4 *>(g.image) + (size_t)at * A_CHUNKS * 2;
        for (int u0 = pt; u0 - pt < n_units; u0 += PER * PRODUCERS) {
          uint4 e[PER][2];
#pragma unroll
          for (int i = 0; i < PER; ++i) {
            const int u = u0 + i * PRODUCERS;
            if (u < n_units) e[i][0] = __ldg(im + 2 * u), e[i][1] = __ldg(im + 2 * u + 1);
          }
          if (s > 0) mbar_wait(accbar, (s - 1) & 1, g.status, 620, alive, g.wait_limit);   // the image is free again
#pragma unroll
          for (int i = 0; i < PER; ++i) {
            const int u = u0 + i * PRODUCERS;
            if (u < n_units) put(u % A_CHUNKS, u / A_CHUNKS, e[i][0], e[i][1]);
          }
        }
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(ebar);
        if (!met) {
          // every CTA has written its part of the batch before (a CTA without rows in a batch arrives at once, which
          // is why every batch has a counter of its own)
          met = true;
          if (pt == 0 && alive) {
            const long long t0 = clock64();
            for (;;) {
              int v;
              asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(&a.cnt->arrived[n - 1]) : "memory");
              if (v >= n_cta * EPI_WARPS) break;
              if (clock64() - t0 > g.wait_limit) {
                report(g.status, ORCA_E_TIMEOUT, 621);
                alive = false;
                break;
              }
            }
          }
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");     // (and the memory rows' numbers are known)
        // own and other memory
        for (int u0 = pt; u0 - pt < n_units; u0 += PER * PRODUCERS) {
          float4 x[PER][2];
#pragma unroll
          for (int i = 0; i < PER; ++i) {
            const int u = u0 + i * PRODUCERS, row = u / A_CHUNKS, c = u - row * A_CHUNKS;
            x[i][0] = x[i][1] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (u < n_units) {
              const int cc = c < PART_CHUNKS ? c : c - PART_CHUNKS;
              const float4 *m = reinterpret_cast<const float4 *>(mem_row(c < PART_CHUNKS ? s_self[q][row] : s_other[q][row])) + 2 * cc;
              x[i][0] = __ldcg(m);
              if (cc < PART_CHUNKS - 1) x[i][1] = __ldcg(m + 1);
            }
          }
          mbar_wait(edone, s & 1, g.status, 622, alive, g.wait_limit);     // the first two parts have been read
#pragma unroll
          for (int i = 0; i < PER; ++i) {
            const int u = u0 + i * PRODUCERS, row = u / A_CHUNKS, c = u - row * A_CHUNKS;
            if (u < n_units) {
              uint4 hi, lo;
              split_chunk(x[i][0], x[i][1], hi, lo);
              put(c, row, hi, lo);
            }
          }
        }
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(mbar);
      }
    }
  } else {
    // ------------------------------------------------------------------ MMA issue
    constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(COLS >> 3) << 17) | ((uint32_t)(ROWS >> 4) << 24);
    mbar_wait(wbar, 0, g.status, 630, alive, g.wait_limit);
    for (int n = 0; n < nb; ++n) {
      const int rows = rows_per(s_win[n]);
      for (int r0 = rb * rows; r0 < s_win[n]; r0 += n_rb * rows, ++s) {
        const uint32_t d = tmem + (s & 1) * BUF_COLS;
        if (s >= 2) mbar_wait(tfree(s & 1), ((s >> 1) & 1) ^ 1, g.status, 631, alive, g.wait_limit);
        // parts of K: edge features, time encoding | own memory, other memory, own memory again
#pragma unroll
        for (int part = 0; part < 5; ++part) {
          if (part == 0) mbar_wait(ebar, s & 1, g.status, 632, alive, g.wait_limit);
          if (part == 2) mbar_wait(mbar, s & 1, g.status, 633, alive, g.wait_limit);
          if (part == 0 || part == 2) tc_fence_after();
          if (elect_one()) {
            const int ap = part == 4 ? 0 : part & 1;      // place of the part's rows in the image
#pragma unroll
            for (int ks = 0; ks < PART_STEPS; ++ks) {
              const uint32_t ao = (ap * PART_STEPS + ks) * 2 * A_LBO, wo = (part * PART_STEPS + ks) * 2 * W_LBO;
              const uint64_t ah = make_desc(a_hi + ao, A_LBO, 128), al = make_desc(a_lo + ao, A_LBO, 128);
              const uint64_t bh = make_desc(w_hi + wo, W_LBO, 128), bl = make_desc(w_lo + wo, W_LBO, 128);
              const uint32_t more = part > 0 || ks > 0 ? 1u : 0u;
              mma_bf16(d, ah, bh, idesc, more);
              mma_bf16(d + SMALL, al, bh, idesc, more);
              mma_bf16(d + SMALL, ah, bl, idesc, 1u);
            }
            if (part == 1) mma_commit(edone);
            if (part == 4) mma_commit(accbar);
          }
          __syncwarp();
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 12) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}

// Message table, times and flags of every node that the group updated, as its last update leaves them (the rows of
// batches in between are never looked at).  Runs behind the chain and before the memory table is written.
// An update: 172 pieces of 16 bytes (own memory, other memory, edge features, time encoding).  A group has thousands of them
// and gives each a warp (a block each waited for one chain of loads after the other: 24 -> 9 us for 6000); where all can have
// a block of four side by side, they do (5.0 us for 60, 5.4 with a warp each).
template <int WARPS>
__global__ void __launch_bounds__(256) last_messages_kernel(const __grid_constant__ ChainArgs g) {
  const Args &a = g.a;
  dep_trigger();
  dep_wait();
  constexpr int PIECES = MSG / 4, ROW_PIECES = D / 4;
  constexpr int LANES = 32 * WARPS;      // of an update
  const int lane = threadIdx.x % LANES, step = gridDim.x * (blockDim.x / LANES);
  const int n = a.cnt->n_last;
  for (int l = (blockIdx.x * blockDim.x + threadIdx.x) / LANES; l < n; l += step) {
    const int i = a.last_at[l];
    const int node = a.win_node[i], self = a.win_mem[i], other = a.win_other[i];
    const float t = a.win_t[i], gap = a.win_gap[i];
    const float4 *src[3] = {reinterpret_cast<const float4 *>((self >= a.n_nodes ? g.log : g.mem.memory) + (size_t)self * D),
                            reinterpret_cast<const float4 *>((other >= a.n_nodes ? g.log : g.mem.memory) + (size_t)other * D),
                            reinterpret_cast<const float4 *>(g.edge_table + (size_t)a.win_eid[i] * D)};
    constexpr int TURNS = (PIECES + LANES - 1) / LANES;
    float4 x[TURNS];
#pragma unroll
    for (int q = 0; q < TURNS; ++q) {
      const int at = lane + LANES * q, part = at / ROW_PIECES, c = at - part * ROW_PIECES;
      if (part < 3) x[q] = src[part][c];
      else if (at < PIECES) {
        const float4 w = __ldg(reinterpret_cast<const float4 *>(g.time_w) + c);
        x[q] = make_float4(cos_any(gap * w.x), cos_any(gap * w.y), cos_any(gap * w.z), cos_any(gap * w.w));
      }
    }
    float4 *dst = reinterpret_cast<float4 *>(g.mem.messages + (size_t)node * MSG);
#pragma unroll
    for (int q = 0; q < TURNS; ++q) {
      const int at = lane + LANES * q;
      if (at < PIECES) dst[at] = x[q];
      if (WARPS == 1 && g.msg_image != nullptr && at < PIECES) put_message(g.msg_image, l, at / ROW_PIECES, at % ROW_PIECES, x[q]);
    }
    if (WARPS > 1) __syncthreads();     // (the last update has been read)
    else __syncwarp();
    if (lane == 0) {
      g.mem.msg_ts[node] = t;
      g.mem.last_update[node] = t;
      g.mem.msg_flag[node] = 0;
    }
  }
}

int launch_gru_chain(const ChainArgs &args, cudaStream_t s) {
  Ctx *c = cur();
  if (c == nullptr) return set_error(ORCA_E_CUDA, "launch_gru_chain: no context for the current device");
  static thread_local int configured_device = -1;
  if (configured_device != c->device) {
    ORCA_CUDA(cudaFuncSetAttribute(gru_chain_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
    configured_device = c->device;
  }
  ChainArgs g = args;
  g.status = c->status_word;
  g.wait_limit = c->wait_limit;
  const int most = g.a.nb * 2 * g.a.bs;
  ORCA_CUDA(launch_dep(update_image_kernel, std::min(ceil_div(most, 8), c->sm_count * 8), 256, 0, s, g));
  ORCA_COUNT_LAUNCH();
  cudaLaunchConfig_t cfg = {};
  // As many row blocks as fit (a batch with more updates than rows takes another turn), less one, whose SMs are left to the
  // layers that run beside the chain: 48 batches of 1000 3.12 -> 3.08 ms, 50 of 2000 6.56 -> 6.49, others unchanged; two row
  // blocks fewer cost batches of 600 3 %.
  cfg.gridDim = dim3(COL_TILES, std::max(1, std::min(ceil_div(2 * g.a.bs, 8), c->sm_count / COL_TILES - 1)));
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = SMEM;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;     // the CTAs wait for one another
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  ORCA_CUDA(cudaLaunchKernelEx(&cfg, gru_chain_kernel, g));
  ORCA_COUNT_LAUNCH();
  if (most > c->sm_count * 8) ORCA_CUDA(launch_dep(last_messages_kernel<1>, std::min(ceil_div(most, 8), c->sm_count * 6), 256, 0, s, g));
  else ORCA_CUDA(launch_dep(last_messages_kernel<4>, std::min(most, c->sm_count * 8), 128, 0, s, g));
  ORCA_COUNT_LAUNCH();
  ORCA_LAUNCH_CHECK();
  return ORCA_OK;
}

}  // namespace grp
}  // namespace orca
