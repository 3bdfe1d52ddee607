// The memory updates of a group of batches in one launch: raw message + GRU of batch 0, 1, ..., each reading the memory
// rows that the batches before it wrote.
//
// As launches of the general projection kernel this chain costs 43 us a batch (message rows written and read back,
// a pipeline filled and drained, two launches) whatever the batch size, and it is the only part of a group that is
// serial: with small batches it is what a stream waits for.  What a batch really waits for is its memory rows.  So
// one cooperative grid walks the batches:
//   - 22 column tiles of 32 gate columns (eight units) times RB row blocks of 32 updates, one CTA each.  A CTA keeps
//     its weight columns (880 x 32, bf16 head and tail, 113 KB) in shared memory for the whole launch.
//   - K is laid out so that what does not depend on the batch before comes first: edge features and time encoding
//     (352 columns) are gathered, converted and multiplied for batch n + 1 while batch n is still being finished.
//   - Then the grid meets at a counter, and only the node's own and the other endpoint's memory rows (2 x 688 bytes
//     an update) are gathered, converted and multiplied; the GRU's hidden operand is the own row's image again.
//   - The result goes to the log row of the update; message table, times and flags follow in one launch at the end.
// A step's products are the ones of the projection kernel, k-step by k-step, so the results are the same bits.
// Warp 0: epilogue (gates; thread = update).  Warps 1-8: gather and split.  Warp 9: MMA issue, tensor memory.
// Every wait is bounded; one that gives up reports ORCA_E_TIMEOUT and the kernel runs to its end.
#include "chain.cuh"
#include "context.cuh"
#include "tc_gemm.cuh"
#include "tc_ptx.cuh"

namespace orca {
namespace grp {

constexpr int ROWS = 32;                       // updates per row block (the MMA's other 96 rows are never read back)
constexpr int COLS = 32, UNITS = COLS / 4;     // gate columns / units per CTA
constexpr int COL_TILES = (4 * D + COLS - 1) / COLS;   // 22
constexpr int PART_CHUNKS = tc::GRU_PART / 8;  // 22 chunks of 8 K elements per part
constexpr int PART_STEPS = tc::GRU_PART / 16;  // 11 MMA steps per part
constexpr int W_LBO = COLS * 16, W_BYTES = 5 * PART_CHUNKS * W_LBO;
constexpr int A_LBO = ROWS * 16 + 16, A_BYTES = 4 * PART_CHUNKS * A_LBO;   // (+16: conflict-free 16-byte stores)
// (an MMA reads 128 rows of a chunk, of which 32 are there: the last chunk's reads run 1520 bytes further)
constexpr int SMEM = 2 * W_BYTES + 2 * A_BYTES + 2048 + 1024 + 256;
constexpr int PRODUCERS = 256, THREADS = 64 + PRODUCERS;
constexpr int TMEM_COLS = 128, BUF_COLS = 64, SMALL = 32;   // two accumulator buffers of main + cross terms
constexpr int META = 4;                        // steps whose row indices are kept

__global__ void __launch_bounds__(THREADS, 1) gru_chain_kernel(const __grid_constant__ ChainArgs g) {
  using namespace tc;
  extern __shared__ unsigned char raw[];
  __shared__ int s_win[MAX_BATCHES];
  __shared__ int s_self[META][ROWS], s_other[META][ROWS], s_eid[META][ROWS];
  __shared__ float s_gap[META][ROWS];
  __shared__ __align__(16) float s_bias[COLS];
  __shared__ __align__(8) unsigned long long s_bar[8];
  __shared__ uint32_t s_tmem;
  const Args &a = g.a;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int ct = blockIdx.x, rb = blockIdx.y, n_cta = gridDim.x * gridDim.y, stride = gridDim.y * ROWS;
  const uint32_t base = (smem_addr(raw) + 1023u) & ~1023u;
  const uint32_t w_hi = base, w_lo = base + W_BYTES, a_hi = base + 2 * W_BYTES, a_lo = a_hi + A_BYTES;
  const uint32_t wbar = smem_addr(&s_bar[0]), ebar = smem_addr(&s_bar[1]), mbar = smem_addr(&s_bar[2]),
                 accbar = smem_addr(&s_bar[3]);
  auto tfree = [&](int b) { return smem_addr(&s_bar[4 + b]); };
  if (tid == 0) {
    mbar_init(wbar, 1);
    mbar_init(ebar, PRODUCERS / 32);
    mbar_init(mbar, PRODUCERS / 32);
    mbar_init(accbar, 1);
    mbar_init(tfree(0), 1);
    mbar_init(tfree(1), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_expect_tx(wbar, 2 * W_BYTES);
    bulk_g2s(w_hi, reinterpret_cast<const char *>(g.w) + (size_t)ct * 2 * W_BYTES, 2 * W_BYTES, wbar);
  }
  if (warp == 9) {
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
  auto mem_row = [&](int r) { return (r >= a.n_nodes ? g.log : g.mem.memory) + (size_t)r * D; };

  int s = 0;    // steps of this CTA so far: 32 updates of one batch each
  if (warp == 0) {
    // ------------------------------------------------------------------ gates
    for (int n = 0; n < a.nb; ++n) {
      for (int r0 = rb * ROWS; r0 < s_win[n]; r0 += stride, ++s) {
        const bool live = r0 + lane < s_win[n];
        mbar_wait(mbar, s & 1, g.status, 610, alive, g.wait_limit);   // (the batches before are complete then)
        float4 h0 = make_float4(0.f, 0.f, 0.f, 0.f), h1 = h0;
        const bool two = ct * UNITS + 4 < D;      // the last tile has four units
        if (live) {
          const float4 *h = reinterpret_cast<const float4 *>(mem_row(s_self[s & (META - 1)][lane]) + ct * UNITS);
          h0 = __ldcg(h);
          if (two) h1 = __ldcg(h + 1);
        }
        mbar_wait(accbar, s & 1, g.status, 611, alive, g.wait_limit);
        tc_fence_after();
        float v[32];
        {
          float x[16];
          const uint32_t t = tmem + (s & 1) * BUF_COLS;
          tmem_ld16_sum(t, SMALL, x);
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = x[i];
          tmem_ld16_sum(t + 16, SMALL, x);
#pragma unroll
          for (int i = 0; i < 16; ++i) v[16 + i] = x[i];
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(tfree(s & 1));
        float y[8];
        const float ho[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
#pragma unroll
        for (int u = 0; u < 8; ++u)
          y[u] = gru_gates(make_float4(v[4 * u] + s_bias[4 * u], v[4 * u + 1] + s_bias[4 * u + 1],
                                       v[4 * u + 2] + s_bias[4 * u + 2], v[4 * u + 3] + s_bias[4 * u + 3]), ho[u]);
        if (live) {
          float4 *o = reinterpret_cast<float4 *>(g.log_out + (size_t)(n * 2 * a.bs + r0 + lane) * D + ct * UNITS);
          o[0] = make_float4(y[0], y[1], y[2], y[3]);
          if (two) o[1] = make_float4(y[4], y[5], y[6], y[7]);
        }
      }
      __threadfence();
      __syncwarp();
      if (lane == 0) asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(&a.cnt->arrived[n]) : "memory");
    }
  } else if (warp < 9) {
    // ------------------------------------------------------------------ gather and split
    const int pt = tid - 32;
    auto put = [&](int chunk, int row, const float4 x, const float4 y) {
      uint4 hi, lo;
      split_chunk(x, y, hi, lo);
      st_shared_v4(a_hi + chunk * A_LBO + row * 16, hi);
      st_shared_v4(a_lo + chunk * A_LBO + row * 16, lo);
    };
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    constexpr int N_UNITS = ROWS * 2 * PART_CHUNKS;     // 16-byte image chunks of two parts
    constexpr int PER = (N_UNITS + PRODUCERS - 1) / PRODUCERS;
    for (int n = 0; n < a.nb; ++n) {
      bool met = n == 0;
      for (int r0 = rb * ROWS; r0 < s_win[n]; r0 += stride, ++s) {
        const int q = s & (META - 1), rows = min(ROWS, s_win[n] - r0);
        if (pt < rows) {
          const int at = n * 2 * a.bs + r0 + pt;
          s_self[q][pt] = a.win_mem[at];
          s_other[q][pt] = a.win_other[at];
          s_eid[q][pt] = a.win_eid[at];
          s_gap[q][pt] = a.win_gap[at];
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");
        // edge features and time encoding: chunks 0 .. 43
        float4 x[PER][2];
#pragma unroll
        for (int i = 0; i < PER; ++i) {
          const int u = pt + i * PRODUCERS, row = u / (2 * PART_CHUNKS), c = u - row * (2 * PART_CHUNKS);
          x[i][0] = x[i][1] = zero;
          if (row < rows && c < PART_CHUNKS) {
            const float4 *e = reinterpret_cast<const float4 *>(g.edge_table + (size_t)s_eid[q][row] * D) + 2 * c;
            x[i][0] = __ldg(e);
            if (c < PART_CHUNKS - 1) x[i][1] = __ldg(e + 1);
          } else if (row < rows) {
            const float gap = s_gap[q][row];
            const int d = (c - PART_CHUNKS) * 8;
            const float4 w0 = __ldg(reinterpret_cast<const float4 *>(g.time_w + d));
            x[i][0] = make_float4(cos_any(gap * w0.x), cos_any(gap * w0.y), cos_any(gap * w0.z), cos_any(gap * w0.w));
            if (d + 4 < D) {
              const float4 w1 = __ldg(reinterpret_cast<const float4 *>(g.time_w + d + 4));
              x[i][1] = make_float4(cos_any(gap * w1.x), cos_any(gap * w1.y), cos_any(gap * w1.z), cos_any(gap * w1.w));
            }
          }
        }
        if (s > 0) mbar_wait(accbar, (s - 1) & 1, g.status, 620, alive, g.wait_limit);   // the image is free again
#pragma unroll
        for (int i = 0; i < PER; ++i) {
          const int u = pt + i * PRODUCERS, row = u / (2 * PART_CHUNKS), c = u - row * (2 * PART_CHUNKS);
          if (row < rows) put(c, row, x[i][0], x[i][1]);
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
              if (v >= n_cta) break;
              if (clock64() - t0 > g.wait_limit) {
                report(g.status, ORCA_E_TIMEOUT, 621);
                alive = false;
                break;
              }
            }
          }
          asm volatile("bar.sync 1, 256;" ::: "memory");
        }
        // own and other memory: chunks 44 .. 87
#pragma unroll
        for (int i = 0; i < PER; ++i) {
          const int u = pt + i * PRODUCERS, row = u / (2 * PART_CHUNKS), c = u - row * (2 * PART_CHUNKS);
          x[i][0] = x[i][1] = zero;
          if (row < rows) {
            const int cc = c < PART_CHUNKS ? c : c - PART_CHUNKS;
            const float4 *m = reinterpret_cast<const float4 *>(mem_row(c < PART_CHUNKS ? s_self[q][row] : s_other[q][row])) + 2 * cc;
            x[i][0] = __ldcg(m);
            if (cc < PART_CHUNKS - 1) x[i][1] = __ldcg(m + 1);
          }
        }
#pragma unroll
        for (int i = 0; i < PER; ++i) {
          const int u = pt + i * PRODUCERS, row = u / (2 * PART_CHUNKS), c = u - row * (2 * PART_CHUNKS);
          if (row < rows) put(2 * PART_CHUNKS + c, row, x[i][0], x[i][1]);
        }
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(mbar);
      }
    }
  } else {
    // ------------------------------------------------------------------ MMA issue
    constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(COLS >> 3) << 17) | (8u << 24);   // M = 128
    mbar_wait(wbar, 0, g.status, 630, alive, g.wait_limit);
    for (int n = 0; n < a.nb; ++n)
      for (int r0 = rb * ROWS; r0 < s_win[n]; r0 += stride, ++s) {
        const uint32_t d = tmem + (s & 1) * BUF_COLS;
        if (s >= 2) mbar_wait(tfree(s & 1), ((s >> 1) & 1) ^ 1, g.status, 631, alive, g.wait_limit);
        // parts of K: edge features, time encoding | own memory, other memory, own memory again
#pragma unroll
        for (int part = 0; part < 5; ++part) {
          if (part == 0) mbar_wait(ebar, s & 1, g.status, 632, alive, g.wait_limit);
          if (part == 2) mbar_wait(mbar, s & 1, g.status, 633, alive, g.wait_limit);
          if (part == 0 || part == 2) tc_fence_after();
          if (elect_one()) {
            const int ap = part < 4 ? part : 2;
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
            if (part == 4) mma_commit(accbar);
          }
          __syncwarp();
        }
      }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}

// Message table, times and flags of every node that the group updated, as its last update leaves them (the rows of
// batches in between are never looked at).  Runs behind the chain and before the memory table is written.
__global__ void __launch_bounds__(256) last_messages_kernel(const __grid_constant__ ChainArgs g) {
  const Args &a = g.a;
  dep_trigger();
  dep_wait();
  const int part = threadIdx.x / 64, lane = threadIdx.x % 64;
  for (int i = blockIdx.x; i < a.nb * 2 * a.bs; i += gridDim.x) {
    const int n = i / (2 * a.bs), w = i - n * 2 * a.bs;
    if (w >= a.cnt->n_win[n]) continue;
    const int node = a.win_node[i];
    if ((unsigned long long)a.bits[node].positive >> (n + 1)) continue;
    float *dst = g.mem.messages + (size_t)node * MSG + part * D;
    auto row = [&](int r) { return (r >= a.n_nodes ? g.log : g.mem.memory) + (size_t)r * D; };
    if (part < 3) {
      const float *src = part == 0 ? row(a.win_mem[i]) : part == 1 ? row(a.win_other[i])
                                                                  : g.edge_table + (size_t)a.win_eid[i] * D;
      if (lane < D / 4) reinterpret_cast<float4 *>(dst)[lane] = reinterpret_cast<const float4 *>(src)[lane];
    } else {
      const float gap = a.win_gap[i];
      for (int d = lane; d < D; d += 64) dst[d] = cos_any(gap * __ldg(g.time_w + d));
    }
    if (threadIdx.x == 0) {
      const float t = a.win_t[i];
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
  // all row blocks that fit at one CTA per SM: a batch with more updates than rows takes another turn per batch
  const int blocks = std::max(1, std::min(ceil_div(2 * g.a.bs, ROWS), c->sm_count / COL_TILES));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(COL_TILES, blocks);
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
  ORCA_CUDA(launch_dep(last_messages_kernel, c->sm_count * 4, 256, 0, s, g));
  ORCA_COUNT_LAUNCH();
  ORCA_LAUNCH_CHECK();
  return ORCA_OK;
}

}  // namespace grp
}  // namespace orca
