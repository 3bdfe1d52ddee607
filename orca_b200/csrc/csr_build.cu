// Time-sorted adjacency built on the device (utils/util.py:91-105, get_neighbor_finder).
//
// Every edge i contributes two records: 2i under its source (neighbour = destination) and 2i + 1 under
// its destination.  The reference appends them in this order and then sorts each node's list by
// timestamp with Python's stable sort, so the wanted order of all records is (node, timestamp, record
// number).  That is a stable least-significant-digit radix sort: the edges by the eight bytes of the
// timestamp (mapped to an unsigned key of the same order), then the records by the bytes of the node id.
// A stream that is in time order already -- they nearly always are -- needs no time pass.
//
// What bounds it: the edges come from host memory.  7.8 M edges are 250 MB as the caller holds them (64-bit ids);
// a few threads narrow them to 20 bytes an edge on the way into pinned chunks, so that 157 MB cross the bus while
// the next chunks are packed.  The sort itself moves (node, record) pairs: one pass reads them twice and writes
// them once, all coalesced but for the scatter by digit.
//
// One pass = a per-block digit histogram, a scan of the counts of every digit over the blocks (one block per digit),
// and a stable scatter.  Inside a block every warp owns a contiguous run of the tile and walks it 32 records at a
// time (eight loads in flight); lanes with the same digit find one another with match.any, so a record's rank among
// its digit is the warp's running count plus the number of lower lanes in its group.
#include <algorithm>

#include "common.cuh"
#include "context.cuh"
#include "host_threads.cuh"

namespace orca {
namespace csr {

constexpr int THREADS = 256;
constexpr int WARPS = THREADS / 32;
constexpr int RUN = 1024;            // records per warp
constexpr int TILE = WARPS * RUN;    // records per block
constexpr int BINS = 256;
constexpr int UNROLL = 8;            // loads in flight per lane

// Edges on the device: chunks of CHUNK edges, each [sources | destinations | edge ids | times], so that a chunk is
// one copy from the host.
constexpr int CHUNK_LOG = 16;
constexpr int CHUNK = 1 << CHUNK_LOG;
constexpr size_t CHUNK_BYTES = (size_t)CHUNK * 20;

struct Edges {
  char *p;
  __host__ __device__ char *chunk(int64_t e) const { return p + (e >> CHUNK_LOG) * CHUNK_BYTES; }
  __device__ int32_t &src(int64_t e) const { return reinterpret_cast<int32_t *>(chunk(e))[e & (CHUNK - 1)]; }
  __device__ int32_t &dst(int64_t e) const { return reinterpret_cast<int32_t *>(chunk(e))[CHUNK + (e & (CHUNK - 1))]; }
  __device__ int32_t &eid(int64_t e) const { return reinterpret_cast<int32_t *>(chunk(e))[2 * CHUNK + (e & (CHUNK - 1))]; }
  __device__ double &ts(int64_t e) const {
    return reinterpret_cast<double *>(chunk(e) + (size_t)CHUNK * 12)[e & (CHUNK - 1)];
  }
};

// unsigned key with the order of the doubles (-0.0 and +0.0 equal)
__device__ __forceinline__ uint64_t time_key(double t) {
  const uint64_t u = (uint64_t)__double_as_longlong(t + 0.0);
  return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}

// ---- what a pass sorts: item(i) and the digit it is sorted by
struct ByTime {   // edge numbers, by one byte of their time
  typedef uint32_t Item;
  Edges e;
  const uint32_t *in;         // nullptr: the edges in their own order
  int shift;
  const int32_t *unsorted;    // device word, 0: the stream is in time order and the pass has nothing to do
  __device__ bool skip() const { return *unsorted == 0; }
  __device__ Item load(int64_t i) const { return in ? in[i] : (uint32_t)i; }
  __device__ int digit(Item x) const { return (int)((time_key(e.ts(x)) >> shift) & 0xff); }
};
struct ByNodeFirst {   // (node, record) pairs made from the edges in time order, by the node's lowest byte
  typedef uint2 Item;
  Edges e;
  const uint32_t *order;      // nullptr: the edges in their own order
  const int32_t *unsorted;    // nullptr, or as above: 0 = `order` was not written
  __device__ bool skip() const { return false; }
  __device__ Item load(int64_t i) const {
    int64_t edge = i >> 1;
    if (order != nullptr && (unsorted == nullptr || *unsorted != 0)) edge = order[edge];
    return make_uint2((uint32_t)((i & 1) ? e.dst(edge) : e.src(edge)), (uint32_t)(2 * edge + (i & 1)));
  }
  __device__ int digit(Item x) const { return (int)(x.x & 0xff); }
};
struct ByNode {
  typedef uint2 Item;
  const uint2 *in;
  int shift;
  __device__ bool skip() const { return false; }
  __device__ Item load(int64_t i) const { return in[i]; }
  __device__ int digit(Item x) const { return (int)((x.x >> shift) & 0xff); }
};

// Walks the warp's run, advancing the warp's digit counts; SCATTER: writes every item at its digit's count.
template <bool SCATTER, class S>
__device__ __forceinline__ void walk_run(const S &s, typename S::Item *out, int64_t first, int64_t n,
                                         int32_t *count /* [BINS] of this warp */) {
  const int lane = threadIdx.x & 31;
  const uint32_t lower = (1u << lane) - 1u;
  for (int r = 0; r < RUN && first + r < n; r += 32 * UNROLL) {
    typename S::Item x[UNROLL];
    int d[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      const int64_t i = first + r + 32 * u + lane;
      if (i < n) x[u] = s.load(i);
    }
#pragma unroll
    for (int u = 0; u < UNROLL; ++u)   // lanes past the end group with nobody
      d[u] = first + r + 32 * u + lane < n ? s.digit(x[u]) : BINS + lane;
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      const uint32_t group = __match_any_sync(0xffffffffu, d[u]);
      const bool valid = d[u] < BINS;
      if (SCATTER && valid) out[count[d[u]] + __popc(group & lower)] = x[u];
      __syncwarp();
      if (valid && (group & lower) == 0) count[d[u]] += __popc(group);
      __syncwarp();
    }
  }
}

// counts[digit * n_blocks + block] = items of the block's tile with that digit
template <class S>
__global__ void __launch_bounds__(THREADS) digit_count_kernel(S s, int64_t n, int32_t *counts, int n_blocks) {
  __shared__ int32_t count[WARPS][BINS];
  if (s.skip()) return;
  for (int i = threadIdx.x; i < WARPS * BINS; i += THREADS) (&count[0][0])[i] = 0;
  __syncthreads();
  const int warp = threadIdx.x >> 5;
  walk_run<false>(s, (typename S::Item *)nullptr, (int64_t)blockIdx.x * TILE + (int64_t)warp * RUN, n, count[warp]);
  __syncthreads();
  int total = 0;
  for (int w = 0; w < WARPS; ++w) total += count[w][threadIdx.x];
  counts[(int64_t)threadIdx.x * n_blocks + blockIdx.x] = total;
}

__device__ __forceinline__ int32_t block_scan(int32_t v, int32_t *warp_sum, int32_t &total) {   // exclusive, THREADS threads
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int32_t up = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += up;
  }
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  int32_t before = 0;
  total = 0;
  for (int w = 0; w < WARPS; ++w) {
    if (w < warp) before += warp_sum[w];
    total += warp_sum[w];
  }
  __syncthreads();
  return before + incl - v;
}

// exclusive scan of one digit's counts over the blocks, in place; totals[digit] = their sum
__global__ void __launch_bounds__(THREADS) digit_scan_kernel(int32_t *counts, int n_blocks, int32_t *totals,
                                                             const int32_t *unsorted) {
  __shared__ int32_t warp_sum[WARPS];
  if (unsorted != nullptr && *unsorted == 0) return;
  int32_t *c = counts + (int64_t)blockIdx.x * n_blocks;
  int32_t carry = 0;
  for (int base = 0; base < n_blocks; base += 4 * THREADS) {
    const int i = base + 4 * (int)threadIdx.x;
    int32_t v[4], mine = 0, total;
#pragma unroll
    for (int j = 0; j < 4; ++j) mine += v[j] = i + j < n_blocks ? c[i + j] : 0;
    int32_t run = carry + block_scan(mine, warp_sum, total);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (i + j < n_blocks) c[i + j] = run;
      run += v[j];
    }
    carry += total;
  }
  if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

// stable scatter of the block's tile: a digit's items of this block start behind all lower digits and behind the
// same digit's items of the blocks before
template <class S>
__global__ void __launch_bounds__(THREADS) digit_scatter_kernel(S s, int64_t n, typename S::Item *out,
                                                                const int32_t *offsets, const int32_t *totals,
                                                                int n_blocks) {
  __shared__ int32_t count[WARPS][BINS];
  __shared__ int32_t warp_sum[WARPS];
  if (s.skip()) return;
  for (int i = threadIdx.x; i < WARPS * BINS; i += THREADS) (&count[0][0])[i] = 0;
  int32_t all;
  int32_t at = block_scan(totals[threadIdx.x], warp_sum, all) + offsets[(int64_t)threadIdx.x * n_blocks + blockIdx.x];
  const int warp = threadIdx.x >> 5;
  const int64_t first = (int64_t)blockIdx.x * TILE + (int64_t)warp * RUN;
  walk_run<false>(s, (typename S::Item *)nullptr, first, n, count[warp]);
  __syncthreads();
  for (int w = 0; w < WARPS; ++w) {
    const int32_t c = count[w][threadIdx.x];
    count[w][threadIdx.x] = at;
    at += c;
  }
  __syncthreads();
  walk_run<true>(s, out, first, n, count[warp]);
}

// The adjacency arrays from the sorted records, and indptr: a thread whose record opens a new node fills the
// entries of that node and of the nodes without records before it (the warp fills one lane's stretch together: a
// stretch can be most of the table).
__global__ void __launch_bounds__(256) emit_kernel(Edges e, const uint2 *rec, int64_t n, int64_t n_nodes, int64_t *indptr,
                                                   int32_t *nbr, int32_t *eid, double *adj_ts) {
  const int lane = threadIdx.x & 31;
  for (int64_t p0 = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); p0 <= n; p0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t p = p0 + lane;
    int64_t lo = 0, hi = 0;    // indptr[lo .. hi) = p
    if (p <= n) {
      const uint2 r = p < n ? rec[p] : make_uint2((uint32_t)n_nodes, 0u);
      lo = p > 0 ? (int64_t)rec[p - 1].x + 1 : 0;
      hi = (int64_t)r.x + 1;
      if (p < n) {
        const int64_t edge = r.y >> 1;
        nbr[p] = (r.y & 1) ? e.src(edge) : e.dst(edge);
        eid[p] = e.eid(edge);
        adj_ts[p] = e.ts(edge);
      }
    }
    unsigned todo = __ballot_sync(0xffffffffu, lo < hi);
    while (todo) {
      const int l = __ffs(todo) - 1;
      todo &= todo - 1;
      const int64_t a = __shfl_sync(0xffffffffu, lo, l), b = __shfl_sync(0xffffffffu, hi, l);
      for (int64_t v = a + lane; v < b; v += 32) indptr[v] = p0 + l;
    }
  }
}

// device arrays -> chunks; ids outside the table are reported (and read as node 0), `unsorted` is set when a time is
// smaller than the one before it
__global__ void narrow_kernel(const int64_t *src, const int64_t *dst, const int64_t *eidx, const double *ts, int64_t n_edges,
                              int64_t n_nodes, Edges e, int32_t *unsorted, int32_t *status) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n_edges; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t s = src[i], d = dst[i];
    const bool ok = s >= 0 && s < n_nodes && d >= 0 && d < n_nodes;
    if (!ok) report(status, ORCA_E_BOUNDS, (int)(i < 0x7fffffff ? i : 0x7fffffff));
    e.src(i) = ok ? (int32_t)s : 0;
    e.dst(i) = ok ? (int32_t)d : 0;
    e.eid(i) = (int32_t)eidx[i];
    e.ts(i) = ts[i];
    if (i > 0 && time_key(ts[i]) < time_key(ts[i - 1])) *unsorted = 1;
  }
}

static int sm_count() {
  Ctx *c = cur();
  return c != nullptr ? c->sm_count : 148;
}

static int node_passes(int64_t n_nodes) {
  int p = 1;
  while (p < 4 && ((n_nodes - 1) >> (8 * p)) != 0) ++p;
  return p;
}

struct Layout {
  int64_t edges, rec_a, rec_b, counts, totals, flag, total;
  int n_blocks;
};
static Layout layout(int64_t n_edges) {
  Layout L;
  const int64_t n = 2 * n_edges;
  L.n_blocks = (int)((n + TILE - 1) / TILE);
  auto up = [](int64_t b) { return (b + 255) & ~255ll; };
  L.edges = 0;
  L.rec_a = L.edges + ((n_edges + CHUNK - 1) >> CHUNK_LOG) * (int64_t)CHUNK_BYTES;
  L.rec_b = L.rec_a + up(n * 8);      // (the time passes keep their edge numbers here: half the items, half the bytes)
  L.counts = L.rec_b + up(n * 8);
  L.totals = L.counts + up((int64_t)BINS * L.n_blocks * 4);
  L.flag = L.totals + up(BINS * 4);
  L.total = L.flag + 256;
  return L;
}

template <class S>
static int one_pass(const S &s, int64_t n, typename S::Item *out, int32_t *counts, int32_t *totals,
                    const int32_t *unsorted, cudaStream_t stream) {
  const int blocks = (int)((n + TILE - 1) / TILE);
  digit_count_kernel<S><<<blocks, THREADS, 0, stream>>>(s, n, counts, blocks);
  ORCA_COUNT_LAUNCH();
  ORCA_LAUNCH_CHECK();
  digit_scan_kernel<<<BINS, THREADS, 0, stream>>>(counts, blocks, totals, unsorted);
  ORCA_COUNT_LAUNCH();
  ORCA_LAUNCH_CHECK();
  digit_scatter_kernel<S><<<blocks, THREADS, 0, stream>>>(s, n, out, counts, totals, blocks);
  ORCA_COUNT_LAUNCH();
  ORCA_LAUNCH_CHECK();
  return ORCA_OK;
}

// the sort over edges that are in the workspace; `in_order`: the caller knows that the times do not fall
static int sort_and_emit(const Layout &L, char *base, int64_t n_edges, int64_t n_nodes, bool in_order, int64_t *d_indptr,
                         int32_t *d_nbr, int32_t *d_eid, double *d_adj_ts, cudaStream_t s) {
  const Edges e{base + L.edges};
  int32_t *counts = (int32_t *)(base + L.counts), *totals = (int32_t *)(base + L.totals);
  const int32_t *unsorted = in_order ? nullptr : (const int32_t *)(base + L.flag);
  char *half[2] = {base + L.rec_a, base + L.rec_b};
  const uint32_t *order = nullptr;
  int out = 0;
  if (!in_order) {
    for (int pass = 0; pass < 8; ++pass, out ^= 1) {
      const int rc = one_pass(ByTime{e, order, 8 * pass, unsorted}, n_edges, (uint32_t *)half[out], counts, totals,
                              unsorted, s);
      if (rc) return rc;
      order = (const uint32_t *)half[out];
    }
  }
  const uint2 *rec = nullptr;
  for (int pass = 0; pass < node_passes(n_nodes); ++pass, out ^= 1) {
    const int rc = pass == 0
        ? one_pass(ByNodeFirst{e, order, unsorted}, 2 * n_edges, (uint2 *)half[out], counts, totals, nullptr, s)
        : one_pass(ByNode{rec, 8 * pass}, 2 * n_edges, (uint2 *)half[out], counts, totals, nullptr, s);
    if (rc) return rc;
    rec = (const uint2 *)half[out];
  }
  const int grid = (int)std::min<int64_t>((2 * n_edges + 256) / 256, sm_count() * 16);
  emit_kernel<<<grid, 256, 0, s>>>(e, rec, 2 * n_edges, n_nodes, d_indptr, d_nbr, d_eid, d_adj_ts);
  ORCA_COUNT_LAUNCH();
  ORCA_LAUNCH_CHECK();
  return ORCA_OK;
}

// One host thread's share of the edges: every `step`-th chunk, narrowed into one of the thread's two pinned slots and
// copied from there.  Returns through `out` what it saw.
struct Packed {
  int rc = ORCA_OK;
  int64_t bad_edge = -1;
  bool in_order = true;
  char err[256] = "";
};
static void pack_chunks(const int64_t *src, const int64_t *dst, const int64_t *eidx, const double *ts, int64_t n_edges,
                        int64_t n_nodes, int64_t first, int64_t step, char *slots, Edges e, int device, cudaStream_t s,
                        Packed *out) {
  auto body = [&]() -> int {
    ORCA_CUDA(cudaSetDevice(device));
    cudaEvent_t done[2] = {nullptr, nullptr};
    int rc = ORCA_OK;
    const int64_t n_chunks = (n_edges + CHUNK - 1) >> CHUNK_LOG;
    auto copy_all = [&]() -> int {
      for (cudaEvent_t &ev : done) ORCA_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
      int64_t k = 0;
      for (int64_t c = first; c < n_chunks; c += step, ++k) {
        const int64_t lo = c << CHUNK_LOG, m = std::min<int64_t>(CHUNK, n_edges - lo);
        char *slot = slots + (k & 1) * CHUNK_BYTES;
        if (k >= 2) ORCA_CUDA(cudaEventSynchronize(done[k & 1]));
        int32_t *a = (int32_t *)slot, *b = a + CHUNK, *w = b + CHUNK;
        double *t = (double *)(slot + (size_t)CHUNK * 12);
        uint64_t wide = 0;      // set where an id is negative or not below n_nodes
        const uint64_t lim = (uint64_t)n_nodes;
        for (int64_t i = 0; i < m; ++i) {
          const uint64_t u = (uint64_t)src[lo + i], v = (uint64_t)dst[lo + i];
          wide |= (u >= lim) | (v >= lim);
          a[i] = (int32_t)u;
          b[i] = (int32_t)v;
          w[i] = (int32_t)eidx[lo + i];
        }
        int falls = 0;
        double before = lo > 0 ? ts[lo - 1] : ts[0];
        for (int64_t i = 0; i < m; ++i) {
          const double x = ts[lo + i];
          falls |= !(before <= x);     // (a time that is not a number counts as out of order)
          t[i] = x;
          before = x;
        }
        if (falls) out->in_order = false;
        if (wide) {
          for (int64_t i = lo; out->bad_edge < 0 && i < lo + m; ++i)
            if ((uint64_t)src[i] >= lim || (uint64_t)dst[i] >= lim) out->bad_edge = i;
          return ORCA_OK;
        }
        // (a short last chunk: the four parts up to the last one's end)
        const size_t bytes = m == CHUNK ? CHUNK_BYTES : (size_t)CHUNK * 12 + (size_t)m * 8;
        ORCA_CUDA(cudaMemcpyAsync(e.chunk(lo), slot, bytes, cudaMemcpyHostToDevice, s));
        ORCA_CUDA(cudaEventRecord(done[k & 1], s));
      }
      return ORCA_OK;
    };
    rc = copy_all();
    for (cudaEvent_t ev : done)
      if (ev != nullptr) cudaEventDestroy(ev);
    return rc;
  };
  out->rc = body();
  if (out->rc != ORCA_OK) snprintf(out->err, sizeof(out->err), "%s", orca_last_error());
}

}  // namespace csr
}  // namespace orca

using namespace orca;

extern "C" int64_t orca_csr_build_workspace_bytes(int64_t n_edges, int64_t n_nodes) {
  if (n_edges < 0 || n_nodes <= 0) return -1;
  return csr::layout(n_edges).total;
}

// slots of the packing threads; a thread is worth starting for a chunk or more.  7.8 M edges, the whole call: 24.9 ms
// with one thread, 13.2 / 8.6 / 5.9 / 6.1 with 2 / 4 / 8 / 16 on 16 cores (another box: 6.6 with 16): from eight on the threads are not
// what it waits for.  The copies are: 120 chunks of 1.3 MB, most of them at the bus's rate (28 us) and others three to six times
// that, 5.9 ms in all where the bus alone would take 2.9; then the sort (0.5 ms) and the gathers of emit_kernel (0.35).
constexpr int MOST_THREADS = 16;
static int pack_threads(int64_t n_edges) {
  const int64_t chunks = (n_edges + csr::CHUNK - 1) >> csr::CHUNK_LOG;
  return (int)std::max<int64_t>(1, std::min<int64_t>({MOST_THREADS, chunks, (int64_t)std::thread::hardware_concurrency()}));
}

extern "C" int64_t orca_csr_build_pinned_bytes(int64_t n_edges) {
  return n_edges < 0 ? -1 : (int64_t)(2 * csr::CHUNK_BYTES) * pack_threads(n_edges);
}

static int csr_args_ok(const void *indptr, const void *ws, const void *nbr, const void *eid, const void *ts, int64_t n_edges,
                       int64_t n_nodes, int64_t ws_bytes, int64_t need) {
  ORCA_CHECK_ARG(indptr && ws);
  ORCA_CHECK_ARG(n_edges >= 0 && n_nodes > 0 && n_nodes < (1ll << 31) && n_edges < (1ll << 30));
  ORCA_CHECK_ARG(n_edges == 0 || (nbr && eid && ts));
  ORCA_CHECK_ARG(((uintptr_t)ws & 255) == 0);
  if (ws_bytes < need)
    return set_error(ORCA_E_CAPACITY, "orca_csr_build: workspace of %lld bytes, %lld needed", (long long)ws_bytes,
                     (long long)need);
  return ORCA_OK;
}

extern "C" int orca_csr_build(const int64_t *d_src, const int64_t *d_dst, const int64_t *d_eidx, const double *d_ts,
                              int64_t n_edges, int64_t n_nodes, int64_t *d_indptr, int32_t *d_nbr, int32_t *d_eid,
                              double *d_adj_ts, int32_t *d_status, void *d_workspace, int64_t workspace_bytes,
                              void *stream) {
  const csr::Layout L = csr::layout(n_edges > 0 ? n_edges : 0);
  const int rc = csr_args_ok(d_indptr, d_workspace, d_nbr, d_eid, d_adj_ts, n_edges, n_nodes, workspace_bytes, L.total);
  if (rc) return rc;
  ORCA_CHECK_ARG(d_status && (n_edges == 0 || (d_src && d_dst && d_eidx && d_ts)));
  cudaStream_t s = (cudaStream_t)stream;
  char *base = (char *)d_workspace;
  if (n_edges == 0) {
    ORCA_CUDA(cudaMemsetAsync(d_indptr, 0, (size_t)(n_nodes + 1) * sizeof(int64_t), s));
    return ORCA_OK;
  }
  ORCA_CUDA(cudaMemsetAsync(base + L.flag, 0, sizeof(int32_t), s));
  const int grid = (int)std::min<int64_t>((n_edges + 255) / 256, csr::sm_count() * 16);
  csr::narrow_kernel<<<grid, 256, 0, s>>>(d_src, d_dst, d_eidx, d_ts, n_edges, n_nodes, csr::Edges{base + L.edges},
                                          (int32_t *)(base + L.flag), d_status);
  ORCA_COUNT_LAUNCH();
  ORCA_LAUNCH_CHECK();
  return csr::sort_and_emit(L, base, n_edges, n_nodes, false, d_indptr, d_nbr, d_eid, d_adj_ts, s);
}

extern "C" int orca_csr_build_from_host(const int64_t *h_src, const int64_t *h_dst, const int64_t *h_eidx,
                                        const double *h_ts, int64_t n_edges, int64_t n_nodes, void *h_pinned,
                                        int64_t pinned_bytes, int64_t *d_indptr, int32_t *d_nbr, int32_t *d_eid,
                                        double *d_adj_ts, void *d_workspace, int64_t workspace_bytes, void *stream) {
  const csr::Layout L = csr::layout(n_edges > 0 ? n_edges : 0);
  int rc = csr_args_ok(d_indptr, d_workspace, d_nbr, d_eid, d_adj_ts, n_edges, n_nodes, workspace_bytes, L.total);
  if (rc) return rc;
  ORCA_CHECK_ARG(n_edges == 0 || (h_src && h_dst && h_eidx && h_ts && h_pinned));
  cudaStream_t s = (cudaStream_t)stream;
  char *base = (char *)d_workspace;
  if (n_edges == 0) {
    ORCA_CUDA(cudaMemsetAsync(d_indptr, 0, (size_t)(n_nodes + 1) * sizeof(int64_t), s));
    return ORCA_OK;
  }
  const int threads = (int)std::min<int64_t>(pack_threads(n_edges), pinned_bytes / (int64_t)(2 * csr::CHUNK_BYTES));
  if (threads < 1)
    return set_error(ORCA_E_CAPACITY, "orca_csr_build_from_host: %lld bytes of pinned memory, %lld needed",
                     (long long)pinned_bytes, (long long)(2 * csr::CHUNK_BYTES));
  int device = 0;
  ORCA_CUDA(cudaGetDevice(&device));
  csr::Packed seen[MOST_THREADS];
  auto part = [&](int t) {
    csr::pack_chunks(h_src, h_dst, h_eidx, h_ts, n_edges, n_nodes, t, threads,
                     (char *)h_pinned + (size_t)t * 2 * csr::CHUNK_BYTES, csr::Edges{base + L.edges}, device, s, &seen[t]);
  };
  rc = on_threads(threads, part, "orca_csr_build_from_host");
  bool in_order = true;
  int64_t bad = -1;
  for (int t = 0; t < threads; ++t) {
    const csr::Packed &p = seen[t];
    if (p.rc != ORCA_OK) rc = set_error(p.rc, "%s", p.err);
    in_order = in_order && p.in_order;
    if (p.bad_edge >= 0 && (bad < 0 || p.bad_edge < bad)) bad = p.bad_edge;
  }
  if (rc || bad >= 0) cudaStreamSynchronize(s);     // (copies from the pinned slots may be in flight)
  if (rc) return rc;
  if (bad >= 0) {
    return set_error(ORCA_E_BOUNDS, "orca_csr_build_from_host: edge %lld has an endpoint outside [0,%lld)", (long long)bad,
                     (long long)n_nodes);
  }
  if (!in_order) ORCA_CUDA(cudaMemsetAsync(base + L.flag, 1, sizeof(int32_t), s));
  return csr::sort_and_emit(L, base, n_edges, n_nodes, in_order, d_indptr, d_nbr, d_eid, d_adj_ts, s);
}
