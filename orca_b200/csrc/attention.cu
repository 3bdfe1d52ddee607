// The fused gather-attention kernel: per query row, gather the valid neighbour rows and edge-feature
// rows (688 B each) with direct 128-bit loads, compute the time encoding cos(delta * w) in registers,
// and run the masked two-head attention over the slots on chip.  No weight matrix is touched: the K
// and V projections are folded into the query (qt) and into the output GEMM, so the memory side of
// this kernel is pure HBM traffic:
//   in : qt row (2 x 2064 B) + valid slots x (688 + 688) B of gathered rows + K * 12 B of indices
//   out: ctx row (4128 B, fp32 or as bf16 head / tail operand image) + 1 flag
#include <algorithm>
#include <vector>

#include "common.cuh"
#include "attn_out.cuh"
#include "context.cuh"
#include "index_ops.cuh"
#include "tc_ptx.cuh"

namespace orca {

// One warp per query row.  A row's slots are taken two or four at a time: their pieces are loaded into registers -- every
// lane owns 16-byte pieces l, l + 32, l + 64 of the gathered [neighbour | edge feature] part and column PAIRS l, l + 32,
// l + 64 of the time-encoding part, which is computed (cos of delta * w) two columns at a time with the packed
// two-wide fp32 instructions of this architecture while the loads are in flight -- then come the partial dot products
// with the two query heads, one cross-lane sum of all logits of the step at once, a running softmax and the weighted sums,
// all from the same registers.
// What bounds it: the instructions of a row and the SM's load path, against the 16 or 12 warps an SM that the registers allow
// (66 k rows of the largest graph, counters: 0.42 GB to and from DRAM in layer 1, 0.56 in layer 2, 2.5 and 3.4 TB/s or 39 and
// 52 % of what a copy reaches; 36 and 54 k rows of 194 k nodes: issue slots 55 % busy, L1 66 %, L2 28 %, DRAM 22 to 35 %).
// Loads of the slots' rows cost next to nothing: with all of them in L1 a launch took 2 % less.  So what helps is fewer instructions a slot (193 -> 160, and 143 four at a time, of 75 that the sums,
// products and cosines cannot do without) and queries that do not pass through L1 once a step:
//   - what all lanes need of a slot (addresses, time difference) is worked out once a row, a slot a lane, and read back from
//     shared memory; so are the weights, twice each, as the packed instructions take them;
//   - one exponential a step gives weights and scales, in lanes of their own; sums are rescaled where a maximum rose;
//   - a row's query is brought to shared memory by one bulk copy while the row before it is written.
// us a launch (queries written by the kernel before; 66 k rows of the largest graph, K 10 / 60 k of c4, K 10 / 54 k, K 20):
// before 197 / 197 / 340; so 166 / 162 / 254.  Valid slots side by side wherever their places are, no query for a row without any:
// 40 k rows of ten / twenty slots 149 / 217 (152 / 220 from the first valid place to the last), half of the places empty 107 / 150
// (127 / 199), none valid 31 (45).  Four slots a step at 168 registers against two at 128, 27 k rows, K 8 / 10 / 12 /
// 14 / 16 / 20 / 32: 79 / 97 / 97 / 116 / 117 / 136 / 187 against 83 / 93 / 106 / 118 / 130 / 152 / 214; 30 k of c4, where rows are
// shorter: 81 / 95 / 97 / 112 / 112 / 128 / 175 against 80 / 89 / 97 / 108 / 116 / 136 / 192: four from K 11 on.
// Measured against it: queries in registers at 12 warps (181 / 175 / 288); a row's first slots loaded before the row in front
// of it is written (177 / 173 / 307); four slots and a tail of two (176 / 172 / 260).  Of the form before: two passes over the
// rows with parked logits 8 % slower, slots copied ahead with cp.async up to 20 %, the long cosine inlined with a variant of
// the loop per range twice the time (instruction cache).  The 688-byte rows are not moved by cp.async.bulk: an SM retires
// only about one small bulk copy per ~130 cycles.
//
// Work distribution.  Rows differ tenfold in cost (0 to k valid slots) and a launch of a single batch holds only two
// to three rows per resident warp, so WHO gets WHICH row decides the length of the launch:
//   - rows are handed out by ticket (one atomic per row on a counter the launch leaves at zero again);
//   - tickets walk the rows in the order of `order` (rows sorted by falling number of valid slots,
//     made by row_order_kernel beside the sampling), so that the launch ends on its lightest rows.
// A warp draws its next ticket when it starts a row and reads it after the row's first slots; the indices of the next
// row are loaded while the rest of the row is worked on.  No block-level synchronisation.
constexpr int GA_THREADS = 64, GA_WARPS = GA_THREADS / 32;
constexpr int ga_blocks(int slots) { return slots == 2 ? 8 : 6; }   // an SM: 16 warps at 128 registers, 12 at 168
constexpr int GA_WIDE_FROM = 11;                // slots a row from which they are taken four at a time
constexpr int GA_MEM_F4 = 2 * D / 4;            // 86 sixteen-byte pieces of [neighbour | edge feature]
constexpr int GA_ROW_F4 = D / 4;                // 43 pieces per table row
constexpr int GA_P_ITERS = 3;                   // pieces / time-column pairs per lane (the third for lanes 0..21)

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 dup2(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 lo2(const float4 &v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4 &v) { return make_float2(v.z, v.w); }

// cos of two arguments below COS_SMALL at once: the reduction of cos_small in packed arithmetic with fewer steps.  The
// nearest integer k of x / 2pi comes from adding and subtracting 1.5 * 2^23, in one fused step, and 2pi is split in two:
// x - k * C1 is a multiple of 2^-22 below 4 (C1 has 24 bits, the last of them 2^-21), so the first difference is exact.
__device__ __forceinline__ float2 cos_small2(float2 x) {
  const float2 t = fma2(x, dup2(0.15915494309189535f), dup2(12582912.f));
  const float2 kk = add2(t, dup2(-12582912.f));
  float2 r = fma2(kk, dup2(-6.2831855f), x);
  r = fma2(kk, dup2(1.7484556e-07f), r);
  return make_float2(__cosf(r.x), __cosf(r.y));
}

// Arguments beyond the fixed-point range (or not finite) are rare: their cosine is a call, so that its long code does
// not stand in the loops six times over (the kernel has to stay within the instruction cache).
__device__ __noinline__ float cos_far(float x) { return cos_any(x); }

// Time encodings of one slot for this lane's column pairs: the first nl pair groups (64 columns each) hold large
// arguments (fixed-point reduction), the others small ones (packed fp32 reduction); nl < 0: beyond both.  w decreases
// with the column, so "large" groups are always a prefix; nl is uniform over the warp.
__device__ __forceinline__ void time_terms(float dt, int nl, const float2 (&wt)[GA_P_ITERS], float2 (&te)[GA_P_ITERS]) {
#pragma unroll
  for (int i = 0; i < GA_P_ITERS; ++i) {
    const float2 x = mul2(dup2(dt), wt[i]);
    if (nl < 0) te[i] = make_float2(cos_far(x.x), cos_far(x.y));
    else if (i < nl) te[i] = make_float2(cos_fixed(x.x), cos_fixed(x.y));
    else te[i] = cos_small2(x);
  }
}

// Rows sorted by falling number of valid slots (counting sort, one block): order[0 .. n) = row ids.  The
// tables are right-aligned (padding first), so a row's count is k minus the position of its first neighbour, which is bisected
// for, eight rows of a thread side by side.  (A slot that stayed empty among the others may make a count wrong: a row then comes
// earlier or later, no more.)  Counting all slots, twice, took a wavefront of L1 per entry, 5000 rows of 32 slots 161 us and 250
// beside a gather launch on the same SM, which single calls waited for (1500 edges 250 to 380 us, 152 now); now 20.
constexpr int RO_ROWS = 8;
__global__ void __launch_bounds__(1024)
row_order_kernel(const int32_t *__restrict__ nbr_a, int n_cap_a, const int32_t *__restrict__ d_n_a,
                 int32_t *__restrict__ order_a, const int32_t *__restrict__ nbr_b, int n_cap_b,
                 const int32_t *__restrict__ d_n_b, int32_t *__restrict__ order_b, int k) {
  __shared__ int s_bin[ORCA_MAX_K + 1];
  dep_trigger();
  dep_wait();
  // block 0 orders table a, block 1 table b
  const int32_t *nbr = blockIdx.x == 0 ? nbr_a : nbr_b;
  int32_t *order = blockIdx.x == 0 ? order_a : order_b;
  const int n = blockIdx.x == 0 ? rows_of(n_cap_a, d_n_a) : rows_of(n_cap_b, d_n_b);
  const int tid = threadIdx.x;
  if (tid <= ORCA_MAX_K) s_bin[tid] = 0;
  __syncthreads();
  // the counts of rows r0 + 1024 u (u < RO_ROWS); rows past the last: -1
  auto counts = [&](int r0, int (&c)[RO_ROWS]) {
    int empty[RO_ROWS] = {};
#pragma unroll
    for (int s = 32; s > 0; s >>= 1)
#pragma unroll
      for (int u = 0; u < RO_ROWS; ++u)
        if (r0 + 1024 * u < n && empty[u] + s <= k && nbr[(size_t)(r0 + 1024 * u) * k + empty[u] + s - 1] == 0) empty[u] += s;
#pragma unroll
    for (int u = 0; u < RO_ROWS; ++u) c[u] = r0 + 1024 * u < n ? k - empty[u] : -1;
  };
  static_assert(ORCA_MAX_K == 32, "the bisection's first step");
  int first[RO_ROWS];      // (of up to 8192 rows the counts are kept)
  counts(tid, first);
#pragma unroll
  for (int u = 0; u < RO_ROWS; ++u)
    if (first[u] >= 0) atomicAdd(&s_bin[first[u]], 1);
  for (int r = tid + 1024 * RO_ROWS; r < n; r += 1024 * RO_ROWS) {
    int c[RO_ROWS];
    counts(r, c);
#pragma unroll
    for (int u = 0; u < RO_ROWS; ++u)
      if (c[u] >= 0) atomicAdd(&s_bin[c[u]], 1);
  }
  __syncthreads();
  if (tid == 0) {   // bins -> first position, heaviest bin first
    int pos = 0;
    for (int c = k; c >= 0; --c) {
      const int m = s_bin[c];
      s_bin[c] = pos;
      pos += m;
    }
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < RO_ROWS; ++u)
    if (first[u] >= 0) order[atomicAdd(&s_bin[first[u]], 1)] = tid + 1024 * u;
  for (int r = tid + 1024 * RO_ROWS; r < n; r += 1024 * RO_ROWS) {
    int c[RO_ROWS];
    counts(r, c);
#pragma unroll
    for (int u = 0; u < RO_ROWS; ++u)
      if (c[u] >= 0) order[atomicAdd(&s_bin[c[u]], 1)] = r + 1024 * u;
  }
}

// What a step needs of a slot, by all lanes at once: where its two rows start, its time difference (twice: an operand of
// the packed instructions) and how many pair groups of its time encoding hold large arguments (time_terms).  The edge row's
// address is a row early, so that a lane's pieces l, l + 32, l + 64 of [neighbour | edge feature] lie 0, 512 and 1024 bytes
// behind 16 l of the one or the other.
struct __align__(16) SlotRec {
  const char *nbr, *edge;
  float dt[2];
  int large, unused;
};
__device__ __forceinline__ float4 ldg4(const char *p) { return __ldg(reinterpret_cast<const float4 *>(p)); }

// Sums V values (V a power of two up to 32) over the warp: lane l returns the total of value l / (32 / V).
template <int V>
__device__ __forceinline__ float warp_sum_many(float (&v)[V], int lane) {
  constexpr unsigned FULL = 0xffffffffu;
  int o = 16;
#pragma unroll
  for (int n = V / 2; n > 0; n >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < n; ++i) {   // a lane keeps the half of the values that its bit names and hands over the other
      const float give = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
      v[i] = keep + __shfl_xor_sync(FULL, give, o);
    }
  }
  float s = v[0];
  for (; o > 0; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
  return s;
}

template <bool IMAGE, int GS>
__global__ void __launch_bounds__(GA_THREADS, ga_blocks(GS))
attn_gather_kernel(const float *__restrict__ qt, const float *__restrict__ nbr_table,
                   const float *__restrict__ nbr_table2, int nbr_split,
                   const float *__restrict__ edge_table, const float *__restrict__ time_w,
                   const int32_t *__restrict__ nbr, const int32_t *__restrict__ eid,
                   const float *__restrict__ delta, int k, int n_cap, const int32_t *__restrict__ d_n,
                   const int32_t *__restrict__ order, const int32_t *__restrict__ q_row, void *__restrict__ ctx,
                   uint8_t *__restrict__ valid_out, int32_t *__restrict__ ticket, unsigned long long *__restrict__ prof,
                   int32_t *status, long long wait_limit) {
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ __align__(128) float s_q[GA_WARPS][QT_LD];
  __shared__ SlotRec s_rec[GA_WARPS][ORCA_MAX_K + GS - 1];
  __shared__ __align__(16) float s_p[GA_WARPS][4 * GS + 4];
  __shared__ __align__(8) unsigned long long s_bar[GA_WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t qbar = tc::smem_addr(&s_bar[warp]);
  if (lane == 0) {
    tc::mbar_init(qbar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  dep_trigger();
  dep_wait();
  const int n = rows_of(n_cap, d_n);
  const bool third = lane + 64 < GA_MEM_F4;       // lanes 0..21 own a third piece / pair
  const bool from_edge = lane >= GA_ROW_F4 - 32;  // whose piece l + 32 is one of the edge row
  float2 wt[GA_P_ITERS];
#pragma unroll
  for (int i = 0; i < GA_P_ITERS; ++i)
    wt[i] = (i < 2 || third) ? __ldg(reinterpret_cast<const float2 *>(time_w) + lane + 32 * i) : make_float2(0.f, 0.f);
  const float wg0 = __ldg(time_w), wg1 = __ldg(time_w + 64), wg2 = __ldg(time_w + 128);
  unsigned long long prof_rows = 0, prof_slots = 0;

  // (A group's rows from the last one back: the images of the rows that the output kernel starts with are still in L2, and so,
  // where every row has a query of its own, are the queries written last.  Measured when both layers' rows had: 200 MB of
  // queries a launch do not fit L2, 50 batches of 2000 5.80 -> 5.68 ms, 51 of 600 3.00 -> 2.96, without reuse 2.36 -> 2.30.)
  auto row_of_ticket = [&](int t) -> int { return order != nullptr ? order[t] : n - 1 - t; };
  auto load_indices = [&](int r, int &o_nbr, int &o_eid, float &o_dt, int &o_q) {
    o_q = q_row != nullptr ? q_row[r] : r;
    o_nbr = 0, o_eid = 0, o_dt = 0.f;
    if (lane < k) {
      const size_t o = (size_t)r * k + lane;
      o_nbr = nbr[o];
      o_eid = eid[o];
      o_dt = delta[o];
    }
  };
  bool alive = true;
  uint32_t phase = 0;
  auto fetch_query = [&](int r) {
    if (lane == 0 && alive) {
      tc::mbar_expect_tx(qbar, QT_LD * 4);
      tc::bulk_g2s(tc::smem_addr(s_q[warp]), qt + (size_t)r * QT_LD, QT_LD * 4, qbar);
    }
  };
  int tkt = 0;
  if (lane == 0) tkt = atomicAdd(&ticket[0], 1);
  tkt = __shfl_sync(FULL, tkt, 0);
  int row = tkt < n ? row_of_ticket(tkt) : -1;
  int my_nbr = 0, my_eid = 0;
  float my_dt = 0.f;
  if (row >= 0) {
    int q;
    load_indices(row, my_nbr, my_eid, my_dt, q);
    if (__any_sync(FULL, my_nbr != 0)) fetch_query(q);
  }
  float4 x[GS][3];                                 // (the third piece of the lanes that have none stays zero)
#pragma unroll
  for (int s = 0; s < GS; ++s) x[s][2] = make_float4(0.f, 0.f, 0.f, 0.f);
  float *const pbuf = s_p[warp];
  while (row >= 0) {
    // the next ticket is drawn now and its row's indices are requested after the first slots (see above)
    if (lane == 0) tkt = atomicAdd(&ticket[0], 1);
    int next = -1, nx_nbr = 0, nx_eid = 0, nx_q = 0;
    float nx_dt = 0.f;
    auto draw_next = [&]() {
      const int t = __shfl_sync(FULL, tkt, 0);
      if (t < n) {
        next = row_of_ticket(t);
        load_indices(next, nx_nbr, nx_eid, nx_dt, nx_q);
      }
    };
    float4 am0[3], am1[3];                         // weighted sums of the gathered part, heads 0 / 1
    float2 at0[GA_P_ITERS], at1[GA_P_ITERS];       // and of the time part
#pragma unroll
    for (int i = 0; i < 3; ++i) am0[i] = am1[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < GA_P_ITERS; ++i) at0[i] = at1[i] = make_float2(0.f, 0.f);
    float sum0 = 0.f, sum1 = 0.f;
    const unsigned vmask = __ballot_sync(FULL, my_nbr != 0);
    const int n_valid = __popc(vmask);
    if (n_valid > 0) {
      tc::mbar_wait(qbar, phase, status, 800, alive, wait_limit);
      phase ^= alive;      // (stays at a query that did not come)
      {
        // which pair groups of the slot need the fixed-point cosine (see time_terms)
        const float adt = fabsf(my_dt);
        int large = (adt * wg0 >= COS_SMALL ? 1 : 0) + (adt * wg1 >= COS_SMALL ? 1 : 0) + (adt * wg2 >= COS_SMALL ? 1 : 0);
        if (!(adt * wg0 < 1073741824.f)) large = -1;   // beyond the fixed-point range (or not finite)
        SlotRec rec;
        rec.nbr = reinterpret_cast<const char *>(my_nbr >= nbr_split ? nbr_table2 : nbr_table) + (size_t)my_nbr * ROW_BYTES;
        rec.edge = reinterpret_cast<const char *>(edge_table) + (size_t)my_eid * ROW_BYTES - ROW_BYTES;
        rec.dt[0] = rec.dt[1] = my_dt;
        rec.large = large;
        rec.unused = 0;
        // the valid slots one behind the other; behind them, up to a whole step, the first one again with weight zero
        const int at = __popc(vmask & ((1u << lane) - 1u));
        if (my_nbr != 0) s_rec[warp][at] = rec;
        if (my_nbr != 0 && at == 0)
          for (int u = 0; u < GS - 1; ++u) s_rec[warp][n_valid + u] = rec;
        __syncwarp();
      }
      const float *q_src = s_q[warp];
      float m = -INFINITY;     // running maximum of this lane's head
      // GS slots at a time, each row of them in registers from its dot products to its weighted sum: nothing is
      // loaded twice, and the cross-lane sums of 2 * GS logits cost little more than those of one
      constexpr int V = 2 * GS, LPV = 32 / V;
      for (int at = 0; at < n_valid; at += GS) {
        float2 te[GS][GA_P_ITERS];
        float4 dts[GS];
#pragma unroll
        for (int s = 0; s < GS; ++s) {
          const ulonglong2 p = *reinterpret_cast<const ulonglong2 *>(&s_rec[warp][at + s].nbr);
          const char *nrow = reinterpret_cast<const char *>(p.x) + 16 * lane, *erow = reinterpret_cast<const char *>(p.y) + 16 * lane;
          x[s][0] = ldg4(nrow);
          x[s][1] = ldg4((from_edge ? erow : nrow) + 512);
          if (third) x[s][2] = ldg4(erow + 1024);
          dts[s] = *reinterpret_cast<const float4 *>(&s_rec[warp][at + s].dt);
        }
        int any = 0;        // (of all slots of the step: one branch, and the usual case is straight code)
#pragma unroll
        for (int s = 0; s < GS; ++s) any |= __float_as_int(dts[s].z);
        if (any == 0) {
#pragma unroll
          for (int s = 0; s < GS; ++s)
#pragma unroll
            for (int i = 0; i < GA_P_ITERS; ++i) te[s][i] = cos_small2(mul2(make_float2(dts[s].x, dts[s].y), wt[i]));
        } else {
#pragma unroll
          for (int s = 0; s < GS; ++s) time_terms(dts[s].x, __float_as_int(dts[s].z), wt, te[s]);
        }
        // partial logits: value 2 * s + head
        float2 a0[GS], a1[GS];
#pragma unroll
        for (int s = 0; s < GS; ++s) a0[s] = a1[s] = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < GA_P_ITERS; ++i) {
          // (a lane without a third piece multiplies zeros by what lies there; its third time pair is cos(0))
          const float4 qa = *(reinterpret_cast<const float4 *>(q_src) + lane + 32 * i);
          const float4 qb = *(reinterpret_cast<const float4 *>(q_src + QT_HEAD) + lane + 32 * i);
          float2 qta = make_float2(0.f, 0.f), qtb = qta;
          if (i < 2 || third) {
            qta = *(reinterpret_cast<const float2 *>(q_src + 2 * D) + lane + 32 * i);
            qtb = *(reinterpret_cast<const float2 *>(q_src + QT_HEAD + 2 * D) + lane + 32 * i);
          }
#pragma unroll
          for (int s = 0; s < GS; ++s) {
            a0[s] = fma2(te[s][i], qta, a0[s]);
            a1[s] = fma2(te[s][i], qtb, a1[s]);
            a0[s] = fma2(lo2(x[s][i]), lo2(qa), a0[s]);
            a0[s] = fma2(hi2(x[s][i]), hi2(qa), a0[s]);
            a1[s] = fma2(lo2(x[s][i]), lo2(qb), a1[s]);
            a1[s] = fma2(hi2(x[s][i]), hi2(qb), a1[s]);
          }
        }
        float v[V];
#pragma unroll
        for (int s = 0; s < GS; ++s) v[2 * s] = a0[s].x + a0[s].y, v[2 * s + 1] = a1[s].x + a1[s].y;
        // lane l holds value l / LPV = 2 * slot + head; head = one lane bit
        float lg = warp_sum_many<V>(v, lane);
        // the next row of this warp: its indices land while this one is finished
        if (at == 0) draw_next();
        if (at + lane / (2 * LPV) >= n_valid) lg = -INFINITY;
        float top = lg;
#pragma unroll
        for (int o = 2 * LPV; o < 32; o <<= 1) top = fmaxf(top, __shfl_xor_sync(FULL, top, o));
        const float m_new = fmaxf(m, top);
        // even lanes: the slot's weight; odd lanes: what the sums so far are scaled by (0 the first time)
        const float p = expf((lane & 1 ? m : lg) - m_new);
        m = m_new;
        // [slot][head] weights, [head] scales, each twice (operands of the packed instructions)
        const int where = lane & 1 ? 2 * GS + (lane / LPV & 1) : lane / LPV;
        reinterpret_cast<float2 *>(pbuf)[where] = dup2(p);
        __syncwarp();
        const float4 S = *reinterpret_cast<const float4 *>(pbuf + 4 * GS);
        sum0 *= S.x, sum1 *= S.z;
        if (at > 0 && (S.x != 1.f || S.z != 1.f)) {
          const float2 S0 = lo2(S), S1 = hi2(S);
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            float2 r;
            r = mul2(S0, lo2(am0[i])); am0[i].x = r.x; am0[i].y = r.y;
            r = mul2(S0, hi2(am0[i])); am0[i].z = r.x; am0[i].w = r.y;
            r = mul2(S1, lo2(am1[i])); am1[i].x = r.x; am1[i].y = r.y;
            r = mul2(S1, hi2(am1[i])); am1[i].z = r.x; am1[i].w = r.y;
            at0[i] = mul2(S0, at0[i]);
            at1[i] = mul2(S1, at1[i]);
          }
        }
#pragma unroll
        for (int s = 0; s < GS; ++s) {
          const float4 P = *reinterpret_cast<const float4 *>(pbuf + 4 * s);
          const float2 P0 = lo2(P), P1 = hi2(P);
          sum0 += P.x, sum1 += P.z;
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            float2 r;
            r = fma2(P0, lo2(x[s][i]), lo2(am0[i])); am0[i].x = r.x; am0[i].y = r.y;
            r = fma2(P0, hi2(x[s][i]), hi2(am0[i])); am0[i].z = r.x; am0[i].w = r.y;
            r = fma2(P1, lo2(x[s][i]), lo2(am1[i])); am1[i].x = r.x; am1[i].y = r.y;
            r = fma2(P1, hi2(x[s][i]), hi2(am1[i])); am1[i].z = r.x; am1[i].w = r.y;
            at0[i] = fma2(P0, te[s][i], at0[i]);
            at1[i] = fma2(P1, te[s][i], at1[i]);
          }
        }
        __syncwarp();
      }
      prof_rows += 1;
      prof_slots += (unsigned long long)n_valid;
    } else {
      draw_next();
    }
    __syncwarp();        // (the query has been read by all lanes: the next one may land)
    if (__any_sync(FULL, nx_nbr != 0)) fetch_query(nx_q);      // (a row without valid slots asks for nothing)
    // write the row: [head 0: gathered 344 | time 172][head 1: ...].  A row whose slots are all padding has no attention
    // term: the image gets zeros (the fp32 form leaves such a row alone, `valid` says so).
    const float inv0 = n_valid > 0 ? 1.f / sum0 : 0.f, inv1 = n_valid > 0 ? 1.f / sum1 : 0.f;
    if (IMAGE) {
      char *im = (char *)ctx + (size_t)(row / img::ROWS) * (img::CTX_STAGES * img::STAGE_BYTES) + (row % img::ROWS) * 64;
      const int sw = (row << 3) & 0x30;
      // (img::at, with the row's part taken out: the four pieces of a lane advance by whole stages)
      auto place = [&](int c) { return im + (((c >> 5) * img::STAGE_BYTES + (c >> 3 & 3) * 16 + 2 * (c & 7)) ^ sw); };
      char *o0 = place(4 * lane), *o1 = place(KEY + 4 * lane), *o2 = place(2 * D + 2 * lane), *o3 = place(KEY + 2 * D + 2 * lane);
      auto put4 = [&](char *p, float4 v, float inv) {
        const float2 a = mul2(dup2(inv), lo2(v)), b = mul2(dup2(inv), hi2(v));
        uint2 hi, lo;
        hi.x = tc::pack_split(a.x, a.y, lo.x);
        hi.y = tc::pack_split(b.x, b.y, lo.y);
        *reinterpret_cast<uint2 *>(p) = hi;
        *reinterpret_cast<uint2 *>(p + img::STAGE_BYTES / 2) = lo;
      };
      auto put2 = [&](char *p, float2 v, float inv) {
        const float2 a = mul2(dup2(inv), v);
        uint32_t lo;
        const uint32_t hi = tc::pack_split(a.x, a.y, lo);
        *reinterpret_cast<uint32_t *>(p) = hi;
        *reinterpret_cast<uint32_t *>(p + img::STAGE_BYTES / 2) = lo;
      };
#pragma unroll
      for (int i = 0; i < 3; ++i)
        if (i < 2 || third) {
          put4(o0 + i * 4 * img::STAGE_BYTES, am0[i], inv0);
          put4(o1 + i * 4 * img::STAGE_BYTES, am1[i], inv1);
          put2(o2 + i * 2 * img::STAGE_BYTES, at0[i], inv0);
          put2(o3 + i * 2 * img::STAGE_BYTES, at1[i], inv1);
        }
      if (lane < (img::CTX_STAGES * img::STAGE_K - QT) / 4) {    // padding
        char *p = place(QT + 4 * lane);
        *reinterpret_cast<uint2 *>(p) = make_uint2(0, 0);
        *reinterpret_cast<uint2 *>(p + img::STAGE_BYTES / 2) = make_uint2(0, 0);
      }
    } else if (n_valid > 0) {
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const int f = lane + 32 * i;
        if (i < 2 || third) {
          float *out = (float *)ctx + (size_t)row * QT;
          reinterpret_cast<float4 *>(out)[f] = make_float4(am0[i].x * inv0, am0[i].y * inv0, am0[i].z * inv0, am0[i].w * inv0);
          reinterpret_cast<float4 *>(out + KEY)[f] = make_float4(am1[i].x * inv1, am1[i].y * inv1, am1[i].z * inv1, am1[i].w * inv1);
          reinterpret_cast<float2 *>(out + 2 * D)[f] = make_float2(at0[i].x * inv0, at0[i].y * inv0);
          reinterpret_cast<float2 *>(out + KEY + 2 * D)[f] = make_float2(at1[i].x * inv1, at1[i].y * inv1);
        }
      }
    }
    if (lane == 0) valid_out[row] = n_valid > 0 ? 1 : 0;
    row = next;
    my_nbr = nx_nbr;
    my_eid = nx_eid;
    my_dt = nx_dt;
  }
  if (lane == 0) {
    if (!alive) tc::mbar_settle(qbar, phase);
    // the last warp to run out of tickets leaves the counters at zero for the next launch
    const int total = (int)(gridDim.x * (blockDim.x >> 5));
    if (atomicAdd(&ticket[1], 1) == total - 1) {
      atomicExch(&ticket[0], 0);
      atomicExch(&ticket[1], 0);
    }
    if (prof != nullptr && prof_rows) {
      atomicAdd(&prof[0], prof_rows);     // rows that gathered
      atomicAdd(&prof[1], prof_slots);    // gathered neighbour slots
    }
  }
}

// d_nbr_table2 (optional): neighbour rows >= nbr_split are read from it; its address is already moved back by
// nbr_split rows
// d_q_row (optional): row r's query is row d_q_row[r] of d_qt
// d_status (optional): where a wait that gave up is reported instead of the context's status word
// `ticket`: two zeroed device words that the launch leaves at zero; launches that may overlap on the GPU
// need words of their own
int launch_attn_gather(const float *d_qt, const float *d_nbr_table, const float *d_edge_table,
                       const float *d_time_w, const int32_t *d_nbr, const int32_t *d_eid, const float *d_delta,
                       int k, int n_rows_cap, const int32_t *d_n_rows, int rows_hint, const int32_t *d_order,
                       void *d_ctx, bool image, uint8_t *d_valid, int32_t *d_ticket, cudaStream_t stream,
                       const float *d_nbr_table2, int nbr_split, const int32_t *d_q_row, int32_t *d_status) {
  if (d_nbr_table2 == nullptr) nbr_split = 0x7fffffff;
  ORCA_CHECK_ARG(d_qt && d_nbr_table && d_edge_table && d_time_w && d_nbr && d_eid && d_delta && d_ctx &&
                 d_valid && d_ticket);
  ORCA_CHECK_ARG(k >= 1 && k <= ORCA_MAX_K && n_rows_cap >= 0);
  ORCA_CHECK_ARG(((uintptr_t)d_qt % 16 == 0) && ((uintptr_t)d_nbr_table % 16 == 0) &&
                 ((uintptr_t)d_edge_table % 16 == 0));
  if (n_rows_cap == 0) return ORCA_OK;
  Ctx *c = cur();
  if (c == nullptr) return set_error(ORCA_E_CUDA, "orca_attn_gather: no context for the current device");
  GatherProfile &pf = c->prof;
  if (pf.on) {
    if (pf.used + 2 > pf.ev.size()) {
      cudaEvent_t a, b;
      ORCA_CUDA(cudaEventCreate(&a));
      ORCA_CUDA(cudaEventCreate(&b));
      pf.ev.push_back(a);
      pf.ev.push_back(b);
    }
    ORCA_CUDA(cudaEventRecord(pf.ev[pf.used], stream));
  }
  if (d_status == nullptr) d_status = c->status_word;
  // one resident wave at most; fewer blocks when the caller expects fewer rows than the capacity
  const int rows = rows_hint > 0 ? std::min(rows_hint, n_rows_cap) : n_rows_cap;
  const bool wide = k >= GA_WIDE_FROM;
  const int grid = std::min(ceil_div(rows, GA_WARPS), c->sm_count * ga_blocks(wide ? 4 : 2));
  auto kernel = image ? (wide ? attn_gather_kernel<true, 4> : attn_gather_kernel<true, 2>)
                      : (wide ? attn_gather_kernel<false, 4> : attn_gather_kernel<false, 2>);
  // (the profiling events would sit between this kernel and its neighbours: plain launch then)
  if (pf.on)
    kernel<<<grid, GA_THREADS, 0, stream>>>(d_qt, d_nbr_table, d_nbr_table2, nbr_split, d_edge_table, d_time_w, d_nbr, d_eid,
                                            d_delta, k, n_rows_cap, d_n_rows, d_order, d_q_row, d_ctx, d_valid, d_ticket,
                                            pf.d_counters, d_status, c->wait_limit);
  else
    ORCA_CUDA(launch_dep(kernel, grid, GA_THREADS, 0, stream, d_qt, d_nbr_table, d_nbr_table2, nbr_split, d_edge_table,
                         d_time_w, d_nbr, d_eid, d_delta, (int)k, (int)n_rows_cap, d_n_rows, d_order, d_q_row, d_ctx, d_valid,
                         d_ticket, (unsigned long long *)nullptr, d_status, c->wait_limit));
  if (pf.on) {
    ORCA_CUDA(cudaEventRecord(pf.ev[pf.used + 1], stream));
    pf.used += 2;
  }
  ORCA_COUNT_LAUNCH();
  ORCA_LAUNCH_CHECK();
  return ORCA_OK;
}

// rows of two neighbour tables (the two attention layers of a batch) in the order the gather kernel should
// take them: heaviest first
int launch_row_order(const int32_t *d_nbr_a, int n_cap_a, const int32_t *d_n_a, int32_t *d_order_a,
                     const int32_t *d_nbr_b, int n_cap_b, const int32_t *d_n_b, int32_t *d_order_b, int k,
                     cudaStream_t stream) {
  ORCA_CHECK_ARG(d_nbr_a && d_order_a && d_nbr_b && d_order_b && k >= 1 && k <= ORCA_MAX_K && n_cap_a >= 0 &&
                 n_cap_b >= 0);
  ORCA_CUDA(launch_dep(row_order_kernel, 2, 1024, 0, stream, d_nbr_a, (int)n_cap_a, d_n_a, d_order_a, d_nbr_b,
                       (int)n_cap_b, d_n_b, d_order_b, (int)k));
  ORCA_COUNT_LAUNCH();
  ORCA_LAUNCH_CHECK();
  return ORCA_OK;
}

}  // namespace orca

using namespace orca;

extern "C" int orca_attn_gather(const float *d_qt, const float *d_nbr_table, const float *d_edge_table,
                                const float *d_time_w, const int32_t *d_nbr, const int32_t *d_eid,
                                const float *d_delta, int32_t k, int32_t n_rows_cap,
                                const int32_t *d_n_rows, float *d_ctx, uint8_t *d_valid,
                                int32_t *d_status, void *stream) {
  Ctx *c = cur();
  if (c == nullptr) return set_error(ORCA_E_CUDA, "orca_attn_gather: no context for the current device");
  return launch_attn_gather(d_qt, d_nbr_table, d_edge_table, d_time_w, d_nbr, d_eid, d_delta, k, n_rows_cap,
                            d_n_rows, 0, nullptr, d_ctx, false, d_valid, c->d_words + CTX_TICKET_MAIN, (cudaStream_t)stream, nullptr, 0,
                            nullptr, d_status);
}
