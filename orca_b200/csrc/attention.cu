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

// One warp per query row.  A row's slots are taken two at a time: their pieces are loaded into registers -- every lane
// owns 16-byte pieces l, l + 32, l + 64 of the gathered [neighbour | edge feature] part and column PAIRS l, l + 32,
// l + 64 of the time-encoding part, which is computed (cos of delta * w) two columns at a time with the packed
// two-wide fp32 instructions of this architecture while the loads are in flight -- then come the partial dot products
// with the two query heads, one cross-lane sum of all four logits at once, a running softmax and the weighted sums, all
// from the same registers.
// What bounds it (48 k rows of ten slots, 165 us; under the profiler 169): the instructions of a row (1800 a warp, a
// third of them the time encodings) against 16 resident warps per SM: issue slots 49 % busy, a warp issues every 8
// cycles (3 of them for loads), DRAM 29 %, L2 25 %, L1 50 %.  Measured against it: two passes over the rows with parked
// logits and time encodings (the form before) 178 us; four slots a step at 12 warps 186; slots copied ahead with
// cp.async, two or four at a time, 167 to 201; the long cosine inlined with a variant of the loop per range, 360
// (instruction cache).  A launch of a single batch is no faster than the two passes were (6000 rows 29.2 us, before
// 28.9): there the two or three rows of each warp, one after the other, are what it takes.  The 688-byte rows are not moved by cp.async.bulk: an SM retires only
// about one small bulk copy per ~130 cycles.
//
// Work distribution.  Rows differ tenfold in cost (0 to k valid slots) and a launch of a single batch holds only two
// to three rows per resident warp, so WHO gets WHICH row decides the length of the launch:
//   - rows are handed out by ticket (one atomic per row on a counter the launch leaves at zero again);
//   - tickets walk the rows in the order of `order` (rows sorted by falling number of valid slots,
//     made by row_order_kernel beside the sampling), so that the launch ends on its lightest rows.
// A warp draws its next ticket when it starts a row and reads it after the row's first slots; the indices of the next
// row are loaded while the rest of the row is worked on.  No block-level synchronisation, no shared memory.
constexpr int GA_THREADS = 64, GA_BLOCKS = 8;    // 16 warps per SM at 128 registers
constexpr int GS = 2;                           // slots per step
constexpr int GA_MEM_F4 = 2 * D / 4;            // 86 sixteen-byte pieces of [neighbour | edge feature]
constexpr int GA_ROW_F4 = D / 4;                // 43 pieces per table row
constexpr int GA_P_ITERS = 3;                   // pieces / time-column pairs per lane (the third for lanes 0..21)

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 dup2(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 lo2(const float4 &v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4 &v) { return make_float2(v.z, v.w); }

// cos of two arguments below COS_SMALL at once: the Cody-Waite reduction of cos_small in packed arithmetic;
// the nearest integer of x / 2pi comes from adding and subtracting 1.5 * 2^23
__device__ __forceinline__ float2 cos_small2(float2 x) {
  const float2 t = mul2(x, dup2(0.15915494309189535f));
  const float2 kk = add2(add2(t, dup2(12582912.f)), dup2(-12582912.f));
  float2 r = fma2(kk, dup2(-6.28125f), x);
  r = fma2(kk, dup2(-0.0019350051879882812f), r);
  r = fma2(kk, dup2(-3.019916050561733e-07f), r);
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
// tables are right-aligned (padding first), so a row's count is k minus the position of its first neighbour.
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
  auto count = [&](int r) {
    const int32_t *row = nbr + (size_t)r * k;
    int c = 0;
    for (int j = 0; j < k; ++j) c += row[j] != 0 ? 1 : 0;
    return c;
  };
  for (int r = tid; r < n; r += 1024) atomicAdd(&s_bin[count(r)], 1);
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
  for (int r = tid; r < n; r += 1024) order[atomicAdd(&s_bin[count(r)], 1)] = r;
}

// Loads one slot's pieces of this lane: piece l of the neighbour row; piece l + 32 of the concatenation (neighbour row
// for l < 11, else edge row piece l - 11); piece l + 64 (edge row piece l + 21, l < 22; the other lanes re-read piece 0
// of the edge row, which is never used).
struct SlotRows {
  const float4 *n0, *n1;
  int at1, at2, split;
  bool from_edge;
  const float4 *e_tab;
  __device__ __forceinline__ void load(int nb, int ei, int lane, float4 (&x)[3]) const {
    const float4 *nrow = (nb >= split ? n1 : n0) + (size_t)nb * GA_ROW_F4;
    const float4 *erow = e_tab + (size_t)ei * GA_ROW_F4;
    x[0] = __ldg(nrow + lane);
    x[1] = __ldg((from_edge ? erow : nrow) + at1);
    x[2] = __ldg(erow + at2);
  }
};

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

template <bool IMAGE>
__global__ void __launch_bounds__(GA_THREADS, GA_BLOCKS)
attn_gather_kernel(const float *__restrict__ qt, const float *__restrict__ nbr_table,
                   const float *__restrict__ nbr_table2, int nbr_split,
                   const float *__restrict__ edge_table, const float *__restrict__ time_w,
                   const int32_t *__restrict__ nbr, const int32_t *__restrict__ eid,
                   const float *__restrict__ delta, int k, int n_cap, const int32_t *__restrict__ d_n,
                   const int32_t *__restrict__ order, void *__restrict__ ctx, uint8_t *__restrict__ valid_out,
                   int32_t *__restrict__ ticket, unsigned long long *__restrict__ prof) {
  constexpr unsigned FULL = 0xffffffffu;
  dep_trigger();
  dep_wait();
  const int n = rows_of(n_cap, d_n);
  const int lane = threadIdx.x & 31;
  const bool third = lane + 64 < GA_MEM_F4;       // lanes 0..21 own a third piece / pair
  // this lane's time-encoding frequencies, as column pairs, and the largest frequency of each pair group
  float2 wt[GA_P_ITERS];
#pragma unroll
  for (int i = 0; i < GA_P_ITERS; ++i)
    wt[i] = (i < 2 || third) ? __ldg(reinterpret_cast<const float2 *>(time_w) + lane + 32 * i) : make_float2(0.f, 0.f);
  const float wg0 = __ldg(time_w), wg1 = __ldg(time_w + 64), wg2 = __ldg(time_w + 128);
  unsigned long long prof_rows = 0, prof_slots = 0;
  SlotRows rows;
  rows.n0 = reinterpret_cast<const float4 *>(nbr_table), rows.n1 = reinterpret_cast<const float4 *>(nbr_table2);
  rows.e_tab = reinterpret_cast<const float4 *>(edge_table);
  rows.from_edge = lane >= GA_ROW_F4 - 32;
  rows.at1 = rows.from_edge ? lane - (GA_ROW_F4 - 32) : lane + 32;
  rows.at2 = third ? lane + 64 - GA_ROW_F4 : 0;
  rows.split = nbr_split;

  // (A group's rows from the last one back: the queries written last are still in L2, and so are the images of the rows
  // that the output kernel starts with.  200 MB of queries a launch do not fit it: 50 batches of 2000 5.80 -> 5.68 ms, 51 of
  // 600 3.00 -> 2.96, without reuse 2.36 -> 2.30.)
  auto row_of_ticket = [&](int t) -> int { return order != nullptr ? order[t] : n - 1 - t; };
  auto load_indices = [&](int r, int &o_nbr, int &o_eid, float &o_dt) {
    o_nbr = 0, o_eid = 0, o_dt = 0.f;
    if (lane < k) {
      const size_t o = (size_t)r * k + lane;
      o_nbr = nbr[o];
      o_eid = eid[o];
      o_dt = delta[o];
    }
  };
  int tkt = 0;
  if (lane == 0) tkt = atomicAdd(&ticket[0], 1);
  tkt = __shfl_sync(FULL, tkt, 0);
  int row = tkt < n ? row_of_ticket(tkt) : -1;
  int my_nbr = 0, my_eid = 0;
  float my_dt = 0.f;
  if (row >= 0) load_indices(row, my_nbr, my_eid, my_dt);
  while (row >= 0) {
    // the next ticket is drawn now and its row's indices are requested after the first slots (see above)
    if (lane == 0) tkt = atomicAdd(&ticket[0], 1);
    int next = -1, nx_nbr = 0, nx_eid = 0;
    float nx_dt = 0.f;
    bool drawn = false;
    auto draw_next = [&]() {
      const int t = __shfl_sync(FULL, tkt, 0);
      if (t < n) {
        next = row_of_ticket(t);
        load_indices(next, nx_nbr, nx_eid, nx_dt);
      }
    };
    const unsigned vmask = __ballot_sync(FULL, my_nbr != 0);
    const int n_valid = __popc(vmask);
    float4 am0[3], am1[3];                         // weighted sums of the gathered part, heads 0 / 1
    float2 at0[GA_P_ITERS], at1[GA_P_ITERS];       // and of the time part
#pragma unroll
    for (int i = 0; i < 3; ++i) am0[i] = am1[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < GA_P_ITERS; ++i) at0[i] = at1[i] = make_float2(0.f, 0.f);
    float inv0 = 0.f, inv1 = 0.f;
    if (n_valid > 0) {
      // which pair groups of this lane's slot need the fixed-point cosine (see time_terms)
      int my_nl;
      {
        const float adt = fabsf(my_dt);
        my_nl = (adt * wg0 >= COS_SMALL ? 1 : 0) + (adt * wg1 >= COS_SMALL ? 1 : 0) + (adt * wg2 >= COS_SMALL ? 1 : 0);
        if (!(adt * wg0 < 1073741824.f)) my_nl = -1;   // beyond the fixed-point range (or not finite)
      }
      const float *q_src = qt + (size_t)row * QT_LD;
      float m = -INFINITY, sum = 0.f;     // running maximum / sum of this lane's head
      unsigned todo = vmask;
      // GS slots at a time, each row of them in registers from its dot products to its weighted sum: nothing is
      // loaded twice, and the cross-lane sums of 2 * GS logits cost little more than those of one
      constexpr int V = 2 * GS, LPV = 32 / V;
      for (int left = n_valid; left > 0; left -= GS) {
        float4 x[GS][3];
        float2 te[GS][GA_P_ITERS];
        int js[GS];
#pragma unroll
        for (int s = 0; s < GS; ++s) {
          const int j = todo ? __ffs(todo) - 1 : -1;
          js[s] = j;
          todo &= todo - 1;
          const int jj = j >= 0 ? j : js[0];      // (an empty place repeats the first slot with weight zero)
          rows.load(__shfl_sync(FULL, my_nbr, jj), __shfl_sync(FULL, my_eid, jj), lane, x[s]);
        }
#pragma unroll
        for (int s = 0; s < GS; ++s) {
          const int jj = js[s] >= 0 ? js[s] : js[0];
          const float dt = __shfl_sync(FULL, my_dt, jj);
          const int nl = __shfl_sync(FULL, my_nl, jj);
          time_terms(dt, nl, wt, te[s]);
        }
        // partial logits: value 2 * s + head
        float2 a0[GS], a1[GS];
#pragma unroll
        for (int s = 0; s < GS; ++s) a0[s] = a1[s] = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < GA_P_ITERS; ++i) {
          if (i < 2 || third) {
            const float4 qa = __ldg(reinterpret_cast<const float4 *>(q_src) + lane + 32 * i);
            const float4 qb = __ldg(reinterpret_cast<const float4 *>(q_src + QT_HEAD) + lane + 32 * i);
            const float2 qta = __ldg(reinterpret_cast<const float2 *>(q_src + 2 * D) + lane + 32 * i);
            const float2 qtb = __ldg(reinterpret_cast<const float2 *>(q_src + QT_HEAD + 2 * D) + lane + 32 * i);
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
        }
        float v[V];
#pragma unroll
        for (int s = 0; s < GS; ++s) v[2 * s] = a0[s].x + a0[s].y, v[2 * s + 1] = a1[s].x + a1[s].y;
        // lane l holds value l / LPV = 2 * slot + head; head = one lane bit
        float lg = warp_sum_many<V>(v, lane);
        const int slot = lane / (2 * LPV);
#pragma unroll
        for (int s = 1; s < GS; ++s)
          if (slot == s && js[s] < 0) lg = -INFINITY;
        float top = lg;
#pragma unroll
        for (int o = 2 * LPV; o < 32; o <<= 1) top = fmaxf(top, __shfl_xor_sync(FULL, top, o));
        const float m_new = fmaxf(m, top);
        const float scale = expf(m - m_new);       // (0 the first time)
        const float p = expf(lg - m_new);
        float ps = p;
#pragma unroll
        for (int o = 2 * LPV; o < 32; o <<= 1) ps += __shfl_xor_sync(FULL, ps, o);
        sum = sum * scale + ps;
        m = m_new;
        const float2 S0 = dup2(__shfl_sync(FULL, scale, 0)), S1 = dup2(__shfl_sync(FULL, scale, LPV));
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
#pragma unroll
        for (int s = 0; s < GS; ++s) {
          const float2 P0 = dup2(__shfl_sync(FULL, p, 2 * s * LPV)), P1 = dup2(__shfl_sync(FULL, p, (2 * s + 1) * LPV));
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
        if (!drawn) {
          // the next row of this warp: its indices land while this one is finished
          drawn = true;
          draw_next();
        }
      }
      inv0 = 1.f / __shfl_sync(FULL, sum, 0), inv1 = 1.f / __shfl_sync(FULL, sum, LPV);
      prof_rows += 1;
      prof_slots += (unsigned long long)n_valid;
    }
    if (!drawn) draw_next();
    // write the row: [head 0: gathered 344 | time 172][head 1: ...].  A row whose slots are all padding has no attention
    // term: the image gets zeros (the fp32 form leaves such a row alone, `valid` says so).
    if (IMAGE || n_valid > 0) {
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const int f = lane + 32 * i;
        if (i < 2 || third) {
          const float4 m0 = make_float4(am0[i].x * inv0, am0[i].y * inv0, am0[i].z * inv0, am0[i].w * inv0);
          const float4 m1 = make_float4(am1[i].x * inv1, am1[i].y * inv1, am1[i].z * inv1, am1[i].w * inv1);
          const float2 t0 = make_float2(at0[i].x * inv0, at0[i].y * inv0);
          const float2 t1 = make_float2(at1[i].x * inv1, at1[i].y * inv1);
          if (IMAGE) {
            char *im = (char *)ctx;
            img::put4<img::CTX_STAGES>(im, row, 4 * f, m0);
            img::put4<img::CTX_STAGES>(im, row, KEY + 4 * f, m1);
            img::put2<img::CTX_STAGES>(im, row, 2 * D + 2 * f, t0);
            img::put2<img::CTX_STAGES>(im, row, KEY + 2 * D + 2 * f, t1);
          } else {
            float *out = (float *)ctx + (size_t)row * QT;
            reinterpret_cast<float4 *>(out)[f] = m0;
            reinterpret_cast<float4 *>(out + KEY)[f] = m1;
            reinterpret_cast<float2 *>(out + 2 * D)[f] = t0;
            reinterpret_cast<float2 *>(out + KEY + 2 * D)[f] = t1;
          }
        }
      }
    }
    if (IMAGE && lane < (img::CTX_STAGES * img::STAGE_K - QT) / 4)    // padding
      img::put4<img::CTX_STAGES>((char *)ctx, row, QT + 4 * lane, make_float4(0.f, 0.f, 0.f, 0.f));
    if (lane == 0) valid_out[row] = n_valid > 0 ? 1 : 0;
    row = next;
    my_nbr = nx_nbr;
    my_eid = nx_eid;
    my_dt = nx_dt;
  }
  if (lane == 0) {
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
// `ticket`: two zeroed device words that the launch leaves at zero; launches that may overlap on the GPU
// need words of their own
int launch_attn_gather(const float *d_qt, const float *d_nbr_table, const float *d_edge_table,
                       const float *d_time_w, const int32_t *d_nbr, const int32_t *d_eid, const float *d_delta,
                       int k, int n_rows_cap, const int32_t *d_n_rows, int rows_hint, const int32_t *d_order,
                       void *d_ctx, bool image, uint8_t *d_valid, int32_t *d_ticket, cudaStream_t stream,
                       const float *d_nbr_table2, int nbr_split) {
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
  // one resident wave at most; fewer blocks when the caller expects fewer rows than the capacity
  const int rows = rows_hint > 0 ? std::min(rows_hint, n_rows_cap) : n_rows_cap;
  const int grid = std::min(ceil_div(rows, GA_THREADS / 32), c->sm_count * GA_BLOCKS);
  auto kernel = image ? attn_gather_kernel<true> : attn_gather_kernel<false>;
  // (the profiling events would sit between this kernel and its neighbours: plain launch then)
  if (pf.on)
    kernel<<<grid, GA_THREADS, 0, stream>>>(d_qt, d_nbr_table, d_nbr_table2, nbr_split, d_edge_table, d_time_w, d_nbr, d_eid,
                                            d_delta, k, n_rows_cap, d_n_rows, d_order, d_ctx, d_valid, d_ticket,
                                            pf.d_counters);
  else
    ORCA_CUDA(launch_dep(kernel, grid, GA_THREADS, 0, stream, d_qt, d_nbr_table, d_nbr_table2, nbr_split, d_edge_table,
                         d_time_w, d_nbr, d_eid, d_delta, (int)k, (int)n_rows_cap, d_n_rows, d_order, d_ctx, d_valid,
                         d_ticket, (unsigned long long *)nullptr));
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
  (void)d_status;
  Ctx *c = cur();
  if (c == nullptr) return set_error(ORCA_E_CUDA, "orca_attn_gather: no context for the current device");
  return launch_attn_gather(d_qt, d_nbr_table, d_edge_table, d_time_w, d_nbr, d_eid, d_delta, k, n_rows_cap,
                            d_n_rows, 0, nullptr, d_ctx, false, d_valid, c->d_words + CTX_TICKET_MAIN, (cudaStream_t)stream);
}
