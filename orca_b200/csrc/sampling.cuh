// Device code of the temporal neighbour sampling, shared by the sampling launches and the batch pipelines.
#pragma once

#include "common.cuh"

namespace orca {

// ---------------------------------------------------------------------------------------------
// Sampling.  A group of G lanes (16 when k <= 16, else 32) serves one query.  The lower bound of
// the query time inside the node's time-sorted segment is found by a G-ary search: every round the
// lanes probe G evenly spaced timestamps, a ballot counts how many are smaller than the query time
// and the segment shrinks by a factor G+1, so a hub with millions of interactions needs five or six
// dependent loads instead of twenty-two.  The lanes then copy the k entries in front of the bound.
// ---------------------------------------------------------------------------------------------
template <int G>
__device__ __forceinline__ long long lower_bound_group(const double *__restrict__ ts, long long lo,
                                                       long long hi, double t, int lane,
                                                       unsigned gmask, int gshift) {
  // invariant: every index < lo has ts < t, every index >= hi has ts >= t
  while (hi - lo > G) {
    long long len = hi - lo;
    long long p = lo + (len * (lane + 1)) / (G + 1);
    bool less = ts[p] < t;
    unsigned b = (__ballot_sync(gmask, less) >> gshift) & ((G == 32) ? 0xffffffffu : ((1u << G) - 1u));
    int cnt = __popc(b);  // probes are increasing, so `less` holds for a prefix of the lanes
    long long nlo = cnt > 0 ? lo + (len * cnt) / (G + 1) + 1 : lo;
    long long nhi = cnt < G ? lo + (len * (cnt + 1)) / (G + 1) : hi;
    lo = nlo;
    hi = nhi;
  }
  long long p = lo + lane;
  bool less = (p < hi) && (ts[p] < t);
  unsigned b = (__ballot_sync(gmask, less) >> gshift) & ((G == 32) ? 0xffffffffu : ((1u << G) - 1u));
  return lo + __popc(b);
}

// The largest neighbour and edge id that the caller's tables have rows for (left alone: it reads none).
struct KnownIds {
  uint32_t nbr = 0xffffffffu, edge = 0xffffffffu;
};

// One query: lower bound, copy of the k entries in front of it (right-aligned, zero padded; an id that is not `known` is
// reported and its slot left empty), and --
// optionally -- marking of the sampled neighbours as candidates of the uncached set: the neighbour
// (the padding node 0 for an empty slot) gets its bit in `cand_bitmap` when its cache flag is clear.
// Hub nodes are sampled thousands of times per batch, so the bit is tested first and only the first
// few writers pay for an atomic on the same word; the one writer that flips the bit also appends the id
// to `cand_list` (if given), which lets the finishing kernel skip the scan of the whole bitmap.
template <int G>
__device__ __forceinline__ void sample_query(const int64_t *__restrict__ indptr, const int32_t *__restrict__ adj_nbr,
                                             const int32_t *__restrict__ adj_eid, const double *__restrict__ adj_ts,
                                             int64_t n_nodes, KnownIds known, int node, double t, int q, int k, int lane,
                                             unsigned gmask, int gshift, int32_t *__restrict__ o_nbr,
                                             int32_t *__restrict__ o_eid, float *__restrict__ o_et,
                                             float *__restrict__ o_dt, int32_t *status,
                                             const uint8_t *__restrict__ cache_flag, uint32_t *__restrict__ cand_bitmap,
                                             int32_t *__restrict__ cand_count, int32_t *__restrict__ cand_list,
                                             const unsigned long long *__restrict__ last_pos = nullptr,
                                             unsigned long long base = 0) {
  long long beg = 0, end = 0;
  if (node >= 0 && node < n_nodes) {
    beg = indptr[node];
    end = indptr[node + 1];
  } else {
    report(status, ORCA_E_BOUNDS, q);
  }
  const long long bound = lower_bound_group<G>(adj_ts, beg, end, t, lane, gmask, gshift);
  if (lane < k) {
    const long long src = bound - k + lane;
    int nb = 0, ei = 0;
    float et = 0.f;
    if (src >= beg) {
      nb = adj_nbr[src];
      ei = adj_eid[src];
      et = (float)adj_ts[src];
      if ((uint32_t)nb > known.nbr || (uint32_t)ei > known.edge) {
        report(status, ORCA_E_BOUNDS, q);
        nb = ei = 0;
        et = 0.f;
      }
    }
    const size_t o = (size_t)q * k + lane;
    o_nbr[o] = nb;
    o_eid[o] = ei;
    if (o_et) o_et[o] = et;
    if (o_dt) o_dt[o] = (float)(t - (double)et);
    // (with `last_pos`: a neighbour whose record already carries this batch's epoch is a row of the
    // batch and can be skipped; rows recorded later than this test slip through and are removed by the
    // finishing kernel, which sees all records)
    if (cand_bitmap != nullptr && cache_flag[nb] == 0 && (last_pos == nullptr || __ldcg(&last_pos[nb]) < base)) {
      const uint32_t bit = 1u << (nb & 31);
      if ((__ldcg(&cand_bitmap[nb >> 5]) & bit) == 0) {
        const uint32_t old = atomicOr(&cand_bitmap[nb >> 5], bit);
        if (cand_list != nullptr && (old & bit) == 0) {
          const int pos = atomicAdd(cand_count, 1);
          if (pos < ORCA_CAND_CAP) cand_list[pos] = nb;
        }
      }
    }
  }
}

}  // namespace orca
