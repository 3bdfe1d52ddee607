// Link-prediction metrics of every batch of a scored stream (evaluation/evaluation.py:30-44): average precision,
// area under the ROC curve and the share of edges whose positive score is not below the negative one's.
//
// Host form: the scores have just arrived on the host, and a batch is a few hundred to a few thousand numbers.  Both
// metrics only need the counts of positives and negatives at or above every distinct score, so the two sides are
// sorted on their own (radix sort of the order-preserving 32-bit keys) and merged once.  40 batches of 200 edges
// take 0.44 ms on one core; scikit-learn's three calls per batch took 75 ms for the same (argument checks and
// temporaries, not arithmetic).  Batches are dealt out to a few threads when there is work for more than one.
//
// Scores that are still on the device are evaluated there, behind the scores of their group (launch_link_metrics): no
// sort, every score is compared with all scores of its batch.  Up to 4096 edges a batch, whose keys fit a block's static
// shared memory.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "host_threads.cuh"

namespace orca {
namespace metrics {

// unsigned key that falls as the score rises (-0.0 and +0.0 equal): ascending keys = descending scores
static inline uint32_t falling_key(float x) {
  uint32_t u;
  x += 0.f;
  memcpy(&u, &x, 4);
  return (u >> 31) ? u : ~(u | 0x80000000u);
}

struct Scratch {
  std::vector<uint32_t> pos, neg, tmp;
  uint32_t count[3][2048];
};

static void sort_keys(std::vector<uint32_t> &v, Scratch &s) {
  std::vector<uint32_t> &tmp = s.tmp;
  uint32_t (&count)[3][2048] = s.count;
  const size_t n = v.size();
  if (n < 128) {   // (three passes over 2048 counters cost more than the comparisons)
    std::sort(v.begin(), v.end());
    return;
  }
  tmp.resize(n);
  memset(count, 0, sizeof(count));
  for (uint32_t k : v) ++count[0][k & 2047], ++count[1][(k >> 11) & 2047], ++count[2][k >> 22];
  for (int p = 0; p < 3; ++p) {
    uint32_t at = 0;
    for (uint32_t &c : count[p]) {
      const uint32_t m = c;
      c = at;
      at += m;
    }
    const int shift = 11 * p;
    for (uint32_t k : v) tmp[count[p][(k >> shift) & 2047]++] = k;
    v.swap(tmp);
  }
}

// false: a score is not finite
static bool one_batch(const float *pos, const float *neg, int64_t n, double *out, Scratch &s) {
  s.pos.resize(n);
  s.neg.resize(n);
  int64_t wins = 0;
  bool finite = true;
  for (int64_t i = 0; i < n; ++i) {
    finite = finite && isfinite(pos[i]) && isfinite(neg[i]);
    wins += pos[i] >= neg[i] ? 1 : 0;
    s.pos[i] = falling_key(pos[i]);
    s.neg[i] = falling_key(neg[i]);
  }
  if (!finite) return false;
  sort_keys(s.pos, s);
  sort_keys(s.neg, s);
  double ap = 0, twice_area = 0;   // (counts are whole numbers: the area is exact up to 2^53)
  int64_t tp = 0, fp = 0;
  while (tp < n || fp < n) {
    uint32_t key = 0xffffffffu;
    if (tp < n) key = s.pos[tp];
    if (fp < n) key = std::min(key, s.neg[fp]);
    int64_t t = tp, f = fp;
    while (t < n && s.pos[t] == key) ++t;
    while (f < n && s.neg[f] == key) ++f;
    if (t > tp) ap += (double)(t - tp) * ((double)t / (double)(t + f));
    twice_area += (double)(f - fp) * (double)(t + tp);
    tp = t;
    fp = f;
  }
  out[0] = ap / (double)n;
  out[1] = twice_area / (2.0 * (double)n * (double)n);
  out[2] = (double)wins / (double)n;
  return true;
}

// Sums over a part of a batch (PART edges): precisions of its positives, for its negatives the positives above and twice
// counted ties, edges whose positive is not below the negative, scores that are not finite.
constexpr int PART = 256, MOST_EDGES = 4096;
__device__ __forceinline__ uint32_t device_key(float x) {
  const uint32_t u = __float_as_uint(x + 0.f);
  return (u >> 31) ? u : ~(u | 0x80000000u);
}
// Blocks (part, batch).  Eight instructions a pair of edges: 8 batches of 2000 take 22 us on the 64 SMs that they use, 40
// of 200 take 5.
__global__ void __launch_bounds__(PART) link_metrics_kernel(const float *__restrict__ prob, int nb, int bs, int b_last,
                                                            double *__restrict__ out) {
  __shared__ __align__(16) uint32_t s_pos[MOST_EDGES], s_neg[MOST_EDGES];
  dep_trigger();
  dep_wait();
  const int b = blockIdx.y, n = b == nb - 1 ? b_last : bs, tid = threadIdx.x, i = blockIdx.x * PART + tid;
  const float *pos = prob + (size_t)b * 2 * bs, *neg = pos + n;
  const int padded = (n + 3) & ~3;
  for (int j = tid; j < padded; j += PART) {     // (padding: below every score)
    s_pos[j] = j < n ? device_key(pos[j]) : 0xffffffffu;
    s_neg[j] = j < n ? device_key(neg[j]) : 0xffffffffu;
  }
  __syncthreads();
  double ap = 0, area = 0;
  int wins = 0, bad = 0;
  if (i < n) {
    const uint32_t p = s_pos[i], q = s_neg[i];
    int tp = 0, fp = 0, above = 0, level = 0;    // (a smaller key is a higher score)
    for (int j = 0; j < padded; j += 4) {
      const uint4 x = *reinterpret_cast<const uint4 *>(s_pos + j), y = *reinterpret_cast<const uint4 *>(s_neg + j);
      tp += (x.x <= p) + (x.y <= p) + (x.z <= p) + (x.w <= p);
      fp += (y.x <= p) + (y.y <= p) + (y.z <= p) + (y.w <= p);
      above += (x.x < q) + (x.y < q) + (x.z < q) + (x.w < q);
      level += (x.x <= q) + (x.y <= q) + (x.z <= q) + (x.w <= q);
    }
    const float a = pos[i], c = neg[i];
    ap = (double)tp / (double)(tp + fp);
    area = (double)(above + level);
    wins = a >= c ? 1 : 0;
    bad = isfinite(a) && isfinite(c) ? 0 : 1;
  }
  __shared__ double s_sum[PART / 32][4];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ap += __shfl_xor_sync(0xffffffffu, ap, o);
    area += __shfl_xor_sync(0xffffffffu, area, o);
  }
  wins = __reduce_add_sync(0xffffffffu, wins);
  bad = __reduce_add_sync(0xffffffffu, bad);
  if ((tid & 31) == 0) s_sum[tid >> 5][0] = ap, s_sum[tid >> 5][1] = area, s_sum[tid >> 5][2] = wins, s_sum[tid >> 5][3] = bad;
  __syncthreads();
  if (tid < 4) {
    double sum = 0;
    for (int w = 0; w < PART / 32; ++w) sum += s_sum[w][tid];
    out[((size_t)b * gridDim.x + blockIdx.x) * 4 + tid] = sum;
  }
}

}  // namespace metrics

int launch_link_metrics(const float *d_prob, int nb, int bs, int b_last, double *d_out, cudaStream_t s) {
  ORCA_CUDA(launch_dep(metrics::link_metrics_kernel, dim3(orca_link_metric_parts(bs), nb), metrics::PART, 0, s, d_prob, nb, bs,
                       b_last, d_out));
  ORCA_COUNT_LAUNCH();
  ORCA_LAUNCH_CHECK();
  return ORCA_OK;
}
}  // namespace orca

using namespace orca;

extern "C" int orca_link_metrics(const float *h_pos, const float *h_neg, int64_t n_edges, int32_t bs, double *h_out) {
  ORCA_CHECK_ARG(h_pos && h_neg && h_out && n_edges >= 0 && bs > 0);
  const int64_t nb = (n_edges + bs - 1) / bs;
  // a thread is worth starting for about 64 k scores (a millisecond); at most eight
  constexpr int MOST = 8;
  const int want = (int)std::min<int64_t>({MOST, nb, 1 + n_edges / 65536, (int64_t)std::max(1u, std::thread::hardware_concurrency())});
  int64_t bad[MOST];
  auto work = [&](int t) {
    bad[t] = -1;
    metrics::Scratch s;
    for (int64_t i = t; i < nb; i += want) {
      const int64_t lo = i * bs, n = std::min<int64_t>(bs, n_edges - lo);
      if (!metrics::one_batch(h_pos + lo, h_neg + lo, n, h_out + 3 * i, s) && bad[t] < 0) bad[t] = i;
    }
  };
  const int rc = on_threads(want, work, "orca_link_metrics");
  if (rc) return rc;
  for (int t = 0; t < want; ++t)
    if (bad[t] >= 0) return set_error(ORCA_E_BADARG, "orca_link_metrics: a score of batch %lld is not finite", (long long)bad[t]);
  return ORCA_OK;
}

extern "C" int32_t orca_link_metric_parts(int32_t bs) {
  return bs > 0 && bs <= metrics::MOST_EDGES ? ceil_div(bs, metrics::PART) : 0;
}

extern "C" int orca_link_metrics_of_parts(const double *h_parts, int64_t n_edges, int32_t bs, double *h_out) {
  ORCA_CHECK_ARG(h_parts && h_out && n_edges >= 0 && orca_link_metric_parts(bs) > 0);
  const int parts = orca_link_metric_parts(bs);
  for (int64_t lo = 0, i = 0; lo < n_edges; lo += bs, ++i) {
    const double n = (double)std::min<int64_t>(bs, n_edges - lo);
    double sum[4] = {0, 0, 0, 0};
    for (int p = 0; p < parts; ++p)
      for (int c = 0; c < 4; ++c) sum[c] += h_parts[(i * parts + p) * 4 + c];
    if (sum[3] != 0) return set_error(ORCA_E_BADARG, "orca_link_metrics: a score of batch %lld is not finite", (long long)i);
    h_out[3 * i] = sum[0] / n, h_out[3 * i + 1] = sum[1] / (2.0 * n * n), h_out[3 * i + 2] = sum[2] / n;
  }
  return ORCA_OK;
}
