// Shared helpers of the orca_b200 kernels: error reporting, launch checks, small device utilities.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "../../include/orca_b200.h"

namespace orca {

constexpr int D = ORCA_DIM;          // 172 floats = 688 bytes = 43 x 16 bytes
constexpr int H = ORCA_HEADS;        // 2
constexpr int KEY = ORCA_KEY_DIM;    // 516
constexpr int QT = ORCA_QT_DIM;      // 1032
constexpr int QT_LD = ORCA_QT_LD;    // 1056: head h of a projected query starts at h * 528
constexpr int QT_HEAD = QT_LD / H;   // 528
constexpr int OWN_LD = 192;          // floats a row of the own features' part of the merger's hidden layer (172 used; whole lines)
constexpr int MSG = ORCA_MSG_DIM;    // 688
constexpr int ROW_BYTES = D * 4;     // 688

// status word layout (int32[4]): [0] first error code, [1] rows at layer 1, [2] unique positives,
// [3] detail of the error (row / id)
int set_error(int code, const char *fmt, ...);

#define ORCA_CHECK_ARG(cond)                                                        \
  do {                                                                              \
    if (!(cond)) return orca::set_error(ORCA_E_BADARG, "%s: bad argument: %s", __func__, #cond); \
  } while (0)

#define ORCA_CUDA(call)                                                             \
  do {                                                                              \
    cudaError_t e_ = (call);                                                        \
    if (e_ != cudaSuccess)                                                          \
      return orca::set_error(ORCA_E_CUDA, "%s: %s failed: %s", __func__, #call,     \
                             cudaGetErrorString(e_));                               \
  } while (0)

#define ORCA_LAUNCH_CHECK()                                                         \
  do {                                                                              \
    cudaError_t e_ = cudaGetLastError();                                            \
    if (e_ != cudaSuccess)                                                          \
      return orca::set_error(ORCA_E_CUDA, "%s: kernel launch failed: %s", __func__, \
                             cudaGetErrorString(e_));                               \
  } while (0)

// number of kernels launched by this thread since the counter was last reset
int &launch_counter();
#define ORCA_COUNT_LAUNCH() (++orca::launch_counter())

// Programmatic dependent launch: a kernel launched through launch_dep() may begin (block scheduling,
// set-up that touches nothing an earlier kernel wrote) while its predecessor in the stream is still
// draining.  EVERY such kernel calls dep_wait() before its first access to memory another kernel
// produced -- and before returning, even when it has nothing to do, so that completion stays
// transitive along the stream -- and dep_trigger() as early as it likes.  Both are no-ops in a kernel
// that was launched the plain way.
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dep_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
bool dependent_launch_enabled();   // switch of the context in effect (context.cuh)
template <typename... KArgs, typename... Args>
inline cudaError_t launch_dep(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                              Args &&...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  int n = 0;
  if (dependent_launch_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}

__device__ __forceinline__ int rows_of(int cap, const int32_t *d_n) {
  if (d_n == nullptr) return cap;
  int n = *d_n;
  return n < cap ? n : cap;
}

__device__ __forceinline__ void report(int32_t *status, int code, int detail) {
  if (status != nullptr && atomicCAS(status, 0, code) == 0) status[3] = detail;
}

// torch's relu: a value that is not a number stays one (fmaxf would make it 0, and what follows plausible)
__device__ __forceinline__ float relu(float x) {
  float y;
  asm("max.NaN.f32 %0, %1, 0f00000000;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// cos(x) for an fp32 argument of any magnitude, accurate to about 1e-6 absolute.
// The arguments here are delta * w with delta up to 3e8 seconds and w down from 1, so many of them are
// far outside the range where cosf() stays on its fast path, and its slow path (Payne-Hanek) costs a
// hundred instructions; double-precision reduction is no way out either (the fp64 and conversion
// pipes of this GPU made a warp-wide cosine cost ~160 cycles).  fp32 and integer pipes only:
//   |x| < 2^24   Cody-Waite: k = rint(x / 2pi) (< 2^22) by adding and subtracting 1.5 * 2^23, r = x - k*C1 - k*C2 with C1 the
//                nearest float to 2pi: its last bit is 2^-21, so x - k*C1 has at most 24 bits and is exact; reduction error
//                1.3e-7 at most.  1/2pi is a float, too: k can be one off, and |r| reaches 3.15 / 3.23 / 3.48 / 3.82 below
//                2^17 / 2^21 / 2^23 / 2^24;
//   |x| < 2^30   fixed point: x = m * 2^e with a 24-bit m; the fraction of x / 2pi is the low part of
//                m * F (F = 2^64 / 2pi) shifted by e, of which the top 32 bits are kept (96-bit product
//                from two 32 x 32 multiplies); cos is even, so |fraction| (24 bits) goes back to a
//                float through the 2^23 exponent trick; reduction error 3.8e-7 at most, 1.3e-7 rms;
//   else         cosf().
// The hardware cosine approximation is applied to the remainder.  CUDA states its error for [-pi, pi] only (2^-21.19);
// measured against 64 bits over every float: 4.0e-7 at most up to pi, 2.2e-7 up to 3.5, 4.0e-7 up to 4.
// So what decides is the error of the whole, over every float of a binade: Cody-Waite 4.9e-7 at most and 1.3e-7 rms below
// 2^24; fixed point 7.1e-7 at most, 2.1e-7 rms, up to 2^24.
constexpr float COS_SMALL = 16777216.f;    // 2^24
// |x| < COS_SMALL, branch free
__device__ __forceinline__ float cos_small(float x) {
  const float ax = fabsf(x);
  const float k = fmaf(ax, 0.15915494309189535f, 12582912.f) - 12582912.f;
  float r = fmaf(-k, 6.2831855f, ax);
  r = fmaf(k, 1.7484556e-07f, r);
  return __cosf(r);
}
// 2^-8 <= |x| < 2^30, branch free
__device__ __forceinline__ float cos_fixed(float x) {
  const uint32_t bits = __float_as_uint(fabsf(x));
  const int e = (int)(bits >> 23) - 150;           // |x| = m * 2^e, e in [-31, 6]
  const uint32_t m = (bits & 0x7fffffu) | 0x800000u;
  const unsigned long long a = (unsigned long long)m * 0x9391054aull;   // m * low word of F
  const unsigned long long mid = (a >> 32) + (unsigned long long)m * 0x28be60dbull;
  const uint32_t w0 = (uint32_t)a, w1 = (uint32_t)mid, w2 = (uint32_t)(mid >> 32);
  // top 32 bits of frac(m * F * 2^e / 2^64)
  const uint32_t top = e >= 0 ? __funnelshift_l(w0, w1, e) : __funnelshift_r(w1, w2, -e);
  const int t = (int)top;                          // turns in [-1/2, 1/2) scaled by 2^32
  const uint32_t u = min((uint32_t)(t < 0 ? -t : t) >> 8, 0x7fffffu);
  const float f = __uint_as_float(0x4b000000u | u) - 8388608.f;   // (float)u, exact
  return __cosf(f * 3.7450702829239286e-07f);      // 2pi / 2^24
}
__device__ __forceinline__ float cos_any(float x) {
  const float ax = fabsf(x);
  if (ax < COS_SMALL) return cos_small(x);
  if (ax < 1073741824.f) return cos_fixed(x);
  return cosf(x);
}

static inline int ceil_div(int a, int b) { return (a + b - 1) / b; }

}  // namespace orca
