// tcgen05 / mbarrier primitives and the bf16 head / tail split, shared by the tensor-core kernels.
#pragma once

#include <cuda_bf16.h>

#include "common.cuh"

namespace orca {
namespace tc {

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// bounded wait (`limit` SM clocks, about a second by default); records the failure if the barrier never
// flipped.  `alive` makes the failure sticky: a thread that gave up once does not wait again, so a
// broken pipeline drains in one limit instead of one time-out per stage.
__device__ __forceinline__ void mbar_wait(uint32_t bar, uint32_t parity, int32_t *status, int where, bool &alive,
                                          long long limit) {
  if (!alive) return;
  if (mbar_try(bar, parity)) return;
  const long long t0 = clock64();
  while (!mbar_try(bar, parity)) {
    if (clock64() - t0 > limit) {
      report(status, ORCA_E_TIMEOUT, where);
      alive = false;
      return;
    }
  }
}
// The last wait for what a thread has in flight itself, before its CTA ends: a thread that gave up on another wait
// (mbar_wait) must not leave a copy behind that would land in the next CTA's shared memory.  Bounded like the others; a
// barrier that has flipped, which is the usual case, costs one look at it.
__device__ __forceinline__ void mbar_settle(uint32_t bar, uint32_t parity) {
  if (mbar_try(bar, parity)) return;
  const long long t0 = clock64();
  while (!mbar_try(bar, parity) && clock64() - t0 < 2000000000ll) {
  }
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
// L2 policy of data that is read once more and never again: its lines go first
__device__ __forceinline__ uint64_t policy_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ void bulk_g2s_hint(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar, uint64_t policy) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar), "l"(policy)
               : "memory");
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// shared-memory matrix descriptor, no swizzle, K-major: 8 rows x 16 bytes form one contiguous
// 128-byte core matrix; `lbo` = bytes between the two 16-byte K chunks of one MMA, `sbo` = bytes
// between consecutive 8-row groups
__device__ __forceinline__ uint64_t make_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3fff);
  d |= (uint64_t)((lbo >> 4) & 0x3fff) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3fff) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version of this architecture
  return d;
}

// One lane of a converged warp.  The MMA loops are run by a whole warp with the instructions themselves under this
// predicate: descriptors and addresses then live in uniform registers.  Issued from a branch that only one lane takes,
// every operand has to be brought there first, and an MMA took 110 to 160 cycles to issue -- longer than to execute (56
// cycles at 96 columns, 88 at 176).
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n.reg .pred q;\nelect.sync _|q, 0xffffffff;\nselp.u32 %0, 1, 0, q;\n}\n" : "=r"(p));
  return p != 0;
}
// D[tmem] (+)= A[smem] . B[smem]^T, K = 16, bf16 inputs, fp32 accumulate
__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// 16 consecutive accumulator columns of this thread's lane (= tile row); complete after tcgen05.wait::ld
__device__ __forceinline__ void tmem_ld16_nowait(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
// main accumulator + cross-term accumulator (`small` columns further): both loads in flight, one wait
__device__ __forceinline__ void tmem_ld16_sum(uint32_t taddr, uint32_t small, float (&v)[16]) {
  uint32_t a[16], b[16];
  tmem_ld16_nowait(taddr, a);
  tmem_ld16_nowait(taddr + small, b);
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(a[i]) + __uint_as_float(b[i]);
}

__device__ __forceinline__ float4 ld_shared_f4(uint32_t saddr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(saddr));
  return v;
}
__device__ __forceinline__ void st_shared_f4(uint32_t saddr, float4 v) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(saddr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
               : "memory");
}

// x ~ head + tail, both bf16 (round to nearest even), for 8 consecutive K elements: one 16-byte chunk
// of the head image and one of the tail image.  Packed conversions (two floats per instruction).
__device__ __forceinline__ uint32_t pack_split(float x0, float x1, uint32_t &lo) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(x0, x1);
  const uint32_t hb = *reinterpret_cast<const uint32_t *>(&h);
  const float r0 = x0 - __uint_as_float(hb << 16);
  const float r1 = x1 - __uint_as_float(hb & 0xffff0000u);
  const __nv_bfloat162 l = __floats2bfloat162_rn(r0, r1);
  lo = *reinterpret_cast<const uint32_t *>(&l);
  return hb;
}
__device__ __forceinline__ void split_chunk(const float4 a, const float4 b, uint4 &hi, uint4 &lo) {
  hi.x = pack_split(a.x, a.y, lo.x);
  hi.y = pack_split(a.z, a.w, lo.y);
  hi.z = pack_split(b.x, b.y, lo.z);
  hi.w = pack_split(b.z, b.w, lo.w);
}

__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint4 v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
               : "memory");
}


// GRU gates of one unit from its four gate sums (r, z, n of the message, n of the memory) and its old memory value
__device__ __forceinline__ float gru_gates(const float4 a, float h_old) {
  const float rg = 1.f / (1.f + expf(-a.x)), z = 1.f / (1.f + expf(-a.y));
  return (1.f - z) * tanhf(a.z + rg * a.w) + z * h_old;
}

}  // namespace tc
}  // namespace orca
