// What the tcgen05 GEMM kernels share: PTX wrappers (TMA tiles, TMEM, MMA, clusters), descriptors, activation arithmetic of
// the epilogues.
#pragma once

#include "planmoe.h"
#include "kernels/common.cuh"

#include <cuda.h>

namespace planmoe {
namespace {

constexpr int BM = 128, BN = 256, BK = 64;       // BM = accumulator rows per CTA (TMEM lanes)
constexpr int UMMA_K = 16;

// ---------------------------------------------------------------------------------------------
// PTX wrappers
// ---------------------------------------------------------------------------------------------
// TMA load into this CTA's shared memory.  `bar` is a shared::cluster address: the CTA's own barrier,
// or (cta_group::2) the barrier of the even CTA of the pair, which collects the bytes of both CTAs.
// No cluster multicast is used anywhere: every CTA fetches its own tiles.
template <int CG>
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0,
                                            int c1, int c2, int c3) {
  if constexpr (CG == 1) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
  } else {
    asm volatile(
        "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
  }
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
template <int CG>
__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t cols) {
  if constexpr (CG == 1)
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(cols) : "memory");
  else
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(cols) : "memory");
}
template <int CG>
__device__ __forceinline__ void tmem_relinquish() {
  if constexpr (CG == 1) asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  else                   asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
template <int CG>
__device__ __forceinline__ void tmem_dealloc(uint32_t addr, uint32_t cols) {
  if constexpr (CG == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
  else                   asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
template <int CG>
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
  if constexpr (CG == 1) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
  }
}
// Arrive on `bar` (a shared::cluster address, possibly in the other CTA of the pair) once every
// tcgen05.mma issued so far by this thread has completed.
template <int CG>
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  if constexpr (CG == 1)
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
  else
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// The same on the barrier at this offset of every CTA of the group.
template <int CG>
__device__ __forceinline__ void umma_commit_group(uint32_t bar) {
  if constexpr (CG == 1)
    umma_commit<1>(bar);
  else
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"((unsigned short)3) : "memory");
}
// One lane of a converged warp.
__device__ __forceinline__ bool elect_one() {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
  return r != 0u;
}
// ---- thread-block cluster helpers (CG = 2) ----
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// shared::cluster address of the same shared-memory location in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t saddr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr) : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
        "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
        "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// Ties the loaded values to the wait in front of it: no arithmetic on them is moved above it.
__device__ __forceinline__ void tmem_ld_ready(uint32_t* v) {
#pragma unroll
  for (int i = 0; i < 32; ++i) asm volatile("" : "+r"(v[i]));
}
__device__ __forceinline__ void epi_bar_sync() {
  asm volatile("bar.sync 1, 256;" ::: "memory");
}

// Shared-memory matrix descriptor, 128-byte swizzle, Blackwell descriptor version 1.
//   bits [0,14) start address >> 4, [16,30) leading byte offset >> 4, [32,46) stride byte offset >> 4,
//   [46,48) version = 1, [61,64) layout = 2 (SWIZZLE_128B).
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// Instruction descriptor for kind::f16 with bf16 inputs and fp32 accumulation:
//   [4,6) D format = 1 (f32), [7,10) A format = 1 (bf16), [10,13) B format = 1 (bf16),
//   [15] A MN-major, [16] B MN-major, [17,23) N >> 3, [24,29) M >> 4.
__host__ __device__ constexpr uint32_t make_idesc(bool a_mn, bool b_mn, int m, int n = BN) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) |
         ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, uint32_t src_smem, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
               ::"l"(map), "r"(src_smem), "r"(c0), "r"(c1), "r"(c2) : "memory");
}

// Bounded mbarrier wait: false on timeout or when another role already aborted.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort, unsigned long long budget_ns,
                                          int* status, int role, int detail) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = global_timer_ns();
  uint32_t spins = 0;
  while (!mbar_try_wait(bar, parity)) {
    if ((++spins & 63u) == 0u) {
      if (*abort) return false;
      if (global_timer_ns() - t0 > budget_ns) {
        *abort = 1;
        report_status(status, kStatusMbarTimeout, role, detail, (int)parity);
        return false;
      }
    }
  }
  return true;
}

__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float ex2_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

using pair_t = unsigned long long;                 // two fp32 values, see common.cuh

__device__ __forceinline__ pair_t rcp_pair(pair_t x) {
  const float2 f = unpair(x);
  return pair_of(rcp_approx(f.x), rcp_approx(f.y));
}
__device__ __forceinline__ pair_t ex2_pair(pair_t x) {
  const float2 f = unpair(x);
  return pair_of(ex2_approx(f.x), ex2_approx(f.y));
}

// Activation value and derivative of two values in one go (they share the transcendental work).  ACT is a compile-time
// constant in the epilogue's inner loops.
//
// GELU: Phi(x) from erf by the Abramowitz-Stegun 7.1.26 rational approximation (|error| < 1.5e-7, far below bf16
// resolution), one exp2 and one approximate reciprocal; exp(-x^2/2) serves Phi and its derivative.  h = (1 - erf(|x| /
// sqrt 2)) / 2 is Phi(-|x|) itself, so that the lower tail keeps its relative accuracy.
template <int ACT>
__device__ __forceinline__ void act_both(pair_t x, pair_t& out, pair_t& deriv) {
  if constexpr (ACT == kActRelu) {
    const float2 f = unpair(x);
    out = pair_of(fmaxf(f.x, 0.f), fmaxf(f.y, 0.f));
    deriv = pair_of(f.x > 0.f ? 1.f : 0.f, f.y > 0.f ? 1.f : 0.f);
  } else if constexpr (ACT == kActGelu) {
    const pair_t e = ex2_pair(mul_pair(mul_pair(x, x), pair_const(-0.72134752044448170f)));
    const pair_t ax = x & 0x7fffffff7fffffffull;
    const pair_t t = rcp_pair(fma_pair(ax, pair_const(0.3275911f * 0.70710678118654752f), pair_const(1.f)));
    pair_t poly = fma_pair(t, pair_const(0.5f * 1.061405429f), pair_const(-0.5f * 1.453152027f));
    poly = fma_pair(poly, t, pair_const(0.5f * 1.421413741f));
    poly = fma_pair(poly, t, pair_const(-0.5f * 0.284496736f));
    poly = fma_pair(poly, t, pair_const(0.5f * 0.254829592f));
    const pair_t h = mul_pair(poly, mul_pair(t, e));
    const float2 fx = unpair(x), lower = unpair(h), upper = unpair(fma_pair(h, pair_const(-1.f), pair_const(1.f)));
    const pair_t cdf = pair_of(fx.x < 0.f ? lower.x : upper.x, fx.y < 0.f ? lower.y : upper.y);
    out = mul_pair(x, cdf);
    deriv = fma_pair(x, mul_pair(e, pair_const(0.3989422804014327f)), cdf);
  } else if constexpr (ACT == kActSilu) {
    const pair_t sg = rcp_pair(add_pair(ex2_pair(mul_pair(x, pair_const(-1.4426950408889634f))), pair_const(1.f)));
    out = mul_pair(x, sg);
    deriv = mul_pair(sg, fma_pair(x, fma_pair(sg, pair_const(-1.f), pair_const(1.f)), pair_const(1.f)));
  } else {
    out = x; deriv = pair_const(1.f);
  }
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

__device__ __forceinline__ uint32_t pack_pair(pair_t v) {
  const float2 f = unpair(v);
  return pack_bf16(f.x, f.y);
}

}  // namespace
}  // namespace planmoe
