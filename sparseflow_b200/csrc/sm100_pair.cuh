// Inline-PTX wrappers for CTA pairs (tcgen05 cta_group::2, TMA copies that signal the pair's even CTA) and the register
// helpers of their accumulator drain, shared by the kernels that run on SM pairs.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels.h"
#include "sm100_ptx.cuh"

namespace sfb200 {

// ---------------------------------------------------------------- cluster / pair PTX
// Arrive on a barrier of the pair's even CTA.  Default semantics (release at CTA scope) on purpose:
// a cluster-scope release would hold the arrive back until this thread's global stores of the
// previous tile have reached L2, and the arrive only has to order tensor-memory reads, which
// tcgen05.wait::ld + tcgen05.fence::before_thread_sync already do.
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// Pair forms: the copy lands in this CTA's shared memory, the byte count is credited to the
// barrier of the even CTA of the pair.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* m, int x, int y,
                                                 uint32_t leader_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(x), "r"(y), "r"(leader_bar)
      : "memory");
}
// L2 eviction policies: outputs are written once and never read by this kernel (evict first, so
// they do not push operand tiles out of L2); the token operand is re-read by every row block
// (evict last).
__device__ __forceinline__ uint64_t l2_policy_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t l2_policy_evict_last() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ void tma_load_2d_pair_hint(uint32_t dst, const CUtensorMap* m, int x, int y,
                                                      uint32_t leader_bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint "
      "[%0], [%1, {%2, %3}], [%4], %5;" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(x), "r"(y), "r"(leader_bar), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void tma_load_1d_pair(uint32_t dst, const CUtensorMap* m, int x,
                                                 uint32_t leader_bar) {
  asm volatile(
      "cp.async.bulk.tensor.1d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2}], [%3];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(x), "r"(leader_bar)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_result),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
// Arrive on the barrier at the same shared-memory offset in both CTAs of the pair once every
// tcgen05 operation issued so far by this thread has completed.
// `mask`: the cluster ranks of the two CTAs (a cluster of one pair: ranks 0 and 1).
__device__ __forceinline__ void tc_commit_pair(uint32_t bar, uint16_t mask = 3) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 "
      "[%0], %1;" ::"r"(bar),
      "h"(mask)
      : "memory");
}
__device__ __forceinline__ void tc_cp_128x128b_pair(uint32_t taddr, uint64_t sdesc) {
  asm volatile("tcgen05.cp.cta_group::2.128x128b [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
}
__device__ __forceinline__ void tc_mma_sp_f16_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc,
                                                   uint32_t e_tmem, uint32_t idesc,
                                                   uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "tcgen05.mma.sp.cta_group::2.kind::f16 [%0], %1, %2, [%3], %4, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(e_tmem), "r"(idesc), "r"(accumulate)
      : "memory");
}

// ---------------------------------------------------------------- accumulator drain
__device__ __forceinline__ float act_fn(float v, int act) {
  switch (act) {
    case kActRelu: return fmaxf(v, 0.f);
    case kActSilu: return v * __fdividef(1.f, 1.f + __expf(-v));
    case kActGelu: return 0.5f * v * (1.f + erff(v * 0.70710678118654752f));
    default: return v;
  }
}
__device__ __forceinline__ float bias_at(const void* bias, int o, int fmt) {
  const uint16_t b = static_cast<const uint16_t*>(bias)[o];
  if (fmt == 1) return __uint_as_float(static_cast<uint32_t>(b) << 16);
  return __half2float(__ushort_as_half(b));
}
// 16 lanes x 16 columns: thread l gets, for repetition n (8 columns each), r[4n], r[4n+1] =
// (lane l/4, columns 8n + 2(l%4), +1) and r[4n+2], r[4n+3] = (lane l/4 + 8, same columns): the
// accumulator-fragment layout of warp-level MMA, which stmatrix can transpose.  Two repetitions: 8 registers.
__device__ __forceinline__ void tmem_ld_16x256b_x2(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
// 32 lanes x 16 columns of fp32: thread i = lane base + i, one register per column
__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, uint32_t r0, uint32_t r1, uint32_t r2,
                                                  uint32_t r3) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr),
               "r"(r0), "r"(r1), "r"(r2), "r"(r3)
               : "memory");
}
__device__ __forceinline__ uint32_t pack16(float a, float b, int fmt) {
  if (fmt == 1) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
  }
  const __half2 v = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float silu_mul(uint32_t g, uint32_t u) {
  const float gf = __uint_as_float(g);
  return (gf * __fdividef(1.f, 1.f + __expf(-gf))) * __uint_as_float(u);
}

__device__ __forceinline__ float silu_mul_bias(uint32_t g, uint32_t u, float bias_g, float bias_u) {
  const float gf = __uint_as_float(g) + bias_g;
  return (gf * __fdividef(1.f, 1.f + __expf(-gf))) * (__uint_as_float(u) + bias_u);
}
// SiLU.mul epilogue: bias of gate features f = row_w / 2 + g, f + 8 (b0, b1) and of the matching up features (b2, b3), for a
// warp whose 32 interleaved rows start at row_w.  Either bias may be null.
__device__ __forceinline__ void load_gate_up_bias(const void* gate, const void* up, int row_w, int g, int n_out, int fmt, float& b0,
                                                  float& b1, float& b2, float& b3) {
  const int f = row_w / 2 + g;
  if (row_w >= n_out) return;      // whole blocks of 32 rows
  if (gate != nullptr) {
    b0 = bias_at(gate, f, fmt);
    b1 = bias_at(gate, f + 8, fmt);
  }
  if (up != nullptr) {
    b2 = bias_at(up, f, fmt);
    b3 = bias_at(up, f + 8, fmt);
  }
}
}  // namespace sfb200
