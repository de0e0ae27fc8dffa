// The tensor-core plumbing the convolution kernels share: mbarriers with bounded waits, shared-memory
// matrix descriptors, tcgen05.mma / commit / ld, cp.async.
#pragma once

#include "common.cuh"

namespace ocnn {
namespace {

constexpr unsigned kSpinLimit = 1u << 20;

enum : int { kErrFullWait = 1, kErrEmptyWait = 2, kErrAccumWait = 3, kErrWeightWait = 4 };

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait.  Returns false when the limit ran out or another role already gave up.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                          int* status, int code) {
  for (unsigned it = 0; it < kSpinLimit; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 255u) == 255u && *abort_flag != 0) return false;
  }
  *abort_flag = 1;
  atomicCAS(status, 0, code);
  return false;
}

// K-major, 128-byte-swizzled shared memory matrix descriptor (sm_100 format): start address >> 4
// in bits [0,14), leading byte offset (unused for swizzled K-major, 1) in [16,30), stride byte
// offset = 1024 B between 8-row groups in [32,46), descriptor version 1 in [46,48), layout type
// SWIZZLE_128B = 2 in [61,64).
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr) {
  return (uint64_t)((addr & 0x3ffffu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) |
         (1ull << 46) | (2ull << 61);
}

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                          uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}

// TMEM for a CTA (by one whole warp); its base goes to *holder.  Only a CTA that has its columns lets the stream's next
// kernel in: an allocation waits until enough columns of its SM are free, and a CTA of the next kernel that took them first
// would keep them until this grid has ended, each waiting for the other.
__device__ __forceinline__ void tmem_alloc(uint32_t* holder, uint32_t columns) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(holder)), "r"(columns)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  grid_dependency_trigger();
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]),
                 "=r"(v[6]), "=r"(v[7])
               : "r"(taddr));
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes)
               : "memory");
}

// What a gather thread's rows of every ring stage hold: one bit per row (R of them) and stage, set while
// the thread's piece of the row is zeros.  A missing neighbour's row is then left alone where the stage's
// last occupant was missing too: a zero-filling copy takes the load/store path like any other, and most
// rows are missing (of 27 neighbours, 2.4 to 11 exist per node on the non-empty nodes of a scene, about
// half on a shape's finest level).  128 -> 96 at 192 k non-empty nodes of depth 9: 179 -> 153 us, the U-Net on
// 200 k points 3.79 -> 3.64 ms; what bounds those layers next are the weight tiles (756 of 894 MB read
// from L2).  Levels whose neighbours mostly exist run as before.
template <int R>
struct ZeroRows {
  uint64_t zero = 0;
  // The rows of stage s to copy when `live` have a source; the others hold zeros afterwards.
  __device__ __forceinline__ uint32_t copies(int s, uint32_t live) {
    constexpr uint32_t kAll = (1u << R) - 1u;
    const int at = R * s;
    const uint32_t was = (uint32_t)(zero >> at) & kAll;
    zero ^= (uint64_t)(was ^ (~live & kAll)) << at;
    return live | (~was & kAll);
  }
};
template <int R>
__device__ __forceinline__ uint32_t live_rows(const int (&p)[R]) {
  uint32_t live = 0;
#pragma unroll
  for (int i = 0; i < R; ++i) live |= (uint32_t)(p[i] >= 0) << i;
  return live;
}

// One contiguous copy global -> shared memory, its bytes counted on `bar`.
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
      "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}

}  // namespace
}  // namespace ocnn
