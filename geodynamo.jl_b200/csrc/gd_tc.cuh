// gd_tc.cuh -- sm_100a tensor-core primitives used by the mixed-precision
// Legendre kernels: tcgen05 MMA (kind::tf32) with FP32 accumulators in tensor
// memory, shared-memory matrix descriptors for K-major SWIZZLE_128B tiles,
// mbarrier waits with a clock bound, TF32 splitting.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace gd {
namespace tc {

// Byte offset of element (row, k) of a K-major SWIZZLE_128B tile whose rows are
// 128 bytes (32 four-byte elements): 8-row atoms of 1024 bytes, 16-byte chunk
// index XOR-ed with row % 8.  The tile base must be 1024-byte aligned.
__host__ __device__ __forceinline__ uint32_t sw128_offset(uint32_t row, uint32_t k) {
  return (row >> 3) * 1024u + (row & 7u) * 128u + ((((k >> 2) ^ (row & 7u)) & 7u) << 4) + (k & 3u) * 4u;
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Shared-memory matrix descriptor: start >> 4 in [0,14), LBO = 1 (16 B) in
// [16,30), SBO = 1024 B between 8-row groups in [32,46), version 1 in [46,48),
// layout SWIZZLE_128B (2) in [61,64).
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)1u << 16) | ((uint64_t)(1024u >> 4) << 32) |
         ((uint64_t)1u << 46) | ((uint64_t)2u << 61);
}

// Instruction descriptor, kind::tf32: D F32 (bits 4-5 = 1), A/B TF32 (bits 7-9 and
// 10-12 = 2), both K-major, N >> 3 in [17,23), M >> 4 in [24,29).
__host__ __device__ __forceinline__ constexpr uint32_t idesc_tf32(int M, int N) {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma_tf32(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}

// One lane of a converged warp.  elect.sync names the same lane each time for the
// same mask (PTX ISA), so MMAs and the commits that cover them, all issued under
// it, come from one thread.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred P;\n\telect.sync _|P, 0xffffffff;\n\tselp.u32 %0, 1, 0, P;\n\t}\n" : "=r"(p));
  return p != 0;
}

__device__ __forceinline__ void mma_commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}

__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Warp-wide TMEM allocation of ncols (power of two >= 32); address written to *dst.
__device__ __forceinline__ void tmem_alloc(uint32_t* dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(dst)), "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// 32 lanes x 8 columns of 32-bit accumulators into v[0..7] (lane = row within the warp's quarter).
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float* v) {
  uint32_t r[8];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Adds tx_bytes to the transaction count of the mbarrier's current phase
// (without arriving); the phase then also waits for that many bytes of bulk
// copies that signal complete_tx on it.
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t tx_bytes) {
  asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(tx_bytes)
               : "memory");
}

// 1-D bulk copy global -> this CTA's shared memory (no multicast); both
// addresses 16-byte aligned, bytes a multiple of 16.  Completion is signalled
// as transaction bytes on the mbarrier.
__device__ __forceinline__ void bulk_g2s(void* smem_dst, const void* gmem_src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_addr(smem_dst)),
      "l"(gmem_src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}

// One arrival that also adds tx_bytes to the current phase's transaction count.
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t tx_bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(tx_bytes)
               : "memory");
}

// Barrier among `count` threads (a multiple of 32) on named barrier `id` (1..15).
__device__ __forceinline__ void named_bar_sync(int id, int count) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}

// One arrival (release, CTA scope) on an mbarrier.
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// Clock cycles a bounded wait allows by default (about a second at 2 GHz).
constexpr long long kWaitCycles = 1LL << 31;

// Waits for the phase with the given parity to complete.  Gives up after
// `limit` clock cycles (kWaitCycles when limit <= 0), raising *err; returns
// false then.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* err, long long limit = 0) {
  const uint32_t addr = smem_addr(bar);
  auto test = [&] {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    return done != 0;
  };
  if (test()) return true;  // without reading the clock
  const long long bound = limit > 0 ? limit : kWaitCycles;
  const long long t0 = clock64();
  while (true) {
    if (test()) return true;
    if (clock64() - t0 > bound) {
      atomicExch(err, 1);
      return false;
    }
  }
}

// The same with one outcome for the whole warp, for warps that go on to warp-wide
// instructions (elect.sync, tcgen05.ld, __syncwarp): near the bound some lanes
// could see the phase complete and others give up.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, int* err, long long limit = 0) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, err, limit));
}

// Round-to-nearest TF32 value of x (low 13 bits of the FP32 pattern zero).
__device__ __forceinline__ float tf32_rn(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}

}  // namespace tc
}  // namespace gd
