// umma.cuh — inline-PTX building blocks for the 5th-generation tensor cores
// (tcgen05) of sm_103a: shared-memory operand descriptors, TMEM allocation,
// MMA issue and commit, TMEM -> register loads, mbarriers and TMA tile loads.
//
// Operand layout used throughout: K-major tiles of bf16 with the 128-byte
// swizzle. A tile of R rows x 64 elements (128 bytes per row) occupies R*128
// bytes starting at a 1024-byte aligned address; row r's 16-byte chunk c sits
// at r*128 + ((c ^ (r & 7)) * 16). This is the layout a TMA load with
// CU_TENSOR_MAP_SWIZZLE_128B and a 64-element inner box writes, and the one
// the descriptor below describes (8-row groups 1024 bytes apart).
#pragma once

#include <stdint.h>

#include "bounded_wait.h"

namespace amca {
namespace umma {

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Programmatic dependent launch: lets the next kernel of the stream start its
// blocks; waits until the kernels before this one have completed.
__device__ __forceinline__ void launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_prerequisites() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ---- mbarrier -------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
// makes barrier initialisation visible to the async proxy (TMA, tcgen05.commit)
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
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

// Waits until the barrier's phase with the given parity has completed, for at
// most limit_ns nanoseconds; false when the wait ran out.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, unsigned long long limit_ns) {
  if (mbar_test(bar, parity)) return true;
  const unsigned long long t0 = global_ns();
  while (!mbar_test(bar, parity))
    if (global_ns() - t0 > limit_ns) return false;
  return true;
}

// The same for blocks whose warps have separate roles: a wait that runs out
// sets *abort, and every wait ends (false) once it is set. For a role that is
// one thread; a role of whole warps waits by mbar_wait_warp, whose verdict is
// the same in every lane.
__device__ __forceinline__ bool mbar_wait_role(uint32_t bar, uint32_t parity, unsigned long long limit_ns,
                                               volatile int *abort) {
  return wait_or_abort([&] { return mbar_test(bar, parity); }, [] { return global_ns(); }, limit_ns, abort);
}
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, unsigned long long limit_ns,
                                               volatile int *abort) {
  return wait_or_abort_together([&] { return mbar_test(bar, parity); }, [] { return global_ns(); }, limit_ns, abort,
                                [](bool ok) { return __all_sync(0xffffffffu, ok) != 0; });
}

// ---- TMA ------------------------------------------------------------------
// 2-D tiled load of the box at (x = inner coordinate, y = row) into shared
// memory; completion is counted on `bar` in bytes. x must be a multiple of 8
// for bf16 (16 bytes).
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const void *tmap, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          dst),
      "l"((uint64_t)tmap), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

// 2-D tiled store of a shared-memory box to (x = inner coordinate, y = row);
// part of this thread's current bulk group.
__device__ __forceinline__ void tma_store_2d(const void *tmap, uint32_t src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"((uint64_t)tmap),
               "r"(x), "r"(y), "r"(src)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// every committed bulk store of this thread has read its shared memory / has completed
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ void tma_prefetch_desc(const void *tmap) {
  asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)tmap) : "memory");
}

// ---- fences ---------------------------------------------------------------
// generic-proxy shared-memory writes -> visible to the async proxy (MMA reads)
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// ---- TMEM -----------------------------------------------------------------
// Executed by all 32 lanes of one warp. The TMEM address is written to `dst`
// (shared memory). ncols: a power of two, 32..512.
__device__ __forceinline__ void tmem_alloc(uint32_t dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst), "r"(ncols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// ---- descriptors ------------------------------------------------------------
// Shared-memory matrix descriptor of a K-major, 128-byte-swizzled bf16 tile
// starting at `saddr` (1024-byte aligned for the first K step; +32 bytes per
// further K step of 16 elements inside the 128-byte row): start address
// bits 0-13 (>> 4), leading offset 16 bytes (unused by swizzled K-major
// layouts), stride offset 1024 bytes between 8-row groups (bits 32-45),
// descriptor version 1 (bit 46), swizzle mode 2 = 128 bytes (bits 61-63).
__device__ __forceinline__ uint64_t sdesc_sw128(uint32_t saddr) {
  uint64_t d = (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// Descriptor of an MN-major operand (its M or N index contiguous in memory, K
// the row index) in the same tiles: 64 M/N elements per 128-byte row, one row
// per K index. A K step of 16 starts 2048 bytes (16 rows) after the previous
// one; the 8-row groups of a step lie 1024 bytes apart (stride offset, bits
// 32-45) and the next 64 M/N elements `block_bytes` further on (leading offset,
// bits 16-29).
__device__ __forceinline__ uint64_t sdesc_sw128_mn(uint32_t saddr, uint32_t block_bytes) {
  uint64_t d = (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)(block_bytes >> 4) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// Instruction descriptor of tcgen05.mma.kind::f16: D in FP32 (bits 4-5 = 1),
// A and B bf16 (bits 7-9 = 1, 10-12 = 1), A MN-major in bit 15, B MN-major in
// bit 16 (0: K-major), N >> 3 in bits 17-22, M >> 4 in bits 24-28.
__host__ __device__ constexpr uint32_t idesc_bf16_f32(int M, int N, bool a_mn = false, bool b_mn = false) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (a_mn ? 1u << 15 : 0u) | (b_mn ? 1u << 16 : 0u) |
         ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// ---- MMA ------------------------------------------------------------------
// D[tmem] (+)= A[smem] * B[smem]^T for one K step of 16; issued by one thread.
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Arrives once on `bar` when every MMA this thread issued before has completed.
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// ---- TMEM -> registers ---------------------------------------------------------
// 32 lanes x 32 consecutive 32-bit columns: thread t of the warp gets lane
// (taddr lane + t), columns col..col+31. A warp may only address the 32-lane
// quarter (warp id % 4) of TMEM.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// Byte offset of element (row r, column k) inside a K-major 128-byte-swizzled
// bf16 tile of 64-column blocks, each block rows*128 bytes.
__host__ __device__ __forceinline__ uint32_t sw128_offset(uint32_t r, uint32_t k, uint32_t rows) {
  const uint32_t kb = k >> 6, kin = k & 63, chunk = kin >> 3;
  return kb * rows * 128u + r * 128u + (((chunk ^ (r & 7u)) << 4) | ((kin & 7u) << 1));
}

}  // namespace umma
}  // namespace amca
