// Wrappers for kernels that run on CTA pairs (thread-block clusters of two, tcgen05
// cta_group::2): tensor memory, MMA and commit forms of the pair, barriers in the peer's shared
// memory, TMA loads that complete on the leader's barrier.  No load here uses multicast.
#pragma once
#include "woq_tc_common.cuh"

namespace woq {

__device__ __forceinline__ uint32_t pair_cta_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void pair_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of `p` (an address of this CTA) in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t pair_map(const void* p, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  return a;
}
// Arrive on a barrier of either CTA (a shared::cluster address).  What such an arrival hands over here
// is tensor memory (ordered by tcgen05.wait and tcgen05.fence before it), never ordinary memory, so it
// carries no cluster-scope release: with one it took 2000 cycles, four times the stage it ends.
__device__ __forceinline__ void pair_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ float pair_ld_f32(uint32_t a) {  // from a shared::cluster address
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
// true in exactly one lane of a converged warp
__device__ __forceinline__ bool elect_one() {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok));
  return ok != 0;
}

// tensor memory of the pair: one warp of each CTA executes these together
__device__ __forceinline__ void pair_tmem_alloc(uint32_t* smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void pair_tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void pair_tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// D[tmem of both CTAs] (+)= A[tmem of both CTAs, 128 rows each] * B[half of the columns in each CTA's
// shared memory]; M = 256, K = 16 (16-bit inputs).  Issued by one thread of the leader.
__device__ __forceinline__ void pair_mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                                uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      :
      : "r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrive on the barrier at this offset in both CTAs of the pair (`mask`: their ranks in the cluster) once
// everything this thread has issued is done
__device__ __forceinline__ void pair_commit(uint64_t* bar, uint16_t mask = 3) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"(mask)
      : "memory");
}
// Instruction descriptor of a pair's MMA (M = 256); formats as umma_idesc.
__host__ __device__ inline uint32_t pair_idesc(int n, int a_format, int b_format, int c_format) {
  return (static_cast<uint32_t>(c_format) << 4) | (static_cast<uint32_t>(a_format) << 7) |
         (static_cast<uint32_t>(b_format) << 10) | (static_cast<uint32_t>(n >> 3) << 17) |
         (static_cast<uint32_t>(256 >> 4) << 24);
}

// 3-D tiled TMA load (no multicast) into this CTA's shared memory that completes on a barrier of
// either CTA of the pair (a shared::cluster address).
__device__ __forceinline__ void pair_tma_load_3d(void* dst_smem, const CUtensorMap* map, int x, int y, int z,
                                                 uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, "
      "%4}], [%5];" ::"r"(smem_u32(dst_smem)),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}

// 32 lanes x 16 columns of 32-bit accumulators -> registers
__device__ __forceinline__ void tmem_ld_x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

}  // namespace woq
