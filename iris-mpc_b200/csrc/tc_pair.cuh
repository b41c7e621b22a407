// Device primitives of the two-SM tensor-core kernels (cta_group::2, internal
// to the library): cluster addressing, TMA loads that complete on the leader's
// barrier, the paired MMA and its multicast commit.  Used by the two-SM limb
// GEMM (gemm_limb.cu) and the rotation-structured GEMM (quad_gemm.cu).
#pragma once
#include "gemm_limb.h"
#include "tc_sm100.cuh"

namespace irs {
namespace {

constexpr int kBM2 = 256;  // DB entries per CTA pair (MMA M)

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

__device__ __forceinline__ uint32_t map_to_rank(const void* p, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
  return r;
}

__device__ __forceinline__ uint32_t ld_cluster(uint32_t cluster_addr) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(cluster_addr) : "memory");
  return v;
}

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// QuadFlags::all_set as the cluster's first CTA reads it, for every thread of
// the cluster.  Its CTAs share barriers and tensor memory, so none may work
// where another has left; and the words can change between two readings, where
// the program writes an engine's rows while a graph over it runs.  `slot` is a
// word of shared memory at the same offset in every CTA.
__device__ __forceinline__ bool cluster_reads(const QuadFlags& flags, uint32_t* slot) {
  if (threadIdx.x == 0) *slot = flags.all_set();
  __syncthreads();
  cluster_sync_all();
  const bool all = ld_cluster(map_to_rank(slot, 0)) != 0;
  cluster_sync_all();  // the first CTA stays until the others have read its word
  return all;
}

__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, uint32_t bar_cluster_addr, int x,
                                                 int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
      "[%4];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar_cluster_addr)
      : "memory");
}

__device__ __forceinline__ void mma_u8_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate));
}

// Arrives on the barrier at the same offset in both CTAs of the pair once the
// leader's preceding MMAs have completed.
__device__ __forceinline__ void mma_commit_pair(uint64_t* bar) {
  const uint16_t mask = 0x3;
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"(mask)
      : "memory");
}

// Instruction descriptor: u8 x u8 -> s32, K-major A and B, M = 256, N = bn.
__host__ __device__ constexpr uint32_t idesc_u8_m256(int bn) {
  return (2u << 4) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(kBM2 >> 4) << 24);
}

}  // namespace
}  // namespace irs
