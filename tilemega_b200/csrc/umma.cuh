// Issue of tcgen05 products from a warp that stays together: one elected lane, operands formed once a warp.
#pragma once
#include "ptx.cuh"

namespace tmb {

// Products of one step of 16 columns, as umma_bf16, with the descriptors' words apart: the low ones differ between steps by a
// constant (an issuing thread that builds each descriptor anew is slower than the tensor pipe), the high ones never.
__device__ __forceinline__ void umma_step(uint32_t d, uint32_t a_low, uint32_t b_low, uint32_t high, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n"
      " .reg .pred p;\n"
      " .reg .b64 a, b;\n"
      " mov.b64 a, {%1, %3};\n"
      " mov.b64 b, {%2, %3};\n"
      " setp.ne.b32 p, %5, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, p;\n"
      "}\n" ::"r"(d),
      "r"(a_low), "r"(b_low), "r"(high), "r"(idesc), "r"(uint32_t(accumulate))
      : "memory");
}
// The same with A in tensor memory: a row a lane, two bf16 a column.
__device__ __forceinline__ void umma_step_tmem(uint32_t d, uint32_t a, uint32_t b_low, uint32_t high, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n"
      " .reg .pred p;\n"
      " .reg .b64 b;\n"
      " mov.b64 b, {%2, %3};\n"
      " setp.ne.b32 p, %5, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %4, p;\n"
      "}\n" ::"r"(d),
      "r"(a), "r"(b_low), "r"(high), "r"(idesc), "r"(uint32_t(accumulate))
      : "memory");
}
__device__ __forceinline__ bool elect_one() {
  uint32_t elected;
  asm volatile(
      "{\n"
      " .reg .pred p;\n"
      " elect.sync _|p, 0xffffffff;\n"
      " selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(elected));
  return elected != 0;
}

// ---- pairs of CTAs (a cluster of two; the first issues) --------------------------------------------------------
// Tensor memory of both, taken and freed by one warp of each.
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* base_in_smem, uint32_t columns) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(base_in_smem)), "r"(columns) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t base, uint32_t columns) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(columns));
}
// The address of a shared variable in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t address_in(const void* local, uint32_t rank) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(local)), "r"(rank));
  return remote;
}
__device__ __forceinline__ void arrive_at(uint64_t* bar, uint32_t rank) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(address_in(bar, rank)) : "memory");
}
__device__ __forceinline__ void store_at(int* local, uint32_t rank, int v) {
  asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(address_in(local, rank)), "r"(v) : "memory");
}
// As tma_load_2d into this CTA's memory, counted on the first CTA's barrier.
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const void* tensor_map, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
      "l"(tensor_map), "r"(x), "r"(y), "r"(address_in(bar, 0))
      : "memory");
}
// umma_step over both CTAs: each has half of A's rows, half of B's and the sums of its rows of A.
__device__ __forceinline__ void umma_step_pair(uint32_t d, uint32_t a_low, uint32_t b_low, uint32_t high, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n"
      " .reg .pred p;\n"
      " .reg .b64 a, b;\n"
      " mov.b64 a, {%1, %3};\n"
      " mov.b64 b, {%2, %3};\n"
      " setp.ne.b32 p, %5, 0;\n"
      " tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %4, p;\n"
      "}\n" ::"r"(d),
      "r"(a_low), "r"(b_low), "r"(high), "r"(idesc), "r"(uint32_t(accumulate))
      : "memory");
}
// One arrival on `bar` of both CTAs.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"(uint16_t(3))
               : "memory");
}

}  // namespace tmb
