// CTA-pair bf16 GEMM (`gemm_pair.cu`): launch interface used by `gemm_tcgen05.cu`.
#pragma once
#include "common.cuh"

namespace cm {
namespace pair2 {

// ---- device helpers of the CTA-pair kernels ----
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t map_to_rank(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
// Loads into this CTA's shared memory whose completion is counted on a barrier of either CTA of the pair.
__device__ __forceinline__ void load_2d(void* dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void load_3d(void* dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
// Arrive on the barrier at this offset in both CTAs once the MMAs issued so far have retired.
__device__ __forceinline__ void commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "h"((uint16_t)3)
               : "memory");
}

}  // namespace pair2

enum PairMode : int { PAIR_DENSE = 0, PAIR_GROUPED_ROWS = 1, PAIR_GROUPED_K = 2 };

struct PairArgs {
  int M, N, K;             // as GemmArgs: GROUPED_ROWS M = allocated rows; GROUPED_K M, N = one expert's output, K unused
  int bn;                  // columns of a tile: K-major B any multiple of 32 up to 256, MN-major B 128 or 256
  long long ldc;
  int num_experts;
  int accumulate;          // C += result
  int tma_store;           // C tiles leave through shared memory and a bulk tensor store (C, pitch and width multiples of 16 bytes)
  const int* tile_expert;
  const int* seg_offsets;
  int* err;
  int c_vec;               // rows of C start on 16-byte boundaries; set at the launch like tma_store
};

// A, B as in cm_gemm_bf16 / cm_grouped_gemm_*; returns 0 or an error code.
int launch_gemm_pair(int mode, bool a_mn, bool b_mn, bool out_fp32, const void* A, const void* B, void* C, long long lda, long long ldb,
                     int k_rows, const PairArgs& args, cudaStream_t stream);

}  // namespace cm
