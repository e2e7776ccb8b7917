// CTA-pair bf16 GEMM (`gemm_pair.cu`): launch interface used by `gemm_tcgen05.cu`.
#pragma once
#include "common.cuh"

namespace cm {

enum PairMode : int { PAIR_DENSE = 0, PAIR_GROUPED_ROWS = 1, PAIR_GROUPED_K = 2 };

struct PairArgs {
  int M, N, K;             // as GemmArgs: GROUPED_ROWS M = allocated rows; GROUPED_K M, N = one expert's output, K unused
  int bn;                  // columns of a tile: K-major B any multiple of 32 up to 256, MN-major B 128 or 256
  long long ldc;
  int num_experts;
  int accumulate;          // C += result
  int tma_store;           // C tiles leave through shared memory and a bulk tensor store (16-byte aligned C and pitch)
  const int* tile_expert;
  const int* seg_offsets;
  int* err;
};

// A, B as in cm_gemm_bf16 / cm_grouped_gemm_*; returns 0 or an error code.
int launch_gemm_pair(int mode, bool a_mn, bool b_mn, bool out_fp32, const void* A, const void* B, void* C, long long lda, long long ldb,
                     int k_rows, const PairArgs& args, cudaStream_t stream);

}  // namespace cm
