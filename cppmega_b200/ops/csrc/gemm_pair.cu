// bf16 GEMM on CTA pairs: two CTAs of a cluster (two SMs) work on one 256 x 256 tile with tcgen05.mma.cta_group::2.
// Each CTA loads 128 rows of A and half of the tile's B columns, the pair's tensor cores read both halves, and each CTA
// keeps its own 128 x 256 fp32 accumulator rows in TMEM (two of them, so that the epilogue of a tile runs under the main
// loop of the next).  Roles per CTA as in gemm_tcgen05.cu: warp 0 TMA producer, warp 1 MMA issuer (first CTA of the pair
// only), warps 2..5 epilogue.
//
// What bounds it: at 128 x 256 per SM the one-CTA kernel moves 48 KB through shared memory per 64-deep k block and keeps
// 4 of them in flight; the pair moves 32 KB per SM for the same products, which leaves room for 6 stages and 32 KB of
// store staging, and halves the B traffic from L2.  The epilogue writes whole 128-byte rows with bulk tensor stores
// instead of 16-byte pieces of 32 different rows per instruction.  The tensor pipe is then busy 94 % of the time at 8192^3
// (1.63 PFLOP/s; the one-CTA kernel 1.30).  16384 x 24960 x 4096 runs in 2.06 ms against 2.42 with time between launches to
// cool, and in 2.55 ms in a loop: there the chip is at its 1 kW limit with either kernel (1.2 GHz), and the gain is 0 to 3 %.
//
// Barriers: `full` of the first CTA counts the bytes of both CTAs' loads; `empty` and `tmem_full` exist in both CTAs and
// are signalled together by tcgen05.commit; `tmem_empty` of the first CTA collects the epilogue warps of both.  No load is
// multicast.  Every wait is bounded; a CTA that gives up sets the error word, which ends its partner's waits as well, and
// both meet at the cluster barrier before either releases its shared memory.
#include "gemm_pair.cuh"

namespace cm {
namespace pair2 {

constexpr int BM = 128;          // rows of one CTA; a tile has 2 * BM
constexpr int BN_MAX = 256;
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int THREADS = 192;
constexpr int STAGES = 6;
constexpr int A_BYTES = BM * BK * 2;
constexpr int STAGE_BYTES = 2 * A_BYTES;                     // B: at most 128 rows of 128 bytes
constexpr int STORE_BYTES = 32 * 128;                        // one warp's 32 rows x 128 bytes
constexpr int STORE_OFF = STAGES * STAGE_BYTES;
constexpr int BAR_OFF = STORE_OFF + 4 * 2 * STORE_BYTES;
constexpr int SMEM_TOTAL = BAR_OFF + 256 + 1024;

__device__ __forceinline__ void mma_pair(uint32_t d, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d), "l"(ad), "l"(bd), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void store_2d(const CUtensorMap* map, const void* src, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(reinterpret_cast<uint64_t>(map)),
               "r"(smem_u32(src)), "r"(c0), "r"(c1)
               : "memory");
}
__device__ __forceinline__ void store_3d(const CUtensorMap* map, const void* src, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(reinterpret_cast<uint64_t>(map)),
               "r"(smem_u32(src)), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}

// One tile of a role's walk: expert, first row / column, k blocks, and which CTAs of the pair store their rows.
struct Tile {
  int e, m0, n0, kb0, nkb, store_mask;
};

template <int MODE>
struct Walk {
  const PairArgs& a;
  int tiles_m, tiles_n, per_problem, total, dense_kb;
  __device__ explicit Walk(const PairArgs& args) : a(args) {
    tiles_n = (a.N + a.bn - 1) / a.bn;
    tiles_m = (a.M + 2 * BM - 1) / (2 * BM);
    per_problem = tiles_m * tiles_n;
    total = MODE == PAIR_GROUPED_K ? per_problem * a.num_experts : per_problem;
    dense_kb = (a.K + BK - 1) / BK;
  }
  // `sub`: GROUPED_ROWS only.  A row pair whose halves belong to two experts is worked on twice, once with each expert's
  // weights, and each pass stores one half.  Returns false when there is no such pass.
  __device__ __forceinline__ bool get(int tile, int sub, Tile& t) const {
    int r = tile;
    t.e = 0;
    if (MODE == PAIR_GROUPED_K) {
      t.e = tile / per_problem;
      r = tile - t.e * per_problem;
    }
    // bands of 8 row tiles: the 74 tiles in flight then read about 8 row and 9 column blocks (tools/kernel_bench.py gemm)
    const int band_tiles = 8 * tiles_n, b = r / band_tiles, in = r - b * band_tiles;
    const int rows = min(8, tiles_m - b * 8);
    const int mt = b * 8 + in % rows;
    t.m0 = mt * 2 * BM;
    t.n0 = (in / rows) * a.bn;
    t.kb0 = 0;
    t.nkb = dense_kb;
    t.store_mask = 3;
    if (MODE == PAIR_GROUPED_ROWS) {
      const int e0 = a.tile_expert[2 * mt], e1 = t.m0 + BM < a.M ? a.tile_expert[2 * mt + 1] : -1;
      if (e0 == e1) {
        if (sub == 1) return false;
      } else {
        t.store_mask = 1 << sub;
      }
      t.e = sub ? e1 : e0;
      return t.e >= 0;
    }
    if (MODE == PAIR_GROUPED_K) {
      const int s0 = a.seg_offsets[t.e], s1 = a.seg_offsets[t.e + 1];
      t.kb0 = s0 / BK;
      t.nkb = (s1 - s0) / BK;
    }
    return sub == 0;
  }
};

template <bool A_MN, bool B_MN, typename OutT, int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmC,
                 OutT* __restrict__ C, const PairArgs args) {
  extern __shared__ uint8_t smem_raw[];
  // the dynamic segment starts at the same offset in both CTAs, so the aligned offsets agree as the descriptors need
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + BAR_OFF);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tmem_full = empty_bar + STAGES;
  uint64_t* tmem_empty = tmem_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int first_tile = blockIdx.x >> 1, tile_step = gridDim.x >> 1;
  const Walk<MODE> walk(args);

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tmem_full[b], 1);
      mbar_init(&tmem_empty[b], 8);
    }
    *abort_flag = (args.err && *reinterpret_cast<volatile int*>(args.err) != 0) ? 1 : 0;   // an earlier kernel gave up: drain
    fence_mbar_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int half = args.bn >> 1;

  if (warp == 0) {
    // ------------------------------ TMA producer (both CTAs) ------------------------------
    if (elect_one()) {
      tma_prefetch_desc(&tmA);
      tma_prefetch_desc(&tmB);
      const uint32_t pair_bytes = 2 * (A_BYTES + half * 128);
      uint32_t stage = 0, phase = 0, used = 0;
      bool ok = *abort_flag == 0;
      for (int tile = first_tile; tile < walk.total && ok; tile += tile_step) {
        for (int sub = 0; sub < (MODE == PAIR_GROUPED_ROWS ? 2 : 1) && ok; ++sub) {
          Tile t;
          if (!walk.get(tile, sub, t)) continue;
          const int ma = t.m0 + rank * BM, nb = t.n0 + rank * half;
          for (int kb = 0; kb < t.nkb; ++kb) {
            ok = mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, args.err, ERR_WAIT_EMPTY);
            if (!ok) break;
            uint8_t* sa = smem + stage * STAGE_BYTES;
            uint8_t* sb = sa + A_BYTES;
            if (rank == 0) mbar_expect_tx(&full_bar[stage], pair_bytes);
            const uint32_t bar = map_to_rank(smem_u32(&full_bar[stage]), 0);
            const int k0 = (t.kb0 + kb) * BK;
            if (!A_MN) {
              load_2d(sa, &tmA, bar, k0, ma);                                           // box [128 rows, 64 k]
            } else {
#pragma unroll
              for (int c = 0; c < BM / 64; ++c) load_2d(sa + c * (BK * 128), &tmA, bar, ma + c * 64, k0);   // boxes [64 k, 64 m]
            }
            if (!B_MN) {
              if (MODE == PAIR_GROUPED_ROWS) load_3d(sb, &tmB, bar, k0, nb, t.e);
              else load_2d(sb, &tmB, bar, k0, nb);                                      // box [bn / 2 rows, 64 k]
            } else {
              for (int c = 0; c < half / 64; ++c) {                                     // boxes [64 k, 64 n]
                if (MODE == PAIR_GROUPED_ROWS) load_3d(sb + c * (BK * 128), &tmB, bar, nb + c * 64, k0, t.e);
                else load_2d(sb + c * (BK * 128), &tmB, bar, nb + c * 64, k0);
              }
            }
            if (used < STAGES) ++used;
            if (++stage == STAGES) { stage = 0; phase ^= 1; }
          }
        }
      }
      // the last releases of this CTA's stages come from the partner: see them arrive before the barriers go away
      for (uint32_t i = 0; i < used && ok; ++i) {
        const uint32_t s = (stage + STAGES - 1 - i) % STAGES;
        const uint32_t ph = (stage >= i + 1) ? phase : phase ^ 1;
        ok = mbar_wait(&empty_bar[s], ph, abort_flag, args.err, ERR_WAIT_EMPTY);
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (first CTA) ------------------------------
    if (rank == 0 && elect_one()) {
      const uint32_t idesc = umma_idesc_bf16(2 * BM, args.bn, A_MN, B_MN);
      uint32_t stage = 0, phase = 0, acc = 0, acc_phase = 0;
      bool ok = *abort_flag == 0;
      for (int tile = first_tile; tile < walk.total && ok; tile += tile_step) {
        for (int sub = 0; sub < (MODE == PAIR_GROUPED_ROWS ? 2 : 1) && ok; ++sub) {
          Tile t;
          if (!walk.get(tile, sub, t) || t.nkb == 0) continue;
          ok = mbar_wait(&tmem_empty[acc], acc_phase ^ 1, abort_flag, args.err, ERR_WAIT_TMEM_EMPTY);
          if (!ok) break;
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + acc * BN_MAX;
          for (int kb = 0; kb < t.nkb; ++kb) {
            ok = mbar_wait(&full_bar[stage], phase, abort_flag, args.err, ERR_WAIT_FULL);
            if (!ok) break;
            tc_fence_after();
            const uint32_t sa = smem_u32(smem + stage * STAGE_BYTES);
            const uint32_t sb = sa + A_BYTES;
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k) {
              const uint64_t ad = A_MN ? umma_desc_sw128(sa + k * (UMMA_K * 128), BK * 128, 1024)
                                       : umma_desc_sw128(sa + k * (UMMA_K * 2), 16, 1024);
              const uint64_t bd = B_MN ? umma_desc_sw128(sb + k * (UMMA_K * 128), BK * 128, 1024)
                                       : umma_desc_sw128(sb + k * (UMMA_K * 2), 16, 1024);
              mma_pair(d_tmem, ad, bd, idesc, (kb | k) != 0);
            }
            commit_pair(&empty_bar[stage]);
            if (++stage == STAGES) { stage = 0; phase ^= 1; }
          }
          if (!ok) break;
          commit_pair(&tmem_full[acc]);
          acc ^= 1;
          if (acc == 0) acc_phase ^= 1;
        }
      }
    }
  } else {
    // ------------------------------ epilogue (both CTAs) ------------------------------
    const int q = warp & 3;                       // TMEM lane quadrant this warp may read
    constexpr int CHUNK = 128 / int(sizeof(OutT));      // columns that make 128 bytes
    uint8_t* stage_buf = smem + STORE_OFF + q * 2 * STORE_BYTES;
    uint32_t acc = 0, acc_phase = 0, buf = 0;
    bool ok = *abort_flag == 0;
    for (int tile = first_tile; tile < walk.total && ok; tile += tile_step) {
      for (int sub = 0; sub < (MODE == PAIR_GROUPED_ROWS ? 2 : 1) && ok; ++sub) {
        Tile t;
        if (!walk.get(tile, sub, t)) continue;
        const int row0 = t.m0 + rank * BM + q * 32, row = row0 + lane;
        const int n_end = min(t.n0 + args.bn, args.N);
        OutT* crow = C + (MODE == PAIR_GROUPED_K ? (long long)t.e * args.M * args.ldc : 0ll) + (long long)row * args.ldc;
        if (t.nkb == 0) {
          if (MODE == PAIR_GROUPED_K && !args.accumulate && row < args.M)
            for (int c = t.n0; c < n_end; ++c) crow[c] = OutT(0.f);
          continue;
        }
        ok = __all_sync(0xffffffffu, mbar_wait(&tmem_full[acc], acc_phase, abort_flag, args.err, ERR_WAIT_TMEM_FULL));
        if (!ok) break;
        tc_fence_after();
        const uint32_t t_base = tmem_base + acc * BN_MAX + (uint32_t(q * 32) << 16);
        if (!(t.store_mask >> rank & 1) || row0 >= args.M) {
          // the rows of this warp belong to another expert, or lie past the matrix
        } else if (args.tma_store) {
          for (int c = 0; t.n0 + c < n_end; c += CHUNK) {
            if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");    // this buffer's last store has been read
            __syncwarp();
            uint8_t* dst = stage_buf + buf * STORE_BYTES + lane * 128;
#pragma unroll
            for (int h = 0; h < CHUNK / 32; ++h) {
              uint32_t r[32];
              tmem_ld_32x32(t_base + c + h * 32, r);
              tmem_ld_wait();
              if constexpr (sizeof(OutT) == 2) {
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                  uint4 o;
                  o.x = pack_bf16(__uint_as_float(r[v * 8 + 0]), __uint_as_float(r[v * 8 + 1]));
                  o.y = pack_bf16(__uint_as_float(r[v * 8 + 2]), __uint_as_float(r[v * 8 + 3]));
                  o.z = pack_bf16(__uint_as_float(r[v * 8 + 4]), __uint_as_float(r[v * 8 + 5]));
                  o.w = pack_bf16(__uint_as_float(r[v * 8 + 6]), __uint_as_float(r[v * 8 + 7]));
                  *reinterpret_cast<uint4*>(dst + (((h * 4 + v) ^ (lane & 7)) << 4)) = o;
                }
              } else {
#pragma unroll
                for (int v = 0; v < 8; ++v)
                  *reinterpret_cast<uint4*>(dst + ((v ^ (lane & 7)) << 4)) = make_uint4(r[v * 4], r[v * 4 + 1], r[v * 4 + 2], r[v * 4 + 3]);
              }
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              if (MODE == PAIR_GROUPED_K) store_3d(&tmC, stage_buf + buf * STORE_BYTES, t.n0 + c, row0, t.e);
              else store_2d(&tmC, stage_buf + buf * STORE_BYTES, t.n0 + c, row0);
              asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
            buf ^= 1;
          }
        } else {
#pragma unroll 1
          for (int c = 0; t.n0 + c < n_end; c += 32) {
            uint32_t r[32];
            tmem_ld_32x32(t_base + c, r);
            tmem_ld_wait();
            const int col = t.n0 + c;
            if (row >= args.M) continue;
            if (col + 32 <= args.N && args.c_vec) {
              if constexpr (sizeof(OutT) == 2) {
                uint4* dst = reinterpret_cast<uint4*>(crow + col);
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                  float f[8];
                  if (args.accumulate) {
                    const uint4 old = dst[v];
                    const __nv_bfloat162* ob = reinterpret_cast<const __nv_bfloat162*>(&old);
#pragma unroll
                    for (int j = 0; j < 4; ++j) { const float2 p = __bfloat1622float2(ob[j]); f[2 * j] = p.x; f[2 * j + 1] = p.y; }
                  } else {
#pragma unroll
                    for (int j = 0; j < 8; ++j) f[j] = 0.f;
                  }
                  uint4 o;
                  o.x = pack_bf16(__uint_as_float(r[v * 8 + 0]) + f[0], __uint_as_float(r[v * 8 + 1]) + f[1]);
                  o.y = pack_bf16(__uint_as_float(r[v * 8 + 2]) + f[2], __uint_as_float(r[v * 8 + 3]) + f[3]);
                  o.z = pack_bf16(__uint_as_float(r[v * 8 + 4]) + f[4], __uint_as_float(r[v * 8 + 5]) + f[5]);
                  o.w = pack_bf16(__uint_as_float(r[v * 8 + 6]) + f[6], __uint_as_float(r[v * 8 + 7]) + f[7]);
                  dst[v] = o;
                }
              } else {
                float4* dst = reinterpret_cast<float4*>(crow + col);
                float4 old[8];
                if (args.accumulate) {
#pragma unroll
                  for (int v = 0; v < 8; ++v) old[v] = dst[v];
                } else {
#pragma unroll
                  for (int v = 0; v < 8; ++v) old[v] = make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
                for (int v = 0; v < 8; ++v)
                  dst[v] = make_float4(__uint_as_float(r[v * 4]) + old[v].x, __uint_as_float(r[v * 4 + 1]) + old[v].y,
                                       __uint_as_float(r[v * 4 + 2]) + old[v].z, __uint_as_float(r[v * 4 + 3]) + old[v].w);
              }
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) {
                if (col + j < n_end) {
                  float v = __uint_as_float(r[j]);
                  if (args.accumulate) v += float(crow[col + j]);
                  crow[col + j] = OutT(v);
                }
              }
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(map_to_rank(smem_u32(&tmem_empty[acc]), 0));
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1;
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    __syncwarp();
  }

  // ------------------------------ teardown ------------------------------
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    // let TMA copies and MMAs still in flight land before the pair's shared memory is released
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
    __syncthreads();
  }
  cluster_sync();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

// C as the target of bulk tensor stores: boxes of 32 rows x 128 bytes.
static int make_store_map(CUtensorMap* out, void* C, bool fp32, int rank3, const PairArgs& a) {
  EncodeTiledFn enc = get_encode_tiled();
  if (!enc) return -1;
  const cuuint64_t es = fp32 ? 4 : 2;
  cuuint64_t dims[3] = {(cuuint64_t)a.N, (cuuint64_t)a.M, (cuuint64_t)a.num_experts};
  cuuint64_t strides[2] = {(cuuint64_t)a.ldc * es, (cuuint64_t)a.ldc * es * (cuuint64_t)a.M};
  cuuint32_t box[3] = {(cuuint32_t)(128 / es), 32, 1};
  cuuint32_t one[3] = {1, 1, 1};
  CUresult r = enc(out, fp32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank3 ? 3 : 2, C, dims, strides, box, one,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : int(r);
}

template <bool A_MN, bool B_MN, typename OutT, int MODE>
static int launch(const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmC, void* C, const PairArgs& args, int tiles,
                  cudaStream_t stream) {
  auto kern = gemm_pair_kernel<A_MN, B_MN, OutT, MODE>;
  static PerDevice configured;
  if (configured.first()) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_TOTAL) != cudaSuccess) return -2;
    configured.done();
  }
  const int pairs = sm_count() / 2;
  const int grid = 2 * (tiles < pairs ? tiles : pairs);
  kern<<<grid, THREADS, SMEM_TOTAL, stream>>>(tmA, tmB, tmC, (OutT*)C, args);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

}  // namespace pair2

int launch_gemm_pair(int mode, bool a_mn, bool b_mn, bool out_fp32, const void* A, const void* B, void* C, long long lda, long long ldb,
                     int k_rows, const PairArgs& in, cudaStream_t stream) {
  PairArgs args = in;
  CUtensorMap tmA, tmB, tmC;
  int rc = a_mn ? make_tmap_2d_bf16(&tmA, A, k_rows, args.M, lda, 64) : make_tmap_2d_bf16(&tmA, A, args.M, args.K, lda, pair2::BM);
  if (rc) return rc;
  const uint32_t half = args.bn / 2;
  if (mode == PAIR_GROUPED_ROWS)
    rc = b_mn ? make_tmap_3d_bf16(&tmB, B, args.num_experts, args.K, args.N, ldb, 64)
              : make_tmap_3d_bf16(&tmB, B, args.num_experts, args.N, args.K, ldb, half);
  else
    rc = b_mn ? make_tmap_2d_bf16(&tmB, B, k_rows, args.N, ldb, 64) : make_tmap_2d_bf16(&tmB, B, args.N, args.K, ldb, half);
  if (rc) return rc;
  const int es = out_fp32 ? 4 : 2;
  const bool c_aligned = (reinterpret_cast<uintptr_t>(C) & 15) == 0;
  // a bulk store cuts a row off at the next multiple of 16 bytes, not at its last element: rows that end elsewhere go element-wise
  args.tma_store = !args.accumulate && c_aligned && (args.ldc * es) % 16 == 0 && ((long long)args.N * es) % 16 == 0 &&
                   args.ldc >= args.N;     // a single row may come with any pitch, which a tensor map does not take
  args.c_vec = c_aligned && args.ldc % 8 == 0;
  if (args.tma_store) {
    rc = pair2::make_store_map(&tmC, C, out_fp32, mode == PAIR_GROUPED_K, args);
    if (rc) return rc;
  } else {
    tmC = tmA;                                   // not used by the kernel
  }
  const int tiles = ((args.M + 2 * pair2::BM - 1) / (2 * pair2::BM)) * ((args.N + args.bn - 1) / args.bn) *
                    (mode == PAIR_GROUPED_K ? args.num_experts : 1);
  if (tiles <= 0) return 0;
#define CM_PAIR(AMN, BMN, OUT, MODE) pair2::launch<AMN, BMN, OUT, MODE>(tmA, tmB, tmC, C, args, tiles, stream)
  if (mode == PAIR_DENSE) {
    if (!a_mn && !b_mn) return out_fp32 ? CM_PAIR(false, false, float, PAIR_DENSE) : CM_PAIR(false, false, __nv_bfloat16, PAIR_DENSE);
    if (!a_mn) return out_fp32 ? CM_PAIR(false, true, float, PAIR_DENSE) : CM_PAIR(false, true, __nv_bfloat16, PAIR_DENSE);
    if (b_mn) return out_fp32 ? CM_PAIR(true, true, float, PAIR_DENSE) : CM_PAIR(true, true, __nv_bfloat16, PAIR_DENSE);
    return out_fp32 ? CM_PAIR(true, false, float, PAIR_DENSE) : CM_PAIR(true, false, __nv_bfloat16, PAIR_DENSE);
  }
  if (mode == PAIR_GROUPED_ROWS)
    return b_mn ? CM_PAIR(false, true, __nv_bfloat16, PAIR_GROUPED_ROWS) : CM_PAIR(false, false, __nv_bfloat16, PAIR_GROUPED_ROWS);
  return out_fp32 ? CM_PAIR(true, true, float, PAIR_GROUPED_K) : CM_PAIR(true, true, __nv_bfloat16, PAIR_GROUPED_K);
#undef CM_PAIR
}

}  // namespace cm
