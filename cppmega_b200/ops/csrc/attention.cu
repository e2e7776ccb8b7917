// Dense causal multi-head attention for the full-attention MLA layers and the MTP layers (q/k head dim 128 = 64 "nope"
// + 64 rope dims, value head dim 64), forward and backward, on tcgen05 with the scores in TMEM.
//
//   s[i,j] = scale * q[i,:] . k[j,:]  (j <= i)      p = softmax_j(s)      o[i,:] = sum_j p[i,j] v[j,:]
//
// forward   one CTA per (pair of 128-query tiles, head, batch).  A TMA warp keeps up to three (K, V) tiles in shared memory, an
//           MMA warp issues S_t = Q_t K^T and O_t += P_t V for the two query tiles t in turn, and one warpgroup per query
//           tile (thread <-> query row <-> TMEM lane) does the softmax: half of S is read twice (maximum, exponentials), P goes back to
//           TMEM as the bf16 A operand of P V, and O stays in TMEM.  O is rescaled only when a row maximum has grown by more
//           than 2^8 since the last rescale (the softmax is the same for any reference value; l and O use the same one).
//           What bounds it: the exponentials, 128 x 128 of them per tile at 16 a cycle = 1024 cycles against 768 of tensor
//           work; the two warpgroups and the products of the other tile overlap.
// backward  one CTA per (128-key tile, head, batch) looping over the query tiles at or below the diagonal:
//           S = Q K^T, dP = dO V^T  ->  P = exp2(S - lse), dS = scale * P o (dP - delta)  ->  dV += P^T dO, dK += dS^T Q
//           (both stay in TMEM for the whole loop), dQ_i = dS K, added to an fp32 buffer by bulk tensor reductions
//           (cp.reduce.async.bulk.tensor .add.f32) - the only atomics, issued by the copy engine.
//           Warp roles: 8 compute warps (a query row's 128 columns are split over two threads), 4 warps that drain dQ, one
//           MMA warp, one TMA warp.  S and dP of the next query tile are multiplied while the current one is in registers;
//           dQ goes through 64 TMEM columns in two halves, since S, dP, dV and dK take the other 448.
//           What bounds it: shared-memory bandwidth - 272 KB of MMA operand reads, 64 KB of P / dS writes and 128 KB of dQ
//           staging a tile are about 3,700 cycles at 128 bytes a cycle, against 2,048 of tensor work.
// All operand tiles are 128-byte-swizzled [128 x 64] bf16 slabs written by TMA (2-D maps over [B*S, H*dim]); the same
// slab is read K-major or MN-major by choosing the descriptor.  Every wait is bounded and reports through the error word.
// Measured at batch 2, seq 4096, 32 heads: forward 262 us (633 with one 128-thread CTA per query tile, K and V loaded in line and
// two passes of exp2f with range handling), backward 697 us (1660 with 128 threads walking the phases one after the other; 587
// when the dQ reductions are left out, so they are a sixth of it).
// The reference takes this operator from cuDNN / FlashAttention (`--attention-backend flash`,
// scripts/remote_smoke_h200_dsa_9_4_m.sh:727-728; MLA adapter at cppmega/megatron/mla_shared.py:39-97).
#include "common.cuh"

namespace cm {
namespace attn {

constexpr int BQ = 128;          // query rows per tile
constexpr int BK = 128;          // key rows per tile
constexpr int D = 128;           // q / k head dim
constexpr int DV = 64;           // v head dim
constexpr int SLAB = 128 * 128;  // bytes of one [128 rows x 64 bf16] swizzled slab

__device__ __forceinline__ int sw_off(int row, int c) { return row * 128 + ((c ^ (row & 7)) << 4); }

// [128 x 128] operand, K-major (two slabs side by side along K), 16-element k step `k` (0..7)
__device__ __forceinline__ uint64_t desc_k(uint32_t tile, int k) {
  return umma_desc_sw128(tile + (k >> 2) * SLAB + (k & 3) * 32, 16, 1024);
}
// [128(K) rows x 64] slab read MN-major (M/N = the 64 columns), 16-row k step
__device__ __forceinline__ uint64_t desc_mn1(uint32_t slab, int k) { return umma_desc_sw128(slab + k * 2048, SLAB, 1024); }
// [128(K) rows x 128] two-slab tile read MN-major (M/N = the 128 columns)
__device__ __forceinline__ uint64_t desc_mn2(uint32_t tile, int k) { return umma_desc_sw128(tile + k * 2048, SLAB, 1024); }

__device__ __forceinline__ uint4 pack8f(const float* f) {
  uint4 o;
  o.x = pack_bf16(f[0], f[1]); o.y = pack_bf16(f[2], f[3]);
  o.z = pack_bf16(f[4], f[5]); o.w = pack_bf16(f[6], f[7]);
  return o;
}

// A in TMEM (row = lane, two consecutive bf16 of K per 32-bit column), B in shared memory
__device__ __forceinline__ void umma_f16_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
      "}\n" ::"r"(d_tmem),
      "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// 32 registers per thread -> 32 lanes x 32 consecutive columns (thread = TMEM lane)
__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]),
      "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// A wait by a whole warp whose lanes then stay together: one lane that gives up takes the warp with it
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* err, int code) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, err, code));
}
struct Diagonal { static constexpr bool value = true; };
struct Interior { static constexpr bool value = false; };

struct FwdArgs {
  __nv_bfloat16* out;   // [B, S, H, DV]
  float* lse2;          // [B, H, S]: log2-domain log-sum-exp of the scaled scores
  int S, H, n_qt;
  float scale_log2;     // softmax scale * log2(e)
  int* err;
};

constexpr int FWD_THREADS = 320;          // warps 0-3 / 4-7: softmax of query tile 0 / 1; 8: MMA; 9: TMA
constexpr int KV_STAGES = 3;
constexpr float RESCALE_AT = 8.f;         // log2 growth of a row maximum that triggers a rescale: P stays below 2^8

struct FwdShared {
  uint64_t q_full[2], kv_full[KV_STAGES], kv_empty[KV_STAGES];
  uint64_t s_full[2], s_free[2], p_full[2], o_done[2];
  uint32_t tmem_slot;
  int abort_flag;
};

constexpr int fwd_smem() { return 4 * SLAB + KV_STAGES * 3 * SLAB + (int)sizeof(FwdShared) + 1024; }

__global__ void __launch_bounds__(FWD_THREADS, 1) attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQ,
                                                                  const __grid_constant__ CUtensorMap tmK,
                                                                  const __grid_constant__ CUtensorMap tmV, const FwdArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;                      // 2 query tiles [128 x 128]
  uint8_t* sKV = sQ + 4 * SLAB;            // stages of K [128 x 128], V [128 x 64]
  FwdShared* sh = reinterpret_cast<FwdShared*>(sKV + KV_STAGES * 3 * SLAB);

  // pairs with many key tiles first
  const int n_pairs = (a.n_qt + 1) >> 1;
  const int bh_count = gridDim.x / n_pairs;
  const int bh = blockIdx.x % bh_count;
  const int pair = n_pairs - 1 - blockIdx.x / bh_count;
  const int h = bh % a.H, b = bh / a.H;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tiles = min(2, a.n_qt - 2 * pair);                 // an odd tile count leaves the last pair with one tile
  const int n_kt = 2 * pair + tiles;                           // key tiles of the last query tile; tile t sees 2 pair + t + 1
  const int row0 = b * a.S;                                    // first row of this batch in the [B*S, .] views
  volatile int* abort_flag = &sh->abort_flag;
  if (tid == 0) {
    for (int t = 0; t < 2; ++t) {
      mbar_init(&sh->q_full[t], 1);
      mbar_init(&sh->s_full[t], 1);
      mbar_init(&sh->s_free[t], 4);
      mbar_init(&sh->p_full[t], 4);
      mbar_init(&sh->o_done[t], 1);
    }
    for (int s = 0; s < KV_STAGES; ++s) {
      mbar_init(&sh->kv_full[s], 1);
      mbar_init(&sh->kv_empty[s], 1);
    }
    sh->abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 8) { tmem_alloc(&sh->tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  const bool drain = setup_barrier(a.err);
  tc_fence_after();
  const uint32_t tmem = sh->tmem_slot;     // S_t at 128 t, O_t at 256 + 64 t, P_t at 384 + 64 t
  if (drain) {
    if (warp == 8) tmem_dealloc(tmem, 512);
    return;
  }

  if (warp == 9) {
    // ------------------------------ TMA producer ------------------------------
    if (elect_one()) {
      for (int t = 0; t < tiles; ++t) {
        const int qrow = row0 + (2 * pair + t) * BQ;
        mbar_expect_tx(&sh->q_full[t], 2 * SLAB);
        tma_load_2d(sQ + t * 2 * SLAB, &tmQ, &sh->q_full[t], h * D, qrow);
        tma_load_2d(sQ + t * 2 * SLAB + SLAB, &tmQ, &sh->q_full[t], h * D + 64, qrow);
      }
      for (int j = 0; j < n_kt; ++j) {
        const int s = j % KV_STAGES;
        if (!mbar_wait(&sh->kv_empty[s], ((j / KV_STAGES) & 1) ^ 1, abort_flag, a.err, ERR_WAIT_EMPTY)) break;
        uint8_t* st = sKV + s * 3 * SLAB;
        mbar_expect_tx(&sh->kv_full[s], 3 * SLAB);
        tma_load_2d(st, &tmK, &sh->kv_full[s], h * D, row0 + j * BK);
        tma_load_2d(st + SLAB, &tmK, &sh->kv_full[s], h * D + 64, row0 + j * BK);
        tma_load_2d(st + 2 * SLAB, &tmV, &sh->kv_full[s], h * DV, row0 + j * BK);
      }
    }
  } else if (warp == 8) {
    // ------------------------------ MMA issuer ------------------------------
    if (elect_one()) {
      constexpr uint32_t id_s = umma_idesc_bf16(BQ, BK, false, false);
      constexpr uint32_t id_o = umma_idesc_bf16(BQ, DV, false, true);
      bool ok = true;
      auto scores = [&](int t, int j) {     // S_t = Q_t K_j^T
        const uint32_t aQ = smem_u32(sQ + t * 2 * SLAB), aK = smem_u32(sKV + (j % KV_STAGES) * 3 * SLAB);
#pragma unroll
        for (int k = 0; k < D / 16; ++k) umma_f16(tmem + t * 128, desc_k(aQ, k), desc_k(aK, k), id_s, k != 0);
        umma_commit(&sh->s_full[t]);
      };
      auto kv_wait = [&](int j) {
        return mbar_wait(&sh->kv_full[j % KV_STAGES], (j / KV_STAGES) & 1, abort_flag, a.err, ERR_WAIT_FULL);
      };
      ok = kv_wait(0);
      for (int t = 0; t < tiles && ok; ++t) {
        ok = mbar_wait(&sh->q_full[t], 0, abort_flag, a.err, ERR_WAIT_FULL);
        tc_fence_after();
        if (ok) scores(t, 0);
      }
      for (int j = 0; j < n_kt && ok; ++j) {
        // per tile: the next scores as soon as its softmax has read the current ones, then the product of P with V
        if (j + 1 < n_kt) ok = kv_wait(j + 1);
        const uint32_t aV = smem_u32(sKV + (j % KV_STAGES) * 3 * SLAB + 2 * SLAB);
        for (int t = 0; t < tiles && ok; ++t) {
          if (j > 2 * pair + t) continue;
          if (j + 1 <= 2 * pair + t) {
            ok = mbar_wait(&sh->s_free[t], j & 1, abort_flag, a.err, ERR_WAIT_TMEM_EMPTY);
            tc_fence_after();
            if (!ok) break;
            scores(t, j + 1);
          }
          ok = mbar_wait(&sh->p_full[t], j & 1, abort_flag, a.err, ERR_WAIT_TMEM_EMPTY);
          tc_fence_after();
          if (!ok) break;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            umma_f16_ta(tmem + 256 + t * 64, tmem + 384 + t * 64 + k * 8, desc_mn1(aV, k), id_o, (j | k) != 0);
          umma_commit(&sh->o_done[t]);
        }
        if (ok) umma_commit(&sh->kv_empty[j % KV_STAGES]);
      }
    }
  } else if ((warp >> 2) < tiles) {
    // ------------------------------ softmax of query tile t ------------------------------
    const int t = warp >> 2, r = tid & 127, qt = 2 * pair + t;
    const uint32_t lane_addr = uint32_t((warp & 3) * 32) << 16;
    const uint32_t tS = tmem + t * 128 + lane_addr, tO = tmem + 256 + t * 64 + lane_addr, tP = tmem + 384 + t * 64 + lane_addr;
    float m_ref = -INFINITY, l = 0.f;
    auto tile = [&](int j, auto where) {
      constexpr bool DIAG = decltype(where)::value;         // columns past the row drop out
      bool ok = warp_wait(&sh->s_full[t], j & 1, abort_flag, a.err, ERR_WAIT_TMEM_FULL);
      if (!ok) return false;
      tc_fence_after();
      // first pass over the row: its maximum.  The first half of the row is read last and kept for the second pass.
      float m_new = -INFINITY;
      uint32_t s0[32], s1[32], s2[32];
#pragma unroll
      for (int c = 1; c >= 0; --c) {
        tmem_ld_32x32(tS + c * 64, s0);
        tmem_ld_32x32(tS + c * 64 + 32, s1);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          if (!DIAG || c * 64 + e <= r) m_new = fmaxf(m_new, __uint_as_float(s0[e]));
          if (!DIAG || c * 64 + 32 + e <= r) m_new = fmaxf(m_new, __uint_as_float(s1[e]));
        }
      }
      m_new *= a.scale_log2;
      float alpha = 1.f;
      if (j == 0) {
        m_ref = m_new;
      } else {
        if (m_new > m_ref + RESCALE_AT) {
          alpha = ex2(m_ref - m_new);
          m_ref = m_new;
          l *= alpha;
        }
        ok = warp_wait(&sh->o_done[t], (j - 1) & 1, abort_flag, a.err, ERR_WAIT_TMEM_FULL);      // P_t and O_t are free
        if (!ok) return false;
        tc_fence_after();
        if (__any_sync(0xffffffffu, alpha != 1.f)) {
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t o[32];
            tmem_ld_32x32(tO + c * 32, o);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
            tmem_st_32x32(tO + c * 32, o);
          }
        }
      }
      float sum[4] = {0.f, 0.f, 0.f, 0.f};  // second pass: P in bf16, row sum in fp32
      uint32_t p[32];
      auto quarter = [&](const uint32_t (&sc)[32], int col0, int at) {
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          float x = ex2(fmaf(__uint_as_float(sc[2 * e]), a.scale_log2, -m_ref));
          float y = ex2(fmaf(__uint_as_float(sc[2 * e + 1]), a.scale_log2, -m_ref));
          if (DIAG) {
            x = col0 + 2 * e <= r ? x : 0.f;
            y = col0 + 2 * e + 1 <= r ? y : 0.f;
          }
          sum[(2 * e) & 3] += x;
          sum[(2 * e + 1) & 3] += y;
          p[at + e] = pack_bf16(x, y);
        }
      };
      quarter(s0, 0, 0);
      quarter(s1, 32, 16);
      tmem_st_32x32(tP, p);
      tmem_ld_32x32(tS + 64, s2);
      tmem_ld_32x32(tS + 96, s1);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh->s_free[t]);
      quarter(s2, 64, 0);
      quarter(s1, 96, 16);
      tmem_st_32x32(tP + 32, p);
      l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh->p_full[t]);
      return true;
    };
    bool ok = true;
    for (int j = 0; j < qt && ok; ++j) ok = tile(j, Interior{});
    ok = ok && tile(qt, Diagonal{});
    if (ok) ok = warp_wait(&sh->o_done[t], qt & 1, abort_flag, a.err, ERR_WAIT_TMEM_FULL);
    if (ok) {
      tc_fence_after();
      const float inv = l > 0.f ? __fdividef(1.f, l) : 0.f;
      __nv_bfloat16* orow = a.out + ((size_t)(row0 + qt * BQ + r) * a.H + h) * DV;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t o[32];
        tmem_ld_32x32(tO + c * 32, o);
        tmem_ld_wait();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float f[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(o[q * 8 + e]) * inv;
          reinterpret_cast<uint4*>(orow)[c * 4 + q] = pack8f(f);
        }
      }
      a.lse2[((size_t)b * a.H + h) * a.S + qt * BQ + r] = m_ref + log2f(l);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(2000);      // copies in flight land before the shared memory is released
    __syncthreads();
  }
  if (warp == 8) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

// delta[b,h,s] = sum_d dO[b,s,h,d] * O[b,s,h,d]: eight lanes per (token, head), one 16-byte vector of each operand per lane
__global__ void __launch_bounds__(256) attn_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ dout,
                                                         float* __restrict__ delta, long long rows, int S, int H) {
  const long long w = blockIdx.x * 32LL + (threadIdx.x >> 3);
  const int part = threadIdx.x & 7;
  float d = 0.f;
  if (w < rows) {
    const uint4 ov = reinterpret_cast<const uint4*>(o + w * DV)[part], gv = reinterpret_cast<const uint4*>(dout + w * DV)[part];
    const __nv_bfloat162* ob = reinterpret_cast<const __nv_bfloat162*>(&ov);
    const __nv_bfloat162* gb = reinterpret_cast<const __nv_bfloat162*>(&gv);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 x = __bfloat1622float2(ob[i]), y = __bfloat1622float2(gb[i]);
      d += x.x * y.x + x.y * y.y;
    }
  }
  d += __shfl_xor_sync(0xffffffffu, d, 1);
  d += __shfl_xor_sync(0xffffffffu, d, 2);
  d += __shfl_xor_sync(0xffffffffu, d, 4);
  if (part == 0 && w < rows) {
    const long long tok = w / H;
    const int h = (int)(w % H);
    const long long b = tok / S, s = tok % S;
    delta[(b * H + h) * S + s] = d;
  }
}

struct BwdArgs {
  const float* lse2;    // [B, H, S]
  const float* delta;   // [B, H, S]
  __nv_bfloat16* dk;    // [B, S, H, D]
  __nv_bfloat16* dv;    // [B, S, H, DV]
  int S, H, n_kt;
  float scale, scale_log2;
  int heads_per_group;
  int* err;
};

// CTA -> ((batch, head), key tile in descending order of work).  Groups of heads that fill the SMs about once run one after the
// other, so that the operands and the dQ rows in use stay in L2: with all heads at once 10.7 GB went through DRAM at batch 4,
// seq 4096, of which 0.9 GB are needed (755 -> 700 us at batch 2).  The forward, whose operands are read only, keeps the order
// over all heads: its longest CTAs then start first over the whole grid (276 us against 314 in groups).
__device__ __forceinline__ void decode_cta(int x, int tiles, int heads, int per_group, int& bh, int& tile) {
  const int grp = x / (per_group * tiles), in = x - grp * per_group * tiles;
  const int n = min(per_group, heads - grp * per_group);
  tile = in / n;
  bh = grp * per_group + in - tile * n;
}

constexpr int BWD_THREADS = 448;          // warps 0-7: P and dS (warp >> 2 = half of the key columns); 8-11: dQ; 12: MMA; 13: TMA

struct BwdShared {
  uint64_t kv_full, q_full[2], q_empty[2];
  uint64_t sdp_full, sdp_free;              // S and dP multiplied / read into registers
  uint64_t pds_full, pds_free;              // P and dS written to shared memory / read by the products
  uint64_t dq_full, dq_free;                // a 64-column half of dQ multiplied / read
  uint64_t acc_done;
  uint32_t tmem_slot;
  int abort_flag;
};

// K 2, V 1, Q 2 x 2, dO 2 x 1, P 2, dS 2 slabs and a dQ staging slab (32 rows x 32 fp32 columns per dQ warp)
constexpr int bwd_smem() { return 14 * SLAB + (int)sizeof(BwdShared) + 1024; }

__device__ __forceinline__ void reduce_add_2d(const CUtensorMap* map, const void* src, int c0, int c1) {
  asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(smem_u32(src)), "r"(c0), "r"(c1)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read_all() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

__global__ void __launch_bounds__(BWD_THREADS, 1) attn_bwd_kernel(const __grid_constant__ CUtensorMap tmQ,
                                                                  const __grid_constant__ CUtensorMap tmK,
                                                                  const __grid_constant__ CUtensorMap tmV,
                                                                  const __grid_constant__ CUtensorMap tmdO,
                                                                  const __grid_constant__ CUtensorMap tmdQ, const BwdArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem;                       // [128 keys x 128]
  uint8_t* sV = sK + 2 * SLAB;              // [128 keys x 64]
  uint8_t* sQ = sV + SLAB;                  // 2 stages x [128 queries x 128]
  uint8_t* sdO = sQ + 4 * SLAB;             // 2 stages x [128 queries x 64]
  uint8_t* sP = sdO + 2 * SLAB;             // [128 queries x 128 keys] bf16
  uint8_t* sdS = sP + 2 * SLAB;
  uint8_t* sdQ = sdS + 2 * SLAB;            // 4 warps x [32 queries x 32 fp32], 128-byte-swizzled
  BwdShared* sh = reinterpret_cast<BwdShared*>(sdQ + SLAB);

  int bh, kt;                               // key tile 0 has the longest loop
  decode_cta(blockIdx.x, a.n_kt, gridDim.x / a.n_kt, a.heads_per_group, bh, kt);
  const int h = bh % a.H, b = bh / a.H;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int k0 = kt * BK;
  volatile int* abort_flag = &sh->abort_flag;
  if (tid == 0) {
    mbar_init(&sh->kv_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&sh->q_full[s], 1);
      mbar_init(&sh->q_empty[s], 1);
    }
    mbar_init(&sh->sdp_full, 1);
    mbar_init(&sh->sdp_free, 8);
    mbar_init(&sh->pds_full, 8);
    mbar_init(&sh->pds_free, 1);
    mbar_init(&sh->dq_full, 1);
    mbar_init(&sh->dq_free, 4);
    mbar_init(&sh->acc_done, 1);
    sh->abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 12) { tmem_alloc(&sh->tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  const bool drain = setup_barrier(a.err);
  tc_fence_after();
  const uint32_t tmem = sh->tmem_slot;
  if (drain) {
    if (warp == 12) tmem_dealloc(tmem, 512);
    return;
  }
  const uint32_t tS = tmem, tdP = tmem + 128, tdV = tmem + 256, tdK = tmem + 320, tdQ = tmem + 448;
  const uint32_t lane_addr = uint32_t((warp & 3) * 32) << 16;
  const int row0 = b * a.S;
  const int n_it = a.n_kt - kt;              // query tiles kt .. n_kt - 1

  if (warp == 13) {
    // ------------------------------ TMA producer ------------------------------
    if (elect_one()) {
      mbar_expect_tx(&sh->kv_full, 3 * SLAB);
      tma_load_2d(sK, &tmK, &sh->kv_full, h * D, row0 + k0);
      tma_load_2d(sK + SLAB, &tmK, &sh->kv_full, h * D + 64, row0 + k0);
      tma_load_2d(sV, &tmV, &sh->kv_full, h * DV, row0 + k0);
      for (int it = 0; it < n_it; ++it) {
        const int s = it & 1, qrow = row0 + (kt + it) * BQ;
        if (!mbar_wait(&sh->q_empty[s], ((it >> 1) & 1) ^ 1, abort_flag, a.err, ERR_WAIT_EMPTY)) break;
        mbar_expect_tx(&sh->q_full[s], 3 * SLAB);
        tma_load_2d(sQ + s * 2 * SLAB, &tmQ, &sh->q_full[s], h * D, qrow);
        tma_load_2d(sQ + s * 2 * SLAB + SLAB, &tmQ, &sh->q_full[s], h * D + 64, qrow);
        tma_load_2d(sdO + s * SLAB, &tmdO, &sh->q_full[s], h * DV, qrow);
      }
    }
  } else if (warp == 12) {
    // ------------------------------ MMA issuer ------------------------------
    if (elect_one()) {
      constexpr uint32_t id_s = umma_idesc_bf16(BQ, BK, false, false);
      constexpr uint32_t id_dv = umma_idesc_bf16(BK, DV, true, true);     // dV [keys x 64] += P^T dO
      constexpr uint32_t id_dk = umma_idesc_bf16(BK, D, true, true);      // dK [keys x 128] += dS^T Q
      constexpr uint32_t id_dq = umma_idesc_bf16(BQ, 64, false, true);    // half of dQ [queries x 128] = dS K
      const uint32_t aK = smem_u32(sK), aV = smem_u32(sV), aP = smem_u32(sP), adS = smem_u32(sdS);
      auto scores = [&](int it) {            // S = Q K^T and dP = dO V^T of query tile `it`
        const int s = it & 1;
        const uint32_t aQ = smem_u32(sQ + s * 2 * SLAB), adO = smem_u32(sdO + s * SLAB);
        if (!mbar_wait(&sh->q_full[s], (it >> 1) & 1, abort_flag, a.err, ERR_WAIT_FULL)) return false;
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < D / 16; ++k) umma_f16(tS, desc_k(aQ, k), desc_k(aK, k), id_s, k != 0);
#pragma unroll
        for (int k = 0; k < DV / 16; ++k)                                 // both K-major over the 64 value dims
          umma_f16(tdP, umma_desc_sw128(adO + k * 32, 16, 1024), umma_desc_sw128(aV + k * 32, 16, 1024), id_s, k != 0);
        umma_commit(&sh->sdp_full);
        return true;
      };
      auto dq_half = [&](int half) {         // columns 64 half .. 64 half + 63: one slab of K, read MN-major
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) umma_f16(tdQ, desc_k(adS, k), desc_mn1(aK + half * SLAB, k), id_dq, k != 0);
        umma_commit(&sh->dq_full);
      };
      bool ok = mbar_wait(&sh->kv_full, 0, abort_flag, a.err, ERR_WAIT_FULL) && scores(0);
      for (int it = 0; it < n_it && ok; ++it) {
        const uint32_t aQ = smem_u32(sQ + (it & 1) * 2 * SLAB), adO = smem_u32(sdO + (it & 1) * SLAB);
        if (it + 1 < n_it) {
          ok = mbar_wait(&sh->sdp_free, it & 1, abort_flag, a.err, ERR_WAIT_TMEM_EMPTY);
          tc_fence_after();
          ok = ok && scores(it + 1);
          if (!ok) break;
        }
        ok = mbar_wait(&sh->pds_full, it & 1, abort_flag, a.err, ERR_WAIT_TMEM_EMPTY);
        // dq_free completes twice a tile; the first half of this tile follows the second of the previous one
        if (ok && it > 0) ok = mbar_wait(&sh->dq_free, 1, abort_flag, a.err, ERR_WAIT_TMEM_EMPTY);
        if (!ok) break;
        tc_fence_after();
        dq_half(0);
#pragma unroll
        for (int k = 0; k < BQ / 16; ++k) umma_f16(tdV, desc_mn2(aP, k), desc_mn1(adO, k), id_dv, (it | k) != 0);
#pragma unroll
        for (int k = 0; k < BQ / 16; ++k) umma_f16(tdK, desc_mn2(adS, k), desc_mn2(aQ, k), id_dk, (it | k) != 0);
        umma_commit(&sh->q_empty[it & 1]);
        ok = mbar_wait(&sh->dq_free, 0, abort_flag, a.err, ERR_WAIT_TMEM_EMPTY);
        if (!ok) break;
        tc_fence_after();
        dq_half(1);
        umma_commit(&sh->pds_free);
      }
      if (ok) umma_commit(&sh->acc_done);
    }
  } else if (warp >= 8) {
    // ------------------------------ dQ: TMEM -> shared memory -> reductions into global memory ------------------------------
    uint8_t* stage = sdQ + (warp - 8) * 4096;
    bool ok = true;
    for (int n = 0; n < 2 * n_it; ++n) {
      ok = warp_wait(&sh->dq_full, n & 1, abort_flag, a.err, ERR_WAIT_TMEM_FULL);
      if (!ok) break;
      tc_fence_after();
      uint32_t r[2][32];
      tmem_ld_32x32(tdQ + lane_addr, r[0]);
      tmem_ld_32x32(tdQ + lane_addr + 32, r[1]);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh->dq_free);
      const int qrow = row0 + (kt + (n >> 1)) * BQ + (warp - 8) * 32;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        if (lane == 0) bulk_wait_read_all();        // the engine has read the previous box out of the staging rows
        __syncwarp();
#pragma unroll
        for (int v = 0; v < 8; ++v)
          *reinterpret_cast<uint4*>(stage + sw_off(lane, v)) = make_uint4(r[c][4 * v], r[c][4 * v + 1], r[c][4 * v + 2], r[c][4 * v + 3]);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          reduce_add_2d(&tmdQ, stage, h * D + (n & 1) * 64 + c * 32, qrow);
          bulk_commit();
        }
      }
    }
    if (lane == 0) bulk_wait_all();                 // this warp's reductions have reached memory
    __syncwarp();
  } else {
    // ------------------------------ P and dS ------------------------------
    const int half = warp >> 2, r = tid & 127;
    const size_t stat = ((size_t)b * a.H + h) * a.S + (size_t)kt * BQ + r;
    float lse = a.lse2[stat], dlt = a.delta[stat];
    auto tile = [&](int it, auto where) {
      constexpr bool DIAG = decltype(where)::value;         // columns past the row drop out
      float lse_next = 0.f, dlt_next = 0.f;
      if (it + 1 < n_it) { lse_next = a.lse2[stat + (size_t)(it + 1) * BQ]; dlt_next = a.delta[stat + (size_t)(it + 1) * BQ]; }
      if (!warp_wait(&sh->sdp_full, it & 1, abort_flag, a.err, ERR_WAIT_TMEM_FULL)) return false;
      tc_fence_after();
      uint32_t pp[2][16], dd[2][16];                // bf16 pairs of this thread's 64 columns
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int col0 = half * 64 + c * 32;
        uint32_t rs[32], rp[32];
        tmem_ld_32x32(tS + lane_addr + col0, rs);
        tmem_ld_32x32(tdP + lane_addr + col0, rp);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          float x = ex2(fmaf(__uint_as_float(rs[2 * e]), a.scale_log2, -lse));
          float y = ex2(fmaf(__uint_as_float(rs[2 * e + 1]), a.scale_log2, -lse));
          if (DIAG) {
            x = col0 + 2 * e <= r ? x : 0.f;
            y = col0 + 2 * e + 1 <= r ? y : 0.f;
          }
          pp[c][e] = pack_bf16(x, y);
          dd[c][e] = pack_bf16(x * (__uint_as_float(rp[2 * e]) - dlt) * a.scale, y * (__uint_as_float(rp[2 * e + 1]) - dlt) * a.scale);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh->sdp_free);
      if (it > 0 && !warp_wait(&sh->pds_free, (it - 1) & 1, abort_flag, a.err, ERR_WAIT_EMPTY)) return false;
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const int off = half * SLAB + sw_off(r, c * 4 + v);
          *reinterpret_cast<uint4*>(sP + off) = make_uint4(pp[c][4 * v], pp[c][4 * v + 1], pp[c][4 * v + 2], pp[c][4 * v + 3]);
          *reinterpret_cast<uint4*>(sdS + off) = make_uint4(dd[c][4 * v], dd[c][4 * v + 1], dd[c][4 * v + 2], dd[c][4 * v + 3]);
        }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh->pds_full);
      lse = lse_next;
      dlt = dlt_next;
      return true;
    };
    bool ok = tile(0, Diagonal{});
    for (int it = 1; it < n_it && ok; ++it) ok = tile(it, Interior{});
    ok = ok && warp_wait(&sh->acc_done, 0, abort_flag, a.err, ERR_WAIT_TMEM_FULL);
    if (ok) {
      tc_fence_after();
      __nv_bfloat16* krow = a.dk + ((size_t)(row0 + k0 + r) * a.H + h) * D + half * 64;
      __nv_bfloat16* vrow = a.dv + ((size_t)(row0 + k0 + r) * a.H + h) * DV + half * 32;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        uint32_t x[32];
        tmem_ld_32x32((c < 2 ? tdK + half * 64 + c * 32 : tdV + half * 32) + lane_addr, x);
        tmem_ld_wait();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float f[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(x[q * 8 + e]);
          reinterpret_cast<uint4*>(c < 2 ? krow + c * 32 : vrow)[q] = pack8f(f);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(2000);      // copies in flight land before the shared memory is released
    __syncthreads();
  }
  if (warp == 12) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

}  // namespace attn
}  // namespace cm

using namespace cm;
using namespace cm::attn;

static int attn_shape_ok(int B, int S, int H, int Dq, int Dv) {
  if (Dq != D || Dv != DV || S % BQ || H <= 0) return 0;
  if ((long long)B * S > 0x7fffffffLL / 4) return 0;
  return 1;
}

// q, k [B,S,H,128] bf16, v [B,S,H,64] bf16 (all packed) -> out [B,S,H,64] bf16, lse2 [B,H,S] fp32 (log2 domain).  S % 128 == 0.
extern "C" int cm_attn_fwd(const void* q, const void* k, const void* v, void* out, float* lse2, int B, int S, int H, int Dq,
                           int Dv, float scale, int* err, cudaStream_t stream) {
  if (B <= 0 || S <= 0) return 0;
  if (!attn_shape_ok(B, S, H, Dq, Dv)) return -10;
  CUtensorMap tmQ, tmK, tmV;
  const uint64_t rows = (uint64_t)B * S;
  int rc = make_tmap_2d_bf16(&tmQ, q, rows, (uint64_t)H * D, (uint64_t)H * D, BQ, 64);
  if (rc) return rc;
  rc = make_tmap_2d_bf16(&tmK, k, rows, (uint64_t)H * D, (uint64_t)H * D, BK, 64);
  if (rc) return rc;
  rc = make_tmap_2d_bf16(&tmV, v, rows, (uint64_t)H * DV, (uint64_t)H * DV, BK, 64);
  if (rc) return rc;
  static PerDevice cfg;
  if (cfg.first()) {
    if (cudaFuncSetAttribute(attn_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, fwd_smem()) != cudaSuccess) return -2;
    cfg.done();
  }
  const int n_qt = S / BQ;
  FwdArgs a{(__nv_bfloat16*)out, lse2, S, H, n_qt, scale * 1.4426950408889634f, err};
  attn_fwd_kernel<<<(unsigned)((n_qt + 1) / 2 * B * H), FWD_THREADS, fwd_smem(), stream>>>(tmQ, tmK, tmV, a);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

// delta [B,H,S] fp32 scratch; dq_acc [B,S,H,128] fp32 ZEROED by the caller (query gradients are reduced into it);
// dk [B,S,H,128], dv [B,S,H,64] bf16 are written.
extern "C" int cm_attn_bwd(const void* q, const void* k, const void* v, const void* o, const void* dout, const float* lse2,
                           float* delta, float* dq_acc, void* dk, void* dv, int B, int S, int H, int Dq, int Dv, float scale,
                           int* err, cudaStream_t stream) {
  if (B <= 0 || S <= 0) return 0;
  if (!attn_shape_ok(B, S, H, Dq, Dv)) return -10;
  CUtensorMap tmQ, tmK, tmV, tmdO;
  const uint64_t rows = (uint64_t)B * S;
  int rc = make_tmap_2d_bf16(&tmQ, q, rows, (uint64_t)H * D, (uint64_t)H * D, BQ, 64);
  if (rc) return rc;
  rc = make_tmap_2d_bf16(&tmK, k, rows, (uint64_t)H * D, (uint64_t)H * D, BK, 64);
  if (rc) return rc;
  rc = make_tmap_2d_bf16(&tmV, v, rows, (uint64_t)H * DV, (uint64_t)H * DV, BK, 64);
  if (rc) return rc;
  rc = make_tmap_2d_bf16(&tmdO, dout, rows, (uint64_t)H * DV, (uint64_t)H * DV, BQ, 64);
  if (rc) return rc;
  EncodeTiledFn enc = get_encode_tiled();
  if (!enc) return -1;
  CUtensorMap tmdQ;                       // fp32 [B*S, H*128], boxes of 32 rows x 32 columns
  {
    cuuint64_t dims[2] = {(cuuint64_t)H * D, rows}, strides[1] = {(cuuint64_t)H * D * 4};
    cuuint32_t box[2] = {32, 32}, one[2] = {1, 1};
    CUresult r = enc(&tmdQ, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, dq_acc, dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return int(r);
  }
  static PerDevice cfg;
  if (cfg.first()) {
    if (cudaFuncSetAttribute(attn_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bwd_smem()) != cudaSuccess) return -2;
    cfg.done();
  }
  const long long nrows = (long long)rows * H;
  attn_delta_kernel<<<(unsigned)((nrows + 31) / 32), 256, 0, stream>>>((const __nv_bfloat16*)o, (const __nv_bfloat16*)dout, delta,
                                                                      nrows, S, H);
  const int n_kt = S / BK;
  BwdArgs a{lse2, delta, (__nv_bfloat16*)dk, (__nv_bfloat16*)dv, S, H, n_kt, scale, scale * 1.4426950408889634f,
            (sm_count() + n_kt - 1) / n_kt, err};
  attn_bwd_kernel<<<(unsigned)(n_kt * B * H), BWD_THREADS, bwd_smem(), stream>>>(tmQ, tmK, tmV, tmdO, tmdQ, a);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}
