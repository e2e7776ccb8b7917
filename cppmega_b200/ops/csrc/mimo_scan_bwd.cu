// Mamba3 MIMO scan, backward (see mimo_common.cuh for the forward math and notation).
//
//   grad_state   per chunk:  Gc = Qr^T (e^{cs} o dO),  dO[4t+r] = dy[t] * Phi[r] * silu(Z[t] Zeta[r])
//   state_scan   per (b,h), reverse:  dEnd_c = dStart_{c+1},  dStart_c = e^{tot_c} dEnd_c + Gc
//   chunk_grad   per chunk: everything else, on tcgen05 with all accumulators in TMEM:
//       phase 1  S1 = Qr Kr^T | dPm = dO PV^T | O2 = Qr St | X = Kr dEnd | dQb = dO St^T
//       phase A  M, Pm = S1 o M, dS1 = dPm o M -> smem (bf16);  scalar gradients from dPm o S1
//       phase 2  O1 = Pm PV | dPV1 = Pm^T dO | dQ = dS1 Kr
//       epil. B  O = O1 + e O2 + D PV -> dPhi, dZeta, dZ;  dPV = dPV1 + D dO + w X -> dV, dPsi, dD;  dw, de
//       phase 3  dK = dS1^T Qr + (w o PV) dEnd^T
//       epil. C  dQr = dQ + e dQb, dKr;  inverse rotation -> per-head dQ/dK rows, d(angles)
//   Per-token scalar gradients (d cs, d ts, d gamma) are reduced in shared memory and written as
//   d(ADT) (reverse cumulative sum), d(ts), d(gamma) [B,H,S].
// Replaces the two TileLang backward kernels of the reference (bwd_fwd state recompute + bwd_bwd,
// cppmega/megatron/tilelang_mimo_autograd.py:160-219; mathematics restated at
// cppmega/megatron/cute_dsl_mimo/full_bwd_bwd_epilogue.py:9-348).
#include "mimo_common.cuh"

namespace cm {
namespace mimo {

__device__ __forceinline__ void tma_load_5d_b(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2,
                                              int c3, int c4) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2),
      "r"(c3), "r"(c4)
      : "memory");
}

struct BwdArgs {
  const __nv_bfloat16* V;       // [B,S,H,P]
  const __nv_bfloat16* Z;
  const __nv_bfloat16* dY;      // [B,S,H,P]
  const float* ADT;             // [B,H,S]
  const float* DT;
  const float* Trap;
  const float* Qb;              // [H,R,N]
  const float* Kb;
  const float* Psi;             // [H,R,P]
  const float* Zeta;
  const float* Phi;
  const float* angles;          // [B,S,H,NROT]
  const float* Dskip;           // [H]
  float* gbuf;                  // [B,H,C,N,P] fp32 (grad_state output)
  __nv_bfloat16* dQh;           // [B,S,H,R,N]
  __nv_bfloat16* dKh;
  __nv_bfloat16* dV;            // [B,S,H,P]
  __nv_bfloat16* dZ;
  float* dAngles;               // [B,S,H,NROT]
  float* dADT;                  // [B,H,S]
  float* dTs;
  float* dGam;
  float* dPsi;                  // [H,R,P] (atomics)
  float* dZeta;
  float* dPhi;
  float* dD;                    // [H]
  float* dQb;                   // [H,R,N] sums over tokens of dQh / dKh (may be null); zeroed by grad_state like the four above
  float* dKb;
  int B, S, H, G, C;
  long long ldV, ldZ;           // token strides of V and Z in elements
  int* err;
  int total_blocks;             // B * H * C
};

__device__ __forceinline__ void decode_block_b(const BwdArgs& a, int x, int& b, int& g, int& c, int& h) {
  const int hpg = a.H / a.G;
  const int hl = x % hpg; x /= hpg;
  c = x % a.C; x /= a.C;
  g = x % a.G; x /= a.G;
  b = x;
  h = g * hpg + hl;
}
__device__ __forceinline__ void decode_block_b(const BwdArgs& a, int& b, int& g, int& c, int& h) {
  decode_block_b(a, (int)blockIdx.x, b, g, c, h);
}

// gating of this thread's row: gate[p] = Phi[r,p] * silu(Z[t,p] * Zeta[r,p]); also returns silu' pieces on demand
__device__ __forceinline__ void load_row_bf16(float (&x)[P], const __nv_bfloat16* __restrict__ base) {
  const uint4* v = reinterpret_cast<const uint4*>(base);
#pragma unroll
  for (int c = 0; c < P / 8; ++c) {
    float f[8];
    unpack8(v[c], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) x[c * 8 + j] = f[j];
  }
}

// this thread's half row (columns [wg*32, wg*32+32)) of a [.., P] bf16 tensor; `base` points at the row start
__device__ __forceinline__ void load_half_bf16(float (&x)[P / 2], const __nv_bfloat16* __restrict__ base) {
  const uint4* v = reinterpret_cast<const uint4*>(base + (threadIdx.x >> 7) * 32);
#pragma unroll
  for (int c = 0; c < P / 16; ++c) {
    float f[8];
    unpack8(v[c], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) x[c * 8 + j] = f[j];
  }
}

constexpr int NROT_MAX = 32;
constexpr int THREADS2 = 256;      // two warpgroups: thread (i = tid & 127, wg = tid >> 7) owns half of fused row i

// ------------------------------------------------------------------------------------------
// grad_state: Gc[n,p] = sum_i Qr[i,n] e^{cs_ti} dO[i,p]
// ------------------------------------------------------------------------------------------
template <int N, int NROT>
__global__ void __launch_bounds__(THREADS2) mimo_grad_state_kernel(const __grid_constant__ CUtensorMap tmQ, const BwdArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int QT = (N / 64) * SLAB;
  uint8_t* sQ = smem;
  uint8_t* sdO = sQ + QT;
  float* cos_tab = reinterpret_cast<float*>(sdO + SLAB);
  float* sin_tab = cos_tab + tab_floats<NROT>();
  HeadBias<N>* hb = reinterpret_cast<HeadBias<N>*>(sin_tab + tab_floats<NROT>());
  HeadVecs* hv = reinterpret_cast<HeadVecs*>(hb + 1);
  ChunkScalars* sc = reinterpret_cast<ChunkScalars*>(hv + 1);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sc + 1);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int b, g, c, h;
  decode_block_b(a, b, g, c, h);
  const int t0 = c * LT;
  const int i = threadIdx.x & 127, wg = threadIdx.x >> 7, t = i >> 2, r = i & 3, warp = threadIdx.x >> 5;
  if (b == 0 && c == 0) {                          // the accumulators of head h that later kernels add to
    static_assert(R * P == THREADS2 && R * N == 2 * THREADS2, "one element of each [R,P] vector per thread");
    a.dPsi[h * R * P + threadIdx.x] = 0.f;
    a.dZeta[h * R * P + threadIdx.x] = 0.f;
    a.dPhi[h * R * P + threadIdx.x] = 0.f;
    if (threadIdx.x == 0) a.dD[h] = 0.f;
    if (a.dQb) {
      reinterpret_cast<float2*>(a.dQb + (size_t)h * R * N)[threadIdx.x] = make_float2(0.f, 0.f);
      reinterpret_cast<float2*>(a.dKb + (size_t)h * R * N)[threadIdx.x] = make_float2(0.f, 0.f);
    }
  }
  // every global load of the prologue is issued here, ahead of the set-up, and consumed further down
  const ScalarLoads sl = load_chunk_scalars(a.ADT, a.DT, a.Trap, ((size_t)b * a.H + h) * a.S + t0, t0, a.S);
  const float4 ang4 = load_angles4<NROT>(a.angles, b, t0, h, a.S, a.H);
  const HalfRowRaw yraw = load_half_raw(a.dY, b, t0, h, a.S, (long long)a.H * P);
  const HalfRowRaw zraw = load_half_raw(a.Z, b, t0, h, a.S, a.ldZ);
  const float* qbh = a.Qb + (size_t)h * R * N + 2 * threadIdx.x;
  const float qb0 = qbh[0], qb1 = qbh[1];
  const float zeta1 = a.Zeta[(size_t)h * R * P + threadIdx.x], phi1 = a.Phi[(size_t)h * R * P + threadIdx.x];
  if (threadIdx.x == 0) {
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 0) { tmem_alloc(tmem_slot, 64); tmem_relinquish(); }
  tc_fence_before();
  const bool drain = setup_barrier(a.err);
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  if (drain) {
    if (warp == 0) tmem_dealloc(tmem, 64);
    return;
  }
  if (threadIdx.x == 0) {
    mbar_expect_tx(&bars[0], QT);
#pragma unroll
    for (int s = 0; s < N / 64; ++s) tma_load_5d_b(sQ + s * SLAB, &tmQ, &bars[0], s * 64, 0, g, t0, b);
  }
  {
    const int bias_at = (2 * threadIdx.x / N) * HeadBias<N>::LD + 2 * threadIdx.x % N;
    hb->qb[bias_at] = qb0;
    hb->qb[bias_at + 1] = qb1;
    hv->zeta[vec_idx(threadIdx.x)] = zeta1;
    hv->phi[vec_idx(threadIdx.x)] = phi1;
  }
  finish_chunk_scalars(sc, sl, t0, a.S);
  fill_sincos4<NROT>(cos_tab, sin_tab, ang4);
  __syncthreads();
  bool ok = mbar_wait(&bars[0], 0, abort_flag, a.err, ERR_WAIT_FULL);
  if (ok) {
    transform_rows<N, NROT, 2, HeadBias<N>::LD>(sQ, hb->qb, cos_tab, sin_tab);
    float dy[P / 2], z[P / 2];
    half_raw_to_float(dy, yraw);
    half_raw_to_float(z, zraw);
    const float* zeta = hv->zeta + r * VLD + wg * 32;
    const float* phi = hv->phi + r * VLD + wg * 32;
    const float e = __expf(sc->cs[t]);
#pragma unroll
    for (int p = 0; p < P / 2; ++p) dy[p] = dy[p] * phi[p] * fast_silu(z[p] * zeta[p]);
    store_half64(sdO, dy, e);
    fence_proxy_async_smem();
  }
  __syncthreads();
  if (threadIdx.x == 0 && !*abort_flag) {
    constexpr uint32_t idesc = umma_idesc_bf16(N, P, true, true);
    const uint32_t aQ = smem_u32(sQ), aO = smem_u32(sdO);
#pragma unroll
    for (int k = 0; k < ROWS / 16; ++k) umma_f16(tmem, desc_mnmajor_2slab(aQ, k), desc_mnmajor_rows(aO, k), idesc, k != 0);
    umma_commit(&bars[1]);
  }
  ok = mbar_wait(&bars[1], 0, abort_flag, a.err, ERR_WAIT_TMEM_FULL);
  tc_fence_after();
  static_assert(N == ROWS, "one TMEM lane per state row");
  store_state_tile(a.gbuf + (((size_t)b * a.H + h) * a.C + c) * N * P, sQ, tmem, ok);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) { tc_fence_after(); tmem_dealloc(tmem, 64); }
}

// reverse scan: dEnd[c] = state; state = e^{tot_c} state + G[c]  for c = C-1 .. 0
__global__ void __launch_bounds__(256) mimo_state_scan_rev_kernel(const float* __restrict__ gbuf, const float* __restrict__ tot,
                                                                  __nv_bfloat16* __restrict__ dend, int C, int NP) {
  const size_t bh = blockIdx.x;
  const int e = (blockIdx.y * 256 + threadIdx.x) * 4;
  if (e >= NP) return;
  float4 st = make_float4(0.f, 0.f, 0.f, 0.f);
  const float* gp = gbuf + bh * (size_t)C * NP + e;
  __nv_bfloat16* dp = dend + bh * (size_t)C * NP + e;
  const float* tp = tot + bh * C;
  for (int c = C - 1; c >= 0; --c) {
    const float4 cur = *reinterpret_cast<const float4*>(gp + (size_t)c * NP);
    uint2 o;
    o.x = pack_bf16(st.x, st.y);
    o.y = pack_bf16(st.z, st.w);
    *reinterpret_cast<uint2*>(dp + (size_t)c * NP) = o;
    const float d = __expf(tp[c]);
    st.x = d * st.x + cur.x; st.y = d * st.y + cur.y; st.z = d * st.z + cur.z; st.w = d * st.w + cur.w;
  }
}

// ------------------------------------------------------------------------------------------
// chunk_grad
// ------------------------------------------------------------------------------------------
// A chunk is a chain of phases on 8 warps (one CTA per SM: 228 KB of tiles, 255 registers), so instructions and latencies
// between its three products are its time (measured per phase: the products themselves are waited for 600 cycles of 48,000).
// Hence partial sums in slots of their own instead of shared-memory atomics, reductions that halve the values they exchange,
// head constants requested with the operands, and the next chunk's operands requested into L2 a chunk ahead:
// 2,532 -> 2,152 us for 16,384 chunks (B 1, S 4096, H 128).
struct GradScratch {
  float row[3][2][LT];       // d cs, d ts, d gamma of a token from its rows: one slot per warpgroup
  float dtot[8];             // one slot per warp
  float dD[8];
  float par[3][4][R][VLD];   // per-lane-quarter partials of dPsi, dZeta, dPhi (each warpgroup fills its own columns)
  alignas(16) float dang[LT][NROT_MAX + 4];  // K-side d(angle) partials (padded rows: eight tokens of a warp write one column) handed from warpgroup 1 to warpgroup 0
};

// Ask for the next chunk's operands while this one runs: they are in L2 when its turn comes.
__device__ __forceinline__ void prefetch_line(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ void prefetch_tile(const CUtensorMap* map, int c0, int c1) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1)
               : "memory");
}

template <int N, int NROT>
__global__ void __launch_bounds__(THREADS2, 1) mimo_chunk_grad_kernel(const __grid_constant__ CUtensorMap tmQ,
                                                                      const __grid_constant__ CUtensorMap tmK,
                                                                      const __grid_constant__ CUtensorMap tmS,
                                                                      const __grid_constant__ CUtensorMap tmE, const BwdArgs a) {
  static_assert(N == 128, "chunk_grad is written for a 128-wide state");
  static_assert(NROT <= NROT_MAX && NROT / 8 == R, "rank r writes the r-th group of eight angles");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;                    // 32 KB
  uint8_t* sK = sQ + 2 * SLAB;           // 32 KB
  uint8_t* sPV = sK + 2 * SLAB;          // 16 KB
  uint8_t* sdO = sPV + SLAB;             // 16 KB
  uint8_t* sSt = sdO + SLAB;             // 16 KB  start state [n x p]
  uint8_t* sdE = sSt + SLAB;             // 16 KB  gradient of the end state [n x p]
  uint8_t* sPm = sdE + SLAB;             // 32 KB
  uint8_t* sdS = sPm + 2 * SLAB;         // 32 KB
  uint8_t* sPVw = sdS + 2 * SLAB;        // 16 KB
  float* cos_tab = reinterpret_cast<float*>(sPVw + SLAB);
  float* sin_tab = cos_tab + tab_floats<NROT>();
  HeadVecs* hv = reinterpret_cast<HeadVecs*>(sin_tab + tab_floats<NROT>());
  ChunkScalars* sc = reinterpret_cast<ChunkScalars*>(hv + 1);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sc + 1);             // tma, ph1, ph2, ph3
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  // colsum [8 warps][2][16] floats follow the abort flag; the head biases and later the reduction scratch alias Pm
  // (biases die before phase A writes Pm; the scratch is used only after phase 2 has read it)
  static_assert(sizeof(GradScratch) <= 2 * SLAB && sizeof(HeadBias<N>) <= 2 * SLAB, "scratch must fit the Pm tile");

  const int tid = threadIdx.x;
  const int i = tid & 127, wg = tid >> 7, t = i >> 2, r = i & 3, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int q = 0; q < 4; ++q) mbar_init(&bars[q], 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 0) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  const bool drain = setup_barrier(a.err);
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  if (drain) {
    if (warp == 0) tmem_dealloc(tmem, 512);
    return;
  }
  // Persistent: one CTA per SM walks the chunks with a grid stride; barriers, TMEM and the kernel prologue are paid
  // once, and every barrier completes exactly one phase per chunk, so its parity is the iteration's low bit.
  uint32_t par = 0;
#pragma unroll 1
  for (int xblk = blockIdx.x; xblk < a.total_blocks; xblk += gridDim.x, par ^= 1) {
  // Re-derive every shared-memory address from a value the compiler cannot see through: otherwise the addresses and
  // the ~80 MMA descriptors built from them are hoisted out of this loop and spill the 255-register budget.
  uint8_t* smem_l;
  asm volatile("mov.u64 %0, %1;" : "=l"(smem_l) : "l"(smem));
  uint8_t* sQ = smem_l;
  uint8_t* sK = sQ + 2 * SLAB;
  uint8_t* sPV = sK + 2 * SLAB;
  uint8_t* sdO = sPV + SLAB;
  uint8_t* sSt = sdO + SLAB;
  uint8_t* sdE = sSt + SLAB;
  uint8_t* sPm = sdE + SLAB;
  uint8_t* sdS = sPm + 2 * SLAB;
  uint8_t* sPVw = sdS + 2 * SLAB;
  float* cos_tab = reinterpret_cast<float*>(sPVw + SLAB);
  float* sin_tab = cos_tab + tab_floats<NROT>();
  HeadVecs* hv = reinterpret_cast<HeadVecs*>(sin_tab + tab_floats<NROT>());
  ChunkScalars* sc = reinterpret_cast<ChunkScalars*>(hv + 1);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sc + 1);
  float* colsum = reinterpret_cast<float*>(reinterpret_cast<uint32_t*>(bars + 4) + 4);
  HeadBias<N>* hb = reinterpret_cast<HeadBias<N>*>(sPm);
  GradScratch* gs = reinterpret_cast<GradScratch*>(sPm);
  int b, g, c, h;
  decode_block_b(a, xblk, b, g, c, h);
  const int t0 = c * LT;
  // every global load of the prologue is issued here, ahead of the set-up, and consumed further down
  const ScalarLoads sl = load_chunk_scalars(a.ADT, a.DT, a.Trap, ((size_t)b * a.H + h) * a.S + t0, t0, a.S);
  const float4 ang4 = load_angles4<NROT>(a.angles, b, t0, h, a.S, a.H);
  const HalfRowRaw vraw = load_half_raw(a.V, b, t0, h, a.S, a.ldV);
  const HalfRowRaw yraw = load_half_raw(a.dY, b, t0, h, a.S, (long long)a.H * P);
  const HalfRowRaw zraw = load_half_raw(a.Z, b, t0, h, a.S, a.ldZ);
  static_assert(R * N == 2 * THREADS2 && R * P == THREADS2, "two bias elements and one of each [R,P] vector per thread");
  const float* qbh = a.Qb + (size_t)h * R * N + 2 * tid;
  const float* kbh = a.Kb + (size_t)h * R * N + 2 * tid;
  const float2 qb2 = make_float2(qbh[0], qbh[1]), kb2 = make_float2(kbh[0], kbh[1]);
  const float psi1 = a.Psi[h * R * P + tid], zeta1 = a.Zeta[h * R * P + tid], phi1 = a.Phi[h * R * P + tid];
  if (tid < 4 * LT && xblk + (int)gridDim.x < a.total_blocks) {
    int nb, ng, nc, nh;
    decode_block_b(a, xblk + gridDim.x, nb, ng, nc, nh);
    const size_t tok = (size_t)nb * a.S + nc * LT + (tid & 31);
    prefetch_line(warp == 0   ? (const void*)(a.V + tok * a.ldV + nh * P)
                  : warp == 1 ? (const void*)(a.dY + (tok * a.H + nh) * P)
                  : warp == 2 ? (const void*)(a.Z + tok * a.ldZ + nh * P)
                              : (const void*)(a.angles + (tok * a.H + nh) * NROT));
    if (tid == 0) {
      const int nrow = (int)((((size_t)nb * a.H + nh) * a.C + nc) * N);
      prefetch_tile(&tmS, 0, nrow);
      prefetch_tile(&tmE, 0, nrow);
    }
  }
  const uint32_t lane_addr = uint32_t((warp & 3) * 32) << 16;
  // phase 1 accumulators                      phase 2 / 3 accumulators
  const uint32_t tS1 = tmem, tdPm = tmem + 128, tO2 = tmem + 256, tX = tmem + 320, tdQb = tmem + 384;
  const uint32_t tO1 = tmem, tdPV1 = tmem + 64, tdQ = tmem + 128, tdK = tmem + 256;

  if (tid == 0) {
    mbar_expect_tx(&bars[0], 4 * SLAB + 2 * SLAB);
    for (int s = 0; s < 2; ++s) {
      tma_load_5d_b(sQ + s * SLAB, &tmQ, &bars[0], s * 64, 0, g, t0, b);
      tma_load_5d_b(sK + s * SLAB, &tmK, &bars[0], s * 64, 0, g, t0, b);
    }
    const int srow = (int)((((size_t)b * a.H + h) * a.C + c) * N);
    tma_load_2d(sSt, &tmS, &bars[0], 0, srow);
    tma_load_2d(sdE, &tmE, &bars[0], 0, srow);
  }
  {
    const int bias_at = (2 * tid / N) * HeadBias<N>::LD + 2 * tid % N;
    *reinterpret_cast<float2*>(hb->qb + bias_at) = qb2;
    *reinterpret_cast<float2*>(hb->kb + bias_at) = kb2;
    hv->psi[vec_idx(tid)] = psi1;
    hv->zeta[vec_idx(tid)] = zeta1;
    hv->phi[vec_idx(tid)] = phi1;
  }
  finish_chunk_scalars(sc, sl, t0, a.S);
  fill_sincos4<NROT>(cos_tab, sin_tab, ang4);
  __syncthreads();
  const size_t rowoff = (((size_t)b * a.S + t0 + t) * a.H + h) * P + wg * 32;     // this thread's half row
  const float* zeta = hv->zeta + r * VLD + wg * 32;
  const float* phi = hv->phi + r * VLD + wg * 32;
  const float* psi = hv->psi + r * VLD + wg * 32;
  const float csi = sc->cs[t], gi = sc->gam[t], tsi = sc->ts[t], tot = sc->tot;
  const float ei = __expf(csi);
  const float wi = tsi * __expf(tot - csi);
  const float dsk = a.Dskip[h];

  bool ok = mbar_wait(&bars[0], par, abort_flag, a.err, ERR_WAIT_FULL);
  if (ok) {
    transform_rows<N, NROT, 2, HeadBias<N>::LD>(sQ, hb->qb, cos_tab, sin_tab);
    transform_rows<N, NROT, 2, HeadBias<N>::LD>(sK, hb->kb, cos_tab, sin_tab);
    {
      float pv[P / 2];
      pv_from_raw(pv, vraw, hv->psi);
      store_half64(sPV, pv, 1.f);
      store_half64(sPVw, pv, wi);
    }
    {
      float dy[P / 2], z[P / 2];
      half_raw_to_float(dy, yraw);
      half_raw_to_float(z, zraw);
#pragma unroll
      for (int p = 0; p < P / 2; ++p) dy[p] = dy[p] * phi[p] * fast_silu(z[p] * zeta[p]);
      store_half64(sdO, dy, 1.f);
    }
    fence_proxy_async_smem();
  }
  __syncthreads();
  const uint32_t aQ = smem_u32(sQ), aK = smem_u32(sK), aPV = smem_u32(sPV), adO = smem_u32(sdO), aSt = smem_u32(sSt),
                 adE = smem_u32(sdE), aPm = smem_u32(sPm), adS = smem_u32(sdS), aPVw = smem_u32(sPVw);
  constexpr uint32_t id_128_kk = umma_idesc_bf16(ROWS, 128, false, false);
  constexpr uint32_t id_64_km = umma_idesc_bf16(ROWS, P, false, true);
  constexpr uint32_t id_64_mm = umma_idesc_bf16(ROWS, P, true, true);
  constexpr uint32_t id_128_km = umma_idesc_bf16(ROWS, 128, false, true);
  constexpr uint32_t id_128_mm = umma_idesc_bf16(ROWS, 128, true, true);
  if (tid == 0 && !*abort_flag) {
#pragma unroll
    for (int k = 0; k < 8; ++k) umma_f16(tS1, desc_kmajor(aQ, k), desc_kmajor(aK, k), id_128_kk, k != 0);
#pragma unroll
    for (int k = 0; k < 4; ++k) umma_f16(tdPm, desc_kmajor(adO, k), desc_kmajor(aPV, k), id_128_kk, k != 0);
#pragma unroll
    for (int k = 0; k < 8; ++k) umma_f16(tO2, desc_kmajor(aQ, k), desc_mnmajor_rows(aSt, k), id_64_km, k != 0);
#pragma unroll
    for (int k = 0; k < 8; ++k) umma_f16(tX, desc_kmajor(aK, k), desc_mnmajor_rows(adE, k), id_64_km, k != 0);
#pragma unroll
    for (int k = 0; k < 4; ++k) umma_f16(tdQb, desc_kmajor(adO, k), desc_kmajor(aSt, k), id_128_kk, k != 0);
    umma_commit(&bars[1]);
  }
  // while the tensor core works: d tot from the state decay, e^{tot} * <dEnd, St> (state row n = i, half of its columns)
  float dtot_part = 0.f;
  if (ok) {
#pragma unroll
    for (int c2 = 0; c2 < 4; ++c2) {
      const int cidx = wg * 4 + c2;
      float s8[8], e8[8];
      unpack8(*reinterpret_cast<const uint4*>(sSt + sw_off(i, cidx)), s8);
      unpack8(*reinterpret_cast<const uint4*>(sdE + sw_off(i, cidx)), e8);
#pragma unroll
      for (int j = 0; j < 8; ++j) dtot_part += s8[j] * e8[j];
    }
    dtot_part *= __expf(tot);
  }
  ok = __syncthreads_and(mbar_wait(&bars[1], par, abort_flag, a.err, ERR_WAIT_TMEM_FULL));
  tc_fence_after();

  // ---------------- phase A: masks, Pm, dS1, scalar gradients from dM = dPm o S1 ----------------
  // this warpgroup's key tokens: [16 wg, 16 wg + 16)
  float rowR = 0.f, dgam_i = 0.f;
  float col_part[LT];                // column sums of dM o M (0..15) and dM o e^{..} (16..31) for this warpgroup's key tokens
  if (ok) {
#pragma unroll
    for (int c2 = 0; c2 < 2; ++c2) {
      const int cc = wg * 2 + c2;
      uint32_t s1[32], dp[32];
      tmem_ld_32x32(tS1 + lane_addr + cc * 32, s1);
      tmem_ld_32x32(tdPm + lane_addr + cc * 32, dp);
      tmem_ld_wait();
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float fp[8], fd[8];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int tl = c2 * 8 + q * 2 + u;          // local key-token index, 0..15
          const int tj = wg * 16 + tl;
          float ex = 0.f, m = 0.f;
          if (tj < t) { ex = __expf(csi - sc->cs[tj]); m = sc->ts[tj] * ex; }
          else if (tj == t) m = gi;
          float dmsum = 0.f;
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            const float sv = __uint_as_float(s1[q * 8 + u * 4 + v]);
            const float dv = __uint_as_float(dp[q * 8 + u * 4 + v]);
            fp[u * 4 + v] = sv * m;
            fd[u * 4 + v] = dv * m;
            dmsum += sv * dv;
          }
          if (tj < t) {
            rowR += dmsum * m;
            col_part[tl] = dmsum * m;
            col_part[16 + tl] = dmsum * ex;
          } else {
            col_part[tl] = 0.f;
            col_part[16 + tl] = 0.f;
            if (tj == t) dgam_i += dmsum;
          }
        }
        const int col = cc * 32 + q * 8;
        *reinterpret_cast<uint4*>(sPm + (col / 64) * SLAB + sw_off(i, (col % 64) / 8)) = pack8(fp);
        *reinterpret_cast<uint4*>(sdS + (col / 64) * SLAB + sw_off(i, (col % 64) / 8)) = pack8(fd);
      }
    }
    fence_proxy_async_smem();
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && !*abort_flag) {
    tc_fence_after();
#pragma unroll
    for (int k = 0; k < 8; ++k) umma_f16(tO1, desc_kmajor(aPm, k), desc_mnmajor_rows(aPV, k), id_64_km, k != 0);
#pragma unroll
    for (int k = 0; k < 8; ++k) umma_f16(tdPV1, desc_mnmajor_2slab(aPm, k), desc_mnmajor_rows(adO, k), id_64_mm, k != 0);
#pragma unroll
    for (int k = 0; k < 8; ++k) umma_f16(tdQ, desc_kmajor(adS, k), desc_mnmajor_2slab(aK, k), id_128_km, k != 0);
    umma_commit(&bars[2]);
  }
  // column sums over the rows of this warp while phase 2 runs
  if (ok) {
    colsum[warp * LT + lane] = xreduce32<false>(col_part, lane);
  }
  ok = __syncthreads_and(mbar_wait(&bars[2], par, abort_flag, a.err, ERR_WAIT_TMEM_FULL));
  tc_fence_after();
  // Pm has been consumed by phase 2: its space becomes the reduction scratch

  // ---------------- epilogue B: gating gradients, dPV, dw, de (this warpgroup's 32 columns) ----------------
  float dw_i = 0.f, de_i = 0.f;
  if (ok) {
    const uint4* vrow = vraw.v;
    const uint4* yrow = yraw.v;
    const uint4* zrow = zraw.v;
    const int wq = warp & 3;
    float dD_part = 0.f;
    float dvrow[32];
    const int pcol = reduce8_first_col(lane);         // first of the two columns (per 16) this lane owns after reduce8
    {   // pass 1: O = O1 + e O2 + D PV  ->  dPhi, dZeta, dZ, de, dD and the D dO part of dPV
      uint32_t o1[32], o2[32];
      tmem_ld_32x32(tO1 + lane_addr + wg * 32, o1);
      tmem_ld_32x32(tO2 + lane_addr + wg * 32, o2);
      tmem_ld_wait();
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        float aphi[16], azeta[16], apsi[16], adz[16];
#pragma unroll
        for (int q2 = 0; q2 < 2; ++q2) {
          const int q = half * 2 + q2;
          float vf[8], yf[8], zf[8];
          unpack8(vrow[q], vf);
          unpack8(yrow[q], yf);
          unpack8(zrow[q], zf);
#pragma unroll
          for (int v = 0; v < 8; ++v) {
            const int e = q * 8 + v, c = q2 * 8 + v;
            const float pvv = vf[v] * psi[e];
            const float o2v = __uint_as_float(o2[e]);
            const float o = __uint_as_float(o1[e]) + ei * o2v + dsk * pvv;
            const float zz = zf[v] * zeta[e];
            const float sg = __fdividef(1.f, 1.f + __expf(-zz));
            const float sil = zz * sg;
            const float dO = yf[v] * phi[e] * sil;
            const float dgate = yf[v] * o;
            const float dzz = dgate * phi[e] * sg * (1.f + zz * (1.f - sg));
            aphi[c] = dgate * sil;
            azeta[c] = dzz * zf[v];
            apsi[c] = dsk * dO * vf[v];
            adz[c] = dzz * zeta[e];
            de_i += dO * o2v;
            dD_part += dO * pvv;
            dvrow[e] = dsk * dO * psi[e];
          }
        }
        float r2[2], mz[4];
        const int col = wg * 32 + half * 16 + pcol;
        reduce8_keep2_of16(apsi, r2);
        gs->par[0][wq][r][col] = r2[0]; gs->par[0][wq][r][col + 1] = r2[1];
        reduce8_keep2_of16(azeta, r2);
        gs->par[1][wq][r][col] = r2[0]; gs->par[1][wq][r][col + 1] = r2[1];
        reduce8_keep2_of16(aphi, r2);
        gs->par[2][wq][r][col] = r2[0]; gs->par[2][wq][r][col + 1] = r2[1];
        reduce4_keep4_of16(adz, mz);
        uint2 oz;
        oz.x = pack_bf16(mz[0], mz[1]);
        oz.y = pack_bf16(mz[2], mz[3]);
        *reinterpret_cast<uint2*>(a.dZ + rowoff + half * 16 + r * 4) = oz;
      }
    }
    {   // pass 2: dPV = dPV1 + w X (+ D dO from pass 1)  ->  dV, dPsi, dw
      uint32_t d1[32], xx[32];
      tmem_ld_32x32(tdPV1 + lane_addr + wg * 32, d1);
      tmem_ld_32x32(tX + lane_addr + wg * 32, xx);
      tmem_ld_wait();
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        float apsi[16];
#pragma unroll
        for (int q2 = 0; q2 < 2; ++q2) {
          const int q = half * 2 + q2;
          float vf[8];
          unpack8(vrow[q], vf);
#pragma unroll
          for (int v = 0; v < 8; ++v) {
            const int e = q * 8 + v;
            const float xv = __uint_as_float(xx[e]);
            const float dpv = __uint_as_float(d1[e]) + wi * xv;
            dw_i += vf[v] * psi[e] * xv;
            apsi[q2 * 8 + v] = dpv * vf[v];
            dvrow[e] += dpv * psi[e];
          }
        }
        float r2[2];
        const int col = wg * 32 + half * 16 + pcol;
        reduce8_keep2_of16(apsi, r2);                 // same lane owns the same columns as in pass 1
        gs->par[0][wq][r][col] += r2[0]; gs->par[0][wq][r][col + 1] += r2[1];
      }
      float mv[8];
      reduce4_keep8(dvrow, mv);
      *reinterpret_cast<uint4*>(a.dV + rowoff + r * 8) = pack8(mv);
    }
    dD_part = warp_sum(dD_part);
    if (lane == 0) gs->dD[warp] = dD_part;
    // per-token scalar gradients (each warpgroup adds the part that comes from its columns)
    //   cs_ti:  + rowR + e_i de_i - w_i dw_i         ts_ti: + dw_i e^{tot-cs_ti}       gamma_ti: + dgam_i
    const float ewi = __expf(tot - csi);
    float dcs_row = rowR + ei * de_i - wi * dw_i;
    float dts_row = dw_i * ewi;
    float dgm_row = dgam_i;
    float dtot_row = wi * dw_i + dtot_part;
    dcs_row += __shfl_xor_sync(0xffffffffu, dcs_row, 1); dcs_row += __shfl_xor_sync(0xffffffffu, dcs_row, 2);
    dts_row += __shfl_xor_sync(0xffffffffu, dts_row, 1); dts_row += __shfl_xor_sync(0xffffffffu, dts_row, 2);
    dgm_row += __shfl_xor_sync(0xffffffffu, dgm_row, 1); dgm_row += __shfl_xor_sync(0xffffffffu, dgm_row, 2);
    dtot_row = warp_sum(dtot_row);
    if (r == 0) {
      gs->row[0][wg][t] = dcs_row;
      gs->row[1][wg][t] = dts_row;
      gs->row[2][wg][t] = dgm_row;
    }
    if (lane == 0) gs->dtot[warp] = dtot_row;
  }
  tc_fence_before();
  __syncthreads();
  // ---------------- phase 3: dK ----------------
  if (tid == 0 && !*abort_flag) {
    tc_fence_after();
#pragma unroll
    for (int k = 0; k < 8; ++k) umma_f16(tdK, desc_mnmajor_2slab(adS, k), desc_mnmajor_2slab(aQ, k), id_128_mm, k != 0);
#pragma unroll
    for (int k = 0; k < 4; ++k) umma_f16(tdK, desc_kmajor(aPVw, k), desc_kmajor(adE, k), id_128_kk, 1);
    umma_commit(&bars[3]);
  }
  // finish the scalar and parameter gradients while phase 3 runs
  if (ok) {
    if (warp == 0) {
      // d(ADT)[s] = sum_{t >= s} dcs[t]  (+ dtot on the last token)
      // token `lane`: the rows of both warpgroups, and the column sums of the four warps whose key tokens include it
      float v = gs->row[0][0][lane] + gs->row[0][1][lane], ts_ = gs->row[1][0][lane] + gs->row[1][1][lane], tot_ = 0.f;
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        v -= colsum[((lane >> 4) * 4 + w) * LT + (lane & 15)];
        ts_ += colsum[((lane >> 4) * 4 + w) * LT + 16 + (lane & 15)];
      }
#pragma unroll
      for (int w = 0; w < 8; ++w) tot_ += gs->dtot[w];
      if (lane == LT - 1) v += tot_;
#pragma unroll
      for (int o_ = 1; o_ < 32; o_ <<= 1) {
        const float n_ = __shfl_down_sync(0xffffffffu, v, o_);
        if (lane + o_ < 32) v += n_;
      }
      const size_t sb = ((size_t)b * a.H + h) * a.S + t0 + lane;
      a.dADT[sb] = v;
      a.dTs[sb] = ts_;
      a.dGam[sb] = gs->row[2][0][lane] + gs->row[2][1][lane];
    }
    {
      const int e = tid;                                   // R * P == 256 == THREADS2
      const int rr = e / P, pp = e % P;
      float s0 = 0.f, s1 = 0.f, s2 = 0.f;
#pragma unroll
      for (int w = 0; w < 4; ++w) { s0 += gs->par[0][w][rr][pp]; s1 += gs->par[1][w][rr][pp]; s2 += gs->par[2][w][rr][pp]; }
      atomicAdd(a.dPsi + (size_t)h * R * P + e, s0);
      atomicAdd(a.dZeta + (size_t)h * R * P + e, s1);
      atomicAdd(a.dPhi + (size_t)h * R * P + e, s2);
    }
    if (tid == THREADS2 - 1) {
      float d = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) d += gs->dD[w];
      atomicAdd(a.dD + h, d);
    }
  }
  ok = __syncthreads_and(mbar_wait(&bars[3], par, abort_flag, a.err, ERR_WAIT_TMEM_FULL));
  tc_fence_after();
  // ---------------- epilogue C: dQr = dQ + e dQb (warpgroup 0), dKr (warpgroup 1); inverse rotation; d(angles) ----
  float dang8[8];
  if (ok) {
    constexpr int HALF = N / 2;
    float dang[NROT];
    const bool isq = wg == 0;
    const uint8_t* tile = isq ? sQ : sK;                 // rotated operand rows (bf16) for d(angle)
    __nv_bfloat16* drow = (isq ? a.dQh : a.dKh) + ((((size_t)b * a.S + t0 + t) * a.H + h) * R + r) * N;
    const uint32_t tacc = isq ? tdQ : tdK;
    // columns [0,32) pair with [64,96); [32,64) and [96,128) are not rotated
    uint32_t lo[32], hi[32];
    tmem_ld_32x32(tacc + lane_addr + 0, lo);
    tmem_ld_32x32(tacc + lane_addr + HALF, hi);
    tmem_ld_wait();
    if (isq) {
      uint32_t lob[32], hib[32];
      tmem_ld_32x32(tdQb + lane_addr + 0, lob);
      tmem_ld_32x32(tdQb + lane_addr + HALF, hib);
      tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 32; ++e) {
        lo[e] = __float_as_uint(__uint_as_float(lo[e]) + ei * __uint_as_float(lob[e]));
        hi[e] = __float_as_uint(__uint_as_float(hi[e]) + ei * __uint_as_float(hib[e]));
      }
    }
#pragma unroll
    for (int x = 0; x < NROT / 8; ++x) {
      float xa[8], xb[8], ga[8], gb[8], cs8[8], sn8[8];
      ld8(cs8, cos_tab + t * tab_stride<NROT>() + x * 8);
      ld8(sn8, sin_tab + t * tab_stride<NROT>() + x * 8);
      unpack8(*reinterpret_cast<const uint4*>(tile + sw_off(i, x)), xa);                 // rotated values, cols 8x..
      unpack8(*reinterpret_cast<const uint4*>(tile + SLAB + sw_off(i, x)), xb);          // cols 64+8x..
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float da = __uint_as_float(lo[x * 8 + j]), db = __uint_as_float(hi[x * 8 + j]);
        dang[x * 8 + j] = db * xa[j] - da * xb[j];
        ga[j] = cs8[j] * da + sn8[j] * db;
        gb[j] = -sn8[j] * da + cs8[j] * db;
      }
      *reinterpret_cast<uint4*>(drow + x * 8) = pack8(ga);
      *reinterpret_cast<uint4*>(drow + HALF + x * 8) = pack8(gb);
    }
    // un-rotated halves
    tmem_ld_32x32(tacc + lane_addr + NROT, lo);
    tmem_ld_32x32(tacc + lane_addr + HALF + NROT, hi);
    tmem_ld_wait();
    if (isq) {
      uint32_t lob[32], hib[32];
      tmem_ld_32x32(tdQb + lane_addr + NROT, lob);
      tmem_ld_32x32(tdQb + lane_addr + HALF + NROT, hib);
      tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 32; ++e) {
        lo[e] = __float_as_uint(__uint_as_float(lo[e]) + ei * __uint_as_float(lob[e]));
        hi[e] = __float_as_uint(__uint_as_float(hi[e]) + ei * __uint_as_float(hib[e]));
      }
    }
#pragma unroll
    for (int x = 0; x < (HALF - NROT) / 8; ++x) {
      float ga[8], gb[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        ga[j] = __uint_as_float(lo[x * 8 + j]);
        gb[j] = __uint_as_float(hi[x * 8 + j]);
      }
      *reinterpret_cast<uint4*>(drow + NROT + x * 8) = pack8(ga);
      *reinterpret_cast<uint4*>(drow + HALF + NROT + x * 8) = pack8(gb);
    }
    // sum over the four ranks (lane r keeps the r-th group of eight); the K side hands its part over through shared memory
    reduce4_keep8(dang, dang8);
    if (!isq) {
      float4* d = reinterpret_cast<float4*>(&gs->dang[t][r * 8]);
      d[0] = make_float4(dang8[0], dang8[1], dang8[2], dang8[3]);
      d[1] = make_float4(dang8[4], dang8[5], dang8[6], dang8[7]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (ok && wg == 0) {
    float kd[8];
    ld8(kd, &gs->dang[t][r * 8]);
    float4* d = reinterpret_cast<float4*>(a.dAngles + (((size_t)b * a.S + t0 + t) * a.H + h) * NROT + r * 8);
    d[0] = make_float4(dang8[0] + kd[0], dang8[1] + kd[1], dang8[2] + kd[2], dang8[3] + kd[3]);
    d[1] = make_float4(dang8[4] + kd[4], dang8[5] + kd[5], dang8[6] + kd[6], dang8[7] + kd[7]);
  }
  // the next chunk's TMA loads and MMAs overwrite the tiles and accumulators every thread has just finished with
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (*abort_flag) break;
  }
  if (warp == 0) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

// Trapezoid coefficients: gamma_t = DT_t sig(Trap_t), ts_t = gamma_t + DT_{t+1} sig(-Trap_{t+1}); their gradients to DT, Trap.
// One launch instead of the dozen elementwise launches of the tensor library that cost a small call more than its kernels.
__global__ void __launch_bounds__(256) mimo_trapezoid_grad_kernel(const float* __restrict__ dts, const float* __restrict__ dgam,
                                                                  const float* __restrict__ DT, const float* __restrict__ Trap,
                                                                  float* __restrict__ dDT, float* __restrict__ dTrap, long long n, int S) {
  for (long long x = blockIdx.x * 256ll + threadIdx.x; x < n; x += gridDim.x * 256ll) {
    const float sg = 1.f / (1.f + expf(-Trap[x]));
    const float dgt = dgam[x] + dts[x], prev = x % S ? dts[x - 1] : 0.f;
    dDT[x] = dgt * sg + prev * (1.f - sg);
    dTrap[x] = (dgt - prev) * DT[x] * sg * (1.f - sg);
  }
}

constexpr int grad_state_smem() {
  return 2 * SLAB + SLAB + 2 * tab_floats<32>() * 4 + (int)sizeof(HeadBias<128>) + (int)sizeof(HeadVecs) + (int)sizeof(ChunkScalars) + 64 + 1024;
}
constexpr int chunk_grad_smem() {
  return 13 * SLAB + 2 * tab_floats<32>() * 4 + (int)sizeof(HeadVecs) + (int)sizeof(ChunkScalars) + 64 + 1024 + 1024;
}

}  // namespace mimo
}  // namespace cm

using namespace cm;
using namespace cm::mimo;

// Inputs as in cm_mimo_scan_fwd plus dY [B,S,H,P] bf16, the forward's `states` (start states, bf16) and `tot`.
// Scratch: gbuf [B,H,C,N,P] fp32, dend [B,H,C,N,P] bf16.
// Outputs: dQh, dKh [B,S,H,R,N] bf16 (per head, before the group reduction); dV, dZ [B,S,H,P] bf16;
// dAngles [B,S,H,N/4] fp32; dADT, dTs, dGam [B,H,S] fp32; dPsi, dZeta, dPhi [H,R,P], dD [H] fp32;
// dDT, dTrap [B,H,S] fp32.  dQg, dKg [B,S,G,R,N] bf16 and dQb, dKb [H,R,N] fp32 (all or none; H / G in 1, 2, 4, 8, 16): the
// sums of dQh, dKh over the heads of a group and over the tokens.
extern "C" int cm_head_reduce(const void* dh, void* dgrp, float* dbias, long long T, int H, int G, int C, cudaStream_t s);
extern "C" int cm_mimo_scan_bwd(const void* Qn, const void* Kn, const void* V, const void* Z, const void* dY,
                                const float* ADT, const float* DT, const float* Trap, const float* Qb, const float* Kb,
                                const float* Psi, const float* Zeta, const float* Phi, const float* angles,
                                const float* Dskip, const void* states, const float* tot, float* gbuf, void* dend,
                                void* dQh, void* dKh, void* dV, void* dZ, float* dAngles, float* dADT, float* dTs,
                                float* dGam, float* dPsi, float* dZeta, float* dPhi, float* dD_, float* dDT, float* dTrap, void* dQg,
                                void* dKg, float* dQb, float* dKb, int B, int S, int H, int G,
                                int N, long long ldV, long long ldZ, int* err, cudaStream_t stream) {
  if (B <= 0 || S <= 0) return 0;
  if (S % LT || N != 128 || H % G) return -10;
  if (ldV < (long long)H * P || ldZ < (long long)H * P || ldV % 8 || ldZ % 8) return -11;
  const int C = S / LT;
  CUtensorMap tmQ, tmK, tmS, tmE;
  int rc = make_tmap_qk(&tmQ, Qn, B, S, G, N);
  if (rc) return rc;
  rc = make_tmap_qk(&tmK, Kn, B, S, G, N);
  if (rc) return rc;
  rc = make_tmap_2d_bf16(&tmS, states, (uint64_t)B * H * C * N, 64, 64, 128, 64);
  if (rc) return rc;
  rc = make_tmap_2d_bf16(&tmE, dend, (uint64_t)B * H * C * N, 64, 64, 128, 64);
  if (rc) return rc;
  BwdArgs a{(const __nv_bfloat16*)V, (const __nv_bfloat16*)Z, (const __nv_bfloat16*)dY, ADT, DT, Trap, Qb, Kb, Psi, Zeta,
            Phi, angles, Dskip, gbuf, (__nv_bfloat16*)dQh, (__nv_bfloat16*)dKh, (__nv_bfloat16*)dV, (__nv_bfloat16*)dZ,
            dAngles, dADT, dTs, dGam, dPsi, dZeta, dPhi, dD_, dQg ? dQb : nullptr, dKb, B, S, H, G, C, ldV, ldZ, err, B * H * C};
  auto k0 = mimo_grad_state_kernel<128, 32>;
  auto k2 = mimo_chunk_grad_kernel<128, 32>;
  static PerDevice cfg;
  if (cfg.first()) {
    if (cudaFuncSetAttribute(k0, cudaFuncAttributeMaxDynamicSharedMemorySize, grad_state_smem()) != cudaSuccess) return -2;
    if (cudaFuncSetAttribute(k2, cudaFuncAttributeMaxDynamicSharedMemorySize, chunk_grad_smem()) != cudaSuccess) return -2;
    cfg.done();
  }
  const int grid = B * H * C;
  k0<<<grid, THREADS2, grad_state_smem(), stream>>>(tmQ, a);
  dim3 g2(B * H, (128 * P + 1023) / 1024);
  mimo_state_scan_rev_kernel<<<g2, 256, 0, stream>>>(gbuf, tot, (__nv_bfloat16*)dend, C, 128 * P);
  k2<<<grid < sm_count() ? grid : sm_count(), THREADS2, chunk_grad_smem(), stream>>>(tmQ, tmK, tmS, tmE, a);
  const long long n = (long long)B * H * S;
  const long long blocks = (n + 255) / 256;
  mimo_trapezoid_grad_kernel<<<(unsigned)(blocks < sm_count() * 8ll ? blocks : sm_count() * 8ll), 256, 0, stream>>>(dTs, dGam, DT, Trap, dDT,
                                                                                                                  dTrap, n, S);
  if (dQg) {
    rc = cm_head_reduce(dQh, dQg, dQb, (long long)B * S, H, G, R * N, stream);
    if (!rc) rc = cm_head_reduce(dKh, dKg, dKb, (long long)B * S, H, G, R * N, stream);
    if (rc) return rc;
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

