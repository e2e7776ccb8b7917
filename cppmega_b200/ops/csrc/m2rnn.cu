// M2RNN matrix-state recurrence, forward and backward.
//
//   a_t = h_{t-1} W + k_t (x) v_t ;  h_t = f_t h_{t-1} + (1 - f_t) tanh(a_t) ;  y_t = q_t . h_t
//
// One CTA per (batch, head), one warp per 16 rows of the state h [KD x 16], which stays in registers for the whole sequence
// in the accumulator layout of mma.m16n8k16 (lane (g, t): rows g and g + 8, columns 2t, 2t + 1 of each 8-column half).  That
// layout is also the A operand of the next step's product with W, so a step exchanges nothing between lanes.  The products
// keep fp32 operands: a bf16 factor enters as it is, an fp32 one as the sum of three bf16 parts (8 + 8 + 8 mantissa bits), each
// multiplied exactly and added in fp32; of the nine products of two such factors those below 2^-24 are left out.
//
// What bounds it: the instructions of a step - one warp per scheduler, each instruction 2.3 cycles at the dependences of a chain -
// not arithmetic or memory.  So every sum that can be one is a matrix product: the gradients of k and q against an operand
// with v and dy in two of its columns, the gradient of v against one with k in a row.  With four
// threads per row, 12 shuffles and 64 dependent multiply-adds a step and the state history fetched one step ahead, the
// backward took 1.23 us and the forward 0.29 us a step at batch 2, 51 heads; now 0.45 and 0.26.
// The history is requested four steps ahead.  Two warps per 16 rows, the second forming the gradients a block of steps behind,
// were slower (0.61 us a step: 589 instructions between them instead of 378 then in one warp).
// Only dh_{t-1} = f_t dh_t + da_t W^T is on the backward's chain; the replay of tanh(a_t) and all other gradients hang off it.
//
// Inputs are staged through shared memory in blocks of 16 steps (the next block is loaded into registers while the current
// one runs, one block barrier per 16 steps).  The forward writes the state history (fp32) that the backward replays in
// reverse.  q and k gradients are produced per head (the caller sums the head axis when q / k are shared by all heads).
// The reference runs this recurrence as Triton kernels with 64-token checkpoints
// (cppmega/megatron/m2rnn_triton.py:243-415 forward, :662-758 backward).
#include "common.cuh"

namespace cm {

constexpr int VD = 16;       // value head dim (fixed)
constexpr int TB = 16;       // time steps per staging block

__device__ __forceinline__ float fast_tanh(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// c (two 16 x 8 accumulators) = hi + mid + lo, each part as the A fragment of a 16 x 16 bf16 operand
struct Split3 {
  uint32_t hi[4], mid[4], lo[4];
};
__device__ __forceinline__ float bf_lo(uint32_t p) { return __uint_as_float(p << 16); }
__device__ __forceinline__ float bf_hi(uint32_t p) { return __uint_as_float(p & 0xffff0000u); }
__device__ __forceinline__ void split3(const float (&c)[8], Split3& s) {
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    float x = c[2 * p], y = c[2 * p + 1];
    s.hi[p] = pack_bf16(x, y);
    x -= bf_lo(s.hi[p]); y -= bf_hi(s.hi[p]);
    s.mid[p] = pack_bf16(x, y);
    x -= bf_lo(s.mid[p]); y -= bf_hi(s.mid[p]);
    s.lo[p] = pack_bf16(x, y);
  }
}
// d = a b + c.  Sums start from a constant or from a term of the step, so that no accumulator is cleared or added separately.
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2], const float (&c)[4]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %11, %12, %13};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  const float z[4] = {0.f, 0.f, 0.f, 0.f};
  mma16816(d, a, b, z);
}
// out = (lo + mid) M on top of `init`, plus hi M: the large part is added last, in fp32 rounding
__device__ __forceinline__ void times16(float (&out)[8], const Split3& x, const uint32_t (&m)[2][2], const float (&init)[8]) {
#pragma unroll
  for (int n = 0; n < 2; ++n) {
    float a[4], b[4];
    const float c[4] = {init[n * 4], init[n * 4 + 1], init[n * 4 + 2], init[n * 4 + 3]};
    mma16816(a, x.lo, m[n], c);
    mma16816(b, x.hi, m[n]);
    mma16816(a, x.mid, m[n], a);
#pragma unroll
    for (int i = 0; i < 4; ++i) out[n * 4 + i] = a[i] + b[i];
  }
}
// The forward's chain: the same with the products kept in this order (free to move, the compiler delays the first by the
// instructions of the step's other work: 1,155 us against 1,082 at batch 2, 51 heads) and nothing to start from
__device__ __forceinline__ void times16_in_order(float (&out)[8], const Split3& x, const uint32_t (&m)[2][2]) {
  auto mma = [](float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
  };
#pragma unroll
  for (int n = 0; n < 2; ++n) {
    float a[4] = {0.f, 0.f, 0.f, 0.f}, b[4] = {0.f, 0.f, 0.f, 0.f};
    mma(a, x.lo, m[n]);
    mma(b, x.hi, m[n]);
    mma(a, x.mid, m[n]);
#pragma unroll
    for (int i = 0; i < 4; ++i) out[n * 4 + i] = a[i] + b[i];
  }
}
__device__ __forceinline__ uint32_t transpose8x8(uint32_t x) {
  uint32_t y;
  asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}
// Sum of x[0..3] over the 8 lanes with equal (lane & 3); lane returns the sum of element 2 * bit4 + bit3 (bit2 is redundant).
__device__ __forceinline__ float reduce_rows4(const float (&x)[4], int lane) {
  const bool u4 = lane & 16, u3 = lane & 8;
  const float a0 = (u4 ? x[2] : x[0]) + __shfl_xor_sync(0xffffffffu, u4 ? x[0] : x[2], 16);
  const float a1 = (u4 ? x[3] : x[1]) + __shfl_xor_sync(0xffffffffu, u4 ? x[1] : x[3], 16);
  float r = (u3 ? a1 : a0) + __shfl_xor_sync(0xffffffffu, u3 ? a0 : a1, 8);
  return r + __shfl_xor_sync(0xffffffffu, r, 4);
}
// column (0..15) of the element that reduce_rows4 leaves in this lane, for x = columns {2t, 2t + 1, 8 + 2t, 9 + 2t}
__device__ __forceinline__ int reduced_col(int lane) { return 2 * (lane & 3) + ((lane >> 3) & 1) + ((lane & 16) ? 8 : 0); }

// 8 consecutive bf16; `vec`: the address is 16-byte aligned
__device__ __forceinline__ uint4 load8(const __nv_bfloat16* p, bool vec) {
  if (vec) return *reinterpret_cast<const uint4*>(p);
  const unsigned short* u = reinterpret_cast<const unsigned short*>(p);
  uint4 r;
  r.x = u[0] | (uint32_t(u[1]) << 16); r.y = u[2] | (uint32_t(u[3]) << 16);
  r.z = u[4] | (uint32_t(u[5]) << 16); r.w = u[6] | (uint32_t(u[7]) << 16);
  return r;
}
__device__ __forceinline__ void spread8(float* dst, uint4 v) {
  reinterpret_cast<float4*>(dst)[0] = make_float4(bf_lo(v.x), bf_hi(v.x), bf_lo(v.y), bf_hi(v.y));
  reinterpret_cast<float4*>(dst)[1] = make_float4(bf_lo(v.z), bf_hi(v.z), bf_lo(v.w), bf_hi(v.w));
}

// One block of inputs: TB steps of q, k (this head's or the shared one), v, dy and f
template <int KD, bool BWD>
struct Stage {
  float q[TB][KD], k[TB][KD], v[TB][VD], g[BWD ? TB : 1][VD], f[TB];
  // the backward also wants k, v and dy as they are, as MMA operands: pairs of bf16
  __align__(16) uint32_t kb[BWD ? TB : 1][KD / 2];
  __align__(16) uint32_t vg[BWD ? TB : 1][2][VD / 2];
};

template <int KD, bool BWD>
struct Loader {
  static constexpr int NT = KD * 2;            // threads: one 8-wide vector of q and of k each per block
  const __nv_bfloat16 *q, *k, *v, *g;
  const float* f;
  size_t q_step, k_step, v_step, f_step;
  int S;
  bool vec;
  uint4 rq, rk, rv, rg;
  float rf;
  __device__ __forceinline__ void fetch(int t0, int tid) {
    const int t = tid / (KD / 8), c = (tid % (KD / 8)) * 8;
    const bool in = t0 + t < S;
    rq = in ? load8(q + (size_t)(t0 + t) * q_step + c, vec) : make_uint4(0, 0, 0, 0);
    rk = in ? load8(k + (size_t)(t0 + t) * k_step + c, vec) : make_uint4(0, 0, 0, 0);
    if (tid < 2 * TB) {
      const int tv = tid >> 1, cv = (tid & 1) * 8;
      const bool inv = t0 + tv < S;
      rv = inv ? load8(v + (size_t)(t0 + tv) * v_step + cv, vec) : make_uint4(0, 0, 0, 0);
      if (BWD) rg = inv ? load8(g + (size_t)(t0 + tv) * v_step + cv, vec) : make_uint4(0, 0, 0, 0);
      if (tid < TB) rf = t0 + tid < S ? f[(size_t)(t0 + tid) * f_step] : 1.f;
    }
  }
  __device__ __forceinline__ void commit(Stage<KD, BWD>& s, int tid) const {
    const int t = tid / (KD / 8), c = (tid % (KD / 8)) * 8;
    spread8(&s.q[t][c], rq);
    spread8(&s.k[t][c], rk);
    if (BWD) *reinterpret_cast<uint4*>(&s.kb[BWD ? t : 0][c / 2]) = rk;
    if (tid < 2 * TB) {
      spread8(&s.v[tid >> 1][(tid & 1) * 8], rv);
      if (BWD) {
        spread8(&s.g[BWD ? tid >> 1 : 0][(tid & 1) * 8], rg);
        *reinterpret_cast<uint4*>(&s.vg[BWD ? tid >> 1 : 0][0][(tid & 1) * 4]) = rv;
        *reinterpret_cast<uint4*>(&s.vg[BWD ? tid >> 1 : 0][1][(tid & 1) * 4]) = rg;
      }
      if (tid < TB) s.f[tid] = rf;
    }
  }
};

// B fragments of W (out[v] = sum_u x[u] W[u][v]) or of its transpose (out[u] = sum_v x[v] W[u][v])
__device__ __forceinline__ void load_matrix(uint32_t (&m)[2][2], const __nv_bfloat16* w, int lane, bool transposed) {
  const int g = lane >> 2, t = lane & 3;
  const unsigned short* u = reinterpret_cast<const unsigned short*>(w);
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int kk = h * 8 + 2 * t, nn = n * 8 + g;
      const unsigned short a = transposed ? u[nn * VD + kk] : u[kk * VD + nn];
      const unsigned short b = transposed ? u[nn * VD + kk + 1] : u[(kk + 1) * VD + nn];
      m[n][h] = a | (uint32_t(b) << 16);
    }
}

template <int KD>
__global__ void __launch_bounds__(KD * 2) m2rnn_fwd_kernel(
    const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k, const __nv_bfloat16* __restrict__ v,
    const __nv_bfloat16* __restrict__ W, const float* __restrict__ f, __nv_bfloat16* __restrict__ y, float* __restrict__ hist,
    float* __restrict__ h_last, int S, int H, int Hq, int Hk, bool vec) {
  constexpr int NT = KD * 2, NW = KD / 16;
  __shared__ __align__(16) Stage<KD, false> stage[2];
  __shared__ float ypart[2][TB][NW][VD];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const int b = blockIdx.x / H, h = blockIdx.x % H;
  const int r0 = warp * 16 + g;                  // state rows r0 and r0 + 8
  Loader<KD, false> in;
  in.q = q + ((size_t)b * S * Hq + (Hq == 1 ? 0 : h)) * KD;
  in.k = k + ((size_t)b * S * Hk + (Hk == 1 ? 0 : h)) * KD;
  in.v = v + ((size_t)b * S * H + h) * VD;
  in.g = nullptr;
  in.f = f + (size_t)b * S * H + h;
  in.q_step = (size_t)Hq * KD; in.k_step = (size_t)Hk * KD; in.v_step = (size_t)H * VD; in.f_step = H;
  in.S = S; in.vec = vec;
  uint32_t w[2][2];
  load_matrix(w, W + (size_t)h * VD * VD, lane, false);
  float hs[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) hs[i] = 0.f;
  float* hrow = hist ? hist + ((size_t)blockIdx.x * S * KD + r0) * VD + 2 * t4 : nullptr;
  const int col = reduced_col(lane);
  in.fetch(0, tid);
  in.commit(stage[0], tid);
  auto write_y = [&](int blk) {                  // sum of the warps' parts of block `blk`
    const int t0 = blk * TB, nt = min(TB, S - t0);
    for (int e = tid; e < nt * VD; e += NT) {
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < NW; ++i) s += ypart[blk & 1][e / VD][i][e % VD];
      y[((size_t)(b * S + t0 + e / VD) * H + h) * VD + e % VD] = __float2bfloat16(s);
    }
  };
  const int nblocks = (S + TB - 1) / TB;
  for (int blk = 0; blk < nblocks; ++blk) {
    __syncthreads();                              // inputs of this block and y parts of the previous one are complete
    const Stage<KD, false>& st = stage[blk & 1];
    if (blk + 1 < nblocks) in.fetch((blk + 1) * TB, tid);
    if (blk > 0) write_y(blk - 1);
    const int nt = min(TB, S - blk * TB);
#pragma unroll 2
    for (int t = 0; t < nt; ++t) {
      const float k0 = st.k[t][r0], k1 = st.k[t][r0 + 8], q0 = st.q[t][r0], q1 = st.q[t][r0 + 8], ft = st.f[t];
      const float2 va = *reinterpret_cast<const float2*>(&st.v[t][2 * t4]), vb = *reinterpret_cast<const float2*>(&st.v[t][8 + 2 * t4]);
      const float vv[4] = {va.x, va.y, vb.x, vb.y};
      Split3 s;
      split3(hs, s);
      float a[8], yp[4];
      times16_in_order(a, s, w);
      const float omf = 1.f - ft;
#pragma unroll
      for (int i = 0; i < 8; ++i)                  // elements 2, 3, 6, 7 are row r0 + 8
        hs[i] = fmaf(ft, hs[i], omf * fast_tanh(fmaf((i & 2) ? k1 : k0, vv[(i >> 2) * 2 + (i & 1)], a[i])));
      if (hist) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<float2*>(hrow + ((i & 1) ? 8 * VD : 0) + (i >> 1) * 8) = make_float2(hs[2 * i], hs[2 * i + 1]);
        hrow += (size_t)KD * VD;
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int i = (c >> 1) * 4 + (c & 1);
        yp[c] = fmaf(q1, hs[i + 2], q0 * hs[i]);
      }
      const float r = reduce_rows4(yp, lane);
      if ((lane & 4) == 0) ypart[blk & 1][t][warp][col] = r;
    }
    if (blk + 1 < nblocks) in.commit(stage[(blk + 1) & 1], tid);     // its last readers passed the barrier above
  }
  __syncthreads();
  write_y(nblocks - 1);
  if (h_last) {
    float* o = h_last + ((size_t)blockIdx.x * KD + r0) * VD + 2 * t4;
#pragma unroll
    for (int i = 0; i < 4; ++i) *reinterpret_cast<float2*>(o + ((i & 1) ? 8 * VD : 0) + (i >> 1) * 8) = make_float2(hs[2 * i], hs[2 * i + 1]);
  }
}

template <int KD>
struct BwdShared {
  Stage<KD, true> stage[2];
  float dq[2][TB][KD], dk[2][TB][KD];
  float dv[2][TB][KD / 16][VD];
  float df[2][TB][KD * 2 + 8];                  // one partial per lane; rows 8 banks apart
  float dw[VD][VD];
};

// One resident CTA is asked for, so that the compiler keeps a step's independent products apart in up to 255 registers: left to
// choose, it takes 182 and 602 us for 1,024 steps of 102 heads, against 511 (16 and 32 rows: 639 and 596 against 501 and 513).
// Calls of more CTAs than fit at two an SM lose by it (1,351 -> 1,212 us at 408 of them, 1,012 with the 167 registers and the
// lower precision of two parts).
template <int KD>
__global__ void __launch_bounds__(KD * 2, 1) m2rnn_bwd_kernel(
    const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k, const __nv_bfloat16* __restrict__ v,
    const __nv_bfloat16* __restrict__ W, const float* __restrict__ f, const float* __restrict__ hist,
    const __nv_bfloat16* __restrict__ dy, float* __restrict__ dq_h, float* __restrict__ dk_h,
    float* __restrict__ dv, float* __restrict__ df, float* __restrict__ dW, int S, int H, int Hq, int Hk, bool vec) {
  constexpr int NT = KD * 2, NW = KD / 16;
  constexpr int AHEAD = 4;                       // steps between the request of a state and its use
  extern __shared__ __align__(16) uint8_t smem_raw[];
  BwdShared<KD>& sh = *reinterpret_cast<BwdShared<KD>*>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const int b = blockIdx.x / H, h = blockIdx.x % H;
  const int r0 = warp * 16 + g;
  Loader<KD, true> in;
  in.q = q + ((size_t)b * S * Hq + (Hq == 1 ? 0 : h)) * KD;
  in.k = k + ((size_t)b * S * Hk + (Hk == 1 ? 0 : h)) * KD;
  in.v = v + ((size_t)b * S * H + h) * VD;
  in.g = dy + ((size_t)b * S * H + h) * VD;
  in.f = f + (size_t)b * S * H + h;
  in.q_step = (size_t)Hq * KD; in.k_step = (size_t)Hk * KD; in.v_step = (size_t)H * VD; in.f_step = H;
  in.S = S; in.vec = vec;
  uint32_t w[2][2], wt[2][2];
  load_matrix(w, W + (size_t)h * VD * VD, lane, false);
  load_matrix(wt, W + (size_t)h * VD * VD, lane, true);
  for (int i = tid; i < VD * VD; i += NT) (&sh.dw[0][0])[i] = 0.f;
  const float* hbase = hist + ((size_t)blockIdx.x * S * KD + r0) * VD + 2 * t4;
  auto load_state = [&](float (&x)[8], int t) {   // h_t, zero before the first step and (never used) past the last
    const float* hp = hbase + (long long)t * (KD * VD);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 p = make_float2(0.f, 0.f);
      if (t >= 0 && t < S) p = *reinterpret_cast<const float2*>(hp + ((i & 1) ? 8 * VD : 0) + (i >> 1) * 8);
      x[2 * i] = p.x; x[2 * i + 1] = p.y;
    }
  };
  const int nblocks = (S + TB - 1) / TB;
  float ring[AHEAD][8], dh[8], dw_sum[2][4];
  Split3 hcur;                                    // h_t of the step at hand
  {
    float h_end[8];
    load_state(h_end, S - 1);
    split3(h_end, hcur);
  }
#pragma unroll
  for (int i = 0; i < AHEAD; ++i) load_state(ring[AHEAD - 1 - i], nblocks * TB - 2 - i);     // slot of step s: s % AHEAD, holds h_{s-1}
#pragma unroll
  for (int i = 0; i < 8; ++i) dh[i] = 0.f;
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) dw_sum[n][i] = 0.f;
  in.fetch((nblocks - 1) * TB, tid);
  in.commit(sh.stage[(nblocks - 1) & 1], tid);
  const uint32_t row0_mask = g == 0 ? 0xffffffffu : 0u, col01_mask = g < 2 ? 0xffffffffu : 0u;
  auto write_out = [&](int blk) {                 // the gradients of block `blk` from its shared-memory parts
    const int t0 = blk * TB, nt = min(TB, S - t0), p = blk & 1;
    for (int e = tid; e < nt * KD; e += NT) {
      const size_t o = ((size_t)(b * S + t0 + e / KD) * H + h) * KD + e % KD;
      dq_h[o] = sh.dq[p][e / KD][e % KD];
      dk_h[o] = sh.dk[p][e / KD][e % KD];
    }
    for (int e = tid; e < nt * VD; e += NT) {
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < NW; ++i) s += sh.dv[p][e / VD][i][e % VD];
      dv[((size_t)(b * S + t0 + e / VD) * H + h) * VD + e % VD] = s;
    }
    for (int e = tid; e < TB * 8; e += NT) {      // eight threads per step
      const int t = e >> 3, part = e & 7;
      float s = 0.f;
      if (t < nt) {
#pragma unroll
        for (int i = 0; i < NT / 8; ++i) s += sh.df[p][t][part + 8 * i];
      }
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      s += __shfl_xor_sync(0xffffffffu, s, 4);
      if (part == 0 && t < nt) df[(size_t)(b * S + t0 + t) * H + h] = s;
    }
  };
  for (int blk = nblocks - 1; blk >= 0; --blk) {
    __syncthreads();                              // inputs of this block and gradient parts of the previous one are complete
    const int p = blk & 1;
    const Stage<KD, true>& st = sh.stage[p];
    if (blk > 0) in.fetch((blk - 1) * TB, tid);
    if (blk + 1 < nblocks) write_out(blk + 1);
    const int t0 = blk * TB;
#pragma unroll 1
    for (int t1 = TB - AHEAD; t1 >= 0; t1 -= AHEAD) {
#pragma unroll
      for (int sl = AHEAD - 1; sl >= 0; --sl) {
        const int t = t1 + sl;
        float hprev[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) hprev[i] = ring[sl][i];
        load_state(ring[sl], t0 + t - 1 - AHEAD);
        if (t0 + t >= S) continue;                // past the end: the whole CTA skips
        const float k0 = st.k[t][r0], k1 = st.k[t][r0 + 8], q0 = st.q[t][r0], q1 = st.q[t][r0 + 8], ft = st.f[t];
        const float2 va = *reinterpret_cast<const float2*>(&st.v[t][2 * t4]), vb = *reinterpret_cast<const float2*>(&st.v[t][8 + 2 * t4]);
        const float2 ga = *reinterpret_cast<const float2*>(&st.g[t][2 * t4]), gb = *reinterpret_cast<const float2*>(&st.g[t][8 + 2 * t4]);
        const float vv[4] = {va.x, va.y, vb.x, vb.y}, gg[4] = {ga.x, ga.y, gb.x, gb.y};
        // replay of tanh(a_t); off the chain
        Split3 sp;
        split3(hprev, sp);
        float a[8], kv[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) kv[i] = ((i & 2) ? k1 : k0) * vv[(i >> 2) * 2 + (i & 1)];
        times16(a, sp, w, kv);
        float da[8], dfp = 0.f;
        const float omf = 1.f - ft;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float hn = fast_tanh(a[i]);
          dh[i] = fmaf((i & 2) ? q1 : q0, gg[(i >> 2) * 2 + (i & 1)], dh[i]);
          dfp = fmaf(dh[i], hprev[i] - hn, dfp);
          da[i] = dh[i] * fmaf(-omf, hn * hn, omf);
        }
        Split3 sd;
        split3(da, sd);
        float back[8];
        const float none[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        times16(back, sd, wt, none);
#pragma unroll
        for (int i = 0; i < 8; ++i) dh[i] = fmaf(ft, dh[i], back[i]);
        // dk[row] = sum_v da[row][v] v[v], dq[row] = sum_v h_t[row][v] dy[v]: one operand with v in column 0 and dy in column 1
        {
          const uint32_t vg[2] = {st.vg[t][g & 1][t4] & col01_mask, st.vg[t][g & 1][4 + t4] & col01_mask};
          float rk[4], rq[4];
          mma16816(rk, sd.lo, vg);
          mma16816(rq, hcur.lo, vg);
          mma16816(rk, sd.mid, vg, rk);
          mma16816(rq, hcur.mid, vg, rq);
          mma16816(rk, sd.hi, vg, rk);
          mma16816(rq, hcur.hi, vg, rq);
          if (t4 == 0) {
            sh.dk[p][t][r0] = rk[0];
            sh.dk[p][t][r0 + 8] = rk[2];
            sh.dq[p][t][r0] = rq[1];
            sh.dq[p][t][r0 + 8] = rq[3];
          }
        }
        // dW[u][v] += sum_rows h_{t-1}[row][u] da[row][v] and dv[v] = sum_rows k[row] da[row][v]: da as the right factor, h as the
        // left one, both transposed within the warp.  All parts of both factors, down to the products of 2^-24 (k is exact); a
        // step's sum starts from zero and is added to the running one in fp32 rounding.
        {
          uint32_t hh[4], hm[4], hl[4], dd[4], dm[4], dl[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int j = (i & 1) * 2 + (i >> 1);  // block (row half, column half) -> (column half, row half)
            hh[j] = transpose8x8(sp.hi[i]); hm[j] = transpose8x8(sp.mid[i]); hl[j] = transpose8x8(sp.lo[i]);
            dd[i] = transpose8x8(sd.hi[i]); dm[i] = transpose8x8(sd.mid[i]); dl[i] = transpose8x8(sd.lo[i]);
          }
          const uint32_t kr[4] = {st.kb[t][warp * 8 + t4] & row0_mask, 0u, st.kb[t][warp * 8 + 4 + t4] & row0_mask, 0u};
          float dvp[2][4];
#pragma unroll
          for (int n = 0; n < 2; ++n) {
            const uint32_t bh[2] = {dd[n * 2], dd[n * 2 + 1]}, bm[2] = {dm[n * 2], dm[n * 2 + 1]}, bl[2] = {dl[n * 2], dl[n * 2 + 1]};
            float dwp[4];
            mma16816(dvp[n], kr, bl);
            mma16816(dwp, hl, bh);
            mma16816(dvp[n], kr, bm, dvp[n]);
            mma16816(dwp, hh, bl, dwp);
            mma16816(dvp[n], kr, bh, dvp[n]);
            mma16816(dwp, hm, bm, dwp);
            mma16816(dwp, hm, bh, dwp);
            mma16816(dwp, hh, bm, dwp);
            mma16816(dwp, hh, bh, dwp);
#pragma unroll
            for (int i = 0; i < 4; ++i) dw_sum[n][i] += dwp[i];
          }
          if (g == 0) {
            *reinterpret_cast<float2*>(&sh.dv[p][t][warp][2 * t4]) = make_float2(dvp[0][0], dvp[0][1]);
            *reinterpret_cast<float2*>(&sh.dv[p][t][warp][8 + 2 * t4]) = make_float2(dvp[1][0], dvp[1][1]);
          }
        }
        sh.df[p][t][tid] = dfp;
        hcur = sp;
      }
    }
    if (blk > 0) in.commit(sh.stage[(blk - 1) & 1], tid);
  }
  __syncthreads();
  write_out(0);
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) atomicAdd(&sh.dw[g + ((i & 2) ? 8 : 0)][n * 8 + 2 * t4 + (i & 1)], dw_sum[n][i]);
  __syncthreads();
  for (int i = tid; i < VD * VD; i += NT) atomicAdd(dW + (size_t)h * VD * VD + i, (&sh.dw[0][0])[i]);
}

template <int KD>
static int launch_bwd(const __nv_bfloat16* q, const __nv_bfloat16* k, const __nv_bfloat16* v, const __nv_bfloat16* W, const float* f,
                      const float* hist, const __nv_bfloat16* dy, float* dq_h, float* dk_h, float* dv, float* df, float* dW, int B, int S,
                      int H, int Hq, int Hk, bool vec, cudaStream_t s) {
  static PerDevice cfg;
  if (cfg.first()) {
    if (cudaFuncSetAttribute(m2rnn_bwd_kernel<KD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BwdShared<KD>)) != cudaSuccess)
      return -2;
    cfg.done();
  }
  m2rnn_bwd_kernel<KD><<<B * H, KD * 2, sizeof(BwdShared<KD>), s>>>(q, k, v, W, f, hist, dy, dq_h, dk_h, dv, df, dW, S, H, Hq, Hk, vec);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

}  // namespace cm

using namespace cm;

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// q [B,S,Hq,KD], k [B,S,Hk,KD], v [B,S,H,16], W [H,16,16] (bf16); f [B,S,H] fp32.
// y [B,S,H,16] bf16; hist (nullable) [B,H,S,KD,16] fp32; h_last (nullable) [B,H,KD,16] fp32.
extern "C" int cm_m2rnn_fwd(const void* q, const void* k, const void* v, const void* W, const float* f, void* y, float* hist, float* h_last,
                            int B, int S, int H, int Hq, int Hk, int KD, int VDim, cudaStream_t s) {
  if (B <= 0 || S <= 0) return 0;
  if (VDim != VD) return -10;
  auto qp = (const __nv_bfloat16*)q; auto kp = (const __nv_bfloat16*)k; auto vp = (const __nv_bfloat16*)v;
  auto wp = (const __nv_bfloat16*)W; auto yp = (__nv_bfloat16*)y;
  const bool vec = aligned16(q) && aligned16(k) && aligned16(v);
  if (KD == 64) m2rnn_fwd_kernel<64><<<B * H, 128, 0, s>>>(qp, kp, vp, wp, f, yp, hist, h_last, S, H, Hq, Hk, vec);
  else if (KD == 32) m2rnn_fwd_kernel<32><<<B * H, 64, 0, s>>>(qp, kp, vp, wp, f, yp, hist, h_last, S, H, Hq, Hk, vec);
  else if (KD == 16) m2rnn_fwd_kernel<16><<<B * H, 32, 0, s>>>(qp, kp, vp, wp, f, yp, hist, h_last, S, H, Hq, Hk, vec);
  else return -10;
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

// dq_h, dk_h [B,S,H,KD] fp32 (per head), dv [B,S,H,16] and df [B,S,H] fp32 are written; dW [H,16,16] fp32 is accumulated over
// the batch: the caller zeroes it.
extern "C" int cm_m2rnn_bwd(const void* q, const void* k, const void* v, const void* W, const float* f, const float* hist,
                            const void* dy, float* dq_h, float* dk_h, float* dv, float* df, float* dW, int B, int S, int H,
                            int Hq, int Hk, int KD, int VDim, cudaStream_t s) {
  if (B <= 0 || S <= 0) return 0;
  if (VDim != VD) return -10;
  auto qp = (const __nv_bfloat16*)q; auto kp = (const __nv_bfloat16*)k; auto vp = (const __nv_bfloat16*)v;
  auto wp = (const __nv_bfloat16*)W; auto gp = (const __nv_bfloat16*)dy;
  const bool vec = aligned16(q) && aligned16(k) && aligned16(v) && aligned16(dy);
  if (KD == 64) return launch_bwd<64>(qp, kp, vp, wp, f, hist, gp, dq_h, dk_h, dv, df, dW, B, S, H, Hq, Hk, vec, s);
  if (KD == 32) return launch_bwd<32>(qp, kp, vp, wp, f, hist, gp, dq_h, dk_h, dv, df, dW, B, S, H, Hq, Hk, vec, s);
  if (KD == 16) return launch_bwd<16>(qp, kp, vp, wp, f, hist, gp, dq_h, dk_h, dv, df, dW, B, S, H, Hq, Hk, vec, s);
  return -10;
}
