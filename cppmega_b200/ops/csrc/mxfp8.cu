// MXFP8 quantisation: E4M3 payload with one E8M0 scale per 32 values.
//
//   scale byte = clamp(ceil(log2(amax / 448)) + 127, 1, 254)   (127 for an all-zero block)
//   payload    = e4m3(x * 2^(127 - scale))
//
//   rowwise      blocks of 32 along the contiguous (last) dimension: the operand layout of a product that reduces
//                over that dimension (forward GEMM: x and W both along K);
//   columnwise   blocks of 32 along the rows, written TRANSPOSED ([cols, rows] payload, [cols, rows/32] scales), so
//                that the result is again a K-major operand for the products that reduce over rows (wgrad over
//                tokens, dgrad over output features);
//   dequantise   payload * 2^(scale - 127) -> bf16;
//   swizzle      row-major [rows, kb] scales -> the 128x4 tile order ([32][4][4] per tile) that block-scaled
//                tensor-core instructions read.
// These replace the reference's cast/transposed-cast kernels and its scale swizzle (Transformer-Engine MXFP8 tensors
// re-used by cppmega/megatron/cutlass_mxfp8_gemm.py:102-506; layout of the swizzle at
// cppmega/megatron/flashinfer_mxfp8_gemm.py:146-160; scale byte at cuda_ext/quantized_muon_momentum.cu:75-91).
#include "common.cuh"

namespace cm {
namespace mx {

// ceil(log2(amax / 448)) + 127 from the bits of the quotient: its exponent field, one more unless it is a power of two (a bf16
// amax makes it one only for 224 * 2^k, whose product with fl(1/448) rounds to the power of two itself).
__device__ __forceinline__ uint8_t e8m0_from_amax(float amax) {
  if (!(amax > 0.f)) return 127;
  const uint32_t u = __float_as_uint(amax * (1.f / 448.f));
  int e = (int)(u >> 23) + ((u & 0x7fffffu) != 0);
  if (e == 255) return 1;                         // an infinity has no scale
  e = e < 1 ? 1 : (e > 254 ? 254 : e);
  return (uint8_t)e;
}
// The same for a tensor-wide amax, which the caller may give as any fp32 value: the bits above differ from the definition's
// logarithm, which rounds to k for the values closest above 448 * 2^k.
__device__ __forceinline__ uint8_t e8m0_from_tensor_amax(float amax) {
  if (!(amax > 0.f)) return 127;
  if (isinf(amax)) return 1;
  const int e = (int)ceilf(log2f(amax * (1.f / 448.f))) + 127;
  return (uint8_t)(e < 1 ? 1 : (e > 254 ? 254 : e));
}
__device__ __forceinline__ uint8_t scale_byte(const float* tamax, float block_amax) {
  return tamax ? e8m0_from_tensor_amax(*tamax) : e8m0_from_amax(block_amax);
}
// 2^(127 - sb), sb in 1..254
__device__ __forceinline__ float inverse_scale(uint8_t sb) { return __uint_as_float(sb == 254 ? 0x00400000u : (254u - sb) << 23); }
// two floats -> two e4m3 bytes (lo in bits 0..7)
__device__ __forceinline__ uint16_t to_e4m3x2(float lo, float hi) {
  uint16_t r;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ float e4m3_to_float(uint8_t b) {
  // sign 1, exponent 4 (bias 7), mantissa 3; no infinities, 0x7f / 0xff are NaN
  const uint32_t s = (uint32_t)(b & 0x80) << 24;
  const uint32_t e = (b >> 3) & 0xf, m = b & 7;
  float v;
  if (e == 0) v = (float)m * 0.001953125f;                            // subnormal: m * 2^-9
  else v = __uint_as_float(((e + 120u) << 23) | (m << 20));
  return __uint_as_float(__float_as_uint(v) | s);
}

// position of scale (row, k block) in the 128x4 tile order
__device__ __forceinline__ size_t swizzled_index(long long row, int kb, int kb_tiles) {
  return ((size_t)(row >> 7) * kb_tiles + (kb >> 2)) * 512 + (size_t)(row & 31) * 16 + ((row >> 5) & 3) * 4 + (kb & 3);
}

// one thread = 8 consecutive values; 4 threads = one block of 32
__global__ void __launch_bounds__(256) quantize_rowwise_kernel(const __nv_bfloat16* __restrict__ x, uint8_t* __restrict__ payload,
                                                               uint8_t* __restrict__ scales, uint8_t* __restrict__ sw, long long rows,
                                                               int cols, const float* __restrict__ tamax) {
  const int kb_row = cols / 32, kb_tiles = (kb_row + 3) / 4;
  const long long nvec = rows * (cols / 8);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nvec; i += (long long)gridDim.x * blockDim.x) {
    const uint4 raw = reinterpret_cast<const uint4*>(x)[i];
    const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&raw);
    float f[8];
    float am = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 t = __bfloat1622float2(b[j]);
      f[2 * j] = t.x; f[2 * j + 1] = t.y;
      am = fmaxf(am, fmaxf(fabsf(t.x), fabsf(t.y)));
    }
    const unsigned live = __activemask();          // whole groups of four threads enter or leave the loop together
    am = fmaxf(am, __shfl_xor_sync(live, am, 1));
    am = fmaxf(am, __shfl_xor_sync(live, am, 2));
    const uint8_t sb = scale_byte(tamax, am);
    const float mult = inverse_scale(sb);
    uint2 o;
    o.x = (uint32_t)to_e4m3x2(f[0] * mult, f[1] * mult) | ((uint32_t)to_e4m3x2(f[2] * mult, f[3] * mult) << 16);
    o.y = (uint32_t)to_e4m3x2(f[4] * mult, f[5] * mult) | ((uint32_t)to_e4m3x2(f[6] * mult, f[7] * mult) << 16);
    reinterpret_cast<uint2*>(payload)[i] = o;
    if ((threadIdx.x & 3) == 0) {
      scales[i >> 2] = sb;
      if (sw) {
        const long long blk = i >> 2;
        sw[swizzled_index(blk / kb_row, (int)(blk % kb_row), kb_tiles)] = sb;
      }
    }
  }
}

// CTA = tile of 32 rows x 128 columns; thread c owns one column: 32 values -> one block
__global__ void __launch_bounds__(128) quantize_colwise_kernel(const __nv_bfloat16* __restrict__ x, uint8_t* __restrict__ payload_t,
                                                               uint8_t* __restrict__ scales_t, uint8_t* __restrict__ sw, long long rows,
                                                               int cols, const float* __restrict__ tamax) {
  const long long r0 = (long long)blockIdx.y * 32;
  const int c = blockIdx.x * 128 + threadIdx.x;
  if (c >= cols) return;
  float f[32];
  float am = 0.f;
#pragma unroll
  for (int r = 0; r < 32; ++r) {
    f[r] = (r0 + r < rows) ? __bfloat162float(x[(size_t)(r0 + r) * cols + c]) : 0.f;
    am = fmaxf(am, fabsf(f[r]));
  }
  const uint8_t sb = scale_byte(tamax, am);
  const float mult = inverse_scale(sb);
  uint32_t w[8];
#pragma unroll
  for (int q = 0; q < 8; ++q)
    w[q] = (uint32_t)to_e4m3x2(f[4 * q] * mult, f[4 * q + 1] * mult) | ((uint32_t)to_e4m3x2(f[4 * q + 2] * mult, f[4 * q + 3] * mult) << 16);
  uint4* dst = reinterpret_cast<uint4*>(payload_t + (size_t)c * rows + r0);
  dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
  dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
  scales_t[(size_t)c * (rows / 32) + blockIdx.y] = sb;
  if (sw) sw[swizzled_index(c, (int)blockIdx.y, (int)((rows / 32 + 3) / 4))] = sb;
}

// Both orientations from one read of x: CTA = tile of 128 rows x 128 columns.  Phase 1 is the row-wise kernel (8 values per
// thread, 4 threads per block) and parks the raw values in shared memory; in phase 2 a thread takes two neighbouring columns
// of one 32-row block, so a bank word is one read.  A tile is one line (128 bytes) of every row and of every transposed row,
// and exactly one 128x4 scale tile of each orientation, which leaves as whole words.  Memory-bound; with 32 x 256 tiles of
// fp32 in shared memory, 32-byte transposed runs and log2 / exp2 per block, 8192 x 8192
// and 8192 x 4096 together took 201 us; now 104 to 137.
constexpr int QB_LD = 65;                                   // words per row of 128 bf16; each 32-row block is 8 words further
__device__ __forceinline__ int qb_word(int row, int pair) { return row * QB_LD + (row >> 5) * 8 + pair; }

__global__ void __launch_bounds__(256) quantize_both_kernel(const __nv_bfloat16* __restrict__ x, uint8_t* __restrict__ pay_r,
                                                            uint8_t* __restrict__ sc_r, uint8_t* __restrict__ sw_r,
                                                            uint8_t* __restrict__ pay_t, uint8_t* __restrict__ sc_t,
                                                            uint8_t* __restrict__ sw_t, long long rows, int cols,
                                                            const float* __restrict__ tamax) {
  __shared__ uint32_t tile[128 * QB_LD + 32];
  __shared__ __align__(4) uint8_t s_r[128][4], s_t[128][4];
  const long long r0 = (long long)blockIdx.y * 128;
  const int c0 = blockIdx.x * 128;
  const int nrows = (int)min(128ll, rows - r0), ncols = min(128, cols - c0);        // multiples of 32
  const int kb_row = cols / 32, kbt_row = (kb_row + 3) / 4;
  const int kb_col = (int)(rows / 32), kbt_col = (kb_col + 3) / 4;
  const int tid = threadIdx.x, lane = tid & 31;
  uint4 raw[8];
#pragma unroll
  for (int it = 0; it < 8; ++it) {
    const int row = it * 16 + (tid >> 4), v = tid & 15;
    raw[it] = make_uint4(0, 0, 0, 0);
    if (row < nrows && v * 8 < ncols) raw[it] = *reinterpret_cast<const uint4*>(x + (size_t)(r0 + row) * cols + c0 + v * 8);
  }
#pragma unroll
  for (int it = 0; it < 8; ++it) {
    const int row = it * 16 + (tid >> 4), v = tid & 15;
    const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&raw[it]);
    float f[8], am = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 t = __bfloat1622float2(b[j]);
      f[2 * j] = t.x; f[2 * j + 1] = t.y;
      am = fmaxf(am, fmaxf(fabsf(t.x), fabsf(t.y)));
    }
    uint32_t* w = &tile[qb_word(row, v * 4)];
    w[0] = raw[it].x; w[1] = raw[it].y; w[2] = raw[it].z; w[3] = raw[it].w;
    am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 1));
    am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 2));
    const uint8_t sb = scale_byte(tamax, am);
    const float mult = inverse_scale(sb);
    if ((lane & 3) == 0) s_r[row][v >> 2] = sb;
    if (row < nrows && v * 8 < ncols) {
      uint2 o;
      o.x = (uint32_t)to_e4m3x2(f[0] * mult, f[1] * mult) | ((uint32_t)to_e4m3x2(f[2] * mult, f[3] * mult) << 16);
      o.y = (uint32_t)to_e4m3x2(f[4] * mult, f[5] * mult) | ((uint32_t)to_e4m3x2(f[6] * mult, f[7] * mult) << 16);
      *reinterpret_cast<uint2*>(pay_r + (size_t)(r0 + row) * cols + c0 + v * 8) = o;
    }
  }
  __syncthreads();
  {
    const int blk = lane & 3, pair = (tid >> 5) * 8 + (lane >> 2);        // 32-row block, column pair
    uint32_t w[32];
    float am[2] = {0.f, 0.f};
#pragma unroll
    for (int r = 0; r < 32; ++r) {
      w[r] = tile[qb_word(blk * 32 + r, pair)];
      am[0] = fmaxf(am[0], fabsf(__uint_as_float(w[r] << 16)));
      am[1] = fmaxf(am[1], fabsf(__uint_as_float(w[r] & 0xffff0000u)));
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint8_t sb = scale_byte(tamax, am[h]);
      const float mult = inverse_scale(sb);
      s_t[pair * 2 + h][blk] = sb;
      uint32_t o[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        float f[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) f[j] = __uint_as_float(h ? (w[q * 4 + j] & 0xffff0000u) : (w[q * 4 + j] << 16)) * mult;
        o[q] = (uint32_t)to_e4m3x2(f[0], f[1]) | ((uint32_t)to_e4m3x2(f[2], f[3]) << 16);
      }
      // neighbouring lanes hold neighbouring 32-byte blocks of the transposed row: they swap halves so that each of the two
      // stores covers whole sectors
      const bool odd = lane & 1;
      uint4 got, a = make_uint4(o[0], o[1], o[2], o[3]), b = make_uint4(o[4], o[5], o[6], o[7]);
      const uint4 give = odd ? a : b;
      got.x = __shfl_xor_sync(0xffffffffu, give.x, 1); got.y = __shfl_xor_sync(0xffffffffu, give.y, 1);
      got.z = __shfl_xor_sync(0xffffffffu, give.z, 1); got.w = __shfl_xor_sync(0xffffffffu, give.w, 1);
      const int col = pair * 2 + h, even_blk = blk & 2;
      if (col < ncols) {
        uint8_t* dst = pay_t + (size_t)(c0 + col) * rows + r0 + even_blk * 32 + (odd ? 16 : 0);
        if (even_blk * 32 < nrows) *reinterpret_cast<uint4*>(dst) = odd ? got : a;                 // the even block
        if (even_blk * 32 + 32 < nrows) *reinterpret_cast<uint4*>(dst + 32) = odd ? b : got;       // the odd block
      }
    }
  }
  __syncthreads();
  // scales: thread < 128 one row, the others one column; whole words where all four blocks exist
  const bool is_row = tid < 128;
  const int k = tid & 127;
  if (k < (is_row ? nrows : ncols)) {
    const uint8_t* src = is_row ? s_r[k] : s_t[k];
    const int nkb = (is_row ? ncols : nrows) / 32, kb0 = (is_row ? c0 : (int)r0) / 32, kbs = is_row ? kb_row : kb_col;
    uint8_t* plain = (is_row ? sc_r + (size_t)(r0 + k) * kbs : sc_t + (size_t)(c0 + k) * kbs) + kb0;
    uint8_t* sw = is_row ? sw_r : sw_t;
    if (sw) sw += swizzled_index((is_row ? r0 : c0) + k, kb0, is_row ? kbt_row : kbt_col);
    if (nkb == 4) {
      const uint32_t v = *reinterpret_cast<const uint32_t*>(src);
      if ((kbs & 3) == 0) *reinterpret_cast<uint32_t*>(plain) = v;
      else for (int q = 0; q < 4; ++q) plain[q] = src[q];
      if (sw) *reinterpret_cast<uint32_t*>(sw) = v;
    } else {
      for (int q = 0; q < nkb; ++q) {
        plain[q] = src[q];
        if (sw) sw[q] = src[q];
      }
    }
  }
}

// absolute maximum of a bf16 tensor: non-negative floats order like their bit patterns, so an integer atomicMax works
__global__ void __launch_bounds__(256) amax_kernel(const __nv_bfloat16* __restrict__ x, long long nvec, float* __restrict__ out) {
  float am = 0.f;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nvec; i += (long long)gridDim.x * blockDim.x) {
    const uint4 raw = reinterpret_cast<const uint4*>(x)[i];
    const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 t = __bfloat1622float2(b[j]);
      am = fmaxf(am, fmaxf(fabsf(t.x), fabsf(t.y)));
    }
  }
  am = warp_max(am);
  __shared__ float red[8];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = am;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) am = fmaxf(am, red[w]);
    if (am == am) atomicMax(reinterpret_cast<unsigned int*>(out), __float_as_uint(am));
  }
}

__global__ void __launch_bounds__(256) dequantize_kernel(const uint8_t* __restrict__ payload, const uint8_t* __restrict__ scales,
                                                         __nv_bfloat16* __restrict__ out, long long n) {
  const long long nvec = n / 8;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nvec; i += (long long)gridDim.x * blockDim.x) {
    const uint2 raw = reinterpret_cast<const uint2*>(payload)[i];
    const float mult = exp2f((float)scales[i >> 2] - 127.f);
    const uint8_t* b = reinterpret_cast<const uint8_t*>(&raw);
    uint4 o;
    o.x = pack_bf16(e4m3_to_float(b[0]) * mult, e4m3_to_float(b[1]) * mult);
    o.y = pack_bf16(e4m3_to_float(b[2]) * mult, e4m3_to_float(b[3]) * mult);
    o.z = pack_bf16(e4m3_to_float(b[4]) * mult, e4m3_to_float(b[5]) * mult);
    o.w = pack_bf16(e4m3_to_float(b[6]) * mult, e4m3_to_float(b[7]) * mult);
    reinterpret_cast<uint4*>(out)[i] = o;
  }
}

// out is the flat 128x4-tiled buffer of ceil(rows/128) x ceil(kb/4) tiles of 512 bytes, padded with the neutral scale
__global__ void __launch_bounds__(256) swizzle_scales_kernel(const uint8_t* __restrict__ scales, uint8_t* __restrict__ out, long long rows,
                                                             int kb, int kb_tiles, long long total) {
  for (long long o = blockIdx.x * (long long)blockDim.x + threadIdx.x; o < total; o += (long long)gridDim.x * blockDim.x) {
    const long long tile = o >> 9;
    const int in = (int)(o & 511);
    const int r32 = in >> 4, rg = (in >> 2) & 3, k4 = in & 3;
    const long long row = (tile / kb_tiles) * 128 + rg * 32 + r32;
    const int k = (int)(tile % kb_tiles) * 4 + k4;
    out[o] = (row < rows && k < kb) ? scales[row * kb + k] : (uint8_t)127;
  }
}

}  // namespace mx
}  // namespace cm

using namespace cm;
using namespace cm::mx;

static int grid1d(long long work) {
  long long blocks = (work + 255) / 256;
  long long cap = (long long)sm_count() * 16;
  return (int)(blocks < cap ? (blocks > 0 ? blocks : 1) : cap);
}

// x [rows, cols] bf16, cols % 32 == 0 -> payload [rows, cols] u8, scales [rows, cols/32] u8; `swizzled` (optional) also
// receives the scales in the 128x4 tile order (its padding entries must already hold the neutral scale)
// `tensor_amax` (optional, every quantise entry point): a device float holding the absolute maximum of the WHOLE tensor.
// When given, every block uses the one scale derived from it (per-tensor "current scaling" with a power-of-two scale)
// instead of its own: the tensorwise FP8 recipe on the same payload / scale-byte data path.
extern "C" int cm_mxfp8_quantize_rowwise(const void* x, void* payload, void* scales, void* swizzled, long long rows, int cols,
                                         const float* tensor_amax, cudaStream_t s) {
  if (rows <= 0) return 0;
  if (cols % 32) return -10;
  quantize_rowwise_kernel<<<grid1d(rows * (cols / 8)), 256, 0, s>>>((const __nv_bfloat16*)x, (uint8_t*)payload, (uint8_t*)scales,
                                                                  (uint8_t*)swizzled, rows, cols, tensor_amax);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

// x [rows, cols] bf16, rows % 32 == 0 -> payload_t [cols, rows] u8, scales_t [cols, rows/32] u8 (+ optional swizzled copy)
extern "C" int cm_mxfp8_quantize_colwise(const void* x, void* payload_t, void* scales_t, void* swizzled, long long rows, int cols,
                                         const float* tensor_amax, cudaStream_t s) {
  if (rows <= 0) return 0;
  if (rows % 32) return -10;
  dim3 grid((cols + 127) / 128, (unsigned)(rows / 32));
  quantize_colwise_kernel<<<grid, 128, 0, s>>>((const __nv_bfloat16*)x, (uint8_t*)payload_t, (uint8_t*)scales_t, (uint8_t*)swizzled, rows, cols, tensor_amax);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

// x [rows, cols] bf16 (rows % 32 == 0, cols % 32 == 0) -> row-wise payload / scales and the transposed column-wise pair in
// one pass; the swizzled scale outputs are optional
extern "C" int cm_mxfp8_quantize_both(const void* x, void* pay_r, void* sc_r, void* sw_r, void* pay_t, void* sc_t, void* sw_t,
                                      long long rows, int cols, const float* tensor_amax, cudaStream_t s) {
  if (rows <= 0) return 0;
  if ((rows % 32) || (cols % 32)) return -10;
  dim3 grid((cols + 127) / 128, (unsigned)((rows + 127) / 128));
  quantize_both_kernel<<<grid, 256, 0, s>>>((const __nv_bfloat16*)x, (uint8_t*)pay_r, (uint8_t*)sc_r, (uint8_t*)sw_r, (uint8_t*)pay_t,
                                           (uint8_t*)sc_t, (uint8_t*)sw_t, rows, cols, tensor_amax);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

// out (device float, zeroed by the caller) = max(out, max |x|) over n bf16 values (n % 8 == 0)
extern "C" int cm_amax_bf16(const void* x, long long n, float* out, cudaStream_t s) {
  if (n <= 0) return 0;
  if (n % 8) return -10;
  amax_kernel<<<grid1d(n / 8), 256, 0, s>>>((const __nv_bfloat16*)x, n / 8, out);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

// payload [n] u8 with scales [n/32] (blocks of 32 consecutive values) -> bf16 [n]
extern "C" int cm_mxfp8_dequantize(const void* payload, const void* scales, void* out, long long n, cudaStream_t s) {
  if (n <= 0) return 0;
  if (n % 32) return -10;
  dequantize_kernel<<<grid1d(n / 8), 256, 0, s>>>((const uint8_t*)payload, (const uint8_t*)scales, (__nv_bfloat16*)out, n);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

// scales [rows, kb] -> out [ceil(rows/128) * ceil(kb/4) * 512]
extern "C" int cm_mxfp8_swizzle_scales(const void* scales, void* out, long long rows, int kb, cudaStream_t s) {
  if (rows <= 0 || kb <= 0) return 0;
  const int kb_tiles = (kb + 3) / 4;
  const long long total = ((rows + 127) / 128) * (long long)kb_tiles * 512;
  swizzle_scales_kernel<<<grid1d(total), 256, 0, s>>>((const uint8_t*)scales, (uint8_t*)out, rows, kb, kb_tiles, total);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}
