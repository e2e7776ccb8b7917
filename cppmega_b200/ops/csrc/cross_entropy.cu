// Softmax cross-entropy over a chunk of bf16 logits, fused with its own backward:
// per row compute max / log-sum-exp / target logit (one pass, online rescaling), write the
// per-token loss, then overwrite the logits in place with
//     dlogits = weight[row] * (softmax - onehot(label))
// so the caller can feed them straight into the dgrad / wgrad GEMMs.  The logits chunk is read
// twice (second read mostly from L2) and written once; full logits never exist.
// Stands in for the Liger / CCE / native fused linear-CE paths of the reference
// (cppmega/megatron/apply_linear_ce_patch.py:251-527) with a true per-token `none` reduction.
#include "common.cuh"

namespace cm {

constexpr int CE_THREADS = 512;
constexpr float LOG2E = 1.4426950408889634f;

__device__ __forceinline__ float ce_ex2(float x) {
  float y;
  asm("ex2.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void ce_unpack(const uint4& v, float (&f)[8]) {
  const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int j = 0; j < 4; ++j) { const float2 t = __bfloat1622float2(b[j]); f[2 * j] = t.x; f[2 * j + 1] = t.y; }
}

// U: 16-byte vectors a thread requests before it uses the first.  With gradients 4096 x 131072 takes 491 us with four and 603 with
// one (floor 325: one read and one write; the second read comes mostly from L2, and 2 x 537 M exponentials take 245), 4096 x 65536
// 247 and 266; shorter rows leave most of a group empty (4096 x 8192: 59.5 us with four, 55.2 with one; 4096 x 1024: 31 and 27), and
// without gradients it never pays (512 x 65536: 22.7 and 21.2).
template <int U>
__global__ void __launch_bounds__(CE_THREADS) ce_fwd_bwd_kernel(__nv_bfloat16* __restrict__ logits, const long long* __restrict__ labels,
                                                                const float* __restrict__ weights, float* __restrict__ loss_out,
                                                                float* __restrict__ lse_out, int rows, int V, long long ld,
                                                                int ignore_index, int write_grad) {
  __shared__ float s_max[CE_THREADS / 32], s_sum[CE_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nvec = V / 8;
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    __nv_bfloat16* lr = logits + (long long)row * ld;
    uint4* lv = reinterpret_cast<uint4*>(lr);
    const long long label = labels[row];
    const bool ignored = (label == ignore_index) || label < 0 || label >= V;
    if (ignored) {
      if (threadIdx.x == 0) { loss_out[row] = 0.f; if (lse_out) lse_out[row] = 0.f; }
      if (write_grad) {
        const uint4 z = make_uint4(0, 0, 0, 0);
        for (int i = threadIdx.x; i < nvec; i += CE_THREADS) lv[i] = z;
      }
      continue;
    }
    float mx = -INFINITY, sm = 0.f;
    for (int i0 = threadIdx.x; i0 < nvec; i0 += CE_THREADS * U) {
      uint4 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (i0 + u * CE_THREADS < nvec) v[u] = lv[i0 + u * CE_THREADS];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (i0 + u * CE_THREADS >= nvec) break;
        float f[8];
        ce_unpack(v[u], f);
        float vm = f[0];
#pragma unroll
        for (int j = 1; j < 8; ++j) vm = fmaxf(vm, f[j]);
        if (vm > mx) { sm *= __expf(mx - vm); mx = vm; }
#pragma unroll
        for (int j = 0; j < 8; ++j) sm += ce_ex2((f[j] - mx) * LOG2E);
      }
    }
    // block reduce (max, sum)
    float wm = warp_max(mx);
    sm = (mx == -INFINITY) ? 0.f : sm * __expf(mx - wm);     // lanes / warps that saw no element
    sm = warp_sum(sm);
    if (lane == 0) { s_max[warp] = wm; s_sum[warp] = sm; }
    __syncthreads();
    float gm = s_max[0];
#pragma unroll
    for (int i = 1; i < CE_THREADS / 32; ++i) gm = fmaxf(gm, s_max[i]);
    float gs = 0.f;
#pragma unroll
    for (int i = 0; i < CE_THREADS / 32; ++i) gs += (s_max[i] == -INFINITY) ? 0.f : s_sum[i] * __expf(s_max[i] - gm);
    const float lse = gm + __logf(gs);
    const float tgt = __bfloat162float(lr[label]);
    __syncthreads();          // everyone has read the target logit and the shared partials
    if (threadIdx.x == 0) { loss_out[row] = lse - tgt; if (lse_out) lse_out[row] = lse; }
    if (!write_grad) continue;
    const float wgt = weights ? weights[row] : 1.f;
    const int lvec = int(label >> 3), lsub = int(label & 7);
    for (int i0 = threadIdx.x; i0 < nvec; i0 += CE_THREADS * U) {
      uint4 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (i0 + u * CE_THREADS < nvec) v[u] = lv[i0 + u * CE_THREADS];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + u * CE_THREADS;
        if (i >= nvec) break;
        float f[8];
        ce_unpack(v[u], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = ce_ex2((f[j] - lse) * LOG2E);
        if (i == lvec) {
#pragma unroll
          for (int j = 0; j < 8; ++j) if (j == lsub) f[j] -= 1.f;
        }
        uint4 o;
        uint32_t* op = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
        for (int j = 0; j < 4; ++j) op[j] = pack_bf16(f[2 * j] * wgt, f[2 * j + 1] * wgt);
        lv[i] = o;
      }
    }
  }
}

// out = bf16(in * g) with the scalar on the device: the upstream factor of the stored gradients, applied and rounded in one
// pass: 559 us for 131072 x 4096 fp32 (485 at the copy rate), where the library's product and cast took 2,170 (fp32 in: multiplied in fp32; bf16 in: multiplied by bf16(g), as the tensor library multiplies two bf16 values)
template <typename T>
__global__ void __launch_bounds__(256) scale_to_bf16_kernel(const T* __restrict__ in, __nv_bfloat16* __restrict__ out,
                                                            const float* __restrict__ g_ptr, long long nvec) {
  const float g = sizeof(T) == 4 ? *g_ptr : __bfloat162float(__float2bfloat16(*g_ptr));
  constexpr int U = 2;
  const long long step = (long long)gridDim.x * blockDim.x;
  for (long long i0 = blockIdx.x * (long long)blockDim.x + threadIdx.x; i0 < nvec; i0 += step * U) {
    uint4 raw[U][sizeof(T) == 4 ? 2 : 1];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = i0 + u * step;
      if (i < nvec) {
        const uint4* src = reinterpret_cast<const uint4*>(in + i * 8);
        raw[u][0] = src[0];
        if constexpr (sizeof(T) == 4) raw[u][1] = src[1];
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = i0 + u * step;
      if (i >= nvec) break;
      float f[8];
      if constexpr (sizeof(T) == 4) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          f[4 * j] = __uint_as_float(raw[u][j].x); f[4 * j + 1] = __uint_as_float(raw[u][j].y);
          f[4 * j + 2] = __uint_as_float(raw[u][j].z); f[4 * j + 3] = __uint_as_float(raw[u][j].w);
        }
      } else {
        ce_unpack(raw[u][0], f);
      }
      uint4 o;
      uint32_t* op = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
      for (int j = 0; j < 4; ++j) op[j] = pack_bf16(f[2 * j] * g, f[2 * j + 1] * g);
      reinterpret_cast<uint4*>(out)[i] = o;
    }
  }
}

}  // namespace cm

// out[n] bf16 = in[n] * g[0]; in fp32 or bf16, n % 8 == 0, 16-byte aligned
extern "C" int cm_scale_to_bf16(const void* in, int in_fp32, void* out, const float* g, long long n, cudaStream_t s) {
  if (n <= 0) return 0;
  if (n % 8 || (reinterpret_cast<uintptr_t>(in) & 15) || (reinterpret_cast<uintptr_t>(out) & 15)) return -10;
  const long long nvec = n / 8, blocks = (nvec + 511) / 512;
  const int grid = (int)(blocks < (long long)cm::sm_count() * 8 ? blocks : (long long)cm::sm_count() * 8);
  if (in_fp32) cm::scale_to_bf16_kernel<float><<<grid, 256, 0, s>>>((const float*)in, (__nv_bfloat16*)out, g, nvec);
  else cm::scale_to_bf16_kernel<__nv_bfloat16><<<grid, 256, 0, s>>>((const __nv_bfloat16*)in, (__nv_bfloat16*)out, g, nvec);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

// logits [rows, V] bf16 (row pitch ld, V % 8 == 0) are replaced by weighted dlogits when
// write_grad != 0.  loss_out[rows] receives lse - target (0 for ignored rows).
extern "C" int cm_ce_fwd_bwd(void* logits, const long long* labels, const float* weights, float* loss_out,
                             float* lse_out, int rows, int V, long long ld, int ignore_index, int write_grad,
                             cudaStream_t s) {
  if (rows <= 0) return 0;
  if (V % 8 || ld % 8) return -10;
  int grid = rows < cm::sm_count() * 2 ? rows : cm::sm_count() * 2;
  const auto kernel = write_grad && V >= 65536 ? cm::ce_fwd_bwd_kernel<4> : cm::ce_fwd_bwd_kernel<1>;
  kernel<<<grid, cm::CE_THREADS, 0, s>>>((__nv_bfloat16*)logits, labels, weights, loss_out, lse_out, rows, V, ld, ignore_index, write_grad);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}
