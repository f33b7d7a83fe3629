// Flat-buffer optimizer kernels: sum of squares of the fp32 gradient shard, and AdamW on fp32 master
// weights that also writes the bf16 compute copy. The clip coefficient is derived on the device from
// the squared-norm word, so the step needs no host synchronisation. This is the single-rank case of
// the reference's clip_grad_norm_ + AdamW step (gpu_process_worker.py:1052-1079).
#include <cuda_bf16.h>

#include "../launchers.h"

namespace agrpo {

namespace {

__global__ void sumsq_kernel(const float* __restrict__ g, long long n, float scale, float* __restrict__ out) {
  float acc = 0.f;
  const long long n4 = n / 4;
  const float4* g4 = reinterpret_cast<const float4*>(g);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) {
    const float4 v = g4[i];
    acc += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
  }
  for (long long i = n4 * 4 + blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    acc += g[i] * g[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  __shared__ float sm[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) sm[warp] = acc;
  __syncthreads();
  if (warp == 0) {
    acc = lane < (blockDim.x >> 5) ? sm[lane] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) atomicAdd(out, acc * scale * scale);
  }
}

struct AdamW {
  float lr, beta1, beta2, eps, wd, inv_bc1, inv_sqrt_bc2, coef;

  __device__ __forceinline__ void update(float g, float& p, float& m, float& v) const {
    g *= coef;
    p *= (1.f - lr * wd);
    m = beta1 * m + (1.f - beta1) * g;
    v = beta2 * v + (1.f - beta2) * g * g;
    const float denom = sqrtf(v) * inv_sqrt_bc2 + eps;
    p -= lr * inv_bc1 * m / denom;
  }
};

// norm_sq points at the squared global gradient norm (already scaled by grad_scale^2).
// clip coefficient = min(1, max_norm / (sqrt(norm_sq) + 1e-6)); max_norm <= 0 disables clipping.
// Bound by memory: 34 bytes a parameter (p, m, v, g read and written, the bf16 copy written). Four parameters a thread, so that
// every access is a whole 16 bytes: 607 M parameters took 4.04 ms (5.1 TB/s) with one parameter a thread, 3.69 ms (5.6 TB/s) with four.
__global__ void __launch_bounds__(256)
adamw_kernel(float* __restrict__ p, float* __restrict__ m, float* __restrict__ v, float* __restrict__ g, __nv_bfloat16* __restrict__ p16,
             long long n, int vec, AdamW k, float bc1, float bc2, const float* __restrict__ norm_sq, float max_norm, int zero_grad) {
  if (max_norm > 0.f && norm_sq != nullptr) {
    const float nrm = sqrtf(*norm_sq);
    k.coef *= fminf(1.f, max_norm / (nrm + 1e-6f));
  }
  k.inv_bc1 = 1.f / bc1;
  k.inv_sqrt_bc2 = rsqrtf(bc2);
  const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
  const long long n4 = vec ? n / 4 : 0;
  for (long long i = first; i < n4; i += stride) {
    const float4 gi = __ldcs(reinterpret_cast<const float4*>(g) + i);
    float4 pi = __ldcs(reinterpret_cast<const float4*>(p) + i);
    float4 mi = __ldcs(reinterpret_cast<const float4*>(m) + i);
    float4 vi = __ldcs(reinterpret_cast<const float4*>(v) + i);
    k.update(gi.x, pi.x, mi.x, vi.x);
    k.update(gi.y, pi.y, mi.y, vi.y);
    k.update(gi.z, pi.z, mi.z, vi.z);
    k.update(gi.w, pi.w, mi.w, vi.w);
    __stcs(reinterpret_cast<float4*>(p) + i, pi);
    __stcs(reinterpret_cast<float4*>(m) + i, mi);
    __stcs(reinterpret_cast<float4*>(v) + i, vi);
    if (zero_grad) __stcs(reinterpret_cast<float4*>(g) + i, make_float4(0.f, 0.f, 0.f, 0.f));
    if (p16 != nullptr) {
      const __nv_bfloat162 lo = __floats2bfloat162_rn(pi.x, pi.y), hi = __floats2bfloat162_rn(pi.z, pi.w);
      uint2 o;
      o.x = *reinterpret_cast<const uint32_t*>(&lo);
      o.y = *reinterpret_cast<const uint32_t*>(&hi);
      reinterpret_cast<uint2*>(p16)[i] = o;
    }
  }
  for (long long i = n4 * 4 + first; i < n; i += stride) {
    k.update(g[i], p[i], m[i], v[i]);
    if (p16 != nullptr) p16[i] = __float2bfloat16(p[i]);
    if (zero_grad) g[i] = 0.f;
  }
}

__global__ void cast_f32_bf16_kernel(const float* __restrict__ in, __nv_bfloat16* __restrict__ out, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = __float2bfloat16(in[i]);
}

}  // namespace

void launch_sumsq(const float* g, long long n, float scale, float* out, cudaStream_t s) {
  if (n == 0) return;
  long long blocks = (n / 4 + 255) / 256;
  if (blocks < 1) blocks = 1;
  if (blocks > 148 * 8) blocks = 148 * 8;
  sumsq_kernel<<<(int)blocks, 256, 0, s>>>(g, n, scale, out);
  check_cuda(cudaGetLastError(), "sumsq");
}

void launch_adamw(float* p, float* m, float* v, float* g, void* p16, long long n, float lr, float beta1, float beta2,
                  float eps, float wd, int step, float grad_scale, const float* norm_sq, float max_norm, bool zero_grad,
                  cudaStream_t s) {
  if (n == 0) return;
  const float bc1 = 1.f - powf(beta1, (float)step);
  const float bc2 = 1.f - powf(beta2, (float)step);
  const auto aligned = [](const void* q, uintptr_t to) { return (reinterpret_cast<uintptr_t>(q) & (to - 1)) == 0; };
  const int vec = aligned(p, 16) && aligned(m, 16) && aligned(v, 16) && aligned(g, 16) && aligned(p16, 8) ? 1 : 0;
  long long blocks = ((vec ? n / 4 : n) + 255) / 256;
  if (blocks < 1) blocks = 1;
  if (blocks > 148 * 16) blocks = 148 * 16;
  const AdamW k{lr, beta1, beta2, eps, wd, 0.f, 0.f, grad_scale};
  adamw_kernel<<<(int)blocks, 256, 0, s>>>(p, m, v, g, (__nv_bfloat16*)p16, n, vec, k, bc1, bc2, norm_sq, max_norm, zero_grad ? 1 : 0);
  check_cuda(cudaGetLastError(), "adamw");
}

void launch_cast_f32_bf16(const float* in, void* out, long long n, cudaStream_t s) {
  if (n == 0) return;
  long long blocks = (n + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  cast_f32_bf16_kernel<<<(int)blocks, 256, 0, s>>>(in, (__nv_bfloat16*)out, n);
  check_cuda(cudaGetLastError(), "cast_f32_bf16");
}

}  // namespace agrpo
