// Flat-buffer optimizer kernels: sum of squares of the fp32 gradient shard, and AdamW on fp32 master
// weights that also writes the bf16 compute copy. The clip coefficient is derived on the device from
// the squared-norm word, so the step needs no host synchronisation. This is the single-rank case of
// the reference's clip_grad_norm_ + AdamW step (gpu_process_worker.py:1052-1079).
#include <cuda_bf16.h>

#include "../common/ptx.cuh"
#include "../launchers.h"

namespace agrpo {

namespace {

__global__ void sumsq_kernel(const float* __restrict__ g, long long n, float scale, float* __restrict__ out) {
  float acc = 0.f;
  const long long n4 = n / 4;
  const float4* g4 = reinterpret_cast<const float4*>(g);
  // four loads in flight a thread: 1550 M values 0.98 -> 0.95 ms (6.5 TB/s)
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n4; i += 4 * stride) {
    float4 w[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) w[u] = i + u * stride < n4 ? g4[i + u * stride] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int u = 0; u < 4; ++u) acc += w[u].x * w[u].x + w[u].y * w[u].y + w[u].z * w[u].z + w[u].w * w[u].w;
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

// kVec fp32 values with one access of 32 or 16 bytes.
template <int kVec>
__device__ __forceinline__ void ld_vec(const float* p, uint32_t (&r)[kVec]) {
  if constexpr (kVec == 8) {
    ld_global_32b(p, r);
  } else {
    const uint4 w = *reinterpret_cast<const uint4*>(p);
    r[0] = w.x; r[1] = w.y; r[2] = w.z; r[3] = w.w;
  }
}
template <int kVec>
__device__ __forceinline__ void st_vec(float* p, const uint32_t (&r)[kVec]) {
  if constexpr (kVec == 8) st_global_32b(p, r);
  else *reinterpret_cast<uint4*>(p) = make_uint4(r[0], r[1], r[2], r[3]);
}

// norm_sq points at the squared global gradient norm (already scaled by grad_scale^2).
// clip coefficient = min(1, max_norm / (sqrt(norm_sq) + 1e-6)); max_norm <= 0 disables clipping.
// Bound by memory: 34 bytes a parameter (p, m, v, g read and written, the bf16 copy written). Eight parameters a thread, every access
// 32 bytes, and as many blocks as that takes: 607 M parameters took 3.52 ms (5.9 TB/s) with four a thread and 148 x 16 blocks that
// stride over them, 3.38 ms with eight, 2.99 ms (6.9 TB/s) without the stride: blocks that start in order keep to a few DRAM pages
// of each of the nine streams. Slices whose buffers keep to 16 bytes (8 for the bf16 copy) but not to 32 take four
// a thread: 64 M parameters 0.346 ms, 0.341 aligned, 0.683 one by one.
template <int kVec>  // 1: buffers that no wide access fits
__global__ void __launch_bounds__(256)
adamw_kernel(float* __restrict__ p, float* __restrict__ m, float* __restrict__ v, float* __restrict__ g, __nv_bfloat16* __restrict__ p16,
             long long n, AdamW k, float bc1, float bc2, const float* __restrict__ norm_sq, float max_norm, int zero_grad) {
  if (max_norm > 0.f && norm_sq != nullptr) {
    const float nrm = sqrtf(*norm_sq);
    k.coef *= fminf(1.f, max_norm / (nrm + 1e-6f));
  }
  k.inv_bc1 = 1.f / bc1;
  k.inv_sqrt_bc2 = rsqrtf(bc2);
  const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
  const long long whole = kVec > 1 ? n / kVec * kVec : 0;
  if constexpr (kVec > 1) {
    const long long at = kVec * first;
    if (at < whole) {  // the launcher starts a thread for each
      uint32_t gi[kVec], pi[kVec], mi[kVec], vi[kVec];
      ld_vec(g + at, gi);
      ld_vec(p + at, pi);
      ld_vec(m + at, mi);
      ld_vec(v + at, vi);
      float q[kVec];
#pragma unroll
      for (int j = 0; j < kVec; ++j) {
        float mj = __uint_as_float(mi[j]), vj = __uint_as_float(vi[j]);
        q[j] = __uint_as_float(pi[j]);
        k.update(__uint_as_float(gi[j]), q[j], mj, vj);
        pi[j] = __float_as_uint(q[j]);
        mi[j] = __float_as_uint(mj);
        vi[j] = __float_as_uint(vj);
        gi[j] = 0u;
      }
      st_vec(p + at, pi);
      st_vec(m + at, mi);
      st_vec(v + at, vi);
      if (zero_grad) st_vec(g + at, gi);
      if (p16 != nullptr) {
        if constexpr (kVec == 8)
          *reinterpret_cast<uint4*>(p16 + at) =
              make_uint4(pack_bf16x2(q[0], q[1]), pack_bf16x2(q[2], q[3]), pack_bf16x2(q[4], q[5]), pack_bf16x2(q[6], q[7]));
        else
          *reinterpret_cast<uint2*>(p16 + at) = make_uint2(pack_bf16x2(q[0], q[1]), pack_bf16x2(q[2], q[3]));
      }
    }
  }
  for (long long i = whole + first; i < n; i += stride) {
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
  const auto all = [&](uintptr_t to) { return aligned(p, to) && aligned(m, to) && aligned(v, to) && aligned(g, to) && aligned(p16, to / 2); };
  const int vec = all(32) ? 8 : all(16) ? 4 : 1;
  long long blocks = (n / vec + 255) / 256;
  if (blocks < 1) blocks = 1;
  if (vec == 1 && blocks > 148 * 16) blocks = 148 * 16;
  const AdamW k{lr, beta1, beta2, eps, wd, 0.f, 0.f, grad_scale};
  const auto kernel = vec == 8 ? adamw_kernel<8> : vec == 4 ? adamw_kernel<4> : adamw_kernel<1>;
  kernel<<<(int)blocks, 256, 0, s>>>(p, m, v, g, (__nv_bfloat16*)p16, n, k, bc1, bc2, norm_sq, max_norm, zero_grad ? 1 : 0);
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
