// 16-byte bf16 vectors and block reductions shared by the memory-bound kernels.
#pragma once
#include "common.cuh"

namespace pb {

struct alignas(16) Bf8 {
  __nv_bfloat162 v[4];
};

PB_DEVICE void bf8_to_f(const Bf8& b, float* f) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(b.v[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
PB_DEVICE Bf8 f_to_bf8(const float* f) {
  Bf8 b;
#pragma unroll
  for (int i = 0; i < 4; ++i) b.v[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return b;
}

template <int THREADS>
PB_DEVICE float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  float r = (l < THREADS / 32) ? red[l] : 0.f;
  r = warp_sum(r);
  return r;
}
template <int THREADS>
PB_DEVICE float block_max(float v, float* red) {
  v = warp_max(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  float r = (l < THREADS / 32) ? red[l] : -INFINITY;
  r = warp_max(r);
  return r;
}

// 16-byte asynchronous copy global -> shared (a thread waits for its own copies with cp_async_wait)
PB_DEVICE void cp_async_16(void* smem_dst, const void* gsrc) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem_dst)), "l"(gsrc) : "memory");
}
PB_DEVICE void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
PB_DEVICE void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

}  // namespace pb
