// Device helpers shared by the kernels of layer-list decoders (stack_ops.cu, stack_gqa.cu, stack_moe.cu): typed loads and
// stores of weight / cache elements (bf16 or fp32), warp and block reductions with a fixed summation order.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

#include "kernels.h"

namespace hb {
namespace {

template <typename T> __device__ __forceinline__ float ldf(const T* p, size_t i);
template <> __device__ __forceinline__ float ldf<float>(const float* p, size_t i) { return p[i]; }
template <> __device__ __forceinline__ float ldf<bf16>(const bf16* p, size_t i) { return __bfloat162float(p[i]); }
template <typename T> __device__ __forceinline__ void stf(T* p, size_t i, float v);
template <> __device__ __forceinline__ void stf<float>(float* p, size_t i, float v) { p[i] = v; }
template <> __device__ __forceinline__ void stf<bf16>(bf16* p, size_t i, float v) { p[i] = __float2bfloat16(v); }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// sum over the block; every thread gets the result.  red: >= 32 floats of shared memory.
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  float t = (l < nw) ? red[l] : 0.f;
  return warp_sum(t);
}
// sums of a product's slabs, in slab order: four columns from n (a multiple of four) of row m, or column n
__device__ __forceinline__ float4 slab_sum4(const Slabs& s, size_t m, int n) {
  const int ns = s.segs[n >> 7];
  const size_t step = (size_t)s.M * s.N;
  const float* p = s.ws + m * s.N + n;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  int i = 0;
  for (; i + 4 <= ns; i += 4) {  // four loads in flight
    float4 v[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = *reinterpret_cast<const float4*>(p + (i + e) * step);
#pragma unroll
    for (int e = 0; e < 4; ++e) acc = make_float4(acc.x + v[e].x, acc.y + v[e].y, acc.z + v[e].z, acc.w + v[e].w);
  }
  for (; i < ns; ++i) {
    const float4 v = *reinterpret_cast<const float4*>(p + i * step);
    acc = make_float4(acc.x + v.x, acc.y + v.y, acc.z + v.z, acc.w + v.w);
  }
  return acc;
}
__device__ __forceinline__ float slab_sum1(const Slabs& s, size_t m, int n) {
  const int ns = s.segs[n >> 7];
  const size_t step = (size_t)s.M * s.N;
  const float* p = s.ws + m * s.N + n;
  float acc = 0.f;
  for (int i = 0; i < ns; ++i) acc += p[i * step];
  return acc;
}
__device__ __forceinline__ float sigmoidf_(float z) { return 1.f / (1.f + expf(-z)); }

}  // namespace
}  // namespace hb
