// What the epilogues of the tcgen05 GEMM kernels share: bf16 pieces of eight and activations over a register array.
#pragma once
#include "common.cuh"

namespace rb { namespace {

__device__ __forceinline__ uint4 pack8(const float* v) {
  uint4 r;
  __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]);
  __nv_bfloat162 b = __floats2bfloat162_rn(v[2], v[3]);
  __nv_bfloat162 c = __floats2bfloat162_rn(v[4], v[5]);
  __nv_bfloat162 d = __floats2bfloat162_rn(v[6], v[7]);
  r.x = *reinterpret_cast<uint32_t*>(&a);
  r.y = *reinterpret_cast<uint32_t*>(&b);
  r.z = *reinterpret_cast<uint32_t*>(&c);
  r.w = *reinterpret_cast<uint32_t*>(&d);
  return r;
}
__device__ __forceinline__ void unpack8(const uint4& u, float* v) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __bfloat1622float2(h[i]);
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}

__device__ __forceinline__ float tanh_fast(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Activation over a register array with the selector hoisted out of the element loop
// (rai-core/src/hlops/activations.rs:20-32); fast-math forms, results are rounded to bf16 anyway.
template <int N>
__device__ __forceinline__ void act_inplace(int act, float (&v)[N], float2 ac) {
  if (act == RB_ACT_SILU) {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = __fdividef(v[i], 1.0f + __expf(-v[i]));
  } else if (act == RB_ACT_GELU_TANH) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const float x = v[i];
      v[i] = 0.5f * x * (1.0f + tanh_fast(0.7978845608028654f * (x + 0.044715f * x * x * x)));
    }
  } else if (act == RB_ACT_GELU_ERF) {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = v[i] * 0.5f * (1.0f + erff(v[i] * 0.7071067811865476f));
  } else if (act == RB_ACT_RELU) {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = fmaxf(v[i], 0.f);
  } else if (act == RB_ACT_RELU2) {
#pragma unroll
    for (int i = 0; i < N; ++i) { const float r = fmaxf(v[i], 0.f); v[i] = r * r; }
  } else if (act == RB_ACT_XIELU) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const float z = v[i];
      const float curve = z > 0.f ? ac.x * z * z : ac.y * (__expf(fminf(z, 0.f)) - 1.0f - z);
      v[i] = fmaf(0.5f, z, curve);
    }
  }
}

}}  // namespace rb::(anonymous)
