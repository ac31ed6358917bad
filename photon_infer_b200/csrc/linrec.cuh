// What the kernels of the recurrent mixers share: gates, asynchronous copies, packed 32-bit arithmetic, and the sums of
// lanes that share a column.
#pragma once
#include "common.cuh"
#include <math.h>

__device__ __forceinline__ float lr_softplus(float x) { return x > 20.f ? x : log1pf(expf(x)); }
__device__ __forceinline__ float lr_logsigmoid(float x) { return fminf(x, 0.f) - log1pf(expf(-fabsf(x))); }
// Inputs of mode 2 (forget and write).
__device__ __forceinline__ float lr_silu(float x) { return x / (1.0f + expf(-x)); }
__device__ __forceinline__ float lr_write_gate(float z, float bias, float lower) { return (1.0f - lower) / (1.0f + expf(z + bias)); }
// The product b of decays and what it lacks to 1, B = 1 - b, brought forward by a decay that lacks `gone` to 1 (`scaled` is that
// decay times b).  Near 1 a product rounds to 2^-25 of itself at every token, always alike where the decays hardly change, which over
// hundreds of tokens is far more than the state's own roundings; B keeps all its bits there.  Below 1/2 the product is the exact one.
__device__ __forceinline__ void lr_decay(float scaled, float gone, float& b, float& B) {
  B = fmaf(gone, b, B);
  b = B < 0.5f ? 1.0f - B : scaled;
}
// A decay as one number: -B (minus zero for a decay of 1) where B lies between 0 and 1/2, else b (also behind a decay that the
// rounding of a running maximum has put above 1).  x decays to fma(code, x, x or 0): the sign says which.
__device__ __forceinline__ float lr_code(float b, float B) { return B >= 0.f && B < 0.5f ? -fabsf(B) : b; }
__device__ __forceinline__ uint32_t lr_mask(float code) { return (uint32_t)(__float_as_int(code) >> 31); }
__device__ __forceinline__ float lr_apply(float code, float x) { return fmaf(code, x, __uint_as_float(__float_as_uint(x) & lr_mask(code))); }
__device__ __forceinline__ void lr_cp4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void lr_cp16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void lr_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int K> __device__ __forceinline__ void lr_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(K) : "memory"); }

// ---------------------------------------------------------------- packed pairs of neighbouring rows
#define LRR_C 4                 // columns of a lane: 2 or 4
typedef unsigned long long lr_pair;
struct alignas(LRR_C * 4) LrCols { float x[LRR_C]; };   // the lane's columns of one row
__device__ __forceinline__ lr_pair lr_dup(float x) { lr_pair d; asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(x)); return d; }
__device__ __forceinline__ lr_pair lr_mul2(lr_pair a, lr_pair b) { lr_pair d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ lr_pair lr_fma2(lr_pair a, lr_pair b, lr_pair c) {
  lr_pair d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ float lr_sum2(lr_pair a) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a));
  return x + y;
}
__device__ __forceinline__ lr_pair lr_make(float x, float y) { lr_pair d; asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y)); return d; }
__device__ __forceinline__ void lr_split(lr_pair a, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a)); }

// The lanes' shares of NV sums meet over the distances D, D / 2 .. 1: while a lane holds several sums it keeps half of them (the
// upper half where the distance's bit of its number is set) and hands over the others.
template <int D, int NV, int M>
__device__ __forceinline__ void lr_meet(float (&val)[M], int sub) {
  if constexpr (D > 0) {
    if constexpr (NV > 1) {
      const bool up = sub & D;
#pragma unroll
      for (int i = 0; i < NV / 2; ++i) {
        const float own = up ? val[i + NV / 2] : val[i], other = up ? val[i] : val[i + NV / 2];
        val[i] = own + __shfl_xor_sync(0xffffffffu, other, D);
      }
      lr_meet<D / 2, NV / 2>(val, sub);
    } else {
      val[0] += __shfl_xor_sync(0xffffffffu, val[0], D);
      lr_meet<D / 2, 1>(val, sub);
    }
  }
}

