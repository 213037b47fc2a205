// Shared helpers of libb200seq (sequence-mixer kernels, sm_100a only).
#pragma once
#include "../../include/b2l_seq.h"
#include "b2l_common.cuh"

namespace b2l {

// An "act" element is bf16 or f32; kernels are templated on it and compute in f32.
template <typename T> __device__ __forceinline__ float ld_act(const T* p, size_t i);
template <> __device__ __forceinline__ float ld_act<__nv_bfloat16>(const __nv_bfloat16* p, size_t i) { return __bfloat162float(p[i]); }
template <> __device__ __forceinline__ float ld_act<float>(const float* p, size_t i) { return p[i]; }
template <typename T> __device__ __forceinline__ void st_act(T* p, size_t i, float v);
template <> __device__ __forceinline__ void st_act<__nv_bfloat16>(__nv_bfloat16* p, size_t i, float v) { p[i] = __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ void st_act<float>(float* p, size_t i, float v) { p[i] = v; }

// Four elements at once, p aligned to all four of them.
__device__ __forceinline__ float4 ld_act4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 ld_act4(const __nv_bfloat16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
}
__device__ __forceinline__ void st_act4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void st_act4(__nv_bfloat16* p, float4 v) {
  const __nv_bfloat162 y[2] = {__floats2bfloat162_rn(v.x, v.y), __floats2bfloat162_rn(v.z, v.w)};
  *reinterpret_cast<uint2*>(p) = *reinterpret_cast<const uint2*>(y);
}

// x / y for y >= 1/4 without a branch: the approximate reciprocal (at most 1 ulp off, as documented), one Newton step, and the quotient corrected by its own
// remainder (Markstein).  While 1/y is a normal number, so for y up to 2^126, that is the correctly rounded quotient, subnormal ones as well: 2 in 10^8 are 1
// ulp off, over all mantissas of y and reciprocals off by up to 1 ulp.  Four gated outputs in a row took the attention kernel 730 cycles with the
// division operator, 190 so.
__device__ __forceinline__ float over_f(float x, float y) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
  r = fmaf(r, fmaf(-y, r, 1.0f), r);
  const float q = x * r, d = fmaf(fmaf(-y, q, x), r, q);
  if (y == INFINITY) return x * 0.0f;
  return fabsf(q) < INFINITY ? d : q;                 // an infinite quotient has no remainder
}
// a quarter of both sides of the fraction: 1 + e^-z up to the largest f32 then has a normal reciprocal (down to z = -88.7), and no rounding changes
__device__ __forceinline__ float sigmoid_f(float z) { return over_f(0.25f, fmaf(expf(-z), 0.25f, 0.25f)); }
__device__ __forceinline__ float silu_f(float z) { return over_f(0.25f * z, fmaf(expf(-z), 0.25f, 0.25f)); }
// log(1 + e^z) = max(z, 0) + log(1 + u), u = e^-|z| <= 1, and log(1 + u) = 2 atanh(s), s = u / (2 + u) <= 1/3, by atanh's series to s^15 (the next term is
// below 2e-9 of the sum): no branch and some 20 operations, where log1pf(expf(z)) took twice as many.
__device__ __forceinline__ float softplus_f(float z) {
  const float u = expf(-fabsf(z)), s = over_f(u, 2.0f + u), t = s * s;
  float p = 1.0f / 15.0f;
  p = fmaf(p, t, 1.0f / 13.0f);
  p = fmaf(p, t, 1.0f / 11.0f);
  p = fmaf(p, t, 1.0f / 9.0f);
  p = fmaf(p, t, 1.0f / 7.0f);
  p = fmaf(p, t, 1.0f / 5.0f);
  p = fmaf(p, t, 1.0f / 3.0f);
  return fmaxf(z, 0.0f) + 2.0f * fmaf(p * t, s, s);
}
__device__ __forceinline__ float gelu_tanh_f(float z) {
  return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
}

// A gated unit from the two halves of one product: act(a) * b, or the clamped unit g = min(a, limit),
// u = clamp(b, -limit, limit), g * sigmoid(1.702 g) * (u + 1).
__device__ __forceinline__ float gated_pair(float a, float b, int act, float limit) {
  if (act == B2L_SEQ_ACT_CLAMPED_SWISH) {
    const float g = fminf(a, limit), u = fminf(fmaxf(b, -limit), limit);
    return g * sigmoid_f(1.702f * g) * (u + 1.0f);
  }
  return (act == B2L_SEQ_ACT_GELU_TANH ? gelu_tanh_f(a) : (act == B2L_SEQ_ACT_SILU ? silu_f(a) : sigmoid_f(a))) * b;
}

// Dot product of a weight row with a vector in shared memory (f32); the warp's lanes stride the row.
template <typename act_t>
__device__ __forceinline__ float row_dot(const act_t* __restrict__ w, const float* __restrict__ x, int n, int lane, bool vec) {
  float acc = 0.f;
  if (vec) {                                         // 16-byte loads: n a multiple of 8 (bf16) / 4 (f32), aligned rows
    constexpr int PER = 16 / sizeof(act_t);
    for (int i = lane * PER; i < n; i += 32 * PER) {
      const uint4 u = *reinterpret_cast<const uint4*>(w + i);
      if (sizeof(act_t) == 2) {
        const uint32_t ww[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          acc = fmaf(__uint_as_float(ww[q] << 16), x[i + 2 * q], acc);
          acc = fmaf(__uint_as_float(ww[q] & 0xffff0000u), x[i + 2 * q + 1], acc);
        }
      } else {
        acc = fmaf(__uint_as_float(u.x), x[i], acc);
        acc = fmaf(__uint_as_float(u.y), x[i + 1], acc);
        acc = fmaf(__uint_as_float(u.z), x[i + 2], acc);
        acc = fmaf(__uint_as_float(u.w), x[i + 3], acc);
      }
    }
  } else {
    for (int i = lane; i < n; i += 32) acc = fmaf(ld_act(w, i), x[i], acc);
  }
  return warp_sum(acc);
}

// whether p may be read by fours of elements of `size` bytes
static inline bool al4(const void* p, size_t size) { return (reinterpret_cast<uintptr_t>(p) & (4 * size - 1)) == 0; }
static inline bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Calls `fn.template operator()<T>()` with the element type of act_dtype.
#define B2L_SEQ_DISPATCH(act_dtype, ...)                                   \
  do {                                                                     \
    if ((act_dtype) == B2L_BF16) { using act_t = __nv_bfloat16; __VA_ARGS__; } \
    else if ((act_dtype) == B2L_F32) { using act_t = float; __VA_ARGS__; }  \
    else { b2l::set_error("act_dtype %d unsupported", (int)(act_dtype)); return B2L_E_UNSUPPORTED; } \
  } while (0)

}  // namespace b2l
