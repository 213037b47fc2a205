// Row-wise and element-wise mechanisms of the sequence mixers: embedding into an f32 residual stream, RMS norms
// (pre, post + residual + next pre fused), gated activations, short causal convolution with carried inputs, unit
// norms, decay factors, grouped read-out norm with its gate.  All arithmetic is f32; `act_t` is only the storage
// type of projection outputs and weights.
#include <type_traits>

#include "seq_common.cuh"

namespace b2l {

template <typename act_t, typename idx_t>
__global__ void seq_embed_kernel(const idx_t* __restrict__ tok, const act_t* __restrict__ table, float scale,
                                 float* __restrict__ x, act_t* __restrict__ h, int D, int vocab) {
  long long t = (long long)tok[blockIdx.x];
  if (t < 0 || t >= vocab) t = 0;
  const act_t* src = table + (size_t)t * D;
  float* dst = x + (size_t)blockIdx.x * D;
  for (int i = threadIdx.x; i < D; i += blockDim.x) {
    const float v = ld_act(src, i) * scale;
    dst[i] = v;
    if (h) st_act(h, (size_t)blockIdx.x * D + i, v);
  }
}

// The same by fours of elements (D a multiple of 4, aligned tables): the loop above makes D / 128 dependent rounds to memory.  Measured (us, above / this): one
// row of 1024 2.6 / 1.6, of 4096 6.6 / 2.9; 777 rows of 1024 3.1 / 2.1; 2048 rows of 4096 9.5 / 6.8.
template <typename act_t, typename idx_t>
__global__ void seq_embed_vec_kernel(const idx_t* __restrict__ tok, const act_t* __restrict__ table, float scale,
                                     float* __restrict__ x, act_t* __restrict__ h, int D, int vocab) {
  long long t = (long long)tok[blockIdx.x];
  if (t < 0 || t >= vocab) t = 0;
  const act_t* src = table + (size_t)t * D;
  const size_t row = (size_t)blockIdx.x * D;
#pragma unroll 2
  for (int i = threadIdx.x * 4; i < D; i += blockDim.x * 4) {
    float4 v = ld_act4(src + i);
    v = make_float4(v.x * scale, v.y * scale, v.z * scale, v.w * scale);
    st_act4(x + row + i, v);
    if (h) st_act4(h + row + i, v);
  }
}

template <typename act_t>
__global__ void __launch_bounds__(256) seq_rmsnorm_kernel(const float* __restrict__ x, const act_t* __restrict__ w, float eps,
                                                          act_t* __restrict__ out, const int* __restrict__ rows, int D) {
  __shared__ float red[32];
  const int r = rows ? rows[blockIdx.x] : blockIdx.x;
  const float* xr = x + (size_t)r * D;
  act_t* o = out + (size_t)blockIdx.x * D;
  float ss = 0.f;
  for (int i = threadIdx.x; i < D; i += blockDim.x) ss += xr[i] * xr[i];
  ss = block_sum(ss, red);
  const float rinv = 1.0f / sqrtf(ss / (float)D + eps);
  for (int i = threadIdx.x; i < D; i += blockDim.x) st_act(o, i, xr[i] * rinv * ld_act(w, i));
}

// The same by fours of elements with the row and its weights in registers (D a multiple of 4, at most 1024 * EPV; aligned rows): one round to memory instead of
// D / 128.  Measured (us, above / this): one row of 1024 2.7 / 1.6, of 4096 6.8 / 1.8; 777 rows of 1024 3.3 / 2.4; 2048 rows of 4096 16.3 / 6.4.
template <typename act_t, int EPV>
__global__ void __launch_bounds__(256) seq_rmsnorm_vec_kernel(const float* __restrict__ x, const act_t* __restrict__ w, float eps,
                                                              act_t* __restrict__ out, const int* __restrict__ rows, int D) {
  __shared__ float red[32];
  const float* xr = x + (size_t)(rows ? rows[blockIdx.x] : blockIdx.x) * D;
  act_t* o = out + (size_t)blockIdx.x * D;
  float4 v[EPV], wv[EPV];
  float ss = 0.f;
#pragma unroll
  for (int e = 0; e < EPV; ++e) {
    const int i = (threadIdx.x + e * 256) * 4;
    v[e] = i < D ? ld_act4(xr + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    wv[e] = i < D ? ld_act4(w + i) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int e = 0; e < EPV; ++e) ss += v[e].x * v[e].x + v[e].y * v[e].y + v[e].z * v[e].z + v[e].w * v[e].w;
  ss = block_sum(ss, red);
  const float r = 1.0f / sqrtf(ss / (float)D + eps);
#pragma unroll
  for (int e = 0; e < EPV; ++e) {
    const int i = (threadIdx.x + e * 256) * 4;
    if (i < D) st_act4(o + i, make_float4(v[e].x * r * wv[e].x, v[e].y * r * wv[e].y, v[e].z * r * wv[e].z, v[e].w * r * wv[e].w));
  }
}

// x += mult * rmsnorm(y) * w_post; optionally h = rmsnorm(x) * w_next, or x in the activation type (no w_next).  One CTA per row; the updated row stays in
// registers between the two passes when it fits (D <= 256 * 8), else it is re-read.
template <typename act_t>
__global__ void __launch_bounds__(256) seq_norm_add_norm_kernel(const act_t* __restrict__ y, const act_t* __restrict__ wp, float eps, float mult,
                                                                float* __restrict__ x, const act_t* __restrict__ wn,
                                                                act_t* __restrict__ h, int D) {
  __shared__ float red[32];
  const act_t* yr = y + (size_t)blockIdx.x * D;
  float* xr = x + (size_t)blockIdx.x * D;
  float ss = 0.f;
  for (int i = threadIdx.x; i < D; i += blockDim.x) {
    const float v = ld_act(yr, i);
    ss += v * v;
  }
  ss = block_sum(ss, red);
  const float rinv = mult / sqrtf(ss / (float)D + eps);
  float s2 = 0.f;
  for (int i = threadIdx.x; i < D; i += blockDim.x) {
    const float v = xr[i] + ld_act(yr, i) * rinv * ld_act(wp, i);
    xr[i] = v;
    s2 += v * v;
    if (h && wn == nullptr) st_act(h, (size_t)blockIdx.x * D + i, v);
  }
  if (wn == nullptr) return;
  s2 = block_sum(s2, red);
  const float r2 = 1.0f / sqrtf(s2 / (float)D + eps);
  act_t* hr = h + (size_t)blockIdx.x * D;
  for (int i = threadIdx.x; i < D; i += blockDim.x) st_act(hr, i, xr[i] * r2 * ld_act(wn, i));   // own writes: visible to this thread
}

// The same with the row held in registers (D <= 256 * EPT): every operand is requested before the first reduction, so
// a single-token step pays one memory latency instead of three.
template <typename act_t, int EPT>
__global__ void __launch_bounds__(256) seq_norm_add_norm_reg_kernel(const act_t* __restrict__ y, const act_t* __restrict__ wp, float eps, float mult,
                                                                    float* __restrict__ x, const act_t* __restrict__ wn,
                                                                    act_t* __restrict__ h, int D) {
  __shared__ float red[32];
  const act_t* yr = y + (size_t)blockIdx.x * D;
  float* xr = x + (size_t)blockIdx.x * D;
  float yv[EPT], xv[EPT], pv[EPT], nv[EPT];
#pragma unroll
  for (int e = 0; e < EPT; ++e) {
    const int i = threadIdx.x + e * 256;
    const bool in = i < D;
    yv[e] = in ? ld_act(yr, i) : 0.f;
    xv[e] = in ? xr[i] : 0.f;
    pv[e] = in ? ld_act(wp, i) : 0.f;
    nv[e] = (in && wn) ? ld_act(wn, i) : 0.f;
  }
  float ss = 0.f;
#pragma unroll
  for (int e = 0; e < EPT; ++e) ss += yv[e] * yv[e];
  ss = block_sum(ss, red);
  const float rinv = mult / sqrtf(ss / (float)D + eps);
  float s2 = 0.f;
#pragma unroll
  for (int e = 0; e < EPT; ++e) {
    const int i = threadIdx.x + e * 256;
    xv[e] += yv[e] * rinv * pv[e];
    if (i < D) {
      xr[i] = xv[e];
      if (h && wn == nullptr) st_act(h, (size_t)blockIdx.x * D + i, xv[e]);
    }
    s2 += xv[e] * xv[e];
  }
  if (wn == nullptr) return;
  s2 = block_sum(s2, red);
  const float r2 = 1.0f / sqrtf(s2 / (float)D + eps);
  act_t* hr = h + (size_t)blockIdx.x * D;
#pragma unroll
  for (int e = 0; e < EPT; ++e) {
    const int i = threadIdx.x + e * 256;
    if (i < D) st_act(hr, i, xv[e] * r2 * nv[e]);
  }
}

// The same by fours of elements (D a multiple of 4, aligned rows; D <= 1024 * EPV).  Loads and stores of one element bound the form above: a warp asked for
// 64 or 128 bytes at a time, 16 requests a thread and operand at 4096.  Measured on bf16 rows (us, above / this): one row of 1024 2.1 / 1.9, of 4096 5.0 / 2.4;
// 777 rows of 1024 4.0 / 3.2, of 2048 5.7 / 4.4, of 4096 13.7 / 7.0; 2048 rows of 4096 31 / 15.  The form above keeps the rows that have no such boundary.
template <typename act_t, int EPV>
__global__ void __launch_bounds__(256) seq_norm_add_norm_vec_kernel(const act_t* __restrict__ y, const act_t* __restrict__ wp, float eps, float mult,
                                                                    float* __restrict__ x, const act_t* __restrict__ wn,
                                                                    act_t* __restrict__ h, int D) {
  __shared__ float red[32];
  const act_t* yr = y + (size_t)blockIdx.x * D;
  float* xr = x + (size_t)blockIdx.x * D;
  act_t* hr = h + (size_t)blockIdx.x * D;
  const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 yv[EPV], xv[EPV], pv[EPV], nv[EPV];
#pragma unroll
  for (int e = 0; e < EPV; ++e) {
    const int i = (threadIdx.x + e * 256) * 4;
    const bool in = i < D;
    yv[e] = in ? ld_act4(yr + i) : none;
    xv[e] = in ? ld_act4(xr + i) : none;
    pv[e] = in ? ld_act4(wp + i) : none;
    nv[e] = in && wn ? ld_act4(wn + i) : none;
  }
  float ss = 0.f;
#pragma unroll
  for (int e = 0; e < EPV; ++e) ss += yv[e].x * yv[e].x + yv[e].y * yv[e].y + yv[e].z * yv[e].z + yv[e].w * yv[e].w;
  ss = block_sum(ss, red);
  const float rinv = mult / sqrtf(ss / (float)D + eps);
  float s2 = 0.f;
#pragma unroll
  for (int e = 0; e < EPV; ++e) {
    const int i = (threadIdx.x + e * 256) * 4;
    xv[e].x += yv[e].x * rinv * pv[e].x;
    xv[e].y += yv[e].y * rinv * pv[e].y;
    xv[e].z += yv[e].z * rinv * pv[e].z;
    xv[e].w += yv[e].w * rinv * pv[e].w;
    if (i < D) {
      st_act4(xr + i, xv[e]);
      if (h && wn == nullptr) st_act4(hr + i, xv[e]);
    }
    s2 += xv[e].x * xv[e].x + xv[e].y * xv[e].y + xv[e].z * xv[e].z + xv[e].w * xv[e].w;
  }
  if (wn == nullptr) return;
  s2 = block_sum(s2, red);
  const float r2 = 1.0f / sqrtf(s2 / (float)D + eps);
#pragma unroll
  for (int e = 0; e < EPV; ++e) {
    const int i = (threadIdx.x + e * 256) * 4;
    if (i < D) st_act4(hr + i, make_float4(xv[e].x * r2 * nv[e].x, xv[e].y * r2 * nv[e].y, xv[e].z * r2 * nv[e].z, xv[e].w * r2 * nv[e].w));
  }
}

// Moved to seq_common.cuh: gated_pair(a, b, act, limit) = act(a) * b, or the clamped unit.

// 16-byte form (F and ldgu multiples of 8 elements, aligned pointers): eight bf16 or four f32 numbers per load.
template <typename act_t>
__global__ void seq_gated_act_vec_kernel(const act_t* __restrict__ gu, int ldgu, act_t* __restrict__ out, int F, int act, float limit) {
  constexpr int PER = 16 / sizeof(act_t);
  const act_t* g = gu + (size_t)blockIdx.x * ldgu;
  act_t* o = out + (size_t)blockIdx.x * F;
  for (int j = (blockIdx.y * blockDim.x + threadIdx.x) * PER; j < F; j += gridDim.y * blockDim.x * PER) {
    const uint4 a4 = *reinterpret_cast<const uint4*>(g + j), b4 = *reinterpret_cast<const uint4*>(g + F + j);
    uint4 r4;
    if (sizeof(act_t) == 2) {
      const uint32_t aw[4] = {a4.x, a4.y, a4.z, a4.w}, bw[4] = {b4.x, b4.y, b4.z, b4.w};
      uint32_t rw[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float lo = gated_pair(__uint_as_float(aw[q] << 16), __uint_as_float(bw[q] << 16), act, limit);
        const float hi = gated_pair(__uint_as_float(aw[q] & 0xffff0000u), __uint_as_float(bw[q] & 0xffff0000u), act, limit);
        const __nv_bfloat162 t = __floats2bfloat162_rn(lo, hi);
        rw[q] = *reinterpret_cast<const uint32_t*>(&t);
      }
      r4 = make_uint4(rw[0], rw[1], rw[2], rw[3]);
    } else {
      r4.x = __float_as_uint(gated_pair(__uint_as_float(a4.x), __uint_as_float(b4.x), act, limit));
      r4.y = __float_as_uint(gated_pair(__uint_as_float(a4.y), __uint_as_float(b4.y), act, limit));
      r4.z = __float_as_uint(gated_pair(__uint_as_float(a4.z), __uint_as_float(b4.z), act, limit));
      r4.w = __float_as_uint(gated_pair(__uint_as_float(a4.w), __uint_as_float(b4.w), act, limit));
    }
    *reinterpret_cast<uint4*>(o + j) = r4;
  }
}

template <typename act_t>
__global__ void seq_gated_act_kernel(const act_t* __restrict__ gu, int ldgu, act_t* __restrict__ out, int F, int act, float limit) {
  const act_t* g = gu + (size_t)blockIdx.x * ldgu;
  act_t* o = out + (size_t)blockIdx.x * F;
  for (int j = blockIdx.y * blockDim.x + threadIdx.x; j < F; j += gridDim.y * blockDim.x) {
    const float a = ld_act(g, j), b = ld_act(g, (size_t)F + j);
    st_act(o, j, gated_pair(a, b, act, limit));
  }
}

// Causal convolution + silu.  Thread = one channel over a tile of CONV_TT tokens with a sliding window in registers.
// Tile 0 reads the carried inputs, and the thread that has read a channel's advances them: to its last inputs, or, where
// the portion has several tiles (and so more tokens than taps), to the portion's (no second launch: 2.5 us of a portion).
constexpr int CONV_TT = 32;
constexpr int CONV_MAX_TAPS = 8;
template <typename act_t>
__global__ void seq_conv_silu_kernel(const act_t* __restrict__ in, int ldin, const act_t* __restrict__ w,
                                     const act_t* __restrict__ bias, act_t* state, const int* __restrict__ meta,
                                     float* __restrict__ out, int ldout, int T, int C, int taps) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  const int t0 = blockIdx.y * CONV_TT, t1 = min(T, t0 + CONV_TT);
  act_t* st = state + (size_t)meta[0] * (taps - 1) * C;
  float wr[CONV_MAX_TAPS], win[CONV_MAX_TAPS];   // win[j] = input at t - (taps-1) + j
#pragma unroll
  for (int j = 0; j < CONV_MAX_TAPS; ++j) wr[j] = j < taps ? ld_act(w, (size_t)c * taps + j) : 0.f;
  const float b = bias ? ld_act(bias, c) : 0.f;
#pragma unroll
  for (int j = 0; j < CONV_MAX_TAPS; ++j) {
    win[j] = 0.f;
    if (j < taps - 1) {
      const int t = t0 - (taps - 1) + j;   // input index relative to the portion
      win[j] = t >= 0 ? ld_act(in, (size_t)t * ldin + c) : ld_act(st, (size_t)(taps - 1 + t) * C + c);
    }
  }
  for (int t = t0; t < t1; ++t) {
    const float cur = ld_act(in, (size_t)t * ldin + c);
    float acc = b;
#pragma unroll
    for (int j = 0; j < CONV_MAX_TAPS; ++j) {
      if (j < taps - 1) acc += wr[j] * win[j];
    }
#pragma unroll
    for (int j = 0; j < CONV_MAX_TAPS; ++j) {
      if (j == taps - 1) acc += wr[j] * cur;
    }
    out[(size_t)t * ldout + c] = silu_f(acc);
#pragma unroll
    for (int j = 0; j < CONV_MAX_TAPS - 1; ++j) {
      if (j < taps - 2) win[j] = win[j + 1];
    }
#pragma unroll
    for (int j = 0; j < CONV_MAX_TAPS; ++j) {
      if (j == taps - 2) win[j] = cur;
    }
  }
  if (blockIdx.y == 0) {   // single tile: win[] now holds the last taps-1 inputs of the sequence
#pragma unroll
    for (int j = 0; j < CONV_MAX_TAPS; ++j) {
      if (j < taps - 1) st_act(st, (size_t)j * C + c, gridDim.y == 1 ? win[j] : ld_act(in, (size_t)(T - (taps - 1) + j) * ldin + c));
    }
  }
}

// Four taps over long portions in bf16: a thread owns V neighbouring channels and CONV_VT tokens, so the bytes in flight suffice for HBM.  Four
// channels (8-byte loads, one 16-byte store, 64 registers) keep twice the warps of eight on an SM: 6144 channels x 2048 tokens with the unit
// heads 26.5 us against 30.3 (73 one channel at a time, 35 with eight channels and 16 tokens).  Eight only where a head of more than 128
// channels is to lie in one warp.  Sums in the order of the kernel above.
// Portions that give the SMs fewer than eight CTAs of eight tokens go by four tokens a thread: their time is a thread's chain of loads and gates.
// A thread takes four tokens at once, the next four requested before: each token by itself waited for its load, its gates and, with unit heads, five
// exchanges, a root and a quotient in every lane; for four tokens together a lane adds up one token's squares and takes its root alone.  us, token by token /
// by fours, unit heads of 128, calls back to back on inputs that the L2 holds: 6144 channels x 2048 tokens 27.1 / 24.9, 3072 x 512 8.5 / 6.6; each call by itself on inputs
// from memory 37.8 / 33.8, 13.3 / 11.2, 3072 x 9 11.3 / 9.6; in the delta layer of 2048 tokens the kernel takes 26.  Without heads 3072 x 9 3.7 / 3.2, but
// 6144 x 2048 19.2 / 19.9 (80 registers), so those go token by token, as do heads of fewer than four lanes.
constexpr int CONV_VT = 8, CONV_VT_FEW = 4;
__device__ __forceinline__ void ld8_bf16(const __nv_bfloat16* p, float (&x)[8]) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    x[2 * i] = __uint_as_float(w[i] << 16);
    x[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
// UNIT: the heads of `size` channels at a0 .. and at b0 .. become unit vectors times ma or mb on the way (size / V neighbouring lanes hold a head).
struct UnitHeads { int a0, a1, b0, b1, size; float eps, ma, mb; };
template <int V> __device__ __forceinline__ void ldv_bf16(const __nv_bfloat16* p, float (&x)[V]) {
  if constexpr (V == 8) {
    ld8_bf16(p, x);
  } else {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    x[0] = __uint_as_float(u.x << 16); x[1] = __uint_as_float(u.x & 0xffff0000u);
    x[2] = __uint_as_float(u.y << 16); x[3] = __uint_as_float(u.y & 0xffff0000u);
  }
}
template <bool UNIT, int V, int VT>
__global__ void __launch_bounds__(128) seq_conv4_silu_kernel(const __nv_bfloat16* __restrict__ in, int ldin, const __nv_bfloat16* __restrict__ w,
                                                            const __nv_bfloat16* __restrict__ bias, __nv_bfloat16* state,
                                                            const int* __restrict__ meta, float* __restrict__ out, int ldout, int T, int C, UnitHeads u) {
  const int c0 = (blockIdx.x * 128 + threadIdx.x) * V, c = min(c0, C - V);      // lanes past the last channel repeat it
  const float mult = !UNIT ? 0.f : c >= u.a0 && c < u.a1 ? u.ma : c >= u.b0 && c < u.b1 ? u.mb : 0.f;
  const bool any = UNIT && __any_sync(0xffffffffu, mult != 0.f);
  static_assert(VT >= 3, "only the first tile may read the carried inputs, which it overwrites");
  const int t0 = blockIdx.y * VT, nt = min(VT, T - t0);
  __nv_bfloat16* st = state + (size_t)meta[0] * 3 * C;
  float wr[4][V], win[3][V], b[V];
#pragma unroll
  for (int i = 0; i < V / 2; ++i) {                         // w is [channel][tap]
    float x[8];
    ld8_bf16(w + (size_t)c * 4 + 8 * i, x);
#pragma unroll
    for (int e = 0; e < 8; ++e) wr[e & 3][2 * i + (e >> 2)] = x[e];
  }
#pragma unroll
  for (int e = 0; e < V; ++e) b[e] = 0.f;
  if (bias) {
#pragma unroll
    for (int e = 0; e < V; ++e) b[e] = __bfloat162float(bias[c + e]);
  }
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const int t = t0 - 3 + j;
    if (t >= 0 || c0 < C) ldv_bf16<V>(t >= 0 ? in + (size_t)t * ldin + c : st + (size_t)(3 + t) * C + c, win[j]);
    else                                                    // a lane that repeats the last channels stays off what their own lane writes below
#pragma unroll
      for (int e = 0; e < V; ++e) win[j][e] = 0.f;
  }
  if (blockIdx.y == 0 && c0 < C) {                          // the thread that has read the carried inputs of its channels leaves the portion's last ones
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      using Word = std::conditional_t<V == 8, uint4, uint2>;
      const int t = T - 3 + j;                              // of fewer than three tokens: a carried input, row j is written after row T + j is read
      *reinterpret_cast<Word*>(st + (size_t)j * C + c) = *reinterpret_cast<const Word*>(t >= 0 ? in + (size_t)t * ldin + c : st + (size_t)(T + j) * C + c);
    }
  }
  if (UNIT ? u.size < 4 * V : VT == CONV_VT) {               // token by token: heads of one or two lanes, and long portions without heads
#pragma unroll 4
    for (int r = 0; r < nt; ++r) {
      float cur[V], y[V];
      ldv_bf16<V>(in + (size_t)(t0 + r) * ldin + c, cur);
#pragma unroll
      for (int e = 0; e < V; ++e) {
        float acc = b[e];
        acc += wr[0][e] * win[0][e];
        acc += wr[1][e] * win[1][e];
        acc += wr[2][e] * win[2][e];
        acc += wr[3][e] * cur[e];
        y[e] = silu_f(acc);
        win[0][e] = win[1][e];
        win[1][e] = win[2][e];
        win[2][e] = cur[e];
      }
      if (any) {
        float ss = 0.f;
#pragma unroll
        for (int e = 0; e < V; ++e) ss += y[e] * y[e];
        if (u.size > V) ss += __shfl_xor_sync(0xffffffffu, ss, 1);
        const float f = mult != 0.f ? mult / sqrtf(ss + u.eps) : 1.f;
#pragma unroll
        for (int e = 0; e < V; ++e) y[e] *= f;
      }
      float4* o = reinterpret_cast<float4*>(out + (size_t)(t0 + r) * ldout + c);
      if (c0 >= C) continue;
      o[0] = make_float4(y[0], y[1], y[2], y[3]);
      if constexpr (V == 8) o[1] = make_float4(y[4], y[5], y[6], y[7]);
    }
    return;
  }
  // four tokens at a time, the next four on their way meanwhile
  using Word = std::conditional_t<V == 8, uint4, uint2>;
  const __nv_bfloat16* row = in + (size_t)t0 * ldin + c;
  float* o = out + (size_t)t0 * ldout + c;
  Word raw[4];
  auto fetch = [&](int from) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
      raw[r] = from + r < nt ? *reinterpret_cast<const Word*>(row + (size_t)(from + r) * ldin) : Word{};
  };
  fetch(0);
#pragma unroll 1
  for (int r0 = 0; r0 < nt; r0 += 4) {
    float cur[4][V], y[4][V] = {};
#pragma unroll
    for (int r = 0; r < 4; ++r) ldv_bf16<V>(reinterpret_cast<const __nv_bfloat16*>(&raw[r]), cur[r]);
    fetch(r0 + 4);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      if (VT == CONV_VT_FEW && (r == 1 || r == 2) && nt == r) break;
#pragma unroll
      for (int e = 0; e < V; ++e) {
        float acc = b[e];
#pragma unroll
        for (int j = 0; j < 4; ++j) acc += wr[j][e] * (r + j < 3 ? win[r + j][e] : cur[r + j - 3][e]);
        y[r][e] = silu_f(acc);
      }
    }
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int e = 0; e < V; ++e) win[j][e] = cur[1 + j][e];
    if (any) {
      float ss[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        ss[r] = 0.f;
#pragma unroll
        for (int e = 0; e < V; ++e) ss[r] += y[r][e] * y[r][e];
      }
      float f[4];
      // a lane adds up one token's squares, and takes its root
      const bool odd = threadIdx.x & 1, high = threadIdx.x & 2;
#pragma unroll
      for (int r = 0; r < 2; ++r) ss[r] = (odd ? ss[r + 2] : ss[r]) + __shfl_xor_sync(0xffffffffu, odd ? ss[r] : ss[r + 2], 1);
      float all = (high ? ss[1] : ss[0]) + __shfl_xor_sync(0xffffffffu, high ? ss[0] : ss[1], 2);
      for (int d = 4; d < u.size / V; d <<= 1) all += __shfl_xor_sync(0xffffffffu, all, d);
      all = mult != 0.f ? mult / sqrtf(all + u.eps) : 1.f;
#pragma unroll
      for (int r = 0; r < 4; ++r) f[r] = __shfl_sync(0xffffffffu, all, (r >> 1) | (r & 1) << 1, 4);
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int e = 0; e < V; ++e) y[r][e] *= f[r];
    }
    if (c0 < C) {
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if (r0 + r < nt) {
          float4* q = reinterpret_cast<float4*>(o + (size_t)(r0 + r) * ldout);
          q[0] = make_float4(y[r][0], y[r][1], y[r][2], y[r][3]);
          if constexpr (V == 8) q[1] = make_float4(y[r][4], y[r][5], y[r][6], y[r][7]);
        }
    }
  }
}

template <typename act_t>
__global__ void seq_cast_f32_kernel(const act_t* __restrict__ in, int ldin, float* __restrict__ out, int ldout, int n) {
  const act_t* p = in + (size_t)blockIdx.x * ldin;
  float* q = out + (size_t)blockIdx.x * ldout;
  for (int j = blockIdx.y * blockDim.x + threadIdx.x; j < n; j += gridDim.y * blockDim.x) q[j] = ld_act(p, j);
}

// The same by fours of elements (n and both strides multiples of 4, aligned rows).  Measured (us, above / this): few rows the same; 777 rows of 1024 2.8 / 1.9,
// 2048 rows of 2048 9.7 / 3.9.
template <typename act_t>
__global__ void seq_cast_f32_vec_kernel(const act_t* __restrict__ in, int ldin, float* __restrict__ out, int ldout, int n) {
  const act_t* p = in + (size_t)blockIdx.x * ldin;
  float* q = out + (size_t)blockIdx.x * ldout;
  for (int j = (blockIdx.y * blockDim.x + threadIdx.x) * 4; j < n; j += gridDim.y * blockDim.x * 4) st_act4(q + j, ld_act4(p + j));
}

// One warp per (token, head): x * mult / sqrt(sum x^2 + eps), in place.
__global__ void seq_unit_norm_kernel(float* __restrict__ x, int ld, int n_groups, int heads, int size, float eps, float mult) {
  const int g = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (g >= n_groups) return;
  float* p = x + (size_t)(g / heads) * ld + (size_t)(g % heads) * size;
  float ss = 0.f;
  for (int i = lane; i < size; i += 32) ss += p[i] * p[i];
  ss = warp_sum(ss);
  const float r = mult / sqrtf(ss + eps);
  for (int i = lane; i < size; i += 32) p[i] *= r;
}

template <typename act_t>
__global__ void seq_decay_kernel(const act_t* __restrict__ a, int lda, const act_t* __restrict__ bias,
                                 const act_t* __restrict__ A_log, int mode, float inv_tau, float* __restrict__ out,
                                 float* __restrict__ dt_out, int heads, int size) {
  const int n = heads * size;
  const act_t* ar = a + (size_t)blockIdx.x * lda;
  for (int j = blockIdx.y * blockDim.x + threadIdx.x; j < n; j += gridDim.y * blockDim.x) {
    const float z = ld_act(ar, j) + (bias ? ld_act(bias, j) : 0.f);
    float r;
    if (mode == B2L_SEQ_DECAY_EXP_SOFTPLUS) {
      const float dt = softplus_f(z);
      if (dt_out) dt_out[(size_t)blockIdx.x * n + j] = dt;
      r = expf(-expf(ld_act(A_log, j / size)) * dt);
    } else {
      // sigmoid(z)^(1/tau) = exp(-softplus(-z) / tau): no underflow of the sigmoid for very negative z
      r = expf(-softplus_f(-z) * inv_tau);
    }
    out[(size_t)blockIdx.x * n + j] = r;
  }
}

// The same for bf16 layers whose heads are whole groups of 8 channels: a thread owns 8 channels (one 16-byte load, two stores), so a head's coefficient is
// formed once for them (2048 channels x 2048 tokens: 23 us one channel at a time, now 9.6; 24 MB move).
__device__ __forceinline__ void ld8_bf16(const __nv_bfloat16* p, float (&x)[8]);
__global__ void __launch_bounds__(256) seq_decay8_kernel(const __nv_bfloat16* __restrict__ a, int lda, const __nv_bfloat16* __restrict__ bias,
                                                        const __nv_bfloat16* __restrict__ A_log, int mode, float inv_tau, float* __restrict__ out,
                                                        float* __restrict__ dt_out, int n, int size) {
  const int j = 8 * (blockIdx.y * blockDim.x + threadIdx.x);
  if (j >= n) return;
  float z[8], b[8] = {}, r[8], dt[8];
  ld8_bf16(a + (size_t)blockIdx.x * lda + j, z);
  if (bias) ld8_bf16(bias + j, b);
  const float coef = mode == B2L_SEQ_DECAY_EXP_SOFTPLUS ? -expf(__bfloat162float(A_log[j / size])) : 0.f;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    z[e] += b[e];
    dt[e] = softplus_f(mode == B2L_SEQ_DECAY_EXP_SOFTPLUS ? z[e] : -z[e]);
    r[e] = expf(mode == B2L_SEQ_DECAY_EXP_SOFTPLUS ? coef * dt[e] : -dt[e] * inv_tau);
  }
  float4* o = reinterpret_cast<float4*>(out + (size_t)blockIdx.x * n + j);
  o[0] = make_float4(r[0], r[1], r[2], r[3]);
  o[1] = make_float4(r[4], r[5], r[6], r[7]);
  if (dt_out && mode == B2L_SEQ_DECAY_EXP_SOFTPLUS) {
    float4* d = reinterpret_cast<float4*>(dt_out + (size_t)blockIdx.x * n + j);
    d[0] = make_float4(dt[0], dt[1], dt[2], dt[3]);
    d[1] = make_float4(dt[4], dt[5], dt[6], dt[7]);
  }
}

// One warp per (token, group).
template <typename act_t>
__global__ void seq_group_norm_gate_kernel(const float* __restrict__ o, int ldo, const act_t* __restrict__ w, int w_shared,
                                           const act_t* __restrict__ gate, int ldg, int gate_act, int gate_first, float eps,
                                           float out_mult, act_t* __restrict__ out, int ldout, int n_rows, int groups, int group) {
  const int id = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (id >= n_rows * groups) return;
  const int t = id / groups, g = id % groups;
  const float* p = o + (size_t)t * ldo + (size_t)g * group;
  const act_t* gp = gate ? gate + (size_t)t * ldg + (size_t)g * group : nullptr;
  auto gate_of = [&](int i) {
    const float z = ld_act(gp, i);
    return gate_act == B2L_SEQ_ACT_SILU ? silu_f(z) : (gate_act == B2L_SEQ_ACT_SIGMOID ? sigmoid_f(z) : gelu_tanh_f(z));
  };
  float ss = 0.f;
  for (int i = lane; i < group; i += 32) {
    float v = p[i];
    if (gp && gate_first) v *= gate_of(i);
    ss += v * v;
  }
  ss = warp_sum(ss);
  const float r = out_mult / sqrtf(ss / (float)group + eps);
  act_t* q = out + (size_t)t * ldout + (size_t)g * group;
  for (int i = lane; i < group; i += 32) {
    float v = p[i];
    if (gp && gate_first) v *= gate_of(i);
    v = v * r * ld_act(w, w_shared ? i : g * group + i);
    if (gp && !gate_first) v *= gate_of(i);
    st_act(q, i, v);
  }
}

// The same for bf16 groups of 32 PER channels: a lane owns PER neighbouring ones and keeps them in registers (2048 tokens of 16 groups of 128: 16 us
// with two-byte accesses, now 10; 32 MB move).
template <int PER>
__global__ void __launch_bounds__(128) seq_group_norm_gate_vec_kernel(const float* __restrict__ o, int ldo, const __nv_bfloat16* __restrict__ w, int w_shared,
                                                                     const __nv_bfloat16* __restrict__ gate, int ldg, int gate_act, int gate_first, float eps,
                                                                     float out_mult, __nv_bfloat16* __restrict__ out, int ldout, int n_rows, int groups) {
  const int id = blockIdx.x * 4 + (threadIdx.x >> 5), c = (threadIdx.x & 31) * PER;
  if (id >= n_rows * groups) return;
  const int t = id / groups, at = (id - t * groups) * (32 * PER) + c;
  struct alignas(2 * PER) Row { __nv_bfloat16 e[PER]; };
  float v[PER], g[PER];
#pragma unroll
  for (int i = 0; i < PER; i += 4) *reinterpret_cast<float4*>(&v[i]) = *reinterpret_cast<const float4*>(o + (size_t)t * ldo + at + i);
  const Row wr = *reinterpret_cast<const Row*>(w + (w_shared ? c : at));
  if (gate) {
    const Row gr = *reinterpret_cast<const Row*>(gate + (size_t)t * ldg + at);
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const float z = __bfloat162float(gr.e[i]);
      g[i] = gate_act == B2L_SEQ_ACT_SILU ? silu_f(z) : (gate_act == B2L_SEQ_ACT_SIGMOID ? sigmoid_f(z) : gelu_tanh_f(z));
      if (gate_first) v[i] *= g[i];
    }
  }
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < PER; ++i) ss += v[i] * v[i];
  const float r = out_mult / sqrtf(warp_sum(ss) / (float)(32 * PER) + eps);
  Row y;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    float x = v[i] * r * __bfloat162float(wr.e[i]);
    if (gate && !gate_first) x *= g[i];
    y.e[i] = __float2bfloat16_rn(x);
  }
  *reinterpret_cast<Row*>(out + (size_t)t * ldout + at) = y;
}

// The same with four neighbouring groups a warp: their loads together, and a lane adds up one group's squares and takes its root alone.
// Groups of 128 from 56 an SM on: 2048 tokens of 16, sigmoid gates, 8.7 us above and 6.9 so (32 MB move), of 32 with silu 16.9 / 12.3, 777 of 16 4.3 / 4.0, 512 of 16
// 3.4 / 3.3; 300 of 16 2.7 / 3.0, one token 1.6 / 2.3.  Groups of 256 take 110 registers so and 2048 tokens 16.6 us for 13.5.
template <int PER>
__global__ void __launch_bounds__(128) seq_group_norm_gate_fours_kernel(const float* __restrict__ o, int ldo, const __nv_bfloat16* __restrict__ w, int w_shared,
                                                                       const __nv_bfloat16* __restrict__ gate, int ldg, int gate_act, int gate_first, float eps,
                                                                       float out_mult, __nv_bfloat16* __restrict__ out, int ldout, int n_rows, int groups) {
  const int id = (blockIdx.x * 4 + (threadIdx.x >> 5)) * 4, lane = threadIdx.x & 31, c = lane * PER, t = id / groups;      // groups a multiple of four: of one token
  if (t >= n_rows) return;
  const int at = (id - t * groups) * (32 * PER) + c;
  struct alignas(2 * PER) Row { __nv_bfloat16 e[PER]; };
  float v[4][PER];
  Row gr[4], wr[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
#pragma unroll
    for (int i = 0; i < PER; i += 4) *reinterpret_cast<float4*>(&v[k][i]) = *reinterpret_cast<const float4*>(o + (size_t)t * ldo + at + k * (32 * PER) + i);
    if (gate) gr[k] = *reinterpret_cast<const Row*>(gate + (size_t)t * ldg + at + k * (32 * PER));
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) wr[k] = *reinterpret_cast<const Row*>(w + (w_shared ? c : at + k * (32 * PER)));
  float g[4][PER], ss[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    ss[k] = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      if (gate) {
        const float z = __bfloat162float(gr[k].e[i]);
        g[k][i] = gate_act == B2L_SEQ_ACT_SILU ? silu_f(z) : (gate_act == B2L_SEQ_ACT_SIGMOID ? sigmoid_f(z) : gelu_tanh_f(z));
        if (gate_first) v[k][i] *= g[k][i];
      }
      ss[k] += v[k][i] * v[k][i];
    }
  }
  const bool odd = lane & 1, high = lane & 2;
#pragma unroll
  for (int k = 0; k < 2; ++k) ss[k] = (odd ? ss[k + 2] : ss[k]) + __shfl_xor_sync(0xffffffffu, odd ? ss[k] : ss[k + 2], 1);
  float all = (high ? ss[1] : ss[0]) + __shfl_xor_sync(0xffffffffu, high ? ss[0] : ss[1], 2);
#pragma unroll
  for (int d = 4; d < 32; d <<= 1) all += __shfl_xor_sync(0xffffffffu, all, d);
  all = out_mult / sqrtf(all / (float)(32 * PER) + eps);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float r = __shfl_sync(0xffffffffu, all, (k >> 1) | (k & 1) << 1, 4);
    Row y;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      float x = v[k][i] * r * __bfloat162float(wr[k].e[i]);
      if (gate && !gate_first) x *= g[k][i];
      y.e[i] = __float2bfloat16_rn(x);
    }
    *reinterpret_cast<Row*>(out + (size_t)t * ldout + at + k * (32 * PER)) = y;
  }
}

// The same for large groups (a whole layer's channels normalised together): one CTA per (token, group).
template <typename act_t>
__global__ void __launch_bounds__(256) seq_group_norm_gate_block_kernel(const float* __restrict__ o, int ldo, const act_t* __restrict__ w, int w_shared,
                                                                        const act_t* __restrict__ gate, int ldg, int gate_act, int gate_first,
                                                                        float eps, float out_mult, act_t* __restrict__ out, int ldout, int groups,
                                                                        int group) {
  __shared__ float red[32];
  const int t = blockIdx.x / groups, g = blockIdx.x % groups;
  const float* p = o + (size_t)t * ldo + (size_t)g * group;
  const act_t* gp = gate ? gate + (size_t)t * ldg + (size_t)g * group : nullptr;
  auto gate_of = [&](int i) {
    const float z = ld_act(gp, i);
    return gate_act == B2L_SEQ_ACT_SILU ? silu_f(z) : (gate_act == B2L_SEQ_ACT_SIGMOID ? sigmoid_f(z) : gelu_tanh_f(z));
  };
  float ss = 0.f;
  for (int i = threadIdx.x; i < group; i += blockDim.x) {
    float v = p[i];
    if (gp && gate_first) v *= gate_of(i);
    ss += v * v;
  }
  ss = block_sum(ss, red);
  const float r = out_mult / sqrtf(ss / (float)group + eps);
  act_t* q = out + (size_t)t * ldout + (size_t)g * group;
  for (int i = threadIdx.x; i < group; i += blockDim.x) {
    float v = p[i];
    if (gp && gate_first) v *= gate_of(i);
    v = v * r * ld_act(w, w_shared ? i : g * group + i);
    if (gp && !gate_first) v *= gate_of(i);
    st_act(q, i, v);
  }
}

// The same in bf16 where every row starts on 16 bytes: eight neighbouring channels a thread and step, NV steps kept in registers, so each gate is taken once and
// nothing is read twice (512 tokens of 2048 channels with silu gates, device time 11.5 -> 5.6 us; their 8 MB take 1.3).
template <int NV>
__global__ void __launch_bounds__(256) seq_group_norm_gate_wide_kernel(const float* __restrict__ o, int ldo, const __nv_bfloat16* __restrict__ w, int w_shared,
                                                                       const __nv_bfloat16* __restrict__ gate, int ldg, int gate_act, int gate_first, float eps,
                                                                       float out_mult, __nv_bfloat16* __restrict__ out, int ldout, int groups, int group) {
  __shared__ float red[32];
  const int t = blockIdx.x / groups, g = blockIdx.x % groups;
  const size_t at = (size_t)g * group;
  float v[NV][8], z[NV][8], ss = 0.f;
#pragma unroll
  for (int c = 0; c < NV; ++c) {
    const int i = (c * 256 + threadIdx.x) * 8;
    if (i >= group) continue;
    const float4 a = *reinterpret_cast<const float4*>(o + (size_t)t * ldo + at + i), b = *reinterpret_cast<const float4*>(o + (size_t)t * ldo + at + i + 4);
    v[c][0] = a.x; v[c][1] = a.y; v[c][2] = a.z; v[c][3] = a.w; v[c][4] = b.x; v[c][5] = b.y; v[c][6] = b.z; v[c][7] = b.w;
    if (gate) {
      ld8_bf16(gate + (size_t)t * ldg + at + i, z[c]);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        z[c][e] = gate_act == B2L_SEQ_ACT_SILU ? silu_f(z[c][e]) : gate_act == B2L_SEQ_ACT_SIGMOID ? sigmoid_f(z[c][e]) : gelu_tanh_f(z[c][e]);
        if (gate_first) v[c][e] *= z[c][e];
      }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) ss += v[c][e] * v[c][e];
  }
  ss = block_sum(ss, red);
  const float r = out_mult / sqrtf(ss / (float)group + eps);
#pragma unroll
  for (int c = 0; c < NV; ++c) {
    const int i = (c * 256 + threadIdx.x) * 8;
    if (i >= group) continue;
    float x[8];
    ld8_bf16(w + (w_shared ? 0 : at) + i, x);
    __nv_bfloat162 y[4];
#pragma unroll
    for (int e = 0; e < 8; e += 2) {
      float p[2] = {v[c][e] * r * x[e], v[c][e + 1] * r * x[e + 1]};
      if (gate && !gate_first) { p[0] *= z[c][e]; p[1] *= z[c][e + 1]; }
      y[e / 2] = __floats2bfloat162_rn(p[0], p[1]);
    }
    *reinterpret_cast<uint4*>(out + (size_t)t * ldout + at + i) = *reinterpret_cast<const uint4*>(y);
  }
}

// Per-head RMS norm + partial rotation.  One warp per (token, head).
template <typename act_t, typename out_t>
__global__ void seq_headnorm_rope_kernel(const act_t* __restrict__ x, int ldx, const act_t* __restrict__ w, float eps,
                                         const float* __restrict__ freq, int rot_dims, float rot_mult,
                                         const int* __restrict__ meta, out_t* __restrict__ out, int n_rows, int heads, int size) {
  const int id = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (id >= n_rows * heads) return;
  const int t = id / heads, hd = id % heads;
  const act_t* p = x + (size_t)t * ldx + (size_t)hd * size;
  out_t* q = out + ((size_t)t * heads + hd) * size;
  float r = 1.f;
  if (w) {
    float ss = 0.f;
    for (int i = lane; i < size; i += 32) {
      const float v = ld_act(p, i);
      ss += v * v;
    }
    ss = warp_sum(ss);
    r = 1.0f / sqrtf(ss / (float)size + eps);
  }
  const float pos = (float)(meta[1] + t);
  const int half = rot_dims / 2;
  for (int i = lane; i < half; i += 32) {
    const float u = ld_act(p, i) * r * (w ? ld_act(w, i) : 1.f);
    const float v = ld_act(p, i + half) * r * (w ? ld_act(w, i + half) : 1.f);
    float s, c;
    sincosf(pos * freq[i], &s, &c);
    s *= rot_mult;
    c *= rot_mult;
    st_act(q, i, u * c - v * s);
    st_act(q, i + half, v * c + u * s);
  }
  for (int i = rot_dims + lane; i < size; i += 32) st_act(q, i, ld_act(p, i) * r * (w ? ld_act(w, i) : 1.f));
}

}  // namespace b2l

using namespace b2l;

extern "C" int b2l_seq_embed(const void* tokens, int tokens_i64, const void* table, int act_dtype, float scale, float* x, void* h,
                             int T, int D, int vocab, b2l_stream_t stream) {
  B2L_CHECK_ARG(tokens && table && x, "b2l_seq_embed: null pointer");
  B2L_CHECK_ARG(T >= 0 && D > 0 && vocab > 0, "b2l_seq_embed: bad size");
  if (T == 0) return 0;
  const size_t es = act_dtype == B2L_F32 ? 4 : 2;
  const bool vec = D % 4 == 0 && al4(table, es) && al4(x, 4) && al4(h, es);
  B2L_SEQ_DISPATCH(act_dtype, {
    if (vec && tokens_i64)
      seq_embed_vec_kernel<act_t, long long><<<T, 128, 0, (cudaStream_t)stream>>>((const long long*)tokens, (const act_t*)table, scale, x, (act_t*)h, D, vocab);
    else if (vec)
      seq_embed_vec_kernel<act_t, int><<<T, 128, 0, (cudaStream_t)stream>>>((const int*)tokens, (const act_t*)table, scale, x, (act_t*)h, D, vocab);
    else if (tokens_i64)
      seq_embed_kernel<act_t, long long><<<T, 128, 0, (cudaStream_t)stream>>>((const long long*)tokens, (const act_t*)table, scale, x, (act_t*)h, D, vocab);
    else
      seq_embed_kernel<act_t, int><<<T, 128, 0, (cudaStream_t)stream>>>((const int*)tokens, (const act_t*)table, scale, x, (act_t*)h, D, vocab);
  });
  B2L_LAUNCH_CHECK("seq_embed_kernel");
  return 0;
}

extern "C" int b2l_seq_rmsnorm(const float* x, const void* w, float eps, void* out, const int* rows, int n_rows, int D,
                               int act_dtype, b2l_stream_t stream) {
  B2L_CHECK_ARG(x && w && out, "b2l_seq_rmsnorm: null pointer");
  B2L_CHECK_ARG(n_rows >= 0 && D > 0, "b2l_seq_rmsnorm: bad size");
  if (n_rows == 0) return 0;
  const size_t es = act_dtype == B2L_F32 ? 4 : 2;
  const bool vec = D % 4 == 0 && al4(x, 4) && al4(w, es) && al4(out, es);
  B2L_SEQ_DISPATCH(act_dtype, {
    cudaStream_t s_ = (cudaStream_t)stream;
    if (vec && D <= 1024) seq_rmsnorm_vec_kernel<act_t, 1><<<n_rows, 256, 0, s_>>>(x, (const act_t*)w, eps, (act_t*)out, rows, D);
    else if (vec && D <= 2048) seq_rmsnorm_vec_kernel<act_t, 2><<<n_rows, 256, 0, s_>>>(x, (const act_t*)w, eps, (act_t*)out, rows, D);
    else if (vec && D <= 4096) seq_rmsnorm_vec_kernel<act_t, 4><<<n_rows, 256, 0, s_>>>(x, (const act_t*)w, eps, (act_t*)out, rows, D);
    else seq_rmsnorm_kernel<act_t><<<n_rows, 256, 0, s_>>>(x, (const act_t*)w, eps, (act_t*)out, rows, D);
  });
  B2L_LAUNCH_CHECK("seq_rmsnorm_kernel");
  return 0;
}

extern "C" int b2l_seq_norm_add_norm(const void* y, const void* w_post, float eps, float mult, float* x, const void* w_next, void* h,
                                     int T, int D, int act_dtype, b2l_stream_t stream) {
  B2L_CHECK_ARG(y && w_post && x, "b2l_seq_norm_add_norm: null pointer");
  B2L_CHECK_ARG(w_next == nullptr || h != nullptr, "b2l_seq_norm_add_norm: a next norm without its output");
  B2L_CHECK_ARG(T >= 0 && D > 0, "b2l_seq_norm_add_norm: bad size");
  if (T == 0) return 0;
#define B2L_NAN_ARGS (const act_t*)y, (const act_t*)w_post, eps, mult, x, (const act_t*)w_next, (act_t*)h, D
  B2L_SEQ_DISPATCH(act_dtype, {
    cudaStream_t s_ = (cudaStream_t)stream;
    const bool vec = D % 4 == 0 && al4(y, sizeof(act_t)) && al4(w_post, sizeof(act_t)) && al4(x, 4) && al4(w_next, sizeof(act_t)) && al4(h, sizeof(act_t));
    if (vec && D <= 1024) seq_norm_add_norm_vec_kernel<act_t, 1><<<T, 256, 0, s_>>>(B2L_NAN_ARGS);
    else if (vec && D <= 2048) seq_norm_add_norm_vec_kernel<act_t, 2><<<T, 256, 0, s_>>>(B2L_NAN_ARGS);
    else if (vec && D <= 4096) seq_norm_add_norm_vec_kernel<act_t, 4><<<T, 256, 0, s_>>>(B2L_NAN_ARGS);
    else if (D <= 1024) seq_norm_add_norm_reg_kernel<act_t, 4><<<T, 256, 0, s_>>>(B2L_NAN_ARGS);
    else if (D <= 2048) seq_norm_add_norm_reg_kernel<act_t, 8><<<T, 256, 0, s_>>>(B2L_NAN_ARGS);
    else if (D <= 4096) seq_norm_add_norm_reg_kernel<act_t, 16><<<T, 256, 0, s_>>>(B2L_NAN_ARGS);
    else seq_norm_add_norm_kernel<act_t><<<T, 256, 0, s_>>>(B2L_NAN_ARGS);
  });
#undef B2L_NAN_ARGS
  B2L_LAUNCH_CHECK("seq_norm_add_norm_kernel");
  return 0;
}

extern "C" int b2l_seq_gated_act(const void* gu, int ldgu, void* out, int T, int F, int act, float limit, int act_dtype, b2l_stream_t stream) {
  B2L_CHECK_ARG(gu && out, "b2l_seq_gated_act: null pointer");
  B2L_CHECK_ARG(T >= 0 && F > 0 && ldgu >= 2 * F, "b2l_seq_gated_act: bad size");
  B2L_CHECK_ARG(act >= 0 && act <= 3, "b2l_seq_gated_act: unknown activation %d", act);
  B2L_CHECK_ARG(act != B2L_SEQ_ACT_CLAMPED_SWISH || limit > 0.f, "b2l_seq_gated_act: the clamped unit needs a positive limit");
  if (T == 0) return 0;
  const bool vec = F % 8 == 0 && ldgu % 8 == 0 && (((uintptr_t)gu | (uintptr_t)out) & 15) == 0;
  B2L_SEQ_DISPATCH(act_dtype, {
    if (vec) {
      const int per = 16 / (int)sizeof(act_t);
      dim3 grid((unsigned)T, (unsigned)std::min((F / per + 255) / 256, 64));
      seq_gated_act_vec_kernel<act_t><<<grid, 256, 0, (cudaStream_t)stream>>>((const act_t*)gu, ldgu, (act_t*)out, F, act, limit);
    } else {
      dim3 grid((unsigned)T, (unsigned)std::min((F + 255) / 256, 64));
      seq_gated_act_kernel<act_t><<<grid, 256, 0, (cudaStream_t)stream>>>((const act_t*)gu, ldgu, (act_t*)out, F, act, limit);
    }
  });
  B2L_LAUNCH_CHECK("seq_gated_act_kernel");
  return 0;
}

// `unit`: heads to normalise; done here where the four-tap kernel runs (*unit_done), left to the caller otherwise
static int conv_silu(const void* in, int ldin, const void* w, const void* bias, void* state, const int* meta, float* out, int ldout, int T, int C, int taps, int act_dtype,
                     const UnitHeads* unit, bool* unit_done, b2l_stream_t stream) {
  B2L_CHECK_ARG(in && w && (state || taps == 1) && meta && out, "b2l_seq_conv_silu: null pointer");
  B2L_CHECK_ARG(T >= 0 && C > 0 && ldin >= C && ldout >= C, "b2l_seq_conv_silu: bad size");
  B2L_CHECK_SUPPORTED(taps >= 1 && taps <= CONV_MAX_TAPS, "b2l_seq_conv_silu: taps %d outside 1..%d", taps, CONV_MAX_TAPS);
  if (T == 0) return 0;
  const int tiles = (T + CONV_TT - 1) / CONV_TT;
  dim3 grid((unsigned)((C + 127) / 128), (unsigned)tiles);
  if (act_dtype == B2L_BF16 && taps == 4 && C % 8 == 0 && ldin % 8 == 0 && ldout % 4 == 0 && al16(in) && al16(w) && al16(state) && al16(out) &&
      (T + CONV_VT - 1) / CONV_VT <= 65535) {      // with fewer CTAs than eight an SM, four tokens a thread stay below as well
    const int wide = unit && unit->size > 128 ? 8 : 4, lanes = unit ? unit->size / wide : 0;       // a head of the unit vectors lies in one warp
    const bool fits = unit && unit->size % wide == 0 && lanes >= 1 && lanes <= 32 && (lanes & (lanes - 1)) == 0 && unit->a0 % unit->size == 0 && unit->b0 % unit->size == 0 &&
                      unit->ma != 0.f && unit->mb != 0.f;
    const long long across = (C / (fits ? wide : 4) + 127) / 128;
    const bool few = across * ((T + CONV_VT - 1) / CONV_VT) < 8LL * sm_count();
    const int vt = few ? CONV_VT_FEW : CONV_VT;
    const dim3 grid4((unsigned)across, (unsigned)((T + vt - 1) / vt));
    auto pick = [&](auto n) {
      constexpr int N = decltype(n)::value;
      return !fits ? seq_conv4_silu_kernel<false, 4, N> : wide == 8 ? seq_conv4_silu_kernel<true, 8, N> : seq_conv4_silu_kernel<true, 4, N>;
    };
    auto kernel = few ? pick(std::integral_constant<int, CONV_VT_FEW>{}) : pick(std::integral_constant<int, CONV_VT>{});
    kernel<<<grid4, 128, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)in, ldin, (const __nv_bfloat16*)w, (const __nv_bfloat16*)bias, (__nv_bfloat16*)state, meta, out, ldout,
                                                    T, C, fits ? *unit : UnitHeads{});
    if (unit_done) *unit_done = fits;
    B2L_LAUNCH_CHECK("seq_conv4_silu_kernel");
    return 0;
  }
  B2L_SEQ_DISPATCH(act_dtype, {
    seq_conv_silu_kernel<act_t><<<grid, 128, 0, (cudaStream_t)stream>>>((const act_t*)in, ldin, (const act_t*)w, (const act_t*)bias,
                                                                        (act_t*)state, meta, out, ldout, T, C, taps);
  });
  B2L_LAUNCH_CHECK("seq_conv_silu_kernel");
  return 0;
}

extern "C" int b2l_seq_conv_silu(const void* in, int ldin, const void* w, const void* bias, void* state, const int* meta,
                                 float* out, int ldout, int T, int C, int taps, int act_dtype, b2l_stream_t stream) {
  return conv_silu(in, ldin, w, bias, state, meta, out, ldout, T, C, taps, act_dtype, nullptr, nullptr, stream);
}

extern "C" int b2l_seq_conv_silu_unit(const void* in, int ldin, const void* w, const void* bias, void* state, const int* meta, float* out, int ldout, int T, int C, int taps,
                                      int q_at, int k_at, int heads, int size, float eps, float q_mult, float k_mult, int act_dtype, b2l_stream_t stream) {
  B2L_CHECK_ARG(heads > 0 && size > 0 && q_at >= 0 && k_at >= 0 && q_at + heads * size <= C && k_at + heads * size <= C, "b2l_seq_conv_silu_unit: heads outside the channels");
  B2L_CHECK_ARG(q_at + heads * size <= k_at || k_at + heads * size <= q_at, "b2l_seq_conv_silu_unit: the two rows of heads overlap");
  const UnitHeads u{q_at, q_at + heads * size, k_at, k_at + heads * size, size, eps, q_mult, k_mult};
  bool done = false;
  if (int rc = conv_silu(in, ldin, w, bias, state, meta, out, ldout, T, C, taps, act_dtype, &u, &done, stream)) return rc;
  if (done || T == 0) return 0;
  if (int rc = b2l_seq_unit_norm(out + q_at, ldout, T, heads, size, eps, q_mult, stream)) return rc;
  return b2l_seq_unit_norm(out + k_at, ldout, T, heads, size, eps, k_mult, stream);
}

extern "C" int b2l_seq_cast_f32(const void* in, int ldin, float* out, int ldout, int T, int n, int act_dtype, b2l_stream_t stream) {
  B2L_CHECK_ARG(in && out, "b2l_seq_cast_f32: null pointer");
  B2L_CHECK_ARG(T >= 0 && n > 0 && ldin >= n && ldout >= n, "b2l_seq_cast_f32: bad size");
  if (T == 0) return 0;
  const bool vec = n % 4 == 0 && ldin % 4 == 0 && ldout % 4 == 0 && al4(in, act_dtype == B2L_F32 ? 4 : 2) && al4(out, 4);
  const int items = vec ? n / 4 : n;
  dim3 grid((unsigned)T, (unsigned)std::min((items + 255) / 256, 64));
  B2L_SEQ_DISPATCH(act_dtype, {
    if (vec) seq_cast_f32_vec_kernel<act_t><<<grid, 256, 0, (cudaStream_t)stream>>>((const act_t*)in, ldin, out, ldout, n);
    else seq_cast_f32_kernel<act_t><<<grid, 256, 0, (cudaStream_t)stream>>>((const act_t*)in, ldin, out, ldout, n);
  });
  B2L_LAUNCH_CHECK("seq_cast_f32_kernel");
  return 0;
}

extern "C" int b2l_seq_unit_norm(float* x, int ld, int T, int heads, int size, float eps, float mult, b2l_stream_t stream) {
  B2L_CHECK_ARG(x != nullptr, "b2l_seq_unit_norm: null pointer");
  B2L_CHECK_ARG(T >= 0 && heads > 0 && size > 0 && ld >= heads * size, "b2l_seq_unit_norm: bad size");
  if (T == 0) return 0;
  const int n = T * heads;
  seq_unit_norm_kernel<<<(n + 3) / 4, 128, 0, (cudaStream_t)stream>>>(x, ld, n, heads, size, eps, mult);
  B2L_LAUNCH_CHECK("seq_unit_norm_kernel");
  return 0;
}

extern "C" int b2l_seq_decay(const void* a, int lda, const void* bias, const void* A_log, int mode, float tau, float* out,
                             float* dt_out, int T, int heads, int size, int act_dtype, b2l_stream_t stream) {
  B2L_CHECK_ARG(a && out, "b2l_seq_decay: null pointer");
  B2L_CHECK_ARG(T >= 0 && heads > 0 && size > 0 && lda >= heads * size, "b2l_seq_decay: bad size");
  B2L_CHECK_ARG(mode == B2L_SEQ_DECAY_SIGMOID_ROOT || (mode == B2L_SEQ_DECAY_EXP_SOFTPLUS && A_log), "b2l_seq_decay: bad mode or no A_log");
  B2L_CHECK_ARG(mode != B2L_SEQ_DECAY_SIGMOID_ROOT || tau > 0.f, "b2l_seq_decay: tau must be positive");
  if (T == 0) return 0;
  const int n = heads * size;
  if (act_dtype == B2L_BF16 && size % 8 == 0 && lda % 8 == 0 && al16(a) && al16(out) && (!bias || al16(bias)) && (!dt_out || al16(dt_out))) {
    const int threads = n >= 2048 ? 256 : 64;
    seq_decay8_kernel<<<dim3((unsigned)T, (unsigned)((n / 8 + threads - 1) / threads)), threads, 0, (cudaStream_t)stream>>>(
        (const __nv_bfloat16*)a, lda, (const __nv_bfloat16*)bias, (const __nv_bfloat16*)A_log, mode, mode == B2L_SEQ_DECAY_SIGMOID_ROOT ? 1.0f / tau : 0.f, out, dt_out, n, size);
    B2L_LAUNCH_CHECK("seq_decay8_kernel");
    return 0;
  }
  dim3 grid((unsigned)T, (unsigned)std::min((n + 255) / 256, 64));
  B2L_SEQ_DISPATCH(act_dtype, (seq_decay_kernel<act_t><<<grid, 256, 0, (cudaStream_t)stream>>>(
                                  (const act_t*)a, lda, (const act_t*)bias, (const act_t*)A_log, mode, mode == B2L_SEQ_DECAY_SIGMOID_ROOT ? 1.0f / tau : 0.f,
                                  out, dt_out, heads, size)));
  B2L_LAUNCH_CHECK("seq_decay_kernel");
  return 0;
}

extern "C" int b2l_seq_group_norm_gate(const float* o, int ldo, const void* w, int w_shared, const void* gate, int ldg,
                                       int gate_act, int gate_first, float eps, float out_mult, void* out, int ldout, int T,
                                       int n, int group, int act_dtype, b2l_stream_t stream) {
  B2L_CHECK_ARG(o && w && out, "b2l_seq_group_norm_gate: null pointer");
  B2L_CHECK_ARG(T >= 0 && n > 0 && group > 0 && n % group == 0 && ldo >= n && ldout >= n, "b2l_seq_group_norm_gate: bad size");
  if (T == 0) return 0;
  const int ids = T * (n / group);
  auto al = [](const void* p, int bytes) { return ((uintptr_t)p & (bytes - 1)) == 0; };
  if (act_dtype == B2L_BF16 && (group == 128 || group == 256) && ldo % 4 == 0 && al16(o)) {
    const int per = group / 32;
    if (ldout % per == 0 && al(out, 2 * per) && al(w, 2 * per) && (!gate || (ldg % per == 0 && al(gate, 2 * per)))) {
      const bool fours = per == 4 && n / group % 4 == 0 && ids >= 56 * sm_count();
      auto kernel = fours ? seq_group_norm_gate_fours_kernel<4> : per == 4 ? seq_group_norm_gate_vec_kernel<4> : seq_group_norm_gate_vec_kernel<8>;
      kernel<<<fours ? (ids + 15) / 16 : (ids + 3) / 4, 128, 0, (cudaStream_t)stream>>>(o, ldo, (const __nv_bfloat16*)w, w_shared, (const __nv_bfloat16*)gate, ldg, gate_act, gate_first, eps, out_mult,
                                                              (__nv_bfloat16*)out, ldout, T, n / group);
      B2L_LAUNCH_CHECK("seq_group_norm_gate_vec_kernel");
      return 0;
    }
  }
  if (act_dtype == B2L_BF16 && group >= 512 && group <= 8192 && group % 8 == 0 && ldo % 4 == 0 && ldout % 8 == 0 && al16(o) && al16(w) && al16(out) &&
      (!gate || (ldg % 8 == 0 && al16(gate)))) {
    auto kernel = group <= 2048 ? seq_group_norm_gate_wide_kernel<1> : group <= 4096 ? seq_group_norm_gate_wide_kernel<2> : seq_group_norm_gate_wide_kernel<4>;
    kernel<<<ids, 256, 0, (cudaStream_t)stream>>>(o, ldo, (const __nv_bfloat16*)w, w_shared, (const __nv_bfloat16*)gate, ldg, gate_act, gate_first, eps, out_mult,
                                                  (__nv_bfloat16*)out, ldout, n / group, group);
    B2L_LAUNCH_CHECK("seq_group_norm_gate_wide_kernel");
    return 0;
  }
  B2L_SEQ_DISPATCH(act_dtype, {
    if (group >= 512)
      seq_group_norm_gate_block_kernel<act_t><<<ids, 256, 0, (cudaStream_t)stream>>>(
          o, ldo, (const act_t*)w, w_shared, (const act_t*)gate, ldg, gate_act, gate_first, eps, out_mult, (act_t*)out, ldout, n / group, group);
    else
      seq_group_norm_gate_kernel<act_t><<<(ids + 3) / 4, 128, 0, (cudaStream_t)stream>>>(
          o, ldo, (const act_t*)w, w_shared, (const act_t*)gate, ldg, gate_act, gate_first, eps, out_mult, (act_t*)out, ldout, T, n / group, group);
  });
  B2L_LAUNCH_CHECK("seq_group_norm_gate_kernel");
  return 0;
}

extern "C" int b2l_seq_headnorm_rope(const void* x, int ldx, const void* w, float eps, const float* freq, int rot_dims,
                                     float rot_mult, const int* meta, void* out, int out_f32, int T, int heads, int size,
                                     int act_dtype, b2l_stream_t stream) {
  B2L_CHECK_ARG(x && meta && out, "b2l_seq_headnorm_rope: null pointer");
  B2L_CHECK_ARG(T >= 0 && heads > 0 && size > 0 && ldx >= heads * size, "b2l_seq_headnorm_rope: bad size");
  B2L_CHECK_ARG(rot_dims >= 0 && rot_dims <= size && rot_dims % 2 == 0 && (rot_dims == 0 || freq), "b2l_seq_headnorm_rope: bad rotation");
  if (T == 0) return 0;
  const int ids = T * heads;
  B2L_SEQ_DISPATCH(act_dtype, {
    if (out_f32)
      seq_headnorm_rope_kernel<act_t, float><<<(ids + 3) / 4, 128, 0, (cudaStream_t)stream>>>(
          (const act_t*)x, ldx, (const act_t*)w, eps, freq, rot_dims, rot_mult, meta, (float*)out, T, heads, size);
    else
      seq_headnorm_rope_kernel<act_t, act_t><<<(ids + 3) / 4, 128, 0, (cudaStream_t)stream>>>(
          (const act_t*)x, ldx, (const act_t*)w, eps, freq, rot_dims, rot_mult, meta, (act_t*)out, T, heads, size);
  });
  B2L_LAUNCH_CHECK("seq_headnorm_rope_kernel");
  return 0;
}

// ---- residual streams with two sublayers on the same input ----
namespace b2l {

// x += y1 + y2 (each may be null), then up to two RMS norms of the new row with weights stored around `w_offset`
// (h = x / rms(x) * (w_offset + w)): a layer whose mixer and feed-forward read the same x with a norm each.  `rows`
// picks the rows (out row r <- x row rows[r]) when nothing is added.  One CTA per row; the sum is f32.
template <typename act_t>
__global__ void __launch_bounds__(256) seq_add_norm2_kernel(const act_t* __restrict__ y1, const act_t* __restrict__ y2, float* __restrict__ x,
                                                            const act_t* __restrict__ w1, act_t* __restrict__ h1,
                                                            const act_t* __restrict__ w2, act_t* __restrict__ h2, float w_offset, float eps,
                                                            const int* __restrict__ rows, int D) {
  __shared__ float red[32];
  const int r = rows ? rows[blockIdx.x] : blockIdx.x;
  float* xr = x + (size_t)r * D;
  float ss = 0.f;
  for (int i = threadIdx.x; i < D; i += blockDim.x) {
    float v = xr[i];
    if (y1) {
      float add = ld_act(y1, (size_t)r * D + i);
      if (y2) add += ld_act(y2, (size_t)r * D + i);
      v += add;
      xr[i] = v;
    }
    ss += v * v;
  }
  if (w1 == nullptr) return;
  ss = block_sum(ss, red);
  const float rinv = 1.0f / sqrtf(ss / (float)D + eps);
  for (int i = threadIdx.x; i < D; i += blockDim.x) {       // own writes of xr: visible to this thread
    const float v = xr[i] * rinv;
    st_act(h1, (size_t)blockIdx.x * D + i, v * (w_offset + ld_act(w1, i)));
    if (w2) st_act(h2, (size_t)blockIdx.x * D + i, v * (w_offset + ld_act(w2, i)));
  }
}

__global__ void seq_softcap_kernel(float* __restrict__ z, size_t n, float cap) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) z[i] = cap * tanhf(z[i] / cap);
}

}  // namespace b2l

extern "C" int b2l_seq_add_norm2(const void* y1, const void* y2, float* x, const void* w1, void* h1, const void* w2, void* h2,
                                 float w_offset, float eps, const int* rows, int n_rows, int D, int act_dtype, b2l_stream_t stream) {
  B2L_CHECK_ARG(x != nullptr && (y1 != nullptr || y2 == nullptr), "b2l_seq_add_norm2: null pointer");
  B2L_CHECK_ARG((w1 == nullptr) == (h1 == nullptr) && (w2 == nullptr) == (h2 == nullptr) && (w1 != nullptr || w2 == nullptr),
                "b2l_seq_add_norm2: every norm needs its weight and its output, the second norm needs the first");
  B2L_CHECK_ARG(rows == nullptr || y1 == nullptr, "b2l_seq_add_norm2: rows are picked only when nothing is added");
  B2L_CHECK_ARG(n_rows >= 0 && D > 0, "b2l_seq_add_norm2: bad size");
  if (n_rows == 0 || (y1 == nullptr && w1 == nullptr)) return 0;
  B2L_SEQ_DISPATCH(act_dtype, {
    seq_add_norm2_kernel<act_t><<<n_rows, 256, 0, (cudaStream_t)stream>>>((const act_t*)y1, (const act_t*)y2, x, (const act_t*)w1, (act_t*)h1,
                                                                         (const act_t*)w2, (act_t*)h2, w_offset, eps, rows, D);
  });
  B2L_LAUNCH_CHECK("seq_add_norm2_kernel");
  return 0;
}

extern "C" int b2l_seq_softcap(float* z, size_t n, float cap, b2l_stream_t stream) {
  B2L_CHECK_ARG(z != nullptr && cap > 0.f, "b2l_seq_softcap: null pointer or cap <= 0");
  if (n == 0) return 0;
  const int grid = (int)((n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096);
  b2l::seq_softcap_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(z, n, cap);
  B2L_LAUNCH_CHECK("seq_softcap_kernel");
  return 0;
}
