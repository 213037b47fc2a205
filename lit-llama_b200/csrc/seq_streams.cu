// Several residual streams (hyper-connections), a hashed token-pair embedding beside the token embedding, and the
// preparation of attention operands from one stacked projection: RMS norm of queries and keys (over the whole
// projection or per head), partial rotation, and the mixing of values with those of an earlier layer.
// All arithmetic is f32; `act_t` is only the storage type of projection outputs and weights.
#include "seq_common.cuh"

namespace b2l {

constexpr int HC_MAX_STREAMS = 16;

// x[t, s, :] = table[token[t]] * scale + pair[row(t)] for every stream s, with
//   row(t) = (previous token * mul_prev + token[t] * mul_cur) mod buckets, and row `buckets` at position 0.
// The previous token of the portion's first token is the sequence's state (int32 per slot); the CTA of token 0 reads
// it and then stores the portion's last token there, so no other CTA touches the state.
template <typename act_t, typename idx_t>
__global__ void seq_embed_pair_kernel(const idx_t* __restrict__ tok, const act_t* __restrict__ table, const act_t* __restrict__ pair,
                                      float scale, int* __restrict__ prev_state, const int* __restrict__ meta, long long mul_prev,
                                      long long mul_cur, int buckets, float* __restrict__ x, int T, int D, int vocab, int streams) {
  const int t = blockIdx.x;
  long long cur = (long long)tok[t];
  if (cur < 0 || cur >= vocab) cur = 0;
  long long row = -1;
  if (pair != nullptr) {
    __shared__ long long s_prev;
    if (threadIdx.x == 0) {
      long long prev;
      if (t > 0) {
        prev = (long long)tok[t - 1];
        if (prev < 0 || prev >= vocab) prev = 0;
      } else {
        prev = meta[1] > 0 ? (long long)prev_state[meta[0]] : -1;
        long long last = (long long)tok[T - 1];
        if (last < 0 || last >= vocab) last = 0;
        prev_state[meta[0]] = (int)last;
      }
      s_prev = prev;
    }
    __syncthreads();
    const long long prev = s_prev;
    // (prev * mul_prev + cur * mul_cur) mod buckets with every factor reduced first: no overflow for any multiplier
    const long long b = buckets;
    row = prev < 0 ? b : ((prev % b) * (mul_prev % b) + (cur % b) * (mul_cur % b)) % b;
  }
  const act_t* src = table + (size_t)cur * D;
  const act_t* add = row >= 0 ? pair + (size_t)row * D : nullptr;
  float* dst = x + (size_t)t * streams * D;
  for (int i = threadIdx.x; i < D; i += blockDim.x) {
    float v = ld_act(src, i) * scale;
    if (add) v += ld_act(add, i);
    for (int s = 0; s < streams; ++s) dst[(size_t)s * D + i] = v;
  }
}

// One sublayer's step on S residual streams X [rows][S][D] (f32), one CTA per row:
//   write (y given):        X_t <- sum_s mix[s, t] X_s + out[t] y           (all streams at once from the old ones)
//   read  (w_next given):   h = rmsnorm(sum_s in_next[s] X_s) * w_next      (of the new streams)
// `rows` picks the rows that are read when nothing is written (h row r <- X row rows[r]).  The mixed row u stays in
// shared memory between the sum of squares and the scaling.
template <typename act_t, int S>
__global__ void __launch_bounds__(256) seq_hc_step_kernel(const act_t* __restrict__ y, float* __restrict__ X, const float* __restrict__ mix,
                                                          const float* __restrict__ outw, const float* __restrict__ in_next,
                                                          const act_t* __restrict__ w_next, act_t* __restrict__ h, float eps,
                                                          const int* __restrict__ rows, int D, int s_rt) {
  extern __shared__ float hc_u[];
  __shared__ float red[32];
  const int n_s = S > 0 ? S : s_rt;
  const int r = rows ? rows[blockIdx.x] : blockIdx.x;
  float* xr = X + (size_t)r * n_s * D;
  float m[HC_MAX_STREAMS * HC_MAX_STREAMS], o[HC_MAX_STREAMS], a[HC_MAX_STREAMS];
#pragma unroll
  for (int s = 0; s < HC_MAX_STREAMS; ++s) {
    if (s >= n_s) break;
    o[s] = y ? outw[s] : 0.f;
    a[s] = in_next ? in_next[s] : 0.f;
#pragma unroll
    for (int t = 0; t < HC_MAX_STREAMS; ++t) {
      if (t >= n_s) break;
      m[s * HC_MAX_STREAMS + t] = y ? mix[s * n_s + t] : 0.f;
    }
  }
  float ss = 0.f;
  for (int i = threadIdx.x; i < D; i += blockDim.x) {
    float xs[HC_MAX_STREAMS];
#pragma unroll
    for (int s = 0; s < HC_MAX_STREAMS; ++s) {
      if (s >= n_s) break;
      xs[s] = xr[(size_t)s * D + i];
    }
    float u = 0.f;
    if (y) {
      const float yv = ld_act(y, (size_t)r * D + i);
#pragma unroll
      for (int t = 0; t < HC_MAX_STREAMS; ++t) {
        if (t >= n_s) break;
        float v = o[t] * yv;
#pragma unroll
        for (int s = 0; s < HC_MAX_STREAMS; ++s) {
          if (s >= n_s) break;
          v = fmaf(m[s * HC_MAX_STREAMS + t], xs[s], v);
        }
        xr[(size_t)t * D + i] = v;
        u = fmaf(a[t], v, u);
      }
    } else {
#pragma unroll
      for (int s = 0; s < HC_MAX_STREAMS; ++s) {
        if (s >= n_s) break;
        u = fmaf(a[s], xs[s], u);
      }
    }
    if (w_next) {
      hc_u[i] = u;
      ss += u * u;
    }
  }
  if (w_next == nullptr) return;
  ss = block_sum(ss, red);
  const float rinv = 1.0f / sqrtf(ss / (float)D + eps);
  act_t* hr = h + (size_t)blockIdx.x * D;
  for (int i = threadIdx.x; i < D; i += blockDim.x) st_act(hr, i, hc_u[i] * rinv * ld_act(w_next, i));     // own writes of hc_u
}

// out[t, :] = sum_s X[t, s, :]  (diagnostics: the residual stream as one vector).
__global__ void seq_hc_sum_kernel(const float* __restrict__ X, float* __restrict__ out, int D, int n_s) {
  const float* xr = X + (size_t)blockIdx.x * n_s * D;
  for (int i = threadIdx.x; i < D; i += blockDim.x) {
    float v = 0.f;
    for (int s = 0; s < n_s; ++s) v += xr[(size_t)s * D + i];
    out[(size_t)blockIdx.x * D + i] = v;
  }
}

__global__ void seq_scale_kernel(float* __restrict__ z, size_t n, float mult) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) z[i] *= mult;
}

constexpr int MOST_PAIRS = 4096;      // rotated pairs whose cos and sin fit the 48 KB of a launch without an attribute

// Attention operands of one token from the stacked projection row, one CTA per token.  `quads`: four neighbouring pairs per thread with 8-byte loads, where
// whole heads turn and a row has one factor (40960 entries with norms, us with them and a pair of two bytes at a time: one token 41 / 115, 2048 tokens 153 / 351).
//   q_out (f32) and k_out (act): RMS norm (whole_row: over all heads*K entries with a weight of that size; else per
//   head with a weight of K entries shared by the heads; no weight: no norm), then rotation of the first rot_dims
//   entries of every head (entry i with entry i + rot_dims/2) by the angle (pos0 + t) * freq[i]; unit_rms (no weights): the
//   rotated head divided by its root mean square.  A rotation keeps the length of the pairs it turns up to rot_mult, so
//   the sum of squares is taken from the entries before it.
//   q_out is multiplied by the query temperature of its position when temp_every > 0.
//   v_out (act): (1 - lambda) v + lambda v_first when v_first is given (lambda read on the device), else not written.
template <typename act_t, bool TABLE>      // TABLE: up to MOST_PAIRS pairs
__global__ void __launch_bounds__(256) seq_qkv_prep_kernel(b2l_seq_qkv_prep_args a, int quads) {
  __shared__ float red[32];
  const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const act_t* row = (const act_t*)a.proj + (size_t)t * a.ld;
  const float pos = (float)(a.meta[1] + t);
  const int half = a.rot_dims / 2, K = a.K;
  const float temp = a.temp_every > 0 ? 1.0f + a.temp_coef * logf((float)((a.meta[1] + t + 1) / a.temp_every + 1)) : 1.0f;
  // every head turns by the same angles: once per token instead of once per head (16 + 4 heads, 2048 tokens: 29 -> 27 us)
  extern __shared__ float turn[];                       // cos | sin of the pairs, times rot_mult
  for (int i = threadIdx.x; TABLE && i < half; i += blockDim.x) {
    float s, c;
    sincosf(pos * a.freq[i], &s, &c);
    turn[i] = c * a.rot_mult;
    turn[half + i] = s * a.rot_mult;
  }
  __syncthreads();
  for (int which = 0; which < 2; ++which) {
    const act_t* x = row + (which == 0 ? a.q_off : a.k_off);
    const act_t* w = (const act_t*)(which == 0 ? a.q_norm : a.k_norm);
    const int heads = which == 0 ? a.heads : a.kv_heads;
    float r_row = 1.f;
    if (w && a.whole_row) {
      float ss = 0.f;
      if (quads && sizeof(act_t) == 2) {
        for (int i = threadIdx.x * 4; i < heads * K; i += blockDim.x * 4) {
          const uint2 u = *reinterpret_cast<const uint2*>(x + i);
          const float v0 = __uint_as_float(u.x << 16), v1 = __uint_as_float(u.x & 0xffff0000u), v2 = __uint_as_float(u.y << 16), v3 = __uint_as_float(u.y & 0xffff0000u);
          ss += (v0 * v0 + v1 * v1) + (v2 * v2 + v3 * v3);
        }
      } else {
        for (int i = threadIdx.x; i < heads * K; i += blockDim.x) {
          const float v = ld_act(x, i);
          ss += v * v;
        }
      }
      ss = block_sum(ss, red);
      r_row = 1.0f / sqrtf(ss / (float)(heads * K) + a.eps);
    }
    if (quads && sizeof(act_t) == 2) {
      // one factor for the whole row: four neighbouring pairs per thread, 8-byte loads (a lane per pair with 2-byte loads took 27 us for 2048 tokens of 16 + 4 heads, so 17)
      const int per = half / 4;
      for (int u = threadIdx.x; u < heads * per; u += blockDim.x) {
        const int hd = u / per, i = (u - hd * per) * 4;
        const __nv_bfloat16* p = reinterpret_cast<const __nv_bfloat16*>(x) + (size_t)hd * K + i;
        const __nv_bfloat16* pw = reinterpret_cast<const __nv_bfloat16*>(w) + (size_t)hd * K + i;
        const uint2 a0 = *reinterpret_cast<const uint2*>(p), a1 = *reinterpret_cast<const uint2*>(p + half);
        const uint2 w0 = w ? *reinterpret_cast<const uint2*>(pw) : make_uint2(0x3f803f80u, 0x3f803f80u);
        const uint2 w1 = w ? *reinterpret_cast<const uint2*>(pw + half) : make_uint2(0x3f803f80u, 0x3f803f80u);
        const uint32_t ua[4] = {a0.x, a0.y, a1.x, a1.y}, uw[4] = {w0.x, w0.y, w1.x, w1.y};
        float lo[4], hi[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int j = e >> 1;
          const float xu = __uint_as_float(e & 1 ? ua[j] & 0xffff0000u : ua[j] << 16), wu = __uint_as_float(e & 1 ? uw[j] & 0xffff0000u : uw[j] << 16);
          const float xv = __uint_as_float(e & 1 ? ua[2 + j] & 0xffff0000u : ua[2 + j] << 16), wv = __uint_as_float(e & 1 ? uw[2 + j] & 0xffff0000u : uw[2 + j] << 16);
          const float pu = xu * r_row * wu, pv = xv * r_row * wv, c = turn[i + e], s = turn[half + i + e];
          lo[e] = pu * c - pv * s;
          hi[e] = pv * c + pu * s;
        }
        if (which == 0) {
          float* qo = a.q_out + ((size_t)t * heads + hd) * K + i;
          *reinterpret_cast<float4*>(qo) = make_float4(lo[0] * temp, lo[1] * temp, lo[2] * temp, lo[3] * temp);
          *reinterpret_cast<float4*>(qo + half) = make_float4(hi[0] * temp, hi[1] * temp, hi[2] * temp, hi[3] * temp);
        } else {
          __nv_bfloat16* ko = (__nv_bfloat16*)a.k_out + ((size_t)t * heads + hd) * K + i;
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            const float (&y)[4] = b ? hi : lo;
            const __nv_bfloat162 y0 = __floats2bfloat162_rn(y[0], y[1]), y1 = __floats2bfloat162_rn(y[2], y[3]);
            *reinterpret_cast<uint2*>(ko + b * half) = make_uint2(*reinterpret_cast<const uint32_t*>(&y0), *reinterpret_cast<const uint32_t*>(&y1));
          }
        }
      }
      continue;
    }
    for (int hd = warp; hd < heads; hd += nw) {
      const act_t* p = x + (size_t)hd * K;
      const act_t* wh = w ? (a.whole_row ? w + (size_t)hd * K : w) : nullptr;
      float r = r_row;
      if (a.unit_rms || (w && !a.whole_row)) {
        const float turned = a.unit_rms ? a.rot_mult : 1.f;
        float ss = 0.f;
        for (int i = lane; i < K; i += 32) {
          const float v = ld_act(p, i) * (i < a.rot_dims ? turned : 1.f);
          ss += v * v;
        }
        ss = warp_sum(ss);
        r = 1.0f / sqrtf(ss / (float)K + a.eps);
      }
      float* qo = a.q_out + ((size_t)t * heads + hd) * K;
      act_t* ko = (act_t*)a.k_out + ((size_t)t * heads + hd) * K;
      for (int i = lane; i < half; i += 32) {
        const float u = ld_act(p, i) * r * (wh ? ld_act(wh, i) : 1.f);
        const float v = ld_act(p, i + half) * r * (wh ? ld_act(wh, i + half) : 1.f);
        float c, s;
        if constexpr (TABLE) {
          c = turn[i];
          s = turn[half + i];
        } else {
          sincosf(pos * a.freq[i], &s, &c);
          s *= a.rot_mult;
          c *= a.rot_mult;
        }
        if (which == 0) {
          qo[i] = (u * c - v * s) * temp;
          qo[i + half] = (v * c + u * s) * temp;
        } else {
          st_act(ko, i, u * c - v * s);
          st_act(ko, i + half, v * c + u * s);
        }
      }
      for (int i = a.rot_dims + lane; i < K; i += 32) {
        const float v = ld_act(p, i) * r * (wh ? ld_act(wh, i) : 1.f);
        if (which == 0) qo[i] = v * temp;
        else st_act(ko, i, v);
      }
    }
  }
  if (a.v_first != nullptr) {
    const float lam = ld_act((const act_t*)a.lambda, 0);
    const act_t* v = row + a.v_off;
    const act_t* vf = (const act_t*)a.v_first + (size_t)t * a.ldvf;
    act_t* vo = (act_t*)a.v_out + (size_t)t * a.kv_heads * a.V;
    for (int i = threadIdx.x; i < a.kv_heads * a.V; i += blockDim.x) st_act(vo, i, (1.f - lam) * ld_act(v, i) + lam * ld_act(vf, i));
  }
}

// The same where whole heads turn and a row has one factor: four neighbouring pairs (u: 16 bytes of x in bf16) are a unit, a thread holds NU of the
// token's units in registers, so x is read once, with its norm weights for all of the CTA's tokens, and the next token's x travels meanwhile.
// Bound by the chain from launch to store, a barrier for the norms and the angles in it: 2048 tokens of 16 + 4 heads of 128 with norms take 9.1 us, their bytes
// 4.8.
constexpr int QUAD_THREADS = 512;
// four elements as they lie in memory
template <typename act_t> struct Quad;
template <> struct Quad<__nv_bfloat16> {
  uint2 v;
  __device__ __forceinline__ void ones() { v = make_uint2(0x3f803f80u, 0x3f803f80u); }
  __device__ __forceinline__ void load(const __nv_bfloat16* p) { v = *reinterpret_cast<const uint2*>(p); }
  __device__ __forceinline__ float operator[](int e) const {
    const uint32_t w = e & 2 ? v.y : v.x;
    return __uint_as_float(e & 1 ? w & 0xffff0000u : w << 16);
  }
};
template <> struct Quad<float> {
  float4 v;
  __device__ __forceinline__ void ones() { v = make_float4(1.f, 1.f, 1.f, 1.f); }
  __device__ __forceinline__ void load(const float* p) { v = *reinterpret_cast<const float4*>(p); }
  __device__ __forceinline__ float operator[](int e) const { return e & 2 ? (e & 1 ? v.w : v.z) : (e & 1 ? v.y : v.x); }
};
template <typename act_t, int NU>
__global__ void __launch_bounds__(QUAD_THREADS) seq_qkv_prep_quads_kernel(b2l_seq_qkv_prep_args a, int tokens) {
  __shared__ float red[2][2][QUAD_THREADS / 32];
  extern __shared__ __align__(16) float turn_quads[];   // per token: cos | sin of the pairs, times rot_mult
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
  const int K = a.K, half = K / 2, per = half / 4, units_q = a.heads * per, units = units_q + a.kv_heads * per;
  const int t0 = blockIdx.x * tokens, nt = min(tokens, a.T - t0);
  const act_t* qw = (const act_t*)a.q_norm;
  const act_t* kw = (const act_t*)a.k_norm;
  Quad<act_t> x0[NU], x1[NU], w0[NU], w1[NU];
  int at[NU], xat[NU];                                  // first entry of the unit: in its row of heads, in the projection's row
#pragma unroll
  for (int i = 0; i < NU; ++i) {
    const int u = min(tid + i * (int)blockDim.x, units - 1), uu = u < units_q ? u : u - units_q, hd = uu / per;
    at[i] = hd * K + (uu - hd * per) * 4;
    xat[i] = at[i] + (u < units_q ? a.q_off : a.k_off);
  }
  auto load = [&](int t) {
    const act_t* row = (const act_t*)a.proj + (size_t)t * a.ld;
#pragma unroll
    for (int i = 0; i < NU; ++i) {
      x0[i].load(row + xat[i]);
      x1[i].load(row + xat[i] + half);
    }
  };
  load(t0);
#pragma unroll
  for (int i = 0; i < NU; ++i) {
    const act_t* w = tid + i * (int)blockDim.x < units_q ? qw : kw;
    if (w) {
      w0[i].load(w + at[i]);
      w1[i].load(w + at[i] + half);
    } else {
      w0[i].ones();
      w1[i].ones();
    }
  }
  const int pos0 = a.meta[1] + t0;
  for (int i = tid; i < nt * half; i += blockDim.x) {
    const int n = i / half, j = i - n * half;
    float s, c;
    sincosf((float)(pos0 + n) * a.freq[j], &s, &c);
    turn_quads[n * K + j] = c * a.rot_mult;
    turn_quads[n * K + half + j] = s * a.rot_mult;
  }
  for (int n = 0; n < nt; ++n) {
    const int t = t0 + n;
    float rq = 1.f, rk = 1.f;
    if (qw || kw) {
      float sq = 0.f, sk = 0.f;
#pragma unroll
      for (int i = 0; i < NU; ++i) {
        const int u = tid + i * (int)blockDim.x;
        float ss = 0.f;
#pragma unroll
        for (int e = 0; e < 4; e += 2) ss += x0[i][e] * x0[i][e] + x0[i][e + 1] * x0[i][e + 1];
#pragma unroll
        for (int e = 0; e < 4; e += 2) ss += x1[i][e] * x1[i][e] + x1[i][e + 1] * x1[i][e + 1];
        if (u < units_q) sq += ss;
        else if (u < units) sk += ss;
      }
      sq = warp_sum(sq);
      sk = warp_sum(sk);
      if (lane == 0) { red[n & 1][0][warp] = sq; red[n & 1][1][warp] = sk; }
    }
    if (n == 0 || qw || kw) __syncthreads();            // the angles; the sums (the other buffer is read until the next token's barrier)
    if (qw || kw) {
      float sq = 0.f, sk = 0.f;
      for (int w = 0; w < nw; ++w) { sq += red[n & 1][0][w]; sk += red[n & 1][1][w]; }
      if (qw) rq = 1.0f / sqrtf(sq / (float)(a.heads * K) + a.eps);
      if (kw) rk = 1.0f / sqrtf(sk / (float)(a.kv_heads * K) + a.eps);
    }
    const float temp = a.temp_every > 0 ? 1.0f + a.temp_coef * logf((float)((pos0 + n + 1) / a.temp_every + 1)) : 1.0f;
    const float* tn = turn_quads + n * K;
    float y[NU][8];
#pragma unroll
    for (int i = 0; i < NU; ++i) {
      const bool is_q = tid + i * (int)blockDim.x < units_q;
      const float r = is_q ? rq : rk;
      const int j = at[i] % K;                          // the unit's first pair
      const float4 c4 = *reinterpret_cast<const float4*>(tn + j), s4 = *reinterpret_cast<const float4*>(tn + half + j);
      const float c[4] = {c4.x, c4.y, c4.z, c4.w}, s[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float pu = x0[i][e] * r * w0[i][e], pv = x1[i][e] * r * w1[i][e];
        y[i][e] = pu * c[e] - pv * s[e];
        y[i][4 + e] = pv * c[e] + pu * s[e];
      }
    }
    if (n + 1 < nt) load(t + 1);
#pragma unroll
    for (int i = 0; i < NU; ++i) {
      const int u = tid + i * (int)blockDim.x;
      if (u < units_q) {
        float* qo = a.q_out + (size_t)t * a.heads * K + at[i];
        *reinterpret_cast<float4*>(qo) = make_float4(y[i][0] * temp, y[i][1] * temp, y[i][2] * temp, y[i][3] * temp);
        *reinterpret_cast<float4*>(qo + half) = make_float4(y[i][4] * temp, y[i][5] * temp, y[i][6] * temp, y[i][7] * temp);
      } else if (u < units) {
        act_t* ko = (act_t*)a.k_out + (size_t)t * a.kv_heads * K + at[i];
        st_act4(ko, make_float4(y[i][0], y[i][1], y[i][2], y[i][3]));
        st_act4(ko + half, make_float4(y[i][4], y[i][5], y[i][6], y[i][7]));
      }
    }
    if (a.v_first != nullptr) {
      const float lam = ld_act((const act_t*)a.lambda, 0);
      const act_t* v = (const act_t*)a.proj + (size_t)t * a.ld + a.v_off;
      const act_t* vf = (const act_t*)a.v_first + (size_t)t * a.ldvf;
      act_t* vo = (act_t*)a.v_out + (size_t)t * a.kv_heads * a.V;
      for (int i = tid; i < a.kv_heads * a.V; i += blockDim.x) st_act(vo, i, (1.f - lam) * ld_act(v, i) + lam * ld_act(vf, i));
    }
  }
}

}  // namespace b2l

using namespace b2l;

extern "C" int b2l_seq_embed_pair(const void* tokens, int tokens_i64, const void* table, const void* pair_table, float scale,
                                  int* prev_state, const int* meta, long long mul_prev, long long mul_cur, int buckets, float* x, int T,
                                  int D, int vocab, int streams, int act_dtype, b2l_stream_t stream) {
  B2L_CHECK_ARG(tokens && table && x, "b2l_seq_embed_pair: null pointer");
  B2L_CHECK_ARG(pair_table == nullptr || (prev_state && meta && buckets > 0 && mul_prev >= 0 && mul_cur >= 0),
                "b2l_seq_embed_pair: the pair table needs its state, the slot and position pair and a positive bucket count");
  B2L_CHECK_ARG(T >= 0 && D > 0 && vocab > 0 && streams >= 1, "b2l_seq_embed_pair: bad size");
  if (T == 0) return 0;
  cudaStream_t s_ = (cudaStream_t)stream;
  B2L_SEQ_DISPATCH(act_dtype, {
    if (tokens_i64)
      seq_embed_pair_kernel<act_t, long long><<<T, 128, 0, s_>>>((const long long*)tokens, (const act_t*)table, (const act_t*)pair_table, scale,
                                                                  prev_state, meta, mul_prev, mul_cur, buckets, x, T, D, vocab, streams);
    else
      seq_embed_pair_kernel<act_t, int><<<T, 128, 0, s_>>>((const int*)tokens, (const act_t*)table, (const act_t*)pair_table, scale, prev_state,
                                                            meta, mul_prev, mul_cur, buckets, x, T, D, vocab, streams);
  });
  B2L_LAUNCH_CHECK("seq_embed_pair_kernel");
  return 0;
}

extern "C" int b2l_seq_hc_step(const void* y, float* X, const float* mix, const float* out_w, const float* in_next, const void* w_next,
                               void* h, float eps, const int* rows, int n_rows, int D, int streams, int act_dtype, b2l_stream_t stream) {
  B2L_CHECK_ARG(X != nullptr, "b2l_seq_hc_step: null pointer");
  B2L_CHECK_ARG((y == nullptr) == (mix == nullptr) && (y == nullptr) == (out_w == nullptr), "b2l_seq_hc_step: y, mix and out_w go together");
  B2L_CHECK_ARG((w_next == nullptr) == (h == nullptr) && (w_next == nullptr) == (in_next == nullptr),
                "b2l_seq_hc_step: in_next, w_next and h go together");
  B2L_CHECK_ARG(rows == nullptr || y == nullptr, "b2l_seq_hc_step: rows are picked only when nothing is written");
  B2L_CHECK_ARG(n_rows >= 0 && D > 0 && streams >= 1, "b2l_seq_hc_step: bad size");
  B2L_CHECK_SUPPORTED(streams <= HC_MAX_STREAMS, "b2l_seq_hc_step: %d streams, at most %d", streams, HC_MAX_STREAMS);
  if (n_rows == 0 || (y == nullptr && w_next == nullptr)) return 0;
  const size_t smem = w_next ? sizeof(float) * (size_t)D : 0;
  B2L_CHECK_SUPPORTED(smem <= 200 * 1024, "b2l_seq_hc_step: width %d too large", D);
  static DynSmemCache cache[2 * 9];
  cudaStream_t s_ = (cudaStream_t)stream;
#define B2L_HC_ARGS (const act_t*)y, X, mix, out_w, in_next, (const act_t*)w_next, (act_t*)h, eps, rows, D, streams
#define B2L_HC_LAUNCH(SV, slot)                                                                                   \
  do {                                                                                                            \
    const int rc_ = ensure_dyn_smem(seq_hc_step_kernel<act_t, SV>, smem, cache[(sizeof(act_t) == 2 ? 0 : 9) + slot]); \
    if (rc_ != 0) return rc_;                                                                                     \
    seq_hc_step_kernel<act_t, SV><<<n_rows, 256, smem, s_>>>(B2L_HC_ARGS);                                         \
  } while (0)
  B2L_SEQ_DISPATCH(act_dtype, {
    switch (streams) {          // the usual stream counts are compiled with their loops unrolled
      case 1: B2L_HC_LAUNCH(1, 0); break;
      case 2: B2L_HC_LAUNCH(2, 1); break;
      case 3: B2L_HC_LAUNCH(3, 2); break;
      case 4: B2L_HC_LAUNCH(4, 3); break;
      case 5: B2L_HC_LAUNCH(5, 4); break;
      case 6: B2L_HC_LAUNCH(6, 5); break;
      case 7: B2L_HC_LAUNCH(7, 6); break;
      case 8: B2L_HC_LAUNCH(8, 7); break;
      default: B2L_HC_LAUNCH(0, 8); break;     // more streams: loops with run-time bounds
    }
  });
#undef B2L_HC_LAUNCH
#undef B2L_HC_ARGS
  B2L_LAUNCH_CHECK("seq_hc_step_kernel");
  return 0;
}

extern "C" int b2l_seq_hc_sum(const float* X, float* out, int T, int D, int streams, b2l_stream_t stream) {
  B2L_CHECK_ARG(X && out && T >= 0 && D > 0 && streams >= 1, "b2l_seq_hc_sum: null pointer or bad size");
  if (T == 0) return 0;
  seq_hc_sum_kernel<<<T, 256, 0, (cudaStream_t)stream>>>(X, out, D, streams);
  B2L_LAUNCH_CHECK("seq_hc_sum_kernel");
  return 0;
}

extern "C" int b2l_seq_scale(float* z, size_t n, float mult, b2l_stream_t stream) {
  B2L_CHECK_ARG(z != nullptr, "b2l_seq_scale: null pointer");
  if (n == 0) return 0;
  const int grid = (int)((n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096);
  seq_scale_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(z, n, mult);
  B2L_LAUNCH_CHECK("seq_scale_kernel");
  return 0;
}

extern "C" int b2l_seq_qkv_prep(const b2l_seq_qkv_prep_args* a, b2l_stream_t stream) {
  B2L_CHECK_ARG(a != nullptr, "b2l_seq_qkv_prep: null argument block");
  B2L_CHECK_ARG(a->proj && a->meta && a->q_out && a->k_out, "b2l_seq_qkv_prep: null pointer");
  B2L_CHECK_ARG(a->T >= 0 && a->heads > 0 && a->kv_heads > 0 && a->K > 0 && a->V > 0, "b2l_seq_qkv_prep: bad size");
  B2L_CHECK_ARG(a->rot_dims >= 0 && a->rot_dims <= a->K && a->rot_dims % 2 == 0 && (a->rot_dims == 0 || a->freq), "b2l_seq_qkv_prep: bad rotation");
  B2L_CHECK_ARG((a->v_first == nullptr) || (a->v_out && a->lambda), "b2l_seq_qkv_prep: value mixing needs lambda and an output");
  B2L_CHECK_ARG(a->temp_every >= 0, "b2l_seq_qkv_prep: negative temperature step");
  B2L_CHECK_ARG(!a->unit_rms || (a->q_norm == nullptr && a->k_norm == nullptr), "b2l_seq_qkv_prep: the norm after the rotation has no weight");
  if (a->T == 0) return 0;
  const size_t es = a->act_dtype == B2L_F32 ? 4 : 2;
  // whole heads turn, in groups of four pairs, and no factor per head; both norms or none, so that both rows take the same form
  const bool table = a->rot_dims / 2 <= MOST_PAIRS;
  const int quads = table && (a->act_dtype == B2L_BF16 || a->act_dtype == B2L_F32) && a->rot_dims == a->K && a->K % 8 == 0 && !a->unit_rms && (a->whole_row || (!a->q_norm && !a->k_norm)) && a->q_off % 4 == 0 &&
                    a->k_off % 4 == 0 && a->ld % 4 == 0 && al4(a->proj, es) && al4(a->q_norm, es) && al4(a->k_norm, es) && al16(a->q_out) && al4(a->k_out, es);
  const long long units = (long long)(a->heads + a->kv_heads) * (a->K / 8);
  // Rows of more than 32768 entries do not fit a CTA's registers.  From 16384 on they take eight units a thread, at 128 registers with spills: faster where
  // few CTAs wait for one another's loads (us, registers / a pass per row: 17408 entries with norms, 1 token 12 / 23, 256 18 / 23, 2048 82 / 68; without, 16
  // tokens 10 / 14, 256 17 / 16, 2048 65 / 47; 32768 with norms, 2048 tokens 114 / 122).
  // In f32 a unit takes twice the registers: rows of up to 8192 entries.  us, a pass per row / so, 8 + 2 heads of 128 with norms: 1 token
  // 4.6 / 2.8, 777 6.6 / 3.8, 2048 12.5 / 8.1; 2048 of 48 + 8 64 / 40.
  const bool norms = a->q_norm || a->k_norm, held = a->act_dtype == B2L_F32 ? units <= 2 * QUAD_THREADS : units <= 4 * QUAD_THREADS || (units <= 8 * QUAD_THREADS && (a->T <= sm_count() * (norms ? 2 : 1) || (norms && units >= 7 * QUAD_THREADS)));
  if (quads && held) {
    // Tokens per CTA: one until the tokens' threads no longer fit the SMs at once (some 1000 an SM, two units each), then two, whose angles come together and the
    // second of which is on its way early; four only for rows of more than 768 units, of which an SM holds two CTAs.  As far as their angles fit, and two CTAs
    // an SM.  us by 1 / 2 / 4 tokens, heads of 128 with norms: 600 tokens of 16 + 4 heads 4.3 / 5.1 / 7.2, 1024 6.0 / 5.7 / 7.5, 2048 9.1 / 9.1 / 9.4; 1024 of 8 + 2
    // 4.0 / 4.9 / 6.7, 4096 10.2 / 9.9 / 10.3; 2048 of 32 + 8 15.1 / 14.1 / 16.2, of 40 + 8 20.2 / 18.6 / 18.0.
    const int fill = a->T / (2 * sm_count());
    const bool many = a->T * units > 2000LL * sm_count();
    const int tokens = a->K > 2048 || fill < 2 || !many ? 1 : units > 768 && fill >= 4 ? 4 : 2;
    // Units per thread: two, but one for the shortest rows and few tokens (160 units: 512 tokens 3.4 / 3.5, 600 3.8 / 3.6, 4096 11.2 / 9.9; 40: 3.9 / 4.2); four
    // from 384 on where tokens are many (480, 2048 tokens: 11.9 / 10.6; 320 9.1 / 10.0) and otherwise where they have to.
    const int nu = units <= 64 || (units <= QUAD_THREADS / 2 && a->T < 4 * sm_count()) ? 1 : units <= (many ? 384 : QUAD_THREADS) || a->act_dtype == B2L_F32 ? 2 : units <= 4 * QUAD_THREADS ? 4 : 8;
    const int threads = (int)((units + 32 * nu - 1) / (32 * nu)) * 32;
    auto kernel = nu == 1 ? seq_qkv_prep_quads_kernel<__nv_bfloat16, 1> : nu == 2 ? seq_qkv_prep_quads_kernel<__nv_bfloat16, 2>
                  : nu == 4 ? seq_qkv_prep_quads_kernel<__nv_bfloat16, 4> : seq_qkv_prep_quads_kernel<__nv_bfloat16, 8>;
    if (a->act_dtype == B2L_F32) kernel = nu == 1 ? seq_qkv_prep_quads_kernel<float, 1> : seq_qkv_prep_quads_kernel<float, 2>;
    kernel<<<(a->T + tokens - 1) / tokens, threads, sizeof(float) * a->K * tokens, (cudaStream_t)stream>>>(*a, tokens);
    B2L_LAUNCH_CHECK("seq_qkv_prep_quads_kernel");
    return 0;
  }
  B2L_SEQ_DISPATCH(a->act_dtype, {
    if (table) seq_qkv_prep_kernel<act_t, true><<<a->T, 256, sizeof(float) * a->rot_dims, (cudaStream_t)stream>>>(*a, quads);
    else seq_qkv_prep_kernel<act_t, false><<<a->T, 256, 0, (cudaStream_t)stream>>>(*a, quads);
  });
  B2L_LAUNCH_CHECK("seq_qkv_prep_kernel");
  return 0;
}
