// Linear recurrences with a matrix state per head (gated delta rule, gated linear attention, state-space duality)
// as ONE kernel: S <- diag(d) S; [u = sigmoid(beta)(v - S^T k)]; S <- S + k u^T; o = S^T q.
//
// A CTA owns one head and a tile of value columns; a column of S (K numbers) lives in the registers of R adjacent
// lanes (SCAN_KPT numbers each), so a step is R-lane shuffles and no shared-memory traffic for S.  The state is
// read once, carried through all T tokens of the portion and written once ([V][K] per head, K fastest, so the R
// lanes of a column read consecutive 16-byte words).  With `ones` the state has one column more whose value is 1 at every
// step (a normaliser: the decayed sum of the keys), kept and read out beside the others.  Inputs of SCAN_TC steps are staged in shared memory by the
// whole CTA with asynchronous copies, one stage ahead of the recurrence.  All arithmetic is f32.
#include <climits>
#include <type_traits>

#include "seq_common.cuh"

namespace b2l {

constexpr int SCAN_KPT = 16;       // state numbers per lane
constexpr int SCAN_TC = 16;        // steps per shared-memory stage
constexpr int SCAN_THREADS = 128;

__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Inputs of SCAN_TC steps go to shared memory with cp.async, two stages deep: stage s+1 is in flight while the
// recurrence runs over stage s, so the sequential loop never waits on global memory after the first stage.
// Stage layout: q[TC][KP] k[TC][KP] d[TC][DP] v[TC][cols] vs[TC] beta[TC] (+ 2*TC unused: stages stay 16-byte aligned).
// PASS 0: the recurrence with outputs, from the slot's state (one chunk) or from a chunk's start state in the workspace.
// PASS 1: a chunk's local end state from zero and its total decay, no outputs (first pass of a chunked portion).
// CPL: value columns per lane.  A step reads k, q and d from shared memory once per lane, so with one column the loop is
// bound by shared-memory bandwidth (12 16-byte reads for 48 FMAs); two columns halve that where throughput matters (long
// portions without the delta rule); one column keeps the most CTAs for single tokens and the latency-bound delta rule.
template <int DELTA, typename act_t, int PASS, int CPL>
__global__ void __launch_bounds__(SCAN_THREADS, DELTA ? 2 : 3) seq_scan_kernel(b2l_seq_scan_args a, int R, int vec, int chunk_len) {
  extern __shared__ __align__(16) float smem[];
  const int KP = R * SCAN_KPT;                 // padded key size
  const int ncg = SCAN_THREADS / R;            // column groups: lane cidx holds columns cidx + j * ncg
  const int cols = ncg * CPL;                  // value columns of this CTA
  const int DP = a.decay_per_channel ? KP : 4;
  const int stage = SCAN_TC * (2 * KP + DP + cols + 4);
  const int beta_at = SCAN_TC * (2 * KP + DP + cols + 1);
  float* so = smem + 2 * stage;                // [TC][cols]

  const int tid = threadIdx.x, r = tid % R, cidx = tid / R;
  const int h = blockIdx.y, hq = h / (a.heads / a.qk_heads);
  const int v0 = blockIdx.x * cols;
  const int K = a.K, V = a.V;
  const int slot = a.meta[0];
  const bool chunked = a.n_chunks > 1;
  const int t_begin = blockIdx.z * chunk_len, t_end = min(a.T, t_begin + chunk_len);
  float* st = chunked ? a.work_state + ((size_t)blockIdx.z * a.heads + h) * (size_t)(V + (a.ones ? 1 : 0)) * K
                      : a.state + ((size_t)slot * a.heads + h) * (size_t)V * K;
  float* st1 = chunked ? st + (size_t)V * K : (a.ones ? a.state_ones + ((size_t)slot * a.heads + h) * (size_t)K : nullptr);   // the column of ones
  const float skip = a.skip ? ld_act((const act_t*)a.skip, h) : 0.f;
  const float* gq = a.q + (size_t)hq * K;
  const float* gk = a.k + (size_t)hq * K;
  const float* gv = a.v + (size_t)h * V + v0;
  const float* gd = a.decay + (a.decay_per_channel ? (size_t)h * K : (size_t)h);
  const int VT = V + (a.ones ? 1 : 0);         // state columns
  const int ncol = min(cols, VT - v0);         // ... of this CTA
  const int nval = min(ncol, V - v0);          // ... of which values (the column of ones is the last of all)
  const bool warp_live = (tid & ~31) / R < ncol;   // a warp whose column groups all lie past the last column has nothing to compute

  // padding that no copy ever touches: q = k = 0 and d = 1 beyond K, v = 1 in the column of ones and 0 beyond it, vs = 1
  // without a value scale
  for (int b = 0; b < 2; ++b) {
    float* sq = smem + b * stage;
    float* sk = sq + SCAN_TC * KP;
    float* sd = sk + SCAN_TC * KP;
    float* sv = sd + SCAN_TC * DP;
    float* svs = sv + SCAN_TC * cols;
    for (int i = tid; i < SCAN_TC * KP; i += SCAN_THREADS) {
      if (i % KP >= K) {
        sq[i] = 0.f;
        sk[i] = 0.f;
        if (a.decay_per_channel) sd[i] = 1.f;
      }
    }
    for (int i = tid; i < SCAN_TC * cols; i += SCAN_THREADS)
      if (i % cols >= nval) sv[i] = i % cols < ncol ? 1.f : 0.f;
    if (tid < SCAN_TC) svs[tid] = 1.f;
  }

  auto prefetch = [&](int t0, int b) {
    const int nt = min(SCAN_TC, t_end - t0);
    float* sq = smem + b * stage;
    float* sk = sq + SCAN_TC * KP;
    float* sd = sk + SCAN_TC * KP;
    float* sv = sd + SCAN_TC * DP;
    float* svs = sv + SCAN_TC * cols;
    if (vec) {
      const int K4 = K >> 2;
      for (int i = tid; i < nt * K4; i += SCAN_THREADS) {
        const int t = i / K4, kk = (i - t * K4) << 2;
        cp_async16(sq + t * KP + kk, gq + (size_t)(t0 + t) * a.ldq + kk);
        cp_async16(sk + t * KP + kk, gk + (size_t)(t0 + t) * a.ldk + kk);
        if (a.decay_per_channel) cp_async16(sd + t * KP + kk, gd + (size_t)(t0 + t) * a.ldd + kk);
      }
    } else {
      for (int i = tid; i < nt * K; i += SCAN_THREADS) {
        const int t = i / K, kk = i - t * K;
        cp_async4(sq + t * KP + kk, gq + (size_t)(t0 + t) * a.ldq + kk);
        cp_async4(sk + t * KP + kk, gk + (size_t)(t0 + t) * a.ldk + kk);
        if (a.decay_per_channel) cp_async4(sd + t * KP + kk, gd + (size_t)(t0 + t) * a.ldd + kk);
      }
    }
    for (int i = tid; i < nt * nval; i += SCAN_THREADS) {
      const int t = i / nval, c = i - t * nval;
      cp_async4(sv + t * cols + c, gv + (size_t)(t0 + t) * a.ldv + c);
    }
    if (tid < nt) {
      if (!a.decay_per_channel) cp_async4(sd + tid, gd + (size_t)(t0 + tid) * a.ldd);
      if (a.vscale) cp_async4(svs + tid, a.vscale + (size_t)(t0 + tid) * a.ldvs + h);
    }
    cp_async_commit();
  };
  auto beta_of = [&](int t0) -> float {   // raw gate of step t0 + tid: act-typed, so a plain load kept in a register
    return (DELTA && tid < min(SCAN_TC, t_end - t0)) ? ld_act((const act_t*)a.beta, (size_t)(t0 + tid) * a.ldb + h) : 0.f;
  };

  float S[CPL][SCAN_KPT];
#pragma unroll
  for (int j = 0; j < CPL; ++j) {
    const int vcol = v0 + cidx + j * ncg;
#pragma unroll
    for (int i = 0; i < SCAN_KPT; ++i) {
      const int kk = ((i >> 2) * R + r) * 4 + (i & 3);
      S[j][i] = (PASS == 0 && kk < K && vcol < VT) ? (vcol < V ? st[(size_t)vcol * K + kk] : st1[kk]) : 0.f;
    }
  }
  float P[PASS ? SCAN_KPT : 1];       // PASS 1: the chunk's total decay of this lane's key channels
#pragma unroll
  for (int i = 0; i < (PASS ? SCAN_KPT : 1); ++i) P[i] = 1.f;

  __syncthreads();                    // the padding is written before any copy lands next to it
  prefetch(t_begin, 0);
  if (DELTA && tid < SCAN_TC) smem[beta_at + tid] = sigmoid_f(beta_of(t_begin));

  int b = 0;
  for (int t0 = t_begin; t0 < t_end; t0 += SCAN_TC, b ^= 1) {
    const int nt = min(SCAN_TC, t_end - t0);
    const bool more = t0 + SCAN_TC < t_end;
    float beta_next = 0.f;
    if (more) {
      prefetch(t0 + SCAN_TC, b ^ 1);
      beta_next = beta_of(t0 + SCAN_TC);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();                  // stage t0 has landed for every thread; so[] of the previous stage is written out
    const float* sq = smem + b * stage;
    const float* sk = sq + SCAN_TC * KP;
    const float* sd = sk + SCAN_TC * KP;
    const float* sv = sd + SCAN_TC * DP;
    const float* svs = sv + SCAN_TC * cols;
    const float* sb = svs + SCAN_TC;

#pragma unroll(DELTA ? 2 : 1)
    for (int t = 0; t < (warp_live ? nt : 0); ++t) {
      const float4* q4 = reinterpret_cast<const float4*>(sq + t * KP);
      const float4* k4 = reinterpret_cast<const float4*>(sk + t * KP);
      float kr[SCAN_KPT], qr[SCAN_KPT];
#pragma unroll
      for (int i4 = 0; i4 < SCAN_KPT / 4; ++i4) {
        const float4 kv = k4[i4 * R + r], qv = q4[i4 * R + r];
        kr[i4 * 4 + 0] = kv.x; kr[i4 * 4 + 1] = kv.y; kr[i4 * 4 + 2] = kv.z; kr[i4 * 4 + 3] = kv.w;
        qr[i4 * 4 + 0] = qv.x; qr[i4 * 4 + 1] = qv.y; qr[i4 * 4 + 2] = qv.z; qr[i4 * 4 + 3] = qv.w;
      }
      if (a.decay_per_channel) {
        const float4* d4 = reinterpret_cast<const float4*>(sd + t * KP);
#pragma unroll
        for (int i4 = 0; i4 < SCAN_KPT / 4; ++i4) {
          const float4 dv = d4[i4 * R + r];
#pragma unroll
          for (int j = 0; j < CPL; ++j) {
            S[j][i4 * 4 + 0] *= dv.x; S[j][i4 * 4 + 1] *= dv.y; S[j][i4 * 4 + 2] *= dv.z; S[j][i4 * 4 + 3] *= dv.w;
          }
          if (PASS) { P[i4 * 4 + 0] *= dv.x; P[i4 * 4 + 1] *= dv.y; P[i4 * 4 + 2] *= dv.z; P[i4 * 4 + 3] *= dv.w; }
        }
      } else {
        const float d = sd[t];
#pragma unroll
        for (int j = 0; j < CPL; ++j)
#pragma unroll
          for (int i = 0; i < SCAN_KPT; ++i) S[j][i] *= d;
        if (PASS) P[0] *= d;
      }
      float vraw[CPL], u[CPL], o[CPL];
#pragma unroll
      for (int j = 0; j < CPL; ++j) {
        vraw[j] = sv[t * cols + cidx + j * ncg];
        u[j] = vraw[j] * svs[t];
      }
      if (PASS) {
#pragma unroll
        for (int j = 0; j < CPL; ++j)
#pragma unroll
          for (int i = 0; i < SCAN_KPT; ++i) S[j][i] = fmaf(kr[i], u[j], S[j][i]);
        continue;
      }
      if (DELTA) {
        // With S' = diag(d) S:  u = beta (v - S'^T k)  and  o = (S' + k u^T)^T q = S'^T q + u (k.q): the dot products
        // over this lane's channels are reduced together, so a step has ONE shuffle chain on its critical path.
        float c0 = 0.f, c1 = 0.f;
#pragma unroll
        for (int i = 0; i < SCAN_KPT; i += 2) {
          c0 = fmaf(kr[i], qr[i], c0);
          c1 = fmaf(kr[i + 1], qr[i + 1], c1);
        }
        float kq = c0 + c1, p[CPL], oq[CPL];
#pragma unroll
        for (int j = 0; j < CPL; ++j) {
          float p0 = 0.f, p1 = 0.f, o0 = 0.f, o1 = 0.f;
#pragma unroll
          for (int i = 0; i < SCAN_KPT; i += 2) {
            p0 = fmaf(S[j][i], kr[i], p0); p1 = fmaf(S[j][i + 1], kr[i + 1], p1);
            o0 = fmaf(S[j][i], qr[i], o0); o1 = fmaf(S[j][i + 1], qr[i + 1], o1);
          }
          p[j] = p0 + p1;
          oq[j] = o0 + o1;
        }
        for (int w = 1; w < R; w <<= 1) {
          kq += __shfl_xor_sync(0xffffffffu, kq, w);
#pragma unroll
          for (int j = 0; j < CPL; ++j) {
            p[j] += __shfl_xor_sync(0xffffffffu, p[j], w);
            oq[j] += __shfl_xor_sync(0xffffffffu, oq[j], w);
          }
        }
#pragma unroll
        for (int j = 0; j < CPL; ++j) {
          u[j] = sb[t] * (u[j] - p[j]);
#pragma unroll
          for (int i = 0; i < SCAN_KPT; ++i) S[j][i] = fmaf(kr[i], u[j], S[j][i]);
          o[j] = fmaf(u[j], kq, oq[j]);
        }
      } else {
#pragma unroll
        for (int j = 0; j < CPL; ++j) {
          float o0 = 0.f, o1 = 0.f, o2 = 0.f, o3 = 0.f;
#pragma unroll
          for (int i = 0; i < SCAN_KPT; i += 4) {
            S[j][i] = fmaf(kr[i], u[j], S[j][i]); S[j][i + 1] = fmaf(kr[i + 1], u[j], S[j][i + 1]);
            S[j][i + 2] = fmaf(kr[i + 2], u[j], S[j][i + 2]); S[j][i + 3] = fmaf(kr[i + 3], u[j], S[j][i + 3]);
            o0 = fmaf(S[j][i], qr[i], o0); o1 = fmaf(S[j][i + 1], qr[i + 1], o1);
            o2 = fmaf(S[j][i + 2], qr[i + 2], o2); o3 = fmaf(S[j][i + 3], qr[i + 3], o3);
          }
          o[j] = (o0 + o1) + (o2 + o3);
        }
        for (int w = 1; w < R; w <<= 1) {
#pragma unroll
          for (int j = 0; j < CPL; ++j) o[j] += __shfl_xor_sync(0xffffffffu, o[j], w);
        }
      }
      if (r == 0) {
#pragma unroll
        for (int j = 0; j < CPL; ++j) so[t * cols + cidx + j * ncg] = o[j] * a.q_mult + skip * vraw[j];
      }
    }
    __syncthreads();
    if (PASS == 0) {
      for (int i = tid; i < nt * ncol; i += SCAN_THREADS) {
        const int t = i / ncol, c = i - t * ncol;
        if (c < nval) a.out[(size_t)(t0 + t) * a.ldo + (size_t)h * V + v0 + c] = so[t * cols + c];
        else a.out_ones[(size_t)(t0 + t) * a.heads + h] = so[t * cols + c];
      }
    }
    if (DELTA && more && tid < SCAN_TC) smem[(b ^ 1) * stage + beta_at + tid] = sigmoid_f(beta_next);
  }

  if (PASS == 0 && chunked) return;   // chunk outputs: the slot's state is written by the combine kernel
#pragma unroll
  for (int j = 0; j < CPL; ++j) {
    const int vcol = v0 + cidx + j * ncg;
#pragma unroll
    for (int i = 0; i < SCAN_KPT; ++i) {
      const int kk = ((i >> 2) * R + r) * 4 + (i & 3);
      if (kk < K && vcol < VT) (vcol < V ? st[(size_t)vcol * K + kk] : st1[kk]) = S[j][i];
    }
  }
  if (PASS && blockIdx.x == 0 && cidx == 0) {
    float* wd = a.work_decay + ((size_t)blockIdx.z * a.heads + h) * (a.decay_per_channel ? K : 1);
    if (a.decay_per_channel) {
#pragma unroll
      for (int i = 0; i < SCAN_KPT; ++i) {
        const int kk = ((i >> 2) * R + r) * 4 + (i & 3);
        if (kk < K) wd[kk] = P[i];
      }
    } else if (r == 0) {
      wd[0] = P[0];
    }
  }
}

// Between the passes of a chunked portion: work_state[c] (a chunk's local end state) becomes the chunk's START state,
// s_0 = the slot's state, s_(c+1) = D_c s_c + local_c, and the slot's state becomes s_n.  One thread per state entry.
__global__ void seq_scan_combine_kernel(b2l_seq_scan_args a) {
  const size_t per_head = (size_t)(a.V + (a.ones ? 1 : 0)) * a.K, n = (size_t)a.heads * per_head, n_val = (size_t)a.V * a.K;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int h = (int)(i / per_head), kk = (int)(i % a.K);
  const size_t in_head = i % per_head;
  float* st = in_head < n_val ? a.state + ((size_t)a.meta[0] * a.heads + h) * n_val + in_head
                              : a.state_ones + ((size_t)a.meta[0] * a.heads + h) * a.K + (in_head - n_val);
  float s = *st;
  const size_t dstep = (size_t)a.heads * (a.decay_per_channel ? a.K : 1);
  const float* dp = a.work_decay + (size_t)h * (a.decay_per_channel ? a.K : 1) + (a.decay_per_channel ? kk : 0);
  for (int c0 = 0; c0 < a.n_chunks; c0 += 8) {        // eight chunks' operands are requested together
    float d[8], local[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const bool in = c0 + u < a.n_chunks;
      d[u] = in ? dp[(size_t)(c0 + u) * dstep] : 1.f;
      local[u] = in ? a.work_state[(size_t)(c0 + u) * n + i] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (c0 + u < a.n_chunks) a.work_state[(size_t)(c0 + u) * n + i] = s;
      s = fmaf(d[u], s, local[u]);
    }
  }
  *st = s;
}

// ---- a portion 16 tokens at a time.  With G_t the product of the decays of a chunk's tokens up to t (per channel) and D_(t,i) that of the
// tokens after i up to t, S_0 the state before the chunk, B[t,i] = q_t . D_(t,i) k_i for i <= t, R_t = S_0^T (G_t q_t):
//   without the delta rule:  u_i = vscale_i v_i;  o = R + B u
//   delta rule:  P_t = S_0^T (G_t k_t);  u = T (v - P),  T = (I + diag(beta) A)^-1 diag(beta),  A[t,i] = k_t . D_(t,i) k_i for i < t;
//                o = R + (B T) (v - P)
//   S_16 = G_16 S_0 + sum_i (D_(16,i) k_i) u_i^T
// Decays only ever multiply (no quotient of cumulative products, which overflows where a channel forgets fast).  T is the product of the
// chunk's transition matrices seen from k: its entries stay below 1 for unit keys.  Long portions with 128 keys take the form on the tensor cores
// (seq_scan_mma.cuh); here all is f32 on the CUDA cores, like the step-by-step form.
//   seq_chunk_kernel  a CTA per (chunk, head): T and B T (or B), 16 x 16 each, into the workspace; all chunks in parallel
//   seq_walk_kernel   a CTA per (head, VT = 16 or 8 value columns) walks the chunks: warps 4..11 (a thread per key channel, the two groups on
//                     alternate chunks) load and form G k, G q, D k a chunk ahead, while warps 0..3 run P / R (K split over the warps),
//                     u / o and the state update in 4 x 4 tiles
// What bounds it: the walk over T / 16 chunks, 832 FMA cycles per chunk (delta rule) and four barriers.  The step-by-step kernel spends 0.38 us
// per token on one dependent chain of FMAs and shuffles, whatever the width (16 heads of 128 x 128, 2048 tokens: 780 us).
// With 8 columns per CTA, where the chip has SMs for twice the CTAs, a chunk's products halve (8 heads of 128 x 128, 2048 tokens, us with 16 / 8
// columns: 171 / 128 without the delta rule, 211 / 163 with it); with more CTAs than SMs two would share an SM's shared-memory reads, which bound it.
constexpr int CH_C = 16, CH_VT = 16, CH_NARROW = 8, CH_MAT = CH_C * CH_C;      // tokens per chunk, value columns per CTA

// v[0..7] of every lane summed over the warp: lane l holds sum number ((l >> 4) & 1) * 4 + ((l >> 3) & 1) * 2 + ((l >> 2) & 1)
__device__ __forceinline__ float warp_sum8(float (&v)[8], int lane) {
#pragma unroll
  for (int half = 4, w = 16; half >= 1; half >>= 1, w >>= 1) {
    const bool up = lane & w;
#pragma unroll
    for (int j = 0; j < half; ++j) {
      const float send = up ? v[j] : v[j + half], keep = up ? v[j + half] : v[j];
      v[j] = keep + __shfl_xor_sync(0xffffffffu, send, w);
    }
  }
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// Two warps: warp 0 the columns 0..3 and 12..15 of A and B, warp 1 the columns 4..11 (20 rows of four columns each).  A row of k, q and decays is
// read from shared memory once for four columns: with a column at a time those reads were what bounded the kernel (1632 warp reads a chunk, 480 so),
// 16 heads of 128 x 128, 2048 tokens: 34 us then.
constexpr int CHUNK_THREADS = 64;
template <typename act_t, int K, bool DELTA>
__global__ void __launch_bounds__(CHUNK_THREADS) seq_chunk_kernel(b2l_seq_scan_args a, int vec) {
  __shared__ __align__(16) float sk[CH_C][K], sq[CH_C][K], sg[CH_C][K];
  __shared__ float sA[CH_C][CH_C + 1], sB[CH_C][CH_C + 1], sbeta[CH_C];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, chunk = blockIdx.x, h = blockIdx.y, hq = h / (a.heads / a.qk_heads);
  const int t0 = chunk * CH_C, nt = min(CH_C, a.T - t0);
  const float* gk = a.k + (size_t)t0 * a.ldk + (size_t)hq * K;
  const float* gq = a.q + (size_t)t0 * a.ldq + (size_t)hq * K;
  const float* gd = a.decay + (size_t)t0 * a.ldd + (a.decay_per_channel ? (size_t)h * K : (size_t)h);
  if (vec) {
#pragma unroll 4
    for (int i = tid; i < CH_C * K / 4; i += CHUNK_THREADS) {
      const int t = i / (K / 4), c = (i - t * (K / 4)) * 4;
      if (t < nt) {
        cp_async16(&sk[t][c], gk + (size_t)t * a.ldk + c);
        cp_async16(&sq[t][c], gq + (size_t)t * a.ldq + c);
        if (a.decay_per_channel) cp_async16(&sg[t][c], gd + (size_t)t * a.ldd + c);
      } else {
        *reinterpret_cast<float4*>(&sk[t][c]) = *reinterpret_cast<float4*>(&sq[t][c]) = make_float4(0.f, 0.f, 0.f, 0.f);
        if (a.decay_per_channel) *reinterpret_cast<float4*>(&sg[t][c]) = make_float4(1.f, 1.f, 1.f, 1.f);
      }
    }
    cp_async_commit();
  } else {
    for (int i = tid; i < CH_C * K; i += CHUNK_THREADS) {
      const int t = i / K, c = i - t * K;
      const bool in = t < nt;
      sk[t][c] = in ? gk[(size_t)t * a.ldk + c] : 0.f;
      sq[t][c] = in ? gq[(size_t)t * a.ldq + c] : 0.f;
      if (a.decay_per_channel) sg[t][c] = in ? gd[(size_t)t * a.ldd + c] : 1.f;
    }
  }
  if (!a.decay_per_channel)
    for (int i = tid; i < CH_C * K; i += CHUNK_THREADS) {
      const int t = i / K;
      sg[t][i - t * K] = t < nt ? gd[(size_t)t * a.ldd] : 1.f;
    }
  if (DELTA && tid < CH_C) sbeta[tid] = tid < nt ? sigmoid_f(ld_act((const act_t*)a.beta, (size_t)(t0 + tid) * a.ldb + h)) : 0.f;
  cp_async_wait<0>();
  __syncthreads();
  // the eight sums of row t: k_t and q_t with the decayed keys of columns i0 .. i0 + 3
  const int col = ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
  auto put = [&](float (&p)[8], int t, int i0) {
    const float v = warp_sum8(p, lane);
    if ((lane & 3) == 0) {
      if (lane & 16) sB[t][i0 + col] = v;
      else if (DELTA) sA[t][i0 + col] = v;
    }
  };
#pragma unroll 1
  for (int n = 0; n < 2; ++n) {
    const int i0 = 4 * (warp ? 1 + n : 3 * n);
    float x[4][K / 32];
#pragma unroll
    for (int r = 0; r < 4; ++r) {                      // rows of the diagonal's 4 x 4
      const int t = i0 + r;
      float p[8] = {};
#pragma unroll
      for (int e = 0; e < K / 32; ++e) {
        const float kv = sk[t][lane + 32 * e], qv = sq[t][lane + 32 * e], gv = sg[t][lane + 32 * e];
#pragma unroll
        for (int c = 0; c < r; ++c) {
          x[c][e] *= gv;
          if (DELTA) p[c] = fmaf(kv, x[c][e], p[c]);
          p[4 + c] = fmaf(qv, x[c][e], p[4 + c]);
        }
        x[r][e] = kv;
        p[4 + r] = fmaf(qv, kv, p[4 + r]);
      }
      put(p, t, i0);
    }
#pragma unroll 2
    for (int t = i0 + 4; t < CH_C; ++t) {
      float p[8] = {};
#pragma unroll
      for (int e = 0; e < K / 32; ++e) {
        const float kv = sk[t][lane + 32 * e], qv = sq[t][lane + 32 * e], gv = sg[t][lane + 32 * e];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          x[c][e] *= gv;
          if (DELTA) p[c] = fmaf(kv, x[c][e], p[c]);
          p[4 + c] = fmaf(qv, x[c][e], p[4 + c]);
        }
      }
      put(p, t, i0);
    }
  }
  __syncthreads();
  float* out = a.work_state + ((size_t)chunk * a.heads + h) * (2 * CH_MAT);
  if (!DELTA) {
    for (int e = tid; e < CH_MAT; e += CHUNK_THREADS) out[CH_MAT + e] = e % CH_C <= e / CH_C ? sB[e / CH_C][e % CH_C] : 0.f;
    return;
  }
  if (warp) return;
  const int j = lane & (CH_C - 1), half = lane >> 4;   // column j of T by forward substitution, in both halves of the warp; B T: a half the even rows, the other the odd ones
  float c[CH_C];
#pragma unroll
  for (int t = 0; t < CH_C; ++t) {
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int i = 0; i < t; ++i) {
      if (i & 1) s1 = fmaf(sA[t][i], c[i], s1);
      else s0 = fmaf(sA[t][i], c[i], s0);
    }
    c[t] = t < j ? 0.f : (t == j ? sbeta[t] : -sbeta[t] * (s0 + s1));
    if ((t & 1) == half) out[t * CH_C + j] = c[t];
  }
#pragma unroll
  for (int s = 0; s < CH_C; s += 2) {
    const int t = s + half;
    float m = 0.f;
#pragma unroll
    for (int i = 0; i <= s + 1; ++i)
      if (i >= j && i <= t) m = fmaf(sB[t][i], c[i], m);          // the rest is zero times a token that t has not seen, which may be infinite
    out[CH_MAT + t * CH_C + j] = m;
  }
}

template <int K, bool DELTA, int VT>
struct WalkStage {
  static constexpr int ROWS = DELTA ? 32 : 16, LD = ROWS + 4;      // padded: 16-byte rows of a channel on distinct banks
  float kq[K][LD];                 // [channel][(delta: 16 tokens of G k) | 16 of G q | padding]
  float kd[CH_C][K];               // D k
  float tm[ROWS][CH_C];            // (T over) B T, or B
  float v[CH_C][VT], u[CH_C][VT];            // values, and (no delta rule) values times vscale
  float gc[K];                     // G of the whole chunk
};
template <int K, bool DELTA, int VT>
struct WalkSmem {
  WalkStage<K, DELTA, VT> st[2];
  float S[K][VT];
  float part[64 / VT][WalkStage<K, DELTA, VT>::ROWS][VT + 4];
  float w[CH_C][VT], u[CH_C][VT];
};
__device__ __forceinline__ void walk_bar() { asm volatile("bar.sync 1, 128;" ::: "memory"); }
__device__ __forceinline__ void fma4(float4& d, float s, const float4& v) {
  d.x = fmaf(s, v.x, d.x); d.y = fmaf(s, v.y, d.y); d.z = fmaf(s, v.z, d.z); d.w = fmaf(s, v.w, d.w);
}
template <int N> struct alignas(4 * N) Cols {           // neighbouring value columns of a thread
  float v[N];
  __device__ __forceinline__ void fma(float s, const Cols& o) {
#pragma unroll
    for (int e = 0; e < N; ++e) v[e] = fmaf(s, o.v[e], v[e]);
  }
};

template <typename act_t, int K, bool DELTA, int VT>
__global__ void __launch_bounds__(384) seq_walk_kernel(b2l_seq_scan_args a) {
  extern __shared__ __align__(16) unsigned char walk_raw[];
  using Stage = WalkStage<K, DELTA, VT>;
  constexpr int VW = VT / 4;                           // columns per thread of the walk, but in its product P / R
  using Vec = Cols<VW>;
  WalkSmem<K, DELTA, VT>& sm = *reinterpret_cast<WalkSmem<K, DELTA, VT>*>(walk_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = blockIdx.y, hq = h / (a.heads / a.qk_heads), v0 = blockIdx.x * VT;
  const int n_chunks = (a.T + CH_C - 1) / CH_C;
  float* st = a.state + ((size_t)a.meta[0] * a.heads + h) * (size_t)a.V * K;

  if (warp >= 4) {
    // ===================== operands: warps 4..7 the even chunks, 8..11 the odd ones =====================
    const int par = warp >= 8, c = tid - 128 - 128 * par;
    const bool chan = c < K;
    float k[CH_C], q[CH_C], g[CH_C], v[VT / 8], vs[VT / 8], G = 1.f;
    float4 tm;
    auto load = [&](int n) {
      if (n >= n_chunks) return;
      const int t0 = n * CH_C, nt = min(CH_C, a.T - t0);
      if (c < Stage::ROWS * CH_C / 4)
        tm = reinterpret_cast<const float4*>(a.work_state + ((size_t)n * a.heads + h) * (2 * CH_MAT) + (DELTA ? 0 : CH_MAT))[c];
#pragma unroll
      for (int i = 0; i < VT / 8; ++i) {
        const int t = c / VT + 8 * i, e = c % VT;
        v[i] = t < nt ? a.v[(size_t)(t0 + t) * a.ldv + (size_t)h * a.V + v0 + e] : 0.f;
        vs[i] = (!DELTA && a.vscale && t < nt) ? a.vscale[(size_t)(t0 + t) * a.ldvs + h] : 1.f;
      }
      if (!chan) return;
      const float* pg = a.decay + (size_t)t0 * a.ldd + (a.decay_per_channel ? (size_t)h * K + c : (size_t)h);
      const float* pk = a.k + (size_t)t0 * a.ldk + (size_t)hq * K + c;
      const float* pq = a.q + (size_t)t0 * a.ldq + (size_t)hq * K + c;
      if (nt == CH_C) {
#pragma unroll
        for (int t = 0; t < CH_C; ++t, pg += a.ldd, pk += a.ldk, pq += a.ldq) { g[t] = *pg; k[t] = *pk; q[t] = *pq; }
      } else {
#pragma unroll
        for (int t = 0; t < CH_C; ++t, pg += a.ldd, pk += a.ldk, pq += a.ldq) {
          const bool in = t < nt;
          g[t] = in ? *pg : 1.f;
          k[t] = in ? *pk : 0.f;
          q[t] = in ? *pq : 0.f;
        }
      }
    };
    float kd[CH_C];
    auto form = [&](int n) {                           // in registers: the stage's buffer is still in use
      if (n >= n_chunks || !chan) return;
      float d = 1.f;
#pragma unroll
      for (int t = CH_C - 1; t >= 0; --t) {
        kd[t] = d * k[t];
        d *= g[t];
      }
      G = 1.f;
#pragma unroll
      for (int t = 0; t < CH_C; ++t) {
        G *= g[t];
        k[t] *= G;
        q[t] *= G;
      }
    };
    auto store = [&](int n) {
      if (n >= n_chunks) return;
      Stage& s = sm.st[n & 1];
      if (c < Stage::ROWS * CH_C / 4) reinterpret_cast<float4*>(&s.tm[0][0])[c] = tm;
#pragma unroll
      for (int i = 0; i < VT / 8; ++i) {
        const int t = c / VT + 8 * i, e = c % VT;
        s.v[t][e] = v[i];
        if (!DELTA) s.u[t][e] = v[i] * vs[i];
      }
      if (!chan) return;
      s.gc[c] = G;
#pragma unroll
      for (int t = 0; t < CH_C; ++t) s.kd[t][c] = kd[t];
#pragma unroll
      for (int t = 0; t < CH_C; t += 4) {
        if (DELTA) *reinterpret_cast<float4*>(&s.kq[c][t]) = make_float4(k[t], k[t + 1], k[t + 2], k[t + 3]);
        *reinterpret_cast<float4*>(&s.kq[c][Stage::ROWS - CH_C + t]) = make_float4(q[t], q[t + 1], q[t + 2], q[t + 3]);
      }
    };
    load(par);
    form(par);
    if (par == 0) {
      store(0);
      load(2);
    }
    __syncthreads();
    for (int n = 0; n < n_chunks; ++n) {
      if (((n + 1) & 1) == par) {
        store(n + 1);
        load(n + 3);
      } else {
        form(n + 2);
      }
      __syncthreads();
    }
    return;
  }
  // ===================== the walk =====================
  const int cg = tid >> 2, vg = tid & 3;               // channels 4 cg .. + 3 (K = 64: half of the threads), columns VW vg .. + VW - 1
  const bool own = cg < K / 4;
  const float skip = a.skip ? ld_act((const act_t*)a.skip, h) : 0.f;
  auto at = [&](auto& row) -> Vec& { return *reinterpret_cast<Vec*>(&row[VW * vg]); };            // this thread's columns of a row in shared memory
  auto of = [&](const auto& row) -> const Vec& { return *reinterpret_cast<const Vec*>(&row[VW * vg]); };
  Vec S[4];                                            // S[j]: channel 4 cg + j
  if (own) {
#pragma unroll
    for (int e = 0; e < VW; ++e) {
      const float4 c = *reinterpret_cast<const float4*>(st + (size_t)(v0 + VW * vg + e) * K + 4 * cg);
      S[0].v[e] = c.x; S[1].v[e] = c.y; S[2].v[e] = c.z; S[3].v[e] = c.w;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) at(sm.S[4 * cg + j]) = S[j];
  }
  __syncthreads();
  for (int n = 0; n < n_chunks; ++n) {
    const Stage& s = sm.st[n & 1];
    constexpr int RT = Stage::ROWS / 8;                // rows per lane
    // (P and) R in tiles of RT rows x 4 columns: a quarter of the channels per warp, with 8 columns an eighth per half warp
    constexpr int SLICES = 64 / VT;
    const int slice = VT == 16 ? warp : 2 * warp + (lane >> 4), tg = VT == 16 ? lane >> 2 : (lane >> 1) & 7, c4 = 4 * (VT == 16 ? vg : lane & 1);
    float4 acc[RT] = {};
#pragma unroll 8
    for (int c = slice * (K / SLICES); c < (slice + 1) * (K / SLICES); ++c) {
      const float4 y = *reinterpret_cast<const float4*>(&sm.S[c][c4]);
      if (DELTA) {
        const float4 x = *reinterpret_cast<const float4*>(&s.kq[c][4 * tg]);
        fma4(acc[0], x.x, y); fma4(acc[1], x.y, y); fma4(acc[RT - 2], x.z, y); fma4(acc[RT - 1], x.w, y);
      } else {
        const float2 x = *reinterpret_cast<const float2*>(&s.kq[c][2 * tg]);
        fma4(acc[0], x.x, y); fma4(acc[1], x.y, y);
      }
    }
#pragma unroll
    for (int j = 0; j < RT; ++j) *reinterpret_cast<float4*>(&sm.part[slice][RT * tg + j][c4]) = acc[j];
    walk_bar();
    // row cg: v - P, or R
    Vec r = {};
    if (cg < Stage::ROWS) {
#pragma unroll
      for (int w = 0; w < SLICES; ++w) {
        const Vec p = of(sm.part[w][cg]);
#pragma unroll
        for (int e = 0; e < VW; ++e) r.v[e] += p.v[e];
      }
    }
    if (DELTA) {
      if (cg < CH_C) {
        const Vec v = of(s.v[cg]);
#pragma unroll
        for (int e = 0; e < VW; ++e) r.v[e] = v.v[e] - r.v[e];
        at(sm.w[cg]) = r;
        r = Vec{};
      }
      walk_bar();
    }
    const float (*in)[VT] = DELTA ? sm.w : s.u;
    if (cg < Stage::ROWS) {
      const int tt = cg & (CH_C - 1);                  // tokens up to this row's: a zero weight would turn a later token's infinity into NaN
#pragma unroll
      for (int i = 0; i < CH_C; i += 4) {
        const float4 m = *reinterpret_cast<const float4*>(&s.tm[cg][i]);
        if (i <= tt) r.fma(m.x, of(in[i]));
        if (i + 1 <= tt) r.fma(m.y, of(in[i + 1]));
        if (i + 2 <= tt) r.fma(m.z, of(in[i + 2]));
        if (i + 3 <= tt) r.fma(m.w, of(in[i + 3]));
      }
      if (DELTA && cg < CH_C) {
        at(sm.u[cg]) = r;
      } else {
        const int t = n * CH_C + tt;
        if (t < a.T) {
          const Vec v = of(s.v[tt]);
          float* o = a.out + (size_t)t * a.ldo + (size_t)h * a.V + v0 + VW * vg;
#pragma unroll
          for (int e = 0; e < VW; ++e) o[e] = r.v[e] * a.q_mult + skip * v.v[e];
        }
      }
    }
    if (DELTA) walk_bar();
    const float (*add)[VT] = DELTA ? sm.u : s.u;
    if (own) {
      const float4 g = *reinterpret_cast<const float4*>(&s.gc[4 * cg]);
      const float gj[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < VW; ++e) S[j].v[e] *= gj[j];
#pragma unroll 8
      for (int i = 0; i < CH_C; ++i) {
        const float4 x = *reinterpret_cast<const float4*>(&s.kd[i][4 * cg]);
        const Vec y = of(add[i]);
        S[0].fma(x.x, y); S[1].fma(x.y, y); S[2].fma(x.z, y); S[3].fma(x.w, y);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) at(sm.S[4 * cg + j]) = S[j];
    }
    __syncthreads();                                   // the next chunk's operands and the state are in place
  }
  if (own) {
#pragma unroll
    for (int e = 0; e < VW; ++e)
      *reinterpret_cast<float4*>(st + (size_t)(v0 + VW * vg + e) * K + 4 * cg) = make_float4(S[0].v[e], S[1].v[e], S[2].v[e], S[3].v[e]);
  }
}

}  // namespace b2l

#include "seq_scan_mma.cuh"

namespace b2l {

constexpr int SCAN_CHUNK = 128;      // tokens per chunk of a chunked portion (a multiple of SCAN_TC)

static bool walk_sizes(int T, int K, int V, int ones) { return T >= 2 * CH_C && (K == 64 || K == 128) && V % CH_VT == 0 && !ones; }
// Where the walk is the faster form.  Against the step-by-step form (0.35 us per token): from 48 tokens on where every CTA of the walk has an SM
// of its own (16 heads of 128 x 128, 48 tokens: 20..26 against 27..29 us; 32 tokens: 17..24 against 21..23), from 64 on otherwise (64 heads of
// 64 x 64, 33 tokens: 26..30 against 21..23; 64 tokens: 28..32 against 35..39).  Against the chunked form without the delta rule, which
// stays flat until its CTAs fill the SMs while the walk takes 1.3 us (1.0 with 64 keys) per 16 tokens and turn of CTAs whatever the heads:
// both times from the fits below, in ns (128 x 128, us walk with 16 columns per CTA / chunked: 1024 tokens of 4 heads 95 / 103; 2048 of 4 173 / 130,
// of 8 179 / 240; 4096 of 4 333 / 251, of 8 345 / 388; 8192 of 1 634 / 134, of 8 673 / 667, of 16 710 / 1285; walk with 8 columns: 512 tokens of 4
// and 8 43, 2048 of 4 124, of 8 128; with 64 keys 512 tokens 38, 1024 of 18 63).  The fits are the FMA walk's also where the tensor cores walk (2048 and 4096 tokens of 4
// heads 84 and 162): those portions still go in chunks, 130 and 240 us, until the rule weighs that walk by its own times.
static bool walk_narrow(int heads, int V) { return (long long)heads * (V / CH_NARROW) <= sm_count(); }
static bool walk_pays(int T, int heads, int K, int V, int delta) {
  const long long sms = sm_count(), ctas = (long long)heads * (V / CH_VT), turns = (ctas + sms - 1) / sms;
  if (T < (turns <= 1 ? 48 : 64)) return false;
  if (delta || T < 2 * SCAN_CHUNK) return true;
  const long long cols = K == 64 ? 64 : 32, chunked = (V + cols - 1) / cols * heads * ((T + SCAN_CHUNK - 1) / SCAN_CHUNK), load = (chunked + sms - 1) / sms;
  const long long t_chunked = load == 1 ? 104000 : load == 2 ? 131000 : 60000 + 45000 * load, t_walk = 15000 + (long long)(T / CH_C) * (walk_narrow(heads, V) ? (K == 64 ? 800 : 920) : (K == 64 ? 1050 : 1350)) * turns;
  return t_walk <= t_chunked;
}
// Portions of two chunks or more with key sizes 64 or 128 and whole groups of 16 values, given room for the chunks' matrices (or operands); other sizes, the
// column of ones and single tokens go step by step.  A caller that asks for the chunked form gets a walk where it is faster and its space suffices.
static long long walk_floats(int T, int heads) { return (long long)((T + CH_C - 1) / CH_C) * heads * (2 * CH_MAT); }
enum { WALK_NONE, WALK_FMA, WALK_MMA };
static int walk_form(const b2l_seq_scan_args* a, long long room) {      // room: floats of work_state
  if (a->work_state == nullptr || !walk_sizes(a->T, a->K, a->V, a->ones) || (a->delta && (!a->decay_per_channel || a->vscale)) || ((uintptr_t)a->state & 15) != 0 ||
      ((uintptr_t)a->work_state & 15) != 0 || a->heads > 65535)
    return WALK_NONE;
  if (a->n_chunks > 1 && !walk_pays(a->T, a->heads, a->K, a->V, a->delta)) return WALK_NONE;
  if (mma_walk(a->T, a->heads, a->K, a->V, a->delta) && mma_walk_floats(a->T, a->heads, a->qk_heads, a->K, a->V, a->delta, a->decay_per_channel) <= room) return WALK_MMA;
  return walk_floats(a->T, a->heads) <= room ? WALK_FMA : WALK_NONE;
}

template <typename act_t, int K, bool DELTA>
static int launch_walk(const b2l_seq_scan_args* a, cudaStream_t s) {
  auto al = [](const void* p) { return ((uintptr_t)p & 15) == 0; };
  const int vec = a->ldq % 4 == 0 && a->ldk % 4 == 0 && al(a->q) && al(a->k) && (!a->decay_per_channel || (a->ldd % 4 == 0 && al(a->decay)));
  seq_chunk_kernel<act_t, K, DELTA><<<dim3((unsigned)((a->T + CH_C - 1) / CH_C), (unsigned)a->heads), CHUNK_THREADS, 0, s>>>(*a, vec);
  B2L_LAUNCH_CHECK("seq_chunk_kernel");
  auto walk = [&](auto vt) {
    constexpr int VT = decltype(vt)::value;
    static DynSmemCache cache;
    if (int rc = ensure_dyn_smem(seq_walk_kernel<act_t, K, DELTA, VT>, sizeof(WalkSmem<K, DELTA, VT>), cache)) return rc;
    seq_walk_kernel<act_t, K, DELTA, VT><<<dim3((unsigned)(a->V / VT), (unsigned)a->heads), 384, sizeof(WalkSmem<K, DELTA, VT>), s>>>(*a);
    B2L_LAUNCH_CHECK("seq_walk_kernel");
    return 0;
  };
  return walk_narrow(a->heads, a->V) ? walk(std::integral_constant<int, CH_NARROW>{}) : walk(std::integral_constant<int, CH_VT>{});
}

static DynSmemCache g_scan_smem[10];

}  // namespace b2l

using namespace b2l;

extern "C" int b2l_seq_scan_chunks(int T, int delta) {
  if (delta || T < 2 * SCAN_CHUNK) return 1;
  return (T + SCAN_CHUNK - 1) / SCAN_CHUNK;
}

extern "C" long long b2l_seq_scan_work_floats(int T, int heads) {
  if (T < 2 * CH_C || heads <= 0) return 0;
  const long long fma = walk_floats(T, heads), mma = T >= MW_LEAST && heads <= MW_HEADS ? mma_walk_most_floats(T, heads) : 0;
  return fma > mma ? fma : mma;                        // for either, whatever the key size
}

static bool plan_walks(int T, int heads, int K, int V, int per_channel, int delta, int ones, int vscale) {
  return walk_sizes(T, K, V, ones) && (!delta || (per_channel && !vscale)) && heads <= 65535 && walk_pays(T, heads, K, V, delta);
}
static long long plan_chunks(int T, int heads, int K, int V, int delta, int ones, int* n_chunks) {
  const int n = b2l_seq_scan_chunks(T, delta);
  if (n_chunks) *n_chunks = n;
  return n > 1 ? (long long)n * heads * (V + (ones ? 1 : 0)) * K : 0;
}

extern "C" long long b2l_seq_scan_plan(int T, int heads, int K, int V, int per_channel, int delta, int ones, int vscale, int* n_chunks) {
  if (n_chunks) *n_chunks = 1;
  if (T <= 0 || heads <= 0 || K <= 0 || V <= 0) return 0;
  if (plan_walks(T, heads, K, V, per_channel, delta, ones, vscale)) return b2l_seq_scan_work_floats(T, heads);
  return plan_chunks(T, heads, K, V, delta, ones, n_chunks);
}

extern "C" long long b2l_seq_scan_space(int T, int heads, int qk_heads, int K, int V, int per_channel, int delta, int ones, int vscale, int* n_chunks, long long* least) {
  if (n_chunks) *n_chunks = 1;
  if (least) *least = 0;
  if (T <= 0 || heads <= 0 || qk_heads <= 0 || K <= 0 || V <= 0) return 0;
  if (!plan_walks(T, heads, K, V, per_channel, delta, ones, vscale)) return plan_chunks(T, heads, K, V, delta, ones, n_chunks);
  const long long fma = walk_floats(T, heads);
  if (!mma_walk(T, heads, K, V, delta)) return fma;
  const long long mma = mma_walk_floats(T, heads, qk_heads, K, V, delta, per_channel);
  if (least && fma < mma) *least = fma;
  return mma;
}

static int scan(const b2l_seq_scan_args* a, long long room, b2l_stream_t stream) {
  B2L_CHECK_ARG(a != nullptr, "b2l_seq_scan: null argument block");
  B2L_CHECK_ARG(a->q && a->k && a->v && a->decay && a->state && a->meta && a->out, "b2l_seq_scan: null pointer");
  B2L_CHECK_ARG(!a->delta || a->beta, "b2l_seq_scan: the delta rule needs beta");
  B2L_CHECK_ARG(a->T >= 0 && a->heads > 0 && a->qk_heads > 0 && a->K > 0 && a->V > 0, "b2l_seq_scan: bad size");
  B2L_CHECK_ARG(a->heads % a->qk_heads == 0, "b2l_seq_scan: heads %d not a multiple of qk_heads %d", a->heads, a->qk_heads);
  B2L_CHECK_SUPPORTED(a->K <= 32 * SCAN_KPT, "b2l_seq_scan: key size %d above %d", a->K, 32 * SCAN_KPT);
  B2L_CHECK_ARG(a->n_chunks <= 1 || (!a->delta && a->work_state && a->work_decay && a->n_chunks == (a->T + SCAN_CHUNK - 1) / SCAN_CHUNK),
                "b2l_seq_scan: chunked portions need the workspace, no delta rule and n_chunks from b2l_seq_scan_chunks");
  B2L_CHECK_ARG(!a->ones || (a->state_ones && a->out_ones && !a->skip && !a->delta), "b2l_seq_scan: the column of ones needs its state and its output, no skip and no delta rule");
  if (a->T == 0) return 0;
  const int form = walk_form(a, room);
  if (form != WALK_NONE && (a->act_dtype == B2L_BF16 || a->act_dtype == B2L_F32)) {
    cudaStream_t st = (cudaStream_t)stream;
    B2L_SEQ_DISPATCH(a->act_dtype, {
      if (form == WALK_MMA) {
        if (a->delta) return launch_mma_walk<act_t, 128, true, false>(a, st);
        if (!a->decay_per_channel) return a->K == 64 ? launch_mma_walk<act_t, 64, false, true>(a, st) : launch_mma_walk<act_t, 128, false, true>(a, st);
        return a->K == 64 ? launch_mma_walk<act_t, 64, false, false>(a, st) : launch_mma_walk<act_t, 128, false, false>(a, st);
      }
      if (a->delta) return a->K == 64 ? launch_walk<act_t, 64, true>(a, st) : launch_walk<act_t, 128, true>(a, st);
      return a->K == 64 ? launch_walk<act_t, 64, false>(a, st) : launch_walk<act_t, 128, false>(a, st);
    });
  }
  const int VT = a->V + (a->ones ? 1 : 0);
  const int n_chunks = a->n_chunks > 1 ? a->n_chunks : 1;
  const int chunk_len = n_chunks > 1 ? SCAN_CHUNK : a->T;
  int R = 1;
  while (R * SCAN_KPT < a->K) R <<= 1;
  // two columns per lane where the loop is bound by shared-memory reads: long portions without the delta rule
  const int cpl = (!a->delta && a->T >= 64 && a->V >= 2 * (SCAN_THREADS / R)) ? 2 : 1;
  const int KP = R * SCAN_KPT, cols = (SCAN_THREADS / R) * cpl;
  const size_t smem = sizeof(float) * (2 * (size_t)SCAN_TC * (2 * KP + (a->decay_per_channel ? KP : 4) + cols + 4) + (size_t)SCAN_TC * cols);
  auto al16 = [](const void* p) { return ((uintptr_t)p & 15) == 0; };
  const int vec = a->K % 4 == 0 && a->ldq % 4 == 0 && a->ldk % 4 == 0 && al16(a->q) && al16(a->k) &&
                  (!a->decay_per_channel || (a->ldd % 4 == 0 && al16(a->decay)));
  dim3 grid((unsigned)((VT + cols - 1) / cols), (unsigned)a->heads, (unsigned)n_chunks);
  cudaStream_t s = (cudaStream_t)stream;
#define B2L_SCAN_LAUNCH(D, T_, P_, C_, slot_)                                                 \
  do {                                                                                        \
    int rc_ = ensure_dyn_smem(seq_scan_kernel<D, T_, P_, C_>, smem, g_scan_smem[slot_]);      \
    if (rc_) return rc_;                                                                      \
    seq_scan_kernel<D, T_, P_, C_><<<grid, SCAN_THREADS, smem, s>>>(*a, R, vec, chunk_len);   \
  } while (0)
  const bool bf = a->act_dtype == B2L_BF16;
  if (!bf && a->act_dtype != B2L_F32) {
    set_error("b2l_seq_scan: act_dtype %d unsupported", a->act_dtype);
    return B2L_E_UNSUPPORTED;
  }
  if (n_chunks > 1) {   // local end states, combine, then the outputs below start from the workspace
    if (cpl == 2) { if (bf) B2L_SCAN_LAUNCH(0, __nv_bfloat16, 1, 2, 4); else B2L_SCAN_LAUNCH(0, float, 1, 2, 5); }
    else { if (bf) B2L_SCAN_LAUNCH(0, __nv_bfloat16, 1, 1, 6); else B2L_SCAN_LAUNCH(0, float, 1, 1, 7); }
    B2L_LAUNCH_CHECK("seq_scan_kernel (local states)");
    const size_t n = (size_t)a->heads * VT * a->K;
    seq_scan_combine_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(*a);
    B2L_LAUNCH_CHECK("seq_scan_combine_kernel");
  }
  if (a->delta) { if (bf) B2L_SCAN_LAUNCH(1, __nv_bfloat16, 0, 1, 0); else B2L_SCAN_LAUNCH(1, float, 0, 1, 1); }
  else if (cpl == 2) { if (bf) B2L_SCAN_LAUNCH(0, __nv_bfloat16, 0, 2, 2); else B2L_SCAN_LAUNCH(0, float, 0, 2, 3); }
  else { if (bf) B2L_SCAN_LAUNCH(0, __nv_bfloat16, 0, 1, 8); else B2L_SCAN_LAUNCH(0, float, 0, 1, 9); }
#undef B2L_SCAN_LAUNCH
  B2L_LAUNCH_CHECK("seq_scan_kernel");
  return 0;
}

extern "C" int b2l_seq_scan(const b2l_seq_scan_args* a, b2l_stream_t stream) {
  // the space that the declarations ask for: a chunked portion's end states, else b2l_seq_scan_work_floats
  return scan(a, a && a->n_chunks > 1 ? (long long)a->n_chunks * a->heads * a->V * a->K : LLONG_MAX, stream);
}

extern "C" int b2l_seq_scan_within(const b2l_seq_scan_args* a, long long work_floats, b2l_stream_t stream) {
  B2L_CHECK_ARG(!a || a->n_chunks <= 1 || work_floats >= (long long)a->n_chunks * a->heads * (a->V + (a->ones ? 1 : 0)) * a->K,
                "b2l_seq_scan_within: %lld floats do not hold the chunks' end states", work_floats);
  return scan(a, work_floats, stream);
}
