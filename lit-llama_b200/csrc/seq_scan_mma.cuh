// Scans 16 tokens at a time on the tensor cores, in f32 by way of three bf16 parts per operand.  With the symbols of the chunked form in seq_scan.cu (G_t the decays
// up to token t of a chunk, D k_i the key decayed to the chunk's end, T, A, B 16 x 16):
//   delta rule:  u = T v - W S_0,  W = T (G k);   o = B T v + Q S_0,  Q = G q - B T (G k)
//   without:     u = vscale v;                    o = B u + Q S_0,    Q = G q
//   S_16 = G_16 S_0 + sum_i (D k_i) u_i^T
// W, Q, D k, T v and B T v need no state, so all chunks make them at once:
//   seq_chunk_ops_kernel   a CTA per (chunk, head): A and B by FMAs, T by forward substitution, the rest as products; W, Q and D k go to the workspace cut into
//                          parts, in the order in which the walk's products take them; B T v goes to the output
//   seq_walk_mma_kernel    a CTA per (head, 16 value columns) walks the chunks: [W; Q] S, the difference, the update.  S^T lies in registers, 16 columns by 16
//                          channels a warp, as the result of one product and, cut into parts, the first operand of the next
// Decays only multiply, as there.  Every product is six bf16 products of parts (those above 2^-24).  The tensor core truncates its sums: a seventh product takes that back
// where it showed beside the FMAs' roundings, in T v, in a chunk's own outputs (B T v, or B u) and in the update; in W S, Q S and the operands it does not show.
// Relative errors against float64, outputs / state, 2048 tokens of 4 heads of 128 x 128, unit keys, the FMA form and this one: delta rule, decays of 0.5 to 1 1.07e-7 / 7.3e-8
// and 1.02e-7 / 6.5e-8, values of mean 2 with decays of 0.99 to 1 2.8e-7 / 2.7e-7 and 1.9e-7 / 1.8e-7, keys that share half of themselves 8.0e-8 / 1.2e-7 and 5.8e-8 / 9.5e-8;
// without it 8.9e-8 / 4.9e-8 and 8.6e-8 / 4.1e-8, with one decay per head 8.9e-8 / 4.8e-8 and 8.9e-8 / 3.9e-8.  Where all is forgotten within a few tokens (decays uniform
// from 0) a result is one or two roundings in either form: 8.1e-8 / 3.5e-8 and 8.4e-8 / 4.6e-8.  Decays within 0.001 of 1 round their products low, here by 16 at
// once: outputs 1.8e-7 and 2.6e-7, state 7.1e-7 and 5.5e-7.  W grows with the keys, and T v - W S loses what T (v - k S) keeps: keys of norm 2 5.5e-7 and 4.2e-7, of norm 3, whose
// recurrence is no longer stable, 512 tokens 1.4e-6 and 2.4e-6.
//
// What bounds it: the walk's chain per chunk, 1500 cycles with the delta rule and 940 without, of which the products are 615 and 390 (m16n8k16 every 8 cycles a
// scheduler): products 370, W S through shared memory 20 + 300 + 40, the update 500, cutting S 150.  An instruction cache next to the schedulers holds a fraction of the
// loop, which is why the operands are made by another kernel (in the same CTAs they cost as much again: 2900 cycles).  At 128 CTAs without the delta rule the operands' way
// from the L2 shows as well (27 KB a chunk and CTA, 5 TB/s: 1280 cycles).  The chunk kernel: 20000 cycles a CTA, three on an SM, instruction fetches and its 58 KB of
// results.  us, FMA form / this one: 2048 tokens, delta rule, 8 / 16 / 32 heads of 128 x 128 156 / 133, 213 / 158, 426 / 321; 512 tokens of 8 heads 49 / 41, of 32 heads of
// 128 x 64 with one decay per head and no delta rule 56 / 44; 2048 and 4096 tokens of 4 heads without it 119 / 84, 226 / 162 (calls back to back).
// With both in f32 FMAs a chunk's products read 0.5 words of shared memory per FMA, 1300 + 750 cycles where the FMAs are 770.
#pragma once
#include "seq_walk_schedule.h"
#include "tc_common.cuh"

namespace b2l {

// ---- x = hi + mid + lo, each rounded to bf16: 24 bits and more between them
__device__ __forceinline__ uint32_t pack_bf16(float x, float y) {      // x in the low half
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(y), "f"(x));
  return r;
}
__device__ __forceinline__ void split2(float x, float y, uint32_t& h, uint32_t& m, uint32_t& l) {      // two values a word
  h = pack_bf16(x, y);
  x -= __uint_as_float(h << 16);
  y -= __uint_as_float(h & 0xffff0000u);
  m = pack_bf16(x, y);
  x -= __uint_as_float(m << 16);
  y -= __uint_as_float(m & 0xffff0000u);
  l = pack_bf16(x, y);
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
struct Parts { uint32_t a[3][4]; };                    // a 16 x 16 operand: rows lane / 4 and + 8, columns 2 (lane % 4), + 1 and + 8
// from two 16 x 8 results side by side, whose lanes hold the same rows and columns
__device__ __forceinline__ void split_pair(const float (&x)[2][4], Parts& p) {
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    split2(x[j][0], x[j][1], p.a[0][2 * j], p.a[1][2 * j], p.a[2][2 * j]);
    split2(x[j][2], x[j][3], p.a[0][2 * j + 1], p.a[1][2 * j + 1], p.a[2][2 * j + 1]);
  }
}
struct PartsB { uint32_t b[3][2]; };
__device__ __forceinline__ void load_b(PartsB& p, const uint32_t* at) {      // six neighbouring words
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const uint2 v = *reinterpret_cast<const uint2*>(at + 2 * i);
    p.b[i][0] = v.x; p.b[i][1] = v.y;
  }
}
// N 16 x 8 results big + small of the six products of parts above 2^-24, in short chains (a product that waits for another's sum takes 22 cycles, one that does
// not 8).  The tensor core truncates its sums: COMP takes the largest product again with its first result as the subtrahend, which leaves what was cut off.
template <int N, bool COMP> __device__ __forceinline__ void mma_parts(float (&big)[N][4], float (&small)[N][4], const Parts& a, const PartsB (&b)[N]) {
  float s1[N][4] = {}, s2[N][4] = {}, s3[N][4] = {};
#pragma unroll
  for (int j = 0; j < N; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) big[j][e] = 0.f;
#pragma unroll
  for (int j = 0; j < N; ++j) mma_bf16(big[j], a.a[0], b[j].b[0]);
#pragma unroll
  for (int j = 0; j < N; ++j) mma_bf16(s1[j], a.a[2], b[j].b[0]);
#pragma unroll
  for (int j = 0; j < N; ++j) mma_bf16(s2[j], a.a[1], b[j].b[0]);
  if (COMP) {
#pragma unroll
    for (int j = 0; j < N; ++j) {
#pragma unroll
      for (int e = 0; e < 4; ++e) s3[j][e] = -big[j][e];
      mma_bf16(s3[j], a.a[0], b[j].b[0]);
    }
  }
#pragma unroll
  for (int j = 0; j < N; ++j) mma_bf16(s1[j], a.a[0], b[j].b[2]);
#pragma unroll
  for (int j = 0; j < N; ++j) mma_bf16(s2[j], a.a[0], b[j].b[1]);
#pragma unroll
  for (int j = 0; j < N; ++j) mma_bf16(s1[j], a.a[1], b[j].b[1]);
#pragma unroll
  for (int j = 0; j < N; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) small[j][e] = COMP ? (s1[j][e] + s2[j][e]) + s3[j][e] : s1[j][e] + s2[j][e];
}
__device__ __forceinline__ bool finite4(const float (&x)[4]) { return fabsf(x[0]) < INFINITY && fabsf(x[1]) < INFINITY && fabsf(x[2]) < INFINITY && fabsf(x[3]) < INFINITY; }
// Tokens x (lane: rows lane / 4, + 8; tokens 2 (lane % 4), + 1, of x[1] + 8) with something infinite or NaN are left out of the products, where a zero weight
// would carry them to earlier tokens; returned: each row's first such token, from which on its results are NaN.
__device__ __forceinline__ void leave_out(float (&x)[2][4], int lane, int (&first)[2]) {
  first[0] = first[1] = CH_C;
#pragma unroll
  for (int j = 1; j >= 0; --j)
#pragma unroll
    for (int e = 3; e >= 0; --e)
      if (!(fabsf(x[j][e]) < INFINITY)) {
        x[j][e] = 0.f;
        first[e >> 1] = min(first[e >> 1], 8 * j + 2 * (lane & 3) + (e & 1));
      }
#pragma unroll
  for (int o = 1; o <= 2; o <<= 1) {
    first[0] = min(first[0], __shfl_xor_sync(0xffffffffu, first[0], o));
    first[1] = min(first[1], __shfl_xor_sync(0xffffffffu, first[1], o));
  }
}
__device__ __forceinline__ void lose_from(float (&x)[2][4], int lane, const int (&first)[2]) {
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (8 * j + 2 * (lane & 3) + (e & 1) >= first[e >> 1]) x[j][e] = __int_as_float(0x7fc00000);
}

// What the walk reads of a chunk, as the chunk kernel writes it.  Operands lie as the walk's products take them, three parts of 16 bits each.
template <int K, bool DELTA>
struct alignas(16) ChunkOps {
  static constexpr int NT = DELTA ? 4 : 2, QT = DELTA ? 2 : 0;       // groups of 8 tokens: (delta: 16 tokens of W,) 16 of Q
  uint32_t wq[K / 16 * NT * 192];  // [16 channels][8 tokens][lane][part][8 channels]
  uint32_t kd[K / 8 * 192];        // [8 channels][lane][part][8 tokens]
  float gc[K];                     // G of the whole chunk
};
// Words per chunk, head and 16 value columns: T v (256), or without the delta rule the parts of v vscale; with one decay per head the parts of D v vscale, and G of
// the 16 tokens behind them.
constexpr int MW_TILE = 384, MW_TILE_G = MW_TILE + CH_C;

struct MwWork { void* ops; uint32_t* tile; };   // of a segment: [chunk][head, or head of q and k] ChunkOps, then [chunk][head][16 value columns] tiles
// What a chunk gives by itself, a CTA per chunk and head; a decay per channel.
constexpr int MW_CHUNK_THREADS = 256;
template <typename act_t, int K, bool DELTA>
__global__ void __launch_bounds__(MW_CHUNK_THREADS, 3) seq_chunk_ops_kernel(b2l_seq_scan_args a, int vec, int t_lo, int t_hi, MwWork work) {
  using Ops = ChunkOps<K, DELTA>;
  constexpr int LD = K + 4, TILES = K / 64;            // TILES groups of 8 channels a warp
  extern __shared__ __align__(16) unsigned char chunk_raw[];
  float (*sq)[LD] = reinterpret_cast<float (*)[LD]>(chunk_raw), (*sk)[LD] = sq + CH_C, (*sg)[LD] = sk + CH_C;
  Ops& ops = *reinterpret_cast<Ops*>(chunk_raw + sizeof(float) * 3 * CH_C * LD);
  __shared__ __align__(16) float sT[2 * CH_C][24];     // T over B T, or B; rows on banks of their own for pairs of columns
  __shared__ float sA[CH_C][CH_C + 1], sB[CH_C][CH_C + 1], sbeta[CH_C];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3, chunk = blockIdx.x, h = blockIdx.y, hq = h / (a.heads / a.qk_heads);
  const int t0 = t_lo + chunk * CH_C, nt = min(CH_C, t_hi - t0);
  const float* gk = a.k + (size_t)t0 * a.ldk + (size_t)hq * K;
  const float* gq = a.q + (size_t)t0 * a.ldq + (size_t)hq * K;
  const float* gd = a.decay + (size_t)t0 * a.ldd + (size_t)h * K;
  if (vec) {
#pragma unroll 2
    for (int i = tid; i < CH_C * K / 4; i += MW_CHUNK_THREADS) {
      const int t = i / (K / 4), c = (i - t * (K / 4)) * 4;
      if (t < nt) {
        cp_async16(&sk[t][c], gk + (size_t)t * a.ldk + c);
        cp_async16(&sq[t][c], gq + (size_t)t * a.ldq + c);
        cp_async16(&sg[t][c], gd + (size_t)t * a.ldd + c);
      } else {
        *reinterpret_cast<float4*>(&sk[t][c]) = *reinterpret_cast<float4*>(&sq[t][c]) = make_float4(0.f, 0.f, 0.f, 0.f);
        *reinterpret_cast<float4*>(&sg[t][c]) = make_float4(1.f, 1.f, 1.f, 1.f);
      }
    }
    cp_async_commit();
  } else {
    for (int i = tid; i < CH_C * K; i += MW_CHUNK_THREADS) {
      const int t = i / K, c = i - t * K;
      const bool in = t < nt;
      sk[t][c] = in ? gk[(size_t)t * a.ldk + c] : 0.f;
      sq[t][c] = in ? gq[(size_t)t * a.ldq + c] : 0.f;
      sg[t][c] = in ? gd[(size_t)t * a.ldd + c] : 1.f;
    }
  }
  if (DELTA && tid < CH_C) sbeta[tid] = tid < nt ? sigmoid_f(ld_act((const act_t*)a.beta, (size_t)(t0 + tid) * a.ldb + h)) : 0.f;
  const bool values = warp * CH_VT < a.V;              // 16 value columns a warp: columns g, g + 8; tokens 2 t4, + 1, + 8, + 9
  float v[2][4] = {}, vs[2][2];
  if (values) {
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int t = 8 * j + 2 * t4 + (e & 1);
        if (t < nt) v[j][e] = a.v[(size_t)(t0 + t) * a.ldv + (size_t)h * a.V + warp * CH_VT + g + 8 * (e >> 1)];
        if (e < 2) vs[j][e] = (!DELTA && a.vscale && t < nt) ? a.vscale[(size_t)(t0 + t) * a.ldvs + h] : 1.f;
      }
  }
  cp_async_wait<0>();
  __syncthreads();
  {
    // A and B by columns i0 .. i0 + 3 and rows r0 .. r1 - 1 a warp, the work spread evenly; the columns' decayed keys are carried from row to row
    const int i0 = 4 * (0x32211000u >> 4 * warp & 15), r0 = (int)(0xcc8a4b60u >> 4 * warp & 15), r1 = (int)(0xffbf9fa5u >> 4 * warp & 15) + 1;
    const int col = ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
    float x[4][K / 32] = {};
#pragma unroll 1
    for (int t = i0; t < r0; ++t)
#pragma unroll
      for (int e = 0; e < K / 32; ++e) {
        const float gv = sg[t][lane + 32 * e];
#pragma unroll
        for (int c = 0; c < 4; ++c) x[c][e] = t == i0 + c ? sk[t][lane + 32 * e] : x[c][e] * gv;
      }
#pragma unroll 1
    for (int t = r0; t < r1; ++t) {
      float p[8] = {};
#pragma unroll
      for (int e = 0; e < K / 32; ++e) {
        const float kv = sk[t][lane + 32 * e], qv = sq[t][lane + 32 * e], gv = sg[t][lane + 32 * e];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          x[c][e] = t == i0 + c ? kv : x[c][e] * gv;
          if (DELTA) p[c] = fmaf(kv, x[c][e], p[c]);
          p[4 + c] = fmaf(qv, x[c][e], p[4 + c]);
        }
      }
      const float s = warp_sum8(p, lane);
      if ((lane & 3) == 0) {
        if (lane & 16) sB[t][i0 + col] = s;
        else if (DELTA) sA[t][i0 + col] = s;
      }
    }
  }
  __syncthreads();
  if (!DELTA) {
    sT[tid / CH_C][tid % CH_C] = tid % CH_C <= tid / CH_C ? sB[tid / CH_C][tid % CH_C] : 0.f;
  } else {
    // columns 2 warp, + 1 of T by forward substitution, a lane per row, and of B T beside it.  Rows up to a token's own only.
    const int t = lane & 15, j = 2 * warp + (lane >> 4);
    float r = t == j ? 1.f : 0.f, m = 0.f;
    const float beta = sbeta[t];
#pragma unroll 4
    for (int i = 0; i < CH_C; ++i) {
      const float c = __shfl_sync(0xffffffffu, beta * r, (lane & 16) + i), av = sA[t][i], bv = sB[t][i];
      if (i < t) r = fmaf(-av, c, r);
      if (i <= t && i >= j) m = fmaf(bv, c, m);
    }
    sT[t][j] = beta * r;
    sT[CH_C + t][j] = m;
  }
  // products over a channel's decays, tokens 2 t4, + 1, + 8, + 9 of channel g of the warp's groups; G k and G q over k and q
#pragma unroll 1
  for (int tile = warp * TILES; tile < (warp + 1) * TILES; ++tile) {
    const int ch = 8 * tile + g;
    float d[4], k[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int t = 2 * t4 + (e & 1) + 8 * (e >> 1);
      d[e] = sg[t][ch]; k[e] = sk[t][ch];
    }
    float up[2], down[2], all[2];                      // product of the pairs of tokens before, after this one, of 0..7 and of 8..15
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      const float p = d[2 * hf] * d[2 * hf + 1], p1 = __shfl_xor_sync(0xffffffffu, p, 1), pp = t4 & 1 ? p1 * p : p * p1, p2 = __shfl_xor_sync(0xffffffffu, pp, 2);
      up[hf] = t4 & 1 ? p1 : 1.f;
      if (t4 & 2) up[hf] *= p2;
      down[hf] = t4 & 1 ? 1.f : p1;
      if (!(t4 & 2)) down[hf] *= p2;
      all[hf] = pp * p2;
    }
    up[1] *= all[0];
    down[0] *= all[1];
    uint32_t* at = ops.kd + tile * 192 + lane * 6;
    uint32_t p[3][2];
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      split2(down[hf] * d[2 * hf + 1] * k[2 * hf], down[hf] * k[2 * hf + 1], p[0][hf], p[1][hf], p[2][hf]);
      const float G0 = up[hf] * d[2 * hf], G1 = G0 * d[2 * hf + 1];
      const int t = 2 * t4 + 8 * hf;
      if (DELTA) {
        sk[t][ch] = k[2 * hf] * G0;
        sk[t + 1][ch] = k[2 * hf + 1] * G1;
      }
      sq[t][ch] *= G0;
      sq[t + 1][ch] *= G1;
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(at + 2 * i) = make_uint2(p[i][0], p[i][1]);
    if (t4 == 0) ops.gc[ch] = all[0] * all[1];
  }
  __syncthreads();
  Parts ta, oa;                                        // T, and B T or B: as the first operand, and transposed as the second
  auto matrix = [&](const float (*m)[24], Parts& p) {
    float x[2][4];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float2 y = *reinterpret_cast<const float2*>(&m[g + 8 * r][2 * t4 + 8 * j]);
        x[j][2 * r] = y.x; x[j][2 * r + 1] = y.y;
      }
    split_pair(x, p);
  };
  auto transposed = [](const Parts& p, PartsB (&b)[2]) {
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int i = 0; i < 3; ++i) { b[j].b[i][0] = p.a[i][j]; b[j].b[i][1] = p.a[i][j + 2]; }
  };
  if (DELTA) matrix(sT, ta);
  matrix(sT + (DELTA ? CH_C : 0), oa);
  // W = T (G k) and Q = G q - B T (G k), or G q: lanes hold tokens g, g + 8 and two neighbouring channels, which is a word of the walk's operands
#pragma unroll 1
  for (int tile = warp * TILES; tile < (warp + 1) * TILES; ++tile) {
    float q[4];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const float2 y = *reinterpret_cast<const float2*>(&sq[g + 8 * r][8 * tile + 2 * t4]);
      q[2 * r] = y.x; q[2 * r + 1] = y.y;
    }
    uint32_t* at = ops.wq + (tile >> 1) * (Ops::NT * 192) + lane * 6 + (tile & 1);
    auto put = [&](const float (&y)[4], int group) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        uint32_t p[3];
        split2(y[2 * r], y[2 * r + 1], p[0], p[1], p[2]);
#pragma unroll
        for (int i = 0; i < 3; ++i) at[(group + r) * 192 + 2 * i] = p[i];
      }
    };
    if (DELTA) {
      float k[4], w[1][4], ws[1][4], o[1][4], os[1][4];
#pragma unroll
      for (int e = 0; e < 4; ++e) k[e] = sk[2 * t4 + (e & 1) + 8 * (e >> 1)][8 * tile + g];
      int first = CH_C;                                // of channel g, as leave_out
      const bool bad = __any_sync(0xffffffffu, !finite4(k));
      if (bad) {
#pragma unroll
        for (int e = 3; e >= 0; --e)
          if (!(fabsf(k[e]) < INFINITY)) {
            k[e] = 0.f;
            first = 2 * t4 + (e & 1) + 8 * (e >> 1);
          }
        first = min(first, __shfl_xor_sync(0xffffffffu, first, 1));
        first = min(first, __shfl_xor_sync(0xffffffffu, first, 2));
      }
      PartsB b[1];
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) split2(k[2 * hf], k[2 * hf + 1], b[0].b[0][hf], b[0].b[1][hf], b[0].b[2][hf]);
      mma_parts<1, false>(w, ws, ta, b);
      mma_parts<1, false>(o, os, oa, b);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        w[0][e] += ws[0][e];
        q[e] -= o[0][e] + os[0][e];
      }
      if (bad) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int f = __shfl_sync(0xffffffffu, first, 4 * (2 * t4 + e));
#pragma unroll
          for (int r = 0; r < 2; ++r)
            if (g + 8 * r >= f) w[0][2 * r + e] = q[2 * r + e] = __int_as_float(0x7fc00000);
        }
      }
      put(w[0], 0);
    }
    put(q, Ops::QT);
  }
  // T v for the walk (without the delta rule: v vscale as it is), and what a chunk's values give its outputs
  if (values) {
    const float skip = a.skip ? ld_act((const act_t*)a.skip, h) : 0.f;
    uint32_t* tile = work.tile + (((size_t)chunk * a.heads + h) * (a.V / CH_VT) + warp) * MW_TILE;
    float x[2][4], y[2][4], ys[2][4];
    Parts va;
    PartsB b[2];
    int first[2];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) x[j][e] = DELTA ? v[j][e] : v[j][e] * vs[j][e & 1];
    if (!DELTA) {
      split_pair(x, va);
#pragma unroll
      for (int i = 0; i < 3; ++i) *reinterpret_cast<uint4*>(tile + 128 * i + 4 * lane) = make_uint4(va.a[i][0], va.a[i][1], va.a[i][2], va.a[i][3]);
    }
    const bool bad = __any_sync(0xffffffffu, !(finite4(x[0]) && finite4(x[1])));
    if (bad) leave_out(x, lane, first);
    if (DELTA || bad) split_pair(x, va);
    if (DELTA) {
      transposed(ta, b);
      if (t4 == (g >> 1)) {                            // without the diagonal, which is beta
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int i = 0; i < 3; ++i) b[j].b[i][j] &= g & 1 ? 0x0000ffffu : 0xffff0000u;
      }
      mma_parts<2, true>(y, ys, va, b);
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) y[j][e] = fmaf(sbeta[8 * j + 2 * t4 + (e & 1)], x[j][e], y[j][e] + ys[j][e]);
      if (bad) lose_from(y, lane, first);
#pragma unroll
      for (int j = 0; j < 2; ++j) *reinterpret_cast<float4*>(tile + 128 * j + 4 * lane) = make_float4(y[j][0], y[j][1], y[j][2], y[j][3]);
    }
    transposed(oa, b);
    mma_parts<2, true>(y, ys, va, b);
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) y[j][e] += ys[j][e];
    if (bad) lose_from(y, lane, first);
    float* out = a.out + (size_t)t0 * a.ldo + (size_t)h * a.V + warp * CH_VT + g;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int t = 8 * j + 2 * t4 + (e & 1);
        if (t < nt) out[(size_t)t * a.ldo + 8 * (e >> 1)] = fmaf(y[j][e], a.q_mult, skip * v[j][e]);
      }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();
  if (tid == 0) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(reinterpret_cast<Ops*>(work.ops) + (size_t)chunk * a.heads + h),
                 "r"((uint32_t)__cvta_generic_to_shared(&ops)), "r"((uint32_t)sizeof(Ops)) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
  }
}

// The same with one decay per head and no delta rule: q, k and their products are those of all heads that share them, and a head's decays weight outputs, values and the
// 16 x 16 matrix.  So a CTA per (chunk, head of q and k, up to eight heads) multiplies q and k once, and the first of them leaves the walk one set of operands for all
// heads, which the L2 then holds once.  us, both kernels, a CTA per head / this form: 32 heads of 128 x 64 over one q and k, 512 and 2048 tokens 44 / 32, 184 / 103; over 32 of
// their own 44 / 44 and 197 / 188; 8 heads of 128 x 128 over one, 2048 tokens 93 / 84.
template <typename act_t, int K>
__global__ void __launch_bounds__(MW_CHUNK_THREADS, 3) seq_chunk_shared_kernel(b2l_seq_scan_args a, int vec, int t_lo, int t_hi, int per, MwWork work) {
  using Ops = ChunkOps<K, false>;
  constexpr int LD = K + 4, TILES = K / 64;
  extern __shared__ __align__(16) unsigned char chunk_raw[];
  float (*sq)[LD] = reinterpret_cast<float (*)[LD]>(chunk_raw), (*sk)[LD] = sq + CH_C;
  Ops& ops = *reinterpret_cast<Ops*>(chunk_raw + sizeof(float) * 2 * CH_C * LD);
  __shared__ __align__(16) float sB[8][CH_C][24];
  __shared__ float sqk[CH_C][CH_C + 1];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3, chunk = blockIdx.x, hq = blockIdx.y;
  // a warp takes a head; where a CTA has fewer than eight, several take one, and its value columns in turn
  const int rep = a.heads / a.qk_heads, here = min(per, rep - per * (int)blockIdx.z), share = 8 / here, h = hq * rep + per * blockIdx.z + warp % here;
  const int t0 = t_lo + chunk * CH_C, nt = min(CH_C, t_hi - t0);
  const float* gk = a.k + (size_t)t0 * a.ldk + (size_t)hq * K;
  const float* gq = a.q + (size_t)t0 * a.ldq + (size_t)hq * K;
  if (vec) {
#pragma unroll 2
    for (int i = tid; i < CH_C * K / 4; i += MW_CHUNK_THREADS) {
      const int t = i / (K / 4), c = (i - t * (K / 4)) * 4;
      if (t < nt) {
        cp_async16(&sk[t][c], gk + (size_t)t * a.ldk + c);
        cp_async16(&sq[t][c], gq + (size_t)t * a.ldq + c);
      } else {
        *reinterpret_cast<float4*>(&sk[t][c]) = *reinterpret_cast<float4*>(&sq[t][c]) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    cp_async_commit();
  } else {
    for (int i = tid; i < CH_C * K; i += MW_CHUNK_THREADS) {
      const int t = i / K, c = i - t * K;
      sk[t][c] = t < nt ? gk[(size_t)t * a.ldk + c] : 0.f;
      sq[t][c] = t < nt ? gq[(size_t)t * a.ldq + c] : 0.f;
    }
  }
  const bool live = warp < share * here;
  const int tt = lane & 15;
  const float d = live && tt < nt ? a.decay[(size_t)(t0 + tt) * a.ldd + h] : 1.f, scale = live && a.vscale && tt < nt ? a.vscale[(size_t)(t0 + tt) * a.ldvs + h] : 1.f;
  cp_async_wait<0>();
  __syncthreads();
  {
    const int t = tid >> 4, i = tid & 15;              // q_t . k_i; of later tokens k_i nothing is used
    float s[4][4] = {};                                // short chains: a sum's error is that of all value columns
#pragma unroll 2
    for (int c = 0; c < K; c += 16)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float4 x = *reinterpret_cast<const float4*>(&sq[t][c + 4 * j]), y = *reinterpret_cast<const float4*>(&sk[i][c + 4 * j]);
        s[j][0] = fmaf(x.x, y.x, s[j][0]); s[j][1] = fmaf(x.y, y.y, s[j][1]); s[j][2] = fmaf(x.z, y.z, s[j][2]); s[j][3] = fmaf(x.w, y.w, s[j][3]);
      }
#pragma unroll
    for (int j = 0; j < 4; ++j) s[j][0] = (s[j][0] + s[j][1]) + (s[j][2] + s[j][3]);
    sqk[t][i] = (s[0][0] + s[1][0]) + (s[2][0] + s[3][0]);
  }
  if (blockIdx.z == 0) {
#pragma unroll 1
    for (int tile = warp * TILES; tile < (warp + 1) * TILES; ++tile) {
      uint32_t p[3][2];
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) split2(sk[2 * t4 + 8 * hf][8 * tile + g], sk[2 * t4 + 8 * hf + 1][8 * tile + g], p[0][hf], p[1][hf], p[2][hf]);
#pragma unroll
      for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(ops.kd + tile * 192 + lane * 6 + 2 * i) = make_uint2(p[i][0], p[i][1]);
      uint32_t* at = ops.wq + (tile >> 1) * (Ops::NT * 192) + lane * 6 + (tile & 1);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float2 y = *reinterpret_cast<const float2*>(&sq[g + 8 * r][8 * tile + 2 * t4]);
        uint32_t w[3];
        split2(y.x, y.y, w[0], w[1], w[2]);
#pragma unroll
        for (int i = 0; i < 3; ++i) at[r * 192 + 2 * i] = w[i];
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  if (blockIdx.z == 0 && tid == 0) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(reinterpret_cast<Ops*>(work.ops) + (size_t)chunk * a.qk_heads + hq),
                 "r"((uint32_t)__cvta_generic_to_shared(&ops)), "r"((uint32_t)sizeof(Ops)) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  }
  __syncwarp();
  if (live) {
    float G = d, D = d;                                // products of the decays up to a token, after it
#pragma unroll
    for (int o = 1; o < CH_C; o <<= 1) {
      const float p = __shfl_up_sync(0xffffffffu, G, o, 16), n = __shfl_down_sync(0xffffffffu, D, o, 16);
      if (tt >= o) G *= p;
      if (tt + o < CH_C) D *= n;
    }
    D = __shfl_down_sync(0xffffffffu, D, 1, 16);
    if (tt == CH_C - 1) D = 1.f;
    float x = 1.f;                                     // column tt of B, the upper half of the warp the odd rows
#pragma unroll 4
    for (int t = 0; t < CH_C; ++t) {
      const float dt = __shfl_sync(0xffffffffu, d, t);
      if (t > tt) x *= dt;
      if ((t & 1) == lane >> 4) sB[warp][t][tt] = t >= tt ? x * sqk[t][tt] : 0.f;
    }
    __syncwarp();
    PartsB b[2];                                       // B transposed
    float dec[2][2], vs[2][2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float2 y = *reinterpret_cast<const float2*>(&sB[warp][g + 8 * j][2 * t4 + 8 * r]);
        split2(y.x, y.y, b[j].b[0][r], b[j].b[1][r], b[j].b[2][r]);
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        dec[j][e] = __shfl_sync(0xffffffffu, D, 8 * j + 2 * t4 + e);
        vs[j][e] = __shfl_sync(0xffffffffu, scale, 8 * j + 2 * t4 + e);
      }
    }
    const float skip = a.skip ? ld_act((const act_t*)a.skip, h) : 0.f;
#pragma unroll 1
    for (int vt = warp / here; vt < a.V / CH_VT; vt += share) {
      uint32_t* tile = work.tile + (((size_t)chunk * a.heads + h) * (a.V / CH_VT) + vt) * MW_TILE_G;
      const size_t col = (size_t)h * a.V + vt * CH_VT + g;
      float v[2][4] = {}, u[2][4], y[2][4], ys[2][4];
      Parts ua;
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int t = 8 * j + 2 * t4 + (e & 1);
          if (t < nt) v[j][e] = a.v[(size_t)(t0 + t) * a.ldv + col + 8 * (e >> 1)];
        }
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) y[j][e] = v[j][e] * vs[j][e & 1] * dec[j][e & 1];
      split_pair(y, ua);
#pragma unroll
      for (int i = 0; i < 3; ++i) *reinterpret_cast<uint4*>(tile + 128 * i + 4 * lane) = make_uint4(ua.a[i][0], ua.a[i][1], ua.a[i][2], ua.a[i][3]);
      if (lane < CH_C) tile[MW_TILE + lane] = __float_as_uint(G);
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) u[j][e] = v[j][e] * vs[j][e & 1];
      int first[2];
      const bool bad = __any_sync(0xffffffffu, !(finite4(u[0]) && finite4(u[1])));
      if (bad) leave_out(u, lane, first);
      split_pair(u, ua);
      mma_parts<2, true>(y, ys, ua, b);
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) y[j][e] += ys[j][e];
      if (bad) lose_from(y, lane, first);
      float* out = a.out + (size_t)t0 * a.ldo + col;
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int t = 8 * j + 2 * t4 + (e & 1);
          if (t < nt) out[(size_t)t * a.ldo + 8 * (e >> 1)] = fmaf(y[j][e], a.q_mult, skip * v[j][e]);
        }
    }
  }
  if (blockIdx.z == 0 && tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

constexpr int MW_WARPS = 8, MW_THREADS = 32 * (MW_WARPS + 4);      // the walk, warp 8 operands, 9 and 10 outputs
template <int K, bool DELTA>
struct MwStage {
  ChunkOps<K, DELTA> ops;
  uint32_t tile[MW_TILE_G];
  float4 rx[MW_WARPS][2][32];    // R of the walk's warps, tokens 0..7 and 8..15
};
template <int K, bool DELTA>
struct MwSmem {
  static constexpr int STAGES = 4;
  MwStage<K, DELTA> st[STAGES];
  float4 px[DELTA ? MW_WARPS : 1][2][32];      // W S of the walk's warps
  uint32_t u[MW_TILE];           // parts of u
  uint64_t bars[STAGES];
  uint32_t bad_columns;          // value columns with something infinite or NaN in them
};
__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void as4(float (&d)[4], const float4& v) { d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w; }
__device__ __forceinline__ void plus4(float (&d)[4], const float4& v) { d[0] += v.x; d[1] += v.y; d[2] += v.z; d[3] += v.w; }
__device__ __forceinline__ float4 sum4(const float (&a)[4], const float (&b)[4]) { return make_float4(a[0] + b[0], a[1] + b[1], a[2] + b[2], a[3] + b[3]); }

// Columns whose results are infinite or NaN (bits of `bad`), token by token in f32 from the state before the segment: what came out finite stays.  `fin` [16][K]: the
// walk's state.  A column is settled once its state holds a NaN and all that is to be replaced in it is one: every later output is NaN then.  us, 2048 tokens of 16
// heads of 128 x 128, delta rule: 169 without anything infinite, 1050 with one infinite value in the middle (2880 before columns settled), 240 with a NaN key at the start.
// Inlined: as a function of its own it cost the walk's loop up to 4 % of its time by where it lay.
template <typename act_t, int K, bool DELTA>
__device__ __forceinline__ void walk_redo(const b2l_seq_scan_args& a, int t_lo, int t_hi, const float* fin, uint32_t bad) {
  constexpr int L = 16, PER = K / L;                   // lanes per column
  const int tid = threadIdx.x;
  if (tid >= CH_VT * L) return;
  const int h = blockIdx.y, hq = h / (a.heads / a.qk_heads), col = blockIdx.x * CH_VT + tid / L, l = tid % L;
  const bool mine = bad >> (tid / L) & 1;
  float* st = a.state + ((size_t)a.meta[0] * a.heads + h) * (size_t)a.V * K + (size_t)col * K;
  fin += (tid / L) * K + l;
  const float skip = a.skip ? ld_act((const act_t*)a.skip, h) : 0.f;
  float S[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) S[i] = st[l + L * i];
  int t = __any_sync(0xffffffffu, mine) ? t_lo : t_hi;
#pragma unroll 1
  while (t < t_hi) {
    float k[PER], q[PER], d[PER];                      // all loads before the first store, which they might alias
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      k[i] = a.k[(size_t)t * a.ldk + (size_t)hq * K + l + L * i];
      q[i] = a.q[(size_t)t * a.ldq + (size_t)hq * K + l + L * i];
      d[i] = a.decay[(size_t)t * a.ldd + (a.decay_per_channel ? (size_t)h * K + l + L * i : (size_t)h)];
    }
    float* out = a.out + (size_t)t * a.ldo + (size_t)h * a.V + col;
    const float v = a.v[(size_t)t * a.ldv + (size_t)h * a.V + col], was = *out,
                gate = DELTA ? sigmoid_f(ld_act((const act_t*)a.beta, (size_t)t * a.ldb + h)) : a.vscale ? a.vscale[(size_t)t * a.ldvs + h] : 1.f;
    float p = 0.f, kq = 0.f, o = 0.f, u = v;           // delta rule: o = S'^T q + u (k . q), as the step by step form takes it
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      S[i] *= d[i];
      if (DELTA) {
        p = fmaf(S[i], k[i], p);
        o = fmaf(S[i], q[i], o);
        kq = fmaf(k[i], q[i], kq);
      }
    }
    if (DELTA) {
#pragma unroll
      for (int w = 1; w < L; w <<= 1) {
        p += __shfl_xor_sync(0xffffffffu, p, w);
        kq += __shfl_xor_sync(0xffffffffu, kq, w);
      }
      u = gate * (v - p);
    } else if (a.vscale) {
      u *= gate;
    }
    bool held = false, open = false;                   // a NaN in the state; something to be replaced that is none yet
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      S[i] = fmaf(k[i], u, S[i]);
      if (!DELTA) o = fmaf(S[i], q[i], o);
      const bool nan = S[i] != S[i];
      held |= nan;
      open |= !nan && !(fabsf(fin[L * i]) < INFINITY);
    }
#pragma unroll
    for (int w = 1; w < L; w <<= 1) o += __shfl_xor_sync(0xffffffffu, o, w);
    if (DELTA) o = fmaf(u, kq, o);
    if (mine && l == 0 && !(fabsf(was) < INFINITY)) *out = o * a.q_mult + skip * v;
    const uint32_t half = 0xffffu << (tid & 16), holds = __ballot_sync(0xffffffffu, held) & half, opens = __ballot_sync(0xffffffffu, open) & half;
    ++t;
    if (__all_sync(0xffffffffu, !mine || (holds && !opens))) break;
  }
  for (t += l; mine && t < t_hi; t += L) {
    float* out = a.out + (size_t)t * a.ldo + (size_t)h * a.V + col;
    if (!(fabsf(*out) < INFINITY)) *out = __int_as_float(0x7fc00000);
  }
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const float x = fin[L * i];
    st[l + L * i] = fabsf(x) < INFINITY ? x : S[i];
  }
}

// tokens t_lo .. t_hi - 1.  SHARED: operands of seq_chunk_shared_kernel; a head's decays are in its tiles
template <typename act_t, int K, bool DELTA, bool SHARED>
__global__ void __launch_bounds__(MW_THREADS) seq_walk_mma_kernel(b2l_seq_scan_args a, int t_lo, int t_hi, MwWork work) {
  using namespace tc;
  extern __shared__ __align__(16) unsigned char walk_raw[];
  using Ops = ChunkOps<K, DELTA>;
  using Stage = MwStage<K, DELTA>;
  using Smem = MwSmem<K, DELTA>;
  constexpr int STAGES = Smem::STAGES, WT = 32 * MW_WARPS;
  Smem& sm = *reinterpret_cast<Smem*>(walk_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3, h = blockIdx.y, v0 = blockIdx.x * CH_VT;
  const int n_chunks = (t_hi - t_lo + CH_C - 1) / CH_C;
  float* st = a.state + ((size_t)a.meta[0] * a.heads + h) * (size_t)a.V * K;
  enum { PX = 1, UX = 2, FULL = 3, DONE = FULL + STAGES, EMPTY = DONE + STAGES };      // barriers: W S and u exchanged; operands of a stage there, walked, read out
  if (tid == 0) {
    sm.bad_columns = 0u;
    for (int i = 0; i < STAGES; ++i) mbar_init(smem_u32(sm.bars + i), 1);
    mbar_init_fence();
  }
  __syncthreads();
  uint32_t dead = 0;
  bool odd[2] = {};                                    // this thread saw something infinite or NaN in value column g, g + 8
  constexpr int WC = K / MW_WARPS, UN = WC / 8;      // channels of a warp of the walk: 16, or 8 (the other half of the products' 16 is zero), groups of 8
  float S[2][4] = {};                                  // value columns lane / 4, + 8; channels 2 (lane % 4), + 1 of the group
  const float lost = __int_as_float(0x7fc00000);

  if (warp < MW_WARPS) {
    // ===================== the walk: channels WC warp .. of S =====================
    const int c0 = warp * WC, at0 = UN == 1 ? warp & 1 : 0;
    Parts sa;
#pragma unroll
    for (int j = 0; j < 2; ++j)
      if (j >= at0 && j < at0 + UN) {
        const float* p = st + (size_t)(v0 + g) * K + c0 + 8 * (j - at0) + 2 * t4;
        const float2 x = *reinterpret_cast<const float2*>(p), y = *reinterpret_cast<const float2*>(p + 8 * (size_t)K);
        S[j][0] = x.x; S[j][1] = x.y; S[j][2] = y.x; S[j][3] = y.y;
      }
    split_pair(S, sa);
    // the element of u that this thread forms (delta rule): number tid of the 256 as the results lie
    uint16_t* const u_at = reinterpret_cast<uint16_t*>(sm.u) + (tid >> 2 & 31) * 8 + 2 * (2 * (tid >> 7) + (tid >> 1 & 1)) + (tid & 1);
    int sti = 0;
    for (int n = 0; n < n_chunks; ++n) {
      Stage& s = sm.st[sti];
      bar_sync(FULL + sti, WT + 32);
      const uint32_t* wq = s.ops.wq + (size_t)(UN == 1 ? warp >> 1 : warp) * (Ops::NT * 192) + lane * 6;
      PartsB b[2], br[2], bd[UN];
      float r[2][4], rs[2][4];
      load_b(br[0], wq + Ops::QT * 192);
      load_b(br[1], wq + Ops::QT * 192 + 192);
      if (DELTA) {
        load_b(b[0], wq);
        load_b(b[1], wq + 192);
        float big[2][4], small[2][4];
        mma_parts<2, false>(big, small, sa, b);
        sm.px[warp][0][lane] = sum4(big[0], small[0]);
        sm.px[warp][1][lane] = sum4(big[1], small[1]);
        bar_sync(PX, WT);
        const float* at = reinterpret_cast<const float*>(sm.px) + tid;
        float p[MW_WARPS], u = __uint_as_float(s.tile[tid]);
#pragma unroll
        for (int w = 0; w < MW_WARPS; ++w) p[w] = at[256 * w];
        mma_parts<2, false>(r, rs, sa, br);
#pragma unroll
        for (int w = 1; w < MW_WARPS; w += 2) p[w] += p[w - 1];
        u -= (p[1] + p[3]) + (p[5] + p[7]);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const uint32_t w = pack_bf16(u, 0.f);
          u_at[256 * i] = (uint16_t)w;
          u -= __uint_as_float(w << 16);
        }
      } else {
        mma_parts<2, false>(r, rs, sa, br);
      }
#pragma unroll
      for (int j = 0; j < UN; ++j) {
        load_b(bd[j], s.ops.kd + (warp * UN + j) * 192 + lane * 6);
      }
      if (DELTA) bar_sync(UX, WT);
      Parts ua;
      {
        const uint4* at = reinterpret_cast<const uint4*>(DELTA ? sm.u : s.tile) + lane;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const uint4 w = at[32 * i];
          ua.a[i][0] = w.x; ua.a[i][1] = w.y; ua.a[i][2] = w.z; ua.a[i][3] = w.w;
        }
      }
      float d[UN][4], ds[UN][4];
      mma_parts<UN, true>(d, ds, ua, bd);
#pragma unroll
      for (int j = 0; j < UN; ++j) {
        float2 gc;
        if (SHARED) gc.x = gc.y = __uint_as_float(s.tile[MW_TILE_G - 1]);
        else gc = *reinterpret_cast<const float2*>(&s.ops.gc[c0 + 8 * j + 2 * t4]);
#pragma unroll
        for (int e = 0; e < 4; ++e) d[j][e] += fmaf(UN == 1 ? S[0][e] + S[1][e] : S[j][e], e & 1 ? gc.y : gc.x, ds[j][e]);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[j][e] = UN == 2 ? d[j % UN][e] : (j == at0 ? d[0][e] : 0.f);
      s.rx[warp][0][lane] = sum4(r[0], rs[0]);
      s.rx[warp][1][lane] = sum4(r[1], rs[1]);
      bar_arrive(DONE + sti, WT + 64);
      split_pair(S, sa);
      if (++sti == STAGES) sti = 0;
    }
    for (int e = 0; e < 4; ++e) odd[e >> 1] |= !(fabsf(S[0][e]) < INFINITY && fabsf(S[1][e]) < INFINITY);
  } else if (warp == MW_WARPS) {
    // ===================== operands, as the chunk kernel wrote them: STAGES - 1 copies ahead of the chunk that is handed over =====================
    constexpr int WORDS = SHARED ? MW_TILE_G : MW_TILE;
    const int sets = SHARED ? a.qk_heads : a.heads;    // of operands, of a chunk
    const Ops* ops = reinterpret_cast<const Ops*>(work.ops) + (SHARED ? h / (a.heads / a.qk_heads) : h);
    const uint32_t* tile = work.tile + ((size_t)h * gridDim.x + blockIdx.x) * WORDS;
    auto copy = [&](int n, int to) {
      if (lane == 0) {
        const uint32_t bar = smem_u32(sm.bars + to);
        mbar_expect_tx(bar, sizeof(Ops) + 4 * WORDS);
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(&sm.st[to].ops)), "l"(ops + (size_t)n * sets),
                     "r"((uint32_t)sizeof(Ops)), "r"(bar) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(sm.st[to].tile)),
                     "l"(tile + (size_t)n * a.heads * gridDim.x * WORDS), "r"((uint32_t)(4 * WORDS)), "r"(bar) : "memory");
      }
    };
    walk_operands<STAGES>(
        n_chunks, [&](int n) { copy(n, n % STAGES); },
        [&](int n) {
          mbar_wait_warp(smem_u32(sm.bars + n % STAGES), (uint32_t)(n / STAGES) & 1u, dead);
          return !dead;
        },
        [&](int n) { bar_arrive(FULL + n % STAGES, WT + 32); }, [&](int n) { bar_sync(EMPTY + n % STAGES, 96); },
        [&](int n) {
          uint32_t late = 0;
          mbar_wait(smem_u32(sm.bars + n % STAGES), (uint32_t)(n / STAGES) & 1u, late);
        });
  } else if (warp < MW_WARPS + 3) {
    // ===================== outputs: 8 tokens of a chunk each, beside what the chunk kernel wrote =====================
    const int ow = warp - MW_WARPS - 1;
    int sti = 0;
    for (int n = 0; n < n_chunks; ++n) {
      const Stage& s = sm.st[sti];
      float y[4], r[4];
      const int t0 = t_lo + n * CH_C + 8 * ow + 2 * t4;
      float* out = a.out + (size_t)t0 * a.ldo + (size_t)h * a.V + v0 + g;
#pragma unroll
      for (int e = 0; e < 4; ++e) y[e] = t0 + (e & 1) < t_hi ? out[(e & 1) * (size_t)a.ldo + 8 * (e >> 1)] : 0.f;
      bar_sync(DONE + sti, WT + 64);
      as4(r, s.rx[0][ow][lane]);
#pragma unroll
      for (int w = 1; w < MW_WARPS; ++w) plus4(r, s.rx[w][ow][lane]);
      if (SHARED) {
#pragma unroll
        for (int e = 0; e < 4; ++e) r[e] *= __uint_as_float(s.tile[MW_TILE + 8 * ow + 2 * t4 + (e & 1)]);
      }
      bar_arrive(EMPTY + sti, 96);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        y[e] = fmaf(r[e], a.q_mult, y[e]);
        odd[e >> 1] |= !(fabsf(y[e]) < INFINITY);
        if (t0 + (e & 1) < t_hi) out[(e & 1) * (size_t)a.ldo + 8 * (e >> 1)] = y[e];
      }
      if (++sti == STAGES) sti = 0;
    }
  }
  if (odd[0] || odd[1]) atomicOr(&sm.bad_columns, (uint32_t)odd[0] << g | (uint32_t)odd[1] << (g + 8));
  const int gone = __syncthreads_or((int)dead), redo = (int)sm.bad_columns;
  if (warp < MW_WARPS) {
    float* fin = reinterpret_cast<float*>(&sm.st[0]);  // [16][K]
    const int at0 = UN == 1 ? warp & 1 : 0;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int r = 0; r < 2; ++r)
        if (j >= at0 && j < at0 + UN) {
          const int col = g + 8 * r, ch = warp * WC + 8 * (j - at0) + 2 * t4;
          *reinterpret_cast<float2*>(walk_state_to_scratch(redo, gone) ? fin + col * K + ch : st + (size_t)(v0 + col) * K + ch) = gone ? make_float2(lost, lost) : make_float2(S[j][2 * r], S[j][2 * r + 1]);
        }
  }
  if (gone) {
    for (int i = tid; i < (t_hi - t_lo) * CH_VT; i += MW_THREADS) a.out[(size_t)(t_lo + i / CH_VT) * a.ldo + (size_t)h * a.V + v0 + i % CH_VT] = lost;
  } else if (redo) {
    __syncthreads();
    walk_redo<act_t, K, DELTA>(a, t_lo, t_hi, reinterpret_cast<const float*>(&sm.st[0]), (uint32_t)redo);
  }
}

// Where this form is taken: key size 128 (64 without the delta rule: 16 heads of 64 x 64, 512 tokens 33 / 29 us, 64 heads, 2048 tokens 281 / 221 us; with it 42 / 44
// and 166 / 177), a CTA's worth of value columns, and portions long enough for the second kernel's launch and the chunks' operands to pay: 64 tokens where the walk
// has more than 64 CTAs (16 heads of 128 x 128 19.8 / 17.7 us with the delta rule, 15.7 / 14.5 without; 32 of 128 x 64 15.8 / 13.6), 144 otherwise (8 heads, 128 / 144 / 192 tokens: 16.7 / 16.7, 18.8 / 16.6, 20.8 / 18.6).
constexpr int MW_HEADS = 256, MW_V = 128, MW_LEAST = 64, MW_SEGMENT = 2048;      // most heads, value columns; least tokens; chunks times heads of a segment
static bool mma_walk(int T, int heads, int K, int V, int delta) {
  if (heads > MW_HEADS || V > MW_V || V % CH_VT) return false;
  return K == 128 ? T >= (heads * (V / CH_VT) > 64 ? MW_LEAST : 144) : K == 64 && !delta && T >= 512;
}
// Tokens of a segment.  A portion goes through the two kernels by segments so that the workspace stays below 103 MB (2048 chunks and heads of 50 KB with the delta rule
// and 128 value columns), most of which the L2 keeps; a segment more costs some 8 us beside 160 or more.
static int mma_segment(int heads) { return MW_SEGMENT / heads * CH_C; }
// Floats of the workspace: of the largest segment, each chunk's operands once for every head (or, with one decay per head, every head of q and k), then its tiles.
static long long mma_walk_floats(int T, int heads, int qk_heads, int K, int V, int delta, int per_channel) {
  const long long chunks = ((T < mma_segment(heads) ? T : mma_segment(heads)) + CH_C - 1) / CH_C;
  const long long ops = (K == 64 ? sizeof(ChunkOps<64, false>) : delta ? sizeof(ChunkOps<128, true>) : sizeof(ChunkOps<128, false>)) / 4;
  return chunks * ((per_channel ? heads : qk_heads) * ops + (long long)heads * (V / CH_VT) * (per_channel ? MW_TILE : MW_TILE_G));
}
// At least that, whatever the sizes but these two; grows with both of them.
static long long mma_walk_most_floats(int T, int heads) {
  const long long all = (long long)((T + CH_C - 1) / CH_C) * heads;
  return (all < MW_SEGMENT ? all : MW_SEGMENT) * (long long)(sizeof(ChunkOps<128, true>) / 4 + MW_V / CH_VT * MW_TILE_G);
}

template <typename act_t, int K, bool DELTA, bool SHARED>
static int launch_mma_walk(const b2l_seq_scan_args* a, cudaStream_t s) {
  using Ops = ChunkOps<K, DELTA>;
  auto al = [](const void* p) { return ((uintptr_t)p & 15) == 0; };
  const int vec = a->ldq % 4 == 0 && a->ldk % 4 == 0 && al(a->q) && al(a->k) && (!a->decay_per_channel || (a->ldd % 4 == 0 && al(a->decay)));
  static DynSmemCache chunk_cache, walk_cache;
  const size_t chunk_smem = sizeof(Ops) + sizeof(float) * (SHARED ? 2 : 3) * CH_C * (K + 4), walk_smem = sizeof(MwSmem<K, DELTA>);
  if constexpr (SHARED) {
    if (int rc = ensure_dyn_smem(seq_chunk_shared_kernel<act_t, K>, chunk_smem, chunk_cache)) return rc;
  } else {
    if (int rc = ensure_dyn_smem(seq_chunk_ops_kernel<act_t, K, DELTA>, chunk_smem, chunk_cache)) return rc;
  }
  if (int rc = ensure_dyn_smem(seq_walk_mma_kernel<act_t, K, DELTA, SHARED>, walk_smem, walk_cache)) return rc;
  const int seg = mma_segment(a->heads), rep = a->heads / a->qk_heads, sms = sm_count();
  for (int t = 0; t < a->T; t += seg) {
    const int hi = a->T - t < seg ? a->T : t + seg, chunks = (hi - t + CH_C - 1) / CH_C;
    const MwWork work{a->work_state, reinterpret_cast<uint32_t*>(reinterpret_cast<Ops*>(a->work_state) + (size_t)chunks * (SHARED ? a->qk_heads : a->heads))};
    if constexpr (SHARED) {
      int per = 8;                                       // heads of a CTA: fewer where CTAs of eight leave SMs idle (8 heads, 512 tokens: 35 us with eight, 32 with two)
      while (per > 1 && (long long)chunks * a->qk_heads * ((rep + per - 1) / per) * 8 < 7LL * sms) per /= 2;
      seq_chunk_shared_kernel<act_t, K><<<dim3((unsigned)chunks, (unsigned)a->qk_heads, (unsigned)((rep + per - 1) / per)), MW_CHUNK_THREADS, chunk_smem, s>>>(*a, vec, t, hi, per,
                                                                                                                                                             work);
    } else
      seq_chunk_ops_kernel<act_t, K, DELTA><<<dim3((unsigned)chunks, (unsigned)a->heads), MW_CHUNK_THREADS, chunk_smem, s>>>(*a, vec, t, hi, work);
    B2L_LAUNCH_CHECK("seq_chunk_ops_kernel");
    seq_walk_mma_kernel<act_t, K, DELTA, SHARED><<<dim3((unsigned)(a->V / CH_VT), (unsigned)a->heads), MW_THREADS, walk_smem, s>>>(*a, t, hi, work);
    B2L_LAUNCH_CHECK("seq_walk_mma_kernel");
  }
  return 0;
}

}  // namespace b2l
