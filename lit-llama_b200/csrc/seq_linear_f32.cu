// f32 linear on the tensor cores: y[M, N] = x[M, K] . W[N, K]^T with f32 operands, f32 sums and f32 results (models that run in 32 bits).
//
// An f32 number is the sum of three bf16 numbers (hi + mid + lo, each rounded: 24 bits in three times eight).  Of the nine products of parts the six
// above 2^-24 are taken (entries below 2^-109 keep fewer bits: the parts have f32's exponents and no more); each is exact in f32, and the sum of 64 k is added to f32 registers, since the tensor core truncates where it adds to its
// accumulator (1024 k in one accumulator: a bias of 2e-6; so errors against float64 are those of f32 FMAs or smaller).
//
// A CTA computes 128 output features x bt tokens (16..112), the WEIGHT as the 128-row operand in tensor memory; per stage of 64 k
//   warp 0        TMA: 128 x 64 weights as they lie (two 128-byte swizzled boxes)
//   warps 4..11   a thread owns half of one weight row: 32 entries into three parts, tcgen05.st into the stage's 3 x 32 columns; then the sum of the
//                 stage before last is added to registers (one feature and half of the tokens a thread)
//   warps 12..15  tokens straight from global memory, 8 entries a thread, into three swizzled bf16 tiles
//   warp 1        24 MMAs (M 128, N bt, K 16), smallest products first, into one of two accumulators; one barrier and one commit per stage
// What bounds it: a stage takes 1.1 us with few tokens, about half of it the 24 MMAs (some 45 cycles each however narrow), the rest the chain from
// operands through one issuing warp to the sums; 1.6 us with 112 tokens on every SM (shared memory: weights in and out, token parts in once and out
// 24 times).  The library's f32 product is FMAs: us here / there, 777 x 1024 -> 2560 39 / 98, -> 1024 33 / 60, 1024 x 2048 -> 5120 158 / 425,
// 400 x 1024 -> 8192 66 / 160; 64 x 1024 -> 1024 32 / 31.  Error against float64: 1024 k 1.1e-7 / 5.7e-7, 4096 k 1.7e-7 / 1.2e-6.
#include "seq_common.cuh"
#include "tc_common.cuh"

namespace b2l {
namespace lf32 {

using namespace tc;

constexpr int BN = 128, BK = 64, NTHREADS = 512, MAX_BT = 112;
constexpr int W_BYTES = BN * BK * 4, A_COLS = 96, BUFS = 3, WS = 4, COL_ACC = BUFS * A_COLS;      // a stage's weight parts: 3 x 32 columns; two accumulators of MAX_BT columns

struct Params {
  CUtensorMap wmap;        // W as 2-D f32, boxes of 32 columns x 128 rows; first member (64-byte alignment)
  const float* x; long long ldx;
  const float* w; long long ldw;
  float* y; long long ldy;
  int M, N, K, bt;
};

// x[0..7] as three rounded bf16 parts, pairs packed
__device__ __forceinline__ void cut8(float (&x)[8], uint32_t (&w)[3][4]) {
#pragma unroll
  for (int p = 0; p < 3; ++p)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const __nv_bfloat162 h = __floats2bfloat162_rn(x[2 * e], x[2 * e + 1]);
      w[p][e] = *reinterpret_cast<const uint32_t*>(&h);
      if (p < 2)
        asm("{\n\t.reg .b64 a, b;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 b, {%2, %3};\n\tsub.rn.f32x2 a, a, b;\n\tmov.b64 {%0, %1}, a;\n\t}"
            : "+f"(x[2 * e]), "+f"(x[2 * e + 1]) : "f"(__uint_as_float(w[p][e] << 16)), "f"(__uint_as_float(w[p][e] & 0xffff0000u)));
    }
}
// A result that came out infinite or NaN, again with FMAs: an infinite entry has no finite rest, so its parts give NaN
__device__ __noinline__ float plain_dot(const float* x, const float* w, int K) {
  float s = 0.f;
  for (int k = 0; k < K; ++k) s = fmaf(x[k], w[k], s);
  return s;
}

__global__ void __launch_bounds__(NTHREADS, 1) seq_linear_f32_kernel(const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[17];
  __shared__ uint32_t tmem_slot;
  const uint32_t sw = (smem_u32(smem_raw) + 1023u) & ~1023u, part = (uint32_t)p.bt * 128, sx = sw + WS * W_BYTES;      // [WS] weights, [2][3] token tiles
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t w_full = smem_u32(bars), w_free = w_full + 32, full = w_full + 64, done = w_full + 88, acc_free = w_full + 112, gave_up = w_full + 128;
  const int n0 = blockIdx.x * BN, m0 = blockIdx.y * p.bt, ns = (p.K + BK - 1) / BK;
  uint32_t dead = 0;
  if (tid == 0) {
    for (int i = 0; i < WS; ++i) { mbar_init(w_full + 8 * i, 1); mbar_init(w_free + 8 * i, 8); }
    for (int i = 0; i < 2; ++i) mbar_init(acc_free + 8 * i, 8);
    for (int i = 0; i < BUFS; ++i) { mbar_init(full + 8 * i, 12); mbar_init(done + 8 * i, 1); }
    mbar_init(gave_up, 1);
    mbar_init_fence();
  }
  if (warp == 1) tmem_alloc(smem_u32(&tmem_slot), 512);
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      int s = 0;
      for (; s < ns; ++s) {
        const int st = s % WS;
        if (s >= WS) mbar_wait(w_free + 8 * st, (uint32_t)(s / WS - 1) & 1u, dead);
        if (dead) break;
        mbar_expect_tx(w_full + 8 * st, W_BYTES);
        for (int h = 0; h < 2; ++h) tma_load_2d(sw + st * W_BYTES + h * (W_BYTES / 2), &p.wmap, s * BK + 32 * h, n0, w_full + 8 * st);
      }
      uint32_t late = 0;                                     // no copy outlives the CTA
      for (int i = max(0, s - WS); i < s; ++i) mbar_wait(w_full + 8 * (i % WS), (uint32_t)(i / WS) & 1u, late);
    }
  } else if (warp == 1) {
    const uint32_t lead = elect_lane();
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.bt >> 3) << 17) | ((uint32_t)(BN >> 4) << 24);      // f32 += bf16 x bf16, K-major
    int st = 0;
    uint32_t ph = 0, ready = 0;                              // the next stage's operands are there: asked while this one's MMAs are issued
    for (int s = 0; s < ns; ++s) {
      if (s >= 2) mbar_wait(acc_free + 8 * (s & 1), (uint32_t)((s >> 1) - 1) & 1u, dead);
      if (!__all_sync(0xffffffffu, ready)) mbar_wait_warp(full + 8 * st, ph, dead);
      dead = __any_sync(0xffffffffu, dead) ? 1u : 0u;
      if (dead) break;
      fence_after();
      ready = mbar_test(full + 8 * (st + 1 < BUFS ? st + 1 : 0), st + 1 < BUFS ? ph : ph ^ 1u);
      const uint32_t d = tmem + COL_ACC + MAX_BT * (s & 1), a = tmem + A_COLS * st;
      const uint64_t b = desc_sw128(sx + (s & 1) * 3 * part);
      constexpr int PW[6] = {2, 1, 0, 1, 0, 0}, PX[6] = {0, 1, 2, 0, 1, 0};      // parts of the weight and of the tokens, smallest products first
      const uint32_t step = part >> 4;
#pragma unroll
      for (int i = 0; i < 6; ++i)                            // written out: from a loop an MMA takes twice as long to issue
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) mma_ts(d, a + 32 * PW[i] + 8 * k, b + PX[i] * step + 2 * k, idesc, (i > 0 || k > 0) ? 1u : 0u, lead);
      if (lead) commit(done + 8 * st);
      __syncwarp();
      if (++st == BUFS) { st = 0; ph ^= 1u; }
    }
    if (dead) {
      uint32_t late = 0;
      if (lead) commit(gave_up);
      mbar_wait(gave_up, 0, late);
    }
  } else if (warp >= 4 && warp < 12) {
    // two groups of four: half of a stage's k each, and half of the tokens' sums
    const int half = (warp - 4) >> 2, row = (warp & 3) * 32 + lane, blocks = p.bt / 16, first = half ? (blocks + 1) / 2 : 0, mine = half ? blocks / 2 : (blocks + 1) / 2;
    const uint32_t lane_at = (uint32_t)((warp & 3) * 32) << 16, acc_at = tmem + lane_at + COL_ACC + 16 * first;
    float acc[4][16] = {};
    int d_st = 0;
    uint32_t d_ph = 0;
    auto add = [&](int s) {                                  // the sum of stage s, once its MMAs are done
      mbar_wait(done + 8 * d_st, d_ph, dead);
      if (++d_st == BUFS) { d_st = 0; d_ph ^= 1u; }
      fence_after();
      __syncwarp();
#pragma unroll
      for (int b = 0; b < 4; ++b)
        if (b < mine) {
          uint32_t r[16];
          tmem_ld16(acc_at + MAX_BT * (s & 1) + 16 * b, r);
#pragma unroll
          for (int i = 0; i < 16; ++i) acc[b][i] += __uint_as_float(r[i]);
        }
      fence_before();
      __syncwarp();
      if (lane == 0 && !dead) mbar_arrive(acc_free + 8 * (s & 1));
    };
    int st = 0;
    for (int s = 0; s < ns; ++s) {
      mbar_wait(w_full + 8 * (s % WS), (uint32_t)(s / WS) & 1u, dead);      // the buffer's MMAs, of stage s - 3, were waited for with their sum
      fence_after();
      const uint32_t src = sw + s % WS * W_BYTES + half * (W_BYTES / 2) + row * 128;
#pragma unroll
      for (int c = 0; c < 2; ++c) {                          // 16 entries: four 16-byte pieces of the row's swizzled half
        uint32_t w[3][8];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float x[8];
          uint32_t o[3][4];
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int j = 4 * c + 2 * h + q;
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x[4 * q]), "=f"(x[4 * q + 1]), "=f"(x[4 * q + 2]), "=f"(x[4 * q + 3]) : "r"(src + ((j ^ (row & 7)) << 4)) : "memory");
          }
          cut8(x, o);
#pragma unroll
          for (int q = 0; q < 3; ++q)
#pragma unroll
            for (int e = 0; e < 4; ++e) w[q][4 * h + e] = o[q][e];
        }
#pragma unroll
        for (int q = 0; q < 3; ++q)
          asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(tmem + lane_at + A_COLS * st + 32 * q + 16 * half + 8 * c), "r"(w[q][0]),
                       "r"(w[q][1]), "r"(w[q][2]), "r"(w[q][3]), "r"(w[q][4]), "r"(w[q][5]), "r"(w[q][6]), "r"(w[q][7]) : "memory");
      }
      tmem_wait_st();
      fence_before();
      __syncwarp();
      if (lane == 0 && !dead) {
        mbar_arrive(full + 8 * st);
        mbar_arrive(w_free + 8 * (s % WS));
      }
      if (++st == BUFS) st = 0;
      if (s >= 2) add(s - 2);
    }
    if (ns > 1) add(ns - 2);
    add(ns - 1);
    const int n = n0 + (warp & 3) * 32 + lane;
    if (n < p.N) {
#pragma unroll
      for (int b = 0; b < 4; ++b)
        if (b < mine) {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int m = m0 + 16 * (first + b) + i;
            if (m >= p.M) continue;
            float v = acc[b][i];
            if (dead) v = __int_as_float(0x7fc00000);
            else if (!(fabsf(v) < INFINITY)) v = plain_dot(p.x + (long long)m * p.ldx, p.w + (long long)n * p.ldw, p.K);
            p.y[(long long)m * p.ldy + n] = v;
          }
        }
    }
  } else if (warp >= 12) {
    const int t = tid - 384, chunk = t & 7, r0 = t >> 3;      // 8 entries of rows r0, r0 + 16, ...
    constexpr int ROUNDS = MAX_BT / 16;
    float x[ROUNDS][8];
    auto fetch = [&](int s) {
      const int k = s * BK + 8 * chunk;
#pragma unroll
      for (int i = 0; i < ROUNDS; ++i) {
        const int r = r0 + 16 * i;
        float4 u = make_float4(0.f, 0.f, 0.f, 0.f), v = u;
        if (r < p.bt && m0 + r < p.M && k < p.K) {            // K in groups of 8
          const float4* q = reinterpret_cast<const float4*>(p.x + (long long)(m0 + r) * p.ldx + k);
          u = q[0];
          v = q[1];
        }
        x[i][0] = u.x; x[i][1] = u.y; x[i][2] = u.z; x[i][3] = u.w; x[i][4] = v.x; x[i][5] = v.y; x[i][6] = v.z; x[i][7] = v.w;
      }
    };
    fetch(0);
    int st = 0, d_st = 0;
    uint32_t d_ph = 0;
    for (int s = 0; s < ns; ++s) {
      if (s >= 2) {                                          // the MMAs that read these tiles
        mbar_wait(done + 8 * d_st, d_ph, dead);
        if (++d_st == BUFS) { d_st = 0; d_ph ^= 1u; }
      }
#pragma unroll
      for (int i = 0; i < ROUNDS; ++i) {
        const int r = r0 + 16 * i;
        if (r >= p.bt) break;
        uint32_t w[3][4];
        cut8(x[i], w);
#pragma unroll
        for (int q = 0; q < 3; ++q)
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sx + ((s & 1) * 3 + q) * part + r * 128 + ((chunk ^ (r & 7)) << 4)), "r"(w[q][0]), "r"(w[q][1]), "r"(w[q][2]), "r"(w[q][3]) : "memory");
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0 && !dead) mbar_arrive(full + 8 * st);
      if (s + 1 < ns) fetch(s + 1);
      if (++st == BUFS) st = 0;
    }
  }
  __syncwarp();
  fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

static size_t smem_of(int bt) {
  const size_t n = WS * W_BYTES + 6 * (size_t)bt * 128 + 1024;
  return n < 120 * 1024 ? 120 * 1024 : n;                    // one CTA per SM: each takes all of tensor memory
}
// Tokens per tile: the fewest rounds of tiles over the SMs, a stage at 2100 cycles (16..64 tokens) and 18 more for each token above 64.
static int tile_for(int M, int N) {
  const int sms = sm_count(), nt = (N + BN - 1) / BN;
  int best = 16;
  long long best_cost = -1;
  for (int bt = 16; bt <= MAX_BT; bt += 16) {
    const long long rounds = ((long long)nt * ((M + bt - 1) / bt) + sms - 1) / sms, cost = rounds * (2100 + (bt > 64 ? 18 * (bt - 64) : 0));
    if (best_cost < 0 || cost <= best_cost) { best_cost = cost; best = bt; }
  }
  return best;
}

}  // namespace lf32
}  // namespace b2l

using namespace b2l;
using namespace b2l::lf32;

extern "C" int b2l_seq_linear_f32(const float* x, long long ldx, const float* w, long long ldw, float* y, long long ldy, int M, int N, int K, b2l_stream_t stream) {
  B2L_CHECK_ARG(x && w && y, "b2l_seq_linear_f32: null pointer");
  B2L_CHECK_ARG(M >= 0 && N > 0 && K > 0 && ldx >= K && ldw >= K && ldy >= N, "b2l_seq_linear_f32: bad size");
  B2L_CHECK_SUPPORTED(K % 8 == 0 && ldx % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)x & 15) == 0 && ((uintptr_t)w & 15) == 0,
                      "b2l_seq_linear_f32: K in groups of 8, rows 16-byte aligned");
  if (M == 0) return 0;
  const int bt = tile_for(M, N), mt = (M + bt - 1) / bt;
  B2L_CHECK_SUPPORTED(mt <= 65535, "b2l_seq_linear_f32: %d rows", M);
  Params p;
  if (int rc = map_sw128(&p.wmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, w, N, K, ldw, 32, BN)) return rc;
  p.x = x; p.ldx = ldx; p.w = w; p.ldw = ldw; p.y = y; p.ldy = ldy; p.M = M; p.N = N; p.K = K; p.bt = bt;
  static DynSmemCache cache;
  if (int rc = ensure_dyn_smem(seq_linear_f32_kernel, smem_of(MAX_BT), cache)) return rc;
  seq_linear_f32_kernel<<<dim3((unsigned)((N + BN - 1) / BN), (unsigned)mt), NTHREADS, smem_of(bt), (cudaStream_t)stream>>>(p);
  B2L_LAUNCH_CHECK("seq_linear_f32_kernel");
  return 0;
}
