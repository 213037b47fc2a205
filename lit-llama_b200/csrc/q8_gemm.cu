// LLM.int8() linear for several activation rows (prompts, batched decoding): y[M, N] from x[M, K] bf16 and the int8 weight CB[N, K].
//
// Replaces Linear8bitLt.forward (lit_llama/quantization.py:38-77 + the published LLM.int8() algorithm) for M > 1; the arithmetic is that of
// q8_gemv.cu value by value (integer contraction, the same f32 / fp16 roundings, outlier terms added in ascending k).  Three launches:
//   q8_mask_kernel    outlier columns of the batch as a K-bit mask (any |fp16(x)| >= threshold);
//   q8_rows_kernel    a CTA per row: absmax over the other columns, int8 row, the row's outlier activations (fp16, [outlier][row]), and,
//                     by the first CTA, the ascending list of outlier columns;
//   q8_gemm_kernel    tcgen05.mma kind::i8 (s8 x s8 -> s32): 128 weight rows x up to 256 tokens per CTA over K (or a part of it).
//
// The GEMM takes the WEIGHT as the 128-row operand, so a prompt of up to 256 tokens reads every weight once: bound by HBM up to ~400
// rows (N K bytes against 2 M N K operations), by the tensor pipe beyond.  CB is read in the checkpoint's layout: a 128-byte swizzled TMA
// box is 128 rows x 128 k.  Where N / 128 tiles do not fill the chip a cluster of 2, 4 or 8 CTAs splits K; the partial sums are integers,
// so adding them through distributed shared memory changes nothing in the result.
// One row at a time through the single-row kernel took 3956 us for 137 x 4096 -> 11008 (137 launches that each stream the weight); the
// three launches took 36.5 us with the call's host side one after the other, and 30.7 each launched while the one before it runs (the rows wait for
// the mask after loading their x, the product for the rows after requesting its first weights); the results have the same bits.
#include <cuda_fp16.h>

#include "tc_common.cuh"

namespace b2l {
namespace q8gm {

using namespace tc;

constexpr int BN = 128;                    // weight rows per CTA = rows of the MMA
constexpr int BK = 128;                    // k (bytes) per stage: one swizzled row
constexpr int A_BYTES = BN * BK;           // 16 KB
constexpr int NTHREADS = 192;              // warp 0: TMA, warp 1: MMA issue and tensor memory, warps 2..5: epilogue
constexpr int MAX_STAGES = 8;
constexpr int SM_OUT = 16;                 // outlier columns whose activations wait in shared memory; more are read from the workspace,
constexpr int WS_OUT = 128;                // and beyond these from x
constexpr int SLAB = 4096;                 // rows per pass: bounds the workspace (16 tiles of 256 rows fill the chip whatever N)

// ---------------------------------------------------------------- outlier columns: 64 columns per CTA, 32 rows at a time
__global__ void __launch_bounds__(256) q8_mask_kernel(const __nv_bfloat16* __restrict__ x, int ldx, int M, int K, float threshold, uint32_t* __restrict__ mask) {
  pdl_launch_dependents();                            // the rows' kernel loads its row meanwhile
  __shared__ uint32_t bits[2];
  const int tid = threadIdx.x, k = blockIdx.x * 64 + (tid & 7) * 8;
  if (tid < 2) bits[tid] = 0u;
  __syncthreads();
  uint32_t o = 0;
  if (k < K) {
#pragma unroll 4
    for (int m = tid >> 3; m < M; m += 32) {
      const uint4 u = *reinterpret_cast<const uint4*>(x + (size_t)m * ldx + k);
      const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (fabsf(__half2float(__float2half_rn(__uint_as_float(w[q] << 16)))) >= threshold) o |= 1u << (2 * q);
        if (fabsf(__half2float(__float2half_rn(__uint_as_float(w[q] & 0xffff0000u)))) >= threshold) o |= 2u << (2 * q);
      }
    }
  }
  if (o) atomicOr(&bits[(tid & 7) >> 2], o << (8 * (tid & 3)));
  __syncthreads();
  if (tid < 2 && blockIdx.x * 64 + tid * 32 < K) mask[blockIdx.x * 2 + tid] = bits[tid];
}

// ---------------------------------------------------------------- a row: int8 values, scale, outlier activations
constexpr int ROW_THREADS = 256;
constexpr int MAX_K = 12288;
__global__ void __launch_bounds__(ROW_THREADS) q8_rows_kernel(const __nv_bfloat16* __restrict__ x, int ldx, int K, int Mp, const uint32_t* __restrict__ mask_g,
                                                              int8_t* __restrict__ xq, float* __restrict__ sca_out, __half* __restrict__ aout,
                                                              int* __restrict__ list, int* __restrict__ n_out) {
  __shared__ uint32_t mask[MAX_K / 32];
  __shared__ int before[MAX_K / 32];          // outliers before each word
  __shared__ float red[ROW_THREADS / 32];
  __shared__ int wsum[ROW_THREADS / 32];
  constexpr int MAXC = MAX_K / (ROW_THREADS * 8);
  const int m = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, words = K / 32;
  pdl_launch_dependents();                            // the product starts on its weights
  float av[MAXC][8];
#pragma unroll
  for (int c = 0; c < MAXC; ++c) {
    const int k = (c * ROW_THREADS + tid) * 8;
    if (k < K) {
      const uint4 u = *reinterpret_cast<const uint4*>(x + (size_t)m * ldx + k);
      const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        av[c][2 * q] = __half2float(__float2half_rn(__uint_as_float(w[q] << 16)));
        av[c][2 * q + 1] = __half2float(__float2half_rn(__uint_as_float(w[q] & 0xffff0000u)));
      }
    }
  }
  pdl_wait();                                         // the mask is complete; read by coherent loads only (x was there before the mask's kernel began)
  // two neighbouring words per thread (K <= 12288: at most 384 words), an exclusive scan of their outlier counts
  auto word = [&](int i) {
    uint32_t v = 0u;
    if (i < words) asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(mask_g + i) : "memory");
    return v;
  };
  const uint32_t w0 = word(2 * tid), w1 = word(2 * tid + 1);
  const int mine = __popc(w0) + __popc(w1);
  int sum = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, sum, o);
    if (lane >= o) sum += v;
  }
  if (lane == 31) wsum[warp] = sum;
  __syncthreads();
  int at = sum - mine;
  for (int w = 0; w < warp; ++w) at += wsum[w];
  if (2 * tid < words) { mask[2 * tid] = w0; before[2 * tid] = at; }
  if (2 * tid + 1 < words) { mask[2 * tid + 1] = w1; before[2 * tid + 1] = at + __popc(w0); }
  if (m == 0) {
    int j = at;
    for (uint32_t b = w0; b; b &= b - 1) list[j++] = 64 * tid + __ffs(b) - 1;
    for (uint32_t b = w1; b; b &= b - 1) list[j++] = 64 * tid + 32 + __ffs(b) - 1;
    if (tid == ROW_THREADS - 1) *n_out = at + mine;
  }
  __syncthreads();
  float amax = 0.f;
#pragma unroll
  for (int c = 0; c < MAXC; ++c) {
    const int k = (c * ROW_THREADS + tid) * 8;
    if (k < K) {
      const uint32_t word = mask[k >> 5], mb = (word >> (k & 31)) & 0xFFu;
      if (mb == 0) {
#pragma unroll
        for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(av[c][e]));
      } else {
        int j = before[k >> 5] + __popc(word & ((1u << (k & 31)) - 1u));
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          if ((mb >> e) & 1u) {
            if (j < WS_OUT) aout[(size_t)j * Mp + m] = __float2half_rn(av[c][e]);
            ++j;
          } else {
            amax = fmaxf(amax, fabsf(av[c][e]));
          }
        }
      }
    }
  }
  amax = warp_max(amax);
  if (lane == 0) red[warp] = amax;
  __syncthreads();
  float sca = 0.f;
#pragma unroll
  for (int w = 0; w < ROW_THREADS / 32; ++w) sca = fmaxf(sca, red[w]);
  const float qs = sca > 0.f ? 127.0f / sca : 0.f;
#pragma unroll
  for (int c = 0; c < MAXC; ++c) {
    const int k = (c * ROW_THREADS + tid) * 8;
    if (k < K) {
      const uint32_t mb = (mask[k >> 5] >> (k & 31)) & 0xFFu;
      uint32_t pk[2] = {0u, 0u};
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        int qv = ((mb >> e) & 1u) ? 0 : __float2int_rn(av[c][e] * qs);
        qv = max(-127, min(127, qv));
        pk[e >> 2] |= (uint32_t)(qv & 0xFF) << (8 * (e & 3));
      }
      *reinterpret_cast<uint2*>(xq + (size_t)m * K + k) = make_uint2(pk[0], pk[1]);
    }
  }
  if (tid == 0) sca_out[m] = sca;
}

// ---------------------------------------------------------------- the product
struct Params {
  CUtensorMap wmap, xmap;      // CB [N][K], xq [M][K]: boxes of 128 bytes x 128 / bt rows
  const int8_t* cb; const float* scb; const float* sca; const __half* aout; const int* list; const int* n_out;
  const __nv_bfloat16* x;
  __nv_bfloat16* y;
  int M, N, K, Mp, ldx, ldy, bt, nst, splits;
};

__device__ __forceinline__ void mma_i8(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc, uint32_t lead) {
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t@q tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a),
               "l"(b), "r"(idesc), "r"(acc), "r"(lead)
               : "memory");
}
__global__ void __launch_bounds__(NTHREADS, 2) q8_gemm_kernel(const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[2 * MAX_STAGES + 2];
  __shared__ uint32_t tmem_slot, failed;
  __shared__ __align__(16) __half s_act[SM_OUT][256];        // the first outliers' activations of the CTA's tokens
  __shared__ float s_sca[256];
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;            // 128-byte swizzle atoms are 1024-byte aligned
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t bar_full = smem_u32(bars), bar_empty = bar_full + 8 * MAX_STAGES, bar_acc = bar_full + 16 * MAX_STAGES,
                 gave_up = bar_acc + 8;
  const uint32_t stage_bytes = A_BYTES + (uint32_t)p.bt * BK;
  const int n0 = (blockIdx.x / p.splits) * BN, m0 = blockIdx.y * p.bt;
  const uint32_t rank = p.splits > 1 ? cluster_rank() : 0u;
  const int n_kb = p.K / BK, kb_lo = (int)((long long)rank * n_kb / p.splits), kb_hi = (int)((long long)(rank + 1) * n_kb / p.splits);
  const uint32_t cols = p.bt > 128 ? 256u : p.bt > 64 ? 128u : p.bt > 32 ? 64u : 32u;
  uint32_t dead = 0;

  if (tid == 0) {
    for (int i = 0; i < p.nst; ++i) { mbar_init(bar_full + 8 * i, 1); mbar_init(bar_empty + 8 * i, 1); }
    mbar_init(bar_acc, 1);
    mbar_init(gave_up, 1);
    failed = 0u;
    mbar_init_fence();
  }
  if (warp == 1) tmem_alloc(smem_u32(&tmem_slot), cols);
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      int st = 0;
      uint32_t ph = 1;                                       // parity of a stage's previous use: passes at once the first time
      const int early = min(kb_lo + p.nst, kb_hi);           // weights of the first stages on their way while the rows' kernel still runs
      for (int kb = kb_lo; kb < early; ++kb) {
        mbar_expect_tx(bar_full + 8 * (kb - kb_lo), stage_bytes);
        tma_load_2d(sbase + (kb - kb_lo) * stage_bytes, &p.wmap, kb * BK, n0, bar_full + 8 * (kb - kb_lo));
      }
      pdl_wait();
      asm volatile("fence.proxy.async;" ::: "memory");         // ordinary stores of the kernel before, read by the async proxy
      for (int kb = kb_lo; kb < kb_hi; ++kb) {
        mbar_wait(bar_empty + 8 * st, ph, dead);
        if (dead) break;
        if (kb >= early) {
          mbar_expect_tx(bar_full + 8 * st, stage_bytes);
          tma_load_2d(sbase + st * stage_bytes, &p.wmap, kb * BK, n0, bar_full + 8 * st);
        }
        tma_load_2d(sbase + st * stage_bytes + A_BYTES, &p.xmap, kb * BK, m0, bar_full + 8 * st);
        if (++st == p.nst) { st = 0; ph ^= 1u; }
      }
      uint32_t late = 0;
      for (int i = 0; i < p.nst; ++i) {                      // no copy outlives the CTA; all have landed unless a wait ran out
        mbar_wait(bar_full + 8 * st, ph, late);
        if (++st == p.nst) { st = 0; ph ^= 1u; }
      }
    }
  } else if (warp == 1) {
    const uint32_t lead = elect_lane();
    // kind::i8: D = s32, A = B = s8, K-major, 128 x bt
    const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.bt >> 3) << 17) | ((uint32_t)(BN >> 4) << 24);
    int st = 0;
    uint32_t ph = 0, acc = 0;
    for (int kb = kb_lo; kb < kb_hi; ++kb) {
      mbar_wait_warp(bar_full + 8 * st, ph, dead);
      if (dead) break;
      fence_after();
      const uint64_t ad = desc_sw128(sbase + st * stage_bytes), bd = desc_sw128(sbase + st * stage_bytes + A_BYTES);
#pragma unroll
      for (int j = 0; j < BK / 32; ++j) mma_i8(tmem, ad + 2 * j, bd + 2 * j, idesc, j > 0 ? 1u : acc, lead);
      acc = 1;
      if (lead) commit(bar_empty + 8 * st);
      __syncwarp();
      if (++st == p.nst) { st = 0; ph ^= 1u; }
    }
    if (lead) commit(dead ? gave_up : bar_acc);
    if (dead) {
      uint32_t late = 0;
      mbar_wait(gave_up, 0, late);
    }
  } else {
    // while the product runs: row scales and outlier activations of these tokens (read from the workspace group by group they took 1000 cycles each)
    pdl_wait();
    const int e = tid - 64, n_sm = min(*p.n_out, SM_OUT);
    for (int i = e; i < p.bt; i += 128) s_sca[i] = m0 + i < p.M ? p.sca[m0 + i] : 0.f;
    for (int i = e; i < n_sm * (p.bt / 8); i += 128) {
      const int j = i / (p.bt / 8), c = (i - j * (p.bt / 8)) * 8;
      if (m0 + c < p.Mp) *reinterpret_cast<uint4*>(&s_act[j][c]) = *reinterpret_cast<const uint4*>(p.aout + (size_t)j * p.Mp + m0 + c);
    }
    asm volatile("bar.sync 1, 128;" ::: "memory");
    mbar_wait(bar_acc, 0, dead);
    fence_after();
    if (dead) failed = 1u;
  }
  __syncwarp();
  // ---- epilogue: a thread owns weight row n, 16 tokens at a time; split K: slices of 16 tokens are summed by one CTA each
  const int q = warp & 3, row = q * 32 + lane, n = n0 + row, nb = p.bt / 16;
  if (p.splits > 1) {
    // stage memory is free (every MMA has completed): int32 [token group][128 rows][16 tokens]; rows of 64 bytes, the 16-byte piece
    // rotated by the row so that a warp's stores touch every bank
    if (warp >= 2 && !__any_sync(0xffffffffu, dead)) {
      for (int b = 0; b < nb; ++b) {
        uint32_t r[16];
        tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + 16u * b, r);
        const uint32_t dst = sbase + (uint32_t)(b * BN + row) * 64;
#pragma unroll
        for (int c = 0; c < 4; ++c)
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + 16 * ((c + (row >> 1)) & 3)), "r"(r[4 * c]), "r"(r[4 * c + 1]), "r"(r[4 * c + 2]), "r"(r[4 * c + 3]) : "memory");
      }
    }
    cluster_sync_all();
  }
  if (warp >= 2) {
    for (int s = 0; s < p.splits; ++s)
      if (p.splits > 1) dead |= ld_dsmem_u32(smem_u32(&failed), (uint32_t)s);
    const int n_out = *p.n_out;
    const float scb = n < p.N ? p.scb[n] : 0.f, wsc = scb / 127.0f;
    const int8_t* cbrow = p.cb + (size_t)min(n, p.N - 1) * p.K;
    // outlier weights by eights: their loads, and those of the activations below, travel together (one by one the six outlier columns of
    // 137 x 4096 -> 11008 took 30 of the kernel's 44 us); the first eight stay for all token groups
    float w_first[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) w_first[u] = u < n_out ? __half2float(__float2half_rn((float)cbrow[p.list[u]] * wsc)) : 0.f;
    for (int b = (int)rank; b < nb; b += p.splits) {
      __syncwarp();
      int t[16];
      if (p.splits == 1) {
        uint32_t r[16];
        tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + 16u * b, r);
#pragma unroll
        for (int i = 0; i < 16; ++i) t[i] = (int)r[i];
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) t[i] = 0;
        for (int s = 0; s < p.splits; ++s) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const uint4 v = ld_dsmem(sbase + (uint32_t)(b * BN + row) * 64 + 16 * ((c + (row >> 1)) & 3), (uint32_t)s);
            t[4 * c] += (int)v.x; t[4 * c + 1] += (int)v.y; t[4 * c + 2] += (int)v.z; t[4 * c + 3] += (int)v.w;
          }
        }
      }
      const int m = m0 + 16 * b;
      if (n < p.N && m < p.M) {
        float term[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) term[i] = 0.f;
        const int n_ws = min(n_out, WS_OUT);
        for (int j0 = 0; j0 < n_ws; j0 += 8) {       // ascending k, one fma each: the order of the single-row kernel
          float w[8];
          uint4 act[8][2];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            if (j0 + u < n_ws) {
              // the same for the whole warp
              const uint4* ap = reinterpret_cast<const uint4*>(j0 + u < SM_OUT ? &s_act[j0 + u][16 * b] : p.aout + (size_t)(j0 + u) * p.Mp + m);
              act[u][0] = ap[0];
              act[u][1] = ap[1];
              w[u] = j0 == 0 ? w_first[u] : __half2float(__float2half_rn((float)cbrow[p.list[j0 + u]] * wsc));
            }
          }
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            if (j0 + u < n_ws) {
              const uint32_t aw[8] = {act[u][0].x, act[u][0].y, act[u][0].z, act[u][0].w, act[u][1].x, act[u][1].y, act[u][1].z, act[u][1].w};
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&aw[i]));
                term[2 * i] = fmaf(f.x, w[u], term[2 * i]);
                term[2 * i + 1] = fmaf(f.y, w[u], term[2 * i + 1]);
              }
            }
          }
        }
        for (int j = WS_OUT; j < n_out; ++j) {
          const int k = p.list[j];
          const float w = __half2float(__float2half_rn((float)cbrow[k] * wsc));
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (m + i < p.M) term[i] = fmaf(__half2float(__float2half_rn(bf2f(p.x[(size_t)(m + i) * p.ldx + k]))), w, term[i]);
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          if (m + i >= p.M) break;
          const float sca = s_sca[16 * b + i];
          float v = __half2float(__float2half_rn((float)t[i] * (sca * scb * (1.0f / (127.0f * 127.0f)))));
          if (n_out > 0) v = __half2float(__float2half_rn(v + __half2float(__float2half_rn(term[i]))));
          if (dead) v = __int_as_float(0x7fc00000);
          p.y[(size_t)(m + i) * p.ldy + n] = f2bf(v);
        }
      }
    }
  }
  __syncwarp();
  if (p.splits > 1) cluster_sync_all();              // nobody leaves while a peer reads its partial sums
  fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, cols);
}

constexpr size_t MOST_SMEM = 201 * 1024;
struct Plan { int bt, m_tiles, splits, nst; size_t smem; };
// Tiles of equal height and a split of K over clusters, by a model of the time in ns.  A CTA takes 4400, 210 per stage of 128 k, and per token of its tile
// 85 for the epilogue's roundings (a rank of a split stores its share) and 1.6 per stage; two CTAs on an SM (tiles of up to 128 tokens) take 1.2 times
// one's time, a last one alone 0.95; a split in 2, 4, 8 adds 3000, 3900, 4800 for its barriers and 3 per token and rank.  Device time in us, one row of
// tiles and the plan so: 137 x 4096 -> 12288 29 / 21, 300 x 4096 -> 12288 58 / 32, 512 x 4096 -> 11008 88 / 58, 256 x 5120 -> 5120 31 / 22, 1000 x 4096 ->
// 4096 46 / 34; up to 64 tokens the plans are mostly the same (16 x 4096 -> 11008 13.3).
static Plan plan_for(int M, int N, int K) {
  static std::atomic<int> known[9];
  const int sms = sm_count(), n_tiles = (N + BN - 1) / BN, least = (M + 255) / 256;
  Plan q{};
  long long best = -1;
  for (int mt = least; mt <= least + 4; ++mt) {
    const int bt = ((M + mt - 1) / mt + 15) / 16 * 16, tiles = n_tiles * ((M + bt - 1) / bt), two = bt <= 128;
    for (int sp = 1; sp <= 8; sp *= 2) {
      const int stages = (K / BK + sp - 1) / sp, at_once = clusters_at_once(q8_gemm_kernel, NTHREADS, sp, sms, known);
      if (sp > 1 && (K / BK / sp < 4 || tiles > at_once * (two && sp == 2 ? 2 : 1))) break;      // a split only where its clusters run at once; four and eight alone on their SMs
      const long long one = 4400 + 210 * stages + bt * (85 / sp + 16 * stages / 10), deep = ((long long)tiles * sp + sms - 1) / sms;
      const long long cost = (deep == 1 ? one : two ? one * (deep / 2 * 24 + deep % 2 * 19) / 20 : one * deep) + (sp == 1 ? 0 : (sp == 2 ? 3000 : sp == 4 ? 3900 : 4800) + 3 * bt * sp);
      if (best < 0 || cost < best) {
        best = cost;
        q.bt = bt; q.m_tiles = (M + bt - 1) / bt; q.splits = sp;
      }
    }
  }
  const size_t stage = A_BYTES + (size_t)q.bt * BK;
  // Two CTAs per SM for tiles of up to 128 tokens, one's epilogue under the other's loads: half of an SM's 228 KB less the 1 KB the system
  // keeps per CTA, the static arrays and the alignment of the stages.  Wider tiles take one.
  constexpr size_t STATIC = sizeof(__half) * SM_OUT * 256 + sizeof(float) * 256 + 8 * (2 * MAX_STAGES + 4);
  const size_t budget = q.bt <= 128 ? 114 * 1024 - 1024 - STATIC - 1024 : MOST_SMEM - 1024;
  q.nst = (int)(budget / stage);
  if (q.nst > MAX_STAGES) q.nst = MAX_STAGES;
  q.smem = q.nst * stage + 1024;
  const size_t part = (size_t)BN * q.bt * 4 + 1024;                  // partial sums of a split
  if (q.splits > 1 && part > q.smem) q.smem = part;
  return q;
}
static size_t up16(size_t v) { return (v + 255) & ~(size_t)255; }

}  // namespace q8gm
}  // namespace b2l

using namespace b2l;
using namespace b2l::q8gm;

static inline int slab_rows(int M) { return M < SLAB ? M : SLAB; }

// Of one slab of rows: int8 rows, scales, activations of the first outlier columns; the list of outlier columns and their mask.
extern "C" size_t b2l_q8_linear_workspace_bytes(int M, int K) {
  if (M <= 0 || K <= 0) return 0;
  const size_t R = (size_t)slab_rows(M), Rp = (R + 15) / 16 * 16;
  return up16(R * K) + up16(Rp * 4) + up16(WS_OUT * Rp * 2) + up16((size_t)K * 4) + up16((size_t)(K + 31) / 32 * 4) + 256;
}

extern "C" int b2l_q8_linear(const void* x, int ldx, const void* cb, const void* scb, void* y, int ldy, void* workspace, int M, int N, int K, float threshold,
                             b2l_stream_t stream) {
  B2L_CHECK_ARG(x && cb && scb && y && workspace, "b2l_q8_linear: null pointer");
  B2L_CHECK_ARG(M > 0 && N > 0 && ldx >= K && ldx % 8 == 0 && ldy >= N, "b2l_q8_linear: bad shape");
  B2L_CHECK_SUPPORTED(K > 0 && K % BK == 0 && K <= MAX_K, "b2l_q8_linear: K=%d must be a multiple of %d and <= %d", K, BK, MAX_K);
  B2L_CHECK_ARG((((uintptr_t)x | (uintptr_t)cb | (uintptr_t)workspace) % 16) == 0, "b2l_q8_linear: x, cb and workspace must be 16-byte aligned");
  cudaStream_t s = (cudaStream_t)stream;
  const int R = slab_rows(M), Rp = (R + 15) / 16 * 16;
  uint8_t* w = (uint8_t*)workspace;
  int8_t* xq = (int8_t*)w;              w += up16((size_t)R * K);
  float* sca = (float*)w;               w += up16((size_t)Rp * 4);
  __half* aout = (__half*)w;            w += up16((size_t)WS_OUT * Rp * 2);
  int* list = (int*)w;                  w += up16((size_t)K * 4);
  uint32_t* mask = (uint32_t*)w;        w += up16((size_t)(K + 31) / 32 * 4);
  int* n_out = (int*)w;
  q8_mask_kernel<<<(K + 63) / 64, 256, 0, s>>>((const __nv_bfloat16*)x, ldx, M, K, threshold, mask);      // outlier columns are the whole batch's
  B2L_LAUNCH_CHECK("q8_mask_kernel");
  static DynSmemCache smem_cache;
  if (int rc = ensure_dyn_smem(q8_gemm_kernel, MOST_SMEM, smem_cache)) return rc;
  for (int at = 0; at < M; at += SLAB) {
    const int rows = M - at < SLAB ? M - at : SLAB;
    const Plan q = plan_for(rows, N, K);
    Params p;
    if (int rc = map_sw128(&p.wmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, cb, N, K, K, BK, BN)) return rc;
    if (int rc = map_sw128(&p.xmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, xq, rows, K, K, BK, q.bt)) return rc;
    p.x = (const __nv_bfloat16*)x + (size_t)at * ldx;
    p.y = (__nv_bfloat16*)y + (size_t)at * ldy;
    LaunchCfg lr(dim3((unsigned)rows), dim3(ROW_THREADS), 0, s, true, 1);      // each kernel is launched while the one before it runs, and waits for it where it reads its results
    B2L_CUDA(cudaLaunchKernelEx(&lr.cfg, q8_rows_kernel, p.x, ldx, K, (int)Rp, (const uint32_t*)mask, xq, sca, aout, list, n_out));
    p.cb = (const int8_t*)cb; p.scb = (const float*)scb; p.sca = sca; p.aout = aout; p.list = list; p.n_out = n_out;
    p.M = rows; p.N = N; p.K = K; p.Mp = Rp; p.ldx = ldx; p.ldy = ldy; p.bt = q.bt; p.nst = q.nst; p.splits = q.splits;
    LaunchCfg lc(dim3((unsigned)((N + BN - 1) / BN * q.splits), (unsigned)q.m_tiles), dim3(NTHREADS), q.smem, s, true, q.splits);
    B2L_CUDA(cudaLaunchKernelEx(&lc.cfg, q8_gemm_kernel, p));
  }
  return 0;
}
