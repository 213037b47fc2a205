// Prompt-shaped int4 weight-only GEMM on the 5th-generation tensor cores: y[M, N] = x[M, K] . dequant(W)[N, K]^T for M > 16 (prompt
// processing, no-cache forward, evaluation).
//
// Replaces ColBlockQuantizedLinear.forward (lit_llama/quantization.py:413-423) and the Triton kernel linear_kernel_4bit_weight
// (quantization.py:187-333: tiles up to 256 x 256, dequantise inside the tile loop) for 4-bit weights with one (scale, zero) per row.
//
// A CTA computes 128 output features x `bt` tokens (16..256), the WEIGHT as the 128-row operand in tensor memory:
//   warp 0       TMA: per 64-wide k stage the 4 KB of packed levels (load-time tiling b2l_q4_tile: contiguous) and the activation tile
//                [bt tokens][64 k] as one 128-byte swizzled box, on one mbarrier; rows beyond M are zero-filled by the TMA unit
//   warps 4..19  four groups, a stage each in turn: a thread owns one weight row: LDS.128 of 32 levels, nibble order chosen so that
//                (w >> 4s) & 0x000f000f | 0x43004300 IS the bf16 pair (128 + level[k], 128 + level[k+1]), then level - zero and * scale with
//                get_weight's own bf16 roundings (quantization.py:392-411), so the product sees exactly the matrix the reference's dense
//                branch multiplies; tcgen05.st into the stage's 32 columns
//   warp 1       tcgen05.mma.cta_group::1.kind::f16, A from tensor memory, B from shared memory, M 128, N bt, K 16
//   afterwards the dequantising warps are the epilogue: tcgen05.ld, bf16, a warp writes 32 neighbouring features per token.
//
// Why this form: with both operands in shared memory a 256 x 256 tile moves 160 bytes per cycle through it (dequantised weights written
// and read, activations written and read) where 128 fit, and held the tensor pipe at 42 % (4096 x 5120 -> 5120: 291 us on the device,
// now 168 under the profiler); a prompt of 203 tokens gave 86 CTAs that each dequantised every second weight row twice (4096 -> 11008: 45 us, now 28).
// What bounds it now is L2: a stage of bt = 240 brings 35 KB to the SM in some 750 cycles (480 of them the tensor pipe's).  Where tiles
// are few a cluster of up to 8 CTAs splits K and adds its f32 sums through distributed shared memory in rank order (the result does not
// depend on timing).
#include "tc_common.cuh"

namespace b2l {
namespace q4gm {

using namespace tc;

constexpr int BN = 128, BK = 64;
constexpr int W_BYTES = BN * BK / 2;           // packed levels of a stage
constexpr int GROUPS = 4, NTHREADS = 128 + 128 * GROUPS;
constexpr int MAX_STAGES = 8, A_COLS = BK / 2;      // a stage owns a weight buffer of 32 tensor-memory columns; the accumulator follows from COL_ACC on
constexpr int COL_ACC = 512 - 256;

struct Params {
  CUtensorMap xmap;        // x as 2-D, boxes of 64 columns x bt rows; must stay the first member (64-byte alignment)
  const uint8_t* qwt;      // b2l_q4_tile layout: [N/128 tiles][K/32 slabs][128 rows][16 B]
  const void* scales; const void* zeros; int szdt;
  __nv_bfloat16* y; int ldy;
  int M, N, K, bt, nst, splits;
  int expired;             // cluster rank that ends as if its last wait had run out, or -1
};

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t mbar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(mbar) : "memory");
}
__global__ void __launch_bounds__(NTHREADS, 1) q4_gemm_kernel(const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[3 * MAX_STAGES + 2];
  __shared__ uint32_t tmem_slot, failed;
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;            // 128-byte swizzle atoms are 1024-byte aligned
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t full = smem_u32(bars), empty = full + 8 * MAX_STAGES, a_full = empty + 8 * MAX_STAGES, acc_done = a_full + 8 * MAX_STAGES,
                 gave_up = acc_done + 8;
  const uint32_t stage_bytes = W_BYTES + (uint32_t)p.bt * (BK * 2);
  const int tile_n = blockIdx.x / p.splits, n0 = tile_n * BN, m0 = blockIdx.y * p.bt;
  const uint32_t rank = p.splits > 1 ? cluster_rank() : 0u;
  const int n_kt = p.K / BK, kt_lo = (int)((long long)rank * n_kt / p.splits), kt_hi = (int)((long long)(rank + 1) * n_kt / p.splits);
  uint32_t dead = 0;

  if (tid == 0) {
    for (int i = 0; i < p.nst; ++i) { mbar_init(full + 8 * i, 1); mbar_init(empty + 8 * i, 1); mbar_init(a_full + 8 * i, 4); }
    mbar_init(acc_done, 1);
    mbar_init(gave_up, 1);
    failed = 0u;
    mbar_init_fence();
  }
  if (warp == 1) tmem_alloc(smem_u32(&tmem_slot), 512);
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      const uint8_t* wsrc = p.qwt + ((size_t)tile_n * (p.K / 32) + (size_t)kt_lo * 2) * 2048;
      int st = 0;
      uint32_t ph = 1;                                       // parity of a stage's previous use: passes at once the first time
      for (int kt = kt_lo; kt < kt_hi; ++kt, wsrc += W_BYTES) {
        mbar_wait(empty + 8 * st, ph, dead);
        if (dead) break;
        const uint32_t base = sbase + st * stage_bytes;
        mbar_expect_tx(full + 8 * st, stage_bytes);
        bulk_load(base, wsrc, W_BYTES, full + 8 * st);
        tma_load_2d(base + W_BYTES, &p.xmap, kt * BK, m0, full + 8 * st);
        if (++st == p.nst) { st = 0; ph ^= 1u; }
      }
      uint32_t late = 0;
      for (int i = 0; i < p.nst; ++i) {                      // no copy outlives the CTA; all have landed unless a wait ran out
        mbar_wait(full + 8 * st, ph, late);
        if (++st == p.nst) { st = 0; ph ^= 1u; }
      }
    }
  } else if (warp == 1) {
    const uint32_t lead = elect_lane();
    // kind::f16: D = f32, A = B = bf16 (K-major), 128 x bt
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.bt >> 3) << 17) | ((uint32_t)(BN >> 4) << 24);
    int st = 0;
    uint32_t ph = 0, acc = 0;
    for (int kt = kt_lo; kt < kt_hi; ++kt) {
      mbar_wait(full + 8 * st, ph, dead);
      mbar_wait_warp(a_full + 8 * st, ph, dead);
      if (dead) break;
      fence_after();
      const uint64_t bd = desc_sw128(sbase + st * stage_bytes + W_BYTES);
      const uint32_t ad = tmem + st * A_COLS;
#pragma unroll
      for (int k = 0; k < BK / 16; ++k) mma_ts(tmem + COL_ACC, ad + 8 * k, bd + 2 * k, idesc, k > 0 ? 1u : acc, lead);
      acc = 1;
      if (lead) commit(empty + 8 * st);                      // one per stage: it frees both halves, and each holds the pipe up for 100 cycles
      __syncwarp();
      if (++st == p.nst) { st = 0; ph ^= 1u; }
    }
    if (lead) commit(dead ? gave_up : acc_done);
    if (dead) {
      uint32_t late = 0;
      mbar_wait(gave_up, 0, late);
    }
  } else if (warp >= 4) {
    const int qtr = warp & 3, grp = (warp >> 2) - 1, row = qtr * 32 + lane, n = n0 + row;
    const uint32_t lane_at = (uint32_t)(qtr * 32) << 16;
    float sc_f = 0.f, z_f = 0.f;
    if (n < p.N) { sc_f = load_sz(p.scales, p.szdt, n); z_f = load_sz(p.zeros, p.szdt, n); }
    const __nv_bfloat162 sc2 = __float2bfloat162_rn(sc_f), z2 = __float2bfloat162_rn(z_f), c128 = __float2bfloat162_rn(128.f);
    int st = grp;
    uint32_t ph = 0;
    if (st >= p.nst) { st -= p.nst; ph ^= 1u; }
    for (int it = grp; it < kt_hi - kt_lo; it += GROUPS) {
      mbar_wait(full + 8 * st, ph, dead);                    // also: the MMAs of the stage's previous use are done
      uint32_t w[8];
      const uint32_t src = sbase + st * stage_bytes + row * 16;
#pragma unroll
      for (int h = 0; h < 2; ++h)
        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(w[4 * h]), "=r"(w[4 * h + 1]), "=r"(w[4 * h + 2]), "=r"(w[4 * h + 3]) : "r"(src + h * 2048) : "memory");
      fence_after();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t o[16];
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int s = 0; s < 4; ++s) {
            const uint32_t v = ((w[4 * h + c] >> (4 * s)) & 0x000f000fu) | 0x43004300u;      // (128 + level) pair, exact
            __nv_bfloat162 t = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&v), c128);     // level, exact
            t = __hmul2(__hsub2(t, z2), sc2);                                                 // the reference's bf16 roundings
            o[4 * c + s] = *reinterpret_cast<const uint32_t*>(&t);
          }
        tmem_st16(tmem + lane_at + st * A_COLS + 16 * h, o);
      }
      tmem_wait_st();
      fence_before();
      __syncwarp();
      if (lane == 0 && !dead) mbar_arrive(a_full + 8 * st);
      st += GROUPS;
      if (st >= p.nst) { st -= p.nst; ph ^= 1u; }
    }
    mbar_wait(acc_done, 0, dead);
    fence_after();
    if (p.expired == (int)rank) dead = 1u;
    if (dead) failed = 1u;
  }
  __syncwarp();
  // ---- epilogue: a thread owns weight row n, 16 tokens at a time, the groups in turn; split K: a token group is summed by one CTA
  const int qtr = warp & 3, grp = (warp >> 2) - 1, row = qtr * 32 + lane, n = n0 + row, nb = p.bt / 16;
  const uint32_t acc_at = tmem + ((uint32_t)(qtr * 32) << 16) + COL_ACC;
  if (p.splits > 1) {
    // stage memory is free (every MMA has completed): f32 [token group][128 rows][16 tokens], the 16-byte pieces of a row rotated
    if (warp >= 4 && !__any_sync(0xffffffffu, dead)) {
      for (int b = grp; b < nb; b += GROUPS) {
        uint32_t r[16];
        tmem_ld16(acc_at + 16 * b, r);
        const uint32_t dst = sbase + (uint32_t)(b * BN + row) * 64;
#pragma unroll
        for (int c = 0; c < 4; ++c)
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + 16 * ((c + (row >> 1)) & 3)), "r"(r[4 * c]), "r"(r[4 * c + 1]), "r"(r[4 * c + 2]), "r"(r[4 * c + 3]) : "memory");
      }
    }
    __syncwarp();
    cluster_sync_all();
  }
  if (warp >= 4) {
    for (int s = 0; s < p.splits; ++s)
      if (p.splits > 1) dead |= ld_dsmem_u32(smem_u32(&failed), (uint32_t)s);
    for (int b = (int)rank + grp * p.splits; b < nb; b += GROUPS * p.splits) {
      __syncwarp();
      float v[16];
      if (p.splits == 1) {
        uint32_t r[16];
        tmem_ld16(acc_at + 16 * b, r);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = 0.f;
        for (int s = 0; s < p.splits; ++s) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const uint4 u = ld_dsmem(sbase + (uint32_t)(b * BN + row) * 64 + 16 * ((c + (row >> 1)) & 3), (uint32_t)s);
            v[4 * c] += __uint_as_float(u.x); v[4 * c + 1] += __uint_as_float(u.y); v[4 * c + 2] += __uint_as_float(u.z); v[4 * c + 3] += __uint_as_float(u.w);
          }
        }
      }
      const int m = m0 + 16 * b;
      if (n < p.N) {
        __nv_bfloat16* dst = p.y + (size_t)m * p.ldy + n;
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if (m + i < p.M) dst[(size_t)i * p.ldy] = f2bf(dead ? __int_as_float(0x7fc00000) : v[i]);
      }
    }
  }
  __syncwarp();
  if (p.splits > 1) cluster_sync_all();              // nobody leaves while a peer reads its partial sums
  fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

struct Plan { int bt, m_tiles, splits, nst; size_t smem; };
// Tile height and K split by a model of the time in tensor cycles: rounds of CTAs over the SMs times (stages of max(2 bt, the 200 a stage's
// dequantisation takes) + a fixed part: first copies, epilogue, and the sums of a split).
static Plan plan_for(int M, int N, int K) {
  const int sms = sm_count(), n_tiles = (N + BN - 1) / BN, n_kt = K / BK;
  Plan best{};
  long long best_cost = -1;
  const int least = (M + 255) / 256;
  for (int mt = least; mt <= least + 3; ++mt) {
    const int bt = ((M + mt - 1) / mt + 15) / 16 * 16, tiles = (M + bt - 1) / bt;
    for (int sp = 1; sp <= 8; ++sp) {
      if (sp > 1 && n_kt / sp < 8) break;
      const long long ctas = (long long)n_tiles * tiles * sp, rounds = (ctas + sms - 1) / sms;
      const long long stages = (n_kt + sp - 1) / sp, per = bt * 2 > 200 ? bt * 2 : 200;
      const long long cost = rounds * (stages * per + 3000 + 8 * bt + (sp > 1 ? 1500 + 10 * bt : 0));
      if (best_cost < 0 || cost < best_cost) {
        best_cost = cost;
        best.bt = bt; best.m_tiles = tiles; best.splits = sp;
      }
    }
  }
  const size_t stage = W_BYTES + (size_t)best.bt * BK * 2;
  best.nst = (int)(216 * 1024 / stage);
  if (best.nst > MAX_STAGES) best.nst = MAX_STAGES;
  best.smem = best.nst * stage + 1024;
  const size_t part = (size_t)BN * best.bt * 4 + 1024;
  if (best.splits > 1 && part > best.smem) best.smem = part;
  // One CTA per SM by its shared memory, whatever its registers: each takes all of tensor memory, and a CTA of a cluster that waited for another's
  // would wait for good if that one waits for it at the cluster's barrier.
  if (best.smem < 120 * 1024) best.smem = 120 * 1024;
  return best;
}

}  // namespace q4gm
}  // namespace b2l

using namespace b2l;
using namespace b2l::q4gm;

extern "C" int b2l_q4_gemm(const b2l_q4_linear_args* a, b2l_stream_t stream) {
  B2L_CHECK_ARG(a != nullptr, "b2l_q4_gemm: null args");
  B2L_CHECK_ARG(a->x && a->qw_tiled && a->scales && a->zeros && a->y, "b2l_q4_gemm: null pointer");
  B2L_CHECK_ARG(a->M > 0 && a->N > 0 && a->K > 0, "b2l_q4_gemm: bad shape");
  B2L_CHECK_SUPPORTED(a->K % BK == 0, "b2l_q4_gemm: K=%d must be a multiple of %d", a->K, BK);
  B2L_CHECK_ARG(a->ldx >= a->K && a->ldx % 8 == 0 && a->ldy >= a->N, "b2l_q4_gemm: bad leading dimension (ldx %% 8 == 0)");
  B2L_CHECK_ARG(((uintptr_t)a->x % 16 == 0) && ((uintptr_t)a->qw_tiled % 16 == 0), "b2l_q4_gemm: x / qw_tiled must be 16-byte aligned");
  B2L_CHECK_ARG(a->sz_dtype == B2L_BF16 || a->sz_dtype == B2L_F32, "b2l_q4_gemm: bad sz_dtype");
  B2L_CHECK_SUPPORTED(a->prologue == B2L_PRO_NONE && a->epilogue == B2L_EPI_STORE, "b2l_q4_gemm: plain linear only (no fused prologue / epilogue)");
  const Plan q = plan_for(a->M, a->N, a->K);
  Params p;
  if (int rc = map_sw128(&p.xmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a->x, a->M, a->K, a->ldx, BK, q.bt)) return rc;
  p.qwt = (const uint8_t*)a->qw_tiled;
  p.scales = a->scales; p.zeros = a->zeros; p.szdt = a->sz_dtype;
  p.y = (__nv_bfloat16*)a->y; p.ldy = a->ldy;
  p.M = a->M; p.N = a->N; p.K = a->K; p.bt = q.bt; p.nst = q.nst; p.splits = q.splits;
  p.expired = (a->flags >> B2L_F_EXPIRED_SHIFT & 15) - 1;
  static DynSmemCache smem_cache;
  if (int rc = ensure_dyn_smem(q4_gemm_kernel, q.smem, smem_cache)) return rc;
  LaunchCfg lc(dim3((unsigned)((a->N + BN - 1) / BN * q.splits), (unsigned)q.m_tiles), dim3(NTHREADS), q.smem, (cudaStream_t)stream, false, q.splits);
  B2L_CUDA(cudaLaunchKernelEx(&lc.cfg, q4_gemm_kernel, p));
  return 0;
}
