// Prompt-shaped int4 weight-only GEMM on the 5th-generation tensor cores: y[M, N] = x[M, K] . dequant(W)[N, K]^T for M > 8 (prompt
// processing, no-cache forward, evaluation, linears of 9..16 sequences; a tile has 16 tokens or more, so 9..16 rows take as long as 17 less the extra tile).
//
// Replaces ColBlockQuantizedLinear.forward (lit_llama/quantization.py:413-423) and the Triton kernel linear_kernel_4bit_weight
// (quantization.py:187-333: tiles up to 256 x 256, dequantise inside the tile loop) for 4-bit weights with one (scale, zero) per row.
//
// Work is in items of 128 output features x `bt` tokens (16..256), the WEIGHT as the 128-row operand in tensor memory; a CTA takes items in turn.
// Operands move in units of 128 k:
//   warp 0       TMA: the activation tile [bt tokens][128 k] as two 128-byte swizzled boxes, three or four units in flight; rows beyond M are zero-filled
//   warp 2       TMA: the 8 KB of packed levels (load-time tiling b2l_q4_tile: contiguous), four or eight units ahead
//   warps 4..19  four groups, a unit each in turn: a thread owns one weight row: LDS.128 of 32 levels, nibbles as bf16 subnormals, so that one fma gives
//                level - zero and one product the weight, with get_weight's own bf16 roundings (quantization.py:392-411): the product sees exactly the
//                matrix the reference's dense branch multiplies; tcgen05.st into the unit's 64 columns
//   warp 1       tcgen05.mma.cta_group::1.kind::f16, A from tensor memory, B from shared memory, M 128, N bt, K 16: one barrier (activations landed and
//                weights stored) and one commit per unit
//   warps 20..27 the epilogue: tcgen05.ld, bf16, a warp writes 32 neighbouring features per token, while the next item's operands are on their way
//                (two accumulators where bt <= 128); of a CTA's last item the dequantising warps store a share.
//
// Why this form: with both operands in shared memory a 256 x 256 tile moves 160 bytes per cycle through it (dequantised weights written
// and read, activations written and read) where 128 fit, and held the tensor pipe at 42 % (4096 x 5120 -> 5120: 291 us on the device);
// a prompt of 203 tokens gave 86 CTAs that each dequantised every second weight row twice.
// What bounds it: from some 200 tokens per tile on the tensor pipe and the power it may draw (148 tiles of 256: 346 ns per 64 k, 512 cycles at the 1.5 GHz
// the chip then keeps; 4096 x 5120 -> 5120 163 -> 153 us); below that the issuing warp and the dequantisation (64 tokens: 200 ns per 64 k).  A barrier that is
// complete still costs the issuing warp 120..190 cycles beside four dequantising warps on its scheduler, and a bf16x2 operation takes a scheduler two
// cycles: units of 128 k instead of 64, one barrier for both operands and two operations per pair of weights instead of three took 64 tokens from 280 to
// 200 ns per 64 k (device time of 64 / 512 / 777 x 4096 -> 11008: 23.2 / 50.9 / 74.7 -> 16.8 / 41.9 / 55.7 us).  Where tiles are few a cluster of up to
// 8 CTAs splits K and adds its f32 sums through distributed shared memory in rank order (the result does not depend on timing).
#include "tc_common.cuh"

namespace b2l {
namespace q4gm {

using namespace tc;

constexpr int BN = 128, BK = 64, UNIT = 2 * BK;      // k of an activation box, and of a pipeline unit (the last one of an odd count is half full)
constexpr int W_BYTES = BN * UNIT / 2;         // packed levels of a unit
constexpr int GROUPS = 4, EPI = 2, NTHREADS = 128 + 128 * (GROUPS + EPI);
constexpr int A_BUFS = 4, A_COLS = UNIT / 2, MAX_W = 8;      // a weight buffer is 64 tensor-memory columns; accumulators follow from COL_ACC on
constexpr int COL_ACC = 512 - 256;

struct Params {
  CUtensorMap xmap;        // x as 2-D, boxes of 64 columns x bt rows; must stay the first member (64-byte alignment)
  const uint8_t* qwt;      // b2l_q4_tile layout: [N/128 tiles][K/32 slabs][128 rows][16 B]
  const void* scales; const void* zeros; int szdt;
  __nv_bfloat16* y; int ldy;
  int M, N, K, bt, nx, nw, splits, n_tiles, items;
  int expired;             // cluster rank that ends as if its last wait had run out, or -1
};

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t mbar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(mbar) : "memory");
}
__global__ void __launch_bounds__(NTHREADS, 1) q4_gemm_kernel(const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[2 * MAX_W + 2 * A_BUFS + 6];
  __shared__ uint32_t tmem_slot, failed;
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;            // 128-byte swizzle atoms are 1024-byte aligned
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t w_full = smem_u32(bars), w_empty = w_full + 8 * MAX_W, full = w_empty + 8 * MAX_W, done = full + 8 * A_BUFS, acc_full = done + 8 * A_BUFS,
                 acc_empty = acc_full + 16, gave_up = acc_empty + 16, last_full = gave_up + 8;
  const uint32_t box = (uint32_t)p.bt * (BK * 2), wbase = sbase + p.nx * 2 * box;
  const uint32_t rank = p.splits > 1 ? cluster_rank() : 0u;
  const int n_kt = p.K / BK, kt_lo = (int)((long long)rank * n_kt / p.splits), kt_hi = (int)((long long)(rank + 1) * n_kt / p.splits), nk = kt_hi - kt_lo;
  // a CTA takes items blockIdx.x, + gridDim.x, ...; its units are counted through all of them.  Split K: one item for the whole cluster.
  const int item0 = p.splits > 1 ? (int)(blockIdx.x / p.splits) : (int)blockIdx.x, step = p.splits > 1 ? p.items : (int)gridDim.x;
  const int accs = p.bt <= 128 ? 2 : 1;                                    // accumulators in turn, or one
  uint32_t dead = 0;

  if (tid == 0) {
    for (int i = 0; i < p.nw; ++i) { mbar_init(w_full + 8 * i, 1); mbar_init(w_empty + 8 * i, 4); }
    for (int i = 0; i < A_BUFS; ++i) { mbar_init(full + 8 * i, 5); mbar_init(done + 8 * i, 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(acc_full + 8 * i, 1); mbar_init(acc_empty + 8 * i, 4 * EPI); }      // nobody waits for the last item's
    mbar_init(gave_up, 1);
    mbar_init(last_full, 1);
    failed = 0u;
    mbar_init_fence();
  }
  if (warp == 1) tmem_alloc(smem_u32(&tmem_slot), 512);
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = tmem_slot;

  // output of the CTA's n-th item, its 16-token groups first, first + stride, ...: a thread owns weight row 32 (warp % 4) + lane
  auto put = [&](int item, int n, int first, int stride, uint32_t bar, uint32_t parity) {
    const int qtr = warp & 3, ab = accs == 2 ? n & 1 : 0, row = item % p.n_tiles * BN + qtr * 32 + lane, m0 = item / p.n_tiles * p.bt;
    mbar_wait_warp(bar, parity, dead);
    fence_after();
    const bool lost = dead || p.expired == 0;
    const uint32_t at = tmem + ((uint32_t)(qtr * 32) << 16) + COL_ACC + 128 * ab;
#pragma unroll 1
    for (int b = first; b < p.bt / 16; b += stride) {
      uint32_t r[16];
      __syncwarp();
      tmem_ld16(at + 16 * b, r);
      const int m = m0 + 16 * b;
      if (row < p.N) {
        __nv_bfloat16* dst = p.y + (size_t)m * p.ldy + row;
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if (m + i < p.M) dst[(size_t)i * p.ldy] = f2bf(lost ? __int_as_float(0x7fc00000) : __uint_as_float(r[i]));
      }
    }
    fence_before();
    __syncwarp();
    if (lane == 0 && !dead) mbar_arrive(acc_empty + 8 * ab);
  };

  if (warp == 0) {
    if (lane == 0) {                                         // activations: unit u on the barrier of its weight buffer; its memory is free when the MMAs
      int u = 0, st = 0;                                     // of unit u - nx are done
      for (int item = item0; item < p.items && !dead; item += step) {
        const int m0 = item / p.n_tiles * p.bt;
        for (int kt = kt_lo; kt < kt_hi; kt += 2, ++u) {
          if (u >= p.nx) mbar_wait(done + 8 * ((u - p.nx) % A_BUFS), (uint32_t)((u - p.nx) / A_BUFS) & 1u, dead);
          if (dead) break;
          const uint32_t bar = full + 8 * (u % A_BUFS), dst = sbase + st * 2 * box;
          const bool two = kt + 1 < kt_hi;
          mbar_expect_tx(bar, two ? 2 * box : box);
          tma_load_2d(dst, &p.xmap, kt * BK, m0, bar);
          if (two) tma_load_2d(dst + box, &p.xmap, kt * BK + BK, m0, bar);
          if (++st == p.nx) st = 0;
        }
      }
      uint32_t late = 0;                                     // no copy outlives the CTA: the latest phases of all barriers, complete unless a wait ran out
      for (int i = max(0, u - A_BUFS); i < u; ++i) mbar_wait(full + 8 * (i % A_BUFS), (uint32_t)(i / A_BUFS) & 1u, late);
    }
  } else if (warp == 2) {
    if (lane == 0) {                                         // packed levels, far ahead: they come from HBM
      int st = 0, u = 0;
      uint32_t ph = 1;                                       // parity of a slot's previous use: passes at once the first time
      for (int item = item0; item < p.items && !dead; item += step) {
        const uint8_t* wsrc = p.qwt + ((size_t)(item % p.n_tiles) * (p.K / 32) + (size_t)kt_lo * 2) * 2048;
        for (int left = nk; left > 0; left -= 2, ++u, wsrc += W_BYTES) {
          const uint32_t bytes = left > 1 ? W_BYTES : W_BYTES / 2;
          mbar_wait(w_empty + 8 * st, ph, dead);
          if (dead) break;
          mbar_expect_tx(w_full + 8 * st, bytes);
          bulk_load(wbase + st * W_BYTES, wsrc, bytes, w_full + 8 * st);
          if (++st == p.nw) { st = 0; ph ^= 1u; }
        }
      }
      uint32_t late = 0;
      for (int i = max(0, u - p.nw); i < u; ++i) mbar_wait(w_full + 8 * (i % p.nw), (uint32_t)(i / p.nw) & 1u, late);
    }
  } else if (warp == 1) {
    const uint32_t lead = elect_lane();
    // kind::f16: D = f32, A = B = bf16 (K-major), 128 x bt
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.bt >> 3) << 17) | ((uint32_t)(BN >> 4) << 24);
    int st = 0, u = 0, n = 0;
    uint32_t ready = 0;                                      // the next unit's operands are there: asked while this one's MMAs are issued
    for (int item = item0; item < p.items; item += step, ++n) {
      const int ab = accs == 2 ? n & 1 : 0, use = accs == 2 ? n >> 1 : n;
      if (use > 0) mbar_wait_warp(acc_empty + 8 * ab, (uint32_t)(use - 1) & 1u, dead);
      const uint32_t d = tmem + COL_ACC + 128 * ab;
      uint32_t acc = 0;
      for (int left = nk; left > 0; left -= 2) {
        const int buf = u % A_BUFS;
        if (!__all_sync(0xffffffffu, ready)) mbar_wait_warp(full + 8 * buf, (uint32_t)(u / A_BUFS) & 1u, dead);
        if (dead) break;
        fence_after();
        ++u;
        ready = mbar_test(full + 8 * (u % A_BUFS), (uint32_t)(u / A_BUFS) & 1u);
        const uint64_t bd = desc_sw128(sbase + st * 2 * box);
        const uint32_t ad = tmem + buf * A_COLS;
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) mma_ts(d, ad + 8 * k, bd + 2 * k, idesc, k > 0 ? 1u : acc, lead);
        acc = 1;
        if (left > 1) {
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) mma_ts(d, ad + A_COLS / 2 + 8 * k, bd + (box >> 4) + 2 * k, idesc, 1u, lead);
        }
        if (lead) commit(done + 8 * buf);                    // frees the weight buffer and the activations' memory
        __syncwarp();
        if (++st == p.nx) st = 0;
      }
      if (dead) break;
      if (lead) {
        commit(acc_full + 8 * ab);
        if (item + step >= p.items) commit(last_full);
      }
      __syncwarp();
    }
    if (dead) {
      uint32_t late = 0;
      if (lead) commit(gave_up);
      mbar_wait(gave_up, 0, late);
    }
  } else if (warp >= 4 && warp < 4 + 4 * GROUPS) {
    const int qtr = warp & 3, grp = (warp >> 2) - 1, row = qtr * 32 + lane;
    const uint32_t lane_at = (uint32_t)(qtr * 32) << 16;
    float sc_f = 0.f, z_f = 0.f;
    auto row_values = [&](int item) {
      const int n = item % p.n_tiles * BN + row;
      const bool in = item < p.items && n < p.N;
      sc_f = in ? load_sz(p.scales, p.szdt, n) : 0.f;
      z_f = in ? load_sz(p.zeros, p.szdt, n) : 0.f;
    };
    int st = grp, turn = grp, u0 = 0;                        // a group takes every fourth unit, counted through all items
    uint32_t ph = 0;
    const int nu = (nk + 1) / 2;
    row_values(item0);
    for (int item = item0; item < p.items; item += step, u0 += nu) {
      // levels as they lie, bf16 subnormals of 2^-133 (low four bits) or 2^-130 (bits 3..6) each, times 2^127: (level - z) 2^-6 or 2^-3 in one fma
      // with get_weight's rounding, since a power of two changes none; its product with scale 2^6 or 2^3 is rounded as the product with scale.
      // Rows whose zero point or scale leaves bf16's normal range so, or is no bf16 number (kept in f32: rounding it first gave sums 0.0037 off, 0.0017 so), look
      // their 16 weights up: get_weight's two roundings of each, low and high bytes in registers.  27 operations for 8 weights where the products take 12: us, bf16 / f32
      // scales, 9 rows of 4096 -> 11008 19 / 28, 203 25 / 31, 2048 135 / 147; 512 rows of 13824 -> 5120 58 / 78.
      const bool fits = (z_f == 0.f || fabsf(z_f) >= 0x1p-100f) && fabsf(sc_f) <= 0x1p100f && rbf(z_f) == z_f && rbf(sc_f) == sc_f, all_fit = __all_sync(0xffffffffu, fits);
      const __nv_bfloat162 up = __float2bfloat162_rn(0x1p127f);
      uint32_t row_w[8];                                     // zero point and scale for levels in the low four bits and in bits 3..6, or the weights' bytes
      if (all_fit) {
        auto pair = [](float v) { const __nv_bfloat162 b = __float2bfloat162_rn(v); return *reinterpret_cast<const uint32_t*>(&b); };
        row_w[0] = pair(z_f * -0x1p-6f); row_w[1] = pair(z_f * -0x1p-3f); row_w[2] = pair(sc_f * 0x1p6f); row_w[3] = pair(sc_f * 0x1p3f);
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint32_t b[4];
#pragma unroll
          for (int l = 0; l < 4; ++l) b[l] = __float_as_uint(rbf(rbf((float)(4 * q + l) - z_f) * sc_f)) >> 16;
          row_w[q] = __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410);
          row_w[4 + q] = __byte_perm(__byte_perm(b[0], b[1], 0x0051), __byte_perm(b[2], b[3], 0x0051), 0x5410);
        }
      }
      row_values(item + step);
      for (; turn < nu; turn += GROUPS) {
        mbar_wait(w_full + 8 * st, ph, dead);
        const int u = u0 + turn, buf = u % A_BUFS, halves = min(2, nk - 2 * turn);
#pragma unroll 1
        for (int h = 0; h < halves; ++h) {
          uint32_t w[8];
          const uint32_t src = wbase + st * W_BYTES + h * (W_BYTES / 2) + row * 16;
#pragma unroll
          for (int i = 0; i < 2; ++i)
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(w[4 * i]), "=r"(w[4 * i + 1]), "=r"(w[4 * i + 2]), "=r"(w[4 * i + 3]) : "r"(src + i * 2048) : "memory");
          if (h + 1 == halves) {                             // the levels are in registers: their memory is free
            __syncwarp();
            if (lane == 0 && !dead) mbar_arrive(w_empty + 8 * st);
          }
          if (h == 0) {
            if (u >= A_BUFS) mbar_wait(done + 8 * buf, (uint32_t)(u / A_BUFS - 1) & 1u, dead);
            fence_after();
          }
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            uint32_t o[16];
            if (all_fit) {
              const __nv_bfloat162 *zl = reinterpret_cast<const __nv_bfloat162*>(row_w), *zh = zl + 1, *sl = zl + 2, *sh = zl + 3;
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                const uint32_t v = w[4 * i + c], lo[2] = {v & 0x000f000fu, (v >> 8) & 0x000f000fu}, hi[2] = {(v >> 1) & 0x00780078u, (v >> 9) & 0x00780078u};
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                  const __nv_bfloat162 l = __hmul2(__hfma2(*reinterpret_cast<const __nv_bfloat162*>(&lo[s]), up, *zl), *sl),
                                       m = __hmul2(__hfma2(*reinterpret_cast<const __nv_bfloat162*>(&hi[s]), up, *zh), *sh);
                  o[4 * c + 2 * s] = *reinterpret_cast<const uint32_t*>(&l);
                  o[4 * c + 2 * s + 1] = *reinterpret_cast<const uint32_t*>(&m);
                }
              }
            } else {
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                const uint32_t v = w[4 * i + c];
                uint32_t e[2][2];                            // the even k's pairs of levels (low half of the word), then the odd k's
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                  const uint32_t at = v >> (16 * s) & 0x7777u, top = __byte_perm(0x0000ff00u, 0u, v >> (16 * s + 3) & 0x1111u);      // levels 8..15: all bits of the byte
                  const uint32_t lo = (__byte_perm(row_w[0], row_w[1], at) & ~top) | (__byte_perm(row_w[2], row_w[3], at) & top),
                                 hi = (__byte_perm(row_w[4], row_w[5], at) & ~top) | (__byte_perm(row_w[6], row_w[7], at) & top);
                  e[s][0] = __byte_perm(lo, hi, 0x5140);
                  e[s][1] = __byte_perm(lo, hi, 0x7362);
                }
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                  o[4 * c + 2 * s] = __byte_perm(e[0][s], e[1][s], 0x5410);
                  o[4 * c + 2 * s + 1] = __byte_perm(e[0][s], e[1][s], 0x7632);
                }
              }
            }
            tmem_st16(tmem + lane_at + buf * A_COLS + 32 * h + 16 * i, o);
          }
        }
        tmem_wait_st();
        fence_before();
        __syncwarp();
        if (lane == 0 && !dead) mbar_arrive(full + 8 * buf);
        st += GROUPS;
        if (st >= p.nw) { st -= p.nw; ph ^= 1u; }
      }
      turn -= nu;                                            // counted from the next item's first unit
    }
    if (p.splits > 1) {
      mbar_wait(acc_full, 0, dead);
      fence_after();
      if (p.expired == (int)rank) dead = 1u;
      if (dead) failed = 1u;
    } else {
      const int n = (p.items - 1 - item0) / step;            // the last item's output together with the other groups
      put(item0 + n * step, n, EPI + grp, EPI + GROUPS, last_full, 0u);      // a barrier of its own: they have not followed the phases of the others
    }
  } else if (warp >= 4 + 4 * GROUPS && p.splits == 1) {
    // the accumulator of an item while the next item's weights are on their way
    const int grp = (warp >> 2) - 1 - GROUPS;
    int n = 0;
    for (int item = item0; item < p.items; item += step, ++n)
      put(item, n, grp, item + step < p.items ? EPI : EPI + GROUPS, acc_full + 8 * (accs == 2 ? n & 1 : 0), (uint32_t)(accs == 2 ? n >> 1 : n) & 1u);
  }
  __syncwarp();
  // ---- split K: a thread owns weight row n, 16 tokens at a time, the groups in turn; a token group is summed by one CTA
  if (p.splits > 1) {
    const int qtr = warp & 3, grp = (warp >> 2) - 1, row = qtr * 32 + lane, n = item0 % p.n_tiles * BN + row, m0 = item0 / p.n_tiles * p.bt, nb = p.bt / 16;
    const bool mine = warp >= 4 && warp < 4 + 4 * GROUPS;
    // stage memory is free (every MMA has completed): f32 [token group][128 rows][16 tokens], the 16-byte pieces of a row rotated
    if (mine && !__any_sync(0xffffffffu, dead)) {
      for (int b = grp; b < nb; b += GROUPS) {
        uint32_t r[16];
        tmem_ld16(tmem + ((uint32_t)(qtr * 32) << 16) + COL_ACC + 16 * b, r);
        const uint32_t dst = sbase + (uint32_t)(b * BN + row) * 64;
#pragma unroll
        for (int c = 0; c < 4; ++c)
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + 16 * ((c + (row >> 1)) & 3)), "r"(r[4 * c]), "r"(r[4 * c + 1]), "r"(r[4 * c + 2]), "r"(r[4 * c + 3]) : "memory");
      }
    }
    __syncwarp();
    cluster_sync_all();
    if (mine) {
      for (int s = 0; s < p.splits; ++s) dead |= ld_dsmem_u32(smem_u32(&failed), (uint32_t)s);
      for (int b = (int)rank + grp * p.splits; b < nb; b += GROUPS * p.splits) {
        __syncwarp();
        float v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = 0.f;
        for (int s = 0; s < p.splits; ++s) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const uint4 u = ld_dsmem(sbase + (uint32_t)(b * BN + row) * 64 + 16 * ((c + (row >> 1)) & 3), (uint32_t)s);
            v[4 * c] += __uint_as_float(u.x); v[4 * c + 1] += __uint_as_float(u.y); v[4 * c + 2] += __uint_as_float(u.z); v[4 * c + 3] += __uint_as_float(u.w);
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
    cluster_sync_all();                              // nobody leaves while a peer reads its partial sums
  }
  fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

constexpr size_t MOST_SMEM = 226 * 1024;
struct Plan { int bt, m_tiles, splits, nx, nw; size_t smem; };
// Tile height and K split by a model of the time in ns: a CTA's items one after the other, each of so many 64-wide stages (60 + 1.15 per token of the
// tile, and no less than the 200 that dequantising and issuing take; 18944 features, 64 / 128 / 208 / 256 tokens: 200 / 209 / 286 / 346) and 1000 for
// each; first copies and the last output once, 4000 and 15 per token.  A split adds 3500 for its barriers and, for every further rank, 12 per token
// (partial sums to and from shared memory; seen: 32 tokens in four 4500, 112 in four 7000, 208 in two 5000), and every round of it starts anew.
static Plan plan_for(int M, int N, int K) {
  static std::atomic<int> known[9];
  const int sms = sm_count(), n_tiles = (N + BN - 1) / BN, n_kt = K / BK;
  Plan best{};
  long long best_cost = -1;
  const int least = (M + 255) / 256;
  for (int mt = least; mt <= least + 3; ++mt) {
    const int bt = ((M + mt - 1) / mt + 15) / 16 * 16, tiles = (M + bt - 1) / bt;
    for (int sp = 1; sp <= 8; ++sp) {
      if (sp > 1 && n_kt / sp < 8) break;
      const int at_once = clusters_at_once(q4_gemm_kernel, NTHREADS, sp, sms, known);
      const long long rounds = (n_tiles * tiles + at_once - 1) / at_once, stages = (n_kt + sp - 1) / sp;
      const long long per = 600 + bt * 23 / 2 > 2000 ? 600 + bt * 23 / 2 : 2000, once = 4000 + 15 * bt;
      const long long cost = sp == 1 ? rounds * (stages * per / 10 + 1000) + once : rounds * (stages * per / 10 + once + 3500 + (sp - 1) * 12 * bt);
      if (best_cost < 0 || cost < best_cost) {
        best_cost = cost;
        best.bt = bt; best.m_tiles = tiles; best.splits = sp;
      }
    }
  }
  // four units of activations where they fit beside eight of weights, three beside four otherwise
  const size_t x = (size_t)best.bt * UNIT * 2, room = MOST_SMEM - 1024;
  best.nx = A_BUFS * x + MAX_W * W_BYTES <= room ? A_BUFS : 3;
  best.nw = best.nx == A_BUFS ? MAX_W : 4;
  best.smem = best.nx * x + best.nw * W_BYTES + 1024;
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
  static DynSmemCache smem_cache;
  if (int rc = ensure_dyn_smem(q4_gemm_kernel, MOST_SMEM, smem_cache)) return rc;
  const Plan q = plan_for(a->M, a->N, a->K);
  Params p;
  if (int rc = map_sw128(&p.xmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a->x, a->M, a->K, a->ldx, BK, q.bt)) return rc;
  p.qwt = (const uint8_t*)a->qw_tiled;
  p.scales = a->scales; p.zeros = a->zeros; p.szdt = a->sz_dtype;
  p.y = (__nv_bfloat16*)a->y; p.ldy = a->ldy;
  p.M = a->M; p.N = a->N; p.K = a->K; p.bt = q.bt; p.nx = q.nx; p.nw = q.nw; p.splits = q.splits;
  p.n_tiles = (a->N + BN - 1) / BN; p.items = p.n_tiles * q.m_tiles;
  p.expired = (a->flags >> B2L_F_EXPIRED_SHIFT & 15) - 1;
  const int ctas = q.splits > 1 ? p.items * q.splits : (p.items < sm_count() ? p.items : sm_count());
  LaunchCfg lc(dim3((unsigned)ctas), dim3(NTHREADS), q.smem, (cudaStream_t)stream, false, q.splits);
  B2L_CUDA(cudaLaunchKernelEx(&lc.cfg, q4_gemm_kernel, p));
  return 0;
}
