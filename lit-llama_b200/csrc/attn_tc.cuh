// Prompt attention on tcgen05 with f32 scores and weights: 128 query rows of one head against tiles of 64 keys.
//
// Keys and values are bf16.  A query in f32 is cut into NQ = 3 bf16 parts that add up to it exactly (8 bits each, by truncation), and so is
// every softmax weight (NP = 3): the products of the parts with bf16 keys or values are exact, the tensor core adds them in f32, so
// the result is that of an f32 kernel up to the order of the sums.  Three bf16 MMAs cost 3 / 16 of what one f32 FMA costs on the CUDA cores.
//
//   warps 0..7   softmax: a thread owns one row (tensor-memory lane) and half of a tile's keys; scores by tcgen05.ld, maxima of the two
//                halves through shared memory, weights back to tensor memory as the A operand of the second product.  The reference
//                maximum of a row moves only when it is exceeded by more than 8 (weights reach e^8; nothing is rounded by that), so the
//                output accumulator is rescaled a few times per row instead of once per tile.
//   warps 8, 9   keys, warps 10, 11 values: rows gathered from the fresh projections or the cache ring by 16-byte cp.async into 128-byte
//                swizzled rows (keys K-major, values MN-major for the second product), two or three stages
//   warp 12      issues the MMAs: S(t+2) = Q K^T goes behind O += P(t) V, so the tensor pipe works while tile t+1 is exponentiated
// Tensor memory: S 2 x 64 columns, O 128, P 2 x 3 x 32.  One CTA per SM.
//
// Bound by the softmax warps and the tensor pipe alike: per 128 x 64 tile 1536 tensor cycles (head size 128) and about 20 instructions
// per score on the CUDA cores.  The f32 kernel on the CUDA cores ran at 9-19 TFLOP/s.
#pragma once
#include "tc_common.cuh"

namespace b2l {
namespace atc {

using namespace tc;

constexpr int ROWS = 128, KEYS = 64;
constexpr int SOFT_WARPS = 8, THREADS = 32 * (SOFT_WARPS + 5);
constexpr int Q_ATOM = ROWS * 128, K_ATOM = KEYS * 128;      // bytes of 64 columns of a query / key / value tile
constexpr uint32_t COL_S = 0, COL_O = 128, COL_P = 256;
constexpr int MAX_DK = 192, MAX_DV = 128;

__host__ __device__ inline int atoms(int d) { return (d + 63) / 64; }
constexpr int CONTROL = 3072;                                // barriers, tensor-memory address, row maxima
struct Layout { int stages; size_t smem; };
static inline Layout layout(int nq, int dk, int dv) {
  Layout l;
  const size_t q = (size_t)nq * atoms(dk) * Q_ATOM, st = (size_t)(atoms(dk) + atoms(dv)) * K_ATOM;
  l.stages = CONTROL + q + 3 * st <= 227 * 1024 ? 3 : 2;
  l.smem = CONTROL + q + l.stages * st;                    // head sizes 192 and 128: all of the 227 KB
  if (l.smem < 120 * 1024) l.smem = 120 * 1024;            // one CTA per SM: each takes all of tensor memory
  return l;
}

__device__ __forceinline__ void cp16(uint32_t dst, const void* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void st_zero16(uint32_t dst) { asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(dst), "r"(0) : "memory"); }
__device__ __forceinline__ void bar_named(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }

__device__ __forceinline__ void mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}
// MN-major operand, 128-byte swizzle: rows of 64 consecutive MN entries, one row per k; `lbo` bytes to the next 64 entries
__device__ __forceinline__ uint64_t desc_mn(uint32_t addr, uint32_t lbo) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
#define B2L_R16(r, o) "=r"(r[o]), "=r"(r[o + 1]), "=r"(r[o + 2]), "=r"(r[o + 3]), "=r"(r[o + 4]), "=r"(r[o + 5]), "=r"(r[o + 6]), "=r"(r[o + 7]), \
                      "=r"(r[o + 8]), "=r"(r[o + 9]), "=r"(r[o + 10]), "=r"(r[o + 11]), "=r"(r[o + 12]), "=r"(r[o + 13]), "=r"(r[o + 14]), "=r"(r[o + 15])
__device__ __forceinline__ void tmem_ld32(uint32_t a, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, "
      "%25, %26, %27, %28, %29, %30, %31}, [%32];"
      : B2L_R16(r, 0), B2L_R16(r, 16)
      : "r"(a)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
#undef B2L_R16
__device__ __forceinline__ void tmem_st16(uint32_t a, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(a), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
               : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// The upper halves of x and y as a bf16 pair (truncation), x in the low half
__device__ __forceinline__ uint32_t hi_pair(float x, float y) { return __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632); }
__device__ __forceinline__ float rest(float x) { return x - __uint_as_float(__float_as_uint(x) & 0xffff0000u); }

// Prob: what a family's attention is made of.  Members, all __device__:
//   Tile tile()                           blockIdx -> {first row, rows, [j_begin, j_end) keys, ...}; per-CTA values in Prob::Tile
//   Row row(tile, j)                      pointers of key j: ka (score entries 0 .. split8*8), kb (the rest), v
//   void query(tile, r, c, float x[8])    query entries 8c .. 8c+7 of row r
//   void range(tile, r, lo, hi)           keys lo .. hi are visible to row r
//   float sink(tile)                      score of the sink, -inf without one
//   bool partial(tile); void store_part(tile, r, c0, x[16]); void store_ml(tile, r, m, l)
//   void store(tile, r, c0, x[16])        normalised outputs c0 .. c0+15
// and the host-visible ints DK, DV, stages, split8, floats scale, softcap.
template <class Prob, int NQ, int NP>
__global__ void __launch_bounds__(THREADS, 1) attn_tc_kernel(const __grid_constant__ Prob pr) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  float (&s_max)[2][2][ROWS] = *reinterpret_cast<float (*)[2][2][ROWS]>(smem_raw);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + sizeof(s_max));      // 18
  uint32_t& tmem_slot = *reinterpret_cast<uint32_t*>(bars + 18);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ka = atoms(pr.DK), va = atoms(pr.DV), nst = pr.stages;
  const uint32_t sq = smem_u32(smem_raw) + CONTROL, sk = sq + NQ * ka * Q_ATOM, sv = sk + nst * ka * K_ATOM;
  const uint32_t b0 = smem_u32(bars);
  const uint32_t k_full = b0, k_empty = b0 + 24, v_full = b0 + 48, v_empty = b0 + 72, s_full = b0 + 96, p_full = b0 + 112, pv_done = b0 + 128;
  uint32_t dead = (sq & 1023u) ? 1u : 0u;                    // swizzle atoms need 1024-byte alignment (shared memory starts on one)
  if (tid == 0) {
    for (int i = 0; i < 3; ++i) {
      mbar_init(k_full + 8 * i, 2); mbar_init(k_empty + 8 * i, 1);
      mbar_init(v_full + 8 * i, 2); mbar_init(v_empty + 8 * i, 1);
    }
    for (int i = 0; i < 2; ++i) { mbar_init(s_full + 8 * i, 1); mbar_init(p_full + 8 * i, SOFT_WARPS); mbar_init(pv_done + 8 * i, 1); }
    mbar_init_fence();
  }
  if (warp == SOFT_WARPS + 4) tmem_alloc(smem_u32(&tmem_slot), 512);
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = tmem_slot;
  const typename Prob::Tile tl = pr.tile();
  const int n = (tl.j_end - tl.j_begin + KEYS - 1) / KEYS;

  if (warp >= SOFT_WARPS && warp < SOFT_WARPS + 4) {
    // ===================== keys (two warps) and values (two warps) =====================
    const bool keys = warp < SOFT_WARPS + 2;
    const int lt = tid - 32 * (keys ? SOFT_WARPS : SOFT_WARPS + 2), r0 = lt >> 3, c0 = lt & 7;
    const int chunks = (keys ? pr.DK : pr.DV) / 8;
    const uint32_t base = keys ? sk : sv, stage = (uint32_t)(keys ? ka : va) * K_ATOM, full = keys ? k_full : v_full, empty = keys ? k_empty : v_empty;
    for (int t = 0; t < n; ++t) {
      const int st = t % nst;
      if (t >= nst) mbar_wait(empty + 8 * st, (uint32_t)(t / nst - 1) & 1u, dead);
      const uint32_t dst0 = base + st * stage;
#pragma unroll 2
      for (int i = 0; i < KEYS / 8; ++i) {
        const int r = r0 + 8 * i, j = tl.j_begin + t * KEYS + r;
        const uint32_t dst = dst0 + r * 128 + ((c0 ^ (r & 7)) << 4);
        if (j < tl.j_end) {
          const typename Prob::Row row = pr.row(tl, j);
          for (int c = c0; c < chunks; c += 8)
            cp16(dst + (c >> 3) * K_ATOM, keys ? (c < pr.split8 ? row.ka + c * 8 : row.kb + (c - pr.split8) * 8) : row.v + c * 8);
        } else {
          for (int c = c0; c < chunks; c += 8) st_zero16(dst + (c >> 3) * K_ATOM);
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(full + 8 * st);
    }
  } else if (warp == SOFT_WARPS + 4) {
    // ===================== MMA issue =====================
    bar_named(9, 32 * (SOFT_WARPS + 1));                     // the query tile is in shared memory
    if (lane == 0) {
      fence_after();
      const uint32_t id_s = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(KEYS >> 3) << 17) | ((uint32_t)(ROWS >> 4) << 24);
      const uint32_t id_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(pr.DV >> 3) << 17) | ((uint32_t)(ROWS >> 4) << 24);
      const int ks = pr.DK / 16;
      auto score = [&](int t) {
        const int st = t % nst;
        mbar_wait(k_full + 8 * st, (uint32_t)(t / nst) & 1u, dead);
        if (dead) return;
        fence_after();
        const uint32_t kb = sk + st * ka * K_ATOM;
#pragma unroll 1
        for (int s = NQ - 1; s >= 0; --s) {                  // the smallest parts first
          const uint32_t qb = sq + s * ka * Q_ATOM;
          for (int k = 0; k < ks; ++k)
            mma_ss(tmem + COL_S + 64 * (t & 1), desc_sw128(qb + (k >> 2) * Q_ATOM) + 2 * (k & 3), desc_sw128(kb + (k >> 2) * K_ATOM) + 2 * (k & 3), id_s,
                   (s < NQ - 1 || k > 0) ? 1u : 0u);
        }
        commit(s_full + 8 * (t & 1));
        commit(k_empty + 8 * st);
      };
      if (n > 0) score(0);                                   // an empty key split has no tile
      if (n > 1) score(1);
      for (int t = 0; t < n && !dead; ++t) {
        const int st = t % nst;
        mbar_wait(p_full + 8 * (t & 1), (uint32_t)(t >> 1) & 1u, dead);
        mbar_wait(v_full + 8 * st, (uint32_t)(t / nst) & 1u, dead);
        if (dead) break;
        fence_after();
        const uint32_t vb = sv + st * va * K_ATOM, pc = tmem + COL_P + 96 * (t & 1);
#pragma unroll
        for (int s = NP - 1; s >= 0; --s)
#pragma unroll
          for (int k = 0; k < KEYS / 16; ++k)
            mma_ts(tmem + COL_O, pc + 32 * s + 8 * k, desc_mn(vb + k * 16 * 128, K_ATOM), id_o, (t > 0 || s < NP - 1 || k > 0) ? 1u : 0u);
        commit(v_empty + 8 * st);
        commit(pv_done + 8 * (t & 1));
        if (t + 2 < n) score(t + 2);                         // its scores' buffer was read before the weights of tile t arrived
      }
    }
    __syncwarp();
  } else {
    // ===================== queries, softmax, output =====================
    const int qtr = warp & 3, half = warp >> 2, r = qtr * 32 + lane;
    for (int i = tid; i < ROWS * (pr.DK / 8); i += 32 * SOFT_WARPS) {
      const int rr = i / (pr.DK / 8), c = i - rr * (pr.DK / 8);
      float x[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] = 0.f;
      if (rr < tl.rows) pr.query(tl, rr, c, x);
      const uint32_t dst = sq + (c >> 3) * Q_ATOM + rr * 128 + (((c & 7) ^ (rr & 7)) << 4);
#pragma unroll
      for (int s = 0; s < NQ; ++s) {
        const uint32_t w0 = hi_pair(x[0], x[1]), w1 = hi_pair(x[2], x[3]), w2 = hi_pair(x[4], x[5]), w3 = hi_pair(x[6], x[7]);
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + s * ka * Q_ATOM), "r"(w0), "r"(w1), "r"(w2), "r"(w3) : "memory");
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = fabsf(x[e]) < INFINITY ? rest(x[e]) : 0.f;
      }
    }
    fence_proxy_async();
    bar_named(9, 32 * (SOFT_WARPS + 1));

    int lo, hi;
    pr.range(tl, r, lo, hi);
    if (r >= tl.rows) { lo = 1; hi = 0; }
    const uint32_t lane_at = (uint32_t)(qtr * 32) << 16;
    float m = -INFINITY, l = 0.f;
    for (int t = 0; t < n; ++t) {
      const int b = t & 1;
      mbar_wait(s_full + 8 * b, (uint32_t)(t >> 1) & 1u, dead);
      fence_after();
      uint32_t sr[32];
      tmem_ld32(tmem + lane_at + COL_S + 64 * b + 32 * half, sr);
      float s[32], mx = -INFINITY;
      const int at = tl.j_begin + t * KEYS + 32 * half, first = lo - at, last = hi - at;      // keys first .. last of these 32 are seen
#pragma unroll
      for (int i = 0; i < 32; ++i) s[i] = __uint_as_float(sr[i]) * pr.scale;
      if (pr.softcap > 0.f) {
#pragma unroll
        for (int i = 0; i < 32; ++i) s[i] = pr.softcap * tanhf(s[i] / pr.softcap);
      }
      if (first > 0 || last < 31) {
#pragma unroll
        for (int i = 0; i < 32; ++i) s[i] = (i >= first && i <= last) ? s[i] : -INFINITY;
      }
#pragma unroll
      for (int i = 0; i < 32; ++i) mx = fmaxf(mx, s[i]);
      s_max[b][half][r] = mx;
      bar_named(1 + qtr, 64);
      mx = fmaxf(mx, s_max[b][half ^ 1][r]);
      if (t >= 2) mbar_wait(pv_done + 8 * b, (uint32_t)((t >> 1) - 1) & 1u, dead);            // P[b] has been read
      float f = 1.f;
      if (mx > m + 8.f) {                                   // also the first key a row sees (m = -inf)
        f = m == -INFINITY ? 1.f : expf(m - mx);            // nothing has been added to a row that has seen no key
        m = mx;
      }
      l *= f;
      if (__any_sync(0xffffffffu, f != 1.f)) {              // t > 0 here
        mbar_wait(pv_done + 8 * (b ^ 1), (uint32_t)((t - 1) >> 1) & 1u, dead);
        fence_after();
        for (int g = half; g < pr.DV / 16; g += 2) {
          uint32_t o[16];
          tmem_ld16(tmem + lane_at + COL_O + 16 * g, o);
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
          tmem_st16(tmem + lane_at + COL_O + 16 * g, o);
        }
      }
      float sum = 0.f;
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        s[i] = s[i] == -INFINITY ? 0.f : expf(s[i] - m);
        sum += s[i];
      }
      l += sum;
#pragma unroll
      for (int q = 0; q < NP; ++q) {
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          w[i] = hi_pair(s[2 * i], s[2 * i + 1]);
          s[2 * i] = rest(s[2 * i]);
          s[2 * i + 1] = rest(s[2 * i + 1]);
        }
        tmem_st16(tmem + lane_at + COL_P + 96 * b + 32 * q + 16 * half, w);
      }
      tmem_wait_st();
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full + 8 * b);
    }
    s_max[n & 1][half][r] = l;                               // the buffer of tile n - 2: both warps are past it
    bar_named(1 + qtr, 64);
    l = s_max[n & 1][0][r] + s_max[n & 1][1][r];
    if (n > 0) mbar_wait(pv_done + 8 * ((n - 1) & 1), (uint32_t)((n - 1) >> 1) & 1u, dead);
    fence_after();
    const bool part = pr.partial(tl), live = r < tl.rows;
    const float sink = pr.sink(tl), M = fmaxf(m, sink);
    const float e = m == -INFINITY ? 0.f : expf(m - M);
    float inv = e / (l * e + (sink == -INFINITY ? 0.f : expf(sink - M)));
    if (dead) inv = l = __int_as_float(0x7fc00000);
    if (part && live && half == 0) pr.store_ml(tl, r, m, l);
    for (int g = half; g < pr.DV / 16; g += 2) {
      uint32_t o[16];
      __syncwarp();
      tmem_ld16(tmem + lane_at + COL_O + 16 * g, o);
      float x[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) x[i] = n > 0 ? __uint_as_float(o[i]) * (part ? 1.f : inv) : 0.f;
      if (live) {
        if (part) pr.store_part(tl, r, 16 * g, x);
        else pr.store(tl, r, 16 * g, x);
      }
    }
  }
  fence_before();
  __syncthreads();
  if (warp == SOFT_WARPS + 4) tmem_dealloc(tmem, 512);
}

template <class Prob, int NQ, int NP>
static int launch(const Prob& p, dim3 grid, size_t smem, DynSmemCache& cache, cudaStream_t st) {
  if (int rc = ensure_dyn_smem(attn_tc_kernel<Prob, NQ, NP>, smem, cache)) return rc;
  attn_tc_kernel<Prob, NQ, NP><<<grid, THREADS, smem, st>>>(p);
  B2L_LAUNCH_CHECK("attn_tc_kernel");
  return 0;
}

}  // namespace atc
}  // namespace b2l
