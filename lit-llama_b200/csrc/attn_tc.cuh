// Prompt attention on tcgen05 with f32 scores and weights: 128 query rows of one head against tiles of 64 keys.
//
// Keys and values are bf16.  A query in f32 is cut into NQ = 3 bf16 parts that add up to it exactly (8 bits each, by truncation), and so is
// every softmax weight (NP = 3): the products of the parts with bf16 keys or values are exact, and the tensor core adds them in f32, but it
// truncates where an f32 add rounds: left in the accumulator, the output's error grew with the keys as a bias towards zero (1024 keys 1.6e-6 of
// the norm, 2048 keys 7e-6, 4096 keys with values of mean 2 2.4e-5; the f32 kernel 4e-7, 9e-7 and 7e-7).  So (REGS) every tile's product
// starts from zero and is added to f32 registers: 2.3e-7, 3.2e-7 and 1.2e-7 in these cases, below the f32 kernel in every size measured.
// Three bf16 MMAs cost 3 / 32 of what the f32 FMAs cost on the CUDA cores (4096 against 128 per cycle).
//
// f32 keys and values (KP = 3) are cut into three rounded parts beforehand, and of the nine products the six above 2^-24 are taken: twice the MMAs
// of bf16 keys (entries below 2^-109 keep fewer than 24 bits: the parts have f32's exponents and no more); against the f32 FMAs on the CUDA cores 777 tokens of 8 heads, window 512, take 40 us instead of 217, with errors of 2.1e-7 instead of
// 3.8e-7 against float64 (between a quarter and two thirds of the FMAs' in all sizes measured).
//
//   warp 0       issues the MMAs of the scores S(t) = Q K^T, three tiles ahead at most, warp 13 those of the outputs, P(t) V
//   warps 1, 2   keys, warps 3, 12 values, into 128-byte swizzled rows (keys K-major, values MN-major for the second product), three
//                stages.  Tiles of 64 consecutive rows (the fresh projections, an expanded latent) come by tiled TMA copies; tiles that touch
//                the cache ring or end early by 16-byte cp.async, which arrive on the stage's barrier by themselves but take 3000 cycles
//                to issue, more than the rest of a tile takes
//   warps 4..7   softmax of the even tiles, warps 8..11 of the odd ones: a thread owns one row (tensor-memory lane) of a tile.  The two
//                groups are half a period apart, so one exponentiates while the other waits for tensor memory.  A row's reference maximum
//                travels from tile to tile through shared memory and moves only when it is exceeded by more than 11 (weights reach 2^11;
//                nothing is rounded by that), so the output is rescaled a few times per row instead of once per tile.  The output of a row, half of
//                its columns in each group, is in registers: a group adds the product of its tile before when it has the maximum of this one, and the
//                other group's before it hands over its own weights.
// Tensor memory: 3 x 96 columns for a tile's scores (the upper 64) and, behind the reader, its weights (24 columns per 16 keys: three
// parts of 8); O 128; the smallest part of an f32 query (of 64..192 entries) 96.  Its other parts, and a bf16 query as it lies, are in shared
// memory: an N = 64 MMA then reads 6 KB in its 48 cycles, all that shared memory gives, so nothing else uses it much.  One CTA per SM.
//
// Scores are powers of two: an f32 query takes scale * log2(e) with it (two parts, rounded once), so a weight is one subtraction and ex2,
// and additions go in pairs (f32x2): 9 instructions per score and weight, of which expf and its scaling alone were as many.  f32 outputs
// against float64 as before or closer (1024 keys 3.1e-7 -> 2.8e-7 of the norm, 2048 keys 3.2e-7 -> 2.9e-7).
//
// All roles' loops together stay under the 12 KB or so that an instruction cache next to the schedulers holds: with the softmax written out
// over 64 keys (26 KB) every role ran into instruction fetches (2.7 stalled warps per issued instruction) and an MMA took 120 cycles to
// issue.  So a tile is taken in four steps of 16 keys, read from tensor memory once for the maximum and once for the weights.
//
// What bounds it: a 128 x 64 tile of head size 128 is 24 MMAs of 48 cycles and 12 of 64, 1920 in all; it takes 2400..2700 (2950 with two score
// regions and one issuing warp, 5250 of softmax and issue in the first form); queries, outputs and the first tile's chain of waits take 12 us per CTA
// whatever its tiles (16, latent heads 30, with a row per lane in both).  Kernel time in us, before this form and now: 16 heads, window 1024, 2048
// tokens 85 / 68, latent 16 heads of 192, 128 / 2048 tokens 36 / 16 and 110 / 77, LLaMA's 32 heads, 2048 tokens 111 / 86.
#pragma once
#include "tc_common.cuh"

namespace b2l {
namespace atc {

using namespace tc;

constexpr int ROWS = 128, KEYS = 64;
constexpr int K_THREADS = 64, V_THREADS = 64, THREADS = 448;
constexpr int Q_ATOM = ROWS * 128, K_ATOM = KEYS * 128;      // bytes of 64 columns of a query / key / value tile
constexpr uint32_t REGION = 96, S_AT = 32, COL_O = 288, COL_Q = 416;      // tile t: region at 96 (t % 3), scores at + 32, weights over them
constexpr int MAX_DK = 192, MAX_DV = 128;
constexpr int CONTROL = 3072;                                // barriers, tensor-memory address, row maxima

__host__ __device__ inline int atoms(int d) { return (d + 63) / 64; }
struct Layout { int stages, v_stages, q_tmem; size_t smem; };      // no stages: the sizes do not fit
static inline Layout layout(int nq, int dk, int dv, int kp = 1) {
  Layout l;
  l.q_tmem = nq > 1 ? 1 : 0;                                 // the smallest part of a query in tensor memory, the others in shared memory
  const size_t room = 227 * 1024 - CONTROL - (size_t)(nq - l.q_tmem) * atoms(dk) * Q_ATOM, k = (size_t)kp * atoms(dk) * K_ATOM, v = (size_t)kp * atoms(dv) * K_ATOM;
  l.stages = l.v_stages = 0;
  while (l.stages < 3 && (l.stages + 1) * k + (l.v_stages ? l.v_stages : 1) * v <= room) {      // keys first: their products run three tiles ahead
    ++l.stages;
    if (l.v_stages < 3 && l.stages * k + (l.v_stages + 1) * v <= room) ++l.v_stages;
  }
  l.smem = 227 * 1024 - room + l.stages * k + l.v_stages * v;
  if (l.smem < 120 * 1024) l.smem = 120 * 1024;              // one CTA per SM: each takes all of tensor memory
  return l;
}

// 16 bytes, or zeros where `in` is false
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}
// one arrival on the barrier when the thread's copies so far have landed
__device__ __forceinline__ void cp_arrive(uint32_t bar) { asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void bar_named(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_named_arrive(int id, int n) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory"); }

__device__ __forceinline__ void mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc, uint32_t lead) {
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
               "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"(lead)
               : "memory");
}
// MN-major operand, 128-byte swizzle: rows of 64 consecutive MN entries, one row per k; `lbo` bytes to the next 64 entries
__device__ __forceinline__ uint64_t desc_mn(uint32_t addr, uint32_t lbo) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// 16 columns on their way; the registers hold them after the wait below, which takes them as operands so that nothing uses them before it
__device__ __forceinline__ void tmem_ld16_issue(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&a)[16], uint32_t (&b)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7]), "+r"(a[8]), "+r"(a[9]), "+r"(a[10]), "+r"(a[11]),
                 "+r"(a[12]), "+r"(a[13]), "+r"(a[14]), "+r"(a[15])
               :
               : "memory");
  asm volatile("" : "+r"(b[0]), "+r"(b[1]), "+r"(b[2]), "+r"(b[3]), "+r"(b[4]), "+r"(b[5]), "+r"(b[6]), "+r"(b[7]), "+r"(b[8]), "+r"(b[9]), "+r"(b[10]), "+r"(b[11]),
               "+r"(b[12]), "+r"(b[13]), "+r"(b[14]), "+r"(b[15]) : : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t a, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(a), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]),
               "r"(r[6]), "r"(r[7])
               : "memory");
}

// The upper halves of x and y as a bf16 pair (truncation), x in the low half
__device__ __forceinline__ uint32_t hi_pair(float x, float y) { return __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632); }
// Two f32 operations in one instruction: half the issue slots at the same rate.  a += c, b += d
__device__ __forceinline__ void add2(float& a, float& b, float c, float d) {
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %3};\n\tadd.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}" : "+f"(a), "+f"(b) : "f"(c), "f"(d));
}
__device__ __forceinline__ void sub2(float& a, float& b, float c, float d) {
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %3};\n\tsub.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}" : "+f"(a), "+f"(b) : "f"(c), "f"(d));
}
// a = a * f + c, b = b * f + d
__device__ __forceinline__ void fma2(float& a, float& b, float f, float c, float d) {
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %2};\n\tmov.b64 z, {%3, %4};\n\tfma.rn.f32x2 x, x, y, z;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "+f"(a), "+f"(b) : "f"(f), "f"(c), "f"(d));
}
__device__ __forceinline__ float high_part(float x) { return __uint_as_float(__float_as_uint(x) & 0xffff0000u); }
// 2^x, documented to 2^-22 of the result and without subnormals: as a weight that leaves out what is below 2^-126 of the largest
__device__ __forceinline__ float exp2_f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
constexpr float LOG2E = 1.44269502162933349609375f, LOG2E_LO = 1.925963033500011e-8f, LN2 = 0.693147180559945309f;      // log2(e): the nearest f32 and its remainder

__device__ __forceinline__ void st4_bf16(__nv_bfloat16* p, const float (&y)[4]) {      // 8-byte aligned
  const __nv_bfloat162 u = __floats2bfloat162_rn(y[0], y[1]), v = __floats2bfloat162_rn(y[2], y[3]);
  *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&u), *reinterpret_cast<const uint32_t*>(&v));
}
__device__ __forceinline__ void tmem_st4(uint32_t a, const uint32_t (&r)[4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}

// Prob: what a family's attention is made of.  Members, all __device__:
//   Tile tile()                           blockIdx -> {first row, rows, [j_begin, j_end) keys, ...}; per-CTA values in Prob::Tile
//   Row row(tile, j)                      pointers of key j: ka (score entries 0 .. split8*8), kb (the rest), v
//   bool bulk(tile, j0, ra, rb, rv)       keys j0 .. j0+63 are rows ra.. of map_a (64-column boxes from column tile.xa; the columns from
//                                         split8*8 on: rows rb.. of map_b from tile.xb) and values rows rv.. of map_v from tile.xv
//   void query(tile, r, c, float x[8])    query entries 8c .. 8c+7 of row r
//   bool pieces(); const void* piece(tile, r, p)      the same by 16-byte aligned pieces (4 f32 or, one part, 8 bf16), where they are
//   void range(tile, r, lo, hi)           keys lo .. hi are visible to row r
//   float sink(tile)                      score of the sink, -inf without one
//   bool partial(tile); void store_part(tile, r, c0, x[4]); void store_ml(tile, r, m, l)
//   float factor(tile, r)                 what the row's outputs are multiplied with
//   Gate gate(tile, r, c0)                and what outputs c0 .. c0+3 are, as it lies in memory
//   bool gate_pieces(); const void* gate_piece(tile, r, p)      the same by 16-byte aligned pieces, where it is
//   void store(tile, r, c0, x[4], gate)   normalised outputs c0 .. c0+3, already with the factor
//   KP                                    parts of a key or value: 1, bf16 as they lie; 3, f32 cut beforehand, the parts `plane` rows apart in map_a and map_v
//                                         (keys and values in Row are f32 then, and bulk() is always true)
//   REGS                                  every tile's product is added to f32 registers: the tensor core truncates when it adds to its
//                                         accumulator, which over many tiles is a bias towards zero (see above)
// and the tensor maps, the host-visible ints DK, DV, stages, v_stages, split8, q_tmem, floats scale, softcap.
// Rows whose result is infinite or NaN, again on the CUDA cores over the keys that they see, one row after the other with the whole CTA (a key
// per thread for the scores, three threads per value column).  The products above cannot tell an infinite key or value from NaN: the lower
// parts of a query or weight are often zero, and a key that the row does not see, with its weight of zero, counts as well.  Where all is
// finite it costs the test alone.
template <class Prob, bool CAP>
__device__ __noinline__ void redo_rows(const Prob& pr, const uint32_t* s_bad, float* sm) {
  constexpr int WARPS = THREADS / 32, GROUPS = THREADS / MAX_DV;
  float *q = sm, *w = q + MAX_DK, *s_acc = w + THREADS, *red = s_acc + GROUPS * MAX_DV, *red2 = red + WARPS;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, d = tid % MAX_DV, grp = tid / MAX_DV;
  const typename Prob::Tile tl = pr.tile();
  for (int r = 0; r < tl.rows; ++r) {
    if (!((s_bad[r >> 5] >> (r & 31)) & 1u)) continue;
    __syncthreads();
    if (tid < pr.DK / 8) {
      float x[8];
      pr.query(tl, r, tid, x);
#pragma unroll
      for (int e = 0; e < 8; ++e) q[8 * tid + e] = x[e];
    }
    int lo, hi;
    pr.range(tl, r, lo, hi);
    lo = max(lo, tl.j_begin);
    hi = min(hi, tl.j_end - 1);
    float m = -INFINITY, l = 0.f, acc = 0.f;
    __syncthreads();
    for (int j0 = lo; j0 <= hi; j0 += THREADS) {
      const int j = j0 + tid, count = min(THREADS, hi - j0 + 1);
      float s = -INFINITY;
      if (j <= hi) {
        const typename Prob::Row row = pr.row(tl, j);
        s = 0.f;
        for (int c = 0; c < pr.DK / 8; ++c) {
          const auto* k = c < pr.split8 ? row.ka + 8 * c : row.kb + 8 * (c - pr.split8);
#pragma unroll
          for (int e = 0; e < 8; ++e) s = fmaf(q[8 * c + e], (float)k[e], s);
        }
        s *= pr.scale;
        if (CAP) s = pr.softcap * tanhf(s / pr.softcap);
      }
      const float top = warp_max(s);
      if (lane == 0) red[warp] = top;
      __syncthreads();
      float now = m;
      for (int i = 0; i < WARPS; ++i) now = fmaxf(now, red[i]);
      const float weight = s == -INFINITY ? 0.f : expf(s - now), corr = m == now ? 1.f : expf(m - now), part = warp_sum(weight);
      w[tid] = weight;
      if (lane == 0) red2[warp] = part;
      __syncthreads();
      float sum = 0.f;
      for (int i = 0; i < WARPS; ++i) sum += red2[i];
      l = l * corr + sum;
      acc *= corr;
      m = now;
      if (grp < GROUPS && d < pr.DV)
        for (int i = grp; i < count; i += GROUPS) acc = fmaf(w[i], (float)pr.row(tl, j0 + i).v[d], acc);
      __syncthreads();
    }
    if (grp < GROUPS) s_acc[grp * MAX_DV + d] = acc;
    __syncthreads();
    const bool part = pr.partial(tl);
    const float sink = pr.sink(tl), M = fmaxf(m, sink), e = m == -INFINITY ? 0.f : expf(m - M);
    const float inv = part ? 1.f : e / (l * e + (sink == -INFINITY ? 0.f : expf(sink - M)));
    if (tid == 0 && part) pr.store_ml(tl, r, m, l);
    if (tid < pr.DV / 4) {
      float x[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float t = 0.f;
        for (int g = 0; g < GROUPS; ++g) t += s_acc[g * MAX_DV + 4 * tid + i];
        x[i] = t * inv * (part ? 1.f : pr.factor(tl, r));
      }
      if (part) pr.store_part(tl, r, 4 * tid, x);
      else pr.store(tl, r, 4 * tid, x, pr.gate(tl, r, 4 * tid));
    }
  }
}

template <class Prob, int NQ, int NP, bool CAP>
__global__ void __launch_bounds__(THREADS, 1) attn_tc_kernel(const __grid_constant__ Prob pr) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  float* s_ref = reinterpret_cast<float*>(smem_raw);         // [ROWS] a row's reference maximum after the latest tile
  float* s_end = s_ref + ROWS;                               // [2][ROWS] maximum and sum of the other group at the end
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_end + 2 * ROWS);      // 23
  uint32_t& tmem_slot = *reinterpret_cast<uint32_t*>(bars + 23);
  uint32_t* s_bad = &tmem_slot + 1;                          // [ROWS / 32] rows with an infinite or NaN result
  uint32_t& failed = s_bad[ROWS / 32];                       // a wait of the CTA's softmax groups ran out
  constexpr bool REGS = Prob::REGS;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int KP = Prob::KP;
  const int ka = atoms(pr.DK), va = atoms(pr.DV), nsm = NQ - pr.q_tmem;      // query parts 0 .. nsm-1 lie in shared memory
  const uint32_t sq = smem_u32(smem_raw) + CONTROL, sk = sq + nsm * ka * Q_ATOM, sv = sk + pr.stages * KP * ka * K_ATOM;
  const uint32_t b0 = smem_u32(bars);
  const uint32_t k_full = b0, k_empty = b0 + 24, v_full = b0 + 48, v_empty = b0 + 72, s_full = b0 + 96, p_full = b0 + 120, pv_done = b0 + 136, gave_up = b0 + 160, o_free = b0 + 176;
  uint32_t dead = (sq & 1023u) ? 1u : 0u;                    // swizzle atoms need 1024-byte alignment (shared memory starts on one)
  if (tid == 0) {
    for (int i = 0; i < 3; ++i) {
      mbar_init(k_full + 8 * i, K_THREADS); mbar_init(k_empty + 8 * i, 1);
      mbar_init(v_full + 8 * i, V_THREADS); mbar_init(v_empty + 8 * i, 1);
      mbar_init(s_full + 8 * i, 1);
      mbar_init(pv_done + 8 * i, 1);
    }
    for (int i = 0; i < 2; ++i) mbar_init(p_full + 8 * i, 4);
    mbar_init(gave_up, 1);
    mbar_init(gave_up + 8, 1);
    mbar_init(o_free, 4);
    failed = 0u;
    mbar_init_fence();
  }
  if (tid < ROWS) s_ref[tid] = -INFINITY;
  if (tid < ROWS / 32) s_bad[tid] = 0u;
  if (warp == 0) tmem_alloc(smem_u32(&tmem_slot), 512);
  const typename Prob::Tile tl = pr.tile();
  const int n = (tl.j_end - tl.j_begin + KEYS - 1) / KEYS;
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = tmem_slot;
  if (warp == 0 || warp == 13) {
    // ===================== MMA issue: warp 0 the scores, warp 13 the outputs =====================
    // One warp for both spent 2800 cycles on a tile: a batch is issued about as fast as it is executed (some 50 cycles an MMA), so every wait, 65..240
    // cycles even on a barrier that is complete, left the tensor pipe idle.
    const uint32_t lead = elect_lane();
    auto copied = [&](int t) {                               // cp.async writes through the generic proxy; the fence costs some 300 cycles
      int ra, rb, rv;
      if (!pr.bulk(tl, tl.j_begin + t * KEYS, ra, rb, rv)) fence_proxy_async();
    };
    const int nst = warp ? pr.v_stages : pr.stages;
    int st = 0, reg = 0;                                     // stage and region, counted instead of divided out
    // Keys and values of one part meet every part of a query or weight; of three parts, the products above 2^-24 (indexes two bits each)
    static_assert(KP == 1 || (NQ == 3 && NP == 3), "three parts meet three parts");
    constexpr int PAIRS = KP == 3 ? 6 : NQ, QS = 0x046, KS = 0x124;
    uint32_t ph = 0;
    if (warp == 0) {
      bar_named(9, 32 + 2 * ROWS);                           // the queries are in place
      fence_after();
      const uint32_t id_s = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(KEYS >> 3) << 17) | ((uint32_t)(ROWS >> 4) << 24);
      const int full = pr.DK / 64, odd = pr.DK / 16 % 4;      // steps of 16 entries: four per 64, and the rest
      for (int t = 0; t < n; ++t) {
        mbar_wait(k_full + 8 * st, ph, dead);
        if (t >= 3) mbar_wait(pv_done + 8 * reg, (uint32_t)(t / 3 - 1) & 1u, dead);      // over the weights of tile t - 3
        dead = __any_sync(0xffffffffu, dead) ? 1u : 0u;
        if (dead) break;
        copied(t);
        fence_after();
        const uint32_t kb = sk + st * KP * ka * K_ATOM, d = tmem + REGION * reg + S_AT;
        const uint64_t kd0 = desc_sw128(kb);
        uint32_t acc = 0;
#pragma unroll 1
        for (int i = 0; i < PAIRS; ++i) {                    // the smallest parts first
          const int s = KP == 3 ? QS >> 2 * i & 3 : NQ - 1 - i;
          uint64_t kd = kd0 + (KP == 3 ? (uint32_t)((KS >> 2 * i & 3) * ka * K_ATOM) >> 4 : 0u);
          if (s >= nsm) {
            uint32_t qa = tmem + COL_Q + (s - nsm) * (pr.DK / 2);
#pragma unroll 1
            for (int a = 0; a < full; ++a, qa += 32, kd += K_ATOM >> 4) {
#pragma unroll
              for (int k = 0; k < 4; ++k) mma_ts(d, qa + 8 * k, kd + 2 * k, id_s, k > 0 ? 1u : acc, lead);
              acc = 1;
            }
#pragma unroll 1
            for (int k = 0; k < odd; ++k, acc = 1) mma_ts(d, qa + 8 * k, kd + 2 * k, id_s, acc, lead);
          } else {
            uint64_t qd = desc_sw128(sq + s * ka * Q_ATOM);
#pragma unroll 1
            for (int a = 0; a < full; ++a, qd += Q_ATOM >> 4, kd += K_ATOM >> 4) {
#pragma unroll
              for (int k = 0; k < 4; ++k) mma_ss(d, qd + 2 * k, kd + 2 * k, id_s, k > 0 ? 1u : acc, lead);
              acc = 1;
            }
#pragma unroll 1
            for (int k = 0; k < odd; ++k, acc = 1) mma_ss(d, qd + 2 * k, kd + 2 * k, id_s, acc, lead);
          }
        }
        if (lead) {
          commit(s_full + 8 * reg);
          commit(k_empty + 8 * st);
        }
        if (++reg == 3) reg = 0;
        if (++st == nst) { st = 0; ph ^= 1u; }
        __syncwarp();
      }
    } else {
      const uint32_t id_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(pr.DV >> 3) << 17) | ((uint32_t)(ROWS >> 4) << 24);
      for (int t = 0; t < n; ++t) {
        mbar_wait(v_full + 8 * st, ph, dead);
        if (REGS && t > 0) mbar_wait(o_free, (uint32_t)(t - 1) & 1u, dead);      // the group of the tile before has taken that product
        mbar_wait_warp(p_full + 8 * (t & 1), (uint32_t)(t >> 1) & 1u, dead);     // and so has this tile's
        if (dead) break;
        copied(t);
        fence_after();
        const uint64_t vd0 = desc_mn(sv + st * KP * va * K_ATOM, K_ATOM);
        const uint32_t pc = tmem + REGION * reg;
#pragma unroll 1
        for (int i = 0; i < (KP == 3 ? 6 : NP); ++i) {
          const int q = KP == 3 ? QS >> 2 * i & 3 : NP - 1 - i;
          const uint64_t vd = vd0 + (KP == 3 ? (uint32_t)((KS >> 2 * i & 3) * va * K_ATOM) >> 4 : 0u);
#pragma unroll
          for (int k = 0; k < KEYS / 16; ++k) mma_ts(tmem + COL_O, pc + 24 * k + 8 * q, vd + k * (16 * 128 / 16), id_o, ((!REGS && t > 0) || i > 0 || k > 0) ? 1u : 0u, lead);
        }
        if (lead) {
          commit(pv_done + 8 * reg);
          commit(v_empty + 8 * st);
        }
        if (++reg == 3) reg = 0;
        if (++st == nst) { st = 0; ph ^= 1u; }
        __syncwarp();
      }
    }
    if (dead) {                                              // what was issued ends before tensor memory is given back
      const uint32_t bar = gave_up + (warp ? 8 : 0);
      uint32_t late = 0;
      if (lead) commit(bar);
      mbar_wait(bar, 0, late);
    }
    __syncwarp();
  } else if (warp < 4 || warp == 12) {
    // ===================== keys and values, two warps each =====================
    const bool keys = warp < 3;
    const int lt = keys ? tid - 32 : (warp == 12 ? 32 : 0) + lane, r0 = lt >> 3, c0 = lt & 7;
    const int chunks = (keys ? pr.DK : pr.DV) / 8;
    const uint32_t base = keys ? sk : sv, stage = (uint32_t)(KP * (keys ? ka : va)) * K_ATOM, full = keys ? k_full : v_full, empty = keys ? k_empty : v_empty;
    const int nst = keys ? pr.stages : pr.v_stages;
    int st = -1;
    uint32_t phase = 0;                                      // parity of the stage's previous use
    int t = 0;
    for (; t < n; ++t) {
      if (++st == nst) { st = 0; phase ^= t > nst ? 1u : 0u; }
      if (t >= nst) mbar_wait(empty + 8 * st, phase, dead);
      if (dead) break;                                       // the stage may still be read: no copy, no arrival
      const uint32_t dst0 = base + st * stage;
      const int j0 = tl.j_begin + t * KEYS;
      int row_a, row_b, row_v;
      if (pr.bulk(tl, j0, row_a, row_b, row_v)) {            // 64 consecutive rows: a tiled copy per 64 columns
        if (lt == 0) {
          mbar_expect_tx(full + 8 * st, stage);
          for (int part = 0; part < KP; ++part) {
            const uint32_t dst = dst0 + part * (keys ? ka : va) * K_ATOM;
            int below = 0;
            if constexpr (KP > 1) below = part * pr.plane;
            if (keys) {
              for (int a = 0; a < ka; ++a) {
                if (8 * a < pr.split8) tma_load_2d(dst + a * K_ATOM, &pr.map_a, tl.xa + 64 * a, row_a + below, full + 8 * st);
                else tma_load_2d(dst + a * K_ATOM, &pr.map_b, tl.xb + 64 * a - 8 * pr.split8, row_b + below, full + 8 * st);
              }
            } else {
              for (int a = 0; a < va; ++a) tma_load_2d(dst + a * K_ATOM, &pr.map_v, tl.xv + 64 * a, row_v + below, full + 8 * st);
            }
          }
        } else {
          mbar_arrive(full + 8 * st);
        }
        continue;
      }
      if constexpr (KP == 1) {
#pragma unroll 2
      for (int i = 0; i < KEYS / 8; ++i) {
        const int r = r0 + 8 * i, j = j0 + r;
        const bool in = j < tl.j_end;
        const uint32_t dst = dst0 + r * 128 + ((c0 ^ (r & 7)) << 4);
        const typename Prob::Row row = pr.row(tl, in ? j : tl.j_begin);
#pragma unroll
        for (int a = 0; a < MAX_DK / 64; ++a) {
          const int c = c0 + 8 * a;
          if (c < chunks) cp16(dst + a * K_ATOM, keys ? (c < pr.split8 ? row.ka + c * 8 : row.kb + (c - pr.split8) * 8) : row.v + c * 8, in);
        }
      }
      cp_arrive(full + 8 * st);
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");         // no copy outlives its thread
    if (lt == 0) {                                           // nor a tiled one: the latest use of every stage, all landed unless a wait ran out
      uint32_t late = 0;
      for (int s = 0; s < nst && s < t; ++s) mbar_wait(full + 8 * s, (uint32_t)((t - 1 - s) / nst) & 1u, late);
    }
  } else {
    // ===================== queries, softmax, output =====================
    const int qtr = warp & 3, b = (warp >> 2) - 1, r = qtr * 32 + lane;      // b: the parity of the group's tiles
    const uint32_t lane_at = (uint32_t)(qtr * 32) << 16;
    // Queries: 16-byte pieces, a warp on one row after the other, to where the parts go that the row's threads make of them (of 8 f32 entries in two
    // pieces: to the places of the two parts in shared memory).  A row per lane kept the load unit busy with 32 lines for every instruction.
    const int sw = warp - 4, pieces = pr.DK / (NQ > 1 ? 4 : 8);
    auto slot = [&](int s, int c, int row) { return sq + (s * ka + (c >> 3)) * Q_ATOM + row * 128 + (((c & 7) ^ (row & 7)) << 4); };
    if (pr.pieces()) {
      for (int p = lane; p < pieces; p += 32)
#pragma unroll 4
        for (int q = sw; q < ROWS; q += 2 * ROWS / 32)
          cp16(NQ > 1 ? slot(p & 1, p >> 1, q) : slot(0, p, q), pr.piece(tl, q < tl.rows ? q : 0, p), q < tl.rows);
      asm volatile("cp.async.wait_all;" ::: "memory");
      bar_named(10, 2 * ROWS);
    }
    // f32 queries take the scale with them, as a factor in two parts; a bf16 query, which is one part as it lies, leaves it to the weights.
    constexpr bool FOLD = NQ > 1;
    const float by = CAP ? pr.scale / pr.softcap : pr.scale * LOG2E, by_lo = CAP ? fmaf(-by, pr.softcap, pr.scale) / pr.softcap : fmaf(pr.scale, LOG2E, -by) + pr.scale * LOG2E_LO;
    const float after = FOLD ? 1.f : CAP ? 1.f : by;
#pragma unroll 1
    for (int c = b; NQ > 1 && c < pr.DK / 8; c += 2) {        // rolled up: code that runs once is fetched at some 12 cycles an instruction
      float x[8];
      if (pr.pieces()) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
          asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x[4 * h]), "=f"(x[4 * h + 1]), "=f"(x[4 * h + 2]), "=f"(x[4 * h + 3]) : "r"(slot(h, c, r)) : "memory");
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = 0.f;
        if (r < tl.rows) pr.query(tl, r, c, x);
        __syncwarp();
      }
      // scores come out in powers of two (with a cap: as its argument); rounded once
#pragma unroll
      for (int e = 0; e < 8; e += 2) {
        float lo[2] = {x[e] * by_lo, x[e + 1] * by_lo};
        fma2(x[e], x[e + 1], by, lo[0], lo[1]);
      }
#pragma unroll
      for (int s = 0; s < NQ; ++s) {
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) w[e] = hi_pair(x[2 * e], x[2 * e + 1]);
        if (s >= nsm) tmem_st4(tmem + lane_at + COL_Q + (s - nsm) * (pr.DK / 2) + 4 * c, w);
        else asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(slot(s, c, r)), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
        if (s + 1 < NQ) {
#pragma unroll
          for (int e = 0; e < 8; e += 2) sub2(x[e], x[e + 1], high_part(x[e]), high_part(x[e + 1]));      // an infinite entry: NaN, and the row is taken again
        }
      }
    }
    tmem_wait_st();
    fence_before();
    fence_proxy_async();
    bar_named(9, 32 + 2 * ROWS);

    int lo, hi;
    pr.range(tl, r, lo, hi);
    if (r >= tl.rows) { lo = 1; hi = 0; }
    float m = -INFINITY, l = 0.f;                            // reference maximum, and the sum over this group's tiles relative to it
    float acc[MAX_DV / 32][16], acc_ref = -INFINITY;         // output columns 16 (b + 2 i) .. of the tiles so far, relative to acc_ref
#pragma unroll
    for (int i = 0; i < MAX_DV / 32; ++i)
#pragma unroll
      for (int e = 0; e < 16; ++e) acc[i][e] = 0.f;
    int s_reg = b;                                           // tile t's region, and the phase of its barrier (this group meets every second one; the one
    uint32_t s_ph = 0;                                       // between, tile t - 3, came before the scores of this group's tile before)
    float base[2] = {-INFINITY, -INFINITY};                  // the references of tiles t - 2 and t - 1
    uint32_t d_bar = 0, d_ph = 0;                            // REGS: barrier and phase of the next product; a group adds all of them in order
    for (int t = b; t < n + (REGS ? 2 : 0); t += 2) {        // REGS, tiles n and n + 1: nothing but the products still to be added
     float now = -INFINITY;
     float mm = 0.f, scale = 1.f;
     const uint32_t reg = tmem + lane_at + REGION * s_reg;
     if (t < n) {
      mbar_wait(s_full + 8 * s_reg, s_ph, dead);
      fence_after();
      s_reg += 2;
      if (s_reg >= 3) { s_reg -= 3; s_ph ^= 1u; }
      const int at = tl.j_begin + t * KEYS, first = lo - at, last = hi - at;      // keys first .. last of these 64 are seen
      const bool cut = __any_sync(0xffffffffu, first > 0 || last < KEYS - 1);
      float mx = -INFINITY;
#pragma unroll 1
      for (int c = 0; c < KEYS / 16; ++c) {
        uint32_t u[16];
        tmem_ld16(reg + S_AT + 16 * c, u);
        float s[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          s[i] = __uint_as_float(u[i]);
          if (CAP) s[i] = pr.softcap * LOG2E * tanhf(FOLD ? s[i] : s[i] * by);
          else if (!FOLD) s[i] *= by;
        }
        if (cut) {
#pragma unroll
          for (int i = 0; i < 16; ++i) s[i] = (16 * c + i >= first && 16 * c + i <= last) ? s[i] : -INFINITY;
        }
        if (CAP || cut) {                                    // the weights are taken from what is left here
#pragma unroll
          for (int i = 0; i < 16; ++i) u[i] = __float_as_uint(s[i]);
          tmem_st16(reg + S_AT + 16 * c, u);
        }
        float m2[2] = {mx, s[0]};
#pragma unroll
        for (int i = 1; i < 16; ++i) m2[i & 1] = fmaxf(m2[i & 1], s[i]);
        mx = fmaxf(m2[0], m2[1]);
      }
      scale = (CAP || cut) ? 1.f : after;
      if (CAP || cut) tmem_wait_st();
      // the row's reference after tile t - 1, from the other group; this tile's goes to it (barriers 1..4 even -> odd, 5..8 odd -> even)
      if (t > 0) bar_named(1 + 4 * (b ^ 1) + qtr, 64);
      const float ref = s_ref[r];
      const bool up = mx > ref + 11.f;                       // also the first key a row sees (ref = -inf)
      now = up ? mx : ref;
      if (up) s_ref[r] = now;
      if (REGS || t + 1 < n) bar_named_arrive(1 + 4 * b + qtr, 64);
      base[1] = ref;
      if (m != now) {
        l *= m == -INFINITY ? 0.f : exp2_f(m - now);
        m = now;
      }
      if (!REGS) {                                           // what is in tensor memory follows the reference
        const float f = (up && ref != -INFINITY) ? exp2_f(ref - now) : 1.f;    // nothing was added to a row that saw no key
        if (__any_sync(0xffffffffu, f != 1.f)) {             // t > 0 here; the scores of this tile came after PV(t - 3), the phase before on this barrier is complete
          mbar_wait(pv_done + 8 * ((t - 1) % 3), (uint32_t)((t - 1) / 3) & 1u, dead);
          fence_after();
          for (int g = 0; g < pr.DV / 16; ++g) {
            uint32_t o[16];
            tmem_ld16(tmem + lane_at + COL_O + 16 * g, o);
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
            tmem_st16(tmem + lane_at + COL_O + 16 * g, o);
          }
        }
      }
      mm = m == -INFINITY ? 0.f : m;                         // a row that has seen no key: every score is -inf, every weight 0
     }
     // REGS: the product of tile t - 2 into the registers, then this tile's weights, then the product of tile t - 1 before PV(t) may overwrite it.
     // The product of this group's tile before comes while the other group exponentiates, and the scores of tile t + 2 need none of it.
#pragma unroll 1
     for (int k = 0; k < 2; ++k) {
      if (REGS) {
        const int u = t - 2 + k;
        if (k == 1 && t == n && n > 0) {
          bar_named(1 + 4 * (b ^ 1) + qtr, 64);
          base[1] = s_ref[r];
        }
        if (u >= 0 && u < n) {
          mbar_wait(pv_done + 8 * d_bar, d_ph, dead);
          if (++d_bar == 3) { d_bar = 0; d_ph ^= 1u; }
          fence_after();
          const float to = k ? base[1] : base[0];
          if (__any_sync(0xffffffffu, acc_ref != to)) {
            const float f = acc_ref == to ? 1.f : acc_ref == -INFINITY ? 0.f : exp2_f(acc_ref - to);
            acc_ref = to;
#pragma unroll
            for (int i = 0; i < MAX_DV / 32; ++i)
#pragma unroll
              for (int e = 0; e < 16; ++e) acc[i][e] *= f;
          }
#pragma unroll
          for (int i = 0; i < MAX_DV / 32; i += 2) {         // two loads on their way together (columns beyond the head are loaded, not used)
            if (b + 2 * i >= pr.DV / 16) break;
            uint32_t o[2][16];
            tmem_ld16_issue(tmem + lane_at + COL_O + 16 * (b + 2 * i), o[0]);
            tmem_ld16_issue(tmem + lane_at + COL_O + 16 * (b + 2 * i + 2), o[1]);
            tmem_wait_ld(o[0], o[1]);
#pragma unroll
            for (int e = 0; e < 16; e += 2) {
              add2(acc[i][e], acc[i][e + 1], __uint_as_float(o[0][e]), __uint_as_float(o[0][e + 1]));
              add2(acc[i + 1][e], acc[i + 1][e + 1], __uint_as_float(o[1][e]), __uint_as_float(o[1][e + 1]));
            }
          }
          if (k == 0) {
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(o_free);
          }
        }
      }
      if (t >= n) continue;
      if (k == 1) {
        fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full + 8 * b);
        continue;
      }
      float sum[2] = {0.f, 0.f};
#pragma unroll 1
      for (int c = 0; c < KEYS / 16; ++c) {
        uint32_t u[16];
        tmem_ld16(reg + S_AT + 16 * c, u);
        float s[16];
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
          s[i] = __uint_as_float(u[i]);
          s[i + 1] = __uint_as_float(u[i + 1]);
          if (FOLD) sub2(s[i], s[i + 1], mm, mm);
          else fma2(s[i], s[i + 1], scale, -mm, -mm);
          s[i] = exp2_f(s[i]);
          s[i + 1] = exp2_f(s[i + 1]);
          add2(sum[0], sum[1], s[i], s[i + 1]);
        }
#pragma unroll
        for (int q = 0; q < NP; ++q) {
          uint32_t w[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            w[i] = hi_pair(s[2 * i], s[2 * i + 1]);
            if (q + 1 < NP) sub2(s[2 * i], s[2 * i + 1], high_part(s[2 * i]), high_part(s[2 * i + 1]));
          }
          tmem_st8(reg + 24 * c + 8 * q, w);
        }
      }
      l += sum[0] + sum[1];
      tmem_wait_st();
     }
     base[0] = now;
    }
    // the even group ends with the sum of both (relative to the last reference); each group stores every other 16 columns.  Without REGS only
    // the group of the last tile waits for its product (the other may not have seen the phase before it, whose parity would let it pass);
    // the barriers below carry that to the other group.
    if (!REGS && n > 0 && b == ((n - 1) & 1)) {
      mbar_wait(pv_done + 8 * ((n - 1) % 3), (uint32_t)((n - 1) / 3) & 1u, dead);
      fence_after();
    }
    if (!REGS) fence_before();
    // Gates along the rows into the memory of the queries, which every score has read by now
    const uint32_t gate_row = pr.DV / 4 * sizeof(typename Prob::Gate);
    const bool staged = REGS && !pr.partial(tl) && pr.gate_pieces() && ROWS * gate_row <= nsm * ka * Q_ATOM;
    if (staged) {
      const int per = gate_row / 16, at_once = 32 / per, sub = lane / per, p = lane - sub * per;
      if (sub < at_once) {
#pragma unroll 4
        for (int q = (warp - 4) * at_once + sub; q < tl.rows; q += 2 * ROWS / 32 * at_once) cp16(sq + q * gate_row + 16 * p, pr.gate_piece(tl, q, p), true);
      }
    }
    if (dead) failed = 1u;
    if (b == 1) { s_end[r] = m; s_end[ROWS + r] = l; }
    bar_named(10, 2 * ROWS);
    const float ref = s_ref[r];
    float* tot = s_end;                                      // [ROWS]: the sum, for both groups
    if (b == 0) {
      const float m1 = s_end[r], l1 = s_end[ROWS + r];
      l = (m == -INFINITY ? 0.f : l * exp2_f(m - ref)) + (m1 == -INFINITY ? 0.f : l1 * exp2_f(m1 - ref));
      tot[r] = l;
    }
    bar_named(10, 2 * ROWS);
    if (!REGS) fence_after();
    dead |= failed;
    l = tot[r];
    m = ref;
    const bool part = pr.partial(tl), live = r < tl.rows;
    const float sink = pr.sink(tl), M = fmaxf(m, sink * LOG2E);
    const float e = m == -INFINITY ? 0.f : exp2_f(m - M);
    float inv = e / (l * e + (sink == -INFINITY ? 0.f : exp2_f(fmaf(sink, LOG2E, fmaf(sink, LOG2E_LO, -M)))));
    if (part) {                                              // maxima outside are in powers of e: what rounding changes about this one goes into the sums
      const float me = m == -INFINITY ? m : m * LN2;
      inv = fabsf(me) < INFINITY ? exp2_f(fmaf(-me, LOG2E_LO, fmaf(-me, LOG2E, m))) : 1.f;
      m = me;
      l *= inv;
    }
    if (dead) inv = l = __int_as_float(0x7fc00000);
    if (part && live && b == 0) pr.store_ml(tl, r, m, l);
    if (!part && live) inv *= pr.factor(tl, r);
    float odd = part ? l * 0.f : 0.f;                        // NaN as soon as something infinite or NaN came out
    // Outputs through shared memory (the stages are free: every product is done), rows apart by 16 bytes more than they take; then lanes side by side
    // along a row.
    const uint32_t row_bytes = pr.DV * 4 + 16, mine = sk + r * row_bytes;
    auto keep = [&](int c0, float (&x)[16]) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        x[i] = n > 0 ? x[i] * inv : 0.f;
        odd = fmaf(x[i], 0.f, odd);
      }
#pragma unroll
      for (int i = 0; i < 16; i += 4)
        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(mine + 4 * (c0 + i)), "f"(x[i]), "f"(x[i + 1]), "f"(x[i + 2]), "f"(x[i + 3]) : "memory");
    };
    if (REGS) {
#pragma unroll
      for (int i = 0; i < MAX_DV / 32; ++i)
        if (b + 2 * i < pr.DV / 16) keep(16 * (b + 2 * i), acc[i]);
    } else {
#pragma unroll 1
      for (int g = b; g < pr.DV / 16; g += 2) {
        uint32_t o[16];
        tmem_ld16(tmem + lane_at + COL_O + 16 * g, o);
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = __uint_as_float(o[i]);
        keep(16 * g, x);
      }
    }
    if (staged) asm volatile("cp.async.wait_all;" ::: "memory");
    bar_named(10, 2 * ROWS);
    const int per = pr.DV / 4, at_once = 32 / per, sub = lane / per, c0 = 4 * (lane - sub * per), stride = 2 * ROWS / 32 * at_once;      // rows a turn
    const int first_row = sub < at_once ? sw * at_once + sub : ROWS;
#pragma unroll 1
    for (int k = first_row; k < tl.rows; k += stride) {
      float x[4];
      asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]) : "r"(sk + k * row_bytes + 4 * c0) : "memory");
      if (part) {
        pr.store_part(tl, k, c0, x);
      } else {
        const typename Prob::Gate g = staged ? *reinterpret_cast<const typename Prob::Gate*>(smem_raw + CONTROL + k * gate_row + c0 / 4 * sizeof(typename Prob::Gate)) : pr.gate(tl, k, c0);
        pr.store(tl, k, c0, x, g);
      }
    }
    const uint32_t bad = __ballot_sync(0xffffffffu, live && !dead && odd != odd);
    if (lane == 0 && bad) atomicOr(&s_bad[qtr], bad);
  }
  fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
  if (s_bad[0] | s_bad[1] | s_bad[2] | s_bad[3]) redo_rows<Prob, CAP>(pr, s_bad, reinterpret_cast<float*>(smem_raw + CONTROL));
}

template <class Prob, int NQ, int NP, bool CAP>
static int launch(const Prob& p, dim3 grid, size_t smem, DynSmemCache& cache, cudaStream_t st) {
  if (int rc = ensure_dyn_smem(attn_tc_kernel<Prob, NQ, NP, CAP>, smem, cache)) return rc;
  attn_tc_kernel<Prob, NQ, NP, CAP><<<grid, THREADS, smem, st>>>(p);
  B2L_LAUNCH_CHECK("attn_tc_kernel");
  return 0;
}

}  // namespace atc
}  // namespace b2l
