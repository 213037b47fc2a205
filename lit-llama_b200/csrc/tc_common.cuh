// tcgen05 / TMA pieces shared by the tensor-core kernels (sm_100a): mbarriers with bounded waits, tiled TMA loads, shared-memory matrix
// descriptors (K-major, 128-byte swizzle), tensor-memory loads, and the host-side tensor-map encoder.
#pragma once
#include <cuda.h>   // CUtensorMap and its enums only: the encoder is fetched with cudaGetDriverEntryPoint (no libcuda link)

#include <atomic>

#include "b2l_common.cuh"

namespace b2l {
namespace tc {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t a, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(count) : "memory"); }
__device__ __forceinline__ void mbar_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(uint32_t a) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(a) : "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint32_t a, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(a), "r"(bytes) : "memory");
}
// Waits for the phase with this parity.  `dead` is the thread's sticky error word: a wait that runs out (about a second; a kernel here
// takes milliseconds at most) sets it and every later wait of the thread returns at once, so the kernel ends.  A thread whose word is set
// passes nothing on: it issues no copy and no MMA, and leaves the barriers that follow without their arrival, so the waits of those that depend on it
// run out too, down to the threads that store the result; they store NaN, and a CTA whose sums others add says so in its `failed` word.
// Copies and MMAs in flight are waited for (with the same limit) by the warp that issued them, with a word of its own.
__device__ __forceinline__ void mbar_wait(uint32_t a, uint32_t parity, uint32_t& dead) {
  if (dead) return;
  uint32_t ok = 0;
  for (uint32_t tries = 0; tries < (1u << 22); ++tries) {
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(a), "r"(parity) : "memory");
    if (ok) return;
  }
  dead = 1u;
}
// The same for a whole warp that acts on the outcome together (aligned instructions, loops with barriers in them).
__device__ __forceinline__ void mbar_wait_warp(uint32_t a, uint32_t parity, uint32_t& dead) {
  mbar_wait(a, parity, dead);
  dead = __any_sync(0xffffffffu, dead) ? 1u : 0u;
}
// Whether the phase with this parity is complete, without waiting: a wait on a barrier that is complete takes 120..300 cycles, so a loop
// asks for its next barrier before it works on this one.
__device__ __forceinline__ uint32_t mbar_test(uint32_t a, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(a), "r"(parity) : "memory");
  return ok;
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t tmem, uint32_t cols) { asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory"); }

// 16 consecutive 32-bit columns of this warp's 32 tensor-memory lanes
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// K-major operand in 128-byte swizzled rows (what a tiled TMA copy with SWIZZLE_128B writes): 8-row groups of 1024 bytes.  A step along
// K inside the 128-byte row adds its byte offset to the start address.
__device__ __forceinline__ uint64_t desc_sw128(uint32_t smem_addr) {
  return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// 2-D tiled copy: box at element (c0 along the row, c1 = row); c0 * element size must be a multiple of 16 bytes
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t mbar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst), "l"(map), "r"(mbar), "r"(c0),
               "r"(c1)
               : "memory");
}

// The whole warp runs an issuing loop, so descriptors stay in uniform registers (issued from one lane's branch an MMA took up to four times
// as long); `lead` is set in the one lane that issues.
__device__ __forceinline__ uint32_t elect_lane() {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
  return r;
}
// kind::f16, A from tensor memory
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc, uint32_t lead) {
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
               "r"(a), "l"(b), "r"(idesc), "r"(acc), "r"(lead)
               : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t a, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(a), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
               : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ---- thread-block clusters
__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t dsmem_addr(uint32_t addr, uint32_t rank) {      // the same shared-memory address in CTA `rank`
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
  return a;
}
__device__ __forceinline__ uint32_t ld_dsmem_u32(uint32_t addr, uint32_t rank) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(dsmem_addr(addr, rank)) : "memory");
  return v;
}
__device__ __forceinline__ uint4 ld_dsmem(uint32_t addr, uint32_t rank) {
  uint4 v;
  asm volatile("ld.shared::cluster.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(dsmem_addr(addr, rank)) : "memory");
  return v;
}

// ---- host side
typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                             CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline EncodeFn encoder() {
  static EncodeFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) p = nullptr;
    return (EncodeFn)p;
  }();
  return fn;
}
// Row-major [rows][cols] matrix, leading dimension ld (elements), boxes of box_cols x box_rows with box_cols * size == 128 bytes,
// 128-byte swizzle; rows and columns beyond the matrix read as zeros.  Returns 0 or a B2L_E_* code with the error set.
inline int map_sw128(CUtensorMap* m, CUtensorMapDataType type, int esize, const void* base, long long rows, long long cols, long long ld, int box_cols, int box_rows) {
  EncodeFn fn = encoder();
  if (fn == nullptr) {
    set_error("cuTensorMapEncodeTiled is not available from this driver");
    return B2L_E_STATE;
  }
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)(ld * esize)};
  const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult cr = fn(m, type, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (cr != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed (%d) for %lld x %lld, leading dimension %lld", (int)cr, rows, cols, ld);
    return B2L_E_ARG;
  }
  return 0;
}

// Clusters of `size` (1..8) CTAs of a kernel, one per SM by 120 KB of shared memory, that run at once (B200: 148, 74, 45, 33, 26, 22, 15, 15: clusters do not
// cross the SM groups).  Asked of the driver once; the kernel's limit of dynamic shared memory has been raised before.
template <class Kernel> inline int clusters_at_once(Kernel kernel, int threads, int size, int sms, std::atomic<int> (&known)[9]) {
  if (size == 1) return sms;
  int n = known[size].load(std::memory_order_relaxed);
  if (n == 0) {
    LaunchCfg lc(dim3((unsigned)size), dim3((unsigned)threads), 120 * 1024, nullptr, false, size);
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &lc.cfg) != cudaSuccess || n <= 0) {
      (void)cudaGetLastError();
      n = sms / size > 0 ? sms / size : 1;
    }
    known[size].store(n, std::memory_order_relaxed);
  }
  return n;
}

}  // namespace tc
}  // namespace b2l
