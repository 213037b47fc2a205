// Error state and version of libb200seq (a library of its own: it is built without the quantized-LLaMA kernels).
#include "seq_common.cuh"

namespace b2l {

static thread_local char g_seq_err[512] = "";

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_seq_err, sizeof(g_seq_err), fmt, ap);
  va_end(ap);
}

int cuda_fail(cudaError_t e, const char* what) {
  set_error("%s: %s (%s)", what, cudaGetErrorString(e), cudaGetErrorName(e));
  (void)cudaGetLastError();
  return (int)e;
}

int sm_count() {
  int dev = 0, v = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 148;
  if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
  return v;
}

}  // namespace b2l

extern "C" int b2l_seq_version(void) { return 100; }
extern "C" const char* b2l_seq_last_error(void) { return b2l::g_seq_err; }

extern "C" int b2l_seq_zero_slot(void* state, size_t slot_bytes, int slot, b2l_stream_t stream) {
  B2L_CHECK_ARG(state != nullptr && slot >= 0, "b2l_seq_zero_slot: null pointer or negative slot");
  if (slot_bytes == 0) return 0;
  B2L_CUDA(cudaMemsetAsync(static_cast<char*>(state) + (size_t)slot * slot_bytes, 0, slot_bytes, (cudaStream_t)stream));
  return 0;
}

namespace b2l {
// Several ranges of 16-byte words at once: a new sequence's state is a range per layer and tensor, and a memset each took 1.5 us of the device and 4 of the host.
constexpr int ZERO_RANGES = 16, ZERO_BLOCK = 256 * 8;      // words per block
struct ZeroRanges { uint4* p[ZERO_RANGES]; unsigned long long words[ZERO_RANGES]; unsigned first[ZERO_RANGES + 1]; };
__global__ void __launch_bounds__(256) seq_zero_kernel(const __grid_constant__ ZeroRanges r) {
  int i = 0;
  while (blockIdx.x >= r.first[i + 1]) ++i;
  const unsigned long long at = (unsigned long long)(blockIdx.x - r.first[i]) * ZERO_BLOCK + threadIdx.x;
#pragma unroll
  for (int k = 0; k < ZERO_BLOCK / 256; ++k)
    if (at + 256 * k < r.words[i]) r.p[i][at + 256 * k] = make_uint4(0u, 0u, 0u, 0u);
}
}  // namespace b2l

extern "C" int b2l_seq_zero_slots(void* const* states, const size_t* slot_bytes, int n, int slot, b2l_stream_t stream) {
  using namespace b2l;
  B2L_CHECK_ARG(n >= 0 && (n == 0 || (states && slot_bytes)) && slot >= 0, "b2l_seq_zero_slots: null pointer or negative size");
  ZeroRanges r{};
  int k = 0;
  auto flush = [&]() -> int {
    if (k == 0) return 0;
    for (int i = k; i < ZERO_RANGES; ++i) r.first[i + 1] = r.first[k];
    seq_zero_kernel<<<r.first[k], 256, 0, (cudaStream_t)stream>>>(r);
    k = 0;
    B2L_LAUNCH_CHECK("seq_zero_kernel");
    return 0;
  };
  for (int i = 0; i < n; ++i) {
    if (slot_bytes[i] == 0) continue;
    char* p = static_cast<char*>(states[i]) + (size_t)slot * slot_bytes[i];
    const unsigned long long words = slot_bytes[i] / 16, blocks = (words + ZERO_BLOCK - 1) / ZERO_BLOCK;
    B2L_CHECK_ARG(states[i] != nullptr, "b2l_seq_zero_slots: null pointer");
    if (slot_bytes[i] % 16 != 0 || ((uintptr_t)p & 15) != 0 || blocks > (1u << 24)) {      // ranges that start or end within a word, and huge ones
      B2L_CUDA(cudaMemsetAsync(p, 0, slot_bytes[i], (cudaStream_t)stream));
      continue;
    }
    r.p[k] = reinterpret_cast<uint4*>(p);
    r.words[k] = words;
    r.first[k + 1] = r.first[k] + (unsigned)blocks;
    if (++k == ZERO_RANGES)
      if (int rc = flush()) return rc;
  }
  return flush();
}

extern "C" int b2l_seq_stream_create(void** stream) {
  B2L_CHECK_ARG(stream != nullptr, "b2l_seq_stream_create: null pointer");
  cudaStream_t s = nullptr;
  B2L_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  *stream = s;
  return 0;
}
