// Library-level state of libb200gpt: error string, launch counter, PDL switch, device info.
#include <mutex>

#include "tc05.cuh"

namespace b200 {

static thread_local char g_err[512] = "";
std::atomic<int64_t> g_launches{0};
std::atomic<int> g_pdl{1};

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}

int sm_count() {
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (cached[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev] = n;
  }
  return cached[dev];
}

// Raised by a kernel that gave up a bounded wait (tc05.cuh): a word per device in pinned host memory, which the device writes and the host
// reads without a copy or a synchronisation.  Kept for the life of the process (captured graphs hold its address).
static std::atomic<unsigned*> g_wait_word[64];

unsigned* wait_error_word() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  unsigned* p = g_wait_word[dev].load(std::memory_order_acquire);
  if (p) return p;
  static std::mutex once;
  std::lock_guard<std::mutex> hold(once);
  p = g_wait_word[dev].load(std::memory_order_acquire);
  if (p) return p;
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;   // the allocation is no part of a graph that this thread may be capturing
  cudaThreadExchangeStreamCaptureMode(&mode);
  void* a = nullptr;
  const cudaError_t e = cudaHostAlloc(&a, sizeof(unsigned), cudaHostAllocMapped | cudaHostAllocPortable);
  cudaThreadExchangeStreamCaptureMode(&mode);
  if (e != cudaSuccess) return nullptr;
  p = static_cast<unsigned*>(a);   // (unified addressing: the device's address is the host's)
  __atomic_store_n(p, 0u, __ATOMIC_RELEASE);
  g_wait_word[dev].store(p, std::memory_order_release);
  return p;
}

bool take_wait_error(int dev) {
  if (dev < 0 && cudaGetDevice(&dev) != cudaSuccess) return false;
  unsigned* p = dev >= 0 && dev < 64 ? g_wait_word[dev].load(std::memory_order_acquire) : nullptr;
  return p && __atomic_load_n(p, __ATOMIC_RELAXED) != 0u && __atomic_exchange_n(p, 0u, __ATOMIC_ACQ_REL) != 0u;
}

// one barrier that nothing arrives on
__global__ void wait_probe_kernel(uint64_t limit_ns, unsigned* err) {
  __shared__ __align__(8) uint64_t s_bar;
  griddep_launch();
  griddep_wait();
  tc::mbar_init(tc::smem_u32(&s_bar), 1);
  tc::mbar_init_fence();
  if (!tc::mbar_wait_slow(tc::smem_u32(&s_bar), 0, limit_ns)) *err = 1u;
}

}  // namespace b200

extern "C" {

uint64_t b200_wait_errors_take(uint64_t devices) {
  uint64_t raised = 0;
  for (int d = 0; d < 64; ++d)
    if (((devices >> d) & 1u) && b200::take_wait_error(d)) raised |= 1ull << d;
  return raised;
}

int b200_wait_error(b200_stream_t stream, unsigned int* code) {
  B200_CHECK_ARG(code, "b200_wait_error: null argument");
  B200_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
  *code = b200::take_wait_error(-1) ? 1u : 0u;
  return B200_OK;
}

int b200_wait_probe(uint64_t limit_ns, b200_stream_t stream) {
  B200_CHECK_ARG(limit_ns <= 2000000000ull, "b200_wait_probe: limit of at most two seconds");
  unsigned* word = b200::wait_error_word();
  B200_CHECK_ARG(word, "b200_wait_probe: no device");
  B200_CUDA(b200::launch(b200::wait_probe_kernel, dim3(1), dim3(1), 0, (cudaStream_t)stream, limit_ns, word));
  return B200_OK;
}

int b200_abi_version(void) { return B200GPT_ABI_VERSION; }

const char* b200_last_error(void) { return b200::g_err; }

int b200_device_info(int* sm_count, int* cc_major, int* cc_minor) {
  int dev = 0;
  B200_CUDA(cudaGetDevice(&dev));
  int n = 0, maj = 0, min = 0;
  B200_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
  B200_CUDA(cudaDeviceGetAttribute(&maj, cudaDevAttrComputeCapabilityMajor, dev));
  B200_CUDA(cudaDeviceGetAttribute(&min, cudaDevAttrComputeCapabilityMinor, dev));
  if (sm_count) *sm_count = n;
  if (cc_major) *cc_major = maj;
  if (cc_minor) *cc_minor = min;
  return B200_OK;
}

int b200_set_pdl(int enabled) { return b200::g_pdl.exchange(enabled ? 1 : 0); }

int64_t b200_launch_count(void) { return b200::g_launches.load(); }

}  // extern "C"
