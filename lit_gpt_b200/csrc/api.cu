// Library-level state of libb200gpt: error string, launch counter, PDL switch, device info.
#include "common.cuh"

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

// Raised by a kernel that gave up a bounded wait (tc05.cuh); one word per device, as every __device__ variable.
__device__ unsigned d_wait_error;

unsigned* wait_error_word() {
  static std::atomic<unsigned*> cached[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  unsigned* p = cached[dev].load(std::memory_order_acquire);
  if (!p) {
    void* a = nullptr;
    if (cudaGetSymbolAddress(&a, d_wait_error) != cudaSuccess) return nullptr;
    p = static_cast<unsigned*>(a);
    cached[dev].store(p, std::memory_order_release);
  }
  return p;
}

}  // namespace b200

extern "C" {

int b200_wait_error(b200_stream_t stream, unsigned int* code) {
  B200_CHECK_ARG(code, "b200_wait_error: null argument");
  unsigned* word = b200::wait_error_word();
  B200_CHECK_ARG(word, "b200_wait_error: no device");
  cudaStream_t st = (cudaStream_t)stream;
  B200_CUDA(cudaMemcpyAsync(code, word, sizeof(unsigned), cudaMemcpyDeviceToHost, st));
  B200_CUDA(cudaStreamSynchronize(st));
  if (*code) B200_CUDA(cudaMemsetAsync(word, 0, sizeof(unsigned), st));
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
