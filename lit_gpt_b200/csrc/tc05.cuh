// tcgen05 / TMA / mbarrier helpers: the kernels that keep their accumulators in tensor memory (qgemm.cu, qgemm_short.cu, int8.cu, attn_tc05.cu), and delta_chunk.cu, whose
// chain of chunks takes the barriers and the report of waits.
//
// Every wait is bounded: after about two seconds mbar_wait() gives up and returns false, the kernel raises the word wait_error_word()
// hands out and leaves through its ordinary teardown, so that a mistake costs one wrong result and not a hung GPU.  The host reports it: the
// entry points of these kernels refuse the next call (B200_CHECK_WAITS), and the serving loops read the word (b200_wait_errors_take) wherever they
// read a result back.
// Before it leaves, the thread that issues copies waits for the last one into each of its stages, and the thread that issues products, when it
// gave up, for those issued so far: neither may still write into memory that then belongs to another CTA.
#pragma once
#include <cuda.h>  // CUtensorMap (type only; the encoder is resolved at run time through the runtime, no -lcuda)

#include "common.cuh"

namespace b200 {

unsigned* wait_error_word();         // the current device's error word (api.cu); null when it cannot be had
bool take_wait_error(int device);    // true, once, after a kernel on `device` (-1: the current one) raised it

#define B200_CHECK_WAITS(what)                                                                                                       \
  do {                                                                                                                               \
    if (b200::take_wait_error(-1)) {                                                                                                 \
      b200::set_error(what ": a kernel launched earlier on this device gave up a bounded wait; outputs since then are invalid");     \
      return B200_ERR_CUDA;                                                                                                          \
    }                                                                                                                                \
  } while (0)

typedef CUresult (*TensorMapEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                      const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline TensorMapEncodeFn tensor_map_encoder() {
  static TensorMapEncodeFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) p = nullptr;
    return reinterpret_cast<TensorMapEncodeFn>(p);
  }();
  return fn;
}

// A row-major matrix (rows x cols elements, rows `ld_bytes` apart) read in boxes of box_rows x 128 bytes, 128-byte swizzle (or x 64 bytes, 64-byte
// swizzle), zeros outside.  base must be 16-byte aligned and ld_bytes a multiple of 16.
inline bool tensor_map_2d(CUtensorMap* map, CUtensorMapDataType type, int elem_bytes, const void* base, int64_t rows, int64_t cols, int64_t ld_bytes, int box_rows,
                          int box_bytes = 128) {
  const TensorMapEncodeFn enc = tensor_map_encoder();
  if (!enc) return false;
  const cuuint64_t dim[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t stride[1] = {(cuuint64_t)ld_bytes};
  const cuuint32_t box[2] = {(cuuint32_t)(box_bytes / elem_bytes), (cuuint32_t)box_rows};
  const cuuint32_t step[2] = {1u, 1u};
  return enc(map, type, 2, const_cast<void*>(base), dim, stride, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE, box_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

namespace tc {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count)); }
__device__ __forceinline__ void mbar_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// SLEEP: how long one try may sleep, ns.  Waiting threads that come back sooner take issue slots from those that work (qgemm.cu, 4096 -> 14336 int4, 64 rows: 28.5 -> 27.1 us
// with 100000); 0 is the hardware's own limit, for warps that wait in turns for short times (delta_chunk.cu: delta rule per head, fp32, two prompts of 1900 rows in all, 16 heads: the layer 875 us, 882 with 100000).
constexpr uint32_t kTrySleepNs = 100000;
template <uint32_t SLEEP = kTrySleepNs>
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t done;
  if constexpr (SLEEP > 0)
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(done) : "r"(bar), "r"(parity), "r"(SLEEP) : "memory");
  else
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done != 0;
}
// (64 tries take far less than 50 ms: where more went by, the GPU was held up, and the time does not count)
template <uint32_t SLEEP = kTrySleepNs>
__device__ __forceinline__ bool mbar_wait_here(uint32_t bar, uint32_t parity, uint64_t limit_ns = 2000000000ull) {
  if (mbar_try<SLEEP>(bar, parity)) return true;
  uint64_t last, t, spent = 0;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(last));
  for (;;) {
    for (int i = 0; i < 64; ++i)
      if (mbar_try<SLEEP>(bar, parity)) return true;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    spent += t - last < 50000000ull ? t - last : 50000000ull;
    last = t;
    if (spent > limit_ns) return false;
  }
}
// The same behind a call, which keeps it out of the way of the code around.  Where that code issues products, mbar_wait_here took part in what elect() below gained.
template <uint32_t SLEEP = kTrySleepNs>
static __device__ __noinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity, uint64_t limit_ns = 2000000000ull) { return mbar_wait_here<SLEEP>(bar, parity, limit_ns); }
template <uint32_t SLEEP = kTrySleepNs>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  return mbar_try<SLEEP>(bar, parity) || mbar_try<SLEEP>(bar, parity) || mbar_wait_slow<SLEEP>(bar, parity);
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
// True in one lane of a warp whose 32 lanes are all here, the same one every time.  Products and commits, and the copies of the GEMMs, are issued behind `if (elect())` in code
// that the whole warp walks (attn_tc05.cu's two copies for 128 keys stand behind a test of the lane).  Measured: four products and a commit issued behind `lane == 0` take
// 235 clk whatever their width, this way 129 for 128 x 64 x 16 and 502 for 128 x 256 x 16, the tensor core's own time.  The likely cause is that the compiler
// has to take operands of a branch on the lane's number for different ones in each lane.
__device__ __forceinline__ bool elect() {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r)::"memory");
  return r != 0;
}
__device__ __forceinline__ void prefetch_map(const CUtensorMap* map) { asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory"); }

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_smem_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Tensor memory is taken after griddep_wait() only: a CTA that started early and held columns while it waited for the grid before it would
// keep them from that grid's own CTAs.  Past the wait a CTA that blocks here waits for CTAs that run to their end.
template <int COLS>
__device__ __forceinline__ void tmem_alloc(uint32_t slot) {   // one whole warp; the address lands in shared memory
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "n"(COLS) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
template <int COLS>
__device__ __forceinline__ void tmem_free(uint32_t tmem) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(COLS) : "memory");
}

// Shared-memory matrix descriptor of a K-major operand in 128-byte-swizzled rows of 128 bytes (8-row groups 1024 bytes apart): start
// address / 16 | leading offset (unused: 1) | stride offset / 16 | version 1 | SWIZZLE_128B.  +2 in the address field is 32 bytes along K.
__device__ __forceinline__ uint64_t desc_sw128(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// The two words apart: the high one is the same for every address, so that the low one, 32-bit sums, is all that a loop over operands moves.
constexpr uint32_t kDescSw128High = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t desc_sw128_low(uint32_t addr) { return ((addr & 0x3FFFFu) >> 4) | (1u << 16); }
__device__ __forceinline__ uint64_t desc_of(uint32_t low, uint32_t high) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(low), "r"(high));
  return d;
}
__device__ __forceinline__ void commit(uint32_t bar) {   // arrives on `bar` once every MMA issued so far has completed
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// ---- CTA pairs (clusters of two, cta_group::2): the even CTA issues the products of both, each CTA holds half of A's and of B's rows and the
// accumulator rows of its own half of A ----
__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t at_rank(uint32_t addr, uint32_t rank) {   // the same shared-memory address in CTA `rank` of the cluster
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_at(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_cluster(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done != 0;
}
// a wait on a barrier that the other CTA of the pair arrives on
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity) {
  return mbar_try_cluster(bar, parity) || mbar_try_cluster(bar, parity) || (mbar_wait_slow(bar, parity) && mbar_try_cluster(bar, parity));
}
__device__ __forceinline__ bool mbar_wait_cluster_here(uint32_t bar, uint32_t parity) {
  return mbar_try_cluster(bar, parity) || (mbar_wait_here(bar, parity) && mbar_try_cluster(bar, parity));
}
// a box into this CTA's shared memory whose bytes count on a barrier of either CTA of the pair
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t cluster_bar) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(cluster_bar) : "memory");
}
// Two pairs that shared their SMs could each hold one half of what both need: a kernel with pairs takes more than half of an SM's shared memory.
constexpr int kPairMinSmem = 114 * 1024 + 1;
template <int COLS>
__device__ __forceinline__ void tmem_alloc_pair(uint32_t slot) {   // one warp of EACH CTA
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "n"(COLS) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
// bytes (a multiple of 16) of this CTA's shared memory into another CTA's, counted on a barrier there
__device__ __forceinline__ void copy_to_cta(uint32_t cluster_dst, uint32_t src, uint32_t bytes, uint32_t cluster_bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(cluster_dst), "r"(src), "r"(bytes), "r"(cluster_bar) : "memory");
}
template <int COLS>
__device__ __forceinline__ void tmem_free_pair(uint32_t tmem) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(COLS) : "memory");
}
__device__ __forceinline__ void commit_pair(uint32_t bar) {   // arrives on `bar` of both CTAs
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}

// 32 lanes x 32 columns of 32-bit accumulators: thread = lane (row), v[j] = column j.  v is valid after wait_ld(v).
__device__ __forceinline__ void ld32(uint32_t (&v)[32], uint32_t addr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,"
      "%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
        "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]),
        "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]),
        "=r"(v[31])
      : "r"(addr));
}
__device__ __forceinline__ void wait_ld(uint32_t (&v)[32]) {   // v as an operand: nothing that reads it moves ahead of the wait
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]), "+r"(v[9]),
                 "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]), "+r"(v[16]), "+r"(v[17]), "+r"(v[18]), "+r"(v[19]),
                 "+r"(v[20]), "+r"(v[21]), "+r"(v[22]), "+r"(v[23]), "+r"(v[24]), "+r"(v[25]), "+r"(v[26]), "+r"(v[27]), "+r"(v[28]), "+r"(v[29]),
                 "+r"(v[30]), "+r"(v[31])
               ::"memory");
}

// the same with 16 columns
__device__ __forceinline__ void ld16(uint32_t (&v)[16], uint32_t addr) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
                 "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
               : "r"(addr));
}
__device__ __forceinline__ void wait_ld(uint32_t (&v)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]), "+r"(v[9]),
                 "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15])
               ::"memory");
}

}  // namespace tc
}  // namespace b200
