// Prompt GEMM of up to 256 rows: y (M, N) = x (M, K) . dequant(W)^T with the WEIGHTS as the left operand, in tensor memory.
//
// With a few dozen rows the other kernel (qgemm.cu: rows left, 128 of them whatever there are) is bound by its operands' way through shared memory: 16 KB
// of padded rows and 16 KB of weights written and read per k-block of 128 features.  Here 128 features are the 128 lanes of tensor memory: a thread rebuilds 64 k
// of its own feature from the packed codes and writes them there with tcgen05.st; the rows are the right operand, in shared memory and no wider than they are,
// and the accumulator has a column per row.  Per CTA:
//   * warp 17 fetches 256 k of 128 features at a time (16 KB, 128 bytes a row) by TMA, warp 18 their scales by cp.async (8 or 16 bytes a row), ahead of the rest;
//   * warps 0-15, four groups of 128 threads, rebuild every fourth k-block each with exactly the dequantise kernel's arithmetic (bf16_rn(code_fp32 *
//     absmax_fp32), bf16_rn(scale * (q - zero))).  nf4 / fp4 look up BOTH codes of a byte at once: 256 entries of two fp32 numbers, a copy for every lane, at a
//     shared-memory address whose second byte is the code byte, so that one PRMT makes the address: PRMT + LDS.64 + 2 FMUL + a conversion for two codes;
//   * warp 16 fetches the rows by TMA, zeros past the last; warp 19 issues tcgen05.mma (128 x rows x 16, A in tensor memory);
//   * the sixteen warps read the accumulator and store 32 neighbouring features of a row per access.
// K is walked by CTAs in equal ranges of all the k there is to do (tiles x K / 256 units): a tile that a range's end cuts is finished by
// short_reduce_kernel, which adds the ranges' fp32 sums in their order.  Nothing waits for another CTA.
// PAIR: gate and up projection of a gated MLP, two accumulators per tile of 128 features, each stage of rows used twice; stores silu(gate) * up with
// the roundings of the separate launches.
// Bound: the rebuilding warps, issue slots and the latency of their chain (wait, codes, arithmetic, tensor memory, hand-over): 0.87 us a unit of 256 k, nf4 and int4, at 17
// rows, 1.3 at 203, where 0.42 is what the weights take from HBM.  us, qgemm.cu / here, weights in turn: 4096 -> 14336 nf4 at 17, 64, 129, 203 rows 35 / 21, 36 / 23,
// 42 / 27, 42 / 32, int4 26 / 21, 27 / 22, 34 / 27, 34 / 31; 14336 -> 4096 at 64 nf4 37 / 25, int4 29 / 24; the pair of 4096 -> 14336 in one launch, against two and the
// product, at 17 / 64 rows nf4 74 / 37, 75 / 41, int4 55 / 38, 57 / 41,
// and against one launch of qgemm.cu at 129 / 203 80 / 50, 80 / 66, int4 63 / 52, 63 / 65.
#include "qgemm_short.cuh"
#include "tc05.cuh"

namespace b200 {

namespace {

constexpr int kShGroups = 4, kShWarps = 4 * kShGroups, kShThreads = (kShWarps + 4) * 32;   // rebuilding; rows, weights, scales, products
constexpr int kShStage = 128 * 128 + 128 * 16;        // 256 k of 128 features: packed codes and scales
constexpr int kShLow = 3;                             // stages below the table of byte pairs
constexpr int kShTable = 256 * 256;
constexpr int kShMaxPair = 208;                       // rows of a gate / up pair: two accumulators beside the rebuilt weights
constexpr int kShSmem = 227 * 1024 - 2048;            // dynamic shared memory (static: barriers)
constexpr int kShMaxW = 8, kShMaxB = 4, kShA = 2, kShMaxRing = 8;   // most stages of weights and rows; stages of rebuilt weights (256 k: 128 columns each, handed over in halves)

struct ShortParams {
  ShortArgs a;
  int tiles, nq, shared, nb;                          // tiles of 128 features, units (256 k) a tile, ..., accumulator columns (rows up to a multiple of 16)
  int ws, bs, ring;                                   // stages of weights and of rows; of single rebuilt k-blocks (a pair of more than 128 rows)
};

// Room for the partial sums of CTA c's part of tile t.  Parts in the order of their k step on by a CTA, a tile or both, so that c + t is another number for each; where
// tiles are more than CTAs, a CTA has two cut ones at most: the one its range begins in and the one (`head`) that it ends in.
__device__ __forceinline__ int64_t part_slot(int64_t c, int64_t t, bool head, int64_t ctas, int64_t tiles) { return tiles <= ctas ? c + t : 2 * c + head; }

__device__ __forceinline__ int64_t unit_begin(int64_t c, int64_t ctas, int64_t tiles, int64_t nq, bool shared) {
  return shared ? c * (tiles * nq) / ctas : (c * tiles / ctas) * nq;
}

// b: the low word of a tc::desc_sw128 descriptor, whose high word is the same for every address
__device__ __forceinline__ void umma_ts(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 bd;\n\tsetp.ne.b32 p, %4, 0;\n\tmov.b64 bd, {%2, %5};\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], bd, %3, p;\n\t}"
               ::"r"(d), "r"(a), "r"(b), "r"(idesc), "r"(accumulate), "n"(tc::kDescSw128High) : "memory");
}
__device__ __forceinline__ void st8(uint32_t addr, const uint32_t (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
               ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}

// 64 int4 codes of one group to bf16_rn(scale * (q - zero)).  A zero point that is a whole number up to 16 (the quantiser's are 0 .. 15): two codes at a time, as
// halves of a word.  128 + q is a bf16 number with the code in its last bits, d = q - zero is exact, and with the scale's eleven bits as a sum of two bf16 numbers
// d * lo is exact too (5 bits x 3), so that the fused d * hi + d * lo is rounded once: PRMT + LOP3 + HADD2 + HMUL2 + HFMA2 for two codes, and a shift for eight.
// Other zero points: one mixed-precision FMA for each code, as in qgemm.cu.
__device__ __forceinline__ void rebuild_int4(uint32_t to, const uint32_t (&qw)[8], uint32_t sc) {
  const __half2 h2 = *reinterpret_cast<const __half2*>(&sc);
  const float scale = __low2float(h2), zero = __high2float(h2);
  if (__all_sync(0xffffffffu, zero >= 0.f && zero <= 16.f && zero == rintf(zero))) {
    const __nv_bfloat162 hi = __float2bfloat162_rn(scale), lo = __float2bfloat162_rn(scale - __low2float(hi)), z = __float2bfloat162_rn(128.f + zero);
    uint32_t mask, base;   // (in registers: an instruction takes one constant)
    asm volatile("mov.b32 %0, 0x000f000f;\n\tmov.b32 %1, 0x43004300;" : "=r"(mask), "=r"(base));
#pragma unroll
    for (int w = 0; w < 8; w += 2) {
      uint32_t o[8];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const uint32_t odd = qw[w + i] >> 4;
#pragma unroll
        for (int e = 0; e < 4; ++e) {   // byte e: codes 2 e and 2 e + 1
          uint32_t x;
          asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(x) : "r"(__byte_perm(qw[w + i], odd, 0x4400 + 0x1111 * e)), "r"(mask), "r"(base));
          const __nv_bfloat162 d = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&x), z), v = __hfma2(d, hi, __hmul2(d, lo));
          o[4 * i + e] = *reinterpret_cast<const uint32_t*>(&v);
        }
      }
      st8(to + 4 * w, o);
    }
    return;
  }
  const float c0 = -scale * (16.0f + zero);
  const uint16_t hs = (uint16_t)(sc & 0xffffu);
#pragma unroll
  for (int w = 0; w < 8; w += 2) {
    uint32_t o[8];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float f[8];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint32_t sh = e < 2 ? qw[w + i] << (6 - 4 * e) : qw[w + i] >> (4 * e - 6);
        asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %2;\n\tfma.rn.f32.f16 %0, l, %3, %4;\n\tfma.rn.f32.f16 %1, h, %3, %4;\n\t}"
            : "=f"(f[e]), "=f"(f[e + 4]) : "r"((sh & 0x03c003c0u) | 0x4c004c00u), "h"(hs), "f"(c0));
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) o[4 * i + e] = pack_bf16(f[2 * e], f[2 * e + 1]);
    }
    st8(to + 4 * w, o);
  }
}

__device__ __forceinline__ float silu_mul(float g, float u) {   // the roundings of two GEMMs and b200_swiglu
  const float a = round_bf16(g);
  return round_bf16(a / (1.0f + expf(-a))) * round_bf16(u);
}

template <bool INT4, bool PAIR, int BQ>   // BQ: k-blocks (64 k) of a stage of rows
__global__ void __launch_bounds__(kShThreads, 1)
qgemm_short_kernel(const __grid_constant__ ShortParams p, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                   const __grid_constant__ CUtensorMap map_w2, unsigned* err) {
  constexpr int NACC = PAIR ? 2 : 1;
  constexpr bool RING = PAIR && BQ == 1;   // accumulators that leave less than two stages of rebuilt weights: single k-blocks in turn (p.ring of them)
  extern __shared__ __align__(1024) uint8_t sh_smem[];
  __shared__ __align__(8) uint64_t s_bars[2 * (kShMaxW + kShMaxB + kShMaxRing) + 3];
  __shared__ uint32_t s_tmem;
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // (uniform, and known to be)
  const uint32_t base = (tc::smem_u32(sh_smem) + 1023u) & ~1023u;
  // the table's address is a multiple of 64 KB: the code byte is then the second byte of its entry's address
  const uint32_t table = (base + kShLow * kShStage + 0xffffu) & ~0xffffu;
  const uint32_t above = INT4 ? base + (uint32_t)p.ws * kShStage : table + kShTable;
  auto w_stage = [&](int i) { return INT4 || i < kShLow ? base + (uint32_t)i * kShStage : above + (uint32_t)(i - kShLow) * kShStage; };
  const uint32_t rows = ((INT4 ? above : above + (uint32_t)(p.ws > kShLow ? p.ws - kShLow : 0) * kShStage) + 1023u) & ~1023u;
  const uint32_t row_block = (uint32_t)p.nb * 128u, row_stage = BQ * row_block;
  const uint32_t bars = tc::smem_u32(s_bars);
  const uint32_t w_full = bars, w_empty = w_full + 8 * kShMaxW, b_full = w_empty + 8 * kShMaxW, b_empty = b_full + 8 * kShMaxB, a_full = b_empty + 8 * kShMaxB,
                 a_empty = a_full + 8 * kShMaxRing, acc_full = a_empty + 8 * kShMaxRing, acc_free = acc_full + 8, idle = acc_full + 16;
  if (rows + (uint32_t)p.bs * row_stage > tc::smem_u32(sh_smem) + (uint32_t)kShSmem) {   // (a layout of shared memory other than the host counts with)
    if (tid == 0) *err = 1u;
    return;
  }
  if (tid == 0) {
    for (int i = 0; i < p.ws; ++i) { tc::mbar_init(w_full + 8 * i, 1 + 32); tc::mbar_init(w_empty + 8 * i, 1); }
    for (int i = 0; i < p.bs; ++i) { tc::mbar_init(b_full + 8 * i, 1); tc::mbar_init(b_empty + 8 * i, 1); }
    for (int i = 0; i < (RING ? 8 : 2 * kShA); ++i) { tc::mbar_init(a_full + 8 * i, RING ? 4 : kShWarps / 2); tc::mbar_init(a_empty + 8 * i, 1); }
    tc::mbar_init(acc_full, 1);
    tc::mbar_init(acc_free, kShWarps);
    tc::mbar_init(idle, 1);
    tc::mbar_init_fence();
    tc::prefetch_map(&map_x);
    tc::prefetch_map(&map_w);
  }
  if (!INT4) {   // entry e: the values of byte e's high and low nibble (even element first), once per lane
    const float code = code_value(p.a.qtype, lane & 15);
    for (int e = warp; e < 256; e += kShThreads / 32)
      asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(table + (uint32_t)(e * 256 + lane * 8)), "f"(__shfl_sync(0xffffffffu, code, e >> 4)), "f"(__shfl_sync(0xffffffffu, code, e & 15)));
  }
  const int64_t nq = p.nq, u0 = unit_begin(blockIdx.x, gridDim.x, p.tiles, nq, p.shared != 0), u1 = unit_begin(blockIdx.x + 1, gridDim.x, p.tiles, nq, p.shared != 0);
  griddep_launch();
  if (warp == kShWarps + 1 && lane == 0)   // the first weights on their way to L2, where nothing can be stale
    for (int64_t u = u0; u < u1 && u < u0 + (PAIR ? 2 : 4); ++u) {
      const int tile = (int)(u / nq), k = (int)(u - tile * nq);
#pragma unroll
      for (int m = 0; m < NACC; ++m)
        asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(m ? &map_w2 : &map_w), "r"(k * 128), "r"(tile * 128) : "memory");
    }
  griddep_wait();
  if (warp == kShWarps + 3) tc::tmem_alloc<512>(tc::smem_u32(&s_tmem));
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = s_tmem, acc0 = tmem + (RING ? 32u * (uint32_t)p.ring : 128u * kShA);   // rebuilt weights, then the accumulators
  struct Segment { int tile, q0, n; };
  auto segment = [&](int64_t u) {
    Segment s;
    s.tile = (int)(u / nq);
    s.q0 = (int)(u - s.tile * nq);
    s.n = (int)(u1 - u < nq - s.q0 ? u1 - u : nq - s.q0);
    return s;
  };
  bool ok = true;
  // before a warp that issues copies leaves: the last one into each of its `n` stages.  `s`, `ph`: its next stage, and the parity it would wait for there
  auto drain = [&](uint32_t full, int n, int s, uint32_t ph) {
    for (int i = 0; i < n; ++i) {   // (a stage never used: the phase before the first)
      if (--s < 0) { s = n - 1; ph ^= 1u; }
      ok = __all_sync(0xffffffffu, tc::mbar_wait(full + 8 * s, ph ^ 1u)) && ok;
    }
  };

  if (warp < kShWarps) {
    // =========================================== REBUILD, THEN STORE ============================================
    const int g = warp >> 2, row = (warp & 3) * 32 + lane;       // group: every fourth k-block; this thread's feature in the tile
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16, lane_table = table | (uint32_t)lane * 8u;
    int sw = 0;                                                   // next stage of weights, and its parity
    uint32_t pw = 0u, acc_ph = 0u, i = 0u;                        // i: tiles of rebuilt weights so far
    uint32_t qw[8], sc;
    int left = (int)(u1 - u0) * NACC, at = (int)(u0 - (u0 / nq) * nq) * NACC, done = 0;   // tiles to come; in the output tile so far, before and in this segment
    const uint32_t code0 = (uint32_t)(row * 128 + (((2 * g) ^ (row & 7)) << 4)), code1 = (uint32_t)(row * 128 + (((2 * g + 1) ^ (row & 7)) << 4));
    const uint32_t scale0 = 16384u + (uint32_t)(INT4 ? row * 8 + (g >> 1) * 4 : row * 16 + g * 4);
    const uint32_t half_full = a_full + 8 * (g >> 1), half_empty = a_empty + 8 * (g >> 1), to0 = tmem + lanes + 32u * (uint32_t)g;
    auto fetch = [&]() {                                          // the next stage's codes and scale into registers
      ok = ok && __all_sync(0xffffffffu, tc::mbar_wait_here(w_full + 8 * sw, pw));
      if (!ok) return;
      const uint32_t st = w_stage(sw);
      asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(qw[0]), "=r"(qw[1]), "=r"(qw[2]), "=r"(qw[3]) : "r"(st + code0));
      asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(qw[4]), "=r"(qw[5]), "=r"(qw[6]), "=r"(qw[7]) : "r"(st + code1));
      asm volatile("ld.shared.u32 %0, [%1];" : "=r"(sc) : "r"(st + scale0));
      if (++sw == p.ws) { sw = 0; pw ^= 1u; }
    };
    // A ring's k-blocks stand in the order of their products: of a unit the gate's and the up projection's first two, then their last two.  Number n takes the room of
    // n - ring; either's hand-overs go by barrier n % 8, so that no wait is for a phase but the present one: a group's steps from one k-block to its next are 2 and 6.
    int n = (g >> 1) * 4 + (g & 1);
    fetch();
    for (int64_t u = u0; ok;) {
      const uint32_t full = RING ? a_full + 8 * (n & 7) : half_full + 16 * (i & 1u), to = RING ? tmem + lanes + 32u * (uint32_t)(n % p.ring) : to0 + 128u * (i & 1u);
      if constexpr (RING) {
        const int before = n - p.ring;
        if (before >= 0) ok = __all_sync(0xffffffffu, tc::mbar_wait_here(a_empty + 8 * (before & 7), (uint32_t)(before >> 3) & 1u));
      } else {
        ok = __all_sync(0xffffffffu, tc::mbar_wait_here(half_empty + 16 * (i & 1u), ((i >> 1) & 1u) ^ 1u));
      }
      if (!ok) break;
      tc::fence_after();
      if constexpr (INT4) {
        rebuild_int4(to, qw, sc);
      } else {
        const float am = __uint_as_float(sc);
#pragma unroll
        for (int w = 0; w < 8; w += 2) {
          uint32_t o[8];
#pragma unroll
          for (int b = 0; b < 8; ++b) {
            float hi, lo;
            const uint32_t addr = __byte_perm(qw[w + (b >> 2)], lane_table, 0x7604 | ((b & 3) << 4));   // table | byte << 8 | lane << 3
            asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(hi), "=f"(lo) : "r"(addr));
            o[b] = pack_bf16(hi * am, lo * am);
          }
          st8(to + 4 * w, o);
        }
      }
      if (--left > 0) fetch();                                    // while tensor memory is written
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc::fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(full);
      if (RING) n += i & 1u ? 6 : 2;
      ++i;
      ++done;
      if (left > 0 && at + done < (int)nq * NACC) continue;
      const Segment t = segment(u);
      at = done = 0;
      // ---- accumulator(s) -> y or partial sums: lane = feature, column = row ----
      ok = ok && __all_sync(0xffffffffu, tc::mbar_wait(acc_full, acc_ph));
      acc_ph ^= 1u;
      if (!ok) break;
      tc::fence_after();
      const bool whole = t.n == p.nq;
      const int64_t n = (int64_t)t.tile * 128 + row, M = p.a.M, N = p.a.N;
      float* const part = p.a.partial + part_slot(blockIdx.x, t.tile, t.q0 == 0, gridDim.x, p.tiles) * NACC * M * 128 + row;
      const float bias = !PAIR && whole && p.a.bias && n < N ? __bfloat162float(p.a.bias[n]) : 0.f;
#pragma unroll 1
      for (int c0 = g * 16; c0 < p.nb; c0 += kShGroups * 16) {
        uint32_t v[16], w[16];
        tc::ld16(v, acc0 + lanes + (uint32_t)c0);
        if constexpr (PAIR) tc::ld16(w, acc0 + lanes + (uint32_t)(p.nb + c0));
        tc::wait_ld(v);
        if constexpr (PAIR) tc::wait_ld(w);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int64_t r = c0 + j;
          if (r < M) {
            if (!whole) {
              part[r * 128] = __uint_as_float(v[j]);
              if constexpr (PAIR) part[(M + r) * 128] = __uint_as_float(w[j]);
            } else if (n < N) {
              if constexpr (PAIR) p.a.y[r * N + n] = __float2bfloat16_rn(silu_mul(__uint_as_float(v[j]), __uint_as_float(w[j])));
              else p.a.y[r * N + n] = __float2bfloat16_rn(__uint_as_float(v[j]) + bias);
            }
          }
        }
        __syncwarp();   // (the next loads of tensor memory want the whole warp)
      }
      tc::fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(acc_free);
      u += t.n;
      if (u >= u1) break;
    }
  } else if (warp == kShWarps) {
    // =========================================== ROWS ===========================================================
    int s = 0;
    uint32_t ph = 1u;
    for (int64_t u = u0; u < u1 && ok; ++u) {
      const int k0 = (int)(u - (u / nq) * nq) * 256;
      for (int l = 0; l < 4; l += BQ) {
        ok = __all_sync(0xffffffffu, tc::mbar_wait(b_empty + 8 * s, ph));
        if (!ok) break;
        if (tc::elect()) {
          tc::mbar_expect_tx(b_full + 8 * s, row_stage);
#pragma unroll
          for (int e = 0; e < BQ; ++e) tc::tma_load_2d(rows + s * row_stage + e * row_block, &map_x, k0 + (l + e) * 64, 0, b_full + 8 * s);
        }
        __syncwarp();
        if (++s == p.bs) { s = 0; ph ^= 1u; }
      }
    }
    drain(b_full, p.bs, s, ph);
  } else if (warp == kShWarps + 1) {
    // =========================================== PACKED WEIGHTS =================================================
    int s = 0;
    uint32_t ph = 1u;
    for (int64_t u = u0; u < u1 && ok; ++u) {
      const int tile = (int)(u / nq), k = (int)(u - tile * nq);
#pragma unroll
      for (int m = 0; m < NACC; ++m) {
        ok = ok && __all_sync(0xffffffffu, tc::mbar_wait(w_empty + 8 * s, ph));
        if (!ok) break;
        if (tc::elect()) {
          tc::mbar_expect_tx(w_full + 8 * s, 16384u);
          tc::tma_load_2d(w_stage(s), m ? &map_w2 : &map_w, k * 128, tile * 128, w_full + 8 * s);
        }
        __syncwarp();
        if (++s == p.ws) { s = 0; ph ^= 1u; }
      }
    }
    drain(w_full, p.ws, s, ph);
  } else if (warp == kShWarps + 2) {
    // =========================================== SCALES =========================================================
    // (a warp of their own: a thread's next arrival on a barrier waits for the copies it has under way)
    uint32_t i = 0;
    for (int64_t u = u0; u < u1 && ok; ++u) {
      const int tile = (int)(u / nq), k = (int)(u - tile * nq);
#pragma unroll
      for (int m = 0; m < NACC; ++m, ++i) {
        const uint32_t s = i % (uint32_t)p.ws, dst = w_stage((int)s) + 16384u;
        ok = ok && __all_sync(0xffffffffu, tc::mbar_wait(w_empty + 8 * s, ((i / (uint32_t)p.ws) & 1u) ^ 1u));
        if (!ok) break;
#pragma unroll
        for (int e = 0; e < 4; ++e) {   // rows past the last feature take its scales: their sums are not stored
          const int r = e * 32 + lane;
          int64_t n = (int64_t)tile * 128 + r;
          if (n >= p.a.N) n = p.a.N - 1;
          if constexpr (INT4)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + (uint32_t)r * 8u), "l"(p.a.scale[m] + n * (p.a.K >> 7) + k * 2) : "memory");
          else
            asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst + (uint32_t)r * 16u), "l"(p.a.scale[m] + n * (p.a.K >> 6) + k * 4) : "memory");
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared.b64 [%0];" ::"r"(w_full + 8 * s) : "memory");
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (tc::elect()) {
    // =========================================== PRODUCTS =======================================================
    // One thread, chosen by tc::elect.  A stage's number is a constant of its copy of the code, and addresses are 32-bit
    // sums of constants and what stands before the loop.  (Two and four issuing warps with an accumulator each took as long: a stage's
    // chain of wait, rebuilding and hand-over in the sixteen warps is what a unit takes.)
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.nb >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
    const uint32_t row_desc = (rows >> 4) | (1u << 16), block_step = row_block >> 4, stage_step = row_stage >> 4;
    int sb = 0, sw = 0, at = (int)(u0 - (u0 / nq) * nq);      // the unit's first stage of rows; next stage of weights; unit within the tile
    uint32_t pa = 0u, pb = 0u, free_ph = 1u, fresh = 1u;      // fresh: a segment's first unit
    int left = (int)(u1 - u0);
    if constexpr (RING) {
      int slot = 0;
      for (; left > 0 && ok; --left) {
        if (fresh) {
          ok = tc::mbar_wait_here(acc_free, free_ph);
          free_ph ^= 1u;
        }
#pragma unroll
        for (int c = 0; c < 8; ++c) {                         // k-blocks 0 and 1 of the gate, of the up projection, 2 and 3 likewise
          const int l = (c >> 2) * 2 + (c & 1), m = (c >> 1) & 1;
          int s = sb + l;
          uint32_t ph = pb;
          if (s >= p.bs) { s -= p.bs; ph ^= 1u; }
          if (m == 0) ok = ok && tc::mbar_wait_here(b_full + 8 * s, ph);
          ok = ok && tc::mbar_wait_here(a_full + 8 * c, pa);
          if (!ok) break;
          tc::fence_after();
          const uint32_t db = row_desc + s * stage_step, ta = tmem + 32u * (uint32_t)slot;
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_ts(acc0 + (m ? (uint32_t)p.nb : 0u), ta + (uint32_t)(8 * k), db + 2 * k, idesc, l | k ? 1u : fresh ^ 1u);
          tc::commit(a_empty + 8 * c);
          if (m == 1) tc::commit(b_empty + 8 * s);
          if (l == 3) {
            tc::commit(w_empty + 8 * sw);
            if (++sw == p.ws) sw = 0;
          }
          if (++slot == p.ring) slot = 0;
        }
        pa ^= 1u;
        sb += 4;
        while (sb >= p.bs) { sb -= p.bs; pb ^= 1u; }
        fresh = 0u;
        if (++at == p.nq || left == 1) {
          if (ok) tc::commit(acc_full);
          at = 0;
          fresh = 1u;
        }
      }
    }
    while (left > 0 && ok) {
#pragma unroll
      for (int sa = 0; sa < kShA; ++sa) {                     // one unit a stage; of a pair one unit, its gate and its up projection
        if (left <= 0 || !ok) break;
        if (fresh && (!PAIR || sa == 0)) {
          ok = tc::mbar_wait_here(acc_free, free_ph);
          free_ph ^= 1u;
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          ok = ok && tc::mbar_wait_here(a_full + 16 * sa + 8 * q, pa);
          if (!ok) break;
#pragma unroll
          for (int l = 2 * q; l < 2 * q + 2; ++l) {
            int s = sb + l / BQ;
            uint32_t ph = pb;
            if (s >= p.bs) { s -= p.bs; ph ^= 1u; }
            if ((!PAIR || sa == 0) && l % BQ == 0) ok = ok && tc::mbar_wait_here(b_full + 8 * s, ph);
            if (!ok) break;
            tc::fence_after();
            const uint32_t db = row_desc + s * stage_step + (l % BQ) * block_step;
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_ts(acc0 + (PAIR && sa ? (uint32_t)p.nb : 0u), tmem + (uint32_t)(128 * sa + 32 * l + 8 * k), db + 2 * k, idesc, l | k ? 1u : fresh ^ 1u);
            if ((!PAIR || sa == 1) && (l + 1) % BQ == 0) tc::commit(b_empty + 8 * s);
          }
          if (!ok) break;
          tc::commit(a_empty + 16 * sa + 8 * q);
          if (q == 1) tc::commit(w_empty + 8 * sw);           // (what was rebuilt from them is multiplied)
        }
        if (++sw == p.ws) sw = 0;
        if (!PAIR || sa == 1) {
          sb += 4 / BQ;
          while (sb >= p.bs) { sb -= p.bs; pb ^= 1u; }       // (a unit's four stages can be more than all there are)
          fresh = 0u;
          --left;
          if (++at == p.nq || left == 0) {
            if (ok) tc::commit(acc_full);
            at = 0;
            fresh = 1u;
          }
        }
      }
      pa ^= 1u;
    }
    if (!ok) {
      tc::commit(idle);
      tc::mbar_wait(idle, 0);
    }
  }
  if (!ok) *err = 1u;
  tc::fence_before();
  __syncthreads();
  if (warp == kShWarps + 3) {
    __syncwarp();
    tc::tmem_free<512>(tmem);
  }
}

// Tiles that two CTAs or more share: their sums in the order of the ranges, + bias.  A CTA takes eight rows of a tile, a thread four features.
template <bool PAIR>
__global__ void __launch_bounds__(256) short_reduce_kernel(const ShortArgs a, int tiles, int nq, int ctas) {
  griddep_launch();
  const int64_t t = blockIdx.y, total = (int64_t)tiles * nq;
  const int64_t first = ((t * nq + 1) * ctas - 1) / total, last = ((t + 1) * nq * (int64_t)ctas - 1) / total;   // the CTAs of its first and last unit
  griddep_wait();   // (by every CTA: a grid that ended before the one ahead of it would let the next one start on unfinished results)
  if (first == last) return;
  const int64_t r = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5), f = (threadIdx.x & 31) * 4, n = t * 128 + f;
  if (r >= a.M || n >= a.N) return;
  constexpr int NACC = PAIR ? 2 : 1;
  float s[NACC][4] = {};
  for (int64_t c = first; c <= last; ++c) {
#pragma unroll
    for (int m = 0; m < NACC; ++m) {
      const float4 v = *reinterpret_cast<const float4*>(a.partial + ((part_slot(c, t, c == first, ctas, tiles) * NACC + m) * a.M + r) * 128 + f);
      s[m][0] += v.x; s[m][1] += v.y; s[m][2] += v.z; s[m][3] += v.w;
    }
  }
  uint32_t o[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    float v[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      if constexpr (PAIR) v[i] = silu_mul(s[0][2 * e + i], s[NACC - 1][2 * e + i]);
      else v[i] = s[0][2 * e + i] + (a.bias ? __bfloat162float(a.bias[n + 2 * e + i]) : 0.f);
    }
    o[e] = pack_bf16(v[0], v[1]);
  }
  *reinterpret_cast<uint2*>(a.y + r * a.N + n) = make_uint2(o[0], o[1]);
}

template <bool INT4, bool PAIR, int BQ>
cudaError_t launch_kind(const ShortArgs& a, const ShortPlan& plan, cudaStream_t st) {
  static PerDeviceOnce once;
  if (once.need()) {
    const cudaError_t e = cudaFuncSetAttribute(qgemm_short_kernel<INT4, PAIR, BQ>, cudaFuncAttributeMaxDynamicSharedMemorySize, kShSmem);
    if (e != cudaSuccess) return e;
    once.done();
  }
  ShortParams p{};
  p.a = a;
  p.tiles = (int)((a.N + 127) / 128);
  p.nq = (int)(a.K / 256);
  p.shared = plan.shared;
  p.nb = (int)((a.M + 15) / 16 * 16);
  // rows: up to kShMaxB stages; what they leave is the weights'
  const int all = INT4 ? kShSmem - 2048 : kShSmem + 1024 - 0x20000;   // (int4: no table; else what lies above it, at 128 KB, whatever the kernel's own first address)
  const int stage = BQ * p.nb * 128;
  p.bs = (all - (INT4 ? 4 : PAIR ? 1 : 0) * kShStage) / stage;
  if (p.bs > kShMaxB) p.bs = kShMaxB;
  p.ring = (512 - 2 * p.nb) / 32 < kShMaxRing ? (512 - 2 * p.nb) / 32 : kShMaxRing;
  p.ws = (INT4 ? 0 : kShLow) + (all - p.bs * stage) / kShStage;
  if (p.ws > kShMaxW) p.ws = kShMaxW;
  alignas(64) CUtensorMap mx, mw, mw2;
  if (!tensor_map_2d(&mx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a.x, a.M, a.K, a.K * 2, p.nb) ||
      !tensor_map_2d(&mw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a.packed[0], a.N, a.K / 2, a.K / 2, 128) ||
      !tensor_map_2d(&mw2, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a.packed[PAIR ? 1 : 0], a.N, a.K / 2, a.K / 2, 128))
    return cudaErrorInvalidValue;
  unsigned* const err = wait_error_word();
  if (!err) return cudaErrorMemoryAllocation;
  const cudaError_t e = launch(qgemm_short_kernel<INT4, PAIR, BQ>, dim3((unsigned)plan.ctas), dim3(kShThreads), (size_t)kShSmem, st, p, mx, mw, mw2, err);
  if (e != cudaSuccess || !plan.shared) return e;
  return launch(short_reduce_kernel<PAIR>, dim3((unsigned)((a.M + 7) / 8), (unsigned)p.tiles), dim3(256), (size_t)0, st, a, p.tiles, p.nq, plan.ctas);
}

// k-blocks a stage of rows: as many as 32 KB hold, so that few rows, whose products are short, are waited for less often
template <bool INT4, bool PAIR>
cudaError_t launch_rows(const ShortArgs& a, const ShortPlan& plan, cudaStream_t st) {
  if (a.M <= 64) return launch_kind<INT4, PAIR, 4>(a, plan, st);
  return a.M <= 128 ? launch_kind<INT4, PAIR, 2>(a, plan, st) : launch_kind<INT4, PAIR, 1>(a, plan, st);
}

}  // namespace

bool short_takes(const ShortArgs& a, bool pair) {
  if (a.M < 1 || a.M > (pair ? kShMaxPair : 256) || a.K % 256 || a.N % 8 || a.N > 65535 * 128LL) return false;
  uintptr_t low = 0;
  for (int i = 0; i < (pair ? 2 : 1); ++i) low |= reinterpret_cast<uintptr_t>(a.packed[i]) | reinterpret_cast<uintptr_t>(a.scale[i]);
  return ((low | reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.y)) & 15) == 0;
}

// us of a launch: what it starts and ends with, what a unit (256 k of 128 features, of a pair both matrices') takes, per accumulator column more, and what is
// stored or summed by its CTAs.  Fitted to 13 shapes x 12 numbers of rows from 17 to 256 (one round of CTAs, weights in turn: 2 to 5 % rms).
struct ShortCost {
  double start, unit, column, out;
};
static double short_time(int64_t units, int64_t ctas, int nb, const ShortCost& c) {
  return c.start + (double)units * (c.unit + c.column * nb) + c.out * 1e-3 * (double)ctas * nb;
}

ShortPlan short_shape(int64_t N, int64_t K, bool shared) {
  const int64_t tiles = (N + 127) / 128, sms = sm_count(), most = shared ? tiles * (K / 256) : tiles;
  return {(int)(most < sms ? most : sms), shared, 0.0};
}

ShortPlan short_plan(int64_t M, int64_t N, int64_t K, int qtype, bool pair, bool scratch) {
  // [int4][rows up to 64, 128, 256][whole tiles, shared]; pairs [int4][rows up to 128, 208][whole, shared]
  static const ShortCost one[2][3][2] = {{{{4.53, 0.856, 0.0018, 0.512}, {7.04, 1.028, 0.0025, 0.275}},
                                          {{5.40, 0.766, 0.0024, 0.298}, {7.32, 0.980, 0.0036, 0.217}},
                                          {{7.44, 0.433, 0.0041, 0.218}, {6.17, 1.159, 0.0033, 0.241}}},
                                         {{{4.71, 0.930, 0.0, 0.547}, {6.96, 1.108, 0.0, 0.273}},
                                          {{5.75, 0.839, 0.0012, 0.306}, {7.30, 1.004, 0.0022, 0.218}},
                                          {{7.53, 0.584, 0.0029, 0.234}, {5.95, 1.058, 0.0031, 0.246}}}};
  static const ShortCost two[2][2][2] = {{{{3.79, 2.009, 0.00335, 0.17}, {9.85, 1.836, 0.00676, 0.29}}, {{10.91, 0.202, 0.0143, 0.222}, {8.19, 2.219, 0.0086, 0.373}}},
                                         {{{2.43, 2.244, 0.00124, 0.25}, {9.13, 2.103, 0.00399, 0.29}}, {{10.76, 0.703, 0.0112, 0.246}, {8.19, 2.117, 0.0089, 0.328}}}};
  ShortPlan best{0, false, 0.0};
  if (M < 1 || M > (pair ? kShMaxPair : 256) || N < 1 || K < 256 || K % 256 || N % 8) return best;
  const int64_t tiles = (N + 127) / 128, nq = K / 256, sms = sm_count(), total = tiles * nq;
  const int nb = (int)((M + 15) / 16 * 16), rows = M <= 64 ? 0 : M <= 128 ? 1 : 2;
  const bool int4 = qtype == B200_Q_INT4;
  const ShortCost* const cost = pair ? two[int4][rows == 2] : one[int4][rows];
  best = short_shape(N, K, false);
  best.time = short_time((tiles + sms - 1) / sms * nq, best.ctas, nb, cost[0]);
  if (scratch) {
    ShortPlan s = short_shape(N, K, true);
    const int64_t units = (total + s.ctas - 1) / s.ctas;
    s.time = short_time(units, s.ctas, nb, cost[1]);
    if (units < (tiles + sms - 1) / sms * nq && s.time < best.time) best = s;
  }
  return best;
}

size_t short_scratch_bytes(int64_t M, int64_t N, const ShortPlan& plan, bool pair) {
  const int64_t tiles = (N + 127) / 128, slots = tiles <= plan.ctas ? plan.ctas + tiles - 1 : 2 * (int64_t)plan.ctas;   // (part_slot)
  return plan.shared ? (size_t)slots * (pair ? 2 : 1) * (size_t)M * 128 * sizeof(float) : 0;
}

cudaError_t launch_short(const ShortArgs& a, const ShortPlan& plan, bool pair, cudaStream_t st) {
  const bool int4 = a.qtype == B200_Q_INT4;
  if (pair) return int4 ? launch_rows<true, true>(a, plan, st) : launch_rows<false, true>(a, plan, st);
  return int4 ? launch_rows<true, false>(a, plan, st) : launch_rows<false, false>(a, plan, st);
}

}  // namespace b200
