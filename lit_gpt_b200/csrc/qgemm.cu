// Prefill GEMM: y (M, N) = x (M, K) . dequant(W)^T on the 5th-generation tensor cores (tcgen05 + TMEM).  Up to 256 rows most sizes run in qgemm_short.cu, which
// b200_qgemm picks by the times of both (K a multiple of 256, addresses on 16 bytes); this kernel takes the others and every longer prompt.
//
// Replaces, for T > 16 rows, bnb.nn.Linear4bit.forward's "dequantize_4bit of the WHOLE weight to bf16, then F.linear"
// (call sites lit_gpt/model.py:519,619,656,713,714,716): the bf16 weight is never materialised in HBM.
// Persistent over output tiles of up to 256 features x 256 MT tokens, a CTA PAIR each (cta_group::2; up to 128 tokens: one CTA on up to 128 x 128; up to 256 of
// small matrices: one on 128 x 256), walking K in blocks of 64.  Per CTA:
//   * warp 18 fetches packed weights, two k-blocks of the CTA's features at a time, into buffers of their own by TMA, ahead of the stages.  (Read by the
//     dequantising warps themselves, sixteen rows of 32 bytes an access, they took 128 of the 810 shared-memory and L1 cycles of a k-block: nf4, 64 rows
//     x 11008 -> 4096 33 -> 27 us, 4096 -> 12288 at 613 rows 93 -> 88; int4, which has cycles to spare, 1 % longer.)
//   * warps 0-15 rebuild the bf16 values of up to 128 features from the packed 4-bit weights and their absmax / {scale, zero} with exactly the
//     dequantise kernel's arithmetic (bf16_rn(code_fp32 * absmax_fp32), resp. bf16_rn(scale * (q - zero))) and write them into shared memory in
//     the tensor core's K-major 128-byte-swizzled layout.  Even and odd k-blocks belong to eight warps each: a warp has two blocks' time
//     for its look-ups and the proxy fence, and 32 codes a thread to overlap.  (Three groups of eight take the same time to a tenth of a us: what bounds
//     them is throughput.);
//   * warp 16 fetches the activation tiles (128 tokens x 64 k per CTA and sub-tile) by TMA, rows past M zero-filled by the hardware;
//   * warp 17 (of the pair's first CTA) issues tcgen05.mma (kind::f16, bf16 x bf16 -> fp32, 256 x 256 x 16) into TENSOR MEMORY; tcgen05.commit
//     hands each stage back to both CTAs;
//   * across the pair every hand-over has cluster scope.  A dequantising warp of the second CTA announces its rows with 16 bytes of them, a bulk
//     copy to the first CTA whose arrival there is the release (it is started after the writes, so it follows them), and each CTA's warp 16 passes a
//     stage's return on to the dequantising warps.  Those wait on barriers of their own CTA only.  (An arrival with release at cluster scope takes 1400
//     clocks, whichever thread makes it: the SM's weight loads under way hold it up.  4096 -> 11008 at 203 rows, nf4: 49.7 us; with one thread that
//     passes the second CTA's tiles on with such arrivals 69.4, with two in turn 50.8; 14336 -> 4096 at 4096 rows, int4: 366, 437, 360.)
//   * the sixteen warps read the accumulators with tcgen05.ld, add the bias, round to bf16 and store rows of y.
// SWIGLU: the pair's first CTA dequantises 128 rows of the gate projection and the second the same rows of the up projection, so that a
// thread holds both halves of its outputs and stores silu(gate) * up, with the roundings of the separate launches.
// Bound: long prompts by power (1.3 GHz and 80 % tensor pipe at 4096 tokens, 4096 -> 14336, int4: 1106 clk a k-block of 512 tokens, 1024 of them products);
// one sub-tile by the look-ups and stores of a tile's features (606 clk a k-block without, at 256 features int4 about 800 and nf4 950).
#include "qgemm_short.cuh"
#include "tc05.cuh"

namespace b200 {

struct GemmParams {
  const uint8_t* packed;      // reference layout: nf4/fp4 bytes (N, K/2); int4 words (N, K/8)
  const uint32_t* scale;      // fp32 absmax (N, K/64) or half2 {scale, zero} (N, K/128)
  const uint8_t* packed2;     // the up-projection beside the gate (SWIGLU)
  const uint32_t* scale2;
  const __nv_bfloat16* x;     // (M, K)
  const __nv_bfloat16* bias;  // (N) or null
  __nv_bfloat16* y;           // (M, N)
  int64_t M, N, K;
  int qtype;
  int ksplit;                 // > 1 (too few tiles for the SMs): an item owns a range of k-blocks and writes fp32 partial sums
  float* partial;             // (ksplit, M, N) fp32, summed in range order by qgemm_splitk_reduce_kernel
  int n_tiles, m_tiles;
  int bn;                     // features per tile: a multiple of 16 (of 32 for a gate / up pair) up to 128 per CTA
};

constexpr int kGGroups = 2, kGDequantWarps = 8 * kGGroups, kGThreads = (kGDequantWarps + 3) * 32;   // groups of dequantising warps, the activations', the products' and the weights' warp
constexpr int kBK = 64;
constexpr int kTileBytes = 128 * kBK * 2;   // one 128-row x 64-k bf16 operand tile = 16 KB

// byte offset of the 16-byte chunk `c` (0..7) of row `r` inside a 128-row K-major SWIZZLE_128B tile
__device__ __forceinline__ uint32_t sw128(int r, int c) { return (uint32_t)((r >> 3) * 1024 + (r & 7) * 128 + ((c ^ (r & 7)) << 4)); }

template <int CTAS>
__device__ __forceinline__ void umma_bf16(uint32_t d, uint64_t a, uint64_t b, int n, uint32_t accumulate) {
  // D = f32, A = B = bf16, both K-major, M = 128 per CTA of the group
  const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 * CTAS >> 4) << 24);
  if constexpr (CTAS == 2)
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
  else
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}

template <int MT>
struct GemmTile {
  static constexpr int kStages = MT == 2 ? 4 : 6;
  static constexpr int kStage = (MT + 1) * kTileBytes;     // MT activation tiles + 1 weight tile
  // Buffers of packed weights: two k-blocks of 128 features each.  Every warp that gives one back has waited for that very pair, so that its arrival cannot
  // be counted into the phase of the pair before it in the buffer, whatever the numbers of stages and buffers (the stages alone would let one group of warps run
  // five blocks ahead of the other).
  static constexpr int kPairs = 3, kPair = 128 * 64;
  static constexpr int kSmem = kStages * kStage + kPairs * kPair + 1024;
  static_assert(kSmem >= tc::kPairMinSmem, "one CTA of a pair per SM");
};

template <int CTAS, int MT, bool INT4, bool SWIGLU>
__global__ void __launch_bounds__(kGThreads, 1) qgemm_tcgen05_kernel(const GemmParams p, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                     const __grid_constant__ CUtensorMap map_w2, unsigned* err) {
  using C = GemmTile<MT>;
  extern __shared__ __align__(1024) uint8_t g_smem[];
  constexpr int BM = 128 * CTAS, BN = BM;           // tokens per sub-tile; columns of an accumulator
  const int bn = p.bn, half = bn / CTAS, busy = (half + 15) / 16;   // features of a tile, of a CTA; dequantising warps of a group that have some
  __shared__ __align__(8) uint64_t s_bars[3 * C::kStages + 3 + 2 * C::kPairs];
  __shared__ uint32_t s_tmem;
  __shared__ uint4 s_token[CTAS == 2 ? C::kStages : 1][8];   // where the bytes of the other CTA's warps land
  __shared__ float s_code[16 * 32];                 // fp32 code book, one copy per lane (conflict-free look-ups)
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // (known to be the same in all lanes)
  const uint32_t rank = CTAS == 2 ? tc::cluster_rank() : 0u;
  const uint32_t tiles = (tc::smem_u32(g_smem) + 1023u) & ~1023u;
  const uint32_t full = tc::smem_u32(&s_bars[0]), empty = tc::smem_u32(&s_bars[C::kStages]), acc_full = tc::smem_u32(&s_bars[2 * C::kStages]), acc_free = acc_full + 8, idle = acc_full + 16;
  const uint32_t room = CTAS == 2 ? idle + 8 : empty;   // where the dequantising warps learn that a stage is theirs
  const uint32_t packed = tiles + C::kStages * C::kStage, w_full = tc::smem_u32(&s_bars[3 * C::kStages + 3]), w_empty = w_full + 8 * C::kPairs;
  if (tid == 0) {
    for (int s = 0; s < C::kStages; ++s) {
      tc::mbar_init(full + 8 * s, 1 + busy);   // a group of dequantising warps and the copies
      tc::mbar_init(empty + 8 * s, 1);
      if (CTAS == 2) tc::mbar_init(room + 8 * s, 1);
    }
    tc::mbar_init(acc_full, 1);
    tc::mbar_init(acc_free, kGDequantWarps * CTAS);
    tc::mbar_init(idle, 1);
    for (int i = 0; i < C::kPairs; ++i) { tc::mbar_init(w_full + 8 * i, 1); tc::mbar_init(w_empty + 8 * i, kGGroups * busy); }
    tc::mbar_init_fence();
    tc::prefetch_map(&map_x);
    tc::prefetch_map(SWIGLU && rank ? &map_w2 : &map_w);
  }
  if (!INT4)
    for (int i = tid; i < 16 * 32; i += kGThreads) s_code[i] = code_value(p.qtype, i >> 5);
  griddep_launch();
  griddep_wait();
  if (warp == kGDequantWarps + 1) {
    if constexpr (CTAS == 2) tc::tmem_alloc_pair<BN * MT>(tc::smem_u32(&s_tmem));
    else tc::tmem_alloc<BN * MT>(tc::smem_u32(&s_tmem));
  }
  tc::fence_before();
  if constexpr (CTAS == 2) tc::cluster_sync();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = s_tmem;

  const int nkb_all = (int)(p.K / kBK), total = p.n_tiles * p.m_tiles * p.ksplit;
  struct Item { int64_t m0, n0; int z, kb0, nkb, mts; };
  auto item = [&](int i) {
    Item t;
    const int z = i / (p.n_tiles * p.m_tiles), r = i - z * (p.n_tiles * p.m_tiles), m = r / p.n_tiles;
    t.z = z;
    t.m0 = (int64_t)m * (BM * MT);
    t.n0 = (int64_t)(r - m * p.n_tiles) * (SWIGLU ? half : bn);
    t.kb0 = (int)(((int64_t)nkb_all * z) / p.ksplit);
    t.nkb = (int)(((int64_t)nkb_all * (z + 1)) / p.ksplit) - t.kb0;
    t.mts = MT == 1 || p.M - t.m0 <= BM ? 1 : MT;     // sub-tiles with tokens in them
    return t;
  };
  const int first = (int)blockIdx.x / CTAS, step = (int)gridDim.x / CTAS;
  bool ok = true;
  int q = 0;                                          // k-blocks so far: stage q % kStages
  auto wait = [](uint32_t bar, uint32_t parity) {     // on a barrier that the other CTA of a pair arrives on
    return CTAS == 2 ? tc::mbar_wait_cluster(bar, parity) : tc::mbar_wait(bar, parity);
  };

  if (warp < kGDequantWarps) {
    // =========================================== DEQUANTISE, THEN STORE =========================================
    constexpr int LAG = 2;
    const int g = warp >> 3, at = ((warp & 7) - 2 * g) & 7, wr = at * 16 + (lane & 15), wh = lane >> 4;   // group of warps, place in it, feature, half of
    // the k-block (a tile of fewer features leaves the last places idle: two warps on, so that the groups' idle ones belong to different schedulers)
    uint32_t acc_ph = 0;
    int pairs = 0;                                    // buffers of weights so far
    for (int i = first; i < total && ok; i += step) {
      const Item t = item(i);
      const int64_t wn = t.n0 + (SWIGLU ? 0 : (int)rank * half) + wr;   // (rows of a warp past the CTA's features are written and not read)
      const uint32_t* sp = (SWIGLU && rank ? p.scale2 : p.scale) + (wn < p.N ? wn : 0) * (INT4 ? (p.K >> 7) : (p.K >> 6));
      const int l0 = (g + kGGroups - q % kGGroups) % kGGroups;   // this group's first k-block of the item
      uint32_t sn[LAG];
#pragma unroll
      for (int e = 0; e < LAG; ++e) {
        const int l = l0 + kGGroups * e;
        sn[e] = l < t.nkb ? sp[INT4 ? ((t.kb0 + l) >> 1) : (t.kb0 + l)] : 0u;
      }
      for (int l = at < busy ? l0 : t.nkb; l < t.nkb; l += kGGroups) {
        const int s = (q + l) % C::kStages;
        const uint32_t ph = (uint32_t)((q + l) / C::kStages) & 1u;
        const uint32_t sc = sn[0];
#pragma unroll
        for (int e = 0; e + 1 < LAG; ++e) sn[e] = sn[e + 1];
        const int ln = l + kGGroups * LAG;
        if (ln < t.nkb) sn[LAG - 1] = sp[INT4 ? ((t.kb0 + ln) >> 1) : (t.kb0 + ln)];
        const int pair = pairs + (l >> 1), buf = pair % C::kPairs;
        const uint32_t dst = tiles + s * C::kStage + MT * kTileBytes;
        ok = __all_sync(0xffffffffu, tc::mbar_wait(w_full + 8 * buf, (uint32_t)(pair / C::kPairs) & 1u));
        if (!ok) break;
        uint32_t qw[4];
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(qw[0]), "=r"(qw[1]), "=r"(qw[2]), "=r"(qw[3])
                     : "r"(packed + buf * C::kPair + wr * 64 + ((((l & 1) * 2 + wh) ^ ((wr >> 1) & 3)) << 4)));
        ok = __all_sync(0xffffffffu, tc::mbar_wait(room + 8 * s, CTAS == 2 ? ph : ph ^ 1u));
        if (!ok) break;
        if (INT4) {
          // bf16_rn(scale * (q - zero)) with two instructions per code and half a conversion: two nibbles at a time are moved to the top four mantissa
          // bits of halves of 16.0 (SHF + LOP3: f = 16 + q exactly, five significant bits), then ONE mixed FMA each, scale * f - scale * (16 + zero) with the
          // fp16 factors as they are: both products are exact in fp32 (11-bit fp16 scale x 6-bit integer), so the result is the exact scale * (q - zero).
          // (8192 codes by sixteen warps, stores included: 288 clk; with every code brought to fp32 of its own 387.)
          const __half2 h2 = *reinterpret_cast<const __half2*>(&sc);
          const float c0 = -__low2float(h2) * (16.0f + __high2float(h2));
          const uint16_t hs = (uint16_t)(sc & 0xffffu);
#pragma unroll
          for (int j = 0; j < 4; ++j) {  // word j = k [32 wh + 8j, +8), element e in bits 4e
            float f[8];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const uint32_t sh = e < 2 ? qw[j] << (6 - 4 * e) : qw[j] >> (4 * e - 6);
              asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %2;\n\tfma.rn.f32.f16 %0, l, %3, %4;\n\tfma.rn.f32.f16 %1, h, %3, %4;\n\t}"
                  : "=f"(f[e]), "=f"(f[e + 4]) : "r"((sh & 0x03c003c0u) | 0x4c004c00u), "h"(hs), "f"(c0));
            }
            uint32_t o[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) o[e] = pack_bf16(f[2 * e], f[2 * e + 1]);
            asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(dst + sw128(wr, wh * 4 + j)), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]) : "memory");
          }
        } else {
          // bf16_rn(code_fp32 * absmax_fp32): look-up offset = nibble << 7 | lane << 2 from the table's (link-time constant) address:
          // SHF + LOP3 + LDS per code
          const float am = __uint_as_float(sc);
          const uint32_t lane4 = (uint32_t)lane * 4u;
          auto deq = [&](uint32_t v, int bit) -> float {   // the nibble at bits bit .. bit + 3 of word v
            const uint32_t sh = bit <= 7 ? v << (7 - bit) : v >> (bit - 7);
            return *reinterpret_cast<const float*>(reinterpret_cast<const char*>(s_code) + ((sh & 0x780u) | lane4)) * am;
          };
#pragma unroll
          for (int j = 0; j < 4; ++j) {  // word j = bytes 4j..4j+3 = k [32 wh + 8j, +8); even element in the HIGH nibble
            uint32_t o[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) o[e] = pack_bf16(deq(qw[j], 8 * e + 4), deq(qw[j], 8 * e));
            asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(dst + sw128(wr, wh * 4 + j)), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]) : "memory");
          }
        }
        tc::fence_smem_async();                       // generic-proxy writes -> visible to the tensor core
        __syncwarp();
        if (lane == 0) {
          tc::mbar_arrive(w_empty + 8 * buf);
          if (CTAS == 2 && rank == 1) tc::copy_to_cta(tc::at_rank(tc::smem_u32(&s_token[s][warp & 7]), 0), dst + sw128(wr, wh * 4), 16, tc::at_rank(full + 8 * s, 0));
          else tc::mbar_arrive(full + 8 * s);
        }
      }
      if ((t.nkb & 1) && l0 == 1 && at < busy && ok) {   // the last pair's second block, which does not exist: its buffer is given back like any other, once it has been filled
        const int pair = pairs + (t.nkb >> 1), buf = pair % C::kPairs;
        ok = __all_sync(0xffffffffu, tc::mbar_wait(w_full + 8 * buf, (uint32_t)(pair / C::kPairs) & 1u));
        if (ok && lane == 0) tc::mbar_arrive(w_empty + 8 * buf);
      }
      pairs += (t.nkb + 1) >> 1;
      q += t.nkb;
      // ---- accumulators -> y (or partial sums): warp w has rows 32 (w % 4) .. + 31 and a quarter of the columns ----
      ok = ok && __all_sync(0xffffffffu, wait(acc_full, acc_ph));
      acc_ph ^= 1u;
      if (!ok) break;
      tc::fence_after();
#pragma unroll 1
      for (int mt = 0; mt < t.mts; ++mt) {
        const int64_t m = t.m0 + mt * BM + rank * 128 + (warp & 3) * 32 + lane;        // this thread's output row (TMEM lane = row)
        const uint32_t acc = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(mt * BN);
        if constexpr (SWIGLU) {   // the first half of the columns is the gate, the other the up projection of the same features
#pragma unroll 1
          for (int c0 = (warp >> 2) * 16; c0 < half; c0 += kGDequantWarps * 4) {
            uint32_t v[16], u[16];
            tc::ld16(v, acc + c0);
            tc::ld16(u, acc + c0 + half);
            tc::wait_ld(v);
            tc::wait_ld(u);
            if (m < p.M) {
#pragma unroll
              for (int j = 0; j < 16; j += 8) {
                const int64_t n = t.n0 + c0 + j;
                if (n < p.N) {
                  uint32_t o[4];
#pragma unroll
                  for (int e = 0; e < 4; ++e) {
                    auto act = [](uint32_t g, uint32_t w) {
                      const float a = round_bf16(__uint_as_float(g));
                      return round_bf16(a / (1.0f + expf(-a))) * round_bf16(__uint_as_float(w));
                    };
                    o[e] = pack_bf16(act(v[j + 2 * e], u[j + 2 * e]), act(v[j + 2 * e + 1], u[j + 2 * e + 1]));
                  }
                  *reinterpret_cast<uint4*>(p.y + m * p.N + n) = make_uint4(o[0], o[1], o[2], o[3]);
                }
              }
            }
            __syncwarp();   // (the next loads of tensor memory want the whole warp, lanes without a row too)
          }
          continue;
        }
#pragma unroll 1
        for (int c0 = (warp >> 2) * 16; c0 < bn; c0 += kGDequantWarps * 4) {
          uint32_t v[16];
          tc::ld16(v, acc + c0);
          tc::wait_ld(v);
          if (m < p.M && p.ksplit > 1) {
            float* dst = p.partial + ((int64_t)t.z * p.M + m) * p.N;   // raw fp32 sums of this k range; bias and rounding in the reduce kernel
#pragma unroll
            for (int j = 0; j < 16; j += 4) {
              const int64_t n = t.n0 + c0 + j;
              if (n < p.N) *reinterpret_cast<uint4*>(dst + n) = make_uint4(v[j], v[j + 1], v[j + 2], v[j + 3]);
            }
          } else if (m < p.M) {
#pragma unroll
            for (int j = 0; j < 16; j += 8) {
              const int64_t n = t.n0 + c0 + j;
              if (n < p.N) {  // N % 8 == 0 (host check): a chunk is either fully inside or fully outside
                uint32_t o[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  float a = __uint_as_float(v[j + 2 * e]), b = __uint_as_float(v[j + 2 * e + 1]);
                  if (p.bias) { a += __bfloat162float(p.bias[n + 2 * e]); b += __bfloat162float(p.bias[n + 2 * e + 1]); }
                  o[e] = pack_bf16(a, b);
                }
                *reinterpret_cast<uint4*>(p.y + m * p.N + n) = make_uint4(o[0], o[1], o[2], o[3]);
              }
            }
          }
          __syncwarp();
        }
      }
      tc::fence_before();
      __syncwarp();
      if (lane == 0) {
        if constexpr (CTAS == 2) tc::mbar_arrive_at(tc::at_rank(acc_free, 0));
        else tc::mbar_arrive(acc_free);
      }
    }
  } else if (warp == kGDequantWarps) {
    // =========================================== ACTIVATIONS ====================================================
    if (tc::elect()) {
      for (int i = first; i < total && ok; i += step) {
        const Item t = item(i);
        for (int l = 0; l < t.nkb; ++l, ++q) {
          const int s = q % C::kStages;
          ok = wait(empty + 8 * s, ((uint32_t)(q / C::kStages) & 1u) ^ 1u);
          if (!ok) break;
          if (CTAS == 2) tc::mbar_arrive(room + 8 * s);
          if (rank == 0) tc::mbar_expect_tx(full + 8 * s, CTAS * t.mts * kTileBytes + (CTAS - 1) * busy * 16);
          const uint32_t st = tiles + s * C::kStage, bar = CTAS == 2 ? tc::at_rank(full + 8 * s, 0) : full + 8 * s;
          for (int mt = 0; mt < t.mts; ++mt) {
            const int row = (int)(t.m0 + mt * BM + rank * 128), col = (t.kb0 + l) * kBK;
            if constexpr (CTAS == 2) tc::tma_load_2d_pair(st + mt * kTileBytes, &map_x, col, row, bar);
            else tc::tma_load_2d(st + mt * kTileBytes, &map_x, col, row, bar);
          }
        }
      }
      if (rank == 0)
        for (int i = 0; i < C::kStages; ++i)   // (a stage never used: the phase before the first)
          ok = wait(full + 8 * i, (uint32_t)((q + C::kStages - 1 - i) / C::kStages + 1) & 1u) && ok;
    }
  } else if (warp == kGDequantWarps + 2) {
    // =========================================== PACKED WEIGHTS =================================================
    if (tc::elect()) {   // ahead of the stages by as many k-blocks as the buffers hold
      int pair = 0;
      for (int i = first; i < total && ok; i += step) {
        const Item t = item(i);
        const int row = (int)(t.n0 + (SWIGLU ? 0 : (int)rank * half));
        for (int l = 0; l < t.nkb; l += 2, ++pair) {
          const int buf = pair % C::kPairs;
          ok = tc::mbar_wait(w_empty + 8 * buf, ((uint32_t)(pair / C::kPairs) & 1u) ^ 1u);
          if (!ok) break;
          tc::mbar_expect_tx(w_full + 8 * buf, (uint32_t)half * 64u);
          tc::tma_load_2d(packed + buf * C::kPair, SWIGLU && rank ? &map_w2 : &map_w, (t.kb0 + l) * 32, row, w_full + 8 * buf);
        }
      }
      for (int i = 0; i < C::kPairs; ++i)   // (a buffer never used: the phase before the first)
        ok = tc::mbar_wait(w_full + 8 * i, (uint32_t)((pair + C::kPairs - 1 - i) / C::kPairs + 1) & 1u) && ok;
    }
  } else if (rank == 0 && tc::elect()) {
    // =========================================== PRODUCTS =======================================================
    auto wait_here = [](uint32_t bar, uint32_t parity) { return CTAS == 2 ? tc::mbar_wait_cluster_here(bar, parity) : tc::mbar_wait_here(bar, parity); };
    uint32_t free_ph = 1, ph = 0;
    int s = 0;
    for (int i = first; i < total && ok; i += step) {
      const Item t = item(i);
      ok = wait_here(acc_free, free_ph);
      free_ph ^= 1u;
      for (int l = 0; l < t.nkb && ok; ++l) {
        ok = wait_here(full + 8 * s, ph);
        if (!ok) break;
        tc::fence_after();
        const uint32_t st = tc::desc_sw128_low(tiles + s * C::kStage), db = st + MT * (kTileBytes >> 4);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          if (mt > 0 && t.mts == 1) break;
#pragma unroll
          for (int k = 0; k < kBK / 16; ++k)  // +32 B along K inside the swizzle atom = +2 in the address field
            umma_bf16<CTAS>(tmem + mt * BN, tc::desc_of(st + mt * (kTileBytes >> 4) + 2 * k, tc::kDescSw128High), tc::desc_of(db + 2 * k, tc::kDescSw128High), bn, (l | k) != 0);
        }
        if constexpr (CTAS == 2) tc::commit_pair(empty + 8 * s);   // the stage is free once these products have read it
        else tc::commit(empty + 8 * s);
        if (++s == C::kStages) { s = 0; ph ^= 1u; }
      }
      if (ok) {
        if constexpr (CTAS == 2) tc::commit_pair(acc_full);
        else tc::commit(acc_full);
      }
    }
    if (!ok) {
      if constexpr (CTAS == 2) tc::commit_pair(idle);
      else tc::commit(idle);
      tc::mbar_wait(idle, 0);
    }
  }
  if (!ok) *err = 1u;
  tc::fence_before();
  if constexpr (CTAS == 2) tc::cluster_sync();   // the other CTA's shared memory is read until its last product
  __syncthreads();
  if (warp == kGDequantWarps + 1) {
    __syncwarp();
    if constexpr (CTAS == 2) tc::tmem_free_pair<BN * MT>(tmem);
    else tc::tmem_free<BN * MT>(tmem);
  }
}

// y = bf16(sum over the k ranges, in range order, + bias): eight outputs per thread (N % 8 == 0)
__global__ void __launch_bounds__(256) qgemm_splitk_reduce_kernel(const float* __restrict__ partial, const __nv_bfloat16* __restrict__ bias,
                                                                  __nv_bfloat16* __restrict__ y, int64_t MN, int64_t N, int ksplit) {
  griddep_launch();
  griddep_wait();
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (i >= MN) return;
  float acc[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) acc[e] = 0.f;
  for (int z = 0; z < ksplit; ++z) {
    const float4 a = *reinterpret_cast<const float4*>(partial + (int64_t)z * MN + i);
    const float4 b = *reinterpret_cast<const float4*>(partial + (int64_t)z * MN + i + 4);
    acc[0] += a.x; acc[1] += a.y; acc[2] += a.z; acc[3] += a.w; acc[4] += b.x; acc[5] += b.y; acc[6] += b.z; acc[7] += b.w;
  }
  const int64_t n = i % N;
  uint32_t o[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    float a = acc[2 * e], b = acc[2 * e + 1];
    if (bias) { a += __bfloat162float(bias[n + 2 * e]); b += __bfloat162float(bias[n + 2 * e + 1]); }
    o[e] = pack_bf16(a, b);
  }
  *reinterpret_cast<uint4*>(y + i) = make_uint4(o[0], o[1], o[2], o[3]);
}

static std::atomic<int> g_gemm_wide{1};   // development switch (b200_qgemm_tune): 0 keeps to one sub-tile of 256 tokens

struct GemmPlan {
  int ctas, mt, ksplit, bn;
};

// Tile and k ranges by the time of the last SM to finish, us.  A k-block takes `block + feature * bn` -- products and hand-overs, and the look-ups or
// conversions of a tile's features, which its tokens share -- a launch `start`, a further round of tiles `round` more, k ranges 0.88 and 2.3 for every
// million partial sums.  Fitted to some 700 launches of one to three rounds (24 shapes of 64 to 2000 rows, every tile and count of ranges: 4 % rms) from before an
// elected thread issued the products.  Against every tile and count of ranges timed since at 257 to 3000 rows (8 shapes, 160 sizes and types) the choice is 1.2 % off the best on
// average and more than 5 % in 17: int4 5120 -> 5120 at 257 rows 29 %, 5120 -> 15360 at 613 17 %, 4096 -> 4096 at 257 14 %; nf4 4096 -> 4096 at 512 13 %.
// Fewer features than 128 per CTA pay where they fill SMs that would have idled: 4096 -> 11008, nf4 / int4, at 64 rows 86 CTAs of 128 features and 138 of 80 39.0
// and 30.8 / 30.6 and 25.6; at 203 rows 43 pairs of 256 and 69 of 160 46.2 and 38.0 / 36.7 and 31.6.
// k ranges are for launches that leave SMs idle all the same: at least four k-blocks per range, at most 16 ranges and 64 MB of partial sums, and no more
// than fill the SMs once.
struct GemmCost {
  double start, block, feature, round;
};
static const GemmCost& gemm_cost(bool int4, int ctas, int mt) {
  static const GemmCost cost[2][2][2] = {{{{4.7, 0.207, 0.00239, 1.6}, {5.9, 0.425, 0.00182, 2.9}}, {{7.3, 0.211, 0.00150, 2.8}, {8.7, 0.410, 0.00125, 1.2}}},
                                         {{{5.5, 0.210, 0.00148, 2.2}, {5.6, 0.425, 0.00179, 2.9}}, {{7.4, 0.237, 0.00083, 3.1}, {8.5, 0.416, 0.00113, 0.9}}}};
  return cost[int4][ctas - 1][mt - 1];
}
// `per_tile`: features of the output that a tile of bn covers
static double gemm_time(int64_t M, int64_t N, int64_t K, bool int4, const GemmPlan& g, int per_tile) {
  const GemmCost& c = gemm_cost(int4, g.ctas, g.mt);
  const int64_t nkb = K / kBK, units = sm_count() / g.ctas, rows = 128 * g.ctas * g.mt;
  const int64_t tiles = ((N + per_tile - 1) / per_tile) * ((M + rows - 1) / rows), rounds = (tiles * g.ksplit + units - 1) / units;
  return c.start + (double)rounds * (double)((nkb + g.ksplit - 1) / g.ksplit) * (c.block + c.feature * g.bn) + c.round * (double)(rounds - 1) +
         (g.ksplit > 1 ? 0.88 + 2.3e-6 * (double)g.ksplit * (double)M * (double)N : 0.0);
}

// (0.1 to 0.3 us on the host)
static GemmPlan gemm_plan(int64_t M, int64_t N, int64_t K, bool int4, bool split_ok) {
  const int nkb = (int)(K / kBK);
  GemmPlan best{1, 1, 1, 128};
  double best_t = -1.0;
  for (int kind = 0; kind < 4; ++kind) {
    const int ctas = kind < 2 ? 1 : 2, mt = kind & 1 ? 2 : 1;
    if (kind == 0 ? M > 128 : M <= 128) continue;            // a second half would be padding; a CTA alone on 128 tokens would dequantise twice
    if (kind == 1 && M > 256) continue;
    if (kind == 3 && (M <= 256 || !g_gemm_wide.load())) continue;
    const int64_t units = sm_count() / ctas, row_tiles = (M + 128 * ctas * mt - 1) / (128 * ctas * mt);
    for (int bn = 128 * ctas; bn >= (ctas == 2 ? 160 : 64); bn -= 16 * ctas) {   // (smaller pairs won nothing over k ranges)
      const int64_t tiles = ((N + bn - 1) / bn) * row_tiles;
      int64_t most = split_ok ? units / tiles : 1;
      if (most > nkb / 4) most = nkb / 4;
      if (most > 16) most = 16;
      while (most > 1 && most * M * N * (int64_t)sizeof(float) > (64ll << 20)) --most;
      for (int64_t s = 1; s <= (most < 1 ? 1 : most); ++s) {
        const GemmPlan g{ctas, mt, (int)s, bn};
        const double t = gemm_time(M, N, K, int4, g, bn);
        if (best_t < 0.0 || t < best_t) { best_t = t; best = g; }
      }
    }
  }
  return best;
}

// What gemm_time is off by at up to 256 rows since its products are issued by an elected thread (measured over the sizes that short_time was fitted to)
static double short_margin(bool int4, const GemmPlan& g) {
  const double off = !int4 ? (g.mt == 2 ? 0.92 : 1.0) : g.ctas == 2 ? 0.96 : g.mt == 2 ? 0.87 : g.ksplit > 1 ? 0.97 : 0.88;
  return off * 0.97;
}

template <int CTAS, int MT, bool INT4, bool SWIGLU = false>
static cudaError_t launch_gemm(GemmParams p, cudaStream_t st) {
  constexpr int smem = GemmTile<MT>::kSmem;
  static PerDeviceOnce once;
  if (once.need()) {
    cudaError_t e = cudaFuncSetAttribute(qgemm_tcgen05_kernel<CTAS, MT, INT4, SWIGLU>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    once.done();
  }
  alignas(64) CUtensorMap map;
  alignas(64) CUtensorMap weights, weights2;
  const int half = p.bn / CTAS;
  if (!tensor_map_2d(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, p.x, p.M, p.K, p.K * 2, 128) ||
      !tensor_map_2d(&weights, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, p.packed, p.N, p.K / 2, p.K / 2, half, 64) ||
      !tensor_map_2d(&weights2, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, SWIGLU ? p.packed2 : p.packed, p.N, p.K / 2, p.K / 2, half, 64))
    return cudaErrorInvalidValue;
  unsigned* const err = wait_error_word();
  if (!err) return cudaErrorMemoryAllocation;
  const int features = SWIGLU ? p.bn / 2 : p.bn;
  p.n_tiles = (int)((p.N + features - 1) / features);
  p.m_tiles = (int)((p.M + 128 * CTAS * MT - 1) / (128 * CTAS * MT));
  const int64_t items = (int64_t)p.n_tiles * p.m_tiles * p.ksplit, units = sm_count() / CTAS;
  const cudaError_t e = launch_cluster(qgemm_tcgen05_kernel<CTAS, MT, INT4, SWIGLU>, dim3((unsigned)((items < units ? items : units) * CTAS)), dim3(kGThreads), CTAS,
                                       (size_t)smem, st, p, map, weights, weights2, err);
  if (e != cudaSuccess || p.ksplit == 1) return e;
  const int64_t MN = p.M * p.N;
  return launch(qgemm_splitk_reduce_kernel, dim3((unsigned)((MN / 8 + 255) / 256)), dim3(256), (size_t)0, st, (const float*)p.partial, p.bias, p.y, MN, p.N, p.ksplit);
}

template <bool INT4>
static cudaError_t launch_plan(const GemmParams& p, const GemmPlan& g, cudaStream_t st) {
  if (g.ctas == 1) return g.mt == 2 ? launch_gemm<1, 2, INT4>(p, st) : launch_gemm<1, 1, INT4>(p, st);
  return g.mt == 2 ? launch_gemm<2, 2, INT4>(p, st) : launch_gemm<2, 1, INT4>(p, st);
}

// Tile of a gate / up pair in one launch (from 129 rows)
static GemmPlan swiglu_tile(int64_t M, int64_t N, int64_t K, bool int4) {
  GemmPlan best{2, 0, 1, 256};
  double best_t = -1.0;
  for (int mt = 1; mt <= (M > 256 && g_gemm_wide.load() ? 2 : 1); ++mt)
    for (int bn = 256; bn >= 128; bn -= 32) {
      const GemmPlan g{2, mt, 1, bn};
      const double t = gemm_time(M, N, K, int4, g, bn / 2);
      if (best_t < 0.0 || t < best_t) { best_t = t; best = g; }
    }
  return best;
}

// The same, no sub-tiles (mt 0) where b200_qgemm_swiglu refuses.  us, two launches and the product, each
// with its best tile, against one, nf4 / int4: 4096 -> 11008 at 203 rows 83 -> 76 / 70 -> 65, at 400 115 -> 95 / 116 -> 101, at 1000 223 -> 158 / 228 -> 171;
// 5120 -> 13824 at 300 131 -> 124 / 134 -> 133, at 2000 470 -> 435 / 462 -> 438; 4096 -> 14336 at 4096 859 -> 769 / 883 -> 776.  Up to 512 rows the two ways' times
// as modelled decide.  Beyond, an older line stands, which counts rounds of full tiles in clocks of an older kernel (1500 and 1130 a k-block).  One launch is shorter
// where it refuses too, in all of 104 shapes and types measured, and b200_qgemm_pair takes those: 4096 -> 11008 at 513 rows 180 / 137 (nf4), 139 / 118 (int4),
// at 2400 378 / 336; 4096 -> 14336 at 1024 219 / 201, 205 / 185; 5120 -> 13824 at 2000 446 / 412, 433 / 408.
static GemmPlan swiglu_plan(int64_t M, int64_t N, int64_t K, bool int4) {
  const GemmPlan none{2, 0, 1, 256};
  if (M <= 128) return none;
  const int64_t units = sm_count() / 2, n = (N + 127) / 128, nkb = K / kBK;
  const GemmPlan best = swiglu_tile(M, N, K, int4);
  const double best_t = gemm_time(M, N, K, int4, best, best.bn / 2);
  if (M <= 512) {
    const GemmPlan one = gemm_plan(M, N, K, int4, true);
    const double apart = 2.0 * gemm_time(M, N, K, int4, one, one.bn) - gemm_cost(int4, one.ctas, one.mt).start + 4.0 + 1e-6 * (double)M * (double)N;   // (and the product)
    return best_t < apart ? best : none;
  }
  auto rounds = [&](int64_t feature_tiles, int mt) { return (feature_tiles * ((M + 256 * mt - 1) / (256 * mt)) + units - 1) / units * (nkb * (mt == 2 ? 1500 : 1130) + 6000); };
  const int64_t one2 = rounds((N + 255) / 256, 2) - ((M - 1) % 512 < 256 ? 370 * nkb : 0), one1 = rounds((N + 255) / 256, 1);   // clocks
  const int64_t pair1 = rounds(n, 1), pair2 = g_gemm_wide.load() ? rounds(n, 2) : pair1;
  const int64_t worth = (2 * (one1 < one2 || !g_gemm_wide.load() ? one1 : one2) + 2000 + M * N / 1100) / 20 * 19;
  return (pair1 < pair2 ? pair1 : pair2) < worth ? best : none;
}

// Gate, up projection and product of 129 to 256 rows by the kernels of this file, as modelled.  us, in one launch here / in one of qgemm_short.cu, 4096 -> 14336 at 129 / 203 rows
// nf4 80 / 50, 80 / 66, int4 63 / 52, 63 / 65; 4096 -> 6144 39 / 36, 39 / 44, 31 / 34, 31 / 42; 2048 -> 5632 23 / 26, 23 / 32, 19 / 26, 19 / 32.
static double swiglu_time(int64_t M, int64_t N, int64_t K, bool int4) {
  const GemmPlan one = gemm_plan(M, N, K, int4, true);
  double best = 2.0 * gemm_time(M, N, K, int4, one, one.bn) - gemm_cost(int4, one.ctas, one.mt).start + 4.0 + 1e-6 * (double)M * (double)N;
  for (int bn = 256; bn >= 128; bn -= 32) {
    const double t = gemm_time(M, N, K, int4, GemmPlan{2, 1, 1, bn}, bn / 2);
    if (t < best) best = t;
  }
  return best * (int4 ? 0.93 : 0.97);   // (int4: what the model is off by since an elected thread issues the products; and something has to be won)
}

}  // namespace b200

using namespace b200;

extern "C" {

int b200_qgemm_tune(int wide) { g_gemm_wide = wide ? 1 : 0; return B200_OK; }

size_t b200_qgemm_workspace_bytes(int64_t M, int64_t N, int64_t K) {
  // accumulators live in tensor memory; only a launch split over k ranges (short prompts: too few output tiles for the SMs) stages fp32 partial sums
  if (M <= 0 || N <= 0 || K < kBK) return 0;
  const int nf4 = gemm_plan(M, N, K, false, true).ksplit, int4 = gemm_plan(M, N, K, true, true).ksplit, s = nf4 > int4 ? nf4 : int4;   // either type's
  const size_t ranges = s > 1 ? (size_t)s * (size_t)M * (size_t)N * sizeof(float) : 0;
  const size_t a = short_scratch_bytes(M, N, short_plan(M, N, K, B200_Q_NF4, false, true), false), b = short_scratch_bytes(M, N, short_plan(M, N, K, B200_Q_INT4, false, true), false);
  return ranges > a ? (ranges > b ? ranges : b) : (a > b ? a : b);
}

static int gemm_args(const b200_qgemm_args* a, GemmParams& p) {
  B200_CHECK_WAITS("b200_qgemm");
  B200_CHECK_ARG(a != nullptr, "b200_qgemm: null args");
  B200_CHECK_ARG(a->packed && a->scale && a->x && a->y, "b200_qgemm: null packed/scale/x/y pointer");
  B200_CHECK_ARG(a->M > 0 && a->N > 0 && a->K > 0, "b200_qgemm: M, N, K must be positive");
  B200_CHECK_ARG(a->qtype == B200_Q_NF4 || a->qtype == B200_Q_FP4 || a->qtype == B200_Q_INT4, "b200_qgemm: bad qtype %d", a->qtype);
  const bool int4 = a->qtype == B200_Q_INT4;
  if (a->blocksize != (int4 ? 128 : 64) || a->K % (int4 ? 128 : 64) != 0 || a->N % 8 != 0) {
    set_error("b200_qgemm: needs blocksize %d, K %% %d == 0 and N %% 8 == 0 (blocksize=%d N=%lld K=%lld)", int4 ? 128 : 64, int4 ? 128 : 64,
              a->blocksize, (long long)a->N, (long long)a->K);
    return B200_ERR_UNSUPPORTED;
  }
  B200_CHECK_ARG(a->N <= 65535LL * 128 && a->M <= 65535LL * 128, "b200_qgemm: shape too large for the grid");
  B200_CHECK_ARG(((reinterpret_cast<uintptr_t>(a->packed) | reinterpret_cast<uintptr_t>(a->x) | reinterpret_cast<uintptr_t>(a->y)) & 15) == 0,
                 "b200_qgemm: packed / x / y must be 16-byte aligned");
  p.packed = reinterpret_cast<const uint8_t*>(a->packed);
  p.scale = reinterpret_cast<const uint32_t*>(a->scale);
  p.x = reinterpret_cast<const __nv_bfloat16*>(a->x);
  p.bias = reinterpret_cast<const __nv_bfloat16*>(a->bias);
  p.y = reinterpret_cast<__nv_bfloat16*>(a->y);
  p.M = a->M; p.N = a->N; p.K = a->K; p.qtype = a->qtype;
  return B200_OK;
}

int b200_qgemm(const b200_qgemm_args* a, b200_stream_t stream) {
  GemmParams p{};
  if (const int rc = gemm_args(a, p)) return rc;
  // k ranges only when the caller provided the workspace b200_qgemm_workspace_bytes asks for (none: one k range)
  const bool int4 = a->qtype == B200_Q_INT4;
  GemmPlan g = gemm_plan(a->M, a->N, a->K, int4, true);
  if (g.ksplit > 1 && (a->workspace == nullptr || a->workspace_bytes < (size_t)g.ksplit * a->M * a->N * sizeof(float) ||
                       (reinterpret_cast<uintptr_t>(a->workspace) & 15)))
    g = gemm_plan(a->M, a->N, a->K, int4, false);
  // Up to 256 rows the kernel with the weights on the left is the shorter way but for some matrices of 2560 x 7680 and less and int4 from 200 rows: us, this one / that
  // one, 4096 -> 14336 at 17 / 64 / 129 / 203 rows nf4 35 / 21, 36 / 23, 42 / 27, 42 / 32, int4 26 / 21, 27 / 23, 34 / 27, 34 / 31; 14336 -> 4096 nf4 36 / 22,
  // 37 / 25, 47 / 31, 47 / 35; 2048 -> 5632 int4 at 128 rows 13.4 / 15.3.  Each has a model of its times.
  const ShortArgs sa{{p.packed, nullptr}, {p.scale, nullptr}, p.x, p.bias, p.y, reinterpret_cast<float*>(a->workspace), p.M, p.N, p.K, p.qtype};
  if (short_takes(sa, false)) {
    ShortPlan s = short_plan(p.M, p.N, p.K, p.qtype, false, true);
    if (s.shared && (a->workspace == nullptr || a->workspace_bytes < short_scratch_bytes(p.M, p.N, s, false) || (reinterpret_cast<uintptr_t>(a->workspace) & 15)))
      s = short_plan(p.M, p.N, p.K, p.qtype, false, false);
    if (s.ctas && s.time < gemm_time(p.M, p.N, p.K, int4, g, g.bn) * short_margin(int4, g)) {
      const cudaError_t e = launch_short(sa, s, false, (cudaStream_t)stream);
      if (e != cudaSuccess) {
        set_error("b200_qgemm: launch failed: %s", cudaGetErrorString(e));
        return B200_ERR_CUDA;
      }
      return B200_OK;
    }
  }
  p.ksplit = g.ksplit;
  p.bn = g.bn;
  p.partial = reinterpret_cast<float*>(a->workspace);
  const cudaError_t e = int4 ? launch_plan<true>(p, g, (cudaStream_t)stream) : launch_plan<false>(p, g, (cudaStream_t)stream);
  if (e != cudaSuccess) {
    set_error("b200_qgemm: launch failed: %s", cudaGetErrorString(e));
    return B200_ERR_CUDA;
  }
  return B200_OK;
}

static int launch_swiglu(const b200_qgemm_args* a, GemmParams p, const GemmPlan& g, const void* packed2, const void* scale2, b200_stream_t stream, const char* what) {
  p.packed2 = reinterpret_cast<const uint8_t*>(packed2);
  p.scale2 = reinterpret_cast<const uint32_t*>(scale2);
  p.ksplit = 1;
  p.bn = g.bn;
  const cudaStream_t st = (cudaStream_t)stream;
  const bool int4 = a->qtype == B200_Q_INT4;
  const cudaError_t e = g.mt == 2 ? (int4 ? launch_gemm<2, 2, true, true>(p, st) : launch_gemm<2, 2, false, true>(p, st))
                                : (int4 ? launch_gemm<2, 1, true, true>(p, st) : launch_gemm<2, 1, false, true>(p, st));
  if (e != cudaSuccess) {
    set_error("%s: launch failed: %s", what, cudaGetErrorString(e));
    return B200_ERR_CUDA;
  }
  return B200_OK;
}

int64_t b200_qgemm_pair_workspace(int64_t M, int64_t N, int64_t K, int qtype, int blocksize) {
  const int block = qtype == B200_Q_INT4 ? 128 : 64;
  if ((qtype != B200_Q_NF4 && qtype != B200_Q_FP4 && qtype != B200_Q_INT4) || blocksize != block || M <= 0 || N <= 0 || K <= 0) return -1;
  if (M > 512) return K % block == 0 && N % 8 == 0 && N <= 65535LL * 128 && M <= 65535LL * 128 && swiglu_plan(M, N, K, qtype == B200_Q_INT4).mt == 0 ? 0 : -1;
  const ShortPlan s = short_plan(M, N, K, qtype, true, true);
  // (up to 128 rows there is no other launch for both; from 129 it is b200_qgemm_swiglu's or two)
  if (s.ctas == 0 || (M > 128 && s.time >= swiglu_time(M, N, K, qtype == B200_Q_INT4))) return -1;
  return (int64_t)short_scratch_bytes(M, N, s, true);
}

int b200_qgemm_pair(const b200_qgemm_args* a, const void* packed2, const void* scale2, b200_stream_t stream) {
  GemmParams p{};
  if (const int rc = gemm_args(a, p)) return rc;
  B200_CHECK_ARG(packed2 && scale2 && (reinterpret_cast<uintptr_t>(packed2) & 15) == 0, "b200_qgemm_pair: null or misaligned second matrix");
  B200_CHECK_ARG(!a->bias, "b200_qgemm_pair: takes no bias");
  if (p.M > 512 && b200_qgemm_pair_workspace(p.M, p.N, p.K, p.qtype, a->blocksize) >= 0)
    return launch_swiglu(a, p, swiglu_tile(p.M, p.N, p.K, p.qtype == B200_Q_INT4), packed2, scale2, stream, "b200_qgemm_pair");
  ShortArgs sa{{p.packed, reinterpret_cast<const uint8_t*>(packed2)}, {p.scale, reinterpret_cast<const uint32_t*>(scale2)}, p.x, nullptr, p.y,
               reinterpret_cast<float*>(a->workspace), p.M, p.N, p.K, p.qtype};
  ShortPlan s = short_plan(p.M, p.N, p.K, p.qtype, true, true);
  if (s.shared && (a->workspace == nullptr || a->workspace_bytes < short_scratch_bytes(p.M, p.N, s, true) || (reinterpret_cast<uintptr_t>(a->workspace) & 15)))
    s = short_plan(p.M, p.N, p.K, p.qtype, true, false);
  if (s.ctas == 0 || !short_takes(sa, true) || b200_qgemm_pair_workspace(p.M, p.N, p.K, p.qtype, a->blocksize) < 0) {
    set_error("b200_qgemm_pair: (M=%lld N=%lld K=%lld) or its addresses run as two b200_qgemm and b200_swiglu", (long long)a->M, (long long)a->N, (long long)a->K);
    return B200_ERR_UNSUPPORTED;
  }
  const cudaError_t e = launch_short(sa, s, true, (cudaStream_t)stream);
  if (e != cudaSuccess) {
    set_error("b200_qgemm_pair: launch failed: %s", cudaGetErrorString(e));
    return B200_ERR_CUDA;
  }
  return B200_OK;
}

int64_t b200_qgemm_short_workspace(int64_t M, int64_t N, int64_t K, int pair, int ranges) {
  if (M < 1 || N < 1 || K < 256) return -1;
  return (int64_t)short_scratch_bytes(M, N, short_shape(N, K, ranges != 0), pair != 0);
}

int b200_qgemm_short(const b200_qgemm_args* a, const void* packed2, const void* scale2, int ranges, b200_stream_t stream) {
  GemmParams p{};
  if (const int rc = gemm_args(a, p)) return rc;
  const bool pair = packed2 != nullptr;
  B200_CHECK_ARG(!pair || (scale2 && !a->bias), "b200_qgemm_short: a pair takes scale2 and no bias");
  const ShortArgs sa{{p.packed, reinterpret_cast<const uint8_t*>(packed2)}, {p.scale, reinterpret_cast<const uint32_t*>(scale2)}, p.x, p.bias, p.y,
                     reinterpret_cast<float*>(a->workspace), p.M, p.N, p.K, p.qtype};
  if (!short_takes(sa, pair)) {
    set_error("b200_qgemm_short: (M=%lld N=%lld K=%lld) or its addresses are not the kernel's", (long long)a->M, (long long)a->N, (long long)a->K);
    return B200_ERR_UNSUPPORTED;
  }
  const ShortPlan s = short_shape(p.N, p.K, ranges != 0);
  B200_CHECK_ARG(!s.shared || (a->workspace && a->workspace_bytes >= short_scratch_bytes(p.M, p.N, s, pair) && (reinterpret_cast<uintptr_t>(a->workspace) & 15) == 0),
                 "b200_qgemm_short: ranges of k want b200_qgemm_short_workspace bytes on a 16-byte boundary");
  B200_CUDA(launch_short(sa, s, pair, (cudaStream_t)stream));
  return B200_OK;
}

int b200_qgemm_swiglu_supported(int64_t M, int64_t N, int64_t K, int qtype, int blocksize) {
  const int block = qtype == B200_Q_INT4 ? 128 : 64;
  if ((qtype != B200_Q_NF4 && qtype != B200_Q_FP4 && qtype != B200_Q_INT4) || blocksize != block) return 0;
  if (M <= 0 || N <= 0 || K <= 0 || K % block || N % 8 || N > 65535LL * 128 || M > 65535LL * 128) return 0;
  return swiglu_plan(M, N, K, qtype == B200_Q_INT4).mt > 0;
}

int b200_qgemm_swiglu(const b200_qgemm_args* a, const void* packed2, const void* scale2, b200_stream_t stream) {
  GemmParams p{};
  if (const int rc = gemm_args(a, p)) return rc;
  B200_CHECK_ARG(packed2 && scale2 && (reinterpret_cast<uintptr_t>(packed2) & 15) == 0, "b200_qgemm_swiglu: null or misaligned second matrix");
  B200_CHECK_ARG(!a->bias, "b200_qgemm_swiglu: takes no bias");
  const GemmPlan g = swiglu_plan(a->M, a->N, a->K, a->qtype == B200_Q_INT4);
  if (g.mt == 0) {
    set_error("b200_qgemm_swiglu: (M=%lld N=%lld K=%lld) runs as two b200_qgemm and b200_swiglu", (long long)a->M, (long long)a->N, (long long)a->K);
    return B200_ERR_UNSUPPORTED;
  }
  return launch_swiglu(a, p, g, packed2, scale2, stream, "b200_qgemm_swiglu");
}

}  // extern "C"
