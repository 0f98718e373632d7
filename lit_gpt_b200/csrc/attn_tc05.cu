// Causal attention of a prompt's rows over a key-value cache or packed rows, head sizes 64 and 128, on the 5th-generation tensor cores.
//
// One CTA = 256 query rows of one head as two tiles of 128, key tiles of 128, one tile's softmax beside the other's products:
//   (small launches: 128 rows per CTA, the second tile empty)
//   * warps 0-3 and 4-7: the softmax of query tile 0 and 1, one row per thread.  S (128 columns of tensor memory) is read into registers, the
//     probabilities go back over it as bf16, the left operand of P V, in two halves so that P V starts on the first.  Half of S is
//     kept in registers from the maximum to the exponentials, the other half read again: 128 registers a thread are all that 16 warps have;
//   * warps 8-11: when a row's maximum grew, they shrink its O in tensor memory while its exponentials are still being taken;
//   * warp 12: one thread issues S = Q K^T (operands in shared memory) and O += P V (P from tensor memory, V as it lies, MN-major), 128 x 128 x
//     16 each, S of a tile's next step right behind its P V;
//   * warp 13 brings the keys, warp 14 the values, two stages each, 128-byte-swizzled: whole tiles by TMA, a tile that ends past the last visible
//     key row by row with cp.async, zeros behind it -- what lies there may be anything, or not be memory at all.  The softmax warps bring Q.
// A masked key has weight 0, and 0 times an infinite or NaN value is NaN: a value that is not finite reaches the rows before its own, within its
// tile of 128 keys and 128 query rows.
// Softmax in fp32 with the exact running maximum, so that the largest probability is 1 and loses nothing to its rounding; probabilities are
// summed as rounded, as they multiply V (the sum of the unrounded ones makes the error against 64 bits 0.1 to 0.4 % larger).  (Moving the maximum only when it grew by 2^8 saves a tenth of the time and raises the error against 64 bits by half.)
//
// Bound: the chain of one tile -- 128 exponentials a row on the special-function units (16 a clock and SM), then its two products, 1270 clocks
// where shared memory feeds them -- of which the other tile's fills the gaps.  32 heads of 128 over 8 key-value heads, 4096 rows: 158 us, 870
// TFLOP/s of the causal half (589 us with the mma.sync tiles of attn_prefill.cu).  Taking a quarter of the exponentials with multiply-adds instead: 225 us, issue slots.
#include "attn_tc05.cuh"
#include "tc05.cuh"

namespace b200 {

namespace {

constexpr int kAtThreads = 480, kAtBM = 128, kAtBN = 128;

typedef unsigned long long f2;   // two packed floats
__device__ __forceinline__ f2 pk2(float a, float b) { f2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ void un2(f2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) { f2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ f2 add2(f2 a, f2 b) { f2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ float ex2(float x) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }

// S = Q K^T: both K-major in shared memory
__device__ __forceinline__ void mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
               ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// O += P V: P in tensor memory
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
               ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void st16(uint32_t addr, const uint32_t (&v)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
               ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
               "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
               : "memory");
}
__device__ __forceinline__ float max3(float a, float b, float c) { float r; asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c)); return r; }
__device__ __forceinline__ void wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

template <int HS>
struct AtTile {
  static constexpr int kPanels = HS / 64;                  // 128-byte-wide panels of a tile of 128 rows
  static constexpr int kBytes = kPanels * 128 * 128;       // one operand tile
  static constexpr int kSmem = 6 * kBytes + 1024;          // Q0 Q1 | K x 2 | V x 2
  static constexpr uint32_t kIdescS = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kAtBN >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
  static constexpr uint32_t kIdescO = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(HS >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
  static constexpr uint32_t kS = 0, kO = 256;              // tensor-memory columns: S0 S1 (P over them) | O0 O1
};

// V tile as the right operand: N = HS contiguous (MN-major), 64 numbers per 128-byte row, one row per key: 8-key groups 1024 bytes apart
// (stride offset), the second panel of 64 numbers 16 KB on (leading offset).  +128 in the address field is 16 keys.
// The low word of the descriptor; the high one is tc::kDescSw128High.
__device__ __forceinline__ uint32_t desc_v_low(uint32_t addr) { return ((addr & 0x3FFFFu) >> 4) | ((16384u >> 4) << 16); }

// Rows [first, first + 128) of a matrix into a swizzled tile by N threads (this one `id`), zeros from row `end` on
template <int HS, int N>
__device__ __forceinline__ void copy_tile(uint32_t dst, const __nv_bfloat16* src, int64_t ld, int first, int end, int id) {
  constexpr int CH = HS / 8, RP = N / CH;   // 16-byte pieces per row, rows per pass
  const int c = id % CH, rr = id / CH;
  const __nv_bfloat16* p = src + (int64_t)(first + rr) * ld + c * 8;
  dst += (uint32_t)(c >> 3) * 16384u;
#pragma unroll 8
  for (int i = 0; i < 128 / RP; ++i) {
    const int r = rr + i * RP;
    const bool in = first + r < end;
    cp16(dst + (uint32_t)(r * 128 + (((c & 7) ^ (r & 7)) << 4)), in ? p + (int64_t)(i * RP) * ld : src, in);
  }
}

template <int HS>
__global__ void __launch_bounds__(kAtThreads, 1)
attn_tc05_kernel(const AttnTc05Args A, const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, unsigned* err) {
  using C = AtTile<HS>;
  extern __shared__ __align__(1024) uint8_t at_smem[];
  __shared__ __align__(8) uint64_t s_bars[26];
  __shared__ float s_shrink[2 * kAtBM];   // per row: what its O and sum shrink by in this step
  __shared__ uint32_t s_tmem;
  __shared__ int s_max[8];
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // (known to be the same in all lanes)
  // Late rows, which see most keys, are scheduled first, those of all heads before any head's earlier ones: with a head's rows next to each other the last heads'
  // late rows started when the others were nearly done (32 heads of 128, 4096 rows: 512 CTAs on 148 SMs, 196 us; 158 in this order).
  const int late = (int)blockIdx.x / A.n_head, h = (int)blockIdx.x - late * A.n_head, b = blockIdx.y, grp = h / (A.n_head / A.n_groups);
  const int block = (int)gridDim.x / A.n_head - 1 - late;                   // the first A.pairs blocks of rows have two tiles, those behind one
  const int r0 = (block + min(block, A.pairs)) * kAtBM, r1 = r0 + (block < A.pairs ? 2 * kAtBM : kAtBM);
  const uint32_t smem = (tc::smem_u32(at_smem) + 1023u) & ~1023u;
  const uint32_t sq_ = smem, sk_ = smem + 2 * C::kBytes, sv_ = smem + 4 * C::kBytes;
  const uint32_t bars = tc::smem_u32(s_bars);
  const uint32_t k_full = bars, v_full = bars + 16, k_empty = bars + 32, v_empty = bars + 48, s_full = bars + 64, p_half = bars + 80, p_full = bars + 96,
                 o_done = bars + 112, q_full = bars + 128, shrink = bars + 136, idle = bars + 200;   // shrink: one per softmax warp; idle: products that gave up

  griddep_launch();
  griddep_wait();
  int T = A.T, pos0 = 0, max_seq = A.max_seq;
  int64_t qrow0 = 0, kvrow0 = 0;
  if (A.seqs) {
    const int4 s = A.seqs[b];
    T = s.y;
    pos0 = s.z;
    max_seq = s.z + s.y;
    qrow0 = s.x;
    kvrow0 = A.kv_first_row ? s.x : s.w;
    if (r0 >= T) return;
  }
  if (tid == 0) {
    tc::mbar_init(q_full, 8);
    tc::mbar_init(idle, 1);
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(k_full + 8 * i, 1);
      tc::mbar_init(v_full + 8 * i, 1);
      tc::mbar_init(k_empty + 8 * i, 1);
      tc::mbar_init(v_empty + 8 * i, 1);
      tc::mbar_init(s_full + 8 * i, 1);
      tc::mbar_init(p_half + 8 * i, 8);   // the softmax and the shrinking warps
      tc::mbar_init(p_full + 8 * i, 4);
      tc::mbar_init(o_done + 8 * i, 1);
    }
    for (int i = 0; i < 8; ++i) tc::mbar_init(shrink + 8 * i, 1);
    tc::mbar_init_fence();
  }
  if (warp == 12) tc::tmem_alloc<512>(tc::smem_u32(&s_tmem));
  // the last key each row sees; a tile's keys end at its rows' maximum
  int lim = -1;
  if (warp < 8) {
    const int r = r0 + tid;
    if (r < T && r < r1) {
      const int64_t p = A.seqs ? (int64_t)pos0 + r : (A.pos64 ? reinterpret_cast<const int64_t*>(A.pos)[r] : (int64_t)reinterpret_cast<const int32_t*>(A.pos)[r]);
      lim = (int)(p < 0 ? 0 : (p >= max_seq ? max_seq - 1 : p));
    }
    const int wl = __reduce_max_sync(0xffffffffu, lim);
    if (lane == 0) s_max[warp] = wl;
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = s_tmem;
  const int window = A.seqs ? A.window : 0;
  int lo[2], hi[2], last = -1;   // key tiles [lo, hi) of either query tile (hi 0: no rows)
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int m = max(max(s_max[4 * t], s_max[4 * t + 1]), max(s_max[4 * t + 2], s_max[4 * t + 3]));
    hi[t] = (m + kAtBN) / kAtBN;
    lo[t] = window > 0 ? max(0, pos0 + r0 + t * kAtBM - window + 1) / kAtBN : 0;
    if (lo[t] > hi[t]) lo[t] = hi[t];
    last = max(last, m);
  }
  const int t_lo = hi[1] > 0 ? min(lo[0], lo[1]) : lo[0], t_hi = max(hi[0], hi[1]);
  bool ok = true;

  if (warp >= 13) {
    // ================================ loads ================================
    auto publish = [&](uint32_t bar) {
      asm volatile("cp.async.wait_all;" ::: "memory");
      tc::fence_smem_async();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(bar);
    };
    const bool keys = warp == 13;
    const __nv_bfloat16* src = keys ? A.k + (int64_t)b * A.k_b + (int64_t)grp * A.k_h + kvrow0 * A.k_r : A.v + (int64_t)b * A.v_b + (int64_t)grp * A.v_h + kvrow0 * A.v_r;
    const int64_t ld = keys ? A.k_r : A.v_r;
    const uint32_t dst = keys ? sk_ : sv_, full = keys ? k_full : v_full, empty = keys ? k_empty : v_empty;
    // the map's column and row of position 0: heads are planes of rows (a cache) or column blocks (packed rows)
    const int x0 = A.seqs ? grp * HS : 0;
    const int64_t row0 = A.seqs ? kvrow0 : ((int64_t)b * A.n_groups + grp) * A.max_seq;
    int i = 0;   // tiles so far
    for (int j = t_lo; j < t_hi; ++j, ++i) {
      const int s = i & 1;
      ok = __all_sync(0xffffffffu, tc::mbar_wait(empty + 8 * s, ((uint32_t)(i >> 1) & 1u) ^ 1u));
      if (!ok) break;
      // (what a cache holds behind the last key does not matter to the scores, which are masked there)
      if ((j + 1) * kAtBN <= (keys && !A.seqs ? A.max_seq : last + 1)) {
        if (lane == 0) {
          tc::mbar_expect_tx(full + 8 * s, C::kBytes);
#pragma unroll
          for (int e = 0; e < C::kPanels; ++e)
            tc::tma_load_2d(dst + s * C::kBytes + e * 16384u, keys ? &map_k : &map_v, x0 + e * 64, (int)(row0 + j * kAtBN), full + 8 * s);
        }
      } else {
        copy_tile<HS, 32>(dst + s * C::kBytes, src, ld, j * kAtBN, last + 1, lane);
        publish(full + 8 * s);
      }
    }
    for (int e = max(i - 2, 0); e < i; ++e) ok = __all_sync(0xffffffffu, tc::mbar_wait(full + 8 * (e & 1), (uint32_t)(e >> 1) & 1u)) && ok;
  } else if (warp == 12) {
    // ================================ products ================================
    if (tc::elect()) {
      const uint32_t q_low = tc::desc_sw128_low(sq_), k_low = tc::desc_sw128_low(sk_), v_low = desc_v_low(sv_);
      auto scores = [&](int t, int s) {                    // S of query tile t with the keys of stage s
        const uint32_t q = q_low + t * (C::kBytes >> 4), k = k_low + s * (C::kBytes >> 4);
#pragma unroll
        for (int e = 0; e < HS / 16; ++e) {
          const uint32_t off = ((uint32_t)(e >> 2) * 16384u + (uint32_t)(e & 3) * 32u) >> 4;
          mma_ss(tmem + C::kS + t * 128, tc::desc_of(q + off, tc::kDescSw128High), tc::desc_of(k + off, tc::kDescSw128High), C::kIdescS, e != 0);
        }
        tc::commit(s_full + 8 * t);
      };
      uint32_t n[2] = {0u, 0u};                            // steps of either tile so far
      ok = tc::mbar_wait_here(q_full, 0) && tc::mbar_wait_here(k_full, 0);
      if (ok) {
        tc::fence_after();
#pragma unroll
        for (int t = 0; t < 2; ++t)
          if (lo[t] == t_lo && lo[t] < hi[t]) scores(t, 0);
        tc::commit(k_empty);
      }
      for (int j = t_lo; j < t_hi && ok; ++j) {
        const int i = j - t_lo, s = i & 1, s1 = s ^ 1;
        const bool more = j + 1 < t_hi;
        ok = tc::mbar_wait_here(v_full + 8 * s, (uint32_t)(i >> 1) & 1u) && (!more || tc::mbar_wait_here(k_full + 8 * s1, (uint32_t)((i + 1) >> 1) & 1u));
        if (!ok) break;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          if (j >= lo[t] && j < hi[t]) {
            const uint32_t dv = v_low + s * (C::kBytes >> 4);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              ok = ok && tc::mbar_wait_here((half ? p_full : p_half) + 8 * t, n[t] & 1u);
              if (!ok) break;
              tc::fence_after();
#pragma unroll
              for (int e = 4 * half; e < 4 * half + 4; ++e)
                mma_ts(tmem + C::kO + t * HS, tmem + C::kS + t * 128 + e * 8, tc::desc_of(dv + 128 * e, tc::kDescSw128High), C::kIdescO, (n[t] | (uint32_t)e) != 0);
            }
            if (!ok) break;
            tc::commit(o_done + 8 * t);
            ++n[t];
          }
          if (more && j + 1 >= lo[t] && j + 1 < hi[t]) scores(t, s1);
        }
        if (!ok) break;
        tc::commit(v_empty + 8 * s);
        if (more) tc::commit(k_empty + 8 * s1);
      }
      if (!ok) {
        tc::commit(idle);
        tc::mbar_wait(idle, 0);
      }
    }
  } else if (warp >= 8) {
    // ================================ shrinking O ================================
    const int w = warp - 8;
    uint32_t n[2] = {0u, 0u};
    for (int j = t_lo; j < t_hi && ok; ++j) {
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        if (j < lo[t] || j >= hi[t]) continue;
        ok = ok && __all_sync(0xffffffffu, tc::mbar_wait(shrink + 8 * (4 * t + w), n[t] & 1u));
        if (!ok) break;
        const float f = s_shrink[t * kAtBM + w * 32 + lane];
        if (n[t] > 0 && __any_sync(0xffffffffu, f != 1.0f)) {   // (S of this step is there, so P V of the last one is done)
          tc::fence_after();
          const uint32_t to = tmem + ((uint32_t)(w * 32) << 16) + C::kO + t * HS;
#pragma unroll 1
          for (int c = 0; c < HS; c += 32) {
            uint32_t o[32];
            tc::ld32(o, to + c);
            tc::wait_ld(o);
            uint32_t a[16], bb[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              a[e] = __float_as_uint(__uint_as_float(o[e]) * f);
              bb[e] = __float_as_uint(__uint_as_float(o[16 + e]) * f);
            }
            st16(to + c, a);
            st16(to + c + 16, bb);
          }
          wait_st();
          tc::fence_before();
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(p_half + 8 * t);
        ++n[t];
      }
    }
  } else {
    // ================================ softmax: a row per thread ================================
    const int t = warp >> 2, r = r0 + tid;
    copy_tile<HS, 128>(sq_ + t * C::kBytes, A.q + (int64_t)b * A.q_b + (int64_t)h * A.q_h + qrow0 * A.q_r, A.q_r, r0 + t * kAtBM, min(T, r1), tid & 127);
    asm volatile("cp.async.wait_all;" ::: "memory");
    tc::fence_smem_async();
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(q_full);
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t ts = tmem + lanes + C::kS + t * 128, to = tmem + lanes + C::kO + t * HS;
    const int low = window > 0 ? lim - window + 1 : 0;
    const int w_lim = __reduce_min_sync(0xffffffffu, lim < 0 ? 0x7fffffff : lim), w_low = __reduce_max_sync(0xffffffffu, lim < 0 ? 0 : low);
    const float sl = A.scale_log2;
    float m = -INFINITY;
    f2 l2[2] = {0ull, 0ull};
    uint32_t n = 0;
    const int j_lo = t ? lo[1] : lo[0], j_hi = t ? hi[1] : hi[0];
    for (int j = j_lo; j < j_hi; ++j, ++n) {
      ok = ok && __all_sync(0xffffffffu, tc::mbar_wait(s_full + 8 * t, n & 1u));
      if (!ok) break;
      tc::fence_after();
      const int j0 = j * kAtBN;
      const bool masked = j0 + kAtBN - 1 > w_lim || j0 < w_low;   // (rows past the sequence are computed and not stored)
      auto mask = [&](uint32_t (&s)[32], int i) {
        if (masked) {
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            const int key = j0 + i * 32 + e;
            if (key > lim || key < low) s[e] = 0xff800000u;
          }
        }
      };
      auto most = [](const uint32_t (&s)[32], float mx) {
#pragma unroll
        for (int e = 0; e < 32; e += 2) mx = max3(mx, __uint_as_float(s[e]), __uint_as_float(s[e + 1]));
        return mx;
      };
      uint32_t s0[32], s1[32];
      float mx[4];
      tc::ld32(s0, ts + 64);
      tc::ld32(s1, ts + 96);
      tc::wait_ld(s0);
      tc::wait_ld(s1);
      mask(s0, 2);
      mask(s1, 3);
      mx[2] = most(s0, -INFINITY);
      mx[3] = most(s1, -INFINITY);
      tc::ld32(s0, ts);
      tc::ld32(s1, ts + 32);
      tc::wait_ld(s0);
      tc::wait_ld(s1);
      mask(s0, 0);
      mask(s1, 1);
      mx[0] = most(s0, -INFINITY);
      mx[1] = most(s1, -INFINITY);
      const float nm = fmaxf(m, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])));
      const float f = m == -INFINITY ? 1.0f : ex2((m - nm) * sl);   // nothing seen so far: O and the sum are zero
      m = nm;
      s_shrink[tid] = f;
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(shrink + 8 * warp);
      const f2 ff = pk2(f, f);
      l2[0] = fma2(l2[0], ff, 0ull);
      l2[1] = fma2(l2[1], ff, 0ull);
      const float org = m == -INFINITY ? 0.f : m * sl;   // rows with nothing visible yet: exp2(-inf) = 0
      const f2 sl2 = pk2(sl, sl), org2 = pk2(-org, -org);
      auto exps = [&](const uint32_t (&s)[32], int i) {
        uint32_t p[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          float a, c;
          un2(fma2(pk2(__uint_as_float(s[2 * e]), __uint_as_float(s[2 * e + 1])), sl2, org2), a, c);
          p[e] = pack_bf16(ex2(a), ex2(c));
          l2[e & 1] = add2(l2[e & 1], pk2(bf16lo(p[e]), bf16hi(p[e])));
        }
        st16(ts + i * 16, p);
      };
      auto hand_over = [&](uint32_t bar) {
        wait_st();
        tc::fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(bar + 8 * t);
      };
      exps(s0, 0);
      tc::ld32(s0, ts + 64);   // (P so far lies in columns 0 .. 31, at most 0 .. 63: scores 64 .. 127 are still there)
      exps(s1, 1);
      tc::wait_ld(s0);
      tc::ld32(s1, ts + 96);
      hand_over(p_half);
      mask(s0, 2);
      exps(s0, 2);
      tc::wait_ld(s1);
      mask(s1, 3);
      exps(s1, 3);
      hand_over(p_full);
    }
    if (n > 0 && ok) {
      ok = __all_sync(0xffffffffu, tc::mbar_wait(o_done + 8 * t, (n - 1) & 1u));
      tc::fence_after();
    }
    if (ok && j_hi > 0) {
      float a, c, d, e;
      un2(l2[0], a, c);
      un2(l2[1], d, e);
      const float l = (a + c) + (d + e);
      float inv = l > 0.f ? 1.0f / l : 0.f;
      if (A.seqs && A.sink) {   // the sink joins the denominator once: l is in units of exp2(m * scale_log2)
        const float sk = __bfloat162float(A.sink[h]) * 1.4426950408889634f;
        const float o = m == -INFINITY ? sk : fmaxf(m * sl, sk), f = m == -INFINITY ? 0.f : exp2f(m * sl - o);
        inv = f / (l * f + exp2f(sk - o));
      }
      __nv_bfloat16* const yr = A.y + (int64_t)b * A.y_b + (qrow0 + r) * A.y_r + (int64_t)h * HS;
      const bool wide = (reinterpret_cast<uintptr_t>(A.y) & 15) == 0 && ((A.y_r | A.y_b) & 7) == 0;
#pragma unroll 1
      for (int c0 = 0; c0 < HS; c0 += 32) {
        uint32_t o[32], w[16];
        tc::ld32(o, to + c0);
        tc::wait_ld(o);
#pragma unroll
        for (int i = 0; i < 16; ++i) w[i] = n > 0 ? pack_bf16(__uint_as_float(o[2 * i]) * inv, __uint_as_float(o[2 * i + 1]) * inv) : 0u;
        if (r < T) {
          if (wide) {
#pragma unroll
            for (int i = 0; i < 16; i += 4) *reinterpret_cast<uint4*>(yr + c0 + 2 * i) = make_uint4(w[i], w[i + 1], w[i + 2], w[i + 3]);
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) *reinterpret_cast<uint32_t*>(yr + c0 + 2 * i) = w[i];
          }
        }
      }
    }
  }
  if (!ok) *err = 1u;
  tc::fence_before();
  __syncthreads();
  if (warp == 12) {
    __syncwarp();
    tc::tmem_free<512>(tmem);
  }
}

template <int HS>
cudaError_t launch_hs(AttnTc05Args a, int batch, cudaStream_t st) {
  constexpr int smem = AtTile<HS>::kSmem;
  static PerDeviceOnce once;
  if (once.need()) {
    const cudaError_t e = cudaFuncSetAttribute(attn_tc05_kernel<HS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    once.done();
  }
  // The maps bound the columns only: boxes stay inside the rows a sequence has by the kernel's own choice of tiles
  alignas(64) CUtensorMap mk, mv;
  const int64_t rows = 0x7fffffff, cols = a.seqs ? (int64_t)a.n_groups * HS : HS;
  if (!tensor_map_2d(&mk, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a.k, rows, cols, a.k_r * 2, 128) ||
      !tensor_map_2d(&mv, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a.v, rows, cols, a.v_r * 2, 128))
    return cudaErrorInvalidValue;
  // Two tiles take turns on one SM's issue slots and special-function units; a CTA with one goes through its keys in 0.85 of the time.  So as many blocks of rows have
  // one tile as still run at once, the late ones, which see most keys; where even pairs take more than a round, all are pairs.  32 heads of 128, 160 / 256 / 400 rows
  // from position 0, us with two tiles and with one: 12.6, 10.8 / 13.2, 11.3 / 17.9, 16.0; from position 4000 80.6, 70.6 / 84.9, 72.6 / 86.7, 77.4.  A pair and three of one,
  // all pairs before: 613 rows of 32 heads from position 1500 44.9, 41.4, 500 of 40 heads from 700 34.0, 30.3; 300 of 40 heads from 0, one each, 14.2, 12.9.
  const int64_t tiles = ((int64_t)a.T + kAtBM - 1) / kAtBM, chains = (int64_t)a.n_head * batch, fit = sm_count() / chains;
  const int64_t pairs = tiles <= fit ? 0 : tiles - fit <= tiles / 2 ? tiles - fit : tiles / 2;
  a.pairs = (int)pairs;
  const dim3 grid((unsigned)((tiles - pairs) * a.n_head), (unsigned)batch);
  unsigned* const err = wait_error_word();
  if (!err) return cudaErrorMemoryAllocation;
  return launch(attn_tc05_kernel<HS>, grid, dim3(kAtThreads), (size_t)smem, st, a, mk, mv, err);
}

}  // namespace

cudaError_t launch_attn_tc05(const AttnTc05Args& a, int head_size, int batch, cudaStream_t st) {
  return head_size == 128 ? launch_hs<128>(a, batch, st) : launch_hs<64>(a, batch, st);
}

}  // namespace b200
