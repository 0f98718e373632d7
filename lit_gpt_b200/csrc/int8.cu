// bnb.int8 -- LLM.int8() inference Linear (bitsandbytes 0.41 nn.Linear8bitLt(has_fp16_weights=False, threshold=6.0),
// selected by `--quantize bnb.int8` at generate/base.py:105,129-134; semantics restated in oracle/quant_ref.py:310-345).
//
//   weight:      CB  = rint(W * 127 / absmax_row)  int8 (N, K),   SCB = absmax_row fp32 (N)
//   activation:  columns k with any |x[m,k]| >= threshold are OUTLIERS: they leave the int8 product and go through an
//                fp16 side product against the dequantised weight columns; the rest is quantised per row,
//                CA = rint(x * 127 / absmax_row), SCA = absmax_row
//   y = f16( int32(CA . CB^T) * (SCA * SCB / 127^2) )  [+ bias -> f16]  [+ f16(x_out . f16(CB_out * SCB / 127)^T) -> f16]
//
// The int8 x int8 -> int32 products are exact and order-free.  Two mappings:
//   rows <= 16 (decode): mma.sync m16n8k32 s8, the weights loaded straight from HBM in fragment order (16 contiguous bytes of one row per
//   lane; the K permutation this implies is applied to both operands); one CTA per 16 weight rows, its 8 warps split K, int32 partials
//   meet in shared memory;
//   rows  > 16 (prefill): tcgen05.mma kind::i8 over TMA-fed tiles of both operands, int32 accumulators in tensor memory (int8_gemm_kernel).
#include "tc05.cuh"

namespace b200 {

constexpr int kI8Threads = 256;
constexpr int kI8Warps = 8;

__device__ __forceinline__ void imma16832(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// ---- weight quantisation: one CTA per output row ---------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) quantize_int8_rows_kernel(const T* __restrict__ w, int64_t K, int8_t* __restrict__ cb,
                                                                 float* __restrict__ scb) {
  __shared__ float s_max[8];
  const int64_t n = blockIdx.x;
  const T* row = w + n * K;
  float m = 0.f;
  for (int64_t k = threadIdx.x; k < K; k += 256) m = fmaxf(m, fabsf(load_as_float<T>(row, k)));
  m = warp_max(m);
  if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = m;
  __syncthreads();
  m = s_max[0];
#pragma unroll
  for (int i = 1; i < 8; ++i) m = fmaxf(m, s_max[i]);
  if (threadIdx.x == 0) scb[n] = m;
  const float inv = __fdiv_rn(127.0f, m);  // inf for an all-zero row: 0 * inf = NaN -> 0 below (np.nan_to_num)
  for (int64_t k = threadIdx.x; k < K; k += 256) {
    const float v = __fmul_rn(load_as_float<T>(row, k), inv);
    cb[n * K + k] = (v != v) ? (int8_t)0 : (int8_t)__float2int_rn(v);
  }
}

template <typename T>
__global__ void __launch_bounds__(256) dequantize_int8_rows_kernel(const int8_t* __restrict__ cb, const float* __restrict__ scb, int64_t N,
                                                                   int64_t K, T* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= N * K) return;
  store_from_float<T>(out, i, __fmul_rn((float)cb[i], __fdiv_rn(scb[i / K], 127.0f)));
}

// ---- activation side ------------------------------------------------------------------------------------------
// flags[k] = 1 when any row has |x[m,k]| >= threshold.  A thread looks at eight neighbouring columns of `block_rows` rows; with one row block
// the flags are written outright, with more they start at zero and only hits are written.  (One thread per column walking every row kept
// 16 CTAs busy for 4096 columns: 250 us of the 750 at 777 rows.)
__global__ void __launch_bounds__(128) int8_outlier_flags_kernel(const __half* __restrict__ x, int64_t M, int64_t K, float threshold, int block_rows, int* __restrict__ flags) {
  griddep_launch();
  griddep_wait();
  const int64_t k = ((int64_t)blockIdx.x * 128 + threadIdx.x) * 8;
  if (k >= K) return;
  const int64_t m0 = (int64_t)blockIdx.y * block_rows;
  const int rows = (int)(M - m0 < block_rows ? M - m0 : block_rows);
  const __half* px = x + m0 * K + k;
  unsigned hit = 0;
  if (threshold > 0.f) {
#pragma unroll 8
    for (int r = 0; r < rows; ++r) {
      const uint4 v = *reinterpret_cast<const uint4*>(px + (int64_t)r * K);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[j]));
        hit |= (fabsf(f.x) >= threshold ? 1u : 0u) << (2 * j) | (fabsf(f.y) >= threshold ? 1u : 0u) << (2 * j + 1);
      }
    }
  }
  if (gridDim.y == 1) {
#pragma unroll
    for (int j = 0; j < 8; ++j) flags[k + j] = (hit >> j) & 1u;
  } else if (hit) {
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if ((hit >> j) & 1u) flags[k + j] = 1;
  }
}

// ordered compaction of the flagged columns (ascending k: the fp32 side product is summed in this order), by one CTA of 256 threads
__device__ __forceinline__ void int8_compact(const int* __restrict__ flags, int64_t K, int* __restrict__ idx, int* __restrict__ count) {
  __shared__ int s_sum[8];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int64_t per = (K / 4 + 255) / 256, beg = t * per < K / 4 ? t * per : K / 4, end = beg + per < K / 4 ? beg + per : K / 4;   // fours of columns
  int c = 0;
  for (int64_t i = beg; i < end; ++i) {
    const int4 f = reinterpret_cast<const int4*>(flags)[i];
    c += f.x + f.y + f.z + f.w;
  }
  int incl = c;   // inclusive scan over the warp, then over the warps' sums
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) s_sum[warp] = incl;
  __syncthreads();
  int before = 0;
  for (int w = 0; w < warp; ++w) before += s_sum[w];
  int pos = before + incl - c;
  if (c) {
    for (int64_t i = beg; i < end; ++i) {
      const int4 f = reinterpret_cast<const int4*>(flags)[i];
      const int k = (int)(4 * i);
      if (f.x) idx[pos++] = k;
      if (f.y) idx[pos++] = k + 1;
      if (f.z) idx[pos++] = k + 2;
      if (f.w) idx[pos++] = k + 3;
    }
  }
  if (t == 255) *count = before + incl;
}

// one CTA per activation row: SCA = absmax over the non-outlier columns, CA = rint(x * 127 / SCA) (0 in outlier columns)
// (K is a multiple of 64 and the rows start on 16-byte boundaries: eight columns per access, the first 8192 kept in registers between
// the maximum and the rounding); the first CTA makes the list of outlier columns beside them (a launch of its own between the flags and the rows took 4 us of
// a call's 62)
__global__ void __launch_bounds__(256) int8_rowquant_kernel(const __half* __restrict__ x, int64_t K, const int* __restrict__ flags,
                                                            int8_t* __restrict__ ca, float* __restrict__ sca, int* __restrict__ idx, int* __restrict__ count) {
  __shared__ float s_max[8];
  constexpr int KEEP = 4;
  griddep_launch();
  griddep_wait();
  if (blockIdx.x == 0) {
    int8_compact(flags, K, idx, count);
    return;
  }
  const int64_t m = (int64_t)blockIdx.x - 1;
  const __half* row = x + m * K;
  const int nv = (int)(K >> 3);
  auto load = [&](int i, float (&f)[8]) {   // eight columns, outliers as 0
    const uint4 v = reinterpret_cast<const uint4*>(row)[i];
    const int4 fa = reinterpret_cast<const int4*>(flags)[2 * i], fb = reinterpret_cast<const int4*>(flags)[2 * i + 1];
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    const int fl[8] = {fa.x, fa.y, fa.z, fa.w, fb.x, fb.y, fb.z, fb.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&w[j]));
      f[2 * j] = fl[2 * j] ? 0.f : h.x;
      f[2 * j + 1] = fl[2 * j + 1] ? 0.f : h.y;
    }
  };
  float kept[KEEP][8];
  float mx = 0.f;
#pragma unroll
  for (int u = 0; u < KEEP; ++u) {
    const int i = (int)threadIdx.x + u * 256;
    if (i < nv) {
      load(i, kept[u]);
#pragma unroll
      for (int j = 0; j < 8; ++j) mx = fmaxf(mx, fabsf(kept[u][j]));
    }
  }
  for (int i = (int)threadIdx.x + KEEP * 256; i < nv; i += 256) {
    float f[8];
    load(i, f);
#pragma unroll
    for (int j = 0; j < 8; ++j) mx = fmaxf(mx, fabsf(f[j]));
  }
  mx = warp_max(mx);
  if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = mx;
  __syncthreads();
  mx = s_max[0];
#pragma unroll
  for (int i = 1; i < 8; ++i) mx = fmaxf(mx, s_max[i]);
  if (threadIdx.x == 0) sca[m] = mx;
  const float inv = __fdiv_rn(127.0f, mx);
  auto store = [&](int i, const float (&f)[8]) {
    uint32_t o[2] = {0u, 0u};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float v = __fmul_rn(f[j], inv);
      const int8_t q = (v != v) ? (int8_t)0 : (int8_t)__float2int_rn(v);
      o[j >> 2] |= (uint32_t)(uint8_t)q << (8 * (j & 3));
    }
    *reinterpret_cast<uint2*>(ca + m * K + (int64_t)i * 8) = make_uint2(o[0], o[1]);
  };
#pragma unroll
  for (int u = 0; u < KEEP; ++u) {
    const int i = (int)threadIdx.x + u * 256;
    if (i < nv) store(i, kept[u]);
  }
  for (int i = (int)threadIdx.x + KEEP * 256; i < nv; i += 256) {
    float f[8];
    load(i, f);
    store(i, f);
  }
}

struct I8Params {
  const int8_t* cb;      // (N, K)
  const float* scb;      // (N)
  const __half* x;       // (M, K) original activations (outlier side product)
  const int8_t* ca;      // (M, K)
  const float* sca;      // (M)
  const int* idx;        // outlier columns, ascending
  const int* count;
  const __half* bias;    // (N) or null
  __half* y;             // (M, N)
  int64_t M, N, K;
};

__device__ __forceinline__ float round_f16(float v) { return __half2float(__float2half_rn(v)); }

// oracle/quant_ref.py:337-345: scale, round, bias, round, outlier side product, round
__device__ __forceinline__ void i8_store(const I8Params& p, int64_t m, int64_t n, int acc) {
  const float scale = __fdiv_rn(__fmul_rn(p.sca[m], p.scb[n]), 127.0f * 127.0f);
  float out = round_f16(__fmul_rn((float)acc, scale));
  if (p.bias) out = round_f16(out + __half2float(p.bias[n]));
  const int no = *p.count;
  if (no > 0) {
    const float wscale = __fdiv_rn(p.scb[n], 127.0f);
    float sub = 0.f;
    for (int j = 0; j < no; ++j) {
      const int k = p.idx[j];
      sub = fmaf(__half2float(p.x[m * p.K + k]), round_f16(__fmul_rn((float)p.cb[n * p.K + k], wscale)), sub);
    }
    out = round_f16(out + round_f16(sub));
  }
  p.y[m * p.N + n] = __float2half_rn(out);
}

// ---- decode: M <= 16.  grid = ceil(N / 16); 8 warps split K in 64-byte chunks ------------------------------------
template <int MB>
__global__ void __launch_bounds__(kI8Threads) int8_gemv_kernel(const I8Params p) {
  __shared__ int s_red[kI8Warps][16][8 * MB];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int64_t n0 = (int64_t)blockIdx.x * 16;
  const int64_t ra = n0 + g < p.N ? n0 + g : p.N - 1, rb = n0 + g + 8 < p.N ? n0 + g + 8 : p.N - 1;
  const int8_t* wa = p.cb + ra * p.K + 16 * t;
  const int8_t* wb = p.cb + rb * p.K + 16 * t;
  const int nchunks = (int)(p.K >> 6);
  int acc[MB][4];
#pragma unroll
  for (int mb = 0; mb < MB; ++mb) acc[mb][0] = acc[mb][1] = acc[mb][2] = acc[mb][3] = 0;

  constexpr int U = 4;  // chunks in flight per warp
  uint4 a[U], b[U];
  // the weights do not depend on the previous kernel: request the first chunks before waiting for it
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int c = warp + u * kI8Warps;
    a[u] = b[u] = make_uint4(0u, 0u, 0u, 0u);
    if (c < nchunks) { a[u] = ldg_stream_v4(wa + (int64_t)c * 64); b[u] = ldg_stream_v4(wb + (int64_t)c * 64); }
  }
  griddep_launch();
  griddep_wait();
  for (int c0 = warp; c0 < nchunks; c0 += U * kI8Warps) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int c = c0 + u * kI8Warps;
      if (c < nchunks) {
        const uint4 av = a[u], bv = b[u];
        const int cn = c + U * kI8Warps;
        if (cn < nchunks) { a[u] = ldg_stream_v4(wa + (int64_t)cn * 64); b[u] = ldg_stream_v4(wb + (int64_t)cn * 64); }
#pragma unroll
        for (int mb = 0; mb < MB; ++mb) {
          const int64_t m = mb * 8 + g;
          uint4 xv = make_uint4(0u, 0u, 0u, 0u);
          if (m < p.M) xv = *reinterpret_cast<const uint4*>(p.ca + m * p.K + (int64_t)c * 64 + 16 * t);
          imma16832(acc[mb], av.x, bv.x, av.y, bv.y, xv.x, xv.y);
          imma16832(acc[mb], av.z, bv.z, av.w, bv.w, xv.z, xv.w);
        }
      }
    }
  }
#pragma unroll
  for (int mb = 0; mb < MB; ++mb) {
    s_red[warp][g][8 * mb + 2 * t] = acc[mb][0];
    s_red[warp][g][8 * mb + 2 * t + 1] = acc[mb][1];
    s_red[warp][g + 8][8 * mb + 2 * t] = acc[mb][2];
    s_red[warp][g + 8][8 * mb + 2 * t + 1] = acc[mb][3];
  }
  __syncthreads();
  for (int o = tid; o < 16 * 8 * MB; o += kI8Threads) {
    const int r = o / (8 * MB), c = o % (8 * MB);
    if (c < p.M && n0 + r < p.N) {
      int s = 0;
#pragma unroll
      for (int w = 0; w < kI8Warps; ++w) s += s_red[w][r][c];
      i8_store(p, c, n0 + r, s);
    }
  }
}

// ---- prefill: M > 16 ----------------------------------------------------------------------------------------------
// Persistent over output tiles, neighbouring CTAs on the same weight rows.  One thread loads 128-byte-wide boxes of both operands by TMA into a
// ring of stages, one issues tcgen05.mma kind::i8 (K = 32) into one of two tensor-memory accumulators, and sixteen epilogue warps scale, round
// and store the other: the epilogue (a division, three roundings and the outlier columns per output) hides behind the next tile's products.
//   PAIR = true: a CTA pair on 256 rows x up to 256 features (i8_features), each CTA holding 128 rows of the activations and half of the features.  The
//   copies are the limit of the int8 pipe: an SM takes 48.7 bytes a clock of 128-byte boxes from L2 (measured with copies alone), the pair's products at
//   full rate 64, a CTA alone on 128 x 128 twice that.  777 x 4096 -> 11008 with its preparing kernels, six outlier columns: 780 us with fragments read
//   from L2, 100 us with 128 x 128 tiles, 66.6 us with pairs of 256 features and eight epilogue warps, 62.7 with sixteen and 224 features (4096 rows ->
//   12288: 338, 220 and 221 us, 1.9 POP/s).  The list of outlier columns beside the row quantisation takes 2 us off all of these.
//   PAIR = false: one CTA on 128 x 128, for up to 128 rows, where the second half of a pair's rows would be padding.
constexpr int kI8EpiWarps = 16, kI8GemmThreads = (kI8EpiWarps + 2) * 32;
constexpr int kI8KB = 128;                       // int8 columns per stage: one 128-byte swizzle row
constexpr int kI8Stages = 6, kI8Stage = 256 * kI8KB, kI8Smem = kI8Stages * kI8Stage + 1024;   // 128 rows of either operand
static_assert(kI8Smem >= tc::kPairMinSmem, "one CTA of a pair per SM");

// kind::i8: D = int32, A = B = signed 8 bit, both K-major
template <bool PAIR>
__device__ __forceinline__ void umma_i8(uint32_t tmem_d, uint64_t da, uint64_t db, int n, uint32_t accumulate) {
  constexpr uint32_t kM = PAIR ? 256 : 128;
  const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((kM >> 4) << 24);
  if constexpr (PAIR)
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}

// x / 127^2 rounded as the division is: the reciprocal, then one Newton step on the remainder (Markstein); beyond 1e30 the division itself
__device__ __forceinline__ float i8_scale(float x) {
  constexpr float d = 127.0f * 127.0f, r = 1.0f / d;
  if (!(x < 1e30f)) return __fdiv_rn(x, d);
  const float q = __fmul_rn(x, r);
  return fmaf(fmaf(-q, d, x), r, q);
}
__device__ __forceinline__ float2 round_f16x2(float a, float b) { return __half22float2(__floats2half2_rn(a, b)); }

template <bool PAIR>
__global__ void __launch_bounds__(kI8GemmThreads, 1)
int8_gemm_kernel(const I8Params p, const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, int m_tiles, int n_tiles, int bn, unsigned* err) {
  constexpr int CTAS = PAIR ? 2 : 1, BM = 128 * CTAS, BN = BM;   // bn: features of a tile, a multiple of 32 up to BN
  extern __shared__ __align__(1024) uint8_t i8_smem[];
  __shared__ __align__(8) uint64_t s_bars[2 * kI8Stages + 5];
  __shared__ uint32_t s_tmem;
  __shared__ __align__(16) float s_feat[10][BN];               // per feature of the tile: weight scale, bias, weight in the first eight outlier columns
  __shared__ __align__(16) float s_more[kI8EpiWarps][8][16];   // per epilogue warp: the weights of 16 features in the next eight
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // (known to be the same in all lanes)
  const uint32_t rank = PAIR ? tc::cluster_rank() : 0u;
  const uint32_t tiles = (tc::smem_u32(i8_smem) + 1023u) & ~1023u;
  const uint32_t full = tc::smem_u32(&s_bars[0]), empty = tc::smem_u32(&s_bars[kI8Stages]);
  const uint32_t acc_full = tc::smem_u32(&s_bars[2 * kI8Stages]), acc_empty = acc_full + 16, idle = acc_full + 32;
  if (tid == 0) {
    for (int s = 0; s < kI8Stages; ++s) { tc::mbar_init(full + 8 * s, 1); tc::mbar_init(empty + 8 * s, 1); }
    for (int a = 0; a < 2; ++a) { tc::mbar_init(acc_full + 8 * a, 1); tc::mbar_init(acc_empty + 8 * a, kI8EpiWarps * CTAS); }
    tc::mbar_init(idle, 1);
    tc::mbar_init_fence();
    tc::prefetch_map(&map_a);
    tc::prefetch_map(&map_b);
  }
  griddep_launch();
  griddep_wait();
  if (warp == kI8EpiWarps) {
    if constexpr (PAIR) tc::tmem_alloc_pair<2 * BN>(tc::smem_u32(&s_tmem));
    else tc::tmem_alloc<2 * BN>(tc::smem_u32(&s_tmem));
  }
  tc::fence_before();
  if constexpr (PAIR) tc::cluster_sync();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = s_tmem;
  const int nkb = (int)((p.K + kI8KB - 1) / kI8KB), total = m_tiles * n_tiles;
  const int first = (int)blockIdx.x / CTAS, step = (int)gridDim.x / CTAS;
  bool ok = true;

  if (warp == kI8EpiWarps) {
    // ---- copies: 128 rows of either operand into this CTA's stage, counted on the issuing CTA's barrier ----
    if (tc::elect()) {
      int s = 0;
      uint32_t ph = 1;
      for (int t = first; t < total && ok; t += step) {
        const int m0 = (t % m_tiles) * BM + (int)rank * 128, n0 = (t / m_tiles) * bn + (int)rank * (bn / CTAS);
        for (int kb = 0; kb < nkb; ++kb) {
          ok = PAIR ? tc::mbar_wait_cluster(empty + 8 * s, ph) : tc::mbar_wait(empty + 8 * s, ph);
          if (!ok) break;
          const uint32_t st = tiles + s * kI8Stage;
          if (rank == 0) tc::mbar_expect_tx(full + 8 * s, (BM + bn) * kI8KB);
          if constexpr (PAIR) {
            const uint32_t bar = tc::at_rank(full + 8 * s, 0);
            tc::tma_load_2d_pair(st, &map_a, kb * kI8KB, m0, bar);
            tc::tma_load_2d_pair(st + 128 * kI8KB, &map_b, kb * kI8KB, n0, bar);
          } else {
            tc::tma_load_2d(st, &map_a, kb * kI8KB, m0, full + 8 * s);
            tc::tma_load_2d(st + 128 * kI8KB, &map_b, kb * kI8KB, n0, full + 8 * s);
          }
          if (++s == kI8Stages) { s = 0; ph ^= 1u; }
        }
      }
      if (rank == 0)
        for (int i = 0; i < kI8Stages; ++i) {
          const uint32_t last = i < s ? ph ^ 1u : ph;   // (a stage never used: the phase before the first)
          ok = (PAIR ? tc::mbar_wait_cluster(full + 8 * i, last) : tc::mbar_wait(full + 8 * i, last)) && ok;
        }
    }
  } else if (warp == kI8EpiWarps + 1) {
    // ---- products ----
    if (rank == 0 && tc::elect()) {
      auto wait_here = [](uint32_t bar, uint32_t parity) { return PAIR ? tc::mbar_wait_cluster_here(bar, parity) : tc::mbar_wait_here(bar, parity); };
      int s = 0, acc = 0;
      uint32_t ph = 0, aph = 1;
      for (int t = first; t < total && ok; t += step) {
        ok = wait_here(acc_empty + 8 * acc, aph);
        for (int kb = 0; kb < nkb && ok; ++kb) {
          ok = wait_here(full + 8 * s, ph);
          if (!ok) break;
          tc::fence_after();
          const uint32_t da = tc::desc_sw128_low(tiles + s * kI8Stage), db = da + (128 * kI8KB >> 4);
#pragma unroll
          for (int k = 0; k < kI8KB / 32; ++k)
            umma_i8<PAIR>(tmem + acc * BN, tc::desc_of(da + 2 * k, tc::kDescSw128High), tc::desc_of(db + 2 * k, tc::kDescSw128High), bn, (kb | k) != 0);
          if constexpr (PAIR) tc::commit_pair(empty + 8 * s);
          else tc::commit(empty + 8 * s);
          if (++s == kI8Stages) { s = 0; ph ^= 1u; }
        }
        if (ok) {
          if constexpr (PAIR) tc::commit_pair(acc_full + 8 * acc);
          else tc::commit(acc_full + 8 * acc);
        }
        acc ^= 1;
        if (acc == 0) aph ^= 1u;
      }
      if (!ok) {
        if constexpr (PAIR) tc::commit_pair(idle);
        else tc::commit(idle);
        tc::mbar_wait(idle, 0);
      }
    }
  } else {
    // ---- epilogue: warp w holds rows 32 (w % 4) .. + 31 and every fourth sixteen of the columns ----
    int acc = 0;
    uint32_t ph = 0;
    const int no = *p.count;
    const bool vec = (p.N & 7) == 0 && (reinterpret_cast<uintptr_t>(p.y) & 15) == 0;
    int k0[8];   // the first eight outlier columns
#pragma unroll
    for (int j = 0; j < 8; ++j) k0[j] = j < no ? p.idx[j] : 0;
    float(&more)[8][16] = s_more[warp];
    for (int t = first; t < total; t += step) {
      const int64_t mw = (int64_t)(t % m_tiles) * BM + rank * 128 + (warp & 3) * 32, m = mw + lane, n0 = (int64_t)(t / m_tiles) * bn;
      const bool mok = m < p.M;
      const float sca = mok ? p.sca[m] : 0.f;
      const __half* const xr = p.x + (mok ? m : 0) * p.K;
      float x0[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) x0[j] = j < no ? __half2float(xr[k0[j]]) : 0.f;
      // the tile's features, one per thread, while its products are still running (a gather per 32 columns in the loop below cost more than
      // the products: 72 us of 266 at 4096 rows with six outlier columns)
      asm volatile("bar.sync 1, %0;" ::"n"(kI8EpiWarps * 32) : "memory");   // the last tile's readers are done
      if (tid < bn) {
        const int64_t n = n0 + tid;
        const bool nok = n < p.N;
        const float scb = nok ? p.scb[n] : 0.f, ws = __fdiv_rn(scb, 127.0f);
        const int8_t* const cb = p.cb + (nok ? n : 0) * p.K;
        float w[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) w[j] = j < no ? (float)cb[k0[j]] : 0.f;
        s_feat[0][tid] = scb;
        s_feat[1][tid] = nok && p.bias ? __half2float(p.bias[n]) : 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (j < no) s_feat[2 + j][tid] = round_f16(__fmul_rn(w[j], ws));
      }
      asm volatile("bar.sync 1, %0;" ::"n"(kI8EpiWarps * 32) : "memory");
      ok = ok && __all_sync(0xffffffffu, PAIR ? tc::mbar_wait_cluster(acc_full + 8 * acc, ph) : tc::mbar_wait(acc_full + 8 * acc, ph));
      tc::fence_after();
      const int c_end = mw < p.M && ok ? bn : 0;   // (a warp whose rows are all past the last one has nothing to do)
#pragma unroll 1
      for (int c0 = (warp >> 2) * 16; c0 < c_end; c0 += 64) {
        uint32_t v[16];
        tc::ld16(v, tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(acc * BN + c0));
        tc::wait_ld(v);
        float out[16];
#pragma unroll
        for (int e = 0; e < 16; e += 2) {
          const float2 sc = *reinterpret_cast<const float2*>(&s_feat[0][c0 + e]);
          const float2 o = round_f16x2(__fmul_rn((float)(int)v[e], i8_scale(__fmul_rn(sca, sc.x))), __fmul_rn((float)(int)v[e + 1], i8_scale(__fmul_rn(sca, sc.y))));
          out[e] = o.x;
          out[e + 1] = o.y;
        }
        if (p.bias) {
#pragma unroll
          for (int e = 0; e < 16; e += 2) {
            const float2 b = *reinterpret_cast<const float2*>(&s_feat[1][c0 + e]);
            const float2 o = round_f16x2(out[e] + b.x, out[e + 1] + b.y);
            out[e] = o.x;
            out[e + 1] = o.y;
          }
        }
        if (no > 0) {
          float sub[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) sub[e] = 0.f;
          auto add = [&](int j0, const float (&xv)[8], const float* rows, int ld) {   // ascending columns
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              if (j0 + j < no) {
#pragma unroll
                for (int e = 0; e < 16; e += 4) {
                  const float4 w = *reinterpret_cast<const float4*>(rows + j * ld + e);
                  sub[e] = fmaf(xv[j], w.x, sub[e]);
                  sub[e + 1] = fmaf(xv[j], w.y, sub[e + 1]);
                  sub[e + 2] = fmaf(xv[j], w.z, sub[e + 2]);
                  sub[e + 3] = fmaf(xv[j], w.w, sub[e + 3]);
                }
              }
            }
          };
          add(0, x0, &s_feat[2][c0], BN);
          for (int j0 = 8; j0 < no; j0 += 8) {
            const int f = lane & 15;
            const int64_t n = n0 + c0 + f;
            const bool nok = n < p.N;
            const float ws = __fdiv_rn(s_feat[0][c0 + f], 127.0f);
            const int8_t* const cb = p.cb + (nok ? n : 0) * p.K;
            float xv[8], w[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const int k = j0 + j < no ? p.idx[j0 + j] : 0;
              xv[j] = j0 + j < no ? __half2float(xr[k]) : 0.f;
              w[j] = j0 + j < no ? (float)cb[k] : 0.f;
            }
            __syncwarp();
            if (lane < 16) {
#pragma unroll
              for (int j = 0; j < 8; ++j) more[j][lane] = round_f16(__fmul_rn(w[j], ws));
            }
            __syncwarp();
            add(j0, xv, &more[0][0], 16);
          }
#pragma unroll
          for (int e = 0; e < 16; e += 2) {
            const float2 r = round_f16x2(sub[e], sub[e + 1]);
            out[e] += r.x;      // rounded by the store
            out[e + 1] += r.y;
          }
        }
        if (mok) {
          __half* const yr = p.y + m * p.N + n0 + c0;
          if (vec) {
#pragma unroll
            for (int e = 0; e < 16; e += 8) {
              if (n0 + c0 + e < p.N) {
                uint32_t o[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  const __half2 h = __floats2half2_rn(out[e + 2 * i], out[e + 2 * i + 1]);
                  o[i] = *reinterpret_cast<const uint32_t*>(&h);
                }
                *reinterpret_cast<uint4*>(yr + e) = make_uint4(o[0], o[1], o[2], o[3]);
              }
            }
          } else {
#pragma unroll
            for (int e = 0; e < 16; ++e)
              if (n0 + c0 + e < p.N) yr[e] = __float2half_rn(out[e]);
          }
        }
        __syncwarp();   // (the next load of tensor memory wants the whole warp, lanes without a row too)
      }
      tc::fence_before();
      __syncwarp();
      if (lane == 0) {
        if constexpr (PAIR) tc::mbar_arrive_at(tc::at_rank(acc_empty + 8 * acc, 0));
        else tc::mbar_arrive(acc_empty + 8 * acc);
      }
      acc ^= 1;
      if (acc == 0) ph ^= 1u;
    }
  }
  if (!ok) *err = 1u;
  tc::fence_before();
  if constexpr (PAIR) tc::cluster_sync();   // the other CTA's shared memory is read until its last product
  __syncthreads();
  if (warp == kI8EpiWarps) {
    __syncwarp();
    if constexpr (PAIR) tc::tmem_free_pair<2 * BN>(tmem);
    else tc::tmem_free<2 * BN>(tmem);
  }
}

// Features of a pair's tile: a round of tiles takes about 235 + bn for each k-block, so that fewer features pay where they cost no further round.  us of the
// whole call at 256, 224, 192, 160, 128, 64 features, six outlier columns: 4096 -> 11008 at 777 rows (3, 3, 4, 4, 5, 10 rounds) 64.5, 62.7, 69.9, 67.8, 72.4, 111;
// 4096 -> 12288 at 512 rows (2, 2, 2, 3, 3, 6) 51.7, 50.1, 47.8, 58.1, 54.4, 79.6; 4096 -> 4096 at 200 rows (all 1) 32.3, 31.6, 29.8, 29.2, 27.9, 26.6.
// A CTA alone (up to 128 rows) keeps 128: with 64 it is 2 us shorter at 4096 features and 4 to 9 longer from 6144 on.
static int i8_features(int64_t N, int64_t row_tiles, int64_t pairs) {
  int best = 256;
  int64_t best_t = -1;
  for (int bn = 256; bn >= 64; bn -= 32) {
    const int64_t t = (row_tiles * ((N + bn - 1) / bn) + pairs - 1) / pairs * (235 + bn);
    if (best_t < 0 || t < best_t) { best_t = t; best = bn; }
  }
  return best;
}

template <bool PAIR>
static cudaError_t launch_i8_gemm(const I8Params& p, cudaStream_t st) {
  static PerDeviceOnce once;
  if (once.need()) {
    const cudaError_t e = cudaFuncSetAttribute(int8_gemm_kernel<PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, kI8Smem);
    if (e != cudaSuccess) return e;
    once.done();
  }
  constexpr int CTAS = PAIR ? 2 : 1, BM = 128 * CTAS;
  const int64_t most = sm_count() / CTAS;
  const int mt = (int)((p.M + BM - 1) / BM), bn = PAIR ? i8_features(p.N, mt, most) : BM, nt = (int)((p.N + bn - 1) / bn);
  const int64_t tiles = (int64_t)mt * nt;
  alignas(64) CUtensorMap ma, mb;
  if (!tensor_map_2d(&ma, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, p.ca, p.M, p.K, p.K, 128) || !tensor_map_2d(&mb, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, p.cb, p.N, p.K, p.K, bn / CTAS))
    return cudaErrorInvalidValue;
  const dim3 grid((unsigned)((tiles < most ? tiles : most) * CTAS));
  unsigned* const err = wait_error_word();
  if (!err) return cudaErrorMemoryAllocation;
  return launch_cluster(int8_gemm_kernel<PAIR>, grid, dim3(kI8GemmThreads), CTAS, (size_t)kI8Smem, st, p, ma, mb, mt, nt, bn, err);
}

}  // namespace b200

using namespace b200;

extern "C" {

int b200_quantize_int8(const void* w, int w_dtype, int64_t N, int64_t K, int8_t* cb, float* scb, b200_stream_t stream) {
  B200_CHECK_ARG(w && cb && scb, "b200_quantize_int8: null pointer");
  B200_CHECK_ARG(N > 0 && K > 0 && N <= 0x7fffffffLL, "b200_quantize_int8: bad shape (N=%lld K=%lld)", (long long)N, (long long)K);
  cudaStream_t st = (cudaStream_t)stream;
  cudaError_t e;
  if (w_dtype == B200_BF16) e = launch(quantize_int8_rows_kernel<__nv_bfloat16>, dim3((unsigned)N), dim3(256), 0, st, (const __nv_bfloat16*)w, K, cb, scb);
  else if (w_dtype == B200_F16) e = launch(quantize_int8_rows_kernel<__half>, dim3((unsigned)N), dim3(256), 0, st, (const __half*)w, K, cb, scb);
  else if (w_dtype == B200_F32) e = launch(quantize_int8_rows_kernel<float>, dim3((unsigned)N), dim3(256), 0, st, (const float*)w, K, cb, scb);
  else { set_error("b200_quantize_int8: bad dtype code %d", w_dtype); return B200_ERR_INVALID; }
  if (e != cudaSuccess) { set_error("b200_quantize_int8: launch failed: %s", cudaGetErrorString(e)); return B200_ERR_CUDA; }
  return B200_OK;
}

int b200_dequantize_int8(const int8_t* cb, const float* scb, int64_t N, int64_t K, void* out, int out_dtype, b200_stream_t stream) {
  B200_CHECK_ARG(cb && scb && out, "b200_dequantize_int8: null pointer");
  B200_CHECK_ARG(N > 0 && K > 0, "b200_dequantize_int8: bad shape");
  cudaStream_t st = (cudaStream_t)stream;
  const dim3 grid((unsigned)((N * K + 255) / 256));
  cudaError_t e;
  if (out_dtype == B200_BF16) e = launch(dequantize_int8_rows_kernel<__nv_bfloat16>, grid, dim3(256), 0, st, cb, scb, N, K, (__nv_bfloat16*)out);
  else if (out_dtype == B200_F16) e = launch(dequantize_int8_rows_kernel<__half>, grid, dim3(256), 0, st, cb, scb, N, K, (__half*)out);
  else if (out_dtype == B200_F32) e = launch(dequantize_int8_rows_kernel<float>, grid, dim3(256), 0, st, cb, scb, N, K, (float*)out);
  else { set_error("b200_dequantize_int8: bad dtype code %d", out_dtype); return B200_ERR_INVALID; }
  if (e != cudaSuccess) { set_error("b200_dequantize_int8: launch failed: %s", cudaGetErrorString(e)); return B200_ERR_CUDA; }
  return B200_OK;
}

size_t b200_linear_int8_workspace_bytes(int64_t M, int64_t K) {
  // flags int32[K] | idx int32[K] | count (16 B) | sca fp32[M] (padded to 16) | ca int8[M * K]
  return (size_t)K * 8 + 16 + (((size_t)M * 4 + 15) & ~(size_t)15) + (size_t)M * K;
}

int b200_linear_int8(const b200_linear_int8_args* a, b200_stream_t stream) {
  B200_CHECK_ARG(a != nullptr, "b200_linear_int8: null args");
  B200_CHECK_WAITS("b200_linear_int8");
  B200_CHECK_ARG(a->x && a->cb && a->scb && a->y && a->workspace, "b200_linear_int8: null x/cb/scb/y/workspace pointer");
  B200_CHECK_ARG(a->M > 0 && a->N > 0 && a->K > 0, "b200_linear_int8: M, N, K must be positive");
  B200_CHECK_ARG(a->workspace_bytes >= b200_linear_int8_workspace_bytes(a->M, a->K), "b200_linear_int8: workspace too small (%zu < %zu)",
                 a->workspace_bytes, b200_linear_int8_workspace_bytes(a->M, a->K));
  B200_CHECK_ARG(((reinterpret_cast<uintptr_t>(a->x) | reinterpret_cast<uintptr_t>(a->cb) | reinterpret_cast<uintptr_t>(a->workspace)) & 15) == 0,
                 "b200_linear_int8: x / cb / workspace must be 16-byte aligned");
  if (a->K % 64 != 0) {
    set_error("b200_linear_int8: K must be a multiple of 64 (got %lld)", (long long)a->K);
    return B200_ERR_UNSUPPORTED;
  }
  B200_CHECK_ARG((a->M + 63) / 64 <= 65535, "b200_linear_int8: too many activation rows for the grid");
  uint8_t* ws = reinterpret_cast<uint8_t*>(a->workspace);
  int* flags = reinterpret_cast<int*>(ws);
  int* idx = flags + a->K;
  int* count = idx + a->K;
  float* sca = reinterpret_cast<float*>(ws + (size_t)a->K * 8 + 16);
  int8_t* ca = reinterpret_cast<int8_t*>(ws + (size_t)a->K * 8 + 16 + (((size_t)a->M * 4 + 15) & ~(size_t)15));
  const __half* x = reinterpret_cast<const __half*>(a->x);
  cudaStream_t st = (cudaStream_t)stream;
  const int block_rows = a->M <= 8 * 65535 ? 8 : 64;   // eight loads in flight per thread, as many CTAs as the grid allows
  const dim3 fg((unsigned)((a->K / 8 + 127) / 128), (unsigned)((a->M + block_rows - 1) / block_rows));
  cudaError_t e = fg.y > 1 ? cudaMemsetAsync(flags, 0, (size_t)a->K * sizeof(int), st) : cudaSuccess;
  if (e == cudaSuccess) e = launch(int8_outlier_flags_kernel, fg, dim3(128), 0, st, x, a->M, a->K, a->threshold, block_rows, flags);
  if (e == cudaSuccess) e = launch(int8_rowquant_kernel, dim3((unsigned)a->M + 1), dim3(256), 0, st, x, a->K, (const int*)flags, ca, sca, idx, count);
  I8Params p{};
  p.cb = reinterpret_cast<const int8_t*>(a->cb);
  p.scb = reinterpret_cast<const float*>(a->scb);
  p.x = x; p.ca = ca; p.sca = sca; p.idx = idx; p.count = count;
  p.bias = reinterpret_cast<const __half*>(a->bias);
  p.y = reinterpret_cast<__half*>(a->y);
  p.M = a->M; p.N = a->N; p.K = a->K;
  if (e == cudaSuccess) {
    const dim3 gv((unsigned)((a->N + 15) / 16));
    if (a->M <= 8) e = launch(int8_gemv_kernel<1>, gv, dim3(kI8Threads), 0, st, p);
    else if (a->M <= 16) e = launch(int8_gemv_kernel<2>, gv, dim3(kI8Threads), 0, st, p);
    else e = a->M > 128 ? launch_i8_gemm<true>(p, st) : launch_i8_gemm<false>(p, st);
  }
  if (e != cudaSuccess) {
    set_error("b200_linear_int8: launch failed: %s", cudaGetErrorString(e));
    return B200_ERR_CUDA;
  }
  return B200_OK;
}

}  // extern "C"
