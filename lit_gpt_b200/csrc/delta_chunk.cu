// Gated delta rule over prompts, 32 tokens at a time (delta.cu walks the same recurrence token by token and serves everything else).
//
//   per token:  S <- g S;  u = beta (v - S^T k);  S <- S + k u^T;  o = S^T q          (g per head, or per head and key channel)
//
// Within a chunk that starts from state S0, with R_ij = g_{j+1} ... g_i (per channel) and P_i = g_0 ... g_i, the writes u_i solve the lower
// triangular system u_i + beta_i sum_{j<i} A_ij u_j = beta_i (v_i - (P_i k_i)^T S0), A_ij = sum_c k_i R_ij k_j.  Its solution is linear in S0:
//   u = U - W S0,   o = O + Q S0,   S' = P S0 + K^T u       with   Q = (P q) - B W,  O = B U,  B_ij = sum_c q_i R_ij k_j (j <= i),  K_j = R_Cj k_j
// so everything but S0 is computed for all chunks side by side (delta_chunk_kernel), and what is left to do in order per chunk is three
// small products on a slice of S0's columns (delta_carry_kernel; the columns never mix).
//
// All of it is fp32.  The decays enter as running products, as in the token-by-token walk: no logarithm or quotient is taken, so any decay
// in [0, 1] is safe.  W, U come from the forward substitution in token order.
//
// Bound: the carry's chain of chunks, three products and as many barriers each, and the per-chunk work, which fills the GPU.  The walk of
// delta.cu costs 0.4 us (one decay per head) to 0.65 us (per channel) a token whatever the width: a layer of 16 heads of 128 x 128 with
// decays per channel takes 1413 us for 2048 tokens with it and 467 us with this one.
#include "tc05.cuh"

namespace b200 {

namespace {

constexpr int kDcC = 32;            // tokens per chunk
constexpr int kDcThreads = 128;
constexpr int kDcMinRows = 64;

struct DcArgs {
  const float* q; const float* k; const float* v;
  int64_t ldq, ldk, ldv;
  const void* beta_in; int64_t ld_beta;
  const void* decay_in; int64_t ld_decay;
  const void* a_log; const void* dt_bias;
  float* state; int64_t state_slot_stride;
  float* out; int64_t ldo;
  const int4* seqs;
  int heads, kv_heads, dk, dv;
  int n_seqs, longs, min_rows;      // sequences, how many of them can have chunks, and from how many rows on they have
  int item0, n_items, most;         // this launch's chunks, counted through all sequences, of `most` in all
  int dvb;                          // blocks of eight value columns (an even number)
  float* ws; int64_t item;          // per (chunk, head): W | K | Q, rows of DK + 4 | P (DK) | U [dvb][32][8] | O [dvb][32][8]
  unsigned* err;
};

template <int DK>
struct DcItem {
  static constexpr int kPitch = DK + 4, kMat = kDcC * kPitch, kHead = 3 * kMat + DK;   // floats; rows four floats apart in their banks
};

typedef unsigned long long f2;   // two packed floats
__device__ __forceinline__ f2 pk2(float a, float b) { f2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ void un2(f2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) { f2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ f2 mul2(f2 a, f2 b) { f2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ float sum2(f2 v) { float a, b; un2(v, a, b); return a + b; }

__device__ __forceinline__ float dc_softplus(float x) { return x > 20.0f ? x : log1pf(expf(x)); }

// Chunks are counted through the sequences in their order, each with as many as its rows take; among several sequences, those of fewer than
// kDcMinRows have none and go token by token.  (A single one always has a chunk, which without rows keeps or clears the slot's state as the walk
// would.)  The functions below are called by whole warps.
__device__ __forceinline__ int dc_chunks(const DcArgs& A, const int4& sq) { return sq.y >= A.min_rows ? (max(sq.y, 1) + kDcC - 1) / kDcC : 0; }
// the sequence of chunk `at` and the chunk's number there; -1: there are not that many
__device__ __forceinline__ int dc_find(const DcArgs& A, int at, int& chunk) {
  const int lane = threadIdx.x & 31;
  int before = 0;
  for (int s0 = 0; s0 < A.n_seqs; s0 += 32) {
    const int n = s0 + lane < A.n_seqs ? dc_chunks(A, A.seqs[s0 + lane]) : 0;
    int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    const unsigned past = __ballot_sync(0xffffffffu, before + incl > at);
    if (past) {
      const int w = __ffs(past) - 1;
      chunk = at - before - __shfl_sync(0xffffffffu, incl - n, w);
      return s0 + w;
    }
    before += __shfl_sync(0xffffffffu, incl, 31);
  }
  return -1;
}
// the z-th of the sequences that have chunks, and how many chunks lie before its own; -1: there are not that many
__device__ __forceinline__ int dc_nth(const DcArgs& A, int z, int& before) {
  const int lane = threadIdx.x & 31;
  before = 0;
  for (int s0 = 0; s0 < A.n_seqs; s0 += 32) {
    const int n = s0 + lane < A.n_seqs ? dc_chunks(A, A.seqs[s0 + lane]) : 0;
    const unsigned have = __ballot_sync(0xffffffffu, n > 0);
    if (z < __popc(have)) {
      const int w = (int)__fns(have, 0, z + 1);
      before += __reduce_add_sync(0xffffffffu, lane < w ? n : 0);
      return s0 + w;
    }
    z -= __popc(have);
    before += __reduce_add_sync(0xffffffffu, n);
  }
  return -1;
}

// One chunk of one head: grid (chunks, heads).  Tokens past the sequence's end count as k = q = v = 0, beta = 0, g = 1.
template <typename T, int DK, bool CHANNEL>
__global__ void __launch_bounds__(kDcThreads, 2) delta_chunk_kernel(DcArgs A, int vec) {
  using I = DcItem<DK>;
  constexpr int C = kDcC, CPW = DK / 4;                 // channels per warp
  extern __shared__ __align__(128) float dc_smem[];
  float* const ks = dc_smem;                            // [C][DK]
  float* const qs = ks + C * DK;                        // [C][DK]
  float* const gs = qs + C * DK;                        // [C][DK] (per channel) or [C]
  float* const bs = gs + (CHANNEL ? C * DK : C);        // [C]
  float* const part = bs + C;                           // [4 warps][A, B][C][C]
  float2* const a2 = reinterpret_cast<float2*>(part + 8 * C * C);   // [C][C]  -beta_i A_ij, twice
  float2* const b2 = a2 + C * C;                                    // [C][C]  B_ij, twice
  griddep_launch();
  griddep_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int h = blockIdx.y, hk = h / (A.heads / A.kv_heads);
  int chunk;
  const int z = dc_find(A, A.item0 + (int)blockIdx.x, chunk);
  if (z < 0) return;
  const int4 sq = A.seqs[z];
  const int t0 = chunk * C;
  const int nt = min(C, sq.y - t0);
  const int64_t row0 = (int64_t)sq.x + t0;
  const int dk = A.dk, dv = A.dv;
  float* const item = A.ws + ((int64_t)blockIdx.x * A.heads + h) * A.item;

  // ---- the chunk's keys, queries, decays and write strengths ----
  const float* const kp = A.k + row0 * A.ldk + (int64_t)hk * dk;
  const float* const qp = A.q + row0 * A.ldq + (int64_t)hk * dk;
#pragma unroll 4
  for (int i = tid * 4; i < C * DK; i += kDcThreads * 4) {
    const int t = i / DK, c = i % DK;
    float4 kv = make_float4(0.f, 0.f, 0.f, 0.f), qv = kv;
    if (t < nt && c < dk) {
      if (vec) {
        kv = *reinterpret_cast<const float4*>(kp + (int64_t)t * A.ldk + c);
        qv = *reinterpret_cast<const float4*>(qp + (int64_t)t * A.ldq + c);
      } else {
        float a[4] = {0.f, 0.f, 0.f, 0.f}, b[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (c + e < dk) { a[e] = kp[(int64_t)t * A.ldk + c + e]; b[e] = qp[(int64_t)t * A.ldq + c + e]; }
        kv = make_float4(a[0], a[1], a[2], a[3]);
        qv = make_float4(b[0], b[1], b[2], b[3]);
      }
    }
    *reinterpret_cast<float4*>(ks + i) = kv;
    *reinterpret_cast<float4*>(qs + i) = qv;
  }
  const float neg_a = -expf(load_as_float(reinterpret_cast<const T*>(A.a_log), h));
  const T* const bias = reinterpret_cast<const T*>(A.dt_bias);
  const T* const dec = reinterpret_cast<const T*>(A.decay_in);
  if constexpr (CHANNEL) {
#pragma unroll 4
    for (int i = tid; i < C * DK; i += kDcThreads) {
      const int t = i / DK, c = i % DK;
      float g = 1.f;
      if (t < nt && c < dk) g = expf(neg_a * dc_softplus(load_as_float(dec, (row0 + t) * A.ld_decay + (int64_t)h * dk + c) + load_as_float(bias, (int64_t)h * dk + c)));
      gs[i] = g;
    }
  } else if (tid < C) {
    gs[tid] = tid < nt ? expf(neg_a * dc_softplus(load_as_float(dec, (row0 + tid) * A.ld_decay + h) + load_as_float(bias, h))) : 1.f;
  }
  if (tid < C) bs[tid] = tid < nt ? 1.0f / (1.0f + expf(-load_as_float(reinterpret_cast<const T*>(A.beta_in), (row0 + tid) * A.ld_beta + h))) : 0.f;
  __syncthreads();

  // ---- A and B: lane j carries R_ij k_j in this warp's channels from token to token ----
  {
    f2 r[CPW / 2];
    float rs = 0.f;
#pragma unroll
    for (int p = 0; p < CPW / 2; ++p) r[p] = 0ull;
    if constexpr (!CHANNEL) {
#pragma unroll
      for (int p = 0; p < CPW / 2; ++p) r[p] = *reinterpret_cast<const f2*>(ks + lane * DK + warp * CPW + 2 * p);
    }
#pragma unroll 1
    for (int i = 0; i < C; ++i) {
      const int at = i * DK + warp * CPW;
      f2 a = 0ull, b = 0ull, a_ = 0ull, b_ = 0ull;
#pragma unroll
      for (int p = 0; p < CPW / 2; p += 2) {
        const ulonglong2 kk = *reinterpret_cast<const ulonglong2*>(ks + at + 2 * p), qq = *reinterpret_cast<const ulonglong2*>(qs + at + 2 * p);
        if constexpr (CHANNEL) {
          const ulonglong2 gg = *reinterpret_cast<const ulonglong2*>(gs + at + 2 * p);
          r[p] = lane == i ? kk.x : mul2(r[p], gg.x);
          r[p + 1] = lane == i ? kk.y : mul2(r[p + 1], gg.y);
        }
        a = fma2(kk.x, r[p], a);
        b = fma2(qq.x, r[p], b);
        a_ = fma2(kk.y, r[p + 1], a_);
        b_ = fma2(qq.y, r[p + 1], b_);
      }
      float sa = sum2(a) + sum2(a_), sb = sum2(b) + sum2(b_);
      if constexpr (!CHANNEL) {
        rs = lane == i ? 1.f : rs * gs[i];
        sa *= rs;
        sb *= rs;
      }
      part[(warp * 2 * C + i) * C + lane] = sa;
      part[(warp * 2 * C + C + i) * C + lane] = sb;
    }
    // K: what the write of token j leaves at the chunk's end
    float* const kh = item + I::kMat + lane * I::kPitch + warp * CPW;
#pragma unroll
    for (int p = 0; p < CPW / 2; p += 2) {
      const f2 m = CHANNEL ? 0ull : pk2(rs, rs);
      *reinterpret_cast<ulonglong2*>(kh + 2 * p) = CHANNEL ? make_ulonglong2(r[p], r[p + 1]) : make_ulonglong2(mul2(r[p], m), mul2(r[p + 1], m));
    }
  }
  __syncthreads();
  for (int i = tid; i < C * C; i += kDcThreads) {
    const int t = i / C, j = i % C;
    float sa = 0.f, sb = 0.f;
#pragma unroll
    for (int w = 0; w < 4; ++w) { sa += part[w * 2 * C * C + i]; sb += part[(w * 2 + 1) * C * C + i]; }
    const float a = j < t ? -bs[t] * sa : 0.f, b = j <= t ? sb : 0.f;
    a2[i] = make_float2(a, a);
    b2[i] = make_float2(b, b);
  }
  // ---- decays from the chunk's start: k becomes beta P k (the right-hand side of W), q becomes P q ----
  for (int c = tid; c < DK; c += kDcThreads) {
    float cum = 1.f;
#pragma unroll 4
    for (int i = 0; i < C; ++i) {
      cum *= CHANNEL ? gs[i * DK + c] : gs[i];
      ks[i * DK + c] *= bs[i] * cum;
      qs[i * DK + c] *= cum;
    }
    item[3 * I::kMat + c] = cum;
  }
  __syncthreads();

  // ---- forward substitution, two columns per thread: the columns of W, then those of U ----
  float* const uo = item + I::kHead;
  const int64_t o_off = (int64_t)A.dvb * C * 8;
  const int pairs = DK / 2 + A.dvb * 4;
  for (int p = tid; p < pairs; p += kDcThreads) {
    const bool is_w = p < DK / 2;
    const int vc = 2 * (p - DK / 2);
    f2 x[C];
    if (is_w) {
#pragma unroll
      for (int i = 0; i < C; ++i) x[i] = *reinterpret_cast<const f2*>(ks + i * DK + 2 * p);
    } else {
      const float* vp = A.v + row0 * A.ldv + (int64_t)h * dv + vc;
#pragma unroll
      for (int i = 0; i < C; ++i) {
        const float b = bs[i];
        x[i] = pk2(i < nt && vc < dv ? b * vp[(int64_t)i * A.ldv] : 0.f, i < nt && vc + 1 < dv ? b * vp[(int64_t)i * A.ldv + 1] : 0.f);
      }
    }
#pragma unroll
    for (int i = 1; i < C; ++i) {
#pragma unroll
      for (int j = 0; j + 1 < i; j += 2) {
        const ulonglong2 m = *reinterpret_cast<const ulonglong2*>(a2 + i * C + j);
        x[i] = fma2(m.x, x[j], x[i]);
        x[i] = fma2(m.y, x[j + 1], x[i]);
      }
      if (i & 1) x[i] = fma2(*reinterpret_cast<const f2*>(a2 + i * C + i - 1), x[i - 1], x[i]);
    }
    float* const dst = is_w ? item + 2 * p : uo + (int64_t)(vc >> 3) * C * 8 + (vc & 7);
    const int pitch = is_w ? I::kPitch : 8;
#pragma unroll
    for (int i = 0; i < C; ++i) *reinterpret_cast<f2*>(dst + i * pitch) = x[i];
#pragma unroll
    for (int i = 0; i < C; ++i) {
      f2 y = 0ull, z = 0ull;
#pragma unroll
      for (int j = 0; j < i; j += 2) {   // pairs (j, j + 1); the last pair of an odd row ends with B_ii
        const ulonglong2 m = *reinterpret_cast<const ulonglong2*>(b2 + i * C + j);
        y = fma2(m.x, x[j], y);
        z = fma2(m.y, x[j + 1], z);
      }
      if (!(i & 1)) y = fma2(*reinterpret_cast<const f2*>(b2 + i * C + i), x[i], y);
      float y0, y1, z0, z1;
      un2(y, y0, y1);
      un2(z, z0, z1);
      y0 += z0;
      y1 += z1;
      if (is_w) {
        const float2 qh = *reinterpret_cast<const float2*>(qs + i * DK + 2 * p);
        *reinterpret_cast<float2*>(dst + 2 * I::kMat + i * pitch) = make_float2(qh.x - y0, qh.y - y1);
      } else {
        *reinterpret_cast<float2*>(dst + o_off + i * pitch) = make_float2(y0, y1);
      }
    }
  }
}

// The state through the chunks, in order: grid (slices of NC value columns, heads, sequences that can have chunks), 16 NC threads.  Chunk c + 1 is on its way into
// the second stage (bulk copies) while chunk c is worked on; the slice of S lies in shared memory by column, so that four keys' numbers are
// one access for either factor of W S and Q S.
template <int DK, int NC>
struct DcCarry {
  using I = DcItem<DK>;
  static constexpr int kThreads = 16 * NC;
  static constexpr int kSlice = kDcC * NC;                         // floats of U (of O) per chunk and slice
  static constexpr int kStage = I::kHead + 2 * kSlice;             // floats
  static constexpr int kFloats = 2 * kStage + NC * I::kPitch + 8 * (kThreads / 2) + 2 * kDcC * NC;
  static constexpr int kSmem = kFloats * 4;
};

template <int DK, int NC>
__global__ void __launch_bounds__(16 * NC) delta_carry_kernel(DcArgs A, int L) {
  using I = DcItem<DK>;
  using Y = DcCarry<DK, NC>;
  constexpr int C = kDcC, PT = I::kPitch, TILES = Y::kThreads / 2, CG = NC / 4;
  extern __shared__ __align__(128) float dc_smem[];
  float* const st = dc_smem + 2 * Y::kStage;            // S by column: [NC][DK + 4]
  float* const red = st + NC * PT;                      // [2][TILES] float4: the second half's sums
  float2* const u2 = reinterpret_cast<float2*>(red + 8 * TILES);   // [C][NC] u, twice
  __shared__ __align__(8) uint64_t s_full[2];
  const int tid = threadIdx.x, h = blockIdx.y, col0 = (int)blockIdx.x * NC;
  const uint32_t full = tc::smem_u32(s_full);
  if (tid == 0) {
    tc::mbar_init(full, 1);
    tc::mbar_init(full + 8, 1);
    tc::mbar_init_fence();
  }
  griddep_launch();
  griddep_wait();
  int before;
  const int z = dc_nth(A, blockIdx.z, before);
  if (z < 0) return;
  const int4 sq = A.seqs[z];
  const int all = dc_chunks(A, sq);
  const int c_first = max(0, A.item0 - before), chunks = min(all, A.item0 + A.n_items - before) - c_first, t_first = c_first * C;
  if (tid == 0 && before + all > A.most) *A.err = 1u;   // more rows than the caller said
  if (chunks <= 0) return;
  const int dk = A.dk, dv = A.dv;
  const float* const items = A.ws + ((int64_t)(before + c_first - A.item0) * A.heads + h) * A.item;
  const int64_t step = (int64_t)A.heads * A.item;

  auto fetch = [&](int c) {   // one thread
    const float* src = items + c * step;
    const uint32_t bar = full + 8 * (c & 1), dst = tc::smem_u32(dc_smem + (c & 1) * Y::kStage);
    tc::mbar_expect_tx(bar, Y::kStage * 4);
    auto copy = [&](uint32_t to, const float* from, uint32_t bytes) {
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(to), "l"(from), "r"(bytes), "r"(bar) : "memory");
    };
    copy(dst, src, I::kHead * 4);
    copy(dst + I::kHead * 4, src + I::kHead + (int64_t)(col0 >> 3) * C * 8, Y::kSlice * 4);
    copy(dst + (I::kHead + Y::kSlice) * 4, src + I::kHead + (int64_t)(A.dvb + (col0 >> 3)) * C * 8, Y::kSlice * 4);
  };
  if (tid == 0) {
    fetch(0);
    if (chunks > 1) fetch(1);
  }
  const int krows = (dk + L - 1) / L;
  float* const slot = A.state + (int64_t)sq.w * A.state_slot_stride + (int64_t)h * krows * L * dv;
  const bool from_slot = sq.z > 0 || c_first > 0;
  for (int i = tid; i < DK * NC; i += Y::kThreads) {
    const int n = i % NC, c = i / NC;
    st[n * PT + c] = from_slot && c < dk && col0 + n < dv ? slot[((int64_t)(c / L) * dv + col0 + n) * L + c % L] : 0.f;
  }
  // W S and Q S: a thread has row `rp` of both, columns cg + CG {0 .. 3}, half of the keys
  const int half = tid / TILES, tile = tid % TILES, cg = tile % CG, rp = tile / CG;
  // K^T u: four keys, two columns
  const int kc = (tid % (DK / 4)) * 4, n0 = (tid / (DK / 4)) * 2;
  constexpr int NSTEP = Y::kThreads / (DK / 4) * 2;    // columns covered at a time
  bool ok = true;
  __syncthreads();
  for (int c = 0; c < chunks; ++c) {
    const float* const sg = dc_smem + (c & 1) * Y::kStage;
    ok = __syncthreads_and(tc::mbar_wait(full + 8 * (c & 1), (uint32_t)(c >> 1) & 1u)) != 0;
    if (!ok) {   // given up: let the copies of this and the next chunk land before leaving
      if (tid == 0) {
        tc::mbar_wait(full + 8 * (c & 1), (uint32_t)(c >> 1) & 1u);
        if (c + 1 < chunks) tc::mbar_wait(full + 8 * ((c + 1) & 1), (uint32_t)((c + 1) >> 1) & 1u);
      }
      break;
    }
    {
      f2 w[4], o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) w[e] = o[e] = 0ull;
      const float* const wr = sg + rp * PT + half * (DK / 2);
      const float* const qr = wr + 2 * I::kMat;
      const float* const sc = st + cg * PT + half * (DK / 2);
#pragma unroll 4
      for (int k = 0; k < DK / 2; k += 4) {
        const ulonglong2 w4 = *reinterpret_cast<const ulonglong2*>(wr + k), q4 = *reinterpret_cast<const ulonglong2*>(qr + k);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const ulonglong2 s4 = *reinterpret_cast<const ulonglong2*>(sc + e * CG * PT + k);
          w[e] = fma2(w4.x, s4.x, w[e]);
          o[e] = fma2(q4.x, s4.x, o[e]);
          w[e] = fma2(w4.y, s4.y, w[e]);
          o[e] = fma2(q4.y, s4.y, o[e]);
        }
      }
      const float4 sw = make_float4(sum2(w[0]), sum2(w[1]), sum2(w[2]), sum2(w[3])), so = make_float4(sum2(o[0]), sum2(o[1]), sum2(o[2]), sum2(o[3]));
      float4* const rd = reinterpret_cast<float4*>(red);
      if (half == 1) {
        rd[tile] = sw;
        rd[TILES + tile] = so;
      }
      __syncthreads();
      if (half == 0) {
        const float4 a = rd[tile], b = rd[TILES + tile];
        const float uw[4] = {sw.x + a.x, sw.y + a.y, sw.z + a.z, sw.w + a.w}, oq[4] = {so.x + b.x, so.y + b.y, so.z + b.z, so.w + b.w};
        const int t = t_first + c * C + rp;
        float* const orow = A.out + ((int64_t)sq.x + t) * A.ldo + (int64_t)h * dv;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int n = cg + e * CG, at = I::kHead + (n >> 3) * C * 8 + rp * 8 + (n & 7);
          const float u = sg[at] - uw[e];
          u2[rp * NC + n] = make_float2(u, u);
          if (t < sq.y && col0 + n < dv) orow[col0 + n] = sg[at + Y::kSlice] + oq[e];
        }
      }
      __syncthreads();
    }
    {
      const float* const kr = sg + I::kMat + kc;
      const ulonglong2 p4 = *reinterpret_cast<const ulonglong2*>(sg + 3 * I::kMat + kc);
#pragma unroll
      for (int n = n0; n < NC; n += NSTEP) {
        float* const s0 = st + n * PT + kc;
        ulonglong2 a = *reinterpret_cast<const ulonglong2*>(s0), b = *reinterpret_cast<const ulonglong2*>(s0 + PT);
        a.x = mul2(a.x, p4.x); a.y = mul2(a.y, p4.y); b.x = mul2(b.x, p4.x); b.y = mul2(b.y, p4.y);
#pragma unroll 8
        for (int j = 0; j < C; ++j) {
          const ulonglong2 k4 = *reinterpret_cast<const ulonglong2*>(kr + j * PT), uu = *reinterpret_cast<const ulonglong2*>(u2 + j * NC + n);
          a.x = fma2(k4.x, uu.x, a.x); a.y = fma2(k4.y, uu.x, a.y);
          b.x = fma2(k4.x, uu.y, b.x); b.y = fma2(k4.y, uu.y, b.y);
        }
        *reinterpret_cast<ulonglong2*>(s0) = a;
        *reinterpret_cast<ulonglong2*>(s0 + PT) = b;
      }
    }
    __syncthreads();   // S complete, this stage free
    if (tid == 0 && c + 2 < chunks) fetch(c + 2);
  }
  if (!ok) *A.err = 1u;
  for (int i = tid; i < DK * NC; i += Y::kThreads) {
    const int n = i % NC, c = i / NC;
    if (c < krows * L && col0 + n < dv) slot[((int64_t)(c / L) * dv + col0 + n) * L + c % L] = c < dk ? st[n * PT + c] : 0.f;
  }
}

template <typename T, int DK, bool CHANNEL>
cudaError_t chunk_launch(const DcArgs& A, int vec, cudaStream_t st) {
  constexpr int C = kDcC;
  constexpr int smem = (2 * C * DK + (CHANNEL ? C * DK : C) + C + 8 * C * C + 4 * C * C) * 4;
  static PerDeviceOnce once;
  if (once.need()) {
    const cudaError_t e = cudaFuncSetAttribute(delta_chunk_kernel<T, DK, CHANNEL>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    once.done();
  }
  return launch(delta_chunk_kernel<T, DK, CHANNEL>, dim3((unsigned)A.n_items, (unsigned)A.heads), dim3(kDcThreads), smem, st, A, vec);
}

template <int DK, int NC>
cudaError_t carry_launch(const DcArgs& A, int L, cudaStream_t st) {
  using Y = DcCarry<DK, NC>;
  static PerDeviceOnce once;
  if (once.need()) {
    const cudaError_t e = cudaFuncSetAttribute(delta_carry_kernel<DK, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, Y::kSmem);
    if (e != cudaSuccess) return e;
    once.done();
  }
  return launch(delta_carry_kernel<DK, NC>, dim3((unsigned)((A.dv + NC - 1) / NC), (unsigned)A.heads, (unsigned)A.longs), dim3(Y::kThreads), Y::kSmem, st, A, L);
}

template <typename T, int DK>
cudaError_t segment_launch(const DcArgs& A, bool channel, int vec, int L, cudaStream_t st) {
  const cudaError_t e = channel ? chunk_launch<T, DK, true>(A, vec, st) : chunk_launch<T, DK, false>(A, vec, st);
  if (e != cudaSuccess) return e;
  // Slices of 8 columns: the shorter chain.  Slices of 16, which read W, Q and K half as often, are 2 - 60 % slower at every number of heads (512
  // rows, decays per channel, us with 8 and 16: 4 heads of 128 x 128 67 and 82, 16 heads 83 and 86, 32 heads 181 and 191; 16 heads of 64 x 128 62 and 94).
  return carry_launch<DK, 8>(A, L, st);
}

int dc_dvb(int dv) { return (dv + 15) / 16 * 2; }
int64_t dc_item(int dk, int dv) { return (dk <= 64 ? (int64_t)DcItem<64>::kHead : (int64_t)DcItem<128>::kHead) + 2 * (int64_t)dc_dvb(dv) * kDcC * 8; }

constexpr int64_t kDcMaxBytes = 256ll << 20;   // scratch of one launch's chunks

}  // namespace

int delta_rule_walk(const b200_delta_rule_args* a, int below, b200_stream_t stream);   // delta.cu

}  // namespace b200

using namespace b200;

extern "C" {

int b200_delta_rule_in_chunks(int64_t rows, int max_rows, int n_seqs, int heads, int dk, int dv, int channel_decay) {
  if (max_rows < kDcMinRows || rows < max_rows || n_seqs <= 0 || heads <= 0 || dk <= 0 || dk > 128 || dv <= 0) return 0;
  // us of either way, fitted to launches of 4 to 256 heads (times sequences of the longest one's length) of 128 x 128: a walk's token takes what its
  // chain of reductions takes until the heads fill the GPU, a chunk's as long as the carry's chain, and both the same work beyond; the short sequences'
  // walk comes on top of the chunks and runs half beside the long one's.  Measured, walk / chunks, 16 heads, 64, 128, 512 rows alone: decays per channel
  // 54 / 43, 104 / 49, 404 / 82; per head 28 / 31, 50 / 35, 181 / 69.  Beside 32 single rows: 76 / 104, 91 / 109, 316 / 159; 56 / 75, 66 / 80, 217 / 118.
  // 16 sequences of 64, of 256 rows: 207 / 245, 822 / 682; 145 / 202, 528 / 539.
  const double n = max_rows, same = (double)rows / max_rows < n_seqs ? (double)rows / max_rows : n_seqs, one = heads * (dk * (double)dv / 16384.0), load = one * same;
  const int64_t shorts = n_seqs - (rows + max_rows - 1) / max_rows;
  auto most = [](double a, double b) { return a > b ? a : b; };
  double walk, chunks, few;
  if (channel_decay) {
    const bool wide = (int64_t)heads * n_seqs * ((dv + 15) / 16) < sm_count() * 3 / 2;   // (delta_rule_walk's choice)
    walk = 5.0 + n * most(0.35, wide ? 0.17 + 0.038 * load : most(0.36 + 0.01 * load, 0.0126 * load));
    chunks = 28.0 + (n + 24.0) * most(0.1, 0.0114 * load);
    few = 0.13 * one;
  } else {
    walk = 5.0 + n * most(most(0.35, 0.25 + 0.0062 * load), 0.0088 * load);
    chunks = 20.0 + (n + 24.0) * most(0.085, 0.009 * load);
    few = 0.09 * one;
  }
  if (shorts > 0) {
    walk += 0.5 * few * shorts;
    chunks += few * shorts;
  }
  return chunks < walk;
}

size_t b200_delta_rule_workspace_bytes(int max_rows, int n_seqs, int heads, int dk, int dv) {
  if (max_rows < kDcMinRows || n_seqs <= 0 || heads <= 0 || dk <= 0 || dk > 128 || dv <= 0) return 0;
  const int64_t per_chunk = (int64_t)n_seqs * heads * dc_item(dk, dv) * 4;
  int64_t chunks = (max_rows + kDcC - 1) / kDcC;
  if (chunks * per_chunk > kDcMaxBytes) chunks = kDcMaxBytes / per_chunk;
  return chunks < 2 ? 0 : (size_t)(chunks * per_chunk);
}

int b200_delta_rule_chunked(const b200_delta_rule_args* a, void* workspace, size_t workspace_bytes, b200_stream_t stream) {
  B200_CHECK_ARG(a && a->q && a->k && a->v && a->beta_in && a->decay_in && a->a_log && a->dt_bias && a->state && a->out && a->seqs && workspace,
                 "b200_delta_rule_chunked: null pointer");
  B200_CHECK_WAITS("b200_delta_rule_chunked");
  B200_CHECK_ARG(a->n_seqs > 0 && a->n_seqs <= 65535 && a->heads > 0 && a->heads <= 65535 && a->kv_heads > 0 && a->heads % a->kv_heads == 0,
                 "b200_delta_rule_chunked: bad head counts");
  B200_CHECK_ARG(a->dk > 0 && a->dk <= 128 && a->dv > 0 && a->rows >= 0 && (a->rows > 0 || a->max_rows > 0),
                 "b200_delta_rule_chunked: key size must be 1 .. 128; the rows of all sequences (or the longest sequence's) are needed");
  B200_CHECK_ARG(((reinterpret_cast<uintptr_t>(a->seqs) | reinterpret_cast<uintptr_t>(workspace)) & 15) == 0,
                 "b200_delta_rule_chunked: seqs and workspace must be 16-byte aligned");
  const int64_t item = dc_item(a->dk, a->dv);
  int64_t fit = (int64_t)(workspace_bytes / (size_t)(item * 4)) / a->heads;   // chunks
  B200_CHECK_ARG(fit > 0, "b200_delta_rule_chunked: workspace too small (%zu bytes)", workspace_bytes);
  // n sequences of `rows` rows in all have at most (rows + 31 n) / 32 chunks, and n of them kDcMinRows rows each at least
  const int64_t longs = a->rows > 0 && a->rows / kDcMinRows < a->n_seqs ? a->rows / kDcMinRows : a->n_seqs;
  const int64_t most = a->rows > 0 ? (longs > 0 ? (a->rows + (kDcC - 1) * longs) / kDcC : 0) : longs * ((a->max_rows + kDcC - 1) / kDcC);
  B200_CHECK_ARG(most <= 0x3fffffff, "b200_delta_rule_chunked: too many rows");
  if (fit > most) fit = most;
  // In a step of several sequences the short ones -- single rows beside a prompt -- keep the walk: a row alone would cost a whole chunk and a link of
  // the carry.  One prompt of 1024 rows beside 32 single rows, 16 heads of 128 x 128 with decays per channel: 250 us; 494 with chunks for all, 679 with
  // the walk for all.
  if (a->n_seqs > 1 || most == 0) {
    b200_delta_rule_args few = *a;
    if (few.max_rows >= kDcMinRows) few.max_rows = kDcMinRows - 1;
    const int rc = delta_rule_walk(&few, kDcMinRows, stream);
    if (rc != B200_OK || most == 0) return rc;
  }
  DcArgs A{a->q, a->k, a->v, a->ldq, a->ldk, a->ldv, a->beta_in, a->ld_beta, a->decay_in, a->ld_decay, a->a_log, a->dt_bias, a->state, a->state_slot_stride,
           a->out, a->ldo, reinterpret_cast<const int4*>(a->seqs), a->heads, a->kv_heads, a->dk, a->dv, a->n_seqs, (int)longs, a->n_seqs > 1 ? kDcMinRows : 0, 0, (int)fit, (int)most, dc_dvb(a->dv),
           reinterpret_cast<float*>(workspace), item, wait_error_word()};
  B200_CHECK_ARG(A.err, "b200_delta_rule_chunked: no error word");
  auto al = [](const void* p, int64_t ld) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && ld % 4 == 0; };
  const int vec = a->dk % 4 == 0 && al(a->q, a->ldq) && al(a->k, a->ldk);
  const int L = a->dk <= 64 ? 4 : 8;   // the stored layout of a state (delta.cu)
  const bool ch = a->channel_decay != 0;
  cudaStream_t st = (cudaStream_t)stream;
  for (int64_t at = 0; at < most; at += fit) {
    A.item0 = (int)at;
    A.n_items = (int)(most - at < fit ? most - at : fit);
    B200_FLOAT_TYPES(a->dtype, T, {
      if (a->dk <= 64) B200_CUDA((segment_launch<T, 64>(A, ch, vec, L, st)));
      else B200_CUDA((segment_launch<T, 128>(A, ch, vec, L, st)));
    });
  }
  return B200_OK;
}

}  // extern "C"
