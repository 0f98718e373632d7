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
// All numbers are fp32 and products of them are formed on the tensor cores as three products of tf32 halves (tf32x3.cuh); those of T and B T with the
// right-hand sides, whose errors all results share, give back what the tensor core cuts off and keep the last bit of the right-hand sides, and B T itself is fp32
// multiply-adds.  The decays enter as running products, as in the token-by-token walk: no logarithm or quotient is taken, so any decay in [0, 1] is safe.
// Error against 64 bits, relative, 1e-7, mean of six shapes of 96 to 2048 tokens, read-out and state: this / every product as fp32 multiply-adds / token by token
//   decays per channel, q, k, v of either sign  2.37, 2.29 / 2.56, 2.64 / 2.38, 2.37    past a silu  1.57, 2.34 / 1.69, 2.66 / 1.52, 2.44    with a mean of 1  0.87, 2.45 / 0.94, 2.74 / 0.69, 2.60
//   decays per head                             2.26, 1.97 / 2.32, 2.27 / 2.17, 2.00                 1.63, 1.92 / 1.67, 2.21 / 1.46, 1.97                      1.01, 1.87 / 1.05, 2.04 / 0.74, 1.82
// (with plain products of halves everywhere, read-outs of numbers of one sign with decays per head 1.19).
//
// Bound: the chain of chunks (1.6 us each at sixteen columns a CTA, a third of it tensor pipe, the rest latency between its two products and three
// barriers), then the per-chunk work (two CTAs an SM; issue slots).  16 heads of 128 x 128 with decays per channel, 2048 tokens: 344 -> 209 us (chunks
// 155 -> 97, chain 180 -> 108) against all of it in fp32 multiply-adds read from shared memory, 1640 token by token.
#include "seq_pieces.cuh"
#include "tc05.cuh"
#include "tf32x3.cuh"

namespace b200 {

namespace {

constexpr int kDcC = 32;            // tokens per chunk
constexpr int kDcChunkThreads = 256;
constexpr int kDcMinRows = 64;

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) { return tc::mbar_wait<0>(bar, parity); }   // (a try's length: tc05.cuh)

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
  int dvb;                          // blocks of eight value columns (a multiple of four)
  float* ws; int64_t item;          // per (chunk, head): W | Q (32 rows of DK) | K by key (DK rows of 32) | P (DK) | U [dvb][32][8] | O [dvb][32][8]
  unsigned* err;
};

template <int DK>
struct DcItem {
  static constexpr int kMat = kDcC * DK, kHead = 3 * kMat + DK;   // floats
};

typedef unsigned long long f2;   // two packed floats
__device__ __forceinline__ void un2(f2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) { f2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ f2 mul2(f2 a, f2 b) { f2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ float sum2(f2 v) { float a, b; un2(v, a, b); return a + b; }

__device__ __forceinline__ float dc_softplus(float x) { return x > 20.0f ? x : log1pf(expf(x)); }

// Chunks are counted through the sequences (seq_pieces.cuh); among several sequences, those of fewer than kDcMinRows have none and go token by token.
// (A single one always has a chunk, which without rows keeps or clears the slot's state as the walk would.)
// One chunk of one head: grid (chunks, heads).  Tokens past the sequence's end count as k = q = v = 0, beta = 0, g = 1.
//
// The tokens form four blocks of eight.  Per channel, a decay from token j of an earlier block to token i is the product of the one from j to the end of
// its block, those of the blocks between, and the one from the start of i's block to i: the pairs of different blocks are then matrix products of scaled
// rows (16 rows of a tile: eight k, eight q), and only the pairs within a block walk the decays one by one.  With one decay per head all pairs are matrix
// products of the plain rows and the decay a factor of the result.  T = (1 + beta A)^-1 by forward substitution; W = T (beta P k), U = T (beta v), and
// B W, B U as (B T) times the same.
template <int DK>
struct DcChunk {
  static constexpr int NW = DK / 16;                     // warps with channels (sixteen each) in A and B
  static constexpr int kPart = 1280;                     // floats of a warp's share of A and B
  static constexpr int kPK = DK + 2, kPV = 130;          // pitches of the right-hand sides: the four tokens of a quarter warp on different banks
  static constexpr int kRhs = kDcC * (kPK + kPV);
  static constexpr int kScratch = NW * kPart > kRhs ? NW * kPart : kRhs;
  static constexpr int kFloats = 3 * kDcC * DK + kScratch + 4 * kDcC * kDcC + 4 * DK + 3 * kDcC;
  static constexpr int kSmem = kFloats * 4;
};

template <int DK>
__device__ __forceinline__ int dc_at(int row, int c) { return row * DK + ((((c >> 2) ^ (row >> 3) ^ ((row & 1) << 2)) << 2) | (c & 3)); }
__device__ __forceinline__ int dc_at32(int row, int c) { return row * kDcC + (x3::unit_row(row, c >> 2) << 2) + (c & 3); }

template <typename T, int DK, bool CHANNEL>
__global__ void __launch_bounds__(kDcChunkThreads, 2) delta_chunk_kernel(DcArgs A, int vec, int vec_v) {
  using I = DcItem<DK>;
  using Y = DcChunk<DK>;
  constexpr int C = kDcC, NT = kDcChunkThreads;
  extern __shared__ __align__(128) float dc_smem[];
  float* const ks = dc_smem;                            // [C][DK] k; then k P within the block
  float* const qs = ks + C * DK;                        // [C][DK] q; then q P within the block; then q P
  float* const gs = qs + C * DK;                        // [C][DK] g; then k times the decay to its block's end   (per head: [C][C] decays R)
  float* const part = gs + C * DK;                      // [NW][kPart] shares of A and B; then the right-hand sides
  float* const pk = part;                               // [C][kPK]  beta P k
  float* const vb = part + C * Y::kPK;                  // [C][kPV]  beta v
  float* const am = part + Y::kScratch;                 // [C][C]    -beta_i A_ij
  float* const bm = am + C * C;                         // [C][C]    B_ij
  float* const tm = bm + C * C;                         // [2 C][C]  T, then B T
  float* const dd = tm + 2 * C * C;                     // [4][DK]   decays of whole blocks
  float* const bs = dd + 4 * DK;                        // [C] beta
  float* const gh = bs + C;                             // [C] g per head
  float* const ph = gh + C;                             // [C] P per head
  griddep_launch();
  griddep_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g8 = lane >> 2, t4 = lane & 3;
  const int h = blockIdx.y, hk = h / (A.heads / A.kv_heads);
  int chunk;
  const int z = seq_of_piece(A.seqs, A.n_seqs, A.min_rows, C, A.item0 + (int)blockIdx.x, chunk);
  if (z < 0) return;
  const int4 sq = A.seqs[z];
  const int t0 = chunk * C;
  const int nt = min(C, sq.y - t0);
  const int64_t row0 = (int64_t)sq.x + t0;
  const int dk = A.dk, dv = A.dv;
  float* const item = A.ws + ((int64_t)blockIdx.x * A.heads + h) * A.item;
  bool odd = false;                                     // a number that is not finite
  auto seen = [&](float x) { odd = odd || !(fabsf(x) <= 3.4028234e38f); };

  // ---- the chunk's keys, queries, decays, values and write strengths: every load is on its way before the first number is used ----
  const float* const kp = A.k + row0 * A.ldk + (int64_t)hk * dk;
  const float* const qp = A.q + row0 * A.ldq + (int64_t)hk * dk;
  const float* const vp = A.v + row0 * A.ldv + (int64_t)h * dv;
  const T* const bias = reinterpret_cast<const T*>(A.dt_bias);
  const T* const dec = reinterpret_cast<const T*>(A.decay_in);
  constexpr int KN = C * DK / (NT * 4);
  float4 kv[KN], qv[KN];
#pragma unroll
  for (int n = 0; n < KN; ++n) {
    const int i = tid * 4 + n * NT * 4, t = i / DK, c = i % DK;
    kv[n] = qv[n] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t < nt && c < dk) {
      const float *const a = kp + (int64_t)t * A.ldk + c, *const b = qp + (int64_t)t * A.ldq + c;
      if (vec) {
        kv[n] = *reinterpret_cast<const float4*>(a);
        qv[n] = *reinterpret_cast<const float4*>(b);
      } else {
        kv[n] = make_float4(a[0], c + 1 < dk ? a[1] : 0.f, c + 2 < dk ? a[2] : 0.f, c + 3 < dk ? a[3] : 0.f);
        qv[n] = make_float4(b[0], c + 1 < dk ? b[1] : 0.f, c + 2 < dk ? b[2] : 0.f, c + 3 < dk ? b[3] : 0.f);
      }
    }
  }
  constexpr int STEP = NT / DK, GN = CHANNEL ? C / STEP : 1;   // decays per channel: a thread's channel stays the same
  const int gc = tid % DK, gt = tid / DK;
  float x[GN], bc = 0.f;
  if constexpr (CHANNEL) {
    if (gc < dk) bc = load_as_float(bias, (int64_t)h * dk + gc);
#pragma unroll
    for (int n = 0; n < GN; ++n) {
      const int t = gt + n * STEP;
      x[n] = t < nt && gc < dk ? load_as_float(dec, (row0 + t) * A.ld_decay + (int64_t)h * dk + gc) : 0.f;
    }
  }
  auto values = [&](int c0, float4 (&v)[4]) {           // columns c0 .. c0 + 127: four of a row per access
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const int t = warp + 8 * n, c = c0 + lane * 4;
      v[n] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (t < nt && c < dv) {
        const float* p = vp + (int64_t)t * A.ldv + c;
        if (vec_v) v[n] = *reinterpret_cast<const float4*>(p);
        else v[n] = make_float4(p[0], c + 1 < dv ? p[1] : 0.f, c + 2 < dv ? p[2] : 0.f, c + 3 < dv ? p[3] : 0.f);
      }
    }
  };
  auto put_values = [&](const float4 (&v)[4]) {
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const int t = warp + 8 * n;
      const float b = bs[t];
      float* const d = vb + t * Y::kPV + lane * 4;
      *reinterpret_cast<float2*>(d) = make_float2(b * v[n].x, b * v[n].y);
      *reinterpret_cast<float2*>(d + 2) = make_float2(b * v[n].z, b * v[n].w);
    }
  };
  float4 v0[4];
  values(0, v0);
  const float neg_a = -expf(load_as_float(reinterpret_cast<const T*>(A.a_log), h));
  if constexpr (CHANNEL) {
#pragma unroll
    for (int n = 0; n < GN; ++n) {
      const int t = gt + n * STEP;
      const float g = t < nt && gc < dk ? expf(neg_a * dc_softplus(x[n] + bc)) : 1.f;
      seen(g);
      gs[dc_at<DK>(t, gc)] = g;
    }
  } else if (tid < C) {
    const float g = tid < nt ? expf(neg_a * dc_softplus(load_as_float(dec, (row0 + tid) * A.ld_decay + h) + load_as_float(bias, h))) : 1.f;
    seen(g);
    gh[tid] = g;
  }
  if (tid < C) {
    const float b = tid < nt ? 1.0f / (1.0f + expf(-load_as_float(reinterpret_cast<const T*>(A.beta_in), (row0 + tid) * A.ld_beta + h))) : 0.f;
    seen(b);
    bs[tid] = b;
  }
#pragma unroll
  for (int n = 0; n < KN; ++n) {
    const int i = tid * 4 + n * NT * 4, t = i / DK, c = i % DK;
    seen(kv[n].x + kv[n].y + kv[n].z + kv[n].w);
    seen(qv[n].x + qv[n].y + qv[n].z + qv[n].w);
    *reinterpret_cast<float4*>(ks + dc_at<DK>(t, c)) = kv[n];
    *reinterpret_cast<float4*>(qs + dc_at<DK>(t, c)) = qv[n];
  }
#pragma unroll
  for (int n = 0; n < 4; ++n) seen(v0[n].x + v0[n].y + v0[n].z + v0[n].w);
  __syncthreads();

  // ---- A and B, a warp's sixteen channels ----
  if (warp < Y::NW) {
    float* const mine = part + warp * Y::kPart;
    if constexpr (CHANNEL) {
      // pairs within a block: lane j carries R_ij k_j from token to token.  [block][A, B][i][j]
      const int b = lane >> 3, jl = lane & 7;
      f2 r[8];
#pragma unroll
      for (int p = 0; p < 8; ++p) r[p] = 0ull;
#pragma unroll 1
      for (int il = 0; il < 8; ++il) {
        f2 a = 0ull, c = 0ull, a_ = 0ull, c_ = 0ull;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int at = dc_at<DK>(8 * b + il, warp * 16 + 4 * e);
          const ulonglong2 kk = *reinterpret_cast<const ulonglong2*>(ks + at), qq = *reinterpret_cast<const ulonglong2*>(qs + at),
                           gg = *reinterpret_cast<const ulonglong2*>(gs + at);
          r[2 * e] = jl == il ? kk.x : mul2(r[2 * e], gg.x);
          r[2 * e + 1] = jl == il ? kk.y : mul2(r[2 * e + 1], gg.y);
          a = fma2(kk.x, r[2 * e], a);
          c = fma2(qq.x, r[2 * e], c);
          a_ = fma2(kk.y, r[2 * e + 1], a_);
          c_ = fma2(qq.y, r[2 * e + 1], c_);
        }
        mine[b * 128 + il * 8 + jl] = sum2(a) + sum2(a_);
        mine[b * 128 + 64 + il * 8 + jl] = sum2(c) + sum2(c_);
      }
    }
  }
  if constexpr (CHANNEL) {
    __syncthreads();
    for (int n = tid; n < 4 * DK; n += NT) {
      const int c = n % DK, b = n / DK;
      float k[8], g[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) { k[e] = ks[dc_at<DK>(8 * b + e, c)]; g[e] = gs[dc_at<DK>(8 * b + e, c)]; }
      float cum = 1.f, rest = 1.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        cum *= g[e];
        ks[dc_at<DK>(8 * b + e, c)] = k[e] * cum;
        qs[dc_at<DK>(8 * b + e, c)] *= cum;
      }
#pragma unroll
      for (int e = 7; e >= 0; --e) {
        gs[dc_at<DK>(8 * b + e, c)] = k[e] * rest;
        rest *= g[e];
      }
      dd[b * DK + c] = cum;
    }
    __syncthreads();
  } else if (warp == 7) {   // decays per head: R_ij, P_i
    float r = 0.f, p = 1.f;
    for (int i = 0; i < C; ++i) {
      const float g = gh[i];
      p *= g;
      r = lane == i ? 1.f : r * g;
      gs[i * C + lane] = r;
      if (lane == i) ph[i] = p;
    }
  }
  if (warp < Y::NW) {
    // pairs of different blocks (per head: of all blocks up to the row's own): rows g8 of a tile are k, rows g8 + 8 are q
    float* const mine = part + warp * Y::kPart + (CHANNEL ? 512 : 0);
    const int c = warp * 16 + 4 * t4;
    const float* const rhs = CHANNEL ? gs : ks;
    int tile = 0;
#pragma unroll
    for (int bi = CHANNEL ? 1 : 0; bi < 4; ++bi) {
      x3::Split<8> a;
      a.set4(0, *reinterpret_cast<const float4*>(ks + dc_at<DK>(8 * bi + g8, c)));
      a.set4(4, *reinterpret_cast<const float4*>(qs + dc_at<DK>(8 * bi + g8, c)));
#pragma unroll
      for (int bj = 0; bj < (CHANNEL ? bi : bi + 1); ++bj, ++tile) {
        float4 r = *reinterpret_cast<const float4*>(rhs + dc_at<DK>(8 * bj + g8, c));
        if constexpr (CHANNEL) {
#pragma unroll
          for (int m = bj + 1; m < bi; ++m) {
            const float4 f = *reinterpret_cast<const float4*>(dd + m * DK + c);
            r.x *= f.x; r.y *= f.y; r.z *= f.z; r.w *= f.w;
          }
        }
        x3::Split<4> b;
        b.set4(0, r);
        float d[4];
        x3::mma16(d, a, b);
        *reinterpret_cast<float2*>(mine + tile * 128 + g8 * 8 + 2 * t4) = make_float2(d[0], d[1]);
        *reinterpret_cast<float2*>(mine + tile * 128 + 64 + g8 * 8 + 2 * t4) = make_float2(d[2], d[3]);
      }
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int n = tid; n < C * C; n += NT) {
    const int t = n / C, j = n % C, bi = t >> 3, bj = j >> 3;
    float sa = 0.f, sb = 0.f;
    if (j <= t) {
      const int tile = CHANNEL ? (bi == bj ? bi : 4 + bi * (bi - 1) / 2 + bj) : bi * (bi + 1) / 2 + bj;
      const float* const p = part + tile * 128 + (t & 7) * 8 + (j & 7);
#pragma unroll
      for (int w = 0; w < Y::NW; ++w) { sa += p[w * Y::kPart]; sb += p[w * Y::kPart + 64]; }
      if constexpr (!CHANNEL) { const float r = gs[t * C + j]; sa *= r; sb *= r; }
    }
    am[n] = j < t ? -bs[t] * sa : 0.f;
    bm[dc_at32(t, j)] = sb;
  }
  odd = __syncthreads_or(odd) != 0;

  // ---- T in one warp; the right-hand sides, K and P in the others ----
  put_values(v0);
  if (warp == 0) {
    float x[C];
#pragma unroll
    for (int i = 0; i < C; ++i) {
      float s = lane == i ? 1.f : 0.f, s_ = 0.f;
#pragma unroll
      for (int l = 0; l < i; l += 4) {
        const float4 m = *reinterpret_cast<const float4*>(am + i * C + l);
        if (l < i) s = fmaf(m.x, x[l], s);
        if (l + 1 < i) s_ = fmaf(m.y, x[l + 1], s_);
        if (l + 2 < i) s = fmaf(m.z, x[l + 2], s);
        if (l + 3 < i) s_ = fmaf(m.w, x[l + 3], s_);
      }
      x[i] = lane <= i ? s + s_ : 0.f;
      tm[dc_at32(i, lane)] = x[i];
    }
  } else {
    for (int n = tid - 32; n < 4 * DK; n += NT - 32) {
      const int c = n % DK, b = n / DK;
      float before = 1.f, after = 1.f;
      if constexpr (CHANNEL) {
        for (int m = 0; m < b; ++m) before *= dd[m * DK + c];
        for (int m = b + 1; m < 4; ++m) after *= dd[m * DK + c];
      }
      float kl[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int i = 8 * b + e, at = dc_at<DK>(i, c);
        if constexpr (!CHANNEL) { before = ph[i]; after = gs[(C - 1) * C + i]; }
        const float kv = ks[at];
        kl[e] = (CHANNEL ? gs[at] : kv) * after;
        pk[i * Y::kPK + c] = kv * before * bs[i];
        qs[at] *= before;
      }
      float* const kt = item + 2 * I::kMat + c * C;
#pragma unroll
      for (int u = 0; u < 2; ++u)
        *reinterpret_cast<float4*>(kt + (x3::unit_row(c, 2 * b + u) << 2)) = make_float4(kl[4 * u], kl[4 * u + 1], kl[4 * u + 2], kl[4 * u + 3]);
      if (b == 3) item[3 * I::kMat + c] = CHANNEL ? before * dd[3 * DK + c] : ph[C - 1];
    }
  }
  __syncthreads();

  // ---- B T: a warp's rows warp, warp + 8, .., a lane's column, in fp32 multiply-adds (B T is a factor of Q and O, and its sums are few) ----
  auto dot = [&](const float* m, int i, const float* x, int pitch) {   // sum over j <= i of m_ij x_j
    float s = 0.f;
    for (int j = 0; j <= i; ++j) s = fmaf(m[dc_at32(i, j)], x[j * pitch], s);
    return s;
  };
  if (odd) {
    for (int n = tid; n < C * C; n += NT) {
      const int i = n / C, j = n % C;
      float s = 0.f;
      for (int l = j; l <= i; ++l) s = fmaf(bm[dc_at32(i, l)], tm[dc_at32(l, j)], s);
      tm[dc_at32(C + i, j)] = s;
    }
  } else {
    float s[C / 8];
#pragma unroll
    for (int r = 0; r < C / 8; ++r) s[r] = 0.f;
#pragma unroll 2
    for (int l = 0; l < C; l += 4) {                    // (T is zero above its diagonal, B above its own)
      float4 m[C / 8];
#pragma unroll
      for (int r = 0; r < C / 8; ++r) m[r] = *reinterpret_cast<const float4*>(bm + dc_at32(warp + 8 * r, l));
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float t = tm[dc_at32(l + e, lane)];
#pragma unroll
        for (int r = 0; r < C / 8; ++r) s[r] = fmaf(e == 0 ? m[r].x : e == 1 ? m[r].y : e == 2 ? m[r].z : m[r].w, t, s[r]);
      }
    }
#pragma unroll
    for (int r = 0; r < C / 8; ++r) tm[dc_at32(C + warp + 8 * r, lane)] = s[r];
  }
  __syncthreads();

  // ---- [T; B T] times the right-hand sides: W, U and, from B T, Q = P q - B W and O ----
  float* const uo = item + I::kHead;
  const int64_t o_off = (int64_t)A.dvb * C * 8;
  auto keys_at = [](int row, int c) { return row * DK + (x3::unit_row(row, c >> 2) << 2) + (c & 3); };
  for (int c0 = 0;; c0 += 128) {                        // blocks of 128 value columns; the key columns go with the first
    const int vn = min(128, A.dvb * 8 - c0), first = c0 == 0 ? 0 : DK, cols = DK + vn;
    if (odd) {
      for (int n = first * C + tid; n < cols * C; n += NT) {
        const int i = n % C, c = n / C;
        const float* const x = c < DK ? pk + c : vb + c - DK;
        const int pitch = c < DK ? Y::kPK : Y::kPV;
        const float t = dot(tm, i, x, pitch), y = dot(tm + C * C, i, x, pitch);
        if (c < DK) {
          item[keys_at(i, c)] = t;
          item[I::kMat + keys_at(i, c)] = qs[dc_at<DK>(i, c)] - y;
        } else {
          float* const d = uo + ((c0 + c - DK) >> 3) * (C * 8) + i * 8 + ((c - DK) & 7);
          d[0] = t;
          d[o_off] = y;
        }
      }
    } else {
      for (int p = first / 16 + warp; p < cols / 16; p += NT / 32) {   // sixteen columns at a time
        const bool keys = p * 16 < DK;
        const float* const src = keys ? pk + p * 16 : vb + p * 16 - DK;
        const int pitch = keys ? Y::kPK : Y::kPV;
        x3::Split3<4> b[2][2];
#pragma unroll
        for (int kk = 0; kk < 2; ++kk)
#pragma unroll
          for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) b[kk][n].set(e, src[(16 * kk + 4 * t4 + e) * pitch + 8 * n + g8]);
#pragma unroll
        for (int mt = 0; mt < 4; ++mt) {
          float d[2][4];
#pragma unroll
          for (int kk = 0; kk <= (mt & 1); ++kk) {
            x3::Split<8> a;
            a.set4(0, *reinterpret_cast<const float4*>(tm + dc_at32(16 * mt + g8, 16 * kk + 4 * t4)));
            a.set4(4, *reinterpret_cast<const float4*>(tm + dc_at32(16 * mt + g8 + 8, 16 * kk + 4 * t4)));
            float s[2][4];
            x3::mma16_mean<2, x3::Split3<4>>(s, {&a, &a}, {&b[kk][0], &b[kk][1]});
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
              for (int e = 0; e < 4; ++e) d[n][e] = kk == 0 ? s[n][e] : d[n][e] + s[n][e];
          }
#pragma unroll
          for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              const int i = 16 * (mt & 1) + g8 + 8 * r, c = p * 16 + 8 * n + 2 * t4;
              float2 y = make_float2(d[n][2 * r], d[n][2 * r + 1]);
              if (keys) {
                if (mt >= 2) {
                  const float2 x = *reinterpret_cast<const float2*>(qs + dc_at<DK>(i, c));
                  y = make_float2(x.x - y.x, x.y - y.y);
                }
                *reinterpret_cast<float2*>(item + (mt >= 2 ? I::kMat : 0) + keys_at(i, c)) = y;
              } else {
                *reinterpret_cast<float2*>(uo + (mt >= 2 ? o_off : 0) + ((c0 + c - DK) >> 3) * (C * 8) + i * 8 + 2 * t4) = y;
              }
            }
        }
      }
    }
    if (c0 + 128 >= A.dvb * 8) break;
    values(c0 + 128, v0);
#pragma unroll
    for (int n = 0; n < 4; ++n) seen(v0[n].x + v0[n].y + v0[n].z + v0[n].w);
    odd = __syncthreads_or(odd) != 0;                   // (this block's columns have been read, too)
    put_values(v0);
    __syncthreads();
  }
}

// The state through the chunks, in order: grid (slices of NC = 8 NT G value columns, heads, sequences that can have chunks).  The next chunks are on their
// way (bulk copies) while one is worked on.  G groups of eight warps have 8 NT columns each and go their own way through the same chunks, so that one
// group's products fill the other's waits.  The slice of S lies in registers as the accumulators of K^T u, sixteen keys a warp, and for W S and Q S in
// shared memory by column as hi and lo; those two are tiles of sixteen tokens, half of the keys per warp.
template <int DK, int NT, int G>
struct DcCarry {
  using I = DcItem<DK>;
  static constexpr int NC = 8 * NT, kThreads = 256 * G, kStages = 3;
  static constexpr int kSlice = kDcC * NC * G;                     // floats of U (of O) per chunk and slice
  static constexpr int kStage = I::kHead + 2 * kSlice;             // floats
  static constexpr int kGroup = 2 * NC * DK + 2 * kDcC * NC + 4 * NT * 128;
  static constexpr int kFloats = kStages * kStage + G * kGroup;
  static constexpr int kSmem = kFloats * 4;
};

template <int DK, int NT, int G>
__global__ void __launch_bounds__(256 * G, 1) delta_carry_kernel(DcArgs A, int L, int vec_o) {
  using I = DcItem<DK>;
  using Y = DcCarry<DK, NT, G>;
  constexpr int C = kDcC, NC = Y::NC, STAGES = Y::kStages, KK = DK / 16;   // KK: tiles of sixteen keys
  extern __shared__ __align__(128) float dc_smem[];
  __shared__ __align__(8) uint64_t s_full[STAGES];
  __shared__ unsigned s_done[STAGES];                   // groups that are done with the stage, ever
  __shared__ int s_gave_up[G];                          // a wait of this group gave up: its warps decide by one word of their own, between two of their barriers
  const int tid = threadIdx.x & 255, group = threadIdx.x >> 8, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3, h = blockIdx.y;
  const int col0 = ((int)blockIdx.x * G + group) * NC;
  float* const st = dc_smem + STAGES * Y::kStage + group * Y::kGroup;   // S by column, as hi and lo: 2 x [NC][DK]
  float* const ut = st + 2 * NC * DK;                   // u by column: 2 x [NC][C]
  float* const red = ut + 2 * C * NC;                   // [4][NT][32] float4: the second half's sums
  const uint32_t full = tc::smem_u32(s_full);
  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; ++i) { tc::mbar_init(full + 8 * i, 1); s_done[i] = 0u; }
    for (int i = 0; i < G; ++i) s_gave_up[i] = 0;
    tc::mbar_init_fence();
  }
  griddep_launch();
  griddep_wait();
  int before;
  const int z = seq_with_pieces(A.seqs, A.n_seqs, A.min_rows, C, blockIdx.z, before);
  if (z < 0) return;
  const int4 sq = A.seqs[z];
  const int all = seq_pieces(sq, A.min_rows, C);
  const int c_first = max(0, A.item0 - before), chunks = min(all, A.item0 + A.n_items - before) - c_first, t_first = c_first * C;
  if (threadIdx.x == 0 && before + all > A.most) *A.err = 1u;   // more rows than the caller said
  if (chunks <= 0) return;
  const int dk = A.dk, dv = A.dv;
  const float* const items = A.ws + ((int64_t)(before + c_first - A.item0) * A.heads + h) * A.item;
  const int64_t step = (int64_t)A.heads * A.item;
  const int block0 = (int)blockIdx.x * G * NT;          // of eight columns

  auto fetch = [&](int c) {   // one thread
    const float* src = items + c * step;
    const uint32_t bar = full + 8 * (c % STAGES), dst = tc::smem_u32(dc_smem + (c % STAGES) * Y::kStage);
    tc::mbar_expect_tx(bar, Y::kStage * 4);
    auto copy = [&](uint32_t to, const float* from, uint32_t bytes) {
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(to), "l"(from), "r"(bytes), "r"(bar) : "memory");
    };
    copy(dst, src, I::kHead * 4);
    copy(dst + I::kHead * 4, src + I::kHead + (int64_t)block0 * C * 8, Y::kSlice * 4);
    copy(dst + (I::kHead + Y::kSlice) * 4, src + I::kHead + (int64_t)(A.dvb + block0) * C * 8, Y::kSlice * 4);
  };
  auto group_sync = [&] { asm volatile("bar.sync %0, 256;" ::"r"(group + 1) : "memory"); };
  if (threadIdx.x == 0) {
    for (int c = 0; c < STAGES && c < chunks; ++c) fetch(c);
  }
  const int krows = (dk + L - 1) / L;
  float* const slot = A.state + (int64_t)sq.w * A.state_slot_stride + (int64_t)h * krows * L * dv;
  const bool from_slot = sq.z > 0 || c_first > 0;
  auto at = [](int n, int c) { return n * DK + (x3::unit_col(n, c >> 2) << 2) + (c & 3); };
  auto put = [](float* p, int plane, int i, float x) {
    x3::Split<1> v;
    v.set(0, x);
    p[i] = __uint_as_float(v.hi[0]);
    p[plane + i] = __uint_as_float(v.lo[0]);
  };
  for (int i = tid; i < DK * NC; i += 256) {
    const int n = i % NC, c = i / NC;
    put(st, NC * DK, at(n, c), from_slot && c < dk && col0 + n < dv ? slot[((int64_t)(c / L) * dv + col0 + n) * L + c % L] : 0.f);
  }
  __syncthreads();
  const bool mine = warp < KK;
  const int key = 16 * warp + g;                        // K^T u: keys key, key + 8
  const int mt = warp & 3, kh = warp >> 2, row = 16 * (mt & 1) + g;   // W S, Q S: tokens row, row + 8 of W (mt < 2) or Q, keys of half kh
  float S[NT][4];                                       // columns 8 n + 2 t4, + 1
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = at(8 * n + 2 * t4 + (e & 1), key + 8 * (e >> 1));
      S[n][e] = mine ? st[i] + st[NC * DK + i] : 0.f;
    }
  bool ok = true;
  for (int c = 0; c < chunks; ++c) {
    const float* const sg = dc_smem + (c % STAGES) * Y::kStage;
    if (!mbar_wait(full + 8 * (c % STAGES), (uint32_t)(c / STAGES) & 1u)) *(volatile int*)&s_gave_up[group] = 1;
    float acc[NT][4];
    const float* const wr = sg + (mt >> 1) * I::kMat + row * DK;
#pragma unroll
    for (int k0 = 0; k0 < KK / 2; k0 += 2) {            // two tiles of keys at a time
      x3::Split<8> a[2];
      x3::Split<4> b[2 * NT];
      const x3::Split<8>* pa[2 * NT];
      const x3::Split<4>* pb[2 * NT];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int u = 4 * (kh * (KK / 2) + k0 + k) + t4;
        a[k].set4(0, *reinterpret_cast<const float4*>(wr + (x3::unit_row(row, u) << 2)));
        a[k].set4(4, *reinterpret_cast<const float4*>(wr + 8 * DK + (x3::unit_row(row, u) << 2)));
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          const float* const p = st + (8 * n + g) * DK + (x3::unit_col(g, u) << 2);
          b[k * NT + n].load4(0, p, p + NC * DK);
          pa[k * NT + n] = &a[k];
          pb[k * NT + n] = &b[k * NT + n];
        }
      }
      float s[2 * NT][4];
      x3::mma16<2 * NT>(s, pa, pb);
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float x = s[n][e] + s[NT + n][e];
          acc[n][e] = k0 == 0 ? x : acc[n][e] + x;
        }
    }
    float4* const rd = reinterpret_cast<float4*>(red) + mt * NT * 32 + lane;
    if (kh == 1) {
#pragma unroll
      for (int n = 0; n < NT; ++n) rd[n * 32] = make_float4(acc[n][0], acc[n][1], acc[n][2], acc[n][3]);
    }
    group_sync();
    if (*(volatile int*)&s_gave_up[group]) { ok = false; break; }
    if (kh == 0) {
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        const float4 x = rd[n * 32];
        const float y[4] = {acc[n][0] + x.x, acc[n][1] + x.y, acc[n][2] + x.z, acc[n][3] + x.w};
        const float* const uo = sg + I::kHead + (mt >= 2 ? Y::kSlice : 0) + (group * NT + n) * C * 8 + 2 * t4;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int tok = row + 8 * r;
          const float2 f = *reinterpret_cast<const float2*>(uo + tok * 8);
          if (mt < 2) {
#pragma unroll
            for (int e = 0; e < 2; ++e) put(ut, C * NC, (8 * n + 2 * t4 + e) * C + (x3::unit_col(2 * t4 + e, tok >> 2) << 2) + (tok & 3), (e ? f.y : f.x) - y[2 * r + e]);
          } else {
            const int t = t_first + c * C + tok, col = col0 + 8 * n + 2 * t4;
            float* const o = A.out + ((int64_t)sq.x + t) * A.ldo + (int64_t)h * dv + col;
            if (t < sq.y) {
              if (vec_o && col < dv) *reinterpret_cast<float2*>(o) = make_float2(f.x + y[2 * r], f.y + y[2 * r + 1]);
              else {
                if (col < dv) o[0] = f.x + y[2 * r];
                if (col + 1 < dv) o[1] = f.y + y[2 * r + 1];
              }
            }
          }
        }
      }
    }
    x3::Split<8> a[2];
    if (mine) {                                         // (what does not depend on u, ahead of the barrier)
      const float* const kt = sg + 2 * I::kMat + key * C;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        a[k].set4(0, *reinterpret_cast<const float4*>(kt + (x3::unit_row(key, 4 * k + t4) << 2)));
        a[k].set4(4, *reinterpret_cast<const float4*>(kt + 8 * C + (x3::unit_row(key, 4 * k + t4) << 2)));
      }
      const float p0 = sg[3 * I::kMat + key], p1 = sg[3 * I::kMat + key + 8];
#pragma unroll
      for (int n = 0; n < NT; ++n) { S[n][0] *= p0; S[n][1] *= p0; S[n][2] *= p1; S[n][3] *= p1; }
    }
    group_sync();
    if (mine) {
      x3::Split<4> b[2 * NT];
      const x3::Split<8>* pa[2 * NT];
      const x3::Split<4>* pb[2 * NT];
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          const float* const p = ut + (8 * n + g) * C + (x3::unit_col(g, 4 * k + t4) << 2);
          b[k * NT + n].load4(0, p, p + C * NC);
          pa[k * NT + n] = &a[k];
          pb[k * NT + n] = &b[k * NT + n];
        }
      float s[2 * NT][4];
      x3::mma16<2 * NT>(s, pa, pb);
#pragma unroll
      for (int n = 0; n < NT; ++n) {
#pragma unroll
        for (int e = 0; e < 4; ++e) S[n][e] += s[n][e] + s[NT + n][e];
#pragma unroll
        for (int e = 0; e < 4; ++e) put(st, NC * DK, at(8 * n + 2 * t4 + (e & 1), key + 8 * (e >> 1)), S[n][e]);
      }
    }
    group_sync();   // S complete, this group done with the stage
    if (tid == 0 && c + STAGES < chunks) {   // the last group to be done sends for the next chunk
      __threadfence_block();
      if (atomicAdd(&s_done[c % STAGES], 1u) % G == G - 1) {
        __threadfence_block();
        fetch(c + STAGES);
      }
    }
  }
  if (!ok) {   // given up: the copies under way land before the CTA leaves
    if (tid == 0) {
      *A.err = 1u;
      for (int e = 0; e < chunks && e < STAGES; ++e) mbar_wait(full + 8 * e, *(volatile unsigned*)&s_done[e] / G & 1u);   // (sent once and once per G counts)
    }
  }
  for (int i = tid; i < DK * NC; i += 256) {
    const int n = i % NC, c = i / NC;
    if (c < krows * L && col0 + n < dv) slot[((int64_t)(c / L) * dv + col0 + n) * L + c % L] = c < dk ? st[at(n, c)] + st[NC * DK + at(n, c)] : 0.f;
  }
}

template <typename T, int DK, bool CHANNEL>
cudaError_t chunk_launch(const DcArgs& A, int vec, int vec_v, cudaStream_t st) {
  constexpr int smem = DcChunk<DK>::kSmem;
  static PerDeviceOnce once;
  if (once.need()) {
    const cudaError_t e = cudaFuncSetAttribute(delta_chunk_kernel<T, DK, CHANNEL>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    once.done();
  }
  return launch(delta_chunk_kernel<T, DK, CHANNEL>, dim3((unsigned)A.n_items, (unsigned)A.heads), dim3(kDcChunkThreads), smem, st, A, vec, vec_v);
}

template <int DK, int NT, int G>
cudaError_t carry_launch(const DcArgs& A, int L, int vec_o, cudaStream_t st) {
  using Y = DcCarry<DK, NT, G>;
  static PerDeviceOnce once;
  if (once.need()) {
    const cudaError_t e = cudaFuncSetAttribute(delta_carry_kernel<DK, NT, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, Y::kSmem);
    if (e != cudaSuccess) return e;
    once.done();
  }
  constexpr int cols = Y::NC * G;
  return launch(delta_carry_kernel<DK, NT, G>, dim3((unsigned)((A.dv + cols - 1) / cols), (unsigned)A.heads, (unsigned)A.longs), dim3(Y::kThreads), Y::kSmem, st, A, L, vec_o);
}

template <typename T, int DK>
cudaError_t segment_launch(const DcArgs& A, bool channel, int vec, int vec_v, int vec_o, int L, int64_t walks, cudaStream_t st) {
  const cudaError_t e = channel ? chunk_launch<T, DK, true>(A, vec, vec_v, st) : chunk_launch<T, DK, false>(A, vec, vec_v, st);
  if (e != cudaSuccess) return e;
  // The fewest columns a CTA with which all CTAs run at once, one an SM.  us of both kernels, 512 tokens with decays per channel, 8, 16 (one or two column
  // tiles in one group) and 32 (two groups) columns a CTA: 8 heads 44, 55, 71; 16 heads 65, 57, 73; 32 heads 128, 112, 98.
  if (walks * ((A.dv + 7) / 8) <= sm_count()) return carry_launch<DK, 1, 1>(A, L, vec_o, st);
  if (walks * ((A.dv + 15) / 16) <= sm_count()) return carry_launch<DK, 2, 1>(A, L, vec_o, st);
  return carry_launch<DK, 2, 2>(A, L, vec_o, st);
}

int dc_dvb(int dv) { return (dv + 31) / 32 * 4; }
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
  // 56 / 29, 108 / 33, 422 / 55; per head 29 / 24, 53 / 28, 194 / 50.  Beside 32 single rows: 75 / 95, 90 / 100, 312 / 138; 55 / 72, 65 / 76, 216 / 114.
  // 16 sequences of 64, of 256 rows: 206 / 121, 818 / 344; 144 / 107, 526 / 300.
  const double n = max_rows, same = (double)rows / max_rows < n_seqs ? (double)rows / max_rows : n_seqs, one = heads * (dk * (double)dv / 16384.0), load = one * same;
  const int64_t shorts = n_seqs - (rows + max_rows - 1) / max_rows;
  auto most = [](double a, double b) { return a > b ? a : b; };
  double walk, chunks, few;
  if (channel_decay) {
    const bool wide = (int64_t)heads * n_seqs * ((dv + 15) / 16) < sm_count() * 3 / 2;   // (delta_rule_walk's choice)
    walk = 5.0 + n * most(0.35, wide ? 0.17 + 0.038 * load : most(0.36 + 0.01 * load, 0.0126 * load));
    chunks = 22.0 + (n + 24.0) * most(0.022, 0.0053 * load);
    few = 0.13 * one;
  } else {
    walk = 5.0 + n * most(0.25 + 0.0062 * load, 0.0088 * load);
    chunks = 20.0 + (n + 24.0) * most(0.02, 0.0047 * load);
    few = 0.09 * one;
  }
  if (shorts > 0) {
    walk += 0.3 * few * shorts;
    chunks += few * shorts;
  }
  // Two chunks at most in any sequence: little but starts to save, and scratch for every row to be had for it; the walk stays unless it takes 1.7 times as long.
  return (max_rows <= 2 * kDcC ? 1.7 : 1.0) * chunks < walk;
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
  const int vec_v = a->dv % 4 == 0 && al(a->v, a->ldv), vec_o = a->dv % 2 == 0 && a->ldo % 2 == 0 && (reinterpret_cast<uintptr_t>(a->out) & 7) == 0;
  const int L = a->dk <= 64 ? 4 : 8;   // the stored layout of a state (delta.cu)
  // Chains that go on side by side.  Sequences that have chunks are as many as there can be, unless most of the others are too short to have any: one of 1000 rows
  // beside 40 single ones, 4 heads of 64 x 64, decays per channel, 94 us with slices for sixteen, 58 for one.
  int64_t chains = longs;
  if (a->max_rows > 0 && a->n_seqs > 1 && a->rows - a->max_rows < (int64_t)(a->n_seqs - 1) * kDcMinRows) chains = 1 + (a->rows > a->max_rows ? (a->rows - a->max_rows) / a->max_rows : 0);
  if (chains > longs) chains = longs;
  const bool ch = a->channel_decay != 0;
  cudaStream_t st = (cudaStream_t)stream;
  for (int64_t at = 0; at < most; at += fit) {
    A.item0 = (int)at;
    A.n_items = (int)(most - at < fit ? most - at : fit);
    B200_FLOAT_TYPES(a->dtype, T, {
      if (a->dk <= 64) B200_CUDA((segment_launch<T, 64>(A, ch, vec, vec_v, vec_o, L, chains * a->heads, st)));
      else B200_CUDA((segment_launch<T, 128>(A, ch, vec, vec_v, vec_o, L, chains * a->heads, st)));
    });
  }
  return B200_OK;
}

}  // extern "C"
