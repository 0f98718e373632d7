// Long prompts of the decaying linear attention with decays per channel (linear_attn.cu) in pieces of 64 tokens whose sums run on the tensor cores:
//
//   within a piece, with R_ij = g_{j+1} ... g_i and P_i = g_0 ... g_i:   o_i = sum_{j <= i} (q_i R_ij k_j) v_j + (P_i q_i)^T S0,   S' = P S0 + sum_j (R_last,j k_j) v_j^T
//
// piece_kernel does everything but the terms of S0, for all pieces side by side: the read-out of the piece's own writes, its contribution to the state, the
// product of its decays, and the queries P q.  scan_kernel (linear_attn.cu) turns the contributions into starting states, and read_kernel adds (P q)^T S0.
// Products are sums of tf32 halves (tf32x3.cuh).  The decays enter as running products as in the walk: pairs of tokens in one block of eight walk
// them one by one, those of different blocks are matrix products of rows scaled from their block's start and to their block's end, times the
// products of the blocks between.  No logarithm or quotient is taken, so any decay in [0, 1] is safe.
// Fixed decays keep the walk: there queries, keys and values have passed silu and are mostly positive, sums without cancellation, in which what the tensor core cuts
// off adds up (read-out of 8 sequences of 256: 1.9e-7 from 64 bits, the walk 0.9e-7).
// (With decays per channel their rounding is ten times that: on forty kinds of input, with silu and without, with a mean and without, the errors are no larger than the
// walk's.)  8 heads of 128 x 128 over 2048 rows (bf16): 119 us -> 74, 72 without the path for numbers that are not finite; error against 64 bits 1.98e-6 (walk 2.01e-6)
// read-out and 2.39e-6 (2.40e-6) state.  Bound by the instructions and
// latencies of one wave of CTAs, 256 of them two on an SM: piece_kernel 40 us, some 65k clocks a CTA, a sixth of them loads and decays, a fifth pairs
// within a block, the rest shared memory reads and splits for the products; scan_kernel 12 us, read_kernel 19 us.
// A piece's instructions run once or twice per warp: loops are kept rolled where they can be, since fetching the code took longer than running it.
#pragma once
#include "tf32x3.cuh"

namespace b200 {

namespace {

constexpr int kLcC = 64, kLcThreads = 256, kLcPV = 130;   // tokens of a piece; pitch of the values and of a starting state

template <int DK>
struct LcPiece {
  static constexpr int kRow = kLcC * DK, kValues = kLcC * kLcPV;
  static constexpr int kQ = kRow > kLcC * kLcC ? kRow : kLcC * kLcC, kK = kRow > kValues ? kRow : kValues;   // (B and the values take their places)
  static constexpr int kFloats = kQ + kK + kRow + 3 * 8 * DK;
  static constexpr int kSmem = kFloats * 4;
  static_assert(kFloats >= DK * 128 + 3 * DK + 128, "walk_piece");
};
template <int DK>
struct LcRead {
  static_assert(kLcC * DK + DK * kLcPV >= DK * 128 + 3 * DK + 128, "walk_piece");
  static constexpr int kSmem = (kLcC * DK + DK * kLcPV) * 4;
};

// element (row, c) of 64 rows of DK: rows of one parity, and fours of rows, on different banks for the fragments' 16-byte and 4-byte reads alike
template <int DK>
__device__ __forceinline__ int lc_at(int row, int c) { return row * DK + ((((c >> 2) ^ ((row & 1) << 2) ^ (((row >> 2) & 3) << 1)) << 2) | (c & 3)); }

// Four times eight columns of sixteen terms each; EXACT: 16-bit numbers as they are, whose lo is zero.
template <bool EXACT>
struct LcCols {
  x3::Split<4> v[4];
  __device__ __forceinline__ void load(const float* p, int t4, int g) {   // p: the first of the sixteen rows, kLcPV apart
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float x = p[(4 * t4 + e) * kLcPV + 8 * n + g];
        if constexpr (EXACT) v[n].hi[e] = __float_as_uint(x);
        else v[n].set(e, x);
      }
  }
  // acc += a times these columns
  __device__ __forceinline__ void add(float (&acc)[4][4], const x3::Split<8>& a) const {
    float c[4][4];
    if constexpr (EXACT) {
      float d[4][4];
#pragma unroll
      for (int n = 0; n < 4; ++n) x3::mma0(c[n], a.lo[0], a.lo[4], a.lo[1], a.lo[5], v[n].hi[0], v[n].hi[1]);
#pragma unroll
      for (int n = 0; n < 4; ++n) x3::mma0(d[n], a.hi[2], a.hi[6], a.hi[3], a.hi[7], v[n].hi[2], v[n].hi[3]);
#pragma unroll
      for (int n = 0; n < 4; ++n) x3::mma(c[n], a.lo[2], a.lo[6], a.lo[3], a.lo[7], v[n].hi[2], v[n].hi[3]);
#pragma unroll
      for (int n = 0; n < 4; ++n) x3::mma(c[n], a.hi[0], a.hi[4], a.hi[1], a.hi[5], v[n].hi[0], v[n].hi[1]);
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) c[n][e] += d[n][e];
    } else {
      x3::mma16<4>(c, {&a, &a, &a, &a}, {&v[0], &v[1], &v[2], &v[3]});
    }
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[n][e] += c[n][e];
  }
};

// A piece with numbers that are not finite, token by token as in the walk, whose infinities stay what they are (halves of an infinity give NaN): from `src` (null: from
// nothing), with read-out, the state at its end to `dst` if there is one.  A function of its own: inlined it takes registers from the kernels (8 heads of 8192
// rows 282 us, 270 so, 267 without it).  smem: DK rows of 128 columns of the state, a token's key, query and decays, 128 sums.
template <typename T, int DK>
__device__ __noinline__ void walk_piece(const LaArgs& A, float* smem, int64_t row0, int nt, int h, int col0, const float* src, float* dst) {
  constexpr int HALF = DK / 2;
  const int tid = threadIdx.x, c = tid & 127, k0 = (tid >> 7) * HALF, dk = A.dk, dv = A.dv;
  const bool in = col0 + c < dv;
  float* const S = smem + k0 * 128 + c;
  float* const tok = smem + DK * 128;        // key | query | decays
  float* const sum = tok + 3 * DK;
#pragma unroll 1
  for (int i = 0; i < HALF; ++i) S[i * 128] = src && in && k0 + i < dk ? src[(int64_t)(k0 + i) * dv + c] : 0.f;
#pragma unroll 1
  for (int t = 0; t < nt; ++t) {
    const int64_t row = row0 + t;
    if (tid < DK) {
      float k = 0.f, q = 0.f, g = 1.f;
      if (tid < dk) {
        const int64_t at = (int64_t)h * dk + tid;
        k = load_as_float(reinterpret_cast<const T*>(A.k), row * A.ldk + at);
        q = load_as_float(reinterpret_cast<const T*>(A.q), row * A.ldq + at);
        if (A.act) { k = silu_f<T>(k); q = silu_f<T>(q); }
        q *= A.q_scale;
        g = channel_decay(A.z[row * A.ldz + at] + load_as_float(reinterpret_cast<const T*>(A.bias), at), A.inv_tau);
      }
      tok[tid] = k;
      tok[DK + tid] = q;
      tok[2 * DK + tid] = g;
    }
    float v = in ? load_as_float(reinterpret_cast<const T*>(A.v), row * A.ldv + (int64_t)h * dv + col0 + c) : 0.f, o = 0.f;
    if (A.act) v = silu_f<T>(v);
    __syncthreads();
#pragma unroll 1
    for (int i = k0; i < k0 + HALF && i < dk; ++i) {
      float& x = smem[i * 128 + c];
      x = fmaf(tok[2 * DK + i], x, tok[i] * v);
      o = fmaf(x, tok[DK + i], o);
    }
    if (k0) sum[c] = o;
    __syncthreads();
    if (!k0 && in) A.out[row * A.ldo + (int64_t)h * dv + col0 + c] = o + sum[c];
  }
#pragma unroll 1
  for (int i = 0; i < HALF && dst; ++i)
    if (in && k0 + i < dk) dst[(int64_t)(k0 + i) * dv + c] = S[i * 128];
}

// EXACT: the values are 16-bit numbers and pass no activation
template <typename T, int DK, bool EXACT>
__global__ void __launch_bounds__(kLcThreads, 2) piece_kernel(const __grid_constant__ LaArgs A, float* __restrict__ qp_out) {
  using Y = LcPiece<DK>;
  constexpr int C = kLcC, NT = kLcThreads;
  extern __shared__ __align__(128) float lc_smem[];
  float* const qs = lc_smem;                 // [C][DK] q; then q P within its block of eight
  float* const bm = qs;                      // [C][C]  then B_ij = q_i R_ij k_j
  float* const ks = qs + Y::kQ;              // [C][DK] k
  float* const vb = ks;                      // [C][kLcPV] then the values
  float* const gs = ks + Y::kK;              // [C][DK] decays; then k times the decay to its block's end; then to the piece's end
  float* const dd = gs + Y::kRow;            // [8][DK] decays of whole blocks
  float* const before = dd + 8 * DK;         // [8][DK] of all blocks before one
  float* const after = before + 8 * DK;      // [8][DK] and after it
  griddep_launch();
  griddep_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3, h = blockIdx.y;
  int piece;
  const int sidx = seq_of_piece(A.seqs, A.n_seqs, A.least, C, A.item0 + (int)blockIdx.z, piece);
  if (sidx < 0) return;
  const int4 sq = A.seqs[sidx];
  const int begin = piece * C, nt = min(C, sq.y - begin);
  const int64_t row0 = (int64_t)sq.x + begin;
  const int dk = A.dk, dv = A.dv, col0 = (int)blockIdx.x * 128;
  const int64_t wrow = (int64_t)blockIdx.z * A.heads + h;
  const T* const kp = reinterpret_cast<const T*>(A.k) + row0 * A.ldk + (int64_t)h * dk;
  const T* const qp = reinterpret_cast<const T*>(A.q) + row0 * A.ldq + (int64_t)h * dk;
  const T* const vp = reinterpret_cast<const T*>(A.v) + row0 * A.ldv + (int64_t)h * dv;
  bool odd = false;                          // a number that is not finite
  auto seen = [&](const float (&f)[8]) {
    float m = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) m += fabsf(f[j]);
    odd = odd || !(m <= 3.4028234e38f);
  };
  auto activate = [&](float (&f)[8]) {
    if (A.act) {
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = silu_f<T>(f[j]);
    }
  };
  auto put8 = [&](float* p, int t, int c, const float (&f)[8]) {
    *reinterpret_cast<float4*>(p + lc_at<DK>(t, c)) = make_float4(f[0], f[1], f[2], f[3]);
    *reinterpret_cast<float4*>(p + lc_at<DK>(t, c + 4)) = make_float4(f[4], f[5], f[6], f[7]);
  };
  // ---- queries, keys and decays: a thread's channels stay the same, the next rows' loads run ahead ----
  constexpr int KN = C * DK / (NT * 8), STEP = NT * 8 / DK;
  const int lc = (tid * 8) % DK, lt = (tid * 8) / DK;
  Raw8<T> rq, rk;
  Raw8<float> rz;
  auto fetch = [&](int t) {
    rq.load(qp + (int64_t)t * A.ldq, lc, dk, A.vec_k, t < nt);
    rk.load(kp + (int64_t)t * A.ldk, lc, dk, A.vec_k, t < nt);
    rz.load(A.z + (row0 + t) * A.ldz + (int64_t)h * dk, lc, dk, A.vec_z, t < nt);
  };
  fetch(lt);
  float bias[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) bias[j] = lc + j < dk ? load_as_float(reinterpret_cast<const T*>(A.bias), (int64_t)h * dk + lc + j) : 0.f;
#pragma unroll 1
  for (int n = 0; n < KN; ++n) {
    const int t = lt + n * STEP;
    float fq[8], fk[8], f[8];
    rq.floats(fq);
    rk.floats(fk);
    rz.floats(f);
    if (n + 1 < KN) fetch(t + STEP);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = t < nt && lc + j < dk ? channel_decay(f[j] + bias[j], A.inv_tau) : 1.f;
    seen(f);
    put8(gs, t, lc, f);
    activate(fk);
    seen(fk);
    put8(ks, t, lc, fk);
    activate(fq);
#pragma unroll
    for (int j = 0; j < 8; ++j) fq[j] *= A.q_scale;
    seen(fq);
    put8(qs, t, lc, fq);
  }
  __syncthreads();

  // ---- B ----
  // pairs within a block: lane (j, quarter of the channels) carries R_ij k_j from token to token, and keeps i = 2 t4, 2 t4 + 1
  float diag0 = 0.f, diag1 = 0.f;
  {
    f2 r[DK / 8];
#pragma unroll
    for (int e = 0; e < DK / 8; ++e) r[e] = 0ull;
#pragma unroll 2
    for (int il = 0; il < 8; ++il) {
      f2 a = 0ull, a_ = 0ull;
      const float first = g == il ? 1.f : 0.f;
      const f2 m = pk2(first, first);
#pragma unroll
      for (int e = 0; e < DK / 16; ++e) {
        const int at = lc_at<DK>(8 * warp + il, 16 * e + 4 * t4);
        const ulonglong2 kk = *reinterpret_cast<const ulonglong2*>(ks + at), qq = *reinterpret_cast<const ulonglong2*>(qs + at),
                         gg = *reinterpret_cast<const ulonglong2*>(gs + at);
        r[2 * e] = fma2(m, kk.x, mul2(r[2 * e], gg.x));
        r[2 * e + 1] = fma2(m, kk.y, mul2(r[2 * e + 1], gg.y));
        a = fma2(qq.x, r[2 * e], a);
        a_ = fma2(qq.y, r[2 * e + 1], a_);
      }
      float x0, x1, y0, y1;
      un2(a, x0, x1);
      un2(a_, y0, y1);
      float s = (x0 + x1) + (y0 + y1);
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      if (il < g) s = 0.f;
      if ((il >> 1) == t4) {
        if (il & 1) diag1 = s;
        else diag0 = s;
      }
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int n = tid; n < 8 * DK; n += NT) {
    const int c = n % DK, b = n / DK;
    float k[8], d[8], cum = 1.f, rest = 1.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) { k[e] = ks[lc_at<DK>(8 * b + e, c)]; d[e] = gs[lc_at<DK>(8 * b + e, c)]; }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      cum *= d[e];
      qs[lc_at<DK>(8 * b + e, c)] *= cum;
    }
#pragma unroll
    for (int e = 7; e >= 0; --e) {
      gs[lc_at<DK>(8 * b + e, c)] = k[e] * rest;
      rest *= d[e];
    }
    dd[b * DK + c] = cum;
  }
  __syncthreads();
  if (tid < 2 * DK) {
    const int c = tid % DK;
    float x[8], f = 1.f;
#pragma unroll
    for (int b = 0; b < 8; ++b) x[b] = dd[b * DK + c];
    if (tid < DK) {
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        before[b * DK + c] = f;
        f *= x[b];
      }
    } else {
#pragma unroll
      for (int b = 7; b >= 0; --b) {
        after[b * DK + c] = f;
        f *= x[b];
      }
    }
  }
  __syncthreads();
  // the values are on their way while the other pairs are worked on
  constexpr int VN = C * 128 / (NT * 8);
  Raw8<T> rv[VN];
#pragma unroll
  for (int n = 0; n < VN; ++n) {
    const int t = (tid + n * NT) / 16, c = (tid % 16) * 8;
    rv[n].load(vp + (int64_t)t * A.ldv, col0 + c, dv, A.vec_v, t < nt && col0 + c < dv);
  }
  // tiles of sixteen queries (row tile a) and eight keys (block bj), two a warp: the blocks before the row tile's first (0 .. 11), and that one against
  // the rows of the second (12 .. 15)
  auto place = [](int i, int& a, int& bj) {
    if (i >= 12) {
      a = i - 12;
      bj = 2 * a;
    } else {
      a = i < 2 ? 1 : i < 6 ? 2 : 3;
      bj = i - a * (a - 1);
    }
  };
  float d[2][4] = {};
  {
    int a[2], bj[2];
#pragma unroll
    for (int m = 0; m < 2; ++m) place(m == 0 ? warp : 15 - warp, a[m], bj[m]);   // (long chains of blocks with short ones)
#pragma unroll 1
    for (int kk = 0; kk < DK / 16; ++kk) {
      const int c = 16 * kk + 4 * t4;
      x3::Split<8> qa[2];
      x3::Split<4> kb[2];
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const float4 q0 = *reinterpret_cast<const float4*>(qs + lc_at<DK>(16 * a[m] + g, c));
        float4 q1 = *reinterpret_cast<const float4*>(qs + lc_at<DK>(16 * a[m] + 8 + g, c)), kr = *reinterpret_cast<const float4*>(gs + lc_at<DK>(8 * bj[m] + g, c));
        auto times = [](float4& x, const float* f) { const float4 y = *reinterpret_cast<const float4*>(f); x.x *= y.x; x.y *= y.y; x.z *= y.z; x.w *= y.w; };
        if (m == 0 || warp > 3) {
          times(q1, dd + 2 * a[m] * DK + c);
#pragma unroll 1
          for (int b = bj[m] + 1; b < 2 * a[m]; ++b) times(kr, dd + b * DK + c);
        }
        qa[m].set4(0, q0);
        qa[m].set4(4, q1);
        kb[m].set4(0, kr);
      }
      float s[2][4];
      x3::mma16<2>(s, {&qa[0], &qa[1]}, {&kb[0], &kb[1]});
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e) d[m][e] += s[m][e];
    }
  }
  // the queries from the piece's start
  if (blockIdx.x == 0) {
#pragma unroll 2
    for (int n = tid; n < 8 * DK; n += NT) {
      const int c = n % DK, b = n / DK;
      const float f = before[n];
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (8 * b + e < nt && c < dk) qp_out[(((int64_t)blockIdx.z * C + 8 * b + e) * A.heads + h) * dk + c] = qs[lc_at<DK>(8 * b + e, c)] * f;
      if (b == 7 && c < dk) A.ws_prod[wrow * dk + c] = f * dd[n];
    }
  }
  __syncthreads();                           // (queries and keys as they were have been read)
  auto bat = [](int row, int c) { return row * C + (x3::unit_row(row, c >> 2) << 2) + (c & 3); };
  bm[bat(8 * warp + 2 * t4, 8 * warp + g)] = diag0;
  bm[bat(8 * warp + 2 * t4 + 1, 8 * warp + g)] = diag1;
  if (!(warp & 1)) bm[bat(8 * warp + 2 * t4, 8 * warp + 8 + g)] = bm[bat(8 * warp + 2 * t4 + 1, 8 * warp + 8 + g)] = 0.f;   // (later keys)
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const int i = m == 0 ? warp : 15 - warp;
    int a, bj;
    place(i, a, bj);
    if (i < 12) *reinterpret_cast<float2*>(bm + bat(16 * a + g, 8 * bj + 2 * t4)) = make_float2(d[m][0], d[m][1]);
    *reinterpret_cast<float2*>(bm + bat(16 * a + 8 + g, 8 * bj + 2 * t4)) = make_float2(d[m][2], d[m][3]);
  }
#pragma unroll
  for (int n = 0; n < VN; ++n) {
    const int t = (tid + n * NT) / 16, c = (tid % 16) * 8;
    float f[8];
    rv[n].floats(f);
    activate(f);
    seen(f);
#pragma unroll
    for (int j = 0; j < 8; j += 2) *reinterpret_cast<float2*>(vb + t * kLcPV + c + j) = make_float2(f[j], f[j + 1]);
  }
#pragma unroll 2
  for (int n = tid; n < 7 * DK; n += NT) {   // keys to the piece's end
    const int c = n % DK, b = n / DK;
    const float f = after[n];
#pragma unroll
    for (int e = 0; e < 8; ++e) gs[lc_at<DK>(8 * b + e, c)] *= f;
  }
  if (__syncthreads_or(odd)) {
    walk_piece<T, DK>(A, lc_smem, row0, nt, h, col0, nullptr, A.ws_state + wrow * dk * dv + col0);
    return;
  }

  // ---- the read-out of the piece's own writes: B v ----
  float* const orow = A.out + row0 * A.ldo + (int64_t)h * dv + col0;
  // a warp's thirty-two columns: row tiles 0 and 3 or 1 and 2 of B v, then every second tile of sixteen keys of the contribution to the state, keys by
  // values; what is read of the values serves all of a warp's tiles
  const int n0 = (warp & 3) * 4, half = warp >> 2;
  const float* const vc = vb + 8 * n0;
  auto store = [&](float* to, int64_t ld, int rows, int a, const float (&acc)[4][4]) {
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int i = 16 * a + g + 8 * r, c = 8 * (n0 + n) + 2 * t4;
        float* const o = to + (int64_t)i * ld + c;
        if (i >= rows) continue;
        if (A.pair_o && col0 + c < dv) *reinterpret_cast<float2*>(o) = make_float2(acc[n][2 * r], acc[n][2 * r + 1]);
        else {
          if (col0 + c < dv) o[0] = acc[n][2 * r];
          if (col0 + c + 1 < dv) o[1] = acc[n][2 * r + 1];
        }
      }
  };
  LcCols<EXACT> v;
  {
    const int a0 = half, a1 = 3 - half;      // a0 < a1
    float acc[2][4][4] = {};
#pragma unroll 1
    for (int kk = 0; kk <= a1; ++kk) {
      v.load(vc + 16 * kk * kLcPV, t4, g);
      x3::Split<8> x;
      auto rows = [&](int a) {
        x.set4(0, *reinterpret_cast<const float4*>(bm + bat(16 * a + g, 16 * kk + 4 * t4)));
        x.set4(4, *reinterpret_cast<const float4*>(bm + bat(16 * a + 8 + g, 16 * kk + 4 * t4)));
      };
      rows(a1);
      v.add(acc[1], x);
      if (kk <= a0) {
        rows(a0);
        v.add(acc[0], x);
      }
    }
    store(orow, A.ldo, nt, a0, acc[0]);
    store(orow, A.ldo, nt, a1, acc[1]);
  }
  float acc[DK / 32][4][4] = {};
#pragma unroll 1
  for (int kk = 0; kk < C / 16; ++kk) {
    v.load(vc + 16 * kk * kLcPV, t4, g);
#pragma unroll
    for (int m = 0; m < DK / 32; ++m) {
      const int key = 16 * (2 * m + half) + g;
      x3::Split<8> x;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        x.set(e, gs[lc_at<DK>(16 * kk + 4 * t4 + e, key)]);
        x.set(4 + e, gs[lc_at<DK>(16 * kk + 4 * t4 + e, key + 8)]);
      }
      v.add(acc[m], x);
    }
  }
#pragma unroll
  for (int m = 0; m < DK / 32; ++m) store(A.ws_state + wrow * dk * dv + col0, dv, dk, 2 * m + half, acc[m]);
}

// out += (P q)^T S0: a piece's rows from its starting state
template <typename T, int DK>
__global__ void __launch_bounds__(kLcThreads, 2) read_kernel(const __grid_constant__ LaArgs A, const float* __restrict__ qp) {
  constexpr int C = kLcC, NT = kLcThreads;
  extern __shared__ __align__(128) float lc_smem[];
  float* const qs = lc_smem;                 // [C][DK]
  float* const ss = qs + C * DK;             // [DK][kLcPV]
  griddep_launch();
  griddep_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3, h = blockIdx.y;
  int piece;
  const int sidx = seq_of_piece(A.seqs, A.n_seqs, A.least, C, A.item0 + (int)blockIdx.z, piece);
  if (sidx < 0) return;
  const int4 sq = A.seqs[sidx];
  if (piece == 0 && sq.z == 0) return;                // (from nothing)
  const int begin = piece * C, nt = min(C, sq.y - begin);
  const int64_t row0 = (int64_t)sq.x + begin;
  const int dk = A.dk, dv = A.dv, col0 = (int)blockIdx.x * 128;
  const float* const st = A.ws_state + ((int64_t)blockIdx.z * A.heads + h) * dk * dv + col0;
  const bool q4 = (dk & 3) == 0;
  bool odd = false;                          // a number that is not finite
  auto seen = [&](const float4& x) { odd = odd || !(fabsf(x.x) + fabsf(x.y) + fabsf(x.z) + fabsf(x.w) <= 3.4028234e38f); };
  auto four = [](const float* p, int left, bool vec) {
    if (left <= 0) return make_float4(0.f, 0.f, 0.f, 0.f);
    if (vec) return *reinterpret_cast<const float4*>(p);
    return make_float4(p[0], left > 1 ? p[1] : 0.f, left > 2 ? p[2] : 0.f, left > 3 ? p[3] : 0.f);
  };
#pragma unroll 4
  for (int i = tid * 4; i < C * DK; i += NT * 4) {
    const int t = i / DK, c = i % DK;
    const float4 x = four(qp + (((int64_t)blockIdx.z * C + t) * A.heads + h) * dk + c, t < nt ? dk - c : 0, q4);
    seen(x);
    *reinterpret_cast<float4*>(qs + lc_at<DK>(t, c)) = x;
  }
#pragma unroll 8
  for (int i = tid * 4; i < DK * 128; i += NT * 4) {
    const int k = i / 128, c = i % 128;
    const float4 x = four(st + (int64_t)k * dv + c, k < dk ? dv - col0 - c : 0, A.vec_s);
    seen(x);
    float* const d = ss + k * kLcPV + c;
    *reinterpret_cast<float2*>(d) = make_float2(x.x, x.y);
    *reinterpret_cast<float2*>(d + 2) = make_float2(x.z, x.w);
  }
  if (__syncthreads_or(odd)) {               // from the starting state: what the piece wrote of its own cannot be told from it any more
    walk_piece<T, DK>(A, lc_smem, row0, nt, h, col0, st, nullptr);
    return;
  }
  float* const orow = A.out + row0 * A.ldo + (int64_t)h * dv + col0;
  const int n0 = (warp & 3) * 4, half = warp >> 2;   // a warp's thirty-two columns; its row tiles half, half + 2
  float acc[2][4][4];
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = 16 * (half + 2 * m) + g + 8 * (e >> 1), c = 8 * (n0 + n) + 2 * t4 + (e & 1);
        acc[m][n][e] = i < nt && col0 + c < dv ? orow[(int64_t)i * A.ldo + c] : 0.f;
      }
#pragma unroll 1
  for (int kk = 0; kk < DK / 16; ++kk) {
    LcCols<false> s0;
    s0.load(ss + 16 * kk * kLcPV + 8 * n0, t4, g);
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int row = 16 * (half + 2 * m) + g;
      x3::Split<8> x;
      x.set4(0, *reinterpret_cast<const float4*>(qs + lc_at<DK>(row, 16 * kk + 4 * t4)));
      x.set4(4, *reinterpret_cast<const float4*>(qs + lc_at<DK>(row + 8, 16 * kk + 4 * t4)));
      s0.add(acc[m], x);
    }
  }
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int i = 16 * (half + 2 * m) + g + 8 * r, c = 8 * (n0 + n) + 2 * t4;
        float* const o = orow + (int64_t)i * A.ldo + c;
        if (i >= nt) continue;
        if (A.pair_o && col0 + c < dv) *reinterpret_cast<float2*>(o) = make_float2(acc[m][n][2 * r], acc[m][n][2 * r + 1]);
        else {
          if (col0 + c < dv) o[0] = acc[m][n][2 * r];
          if (col0 + c + 1 < dv) o[1] = acc[m][n][2 * r + 1];
        }
      }
}

template <typename T, int DK, bool EXACT>
cudaError_t piece_start(const LaArgs& A, dim3 grid, float* qp, cudaStream_t st) {
  static PerDeviceOnce once;
  if (once.need()) {
    cudaError_t e = cudaFuncSetAttribute(piece_kernel<T, DK, EXACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, LcPiece<DK>::kSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(read_kernel<T, DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, LcRead<DK>::kSmem);
    if (e != cudaSuccess) return e;
    once.done();
  }
  return launch(piece_kernel<T, DK, EXACT>, grid, dim3(kLcThreads), LcPiece<DK>::kSmem, st, A, qp);
}

template <typename T, int DK>
cudaError_t piece_launch(const LaArgs& A, float* qp, cudaStream_t st) {
  const dim3 grid((unsigned)((A.dv + 127) / 128), (unsigned)A.heads, (unsigned)A.n_items);
  cudaError_t e;
  if constexpr (sizeof(T) == 2) e = A.act ? piece_start<T, DK, false>(A, grid, qp, st) : piece_start<T, DK, true>(A, grid, qp, st);
  else e = piece_start<T, DK, false>(A, grid, qp, st);
  if (e != cudaSuccess) return e;
  e = states_launch(A, A.longs, st);
  if (e != cudaSuccess) return e;
  return launch(read_kernel<T, DK>, grid, dim3(kLcThreads), LcRead<DK>::kSmem, st, A, (const float*)qp);
}

}  // namespace

}  // namespace b200
