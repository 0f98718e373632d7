// Short causal convolution over time on the channels of a projection, with the per-head step that follows it fused in.
//
//   y[t, c] = sum_j w[c, j] * u[t - taps + 1 + j, c]            (zeros before a sequence's first position)
//
// A step brings the rows of several sequences packed into one matrix (seqs[s] = {first row, rows, first position, state
// slot}).  Inputs from before the step's first row come from the sequence's tail: the last taps - 1 projected rows that
// earlier steps left in its state slot.  Whether a tap lies before the sequence start, in the tail or in the step is decided
// by its POSITION alone, so a slot that another sequence used before needs no clearing.
//
// The channels form up to three groups of heads (e.g. queries, keys, values); the lanes of a head apply after the convolution, in fp32:
//   act  : none | silu
//   post : none
//        | rotate + norm : rotary positions on the first rot_dims dimensions, interleaved pairs (2i, 2i + 1) turned by the
//                          angle position * inv_freq[i], cos and sin times rot_mscale; then x / sqrt(mean(x^2) + eps)
//        | unit          : x / sqrt(sum(x^2) + eps)
//   and a final multiplier post_scale.
// b200_conv_tail_update then stores each sequence's new tail.
#include "common.cuh"

namespace b200 {

namespace {

constexpr int kCvThreads = 128, kCvMaxTaps = 8, kCvMaxGroups = 3, kCvMaxIt = 8;   // head size <= 64 * kCvMaxIt

struct CvGroup {
  const void* w;
  void* out;
  int64_t ld_out;
  const double* inv_freq;
  int col0, heads, dim, act, post, rot_dims, out_f32;
  float rot_mscale, post_scale, eps;
};

struct CvParams {
  CvGroup g[kCvMaxGroups];
  int n_groups, taps, total_heads;
};

// two neighbouring elements at once when the caller vouches for the alignment (one 4- or 8-byte access)
template <typename T>
__device__ __forceinline__ void load_pair(const T* p, int64_t i, bool pair, bool second, float& a, float& b);
template <>
__device__ __forceinline__ void load_pair<__nv_bfloat16>(const __nv_bfloat16* p, int64_t i, bool pair, bool second, float& a, float& b) {
  if (pair) {
    const uint32_t v = *reinterpret_cast<const uint32_t*>(p + i);
    a = bf16lo(v);
    b = bf16hi(v);
  } else {
    a = __bfloat162float(p[i]);
    b = second ? __bfloat162float(p[i + 1]) : 0.f;
  }
}
template <>
__device__ __forceinline__ void load_pair<float>(const float* p, int64_t i, bool pair, bool second, float& a, float& b) {
  if (pair) {
    const float2 v = *reinterpret_cast<const float2*>(p + i);
    a = v.x;
    b = v.y;
  } else {
    a = p[i];
    b = second ? p[i + 1] : 0.f;
  }
}

// NIT: 64-element pieces of the widest head; TAPS: the number of taps when it is one of the unrolled ones, else 0 (read at run time).
// A warp walks rows_per_warp neighbouring rows of its head: the taps' weights are read once and, with unrolled taps, the rows that earlier
// taps need stay in registers, so a row is read once instead of once per tap (and fetched one row ahead).  Bound: instructions -- the
// division of silu, the norm's reduction, the rotation's sine.
template <typename T, int NIT, int TAPS>
__global__ void __launch_bounds__(kCvThreads) short_conv_kernel(const T* __restrict__ in, int64_t ld_in, CvParams P,
                                                                 const T* __restrict__ tail, int64_t tail_slot_stride, int tail_cols,
                                                                 const int4* __restrict__ seqs, const int* __restrict__ row_seq, int64_t rows,
                                                                 int rows_per_warp, int pairs) {
  griddep_launch();
  griddep_wait();
  const int lane = threadIdx.x & 31;
  int hh = (int)blockIdx.y * (kCvThreads / 32) + (threadIdx.x >> 5);
  if (hh >= P.total_heads) return;
  int gi = 0;
  while (gi + 1 < P.n_groups && hh >= P.g[gi].heads) { hh -= P.g[gi].heads; ++gi; }
  const CvGroup& G = P.g[gi];
  const int64_t row0 = (int64_t)blockIdx.x * rows_per_warp, row1 = row0 + rows_per_warp < rows ? row0 + rows_per_warp : rows;
  const int taps = TAPS ? TAPS : P.taps;
  const T* wt = reinterpret_cast<const T*>(G.w);
  const int c_head = G.col0 + hh * G.dim;     // first channel of this head among the convolved columns
  const bool pair = (pairs & 1) != 0;
  const bool wvec = TAPS == 4 && (pairs & 2) != 0;   // the eight taps of two neighbouring channels in one 16-byte (fp32: 32-byte) access
  const bool out_pair = (pairs & 4) != 0;
  constexpr int HIST = TAPS ? TAPS - 1 : 0, WT = TAPS ? TAPS : 1;

  float w[NIT][2][WT];                        // the taps of this lane's channels
  if constexpr (TAPS != 0) {
#pragma unroll
    for (int it = 0; it < NIT; ++it) {
      const int d = it * 64 + lane * 2;
#pragma unroll
      for (int j = 0; j < TAPS; ++j) w[it][0][j] = w[it][1][j] = 0.f;
      if (d < G.dim) {
        const T* wc = wt + (int64_t)(hh * G.dim + d) * TAPS;
        if constexpr (TAPS == 4) {
          if (wvec) {
            float wf[8];
            load8(wc, wf);
#pragma unroll
            for (int j = 0; j < 4; ++j) { w[it][0][j] = wf[j]; w[it][1][j] = wf[4 + j]; }
            continue;
          }
        }
#pragma unroll
        for (int j = 0; j < TAPS; ++j) {
          w[it][0][j] = load_as_float(wc, j);
          if (d + 1 < G.dim) w[it][1][j] = load_as_float(wc, TAPS + j);
        }
      }
    }
  }
  // the value `back` positions before row `row` (whose sequence's description is sq) in this lane's channels of piece `it`
  auto fetch = [&](int64_t row, const int4& sq, int back, int it, float& u0, float& u1) {
    u0 = u1 = 0.f;
    const int d = it * 64 + lane * 2;
    if (d >= G.dim) return;
    const bool second = d + 1 < G.dim;
    const int c = c_head + d, r = (int)(row - sq.x);   // row within the step's part of its sequence
    if (back > sq.z + r) return;                       // before the sequence's first token: zero
    if (back <= r) load_pair(in, (row - back) * ld_in + c, pair, second, u0, u1);
    else load_pair(tail + (int64_t)sq.w * tail_slot_stride, (int64_t)(taps - 1 - (back - r)) * tail_cols + c, pair, second, u0, u1);   // tail row taps-1-k: the k-th row before the step
  };

  float hist[HIST ? HIST : 1][NIT][2], next[NIT][2];   // hist[j]: the input of tap j
  int seq = -1;
  int4 sq = make_int4(0, 0, 0, 0);
  for (int64_t row = row0; row < row1; ++row) {
    const int s = row_seq[row];
    if (s != seq) {
      seq = s;
      sq = seqs[s];
      if constexpr (TAPS != 0) {
#pragma unroll
        for (int it = 0; it < NIT; ++it) {
#pragma unroll
          for (int j = 0; j < HIST; ++j) fetch(row, sq, TAPS - 1 - j, it, hist[j][it][0], hist[j][it][1]);
          fetch(row, sq, 0, it, next[it][0], next[it][1]);
        }
      }
    }
    const int pos = sq.z + (int)(row - sq.x);
    float val[NIT][2];
    float ss = 0.f;
    float cur[NIT][2];
    if constexpr (TAPS != 0) {
#pragma unroll
      for (int it = 0; it < NIT; ++it) {
        cur[it][0] = next[it][0];
        cur[it][1] = next[it][1];
        if (row + 1 < row1 && row + 1 < (int64_t)sq.x + sq.y) fetch(row + 1, sq, 0, it, next[it][0], next[it][1]);
      }
    }
#pragma unroll
    for (int it = 0; it < NIT; ++it) {
      const int d = it * 64 + lane * 2;
      float acc0 = 0.f, acc1 = 0.f;
      if constexpr (TAPS != 0) {
#pragma unroll
        for (int j = 0; j < HIST; ++j) {
          acc0 = fmaf(w[it][0][j], hist[j][it][0], acc0);
          acc1 = fmaf(w[it][1][j], hist[j][it][1], acc1);
        }
        acc0 = fmaf(w[it][0][WT - 1], cur[it][0], acc0);
        acc1 = fmaf(w[it][1][WT - 1], cur[it][1], acc1);
#pragma unroll
        for (int j = 0; j + 1 < HIST; ++j) { hist[j][it][0] = hist[j + 1][it][0]; hist[j][it][1] = hist[j + 1][it][1]; }
        if constexpr (HIST > 0) { hist[HIST - 1][it][0] = cur[it][0]; hist[HIST - 1][it][1] = cur[it][1]; }
      } else if (d < G.dim) {
        const T* wc = wt + (int64_t)(hh * G.dim + d) * taps;
#pragma unroll
        for (int j = 0; j < kCvMaxTaps + 1; ++j) {
          if (j >= taps) break;
          float u0, u1;
          fetch(row, sq, taps - 1 - j, it, u0, u1);
          acc0 = fmaf(load_as_float(wc, j), u0, acc0);
          if (d + 1 < G.dim) acc1 = fmaf(load_as_float(wc, taps + j), u1, acc1);
        }
      }
      if (G.act == 1) {
        acc0 = acc0 / (1.0f + expf(-acc0));
        acc1 = acc1 / (1.0f + expf(-acc1));
      }
      val[it][0] = acc0;
      val[it][1] = acc1;
    }
    if (G.post == 1) {
#pragma unroll
      for (int it = 0; it < NIT; ++it) {
        const int d = it * 64 + lane * 2;
        if (d + 1 < G.rot_dims && d + 1 < G.dim) {
          // the angle in double, reduced to [-pi, pi] before the fp32 sine and cosine: exact to fp32 at any position
          double a = (double)pos * G.inv_freq[d >> 1];
          a -= 6.283185307179586476925286766559 * rint(a * 0.15915494309189533576888376337251);
          float sn, cs;
          sincosf((float)a, &sn, &cs);
          sn *= G.rot_mscale;
          cs *= G.rot_mscale;
          const float u = val[it][0], v = val[it][1];
          val[it][0] = u * cs - v * sn;
          val[it][1] = v * cs + u * sn;
        }
      }
    }
    if (G.post != 0) {
#pragma unroll
      for (int it = 0; it < NIT; ++it) ss += val[it][0] * val[it][0] + val[it][1] * val[it][1];   // lanes past dim hold zeros
      ss = warp_sum(ss);
    }
    float mul = G.post_scale;
    if (G.post == 1) mul *= 1.0f / sqrtf(ss / (float)G.dim + G.eps);
    else if (G.post == 2) mul *= 1.0f / sqrtf(ss + G.eps);
#pragma unroll
    for (int it = 0; it < NIT; ++it) {
      const int d = it * 64 + lane * 2;
      if (d >= G.dim) continue;
      const int64_t o = row * G.ld_out + (int64_t)hh * G.dim + d;
      const float v0 = val[it][0] * mul, v1 = val[it][1] * mul;
      if (out_pair) {
        if (G.out_f32 || sizeof(T) == 4) *reinterpret_cast<float2*>(reinterpret_cast<float*>(G.out) + o) = make_float2(v0, v1);
        else *reinterpret_cast<uint32_t*>(reinterpret_cast<T*>(G.out) + o) = pack_bf16(v0, v1);
        continue;
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        if (d + e >= G.dim) break;
        if (G.out_f32) reinterpret_cast<float*>(G.out)[o + e] = e ? v1 : v0;
        else store_from_float(reinterpret_cast<T*>(G.out), o + e, e ? v1 : v0);
      }
    }
  }
}

// x / (1 + exp(-x)) by the approximate reciprocal and one correction of the quotient by its remainder (Markstein): as close as the division, without
// its branches.  Beyond 80 the quotient is x or below 1e-32 and the remainder could overflow: left as it is (infinities and NaN as by the division).
__device__ __forceinline__ float silu_cv(float x) {
  const float y = 1.0f + expf(-x), r = __fdividef(1.0f, y), q = x * r;
  return fabsf(x) < 80.0f ? fmaf(fmaf(-q, y, x), r, q) : q;
}
// 1 / sqrt(x): the approximation and one Newton step
__device__ __forceinline__ float rsqrt_cv(float x) {
  const float r = rsqrtf(x), h = 0.5f * x * r;
  return x > 1e-30f && x < 1e30f ? fmaf(r, fmaf(-h, r, 0.5f), r) : r;
}

// Four neighbouring channels of a row as they lie in memory
template <typename T>
struct CvRaw;
template <>
struct CvRaw<__nv_bfloat16> {
  uint2 w;
  __device__ __forceinline__ void load(const __nv_bfloat16* p) { w = *reinterpret_cast<const uint2*>(p); }
  __device__ __forceinline__ void zero() { w = make_uint2(0, 0); }
  __device__ __forceinline__ void floats(float (&f)[8], int at) const { f[at] = bf16lo(w.x); f[at + 1] = bf16hi(w.x); f[at + 2] = bf16lo(w.y); f[at + 3] = bf16hi(w.y); }
};
template <>
struct CvRaw<float> {
  float4 w;
  __device__ __forceinline__ void load(const float* p) { w = *reinterpret_cast<const float4*>(p); }
  __device__ __forceinline__ void zero() { w = make_float4(0.f, 0.f, 0.f, 0.f); }
  __device__ __forceinline__ void floats(float (&f)[8], int at) const { f[at] = w.x; f[at + 1] = w.y; f[at + 2] = w.z; f[at + 3] = w.w; }
};
__device__ __forceinline__ void store4(float* p, const float (&f)[8], int at) { *reinterpret_cast<float4*>(p) = make_float4(f[at], f[at + 1], f[at + 2], f[at + 3]); }
__device__ __forceinline__ void store4(__nv_bfloat16* p, const float (&f)[8], int at) {
  *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16(f[at], f[at + 1]), pack_bf16(f[at + 2], f[at + 3]));
}

constexpr int kCv8Taps = 4;
struct Cv8Blocks {   // per group: heads of a CTA (a power of two, the other lanes take further strips of rows), first CTA along y
  int heads[kCvMaxGroups], first[kCvMaxGroups];
};

// Four taps, heads of a multiple of eight channels on 16-byte boundaries: a lane has two times four channels of its head, LPR lanes a head, R neighbouring
// rows a lane.  All rows that R outputs read are fetched before the first is used, and the R chains of activation, norm and store run side by
// side; the cosines and sines of a CTA's rows are computed once for all its heads.
// Bound: the rows' way from L2 (R + 3 rows for R outputs), then the activation's instructions.  us against two channels a lane, each row's activation,
// norm and store before the next row's, rows of 24 heads of 128 rotated and normed / 48 heads with silu and unit norm, four taps: bf16 300 rows 12.4 -> 6.3
// / 16.3 -> 8.3, 2048 rows 31.2 -> 15.1 / 59.6 -> 29.8; fp32 2048 rows 24.9 -> 20.6 / 45.6 -> 39.2.  Eight neighbouring channels a lane: 17.3 / 31.7 and
// fp32 26.5 / 44.9 (half of every 32-byte sector per access).  R = 8: 23.4 / 41.1 (registers).
template <typename T, int LPR, int R>
__global__ void __launch_bounds__(kCvThreads, 4) short_conv8_kernel(const T* __restrict__ in, int64_t ld_in, CvParams P, Cv8Blocks B, const T* __restrict__ tail,
                                                                    int64_t tail_slot_stride, int tail_cols, const int4* __restrict__ seqs,
                                                                    const int* __restrict__ row_seq, int64_t rows) {
  constexpr int UNITS = kCvThreads / LPR, H = kCv8Taps - 1;
  __shared__ float2 s_turn[UNITS * R * LPR * 4];   // [row of the CTA][pair of channels]: cosine and sine
  griddep_launch();
  griddep_wait();
  const int tid = threadIdx.x, unit = tid / LPR, sub = tid % LPR;
  int gi = 0;
  while (gi + 1 < P.n_groups && (int)blockIdx.y >= B.first[gi + 1]) ++gi;
  const CvGroup& G = P.g[gi];
  const int hb = B.heads[gi], strips = UNITS / hb;
  const int hh = ((int)blockIdx.y - B.first[gi]) * hb + unit % hb;
  const int64_t cta0 = (int64_t)blockIdx.x * (strips * R), row0 = cta0 + (unit / hb) * R;
  if (cta0 >= rows) return;
  const int dim = G.dim, d[2] = {4 * sub, 4 * (LPR + sub)};
  const bool has[2] = {d[0] < dim, d[1] < dim};
  const int c = G.col0 + hh * dim;

  CvRaw<T> win[R + H][2];   // rows row0 - 3 .. row0 + R - 1 of the step
#pragma unroll
  for (int i = 0; i < R + H; ++i) {
    const int64_t row = row0 + i - H;
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      if (has[p] && row >= 0 && row < rows) win[i][p].load(in + row * ld_in + c + d[p]);
      else win[i][p].zero();
    }
  }
  float w[8][kCv8Taps];
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    const T* wt = reinterpret_cast<const T*>(G.w) + ((int64_t)hh * dim + d[p]) * kCv8Taps;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (has[p]) load8(wt + 8 * i, f);
#pragma unroll
      for (int j = 0; j < 4; ++j) { w[4 * p + 2 * i][j] = f[j]; w[4 * p + 2 * i + 1][j] = f[4 + j]; }
    }
  }
  int4 sq[R];
#pragma unroll
  for (int r = 0; r < R; ++r) sq[r] = row0 + r < rows ? seqs[row_seq[row0 + r]] : make_int4(0, 0, 0, 0);
  const int half = G.rot_dims >> 1;
  if (G.post == 1) {
    for (int i = tid; i < strips * R * half; i += kCvThreads) {
      const int r = i / half, p = i - r * half;
      const int64_t row = cta0 + r;
      if (row >= rows) break;
      const int4 s = seqs[row_seq[row]];
      // the angle in double, reduced to [-pi, pi] before the fp32 sine and cosine: exact to fp32 at any position
      double a = (double)(s.z + (int)(row - s.x)) * G.inv_freq[p];
      a -= 6.283185307179586476925286766559 * rint(a * 0.15915494309189533576888376337251);
      float sn, cs;
      sincosf((float)a, &sn, &cs);
      s_turn[r * (LPR * 4) + p] = make_float2(cs * G.rot_mscale, sn * G.rot_mscale);
    }
    __syncthreads();
  }

  float val[R][8], ss[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int at = (int)(row0 + r - sq[r].x);   // row within the step's part of its sequence
    float u[kCv8Taps][8];
#pragma unroll
    for (int j = 0; j < kCv8Taps; ++j)
#pragma unroll
      for (int p = 0; p < 2; ++p) win[r + j][p].floats(u[j], 4 * p);
    if (at < H && row0 + r < rows) {   // some taps lie before the step: in the tail, or before the sequence's first token
#pragma unroll
      for (int j = 0; j < H; ++j) {
        const int back = H - j;
        if (back <= at) continue;
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          CvRaw<T> t;
          if (has[p] && back <= sq[r].z + at) t.load(tail + (int64_t)sq[r].w * tail_slot_stride + (int64_t)(H - (back - at)) * tail_cols + c + d[p]);
          else t.zero();
          t.floats(u[j], 4 * p);
        }
      }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      float a = 0.f;
#pragma unroll
      for (int j = 0; j < kCv8Taps; ++j) a = fmaf(w[e][j], u[j][e], a);
      val[r][e] = a;
    }
    if (G.act == 1) {
#pragma unroll
      for (int e = 0; e < 8; ++e) val[r][e] = silu_cv(val[r][e]);
    }
    if (G.post == 1) {
#pragma unroll
      for (int e = 0; e < 8; e += 2) {
        const int dim0 = d[e >> 2] + (e & 3);
        if (dim0 + 1 < G.rot_dims) {
          const float2 t = s_turn[((unit / hb) * R + r) * (LPR * 4) + (dim0 >> 1)];
          const float x = val[r][e], y = val[r][e + 1];
          val[r][e] = x * t.x - y * t.y;
          val[r][e + 1] = y * t.x + x * t.y;
        }
      }
    }
    ss[r] = 0.f;
    if (G.post != 0) {
#pragma unroll
      for (int e = 0; e < 8; ++e) ss[r] = fmaf(val[r][e], val[r][e], ss[r]);   // lanes past dim hold zeros
    }
  }
  if (G.post != 0) {
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1)
#pragma unroll
      for (int r = 0; r < R; ++r) ss[r] += __shfl_xor_sync(0xffffffffu, ss[r], o);
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (row0 + r >= rows) continue;
    float mul = G.post_scale;
    if (G.post == 1) mul *= rsqrt_cv(ss[r] / (float)dim + G.eps);
    else if (G.post == 2) mul *= rsqrt_cv(ss[r] + G.eps);
#pragma unroll
    for (int e = 0; e < 8; ++e) val[r][e] *= mul;
    const int64_t o = (row0 + r) * G.ld_out + (int64_t)hh * dim;
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      if (!has[p]) continue;
      if (G.out_f32) store4(reinterpret_cast<float*>(G.out) + o + d[p], val[r], 4 * p);
      else store4(reinterpret_cast<T*>(G.out) + o + d[p], val[r], 4 * p);
    }
  }
}

// Four rows a lane from about eight CTAs per SM on, else one.  us with one and four, bf16, 24 heads of 128: 300 rows 6.3, 6.9, 1024 rows 12.5, 10.8; 24 heads
// of 64: 1024 rows 7.5, 8.1, 2048 rows 11.9, 11.0.
bool conv8_four(int64_t rows, int heads, int lanes_per_head) { return rows * heads >= (int64_t)sm_count() * (kCvThreads / lanes_per_head) * 8; }

template <typename T, int LPR>
cudaError_t short_conv8_launch(cudaStream_t st, const T* in, int64_t ld_in, const CvParams& P, const T* tail, int64_t tail_slot_stride, int tail_cols,
                               const int4* seqs, const int* row_seq, int64_t rows) {
  constexpr int UNITS = kCvThreads / LPR;
  Cv8Blocks B{};
  int y = 0, strips = 1;
  for (int g = 0; g < P.n_groups; ++g) {
    int hb = UNITS;
    while (P.g[g].heads % hb) hb >>= 1;
    B.heads[g] = hb;
    B.first[g] = y;
    y += P.g[g].heads / hb;
    strips = g == 0 || UNITS / hb < strips ? UNITS / hb : strips;
  }
  const bool four = conv8_four(rows, P.total_heads, LPR);
  const int per = strips * (four ? 4 : 1);
  const dim3 grid((unsigned)((rows + per - 1) / per), (unsigned)y);
  return four ? launch(short_conv8_kernel<T, LPR, 4>, grid, dim3(kCvThreads), 0, st, in, ld_in, P, B, tail, tail_slot_stride, tail_cols, seqs, row_seq, rows)
              : launch(short_conv8_kernel<T, LPR, 1>, grid, dim3(kCvThreads), 0, st, in, ld_in, P, B, tail, tail_slot_stride, tail_cols, seqs, row_seq, rows);
}

template <typename T, int NIT>
cudaError_t short_conv_launch(int taps, dim3 grid, cudaStream_t st, const T* in, int64_t ld_in, const CvParams& P, const T* tail,
                              int64_t tail_slot_stride, int tail_cols, const int4* seqs, const int* row_seq, int64_t rows, int rows_per_warp, int pairs) {
  auto go = [&](auto kernel) {
    return launch(kernel, grid, dim3(kCvThreads), 0, st, in, ld_in, P, tail, tail_slot_stride, tail_cols, seqs, row_seq, rows, rows_per_warp, pairs);
  };
  switch (taps) {
    case 2: return go(short_conv_kernel<T, NIT, 2>);
    case 3: return go(short_conv_kernel<T, NIT, 3>);
    case 4: return go(short_conv_kernel<T, NIT, 4>);
    default: return go(short_conv_kernel<T, NIT, 0>);
  }
}

// tail[slot][i] <- the (taps - 1 - i)-th last projected row of the sequence after this step, i = 0 .. taps - 2; rows that
// the step did not bring move up from the old tail.  One thread per (sequence, channel) reads all it needs before writing.
template <typename T>
__global__ void __launch_bounds__(256) conv_tail_kernel(const T* __restrict__ in, int64_t ld_in, T* __restrict__ tail,
                                                        int64_t tail_slot_stride, int tail_cols, int taps, const int4* __restrict__ seqs) {
  griddep_launch();
  griddep_wait();
  const int c = (int)blockIdx.x * 256 + threadIdx.x;
  if (c >= tail_cols) return;
  const int4 sq = seqs[blockIdx.y];
  const int L = sq.y, n = taps - 1;
  T* tl = tail + (int64_t)sq.w * tail_slot_stride;
  T keep[kCvMaxTaps];
#pragma unroll
  for (int i = 0; i < kCvMaxTaps; ++i) {
    if (i >= n) break;
    const int back = n - 1 - i;                 // rows before the sequence's last row
    if (back < L) keep[i] = in[(int64_t)(sq.x + L - 1 - back) * ld_in + c];
    else if (i + L < n) keep[i] = tl[(int64_t)(i + L) * tail_cols + c];
    else keep[i] = tl[(int64_t)i * tail_cols + c];   // unreachable: back >= L implies i + L < n
  }
#pragma unroll
  for (int i = 0; i < kCvMaxTaps; ++i) {
    if (i >= n) break;
    tl[(int64_t)i * tail_cols + c] = keep[i];
  }
}

}  // namespace

}  // namespace b200

using namespace b200;

extern "C" {

int b200_short_conv(const void* in, int64_t ld_in, const b200_conv_group* groups, int n_groups, int taps, const void* tail,
                    int64_t tail_slot_stride, int tail_cols, const int32_t* seqs, const int32_t* row_seq, int64_t rows, int dtype,
                    b200_stream_t stream) {
  B200_CHECK_ARG(in && groups && seqs && row_seq, "b200_short_conv: null pointer");
  B200_CHECK_ARG(n_groups >= 1 && n_groups <= kCvMaxGroups, "b200_short_conv: one to three groups");
  B200_CHECK_ARG(taps >= 1 && taps <= kCvMaxTaps + 1, "b200_short_conv: 1 to %d taps", kCvMaxTaps + 1);
  B200_CHECK_ARG(taps == 1 || tail, "b200_short_conv: a convolution over more than one tap needs the tail state");
  B200_CHECK_ARG(rows > 0 && rows <= 0x7fffffff, "b200_short_conv: bad row count");
  B200_CHECK_ARG((reinterpret_cast<uintptr_t>(seqs) & 15) == 0, "b200_short_conv: seqs must be 16-byte aligned");
  CvParams P{};
  P.n_groups = n_groups;
  P.taps = taps;
  for (int i = 0; i < n_groups; ++i) {
    const b200_conv_group& a = groups[i];
    B200_CHECK_ARG(a.w && a.out && a.heads > 0 && a.dim > 0 && a.dim <= 64 * kCvMaxIt, "b200_short_conv: bad group (head size up to %d)", 64 * kCvMaxIt);
    B200_CHECK_ARG(a.post != 1 || (a.rot_dims >= 0 && a.rot_dims <= a.dim && a.rot_dims % 2 == 0 && (a.rot_dims == 0 || a.inv_freq)),
                   "b200_short_conv: rotation needs an even number of dimensions and their frequencies");
    P.g[i] = CvGroup{a.w, a.out, a.ld_out, a.inv_freq, a.col0, a.heads, a.dim, a.act, a.post, a.rot_dims, a.out_f32, a.rot_mscale, a.post_scale, a.eps};
    P.total_heads += a.heads;
  }
  const int per = kCvThreads / 32;
  B200_CHECK_ARG((P.total_heads + per - 1) / per <= 65535, "b200_short_conv: too many heads");
  // Rows per warp, by (row, head) pairs per SM: more rows spare re-reads and set-up, fewer fill the SMs.  us with 1, 4 and 8 rows a warp, 40 heads of
  // 128 rotated and normed / 48 heads of 128 with silu and unit norm / 12 heads of 64, four taps: 128 rows (35, 42, 10 pairs per SM) 11.4, 12.4, 18.0 /
  // 11.2, 11.1, 16.3 / 6.4, 9.1, 12.4; 300 rows (81, 97, 24) 18.4, 13.5, 19.0 / 20.2, 17.1, 16.9 / 6.3, 8.9, 12.4; 1024 rows (277, 332, 83)
  // 47, 30, 34 / 53, 34, 31 / 10.9, 9.7, 13.0; 4096 rows (1107, 1328, 332) 194, 117, 104 / 236, 150, 137 / 27, 20, 19.
  const int64_t per_sm = rows * P.total_heads / sm_count();
  const int rpw = per_sm >= 320 ? 8 : (per_sm >= 64 ? 4 : 1);
  const dim3 grid((unsigned)((rows + rpw - 1) / rpw), (unsigned)((P.total_heads + per - 1) / per));
  // pairs of neighbouring channels are read with one access when every head starts on an even channel of even-pitched, aligned rows
  const size_t esz = dtype == B200_F32 ? 4 : 2;
  int pairs = (ld_in % 2 == 0) && (tail_cols % 2 == 0) && (tail_slot_stride % 2 == 0) && (reinterpret_cast<uintptr_t>(in) % (2 * esz) == 0) &&
              (reinterpret_cast<uintptr_t>(tail) % (2 * esz) == 0);
  int max_dim = 0;
  bool w16 = true, out2 = true;
  for (int i = 0; i < n_groups; ++i) {
    pairs = pairs && groups[i].dim % 2 == 0 && groups[i].col0 % 2 == 0;
    w16 = w16 && reinterpret_cast<uintptr_t>(groups[i].w) % 16 == 0;
    out2 = out2 && groups[i].dim % 2 == 0 && groups[i].ld_out % 2 == 0 && reinterpret_cast<uintptr_t>(groups[i].out) % (groups[i].out_f32 ? 8 : 2 * esz) == 0;
    max_dim = groups[i].dim > max_dim ? groups[i].dim : max_dim;
  }
  if (pairs && w16) pairs |= 2;   // even channels times four taps: every pair's taps start on a 16-byte boundary
  if (out2) pairs |= 4;
  // Four taps, eight channels a lane where every head's channels lie on 16-byte boundaries; fp32 only with four rows a lane: with one, 64 rows of 24 heads
  // take 6.5 us against 5.4.
  const int64_t e16 = 16 / (int64_t)esz;
  bool vec8 = taps == kCv8Taps && max_dim <= 256 && P.total_heads <= 65535 && ld_in % e16 == 0 && tail_cols % e16 == 0 && tail_slot_stride % e16 == 0 && w16 &&
              ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(tail)) & 15) == 0;
  vec8 = vec8 && (dtype != B200_F32 || conv8_four(rows, P.total_heads, max_dim <= 64 ? 8 : (max_dim <= 128 ? 16 : 32)));
  for (int i = 0; i < n_groups; ++i)
    vec8 = vec8 && groups[i].dim % 8 == 0 && groups[i].col0 % e16 == 0 && reinterpret_cast<uintptr_t>(groups[i].out) % 16 == 0 &&
           groups[i].ld_out % (groups[i].out_f32 ? 4 : e16) == 0;
  cudaStream_t st = (cudaStream_t)stream;
  const int4* sq = reinterpret_cast<const int4*>(seqs);
  if (vec8) {
    B200_FLOAT_TYPES(dtype, T, {
      if (max_dim <= 64) B200_CUDA((short_conv8_launch<T, 8>(st, (const T*)in, ld_in, P, (const T*)tail, tail_slot_stride, tail_cols, sq, row_seq, rows)));
      else if (max_dim <= 128) B200_CUDA((short_conv8_launch<T, 16>(st, (const T*)in, ld_in, P, (const T*)tail, tail_slot_stride, tail_cols, sq, row_seq, rows)));
      else B200_CUDA((short_conv8_launch<T, 32>(st, (const T*)in, ld_in, P, (const T*)tail, tail_slot_stride, tail_cols, sq, row_seq, rows)));
    });
    return B200_OK;
  }
  B200_FLOAT_TYPES(dtype, T, {
    if (max_dim <= 64) B200_CUDA((short_conv_launch<T, 1>(taps, grid, st, (const T*)in, ld_in, P, (const T*)tail, tail_slot_stride, tail_cols, sq, row_seq, rows, rpw, pairs)));
    else if (max_dim <= 128) B200_CUDA((short_conv_launch<T, 2>(taps, grid, st, (const T*)in, ld_in, P, (const T*)tail, tail_slot_stride, tail_cols, sq, row_seq, rows, rpw, pairs)));
    else if (max_dim <= 256) B200_CUDA((short_conv_launch<T, 4>(taps, grid, st, (const T*)in, ld_in, P, (const T*)tail, tail_slot_stride, tail_cols, sq, row_seq, rows, rpw, pairs)));
    else B200_CUDA((short_conv_launch<T, kCvMaxIt>(taps, grid, st, (const T*)in, ld_in, P, (const T*)tail, tail_slot_stride, tail_cols, sq, row_seq, rows, rpw, pairs)));
  });
  return B200_OK;
}

int b200_conv_tail_update(const void* in, int64_t ld_in, void* tail, int64_t tail_slot_stride, int tail_cols, int taps, const int32_t* seqs,
                          int n_seqs, int dtype, b200_stream_t stream) {
  B200_CHECK_ARG(taps >= 1 && taps <= kCvMaxTaps + 1, "b200_conv_tail_update: 1 to %d taps", kCvMaxTaps + 1);
  if (taps == 1) return B200_OK;   // nothing is carried
  B200_CHECK_ARG(in && tail && seqs && n_seqs > 0 && n_seqs <= 65535 && tail_cols > 0, "b200_conv_tail_update: bad argument");
  B200_CHECK_ARG((reinterpret_cast<uintptr_t>(seqs) & 15) == 0, "b200_conv_tail_update: seqs must be 16-byte aligned");
  const dim3 grid((unsigned)((tail_cols + 255) / 256), (unsigned)n_seqs);
  B200_FLOAT_TYPES(dtype, T, B200_CUDA(launch(conv_tail_kernel<T>, grid, dim3(256), 0, (cudaStream_t)stream, (const T*)in, ld_in, (T*)tail,
                                               tail_slot_stride, tail_cols, taps, reinterpret_cast<const int4*>(seqs))));
  return B200_OK;
}

}  // extern "C"
