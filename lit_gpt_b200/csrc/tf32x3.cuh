// fp32 products on the tensor cores: every factor as the sum of two tf32 numbers (hi the nearest, lo what is left of it),
// x y = hi lo' + lo hi' + hi hi' with fp32 accumulation (the dropped lo lo' is below 2^-22 of the product).
//
// The tensor core cuts off what its accumulator cannot hold where an fp32 addition rounds, so sums are kept short: a chain of products starts from zero
// and is added to the running sum by an ordinary fp32 addition.  Non-finite factors give NaN (inf - inf in lo).
//
// m16n8k8 fragments (g = lane / 4, t = lane % 4): A rows g, g + 8; B column g; C rows g, g + 8, columns 2 t, 2 t + 1.  The order of the summed index is
// free as long as both factors agree: a lane reads four neighbouring ones (4 t .. 4 t + 3 of sixteen) with one 16-byte access, numbers 0, 1 for the first
// product of eight and 2, 3 for the second.
#pragma once
#include "common.cuh"

namespace b200 {
namespace x3 {

template <int N>
struct Split {
  uint32_t hi[N], lo[N];
  __device__ __forceinline__ void set(int i, float x) {   // (the product reads the upper nineteen bits: lo loses at most the last bit of x)
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hi[i]) : "f"(x));
    lo[i] = __float_as_uint(x - __uint_as_float(hi[i]));
  }
  __device__ __forceinline__ void set4(int i, const float4& v) { set(i, v.x); set(i + 1, v.y); set(i + 2, v.z); set(i + 3, v.w); }
  __device__ __forceinline__ void load4(int i, const float* h, const float* l) {   // kept apart in memory
    const uint4 x = *reinterpret_cast<const uint4*>(h), y = *reinterpret_cast<const uint4*>(l);
    hi[i] = x.x; hi[i + 1] = x.y; hi[i + 2] = x.z; hi[i + 3] = x.w;
    lo[i] = y.x; lo[i + 1] = y.y; lo[i + 2] = y.z; lo[i + 3] = y.w;
  }
};

// the same with the bit that lo loses
template <int N>
struct Split3 : Split<N> {
  uint32_t last[N];
  __device__ __forceinline__ void set(int i, float x) {
    Split<N>::set(i, x);
    last[i] = __float_as_uint(__uint_as_float(this->lo[i]) - __uint_as_float(this->lo[i] & 0xffffe000u));
  }
};

__device__ __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma0(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {   // from zero
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

// sixteen terms of the sum: a holds row g's four numbers in 0 .. 3 and row g + 8's in 4 .. 7, b column g's.  The two products of hi and hi start chains of
// their own, which an fp32 addition joins.
// N such sums side by side, product by product: a product's successor in its chain waits some thirty clocks for it.
template <int N>
__device__ __forceinline__ void mma16(float (&c)[N][4], const Split<8>* const (&a)[N], const Split<4>* const (&b)[N]) {
  float d[N][4];
#pragma unroll
  for (int n = 0; n < N; ++n) mma0(c[n], a[n]->lo[0], a[n]->lo[4], a[n]->lo[1], a[n]->lo[5], b[n]->hi[0], b[n]->hi[1]);
#pragma unroll
  for (int n = 0; n < N; ++n) mma0(d[n], a[n]->hi[2], a[n]->hi[6], a[n]->hi[3], a[n]->hi[7], b[n]->hi[2], b[n]->hi[3]);
#pragma unroll
  for (int n = 0; n < N; ++n) mma(c[n], a[n]->hi[0], a[n]->hi[4], a[n]->hi[1], a[n]->hi[5], b[n]->lo[0], b[n]->lo[1]);
#pragma unroll
  for (int n = 0; n < N; ++n) mma(c[n], a[n]->lo[2], a[n]->lo[6], a[n]->lo[3], a[n]->lo[7], b[n]->hi[2], b[n]->hi[3]);
#pragma unroll
  for (int n = 0; n < N; ++n) mma(c[n], a[n]->hi[2], a[n]->hi[6], a[n]->hi[3], a[n]->hi[7], b[n]->lo[2], b[n]->lo[3]);
#pragma unroll
  for (int n = 0; n < N; ++n) mma(c[n], a[n]->hi[0], a[n]->hi[4], a[n]->hi[1], a[n]->hi[5], b[n]->hi[0], b[n]->hi[1]);
#pragma unroll
  for (int n = 0; n < N; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) c[n][e] += d[n][e];
}
// The same where more is made of the sums than a total: what the tensor core cuts off is half a unit in the last place on average (0.43 to 0.48 measured, products of one
// sign), always towards zero, and adds up.  Either product of hi and hi starts from zero and its half unit goes to the small products' sum, as does the last bit of a
// b that has it (Split3).
__device__ __forceinline__ float half_unit(float x, float c) { return fmaf(__uint_as_float(__float_as_uint(x) & 0xff800000u), 5.9604644775390625e-8f, c); }   // c + 2^(exponent - 24)
__device__ __forceinline__ void mma_last(float (&c)[4], const Split<8>& a, const Split3<4>& b) {
  mma(c, a.hi[0], a.hi[4], a.hi[1], a.hi[5], b.last[0], b.last[1]);
  mma(c, a.hi[2], a.hi[6], a.hi[3], a.hi[7], b.last[2], b.last[3]);
}
__device__ __forceinline__ void mma_last(float (&)[4], const Split<8>&, const Split<4>&) {}
template <int N, typename B>
__device__ __forceinline__ void mma16_mean(float (&c)[N][4], const Split<8>* const (&a)[N], const B* const (&b)[N]) {
  float d[N][4], f[N][4];
#pragma unroll
  for (int n = 0; n < N; ++n) mma0(c[n], a[n]->lo[0], a[n]->lo[4], a[n]->lo[1], a[n]->lo[5], b[n]->hi[0], b[n]->hi[1]);
#pragma unroll
  for (int n = 0; n < N; ++n) mma0(d[n], a[n]->hi[2], a[n]->hi[6], a[n]->hi[3], a[n]->hi[7], b[n]->hi[2], b[n]->hi[3]);
#pragma unroll
  for (int n = 0; n < N; ++n) mma(c[n], a[n]->hi[0], a[n]->hi[4], a[n]->hi[1], a[n]->hi[5], b[n]->lo[0], b[n]->lo[1]);
#pragma unroll
  for (int n = 0; n < N; ++n) mma0(f[n], a[n]->hi[0], a[n]->hi[4], a[n]->hi[1], a[n]->hi[5], b[n]->hi[0], b[n]->hi[1]);
#pragma unroll
  for (int n = 0; n < N; ++n) mma(c[n], a[n]->lo[2], a[n]->lo[6], a[n]->lo[3], a[n]->lo[7], b[n]->hi[2], b[n]->hi[3]);
#pragma unroll
  for (int n = 0; n < N; ++n) mma(c[n], a[n]->hi[2], a[n]->hi[6], a[n]->hi[3], a[n]->hi[7], b[n]->lo[2], b[n]->lo[3]);
#pragma unroll
  for (int n = 0; n < N; ++n) mma_last(c[n], *a[n], *b[n]);
#pragma unroll
  for (int n = 0; n < N; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) c[n][e] = (d[n][e] + f[n][e]) + half_unit(f[n][e], half_unit(d[n][e], c[n][e]));
}
__device__ __forceinline__ void mma16(float (&c)[4], const Split<8>& a, const Split<4>& b) {
  const Split<8>* const pa[1] = {&a};
  const Split<4>* const pb[1] = {&b};
  mma16<1>(reinterpret_cast<float (&)[1][4]>(c), pa, pb);
}

// Rows of a multiple of 32 floats in shared memory, read by lanes (g, t) at 16-byte unit 4 kk + t of row g: neighbouring rows swap halves of eight units,
// so that a quarter warp covers all banks
__device__ __forceinline__ int unit_row(int row, int unit) { return unit ^ ((row & 1) << 2); }
// The same for a column of a factor whose C fragments are written by lanes (g, t) at (unit g / 4, column 2 t or 2 t + 1)
__device__ __forceinline__ int unit_col(int col, int unit) { return unit ^ (((col >> 1) & 3) << 1) ^ ((col & 1) << 2); }

}  // namespace x3
}  // namespace b200
