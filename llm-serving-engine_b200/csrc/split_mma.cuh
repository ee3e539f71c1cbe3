// Products of float32 matrices on the tensor cores, as exact as on the CUDA cores.
//
// A float32 number has 24 bits: rounded to bfloat16 (8 bits), and what is left rounded to bfloat16, it is the sum of
// three such numbers, h + m + l, without a remainder. Of the nine products of two such sums six are taken (h h, h m, m h,
// h l, l h, m m; each is exact in float32); the other three together are below 2^-25 of the product. The tensor cores
// add sixteen products and cut the sum off (they do not round it), so a sum must not run on in them for long: the
// products h h of sixteen terms, which hardly lose a bit, are summed from zero and added to a float32 accumulator by the
// CUDA cores, as is the sum of the others. 1017 multiply-adds a clock and SM / 6 = 170, where the CUDA cores have 126 at
// best, and what counts more: a warp's tile of 32 x 32 reads 16 numbers of shared memory for 128 multiply-adds of a lane.
// (tf32 numbers, of 11 bits, would need three products of half the rate, and their remainders are 2^-22 each.)
//
// A number that is not finite has no such sum: its products are NaN. Whoever uses these products looks at the sums and
// takes those that are not finite again with fmaf.
#pragma once

#include "common.cuh"

namespace lse {
namespace split {

// Two neighbouring terms (the first in the lower half), as the operand registers of mma.sync hold them.
__device__ __forceinline__ void cut(float x0, float x1, uint32_t& h, uint32_t& m, uint32_t& l) {
  auto pack = [](float a, float b) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
    return r;
  };
  auto rest = [](float& a, float& b, uint32_t r) {
    a -= __uint_as_float(r << 16);
    b -= __uint_as_float(r & 0xffff0000u);
  };
  h = pack(x0, x1);
  rest(x0, x1, h);
  m = pack(x0, x1);
  rest(x0, x1, m);
  l = pack(x0, x1);
}

// Operands of one m16n8k16 product. Lane = 4 g + q. A: terms (0, 1) of row g, of row g + 8, terms (2, 3) of row g, of
// row g + 8; B: terms (0, 1) and (2, 3) of column g. Which four of the sixteen terms a lane holds (by its q) is free as
// long as A and B agree. C: columns 2 q, 2 q + 1 of row g, then of row g + 8.
struct A {
  uint32_t h[4], m[4], l[4];
  __device__ __forceinline__ void set(int i, float x0, float x1) { cut(x0, x1, h[i], m[i], l[i]); }
};
struct B {
  uint32_t h[2], m[2], l[2];
  __device__ __forceinline__ void set(int i, float x0, float x1) { cut(x0, x1, h[i], m[i], l[i]); }
};

__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// acc[j] += a b[j] for N tiles beside one another: their chains take turns. The largest products are summed by
// themselves: they have 16 bits each, so hardly anything of their sum is cut off.
template <int N>
__device__ __forceinline__ void multiply_add(float (&acc)[N][4], const A& a, const B (&b)[N]) {
  float d[N][4], t[N][4];
#pragma unroll
  for (int j = 0; j < N; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) d[j][e] = t[j][e] = 0.f;
#pragma unroll
  for (int j = 0; j < N; ++j) mma(d[j], a.l, b[j].h);
#pragma unroll
  for (int j = 0; j < N; ++j) mma(d[j], a.h, b[j].l);
#pragma unroll
  for (int j = 0; j < N; ++j) mma(d[j], a.m, b[j].m);
#pragma unroll
  for (int j = 0; j < N; ++j) mma(d[j], a.m, b[j].h);
#pragma unroll
  for (int j = 0; j < N; ++j) mma(d[j], a.h, b[j].m);
#pragma unroll
  for (int j = 0; j < N; ++j) mma(t[j], a.h, b[j].h);
#pragma unroll
  for (int j = 0; j < N; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[j][e] += t[j][e] + d[j][e];
}

// The same for accumulators that can afford a second register each: the small products of all terms run on in `low`,
// 2^-8 of the sum, which is added at the end (one rounding where `multiply_add` has one for every sixteen terms).
template <int N>
__device__ __forceinline__ void multiply_add(float (&acc)[N][4], float (&low)[N][4], const A& a, const B (&b)[N]) {
  float t[N][4];
#pragma unroll
  for (int j = 0; j < N; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) t[j][e] = 0.f;
#pragma unroll
  for (int j = 0; j < N; ++j) mma(t[j], a.h, b[j].h);
#pragma unroll
  for (int j = 0; j < N; ++j) mma(low[j], a.l, b[j].h);
#pragma unroll
  for (int j = 0; j < N; ++j) mma(low[j], a.h, b[j].l);
#pragma unroll
  for (int j = 0; j < N; ++j) mma(low[j], a.m, b[j].m);
#pragma unroll
  for (int j = 0; j < N; ++j) mma(low[j], a.m, b[j].h);
#pragma unroll
  for (int j = 0; j < N; ++j) mma(low[j], a.h, b[j].m);
#pragma unroll
  for (int j = 0; j < N; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[j][e] += t[j][e];
}
// One tile, 16 N terms at a time: acc += a[0] b[0] + .. + a[N - 1] b[N - 1], small products in `low[i]`.
template <int N>
__device__ __forceinline__ void multiply_add_terms(float (&acc)[4], float (&low)[N][4], const A (&a)[N], const B (&b)[N]) {
  float t[N][4];
#pragma unroll
  for (int j = 0; j < N; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) t[j][e] = 0.f;
#pragma unroll
  for (int j = 0; j < N; ++j) mma(t[j], a[j].h, b[j].h);
#pragma unroll
  for (int j = 0; j < N; ++j) mma(low[j], a[j].l, b[j].h);
#pragma unroll
  for (int j = 0; j < N; ++j) mma(low[j], a[j].h, b[j].l);
#pragma unroll
  for (int j = 0; j < N; ++j) mma(low[j], a[j].m, b[j].m);
#pragma unroll
  for (int j = 0; j < N; ++j) mma(low[j], a[j].m, b[j].h);
#pragma unroll
  for (int j = 0; j < N; ++j) mma(low[j], a[j].h, b[j].m);
#pragma unroll
  for (int j = 0; j < N; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[e] += t[j][e];
}

// Sixteen terms that lie side by side, rows `ld` apart (16 more than a multiple of 32: no bank conflicts): a lane has
// the four from 4 q on. `p` points to the first term of the lane's row (A: row g) or column (B: column g) of the tile.
__device__ __forceinline__ void along(A& a, const float* p, int ld, int q) {
  const float4 x = *reinterpret_cast<const float4*>(p + 4 * q), y = *reinterpret_cast<const float4*>(p + 8 * ld + 4 * q);
  a.set(0, x.x, x.y), a.set(1, y.x, y.y), a.set(2, x.z, x.w), a.set(3, y.z, y.w);
}
__device__ __forceinline__ void along(B& b, const float* p, int q) {
  const float4 x = *reinterpret_cast<const float4*>(p + 4 * q);
  b.set(0, x.x, x.y), b.set(1, x.z, x.w);
}
// Sixteen terms below one another, `ld` apart (4 more than a multiple of 16): a lane has 2 q, 2 q + 1 and those 8 on.
__device__ __forceinline__ void down(A& a, const float* p, int ld, int q) {
  p += 2 * q * ld;
#pragma unroll
  for (int i = 0; i < 2; ++i, p += 8 * ld) a.set(2 * i, p[0], p[ld]), a.set(2 * i + 1, p[8], p[ld + 8]);
}
__device__ __forceinline__ void down(B& b, const float* p, int ld, int q) {
  p += 2 * q * ld;
  b.set(0, p[0], p[ld]), b.set(1, p[8 * ld], p[9 * ld]);
}
// The same terms as `down`, side by side, rows `ld` apart (8 more than a multiple of 32).
__device__ __forceinline__ void along_as_down(A& a, const float* p, int ld, int q) {
  p += 2 * q;
#pragma unroll
  for (int i = 0; i < 2; ++i, p += 8) {
    const float2 x = *reinterpret_cast<const float2*>(p), y = *reinterpret_cast<const float2*>(p + 8 * ld);
    a.set(2 * i, x.x, x.y), a.set(2 * i + 1, y.x, y.y);
  }
}

__device__ __forceinline__ bool finite(float x) { return fabsf(x) <= 3.402823466e38f; }
// Is one of n numbers not finite?
template <int N>
__device__ __forceinline__ bool strange(const float (&x)[N][4]) {
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) s = fmaf(x[i][e], 0.f, s);
  return s != 0.f;
}
// The sum of n products, `dx` and `dy` floats apart, one after another.
static __device__ __noinline__ float dot(const float* x, int dx, const float* y, int dy, int n) {
  float s = 0.f;
#pragma unroll 1
  for (int i = 0; i < n; ++i) s = fmaf(x[i * dx], y[i * dy], s);
  return s;
}

}  // namespace split
}  // namespace lse
