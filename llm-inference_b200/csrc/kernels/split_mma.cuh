// Products of 32-bit numbers on the tensor cores.
//
// A number is the sum of three bfloat16 ones, to its last bit: the nearest, the nearest to what is left, and the rest (8 + 8 + 8 bits). Of the
// nine products of two such sums the six largest are taken; the others come to at most 2^-24 of the whole (the second part is up to 2^-8 of a number,
// the third 2^-17), as much as rounding it. Products of 8-bit numbers are exact in
// 32 bits. The tensor core's own sums drop bits below the last, so few are chained: the five small products of a step of 16 first, the large
// one last, and what is summed beyond one step is added with ordinary rounding.
// At the ends of the range: an infinity, like NaN, becomes NaN; the largest numbers, which bfloat16 would round to infinity, keep the largest bfloat16
// as their first part and are exact; below 2^-110 the third part falls under bfloat16's smallest number, 2^-133, half of which is then the error of a number.
#pragma once

#include "common.cuh"

struct Split {  // two neighbouring numbers, packed
  uint32_t part[3];
};
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}
__device__ __forceinline__ uint32_t pack_bf16_within(float lo, float hi) {  // past the largest number: the largest
  uint32_t d;
  asm("cvt.rn.satfinite.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}
__device__ __forceinline__ Split split_pair(float x, float y) {
  Split out;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    out.part[i] = i == 0 ? pack_bf16_within(x, y) : pack_bf16(x, y);
    if (i < 2) x -= __uint_as_float(out.part[i] << 16), y -= __uint_as_float(out.part[i] & 0xffff0000u);
  }
  return out;
}
// D[16][8] += A[16][16] B[16][8]. Of a lane (g = lane / 4, q = lane % 4), over the step's numbers along which is summed, in an order of
// this file's own: it holds 4 q .. + 3 of them. A: row g 4q, + 1; row g + 8 likewise; row g 4q + 2, + 3; row g + 8 likewise. B: column g
// 4q, + 1; 4q + 2, + 3. D: row g columns 2q, + 1; row g + 8 likewise.
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// D = A B.
__device__ __forceinline__ void mma_bf16_fresh(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
struct SplitA {  // a lane's share of A
  uint32_t part[3][4];
  __device__ __forceinline__ void set(int at, const Split& s) { part[0][at] = s.part[0], part[1][at] = s.part[1], part[2][at] = s.part[2]; }
};
// Of A, from four numbers each of rows g and g + 8.
__device__ __forceinline__ SplitA split_rows(float4 low, float4 high) {
  SplitA a;
  a.set(0, split_pair(low.x, low.y)), a.set(1, split_pair(high.x, high.y));
  a.set(2, split_pair(low.z, low.w)), a.set(3, split_pair(high.z, high.w));
  return a;
}
struct SplitB {  // of B
  Split lo, hi;
  __device__ __forceinline__ SplitB() {}
  __device__ __forceinline__ explicit SplitB(float4 v) : lo(split_pair(v.x, v.y)), hi(split_pair(v.z, v.w)) {}
};
// d = a b, over sixteen numbers.
__device__ __forceinline__ void mma_split(float (&d)[4], const SplitA& a, const SplitB& b) {
  constexpr int order[6][2] = {{2, 0}, {0, 2}, {1, 1}, {1, 0}, {0, 1}, {0, 0}};
  mma_bf16_fresh(d, a.part[order[0][0]], b.lo.part[order[0][1]], b.hi.part[order[0][1]]);
#pragma unroll
  for (int i = 1; i < 6; ++i) mma_bf16(d, a.part[order[i][0]], b.lo.part[order[i][1]], b.hi.part[order[i][1]]);
}

// A product whose result is the next one's A has two tiles of eight columns for sixteen: the one that stands as column g = lane / 4 of tile t.
// A lane q, which has columns 2 q and 2 q + 1 of D's either tile, then has four neighbours, 4 q .. + 3, as A wants them.
__device__ __forceinline__ int in_sixteen(int t, int g) { return 4 * (g >> 1) + 2 * t + (g & 1); }
__device__ __forceinline__ bool all_finite(float4 v) { return fmaf(v.x, 0.f, fmaf(v.y, 0.f, fmaf(v.z, 0.f, v.w * 0.f))) == 0.f; }
