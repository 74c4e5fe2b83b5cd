// fp32 products on mma.sync: an operand is split into three bf16 parts, which hold its 24 bits, and six of the nine products of parts are
// taken. The tensor cores then do 1024 / 6 = 171 FMAs a cycle and SM (bf16 1024 and tf32 509 measured), the fp32 pipe's packed FMAs
// 85 to 109; and sums over k need no shuffles.
#pragma once

#include "mma_sync.cuh"

namespace b200 {

// Two fp32 values as three pairs of bf16: x = p0 + p1 + p2 to within 2^-27 of x (each part takes eight bits of what the ones before it left)
__device__ __forceinline__ void split3(float x, float y, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
  p0 = pack_bf16x2(x, y);
  x -= __uint_as_float(p0 << 16); y -= __uint_as_float(p0 & 0xffff0000u);
  p1 = pack_bf16x2(x, y);
  x -= __uint_as_float(p1 << 16); y -= __uint_as_float(p1 & 0xffff0000u);
  p2 = pack_bf16x2(x, y);
}
// An operand of mma.sync.m16n8k16 in its three parts
struct SplitA { uint32_t p[3][4]; };   // 16 rows x 16
struct SplitB { uint32_t p[3][2]; };   // 16 x 8 columns
__device__ __forceinline__ SplitB split_b(float x0, float x1, float x2, float x3) {
  SplitB b;
  split3(x0, x1, b.p[0][0], b.p[1][0], b.p[2][0]);
  split3(x2, x3, b.p[0][1], b.p[1][1], b.p[2][1]);
  return b;
}
// a b to 2^-25 of the largest terms: all products of parts down to that. Those of the leading parts are summed 16 at a time by the tensor core and
// then in fp32; the others, 2^-8 and 2^-16 of them, in accumulators of their own (three short chains wait less than one long one).
struct SplitAcc {
  float lead[4] = {0.f, 0.f, 0.f, 0.f}, mid[4] = {0.f, 0.f, 0.f, 0.f}, low[4] = {0.f, 0.f, 0.f, 0.f};
  __device__ __forceinline__ float sum(int x) const { return lead[x] + (mid[x] + low[x]); }
};
// FIRST: `c` is still zero
template <bool FIRST = false>
__device__ __forceinline__ void mma_split(const SplitA& a, const SplitB& b, SplitAcc& c) {
  float t[4] = {0.f, 0.f, 0.f, 0.f};
  mma_bf16_16816(t, a.p[0][0], a.p[0][1], a.p[0][2], a.p[0][3], b.p[0][0], b.p[0][1]);
  mma_bf16_16816(c.mid, a.p[0][0], a.p[0][1], a.p[0][2], a.p[0][3], b.p[1][0], b.p[1][1]);
  mma_bf16_16816(c.low, a.p[0][0], a.p[0][1], a.p[0][2], a.p[0][3], b.p[2][0], b.p[2][1]);
  mma_bf16_16816(c.mid, a.p[1][0], a.p[1][1], a.p[1][2], a.p[1][3], b.p[0][0], b.p[0][1]);
  mma_bf16_16816(c.low, a.p[1][0], a.p[1][1], a.p[1][2], a.p[1][3], b.p[1][0], b.p[1][1]);
  mma_bf16_16816(c.low, a.p[2][0], a.p[2][1], a.p[2][2], a.p[2][3], b.p[0][0], b.p[0][1]);
#pragma unroll
  for (int x = 0; x < 4; ++x) c.lead[x] = FIRST ? t[x] : c.lead[x] + t[x];
}
__device__ __forceinline__ SplitA load_a(const float* at, int lane) {        // [3 parts][32 lanes][4]
  SplitA a;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const uint4 v = *reinterpret_cast<const uint4*>(at + i * 128 + lane * 4);
    a.p[i][0] = v.x; a.p[i][1] = v.y; a.p[i][2] = v.z; a.p[i][3] = v.w;
  }
  return a;
}

// also where rounding to 16 bits may be an infinity
__device__ __forceinline__ bool not_finite(float x) { return !(fabsf(x) <= 3.3e38f); }

}  // namespace b200
