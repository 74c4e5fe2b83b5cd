// The delta rule with one decay per token and head (mode 3 of linear_scan.cu) over prompts, 64 tokens at a time:
//
//   S <- a_t S ;  u_t = beta_t (v_t - S^T k_t) ;  S <- S + k_t u_t^T ;  o_t = S^T q_t          S [D, Dv] per head
//
// Walked token by token (linear_scan.cu) every token waits for the reduced S^T k of the one before it: a chain of
// shared-memory reads, FMAs and shuffles per token, 8 % of the fp32 rate for one prompt. With the decays' products
// r_ij = a_(j+1) .. a_i inside a chunk, c_i = a_1 .. a_i and S_0 the state in front of the chunk, the same sums are
//
//   (I + A) U = R,  A_ij = beta_i r_ij (k_i . k_j)  (j < i),   R_i = beta_i (v_i - c_i S_0^T k_i)
//   O_i = c_i S_0^T q_i + sum_(j <= i) r_ij (q_i . k_j) u_j,   S = c_64 S_0 + sum_j r_64,j k_j u_j^T
//
// (the chunked form of the gated delta rule, Yang, Kautz and Hatamizadeh 2024), products of small matrices without a chain inside.
//   delta_chunk_prep_kernel   a CTA per (chunk, q/k head): K K^T and Q K^T; then per head, 64 threads each: T = (I + A)^-1 by blocks of 16,
//                             P_ij = r_ij (q_i . k_j), c_i and r_64,j -> workspace, with K and Q. Chunks do not wait for one another.
//   delta_chunk_scan_kernel   a CTA per (run, head, block of 16 value columns) walks the chunks with its columns of S in registers
//                             and, for the products, in shared memory: [K; Q] S_0, U = T R, O += P U, S += K^T U. What the next
//                             chunk needs is on its way (bulk copies) meanwhile.
// The products run on mma.sync with fp32 operands in three bf16 parts (split_mma.cuh), which has the error of fp32 or less: state against 64 bits,
// 2048 and 513 tokens, 16 heads of 128: 1.9e-7 (by packed FMAs 2.2e-7, most of both from the keys). In two fp16 parts, with scales for each
// column, the scan took 145 us instead of 170, with an error 5 to 15 % above that of the FMAs for heads of 64. r_ij is a product of the decays
// themselves, roundings a walk makes too; sums of logarithms would lose digits to cancellation.
// Bound of the scan: mma.sync and the instructions that split operands share the issue slots: a tile of 16 x 8 x 16 takes 48 cycles of a scheduler and
// the split of its fp32 operand 28 more (measured apart: they do not overlap), 2800 + 2500 of a chunk's 6900 cycles; then its four
// barriers. So Q, T and P come split, once for the eight column blocks and four heads; K, wanted in two forms, would not fit so.
// One prompt of 2048 tokens, 16 heads of 128 x 128 over 4 q/k heads: 506 us token by token, 35 + 120 here (by FMAs, with T by substitution over
// all 64 rows: 30 + 194); 2048 and 513 tokens: 35 + 170 (30 + 252; the shorter run's CTAs fill in behind the longer one's).
#include "common.cuh"
#include "split_mma.cuh"
#include "../include/b200_ops.h"

namespace b200 {

constexpr int kDcC = 64, kDcCP = kDcC + 4;                // tokens of a chunk; padded row of a [64, 64] matrix
// The workspace holds a chunk's matrices as the scan's products want them in shared memory, so that they are four bulk copies (a copy for each of their
// rows: 320, and 200 us for a scan that takes 170). Q, T and P: operands of mma.sync in their three bf16 parts (split_mma.cuh), [8 rows x 16 columns][part][lane][2],
// T and P without the blocks above the diagonal. K, which is read as it is and transposed: fp32, rows without padding, bits 3 and 4 of
// the column turned by the row, so that pairs of columns of eight rows, and columns of four pairs of rows, are in different banks.
__device__ __forceinline__ int dc_turn(int row) { return ((row >> 1) & 1) << 3 | ((row ^ (row >> 2)) & 1) << 4; }
constexpr int kDcB = 3 * 64;                              // words of a block
constexpr int dc_block(int j, int s) { return (j >> 1) * ((j >> 1) + 1) + (j & 1) * ((j >> 1) + 1) + s; }     // of T and P: rows 8 j .., columns 16 s ..
constexpr int kDcT = 20 * kDcB, kDcPX = kDcT + 3 * kDcC, kDcHead = kDcT + kDcPX;      // words: T; P, c, r_64, beta
constexpr int dc_q(int D) { return 8 * (D / 16) * kDcB; }
constexpr int dc_kv(int D) { return kDcC * D + dc_q(D); } // K; Q
// What a step's workspace takes at most, for each head: 4.3 MB, 136 MB at 32 heads. That holds all a step needs up to 37 chunks (with a q/k head for each head and
// keys of 128; 82 at four heads to one, 135 with keys of 64 as well); longer ones go by windows of chunks.
constexpr long long kDcMost = 128ll * 8320;

struct DeltaChunkArgs {
  const float *q, *k, *v, *g, *beta;
  long long ldq, ldk, ldv, ldg, ldb;
  float *state, *o, *ws;
  const int* runs;
  int n_runs, H, G, Dv, tile_lo, tile_hi;                 // chunks [tile_lo, tile_hi) of all the step's chunks, counted run by run
  long long kv_ws;                                        // where K and Q begin in ws
};

template <int D> constexpr int prep_smem() {              // K | Q (later the four heads' A and T), K K^T | Q K^T, a of four heads
  constexpr int tiles = 2 * kDcC * D, as = 4 * kDcC * kDcCP;
  return ((tiles > as ? tiles : as) + 2 * kDcC * kDcCP + 4 * kDcC) * 4;
}

// In place: A [64, 64] strictly below the diagonal -> on and above it the transpose of T = (I + A)^-1 (zeros below it in the blocks of 16 it passes). 64 threads, thread j.
// Blocks of 16: those on the diagonal by forward substitution, a column to a thread; then, the nearest to the diagonal first,
// T_IJ = -T_II sum_(J <= M < I) A_IM T_MJ. The substitution of all 64 rows in registers was 2000 FMAs in a row of straight code, read once.
__device__ __forceinline__ void invert_lower(float* As, int j, int barrier) {
  const int blk = j >> 4, col = j & 15;
  {
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float s0 = 0.f, s1 = 0.f;
#pragma unroll
      for (int m = 0; m < i; m += 2) {                    // x is zero above the column's diagonal
        const float2 a = *reinterpret_cast<const float2*>(As + (blk * 16 + i) * kDcCP + blk * 16 + m);
        s0 = fmaf(a.x, x[m], s0);
        if (m + 1 < i) s1 = fmaf(a.y, x[m + 1], s1);
      }
      x[i] = (i == col ? 1.f : 0.f) - (s0 + s1);
    }
    asm volatile("bar.sync %0, 64;" ::"r"(barrier) : "memory");          // A's block is read: all of T's, transposed, takes its place
#pragma unroll
    for (int i = 0; i < 16; i += 4) *reinterpret_cast<float4*>(As + j * kDcCP + blk * 16 + i) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
  }
  const int r0 = blk * 4;                                 // from here on: four rows of a block, column `col`
#pragma unroll 1
  for (int l = 1; l < 4; ++l) {
    float y[3][4];
    asm volatile("bar.sync %0, 64;" ::"r"(barrier) : "memory");
#pragma unroll
    for (int J = 0; J < 3; ++J) {
      if (J + l > 3) break;
      const float* Tc = As + (J * 16 + col) * kDcCP;      // column `col` of block column J of T, as a row
      const float* Ar = As + ((J + l) * 16 + r0) * kDcCP;
#pragma unroll
      for (int i = 0; i < 4; ++i) y[J][i] = 0.f;
#pragma unroll 1
      for (int M = J; M < J + l; ++M) {
#pragma unroll
        for (int k = 0; k < 16; k += 4) {
          const float4 t = *reinterpret_cast<const float4*>(Tc + M * 16 + k);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float4 a = *reinterpret_cast<const float4*>(Ar + i * kDcCP + M * 16 + k);
            y[J][i] = fmaf(a.x, t.x, y[J][i]); y[J][i] = fmaf(a.y, t.y, y[J][i]);
            y[J][i] = fmaf(a.z, t.z, y[J][i]); y[J][i] = fmaf(a.w, t.w, y[J][i]);
          }
        }
      }
    }
#pragma unroll
    for (int J = 0; J < 3; ++J)
      if (J + l < 4) *reinterpret_cast<float4*>(As + (J * 16 + col) * kDcCP + (J + l) * 16 + r0) = make_float4(y[J][0], y[J][1], y[J][2], y[J][3]);
    asm volatile("bar.sync %0, 64;" ::"r"(barrier) : "memory");
#pragma unroll
    for (int J = 0; J < 3; ++J) {
      if (J + l > 3) break;
      const int I = (J + l) * 16;
#pragma unroll
      for (int i = 0; i < 4; ++i) y[J][i] = 0.f;
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        const float4 t = *reinterpret_cast<const float4*>(As + (I + k) * kDcCP + I + r0);       // T_II's column k
        const float v = As[(J * 16 + col) * kDcCP + I + k];
        y[J][0] = fmaf(t.x, v, y[J][0]); y[J][1] = fmaf(t.y, v, y[J][1]); y[J][2] = fmaf(t.z, v, y[J][2]); y[J][3] = fmaf(t.w, v, y[J][3]);
      }
    }
    asm volatile("bar.sync %0, 64;" ::"r"(barrier) : "memory");
#pragma unroll
    for (int J = 0; J < 3; ++J)
      if (J + l < 4) *reinterpret_cast<float4*>(As + (J * 16 + col) * kDcCP + (J + l) * 16 + r0) = make_float4(-y[J][0], -y[J][1], -y[J][2], -y[J][3]);
  }
  asm volatile("bar.sync %0, 64;" ::"r"(barrier) : "memory");
}

template <int D>
__global__ void __launch_bounds__(256, 2)
delta_chunk_prep_kernel(const DeltaChunkArgs p) {
  constexpr int KS = D / 16;
  extern __shared__ __align__(16) float sm[];
  constexpr int kTiles = 2 * kDcC * D, kAs = 4 * kDcC * kDcCP;
  float* Ks = sm;
  float* Qs = sm + kDcC * D;
  float* KK = sm + (kTiles > kAs ? kTiles : kAs);
  float* QK = KK + kDcC * kDcCP;
  float* AB = QK + kDcC * kDcCP;                          // [4 heads][a 64]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tile = p.tile_lo + blockIdx.x, kvh = blockIdx.y, rep = p.H / p.G;
  int first = 0, n = 0;
  for (int r = 0, at = 0; r < p.n_runs; ++r) {
    const int len = p.runs[4 * r + 1], nt = (len + kDcC - 1) / kDcC;
    if (tile < at + nt) { first = p.runs[4 * r] + (tile - at) * kDcC; n = min(kDcC, len - (tile - at) * kDcC); break; }
    at += nt;
  }
  if (n <= 0) return;                                     // the grid counts a chunk more per run than there may be
  float* kv = p.ws + p.kv_ws + ((long long)blockIdx.x * p.G + kvh) * dc_kv(D);
  {
    constexpr int N = kDcC * (D / 4) / 256;
    float4 x[N], y[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int t = (tid + 256 * i) / (D / 4), d = (tid + 256 * i) % (D / 4) * 4;
      x[i] = y[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (t < n) {
        x[i] = *reinterpret_cast<const float4*>(p.k + (long long)(first + t) * p.ldk + (long long)kvh * D + d);
        y[i] = *reinterpret_cast<const float4*>(p.q + (long long)(first + t) * p.ldq + (long long)kvh * D + d);
      }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int t = (tid + 256 * i) / (D / 4), d = (tid + 256 * i) % (D / 4) * 4;
      const int at = t * D + (d ^ dc_turn(t));
      *reinterpret_cast<float4*>(Ks + at) = x[i];
      *reinterpret_cast<float4*>(Qs + at) = y[i];
      *reinterpret_cast<float4*>(kv + at) = x[i];
    }
  }
  __syncthreads();
  {
    // 16 rows of K K^T or Q K^T to a warp, up to the diagonal; the two warps of a scheduler have ten tiles of eight columns together
    const int g = lane >> 2, t2 = (lane & 3) * 2, mt = warp < 4 ? warp : 7 - warp, turn = dc_turn(g);
    const float* rows = (warp < 4 ? Ks : Qs) + (mt * 16 + g) * D;
    float* out = (warp < 4 ? KK : QK) + (mt * 16 + g) * kDcCP + t2;
    SplitA a[KS];
#pragma unroll
    for (int s = 0; s < KS; ++s)
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const float2 v = *reinterpret_cast<const float2*>(rows + (x & 1) * 8 * D + ((16 * s + (x >> 1) * 8 + t2) ^ turn));
        split3(v.x, v.y, a[s].p[0][x], a[s].p[1][x], a[s].p[2][x]);
      }
    if (warp >= 4) {                                      // Q's operands for the scan: their rows are its columns
      uint32_t* qw = reinterpret_cast<uint32_t*>(kv + kDcC * D);
#pragma unroll
      for (int s = 0; s < KS; ++s)
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int e = 0; e < 2; ++e)
            *reinterpret_cast<uint2*>(qw + ((2 * mt + e) * KS + s) * kDcB + i * 64 + lane * 2) = make_uint2(a[s].p[i][e], a[s].p[i][2 + e]);
    }
#pragma unroll 1
    for (int j = 0; j < 2 * mt + 2; ++j) {
      SplitAcc c;
      const float* col = Ks + (8 * j + g) * D;
#pragma unroll
      for (int s = 0; s < KS; ++s) {
        const float2 v = *reinterpret_cast<const float2*>(col + ((16 * s + t2) ^ turn)), w = *reinterpret_cast<const float2*>(col + ((16 * s + 8 + t2) ^ turn));
        mma_split(a[s], split_b(v.x, v.y, w.x, w.y), c);
      }
      *reinterpret_cast<float2*>(out + 8 * j) = make_float2(c.sum(0), c.sum(1));
      *reinterpret_cast<float2*>(out + 8 * kDcCP + 8 * j) = make_float2(c.sum(2), c.sum(3));
    }
  }
  __syncthreads();                                        // K and Q are read: their place takes the heads' A
  const int grp = tid >> 6, i = tid & 63;                 // a head, a row
  float* As = sm + grp * kDcC * kDcCP;
  float* a_ = AB + grp * kDcC;
  const int lane0 = (i & 7) * 4, s_end = (i >> 5) * 2 + 2;         // steps of 16 columns: the same in a warp, of whose rows the last ends at i | 31
  for (int hh = grp; hh < rep; hh += 4) {
    const int h = kvh * rep + hh;
    const float b_i = i < n ? p.beta[(long long)(first + i) * p.ldb + h] : 0.f;
    a_[i] = i < n ? p.g[(long long)(first + i) * p.ldg + h] : 1.f;
    uint32_t* T = reinterpret_cast<uint32_t*>(p.ws + ((long long)blockIdx.x * p.H + h) * kDcHead);
    uint32_t* P = T + kDcT;
    float* X = reinterpret_cast<float*>(P + kDcT);
    // 16 columns of row i as the operand's words: pairs 2 t, 2 t + 1 and 2 t + 8, + 9 are lane t's
    auto store_row = [&](uint32_t* m, int s, const float (&x)[16]) {
      uint32_t w[3][8];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        split3(x[2 * t], x[2 * t + 1], w[0][2 * t], w[1][2 * t], w[2][2 * t]);
        split3(x[2 * t + 8], x[2 * t + 9], w[0][2 * t + 1], w[1][2 * t + 1], w[2][2 * t + 1]);
      }
      if (s > (i >> 4)) return;                           // above the diagonal
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        uint4* at = reinterpret_cast<uint4*>(m + dc_block(i >> 3, s) * kDcB + k * 64 + lane0 * 2);
        at[0] = make_uint4(w[k][0], w[k][1], w[k][2], w[k][3]);
        at[1] = make_uint4(w[k][4], w[k][5], w[k][6], w[k][7]);
      }
    };
    asm volatile("bar.sync %0, 64;" ::"r"(1 + grp) : "memory");
    float r = 1.f;                                        // r_ij, from the row's token to the ones before it
#pragma unroll 1
    for (int s = s_end - 1; s >= 0; --s) {
      float x[16];
#pragma unroll
      for (int e0 = 12; e0 >= 0; e0 -= 4) {
        const int j0 = 16 * s + e0;
        const float4 k4 = *reinterpret_cast<const float4*>(KK + i * kDcCP + j0), q4 = *reinterpret_cast<const float4*>(QK + i * kDcCP + j0);
        const float4 a4 = *reinterpret_cast<const float4*>(a_ + j0);
        const float ka[4] = {k4.x, k4.y, k4.z, k4.w}, qa[4] = {q4.x, q4.y, q4.z, q4.w}, aa[4] = {a4.x, a4.y, a4.z, a4.w};
        float A[4];
#pragma unroll
        for (int e = 3; e >= 0; --e) {
          const bool on = j0 + e <= i;
          x[e0 + e] = on ? r * qa[e] : 0.f;
          A[e] = j0 + e < i ? b_i * (r * ka[e]) : 0.f;
          if (on) r *= aa[e];
        }
        *reinterpret_cast<float4*>(As + i * kDcCP + j0) = make_float4(A[0], A[1], A[2], A[3]);
      }
      store_row(P, s, x);
    }
    X[i] = r;                                             // c_i
    r = 1.f;                                              // r_64 of token i
#pragma unroll 4
    for (int j0 = kDcC - 4; j0 >= (i & 32); j0 -= 4) {
      const float4 a4 = *reinterpret_cast<const float4*>(a_ + j0);
      if (j0 + 3 > i) r *= a4.w;
      if (j0 + 2 > i) r *= a4.z;
      if (j0 + 1 > i) r *= a4.y;
      if (j0 > i) r *= a4.x;
    }
    X[kDcC + i] = r;
    X[2 * kDcC + i] = b_i;
    asm volatile("bar.sync %0, 64;" ::"r"(1 + grp) : "memory");
    invert_lower(As, i, 1 + grp);
#pragma unroll 1
    for (int s = 0; s < s_end; ++s) {
      float x[16];
#pragma unroll
      for (int e = 0; e < 16; ++e) x[e] = 16 * s + e <= i ? As[(16 * s + e) * kDcCP + i] : 0.f;
      store_row(T, s, x);
    }
    asm volatile("bar.sync %0, 64;" ::"r"(1 + grp) : "memory");   // the next head's a and A overwrite these
  }
}

template <int N> struct IntC { static constexpr int value = N; };
constexpr int kDcNC = 16;                                 // value columns of a CTA: 128 CTAs for 16 heads of 128

template <int D> struct DcSmem {                          // float offsets
  static constexpr int NC = kDcNC, KS = D / 16, kThreads = 2 * KS * 32;   // two warps to 16 rows of the state
  static constexpr int K = 0, Q = K + 2 * kDcC * D, T = Q + dc_q(D), P = T + kDcT, Red = P + 2 * kDcPX, S = Red + KS * kDcC * NC,
                       R = S + KS * 3 * 128, U = R + 4 * 3 * 128, UD = U + 4 * 3 * 128, Bar = UD + 4 * 3 * 128, kTotal = Bar + 8;
  static_assert(kTotal * 4 <= 227 * 1024, "shared memory");
};

// half an operand A from an accumulator: columns 2 t, 2 t + 1 of rows g and g + 8 are what the lane holds of either
__device__ __forceinline__ void store_half_a(float* at, int lane, int half, const float (&x)[4]) {
  uint32_t p[3][2];
  split3(x[0], x[1], p[0][0], p[1][0], p[2][0]);
  split3(x[2], x[3], p[0][1], p[1][1], p[2][1]);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(at + i * 128 + lane * 4 + half * 2) = make_uint2(p[i][0], p[i][1]);
}

// an "or" over the first N threads, and a barrier for them
template <int N>
__device__ __forceinline__ int half_or(int x) {
  int r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\t"
      "barrier.cta.red.or.pred q, 1, %2, p;\n\tselp.s32 %0, 1, 0, q;\n\t}" : "=r"(r) : "r"(x), "n"(N) : "memory");
  return r;
}

// Tokens [at, len) of a run one by one, from S [D][16 columns] in shared memory (at Red): what a chunk with an infinity or NaN in R, U or Q S_0 takes,
// since a product with zeros above a diagonal, or of parts of an infinity, would carry it to tokens before its own. A warp has one of the columns (keys of 64: two)
// in registers, so that tokens follow one another without a barrier; their k, q and v come through the front of `sm`, 64 at a time. A NaN in the
// first of 2048 tokens, 16 heads of 128: the mixer 292 -> 1010 us (with S k summed over the CTA and k, q read where they lie, token by token, 2980). Outputs of several tokens
// summed at once take 735 to 780, but the longer code costs steps without a NaN 0.3 to 0.4% more (2048 and 513 tokens: 194.5 us of the two kernels, 195.1 to 195.3).
template <int D>
__device__ __noinline__ void walk_on(const DeltaChunkArgs& p, float* sm, int h, int col0, int first, int at, int len, float* state) {
  constexpr int NT = DcSmem<D>::kThreads, CPW = kDcNC * 32 / NT, RPL = D / 32;
  static_assert(2 * kDcC * D + kDcC * (kDcNC + 2) <= DcSmem<D>::Red, "the staged tokens lie in front of S");
  float *Ks = sm, *Qs = Ks + kDcC * D, *Vs = Qs + kDcC * D, *As = Vs + kDcC * kDcNC, *Bs = As + kDcC;
  const float* s0 = sm + DcSmem<D>::Red;
  const int tid = threadIdx.x, lane = tid & 31, col = (tid >> 5) * CPW, kvh = h / (p.H / p.G);
  float s[CPW][RPL];
#pragma unroll
  for (int c = 0; c < CPW; ++c)
#pragma unroll
    for (int i = 0; i < RPL; ++i) s[c][i] = s0[(lane + 32 * i) * kDcNC + col + c];
  for (int t0 = at; t0 < len; t0 += kDcC) {
    const int n = min(kDcC, len - t0);
    const long long row = first + t0;
    __syncthreads();                                      // the tokens before are read
    for (int i = tid; i < n * (D / 4); i += NT) {
      const int t = i / (D / 4), d = i % (D / 4) * 4;
      *reinterpret_cast<float4*>(Ks + t * D + d) = *reinterpret_cast<const float4*>(p.k + (row + t) * p.ldk + (long long)kvh * D + d);
      *reinterpret_cast<float4*>(Qs + t * D + d) = *reinterpret_cast<const float4*>(p.q + (row + t) * p.ldq + (long long)kvh * D + d);
    }
    for (int i = tid; i < n * kDcNC; i += NT) Vs[i] = p.v[(row + i / kDcNC) * p.ldv + (long long)h * p.Dv + col0 + i % kDcNC];
    if (tid < n) { As[tid] = p.g[(row + tid) * p.ldg + h]; Bs[tid] = p.beta[(row + tid) * p.ldb + h]; }
    __syncthreads();
#pragma unroll 1
    for (int t = 0; t < n; ++t) {
      const float a = As[t], b = Bs[t];
      float k[RPL], q[RPL];
#pragma unroll
      for (int i = 0; i < RPL; ++i) { k[i] = Ks[t * D + lane + 32 * i]; q[i] = Qs[t * D + lane + 32 * i]; }
#pragma unroll
      for (int c = 0; c < CPW; ++c) {
        float d = 0.f, o = 0.f;
#pragma unroll
        for (int i = 0; i < RPL; ++i) { s[c][i] *= a; d = fmaf(s[c][i], k[i], d); }
#pragma unroll
        for (int w = 16; w >= 1; w >>= 1) d += __shfl_xor_sync(0xffffffffu, d, w);
        const float u = b * (Vs[t * kDcNC + col + c] - d);
#pragma unroll
        for (int i = 0; i < RPL; ++i) { s[c][i] = fmaf(k[i], u, s[c][i]); o = fmaf(s[c][i], q[i], o); }
#pragma unroll
        for (int w = 16; w >= 1; w >>= 1) o += __shfl_xor_sync(0xffffffffu, o, w);
        if (lane == 0) p.o[((row + t) * p.H + h) * p.Dv + col0 + col + c] = o;
      }
    }
  }
#pragma unroll
  for (int c = 0; c < CPW; ++c)
#pragma unroll
    for (int i = 0; i < RPL; ++i) state[(long long)(lane + 32 * i) * p.Dv + col0 + col + c] = s[c][i];
}

// The state of 16 columns, transposed, is the 16 rows of an mma.sync tile: S^T K^T, R^T T^T, U^T P^T, S^T Q^T have the chunk's tokens as columns,
// U^T K the state's rows, and every accumulator is, lane by lane, half an operand of the next product. The operands are fp32 in three bf16 parts
// (split_mma.cuh). A warp keeps eight rows of the state, fp32, in its accumulator.
// What the next chunk waits for is only K S_0, U = T R and S += K^T U. All warps do the first, 16 rows of the state and half of the tokens each; their
// parts meet in shared memory, where the first half of the warps forms R and U while the other half reads out Q S_0; all do the last, and
// the second half P U after it.
template <int D>
__global__ void __launch_bounds__(DcSmem<D>::kThreads, 1)
delta_chunk_scan_kernel(const DeltaChunkArgs p) {
  using L = DcSmem<D>;
  constexpr int NC = kDcNC, KS = L::KS, TW = 8 / KS;      // TW: tiles of eight tokens to a warp of one half
  extern __shared__ __align__(16) float sm[];
  const int h = blockIdx.y, col0 = blockIdx.x * NC, run = blockIdx.z;
  int tb = 0;
  for (int r = 0; r < run; ++r) tb += (p.runs[4 * r + 1] + kDcC - 1) / kDcC;
  const int first = p.runs[4 * run], len = p.runs[4 * run + 1], p0 = p.runs[4 * run + 2], slot = p.runs[4 * run + 3];
  const int t_lo = max(tb, p.tile_lo), t_hi = min(tb + (len + kDcC - 1) / kDcC, p.tile_hi);
  if (t_lo >= t_hi) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, half = warp / KS, w = warp % KS;
  const int g = lane >> 2, t2 = (lane & 3) * 2;           // the lane's row and first column of an accumulator
  const int kvh = h / (p.H / p.G), turn = dc_turn(g);

  // What a chunk needs, as delta_chunk_prep_kernel laid it out: K and P | c | r_64 | beta a chunk ahead, Q and T half of one. One thread asks; all have
  // waited for a barrier's last phase when it does.
  const uint32_t bar = smem_u32(sm + L::Bar);
  auto kp_bar = [&](int tile) { return bar + 8u * (tile & 1); };
  const uint32_t qt_bar = bar + 16;
  auto copy = [&](int dst, const float* src, int floats, uint32_t b) { bulk_load_1d(smem_u32(sm + dst), src, floats * 4, b); };
  auto head_ws = [&](int tile) { return p.ws + ((long long)(tile - p.tile_lo) * p.H + h) * kDcHead; };
  auto kv_ws = [&](int tile) { return p.ws + p.kv_ws + ((long long)(tile - p.tile_lo) * p.G + kvh) * dc_kv(D); };
  auto ask_kp = [&](int tile) {
    mbar_arrive_expect_tx(kp_bar(tile), (kDcC * D + kDcPX) * 4u);
    copy(L::K + (tile & 1) * kDcC * D, kv_ws(tile), kDcC * D, kp_bar(tile));
    copy(L::P + (tile & 1) * kDcPX, head_ws(tile) + kDcT, kDcPX, kp_bar(tile));
  };
  auto ask_qt = [&](int tile) {
    mbar_arrive_expect_tx(qt_bar, (dc_q(D) + kDcT) * 4u);
    copy(L::Q, kv_ws(tile) + kDcC * D, dc_q(D), qt_bar);
    copy(L::T, head_ws(tile), kDcT, qt_bar);
  };
  const bool asks = tid == KS * 32;
  if (asks) {
    for (int i = 0; i < 3; ++i) mbar_init(bar + 8 * i, 1);
    fence_mbar_init();
    ask_kp(t_lo);
    ask_qt(t_lo);
  }
  __syncthreads();

  // columns g, g + 8 of the state's rows 16 w + 8 half + t2, + 1
  float S[4];
  float* const sp = p.state + (((long long)slot * p.H + h) * D) * p.Dv;
  auto s_at = [&](int x) { return (long long)(16 * w + 8 * half + t2 + (x & 1)) * p.Dv + col0 + g + (x >> 1) * 8; };
#pragma unroll
  for (int x = 0; x < 4; ++x) S[x] = p0 > 0 || t_lo > tb ? sp[s_at(x)] : 0.f;
  store_half_a(sm + L::S + w * 384, lane, half, S);

  for (int tile = t_lo; tile < t_hi; ++tile) {
    const int buf = tile & 1;
    const int at = (tile - tb) * kDcC, n = min(kDcC, len - at);
    const bool more = tile + 1 < t_hi;
    float v[TW][4];                                       // first half: the values of the tokens whose R this warp forms
    if (half == 0) {
#pragma unroll
      for (int i = 0; i < TW; ++i)
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const int t = 8 * (w + i * KS) + t2 + (x & 1);
          v[i][x] = t < n ? p.v[(long long)(first + at + t) * p.ldv + (long long)h * p.Dv + col0 + g + (x >> 1) * 8] : 0.f;
        }
    }
    mbar_wait(kp_bar(tile), (uint32_t)((tile - t_lo) >> 1) & 1u);
    mbar_wait(qt_bar, (uint32_t)(tile - t_lo) & 1u);
    __syncthreads();                                      // and S; the other K and P are read
    if (asks && more) ask_kp(tile + 1);
    const float* Ks = sm + L::K + buf * kDcC * D;
    const float* Ps = sm + L::P + buf * kDcPX;
    const float* cs = Ps + kDcT;                   // c | r_64 | beta
    int odd = 0;                                          // an infinity or NaN among this thread's part of R, then of U, or of Q S_0
    auto load_b = [&](const float* at) {                  // [part][lane][2]
      SplitB b;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const uint2 u = *reinterpret_cast<const uint2*>(at + i * 64 + lane * 2);
        b.p[i][0] = u.x; b.p[i][1] = u.y;
      }
      return b;
    };
    // eight rows of a lower triangle [64, 64] (from row 8 j) times R or U. The number of steps is chosen by one branch: a branch in front of each
    // step kept the steps apart
    auto times_lower = [&](const float* tri, const float* X, int j, float (&z)[4]) {
      auto steps = [&](auto n) {
        SplitAcc c[2];
#pragma unroll
        for (int s = 0; s < n.value; ++s) {
          const SplitA a = load_a(X + s * 384, lane);
          const SplitB b = load_b(tri + (dc_block(j, 0) + s) * kDcB);
          if (s < 2) mma_split<true>(a, b, c[s & 1]);
          else mma_split(a, b, c[s & 1]);
        }
#pragma unroll
        for (int x = 0; x < 4; ++x) z[x] = n.value > 1 ? c[0].sum(x) + c[1].sum(x) : c[0].sum(x);
      };
      if (j < 2) steps(IntC<1>());
      else if (j < 4) steps(IntC<2>());
      else if (j < 6) steps(IntC<3>());
      else steps(IntC<4>());
    };
    {
      // ---- 16 rows of S in K S_0, half of the tokens ----
      const SplitA a = load_a(sm + L::S + w * 384, lane);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int j = half * 4 + i;
        SplitAcc c;
        const float* row = Ks + (8 * j + g) * D;
        const float2 x = *reinterpret_cast<const float2*>(row + ((16 * w + t2) ^ turn)), y = *reinterpret_cast<const float2*>(row + ((16 * w + 8 + t2) ^ turn));
        mma_split<true>(a, split_b(x.x, x.y, y.x, y.y), c);
        *reinterpret_cast<float4*>(sm + L::Red + (w * 8 + j) * 128 + lane * 4) = make_float4(c.sum(0), c.sum(1), c.sum(2), c.sum(3));
      }
    }
    __syncthreads();
    float y[TW][4];                                       // second half: columns g, g + 8 of tokens t2, t2 + 1 of the read-out
    if (half == 0) {
#pragma unroll
      for (int i = 0; i < TW; ++i) {
        const int j = w + i * KS;
        float z[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < KS; ++k) {
          const float4 r = *reinterpret_cast<const float4*>(sm + L::Red + (k * 8 + j) * 128 + lane * 4);
          z[0] += r.x; z[1] += r.y; z[2] += r.z; z[3] += r.w;
        }
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const int t = 8 * j + t2 + (x & 1);
          z[x] = cs[2 * kDcC + t] * (v[i][x] - cs[t] * z[x]);
          odd |= not_finite(z[x]);
        }
        store_half_a(sm + L::R + (j >> 1) * 384, lane, j & 1, z);
      }
      odd = half_or<KS * 32>(odd);
#pragma unroll
      for (int i = 0; i < TW; ++i) {
        const int j = w + i * KS;
        float z[4];
        times_lower(sm + L::T, sm + L::R, j, z);
#pragma unroll
        for (int x = 0; x < 4; ++x) odd |= not_finite(z[x]);
        store_half_a(sm + L::U + (j >> 1) * 384, lane, j & 1, z);
#pragma unroll
        for (int x = 0; x < 4; ++x) z[x] *= cs[kDcC + 8 * j + t2 + (x & 1)];
        store_half_a(sm + L::UD + (j >> 1) * 384, lane, j & 1, z);
      }
    } else {
      // ---- Q S_0 ----
      SplitAcc c[TW][2];
#pragma unroll
      for (int s = 0; s < KS; ++s) {
        const SplitA a = load_a(sm + L::S + s * 384, lane);
#pragma unroll
        for (int i = 0; i < TW; ++i) {
          const SplitB b = load_b(sm + L::Q + ((w + i * KS) * KS + s) * kDcB);
          if (s < 2) mma_split<true>(a, b, c[i][s & 1]);
          else mma_split(a, b, c[i][s & 1]);
        }
      }
#pragma unroll
      for (int i = 0; i < TW; ++i)
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          y[i][x] = c[i][0].sum(x) + c[i][1].sum(x);
          odd |= not_finite(y[i][x]);
          y[i][x] *= cs[8 * (w + i * KS) + t2 + (x & 1)];
        }
    }
    if (__syncthreads_or(odd)) {                          // S is still the one in front of the chunk
#pragma unroll
      for (int x = 0; x < 4; ++x) sm[L::Red + (16 * w + 8 * half + t2 + (x & 1)) * 16 + g + (x >> 1) * 8] = S[x];
      if (more) mbar_wait(kp_bar(tile + 1), (uint32_t)((tile + 1 - t_lo) >> 1) & 1u);      // what is on its way arrives before the CTA leaves
      __syncthreads();
      walk_on<D>(p, sm, h, col0, first, at, min(len, (t_hi - tb) * kDcC), sp);
      return;
    }
    if (asks && more) ask_qt(tile + 1);
    {
      // ---- S = c_64 S + K^T (r_64 U) ----
      SplitAcc c[2];
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const int d = 16 * w + 8 * half + g, r = 16 * s + t2;
        const float* kc = Ks + r * D;
        const int e0 = d ^ dc_turn(t2), e1 = d ^ dc_turn(t2 + 1);
        const SplitB b = split_b(kc[e0], kc[D + e1], kc[8 * D + e0], kc[9 * D + e1]);
        const SplitA a = load_a(sm + L::UD + s * 384, lane);
        if (s < 2) mma_split<true>(a, b, c[s & 1]);
        else mma_split(a, b, c[s & 1]);
      }
      const float ce = cs[kDcC - 1];
#pragma unroll
      for (int x = 0; x < 4; ++x) S[x] = fmaf(S[x], ce, c[0].sum(x) + c[1].sum(x));
      store_half_a(sm + L::S + w * 384, lane, half, S);
    }
    if (half == 1) {
      // ---- the read-out ----
#pragma unroll
      for (int i = 0; i < TW; ++i) {
        const int t8 = 8 * (w + i * KS);
        float z[4];
        times_lower(Ps, sm + L::U, w + i * KS, z);
        float* orow = p.o + ((long long)(first + at + t8) * p.H + h) * p.Dv + col0 + g;
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const int t = t2 + (x & 1);
          if (t8 + t < n) orow[(long long)t * p.H * p.Dv + (x >> 1) * 8] = y[i][x] + z[x];
        }
      }
    }
  }
#pragma unroll
  for (int x = 0; x < 4; ++x) sp[s_at(x)] = S[x];
}

template <int D>
static int run_windows(DeltaChunkArgs p, int bound, int window, cudaStream_t st) {
  constexpr int smem = prep_smem<D>();
  auto prep = delta_chunk_prep_kernel<D>;
  B200_CHECK(cudaFuncSetAttribute(prep, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  constexpr int scan_smem = DcSmem<D>::kTotal * 4;
  auto scan = delta_chunk_scan_kernel<D>;
  B200_CHECK(cudaFuncSetAttribute(scan, cudaFuncAttributeMaxDynamicSharedMemorySize, scan_smem));
  for (int lo = 0; lo < bound; lo += window) {
    p.tile_lo = lo;
    p.tile_hi = lo + window < bound ? lo + window : bound;
    prep<<<dim3(p.tile_hi - lo, p.G), 256, smem, st>>>(p);
    B200_LAUNCH_CHECK();
    scan<<<dim3(p.Dv / kDcNC, p.H, p.n_runs), DcSmem<D>::kThreads, scan_smem, st>>>(p);
    B200_LAUNCH_CHECK();
  }
  return 0;
}
}  // namespace b200

// Workspace (floats) for a step of `tokens` tokens in n_runs runs, whatever its q/k heads and key size are; bounded, however long the step is.
B200_API long long b200_delta_chunk_workspace(int tokens, int n_runs, int H) {
  using namespace b200;
  const long long all = ((long long)tokens / kDcC + n_runs) * (kDcHead + dc_kv(128));
  return H * (all < kDcMost ? all : kDcMost);
}

// Arguments as in b200_linear_scan (mode 3), `runs` present; `ws`: b200_delta_chunk_workspace floats. B200_ERR_UNSUPPORTED: the caller
// takes b200_linear_scan.
B200_API int b200_delta_chunk_scan(const float* q, long long ldq, const float* k, long long ldk, const float* v, long long ldv, const float* g,
                                   long long ldg, const float* beta, long long ldb, float* state, const int* runs, int n_runs, float* o,
                                   float* ws, int tokens, int H, int G, int D, int Dv, void* stream) {
  using namespace b200;
  if (n_runs <= 0 || tokens <= 0) return 0;
  if (H <= 0 || G <= 0 || H % G || H > 65535 || n_runs > 65535) return B200_ERR_BAD_SHAPE;
  auto al = [](const void* x, long long ld) { return !(reinterpret_cast<uintptr_t>(x) & 15) && ld % 4 == 0; };
  if ((D != 64 && D != 128) || Dv % 16 || !al(q, ldq) || !al(k, ldk) || !al(v, ldv) || !al(state, 0) || !al(o, 0) || !al(ws, 0) || !runs)
    return B200_ERR_UNSUPPORTED;
  DeltaChunkArgs p = {q, k, v, g, beta, ldq, ldk, ldv, ldg, ldb, state, o, ws, runs, n_runs, H, G, Dv, 0, 0, 0};
  const long long bound = (long long)tokens / kDcC + n_runs;      // a run of n tokens has at most n / 64 + 1 chunks
  if (bound > 0x7fffffffLL) return B200_ERR_TOO_LARGE;
  const long long holds = b200_delta_chunk_workspace(tokens, n_runs, H) / ((long long)H * kDcHead + (long long)G * dc_kv(D));
  const long long windows = (bound + holds - 1) / holds;
  const int window = (int)((bound + windows - 1) / windows);
  p.kv_ws = (long long)window * H * kDcHead;
  return D == 64 ? run_windows<64>(p, (int)bound, window, (cudaStream_t)stream) : run_windows<128>(p, (int)bound, window, (cudaStream_t)stream);
}
