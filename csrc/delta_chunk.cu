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
//   delta_chunk_prep_kernel   a CTA per (chunk, q/k head): K K^T and Q K^T; then per head, 64 threads each: T = (I + A)^-1 by forward
//                             substitution (a thread owns a column, rows of A are read as broadcasts), P_ij = r_ij (q_i . k_j),
//                             c_i and r_64,j -> workspace. Chunks do not wait for one another.
//   delta_chunk_scan_kernel   a CTA per (run, head, block of 16 value columns) walks the chunks with its columns of S in registers
//                             and, for the products, in shared memory: [K; Q] S_0, U = T R, O += P U, S += K^T U. What the next
//                             chunk needs is on its way (bulk copies) meanwhile.
// All in fp32 FMAs (two per instruction), no tensor cores: the state is fp32 by definition, and splitting fp32 operands for bf16 or
// tf32 mma.sync takes as many cycles as the FMAs do. r_ij is a product taken from j upwards, the roundings a walk makes too;
// sums of logarithms would lose digits to cancellation. Bound: a packed FMA takes 3.0 cycles of a scheduler with three operands of its own and
// 2.3 where one is the last one's too, as here, not 2 (85 and 109 FMAs a cycle and SM of 128, measured alone, two to four warps per
// scheduler), 4800 of a chunk's 11 800 cycles; then the latency of the sums across lanes and the four barriers of a chunk. One prompt
// of 2048 tokens, 16 heads of 128 x 128 over 4 q/k heads: 502 us token by token, 18 + 194 here; 2048 and 513 tokens: 586 -> 272 (the
// shorter run's CTAs fill in behind the longer one's); error of the state against 64 bits 2e-7 both ways.
#include "common.cuh"
#include "../include/b200_ops.h"

namespace b200 {

constexpr int kDcC = 64, kDcCP = kDcC + 4;                // tokens of a chunk; padded row of a [64, 64] matrix
constexpr long long kDcWs = 2 * kDcC * kDcC + 2 * kDcC;   // floats of workspace per (chunk, head): T, P, c, r_64

struct DeltaChunkArgs {
  const float *q, *k, *v, *g, *beta;
  long long ldq, ldk, ldv, ldg, ldb;
  float *state, *o, *ws;
  const int* runs;
  int n_runs, H, G, Dv, tile_lo, tile_hi;                 // chunks [tile_lo, tile_hi) of all the step's chunks, counted run by run
};

// 16 bytes on their way to shared memory; zeros where `live` is false
__device__ __forceinline__ void dc_copy16(float* dst, const float* src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void dc_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ float2 lo2(const float4& v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4& v) { return make_float2(v.z, v.w); }

template <int D> constexpr int prep_smem() {              // K | Q (later the four heads' A), K K^T | Q K^T, a | beta of four heads
  constexpr int tiles = 2 * kDcC * (D + 4), as = 4 * kDcC * kDcCP;
  return ((tiles > as ? tiles : as) + 2 * kDcC * kDcCP + 4 * 2 * kDcC) * 4;
}

template <int D>
__global__ void __launch_bounds__(256, 2)
delta_chunk_prep_kernel(const DeltaChunkArgs p) {
  constexpr int DP = D + 4;
  extern __shared__ __align__(16) float sm[];
  constexpr int kTiles = 2 * kDcC * DP, kAs = 4 * kDcC * kDcCP;
  float* Ks = sm;
  float* Qs = sm + kDcC * DP;
  float* KK = sm + (kTiles > kAs ? kTiles : kAs);
  float* QK = KK + kDcC * kDcCP;
  float* AB = QK + kDcC * kDcCP;                          // [4 heads][a 64 | beta 64]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tile = p.tile_lo + blockIdx.x, kvh = blockIdx.y, rep = p.H / p.G;
  int first = 0, n = 0;
  for (int r = 0, at = 0; r < p.n_runs; ++r) {
    const int len = p.runs[4 * r + 1], nt = (len + kDcC - 1) / kDcC;
    if (tile < at + nt) { first = p.runs[4 * r] + (tile - at) * kDcC; n = min(kDcC, len - (tile - at) * kDcC); break; }
    at += nt;
  }
  if (n <= 0) return;                                     // the grid counts a chunk more per run than there may be
  for (int i = tid; i < kDcC * (D / 4); i += 256) {
    const int t = i / (D / 4), d = i % (D / 4) * 4;
    const long long row = first + min(t, n - 1);
    dc_copy16(Ks + t * DP + d, p.k + row * p.ldk + (long long)kvh * D + d, t < n);
    dc_copy16(Qs + t * DP + d, p.q + row * p.ldq + (long long)kvh * D + d, t < n);
  }
  dc_wait_all();
  __syncthreads();
  {
    const int rl = lane >> 2, cl = lane & 3, row0 = (warp & 1) * 32 + rl, col0 = (warp >> 1) * 16 + cl;
    float2 ak[4][4], aq[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) ak[i][j] = aq[i][j] = make_float2(0.f, 0.f);
    if ((warp & 1) || warp < 4) {                         // rows 0 .. 31 x columns 32 .. 63 lie above the diagonal
#pragma unroll 2
      for (int d = 0; d < D; d += 4) {
        float4 b[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(Ks + (col0 + 4 * j) * DP + d);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 x = *reinterpret_cast<const float4*>(Ks + (row0 + 8 * i) * DP + d);
          const float4 y = *reinterpret_cast<const float4*>(Qs + (row0 + 8 * i) * DP + d);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            ak[i][j] = __ffma2_rn(lo2(x), lo2(b[j]), ak[i][j]);
            aq[i][j] = __ffma2_rn(lo2(y), lo2(b[j]), aq[i][j]);
            ak[i][j] = __ffma2_rn(hi2(x), hi2(b[j]), ak[i][j]);
            aq[i][j] = __ffma2_rn(hi2(y), hi2(b[j]), aq[i][j]);
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        KK[(row0 + 8 * i) * kDcCP + col0 + 4 * j] = ak[i][j].x + ak[i][j].y;
        QK[(row0 + 8 * i) * kDcCP + col0 + 4 * j] = aq[i][j].x + aq[i][j].y;
      }
  }
  __syncthreads();                                        // K and Q are read: their place takes the heads' A
  const int grp = tid >> 6, j = tid & 63;
  float* As = sm + grp * kDcC * kDcCP;
  float* a_ = AB + grp * 2 * kDcC;
  float* b_ = a_ + kDcC;
  for (int hh = grp; hh < rep; hh += 4) {
    const int h = kvh * rep + hh;
    a_[j] = j < n ? p.g[(long long)(first + j) * p.ldg + h] : 1.f;
    b_[j] = j < n ? p.beta[(long long)(first + j) * p.ldb + h] : 0.f;
    asm volatile("bar.sync %0, 64;" ::"r"(1 + grp) : "memory");
    float* T = p.ws + ((long long)(tile - p.tile_lo) * p.H + h) * kDcWs;
    float* P = T + kDcC * kDcC;
    float r = 1.f, c = 1.f;
    for (int i = 0; i < kDcC; ++i) {
      const float a = a_[i];
      if (i <= j) c *= a;
      if (i > j) r *= a;
      As[i * kDcCP + j] = i > j ? b_[i] * r * KK[i * kDcCP + j] : 0.f;
      P[i * kDcC + j] = i >= j ? r * QK[i * kDcCP + j] : 0.f;
    }
    P[kDcC * kDcC + j] = c;
    P[kDcC * kDcC + kDcC + j] = r;
    asm volatile("bar.sync %0, 64;" ::"r"(1 + grp) : "memory");
    float x[kDcC];                                        // column j of the inverse
#pragma unroll
    for (int i = 0; i < kDcC; ++i) x[i] = 0.f;
#pragma unroll
    for (int i = 0; i < kDcC; ++i) {
      float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
      for (int m = 0; m < i; m += 4) {                    // A is zero from the diagonal on, x from i on
        const float4 a4 = *reinterpret_cast<const float4*>(As + i * kDcCP + m);
        s0 = fmaf(a4.x, x[m], s0); s1 = fmaf(a4.y, x[m + 1], s1); s2 = fmaf(a4.z, x[m + 2], s2); s3 = fmaf(a4.w, x[m + 3], s3);
      }
      x[i] = (i == j ? 1.f : 0.f) - ((s0 + s1) + (s2 + s3));
      T[i * kDcC + j] = x[i];
    }
    asm volatile("bar.sync %0, 64;" ::"r"(1 + grp) : "memory");   // the next head's a, beta and A overwrite these
  }
}

constexpr int kDcNC = 16;                                 // value columns of a CTA: 128 CTAs for 16 heads of 128

template <int D> struct DcSmem {                          // float offsets
  static constexpr int NC = kDcNC;
  static constexpr int DP = D + 4;
  static constexpr int K = 0, Q = K + 2 * kDcC * DP, T = Q + kDcC * DP, P = T + kDcC * kDcCP, V = P + 2 * kDcC * kDcCP, S = V + 2 * kDcC * NC,
                       R = S + D * NC, U = R + kDcC * NC, UD = U + kDcC * NC, X = UD + kDcC * NC,
                       Bar = X + 2 * 3 * kDcC, kTotal = Bar + 8;       // X: c | r_64 | beta, twice; Bar: K, V, P, X of each buffer, Q and T
};

// Where columns c, c + 1 (c even) of the pair of rows pr lie in a [rows / 2][16][2] array: 16 bytes, the two halves of 32 changing places
// with every other two pairs so that the eight lane groups of a warp read and write different banks
__device__ __forceinline__ int pair_at(int pr, int c) { return pr * (2 * kDcNC) + (((c >> 1) ^ (pr >> 1 & 1)) << 2); }

// NR rows' sums over 4 N2 elements (every eighth group of four, the lane's own) times four columns held as pairs of rows: with two warps per scheduler it is the rows beside one
// another that keep the FMA pipe busy
template <int NR, int N2>
__device__ __forceinline__ void dot_rows(const float* rows, int stride, const float2 (&m)[2 * N2][4], float4 (&out)[NR]) {
  float2 acc[NR][4];
#pragma unroll
  for (int r = 0; r < NR; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[r][c] = make_float2(0.f, 0.f);
#pragma unroll
  for (int x = 0; x < N2; ++x) {
    float4 a[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) a[r] = *reinterpret_cast<const float4*>(rows + r * stride + 32 * x);
#pragma unroll
    for (int r = 0; r < NR; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[r][c] = __ffma2_rn(lo2(a[r]), m[2 * x][c], acc[r][c]);
#pragma unroll
    for (int r = 0; r < NR; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[r][c] = __ffma2_rn(hi2(a[r]), m[2 * x + 1][c], acc[r][c]);
  }
#pragma unroll
  for (int r = 0; r < NR; ++r)
    out[r] = make_float4(acc[r][0].x + acc[r][0].y, acc[r][1].x + acc[r][1].y, acc[r][2].x + acc[r][2].y, acc[r][3].x + acc[r][3].y);
}

// Four columns' parts in the eight lanes that share them (lane bits 2, 3, 4) -> the sum of column 2 (bit 4) + (bit 3): each step hands
// half of what is left to the lane across
__device__ __forceinline__ float gather4(const float4& v, int lane) {
  const bool b4 = lane & 16, b3 = lane & 8;
  const float x = (b4 ? v.z : v.x) + __shfl_xor_sync(0xffffffffu, b4 ? v.x : v.z, 16);
  const float y = (b4 ? v.w : v.y) + __shfl_xor_sync(0xffffffffu, b4 ? v.y : v.w, 16);
  const float z = (b3 ? y : x) + __shfl_xor_sync(0xffffffffu, b3 ? x : y, 8);
  return z + __shfl_xor_sync(0xffffffffu, z, 4);
}

// Row t of a lower triangle times column c of X, in the layout of R and U: the columns above the diagonal are zero, and here they are not
// multiplied either. dot_rows multiplies them, which is the same unless X holds an infinity or NaN: then it would reach rows, tokens, that
// come before its own. So a chunk with such an R or U takes this one (a vote with the barriers that are there anyway).
__device__ __forceinline__ float lower_dot(const float* row, const float* X, int t, int c) {
  float s = 0.f;
  for (int j = 0; j <= t; ++j) s = fmaf(row[j], X[pair_at(j >> 1, c) + (c & 1) * 2 + (j & 1)], s);
  return s;
}
__device__ __forceinline__ bool not_finite(float x) { return !(fabsf(x) <= 3.402823466e38f); }

// an "or" over the 256 threads of the chain's warps, and a barrier for them
__device__ __forceinline__ int chain_or(int x) {
  int r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\t"
      "barrier.cta.red.or.pred q, 1, 256, p;\n\tselp.s32 %0, 1, 0, q;\n\t}" : "=r"(r) : "r"(x) : "memory");
  return r;
}

// What limits the walk is shared memory, 128 bytes a cycle into registers against 128 FMAs: a tile of 4 x 4 outputs per thread would
// take two bytes per FMA. So the small side of every product but the last stays in registers — S_0 with 16 rows of four columns in
// every lane of every warp, R and U with eight — and a row of the other side costs one byte per FMA; the lanes' parts of
// a row meet in four shuffles. Shared layouts: S, R and U hold pairs of neighbouring rows of one column side by side
// ([rows / 2][16][2], pair_at), the pairs a packed FMA takes.
// What the next chunk waits for is only K S_0, U = T R and S += K^T U. Warps 0-7, the chain, do these; warps 8-15 read out beside them: Q S_0
// while the chain is at K S_0 and T R, then P U while it is at K^T U. Eight warps for all of it one after the other and copies of 16 bytes
// by all of them: 262 us for runs of 2048 and 513 tokens, 245 now; the halves alone, with those copies, gave nothing (264).
template <int D>
__global__ void __launch_bounds__(512, 1)
delta_chunk_scan_kernel(const DeltaChunkArgs p) {
  using L = DcSmem<D>;
  constexpr int NC = kDcNC, DP = L::DP, DT = D / 32;     // DT: state rows of a thread
  extern __shared__ __align__(16) float sm[];
  const int h = blockIdx.y, col0 = blockIdx.x * NC, run = blockIdx.z;
  int tb = 0;
  for (int r = 0; r < run; ++r) tb += (p.runs[4 * r + 1] + kDcC - 1) / kDcC;
  const int first = p.runs[4 * run], len = p.runs[4 * run + 1], p0 = p.runs[4 * run + 2], slot = p.runs[4 * run + 3];
  const int t_lo = max(tb, p.tile_lo), t_hi = min(tb + (len + kDcC - 1) / kDcC, p.tile_hi);
  if (t_lo >= t_hi) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = (tid >> 5) & 7;    // the warp's place in its half
  const bool chain = tid < 256;
  const int rl = lane >> 2, cb = (lane & 3) * 4;          // this thread's four columns
  const int cg = cb + (lane >> 4) * 2 + (lane >> 3 & 1);  // and the one whose sum over the warp it ends up with (gather4)
  const int kvh = h / (p.H / p.G), t8 = warp * 8;         // a warp's eight tokens of a chunk

  // What a chunk needs comes a row at a time by bulk copies, one to a thread of the reading half: cp.async pieces of 16 bytes took all warps
  // 2400 of a chunk's 12 700 cycles to ask for. A barrier is armed one barrier of the CTA before its copies are asked for.
  const uint32_t bar = smem_u32(sm + L::Bar);
  auto kvp_bar = [&](int tile) { return bar + 8u * (tile & 1); };
  const uint32_t qt_bar = bar + 16;
  auto rows_of = [&](int tile) { return min(kDcC, len - (tile - tb) * kDcC); };
  auto arm_kvp = [&](int tile) { mbar_arrive_expect_tx(kvp_bar(tile), (uint32_t)(rows_of(tile) * (D + NC) + kDcC * kDcC + 2 * kDcC) * 4u); };
  auto arm_qt = [&](int tile) { mbar_arrive_expect_tx(qt_bar, (uint32_t)(rows_of(tile) * D + kDcC * kDcC) * 4u); };
  const int ri = tid - 256;                               // place in the reading half
  auto row_copy = [&](float* dst, const float* src, int floats, bool there, uint32_t b) {
    if (there) bulk_load_1d(smem_u32(dst), src, floats * 4, b);
    else
      for (int i = 0; i < floats; i += 4) *reinterpret_cast<float4*>(dst + i) = make_float4(0.f, 0.f, 0.f, 0.f);     // tokens past the end
  };
  auto ask_kvp = [&](int tile) {
    const int buf = tile & 1, n = rows_of(tile), j = ri & 63;
    const long long row = first + (tile - tb) * kDcC + min(j, n - 1);
    const float* w = p.ws + ((long long)(tile - p.tile_lo) * p.H + h) * kDcWs + kDcC * kDcC;
    if (ri < 64) row_copy(sm + L::K + (buf * kDcC + j) * DP, p.k + row * p.ldk + (long long)kvh * D, D, j < n, kvp_bar(tile));
    else if (ri < 128) row_copy(sm + L::V + (buf * kDcC + j) * NC, p.v + row * p.ldv + (long long)h * p.Dv + col0, NC, j < n, kvp_bar(tile));
    else if (ri < 192) row_copy(sm + L::P + (buf * kDcC + j) * kDcCP, w + j * kDcC, kDcC, true, kvp_bar(tile));
    else {
      if (j == 0) row_copy(sm + L::X + buf * 3 * kDcC, w + kDcC * kDcC, 2 * kDcC, true, kvp_bar(tile));
      sm[L::X + buf * 3 * kDcC + 2 * kDcC + j] = j < n ? p.beta[row * p.ldb + h] : 0.f;
    }
  };
  auto ask_qt = [&](int tile) {
    const int n = rows_of(tile), j = ri & 63;
    const long long row = first + (tile - tb) * kDcC + min(j, n - 1);
    const float* w = p.ws + ((long long)(tile - p.tile_lo) * p.H + h) * kDcWs;
    if (ri < 64) row_copy(sm + L::Q + j * DP, p.q + row * p.ldq + (long long)kvh * D, D, j < n, qt_bar);
    else if (ri < 128) row_copy(sm + L::T + j * kDcCP, w + j * kDcC, kDcC, true, qt_bar);
  };
  if (tid == 256) {
    for (int i = 0; i < 3; ++i) mbar_init(bar + 8 * i, 1);
    fence_mbar_init();
    arm_kvp(t_lo);
    arm_qt(t_lo);
    if (t_lo + 1 < t_hi) arm_kvp(t_lo + 1);
  }
  __syncthreads();
  if (!chain) {
    ask_kvp(t_lo);
    ask_qt(t_lo);
  }

  // the state: rows d0 .. d0 + DT of four columns, in pairs of rows, kept by the first four warps; the chain's other four add up the second
  // half of each chunk's tokens
  const int d0 = ((warp & 3) * 8 + rl) * DT;
  float* sp = p.state + (((long long)slot * p.H + h) * D) * p.Dv + col0 + cb;
  float2 S[DT / 2][4];
  const bool from_state = p0 > 0 || t_lo > tb, owner = tid < 128;
#pragma unroll
  for (int x = 0; x < DT / 2; ++x) {
    float4 s0 = make_float4(0.f, 0.f, 0.f, 0.f), s1 = s0;
    if (from_state && owner) {
      s0 = *reinterpret_cast<const float4*>(sp + (long long)(d0 + 2 * x) * p.Dv);
      s1 = *reinterpret_cast<const float4*>(sp + (long long)(d0 + 2 * x + 1) * p.Dv);
    }
    S[x][0] = make_float2(s0.x, s1.x); S[x][1] = make_float2(s0.y, s1.y); S[x][2] = make_float2(s0.z, s1.z); S[x][3] = make_float2(s0.w, s1.w);
  }
  auto publish_state = [&]() {
#pragma unroll
    for (int x = 0; x < DT / 2; ++x) {
      *reinterpret_cast<float4*>(sm + L::S + pair_at(d0 / 2 + x, cb)) = make_float4(S[x][0].x, S[x][0].y, S[x][1].x, S[x][1].y);
      *reinterpret_cast<float4*>(sm + L::S + pair_at(d0 / 2 + x, cb + 2)) = make_float4(S[x][2].x, S[x][2].y, S[x][3].x, S[x][3].y);
    }
  };
  if (owner) publish_state();

  // N pairs of pairs of rows of S, R or U, every eighth of them the lane's own
  auto hold = [&](const float* X, auto& B) {
    constexpr int N = sizeof(B) / sizeof(B[0]);
#pragma unroll
    for (int x = 0; x < N; ++x) {
      const int pr = ((x >> 1) * 8 + rl) * 2 + (x & 1);
      const float4 b0 = *reinterpret_cast<const float4*>(X + pair_at(pr, cb)), b1 = *reinterpret_cast<const float4*>(X + pair_at(pr, cb + 2));
      B[x][0] = lo2(b0); B[x][1] = hi2(b0); B[x][2] = lo2(b1); B[x][3] = hi2(b1);
    }
  };
  // eight rows of a [64, D] tile times the state: column cg of rows t8 .. t8 + 7
  auto times_state = [&](const float* rows, float (&y)[8]) {
    float2 s0[D / 16][4];
    hold(sm + L::S, s0);
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      float4 z[2];
      dot_rows<2, D / 32>(rows + (t8 + i) * DP + rl * 4, DP, s0, z);
      y[i] = gather4(z[0], lane);
      y[i + 1] = gather4(z[1], lane);
    }
  };
  // eight rows of a lower triangle times X (R or U); `odd`: X holds an infinity or NaN
  auto times_lower = [&](const float* rows, const float* X, int odd, float (&y)[8]) {
    float2 B[4][4];
    hold(X, B);
#pragma unroll
    for (int i = 0; i < 8; i += 4) {
      float4 z[4];
      dot_rows<4, 2>(rows + (t8 + i) * kDcCP + rl * 4, kDcCP, B, z);
#pragma unroll
      for (int e = 0; e < 4; ++e) y[i + e] = gather4(z[e], lane);
    }
    if (odd) {
#pragma unroll
      for (int i = 0; i < 8; ++i) y[i] = lower_dot(rows + (t8 + i) * kDcCP, X, t8 + i, cg);
    }
  };

  for (int tile = t_lo; tile < t_hi; ++tile) {
    const int buf = tile & 1;
    const int at = (tile - tb) * kDcC, n = min(kDcC, len - at);
    const bool more = tile + 1 < t_hi, live = t8 < n;
    mbar_wait(kvp_bar(tile), (uint32_t)((tile - t_lo) >> 1) & 1u);
    mbar_wait(qt_bar, (uint32_t)(tile - t_lo) & 1u);
    __syncthreads();                                      // and S, and beta
    if (!chain && more) {
      if (ri == 0) {
        arm_qt(tile + 1);
        if (tile + 2 < t_hi) arm_kvp(tile + 2);           // this chunk's barrier: all have waited for it
      }
      ask_kvp(tile + 1);
    }
    const float* Ks = sm + L::K + buf * kDcC * DP;
    const float* cs = sm + L::X + buf * 3 * kDcC;         // c | r_64 | beta
    int odd = 0;                                          // an infinity or NaN among this thread's part of R, then of U
    float y[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) y[i] = 0.f;
    if (chain) {
      if (live) {
        times_state(Ks, y);                               // K S_0
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          y[i] = cs[2 * kDcC + t8 + i] * (sm[L::V + (buf * kDcC + t8 + i) * NC + cg] - cs[t8 + i] * y[i]);
          odd |= not_finite(y[i]);
        }
      }
      if (!(lane & 4)) {
#pragma unroll
        for (int i = 0; i < 8; i += 2) *reinterpret_cast<float2*>(sm + L::R + pair_at((t8 + i) / 2, cg) + (cg & 1) * 2) = make_float2(y[i], y[i + 1]);
      }
      odd = chain_or(odd);
      float u[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) u[i] = 0.f;
      if (live) {
        times_lower(sm + L::T, sm + L::R, odd, u);
#pragma unroll
        for (int i = 0; i < 8; ++i) odd |= not_finite(u[i]);
      }
      if (!(lane & 4)) {
#pragma unroll
        for (int i = 0; i < 8; ++i) sm[L::UD + (t8 + i) * NC + cg] = cs[kDcC + t8 + i] * u[i];
#pragma unroll
        for (int i = 0; i < 8; i += 2) *reinterpret_cast<float2*>(sm + L::U + pair_at((t8 + i) / 2, cg) + (cg & 1) * 2) = make_float2(u[i], u[i + 1]);
      }
    } else if (live) {
      times_state(sm + L::Q, y);                          // Q S_0
#pragma unroll
      for (int i = 0; i < 8; ++i) y[i] *= cs[t8 + i];
    }
    odd = __syncthreads_or(odd);
    if (!chain) {
      if (more) ask_qt(tile + 1);
      // ---- the read-out ----
      if (live) {
        float z[8];
        times_lower(sm + L::P + buf * kDcC * kDcCP, sm + L::U, odd, z);
        float* orow = p.o + ((long long)(first + at) * p.H + h) * p.Dv + col0 + cg;
        if (!(lane & 4)) {
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (t8 + i < n) orow[(long long)(t8 + i) * p.H * p.Dv] = y[i] + z[i];
        }
      }
      continue;
    }
    // ---- S = c_64 S + K^T (r_64 U) ----
    const float2 ce = make_float2(cs[kDcC - 1], cs[kDcC - 1]);
#pragma unroll
    for (int x = 0; x < DT / 2; ++x)
#pragma unroll
      for (int c = 0; c < 4; ++c) S[x][c] = owner ? __fmul2_rn(S[x][c], ce) : make_float2(0.f, 0.f);
    const int t_end = owner ? min(n, kDcC / 2) : n;
#pragma unroll 8
    for (int t = owner ? 0 : kDcC / 2; t < t_end; ++t) {
      float2 a[DT / 2];
      if (DT == 4) {
        const float4 a4 = *reinterpret_cast<const float4*>(Ks + t * DP + d0);
        a[0] = lo2(a4); a[DT / 2 - 1] = hi2(a4);
      } else a[0] = *reinterpret_cast<const float2*>(Ks + t * DP + d0);
      const float4 u = *reinterpret_cast<const float4*>(sm + L::UD + t * NC + cb);
#pragma unroll
      for (int x = 0; x < DT / 2; ++x) {
        S[x][0] = __ffma2_rn(a[x], make_float2(u.x, u.x), S[x][0]); S[x][1] = __ffma2_rn(a[x], make_float2(u.y, u.y), S[x][1]);
        S[x][2] = __ffma2_rn(a[x], make_float2(u.z, u.z), S[x][2]); S[x][3] = __ffma2_rn(a[x], make_float2(u.w, u.w), S[x][3]);
      }
    }
    if (!owner) publish_state();                          // the products with the old S ended in front of the last barrier
    asm volatile("bar.sync 1, 256;" ::: "memory");
    if (owner) {
#pragma unroll
      for (int x = 0; x < DT / 2; ++x) {
        const float4 a = *reinterpret_cast<const float4*>(sm + L::S + pair_at(d0 / 2 + x, cb)), b = *reinterpret_cast<const float4*>(sm + L::S + pair_at(d0 / 2 + x, cb + 2));
        S[x][0].x += a.x; S[x][0].y += a.y; S[x][1].x += a.z; S[x][1].y += a.w;
        S[x][2].x += b.x; S[x][2].y += b.y; S[x][3].x += b.z; S[x][3].y += b.w;
      }
      publish_state();
    }
  }
  if (!owner) return;
#pragma unroll
  for (int x = 0; x < DT / 2; ++x) {
    *reinterpret_cast<float4*>(sp + (long long)(d0 + 2 * x) * p.Dv) = make_float4(S[x][0].x, S[x][1].x, S[x][2].x, S[x][3].x);
    *reinterpret_cast<float4*>(sp + (long long)(d0 + 2 * x + 1) * p.Dv) = make_float4(S[x][0].y, S[x][1].y, S[x][2].y, S[x][3].y);
  }
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
    scan<<<dim3(p.Dv / kDcNC, p.H, p.n_runs), 512, scan_smem, st>>>(p);
    B200_LAUNCH_CHECK();
  }
  return 0;
}
}  // namespace b200

// Workspace (floats) for a step of `tokens` tokens in n_runs runs: chunks are taken in windows of at most 128, however long the step is.
B200_API long long b200_delta_chunk_workspace(int tokens, int n_runs, int H) {
  using namespace b200;
  const long long bound = (long long)tokens / kDcC + n_runs;
  return (bound < 128 ? bound : 128) * H * kDcWs;
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
  DeltaChunkArgs p = {q, k, v, g, beta, ldq, ldk, ldv, ldg, ldb, state, o, ws, runs, n_runs, H, G, Dv, 0, 0};
  const long long bound = (long long)tokens / kDcC + n_runs;      // a run of n tokens has at most n / 64 + 1 chunks
  if (bound > 0x7fffffffLL) return B200_ERR_TOO_LARGE;
  const int window = bound < 128 ? (int)bound : 128;
  return D == 64 ? run_windows<64>(p, (int)bound, window, (cudaStream_t)stream) : run_windows<128>(p, (int)bound, window, (cudaStream_t)stream);
}
