// Gated linear attention with a decay per key channel, over the runs of a ragged serving step (see linear_scan.cu for runs,
// state rows and the other scan modes). All arithmetic is fp32.
//
//   b200_lowrank_decay   a[t, c] = sigmoid(sum_r w2[c, r] x[t, r] + bias[c])^(1 / tau), formed as exp(log sigmoid(.) / tau), or
//                        exp(-exp(sum_r w2[c, r] tanh(x[t, r]) + bias[c]))
//   b200_channel_scan    per head, state S [D, Dv] (fp32, in `state` [rows, H, D, Dv]):
//                            S <- diag(g_t) S + k_t v_t^T ;   o_t = S^T q_t                      (u NULL)
//                            o_t = (S + diag(u) k_t v_t^T)^T q_t ;   S <- diag(g_t) S + k_t v_t^T  (u [H, D]: a bonus for the
//                            current token, which the read-out sees before the state decays)
//
// A run is walked token by token, but the recurrence is linear, so a long run need not be walked by one CTA: it is cut into
// tiles (64 tokens), and
//   pass 1  every tile but a run's last forms its local state (from zero) and the product of its decays,
//   carry   per element of S, the tiles of a run are chained: incoming state of tile j + 1 = decay_j * incoming_j + local_j,
//   pass 2  every tile is walked again from its incoming state and writes its outputs; the last one leaves the run's state.
// Runs of at most one tile (decode batches, short pieces) take pass 0: one walk from and to the state row. Passes 1 and 2 of square states (64 or
// 128) on whole vectors go by products of matrices (channel_tile_kernel), other sizes token by token.
//
// Columns of S are independent. A thread owns R rows of CPT columns, LPC lanes share a column and reduce their parts of an
// output by shuffles (each step halves the columns a lane still carries), a CTA owns a block of columns of one (run or tile,
// head). k, q, g and v of a chunk of tokens are staged through shared memory by cp.async, one chunk ahead.
#include "common.cuh"
#include "split_mma.cuh"
#include "../include/b200_ops.h"

namespace b200 {

constexpr int kCsR = 16, kCsCols = 4;                   // rows and columns of a thread

__device__ __forceinline__ void cs_async4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cs_async16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cs_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cs_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

struct ChannelScanArgs {
  const float *q, *k, *v, *g, *u;
  long long ldq, ldk, ldv, ldg;
  float* state;                                          // [rows, H, D, Dv]
  float* part;                                           // [tiles, H, D, Dv]: local, then incoming states
  float* pdec;                                           // [tiles, H, D]: decay products of the tiles
  const int *runs, *pos, *slot;                          // runs NULL: a decode batch
  const int *tiles, *tile_of;
  float* o;
  int H, G, D, Dv, chunk, vec, vecv;
};

// PASS 0: blockIdx.x is a run; 1, 2: a tile
// Four CTAs per SM for short runs and decode batches (0: the compiler's own choice; the tile passes are faster with it).
template <int PASS, int LPC, bool BONUS>
__global__ void __launch_bounds__(128, PASS == 0 ? 4 : 0)
channel_scan_kernel(const ChannelScanArgs a) {
  extern __shared__ __align__(16) float sm[];
  constexpr int R = kCsR, CPT = kCsCols, RP = R + 4, DP = LPC * RP, cpw = 32 / LPC;
  const int b_ = blockIdx.x, h = blockIdx.y;
  int first, n, p0, s;
  bool from_part = false, keep_state = true;
  if (PASS == 0) {
    if (a.runs) { first = a.runs[4 * b_]; n = a.runs[4 * b_ + 1]; p0 = a.runs[4 * b_ + 2]; s = a.runs[4 * b_ + 3]; }
    else { first = b_; n = 1; p0 = a.pos[b_]; s = a.slot[b_]; }
  } else {
    const int place = a.tile_of[4 * b_ + 1], count = a.tile_of[4 * b_ + 2];
    if (PASS == 1 && place + 1 == count) return;         // nobody asks for the last tile's local state
    first = a.tiles[4 * b_]; n = a.tiles[4 * b_ + 1]; p0 = a.tiles[4 * b_ + 2]; s = a.tiles[4 * b_ + 3];
    from_part = PASS == 2;
    keep_state = PASS == 2 && place + 1 == count;
  }
  const int H = a.H, D = a.D, Dv = a.Dv;
  const int kvh = h / (H / a.G);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int l = lane % LPC, jj = lane / LPC;             // the lanes of a column are neighbours: an eighth of a warp reads
  const int ncol = nw * cpw * CPT;                       // different rows of a staged token, without bank conflicts
  const int col0 = blockIdx.z * ncol;
  const int cc0 = (warp * cpw + jj) * CPT;               // first column of this thread inside the CTA's block
  const int j0 = col0 + cc0;
  const int row0 = l * R;
  const int CH = a.chunk;
  constexpr int NS = PASS == 1 ? 2 : 3;                  // staged rows per token: k, g and, where there are outputs, q
  const int per = CH * (NS * DP + ncol);                 // floats per buffer
  auto KS = [&](int b) { return sm + b * per; };
  auto GS = [&](int b) { return sm + b * per + CH * DP; };
  auto QS = [&](int b) { return sm + b * per + 2 * CH * DP; };
  auto VS = [&](int b) { return sm + b * per + NS * CH * DP; };
  auto at = [](int d) { return (d / R) * RP + d % R; };  // key channel d -> its place in a staged row
  if (LPC * R > D) {                                     // rows past D never arrive by copy: zero keys keep their state at zero
    const int padw = LPC * R - D;
    for (int i = threadIdx.x; i < 2 * CH * padw; i += blockDim.x) {
      const int b = i / (CH * padw), r = i % (CH * padw);
      const int x = (r / padw) * DP + at(D + r % padw);
      KS(b)[x] = 0.f;
      GS(b)[x] = 0.f;
      if (PASS != 1) QS(b)[x] = 0.f;
    }
  }
  float2 S2[CPT][R / 2];
  float* sp = a.state + ((long long)s * H + h) * D * (long long)Dv;
  float* pp = PASS == 0 ? nullptr : a.part + ((long long)b_ * H + h) * D * (long long)Dv;
  const float* src = from_part ? pp : (PASS == 0 && p0 > 0 ? sp : nullptr);
  const bool v4 = a.vecv && j0 + CPT <= Dv;              // four whole columns on a 16-byte boundary
#pragma unroll
  for (int i = 0; i < R / 2; ++i) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int d = row0 + 2 * i + e;
      float x[CPT];
#pragma unroll
      for (int c = 0; c < CPT; ++c) x[c] = 0.f;
      if (src && d < D) {
        const float* r = src + (long long)d * Dv + j0;
        if (v4) *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(r);
        else {
#pragma unroll
          for (int c = 0; c < CPT; ++c) if (j0 + c < Dv) x[c] = r[c];
        }
      }
#pragma unroll
      for (int c = 0; c < CPT; ++c) { if (e == 0) S2[c][i].x = x[c]; else S2[c][i].y = x[c]; }
    }
  }
  // the first warp of the first column block also multiplies up the decays of its tile
  const bool owns_dec = PASS == 1 && blockIdx.z == 0 && warp == 0;
  float2 P2[R / 2];
#pragma unroll
  for (int i = 0; i < R / 2; ++i) P2[i] = make_float2(1.f, 1.f);

  // the bonus of a thread's rows stays in registers over a tile; a short run reads it per token instead (occupancy)
  float2 u2[R / 2];
  auto load_u = [&]() {
#pragma unroll
    for (int i = 0; i < R / 2; ++i) {
      u2[i].x = row0 + 2 * i < D ? __ldg(a.u + h * D + row0 + 2 * i) : 0.f;
      u2[i].y = row0 + 2 * i + 1 < D ? __ldg(a.u + h * D + row0 + 2 * i + 1) : 0.f;
    }
  };
  if (BONUS && PASS == 2) load_u();

  auto stage = [&](int b, int c0) {
    const int cn = min(CH, n - c0);
    for (int tt = warp; tt < cn; tt += nw) {
      const long long tr = first + c0 + tt;
      const float* kr = a.k + tr * a.ldk + (long long)kvh * D;
      const float* qr = a.q + tr * a.ldq + (long long)kvh * D;
      const float* gr = a.g + tr * a.ldg + (long long)h * D;
      if (a.vec) {
        for (int d = lane * 4; d < D; d += 128) {
          cs_async16(KS(b) + tt * DP + at(d), kr + d);
          cs_async16(GS(b) + tt * DP + at(d), gr + d);
          if (PASS != 1) cs_async16(QS(b) + tt * DP + at(d), qr + d);
        }
      } else {
        for (int d = lane; d < D; d += 32) {
          cs_async4(KS(b) + tt * DP + at(d), kr + d);
          cs_async4(GS(b) + tt * DP + at(d), gr + d);
          if (PASS != 1) cs_async4(QS(b) + tt * DP + at(d), qr + d);
        }
      }
      const float* vr = a.v + tr * a.ldv + (long long)h * Dv + col0;
      for (int c = lane * 4; c < ncol; c += 128) {
        float* dst = VS(b) + tt * ncol + c;
        if (a.vecv && col0 + c + 4 <= Dv) cs_async16(dst, vr + c);
        else {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            if (col0 + c + e < Dv) cs_async4(dst + e, vr + c + e);
            else dst[e] = 0.f;
          }
        }
      }
    }
  };

  stage(0, 0);
  cs_commit();
  int buf = 0;
  for (int c0 = 0; c0 < n; c0 += CH, buf ^= 1) {
    const int cn = min(CH, n - c0);
    if (c0 + CH < n) stage(buf ^ 1, c0 + CH);
    cs_commit();
    cs_wait<1>();
    __syncthreads();
    const float* ks = KS(buf) + l * RP;
    const float* gs = GS(buf) + l * RP;
    const float* qs = PASS == 1 ? ks : QS(buf) + l * RP;
    const float* vs = VS(buf) + cc0;
    // Pass 2 by two tokens: one's sum over the lanes is a chain of shuffles beside which the other's products run (2345 tokens in three runs,
    // 16 heads of 128 by 128: 281 -> 271 us for two layers; heads of 64: 46 -> 42). Passes 0 and 1 do not gain.
#pragma unroll (PASS == 2 ? 2 : 1)
    for (int tt = 0; tt < cn; ++tt) {
      float2 k2[R / 2], g2[R / 2], q2[R / 2];
#pragma unroll
      for (int i = 0; i < R / 2; i += 2) {
        const float4 kk = *reinterpret_cast<const float4*>(ks + tt * DP + 2 * i);
        const float4 gg = *reinterpret_cast<const float4*>(gs + tt * DP + 2 * i);
        k2[i] = make_float2(kk.x, kk.y); k2[i + 1] = make_float2(kk.z, kk.w);
        g2[i] = make_float2(gg.x, gg.y); g2[i + 1] = make_float2(gg.z, gg.w);
        if (PASS != 1) {
          const float4 qq = *reinterpret_cast<const float4*>(qs + tt * DP + 2 * i);
          q2[i] = make_float2(qq.x, qq.y); q2[i + 1] = make_float2(qq.z, qq.w);
        }
      }
      const float4 vv = *reinterpret_cast<const float4*>(vs + tt * ncol);
      const float vc[CPT] = {vv.x, vv.y, vv.z, vv.w};
      float o[CPT];
      float bonus = 0.f;                                 // this lane's part of q . diag(u) k, the weight of the token's own value
      if (BONUS && PASS != 1) {
        if (PASS == 0) load_u();
        float2 ba = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < R / 2; ++i) ba = __ffma2_rn(__fmul2_rn(u2[i], k2[i]), q2[i], ba);
        bonus = ba.x + ba.y;
      }
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        const float2 v2 = make_float2(vc[c], vc[c]);
        float2 oa = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < R / 2; ++i) {
          if (BONUS && PASS != 1) oa = __ffma2_rn(S2[c][i], q2[i], oa);
          S2[c][i] = __ffma2_rn(g2[i], S2[c][i], __fmul2_rn(k2[i], v2));
          if (!BONUS && PASS != 1) oa = __ffma2_rn(S2[c][i], q2[i], oa);
        }
        o[c] = oa.x + oa.y;
        if (BONUS && PASS != 1) o[c] = fmaf(bonus, vc[c], o[c]);
      }
      if (PASS == 1) {
        if (owns_dec) {
#pragma unroll
          for (int i = 0; i < R / 2; ++i) P2[i] = __fmul2_rn(P2[i], g2[i]);
        }
        continue;
      }
      // sum over the LPC lanes of the columns: the first step sends two columns away and keeps two, the second one and one
      float* orow = a.o + ((long long)(first + c0 + tt) * H + h) * Dv;
      if (LPC == 1) {
        if (v4) *reinterpret_cast<float4*>(orow + j0) = make_float4(o[0], o[1], o[2], o[3]);
        else {
#pragma unroll
          for (int c = 0; c < CPT; ++c) if (j0 + c < Dv) orow[j0 + c] = o[c];
        }
      } else {
        const int b0 = l & 1;
        const float s0 = b0 ? o[0] : o[2], s1 = b0 ? o[1] : o[3];
        float r0 = (b0 ? o[2] : o[0]) + __shfl_xor_sync(0xffffffffu, s0, 1);
        float r1 = (b0 ? o[3] : o[1]) + __shfl_xor_sync(0xffffffffu, s1, 1);
        if (LPC == 2) {
          const int j = j0 + 2 * b0;
          if (j < Dv) orow[j] = r0;
          if (j + 1 < Dv) orow[j + 1] = r1;
        } else {
          const int b1 = (l >> 1) & 1;
          float r = (b1 ? r1 : r0) + __shfl_xor_sync(0xffffffffu, b1 ? r0 : r1, 2);
#pragma unroll
          for (int x = 4; x < LPC; x <<= 1) r += __shfl_xor_sync(0xffffffffu, r, x);
          const int j = j0 + 2 * b0 + b1;
          if (l < 4 && j < Dv) orow[j] = r;
        }
      }
    }
    __syncthreads();
  }
  float* dst = PASS == 1 ? pp : (keep_state ? sp : nullptr);
  if (dst) {
#pragma unroll
    for (int i = 0; i < R / 2; ++i) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int d = row0 + 2 * i + e;
        if (d >= D) continue;
        float* r = dst + (long long)d * Dv + j0;
        float x[CPT];
#pragma unroll
        for (int c = 0; c < CPT; ++c) x[c] = e == 0 ? S2[c][i].x : S2[c][i].y;
        if (v4) *reinterpret_cast<float4*>(r) = *reinterpret_cast<const float4*>(x);
        else {
#pragma unroll
          for (int c = 0; c < CPT; ++c) if (j0 + c < Dv) r[c] = x[c];
        }
      }
    }
  }
  if (owns_dec && jj == 0) {
    float* pd = a.pdec + ((long long)b_ * H + h) * D;
#pragma unroll
    for (int i = 0; i < R / 2; ++i) {
      if (row0 + 2 * i < D) pd[row0 + 2 * i] = P2[i].x;
      if (row0 + 2 * i + 1 < D) pd[row0 + 2 * i + 1] = P2[i].y;
    }
  }
}

// ---- tiles of a prompt by products of matrices: D = Dv, 64 or 128, 16-byte rows -------------------------------------------------
// 16 tokens at a time. With A_i the decays' product over a block's tokens up to i (bonus: up to the one before), B_j that over those after j
// and E that over all 16, per key channel,
//   o_i = (A_i q_i)^T S + sum_(j <= i) W_ij v_j ,  W_ij = sum_d q_id k_jd prod_(j < s <= i) g_sd (bonus: s < i, and u_d for j = i) ,
//   S <- diag(E) S + sum_j (B_j k_j) v_j^T ,
// where every decay is a product of those a walk multiplies too: nothing is divided, and products that underflow do so in a walk as well.
// W is formed by the threads that have the block's q, k and g in registers (two channels each), 120 products running down its columns and nine
// sums over a warp; the rest are products on mma.sync in split bf16 (split_mma.cuh), transposed: 16 columns of S are a warp's 16 rows,
// the state's rows its accumulators, which are an operand of the next product as they lie. The other operand, A q and B k, is split once
// for all columns and read in the order of its lanes.
// A tile with an infinity or NaN, or a product that grows to one, is walked (walk_tile): a product with W's zeros would carry it to tokens before its
// own.
// Bound: the issue slots, which mma.sync and the splits share (split_mma.cuh): of pass 2's 26 000 cycles a tile and head 11 500 are mma.sync, 2800 splits of S,
// 3500 W; pass 1 reads and writes 1.2 TB/s beside it. Two CTAs per SM by registers. Passes 1 / 2, token by token before: 2345 tokens in
// three runs, 16 heads of 128 with a bonus 75 + 146 -> 54 + 104 us (all of the mixer 257 -> 204); 790 tokens, 32 heads of 64: 99 -> 68. Error
// against 64 bits, 500 tokens, decays in 0.9 .. 1 / 0.99 .. 1: state 8.2e-8 / 1.9e-7 (walk 8.6e-8 / 2.3e-7), outputs 1.2e-7 / 1.8e-7 (1.2e-7 / 2.2e-7).
template <int D> struct TileSmem {                        // offsets in 32-bit words
  static constexpr int kWarps = D / 16, KS = D / 16, NT = D / 8, QS = 200, KT = 202, WR = 18;
  static constexpr int E = 0, K = 4 * D, Q = K + 4 * NT * KT, W = Q + 8 * KS * QS, kBoth = W + (D / 64) * 64 * WR, kFirst = K + 4 * NT * KT;
  static constexpr int kWalk = D * D + 2 * D;
  static constexpr int bytes(int pass) { return (pass == 1 ? (kFirst > kWalk ? kFirst : kWalk) : (kBoth > kWalk ? kBoth : kWalk)) * 4; }
};

// 16 values a lane, summed over the warp: lane l keeps the sum of value l / 2
__device__ __forceinline__ float gather16(float (&v)[16], int lane) {
#pragma unroll
  for (int w = 8; w >= 1; w >>= 1) {
    const bool up = lane & (2 * w);
#pragma unroll
    for (int i = 0; i < w; ++i) {
      const float mine = up ? v[w + i] : v[i], theirs = up ? v[i] : v[w + i];
      v[i] = mine + __shfl_xor_sync(0xffffffffu, theirs, 2 * w);
    }
  }
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// Tokens [c0, n) of a tile one by one, from the S [D][D] in shared memory; a state that is kept goes to `dst`. A thread has half of a column in registers; k, q and g
// of 16 tokens come through shared memory, where their halves of the outputs meet. A NaN in one channel of the first of 2345 tokens, 16 heads of 128:
// the mixer 232 -> 336 us, in all channels 480 (with S in shared memory and k, q, g read where they lie, 754 and 1133).
template <int PASS, int D, bool BONUS>
__device__ __noinline__ void walk_tile(const ChannelScanArgs& a, float* sm, int h, int first, int c0, int n, bool keep, float* dst) {
  constexpr int TB = 16, R = D / 2, NT = 2 * D;
  static_assert((5 * TB + 1) * D * 4 <= TileSmem<D>::bytes(1), "the staged tokens fit");
  float *Ks = sm, *Gs = Ks + TB * D, *Qs = Gs + TB * D, *red = Qs + TB * D, *us = red + 2 * TB * D;
  const int tid = threadIdx.x, e = tid % D, half = tid / D, kvh = h / (a.H / a.G);
  float s[R];
#pragma unroll
  for (int i = 0; i < R; ++i) s[i] = sm[(half * R + i) * D + e];
  __syncthreads();
  if (PASS != 1 && BONUS && half == 0) us[e] = a.u[h * D + e];
  for (int t0 = c0; t0 < n; t0 += TB) {
    const int m = min(TB, n - t0);
    const long long row = first + t0;
    for (int i = tid; i < m * D; i += NT) {
      const int t = i / D, d = i % D;
      Ks[i] = a.k[(row + t) * a.ldk + (long long)kvh * D + d];
      Gs[i] = a.g[(row + t) * a.ldg + (long long)h * D + d];
      if (PASS != 1) Qs[i] = a.q[(row + t) * a.ldq + (long long)kvh * D + d];
    }
    __syncthreads();
    for (int t = 0; t < m; ++t) {
      const float v = a.v[(row + t) * a.ldv + (long long)h * D + e];
      float o = 0.f;
#pragma unroll
      for (int i = 0; i < R; i += 4) {
        const int d = half * R + i;
        const float4 k4 = *reinterpret_cast<const float4*>(Ks + t * D + d), g4 = *reinterpret_cast<const float4*>(Gs + t * D + d);
        float4 q4 = {}, u4 = {};
        if (PASS != 1) q4 = *reinterpret_cast<const float4*>(Qs + t * D + d);
        if (PASS != 1 && BONUS) u4 = *reinterpret_cast<const float4*>(us + d);
        const float k[4] = {k4.x, k4.y, k4.z, k4.w}, g[4] = {g4.x, g4.y, g4.z, g4.w}, q[4] = {q4.x, q4.y, q4.z, q4.w}, u[4] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const float kv = k[x] * v;
          if (PASS != 1 && BONUS) o = fmaf(fmaf(u[x], kv, s[i + x]), q[x], o);
          s[i + x] = fmaf(g[x], s[i + x], kv);
          if (PASS != 1 && !BONUS) o = fmaf(s[i + x], q[x], o);
        }
      }
      if (PASS != 1) red[(t * 2 + half) * D + e] = o;
    }
    __syncthreads();
    if (PASS != 1)
      for (int i = tid; i < m * D; i += NT) {
        const int t = i / D, c = i % D;
        a.o[((row + t) * a.H + h) * D + c] = red[2 * t * D + c] + red[(2 * t + 1) * D + c];
      }
  }
  if (keep)
#pragma unroll
    for (int i = 0; i < R; ++i) dst[(half * R + i) * D + e] = s[i];
}

template <int PASS, int D, bool BONUS>
__global__ void __launch_bounds__(TileSmem<D>::kWarps * 32, D == 64 ? 3 : 2)
channel_tile_kernel(const ChannelScanArgs a) {
  using L = TileSmem<D>;
  constexpr int KS = L::KS, NT = L::NT;
  extern __shared__ __align__(16) float sm[];
  uint32_t* smw = reinterpret_cast<uint32_t*>(sm);
  const int b_ = blockIdx.x, h = blockIdx.y, kvh = h / (a.H / a.G);
  const int place = a.tile_of[4 * b_ + 1], count = a.tile_of[4 * b_ + 2];
  if (PASS == 1 && place + 1 == count) return;           // nobody asks for the last tile's local state
  const int first = a.tiles[4 * b_], n = a.tiles[4 * b_ + 1], slot = a.tiles[4 * b_ + 3];
  const bool keep = PASS == 1 || place + 1 == count;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t2 = (lane & 3) * 2;
  float* part = a.part + ((long long)b_ * a.H + h) * D * D;
  float* dst = PASS == 1 ? part : a.state + ((long long)slot * a.H + h) * D * D;

  float S[NT][4];                                         // S^T: columns 16 warp + g and + 8 of the state's rows 8 j + t2, + 1
  auto each = [&](auto f) {
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int x = 0; x < 4; ++x) f(S[j][x], (8 * j + t2 + (x & 1)) * D + warp * 16 + g + (x >> 1) * 8);
  };
  float dec = 1.f;                                        // pass 1: the tile's decay product of channel tid
  for (int c0 = 0; c0 < n; c0 += 64) {
    const int cn = min(64, n - c0);
    int odd = 0;
    // ---- this thread's two channels of one block of 16 tokens ----
    {
      const int blk = tid / (D / 2), c = tid % (D / 2);
      float2 gg[16], kk[16], qq[PASS == 1 ? 1 : 16];
      const long long row0 = first + c0 + blk * 16;
      const float* gp = a.g + row0 * a.ldg + (long long)h * D + 2 * c;
      const float* kp = a.k + row0 * a.ldk + (long long)kvh * D + 2 * c;
      const float* qp = a.q + row0 * a.ldq + (long long)kvh * D + 2 * c;
#pragma unroll
      for (int x = 0; x < 16; ++x) {
        const bool live = blk * 16 + x < cn;
        gg[x] = live ? *reinterpret_cast<const float2*>(gp + x * a.ldg) : make_float2(1.f, 1.f);
        kk[x] = live ? *reinterpret_cast<const float2*>(kp + x * a.ldk) : make_float2(0.f, 0.f);
        if (PASS != 1) qq[PASS == 1 ? 0 : x] = live ? *reinterpret_cast<const float2*>(qp + x * a.ldq) : make_float2(0.f, 0.f);
      }
      if constexpr (PASS != 1) {
        float* Ws = sm + L::W + ((c >> 5) * 4 + blk) * 16 * L::WR;       // each warp of a block its sums
        float v[16];
        const float2 u = BONUS ? *reinterpret_cast<const float2*>(a.u + h * D + 2 * c) : make_float2(1.f, 1.f);
#pragma unroll
        for (int x = 0; x < 16; ++x) v[x] = fmaf(qq[x].x * u.x, kk[x].x, qq[x].y * u.y * kk[x].y);
        float w = gather16(v, lane);
        const int s = lane >> 1;
        odd |= not_finite(w);
        if (!(lane & 1)) Ws[s * L::WR + s] = w;
        // columns j and 15 - j of W together: 15 - j and j elements below the diagonal
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          v[j] = 0.f;
          float2 p = kk[j];
#pragma unroll
          for (int i = j + 1; i < 16; ++i) {
            if (!BONUS) p = __fmul2_rn(p, gg[i]);
            v[i] = fmaf(qq[i].x, p.x, qq[i].y * p.y);
            if (BONUS) p = __fmul2_rn(p, gg[i]);
          }
          p = kk[15 - j];
#pragma unroll
          for (int i = 16 - j; i < 16; ++i) {
            if (!BONUS) p = __fmul2_rn(p, gg[i]);
            v[i - 16 + j] = fmaf(qq[i].x, p.x, qq[i].y * p.y);
            if (BONUS) p = __fmul2_rn(p, gg[i]);
          }
          w = gather16(v, lane);
          odd |= not_finite(w);
          if (!(lane & 1) && s != j) Ws[s > j ? s * L::WR + j : (16 - j + s) * L::WR + 15 - j] = w;
        }
        // A q: pairs of channels of a token
        uint32_t* Qs = smw + L::Q + (blk * 2 * KS + (c >> 3)) * L::QS + (c & 3) * 2 + ((c >> 2) & 1);
        float2 p = make_float2(1.f, 1.f);
#pragma unroll
        for (int x = 0; x < 16; ++x) {
          if (!BONUS) p = __fmul2_rn(p, gg[x]);
          const float2 y = __fmul2_rn(qq[x], p);
          if (BONUS) p = __fmul2_rn(p, gg[x]);
          odd |= not_finite(y.x) | not_finite(y.y);
          uint32_t* at = Qs + (x >> 3) * KS * L::QS + (x & 7) * 8;
          split3(y.x, y.y, at[0], at[64], at[128]);
        }
      }
      // B k: pairs of tokens of a channel
      uint32_t* Kb = smw + L::K + (blk * NT + (c >> 2)) * L::KT + (c & 3) * 16;
      float2 p = make_float2(1.f, 1.f);
#pragma unroll
      for (int x = 14; x >= 0; x -= 2) {
        const float2 y1 = __fmul2_rn(kk[x + 1], p);
        p = __fmul2_rn(p, gg[x + 1]);
        const float2 y0 = __fmul2_rn(kk[x], p);
        p = __fmul2_rn(p, gg[x]);
        odd |= not_finite(y0.x) | not_finite(y0.y) | not_finite(y1.x) | not_finite(y1.y);
        uint32_t* at = Kb + ((x >> 1) & 3) * 2 + (x >> 3);
        split3(y0.x, y1.x, at[0], at[64], at[128]);
        split3(y0.y, y1.y, at[8], at[72], at[136]);
      }
      odd |= not_finite(p.x) | not_finite(p.y);
      *reinterpret_cast<float2*>(sm + L::E + blk * D + 2 * c) = p;
    }
    // the values: 16 columns of this warp
    const float* vp = a.v + (long long)(first + c0) * a.ldv + (long long)h * D + warp * 16 + g;
    auto value = [&](int t, int hi) { return t < cn ? vp[(long long)t * a.ldv + hi * 8] : 0.f; };
    each([&](float& s, int at) { s = PASS == 1 && c0 == 0 ? 0.f : part[at]; });
    __syncthreads();
    const float before = dec;
    if (PASS == 1 && tid < D) dec *= (sm[L::E + tid] * sm[L::E + D + tid]) * (sm[L::E + 2 * D + tid] * sm[L::E + 3 * D + tid]);
    const int nb = (cn + 15) / 16;
#pragma unroll 1
    for (int blk = 0; blk < nb; ++blk) {
      SplitA va;
      {
        const int t = blk * 16 + t2;
        split3(value(t, 0), value(t + 1, 0), va.p[0][0], va.p[1][0], va.p[2][0]);
        split3(value(t, 1), value(t + 1, 1), va.p[0][1], va.p[1][1], va.p[2][1]);
        split3(value(t + 8, 0), value(t + 9, 0), va.p[0][2], va.p[1][2], va.p[2][2]);
        split3(value(t + 8, 1), value(t + 9, 1), va.p[0][3], va.p[1][3], va.p[2][3]);
      }
      auto load_b = [&](const uint32_t* at) {
        SplitB b;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const uint2 v = *reinterpret_cast<const uint2*>(at + i * 64 + lane * 2);
          b.p[i][0] = v.x; b.p[i][1] = v.y;
        }
        return b;
      };
      if (PASS != 1) {
        SplitAcc oa[2];
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          float w[4];
          const int i = 8 * m + g;
#pragma unroll
          for (int x = 0; x < 4; ++x) {                   // W_ij of token i, j = t2, t2 + 1, t2 + 8, t2 + 9
            const int j = t2 + (x & 1) + (x >> 1) * 8;
            const float* at = sm + L::W + (blk * 16 + i) * L::WR + j;
            w[x] = j > i ? 0.f : (D == 128 ? at[0] + at[64 * L::WR] : at[0]);
          }
          mma_split<true>(va, split_b(w[0], w[1], w[2], w[3]), oa[m]);
        }
#pragma unroll
        for (int s = 0; s < KS; ++s) {
          SplitA sa;
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            split3(S[2 * s + j][0], S[2 * s + j][1], sa.p[0][2 * j], sa.p[1][2 * j], sa.p[2][2 * j]);
            split3(S[2 * s + j][2], S[2 * s + j][3], sa.p[0][2 * j + 1], sa.p[1][2 * j + 1], sa.p[2][2 * j + 1]);
          }
#pragma unroll
          for (int m = 0; m < 2; ++m) mma_split(sa, load_b(smw + L::Q + ((blk * 2 + m) * KS + s) * L::QS), oa[m]);
        }
        float* orow = a.o + ((long long)(first + c0 + blk * 16) * a.H + h) * D + warp * 16 + g;
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            const int t = 8 * m + t2 + (x & 1);
            const float o = oa[m].sum(x);
            odd |= not_finite(o);
            if (blk * 16 + t < cn) orow[(long long)t * a.H * D + (x >> 1) * 8] = o;
          }
      }
      if (!keep && c0 + (blk + 1) * 16 >= n) break;       // nobody asks for this state
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        SplitAcc sa;
        mma_split<true>(va, load_b(smw + L::K + (blk * NT + j) * L::KT), sa);
        const float2 e = *reinterpret_cast<const float2*>(sm + L::E + blk * D + 8 * j + t2);
#pragma unroll
        for (int x = 0; x < 4; ++x) S[j][x] = fmaf(x & 1 ? e.y : e.x, S[j][x], sa.sum(x));
      }
    }
    if (keep || c0 + 64 < n) each([&](float& s, int) { odd |= not_finite(s); });      // a state that is used
    if (__syncthreads_or(odd)) {                          // from the state in front of these tokens, which still lies there, again
      each([&](float&, int at) { sm[at] = PASS == 1 && c0 == 0 ? 0.f : part[at]; });
      if (PASS == 1 && tid < D) {
        dec = before;
        for (int t = c0; t < n; ++t) dec *= a.g[(long long)(first + t) * a.ldg + (long long)h * D + tid];
        a.pdec[((long long)b_ * a.H + h) * D + tid] = dec;
      }
      __syncthreads();
      walk_tile<PASS, D, BONUS>(a, sm, h, first, c0, n, keep, dst);
      return;
    }
    if (c0 + 64 < n) each([&](float& s, int at) { part[at] = s; });       // a longer tile: its state waits where it came from
  }
  if (keep) each([&](float& s, int at) { dst[at] = s; });
  if (PASS == 1 && tid < D) a.pdec[((long long)b_ * a.H + h) * D + tid] = dec;
}

template <int PASS, int D, bool BONUS>
static int launch_tiles(const ChannelScanArgs& a, int n_tiles, cudaStream_t st) {
  auto kern = channel_tile_kernel<PASS, D, BONUS>;
  constexpr int smem = TileSmem<D>::bytes(PASS);
  B200_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  kern<<<dim3(n_tiles, a.H), TileSmem<D>::kWarps * 32, smem, st>>>(a);
  return 0;
}

// Chains the tiles of every run: part[tile] (local state) becomes the tile's incoming state. A thread owns V neighbouring
// elements of one head's state; the loads do not depend on the chain, so four tiles are in flight.
template <int V>
__global__ void __launch_bounds__(128)
channel_scan_carry_kernel(float* __restrict__ part, const float* __restrict__ pdec, const float* __restrict__ state,
                          const int* __restrict__ runs, const int* __restrict__ run_tiles, int H, int D, int Dv) {
  const int h = blockIdx.y;
  const long long e0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * V;
  if (e0 >= (long long)D * Dv) return;
  const int d = (int)(e0 / Dv);                          // V divides Dv: the V elements share a row
  const int t0 = run_tiles[4 * blockIdx.z], count = run_tiles[4 * blockIdx.z + 1];
  const int p0 = runs[4 * blockIdx.z + 2], s = runs[4 * blockIdx.z + 3];
  float S[V];
#pragma unroll
  for (int v = 0; v < V; ++v) S[v] = p0 > 0 ? state[((long long)s * H + h) * D * (long long)Dv + e0 + v] : 0.f;
  const long long ts = (long long)H * D * Dv;
  float* p = part + (long long)t0 * ts + (long long)h * D * Dv + e0;
  const float* g = pdec + ((long long)t0 * H + h) * D + d;
  for (int j0 = 0; j0 < count; j0 += 4) {
    float loc[4][V], dec[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      dec[u] = 0.f;
#pragma unroll
      for (int v = 0; v < V; ++v) loc[u][v] = 0.f;
      if (j0 + u + 1 < count) {                          // the last tile of a run has no local state
        if (V == 4) *reinterpret_cast<float4*>(loc[u]) = *reinterpret_cast<const float4*>(p + (j0 + u) * ts);
        else loc[u][0] = p[(j0 + u) * ts];
        dec[u] = g[(long long)(j0 + u) * H * D];
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (j0 + u < count) {
        if (V == 4) *reinterpret_cast<float4*>(p + (j0 + u) * ts) = *reinterpret_cast<const float4*>(S);
        else p[(j0 + u) * ts] = S[0];
#pragma unroll
        for (int v = 0; v < V; ++v) S[v] = fmaf(dec[u], S[v], loc[u][v]);
      }
    }
  }
}

// CPT channels per thread, kLrTok tokens at a time, `groups` times: x rows of all of them are staged once and broadcast.
// FAST (16-bit models): base-2 hardware exponential and logarithm; their absolute error in log sigmoid, 2e-7, is divided by tau.
// Otherwise a decay near 1 is formed as 1 + expm1(.): it is raised to the power of its whole reach, and expf's small bias would
// add up where the rounding of 1 + expm1 does not.
constexpr int kLrTok = 8;
// CPT channels per thread share the reads of x. RK: the rank at compile time, weights then stay in registers (0: any rank)
// EXPO: the inputs pass tanh as they are staged, and the decay is exp(-exp(z)).
template <bool FAST, int CPT, int RK, bool EXPO>
__global__ void __launch_bounds__(128)
lowrank_decay_kernel(const float* __restrict__ x, long long ldx, const float* __restrict__ w2, const float* __restrict__ bias,
                     float* __restrict__ out, int tokens, int C, int rank, float inv_tau, int groups) {
  extern __shared__ __align__(16) float xall[];          // [groups * kLrTok][rank]
  const int tb = blockIdx.y * kLrTok * groups;
  for (int i = threadIdx.x; i < groups * kLrTok * rank; i += blockDim.x) {
    const int t = i / rank;
    const float xv = tb + t < tokens ? x[(long long)(tb + t) * ldx + i % rank] : 0.f;
    xall[i] = EXPO ? tanhf(xv) : xv;
  }
  __syncthreads();
  const int c0 = blockIdx.x * 128 * CPT + threadIdx.x;   // this thread's channels are 128 apart
  const float* w[CPT];
#pragma unroll
  for (int j = 0; j < CPT; ++j) w[j] = w2 + (long long)min(c0 + 128 * j, C - 1) * rank;
  const bool vec = rank % 4 == 0 && (reinterpret_cast<uintptr_t>(w2) & 15) == 0;
  constexpr int RV = RK / 4 > 0 ? RK / 4 : 1;
  float4 wr[CPT][RV];
  if (RK > 0) {
#pragma unroll
    for (int j = 0; j < CPT; ++j)
#pragma unroll
      for (int i = 0; i < RV; ++i) wr[j][i] = *reinterpret_cast<const float4*>(w[j] + 4 * i);
  }
  for (int gi = 0; gi < groups; ++gi) {
    const int t0 = tb + gi * kLrTok, nt = min(kLrTok, tokens - t0);
    if (nt <= 0) break;
    const float* xs = xall + gi * kLrTok * rank;
    float acc[kLrTok][CPT];
#pragma unroll
    for (int j = 0; j < CPT; ++j) {
      const float b = bias[min(c0 + 128 * j, C - 1)];
#pragma unroll
      for (int t = 0; t < kLrTok; ++t) acc[t][j] = b;
    }
    int r = RK;
    if (RK > 0) {
#pragma unroll
      for (int i = 0; i < RV; ++i)
#pragma unroll
        for (int t = 0; t < kLrTok; ++t) {
          const float4 xv = *reinterpret_cast<const float4*>(xs + t * rank + 4 * i);
#pragma unroll
          for (int j = 0; j < CPT; ++j) {
            acc[t][j] = fmaf(wr[j][i].x, xv.x, acc[t][j]);
            acc[t][j] = fmaf(wr[j][i].y, xv.y, acc[t][j]);
            acc[t][j] = fmaf(wr[j][i].z, xv.z, acc[t][j]);
            acc[t][j] = fmaf(wr[j][i].w, xv.w, acc[t][j]);
          }
        }
    } else if (vec) {
      for (; r < rank; r += 4) {
        float4 wv[CPT];
#pragma unroll
        for (int j = 0; j < CPT; ++j) wv[j] = *reinterpret_cast<const float4*>(w[j] + r);
#pragma unroll
        for (int t = 0; t < kLrTok; ++t) {
          const float4 xv = *reinterpret_cast<const float4*>(xs + t * rank + r);
#pragma unroll
          for (int j = 0; j < CPT; ++j) {
            acc[t][j] = fmaf(wv[j].x, xv.x, acc[t][j]);
            acc[t][j] = fmaf(wv[j].y, xv.y, acc[t][j]);
            acc[t][j] = fmaf(wv[j].z, xv.z, acc[t][j]);
            acc[t][j] = fmaf(wv[j].w, xv.w, acc[t][j]);
          }
        }
      }
    }
    for (; r < rank; ++r) {
#pragma unroll
      for (int t = 0; t < kLrTok; ++t)
#pragma unroll
        for (int j = 0; j < CPT; ++j) acc[t][j] = fmaf(w[j][r], xs[t * rank + r], acc[t][j]);
    }
#pragma unroll
    for (int t = 0; t < kLrTok; ++t) {
      if (t >= nt) break;
#pragma unroll
      for (int j = 0; j < CPT; ++j) {
        const float z = acc[t][j];
        float v;
        if (EXPO) {
          const float y = -expf(z);
          v = FAST ? ex2_approx(y * 1.4426950408889634f) : (y > -0.5f ? 1.f + expm1f(y) : expf(y));
        } else if (FAST) {
          const float z2 = z * 1.4426950408889634f;
          v = ex2_approx((fminf(z2, 0.f) - __log2f(1.f + ex2_approx(-fabsf(z2)))) * inv_tau);
        } else {
          const float y = (fminf(z, 0.f) - log1pf(expf(-fabsf(z)))) * inv_tau;        // log sigmoid(z) / tau
          v = y > -0.5f ? 1.f + expm1f(y) : expf(y);
        }
        if (c0 + 128 * j < C) out[(long long)(t0 + t) * C + c0 + 128 * j] = v;
      }
    }
  }
}
}  // namespace b200

// form 0: sigmoid(w2 x + bias)^inv_tau; 1: exp(-exp(w2 tanh(x) + bias))
B200_API int b200_lowrank_decay_ex(const float* x, long long ldx, const float* w2, const float* bias, float* out, int tokens, int C,
                                   int rank, float inv_tau, int form, int fast, void* stream) {
  using namespace b200;
  if (tokens <= 0) return 0;
  if (C <= 0 || rank <= 0 || tokens > 65535 * kLrTok) return B200_ERR_BAD_SHAPE;
  int groups = tokens >= 2048 ? 4 : 1;
  while (groups > 1 && (size_t)groups * kLrTok * rank * 4 > 48 * 1024) groups /= 2;
  const size_t smem = (size_t)groups * kLrTok * rank * 4;
  if (smem > 48 * 1024) return B200_ERR_TOO_LARGE;
  const bool r16 = rank == 16 && !(reinterpret_cast<uintptr_t>(w2) & 15);
  const int cpt = tokens >= 512 ? (r16 ? 2 : 4) : 1;
  dim3 grid((C + 128 * cpt - 1) / (128 * cpt), (tokens + kLrTok * groups - 1) / (kLrTok * groups));
#define LR(FF, CC, RR)                                                                                                         \
  do {                                                                                                                         \
    if (form == 1) lowrank_decay_kernel<FF, CC, RR, true><<<grid, 128, smem, (cudaStream_t)stream>>>(x, ldx, w2, bias, out, tokens, C, rank, inv_tau, groups); \
    else lowrank_decay_kernel<FF, CC, RR, false><<<grid, 128, smem, (cudaStream_t)stream>>>(x, ldx, w2, bias, out, tokens, C, rank, inv_tau, groups); \
  } while (0)
#define LR_F(FF)                                                                                                               \
  do { if (cpt == 2) LR(FF, 2, 16); else if (cpt == 4) LR(FF, 4, 0); else if (r16) LR(FF, 1, 16); else LR(FF, 1, 0); } while (0)
  if (fast) LR_F(true); else LR_F(false);
#undef LR_F
#undef LR
  B200_LAUNCH_CHECK();
  return 0;
}

B200_API int b200_lowrank_decay(const float* x, long long ldx, const float* w2, const float* bias, float* out, int tokens, int C,
                                int rank, float inv_tau, int fast, void* stream) {
  return b200_lowrank_decay_ex(x, ldx, w2, bias, out, tokens, C, rank, inv_tau, 0, fast, stream);
}

B200_API int b200_channel_scan(const float* q, long long ldq, const float* k, long long ldk, const float* v, long long ldv,
                               const float* g, long long ldg, const float* u, float* state, float* part, float* pdec, const int* runs, int n_runs,
                               const int* tiles, int n_tiles, const int* tile_of, const int* run_tiles, int chunk, const int* pos, const int* slot, float* o,
                               int H, int G, int D, int Dv, void* stream) {
  using namespace b200;
  if (n_runs <= 0) return 0;
  if (H <= 0 || G <= 0 || H % G || D <= 0 || Dv <= 0 || H > 65535 || chunk < 1) return B200_ERR_BAD_SHAPE;
  if (n_tiles > 0 && (!part || !pdec || !tiles || !tile_of || !run_tiles || !runs || n_runs > 65535)) return B200_ERR_BAD_SHAPE;
  int LPC = 1;
  while (LPC * kCsR < D) LPC *= 2;
  if (LPC > 32) return B200_ERR_TOO_LARGE;
  const int wcol = 32 / LPC * kCsCols;                   // columns of a warp
  int nw = 4;
  while (nw > 1 && (nw - 1) * wcol >= Dv) --nw;          // no warp without columns
  const int ncol = nw * wcol, zb = (Dv + ncol - 1) / ncol;
  const int DP = LPC * (kCsR + 4);
  int CH = chunk < 16 ? chunk : 16;
  auto bytes = [&](int ch) { return (size_t)2 * ch * (3 * DP + ncol) * 4; };
  while (CH > 1 && bytes(CH) > 100 * 1024) CH /= 2;
  auto al = [](const void* p_, long long ld) { return !(reinterpret_cast<uintptr_t>(p_) & 15) && ld % 4 == 0; };
  ChannelScanArgs a;
  a.q = q; a.k = k; a.v = v; a.g = g; a.u = u; a.ldq = ldq; a.ldk = ldk; a.ldv = ldv; a.ldg = ldg;
  a.state = state; a.part = part; a.pdec = pdec; a.runs = runs; a.pos = pos; a.slot = slot; a.tiles = tiles; a.tile_of = tile_of;
  a.o = o; a.H = H; a.G = G; a.D = D; a.Dv = Dv; a.chunk = CH;
  a.vec = D % 4 == 0 && al(q, ldq) && al(k, ldk) && al(g, ldg);
  a.vecv = Dv % 4 == 0 && al(v, ldv) && al(state, 4) && al(o, 4) && (!part || al(part, 4));
  cudaStream_t st = (cudaStream_t)stream;
  const size_t smem = bytes(CH);
#define CS(PASS, LL, NB) do { if (u) CS_B(PASS, LL, NB, true); else CS_B(PASS, LL, NB, false); } while (0)
#define CS_B(PASS, LL, NB, BB)                                                                                             \
  do {                                                                                                                     \
    auto kern = channel_scan_kernel<PASS, LL, (PASS != 1 && BB)>;                                                                             \
    if (smem > 48 * 1024) B200_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));  \
    kern<<<dim3(NB, H, zb), nw * 32, smem, st>>>(a);                                                                       \
  } while (0)
#define CS_L(PASS, NB)                                                                                                     \
  do {                                                                                                                     \
    if (LPC == 1) CS(PASS, 1, NB); else if (LPC == 2) CS(PASS, 2, NB); else if (LPC == 4) CS(PASS, 4, NB);                  \
    else if (LPC == 8) CS(PASS, 8, NB); else if (LPC == 16) CS(PASS, 16, NB); else CS(PASS, 32, NB);                        \
  } while (0)
  if (n_tiles <= 0) {
    CS_L(0, n_runs);
  } else {
    // runs of several tiles where a head's state is square and rows are whole vectors: by products; else token by token
    const bool mat = (D == 64 || D == 128) && Dv == D && a.vec && a.vecv && (!u || al(u, 4));
    if (mat) { if (int rc = D == 64 ? launch_tiles<1, 64, false>(a, n_tiles, st) : launch_tiles<1, 128, false>(a, n_tiles, st)) return rc; }
    else CS_L(1, n_tiles);
    const int V = Dv % 4 == 0 && al(part, 4) ? 4 : 1;
    const long long n = (long long)D * Dv / V;
    dim3 grid((unsigned)((n + 127) / 128), H, n_runs);
    if (V == 4) channel_scan_carry_kernel<4><<<grid, 128, 0, st>>>(part, pdec, state, runs, run_tiles, H, D, Dv);
    else channel_scan_carry_kernel<1><<<grid, 128, 0, st>>>(part, pdec, state, runs, run_tiles, H, D, Dv);
    if (!mat) CS_L(2, n_tiles);
    else if (int rc = D == 64 ? (u ? launch_tiles<2, 64, true>(a, n_tiles, st) : launch_tiles<2, 64, false>(a, n_tiles, st))
                              : (u ? launch_tiles<2, 128, true>(a, n_tiles, st) : launch_tiles<2, 128, false>(a, n_tiles, st))) return rc;
  }
#undef CS_L
#undef CS_B
#undef CS
  B200_LAUNCH_CHECK();
  return 0;
}
