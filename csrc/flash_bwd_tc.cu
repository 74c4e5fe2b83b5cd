// K4 backward on the 5th-generation tensor cores: dQ, dK, dV of causal flash attention with every product on tcgen05.mma,
// accumulators in TMEM, operands by TMA straight out of the fused qkv / dout matrices, no atomics and no fp32 gradient
// staging buffer.
//
// One kernel body, two modes (launched one after the other):
//   mode KV  CTA = (128-key block, kv head, batch): K, V stay in shared memory; the (query head of the group, 64-row query tile)
//            pairs that see the block stream through a 4-stage TMA ring. TMEM lanes are KEYS:
//              S^T = K Q^T, dP^T = V dO^T   (M 128 x N 64 x K D) -> TMEM, double-buffered, issued one pair AHEAD
//              warps 0-15, thread = (key, quarter of the queries): P = exp2(S c - lse), dS = P (dP - delta) scale -> 16 bit, written
//                                          over S^T and dP^T in TMEM; lse and delta of the pair's 64 queries lie in shared memory
//              dV += P^T dO, dK += dS^T Q   (M 128 x N D x K 64, A from TMEM, B in place), over ALL pairs, GQA group included
//   mode Q   CTA = (128-row query tile, query head, batch): Q, dO stay; the 64-key blocks it sees stream. TMEM lanes are queries:
//              S = Q K^T, dP = dO V^T, dS as above over dP in TMEM, dQ += dS K (M 128 x N D x K 64, A from TMEM)
// What bounds it is shared memory (128 bytes a cycle): a 128 x 64 x 16 product with both operands there takes 48 cycles for 32 of
// tensor time, so P and dS, which are computed in registers anyway, go back to TMEM and only the streamed side of the second
// products is read from shared memory. S and dP are recomputed in mode Q (7 products instead of 5) in exchange for: no
// red.global traffic (the atomics of a one-pass kernel are 64 KB per 128 x 128 pair), no zero-filled fp32 [tokens,
// 3 x heads x D] buffer, bit-reproducible gradients. In mode KV the key block is the slowest grid dimension: block 0, which
// every query sees, starts first for all heads, and the short blocks fill the end.
// Measured (bf16, causal; dK / dV pass, dQ pass, delta), before with 64-key blocks, P and dS through shared memory and eight warps:
// 1 x 4096, 32 / 8 heads of 128: 574, 303, 24 -> 273, 211, 15 us; 4 x 512, 40 / 8 heads: 81, 47, 16 -> 52, 43, 10; eight element-wise
// warps instead of sixteen: 372, 312; 32 x 256, 12 heads of 64 (mma.sync with fp32 atomics before: 144 with its memset,
// cast and delta): 46, 38, 7.
//
// 608 threads: warps 0-15 element-wise (four share a TMEM lane quarter and split the 64 columns: a pair is a chain of TMEM reads, FMAs,
// exponentials and TMEM writes, and it is warps beside one another that hide it), warp 16 TMA producer, warp 17 tcgen05
// issuer, warp 18 the rows' lse and delta of mode KV; 1 CTA per SM (512 TMEM columns). head_dim 64 or
// 128, 16-bit, no dropout — anything else goes to the mma.sync kernel of flash_attn.cu. Reference call sites: the SDPA backward
// behind nn.MultiheadAttention
// (LLM_Distributed_Trainning/PyTorch/ddp_basics/ddp_gpt_wikitext2.py:89-96) and HF Qwen3 attention under the Trainer
// (Fine-Tuning/qwen3-14b-qlora-dist-deepspeed.py:95-107, Fine-Tuning/qwen3-8b-lora-dist.py:118).
#include "common.cuh"
#include "tma_host.h"
#include "../include/b200_ops.h"

namespace b200 {

constexpr int kBwBM = 128, kBwBN = 64;   // rows that stay (TMEM lanes), rows that stream
constexpr int kBwEw = 16;                // element-wise warps
constexpr int kBwThreads = (kBwEw + 3) * 32;
constexpr int kBwStages = 4;
constexpr uint32_t kBwTmemCols = 512;
constexpr uint32_t kBwTS = 0, kBwTdP = 64, kBwTBuf = 128, kBwTAcc = 256;   // S(b) at b*128, dP(b) at 64 + b*128, accumulators from 256

// shared memory: the two resident tiles [128 rows] (halves of 64 columns, 16 KiB each), the stages of two tiles [64 rows], lse | delta
// of the stages' rows, barriers
template <int D> struct BwSmem {
  static constexpr uint32_t kHalves = D / 64, kRes = 16384 * kHalves, kTile = 8192 * kHalves, kStage = 2 * kTile;
  static constexpr uint32_t kRing = 2 * kRes, kStats = kRing + kBwStages * kStage, kBar = kStats + kBwStages * 512, kBytes = kBar + 256;
};

struct FlashBwdTcParams {
  void* dqkv;             // [B*S, W] 16-bit, same layout as qkv
  const float* lse;       // [B, H, S] natural log
  const float* delta;     // [B, H, S] rowsum(dO * O)
  int B, S, H, Hkv;
  long long W;            // row stride of qkv / dqkv in elements
  float scale, scale_log2;
  int causal;
};

// 8 products of 16-bit pairs
template <bool BF16>
__device__ __forceinline__ float bw_dot8(const uint4& a, const uint4& b) {
  const uint32_t x[4] = {a.x, a.y, a.z, a.w}, y[4] = {b.x, b.y, b.z, b.w};
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 u, v;
    if (BF16) { u = unpack_bf16x2(x[i]); v = unpack_bf16x2(y[i]); }
    else { u = __half22float2(*reinterpret_cast<const __half2*>(&x[i])); v = __half22float2(*reinterpret_cast<const __half2*>(&y[i])); }
    s = fmaf(u.x, v.x, s); s = fmaf(u.y, v.y, s);
  }
  return s;
}

// delta[b, h, s] = sum_d dO[b*S + s, h*D + d] * O[...]: D / 8 lanes per (row, head), 16 bytes each, two items per lane on their way
template <bool BF16, int D>
__global__ void __launch_bounds__(256)
flash_delta_tc_kernel(const uint16_t* __restrict__ o, const uint16_t* __restrict__ dout, float* __restrict__ delta, long long items, int S, int H) {
  constexpr int L = D / 8, PER = 256 / L;                  // lanes of an item, items of a block's pass
  const int sub = threadIdx.x % L;
  const long long i0 = (long long)blockIdx.x * (2 * PER) + threadIdx.x / L;
  uint4 a[2], b[2];
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    const long long i = i0 + x * PER;
    a[x] = b[x] = make_uint4(0, 0, 0, 0);
    if (i < items) {
      a[x] = *reinterpret_cast<const uint4*>(o + i * D + sub * 8);
      b[x] = *reinterpret_cast<const uint4*>(dout + i * D + sub * 8);
    }
  }
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    const long long i = i0 + x * PER;                      // item = row * H + head
    float s = bw_dot8<BF16>(a[x], b[x]);
#pragma unroll
    for (int m = L / 2; m > 0; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
    if (sub == 0 && i < items) {
      const long long row = i / H;
      const int h = (int)(i - row * H);
      delta[((row / S) * H + h) * S + (row % S)] = s;
    }
  }
}

__device__ __forceinline__ float bw_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Whole-warp wait, one lane spinning on the non-blocking test_wait (try_wait may park the thread for a while: these
// hand-offs are on the critical path of every pair)
__device__ __forceinline__ void bw_wait_warp(uint32_t bar, uint32_t parity) {
  if ((threadIdx.x & 31) == 0) mbar_wait_spin(bar, parity);
  __syncwarp();
}

// tcgen05.mma / commit issued from CONVERGED warp code (every lane runs the loop, elect.sync picks the issuing lane): measured 5 to 8 %
// faster over the whole kernel than the same instructions inside `if (lane == 0)`.
__device__ __forceinline__ void umma_f16_w(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// the A operand (16-bit, row = lane, two k values per column) comes from TMEM
__device__ __forceinline__ void umma_f16_ts_w(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit_w(uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar) : "memory");
}

// 32 lanes x 8 columns register -> TMEM
__device__ __forceinline__ void tmem_st_32x8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}

template <bool BF16>
__device__ __forceinline__ uint32_t bw_pack16(float a, float b) {
  if (BF16) return pack_bf16x2(a, b);
  const __half2 hh = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&hh);
}

// MODE_Q false: dK / dV of one 128-key block (K, V resident, query tiles stream). MODE_Q true: dQ of one 128-row query tile
// (Q, dO resident, key blocks stream). tmq: tensor map over qkv [B, S, W]; tmd: over dout [B, S, H*D]; both box {64, 64, 1}. The
// entry of the batch is a dimension of its own so that rows past its end arrive as zeros: with their scores masked alone, what lies
// there (the next entry's rows) would still be multiplied by zero, and a NaN among it would arrive in the sums.
template <bool BF16, bool MODE_Q, int D>
__global__ void __launch_bounds__(kBwThreads, 1)
flash_bwd_tc_kernel(const __grid_constant__ CUtensorMap tmq, const __grid_constant__ CUtensorMap tmd, const FlashBwdTcParams p) {
  using L = BwSmem<D>;
  constexpr int kHalves = L::kHalves, NST = kBwStages;
  extern __shared__ __align__(1024) uint8_t smem_bw[];
  const uint32_t sbase = smem_u32(smem_bw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = p.S, H = p.H, Hkv = p.Hkv, G = H / Hkv;

  // ---- what this CTA owns (128 rows from r0 of batch b) and what streams through it ----
  int b, r0, hk, hq = 0, i_min = 0, nqt = 0, n_iter;
  if (!MODE_Q) {
    b = blockIdx.x / Hkv; hk = blockIdx.x % Hkv; r0 = blockIdx.y * kBwBM;
    i_min = p.causal ? r0 / kBwBN : 0;
    nqt = (S + kBwBN - 1) / kBwBN - i_min;
    n_iter = G * nqt;
  } else {
    b = blockIdx.x / H; hq = blockIdx.x % H; hk = hq / G; r0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * kBwBM;
    const int kv_end = p.causal ? min(S, r0 + kBwBM) : S;
    n_iter = (kv_end + kBwBN - 1) / kBwBN;
  }
  const int row_base = b * S;
  // query head and first streamed row of pair n
  auto pair_of = [&](int n, int& qh, int& row) {
    if (!MODE_Q) { const int g = n / nqt; qh = hk * G + g; row = (i_min + n - g * nqt) * kBwBN; }
    else { qh = hq; row = n * kBwBN; }
  };

  const uint32_t sRes = sbase, sRing = sbase + L::kRing;
  const uint32_t bar = sbase + L::kBar;
  const uint32_t res_full = bar, st_full0 = bar + 8, st_empty0 = bar + 40, s_full0 = bar + 72, ds_full0 = bar + 88, acc_done = bar + 104,
                 tmem_slot = bar + 112;
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmq);
    tma_prefetch_desc(&tmd);
    mbar_init(res_full, 1);
    for (int s = 0; s < NST; ++s) { mbar_init(st_full0 + 8 * s, MODE_Q ? 1 : 2); mbar_init(st_empty0 + 8 * s, 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(s_full0 + 8 * s, 1); mbar_init(ds_full0 + 8 * s, kBwEw); }
    mbar_init(acc_done, 1);
    fence_mbar_init();
  }
  if (warp == kBwEw + 1) { tmem_alloc(tmem_slot, kBwTmemCols); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t tmem_base;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));

  if (warp == kBwEw) {
    if (lane == 0) {
      const int kcol = (H + hk) * D, vcol = (H + Hkv + hk) * D;
      // resident tiles: K and V, or Q and dO; per 64-column half two 64-row boxes stacked
      mbar_arrive_expect_tx(res_full, 2 * L::kRes);
      for (int half = 0; half < kHalves; ++half)
        for (int rb = 0; rb < 2; ++rb) {
          const uint32_t dst = sRes + half * 16384 + rb * 8192;
          const int row = r0 + rb * 64;
          tma_load_3d(dst, &tmq, res_full, (MODE_Q ? hq * D : kcol) + half * 64, row, b);
          tma_load_3d(dst + L::kRes, MODE_Q ? &tmd : &tmq, res_full, (MODE_Q ? hq * D : vcol) + half * 64, row, b);
        }
      for (int n = 0; n < n_iter; ++n) {
        const int s = n % NST;
        int qh, row;
        pair_of(n, qh, row);
        mbar_wait(st_empty0 + 8 * s, (((uint32_t)(n / NST)) & 1u) ^ 1u);
        mbar_arrive_expect_tx(st_full0 + 8 * s, L::kStage);
        const uint32_t dst = sRing + s * L::kStage;
        for (int half = 0; half < kHalves; ++half) {       // Q and dO, or K and V
          tma_load_3d(dst + half * 8192, &tmq, st_full0 + 8 * s, (MODE_Q ? kcol : qh * D) + half * 64, row, b);
          tma_load_3d(dst + L::kTile + half * 8192, MODE_Q ? &tmq : &tmd, st_full0 + 8 * s, (MODE_Q ? vcol : qh * D) + half * 64, row, b);
        }
      }
    }
  } else if (warp == kBwEw + 1) {
    {   // the whole warp runs this block (see umma_f16_w)
      constexpr uint32_t kHi = (1024u >> 4) | (1u << 14) | (kSwizzle128B << 29);
      constexpr uint32_t kLoK = (16u >> 4) << 16;
      constexpr uint32_t kLoMN = (8192u >> 4) << 16;     // MN-major 64-row tile: 64-column chunks 8 KB apart
      auto desc = [](uint32_t lo) { return ((uint64_t)kHi << 32) | (uint64_t)lo; };
      const uint32_t idesc_s = make_idesc_f16(kBwBM, kBwBN, BF16, false, false);
      const uint32_t idesc_acc = make_idesc_f16(kBwBM, D, BF16, false, true);
      auto ring = [&](int n) { return sRing + (uint32_t)(n % NST) * L::kStage; };
      auto issue_sdp = [&](int n) {
        const uint32_t buf = tmem_base + (uint32_t)(n & 1) * kBwTBuf;
#pragma unroll
        for (int which = 0; which < 2; ++which) {
          const uint32_t al = ((sRes + which * L::kRes) >> 4) | kLoK, bl = ((ring(n) + which * L::kTile) >> 4) | kLoK;
#pragma unroll
          for (int half = 0; half < kHalves; ++half)
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              umma_f16_w(buf + (which ? kBwTdP : kBwTS), desc(al + half * (16384u >> 4) + ks * 2u), desc(bl + half * (8192u >> 4) + ks * 2u),
                         idesc_s, (half | ks) ? 1u : 0u);
        }
        umma_commit_w(s_full0 + 8 * (n & 1));
      };
      mbar_wait_spin(res_full, 0);
      mbar_wait_spin(st_full0, 0);
      tc_fence_after();
      issue_sdp(0);
      for (int n = 0; n < n_iter; ++n) {
        if (n + 1 < n_iter) {
          mbar_wait_spin(st_full0 + 8 * ((n + 1) % NST), ((uint32_t)((n + 1) / NST)) & 1u);
          // buffer (n + 1) & 1 last held pair n - 1, whose P and dS are read by products issued before this one: the pipe runs in order
          tc_fence_after();
          issue_sdp(n + 1);
        }
        mbar_wait_spin(ds_full0 + 8 * (n & 1), ((uint32_t)n >> 1) & 1u);      // P and dS of pair n are in TMEM
        tc_fence_after();
        const uint32_t buf = tmem_base + (uint32_t)(n & 1) * kBwTBuf;
        const uint32_t first = (ring(n) >> 4) | kLoMN, second = ((ring(n) + L::kTile) >> 4) | kLoMN;
        // the 64 k values lie as 4 x 8 columns, 16 apart: each quarter of the element-wise warps writes where it has read
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          if (!MODE_Q) umma_f16_ts_w(tmem_base + kBwTAcc + D, buf + kBwTS + ks * 16, desc(second + ks * (2048u >> 4)), idesc_acc, (n | ks) ? 1u : 0u);   // dV += P^T dO
        }
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          umma_f16_ts_w(tmem_base + kBwTAcc, buf + kBwTdP + ks * 16, desc(first + ks * (2048u >> 4)), idesc_acc, (n | ks) ? 1u : 0u);   // dK += dS^T Q, or dQ += dS K
        }
        umma_commit_w(st_empty0 + 8 * (n % NST));
      }
      umma_commit_w(acc_done);
    }
  } else if (warp == kBwEw + 2) {
    if (!MODE_Q) {                                         // lse (in units of log 2; rows past the end: infinity, so that P = 0) and delta
      for (int n = 0; n < n_iter; ++n) {
        const int s = n % NST;
        int qh, row;
        pair_of(n, qh, row);
        float lse[2], dl[2];
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          const int q = row + lane + 32 * x;
          const long long o = ((long long)b * H + qh) * S + q;
          lse[x] = q < S ? p.lse[o] * 1.4426950408889634f : INFINITY;
          dl[x] = q < S ? p.delta[o] : 0.f;
        }
        mbar_wait(st_empty0 + 8 * s, (((uint32_t)(n / NST)) & 1u) ^ 1u);
        const uint32_t at = sbase + L::kStats + s * 512;
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + (lane + 32 * x) * 4), "f"(lse[x]) : "memory");
          asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + 256 + (lane + 32 * x) * 4), "f"(dl[x]) : "memory");
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(st_full0 + 8 * s);
      }
    }
  } else {
    // ================= element-wise: thread = (resident row, quarter of the streamed rows) =================
    const int wq = warp & 3, c = warp >> 2;        // TMEM lane quarter, 16-column part of S / dP
    const int r = wq * 32 + lane, own = r0 + r;    // position of this thread's row
    const uint32_t lane_addr = (uint32_t)(wq * 32) << 16;
    const float sl = p.scale_log2, sc = p.scale;
    float lse_own = INFINITY, dl_own = 0.f;
    if (MODE_Q && own < S) {
      const long long o = ((long long)b * H + hq) * S + own;
      lse_own = p.lse[o] * 1.4426950408889634f;
      dl_own = p.delta[o];
    }
    for (int n = 0; n < n_iter; ++n) {
      int qh, row;
      pair_of(n, qh, row);
      const int col0 = row + c * 16;               // position of this thread's first column
      const bool need_mask = MODE_Q ? ((p.causal && row + kBwBN - 1 > r0) || row + kBwBN > S)
                                    : ((p.causal && r0 + kBwBM - 1 > row) || r0 + kBwBM > S || row + kBwBN > S);
      const uint32_t buf = tmem_base + lane_addr + (uint32_t)(n & 1) * kBwTBuf + c * 16;
      const float4* stats = reinterpret_cast<const float4*>(smem_bw + L::kStats + (n % NST) * 512 + c * 64);
      if (!MODE_Q) bw_wait_warp(st_full0 + 8 * (n % NST), ((uint32_t)(n / NST)) & 1u);
      bw_wait_warp(s_full0 + 8 * (n & 1), ((uint32_t)n >> 1) & 1u);
      tc_fence_after();
      uint32_t sv[16], dv[16], pw[8], dw[8];
      tmem_ld_32x16(buf + kBwTS, sv);
      tmem_ld_32x16(buf + kBwTdP, dv);
      float ls[16], de[16];
#pragma unroll
      for (int i = 0; i < 16; i += 4) {
        if (MODE_Q) {
#pragma unroll
          for (int e = 0; e < 4; ++e) { ls[i + e] = lse_own; de[i + e] = dl_own; }
        } else {
          *reinterpret_cast<float4*>(&ls[i]) = stats[i / 4];
          *reinterpret_cast<float4*>(&de[i]) = stats[16 + i / 4];
        }
      }
      tmem_ld_wait();
      if (need_mask) {                             // a masked score is minus infinity and its dP zero, whatever lies there
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const int q = MODE_Q ? own : col0 + i, k = MODE_Q ? col0 + i : own;
          if (q >= S || k >= S || (p.causal && k > q)) { sv[i] = 0xff800000u; dv[i] = 0u; }
        }
      }
      float pv[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) pv[i] = bw_ex2(fmaf(__uint_as_float(sv[i]), sl, -ls[i]));
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        pw[i] = bw_pack16<BF16>(pv[2 * i], pv[2 * i + 1]);
        dw[i] = bw_pack16<BF16>(pv[2 * i] * (__uint_as_float(dv[2 * i]) - de[2 * i]) * sc,
                                pv[2 * i + 1] * (__uint_as_float(dv[2 * i + 1]) - de[2 * i + 1]) * sc);
      }
      if (!MODE_Q) tmem_st_32x8(buf + kBwTS, pw);
      tmem_st_32x8(buf + kBwTdP, dw);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_full0 + 8 * (n & 1));
    }
    // ---- write the accumulators out through shared memory (the resident tiles are dead) for 16-byte coalesced stores. The four warps of
    //      a lane quarter split the columns: of dK (two) and dV (two) in mode KV, of dQ in mode Q ----
    bw_wait_warp(acc_done, 0);
    tc_fence_after();
    constexpr int CH = D / 8, kCols = MODE_Q ? D / 4 : D / 2;      // 16-byte chunks of a row, columns of a warp
    const int which = MODE_Q ? 0 : c >> 1, c0 = (MODE_Q ? c : c & 1) * kCols;
    const uint32_t orow = sRes + (uint32_t)which * L::kRes + (uint32_t)r * (D * 2u);
#pragma unroll 1
    for (int cc = c0; cc < c0 + kCols; cc += 16) {
      uint32_t v[16];
      tmem_ld_32x16(tmem_base + lane_addr + kBwTAcc + which * D + cc, v);
      tmem_ld_wait();
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) w[e] = bw_pack16<BF16>(__uint_as_float(v[g * 8 + e * 2]), __uint_as_float(v[g * 8 + e * 2 + 1]));
        const uint32_t chunk = (uint32_t)(cc / 8 + g);
        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(orow + ((chunk ^ ((uint32_t)r & (CH - 1u))) << 4)), "r"(w[0]),
                     "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
      }
    }
    asm volatile("bar.sync 1, %0;" ::"n"(kBwEw * 32) : "memory");  // every part of every row is in shared memory
    constexpr int kRows = MODE_Q ? 8 : 16;                         // rows a warp copies
    const int part = MODE_Q ? 0 : warp >> 3;                       // dK or dV
    const uint32_t tile = sRes + (uint32_t)part * L::kRes;
    uint16_t* out = reinterpret_cast<uint16_t*>(p.dqkv) + (long long)(MODE_Q ? hq : (part ? H + Hkv + hk : H + hk)) * D;
#pragma unroll
    for (int it = 0; it < kRows * CH / 32; ++it) {
      const int rr = (MODE_Q ? warp : (warp & 7)) * kRows + it * (32 / CH) + lane / CH, chunk = lane % CH;
      uint32_t w0, w1, w2, w3;
      asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(w0), "=r"(w1), "=r"(w2), "=r"(w3)
                   : "r"(tile + (uint32_t)rr * (D * 2u) + (((uint32_t)chunk ^ ((uint32_t)rr & (CH - 1u))) << 4)));
      if (r0 + rr < S) *reinterpret_cast<uint4*>(out + (long long)(row_base + r0 + rr) * p.W + chunk * 8) = make_uint4(w0, w1, w2, w3);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kBwEw + 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kBwTmemCols);
  }
}

template <bool BF16, int D>
static int launch_bwd(const CUtensorMap& tmq, const CUtensorMap& tmd, const FlashBwdTcParams& p, const void* out, const void* dout, float* delta,
                      cudaStream_t st) {
  constexpr int kSmem = (int)BwSmem<D>::kBytes;
  // per call: the attribute belongs to the current device, and a process may use several
  B200_CHECK(cudaFuncSetAttribute(flash_bwd_tc_kernel<BF16, false, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
  B200_CHECK(cudaFuncSetAttribute(flash_bwd_tc_kernel<BF16, true, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
  const long long items = (long long)p.B * p.S * p.H;
  constexpr int per = 2 * 256 / (D / 8);
  flash_delta_tc_kernel<BF16, D><<<(unsigned)((items + per - 1) / per), 256, 0, st>>>((const uint16_t*)out, (const uint16_t*)dout, delta, items, p.S, p.H);
  B200_LAUNCH_CHECK();
  const int blocks = (p.S + kBwBM - 1) / kBwBM;
  flash_bwd_tc_kernel<BF16, false, D><<<dim3(p.Hkv * p.B, blocks), kBwThreads, kSmem, st>>>(tmq, tmd, p);
  B200_LAUNCH_CHECK();
  flash_bwd_tc_kernel<BF16, true, D><<<dim3(p.H * p.B, blocks), kBwThreads, kSmem, st>>>(tmq, tmd, p);
  B200_LAUNCH_CHECK();
  return 0;
}

}  // namespace b200
using namespace b200;

// dqkv [B*S, (H + 2 Hkv) * D] = gradient of the fused projection for dout [B*S, H * D] (16-bit). out / lse are the
// forward's outputs (lse natural log, [B, H, S]); delta [B, H, S] is a caller-provided fp32 work buffer. head_dim 64 or 128, scale > 0,
// no dropout; B200_ERR_UNSUPPORTED otherwise (callers then use b200_flash_attn_bwd).
B200_API int b200_flash_attn_bwd_tc(const void* qkv, const void* out, const void* dout, const float* lse, float* delta, void* dqkv,
                                    int B, int S, int H, int Hkv, int D, int causal, float scale, int dtype, void* stream) {
  // scale > 0: scores are masked before they are multiplied by it (see flash_tc.cu); other scales are the mma.sync kernel's
  if ((D != 64 && D != 128) || (dtype != B200_DT_BF16 && dtype != B200_DT_FP16) || !(scale > 0.f)) return B200_ERR_UNSUPPORTED;
  if (B < 1 || S < 1 || H < 1 || Hkv < 1 || H % Hkv) return B200_ERR_BAD_SHAPE;
  if ((S + kBwBM - 1) / kBwBM > 65535 || (long long)H * B > 0x7fffffffLL) return B200_ERR_UNSUPPORTED;
  if ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(dout) |
       reinterpret_cast<uintptr_t>(dqkv)) & 15) return B200_ERR_BAD_ALIGN;
  // autograd's backward threads have no current driver context until a runtime call binds the primary one; the tensor-map
  // encode below is a driver entry point
  { int dev = 0; B200_CHECK(cudaGetDevice(&dev)); B200_CHECK(cudaSetDevice(dev)); }
  const long long W = (long long)(H + 2 * Hkv) * D;
  CUtensorMap tmq, tmd;
  {
    uint64_t dims[3] = {(uint64_t)W, (uint64_t)S, (uint64_t)B}, str[2] = {(uint64_t)W * 2, (uint64_t)W * 2 * S};
    uint32_t box[3] = {64, 64, 1};
    if (int rc = make_tensor_map(&tmq, qkv, 2, 3, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
    uint64_t dims2[3] = {(uint64_t)H * D, (uint64_t)S, (uint64_t)B}, str2[2] = {(uint64_t)H * D * 2, (uint64_t)H * D * 2 * S};
    if (int rc = make_tensor_map(&tmd, dout, 2, 3, dims2, str2, box, CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
  }
  FlashBwdTcParams p = {};
  p.dqkv = dqkv; p.lse = lse; p.delta = delta; p.B = B; p.S = S; p.H = H; p.Hkv = Hkv; p.W = W;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f; p.causal = causal;
  cudaStream_t st = (cudaStream_t)stream;
  const bool bf = dtype == B200_DT_BF16;
  if (D == 64) return bf ? launch_bwd<true, 64>(tmq, tmd, p, out, dout, delta, st) : launch_bwd<false, 64>(tmq, tmd, p, out, dout, delta, st);
  return bf ? launch_bwd<true, 128>(tmq, tmd, p, out, dout, delta, st) : launch_bwd<false, 128>(tmq, tmd, p, out, dout, delta, st);
}
