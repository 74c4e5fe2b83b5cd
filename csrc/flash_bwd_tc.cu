// K4 backward on the 5th-generation tensor cores: dQ, dK, dV of causal flash attention with every product on tcgen05.mma,
// accumulators in TMEM, operands by TMA straight out of the fused qkv / dout matrices, no atomics and no fp32 gradient
// staging buffer.
//
// One kernel body, two modes, launched one after the other. An item is 128 rows that stay; a CTA (one per SM) takes items in turn, the longest
// first, and the ring of what streams, S and dP of the next item's first pair and its resident tiles run on across the ends of items.
//   mode Q   item = (128-row query tile, query head, batch), first: Q, dO stay; the 64-key blocks it sees stream. TMEM lanes are queries:
//              S = Q K^T, dP = dO V^T   (M 128 x N 64 x K D), double-buffered, issued one pair AHEAD
//              warps 0-15, thread = (row, quarter of the block's keys): P = exp2(S c - lse), dS = P (dP - delta) scale -> 16 bit, over dP in TMEM
//              dQ += dS K               (M 128 x N D x K 64, A from TMEM, B in place)
//            delta = rowsum(dO O) is formed here, from a tile of O that takes a stage of the ring in front of the item's pairs
//   mode KV  item = (128-key block, kv head, batch): K, V stay; the (query head of the group, 64-row query tile) pairs that see the block
//            stream. TMEM lanes are KEYS: S^T = K Q^T, dP^T = V dO^T; P and dS as above over S^T and dP^T, lse and delta of the pair's 64
//            queries in shared memory; dV += P^T dO, dK += dS^T Q over ALL pairs, GQA group included
// What bounds it is shared memory (128 bytes a cycle): a 128 x 64 x 16 product with both operands there takes 48 cycles for 32 of
// tensor time, so P and dS, which are computed in registers anyway, go back to TMEM, and the resident tiles too where its columns are enough
// (mode Q, and mode KV with heads of 64). Then the element-wise warps: two exponentials a cycle and SM at most, and their issue slots.
// S and dP are recomputed in the second mode (7 products instead of 5) in exchange for: no red.global traffic (the atomics of a
// one-pass kernel are 64 KB per 128 x 128 pair), no zero-filled fp32 [tokens, 3 x heads x D] buffer, bit-reproducible gradients.
// Measured (bf16, causal; dK / dV pass + dQ pass + a launch for delta before -> now), one item to a CTA, delta apart and products with both
// operands in shared memory before: 1 x 4096, 32 / 8 heads of 128: 276 + 212 + 15 -> 233 + 179 us; 4 x 512, 40 / 8 heads: 53 + 43 + 11 -> 47 + 39;
// 32 x 256, 12 heads of 64: 46 + 38 + 8 -> 29 + 30; 8 x 1761, 8 heads of 64 (fp16): 129 + 91 + 7 -> 86 + 75. Of it, items in turn and packed
// element-wise arithmetic gave the most (46 -> 29); Q and dO in TMEM 202 -> 181 at 4096. An item's end costs 4000 cycles with them on the
// way (9000 where O came by loads of the element-wise warps: any load on its way holds up every wait of theirs).
//
// 608 threads: warps 0-15 element-wise (four share a TMEM lane quarter and split the 64 columns: a pair is a chain of TMEM reads, FMAs,
// exponentials and TMEM writes, and it is warps beside one another that hide it), warp 16 TMA producer, warp 17 tcgen05
// issuer, warp 18 the rows' lse (and delta, mode KV); 1 CTA per SM (512 TMEM columns). head_dim 64 or
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
constexpr uint32_t kBwTmemCols = 512;
constexpr uint32_t kBwTS = 0, kBwTdP = 64, kBwTBuf = 128, kBwTAcc = 256;   // S(b) at b*128, dP(b) at 64 + b*128, accumulators from 256

// shared memory: the resident tiles [128 rows] of two items, two each (halves of 64 columns, 16 KiB each), the stages of two tiles [64 rows],
// lse | delta of the stages' rows (mode KV) or the parts of delta | lse (mode Q), barriers
template <int D> struct BwSmem {
  static constexpr int NST = D == 64 ? 4 : 3;               // shared memory holds no more for heads of 128
  static constexpr uint32_t kHalves = D / 64, kRes = 16384 * kHalves, kTile = 8192 * kHalves, kStage = 2 * kTile;
  static constexpr uint32_t kRing = 4 * kRes, kStats = kRing + NST * kStage, kBar = kStats + 2560, kBytes = kBar + 256;
  static_assert(kBytes <= 227 * 1024, "shared memory");
};

struct FlashBwdTcParams {
  void* dqkv;             // [B*S, W] 16-bit, same layout as qkv
  const float* lse;       // [B, H, S] natural log
  float* delta;           // [B, H, S] rowsum(dO * O): mode Q forms it, mode KV reads it
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

// A row of tcgen05.mma along k, issued from CONVERGED warp code in one piece: one elect.sync for all of them and the operands of a step a
// constant away from the one before (a product at a time took the issuing warp, which shares its scheduler with four others, longer
// than the tensor pipe). TS: the A operand (16-bit, row = lane, two k values per column) comes from TMEM. The steps are A0 and B0 apart;
// after four, where there are eight, the second halves begin A4 and B4 after the first. `acc`: whether the first step accumulates.
#define BW_MMA(PRED, DSTEP) "@q tcgen05.mma.cta_group::1.kind::f16 [%0], " DSTEP ", %3, " PRED ";\n\t"
template <int STEPS, int A0, int A4, int B0, int B4>
__device__ __forceinline__ void umma_row_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  static_assert(STEPS == 4 || STEPS == 8, "steps");
  asm volatile(
      "{\n\t.reg .pred q, t, f;\n\t.reg .b32 a1, a2, a3;\n\t.reg .b64 b1, b2, b3;\n\t"
      "elect.sync _|q, 0xffffffff;\n\tsetp.ne.b32 f, %4, 0;\n\tsetp.eq.b32 t, %4, %4;\n\t"
      "add.u32 a1, %1, %5;\n\tadd.u32 a2, a1, %5;\n\tadd.u32 a3, a2, %5;\n\t"
      "add.u64 b1, %2, %6;\n\tadd.u64 b2, b1, %6;\n\tadd.u64 b3, b2, %6;\n\t"
      BW_MMA("f", "[%1], %2") BW_MMA("t", "[a1], b1") BW_MMA("t", "[a2], b2") BW_MMA("t", "[a3], b3") "}"
      ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(acc), "n"(A0), "n"(B0) : "memory");
  if constexpr (STEPS == 8) umma_row_ts<4, A0, 0, B0, 0>(d, a + A4, b + B4, idesc, 1u);
}
template <int STEPS, int A0, int A4, int B0, int B4>
__device__ __forceinline__ void umma_row_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  static_assert(STEPS == 4 || STEPS == 8, "steps");
  asm volatile(
      "{\n\t.reg .pred q, t, f;\n\t.reg .b64 a1, a2, a3;\n\t.reg .b64 b1, b2, b3;\n\t"
      "elect.sync _|q, 0xffffffff;\n\tsetp.ne.b32 f, %4, 0;\n\tsetp.eq.b32 t, %4, %4;\n\t"
      "add.u64 a1, %1, %5;\n\tadd.u64 a2, a1, %5;\n\tadd.u64 a3, a2, %5;\n\t"
      "add.u64 b1, %2, %6;\n\tadd.u64 b2, b1, %6;\n\tadd.u64 b3, b2, %6;\n\t"
      BW_MMA("f", "%1, %2") BW_MMA("t", "a1, b1") BW_MMA("t", "a2, b2") BW_MMA("t", "a3, b3") "}"
      ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc), "n"(A0), "n"(B0) : "memory");
  if constexpr (STEPS == 8) umma_row_ss<4, A0, 0, B0, 0>(d, a + A4, b + B4, idesc, 1u);
}
#undef BW_MMA
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

// 32 lanes x 16 (8) columns register -> TMEM
__device__ __forceinline__ void bw_tmem_st(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
               "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void bw_tmem_st(uint32_t taddr, const uint32_t (&r)[8]) { tmem_st_32x8(taddr, r); }

template <bool BF16>
__device__ __forceinline__ uint32_t bw_pack16(float a, float b) {
  if (BF16) return pack_bf16x2(a, b);
  const __half2 hh = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&hh);
}

// MODE_Q false: dK / dV of one 128-key block (K, V resident, query tiles stream). MODE_Q true: dQ of one 128-row query tile
// (Q, dO resident, key blocks stream). tmq: tensor map over qkv [B, S, W]; tmd, tmo: over dout and out [B, S, H*D]; all box {64, 64, 1}. The
// entry of the batch is a dimension of its own so that rows past its end arrive as zeros: with their scores masked alone, what lies
// there (the next entry's rows) would still be multiplied by zero, and a NaN among it would arrive in the sums.
template <bool BF16, bool MODE_Q, int D>
__global__ void __launch_bounds__(kBwThreads, 1)
flash_bwd_tc_kernel(const __grid_constant__ CUtensorMap tmq, const __grid_constant__ CUtensorMap tmd, const __grid_constant__ CUtensorMap tmo,
                    const FlashBwdTcParams p) {
  using L = BwSmem<D>;
  constexpr int kHalves = L::kHalves, NST = L::NST;
  // RT: the resident tiles are the A operands of S and dP from TMEM, where the element-wise warps put them: from shared memory the two
  // products of a pair are bound by its port (16 x 48 cycles for heads of 128), from TMEM by the tensor pipe (16 x 32). dK and dV of heads
  // of 128 leave no columns for them.
  constexpr bool RT = MODE_Q || D == 64;
  constexpr uint32_t kTRes = kBwTAcc + (MODE_Q ? D : 2 * D);
  static_assert(!RT || kTRes + D <= kBwTmemCols, "TMEM");
  extern __shared__ __align__(1024) uint8_t smem_bw[];
  const uint32_t sbase = smem_u32(smem_bw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = p.S, H = p.H, Hkv = p.Hkv, G = H / Hkv;
  const int blocks = (S + kBwBM - 1) / kBwBM, heads = (MODE_Q ? H : Hkv) * p.B, items = heads * blocks;

  // ---- item `index`: 128 rows from r0 of batch b, and what streams through it; the longest items have the lowest indexes ----
  struct Item { int b, hk, hq, r0, i_min, nqt, n_iter; };
  // the k-th item of this CTA, there and back, so that a CTA with a longer one of the first round gets a shorter one of the second
  auto index_of = [&](int k) { return k * (int)gridDim.x + ((k & 1) ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x); };
  auto item_of = [&](int k, Item& t) {
    const int index = index_of(k);
    if (index >= items) return false;
    const int x = index % heads, y = index / heads;
    if (!MODE_Q) {
      t.b = x / Hkv; t.hk = x % Hkv; t.hq = 0; t.r0 = y * kBwBM;
      t.i_min = p.causal ? t.r0 / kBwBN : 0;
      t.nqt = (S + kBwBN - 1) / kBwBN - t.i_min;
      t.n_iter = G * t.nqt;
    } else {
      t.b = x / H; t.hq = x % H; t.hk = t.hq / G; t.r0 = (blocks - 1 - y) * kBwBM; t.i_min = t.nqt = 0;
      const int kv_end = p.causal ? min(S, t.r0 + kBwBM) : S;
      t.n_iter = (kv_end + kBwBN - 1) / kBwBN;
    }
    return true;
  };
  // query head and first streamed row of the item's pair n
  auto pair_of = [&](const Item& t, int n, int& qh, int& row) {
    if (!MODE_Q) { const int g = n / t.nqt; qh = t.hk * G + g; row = (t.i_min + n - g * t.nqt) * kBwBN; }
    else { qh = t.hq; row = n * kBwBN; }
  };
  // stage and phase of the pair that a role has come to
  struct Ring {
    int s = 0;
    uint32_t ph = 0;
    __device__ void next() { if (++s == NST) { s = 0; ph ^= 1u; } }
  };

  const uint32_t sRing = sbase + L::kRing, bar = sbase + L::kBar;
  auto res_at = [&](int k) { return sbase + (uint32_t)(k & 1) * 2 * L::kRes; };
  const uint32_t res_full0 = bar, res_empty0 = bar + 16, s_full0 = bar + 32, ds_full0 = bar + 48, acc_full = bar + 64, tm_full = bar + 72, lse_full = bar + 80, lse_empty = bar + 88,
                 st_full0 = bar + 96, st_empty0 = bar + 128, tmem_slot = bar + 160;
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmq);
    tma_prefetch_desc(&tmd);
    if (MODE_Q) tma_prefetch_desc(&tmo);
    for (int s = 0; s < NST; ++s) { mbar_init(st_full0 + 8 * s, MODE_Q ? 1 : 2); mbar_init(st_empty0 + 8 * s, 1); }
    for (int s = 0; s < 2; ++s) {
      mbar_init(res_full0 + 8 * s, 1); mbar_init(res_empty0 + 8 * s, kBwEw);
      mbar_init(s_full0 + 8 * s, 1); mbar_init(ds_full0 + 8 * s, kBwEw);
    }
    mbar_init(acc_full, 1); mbar_init(tm_full, kBwEw);
    mbar_init(lse_full, 1); mbar_init(lse_empty, kBwEw);
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
      Ring st;
      Item t, u;
      // resident tiles: K and V, or Q and dO; per 64-column half two 64-row boxes stacked
      auto load_resident = [&](int k, const Item& t) {
        const uint32_t rf = res_full0 + 8 * (k & 1);
        mbar_wait(res_empty0 + 8 * (k & 1), (((uint32_t)k >> 1) & 1u) ^ 1u);
        mbar_arrive_expect_tx(rf, 2 * L::kRes);
        for (int half = 0; half < kHalves; ++half)
          for (int rb = 0; rb < 2; ++rb) {
            const uint32_t dst = res_at(k) + half * 16384 + rb * 8192;
            const int row = t.r0 + rb * 64;
            tma_load_3d(dst, &tmq, rf, (MODE_Q ? t.hq : H + t.hk) * D + half * 64, row, t.b);
            tma_load_3d(dst + L::kRes, MODE_Q ? &tmd : &tmq, rf, (MODE_Q ? t.hq : H + Hkv + t.hk) * D + half * 64, row, t.b);
          }
      };
      if (item_of(0, t)) load_resident(0, t);
      for (int k = 0; item_of(k, t); ++k) {
        const int kcol = (H + t.hk) * D, vcol = (H + Hkv + t.hk) * D;
        if (MODE_Q) {                                      // the tile of O, for delta, takes a stage in front of the item's pairs
          mbar_wait(st_empty0 + 8 * st.s, st.ph ^ 1u);
          mbar_arrive_expect_tx(st_full0 + 8 * st.s, L::kRes);
          for (int half = 0; half < kHalves; ++half)
            for (int rb = 0; rb < 2; ++rb)
              tma_load_3d(sRing + st.s * L::kStage + half * 16384 + rb * 8192, &tmo, st_full0 + 8 * st.s, t.hq * D + half * 64, t.r0 + rb * 64, t.b);
          st.next();
        }
        for (int n = 0; n < t.n_iter; ++n, st.next()) {
          int qh, row;
          pair_of(t, n, qh, row);
          mbar_wait(st_empty0 + 8 * st.s, st.ph ^ 1u);
          mbar_arrive_expect_tx(st_full0 + 8 * st.s, L::kStage);
          const uint32_t dst = sRing + st.s * L::kStage;
          for (int half = 0; half < kHalves; ++half) {     // Q and dO, or K and V
            tma_load_3d(dst + half * 8192, &tmq, st_full0 + 8 * st.s, (MODE_Q ? kcol : qh * D) + half * 64, row, t.b);
            tma_load_3d(dst + L::kTile + half * 8192, MODE_Q ? &tmq : &tmd, st_full0 + 8 * st.s, (MODE_Q ? vcol : qh * D) + half * 64, row, t.b);
          }
          // the next item's, early: they come from HBM. Their place is free when the item before this one has been written out, which
          // happens in front of this item's first pair
          if (n == min(2, t.n_iter - 1) && item_of(k + 1, u)) load_resident(k + 1, u);
        }
      }
    }
  } else if (warp == kBwEw + 1) {
    {   // the whole warp runs this block (see umma_row_ts)
      constexpr uint32_t kHi = (1024u >> 4) | (1u << 14) | (kSwizzle128B << 29);
      constexpr uint32_t kLoK = (16u >> 4) << 16;
      constexpr uint32_t kLoMN = (8192u >> 4) << 16;     // MN-major 64-row tile: 64-column chunks 8 KB apart
      auto desc = [](uint32_t lo) { return ((uint64_t)kHi << 32) | (uint64_t)lo; };
      const uint32_t idesc_s = make_idesc_f16(kBwBM, kBwBN, BF16, false, false);
      const uint32_t idesc_acc = make_idesc_f16(kBwBM, D, BF16, false, true);
      auto issue_sdp = [&](int k, int i, int s) {          // of the i-th pair, whose stage is s, of item k
        const uint32_t buf = tmem_base + (uint32_t)(i & 1) * kBwTBuf, ring = sRing + s * L::kStage, res = res_at(k);
#pragma unroll
        for (int which = 0; which < 2; ++which) {
          const uint32_t al = ((res + which * L::kRes) >> 4) | kLoK, bl = ((ring + which * L::kTile) >> 4) | kLoK;
          const uint32_t dst = buf + (which ? kBwTdP : kBwTS);
          if (RT) umma_row_ts<4 * kHalves, 8, 32, 2, 8192 / 16>(dst, tmem_base + kTRes + which * (D / 2), desc(bl), idesc_s, 0u);
          else umma_row_ss<4 * kHalves, 2, 16384 / 16, 2, 8192 / 16>(dst, desc(al), desc(bl), idesc_s, 0u);
        }
        umma_commit_w(s_full0 + 8 * (i & 1));
      };
      // S and dP are asked for one pair ahead of the products that use them, across the ends of items too (RT: there after them, since the
      // element-wise warps put the next item's tiles into TMEM when they are done with the last pair's S and dP)
      Ring st, sa;
      Item t, ta;
      int k = 0, ka = 0, na = 0;
      bool more = item_of(0, ta);
      auto ahead = [&](int i) {
        if (!more) return;
        if (na == 0) {
          if (RT) mbar_wait_spin(tm_full, (uint32_t)ka & 1u);
          if (MODE_Q) sa.next();                           // O's stage
          if (!RT) mbar_wait_spin(res_full0 + 8 * (ka & 1), ((uint32_t)ka >> 1) & 1u);
        }
        mbar_wait_spin(st_full0 + 8 * sa.s, sa.ph);
        __syncwarp();                                      // each lane has looked for itself (see umma_row_ts)
        // buffer i & 1 last held pair i - 2, whose P and dS are read by products issued before this one: the pipe runs in order
        tc_fence_after();
        issue_sdp(ka, i, sa.s);
        sa.next();
        if (++na == ta.n_iter) { na = 0; more = item_of(++ka, ta); }
      };
      ahead(0);
      for (int i = 0; item_of(k, t); ++k) {
        const uint32_t acc = tmem_base + kBwTAcc;
        if (MODE_Q) st.next();
        for (int n = 0; n < t.n_iter; ++n, ++i, st.next()) {
          if (!RT || n + 1 < t.n_iter) ahead(i + 1);
          // P and dS of the pair are in TMEM (and the accumulators of the item before have been read)
          mbar_wait_spin(ds_full0 + 8 * (i & 1), ((uint32_t)i >> 1) & 1u);
          __syncwarp();
          tc_fence_after();
          const uint32_t buf = tmem_base + (uint32_t)(i & 1) * kBwTBuf, ring = sRing + st.s * L::kStage;
          const uint32_t first = (ring >> 4) | kLoMN, second = ((ring + L::kTile) >> 4) | kLoMN;
          // the 64 k values lie as 4 x 8 columns, 16 apart: each quarter of the element-wise warps writes where it has read
          if (!MODE_Q) umma_row_ts<4, 16, 0, 2048 / 16, 0>(acc + D, buf + kBwTS, desc(second), idesc_acc, n ? 1u : 0u);   // dV += P^T dO
          umma_row_ts<4, 16, 0, 2048 / 16, 0>(acc, buf + kBwTdP, desc(first), idesc_acc, n ? 1u : 0u);   // dK += dS^T Q, or dQ += dS K
          umma_commit_w(st_empty0 + 8 * st.s);
        }
        umma_commit_w(acc_full);
        if (RT) ahead(i);
      }
    }
  } else if (warp == kBwEw + 2) {
    if (MODE_Q) {                                          // minus lse of the next item's rows, while the element-wise warps are at the item before
      Item t;
      for (int k = 0; item_of(k, t); ++k) {
        float lse[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const int row = t.r0 + lane + 32 * x;
          lse[x] = row < S ? p.lse[((long long)t.b * H + t.hq) * S + row] * -1.4426950408889634f : -INFINITY;
        }
        mbar_wait(lse_empty, ((uint32_t)k & 1u) ^ 1u);
#pragma unroll
        for (int x = 0; x < 4; ++x)
          asm volatile("st.shared.f32 [%0], %1;" ::"r"(sbase + L::kStats + 2048 + (lane + 32 * x) * 4), "f"(lse[x]) : "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(lse_full);
      }
    } else {                                               // minus lse (in units of log 2; rows past the end: minus infinity, so that P = 0) and minus delta times the scale
      Ring st;
      Item t;
      for (int k = 0; item_of(k, t); ++k)
        for (int n = 0; n < t.n_iter; ++n, st.next()) {
          int qh, row;
          pair_of(t, n, qh, row);
          float lse[2], dl[2];
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const int q = row + lane + 32 * x;
            const long long o = ((long long)t.b * H + qh) * S + q;
            lse[x] = q < S ? p.lse[o] * -1.4426950408889634f : -INFINITY;
            dl[x] = q < S ? p.delta[o] * -p.scale : 0.f;
          }
          mbar_wait(st_empty0 + 8 * st.s, st.ph ^ 1u);
          const uint32_t at = sbase + L::kStats + st.s * 512;
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + (lane + 32 * x) * 4), "f"(lse[x]) : "memory");
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + 256 + (lane + 32 * x) * 4), "f"(dl[x]) : "memory");
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(st_full0 + 8 * st.s);
        }
    }
  } else {
    // ================= element-wise: thread = (resident row, quarter of the streamed rows) =================
    const int wq = warp & 3, c = warp >> 2;        // TMEM lane quarter, 16-column part of S / dP
    const int r = wq * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(wq * 32) << 16;
    const float sl = p.scale_log2, sc = p.scale;
    constexpr int OV = D / 32;                     // 16-byte pieces of a quarter of a row
    Ring st;
    Item t;
    int i = 0;
    bool live = item_of(0, t);
    float lse_own = -INFINITY, dl_own = 0.f;       // minus lse; minus delta times the scale
    // Item k's resident tiles into TMEM, this thread's quarter of its row of each; mode Q: and delta of the row, rowsum(dO * O), whose quarters
    // meet in shared memory
    auto take = [&](const Item& t, int k) {
      if (!RT) return;
      bw_wait_warp(res_full0 + 8 * (k & 1), ((uint32_t)k >> 1) & 1u);
      auto quarter = [&](uint32_t tile, uint32_t (&w)[4 * OV]) {
#pragma unroll
        for (int e = 0; e < OV; ++e) {
          const int chunk = c * OV + e;            // of the row's 16-byte pieces; 8 to a half
          asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(w[4 * e]), "=r"(w[4 * e + 1]), "=r"(w[4 * e + 2]), "=r"(w[4 * e + 3])
                       : "r"(tile + (uint32_t)(chunk >> 3) * 16384 + r * 128 + (((chunk ^ r) & 7) << 4)) : "memory");
        }
      };
      uint32_t w[4 * OV], o[4 * OV];
      quarter(res_at(k), w);
      bw_tmem_st(tmem_base + lane_addr + kTRes + c * (D / 8), w);
      quarter(res_at(k) + L::kRes, w);
      bw_tmem_st(tmem_base + lane_addr + kTRes + D / 2 + c * (D / 8), w);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tm_full);
      if (MODE_Q) {
        bw_wait_warp(st_full0 + 8 * st.s, st.ph);
        quarter(sRing + st.s * L::kStage, o);
        float part = 0.f;
#pragma unroll
        for (int e = 0; e < OV; ++e)
          part += bw_dot8<BF16>(make_uint4(o[4 * e], o[4 * e + 1], o[4 * e + 2], o[4 * e + 3]), make_uint4(w[4 * e], w[4 * e + 1], w[4 * e + 2], w[4 * e + 3]));
        const uint32_t at = sbase + L::kStats + r * 4;
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + c * 512), "f"(part) : "memory");
        bw_wait_warp(lse_full, (uint32_t)k & 1u);
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(lse_own) : "r"(at + 2048) : "memory");
        asm volatile("bar.sync 1, %0;" ::"n"(kBwEw * 32) : "memory");
        if (threadIdx.x == 0) mbar_arrive(st_empty0 + 8 * st.s);       // O is read
        if (lane == 0) mbar_arrive(lse_empty);
        st.next();
        float d[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(d[x]) : "r"(at + x * 512) : "memory");
        asm volatile("bar.sync 1, %0;" ::"n"(kBwEw * 32) : "memory");  // all have read the parts: the next item's may be written
        dl_own = (d[0] + d[1]) + (d[2] + d[3]);
        if (c == 0 && t.r0 + r < S) p.delta[((long long)t.b * H + t.hq) * S + t.r0 + r] = dl_own;
        dl_own *= -sc;
      }
    };
    if (live) take(t, 0);
    for (int k = 0; live; ++k) {
      const int own = t.r0 + r;                    // position of this thread's row
      const uint32_t res = res_at(k);
      const int row_lo = MODE_Q ? 0 : t.i_min * kBwBN, row_hi = MODE_Q ? 0x7fffffff : (t.i_min + t.nqt) * kBwBN;
      int row = row_lo;                            // first streamed row of the pair (pair_of, without its division)
      for (int n = 0; n < t.n_iter; ++n, ++i, st.next(), row = row + kBwBN < row_hi ? row + kBwBN : row_lo) {
        const int col0 = row + c * 16;             // position of this thread's first column
        const bool need_mask = MODE_Q ? ((p.causal && row + kBwBN - 1 > t.r0) || row + kBwBN > S)
                                      : ((p.causal && t.r0 + kBwBM - 1 > row) || t.r0 + kBwBM > S || row + kBwBN > S);
        const uint32_t buf = tmem_base + lane_addr + (uint32_t)(i & 1) * kBwTBuf + c * 16;
        const float4* stats = reinterpret_cast<const float4*>(smem_bw + L::kStats + st.s * 512 + c * 64);
        if (!MODE_Q) bw_wait_warp(st_full0 + 8 * st.s, st.ph);
        bw_wait_warp(s_full0 + 8 * (i & 1), ((uint32_t)i >> 1) & 1u);
        tc_fence_after();
        uint32_t sv[16], dv[16], pw[8], dw[8];
        tmem_ld_32x16(buf + kBwTS, sv);
        tmem_ld_32x16(buf + kBwTdP, dv);
        float ls[16], de[16];
#pragma unroll
        for (int x = 0; x < 16; x += 4) {
          if (MODE_Q) {
#pragma unroll
            for (int e = 0; e < 4; ++e) { ls[x + e] = lse_own; de[x + e] = dl_own; }
          } else {
            *reinterpret_cast<float4*>(&ls[x]) = stats[x / 4];
            *reinterpret_cast<float4*>(&de[x]) = stats[16 + x / 4];
          }
        }
        tmem_ld_wait();
        if (need_mask) {                           // a masked score is minus infinity and its dP zero, whatever lies there
#pragma unroll
          for (int x = 0; x < 16; ++x) {
            const int q = MODE_Q ? own : col0 + x, kk = MODE_Q ? col0 + x : own;
            if (q >= S || kk >= S || (p.causal && kk > q)) { sv[x] = 0xff800000u; dv[x] = 0u; }
          }
        }
        const float2 sl2 = make_float2(sl, sl), sc2 = make_float2(sc, sc);
#pragma unroll
        for (int x = 0; x < 8; ++x) {              // P = exp2(S c - lse), dS = P (dP scale - delta scale)
          float2 e = __ffma2_rn(make_float2(__uint_as_float(sv[2 * x]), __uint_as_float(sv[2 * x + 1])), sl2, make_float2(ls[2 * x], ls[2 * x + 1]));
          e.x = bw_ex2(e.x); e.y = bw_ex2(e.y);
          const float2 f = __fmul2_rn(e, __ffma2_rn(make_float2(__uint_as_float(dv[2 * x]), __uint_as_float(dv[2 * x + 1])), sc2,
                                                    make_float2(de[2 * x], de[2 * x + 1])));
          pw[x] = bw_pack16<BF16>(e.x, e.y);
          dw[x] = bw_pack16<BF16>(f.x, f.y);
        }
        if (!MODE_Q) tmem_st_32x8(buf + kBwTS, pw);
        tmem_st_32x8(buf + kBwTdP, dw);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(ds_full0 + 8 * (i & 1));
      }
      const Item o = t;
      live = item_of(k + 1, t);
      if (live) take(t, k + 1);                    // S and dP of this item have all been read: the products are done with its tiles
      // ---- write the accumulators out through shared memory (the item's resident tiles are dead) for 16-byte coalesced stores. The four
      //      warps of a lane quarter split the columns: of dK (two) and dV (two) in mode KV, of dQ in mode Q ----
      bw_wait_warp(acc_full, (uint32_t)k & 1u);
      tc_fence_after();
      constexpr int CH = D / 8, kCols = MODE_Q ? D / 4 : D / 2;      // 16-byte chunks of a row, columns of a warp
      const int which = MODE_Q ? 0 : c >> 1, c0 = (MODE_Q ? c : c & 1) * kCols;
      const uint32_t orow = res + (uint32_t)which * L::kRes + (uint32_t)r * (D * 2u);
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
      tc_fence_before();
      asm volatile("bar.sync 1, %0;" ::"n"(kBwEw * 32) : "memory");  // every part of every row is in shared memory
      constexpr int kRows = MODE_Q ? 8 : 16;                         // rows a warp copies
      const int part = MODE_Q ? 0 : warp >> 3;                       // dK or dV
      const uint32_t tile = res + (uint32_t)part * L::kRes;
      uint16_t* out = reinterpret_cast<uint16_t*>(p.dqkv) + (long long)(MODE_Q ? o.hq : (part ? H + Hkv + o.hk : H + o.hk)) * D;
      constexpr int kIt = kRows * CH / 32;
      uint4 v[kIt];
      const int rr0 = (MODE_Q ? warp : (warp & 7)) * kRows + lane / CH, chunk = lane % CH;
#pragma unroll
      for (int it = 0; it < kIt; ++it) {
        const int rr = rr0 + it * (32 / CH);
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v[it].x), "=r"(v[it].y), "=r"(v[it].z), "=r"(v[it].w)
                     : "r"(tile + (uint32_t)rr * (D * 2u) + (((uint32_t)chunk ^ ((uint32_t)rr & (CH - 1u))) << 4)) : "memory");
      }
      fence_proxy_async_smem();                    // the tiles' next contents come by TMA; in front of the stores, which it would wait for
      __syncwarp();
      if (lane == 0) mbar_arrive(res_empty0 + 8 * (k & 1));
#pragma unroll
      for (int it = 0; it < kIt; ++it) {
        const int rr = rr0 + it * (32 / CH);
        if (o.r0 + rr < S) *reinterpret_cast<uint4*>(out + (long long)(o.b * S + o.r0 + rr) * p.W + chunk * 8) = v[it];
      }
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
static int launch_bwd(const CUtensorMap& tmq, const CUtensorMap& tmd, const CUtensorMap& tmo, const FlashBwdTcParams& p, cudaStream_t st) {
  constexpr int kSmem = (int)BwSmem<D>::kBytes;
  // per call: the attribute belongs to the current device, and a process may use several
  B200_CHECK(cudaFuncSetAttribute(flash_bwd_tc_kernel<BF16, false, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
  B200_CHECK(cudaFuncSetAttribute(flash_bwd_tc_kernel<BF16, true, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
  const long long blocks = (p.S + kBwBM - 1) / kBwBM, q_items = blocks * p.H * p.B, kv_items = blocks * p.Hkv * p.B;
  flash_bwd_tc_kernel<BF16, true, D><<<(unsigned)(q_items < kNumSMs ? q_items : kNumSMs), kBwThreads, kSmem, st>>>(tmq, tmd, tmo, p);
  B200_LAUNCH_CHECK();
  flash_bwd_tc_kernel<BF16, false, D><<<(unsigned)(kv_items < kNumSMs ? kv_items : kNumSMs), kBwThreads, kSmem, st>>>(tmq, tmd, tmo, p);
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
  if ((long long)((S + kBwBM - 1) / kBwBM) * H * B > 0x3fffffffLL) return B200_ERR_UNSUPPORTED;
  if ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(dout) |
       reinterpret_cast<uintptr_t>(dqkv)) & 15) return B200_ERR_BAD_ALIGN;
  // autograd's backward threads have no current driver context until a runtime call binds the primary one; the tensor-map
  // encode below is a driver entry point
  { int dev = 0; B200_CHECK(cudaGetDevice(&dev)); B200_CHECK(cudaSetDevice(dev)); }
  const long long W = (long long)(H + 2 * Hkv) * D;
  CUtensorMap tmq, tmd, tmo;
  {
    uint64_t dims[3] = {(uint64_t)W, (uint64_t)S, (uint64_t)B}, str[2] = {(uint64_t)W * 2, (uint64_t)W * 2 * S};
    uint32_t box[3] = {64, 64, 1};
    if (int rc = make_tensor_map(&tmq, qkv, 2, 3, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
    uint64_t dims2[3] = {(uint64_t)H * D, (uint64_t)S, (uint64_t)B}, str2[2] = {(uint64_t)H * D * 2, (uint64_t)H * D * 2 * S};
    if (int rc = make_tensor_map(&tmd, dout, 2, 3, dims2, str2, box, CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
    if (int rc = make_tensor_map(&tmo, out, 2, 3, dims2, str2, box, CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
  }
  FlashBwdTcParams p = {};
  p.dqkv = dqkv; p.lse = lse; p.delta = delta; p.B = B; p.S = S; p.H = H; p.Hkv = Hkv; p.W = W;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f; p.causal = causal;
  cudaStream_t st = (cudaStream_t)stream;
  const bool bf = dtype == B200_DT_BF16;
  if (D == 64) return bf ? launch_bwd<true, 64>(tmq, tmd, tmo, p, st) : launch_bwd<false, 64>(tmq, tmd, tmo, p, st);
  return bf ? launch_bwd<true, 128>(tmq, tmd, tmo, p, st) : launch_bwd<false, 128>(tmq, tmd, tmo, p, st);
}
