// K4 on the 5th-generation tensor cores: flash-attention forward with tcgen05.mma, S, P and O in TMEM, Q / K / V tiles brought in
// by TMA in place (no head transposes, GQA by column offset), online softmax by four warps whose threads each own ONE query
// row (TMEM lane = row, so row max and row sum need no shuffles).
//
//   CTA = 128 query rows; 256 threads: warps 0-3 softmax, warp 4 TMA producer, warp 5 tcgen05 issuer (the whole warp runs the
//   issue loop, elect.sync picks the lane); where a CTA goes on from tile to tile (RUN below), warp 6 finds the next one and warp 7
//   writes results out.
//   TMEM (256 columns, two CTAs per SM): S(even j) [0, 64), S(odd j) [64, 128), O [128, 128 + D).
//   per 64-key block j:   S_j = Q K_j^T          (M 128 x N 64 x K D), issued one block AHEAD of the softmax
//                         softmax warps: tcgen05.ld S_j (64 registers), running max, P = exp2(S c - m c) -> 16 bit,
//                                        written over S_j in TMEM (tcgen05.st, two values per column)
//                         O += P V_j             (M 128 x N D x K 64, A operand from TMEM, V MN-major in place)
//   O never leaves TMEM during the loop but to be scaled when a row's maximum rises (see kSlack; a warp whose 32 rows all keep
//   theirs leaves it alone). The tensor pipe therefore sees QK(j+1), PV(j), QK(j+2), ... back to back while the
//   softmax warps work on block j, and the second resident CTA fills the remaining bubbles.
//
// One kernel, three ways to find the rows (MODE):
//   dense    B sequences of S rows of the fused qkv projection; tile = 128 positions of one head
//   varlen   sequences packed back to back (cu_seqlens on the device); tiles past a sequence's end leave at once
//   paged    pieces of at most 64 rows (b200_multimap_attn_mma's tiles) over a paged cache. The two halves of the 128 rows are
//            two heads of one KV group, so short pieces fill the tensor-core tile and their keys are fetched once for both;
//            where a group's heads are odd in number they are two neighbouring tiles of one run and head. A 64-key block is
//            one TMA box per page (page numbers read one block ahead), blocks that neither the window nor the kept first
//            tokens reach are never fetched; sink, cap, chunks, gate as in multimap_attn_mma.cu
// Rows of K and V past the last key of a sequence belong to somebody else (or were never written): their scores are masked, and
// their V rows are zeroed in shared memory before the product, so that not even a NaN there reaches this sequence.
//
// Takes the place of the mma.sync kernels of flash_attn.cu (other head sizes, other scales and dropout stay there) and
// multimap_attn_mma.cu (other sizes, two maps). Measured against them, bf16: six packed prompts of 77 - 2048 tokens, 32 / 8 heads
// of 128: 237 -> 103 us, 16 / 8 heads of 64: 86 -> 51; pages of 64, 16 / 4 heads of 128, pieces of 2048 and 700 (at 512) tokens beside
// two that decode: 171 -> 57 us, window of 1024: 128 -> 42, chunks with capped scores: 194 -> 80; eight packed prompts of 30 - 250
// tokens (fp16): 19.1 -> 16.4.
// Reference call sites: SDPA behind nn.MultiheadAttention (LLM_Distributed_Trainning/PyTorch/ddp_basics/ddp_gpt_wikitext2.py:89-96),
// HF Qwen3 attention (Fine-Tuning/qwen3-14b-qlora-dist-deepspeed.py:95-107).
#include "common.cuh"
#include "tma_host.h"
#include "../include/b200_ops.h"

namespace b200 {

constexpr int kTcBM = 128, kTcBN = 64;
constexpr int kTcThreads = 256;
constexpr uint32_t kTcTmemCols = 256, kTcTmemO = 128;
constexpr float kTcLog2e = 1.4426950408889634f;
constexpr int kTcGridY = 65535;          // largest second (and third) dimension of a grid
enum { kTcDense = 0, kTcVarlen = 1, kTcPaged = 2 };

// shared memory: Q [128 rows] as D / 64 swizzled halves of 16 KiB, the rings of K and of V [64 rows] as halves of 8 KiB, barriers. K and V
// have rings of their own: K's stage is free as soon as its scores are there, a whole block of softmax before V's. With one ring of two
// stages for both, a block's keys were asked for when the product two blocks before had ended, and the softmax waited 500 of 2000 cycles for
// its scores: 1 x 4096, 32 / 8 heads of 128: 160 -> 136 us (200 with the tiles of one head after another), window of 1024: 54 -> 46.
template <int D> struct TcSmem {
  static constexpr uint32_t kHalves = D / 64, kStage = 8192 * kHalves;
  static constexpr int NK = D == 64 ? 4 : 3, NV = D == 64 ? 4 : 2;      // two CTAs fit an SM
  static constexpr uint32_t kQ = 0, kK = 16384 * kHalves, kV = kK + NK * kStage, kBar = kV + NV * kStage, kBytes = kBar + 512;
};

struct FlashTcParams {
  void* out;
  float* lse;         // [B, H, S] natural-log log-sum-exp of the scaled scores (what the backward kernel reads), may be null
  const int* cu;      // varlen: sequence b is rows [cu[b], cu[b + 1])
  int B, S, H, Hkv;
  int group;          // dense, varlen: heads (of all sequences) whose tiles are taken together, see head_group; 0: all
  unsigned h_inv;     // 2^32 / H, rounded up
  long long out_rs;   // elements between output rows
  float scale_log2;   // softmax scale * log2(e) (capped: cap * log2(e))
  int causal;
  // paged
  const int *tiles, *tile_of, *table;   // tile_of (odd head groups): (run, place in the run, tiles of the run, its first tile)
  int max_blocks, bs_log2, window, keep_first;
  float cin, post;    // capped: scores become tanh(cin q . k) before they are scaled
  b200_attn_opts opt;
};

// the largest of three (a NaN gives way, as in fmaxf)
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float ex2f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// tcgen05.mma issued from CONVERGED warp code (every lane of the issuing warp runs the loop, elect.sync picks the lane):
// measured 5 to 8 % faster over the whole kernel than the same instructions inside `if (lane == 0)`.
__device__ __forceinline__ void umma_f16_w(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// the A operand (P, 16-bit, row = lane, two k values per column) comes from TMEM
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

template <bool BF16>
__device__ __forceinline__ uint32_t pack16(float a, float b) {
  if (BF16) return pack_bf16x2(a, b);
  const __half2 hh = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&hh);
}

// tanh for capped scores: by its power series where every score that the row sees in the block is small (|x| <= 1/4: the next term is
// below 3e-9 of x), else 1 - 2 / (1 + e^(2x)) on the hardware's exponential (a few 1e-7 absolute)
__device__ __forceinline__ float tanh_small(float x) {
  const float y = x * x;
  return x * fmaf(y, fmaf(y, fmaf(y, fmaf(y, 62.f / 2835.f, -17.f / 315.f), 2.f / 15.f), -1.f / 3.f), 1.f);
}
__device__ __forceinline__ float tanh_any(float x) { return 1.f - __fdividef(2.f, 1.f + ex2f(x * 2.8853900817779268f)); }

// RUN: a CTA goes on to the tiles of CTAs that have not started (clusterlaunchcontrol). The next tile's Q and keys come, and its first scores are taken,
// while the softmax warps finish the one before; a warp of its own writes that out by TMA. Set-up, the wait for the first scores and the
// end were 13 000 of a CTA's 26 000 cycles for sequences of 512 (8000 or 4600 of them the wait, in the first round and after it). One tile to a CTA
// before: 4 x 512, 40 / 8 heads of 128: packed 37.9 -> 33.9 us; six packed prompts of 77 to 2048
// tokens, 32 / 8 heads: 105 -> 100; eleven of 17 to 1000, 40 / 8 heads: 52 -> 46; eight of 1000, 16 heads of 64: 59 -> 56; one of 4096
// or 8192: the same. A piece of a paged prompt starts with its page numbers either way and gained nothing (102 us for 5596 tokens), with capped scores
// it lost a fifth to registers spilled in the loop; so pieces, and calls of few tiles (see fused_qkv), keep a tile to a CTA.
template <int MODE, int D, bool BF16, bool CAP, bool RUN>
__global__ void __launch_bounds__(kTcThreads, 2)
flash_fwd_tc_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk, const __grid_constant__ CUtensorMap tv,
                    const __grid_constant__ CUtensorMap to, const FlashTcParams p) {
  using L = TcSmem<D>;
  constexpr int kHalves = L::kHalves, NK = L::NK, NV = L::NV;
  // How far a row's maximum may run ahead of the one its weights refer to before O is scaled (an exponent of two). With none the largest
  // weight is 1 and has no rounding error, as in the mma.sync kernels: error of the result against 64 bits 0.00196 (six packed prompts,
  // bf16) and 0.00199 (pieces over pages); with a slack of 8 it was 0.00200 and 0.00206, at 108 and 57 us instead of 114 and 61
  // (before keys and values had rings of their own; with none now 105 and 57). Dense batches with heads of 128 never were on mma.sync here
  // and keep the slack that their kernel was written with.
  constexpr float kSlack = MODE == kTcDense && D == 128 ? 8.f : 0.f;
  extern __shared__ __align__(1024) uint8_t smem_tc[];
  const uint32_t sbase = smem_u32(smem_tc);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // ---- a tile: its rows and keys ----
  struct Tile {
    int h, b, hk, row_base, q0, limit;                    // limit: keys of the sequence; q0: position of row 0; row_base: its row 0
    int nit, nA, bB;                                      // key blocks: [0, nA), then bB, bB + 1, ...; nit 0: no tile any more
    int nrows, low_max, slot;                             // paged
  };
  const int keepW = MODE == kTcPaged && p.window > 0 ? max(p.keep_first, 0) : 0;
  const bool solo = MODE == kTcPaged && ((p.H / p.Hkv) & 1);              // paged: the second half of the rows is the same head's next tile
  auto low_of = [&](int pos) {
    return p.opt.chunk > 0 ? pos / p.opt.chunk * p.opt.chunk : (p.window > 0 ? max(0, pos + 1 - p.window) : 0);
  };
  // the tile that a CTA with this index is for; false: none (a sequence's end, the half of a pair that its other half takes)
  auto tile_of = [&](int bx, int by, int bz, Tile& t) {
    t.h = by; t.b = 0; t.nA = t.bB = 0; t.nrows = kTcBM; t.low_max = 0; t.slot = 0;
    if (MODE == kTcPaged) {
      const int tile = (int)gridDim.x - 1 - bx, rep = p.H / p.Hkv;
      const int* tl = p.tiles + 4 * tile;
      t.row_base = tl[0]; t.nrows = tl[1]; t.q0 = tl[2];
      if (solo) {
        const int place = p.tile_of[4 * tile + 1];
        if (place & 1) return false;                      // the tile before it takes both
        if (place + 1 < p.tile_of[4 * tile + 2]) t.nrows += tl[5];
        t.hk = t.h / rep;
      } else {
        t.hk = t.h / (rep / 2);
        t.h *= 2;
      }
      t.slot = tl[3];
      t.limit = t.q0 + t.nrows;
      const int lo0 = low_of(t.q0);
      t.nA = (min(keepW, lo0) + kTcBN - 1) / kTcBN;
      t.bB = max(lo0 / kTcBN, t.nA);
      t.nit = t.nA + (t.limit + kTcBN - 1) / kTcBN - t.bB;
      t.low_max = low_of(t.q0 + (solo ? kTcBM : kTcBN) - 1);
    } else {
      // Heavy (late) query tiles of all heads and sequences first, or of a group of heads (see head_group): under the causal mask tile t has
      // t + 1 times the work of tile 0, and the short ones fill the end.
      int qt;
      if (p.group == 0) {
        t.h = bx; t.b = by;
        qt = (int)gridDim.z - 1 - bz;
      } else {
        int x = bx;
        qt = (p.S + kTcBM - 1) / kTcBM - 1 - by;
        if (qt >= kTcGridY) {                             // more tiles than the second dimension holds: the first takes the rest
          qt -= x / p.group * kTcGridY;
          x %= p.group;
        }
        const int hb = bz * p.group + x;
        t.b = p.H == 1 ? hb : (int)__umulhi((unsigned)hb, p.h_inv);
        if (t.b >= p.B || qt < 0) return false;
        t.h = hb - t.b * p.H;
      }
      t.hk = t.h / (p.H / p.Hkv);
      t.row_base = MODE == kTcVarlen ? p.cu[t.b] : t.b * p.S;
      t.limit = MODE == kTcVarlen ? p.cu[t.b + 1] - t.row_base : p.S;
      t.q0 = qt * kTcBM;
      if (MODE == kTcVarlen && t.q0 >= t.limit) return false;
      const int kv_end = p.causal ? min(t.limit, t.q0 + kTcBM) : t.limit;
      t.nit = (kv_end + kTcBN - 1) / kTcBN;
    }
    return true;
  };
  Tile t0;
  if (!RUN && !tile_of(blockIdx.x, blockIdx.y, blockIdx.z, t0)) return;

  const uint32_t bar = sbase + L::kBar;
  // P has two barriers: the softmax may be a block ahead of the issuing warp (S(j + 1) is asked for before V(j) and P(j) are waited for).
  // Blocks are counted through all tiles of the CTA (g): buffers, stages and phases go by that.
  const uint32_t q_full = bar, q_empty = bar + 8, s_full0 = bar + 16, p_full0 = bar + 32, o_done = bar + 48, tmem_slot = bar + 56, st_free = bar + 64,
                 tile_full0 = bar + 72, tile_empty0 = bar + 88, ask = bar + 104, clc = bar + 112, clc_at = bar + 256, o_staged = bar + 400;
  auto k_full = [&](int j) { return bar + 120 + 8u * ((uint32_t)j % NK); };
  auto k_empty = [&](int j) { return bar + 120 + 8u * (NK + (uint32_t)j % NK); };
  auto v_full = [&](int j) { return bar + 120 + 8u * (2 * NK + (uint32_t)j % NV); };
  auto v_empty = [&](int j) { return bar + 120 + 8u * (2 * NK + NV + (uint32_t)j % NV); };
  auto k_phase = [&](int j) { return ((uint32_t)j / NK) & 1u; };
  auto v_phase = [&](int j) { return ((uint32_t)j / NV) & 1u; };
  auto k_at = [&](int j) { return sbase + L::kK + ((uint32_t)j % NK) * L::kStage; };
  auto v_at = [&](int j) { return sbase + L::kV + ((uint32_t)j % NV) * L::kStage; };
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tq);
    if (RUN) tma_prefetch_desc(&to);
    if (MODE == kTcPaged) { tma_prefetch_desc(&tk); tma_prefetch_desc(&tv); }
    mbar_init(q_full, 1); mbar_init(q_empty, 1); mbar_init(st_free, 1); mbar_init(o_staged, 4); mbar_init(ask, 1); mbar_init(clc, 1);
    for (int s = 0; s < NK; ++s) { mbar_init(k_full(s), 1); mbar_init(k_empty(s), 1); }
    for (int s = 0; s < NV; ++s) { mbar_init(v_full(s), 1); mbar_init(v_empty(s), 1); }
    for (int s = 0; s < 2; ++s) {
      mbar_init(s_full0 + 8 * s, 1); mbar_init(p_full0 + 8 * s, 4);
      if (RUN) { mbar_init(tile_full0 + 8 * s, 1); mbar_init(tile_empty0 + 8 * s, 7); }   // producer, issuer, four softmax warps, the one that writes out
    }
    mbar_init(o_done, 1);
    fence_mbar_init();
  }
  if (warp == 5) { tmem_alloc(tmem_slot, kTcTmemCols); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t tmem_base;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));

  // The n-th tile of this CTA, for a whole warp; false: there are no more. done_with: its place may be written again
  auto tile_part = [&](int n, int part) {
    int4 x;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w) : "r"(bar + 272 + (n & 1) * 32 + part * 16) : "memory");
    return x;
  };
  auto take_tile = [&](int n, Tile& t) {
    if (!RUN) { t = t0; return n == 0; }
    mbar_wait_warp(tile_full0 + 8 * (n & 1), ((uint32_t)n >> 1) & 1u);
    const int4 a = tile_part(n, 0), b = tile_part(n, 1);
    t.h = a.x; t.b = a.y; t.hk = a.z; t.row_base = a.w; t.q0 = b.x; t.limit = b.y; t.nit = b.z;
    return t.nit > 0;
  };
  auto done_with = [&](int n) {
    if (!RUN) return;
    __syncwarp();
    if (lane == 0) mbar_arrive(tile_empty0 + 8 * (n & 1));
  };

  if (RUN && warp == 6) {
    // ---- tiles: this CTA's own, then those of CTAs that have not started, which need not any more (clusterlaunchcontrol). The next one is taken
    //      when the producer is at the last blocks of the one before: taken early, long tiles would find their turn behind long tiles ----
    if (lane == 0) {
      int bx = blockIdx.x, by = blockIdx.y, bz = blockIdx.z;
      uint32_t clc_phase = 0;
      bool more = true;
      auto next = [&]() {
        mbar_arrive_expect_tx(clc, 16);
        asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(clc_at), "r"(clc) : "memory");
        mbar_wait(clc, clc_phase);
        clc_phase ^= 1u;
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t.reg .b128 r;\n\t"
            "ld.shared.b128 r, [%4];\n\t"
            "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, r;\n\t"
            "selp.u32 %3, 1, 0, p;\n\t"
            "@p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%0, %1, %2, _}, r;\n\t}"
            : "+r"(bx), "+r"(by), "+r"(bz), "=r"(ok) : "r"(clc_at) : "memory");
        fence_proxy_async_smem();                         // the answer is read: the next one may be written there
        return ok != 0;
      };
      for (int n = 0;; ++n) {
        Tile t = {};
        while (more && !tile_of(bx, by, bz, t)) more = next();
        mbar_wait(tile_empty0 + 8 * (n & 1), (((uint32_t)n >> 1) & 1u) ^ 1u);
        int4* at = reinterpret_cast<int4*>(smem_tc + L::kBar + 272 + (n & 1) * 32);
        at[0] = make_int4(t.h, t.b, t.hk, t.row_base);
        at[1] = make_int4(t.q0, t.limit, more ? t.nit : 0, 0);
        mbar_arrive(tile_full0 + 8 * (n & 1));
        if (!more) break;
        mbar_wait(ask, (uint32_t)n & 1u);
        more = next();
      }
    }
  }
  if (RUN && warp == 7) {
    // ---- out: the results that the softmax warps left in the ring of V, 32 rows (a warp's) at a time: by TMA where all of them are the tile's, else
    //      16 bytes to a lane ----
    Tile t;
    for (int n = 0; take_tile(n, t); ++n) {
      done_with(n);
      mbar_wait_warp(o_staged, (uint32_t)n & 1u);
      bool by_hand = false;
#pragma unroll 1
      for (int q = 0; q < 4; ++q) {
        const int live = t.limit - t.q0 - q * 32, first = t.row_base + t.q0 + q * 32;
        const uint32_t at = sbase + L::kV + q * 4096;
        if (live >= 32) {
          if (lane == 0)
            for (int half = 0; half < kHalves; ++half)
              asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%2, %3}], [%1];" ::"l"(&to), "r"(at + half * 16384),
                           "r"(t.h * D + half * 64), "r"(first) : "memory");
        } else if (live > 0) {
          by_hand = true;
          for (int i = lane; i < live * (D / 8); i += 32) {
            const int r = i / (D / 8), c = i % (D / 8);
            uint4 x;
            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w)
                         : "r"(at + (c >> 3) * 16384 + r * 128 + (((c ^ r) & 7) << 4)));
            *reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(p.out) + (long long)(first + r) * p.out_rs + t.h * D + c * 8) = x;
          }
        }
      }
      if (lane == 0) {
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
      }
      if (by_hand) fence_proxy_async_smem();              // the next tile's values come by TMA
      __syncwarp();
      if (lane == 0) mbar_arrive(st_free);
    }
  }
  if (warp == 4) {
    Tile t;
    int g0 = 0;                                           // blocks of the tiles before
    for (int n = 0; take_tile(n, t); g0 += t.nit, ++n) {
      done_with(n);
      const int h = t.h, hk = t.hk, nit = t.nit, limit = t.limit;
      auto block_of = [&](int it) { return MODE == kTcPaged ? (it < t.nA ? it : t.bB + (it - t.nA)) : it; };
      // ---- Q: D / 64 column halves, each 128 rows (two 64-row boxes stacked = one K-major 128B-swizzled tile). The scores before it are done:
      //      with the tile before still in its softmax and its end ----
      if (lane == 0) {
        if (RUN) mbar_wait(q_empty, ((uint32_t)n & 1u) ^ 1u);
        mbar_arrive_expect_tx(q_full, 16384 * kHalves);
        for (int half = 0; half < kHalves; ++half)
          for (int rb = 0; rb < 2; ++rb) {
            const int col = (MODE == kTcPaged && !solo ? h + rb : h) * D + half * 64;
            const int row = MODE == kTcPaged ? t.row_base + (solo ? rb * 64 : 0) : t.row_base + t.q0 + rb * 64;
            tma_load_2d(sbase + L::kQ + half * 16384 + rb * 8192, &tq, q_full, col, row);
          }
      }
      // the ring of V holds the tile before while it is written out
      auto before_v = [&](int j) {
        if (RUN && j == 0 && n > 0) mbar_wait(st_free, (uint32_t)(n - 1) & 1u);
        mbar_wait(v_empty(g0 + j), v_phase(g0 + j) ^ 1u);
      };
      if (MODE == kTcPaged) {
        // a block is `pieces` boxes of `psize` rows; lane i looks up and fetches piece i, its page number one block ahead
        const int* trow = p.table + (long long)t.slot * p.max_blocks;
        const int psl = min(p.bs_log2, 6), psize = 1 << psl, pieces = kTcBN >> psl;
        auto row_of = [&](int it) {
          const int kp = block_of(it) * kTcBN + lane * psize;
          return (it < nit && lane < pieces && kp < limit)
                     ? ((trow[kp >> p.bs_log2] * p.Hkv + hk) << p.bs_log2) + (kp & ((1 << p.bs_log2) - 1)) : -1;
        };
        auto bytes_of = [&](int it) {
          return (uint32_t)(min(pieces, (limit - block_of(it) * kTcBN + psize - 1) >> psl) * psize * 128 * kHalves);
        };
        // block it's keys, then the values of the block before it: a K stage is free long before a V stage
        int row = row_of(0), row_v = -1;
        for (int it = 0; it <= nit; ++it) {
          if (it < nit) {
            const int g = g0 + it;
            if (lane == 0) {
                            mbar_wait(k_empty(g), k_phase(g) ^ 1u);
              mbar_arrive_expect_tx(k_full(g), bytes_of(it));
            }
            __syncwarp();
            if (row >= 0) {
#pragma unroll
              for (int half = 0; half < kHalves; ++half)
                tma_load_2d(k_at(g) + half * 8192 + lane * psize * 128, &tk, k_full(g), half * 64, row);
            }
          }
          const int next = row_of(it + 1);
          if (it > 0) {
            const int j = it - 1, g = g0 + j;
            if (lane == 0) {
              before_v(j);
              mbar_arrive_expect_tx(v_full(g), bytes_of(j));
            }
            __syncwarp();
            if (row_v >= 0) {
#pragma unroll
              for (int half = 0; half < kHalves; ++half)
                tma_load_2d(v_at(g) + half * 8192 + lane * psize * 128, &tv, v_full(g), half * 64, row_v);
            }
          }
          row_v = row;
          row = next;
        }
      } else if (lane == 0) {
        const int kcol = (p.H + hk) * D, vcol = (p.H + p.Hkv + hk) * D;
        for (int j = 0; j <= nit; ++j) {
          if (j < nit) {
            const int g = g0 + j;
            if (RUN && j == max(0, nit - 2)) mbar_arrive(ask);
            mbar_wait(k_empty(g), k_phase(g) ^ 1u);
            mbar_arrive_expect_tx(k_full(g), L::kStage);
            for (int half = 0; half < kHalves; ++half)
              tma_load_2d(k_at(g) + half * 8192, &tk, k_full(g), kcol + half * 64, t.row_base + j * kTcBN);
          }
          if (j > 0) {
            const int g = g0 + j - 1;
            before_v(j - 1);
            mbar_arrive_expect_tx(v_full(g), L::kStage);
            for (int half = 0; half < kHalves; ++half)
              tma_load_2d(v_at(g) + half * 8192, &tv, v_full(g), vcol + half * 64, t.row_base + (j - 1) * kTcBN);
          }
        }
      }
      __syncwarp();
    }
  } else if (warp == 5) {
    {   // the whole warp runs this block (see umma_f16_w)
      // descriptors: hi word = SBO 1024 | version 1 | 128B swizzle; lo word = address >> 4 (| LBO << 16 for MN-major)
      constexpr uint32_t kHi = (1024u >> 4) | (1u << 14) | (kSwizzle128B << 29);
      constexpr uint32_t kLoK = (16u >> 4) << 16, kLoMN = (8192u >> 4) << 16;
      auto desc = [](uint32_t lo) { return ((uint64_t)kHi << 32) | (uint64_t)lo; };
      const uint32_t idesc_qk = make_idesc_f16(kTcBM, kTcBN, BF16, false, false);
      const uint32_t idesc_pv = make_idesc_f16(kTcBM, D, BF16, false, true);
      const uint32_t tS = tmem_base, tO = tmem_base + kTcTmemO;
      const uint32_t qlo = ((sbase + L::kQ) >> 4) | kLoK;
      auto issue_qk = [&](int j) {
        const int s = j & 1;
        const uint32_t klo = (k_at(j) >> 4) | kLoK;
#pragma unroll
        for (int half = 0; half < kHalves; ++half)
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            umma_f16_w(tS + s * kTcBN, desc(qlo + half * (16384u >> 4) + ks * 2u), desc(klo + half * (8192u >> 4) + ks * 2u),
                     idesc_qk, (half | ks) ? 1u : 0u);
        umma_commit_w(s_full0 + 8 * s);
        umma_commit_w(k_empty(j));
      };
      Tile t;
      int g0 = 0;
      for (int n = 0; take_tile(n, t); g0 += t.nit, ++n) {
        done_with(n);
        const int nit = t.nit;
        mbar_wait_spin(q_full, (uint32_t)n & 1u);
        mbar_wait_spin(k_full(g0), k_phase(g0));
        __syncwarp();                                     // each lane has looked for itself (see umma_f16_w)
        tc_fence_after();
        issue_qk(g0);                                     // into the buffer of the last block but one: its P has been read by products issued before
        if (RUN && nit == 1) umma_commit_w(q_empty);
        for (int j = 0; j < nit; ++j) {
          const int g = g0 + j, s = g & 1;
          if (j + 1 < nit) {
            mbar_wait_spin(k_full(g + 1), k_phase(g + 1));
            __syncwarp();
            // S buffer (g+1)&1 last held block g-1: P(g-1) sat in it and PV(g-1) was issued before this UMMA, the pipe runs in order
            tc_fence_after();
            issue_qk(g + 1);
            if (RUN && j + 2 == nit) umma_commit_w(q_empty);     // the tile's scores are done with Q
          }
          mbar_wait_spin(v_full(g), v_phase(g));
          mbar_wait_spin(p_full0 + 8 * s, ((uint32_t)g >> 1) & 1u);     // P(g) is written (and O rescaled where a row needed it; and taken, the tile before)
          __syncwarp();
          tc_fence_after();
          const uint32_t vlo = (v_at(g) >> 4) | kLoMN;
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            umma_f16_ts_w(tO, tS + s * kTcBN + ks * 8, desc(vlo + ks * (2048u >> 4)), idesc_pv, (j | ks) ? 1u : 0u);
          umma_commit_w(o_done);
          umma_commit_w(v_empty(g));
        }
      }
    }
  } else if (warp < 4) {
    // ================= softmax: thread = query row =================
    const int q = warp;                             // TMEM lane quarter this warp may touch (warp index mod 4)
    const int r = q * 32 + lane;                    // row inside the tile
    const int rmask = MODE == kTcPaged && !solo ? 63 : 127;       // two heads: rows 64 .. 127 are the second one's
    const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
    const uint32_t tS = tmem_base + lane_addr, tO = tmem_base + lane_addr + kTcTmemO;
    const float sl = p.scale_log2;
    Tile t;
    int g0 = 0;
    for (int n = 0; take_tile(n, t); g0 += t.nit, ++n) {
    const int nit = t.nit, limit = t.limit, q0 = t.q0, nrows = t.nrows, low_max = t.low_max;
    auto block_of = [&](int it) { return MODE == kTcPaged ? (it < t.nA ? it : t.bB + (it - t.nA)) : it; };
    const int rr = r & rmask, grow = q0 + rr;       // row of the tile, position in the sequence
    const int lim = (MODE == kTcPaged || p.causal) ? min(grow, limit - 1) : limit - 1;      // last visible key of this row
    const int low = MODE == kTcPaged ? low_of(grow) : 0;                                    // first one, besides kept tokens
    float m_ref = -INFINITY, l = 0.f;
    uint32_t v[64];
    for (int j = 0; j < nit; ++j) {
      const int g = g0 + j, kv0 = block_of(j) * kTcBN, sb = g & 1;
      const bool need_mask = MODE == kTcPaged ? (kv0 + kTcBN - 1 > q0 || (kv0 < low_max && kv0 + kTcBN - 1 >= keepW))
                                              : ((p.causal && kv0 + kTcBN - 1 > q0) || (kv0 + kTcBN > limit));
      mbar_wait_warp(s_full0 + 8 * sb, ((uint32_t)g >> 1) & 1u);
      tc_fence_after();
      tmem_ld_32x32(tS + sb * kTcBN, *reinterpret_cast<uint32_t(*)[32]>(&v[0]));
      tmem_ld_32x32(tS + sb * kTcBN + 32, *reinterpret_cast<uint32_t(*)[32]>(&v[32]));
      tmem_ld_wait();
      // Keys the row does not see are taken out before the row chooses its form of tanh, and each row chooses for itself: its result
      // must not depend on what lies behind the sequence, or in its window's other end, nor on the other rows of the tile.
      auto hidden = [&](int kp) { return MODE == kTcPaged ? (kp > lim || (kp < low && kp >= keepW)) : kp > lim; };
      if (CAP) {
        float big = 0.f;
#pragma unroll
        for (int i = 0; i < 64; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * p.cin);
        if (need_mask) {
#pragma unroll
          for (int i = 0; i < 64; ++i)
            if (hidden(kv0 + i)) v[i] = 0u;
        }
#pragma unroll
        for (int i = 0; i < 64; ++i) big = fmaxf(big, fabsf(__uint_as_float(v[i])));
        // Small scores: the series takes fewer cycles than two special functions. Only the warp's branches are decided together (its
        // lanes stay in step for the TMEM accesses below); rows past the end of a short piece go along with the others.
        const bool large = big > 0.25f, dead = MODE == kTcPaged && rr >= nrows;
        if (!__any_sync(0xffffffffu, large && !dead)) {
#pragma unroll
          for (int i = 0; i < 64; ++i) v[i] = __float_as_uint(tanh_small(__uint_as_float(v[i])));
        } else if (__all_sync(0xffffffffu, large || dead)) {
#pragma unroll
          for (int i = 0; i < 64; ++i) v[i] = __float_as_uint(tanh_any(__uint_as_float(v[i])));
        } else {
#pragma unroll
          for (int i = 0; i < 64; ++i) v[i] = __float_as_uint(large ? tanh_any(__uint_as_float(v[i])) : tanh_small(__uint_as_float(v[i])));
        }
      }
      if (need_mask) {
#pragma unroll
        for (int i = 0; i < 64; ++i) {
          if (hidden(kv0 + i)) v[i] = 0xff800000u;        // -inf
        }
      }
      float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};   // four chains: two warps per scheduler hide little
#pragma unroll
      for (int i = 0; i < 64; i += 8)
#pragma unroll
        for (int c = 0; c < 4; ++c) m4[c] = max3(m4[c], __uint_as_float(v[i + 2 * c]), __uint_as_float(v[i + 2 * c + 1]));
      const float mx = fmaxf(max3(m4[0], m4[1], m4[2]), m4[3]);
      const float m_new = fmaxf(m_ref, mx * sl);
      const bool raise = m_new > m_ref + kSlack;
      float alpha = 1.f;
      if (raise) { alpha = ex2f(m_ref - m_new); m_ref = m_new; }
      const float m_use = (m_ref == -INFINITY) ? 0.f : m_ref;
      const bool any_raise = j > 0 && __any_sync(0xffffffffu, raise);
      // PV(j-1) complete: O is stable. A parity wait tells phase c from c + 1, not from c + 2, and S(j) only proves PV(j-2)
      // complete: a warp that skipped this wait for a while is still safe here (o_done has completed j - 1 or j phases), but
      // it must not reach the wait after the loop two phases behind, where the parity of "PV(nit-3) done" reads as
      // "PV(nit-1) done" and O would be taken before the last two products. So the last block always waits.
      if (j > 0 && (any_raise || j == nit - 1)) {
        mbar_wait_warp(o_done, (uint32_t)(g - 1) & 1u);
        tc_fence_after();
      }
      if (any_raise) {
        uint32_t o[32];
#pragma unroll 1
        for (int c = 0; c < D / 32; ++c) {
          tmem_ld_32x32(tO + c * 32, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tmem_st_32x32(tO + c * 32, o);
        }
      }
      l *= alpha;
      float2 rs = make_float2(0.f, 0.f);              // even and odd keys; four sums are no faster
      const float2 nm = make_float2(-m_use, -m_use), sl2 = make_float2(sl, sl);
      uint32_t w[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        float2 e = __ffma2_rn(make_float2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])), sl2, nm);
        e.x = ex2f(e.x); e.y = ex2f(e.y);
        rs = __fadd2_rn(rs, e);
        w[i] = pack16<BF16>(e.x, e.y);
      }
      tmem_st_32x32(tS + sb * kTcBN, w);
      if (kv0 + kTcBN > limit) {                          // the sequence's last block: V rows that are not its own become zeros
        mbar_wait_warp(v_full(g), v_phase(g));
        for (int i = threadIdx.x; i < (kv0 + kTcBN - limit) * 8 * kHalves; i += 128) {
          const int row = limit - kv0 + i / (8 * kHalves), c = i % (8 * kHalves);
          asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(v_at(g) + (c >> 3) * 8192 + row * 128 + (c & 7) * 16),
                       "r"(0) : "memory");
        }
        fence_proxy_async_smem();                         // generic-proxy stores -> visible to tcgen05.mma
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full0 + 8 * sb);
      l += rs.x + rs.y;
    }
    // ---- finish: O / l -> 16 bit through shared memory (the ring of V: every product has completed, and the next tile's values wait) ----
    mbar_wait_warp(o_done, (uint32_t)(g0 + nit - 1) & 1u);
    tc_fence_after();
    const int4 who = RUN ? tile_part(n, 0) : make_int4(t.h, t.b, 0, t.row_base);         // RUN: read again, registers are short in the loop
    const int h = who.x, b = who.y, row_base = who.w;
    const int head = MODE == kTcPaged && !solo ? h + (r >> 6) : h;
    const bool live = MODE == kTcPaged ? rr < nrows : grow < limit;
    if (MODE == kTcPaged && p.opt.sink) l += ex2f(p.opt.sink[head] * kTcLog2e - m_ref);   // no key: not scaled, not capped
    float inv = l > 0.f ? 1.f / l : 0.f;
    if (MODE == kTcPaged) {
      inv *= p.post;
      if (p.opt.gate && live) inv /= 1.f + expf(-p.opt.gate[(long long)(row_base + rr) * p.opt.ld_gate + head]);
    }
    constexpr int CH = D / 8;                             // 16-byte chunks of an output row
    // RUN: in the ring of V, halves of 64 columns, 128 bytes a row, pieces turned by the row (the swizzle of TMA); else over Q, a whole row after another
    const uint32_t orow = RUN ? sbase + L::kV + q * 4096 + lane * 128 : sbase + L::kQ + (uint32_t)r * (D * 2u);
#pragma unroll 1
    for (int c = 0; c < D / 32; ++c) {
      uint32_t o[32];
      tmem_ld_32x32(tO + c * 32, o);
      tmem_ld_wait();
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
          w[e] = pack16<BF16>(__uint_as_float(o[g * 8 + e * 2]) * inv, __uint_as_float(o[g * 8 + e * 2 + 1]) * inv);
        const uint32_t chunk = (uint32_t)(c * 4 + g);
        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(RUN ? orow + (chunk >> 3) * 16384 + (((chunk ^ (uint32_t)lane) & 7u) << 4)
                                                                          : orow + ((chunk ^ ((uint32_t)r & (CH - 1u))) << 4)), "r"(w[0]),
                     "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
      }
    }
    if (RUN) fence_proxy_async_smem();                    // written here, read by TMA
    __syncwarp();
    if (RUN && lane == 0) mbar_arrive(o_staged);
    if (MODE == kTcDense && p.lse && live)
      p.lse[((long long)b * p.H + h) * p.S + grow] = fmaf(__log2f(l), 0.6931471805599453f, __fmul_rn(m_ref, 0.6931471805599453f));
    done_with(n);
    if (!RUN) {
      // each warp copies ITS 32 rows out (written by its own lanes): CH lanes cover the bytes of a row
      uint16_t* obase = reinterpret_cast<uint16_t*>(p.out);
#pragma unroll 4
      for (int it = 0; it < CH; ++it) {
        const int row = q * 32 + it * (32 / CH) + lane / CH, chunk = lane % CH;
        uint32_t w0, w1, w2, w3;
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(w0), "=r"(w1), "=r"(w2), "=r"(w3)
                     : "r"(sbase + L::kQ + (uint32_t)row * (D * 2u) + (((uint32_t)chunk ^ ((uint32_t)row & (CH - 1u))) << 4)));
        const int rw = MODE == kTcPaged && !solo ? (row & 63) : row;
        const bool keep = MODE == kTcPaged ? rw < nrows : q0 + rw < limit;
        const long long at = (long long)(MODE == kTcPaged ? row_base + rw : row_base + q0 + rw) * p.out_rs +
                             (MODE == kTcPaged && !solo ? h + (row >> 6) : h) * D + chunk * 8;
        if (keep) *reinterpret_cast<uint4*>(obase + at) = make_uint4(w0, w1, w2, w3);
      }
    }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 5) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTcTmemCols);
  }
}

template <int MODE, int D, bool BF16, bool CAP, bool RUN>
static int launch_tc(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& to, const FlashTcParams& p, dim3 grid, cudaStream_t st) {
  auto kern = flash_fwd_tc_kernel<MODE, D, BF16, CAP, RUN>;
  // per call: the attribute belongs to the current device, and a process may use several
  B200_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TcSmem<D>::kBytes));
  kern<<<grid, kTcThreads, TcSmem<D>::kBytes, st>>>(tq, tk, tv, to, p);
  B200_LAUNCH_CHECK();
  return 0;
}

// rows [rows, cols] of 16-bit values, boxes of 64 columns
static int rows_map(CUtensorMap* tm, const void* base, uint64_t cols, uint64_t rows, uint32_t box_rows) {
  uint64_t dims[2] = {cols, rows}, str[1] = {cols * 2};
  uint32_t box[2] = {64, box_rows};
  return make_tensor_map(tm, base, 2, 2, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

// autograd's backward threads have no current driver context until a runtime call binds the primary one; the tensor-map encode
// is a driver entry point
static int bind_device() {
  int dev = 0;
  B200_CHECK(cudaGetDevice(&dev));
  B200_CHECK(cudaSetDevice(dev));
  return 0;
}

// Tiles of dense and packed calls go out tile by tile, and a tile of every head reads its keys and values: with heads of 128 they are wanted
// at 9 TB/s, which only L2 has. So where those of all heads are more than its 126 MB, the heads go in groups whose keys and values stay
// there from one tile's turn to the next: 48 MB, less than half of it, since the queries and the results go through it too.
// 16 x 4096, 32 heads of 128 (1.07 GB), causal / full / packed: 2172 / 3949 / 2745 us, in one group 2873 / 5412 / 3231, head by head
// 2701 / 4734 / 2895; 2 x 8192: 1008 / 1916 / 1309, 1127 / 2519 / 1344 and 1346 / 2414 / 1445. 24 to 64 MB differ by 3 %. Heads of 64
// want 3.6 TB/s and stay one group: 64 x 4096, 12 heads (0.8 GB) 3331 us, 3330 in groups; below 126 MB groups gain nothing: 48 x 512
// packed, 40 / 8 heads of 128 (100 MB) 304 us, 310 in groups.
// Sequences of more tiles than a grid's second and third dimension hold (8.4 million rows) take the grouped form as well.
constexpr long long kTcL2Bytes = 126ll << 20, kTcGroupBytes = 48ll << 20;
static int head_group(long long rows, FlashTcParams& p, int D, dim3& grid) {
  const long long tiles = (p.S + kTcBM - 1) / kTcBM, heads = (long long)p.H * p.B, rep = p.H / p.Hkv;
  const long long kv = (rows * D * 4 + p.B - 1) / p.B;    // keys and values of one head of a sequence (packed: of the mean one)
  const bool divides = heads * p.H < (1ll << 32);         // what the kernel's quotient by H takes
  p.group = 0;
  grid = dim3(p.H, p.B, (unsigned)tiles);
  if (tiles <= kTcGridY && (D == 64 || !divides || kv * (heads / rep) <= kTcL2Bytes)) return 0;
  if (!divides) return B200_ERR_UNSUPPORTED;
  const long long over = (tiles + kTcGridY - 1) / kTcGridY;
  long long group = kTcGroupBytes / kv * rep;
  if (group < rep) group = rep;
  if (group * kTcGridY < heads) group = (heads + kTcGridY - 1) / kTcGridY;
  if (group > heads) group = heads;
  const long long groups = (heads + group - 1) / group;
  group = ((heads + groups - 1) / groups + rep - 1) / rep * rep;          // of one size, heads of the same keys together
  if (group * over > 0x7fffffffLL) return B200_ERR_UNSUPPORTED;
  p.group = (int)group;
  p.h_inv = p.H == 1 ? 0 : (unsigned)((1ll << 32) / p.H + 1);
  grid = dim3((unsigned)(group * over), (unsigned)(tiles < kTcGridY ? tiles : kTcGridY), (unsigned)groups);
  return 0;
}

template <int MODE>
static int fused_qkv(const void* qkv, long long rows, FlashTcParams& p, int D, int dtype, void* stream) {
  dim3 grid;
  if (int rc = head_group(rows, p, D, grid)) return rc;
  if (int rc = bind_device()) return rc;
  CUtensorMap tm;
  if (int rc = rows_map(&tm, qkv, (uint64_t)(p.H + 2 * p.Hkv) * D, (uint64_t)rows, 64)) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  const bool bf = dtype == B200_DT_BF16;
  // More tiles than two rounds of two CTAs for each SM: CTAs go on from tile to tile. With none to go on to, or one each, a tile's way through the other
  // warps is not made up for. One tile to a CTA against tiles in turn, us, 8 heads: 400 tiles of 64 tokens, heads of 64: 11.0, 12.2; 352 of 256: 14.6, 16.5; 320 of
  // 1024, heads of 128: 22.0, 22.8; 304 packed of 17: 12.4, 14.2; some are faster in turn (400 of 64, heads of 128: 13.1, 12.5). 592: within 6 % either
  // way. From 640 on: 64 tokens 14.6, 14.5 (heads of 128: 18.7, 16.2), 512 26.9, 24.8 (29.8, 27.1); 896: 18.7, 16.6 (22.9, 18.8), 34.9, 32.1 (41.3, 37.1).
  const bool run = (long long)grid.x * grid.y * grid.z > 4 * kNumSMs;
  CUtensorMap to = tm;
  if (run)
    if (int rc = rows_map(&to, p.out, (uint64_t)p.H * D, (uint64_t)rows, 32)) return rc;
#define TC_ROWS(DD, BB) (run ? launch_tc<MODE, DD, BB, false, true>(tm, tm, tm, to, p, grid, st) : launch_tc<MODE, DD, BB, false, false>(tm, tm, tm, to, p, grid, st))
  return D == 64 ? (bf ? TC_ROWS(64, true) : TC_ROWS(64, false)) : (bf ? TC_ROWS(128, true) : TC_ROWS(128, false));
#undef TC_ROWS
}

}  // namespace b200
using namespace b200;

// The scale is above zero here: scores are masked before they are multiplied by it, and a masked one, minus infinity, would become NaN
// (times 0) or plus infinity. The mma.sync kernels multiply first and take any scale.
static int tc_check(const void* qkv, const void* out, int B, int S, int H, int Hkv, int D, float scale, int dtype) {
  if ((D != 64 && D != 128) || (dtype != B200_DT_BF16 && dtype != B200_DT_FP16) || !(scale > 0.f)) return B200_ERR_UNSUPPORTED;
  if (B < 1 || S < 1 || H < 1 || Hkv < 1 || H % Hkv) return B200_ERR_BAD_SHAPE;
  if (H > 65535 || B > 65535) return B200_ERR_UNSUPPORTED;
  if ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(out)) & 15) return B200_ERR_BAD_ALIGN;
  return 0;
}

// Heads (of all sequences) whose tiles a dense (rows = B * S) or packed call takes together, 0 where it is refused
B200_API int b200_flash_tc_group(long long rows, int B, int S, int H, int Hkv, int D) {
  FlashTcParams p = {};
  dim3 grid;
  p.B = B; p.S = S; p.H = H; p.Hkv = Hkv;
  return rows < 1 || B < 1 || S < 1 || H < 1 || Hkv < 1 || H % Hkv || D < 1 || head_group(rows, p, D, grid) ? 0 : p.group ? p.group : p.H * p.B;
}

// Causal (or full) attention forward on the tcgen05 path. head_dim 64 or 128, 16-bit, no dropout, scale > 0. qkv [B*S, (H + 2 Hkv) * D],
// out [B*S, H * D], lse [B, H, S] or NULL. Returns B200_ERR_UNSUPPORTED for shapes it does not cover (the caller then
// takes b200_flash_attn_fwd).
B200_API int b200_flash_attn_fwd_tc(const void* qkv, void* out, float* lse, int B, int S, int H, int Hkv, int D, int causal,
                                    float scale, int dtype, void* stream) {
  if (int rc = tc_check(qkv, out, B, S, H, Hkv, D, scale, dtype)) return rc;
  FlashTcParams p = {};
  p.out = out; p.lse = lse; p.B = B; p.S = S; p.H = H; p.Hkv = Hkv; p.out_rs = (long long)H * D;
  p.scale_log2 = scale * kTcLog2e; p.causal = causal;
  return fused_qkv<kTcDense>(qkv, (long long)B * S, p, D, dtype, stream);
}

// The packed form (see b200_flash_attn_varlen_fwd): `tokens` rows hold n_seqs sequences back to back, the longest of max_seqlen rows.
B200_API int b200_flash_attn_varlen_fwd_tc(const void* qkv, void* out, const int* cu_seqlens, long long tokens, int n_seqs, int max_seqlen,
                                           int H, int Hkv, int D, int causal, float scale, int dtype, void* stream) {
  if (int rc = tc_check(qkv, out, n_seqs, max_seqlen, H, Hkv, D, scale, dtype)) return rc;
  if (!cu_seqlens || tokens < 1) return B200_ERR_BAD_SHAPE;
  FlashTcParams p = {};
  p.out = out; p.cu = cu_seqlens; p.B = n_seqs; p.S = max_seqlen; p.H = H; p.Hkv = Hkv; p.out_rs = (long long)H * D;
  p.scale_log2 = scale * kTcLog2e; p.causal = causal;
  return fused_qkv<kTcVarlen>(qkv, tokens, p, D, dtype, stream);
}

// Prompt pieces over a paged cache, one map, key and value rows of one size (arguments as in b200_multimap_attn_mma_ex; `tokens`: rows
// of q, `pool_rows`: rows of the pools, blocks * G * block_size; `tile_of` as described above, wanted where H / G is odd).
// B200_ERR_UNSUPPORTED: the caller takes the mma.sync kernel.
B200_API int b200_paged_attn_tc(const void* q, long long tokens, const void* ck, const void* cv, long long pool_rows, const int* tiles,
                                const int* tile_of, int n_tiles, const int* table, int max_blocks, void* out, long long ldo, int H, int G,
                                int D, int block_size, float scale, int window, int keep_first, float post, const b200_attn_opts* opts,
                                int dtype, void* stream) {
  if (n_tiles <= 0) return 0;
  if (int rc = tc_check(q, out, 1, 1, H, G, D, scale, dtype)) return rc;
  const b200_attn_opts opt = opts ? *opts : b200_attn_opts{};
  if (opt.chunk < 0 || (opt.chunk > 0 && window > 0) || !(opt.softcap >= 0.f)) return B200_ERR_UNSUPPORTED;
  const int rep = H / G;
  if ((rep & 1) && !tile_of) return B200_ERR_UNSUPPORTED;
  if (((reinterpret_cast<uintptr_t>(ck) | reinterpret_cast<uintptr_t>(cv)) & 15) || ldo % 8 || pool_rows > 0x7fffffffLL) return B200_ERR_UNSUPPORTED;
  FlashTcParams p = {};
  while ((1 << p.bs_log2) < block_size) ++p.bs_log2;
  if ((1 << p.bs_log2) != block_size || block_size < 8) return B200_ERR_UNSUPPORTED;      // a swizzled box starts on a group of 8 rows
  if (int rc = bind_device()) return rc;
  CUtensorMap tq, tk, tv;
  const uint32_t box = block_size < 64 ? block_size : 64;
  if (int rc = rows_map(&tq, q, (uint64_t)H * D, (uint64_t)tokens, 64)) return rc;
  if (int rc = rows_map(&tk, ck, (uint64_t)D, (uint64_t)pool_rows, box)) return rc;
  if (int rc = rows_map(&tv, cv, (uint64_t)D, (uint64_t)pool_rows, box)) return rc;
  const bool capped = opt.softcap > 0.f;
  p.out = out; p.out_rs = ldo; p.H = H; p.Hkv = G; p.causal = 1; p.tiles = tiles; p.tile_of = tile_of; p.table = table; p.max_blocks = max_blocks;
  p.window = window; p.keep_first = keep_first; p.post = post; p.opt = opt;
  p.scale_log2 = (capped ? opt.softcap : scale) * kTcLog2e;
  p.cin = capped ? scale / opt.softcap : 1.f;
  const dim3 grid(n_tiles, rep & 1 ? H : H / 2);
  cudaStream_t st = (cudaStream_t)stream;
  const bool bf = dtype == B200_DT_BF16;
#define TC_PAGED(DD)                                                                                                           \
  (capped ? (bf ? launch_tc<kTcPaged, DD, true, true, false>(tq, tk, tv, tq, p, grid, st) : launch_tc<kTcPaged, DD, false, true, false>(tq, tk, tv, tq, p, grid, st)) \
          : (bf ? launch_tc<kTcPaged, DD, true, false, false>(tq, tk, tv, tq, p, grid, st) : launch_tc<kTcPaged, DD, false, false, false>(tq, tk, tv, tq, p, grid, st)))
  return D == 64 ? TC_PAGED(64) : TC_PAGED(128);
#undef TC_PAGED
}
