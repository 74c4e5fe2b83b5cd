// Products of 17 to 64 tokens with integer 4-bit codes on the 5th-generation tensor cores: y[m, n] = sum_k x[m, k] w[n, k] (+ bias),
// w = lin_a scale (code - lin_off) - zs, groups of 128, K a multiple of 512 (b200_w4_gemv_linear; other forms stay in gemv.cu).
//
// The weights are the 128-row operand of tcgen05.mma and come from TMEM; the tokens are its N. A code enters as the exact 16-bit value
// b + code with b = 16 (64 for fp16): the nibble OR-ed into the mantissa of b, one logic op per pair. The affine map is applied in fp32 to a
// group's sums:  sum_k w_k x_k = A (sum_k (b + c_k) x_k) - (A (b + lin_off) + zs) sum_k x_k.  sum_k x_k needs no pass over x: lane 31
// of every warp's 32 rows carries codes of zero, so its sums are b sum_k x_k, and it hands them to the warp's other rows. The two
// sums cancel, and their error grows with b; 16 is the smallest that holds a code, and 64 saves fp16 a shift (16: up to 1.2 of 33 us).
// Results that are not the 16-bit number next to the 64-bit one, 64 tokens, N 24576, K 4096: bf16 0.03 %, fp16 1 % (2 % where the
// activations have a mean of 2); with 128 (bf16) and 1024, at the same time: 0.19, 15 and 84 %; mma.sync 0.12, 9 and 38 %.
//
// CTA (one per SM): a slice of k of a tile of R = 4 x (at most 31) rows, tile after tile, two groups (a pair) at a time.
//   warp 0       TMA: codes of a pair (a box of [R rows x 128 bytes]) through a ring as long as fits; scales and zeros of four groups
//   warp 1       tcgen05.mma, sixteen per pair
//   warp 2       TMA: the tokens of a pair. They lie in the order of the codes' pairs ((e0, e4), (e1, e5), (e2, e6), (e3, e7)) in global
//                memory, where a launch of its own puts them; the weights are on their way meanwhile (programmatic dependent launch)
//   warps 4-19   expansion, thread = row: 64 bytes of codes -> 64 TMEM columns; four warps to every fourth group
//   warps 20-27  the groups' sums from TMEM: scaled and added up in fp32, thread = (row, half of the tokens)
// Codes cross shared memory once, as codes, and never as 16-bit values. A cluster of `split` CTAs shares a tile's k; their parts meet
// through distributed shared memory, in the order of the ranks.
// What bounds it: two bytes per weight cross the port of TMEM twice, as tcgen05.st and as the A operand of the products (a step of 16 k takes
// 34 cycles of it whatever the tokens' number), 12 - 18 us for 100 M weights; then the hand-overs between the warps. Both sides in turn, cold
// caches, against mma.sync (w4 of 17 / 32 / 64 tokens, N 24576, K 4096): 77 / 92 / 188 -> 33 / 33 / 51 us; 60 tokens, N 4096, K 12288: 95 -> 39;
// 64 tokens, N 34816, K 5120: 311 -> 61. Up to 16 tokens mma.sync, which expands into registers, is as fast or faster (8 tokens: 25, here 29).
// Eight expanding warps instead of sixteen: 30 and 66 us for 32 and 64 tokens of the first shape.
#include "common.cuh"
#include "tma_host.h"
#include "../include/b200_ops.h"

namespace b200 {

constexpr int kWtTma = 0, kWtMma = 1, kWtTok = 2, kWtExp = 4, kWtSum = 20, kWtThreads = 28 * 32;
constexpr int kWtMaxW = 10, kWtNS = 4, kWtNX = 2;         // stages: codes (at most), scales, tokens
constexpr uint32_t kWtBox = 16384, kWtScale = 4096;       // codes of a pair; scales | zeros of two pairs
constexpr uint32_t kWtSmemMax = 227 * 1024;

struct W4TcArgs {
  const void *x, *packed;
  const float *scale, *zs;      // zs may be null
  const void* bias;             // 16-bit, may be null
  void *y, *ws;
  int M, K;
  long long N, x_rs, y_rs;
  float lin_a, lin_off;
};
// How a product is cut: log2 of the CTAs that share a tile's k (-1: not a form of this kernel), rows of a warp (a tile has four times as
// many), clusters
struct W4TcCut { int split_log2 = -1, rpw = 0, clusters = 0, nw = 0; };

// shared memory: codes | scales | tokens | parts of a tile, twice | sums of tokens | zeros | barriers
struct WtSmem {
  uint32_t sc, x, part, xs, zero, bar, bytes;
  __host__ __device__ WtSmem(int nw, uint32_t xbytes, uint32_t part_bytes) {
    sc = nw * kWtBox; x = sc + kWtNS * kWtScale; part = x + xbytes; xs = part + 2 * part_bytes; zero = xs + 2048; bar = zero + 64; bytes = bar + 512 + 1024;
  }
};

struct W4TcParams {
  const void* bias;
  void* y;
  int M, K, has_zs;
  long long N, y_rs;
  float lin_a, lin_off;
  int split_log2, rpw, nw; // CTAs of a cluster, rows of a warp, stages of codes
  uint32_t part_bytes;
};

__device__ __forceinline__ uint32_t wt_and_or(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ uint4 wt_lds(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void wt_sts(uint32_t a, const uint4& v) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
// The eight products of a group: A (codes) from TMEM, 8 columns a step, B (tokens) from shared memory, 32 bytes a step in each of two
// halves. One elect.sync for all of them, in converged warp code.
template <int HALF>
__device__ __forceinline__ void wt_group(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred q, t, f;\n\t.reg .b32 a1, a2, a3, a4, a5, a6, a7;\n\t.reg .b64 b1, b2, b3, b4, b5, b6, b7;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "setp.eq.b32 t, %3, %3;\n\tsetp.ne.b32 f, %3, %3;\n\t"
      "add.u32 a1, %1, 8;\n\tadd.u32 a2, %1, 16;\n\tadd.u32 a3, %1, 24;\n\tadd.u32 a4, %1, 32;\n\t"
      "add.u32 a5, %1, 40;\n\tadd.u32 a6, %1, 48;\n\tadd.u32 a7, %1, 56;\n\t"
      "add.u64 b1, %2, 2;\n\tadd.u64 b2, %2, 4;\n\tadd.u64 b3, %2, 6;\n\tadd.u64 b4, %2, %4;\n\t"
      "add.u64 b5, b4, 2;\n\tadd.u64 b6, b4, 4;\n\tadd.u64 b7, b4, 6;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, f;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %3, t;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], b2, %3, t;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], b3, %3, t;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a4], b4, %3, t;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a5], b5, %3, t;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a6], b6, %3, t;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a7], b7, %3, t;\n\t}"
      ::"r"(d), "r"(a), "l"(b), "r"(idesc), "n"(HALF) : "memory");
}
__device__ __forceinline__ void wt_commit(uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar) : "memory");
}
// one lane waits for the warp
__device__ __forceinline__ void wt_wait(uint32_t bar, uint32_t parity) {
  if ((threadIdx.x & 31) == 0) mbar_wait(bar, parity);
  __syncwarp();
}
// other CTAs' stores to this one's shared memory, announced on `bar`
__device__ __forceinline__ void wt_wait_cluster(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  const long long t0 = clock64();
  do {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    if (!ok && clock64() - t0 > B200_MBAR_TIMEOUT_CYCLES) {
      printf("b200 w4: wait for the parts of a tile timed out (block %d)\n", blockIdx.x);
      __trap();
    }
  } while (!ok);
}

template <bool BF16>
__device__ __forceinline__ void wt_store(const W4TcParams& p, long long row, int tok, float bias, float v) {
  v += bias;
  if (BF16) reinterpret_cast<__nv_bfloat16*>(p.y)[(long long)tok * p.y_rs + row] = __float2bfloat16_rn(v);
  else reinterpret_cast<__half*>(p.y)[(long long)tok * p.y_rs + row] = __float2half_rn(v);
}

// eight values of a token in the order of the codes' pairs
__device__ __forceinline__ uint4 wt_order(const uint4& w) {
  return make_uint4(__byte_perm(w.x, w.z, 0x5410), __byte_perm(w.x, w.z, 0x7632), __byte_perm(w.y, w.w, 0x5410), __byte_perm(w.y, w.w, 0x7632));
}

// [K / 64][MT tokens][64 values, ordered], zeros past M
__global__ void __launch_bounds__(256)
w4_tc_tokens_kernel(const uint16_t* __restrict__ x, long long x_rs, int M, int K, int mt_log2, uint4* __restrict__ out) {
  pdl_launch_dependents();
  const int i = blockIdx.x * 256 + threadIdx.x, c = i & 7, tok = (i >> 3) & ((1 << mt_log2) - 1), h = i >> (3 + mt_log2);
  if (h >= K / 64) return;
  uint4 v = make_uint4(0, 0, 0, 0);
  if (tok < M) v = wt_order(*reinterpret_cast<const uint4*>(x + tok * x_rs + h * 64 + c * 8));
  out[i] = v;
}

template <bool BF16, int MT>
__global__ void __launch_bounds__(kWtThreads, 1)
w4_tc_kernel(const __grid_constant__ CUtensorMap tw, const __grid_constant__ CUtensorMap tsc, const __grid_constant__ CUtensorMap tzs,
             const __grid_constant__ CUtensorMap tx, const W4TcParams p) {
  constexpr uint32_t kPair = MT * 512;                    // a pair's tokens: four blocks of 64 values
  extern __shared__ uint8_t smem_wt[];
  const WtSmem L(p.nw, kWtNX * kPair, p.part_bytes);
  const uint32_t sb = (smem_u32(smem_wt) + 1023u) & ~1023u;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = 1 << p.split_log2, cr = blockIdx.x & (S - 1), cl = blockIdx.x >> p.split_log2, ncl = gridDim.x >> p.split_log2;
  const int R = 4 * p.rpw;
  const int ntiles = (int)((p.N + R - 1) / R);
  const int T = (ntiles - 1 - cl) / ncl + 1;              // tiles of this cluster: there are no more clusters than tiles
  const int nun = p.K / 512, u0 = nun * cr / S, nu = nun * (cr + 1) / S - u0;      // this CTA's units of four groups in every tile
  const int np = 2 * nu, P = T * np;                      // pairs of a tile, and of all of them

  const uint32_t bar = sb + L.bar;
  auto w_full = [&](int i) { return bar + 8u * i; };
  auto w_empty = [&](int i) { return bar + 8u * (kWtMaxW + i); };
  constexpr int kB = 2 * kWtMaxW;
  auto s_full = [&](int i) { return bar + 8u * (kB + i); };
  auto s_empty = [&](int i) { return bar + 8u * (kB + 4 + i); };
  auto x_full = [&](int i) { return bar + 8u * (kB + 8 + i); };
  auto x_empty = [&](int i) { return bar + 8u * (kB + 10 + i); };
  auto a_full = [&](int i) { return bar + 8u * (kB + 12 + i); };
  auto done = [&](int i) { return bar + 8u * (kB + 14 + i); };          // the pair's products are complete
  auto d_empty = [&](int i) { return bar + 8u * (kB + 16 + i); };
  auto part_full = [&](int i) { return bar + 8u * (kB + 18 + i); };
  const uint32_t tmem_slot = bar + 8u * (kB + 20);
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tw);
    tma_prefetch_desc(&tsc);
    if (p.has_zs) tma_prefetch_desc(&tzs);
    tma_prefetch_desc(&tx);
    for (int i = 0; i < p.nw; ++i) { mbar_init(w_full(i), 1); mbar_init(w_empty(i), 8); }
    for (int i = 0; i < kWtNS; ++i) { mbar_init(s_full(i), 1); mbar_init(s_empty(i), 8); }
    for (int i = 0; i < 2; ++i) {
      mbar_init(x_full(i), 1); mbar_init(x_empty(i), 1); mbar_init(a_full(i), 8); mbar_init(done(i), 1); mbar_init(d_empty(i), 8);
      mbar_init(part_full(i), 8 * S);
    }
    fence_mbar_init();
  }
  if (threadIdx.x < 16) asm volatile("st.shared.u32 [%0], %1;" ::"r"(sb + L.zero + 4 * threadIdx.x), "r"(0) : "memory");
  if (warp == kWtMma) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  if (S > 1) cluster_sync_all();                          // the peers' barriers exist
  tc_fence_after();
  constexpr uint32_t tmem = 0;                            // all 512 columns: the allocation starts at the first

  if (warp == kWtTma) {
    if (lane == 0) {
      const uint32_t sbytes = (uint32_t)R * (p.has_zs ? 32 : 16);
      int st = 0, ss = 0;
      uint32_t ph = 0, sph = 0;
      for (int t = 0; t < T; ++t) {
        const int row0 = (cl + t * ncl) * R;
        for (int n = 0; n < np; ++n) {
          if (!(n & 1)) {
            mbar_wait(s_empty(ss), sph ^ 1u);
            mbar_arrive_expect_tx(s_full(ss), sbytes);
            tma_load_2d(sb + L.sc + ss * kWtScale, &tsc, s_full(ss), u0 * 4 + n * 2, row0);
            if (p.has_zs) tma_load_2d(sb + L.sc + ss * kWtScale + 2048, &tzs, s_full(ss), u0 * 4 + n * 2, row0);
            if (++ss == kWtNS) { ss = 0; sph ^= 1u; }
          }
          mbar_wait(w_empty(st), ph ^ 1u);
          mbar_arrive_expect_tx(w_full(st), (uint32_t)R * 128);
          tma_load_2d(sb + st * kWtBox, &tw, w_full(st), u0 * 256 + n * 128, row0);
          if (++st == p.nw) { st = 0; ph ^= 1u; }
        }
      }
    }
  } else if (warp == kWtTok) {
    if (lane == 0) {
      pdl_wait();                                         // the ordered tokens are there
      for (int t = 0, i = 0; t < T; ++t)
        for (int n = 0; n < np; ++n, ++i) {
          const int xs = i & 1;
          mbar_wait(x_empty(xs), ((uint32_t)(i >> 1) & 1u) ^ 1u);
          mbar_arrive_expect_tx(x_full(xs), kPair);
          tma_load_3d(sb + L.x + xs * kPair, &tx, x_full(xs), 0, 0, u0 * 8 + n * 4);
        }
    }
  } else if (warp == kWtMma) {
    // ================= tcgen05.mma, the whole warp in step =================
    constexpr uint32_t kHi = (1024u >> 4) | (1u << 14) | (kSwizzle128B << 29), kLo = (16u >> 4) << 16;
    const uint32_t idesc = make_idesc_f16(128, MT, BF16, false, false);
    for (int i = 0; i < P; ++i) {
      const int b = i & 1;
      const uint32_t ph = (uint32_t)(i >> 1) & 1u;
      mbar_wait(x_full(b), ph);
      mbar_wait(d_empty(b), ph ^ 1u);
      mbar_wait(a_full(b), ph);
      __syncwarp();                                        // each lane has looked for itself (see wt_group)
      tc_fence_after();
      const uint64_t bd = ((uint64_t)kHi << 32) | ((sb + L.x + b * kPair) >> 4) | kLo;
      wt_group<(MT * 128 >> 4)>(tmem + 256 + b * (2 * MT), tmem + b * 128, bd, idesc);
      wt_group<(MT * 128 >> 4)>(tmem + 256 + b * (2 * MT) + MT, tmem + b * 128 + 64, bd + (kPair / 2 >> 4), idesc);
      wt_commit(done(b));
      wt_commit(x_empty(b));
    }
  } else if (warp >= kWtExp && warp < kWtSum) {
    // ================= codes -> 16-bit values in TMEM, thread = row =================
    const int set = ((warp - kWtExp) >> 2) & 1, b = (warp - kWtExp) >> 3, q = warp & 3, row = q * p.rpw + lane;      // group 2 b + set of every unit
    const bool live = lane < p.rpw;
    constexpr int kUp = BF16 ? 3 : 4;                     // where a nibble lies in the mantissa of 16 or 64
    uint32_t magic = BF16 ? 0x41804180u : 0x54005400u, mask = 0x000F000Fu << kUp;
    asm volatile("" : "+r"(magic), "+r"(mask));           // both stay in registers (one LOP3 per pair of codes)
    const uint32_t ta = tmem + ((uint32_t)(q * 32) << 16) + b * 128 + set * 64;
    uint32_t at[4];                                       // where the group's 64 bytes lie in a stage; other lanes read zeros
#pragma unroll
    for (int c = 0; c < 4; ++c) at[c] = live ? sb + row * 128 + (((uint32_t)(set * 4 + c) ^ (uint32_t)(row & 7)) << 4) : sb + L.zero + c * 16;
    const uint32_t step = live ? kWtBox : 0u;
    int st = b;
    uint32_t ph = 0;
    for (int u = 0; u < P / 2; ++u) {
      wt_wait(w_full(st), ph);
      uint32_t w[16];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const uint4 x = wt_lds(at[c] + st * step);
        w[4 * c] = x.x; w[4 * c + 1] = x.y; w[4 * c + 2] = x.z; w[4 * c + 3] = x.w;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(w_empty(st));
      st += 2;
      if (st >= p.nw) { st -= p.nw; ph ^= 1u; }
      if (u > 0) {                                        // the products that read this buffer a unit ago
        wt_wait(done(b), (uint32_t)(u - 1) & 1u);
        tc_fence_after();
      }
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t o[32];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const uint32_t x = w[hf * 8 + c];
          o[4 * c] = wt_and_or(x >> (4 - kUp), mask, magic);
          o[4 * c + 1] = wt_and_or(x << kUp, mask, magic);
          o[4 * c + 2] = wt_and_or(x >> (12 - kUp), mask, magic);
          o[4 * c + 3] = wt_and_or(x >> (8 - kUp), mask, magic);
        }
        tmem_st_32x32(ta + hf * 32, o);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(a_full(b));
    }
  } else if (warp >= kWtSum) {
    // ================= sums, thread = (row, half of the tokens) =================
    constexpr int MH = MT / 2;
    const int q = warp & 3, row = q * p.rpw + lane, t0 = ((warp - kWtSum) >> 2) * MH;
    const int mh = p.M - t0;                              // tokens of this half
    const bool live = lane < p.rpw;
    constexpr float kBase = BF16 ? 16.f : 64.f;
    const uint32_t td = tmem + ((uint32_t)(q * 32) << 16) + 256 + t0;
    const uint32_t xs = sb + L.xs + (warp - kWtSum) * 256;
    int ss = 0;
    uint32_t sph = 0, u = 0;
    for (int t = 0; t < T; ++t) {
      float2 acc[MH / 2];
#pragma unroll
      for (int k = 0; k < MH / 2; ++k) acc[k] = make_float2(0.f, 0.f);
      for (int n = 0; n < nu; ++n, ++u) {
        wt_wait(s_full(ss), sph);
        float a[4], z[4] = {0.f, 0.f, 0.f, 0.f};
        {
          const uint32_t s = sb + L.sc + ss * kWtScale + row * 16;
          const uint4 v = wt_lds(s);
          a[0] = __uint_as_float(v.x); a[1] = __uint_as_float(v.y); a[2] = __uint_as_float(v.z); a[3] = __uint_as_float(v.w);
          if (p.has_zs) {
            const uint4 w = wt_lds(s + 2048);
            z[0] = __uint_as_float(w.x); z[1] = __uint_as_float(w.y); z[2] = __uint_as_float(w.z); z[3] = __uint_as_float(w.w);
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(s_empty(ss));
        if (++ss == kWtNS) { ss = 0; sph ^= 1u; }
#pragma unroll
        for (int j = 0; j < 2; ++j) {                     // a pair: two groups' sums
          wt_wait(done(j), u & 1u);
          tc_fence_after();
          constexpr int CH = 16;
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const float A = a[2 * j + k] * p.lin_a, C = -fmaf(A, kBase + p.lin_off, z[2 * j + k]) * (1.f / kBase);
            const float2 A2 = make_float2(A, A), C2 = make_float2(C, C);
#pragma unroll
            for (int c = 0; c < MH / CH; ++c) {
              uint32_t d[CH];
              const uint32_t from = td + j * (2 * MT) + k * MT + c * CH;
              tmem_ld_32x16(from, d);
              tmem_ld_wait();
              if (k == 1 && c == MH / CH - 1) {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(d_empty(j));
              }
              const uint32_t at = xs + k * 128 + c * (CH * 4);
              if (lane == 31) {
#pragma unroll
                for (int e = 0; e < CH; e += 4) wt_sts(at + e * 4, make_uint4(d[e], d[e + 1], d[e + 2], d[e + 3]));
              }
              __syncwarp();
#pragma unroll
              for (int e = 0; e < CH; e += 4) {
                const uint4 x = wt_lds(at + e * 4);
                float2& s0 = acc[(c * CH + e) / 2];
                float2& s1 = acc[(c * CH + e) / 2 + 1];
                s0 = __ffma2_rn(C2, make_float2(__uint_as_float(x.x), __uint_as_float(x.y)), s0);
                s1 = __ffma2_rn(C2, make_float2(__uint_as_float(x.z), __uint_as_float(x.w)), s1);
                s0 = __ffma2_rn(A2, make_float2(__uint_as_float(d[e]), __uint_as_float(d[e + 1])), s0);
                s1 = __ffma2_rn(A2, make_float2(__uint_as_float(d[e + 2]), __uint_as_float(d[e + 3])), s1);
              }
            }
          }
        }
      }
      const long long gr = (long long)(cl + t * ncl) * R + row;
      const bool store = live && gr < p.N;
      const float bias = !p.bias || !store ? 0.f : BF16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p.bias)[gr])
                                                       : __half2float(reinterpret_cast<const __half*>(p.bias)[gr]);
      if (S == 1) {
        if (store) {
#pragma unroll
          for (int i = 0; i < MH; ++i)
            if (i < mh) wt_store<BF16>(p, gr, t0 + i, bias, i & 1 ? acc[i / 2].y : acc[i / 2].x);
        }
      } else {
        // of every half's tokens [d MH / S, ..) are CTA d's to finish: [half][rank][token][row] there. Two buffers: whoever has announced its
        // part of tile t - 1 has finished tile t - 2, and all of them have when part_full of t - 1 was seen
        const int pl = (MH == 16 ? 4 : 5) - p.split_log2, per = 1 << pl, pb = t & 1;
        const uint32_t buf = sb + L.part + pb * p.part_bytes + (uint32_t)(t0 * 128 + q * 32 + lane) * 4u;
#pragma unroll
        for (int i = 0; i < MH; ++i) {
          if (i < mh) {
            const uint32_t at = buf + (uint32_t)((cr << pl) + (i & (per - 1))) * 512u;
            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(mapa_shared(at, (uint32_t)(i >> pl))),
                         "f"(i & 1 ? acc[i / 2].y : acc[i / 2].x) : "memory");
          }
        }
        asm volatile("fence.acq_rel.cluster;" ::: "memory");
        __syncwarp();
        if (lane < S)
          asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(mapa_shared(part_full(pb), (uint32_t)lane)) : "memory");
        wt_wait_cluster(part_full(pb), (uint32_t)(t >> 1) & 1u);
        if (store) {
#pragma unroll 4
          for (int tl = 0; tl < per; ++tl) {
            const int tok = (cr << pl) + tl;
            if (tok < mh) {
              float v[4];
#pragma unroll
              for (int w = 0; w < 4; ++w)
                if (w < S) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v[w]) : "r"(buf + (uint32_t)((w << pl) + tl) * 512u) : "memory");
              float s = v[0] + v[1];
              if (S == 4) s = (s + v[2]) + v[3];
              wt_store<BF16>(p, gr, t0 + tok, bias, s);
            }
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (S > 1) cluster_sync_all();                          // peers write to this CTA's shared memory until here
  if (warp == kWtMma) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

template <bool BF16, int MT>
static int wt_launch(const W4TcArgs& a, const W4TcCut& c, cudaStream_t st) {
  auto kern = w4_tc_kernel<BF16, MT>;
  CUtensorMap tw, ts, tz, tx;
  const uint32_t R = 4 * c.rpw;
  {
    uint64_t dims[2] = {(uint64_t)a.K / 2, (uint64_t)a.N}, str[1] = {(uint64_t)a.K / 2};
    uint32_t box[2] = {128, R};
    if (int rc = make_tensor_map(&tw, a.packed, 1, 2, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
    uint64_t sd[2] = {(uint64_t)a.K / 128, (uint64_t)a.N}, ss[1] = {(uint64_t)a.K / 128 * 4};
    uint32_t sbx[2] = {4, R};
    if (int rc = make_tensor_map(&ts, a.scale, 4, 2, sd, ss, sbx, CU_TENSOR_MAP_SWIZZLE_NONE)) return rc;
    tz = ts;
    if (a.zs)
      if (int rc = make_tensor_map(&tz, a.zs, 4, 2, sd, ss, sbx, CU_TENSOR_MAP_SWIZZLE_NONE)) return rc;
    {
      uint64_t xd[3] = {64, MT, (uint64_t)a.K / 64}, xs[2] = {128, 128 * MT};
      uint32_t xb[3] = {64, MT, 4};
      if (int rc = make_tensor_map(&tx, a.ws, 2, 3, xd, xs, xb, CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
    }
  }
  W4TcParams p = {};
  p.bias = a.bias; p.y = a.y; p.M = a.M; p.K = a.K; p.has_zs = a.zs ? 1 : 0;
  p.N = a.N; p.y_rs = a.y_rs; p.lin_a = a.lin_a; p.lin_off = a.lin_off; p.split_log2 = c.split_log2; p.rpw = c.rpw;
  p.nw = c.nw; p.part_bytes = c.split_log2 ? MT * 512 : 0;
  // per call: the attribute belongs to the current device, and a process may use several
  B200_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWtSmemMax));
  w4_tc_tokens_kernel<<<(a.K / 64 * MT * 8 + 255) / 256, 256, 0, st>>>((const uint16_t*)a.x, a.x_rs, a.M, a.K, MT == 32 ? 5 : 6, (uint4*)a.ws);
  B200_LAUNCH_CHECK();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(c.clusters << c.split_log2));
  cfg.blockDim = dim3(kWtThreads);
  cfg.dynamicSmemBytes = kWtSmemMax;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (c.split_log2 > 0) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = 1 << c.split_log2; attr[na].val.clusterDim.y = attr[na].val.clusterDim.z = 1;
    ++na;
  }
  attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // nothing but the tokens depends on the launch before
  attr[na].val.programmaticStreamSerializationAllowed = 1;
  ++na;
  cfg.attrs = attr;
  cfg.numAttrs = na;
  return (int)cudaLaunchKernelEx(&cfg, kern, tw, ts, tz, tx, p);
}

// Clusters of 1, 2 and 4 CTAs that are resident at once (a GPC has no multiple of four SMs); a device property, found once
static const int* wt_resident() {
  static const struct Resident {
    int n[3];
    Resident() {
      n[0] = kNumSMs;
      for (int i = 1; i < 3; ++i) {
        n[i] = 0;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = 1 << i; at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.gridDim = dim3(kNumSMs >> i << i); cfg.blockDim = dim3(kWtThreads); cfg.dynamicSmemBytes = kWtSmemMax;
        cfg.attrs = &at; cfg.numAttrs = 1;
        if (cudaFuncSetAttribute(w4_tc_kernel<true, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWtSmemMax) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&n[i], w4_tc_kernel<true, 32>, &cfg) != cudaSuccess) { n[i] = 0; (void)cudaGetLastError(); }
      }
    }
  } resident;
  return resident.n;
}

// The cut with the shortest time by what a unit (four groups) and the end of a tile take, us: 1.8 (up to 32 tokens) or 2.9, and 0.5, or 3.6
// where parts meet; a unit takes half as long again in clusters of four, whose CTAs wait for one another. From N 24576 and 34816 at K 4096
// and 5120, N 4096 at K 12288 and N 12288 at K 2048, each cut timed: N 24576, 64 tokens: 48 / 50 / 69 with 1 / 2 / 4 CTAs, N 4096: 64 / 38 / 42.
// It takes two CTAs for both: the shortest of the second, 2 us above the shortest of the first.
static W4TcCut w4_tc_cut(int M, long long N, int K, int group) {
  W4TcCut cut;
  if (M < 17 || M > 64 || N < 1 || N > (1 << 30) || K < 512 || K % 512 || group != 128) return cut;
  const int MT = M <= 32 ? 32 : 64, nun = K / 512;
  const int* res = wt_resident();
  double best = 0.;
  for (int i = 0; i < 3 && (1 << i) <= nun; ++i) {
    if (res[i] < 1) continue;
    const uint32_t rest = WtSmem(0, kWtNX * MT * 512, i ? MT * 512 : 0).bytes;
    const int um = (nun + (1 << i) - 1) >> i, nw = (int)((kWtSmemMax - rest) / kWtBox);
    const long long rounds = (N + (long long)res[i] * 124 - 1) / ((long long)res[i] * 124);
    const int rpw = (int)((N + rounds * res[i] * 4 - 1) / (rounds * res[i] * 4));
    const double cost = rounds * (um * (MT == 32 ? 1.8 : 2.9) * (i == 2 ? 1.5 : 1.) + (i ? 3.6 : 0.5));
    if (cut.split_log2 < 0 || cost < best) {
      best = cost;
      cut.split_log2 = i; cut.rpw = rpw; cut.nw = nw < kWtMaxW ? nw : kWtMaxW;
      const long long tiles = (N + 4 * rpw - 1) / (4 * rpw);
      cut.clusters = (int)(tiles < res[i] ? tiles : res[i]);
    }
  }
  return cut;
}

}  // namespace b200
using namespace b200;

// Arguments as in b200_w4_gemv_linear; `ws`: room for K x 32 (up to 32 tokens) or K x 64 16-bit values. B200_ERR_UNSUPPORTED: the caller
// takes that.
B200_API int b200_w4_tc_linear(const void* x, const uint8_t* packed, const float* scale, const float* zs, const void* bias, void* y, void* ws,
                               int M, long long N, int K, int group, long long x_rs, long long y_rs, float lin_a, float lin_off, int dtype,
                               void* stream) {
  if ((dtype != B200_DT_BF16 && dtype != B200_DT_FP16) || lin_off != (float)(int)lin_off || lin_off < -64.f || lin_off > 64.f || x_rs % 8 ||
      !ws || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(packed) | reinterpret_cast<uintptr_t>(scale) |
               reinterpret_cast<uintptr_t>(zs) | reinterpret_cast<uintptr_t>(ws)) & 15)) return B200_ERR_UNSUPPORTED;
  const W4TcCut cut = w4_tc_cut(M, N, K, group);
  if (cut.split_log2 < 0) return B200_ERR_UNSUPPORTED;
  const W4TcArgs a = {x, packed, scale, zs, bias, y, ws, M, K, N, x_rs, y_rs, lin_a, lin_off};
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == B200_DT_BF16) return M <= 32 ? wt_launch<true, 32>(a, cut, st) : wt_launch<true, 64>(a, cut, st);
  return M <= 32 ? wt_launch<false, 32>(a, cut, st) : wt_launch<false, 64>(a, cut, st);
}

// CTAs that share the k of a tile (1, 2, 4) where that call is taken, 0 where it is refused
B200_API int b200_w4_tc_split(int M, long long N, int K, int group) {
  const W4TcCut cut = w4_tc_cut(M, N, K, group);
  return cut.split_log2 < 0 ? 0 : 1 << cut.split_log2;
}
