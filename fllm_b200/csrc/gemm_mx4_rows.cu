// MXFP4 expert stacks x 16-bit activations on the block-scaled tensor cores, without expanding the codes:
//
//   y[row] = W[expert(row)] x[row] (+ bias),  W: e2m1 codes + one e8m0 scale per 32 values, x: bf16 rows, or fp32 values of a gated
//   epilogue
//
// tcgen05.mma kind::mxf8f6f4 multiplies e2m1 codes as they are and applies their scales, but its other operand has 8 bits. So a row is
// written as a sum of P rows of e4m3 with a scale per 32 values each: the first holds the value rounded to four significant bits, the next what
// is left of it, and so on. Two pieces hold the 8 bits of a bf16 value (exact down to 2^-12 of its block's largest, off by less than 2^-21 of that
// below), three 12 bits and a sign of a wider one, one more than fp16. (What this holds less than rows of fp16 with a factor each, which keep eight
// bits down to 2^-31 of a row's largest: small values beside a very large one in the same 32. Error of a layer of 2880 x 2880 x 3 against 64 bits, fp16 rows
// and this: 0.2365 %, 0.2355 % on normal rows; with every 640th value 30 to 3000 times as large the same or less, 3e4 times 0.2359, 0.2391 and 3e5 times 0.236,
// 0.516 where the weights of those values are zeros, 0.235 in both where they are not.) The pieces are further columns of the same product
// (accumulators of their own, added up in fp32 by the epilogue), so a tile of codes is read once for all of them, and a
// piece costs half of a bf16 product.
//
// What bounds it: 128 features x 128 values are 8.7 KB of HBM and 373 clocks at an SM's share of 6.5 TB/s; the product takes
// 64 + 32 per 16 tokens of two pieces, 190 at least, its operands 200 to 330 clocks of shared memory. The form that expands codes to fp16 on the
// ALUs (gemm_w4a16.cu) takes 735 for the same tile however few tokens there are. TMA spreads 16 codes over 16 bytes on the way to shared
// memory (16U4_ALIGN16B). What remains is the issue of the products: a wait costs the issuing lane 80 to 120 clocks even where the barrier has
// flipped. So up to 32 tokens a slot of the ring holds 256 values of K, codes and activations behind one barrier (416 clocks per 128 values; a slot
// of 128 with two waits: 620), and wide tiles, whose activations need the room, ask both barriers before they use either answer (510 to 610). One persistent
// CTA per SM; the epilogue of a tile runs beside the next one's products. 128 experts of 2880 x 2880 x 3, four of them per token, gate to down
// with routing, us per layer, expanded to fp16 -> this: 4 tokens 100 -> 78, 16: 225 -> 163, 121: 477 -> 334, 512: 504 -> 387, 1024: 544 -> 479, 2048: 674 -> 624.
//
// Tokens come in groups of 16: rows [group][piece][16] in the activation array, so that the tokens which a tile really has are its first
// 16 P (their number / 16) rows, and the product's width follows their number, not the tile's.
//
// Reference counterpart: rust/engine/cuda/mxfp4_moe.cu (grouped MXFP4 experts on expanded codes).
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include <algorithm>

#include "fllm_ops.h"
#include "ptx.cuh"
#include "tma_host.h"

namespace fllm {

constexpr int M4_BM = 128, M4_BK = 128, M4_G = 16, M4_ATOM = 512;

struct Mx4Maps {
  CUtensorMap codes, rows[3];        // boxes of 1, 2 and 4 groups of tokens
};

struct Mx4Args {
  int M, K;                          // output features of an expert, inputs
  int m_tiles, k_blocks;
  const uint8_t* sfa;                // [experts][m_tiles][k_blocks][512]
  const uint8_t* sfb;                // [tiles][k_blocks][atoms][512]
  const int *tile_expert, *tile_row0, *tile_rows, *num_tiles;
  const __nv_bfloat16* bias;         // [experts][M]
  __nv_bfloat16* out;                // [rows][ldc]; without a gated epilogue
  long long ldc;
  float alpha;
  // gated epilogue: clamped SwiGLU-OAI of (gate, up) pairs of neighbouring features, written as three pieces for the next product
  float glu_alpha, glu_limit;
  uint8_t* q_out;                    // [rows * 3][M / 2]
  uint8_t* sf_out;                   // [tiles][ceil(M / 256)][atoms of three pieces][512]
  int* status;
};

template <int BN, int P, bool GLU>
struct Mx4Smem {
  // Sets of four epilogue warps, which take the groups of tokens in turn: activation and splitting of one group take a set 3200 clocks, a tile's
  // products 9000 to 10000, and a tile of 80 tokens has five groups.
  static constexpr int kSets = GLU && BN > 32 ? 3 : 1;
  static constexpr int kThreads = (3 + 4 * kSets) * 32;         // codes, MMA, epilogue warps, activations
  static constexpr int kN = BN * P;                             // widest product
  static constexpr int kAtoms = (kN + 127) / 128;
  static constexpr bool kOne = BN <= 32;                        // activations lie in the slot of their codes; else they have a ring of single K blocks
  static constexpr int kABlock = M4_BM * M4_BK;                 // 8 KB of codes take 16
  static constexpr int kBBlock = kN * M4_BK;
  static constexpr int kBSf = kAtoms * M4_ATOM;
  static constexpr int kPer = kOne ? 2 : 1;                     // K blocks of a slot
  static constexpr int kSlot = kPer * (kABlock + M4_ATOM + (kOne ? kBBlock + kBSf : 0));
  static constexpr int kBStages = kOne ? 0 : 4;
  static constexpr int kStageOut = GLU ? kSets * 2 * M4_G * 72 * 4 : 4 * M4_G * 32 * 2;   // a set's two groups of 16 tokens x 64 activations (two blocks of 36 floats); bf16
  static constexpr int kRoom = 226 * 1024 - 1024 - 512 - kStageOut - kBStages * (kBBlock + kBSf);
  static constexpr int kStages = kRoom / kSlot;
  static constexpr int kBSlots = kOne ? 2 * kStages : kBStages; // blocks of activations in shared memory
  static constexpr int kASlots = kPer * kStages;                // and of codes
  static constexpr int kSfCols = 4 + 4 * kAtoms;                // tensor memory of a K block's scales, two of them
  static constexpr int kCols = 2 * kN + 2 * kSfCols;
  static constexpr int kTmemCols = kCols <= 128 ? 128 : kCols <= 256 ? 256 : 512;
  static constexpr int kTotal = 1024 + kASlots * (kABlock + M4_ATOM) + kBSlots * (kBBlock + kBSf) + kStageOut + 512;
  static_assert(kN <= 256 && kCols <= 512, "width of a product, tensor memory");
  static_assert(BN % M4_G == 0 && kBBlock % 1024 == 0, "groups of 16 tokens, swizzle atoms");
  static_assert((2 * kStages + 2 * kBStages + 4) * 8 + 8 <= 512, "barrier block");
  static_assert(kStages >= 3 && kTotal <= 227 * 1024, "shared memory of a CTA");
};

__device__ __forceinline__ uint64_t m4_sf_desc(uint32_t saddr) {   // one scale atom: K-major, no swizzle, 8-row groups 128 bytes apart
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (uint64_t)(128 >> 4) << 32 | (uint64_t)1 << 46;
}

__device__ __forceinline__ void m4_cp_sf(uint32_t tmem_dst, uint64_t sdesc) {
  asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(tmem_dst), "l"(sdesc) : "memory");
}

__device__ __forceinline__ void m4_mma(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t sfa, uint32_t sfb, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%5], [%6], p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb)
      : "memory");
}

__device__ __forceinline__ void m4_bulk_load(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(gsrc)), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

// 32 values, eight on each of four neighbouring lanes -> P pieces of e4m3, and a scale byte each (lanes agree). The scale of a piece is the smallest
// power of two that brings its largest magnitude to 448 or below. Magnitudes are compared as integers, so infinities and
// NaN win; their block's scale becomes the e8m0 NaN and the products of its row are not numbers.
template <int P>
__device__ __forceinline__ void split_e4m3(float (&v)[8], uint2 (&q)[P], uint32_t (&sf)[P]) {
#pragma unroll
  for (int p = 0; p < P; ++p) {
    uint32_t m = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) m = max(m, __float_as_uint(v[i]) & 0x7FFFFFFFu);
    m = max(m, __shfl_xor_sync(0xffffffffu, m, 1));
    m = max(m, __shfl_xor_sync(0xffffffffu, m, 2));
    const int ex = (int)(m >> 23);
    const int byte = max(ex - 8 + ((m & 0x7FFFFFu) > 0x600000u ? 1 : 0), 0);
    const float inv = __uint_as_float((uint32_t)(254 - byte) << 23);
    const float scale = __uint_as_float(byte == 0 ? 0x00400000u : (uint32_t)byte << 23);
    uint32_t w[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t two[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int at = 4 * h + 2 * i;
        const __nv_fp8x2_storage_t c = __nv_cvt_float2_to_fp8x2(make_float2(v[at] * inv, v[at + 1] * inv), __NV_SATFINITE, __NV_E4M3);
        two[i] = c;
        if (p + 1 < P) {                                         // what is left, exactly
          const float2 back = __half22float2(__half2(__nv_cvt_fp8x2_to_halfraw2(c, __NV_E4M3)));
          v[at] = fmaf(-back.x, scale, v[at]);
          v[at + 1] = fmaf(-back.y, scale, v[at + 1]);
        }
      }
      w[h] = two[0] | two[1] << 16;
    }
    q[p] = make_uint2(w[0], w[1]);
    sf[p] = ex == 255 ? 255u : (uint32_t)byte;
  }
}

template <int BN, int P, bool GLU>
__global__ void __launch_bounds__(Mx4Smem<BN, P, GLU>::kThreads, 1)
gemm_mx4_rows_kernel(const __grid_constant__ Mx4Maps maps, const Mx4Args p) {
  using S = Mx4Smem<BN, P, GLU>;
  constexpr int AST = S::kStages, BST = S::kBStages;
  constexpr bool ONE = S::kOne;
  constexpr int PER = S::kPer;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sA = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sB = sA + S::kASlots * S::kABlock;
  uint8_t* sFA = sB + S::kBSlots * S::kBBlock;
  uint8_t* sFB = sFA + S::kASlots * M4_ATOM;
  uint8_t* sOut = sFB + S::kBSlots * S::kBSf;
  uint64_t* afull_bar = reinterpret_cast<uint64_t*>(sOut + S::kStageOut);
  uint64_t* aempty_bar = afull_bar + AST;
  uint64_t* bfull_bar = aempty_bar + AST;
  uint64_t* bempty_bar = bfull_bar + BST;
  uint64_t* tfull_bar = bempty_bar + BST;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = uniform_warp(), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < AST; ++s) { mbar_init(&afull_bar[s], 1); mbar_init(&aempty_bar[s], 1); }
    for (int s = 0; s < BST; ++s) { mbar_init(&bfull_bar[s], 1); mbar_init(&bempty_bar[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&tfull_bar[s], 1); mbar_init(&tempty_bar[s], 4 * S::kSets); }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 0 && lane == 0) { tma_prefetch_desc(&maps.codes); tma_prefetch_desc(&maps.rows[0]); tma_prefetch_desc(&maps.rows[1]); tma_prefetch_desc(&maps.rows[2]); }
  if (warp == 1) { tmem_alloc(tmem_slot, S::kTmemCols); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();
  pdl_wait();                                           // tile list and rows come from the predecessors
  const int total = *p.num_tiles * p.m_tiles;
  auto groups_of = [&](int tile) { return (min(__ldcg(p.tile_rows + tile), BN) + M4_G - 1) / M4_G; };

  // activations of one K block in boxes of 4, 2 and 1 groups of tokens (a box per group was bounded by their issue; values beyond K read as zero),
  // and their scales
  auto load_rows = [&](int block, uint64_t* bar, int kb, int groups, int rows0, const uint8_t* sf, uint32_t sf_bytes) {
    constexpr int GROUP = M4_G * P;
    uint8_t* b = sB + block * S::kBBlock;
    if (BN >= 64 && (groups & 4)) tma_load_2d(b, &maps.rows[2], bar, kb * M4_BK, rows0);
    const int g2 = groups & 4, g1 = groups & 6;
    if (BN >= 32 && (groups & 2)) tma_load_2d(b + g2 * GROUP * M4_BK, &maps.rows[1], bar, kb * M4_BK, rows0 + g2 * GROUP);
    if (groups & 1) tma_load_2d(b + g1 * GROUP * M4_BK, &maps.rows[0], bar, kb * M4_BK, rows0 + g1 * GROUP);
    m4_bulk_load(sFB + block * S::kBSf, sf + (size_t)kb * S::kBSf, sf_bytes, bar);
  };

  if (warp == 0) {
    // ------------------------------------------------ codes and their scales (narrow tiles: activations, too), two K blocks a slot
    int st = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int w = blockIdx.x; w < total && ok; w += gridDim.x) {
      const int tile = w / p.m_tiles, m_idx = w - tile * p.m_tiles;
      const int expert = __ldcg(p.tile_expert + tile);
      const uint8_t* sf = p.sfa + (size_t)(expert * p.m_tiles + m_idx) * p.k_blocks * M4_ATOM;
      const int row0 = expert * p.M + m_idx * M4_BM;
      int groups = 0, rows0 = 0;
      uint32_t sf_bytes = 0, b_bytes = 0;
      const uint8_t* sfb = nullptr;
      if (ONE) {
        groups = groups_of(tile); rows0 = __ldcg(p.tile_row0 + tile) * P;
        sf_bytes = (groups * M4_G * P + 127) / 128 * M4_ATOM;
        b_bytes = groups * M4_G * P * M4_BK + sf_bytes;
        sfb = p.sfb + (size_t)(rows0 / (BN * P)) * p.k_blocks * S::kBSf;
      }
      for (int kb = 0; kb < p.k_blocks; kb += PER) {
        if (!mbar_wait_warp(&aempty_bar[st], phase ^ 1, abort_flag)) { ok = false; break; }
        if (elect_one()) {
          const bool two = PER == 2 && kb + 1 < p.k_blocks;
          uint8_t* a = sA + st * PER * S::kABlock;
          mbar_expect_tx(&afull_bar[st], (two ? 2 : 1) * (S::kABlock / 2 + M4_ATOM + b_bytes));      // packed codes are counted as they leave global memory
          tma_load_2d(a, &maps.codes, &afull_bar[st], kb * M4_BK, row0);
          if (two) tma_load_2d(a + S::kABlock, &maps.codes, &afull_bar[st], (kb + 1) * M4_BK, row0);
          m4_bulk_load(sFA + st * PER * M4_ATOM, sf + (size_t)kb * M4_ATOM, (two ? 2 : 1) * M4_ATOM, &afull_bar[st]);
          if (ONE) {
            load_rows(2 * st, &afull_bar[st], kb, groups, rows0, sfb, sf_bytes);
            if (two) load_rows(2 * st + 1, &afull_bar[st], kb + 1, groups, rows0, sfb, sf_bytes);
          }
        }
        __syncwarp();
        if (++st == AST) { st = 0; phase ^= 1; }
      }
    }
  } else if (warp == 2 + 4 * S::kSets) {
    // ------------------------------------------------ activations of wide tiles
    int st = 0;
    uint32_t phase = 0;
    bool ok = !ONE;
    for (int w = blockIdx.x; w < total && ok; w += gridDim.x) {
      const int tile = w / p.m_tiles;
      const int groups = groups_of(tile), rows0 = __ldcg(p.tile_row0 + tile) * P;
      const uint32_t sf_bytes = (groups * M4_G * P + 127) / 128 * M4_ATOM;
      const uint8_t* sf = p.sfb + (size_t)(rows0 / (BN * P)) * p.k_blocks * S::kBSf;
      for (int kb = 0; kb < p.k_blocks; ++kb) {
        if (!mbar_wait_warp(&bempty_bar[st], phase ^ 1, abort_flag)) { ok = false; break; }
        if (elect_one()) {
          mbar_expect_tx(&bfull_bar[st], groups * M4_G * P * M4_BK + sf_bytes);
          load_rows(st, &bfull_bar[st], kb, groups, rows0, sf, sf_bytes);
        }
        __syncwarp();
        if (++st == BST) { st = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    // e2m1 (format 5) x e4m3 (0), e8m0 scales, fp32 accumulators; the width is set per tile. One lane runs the role: with a region of one elected
    // lane and a vote per slot, leaving and entering it cost 300 clocks each time.
    constexpr uint32_t idesc0 = 5u << 7 | 1u << 23 | (uint32_t)(M4_BM >> 4) << 24;
    const uint64_t da0 = make_smem_desc_sw128(smem_u32(sA)), db0 = make_smem_desc_sw128(smem_u32(sB));
    const uint64_t fa0 = m4_sf_desc(smem_u32(sFA)), fb0 = m4_sf_desc(smem_u32(sFB));
    const uint32_t tmem_sf = tmem_base + 2 * S::kN;
    int as = 0, bs = 0, acc = 0;
    uint32_t aphase = 0, bphase = 0, accphase = 0;
    bool ok = elect_one();
    for (int w = blockIdx.x; w < total && ok; w += gridDim.x) {
      const int n = groups_of(w / p.m_tiles) * M4_G * P;
      const uint32_t idesc = idesc0 | (uint32_t)(n >> 3) << 17;
      if (!mbar_wait(&tempty_bar[acc], accphase ^ 1, abort_flag)) break;
      const uint32_t td = tmem_base + acc * S::kN;
      auto block = [&](int ablk, int bblk, int j, uint32_t first) {
        const uint32_t sfa = tmem_sf + j * S::kSfCols, sfb = sfa + 4;
        m4_cp_sf(sfa, fa0 + (uint64_t)(ablk * (M4_ATOM >> 4)));
        m4_cp_sf(sfb, fb0 + (uint64_t)(bblk * (S::kBSf >> 4)));
        if (S::kAtoms > 1 && n > 128) m4_cp_sf(sfb + 4, fb0 + (uint64_t)(bblk * (S::kBSf >> 4) + (M4_ATOM >> 4)));
        const uint64_t da = da0 + (uint64_t)(ablk * (S::kABlock >> 4)), db = db0 + (uint64_t)(bblk * (S::kBBlock >> 4));
#pragma unroll
        for (int k = 0; k < 4; ++k)
          m4_mma(td, da + 2 * k, db + 2 * k, idesc | (uint32_t)k << 29 | (uint32_t)k << 4, sfa, sfb, k > 0 ? 1u : first);
      };
      for (int kb = 0; kb < p.k_blocks; kb += PER) {
        const bool two = PER == 2 && kb + 1 < p.k_blocks, last = kb + PER >= p.k_blocks;
        if (ONE) {
          if (!mbar_wait(&afull_bar[as], aphase, abort_flag)) { ok = false; break; }
        } else {                                          // both asked before either answer is used: 80 clocks each
          const bool a_in = mbar_try_wait(&afull_bar[as], aphase), b_in = mbar_try_wait(&bfull_bar[bs], bphase);
          if (!(a_in || mbar_wait(&afull_bar[as], aphase, abort_flag)) || !(b_in || mbar_wait(&bfull_bar[bs], bphase, abort_flag))) { ok = false; break; }
        }
        tc_fence_after_sync();
        block(PER * as, ONE ? 2 * as : bs, ONE ? 0 : kb & 1, kb > 0 ? 1u : 0u);
        if (two) block(2 * as + 1, 2 * as + 1, 1, 1u);
        tc_commit(&aempty_bar[as]);
        if (!ONE) tc_commit(&bempty_bar[bs]);
        if (last) tc_commit(&tfull_bar[acc]);
        if (!ONE && ++bs == BST) { bs = 0; bphase ^= 1; }
        if (++as == AST) { as = 0; aphase ^= 1; }
      }
      acc ^= 1;
      if (acc == 0) accphase ^= 1;
    }
    __syncwarp();
  } else {
    // ------------------------------------------------ epilogue: sets of four warps, one per TMEM lane quarter
    const int q = warp & 3, set = (warp - 2) >> 2, etid = threadIdx.x - 64 - set * 128;
    const uint32_t t_lane = tmem_base + ((uint32_t)(q * 32) << 16);
    int acc = 0, turn = 0;
    uint32_t accphase = 0;
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
      const int tile = w / p.m_tiles, m_idx = w - tile * p.m_tiles;
      const int groups = groups_of(tile), row0 = __ldcg(p.tile_row0 + tile);
      const int m = m_idx * M4_BM + q * 32 + lane;
      const float bias_m = (p.bias && m < p.M) ? __bfloat162float(p.bias[(size_t)__ldcg(p.tile_expert + tile) * p.M + m]) : 0.f;
      bool ok = mbar_wait(&tfull_bar[acc], accphase, abort_flag);
      if constexpr (GLU) {                                   // the four warps meet below: they go on, or leave, together
        int all;
        asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbarrier.red.and.pred q, %2, 128, p;\n\tselp.b32 %0, 1, 0, q;\n\t}"
                     : "=r"(all) : "r"((int)ok), "r"(1 + set) : "memory");
        ok = all != 0;
      }
      if (!ok) break;
      tc_fence_after_sync();
#pragma unroll 1
      for (int g = set; g < groups; g += S::kSets) {
        float v[M4_G];
        {
          uint32_t r[P][M4_G];
#pragma unroll
          for (int i = 0; i < P; ++i) tmem_ld_32x16(t_lane + acc * S::kN + (g * P + i) * M4_G, r[i]);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < M4_G; ++c) {                   // the smallest pieces first
            float s = __uint_as_float(r[P - 1][c]);
#pragma unroll
            for (int i = P - 2; i >= 0; --i) s += __uint_as_float(r[i][c]);
            v[c] = s * p.alpha + bias_m;
          }
        }
        if (g + S::kSets >= groups) {                        // the accumulators are in registers
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&tempty_bar[acc]);
        }
        if constexpr (GLU) {
          // even lanes hold gate features, odd lanes their up features: neighbours trade one value per pair of columns, so that each
          // computes the activation of one of the two
          float* stg = reinterpret_cast<float*>(sOut) + (2 * set + (turn & 1)) * M4_G * 72;
          ++turn;
          const bool hi = lane & 1;
          const int at = (q >> 1) * 36 + (q & 1) * 16 + (lane >> 1);
#pragma unroll
          for (int c = 0; c < M4_G; c += 2) {
            const float recv = __shfl_xor_sync(0xffffffffu, hi ? v[c] : v[c + 1], 1);
            const float gate = fminf(hi ? recv : v[c], p.glu_limit);
            const float up = fminf(fmaxf(hi ? v[c + 1] : recv, -p.glu_limit), p.glu_limit);
            stg[(c + (hi ? 1 : 0)) * 72 + at] = __fdividef(gate, 1.f + __expf(-p.glu_alpha * gate)) * (up + 1.f);
          }
          asm volatile("bar.sync %0, 128;" ::"r"(1 + set) : "memory");    // (the other half of sOut is written next: one barrier per group is enough)
          // 16 tokens x 2 blocks of 32 activations, four lanes each
          const int t = etid >> 3, blk = (etid >> 2) & 1, part = etid & 3;
          const float4 lo = *reinterpret_cast<const float4*>(stg + t * 72 + blk * 36 + part * 8);
          const float4 hi4 = *reinterpret_cast<const float4*>(stg + t * 72 + blk * 36 + part * 8 + 4);
          float a[8] = {lo.x, lo.y, lo.z, lo.w, hi4.x, hi4.y, hi4.z, hi4.w};
          constexpr int PO = 3, ATOMS = (BN * PO + 127) / 128;
          uint2 qv[PO];
          uint32_t sf[PO];
          split_e4m3<PO>(a, qv, sf);
          const int half = p.M / 2, kb = m_idx >> 1, j = (m_idx & 1) * 2 + blk;      // (half is a multiple of 64)
          // a K block that ends in the middle: its last two scales, of values that do not exist, must be numbers
          const bool pad = (m_idx & 1) == 0 && m_idx + 1 == p.m_tiles;
#pragma unroll
          for (int i = 0; i < PO; ++i) {
            const int r = (g * PO + i) * M4_G + t;           // row within the tile
            *reinterpret_cast<uint2*>(p.q_out + ((size_t)row0 * PO + r) * half + m_idx * 64 + blk * 32 + part * 8) = qv[i];
            if (part == 0) {
              uint8_t* atom = p.sf_out + (((size_t)(row0 / BN) * ((half + 127) / 128) + kb) * ATOMS + (r >> 7)) * M4_ATOM + (r & 31) * 16 + ((r >> 5) & 3) * 4;
              atom[j] = (uint8_t)sf[i];
              if (pad) atom[j + 2] = 127;
            }
          }
        } else {
          __nv_bfloat16* stg = reinterpret_cast<__nv_bfloat16*>(sOut) + q * (M4_G * 32);
#pragma unroll
          for (int c = 0; c < M4_G; ++c) stg[c * 32 + lane] = __float2bfloat16(v[c]);
          __syncwarp();
          const int f0 = 8 * (lane & 3), mm0 = m_idx * M4_BM + q * 32 + f0;
#pragma unroll
          for (int rnd = 0; rnd < M4_G / 8; ++rnd) {
            const int c = (lane >> 2) + 8 * rnd;
            if (mm0 < p.M)
              *reinterpret_cast<uint4*>(p.out + (size_t)(row0 + g * M4_G + c) * p.ldc + mm0) = *reinterpret_cast<const uint4*>(stg + c * 32 + f0);
          }
          __syncwarp();
        }
      }
      if (S::kSets > 1 && set >= groups && lane == 0) mbar_arrive(&tempty_bar[acc]);      // nothing to read for this set
      acc ^= 1;
      if (acc == 0) accphase ^= 1;
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) { tc_fence_after_sync(); tmem_dealloc(tmem_base, S::kTmemCols); }
  if (threadIdx.x == 0 && *abort_flag && p.status) atomicCAS(p.status, FLLM_OK, FLLM_ERR_MBAR_TIMEOUT);
}

// Rows of bf16 -> two pieces of e4m3 and their scale atoms, in the order of gemm_mx4_rows_kernel: row r of a tile of bn tokens goes to rows
// (r / 16) 32 + r % 16 and + 16 of the tile. One CTA per row, half a warp per 128 values. token_of (optional): rows without a token (-1) become
// zeros, groups of 16 without any are left out. placed: x has the rows of the tiles already (an activation between the products). row_weight
// (optional): routers that weigh an expert's input (rounded to bf16, as there).
__global__ void __launch_bounds__(192) rows_mx_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, const int* __restrict__ token_of, int placed,
                                                      const float* __restrict__ row_weight, uint8_t* __restrict__ xq, uint8_t* __restrict__ sf, int K, int bn) {
  pdl_launch_dependents();
  pdl_wait();
  const int row = blockIdx.x;
  int t = row;
  if (token_of != nullptr) {
    if (token_of[row & ~(M4_G - 1)] < 0) return;              // tokens fill a tile from its start
    t = token_of[row];
    if (placed && t >= 0) t = row;
  }
  const float rw = row_weight != nullptr && t >= 0 ? row_weight[row] : 1.f;
  const int tile = row / bn, in = row - tile * bn, r0 = (in / M4_G) * (2 * M4_G) + (in % M4_G), atoms = (2 * bn + 127) / 128;
  const int kbs = (K + 127) / 128, l = threadIdx.x & 15;
  for (int kb0 = 0; kb0 < kbs; kb0 += 12) {                   // whole warps: the shuffles need both halves
    const int kb = kb0 + (threadIdx.x >> 4), k = kb * 128 + l * 8;
    uint4 raw = make_uint4(0, 0, 0, 0);
    if (t >= 0 && k < K) raw = *reinterpret_cast<const uint4*>(x + (size_t)t * ldx + k);
    const uint32_t u[4] = {raw.x, raw.y, raw.z, raw.w};
    float v[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 f = unpack_bf16x2(u[i]);
      if (row_weight != nullptr) f = unpack_bf16x2(pack_bf16x2(f.x * rw, f.y * rw));
      v[2 * i] = f.x;
      v[2 * i + 1] = f.y;
    }
    uint2 q[2];
    uint32_t s[2];
    split_e4m3<2>(v, q, s);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      uint32_t word = s[i] << (8 * (l >> 2));                 // four scales of 32 values
      word |= __shfl_xor_sync(0xffffffffu, word, 4);
      word |= __shfl_xor_sync(0xffffffffu, word, 8);
      const int r = r0 + i * M4_G;
      if (kb < kbs && k < K) *reinterpret_cast<uint2*>(xq + ((size_t)tile * bn * 2 + r) * K + k) = q[i];
      if (kb < kbs && l == 0)
        *reinterpret_cast<uint32_t*>(sf + (((size_t)tile * kbs + kb) * atoms + (r >> 7)) * M4_ATOM + (r & 31) * 16 + ((r >> 5) & 3) * 4) = word;
    }
  }
}

void rows_mx(const void* x, long long ldx, const int* token_of, bool placed, const float* row_weight, void* xq, void* sf, int rows, int K, int bn,
             cudaStream_t s) {
  if (rows <= 0) return;
  if ((K & 63) || (ldx & 7) || (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(xq) & 15) || (reinterpret_cast<uintptr_t>(sf) & 15))
    throw std::runtime_error("rows_mx: K % 64 and 16-byte rows required");
  if (bn % M4_G || rows % bn) throw std::runtime_error("rows_mx: whole tiles of a multiple of 16 rows");
  launch_pdl(rows_mx_kernel, dim3(rows), dim3(192), 0, s, (const __nv_bfloat16*)x, ldx, token_of, placed ? 1 : 0, row_weight, (uint8_t*)xq, (uint8_t*)sf, K, bn);
}

template <int BN, int P, bool GLU>
static void launch_mx4(const Mx4Maps& maps, const Mx4Args& a, int items, cudaStream_t s) {
  using S = Mx4Smem<BN, P, GLU>;
  static bool configured[kMaxDevices] = {};
  if (first_call_on_device(configured))
    cuda_check(cudaFuncSetAttribute(gemm_mx4_rows_kernel<BN, P, GLU>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kTotal),
               "cudaFuncSetAttribute(gemm_mx4_rows_kernel)");
  launch_pdl(gemm_mx4_rows_kernel<BN, P, GLU>, dim3(std::min(items, sm_count())), dim3(S::kThreads), S::kTotal, s, maps, a);
}

template <int BN>
static void launch_mx4_form(int pieces, bool glu, const Mx4Maps& maps, const Mx4Args& a, int items, cudaStream_t s) {
  if (pieces == 3) launch_mx4<BN, 3, false>(maps, a, items, s);
  else if (glu) launch_mx4<BN, 2, true>(maps, a, items, s);
  else launch_mx4<BN, 2, false>(maps, a, items, s);
}

// Bytes of the scale atoms of `rows` rows of K values in tiles of bn tokens.
size_t mx4_scale_bytes(int rows, int K, int bn, int pieces) {
  return (size_t)(rows / bn) * ((K + 127) / 128) * ((bn * pieces + 127) / 128) * M4_ATOM;
}

int moe_grouped_linear_mx4(const Mx4Rows& x, const void* codes, const void* sfa, int experts, int n_out, int K, float alpha, const void* bias, void* y,
                           long long ldy, const Mx4Glu* glu, const Mx4Tiles& tiles, int* status, cudaStream_t stream) {
  if (x.rows <= 0 || tiles.max_tiles <= 0) return 0;
  const int bn = tiles.bn;
  if (bn != 16 && bn != 32 && bn != 80) throw std::runtime_error("moe_grouped_linear_mx4: tiles of 16, 32 or 80 tokens");
  if (x.rows % bn || K % 64 || n_out % 8) throw std::runtime_error("moe_grouped_linear_mx4: whole tiles, K % 64 and N % 8 required");
  if (x.pieces != 2 && (x.pieces != 3 || glu)) throw std::runtime_error("moe_grouped_linear_mx4: two pieces, or three without an activation");
  if ((reinterpret_cast<uintptr_t>(codes) & 31) || (reinterpret_cast<uintptr_t>(sfa) & 15) || (reinterpret_cast<uintptr_t>(x.sf) & 15))
    throw std::runtime_error("moe_grouped_linear_mx4: codes must be 32-byte, scales 16-byte aligned");
  Mx4Args a{};
  a.M = n_out; a.K = K; a.m_tiles = (n_out + M4_BM - 1) / M4_BM; a.k_blocks = (K + M4_BK - 1) / M4_BK;
  a.sfa = (const uint8_t*)sfa; a.sfb = (const uint8_t*)x.sf;
  a.tile_expert = tiles.expert; a.tile_row0 = tiles.row0; a.tile_rows = tiles.rows; a.num_tiles = tiles.count;
  a.bias = (const __nv_bfloat16*)bias; a.alpha = alpha; a.status = status;
  if (glu != nullptr) {
    if (n_out % 128) throw std::runtime_error("moe_grouped_linear_mx4: a gated epilogue needs N % 128 == 0");
    a.glu_alpha = glu->alpha; a.glu_limit = glu->limit; a.q_out = (uint8_t*)glu->q; a.sf_out = (uint8_t*)glu->sf;
  } else {
    if ((ldy & 7) || (reinterpret_cast<uintptr_t>(y) & 15)) throw std::runtime_error("moe_grouped_linear_mx4: 16-byte output rows required");
    a.out = (__nv_bfloat16*)y; a.ldc = ldy;
  }
  // The map's rows are whole blocks of 128 codes: where K ends in the middle of one, the second half of the last block is the next row's first codes (or
  // up to 32 bytes behind the stack, which its owner provides), which meet zeros in the activations.
  Mx4Maps maps;
  maps.codes = make_tmap_2d(codes, CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B, 1, (uint64_t)experts * n_out, (uint64_t)a.k_blocks * M4_BK, K / 2, M4_BM, M4_BK,
                            true);
  for (int i = 0; i < 3; ++i)
    maps.rows[i] = make_tmap_2d(x.q, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)x.rows * x.pieces, K, K, (M4_G * x.pieces) << i, M4_BK, true);
  const int items = tiles.max_tiles * a.m_tiles;
  if (bn == 16) launch_mx4_form<16>(x.pieces, glu != nullptr, maps, a, items, stream);
  else if (bn == 32) launch_mx4_form<32>(x.pieces, glu != nullptr, maps, a, items, stream);
  else launch_mx4_form<80>(x.pieces, glu != nullptr, maps, a, items, stream);
  return 1;
}

}  // namespace fllm
