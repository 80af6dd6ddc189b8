// Packed 4-bit weights x 16-bit activations on tcgen05 (weights stay packed in HBM):
//
//   NVFP4   e2m1 codes, two per byte, + one e4m3 scale per 16 values + an fp32 tensor scale
//   MXFP4   e2m1 codes, two per byte, + one e8m0 (power of two) scale per 32 values
//   INT4G   unsigned 4-bit codes + one (scale, min) pair of bf16 per 32 values: value = q * scale - min.
//           This is the device form of GGUF Q4_K / Q4_0 / Q4_1 and of AWQ / GPTQ int4 groups, re-laid at
//           load time (planar codes, nibbles ordered so that two shifts-and-masks yield K-ordered pairs).
//
// Decode is bound by the bytes of weight read, so reading 4.5 bit/weight instead of 16 is the
// point. The kernel is the swap-AB GEMM of gemm_bf16.cu with one extra stage in the operand path:
// TMA brings the raw code tile (128 features x 128 bytes) into shared memory, groups of four warps expand it
// into tensor memory, publish it with an mbarrier, and the single issuing thread runs tcgen05.mma kind::f16 with
// A from there. Four further warps run the epilogue of one tile while the next is expanded; one persistent CTA per SM.
//
// What bounds it: at 6.5 TB/s an SM receives 46 codes per clock, so the expansion may cost 128 lanes x 1 / 46 = 2.8
// instructions per value and everything else that the expanding warps do must fit into the same. The fp16 form takes one:
// a conversion instruction yields two fp16 values of two codes and one multiplication applies their block scale. e2m1 times
// e4m3 (6 significant bits, 2^-10 .. 2688) and e2m1 times e8m0 within [104, 140] are exact in fp16; activations come as fp16
// rows times a power of two per row (rows_f16_kernel: exact, too), which the epilogue multiplies back in. The bf16 form
// (byte permutes through register tables, 2.75 instructions per value) is for INT4G, for block scales outside that range
// and for callers without converted rows.
//
// Reference counterparts: rust/engine/cuda/nvfp4.cu:132-307 (mma.sync mxf4nvf4, GeForce Blackwell
// only), rust/engine/cuda/marlin_vllm (W4A16 Marlin, the sm_100 default), MXFP4 through the
// IQ4_NL look-up path (rust/engine/cuda/common.cuh:154).
#include <cuda_fp8.h>

#include <algorithm>

#include "fllm_ops.h"
#include "ptx.cuh"
#include "tma_host.h"

namespace fllm {

constexpr int W4_BM = 128;
constexpr int W4_BK = 64;             // values per step = one 128-byte swizzled row of 16-bit activations

struct W4Args {
  int M, N, K;                        // M = output features, N = tokens
  int m_tiles, k_blocks;
  int k_splits, kb_per_split;         // splits of the K loop; partial sums go to `ws`
  float* ws;                          // [k_splits][N][M] fp32 when k_splits > 1
  int fmt;                            // 0 NVFP4 (e4m3 / 16), 1 MXFP4 (e8m0 / 32), 2 INT4G ((scale, min) bf16 / 32)
  int f16;                            // activations and expanded weights are fp16 (fmt 0 and 1)
  long long ldc;
  uint16_t* out;                      // bf16 (fp16 with a gated epilogue)
  const uint8_t* scales;              // [M][K/16] bytes, [M][K/32] bytes, or [M][K/32] x {bf16 scale, bf16 min}
  const float* row_factor;            // per activation row, multiplied back in (null: 1)
  float alpha;                        // tensor scale (NVFP4), 1 otherwise
  const __nv_bfloat16* bias;
  int* status;
  int glu;                            // 1: clamped SwiGLU-OAI over (gate, up) pairs of neighbouring features, stored as fp16 times glu_scale
  float glu_alpha, glu_limit, glu_scale;
  // grouped (mixture of experts): items walk a device-built tile list; tile i multiplies rows
  // [row0, row0 + BN) of the permuted activations with expert e's matrix (codes / scales / bias stacked
  // over experts, g_rows output features each)
  const int* g_tile_expert;
  const int* g_tile_row0;
  const int* g_num_tiles;
  int g_rows;
};

template <int BN>
struct W4Smem {
  // The unit of every ring is a slot of 256 values of K: 128-byte rows of codes (narrower rows waste HBM bursts) and four
  // 128-byte rows of activations per token; 96 - 128 KB of codes in flight. The expanded operand never touches
  // shared memory: the expanding warps store it into tensor memory (128 columns per slot) and the MMA reads A from there.
  static constexpr int kThreads = 64 + 16 * 32 + 4 * 32 + 32;  // codes, MMA, four groups of four expanding warps, four epilogue warps, activations
  static constexpr int kRawBytes = W4_BM * 128;
  static constexpr int kBStep = BN * W4_BK * 2;                // activations of one 64-value step
  static constexpr int kBBytes = 4 * kBStep;
  static constexpr int kRStages = BN == 128 ? 4 : BN == 96 ? 5 : BN == 64 ? 6 : 8;
  static constexpr int kBStages = BN >= 96 ? 2 : BN == 64 ? 3 : BN == 32 ? 4 : 6;
  // tensor memory: two accumulators, then kAStages slots of expanded weights
  static constexpr int kDCols = BN < 32 ? 32 : BN;
  static constexpr int kTmemCols = 512;
  static constexpr int kAStages = (kTmemCols - 2 * kDCols) / 128;
  static constexpr int kBarBytes = 512;
  static constexpr int kLutBytes = 1024;                       // scale byte -> pair of 16-bit values
  static constexpr int kStageOutBytes = 4 * 32 * 32 * 2;       // per-epilogue-warp transpose tile
  static constexpr int kTotal = kRStages * kRawBytes + kBStages * kBBytes + kBarBytes + kLutBytes + kStageOutBytes + 1024;
  static_assert(kAStages >= 2, "one slot in the MMA, one being expanded");
  static_assert((2 * kRStages + 2 * kBStages + 2 * kAStages + 4) * 8 + 8 <= kBarBytes, "barrier block");
  static_assert(kTotal <= 226 * 1024, "shared memory of a CTA");
};

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}

// 8 e2m1 codes (one 32-bit word, low nibble first) -> 8 bf16, scaled by `s2` (bf16x2 of the block scale).
// Four codes per step: two byte-permutes look the high and low bf16 bytes up in 8-entry tables held in
// registers (selector = the codes' three magnitude bits), a sign-replicating permute spreads the four sign
// bits, two more permutes interleave the bytes into bf16 pairs: about 2.75 instructions per value.
__device__ __forceinline__ void e2m1x8_to_bf16(uint32_t codes, uint32_t s2, uint32_t (&out)[4]) {
  // bf16 of {0, .5, 1, 1.5, 2, 3, 4, 6}: high bytes 00 3F 3F 3F 40 40 40 40, low bytes 00 00 80 C0 00 40 80 C0
  constexpr uint32_t HI_LO = 0x3F3F3F00u, HI_HI = 0x40404040u, LO_LO = 0xC0800000u, LO_HI = 0xC0804000u;
  const __nv_bfloat162 sc = *reinterpret_cast<const __nv_bfloat162*>(&s2);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t w = codes >> (16 * h);                          // selectors read the low 16 bits only
    const uint32_t sel = w & 0x7777u;
    uint32_t hi4 = prmt(HI_LO, HI_HI, sel);
    const uint32_t lo4 = prmt(LO_LO, LO_HI, sel);
    const uint32_t sg = prmt(w, w << 4, 0x9D8Cu);                  // byte i = 0xFF where code i is negative
    hi4 |= sg & 0x80808080u;
    uint32_t v0 = prmt(lo4, hi4, 0x5140u);                         // [lo0, hi0, lo1, hi1]
    uint32_t v1 = prmt(lo4, hi4, 0x7362u);                         // [lo2, hi2, lo3, hi3]
    __nv_bfloat162 r0 = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&v0), sc);
    __nv_bfloat162 r1 = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&v1), sc);
    out[2 * h] = *reinterpret_cast<uint32_t*>(&r0);
    out[2 * h + 1] = *reinterpret_cast<uint32_t*>(&r1);
  }
}

// The same codes -> 8 fp16: one conversion and one multiplication per pair.
__device__ __forceinline__ void e2m1x8_to_f16(uint32_t codes, uint32_t s2, uint32_t (&out)[4]) {
  asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
      "mov.b32 {b0, b1, b2, b3}, %4;\n\t"
      "cvt.rn.f16x2.e2m1x2 %0, b0;\n\t"
      "cvt.rn.f16x2.e2m1x2 %1, b1;\n\t"
      "cvt.rn.f16x2.e2m1x2 %2, b2;\n\t"
      "cvt.rn.f16x2.e2m1x2 %3, b3;\n\t}"
      : "=r"(out[0]), "=r"(out[1]), "=r"(out[2]), "=r"(out[3]) : "r"(codes));
  const __half2 sc = *reinterpret_cast<const __half2*>(&s2);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __half2 r = __hmul2(*reinterpret_cast<const __half2*>(&out[i]), sc);
    out[i] = *reinterpret_cast<const uint32_t*>(&r);
  }
}

// 8 unsigned 4-bit codes -> 8 bf16 of q * s - m. Storage order: nibble j of the word holds value 2j (j < 4)
// or 2(j - 4) + 1, so ((w >> 4j) & 0x000F000F) is the K-ordered pair (2j, 2j + 1). OR-ing 0x4300 makes the
// bf16 number 128 + q exactly; one subtract and one fused multiply-add finish it.
__device__ __forceinline__ void int4x8_to_bf16(uint32_t w, uint32_t s2, uint32_t negm2, uint32_t (&out)[4]) {
  const __nv_bfloat162 sc = *reinterpret_cast<const __nv_bfloat162*>(&s2);
  const __nv_bfloat162 nm = *reinterpret_cast<const __nv_bfloat162*>(&negm2);
  const uint32_t c128 = 0x43004300u;
  const __nv_bfloat162 b128 = *reinterpret_cast<const __nv_bfloat162*>(&c128);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint32_t t = ((w >> (4 * j)) & 0x000F000Fu) | c128;
    const __nv_bfloat162 q = __hsub2(*reinterpret_cast<__nv_bfloat162*>(&t), b128);
    const __nv_bfloat162 r = __hfma2(q, sc, nm);
    out[j] = *reinterpret_cast<const uint32_t*>(&r);
  }
}

__device__ __forceinline__ float scale_to_float(uint8_t s, int fmt) {
  if (fmt == 0) {
    __nv_fp8_e4m3 v;
    v.__x = s;
    return static_cast<float>(v);
  }
  return __uint_as_float((uint32_t)s << 23);                       // e8m0: 2^(s - 127); s = 0 -> 0 (denormal floor)
}

// One unit of work: a feature tile of a split of K, or of a tile of the list.
struct W4Item {
  int m_idx, split, kb0, nkb, expert, row0;
};

__device__ __forceinline__ W4Item w4_item(const W4Args& p, int w) {
  W4Item it;
  const int outer = w / p.m_tiles;
  it.m_idx = w - outer * p.m_tiles;
  if (p.g_tile_expert != nullptr) {
    it.split = 0; it.kb0 = 0; it.nkb = p.k_blocks;
    it.expert = __ldcg(p.g_tile_expert + outer);
    it.row0 = __ldcg(p.g_tile_row0 + outer);
  } else {
    it.split = outer;
    it.kb0 = outer * p.kb_per_split;                    // multiple of 4: code slots start on 256 values
    it.nkb = min(p.k_blocks, it.kb0 + p.kb_per_split) - it.kb0;
    it.expert = 0; it.row0 = 0;
  }
  return it;
}

// F16: activations and expanded weights are fp16 (formats 0 and 1). A template parameter: tested at every word of codes, the branches
// were a tenth of the expanding warps' time.
template <int BN, bool F16>
__global__ void __launch_bounds__(W4Smem<BN>::kThreads, 1)
gemm_w4a16_kernel(const __grid_constant__ CUtensorMap tma_raw, const __grid_constant__ CUtensorMap tma_b, const W4Args p) {
  using S = W4Smem<BN>;
  constexpr int RST = S::kRStages, BST = S::kBStages, AST = S::kAStages;
  extern __shared__ uint8_t smem_raw_[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw_) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sR = smem;                                   // code slots, 16 KB each (128-byte swizzled rows)
  uint8_t* sB = sR + RST * S::kRawBytes;                // activations, four steps of BN x 128 B each
  uint64_t* bars = reinterpret_cast<uint64_t*>(sB + BST * S::kBBytes);
  uint64_t* rfull_bar = bars;                           // codes landed
  uint64_t* rempty_bar = rfull_bar + RST;               // every expanding warp is done with the slot
  uint64_t* bfull_bar = rempty_bar + RST;               // activations landed
  uint64_t* bempty_bar = bfull_bar + BST;               // MMA retired
  uint64_t* ready_bar = bempty_bar + BST;               // expanded operand stored to tensor memory (16 warps)
  uint64_t* aempty_bar = ready_bar + AST;               // its columns consumed by the MMA
  uint64_t* tfull_bar = aempty_bar + AST;               // accumulator complete
  uint64_t* tempty_bar = tfull_bar + 2;                 // accumulator read by the epilogue (4 warps)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint32_t* lut = reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(bars) + S::kBarBytes);
  uint16_t* stage_out = reinterpret_cast<uint16_t*>(lut + S::kLutBytes / 4);
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const bool grouped = p.g_tile_expert != nullptr;

  if (threadIdx.x == 0) {
    for (int s = 0; s < RST; ++s) { mbar_init(&rfull_bar[s], 1); mbar_init(&rempty_bar[s], 16); }
    for (int s = 0; s < BST; ++s) { mbar_init(&bfull_bar[s], 1); mbar_init(&bempty_bar[s], 1); }
    for (int s = 0; s < AST; ++s) { mbar_init(&ready_bar[s], 16); mbar_init(&aempty_bar[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&tfull_bar[s], 1); mbar_init(&tempty_bar[s], 4); }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (threadIdx.x >= 64 && threadIdx.x < 64 + 256 && !(F16 && p.fmt == 0)) {    // scale byte -> {s, s} (fp16 NVFP4 converts its scales)
    const int i = threadIdx.x - 64;
    const float f = scale_to_float((uint8_t)i, p.fmt);
    const __half2 h = __floats2half2_rn(f, f);
    lut[i] = F16 ? *reinterpret_cast<const uint32_t*>(&h) : pack_bf16x2(f, f);
  }
  if (warp == 0 && lane == 0) { tma_prefetch_desc(&tma_raw); tma_prefetch_desc(&tma_b); }
  if (warp == 1) { tmem_alloc(tmem_slot, S::kTmemCols); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();
  if (grouped) pdl_wait();                              // the tile list comes from the predecessor
  const int total = grouped ? *p.g_num_tiles * p.m_tiles : p.m_tiles * p.k_splits;

  if (warp == 0) {
    // ------------------------------------------------ codes: static, so without a list they do not even wait for the predecessor
    int rs = 0;
    uint32_t rphase = 0;
    bool ok = true;
    for (int w = blockIdx.x; w < total && ok; w += gridDim.x) {
      const W4Item it = w4_item(p, w);
      const int code_row0 = it.expert * p.g_rows + it.m_idx * W4_BM;
      for (int kb = 0; kb < it.nkb; kb += 4) {
        if (!mbar_wait_warp(&rempty_bar[rs], rphase ^ 1, abort_flag)) { ok = false; break; }
        if (elect_one()) {
          mbar_expect_tx(&rfull_bar[rs], S::kRawBytes);
          tma_load_2d(sR + rs * S::kRawBytes, &tma_raw, &rfull_bar[rs], (it.kb0 + kb) * 32, code_row0);
        }
        __syncwarp();
        if (++rs == RST) { rs = 0; rphase ^= 1; }
      }
    }
  } else if (warp == 22) {
    // ------------------------------------------------ activations: four steps in one box (steps beyond K read as zero)
    if (!grouped) pdl_wait();
    int bs = 0;
    uint32_t bphase = 0;
    bool ok = true;
    for (int w = blockIdx.x; w < total && ok; w += gridDim.x) {
      const W4Item it = w4_item(p, w);
      for (int kb = 0; kb < it.nkb; kb += 4) {
        if (!mbar_wait_warp(&bempty_bar[bs], bphase ^ 1, abort_flag)) { ok = false; break; }
        if (elect_one()) {
          mbar_expect_tx(&bfull_bar[bs], S::kBBytes);
          tma_load_3d(sB + bs * S::kBBytes, &tma_b, &bfull_bar[bs], 0, it.row0, it.kb0 + kb);
        }
        __syncwarp();
        if (++bs == BST) { bs = 0; bphase ^= 1; }
      }
    }
  } else if (warp == 1) {
    const uint32_t idesc = F16 ? make_idesc(W4_BM, BN, 0, 0) : make_idesc(W4_BM, BN, 1, 1);
    const uint64_t db0 = make_smem_desc_sw128(smem_u32(sB));
    int bs = 0, as = 0, acc = 0;
    uint32_t bphase = 0, aphase = 0, accphase = 0;
    bool ok = true;
    for (int w = blockIdx.x; w < total && ok; w += gridDim.x) {
      const int split = w / p.m_tiles;
      const int nkb = grouped ? p.k_blocks : min(p.k_blocks, (split + 1) * p.kb_per_split) - split * p.kb_per_split;
      if (!mbar_wait_warp(&tempty_bar[acc], accphase ^ 1, abort_flag)) break;
      tc_fence_after_sync();
      const uint32_t td = tmem_base + acc * S::kDCols;
      for (int kb = 0; kb < nkb; kb += 4) {
        if (!mbar_wait_warp(&bfull_bar[bs], bphase, abort_flag) || !mbar_wait_warp(&ready_bar[as], aphase, abort_flag)) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t ta = tmem_base + 2 * S::kDCols + as * 128;
        const uint64_t db = db0 + (uint64_t)(bs * (S::kBBytes >> 4));
        const int steps = min(4, nkb - kb);
        if (elect_one()) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (i < steps) {
#pragma unroll
              for (int k = 0; k < W4_BK / 16; ++k)
                tc_mma_bf16_ts(td, ta + 32 * i + 8 * k, db + i * (S::kBStep >> 4) + 2 * k, idesc, (kb > 0 || i > 0 || k > 0) ? 1u : 0u);
            }
          }
          tc_commit(&bempty_bar[bs]);
          tc_commit(&aempty_bar[as]);
          if (kb + 4 >= nkb) tc_commit(&tfull_bar[acc]);
        }
        __syncwarp();
        if (++bs == BST) { bs = 0; bphase ^= 1; }
        if (++as == AST) { as = 0; aphase ^= 1; }
      }
      acc ^= 1;
      if (acc == 0) accphase ^= 1;
    }
  } else if (warp < 2 + 16) {
    // ------------------------------------------------ expand codes into tensor memory
    // Group g expands step g of every slot. Every thread owns one row (= TMEM lane).
    const int q = warp & 3;                             // TMEM lane quarter this warp may touch
    const int g = (warp - 2) >> 2;
    const int row = q * 32 + lane;
    const uint32_t t_lane = tmem_base + ((uint32_t)(q * 32) << 16) + 2 * S::kDCols + g * 32;
    const int sbytes = p.fmt == 0 ? 4 : p.fmt == 1 ? 2 : 8;   // scale bytes per row per step
    auto scale_row = [&](const W4Item& it) {
      const int m_row = it.expert * p.g_rows + min(it.m_idx * W4_BM + row, p.M - 1);
      return p.scales + ((size_t)m_row * (p.K / 64) + it.kb0) * sbytes;
    };
    auto load_scales = [&](const uint8_t* srow, int kb, int nkb) -> uint2 {           // this row's scales of step kb
      if (kb >= nkb) return make_uint2(0, 0);
      if (p.fmt == 0) return make_uint2(__ldg(reinterpret_cast<const uint32_t*>(srow + kb * 4)), 0);
      if (p.fmt == 1) return make_uint2((uint32_t)__ldg(reinterpret_cast<const uint16_t*>(srow + kb * 2)), 0);
      return __ldg(reinterpret_cast<const uint2*>(srow + kb * 8));
    };
    int rs = 0, as = 0;
    uint32_t rphase = 0, aphase = 0;
    bool ok = true;
    if ((int)blockIdx.x < total) {
      W4Item it = w4_item(p, blockIdx.x);
      const uint8_t* srow = scale_row(it);
      uint2 sc = load_scales(srow, g, it.nkb);          // one slot ahead, over the end of an item, too
      for (int w = blockIdx.x; w < total && ok; w += gridDim.x) {
        const int nkb = it.nkb;
        const bool more = w + (int)gridDim.x < total;
        if (more) it = w4_item(p, w + gridDim.x);
        const uint8_t* srow_next = scale_row(it);
        for (int kb = g; kb - g < nkb; kb += 4) {
          const uint32_t sraw = sc.x, sraw2 = sc.y;
          if (kb - g + 4 < nkb) sc = load_scales(srow, kb + 4, nkb);
          else if (more) sc = load_scales(srow_next, g, it.nkb);
          uint32_t s2[4];
          if (p.fmt == 0 && F16) {                        // four e4m3 scales: two conversions, no table
            uint32_t h01, h23;
            asm("{\n\t.reg .b16 a, b;\n\tmov.b32 {a, b}, %2;\n\tcvt.rn.f16x2.e4m3x2 %0, a;\n\tcvt.rn.f16x2.e4m3x2 %1, b;\n\t}" : "=r"(h01), "=r"(h23) : "r"(sraw));
            s2[0] = __byte_perm(h01, 0, 0x1010);
            s2[1] = __byte_perm(h01, 0, 0x3232);
            s2[2] = __byte_perm(h23, 0, 0x1010);
            s2[3] = __byte_perm(h23, 0, 0x3232);
          } else if (p.fmt == 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i) s2[i] = lut[(sraw >> (8 * i)) & 0xFF];
          } else if (p.fmt == 1) {
            s2[0] = s2[1] = lut[sraw & 0xFF];
            s2[2] = s2[3] = lut[(sraw >> 8) & 0xFF];
          } else {                                          // {scale, min} bf16 of the two 32-value groups
            s2[0] = __byte_perm(sraw, 0, 0x1010);           // (s, s)
            s2[1] = __byte_perm(sraw, 0, 0x3232) ^ 0x80008000u;   // (-m, -m)
            s2[2] = __byte_perm(sraw2, 0, 0x1010);
            s2[3] = __byte_perm(sraw2, 0, 0x3232) ^ 0x80008000u;
          }
          if (!mbar_wait(&rfull_bar[rs], rphase, abort_flag)) { ok = false; break; }
          const uint8_t* rrow = sR + rs * S::kRawBytes + row * 128;
          const uint4 r0 = *reinterpret_cast<const uint4*>(rrow + (((2 * g) ^ (row & 7)) << 4));
          const uint4 r1 = *reinterpret_cast<const uint4*>(rrow + (((2 * g + 1) ^ (row & 7)) << 4));
          if (!mbar_wait(&aempty_bar[as], aphase ^ 1, abort_flag)) { ok = false; break; }
          tc_fence_after_sync();
          if (kb < nkb) {
            const uint32_t words[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              uint32_t o[16];
#pragma unroll
              for (int c = 0; c < 4; ++c) {                 // 8 codes -> 4 cells of two values each
                uint32_t o4[4];
                if (F16) e2m1x8_to_f16(words[4 * h + c], s2[2 * h + (c >> 1)], o4);
                else if (p.fmt == 2) int4x8_to_bf16(words[4 * h + c], s2[2 * h], s2[2 * h + 1], o4);
                else e2m1x8_to_bf16(words[4 * h + c], s2[2 * h + (c >> 1)], o4);
#pragma unroll
                for (int i = 0; i < 4; ++i) o[4 * c + i] = o4[i];
              }
              tmem_st_32x16(t_lane + as * 128 + 16 * h, o);
            }
            tmem_st_wait();
          }
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) {                                  // one arrival per warp, with or without a step in the slot
            mbar_arrive(&ready_bar[as]);
            mbar_arrive(&rempty_bar[rs]);
          }
          if (++rs == RST) { rs = 0; rphase ^= 1; }
          if (++as == AST) { as = 0; aphase ^= 1; }
        }
        srow = srow_next;
      }
    }
  } else {
    // ------------------------------------------------ epilogue: four warps, one per TMEM lane quarter
    const int q = warp & 3;
    if (!grouped) pdl_wait();                           // outputs and partial sums may still be in use by the predecessor
    constexpr int CH = BN < 32 ? 16 : 32;
    const uint32_t t_lane = tmem_base + ((uint32_t)(q * 32) << 16);
    uint16_t* stg = stage_out + (warp - 18) * (32 * 32);
    int acc = 0;
    uint32_t accphase = 0;
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
      const W4Item it = w4_item(p, w);
      const int m = it.m_idx * W4_BM + q * 32 + lane;
      const float bias_m = (p.bias && m < p.M) ? __bfloat162float(p.bias[(size_t)it.expert * p.g_rows + m]) : 0.f;
      if (!mbar_wait(&tfull_bar[acc], accphase, abort_flag)) break;
      tc_fence_after_sync();
#pragma unroll 1
      for (int c0 = 0; c0 < BN; c0 += CH) {
        float v[CH];
        {
          uint32_t r[CH];
          if constexpr (CH == 32) tmem_ld_32x32(t_lane + acc * S::kDCols + c0, r);
          else tmem_ld_32x16(t_lane + acc * S::kDCols + c0, r);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < CH; ++c) v[c] = __uint_as_float(r[c]);
        }
        const int n0 = it.row0 + c0;
        if (p.row_factor != nullptr) {                  // one load per lane, handed round
          const float f = lane < CH && n0 + lane < p.N ? __ldcg(p.row_factor + n0 + lane) : 0.f;
#pragma unroll
          for (int c = 0; c < CH; ++c) v[c] *= __shfl_sync(0xffffffffu, f, c);
        }
        if (p.k_splits > 1) {                           // fp32 partial sums, lanes along features: coalesced
          float* wsp = p.ws + (size_t)it.split * p.N * p.M;
#pragma unroll
          for (int c = 0; c < CH; ++c)
            if (c0 + c < p.N && m < p.M) wsp[(size_t)(c0 + c) * p.M + m] = v[c];
          continue;
        }
        if (p.glu) {
          // even lanes hold gate features, odd lanes their up features: neighbours trade one value per pair of columns, so that
          // each computes the activation of one of the two; the warp's 16 output features of a row leave as 16-byte stores
          const bool hi = lane & 1;
#pragma unroll
          for (int c = 0; c < CH; c += 2) {
            const float a0 = v[c] * p.alpha + bias_m, a1 = v[c + 1] * p.alpha + bias_m;
            const float recv = __shfl_xor_sync(0xffffffffu, hi ? a0 : a1, 1);
            const float gate = fminf(hi ? recv : a0, p.glu_limit);
            const float up = fminf(fmaxf(hi ? a1 : recv, -p.glu_limit), p.glu_limit);
            const __half r = __float2half_rn(__fdividef(gate, 1.f + __expf(-p.glu_alpha * gate)) * (up + 1.f) * p.glu_scale);
            stg[(c + (hi ? 1 : 0)) * 16 + (lane >> 1)] = __half_as_ushort(r);
          }
          __syncwarp();
          const int f0 = 8 * (lane & 1), fo = (it.m_idx * W4_BM + q * 32) / 2 + f0;
#pragma unroll
          for (int rnd = 0; rnd < CH / 16; ++rnd) {
            const int c = (lane >> 1) + 16 * rnd, n = n0 + c;
            if (n < p.N && 2 * fo < p.M)
              *reinterpret_cast<uint4*>(p.out + (size_t)n * p.ldc + fo) = *reinterpret_cast<const uint4*>(stg + c * 16 + f0);
          }
          __syncwarp();
          continue;
        }
#pragma unroll
        for (int c = 0; c < CH; ++c) stg[c * 32 + lane] = __bfloat16_as_ushort(__float2bfloat16(v[c] * p.alpha + bias_m));
        __syncwarp();
        const int f0 = 8 * (lane & 3);
        const int mm0 = it.m_idx * W4_BM + q * 32 + f0;
#pragma unroll
        for (int rnd = 0; rnd < CH / 8; ++rnd) {
          const int c = (lane >> 2) + 8 * rnd;
          const int n = n0 + c;
          if (n < p.N && mm0 < p.M)
            *reinterpret_cast<uint4*>(p.out + (size_t)n * p.ldc + mm0) = *reinterpret_cast<const uint4*>(stg + c * 32 + f0);
        }
        __syncwarp();
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty_bar[acc]);
      acc ^= 1;
      if (acc == 0) accphase ^= 1;
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) { tc_fence_after_sync(); tmem_dealloc(tmem_base, S::kTmemCols); }
  if (threadIdx.x == 0 && *abort_flag && p.status) atomicCAS(p.status, FLLM_OK, FLLM_ERR_MBAR_TIMEOUT);
}

// Rows of bf16 -> fp16 times a power of two per row, and that power's inverse: out[r] = x[token_of[r]] 2^-e, factor[r] = 2^e, with the
// row's largest finite value in [2^14, 2^15). bf16 has fewer significant bits than fp16, so every value down to 2^-31 of the
// largest is exact. Rows without a token (-1) become zeros. row_weight (optional): routers that weigh an expert's input.
__global__ void __launch_bounds__(128) rows_f16_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, const int* __restrict__ token_of,
                                                       const float* __restrict__ row_weight, __half* __restrict__ out, float* __restrict__ factor, int K) {
  __shared__ uint32_t top[4];
  pdl_launch_dependents();
  pdl_wait();
  const int row = blockIdx.x;
  const int t = token_of != nullptr ? token_of[row] : row;
  uint4* dst = reinterpret_cast<uint4*>(out + (size_t)row * K);
  if (t < 0) {
    for (int i = threadIdx.x; i < K / 8; i += 128) dst[i] = make_uint4(0, 0, 0, 0);
    if (threadIdx.x == 0) factor[row] = 1.f;
    return;
  }
  const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)t * ldx);
  const float rw = row_weight != nullptr ? row_weight[row] : 1.f;
  auto get = [&](int i) {
    uint4 v = src[i];
    if (row_weight != nullptr) {                        // rounded to bf16, as the bf16 path stores it
      uint32_t* u = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
      for (int j = 0; j < 4; ++j) { const float2 f = unpack_bf16x2(u[j]); u[j] = pack_bf16x2(f.x * rw, f.y * rw); }
    }
    return v;
  };
  uint32_t m = 0;                                       // largest magnitude bits of the finite values
  for (int i = threadIdx.x; i < K / 8; i += 128) {
    const uint4 v = get(i);
    const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t lo = u[j] & 0x7FFFu, hi = (u[j] >> 16) & 0x7FFFu;
      if (lo < 0x7F80u) m = max(m, lo);
      if (hi < 0x7F80u) m = max(m, hi);
    }
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) top[threadIdx.x >> 5] = m;
  __syncthreads();
  m = max(max(top[0], top[1]), max(top[2], top[3]));
  const int e = m == 0 ? 0 : min(max((int)(m >> 7) - 127 - 14, -112), 113);      // both powers are normal fp32 numbers
  const float f = __uint_as_float((uint32_t)(127 - e) << 23);
  if (threadIdx.x == 0) factor[row] = __uint_as_float((uint32_t)(127 + e) << 23);
  for (int i = threadIdx.x; i < K / 8; i += 128) {
    const uint4 v = get(i);
    const uint32_t u[4] = {v.x, v.y, v.z, v.w};
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 a = unpack_bf16x2(u[j]);
      const __half2 h = __floats2half2_rn(a.x * f, a.y * f);
      o[j] = *reinterpret_cast<const uint32_t*>(&h);
    }
    dst[i] = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

void rows_f16(const void* x, long long ldx, const int* token_of, const float* row_weight, void* out, float* factor, int rows, int K, cudaStream_t s) {
  if (rows <= 0) return;
  if ((K & 7) || (ldx & 7) || (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(out) & 15))
    throw std::runtime_error("rows_f16: 16-byte rows required");
  launch_pdl(rows_f16_kernel, dim3(rows), dim3(128), 0, s, (const __nv_bfloat16*)x, ldx, token_of, row_weight, (__half*)out, factor, K);
}

// out[n][m] = bf16(alpha * sum_s ws[s][n][m] + bias[m])
template <int B>
__global__ void w4_splitk_reduce_kernel(const float* __restrict__ ws, int splits, int rows, int cols, long long ldc,
                                        float alpha, const __nv_bfloat16* __restrict__ bias, __nv_bfloat16* __restrict__ out) {
  pdl_launch_dependents();
  pdl_wait();
  const size_t n = (size_t)rows * cols;
  const size_t i4 = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (i4 >= n) return;
  const float4 acc = sum_splits4<B>(ws + i4, n, splits);
  const int r = row_of_element(i4, cols);
  const int c = (int)(i4 - (size_t)r * cols);
  float b[4] = {0.f, 0.f, 0.f, 0.f};
  if (bias) for (int i = 0; i < 4; ++i) b[i] = __bfloat162float(bias[c + i]);
  uint2 o;
  o.x = pack_bf16x2(acc.x * alpha + b[0], acc.y * alpha + b[1]);
  o.y = pack_bf16x2(acc.z * alpha + b[2], acc.w * alpha + b[3]);
  *reinterpret_cast<uint2*>(out + (size_t)r * ldc + c) = o;
}

// Expand packed weights to bf16 [M][K] (prefill path: expand once, then the dense GEMM).
__global__ void w4_dequant_kernel(const uint8_t* __restrict__ codes, const uint8_t* __restrict__ scales, int fmt,
                                  float alpha, __nv_bfloat16* __restrict__ out, long long n_groups8, int K) {
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;      // one thread = 8 values
  if (g >= n_groups8) return;
  const long long e0 = g * 8;
  const long long row = e0 / K;
  const int k = (int)(e0 - row * K);
  const uint32_t w = reinterpret_cast<const uint32_t*>(codes)[g];
  if (fmt == 2) {
    const uint32_t sm = reinterpret_cast<const uint32_t*>(scales)[row * (K / 32) + k / 32];
    uint32_t o[4];
    int4x8_to_bf16(w, __byte_perm(sm, 0, 0x1010), __byte_perm(sm, 0, 0x3232) ^ 0x80008000u, o);
    *reinterpret_cast<uint4*>(out + e0) = make_uint4(o[0], o[1], o[2], o[3]);
    return;
  }
  const int bs = fmt == 0 ? 16 : 32;
  const float sf = scale_to_float(scales[row * (K / bs) + k / bs], fmt) * alpha;
  uint32_t o[4];
  e2m1x8_to_bf16(w, pack_bf16x2(1.f, 1.f), o);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = unpack_bf16x2(o[i]);
    o[i] = pack_bf16x2(f.x * sf, f.y * sf);
  }
  *reinterpret_cast<uint4*>(out + e0) = make_uint4(o[0], o[1], o[2], o[3]);
}

void w4_dequant_bf16(const void* codes, const void* scales, int fmt, float alpha, void* out, long long rows, int K,
                     cudaStream_t s) {
  const long long groups = rows * K / 8;
  if (groups <= 0) return;
  w4_dequant_kernel<<<(unsigned)((groups + 255) / 256), 256, 0, s>>>((const uint8_t*)codes, (const uint8_t*)scales, fmt,
                                                                     alpha, (__nv_bfloat16*)out, groups, K);
  cuda_check(cudaGetLastError(), "w4_dequant_kernel");
}

template <int BN, bool F16>
static void launch_w4_form(const CUtensorMap& tr, const CUtensorMap& tb, const W4Args& a, int items, cudaStream_t s) {
  using S = W4Smem<BN>;
  static bool configured[kMaxDevices] = {};
  if (first_call_on_device(configured)) {
    cuda_check(cudaFuncSetAttribute(gemm_w4a16_kernel<BN, F16>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kTotal),
               "cudaFuncSetAttribute(gemm_w4a16_kernel)");
    cuda_check(cudaFuncSetAttribute(gemm_w4a16_kernel<BN, F16>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                    cudaSharedmemCarveoutMaxShared), "cudaFuncSetAttribute(carveout)");
  }
  launch_pdl(gemm_w4a16_kernel<BN, F16>, dim3(std::min(items, sm_count())), dim3(S::kThreads), S::kTotal, s, tr, tb, a);
}

template <int BN>
static void launch_w4(const CUtensorMap& tr, const CUtensorMap& tb, const W4Args& a, int items, cudaStream_t s) {
  if (a.f16) launch_w4_form<BN, true>(tr, tb, a, items, s);
  else launch_w4_form<BN, false>(tr, tb, a, items, s);
}

static void launch_w4_bn(int bn, const CUtensorMap& tr, const CUtensorMap& tb, const W4Args& a, int items, cudaStream_t s) {
  switch (bn) {
    case 16: launch_w4<16>(tr, tb, a, items, s); break;
    case 32: launch_w4<32>(tr, tb, a, items, s); break;
    case 64: launch_w4<64>(tr, tb, a, items, s); break;
    case 96: launch_w4<96>(tr, tb, a, items, s); break;
    default: launch_w4<128>(tr, tb, a, items, s); break;
  }
}

static int w4_token_tile(int T) { return T <= 16 ? 16 : T <= 32 ? 32 : T <= 64 ? 64 : T <= 96 ? 96 : 128; }

// fp16 rows and their factors at the end of the workspace: [.. partial sums ..][fp16 rows][row factors]
static size_t w4_rows_bytes(int T, int K) { return ((size_t)T * K * 2 + (size_t)T * 4 + 255) & ~(size_t)255; }

// Form and splits over K of a dense product. One CTA per SM streams whole items, so the time goes by the rounds of items over the SMs. In
// units of 10 ns, fitted to 72 products of 1024 .. 57344 features, K of 1024 .. 28672 and 8 .. 128 tokens (what is chosen is 0.6 % behind the best
// in the mean, 6 % at most): a slot of 256 values of K takes 68 to 88 by the token tile in the fp16 form, 99 to 107 in the bf16 form; an
// item 21 to 301 more until its sums have left; partial sums a kernel of 134, 48 a split, and their bytes at 12.7 TB/s; the conversion of the
// rows 141 and 2 per 10000 values. (By rounds alone 64 x 24576 x 4096 was cut in eight: 52 us for 31. The conversion of 128 rows of
// 1024 took 3 of 12 us.)
W4Plan w4_plan(int T, int N, int K, int sms, bool f16, size_t workspace_bytes) {
  const int bn = w4_token_tile(T);
  const size_t rows_bytes = w4_rows_bytes(T, K) + 256;
  if (workspace_bytes < rows_bytes) f16 = false;
  const int m_tiles = (N + W4_BM - 1) / W4_BM, slots = (K / W4_BK + 3) / 4, tile = bn == 16 ? 0 : bn == 32 ? 1 : bn == 64 ? 2 : bn == 96 ? 3 : 4;
  W4Plan best{1, false};
  long long least = -1;
  for (int form = 0; form <= (f16 ? 1 : 0); ++form) {
    for (int s = 1; s <= std::min(8, slots); ++s) {
      if (s > 1 && (size_t)s * T * N * 4 > workspace_bytes - (form ? rows_bytes : 0)) break;
      const int per = (slots + s - 1) / s, parts = (slots + per - 1) / per;
      const long long rounds = ((long long)m_tiles * parts + sms - 1) / sms;
      const long long cost = rounds * (per * (form ? 68 + 5 * tile : 99 + 2 * tile) + 21 + 70 * tile) + (form ? 141 + (long long)T * K / 5000 : 0) +
                             (parts > 1 ? 134 + 48 * parts + (long long)((double)parts * T * N * 8 / 127000.0) : 0);
      if (least < 0 || cost < least) { least = cost; best = W4Plan{s, form == 1}; }
    }
  }
  return best;
}

// y[T][N] = x[T][K] * dequant(codes, scales)^T * alpha (+ bias); T <= 128. f16: the block scales of the format allow the fp16 form
// (NVFP4 always; MXFP4 with scales of 104 .. 140, or 0), which the plan takes where it is faster: the rows are then converted into the end of
// the workspace first.
int linear_w4a16(const void* x, long long ldx, const void* codes, const void* scales, int fmt, float alpha,
                 const void* bias, void* y, long long ldy, int T, int N, int K, void* workspace, size_t workspace_bytes,
                 int* status, cudaStream_t stream, bool f16) {
  if (T <= 0 || N <= 0) return 0;
  if (T > 128) throw std::runtime_error("linear_w4a16: at most 128 tokens per call (expand the weight for prefill)");
  if (K % 64 || N % 8 || (ldx & 7) || (ldy & 7)) throw std::runtime_error("linear_w4a16: K % 64, N % 8 and 16-byte rows required");
  if (fmt < 0 || fmt > 2) throw std::runtime_error("linear_w4a16: fmt must be 0 (NVFP4), 1 (MXFP4) or 2 (INT4G)");
  W4Args a{};
  a.M = N; a.N = T; a.K = K; a.m_tiles = (N + W4_BM - 1) / W4_BM; a.k_blocks = K / W4_BK; a.fmt = fmt;
  a.ldc = ldy; a.out = reinterpret_cast<uint16_t*>(y); a.scales = reinterpret_cast<const uint8_t*>(scales);
  a.alpha = alpha; a.bias = reinterpret_cast<const __nv_bfloat16*>(bias); a.status = status;
  const int bn = w4_token_tile(T);
  const size_t rows_bytes = w4_rows_bytes(T, K);
  const W4Plan plan = w4_plan(T, N, K, sm_count(), f16 && fmt != 2, workspace ? workspace_bytes : 0);
  const int splits = plan.splits;
  a.f16 = plan.f16;
  int launches = 1;
  if (a.f16) {
    uint8_t* end = reinterpret_cast<uint8_t*>(reinterpret_cast<uintptr_t>(workspace) + workspace_bytes & ~(uintptr_t)255);
    uint8_t* xh = end - rows_bytes;
    float* factor = reinterpret_cast<float*>(xh + (size_t)T * K * 2);
    rows_f16(x, ldx, nullptr, nullptr, xh, factor, T, K, stream);
    x = xh; ldx = K; a.row_factor = factor;
    workspace_bytes -= rows_bytes + 256;
    ++launches;
  }
  a.kb_per_split = ((a.k_blocks + splits - 1) / splits + 3) & ~3;      // code slots cover four K steps
  a.k_splits = (a.k_blocks + a.kb_per_split - 1) / a.kb_per_split;
  a.ws = reinterpret_cast<float*>(workspace);
  CUtensorMap tr = make_tmap_2d(codes, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, N, K / 2, K / 2, W4_BM, 128, true);
  CUtensorMap tb = make_tmap_parts(x, T, K, bn, 4, ldx * 2);
  launch_w4_bn(bn, tr, tb, a, a.m_tiles * a.k_splits, stream);
  if (a.k_splits > 1) {
    const unsigned blocks = (unsigned)(((size_t)T * N / 4 + 255) / 256);
    launch_pdl(eight_planes(blocks, a.k_splits) ? w4_splitk_reduce_kernel<8> : w4_splitk_reduce_kernel<4>, dim3(blocks), dim3(256), 0, stream,
               (const float*)a.ws, a.k_splits, T, N, ldy, alpha, a.bias, reinterpret_cast<__nv_bfloat16*>(a.out));
    ++launches;
  }
  return launches;
}

// Grouped form over a device-built tile list (mixture of experts): y[row, :] = dequant(codes[e(row)]) * xp[row, :]
// (+ bias[e(row)]) for the permuted, per-expert padded rows of xp; `bn` is the token-tile width the list was
// built for (at most 128), `max_tiles` bounds the list. `f16`: xp holds rows of rows_f16 (or fp16 rows of a gated epilogue,
// whose factor the caller folds into alpha); with glu_scale > 0 the epilogue applies the clamped SwiGLU-OAI to the pairs of
// neighbouring features and y receives n_out / 2 fp16 values per row, times glu_scale.
int moe_grouped_linear_w4(const void* xp, long long ldx, const void* codes_stack, const void* scales_stack, int fmt,
                          float alpha, const void* bias_stack, void* y, long long ldy, int rows_cap, int n_out, int K,
                          int experts, const int* tile_expert, const int* tile_row0, const int* num_tiles, int max_tiles,
                          int bn, int* status, cudaStream_t stream, const W4Rows* rows) {
  if (rows_cap <= 0 || max_tiles <= 0) return 0;
  if (K % 64 || n_out % 8 || (ldx & 7) || (ldy & 7)) throw std::runtime_error("moe_grouped_linear_w4: K % 64, n_out % 8 and 16-byte rows required");
  if (fmt < 0 || fmt > 2) throw std::runtime_error("moe_grouped_linear_w4: fmt must be 0, 1 or 2");
  if (bn != 16 && bn != 32 && bn != 64 && bn != 96 && bn != 128) throw std::runtime_error("moe_grouped_linear_w4: token tile must be 16, 32, 64, 96 or 128");
  W4Args a{};
  a.M = n_out; a.N = rows_cap; a.K = K; a.m_tiles = (n_out + W4_BM - 1) / W4_BM; a.k_blocks = K / W4_BK; a.fmt = fmt;
  a.ldc = ldy; a.out = reinterpret_cast<uint16_t*>(y); a.scales = reinterpret_cast<const uint8_t*>(scales_stack);
  a.alpha = alpha; a.bias = reinterpret_cast<const __nv_bfloat16*>(bias_stack); a.status = status;
  a.k_splits = 1; a.kb_per_split = a.k_blocks;
  a.g_tile_expert = tile_expert; a.g_tile_row0 = tile_row0; a.g_num_tiles = num_tiles; a.g_rows = n_out;
  if (rows != nullptr) {
    if (fmt == 2) throw std::runtime_error("moe_grouped_linear_w4: fp16 rows need an FP4 format");
    a.f16 = 1; a.row_factor = rows->factor;
    if (rows->glu_scale > 0.f) {
      if (n_out % 16) throw std::runtime_error("moe_grouped_linear_w4: a gated epilogue needs n_out % 16 == 0");
      a.glu = 1; a.glu_alpha = rows->glu_alpha; a.glu_limit = rows->glu_limit; a.glu_scale = rows->glu_scale;
    }
  }
  // when n_out is not a multiple of 128 the last feature tile of an expert also reads rows of the next expert's
  // codes (or zero fill past the stack); the epilogue never stores those rows
  CUtensorMap tr = make_tmap_2d(codes_stack, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)experts * n_out, K / 2, K / 2,
                                W4_BM, 128, true);
  CUtensorMap tb = make_tmap_parts(xp, rows_cap, K, bn, 4, ldx * 2);
  launch_w4_bn(bn, tr, tb, a, max_tiles * a.m_tiles, stream);
  return 1;
}

}  // namespace fllm
