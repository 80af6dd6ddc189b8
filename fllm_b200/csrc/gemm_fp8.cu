// Block-scaled FP8 (e4m3) GEMM on tcgen05:  y = (x_q * sx) (w_q * sw)^T
//
//   weights      e4m3 [N][K] with one fp32 scale per 128 x 128 block  (sw[N/128][K/128])
//   activations  e4m3 [T][K] with one fp32 scale per token per 128 K  (sx[T][K/128]),
//                produced by quant_fp8_1x128_kernel from bf16 (dynamic, amax / 448)
//
// These scales do not map onto the hardware's 1x32 block-scaled MMA (that needs power-of-two
// scales per 32 values), so every 128-deep K block is multiplied unscaled into a fresh TMEM
// accumulator (tcgen05.mma kind::f8f6f4, four K=32 instructions) and the epilogue warps
// promote it: they read the partial sums out of TMEM, multiply by sx * sw of that K block and
// add them into fp32 registers. TMEM buffers alternate (two of 256 columns, four of fewer), so the
// tensor core works on the next K blocks while one is being promoted. Warp roles, TMA staging (128-byte swizzle, one K block
// = one 128-byte row) and the swap-AB orientation for small token counts are those of
// gemm_bf16.cu.
//
// Reference counterparts: rust/engine/cuda/fp8_block.cu:94-312 (FP32 GEMV / FP16-expanded GEMM for
// block-wise FP8 weights), rust/engine/cuda/fp8_gemm.cu:44-78 (per-128-group activation quant).
// Unlike the reference (docs/multi-gpu.md:166) the format can be cut for tensor parallelism on
// 128-element boundaries.
#include <cuda_fp8.h>

#include <algorithm>

#include "fllm_ops.h"
#include "ptx.cuh"
#include "tma_host.h"

namespace fllm {

constexpr int F8_BM = 128;
constexpr int F8_BK = 128;      // e4m3 elements = bytes per swizzle row = scale block depth
constexpr int F8_UMMA_K = 32;

struct Fp8GemmArgs {
  int M, N, K;              // MMA orientation: D[M][N] = A[M][K] B[N][K]^T
  int m_tiles, n_tiles, k_blocks;
  int transposed;           // 1: A = weights (M = features), tokens in N; out[n * ldc + m]
  long long ldc;
  __nv_bfloat16* out;
  const float* sx;          // [tokens][k_blocks]
  const float* sw;          // [features / 128][k_blocks]
  const __nv_bfloat16* bias;
  int* status;
  int k_splits, kb_per_split;   // work items are (tile, split): few tiles cannot pull the whole HBM bandwidth otherwise
  int whole;                    // the first tiles are one item each, over all of K; only those after them are split
  float* ws;                    // fp32 partial sums when k_splits > 1: [k_splits][tokens][features], or a tile each if whole > 0
};

// Item w of a launch: its tile, its split (-1: a whole tile) and its K blocks.
struct Fp8Item {
  int t, split, kb0, kb1;
  __device__ __forceinline__ Fp8Item(const Fp8GemmArgs& p, int w) : t(w), split(-1), kb0(0), kb1(p.k_blocks) {
    if (w >= p.whole) {                                     // the split is the fastest index
      const int v = w - p.whole;
      split = v % p.k_splits; t = p.whole + v / p.k_splits;
      kb0 = split * p.kb_per_split; kb1 = min(p.k_blocks, kb0 + p.kb_per_split);
    }
  }
};

// Waits for the loads from tensor memory; `r` is used behind it.
__device__ __forceinline__ void tmem_ld_wait_of(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
                 "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]),
                 "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
               :: "memory");
}

template <int BN, bool SWAP, int PER>
struct Fp8Smem {
  static constexpr int kABytes = F8_BM * F8_BK;
  static constexpr int kBBytes = BN * F8_BK;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kScaleFloats = SWAP ? 64 * BN : 0;       // token scales of a swap-AB tile, up to 64 K blocks
  static constexpr int kRing = (PER == 2 ? 96 : 196) * 1024 - kScaleFloats * 4;
  static constexpr int kStages = kRing / kStageBytes > 10 ? 10 : kRing / kStageBytes;
  // A K block's product stays in its buffer until the promoting warps have added it up: the tensor core runs ahead by the other buffers.
  static constexpr int kBuffers = BN == 256 ? 2 : 4;
  static constexpr int kTmemCols = kBuffers * BN < 128 ? (kBuffers * BN < 64 ? 64 : kBuffers * BN) : kBuffers * BN;
  static constexpr int kCols = BN == 256 ? 128 : BN > 64 ? 64 : BN > 32 ? 32 : BN;     // columns of a promoting thread
  static constexpr int kShares = BN / kCols;                        // warps that share a lane quarter split the columns
  static constexpr int kPromote = 128 * kShares;                    // promoting threads: four warps per share
  // TMA warp, MMA warp, promoting warps; with 256 columns two more warps fill up the first four, whose registers go to the others
  static constexpr bool kSplitRegs = BN == 256;
  static constexpr int kFirst = kSplitRegs ? 4 : 2;                 // the first promoting warp
  static constexpr int kThreads = 32 * kFirst + kPromote;
  static constexpr int kTotal = kStages * kStageBytes + kScaleFloats * 4 + 256 + 1024;
  static_assert((2 * kStages + 2 * kBuffers) * 8 + 8 <= 256, "barrier block");
};

// What bounds it: a 128 x 256 x 128 block is 512 clocks of the tensor core, its operands some 700 of L2 with every SM reading (19.6 TB/s in all), its promotion
// 32768 multiply-adds, 256 issue slots of each scheduler, and it takes 1000: the promoting warps go through every block one after the other, and what
// surrounds their multiply-adds (a wait, the first load's latency, the scales, the way back to the top of 2 KB of code) adds up to as much as
// these. So few warps with many columns each: eight of 128, with 224 registers that the first four warps leave them, the next 32 columns on their way
// while 32 are added, the scales read under the first load. Sixteen warps of 64 columns: 141 us for 1965 x 7168 x 8192, this 132 (where the product and wait
// loops were still voted on by whole warps: 147). 128 x 128 tiles read and write shared memory twice as often per product; they remain for few tiles.
template <int BN, bool SWAP, int PER>       // SWAP: tokens in the N dimension; PER: CTAs per SM
__global__ void __launch_bounds__(Fp8Smem<BN, SWAP, PER>::kThreads, PER)
gemm_fp8_block_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                      const Fp8GemmArgs p) {
  using S = Fp8Smem<BN, SWAP, PER>;
  constexpr int STAGES = S::kStages, NBUF = S::kBuffers, COLS = S::kCols;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + STAGES * S::kABytes;
  float* s_scale = reinterpret_cast<float*>(smem + STAGES * S::kStageBytes);
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_scale + S::kScaleFloats);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + STAGES;
  uint64_t* tfull_bar = bars + 2 * STAGES;
  uint64_t* tempty_bar = tfull_bar + NBUF;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + NBUF);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = uniform_warp(), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int a = 0; a < NBUF; ++a) { mbar_init(&tfull_bar[a], 1); mbar_init(&tempty_bar[a], 4 * S::kShares); }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 0 && lane == 0) { tma_prefetch_desc(&tma_a); tma_prefetch_desc(&tma_b); }
  if (warp == 1) { tmem_alloc(tmem_slot, S::kTmemCols); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();
  const int items = p.whole + (p.m_tiles * p.n_tiles - p.whole) * p.k_splits;

  if (warp < S::kFirst) {
    if constexpr (S::kSplitRegs) asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");      // launched with 168 a thread: 128 x 56 + 256 x 224 = 384 x 168
    if (warp == 0) {
      int stage = 0, pre = 0;
      uint32_t phase = 0;
      bool ok = true;
      {                                    // weights are static: the first stages' are requested before waiting for the quantiser
        const Fp8Item it(p, blockIdx.x);
        const int n_idx = it.t / p.m_tiles, m_idx = it.t - n_idx * p.m_tiles;
        const int kb0 = it.kb0;
        pre = min(it.kb1 - kb0, STAGES);
        if (elect_one()) {
          for (int i = 0; i < pre; ++i) {
            mbar_expect_tx(&full_bar[i], S::kStageBytes);
            if (SWAP) tma_load_2d(sA + i * S::kABytes, &tma_a, &full_bar[i], (kb0 + i) * F8_BK, m_idx * F8_BM);
            else tma_load_2d(sB + i * S::kBBytes, &tma_b, &full_bar[i], (kb0 + i) * F8_BK, n_idx * BN);
          }
        }
        __syncwarp();
      }
      pdl_wait();
      ok = elect_one();
      for (int w = blockIdx.x; w < items && ok; w += gridDim.x) {
        const Fp8Item it(p, w);
        const int n_idx = it.t / p.m_tiles, m_idx = it.t - n_idx * p.m_tiles;
        const int kb0 = it.kb0, kb1 = it.kb1;
        for (int kb = kb0; kb < kb1; ++kb) {
          const bool requested = pre > 0;
          if (requested) --pre;
          else if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag)) { ok = false; break; }
          if (!requested) mbar_expect_tx(&full_bar[stage], S::kStageBytes);
          if (!requested || !SWAP) tma_load_2d(sA + stage * S::kABytes, &tma_a, &full_bar[stage], kb * F8_BK, m_idx * F8_BM);
          if (!requested || SWAP) tma_load_2d(sB + stage * S::kBBytes, &tma_b, &full_bar[stage], kb * F8_BK, n_idx * BN);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
      __syncwarp();
    } else if (warp == 1) {
      constexpr uint32_t idesc = make_idesc(F8_BM, BN, 0, 0);      // e4m3 x e4m3
      const uint64_t da0 = make_smem_desc_sw128(smem_u32(sA)), db0 = make_smem_desc_sw128(smem_u32(sB));
      // One lane runs the role and asks both barriers before it uses either answer: an elected region per K block with two waits of the whole warp in front
      // took 750 clocks, half again as many as the products of the block.
      int stage = 0, buf = 0;
      uint32_t phase = 0, buf_phase = 0;
      bool ok = elect_one();
      for (int w = blockIdx.x; w < items && ok; w += gridDim.x) {
        const Fp8Item it(p, w);
        for (int kb = it.kb0; kb < it.kb1; ++kb) {
          // each K block gets its own accumulator: wait until the promoting warps drained this buffer
          const bool drained = mbar_try_wait(&tempty_bar[buf], buf_phase ^ 1), landed = mbar_try_wait(&full_bar[stage], phase);
          if (!(drained || mbar_wait(&tempty_bar[buf], buf_phase ^ 1, abort_flag)) || !(landed || mbar_wait(&full_bar[stage], phase, abort_flag))) { ok = false; break; }
          tc_fence_after_sync();
          const uint64_t da = da0 + (uint64_t)(stage * (S::kABytes >> 4)), db = db0 + (uint64_t)(stage * (S::kBBytes >> 4));
#pragma unroll
          for (int k = 0; k < F8_BK / F8_UMMA_K; ++k)
            tc_mma_f8f6f4(tmem_base + buf * BN, da + 2 * k, db + 2 * k, idesc, k > 0 ? 1u : 0u);
          tc_commit(&empty_bar[stage]);
          tc_commit(&tfull_bar[buf]);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
          if (++buf == NBUF) { buf = 0; buf_phase ^= 1; }
        }
      }
      __syncwarp();
    }
  } else {
    if constexpr (S::kSplitRegs) asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
    const int q = warp & 3, half = (warp - S::kFirst) >> 2;
    const int etid = threadIdx.x - 32 * S::kFirst;
    pdl_wait();                            // scales of the activations; outputs may still be in use by the predecessor
    int buf = 0;
    uint32_t buf_phase = 0;
    bool ok = true;
    for (int w = blockIdx.x; w < items && ok; w += gridDim.x) {
      const Fp8Item it(p, w);
      const int n_idx = it.t / p.m_tiles, m_idx = it.t - n_idx * p.m_tiles;
      const int kb0 = it.kb0, kb1 = it.kb1;
      const int m = m_idx * F8_BM + q * 32 + lane;
      const int n_base = n_idx * BN + half * COLS;
      if (SWAP) {
        // token scales of the tile: s_scale[kb][c] = sx[n + c][kb]
        asm volatile("bar.sync 1, %0;" ::"n"(S::kPromote) : "memory");              // previous tile finished reading
        for (int i = etid; i < (kb1 - kb0) * BN; i += S::kPromote) {
          const int kb = kb0 + i / BN, c = i % BN;
          const int tok = n_idx * BN + c;
          s_scale[i] = tok < p.N ? p.sx[(size_t)tok * p.k_blocks + kb] : 0.f;
        }
        asm volatile("bar.sync 1, %0;" ::"n"(S::kPromote) : "memory");
      }
      // scale of the weights: features lie along the rows (one block of 128 per tile), or along the columns (one per thread: COLS divides 128)
      const float* wrow = p.sw + (size_t)(SWAP ? m_idx : min(n_base, p.N - 1) >> 7) * p.k_blocks;
      const float* xrow = p.sx + (size_t)(SWAP ? 0 : min(m, p.M - 1)) * p.k_blocks;
      // (read ahead as they are: a product of the two scales formed at once would wait for them, 400 clocks a block)
      auto wscale = [&](int kb) { return wrow[min(kb, kb1 - 1)]; };
      auto xscale = [&](int kb) { return SWAP ? 1.f : xrow[min(kb, kb1 - 1)]; };
      float acc[COLS];
#pragma unroll
      for (int c = 0; c < COLS; ++c) acc[c] = 0.f;
      float w0 = wscale(kb0), w1 = wscale(kb0 + 1), x0 = xscale(kb0), x1 = xscale(kb0 + 1);
      for (int kb = kb0; kb < kb1; ++kb) {
        float f = 0.f;
        auto next_scales = [&]() {
          f = SWAP ? w0 : x0 * w0;
          w0 = w1; w1 = wscale(kb + 2);
          x0 = x1; x1 = xscale(kb + 2);
        };
        if (!mbar_wait(&tfull_bar[buf], buf_phase, abort_flag)) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t t_row = tmem_base + buf * BN + half * COLS + ((uint32_t)(q * 32) << 16);
        if constexpr (BN == 256) {                           // the next 32 columns are on their way while these are added
          uint32_t r[2][32];
          tmem_ld_32x32(t_row, r[0]);
          next_scales();
          tmem_ld_wait_of(r[0]);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (i < 3) tmem_ld_32x32(t_row + 32 * (i + 1), r[(i + 1) & 1]);
            else {                                           // all of the buffer is in registers
              tc_fence_before_sync();
              __syncwarp();
              if (lane == 0) mbar_arrive(&tempty_bar[buf]);
            }
#pragma unroll
            for (int c = 0; c < 32; ++c) acc[32 * i + c] += __uint_as_float(r[i & 1][c]) * f;
            if (i < 3) tmem_ld_wait_of(r[(i + 1) & 1]);
          }
        } else {
          next_scales();
          constexpr int CH = COLS < 32 ? 16 : 32;
#pragma unroll
          for (int c0 = 0; c0 < COLS; c0 += CH) {
            uint32_t r[CH];
            if constexpr (CH == 32) tmem_ld_32x32(t_row + c0, r);
            else tmem_ld_32x16(t_row + c0, r);
            tmem_ld_wait();
#pragma unroll
            for (int c = 0; c < CH; ++c) {
              if (SWAP) acc[c0 + c] += __uint_as_float(r[c]) * (f * s_scale[(kb - kb0) * BN + half * COLS + c0 + c]);
              else acc[c0 + c] += __uint_as_float(r[c]) * f;
            }
          }
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&tempty_bar[buf]);
        }
        if (++buf == NBUF) { buf = 0; buf_phase ^= 1; }
      }
      if (!ok) break;
      // store
      if (it.split >= 0) {                                    // fp32 partial sums; bias in the reduction
        float* wsp = p.ws + (size_t)it.split * (size_t)p.N * p.M;
        if (SWAP) {                                           // lanes run along features: coalesced
#pragma unroll
          for (int c = 0; c < COLS; ++c)
            if (n_base + c < p.N && m < p.M) wsp[(size_t)(n_base + c) * p.M + m] = acc[c];
        } else if (p.whole > 0) {
          wsp = p.ws + (((size_t)it.split * (p.m_tiles * p.n_tiles - p.whole) + (it.t - p.whole)) * F8_BM + q * 32 + lane) * BN + half * COLS;
#pragma unroll
          for (int c = 0; c < COLS; c += 4) *reinterpret_cast<float4*>(wsp + c) = make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
        } else if (m < p.M) {
#pragma unroll
          for (int c = 0; c < COLS; c += 4)
            if (n_base + c < p.N) *reinterpret_cast<float4*>(wsp + (size_t)m * p.N + n_base + c) = make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
        }
      } else if (!SWAP) {
        if (m < p.M) {
          __nv_bfloat16* dst = p.out + (size_t)m * p.ldc + n_base;
#pragma unroll
          for (int c = 0; c < COLS; c += 8) {
            if (n_base + c < p.N) {
              float v[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) v[i] = acc[c + i] + (p.bias ? __bfloat162float(p.bias[n_base + c + i]) : 0.f);
              uint4 o;
              o.x = pack_bf16x2(v[0], v[1]); o.y = pack_bf16x2(v[2], v[3]);
              o.z = pack_bf16x2(v[4], v[5]); o.w = pack_bf16x2(v[6], v[7]);
              *reinterpret_cast<uint4*>(dst + c) = o;
            }
          }
        }
      } else {
        const float bias_m = (p.bias && m < p.M) ? __bfloat162float(p.bias[m]) : 0.f;
        const bool odd = lane & 1;
#pragma unroll
        for (int c = 0; c < COLS; c += 2) {
          const float own0 = acc[c] + bias_m, own1 = acc[c + 1] + bias_m;
          const float recv = __shfl_xor_sync(0xffffffffu, odd ? own0 : own1, 1);
          const int n = n_base + c + (odd ? 1 : 0);
          const int mm = odd ? m - 1 : m;
          const uint32_t packed = odd ? pack_bf16x2(recv, own1) : pack_bf16x2(own0, recv);
          if (n < p.N && mm < p.M) *reinterpret_cast<uint32_t*>(p.out + (size_t)n * p.ldc + mm) = packed;
        }
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) { tc_fence_after_sync(); tmem_dealloc(tmem_base, S::kTmemCols); }
  if (threadIdx.x == 0 && *abort_flag && p.status) atomicCAS(p.status, FLLM_OK, FLLM_ERR_MBAR_TIMEOUT);
}

// out[t][n] = bf16(sum_s ws[s][t][n] + bias[n])
template <int B>
__global__ void fp8_splitk_reduce_kernel(const float* __restrict__ ws, int splits, int rows, int cols, long long ldc,
                                         const __nv_bfloat16* __restrict__ bias, __nv_bfloat16* __restrict__ out) {
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
  o.x = pack_bf16x2(acc.x + b[0], acc.y + b[1]);
  o.y = pack_bf16x2(acc.z + b[2], acc.w + b[3]);
  *reinterpret_cast<uint2*>(out + (size_t)r * ldc + c) = o;
}

// The same over the tiles after the whole ones, whose partial sums lie tile by tile: ws[s][tile][128][bn].
__global__ void fp8_tail_reduce_kernel(const Fp8GemmArgs p, int bn) {
  pdl_launch_dependents();
  pdl_wait();
  const size_t tile = (size_t)F8_BM * bn, n = (size_t)(p.m_tiles * p.n_tiles - p.whole) * tile;
  const size_t i4 = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (i4 >= n) return;
  const int t0 = row_of_element(i4, (int)tile), t = p.whole + t0, within = (int)(i4 - t0 * tile);
  const int n_idx = t / p.m_tiles, m_idx = t - n_idx * p.m_tiles;
  const int r = m_idx * F8_BM + within / bn, c = n_idx * bn + within % bn;
  if (r >= p.M || c >= p.N) return;
  const float4 acc = sum_splits4(p.ws + i4, n, p.k_splits);
  float b[4] = {0.f, 0.f, 0.f, 0.f};
  if (p.bias) for (int i = 0; i < 4; ++i) b[i] = __bfloat162float(p.bias[c + i]);
  uint2 o;
  o.x = pack_bf16x2(acc.x + b[0], acc.y + b[1]);
  o.y = pack_bf16x2(acc.z + b[2], acc.w + b[3]);
  *reinterpret_cast<uint2*>(p.out + (size_t)r * p.ldc + c) = o;
}

// x bf16 [T][K] -> e4m3 [T][K] and scales [T][K/128] (amax / 448 per 128 values). Half a warp per group, 16 bytes per lane (one warp per
// group with 8 bytes per lane moved 2.3 TB/s at 1965 x 8192). Groups are counted in 32 bits: with a 64-bit quotient per thread the kernel was bound by
// its instructions (1965 x 8192: 13.1 -> 12.3 us).
__global__ void __launch_bounds__(256) quant_fp8_1x128_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, uint8_t* __restrict__ xq,
                                                              float* __restrict__ sx, int tokens, int K) {
  pdl_launch_dependents();
  pdl_wait();
  const int kb_n = K / 128;
  const unsigned g = blockIdx.x * 16u + (threadIdx.x >> 4);
  const int l = threadIdx.x & 15;
  const bool in = g < (unsigned)tokens * (unsigned)kb_n;
  const int t = in ? (int)(g / (unsigned)kb_n) : 0, kb = in ? (int)(g - (unsigned)t * (unsigned)kb_n) : 0;
  uint4 raw = make_uint4(0, 0, 0, 0);
  if (in) {
    const __nv_bfloat16* src = x + (size_t)t * ldx + kb * 128 + l * 8;
    if ((ldx & 7) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0) {
      raw = *reinterpret_cast<const uint4*>(src);
    } else {
      const uint2 a = reinterpret_cast<const uint2*>(src)[0], b = reinterpret_cast<const uint2*>(src)[1];
      raw = make_uint4(a.x, a.y, b.x, b.y);
    }
  }
  const float2 a = unpack_bf16x2(raw.x), b = unpack_bf16x2(raw.y), c = unpack_bf16x2(raw.z), d = unpack_bf16x2(raw.w);
  float amax = fmaxf(fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(b.x), fabsf(b.y))), fmaxf(fmaxf(fabsf(c.x), fabsf(c.y)), fmaxf(fabsf(d.x), fabsf(d.y))));
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if (!in) return;
  const float scale = fmaxf(amax, 1e-10f) / 448.f, inv = 1.f / scale;
  __nv_fp8x4_e4m3 q0(make_float4(a.x * inv, a.y * inv, b.x * inv, b.y * inv)), q1(make_float4(c.x * inv, c.y * inv, d.x * inv, d.y * inv));
  *reinterpret_cast<uint2*>(xq + (size_t)t * K + kb * 128 + l * 8) = make_uint2(*reinterpret_cast<uint32_t*>(&q0), *reinterpret_cast<uint32_t*>(&q1));
  if (l == 0) sx[(size_t)t * kb_n + kb] = scale;
}

void quant_fp8_1x128(const void* x, long long ldx, void* xq, float* sx, int tokens, int K, cudaStream_t s) {
  if (tokens <= 0) return;
  if (K % 128) throw std::runtime_error("quant_fp8_1x128: K must be a multiple of 128");
  const long long groups = (long long)tokens * (K / 128);
  if (groups >= (1ll << 31)) throw std::runtime_error("quant_fp8_1x128: more than 2^31 groups");
  launch_pdl(quant_fp8_1x128_kernel, dim3((unsigned)((groups + 15) / 16)), dim3(256), 0, s, (const __nv_bfloat16*)x, ldx, (uint8_t*)xq, sx, tokens, K);
}

template <int BN, bool SWAP, int PER = 1>
static void launch_fp8(const CUtensorMap& ta, const CUtensorMap& tb, const Fp8GemmArgs& a, int grid, cudaStream_t s) {
  using S = Fp8Smem<BN, SWAP, PER>;
  static bool configured[kMaxDevices] = {};
  if (first_call_on_device(configured)) {
    cuda_check(cudaFuncSetAttribute(gemm_fp8_block_kernel<BN, SWAP, PER>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kTotal),
               "cudaFuncSetAttribute(gemm_fp8_block_kernel)");
  }
  launch_pdl(gemm_fp8_block_kernel<BN, SWAP, PER>, dim3(grid), dim3(S::kThreads), S::kTotal, s, ta, tb, a);
}

// y[T][N] = dequant(xq, sx) * dequant(wq, sw)^T (+ bias)
int linear_fp8_block(const void* xq, const float* sx, const void* wq, const float* sw, const void* bias, void* y,
                     long long ldy, int T, int N, int K, int* status, cudaStream_t stream, void* workspace,
                     size_t workspace_bytes) {
  if (T <= 0 || N <= 0) return 0;
  if (K % 128 || N % 128) throw std::runtime_error("linear_fp8_block: N and K must be multiples of 128");
  if (K / 128 > 64 * 4) throw std::runtime_error("linear_fp8_block: K above 32768 is not supported");
  Fp8GemmArgs a{};
  a.K = K; a.k_blocks = K / 128;
  a.out = reinterpret_cast<__nv_bfloat16*>(y); a.ldc = ldy;
  a.sx = sx; a.sw = sw; a.bias = reinterpret_cast<const __nv_bfloat16*>(bias); a.status = status;
  const bool swap = T <= 64;                          // decode: features fill the 128-row MMA dimension
  const int sms = sm_count();
  a.M = swap ? N : T; a.N = swap ? T : N; a.transposed = swap;
  a.m_tiles = (a.M + F8_BM - 1) / F8_BM;
  // Tile and K splits by the rounds of items over the SMs, in units of 1/100 us. A K block takes the time in which an SM's share of the HBM
  // bandwidth brings its weights (37 per 128 features) when no other tile of the step reads them, too (64-wide tiles spare few tokens the
  // partial sums or some of them, 28: 128 x 1280 x 8192 13.6 -> 12.0 us, 128 x 8192 x 3584 16.9 -> 15.8; 7168 x 8192 needs them and took 27.7
  // against 24.9); else its operands from L2 and its promotion with every SM busy (256-wide tiles 60, 128-wide 36, of a round of 1965 x 7168 x 8192). Partial sums are
  // written and read once, and cost a launch. With more tiles than SMs either all are split, or those of the last, partly filled
  // round alone (whole > 0): 1965 x 7168 x 8192 has 448 tiles of 256 for 3 x 148, and the last four took as long
  // as a full round (172 -> 149 us). 16-wide tiles may run as two CTAs per SM with half of the ring each, which share its bandwidth: one's
  // scales, last blocks and stores lie under the other's stream, and the rounds are half as many (16 x 57344 x 8192 with its quantiser
  // 89.8 -> 82.0 us, 16 x 28672 x 4096 27.6 -> 23.5); with few tiles one CTA and its whole ring are faster (1 x 16384 x 2048 9.7 against 10.3).
  int bn = T <= 16 ? 16 : (T <= 32 ? 32 : 64), splits = 1, whole = 0, per = 1;
  const int deep = (a.k_blocks + 63) / 64, least = swap ? deep : 1;   // swap-AB: the token scales of a split fit their shared-memory block
  // Tiles of up to 64 tokens store pairs of features, wider ones eight at a time; the kernels that add partial sums store four. So rows
  // aligned to 4 bytes are not split, and more than 64 tokens go into rows aligned to 8 bytes only as partial sums of all tiles.
  auto rows_of = [&](int n) { return ldy % n == 0 && reinterpret_cast<uintptr_t>(y) % (2 * n) == 0; };
  const bool can_split = workspace && rows_of(4), can_store = rows_of(swap ? 2 : 8);
  long long best = -1;
  for (int w : {swap ? bn : 256, swap ? 0 : 128, swap ? 0 : 64}) {
    if (w == 0 || (w == 256 && N % 256)) continue;
    const int n_tiles = (a.N + w - 1) / w;
    const long long block = swap ? 37 : a.m_tiles == 1 ? (w == 256 ? 74 : w == 128 ? 37 : 28) : (w == 256 ? 60 : w == 128 ? 36 : 28);
    for (int s = least; s <= 16 * deep && s <= a.k_blocks; ++s) {
      if (s == 1 && !can_store) continue;
      if (s > 1 && (!can_split || (size_t)s * T * N * 4 > workspace_bytes)) break;
      const long long items = (long long)a.m_tiles * n_tiles * s;
      for (int two = 1; two <= (w == 16 ? 2 : 1); ++two) {
        const long long rounds = (items + sms * two - 1) / (sms * two);
        const long long cost = rounds * ((a.k_blocks + s - 1) / s * (two == 2 && items > sms ? 2 * block : block) + 100) +
                               (s > 1 ? 250 + (long long)((double)s * T * N * 8 / 60000.0) : 0);
        if (best < 0 || cost < best) { best = cost; bn = w; splits = s; whole = 0; per = two; }
      }
    }
    const long long tiles = (long long)a.m_tiles * n_tiles, first = tiles / sms * sms, tail = tiles - first;
    if (swap || !can_split || !can_store || first == 0) continue;
    for (int s = 2; s <= 16 && s <= a.k_blocks && tail; ++s) {
      const long long bytes = s * tail * F8_BM * w * 4;
      if ((size_t)bytes > workspace_bytes) break;
      const long long cost = first / sms * (a.k_blocks * block + 100) + (tail * s + sms - 1) / sms * ((a.k_blocks + s - 1) / s * block + 100) + 250 + bytes / 30000;
      if (best < 0 || cost < best) { best = cost; bn = w; splits = s; whole = (int)first; }
    }
  }
  if (best < 0 && !can_store)
    throw std::runtime_error("linear_fp8_block: output rows must be aligned to 4 bytes for up to 64 tokens, to 16 for more (8 where there is room for partial sums)");
  if (best < 0) throw std::runtime_error("linear_fp8_block: K above 8192 needs a split-K workspace and output rows aligned to 8 bytes");
  a.n_tiles = (a.N + bn - 1) / bn;
  const CUtensorMap tw = make_tmap_2d(wq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, N, K, K, swap ? F8_BM : bn, F8_BK, true);
  const CUtensorMap tx = make_tmap_2d(xq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, T, K, K, swap ? bn : F8_BM, F8_BK, true);
  const CUtensorMap &ta = swap ? tw : tx, &tb = swap ? tx : tw;
  a.kb_per_split = (a.k_blocks + splits - 1) / splits;
  a.k_splits = (a.k_blocks + a.kb_per_split - 1) / a.kb_per_split;
  a.whole = a.k_splits > 1 ? whole : a.m_tiles * a.n_tiles;
  a.ws = reinterpret_cast<float*>(workspace);
  const int grid = std::min(a.whole + (a.m_tiles * a.n_tiles - a.whole) * a.k_splits, sms * per);
  switch (bn) {
    case 16:
      if (per == 2) launch_fp8<16, true, 2>(ta, tb, a, grid, stream);
      else launch_fp8<16, true>(ta, tb, a, grid, stream);
      break;
    case 32: launch_fp8<32, true>(ta, tb, a, grid, stream); break;
    case 64:
      if (swap) launch_fp8<64, true>(ta, tb, a, grid, stream);
      else launch_fp8<64, false>(ta, tb, a, grid, stream);
      break;
    case 128: launch_fp8<128, false>(ta, tb, a, grid, stream); break;
    default: launch_fp8<256, false>(ta, tb, a, grid, stream); break;
  }
  if (a.k_splits > 1 && a.whole > 0) {
    const size_t n = (size_t)(a.m_tiles * a.n_tiles - a.whole) * F8_BM * bn;
    launch_pdl(fp8_tail_reduce_kernel, dim3((unsigned)((n / 4 + 255) / 256)), dim3(256), 0, stream, a, bn);
    return 2;
  }
  if (a.k_splits > 1) {
    const unsigned blocks = (unsigned)(((size_t)T * N / 4 + 255) / 256);
    launch_pdl(eight_planes(blocks, a.k_splits) ? fp8_splitk_reduce_kernel<8> : fp8_splitk_reduce_kernel<4>, dim3(blocks), dim3(256), 0, stream, (const float*)a.ws,
               a.k_splits, T, N, ldy, a.bias, a.out);
    return 2;
  }
  return 1;
}

}  // namespace fllm
