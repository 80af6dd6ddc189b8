// Prefill attention on the fifth-generation tensor cores: S = Q K^T and O += P V both run as
// tcgen05.mma with their accumulators in tensor memory.
//
// One CTA owns 128 packed query rows (row = query position x head of one KV group, so one K/V tile
// serves every head of the group) of one sequence and walks the KV pages 128 tokens at a time:
//
//   warp 0   producer  TMA: the 8 pages of the K tile, then of the V tile, 128-byte swizzled rows
//   warp 1   issuer    S[128x128] = Q K^T   (A, B from shared memory, K-major)
//                      O[128x128] (+)= P V  (A = P from tensor memory, B = V as an MN-major operand:
//                                            the cache keeps [token][dim], which is V^T's K-major form)
//   warps 2-5 softmax  one thread per row: tcgen05.ld of the row of S, mask, running max / sum,
//                      P as bf16 written over S's first columns with tcgen05.st, and the rescale of
//                      O in tensor memory when the row maximum moved by more than 2^8
//
// Tensor memory: S/P 128 columns + O up to 128 columns = 256, shared memory 97 KB at head dim 128, so
// two CTAs share an SM and one CTA's softmax overlaps the other's MMAs. Head dim 64 and 128 are template
// instances (a tile is one or two 64-column halves). Every wait is bounded (ptx.cuh: mbar_wait) and a
// timeout is reported through the status word.
//
// Reference counterpart: rust/engine/cuda/attention3.cu:57-288 (mma.sync prefill tiles).
#include <unordered_map>

#include "fllm_ops.h"
#include "ptx.cuh"
#include "tma_host.h"

namespace fllm {

namespace {

constexpr int kPageT = 16;
constexpr int kRowsT = 128;        // packed query rows per CTA = tensor memory lanes
constexpr int kTileT = 128;        // KV tokens per tile
constexpr int kHalfBytes = kRowsT * 128;           // one 64-column half of a 128-row tile: 16 KB
// head dim D is a template parameter (64 or 128): a 128-row tile of Q, K or V is D / 64 such halves
template <int D> constexpr int tile_bytes() { return (D / 64) * kHalfBytes; }
constexpr int kThreadsT = 192;
template <int D> constexpr int smem_one() { return 3 * tile_bytes<D>() + 256 + 1024; }   // Q, K, V, barriers, alignment slack
constexpr float kLog2eT = 1.4426950408889634f;
constexpr float kLazyRescale = 8.f;                // keep a stale row maximum while exp2 stays below 2^8

struct FaTmemParams {
  const __nv_bfloat16* q;
  long long ldq;
  const int* block_tables;
  int max_blocks;
  const int* q_starts;
  const int* kv_lens;
  __nv_bfloat16* out;
  long long ldo;
  const float* sinks;
  int* status;
  int hkv, group;
  int window;
  int min_q;             // sequences with fewer query rows are not this kernel's
  float scale_log2, softcap, scale;
  int tile_variant;      // 0: pick by shape; 1 / 2: force one / two query tiles per CTA
  int bidir;             // 1: no causal mask, every query row sees all kv_len tokens (encoders)
  int list_seqs;         // > 0: blockIdx.x counts the tiles of these sequences' prompts (tile_of_list), blockIdx.z is 0
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Two fp32 values an instruction.
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// Shared-memory descriptor of an operand stored as 128-byte swizzled rows with 1024 bytes between
// groups of eight rows, in either major-ness. For the MN-major use (V) every MMA covers one 64-wide
// swizzle atom along N, so both offset fields describe the same stride: eight K rows = 1024 bytes.
__device__ __forceinline__ uint64_t smem_desc_sw128_1k(uint32_t saddr, uint32_t lbo_bytes = 1024) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)(lbo_bytes >> 4) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// One row (thread) of the softmax over one 128-token tile: reads S from tensor memory, updates the row's
// reference maximum and sum, writes P as bf16 over S's first 64 columns and, when the maximum of any row of
// the warp moved by more than 2^8, rescales the warp's rows of O. `t_s` / `t_o` already carry the lane offset.
template <int D, bool full, bool capped, bool windowed>
__device__ __forceinline__ void softmax_tile_impl(const FaTmemParams& p, uint32_t t_s, uint32_t t_o, int tok0, int lim,
                                                  int beg, bool have_o, float& m_used, float& l) {
  const float cap_in = capped ? p.scale / p.softcap : 0.f;
  const float cap_out = p.softcap * kLog2eT;
  // One warp per lane quarter runs this alone on its scheduler, so the instruction stream is written for
  // instruction-level parallelism: 64 columns per tensor-memory round trip, four independent max / sum chains.
  uint32_t sa[32], sb[32];
  float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {
    tmem_ld_32x32(t_s + 64 * h, sa);
    tmem_ld_32x32(t_s + 64 * h + 32, sb);
    tmem_ld_wait();
    // columns [lo, hi) of these 64 are visible to this row: one compare (two with a window) per element
    const int hi = lim - (tok0 + 64 * h), lo = beg - (tok0 + 64 * h);
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
      float a0 = __uint_as_float(sa[i]), a1 = __uint_as_float(sa[i + 1]);
      float b0 = __uint_as_float(sb[i]), b1 = __uint_as_float(sb[i + 1]);
      if (capped) {
        a0 = tanhf(a0 * cap_in); a1 = tanhf(a1 * cap_in); b0 = tanhf(b0 * cap_in); b1 = tanhf(b1 * cap_in);
      }
      if (!full) {
        if (i >= hi || (windowed && i < lo)) a0 = -INFINITY;
        if (i + 1 >= hi || (windowed && i + 1 < lo)) a1 = -INFINITY;
        if (i + 32 >= hi || (windowed && i + 32 < lo)) b0 = -INFINITY;
        if (i + 33 >= hi || (windowed && i + 33 < lo)) b1 = -INFINITY;
      }
      mx0 = fmaxf(mx0, a0); mx1 = fmaxf(mx1, a1); mx2 = fmaxf(mx2, b0); mx3 = fmaxf(mx3, b1);
    }
  }
  // the scale is positive, so it commutes with the maximum
  const float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3)) * (capped ? cap_out : p.scale_log2);
  // a row keeps its old reference maximum unless the new one is far above it; the decision is per
  // warp because the tensor memory accesses of the rescale are warp-wide
  const bool grow = mx > m_used + kLazyRescale || (m_used == -INFINITY && mx > -INFINITY);
  const bool warp_grow = __any_sync(0xffffffffu, grow);
  float corr = 1.f;
  if (warp_grow) {
    const float m_new = fmaxf(m_used, mx);
    corr = m_new == -INFINITY ? 1.f : ex2(m_used - m_new);     // m_used = -inf gives 0
    m_used = m_new;
    l *= corr;
  }
  const float m_ref = m_used == -INFINITY ? 0.f : m_used;
  float sum0 = 0.f, sum1 = 0.f, sum2 = 0.f, sum3 = 0.f;
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {
    tmem_ld_32x32(t_s + 64 * h, sa);
    tmem_ld_32x32(t_s + 64 * h + 32, sb);
    tmem_ld_wait();
    const int hi = lim - (tok0 + 64 * h), lo = beg - (tok0 + 64 * h);
    uint32_t pa[16], pb[16];
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
      float a0 = __uint_as_float(sa[i]), a1 = __uint_as_float(sa[i + 1]);
      float b0 = __uint_as_float(sb[i]), b1 = __uint_as_float(sb[i + 1]);
      if (capped) {
        a0 = fmaf(cap_out, tanhf(a0 * cap_in), -m_ref); a1 = fmaf(cap_out, tanhf(a1 * cap_in), -m_ref);
        b0 = fmaf(cap_out, tanhf(b0 * cap_in), -m_ref); b1 = fmaf(cap_out, tanhf(b1 * cap_in), -m_ref);
      } else {
        a0 = fmaf(a0, p.scale_log2, -m_ref); a1 = fmaf(a1, p.scale_log2, -m_ref);
        b0 = fmaf(b0, p.scale_log2, -m_ref); b1 = fmaf(b1, p.scale_log2, -m_ref);
      }
      a0 = ex2(a0); a1 = ex2(a1); b0 = ex2(b0); b1 = ex2(b1);
      if (!full) {
        if (i >= hi || (windowed && i < lo)) a0 = 0.f;
        if (i + 1 >= hi || (windowed && i + 1 < lo)) a1 = 0.f;
        if (i + 32 >= hi || (windowed && i + 32 < lo)) b0 = 0.f;
        if (i + 33 >= hi || (windowed && i + 33 < lo)) b1 = 0.f;
      }
      sum0 += a0; sum1 += a1; sum2 += b0; sum3 += b1;
      pa[i >> 1] = pack_bf16x2(a0, a1);
      pb[i >> 1] = pack_bf16x2(b0, b1);
    }
    // P columns [32h, 32h + 32) hold tokens [64h, 64h + 64): they overwrite S columns that were already read
    tmem_st_32x16(t_s + 32 * h, pa);
    tmem_st_32x16(t_s + 32 * h + 16, pb);
  }
  l += (sum0 + sum1) + (sum2 + sum3);
  if (warp_grow && have_o) {
#pragma unroll 1
    for (int c = 0; c < D / 32; ++c) {
      tmem_ld_32x32(t_o + 32 * c, sa);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 32; ++i) sa[i] = __float_as_uint(__uint_as_float(sa[i]) * corr);
      uint32_t lo[16], hi[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) { lo[i] = sa[i]; hi[i] = sa[16 + i]; }
      tmem_st_32x16(t_o + 32 * c, lo);
      tmem_st_32x16(t_o + 32 * c + 16, hi);
    }
  }
  tmem_st_wait();
}

// The mask and soft-cap tests are compile-time so that the common case (a tile every row sees whole, no cap)
// carries no predicated instructions: this code runs one warp per scheduler and every issue slot counts.
template <int D>
__device__ __forceinline__ void softmax_tile(const FaTmemParams& p, uint32_t t_s, uint32_t t_o, int tok0, int lim,
                                             int beg, bool full, bool have_o, float& m_used, float& l) {
  if (p.softcap > 0.f) softmax_tile_impl<D, false, true, true>(p, t_s, t_o, tok0, lim, beg, have_o, m_used, l);
  else if (full) softmax_tile_impl<D, true, false, false>(p, t_s, t_o, tok0, lim, beg, have_o, m_used, l);
  else if (p.window > 0) softmax_tile_impl<D, false, false, true>(p, t_s, t_o, tok0, lim, beg, have_o, m_used, l);
  else softmax_tile_impl<D, false, false, false>(p, t_s, t_o, tok0, lim, beg, have_o, m_used, l);
}

// The same with a row's 128 scores held in registers between the two passes, for warps that have 208 of them. The first 64 probabilities
// are handed over (`p_half`) before the others are computed.
template <int D, bool full, bool capped, bool windowed>
__device__ __forceinline__ void softmax_row_impl(const FaTmemParams& p, uint32_t t_s, uint32_t t_o, int tok0, int lim, int beg, bool have_o,
                                                 uint64_t* p_half, float& m_used, float& l) {
  const float cap_in = capped ? p.scale / p.softcap : 0.f;
  const float scale = capped ? p.softcap * kLog2eT : p.scale_log2;
  uint32_t s[4][32];
#pragma unroll
  for (int c = 0; c < 4; ++c) tmem_ld_32x32(t_s + 32 * c, s[c]);
  tmem_ld_wait();
  const int hi = lim - tok0, lo = beg - tok0;
  float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
  for (int i = 0; i < 128; i += 2) {
    float a[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      a[k] = __uint_as_float(s[i >> 5][(i & 31) + k]);
      if (capped) { a[k] = tanhf(a[k] * cap_in); s[i >> 5][(i & 31) + k] = __float_as_uint(a[k]); }
      if (!full && (i + k >= hi || (windowed && i + k < lo))) a[k] = -INFINITY;
    }
    mx[(i >> 1) & 3] = fmaxf(fmaxf(mx[(i >> 1) & 3], a[0]), a[1]);
  }
  // the scale is positive, so it commutes with the maximum
  const float m = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * scale;
  const bool grow = m > m_used + kLazyRescale || (m_used == -INFINITY && m > -INFINITY);
  if (__any_sync(0xffffffffu, grow)) {
    const float m_new = fmaxf(m_used, m);
    const float corr = m_new == -INFINITY ? 1.f : ex2(m_used - m_new);     // m_used = -inf gives 0
    m_used = m_new;
    l *= corr;
    if (have_o) {
#pragma unroll 1
      for (int c = 0; c < D / 16; ++c) {
        uint32_t o[16];
        tmem_ld_32x16(t_o + 16 * c, o);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
        tmem_st_32x16(t_o + 16 * c, o);
      }
    }
  }
  const float m_ref = m_used == -INFINITY ? 0.f : m_used;
  uint64_t sum[2] = {0, 0};
  const uint64_t scale2 = pack2(scale, scale), ref2 = pack2(-m_ref, -m_ref);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t w[16];
#pragma unroll
    for (int j = 0; j < 32; j += 2) {
      const int i = 32 * c + j;
      const uint64_t x = fma2(pack2(__uint_as_float(s[c][j]), __uint_as_float(s[c][j + 1])), scale2, ref2);
      float2 e = unpack2(x);
      e.x = ex2(e.x); e.y = ex2(e.y);
      if (!full) {
        if (i >= hi || (windowed && i < lo)) e.x = 0.f;
        if (i + 1 >= hi || (windowed && i + 1 < lo)) e.y = 0.f;
      }
      sum[j >> 1 & 1] = add2(sum[j >> 1 & 1], pack2(e.x, e.y));
      w[j >> 1] = pack_bf16x2(e.x, e.y);
    }
    tmem_st_32x16(t_s + 16 * c, w);
    if (c == 1) {
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      if ((threadIdx.x & 31) == 0) mbar_arrive(p_half);
    }
  }
  const float2 l0 = unpack2(sum[0]), l1 = unpack2(sum[1]);
  l += (l0.x + l0.y) + (l1.x + l1.y);
  tmem_st_wait();
}

template <int D>
__device__ __forceinline__ void softmax_row(const FaTmemParams& p, uint32_t t_s, uint32_t t_o, int tok0, int lim, int beg, bool full, bool have_o,
                                            uint64_t* p_half, float& m_used, float& l) {
  if (p.softcap > 0.f) softmax_row_impl<D, false, true, true>(p, t_s, t_o, tok0, lim, beg, have_o, p_half, m_used, l);
  else if (full) softmax_row_impl<D, true, false, false>(p, t_s, t_o, tok0, lim, beg, have_o, p_half, m_used, l);
  else if (p.window > 0) {
    // Two bounds per score: in one pass over 128 registers their code is twice as long and slower than two passes over 64 (2048 tokens under a
    // window of 128, 32 query and 8 key heads of 64: 33.7 against 30.6 us).
    softmax_tile_impl<D, false, false, true>(p, t_s, t_o, tok0, lim, beg, have_o, m_used, l);
    tc_fence_before_sync();
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(p_half);
  }
  else softmax_row_impl<D, false, false, false>(p, t_s, t_o, tok0, lim, beg, have_o, p_half, m_used, l);
}

// Rows [row0, row0 + 128 TILES) of the CTA's queries to shared memory, in the layout TMA's 128-byte swizzle would have produced, by THREADS threads that
// leave once their part is there and visible to the tensor cores. Asynchronous copies, all of a thread's under way at once: through registers, a
// row's index divided out for each, they took 13,000 clocks for 256 rows of 128 and held back everything else.
template <int D, int TILES, int THREADS>
__device__ __forceinline__ void load_q(const FaTmemParams& p, uint8_t* sq, int t, int first_token, int kvh, int n_rows) {
  const int shift = __ffs(p.group) - 1;                 // the group divides 128
#pragma unroll 4
  for (int i = t; i < TILES * kRowsT * (D / 8); i += THREADS) {
    const int r = i / (D / 8), c = i % (D / 8), rr = r & (kRowsT - 1);
    const int qi = r >> shift, hg = r - (qi << shift);
    const bool valid = r < n_rows;
    const __nv_bfloat16* src = p.q + (size_t)(first_token + (valid ? qi : 0)) * p.ldq + (size_t)(kvh * p.group + hg) * D + c * 8;
    const uint32_t dst = smem_u32(sq + (r >> 7) * tile_bytes<D>() + (c >> 3) * kHalfBytes + rr * 128 + (((c & 7) ^ (rr & 7)) << 4));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  fence_proxy_async_smem();
}

// Final normalisation (with the head's sink, if any) and store of a warp's 32 rows of O, r0 the first. They pass through 64 D bytes of shared memory of the
// warp's own, so that a store instruction writes whole rows: with a row to each lane every one of them touched 32 rows, 16 bytes of each (256 rows
// of 128: 6400 clocks to the end of the CTA, 4400 to 5400 now).
template <int D>
__device__ __forceinline__ void store_rows(const FaTmemParams& p, uint32_t t_o, uint8_t* stage, int r0, int n_rows, int first_token, int kvh,
                                           float m_used, float l) {
  constexpr int C = D / 8;                              // pieces of 16 bytes in a row
  const int lane = threadIdx.x & 31, shift = __ffs(p.group) - 1;
  float ll = l, c = 1.f;
  if (p.sinks && r0 + lane < n_rows) {
    const float sk2 = p.sinks[kvh * p.group + ((r0 + lane) & (p.group - 1))] * kLog2eT;
    const float mn = fmaxf(m_used, sk2);
    c = m_used == -INFINITY ? 0.f : ex2(m_used - mn);
    ll = ll * c + ex2(sk2 - mn);
  }
  const float inv = ll > 0.f ? c / ll : 0.f;
#pragma unroll 1
  for (int cc = 0; cc < D / 32; ++cc) {
    uint32_t orow[32];
    tmem_ld_32x32(t_o + 32 * cc, orow);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 32; i += 8) {
      uint4 w;
      w.x = pack_bf16x2(__uint_as_float(orow[i]) * inv, __uint_as_float(orow[i + 1]) * inv);
      w.y = pack_bf16x2(__uint_as_float(orow[i + 2]) * inv, __uint_as_float(orow[i + 3]) * inv);
      w.z = pack_bf16x2(__uint_as_float(orow[i + 4]) * inv, __uint_as_float(orow[i + 5]) * inv);
      w.w = pack_bf16x2(__uint_as_float(orow[i + 6]) * inv, __uint_as_float(orow[i + 7]) * inv);
      *reinterpret_cast<uint4*>(stage + lane * (2 * D) + (((4 * cc + (i >> 3)) ^ (lane & 7)) << 4)) = w;
    }
  }
  __syncwarp();
#pragma unroll 4
  for (int k = 0; k < C; ++k) {
    const int r = k * (32 / C) + lane / C, piece = lane % C;
    const uint4 w = *reinterpret_cast<const uint4*>(stage + r * (2 * D) + ((piece ^ (r & 7)) << 4));
    const int qi = (r0 + r) >> shift, hg = (r0 + r) - (qi << shift);
    if (r0 + r < n_rows) *reinterpret_cast<uint4*>(p.out + (size_t)(first_token + qi) * p.ldo + (size_t)(kvh * p.group + hg) * D + piece * 8) = w;
  }
}

// The sequence and query tile that are the `want`-th of all prompts; false past the last. (A CTA per tile and sequence
// leaves the decode rows of a mixed step CTAs that find nothing to do, each of which still takes an SM for its launch: 200 rows beside a prompt
// of 1500, 64 query and 8 key heads of 64, window of 128: 442 -> 77 us with the decode rows.) Called by all THREADS; sums over as many sequences
// at a time.
template <int THREADS>
__device__ bool tile_of_list(const FaTmemParams& p, int rq, int want, int& seq, int& tile) {
  __shared__ int warp_sum[THREADS / 32], found[2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) found[0] = -1;
  int before = 0;
  for (int s0 = 0; s0 < p.list_seqs; s0 += THREADS) {
    const int s = s0 + threadIdx.x;
    const int qn = s < p.list_seqs ? p.q_starts[s + 1] - p.q_starts[s] : 0;
    const int mine = qn >= p.min_q ? (qn + rq - 1) / rq : 0;
    int sum = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += v;
    }
    if (lane == 31) warp_sum[warp] = sum;
    __syncthreads();
    int first = before + sum - mine;
    for (int w = 0; w < THREADS / 32; ++w) {
      if (w < warp) first += warp_sum[w];
      before += warp_sum[w];
    }
    if (want >= first && want < first + mine) { found[0] = s; found[1] = mine - 1 - (want - first); }      // the longest KV range first
    __syncthreads();
    if (found[0] >= 0 || want < before) break;
  }
  seq = found[0]; tile = found[1];
  return seq >= 0;
}

template <int D>
__global__ void __launch_bounds__(kThreadsT, 2)
fa_prefill_tmem_kernel(const __grid_constant__ CUtensorMap tma_k, const __grid_constant__ CUtensorMap tma_v,
                       const FaTmemParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sq = smem;
  constexpr int TB = tile_bytes<D>();
  uint8_t* sk = smem + TB;
  uint8_t* sv = smem + 2 * TB;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 3 * TB);
  uint64_t* k_full = bars + 0;
  uint64_t* v_full = bars + 1;
  uint64_t* k_empty = bars + 2;
  uint64_t* v_empty = bars + 3;
  uint64_t* s_full = bars + 4;
  uint64_t* p_ready = bars + 5;
  uint64_t* o_done = bars + 6;
  uint64_t* q_full = bars + 7;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int nth = blockIdx.x / p.hkv, kvh = blockIdx.x - nth * p.hkv;
  int qt = gridDim.x / p.hkv - 1 - nth, seq = blockIdx.z;      // the tiles with the longest KV range start first
  const int G = p.group;
  const int RQ = kRowsT / G;
  if (p.list_seqs > 0 && !tile_of_list<kThreadsT>(p, RQ, nth, seq, qt)) return;
  const int q0 = p.q_starts[seq];
  const int qn = p.q_starts[seq + 1] - q0;
  if (qn < p.min_q) return;
  const int qi0 = qt * RQ;
  if (qi0 >= qn) return;
  const int nq = min(RQ, qn - qi0);
  const int n_rows = nq * G;
  const int kv_len = p.kv_lens[seq];
  const int first_pos = kv_len - qn + qi0;
  const int hi_tok = p.bidir ? kv_len : first_pos + nq;
  const int lo_tok = p.window > 0 ? max(0, first_pos - p.window + 1) : 0;
  const int tile_lo = lo_tok / kTileT;
  const int tile_hi = (hi_tok + kTileT - 1) / kTileT;
  const int n_tiles = tile_hi - tile_lo;

  if (threadIdx.x == 0) {
    mbar_init(k_full, 1); mbar_init(v_full, 1); mbar_init(k_empty, 1); mbar_init(v_empty, 1);
    mbar_init(s_full, 1); mbar_init(p_ready, 4); mbar_init(o_done, 1); mbar_init(q_full, 4);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 0 && lane == 0) { tma_prefetch_desc(&tma_k); tma_prefetch_desc(&tma_v); }
  if (warp == 1) { tmem_alloc(tmem_slot, 256); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();                     // decode rows of a mixed batch, the weights of the next product (not before the allocation)
  const uint32_t t_s = tmem_base;            // S, later P in its first 64 columns
  const uint32_t t_o = tmem_base + 128;

  if (warp == 0) {
    const int* table = p.block_tables + (size_t)seq * p.max_blocks;
    const int last_page = (kv_len + kPageT - 1) / kPageT - 1;
    // first cache row of the tile's pages; pages past the sequence repeat its last page (finite values).
    // The next tile's table entries are requested before this tile's waits, so their latency is hidden.
    int rows[kTileT / kPageT], nxt[kTileT / kPageT];
#pragma unroll
    for (int pg = 0; pg < kTileT / kPageT; ++pg)
      nxt[pg] = table[min(tile_lo * (kTileT / kPageT) + pg, last_page)];
    for (int it = 0; it < n_tiles; ++it) {
      const int page1 = (tile_lo + it + 1) * (kTileT / kPageT);
#pragma unroll
      for (int pg = 0; pg < kTileT / kPageT; ++pg) {
        rows[pg] = (nxt[pg] * p.hkv + kvh) * kPageT;
        nxt[pg] = table[min(page1 + pg, last_page)];
      }
      if (it > 0 && !mbar_wait_warp(k_empty, (it - 1) & 1, abort_flag)) break;
      if (elect_one()) {
        mbar_expect_tx(k_full, TB);
#pragma unroll
        for (int pg = 0; pg < kTileT / kPageT; ++pg) {
#pragma unroll
          for (int h = 0; h < D / 64; ++h) tma_load_2d(sk + h * kHalfBytes + pg * 2048, &tma_k, k_full, 64 * h, rows[pg]);
        }
      }
      __syncwarp();
      if (it > 0 && !mbar_wait_warp(v_empty, (it - 1) & 1, abort_flag)) break;
      if (elect_one()) {
        mbar_expect_tx(v_full, TB);
#pragma unroll
        for (int pg = 0; pg < kTileT / kPageT; ++pg) tma_load_3d(sv + pg * (D / 64) * 2048, &tma_v, v_full, 0, rows[pg], 0);
      }
      __syncwarp();
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc_s = make_idesc(128, 128, 1, 1);
    constexpr uint32_t idesc_pv = make_idesc(128, D, 1, 1) | (1u << 16);     // B is MN-major
    const uint64_t dq = make_smem_desc_sw128(smem_u32(sq)), dk = make_smem_desc_sw128(smem_u32(sk));
    const uint64_t dv = smem_desc_sw128_1k(smem_u32(sv), D == 128 ? 2048 : 1024);     // V lands by pages: [page][D / 64][16][64]
    const bool ok = mbar_wait_warp(q_full, 0, abort_flag);
    for (int it = 0; ok && it < n_tiles; ++it) {
      const uint32_t ph = it & 1;
      if (!mbar_wait_warp(k_full, ph, abort_flag)) break;
      tc_fence_after_sync();
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint32_t off = ((k >> 2) * kHalfBytes + (k & 3) * 32) >> 4;
          tc_mma_bf16(t_s, dq + off, dk + off, idesc_s, k > 0);
        }
        tc_commit(s_full);
        tc_commit(k_empty);
      }
      __syncwarp();
      if (!mbar_wait_warp(p_ready, ph, abort_flag) || !mbar_wait_warp(v_full, ph, abort_flag)) break;
      tc_fence_after_sync();
      if (elect_one()) {
        // at D = 128 the second 64-wide atom of V's rows lies half a page further: the leading offset
#pragma unroll
        for (int k = 0; k < kTileT / 16; ++k)
          tc_mma_bf16_ts(t_o, t_s + 8 * k, dv + (uint64_t)(k * (D / 64) * (2048 >> 4)), idesc_pv, (it > 0 || k > 0) ? 1u : 0u);
        tc_commit(v_empty);
        if (it == n_tiles - 1) tc_commit(o_done);
      }
      __syncwarp();
    }
  } else {
    const int quarter = warp & 3;                       // the lane quarter this warp may touch
    const int r = quarter * 32 + lane;
    const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
    load_q<D, 1, 128>(p, sq, threadIdx.x - 64, q0 + qi0, kvh, n_rows);
    __syncwarp();
    if (lane == 0) mbar_arrive(q_full);
    int lim = 0, beg = 0;
    if (r < n_rows) {
      lim = p.bidir ? kv_len : first_pos + r / G + 1;
      beg = p.window > 0 ? max(0, lim - p.window) : 0;
    }
    float m_used = -INFINITY, l = 0.f;
    bool ok = true;
    for (int it = 0; it < n_tiles; ++it) {
      const int tok0 = (tile_lo + it) * kTileT;
      if (!mbar_wait(s_full, it & 1, abort_flag)) { ok = false; break; }
      tc_fence_after_sync();
      // whole tile visible to every row of the CTA: no per-element mask
      const bool full = p.window == 0 && tok0 + kTileT <= (p.bidir ? kv_len : first_pos + 1) && n_rows == kRowsT;
      softmax_tile<D>(p, t_s + lane_off, t_o + lane_off, tok0, lim, beg, full, it > 0, m_used, l);
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_ready);
    }
    if (ok && mbar_wait(o_done, 0, abort_flag)) {
      tc_fence_after_sync();
      store_rows<D>(p, t_o + lane_off, sq + quarter * 64 * D, quarter * 32, n_rows, q0 + qi0, kvh, m_used, l);      // Q has been read
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) { tc_fence_after_sync(); tmem_dealloc(tmem_base, 256); }
  if (threadIdx.x == 0 && *abort_flag && p.status) atomicCAS(p.status, FLLM_OK, FLLM_ERR_MBAR_TIMEOUT);
}

// The same pipeline with two 128-row query tiles per CTA sharing every K/V tile (half the K/V traffic per
// FLOP, which is what bounds the one-tile kernel: its 64 KB per 8.4 MFLOP tile saturates L2 first). Twelve warps:
// one softmax group of four warps per query tile, three producers, issuer. The issuer interleaves the two tiles
// (PV0, next S0, PV1, next S1) so that one group's softmax runs under the other tile's MMAs; K and V are
// double buffered. Tensor memory: S0 S1 O0 O1 = 512 columns, one CTA per SM.
//
// What bounds it: the chain of a group (softmax, PV, next S), 3000 to 3300 clocks per tile where the tensor pipe and the exponentials need 2048
// each for both groups. A row's scores stay in registers (one pass over tensor memory instead of two; the warps that need no registers leave
// theirs; compiled for the 168 of the launch, a thread spills 48 bytes and reads 188 back), two of them to an instruction, and PV of the first 64 tokens runs while the others' exponentials are computed. (Two S buffers of 64 tokens
// per tile are slower: products of 64 columns read Q twice as often. A share of the exponentials on the multiply-add pipe gave
// 1 % at best.) One lane walks the issuer's loop: five waits voted on by its warp and five elected regions cost 1850 of a tile's 3570
// clocks. The grid runs over the key heads first and from a sequence's longest tiles to its shortest, so that the last CTAs to start are short:
// with a head's tiles next to each other the SMs of 256 CTAs ended up to 40 % apart. K and V are on their way while the queries are
// loaded. 32 query and 8 key heads of 128, us before and now: 2017 tokens at 8161: 292, 230; 2 x 1024: 56, 37.5; 4096: 190, 144; 64 query and
// 8 key heads of 64, 2048 tokens: 102, 80. Under a window the tiles that every row sees whole take the unmasked form.
constexpr int kThreadsT2 = 384;
template <int D> constexpr int smem_two() { return 6 * tile_bytes<D>() + 256 + 1024; }

template <int D>
__global__ void __launch_bounds__(kThreadsT2, 1)
fa_prefill_tmem2_kernel(const __grid_constant__ CUtensorMap tma_k, const __grid_constant__ CUtensorMap tma_v,
                        const FaTmemParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sq = smem;                          // two query tiles
  constexpr int TB = tile_bytes<D>();
  uint8_t* sk = smem + 2 * TB;                 // two stages
  uint8_t* sv = smem + 4 * TB;                 // two stages
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 6 * TB);
  uint64_t* k_full = bars + 0;                 // [2] by stage
  uint64_t* v_full = bars + 2;
  uint64_t* k_empty = bars + 4;
  uint64_t* v_empty = bars + 6;
  uint64_t* s_full = bars + 8;                 // [2] by query tile
  uint64_t* p_ready = bars + 10;
  uint64_t* o_done = bars + 12;
  uint64_t* p_half = bars + 13;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint64_t* q_full = bars + 16;

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int nth = blockIdx.x / p.hkv, kvh = blockIdx.x - nth * p.hkv;
  int qt = gridDim.x / p.hkv - 1 - nth, seq = blockIdx.z;
  const int G = p.group;
  const int RQ = 2 * kRowsT / G;
  if (p.list_seqs > 0 && !tile_of_list<kThreadsT2>(p, RQ, nth, seq, qt)) return;
  const int q0 = p.q_starts[seq];
  const int qn = p.q_starts[seq + 1] - q0;
  if (qn < p.min_q) return;
  const int qi0 = qt * RQ;
  if (qi0 >= qn) return;
  const int nq = min(RQ, qn - qi0);
  const int n_rows = nq * G;
  const int kv_len = p.kv_lens[seq];
  const int first_pos = kv_len - qn + qi0;
  const int hi_tok = p.bidir ? kv_len : first_pos + nq;
  const int lo_tok = p.window > 0 ? max(0, first_pos - p.window + 1) : 0;
  const int tile_lo = lo_tok / kTileT;
  const int tile_hi = (hi_tok + kTileT - 1) / kTileT;
  const int n_tiles = tile_hi - tile_lo;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], D / 64); mbar_init(&v_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1); mbar_init(&p_half[i], 4); mbar_init(&p_ready[i], 4);
    }
    mbar_init(o_done, 1); mbar_init(q_full, 8);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 8 && lane == 0) { tma_prefetch_desc(&tma_k); tma_prefetch_desc(&tma_v); }
  if (warp == 9) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();                     // decode rows of a mixed batch, the weights of the next product (not before the allocation)

  // The block was launched with 168 registers a thread: 256 x 208 + 128 x 88 = 384 x 168.
  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
    if (warp != 9) {
      // Three warps ask for the pages, one box of theirs after the other: warp 8 for the first 64 columns of K, warp 10 for the
      // others, warp 11 for V. (One warp for all 32 boxes of a tile needed longer than the products of the tile.)
      const bool is_v = warp == 11;
      const int half = warp == 10 ? 1 : 0;
      uint64_t *full = is_v ? v_full : k_full, *empty = is_v ? v_empty : k_empty;
      const int* table = p.block_tables + (size_t)seq * p.max_blocks;
      const int last_page = (kv_len + kPageT - 1) / kPageT - 1;
      int rows[kTileT / kPageT], nxt[kTileT / kPageT];
  #pragma unroll
      for (int pg = 0; pg < kTileT / kPageT; ++pg)
        nxt[pg] = table[min(tile_lo * (kTileT / kPageT) + pg, last_page)];
      for (int it = 0; it < n_tiles && (half == 0 || D == 128); ++it) {
        const int b = it & 1;
        const int page1 = (tile_lo + it + 1) * (kTileT / kPageT);
  #pragma unroll
        for (int pg = 0; pg < kTileT / kPageT; ++pg) {
          rows[pg] = (nxt[pg] * p.hkv + kvh) * kPageT;
          nxt[pg] = table[min(page1 + pg, last_page)];
        }
        if (it >= 2 && !mbar_wait_warp(&empty[b], ((it >> 1) - 1) & 1, abort_flag)) break;      // phase of the stage's previous use
        if (elect_one()) {
          if (is_v) {
            mbar_expect_tx(&full[b], TB);
  #pragma unroll
            for (int pg = 0; pg < kTileT / kPageT; ++pg) tma_load_3d(sv + b * TB + pg * (D / 64) * 2048, &tma_v, &full[b], 0, rows[pg], 0);
          } else {
            mbar_expect_tx(&full[b], kHalfBytes);
  #pragma unroll
            for (int pg = 0; pg < kTileT / kPageT; ++pg) tma_load_2d(sk + b * TB + half * kHalfBytes + pg * 2048, &tma_k, &full[b], 64 * half, rows[pg]);
          }
        }
        __syncwarp();
      }
    } else {
      constexpr uint32_t idesc_s = make_idesc(128, 128, 1, 1);
      constexpr uint32_t idesc_pv = make_idesc(128, D, 1, 1) | (1u << 16);     // B is MN-major
      const uint64_t dq = make_smem_desc_sw128(smem_u32(sq)), dk = make_smem_desc_sw128(smem_u32(sk));
      const uint64_t dv = smem_desc_sw128_1k(smem_u32(sv), D == 128 ? 2048 : 1024);     // V lands by pages: [page][D / 64][16][64]
      auto issue_s = [&](int g, int stage) {
  #pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint32_t off = ((k >> 2) * kHalfBytes + (k & 3) * 32) >> 4;
          tc_mma_bf16(tmem_base + 128 * g, dq + g * (TB >> 4) + off, dk + (uint64_t)(stage * (TB >> 4)) + off, idesc_s, k > 0);
        }
      };
      auto issue_pv = [&](int g, int stage, bool first, int part) {            // over tokens [64 part, 64 part + 64)
        const uint32_t t_p = tmem_base + 128 * g, t_o = tmem_base + 256 + 128 * g;
  #pragma unroll
        for (int k = 4 * part; k < 4 * part + 4; ++k)
          tc_mma_bf16_ts(t_o, t_p + 8 * k, dv + (uint64_t)(stage * (TB >> 4)) + k * (D / 64) * (2048 >> 4), idesc_pv, (!first || k > 0) ? 1u : 0u);
      };
      if (elect_one()) {
        bool ok = mbar_wait(&k_full[0], 0, abort_flag) && mbar_wait(q_full, 0, abort_flag);
        if (ok) {
          tc_fence_after_sync();
          issue_s(0, 0);
          tc_commit(&s_full[0]);
          issue_s(1, 0);
          tc_commit(&s_full[1]);
          tc_commit(&k_empty[0]);
        }
        for (int it = 0; ok && it < n_tiles; ++it) {
          const int b = it & 1, nb = b ^ 1;
          const uint32_t ph = (it >> 1) & 1, nph = ((it + 1) >> 1) & 1;
          const bool more = it + 1 < n_tiles;
          ok = mbar_wait(&v_full[b], ph, abort_flag) && mbar_wait(&p_half[0], it & 1, abort_flag);
          if (!ok) break;
          tc_fence_after_sync();
          issue_pv(0, b, it == 0, 0);
          ok = mbar_wait(&p_ready[0], it & 1, abort_flag);
          if (!ok) break;
          tc_fence_after_sync();
          issue_pv(0, b, it == 0, 1);
          if (more) {
            ok = mbar_wait(&k_full[nb], nph, abort_flag);
            if (!ok) break;
            tc_fence_after_sync();
            issue_s(0, nb);
            tc_commit(&s_full[0]);
          }
          ok = mbar_wait(&p_half[1], it & 1, abort_flag);
          if (!ok) break;
          tc_fence_after_sync();
          issue_pv(1, b, it == 0, 0);
          ok = mbar_wait(&p_ready[1], it & 1, abort_flag);
          if (!ok) break;
          tc_fence_after_sync();
          issue_pv(1, b, it == 0, 1);
          tc_commit(&v_empty[b]);
          if (more) {
            issue_s(1, nb);
            tc_commit(&s_full[1]);
            tc_commit(&k_empty[nb]);
          } else {
            tc_commit(o_done);
          }
        }
      }
      __syncwarp();
    }
  } else {                                              // warps 0 - 7
    asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
    const int g = warp >> 2;                            // query tile of this softmax group
    const int quarter = warp & 3;
    const int r = g * kRowsT + quarter * 32 + lane;     // packed row within the CTA
    const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
    load_q<D, 2, 256>(p, sq, threadIdx.x, q0 + qi0, kvh, n_rows);
    __syncwarp();
    if (lane == 0) mbar_arrive(q_full);
    const uint32_t t_s = tmem_base + 128 * g + lane_off, t_o = tmem_base + 256 + 128 * g + lane_off;
    int lim = 0, beg = 0;
    if (r < n_rows) {
      lim = p.bidir ? kv_len : first_pos + r / G + 1;
      beg = p.window > 0 ? max(0, lim - p.window) : 0;
    }
    const int group_first = first_pos + (g * kRowsT) / G;
    // where the last row's window begins: a tile from there on is whole for all rows that see its end
    const int group_beg = p.window > 0 ? (p.bidir ? kv_len : first_pos + ((g + 1) * kRowsT - 1) / G + 1) - p.window : 0;
    const bool group_whole = n_rows >= (g + 1) * kRowsT;
    float m_used = -INFINITY, l = 0.f;
    bool ok = true;
    for (int it = 0; it < n_tiles; ++it) {
      const int tok0 = (tile_lo + it) * kTileT;
      if (!mbar_wait(&s_full[g], it & 1, abort_flag)) { ok = false; break; }
      tc_fence_after_sync();
      const bool full = tok0 >= group_beg && tok0 + kTileT <= (p.bidir ? kv_len : group_first + 1) && group_whole;
      softmax_row<D>(p, t_s, t_o, tok0, lim, beg, full, it > 0, &p_half[g], m_used, l);
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_ready[g]);
    }
    if (ok && mbar_wait(o_done, 0, abort_flag)) {
      tc_fence_after_sync();
      store_rows<D>(p, t_o, sq + g * TB + quarter * 64 * D, r - lane, n_rows, q0 + qi0, kvh, m_used, l);      // Q has been read
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 9) { tc_fence_after_sync(); tmem_dealloc(tmem_base, 512); }
  if (threadIdx.x == 0 && *abort_flag && p.status) atomicCAS(p.status, FLLM_OK, FLLM_ERR_MBAR_TIMEOUT);
}

struct MapKey {
  const void* k;
  const void* v;
  uint64_t rows;
  int d;
  bool operator==(const MapKey& o) const { return k == o.k && v == o.v && rows == o.rows && d == o.d; }
};
struct MapKeyHash {
  size_t operator()(const MapKey& x) const {
    return std::hash<const void*>()(x.k) ^ (std::hash<const void*>()(x.v) * 31) ^ std::hash<uint64_t>()(x.rows * 2 + x.d / 128);
  }
};
struct MapPair { CUtensorMap k, v; };

template <int D>
void launch_tmem(const MapPair& maps, FaTmemParams p, int max_q_len, int num_seqs, int mixed_rows, cudaStream_t s) {
  static bool configured[kMaxDevices] = {};
  if (first_call_on_device(configured)) {
    cuda_check(cudaFuncSetAttribute(fa_prefill_tmem_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_one<D>()),
               "fa_prefill_tmem smem");
    cuda_check(cudaFuncSetAttribute(fa_prefill_tmem2_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_two<D>()),
               "fa_prefill_tmem2 smem");
  }
  // Two query tiles per CTA when that still gives every SM a CTA (tile_variant 1 / 2 forces one: tests only), but not under windows of
  // less than two tiles: of three tiles of keys or so the way in and out is the larger part, and two CTAs of one tile on an SM hide each
  // other's. us with one and two, 2048 tokens, 64 query and 8 key heads of 64: window 128: 48, 54; 256: 61, 62; 512: 83, 67; 32 heads of 128: 35, 37;
  // 43, 41; 54, 48. (With fewer CTAs than SMs two tiles win beside 4096 cached tokens, 832 tokens: 94, 86, and lose without, 25, 27.)
  const int forced = p.tile_variant;
  const int rq2 = 2 * kRowsT / p.group;
  const long long ctas2 = (long long)((max_q_len + rq2 - 1) / rq2) * p.hkv * num_seqs;
  const bool two = forced ? forced == 2 : (max_q_len * p.group >= 2 * kRowsT && ctas2 >= sm_count() && !(p.window > 0 && p.window < 2 * kTileT));
  const int rq = two ? rq2 : kRowsT / p.group, tiles = (max_q_len + rq - 1) / rq;
  dim3 grid((unsigned)tiles * p.hkv, 1, num_seqs);
  if (mixed_rows > 0) {                // P prompts of q rows each have at most sum(q) / rq + P tiles
    const long long bound = max(1, mixed_rows / rq + min(num_seqs, mixed_rows / max(p.min_q, 1)));    // (max_q_len may be an upper bound)
    if (bound < (long long)tiles * num_seqs) { grid = dim3((unsigned)bound * p.hkv, 1, 1); p.list_seqs = num_seqs; }
  }
  if (two) fa_prefill_tmem2_kernel<D><<<grid, kThreadsT2, smem_two<D>(), s>>>(maps.k, maps.v, p);
  else fa_prefill_tmem_kernel<D><<<grid, kThreadsT, smem_one<D>(), s>>>(maps.k, maps.v, p);
  cuda_check(cudaGetLastError(), "fa_prefill_tmem launch");
}

}  // namespace

bool attention_prefill_tmem_supported(int head_dim, int group, int block_size) {
  return (head_dim == 64 || head_dim == 128) && block_size == kPageT && group >= 1 && group <= 16 && (kRowsT % group) == 0;
}

// Tensor maps depend only on the cache tensors, so they are built once per (K, V) pair.
void attention_prefill_tmem(const void* q, long long ldq, const void* k_cache, const void* v_cache, long long num_blocks,
                            const int* block_tables, int max_blocks, const int* q_starts, const int* kv_lens,
                            void* out, long long ldo, int num_seqs, int max_q_len, int min_q, int hq, int hkv,
                            int head_dim, float scale, int window, const float* sinks, float softcap, int* status,
                            cudaStream_t s, int tile_variant, int bidir, int mixed_rows) {
  static std::unordered_map<MapKey, MapPair, MapKeyHash> maps;
  const uint64_t rows = (uint64_t)num_blocks * hkv * kPageT;
  const MapKey key{k_cache, v_cache, rows, head_dim};
  auto it = maps.find(key);
  if (it == maps.end()) {
    if (maps.size() > 4096) maps.clear();
    MapPair mp;
    mp.k = make_tmap_2d(k_cache, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, rows, head_dim, head_dim * 2, kPageT, 64, true);
    mp.v = make_tmap_parts(v_cache, rows, head_dim, kPageT, head_dim / 64);
    it = maps.emplace(key, mp).first;
  }
  FaTmemParams p{};
  p.q = (const __nv_bfloat16*)q; p.ldq = ldq;
  p.block_tables = block_tables; p.max_blocks = max_blocks;
  p.q_starts = q_starts; p.kv_lens = kv_lens;
  p.out = (__nv_bfloat16*)out; p.ldo = ldo;
  p.sinks = sinks; p.status = status;
  p.hkv = hkv; p.group = hq / hkv;
  p.window = window; p.min_q = min_q;
  p.scale = scale; p.scale_log2 = scale * kLog2eT; p.softcap = softcap;
  p.tile_variant = tile_variant;
  p.bidir = bidir;
  if (head_dim == 64) launch_tmem<64>(it->second, p, max_q_len, num_seqs, mixed_rows, s);
  else launch_tmem<128>(it->second, p, max_q_len, num_seqs, mixed_rows, s);
}

}  // namespace fllm
