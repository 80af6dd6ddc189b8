// torch.ops.fllm_b200 bindings of mixture-of-experts kernels over packed weights and over peer memory (expert parallel).
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/library.h>

#include <vector>

#include "fllm_ops.h"

namespace {
using at::Tensor;
using c10::optional;
inline cudaStream_t cur_stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
inline const void* optp(const optional<Tensor>& t) { return t.has_value() && t->defined() ? t->data_ptr() : nullptr; }

// Grouped expert GEMM over packed 4-bit stacks: codes [E, n, k/2] bytes, scales [E, n, k/16] (NVFP4), [E, n, k/32] (MXFP4)
// bytes or [E, n, k/32, 2] bf16 (INT4 group-affine).
int64_t moe_grouped_linear_w4(const Tensor& xp, const Tensor& codes, const Tensor& scales, int64_t fmt, double alpha,
                              const optional<Tensor>& bias_stack, Tensor y, const Tensor& tile_expert,
                              const Tensor& tile_row0, const Tensor& num_tiles, int64_t bn, const optional<Tensor>& status) {
  TORCH_CHECK(codes.dim() == 3 && codes.is_contiguous() && codes.element_size() == 1, "codes: contiguous [E, n, k/2] bytes");
  TORCH_CHECK(scales.is_contiguous() && scales.is_cuda(), "scales: contiguous device tensor");
  TORCH_CHECK(xp.dim() == 2 && xp.stride(1) == 1 && xp.size(1) == codes.size(2) * 2 && xp.scalar_type() == at::kBFloat16, "xp: [rows, k] bf16");
  TORCH_CHECK(y.dim() == 2 && y.stride(1) == 1 && y.size(0) == xp.size(0) && y.size(1) == codes.size(1), "y: [rows, n]");
  c10::cuda::CUDAGuard guard(xp.device());
  int* st = status.has_value() && status->defined() ? status->data_ptr<int>() : nullptr;
  return fllm::moe_grouped_linear_w4(xp.data_ptr(), xp.stride(0), codes.data_ptr(), scales.data_ptr(), (int)fmt, (float)alpha,
                                     optp(bias_stack), y.data_ptr(), y.stride(0), (int)xp.size(0), (int)codes.size(1),
                                     (int)codes.size(2) * 2, (int)codes.size(0), tile_expert.data_ptr<int>(),
                                     tile_row0.data_ptr<int>(), num_tiles.data_ptr<int>(), (int)tile_expert.numel(), (int)bn,
                                     st, cur_stream());
}

// x bf16 [tokens, k] -> xp fp16 [rows, k] times a power of two per row, factor fp32 [rows] (csrc/gemm_w4a16.cu: rows_f16)
void moe_rows_f16(const Tensor& x, const optional<Tensor>& token_of, Tensor xp, Tensor factor, const optional<Tensor>& row_weight) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.dim() == 2 && x.stride(1) == 1, "x: bf16 rows");
  TORCH_CHECK(xp.scalar_type() == at::kHalf && xp.dim() == 2 && xp.is_contiguous() && xp.size(1) == x.size(1), "xp: contiguous [rows, k] fp16");
  TORCH_CHECK(factor.scalar_type() == at::kFloat && factor.is_contiguous() && factor.numel() >= xp.size(0), "factor: fp32 [rows]");
  const int* t = nullptr;
  if (token_of.has_value() && token_of->defined()) {
    TORCH_CHECK(token_of->scalar_type() == at::kInt && token_of->is_contiguous() && token_of->numel() >= xp.size(0), "token_of: int32 [rows]");
    t = token_of->data_ptr<int>();
  } else {
    TORCH_CHECK(xp.size(0) <= x.size(0), "xp: as many rows as x");
  }
  const float* w = nullptr;
  if (row_weight.has_value() && row_weight->defined()) {
    TORCH_CHECK(row_weight->scalar_type() == at::kFloat && row_weight->is_contiguous() && row_weight->numel() >= xp.size(0), "row_weight: fp32 [rows]");
    w = row_weight->data_ptr<float>();
  }
  c10::cuda::CUDAGuard guard(x.device());
  fllm::rows_f16(x.data_ptr(), x.stride(0), t, w, xp.data_ptr(), factor.data_ptr<float>(), (int)xp.size(0), (int)x.size(1), cur_stream());
}

// The same on fp16 rows; factor: per row, or none (folded into alpha). glu_scale > 0: clamped SwiGLU-OAI in the epilogue, y fp16 [rows, n / 2] times it.
int64_t moe_grouped_linear_w4_f16(const Tensor& xp, const optional<Tensor>& factor, const Tensor& codes, const Tensor& scales, int64_t fmt, double alpha,
                                  const optional<Tensor>& bias_stack, Tensor y, const Tensor& tile_expert, const Tensor& tile_row0, const Tensor& num_tiles,
                                  int64_t bn, const optional<Tensor>& status, double glu_alpha, double glu_limit, double glu_scale) {
  const bool glu = glu_scale > 0;
  TORCH_CHECK(codes.dim() == 3 && codes.is_contiguous() && codes.element_size() == 1, "codes: contiguous [E, n, k/2] bytes");
  TORCH_CHECK(scales.is_contiguous() && scales.is_cuda() && scales.element_size() == 1 &&
              scales.numel() == codes.numel() * 2 / (fmt == 0 ? 16 : 32), "scales: one byte per block");
  TORCH_CHECK(xp.dim() == 2 && xp.stride(1) == 1 && xp.size(1) == codes.size(2) * 2 && xp.scalar_type() == at::kHalf, "xp: [rows, k] fp16");
  TORCH_CHECK(y.dim() == 2 && y.stride(1) == 1 && y.size(0) == xp.size(0) && y.size(1) == codes.size(1) / (glu ? 2 : 1) &&
              y.scalar_type() == (glu ? at::kHalf : at::kBFloat16), "y: [rows, n] bf16, or [rows, n / 2] fp16 behind an activation");
  TORCH_CHECK((reinterpret_cast<uintptr_t>(y.data_ptr()) & 15) == 0, "y: 16-byte aligned");
  fllm::W4Rows r{nullptr, (float)glu_alpha, (float)glu_limit, (float)glu_scale};
  if (factor.has_value() && factor->defined()) {
    TORCH_CHECK(factor->scalar_type() == at::kFloat && factor->is_contiguous() && factor->numel() >= xp.size(0), "factor: fp32 [rows]");
    r.factor = factor->data_ptr<float>();
  }
  c10::cuda::CUDAGuard guard(xp.device());
  int* st = status.has_value() && status->defined() ? status->data_ptr<int>() : nullptr;
  return fllm::moe_grouped_linear_w4(xp.data_ptr(), xp.stride(0), codes.data_ptr(), scales.data_ptr(), (int)fmt, (float)alpha,
                                     optp(bias_stack), y.data_ptr(), y.stride(0), (int)xp.size(0), (int)codes.size(1),
                                     (int)codes.size(2) * 2, (int)codes.size(0), tile_expert.data_ptr<int>(),
                                     tile_row0.data_ptr<int>(), num_tiles.data_ptr<int>(), (int)tile_expert.numel(), (int)bn,
                                     st, cur_stream(), &r);
}

// x bf16 [tokens, k] -> two pieces of e4m3 per row, xq bytes [rows * 2, k] in groups of 16 rows, and their scale atoms (csrc/gemm_mx4_rows.cu: rows_mx)
void moe_rows_mx(const Tensor& x, const optional<Tensor>& token_of, Tensor xq, Tensor sf, int64_t bn, const optional<Tensor>& row_weight,
                 bool placed) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.dim() == 2 && x.stride(1) == 1, "x: bf16 rows");
  TORCH_CHECK(xq.is_cuda() && xq.element_size() == 1 && xq.dim() == 2 && xq.is_contiguous() && xq.size(1) == x.size(1) && xq.size(0) % 2 == 0, "xq: contiguous bytes [rows * 2, k]");
  const int64_t rows = xq.size(0) / 2;
  TORCH_CHECK(bn > 0 && bn % 16 == 0 && rows % bn == 0, "whole tiles of a multiple of 16 rows");
  TORCH_CHECK(sf.is_cuda() && sf.is_contiguous() && sf.nbytes() >= fllm::mx4_scale_bytes((int)rows, (int)x.size(1), (int)bn, 2), "sf: scale atoms of every tile");
  const int* t = nullptr;
  if (token_of.has_value() && token_of->defined()) {
    TORCH_CHECK(token_of->scalar_type() == at::kInt && token_of->is_contiguous() && token_of->numel() >= rows, "token_of: int32 [rows]");
    t = token_of->data_ptr<int>();
  }
  TORCH_CHECK((t != nullptr && !placed) || rows <= x.size(0), "xq: as many rows as x");
  const float* w = nullptr;
  if (row_weight.has_value() && row_weight->defined()) {
    TORCH_CHECK(row_weight->scalar_type() == at::kFloat && row_weight->is_contiguous() && row_weight->numel() >= rows, "row_weight: fp32 [rows]");
    w = row_weight->data_ptr<float>();
  }
  c10::cuda::CUDAGuard guard(x.device());
  fllm::rows_mx(x.data_ptr(), x.stride(0), t, placed, w, xq.data_ptr(), sf.data_ptr(), (int)rows, (int)x.size(1), (int)bn, cur_stream());
}

// Grouped product of such rows (`pieces` each) with a stack of MXFP4 matrices: codes [E, n, k/2] bytes, atoms [E, ceil(n / 128), ceil(k / 128), 512] their
// scales. y: bf16 [rows, n]; or, with y_sf, the clamped SwiGLU-OAI of it as bytes [rows * 3, n / 2] with the scale atoms y_sf.
int64_t moe_grouped_linear_mx4(const Tensor& xq, const Tensor& sf, int64_t pieces, const Tensor& codes, const Tensor& atoms, double alpha,
                               const optional<Tensor>& bias_stack, Tensor y, const optional<Tensor>& y_sf, const Tensor& tile_expert, const Tensor& tile_row0,
                               const Tensor& tile_rows, const Tensor& num_tiles, int64_t bn, const optional<Tensor>& status, double glu_alpha,
                               double glu_limit) {
  TORCH_CHECK(codes.is_cuda() && codes.dim() == 3 && codes.is_contiguous() && codes.element_size() == 1, "codes: contiguous [E, n, k/2] bytes");
  const int64_t E = codes.size(0), n = codes.size(1), k = codes.size(2) * 2;
  TORCH_CHECK(k % 128 == 0 || codes.storage().nbytes() >= (size_t)(codes.storage_offset() + codes.numel() + 32), "codes: 32 bytes behind the stack where k % 128 != 0");
  TORCH_CHECK(atoms.is_cuda() && atoms.is_contiguous() && atoms.nbytes() == (size_t)(E * ((n + 127) / 128) * ((k + 127) / 128) * 512), "atoms: scales of every 128 x 128 codes");
  TORCH_CHECK((pieces == 2 || pieces == 3) && xq.is_cuda() && xq.dim() == 2 && xq.is_contiguous() && xq.element_size() == 1 && xq.size(1) == k && xq.size(0) % pieces == 0,
              "xq: bytes [rows * pieces, k]");
  const int64_t rows = xq.size(0) / pieces;
  TORCH_CHECK(bn > 0 && rows % bn == 0 && sf.is_cuda() && sf.is_contiguous() && sf.nbytes() >= fllm::mx4_scale_bytes((int)rows, (int)k, (int)bn, (int)pieces), "sf: scale atoms of every tile");
  TORCH_CHECK(tile_rows.numel() >= tile_expert.numel() && tile_row0.numel() >= tile_expert.numel(), "a row and a number of rows per tile");
  const fllm::Mx4Rows x{xq.data_ptr(), sf.data_ptr(), (int)rows, (int)pieces};
  const fllm::Mx4Tiles tiles{tile_expert.data_ptr<int>(), tile_row0.data_ptr<int>(), tile_rows.data_ptr<int>(), num_tiles.data_ptr<int>(), (int)tile_expert.numel(), (int)bn};
  fllm::Mx4Glu g{(float)glu_alpha, (float)glu_limit, nullptr, nullptr};
  const bool glu = y_sf.has_value() && y_sf->defined();
  if (glu) {
    TORCH_CHECK(y.dim() == 2 && y.is_contiguous() && y.element_size() == 1 && y.size(0) == rows * 3 && y.size(1) == n / 2, "y: bytes [rows * 3, n / 2]");
    TORCH_CHECK(y_sf->is_cuda() && y_sf->is_contiguous() && y_sf->nbytes() >= fllm::mx4_scale_bytes((int)rows, (int)n / 2, (int)bn, 3), "y_sf: scale atoms of every tile");
    g.q = y.data_ptr();
    g.sf = y_sf->data_ptr();
  } else {
    TORCH_CHECK(y.dim() == 2 && y.stride(1) == 1 && y.size(0) == rows && y.size(1) == n && y.scalar_type() == at::kBFloat16, "y: [rows, n] bf16");
  }
  c10::cuda::CUDAGuard guard(xq.device());
  int* st = status.has_value() && status->defined() ? status->data_ptr<int>() : nullptr;
  return fllm::moe_grouped_linear_mx4(x, codes.data_ptr(), atoms.data_ptr(), (int)E, (int)n, (int)k, (float)alpha, optp(bias_stack), y.data_ptr(), y.stride(0),
                                      glu ? &g : nullptr, tiles, st, cur_stream());
}

// ---- expert-parallel all-to-all: a context of every rank's buffer addresses, then the four steps
std::vector<fllm::EpArgs> g_ep;

int64_t ep_ctx_create(int64_t ranks, int64_t my_rank, int64_t cap, int64_t hidden, int64_t experts_per_rank,
                      std::vector<int64_t> recv_x, std::vector<int64_t> recv_meta, std::vector<int64_t> ctrl,
                      std::vector<int64_t> comb_y) {
  TORCH_CHECK(ranks >= 1 && ranks <= fllm::kMaxEp, "1..8 ranks");
  TORCH_CHECK((int64_t)recv_x.size() == ranks && (int64_t)recv_meta.size() == ranks && (int64_t)ctrl.size() == ranks &&
              (int64_t)comb_y.size() == ranks, "one address per rank expected");
  fllm::EpArgs a{};
  for (int i = 0; i < ranks; ++i) {
    a.recv_x[i] = reinterpret_cast<void*>(recv_x[i]);
    a.recv_meta[i] = reinterpret_cast<void*>(recv_meta[i]);
    a.ctrl[i] = reinterpret_cast<void*>(ctrl[i]);
    a.comb_y[i] = reinterpret_cast<void*>(comb_y[i]);
  }
  a.ranks = (int)ranks; a.my_rank = (int)my_rank; a.cap = (int)cap; a.hidden = (int)hidden;
  a.experts_per_rank = (int)experts_per_rank;
  g_ep.push_back(a);
  return (int64_t)g_ep.size() - 1;
}

// the rank's call counter: one int32 / uint32 in device memory, or none (host-passed call number)
unsigned* ctr_ptr(const optional<Tensor>& t) {
  if (!t.has_value() || !t->defined()) return nullptr;
  TORCH_CHECK(t->is_cuda() && t->element_size() == 4 && t->numel() >= 1, "call counter: one 32-bit integer on the device");
  return reinterpret_cast<unsigned*>(t->data_ptr());
}

const fllm::EpArgs& ep_at(int64_t h) {
  TORCH_CHECK(h >= 0 && h < (int64_t)g_ep.size(), "invalid expert-parallel context handle");
  return g_ep[h];
}

void ep_dispatch(int64_t h, const Tensor& x, const Tensor& ids, int64_t epoch, const optional<Tensor>& status,
                 const optional<Tensor>& call_ctr) {
  const auto& a = ep_at(h);
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.dim() == 2 && x.stride(1) == 1 && x.size(1) == a.hidden, "x: [tokens, hidden] bf16");
  TORCH_CHECK(ids.scalar_type() == at::kInt && ids.is_contiguous() && ids.dim() == 2 && ids.size(0) == x.size(0), "ids: [tokens, k] int32");
  c10::cuda::CUDAGuard guard(x.device());
  fllm::ep_dispatch(a, x.data_ptr(), x.stride(0), ids.data_ptr<int>(), (int)x.size(0), (int)ids.size(1), (unsigned)epoch, ctr_ptr(call_ctr),
                    status.has_value() && status->defined() ? status->data_ptr<int>() : nullptr, cur_stream());
}

void ep_ingest(int64_t h, int64_t epoch, Tensor ids_out, Tensor count_out, const optional<Tensor>& status,
               const optional<Tensor>& call_ctr) {
  const auto& a = ep_at(h);
  TORCH_CHECK(ids_out.scalar_type() == at::kInt && ids_out.is_contiguous() && ids_out.numel() == a.cap, "ids_out: [cap] int32");
  TORCH_CHECK(count_out.scalar_type() == at::kInt && count_out.numel() >= 1, "count_out: int32");
  c10::cuda::CUDAGuard guard(ids_out.device());
  fllm::ep_ingest(a, (unsigned)epoch, ctr_ptr(call_ctr), ids_out.data_ptr<int>(), count_out.data_ptr<int>(),
                  status.has_value() && status->defined() ? status->data_ptr<int>() : nullptr, cur_stream());
}

void ep_return(int64_t h, const Tensor& y, const Tensor& row_of, const Tensor& count, int64_t epoch,
               const optional<Tensor>& call_ctr) {
  const auto& a = ep_at(h);
  TORCH_CHECK(y.scalar_type() == at::kBFloat16 && y.dim() == 2 && y.stride(1) == 1 && y.size(1) == a.hidden, "y: [rows, hidden] bf16");
  TORCH_CHECK(row_of.scalar_type() == at::kInt && row_of.is_contiguous() && row_of.numel() == a.cap, "row_of: [cap] int32");
  c10::cuda::CUDAGuard guard(y.device());
  fllm::ep_return(a, y.data_ptr(), y.stride(0), row_of.data_ptr<int>(), count.data_ptr<int>(), (unsigned)epoch, ctr_ptr(call_ctr),
                  cur_stream());
}

void ep_wait_returns(int64_t h, int64_t epoch, const Tensor& status, const optional<Tensor>& call_ctr) {
  c10::cuda::CUDAGuard guard(status.device());
  fllm::ep_wait_returns(ep_at(h), (unsigned)epoch, ctr_ptr(call_ctr), status.data_ptr<int>(), cur_stream());
}
}  // namespace

TORCH_LIBRARY_FRAGMENT(fllm_b200, m) {
  m.def("moe_grouped_linear_w4(Tensor xp, Tensor codes, Tensor scales, int fmt, float alpha, Tensor? bias_stack, Tensor(a!) y, Tensor tile_expert, Tensor tile_row0, Tensor num_tiles, int bn, Tensor? status) -> int", &moe_grouped_linear_w4);
  m.def("moe_rows_f16(Tensor x, Tensor? token_of, Tensor(a!) xp, Tensor(b!) factor, Tensor? row_weight=None) -> ()", &moe_rows_f16);
  m.def("moe_grouped_linear_w4_f16(Tensor xp, Tensor? factor, Tensor codes, Tensor scales, int fmt, float alpha, Tensor? bias_stack, Tensor(a!) y, Tensor tile_expert, Tensor tile_row0, Tensor num_tiles, int bn, Tensor? status, float glu_alpha=1.0, float glu_limit=0.0, float glu_scale=0.0) -> int", &moe_grouped_linear_w4_f16);
  m.def("moe_rows_mx(Tensor x, Tensor? token_of, Tensor(a!) xq, Tensor(b!) sf, int bn, Tensor? row_weight=None, bool placed=False) -> ()", &moe_rows_mx);
  m.def("moe_grouped_linear_mx4(Tensor xq, Tensor sf, int pieces, Tensor codes, Tensor atoms, float alpha, Tensor? bias_stack, Tensor(a!) y, Tensor(b!)? y_sf, Tensor tile_expert, Tensor tile_row0, Tensor tile_rows, Tensor num_tiles, int bn, Tensor? status, float glu_alpha=1.0, float glu_limit=0.0) -> int", &moe_grouped_linear_mx4);
  m.def("ep_ctx_create(int ranks, int my_rank, int cap, int hidden, int experts_per_rank, int[] recv_x, int[] recv_meta, int[] ctrl, int[] comb_y) -> int", &ep_ctx_create);
  m.def("ep_dispatch(int ctx, Tensor x, Tensor ids, int epoch, Tensor? status, Tensor(a!)? call_ctr=None) -> ()", &ep_dispatch);
  m.def("ep_ingest(int ctx, int epoch, Tensor(a!) ids_out, Tensor(b!) count_out, Tensor? status, Tensor? call_ctr=None) -> ()", &ep_ingest);
  m.def("ep_return(int ctx, Tensor y, Tensor row_of, Tensor count, int epoch, Tensor? call_ctr=None) -> ()", &ep_return);
  m.def("ep_wait_returns(int ctx, int epoch, Tensor(a!) status, Tensor? call_ctr=None) -> ()", &ep_wait_returns);
}
