// torch.ops.paired_nvfp4.*: argument validation, output allocation, stream lookup, then one call into the C ABI.
// Mirrors the reference's op layer (csrc/ops.cu) schema for schema: same names, argument meaning, output shapes and
// error substrings.  Every forward op only enqueues work on the current CUDA stream of the tensors' device; nothing
// synchronises or reads device memory.
//
// A decode step makes five of these calls and its kernels take less than 50 us together, so what a call costs on the
// host is what the step costs: registered from Python (torch.library + ctypes) a call took 20-40 us, here 4-8.
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <torch/library.h>

#include <algorithm>
#include <atomic>
#include <list>
#include <mutex>
#include <optional>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/paired_nvfp4_b200.h"

namespace {

using at::Tensor;
using c10::optional;

constexpr int64_t kSfBlock = 32;
constexpr int kArchSm = 100;

std::atomic<int> g_sm_margin{0};

void check_rc(int rc) { TORCH_CHECK(rc == 0, pnv_last_error()); }

struct DeviceInfo { int sm_version = 0, sm_count = 0; };

// (sm_version, sm_count) of a CUDA device, queried once (reference: csrc/ops.cu:86-103)
DeviceInfo device_info(int dev) {
  constexpr int kMax = 64;
  static DeviceInfo info[kMax];
  static std::once_flag once[kMax];
  TORCH_CHECK(dev >= 0 && dev < kMax, "unexpected CUDA device index ", dev);
  std::call_once(once[dev], [dev] {
    int major = 0, minor = 0, sms = 0;
    cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev);
    cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    info[dev] = DeviceInfo{major * 10 + minor, sms};
  });
  return info[dev];
}

int sm_count(const Tensor& t) { return std::max(1, device_info(t.get_device()).sm_count - g_sm_margin.load(std::memory_order_relaxed)); }

void check_arch(const Tensor& t) {
  const int v = device_info(t.get_device()).sm_version;
  TORCH_CHECK(v == kArchSm, "paired_nvfp4 ops in this module are built for SM", kArchSm,
              " but the tensor is on a compute capability ", v / 10, ".", v % 10, " device");
}

cudaStream_t current_stream(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

// An uninitialised tensor.  Through the dispatcher only where torch is to fill uninitialised memory
// (torch.use_deterministic_algorithms): rows past an expert's count then hold the same bytes in every run.
Tensor empty_on(const Tensor& like, at::IntArrayRef sizes, at::ScalarType dtype) {
  const at::Context& ctx = at::globalContext();
  if (C10_UNLIKELY(ctx.deterministicAlgorithms() && ctx.deterministicFillUninitializedMemory()))
    return at::empty(sizes, like.options().dtype(dtype));
  return at::detail::empty_cuda(sizes, dtype, like.device(), c10::nullopt);
}

int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

struct Dims { int m_ac, k_ac, m_e, k_e; };
Dims physical_dims(int64_t features, int64_t k) {
  Dims d;
  check_rc(pnv_physical_dims((int)features, (int)k, &d.m_ac, &d.k_ac, &d.m_e, &d.k_e));
  return d;
}

const float* f32(const Tensor& t) { return static_cast<const float*>(t.const_data_ptr()); }
const int32_t* i32(const Tensor& t) { return static_cast<const int32_t*>(t.const_data_ptr()); }
const uint8_t* u8(const Tensor& t) { return static_cast<const uint8_t*>(t.const_data_ptr()); }

bool is_int(const Tensor& t) { return t.scalar_type() == at::kInt; }
bool is_float(const Tensor& t) { return t.scalar_type() == at::kFloat; }
bool is_bf16(const Tensor& t) { return t.scalar_type() == at::kBFloat16; }
bool is_byte(const Tensor& t) { return t.scalar_type() == at::kByte; }

void check_gscale_counts(const Tensor& gscale, const Tensor& counts, int64_t E) {
  TORCH_CHECK(is_float(gscale), "gscale must be float32");
  TORCH_CHECK(gscale.numel() == E || gscale.numel() == 1, "gscale must be [E] (per expert) or [1] (shared)");
  TORCH_CHECK(is_int(counts) && counts.numel() == E, "expert_num_tokens must be [E] int32");
  TORCH_CHECK(gscale.is_contiguous() && counts.is_contiguous(), "gscale and expert_num_tokens must be contiguous");
}

int act_kind(c10::string_view activation, double beta) {
  if (activation == "silu") return PNV_ACT_SILU;
  if (activation == "situ") {
    TORCH_CHECK(beta > 0, "situ: beta must be positive, got ", beta);
    return PNV_ACT_SITU;
  }
  TORCH_CHECK(false, "activation must be 'silu' or 'situ', got '", activation, "'");
}

// ---- quantizers, compressor ------------------------------------------------------------------------

// csrc/ops.cu:156-223
std::tuple<Tensor, Tensor, Tensor> compress(const Tensor& w_packed, const Tensor& w_blockscale, int64_t K) {
  TORCH_CHECK(w_packed.is_cuda() && w_blockscale.is_cuda(), "inputs must be CUDA tensors");
  check_arch(w_packed);
  TORCH_CHECK(w_packed.dim() == 3, "w_packed must be [E, out_features, K/2]");
  TORCH_CHECK(w_blockscale.dim() == 3, "w_blockscale must be [E, out_features, ceil(K/SFVecSize)]");
  TORCH_CHECK(w_packed.is_contiguous() && w_blockscale.is_contiguous(), "inputs must be contiguous");
  TORCH_CHECK(is_byte(w_packed), "w_packed must be uint8 (2 e2m1 per byte)");
  const int64_t E = w_packed.size(0), M = w_packed.size(1);
  TORCH_CHECK(K % 2 == 0 && w_packed.size(2) == K / 2, "w_packed last dim must equal K/2");
  TORCH_CHECK(w_blockscale.size(0) == E && w_blockscale.size(1) == M, "w_blockscale must match w_packed in [E, out_features]");
  const int64_t kb = ceil_div(K, kSfBlock);
  TORCH_CHECK(w_blockscale.size(2) == kb, "w_blockscale last dim must be ceil(K/", kSfBlock, ") = ", kb, ", got ",
              w_blockscale.size(2), ". The sparse NVFP4 MMA uses one scale per ", kSfBlock,
              " dense K elements; checkpoints quantized with 16-element groups are incompatible");
  TORCH_CHECK(w_blockscale.element_size() == 1, "w_blockscale must be a 1-byte (e4m3) dtype");
  const Dims d = physical_dims(M, K);
  Tensor a_comp = empty_on(w_packed, {E, d.m_ac, d.k_ac / 2}, at::kByte);
  Tensor e_meta = empty_on(w_packed, {E, d.m_e, d.k_e}, at::kByte);
  Tensor sfa = empty_on(w_packed, {pnv_sf_numel((int)M, (int)K, (int)E)}, at::kByte);
  const c10::cuda::CUDAGuard guard(w_packed.device());
  check_rc(pnv_compress(u8(w_packed), u8(w_blockscale), (int)E, (int)M, (int)K, a_comp.mutable_data_ptr<uint8_t>(),
                        e_meta.mutable_data_ptr<uint8_t>(), sfa.mutable_data_ptr<uint8_t>(), current_stream(w_packed)));
  return {a_comp, e_meta, sfa};
}

// csrc/ops.cu:230-262; `features` is accepted for API symmetry, the layouts do not use it
std::tuple<Tensor, Tensor> quant_act(const Tensor& x, const Tensor& gscale, const Tensor& counts, int64_t /*features*/) {
  TORCH_CHECK(x.is_cuda() && gscale.is_cuda() && counts.is_cuda(), "inputs must be CUDA");
  check_arch(x);
  TORCH_CHECK(x.dim() == 3, "x must be [E, max_n, K]");
  TORCH_CHECK(is_bf16(x) && x.is_contiguous(), "x must be contiguous bf16");
  const int64_t E = x.size(0), max_n = x.size(1), K = x.size(2);
  TORCH_CHECK(K % kSfBlock == 0, "K must be a multiple of ", kSfBlock, ", got ", K);
  check_gscale_counts(gscale, counts, E);
  Tensor b_act = empty_on(x, {E, max_n, K / 2}, at::kByte);
  Tensor sfb = empty_on(x, {pnv_sf_numel((int)max_n, (int)K, (int)E)}, at::kByte);
  const c10::cuda::CUDAGuard guard(x.device());
  check_rc(pnv_quant_act(x.const_data_ptr(), f32(gscale), gscale.numel() == E, i32(counts), (int)E, (int)max_n, (int)K,
                         b_act.mutable_data_ptr<uint8_t>(), sfb.mutable_data_ptr<uint8_t>(), sm_count(x), current_stream(x)));
  return {b_act, sfb};
}

// csrc/ops.cu:269-306
std::tuple<Tensor, Tensor> silu_mul_quant_act(const Tensor& x2, const Tensor& gscale, const Tensor& counts, int64_t /*features*/,
                                              bool interleaved, c10::string_view activation, double beta, double linear_beta) {
  TORCH_CHECK(x2.is_cuda() && gscale.is_cuda() && counts.is_cuda(), "inputs must be CUDA");
  check_arch(x2);
  TORCH_CHECK(x2.dim() == 3, "x2 must be [E, max_n, 2N] ([gate | up] halves)");
  TORCH_CHECK(is_bf16(x2) && x2.is_contiguous(), "x2 must be contiguous bf16");
  const int64_t E = x2.size(0), max_n = x2.size(1);
  TORCH_CHECK(x2.size(2) % 2 == 0, "x2 last dim must be even ([gate | up]), got ", x2.size(2));
  const int64_t N = x2.size(2) / 2;
  TORCH_CHECK(N % kSfBlock == 0, "intermediate width N must be a multiple of ", kSfBlock, ", got ", N);
  check_gscale_counts(gscale, counts, E);
  const int kind = act_kind(activation, beta);
  Tensor b_act = empty_on(x2, {E, max_n, N / 2}, at::kByte);
  Tensor sfb = empty_on(x2, {pnv_sf_numel((int)max_n, (int)N, (int)E)}, at::kByte);
  const c10::cuda::CUDAGuard guard(x2.device());
  check_rc(pnv_silu_mul_quant_act(x2.const_data_ptr(), f32(gscale), gscale.numel() == E, i32(counts), (int)E, (int)max_n,
                                  (int)N, interleaved ? 1 : 0, kind, (float)beta, (float)linear_beta,
                                  b_act.mutable_data_ptr<uint8_t>(), sfb.mutable_data_ptr<uint8_t>(), sm_count(x2), current_stream(x2)));
  return {b_act, sfb};
}

// csrc/ops.cu:314-367; expert_num_tokens only supplies E
std::tuple<Tensor, Tensor> scatter_quant_act(const Tensor& a1, const Tensor& flat_tok, const Tensor& dest_global,
                                             const optional<Tensor>& topk_weights, const Tensor& gscale, const Tensor& counts,
                                             int64_t cap) {
  TORCH_CHECK(a1.is_cuda() && flat_tok.is_cuda() && dest_global.is_cuda() && gscale.is_cuda() && counts.is_cuda(), "inputs must be CUDA");
  check_arch(a1);
  TORCH_CHECK(a1.dim() == 2, "a1 must be [T, K] (token-order hidden states)");
  TORCH_CHECK(is_bf16(a1) && a1.is_contiguous(), "a1 must be contiguous bf16");
  const int64_t K = a1.size(1);
  TORCH_CHECK(K % kSfBlock == 0, "K must be a multiple of ", kSfBlock, ", got ", K);
  TORCH_CHECK(flat_tok.scalar_type() == at::kLong && dest_global.scalar_type() == at::kLong, "flat_tok and dest_global must be int64");
  TORCH_CHECK(flat_tok.dim() == 1 && dest_global.dim() == 1 && flat_tok.numel() == dest_global.numel(),
              "flat_tok and dest_global must be same-length 1D");
  TORCH_CHECK(flat_tok.is_contiguous() && dest_global.is_contiguous(), "plan tensors must be contiguous");
  TORCH_CHECK(cap > 0, "cap must be positive");
  const int64_t n = flat_tok.numel(), E = counts.numel();
  check_gscale_counts(gscale, counts, E);
  const float* w = nullptr;
  if (topk_weights.has_value()) {
    TORCH_CHECK(topk_weights->is_cuda() && is_float(*topk_weights) && topk_weights->is_contiguous() && topk_weights->numel() == n,
                "topk_weights must be contiguous float32 [N]");
    w = f32(*topk_weights);
  }
  // one extra trailing row, as in the reference: b_act is a view of an (E*cap + 1)-row buffer
  Tensor b_ext = empty_on(a1, {E * cap + 1, K / 2}, at::kByte);
  Tensor sfb = empty_on(a1, {pnv_sf_numel((int)cap, (int)K, (int)E)}, at::kByte);
  const c10::cuda::CUDAGuard guard(a1.device());
  check_rc(pnv_scatter_quant_act(a1.const_data_ptr(), static_cast<const int64_t*>(flat_tok.const_data_ptr()),
                                 static_cast<const int64_t*>(dest_global.const_data_ptr()), w, f32(gscale), gscale.numel() == E, n,
                                 (int)K, (int)E, (int)cap, b_ext.mutable_data_ptr<uint8_t>(), sfb.mutable_data_ptr<uint8_t>(),
                                 sm_count(a1), current_stream(a1)));
  return {b_ext.narrow(0, 0, E * cap).view({E, cap, K / 2}), sfb};
}

// csrc/ops.cu:374-411: (expert_num_tokens, route_dest, src_tok, src_route).  Beyond the reference's contiguous [T, topk]
// ids, a [T, 1] view with a row stride is accepted (one id per row of a wider buffer: the expert ids inside the wire
// rows of an expert-parallel dispatch).
std::tuple<Tensor, Tensor, Tensor, Tensor> dispatch_plan(const Tensor& ids, int64_t first_expert, int64_t E, int64_t cap) {
  TORCH_CHECK(ids.is_cuda(), "topk_ids must be CUDA");
  TORCH_CHECK(ids.dim() == 2, "topk_ids must be [T, topk]");
  const bool contiguous = ids.is_contiguous();
  const bool strided = !contiguous && ids.size(1) == 1 && ids.stride(0) >= 1;
  TORCH_CHECK(contiguous || strided, "topk_ids must be contiguous [T, topk] (or a strided [T, 1] view)");
  TORCH_CHECK(is_int(ids) || ids.scalar_type() == at::kLong, "topk_ids must be int32 or int64");
  TORCH_CHECK(1 <= E && E <= 4096, "num_local_experts must be in [1, 4096], got ", E);
  TORCH_CHECK(cap >= 1, "cap must be positive");
  TORCH_CHECK(E * cap < (1LL << 31), "E * cap must fit int32");
  const int64_t T = ids.size(0), topk = ids.size(1);
  TORCH_CHECK(T * topk < (1LL << 31), "T * topk must fit int32");
  Tensor counts = empty_on(ids, {E}, at::kInt);
  Tensor route_dest = empty_on(ids, {T, topk}, at::kInt);
  Tensor src_tok = empty_on(ids, {E * cap}, at::kInt);
  Tensor src_route = empty_on(ids, {E * cap}, at::kInt);
  const int64_t n_scratch = pnv_dispatch_plan_scratch_ints(T * topk, (int)E);
  Tensor scratch;
  if (n_scratch > 0) scratch = empty_on(ids, {n_scratch}, at::kInt);
  const c10::cuda::CUDAGuard guard(ids.device());
  check_rc(pnv_dispatch_plan_strided(ids.const_data_ptr(), is_int(ids) ? 0 : 1, strided ? ids.stride(0) : 1, T, (int)topk,
                                     (int)first_expert, (int)E, (int)cap, counts.mutable_data_ptr<int32_t>(),
                                     route_dest.mutable_data_ptr<int32_t>(), src_tok.mutable_data_ptr<int32_t>(),
                                     src_route.mutable_data_ptr<int32_t>(),
                                     scratch.defined() ? scratch.mutable_data_ptr<int32_t>() : nullptr, current_stream(ids)));
  return {counts, route_dest, src_tok, src_route};
}

void check_slots(const Tensor& src_tok, int64_t slots, const char* what) {
  TORCH_CHECK(is_int(src_tok) && src_tok.is_contiguous() && src_tok.numel() == slots, what);
}

// csrc/ops.cu:418-468
std::tuple<Tensor, Tensor> scatter_quant_act_planned(const Tensor& a1, const Tensor& src_tok, const Tensor& src_route,
                                                     const optional<Tensor>& topk_weights, const Tensor& gscale,
                                                     const Tensor& counts, int64_t cap) {
  TORCH_CHECK(a1.is_cuda() && src_tok.is_cuda() && src_route.is_cuda() && gscale.is_cuda() && counts.is_cuda(), "inputs must be CUDA");
  check_arch(a1);
  TORCH_CHECK(a1.dim() == 2, "a1 must be [T, K] (token-order hidden states)");
  TORCH_CHECK(is_bf16(a1) && a1.is_contiguous(), "a1 must be contiguous bf16");
  const int64_t K = a1.size(1);
  TORCH_CHECK(K % kSfBlock == 0, "K must be a multiple of ", kSfBlock, ", got ", K);
  const int64_t E = counts.numel();
  check_gscale_counts(gscale, counts, E);
  TORCH_CHECK(cap > 0, "cap must be positive");
  const char* plan_msg = "src_tok and src_route must be contiguous int32 [E * cap] (dispatch_plan output)";
  check_slots(src_tok, E * cap, plan_msg);
  check_slots(src_route, E * cap, plan_msg);
  const float* w = nullptr;
  if (topk_weights.has_value()) {
    TORCH_CHECK(topk_weights->is_cuda() && is_float(*topk_weights) && topk_weights->is_contiguous(),
                "topk_weights must be contiguous float32 [T * topk]");
    w = f32(*topk_weights);
  }
  Tensor b_act = empty_on(a1, {E, cap, K / 2}, at::kByte);
  Tensor sfb = empty_on(a1, {pnv_sf_numel((int)cap, (int)K, (int)E)}, at::kByte);
  const c10::cuda::CUDAGuard guard(a1.device());
  check_rc(pnv_scatter_quant_act_planned(a1.const_data_ptr(), i32(src_tok), i32(src_route), w, f32(gscale), gscale.numel() == E,
                                         i32(counts), (int)K, (int)E, (int)cap, b_act.mutable_data_ptr<uint8_t>(),
                                         sfb.mutable_data_ptr<uint8_t>(), sm_count(a1), current_stream(a1)));
  return {b_act, sfb};
}

// csrc/ops.cu:476-500
std::tuple<Tensor, Tensor> quant_rows(const Tensor& x, const Tensor& gscale) {
  TORCH_CHECK(x.is_cuda() && gscale.is_cuda(), "inputs must be CUDA");
  check_arch(x);
  TORCH_CHECK(x.dim() == 2 && is_bf16(x) && x.is_contiguous(), "x must be contiguous bf16 [T, K]");
  const int64_t T = x.size(0), K = x.size(1);
  TORCH_CHECK(K % kSfBlock == 0, "K must be a multiple of ", kSfBlock, ", got ", K);
  TORCH_CHECK(is_float(gscale) && gscale.numel() >= 1, "gscale must be float32 with the shared global scale first");
  Tensor q = empty_on(x, {T, K / 2}, at::kByte);
  Tensor sf = empty_on(x, {T, K / kSfBlock}, at::kByte);
  const c10::cuda::CUDAGuard guard(x.device());
  check_rc(pnv_quant_rows(x.const_data_ptr(), f32(gscale), T, (int)K, q.mutable_data_ptr<uint8_t>(), sf.mutable_data_ptr<uint8_t>(),
                          sm_count(x), current_stream(x)));
  return {q, sf};
}

// csrc/ops.cu:502-541
std::tuple<Tensor, Tensor> scatter_fp4_planned(const Tensor& q, const Tensor& q_sf, const Tensor& src_tok, const Tensor& counts, int64_t cap) {
  TORCH_CHECK(q.is_cuda() && q_sf.is_cuda() && src_tok.is_cuda() && counts.is_cuda(), "inputs must be CUDA");
  check_arch(q);
  TORCH_CHECK(q.dim() == 2 && is_byte(q) && q.is_contiguous(), "q must be contiguous uint8 [T, K/2] (quant_rows output)");
  const int64_t K = q.size(1) * 2;
  TORCH_CHECK(K % kSfBlock == 0, "K must be a multiple of ", kSfBlock, ", got ", K);
  TORCH_CHECK(q_sf.dim() == 2 && q_sf.size(0) == q.size(0) && q_sf.size(1) == K / kSfBlock && q_sf.element_size() == 1 && q_sf.is_contiguous(),
              "q_sf must be contiguous 1-byte [T, K/", kSfBlock, "] (quant_rows output)");
  const int64_t E = counts.numel();
  TORCH_CHECK(is_int(counts) && counts.is_contiguous(), "expert_num_tokens must be contiguous int32 [E]");
  TORCH_CHECK(cap > 0, "cap must be positive");
  check_slots(src_tok, E * cap, "src_tok must be contiguous int32 [E * cap] (dispatch_plan output)");
  Tensor b_act = empty_on(q, {E, cap, K / 2}, at::kByte);
  Tensor sfb = empty_on(q, {pnv_sf_numel((int)cap, (int)K, (int)E)}, at::kByte);
  const c10::cuda::CUDAGuard guard(q.device());
  check_rc(pnv_scatter_fp4_planned(u8(q), u8(q_sf), i32(src_tok), i32(counts), (int)K, (int)E, (int)cap,
                                   b_act.mutable_data_ptr<uint8_t>(), sfb.mutable_data_ptr<uint8_t>(), sm_count(q), current_stream(q)));
  return {b_act, sfb};
}

// ---- wire rows of the expert-parallel dispatch ---------------------------------------------------------

struct PackArgs { int64_t K, ranks; };

PackArgs check_pack_args(const Tensor& q, const Tensor& q_sf, const Tensor& ids, const Tensor& slot_tok, const Tensor& slot_route,
                         const Tensor& slab_counts, int64_t slab, int64_t experts_per_rank) {
  TORCH_CHECK(q.is_cuda() && q_sf.is_cuda() && ids.is_cuda() && slot_tok.is_cuda() && slot_route.is_cuda() && slab_counts.is_cuda(),
              "inputs must be CUDA");
  check_arch(q);
  TORCH_CHECK(q.dim() == 2 && is_byte(q) && q.is_contiguous(), "q must be contiguous uint8 [T, K/2]");
  const int64_t K = q.size(1) * 2;
  TORCH_CHECK(K % kSfBlock == 0, "K must be a multiple of ", kSfBlock, ", got ", K);
  TORCH_CHECK(q_sf.dim() == 2 && q_sf.size(0) == q.size(0) && q_sf.size(1) == K / kSfBlock && q_sf.element_size() == 1 && q_sf.is_contiguous(),
              "q_sf must be contiguous 1-byte [T, K/", kSfBlock, "]");
  TORCH_CHECK((is_int(ids) || ids.scalar_type() == at::kLong) && ids.is_contiguous(), "topk_ids must be contiguous int32/int64");
  const int64_t ranks = slab_counts.numel();
  TORCH_CHECK(is_int(slab_counts) && slab_counts.is_contiguous(), "slab_counts must be contiguous int32 [ranks]");
  TORCH_CHECK(slab >= 1 && experts_per_rank >= 1, "slab and experts_per_rank must be positive");
  TORCH_CHECK(is_int(slot_tok) && is_int(slot_route) && slot_tok.is_contiguous() && slot_route.is_contiguous() &&
                  slot_tok.numel() == ranks * slab && slot_route.numel() == ranks * slab,
              "slot_tok and slot_route must be contiguous int32 [ranks * slab] (dispatch_plan output)");
  return {K, ranks};
}

// Device pointers of an output spread over several buffers (each part [rows, width] of dtype).
std::vector<void*> part_pointers(at::TensorList parts, int64_t rows, int64_t width, at::ScalarType dtype, const char* what) {
  TORCH_CHECK(parts.size() >= 1 && parts.size() <= 16, what, ": between 1 and 16 parts, got ", parts.size());
  std::vector<void*> ptrs;
  ptrs.reserve(parts.size());
  for (const Tensor& t : parts) {
    TORCH_CHECK(t.is_cuda() && t.scalar_type() == dtype && t.dim() == 2 && t.is_contiguous() && t.size(0) == rows && t.size(1) == width,
                what, ": every part must be contiguous CUDA ", dtype, " [", rows, ", ", width, "]");
    ptrs.push_back(t.data_ptr());
  }
  return ptrs;
}

Tensor pack_wire_rows(const Tensor& q, const Tensor& q_sf, const Tensor& ids, const Tensor& slot_tok, const Tensor& slot_route,
                      const Tensor& slab_counts, int64_t slab, int64_t experts_per_rank) {
  const PackArgs a = check_pack_args(q, q_sf, ids, slot_tok, slot_route, slab_counts, slab, experts_per_rank);
  Tensor wire = empty_on(q, {a.ranks * slab, pnv_wire_row_bytes((int)a.K)}, at::kByte);
  const c10::cuda::CUDAGuard guard(q.device());
  check_rc(pnv_pack_wire_rows(u8(q), u8(q_sf), ids.const_data_ptr(), is_int(ids) ? 0 : 1, i32(slot_tok), i32(slot_route),
                              i32(slab_counts), (int)a.ranks, (int)slab, (int)experts_per_rank, (int)a.K,
                              wire.mutable_data_ptr<uint8_t>(), current_stream(q)));
  return wire;
}

void pack_wire_rows_parts(const Tensor& q, const Tensor& q_sf, const Tensor& ids, const Tensor& slot_tok, const Tensor& slot_route,
                          const Tensor& slab_counts, int64_t slab, int64_t experts_per_rank, at::TensorList wire_parts) {
  const PackArgs a = check_pack_args(q, q_sf, ids, slot_tok, slot_route, slab_counts, slab, experts_per_rank);
  TORCH_CHECK((int64_t)wire_parts.size() == a.ranks, "one wire part per destination rank: ", a.ranks, ", got ", wire_parts.size());
  std::vector<void*> parts = part_pointers(wire_parts, slab, pnv_wire_row_bytes((int)a.K), at::kByte, "pack_wire_rows_parts");
  const c10::cuda::CUDAGuard guard(q.device());
  check_rc(pnv_pack_wire_rows_parts(u8(q), u8(q_sf), ids.const_data_ptr(), is_int(ids) ? 0 : 1, i32(slot_tok), i32(slot_route),
                                    i32(slab_counts), (int)a.ranks, (int)slab, (int)experts_per_rank, (int)a.K, parts.data(),
                                    current_stream(q)));
}

std::tuple<Tensor, Tensor> scatter_fp4_wire(const Tensor& wire, int64_t K, const Tensor& src_tok, const Tensor& counts, int64_t cap) {
  TORCH_CHECK(wire.is_cuda() && src_tok.is_cuda() && counts.is_cuda(), "inputs must be CUDA");
  check_arch(wire);
  TORCH_CHECK(K % kSfBlock == 0, "K must be a multiple of ", kSfBlock, ", got ", K);
  TORCH_CHECK(wire.dim() == 2 && is_byte(wire) && wire.is_contiguous() && wire.size(1) == pnv_wire_row_bytes((int)K),
              "wire must be contiguous uint8 [rows, wire_row_bytes(K)]");
  const int64_t E = counts.numel();
  TORCH_CHECK(is_int(counts) && counts.is_contiguous(), "expert_num_tokens must be contiguous int32 [E]");
  TORCH_CHECK(cap > 0, "cap must be positive");
  check_slots(src_tok, E * cap, "src_tok must be contiguous int32 [E * cap] (dispatch_plan output)");
  Tensor b_act = empty_on(wire, {E, cap, K / 2}, at::kByte);
  Tensor sfb = empty_on(wire, {pnv_sf_numel((int)cap, (int)K, (int)E)}, at::kByte);
  const c10::cuda::CUDAGuard guard(wire.device());
  check_rc(pnv_scatter_fp4_wire(u8(wire), i32(src_tok), i32(counts), (int)K, (int)E, (int)cap, b_act.mutable_data_ptr<uint8_t>(),
                                sfb.mutable_data_ptr<uint8_t>(), sm_count(wire), current_stream(wire)));
  return {b_act, sfb};
}

// ---- combine, row copies, activation -------------------------------------------------------------------

// csrc/ops.cu:548-575; mutates `out` in place
void moe_finalize(const Tensor& out, const Tensor& fused, const Tensor& route_dest, const optional<Tensor>& topk_weights) {
  TORCH_CHECK(out.is_cuda() && fused.is_cuda() && route_dest.is_cuda(), "inputs must be CUDA");
  TORCH_CHECK(out.dim() == 2 && is_bf16(out) && out.is_contiguous(), "out must be contiguous bf16 [T, K]");
  TORCH_CHECK(is_bf16(fused) && fused.is_contiguous() && fused.dim() >= 2, "fused must be contiguous bf16 [E, cap, K] (or [E * cap, K])");
  const int64_t T = out.size(0), K = out.size(1);
  TORCH_CHECK(fused.size(-1) == K, "fused and out must share K");
  TORCH_CHECK(K % 8 == 0, "K must be a multiple of 8");
  TORCH_CHECK(is_int(route_dest) && route_dest.is_contiguous() && route_dest.dim() == 2 && route_dest.size(0) == T,
              "route_dest must be contiguous int32 [T, topk] (dispatch_plan output)");
  const int64_t topk = route_dest.size(1);
  const float* w = nullptr;
  if (topk_weights.has_value()) {
    TORCH_CHECK(topk_weights->is_cuda() && is_float(*topk_weights) && topk_weights->is_contiguous() && topk_weights->numel() == T * topk,
                "topk_weights must be contiguous float32 [T, topk]");
    w = f32(*topk_weights);
  }
  const c10::cuda::CUDAGuard guard(out.device());
  check_rc(pnv_moe_finalize(out.data_ptr(), fused.const_data_ptr(), i32(route_dest), w, T, (int)topk, (int)K, current_stream(out)));
}

// dst[i] = src[idx[i]] for idx[i] >= 0, a zero row otherwise
Tensor gather_rows(const Tensor& src, const Tensor& idx) {
  TORCH_CHECK(src.is_cuda() && idx.is_cuda(), "inputs must be CUDA");
  TORCH_CHECK(src.dim() == 2 && src.is_contiguous(), "src must be contiguous [rows, width]");
  TORCH_CHECK(is_int(idx) && idx.is_contiguous() && idx.dim() == 1, "idx must be contiguous int32 [n]");
  const int64_t row_bytes = src.size(1) * src.element_size();
  TORCH_CHECK(row_bytes % 16 == 0, "rows must be a multiple of 16 bytes, got ", row_bytes);
  Tensor dst = empty_on(src, {idx.numel(), src.size(1)}, src.scalar_type());
  const c10::cuda::CUDAGuard guard(src.device());
  check_rc(pnv_gather_rows(src.const_data_ptr(), i32(idx), idx.numel(), row_bytes, dst.data_ptr(), current_stream(src)));
  return dst;
}

// dst[i] = 0 where flags[i] < 0; the other rows are left alone
void zero_rows(const Tensor& dst, const Tensor& flags) {
  TORCH_CHECK(dst.is_cuda() && flags.is_cuda(), "inputs must be CUDA");
  TORCH_CHECK(dst.dim() == 2 && dst.is_contiguous(), "dst must be contiguous [rows, width]");
  TORCH_CHECK(is_int(flags) && flags.is_contiguous() && flags.numel() == dst.size(0), "flags must be contiguous int32 [rows]");
  const int64_t row_bytes = dst.size(1) * dst.element_size();
  TORCH_CHECK(row_bytes % 16 == 0, "rows must be a multiple of 16 bytes, got ", row_bytes);
  const c10::cuda::CUDAGuard guard(dst.device());
  check_rc(pnv_zero_rows(dst.data_ptr(), i32(flags), dst.size(0), row_bytes, current_stream(dst)));
}

// zero_rows over a parts table: flags [parts * rows]; row q is row q % rows of parts[q / rows]
void zero_rows_parts(at::TensorList parts, const Tensor& flags) {
  TORCH_CHECK(parts.size() >= 1 && flags.is_cuda(), "inputs must be CUDA");
  const int64_t rows = parts[0].size(0), width = parts[0].size(1);
  std::vector<void*> ptrs = part_pointers(parts, rows, width, parts[0].scalar_type(), "zero_rows_parts");
  TORCH_CHECK(is_int(flags) && flags.is_contiguous() && flags.numel() == (int64_t)parts.size() * rows,
              "flags must be contiguous int32 [parts * rows]");
  const int64_t row_bytes = width * parts[0].element_size();
  TORCH_CHECK(row_bytes % 16 == 0, "rows must be a multiple of 16 bytes, got ", row_bytes);
  const c10::cuda::CUDAGuard guard(flags.device());
  check_rc(pnv_zero_rows_parts(ptrs.data(), (int)parts.size(), rows, i32(flags), row_bytes, current_stream(flags)));
}

// The unfused gated activation (gated_act, csrc/layout.cuh:204-216): bf16 [..., 2N] -> [..., N]
Tensor gated_act(const Tensor& x2, bool interleaved, c10::string_view activation, double beta, double linear_beta) {
  TORCH_CHECK(x2.is_cuda() && is_bf16(x2) && x2.is_contiguous(), "x2 must be contiguous CUDA bf16");
  const int64_t N = x2.size(-1) / 2;
  TORCH_CHECK(N % kSfBlock == 0, "intermediate width N must be a multiple of ", kSfBlock, ", got ", N);
  const int kind = act_kind(activation, beta);
  std::vector<int64_t> sizes = x2.sizes().vec();
  sizes.back() = N;
  Tensor y = empty_on(x2, sizes, at::kBFloat16);
  const c10::cuda::CUDAGuard guard(x2.device());
  check_rc(pnv_gated_act(x2.const_data_ptr(), N ? x2.numel() / (2 * N) : 0, (int)N, interleaved ? 1 : 0, kind, (float)beta,
                         (float)linear_beta, y.data_ptr(), current_stream(x2)));
  return y;
}

// ---- grouped GEMM --------------------------------------------------------------------------------------

// Split-K workspaces (the reference allocates its workspace inside the op as well, csrc/group_mm.cuh:163-165).  One is
// kept per (device, stream, size); the counters are zeroed when a workspace is made and every launch leaves them zero.
// Launches with another number of counters get a workspace of their own: the partial sums follow the counters, so in a
// shared one a launch would leave its sums where the other's counters are.
// The list is short and least recently used entries go back to the caching allocator; a workspace is allocated with its
// stream current, so what the allocator does with a returned one is ordered after the launches that used it.
// While the stream is being captured nothing is kept: the call makes a workspace in the capture's memory pool, zeroes its
// counters inside the graph and gives it back when it returns, like any temporary of the captured program, so a graph never
// shares a buffer with work outside it and holds no memory that outlives it.
struct Workspace {
  int device;
  cudaStream_t stream;
  int64_t counters, bytes;
  Tensor buf;
};
constexpr size_t kMaxWorkspaces = 32;

Tensor new_workspace(const Tensor& t, cudaStream_t stream, int64_t counters, int64_t bytes) {
  Tensor buf = empty_on(t, {bytes}, at::kByte);
  TORCH_CHECK(cudaMemsetAsync(buf.data_ptr(), 0, (size_t)counters, stream) == cudaSuccess, "cudaMemsetAsync failed");
  return buf;
}

Tensor split_workspace(const Tensor& t, cudaStream_t stream, int64_t experts, int64_t features, int64_t k, int64_t max_n, int64_t* bytes) {
  static std::mutex mu;
  static std::list<Workspace>* pool = new std::list<Workspace>;      // never destroyed: tensors must not outlive CUDA at exit
  const int sms = sm_count(t);
  // (a K too short to be split needs none: in a captured decode step the clearing of its counters was a node of its own
  // between two GEMMs and kept the second from starting early: 101.0 -> 99.3 us for 128 tokens on 32 experts)
  *bytes = k < PNV_SPLIT_MIN_K ? 0 : pnv_group_mm_workspace_bytes((int)experts, (int)features, (int)max_n, sms);
  if (*bytes == 0) return Tensor();
  // the counters, one per (expert, 128 features), come first and are the only part that has to start at zero
  const int64_t counters = std::min<int64_t>(*bytes, ceil_div(experts * ceil_div(features, 128) * 4, 256) * 256);
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  TORCH_CHECK(cudaStreamIsCapturing(stream, &status) == cudaSuccess, "cudaStreamIsCapturing failed");
  if (status != cudaStreamCaptureStatusNone) return new_workspace(t, stream, counters, *bytes);
  const int dev = t.get_device();
  std::lock_guard<std::mutex> lock(mu);
  for (auto it = pool->begin(); it != pool->end(); ++it) {
    if (it->device == dev && it->stream == stream && it->counters == counters && it->bytes == *bytes) {
      pool->splice(pool->begin(), *pool, it);
      return pool->front().buf;
    }
  }
  Tensor buf = new_workspace(t, stream, counters, *bytes);
  pool->push_front(Workspace{dev, stream, counters, *bytes, buf});
  if (pool->size() > kMaxWorkspaces) pool->pop_back();
  return buf;
}

struct GemmArgs { int64_t E, M, K, max_n; };

GemmArgs check_gemm_operands(const Tensor& a_comp, const Tensor& e_meta, const Tensor& sfa, const Tensor& b_act, const Tensor& sfb,
                             int64_t M, int64_t K, const char* mismatch) {
  const GemmArgs a{a_comp.size(0), M, K, b_act.size(1)};
  const Dims d = physical_dims(M, K);
  TORCH_CHECK(a_comp.size(1) == d.m_ac && a_comp.size(2) == d.k_ac / 2 && e_meta.size(1) == d.m_e && e_meta.size(2) == d.k_e,
              "a_comp / e_meta shapes do not match compress() output for features=", M, ", k=", K, mismatch);
  TORCH_CHECK(sfa.numel() >= pnv_sf_numel((int)M, (int)K, (int)a.E), "sfa is smaller than the SFA layout");
  TORCH_CHECK(sfb.numel() >= pnv_sf_numel((int)a.max_n, (int)K, (int)a.E), "sfb is smaller than the SFB layout");
  return a;
}

// out / out_parts: exactly one of them; row_map only with 2-D outputs (csrc/ops.cu:672-735)
void group_mm_impl(const Tensor* out, const at::TensorList* out_parts, const Tensor* row_map, const Tensor& a_comp, const Tensor& e_meta,
                   const Tensor& sfa, const Tensor& b_act, const Tensor& sfb, const Tensor& alphas, const Tensor& counts, int64_t M,
                   int64_t K, int64_t config_id, int64_t cluster_m, int64_t cluster_n) {
  TORCH_CHECK(a_comp.is_cuda() && e_meta.is_cuda() && sfa.is_cuda() && b_act.is_cuda() && sfb.is_cuda() && alphas.is_cuda() &&
                  counts.is_cuda() && (out == nullptr || out->is_cuda()), "all tensors must be CUDA");
  check_arch(b_act);
  TORCH_CHECK(b_act.dim() == 3 && a_comp.dim() == 3 && e_meta.dim() == 3, "b_act, a_comp and e_meta must be 3D");
  const int64_t E = a_comp.size(0), max_n = b_act.size(1);
  TORCH_CHECK(b_act.size(0) == E && e_meta.size(0) == E, "expert dim mismatch");
  std::vector<void*> parts;
  if (row_map == nullptr) {
    TORCH_CHECK(out->dim() == 3, "out must be 3D");
    TORCH_CHECK(out->size(0) == E, "expert dim mismatch");
    TORCH_CHECK(out->size(1) == max_n && out->size(2) == M, "out must be [E, max_n, features]");
  } else {
    TORCH_CHECK(row_map->is_cuda() && is_int(*row_map) && row_map->is_contiguous() && row_map->numel() == E * max_n,
                "row_map must be contiguous int32 [E * max_n]");
    if (out_parts == nullptr) {
      TORCH_CHECK(out->dim() == 2 && out->size(1) == M, "out must be [rows, features]");
    } else {
      TORCH_CHECK(out_parts->size() >= 1, "at least one output part");
      parts = part_pointers(*out_parts, (*out_parts)[0].size(0), M, at::kBFloat16, "group_mm_rows_parts");
    }
  }
  TORCH_CHECK(b_act.size(2) == K / 2, "b_act must be [E, max_n, K/2]");
  TORCH_CHECK(out == nullptr || is_bf16(*out), "out must be bf16");
  TORCH_CHECK(is_byte(a_comp) && is_byte(e_meta) && is_byte(b_act) && sfa.element_size() == 1 && sfb.element_size() == 1,
              "a_comp, e_meta and b_act must be uint8; sfa, sfb 1-byte");
  TORCH_CHECK(a_comp.is_contiguous() && e_meta.is_contiguous() && sfa.is_contiguous() && b_act.is_contiguous() && sfb.is_contiguous() &&
                  alphas.is_contiguous() && counts.is_contiguous() && (out == nullptr || out->is_contiguous()),
              "all group_mm tensors must be contiguous");
  TORCH_CHECK(is_float(alphas) && alphas.numel() == E, "alphas must be [E] float32");
  TORCH_CHECK(is_int(counts) && counts.numel() == E, "expert_num_tokens must be [E] int32 (real per-expert token counts, <= max_n)");
  check_gemm_operands(a_comp, e_meta, sfa, b_act, sfb, M, K, " (check the features / k arguments)");
  const c10::cuda::CUDAGuard guard(b_act.device());
  const cudaStream_t stream = current_stream(b_act);
  int64_t ws_bytes = 0;
  const Tensor ws = split_workspace(b_act, stream, E, M, K, max_n, &ws_bytes);
  void* ws_ptr = ws.defined() ? ws.data_ptr() : nullptr;
  const int e = (int)E, m = (int)M, k = (int)K, n = (int)max_n, cfg = (int)config_id, cm = (int)cluster_m, cn = (int)cluster_n;
  const int sms = sm_count(b_act);
  if (row_map == nullptr)
    check_rc(pnv_group_mm(out->data_ptr(), u8(a_comp), u8(e_meta), u8(sfa), u8(b_act), u8(sfb), f32(alphas), i32(counts), e, m, k, n,
                          cfg, cm, cn, sms, 1, ws_ptr, ws_bytes, stream));
  else if (out_parts == nullptr)
    check_rc(pnv_group_mm_rows(out->data_ptr(), i32(*row_map), u8(a_comp), u8(e_meta), u8(sfa), u8(b_act), u8(sfb), f32(alphas),
                               i32(counts), e, m, k, n, cfg, cm, cn, sms, 1, ws_ptr, ws_bytes, stream));
  else
    check_rc(pnv_group_mm_rows_parts(parts.data(), (int)parts.size(), (*out_parts)[0].size(0), i32(*row_map), u8(a_comp), u8(e_meta),
                                     u8(sfa), u8(b_act), u8(sfb), f32(alphas), i32(counts), e, m, k, n, cfg, cm, cn, sms, 1, ws_ptr,
                                     ws_bytes, stream));
}

void group_mm(const Tensor& out, const Tensor& a_comp, const Tensor& e_meta, const Tensor& sfa, const Tensor& b_act, const Tensor& sfb,
              const Tensor& alphas, const Tensor& counts, int64_t features, int64_t k, int64_t config_id, int64_t cluster_m, int64_t cluster_n) {
  group_mm_impl(&out, nullptr, nullptr, a_comp, e_meta, sfa, b_act, sfb, alphas, counts, features, k, config_id, cluster_m, cluster_n);
}

// group_mm whose token row (e, t) lands in row row_map[e * max_n + t] of out [rows, features] (skipped where negative)
void group_mm_rows(const Tensor& out, const Tensor& row_map, const Tensor& a_comp, const Tensor& e_meta, const Tensor& sfa,
                   const Tensor& b_act, const Tensor& sfb, const Tensor& alphas, const Tensor& counts, int64_t features, int64_t k,
                   int64_t config_id, int64_t cluster_m, int64_t cluster_n) {
  group_mm_impl(&out, nullptr, &row_map, a_comp, e_meta, sfa, b_act, sfb, alphas, counts, features, k, config_id, cluster_m, cluster_n);
}

// group_mm_rows whose logical output [parts * rows, features] is spread over out_parts (bf16 [rows, features] each,
// possibly other GPUs' memory opened in this process)
void group_mm_rows_parts(at::TensorList out_parts, const Tensor& row_map, const Tensor& a_comp, const Tensor& e_meta, const Tensor& sfa,
                         const Tensor& b_act, const Tensor& sfb, const Tensor& alphas, const Tensor& counts, int64_t features, int64_t k,
                         int64_t config_id, int64_t cluster_m, int64_t cluster_n) {
  group_mm_impl(nullptr, &out_parts, &row_map, a_comp, e_meta, sfa, b_act, sfb, alphas, counts, features, k, config_id, cluster_m, cluster_n);
}

// csrc/ops.cu:591-658: GEMM1 + gated activation + GEMM2's input quantization in one kernel; returns GEMM2's operands
// (b_act [E, max_n, N/2], sfb)
std::tuple<Tensor, Tensor> group_mm_swiglu_quant(const Tensor& a_comp, const Tensor& e_meta, const Tensor& sfa, const Tensor& b_act,
                                                 const Tensor& sfb, const Tensor& alphas, const Tensor& counts, const Tensor& gscale,
                                                 int64_t M, int64_t K, int64_t config_id, int64_t cluster_m, int64_t cluster_n,
                                                 c10::string_view activation, double beta, double linear_beta) {
  TORCH_CHECK(a_comp.is_cuda() && e_meta.is_cuda() && sfa.is_cuda() && b_act.is_cuda() && sfb.is_cuda() && alphas.is_cuda() &&
                  counts.is_cuda() && gscale.is_cuda(), "all tensors must be CUDA");
  check_arch(b_act);
  TORCH_CHECK(b_act.dim() == 3 && a_comp.dim() == 3 && e_meta.dim() == 3, "b_act, a_comp and e_meta must be 3D");
  const int64_t E = a_comp.size(0), max_n = b_act.size(1), N = M / 2;
  TORCH_CHECK(M % 128 == 0, "features (2N) must be a multiple of 128 (whole 64-row gate/up blocks per CTA), got ", M);
  TORCH_CHECK(b_act.size(0) == E && b_act.size(2) == K / 2, "b_act must be [E, max_n, K/2]");
  TORCH_CHECK(a_comp.is_contiguous() && e_meta.is_contiguous() && sfa.is_contiguous() && b_act.is_contiguous() && sfb.is_contiguous() &&
                  alphas.is_contiguous(), "inputs must be contiguous");
  TORCH_CHECK(is_float(alphas) && alphas.numel() == E, "alphas must be [E] float32");
  check_gscale_counts(gscale, counts, E);
  check_gemm_operands(a_comp, e_meta, sfa, b_act, sfb, M, K, "");
  const int kind = act_kind(activation, beta);
  Tensor b_out = empty_on(b_act, {E, max_n, N / 2}, at::kByte);
  Tensor sfb_out = empty_on(b_act, {pnv_sf_numel((int)max_n, (int)N, (int)E)}, at::kByte);
  const c10::cuda::CUDAGuard guard(b_act.device());
  const cudaStream_t stream = current_stream(b_act);
  int64_t ws_bytes = 0;
  const Tensor ws = split_workspace(b_act, stream, E, M, K, max_n, &ws_bytes);
  check_rc(pnv_group_mm_swiglu_quant(b_out.mutable_data_ptr<uint8_t>(), sfb_out.mutable_data_ptr<uint8_t>(), u8(a_comp), u8(e_meta),
                                     u8(sfa), u8(b_act), u8(sfb), f32(alphas), i32(counts), f32(gscale), gscale.numel() == E, (int)E,
                                     (int)M, (int)K, (int)max_n, (int)config_id, (int)cluster_m, (int)cluster_n, kind, (float)beta,
                                     (float)linear_beta, sm_count(b_act), 1, ws.defined() ? ws.data_ptr() : nullptr, ws_bytes, stream));
  return {b_out, sfb_out};
}

std::vector<std::string> group_mm_configs() {       // csrc/ops.cu:665-670
  std::vector<std::string> names;
  for (int i = 0; i < pnv_group_mm_num_configs(); ++i) names.emplace_back(pnv_group_mm_config_name(i));
  return names;
}

std::vector<std::string> group_mm_swiglu_configs() {      // csrc/ops.cu:585-589
  std::vector<std::string> names;
  for (int i = 0; i < pnv_group_mm_swiglu_num_configs(); ++i) names.emplace_back(pnv_group_mm_swiglu_config_name(i));
  return names;
}

}  // namespace

// Leave `n` SMs out of every persistent launch (see paired_nvfp4_kernels.ops.set_sm_margin).
extern "C" __attribute__((visibility("default"))) void pnv_torch_set_sm_margin(int n) { g_sm_margin.store(std::max(0, n)); }

// The torch this library was built for, looked up in the file by build.py.
extern "C" __attribute__((visibility("default"))) const char* pnv_torch_build_id() { return PNV_TORCH_BUILD_ID; }

#define PNV_GEMM_OPERANDS "Tensor a_comp, Tensor e_meta, Tensor sfa, Tensor b_act, Tensor sfb, Tensor alphas, Tensor expert_num_tokens, "
// the defaults are paired_nvfp4_kernels.DEFAULT_TACTIC
#define PNV_TACTIC "int config_id=0, int cluster_m=2, int cluster_n=1"

TORCH_LIBRARY(paired_nvfp4, m) {
  m.def("compress(Tensor w_packed, Tensor w_blockscale, int k) -> (Tensor, Tensor, Tensor)");
  m.def("quant_act(Tensor x, Tensor gscale, Tensor expert_num_tokens, int features) -> (Tensor, Tensor)");
  m.def("silu_mul_quant_act(Tensor x2, Tensor gscale, Tensor expert_num_tokens, int features, bool interleaved=False, "
        "str activation=\"silu\", float beta=1.0, float linear_beta=-1.0) -> (Tensor, Tensor)");
  m.def("scatter_quant_act(Tensor a1, Tensor flat_tok, Tensor dest_global, Tensor? topk_weights, Tensor gscale, "
        "Tensor expert_num_tokens, int cap) -> (Tensor, Tensor)");
  m.def("dispatch_plan(Tensor topk_ids, int first_expert, int num_local_experts, int cap) -> (Tensor, Tensor, Tensor, Tensor)");
  m.def("scatter_quant_act_planned(Tensor a1, Tensor src_tok, Tensor src_route, Tensor? topk_weights, Tensor gscale, "
        "Tensor expert_num_tokens, int cap) -> (Tensor, Tensor)");
  m.def("quant_rows(Tensor x, Tensor gscale) -> (Tensor, Tensor)");
  m.def("scatter_fp4_planned(Tensor q, Tensor q_sf, Tensor src_tok, Tensor expert_num_tokens, int cap) -> (Tensor, Tensor)");
  m.def("moe_finalize(Tensor(a!) out, Tensor fused, Tensor route_dest, Tensor? topk_weights) -> ()");
  m.def("gather_rows(Tensor src, Tensor idx) -> Tensor");
  m.def("pack_wire_rows(Tensor q, Tensor q_sf, Tensor topk_ids, Tensor slot_tok, Tensor slot_route, Tensor slab_counts, int slab, "
        "int experts_per_rank) -> Tensor");
  m.def("scatter_fp4_wire(Tensor wire, int k, Tensor src_tok, Tensor expert_num_tokens, int cap) -> (Tensor, Tensor)");
  m.def("group_mm(Tensor(a!) out, " PNV_GEMM_OPERANDS "int features, int k, " PNV_TACTIC ") -> ()");
  m.def("group_mm_rows(Tensor(a!) out, Tensor row_map, " PNV_GEMM_OPERANDS "int features, int k, " PNV_TACTIC ") -> ()");
  m.def("zero_rows(Tensor(a!) dst, Tensor flags) -> ()");
  m.def("group_mm_rows_parts(Tensor(a!)[] out_parts, Tensor row_map, " PNV_GEMM_OPERANDS "int features, int k, " PNV_TACTIC ") -> ()");
  m.def("zero_rows_parts(Tensor(a!)[] parts, Tensor flags) -> ()");
  m.def("pack_wire_rows_parts(Tensor q, Tensor q_sf, Tensor topk_ids, Tensor slot_tok, Tensor slot_route, Tensor slab_counts, "
        "int slab, int experts_per_rank, Tensor(a!)[] wire_parts) -> ()");
  m.def("group_mm_configs() -> str[]");
  m.def("group_mm_swiglu_quant(" PNV_GEMM_OPERANDS "Tensor gscale, int features, int k, " PNV_TACTIC
        ", str activation=\"silu\", float beta=1.0, float linear_beta=-1.0) -> (Tensor, Tensor)");
  m.def("group_mm_swiglu_configs() -> str[]");
  m.def("gated_act(Tensor x2, bool interleaved=False, str activation=\"silu\", float beta=1.0, float linear_beta=-1.0) -> Tensor");
}

// The operators whose results are whole numbers (codes, scales, plans) or that only write into their arguments ...
#define PNV_OPS_WITHOUT_FLOAT_RESULTS(X)                                                                               \
  X(compress) X(quant_act) X(silu_mul_quant_act) X(scatter_quant_act) X(dispatch_plan) X(scatter_quant_act_planned)     \
  X(quant_rows) X(scatter_fp4_planned) X(moe_finalize) X(pack_wire_rows) X(scatter_fp4_wire) X(group_mm)                \
  X(group_mm_rows) X(zero_rows) X(group_mm_rows_parts) X(zero_rows_parts) X(pack_wire_rows_parts)                       \
  X(group_mm_swiglu_quant)
// ... and those that return floating-point tensors
#define PNV_OPS_WITH_FLOAT_RESULTS(X) X(gather_rows) X(gated_act)

TORCH_LIBRARY_IMPL(paired_nvfp4, CUDA, m) {
#define PNV_IMPL(name) m.impl(#name, TORCH_FN(name));
  PNV_OPS_WITHOUT_FLOAT_RESULTS(PNV_IMPL)
  PNV_OPS_WITH_FLOAT_RESULTS(PNV_IMPL)
#undef PNV_IMPL
}

// There is no backward for these ops.  torch's autograd fallback says so by a node on every floating-point result of an
// input that requires grad, which warns in backward; it never touches integer results or written arguments, so the ops
// without floating-point results skip it (it is boxed: a microsecond or two a call).
TORCH_LIBRARY_IMPL(paired_nvfp4, AutogradCUDA, m) {
#define PNV_FALLTHROUGH(name) m.impl(#name, torch::CppFunction::makeFallthrough());
  PNV_OPS_WITHOUT_FLOAT_RESULTS(PNV_FALLTHROUGH)
#undef PNV_FALLTHROUGH
}

TORCH_LIBRARY_IMPL(paired_nvfp4, CompositeExplicitAutograd, m) {
  m.impl("group_mm_configs", TORCH_FN(group_mm_configs));
  m.impl("group_mm_swiglu_configs", TORCH_FN(group_mm_swiglu_configs));
}
