// Python extension module `agemm`: the operator surface of ARCQuant's torch extension
// (kernels/src/bindings.cpp:551-582) on top of libarcq.so's C ABI.  Same function names, argument
// order and return types for the four quantized-linear operators; outputs are allocated here with
// torch::empty, inputs are borrowed, kernels run on torch's current CUDA stream.  The reference's
// KV-cache operators (batch_decode_*, init_kv_*, append_kv_*) are not part of this library.
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include <sstream>
#include <stdexcept>
#include <tuple>

#include "arcq.h"

namespace {

// A status of the C side; in Python arcquant_b200._lib.ArcqError, as without the extension (a RuntimeError where this module is
// used without the package).
struct StatusError : std::runtime_error {
  StatusError(int status, const std::string& where, const std::string& text) : std::runtime_error(text), status(status), where(where) {}
  int status;
  std::string where;
};
void check_status(int status, const char* name) {
  if (status == ARCQ_OK) return;
  const std::string where = std::string("Value error in ") + name;
  std::ostringstream os;
  os << where << ": " << arcq_status_string(status);
  if (status == ARCQ_ERR_CUDA) os << " (cudaError " << arcq_last_cuda_error() << ")";
  throw StatusError(status, where, os.str());
}
void translate_status(std::exception_ptr e) {
  try {
    if (e) std::rethrow_exception(e);
  } catch (const StatusError& error) {
    try {
      const py::object type = py::module_::import("arcquant_b200._lib").attr("ArcqError");
      PyErr_SetObject(type.ptr(), type(error.status, error.where).ptr());
    } catch (py::error_already_set&) {
      PyErr_SetString(PyExc_RuntimeError, error.what());
    }
  }
}

void* current_stream(const torch::Tensor& t) {
  return static_cast<void*>(c10::cuda::getCurrentCUDAStream(t.device().index()).stream());
}

void require_cuda(const torch::Tensor& t, const char* name) {
  TORCH_CHECK(t.is_cuda(), name, " must be a CUDA tensor (this library has no CPU path)");
  TORCH_CHECK(t.is_contiguous(), name, " must be contiguous");
}
// Every tensor a kernel will dereference: on the device of `like`, contiguous, of the given type.
void require_on(const torch::Tensor& t, const torch::Tensor& like, at::ScalarType type, const char* name) {
  require_cuda(t, name);
  TORCH_CHECK(t.device() == like.device(), name, " must be on the same device as the first operand");
  TORCH_CHECK(t.scalar_type() == type, name, ": expected ", type, ", got ", t.scalar_type());
}
void require_scalar_f32(const torch::Tensor& t, const torch::Tensor& like, const char* name) {
  require_on(t, like, at::kFloat, name);
  TORCH_CHECK(t.numel() == 1, name, " must hold one fp32 value");
}
// An output on `like`'s device.  Straight from the CUDA allocator's factory: through torch::empty's dispatch an allocation costs the
// host about as much as a third of a launch, and a call makes two to five.  Through the dispatch all the same where somebody wants to see the
// allocation - a dispatch mode, a tracer, a functorch transform: their keys are in the thread's set - or torch is asked to fill it.
bool dispatch_allocations() {
  const auto& context = at::globalContext();
  return !(c10::impl::tls_local_dispatch_key_set().included_ - c10::default_included_set - c10::autocast_dispatch_keyset).empty() ||
         (context.deterministicAlgorithms() && context.deterministicFillUninitializedMemory());
}
torch::Tensor empty_on(const torch::Tensor& like, at::IntArrayRef sizes, at::ScalarType type) {
  if (dispatch_allocations()) return torch::empty(sizes, at::TensorOptions(type).device(like.device()));
  return torch::Tensor(at::detail::empty_cuda(sizes, type, like.device(), c10::nullopt));
}
// Shapes of a block-scaled GEMM's operands; returns M, N, K_eff.
std::tuple<int64_t, int64_t, int64_t> check_gemm_operands(const torch::Tensor& A, const torch::Tensor& B,
                                                          const torch::Tensor& SFA, const torch::Tensor& SFB) {
  require_cuda(A, "A");
  TORCH_CHECK(A.scalar_type() == at::kByte, "A: expected uint8 packed codes");
  require_on(B, A, at::kByte, "B");
  require_on(SFA, A, at::kByte, "SFA");
  require_on(SFB, A, at::kByte, "SFB");
  TORCH_CHECK(A.dim() == 2 && B.dim() == 2, "A and B must be 2-D [rows, K_eff/2]");
  TORCH_CHECK(A.size(1) == B.size(1), "A and B disagree on K");
  const int64_t M = A.size(0), N = B.size(0), K = A.size(1) * 2;
  // what the kernels read: whole 512-byte atoms of every 128-row tile
  const int64_t atoms = (K / 16 + 3) / 4;
  TORCH_CHECK(SFA.numel() >= ((M + 127) / 128) * atoms * 512, "SFA is smaller than the scale layout of A");
  TORCH_CHECK(SFB.numel() >= ((N + 127) / 128) * atoms * 512, "SFB is smaller than the scale layout of B");
  return std::make_tuple(M, N, K);
}

std::tuple<torch::Tensor, torch::Tensor> quantize_common(const torch::Tensor& X, const torch::Tensor* gamma,
                                                         float eps, const torch::Tensor& reorder_index, int KE,
                                                         bool is_weight, const char* where, const torch::Tensor* clear = nullptr) {
  require_cuda(X, "input");
  require_on(reorder_index, X, at::kShort, "reorder_index");
  TORCH_CHECK(X.dim() == 2, "input must be 2-D");
  const int64_t rows = X.size(0);
  const int KQ = static_cast<int>(X.size(1));
  const int K = KQ + KE;
  TORCH_CHECK(KE >= 0 && KE <= KQ, "KE must lie in [0, KQ]");
  TORCH_CHECK(reorder_index.numel() == KQ, "reorder_index must have KQ entries");
  c10::cuda::CUDAGuard guard(X.device());
  auto Q = empty_on(X, {rows, K / 2}, at::kByte);
  auto SF = empty_on(X, {static_cast<int64_t>(arcq_sf_bytes(rows, K))}, at::kByte);
  const void* px = X.data_ptr<at::BFloat16>();                 // throws on a wrong dtype, as the reference does
  const int16_t* pidx = reorder_index.data_ptr<int16_t>();
  int status;
  if (gamma) {
    require_on(*gamma, X, at::kBFloat16, "weight");
    TORCH_CHECK(gamma->numel() == KQ, "weight must have KQ entries");
    if (clear) require_on(*clear, X, at::kFloat, "clear");
    status = arcq_rmsnorm_quantize_x_clear(px, gamma->data_ptr<at::BFloat16>(), eps, pidx, rows, KQ, KE, Q.data_ptr<uint8_t>(),
                                           SF.data_ptr<uint8_t>(), clear ? clear->data_ptr<float>() : nullptr,
                                           clear ? static_cast<int>(clear->numel()) : 0, current_stream(X));
  } else if (is_weight) {
    status = arcq_reorder_quantize_w(px, pidx, rows, KQ, KE, arcq_reference_mode(KQ), Q.data_ptr<uint8_t>(),
                                     SF.data_ptr<uint8_t>(), current_stream(X));
  } else {
    status = arcq_reorder_quantize_x(px, pidx, rows, KQ, KE, arcq_reference_mode(KQ), Q.data_ptr<uint8_t>(),
                                     SF.data_ptr<uint8_t>(), current_stream(X));
  }
  check_status(status, where);
  return std::make_tuple(Q, SF);
}

torch::Tensor matmul(const torch::Tensor& A, const torch::Tensor& B, const torch::Tensor& SFA,
                     const torch::Tensor& SFB, const float scale) {
  int64_t M, N, K;
  std::tie(M, N, K) = check_gemm_operands(A, B, SFA, SFB);
  c10::cuda::CUDAGuard guard(A.device());
  auto C = empty_on(A, {M, N}, at::kBFloat16);
  int status = arcq_matmul_nvfp4_ws(A.data_ptr<uint8_t>(), B.data_ptr<uint8_t>(), SFA.data_ptr<uint8_t>(),
                                    SFB.data_ptr<uint8_t>(), M, N, K, scale, nullptr, nullptr,
                                    C.data_ptr<at::BFloat16>(), nullptr, 0, current_stream(A));
  check_status(status, "matmul_host_nvfp4_bf16");
  return C;
}

// Extra: alpha = alpha_a * alpha_b read on the device (0-dim fp32 CUDA tensors), no host sync.
torch::Tensor matmul_dev_alpha(const torch::Tensor& A, const torch::Tensor& B, const torch::Tensor& SFA,
                               const torch::Tensor& SFB, const torch::Tensor& alpha_a,
                               const c10::optional<torch::Tensor>& alpha_b, const c10::optional<torch::Tensor>& bias) {
  int64_t M, N, K;
  std::tie(M, N, K) = check_gemm_operands(A, B, SFA, SFB);
  require_scalar_f32(alpha_a, A, "alpha_a");
  if (alpha_b.has_value()) require_scalar_f32(*alpha_b, A, "alpha_b");
  c10::cuda::CUDAGuard guard(A.device());
  auto C = empty_on(A, {M, N}, at::kBFloat16);
  const float* pb = alpha_b.has_value() ? alpha_b->data_ptr<float>() : nullptr;
  int status;
  if (bias.has_value()) {
    TORCH_CHECK(bias->scalar_type() == torch::kBFloat16 && bias->is_contiguous() && bias->numel() == N &&
                bias->device() == A.device(), "bias must be a contiguous bf16 vector of N elements on A's device");
    status = arcq_matmul_nvfp4_bias(A.data_ptr<uint8_t>(), B.data_ptr<uint8_t>(), SFA.data_ptr<uint8_t>(),
                                    SFB.data_ptr<uint8_t>(), M, N, K, alpha_a.data_ptr<float>(), pb, bias->data_ptr(),
                                    C.data_ptr<at::BFloat16>(), current_stream(A));
  } else {
    status = arcq_matmul_nvfp4_dev_alpha(A.data_ptr<uint8_t>(), B.data_ptr<uint8_t>(), SFA.data_ptr<uint8_t>(),
                                         SFB.data_ptr<uint8_t>(), M, N, K, alpha_a.data_ptr<float>(), pb,
                                         C.data_ptr<at::BFloat16>(), current_stream(A));
  }
  check_status(status, "matmul_host_nvfp4_bf16");
  return C;
}

// Extra: residual [M, N] + the product, added in the GEMM's epilogue.
torch::Tensor matmul_residual(const torch::Tensor& A, const torch::Tensor& B, const torch::Tensor& SFA,
                              const torch::Tensor& SFB, const torch::Tensor& alpha_a,
                              const c10::optional<torch::Tensor>& alpha_b, const torch::Tensor& residual) {
  int64_t M, N, K;
  std::tie(M, N, K) = check_gemm_operands(A, B, SFA, SFB);
  require_scalar_f32(alpha_a, A, "alpha_a");
  if (alpha_b.has_value()) require_scalar_f32(*alpha_b, A, "alpha_b");
  TORCH_CHECK(residual.scalar_type() == torch::kBFloat16 && residual.is_contiguous() && residual.dim() == 2 &&
              residual.size(0) == M && residual.size(1) == N && residual.device() == A.device(),
              "residual must be a contiguous bf16 [M, N] tensor on A's device");
  c10::cuda::CUDAGuard guard(A.device());
  auto C = empty_on(A, {M, N}, at::kBFloat16);
  int status = arcq_matmul_nvfp4_residual(
      A.data_ptr<uint8_t>(), B.data_ptr<uint8_t>(), SFA.data_ptr<uint8_t>(), SFB.data_ptr<uint8_t>(), M, N, K,
      alpha_a.data_ptr<float>(), alpha_b.has_value() ? alpha_b->data_ptr<float>() : nullptr, residual.data_ptr(),
      C.data_ptr<at::BFloat16>(), current_stream(A));
  check_status(status, "matmul_residual");
  return C;
}

std::tuple<torch::Tensor, torch::Tensor> reorder_quantize_x(const torch::Tensor& X,
                                                            const torch::Tensor& reorder_index, const int KE) {
  return quantize_common(X, nullptr, 0.f, reorder_index, KE, false, "run_reorder_x_bf16_nvfp4");
}

std::tuple<torch::Tensor, torch::Tensor> reorder_quantize_w(const torch::Tensor& W,
                                                            const torch::Tensor& reorder_index, const int KE) {
  return quantize_common(W, nullptr, 0.f, reorder_index, KE, true, "run_reorder_w_bf16_nvfp4");
}

std::tuple<torch::Tensor, torch::Tensor> rmsnorm_quantize_x(const torch::Tensor& X, const torch::Tensor& W,
                                                            const float eps, const torch::Tensor& reorder_index,
                                                            const int KE, const c10::optional<torch::Tensor>& clear) {
  return quantize_common(X, &W, eps, reorder_index, KE, false, "run_rmsnorm_x_bf16_nvfp4", clear.has_value() ? &*clear : nullptr);
}

// ---- extras without a counterpart in the reference's bindings (its layers call torch for these) ----

// reorder_quantize_x on X / scale (scale: 0-dim fp32 CUDA tensor), the division fused into the kernel
// where the row width allows it, done with torch first where it does not.  mode < 0: the reference's
// choice for this KQ.
std::tuple<torch::Tensor, torch::Tensor> reorder_quantize_x_scaled(const torch::Tensor& X, const torch::Tensor& scale,
                                                                   const torch::Tensor& reorder_index, const int KE,
                                                                   int mode) {
  require_cuda(X, "input");
  require_on(reorder_index, X, at::kShort, "reorder_index");
  require_scalar_f32(scale, X, "scale");
  TORCH_CHECK(X.dim() == 2, "input must be 2-D");
  const int64_t rows = X.size(0);
  const int KQ = static_cast<int>(X.size(1));
  const int K = KQ + KE;
  TORCH_CHECK(KE >= 0 && KE <= KQ, "KE must lie in [0, KQ]");
  TORCH_CHECK(reorder_index.numel() == KQ, "reorder_index must have KQ entries");
  if (mode < 0) mode = arcq_reference_mode(KQ);
  c10::cuda::CUDAGuard guard(X.device());
  auto Q = empty_on(X, {rows, K / 2}, at::kByte);
  auto SF = empty_on(X, {static_cast<int64_t>(arcq_sf_bytes(rows, K))}, at::kByte);
  int status = arcq_reorder_quantize_x_scaled(X.data_ptr<at::BFloat16>(), scale.data_ptr<float>(),
                                              reorder_index.data_ptr<int16_t>(), rows, KQ, KE, mode,
                                              Q.data_ptr<uint8_t>(), SF.data_ptr<uint8_t>(), current_stream(X));
  if (status == ARCQ_ERR_UNSUPPORTED_K) {
    auto Xs = X / scale;
    status = arcq_reorder_quantize_x(Xs.data_ptr<at::BFloat16>(), reorder_index.data_ptr<int16_t>(), rows, KQ, KE, mode,
                                     Q.data_ptr<uint8_t>(), SF.data_ptr<uint8_t>(), current_stream(X));
  }
  check_status(status, "run_reorder_x_bf16_nvfp4");
  return std::make_tuple(Q, SF);
}

// (codes, scales, per-tensor scale): x or w divided by max / (448 * 6), then reordered and quantized; see
// arcq_quantize_tensor_scale.  amax: max|x| as a 0-dim fp32 CUDA tensor if the caller has it.
std::tuple<torch::Tensor, torch::Tensor, torch::Tensor> quantize_tensor_scale(const torch::Tensor& X,
                                                                              const torch::Tensor& reorder_index, const int KE,
                                                                              int mode, bool is_weight,
                                                                              const c10::optional<torch::Tensor>& amax) {
  require_cuda(X, "input");
  TORCH_CHECK(X.scalar_type() == at::kBFloat16, "input: expected bfloat16");
  require_on(reorder_index, X, at::kShort, "reorder_index");
  if (amax.has_value()) require_scalar_f32(*amax, X, "amax");
  TORCH_CHECK(X.dim() == 2, "input must be 2-D");
  const int64_t rows = X.size(0);
  const int KQ = static_cast<int>(X.size(1));
  const int K = KQ + KE;
  TORCH_CHECK(KE >= 0 && KE <= KQ, "KE must lie in [0, KQ]");
  TORCH_CHECK(reorder_index.numel() == KQ, "reorder_index must have KQ entries");
  if (mode < 0) mode = arcq_reference_mode(KQ);
  c10::cuda::CUDAGuard guard(X.device());
  auto Q = empty_on(X, {rows, K / 2}, at::kByte);
  auto SF = empty_on(X, {static_cast<int64_t>(arcq_sf_bytes(rows, K))}, at::kByte);
  auto scale = empty_on(X, {}, at::kFloat);
  torch::Tensor scratch;
  if (!amax.has_value()) scratch = empty_on(X, {ARCQ_SCALE_SCRATCH}, at::kFloat);
  check_status(arcq_quantize_tensor_scale(X.data_ptr(), amax.has_value() ? amax->data_ptr<float>() : nullptr, is_weight ? 1 : 0,
                                          reorder_index.data_ptr<int16_t>(), rows, KQ, KE, mode, Q.data_ptr<uint8_t>(),
                                          SF.data_ptr<uint8_t>(), scale.data_ptr<float>(),
                                          amax.has_value() ? nullptr : scratch.data_ptr<float>(), current_stream(X)),
               is_weight ? "run_reorder_w_bf16_nvfp4" : "run_reorder_x_bf16_nvfp4");
  return std::make_tuple(Q, SF, scale);
}

// A scale factor per matrix: `count` values at least, the kernels read one for each.
const float* factors(const torch::Tensor& t, const torch::Tensor& like, int64_t count, const char* name) {
  require_on(t, like, at::kFloat, name);
  TORCH_CHECK(t.numel() >= count, name, " must hold an fp32 value for every matrix");
  return t.data_ptr<float>();
}
const float* factors(const c10::optional<torch::Tensor>& t, const torch::Tensor& like, int64_t count, const char* name) {
  return t.has_value() ? factors(*t, like, count, name) : nullptr;
}

// Gate/up GEMM with the SwiGLU epilogue; see arcq_matmul_nvfp4_swiglu, and _onto for an amax that is zero already.
torch::Tensor swiglu(const torch::Tensor& A, const torch::Tensor& B, const torch::Tensor& SFA, const torch::Tensor& SFB,
                     const torch::Tensor& alpha_a, const c10::optional<torch::Tensor>& alpha_b, torch::Tensor& amax,
                     decltype(arcq_matmul_nvfp4_swiglu)* call) {
  int64_t M, N, K;
  std::tie(M, N, K) = check_gemm_operands(A, B, SFA, SFB);
  const float *aa = factors(alpha_a, A, 1, "alpha_a"), *ab = factors(alpha_b, A, 1, "alpha_b");
  TORCH_CHECK(N % 256 == 0, "N is not a multiple of 256");
  c10::cuda::CUDAGuard guard(A.device());
  auto C = empty_on(A, {M, N / 2}, at::kBFloat16);
  check_status(call(A.data_ptr<uint8_t>(), B.data_ptr<uint8_t>(), SFA.data_ptr<uint8_t>(), SFB.data_ptr<uint8_t>(), M, N, K, aa, ab,
                    C.data_ptr<at::BFloat16>(), amax.data_ptr<float>(), current_stream(A)),
               "swiglu matmul");
  return C;
}
std::tuple<torch::Tensor, torch::Tensor> matmul_swiglu(const torch::Tensor& A, const torch::Tensor& B, const torch::Tensor& SFA,
                                                       const torch::Tensor& SFB, const torch::Tensor& alpha_a,
                                                       const c10::optional<torch::Tensor>& alpha_b,
                                                       const c10::optional<torch::Tensor>& onto) {
  require_cuda(A, "A");
  if (onto.has_value()) factors(*onto, A, 1, "onto");
  auto amax = onto.has_value() ? *onto : empty_on(A, {}, at::kFloat);
  auto call = onto.has_value() ? arcq_matmul_nvfp4_swiglu_onto : arcq_matmul_nvfp4_swiglu;
  return std::make_tuple(swiglu(A, B, SFA, SFB, alpha_a, alpha_b, amax, call), amax);
}

// The grouped forms; groups: the run table [first rows | rows] of exactly these runs (in a table of more the row counts lie
// elsewhere, and the kernels would take first rows for them).
void check_grouped(const torch::Tensor& A, const torch::Tensor& B, const torch::Tensor& tile_group, const torch::Tensor& groups,
                   int64_t ngroups, int64_t n, const torch::Tensor& alpha_a) {
  require_on(tile_group, A, at::kInt, "tile_group");
  require_on(groups, A, at::kInt, "groups");
  TORCH_CHECK(ngroups > 0 && n > 0 && B.size(0) == ngroups * n && tile_group.numel() >= (A.size(0) + 255) / 256 &&
                  alpha_a.numel() == ngroups,
              "operand shapes disagree");
  TORCH_CHECK(groups.numel() == 2 * ngroups, "groups must hold 2 * ngroups entries");
}
std::tuple<torch::Tensor, torch::Tensor> matmul_grouped_swiglu(const torch::Tensor& A, const torch::Tensor& B, const torch::Tensor& SFA,
                                                               const torch::Tensor& SFB, const torch::Tensor& tile_group,
                                                               const torch::Tensor& groups, int64_t ngroups, int64_t n,
                                                               const torch::Tensor& alpha_a,
                                                               const c10::optional<torch::Tensor>& alpha_b,
                                                               const c10::optional<torch::Tensor>& onto) {
  int64_t M, N, K;
  std::tie(M, N, K) = check_gemm_operands(A, B, SFA, SFB);
  check_grouped(A, B, tile_group, groups, ngroups, n, alpha_a);
  const float *aa = factors(alpha_a, A, ngroups, "alpha_a"), *ab = factors(alpha_b, A, ngroups, "alpha_b");
  TORCH_CHECK(n % 256 == 0, "n is not a multiple of 256");
  if (onto.has_value()) factors(*onto, A, ngroups, "onto");
  c10::cuda::CUDAGuard guard(A.device());
  auto C = empty_on(A, {M, n / 2}, at::kBFloat16);
  auto amax = onto.has_value() ? *onto : empty_on(A, {ngroups}, at::kFloat);
  auto call = onto.has_value() ? arcq_matmul_nvfp4_grouped_swiglu_onto : arcq_matmul_nvfp4_grouped_swiglu;
  check_status(call(A.data_ptr<uint8_t>(), B.data_ptr<uint8_t>(), SFA.data_ptr<uint8_t>(), SFB.data_ptr<uint8_t>(), M, n, K,
                    tile_group.data_ptr<int32_t>(), groups.data_ptr<int32_t>(), static_cast<int>(ngroups), aa, ab,
                    C.data_ptr<at::BFloat16>(), amax.data_ptr<float>(), current_stream(A)),
               "grouped swiglu matmul");
  return std::make_tuple(C, amax);
}
torch::Tensor matmul_grouped_runs(const torch::Tensor& A, const torch::Tensor& B, const torch::Tensor& SFA, const torch::Tensor& SFB,
                                  const torch::Tensor& tile_group, const torch::Tensor& groups, int64_t ngroups, int64_t n,
                                  const torch::Tensor& alpha_a, const c10::optional<torch::Tensor>& alpha_b) {
  int64_t M, N, K;
  std::tie(M, N, K) = check_gemm_operands(A, B, SFA, SFB);
  check_grouped(A, B, tile_group, groups, ngroups, n, alpha_a);
  const float *aa = factors(alpha_a, A, ngroups, "alpha_a"), *ab = factors(alpha_b, A, ngroups, "alpha_b");
  c10::cuda::CUDAGuard guard(A.device());
  auto C = empty_on(A, {M, n}, at::kBFloat16);
  check_status(arcq_matmul_nvfp4_grouped_runs(A.data_ptr<uint8_t>(), B.data_ptr<uint8_t>(), SFA.data_ptr<uint8_t>(),
                                              SFB.data_ptr<uint8_t>(), M, n, K, tile_group.data_ptr<int32_t>(),
                                              groups.data_ptr<int32_t>(), static_cast<int>(ngroups), aa, ab,
                                              C.data_ptr<at::BFloat16>(), current_stream(A)),
               "grouped matmul");
  return C;
}

// Grouped rows quantized by their runs' maxima; see arcq_quantize_x_grouped_amax.
std::tuple<torch::Tensor, torch::Tensor, torch::Tensor> quantize_grouped_amax(const torch::Tensor& X, const c10::optional<torch::Tensor>& row_map,
                                                                              const torch::Tensor& amax, const torch::Tensor& indices,
                                                                              const torch::Tensor& groups, int64_t rows_bound, int KE,
                                                                              int mode, const c10::optional<torch::Tensor>& clear) {
  require_cuda(X, "input");
  TORCH_CHECK(X.scalar_type() == at::kBFloat16 && X.dim() >= 1, "input: expected bfloat16 rows");
  require_on(amax, X, at::kFloat, "amax");
  require_on(indices, X, at::kShort, "reorder_indices");
  require_on(groups, X, at::kInt, "groups");
  TORCH_CHECK(indices.dim() == 2, "reorder_indices must be [runs, KQ]");
  const int64_t ngroups = indices.size(0), KQ = indices.size(1);
  TORCH_CHECK(X.size(-1) == KQ && amax.numel() == ngroups && groups.numel() == 2 * ngroups,
              "reorder_indices / groups disagree on the number of runs or on KQ");
  if (row_map.has_value()) {
    require_on(*row_map, X, at::kInt, "row_map");
    TORCH_CHECK(row_map->numel() >= rows_bound, "row_map must cover rows_bound rows");
  } else {
    TORCH_CHECK(X.size(0) >= rows_bound, "input has fewer rows than rows_bound");
  }
  if (clear.has_value()) require_on(*clear, X, at::kFloat, "clear");
  c10::cuda::CUDAGuard guard(X.device());
  auto Q = empty_on(X, {rows_bound, (KQ + KE) / 2}, at::kByte);
  auto SF = empty_on(X, {static_cast<int64_t>(arcq_sf_bytes(rows_bound, KQ + KE))}, at::kByte);
  auto scale = empty_on(X, {ngroups}, at::kFloat);
  check_status(arcq_quantize_x_grouped_amax_clear(X.data_ptr(), row_map.has_value() ? row_map->data_ptr<int32_t>() : nullptr,
                                                  amax.data_ptr<float>(), indices.data_ptr<int16_t>(), groups.data_ptr<int32_t>(),
                                                  static_cast<int>(ngroups), rows_bound, static_cast<int>(KQ), KE, mode,
                                                  Q.data_ptr<uint8_t>(), SF.data_ptr<uint8_t>(), scale.data_ptr<float>(),
                                                  clear.has_value() ? clear->data_ptr<float>() : nullptr,
                                                  clear.has_value() ? static_cast<int>(clear->numel()) : 0, current_stream(X)),
               "grouped x-quantize");
  return std::make_tuple(Q, SF, scale);
}

// One batch of calibration statistics, accumulated in place; see arcq_calib_stats_bf16.
void calib_stats(const torch::Tensor& X, const torch::Tensor& chan_absmax, const c10::optional<torch::Tensor>& above) {
  require_cuda(X, "input");
  TORCH_CHECK(X.scalar_type() == at::kBFloat16, "input: expected bfloat16");
  require_on(chan_absmax, X, at::kFloat, "chan_absmax");
  const int64_t K = X.size(-1);
  TORCH_CHECK(chan_absmax.numel() == K, "chan_absmax must have one entry per channel");
  if (above.has_value()) require_on(*above, X, at::kLong, "above");
  c10::cuda::CUDAGuard guard(X.device());
  check_status(arcq_calib_stats_bf16(X.data_ptr(), K ? X.numel() / K : 0, static_cast<int>(K), chan_absmax.data_ptr<float>(),
                                     above.has_value() ? reinterpret_cast<unsigned long long*>(above->data_ptr<int64_t>()) : nullptr,
                                     current_stream(X)),
               "calib_stats");
}

// Channels by ascending statistic; see arcq_channel_order.
torch::Tensor channel_order(const torch::Tensor& value) {
  require_on(value, value, at::kFloat, "value");
  TORCH_CHECK(value.numel() <= 32768, "value has more channels than an int16 order can hold");
  c10::cuda::CUDAGuard guard(value.device());
  auto order = empty_on(value, {value.numel()}, at::kShort);
  if (value.numel() == 0) return order;
  check_status(arcq_channel_order(value.data_ptr<float>(), static_cast<int>(value.numel()), order.data_ptr<int16_t>(), current_stream(value)),
               "channel_order");
  return order;
}

std::tuple<torch::Tensor, torch::Tensor> silu_mul(const torch::Tensor& GU) {
  require_cuda(GU, "gate_up");
  TORCH_CHECK(GU.dim() == 2 && GU.size(1) % 16 == 0, "gate_up must be [tokens, 2F] with F a multiple of 8");
  c10::cuda::CUDAGuard guard(GU.device());
  const int64_t tokens = GU.size(0);
  const int F = static_cast<int>(GU.size(1) / 2);
  auto out = empty_on(GU, {tokens, F}, at::kBFloat16);
  auto amax = empty_on(GU, {}, at::kFloat);
  check_status(arcq_silu_mul_bf16(GU.data_ptr<at::BFloat16>(), out.data_ptr<at::BFloat16>(), tokens, F,
                                  amax.data_ptr<float>(), current_stream(GU)),
               "silu_mul");
  return std::make_tuple(out, amax);
}

torch::Tensor rope_inplace(torch::Tensor X, const torch::Tensor& cos_t, const torch::Tensor& sin_t, int heads,
                           int head_dim) {
  require_cuda(X, "x");
  require_on(cos_t, X, at::kFloat, "cos");
  require_on(sin_t, X, at::kFloat, "sin");
  TORCH_CHECK(X.dim() == 2 && cos_t.dim() == 2 && cos_t.size(1) == head_dim && cos_t.sizes() == sin_t.sizes(),
              "x must be [tokens, row]; cos / sin [seq, head_dim]");
  c10::cuda::CUDAGuard guard(X.device());
  check_status(arcq_rope_bf16(X.data_ptr<at::BFloat16>(), cos_t.data_ptr<float>(), sin_t.data_ptr<float>(), X.size(0),
                              static_cast<int>(X.size(1)), heads, head_dim, static_cast<int>(cos_t.size(0)),
                              current_stream(X)),
               "rope");
  return X;
}

torch::Tensor absmax(const torch::Tensor& X) {
  require_cuda(X, "input");
  c10::cuda::CUDAGuard guard(X.device());
  auto out = empty_on(X, {}, at::kFloat);
  check_status(arcq_absmax_bf16(X.data_ptr<at::BFloat16>(), X.numel(), out.data_ptr<float>(), 0, current_stream(X)),
               "absmax");
  return out;
}

// A quantized linear's forward: `matmul_dev_alpha` with a bias, the result as [bsz, q_len, N] or [q_len, N].
torch::Tensor linear(const torch::Tensor& A, const torch::Tensor& B, const torch::Tensor& SFA, const torch::Tensor& SFB,
                     const torch::Tensor& alpha_a, const torch::Tensor& alpha_b, const c10::optional<torch::Tensor>& bias,
                     const c10::optional<int64_t>& bsz, int64_t q_len) {
  auto C = matmul_dev_alpha(A, B, SFA, SFB, alpha_a, alpha_b, bias);
  if (bsz.has_value()) return C.reshape({*bsz, q_len, -1});
  return q_len > 0 && q_len == C.size(0) ? C : C.reshape({q_len, -1});
}

// The two halves of a decoder layer as the Python class of that name strings them together, operation for operation: one call each
// instead of a dozen, whose argument handling, views and attribute look-ups took longer than the kernels of a short prompt.
torch::Tensor attention_half(const torch::Tensor& X, const torch::Tensor& gain, double eps, const torch::Tensor& q_index, int q_ke,
                             const torch::Tensor& qkv_W, const torch::Tensor& qkv_SF, const torch::Tensor& qkv_scale,
                             const torch::Tensor& cos_t, const torch::Tensor& sin_t, int64_t heads, int64_t kv_heads, int64_t head_dim,
                             int64_t bsz, int64_t seq, const torch::Tensor& o_index, int o_ke, const torch::Tensor& o_W,
                             const torch::Tensor& o_SF, const torch::Tensor& o_scale, const c10::optional<torch::Tensor>& residual) {
  require_cuda(X, "x");
  TORCH_CHECK(X.dim() == 2 && X.size(0) == bsz * seq, "x must be [bsz * seq, hidden]");
  at::NoGradGuard no_grad;
  c10::cuda::CUDAGuard guard(X.device());
  torch::Tensor a, sfa, so;
  std::tie(a, sfa) = quantize_common(X, &gain, static_cast<float>(eps), q_index, q_ke, false, "run_rmsnorm_x_bf16_nvfp4");
  auto qkv = matmul_dev_alpha(a, qkv_W, sfa, qkv_SF, qkv_scale, c10::nullopt, c10::nullopt);
  const int64_t N = qkv.size(1);
  TORCH_CHECK(N == (heads + 2 * kv_heads) * head_dim, "the q/k/v projection does not hold these heads");
  rope_inplace(qkv, cos_t, sin_t, static_cast<int>(heads + kv_heads), static_cast<int>(head_dim));
  // [bsz, heads, seq, head_dim] views of the fused output; grouped-query heads are not materialised
  auto view = [&](int64_t n, int64_t at) { return qkv.as_strided({bsz, n, seq, head_dim}, {seq * N, head_dim, N, 1}, at); };
  auto attn = at::scaled_dot_product_attention(view(heads, 0), view(kv_heads, heads * head_dim), view(kv_heads, (heads + kv_heads) * head_dim),
                                               c10::nullopt, 0.0, true, c10::nullopt, heads != kv_heads);
  attn = attn.transpose(1, 2).reshape({bsz * seq, heads * head_dim}).contiguous();
  std::tie(a, sfa, so) = quantize_tensor_scale(attn, o_index, o_ke, ARCQ_MODE_16, false, c10::nullopt);
  return residual.has_value() ? matmul_residual(a, o_W, sfa, o_SF, so, o_scale, *residual)
                              : matmul_dev_alpha(a, o_W, sfa, o_SF, so, o_scale, c10::nullopt);
}
torch::Tensor mlp_half(const torch::Tensor& H, const torch::Tensor& gain, double eps, const torch::Tensor& up_index, int up_ke,
                       const torch::Tensor& gu_W, const torch::Tensor& gu_SF, const torch::Tensor& gu_scale,
                       const torch::Tensor& down_index, int down_ke, const torch::Tensor& down_W, const torch::Tensor& down_SF,
                       const torch::Tensor& down_scale, const c10::optional<torch::Tensor>& residual) {
  require_cuda(H, "h");
  at::NoGradGuard no_grad;
  c10::cuda::CUDAGuard guard(H.device());
  torch::Tensor a, sfa, act, amax, scale;
  amax = empty_on(H, {}, at::kFloat);                           // (cleared by the quantizer)
  std::tie(a, sfa) = quantize_common(H, &gain, static_cast<float>(eps), up_index, up_ke, false, "run_rmsnorm_x_bf16_nvfp4", &amax);
  act = swiglu(a, gu_W, sfa, gu_SF, gu_scale, c10::nullopt, amax, arcq_matmul_nvfp4_swiglu_onto);
  std::tie(a, sfa, scale) = quantize_tensor_scale(act, down_index, down_ke, ARCQ_MODE_16, false, amax);
  return residual.has_value() ? matmul_residual(a, down_W, sfa, down_SF, scale, down_scale, *residual)
                              : matmul_dev_alpha(a, down_W, sfa, down_SF, scale, down_scale, c10::nullopt);
}

// Routing and bookkeeping of a MoE block; see arcq_route_topk_bf16, arcq_moe_layout, arcq_absmax_grouped_bf16, arcq_moe_combine_bf16.
std::tuple<torch::Tensor, torch::Tensor> route_topk(const torch::Tensor& logits, int64_t top_k) {
  require_on(logits, logits, at::kBFloat16, "logits");
  TORCH_CHECK(logits.dim() == 2, "logits must be [tokens, experts]");
  c10::cuda::CUDAGuard guard(logits.device());
  const int64_t t = logits.size(0);
  auto ids = empty_on(logits, {t, top_k}, at::kLong);
  auto w = empty_on(logits, {t, top_k}, at::kBFloat16);
  check_status(arcq_route_topk_bf16(logits.data_ptr(), t, static_cast<int>(logits.size(1)), static_cast<int>(top_k),
                                    ids.data_ptr<int64_t>(), w.data_ptr(), current_stream(logits)),
               "route_topk");
  return std::make_tuple(ids, w);
}
std::tuple<torch::Tensor, torch::Tensor, torch::Tensor, torch::Tensor> moe_layout(const torch::Tensor& slot_group, int64_t ngroups,
                                                                                  int64_t tile, int64_t rows_bound, int64_t div) {
  require_on(slot_group, slot_group, at::kLong, "slot_group");
  TORCH_CHECK(tile > 0, "tile must be positive");
  c10::cuda::CUDAGuard guard(slot_group.device());
  const int64_t n = slot_group.numel();
  auto dest = empty_on(slot_group, {n}, at::kInt);
  auto row_map = empty_on(slot_group, {rows_bound}, at::kInt);
  auto groups = empty_on(slot_group, {2 * ngroups}, at::kInt);
  auto tile_group = empty_on(slot_group, {rows_bound / tile}, at::kInt);
  check_status(arcq_moe_layout(slot_group.data_ptr<int64_t>(), static_cast<int>(n), static_cast<int>(ngroups), static_cast<int>(tile),
                               static_cast<int>(rows_bound), static_cast<int>(div), dest.data_ptr<int32_t>(), row_map.data_ptr<int32_t>(),
                               groups.data_ptr<int32_t>(), tile_group.data_ptr<int32_t>(), current_stream(slot_group)),
               "moe_layout");
  return std::make_tuple(dest, row_map, groups, tile_group);
}
torch::Tensor absmax_grouped(const torch::Tensor& X, const c10::optional<torch::Tensor>& row_map, const torch::Tensor& groups,
                             int64_t ngroups) {
  require_on(X, X, at::kBFloat16, "input");
  require_on(groups, X, at::kInt, "groups");
  if (row_map.has_value()) require_on(*row_map, X, at::kInt, "row_map");
  TORCH_CHECK(groups.numel() == 2 * ngroups, "groups must hold 2 * ngroups entries");
  c10::cuda::CUDAGuard guard(X.device());
  auto out = empty_on(X, {ngroups}, at::kFloat);
  check_status(arcq_absmax_grouped_bf16(X.data_ptr(), row_map.has_value() ? row_map->data_ptr<int32_t>() : nullptr,
                                        groups.data_ptr<int32_t>(), static_cast<int>(ngroups), static_cast<int>(X.size(-1)),
                                        out.data_ptr<float>(), current_stream(X)),
               "absmax_grouped");
  return out;
}
torch::Tensor moe_combine(const torch::Tensor& Y, const torch::Tensor& pos, const torch::Tensor& weights) {
  require_on(Y, Y, at::kBFloat16, "y");
  require_on(pos, Y, at::kInt, "pos");
  require_on(weights, Y, at::kBFloat16, "weights");
  TORCH_CHECK(pos.dim() == 2 && Y.dim() == 2 && weights.numel() >= pos.numel(), "y must be [rows, H], pos and weights [tokens, k]");
  c10::cuda::CUDAGuard guard(Y.device());
  auto out = empty_on(Y, {pos.size(0), Y.size(1)}, at::kBFloat16);
  check_status(arcq_moe_combine_bf16(Y.data_ptr(), pos.data_ptr<int32_t>(), weights.data_ptr(), out.data_ptr(), pos.size(0),
                                     static_cast<int>(Y.size(1)), static_cast<int>(pos.size(1)), current_stream(Y)),
               "moe_combine");
  return out;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  py::register_local_exception_translator(&translate_status);
  m.def("matmul", &matmul, "our ARC gemm (sm_100a)", py::arg("A"), py::arg("B"), py::arg("SFA"), py::arg("SFB"),
        py::arg("scale"));
  m.def("reorder_quantize_x", &reorder_quantize_x, "Reorder and quantize activation.", py::arg("X"),
        py::arg("reorder_index"), py::arg("KE"));
  m.def("reorder_quantize_w", &reorder_quantize_w, "Reorder and quantize weight.", py::arg("W"),
        py::arg("reorder_index"), py::arg("KE"));
  m.def("rmsnorm_quantize_x", &rmsnorm_quantize_x, "RMSNorm, reorder and quantize activation.", py::arg("X"),
        py::arg("W"), py::arg("eps"), py::arg("reorder_index"), py::arg("KE"), py::arg("clear") = py::none());
  m.def("matmul_dev_alpha", &matmul_dev_alpha, "gemm with device-resident global scales", py::arg("A"),
        py::arg("B"), py::arg("SFA"), py::arg("SFB"), py::arg("alpha_a"), py::arg("alpha_b") = py::none(),
        py::arg("bias") = py::none());
  m.def("linear", &linear, "forward of a quantized linear", py::arg("A"), py::arg("B"), py::arg("SFA"), py::arg("SFB"), py::arg("alpha_a"),
        py::arg("alpha_b"), py::arg("bias"), py::arg("bsz"), py::arg("q_len"));
  m.def("attention_half", &attention_half, "norm, q/k/v, rotary embedding, attention, o projection of a decoder layer");
  m.def("mlp_half", &mlp_half, "norm, gate/up with SwiGLU, down projection of a decoder layer");
  m.def("route_topk", &route_topk, "(expert ids, weights) of router logits", py::arg("logits"), py::arg("top_k"));
  m.def("moe_layout", &moe_layout, "(dest, row_map, groups, tile_group) of routed rows", py::arg("slot_group"), py::arg("ngroups"),
        py::arg("tile"), py::arg("rows_bound"), py::arg("div"));
  m.def("absmax_grouped", &absmax_grouped, "max|x| over the rows of each run", py::arg("X"), py::arg("row_map"), py::arg("groups"),
        py::arg("ngroups"));
  m.def("moe_combine", &moe_combine, "weighted sums of the routed copies", py::arg("Y"), py::arg("pos"), py::arg("weights"));
  m.def("matmul_residual", &matmul_residual, "residual + gemm with device-resident global scales", py::arg("A"), py::arg("B"),
        py::arg("SFA"), py::arg("SFB"), py::arg("alpha_a"), py::arg("alpha_b"), py::arg("residual"));
  m.def("reorder_quantize_x_scaled", &reorder_quantize_x_scaled, "reorder_quantize_x of X / scale (device scalar)",
        py::arg("X"), py::arg("scale"), py::arg("reorder_index"), py::arg("KE"), py::arg("mode") = -1);
  m.def("quantize_tensor_scale", &quantize_tensor_scale, "(Q, SF, scale) of x or w over its per-tensor scale", py::arg("X"),
        py::arg("reorder_index"), py::arg("KE"), py::arg("mode") = -1, py::arg("is_weight") = false,
        py::arg("amax") = py::none());
  m.def("matmul_swiglu", &matmul_swiglu, "gate/up GEMM with SwiGLU: (act, amax)", py::arg("A"), py::arg("B"), py::arg("SFA"),
        py::arg("SFB"), py::arg("alpha_a"), py::arg("alpha_b"), py::arg("onto") = py::none());
  m.def("matmul_grouped_swiglu", &matmul_grouped_swiglu, "its grouped form", py::arg("A"), py::arg("B"), py::arg("SFA"), py::arg("SFB"),
        py::arg("tile_group"), py::arg("groups"), py::arg("ngroups"), py::arg("n"), py::arg("alpha_a"), py::arg("alpha_b"),
        py::arg("onto") = py::none());
  m.def("matmul_grouped_runs", &matmul_grouped_runs, "grouped GEMM with the run table", py::arg("A"), py::arg("B"), py::arg("SFA"),
        py::arg("SFB"), py::arg("tile_group"), py::arg("groups"), py::arg("ngroups"), py::arg("n"), py::arg("alpha_a"), py::arg("alpha_b"));
  m.def("quantize_grouped_amax", &quantize_grouped_amax, "grouped rows by their runs' maxima: (codes, scales, scale)", py::arg("X"),
        py::arg("row_map"), py::arg("amax"), py::arg("reorder_indices"), py::arg("groups"), py::arg("rows_bound"), py::arg("KE"),
        py::arg("mode"), py::arg("clear") = py::none());
  m.def("channel_order", &channel_order, "channels by ascending statistic, int16", py::arg("value"));
  m.def("calib_stats", &calib_stats, "accumulate the calibration statistics of one batch", py::arg("X"),
        py::arg("chan_absmax"), py::arg("above") = py::none());
  m.def("silu_mul", &silu_mul, "(silu(gate) * up, max|.|) of [gate | up]", py::arg("gate_up"));
  m.def("rope_inplace", &rope_inplace, "rotate-half rotary embedding in place on the first heads of each row",
        py::arg("X"), py::arg("cos"), py::arg("sin"), py::arg("heads"), py::arg("head_dim"));
  m.def("absmax", &absmax, "max|x| of a bf16 tensor as a 0-dim fp32 tensor", py::arg("X"));
  m.def("sf_bytes", [](int64_t rows, int64_t k_eff) { return static_cast<int64_t>(arcq_sf_bytes(rows, k_eff)); },
        "bytes of a scale-factor buffer");
}
