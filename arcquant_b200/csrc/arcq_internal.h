// Internal declarations shared by the translation units of libarcq.so.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "arcq.h"

namespace arcq {

// Records a failing CUDA call for arcq_last_cuda_error() and returns ARCQ_ERR_CUDA.
int cuda_fail(cudaError_t e);

#define ARCQ_CUDA_TRY(expr)                                  \
  do {                                                       \
    cudaError_t _e = (expr);                                 \
    if (_e != cudaSuccess) return ::arcq::cuda_fail(_e);     \
  } while (0)

struct DeviceInfo {
  int device;
  int num_sms;        // SMs that launches may use (arcq_set_sm_limit)
  int all_sms;
  int max_smem_optin;
  // CTAs of a launch of which `per_sm` fit an SM at once.  Under a limit one per SM that may be used: the scheduler fills
  // idle SMs first, so n CTAs may spread over n SMs whatever fits beside them.
  long long resident(int per_sm) const { return num_sms < all_sms ? num_sms : (long long)num_sms * per_sm; }
  // Whether a launch may be set up before the kernel in front of it is done (programmatic dependent launch).  Not under a limit: two
  // grids at once hold twice the SMs, and where the CTAs fill their SMs the second sits on the very ones that are to stay free.  (A
  // chain of GEMMs under a limit of 100: a 40-CTA kernel on another stream had to wait until the GEMM under way was done, 97 us instead of 50.)
  int early_start() const { return num_sms == all_sms; }
};
// Cached properties of the current device (queried once per device).
int get_device_info(DeviceInfo* out);

// How the divisor of a scaled quantization comes about: `scale` times the factor, or - npartials > 0 - the maximum of
// that many values at `scale` times the factor, or - npartials < 0, few rows only - the maximum of the tensor itself; out (device, or
// null) receives it, per run of grouped rows.
struct ScaleOptions {
  float factor = 1.0f;
  float* out = nullptr;
  int npartials = 0;
  // nclear floats (at most 64) that the quantizer sets to zero by the way, for the launch behind it to collect maxima in.  A memset between
  // the two ends the chain of programmatic dependents: the GEMM is set up, and its first weight tiles asked for, only when it is done
  // (SwiGLU [28672, 4224] by weight streaming, call after call, us, behind a memset / behind a kernel that clears: 1 row 18.6 / 14.5, 16 rows
  // 19.9 / 15.2, 64 rows 22.0 / 17.9).
  float* clear = nullptr;
  int nclear = 0;
};

#ifdef __CUDACC__
// One thread of a converged warp, the same on every call.  A role that starts copies or MMAs is entered through this and
// not through `lane == 0`: of elect.sync the compiler knows that a single thread is active and issues those instructions
// directly; behind a comparison it wraps each in a loop over the active threads.  Measured (cycles): a tcgen05.cp 81 -> 27,
// a TMA load about 65 -> 20.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n.reg .pred P;\nelect.sync _|P, 0xffffffff;\nselp.u32 %0, 1, 0, P;\n}" : "=r"(p));
  return p != 0;
}

// early: as a programmatic dependent of the kernel before; the grid may be set up while that one drains, and waits itself
// (griddepcontrol.wait) before it touches global memory.
template <typename... Params, typename... Args>
int launch_kernel(void (*kern)(Params...), unsigned grid, unsigned threads, size_t smem, bool early, cudaStream_t stream, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = early;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  ARCQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, args...));
  return ARCQ_OK;
}
// The same wherever launches may start early (see early_start).
template <typename... Params, typename... Args>
int launch_dependent(void (*kern)(Params...), unsigned grid, unsigned threads, size_t smem, const DeviceInfo& di, cudaStream_t stream,
                     const Args&... args) {
  return launch_kernel(kern, grid, threads, smem, di.early_start() != 0, stream, args...);
}
// Element-wise kernels of many small CTAs only where these are at most one per SM: set up early, more of them crowd on the SMs that the
// kernel before leaves first (rotary embedding of 16 384 tokens behind a GEMM 72 -> 92 us; of 16 tokens it saves 1).
template <typename... Params, typename... Args>
int launch_elementwise(void (*kern)(Params...), unsigned grid, unsigned threads, const DeviceInfo& di, cudaStream_t stream, const Args&... args) {
  return launch_kernel(kern, grid, threads, 0, di.early_start() && grid <= (unsigned)di.num_sms, stream, args...);
}
#endif

// Launchers (defined in arcq_quant.cu / arcq_gemm.cu); arguments are validated by the callers
// in arcq_api.cu.
int launch_quantize(const void* x, const void* gamma, float eps, const int16_t* idx, int64_t rows, int KQ,
                    int KE, int mode, int is_weight, uint8_t* q, uint8_t* sf, cudaStream_t stream,
                    const float* scale = nullptr,    // scale (device): x is divided by it first; plain x only
                    const int* groups = nullptr, int ngroups = 0,   // runs of rows with their own order and scale
                    const int* row_map = nullptr,                   // input row of every output row
                    // further copies of the output (e.g. the peers' gathered buffers), see QuantParams
                    uint8_t* const* q_extra = nullptr, uint8_t* const* sf_extra = nullptr, int nextra = 0,
                    const ScaleOptions& so = ScaleOptions());
int launch_quantize_tensor_scale(const void* x, const float* amax, int is_weight, const int16_t* idx, int64_t rows, int KQ,
                                 int KE, int mode, uint8_t* q, uint8_t* sf, float* scale_out, float* scratch,
                                 cudaStream_t stream, const int* groups = nullptr, int ngroups = 0,
                                 const int* row_map = nullptr, float* clear = nullptr, int nclear = 0);
// n floats (at most 64) to zero, as a programmatic dependent.
int launch_clear(float* p, int n, cudaStream_t stream);
int launch_absmax(const void* x, int64_t n, float* out, int accumulate, cudaStream_t stream);
int launch_gemm(const uint8_t* A, const uint8_t* B, const uint8_t* SFA, const uint8_t* SFB, int64_t M,
                int64_t N, int64_t K_eff, float alpha, const float* alpha_a, const float* alpha_b, void* C,
                cudaStream_t stream, const void* bias = nullptr);   // bias: bf16 [N], added to the bf16-rounded result
size_t gemm_workspace_bytes(int64_t M, int64_t N, int64_t K_eff);
// Kernel choice for a shape (see arcq_matmul_plan).
int gemm_plan(int64_t M, int64_t N, int64_t K_eff, int* kind, int* tile_n, int* splits);
// launch_gemm for callers that must not allocate; refuses what gemm_workspace_bytes() puts above the documented limit.
int launch_gemm_static(const uint8_t* A, const uint8_t* B, const uint8_t* SFA, const uint8_t* SFB, int64_t M,
                       int64_t N, int64_t K_eff, float alpha, const float* alpha_a, const float* alpha_b, void* C,
                       cudaStream_t stream);
// Layer glue (arcq_layer.cu).
int launch_rope(void* x, const float* cos_t, const float* sin_t, int64_t tokens, int row_elems, int heads, int dim,
                int seq, cudaStream_t stream);
int launch_silu_mul(const void* gu, void* out, int64_t tokens, int F, float* amax, cudaStream_t stream);
int launch_moe_combine(const void* y, const int* pos, const void* w, void* out, int64_t tokens, int hidden, int k,
                       cudaStream_t stream);
// One launch over `ngroups` weight matrices stacked in B (each N rows): tile_group (device) names the
// matrix of every 256-row tile of A, alpha_a / alpha_b are per-matrix arrays.
int launch_gemm_grouped(const uint8_t* A, const uint8_t* B, const uint8_t* SFA, const uint8_t* SFB, int64_t M,
                        int64_t N, int64_t K_eff, const int* tile_group, int ngroups, const float* alpha_a,
                        const float* alpha_b, void* C, cudaStream_t stream,
                        // SwiGLU epilogue: C is [M, N/2], swiglu_amax[ngroups] takes max|C| per matrix; tile_group
                        // may be null with ngroups 1 (one matrix); groups: run table of a grouped problem (where
                        // it is known, few rows per matrix take the weight-streaming kernel)
                        // clear_amax: zero them first (else the caller has)
                        float* swiglu_amax = nullptr, const int* groups = nullptr, bool clear_amax = true);
int launch_absmax_grouped(const void* x, const int* row_map, const int* groups, int ngroups, int K, float* out,
                          cudaStream_t stream);
int launch_moe_layout(const long long* slot_group, int n, int ngroups, int tile, int rows_bound, int div, int* dest,
                      int* row_map, int* groups, int* tile_group, cudaStream_t stream);
int launch_route_topk(const void* logits, int64_t tokens, int experts, int top_k, long long* ids, void* weights,
                      cudaStream_t stream);
int launch_calib_stats(const void* x, int64_t rows, int K, float* chan_absmax, unsigned long long* above,
                       cudaStream_t stream);
int launch_channel_order(const float* value, int K, int16_t* order, cudaStream_t stream);
int launch_silu_mul_grouped(const void* gu, void* out, int64_t rows, int F, const int* tile_group, const int* groups,
                            int ngroups, float* amax, cudaStream_t stream);
// GEMM whose result rows go to `ndests` buffers of M / ndests rows each (host array of device addresses; peers'
// memory allowed), and the sum of `n` partial results plus an optional residual (arcq_layer.cu).
int launch_gemm_scatter(const uint8_t* A, const uint8_t* B, const uint8_t* SFA, const uint8_t* SFB, int64_t M,
                        int64_t N, int64_t K_eff, const float* alpha_a, const float* alpha_b, void* const* dests,
                        int ndests, cudaStream_t stream);
int launch_gemm_residual(const uint8_t* A, const uint8_t* B, const uint8_t* SFA, const uint8_t* SFB, int64_t M,
                         int64_t N, int64_t K_eff, const float* alpha_a, const float* alpha_b, const void* residual,
                         void* C, cudaStream_t stream);
// Expert-parallel dispatch through peer memory (arcq_layer.cu): places of this rank's routed copies in the peers'
// receive buffers, and rows into the peers' buffers (both directions).
int launch_ep_send_layout(const long long* ids, int n, int e_local, int ep, int cap, int rank, int* slot,
                          void* const* meta, int* overflow, cudaStream_t stream);
int launch_ep_rows(const void* src, const int* item_src, int div, int src_limit, const int* item_slot, int n, int row_bytes,
                   int cap, int ep, int rank, void* const* dst, cudaStream_t stream);
int launch_peer_barrier(void* const* flags, int rank, int world, unsigned int* counter, cudaStream_t stream);
int peer_poll_error();
int peer_set_wait_limit_ms(int ms);
int launch_sum_partials(const void* const* srcs, int n, int64_t elems, const void* residual, void* out,
                        cudaStream_t stream);
// Few rows: weight streaming (arcq_skinny.cu).
int launch_gemm_skinny(const uint8_t* X, const uint8_t* W, const uint8_t* SFX, const uint8_t* SFW, int64_t M, int64_t N,
                       int64_t K_eff, float alpha, const float* alpha_a, const float* alpha_b, const void* residual, void* C,
                       float* swiglu_amax, const int* groups, int ngroups, cudaStream_t stream, bool residual_is_bias = false);   // (swiglu_amax: cleared by the caller)
int skinny_plan_splits(int64_t M, int64_t N, int64_t K_eff);
int skinny_poll_error();
int gemm_poll_error();

}  // namespace arcq
