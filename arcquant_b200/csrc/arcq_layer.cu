// Element-wise pieces of a decoder layer that sit between the quantized linears: rotary position
// embedding applied in place to the q and k columns of the fused qkv output, and SiLU(gate) * up with
// the per-tensor max|.| of the result (which the next activation quantizer needs) taken in the same
// pass.  The reference's layers call torch for these (model/qLlamaLayer.py of ARCQuant uses the
// Hugging Face `apply_rotary_pos_emb` and `act_fn(gate) * up`); the arithmetic below reproduces the
// eager torch results bit for bit: every product and sum is rounded to fp32 separately, the same
// `expf` and IEEE division, bf16 rounding after SiLU and after the product.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <math.h>
#include <stdlib.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <type_traits>

#include "arcq_internal.h"

namespace arcq {
namespace {

__device__ __forceinline__ float lo_f(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float hi_f(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

__device__ __forceinline__ uint32_t max_bf16x2(uint32_t a, uint32_t b) {
  asm("max.bf16x2 %0, %0, %1;" : "+r"(a) : "r"(b));
  return a;
}
__device__ __forceinline__ uint32_t gt_mask_bf16x2(uint32_t a, uint32_t b) {   // 0xffff per half where a > b
  return __hgt2_mask(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b));
}
// n + (a > b) per half, n a small whole number.
__device__ __forceinline__ uint32_t count_gt_bf16x2(uint32_t n, uint32_t a, uint32_t b) {
  const __nv_bfloat162 r = __hadd2(*reinterpret_cast<__nv_bfloat162*>(&n), __hgt2(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b)));
  return *reinterpret_cast<const uint32_t*>(&r);
}

// x: [tokens, row_elems] bf16; the first `heads` heads of `dim` elements of each row are rotated:
// out[d] = x[d] * cos[d] - x[d + dim/2] * sin[d],  out[d + dim/2] = x[d + dim/2] * cos[..] + x[d] * sin[..]
// (rotate-half convention), cos/sin: [seq, dim] fp32 indexed by token % seq.  One thread = 8 + 8 elements.
// Bound: HBM, 4 bytes an element; few tokens: latency.  I: 32 bits where they count all items (narrow_index) - three divisions in 64 bits were most of
// the kernel's instructions.  us, 64 bits and 16 CTAs per SM / 32 bits / and 32 CTAs per SM: 16 384 tokens of 40 heads 63.9 / 60.4 / 58.5 (floor 51), 4096 16.7 /
// 16.1 / 15.8, 777 5.2 / 4.7 / 4.7, 1 token 2.1 / 1.7 / 1.7.
template <typename I>
__global__ void arcq_rope_kernel(uint16_t* __restrict__ x, const float* cs, const float* sn,
                                 long long tokens, int row_elems, int heads, int dim, int seq) {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int half = dim >> 1, per_head = half >> 3;
  const I total = (I)(tokens * heads * per_head);
  for (I i = blockIdx.x * (I)blockDim.x + threadIdx.x; i < total; i += (I)gridDim.x * blockDim.x) {
    const I th = i / (I)per_head;
    const int d8 = (int)(i - th * (I)per_head);
    const I t = th / (I)heads;
    const int h = (int)(th - t * (I)heads);
    const int pos = (int)(t % (I)seq);
    uint16_t* base = x + (long long)t * row_elems + (long long)h * dim + d8 * 8;
    const uint4 a = *reinterpret_cast<const uint4*>(base), b = *reinterpret_cast<const uint4*>(base + half);
    const float* c0 = cs + (long long)pos * dim + d8 * 8;
    const float* s0 = sn + (long long)pos * dim + d8 * 8;
    const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
    uint32_t oa[4], ob[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float ra[2], rb[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float xa = e ? hi_f(aw[k]) : lo_f(aw[k]), xb = e ? hi_f(bw[k]) : lo_f(bw[k]);
        const int d = 2 * k + e;
        // first half: x_a * cos + (-x_b) * sin;  second half: x_b * cos + x_a * sin
        ra[e] = __fadd_rn(__fmul_rn(xa, c0[d]), __fmul_rn(-xb, s0[d]));
        rb[e] = __fadd_rn(__fmul_rn(xb, c0[half + d]), __fmul_rn(xa, s0[half + d]));
      }
      oa[k] = pack2(ra[0], ra[1]);
      ob[k] = pack2(rb[0], rb[1]);
    }
    *reinterpret_cast<uint4*>(base) = make_uint4(oa[0], oa[1], oa[2], oa[3]);
    *reinterpret_cast<uint4*>(base + half) = make_uint4(ob[0], ob[1], ob[2], ob[3]);
  }
}

__device__ __forceinline__ float silu_bf16(float g) {
  const float s = __fdiv_rn(g, __fadd_rn(1.0f, expf(-g)));
  return __uint_as_float(pack2(s, 0.f) << 16);   // rounded to bf16, as torch's bf16 SiLU returns it
}

// gu: [tokens, 2F] bf16 = [gate | up]; out: [tokens, F] bf16 = bf16(bf16(silu(gate)) * up); amax: max |out|.
__global__ void arcq_silu_mul_kernel(const uint16_t* __restrict__ gu, uint16_t* __restrict__ out, long long tokens, int F,
                                     unsigned int* amax) {
  const int vec_per_row = F >> 3;
  const long long total = tokens * vec_per_row;
  uint32_t m = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long t = i / vec_per_row;
    const int v = (int)(i - t * vec_per_row);
    const uint16_t* row = gu + t * 2LL * F;
    const uint4 g = *reinterpret_cast<const uint4*>(row + v * 8), u = *reinterpret_cast<const uint4*>(row + F + v * 8);
    const uint32_t gw[4] = {g.x, g.y, g.z, g.w}, uw[4] = {u.x, u.y, u.z, u.w};
    uint32_t o[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float a = __fmul_rn(silu_bf16(lo_f(gw[k])), lo_f(uw[k]));
      const float b = __fmul_rn(silu_bf16(hi_f(gw[k])), hi_f(uw[k]));
      o[k] = pack2(a, b);
      uint32_t ab;
      asm("max.u16x2 %0, %1, %2;" : "=r"(ab) : "r"(m), "r"(o[k] & 0x7fff7fffu));
      m = ab;
    }
    *reinterpret_cast<uint4*>(out + t * (long long)F + v * 8) = make_uint4(o[0], o[1], o[2], o[3]);
  }
  if (amax) {
    uint32_t r = max(m & 0xffffu, m >> 16);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) r = max(r, __shfl_xor_sync(0xffffffffu, r, d));
    if ((threadIdx.x & 31) == 0) atomicMax(amax, r << 16);   // non-negative floats order like their bit patterns
  }
}

// Large calls: bf16 SiLU is a function of 65 536 bit patterns, and its exact evaluation (expf, IEEE
// division: ~25 instructions per element) makes the pass above instruction bound at ~0.75 of the HBM
// rate.  g_silu_table holds bf16(silu(g)) for every g, written by arcq_silu_table_kernel with the very
// function above (so the results cannot differ); each CTA of the main kernel copies the 128 KB into
// shared memory and looks SiLU up.
__device__ uint16_t g_silu_table[65536];

__global__ void arcq_silu_table_kernel() {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  g_silu_table[i] = (uint16_t)(__float_as_uint(silu_bf16(__uint_as_float(i << 16))) >> 16);
}

// The table is written once per device: the first call launches the kernel on its own stream and records
// an event, later calls make their stream wait for that event until it has completed (after which the
// table is never touched again, so calls on any number of streams only ever read it).
int ensure_silu_table(int device, cudaStream_t stream) {
  struct State { bool started = false, done = false; cudaEvent_t ev = nullptr; };
  static std::mutex mu;
  static State st[64];
  if (device < 0 || device >= 64) return ARCQ_ERR_CUDA;
  std::lock_guard<std::mutex> lock(mu);
  State& s = st[device];
  if (s.done) return ARCQ_OK;
  if (!s.started) {
    ARCQ_CUDA_TRY(cudaEventCreateWithFlags(&s.ev, cudaEventDisableTiming));
    arcq_silu_table_kernel<<<65536 / 256, 256, 0, stream>>>();
    ARCQ_CUDA_TRY(cudaGetLastError());
    ARCQ_CUDA_TRY(cudaEventRecord(s.ev, stream));
    s.started = true;
    return ARCQ_OK;
  }
  if (cudaEventQuery(s.ev) == cudaSuccess) {
    s.done = true;
    return ARCQ_OK;
  }
  (void)cudaGetLastError();   // (cudaErrorNotReady is not an error)
  ARCQ_CUDA_TRY(cudaStreamWaitEvent(stream, s.ev, 0));
  return ARCQ_OK;
}

__global__ void __launch_bounds__(1024, 1) arcq_silu_mul_table_kernel(const uint16_t* __restrict__ gu, uint16_t* __restrict__ out,
                                                                      long long tokens, int F, unsigned int* amax) {
  extern __shared__ __align__(16) uint16_t tab[];
  {
    const uint4* src = reinterpret_cast<const uint4*>(g_silu_table);
    uint4* dst = reinterpret_cast<uint4*>(tab);
    for (int i = threadIdx.x; i < 65536 / 8; i += blockDim.x) dst[i] = src[i];
  }
  __syncthreads();
  const int vec_per_row = F >> 3;
  const long long total = tokens * vec_per_row;
  const long long step = (long long)gridDim.x * blockDim.x;
  uint32_t m = 0;
  // two vectors per thread and iteration: four 16-byte loads in flight before any is used
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += 2 * step) {
    const long long i1 = i + step;
    const bool two = i1 < total;
    const long long t0 = i / vec_per_row, t1 = two ? i1 / vec_per_row : t0;
    const int v0 = (int)(i - t0 * vec_per_row), v1 = two ? (int)(i1 - t1 * vec_per_row) : v0;
    const uint16_t* r0 = gu + t0 * 2LL * F + v0 * 8;
    const uint16_t* r1 = gu + t1 * 2LL * F + v1 * 8;
    const uint4 g0 = *reinterpret_cast<const uint4*>(r0), u0 = *reinterpret_cast<const uint4*>(r0 + F);
    const uint4 g1 = *reinterpret_cast<const uint4*>(r1), u1 = *reinterpret_cast<const uint4*>(r1 + F);
    auto one = [&](const uint4& g, const uint4& u, long long t, int v) {
      const uint32_t gw[4] = {g.x, g.y, g.z, g.w}, uw[4] = {u.x, u.y, u.z, u.w};
      uint32_t o[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float sa = __uint_as_float((uint32_t)tab[gw[k] & 0xffffu] << 16);
        const float sb = __uint_as_float((uint32_t)tab[gw[k] >> 16] << 16);
        o[k] = pack2(__fmul_rn(sa, lo_f(uw[k])), __fmul_rn(sb, hi_f(uw[k])));
        uint32_t ab;
        asm("max.u16x2 %0, %1, %2;" : "=r"(ab) : "r"(m), "r"(o[k] & 0x7fff7fffu));
        m = ab;
      }
      *reinterpret_cast<uint4*>(out + t * (long long)F + v * 8) = make_uint4(o[0], o[1], o[2], o[3]);
    };
    one(g0, u0, t0, v0);
    if (two) one(g1, u1, t1, v1);
  }
  if (amax) {
    uint32_t r = max(m & 0xffffu, m >> 16);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) r = max(r, __shfl_xor_sync(0xffffffffu, r, d));
    if ((threadIdx.x & 31) == 0) atomicMax(amax, r << 16);   // non-negative floats order like their bit patterns
  }
}

// SiLU(gate) * up over grouped rows (see arcq_silu_mul_grouped_bf16): tiles of 256 rows without rows are
// skipped, padding rows inside a tile are computed but kept out of the maxima, and amax[e] receives max|out|
// over the rows of run e.  F/8 is a multiple of 32, so the 32 vectors a warp takes per step lie in one row
// and the warp's run is uniform: its running maximum is flushed (one atomic per warp) when the run changes.
template <bool TABLE>
__global__ void __launch_bounds__(1024, 1)
arcq_silu_mul_grouped_kernel(const uint16_t* __restrict__ gu, uint16_t* __restrict__ out, long long rows, int F,
                             const int* __restrict__ tile_group, const int* __restrict__ groups, int ngroups,
                             unsigned int* amax) {
  extern __shared__ __align__(16) uint16_t tab[];
  if (TABLE) {
    const uint4* src = reinterpret_cast<const uint4*>(g_silu_table);
    uint4* dst = reinterpret_cast<uint4*>(tab);
    for (int i = threadIdx.x; i < 65536 / 8; i += blockDim.x) dst[i] = src[i];
    __syncthreads();
  }
  const int vec_per_row = F >> 3;
  const long long total = rows * vec_per_row;
  const long long step = (long long)gridDim.x * blockDim.x;
  uint32_t m = 0;
  int cur = -1;
  auto flush = [&]() {
    if (cur >= 0 && amax != nullptr) {
      uint32_t r = max(m & 0xffffu, m >> 16);
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) r = max(r, __shfl_xor_sync(0xffffffffu, r, d));
      if ((threadIdx.x & 31) == 0 && r) atomicMax(amax + cur, r << 16);
    }
    m = 0;
  };
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += step) {
    const long long t = i / vec_per_row;
    const int v = (int)(i - t * vec_per_row);
    const int e = __ldg(tile_group + (t >> 8));
    if (e < 0) continue;                                   // (warp-uniform)
    if (e != cur) { flush(); cur = e; }
    const bool valid = t < (long long)__ldg(groups + e) + __ldg(groups + ngroups + e);
    const uint16_t* row = gu + t * 2LL * F + v * 8;
    const uint4 g = *reinterpret_cast<const uint4*>(row), u = *reinterpret_cast<const uint4*>(row + F);
    const uint32_t gw[4] = {g.x, g.y, g.z, g.w}, uw[4] = {u.x, u.y, u.z, u.w};
    uint32_t o[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float sa, sb;
      if (TABLE) {
        sa = __uint_as_float((uint32_t)tab[gw[k] & 0xffffu] << 16);
        sb = __uint_as_float((uint32_t)tab[gw[k] >> 16] << 16);
      } else {
        sa = silu_bf16(lo_f(gw[k]));
        sb = silu_bf16(hi_f(gw[k]));
      }
      o[k] = pack2(__fmul_rn(sa, lo_f(uw[k])), __fmul_rn(sb, hi_f(uw[k])));
      if (valid) asm("max.u16x2 %0, %0, %1;" : "+r"(m) : "r"(o[k] & 0x7fff7fffu));
    }
    *reinterpret_cast<uint4*>(out + t * (long long)F + v * 8) = make_uint4(o[0], o[1], o[2], o[3]);
  }
  flush();
}

// What the next launch collects maxima in, cleared inside the chain of programmatic dependents, which a memset would end: in front of the
// quantizers of many rows that clear (see ScaleOptions::clear) and of the grouped maxima.  Layout, maxima and quantizer of a MoE block, us, with
// a memset / this: 37 x 4096 14.5 / 11.3, 500 x 4096 19.9 / 15.4, 4096 x 4096 54.7 / 51.0.
__global__ void arcq_clear_kernel(float* p, int n) {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if ((int)threadIdx.x < n) p[threadIdx.x] = 0.f;
}

// out[t] = sum over the k routed copies of token t of bf16(y[pos[t][j]] * w[t][j]), accumulated in the
// output type in the order j = 0..k-1 (a bf16 index_add over the copies adds them in bf16 as well; with
// k = 2 the order does not matter).  One thread = 8 channels of one token, two copies on their way at a time; indices as in the rotary embedding.
// us, one copy after the other and 64 bits / this: 4096 tokens of 4096 channels 19.3 / 18.3, 2222 9.8 / 9.0, 37 1.95 / 1.74.
template <typename I>
__global__ void arcq_moe_combine_kernel(const uint16_t* y, const int* pos,
                                        const uint16_t* w, uint16_t* __restrict__ out, long long tokens,
                                        int hidden, int k) {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int vec_per_row = hidden >> 3;
  const I total = (I)(tokens * vec_per_row);
  for (I i = blockIdx.x * (I)blockDim.x + threadIdx.x; i < total; i += (I)gridDim.x * blockDim.x) {
    const long long t = i / (I)vec_per_row;
    const int v = (int)(i - (I)t * (I)vec_per_row);
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    auto add = [&](const uint4& a, float wj) {
      const uint32_t aw[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        // product rounded to bf16, then a bf16 addition: what `out.index_add_(0, idx, y * w)` computes
        const uint32_t pr = pack2(__fmul_rn(lo_f(aw[q]), wj), __fmul_rn(hi_f(aw[q]), wj));
        const uint32_t sm = pack2(__fadd_rn(acc[2 * q], lo_f(pr)), __fadd_rn(acc[2 * q + 1], hi_f(pr)));
        acc[2 * q] = lo_f(sm);
        acc[2 * q + 1] = hi_f(sm);
      }
    };
    for (int j = 0; j < k; j += 2) {           // (two copies asked for at a time)
      const long long at = t * k + j, next = j + 1 < k ? at + 1 : at;
      const long long r0 = pos[at], r1 = pos[next];
      const uint16_t w0 = w[at], w1 = w[next];
      const uint4 a0 = *reinterpret_cast<const uint4*>(y + r0 * hidden + v * 8), a1 = *reinterpret_cast<const uint4*>(y + r1 * hidden + v * 8);
      add(a0, __uint_as_float((uint32_t)w0 << 16));
      if (j + 1 < k) add(a1, __uint_as_float((uint32_t)w1 << 16));
    }
    uint4 o;
    o.x = pack2(acc[0], acc[1]); o.y = pack2(acc[2], acc[3]); o.z = pack2(acc[4], acc[5]); o.w = pack2(acc[6], acc[7]);
    *reinterpret_cast<uint4*>(out + t * (long long)hidden + v * 8) = o;
  }
}

// out = residual + bf16(src[0] + src[1] + ... + src[n-1]): the partial results of a row-parallel projection
// added in fp32 in the order of the sources (the same on every rank), rounded to the output type once, then
// the bf16 addition of the residual stream.  The sources are this rank's receive slots (local memory that the
// peers' GEMMs wrote) or, for a caller that pulls, addresses in the peers' memory.  One thread = 8 elements.
struct SumSources {
  const uint4* p[8];
};
__global__ void arcq_sum_partials_kernel(const SumSources src, int n, long long nvec, const uint4* __restrict__ residual,
                                         uint4* __restrict__ out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nvec; i += (long long)gridDim.x * blockDim.x) {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int s = 0; s < n; ++s) {
      const uint4 a = __ldcs(src.p[s] + i);
      const uint32_t aw[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        acc[2 * q] = __fadd_rn(acc[2 * q], lo_f(aw[q]));
        acc[2 * q + 1] = __fadd_rn(acc[2 * q + 1], hi_f(aw[q]));
      }
    }
    uint32_t y[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) y[q] = pack2(acc[2 * q], acc[2 * q + 1]);
    if (residual != nullptr) {
      const uint4 r = __ldcs(residual + i);
      const uint32_t rw[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) y[q] = pack2(__fadd_rn(lo_f(rw[q]), lo_f(y[q])), __fadd_rn(hi_f(rw[q]), hi_f(y[q])));
    }
    out[i] = make_uint4(y[0], y[1], y[2], y[3]);
  }
}

// Barrier over the ranks of a tensor-parallel group through flags in peer memory.  Rank r owns a block of
// `world` 32-bit flags; arriving at barrier number e, it writes e into flag [r] of every rank's block and
// waits until all flags of its own block have reached e.  One CTA, thread d talks to rank d.  Everything this
// rank's earlier kernels of the stream wrote (into its own or a peer's memory) is visible to a peer's kernels
// that follow the peer's barrier: the kernel boundary orders those writes before this thread's system-scope
// fence and flag store, the peer's flag load and fence order its later reads after them.
// The wait is bounded: after `limit_ns` the kernel records ARCQ_ERR_TIMEOUT and returns.
struct PeerFlags {
  unsigned int* p[8];
};
__device__ int g_peer_error = 0;   // sticky until polled

__global__ void arcq_peer_barrier_kernel(const PeerFlags f, int rank, int world, unsigned int* counter,
                                         unsigned long long limit_ns) {
  __shared__ unsigned int epoch_s;
  if (threadIdx.x == 0) {
    epoch_s = *counter + 1u;
    *counter = epoch_s;
  }
  __syncthreads();
  const unsigned int epoch = epoch_s;
  const int d = threadIdx.x;
  if (d < world) {
    __threadfence_system();
    *reinterpret_cast<volatile unsigned int*>(f.p[d] + rank) = epoch;
    const volatile unsigned int* in = f.p[rank] + d;
    unsigned long long t0 = 0;
    for (unsigned int it = 0; (int)(*in - epoch) < 0; ++it) {
      if ((it & 255u) == 255u) {
        unsigned long long t1;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t1));
        if (t0 == 0) t0 = t1;
        if (t1 - t0 > limit_ns) {
          atomicExch(&g_peer_error, ARCQ_ERR_TIMEOUT);
          break;
        }
      }
    }
    __threadfence_system();
  }
}

// Per-run max|x| of grouped rows: run e holds rows [groups[e], groups[e] + groups[ngroups + e]) of the
// (padded) row numbering; row r of that numbering is input row row_map[r] (or r).  One warp per row, its loads unrolled by sixteen and eight.
// Bound: latency, many rows: L2.  us, a plain loop and the runs looked at one by one / a plain loop / this: 16 x 4096 of 8 runs 3.6 / 3.3 / 2.8, 74 x 4096 3.8 / 3.5 / 3.0,
// 300 x 4096 of 64 8.4 / 4.3 / 3.8, 74 x 14 336 of 8 7.5 / 7.5 / 5.5, 2222 x 14 336 8.6 / 8.6 / 7.5, 8192 x 4096 10.0 / 9.8 / 9.7.  The assembler takes a batch apart: at 32
// registers, eight CTAs to an SM, some five loads of a lane fit.  Sixteen held together (79 registers, three CTAs per SM) are faster where rows are
// few or wide (74 x 14 336 4.6, 3000 x 8192 7.5 / 6.4) and slower where short ones are many (8192 x 512 of 64 7.4 / 8.8, 300 x 4096 of 64 3.8 / 4.5).
__global__ void arcq_absmax_grouped_kernel(const uint16_t* x, const int* row_map,
                                           const int* groups, int ngroups, int K, unsigned int* out) {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int lane = threadIdx.x & 31;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  const int last = groups[ngroups - 1] + groups[2 * ngroups - 1];   // end of the last run
  // The run of a row is the one in front of the first that starts beyond it: all starts looked at together, not each behind the one before.
  auto run_of = [&](int r) {
    const uint32_t lo = __ballot_sync(0xffffffffu, lane > 0 && lane < ngroups && groups[min(lane, ngroups - 1)] > r);
    const uint32_t hi = __ballot_sync(0xffffffffu, lane + 32 < ngroups && groups[min(lane + 32, ngroups - 1)] > r);
    return (lo ? __ffs(lo) - 1 : hi ? 31 + __ffs(hi) : ngroups) - 1;
  };
  int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, e = run_of(r);
  for (; r < last; r += warps) {
    if (e + 1 < ngroups && r >= groups[e + 1]) e = run_of(r);
    if (r >= groups[e] + groups[ngroups + e]) continue;        // padding between runs
    const uint4* row = reinterpret_cast<const uint4*>(x + (size_t)(row_map ? row_map[r] : r) * (size_t)K);
    uint32_t m = 0;
    const int nvec = K >> 3;
    auto batch = [&](auto n, int at) {
      constexpr int IN = decltype(n)::value;
      uint4 a[IN];
#pragma unroll
      for (int k = 0; k < IN; ++k) a[k] = __ldcg(row + min(at + 32 * k + lane, nvec - 1));
#pragma unroll
      for (int k = 0; k < IN; ++k) {
        asm("max.u16x2 %0, %0, %1;" : "+r"(m) : "r"(a[k].x & 0x7fff7fffu));
        asm("max.u16x2 %0, %0, %1;" : "+r"(m) : "r"(a[k].y & 0x7fff7fffu));
        asm("max.u16x2 %0, %0, %1;" : "+r"(m) : "r"(a[k].z & 0x7fff7fffu));
        asm("max.u16x2 %0, %0, %1;" : "+r"(m) : "r"(a[k].w & 0x7fff7fffu));
      }
    };
    int at = 0;
    for (; at + 32 * 16 <= nvec; at += 32 * 16) batch(std::integral_constant<int, 16>(), at);
    for (; at + 32 * 8 <= nvec; at += 32 * 8) batch(std::integral_constant<int, 8>(), at);
    for (; at < nvec; at += 32) batch(std::integral_constant<int, 1>(), at);
    uint32_t v = max(m & 0xffffu, m >> 16);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, d));
    if (lane == 0) atomicMax(out + e, v << 16);   // non-negative floats order like their bit patterns
  }
}

// Padded layout of routed rows, one CTA: slot i belongs to run slot_group[i] (or to nobody if that is >=
// ngroups); the runs follow one another, each starting at a multiple of `tile` rows, slots of one run in
// their original order.  dest[i] = padded row of slot i (rows_bound for nobody), row_map[r] = i / div for
// the padded row r that holds slot i (0 for padding), groups = [first row of every run | rows of every
// run], tile_group[m] = run of tile m or -1.
// Bound: latency.  Every warp owns a run of slots and counts its runs 32 slots at a time (lanes of one run find each other
// by match, their first adds the count), the 32 warps' counts are scanned per run, and the same walk places the slots:
// 2 n / 1024 steps whatever the number of runs, coalesced.  One scan over all slots per run took 13 us for 74 slots of 8
// runs and 71 us for
// 8192; this takes 4.1 and 9.5.
__global__ void __launch_bounds__(1024, 1)
arcq_moe_layout_kernel(const long long* slot_group, int n, int ngroups, int tile, int rows_bound, int div,
                       int* __restrict__ dest, int* __restrict__ row_map, int* __restrict__ groups,
                       int* __restrict__ tile_group) {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  constexpr int BATCH = 8;
  __shared__ int s_hist[32][65], s_cnt[64], s_off[64];     // (65: a column is read by 32 lanes)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int chunk = ((n + 1023) >> 10) * 32;               // slots per warp
  const int lo = min(n, warp * chunk), hi = min(n, lo + chunk);
  int e[BATCH];                                            // runs of this lane's slots, -1: nobody
  auto load = [&](int at) {
#pragma unroll
    for (int b = 0; b < BATCH; ++b) {
      const int i = at + 32 * b + lane;
      const long long g = i < hi ? slot_group[i] : -1;
      e[b] = g >= 0 && g < ngroups ? (int)g : -1;
    }
  };
  load(lo);
  for (int r = tid; r < rows_bound; r += 1024) row_map[r] = 0;
  for (int g = lane; g < 64; g += 32) s_hist[warp][g] = 0;
  __syncwarp();
  for (int at = lo; at < hi; at += 32 * BATCH) {
    if (at != lo) load(at);
#pragma unroll
    for (int b = 0; b < BATCH; ++b) {
      if (at + 32 * b >= hi) break;
      const uint32_t same = __match_any_sync(0xffffffffu, e[b]);
      if (e[b] >= 0 && lane == __ffs(same) - 1) s_hist[warp][e[b]] += __popc(same);
      __syncwarp();
    }
  }
  __syncthreads();
  for (int g = warp; g < ngroups; g += 32) {               // exclusive scan over the warps
    const int v = s_hist[lane][g];
    int inc = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, inc, d);
      if (lane >= d) inc += u;
    }
    s_hist[lane][g] = inc - v;
    if (lane == 31) s_cnt[g] = inc;
  }
  __syncthreads();
  if (tid == 0) {
    int off = 0;
    for (int g = 0; g < ngroups; ++g) {
      s_off[g] = off;
      groups[g] = off;
      groups[ngroups + g] = s_cnt[g];
      off += (s_cnt[g] + tile - 1) / tile * tile;
    }
  }
  __syncthreads();
  const bool again = hi - lo > 32 * BATCH;                 // (else the first batch is still in registers)
  for (int at = lo; at < hi; at += 32 * BATCH) {
    if (again) load(at);
#pragma unroll
    for (int b = 0; b < BATCH; ++b) {
      if (at + 32 * b >= hi) break;
      const int i = at + 32 * b + lane;
      const uint32_t same = __match_any_sync(0xffffffffu, e[b]);
      const int first = e[b] >= 0 ? s_hist[warp][e[b]] : 0;
      __syncwarp();
      if (e[b] >= 0) {
        const int r = s_off[e[b]] + first + __popc(same & ((1u << lane) - 1u));
        dest[i] = r;
        row_map[r] = i / div;
        if (lane == __ffs(same) - 1) s_hist[warp][e[b]] = first + __popc(same);
      } else if (i < hi) {
        dest[i] = rows_bound;
      }
      __syncwarp();
    }
  }
  for (int m = tid; m < rows_bound / tile; m += 1024) {
    const int start = m * tile;
    int run = -1;
    for (int g = 0; g < ngroups; ++g)
      if (start >= s_off[g] && start < s_off[g] + s_cnt[g]) run = g;
    tile_group[m] = run;
  }
}

// Routing of a MoE block: softmax over a token's logits in fp32, the top_k largest probabilities (of equal ones the
// earliest), their shares of the selected sum rounded to bf16.  width (a power of two >= experts, at most 32) lanes per
// token; sums in the order of a butterfly over them.  Bound: launches - softmax, top-k, its sort, the sum, the division
// and the cast as torch operations were seven launches, 21 us of kernels for 37 tokens and 29 us for 4096; this
// kernel takes 2.8 and 2.6.
__global__ void arcq_route_topk_kernel(const uint16_t* logits, long long tokens, int experts, int width, int top_k,
                                       long long* __restrict__ ids, uint16_t* __restrict__ weights) {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int per_warp = 32 / width, lane = threadIdx.x & 31, sub = lane & (width - 1);
  const long long warps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long t0 = ((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5) * per_warp; t0 < tokens; t0 += warps * per_warp) {
    const long long t = t0 + lane / width;
    const bool in = t < tokens && sub < experts;
    const float l = in ? __uint_as_float((uint32_t)logits[t * experts + sub] << 16) : -INFINITY;
    float mx = l;
    for (int d = width >> 1; d > 0; d >>= 1) {
      const float o = __shfl_xor_sync(0xffffffffu, mx, d);
      mx = mx < o ? o : mx;
    }
    const float ex = in ? expf(l - mx) : 0.f;
    float sum = ex;
    for (int d = width >> 1; d > 0; d >>= 1) sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, d));
    const float p = __fdiv_rn(ex, sum);
    int key = in ? (int)(__float_as_uint(p) & 0x7fffffffu) : -1;       // (a NaN orders above everything)
    float mine = 0.f, total = 0.f;
    int mine_id = 0;
    for (int j = 0; j < top_k; ++j) {
      int bk = key, bi = sub;
      for (int d = width >> 1; d > 0; d >>= 1) {
        const int ok = __shfl_xor_sync(0xffffffffu, bk, d), oi = __shfl_xor_sync(0xffffffffu, bi, d);
        if (ok > bk || (ok == bk && oi < bi)) { bk = ok; bi = oi; }
      }
      const float pv = __shfl_sync(0xffffffffu, p, (lane & ~(width - 1)) | bi);
      total = j == 0 ? pv : __fadd_rn(total, pv);
      if (sub == j) { mine = pv; mine_id = bi; }
      if (sub == bi) key = -1;
    }
    if (t < tokens && sub < top_k) {
      ids[t * top_k + sub] = mine_id;
      weights[t * top_k + sub] = (uint16_t)pack2(__fdiv_rn(mine, total), 0.f);
    }
  }
}

// Expert-parallel dispatch through peer memory, send side, one CTA: copy i of this rank goes to local expert
// ids[i] % e_local of rank d = ids[i] / e_local and takes the next free place j of this rank's block in rank
// d's receive buffer (places in copy order): slot[i] = d * cap + j, and the place's local expert is written
// into rank d's slot table (meta.p[d][rank * cap + j]); places of the block that stay free are marked with
// e_local ("nobody").  Copies beyond a block's capacity are dropped: slot[i] = ep * cap, *overflow set.
struct PeerPtrs {
  void* p[8];
};
__global__ void __launch_bounds__(1024, 1)
arcq_ep_send_layout_kernel(const long long* __restrict__ ids, int n, int e_local, int ep, int cap, int rank,
                           int* __restrict__ slot, const PeerPtrs meta, int* __restrict__ overflow) {
  __shared__ int s_warp[32], s_total;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int per = (n + 1023) >> 10;
  const int lo = min(n, tid * per), hi = min(n, lo + per);
  for (int d = 0; d < ep; ++d) {
    long long* table = static_cast<long long*>(meta.p[d]) + (size_t)rank * cap;
    int mine = 0;
    for (int i = lo; i < hi; ++i) {
      const long long e = ids[i];
      mine += (e >= 0 && e / e_local == d) ? 1 : 0;
    }
    int inc = mine;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc, k);
      if (lane >= k) inc += v;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    if (warp == 0) {
      int w = s_warp[lane], winc = w;
#pragma unroll
      for (int k = 1; k < 32; k <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, winc, k);
        if (lane >= k) winc += v;
      }
      s_warp[lane] = winc - w;
      if (lane == 31) s_total = winc;
    }
    __syncthreads();
    int r = s_warp[warp] + inc - mine;
    const int total = s_total;
    for (int i = lo; i < hi; ++i) {
      const long long e = ids[i];
      if (e >= 0 && e / e_local == d) {
        if (r < cap) {
          slot[i] = d * cap + r;
          table[r] = e - (long long)d * e_local;
        } else {
          slot[i] = ep * cap;
          *overflow = 1;
        }
        ++r;
      }
    }
    for (int j = min(total, cap) + tid; j < cap; j += 1024) table[j] = e_local;
    __syncthreads();                                   // s_warp / s_total are reused by the next rank
  }
  for (int i = lo; i < hi; ++i)
    if (ids[i] < 0 || ids[i] >= (long long)ep * e_local) slot[i] = ep * cap;
}

// Rows into the peers' buffers, one warp per item: item i reads row (item_src ? item_src[i] : i / div) of src
// (skipped if that is >= src_limit) and writes place rank * cap + s % cap of the buffer of rank s / cap, where
// s = item_slot ? item_slot[i] : i (skipped if s >= ep * cap).  Dispatch: items = routed copies, s = their slot;
// return trip: items = the places of this rank's receive buffer, read through the experts' padded layout.
__global__ void arcq_ep_rows_kernel(const uint4* __restrict__ src, const int* __restrict__ item_src, int div, int src_limit,
                                    const int* __restrict__ item_slot, int n, int row_vec, int cap, int ep, int rank,
                                    const PeerPtrs dst) {
  const int lane = threadIdx.x & 31;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
    const int s = item_slot ? __ldg(item_slot + i) : i;
    if (s < 0 || s >= ep * cap) continue;
    const int r = item_src ? __ldg(item_src + i) : i / div;
    if (r < 0 || r >= src_limit) continue;
    const int d = s / cap;
    const uint4* from = src + (size_t)r * row_vec;
    uint4* to = static_cast<uint4*>(dst.p[d]) + ((size_t)rank * cap + (s - d * cap)) * row_vec;
    for (int v = lane; v < row_vec; v += 32) to[v] = __ldg(from + v);
  }
}

// Calibration statistics in one pass over the activations (utilize.py:108 and :546-547 of ARCQuant):
// per-channel running max|x| and the number of elements larger than an eighth of their row's (signed)
// maximum.  Thread t of a CTA owns the 16-byte chunks t, t + 512, ... of every row it meets, so its channels'
// maxima stay in registers; RB rows are in flight together, so that one barrier serves their RB row maxima.
// Bound: HBM in principle (2 bytes per element, 2.5 us of [2000, 4096]); what sets the time is a chain of batches that are
// a wave of CTAs each: start, first bytes, way out of the maxima.
//  * While the batch before is finishing, every CTA pulls its first rows into L2 (a prefetch reads nothing into the CTA, so rows still
//    being written are not read early).
//  * The running maxima come into shared memory beside the rows, and only a larger value costs an atomic: all of a CTA's in the first batch,
//    few afterwards.  Lane after lane takes channel after channel, so that a warp's atomics are one line of memory.  (A thread that took
//    two neighbouring channels: the first batch of [2000, 4096] 11.1 instead of 7.8.  In the order of the chunks an atomic instruction
//    touched 32 sectors, 184 us for 4.85 million.  Clusters of eight that reduced their maxima through distributed shared memory first
//    spent more on meeting than on the atomics saved.)
//  * Row maxima are handed over in halves (see below), and elements above are counted in packed bf16: 20 shuffles, 64 shared loads and 32 popcounts
//    a thread made [2000, 4096] 7.7 us where it takes 6.6.
// us a batch, a first one and then one of eight in turn: [500, 2048] 3.8 and 3.7, [2000, 4096] 6.6 and 6.2, [20000, 4096] 30, [2000, 8192] 9.8 and
// 8.8, [500, 14336] 9.2 and 7.1, [2000, 14336] 16.4 and 15.7, [300, 28672] 10.8 and 10.2, [2000, 28672] 30.2 and 29.5 (clusters of eight, which
// a first batch of some 200 rows of more than 16384 channels would still favour, 9.1, 9.0, 68, 14.1, 9.5, 23.3, 16.0, 49).
// STAGED false: a handful of rows, whose maxima go out as they are.
constexpr int CALIB_THREADS = 512;
template <int CPT, int RB, bool STAGED>
__global__ void __launch_bounds__(CALIB_THREADS, CPT * RB > 8 ? 1 : 2)
arcq_calib_stats_kernel(const uint16_t* __restrict__ x, long long rows, int K, unsigned int* chan_absmax,
                        unsigned long long* above) {
  constexpr int WARPS = CALIB_THREADS / 32;
  extern __shared__ __align__(16) uint32_t s_col[];           // [K/2]: this CTA's channel maxima, two per word; staged [K] more: the running ones
  constexpr int W = RB / 2;                                   // words of two rows' maxima
  __shared__ __align__(16) uint32_t s_max[2][WARPS * W];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nchunks = K >> 3;
  uint32_t* s_run = s_col + (K >> 1);
  const bool aligned = (reinterpret_cast<uintptr_t>(chan_absmax) & 15u) == 0;   // (else the running maxima are read in place)
  asm volatile("griddepcontrol.launch_dependents;");
  if (STAGED && tid == 0) {
    const long long r0 = (long long)blockIdx.x * RB;
    const long long bytes = min((long long)RB, rows - r0) * K * 2;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(x + r0 * (long long)K), "r"((uint32_t)bytes) : "memory");
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  uint32_t cmax[CPT][4];
#pragma unroll
  for (int j = 0; j < CPT; ++j) cmax[j][0] = cmax[j][1] = cmax[j][2] = cmax[j][3] = 0;
  unsigned int count = 0;
  int buf = 0;
  for (long long r0 = (long long)blockIdx.x * RB; r0 < rows; r0 += (long long)gridDim.x * RB, buf ^= 1) {
    uint4 v[RB][CPT];
#pragma unroll
    for (int i = 0; i < RB; ++i) {
#pragma unroll
      for (int j = 0; j < CPT; ++j) {
        const int c = tid + j * CALIB_THREADS;
        v[i][j] = make_uint4(0xff80ff80u, 0xff80ff80u, 0xff80ff80u, 0xff80ff80u);   // -inf: never above, never a maximum
        if (c < nchunks && r0 + i < rows) v[i][j] = __ldcs(reinterpret_cast<const uint4*>(x + (r0 + i) * (long long)K) + c);
      }
    }
    if (STAGED && aligned && r0 == (long long)blockIdx.x * RB) {
      const uint32_t to = (uint32_t)__cvta_generic_to_shared(s_run);
      for (int j = tid; j < (K >> 2); j += CALIB_THREADS)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + 16u * j), "l"(chan_absmax + 4 * j) : "memory");
    }
    uint32_t m[RB / 2];                                        // (row 2i, row 2i + 1): signed maxima
#pragma unroll
    for (int i = 0; i < RB; i += 2) {
      uint32_t a = 0xff80ff80u, b = 0xff80ff80u;
#pragma unroll
      for (int j = 0; j < CPT; ++j) {
        const uint32_t wa[4] = {v[i][j].x, v[i][j].y, v[i][j].z, v[i][j].w};
        const uint32_t wb[4] = {v[i + 1][j].x, v[i + 1][j].y, v[i + 1][j].z, v[i + 1][j].w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          a = max_bf16x2(a, wa[k]);
          b = max_bf16x2(b, wb[k]);
          if (r0 + i < rows) asm("max.u16x2 %0, %0, %1;" : "+r"(cmax[j][k]) : "r"(wa[k] & 0x7fff7fffu));
          if (r0 + i + 1 < rows) asm("max.u16x2 %0, %0, %1;" : "+r"(cmax[j][k]) : "r"(wb[k] & 0x7fff7fffu));
        }
      }
      m[i / 2] = max_bf16x2(__byte_perm(a, b, 0x5410), __byte_perm(a, b, 0x7632));
    }
    // Row maxima across the lanes: W values that 32 lanes hold halve at every step that can hand half of them over (6 shuffles for four words
    // instead of 20), so that the lanes of a 32 / W-th end up with one word; the warps' words likewise.
    {
      int step = 16;
#pragma unroll
      for (int n = W; n > 1; n >>= 1, step >>= 1) {
        const bool up = lane & step;
#pragma unroll
        for (int i = 0; i < n / 2; ++i) {
          const uint32_t keep = up ? m[i + n / 2] : m[i], give = up ? m[i] : m[i + n / 2];
          m[i] = max_bf16x2(keep, __shfl_xor_sync(0xffffffffu, give, step));
        }
      }
#pragma unroll
      for (int d = 16 / W; d > 0; d >>= 1) m[0] = max_bf16x2(m[0], __shfl_xor_sync(0xffffffffu, m[0], d));
      if ((lane & (32 / W - 1)) == 0) s_max[buf][warp * W + lane / (32 / W)] = m[0];
    }
    __syncthreads();
    uint32_t all;                                              // (in lane i at least: word i)
    if constexpr (W == 1) {                                    // (shuffles take longer here: 7 x 2048 2.9 -> 3.2 us)
      uint32_t a[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint4 w = reinterpret_cast<const uint4*>(s_max[buf])[k];
        a[k] = max_bf16x2(max_bf16x2(w.x, w.y), max_bf16x2(w.z, w.w));
      }
      all = max_bf16x2(max_bf16x2(a[0], a[1]), max_bf16x2(a[2], a[3]));
    } else {
      all = s_max[buf][lane];                                  // (word lane % W of some warp)
      if (WARPS * W > 32) all = max_bf16x2(all, s_max[buf][lane + 32]);
#pragma unroll
      for (int d = W; d < 32; d <<= 1) all = max_bf16x2(all, __shfl_xor_sync(0xffffffffu, all, d));
    }
    uint32_t over[2] = {0, 0};                                 // elements above in even and odd rows, per half
    int count16 = 0;                                           // sixteen per element above
#pragma unroll
    for (int i = 0; i < RB; i += 2) {
      const uint32_t rm = W == 1 ? all : __shfl_sync(0xffffffffu, all, i / 2);
      // the threshold in the tensor's own type, as torch computes `max * 0.125` on a bf16 tensor
      const uint32_t t = pack2(__fmul_rn(lo_f(rm), 0.125f), __fmul_rn(hi_f(rm), 0.125f));
      const uint32_t ta = __byte_perm(t, t, 0x1010), tb = __byte_perm(t, t, 0x3232);
#pragma unroll
      for (int j = 0; j < CPT; ++j) {
        const uint32_t wa[4] = {v[i][j].x, v[i][j].y, v[i][j].z, v[i][j].w};
        const uint32_t wb[4] = {v[i + 1][j].x, v[i + 1][j].y, v[i + 1][j].z, v[i + 1][j].w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if constexpr (STAGED) {
            over[0] = count_gt_bf16x2(over[0], wa[k], ta);
            over[1] = count_gt_bf16x2(over[1], wb[k], tb);
          } else {             // (a popcount is shorter than a chain of additions where few warps share the unit: 7 x 2048 2.9 / 3.2 us)
            count16 += __popc(gt_mask_bf16x2(wa[k], ta)) + __popc(gt_mask_bf16x2(wb[k], tb));
          }
        }
      }
    }
    static_assert(2 * RB * CPT <= 256, "counts that bf16 holds exactly");
    if constexpr (STAGED) count += (unsigned int)((lo_f(over[0]) + hi_f(over[0])) + (lo_f(over[1]) + hi_f(over[1])));
    else count += (unsigned int)(count16 >> 4);
  }
  if constexpr (!STAGED) {
#pragma unroll
    for (int j = 0; j < CPT; ++j) {
      const int c = tid + j * CALIB_THREADS;
      if (c < nchunks) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          atomicMax(chan_absmax + 8 * c + 2 * k, cmax[j][k] << 16);
          atomicMax(chan_absmax + 8 * c + 2 * k + 1, cmax[j][k] & 0xffff0000u);
        }
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < CPT; ++j) {
      const int c = tid + j * CALIB_THREADS;
      if (c < nchunks) *reinterpret_cast<uint4*>(s_col + 4 * c) = make_uint4(cmax[j][0], cmax[j][1], cmax[j][2], cmax[j][3]);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // (non-negative floats order like their bit patterns; a running maximum that is stale by now only costs an atomic)
    for (int c = tid; c < K; c += CALIB_THREADS) {
      const uint32_t m = (uint32_t)reinterpret_cast<const uint16_t*>(s_col)[c] << 16;
      if (m > (aligned ? s_run[c] : __ldcg(chan_absmax + c))) atomicMax(chan_absmax + c, m);
    }
  }
  if (above != nullptr) {
    unsigned long long t = count;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) t += __shfl_xor_sync(0xffffffffu, t, d);
    __shared__ unsigned long long s_count[WARPS];
    if (lane == 0) s_count[warp] = t;
    __syncthreads();
    if (tid == 0) {
      t = 0;
      for (int k = 0; k < WARPS; ++k) t += s_count[k];
      if (t) atomicAdd(above, t);
    }
  }
}

// Channel order of K statistics: ascending, equal values in order of their channels (a stable sort; NaN last).  A channel's
// place is the number of channels before it, counted against all others, where a sort is a chain of dependent passes in a
// handful of CTAs.  A CTA serves 32 channels (lane = channel), its 32 warps a share of the keys each; every CTA stages all keys
// for itself.  4096 channels 8.6 us where torch's argsort and its conversion to int16 take 45.7 (with eight warps per CTA:
// 12.7); 17 million comparisons alone would be a microsecond or two of the whole chip, of which 128 CTAs use a part.
constexpr int ORDER_THREADS = 1024, ORDER_BLOCK = 8192;
__device__ __forceinline__ uint32_t order_key(float v) {      // unsigned order = order of the values; below 2^32 - 1
  if (v != v) return 0xfffffffeu;
  const uint32_t b = v == 0.f ? 0u : __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__global__ void __launch_bounds__(ORDER_THREADS) arcq_channel_order_kernel(const float* __restrict__ value, int K, int16_t* __restrict__ order) {
  __shared__ uint4 s_key[ORDER_BLOCK / 4];
  __shared__ int s_place[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int c = blockIdx.x * 32 + lane;
  const uint32_t key = c < K ? order_key(__ldcg(value + c)) : 0u;
  if (tid < 32) s_place[tid] = 0;
  int before = 0;
  for (int b0 = 0; b0 < K; b0 += ORDER_BLOCK) {
    __syncthreads();                                          // (the block before is done with)
    uint32_t* sk = reinterpret_cast<uint32_t*>(s_key);
    const int here = min(ORDER_BLOCK, K - b0), vecs = (here + 3) >> 2;   // vectors of four keys
    for (int j = tid; j < 4 * vecs; j += ORDER_THREADS) sk[j] = j < here ? order_key(__ldcg(value + b0 + j)) : 0xffffffffu;
    __syncthreads();
    // Keys of channels before c's group of four count where they are equal too: against them the bound is one higher.
    const int own = (c - b0) >> 2;                            // (negative, or beyond the block: another block's)
#pragma unroll 4
    for (int at = warp; at < vecs; at += ORDER_THREADS / 32) {
      const uint4 k4 = s_key[at];
      const uint32_t bound = key + (at < own ? 1u : 0u);
      before += (k4.x < bound) + (k4.y < bound) + (k4.z < bound) + (k4.w < bound);
    }
    if (warp == 0 && c >= b0 && c < b0 + here)                // equal keys among the group's own four
      for (int j = 4 * own; j < c - b0; ++j) before += sk[j] == key;
  }
  atomicAdd(&s_place[lane], before);
  __syncthreads();
  if (tid < 32 && c < K) order[s_place[tid]] = (int16_t)c;
}

}  // namespace

int launch_channel_order(const float* value, int K, int16_t* order, cudaStream_t stream) {
  DeviceInfo di;
  int rc = get_device_info(&di);
  if (rc != ARCQ_OK) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((K + 31) / 32));
  cfg.blockDim = dim3(ORDER_THREADS);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = di.early_start();
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  ARCQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, arcq_channel_order_kernel, value, K, order));
  return ARCQ_OK;
}

int launch_calib_stats(const void* x, int64_t rows, int K, float* chan_absmax, unsigned long long* above,
                       cudaStream_t stream) {
  if (rows == 0) return ARCQ_OK;
  DeviceInfo di;
  int rc = get_device_info(&di);
  if (rc != ARCQ_OK) return rc;
  const int cpt = (K / 8 + CALIB_THREADS - 1) / CALIB_THREADS;
  auto xs = static_cast<const uint16_t*>(x);
  auto cm = reinterpret_cast<unsigned int*>(chan_absmax);
  auto launch = [&](auto kern, int rb, bool staged) -> int {
    const size_t smem = staged ? (size_t)K * 6 : 0;
    // Unasked, a launch gets 48 KB, its static part (below 1 KB here) included.  The limit is the kernel's, not this call's:
    // always the same value, so that calls of several threads and widths cannot lower one another's.
    if (smem > 47 * 1024) ARCQ_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 6 * 32768));
    // (one CTA per SM beyond 16384 channels, by its registers and its shared memory)
    const long long grid = std::min<long long>((rows + rb - 1) / rb, di.resident(cpt > 4 ? 1 : 2));
    return launch_dependent(kern, (unsigned)grid, CALIB_THREADS, smem, di, stream, xs, (long long)rows, K, cm, above);
  };
  // Up to 64 rows of up to 4096 channels are one step of a few small CTAs, which a look at the running maxima would only lengthen
  // (2048 channels, with clusters / direct: 7 rows 5.5 / 2.5 us, 40 rows 5.3 / 3.4).
  if (cpt <= 1 && rows <= 64) return launch(arcq_calib_stats_kernel<1, 2, false>, 2, false);
  // (rows in flight per CTA: eight 16-byte loads per thread, two rows at least)
  if (cpt <= 1) return launch(arcq_calib_stats_kernel<1, 8, true>, 8, true);
  if (cpt <= 2) return launch(arcq_calib_stats_kernel<2, 4, true>, 4, true);
  if (cpt <= 4) return launch(arcq_calib_stats_kernel<4, 2, true>, 2, true);
  if (cpt <= 8) return launch(arcq_calib_stats_kernel<8, 2, true>, 2, true);
  return ARCQ_ERR_UNSUPPORTED_K;
}

int launch_clear(float* p, int n, cudaStream_t stream) {
  if (n < 0 || n > 64) return ARCQ_ERR_BAD_SHAPE;
  DeviceInfo di;
  int rc = get_device_info(&di);
  if (rc != ARCQ_OK) return rc;
  return launch_dependent(arcq_clear_kernel, 1, 64, 0, di, stream, p, n);
}

int launch_ep_send_layout(const long long* ids, int n, int e_local, int ep, int cap, int rank, int* slot,
                          void* const* meta, int* overflow, cudaStream_t stream) {
  PeerPtrs m = {};
  for (int d = 0; d < ep; ++d) m.p[d] = meta[d];
  arcq_ep_send_layout_kernel<<<1, 1024, 0, stream>>>(ids, n, e_local, ep, cap, rank, slot, m, overflow);
  ARCQ_CUDA_TRY(cudaGetLastError());
  return ARCQ_OK;
}

int launch_ep_rows(const void* src, const int* item_src, int div, int src_limit, const int* item_slot, int n, int row_bytes,
                   int cap, int ep, int rank, void* const* dst, cudaStream_t stream) {
  if (n == 0) return ARCQ_OK;
  DeviceInfo di;
  int rc = get_device_info(&di);
  if (rc != ARCQ_OK) return rc;
  PeerPtrs b = {};
  for (int d = 0; d < ep; ++d) b.p[d] = dst[d];
  long long blocks = ((long long)n + 7) / 8;              // eight warps (rows) per CTA
  const long long capb = (long long)di.num_sms * 8;
  if (blocks > capb) blocks = capb;
  arcq_ep_rows_kernel<<<(unsigned)blocks, 256, 0, stream>>>(static_cast<const uint4*>(src), item_src, div, src_limit,
                                                           item_slot, n, row_bytes / 16, cap, ep, rank, b);
  ARCQ_CUDA_TRY(cudaGetLastError());
  return ARCQ_OK;
}

int launch_moe_layout(const long long* slot_group, int n, int ngroups, int tile, int rows_bound, int div, int* dest,
                      int* row_map, int* groups, int* tile_group, cudaStream_t stream) {
  DeviceInfo di;
  int rc = get_device_info(&di);
  if (rc != ARCQ_OK) return rc;
  return launch_dependent(arcq_moe_layout_kernel, 1, 1024, 0, di, stream, slot_group, n, ngroups, tile, rows_bound, div, dest,
                          row_map, groups, tile_group);
}

int launch_route_topk(const void* logits, int64_t tokens, int experts, int top_k, long long* ids, void* weights,
                      cudaStream_t stream) {
  if (tokens == 0) return ARCQ_OK;
  DeviceInfo di;
  int rc = get_device_info(&di);
  if (rc != ARCQ_OK) return rc;
  int width = 1;
  while (width < experts) width <<= 1;
  const long long per_block = 4 * (32 / width);            // four warps
  long long blocks = (tokens + per_block - 1) / per_block;
  if (blocks > (long long)di.num_sms * 16) blocks = (long long)di.num_sms * 16;
  return launch_elementwise(arcq_route_topk_kernel, (unsigned)blocks, 128, di, stream, static_cast<const uint16_t*>(logits),
                          (long long)tokens, experts, width, top_k, ids, static_cast<uint16_t*>(weights));
}

int launch_absmax_grouped(const void* x, const int* row_map, const int* groups, int ngroups, int K, float* out,
                          cudaStream_t stream) {
  DeviceInfo di;
  int rc = get_device_info(&di);
  if (rc == ARCQ_OK) rc = launch_clear(out, ngroups, stream);
  if (rc != ARCQ_OK) return rc;
  // Eight CTAs per SM, whatever the rows: early only where a warp's row is short.  Layout, maxima and quantizer of a MoE block in turn, us, early /
  // not: 37 x 1024 9.8 / 10.1, 37 x 4096 11.3 / 11.6, 4096 x 4096 50.2 / 50.4, 8192 x 4096 96.0 / 95.3, 8192 x 5120 108.4 / 107.3, 1000 x 8192 27.6 / 24.9,
  // 2222 x 14 336 91 / 76 (37 x 8192 13.3 / 13.5); in an eager MoE block of 37 x 4096 it saves 1.6 of 181.
  return launch_kernel(arcq_absmax_grouped_kernel, (unsigned)di.num_sms * 8, 256, 0, di.early_start() && K <= 4096, stream,
                       static_cast<const uint16_t*>(x), row_map, groups, ngroups, K, reinterpret_cast<unsigned int*>(out));
}

// Whether 32 bits count the items of a grid-stride loop over CTAs of 256 threads, a step beyond the last among them.
static bool narrow_index(long long total, long long blocks) { return total + blocks * 256 < (1LL << 32); }

int launch_moe_combine(const void* y, const int* pos, const void* w, void* out, int64_t tokens, int hidden, int k,
                       cudaStream_t stream) {
  if (tokens == 0) return ARCQ_OK;
  DeviceInfo di;
  int rc = get_device_info(&di);
  if (rc != ARCQ_OK) return rc;
  const long long total = (long long)tokens * (hidden / 8);
  long long blocks = (total + 255) / 256;
  const long long cap = (long long)di.num_sms * 16;
  if (blocks > cap) blocks = cap;
  return launch_elementwise(narrow_index(total, blocks) ? arcq_moe_combine_kernel<uint32_t> : arcq_moe_combine_kernel<unsigned long long>, (unsigned)blocks, 256, di, stream, static_cast<const uint16_t*>(y), pos,
                          static_cast<const uint16_t*>(w), static_cast<uint16_t*>(out), (long long)tokens, hidden, k);
}

static std::atomic<long long> g_peer_wait_limit_ms{10000};

int peer_set_wait_limit_ms(int ms) {
  return (int)g_peer_wait_limit_ms.exchange(ms < 1 ? 1 : ms);
}

int launch_peer_barrier(void* const* flags, int rank, int world, unsigned int* counter, cudaStream_t stream) {
  PeerFlags f = {};
  for (int d = 0; d < world; ++d) f.p[d] = static_cast<unsigned int*>(flags[d]);
  arcq_peer_barrier_kernel<<<1, 32, 0, stream>>>(f, rank, world, counter,
                                                 (unsigned long long)g_peer_wait_limit_ms.load() * 1000000ull);
  ARCQ_CUDA_TRY(cudaGetLastError());
  return ARCQ_OK;
}

int peer_poll_error() {
  int v = 0, zero = 0;
  ARCQ_CUDA_TRY(cudaDeviceSynchronize());
  ARCQ_CUDA_TRY(cudaMemcpyFromSymbol(&v, g_peer_error, sizeof(int)));
  if (v) ARCQ_CUDA_TRY(cudaMemcpyToSymbol(g_peer_error, &zero, sizeof(int)));
  return v;
}

int launch_sum_partials(const void* const* srcs, int n, int64_t elems, const void* residual, void* out,
                        cudaStream_t stream) {
  if (elems == 0) return ARCQ_OK;
  DeviceInfo di;
  int rc = get_device_info(&di);
  if (rc != ARCQ_OK) return rc;
  SumSources src = {};
  for (int s = 0; s < n; ++s) src.p[s] = static_cast<const uint4*>(srcs[s]);
  const long long nvec = elems / 8;
  long long blocks = (nvec + 255) / 256;
  const long long cap = (long long)di.num_sms * 16;
  if (blocks > cap) blocks = cap;
  arcq_sum_partials_kernel<<<(unsigned)blocks, 256, 0, stream>>>(src, n, nvec, static_cast<const uint4*>(residual),
                                                                static_cast<uint4*>(out));
  ARCQ_CUDA_TRY(cudaGetLastError());
  return ARCQ_OK;
}

int launch_rope(void* x, const float* cos_t, const float* sin_t, int64_t tokens, int row_elems, int heads, int dim,
                int seq, cudaStream_t stream) {
  if (tokens == 0 || heads == 0) return ARCQ_OK;
  DeviceInfo di;
  int rc = get_device_info(&di);
  if (rc != ARCQ_OK) return rc;
  const long long total = (long long)tokens * heads * (dim / 16);
  long long blocks = (total + 255) / 256;
  const long long cap = (long long)di.num_sms * 32;
  if (blocks > cap) blocks = cap;
  return launch_elementwise(narrow_index(total, blocks) ? arcq_rope_kernel<uint32_t> : arcq_rope_kernel<unsigned long long>, (unsigned)blocks, 256, di, stream, static_cast<uint16_t*>(x), cos_t, sin_t,
                          (long long)tokens, row_elems, heads, dim, seq);
}

int launch_silu_mul_grouped(const void* gu, void* out, int64_t rows, int F, const int* tile_group, const int* groups,
                            int ngroups, float* amax, cudaStream_t stream) {
  if (amax) ARCQ_CUDA_TRY(cudaMemsetAsync(amax, 0, sizeof(float) * ngroups, stream));
  if (rows == 0) return ARCQ_OK;
  DeviceInfo di;
  int rc = get_device_info(&di);
  if (rc != ARCQ_OK) return rc;
  const long long total = (long long)rows * (F / 8);
  auto g = static_cast<const uint16_t*>(gu);
  auto o = static_cast<uint16_t*>(out);
  auto am = reinterpret_cast<unsigned int*>(amax);
  if (total >= (1LL << 21) && di.max_smem_optin >= 131072) {
    rc = ensure_silu_table(di.device, stream);
    if (rc != ARCQ_OK) return rc;
    auto kern = arcq_silu_mul_grouped_kernel<true>;
    static thread_local int attr_dev = -1;
    if (attr_dev != di.device) {
      ARCQ_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 131072));
      attr_dev = di.device;
    }
    kern<<<(unsigned)di.num_sms, 1024, 131072, stream>>>(g, o, rows, F, tile_group, groups, ngroups, am);
  } else {
    long long blocks = (total + 1023) / 1024;
    if (blocks > (long long)di.num_sms * 2) blocks = (long long)di.num_sms * 2;
    arcq_silu_mul_grouped_kernel<false><<<(unsigned)blocks, 1024, 0, stream>>>(g, o, rows, F, tile_group, groups, ngroups, am);
  }
  ARCQ_CUDA_TRY(cudaGetLastError());
  return ARCQ_OK;
}

int launch_silu_mul(const void* gu, void* out, int64_t tokens, int F, float* amax, cudaStream_t stream) {
  if (amax) ARCQ_CUDA_TRY(cudaMemsetAsync(amax, 0, sizeof(float), stream));
  if (tokens == 0) return ARCQ_OK;
  DeviceInfo di;
  int rc = get_device_info(&di);
  if (rc != ARCQ_OK) return rc;
  const long long total = (long long)tokens * (F / 8);
  if (total >= (1LL << 22) && di.max_smem_optin >= 131072) {   // 32 M elements and more: table lookups
    rc = ensure_silu_table(di.device, stream);
    if (rc != ARCQ_OK) return rc;
    auto kern = arcq_silu_mul_table_kernel;
    static thread_local int attr_dev = -1;
    if (attr_dev != di.device) {
      ARCQ_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 131072));
      attr_dev = di.device;
    }
    kern<<<(unsigned)di.num_sms, 1024, 131072, stream>>>(static_cast<const uint16_t*>(gu), static_cast<uint16_t*>(out),
                                                        tokens, F, reinterpret_cast<unsigned int*>(amax));
    ARCQ_CUDA_TRY(cudaGetLastError());
    return ARCQ_OK;
  }
  long long blocks = (total + 255) / 256;
  const long long cap = (long long)di.num_sms * 16;
  if (blocks > cap) blocks = cap;
  arcq_silu_mul_kernel<<<(unsigned)blocks, 256, 0, stream>>>(static_cast<const uint16_t*>(gu), static_cast<uint16_t*>(out),
                                                             tokens, F, reinterpret_cast<unsigned int*>(amax));
  ARCQ_CUDA_TRY(cudaGetLastError());
  return ARCQ_OK;
}

}  // namespace arcq
