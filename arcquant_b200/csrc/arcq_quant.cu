// ARC-NVFP4 quantizer for sm_100a: (RMSNorm ->) channel gather -> NVFP4 block quantization ->
// re-quantized residuals of the critical channels, written as packed e2m1 codes plus ue4m3 block
// scales in the 128x4 atom layout of block-scaled tensor-core GEMMs.
//
// The kernels here serve the reference's reorder_x / reorder32_x / down32_x / rmsnorm_x and the three
// weight kernels (kernels/src/reorder.cu, down.cu, rmsnorm.cu of ARCQuant); the arithmetic is theirs,
// the organisation is not.  Three of them: sets of warps for many rows (arcq_quantize_ws_kernel_sets), small CTAs for few rows
// (arcq_quantize_rows_kernel), and one CTA after the other for the widest rows and whatever else is left (arcq_quantize_kernel).
// Common to them:
//
//  * CTAs walk over PAIRS of rows.  A pair is staged in shared memory interleaved at
//    2-byte granularity - word c = (row0[c], row1[c]) - so the random channel gather costs one
//    32-bit shared load per TWO elements, and everything downstream works on both rows at once:
//    packed 16-bit max for the block amax, packed fp32x2 multiplies (FMUL2) for the scaling,
//    cvt.rn.bf16x2 for the RMSNorm rounding;
//  * rows come through registers (128-bit coalesced streaming loads, the next ones in flight while the current
//    pair is quantized); 16-byte chunks are stored XOR-swizzled so the 128-bit shared
//    stores are conflict free;
//  * the channel order becomes, once per CTA, (swizzled) byte offsets - no per-row index traffic;
//  * block scale: ue4m3(clamp(amax/6)) and its fp32 reciprocal without branches (in the last of the three from two tiny tables indexed by
//    the bf16 bits of the amax);
//  * conversions use the hardware cvt.rn.satfinite.{e2m1x2,e4m3x2}.f32 (round to nearest even,
//    saturating), eight codes are packed per 32-bit word and stored 8 bytes per group;
//  * RMSNorm partial sums are taken from the registers of the streaming load, in the reference's
//    accumulation order, and the reciprocal root is the correctly rounded one.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "arcq_internal.h"

namespace arcq {
namespace {

struct QuantParams {
  const uint16_t* x;      // bf16 bits [rows, KQ]
  const uint16_t* gamma;  // bf16 bits [KQ] (RMSNorm gain) or nullptr
  const int16_t* idx;     // [KQ] or nullptr (identity)
  uint8_t* q;             // [rows, (KQ+KE)/2]
  uint8_t* sf;            // swizzled ue4m3 scales
  long long rows;
  long long npairs;
  int KQ, KE;
  int G, G0;      // groups per row, groups without residual
  int natoms;     // ceil(((KQ+KE)/16)/4): 512-byte scale atoms per 128-row tile
  int nchunks;    // KQ/8: 16-byte chunks per row
  int mode;       // 16 or 32 (placement of critical groups, residual flavour)
  int is_weight;  // residual slot = copy of the main codes
  float eps;
  const float* scale;   // plain operator: x is divided by *scale (device) first (see ScaleOptions), or nullptr
  // Grouped rows: the rows form `ngroups` runs, run e starting at output
  // row groups[e] with groups[ngroups + e] rows (device memory, so the host never learns the sizes);
  // run e uses the channel order idx + e*KQ and the scale scale[e].  row_map (or nullptr): input row of
  // every output row.
  const int* groups;
  int ngroups;
  const int* row_map;
};
// (ScaleOptions travels behind it as a kernel parameter of its own: three more members of this struct once made ptxas spill in a kernel whose
// registers were all in use.)

__device__ __forceinline__ float bf16lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

__device__ __forceinline__ uint4 ldg_stream(const uint4* p) {
  uint4 v;
  // (not the read-only path: launched early, a kernel lives while its input may still be written)
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

// (lo, hi) fp32 -> packed bf16x2, round to nearest even.
__device__ __forceinline__ uint32_t pack_bf16x2_rn(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
// a * b + c with a, b bf16 and c, result fp32 (one rounding): the mixed-precision FMA of sm_100.
// With c = -0.0f it is the exact product a * b, signed zeros included.
__device__ __forceinline__ float fma_bf16(uint16_t a, uint16_t b, float c) {
  float d;
  asm("fma.rn.f32.bf16 %0, %1, %2, %3;" : "=f"(d) : "h"(a), "h"(b), "f"(c));
  return d;
}
__device__ __forceinline__ uint16_t half_lo(uint32_t w) { return (uint16_t)(w & 0xffffu); }
__device__ __forceinline__ uint16_t half_hi(uint32_t w) { return (uint16_t)(w >> 16); }
// per-halfword unsigned max
__device__ __forceinline__ uint32_t max_u16x2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

// float -> ue4m3 byte: round to nearest even, saturating at 448 (input is in [2^-9, 448]).
__device__ __forceinline__ uint32_t ue4m3_encode(float s) {
  uint16_t r;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(0.0f), "f"(s));
  return (uint32_t)r & 0xffu;
}
__device__ __forceinline__ float ue4m3_decode(uint32_t c) {
  uint32_t e = (c >> 3) & 15u, m = c & 7u;
  return e ? __uint_as_float(((e + 120u) << 23) | (m << 20)) : (float)m * 0.001953125f;
}

// Eight floats -> eight e2m1 codes in one word, element 0 in the lowest nibble
// (cvt.e2m1x2 puts its first source in the high nibble).
__device__ __forceinline__ uint32_t e2m1x8(float a0, float a1, float a2, float a3, float a4, float a5,
                                           float a6, float a7) {
  uint32_t out;
  asm("{\n"
      ".reg .b8 b0, b1, b2, b3;\n"
      "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n"
      "cvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n"
      "cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n"
      "cvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n"
      "mov.b32 %0, {b0, b1, b2, b3};\n"
      "}"
      : "=r"(out)
      : "f"(a0), "f"(a1), "f"(a2), "f"(a3), "f"(a4), "f"(a5), "f"(a6), "f"(a7));
  return out;
}

// One byte of two e2m1 codes -> their values (exact): x = low nibble, y = high nibble.
__device__ __forceinline__ float2 e2m1x2_decode(uint32_t byte) {
  uint32_t h2;
  const uint16_t b16 = (uint16_t)(byte & 0xffu);
  asm("{\n.reg .b8 t;\nmov.b16 {t, _}, %1;\ncvt.rn.f16x2.e2m1x2 %0, t;\n}" : "=r"(h2) : "h"(b16));
  return __half22float2(*reinterpret_cast<__half2*>(&h2));
}

struct GroupScale {
  uint32_t byte;  // ue4m3 code
  float dec;      // its value
  float raw;      // clamp(amax/6, 2^-9, 448) before rounding
  float rcp;      // fp32(1/dec)
};

// IEEE path: every case, including subnormal and saturated scales.
__device__ __noinline__ GroupScale make_scale_slow(float amax) {
  GroupScale s;
  float t = __fdiv_rn(amax, 6.0f);
  t = fminf(t, 448.0f);
  s.raw = fmaxf(t, 0.001953125f);
  s.byte = ue4m3_encode(s.raw);
  s.dec = ue4m3_decode(s.byte);
  s.rcp = __frcp_rn(s.dec);
  return s;
}

// Table path.  ab = bf16 bits of the amax (15 bits).  For a normal result the scale code is
// T[mantissa] shifted by the exponent, and 1/scale is RB[code mantissa] shifted likewise (powers
// of two do not change any rounding).  Anything outside the normal, unsaturated range takes the
// IEEE path.
struct ScaleLut {
  const uint8_t* T;     // [128] code of amax = 1.m7 (exponent field 127)
  const uint32_t* RB;   // [8]   fp32 bits of 1/(1+m3/8), exponent pre-biased by 7
};
// Both rows of a pair: one (rarely taken) branch covers the IEEE fallback of either row.
__device__ __forceinline__ void scale_of_pair(uint32_t m, const ScaleLut& lut, uint32_t& c0, uint32_t& c1, float& r0,
                                              float& r1) {
  const uint32_t a0 = m & 0xffffu, a1 = m >> 16;
  const int s0 = (int)lut.T[a0 & 127u] + (int)((a0 >> 7) << 3) - 1016;
  const int s1 = (int)lut.T[a1 & 127u] + (int)((a1 >> 7) << 3) - 1016;
  c0 = (uint32_t)s0;
  c1 = (uint32_t)s1;
  r0 = __uint_as_float(lut.RB[s0 & 7] - ((uint32_t)(s0 >> 3) << 23));
  r1 = __uint_as_float(lut.RB[s1 & 7] - ((uint32_t)(s1 >> 3) << 23));
  // (unsigned)(s - 8) > 118  <=>  s < 8 or s > 126
  if (__builtin_expect(((uint32_t)(s0 - 8) > 118u) | ((uint32_t)(s1 - 8) > 118u), 0)) {
    const GroupScale g0 = make_scale_slow(__uint_as_float(a0 << 16));
    const GroupScale g1 = make_scale_slow(__uint_as_float(a1 << 16));
    c0 = g0.byte; r0 = g0.rcp;
    c1 = g1.byte; r1 = g1.rcp;
  }
}

__device__ __forceinline__ size_t sf_row_base(long long r, int natoms) {
  return ((size_t)(r >> 7) * (size_t)natoms) * 512 + (size_t)(r & 31) * 16 + (size_t)((r >> 5) & 3) * 4;
}
__device__ __forceinline__ size_t sf_col(int c) { return (size_t)(c >> 2) * 512 + (size_t)(c & 3); }

// Where a critical group's main / residual codes and scales go.
struct Slot {
  int byte_main, col_main, byte_res, col_res;
};
__device__ __forceinline__ Slot slot_of(int g, int G0, int mode) {
  Slot s;
  if (mode == 32) {
    int j = g - G0, pair = j >> 1, h = j & 1;
    s.col_main = G0 + 4 * pair + h; s.col_res = s.col_main + 2;
    s.byte_main = 8 * G0 + 32 * pair + 8 * h; s.byte_res = s.byte_main + 16;
  } else {
    int j = g - G0;
    s.col_main = G0 + 2 * j; s.col_res = s.col_main + 1;
    s.byte_main = 8 * G0 + 16 * j; s.byte_res = s.byte_main + 8;
  }
  return s;
}

// Both rows of a pair at once: w[i] = (row0 value, row1 value) as bf16x2.  Multiplies every value by
// its row's reciprocal scale (one FMUL2 per word) and converts to e2m1, eight codes per word.
__device__ __forceinline__ void encode_pair(const uint32_t (&w)[16], float rcp0, float rcp1, uint2& c0, uint2& c1) {
  const float2 r = make_float2(rcp0, rcp1);
  uint32_t o0[2], o1[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {   // eight words (one output word per row) at a time: fewer values live
    float2 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __fmul2_rn(make_float2(bf16lo(w[8 * h + i]), bf16hi(w[8 * h + i])), r);
    o0[h] = e2m1x8(v[0].x, v[1].x, v[2].x, v[3].x, v[4].x, v[5].x, v[6].x, v[7].x);
    o1[h] = e2m1x8(v[0].y, v[1].y, v[2].y, v[3].y, v[4].y, v[5].y, v[6].y, v[7].y);
  }
  c0 = make_uint2(o0[0], o0[1]);
  c1 = make_uint2(o1[0], o1[1]);
}

// Packed |.| maximum of the sixteen words: low half = row0 amax bits, high half = row1.
__device__ __forceinline__ uint32_t amax_pair(const uint32_t (&w)[16]) {
  uint32_t m = 0;
#pragma unroll
  for (int i = 0; i < 16; ++i) m = max_u16x2(m, w[i] & 0x7fff7fffu);
  return m;
}

// The same with the packed bf16 maximum of magnitudes (one instruction per word).  A NaN input gives
// the canonical NaN 0x7fff, which the caller clamps like the integer maximum of a NaN pattern.
__device__ __forceinline__ uint32_t amax_pair_h(const uint32_t (&w)[16]) {
  uint32_t m[4] = {w[0], w[1], w[2], w[3]};
#pragma unroll
  for (int i = 4; i < 16; ++i)
    asm("max.NaN.xorsign.abs.bf16x2 %0, %0, %1;" : "+r"(m[i & 3]) : "r"(w[i]));
  asm("max.NaN.xorsign.abs.bf16x2 %0, %0, %1;" : "+r"(m[0]) : "r"(m[1]));
  asm("max.NaN.xorsign.abs.bf16x2 %0, %0, %1;" : "+r"(m[2]) : "r"(m[3]));
  asm("max.NaN.xorsign.abs.bf16x2 %0, %0, %1;" : "+r"(m[0]) : "r"(m[2]));
  return m[0] & 0x7fff7fffu;
}

// Residuals of a critical group, both rows: w[i] <- bf16(x - q*s) per half.
// mode 16 subtracts against the rounded scale (q*s is exact in fp32, so the fused form is the same
// number); mode 32 against the un-rounded one, fused, as the 32-wide reference kernels compile.
__device__ __forceinline__ void residual_pair(uint32_t (&w)[16], uint2 c0, uint2 c1, float s0, float s1) {
#pragma unroll
  for (int i = 0; i < 16; i += 2) {
    const uint32_t b0 = ((i < 8 ? c0.x : c0.y) >> (4 * (i & 7))) & 0xffu;
    const uint32_t b1 = ((i < 8 ? c1.x : c1.y) >> (4 * (i & 7))) & 0xffu;
    const float2 q0 = e2m1x2_decode(b0), q1 = e2m1x2_decode(b1);
    float d00 = __fmaf_rn(-q0.x, s0, bf16lo(w[i])), d01 = __fmaf_rn(-q0.y, s0, bf16lo(w[i + 1]));
    float d10 = __fmaf_rn(-q1.x, s1, bf16hi(w[i])), d11 = __fmaf_rn(-q1.y, s1, bf16hi(w[i + 1]));
    w[i] = pack_bf16x2_rn(d00, d10);
    w[i + 1] = pack_bf16x2_rn(d01, d11);
  }
}

// Quantize one group of both rows and store codes + scales.  Every lane runs the same main path
// (table scale, FMUL2 + cvt); only the residual of a critical group is a divergent extra.
// Row 1 is stored before row 0: for the odd last row of the input the caller aliases row 1's
// output pointers to row 0's, and the later store wins.
__device__ __forceinline__ void quantize_group_pair(uint32_t (&w)[16], int g, const QuantParams& p,
                                                    const ScaleLut& lut, uint8_t* q0, uint8_t* q1, uint8_t* sf0,
                                                    uint8_t* sf1) {
  const uint32_t m = amax_pair(w);
  uint32_t s0, s1;
  float r0, r1;
  scale_of_pair(m, lut, s0, s1, r0, r1);
  uint2 c0, c1;
  encode_pair(w, r0, r1, c0, c1);
  const bool critical = g >= p.G0;
  int byte_main = 8 * g, col_main = g;
  Slot sl;
  if (critical) {
    sl = slot_of(g, p.G0, p.mode);
    byte_main = sl.byte_main;
    col_main = sl.col_main;
  }
  const size_t cm = sf_col(col_main);
  *reinterpret_cast<uint2*>(q1 + byte_main) = c1;
  sf1[cm] = (uint8_t)s1;
  *reinterpret_cast<uint2*>(q0 + byte_main) = c0;
  sf0[cm] = (uint8_t)s0;
  if (!critical) return;

  // critical group: the re-quantized residual (or, for weights, a copy of the main codes)
  uint2 e0 = c0, e1 = c1;
  uint32_t t0 = s0, t1 = s1;
  if (!p.is_weight) {
    float d0 = ue4m3_decode(s0), d1 = ue4m3_decode(s1);
    if (p.mode == 32) {   // against the un-rounded fp32 scale
      d0 = make_scale_slow(__uint_as_float((m & 0xffffu) << 16)).raw;
      d1 = make_scale_slow(__uint_as_float((m >> 16) << 16)).raw;
    }
    residual_pair(w, c0, c1, d0, d1);
    const uint32_t rm = amax_pair(w);
    float h0, h1;
    scale_of_pair(rm, lut, t0, t1, h0, h1);
    encode_pair(w, h0, h1, e0, e1);
  }
  const size_t cr = sf_col(sl.col_res);
  *reinterpret_cast<uint2*>(q1 + sl.byte_res) = e1;
  sf1[cr] = (uint8_t)t1;
  *reinterpret_cast<uint2*>(q0 + sl.byte_res) = e0;
  sf0[cr] = (uint8_t)t0;
}

// Sum-of-squares tree of one row in the reference's order (rmsnorm.cu:131-154 of ARCQuant), done by
// one warp: lane l owns the partials of reference threads l, l+32, ... (zero where none exists).
__device__ __forceinline__ float rms_tree(const float* ps, int nt, int lane) {
  // slot t = lane + 32k, k < 16; the tree adds slots 256, 128, 64 and 32 apart, in that order
  auto slot = [&](int k) { const int t = lane + 32 * k; return t < nt ? ps[t] : 0.f; };
  auto b = [&](int k) { return __fadd_rn(slot(k), slot(k + 8)); };       // +256
  auto c = [&](int k) { return __fadd_rn(b(k), b(k + 4)); };             // +128
  const float d0 = __fadd_rn(c(0), c(2)), d1 = __fadd_rn(c(1), c(3));    // +64
  float s = __fadd_rn(d0, d1);                                           // +32
#pragma unroll
  for (int d2 = 16; d2 > 0; d2 >>= 1) s = __fadd_rn(s, __shfl_down_sync(0xffffffffu, s, d2));
  return s;  // valid in lane 0
}

// Physical position (in 16-byte units) of logical 16-byte unit j of an interleaved row pair.
__device__ __forceinline__ uint32_t swz16(uint32_t j) { return j ^ ((j >> 3) & 1u); }
// Byte offset of channel ch's (row0,row1) word.
__device__ __forceinline__ uint32_t word_offset(uint32_t ch) { return (swz16(ch >> 2) << 4) | ((ch & 3u) << 2); }

// CPT: 16-byte chunks per thread per row; NBUF: shared buffers (2 = the next unit streams in while
// the current one is quantized); PAIRS: row pairs per loop iteration ("unit") - two pairs halve the
// per-row cost of the table reads, the barrier and the loop bookkeeping and double the independent
// shared loads in flight; RMS: fused RMSNorm; RAWIDX: the offset table holds 16-bit channel numbers
// (rows wider than 16384 channels) instead of 32-bit byte offsets.  MAXT / MINB: launch bounds.
template <int CPT, int NBUF, int PAIRS, bool RMS, bool RAWIDX, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) arcq_quantize_kernel(const QuantParams p) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int tid = threadIdx.x, nt = blockDim.x;
  const int KQ = p.KQ, G = p.G, nchunks = p.nchunks;
  const long long rows = p.rows, npairs = p.npairs;

  // shared layout: [scale tables 160 B][offsets][gain (RMS)][partial sums, rstd (RMS)][row-pair buffers]
  uint8_t* lutT = smem;
  uint32_t* lutRB = reinterpret_cast<uint32_t*>(smem + 128);
  size_t cursor = 160;
  uint32_t* offs32 = reinterpret_cast<uint32_t*>(smem + cursor);
  uint16_t* offs16 = reinterpret_cast<uint16_t*>(smem + cursor);
  cursor += ((size_t)KQ * (RAWIDX ? 2 : 4) + 15) & ~(size_t)15;
  float* gperm = reinterpret_cast<float*>(smem + cursor);
  float* psum = nullptr;
  float* rstd_s = nullptr;
  if (RMS) {
    cursor += (size_t)KQ * 4;
    psum = reinterpret_cast<float*>(smem + cursor);
    cursor += (size_t)2 * PAIRS * nt * sizeof(float);
    rstd_s = reinterpret_cast<float*>(smem + cursor);
    cursor += 16;
  }
  uint32_t* bufs = reinterpret_cast<uint32_t*>(smem + cursor);   // [NBUF][PAIRS][KQ] words

  for (int j = tid; j < 128; j += nt)
    lutT[j] = (uint8_t)make_scale_slow(__uint_as_float(((127u << 7) | (uint32_t)j) << 16)).byte;
  if (tid < 8)
    lutRB[tid] = tid ? (__float_as_uint(__frcp_rn(1.0f + 0.125f * (float)tid)) + (7u << 23)) : (134u << 23);
  // Tables are laid out [vector v][group g][4]: consecutive lanes (groups) read consecutive 16 bytes,
  // so every 128-bit table load is conflict free.
  for (int j = tid; j < KQ; j += nt) {
    int c = p.idx ? (int)p.idx[j] : j;
    const int g = j >> 4, i = j & 15;
    const int slot = (((i >> 2) * G + g) << 2) | (i & 3);
    if (RAWIDX) offs16[j] = (uint16_t)c; else offs32[slot] = word_offset((uint32_t)c);
    if (RMS) gperm[slot] = __uint_as_float((uint32_t)p.gamma[c] << 16);
  }
  const ScaleLut lut{lutT, lutRB};

  uint4 ra[PAIRS][CPT], rb[PAIRS][CPT];

  auto load_unit = [&](long long unit) {
#pragma unroll
    for (int u = 0; u < PAIRS; ++u) {
      const long long r0 = 2 * (unit * PAIRS + u);
      const bool has0 = r0 < rows, has1 = (r0 + 1) < rows;
      const uint4* x0 = reinterpret_cast<const uint4*>(p.x + r0 * (long long)KQ);
      const uint4* x1 = reinterpret_cast<const uint4*>(p.x + (r0 + 1) * (long long)KQ);
#pragma unroll
      for (int j = 0; j < CPT; ++j) {
        int c = tid + j * nt;
        if (c < nchunks) {
          ra[u][j] = has0 ? ldg_stream(x0 + c) : make_uint4(0, 0, 0, 0);
          rb[u][j] = has1 ? ldg_stream(x1 + c) : make_uint4(0, 0, 0, 0);
        }
      }
    }
  };

  auto store_unit = [&](uint32_t* buf) {
#pragma unroll
    for (int u = 0; u < PAIRS; ++u) {
      float2 ss = make_float2(0.f, 0.f);
      uint4* b4 = reinterpret_cast<uint4*>(buf + (size_t)u * KQ);
#pragma unroll
      for (int j = 0; j < CPT; ++j) {
        int c = tid + j * nt;
        if (c < nchunks) {
          const uint4 a = ra[u][j], b = rb[u][j];
          uint4 lo, hi;  // words of channels 8c..8c+3 and 8c+4..8c+7: (row0[ch], row1[ch]) per word
          lo.x = __byte_perm(a.x, b.x, 0x5410); lo.y = __byte_perm(a.x, b.x, 0x7632);
          lo.z = __byte_perm(a.y, b.y, 0x5410); lo.w = __byte_perm(a.y, b.y, 0x7632);
          hi.x = __byte_perm(a.z, b.z, 0x5410); hi.y = __byte_perm(a.z, b.z, 0x7632);
          hi.z = __byte_perm(a.w, b.w, 0x5410); hi.w = __byte_perm(a.w, b.w, 0x7632);
          // XOR-swizzled 16-byte units: the eight lanes of a 128-bit store wavefront hit distinct banks
          b4[swz16(2u * c)] = lo;
          b4[swz16(2u * c + 1u)] = hi;
          if (RMS) {
            // reference thread t adds chunk t then chunk t+KQ/16, eight elements each, in order;
            // the two rows ride in the two lanes of a packed FMA
            const uint32_t ws[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float2 v = make_float2(bf16lo(ws[i]), bf16hi(ws[i]));
              ss = __ffma2_rn(v, v, ss);
            }
          }
        }
      }
      if (RMS) {
        psum[(2 * u) * nt + tid] = ss.x;
        psum[(2 * u + 1) * nt + tid] = ss.y;
      }
    }
  };

  // The register prefetch above is scheduled late by the assembler (it holds 16+ registers), so its
  // latency is partly exposed; pulling the rows of the unit after next into L2 ahead of time turns
  // that exposed latency from an HBM access into an L2 hit.
  auto prefetch_unit_l2 = [&](long long unit) {
    if (tid < 2 * PAIRS) {
      const long long r = 2 * unit * PAIRS + tid;
      if (r < rows)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p.x + r * (long long)KQ), "r"(KQ * 2)
                     : "memory");
    }
  };

  const long long nunits = (npairs + PAIRS - 1) / PAIRS;
  long long unit = blockIdx.x;
  if (unit < nunits) { load_unit(unit); store_unit(bufs); }
  if (unit + gridDim.x < nunits) prefetch_unit_l2(unit + gridDim.x);
  __syncthreads();

  int cur = 0;
  const size_t row_bytes = (size_t)(KQ + p.KE) / 2;
  const size_t buf_words = (size_t)PAIRS * KQ;
  for (; unit < nunits; unit += gridDim.x) {
    const long long nxt = unit + gridDim.x;
    const bool more = nxt < nunits;
    if (NBUF == 2 && more) load_unit(nxt);
    if (nxt + gridDim.x < nunits) prefetch_unit_l2(nxt + gridDim.x);

    float2 rstd[PAIRS];
    if (RMS) {
      const int warp = tid >> 5, lane = tid & 31;
      if (warp < 2 * PAIRS) {
        float ss = rms_tree(psum + warp * nt, nt, lane);
        if (lane == 0) rstd_s[warp] = __frsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)KQ), p.eps));
      }
      __syncthreads();
#pragma unroll
      for (int u = 0; u < PAIRS; ++u) rstd[u] = make_float2(rstd_s[2 * u], rstd_s[2 * u + 1]);
    }

    const uint8_t* buf = reinterpret_cast<const uint8_t*>(bufs + (size_t)cur * buf_words);
    uint8_t *q0[PAIRS], *q1[PAIRS], *sf0[PAIRS], *sf1[PAIRS];
    bool live[PAIRS];
#pragma unroll
    for (int u = 0; u < PAIRS; ++u) {
      const long long r0 = 2 * (unit * PAIRS + u), r1 = r0 + 1;
      live[u] = r0 < rows;
      const bool has1 = r1 < rows;
      q0[u] = p.q + (size_t)r0 * row_bytes;
      q1[u] = has1 ? q0[u] + row_bytes : q0[u];          // odd last row: alias, row 0 is stored last
      sf0[u] = p.sf + sf_row_base(r0, p.natoms);
      sf1[u] = has1 ? p.sf + sf_row_base(r1, p.natoms) : sf0[u];
    }

    for (int g = tid; g < G; g += nt) {
      uint32_t w[PAIRS][16];
      if (RAWIDX) {
        const uint4* op = reinterpret_cast<const uint4*>(offs16 + 16 * g);
        const uint4 o0 = op[0], o1 = op[1];
        const uint32_t ow[8] = {o0.x, o0.y, o0.z, o0.w, o1.x, o1.y, o1.z, o1.w};
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const uint32_t ch = (i & 1) ? (ow[i >> 1] >> 16) : (ow[i >> 1] & 0xffffu);
          const uint32_t o = word_offset(ch);
#pragma unroll
          for (int u = 0; u < PAIRS; ++u)
            w[u][i] = *reinterpret_cast<const uint32_t*>(buf + (size_t)u * KQ * 4 + o);
        }
      } else {
        const uint4* op = reinterpret_cast<const uint4*>(offs32) + g;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const uint4 o = op[v * G];
#pragma unroll
          for (int u = 0; u < PAIRS; ++u) {
            const uint8_t* bu = buf + (size_t)u * KQ * 4;
            w[u][4 * v + 0] = *reinterpret_cast<const uint32_t*>(bu + o.x);
            w[u][4 * v + 1] = *reinterpret_cast<const uint32_t*>(bu + o.y);
            w[u][4 * v + 2] = *reinterpret_cast<const uint32_t*>(bu + o.z);
            w[u][4 * v + 3] = *reinterpret_cast<const uint32_t*>(bu + o.w);
          }
        }
      }
      if (RMS) {
        const float4* gp = reinterpret_cast<const float4*>(gperm) + g;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const float4 gm = gp[v * G];
          const float gs[4] = {gm.x, gm.y, gm.z, gm.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int i = 4 * v + k;
#pragma unroll
            for (int u = 0; u < PAIRS; ++u) {
              // bf16 x bf16 is exact in fp32; then one rounding by rstd (both rows in one FMUL2), one to bf16
              const float2 t = make_float2(__fmul_rn(bf16lo(w[u][i]), gs[k]), __fmul_rn(bf16hi(w[u][i]), gs[k]));
              const float2 n = __fmul2_rn(t, rstd[u]);
              w[u][i] = pack_bf16x2_rn(n.x, n.y);
            }
          }
        }
      }
#pragma unroll
      for (int u = 0; u < PAIRS; ++u)
        if (live[u]) quantize_group_pair(w[u], g, p, lut, q0[u], q1[u], sf0[u], sf1[u]);
    }

    if (NBUF == 2) {
      if (more) store_unit(bufs + (size_t)(cur ^ 1) * buf_words);
      __syncthreads();
      cur ^= 1;
    } else {
      __syncthreads();
      if (more) { load_unit(nxt); store_unit(bufs); }
      __syncthreads();
    }
  }
}

// ------------------------------------------------------------------------------------------------
// Pieces of the two kernels below.
//
// Block scales are computed without tables or branches: amax/6 by a multiply and one FMA correction
// (exact for every bf16 amax), the ue4m3 code of both rows by one packed conversion, and 1/scale by
// the approximate reciprocal plus one Newton step (exact here: a scale is k*2^e with k <= 15, so its
// reciprocal lies far from every fp32 rounding boundary).
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sts128(uint32_t a, const uint4& v) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

__device__ __forceinline__ uint32_t min_u16x2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("min.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

// Scales of both rows from the packed amax bits (low half row 0, high half row 1).
// codes = ue4m3(row0) | ue4m3(row1) << 8; dec = their values; rcp = fp32(1/dec); raw = clamp(amax/6) unrounded.
__device__ __forceinline__ void scale_of_pair_fma(uint32_t m, uint32_t& codes, float2& dec, float2& rcp, float2* raw = nullptr) {
  m = min_u16x2(m, 0x7f7f7f7fu);                       // inf/NaN amax -> largest finite (saturates to 448)
  const float2 a = make_float2(bf16lo(m), bf16hi(m));
  const float sixth = 0.16666667163372039794921875f;   // fp32(1/6)
  const float2 c = make_float2(sixth, sixth);
  const float2 q = __fmul2_rn(a, c);
  const float2 r = __ffma2_rn(make_float2(-6.0f, -6.0f), q, a);
  float2 t = __ffma2_rn(r, c, q);                      // = fp32(amax / 6), correctly rounded
  t.x = fmaxf(t.x, 0.001953125f);
  t.y = fmaxf(t.y, 0.001953125f);                      // values above 448 saturate in the conversion
  if (raw) *raw = make_float2(fminf(t.x, 448.0f), fminf(t.y, 448.0f));
  uint16_t c2;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(c2) : "f"(t.y), "f"(t.x));
  uint32_t h2;
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"(c2));
  dec = __half22float2(*reinterpret_cast<__half2*>(&h2));
  float2 r0;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0.x) : "f"(dec.x));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0.y) : "f"(dec.y));
  const float2 e = __ffma2_rn(make_float2(-dec.x, -dec.y), r0, make_float2(1.0f, 1.0f));
  rcp = __ffma2_rn(r0, e, r0);
  codes = c2;
}

// The tensor's divisor from the partial maxima of arcq_max_partials_kernel (one whole warp).
__device__ __forceinline__ float partials_max(const float* part, int n, int lane) {
  float m = -INFINITY;
  bool nan = false;
  for (int i = lane; i < n; i += 32) {
    const float v = __ldcg(part + i);
    nan |= v != v;
    m = fmaxf(m, v);
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
  return __any_sync(0xffffffffu, nan) ? __uint_as_float(0x7fc00000u) : m;
}

// bf16(x / s) for bf16 x and a bf16 divisor s shared by the whole tensor, as one multiplication by
// r = fp32(1/s): the caller rounds the product to bf16, and that rounding cannot differ from the
// rounding of the exact quotient.  With 8-bit significands mx, ms the quotient mx/ms is never within
// 2^-18 (relative) of the midpoint of two bf16 values unless it is a bf16 value itself (a dyadic
// mx/ms has at most 8 significant bits), while x*r is within 2^-23 of it; the same holds for the
// fp32 quotient an IEEE division would round first.  That argument needs a product that is a normal
// number with room to spare.  Products below 2^-60 in magnitude may round differently from the quotient,
// but never visibly: with the smallest block scale 2^-9 and the coarsest step of the e2m1 grid such an
// element (and its residual) quantizes to a zero of its own sign either way, and a group in which every
// element is that small gets the smallest scale either way - the codes and scale bytes, the only outputs,
// are the same.  So there is no per-element guard (it cost more than the multiplication: a third of the
// time of the wide operator); what is checked once is the divisor: when it is zero, not finite, or so
// large or small that 1/s is not a well-scaled normal number, every element takes the IEEE division.
// A large product is as accurate as any other, and where it overflows the quotient is beyond the largest
// bf16 number as well; NaN and infinite elements give the same NaN / infinity either way.
__device__ __forceinline__ bool div_by_reciprocal_ok(float s) {
  const float m = fabsf(s);
  return m >= 7.8886091e-31f && m <= 1.2676506e30f;   // 2^-100 .. 2^100
}
// Words wa, wb: two channels of row 0 and of row 1.  o0 / o1: (row 0, row 1) of the first / second channel.
__device__ __forceinline__ void div_pair_words(uint32_t wa, uint32_t wb, float s, float r, bool fast, uint32_t& o0,
                                               uint32_t& o1) {
  if (fast) {
    const float2 r2 = make_float2(r, r);
    const float2 q0 = __fmul2_rn(make_float2(bf16lo(wa), bf16lo(wb)), r2);
    const float2 q1 = __fmul2_rn(make_float2(bf16hi(wa), bf16hi(wb)), r2);
    o0 = pack_bf16x2_rn(q0.x, q0.y);
    o1 = pack_bf16x2_rn(q1.x, q1.y);
  } else {
    o0 = pack_bf16x2_rn(__fdiv_rn(bf16lo(wa), s), __fdiv_rn(bf16lo(wb), s));
    o1 = pack_bf16x2_rn(__fdiv_rn(bf16hi(wa), s), __fdiv_rn(bf16hi(wb), s));
  }
}

// ------------------------------------------------------------------------------------------------
// Kernel of many rows (of 512 to 16384 channels; RMSNorm 1024 to 8192): one CTA per SM, its 24 warps in sets of TW ("ws": warp sets).
//
// A set takes a pair of rows from global memory to its codes by itself and shares nothing with the others but the tables: the pair is
// interleaved in the set's own buffer, gathered from there group by group, quantized and stored; two barriers of the set (none where a warp is a
// set) stand between.  What bounds it: the pipe of shared memory and L1, 69 % of its cycles at 16 384 x 4096 (of them the gather, whose
// random words meet 3.6 to a bank, is half), issue slots 48 % (plain) to 57 % (fused RMSNorm).  So it is built to ask little of both:
//  * rows come through registers, not through a ring in shared memory (a raw ring costs two more passes over the pair), in slots of four 128-bit
//    loads of a lane: one on its way while the rows before are quantized, one ahead after that, all from L2, where a bulk prefetch puts the pair
//    a pair ahead (without it 43.4 -> 49.9 us);
//  * no roles: with producers and consumers one side waits for the other, and each wait is polled (40 % of the instructions of the
//    warp-specialised kernel that this one replaced, with 4650 instructions a pair of the fused RMSNorm where this one has 3350; a scheduler that gave every warp
//    tasks of both kinds in turn polled no less);
//  * 24 warps of 80 registers rather than 12 of 168 (plain 16 384 x 4096 44 -> 37 us): latency is hidden by warps.  Not one value may spill: shared memory
//    leaves next to no L1, and a spilled word comes back from L2 (100 bytes of spills: 37 -> 45 us);
//  * addresses are a base and constants: every chunk of a row is 32 lanes wide, the last chunk of a ragged row reaches back over the one
//    before (its lanes write the same values twice), the last slot likewise.
// us, the warp-specialised kernel / this one (graphs of ten calls): fused RMSNorm 32 768 x 4096 95.0 / 79.1, 16 384 x 4096 50.7 / 41.9, 4096 x 4096 15.4 /
// 13.2, 8192 x 2048 19.4 / 12.8, 8192 x 5120 40.8 / 28.2, 16 384 x 8192 88.8 / 80.4, 2048 x 8192 14.3 / 13.8, 600 x 8192 8.1 / 7.7;
// plain 16 384 x 4096 42.0 / 36.7, 16 384 x 8192 72.4 / 71.9; over a tensor's maximum 16 384 x 4096 47.7 / 37.7, 8192 x 9216 62.4 / 46,
// 16 384 x 14 336 142.4 / 128.0; eight runs of 8192 rows in all of 4096 channels 30.4 / 21.2, of 14 336 82.2 / 71.1.
// Four rows at a time (64-bit gathers, a sixth less of the pipe) do not fit 80 registers: 47 us where pairs take 43; without spills, 16 warps of
// 128 registers are too few.
// The name of a launch is what tells it from one of the row kernel.
// RMSNorm: lane l of a set's slot k is the reference's thread t = 32 (TW k + warp) + l with its chunks t and t + KQ/16; the sums of a warp's slots
// are added in the lane, those of the warps meet in shared memory, the last 32 are added across the lanes: the reference's tree.
constexpr int WS_WARPS = 24;
// Shared memory in front of the sets' buffers: offsets, gains, and the sums that cross the warps of a set.
__host__ __device__ __forceinline__ uint32_t ws_fixed_bytes(bool rms, int tw, int KQ, int nsets) {
  return (uint32_t)KQ * (rms ? 4 : 2) + (rms && tw > 1 ? (uint32_t)nsets * 512u : 0u);
}

// MG: groups per row at most.
template <bool RMS, bool SCALED, int MG, int TW>
__global__ void __launch_bounds__(WS_WARPS * 32, 1) arcq_quantize_ws_kernel_sets(const QuantParams p, const ScaleOptions so) {
  extern __shared__ __align__(32) uint8_t ws_smem[];      // (buffers begin at multiples of 32: a chunk's two halves are 16 bytes apart, either way round)
  uint8_t* smem = ws_smem;
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int set = warp / TW, sw = warp % TW, nsets = (int)(blockDim.x >> 5) / TW;
  const int KQ = p.KQ, G = p.G, G0 = p.G0;
  uint32_t rows = (uint32_t)p.rows, cta = blockIdx.x, stride = gridDim.x, row_base = 0;
  const int16_t* idx_g = p.idx;
  const float* scale_g = p.scale;
  if (p.groups != nullptr) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t ng = (uint32_t)p.ngroups, e = blockIdx.x % ng;
    cta = blockIdx.x / ng;
    stride = (gridDim.x - e + ng - 1) / ng;
    row_base = (uint32_t)p.groups[e];
    rows = (uint32_t)p.groups[ng + e];
    if (idx_g) idx_g += (size_t)e * (size_t)KQ;
    if (scale_g) scale_g += e;
  }
  const uint32_t npairs = (rows + 1) >> 1;
  if (cta >= npairs) {
    if (SCALED && p.groups != nullptr && so.out != nullptr && blockIdx.x == 0)
      for (int e = tid; e < p.ngroups; e += blockDim.x) so.out[e] = p.scale[e] * so.factor;
    return;
  }
  // shared layout: [offsets][gains (RMS)][sums that cross the warps of a set (RMS)][a buffer per set]
  uint16_t* offs = reinterpret_cast<uint16_t*>(smem);
  uint16_t* gains = offs + KQ;
  const uint32_t exch = smem_addr(smem) + (uint32_t)KQ * 4 + (uint32_t)set * 512u + 4u * lane;
  const uint32_t buf = smem_addr(smem) + ws_fixed_bytes(RMS, TW, KQ, nsets) + (uint32_t)set * (uint32_t)KQ * 4;

  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  auto in_row = [&](uint32_t r) -> const uint4* {
    const uint32_t gr = row_base + r;
    return reinterpret_cast<const uint4*>(p.x + (size_t)(p.row_map ? (uint32_t)p.row_map[gr] : gr) * (size_t)KQ);
  };
  const int slots = (G + 32 * TW - 1 - 32 * sw) / (32 * TW), t0 = 32 * sw + lane;
  uint4 first[4];
  const uint4 *x0 = nullptr, *x1 = nullptr;                // (at this lane's first chunk)
  auto rows_at = [&](uint32_t pr) {
    x0 = in_row(2 * pr) + t0;
    x1 = 2 * pr + 1 < rows ? in_row(2 * pr + 1) + t0 : x0;
  };
  auto load_slot = [&](int k, uint4 (&b)[4]) {
    const int at = RMS ? 32 * TW * k : min(32 * TW * k, G - 32 - 32 * sw);      // (the last slot of a ragged row reaches back)
    b[0] = ldg_stream(x0 + at); b[1] = ldg_stream(x0 + G + at);
    b[2] = ldg_stream(x1 + at); b[3] = ldg_stream(x1 + G + at);
  };
  const uint32_t st0 = buf + (swz16(2u * t0) << 4), st1 = buf + (swz16(2u * (t0 + G)) << 4);    // (+ 1024 TW a slot)
  uint32_t pair = cta + (uint32_t)set * stride;
  const uint32_t step = (uint32_t)nsets * stride;
  if (pair < npairs) {
    rows_at(pair);
    load_slot(0, first);
  }
  const uint32_t divisor = smem_addr(smem) + ws_fixed_bytes(RMS, TW, KQ, nsets);      // (in a buffer that nothing lies in yet)
  // The divisor: by the last warp, which has the least of the tables to set up, and ahead of them (by the first behind them: over maxima 600 x 5120 4.9 / 4.6, over
  // the tensor's own 900 x 4096 8.2 / 7.7, 6000 x 4096 21.2 / 20.6).
  if (SCALED) {
    if (warp == (int)(blockDim.x >> 5) - 1) {
      const float v = (so.npartials > 0 ? partials_max(p.scale, so.npartials, lane) : *scale_g) * so.factor;
      if (lane == 0) asm volatile("st.shared.f32 [%0], %1;" ::"r"(divisor), "f"(v) : "memory");
      if (so.out != nullptr && blockIdx.x == 0) {
        if (so.npartials > 0) {
          if (lane == 0) so.out[0] = v;
        } else {
          for (int e = lane; e < (p.groups != nullptr ? p.ngroups : 1); e += 32) so.out[e] = p.scale[e] * so.factor;
        }
      }
    }
  }
  // The tables.  RMSNorm: the gains come in their own order into a buffer that nothing lies in yet (of set 0), and from there into the order of the
  // groups: gathered from global memory they came a round trip after the channel order.
  uint16_t* gains_in = reinterpret_cast<uint16_t*>(smem + ws_fixed_bytes(RMS, TW, KQ, nsets));
  auto gains_at = [&](int v) { return __ldcg(reinterpret_cast<const uint4*>(p.gamma) + v); };
  // Eight channels that follow one another lie side by side in the tables (half a group).  Stored one by one, and the gains asked for and waited for
  // ahead of the order, they cost every CTA 0.3 to 0.9 us, which few pairs of wide rows did not win back: fused RMSNorm 600 x 8192 8.1 / 7.4, 888 x 8192
  // 8.5 / 7.7 (7.8 and 8.0 in the kernel that this one replaced), 1800 x 4096 7.9 / 7.4, plain 600 x 8192 5.8 / 5.5.
  auto fill = [&](auto channels) {
    for (int v = tid; v < (KQ >> 3); v += blockDim.x) {
      const uint4 c = channels(v);
      if (RMS) {
        const uint4 g = gains_at(v);
        *reinterpret_cast<uint4*>(gains_in + 8 * v) = g;
      }
      const uint32_t at = 8u * (uint32_t)((v & 1) * G + (v >> 1)), cw[4] = {c.x, c.y, c.z, c.w};
      uint32_t o[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) o[k] = __byte_perm(word_offset(cw[k] & 0xffffu), word_offset(cw[k] >> 16), 0x5410);
      *reinterpret_cast<uint4*>(offs + at) = make_uint4(o[0], o[1], o[2], o[3]);
      if (RMS) *reinterpret_cast<uint4*>(gains + at) = c;
    }
  };
  if (idx_g && (reinterpret_cast<uintptr_t>(idx_g) & 15u) == 0) {
    fill([&](int v) { return __ldcg(reinterpret_cast<const uint4*>(idx_g) + v); });
  } else if (idx_g) {
    fill([&](int v) {
      auto two = [&](int j) { return (uint32_t)(uint16_t)idx_g[j] | ((uint32_t)(uint16_t)idx_g[j + 1] << 16); };
      return make_uint4(two(8 * v), two(8 * v + 2), two(8 * v + 4), two(8 * v + 6));
    });
  } else {
    if (RMS)
      for (int v = tid; v < (KQ >> 3); v += blockDim.x) *reinterpret_cast<uint4*>(gains_in + 8 * v) = gains_at(v);
    // (the channels' own order: nothing to be read)
    for (int j = tid; j < KQ; j += blockDim.x) {
      const int at = ((((j & 15) >> 3) * G + (j >> 4)) << 3) | (j & 7);
      offs[at] = (uint16_t)word_offset((uint32_t)j);
      if (RMS) gains[at] = (uint16_t)j;
    }
  }
  if (RMS) {
    __syncthreads();
    for (int j = 2 * tid; j < KQ; j += 2 * blockDim.x) {
      uint32_t& two = *reinterpret_cast<uint32_t*>(gains + j);
      two = (uint32_t)gains_in[two & 0xffffu] | ((uint32_t)gains_in[two >> 16] << 16);
    }
  }
  float sc = 1.0f, rsc = 1.0f;
  bool fast = true;
  __syncthreads();
  if (SCALED) {
    // torch's CUDA kernel for (bf16 tensor) / (fp32 scalar tensor) loads the divisor as bf16
    sc = __uint_as_float(pack_bf16x2_rn(__uint_as_float(lds32(divisor)), 0.f) << 16);
    rsc = __frcp_rn(sc);
    fast = div_by_reciprocal_ok(sc);
    __syncthreads();
  }

  auto set_sync = [&]() {
    if (TW == 1) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(1 + set), "n"(32 * TW) : "memory");
  };
  const uint32_t row_bytes = (uint32_t)(KQ + p.KE) / 2, tile_bytes = (uint32_t)p.natoms * 512;
  const bool mode32 = p.mode == 32, is_weight = p.is_weight != 0;
  // (scales off a 4-byte boundary: every chunk by the loop that stores them byte by byte)
  const int chunks = (G + 31) >> 5, plain_chunks = (reinterpret_cast<uintptr_t>(p.sf) & 3u) ? 0 : G0 >> 5;
  const uint32_t offs_l = smem_addr(offs) + 16u * lane, half = 16u * (uint32_t)G;    // (to the second half of a table)
  const uint32_t sel1 = (lane & 1) ? 0x3715u : 0x6240u, sel2 = (lane & 2) ? 0x3276u : 0x5410u;
  int turn = sw;
  for (; pair < npairs; pair += step) {
    const bool has1 = 2 * pair + 1 < rows;
    // ---- both rows, interleaved
    // Slot k of the warp from registers into the buffer; s0, s1: the sums of squares of its reference thread.
    auto put_slot = [&](int k, const uint4 (&b)[4], float& s0, float& s1) {
      const bool back = !RMS && 32 * (TW * k + sw) > G - 32;
      auto interleave = [&](auto quick) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint4 u = b[h], v = b[2 + h];
          uint4 lo, hi;
          if (RMS) {
            // reference thread t adds chunk t, then chunk t + KQ/16, eight elements each, in order; x*x is exact in fp32
            const uint32_t wa[4] = {u.x, u.y, u.z, u.w}, wb[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              s0 = fma_bf16(half_hi(wa[e]), half_hi(wa[e]), fma_bf16(half_lo(wa[e]), half_lo(wa[e]), s0));
              s1 = fma_bf16(half_hi(wb[e]), half_hi(wb[e]), fma_bf16(half_lo(wb[e]), half_lo(wb[e]), s1));
            }
          }
          if (SCALED) {
            constexpr bool q = decltype(quick)::value;
            div_pair_words(u.x, v.x, sc, rsc, q, lo.x, lo.y); div_pair_words(u.y, v.y, sc, rsc, q, lo.z, lo.w);
            div_pair_words(u.z, v.z, sc, rsc, q, hi.x, hi.y); div_pair_words(u.w, v.w, sc, rsc, q, hi.z, hi.w);
          } else {
            lo.x = __byte_perm(u.x, v.x, 0x5410); lo.y = __byte_perm(u.x, v.x, 0x7632);
            lo.z = __byte_perm(u.y, v.y, 0x5410); lo.w = __byte_perm(u.y, v.y, 0x7632);
            hi.x = __byte_perm(u.z, v.z, 0x5410); hi.y = __byte_perm(u.z, v.z, 0x7632);
            hi.z = __byte_perm(u.w, v.w, 0x5410); hi.w = __byte_perm(u.w, v.w, 0x7632);
          }
          uint32_t at = (h ? st1 : st0) + 1024u * TW * k;
          if (back) at = buf + (swz16(2u * (uint32_t)((h ? G : 0) + G - 32 + lane)) << 4);
          sts128(at, lo);
          sts128(at ^ 16u, hi);
        }
      };
      if (!SCALED || fast) interleave(std::true_type{});     // (asked once per slot: a branch per word kept their work apart)
      else interleave(std::false_type{});
    };
    constexpr int MT = RMS ? 16 / TW : 1, MS = MG / 32 / TW;      // slots of the reference's tree (512 threads); slots of this warp at most
    float d[2][MT > MS ? MT : MS];
    uint4 late[MS][4];                         // (defined in every iteration: else it would stay in registers over the rest of one)
    auto load_late = [&](int k) {
      if (k < slots) load_slot(k, late[k]);
      else late[k][0] = late[k][1] = late[k][2] = late[k][3] = make_uint4(0, 0, 0, 0);
    };
    load_late(1);
#pragma unroll                                 // (a loop that is not: 16 384 x 4096 36.7 -> 38.0 us)
    for (int k = 0; k < MS; ++k) {
      d[0][k] = d[1][k] = 0.f;
      if (k < slots) put_slot(k, k == 0 ? first : late[k], d[0][k], d[1][k]);
      if (k + 2 < MS) load_late(k + 2);
    }
    float2 rstd = make_float2(1.f, 1.f);
    if (RMS) {
      // the reference's tree: slots 256, 128, 64 and 32 threads apart, then across the lanes
#pragma unroll
      for (int k = MS; k < MT; ++k) d[0][k] = d[1][k] = 0.f;
      float s[2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
#pragma unroll
        for (int w = MT / 2; w > 0; w >>= 1)
#pragma unroll
          for (int k = 0; k < w; ++k) d[r][k] = __fadd_rn(d[r][k], d[r][k + w]);
        s[r] = d[r][0];
      }
      auto give = [&](uint32_t at, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(exch + at), "f"(v) : "memory"); };
      auto take = [&](uint32_t at) { return __uint_as_float(lds32(exch + at)); };
      if (TW == 2) {             // [warp][row]
        give(256u * sw, s[0]);
        give(256u * sw + 128u, s[1]);
      } else if (TW == 4) {      // warps 0 and 1 add up row 0 with warps 2 and 3, those row 1 with them; then everyone takes both rows' halves
        give(128u * (sw ^ 2), sw < 2 ? s[1] : s[0]);
      }
      set_sync();
      if (TW == 2) {
        s[0] = __fadd_rn(take(0), take(256));
        s[1] = __fadd_rn(take(128), take(384));
      } else if (TW == 4) {
        give(128u * sw, __fadd_rn(sw < 2 ? s[0] : s[1], take(128u * sw)));
        set_sync();
        s[0] = __fadd_rn(take(0), take(128));
        s[1] = __fadd_rn(take(256), take(384));
      }
#pragma unroll
      for (int m = 16; m > 0; m >>= 1) {
        s[0] = __fadd_rn(s[0], __shfl_down_sync(0xffffffffu, s[0], m));
        s[1] = __fadd_rn(s[1], __shfl_down_sync(0xffffffffu, s[1], m));
      }
      const float s1 = __shfl_sync(0xffffffffu, s[1], 0), ss = lane == 16 ? s1 : s[0];       // (lanes 0 and 16: a row each)
      const float rs = __frsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)KQ), p.eps));
      rstd = make_float2(__shfl_sync(0xffffffffu, rs, 0), __shfl_sync(0xffffffffu, rs, 16));
    } else {
      set_sync();
    }
    const uint32_t nxt = pair + step;
    if (nxt < npairs) {
      rows_at(nxt);
      if (lane == 0 && sw == 0) {
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(x0), "r"((uint32_t)KQ * 2) : "memory");
        if (x1 != x0) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(x1), "r"((uint32_t)KQ * 2) : "memory");
      }
    }
    // ---- gather and quantize
    const uint32_t r0 = row_base + 2 * pair;
    uint8_t* q0 = p.q + (size_t)r0 * row_bytes;
    // 128-row tile, then 16 bytes per row % 32 and 4 per (row / 32) % 4
    uint8_t* sf0 = p.sf + (size_t)(r0 >> 7) * tile_bytes + (((r0 & 31u) << 4) | (((r0 >> 5) & 3u) << 2));
    auto gather = [&](uint32_t at, uint32_t (&w)[16]) {
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        const uint4 o4 = lds128(at + v * half);
        const uint32_t ow[4] = {o4.x, o4.y, o4.z, o4.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          w[8 * v + 2 * k] = lds32(buf + (ow[k] & 0xffffu));
          w[8 * v + 2 * k + 1] = lds32(buf + (ow[k] >> 16));
        }
      }
    };
    auto normalise = [&](uint32_t at, uint32_t (&w)[16]) {
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        const uint4 g4 = lds128(at + v * half);
        const uint32_t gw[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          // bf16 x bf16 is exact in fp32; then one rounding by rstd (both rows in one FMUL2), one to bf16
          const uint16_t gg = (k & 1) ? half_hi(gw[k >> 1]) : half_lo(gw[k >> 1]);
          uint32_t& x = w[8 * v + k];
          const float2 y = __fmul2_rn(make_float2(fma_bf16(half_lo(x), gg, -0.0f), fma_bf16(half_hi(x), gg, -0.0f)), rstd);
          x = pack_bf16x2_rn(y.x, y.y);
        }
      }
    };
    auto all_gathered = [&]() {          // (this warp's last chunk is in registers)
      if (nxt < npairs) load_slot(0, first);
      set_sync();
    };
    const uint32_t ql = 8u * lane, sl = 16u * (lane & 1) + 512u * (lane >> 2);       // (this lane's place in chunk 0)
    const bool word_lane = (lane & 2) == 0 && (has1 || (lane & 1) == 0);
    int cb = turn;
    if (TW > 4) turn = turn + 1 == TW ? 0 : turn + 1;
#pragma unroll 1
    for (; cb < plain_chunks; cb += TW) {
      uint32_t w[16];
      const uint32_t at = offs_l + 512u * (uint32_t)cb;
      gather(at, w);
      if (cb + TW >= chunks) all_gathered();
      if (RMS) normalise(at + 2u * (uint32_t)p.KQ, w);
      uint32_t codes;
      float2 dec, rcp;
      scale_of_pair_fma(amax_pair_h(w), codes, dec, rcp);
      uint2 c0, c1;
      encode_pair(w, rcp.x, rcp.y, c0, c1);
      uint8_t* q = q0 + (ql + 256u * (uint32_t)cb);
      *reinterpret_cast<uint2*>(q) = c0;
      if (has1) *reinterpret_cast<uint2*>(q + row_bytes) = c1;
      // four scale bytes of a row form a word: lanes 4 i and 4 i + 1 store those of the two rows
      const uint32_t tv = __byte_perm(codes, __shfl_xor_sync(0xffffffffu, codes, 1), sel1);
      const uint32_t word = __byte_perm(tv, __shfl_xor_sync(0xffffffffu, tv, 2), sel2);
      if (word_lane) *reinterpret_cast<uint32_t*>(sf0 + (sl + 4096u * (uint32_t)cb)) = word;
    }
#pragma unroll 1
    for (; cb < chunks; cb += TW) {      // chunks with critical groups, or that reach beyond the last group
      const int g = 32 * cb + lane, jc = g - G0;
      const uint32_t at = offs_l - 16u * lane + 16u * (uint32_t)min(g, G - 1);
      uint32_t w[16];
      gather(at, w);
      if (cb + TW >= chunks) all_gathered();
      if (RMS) normalise(at + 2u * (uint32_t)p.KQ, w);
      uint32_t codes;
      float2 dec, rcp, raw;
      scale_of_pair_fma(amax_pair_h(w), codes, dec, rcp, &raw);
      uint2 c0, c1;
      encode_pair(w, rcp.x, rcp.y, c0, c1);
      const bool critical = jc >= 0;
      const uint32_t col = critical ? (mode32 ? (uint32_t)(G0 + ((jc >> 1) << 2) + (jc & 1)) : (uint32_t)(g + jc)) : (uint32_t)g;
      auto put_codes = [&](uint32_t c) {
        const uint32_t sf_at = ((c >> 2) << 9) | (c & 3u);
        *reinterpret_cast<uint2*>(q0 + 8u * c) = c0;
        sf0[sf_at] = (uint8_t)codes;
        if (has1) {
          *reinterpret_cast<uint2*>(q0 + row_bytes + 8u * c) = c1;
          sf0[sf_at + 16] = (uint8_t)(codes >> 8);
        }
      };
      if (g < G) put_codes(col);
      if (critical && g < G) {
        // the re-quantized residual (or, for weights, a copy of the main codes)
        if (!is_weight) {
          if (mode32) dec = raw;         // against the un-rounded fp32 scale
          residual_pair(w, c0, c1, dec.x, dec.y);
          scale_of_pair_fma(amax_pair_h(w), codes, dec, rcp);
          encode_pair(w, rcp.x, rcp.y, c0, c1);
        }
        put_codes(col + (mode32 ? 2u : 1u));
      }
    }
  }
}

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void st_cluster(uint32_t at, uint32_t rank, uint32_t v) {      // to the same place in another CTA's shared memory
  asm volatile("{\n.reg .b32 a;\nmapa.shared::cluster.u32 a, %0, %1;\nst.shared::cluster.u32 [a], %2;\n}" ::"r"(at), "r"(rank), "r"(v) : "memory");
}

// ------------------------------------------------------------------------------------------------
// Row kernel: R rows at a time per CTA, several small CTAs per SM.
//
// Bound: HBM (2*KQ + 9/16*(KQ+KE) bytes per row); what competes with it is shared-memory bandwidth and issue
// slots, and this organisation is the one that needs the least of both:
//  * the two rows are interleaved in shared memory (a word (row0, row1) per channel), so one shared load gathers a
//    channel of both;
//  * a thread keeps the same GPT groups for all the rows it meets: their 16 GPT (swizzled) positions stay in
//    registers, two per register, and no offset table is read;
//  * rows go from global memory through registers straight into the interleaved buffer (no staging copy), with
//    the next unit's loads issued before the current unit is gathered (PF) and the rows after that pulled into L2;
//  * no roles and no rings: the CTAs of an SM are in different phases, which hides the barriers and the latency.
// A warp stores 256 contiguous bytes of codes per row; the scale bytes of four neighbouring groups are brought
// together with two shuffles and leave as one 32-bit word per row.
// RMSNorm: thread t holds chunks t and t + KQ/16, the reference's assignment and summation order (T == KQ/16).
// BY: what a launch does by the way.  Asked for at run time, both cost every launch that wants neither 0.1 us (us, asked for / this:
// plain 1 x 512 2.09 / 1.99, 16 x 5120 2.60 / 2.52; divided by a scale 200 x 4096 3.15 / 3.07, 444 x 5120 4.87 / 4.77; grouped 200 x 2048
// 3.77 / 3.65).  The fused RMSNorm always has the loop that clears: over none it costs nothing there (1.000 in the mean of 42 sizes).
constexpr int MAX_CLUSTER = 8;                  // (as many CTAs as any device takes)
// BY_BYTES: scales that begin off a 4-byte boundary, byte by byte, of rows narrower than the kernel of many rows takes (asked for at run time, by a
// bit of the address or a parameter, it cost every launch up to 0.1 us: fused RMSNorm 16 x 2048 2.74 / 2.87, grouped 74 x 1024 3.56 / 3.62).
enum { BY_NOTHING, BY_CLEAR, BY_OWN_MAX, BY_BYTES };      // so.clear set to zero; the maximum of the tensor itself taken first
// CLUSTERS: the maximum by clusters, a launch of MAX_CLUSTER CTAs each.  CPT: 16-byte chunks per thread and row; two per group of the thread, or more where
// CTAs share rows (see launch_rows).
template <int GPT, int CPT, bool RMS, bool SCALED, bool GROUPED, bool PF, int MAXT, int MINB, bool CLUSTERS, int BY>
__global__ void __launch_bounds__(MAXT, MINB) arcq_quantize_rows_kernel(const QuantParams p, const ScaleOptions so, const int share) {
  static_assert(BY != BY_OWN_MAX || (SCALED && !GROUPED), "the maximum of one tensor");
  static_assert(BY == BY_OWN_MAX || !CLUSTERS, "clusters take a maximum");
  constexpr int R = 2;                                          // rows of a unit
  constexpr bool WIDE = CPT > 2;
  static_assert(!RMS || (GPT == 1 && CPT == 2), "RMSNorm: one group per thread");
  extern __shared__ __align__(16) uint8_t smem[];
  const int tid = threadIdx.x, T = blockDim.x, lane = tid & 31, warp = tid >> 5;
  const int KQ = p.KQ, G = p.G, G0 = p.G0, nchunks = p.nchunks;
  uint8_t* buf = smem;                                          // [KQ][R] bf16
  float* psum = reinterpret_cast<float*>(smem + (size_t)KQ * 2 * R);   // RMS: [R][T] partial sums, then [R] roots
  float* rstd_s = psum + R * T;
  const bool mode32 = p.mode == 32, is_weight = p.is_weight != 0;
  const uint32_t row_bytes = (uint32_t)(KQ + p.KE) >> 1;

  if (CLUSTERS) cluster_arrive();                               // (waited for before the first remote store)
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // ---- the rows: one run, or `ngroups` runs (units of R rows are counted through all of them)
  // Lane l of every warp holds runs l and l + 32 (at most 64): first row, rows, and the units up to and including the run,
  // so that the run of a unit is found by a ballot.  (One round trip to memory: 256 rows over 64 runs 11.5 -> 6.0 us
  // against walking the table run by run.)
  const int ng = GROUPED ? p.ngroups : 1;
  uint32_t t_row0[2] = {0, 0}, t_rows[2] = {0, 0}, t_end[2] = {0, 0};
  uint32_t unit, unit_end, step;
  // Of the rows it stages a CTA of wide rows quantizes the groups [g_begin, g_end) (see launch_rows).
  const int g_begin = WIDE ? (int)blockIdx.y * share : 0, g_end = WIDE ? min(G, g_begin + share) : G;
  if (!GROUPED) {
    unit = blockIdx.x;
    unit_end = ((uint32_t)p.rows + R - 1) / R;
    step = gridDim.x;
  } else {      // a contiguous share: few changes of the run, and with it of the channel order
    uint32_t before = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = lane + 32 * h;
      if (e < ng) {
        t_row0[h] = (uint32_t)p.groups[e];
        t_rows[h] = (uint32_t)p.groups[ng + e];
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t inc = (t_rows[h] + R - 1) / R;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += v;
      }
      t_end[h] = before + inc;
      before = __shfl_sync(0xffffffffu, t_end[h], 31);
    }
    unit = (uint32_t)((unsigned long long)before * blockIdx.x / gridDim.x);
    unit_end = (uint32_t)((unsigned long long)before * (blockIdx.x + 1) / gridDim.x);
    step = 1;
  }
  // (run, first unit of the run) of the unit being worked on
  int e_cur = GROUPED ? -1 : 0;
  uint32_t e_first = 0, e_units = GROUPED ? 0 : unit_end, e_rows = GROUPED ? 0 : (uint32_t)p.rows, e_row0 = 0;
  auto seek = [&](uint32_t u) {                                // (whole warps) -> true if the run changed
    if (!GROUPED || u < e_first + e_units) return false;
    e_cur = __popc(__ballot_sync(0xffffffffu, t_end[0] <= u)) + __popc(__ballot_sync(0xffffffffu, t_end[1] <= u));
    const int h = e_cur >> 5, l = e_cur & 31;
    e_row0 = __shfl_sync(0xffffffffu, h ? t_row0[1] : t_row0[0], l);
    e_rows = __shfl_sync(0xffffffffu, h ? t_rows[1] : t_rows[0], l);
    e_units = (e_rows + R - 1) / R;
    e_first = __shfl_sync(0xffffffffu, h ? t_end[1] : t_end[0], l) - e_units;
    return true;
  };

  // ---- the tensor's divisor: given (times a factor), or from the partial maxima of the pass before
  float sc = 1.0f, rsc = 1.0f;
  bool fast = true;
  auto set_scale = [&](float s) {
    // torch's CUDA kernel for (bf16 tensor) / (fp32 scalar tensor) loads the divisor as bf16
    sc = __uint_as_float(pack_bf16x2_rn(s, 0.f) << 16);
    rsc = __frcp_rn(sc);
    fast = div_by_reciprocal_ok(sc);
  };
  if (SCALED) {
    if (BY == BY_OWN_MAX) {                   // (once this thread's rows and order are on their way)
    } else if (so.npartials > 0) {
      const float m = partials_max(p.scale, so.npartials, lane) * so.factor;
      if (blockIdx.x == 0 && tid == 0 && so.out != nullptr) so.out[0] = m;
      set_scale(m);
    } else {
      if (so.out != nullptr && blockIdx.x == 0)
        for (int e = tid; e < ng; e += T) so.out[e] = p.scale[e] * so.factor;
      if (!GROUPED) set_scale(*p.scale * so.factor);
    }
  }

  // ---- the channel order of this thread's groups
  uint32_t off[GPT][8];
  auto load_order = [&](const int16_t* idx) {
#pragma unroll
    for (int j = 0; j < GPT; ++j) {
      const int g = min(g_begin + tid + j * T, G - 1);
      if (idx == nullptr) {
#pragma unroll
        for (int k = 0; k < 8; ++k) off[j][k] = word_offset(16 * g + 2 * k) | (word_offset(16 * g + 2 * k + 1) << 16);
      } else if ((reinterpret_cast<uintptr_t>(idx) & 15u) == 0) {
        const uint4 lo = reinterpret_cast<const uint4*>(idx)[2 * g], hi = reinterpret_cast<const uint4*>(idx)[2 * g + 1];
        const uint32_t ww[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
        for (int k = 0; k < 8; ++k) off[j][k] = word_offset(ww[k] & 0xffffu) | (word_offset(ww[k] >> 16) << 16);
      } else {
#pragma unroll
        for (int k = 0; k < 8; ++k)
          off[j][k] = word_offset((uint32_t)(uint16_t)idx[16 * g + 2 * k]) | (word_offset((uint32_t)(uint16_t)idx[16 * g + 2 * k + 1]) << 16);
      }
    }
  };
  // RMSNorm gains of this thread's sixteen channels, kept packed (two bf16 per register)
  uint4 gn[2];
  if (RMS) {
    gn[0] = reinterpret_cast<const uint4*>(p.gamma)[tid];
    gn[1] = reinterpret_cast<const uint4*>(p.gamma)[tid + T];
  }

  uint4 a[R][CPT];
  auto in_row = [&](uint32_t out_row) -> const uint4* {
    const uint32_t r = GROUPED && p.row_map != nullptr ? (uint32_t)p.row_map[out_row] : out_row;
    return reinterpret_cast<const uint4*>(p.x + (size_t)r * (size_t)KQ);
  };
  auto load_unit = [&](uint32_t row0, uint32_t rows_here) {     // rows row0 .. row0 + rows_here of the output numbering
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const uint4* src = (uint32_t)i < rows_here ? in_row(row0 + i) : nullptr;
#pragma unroll
      for (int j = 0; j < CPT; ++j) {
        const int c = tid + j * T;
        a[i][j] = (src != nullptr && c < nchunks) ? ldg_stream(src + c) : make_uint4(0, 0, 0, 0);
      }
    }
  };
  auto prefetch_l2 = [&](uint32_t row0, uint32_t rows_here) {
    if ((uint32_t)tid < rows_here)
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(reinterpret_cast<uint64_t>(in_row(row0 + tid))), "r"((uint32_t)(KQ * 2)) : "memory");
  };

  auto clear_for_next = [&]() {      // (last: in front of the loads it cost 0.05 us of a call)
    if (BY == BY_CLEAR && blockIdx.x == 0)
      for (int i = tid; i < so.nclear; i += T) so.clear[i] = 0.f;
  };
  if (BY != BY_OWN_MAX && unit >= unit_end) { clear_for_next(); return; }
  auto rows_of = [&](uint32_t u) -> uint32_t { return min((uint32_t)R, e_rows - (u - e_first) * R); };
  seek(unit);
  auto new_run = [&]() {
    load_order(p.idx == nullptr ? nullptr : p.idx + (size_t)e_cur * (size_t)KQ);
    if (SCALED && GROUPED) set_scale(p.scale[e_cur] * so.factor);
  };
  // Rows and order ahead of the tensor's own maximum where there are registers for both: not with two groups a thread (16 x 14 336 0.8 us slower), nor where
  // every CTA takes the whole maximum and three share an SM (4 x 4096 3.79 / 3.83, 8 x 4096 3.91 / 3.97, 16 x 256 3.05 / 3.30, after / ahead of it).
  constexpr bool EARLY = PF && (BY != BY_OWN_MAX || CLUSTERS || WIDE);
  if (EARLY && (BY != BY_OWN_MAX || unit < unit_end)) load_unit(e_row0 + (unit - e_first) * R, rows_of(unit));
  if (EARLY || BY != BY_OWN_MAX) new_run();
  if constexpr (BY == BY_OWN_MAX) {          // a small tensor: its maximum, taken by every cluster (or CTA alone) for itself
    const uint4* x4 = reinterpret_cast<const uint4*>(p.x);
    const int nvec = (int)p.rows * nchunks;
    constexpr int C = CLUSTERS ? MAX_CLUSTER : 1;
    const int every = C * T, rank = CLUSTERS ? (int)cluster_ctarank() : 0;
    const uint32_t keep = is_weight ? 0xffffffffu : 0x7fff7fffu;     // (weights: the signed maximum)
    uint32_t m = is_weight ? 0xff80ff80u : 0u;
    auto take = [&](uint32_t w) { asm("max.NaN.bf16x2 %0, %0, %1;" : "+r"(m) : "r"(w & keep)); };
    constexpr int IN = 4;
    for (int i = rank * T + tid; i < nvec; i += IN * every) {
      uint4 v[IN];
#pragma unroll
      for (int k = 0; k < IN; ++k) v[k] = __ldcg(x4 + min(i + k * every, nvec - 1));
#pragma unroll
      for (int k = 0; k < IN; ++k) { take(v[k].x); take(v[k].y); take(v[k].z); take(v[k].w); }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) take(__shfl_xor_sync(0xffffffffu, m, d));
    uint32_t* red = reinterpret_cast<uint32_t*>(smem);       // [16 warps][CTAs of the cluster]
    if (lane == 0) red[warp] = m;
    __syncthreads();
    for (int w = 0; w < (T >> 5); ++w) take(red[w]);
    if (CLUSTERS) {
      cluster_wait();                                         // (all have started)
      if (tid < C) st_cluster(smem_addr(red + 16) + 4u * rank, (uint32_t)tid, m);
      __syncwarp();
      cluster_arrive();
      cluster_wait();
      for (int w = 0; w < C; ++w) take(red[16 + w]);
    }
    __syncthreads();                                          // (the rows are about to be staged there)
    const float lo = bf16lo(m), hi = bf16hi(m), top = (lo != lo || hi != hi) ? __uint_as_float(0x7fc00000u) : fmaxf(lo, hi);
    if (blockIdx.x == 0 && tid == 0 && so.out != nullptr) so.out[0] = top * so.factor;
    set_scale(top * so.factor);
    if (PF && !EARLY && unit < unit_end) load_unit(e_row0 + (unit - e_first) * R, rows_of(unit));
    if (!EARLY) new_run();
  }

  for (; unit < unit_end; unit += step) {
    const uint32_t row0 = e_row0 + (unit - e_first) * R, nrows = rows_of(unit);
    if (!PF) {
      load_unit(row0, nrows);
      if (unit + step < e_first + e_units && unit + step < unit_end) prefetch_l2(row0 + step * R, rows_of(unit + step));
    }
    float rstd[R];
    if (RMS) {
#pragma unroll
      for (int i = 0; i < R; ++i) {
        float ss = 0.f;   // x*x is exact in fp32, so each step rounds once, like the fp32 FMA
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const uint32_t w[4] = {a[i][j].x, a[i][j].y, a[i][j].z, a[i][j].w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            ss = fma_bf16(half_lo(w[k]), half_lo(w[k]), ss);
            ss = fma_bf16(half_hi(w[k]), half_hi(w[k]), ss);
          }
        }
        psum[i * T + tid] = ss;
      }
      __syncthreads();            // (also: everyone has gathered the previous unit)
      for (int i = warp; i < R; i += (T >> 5)) {
        const float t = rms_tree(psum + i * T, T, lane);
        if (lane == 0) rstd_s[i] = __frsqrt_rn(__fadd_rn(__fdiv_rn(t, (float)KQ), p.eps));
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < R; ++i) rstd[i] = rstd_s[i];
    } else {
      __syncthreads();            // everyone has gathered the previous unit
    }
    // ---- interleave (and normalise, or divide) into the buffer
#pragma unroll
    for (int j = 0; j < CPT; ++j) {
      const int c = tid + j * T;
      if (c < nchunks) {
        uint32_t o[8];            // a word (row 0, row 1) per channel
        const uint4 x0 = a[0][j], x1 = a[1][j];
        const uint32_t wa[4] = {x0.x, x0.y, x0.z, x0.w}, wb[4] = {x1.x, x1.y, x1.z, x1.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (RMS) {
            // bf16 x bf16 is exact in fp32; then one rounding by rstd (both rows in one FMUL2), one to bf16
            const uint4 g8 = gn[j & 1];
            const uint32_t gw = k == 0 ? g8.x : (k == 1 ? g8.y : (k == 2 ? g8.z : g8.w));
            const uint16_t ga = half_lo(gw), gb = half_hi(gw);
            const float2 r2 = make_float2(rstd[0], rstd[1]);
            const float2 n0 = __fmul2_rn(make_float2(fma_bf16(half_lo(wa[k]), ga, -0.0f), fma_bf16(half_lo(wb[k]), ga, -0.0f)), r2);
            const float2 n1 = __fmul2_rn(make_float2(fma_bf16(half_hi(wa[k]), gb, -0.0f), fma_bf16(half_hi(wb[k]), gb, -0.0f)), r2);
            o[2 * k] = pack_bf16x2_rn(n0.x, n0.y);
            o[2 * k + 1] = pack_bf16x2_rn(n1.x, n1.y);
          } else if (SCALED) {
            div_pair_words(wa[k], wb[k], sc, rsc, fast, o[2 * k], o[2 * k + 1]);
          } else {
            o[2 * k] = __byte_perm(wa[k], wb[k], 0x5410);
            o[2 * k + 1] = __byte_perm(wa[k], wb[k], 0x7632);
          }
        }
        uint4* b4 = reinterpret_cast<uint4*>(buf);
        b4[swz16(2u * c)] = make_uint4(o[0], o[1], o[2], o[3]);
        b4[swz16(2u * c + 1u)] = make_uint4(o[4], o[5], o[6], o[7]);
      }
    }
    __syncthreads();
    // ---- what comes next is on its way while this unit is quantized
    const uint32_t e_G0 = (uint32_t)G0;
    const uint32_t nxt = unit + step;
    bool changed = false;
    if (PF && nxt < unit_end) {
      changed = seek(nxt);
      const uint32_t nrow0 = e_row0 + (nxt - e_first) * R;
      load_unit(nrow0, rows_of(nxt));
      if (nxt + step < e_first + e_units && nxt + step < unit_end) prefetch_l2(nrow0 + step * R, rows_of(nxt + step));
    }
    // ---- gather and quantize this thread's groups
    uint8_t* qrow = p.q + (size_t)row0 * row_bytes;
    uint8_t* sfrow = p.sf + sf_row_base(row0, p.natoms);       // row i of the unit: + 16 i
#pragma unroll
    for (int j = 0; j < GPT; ++j) {
      const int g = g_begin + tid + j * T;
      if (WIDE && (g & ~31) >= g_end) break;                   // (whole warps)
      const bool live = g < g_end;
      auto gather = [&](uint32_t (&w)[16]) {
#pragma unroll
        for (int k = 0; k < 16; ++k)
          w[k] = *reinterpret_cast<const uint32_t*>(buf + ((k & 1) ? off[j][k >> 1] >> 16 : off[j][k >> 1] & 0xffffu));
      };
      uint32_t w[16];
      gather(w);
      const int jc = g - (int)e_G0;
      const bool critical = jc >= 0;
      uint32_t col = (uint32_t)g;
      if (critical) col = mode32 ? (uint32_t)((int)e_G0 + ((jc >> 1) << 2) + (jc & 1)) : (uint32_t)(g + jc);
      uint32_t codes;                                          // scale code of row i in byte i
      {
        float2 dec, rcp;
        scale_of_pair_fma(amax_pair_h(w), codes, dec, rcp);
        uint2 c0, c1;
        encode_pair(w, rcp.x, rcp.y, c0, c1);
        uint8_t* q0 = qrow + 8u * col;
        if (live) *reinterpret_cast<uint2*>(q0) = c0;
        if (live && nrows > 1) *reinterpret_cast<uint2*>(q0 + row_bytes) = c1;
      }
      // scale bytes: four plain groups side by side form a 32-bit word per row
      {
        const uint32_t x = __shfl_xor_sync(0xffffffffu, codes, 1);
        const uint32_t t = (lane & 1) ? __byte_perm(x, codes, 0x7351) : __byte_perm(codes, x, 0x6240);   // row 1 / 0
        const uint32_t y = __shfl_xor_sync(0xffffffffu, t, 2);
        const uint32_t word = (lane & 2) ? __byte_perm(y, t, 0x7632) : __byte_perm(t, y, 0x5410);
        const uint32_t gq = (uint32_t)g & ~3u;
        if (BY != BY_BYTES && gq + 3 < e_G0) {                 // (G0 <= G: all four lanes are live)
          const uint32_t i = (uint32_t)lane & 3u;              // this lane's row of the unit
          if (i < nrows) *reinterpret_cast<uint32_t*>(sfrow + 16u * i + ((gq >> 2) << 9)) = word;
        } else if (live) {
          uint8_t* s0 = sfrow + (((col >> 2) << 9) | (col & 3u));
#pragma unroll
          for (int i = 0; i < R; ++i)
            if ((uint32_t)i < nrows) s0[16 * i] = (uint8_t)(codes >> (8 * i));
        }
      }
      if (critical && live) {
        // the re-quantized residual (or, for weights, a copy of the main codes)
        const uint32_t rcol = col + (mode32 ? 2u : 1u);
        uint32_t v[16];
        gather(v);
        uint32_t rc;
        float2 dec, rcp, raw;
        scale_of_pair_fma(amax_pair_h(v), rc, dec, rcp, &raw);
        uint2 c0, c1;
        encode_pair(v, rcp.x, rcp.y, c0, c1);
        if (!is_weight) {
          if (mode32) dec = raw;        // against the un-rounded fp32 scale
          residual_pair(v, c0, c1, dec.x, dec.y);
          float2 rdec, rrcp;
          scale_of_pair_fma(amax_pair_h(v), rc, rdec, rrcp);
          encode_pair(v, rrcp.x, rrcp.y, c0, c1);
        }
        uint8_t* q0 = qrow + 8u * rcol;
        uint8_t* s0 = sfrow + (((rcol >> 2) << 9) | (rcol & 3u));
        *reinterpret_cast<uint2*>(q0) = c0;
        s0[0] = (uint8_t)rc;
        if (nrows > 1) {
          *reinterpret_cast<uint2*>(q0 + row_bytes) = c1;
          s0[16] = (uint8_t)(rc >> 8);
        }
      }
    }
    if (PF) {
      if (changed) new_run();
    } else if (nxt < unit_end && seek(nxt)) {
      new_run();
    }
  }
  clear_for_next();
}

// `nvec` 16-byte words from src to each of n destinations: the codes and scale tiles a rank has just made of
// its token rows, to the same place in its peers' gathered buffers (peer memory over NVLink).  Storing them from
// inside the quantizer as they are made was measured no faster (the transfer is bound by NVLink either way) and
// needs single-byte stores for the scales, a packet each.
struct BroadcastDests {
  uint4* p[7];
};
__global__ void arcq_broadcast_kernel(const uint4* __restrict__ src, const BroadcastDests dst, int n, long long nvec) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nvec; i += (long long)gridDim.x * blockDim.x) {
    const uint4 v = src[i];
    for (int d = 0; d < n; ++d) dst.p[d][i] = v;
  }
}

__global__ void arcq_absmax_kernel(const uint4* __restrict__ x, long long nvec, const uint16_t* tail,
                                   int ntail, unsigned int* out) {
  uint32_t m = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nvec;
       i += (long long)gridDim.x * blockDim.x) {
    uint4 v = ldg_stream(x + i);
    m = max_u16x2(m, v.x & 0x7fff7fffu);
    m = max_u16x2(m, v.y & 0x7fff7fffu);
    m = max_u16x2(m, v.z & 0x7fff7fffu);
    m = max_u16x2(m, v.w & 0x7fff7fffu);
  }
  uint32_t r = max(m & 0xffffu, m >> 16);
  if (blockIdx.x == 0 && (int)threadIdx.x < ntail) r = max(r, (uint32_t)tail[threadIdx.x] & 0x7fffu);
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) r = max(r, __shfl_xor_sync(0xffffffffu, r, d));
  // non-negative floats order like their bit patterns
  if ((threadIdx.x & 31) == 0) atomicMax(out, r << 16);
}

// One maximum per CTA of a bf16 tensor (16-byte aligned): of the magnitudes, or signed.  The row kernel that follows
// takes the maximum of them, so nothing has to be initialised and no atomic is needed.  The tensor is walked from its
// end: the row kernel then starts with the rows this pass has left in L2.
template <bool SIGNED>
__global__ void __launch_bounds__(512) arcq_max_partials_kernel(const uint4* x, long long nvec, float* __restrict__ out) {
  __shared__ uint32_t red[16];
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const long long step = (long long)gridDim.x * blockDim.x;
  uint32_t m = SIGNED ? 0xff80ff80u : 0u;
  auto take = [&](uint32_t w) {
    if (SIGNED) asm("max.NaN.bf16x2 %0, %0, %1;" : "+r"(m) : "r"(w));
    else m = max_u16x2(m, w & 0x7fff7fffu);
  };
  // IN loads in flight per thread; what is left over at the end goes one by one.
  constexpr int IN = 4;
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const uint4* at = x + (nvec - 1 - i);
#pragma unroll 1
  for (; i + (IN - 1) * step < nvec; i += IN * step, at -= IN * step) {
    uint4 v[IN];
#pragma unroll
    for (int k = 0; k < IN; ++k) v[k] = at[-k * step];
#pragma unroll
    for (int k = 0; k < IN; ++k) { take(v[k].x); take(v[k].y); take(v[k].z); take(v[k].w); }
  }
#pragma unroll 1
  for (; i < nvec; i += step, at -= step) {
    const uint4 v = *at;
    take(v.x); take(v.y); take(v.z); take(v.w);
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) take(__shfl_xor_sync(0xffffffffu, m, d));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) take(red[w]);
    const float lo = __uint_as_float(m << 16), hi = __uint_as_float(m & 0xffff0000u);
    out[blockIdx.x] = (lo != lo || hi != hi) ? __uint_as_float(0x7fc00000u) : fmaxf(lo, hi);
  }
}

// The limit of a launch's dynamic shared memory belongs to the kernel on its device, not to the thread that sets it.  So it
// is always set to what the device has: set to the need of one call, a narrower call of another thread would lower it, and
// the next wide call of the thread that remembers having set it would be refused.
template <typename Kernel>
cudaError_t allow_shared_memory(Kernel kern, const DeviceInfo& di) {
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, di.max_smem_optin);
}

// Whether clusters may share the maximum of a small tensor: not under an SM limit, which a grid in clusters might not keep, and not of narrow
// rows, of which there are many CTAs, each to look at the same few lines (us, every CTA / clusters: 512 x 16 3.7 / 4.3, 130 x 32 3.4 / 3.7; two launches / clusters: 250 x 64
// 5.0 / 7.3, but 32 x 512 4.6 / 4.1).
static bool clusters_take_maximum(int G, const DeviceInfo& di) { return G >= 32 && di.num_sms == di.all_sms; }

// CTAs that share each of `grid` pairs of wide rows.  No more than twelve clusters, one CTA per SM: sixteen are not resident at once (32 x 11 008 over its
// own maximum with 128 CTAs 10.6 us, with 64 5.8).
static int row_parts(long long grid, bool clusters, const DeviceInfo& di) {
  const int most = clusters ? 12 * MAX_CLUSTER : di.num_sms;
  int parts = 1;
  while (parts < 8 && 2 * parts * grid <= most) parts *= 2;
  return parts;
}

template <int GPT, int CPT, bool RMS, bool SCALED, bool GROUPED, bool PF, int MAXT, int MINB, bool CLUSTERS, int BY>
int launch_rows(const QuantParams& p, const ScaleOptions& so, long long units, int T, const DeviceInfo& di, cudaStream_t stream) {
  constexpr int R = 2;
  auto kern = arcq_quantize_rows_kernel<GPT, CPT, RMS, SCALED, GROUPED, PF, MAXT, MINB, CLUSTERS, BY>;
  const size_t smem = (size_t)p.KQ * 2 * R + (RMS ? (size_t)(R * T + R) * sizeof(float) : 64);
  // the attribute and the occupancy query cost host time: once per (device, block size, shared memory)
  static thread_local int c_dev = -1, c_threads = 0, c_occ = 0;
  static thread_local size_t c_smem = 0;
  if (c_dev != di.device || c_threads != T || c_smem != smem) {
    int occ = 0;
    ARCQ_CUDA_TRY(allow_shared_memory(kern, di));
    ARCQ_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, T, smem));
    c_dev = di.device; c_threads = T; c_smem = smem; c_occ = occ;
  }
  if (c_occ < 1) return ARCQ_ERR_UNSUPPORTED_K;
  // No more CTAs per SM than the units need, by shared memory asked for: set up early, while the kernel before still holds
  // most SMs, several of them would crowd on the first SMs that come free
  // (290 rows of 4096 channels, call after call 3.8 -> 2.7 us; with RMSNorm and the GEMM [6144, 4224] 17.3 -> 15.3).
  const long long need = (units + di.num_sms - 1) / di.num_sms;
  const int per_sm = need < c_occ ? (int)need : c_occ;
  const size_t share = per_sm < c_occ ? ((size_t)di.max_smem_optin + 1024) / (per_sm + 1) : 0;
  long long grid = di.resident(per_sm);
  if (grid > (p.rows + R - 1) / R) grid = (p.rows + R - 1) / R;
  // A few wide rows: up to eight CTAs stage the same rows and quantize a part of their groups each, instead of two groups per thread in one
  // CTA (14 336 channels, us, one CTA per pair of rows / this: plain 16 rows 4.6 / 3.6, 74 rows 4.8 / 3.9, 148 rows 4.8 / 4.2.
  // Rows of 4096 channels, one group per thread already, gain nothing.)
  if (CLUSTERS) grid = (grid + MAX_CLUSTER - 1) / MAX_CLUSTER * MAX_CLUSTER;
  const int parts = CPT > 2 && !GROUPED ? row_parts(grid, CLUSTERS, di) : 1;
  const int groups_each = ((p.G + parts - 1) / parts + 31) & ~31;
  if (CPT > 2 * GPT && groups_each > GPT * T) return ARCQ_ERR_UNSUPPORTED_K;      // (chosen where CTAs share rows only)
  // Programmatic dependent launch: the grid may be set up while the previous kernel of the stream is
  // still draining; the kernel itself waits (griddepcontrol.wait) before it touches global memory.
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid, (unsigned)((p.G + groups_each - 1) / groups_each));
  cfg.blockDim = dim3((unsigned)T);
  cfg.dynamicSmemBytes = std::max(smem, share);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = di.early_start();
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim = {MAX_CLUSTER, 1, 1};
  cfg.attrs = attr;
  cfg.numAttrs = CLUSTERS ? 2 : 1;
  ARCQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, p, so, groups_each));
  return ARCQ_OK;
}

template <bool RMS, bool SCALED, int MG, int TW>
int launch_sets(const QuantParams& p, const ScaleOptions& so, const DeviceInfo& di, cudaStream_t stream) {
  auto kern = arcq_quantize_ws_kernel_sets<RMS, SCALED, MG, TW>;
  const size_t buffer = (size_t)p.KQ * 4;
  int nsets = WS_WARPS / TW;
  while (nsets > 1 && ws_fixed_bytes(RMS, TW, p.KQ, nsets) + nsets * buffer > (size_t)di.max_smem_optin) --nsets;
  // Where the sets of an SM take two pairs and more each, no more sets than share them evenly: the last round is a full one (2048 x 8192 12.6 ->
  // 11.7 us, fused RMSNorm 4096 x 4096 14.2 -> 13.8).  Of one round all sets are launched, for their threads set up the tables (900 x 4096 6.9 / 6.3).
  if (p.groups == nullptr) {
    const long long per_sm = (p.npairs + di.num_sms - 1) / di.num_sms, rounds = (per_sm + nsets - 1) / nsets;
    if (rounds > 1) nsets = (int)((per_sm + rounds - 1) / rounds);
  }
  const size_t smem = ws_fixed_bytes(RMS, TW, p.KQ, nsets) + nsets * buffer;
  static thread_local int c_dev = -1;      // (the attribute costs host time: once per device)
  if (c_dev != di.device) {
    ARCQ_CUDA_TRY(allow_shared_memory(kern, di));
    c_dev = di.device;
  }
  long long grid = di.resident(1);
  if (p.groups == nullptr && grid > p.npairs) grid = p.npairs;
  if (p.groups != nullptr && grid < p.ngroups) return ARCQ_ERR_BAD_SHAPE;      // every run needs a CTA
  return launch_dependent(kern, (unsigned)grid, (unsigned)(32 * nsets * TW), smem, di, stream, p, so);
}
// The warps of a set: as few as keep it at four slots (RMSNorm, where they are a power of two for the tree's sake: five), so that sets are many
// and their barriers cheap, and yet all 24 warps have a buffer.  us, with half as many / with these / with more: fused RMSNorm 8192 x 2048
// - / 13.6 / 14.4 (2), 16 384 x 4096 49.1 / 43.0 / 46.6 (4), 8192 x 5120 - / 28.5 / 33.2 (4), 16 384 x 8192 - / 81.2 / 89.7 (8); over a
// tensor's maximum 8192 x 5120 26.2 (2) / 25.7 / 29.3 (4), 8192 x 14 336 75.2 / 68.1 / -.
template <bool SCALED>
int launch_sets_plain(const QuantParams& p, const ScaleOptions& so, const DeviceInfo& di, cudaStream_t stream) {
  if (p.G <= 128) return launch_sets<false, SCALED, 128, 1>(p, so, di, stream);
  if (p.G <= 256) return launch_sets<false, SCALED, 256, 2>(p, so, di, stream);
  if (p.G <= 384) return launch_sets<false, SCALED, 384, 3>(p, so, di, stream);
  if (p.G <= 512) return launch_sets<false, SCALED, 512, 4>(p, so, di, stream);
  if (p.G <= 768) return launch_sets<false, SCALED, 768, 6>(p, so, di, stream);
  return launch_sets<false, SCALED, 1024, 8>(p, so, di, stream);
}
static int launch_sets_rms(const QuantParams& p, const ScaleOptions& so, const DeviceInfo& di, cudaStream_t stream) {
  if (p.G <= 128) return launch_sets<true, false, 128, 1>(p, so, di, stream);
  if (p.G <= 256) return launch_sets<true, false, 256, 2>(p, so, di, stream);
  if (p.G <= 320) return launch_sets<true, false, 320, 2>(p, so, di, stream);
  return launch_sets<true, false, 512, 4>(p, so, di, stream);
}

template <int CPT, int NBUF, int PAIRS, bool RMS, bool RAWIDX, int MAXT, int MINB>
int launch_variant(const QuantParams& p, int nt, size_t smem, const DeviceInfo& di, cudaStream_t stream) {
  auto kern = arcq_quantize_kernel<CPT, NBUF, PAIRS, RMS, RAWIDX, MAXT, MINB>;
  ARCQ_CUDA_TRY(allow_shared_memory(kern, di));
  int occ = 0;
  ARCQ_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, nt, smem));
  if (occ < 1) return ARCQ_ERR_UNSUPPORTED_K;
  const long long nunits = (p.npairs + PAIRS - 1) / PAIRS;
  long long grid = di.resident(occ);
  if (grid > nunits) grid = nunits;
  kern<<<(unsigned)grid, nt, smem, stream>>>(p);
  ARCQ_CUDA_TRY(cudaGetLastError());
  return ARCQ_OK;
}

}  // namespace

static int launch_quantize_one(const void* x, const void* gamma, float eps, const int16_t* idx, int64_t rows, int KQ,
                               int KE, int mode, int is_weight, uint8_t* q, uint8_t* sf, cudaStream_t stream,
                               const float* scale, const int* groups, int ngroups, const int* row_map, const ScaleOptions& so);

int launch_quantize(const void* x, const void* gamma, float eps, const int16_t* idx, int64_t rows, int KQ,
                    int KE, int mode, int is_weight, uint8_t* q, uint8_t* sf, cudaStream_t stream, const float* scale,
                    const int* groups, int ngroups, const int* row_map, uint8_t* const* q_extra,
                    uint8_t* const* sf_extra, int nextra, const ScaleOptions& so) {
  if (rows == 0) return ARCQ_OK;
  if (nextra > 0 && (rows % 128 || nextra > 7)) return ARCQ_ERR_BAD_SHAPE;   // whole scale tiles travel
  int rc = launch_quantize_one(x, gamma, eps, idx, rows, KQ, KE, mode, is_weight, q, sf, stream, scale, groups,
                               ngroups, row_map, so);
  if (rc != ARCQ_OK || nextra == 0) return rc;
  DeviceInfo di;
  rc = get_device_info(&di);
  if (rc != ARCQ_OK) return rc;
  BroadcastDests bq = {}, bs = {};
  for (int d = 0; d < nextra; ++d) {
    bq.p[d] = reinterpret_cast<uint4*>(q_extra[d]);
    bs.p[d] = reinterpret_cast<uint4*>(sf_extra[d]);
  }
  const long long nq = rows * (long long)((KQ + KE) / 2) / 16;
  const long long ns = (rows / 128) * (long long)(((KQ + KE) / 16 + 3) / 4) * 32;
  const long long cap = (long long)di.num_sms * 8;
  long long bl = (nq + 255) / 256;
  arcq_broadcast_kernel<<<(unsigned)(bl < cap ? bl : cap), 256, 0, stream>>>(reinterpret_cast<const uint4*>(q), bq,
                                                                            nextra, nq);
  bl = (ns + 255) / 256;
  arcq_broadcast_kernel<<<(unsigned)(bl < cap ? bl : cap), 256, 0, stream>>>(reinterpret_cast<const uint4*>(sf), bs,
                                                                            nextra, ns);
  ARCQ_CUDA_TRY(cudaGetLastError());
  return ARCQ_OK;
}

// Row kernel: little work per SM.  A unit is a pair of rows; there is no table to set up, and the CTAs of an SM hide one another's
// latency.  The line lies where a CTA would take a second unit (three CTAs of 256 threads per SM, more of narrower rows), a unit per SM where rows
// of one run are divided by a given scale and wider, two (four without a divisor of the caller's) of more than 512 groups.  us just below it, the
// kernel of many rows / this one:
//  * fused RMSNorm 16 x 4096 4.2 / 3.4, 888 x 4096 5.5 / 5.2, 1776 x 2048 5.4 / 5.3, 592 x 5120 5.6 / 5.3, 592 x 8192 6.7 / 6.2;
//  * plain 592 x 5120 4.2 / 4.2, 592 x 8192 5.2 / 5.0, 592 x 14 336 7.3 / 7.3, 1184 x 14 336 12.2 / 12.6;
//  * divided: 296 x 5120 4.3 / 3.6, 880 x 4096 4.8 / 5.2, over maxima 444 x 4096 4.2 / 4.0, 888 x 4096 4.8 / 5.1, 592 x 5120 4.7 / 5.1, 592 x 14 336
//    7.9 / 8.7, 1184 x 14 336 13.0 / 14.9;
//  * grouped, eight runs: 444 x 8192 6.0 / 7.0, 444 x 14 336 8.3 / 10.1, 592 x 14 336 9.9 / 11.0, 1100 x 4096 5.8 / 7.9, 1400 x 4096 6.5 / 8.1.
// (Open: it was drawn against the kernel in use before that of many rows, and where rows are divided it now holds on to too much, by 5 to 10 %, grouped by
// 10 to 35 %.)
struct RowLaunch {
  long long units;   // pairs of rows (grouped: as far as the host knows)
  int threads;       // of a CTA
  bool serves;
};
// given: rows of one run divided by a scale that the caller has.
static RowLaunch row_launch(int G, long long rows, int ngroups, bool given, const DeviceInfo& di) {
  const bool wide = G > 512;
  RowLaunch r;
  r.units = (std::max<long long>(rows - 256LL * ngroups, 1) + 1) / 2;
  r.threads = wide ? ((G + 1) / 2 + 31) / 32 * 32 : (G + 31) / 32 * 32;
  long long per_sm = (ngroups > 0 ? 6 : 3) * 256 / r.threads;
  if (r.threads > 256) per_sm = wide ? (given || ngroups > 0 ? 2 : 4) : (given ? 1 : 2);
  r.serves = r.units <= per_sm * di.num_sms;
  return r;
}

static int launch_quantize_one(const void* x, const void* gamma, float eps, const int16_t* idx, int64_t rows, int KQ,
                               int KE, int mode, int is_weight, uint8_t* q, uint8_t* sf, cudaStream_t stream,
                               const float* scale, const int* groups, int ngroups, const int* row_map, const ScaleOptions& so) {
  if (groups != nullptr && scale == nullptr) return ARCQ_ERR_NULL_POINTER;      // (every run is divided by a scale)
  DeviceInfo di;
  int rc = get_device_info(&di);
  if (rc != ARCQ_OK) return rc;

  QuantParams p;
  p.x = static_cast<const uint16_t*>(x);
  p.gamma = static_cast<const uint16_t*>(gamma);
  p.idx = idx;
  p.q = q;
  p.sf = sf;
  p.rows = rows;
  p.npairs = (rows + 1) / 2;
  p.KQ = KQ;
  p.KE = KE;
  p.G = KQ / 16;
  p.G0 = (KQ - KE) / 16;
  p.natoms = ((KQ + KE) / 16 + 3) / 4;
  p.nchunks = KQ / 8;
  p.mode = mode;
  p.is_weight = is_weight;
  p.eps = eps;
  p.scale = scale;
  p.groups = groups;
  p.ngroups = ngroups;
  p.row_map = row_map;

  const bool rms = gamma != nullptr;
  int nt = p.G;        // (RMSNorm: one reference thread per CUDA thread, which keeps the accumulation order)
  if (!rms) {
    const int gpt = (p.G + 511) / 512;
    nt = (((p.G + gpt - 1) / gpt) + 31) / 32 * 32;
    if ((p.nchunks + nt - 1) / nt > 8) return ARCQ_ERR_UNSUPPORTED_K;
  }
  const bool rawidx = KQ > 16384;
  const bool gamma_ok = !rms || (reinterpret_cast<uintptr_t>(gamma) & 15u) == 0;   // read with 128-bit loads
  const bool wide = p.G > 512;

  const bool given = scale != nullptr && groups == nullptr && so.npartials == 0 && so.out == nullptr;
  const RowLaunch r = row_launch(p.G, rows, groups != nullptr ? ngroups : 0, given, di);
  const long long units = r.units;
  const int T = r.threads;
  const bool own_max = so.npartials < 0;      // (decided by the caller, maybe under another SM limit: the row kernel it is)
  const bool words = (reinterpret_cast<uintptr_t>(sf) & 3u) == 0;        // scales of four groups may be stored at once: else the kernel of many rows
  if (gamma_ok && p.G <= 1024 && !(rms && wide) && (row_map == nullptr || groups != nullptr) && rows < (1LL << 30) &&
      ((r.serves && words) || own_max || (p.G < 32 && !rms))) {
#define ARCQ_ROWS(SC_, GR_, BY_)                                                                                    \
  {                                                                                                                 \
    if (wide) return launch_rows<2, 4, false, SC_, GR_, false, 512, 1, false, BY_>(p, so, units, T, di, stream);    \
    return T <= 256 ? launch_rows<1, 2, false, SC_, GR_, true, 256, 3, false, BY_>(p, so, units, T, di, stream)     \
                    : launch_rows<1, 2, false, SC_, GR_, true, 512, 1, false, BY_>(p, so, units, T, di, stream);    \
  }
    if (!words) {
      rc = so.nclear > 0 ? launch_clear(so.clear, so.nclear, stream) : ARCQ_OK;
      if (rc != ARCQ_OK) return rc;
      if (groups != nullptr) return launch_rows<1, 2, false, true, true, true, 256, 3, false, BY_BYTES>(p, so, units, T, di, stream);
      return scale != nullptr ? launch_rows<1, 2, false, true, false, true, 256, 3, false, BY_BYTES>(p, so, units, T, di, stream)
                              : launch_rows<1, 2, false, false, false, true, 256, 3, false, BY_BYTES>(p, so, units, T, di, stream);
    }
    if (groups != nullptr && so.nclear > 0) ARCQ_ROWS(true, true, BY_CLEAR)
    if (groups != nullptr) ARCQ_ROWS(true, true, BY_NOTHING)
    if (own_max) {
      // A tensor of more than 16 loads a thread: clusters (see launch_quantize_tensor_scale).
      const bool clusters = clusters_take_maximum(p.G, di) && rows * (long long)p.nchunks > 16LL * T;
      // CTAs that share wide rows have one group a thread: rows and order are asked for ahead of the maximum there too.
      if (wide && clusters) return launch_rows<1, 4, false, true, false, true, 512, 1, true, BY_OWN_MAX>(p, so, units, T, di, stream);
      if (wide && row_parts(units, false, di) > 1) return launch_rows<1, 4, false, true, false, true, 512, 1, false, BY_OWN_MAX>(p, so, units, T, di, stream);
      if (clusters)
        return T <= 256 ? launch_rows<1, 2, false, true, false, true, 256, 3, true, BY_OWN_MAX>(p, so, units, T, di, stream)
                        : launch_rows<1, 2, false, true, false, true, 512, 1, true, BY_OWN_MAX>(p, so, units, T, di, stream);
      ARCQ_ROWS(true, false, BY_OWN_MAX)
    }
    if (scale != nullptr) ARCQ_ROWS(true, false, BY_NOTHING)
    if (!rms) ARCQ_ROWS(false, false, BY_NOTHING)
    return T <= 256 ? launch_rows<1, 2, true, false, false, true, 256, 3, false, BY_CLEAR>(p, so, units, T, di, stream)
                    : launch_rows<1, 2, true, false, false, true, 512, 1, false, BY_CLEAR>(p, so, units, T, di, stream);
#undef ARCQ_ROWS
  }

  if (own_max) return ARCQ_ERR_UNSUPPORTED_K;      // (the kernels below have no maximum to divide by)
  // (Only the row kernel clears by the way: in the kernels below it cost registers that are all in use.)
  if (so.nclear > 0) {
    rc = launch_clear(so.clear, so.nclear, stream);
    if (rc != ARCQ_OK) return rc;
  }

  // (RMSNorm: one lane per 16-channel group, in whole warps - the reference's summation order)
  if (gamma_ok && p.G >= 32 && (!rms || (p.G % 32 == 0 && p.G >= 64)) && rows < (1LL << 30) && p.G <= (rms ? 512 : 1024)) {
    if (rms) return launch_sets_rms(p, so, di, stream);
    return scale != nullptr ? launch_sets_plain<true>(p, so, di, stream) : launch_sets_plain<false>(p, so, di, stream);
  }
  // the kernel below neither divides by the scale nor walks grouped rows nor follows a row map
  if (p.scale || p.groups || p.row_map) return ARCQ_ERR_UNSUPPORTED_K;

  const size_t table = 160 + (((size_t)KQ * (rawidx ? 2 : 4) + 15) & ~(size_t)15);
  auto smem_for = [&](int nbuf, int pairs) {
    return table + (rms ? (size_t)KQ * 4 + (size_t)2 * pairs * nt * sizeof(float) + 16 : 0) +
           (size_t)nbuf * pairs * KQ * 4;
  };
  if (rawidx)      // very wide rows: one buffer, loads not overlapped with the arithmetic
    return rms ? ARCQ_ERR_UNSUPPORTED_K : launch_variant<8, 1, 1, false, true, 512, 1>(p, nt, smem_for(1, 1), di, stream);
  const size_t smem = smem_for(2, 1);
  // Narrow rows: one row pair per iteration, three resident CTAs per SM (two pairs per iteration with
  // two resident CTAs were measured slower on B200: fewer warps to hide latency).
  if (rms) return nt <= 256 ? launch_variant<2, 2, 1, true, false, 256, 3>(p, nt, smem, di, stream)
                            : launch_variant<2, 2, 1, true, false, 512, 1>(p, nt, smem, di, stream);
  // (What is left are 2^30 rows and more: of more than 4096 channels, nine terabytes.)
  return nt <= 256 ? launch_variant<2, 2, 1, false, false, 256, 3>(p, nt, smem, di, stream) : ARCQ_ERR_BAD_SHAPE;
}

// x divided by the tensor's own scale, max / (448 * 6): the maximum as one partial result per CTA of a first pass
// (or `amax`, which the caller already has on the device), the rest of it in the quantizer's prologue.  The factor is
// the fp32 reciprocal, as torch's division of a tensor by a host scalar multiplies by it.
int launch_quantize_tensor_scale(const void* x, const float* amax, int is_weight, const int16_t* idx, int64_t rows, int KQ,
                                 int KE, int mode, uint8_t* q, uint8_t* sf, float* scale_out, float* scratch,
                                 cudaStream_t stream, const int* groups, int ngroups, const int* row_map, float* clear, int nclear) {
  if (KQ > 16384) return ARCQ_ERR_UNSUPPORTED_K;
  ScaleOptions so;
  so.factor = 1.0f / 2688.0f;
  so.out = scale_out;
  so.clear = clear;
  so.nclear = nclear;
  if (amax == nullptr) {
    DeviceInfo di;
    int rc = get_device_info(&di);
    if (rc != ARCQ_OK) return rc;
    const long long nvec = rows * (long long)KQ / 8;
    // A small tensor's maximum is taken by the CTAs of the row kernel: less than a second launch costs the device, and one launch less for
    // the host.  Up to 16 loads a thread by every CTA for itself, up to 64 by clusters of eight, eight loads a thread each (without clusters: up to 32
    // by every CTA).  us, two launches / every CTA / clusters: 4 x 4096 4.8 / 3.8 / 4.4, 16 x 4096 5.1 / 4.6 / 4.0, 32 x 4096 4.9 / 5.9 / 4.3, 16 x
    // 8192 5.4 / 5.5 / 4.8, 8 x 14 336 7.1 / 5.9 / 4.9, 16 x 14 336 6.1 / - / 5.3, 32 x 512 4.4 / - / 3.7.  Beyond eight loads each a third round of them
    // begins (with the registers of two groups a thread 20 x 14 336 6.3 / - / 6.5, 20 x 16 384 6.3 / - / 6.6).  Between 32 and 40 two launches stay (open: 20 x
    // 4096, at 40, says that clusters would be faster there too, 4.8 / - / 4.3).  In a graph behind another kernel, where the host's launches do not count, with
    // the GEMM: 20 x 4096 11.8 / - / 11.3, 24 x 8192 15.0 / - / 14.7, 10 x 14 336 13.6 / - / 13.6, 16 x 14 336 14.4 / - / 14.2 (with two groups a thread 14.2 and
    // 14.8).
    const RowLaunch r = row_launch(KQ / 16, rows, 0, false, di);
    const bool small = nvec <= 32LL * r.threads, fits = clusters_take_maximum(KQ / 16, di) && nvec >= 40LL * r.threads && nvec <= 64LL * r.threads;
    if (groups == nullptr && (small || fits) && r.serves && (reinterpret_cast<uintptr_t>(sf) & 3u) == 0) {
      so.npartials = -1;
      return launch_quantize(x, nullptr, 0.f, idx, rows, KQ, KE, mode, is_weight, q, sf, stream, scratch, groups, ngroups, row_map,
                             nullptr, nullptr, 0, so);
    }
    // four 16-byte loads per thread, at most three CTAs per SM
    long long grid = (nvec + 4 * 512 - 1) / (4 * 512);
    if (grid > di.resident(3)) grid = di.resident(3);
    if (grid > ARCQ_SCALE_SCRATCH) grid = ARCQ_SCALE_SCRATCH;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(512);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = di.early_start();
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    auto kern = is_weight ? arcq_max_partials_kernel<true> : arcq_max_partials_kernel<false>;
    ARCQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, static_cast<const uint4*>(x), nvec, scratch));
    so.npartials = (int)grid;
    amax = scratch;
  }
  return launch_quantize(x, nullptr, 0.f, idx, rows, KQ, KE, mode, is_weight, q, sf, stream, amax, groups, ngroups, row_map,
                         nullptr, nullptr, 0, so);
}

int launch_absmax(const void* x, int64_t n, float* out, int accumulate, cudaStream_t stream) {
  DeviceInfo di;
  int rc = get_device_info(&di);
  if (rc != ARCQ_OK) return rc;
  if (!accumulate) ARCQ_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(float), stream));
  if (n == 0) return ARCQ_OK;
  long long nvec = n / 8;
  int ntail = (int)(n - nvec * 8);
  const uint16_t* tail = static_cast<const uint16_t*>(x) + nvec * 8;
  long long blocks = (nvec + 255) / 256;
  long long cap = (long long)di.num_sms * 8;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  arcq_absmax_kernel<<<(unsigned)blocks, 256, 0, stream>>>(static_cast<const uint4*>(x), nvec, tail, ntail,
                                                          reinterpret_cast<unsigned int*>(out));
  ARCQ_CUDA_TRY(cudaGetLastError());
  return ARCQ_OK;
}

}  // namespace arcq
