// Block-scaled NVFP4 GEMM for sm_100a:  C[M,N] = bf16(alpha * (A.SFA)(B.SFB)^T), fp32 accumulation
// in tensor memory.  A [M,K/2] and B [N,K/2] hold packed e2m1 codes (K-major, two per byte), SFA/SFB
// hold one ue4m3 scale per 16 elements in 512-byte atoms of 128 rows x 4 scale columns - exactly
// what one 128-row, K=64 tcgen05 block-scaled MMA consumes, so an atom travels
// global -> shared (bulk copy) -> tensor memory (tcgen05.cp) without being touched by a thread.
//
// Organisation (one CTA per SM, persistent over output tiles of 128 x BN):
//   warp 0    producer: per K stage (256 elements = one 128-byte swizzled row) two tiled TMA loads
//             (A box 128 rows, B box BN rows, 128B swizzle) and the bulk copies of the scale atoms,
//             all completing on the stage's "full" mbarrier
//   warp 1    tensor-core issuer: one thread copies the stage's scale atoms into TMEM and issues
//             four tcgen05.mma.kind::mxf4nvf4.block_scale (M128 x BN x K64) per stage;
//             tcgen05.commit releases the stage ("empty") and finally publishes the accumulator
//   warps 2-5 epilogue: tcgen05.ld 32 lanes x 32 columns, scale by alpha, convert to bf16, 64-byte
//             contiguous global stores per thread; then hand the accumulator back
// Replaces the CUTLASS sm_120 instantiation of kernels/src/nvfp4.cu in ARCQuant.
//
// Every wait on an mbarrier is bounded: after ~2 s without progress the waiting thread raises a
// CTA-wide abort flag, records ARCQ_ERR_TIMEOUT in a device word the host can poll, and all roles
// fall through to the common exit, where tensor memory is released.
#include <algorithm>
#include <mutex>

#include "arcq_tc.cuh"

namespace arcq {
namespace {

constexpr int BM = 128;            // rows of A per tile (MMA M)
constexpr int NUM_THREADS = 192;

template <int BN>
struct Cfg {
  static constexpr int NB = BN > 128 ? BN / 128 : 1;           // scale atoms of B per K step
  static constexpr int A_BYTES = BM * BK_BYTES;                // 16 KB
  static constexpr int B_BYTES = BN * BK_BYTES;
  static constexpr int SFA_BYTES = KSTEPS * ATOM;              // 2 KB
  static constexpr int SFB_BYTES = NB * KSTEPS * ATOM;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES + SFA_BYTES + SFB_BYTES;
  static constexpr int STAGES = (BN == 256) ? 4 : (BN == 128 ? 6 : 7);
  static constexpr int SF_COLS = KSTEPS * 4 + KSTEPS * 4 * NB;  // TMEM columns of one stage's scales
  static constexpr int TMEM_NEED = BN + 2 * SF_COLS;
  static constexpr int TMEM_COLS = TMEM_NEED <= 128 ? 128 : (TMEM_NEED <= 256 ? 256 : 512);
  // 1 KB alignment slack + stages + barriers; at least ~120 KB so that two CTAs never share an SM
  static constexpr int SMEM_RAW = 1024 + STAGES * STAGE_BYTES + 256;
  static constexpr int SMEM_BYTES = SMEM_RAW < 124 * 1024 ? 124 * 1024 : SMEM_RAW;
};

struct GemmParams {
  const uint8_t* sfa;
  const uint8_t* sfb;
  __nv_bfloat16* c;
  const __nv_bfloat16* bias;   // added to the bf16-rounded result, or nullptr: [N], or a residual [M, N] (bias_ld = N)
  int bias_ld;                 // elements between its rows: 0 or N
  const float* alpha_a;
  const float* alpha_b;
  float alpha;
  int M, N;
  int ksteps_total;   // K_eff / 64
  int natoms;         // ceil((K_eff/16)/4): scale atoms per 128-row tile
  int tiles_m, tiles_n;
  int sfb_tiles;      // ceil(N/128): 128-row scale tiles of B that exist
};

// Instruction descriptor of kind::mxf4nvf4 block-scaled MMA: e2m1 x e2m1 (format id 1), ue4m3
// scales (bit 23 = 0), both operands K-major, N>>3 at bit 17, M>>4 at bit 24, K=64 (bit 31 = 0).
template <int BN>
__device__ __forceinline__ constexpr uint32_t instr_desc() {
  return (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}

// Eight bf16 results plus eight bias or residual values, as a bf16 addition behind the GEMM gives them.
__device__ __forceinline__ void add_bf16x8(uint4& o, const uint4& b) {
  auto add = [](uint32_t x, uint32_t y) {
    return pack_bf16x2(__fadd_rn(__uint_as_float(x << 16), __uint_as_float(y << 16)),
                       __fadd_rn(__uint_as_float(x & 0xffff0000u), __uint_as_float(y & 0xffff0000u)));
  };
  o = make_uint4(add(o.x, b.x), add(o.y, b.y), add(o.z, b.z), add(o.w, b.w));
}

// ----------------------------------------------------------------------------- kernel

template <int BN>
__global__ void __launch_bounds__(NUM_THREADS, 1)
arcq_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                 const GemmParams p) {
  using C = Cfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;   // 128B swizzle needs 1 KB alignment
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bar_base = base + C::STAGES * C::STAGE_BYTES;
  volatile uint32_t* misc = reinterpret_cast<volatile uint32_t*>(base_ptr + C::STAGES * C::STAGE_BYTES + 192);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(misc + 1);
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (C::STAGES + s); };
  const uint32_t tmem_full_bar = bar_base + 8u * (2 * C::STAGES);
  const uint32_t tmem_empty_bar = tmem_full_bar + 8u;

  const int warp = warp_index(), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    mbar_init(tmem_full_bar, 1);
    mbar_init(tmem_empty_bar, 4);
    misc[1] = 0;  // abort flag
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)misc)),
                 "r"((uint32_t)C::TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");   // (every thread: everything below reads or writes global memory)
  // (All loads from here on are plain ones: scales, residual and tables may be written by the kernel before while this one is
  // already resident, and a residual by this one, which the read-only path is not for.)
  const uint32_t tmem_base = misc[0];
  const uint32_t tmem_sf = tmem_base + BN;   // two stage-parity buffers of SF_COLS columns each

  const int num_tiles = p.tiles_m * p.tiles_n;
  const int kstages = (p.ksteps_total + KSTEPS - 1) / KSTEPS;

  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    if (elect_one()) {
      uint32_t it = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
        const int tm = tile % p.tiles_m, tn = tile / p.tiles_m;
        const int rtb = (tn * BN) / 128;   // first 128-row scale tile of B this output tile touches
        for (int ks = 0; ks < kstages; ++ks, ++it) {
          const int s = it % C::STAGES;
          const uint32_t ph = (it / C::STAGES) & 1u;
          if (!mbar_wait(empty_bar(s), ph ^ 1u, abort_flag)) { ok = false; break; }
          const int nk = min(KSTEPS, p.ksteps_total - ks * KSTEPS);
          const uint32_t sf_bytes = (uint32_t)nk * ATOM;
          const uint32_t st = base + s * C::STAGE_BYTES;
          // scale tiles of B that exist (a 256-wide tile may hang over the last 128-row scale tile)
          int nb_valid = 0;
#pragma unroll
          for (int a = 0; a < C::NB; ++a) nb_valid += (rtb + a) < p.sfb_tiles ? 1 : 0;
          mbar_expect_tx(full_bar(s), C::A_BYTES + C::B_BYTES + sf_bytes * (1 + nb_valid));
          tma_load_2d(st, &map_a, full_bar(s), ks * BK_BYTES, tm * BM);
          tma_load_2d(st + C::A_BYTES, &map_b, full_bar(s), ks * BK_BYTES, tn * BN);
          const uint8_t* sa = p.sfa + ((size_t)tm * p.natoms + (size_t)ks * KSTEPS) * ATOM;
          bulk_load(st + C::A_BYTES + C::B_BYTES, sa, sf_bytes, full_bar(s));
#pragma unroll
          for (int a = 0; a < C::NB; ++a) {
            if ((rtb + a) < p.sfb_tiles) {
              const uint8_t* sb = p.sfb + ((size_t)(rtb + a) * p.natoms + (size_t)ks * KSTEPS) * ATOM;
              bulk_load(st + C::A_BYTES + C::B_BYTES + C::SFA_BYTES + a * (KSTEPS * ATOM), sb, sf_bytes, full_bar(s));
            }
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      constexpr uint32_t idesc = instr_desc<BN>();
      uint32_t it = 0, tile_it = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x, ++tile_it) {
        const int tn = tile / p.tiles_m;
        // sub-atom column offset when BN = 64: rows 32j..32j+31 of an atom live in TMEM column j, so
        // the upper half of a 128-row scale atom starts two columns in.  (Tiles narrower than 64
        // would need an odd column offset, which the block-scaled MMA rejects as misaligned.)
        const uint32_t sfb_sub = (BN < 128) ? (uint32_t)(((tn * BN) % 128) / 32) : 0u;
        if (!mbar_wait(tmem_empty_bar, (tile_it & 1u) ^ 1u, abort_flag)) { ok = false; break; }
        tc_fence_after();
        for (int ks = 0; ks < kstages; ++ks, ++it) {
          const int s = it % C::STAGES;
          const uint32_t ph = (it / C::STAGES) & 1u;
          if (!mbar_wait(full_bar(s), ph, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint32_t t_sfa = tmem_sf + (it & 1u) * C::SF_COLS, t_sfb = t_sfa + KSTEPS * 4;
          const uint32_t st = base + s * C::STAGE_BYTES;
          const uint64_t ad = smem_desc(st, 1024, LAYOUT_SW128), bd = smem_desc(st + C::A_BYTES, 1024, LAYOUT_SW128);
          const uint64_t sd = smem_desc(st + C::A_BYTES + C::B_BYTES, 128, LAYOUT_NONE);   // (descriptors count 16-byte units)
          auto copy_scales = [&](int k) {
            tc_cp_sf(t_sfa + k * 4, sd + k * (ATOM / 16));
#pragma unroll
            for (int a = 0; a < C::NB; ++a) tc_cp_sf(t_sfb + k * 4 * C::NB + a * 4, sd + ((1 + a) * KSTEPS + k) * (ATOM / 16));
          };
          auto multiply = [&](int k) {
            tc_mma_nvf4(tmem_base, ad + 2 * k, bd + 2 * k, idesc, t_sfa + k * 4, t_sfb + k * 4 * C::NB + sfb_sub, (ks | k) ? 1u : 0u);
          };
          const int nk = p.ksteps_total - ks * KSTEPS;
          if (nk >= KSTEPS) {
#pragma unroll
            for (int k = 0; k < KSTEPS; ++k) copy_scales(k);
#pragma unroll
            for (int k = 0; k < KSTEPS; ++k) multiply(k);
          } else {
            for (int k = 0; k < nk; ++k) copy_scales(k);
            for (int k = 0; k < nk; ++k) multiply(k);
          }
          tc_commit(empty_bar(s));   // stage reusable once these MMAs have read it
        }
        if (ok) tc_commit(tmem_full_bar);
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..5)
    const int quad = warp & 3;       // TMEM lanes 32*quad .. 32*quad+31 belong to this warp
    float alpha = p.alpha;
    if (p.alpha_a) alpha *= *p.alpha_a;
    if (p.alpha_b) alpha *= *p.alpha_b;
    uint32_t tile_it = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x, ++tile_it) {
      const int tm = tile % p.tiles_m, tn = tile / p.tiles_m;
      const int row = tm * BM + quad * 32 + lane;
      __nv_bfloat16* crow = p.c + (size_t)row * p.N;
      // Bias or residual of this thread's row.  Tiles of up to 128 columns ask for all of it while the products are still being
      // formed: behind the accumulator its latency was paid once per 32 columns.  With a residual, us, behind / early (without
      // one): [4096, 576] 512 rows 9.5 / 5.4 (4.4), [4096, 4224] 128 rows 10.1 / 7.8 (7.5), 333 rows 13.4 / 9.1 (8.6),
      // [1024, 7296] 256 rows 11.7 / 10.0 (9.7), [6144, 7296] 200 rows 17.0 / 12.8 (12.4).
      constexpr bool EARLY = BN <= 128;
      uint4 addend[EARLY ? BN / 8 : 4];
      auto fetch = [&](int c0, uint4* to) {
        const int col = tn * BN + c0;
        if (p.bias == nullptr || row >= p.M) return;
#pragma unroll
        for (int v = 0; v < 4; ++v)
          if (col + v * 8 < p.N) to[v] = *reinterpret_cast<const uint4*>(p.bias + (size_t)row * p.bias_ld + col + v * 8);
      };
      if constexpr (EARLY) {
#pragma unroll
        for (int c0 = 0; c0 < BN; c0 += 32) fetch(c0, addend + c0 / 8);
      }
      ok = mbar_wait(tmem_full_bar, tile_it & 1u, abort_flag);
      ok = __all_sync(0xffffffffu, ok);   // keep the warp converged for the .sync.aligned loads
      if (!ok) break;
      tc_fence_after();
      auto store = [&](int c0, const uint4* add) {
        uint32_t r[32];
        tc_ld32(tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0, r);
        tc_wait_ld();
        const int col = tn * BN + c0;
        if (row >= p.M) return;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          if (col + v * 8 < p.N) {   // N is a multiple of 8: whole 16-byte pieces are in or out
            uint4 o;
            o.x = pack_bf16x2(__uint_as_float(r[v * 8 + 0]) * alpha, __uint_as_float(r[v * 8 + 1]) * alpha);
            o.y = pack_bf16x2(__uint_as_float(r[v * 8 + 2]) * alpha, __uint_as_float(r[v * 8 + 3]) * alpha);
            o.z = pack_bf16x2(__uint_as_float(r[v * 8 + 4]) * alpha, __uint_as_float(r[v * 8 + 5]) * alpha);
            o.w = pack_bf16x2(__uint_as_float(r[v * 8 + 6]) * alpha, __uint_as_float(r[v * 8 + 7]) * alpha);
            if (p.bias != nullptr) add_bf16x8(o, add[v]);
            *reinterpret_cast<uint4*>(crow + col + v * 8) = o;
          }
        }
      };
      if constexpr (EARLY) {
#pragma unroll
        for (int c0 = 0; c0 < BN; c0 += 32) store(c0, addend + c0 / 8);
      } else {
#pragma unroll 1
        for (int c0 = 0; c0 < BN; c0 += 32) {
          fetch(c0, addend);
          store(c0, addend);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tmem_empty_bar);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)C::TMEM_COLS)
                 : "memory");
  }
}

// ----------------------------------------------------------------------------- 2-CTA kernel
//
// Same dataflow on a pair of SMs (cluster of two CTAs, cta_group::2): the pair owns a 256 x 256
// output tile.  Each CTA loads its own 128 rows of A, its own 128 rows of B (half of N), its own
// scale atoms of A and all scale atoms of B; the even CTA (leader) issues one
// tcgen05.mma.cta_group::2 (M256 x N256 x K64) per K step, which reads A from both CTAs' shared
// memory, the two halves of B likewise, and accumulates 128 rows x 256 columns in each CTA's TMEM.
// Per SM this is 9.5 KB of operands per K step instead of 13.5 KB, and the smaller stage
// (38 KB) lets five stages fit.
//
// Scale factors go shared memory -> tensor memory with tcgen05.cp (cta_group::2: each CTA's own atoms into its own tensor
// memory), twelve copies in front of a stage's MMAs, issued by the same thread.  Each of the five stages owns 48 TMEM columns, which
// the four warps needed that once carried the scales; copies and MMAs of one thread keep their order, and the single-CTA kernel
// makes do with two sets in turn.
// What bounds the main loop: the tensor pipe, 4 x 128 cycles a stage.  Loads alone need 450 cycles a stage, copies alone 325,
// MMAs alone 512 + what a tile boundary costs (730 a tile); all together 588, of which 76 are the boundary (17 stages
// a tile, [16384, 27648, 4224]).  While every role sat behind `lane == 0` a stage took 866 (see elect_one), and four warps
// carried the scales with tcgen05.st because copies looked as expensive as the MMAs.
//
// Synchronisation: all loads of either CTA complete on the LEADER's "full" barrier (.cta_group::2 form; the barrier address
// is the CTA-local one with the pair's rank bit cleared); tcgen05.commit with a two-CTA mask releases the stage in both
// CTAs and publishes the accumulator to both epilogues; the epilogue warps of both CTAs arrive on the leader's
// "accumulator free" barrier.  No load uses cluster multicast.

constexpr int C2_STAGES = 5;
constexpr int C2_THREADS = 320;                     // producer, MMA, 8 epilogue warps
constexpr int C2_A_BYTES = 128 * BK_BYTES;          // 16 KB
constexpr int C2_B_BYTES = 128 * BK_BYTES;          // 16 KB: this CTA's half of the 256 B rows
constexpr int C2_SFA_BYTES = KSTEPS * ATOM;         // 2 KB
constexpr int C2_SFB_BYTES = 2 * KSTEPS * ATOM;     // 4 KB: both 128-row scale tiles of B
constexpr int C2_STAGE_BYTES = C2_A_BYTES + C2_B_BYTES + C2_SFA_BYTES + C2_SFB_BYTES;   // 38 KB
constexpr int C2_SF_COLS = KSTEPS * 4 + KSTEPS * 8;  // 48 TMEM columns of scales per stage
constexpr int C2_TMEM_COLS = 512;                    // 256 accumulator + 5 x 48 scale columns
constexpr int C2_CSTAGE_BYTES = 8 * 4096;             // output staging: 32 rows x 64 columns of bf16 per epilogue warp
constexpr int C2_SMEM_BYTES = 1024 + C2_STAGES * C2_STAGE_BYTES + C2_CSTAGE_BYTES + 256 + 64;   // + residual barriers
constexpr uint32_t PEER_BIT_MASK = 0xFEFFFFFFu;      // clears the pair-rank bit of a shared address

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Tiled TMA load whose completion is counted on the leader CTA's barrier.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, uint32_t leader_bar, int x,
                                                 int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(map), "r"(leader_bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {   // arrives on `bar` in both CTAs of the pair
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
      ::"r"(bar), "h"((uint16_t)3)
      : "memory");
}
__device__ __forceinline__ void tc_mma_nvf4_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                                 uint32_t tsfa, uint32_t tsfb, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\n"
      "setp.ne.b32 p, %6, 0;\n"
      "tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.block16 [%0], %1, %2, %3, [%4], [%5], p;\n}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(tsfa), "r"(tsfb), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tc_cp_sf_pair(uint32_t taddr, uint64_t desc) {
  asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(desc) : "memory");
}
__device__ __forceinline__ void mbar_arrive_leader(uint32_t bar) {   // remote arrive on the leader's barrier
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar & PEER_BIT_MASK) : "memory");
}
struct Gemm2Params {
  __nv_bfloat16* c;
  const __nv_bfloat16* bias;   // [N], see GemmParams (plain epilogue only)
  const float* alpha_a;
  const float* alpha_b;
  float alpha;
  int M, N;
  int ksteps_total;   // K_eff / 64
  int natoms;         // scale atoms per 128-row tile
  int tiles_m, tiles_n;   // 256 x 256 tiles
  int group_m;            // tile rows per band of the tile order (see pair_tile_coords)
  // Grouped problems (one launch over several weight matrices stacked in B): tile_group[tm] = which
  // matrix the 256-row tile tm of A multiplies, or a negative number for a tile that holds no rows
  // (device memory: the host never learns the split).  Matrix g owns rows [g*N, (g+1)*N) of B and of
  // its scales, and alpha_a[g] * alpha_b[g].
  const int* tile_group;
  // SwiGLU epilogue (template flag of the kernel): B holds gate and up columns interleaved in blocks of 128
  // (tile column tn = gate columns [128 tn, 128 tn + 128) then the same up columns), C is [M, N/2] and
  // receives bf16(bf16(silu(gate)) * up) of the bf16-rounded GEMM outputs; amax[g] (bit pattern of a
  // non-negative float) takes max|.| over the valid rows - rows below M, and for grouped problems below the
  // end of their run, groups[g] + groups[ngroups + g].
  unsigned int* amax;
  const int* groups;
  int ngroups;
  // Scattered output (0 = off): rows [d * rows_per_dest, (d + 1) * rows_per_dest) of the result go to output
  // map d, a [rows_per_dest, N] buffer of its own - in a tensor-parallel group, this rank's slot in the memory
  // of the rank that owns those rows (a peer's memory over NVLink, or local memory).  A multiple of 32: one
  // bulk store carries 32 rows.
  int rows_per_dest;
};

// Output maps of the CTA-pair kernel: one, or one per destination of a scattered output.
constexpr int MAX_DESTS = 8;
struct OutputMaps {
  CUtensorMap m[MAX_DESTS];
};

// Tile order of the persistent pairs: bands of group_m tile rows, and inside a band column by column.
// The ~74 tiles in flight at any time then cover about group_m x (74 / group_m) tiles, so every strip of
// A and of B that is being streamed is shared by several pairs (one column of tiles would share one
// strip of B and nothing of A), and a band's A rows plus all of B stay in L2 while the band lasts.
__device__ __forceinline__ void pair_tile_coords(int tile, const Gemm2Params& p, int& tm, int& tn) {
  const int per_band = p.group_m * p.tiles_n;
  const int band = tile / per_band, in_band = tile - band * per_band;
  const int first = band * p.group_m;
  const int rows = min(p.group_m, p.tiles_m - first);
  tn = in_band / rows;
  tm = first + (in_band - tn * rows);
}

// RESID: the epilogue adds a residual tile (bf16 [M, N], map_r) to the bf16-rounded result before it stores:
// C = bf16(R + bf16(alpha * A B^T)), what a bf16 addition after the GEMM computes.  The tile arrives by TMA in
// the same staging memory the output leaves from (per-thread loads would touch 32 different rows per instruction).
template <bool SWIGLU, bool RESID = false>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(C2_THREADS, 1)
arcq_gemm2_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                  const __grid_constant__ CUtensorMap map_sfa, const __grid_constant__ CUtensorMap map_sfb,
                  const __grid_constant__ OutputMaps maps_c, const Gemm2Params p,
                  const __grid_constant__ CUtensorMap map_r) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t cstage_base = base + C2_STAGES * C2_STAGE_BYTES;   // 1024-byte aligned (swizzled boxes)
  const uint32_t bar_base = cstage_base + C2_CSTAGE_BYTES;
  volatile uint32_t* misc =
      reinterpret_cast<volatile uint32_t*>(base_ptr + C2_STAGES * C2_STAGE_BYTES + C2_CSTAGE_BYTES + 192);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(misc + 1);
  auto full_bar = [&](int s) { return bar_base + 8u * s; };                       // both CTAs' loads landed (leader's is used)
  auto empty_bar = [&](int s) { return bar_base + 8u * (C2_STAGES + s); };        // stage reusable
  const uint32_t tmem_full_bar = bar_base + 8u * (2 * C2_STAGES);
  const uint32_t tmem_empty_bar = tmem_full_bar + 8u;
  auto resid_bar = [&](int w) { return bar_base + 256u + 8u * w; };              // residual box of epilogue warp w landed

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();        // 0 = leader (issues the MMAs), 1 = peer
  const int cluster_id = blockIdx.x >> 1, num_clusters = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < C2_STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(tmem_full_bar, 1);
    mbar_init(tmem_empty_bar, 16);                // eight epilogue warps in each of the two CTAs
    for (int w = 0; w < 8; ++w) mbar_init(resid_bar(w), 1);
    misc[1] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)misc)),
                 "r"((uint32_t)C2_TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                             // both CTAs' barriers exist before anyone signals them
  tc_fence_after();
  // Programmatic dependent launch: what is above overlaps the end of the kernel before, everything below reads or writes
  // global memory (with plain loads, see arcq_gemm_kernel).
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const uint32_t tmem_base = misc[0];
  const uint32_t tmem_sf = tmem_base + 256;       // stage s: scale columns [256 + 48 s, 256 + 48 s + 48)

  const int num_tiles = p.tiles_m * p.tiles_n;
  const int kstages = (p.ksteps_total + KSTEPS - 1) / KSTEPS;

  if (warp == 0) {
    // ------------------------------------------------------------------ producer (both CTAs)
    if (elect_one()) {
      uint32_t it = 0;
      bool ok = true;
      for (int tile = cluster_id; tile < num_tiles && ok; tile += num_clusters) {
        int tm, tn;
        pair_tile_coords(tile, p, tm, tn);
        int grp = 0;
        if (p.tile_group != nullptr) { grp = p.tile_group[tm]; if (grp < 0) continue; }
        const int row_a = tm * 256 + (int)rank * 128;        // this CTA's rows of A (and of the output)
        const int row_b = grp * p.N + tn * 256 + (int)rank * 128;   // this CTA's rows of B (half of the N tile)
        const int sfa_tile = tm * 2 + (int)rank;             // 128-row scale tiles
        const int sfb_tile = grp * (p.N >> 7) + tn * 2;
        for (int ks = 0; ks < kstages; ++ks, ++it) {
          const int s = it % C2_STAGES;
          const uint32_t ph = (it / C2_STAGES) & 1u;
          if (!mbar_wait(empty_bar(s), ph ^ 1u, abort_flag)) { ok = false; break; }
          const uint32_t st = base + s * C2_STAGE_BYTES;
          const uint32_t lbar = full_bar(s) & PEER_BIT_MASK;
          if (rank == 0) mbar_expect_tx(full_bar(s), 2u * C2_STAGE_BYTES);   // what both CTAs deliver
          // scale atoms: rows of the map are atoms (128 words each); one box = the four K atoms of this stage
          tma_load_2d_pair(st + C2_A_BYTES + C2_B_BYTES, &map_sfa, lbar, 0, sfa_tile * p.natoms + ks * KSTEPS);
          tma_load_2d_pair(st + C2_A_BYTES + C2_B_BYTES + C2_SFA_BYTES, &map_sfb, lbar, 0, sfb_tile * p.natoms + ks * KSTEPS);
          tma_load_2d_pair(st + C2_A_BYTES + C2_B_BYTES + C2_SFA_BYTES + KSTEPS * ATOM, &map_sfb, lbar, 0,
                           (sfb_tile + 1) * p.natoms + ks * KSTEPS);
          tma_load_2d_pair(st, &map_a, lbar, ks * BK_BYTES, row_a);
          tma_load_2d_pair(st + C2_A_BYTES, &map_b, lbar, ks * BK_BYTES, row_b);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader CTA only)
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc = (1u << 7) | (1u << 10) | ((uint32_t)(256 >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
      uint32_t it = 0, tile_it = 0;
      bool ok = true;
      for (int tile = cluster_id; tile < num_tiles && ok; tile += num_clusters) {
        if (p.tile_group != nullptr) {
          int tm, tn;
          pair_tile_coords(tile, p, tm, tn);
          if (p.tile_group[tm] < 0) continue;      // a tile without rows: every role skips it
        }
        for (int ks = 0; ks < kstages; ++ks, ++it) {
          const int s = it % C2_STAGES;
          const uint32_t ph = (it / C2_STAGES) & 1u;
          if (!mbar_wait(full_bar(s), ph, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint32_t t_sfa = tmem_sf + s * C2_SF_COLS, t_sfb = t_sfa + KSTEPS * 4;
          const uint32_t st = base + s * C2_STAGE_BYTES;
          const uint64_t ad = smem_desc(st, 1024, LAYOUT_SW128), bd = smem_desc(st + C2_A_BYTES, 1024, LAYOUT_SW128);
          const uint64_t sd = smem_desc(st + C2_A_BYTES + C2_B_BYTES, 128, LAYOUT_NONE);   // (descriptors count 16-byte units)
          auto copy_scales = [&](int k) {
            tc_cp_sf_pair(t_sfa + k * 4, sd + k * (ATOM / 16));
            tc_cp_sf_pair(t_sfb + k * 8, sd + (KSTEPS + k) * (ATOM / 16));
            tc_cp_sf_pair(t_sfb + k * 8 + 4, sd + (2 * KSTEPS + k) * (ATOM / 16));
          };
          auto multiply = [&](int k) {
            tc_mma_nvf4_pair(tmem_base, ad + 2 * k, bd + 2 * k, idesc, t_sfa + k * 4, t_sfb + k * 8, (ks | k) ? 1u : 0u);
          };
          // (the scales do not wait for the accumulator)
          auto accumulator_free = [&]() {
            if (ks != 0) return true;
            if (!mbar_wait(tmem_empty_bar, (tile_it & 1u) ^ 1u, abort_flag)) return false;
            tc_fence_after();
            return true;
          };
          const int nk = p.ksteps_total - ks * KSTEPS;
          if (nk >= KSTEPS) {        // (unrolled: sixteen instructions have to leave in less than the MMAs' 512 cycles)
#pragma unroll
            for (int k = 0; k < KSTEPS; ++k) copy_scales(k);
            if (!accumulator_free()) { ok = false; break; }
#pragma unroll
            for (int k = 0; k < KSTEPS; ++k) multiply(k);
          } else {
            for (int k = 0; k < nk; ++k) copy_scales(k);
            if (!accumulator_free()) { ok = false; break; }
            for (int k = 0; k < nk; ++k) multiply(k);
          }
          tc_commit_pair(empty_bar(s));
        }
        if (ok) tc_commit_pair(tmem_full_bar);
        ++tile_it;
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (both CTAs)
    // Two warps per tensor-memory quadrant, each with half of the columns: [128 half, 128 half + 128), with SwiGLU gate
    // columns [64 half, 64 half + 64) and the up columns that belong to them.
    // (One warp per quadrant, with all 256 columns and SiLU from a table in L2, was busy for longer than a tile's MMAs:
    // SwiGLU [28672, 4224], us, before / eight warps and the table / eight warps and silu_for_bf16: 333 rows 55 / 52 / 49,
    // 2048 rows 147 / 142 / 137, 16384 rows 1057 / 1035 / 978.  The other epilogues are hidden either way.)
    const int quad = warp & 3, ew = warp - 2, half = ew >> 2;
    float alpha = p.alpha;
    if (p.tile_group == nullptr) {
      if (p.alpha_a) alpha *= *p.alpha_a;
      if (p.alpha_b) alpha *= *p.alpha_b;
    }
    uint32_t tile_it = 0, resid_it = 0;
    bool ok = true;
    for (int tile = cluster_id; tile < num_tiles && ok; tile += num_clusters) {
      int tm, tn;
      pair_tile_coords(tile, p, tm, tn);
      int grp = 0;
      if (p.tile_group != nullptr) {
        grp = p.tile_group[tm];
        if (grp < 0) continue;
        alpha = p.alpha;
        if (p.alpha_a) alpha *= p.alpha_a[grp];
        if (p.alpha_b) alpha *= p.alpha_b[grp];
      }
      if (RESID) {
        // the first residual box of this tile is fetched while the tile's MMAs are still running
        const int row0r = tm * 256 + (int)rank * 128 + quad * 32;
        if (lane == 0 && row0r < p.M && tn * 256 + 128 * half < p.N) {
          asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");     // the slot is free again
          mbar_expect_tx(resid_bar(ew), 4096u);
          tma_load_2d_once(cstage_base + (uint32_t)ew * 4096u, &map_r, resid_bar(ew), tn * 256 + 128 * half, row0r);
        }
      }
      ok = mbar_wait(tmem_full_bar, tile_it & 1u, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const int row = tm * 256 + (int)rank * 128 + quad * 32 + lane;
      // Drain the accumulator into registers (128 columns per thread) and hand tensor memory back before anything is done
      // with it: scaling, rounding and the stores then overlap the next tile's MMAs.
      uint32_t o[64];
      {
        uint32_t r[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint32_t col = SWIGLU ? (uint32_t)(128 * (c >> 1) + 64 * half + 32 * (c & 1)) : (uint32_t)(128 * half + 32 * c);
          tc_ld32(tmem_base + ((uint32_t)(quad * 32) << 16) + col, r[c]);
        }
        tc_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_leader(tmem_empty_bar);
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int v = 0; v < 16; ++v)
            o[16 * c + v] = pack_bf16x2(__uint_as_float(r[c][2 * v]) * alpha, __uint_as_float(r[c][2 * v + 1]) * alpha);
      }
      if (SWIGLU) {
        // columns 0..127 of the tile are gate, 128..255 the matching up columns: out = silu(gate) * up in
        // the gate registers, and its maximum over the rows that hold data
        int row_end = p.M;
        if (p.groups != nullptr) row_end = p.groups[grp] + p.groups[p.ngroups + grp];
        uint32_t m = 0;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const uint32_t g = o[j], u = o[32 + j];
          const uint32_t s2 = pack_bf16x2(silu_for_bf16(__uint_as_float(g << 16)), silu_for_bf16(__uint_as_float(g & 0xffff0000u)));
          const float sa = __uint_as_float(s2 << 16), sb = __uint_as_float(s2 & 0xffff0000u);
          o[j] = pack_bf16x2(sa * __uint_as_float(u << 16), sb * __uint_as_float(u & 0xffff0000u));
          asm("max.u16x2 %0, %0, %1;" : "+r"(m) : "r"(o[j] & 0x7fff7fffu));
        }
        uint32_t v = row < row_end ? max(m & 0xffffu, m >> 16) : 0u;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, d));
        if (lane == 0 && v) atomicMax(p.amax + grp, v << 16);
      }
      const int col0 = SWIGLU ? tn * 128 + 64 * half : tn * 256 + 128 * half;
      const int ncols = SWIGLU ? (p.N >> 1) : p.N;
      {
        // Through shared memory: the warp's 32 rows x 128 columns (SwiGLU: 64) leave as boxes of 64 columns
        // (32 rows x 128 bytes, 128-byte swizzle: lane = row, 16-byte chunk c of row r sits at chunk
        // c ^ (r & 7), so a warp's 128-bit stores are conflict free), one after the other from the
        // warp's 4 KB of staging.  The bulk stores write whole 128-byte lines, clip rows >= M and
        // columns >= N themselves.
        const int row0 = tm * 256 + (int)rank * 128 + quad * 32;
        const uint32_t slot = cstage_base + (uint32_t)ew * 4096u;
        const CUtensorMap* map_c = &maps_c.m[0];
        int row_st = row0;
        if (p.rows_per_dest) {       // these 32 rows belong to one destination
          const int d = row0 / p.rows_per_dest;
          map_c = &maps_c.m[d];
          row_st = row0 - d * p.rows_per_dest;
        }
        if (row0 < p.M) {
#pragma unroll
          for (int k = 0; k < (SWIGLU ? 1 : 2); ++k) {
            const int col = col0 + 64 * k;
            if (col >= ncols) break;
            if (RESID) {
              // (box 0 was requested before the accumulator was ready)
              if (k > 0 && lane == 0) {
                asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // box 0 has left the slot
                mbar_expect_tx(resid_bar(ew), 4096u);
                tma_load_2d_once(slot, &map_r, resid_bar(ew), col, row0);
              }
              ok = mbar_wait(resid_bar(ew), resid_it & 1u, abort_flag);
              ok = __all_sync(0xffffffffu, ok);
              if (!ok) break;
              ++resid_it;
            } else {
              if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the slot is free again
              __syncwarp();
            }
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              const int j = 32 * k + 4 * c;
              const uint32_t addr = slot + (uint32_t)lane * 128u + (uint32_t)((c ^ (lane & 7)) << 4);
              uint32_t out4[4] = {o[j], o[j + 1], o[j + 2], o[j + 3]};
              if (!RESID && !SWIGLU && p.bias != nullptr && col + 8 * c < ncols) {
                uint4 b4 = make_uint4(out4[0], out4[1], out4[2], out4[3]);
                add_bf16x8(b4, *reinterpret_cast<const uint4*>(p.bias + col + 8 * c));
                out4[0] = b4.x; out4[1] = b4.y; out4[2] = b4.z; out4[3] = b4.w;
              }
              if (RESID) {
                uint32_t rr[4];
                asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(rr[0]), "=r"(rr[1]), "=r"(rr[2]), "=r"(rr[3]) : "r"(addr) : "memory");
#pragma unroll
                for (int e = 0; e < 4; ++e)
                  out4[e] = pack_bf16x2(__uint_as_float(rr[e] << 16) + __uint_as_float(o[j + e] << 16),
                                        __uint_as_float(rr[e] & 0xffff0000u) + __uint_as_float(o[j + e] & 0xffff0000u));
              }
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(out4[0]), "r"(out4[1]), "r"(out4[2]),
                           "r"(out4[3])
                           : "memory");
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
              asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(map_c),
                           "r"(slot), "r"(col), "r"(row_st)
                           : "memory");
              asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
          }
        }
      }
      ++tile_it;
    }
    // the last boxes must have left shared memory (and reached global memory) before the CTA goes
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    __syncwarp();
  }

  // Neither CTA may leave (or give back tensor memory) while the other can still touch it.
  tc_fence_before();
  __syncthreads();
  __syncwarp();
  cluster_sync_all();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)C2_TMEM_COLS)
                 : "memory");
  }
}

// ----------------------------------------------------------------------------- host side

// Scale-factor buffer as a 2-D tensor of 32-bit words: one row per 512-byte atom; box = four atoms
// (the four K steps of one stage of one 128-row tile).
int make_sf_map(CUtensorMap* map, const void* ptr, int64_t total_atoms) {
  EncodeTiledFn fn;
  int rc = get_encode_fn(&fn);
  if (rc != ARCQ_OK) return rc;
  cuuint64_t dims[2] = {128, (cuuint64_t)total_atoms};
  cuuint64_t strides[1] = {(cuuint64_t)ATOM};
  cuuint32_t box[2] = {128, (cuuint32_t)KSTEPS};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return cuda_fail(cudaErrorInvalidValue);
  return ARCQ_OK;
}

// bf16 output [M, N] with a box of 64 columns x 32 rows, 128-byte swizzle (what one epilogue warp
// hands over per bulk store).
int make_c_map(CUtensorMap* map, const void* ptr, int64_t M, int64_t N) {
  EncodeTiledFn fn;
  int rc = get_encode_fn(&fn);
  if (rc != ARCQ_OK) return rc;
  cuuint64_t dims[2] = {(cuuint64_t)N, (cuuint64_t)M};
  cuuint64_t strides[1] = {(cuuint64_t)N * 2};
  cuuint32_t box[2] = {64, 32};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return cuda_fail(cudaErrorInvalidValue);
  return ARCQ_OK;
}

// ngroups > 1: B and SFB hold `ngroups` matrices of N rows each, tile_group says which one every
// 256-row tile of A multiplies (see Gemm2Params).
// swiglu_amax != nullptr: SwiGLU epilogue (see Gemm2Params), C is [M, N/2]; groups: the run table of a grouped
// problem (for the maxima).
int launch_pair(const uint8_t* A, const uint8_t* B, const uint8_t* SFA, const uint8_t* SFB, int64_t M, int64_t N,
                int64_t K_eff, const GemmParams& gp, const DeviceInfo& di, cudaStream_t stream, const int* tile_group = nullptr,
                int ngroups = 1, float* swiglu_amax = nullptr, const int* groups = nullptr,
                void* const* dests = nullptr, int ndests = 0, const void* residual = nullptr) {
  Gemm2Params p;
  p.rows_per_dest = ndests > 0 ? (int)(M / ndests) : 0;
  p.amax = reinterpret_cast<unsigned int*>(swiglu_amax);
  p.groups = groups;
  p.ngroups = ngroups;
  p.c = gp.c;
  p.bias = gp.bias;
  p.alpha_a = gp.alpha_a;
  p.alpha_b = gp.alpha_b;
  p.alpha = gp.alpha;
  p.M = gp.M;
  p.N = gp.N;
  p.ksteps_total = gp.ksteps_total;
  p.natoms = gp.natoms;
  p.tiles_m = (int)((M + 255) / 256);
  p.tiles_n = (int)((N + 255) / 256);
  // Column by column (one strip of B shared by the whole wave, A streamed from L2 once per column) unless A
  // alone overflows half of L2: then narrow bands of 4 tile rows, whose A rows stay resident next to B while
  // the band lasts.  Measured on B200 (M 16384, PFLOP/s): the down projection (A 118 MB) 4.32 with bands of 32
  // or 64 tile rows, 4.54 with 8 or 16, 4.62 - 4.65 with 4 (bands of 32 read A three times from HBM: 885 MB
  // where the operands and the residual are 282 MB); gate_up, qkv and o (A 35 MB) within 1.5 % of one another
  // for every band height from 8 to 64.
  p.group_m = (double)M * (double)K_eff / 2.0 > 64e6 ? 4 : p.tiles_m;
  // grouped: tile rows of one matrix are neighbours, so narrow bands keep a strip of B shared by the
  // pairs that are in flight together
  if (tile_group != nullptr) p.group_m = 4;
  if (p.group_m > p.tiles_m) p.group_m = p.tiles_m;
  p.tile_group = tile_group;
  CUtensorMap ma, mb, msa, msb;
  OutputMaps mc;
  int rc = ARCQ_OK;
  if (ndests > 0) {
    for (int d = 0; d < ndests && rc == ARCQ_OK; ++d) rc = make_c_map(&mc.m[d], dests[d], M / ndests, N);
    for (int d = ndests; d < MAX_DESTS; ++d) mc.m[d] = mc.m[0];
  } else {
    rc = make_c_map(&mc.m[0], gp.c, M, swiglu_amax != nullptr ? N / 2 : N);
    for (int d = 1; d < MAX_DESTS; ++d) mc.m[d] = mc.m[0];
  }
  if (rc != ARCQ_OK) return rc;
  rc = make_operand_map(&ma, A, M, K_eff / 2, 128);
  if (rc != ARCQ_OK) return rc;
  rc = make_operand_map(&mb, B, N * ngroups, K_eff / 2, 128);
  if (rc != ARCQ_OK) return rc;
  rc = make_sf_map(&msa, SFA, ((M + 127) / 128) * (int64_t)gp.natoms);
  if (rc != ARCQ_OK) return rc;
  rc = make_sf_map(&msb, SFB, ((N * ngroups + 127) / 128) * (int64_t)gp.natoms);
  if (rc != ARCQ_OK) return rc;
  CUtensorMap mr = mc.m[0];
  if (residual != nullptr) {
    rc = make_c_map(&mr, residual, M, N);
    if (rc != ARCQ_OK) return rc;
  }
  auto kern = swiglu_amax != nullptr ? arcq_gemm2_kernel<true, false>
                                     : (residual != nullptr ? arcq_gemm2_kernel<false, true> : arcq_gemm2_kernel<false, false>);
  ARCQ_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C2_SMEM_BYTES));
  long long tiles = (long long)p.tiles_m * p.tiles_n;
  long long clusters = di.num_sms / 2;
  if (clusters > tiles) clusters = tiles;
  return launch_dependent(kern, (unsigned)(2 * clusters), C2_THREADS, C2_SMEM_BYTES, di, stream, ma, mb, msa, msb, mc, p, mr);
}

template <int BN>
int launch_bn(const CUtensorMap& ma, const CUtensorMap& mb, GemmParams p, const DeviceInfo& di, cudaStream_t stream) {
  using C = Cfg<BN>;
  auto kern = arcq_gemm_kernel<BN>;
  ARCQ_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES));
  p.tiles_n = (p.N + BN - 1) / BN;
  long long tiles = (long long)p.tiles_m * p.tiles_n;
  int grid = (int)(tiles < di.num_sms ? tiles : di.num_sms);
  return launch_dependent(kern, (unsigned)grid, NUM_THREADS, C::SMEM_BYTES, di, stream, ma, mb, p);
}

// The single-CTA kernel with tiles of bn columns.
int launch_single(const uint8_t* A, const uint8_t* B, int64_t M, int64_t N, int64_t K_eff, int bn, const GemmParams& p, const DeviceInfo& di,
                  cudaStream_t stream) {
  CUtensorMap ma, mb;
  int rc = make_operand_map(&ma, A, M, K_eff / 2, BM);
  if (rc != ARCQ_OK) return rc;
  rc = make_operand_map(&mb, B, N, K_eff / 2, bn);
  if (rc != ARCQ_OK) return rc;
  switch (bn) {
    case 256: return launch_bn<256>(ma, mb, p, di, stream);
    case 128: return launch_bn<128>(ma, mb, p, di, stream);
    default: return launch_bn<64>(ma, mb, p, di, stream);
  }
}

}  // namespace

// Scratch for partial sums (see gemm_workspace_bytes) and tile width of the single-CTA kernel, by the cost model of a
// single row of tiles (microseconds: ~5 fixed, 0.35 + 0.65 * bn/256 per stage, 2 + 0.35 per MB of partial sums), among
// the choices that fit one wave of CTAs and 8 MB.
static void plan_splitk(int64_t M, int64_t N, int64_t K_eff, int num_sms, int* bn_out, int* splits_out,
                        bool allow_split = true) {
  const int tiles_m = (int)((M + BM - 1) / BM);
  int bn = 256;
  while (bn > 64 && (long long)tiles_m * ((N + bn - 1) / bn) < num_sms) bn >>= 1;
  const long long tiles = (long long)tiles_m * ((N + bn - 1) / bn);
  const int kstages = (int)((K_eff / 64 + KSTEPS - 1) / KSTEPS);
  int splits = 1;
  if (tiles_m == 1) {
    double best = 1e30;
    int best_bn = 64, best_splits = 1;
    for (int cand = 64; cand <= 256; cand <<= 1) {
      const long long t = (N + cand - 1) / cand;
      for (int sp = 1; sp <= (allow_split ? 8 : 1); ++sp) {
        if (t * sp > num_sms && sp > 1) break;
        if (sp > 1 && sp > kstages / 2) break;
        if (sp > 1 && (sp - 1) * ((kstages + sp - 1) / sp) >= kstages) continue;   // an empty range
        const double ws_mb = sp > 1 ? (double)sp * (double)M * (double)N * 4.0 / (1 << 20) : 0.0;
        if (ws_mb > 8.0) break;
        const double waves = (double)((t * sp + num_sms - 1) / num_sms);
        const double cost = 5.0 + waves * ((kstages + sp - 1) / sp) * (0.35 + 0.65 * cand / 256.0) +
                            (sp > 1 ? 2.0 + 0.35 * ws_mb : 0.0);
        if (cost < best) { best = cost; best_bn = cand; best_splits = sp; }
      }
    }
    bn = best_bn;
    splits = best_splits;
  } else if (allow_split && tiles * 2 <= num_sms) {
    splits = (int)(num_sms / tiles);
    if (splits > 8) splits = 8;
    if (splits > kstages / 2) splits = kstages / 2;   // at least two stages per range
    if (splits < 1) splits = 1;
    // ranges of ceil(kstages/splits) stages must all be non-empty
    while (splits > 1 && (splits - 1) * ((kstages + splits - 1) / splits) >= kstages) --splits;
  }
  *bn_out = bn;
  *splits_out = splits;
}

// Width of the single-CTA kernel's tiles for more than 64 rows where its tiles are one wave (the narrowest that are: a narrow
// tile's stages are short), or 0 where another kernel is the faster one.  Its K loop is one chain of stages; weight streaming
// splits K over a cluster of four as long as there are few enough 128 x 128 tiles (of two with more tiles, which never pays:
// 96 tiles and 113 stages 1.11 of this kernel's time).  The more tiles, the longer the chain may be.  Weight streaming over
// this kernel, product alone / with a residual:
//   tiles  97 and more rows, by stages of K                                  65 rows
//     8    17: 1.03 / 1.06   21: 0.96 / 0.97   29: 0.83 / 0.85                9: 1.13 / 1.15   13: 0.99 / 1.03   17: 0.87 / 0.91
//    16    17: 1.03 / 1.07   21: 0.99 / 1.01   25: 0.88 / 0.92                9: 1.17 / 1.16   13: 1.00 / 1.03   17: 0.90 / 0.93
//    24    21: 1.06 / 1.10   25: 0.99 / 1.02   37: 0.90 / 0.97               13: 1.00 / 1.03   17: 0.92 / 0.99   25: 0.90 / 0.98
//    32    29: 1.07 / 1.16   37: 0.99 / 1.05   45: 0.93 / 1.00               21: 1.01 / 1.07   25: 0.96 / 1.04   29: 0.93 / 1.00
//    48    37: 1.05 / 1.10   45: 0.99 / 1.04   57: 0.88 / 0.93               29: 1.02 / 1.08   37: 0.96 / 1.00   45: 0.93 / 0.97
//    64    45: 1.07 / 1.09   57: 0.95 / 0.97   81: 0.89 / 0.90               37: 1.00 / 1.04   45: 0.96 / 1.00   57: 0.95 / 0.98
// (96 rows lie between the two.  The line was drawn in tiles of rows once: narrow outputs of three and more then took the
// chain whatever its length, [1024, 14464] 333 rows 16.6 us instead of 12.5.)
// Tiles of 256 columns lose to CTA pairs (777 rows of [4096, 4224] 14.3 / 11.4), so 128 is the widest here.
static int single_tile(int64_t M, int64_t N, int64_t K_eff, int num_sms) {
  const int64_t rows = (M + BM - 1) / BM, tiles = rows * ((N + 127) / 128), stages = (K_eff / 64 + KSTEPS - 1) / KSTEPS;
  if (M <= ARCQ_SKINNY_ROWS || tiles > num_sms) return 0;
  const int64_t chain = M > 96 ? std::min<int64_t>(std::max<int64_t>(tiles, 18), 48) : std::min<int64_t>(std::max<int64_t>(tiles - 8, 12), 40);
  if (stages > chain && skinny_plan_splits(M, N, K_eff) == 4) return 0;
  return rows * ((N + 63) / 64) <= num_sms ? 64 : 128;
}

// Weight streaming (arcq_skinny.cu): up to 64 rows, and what the rule above leaves to it.
static bool use_skinny_kernel(int64_t M, int64_t N, int num_sms) {
  return M <= ARCQ_SKINNY_ROWS || ((M + 127) / 128) * ((N + 127) / 128) <= num_sms;
}
// With the SwiGLU epilogue (gate and up blocks in different CTAs of a cluster), us, this kernel at 65 and at 128 rows / CTA
// pairs at 129: [2048, 2176] 10.9 and 11.0 / 13.1, [3584, 4224] 11.2 and 12.9 / 15.5, [7168, 4224] 15.2 and 17.2 / 15.5, [14336,
// 4224] 14.9 and 18.9 / 14.9, [28672, 4224] 18.8 and 21.3 / 23.1, [57344, 8320] 60.0 and 64.6 / 68.2.  So CTA pairs from 81 rows
// where their tiles are one wave of at least a third of the pairs (96 rows of [14336, 4224] 17.0 / 14.9, of [7168, 4224] 15.9 / 15.5), and
// beyond 128 rows everywhere.
constexpr int64_t SKINNY_GATED_ROWS = 128;
// (At least two CTAs per 256 columns and 128 rows: under an SM limit only where that many may run, see arcq_set_sm_limit.)
static bool use_skinny_gated(int64_t M, int64_t N, const DeviceInfo& di) {
  const int64_t tiles = N / 256, ctas = 2 * tiles * ((M + 127) / 128);
  if (M > 80 && 6 * tiles >= di.num_sms && 2 * tiles <= di.num_sms) return false;
  return M <= SKINNY_GATED_ROWS && (di.num_sms == di.all_sms || ctas <= di.num_sms);
}

int launch_gemm_grouped(const uint8_t* A, const uint8_t* B, const uint8_t* SFA, const uint8_t* SFB, int64_t M,
                        int64_t N, int64_t K_eff, const int* tile_group, int ngroups, const float* alpha_a,
                        const float* alpha_b, void* Cout, cudaStream_t stream, float* swiglu_amax, const int* groups, bool clear_amax) {
  DeviceInfo di;
  int rc = get_device_info(&di);
  if (rc != ARCQ_OK) return rc;
  if (swiglu_amax != nullptr && clear_amax) ARCQ_CUDA_TRY(cudaMemsetAsync(swiglu_amax, 0, sizeof(float) * ngroups, stream));
  GemmParams p = {};
  p.c = static_cast<__nv_bfloat16*>(Cout);
  p.alpha_a = alpha_a;
  p.alpha_b = alpha_b;
  p.alpha = 1.0f;
  p.M = (int)M;
  p.N = (int)N;
  p.ksteps_total = (int)(K_eff / 64);
  p.natoms = (int)((K_eff / 16 + 3) / 4);
  // Few rows per matrix: the weight bytes are the time, and a 256-row tile holds mostly padding (see arcq_skinny.cu).  Eight
  // experts, down projection [4096, 14464] with the rest of the block, us, CTA pairs / streaming: 5 tokens 183 / 168, 37 tokens
  // 208 / 193, 100 tokens 211 / 197, 200 tokens (beyond the line, CTA pairs) 238 / 234.
  // Of a grouped problem the host knows a bound, M = routed rows rounded up to a tile + a tile per matrix (a tighter buffer is right
  // too, but passes for one of few rows).
  if (tile_group == nullptr && ngroups == 1 && swiglu_amax != nullptr && use_skinny_gated(M, N, di))
    return launch_gemm_skinny(A, B, SFA, SFB, M, N, K_eff, 1.0f, alpha_a, alpha_b, nullptr, Cout, swiglu_amax, nullptr, 1, stream);
  if (groups != nullptr && M - 256LL * ngroups <= 32LL * ngroups)
    return launch_gemm_skinny(A, B, SFA, SFB, M, N, K_eff, 1.0f, alpha_a, alpha_b, nullptr, Cout, swiglu_amax, groups, ngroups,
                              stream);
  return launch_pair(A, B, SFA, SFB, M, N, K_eff, p, di, stream, tile_group, ngroups, swiglu_amax, groups);
}

// The GEMM whose result rows are scattered over `ndests` buffers of M / ndests rows each (see
// Gemm2Params::rows_per_dest): always the CTA-pair kernel, whose epilogue stores through tensor maps.
int launch_gemm_scatter(const uint8_t* A, const uint8_t* B, const uint8_t* SFA, const uint8_t* SFB, int64_t M,
                        int64_t N, int64_t K_eff, const float* alpha_a, const float* alpha_b, void* const* dests,
                        int ndests, cudaStream_t stream) {
  if (ndests < 1 || ndests > MAX_DESTS || M % ndests || (M / ndests) % 32) return ARCQ_ERR_BAD_SHAPE;
  DeviceInfo di;
  int rc = get_device_info(&di);
  if (rc != ARCQ_OK) return rc;
  GemmParams p = {};
  p.c = nullptr;
  p.alpha_a = alpha_a;
  p.alpha_b = alpha_b;
  p.alpha = 1.0f;
  p.M = (int)M;
  p.N = (int)N;
  p.ksteps_total = (int)(K_eff / 64);
  p.natoms = (int)((K_eff / 16 + 3) / 4);
  return launch_pair(A, B, SFA, SFB, M, N, K_eff, p, di, stream, nullptr, 1, nullptr, nullptr, dests, ndests);
}

// C = bf16(residual + bf16(alpha_a * alpha_b * A B^T)), in the kernel that serves the plain product of this shape (so that the
// bits are those of an addition behind it), or CTA pairs.
int launch_gemm_residual(const uint8_t* A, const uint8_t* B, const uint8_t* SFA, const uint8_t* SFB, int64_t M,
                         int64_t N, int64_t K_eff, const float* alpha_a, const float* alpha_b, const void* residual,
                         void* Cout, cudaStream_t stream) {
  DeviceInfo di;
  int rc = get_device_info(&di);
  if (rc != ARCQ_OK) return rc;
  const int bn = single_tile(M, N, K_eff, di.num_sms);
  if (bn == 0 && use_skinny_kernel(M, N, di.num_sms))
    return launch_gemm_skinny(A, B, SFA, SFB, M, N, K_eff, 1.0f, alpha_a, alpha_b, residual, Cout, nullptr, nullptr, 1, stream);
  GemmParams p = {};
  p.sfa = SFA;
  p.sfb = SFB;
  p.c = static_cast<__nv_bfloat16*>(Cout);
  p.alpha_a = alpha_a;
  p.alpha_b = alpha_b;
  p.alpha = 1.0f;
  p.M = (int)M;
  p.N = (int)N;
  p.ksteps_total = (int)(K_eff / 64);
  p.natoms = (int)((K_eff / 16 + 3) / 4);
  p.tiles_m = (int)((M + BM - 1) / BM);
  p.sfb_tiles = (int)((N + 127) / 128);
  if (bn != 0) {
    p.bias = static_cast<const __nv_bfloat16*>(residual);
    p.bias_ld = (int)N;
    return launch_single(A, B, M, N, K_eff, bn, p, di, stream);
  }
  return launch_pair(A, B, SFA, SFB, M, N, K_eff, p, di, stream, nullptr, 1, nullptr, nullptr, nullptr, 0,
                     residual);
}

// What earlier versions put their partial sums in; no kernel touches it any more.
size_t gemm_workspace_bytes(int64_t M, int64_t N, int64_t K_eff) {
  DeviceInfo di;
  if (get_device_info(&di) != ARCQ_OK) return 0;
  int bn, splits;
  plan_splitk(M, N, K_eff, di.num_sms, &bn, &splits);
  return splits > 1 ? (size_t)splits * (size_t)M * (size_t)N * sizeof(float) : 0;
}

// Problems with enough 256 x 256 tiles to occupy at least half of the SM pairs run on CTA pairs
// (about 1.4x the throughput of the single-CTA kernel).
static bool use_pair_kernel(int64_t M, int64_t N, int num_sms) {
  return (long long)((M + 255) / 256) * ((N + 255) / 256) >= num_sms / 4 && M > 128;
}

int gemm_plan(int64_t M, int64_t N, int64_t K_eff, int* kind, int* tile_n, int* splits) {
  DeviceInfo di;
  int rc = get_device_info(&di);
  if (rc != ARCQ_OK) return rc;
  int k = ARCQ_GEMM_KIND_SINGLE, bn = single_tile(M, N, K_eff, di.num_sms), sp = 1;
  if (bn != 0) {
  } else if (use_skinny_kernel(M, N, di.num_sms)) {
    k = ARCQ_GEMM_KIND_SKINNY;
    bn = 128;
    sp = skinny_plan_splits(M, N, K_eff);
  } else if (use_pair_kernel(M, N, di.num_sms)) {
    k = ARCQ_GEMM_KIND_PAIR;
    bn = 256;
  } else {
    plan_splitk(M, N, K_eff, di.num_sms, &bn, &sp, false);
  }
  if (kind) *kind = k;
  if (tile_n) *tile_n = bn;
  if (splits) *splits = sp;
  return ARCQ_OK;
}

int launch_gemm(const uint8_t* A, const uint8_t* B, const uint8_t* SFA, const uint8_t* SFB, int64_t M, int64_t N,
                int64_t K_eff, float alpha, const float* alpha_a, const float* alpha_b, void* Cout, cudaStream_t stream,
                const void* bias) {
  DeviceInfo di;
  int rc = get_device_info(&di);
  if (rc != ARCQ_OK) return rc;
  int bn = single_tile(M, N, K_eff, di.num_sms);
  if (bn == 0 && use_skinny_kernel(M, N, di.num_sms))
    return launch_gemm_skinny(A, B, SFA, SFB, M, N, K_eff, alpha, alpha_a, alpha_b, bias, Cout, nullptr, nullptr, 1, stream,
                              bias != nullptr);

  GemmParams p;
  p.sfa = SFA;
  p.sfb = SFB;
  p.c = static_cast<__nv_bfloat16*>(Cout);
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.bias_ld = 0;
  p.alpha_a = alpha_a;
  p.alpha_b = alpha_b;
  p.alpha = alpha;
  p.M = (int)M;
  p.N = (int)N;
  p.ksteps_total = (int)(K_eff / 64);
  p.natoms = (int)((K_eff / 16 + 3) / 4);
  p.tiles_m = (int)((M + BM - 1) / BM);
  p.tiles_n = 0;
  p.sfb_tiles = (int)((N + 127) / 128);
  if (bn == 0 && use_pair_kernel(M, N, di.num_sms)) return launch_pair(A, B, SFA, SFB, M, N, K_eff, p, di, stream);

  int splits;
  if (bn == 0) plan_splitk(M, N, K_eff, di.num_sms, &bn, &splits, false);
  return launch_single(A, B, M, N, K_eff, bn, p, di, stream);
}

// ----------------------------------------------------------------------------- no-allocation entry point
//
// No kernel needs scratch; the shapes that once needed more than the block inside the library are refused as before.
int launch_gemm_static(const uint8_t* A, const uint8_t* B, const uint8_t* SFA, const uint8_t* SFB, int64_t M,
                       int64_t N, int64_t K_eff, float alpha, const float* alpha_a, const float* alpha_b, void* Cout,
                       cudaStream_t stream) {
  if (gemm_workspace_bytes(M, N, K_eff) > (size_t)ARCQ_STATIC_SCRATCH_BYTES) return ARCQ_ERR_SCRATCH_LIMIT;
  return launch_gemm(A, B, SFA, SFB, M, N, K_eff, alpha, alpha_a, alpha_b, Cout, stream);
}

int gemm_poll_error() {
  const int a = poll_tc_error(), b = skinny_poll_error();
  return a != ARCQ_OK ? a : b;
}

}  // namespace arcq
