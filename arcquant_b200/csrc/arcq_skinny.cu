// Block-scaled NVFP4 GEMM for few rows of A (decoding, short prompts, experts with a handful of tokens): weight streaming.
//
// Bound: HBM, by the packed weight (N * K_eff * 9/16 bytes); the products are a rounding error.  So the operands
// change sides: 128 rows of the WEIGHT are the M side of the MMA and the tokens its N side (16 to 128 columns), so
// that a stage of the ring is weight (16 KB of codes + 2 KB of scales for K = 256) and little else, and the whole
// chip's shared memory is a window of weight bytes in flight: two CTAs per SM, three to five stages each.
//  * K is split over the CTAs of a cluster (up to eight) where N alone gives too few CTAs.  Every CTA pushes its fp32
//    partial sums into the shared memory of the cluster's CTA that owns the token, one cluster barrier later they are
//    added there in rank order (the same bits on every run): no scratch, no second launch.
//  * SwiGLU (gate and up rows interleaved in blocks of 128): half of a cluster's CTAs compute the gate block, half the up
//    block, and the owner of a token forms bf16(bf16(silu(g)) * u) from their sums, and its maximum.  (Grouped: one CTA
//    computes both, one after the other, into two accumulators.)
//  * Grouped problems (the experts of a MoE block; with SwiGLU and plain): persistent CTAs walk over (expert, weight tile, pass of up to NT of
//    its rows); the rows of each expert are read from the device, and experts without rows cost nothing.
//  * Programmatic dependent launch: while the kernel before is still running, every CTA pulls its first weight tiles
//    into L2 (a prefetch reads nothing into the CTA, so a weight still being written is not read early).
//
// Roles: warp 0 producer (TMA), warp 1 issuer of the scale copies (tcgen05.cp) and MMAs, warps 2-5 epilogue; warps 6-9 help
// to add the partial sums.
#include "arcq_tc.cuh"

namespace arcq {
namespace {

constexpr int SK_THREADS = 320;
constexpr int SK_W_BYTES = 128 * BK_BYTES;      // 16 KB: 128 weight rows of one stage
constexpr int SK_SF_BYTES = KSTEPS * ATOM;      // 2 KB: the scale atoms of 128 rows of one stage
constexpr int SK_SF_COLS = 2 * KSTEPS * 4;      // tensor-memory columns of one stage's scales (both sides)

// NT token columns, NA accumulators; SPLIT: room for the cluster's partial sums.  Two CTAs per SM (half of 228 KB, less
// 1 KB per CTA for the system, 1 KB for alignment and the barriers).
template <int NT, int NA, bool SPLIT, bool GROUPED>
struct SkCfg {
  static constexpr int X_BYTES = NT * BK_BYTES;
  static constexpr int XBOX = NT > 64 ? 32 : 16;                       // rows of A per TMA box
  // Up to 32 columns the partial sums have memory of their own and are pushed there; more take the ring's place once the
  // CTA's products are complete, and their owners pull them.  (64 columns pushed left room for two stages only; 64 rows, us:
  // [6144, 4224] 11.2 -> 9.2, [10240, 8320] 19.8 -> 15.3, SwiGLU [14336, 4224] 22.7 -> 18.6.)
  static constexpr bool PULL = SPLIT && NT > 32;
  static constexpr int STAGE_BYTES = SK_W_BYTES + X_BYTES + 2 * SK_SF_BYTES;
  static constexpr int BAR_BYTES = 256;
  static constexpr int PART_BYTES = SPLIT && !PULL ? NA * (NT + 7) * 512 : 0;   // (tokens rounded up to the cluster, at most eight)
  static constexpr int TABLE_BYTES = GROUPED ? 3 * 64 * 4 : 0;         // the run table
  static constexpr int FIT = (113 * 1024 - 1024 - BAR_BYTES - TABLE_BYTES - PART_BYTES) / STAGE_BYTES;
  static constexpr int STAGES = FIT < 5 ? FIT : 5;
  static constexpr int SMEM_BYTES = 1024 + STAGES * STAGE_BYTES + PART_BYTES + BAR_BYTES + TABLE_BYTES;
  static constexpr int TMEM_NEED = NA * NT + STAGES * SK_SF_COLS;
  static constexpr int TMEM_COLS = TMEM_NEED <= 128 ? 128 : 256;
  static_assert(STAGES >= 2 && TMEM_NEED <= 256, "two CTAs share 512 columns of tensor memory");
  static_assert(!PULL || (NA == 1 && STAGES * STAGE_BYTES >= NT * 512), "the partial sums fit the ring");
};

struct SkinnyParams {
  const uint8_t* sfx;
  const uint8_t* sfw;
  __nv_bfloat16* c;                  // [M, N], or [M, N/2] with SwiGLU
  const __nv_bfloat16* residual;     // [M, N] (a bias: [N], residual_ld 0) or nullptr
  int residual_ld;                   // elements between its rows
  const float* alpha_a;
  const float* alpha_b;
  float alpha;
  int M, N;
  int ksteps_total;                  // K_eff / 64
  int natoms;                        // scale atoms per 128-row tile
  int tiles;                         // weight tiles per matrix: ceil(N / 128), halved with SwiGLU
  int ttiles;                        // token tiles of NT rows (grouped problems: counted on the device)
  int splits;                        // K ranges = CTAs per cluster
  const int* groups;                 // run table of a grouped problem (device) or nullptr
  int ngroups;
  unsigned int* amax;                // SwiGLU: max|C| per matrix (bit pattern of a non-negative float)
};

__device__ __forceinline__ void sk_prefetch_tile(const CUtensorMap* map, int x, int y) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(map), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t rank) {   // the same place in another CTA's shared memory
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster_f32(uint32_t addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t swiglu_bf16x2(uint32_t g, uint32_t u) {
  const uint32_t s = pack_bf16x2(silu_for_bf16(__uint_as_float(g << 16)), silu_for_bf16(__uint_as_float(g & 0xffff0000u)));
  return pack_bf16x2(__uint_as_float(s << 16) * __uint_as_float(u << 16), __uint_as_float(s & 0xffff0000u) * __uint_as_float(u & 0xffff0000u));
}
__device__ __forceinline__ uint32_t add_bf16x2(uint32_t a, uint32_t b) {   // in fp32, rounded once
  return pack_bf16x2(__fadd_rn(__uint_as_float(a << 16), __uint_as_float(b << 16)),
                     __fadd_rn(__uint_as_float(a & 0xffff0000u), __uint_as_float(b & 0xffff0000u)));
}

// NT: token columns per pass.  GATED: SwiGLU.  SPLIT: more than one CTA per cluster.  GROUPED: runs of rows, each with its
// own matrix (never split; SwiGLU of one matrix always is).
template <int NT, bool GATED, bool SPLIT, bool GROUPED>
__global__ void __launch_bounds__(SK_THREADS, 2)
arcq_skinny_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const SkinnyParams p) {
  constexpr int NA = GATED && !SPLIT ? 2 : 1;          // accumulators of a CTA
  constexpr int NB = GATED ? 2 : 1;                    // 128-row blocks of weight per work item
  static_assert(!(GROUPED && SPLIT) && (!GATED || GROUPED || SPLIT), "see above");
  using C = SkCfg<NT, NA, SPLIT, GROUPED>;
  constexpr int TMEM_COLS = C::TMEM_COLS;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  constexpr int BAR_AT = C::STAGES * C::STAGE_BYTES + C::PART_BYTES;
  const uint32_t part_base = base + C::STAGES * C::STAGE_BYTES, bar_base = base + BAR_AT;
  volatile uint32_t* misc = reinterpret_cast<volatile uint32_t*>(base_ptr + BAR_AT + 192);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(misc + 1);
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (C::STAGES + s); };
  const uint32_t acc_full_bar = bar_base + 8u * (2 * C::STAGES), acc_empty_bar = acc_full_bar + 8u;
  const int warp = warp_index(), lane = threadIdx.x & 31;

  const int ttiles = NT > 64 ? p.ttiles : 1;           // (a constant up to 64 rows: four divisions less before the first load)
  const int kstages = (p.ksteps_total + KSTEPS - 1) / KSTEPS;
  const int csize = SPLIT ? p.splits * NB : 1;                         // CTAs per cluster
  const int rank = SPLIT ? (int)(blockIdx.x % csize) : 0;
  const int splits = SPLIT ? p.splits : 1, split = SPLIT ? rank % splits : 0;
  const int block = SPLIT ? rank / splits : 0;                         // SwiGLU: 0 = gate, 1 = up
  const int ks_begin = kstages * split / splits, ks_end = kstages * (split + 1) / splits;
  const int first_item = (int)(blockIdx.x / csize), item_step = (int)(gridDim.x / csize);
  int num_items = p.tiles * ttiles;                                  // token tiles of one weight tile are neighbours
  // first weight row of accumulator a of weight tile t of matrix g, in the stacked matrices
  auto weight_row = [&](int g, int t, int a) { return g * p.N + t * (128 * NB) + 128 * (block + a); };

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(acc_full_bar, 1);
    mbar_init(acc_empty_bar, 4);
    misc[1] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    // the first ring of weight tiles on its way into L2 (grouped: as if every run had rows for one pass)
    int n = 0;
    for (int item = first_item; item < (GROUPED ? p.tiles * p.ngroups : num_items) && n < C::STAGES; item += item_step) {
      const int g = GROUPED ? item / p.tiles : 0, t = GROUPED ? item - g * p.tiles : item / ttiles;
      for (int a = 0; a < NA; ++a)
        for (int ks = ks_begin; ks < ks_end && n < C::STAGES; ++ks, ++n) sk_prefetch_tile(&map_w, ks * BK_BYTES, weight_row(g, t, a));
    }
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)misc)),
                 "r"((uint32_t)TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // A CTA's shared memory may be written by its cluster only once it has started: the other half of this barrier is in
  // front of the first such store (waiting here cost 0.6 us a call at 1 to 16 rows).
  if (SPLIT) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  bool met = false;
  auto meet = [&]() {
    if (SPLIT && !met) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    met = true;
  };
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");   // (every thread: everything below reads or writes global memory)
  const uint32_t tmem_base = misc[0];
  const uint32_t tmem_sf = tmem_base + NA * NT;

  // Grouped: per run (up to 64) the items up to and including it, its rows and its first row.  The passes of a long run
  // are items of their own: one CTA after the other taking them in turn made a batch that routes to few experts wait for
  // a few CTAs (256 rows of one run out of eight, [7168, 2176]: 51.3 -> 18.5 us).
  int* const run_end = reinterpret_cast<int*>(base_ptr + BAR_AT + C::BAR_BYTES);
  if (GROUPED) {
    if (warp == 0) {
      int before = 0;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int e = lane + 32 * h;
        const int row0 = e < p.ngroups ? p.groups[e] : 0, cnt = e < p.ngroups ? p.groups[p.ngroups + e] : 0;
        int inc = p.tiles * ((cnt + NT - 1) / NT);
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, inc, d);
          if (lane >= d) inc += v;
        }
        run_end[e] = before + inc;
        run_end[64 + e] = cnt;
        run_end[128 + e] = row0;
        before += __shfl_sync(0xffffffffu, inc, 31);
      }
    }
    __syncthreads();
    num_items = run_end[63];
  }
  // a work item: matrix, weight tile, first row in A / C, rows (at most NT)
  auto locate = [&](int item, int& g, int& t, int& row0, int& cnt) {
    if (GROUPED) {
      g = 0;                                              // the first run that ends beyond the item
#pragma unroll
      for (int d = 32; d > 0; d >>= 1)
        if (run_end[g + d - 1] <= item) g += d;
      const int i = item - (g > 0 ? run_end[g - 1] : 0), passes = (run_end[64 + g] + NT - 1) / NT;
      t = passes > 1 ? i / passes : i;                    // (the passes of one weight tile are neighbours)
      const int at = (i - t * passes) * NT;
      row0 = run_end[128 + g] + at;
      cnt = min(NT, run_end[64 + g] - at);
    } else {
      g = 0;
      t = item / ttiles;
      row0 = (item - t * ttiles) * NT;
      cnt = min(NT, p.M - row0);
    }
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    if (elect_one()) {
      uint32_t it = 0;
      bool ok = true;
      for (int item = first_item; item < num_items && ok; item += item_step) {
        int g, t, row0, cnt;
        locate(item, g, t, row0, cnt);
        const int boxes = (cnt + C::XBOX - 1) / C::XBOX;
        const int xt = row0 >> 7;                                        // 128-row scale tile of these rows
        for (int ai = 0; ai < NA && ok; ++ai) {
          const int wrow = weight_row(g, t, ai), wt = wrow >> 7;
          for (int ks = ks_begin; ks < ks_end; ++ks, ++it) {
            const int s = it % C::STAGES;
            if (!mbar_wait(empty_bar(s), ((it / C::STAGES) & 1u) ^ 1u, abort_flag)) { ok = false; break; }
            const uint32_t sf_bytes = (uint32_t)min(KSTEPS, p.ksteps_total - ks * KSTEPS) * ATOM;
            const uint32_t st = base + s * C::STAGE_BYTES, x_s = st + SK_W_BYTES, sfw_s = x_s + C::X_BYTES, sfx_s = sfw_s + SK_SF_BYTES;
            mbar_expect_tx(full_bar(s), SK_W_BYTES + (uint32_t)(boxes * C::XBOX * BK_BYTES) + 2u * sf_bytes);
            bulk_load(sfw_s, p.sfw + ((size_t)wt * p.natoms + (size_t)ks * KSTEPS) * ATOM, sf_bytes, full_bar(s));
            bulk_load(sfx_s, p.sfx + ((size_t)xt * p.natoms + (size_t)ks * KSTEPS) * ATOM, sf_bytes, full_bar(s));
            tma_load_2d(st, &map_w, full_bar(s), ks * BK_BYTES, wrow);
            for (int b = 0; b < boxes; ++b) tma_load_2d(x_s + b * (C::XBOX * BK_BYTES), &map_x, full_bar(s), ks * BK_BYTES, row0 + C::XBOX * b);
          }
        }
      }
      if (!ok) {
        // giving up with copies possibly in flight: wait (bounded) for those started here, so that none lands in
        // shared memory after the CTA has gone
        const unsigned long long t0 = globaltimer_ns();
        for (uint32_t j = it > (uint32_t)C::STAGES ? it - C::STAGES : 0; j < it; ++j)
          while (!mbar_try_wait(full_bar(j % C::STAGES), (j / C::STAGES) & 1u) && globaltimer_ns() - t0 < WAIT_LIMIT_NS) {}
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      uint32_t it = 0, acc_it = 0;
      bool ok = true;
      for (int item = first_item; item < num_items && ok; item += item_step, ++acc_it) {
        int g, t, row0, cnt;
        locate(item, g, t, row0, cnt);
        const uint32_t ncols = (uint32_t)((cnt + 15) & ~15);
        // e2m1 x e2m1, ue4m3 scales, K-major operands (see arcq_gemm.cu), N = ncols, M = 128
        const uint32_t idesc = (1u << 7) | (1u << 10) | ((ncols >> 3) << 17) | (8u << 24);
        if (!mbar_wait(acc_empty_bar, (acc_it & 1u) ^ 1u, abort_flag)) { ok = false; break; }
        tc_fence_after();
        for (int ai = 0; ai < NA && ok; ++ai) {
          for (int ks = ks_begin; ks < ks_end; ++ks, ++it) {
            const int s = it % C::STAGES;
            if (!mbar_wait(full_bar(s), (it / C::STAGES) & 1u, abort_flag)) { ok = false; break; }
            tc_fence_after();
            const int nk = min(KSTEPS, p.ksteps_total - ks * KSTEPS);
            const uint32_t st = base + s * C::STAGE_BYTES;
            // Scales: shared -> tensor memory, in front of the MMAs (the pipe keeps the order of copies and MMAs that one
            // thread issues; the MMAs that read the stage's old columns are complete, its producer waited for them).
            // `upper`: rows 64.. of a 128-row scale tile are words 2 and 3 of its atoms.
            const uint32_t t_sfw = tmem_sf + s * SK_SF_COLS, t_cpx = t_sfw + KSTEPS * 4, t_sfx = t_cpx + ((row0 & 64) ? 2u : 0u);
            const uint64_t wd = smem_desc(st, 1024, LAYOUT_SW128), xd = smem_desc(st + SK_W_BYTES, 1024, LAYOUT_SW128);
            const uint64_t sd = smem_desc(st + SK_W_BYTES + C::X_BYTES, 128, LAYOUT_NONE);   // (descriptors count 16-byte units)
            auto copy_scales = [&](int k) {
              tc_cp_sf(t_sfw + k * 4, sd + k * (ATOM / 16));
              tc_cp_sf(t_cpx + k * 4, sd + (KSTEPS + k) * (ATOM / 16));
            };
            auto multiply = [&](int k) {
              tc_mma_nvf4(tmem_base + ai * NT, wd + 2 * k, xd + 2 * k, idesc, t_sfw + k * 4, t_sfx + k * 4,
                          (ks > ks_begin || k > 0) ? 1u : 0u);
            };
            if (nk == KSTEPS) {
#pragma unroll
              for (int k = 0; k < KSTEPS; ++k) copy_scales(k);
#pragma unroll
              for (int k = 0; k < KSTEPS; ++k) multiply(k);
            } else {
              for (int k = 0; k < nk; ++k) copy_scales(k);
              for (int k = 0; k < nk; ++k) multiply(k);
            }
            tc_commit(empty_bar(s));
          }
        }
        if (ok) tc_commit(acc_full_bar);
      }
    }
  } else if (warp < 6) {
    // ------------------------------------------------------------------ epilogue (warps 2..5)
    const int quad = warp & 3;       // TMEM lanes 32*quad .. 32*quad+31 belong to this warp: weight rows of the tile
    const uint32_t t_row = tmem_base + ((uint32_t)(quad * 32) << 16);
    const int nl = quad * 32 + lane;                       // weight row within the tile
    uint32_t acc_it = 0;
    bool ok = true;
    const int ncols = GATED ? p.N >> 1 : p.N;
    // (unsplit) the residual of the next AHEAD tokens of this lane's four columns
    constexpr int AHEAD = NT < 64 ? NT : 64;
    uint2 res[AHEAD / 4];
    auto fetch_residual = [&](int row, int rows_here, int col) {
      if constexpr (!GATED) {
        if (p.residual == nullptr) return;
#pragma unroll
        for (int k = 0; k < AHEAD / 4; ++k) {
          const int tok = 4 * k + (lane & 3);
          if (tok < rows_here && col < ncols) res[k] = *reinterpret_cast<const uint2*>(p.residual + (size_t)(row + tok) * p.residual_ld + col);
        }
      }
    };
    for (int item = first_item; item < num_items; item += item_step, ++acc_it) {
      int g, t, row0, here;
      locate(item, g, t, row0, here);
      const int n4 = t * 128 + quad * 32 + (lane & ~3);    // (unsplit) first of this lane's four output columns
      float alpha = p.alpha;
      if (p.alpha_a) alpha *= p.alpha_a[g];
      if (p.alpha_b) alpha *= p.alpha_b[g];
      if (!SPLIT) fetch_residual(row0, here, n4);        // (while the products are still being formed)
      ok = mbar_wait(acc_full_bar, acc_it & 1u, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      if (C::PULL) {
        // fp32 partial sums in place of the ring (every product that reads it is complete): [token][128]
        for (int j0 = 0; j0 < here; j0 += 16) {
          uint32_t v[16];
          tc_ld16(t_row + j0, v);
          tc_wait_ld();
          float* dst = reinterpret_cast<float*>(base_ptr) + j0 * 128 + nl;
#pragma unroll
          for (int j = 0; j < 16; ++j) dst[j * 128] = __uint_as_float(v[j]);
        }
      } else if (SPLIT) {
        // fp32 partial sums to the CTAs that own the tokens: token j belongs to rank j % csize, where it is
        // number j / csize; layout there: [token number][source rank][128]
        meet();
        uint32_t dst[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) dst[r] = cluster_addr(part_base, (uint32_t)min(r, csize - 1));
        int r = 0;                                       // (rank of token j without a division per token)
        uint32_t at = (uint32_t)(rank * 512 + nl * 4);
        for (int j0 = 0; j0 < here; j0 += 16) {
          uint32_t v[16];
          tc_ld16(t_row + j0, v);
          tc_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            if (j0 + j < here) {
              uint32_t d = dst[0];
#pragma unroll
              for (int q = 1; q < 8; ++q) d = r == q ? dst[q] : d;
              st_cluster_f32(d + at, v[j]);
              if (++r == csize) { r = 0; at += (uint32_t)(csize * 512); }
            }
          }
        }
      } else {
        // A lane holds one column of 16 tokens; two exchanges between neighbouring lanes leave it four columns of the
        // tokens 4 k + lane % 4, which go out as 8-byte stores.  (Element by element - 16 stores, 16 dependent loads of
        // the residual - a pass of 64 tokens cost more than its weight stream, us: [256, 576] 128 rows 14.5 -> 6.5, with
        // a residual 33.9 -> 8.9; grouped SwiGLU [7168, 2176], 256 rows of one run out of eight 80.0 -> 51.3.)
        uint32_t m = 0;                                  // max|C| of two tokens
#pragma unroll 1
        for (int h0 = 0; h0 < here; h0 += AHEAD) {
          if (h0 > 0) fetch_residual(row0 + h0, here - h0, n4);
#pragma unroll
          for (int b = 0; b < AHEAD / 16; ++b) {
            const int j0 = h0 + 16 * b;
            if (j0 >= here) break;
            uint32_t r[16], u[16], o[8];
            tc_ld16(t_row + j0, r);
            if (GATED) tc_ld16(t_row + (NA - 1) * NT + j0, u);
            tc_wait_ld();
#pragma unroll
            for (int i = 0; i < 8; ++i) {                // tokens 2 i, 2 i + 1
              o[i] = pack_bf16x2(__uint_as_float(r[2 * i]) * alpha, __uint_as_float(r[2 * i + 1]) * alpha);
              if (GATED) o[i] = swiglu_bf16x2(o[i], pack_bf16x2(__uint_as_float(u[2 * i]) * alpha, __uint_as_float(u[2 * i + 1]) * alpha));
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {                // token 2 i + lane % 2, two columns
              const uint32_t x = __shfl_xor_sync(0xffffffffu, o[i], 1);
              o[i] = (lane & 1) ? __byte_perm(x, o[i], 0x7632) : __byte_perm(o[i], x, 0x5410);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {                // token 4 k + lane % 4, four columns
              const uint32_t x = __shfl_xor_sync(0xffffffffu, (lane & 2) ? o[2 * k] : o[2 * k + 1], 2);
              uint2 v = (lane & 2) ? make_uint2(x, o[2 * k + 1]) : make_uint2(o[2 * k], x);
              const int tok = j0 + 4 * k + (lane & 3);
              if (tok < here && n4 < ncols) {
                if (GATED) {
                  asm("max.u16x2 %0, %0, %1;" : "+r"(m) : "r"(v.x & 0x7fff7fffu));
                  asm("max.u16x2 %0, %0, %1;" : "+r"(m) : "r"(v.y & 0x7fff7fffu));
                } else if (p.residual != nullptr) {
                  v = make_uint2(add_bf16x2(res[4 * b + k].x, v.x), add_bf16x2(res[4 * b + k].y, v.y));
                }
                *reinterpret_cast<uint2*>(p.c + (size_t)(row0 + tok) * ncols + n4) = v;
              }
            }
          }
        }
        if (GATED) {       // (a NaN counts as larger than everything, as in the other epilogues)
          uint32_t mi = max(m & 0xffffu, m >> 16) << 16;
#pragma unroll
          for (int d = 16; d > 0; d >>= 1) mi = max(mi, __shfl_xor_sync(0xffffffffu, mi, d));
          if (lane == 0 && mi) atomicMax(p.amax + g, mi);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty_bar);
    }
  }

  __syncwarp();
  tc_fence_before();
  if (SPLIT) {
    // ------------------------------------------------------------------ the cluster's partial sums
    meet();
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (*abort_flag == 0) {
      int g, t, row0, cnt;
      locate(first_item, g, t, row0, cnt);
      const int ncols = GATED ? p.N >> 1 : p.N;
      float alpha = p.alpha;
      if (p.alpha_a) alpha *= *p.alpha_a;
      if (p.alpha_b) alpha *= *p.alpha_b;
      uint32_t m = 0;                                      // max|C|, two columns
      const float4* part = reinterpret_cast<const float4*>(base_ptr + C::STAGES * C::STAGE_BYTES);
      // four neighbouring columns of one of this CTA's tokens per thread and step
      for (int i = threadIdx.x;; i += SK_THREADS) {
        const int num = i >> 5, tok = num * csize + rank, n4 = (i & 31) * 4;
        if (tok >= cnt) break;
        float v[NB][4];
#pragma unroll
        for (int a = 0; a < NB; ++a) {
          float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
          for (int r = 0; r < splits; ++r) {
            float4 q;
            if (C::PULL) q = ld_cluster_f4(cluster_addr(base + (uint32_t)(tok * 512 + n4 * 4), (uint32_t)(a * splits + r)));
            else q = part[(num * csize + a * splits + r) * 32 + (i & 31)];
            sum.x += q.x; sum.y += q.y; sum.z += q.z; sum.w += q.w;
          }
          v[a][0] = sum.x; v[a][1] = sum.y; v[a][2] = sum.z; v[a][3] = sum.w;
        }
        const int n = t * 128 + n4;
        if (n < ncols) {                                   // (a multiple of four columns is in or out: N % 8 == 0)
          const size_t at = (size_t)(row0 + tok) * ncols + n;
          uint2 o = make_uint2(pack_bf16x2(v[0][0] * alpha, v[0][1] * alpha), pack_bf16x2(v[0][2] * alpha, v[0][3] * alpha));
          if (GATED) {
            o.x = swiglu_bf16x2(o.x, pack_bf16x2(v[NB - 1][0] * alpha, v[NB - 1][1] * alpha));
            o.y = swiglu_bf16x2(o.y, pack_bf16x2(v[NB - 1][2] * alpha, v[NB - 1][3] * alpha));
            asm("max.u16x2 %0, %0, %1;" : "+r"(m) : "r"(o.x & 0x7fff7fffu));
            asm("max.u16x2 %0, %0, %1;" : "+r"(m) : "r"(o.y & 0x7fff7fffu));
          } else if (p.residual != nullptr) {
            const uint2 r2 = *reinterpret_cast<const uint2*>(p.residual + (size_t)(row0 + tok) * p.residual_ld + n);
            o = make_uint2(add_bf16x2(r2.x, o.x), add_bf16x2(r2.y, o.y));
          }
          *reinterpret_cast<uint2*>(p.c + at) = o;
        }
      }
      if (GATED) {
        __syncwarp();
        uint32_t mi = max(m & 0xffffu, m >> 16) << 16;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) mi = max(mi, __shfl_xor_sync(0xffffffffu, mi, d));
        if (lane == 0 && mi) atomicMax(p.amax, mi);
      }
    }
    if (C::PULL) {       // nobody's partial sums go away while another CTA reads them
      __syncwarp();
      asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
  } else {
    __syncthreads();
  }
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)TMEM_COLS) : "memory");
  }
}

template <int NT, bool GATED, bool SPLIT, bool GROUPED = false>
int launch_one(const CUtensorMap& mx, const CUtensorMap& mw, const SkinnyParams& p, int grid, const DeviceInfo& di, cudaStream_t stream) {
  using C = SkCfg<NT, GATED && !SPLIT ? 2 : 1, SPLIT, GROUPED>;
  auto kern = arcq_skinny_kernel<NT, GATED, SPLIT, GROUPED>;
  static thread_local int c_dev = -1;
  int dev = 0;
  ARCQ_CUDA_TRY(cudaGetDevice(&dev));
  if (c_dev != dev) {
    ARCQ_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES));
    c_dev = dev;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(SK_THREADS);
  cfg.dynamicSmemBytes = C::SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = di.early_start();
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)(p.splits * (GATED ? 2 : 1));
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = SPLIT ? 2 : 1;
  ARCQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, mx, mw, p));
  return ARCQ_OK;
}
template <int NT>
int launch_nt(const CUtensorMap& mx, const CUtensorMap& mw, const SkinnyParams& p, bool gated, int grid, const DeviceInfo& di, cudaStream_t stream) {
  if (gated) return launch_one<NT, true, true>(mx, mw, p, grid, di, stream);
  if constexpr (NT > 64) return launch_one<NT, false, true>(mx, mw, p, grid, di, stream);   // (comes here split only)
  else return p.splits > 1 ? launch_one<NT, false, true>(mx, mw, p, grid, di, stream) : launch_one<NT, false, false>(mx, mw, p, grid, di, stream);
}

}  // namespace

// K ranges of a plain problem.  More CTAs shorten each one's chain of stages until the clusters no longer fit the chip
// at once; measured over 1..8 ranges (16 rows, us): [6144, 4224] 10.5 unsplit, 6.6 with 192 CTAs, 6.8 with 240, 10.4 with
// 288; [4096, 4224] 10.5, 5.7 with 192, 6.4 with 256; [4096, 14464] 26.1, 9.8 with 192, 9.7 with 256.  So one and a half
// CTAs per SM (one under an SM limit), at most eight ranges (the portable cluster
// size), each at least two stages long.
static int skinny_splits(int tiles, int kstages, const DeviceInfo& di) {
  const int ctas = di.num_sms == di.all_sms ? di.num_sms * 3 / 2 : di.num_sms;
  int s = ctas / tiles;
  if (s > 8) s = 8;
  if (s > kstages / 2) s = kstages / 2;
  return s < 1 ? 1 : s;
}
// The same for tiles of 128 token columns, whose stages take two to three times as long.  Clusters of two and four only: of
// three or six, CTAs that would fit one by one do not fit the chip at once ([4096, 4224], 333 rows, us: unsplit 20.4, two
// ranges = 192 CTAs 12.2, three = 288 CTAs 19.1; 200 rows: two 11.6, three 11.3, four = 256 CTAs 10.9, six 19.5).  (Two and one
// are used with SwiGLU only: a plain product that would not be split in four is served by single CTAs, see single_tile.)
static int skinny_splits_wide(int tiles, int kstages, const DeviceInfo& di) {
  const bool all = di.num_sms == di.all_sms;
  int s = 1;
  if (2LL * tiles <= (all ? 2 * di.num_sms : di.num_sms)) s = 2;
  if (4LL * tiles <= (all ? di.num_sms * 7 / 4 : di.num_sms)) s = 4;
  while (s > 1 && s > kstages / 2) s >>= 1;
  return s;
}
// See SkinnyParams; `residual` excludes `swiglu_amax` and groups; groups (device): ngroups matrices (at most 64) stacked in W.
int launch_gemm_skinny(const uint8_t* X, const uint8_t* W, const uint8_t* SFX, const uint8_t* SFW, int64_t M, int64_t N,
                       int64_t K_eff, float alpha, const float* alpha_a, const float* alpha_b, const void* residual, void* C,
                       float* swiglu_amax, const int* groups, int ngroups, cudaStream_t stream, bool residual_is_bias) {
  DeviceInfo di;
  int rc = get_device_info(&di);
  if (rc != ARCQ_OK) return rc;
  const bool gated = swiglu_amax != nullptr;
  SkinnyParams p = {};
  p.sfx = SFX;
  p.sfw = SFW;
  p.c = static_cast<__nv_bfloat16*>(C);
  p.residual = static_cast<const __nv_bfloat16*>(residual);
  p.residual_ld = residual_is_bias ? 0 : (int)N;
  p.alpha_a = alpha_a;
  p.alpha_b = alpha_b;
  p.alpha = alpha;
  p.M = (int)M;
  p.N = (int)N;
  p.ksteps_total = (int)(K_eff / 64);
  p.natoms = (int)((K_eff / 16 + 3) / 4);
  p.tiles = gated ? (int)(N / 256) : (int)((N + 127) / 128);
  p.groups = groups;
  p.ngroups = groups != nullptr ? ngroups : 1;
  p.amax = reinterpret_cast<unsigned int*>(swiglu_amax);
  const int kstages = (p.ksteps_total + KSTEPS - 1) / KSTEPS;
  // (runs of a grouped problem may start in the middle of a scale tile only in steps of 64 rows)
  const int nt = groups != nullptr ? 64 : (M > 64 ? 128 : (M > 32 ? 64 : (M <= 16 ? 16 : 32)));
  p.ttiles = groups != nullptr ? 1 : (int)((M + nt - 1) / nt);
  const int blocks = (gated ? 2 * p.tiles : p.tiles) * p.ttiles;
  p.splits = groups != nullptr ? 1 : (nt > 64 ? skinny_splits_wide(blocks, kstages, di) : skinny_splits(blocks, kstages, di));
  if (gated && p.splits > 4) p.splits = 4;
  const int csize = groups != nullptr ? 1 : p.splits * (gated ? 2 : 1);
  // (grouped: of the rows the host knows a bound, see launch_gemm_grouped)
  const long long passes = groups != nullptr ? p.ngroups + (M > 256LL * p.ngroups ? (M - 256LL * p.ngroups) / nt : 0) : p.ttiles;
  long long grid = p.tiles * passes * csize;
  // one CTA per item where several form a cluster; else persistent CTAs, two per SM
  const long long slots = di.num_sms == di.all_sms ? 2LL * di.num_sms : di.num_sms;
  if (csize == 1 && (groups != nullptr || nt <= 64) && grid > slots) grid = slots;
  CUtensorMap mx, mw;
  rc = make_operand_map(&mx, X, M, K_eff / 2, nt > 64 ? 32 : 16);
  if (rc != ARCQ_OK) return rc;
  rc = make_operand_map(&mw, W, N * p.ngroups, K_eff / 2, 128);
  if (rc != ARCQ_OK) return rc;
  if (groups != nullptr)
    return gated ? launch_one<64, true, false, true>(mx, mw, p, (int)grid, di, stream) : launch_one<64, false, false, true>(mx, mw, p, (int)grid, di, stream);
  if (nt == 16) return launch_nt<16>(mx, mw, p, gated, (int)grid, di, stream);
  if (nt == 32) return launch_nt<32>(mx, mw, p, gated, (int)grid, di, stream);
  if (nt == 64) return launch_nt<64>(mx, mw, p, gated, (int)grid, di, stream);
  return launch_nt<128>(mx, mw, p, gated, (int)grid, di, stream);
}

int skinny_plan_splits(int64_t M, int64_t N, int64_t K_eff) {
  DeviceInfo di;
  if (get_device_info(&di) != ARCQ_OK) return 1;
  const int tiles = (int)((N + 127) / 128), kstages = (int)((K_eff / 64 + KSTEPS - 1) / KSTEPS);
  return M > 64 ? skinny_splits_wide(tiles * (int)((M + 127) / 128), kstages, di) : skinny_splits(tiles, kstages, di);
}

int skinny_poll_error() { return poll_tc_error(); }

}  // namespace arcq
