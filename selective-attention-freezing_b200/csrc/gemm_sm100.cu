// Indexed linear on the 5th-generation tensor cores (tcgen05, TMEM accumulators).
//
//   out[m, g*slab + r] = sum_c x[m,c] * W_g[row0_g + r, c]  (+ bias)   [+ RoPE on chosen slabs]
//
// replaces the reference's gather-then-GEMM (kernel/indexed_linear.py:86-98: two
// index_select + cat materialise a (2R, C) weight copy on every call, then cuBLAS;
// RoPE afterwards as 3-4 elementwise kernels, nanogpt/model.py:1007-1008).  Here the
// canonical weights are read in place: every 64-row block of output features has
// its own TMA source (weight matrix, first row), so rows of frozen heads are never
// touched, and the rotation is applied to the fp32 accumulator in the epilogue.
//
// Persistent, warp-specialised CTA (1 per SM):
//   warp 0      TMA producer: x tile 128x64 and four 64x64 weight blocks per stage (128B swizzle)
//   warp 1      MMA issuer: tcgen05.mma 128x256x16, bf16 -> fp32 in TMEM, 2 accumulator buffers (512 columns)
//   warps 4..11 epilogue, two groups of four warps, 64 columns each at a time: TMEM -> registers (bias, RoPE) -> bf16
//               -> swizzled smem -> TMA store (one staging block per group).  The row's cos/sin values are fetched
//               once per row of tiles, before the accumulator is waited for, so their latency hides behind the MMAs.
//               With K = 768 a tile's products take 6144 cycles; one group of four warps needed longer than that for
//               a GELU or (by far) a rotation of 128-row slabs, whose 64 cos and 64 sin values it had to read anew for
//               every tile: 65536 x 1536 -> 1664, 128-row slabs, 692 -> 333 us; 65536 x 768 -> 1920, 64-row, 209 -> 175.
//               A residual comes by TMA into the block's own staging place, fetched into L2 while the products run:
//               65536 x 768 -> 768 with residual 125 -> 86 us (row by row from global memory before).
// Large products run the same kernel as CTA PAIRS (template parameter PAIR, a cluster of two): one 256x256 tile per
// pair through tcgen05.mma.cta_group::2, each CTA loading its 128 rows of x and half of the weight tile (see GCfg).
// All mbarrier waits are bounded; a wait that runs out sets *status and the CTA drains.
#include <algorithm>
#include <atomic>

#include "saf_internal.h"
#include "sm100_prims.cuh"

namespace saf {
namespace {

constexpr int GM = 128, GK = 64;             // rows of one CTA's accumulator, K step
constexpr int A_BYTES = GM * GK * 2;            // 16 KB
constexpr int SUB_BYTES = 64 * GK * 2;          // 8 KB: one 64-row block of weights
constexpr int MAX_STAGES = 8;
// PAIR: two CTAs of a cluster share one 256 x 256 tile through tcgen05 cta_group::2.  Each CTA loads its 128 rows of x
// and HALF of the weight tile (two 64-row blocks), so the operand traffic per SM drops from 96 to 64 bytes per clock at
// the full MMA rate -- what one SM can pull from L2 -- and a stage shrinks to 32 KB (6 stages instead of 4).
// SUBS: 64-column blocks of a tile.  4 (128x256 tiles, 96 B/clk of operand traffic per SM at the full MMA rate) is the form
// for products with tiles to spare; 2 and 1 cut a small product into enough tiles to occupy the SMs (pick_form).
template <bool PAIR, int SUBS>
struct GCfg {
  static constexpr int GN = SUBS * 64;                                 // columns of a tile
  static constexpr int B_SUBS = PAIR ? SUBS / 2 : SUBS;                // weight blocks a CTA loads per stage
  static constexpr int STAGE_BYTES = A_BYTES + B_SUBS * SUB_BYTES;     // 48 / 32 / 24 KB
  static constexpr int STAGES = STAGE_BYTES > 32768 ? 4 : (STAGE_BYTES > 24576 ? 6 : 8);
  static constexpr int ROWS = PAIR ? 2 * GM : GM;                      // rows of a tile
  static constexpr int TMEM_COLS = 2 * GN;                             // two accumulators
};
constexpr int OUT_BYTES = 2 * GM * 64 * 2;      // two 16 KB staging blocks for the TMA stores
constexpr int MAX_SUB = 288;                    // 64-row blocks of output features (N <= 18432)
constexpr int GEMM_THREADS = 384;   // TMA warp, MMA warp, two idle ones; two epilogue groups of four warps
// registers: 384 x 168 at launch; the first four warps keep 72, the epilogue takes 208 (128 * 72 + 256 * 208 <= 384 * 168)
constexpr int REGS_ISSUE = 72, REGS_EPI = 208;

struct SubTable {
  int32_t row0[MAX_SUB];
  uint8_t weight[MAX_SUB];
  uint8_t rope[MAX_SUB];     // 0: none, 1: this 64-block is the first half of a rotated slab... see kernel
  // slabs that are a multiple of 32 but not of 64 rows (head_dim 96): a 64-column block is two runs of 32 weight
  // rows, each with its own source (first run in row0 / weight, second run here)
  int32_t row0b[MAX_SUB];
  uint8_t weightb[MAX_SUB];
};

struct GemmParams {
  int M, N, K, T, slab;
  int tiles_m, tiles_n;
  int group_n, runs;             // column tiles walked together; units walk runs of tiles (see the tile order)
  const void* bias[SAF_MAX_WEIGHTS];
  const float* cosT;
  const float* sinT;
  int* status;
  int act;                       // SAF_ACT_*
  const __nv_bfloat16* residual; // added to the output, or null
  int64_t ldr;
  int residual_tma;              // the residual's blocks come through mapR (no rotation, no gate: columns as the output's)
  int halves;                    // weight blocks arrive as two 32-row TMA boxes (see SubTable)
  int weights_early;             // the first weight tiles may be loaded before the previous kernel is complete
  int32_t* zero2;                // two ints this launch clears for the next one on the stream (a tile queue), or null
};

// Form of a product: 64-column blocks of a single-CTA tile (1, 2, 4), or PAIR_FORM for 256 x 256 tiles of CTA pairs.
// A form takes fixed + waves x K steps x step: the fixed part is launch, first loads and the last tile's way out, a step is
// bound by the operands from L2 (24 / 32 / 48 KB an SM per step of a 1-, 2-, 4-block tile, 32 KB for a pair's 256 x 256).
// Fitted to each form's times over 128 to 8192 rows, K 256 to 3072, N 256 to 17920 on a B200, where the form it takes
// is within 8 % of the best one.  In us, pair / 4 / 2 / 1 blocks: 777 x 768 -> 3072 10.4 / 11.0 / 12.1 / 13.3, 777 x 3072
// -> 768 21.4 / 27.1 / 19.7 / 15.8, 777 x 2048 -> 5120 28.4 / 21.4 / 27.7 / 38.1, 3001 x 768 -> 768 9.7 / 11.0 / 8.7 /
// 10.2, 3001 x 1536 -> 3840 33.0 / 42.1 / 49.0 / 69.3, 8192 x 2048 -> 5120 122 / 150 / 211 / 301.
// `least`: blocks that belong together (a 128-row rotated slab, a gate/up pair).
constexpr int PAIR_FORM = 8;
int pick_form(int M, int N, int KB, int least, int pairs) {
  const int sms = device_sm_count();
  const int rows = (M + GM - 1) / GM, pair_rows = (M + 2 * GM - 1) / (2 * GM);
  int best = 4;
  double best_t = 1e30;
  auto consider = [&](int form, int64_t tiles, int units, double fixed, double step) {
    const double t = fixed + (double)((tiles + units - 1) / units) * KB * step;
    if (t < best_t) {
      best_t = t;
      best = form;
    }
  };
  if (N >= 256 && pairs > 0) consider(PAIR_FORM, (int64_t)pair_rows * ((N + 255) / 256), pairs, 4.9, 0.40);
  consider(4, (int64_t)rows * ((N + 255) / 256), sms, 4.9, 0.53);
  if (least <= 2) consider(2, (int64_t)rows * ((N + 127) / 128), sms, 3.6, 0.38);
  if (least <= 1) consider(1, (int64_t)rows * (N / 64), sms, 3.1, 0.27);
  return best;
}

// exact-form GELU, 0.5 x (1 + erf(x / sqrt 2)), with erf from Abramowitz-Stegun 7.1.26 (|error| < 1.5e-7):
// one reciprocal and one exponential on the special-function unit, the rest FMAs
__device__ __forceinline__ float gelu_erf(float x) {
  // Phi(-|x|) = 0.5 erfc(|x| / sqrt 2) = 0.5 t (a1 + t (a2 + t (a3 + t (a4 + t a5)))) exp(-x^2 / 2)
  const float ax = fabsf(x);
  float t, e;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t) : "f"(fmaf(0.3275911f * 0.70710678118654752f, ax, 1.f)));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(ax * ax * (-0.5f * 1.4426950408889634f)));
  float poly = fmaf(0.5f * 1.061405429f, t, 0.5f * -1.453152027f);
  poly = fmaf(poly, t, 0.5f * 1.421413741f);
  poly = fmaf(poly, t, 0.5f * -0.284496736f);
  poly = fmaf(poly, t, 0.5f * 0.254829592f);
  const float q = poly * t * e;                 // Phi(-|x|)
  return x * (x >= 0.f ? 1.f - q : q);          // x Phi(x)
}

// SiLU gate: g * sigmoid(g) * u, sigmoid through one exponential and one approximate reciprocal
__device__ __forceinline__ float silu_mul(float g, float u) {
  float e, r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(g * -1.4426950408889634f));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.f + e));
  return g * r * u;
}

struct SmemLayout {
  uint64_t full[MAX_STAGES], empty[MAX_STAGES], acc_full[2], acc_empty[2], res[2];
  uint32_t tmem_base;
};

template <bool PAIR, int SUBS>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
indexed_gemm_kernel(const __grid_constant__ CUtensorMap mapX, const __grid_constant__ CUtensorMap mapW0,
                    const __grid_constant__ CUtensorMap mapW1, const __grid_constant__ CUtensorMap mapW2,
                    const __grid_constant__ CUtensorMap mapW3, const __grid_constant__ CUtensorMap mapO,
                    const __grid_constant__ CUtensorMap mapR,
                    const __grid_constant__ GemmParams p, const __grid_constant__ SubTable tb) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  using C = GCfg<PAIR, SUBS>;
  constexpr int STAGES = C::STAGES, STAGE_BYTES = C::STAGE_BYTES, GN = C::GN;
  uint8_t* stage_base = smem;
  uint8_t* out_stage = smem + STAGES * STAGE_BYTES;
  SmemLayout* sl = reinterpret_cast<SmemLayout*>(out_stage + OUT_BYTES);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int KB = (p.K + GK - 1) / GK;
  const int total_tiles = p.tiles_m * p.tiles_n;
  const int rank = PAIR ? (int)cluster_ctarank() : 0;                 // which 128 rows of the tile are this CTA's
  const int unit = PAIR ? blockIdx.x >> 1 : blockIdx.x, n_units = PAIR ? gridDim.x >> 1 : gridDim.x;
  // Tile order: column tiles in groups whose weights stay in L2, inside a group all columns of one row tile first; the
  // units take neighbouring tiles at the same time, so a row of x is fetched from memory once per group, by the units that
  // need it together.  (Each unit walking the columns of rows of its own has 74 x 256 rows of x in use at once: at
  // K = 8960 that is 340 MB, and x comes from memory once per column tile.  65536 x 8960 -> 1536 with that order and its
  // sibling 1536 -> 2 x 8960 2372 us on average, now 1882.)  A rotated product keeps the runs: its epilogue holds the
  // row's cos / sin values over the run, and reading them anew for every tile cost more than x from memory
  // (65536 x 768 -> 1920, before the tables were read as whole lines: 180 us with runs, 260 without; at 128-row slabs no
  // difference).
  const int tile_lo = p.runs ? (int)((int64_t)unit * total_tiles / n_units) : unit;
  const int tile_hi = p.runs ? (int)((int64_t)(unit + 1) * total_tiles / n_units) : total_tiles;
  const int tile_step = p.runs ? 1 : n_units;
  auto decode = [&](int tile, int& tm, int& tn) {
    const int per_group = p.tiles_m * p.group_n;
    const int g = tile / per_group, rem = tile - g * per_group;
    const int width = min(p.group_n, p.tiles_n - g * p.group_n);
    tm = rem / width;
    tn = g * p.group_n + rem - tm * width;
  };

  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&sl->full[s], 1);
      mbar_init(&sl->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sl->acc_full[b], 1);
      mbar_init(&sl->acc_empty[b], PAIR ? 16 : 8);      // one arrival per epilogue warp (of both CTAs)
    }
    mbar_init(&sl->res[0], 1);
    mbar_init(&sl->res[1], 1);
    fence_mbar_init();
  }
  if (warp == 1) {
    if constexpr (PAIR) {
      tmem_alloc_pair(&sl->tmem_base, C::TMEM_COLS);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(&sl->tmem_base, C::TMEM_COLS);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();                 // the peer's barriers exist before anything arrives on them
  tc_fence_after();
  const uint32_t tmem = sl->tmem_base;

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_ISSUE));
    if (warp == 0) {
      if (lane == 0) {
        const CUtensorMap* wm[4] = {&mapW0, &mapW1, &mapW2, &mapW3};
        tma_prefetch_desc(&mapX);
        uint32_t it = 0;
        bool ok = true;
        // announce a stage's bytes and load its weight tile / its rows of x.
        // PAIR: this CTA's 128 rows of x and its two of the tile's four weight blocks.  Every byte of both CTAs is
        // counted on the even CTA's barrier, which its MMA warp waits on: the even CTA's producer announces the
        // pair's bytes there (a local arrive), the odd CTA's producer only issues its loads -- they cannot land
        // before the barrier's previous phase is over, because its own empty barrier opens after that.
        // (a last column tile of two blocks is computed as a 256 x 128 product: one block per CTA)
        auto load_w = [&](int tn, int kb, int s) {
          const int nsub = min(SUBS, (p.N - tn * GN) / 64);
          uint8_t* b = stage_base + s * STAGE_BYTES + A_BYTES;
          const int per = PAIR ? (nsub == 2 ? 1 : C::B_SUBS) : SUBS;
          const int mine = PAIR ? max(0, min(per, nsub - rank * per)) : nsub;
          if (!PAIR) mbar_expect_tx(&sl->full[s], A_BYTES + nsub * SUB_BYTES);
          else if (rank == 0) mbar_expect_tx(&sl->full[s], 2 * A_BYTES + nsub * SUB_BYTES);
          const uint32_t bar = PAIR ? cluster_addr_of(&sl->full[s], 0) : 0;
          for (int u = 0; u < mine; ++u) {
            const int sb = tn * SUBS + rank * per + u;
            if constexpr (PAIR) tma_load_2d_pair(b + u * SUB_BYTES, wm[tb.weight[sb]], bar, kb * GK, tb.row0[sb]);
            else tma_load_2d(b + u * SUB_BYTES, wm[tb.weight[sb]], &sl->full[s], kb * GK, tb.row0[sb]);
            if (p.halves) {   // the maps' boxes are 32 rows: the second run lands behind the first (4 swizzle atoms on)
              if constexpr (PAIR) tma_load_2d_pair(b + u * SUB_BYTES + SUB_BYTES / 2, wm[tb.weightb[sb]], bar, kb * GK, tb.row0b[sb]);
              else tma_load_2d(b + u * SUB_BYTES + SUB_BYTES / 2, wm[tb.weightb[sb]], &sl->full[s], kb * GK, tb.row0b[sb]);
            }
          }
        };
        auto load_x = [&](int tm, int kb, int s) {
          uint8_t* a = stage_base + s * STAGE_BYTES;
          if constexpr (PAIR) tma_load_2d_pair(a, &mapX, cluster_addr_of(&sl->full[s], 0), kb * GK, tm * C::ROWS + rank * GM);
          else tma_load_2d(a, &mapX, &sl->full[s], kb * GK, tm * GM);
        };
        // the first ring of weight tiles depends on no earlier kernel (the caller says so)
        const int early = p.weights_early && tile_lo < tile_hi ? min(KB, STAGES) : 0;
        int tm, tn;
        decode(tile_lo, tm, tn);
        for (int kb = 0; kb < early; ++kb) load_w(tn, kb, kb);
        pdl_wait();
        if (p.zero2 && blockIdx.x == 0) {
          p.zero2[0] = 0;
          p.zero2[1] = 0;
        }
        pdl_trigger();
        for (int tile = tile_lo; tile < tile_hi && ok; tile += tile_step) {
          decode(tile, tm, tn);
          if (p.residual_tma)     // the epilogue's residual blocks are in L2 by the time the products are done
            for (int u = 0; u < min(SUBS, (p.N - tn * GN) / 64); ++u) tma_prefetch_2d(&mapR, tn * GN + u * 64, tm * C::ROWS + rank * GM);
          for (int kb = 0; kb < KB; ++kb, ++it) {
            const int s = it % STAGES;
            if (it >= (uint32_t)early) {
              if (!mbar_wait(&sl->empty[s], ((it / STAGES) & 1) ^ 1)) {
                dev_set_error(p.status, SAF_DEV_TIMEOUT_TMA, 10);
                ok = false;
                break;
              }
              load_w(tn, kb, s);
            }
            load_x(tm, kb, s);
          }
        }
      }
    } else if (warp == 1 && rank == 0) {
      // the whole warp walks the schedule (uniform addresses); one elected lane issues.  In a pair only the even
      // CTA issues: its instructions read both CTAs' stages and write both CTAs' accumulators.
      const bool leader = elect_one();
      const uint32_t idesc_full = umma_idesc_bf16(C::ROWS, GN, 0, 0);
      const uint32_t idesc_half = umma_idesc_bf16(C::ROWS, GN / 2, 0, 0);   // pair: a last column tile of two blocks
      const uint32_t sbase = smem_u32(stage_base);
      uint32_t it = 0, lt = 0;
      bool ok = true;
      // K steps of all this unit's tiles.  The last round of stages is not handed back: nobody loads into them again, and in
      // a pair the hand-back is an arrival that the tensor core makes in both CTAs' shared memory, where another kernel's
      // CTA may follow as soon as this one is done.
      const uint32_t steps = tile_lo < tile_hi ? (uint32_t)((tile_hi - tile_lo + tile_step - 1) / tile_step) * KB : 0;
      pdl_wait();                       // the limits of the waits below do not run while an earlier kernel does
      for (int tile = tile_lo; tile < tile_hi && ok; tile += tile_step, ++lt) {
        const int buf = lt & 1;
        if (!mbar_wait(&sl->acc_empty[buf], ((lt >> 1) & 1) ^ 1)) {
          dev_set_error(p.status, SAF_DEV_TIMEOUT_MMA, 11);
          break;
        }
        tc_fence_after();
        const uint32_t d = tmem + buf * GN;
        int tm_, tn_;
        decode(tile, tm_, tn_);
        const uint32_t idesc = (PAIR && (p.N - tn_ * GN) / 64 == 2) ? idesc_half : idesc_full;
        for (int kb = 0; kb < KB; ++kb, ++it) {
          const int s = it % STAGES;
          if (!mbar_wait(&sl->full[s], (it / STAGES) & 1)) {
            dev_set_error(p.status, SAF_DEV_TIMEOUT_MMA, 12);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a = sbase + s * STAGE_BYTES;
          const uint32_t b = a + A_BYTES;
          if (leader) {
            const uint64_t ad0 = umma_smem_desc_sw128(a, 16, 1024), bd0 = umma_smem_desc_sw128(b, 16, 1024);
#pragma unroll
            for (int k4 = 0; k4 < GK / 16; ++k4) {
              const uint64_t ad = umma_desc_advance(ad0, k4 * 32), bd = umma_desc_advance(bd0, k4 * 32);
              if constexpr (PAIR) umma_ss_pair(d, ad, bd, idesc, (kb | k4) != 0);
              else umma_ss(d, ad, bd, idesc, (kb | k4) != 0);
            }
            if (it + STAGES < steps) {
              if constexpr (PAIR) umma_commit_pair(&sl->empty[s]);    // frees the stage in both CTAs
              else umma_commit(&sl->empty[s]);
            }
          }
          __syncwarp();
        }
        if (ok && leader) {
          if constexpr (PAIR) umma_commit_pair(&sl->acc_full[buf]);
          else umma_commit(&sl->acc_full[buf]);
        }
        __syncwarp();
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_EPI));
    // epilogue warps 4..11 -> TMEM lane quadrant (warp % 4); two groups of four warps take turns over the 64-column blocks
    pdl_wait();
    const int quad = warp & 3, grp = (warp - 4) >> 2;
    const int row = quad * 32 + lane;           // row inside the tile
    const bool chief = (tid & 127) == 0;        // loads and stores its group's blocks
    const bool swiglu = p.act == SAF_ACT_SWIGLU;
    // a rotated 128-row slab is two blocks: group g rotates columns 32g .. 32g+31 of the first with those of the second,
    // so that a thread needs 32 cos and 32 sin values of its row (held over the row's tiles), and both fill both blocks.
    // The second half of a table row repeats the first in every rotary embedding; a block of 128 rows where it does not
    // is noticed as the values arrive, and reads its second halves where it needs them
    const bool wide = p.slab == 128 && p.cosT;
    const int bar_id = wide ? 3 : 1 + grp, bar_n = wide ? 256 : 128;
    uint8_t* stg = out_stage + grp * (OUT_BYTES / 2);
    uint32_t lt = 0;
    int tm_held = -1;                           // row tile whose cos / sin values the registers hold
    float4 cs4[8], sn4[8];
    bool halves_differ = false;
    // the residual block of this group's first output block at or behind (tile, step), into its free staging block
    uint32_t n_res = 0;
    auto ask_residual = [&](int tile, int st) {
      for (; tile < tile_hi; tile += tile_step, st = 0) {
        int tm, tn;
        decode(tile, tm, tn);
        const int nsub = min(SUBS, (p.N - tn * GN) / 64), u = 2 * st + grp;
        if (u >= nsub) continue;
        mbar_expect_tx(&sl->res[grp], GM * 64 * 2);
        tma_load_2d(stg, &mapR, &sl->res[grp], tn * GN + u * 64, tm * C::ROWS + rank * GM);
        return;
      }
    };
    if (p.residual_tma && chief) ask_residual(tile_lo, 0);
    for (int tile = tile_lo; tile < tile_hi; tile += tile_step, ++lt) {
      int tm, tn;
      decode(tile, tm, tn);
      const int nsub = min(SUBS, (p.N - tn * GN) / 64);
      const int buf = lt & 1;
      const int m = tm * C::ROWS + rank * GM + row;
      if (p.cosT && tm != tm_held) {
        tm_held = tm;
        // 32 values of 128 table rows (the tables repeat per half), whole 128-byte pieces of 4 rows per load, handed to
        // the threads of the rows through the group's staging block.  (A thread reading its own row touched 32 lines per
        // load: 8192 cycles of the load path for the two groups, more than the products of a narrow tile.)
        const int l = tid & 127;
        bool differ = false;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int mr = tm * C::ROWS + rank * GM + (l >> 3) + 16 * q;
          const int64_t at = (int64_t)(p.T > 0 ? mr % p.T : 0) * p.slab + (wide ? grp * 32 : 0) + (l & 7) * 4;
          cs4[q] = *reinterpret_cast<const float4*>(p.cosT + at);
          sn4[q] = *reinterpret_cast<const float4*>(p.sinT + at);
          if (wide) {
            const float4 c2 = *reinterpret_cast<const float4*>(p.cosT + at + 64), s2 = *reinterpret_cast<const float4*>(p.sinT + at + 64);
            differ |= c2.x != cs4[q].x || c2.y != cs4[q].y || c2.z != cs4[q].z || c2.w != cs4[q].w || s2.x != sn4[q].x ||
                      s2.y != sn4[q].y || s2.z != sn4[q].z || s2.w != sn4[q].w;
          }
        }
        if (chief) tma_store_wait_read0();
        halves_differ = named_bar_or(1 + grp, 128, differ);
        auto own_row = [&](float4 (&x)[8]) {
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const int r = (l >> 3) + 16 * q;
            *reinterpret_cast<float4*>(stg + r * 128 + (((l & 7) ^ (r & 7)) << 4)) = x[q];
          }
          named_bar_sync(1 + grp, 128);
#pragma unroll
          for (int c = 0; c < 8; ++c) x[c] = *reinterpret_cast<const float4*>(stg + row * 128 + ((c ^ (row & 7)) << 4));
          named_bar_sync(1 + grp, 128);
        };
        own_row(cs4);
        own_row(sn4);
      }
      const uint32_t tsrc = tmem + ((uint32_t)(quad * 32) << 16) + buf * GN;
      // gated MLP: blocks come in (gate, up) pairs, a group takes a pair and produces 64 output columns
      const int n_steps = swiglu ? (nsub + 3) / 4 : (nsub + 1) / 2;
      for (int st = 0; st < n_steps; ++st) {
        const int u = swiglu ? (2 * st + grp) * 2 : 2 * st + grp;
        const bool mine = u < nsub;
        const int out_col = swiglu ? (tn * GN + u * 64) / 2 : tn * GN + u * 64;
        if (st == 0) {
          // threads that meet at named barriers leave together: one whose wait ran out takes the others with it
          if (named_bar_or(bar_id, bar_n, !mbar_wait(&sl->acc_full[buf], (lt >> 1) & 1))) {
            dev_set_error(p.status, SAF_DEV_TIMEOUT_EPI, 13);
            if (p.residual_tma) mbar_wait(&sl->res[grp], n_res & 1);       // a copy may be on its way: let it land
            tile = tile_hi;
            break;
          }
          tc_fence_after();
        }
        const int sb = tn * SUBS + u;
        const bool both = wide && tb.rope[sb];   // (a rotated 128-row slab never meets one-block tiles)
        float v[64];
        if (mine) {
          uint32_t r0[32], r1[32];
          tmem_ld32(tsrc + (both ? 2 * st * 64 + grp * 32 : u * 64), r0);
          tmem_ld32(tsrc + (both ? (2 * st + 1) * 64 + grp * 32 : u * 64 + 32), r1);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            v[j] = __uint_as_float(r0[j]);
            v[32 + j] = __uint_as_float(r1[j]);
          }
          if (SUBS > 1 && swiglu) {   // v holds the gate block; the up block is the next 64 accumulator columns
#pragma unroll
            for (int c = 0; c < 64; c += 16) {
              uint32_t q[16];
              tmem_ld16(tsrc + (u + 1) * 64 + c, q);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 16; ++j) v[c + j] = silu_mul(v[c + j], __uint_as_float(q[j]));
            }
          }
        }
        if (st == n_steps - 1) {   // the accumulator has been read: the MMA warp may overwrite it
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            if constexpr (PAIR) mbar_arrive_cluster(cluster_addr_of(&sl->acc_empty[buf], 0));   // the even CTA's MMA warp waits
            else mbar_arrive(&sl->acc_empty[buf]);
          }
        }
        if (!mine) continue;
        {
          // bias of the columns in v[0..31] and v[32..63]
          const int sa = both ? tn * SUBS + 2 * st : sb;
          const int wa = tb.weight[sa], wb = p.halves ? tb.weightb[sb] : wa;
          const int ra = tb.row0[sa] + (both ? grp * 32 : 0);
          const int rb = both ? tb.row0[sa + 1] + grp * 32 : (p.halves ? tb.row0b[sb] : ra + 32);
          if (p.bias[wa]) {
            const __nv_bfloat16* bp = reinterpret_cast<const __nv_bfloat16*>(p.bias[wa]) + ra;
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] += __bfloat162float(bp[j]);
          }
          if (p.bias[wb]) {
            const __nv_bfloat16* bp = reinterpret_cast<const __nv_bfloat16*>(p.bias[wb]) + rb;
#pragma unroll
            for (int j = 0; j < 32; ++j) v[32 + j] += __bfloat162float(bp[j]);
          }
        }
        if (p.act == SAF_ACT_GELU) {
#pragma unroll
          for (int j = 0; j < 64; ++j) v[j] = gelu_erf(v[j]);
        }
        if (p.residual) {
          if (p.residual_tma) {     // the block is in staging; this thread's row takes its sums back to the same place
            if (!mbar_wait(&sl->res[grp], (n_res++) & 1)) dev_set_error(p.status, SAF_DEV_TIMEOUT_EPI, 14);
          }
          const __nv_bfloat16* rr = p.residual + (int64_t)m * p.ldr + tn * GN;
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            uint4 q = make_uint4(0, 0, 0, 0);
            if (p.residual_tma) q = *reinterpret_cast<const uint4*>(stg + row * 128 + ((c ^ (row & 7)) << 4));
            else if (m < p.M) q = *reinterpret_cast<const uint4*>(rr + (both ? (2 * st + (c >> 2)) * 64 + grp * 32 + (c & 3) * 8 : out_col - tn * GN + c * 8));
            const uint32_t w4[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              v[c * 8 + 2 * e] += __uint_as_float(w4[e] << 16);
              v[c * 8 + 2 * e + 1] += __uint_as_float(w4[e] & 0xffff0000u);
            }
          }
        }
        if (tb.rope[sb]) {   // pairs (d, d + slab/2) are v[j], v[32 + j].  Warp-uniform: rows past M are clipped by the store
#pragma unroll
          for (int j4 = 0; j4 < 8; ++j4) {
            const float cc[4] = {cs4[j4].x, cs4[j4].y, cs4[j4].z, cs4[j4].w}, ss[4] = {sn4[j4].x, sn4[j4].y, sn4[j4].z, sn4[j4].w};
            float4 c2 = cs4[j4], s2 = sn4[j4];
            if (halves_differ) {
              const int64_t at = (int64_t)(p.T > 0 ? m % p.T : 0) * p.slab + 64 + grp * 32 + j4 * 4;
              c2 = *reinterpret_cast<const float4*>(p.cosT + at);
              s2 = *reinterpret_cast<const float4*>(p.sinT + at);
            }
            const float cc2[4] = {c2.x, c2.y, c2.z, c2.w}, ss2[4] = {s2.x, s2.y, s2.z, s2.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int j = j4 * 4 + e;
              const float x1 = v[j], x2 = v[32 + j];
              v[j] = x1 * cc[e] - x2 * ss[e];
              v[32 + j] = x2 * cc2[e] + x1 * ss2[e];
            }
          }
        }
        // a group has one staging block: its last store has read it by now, the accumulator's way to here hid the wait
        if (!p.residual_tma) {
          if (chief) tma_store_wait_read0();
          named_bar_sync(bar_id, bar_n);
        }
        // bf16 pack -> swizzled staging: 16-byte chunk c of row r lands at chunk (c ^ (r & 7))
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          uint4 q;
          q.x = pack_bf16(v[c * 8 + 0], v[c * 8 + 1]);
          q.y = pack_bf16(v[c * 8 + 2], v[c * 8 + 3]);
          q.z = pack_bf16(v[c * 8 + 4], v[c * 8 + 5]);
          q.w = pack_bf16(v[c * 8 + 6], v[c * 8 + 7]);
          uint8_t* dst = (both ? out_stage + (c >> 2) * (OUT_BYTES / 2) : stg) + row * 128;
          const int ch = both ? grp * 4 + (c & 3) : c;
          *reinterpret_cast<uint4*>(dst + ((ch ^ (row & 7)) << 4)) = q;
        }
        fence_proxy_async_smem();
        named_bar_sync(bar_id, bar_n);
        if (chief) {
          tma_store_2d(&mapO, stg, out_col, tm * C::ROWS + rank * GM);
          tma_store_commit();
          if (p.residual_tma) {
            tma_store_wait_read0();
            ask_residual(tile, st + 1);
          }
        }
      }
    }
    if (chief) tma_store_wait_all();
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) {
    cluster_sync_all();               // nothing of the peer's is touched after this point
    if (warp == 1) tmem_dealloc_pair(tmem, C::TMEM_COLS);
  } else {
    if (warp == 1) tmem_dealloc(tmem, C::TMEM_COLS);
  }
}

// Column tiles whose weights are walked together: groups of equal width of at most 32 MB, a quarter of the L2 (its two
// halves may hold a line each).
int columns_together(int tiles_n, int tile_cols, int K) {
  const int64_t bytes = (int64_t)tiles_n * tile_cols * K * 2;
  const int groups = (int)std::min<int64_t>(tiles_n, (bytes + (32 << 20) - 1) / (32 << 20));
  return (tiles_n + groups - 1) / groups;
}

bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

constexpr size_t PAIR_SMEM = 1024 + GCfg<true, 4>::STAGES * GCfg<true, 4>::STAGE_BYTES + OUT_BYTES + sizeof(SmemLayout);
static_assert(PAIR_SMEM <= 227 * 1024, "pair kernel shared memory");

// CTA pairs that can be resident at once (an SM without a free neighbour in its GPC stays out), after the pair kernel
// has its shared memory
int resident_pairs(cudaStream_t st, int* out) {
  auto kernel = indexed_gemm_kernel<true, 4>;
  static PerDeviceOnce smem_once;
  if (int rc = ensure_dyn_smem(kernel, (int)PAIR_SMEM, smem_once)) return rc;
  static std::atomic<int> cache[SAF_MAX_DEVICES];
  const int dev = current_device();
  int pairs = (dev >= 0 && dev < SAF_MAX_DEVICES) ? cache[dev].load(std::memory_order_acquire) : 0;
  if (pairs <= 0) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.blockDim = dim3(GEMM_THREADS);
    cfg.dynamicSmemBytes = PAIR_SMEM;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3(device_sm_count() & ~1);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n <= 0) {
      cudaGetLastError();
      n = device_sm_count() / 2;
    }
    pairs = n;
    if (dev >= 0 && dev < SAF_MAX_DEVICES) cache[dev].store(pairs, std::memory_order_release);
  }
  *out = pairs;
  return SAF_OK;
}

template <int SUBS>
int launch_single(const CUtensorMap& mx, const CUtensorMap* mw, const CUtensorMap& mo, const CUtensorMap& mr, GemmParams p, const SubTable& tb,
                  cudaStream_t st) {
  using C = GCfg<false, SUBS>;
  constexpr size_t smem = 1024 + C::STAGES * C::STAGE_BYTES + OUT_BYTES + sizeof(SmemLayout);
  static_assert(smem <= 227 * 1024, "single-CTA kernel shared memory");
  static PerDeviceOnce smem_once;
  if (int rc = ensure_dyn_smem(indexed_gemm_kernel<false, SUBS>, (int)smem, smem_once)) return rc;
  p.tiles_n = (p.N + C::GN - 1) / C::GN;
  p.group_n = columns_together(p.tiles_n, C::GN, p.K);
  const int grid = std::min(device_sm_count(), p.tiles_m * p.tiles_n);
  return launch_pdl("indexed_gemm_kernel", indexed_gemm_kernel<false, SUBS>, dim3(grid), GEMM_THREADS, smem, st, 1, mx, mw[0], mw[1],
                    mw[2], mw[3], mo, mr, p, tb);
}

}  // namespace

int launch_gemm_sm100(const SafIndexedLinearArgs& a, cudaStream_t st, int32_t* zero2, bool weights_early) {
  if (a.dtype != SAF_BF16) return SAF_ERR_UNSUPPORTED;
  // slabs of 64 or 128 rows are whole 64-row weight blocks; other multiples of 32 (head_dim 96) are served as runs
  // of 32 rows, two per block, when the total width still fills whole 64-column blocks.  The rotation is fused in
  // the epilogue for the first kind only; for the second it runs as a second launch over the output.
  const bool halves = a.slab != 64 && a.slab != 128;
  if (halves && (a.slab % 32 || (a.n_slabs * a.slab) % 64 || a.act != SAF_ACT_NONE || a.residual)) return SAF_ERR_UNSUPPORTED;
  const int N = a.n_slabs * a.slab;
  if (N / 64 > MAX_SUB) return SAF_ERR_UNSUPPORTED;
  if (a.C % 8 || a.ldx % 8 || a.ldo % 8 || !aligned16(a.x) || !aligned16(a.out)) return SAF_ERR_UNSUPPORTED;
  if ((a.rope_cos && !aligned16(a.rope_cos)) || (a.rope_sin && !aligned16(a.rope_sin))) return SAF_ERR_UNSUPPORTED;
  if (a.residual && (!aligned16(a.residual) || a.ldr % 8)) return SAF_ERR_UNSUPPORTED;
  if (a.act == SAF_ACT_SWIGLU) {
    // (gate, up) pairs of 64-row blocks, no bias, no rotation; every tile holds whole pairs (4 blocks per tile)
    if (a.slab != 64 || a.n_slabs % 2 || a.slab_rope) return SAF_ERR_UNSUPPORTED;
    for (int w = 0; w < a.n_weights; ++w)
      if (a.biases[w]) return SAF_ERR_UNSUPPORTED;
  }
  for (int w = 0; w < a.n_weights; ++w) {
    if (!a.weights[w]) continue;
    if (a.ldw[w] % 8 || (a.cdw[w] != 0 && a.cdw[w] != 1) || !aligned16(a.weights[w])) return SAF_ERR_UNSUPPORTED;
  }
  if (!saf_device_supported()) return SAF_ERR_UNSUPPORTED;
  // Tables count only when some slab rotates: the form of the tiles and the epilogue's way through a 128-row slab (both
  // groups on one pair of blocks) have to follow from the same fact.
  bool rotates = false;
  for (int g = 0; g < a.n_slabs && a.slab_rope; ++g) rotates |= a.slab_rope[g] != 0;

  CUtensorMap mx, mw[4], mo, mr;
  int rc;
  {
    uint64_t dims[2] = {(uint64_t)a.C, (uint64_t)a.M};
    uint64_t strides[2] = {0, (uint64_t)a.ldx * 2};
    uint32_t box[2] = {GK, GM};
    if ((rc = make_tensor_map_bf16(&mx, a.x, 2, dims, strides, box, true))) return rc;
  }
  for (int w = 0; w < 4; ++w) {
    const int ww = (w < a.n_weights && a.weights[w]) ? w : 0;
    uint64_t dims[2] = {(uint64_t)a.C, (uint64_t)a.rows_w[ww]};
    uint64_t strides[2] = {0, (uint64_t)a.ldw[ww] * 2};
    uint32_t box[2] = {GK, halves ? 32u : 64u};
    if ((rc = make_tensor_map_bf16(&mw[w], a.weights[ww], 2, dims, strides, box, true))) return rc;
  }
  {
    // gated MLP: the output holds one column per (gate, up) pair
    uint64_t dims[2] = {(uint64_t)(a.act == SAF_ACT_SWIGLU ? N / 2 : N), (uint64_t)a.M};
    uint64_t strides[2] = {0, (uint64_t)a.ldo * 2};
    uint32_t box[2] = {64, GM};
    if ((rc = make_tensor_map_bf16(&mo, a.out, 2, dims, strides, box, false))) return rc;
  }
  // (a residual whose rows overlap, such as one row for all, has no tensor map: it is read row by row)
  const bool residual_tma = a.residual && !rotates && a.act != SAF_ACT_SWIGLU && (a.ldr >= N || a.M == 1);
  mr = mo;
  if (residual_tma) {
    uint64_t dims[2] = {(uint64_t)N, (uint64_t)a.M};
    uint64_t strides[2] = {0, (uint64_t)std::max<int64_t>(a.ldr, N) * 2};     // (M == 1: any stride)
    uint32_t box[2] = {64, GM};
    if ((rc = make_tensor_map_bf16(&mr, a.residual, 2, dims, strides, box, false))) return rc;
  }
  SubTable tb;
  memset(&tb, 0, sizeof(tb));
  if (halves) {
    for (int hb = 0; hb < N / 32; ++hb) {          // 32-column runs of the output, two per block
      const int g = (hb * 32) / a.slab, r = (hb * 32) % a.slab;
      if (hb & 1) {
        tb.row0b[hb >> 1] = a.slab_row0[g] + r;
        tb.weightb[hb >> 1] = (uint8_t)a.slab_weight[g];
      } else {
        tb.row0[hb >> 1] = a.slab_row0[g] + r;
        tb.weight[hb >> 1] = (uint8_t)a.slab_weight[g];
      }
    }
  } else {
    const int per = a.slab / 64;
    for (int g = 0; g < a.n_slabs; ++g)
      for (int u = 0; u < per; ++u) {
        tb.row0[g * per + u] = a.slab_row0[g] + u * 64;
        tb.weight[g * per + u] = (uint8_t)a.slab_weight[g];
        tb.rope[g * per + u] = (uint8_t)(a.slab_rope ? (a.slab_rope[g] != 0) : 0);
      }
  }
  GemmParams p;
  memset(&p, 0, sizeof(p));
  p.M = a.M; p.N = N; p.K = a.C; p.T = a.T; p.slab = a.slab;
  for (int w = 0; w < a.n_weights; ++w) p.bias[w] = a.biases[w];
  p.cosT = rotates && !halves ? a.rope_cos : nullptr;     // halves: rotated by a launch of its own, below
  p.sinT = a.rope_sin;
  p.status = a.status;
  p.act = a.act;
  p.residual = reinterpret_cast<const __nv_bfloat16*>(a.residual);
  p.ldr = a.ldr;
  p.residual_tma = residual_tma ? 1 : 0;
  p.runs = p.cosT ? 1 : 0;
  p.halves = halves ? 1 : 0;
  p.zero2 = zero2;
  p.weights_early = weights_early ? 1 : 0;

  const bool together = a.act == SAF_ACT_SWIGLU || (a.slab == 128 && p.cosT);
  const char* pair_env = getenv("SAF_B200_GEMM_PAIR");
  const bool pair_off = pair_env && pair_env[0] == '0' && pair_env[1] == 0;
  int pairs = 0;
  if (!pair_off && N >= 256 && (rc = resident_pairs(st, &pairs))) return rc;
  const int form = pick_form(a.M, N, (a.C + GK - 1) / GK, together ? 2 : 1, pairs);
  if (form == PAIR_FORM) {
    using C = GCfg<true, 4>;
    p.tiles_m = (a.M + C::ROWS - 1) / C::ROWS;
    p.tiles_n = (N + C::GN - 1) / C::GN;
    p.group_n = columns_together(p.tiles_n, C::GN, p.K);
    pairs = std::min(pairs, p.tiles_m * p.tiles_n);
    if ((rc = launch_pdl("indexed_gemm_kernel<pair>", indexed_gemm_kernel<true, 4>, dim3(2 * pairs), GEMM_THREADS, PAIR_SMEM, st, 2, mx, mw[0], mw[1], mw[2], mw[3],
                         mo, mr, p, tb)))
      return rc;
  } else {
    p.tiles_m = (a.M + GM - 1) / GM;
    switch (form) {
      case 1: rc = launch_single<1>(mx, mw, mo, mr, p, tb, st); break;
      case 2: rc = launch_single<2>(mx, mw, mo, mr, p, tb, st); break;
      default: rc = launch_single<4>(mx, mw, mo, mr, p, tb, st); break;
    }
    if (rc) return rc;
  }
  if (halves && rotates)
    return launch_rope_slabs(a.out, a.ldo, a.M, a.n_slabs, a.slab, a.T, a.slab_rope, a.rope_cos, a.rope_sin, a.dtype, 0, st);
  return SAF_OK;
}

}  // namespace saf
