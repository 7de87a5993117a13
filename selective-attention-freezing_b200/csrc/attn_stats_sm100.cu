// Attention statistics for the freeze controller without the (B, H, T, T) capture.
//
// The reference measures heads by running the eager path with capture on and reducing the retained
// softmax(QK^T) tensor: batch mean per cell, centred sum of squares reduced per head, and sum p log p per head
// (nanogpt/dynamic_freeze.py:96-127 _centered_batch_reduced_moments, :130-143 _merge_reduced_moments,
// :146-173 _negative_entropy_sum, used by _measure :629-745).  Here a CTA takes one 128 x 64 cell tile of one head
// at a time: S_b = Q_b K_b^T of up to four samples on tcgen05 into TMEM, then per cell P_b = exp2(S_b scale - lse_b) with
// the row log-sum-exp (row_lse_sm100.cu), the samples' mean and the squares about it, and the Chan merge into the
// tile of the running mean; the per-head scalars are reduced to one double atomic per CTA and head.
//
// LOGITS: the same walk over the raw scores q k^T * sm_scale of the whole square (nothing masked, tiles above the
// diagonal included), for the priors that sample logits (`_last_logits`, nanogpt/model.py:828-831, reduced at
// nanogpt/dynamic_freeze.py:721-737 with _centered_batch_moments / _merge_moments, :62-93): running mean per cell and,
// when asked for, the centred squares per cell; no per-head scalars.
//
// What bounds it: the running statistics, 8 (LOGITS 16) bytes per cell read and written once.  So they move on their own:
// the running tile arrives in shared memory while the tile before is worked on (two buffers), is updated in place and
// leaves from there, and a thread that owns half a row reads and writes it as 16-byte pieces of 128-byte-swizzled rows.
// All samples of a cell are in TMEM at once, so mean and centred squares need no memory at all; more than four samples
// are merged four at a time into the tile in shared memory.
// 9 heads, T = 4096, four samples on a B200: raw scores with centred squares 1142 -> 400 us (2.4 GB, 6.0 TB/s),
// probabilities 373 -> 263 us (302 M probabilities; their tiles alone take 90 us), and 212 us since two cells go through each
// instruction and a cell's mean and centred squares come from sums over the samples instead of chains of updates.
//
//   warps 0-7: two warpgroups x 32 key columns, thread = query row (TMEM lane)
//   warp 8: TMA producer ([Q_b tile | K_b tile] ring), warp 9: MMA issuer
//   warps 10-11: running tiles in and out: one thread with TMA, or (T not a multiple of 4: rows do not start on 16-byte
//                boundaries) both warps with 4-byte cp.async and coalesced stores
// Every mbarrier wait is bounded; on expiry the kernel records a code in *status and falls through.
#include <type_traits>

#include "saf_internal.h"
#include "sm100_prims.cuh"

namespace saf {
namespace {

constexpr int AS_COMPUTE = 256;
constexpr int AS_THREADS = AS_COMPUTE + 128;
constexpr int AS_COLS = 64;                  // key columns of a tile
constexpr int AS_GROUP = 4;                  // samples of one unit of work: their scores are in TMEM together
constexpr int AS_STATE = 128 * AS_COLS * 4;  // one running tile: two boxes of 128 rows x 32 columns
constexpr float AS_LN2 = 0.6931471805599453f;

struct AsParams {
  int B, U, T, n_it, n_jt;
  float scale_log2;
  float scale;                 // LOGITS: sm_scale itself
  float* cell_m2;              // LOGITS: (U, T, T) or null
  const float* lse;
  int64_t lse_s[3];
  float* mean;                 // (U, T, T)
  long long count_prev;
  double* head_m2;
  double* neg_entropy;
  int* status;
};

struct AsShared {
  uint64_t full[4], empty[4], s_full[2], s_empty[2];
  uint64_t old_full[2], done[2];               // a state buffer holds its running tile (or is free) / is updated
  uint32_t tmem_base;
  double red[2][AS_COMPUTE / 32];
};

template <int HD, bool LOGITS>
struct AsCfg {
  static constexpr int Q_BYTES = 128 * HD * 2, K_BYTES = AS_COLS * HD * 2;
  static constexpr int NS = (HD == 64) ? 4 : 2;
  static constexpr int MATS = LOGITS ? 2 : 1;                // running tiles: mean, centred squares
  static constexpr int SMEM_BYTES = 1024 + NS * (Q_BYTES + K_BYTES) + 2 * MATS * AS_STATE + (int)sizeof(AsShared);
  static constexpr int TMEM_COLS = 512;                      // two units x four samples x 64 columns
  static_assert(SMEM_BYTES <= 227 * 1024, "statistics kernel shared memory");
};

__device__ __forceinline__ float as_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Persistent: CTA c owns tiles c, c + gridDim.x, ... of the list (head, query tile, key tile); probabilities are zero
// above the diagonal, so their list holds the 2 (it + 1) key tiles that query tile `it` can see.
struct AsTile {
  int u, it, jt;
};
template <bool LOGITS>
__host__ __device__ __forceinline__ int64_t as_tiles_per_head(int n_it, int n_jt) {
  if (LOGITS) return (int64_t)n_it * n_jt;
  return (int64_t)n_it * (n_it - 1) + (2 * n_it < n_jt ? 2 * n_it : n_jt);
}
template <bool LOGITS>
__device__ __forceinline__ AsTile as_decode(const AsParams& p, int t) {
  const int per = (int)as_tiles_per_head<LOGITS>(p.n_it, p.n_jt);
  AsTile x;
  x.u = t / per;
  const int rem = t - x.u * per;
  if (LOGITS) {
    x.it = rem / p.n_jt;
    x.jt = rem - x.it * p.n_jt;
  } else {                                                   // it (it + 1) tiles lie before query tile `it`
    x.it = (int)((sqrtf(4.f * (float)rem + 1.f) - 1.f) * 0.5f);
    while (x.it * (x.it + 1) > rem) --x.it;
    while ((x.it + 1) * (x.it + 2) <= rem) ++x.it;
    x.jt = rem - x.it * (x.it + 1);
  }
  return x;
}
// byte offset of cell (r, c) inside a running tile
__device__ __forceinline__ int as_cell(int r, int c) {
  return (c >> 5) * (AS_STATE / 2) + r * 128 + ((((c & 31) >> 2) ^ (r & 7)) << 4) + (c & 3) * 4;
}

// TMA_STATE: running tiles move by TMA (T a multiple of 4)
template <int HD, bool LOGITS, bool TMA_STATE>
__global__ void __launch_bounds__(AS_THREADS, 1)
attn_stats_kernel(const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapK,
                  const __grid_constant__ CUtensorMap mapMean, const __grid_constant__ CUtensorMap mapM2,
                  const __grid_constant__ AsParams p) {
  using C = AsCfg<HD, LOGITS>;
  const int total = (int)as_tiles_per_head<LOGITS>(p.n_it, p.n_jt) * p.U;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n_groups = (p.B + AS_GROUP - 1) / AS_GROUP;
  const bool has_m2 = LOGITS && p.cell_m2;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* ring = smem;                                      // stage s: [Q_b tile | K_b tile]
  constexpr int STAGE = C::Q_BYTES + C::K_BYTES;
  uint8_t* state = ring + C::NS * STAGE;                     // buffer k: [mean | centred squares]
  AsShared* sh = reinterpret_cast<AsShared*>(state + 2 * C::MATS * AS_STATE);
  constexpr int W_TMA = AS_COMPUTE / 32, W_MMA = W_TMA + 1, W_MOVE = W_TMA + 2;

  if (tid == 0) {
    for (int s = 0; s < 4; ++s) {
      mbar_init(&sh->full[s], 1);
      mbar_init(&sh->empty[s], 1);                           // the MMA's commit
    }
    for (int k = 0; k < 2; ++k) {
      mbar_init(&sh->s_full[k], 1);
      mbar_init(&sh->s_empty[k], AS_COMPUTE / 32);           // one lane of every compute warp
      mbar_init(&sh->old_full[k], TMA_STATE ? 1 : 64);
      mbar_init(&sh->done[k], AS_COMPUTE / 32);
    }
    fence_mbar_init();
  }
  if (warp == W_MMA) {
    tmem_alloc(&sh->tmem_base, C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh->tmem_base;

  if (warp == W_TMA) {
    if (elect_one()) {
      tma_prefetch_desc(&mapQ);
      tma_prefetch_desc(&mapK);
      int i = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
        const AsTile x = as_decode<LOGITS>(p, t);
        for (int b = 0; b < p.B; ++b, ++i) {
          const int s = i % C::NS;
          if (!mbar_wait(&sh->empty[s], ((i / C::NS) & 1) ^ 1)) {
            dev_set_error(p.status, SAF_DEV_TIMEOUT_TMA, 80);
            ok = false;
            break;
          }
          uint8_t* dst = ring + s * STAGE;
          mbar_expect_tx(&sh->full[s], STAGE);
#pragma unroll
          for (int hh = 0; hh < HD / 64; ++hh) {
            tma_load_4d(dst + hh * 16384, &mapQ, &sh->full[s], hh * 64, x.it * 128, x.u, b);
            tma_load_4d(dst + C::Q_BYTES + hh * 8192, &mapK, &sh->full[s], hh * 64, x.jt * AS_COLS, x.u, b);
          }
        }
      }
    }
  } else if (warp == W_MMA) {
    const bool leader = elect_one();
    const uint32_t idesc = umma_idesc_bf16(128, AS_COLS, 0, 0);
    const uint32_t aR = smem_u32(ring);
    int i = 0, g = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
      for (int b = 0; b < p.B; ++b, ++i) {
        const int s = i % C::NS, k = g & 1;
        if ((b % AS_GROUP == 0 && !mbar_wait(&sh->s_empty[k], ((g >> 1) & 1) ^ 1)) || !mbar_wait(&sh->full[s], (i / C::NS) & 1)) {
          dev_set_error(p.status, SAF_DEV_TIMEOUT_MMA, 81);
          ok = false;
          break;
        }
        tc_fence_after();
        const bool last = b % AS_GROUP == AS_GROUP - 1 || b == p.B - 1;
        if (leader) {
          const uint32_t aQ = aR + s * STAGE, aK = aQ + C::Q_BYTES;
#pragma unroll
          for (int ks = 0; ks < HD / 16; ++ks)
            umma_ss(tmem + k * 256 + (b % AS_GROUP) * AS_COLS, umma_smem_desc_sw128(aQ + (ks >> 2) * 16384 + (ks & 3) * 32, 16, 1024),
                    umma_smem_desc_sw128(aK + (ks >> 2) * 8192 + (ks & 3) * 32, 16, 1024), idesc, ks > 0);
          umma_commit(&sh->empty[s]);
          if (last) umma_commit(&sh->s_full[k]);
        }
        __syncwarp();
        g += last;
      }
    }
  } else if (warp >= W_MOVE) {
    // ------------------------------------------------------------------ running tiles in and out
    const bool any_old = p.count_prev > 0;                   // the first call only writes
    if constexpr (TMA_STATE) {
      if (warp == W_MOVE && elect_one()) {
        auto fetch = [&](int t, int k) {
          if (t >= total) return;
          if (!any_old) {                                    // nothing to bring: the buffer is free
            mbar_arrive(&sh->old_full[k]);
            return;
          }
          const AsTile x = as_decode<LOGITS>(p, t);
          // (both boxes, also one behind the last column: the cells the merge sees there are zeros)
          mbar_expect_tx(&sh->old_full[k], (has_m2 ? 2 : 1) * AS_STATE);
          for (int h = 0; h < 2; ++h) {
            uint8_t* dst = state + k * C::MATS * AS_STATE + h * (AS_STATE / 2);
            tma_load_4d(dst, &mapMean, &sh->old_full[k], x.jt * AS_COLS + h * 32, x.it * 128, x.u, 0);
            if (has_m2) tma_load_4d(dst + AS_STATE, &mapM2, &sh->old_full[k], x.jt * AS_COLS + h * 32, x.it * 128, x.u, 0);
          }
        };
        fetch(blockIdx.x, 0);
        fetch(blockIdx.x + gridDim.x, 1);
        int n = 0;
        for (int t = blockIdx.x; t < total; t += gridDim.x, ++n) {
          const int k = n & 1;
          if (!mbar_wait(&sh->done[k], (n >> 1) & 1)) {
            dev_set_error(p.status, SAF_DEV_TIMEOUT_EPI, 83);
            break;
          }
          const AsTile x = as_decode<LOGITS>(p, t);
          const int boxes = x.jt * AS_COLS + 32 < p.T ? 2 : 1;
          for (int h = 0; h < boxes; ++h) {
            const uint8_t* src = state + k * C::MATS * AS_STATE + h * (AS_STATE / 2);
            tma_store_4d(&mapMean, src, x.jt * AS_COLS + h * 32, x.it * 128, x.u, 0);
            if (has_m2) tma_store_4d(&mapM2, src + AS_STATE, x.jt * AS_COLS + h * 32, x.it * 128, x.u, 0);
          }
          tma_store_commit();
          tma_store_wait_read0();
          fetch(t + 2 * gridDim.x, k);
        }
        tma_store_wait_all();
      }
    } else {
      // thread (warp w, lane): rows w, w + 2, ...; columns lane and lane + 32.  A thread stores from and loads into the
      // same places of a buffer, so its own order is all the ordering they need.
      const int w = warp - W_MOVE;
      auto fetch = [&](int t, int k) {
        if (t >= total) return;
        const AsTile x = as_decode<LOGITS>(p, t);
        uint8_t* dst = state + k * C::MATS * AS_STATE;
        for (int r = w; any_old && r < 128; r += 2)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int gi = x.it * 128 + r, gj = x.jt * AS_COLS + h * 32 + lane;
            const bool in = gi < p.T && gj < p.T;
            const int64_t at = in ? ((int64_t)x.u * p.T + gi) * p.T + gj : 0;
            cp_async4_zfill(dst + as_cell(r, h * 32 + lane), p.mean + at, in);
            if (has_m2) cp_async4_zfill(dst + AS_STATE + as_cell(r, h * 32 + lane), p.cell_m2 + at, in);
          }
        cp_async_mbar_arrive(&sh->old_full[k]);
      };
      fetch(blockIdx.x, 0);
      fetch(blockIdx.x + gridDim.x, 1);
      int n = 0;
      for (int t = blockIdx.x; t < total; t += gridDim.x, ++n) {
        const int k = n & 1;
        if (!mbar_wait(&sh->done[k], (n >> 1) & 1)) {
          dev_set_error(p.status, SAF_DEV_TIMEOUT_EPI, 83);
          break;
        }
        const AsTile x = as_decode<LOGITS>(p, t);
        const uint8_t* src = state + k * C::MATS * AS_STATE;
#pragma unroll 4
        for (int r = w; r < 128; r += 2)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int gi = x.it * 128 + r, gj = x.jt * AS_COLS + h * 32 + lane;
            if (gi >= p.T || gj >= p.T) continue;
            const int64_t at = ((int64_t)x.u * p.T + gi) * p.T + gj;
            p.mean[at] = *reinterpret_cast<const float*>(src + as_cell(r, h * 32 + lane));
            if (has_m2) p.cell_m2[at] = *reinterpret_cast<const float*>(src + AS_STATE + as_cell(r, h * 32 + lane));
          }
        fetch(t + 2 * gridDim.x, k);
      }
      cp_async_wait_all();
    }
  } else {
    // ------------------------------------------------------------------ compute warpgroups
    const int half = warp >> 2;
    const int r = (warp & 3) * 32 + lane;           // query row of the tile
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const float sc = p.scale_log2;
    // per-head scalars of this thread, handed to the head's two doubles when the CTA moves to another head
    double m2sum = 0.0, esum = 0.0;
    int cur_u = -1;
    auto flush_head = [&]() {
#pragma unroll
      for (int off = 16; off; off >>= 1) {
        m2sum += __shfl_xor_sync(0xffffffffu, m2sum, off);
        esum += __shfl_xor_sync(0xffffffffu, esum, off);
      }
      named_bar_sync(1, AS_COMPUTE);                // the previous flush has been read
      if (lane == 0) {
        sh->red[0][warp] = m2sum;
        sh->red[1][warp] = esum;
      }
      named_bar_sync(1, AS_COMPUTE);
      if (tid < 2) {
        double tot = 0.0;
        for (int wq = 0; wq < AS_COMPUTE / 32; ++wq) tot += sh->red[tid][wq];
        atomicAdd(tid == 0 ? &p.head_m2[cur_u] : &p.neg_entropy[cur_u], tot);
      }
      m2sum = esum = 0.0;
    };
    // row log-sum-exps of a unit's samples, asked for one unit ahead; +inf: rows past T hold zeros
    auto row_lse = [&](int t, int gr, float (&L)[AS_GROUP]) {
      if (t >= total) return;
      const AsTile x = as_decode<LOGITS>(p, t);
      const int gi = x.it * 128 + r;
      const float* lse = p.lse + (int64_t)x.u * p.lse_s[1] + (int64_t)gi * p.lse_s[2];
#pragma unroll
      for (int b = 0; b < AS_GROUP; ++b)
        L[b] = (gi < p.T && gr * AS_GROUP + b < p.B) ? lse[(int64_t)(gr * AS_GROUP + b) * p.lse_s[0]] : INFINITY;
    };
    float Ln[AS_GROUP];
    if constexpr (!LOGITS) row_lse(blockIdx.x, 0, Ln);
    int g = 0, n = 0;
    bool ok = true;
    float w = 0.f, cw = 0.f;                        // weights of the merge: nb / (c0 + nb), c0 nb / (c0 + nb)
    double cwd = 0.0;
    // (a warp whose wait ran out keeps walking its tiles, doing nothing but its part of flush_head's barriers: the others
    // end on their own limits instead of waiting there for it)
    for (int t = blockIdx.x; t < total; t += gridDim.x, ++n) {
      const AsTile x = as_decode<LOGITS>(p, t);
      if (!LOGITS && x.u != cur_u) {
        if (cur_u >= 0) flush_head();
        cur_u = x.u;
      }
      if (!ok) continue;
      const int gi = x.it * 128 + r;
      const int gj0 = x.jt * AS_COLS + half * 32;
      const bool diag = x.jt * AS_COLS + AS_COLS - 1 > x.it * 128;
      uint8_t* mrow = state + (n & 1) * C::MATS * AS_STATE + half * (AS_STATE / 2) + r * 128;
      for (int gr = 0; gr < n_groups; ++gr, ++g) {
        const int k = g & 1, b0 = gr * AS_GROUP, nb = min(AS_GROUP, p.B - b0);
        const long long c0 = p.count_prev + b0;
        if (n_groups > 1 || g == 0) {
          const double tot = (double)c0 + (double)nb;
          w = (float)((double)nb / tot);
          cwd = (double)c0 * (double)nb / tot;
          cw = (float)cwd;
        }
        float L[AS_GROUP];
        if constexpr (!LOGITS) {
#pragma unroll
          for (int b = 0; b < AS_GROUP; ++b) L[b] = Ln[b];
        }
        const bool got = mbar_wait(&sh->s_full[k], (g >> 1) & 1) && (gr > 0 || mbar_wait(&sh->old_full[n & 1], (n >> 1) & 1));
        if (!__all_sync(0xffffffffu, got)) {
          dev_set_error(p.status, SAF_DEV_TIMEOUT_SOFTMAX, 82);
          ok = false;
          break;
        }
        tc_fence_after();
        if constexpr (!LOGITS) row_lse(gr + 1 < n_groups ? t : t + gridDim.x, gr + 1 < n_groups ? gr + 1 : 0, Ln);
        float2 ent2 = make_float2(0.f, 0.f);          // sum p log2 p of this thread's cells
        double corr = 0.0;
        // Two cells at a time on packed pairs: the samples' mean, then the squares about it -- sums instead of a chain of
        // updates.  Compiled per number of samples and for tiles the diagonal crosses.
        auto cells = [&](auto nb_c, auto diag_c) {
          constexpr int NB = decltype(nb_c)::value;
          constexpr bool DIAG = decltype(diag_c)::value;
          const float2 f2 = make_float2(LOGITS ? p.scale : sc, LOGITS ? p.scale : sc), inv2 = make_float2(1.f / NB, 1.f / NB);
          const float2 w2 = make_float2(w, w);
#pragma unroll
          for (int c16 = 0; c16 < 2; ++c16) {
            uint32_t d[NB][16];
#pragma unroll
            for (int b = 0; b < NB; ++b)
              tmem_ld16(tmem + lane_base + k * 256 + b * AS_COLS + half * 32 + c16 * 16, d[b]);
            tmem_ld_wait();
#pragma unroll
            for (int c4 = 0; c4 < 4; ++c4) {
              float4* mp = reinterpret_cast<float4*>(mrow + (((c16 * 4 + c4) ^ (r & 7)) << 4));
              float4* qp = reinterpret_cast<float4*>(reinterpret_cast<uint8_t*>(mp) + AS_STATE);
              float2 mm[2], m2[2];
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                const int c = c4 * 4 + 2 * e;
                float2 pe[NB], sum = make_float2(0.f, 0.f);
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                  const float2 v = make_float2(__uint_as_float(d[b][c]), __uint_as_float(d[b][c + 1]));
                  if constexpr (LOGITS) {
                    pe[b] = __fmul2_rn(v, f2);                                   // the raw scores
                  } else {
                    float2 x2 = __ffma2_rn(v, f2, make_float2(-L[b], -L[b]));    // log2 of the probabilities
                    if constexpr (DIAG) {                                        // causal mask
                      if (gj0 + c16 * 16 + c > gi) x2.x = -INFINITY;
                      if (gj0 + c16 * 16 + c + 1 > gi) x2.y = -INFINITY;
                    }
                    pe[b] = make_float2(as_ex2(x2.x), as_ex2(x2.y));
                    // (p = 0 there, so the clamp only avoids 0 * inf)
                    ent2 = __ffma2_rn(pe[b], make_float2(fmaxf(x2.x, -200.f), fmaxf(x2.y, -200.f)), ent2);
                  }
                  sum = b == 0 ? pe[0] : __fadd2_rn(sum, pe[b]);
                }
                mm[e] = NB == 1 ? sum : __fmul2_rn(sum, inv2);
                m2[e] = make_float2(0.f, 0.f);
                if constexpr (NB > 1) {
#pragma unroll
                  for (int b = 0; b < NB; ++b) {
                    const float2 dlt = __fadd2_rn(pe[b], make_float2(-mm[e].x, -mm[e].y));
                    m2[e] = __ffma2_rn(dlt, dlt, m2[e]);
                  }
                }
              }
              if constexpr (!LOGITS) m2sum += (double)(m2[0].x + m2[0].y) + (double)(m2[1].x + m2[1].y);
              if (c0 > 0) {                               // Chan merge into the running cells
                const float4 old = *mp;
                const float2 ov[2] = {make_float2(old.x, old.y), make_float2(old.z, old.w)};
                float2 o2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)}, cs = make_float2(0.f, 0.f);
                if (has_m2) {
                  const float4 q = *qp;
                  o2[0] = make_float2(q.x, q.y);
                  o2[1] = make_float2(q.z, q.w);
                }
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                  const float2 dlt = __fadd2_rn(mm[e], make_float2(-ov[e].x, -ov[e].y));
                  mm[e] = __ffma2_rn(dlt, w2, ov[e]);
                  if constexpr (LOGITS) m2[e] = __fadd2_rn(m2[e], __ffma2_rn(__fmul2_rn(dlt, dlt), make_float2(cw, cw), o2[e]));
                  else cs = __ffma2_rn(dlt, dlt, cs);
                }
                if constexpr (!LOGITS) corr += (double)(cs.x + cs.y);
              }
              *mp = make_float4(mm[0].x, mm[0].y, mm[1].x, mm[1].y);
              if (has_m2) *qp = make_float4(m2[0].x, m2[0].y, m2[1].x, m2[1].y);
            }
          }
        };
        auto by_count = [&](auto diag_c) {
          switch (nb) {
            case 1: cells(std::integral_constant<int, 1>{}, diag_c); break;
            case 2: cells(std::integral_constant<int, 2>{}, diag_c); break;
            case 3: cells(std::integral_constant<int, 3>{}, diag_c); break;
            default: cells(std::integral_constant<int, AS_GROUP>{}, diag_c);
          }
        };
        if (!LOGITS && diag) by_count(std::integral_constant<bool, !LOGITS>{});
        else by_count(std::false_type{});
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh->s_empty[k]);
        if constexpr (!LOGITS) {
          m2sum += corr * cwd;
          esum += (double)(ent2.x + ent2.y) * (double)AS_LN2;        // natural log, as the reference's xlogy
        }
      }
      if (!ok) continue;
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh->done[n & 1]);
    }
    if (!LOGITS && cur_u >= 0) flush_head();
    if (!LOGITS && p.count_prev == 0) {
      // above the diagonal every probability is zero: the first batch writes the zeros, later ones leave them
      const int64_t rows = (int64_t)p.U * p.T;
      for (int64_t row = (int64_t)blockIdx.x * (AS_COMPUTE / 32) + warp; row < rows; row += (int64_t)gridDim.x * (AS_COMPUTE / 32)) {
        const int i = (int)(row % p.T);
        float* dst = p.mean + row * p.T;
        for (int j = min(p.n_jt, 2 * (i / 128 + 1)) * AS_COLS + lane; j < p.T; j += 32) dst[j] = 0.f;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == W_MMA) tmem_dealloc(tmem, C::TMEM_COLS);
}

template <int HD, bool LOGITS, bool TMA_STATE>
int as_launch(const SafAttnStatsArgs& a, cudaStream_t st) {
  CUtensorMap mq, mk, mm, m2;
  int rc;
  if ((rc = make_row_tile_map_bf16(&mq, a.q, a.B, a.U, a.T, HD))) return rc;
  {
    uint64_t dims[4] = {(uint64_t)HD, (uint64_t)a.T, (uint64_t)a.U, (uint64_t)a.B};
    uint64_t strides[4] = {0, (uint64_t)a.k.stride[2] * 2, (uint64_t)a.k.stride[1] * 2, (uint64_t)a.k.stride[0] * 2};
    uint32_t box[4] = {64, AS_COLS, 1, 1};
    if ((rc = make_tensor_map_bf16(&mk, a.k.ptr, 4, dims, strides, box, true))) return rc;
  }
  mm = m2 = mq;
  if (TMA_STATE) {
    const uint64_t row = (uint64_t)a.T * 4;
    uint64_t dims[4] = {(uint64_t)a.T, (uint64_t)a.T, (uint64_t)a.U, 1};
    uint64_t strides[4] = {0, row, row * a.T, row * a.T * a.U};
    uint32_t box[4] = {32, 128, 1, 1};
    if ((rc = make_tensor_map_f32(&mm, a.mean, 4, dims, strides, box))) return rc;
    m2 = mm;
    if (LOGITS && a.cell_m2 && (rc = make_tensor_map_f32(&m2, a.cell_m2, 4, dims, strides, box))) return rc;
  }
  AsParams p;
  p.B = a.B; p.U = a.U; p.T = a.T;
  p.n_it = (a.T + 127) / 128;
  p.n_jt = (a.T + AS_COLS - 1) / AS_COLS;
  p.scale_log2 = a.sm_scale * 1.4426950408889634f;
  p.scale = a.sm_scale;
  p.cell_m2 = LOGITS ? a.cell_m2 : nullptr;
  p.lse = LOGITS ? nullptr : reinterpret_cast<const float*>(a.lse.ptr);
  for (int i = 0; i < 3; ++i) p.lse_s[i] = LOGITS ? 0 : a.lse.stride[i];
  p.mean = a.mean;
  p.count_prev = a.count_prev;
  p.head_m2 = a.head_m2;
  p.neg_entropy = a.neg_entropy;
  p.status = a.status;
  using C = AsCfg<HD, LOGITS>;
  static PerDeviceOnce smem_once;
  if (int rc2 = ensure_dyn_smem(attn_stats_kernel<HD, LOGITS, TMA_STATE>, C::SMEM_BYTES, smem_once)) return rc2;
  const int64_t tiles = as_tiles_per_head<LOGITS>(p.n_it, p.n_jt) * a.U;
  if ((int64_t)p.n_it * p.n_jt * a.U > 0x7fffffff / 2) return fail(SAF_ERR_LIMIT, "attention statistics: too many tiles");
  const int sm_count = device_sm_count();
  const int grid = (int)(tiles < sm_count ? tiles : sm_count);      // one persistent CTA per SM
  attn_stats_kernel<HD, LOGITS, TMA_STATE><<<(unsigned)grid, AS_THREADS, C::SMEM_BYTES, st>>>(mq, mk, mm, m2, p);
  count_launch();
  return check_launch("attn_stats_kernel");
}

template <int HD, bool LOGITS>
int as_dispatch(const SafAttnStatsArgs& a, cudaStream_t st) {
  // rows of T floats start on 16-byte boundaries when T is a multiple of 4: what TMA asks for
  return a.T % 4 == 0 ? as_launch<HD, LOGITS, true>(a, st) : as_launch<HD, LOGITS, false>(a, st);
}

}  // namespace

int launch_attn_stats_sm100(const SafAttnStatsArgs& a, cudaStream_t st) {
  if (a.dtype != SAF_BF16 || (a.HD != 64 && a.HD != 128)) return fail(SAF_ERR_UNSUPPORTED, "attention statistics: bf16 with head_dim 64 or 128 only");
  if (!tma_rows_ok(a.q) || !tma_rows_ok(a.k))
    return fail(SAF_ERR_UNSUPPORTED, "attention statistics: q, k need 16-byte aligned rows and unit last stride");
  if (a.quantity == SAF_STATS_LSE) {
    if (!saf_device_supported()) return fail(SAF_ERR_UNSUPPORTED, "attention statistics need an sm_100 device");
    return launch_row_lse_sm100(a, st);
  }
  if ((uintptr_t)a.mean & 15) return fail(SAF_ERR_INVALID, "attention statistics: mean must be 16-byte aligned");
  if (!saf_device_supported()) return fail(SAF_ERR_UNSUPPORTED, "attention statistics need an sm_100 device");
  if ((uintptr_t)a.cell_m2 & 15) return fail(SAF_ERR_INVALID, "attention statistics: cell_m2 must be 16-byte aligned");
  if (a.quantity == SAF_STATS_LOGITS) return a.HD == 64 ? as_dispatch<64, true>(a, st) : as_dispatch<128, true>(a, st);
  return a.HD == 64 ? as_dispatch<64, false>(a, st) : as_dispatch<128, false>(a, st);
}

}  // namespace saf
