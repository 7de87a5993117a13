// Row log-sum-exp of causal scores without the attention: lse[b,h,i] = log2 sum_{j<=i} 2^(q_i.k_j * scale * log2 e), what the
// controller statistics need before they can form probabilities.
//
// A forward attention launch gives the same numbers and a product nobody reads; here nothing follows the scores, so nothing
// waits on a softmax: score tiles run four ahead through the four 128-column quarters of tensor memory and four compute
// warpgroups each drain the quarter of their own (one thread per row, 32 columns at a time, running maximum and sum).
//   warp 0      TMA: Q tiles (two), K tiles (a ring of four), in the order the units ask for them
//   warp 1      S = Q K_j^T
//   warps 4-19  group g takes every fourth score tile; at the end of a row tile the four (maximum, sum) pairs of a row meet
//               in shared memory
// Persistent, one CTA per SM over (row tile, batch, head), longest row tiles first, rounds dealt out forwards and backwards.
// The special function unit needs 1024 cycles for 128 x 128 exponentials, so a quarter of them runs on the FMA pipe; the
// products of width 64 need 256.  9 heads x 64, T = 4096, B = 4 on a B200: 149 us through the attention forward, 107 here with all
// exponentials on the special function unit, 94 as it is (1400 cycles a tile: four warps a scheduler, the chains of maxima
// and sums between them).
#include <math.h>

#include <algorithm>

#include "saf_internal.h"
#include "sm100_prims.cuh"

namespace saf {
namespace {

constexpr int RL_GROUPS = 4, RL_THREADS = 128 + RL_GROUPS * 128;
constexpr int RL_KS = 4;                        // K stages
constexpr float RL_LOG2E = 1.4426950408889634f;
constexpr float RL_LOW = -3.402823466e38f;      // a maximum before the first score

template <int HD>
struct RlCfg {
  static constexpr int TILE = 128 * HD * 2;
  static constexpr int SMEM = 1024 + (2 + RL_KS) * TILE + 256 + 2 * RL_GROUPS * 128 * 8;
};
struct RlBars {
  uint64_t q_full[2], q_empty[2], k_full[RL_KS], k_empty[RL_KS], s_full[RL_GROUPS], s_empty[RL_GROUPS];
  uint32_t tmem_base;
};
static_assert(sizeof(RlBars) <= 256, "barrier block");

struct RlParams {
  int B, U, T, n_tiles, total;
  float scale;                 // |sm_scale| log2 e
  int negative;                // sm_scale < 0
  float* lse;
  int64_t s[3];
  int* status;
};

__device__ __forceinline__ float rl_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// the larger one, NaN if either is: a NaN score makes its row's maximum, and so the result, NaN
__device__ __forceinline__ float rl_max(float x, float y) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(x), "f"(y));
  return r;
}
// 2^x for x <= 0 on the FMA pipe: the fraction in [-1/2, 1/2] by a degree-4 polynomial (fitted to the smallest relative
// error, 2.6e-6), the integer part added to the exponent
__device__ __forceinline__ float2 rl_poly2(float2 x) {
  const float magic = 12582912.f;               // 1.5 * 2^23: its sum with x holds the nearest integer in the low bits
  x.x = fmaxf(x.x, -126.f);
  x.y = fmaxf(x.y, -126.f);
  const float2 t = __fadd2_rn(x, make_float2(magic, magic));
  const float2 n = __fadd2_rn(t, make_float2(-magic, -magic));
  const float2 f = __fadd2_rn(x, make_float2(-n.x, -n.y));
  float2 q = __ffma2_rn(f, make_float2(9.570102e-3f, 9.570102e-3f), make_float2(5.5917863e-2f, 5.5917863e-2f));
  q = __ffma2_rn(q, f, make_float2(0.24024744f, 0.24024744f));
  q = __ffma2_rn(q, f, make_float2(0.69312179f, 0.69312179f));
  q = __ffma2_rn(q, f, make_float2(0.99999928f, 0.99999928f));
  return make_float2(__int_as_float(__float_as_int(q.x) + (__float_as_int(t.x) << 23)),
                     __int_as_float(__float_as_int(q.y) + (__float_as_int(t.y) << 23)));
}

template <int HD>
__global__ void __launch_bounds__(RL_THREADS, 1) row_lse_kernel(const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapK,
                                                                const __grid_constant__ RlParams p) {
  using C = RlCfg<HD>;
  extern __shared__ uint8_t rl_smem[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)rl_smem + 1023) & ~(uintptr_t)1023);
  uint8_t *sQ = smem, *sK = smem + 2 * C::TILE;
  RlBars* bars = reinterpret_cast<RlBars*>(sK + RL_KS * C::TILE);
  float2* parts = reinterpret_cast<float2*>(reinterpret_cast<uint8_t*>(bars) + 256);     // [item parity][group][row]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // unit of round k: (batch, head) and row tile
  auto unit = [&](int k, int& bh, int& m) {
    const int i = k * gridDim.x + ((k & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
    if (i >= p.total) return false;
    const int heads = p.B * p.U;
    m = p.n_tiles - 1 - i / heads;
    bh = i % heads;
    return true;
  };
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->q_full[i], 1);
      mbar_init(&bars->q_empty[i], 1);
    }
    for (int i = 0; i < RL_KS; ++i) {
      mbar_init(&bars->k_full[i], 1);
      mbar_init(&bars->k_empty[i], 1);
    }
    for (int i = 0; i < RL_GROUPS; ++i) {
      mbar_init(&bars->s_full[i], 1);
      mbar_init(&bars->s_empty[i], 4);
    }
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_base;

  int bh, m;
  if (warp == 0) {
    if (lane == 0) {
      auto load = [&](uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int row, int h, int b) {
        mbar_expect_tx(bar, C::TILE);
#pragma unroll
        for (int hh = 0; hh < HD / 64; ++hh) tma_load_4d(dst + hh * 16384, map, bar, hh * 64, row, h, b);
      };
      tma_prefetch_desc(&mapQ);
      tma_prefetch_desc(&mapK);
      bool ok = true;
      for (int k = 0, n = 0; ok && unit(k, bh, m); ++k) {
        const int b = bh / p.U, h = bh - b * p.U;
        if (!(ok = mbar_wait(&bars->q_empty[k & 1], ((k >> 1) & 1) ^ 1))) break;
        load(sQ + (k & 1) * C::TILE, &mapQ, &bars->q_full[k & 1], m * 128, h, b);
        for (int j = 0; j <= m; ++j, ++n) {
          const int s = n % RL_KS;
          if (!(ok = mbar_wait(&bars->k_empty[s], ((n / RL_KS) & 1) ^ 1))) break;
          load(sK + s * C::TILE, &mapK, &bars->k_full[s], j * 128, h, b);
        }
      }
      if (!ok) dev_set_error(p.status, SAF_DEV_TIMEOUT_TMA, 90);
    }
  } else if (warp == 1) {
    const bool leader = elect_one();
    const uint32_t idesc = umma_idesc_bf16(128, 128, 0, 0);
    const uint32_t aQ = smem_u32(sQ), aK = smem_u32(sK);
    bool ok = true;
    for (int k = 0, n = 0; ok && unit(k, bh, m); ++k) {
      if (!(ok = mbar_wait(&bars->q_full[k & 1], (k >> 1) & 1))) break;
      const uint64_t dq = umma_smem_desc_sw128(aQ + (k & 1) * C::TILE, 16, 1024);
      for (int j = 0; j <= m; ++j, ++n) {
        const int s = n % RL_KS, g = n % RL_GROUPS;
        if (!(ok = mbar_wait(&bars->k_full[s], (n / RL_KS) & 1) && mbar_wait(&bars->s_empty[g], ((n / RL_GROUPS) & 1) ^ 1))) break;
        tc_fence_after();
        if (leader) {
          const uint64_t dk = umma_smem_desc_sw128(aK + s * C::TILE, 16, 1024);
#pragma unroll
          for (int ks = 0; ks < HD / 16; ++ks) {
            const uint32_t off = (ks >> 2) * 16384 + (ks & 3) * 32;
            umma_ss(tmem + g * 128, umma_desc_advance(dq, off), umma_desc_advance(dk, off), idesc, ks > 0);
          }
          umma_commit(&bars->k_empty[s]);
          umma_commit(&bars->s_full[g]);
          if (j == m) umma_commit(&bars->q_empty[k & 1]);
        }
        __syncwarp();
      }
    }
    if (!ok) dev_set_error(p.status, SAF_DEV_TIMEOUT_MMA, 91);
  } else if (warp >= 4) {
    const int g = (warp - 4) >> 2, row = (warp & 3) * 32 + lane;
    const uint32_t ts = tmem + ((uint32_t)((warp & 3) * 32) << 16) + g * 128;
    bool ok = true;
    for (int k = 0, n = 0; unit(k, bh, m); ++k, n += m + 1) {
      float mx = RL_LOW, l = 0.f;
      // this group's tiles of the row tile: running numbers n + j with (n + j) % 4 == g
      for (int j = (g - n) & (RL_GROUPS - 1); j <= m && ok; j += RL_GROUPS) {
        if (!(ok = __all_sync(0xffffffffu, mbar_wait(&bars->s_full[g], ((n + j) / RL_GROUPS) & 1)))) {
          dev_set_error(p.status, SAF_DEV_TIMEOUT_SOFTMAX, 92);
          break;
        }
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < 128; c += 64) {
          uint32_t x[2][32];
          tmem_ld32(ts + c, x[0]);
          tmem_ld32(ts + c + 32, x[1]);
          tmem_ld_wait();
          if (c == 64) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->s_empty[g]);
          }
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            float v[32];
#pragma unroll
            for (int e = 0; e < 32; ++e) v[e] = __uint_as_float(x[q][e]);
            if (p.negative) {
#pragma unroll
              for (int e = 0; e < 32; ++e) v[e] = -v[e];
            }
            float scale = p.scale;
            if (j == m) {                        // the diagonal tile (keys past the end lie beyond every row)
#pragma unroll
              for (int e = 0; e < 32; ++e) v[e] = c + q * 32 + e > row ? -INFINITY : v[e] * scale;
              scale = 1.f;
            }
            float t[4] = {v[0], v[1], v[2], v[3]};
#pragma unroll
            for (int e = 4; e < 32; ++e) t[e & 3] = rl_max(t[e & 3], v[e]);
            const float mn = rl_max(mx, rl_max(rl_max(t[0], t[1]), rl_max(t[2], t[3])) * scale);
            l *= rl_ex2(mx - mn);
            mx = mn;
            float2 u[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
            for (int e = 0; e < 32; e += 2) {
              const float2 y = __ffma2_rn(make_float2(v[e], v[e + 1]), make_float2(scale, scale), make_float2(-mn, -mn));
              const float2 w = (e & 6) == 0 ? rl_poly2(y) : make_float2(rl_ex2(y.x), rl_ex2(y.y));
              u[(e >> 1) & 1] = __fadd2_rn(u[(e >> 1) & 1], w);
            }
            const float2 w = __fadd2_rn(u[0], u[1]);
            l += w.x + w.y;
          }
        }
      }
      // the four groups' pairs of a row: one barrier per row tile, the buffers alternate
      float2* at = parts + (k & 1) * RL_GROUPS * 128;
      at[g * 128 + row] = make_float2(mx, l);
      named_bar_sync(1, RL_GROUPS * 128);
      if (g == (k & (RL_GROUPS - 1)) && ok) {
        const int t = m * 128 + row;
        float2 q[RL_GROUPS];
        float top = RL_LOW, sum = 0.f;
#pragma unroll
        for (int i = 0; i < RL_GROUPS; ++i) {
          q[i] = at[i * 128 + row];
          top = fmaxf(top, q[i].x);
        }
#pragma unroll
        for (int i = 0; i < RL_GROUPS; ++i) sum += q[i].y * rl_ex2(q[i].x - top);
        if (t < p.T) {
          const int b = bh / p.U, h = bh - b * p.U;
          p.lse[(int64_t)b * p.s[0] + (int64_t)h * p.s[1] + (int64_t)t * p.s[2]] = top + log2f(sum);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

template <int HD>
int launch_typed(const SafAttnStatsArgs& a, cudaStream_t st) {
  CUtensorMap mq, mk;
  int rc;
  if ((rc = make_row_tile_map_bf16(&mq, a.q, a.B, a.U, a.T, HD)) || (rc = make_row_tile_map_bf16(&mk, a.k, a.B, a.U, a.T, HD))) return rc;
  RlParams p;
  p.B = a.B; p.U = a.U; p.T = a.T;
  p.n_tiles = (a.T + 127) / 128;
  const int64_t total = (int64_t)a.B * a.U * p.n_tiles;
  if (total > (1 << 30)) return fail(SAF_ERR_LIMIT, "row log-sum-exp: too many row tiles");
  p.total = (int)total;
  p.scale = fabsf(a.sm_scale) * RL_LOG2E;
  p.negative = a.sm_scale < 0.f;
  p.lse = reinterpret_cast<float*>(a.lse.ptr);
  for (int i = 0; i < 3; ++i) p.s[i] = a.lse.stride[i];
  p.status = a.status;
  static PerDeviceOnce once;
  if ((rc = ensure_dyn_smem(row_lse_kernel<HD>, RlCfg<HD>::SMEM, once))) return rc;
  row_lse_kernel<HD><<<std::min(device_sm_count(), p.total), RL_THREADS, RlCfg<HD>::SMEM, st>>>(mq, mk, p);
  count_launch();
  return check_launch("row_lse_kernel");
}

}  // namespace

int launch_row_lse_sm100(const SafAttnStatsArgs& a, cudaStream_t st) {
  return a.HD == 64 ? launch_typed<64>(a, st) : launch_typed<128>(a, st);
}

}  // namespace saf
