// Backward products of the indexed linear on tcgen05 (kernel/indexed_linear.py:47-55, 107-121):
//
//   DX:  dx[m, c]            = sum_n dout[m, n] * W_g[row0_g + r, c]        n = g*64 + r over the selected 64-row blocks
//   DW:  dW_g[row0_g + r, c] = sum_m dout[m, g*64 + r] * x[m, c]            rows of no block are never written
//
// Neither product needs a transposed or gathered copy: the tensor core reads an operand whose
// contraction index is the slow one ("MN-major") straight from the row-major tile TMA delivers.
//   DX: A = dout tile (K-major), B = 64 selected weight rows x 256 columns (MN-major), one TMA source per block
//   DW: A = dout^T (MN-major: 64 tokens x 128 features), B = x tile (MN-major: 64 tokens x 256 columns);
//       the finished 128 x 256 tile is stored through the weight-gradient maps, 64 rows at a time, at the
//       rows the two blocks own (the reference zero-fills and index_copy_'s a dense product instead).
// Same persistent, warp-specialised CTA as the forward GEMM: warp 0 TMA, warp 1 MMA issuer, warps 2-5
// epilogue; 128x256 tiles, K step 64, 4 stages, two TMEM accumulators.  All mbarrier waits are bounded.
//
// A training layer keeps fp32 master weights and an fp32 residual stream, so both products also exist with an fp32
// result (F32OUT: the accumulator leaves the kernel unrounded, 32 columns per 16 KB staging block), and DW can be
// split over the tokens: work unit (tile, split) writes its partial tile to an fp32 workspace and a finishing kernel
// adds the splits in a fixed order, writes the gradient of whole weight matrices in their own dtype and puts the
// exact zeros of rows no slab owns -- one pass instead of a zero fill, a bf16 product and a conversion.  A narrow layer
// needs the split: at 12 x 64 the products have 18 to 45 tiles for 148 SMs, and their K range is the token count.
// All weight gradients of one layer, 12 x 64, 8192 tokens: 260 us (three products on at most 36 CTAs, without fills
// and conversions) -> 44 + 9 us; 16 x 128, 16384 tokens: 510 -> 495 + 31 us, the zero fills and conversions (0.1 ms) gone.
#include <algorithm>
#include <type_traits>

#include "saf_internal.h"
#include "sm100_prims.cuh"

namespace saf {
namespace {

constexpr int BM = 128, BN = 256, BK = 64;
constexpr int NSTG = 4;
constexpr int ATOM = 64 * 64 * 2;               // 8 KB: 64 rows of 128 bytes
constexpr int BA_BYTES = 2 * ATOM;              // 16 KB
constexpr int BB_BYTES = 4 * ATOM;              // 32 KB
constexpr int BSTAGE = BA_BYTES + BB_BYTES;
constexpr int BOUT_BYTES = 2 * BM * 64 * 2;
constexpr int BMAX_SUB = 160;
constexpr int BGEMM_THREADS = 192;
enum { MODE_DX = 0, MODE_DW = 1 };

struct BlockTable {
  int32_t row0[BMAX_SUB];
  uint8_t weight[BMAX_SUB];
  // slabs that are a multiple of 32 but not of 64 rows (head_dim 96): a 64-row block is two runs of 32 weight
  // rows, each with its own source (first run in row0 / weight, second run here); the weight maps then carry
  // 32-row boxes
  int32_t row0b[BMAX_SUB];
  uint8_t weightb[BMAX_SUB];
};

struct BwdGemmParams {
  int I, J, KB;              // output rows, output columns, K steps of 64
  int tiles_m, tiles_n;
  int subs;                  // DW: 64-column blocks of a tile
  int n_blocks;              // selected 64-row blocks
  const void* bias;          // DX only: bf16 over the J output columns, or null
  int* status;
  int halves;                // see BlockTable
  int splits, split_rows;    // DW into a workspace: parts of the K range, workspace rows of one part
};

struct BSmem {
  uint64_t full[NSTG], empty[NSTG], acc_full[2], acc_empty[2];
  uint32_t tmem_base;
};

// F32OUT: DX writes fp32, DW writes its part of the product to the workspace (mapO: splits * split_rows rows).  SUBS: 64-column
// blocks of a tile, 2, 3 or 4, known to the compiler for DX, whose producer loops over them in every K step (as a parameter of the
// launch it cost 5 to 8 % at 256 columns: 16384 rows, 4608 -> 1536 188 us where it takes 179); 0: the launch's own, for DW (as a
// constant 4 it cost up to 4 % there: dx and dW of 8192 rows, 768 -> 768 76.0 us where they take 73.5)
template <int MODE, bool F32OUT, int SUBS>
__global__ void __launch_bounds__(BGEMM_THREADS, 1)
indexed_gemm_bwd_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                        const __grid_constant__ CUtensorMap mapW0, const __grid_constant__ CUtensorMap mapW1,
                        const __grid_constant__ CUtensorMap mapW2, const __grid_constant__ CUtensorMap mapW3,
                        const __grid_constant__ CUtensorMap mapO, const __grid_constant__ BwdGemmParams p,
                        const __grid_constant__ BlockTable tb) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* stage_base = smem;
  uint8_t* out_stage = smem + NSTG * BSTAGE;
  BSmem* sl = reinterpret_cast<BSmem*>(out_stage + BOUT_BYTES);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int splits = (MODE == MODE_DW && F32OUT) ? p.splits : 1;
  const int total_tiles = p.tiles_m * p.tiles_n * splits;    // work units: (tile, part of the K range)
  // unit -> row tile, column tile and its K steps; the parts of a tile are neighbours, the first ones a step longer
  auto unit = [&](int u, int& tm, int& tn, int& sp, int& kb0, int& kb1) {
    const int tile = u / splits;
    sp = u - tile * splits;
    tm = tile / p.tiles_n;
    tn = tile - tm * p.tiles_n;
    kb0 = (int)((int64_t)p.KB * sp / splits);
    kb1 = (int)((int64_t)p.KB * (sp + 1) / splits);
  };
  const CUtensorMap* wm[4] = {&mapW0, &mapW1, &mapW2, &mapW3};
  const int subs = SUBS ? SUBS : p.subs, bn = subs * 64;     // columns of a tile

  if (tid == 0) {
    for (int s = 0; s < NSTG; ++s) {
      mbar_init(&sl->full[s], 1);
      mbar_init(&sl->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sl->acc_full[b], 1);
      mbar_init(&sl->acc_empty[b], 4);
    }
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(&sl->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sl->tmem_base;

  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&mapA);
      pdl_wait();
      pdl_trigger();
      uint32_t it = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
        int tm, tn, sp, kb0, kb1;
        unit(tile, tm, tn, sp, kb0, kb1);
        const int nsub = min(subs, (p.J - tn * bn + 63) / 64);                      // 64-column blocks of B
        const int nrow = (MODE == MODE_DW) ? min(2, p.n_blocks - tm * 2) : 2;    // 64-feature blocks of A
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int s = it % NSTG;
          if (!mbar_wait(&sl->empty[s], ((it / NSTG) & 1) ^ 1)) {
            dev_set_error(p.status, SAF_DEV_TIMEOUT_TMA, 60);
            ok = false;
            break;
          }
          uint8_t* a = stage_base + s * BSTAGE;
          uint8_t* b = a + BA_BYTES;
          if (MODE == MODE_DX) {
            mbar_expect_tx(&sl->full[s], BA_BYTES + nsub * ATOM);
            tma_load_2d(a, &mapA, &sl->full[s], kb * BK, tm * BM);               // dout[m tile, block kb]
            for (int u = 0; u < nsub; ++u) {
              tma_load_2d(b + u * ATOM, wm[tb.weight[kb]], &sl->full[s], tn * bn + u * 64, tb.row0[kb]);
              if (p.halves)
                tma_load_2d(b + u * ATOM + ATOM / 2, wm[tb.weightb[kb]], &sl->full[s], tn * bn + u * 64, tb.row0b[kb]);
            }
          } else {
            mbar_expect_tx(&sl->full[s], (nrow + nsub) * ATOM);
            for (int u = 0; u < nrow; ++u)
              tma_load_2d(a + u * ATOM, &mapA, &sl->full[s], (tm * 2 + u) * 64, kb * BK);   // dout[token block, features]
            for (int u = 0; u < nsub; ++u)
              tma_load_2d(b + u * ATOM, &mapB, &sl->full[s], tn * bn + u * 64, kb * BK);    // x[token block, columns]
          }
        }
      }
    }
  } else if (warp == 1) {
    const bool leader = elect_one();
    const uint32_t idesc = umma_idesc_bf16(BM, bn, MODE == MODE_DW ? 1 : 0, 1);
    const uint32_t sbase = smem_u32(stage_base);
    uint32_t it = 0, lt = 0;
    bool ok = true;
    pdl_wait();                                 // the limits of the waits below do not run while an earlier kernel does
    for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x, ++lt) {
      const int buf = lt & 1;
      if (!mbar_wait(&sl->acc_empty[buf], ((lt >> 1) & 1) ^ 1)) {
        dev_set_error(p.status, SAF_DEV_TIMEOUT_MMA, 61);
        break;
      }
      tc_fence_after();
      const uint32_t d = tmem + buf * BN;
      int tm, tn, sp, kb0, kb1;
      unit(tile, tm, tn, sp, kb0, kb1);
      for (int kb = kb0; kb < kb1; ++kb, ++it) {
        const int s = it % NSTG;
        if (!mbar_wait(&sl->full[s], (it / NSTG) & 1)) {
          dev_set_error(p.status, SAF_DEV_TIMEOUT_MMA, 62);
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t a = sbase + s * BSTAGE;
        const uint32_t b = a + BA_BYTES;
        if (leader) {
#pragma unroll
          for (int k4 = 0; k4 < BK / 16; ++k4) {
            const uint64_t ad = (MODE == MODE_DW) ? umma_smem_desc_sw128(a + k4 * 2048, ATOM, 1024)
                                                  : umma_smem_desc_sw128(a + k4 * 32, 16, 1024);
            umma_ss(d, ad, umma_smem_desc_sw128(b + k4 * 2048, ATOM, 1024), idesc, kb > kb0 || k4 > 0);
          }
          umma_commit(&sl->empty[s]);
        }
        __syncwarp();
      }
      if (ok && leader) umma_commit(&sl->acc_full[buf]);
      __syncwarp();
    }
  } else {
    pdl_wait();
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const int etid = tid - 64;
    uint32_t lt = 0;
    uint32_t n_out = 0;                         // output blocks stored so far (staging block = parity)
    for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x, ++lt) {
      int tm, tn, sp, kb0, kb1;
      unit(tile, tm, tn, sp, kb0, kb1);
      const int nsub = min(subs, (p.J - tn * bn + 63) / 64);
      const int nrow = (MODE == MODE_DW) ? min(2, p.n_blocks - tm * 2) : 2;
      const int buf = lt & 1;
      // threads that meet at named barriers leave together: one whose wait ran out takes the others with it
      if (named_bar_or(1, 128, !mbar_wait(&sl->acc_full[buf], (lt >> 1) & 1))) {
        dev_set_error(p.status, SAF_DEV_TIMEOUT_EPI, 63);
        break;
      }
      tc_fence_after();
      const uint32_t tsrc = tmem + ((uint32_t)(quad * 32) << 16) + buf * BN;
      if constexpr (F32OUT) {
        const int orow = (MODE == MODE_DW) ? sp * p.split_rows + tm * BM : tm * BM;
        const int n32 = min(2 * nsub, (p.J - tn * bn + 31) / 32);
        for (int u = 0; u < n32; ++u) {             // 32 fp32 columns: 128-byte rows, 16 KB
          const int ob = (n_out++) & 1;
          if (etid == 0) tma_store_wait_read1();
          named_bar_sync(1, 128);
          uint32_t r0[32];
          tmem_ld32(tsrc + u * 32, r0);
          tmem_ld_wait();
          uint8_t* dst = out_stage + ob * (BOUT_BYTES / 2) + row * 128;
#pragma unroll
          for (int c = 0; c < 8; ++c)
            *reinterpret_cast<uint4*>(dst + ((c ^ (row & 7)) << 4)) = make_uint4(r0[c * 4], r0[c * 4 + 1], r0[c * 4 + 2], r0[c * 4 + 3]);
          fence_proxy_async_smem();
          named_bar_sync(1, 128);
          if (etid == 0) {
            tma_store_2d(&mapO, out_stage + ob * (BOUT_BYTES / 2), tn * bn + u * 32, orow);
            tma_store_commit();
          }
        }
      } else
      for (int u = 0; u < nsub; ++u) {
        // the two staging blocks take turns over all stores of the CTA (nsub may be odd)
        const int ob = (n_out++) & 1;
        if (etid == 0) tma_store_wait_read1();
        named_bar_sync(1, 128);
        uint32_t r0[32], r1[32];
        tmem_ld32(tsrc + u * 64, r0);
        tmem_ld32(tsrc + u * 64 + 32, r1);
        tmem_ld_wait();
        float v[64];
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          v[j] = __uint_as_float(r0[j]);
          v[32 + j] = __uint_as_float(r1[j]);
        }
        if (MODE == MODE_DX && p.bias) {
          const __nv_bfloat16* bp = reinterpret_cast<const __nv_bfloat16*>(p.bias) + tn * bn + u * 64;
#pragma unroll
          for (int j = 0; j < 64; ++j)
            if (tn * bn + u * 64 + j < p.J) v[j] += __bfloat162float(bp[j]);
        }
        uint8_t* dst = out_stage + ob * (BOUT_BYTES / 2) + row * 128;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          uint4 q;
          q.x = pack_bf16(v[c * 8 + 0], v[c * 8 + 1]);
          q.y = pack_bf16(v[c * 8 + 2], v[c * 8 + 3]);
          q.z = pack_bf16(v[c * 8 + 4], v[c * 8 + 5]);
          q.w = pack_bf16(v[c * 8 + 6], v[c * 8 + 7]);
          *reinterpret_cast<uint4*>(dst + ((c ^ (row & 7)) << 4)) = q;
        }
        fence_proxy_async_smem();
        named_bar_sync(1, 128);
        if (etid == 0) {
          const uint8_t* src = out_stage + ob * (BOUT_BYTES / 2);
          if (MODE == MODE_DX) {
            tma_store_2d(&mapO, src, tn * bn + u * 64, tm * BM);
          } else {
            for (int hb = 0; hb < nrow; ++hb) {
              const int sb = tm * 2 + hb;
              tma_store_2d(wm[tb.weight[sb]], src + hb * ATOM, tn * bn + u * 64, tb.row0[sb]);
              if (p.halves) tma_store_2d(wm[tb.weightb[sb]], src + hb * ATOM + ATOM / 2, tn * bn + u * 64, tb.row0b[sb]);
            }
          }
          tma_store_commit();
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sl->acc_empty[buf]);
    }
    if (etid == 0) tma_store_wait_all();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

bool al16(const void* q) { return ((uintptr_t)q & 15) == 0; }

int map2(CUtensorMap* m, const void* base, uint64_t cols, uint64_t rows, int64_t ld, uint32_t box_rows) {
  uint64_t dims[2] = {cols, rows};
  uint64_t strides[2] = {0, (uint64_t)ld * 2};
  uint32_t box[2] = {64, box_rows};
  return make_tensor_map_bf16(m, base, 2, dims, strides, box, true);
}

// fp32 output: 32 columns x 128 rows per store, row stride ld elements
int map2_f32(CUtensorMap* m, const void* base, uint64_t cols, uint64_t rows, int64_t ld) {
  uint64_t dims[2] = {cols, rows};
  uint64_t strides[2] = {0, (uint64_t)ld * 4};
  uint32_t box[2] = {32, 128};
  return make_tensor_map_f32(m, base, 2, dims, strides, box);
}

bool common_ok(const SafIndexedLinearArgs& a, const void* dout, int64_t lddo) {
  if (a.dtype != SAF_BF16 || a.slab % 32 || (a.n_slabs * a.slab) % 64 || a.n_slabs <= 0 || a.M <= 0) return false;
  if (a.n_slabs * a.slab / 64 > BMAX_SUB) return false;
  if (a.C % 8 || lddo % 8 || !al16(dout)) return false;
  for (int w = 0; w < a.n_weights; ++w) {
    if (!a.weights[w]) return false;
    if (a.ldw[w] % 8 || (a.cdw[w] != 0 && a.cdw[w] != 1) || !al16(a.weights[w])) return false;
  }
  return saf_device_supported() != 0;
}

bool is_halves(const SafIndexedLinearArgs& a) { return a.slab % 64 != 0; }

void fill_blocks(const SafIndexedLinearArgs& a, BlockTable* tb) {
  memset(tb, 0, sizeof(*tb));
  if (is_halves(a)) {
    for (int hb = 0; hb < a.n_slabs * a.slab / 32; ++hb) {       // 32-row runs, two per block
      const int g = (hb * 32) / a.slab, r = (hb * 32) % a.slab;
      if (hb & 1) {
        tb->row0b[hb >> 1] = a.slab_row0[g] + r;
        tb->weightb[hb >> 1] = (uint8_t)a.slab_weight[g];
      } else {
        tb->row0[hb >> 1] = a.slab_row0[g] + r;
        tb->weight[hb >> 1] = (uint8_t)a.slab_weight[g];
      }
    }
    return;
  }
  const int per = a.slab / 64;
  for (int g = 0; g < a.n_slabs; ++g)
    for (int u = 0; u < per; ++u) {
      tb->row0[g * per + u] = a.slab_row0[g] + u * 64;
      tb->weight[g * per + u] = (uint8_t)a.slab_weight[g];
    }
}

template <int MODE, bool F32OUT = false, int SUBS = 0>
int launch_mode(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap* mw, const CUtensorMap& mo,
                const BwdGemmParams& p, const BlockTable& tb, cudaStream_t st) {
  const int sm_count = device_sm_count();
  const size_t smem = 1024 + NSTG * BSTAGE + BOUT_BYTES + sizeof(BSmem);
  static PerDeviceOnce smem_once;
  if (int rc = ensure_dyn_smem(indexed_gemm_bwd_kernel<MODE, F32OUT, SUBS>, (int)smem, smem_once)) return rc;
  const int grid = std::min(sm_count, p.tiles_m * p.tiles_n * std::max(1, p.splits));
  return launch_pdl(MODE == MODE_DX ? "indexed_gemm_bwd_kernel<dx>" : "indexed_gemm_bwd_kernel<dw>", indexed_gemm_bwd_kernel<MODE, F32OUT, SUBS>,
                    dim3(grid), BGEMM_THREADS, smem, st, 1, ma, mb, mw[0], mw[1], mw[2], mw[3], mo, p, tb);
}

// Columns of a dx tile, in 64-column blocks, by the time the waves should take, in cycles: a K step is bound by its
// operands' way from L2 (16 KB of dout and 8 KB of weights per block).  A last wave that is nearly empty costs as much as a
// full one.  Measured with 256, 192 and 128 columns: 8192 rows, 1920 -> 768 29.0, 26.2 and 32.7 us (192 tiles, 256, 384 on 148
// SMs), 768 -> 768 14.1, 12.9, 15.7; 1024 rows, 1920 -> 768 15.6, 13.7, 12.5; 3001 rows, 3840 -> 1536 29.9, 47, 43.  (With the
// width a parameter of the launch; as a constant 8192 rows, 1920 -> 768 take 24.3 at 192 columns, 1024 rows 11.4 at 128.)
int dx_subs(int tiles_m, int C, int KB) {
  const int sms = device_sm_count();
  int best = 4;
  double cost = 1e30;
  for (int s = 4; s >= 2; --s) {
    const int64_t tiles = (int64_t)tiles_m * ((C + s * 64 - 1) / (s * 64));
    const double t = (double)((tiles + sms - 1) / sms) * (KB * (445.0 + 110.0 * s) + 1000.0 + 300.0 * s);
    if (t < cost) {
      cost = t;
      best = s;
    }
  }
  return best;
}

}  // namespace

int launch_gemm_bwd_dx_sm100(const SafIndexedLinearArgs& a, const void* dout, int64_t lddo, void* dx, int64_t lddx,
                             const void* bias, bool f32_out, cudaStream_t st) {
  if (!common_ok(a, dout, lddo)) return SAF_ERR_UNSUPPORTED;
  if (lddx % (f32_out ? 4 : 8) || !al16(dx) || (f32_out && bias)) return SAF_ERR_UNSUPPORTED;
  const int N = a.n_slabs * a.slab;
  CUtensorMap ma, mw[4], mo;
  int rc;
  if ((rc = map2(&ma, dout, (uint64_t)N, (uint64_t)a.M, lddo, 128))) return rc;
  for (int w = 0; w < 4; ++w) {
    const int ww = w < a.n_weights ? w : 0;
    if ((rc = map2(&mw[w], a.weights[ww], (uint64_t)a.C, (uint64_t)a.rows_w[ww], a.ldw[ww], is_halves(a) ? 32 : 64))) return rc;
  }
  if (f32_out) rc = map2_f32(&mo, dx, (uint64_t)a.C, (uint64_t)a.M, lddx);
  else rc = map2(&mo, dx, (uint64_t)a.C, (uint64_t)a.M, lddx, 128);
  if (rc) return rc;
  BlockTable tb;
  fill_blocks(a, &tb);
  BwdGemmParams p;
  memset(&p, 0, sizeof(p));
  p.halves = is_halves(a) ? 1 : 0;
  p.I = a.M; p.J = a.C; p.KB = N / 64; p.n_blocks = N / 64;
  p.tiles_m = (a.M + BM - 1) / BM;
  const int subs = dx_subs(p.tiles_m, a.C, p.KB);
  p.tiles_n = (a.C + subs * 64 - 1) / (subs * 64);
  p.bias = bias;
  p.status = a.status;
  auto launch = [&](auto f32) {
    constexpr bool F = decltype(f32)::value;
    return subs == 4 ? launch_mode<MODE_DX, F, 4>(ma, ma, mw, mo, p, tb, st)
                     : (subs == 3 ? launch_mode<MODE_DX, F, 3>(ma, ma, mw, mo, p, tb, st) : launch_mode<MODE_DX, F, 2>(ma, ma, mw, mo, p, tb, st));
  };
  return f32_out ? launch(std::true_type{}) : launch(std::false_type{});
}

int launch_gemm_bwd_dw_sm100(const SafIndexedLinearArgs& a, const void* dout, int64_t lddo, cudaStream_t st) {
  if (!common_ok(a, dout, lddo)) return SAF_ERR_UNSUPPORTED;
  if (a.ldx % 8 || !al16(a.x)) return SAF_ERR_UNSUPPORTED;
  for (int w = 0; w < a.n_weights; ++w)
    if (a.biases[w]) return SAF_ERR_UNSUPPORTED;   // bias gradients stay with the generic kernels
  const int N = a.n_slabs * a.slab;
  CUtensorMap ma, mb, mw[4];
  int rc;
  if ((rc = map2(&ma, dout, (uint64_t)N, (uint64_t)a.M, lddo, 64))) return rc;
  if ((rc = map2(&mb, a.x, (uint64_t)a.C, (uint64_t)a.M, a.ldx, 64))) return rc;
  for (int w = 0; w < 4; ++w) {
    const int ww = w < a.n_weights ? w : 0;
    if ((rc = map2(&mw[w], a.weights[ww], (uint64_t)a.C, (uint64_t)a.rows_w[ww], a.ldw[ww], is_halves(a) ? 32 : 64))) return rc;
  }
  BlockTable tb;
  fill_blocks(a, &tb);
  BwdGemmParams p;
  memset(&p, 0, sizeof(p));
  p.halves = is_halves(a) ? 1 : 0;
  p.I = N; p.J = a.C; p.KB = (a.M + BK - 1) / BK; p.n_blocks = N / 64;
  p.tiles_m = (p.n_blocks + 1) / 2;
  p.subs = BN / 64;
  p.tiles_n = (a.C + BN - 1) / BN;
  p.status = a.status;
  return launch_mode<MODE_DW>(ma, mb, mw, ma, p, tb, st);
}

// ---- DW through a workspace: splits over the tokens, whole gradient matrices out ----------------------------------
namespace {

constexpr int FIN_RUNS = 1024;                  // 32-row runs of the gradient matrices of one call
constexpr int FIN_THREADS = 256;
struct FinishTable {
  int16_t src[FIN_RUNS];                        // position of the run in the stacked product (in runs), -1: zeros
};
struct FinishParams {
  const float* ws;
  void* out[SAF_MAX_WEIGHTS];
  int run0[SAF_MAX_WEIGHTS + 1];                // first run of each matrix
  int n, C4, splits;                            // matrices; 16-byte columns; parts
  int64_t part;                                 // floats of one part (split_rows * C)
  int f32;
};

// gradient[row] = sum over the parts of the workspace row its run came from, or zero.  Memory-bound: one float4
// column per thread and row, consecutive threads along the row.
__global__ void __launch_bounds__(FIN_THREADS) dw_finish_kernel(const __grid_constant__ FinishParams p,
                                                                const __grid_constant__ FinishTable tb) {
  pdl_wait();
  pdl_trigger();
  const int run = blockIdx.y;
  int w = 0;
  while (w + 1 < p.n && run >= p.run0[w + 1]) ++w;
  const int src = tb.src[run];
  const int64_t row0 = (int64_t)(run - p.run0[w]) * 32;
  for (int idx = blockIdx.x * FIN_THREADS + threadIdx.x; idx < 32 * p.C4; idx += gridDim.x * FIN_THREADS) {
    const int r = idx / p.C4, c = idx - r * p.C4;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    if (src >= 0) {
      const float4* q = reinterpret_cast<const float4*>(p.ws) + ((int64_t)src * 32 + r) * p.C4 + c;
      const int64_t step = p.part >> 2;
      s = *q;
      for (int k = 1; k < p.splits; ++k) {
        const float4 t = q[k * step];
        s.x += t.x; s.y += t.y; s.z += t.z; s.w += t.w;
      }
    }
    const int64_t o = (row0 + r) * p.C4 + c;
    if (p.f32) reinterpret_cast<float4*>(p.out[w])[o] = s;
    else reinterpret_cast<uint2*>(p.out[w])[o] = make_uint2(pack_bf16(s.x, s.y), pack_bf16(s.z, s.w));
  }
}

struct DwPlan {
  int splits, split_rows;
};

// Parts of the token range.  A row of tiles that does not fill the SMs, or leaves a nearly empty last wave, is split
// until (waves x K steps per unit), plus about 6 K steps of accumulator drain per unit and the workspace traffic of the
// extra part (written and read once, in K steps of 0.28 us over all SMs), is smallest.
DwPlan dw_plan(int n_blocks, int C, int M) {
  const int sms = device_sm_count();
  const int tiles_m = (n_blocks + 1) / 2, tiles = tiles_m * ((C + BN - 1) / BN), KB = (M + BK - 1) / BK;
  int best = 1;
  double best_cost = 1e30;
  for (int s = 1; s <= std::min(16, KB); ++s) {
    const int waves = (tiles * s + sms - 1) / sms;
    const double traffic = 2.0 * s * tiles_m * BM * (double)C * 4.0 / 5e12 / 0.28e-6;
    const double cost = waves * ((KB + s - 1) / s + 6.0) + traffic;
    if (cost < best_cost) {
      best_cost = cost;
      best = s;
    }
  }
  return {best, tiles_m * BM};
}

}  // namespace

int64_t gemm_dw_workspace_bytes(int n_rows, int C, int M) {
  const DwPlan d = dw_plan((n_rows + 63) / 64, C, M);
  return (int64_t)d.splits * d.split_rows * C * 4;
}

// a.weights: the gradient matrices, contiguous (rows_w, C) in fp32 (f32_out) or bf16, every row of them written
int launch_gemm_bwd_dw_full_sm100(const SafIndexedLinearArgs& a, const void* dout, int64_t lddo, float* ws,
                                  int64_t ws_bytes, bool f32_out, cudaStream_t st) {
  if (!common_ok(a, dout, lddo)) return SAF_ERR_UNSUPPORTED;
  if (a.ldx % 8 || !al16(a.x) || !al16(ws)) return SAF_ERR_UNSUPPORTED;
  const int N = a.n_slabs * a.slab;
  FinishTable ft;
  FinishParams fp;
  memset(&fp, 0, sizeof(fp));
  int runs = 0;
  for (int w = 0; w < a.n_weights; ++w) {
    if (a.rows_w[w] % 32 || a.ldw[w] != a.C) return SAF_ERR_UNSUPPORTED;
    fp.run0[w] = runs;
    runs += a.rows_w[w] / 32;
    fp.out[w] = const_cast<void*>(a.weights[w]);
  }
  if (runs > FIN_RUNS) return SAF_ERR_UNSUPPORTED;
  fp.run0[a.n_weights] = runs;
  for (int i = 0; i < runs; ++i) ft.src[i] = -1;
  const int per = a.slab / 32;
  for (int g = 0; g < a.n_slabs; ++g) {
    if (a.slab_row0[g] % 32) return SAF_ERR_UNSUPPORTED;
    for (int u = 0; u < per; ++u) ft.src[fp.run0[a.slab_weight[g]] + a.slab_row0[g] / 32 + u] = (int16_t)(g * per + u);
  }
  const DwPlan d = dw_plan(N / 64, a.C, a.M);
  if (ws_bytes < (int64_t)d.splits * d.split_rows * a.C * 4) return fail(SAF_ERR_INVALID, "dW workspace is too small");
  CUtensorMap ma, mb, mo;
  int rc;
  if ((rc = map2(&ma, dout, (uint64_t)N, (uint64_t)a.M, lddo, 64))) return rc;
  if ((rc = map2(&mb, a.x, (uint64_t)a.C, (uint64_t)a.M, a.ldx, 64))) return rc;
  if ((rc = map2_f32(&mo, ws, (uint64_t)a.C, (uint64_t)d.splits * d.split_rows, a.C))) return rc;
  BlockTable tb;
  memset(&tb, 0, sizeof(tb));
  BwdGemmParams p;
  memset(&p, 0, sizeof(p));
  p.I = N; p.J = a.C; p.KB = (a.M + BK - 1) / BK; p.n_blocks = N / 64;
  p.tiles_m = (p.n_blocks + 1) / 2;
  p.subs = BN / 64;
  p.tiles_n = (a.C + BN - 1) / BN;
  p.splits = d.splits;
  p.split_rows = d.split_rows;
  p.status = a.status;
  const CUtensorMap mw[4] = {ma, ma, ma, ma};
  if ((rc = launch_mode<MODE_DW, true>(ma, mb, mw, mo, p, tb, st))) return rc;
  fp.ws = ws;
  fp.n = a.n_weights;
  fp.C4 = a.C / 4;
  fp.splits = d.splits;
  fp.part = (int64_t)d.split_rows * a.C;
  fp.f32 = f32_out ? 1 : 0;
  const int per_run = (32 * fp.C4 + FIN_THREADS - 1) / FIN_THREADS;
  const dim3 grid((unsigned)std::min(per_run, std::max(1, 8 * device_sm_count() / runs)), (unsigned)runs);
  return launch_pdl("dw_finish_kernel", dw_finish_kernel, grid, FIN_THREADS, 0, st, 1, fp, ft);
}

}  // namespace saf
