// fp32 indexed linear on the tensor cores: every operand element is split into three bf16 parts, x = x0 + x1 + x2
// (split_bf16.cuh), and the product is the sum of the six part products that reach 2^-24 of it.
//
// Precision: the tensor core adds into its fp32 accumulator by truncation, and an error of one sign grows with the length
// of the chain.  So the leading product x0 y0 only runs over 32 of K (two instructions) before the epilogue warps take
// it out and add it in fp32 with rounding, while the next 32 go to the other of two accumulators; the
// five small products (2^-8 and less of the leading one) stay in accumulators of their own for the whole K range, where
// truncation costs 2^-8 of what it would cost beside the leading product.
//
// What bounds it: a slice of a 128 x 128 tile takes 2800 cycles, of which its 16 instructions (128 x 128 x 16 and
// 128 x 256 x 16) need 1536 and the conversion of the next slice most of the rest (without the small products 2400);
// 96 KB of parts are written to shared memory and 256 KB read.  2048 x 768 x 768 on a B200, before (fp32 FMAs, 64 x 64
// tiles) and now: forward 79 -> 24 us, dx 80 -> 23, dW 64 -> 22; 16384 x 2048 x 2048: 3380 -> 800 us = 172 TFLOP/s.
// Relative error against 64 bits, normal inputs: 2.5e-7 -> 1.1e-7 at K = 768, 1.15e-6 -> 4.3e-7 at K = 16384.
// An operand keeps the layout it has in memory: rows of 64 consecutive elements become 128-byte swizzled rows whether they
// run along K (K-major) or along the tile's rows or columns (MN-major), so nothing is transposed.
//   warps 0-15  read fp32 from global memory one slice ahead in registers, split, write the parts
//   warps 16-23 take the leading product out of TMEM; at the end add the small ones and hand the tile over
//   warp 24     issues (25-27 complete the warpgroup that hands registers to the others)
// Few tiles: the K range of a backward product is split over a cluster of 2 or 4 CTAs that add their sums through
// distributed shared memory, in the order of the parts (no atomics, no workspace).  The forward is never split: an output
// then has the same bits whatever other rows and features the call has.
//
// What the parts cannot carry shows in the results: they are not finite, or smaller than what may have been lost of them, which
// follows from the largest operands (split_bf16.cuh).  A tile with such a result, by its largest operands, is computed again with
// fp32 FMAs, and the results that are such by the largest elements of their own row and column are taken from there: what
// a result is depends on these alone.
#include <algorithm>
#include <type_traits>

#include "linear_tables.cuh"
#include "split_bf16.cuh"

namespace saf {
namespace {

constexpr int SI = 128, SK = 64;
constexpr int SPROD = 512, SEPI = 256, STHREADS = SPROD + SEPI + 128;
constexpr int ISSUER = (SPROD + SEPI) / 32;
constexpr int FBK = 32;                        // K slice of the FMA path

template <int BN>
struct SplitShape {
  static constexpr int NBJ = BN / 64, NB = 2 + NBJ;
  static constexpr int A_PART = 2 * SBLK, B_PART = NBJ * SBLK;
  static constexpr int STAGE = 3 * (A_PART + B_PART);
  static constexpr int STAGES = BN == 128 ? 2 : 3;
  static constexpr int LDR = BN + 4;           // row stride of the hand-over tile
  static constexpr int TCOLS = 4 * BN;         // two leading accumulators, two of the small products
  struct Ctrl {
    uint64_t full[STAGES], empty[STAGES], acc_full[2], acc_empty[2];
    uint32_t tmem_base;
    uint32_t top, top_j[BN];                   // largest operand of the tile; in the repeat, of a column (fp32 bits)
    const float* brow[BN];                     // forward: the weight rows of the tile's columns, null beyond the last
  };
  static constexpr int SMEM = 1024 + STAGES * STAGE + (int)sizeof(Ctrl);
};

struct SplitParams {
  const float *A, *X;
  float* out;
  int64_t lda, ldx, ldc;
  int M, C, N, slab, tiles_j, splits;
  int* status;
};

__device__ __forceinline__ float4 ld_cluster4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

// MODE 0: forward, 1: dx, 2: dW (see linear_generic.cu).  I rows, J columns, K depth of the product
template <int MODE, int BN>
__global__ void __launch_bounds__(STHREADS, 1) linear_f32_split_kernel(const __grid_constant__ SplitParams p,
                                                                       const __grid_constant__ WeightSet ws,
                                                                       const __grid_constant__ SlabTable tb) {
  using S = SplitShape<BN>;
  constexpr bool A_KC = MODE != 2, B_KC = MODE == 0;      // K is the operand's contiguous index
  extern __shared__ uint8_t split_smem[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)split_smem + 1023) & ~(uintptr_t)1023);
  typename S::Ctrl* sl = reinterpret_cast<typename S::Ctrl*>(smem + S::STAGES * S::STAGE);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int I = (MODE == 2) ? p.N : p.M;
  const int J = (MODE == 0) ? p.N : p.C;
  const int K = (MODE == 0) ? p.C : (MODE == 1 ? p.N : p.M);
  const int KT = (K + SK - 1) / SK;
  const int tile = blockIdx.x / p.splits, sp = blockIdx.x - tile * p.splits;
  const int ti = tile / p.tiles_j, i0 = ti * SI, j0 = (tile - ti * p.tiles_j) * BN;
  const int kt0 = (int)((int64_t)KT * sp / p.splits), kt1 = (int)((int64_t)KT * (sp + 1) / p.splits);

  if (tid == 0) {
    for (int s = 0; s < S::STAGES; ++s) {
      mbar_init(&sl->full[s], SPROD / 32);
      mbar_init(&sl->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sl->acc_full[b], 1);
      mbar_init(&sl->acc_empty[b], SEPI / 32);
    }
    fence_mbar_init();
  }
  if (tid == 0) sl->top = 0;
  if (tid < BN) sl->top_j[tid] = 0;
  if constexpr (B_KC) {
    if (tid < BN) sl->brow[tid] = j0 + tid < J ? welem<float>(ws, tb, j0 + tid, p.slab, 0) : nullptr;
  }
  pdl_wait();
  pdl_trigger();
  if (warp == ISSUER) {
    tmem_alloc(&sl->tmem_base, S::TCOLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sl->tmem_base;

  if (warp < SPROD / 32) {
    // (512 x 64 + 256 x 104 + 128 x 40 registers = 896 x 72; the narrow tile's epilogue holds half as many sums)
    if constexpr (BN == 128) asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    // 16 bytes of a row, 32 rows apart in every block of 64 x 64 elements
    const int row = tid >> 4, c4 = (tid & 15) * 4;
    const uint32_t off = row * 128 + ((((tid & 15) >> 1) ^ (row & 7)) << 4) + (tid & 1) * 8;
    const bool whole = i0 + SI <= I && j0 + BN <= J;
    // first element of this thread in the slice kt0, and the way to the next 32 rows / 64 columns / slice
    const float* pa = p.A + (A_KC ? (int64_t)(i0 + row) * p.lda + kt0 * SK + c4 : (int64_t)(kt0 * SK + row) * p.lda + i0 + c4);
    const float* pb = MODE == 2 ? p.X + (int64_t)(kt0 * SK + row) * p.ldx + j0 + c4 : nullptr;
    // MODE 1: the selection rows of K, as slab and row inside it, of the slice's two runs of 32 (slabs are whole runs)
    int g[2], r[2];
    if constexpr (MODE == 1) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        g[h] = (kt0 * SK + h * 32) / p.slab;
        r[h] = kt0 * SK + h * 32 - g[h] * p.slab;
      }
    }
    float4 v[S::NB][2];
    // half `op` of the slice kt: 0 the left operand's pieces, 1 the right one's
    auto load_as = [&](auto inside, int op, int kt) {
      constexpr bool all = decltype(inside)::value;       // no piece leaves the operands
      const int k0 = kt * SK;
      if (op == 0) {
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const float* src = pa + (A_KC ? (int64_t)(b * 64 + q * 32) * p.lda : (int64_t)(q * 32) * p.lda + b * 64);
            const int i = i0 + b * 64 + (A_KC ? q * 32 + row : c4), k = k0 + (A_KC ? c4 : q * 32 + row);
            v[b][q] = ld4_or_0(src, all || (i < I && k < K));
          }
        pa += A_KC ? (int64_t)SK : SK * p.lda;
        return;
      }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const float* src = pb;
        if constexpr (MODE == 1) {
          if (all || k0 + q * 32 < K) {
            const int w = tb.weight[g[q]];
            src = reinterpret_cast<const float*>(ws.w[w]) + (int64_t)(tb.row0[g[q]] + r[q] + row) * ws.ldw[w] + j0 + c4;
          }
          for (r[q] += SK; r[q] >= p.slab; r[q] -= p.slab) ++g[q];
        } else if constexpr (MODE == 2) {
          src += (int64_t)(q * 32) * p.ldx;
        }
#pragma unroll
        for (int b = 0; b < S::NBJ; ++b) {
          if constexpr (B_KC) {
            const float* wr = sl->brow[b * 64 + q * 32 + row];
            v[2 + b][q] = ld4_or_0(wr + k0 + c4, all || (wr != nullptr && k0 + c4 < K));
          } else {
            v[2 + b][q] = ld4_or_0(src + b * 64, all || (k0 + q * 32 + row < K && j0 + b * 64 + c4 < J));
          }
        }
      }
      if constexpr (MODE == 2) pb += SK * p.ldx;
    };
    auto load = [&](int op, int kt) {
      if (whole && kt * SK + SK <= K) load_as(std::true_type{}, op, kt);
      else load_as(std::false_type{}, op, kt);
    };
    float top = 0.f;                           // largest operand
    if (kt0 < kt1) {
      load(0, kt0);
      load(1, kt0);
    }
    for (int kt = kt0; kt < kt1; ++kt) {
      const int it = kt - kt0, s = it % S::STAGES;
      if (!mbar_wait(&sl->empty[s], ((it / S::STAGES) & 1) ^ 1)) {
        dev_set_error(p.status, SAF_DEV_TIMEOUT_TMA, 70);
        break;
      }
      uint8_t* st = smem + s * S::STAGE + off;
      // an operand's pieces are loaded again as soon as they are converted; one operand at a time, so that the wait for
      // its pieces does not include newer loads
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        constexpr int PART[2] = {S::A_PART, S::B_PART};
#pragma unroll
        for (int b = 0; b < (o ? S::NBJ : 2); ++b)
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            split_store(st + o * 3 * S::A_PART + b * SBLK + q * 4096, PART[o], v[2 * o + b][q]);
            top = max_abs(top, v[2 * o + b][q]);
          }
        if (kt + 1 < kt1) load(o, kt + 1);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sl->full[s]);
    }
    const uint32_t m = __reduce_max_sync(0xffffffffu, __float_as_uint(top));
    if (lane == 0) atomicMax(&sl->top, m);
    named_bar_arrive(2, SPROD + SEPI);
  } else if (warp >= ISSUER) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (warp == ISSUER) {
    const bool leader = elect_one();
    const uint32_t id1 = umma_idesc_bf16(SI, BN, A_KC ? 0 : 1, B_KC ? 0 : 1);
    const uint32_t id2 = umma_idesc_bf16(SI, 2 * BN, A_KC ? 0 : 1, B_KC ? 0 : 1);
    const uint32_t sbase = smem_u32(smem), small = tmem + 2 * BN;
    for (int kt = kt0; kt < kt1; ++kt) {
      const int it = kt - kt0, s = it % S::STAGES;
      if (!mbar_wait(&sl->full[s], (it / S::STAGES) & 1)) {
        dev_set_error(p.status, SAF_DEV_TIMEOUT_MMA, 71);
        break;
      }
      tc_fence_after();
      uint64_t ad[3], bd[3];
#pragma unroll
      for (int u = 0; u < 3; ++u) {
        const uint32_t aa = sbase + s * S::STAGE + u * S::A_PART, bb = sbase + s * S::STAGE + 3 * S::A_PART + u * S::B_PART;
        ad[u] = A_KC ? umma_smem_desc_sw128(aa, 16, 1024) : umma_smem_desc_sw128(aa, SBLK, 1024);
        bd[u] = B_KC ? umma_smem_desc_sw128(bb, 16, 1024) : umma_smem_desc_sw128(bb, SBLK, 1024);
      }
      constexpr uint32_t SA = A_KC ? 32 : 2048, SB = B_KC ? 32 : 2048;    // 16 steps of K further on
      if (leader) {
#pragma unroll
        for (int k4 = 0; k4 < SK / 16; ++k4) {
          const uint32_t oa = k4 * SA, ob = k4 * SB;
          umma_ss(small, umma_desc_advance(ad[0], oa), umma_desc_advance(bd[1], ob), id2, it > 0 || k4 > 0);   // x0 [y1 y2]
          umma_ss(small, umma_desc_advance(ad[1], oa), umma_desc_advance(bd[0], ob), id2, 1);                 // x1 [y0 y1]
          umma_ss(small, umma_desc_advance(ad[2], oa), umma_desc_advance(bd[0], ob), id1, 1);                 // x2 y0
        }
      }
      __syncwarp();
      bool ok = true;
#pragma unroll
      for (int b = 0; b < 2 && ok; ++b) {        // the leading product: half a slice, two instructions, per accumulator
        if (!(ok = mbar_wait(&sl->acc_empty[b], (it & 1) ^ 1))) {
          dev_set_error(p.status, SAF_DEV_TIMEOUT_MMA, 72);
          break;
        }
        tc_fence_after();
        if (leader) {
#pragma unroll
          for (int k4 = 2 * b; k4 < 2 * b + 2; ++k4)
            umma_ss(tmem + b * BN, umma_desc_advance(ad[0], k4 * SA), umma_desc_advance(bd[0], k4 * SB), id1, k4 & 1);
          if (b == 1) umma_commit(&sl->empty[s]);
          umma_commit(&sl->acc_full[b]);
        }
        __syncwarp();
      }
      if (!ok) break;
    }
    }
  } else {
    if constexpr (BN == 128) asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    else asm volatile("setmaxnreg.inc.sync.aligned.u32 88;");
    constexpr int CW = BN / 2;                   // columns of a warp
    const int ew = warp - SPROD / 32, row = (warp & 3) * 32 + lane, col = (ew >> 2) * CW;
    const uint32_t tsrc = tmem + ((uint32_t)((warp & 3) * 32) << 16) + col;
    float acc[CW];
#pragma unroll
    for (int c = 0; c < CW; ++c) acc[c] = 0.f;
    auto add = [&](uint32_t from) {
#pragma unroll
      for (int c = 0; c < CW; c += 16) {
        uint32_t r[16];
        tmem_ld16(from + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          const float2 t = __fadd2_rn(make_float2(acc[c + j], acc[c + j + 1]), make_float2(__uint_as_float(r[j]), __uint_as_float(r[j + 1])));
          acc[c + j] = t.x;
          acc[c + j + 1] = t.y;
        }
      }
    };
    bool ok = true;
    for (int h = 0; h < 2 * (kt1 - kt0); ++h) {
      const int b = h & 1;
      if (!(ok = __all_sync(0xffffffffu, mbar_wait(&sl->acc_full[b], (h >> 1) & 1)))) {   // (whole warps read tensor memory)
        dev_set_error(p.status, SAF_DEV_TIMEOUT_EPI, 73);
        break;
      }
      tc_fence_after();
      add(tsrc + b * BN);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sl->acc_empty[b]);
    }
    if (ok && kt0 < kt1) {                       // the last slice's commit covers the small products as well
      add(tsrc + 2 * BN);
      add(tsrc + 3 * BN);
    }
    named_bar_sync(2, SPROD + SEPI);             // the largest operand is known
    const float top = __uint_as_float(sl->top), tiny = split_tiny(K, top);
    // (zero is a result like any other unless all the tile's products may have been lost)
    const bool zero = top > 0.f && top * top < 0x1p-90f;
    auto odd = [&](float v, float tiny) { return !(fabsf(v) < INFINITY) || (fabsf(v) < tiny && (zero || v != 0.f)); };
    // two operations a result; what they find is looked at again
    bool any = false;
    float big = 0.f;
#pragma unroll
    for (int c = 0; c < CW; ++c) {
      any |= !(fabsf(acc[c]) >= tiny);
      big = fmaxf(big, fabsf(acc[c]));
    }
    any = (any || big == INFINITY) && i0 + row < I;
    float* dst = reinterpret_cast<float*>(smem) + row * S::LDR + col;
    auto put = [&](int c) { *reinterpret_cast<float4*>(dst + c) = make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]); };
#pragma unroll
    for (int c = 0; c < CW; c += 4) put(c);
    if (any) {
      any = false;
#pragma unroll 4
      for (int c = 0; c < CW; ++c) any |= odd(dst[c], tiny);
    }
    if (named_bar_or(1, SEPI, any)) {
      // plain fp32 over the same K range: slices as [k][row] and [k][column] where the parts were, behind the tile
      float* as = reinterpret_cast<float*>(smem) + SI * S::LDR;
      float* bs = as + FBK * SI;
      float* sum = bs + FBK * BN + row * S::LDR + col;     // of the slices' own sums: short chains, as of the products above
      const int et = tid - SPROD, k1 = min(K, kt1 * SK);
      float top_i = 0.f;
#pragma unroll
      for (int c = 0; c < CW; c += 4) *reinterpret_cast<float4*>(sum + c) = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int k0 = kt0 * SK; k0 < k1; k0 += FBK) {
        for (int idx = et; idx < FBK * (SI + BN); idx += SEPI) {
          const bool isb = idx >= FBK * SI;
          const int x = isb ? idx - FBK * SI : idx, kk = x / (isb ? BN : SI), rr = x - kk * (isb ? BN : SI), k = k0 + kk;
          float val = 0.f;
          if (k < k1) {
            if (!isb) {
              if (i0 + rr < I) val = A_KC ? p.A[(int64_t)(i0 + rr) * p.lda + k] : p.A[(int64_t)k * p.lda + i0 + rr];
            } else if (j0 + rr < J) {
              if constexpr (MODE == 0) val = *welem<float>(ws, tb, j0 + rr, p.slab, k);
              else if constexpr (MODE == 1) val = *welem<float>(ws, tb, k, p.slab, j0 + rr);
              else val = p.X[(int64_t)k * p.ldx + j0 + rr];
            }
          }
          (isb ? bs : as)[x] = val;
          if (isb) atomicMax(&sl->top_j[rr], __float_as_uint(fabsf(val)));
        }
        named_bar_sync(1, SEPI);
        const int kn = min(FBK, k1 - k0);
#pragma unroll
        for (int c = 0; c < CW; ++c) acc[c] = 0.f;
        for (int kk = 0; kk < kn; ++kk) {
          const float av = as[kk * SI + row];
          top_i = fmaxf(top_i, fabsf(av));
#pragma unroll
          for (int c = 0; c < CW; c += 4) {
            const float4 bv = *reinterpret_cast<const float4*>(bs + kk * BN + col + c);
            acc[c] = fmaf(av, bv.x, acc[c]);
            acc[c + 1] = fmaf(av, bv.y, acc[c + 1]);
            acc[c + 2] = fmaf(av, bv.z, acc[c + 2]);
            acc[c + 3] = fmaf(av, bv.w, acc[c + 3]);
          }
        }
#pragma unroll
        for (int c = 0; c < CW; ++c) sum[c] += acc[c];
        named_bar_sync(1, SEPI);
      }
#pragma unroll 4
      for (int c = 0; c < CW; ++c) {
        const float top_j = __uint_as_float(sl->top_j[col + c]);
        if (odd(dst[c], split_tiny(K, fmaxf(top_i, top_j)))) dst[c] = sum[c];
      }
    }
  }

  // ---- the tile lies in shared memory; each CTA of the cluster adds the parts of its share of the rows and stores them
  tc_fence_before();
  __syncthreads();
  if (p.splits > 1) cluster_sync_all();
  if (tid < SPROD + SEPI) {
    const int r0 = SI * sp / p.splits, r1 = SI * (sp + 1) / p.splits;
    for (int idx = r0 * (BN / 4) + tid; idx < r1 * (BN / 4); idx += SPROD + SEPI) {
      const int r = idx / (BN / 4), c = (idx - r * (BN / 4)) * 4;
      const int ii = i0 + r, jj = j0 + c;
      if (ii >= I || jj >= J) continue;
      const float* at = reinterpret_cast<const float*>(smem) + r * S::LDR + c;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (p.splits == 1) {
        v = *reinterpret_cast<const float4*>(at);
      } else {
        for (int s = 0; s < p.splits; ++s) {
          const float4 t = ld_cluster4(cluster_addr_of(at, s));
          v.x += t.x; v.y += t.y; v.z += t.z; v.w += t.w;
        }
      }
      const float* bias = nullptr;
      if constexpr (MODE == 0) {
        const int g = jj / p.slab;
        const float* b = reinterpret_cast<const float*>(ws.b[tb.weight[g]]);
        if (b) bias = b + tb.row0[g] + (jj - g * p.slab);
      } else if constexpr (MODE == 1) {
        if (p.X) bias = p.X + jj;
      }
      if (bias) {
        v.x += bias[0]; v.y += bias[1]; v.z += bias[2]; v.w += bias[3];
      }
      float* o = MODE == 2 ? const_cast<float*>(welem<float>(ws, tb, ii, p.slab, jj)) : p.out + (int64_t)ii * p.ldc + jj;
      *reinterpret_cast<float4*>(o) = v;
    }
  }
  __syncwarp();
  if (p.splits > 1) cluster_sync_all();          // nobody leaves while its tile is read
  if (warp == ISSUER) tmem_dealloc(tmem, S::TCOLS);
}

struct SplitForm {
  int bn, splits;
};

// Tile width and parts of the K range by the time they should take: waves of (a fixed part + slices x time of a slice), in
// cycles as measured (2048 rows, 768 -> 768, forward: 24 us in tiles of 128 columns and 35 in 64; dW: 50 and 39 unsplit, 30
// and 24 in two parts, 37 and 43 in four).
SplitForm pick_split_form(int mode, int I, int J, int KT) {
  const int sms = device_sm_count();
  SplitForm best{128, 1};
  double cost = 1e30;
  for (int bn : {128, 64}) {
    const int64_t tiles = (int64_t)((I + SI - 1) / SI) * ((J + bn - 1) / bn);
    for (int s : {1, 2, 4}) {
      if (s > 1 && (mode == 0 || KT < 2 * s)) break;
      const int64_t room = s == 4 ? sms * 9 / 10 / 4 * 4 : sms / s * s;       // clusters of four leave SMs over
      const double waves = (double)((tiles * s + room - 1) / room);
      const double fixed = s == 1 ? 6000.0 : (s == 2 ? 12000.0 : 14600.0);
      const double t = waves * (fixed + ((KT + s - 1) / s) * (bn == 128 ? 2800.0 : 2100.0));
      if (t < cost) {
        cost = t;
        best = {bn, s};
      }
    }
  }
  return best;
}

template <int MODE, int BN>
int launch_split(const SplitParams& p, int64_t tiles, const WeightSet& ws, const SlabTable& tb, cudaStream_t st) {
  static PerDeviceOnce once;
  if (int rc = ensure_dyn_smem(linear_f32_split_kernel<MODE, BN>, SplitShape<BN>::SMEM, once)) return rc;
  return launch_pdl("linear_f32_split_kernel", linear_f32_split_kernel<MODE, BN>, dim3((unsigned)(tiles * p.splits)), STHREADS,
                    SplitShape<BN>::SMEM, st, p.splits, p, ws, tb);
}

}  // namespace

int launch_linear_f32(int mode, const void* A, int64_t lda, const void* X, int64_t ldx, void* Cout, int64_t ldc,
                      const SafIndexedLinearArgs& a, const WeightSet& ws, const SlabTable& tb, cudaStream_t st) {
  SplitParams p;
  p.A = reinterpret_cast<const float*>(A);
  p.X = reinterpret_cast<const float*>(X);
  p.out = reinterpret_cast<float*>(Cout);
  p.lda = lda; p.ldx = ldx; p.ldc = ldc;
  p.M = a.M; p.C = a.C; p.N = a.n_slabs * a.slab; p.slab = a.slab;
  p.status = a.status;
  const int I = mode == 2 ? p.N : p.M, J = mode == 0 ? p.N : p.C, K = mode == 0 ? p.C : (mode == 1 ? p.N : p.M);
  const SplitForm f = pick_split_form(mode, I, J, (K + SK - 1) / SK);
  p.splits = f.splits;
  p.tiles_j = (J + f.bn - 1) / f.bn;
  const int64_t tiles = (int64_t)((I + SI - 1) / SI) * p.tiles_j;
  if (f.bn == 128)
    return mode == 0 ? launch_split<0, 128>(p, tiles, ws, tb, st)
                     : (mode == 1 ? launch_split<1, 128>(p, tiles, ws, tb, st) : launch_split<2, 128>(p, tiles, ws, tb, st));
  return mode == 0 ? launch_split<0, 64>(p, tiles, ws, tb, st)
                   : (mode == 1 ? launch_split<1, 64>(p, tiles, ws, tb, st) : launch_split<2, 64>(p, tiles, ws, tb, st));
}

}  // namespace saf
