// fp32 attention of the live heads at head_dim 64 on the tensor cores: forward, dK / dV and dQ.
//
// Every fp32 operand, probabilities and score gradients included, is split into three bf16 parts (split_bf16.cuh) and a
// product is the sum of the six part products that reach 2^-24 of it, as in the fp32 projections (linear_f32_sm100.cu).
// The leading part product of a 64-deep step is taken out of tensor memory after the step and added in fp32 with
// rounding; the five small ones have an accumulator of their own.  Exponentials, row maxima and row sums are fp32.
//
//   forward  CTA = 128 query rows, walks 64-key tiles:     S = Q K^T,                       O   += P V
//   dK / dV  CTA = 128 keys, walks 64-row query tiles:     S = K Q^T, dP = V dO^T,          dV  += P^T dO, dK += dS^T Q
//   dQ       CTA = 128 query rows, walks 64-key tiles:     S = Q K^T, dP = dO V^T,          dQ  += dS K
// All three have the same skeleton: one or two resident operands of 128 rows, two streamed ones of 64 rows a step.
//   warps 0-7   read fp32 rows one step ahead, split them into shared memory
//   warps 8-23  four threads per row, 16 columns each: scores out of TMEM, probabilities / score gradients back into the
//               columns the same thread has read, as A operands; they also keep the outputs in registers
//   warp 24     issues (25-27 complete the warpgroup that hands registers to the others)
//
// What bounds it: the 24 to 48 part products of a step, 128 x 64 x 16 at 48 cycles from shared memory and 32 from tensor
// memory (two thirds of the time of the longest walks), and the row tiles' unequal walks.  9 heads, T = 1024, B = 2 on a B200,
// before (fp32 FMAs, 64 x 64 tiles) and now: forward 119 -> 33 us, backward 397 -> 78; relative error against 64 bits 3.3e-7 ->
// 1.6e-7 (y), 4.5e-7 -> 3.0e-7 (dq), 7.9e-7 -> 3.2e-7 (dk), 8.0e-7 -> 2.6e-7 (dv).  Two threads per row instead of four:
// 41 and 196 us; each step's products one after the other: 164.
// Since the issuing warp's descriptors no longer spill (below), whole launches in a row, fills and delta included: forward 34.5 ->
// 33.3 us, backward 91 -> 81; T = 4096, B = 1, 12 heads 182 -> 175 and 700 -> 585.  What is still spilled (-Xptxas -v, bytes of stores and
// loads a thread) is most of it in the repeat of what the split cannot carry: 40 / 40 forward, 268 / 300 backward, none and 84 / 124
// without it.
//
// The same split as the reference (kernel/fused_attn.py:228-289, 415-481, 483-540): no atomics, fixed order of sums.
// What the parts cannot carry shows in the results: they are not finite, or smaller than what may have been lost of them, which
// follows from the tile's largest operand (split_bf16.cuh).  A tile with such results is computed again with fp32 FMAs, and the threads
// that hold one take their 16 columns from there.
#include <string.h>

#include "head_index.cuh"
#include "saf_internal.h"
#include "scan_body.cuh"
#include "split_bf16.cuh"


namespace saf {
namespace {

constexpr int AR = 128, AX = 64, AHD = 64;      // resident rows, streamed rows, head width
constexpr int APROD = 256, ACOMP = 512, ATHREADS = APROD + ACOMP + 128;
constexpr int AISSUER = (APROD + ACOMP) / 32;
constexpr int RES_PART = 2 * SBLK, RES = 3 * RES_PART;        // a resident operand: 48 KB
constexpr int STR = 3 * SBLK, ASTAGE = 2 * STR;               // a streamed one, a stage of two
constexpr float F_LOG2E = 1.4426950408889634f;
enum { A_FWD = 0, A_DKDV = 1, A_DQ = 2 };

template <int MODE>
struct AttnShape {
  static constexpr int NRES = MODE == A_FWD ? 1 : 2, STAGES = MODE == A_FWD ? 3 : 2;
  struct Ctrl {
    uint64_t full[STAGES], empty[STAGES], res_full, s_full[2], dp_full, p_full[2], ds_full, acc_full[2];
    uint32_t tmem_base, top;                    // largest operand (fp32 bits)
    alignas(16) float lse[STAGES][AX], delta[STAGES][AX];   // dK / dV: of the streamed query rows
    float mx[2][4][AR];                         // forward: row maxima, row sums of the four quarters
  };
  static constexpr int SMEM = 1024 + NRES * RES + STAGES * ASTAGE + (int)sizeof(Ctrl);
};
// TMEM columns: every accumulator is 64 columns of the leading product and 64 of the small ones.  The forward alternates its
// scores between T_S and T_DP and its output between T_ACC1 and T_ACC2, dQ its scores between T_S and T_ACC2
constexpr uint32_t T_S = 0, T_DP = 128, T_ACC1 = 256, T_ACC2 = 384;

__device__ __forceinline__ const float* f32_head(const SafTensor& t, int b, int h) {
  return reinterpret_cast<const float*>(t.ptr) + (int64_t)b * t.stride[0] + (int64_t)h * t.stride[1];
}

// The six part products of one 16-deep step, k4; A in shared memory or, as it was put back, in tensor memory.  The parts of
// an operand lie RES_PART / SBLK bytes apart: one descriptor, advanced by constants.
__device__ __forceinline__ void six_ss(uint32_t d, uint64_t a, uint64_t b, int k4, uint32_t idesc) {
  const uint32_t o = k4 * 32;
  auto pa = [&](int u) { return umma_desc_advance(a, u * RES_PART + o); };
  auto pb = [&](int u) { return umma_desc_advance(b, u * SBLK + o); };
  umma_ss(d, pa(0), pb(0), idesc, k4 > 0);
  umma_ss(d + 64, pa(0), pb(1), idesc, k4 > 0);
  umma_ss(d + 64, pa(1), pb(0), idesc, 1);
  umma_ss(d + 64, pa(0), pb(2), idesc, 1);
  umma_ss(d + 64, pa(1), pb(1), idesc, 1);
  umma_ss(d + 64, pa(2), pb(0), idesc, 1);
}
// `at`: the 64 leading columns of the region that held the scores; step k4's parts lie where its thread read them
__device__ __forceinline__ void six_ts(uint32_t d, uint32_t at, uint64_t b, int k4, uint32_t idesc, bool first_small) {
  const uint32_t a0 = at + 16 * k4, a1 = a0 + 8, a2 = a0 + 64, o = k4 * 2048;
  auto pb = [&](int u) { return umma_desc_advance(b, u * SBLK + o); };
  umma_ts(d, a0, pb(0), idesc, k4 > 0);
  umma_ts(d + 64, a0, pb(1), idesc, !first_small);
  umma_ts(d + 64, a1, pb(0), idesc, 1);
  umma_ts(d + 64, a0, pb(2), idesc, 1);
  umma_ts(d + 64, a1, pb(1), idesc, 1);
  umma_ts(d + 64, a2, pb(0), idesc, 1);
}

// 16 columns of an accumulator pair, added
__device__ __forceinline__ void tmem_sum16(uint32_t at, float (&v)[16]) {
  uint32_t x[16], y[16];
  tmem_ld16(at, x);
  tmem_ld16(at + 64, y);
  tmem_ld_wait();
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(x[j]) + __uint_as_float(y[j]);
}
// 16 values -> their parts, in the columns `at`.. the thread read them from
__device__ __forceinline__ void tmem_parts16(uint32_t at, const float (&v)[16]) {
  uint32_t w[3][8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    uint32_t q[3];
    split2(v[2 * j], v[2 * j + 1], q);
#pragma unroll
    for (int u = 0; u < 3; ++u) w[u][j] = q[u];
  }
  tmem_st8(at, w[0]);
  tmem_st8(at + 8, w[1]);
  tmem_st8(at + 64, w[2]);
}

__device__ __forceinline__ void store16(const SafTensor& t, int b, int h, int row, int col, const float (&v)[16], float f) {
  float* p = reinterpret_cast<float*>(t.ptr) + (int64_t)b * t.stride[0] + (int64_t)h * t.stride[1] + (int64_t)row * t.stride[2] + col;
#pragma unroll
  for (int c = 0; c < 16; c += 4) *reinterpret_cast<float4*>(p + c) = make_float4(v[c] * f, v[c + 1] * f, v[c + 2] * f, v[c + 3] * f);
}

// a thread's 16 columns of row t
template <int MODE>
__device__ __forceinline__ void store_results(const SafMixedAttnBwdArgs& g, const HeadIdx& hx, int t, int col, const float (&acc1)[16],
                                              const float (&acc2)[16], float m, float l) {
  const SafMixedAttnArgs& a = g.fwd;
  if constexpr (MODE == A_FWD) {
    const float ls = l == 0.f ? 1.f : l;
    store16(a.out, hx.b, hx.h, t, col, acc1, 1.f / ls);
    if (a.lse.ptr && col == 0)
      reinterpret_cast<float*>(a.lse.ptr)[(int64_t)hx.b * a.lse.stride[0] + (int64_t)hx.h * a.lse.stride[1] + (int64_t)t * a.lse.stride[2]] =
          ((m == -INFINITY) ? 0.f : m) + log2f(ls);
  } else if constexpr (MODE == A_DKDV) {
    store16(g.dv, hx.b, hx.hv, t, col, acc1, 1.f);
    store16(g.dk, hx.b, hx.hk, t, col, acc2, 1.f);
  } else {
    store16(g.dq, hx.b, hx.hq, t, col, acc1, 1.f);
  }
}

// The tile once more with fp32 FMAs, by all compute warps; threads with `odd` set store their results.  Resident and streamed rows, and
// the scores or what is made of them, lie in shared memory as fp32 where the parts were (68 floats a row: 8 neighbouring rows'
// float4 reads hit all banks once), a thread has 16 columns of a row as above.  A row adds up only what it sees, so that what later
// keys hold does not reach it, in sums of 64.  It comes when the tile's registers are free, behind the roles: as a function of its own
// it cost the others 4 to 8 %.  9 heads, T = 1024, B = 2, all of q NaN: forward 383 us, backward 782 (one NaN 54 and 782); the FMA
// kernels that served these calls before 126 and 411, one thread a row through global memory 6.3 and 38 ms.
template <int MODE>
__device__ __forceinline__ void attn_f32_repeat(const SafMixedAttnBwdArgs& g, float* sm, int r0, int x0, int x1, bool odd) {
  constexpr int LD = 68;
  static_assert((AR * LD * (MODE == A_FWD ? 2 : 3) + 2 * AX * LD + 4 * AR) * 4 <= AttnShape<MODE>::NRES * RES + AttnShape<MODE>::STAGES * ASTAGE,
                "fits where the parts were");
  const SafMixedAttnArgs& a = g.fwd;
  const HeadIdx hx = head_index(a, blockIdx.x);
  const int tid = threadIdx.x - APROD, T = a.T;
  const int part = tid >> 7, row = tid & 127, col = part * 16, t = r0 + row;
  float *R0 = sm, *R1 = R0 + AR * LD, *X0 = MODE == A_FWD ? R1 : R1 + AR * LD, *X1 = X0 + AX * LD, *W = X1 + AX * LD, *MX = W + AR * LD;
  auto rows = [&](float* dst, const SafTensor& from, int head, int first, int n) {
    const float* p = f32_head(from, hx.b, head);
    for (int i = tid; i < n * 16; i += ACOMP) {
      const int r = i >> 4, c = (i & 15) * 4;
      *reinterpret_cast<float4*>(dst + r * LD + c) = ld4_or_0(p + (int64_t)(first + r) * from.stride[2] + c, first + r < T);
    }
  };
  // this thread's 8 columns from j on of R X^T
  auto dot8 = [&](const float* R, const float* X, int j, float (&s)[8]) {
#pragma unroll
    for (int e = 0; e < 8; ++e) s[e] = 0.f;
#pragma unroll 1
    for (int d = 0; d < AHD; d += 4) {
      const float4 y = *reinterpret_cast<const float4*>(R + row * LD + d);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float4 x = *reinterpret_cast<const float4*>(X + (col + j + e) * LD + d);
        s[e] = fmaf(y.x, x.x, s[e]);
        s[e] = fmaf(y.y, x.y, s[e]);
        s[e] = fmaf(y.z, x.z, s[e]);
        s[e] = fmaf(y.w, x.w, s[e]);
      }
    }
  };
  // acc += W X over the streamed rows [from, to) of the step
  auto apply = [&](const float* X, int from, int to, float (&acc)[16]) {
    float s[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) s[c] = 0.f;
#pragma unroll 1
    for (int x = from; x < to; ++x) {
      const float w = W[row * LD + x];
#pragma unroll
      for (int c = 0; c < 16; c += 4) {
        const float4 v = *reinterpret_cast<const float4*>(X + x * LD + col + c);
        s[c] = fmaf(w, v.x, s[c]);
        s[c + 1] = fmaf(w, v.y, s[c + 1]);
        s[c + 2] = fmaf(w, v.z, s[c + 2]);
        s[c + 3] = fmaf(w, v.w, s[c + 3]);
      }
    }
#pragma unroll
    for (int c = 0; c < 16; ++c) acc[c] += s[c];
  };
  const bool kv = MODE == A_DKDV;
  rows(R0, kv ? a.k : a.q, kv ? hx.hk : hx.hq, r0, AR);
  if constexpr (MODE != A_FWD) rows(R1, kv ? a.v : g.dout, kv ? hx.hv : hx.h, r0, AR);
  const float scale = a.sm_scale * F_LOG2E;
  const float* lse = MODE == A_FWD ? nullptr : f32_head(a.lse, hx.b, hx.h);
  const float* del = MODE == A_FWD ? nullptr : f32_head(g.delta, hx.b, hx.h);
  float acc1[16], acc2[16], m = -INFINITY, l = 0.f, s[8];
#pragma unroll
  for (int c = 0; c < 16; ++c) acc1[c] = acc2[c] = 0.f;
  for (int xi = x0; xi < x1; ++xi) {
    const int xb = xi * AX;
    named_bar_sync(1, ACOMP);                               // the step before is read
    rows(X0, kv ? a.q : a.k, kv ? hx.hq : hx.hk, xb, AX);
    rows(X1, kv ? g.dout : a.v, kv ? hx.h : hx.hv, xb, AX);
    named_bar_sync(1, ACOMP);
    // the rows of the step that this one sees
    const int from = kv ? min(AX, max(0, t - xb)) : 0, to = t >= T ? from : (kv ? min(AX, T - xb) : max(0, min(AX, t - xb + 1)));
    float* w = W + row * LD + col;
    float mx = -INFINITY;
#pragma unroll 1
    for (int j = 0; j < 16; j += 8) {
      dot8(R0, X0, j, s);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int x = col + j + e;
        const bool seen = x >= from && x < to;
        if constexpr (MODE == A_FWD) {
          w[j + e] = seen ? s[e] * scale : -INFINITY;
          mx = fmaxf(mx, w[j + e]);
        } else {
          w[j + e] = seen ? exp2f(s[e] * scale - lse[(int64_t)(kv ? xb + x : t) * a.lse.stride[2]]) : 0.f;
        }
      }
    }
    if constexpr (MODE == A_FWD) {
      MX[part * AR + row] = mx;
      named_bar_sync(1, ACOMP);
      mx = fmaxf(fmaxf(MX[row], MX[AR + row]), fmaxf(MX[2 * AR + row], MX[3 * AR + row]));
      const float m_new = fmaxf(m, mx), m_safe = (m_new == -INFINITY) ? 0.f : m_new;
      const float f = (m == -INFINITY) ? 0.f : exp2f(m - m_safe);
      float sum = 0.f;
#pragma unroll 4
      for (int j = 0; j < 16; ++j) {
        w[j] = exp2f(w[j] - m_safe);
        sum += w[j];
      }
      l = l * f + sum;
      m = m_new;
      named_bar_sync(1, ACOMP);
#pragma unroll
      for (int c = 0; c < 16; ++c) acc1[c] *= f;
      apply(X1, from, to, acc1);
    } else {
      if constexpr (MODE == A_DKDV) {
        named_bar_sync(1, ACOMP);
        apply(X1, from, to, acc1);
        named_bar_sync(1, ACOMP);                           // P is read
      }
#pragma unroll 1
      for (int j = 0; j < 16; j += 8) {
        dot8(R1, X1, j, s);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int x = col + j + e;
          if (x >= from && x < to) w[j + e] = w[j + e] * (s[e] - del[(int64_t)(kv ? xb + x : t) * g.delta.stride[2]]) * a.sm_scale;
        }
      }
      named_bar_sync(1, ACOMP);
      if constexpr (MODE == A_DKDV) apply(X0, from, to, acc2);
      else apply(X0, from, to, acc1);
    }
  }
  if constexpr (MODE == A_FWD) {
    MX[part * AR + row] = l;
    named_bar_sync(1, ACOMP);
    l = (MX[row] + MX[AR + row]) + (MX[2 * AR + row] + MX[3 * AR + row]);
  }
  if (odd) store_results<MODE>(g, hx, t, col, acc1, acc2, m, l);
}

// the row tile with the `rank`-th longest walk of one (batch, head)
template <int MODE>
__device__ __forceinline__ void attn_f32_tile(const SafMixedAttnBwdArgs& g, int rank, int tiles) {
  using S = AttnShape<MODE>;
  const SafMixedAttnArgs& a = g.fwd;
  extern __shared__ uint8_t attn_smem[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)attn_smem + 1023) & ~(uintptr_t)1023);
  uint8_t* stages = smem + S::NRES * RES;
  typename S::Ctrl* sl = reinterpret_cast<typename S::Ctrl*>(stages + S::STAGES * ASTAGE);
  const HeadIdx hx = head_index(a, blockIdx.x);
  if (hx.state != SAF_LIVE) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, T = a.T;
  const int r0 = (MODE == A_DKDV ? rank : tiles - 1 - rank) * AR;     // first resident row
  // streamed tiles: keys up to the last row's, or queries from the first key's on
  const int x0 = MODE == A_DKDV ? r0 / AX : 0, xt = (T + AX - 1) / AX;
  const int x1 = MODE == A_DKDV ? xt : min(xt, (r0 + AR) / AX);

  if (tid == 0) {
    sl->top = 0;
    for (int s = 0; s < S::STAGES; ++s) {
      mbar_init(&sl->full[s], APROD / 32);
      mbar_init(&sl->empty[s], 1);
    }
    mbar_init(&sl->res_full, APROD / 32);
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sl->s_full[b], 1);
      mbar_init(&sl->p_full[b], ACOMP / 32);
      mbar_init(&sl->acc_full[b], 1);
    }
    mbar_init(&sl->dp_full, 1);
    mbar_init(&sl->ds_full, ACOMP / 32);
    fence_mbar_init();
  }
  if (warp == AISSUER) {
    tmem_alloc(&sl->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sl->tmem_base;
  bool again = false;                           // this thread's results have to be computed again

  if (warp < APROD / 32) {
    // backward: 256 x 64 + 512 x 80 + 128 x 56 registers = 896 x 72, the split with the fewest spills (with 40 the issuing warp
    // spilled its descriptors); the forward is fastest with 72 for all, said role by role: T = 4096, B = 1, 12 heads 173 us, 183 with
    // 80 for the compute warps, 186 without the instructions (the compiler spills more)
    if constexpr (MODE == A_FWD) asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    else asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    const int row = tid >> 4, c4 = (tid & 15) * 4;           // 16 bytes of a row, 16 rows apart
    const uint32_t off = row * 128 + ((((tid & 15) >> 1) ^ (row & 7)) << 4) + (tid & 1) * 8;
    float top = 0.f;
    // the resident operands, block by block
    {
      const SafTensor& t0 = MODE == A_DKDV ? a.k : a.q;
      const SafTensor& t1 = MODE == A_DKDV ? a.v : g.dout;
      const float* p0 = f32_head(t0, hx.b, MODE == A_DKDV ? hx.hk : hx.hq) + c4;
      const float* p1 = S::NRES == 2 ? f32_head(t1, hx.b, MODE == A_DKDV ? hx.hv : hx.h) + c4 : nullptr;
#pragma unroll 1
      for (int n = 0; n < 2 * S::NRES; ++n) {
        const int o = n >> 1, blk = n & 1;
        const float* src = o ? p1 : p0;
        const int64_t ld = (o ? t1 : t0).stride[2];
        float4 v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int t = r0 + blk * 64 + q * 16 + row;
          v[q] = ld4_or_0(src + (int64_t)t * ld, t < T);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          split_store(smem + o * RES + blk * SBLK + q * 2048 + off, RES_PART, v[q]);
          top = max_abs(top, v[q]);
        }
      }
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(&sl->res_full);
    const SafTensor& s0 = MODE == A_DKDV ? a.q : a.k;
    const SafTensor& s1 = MODE == A_DKDV ? g.dout : a.v;
    const float* p0 = f32_head(s0, hx.b, MODE == A_DKDV ? hx.hq : hx.hk) + c4;
    const float* p1 = f32_head(s1, hx.b, MODE == A_DKDV ? hx.h : hx.hv) + c4;
    const float* lse = MODE == A_DKDV ? f32_head(a.lse, hx.b, hx.h) : nullptr;
    const float* del = MODE == A_DKDV ? f32_head(g.delta, hx.b, hx.h) : nullptr;
    float4 v[2][4];
    float stat = 0.f;
    auto load = [&](int o, int xi) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int t = xi * AX + q * 16 + row;
        v[o][q] = ld4_or_0((o ? p1 : p0) + (int64_t)t * (o ? s1 : s0).stride[2], t < T);
      }
      if (MODE == A_DKDV && o == 1 && tid < 2 * AX) {
        const int t = xi * AX + (tid & (AX - 1));
        stat = t < T ? (tid < AX ? lse[(int64_t)t * a.lse.stride[2]] : del[(int64_t)t * g.delta.stride[2]]) : 0.f;
      }
    };
    if (x0 < x1) {
      load(0, x0);
      load(1, x0);
    }
    for (int xi = x0; xi < x1; ++xi) {
      const int it = xi - x0, s = it % S::STAGES;
      if (!mbar_wait(&sl->empty[s], ((it / S::STAGES) & 1) ^ 1)) {
        dev_set_error(a.status, SAF_DEV_TIMEOUT_TMA, 75);
        break;
      }
      uint8_t* st = stages + s * ASTAGE + off;
#pragma unroll
      for (int o = 0; o < 2; ++o) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          split_store(st + o * STR + q * 2048, SBLK, v[o][q]);
          top = max_abs(top, v[o][q]);
        }
        if (MODE == A_DKDV && o == 1 && tid < 2 * AX) (tid < AX ? sl->lse : sl->delta)[s][tid & (AX - 1)] = stat;
        if (xi + 1 < x1) load(o, xi + 1);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sl->full[s]);
    }
    const uint32_t m = __reduce_max_sync(0xffffffffu, __float_as_uint(top));
    if (lane == 0) atomicMax(&sl->top, m);
    named_bar_arrive(2, APROD + ACOMP);
  } else if (warp >= AISSUER) {
    if constexpr (MODE == A_FWD) asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    else asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == AISSUER) {
      const bool leader = elect_one();
      const uint32_t id_k = umma_idesc_bf16(AR, AX, 0, 0), id_mn = umma_idesc_bf16(AR, AHD, 0, 1);
      const uint32_t sb = smem_u32(smem), xb = smem_u32(stages);
      // products of the resident operand o with streamed tile `it`, into `d`
      auto scores = [&](int o, int it, uint32_t d, uint64_t* done) {
        const uint64_t ad = umma_smem_desc_sw128(sb + o * RES, 16, 1024);
        const uint64_t bd = umma_smem_desc_sw128(xb + (it % S::STAGES) * ASTAGE + o * STR, 16, 1024);
        if (leader) {
#pragma unroll
          for (int k4 = 0; k4 < 4; ++k4) six_ss(d, ad, bd, k4, id_k);
          umma_commit(done);
        }
        __syncwarp();
      };
      // products of the parts in region `at` with the rows of streamed operand o, into `d`; a step's leading product starts
      // again, the small ones go on unless `fresh`
      auto apply = [&](uint32_t at, int o, int it, uint32_t d, bool fresh) {
        const uint64_t bd = umma_smem_desc_sw128(xb + (it % S::STAGES) * ASTAGE + o * STR, SBLK, 1024);
        if (leader) {
#pragma unroll
          for (int k4 = 0; k4 < 4; ++k4) six_ts(d, at, bd, k4, id_mn, fresh && k4 == 0);
        }
      };
      auto commit = [&](uint64_t* bar) {
        if (leader) umma_commit(bar);
        __syncwarp();
      };
      auto wait = [&](uint64_t* bar, int phase, int site) {
        if (mbar_wait(bar, phase & 1)) {
          tc_fence_after();
          return true;
        }
        dev_set_error(a.status, SAF_DEV_TIMEOUT_MMA, site);
        return false;
      };
      auto stage_full = [&](int it) { return wait(&sl->full[it % S::STAGES], it / S::STAGES, 76); };
      const int n = x1 - x0;
      bool ok = wait(&sl->res_full, 0, 77);
      // Instructions of one thread run in order: a region is free for the next product once the last one that reads it has
      // been issued and its readers in the compute warps have arrived.
      // A wait by parity tells a phase from the next one only, so a barrier's arrivals for one step must not come before this
      // warp has seen those for the step before.  The forward's scores are two steps ahead of P: the compute warps can hand
      // over the next P while P of this step has yet to be seen here, and take turns on two barriers.
      if constexpr (MODE == A_FWD) {
        for (int it = 0; it < 2 && it < n && ok; ++it)
          if ((ok = stage_full(it))) scores(0, it, tmem + it * 128, &sl->s_full[it]);
        for (int it = 0; it < n && ok; ++it) {
          if (!(ok = wait(&sl->p_full[it & 1], it >> 1, 78))) break;
          apply(tmem + (it & 1) * 128, 1, it, tmem + T_ACC1 + (it & 1) * 128, true);
          commit(&sl->empty[it % S::STAGES]);
          commit(&sl->acc_full[it & 1]);
          if (it + 2 < n && (ok = stage_full(it + 2))) scores(0, it + 2, tmem + (it & 1) * 128, &sl->s_full[it & 1]);
        }
      } else if constexpr (MODE == A_DKDV) {
        // dV of a step and S of the next run while the compute warps make dS; dK and the next dP while they make P
        if (n > 0 && ok && (ok = stage_full(0))) {
          scores(0, 0, tmem + T_S, &sl->s_full[0]);
          scores(1, 0, tmem + T_DP, &sl->dp_full);
        }
        for (int it = 0; it < n && ok; ++it) {
          if (!(ok = wait(&sl->p_full[0], it, 78))) break;
          apply(tmem + T_S, 1, it, tmem + T_ACC1, it == 0);
          if (it + 1 < n) {
            if (!(ok = stage_full(it + 1))) break;
            scores(0, it + 1, tmem + T_S, &sl->s_full[0]);
          }
          if (!(ok = wait(&sl->ds_full, it, 74))) break;
          apply(tmem + T_DP, 0, it, tmem + T_ACC2, it == 0);
          commit(&sl->empty[it % S::STAGES]);
          if (it + 1 < n) scores(1, it + 1, tmem + T_DP, &sl->dp_full);
          else commit(&sl->acc_full[0]);
        }
      } else {
        // S of the next step, in the other of two regions, is ready before a step's dS; its dP runs while they make P
        constexpr uint32_t T_S2[2] = {T_S, T_ACC2};
        if (n > 0 && ok && (ok = stage_full(0))) {
          scores(0, 0, tmem + T_S, &sl->s_full[0]);
          scores(1, 0, tmem + T_DP, &sl->dp_full);
        }
        for (int it = 0; it < n && ok; ++it) {
          if (it + 1 < n) {
            if (!(ok = stage_full(it + 1))) break;
            scores(0, it + 1, tmem + T_S2[(it + 1) & 1], &sl->s_full[(it + 1) & 1]);
          }
          if (!(ok = wait(&sl->ds_full, it, 74))) break;
          apply(tmem + T_DP, 0, it, tmem + T_ACC1, it == 0);
          commit(&sl->empty[it % S::STAGES]);
          if (it + 1 < n) scores(1, it + 1, tmem + T_DP, &sl->dp_full);
          else commit(&sl->acc_full[0]);
        }
      }
    }
  } else {
    if constexpr (MODE == A_FWD) asm volatile("setmaxnreg.inc.sync.aligned.u32 72;");
    else asm volatile("setmaxnreg.inc.sync.aligned.u32 80;");
    const int quad = warp & 3, part = (warp - APROD / 32) >> 2, row = quad * 32 + lane, col = part * 16;
    const int t = r0 + row;                                   // this thread's query (dK / dV: key)
    const uint32_t lanes = tmem + ((uint32_t)(quad * 32) << 16) + col;
    const float scale = a.sm_scale * F_LOG2E;
    float acc1[16], acc2[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) acc1[c] = acc2[c] = 0.f;
    float m = -INFINITY, l = 0.f, L = 0.f, dl = 0.f;
    if (MODE == A_DQ && t < T) {
      L = f32_head(a.lse, hx.b, hx.h)[(int64_t)t * a.lse.stride[2]];
      dl = f32_head(g.delta, hx.b, hx.h)[(int64_t)t * g.delta.stride[2]];
    }
    const int n = x1 - x0;
    // the leading product of the step before (forward: and the small ones, which a new row maximum scales as well)
    auto drain = [&](uint32_t at, float (&acc)[16], bool small) {
      uint32_t x[16];
      tmem_ld16(lanes + at, x);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; ++j) acc[j] += __uint_as_float(x[j]);
      if (small) {
        tmem_ld16(lanes + at + 64, x);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[j] += __uint_as_float(x[j]);
      }
    };
    auto hand_over = [&](uint64_t* bar) {
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    auto wait = [&](uint64_t* bar, int phase, int site) {
      // (a lane's limit is its own, and tensor memory is read by whole warps: they leave together)
      const bool in_time = __all_sync(0xffffffffu, mbar_wait(bar, phase & 1));
      if (!in_time) dev_set_error(a.status, SAF_DEV_TIMEOUT_SOFTMAX, site);
      tc_fence_after();
      return in_time;
    };
    bool ok = true;
    for (int it = 0; it < n; ++it) {
      const int xb = (x0 + it) * AX + col;                    // this thread's first streamed row
      const uint32_t sat = lanes + (MODE == A_FWD ? (it & 1) * 128 : (MODE == A_DQ && (it & 1) ? T_ACC2 : T_S));
      ok = ok && (MODE == A_DKDV ? wait(&sl->s_full[0], it, 79) : wait(&sl->s_full[it & 1], it >> 1, 79));
      if (MODE != A_FWD && !ok) break;                        // (the forward leaves at the vote, where the row's threads meet)
      const bool edge = MODE == A_DKDV ? xb < r0 + AR || xb + 16 > T : xb + 15 > r0;       // some scores may be masked
      float s[16];
      tmem_sum16(sat, s);
      if constexpr (MODE == A_FWD) {
        float mx = -INFINITY;
#pragma unroll
        for (int j = 0; j < 16; ++j) s[j] *= scale;
        if (edge) {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (xb + j > t || xb + j >= T) s[j] = -INFINITY;
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) mx = fmaxf(mx, s[j]);
        sl->mx[it & 1][part][row] = mx;
        if (named_bar_or(1, ACOMP, !ok)) {
          ok = false;
          break;
        }
        mx = fmaxf(fmaxf(sl->mx[it & 1][0][row], sl->mx[it & 1][1][row]), fmaxf(sl->mx[it & 1][2][row], sl->mx[it & 1][3][row]));
        const float m_new = fmaxf(m, mx), m_safe = (m_new == -INFINITY) ? 0.f : m_new;
        const float f = (m == -INFINITY) ? 0.f : exp2f(m - m_safe);
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          s[j] = exp2f(s[j] - m_safe);
          sum += s[j];
        }
        tmem_parts16(sat, s);
        hand_over(&sl->p_full[it & 1]);
        l = l * f + sum;                                      // this thread's columns; added over the row at the end
        m = m_new;
        // the step before, from the other accumulator, under this one's product
        if (it > 0) {
          ok = wait(&sl->acc_full[(it - 1) & 1], (it - 1) >> 1, 80);
          drain(T_ACC1 + ((it - 1) & 1) * 128, acc1, true);
          tc_fence_before();                                  // (ordered before the next hand-over)
        }
#pragma unroll
        for (int c = 0; c < 16; ++c) acc1[c] *= f;
      } else {
        const int st = it % S::STAGES;
        // (the row statistics beside the tile)
        if (MODE == A_DKDV && !(ok = wait(&sl->full[st], it / S::STAGES, 82))) break;
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
          const float4 Lj = MODE == A_DKDV ? *reinterpret_cast<const float4*>(&sl->lse[st][col + j]) : make_float4(L, L, L, L);
          s[j] = exp2f(s[j] * scale - Lj.x);
          s[j + 1] = exp2f(s[j + 1] * scale - Lj.y);
          s[j + 2] = exp2f(s[j + 2] * scale - Lj.z);
          s[j + 3] = exp2f(s[j + 3] * scale - Lj.w);
        }
        if (edge) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const int x = xb + j;
            if (MODE == A_DKDV ? x >= T || t > x : t >= T || x > t) s[j] = 0.f;
          }
        }
        if constexpr (MODE == A_DKDV) {
          tmem_parts16(sat, s);
          if (it > 0) drain(T_ACC1, acc1, false);             // (S was issued after the dV of the step before)
          hand_over(&sl->p_full[0]);
        }
        if (!(ok = wait(&sl->dp_full, it, 83))) break;
        float ds[16];
        tmem_sum16(lanes + T_DP, ds);
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
          const float4 dj = MODE == A_DKDV ? *reinterpret_cast<const float4*>(&sl->delta[st][col + j]) : make_float4(dl, dl, dl, dl);
          ds[j] = s[j] * (ds[j] - dj.x) * a.sm_scale;
          ds[j + 1] = s[j + 1] * (ds[j + 1] - dj.y) * a.sm_scale;
          ds[j + 2] = s[j + 2] * (ds[j + 2] - dj.z) * a.sm_scale;
          ds[j + 3] = s[j + 3] * (ds[j + 3] - dj.w) * a.sm_scale;
        }
        tmem_parts16(lanes + T_DP, ds);
        // (dP was issued after the dK / dQ of the step before)
        if (it > 0) drain(MODE == A_DKDV ? T_ACC2 : T_ACC1, MODE == A_DKDV ? acc2 : acc1, false);
        hand_over(&sl->ds_full);
      }
    }
    if (n > 0 && ok) {
      const int b = MODE == A_FWD ? (n - 1) & 1 : 0;
      ok = wait(&sl->acc_full[b], MODE == A_FWD ? (n - 1) >> 1 : 0, 81);
      drain(T_ACC1 + b * 128, acc1, true);
      if constexpr (MODE == A_DKDV) drain(T_ACC2, acc2, true);
    }
    if (MODE == A_FWD) sl->mx[0][part][row] = l;              // (the last step's maxima were read before its p_full)
    named_bar_sync(2, APROD + ACOMP);                         // row sums and the largest operand are known
    // dP, a sum of 64 products, is off by that much more, and what it is off by comes times an operand
    const float top = fmaxf(1.f, __uint_as_float(sl->top)), tiny = split_tiny(64 * AX * n, top) * top;
    bool odd = false;
    float big = 0.f;
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      odd |= !(fabsf(acc1[c]) >= tiny) && acc1[c] != 0.f;
      big = fmaxf(big, fabsf(acc1[c]));
      if (MODE == A_DKDV) {
        odd |= !(fabsf(acc2[c]) >= tiny) && acc2[c] != 0.f;
        big = fmaxf(big, fabsf(acc2[c]));
      }
    }
    odd |= big == INFINITY;
    if (MODE == A_FWD) {
      l = (sl->mx[0][0][row] + sl->mx[0][1][row]) + (sl->mx[0][2][row] + sl->mx[0][3][row]);
    }
    odd &= t < T;
    if (t < T && !odd) store_results<MODE>(g, hx, t, col, acc1, acc2, m, l);
    again = odd;
  }
  tc_fence_before();
  const bool any = __syncthreads_or(again);
  if (warp == AISSUER) tmem_dealloc(tmem, 512);
  if (any) {
    const bool compute = warp >= APROD / 32 && warp < AISSUER;
    // back to one share for all
    if (compute) asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    else asm volatile("setmaxnreg.inc.sync.aligned.u32 72;");
    if (compute) attn_f32_repeat<MODE>(g, reinterpret_cast<float*>(smem), r0, x0, x1, again);
  }
}

// A structured head's CTA of the first row of the grid runs its scan, a sequential chain that ends long before the longest
// walks (launched on their own before: 17 us forward, 26 backward of the layer's 394 at T = 1024; now 366).  256 x 168 +
// 640 x 24 registers <= 896 x 72; the warps without work leave before the others take theirs, so that the compiler sees one
// path with the larger share.
__device__ __forceinline__ bool attn_f32_scan_head(const SafMixedAttnArgs& a, const ScanArgs& sc) {
  return blockIdx.y == 0 && sc.in != nullptr && head_index(a, blockIdx.x).state == SAF_SINK_DECAY;
}
template <bool BWD>
__device__ __forceinline__ void attn_f32_scan(const SafMixedAttnArgs& a, const ScanArgs& sc) {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 168;");
  extern __shared__ uint8_t attn_smem[];
  const int b = blockIdx.x / a.H, h = blockIdx.x % a.H;
  sink_decay_scan_cta<float, BWD, 0, true>(sc, b, h, 0, 0, -1, reinterpret_cast<float*>(attn_smem));
}

// grid (B * H, row tiles): the longest walks of all heads first
__global__ void __launch_bounds__(ATHREADS, 1) attn_f32_fwd_kernel(const __grid_constant__ SafMixedAttnBwdArgs g,
                                                                   const __grid_constant__ ScanArgs sc) {
  pdl_wait();
  pdl_trigger();
  if (attn_f32_scan_head(g.fwd, sc)) {
    if (threadIdx.x >= SCAN_NT) {
      asm volatile("setmaxnreg.dec.sync.aligned.u32 24;");
      return;
    }
    attn_f32_scan<false>(g.fwd, sc);
    return;
  }
  attn_f32_tile<A_FWD>(g, blockIdx.y, gridDim.y);
}
// grid (B * H, 2 x row tiles): dK / dV and dQ tiles of one length take turns.  One launch for both, because a row tile's walk
// has 2 to 2 tiles' length of steps and a launch of one kind alone ends with most SMs idle
__global__ void __launch_bounds__(ATHREADS, 1) attn_f32_bwd_kernel(const __grid_constant__ SafMixedAttnBwdArgs g,
                                                                   const __grid_constant__ ScanArgs sc) {
  pdl_wait();
  pdl_trigger();
  if (attn_f32_scan_head(g.fwd, sc)) {
    if (threadIdx.x >= SCAN_NT) {
      asm volatile("setmaxnreg.dec.sync.aligned.u32 24;");
      return;
    }
    attn_f32_scan<true>(g.fwd, sc);
    return;
  }
  if (blockIdx.y & 1) attn_f32_tile<A_DQ>(g, blockIdx.y >> 1, gridDim.y >> 1);
  else attn_f32_tile<A_DKDV>(g, blockIdx.y >> 1, gridDim.y >> 1);
}

// 16-byte rows: base, row, head and batch strides (an axis of one element is never stepped over)
bool f32_rows_ok(const SafTensor& t, int B, int Hn, int T) {
  return t.ptr && ((uintptr_t)t.ptr & 15) == 0 && t.stride[3] == 1 && (B < 2 || t.stride[0] % 4 == 0) && (Hn < 2 || t.stride[1] % 4 == 0) &&
         (T < 2 || t.stride[2] % 4 == 0);
}

bool f32_call_ok(const SafMixedAttnArgs& a) {
  const int kv = a.HKV > 0 ? a.HKV : 0;
  // (grid.y holds the row tiles)
  return a.dtype == SAF_F32 && a.HD == AHD && !a.rope && a.U > 0 && a.T <= 65535 * 64 && f32_rows_ok(a.q, a.B, a.U, a.T) &&
         f32_rows_ok(a.k, a.B, kv ? kv : a.U, a.T) && f32_rows_ok(a.v, a.B, kv ? kv : a.H, a.T) && f32_rows_ok(a.out, a.B, a.H, a.T);
}

}  // namespace

// The live heads of an fp32 call whose rows are whole 16-byte pieces and come rotated already; everything else stays
// with the any-type kernels.
int launch_attn_f32_fwd(const SafMixedAttnArgs& a, bool scan, cudaStream_t st) {
  if (!f32_call_ok(a)) return SAF_ERR_UNSUPPORTED;
  SafMixedAttnBwdArgs g;
  memset(&g, 0, sizeof(g));
  g.fwd = a;
  static PerDeviceOnce once;
  if (int rc = ensure_dyn_smem(attn_f32_fwd_kernel, AttnShape<A_FWD>::SMEM, once)) return rc;
  return launch_pdl("attn_f32_fwd_kernel", attn_f32_fwd_kernel, dim3(a.B * a.H, (a.T + AR - 1) / AR), ATHREADS, AttnShape<A_FWD>::SMEM, st, 1, g,
                    scan ? scan_args_fwd(a) : ScanArgs{});
}

bool attn_f32_bwd_ok(const SafMixedAttnBwdArgs& g) {
  const SafMixedAttnArgs& a = g.fwd;
  return f32_call_ok(a) && a.HKV == 0 && f32_rows_ok(g.dout, a.B, a.H, a.T) && f32_rows_ok(g.dv, a.B, a.H, a.T) &&
         f32_rows_ok(g.dq, a.B, a.U, a.T) && f32_rows_ok(g.dk, a.B, a.U, a.T);
}

// dK, dV and dQ; delta is filled already
int launch_attn_f32_bwd(const SafMixedAttnBwdArgs& g, bool scan, cudaStream_t st) {
  const SafMixedAttnArgs& a = g.fwd;
  if (!attn_f32_bwd_ok(g)) return SAF_ERR_UNSUPPORTED;
  constexpr int smem = AttnShape<A_DKDV>::SMEM;
  static_assert(smem >= AttnShape<A_DQ>::SMEM, "both kinds of tile fit");
  static PerDeviceOnce once;
  if (int rc = ensure_dyn_smem(attn_f32_bwd_kernel, smem, once)) return rc;
  return launch_pdl("attn_f32_bwd_kernel", attn_f32_bwd_kernel, dim3(a.B * a.H, 2 * ((a.T + AR - 1) / AR)), ATHREADS, smem, st, 1, g,
                    scan ? scan_args_bwd(g) : ScanArgs{});
}

}  // namespace saf
