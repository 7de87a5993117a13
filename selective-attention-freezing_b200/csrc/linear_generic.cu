// CUDA-core indexed linear (fp32 accumulate): forward for fp32 / shapes the
// tensor-core GEMM does not take, and both backward products.  Weight rows are
// addressed in place through the slab table; no gathered weight copy exists
// (the reference builds one per call, kernel/indexed_linear.py:93).
//
//   fwd : out[m, n]  = sum_c x[m,c] W[n][c] + b[n]          (kernel/indexed_linear.py:28-38, 86-98)
//   dx  : dx[m, c]   = sum_n dout[m,n] W[n][c]              (:47-49, 107-109)
//   dw  : dW[n][c]   = sum_m dout[m,n] x[m,c], db[n] = sum_m dout[m,n]   (:50-55, 110-121)
// where n = g*slab + r addresses row (row0[g] + r) of weight matrix slab_weight[g].
// Also: the freeze-time row normaliser of decomposed patterns (kernel/fused_attn.py:101-116).
#include "saf_internal.h"
#include "sm100_prims.cuh"

namespace saf {
namespace {

constexpr int MAX_SLABS = 2048;
struct SlabTable {
  int32_t row0[MAX_SLABS];
  uint8_t weight[MAX_SLABS];
  uint8_t rope[MAX_SLABS];
};
struct WeightSet {
  const void* w[SAF_MAX_WEIGHTS];
  const void* b[SAF_MAX_WEIGHTS];
  int64_t ldw[SAF_MAX_WEIGHTS];
  int64_t cdw[SAF_MAX_WEIGHTS];
};

constexpr int TM = 64, TN = 64, TK = 16, GNT = 256;

// pointer to element (row n of the selection, column c)
template <typename T>
__device__ __forceinline__ const T* welem(const WeightSet& ws, const SlabTable& tb, int n, int slab, int c) {
  const int g = n / slab, r = n - g * slab;
  const int w = tb.weight[g];
  return reinterpret_cast<const T*>(ws.w[w]) + (int64_t)(tb.row0[g] + r) * ws.ldw[w] + (int64_t)c * ws.cdw[w];
}

__device__ __forceinline__ void mma_tile(const float (*As)[TM + 1], const float (*Bs)[TN + 1], int ty, int tx,
                                         float (&acc)[4][4]) {
#pragma unroll
  for (int k = 0; k < TK; ++k) {
    float a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = As[k][ty * 4 + i];
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = Bs[k][tx + 16 * j];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
  }
}

// MODE 0: fwd, MODE 1: dx, MODE 2: dw
template <typename T, int MODE>
__global__ void __launch_bounds__(GNT) linear_generic_kernel(const T* __restrict__ A, int64_t lda,
                                                             const T* __restrict__ X, int64_t ldx, T* __restrict__ Cout,
                                                             int64_t ldc, int M, int C, int N, int slab,
                                                             const __grid_constant__ WeightSet ws,
                                                             const __grid_constant__ SlabTable tb) {
  __shared__ float As[TK][TM + 1];
  __shared__ float Bs[TK][TN + 1];
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  // problem shape (rows I, cols J, depth K) per mode
  const int I = (MODE == 2) ? N : M;
  const int J = (MODE == 0) ? N : C;
  const int K = (MODE == 0) ? C : (MODE == 1 ? N : M);
  const int i0 = blockIdx.y * TM, j0 = blockIdx.x * TN;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  for (int k0 = 0; k0 < K; k0 += TK) {
    for (int idx = tid; idx < TM * TK; idx += GNT) {
      float av = 0.f, bv = 0.f;
      if (MODE == 0 || MODE == 1) {
        // A(i,k): row-major, k contiguous
        const int ii = idx / TK, kk = idx - ii * TK;
        const int i = i0 + ii, k = k0 + kk;
        if (i < I && k < K) av = to_f<T>(A[(int64_t)i * lda + k]);
        As[kk][ii] = av;
      } else {
        // A(i=n, k=m) = dout[m*lda + n]: n contiguous
        const int kk = idx / TM, ii = idx - kk * TM;
        const int i = i0 + ii, k = k0 + kk;
        if (i < I && k < K) av = to_f<T>(A[(int64_t)k * lda + i]);
        As[kk][ii] = av;
      }
      if (MODE == 0) {
        const int jj = idx / TK, kk = idx - jj * TK;
        const int j = j0 + jj, k = k0 + kk;
        if (j < J && k < K) bv = to_f<T>(*welem<T>(ws, tb, j, slab, k));
        Bs[kk][jj] = bv;
      } else if (MODE == 1) {
        // B(j=c, k=n) = W[n][c]: c contiguous
        const int kk = idx / TN, jj = idx - kk * TN;
        const int j = j0 + jj, k = k0 + kk;
        if (j < J && k < K) bv = to_f<T>(*welem<T>(ws, tb, k, slab, j));
        Bs[kk][jj] = bv;
      } else {
        // B(j=c, k=m) = x[m*ldx + c]
        const int kk = idx / TN, jj = idx - kk * TN;
        const int j = j0 + jj, k = k0 + kk;
        if (j < J && k < K) bv = to_f<T>(X[(int64_t)k * ldx + j]);
        Bs[kk][jj] = bv;
      }
    }
    __syncthreads();
    mma_tile(As, Bs, ty, tx, acc);
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int ii = i0 + ty * 4 + i;
    if (ii >= I) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int jj = j0 + tx + 16 * j;
      if (jj >= J) continue;
      float v = acc[i][j];
      if (MODE == 0) {
        const int g = jj / slab, r = jj - g * slab;
        const int w = tb.weight[g];
        if (ws.b[w]) v += to_f<T>(reinterpret_cast<const T*>(ws.b[w])[tb.row0[g] + r]);
        Cout[(int64_t)ii * ldc + jj] = from_f<T>(v);
      } else if (MODE == 1) {
        if (X) v += to_f<T>(X[jj]);   // optional bias over the output columns
        Cout[(int64_t)ii * ldc + jj] = from_f<T>(v);
      } else {
        *const_cast<T*>(welem<T>(ws, tb, ii, slab, jj)) = from_f<T>(v);
      }
    }
  }
}

// ---- fp32, 16-byte rows ----------------------------------------------------------------------------------------------
// Bound by the FMA pipe once shared memory keeps up: a thread owns 8 x 8 outputs and reads its operands as float4 along
// whichever index they store contiguously, 16 reads for 256 FMAs (the any-shape kernel above: 8 for 16).  An operand
// stays in its own layout, K-contiguous rows (stride 36: 8 neighbouring rows' float4 reads hit all banks once) or
// row-contiguous K slices, so cp.async brings every tile and nothing is transposed.  Training products of one narrow
// layer are only 64 to 400 tiles of 64 x 64, so a CTA is four groups of 64 threads that each take a quarter of every K
// slice and add their sums at the end: four times the warps in flight for the same tiles, and shorter chains of sums.
// 2048 x 768 x 768 on a B200: forward 217 -> 82 us, dx 209 -> 84, dW 380 -> 68.
constexpr int FK = 32, FGROUPS = 4, FKG = FK / FGROUPS, FLD = FK + 4, FSTAGES = 3, FRED = 68;

// acc[i][j] = element (frag_row(i), frag_row(j)) of the group's tile
template <bool KC>
__device__ __forceinline__ int frag_at(int t, int i) { return KC ? t + 8 * i : t * 4 + (i & 3) + 32 * (i >> 2); }
__device__ __forceinline__ float f4c(const float4& v, int e) { return e == 0 ? v.x : (e == 1 ? v.y : (e == 2 ? v.z : v.w)); }

template <int MODE>
__global__ void __launch_bounds__(GNT, 2) linear_f32_kernel(const float* __restrict__ A, int64_t lda, const float* __restrict__ X,
                                                            int64_t ldx, float* __restrict__ Cout, int64_t ldc, int M, int C,
                                                            int N, int slab, const __grid_constant__ WeightSet ws,
                                                            const __grid_constant__ SlabTable tb) {
  constexpr bool A_KC = MODE != 2, B_KC = MODE == 0;
  constexpr int A_F = A_KC ? TM * FLD : FK * TM, B_F = B_KC ? TN * FLD : FK * TN;
  extern __shared__ __align__(16) float lin_smem[];
  const int tid = threadIdx.x, kg = tid >> 6, ty = (tid & 63) >> 3, tx = tid & 7;
  const int I = (MODE == 2) ? N : M;
  const int J = (MODE == 0) ? N : C;
  const int K = (MODE == 0) ? C : (MODE == 1 ? N : M);
  const int i0 = blockIdx.y * TM, j0 = blockIdx.x * TN;
  // MODE 0: the weight rows this thread copies pieces of
  const float* wrow[2] = {nullptr, nullptr};
  if constexpr (MODE == 0) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int j = j0 + ((tid + q * GNT) >> 3);
      if (j < J) wrow[q] = welem<float>(ws, tb, j, slab, 0);
    }
  }
  auto load = [&](int kt, int s) {
    float* as = lin_smem + s * (A_F + B_F);
    float* bs = as + A_F;
    const int k0 = kt * FK;
    const float* wk = nullptr;                 // MODE 1: row k0 of the selection (slabs are whole 32-row runs)
    int64_t wld = 0;
    if constexpr (MODE == 1) {
      wk = welem<float>(ws, tb, k0, slab, 0);
      wld = ws.ldw[tb.weight[k0 / slab]];
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int idx = tid + q * GNT;
      const int r = idx >> 3, rc = (idx & 7) * 4;      // K-contiguous: row, first k
      const int kk = idx >> 4, kc = (idx & 15) * 4;    // K slices: k, first row
      if constexpr (A_KC) {
        const bool ok = i0 + r < I && k0 + rc < K;
        cp_async16_zfill(as + r * FLD + rc, ok ? A + (int64_t)(i0 + r) * lda + k0 + rc : A, ok);
      } else {
        const bool ok = i0 + kc < I && k0 + kk < K;
        cp_async16_zfill(as + kk * TM + kc, ok ? A + (int64_t)(k0 + kk) * lda + i0 + kc : A, ok);
      }
      if constexpr (MODE == 0) {
        const bool ok = wrow[q] && k0 + rc < K;
        cp_async16_zfill(bs + r * FLD + rc, ok ? wrow[q] + k0 + rc : A, ok);
      } else if constexpr (MODE == 1) {
        const bool ok = j0 + kc < J;
        cp_async16_zfill(bs + kk * TN + kc, ok ? wk + kk * wld + j0 + kc : A, ok);
      } else {
        const bool ok = j0 + kc < J && k0 + kk < K;
        cp_async16_zfill(bs + kk * TN + kc, ok ? X + (int64_t)(k0 + kk) * ldx + j0 + kc : A, ok);
      }
    }
  };
  float acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
  const int KT = (K + FK - 1) / FK;
#pragma unroll
  for (int s = 0; s < FSTAGES - 1; ++s) {
    if (s < KT) load(s, s);
    cp_async_commit();
  }
  for (int kt = 0; kt < KT; ++kt) {
    cp_async_wait<FSTAGES - 2>();
    __syncthreads();
    if (kt + FSTAGES - 1 < KT) load(kt + FSTAGES - 1, (kt + FSTAGES - 1) % FSTAGES);
    cp_async_commit();
    const float* as = lin_smem + (kt % FSTAGES) * (A_F + B_F);
    const float* bs = as + A_F;
    if constexpr (A_KC && B_KC) {
#pragma unroll
      for (int h = 0; h < FKG; h += 4) {
        float4 b[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) b[j] = *reinterpret_cast<const float4*>(bs + (tx + 8 * j) * FLD + kg * FKG + h);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 a = *reinterpret_cast<const float4*>(as + (ty + 8 * i) * FLD + kg * FKG + h);
#pragma unroll
          for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(f4c(a, e), f4c(b[j], e), acc[i][j]);
        }
      }
    } else {
#pragma unroll
      for (int h = 0; h < FKG; h += 4) {
        float4 ak[8];
        if constexpr (A_KC) {
#pragma unroll
          for (int i = 0; i < 8; ++i) ak[i] = *reinterpret_cast<const float4*>(as + (ty + 8 * i) * FLD + kg * FKG + h);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int k = kg * FKG + h + e;
          const float4 b0 = *reinterpret_cast<const float4*>(bs + k * TN + tx * 4);
          const float4 b1 = *reinterpret_cast<const float4*>(bs + k * TN + 32 + tx * 4);
          float4 a0, a1;
          if constexpr (!A_KC) {
            a0 = *reinterpret_cast<const float4*>(as + k * TM + ty * 4);
            a1 = *reinterpret_cast<const float4*>(as + k * TM + 32 + ty * 4);
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            float av;
            if constexpr (A_KC) av = f4c(ak[i], e);
            else av = f4c(i < 4 ? a0 : a1, i & 3);
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(av, f4c(j < 4 ? b0 : b1, j & 3), acc[i][j]);
          }
        }
      }
    }
  }
  // ---- the groups' sums, added in order
  cp_async_wait<0>();
  __syncthreads();
  float* red = lin_smem + kg * TM * FRED;
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) red[frag_at<A_KC>(ty, i) * FRED + frag_at<B_KC>(tx, j)] = acc[i][j];
  __syncthreads();
#pragma unroll
  for (int q = 0; q < TM * TN / 4 / GNT; ++q) {
    const int idx = tid + q * GNT, r = idx >> 4, c = (idx & 15) * 4;
    const int ii = i0 + r, jj = j0 + c;
    if (ii >= I || jj >= J) continue;
    float4 v = *reinterpret_cast<const float4*>(lin_smem + r * FRED + c);
#pragma unroll
    for (int g = 1; g < FGROUPS; ++g) {
      const float4 t = *reinterpret_cast<const float4*>(lin_smem + (g * TM + r) * FRED + c);
      v.x += t.x; v.y += t.y; v.z += t.z; v.w += t.w;
    }
    const float* bias = nullptr;
    if constexpr (MODE == 0) {
      const int g = jj / slab;
      const float* b = reinterpret_cast<const float*>(ws.b[tb.weight[g]]);
      if (b) bias = b + tb.row0[g] + (jj - g * slab);
    } else if constexpr (MODE == 1) {
      if (X) bias = X + jj;                    // optional bias over the output columns
    }
    if (bias) {
      v.x += bias[0]; v.y += bias[1]; v.z += bias[2]; v.w += bias[3];
    }
    float* dst = MODE == 2 ? const_cast<float*>(welem<float>(ws, tb, ii, slab, jj)) : Cout + (int64_t)ii * ldc + jj;
    *reinterpret_cast<float4*>(dst) = v;
  }
}

// Whether every row the product touches is made of whole 16-byte pieces and a 32-deep K slice stays inside one slab.
// A: the left operand (x, or dout in the backward); Cout is null for the weight gradient.
bool f32_rows_ok(const SafIndexedLinearArgs& a, const void* A, int64_t lda, const void* X, int64_t ldx, const void* Cout, int64_t ldc) {
  auto ok = [](const void* p, int64_t ld) { return ((uintptr_t)p & 15) == 0 && ld % 4 == 0; };
  if (a.slab % 32 || a.C % 4 || !ok(A, lda) || !ok(X, ldx) || !ok(Cout, ldc)) return false;
  for (int w = 0; w < a.n_weights; ++w)
    if (!ok(a.weights[w], a.ldw[w]) || (a.cdw[w] != 0 && a.cdw[w] != 1)) return false;
  return true;
}

template <int MODE>
int launch_linear_f32(dim3 grid, const void* A, int64_t lda, const void* X, int64_t ldx, void* Cout, int64_t ldc, const SafIndexedLinearArgs& a,
                      const WeightSet& ws, const SlabTable& tb, cudaStream_t st) {
  constexpr int A_F = MODE != 2 ? TM * FLD : FK * TM, B_F = MODE == 0 ? TN * FLD : FK * TN;
  constexpr int smem = 4 * (FSTAGES * (A_F + B_F) > FGROUPS * TM * FRED ? FSTAGES * (A_F + B_F) : FGROUPS * TM * FRED);
  static PerDeviceOnce once;
  if (int rc = ensure_dyn_smem(linear_f32_kernel<MODE>, smem, once)) return rc;
  linear_f32_kernel<MODE><<<grid, GNT, smem, st>>>(reinterpret_cast<const float*>(A), lda, reinterpret_cast<const float*>(X), ldx,
                                                   reinterpret_cast<float*>(Cout), ldc, a.M, a.C, a.n_slabs * a.slab, a.slab, ws, tb);
  count_launch();
  return check_launch("linear_f32_kernel");
}

// db[n] = sum_m dout[m, n], scattered to bias rows
template <typename T>
__global__ void bias_grad_kernel(const T* __restrict__ dout, int64_t lddo, int M, int N, int slab,
                                 const __grid_constant__ WeightSet ws, const __grid_constant__ SlabTable tb) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  const int g = n / slab, r = n - g * slab;
  const int w = tb.weight[g];
  if (!ws.b[w]) return;
  float s = 0.f;
  for (int m = 0; m < M; ++m) s += to_f<T>(dout[(int64_t)m * lddo + n]);
  const_cast<T*>(reinterpret_cast<const T*>(ws.b[w]))[tb.row0[g] + r] = from_f<T>(s);
}

// in-place rotation of the rotated slabs of out (generic path only; the
// tensor-core GEMM rotates in its epilogue)
template <typename T>
__global__ void rope_slabs_kernel(T* __restrict__ out, int64_t ldo, int M, int n_slabs, int slab, int Tlen,
                                  const float* __restrict__ cosT, const float* __restrict__ sinT,
                                  const __grid_constant__ SlabTable tb, float sgn) {
  const int half = slab >> 1;
  const int64_t total = (int64_t)M * n_slabs * half;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x) {
    const int d = (int)(idx % half);
    const int g = (int)((idx / half) % n_slabs);
    const int64_t m = idx / ((int64_t)half * n_slabs);
    if (!tb.rope[g]) continue;
    const int t = (int)(m % Tlen);
    T* p = out + m * ldo + (int64_t)g * slab;
    const float x1 = to_f<T>(p[d]), x2 = to_f<T>(p[d + half]);
    // sgn = -1 gives the adjoint (inverse) rotation; the tables repeat per half
    const float c1 = cosT[(int64_t)t * slab + d], s1 = sgn * sinT[(int64_t)t * slab + d];
    const float c2 = cosT[(int64_t)t * slab + d + half], s2 = sgn * sinT[(int64_t)t * slab + d + half];
    p[d] = from_f<T>(x1 * c1 - x2 * s1);
    p[d + half] = from_f<T>(x2 * c2 + x1 * s2);
  }
}

// bf16, 16-byte accesses: one thread rotates 8 pairs (d .. d+7, d+half .. d+half+7) of one slab of one row
__global__ void __launch_bounds__(256) rope_slabs_vec_kernel(__nv_bfloat16* __restrict__ out, int64_t ldo, int M, int n_slabs,
                                                             int slab, int Tlen, const float* __restrict__ cosT,
                                                             const float* __restrict__ sinT,
                                                             const __grid_constant__ SlabTable tb, float sgn) {
  pdl_wait();
  pdl_trigger();
  const int half = slab >> 1, per_slab = half >> 3;
  const int64_t total = (int64_t)M * n_slabs * per_slab;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x) {
    const int d = (int)(idx % per_slab) * 8;
    const int g = (int)((idx / per_slab) % n_slabs);
    const int64_t m = idx / ((int64_t)per_slab * n_slabs);
    if (!tb.rope[g]) continue;
    const int t = (int)(m % Tlen);
    __nv_bfloat16* p = out + m * ldo + (int64_t)g * slab + d;
    uint4 lo = *reinterpret_cast<const uint4*>(p), hi = *reinterpret_cast<const uint4*>(p + half);
    const float4* c4 = reinterpret_cast<const float4*>(cosT + (int64_t)t * slab + d);
    const float4* s4 = reinterpret_cast<const float4*>(sinT + (int64_t)t * slab + d);
    const float4 ca = c4[0], cb = c4[1], sa = s4[0], sb = s4[1];
    const float cc[8] = {ca.x, ca.y, ca.z, ca.w, cb.x, cb.y, cb.z, cb.w};
    const float ss[8] = {sa.x, sa.y, sa.z, sa.w, sb.x, sb.y, sb.z, sb.w};
    uint32_t lw[4] = {lo.x, lo.y, lo.z, lo.w}, hw[4] = {hi.x, hi.y, hi.z, hi.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float x1a = __uint_as_float(lw[e] << 16), x1b = __uint_as_float(lw[e] & 0xffff0000u);
      const float x2a = __uint_as_float(hw[e] << 16), x2b = __uint_as_float(hw[e] & 0xffff0000u);
      const float sA = sgn * ss[2 * e], sB = sgn * ss[2 * e + 1];   // the tables repeat per half
      const __nv_bfloat162 l2 = __floats2bfloat162_rn(x1a * cc[2 * e] - x2a * sA, x1b * cc[2 * e + 1] - x2b * sB);
      const __nv_bfloat162 h2 = __floats2bfloat162_rn(x2a * cc[2 * e] + x1a * sA, x2b * cc[2 * e + 1] + x1b * sB);
      lw[e] = *reinterpret_cast<const uint32_t*>(&l2);
      hw[e] = *reinterpret_cast<const uint32_t*>(&h2);
    }
    *reinterpret_cast<uint4*>(p) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
    *reinterpret_cast<uint4*>(p + half) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
  }
}

int fill_tables(const SafIndexedLinearArgs& a, WeightSet* ws, SlabTable* tb) {
  if (a.n_slabs > MAX_SLABS) return fail(SAF_ERR_LIMIT, "n_slabs %d exceeds the limit of %d", a.n_slabs, MAX_SLABS);
  memset(ws, 0, sizeof(*ws));
  memset(tb, 0, sizeof(*tb));
  for (int w = 0; w < a.n_weights; ++w) {
    ws->w[w] = a.weights[w];
    ws->b[w] = a.biases[w];
    ws->ldw[w] = a.ldw[w];
    ws->cdw[w] = a.cdw[w] ? a.cdw[w] : 1;
  }
  for (int g = 0; g < a.n_slabs; ++g) {
    tb->row0[g] = a.slab_row0[g];
    tb->weight[g] = (uint8_t)a.slab_weight[g];
    tb->rope[g] = (uint8_t)(a.slab_rope ? (a.slab_rope[g] != 0) : 0);
  }
  return SAF_OK;
}

template <typename T>
int gemm_generic_typed(const SafIndexedLinearArgs& a, int mode, const void* dout, int64_t lddo, void* dx,
                       int64_t lddx, const void* bias, cudaStream_t st) {
  WeightSet ws;
  SlabTable tb;
  int rc = fill_tables(a, &ws, &tb);
  if (rc) return rc;
  const int N = a.n_slabs * a.slab;
  constexpr bool f32 = sizeof(T) == 4;
  if (mode == 0) {
    dim3 grid((N + TN - 1) / TN, (a.M + TM - 1) / TM);
    if (f32 && f32_rows_ok(a, a.x, a.ldx, nullptr, 0, a.out, a.ldo)) {
      if ((rc = launch_linear_f32<0>(grid, a.x, a.ldx, nullptr, 0, a.out, a.ldo, a, ws, tb, st))) return rc;
    } else {
      linear_generic_kernel<T, 0><<<grid, GNT, 0, st>>>(reinterpret_cast<const T*>(a.x), a.ldx, nullptr, 0,
                                                        reinterpret_cast<T*>(a.out), a.ldo, a.M, a.C, N, a.slab, ws, tb);
      count_launch();
      if ((rc = check_launch("linear_generic_kernel<fwd>"))) return rc;
    }
    bool any_rope = false;
    for (int g = 0; g < a.n_slabs; ++g) any_rope |= tb.rope[g] != 0;
    if (any_rope) {
      const int64_t total = (int64_t)a.M * a.n_slabs * (a.slab / 2);
      const int blocks = (int)std::min<int64_t>((total + 255) / 256, 148 * 16);
      rope_slabs_kernel<T><<<blocks, 256, 0, st>>>(reinterpret_cast<T*>(a.out), a.ldo, a.M, a.n_slabs, a.slab, a.T,
                                                  a.rope_cos, a.rope_sin, tb, 1.f);
      count_launch();
      if ((rc = check_launch("rope_slabs_kernel"))) return rc;
    }
  } else if (mode == 1) {
    dim3 grid((a.C + TN - 1) / TN, (a.M + TM - 1) / TM);
    if (f32 && f32_rows_ok(a, dout, lddo, nullptr, 0, dx, lddx))
      return launch_linear_f32<1>(grid, dout, lddo, bias, 0, dx, lddx, a, ws, tb, st);
    linear_generic_kernel<T, 1><<<grid, GNT, 0, st>>>(reinterpret_cast<const T*>(dout), lddo,
                                                      reinterpret_cast<const T*>(bias), 0,
                                                      reinterpret_cast<T*>(dx), lddx, a.M, a.C, N, a.slab, ws, tb);
    count_launch();
    if ((rc = check_launch("linear_generic_kernel<dx>"))) return rc;
  } else {
    dim3 grid((a.C + TN - 1) / TN, (N + TM - 1) / TM);
    if (f32 && f32_rows_ok(a, dout, lddo, a.x, a.ldx, nullptr, 0)) {
      if ((rc = launch_linear_f32<2>(grid, dout, lddo, a.x, a.ldx, nullptr, 0, a, ws, tb, st))) return rc;
    } else {
      linear_generic_kernel<T, 2><<<grid, GNT, 0, st>>>(reinterpret_cast<const T*>(dout), lddo,
                                                        reinterpret_cast<const T*>(a.x), a.ldx, nullptr, 0, a.M, a.C, N,
                                                        a.slab, ws, tb);
      count_launch();
      if ((rc = check_launch("linear_generic_kernel<dw>"))) return rc;
    }
    bool any_bias = false;
    for (int w = 0; w < a.n_weights; ++w) any_bias |= a.biases[w] != nullptr;
    if (any_bias) {
      bias_grad_kernel<T><<<(N + 127) / 128, 128, 0, st>>>(reinterpret_cast<const T*>(dout), lddo, a.M, N, a.slab, ws, tb);
      count_launch();
      if ((rc = check_launch("bias_grad_kernel"))) return rc;
    }
  }
  return SAF_OK;
}

// z[h,i] = logsumexp_{j<=i}(alpha[h,j] + rho[h,i-j]); one warp per row
__global__ void logz_kernel(const float* __restrict__ alpha, const float* __restrict__ rho, float* __restrict__ z,
                            int H, int S, int rows) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= H * S) return;
  const int h = warp / S, i = warp - h * S;
  if (i >= rows) {
    if (lane == 0) z[(int64_t)h * S + i] = 0.f;
    return;
  }
  const float* al = alpha + (int64_t)h * S;
  const float* rh = rho + (int64_t)h * S;
  // the row's maximum first, then the sum against it: short chains instead of one that rescales as it goes
  // (12 heads, 2048 rows: 55 -> 42 us, now bound by the instructions of 25 M expf).
  // Entries that are -inf or NaN take no part.
  float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
  int j = lane;
  for (; j + 96 <= i; j += 128)
#pragma unroll
    for (int e = 0; e < 4; ++e) mx[e] = fmaxf(mx[e], al[j + 32 * e] + rh[i - j - 32 * e]);
  for (; j <= i; j += 32) mx[0] = fmaxf(mx[0], al[j] + rh[i - j]);
  float m = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
#pragma unroll
  for (int off = 16; off; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
  float sm[4] = {0.f, 0.f, 0.f, 0.f};
  auto term = [&](int jj) {
    const float x = al[jj] + rh[i - jj];
    return x > -INFINITY ? expf(x - m) : 0.f;
  };
  j = lane;
  for (; j + 96 <= i; j += 128)
#pragma unroll
    for (int e = 0; e < 4; ++e) sm[e] += term(j + 32 * e);
  for (; j <= i; j += 32) sm[0] += term(j);
  float s = (sm[0] + sm[1]) + (sm[2] + sm[3]);
#pragma unroll
  for (int off = 16; off; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  if (lane == 0) z[(int64_t)h * S + i] = m + logf(s);
}

}  // namespace

int launch_gemm_generic(const SafIndexedLinearArgs& a, cudaStream_t st) {
  if (a.dtype == SAF_F32) return gemm_generic_typed<float>(a, 0, nullptr, 0, nullptr, 0, nullptr, st);
  return gemm_generic_typed<__nv_bfloat16>(a, 0, nullptr, 0, nullptr, 0, nullptr, st);
}
int launch_gemm_bwd_dx(const SafIndexedLinearArgs& a, const void* dout, int64_t lddo, void* dx, int64_t lddx,
                       const void* bias, cudaStream_t st) {
  if (a.dtype == SAF_F32) return gemm_generic_typed<float>(a, 1, dout, lddo, dx, lddx, bias, st);
  return gemm_generic_typed<__nv_bfloat16>(a, 1, dout, lddo, dx, lddx, bias, st);
}
int launch_gemm_bwd_dw(const SafIndexedLinearArgs& a, const void* dout, int64_t lddo, cudaStream_t st) {
  if (a.dtype == SAF_F32) return gemm_generic_typed<float>(a, 2, dout, lddo, nullptr, 0, nullptr, st);
  return gemm_generic_typed<__nv_bfloat16>(a, 2, dout, lddo, nullptr, 0, nullptr, st);
}
int launch_rope_slabs(void* x, int64_t ld, int M, int n_slabs, int slab, int T, const int32_t* slab_rope,
                      const float* cosT, const float* sinT, int dtype, int inverse, cudaStream_t st) {
  if (n_slabs > MAX_SLABS) return fail(SAF_ERR_LIMIT, "n_slabs %d exceeds the limit of %d", n_slabs, MAX_SLABS);
  SlabTable tb;
  memset(&tb, 0, sizeof(tb));
  for (int g = 0; g < n_slabs; ++g) tb.rope[g] = (uint8_t)(slab_rope ? (slab_rope[g] != 0) : 1);
  const int64_t total = (int64_t)M * n_slabs * (slab / 2);
  const int blocks = (int)std::min<int64_t>((total + 255) / 256, 148 * 16);
  const float sgn = inverse ? -1.f : 1.f;
  const bool vec = dtype == SAF_BF16 && slab % 16 == 0 && ld % 8 == 0 && ((uintptr_t)x & 15) == 0 &&
                   ((uintptr_t)cosT & 15) == 0 && ((uintptr_t)sinT & 15) == 0;
  if (vec) {
    const int64_t tv = (int64_t)M * n_slabs * (slab / 16);
    const int bv = (int)std::min<int64_t>((tv + 255) / 256, 148 * 32);
    return launch_pdl("rope_slabs_kernel", rope_slabs_vec_kernel, dim3(bv), 256, 0, st, 1, reinterpret_cast<__nv_bfloat16*>(x), ld, M,
                      n_slabs, slab, T, cosT, sinT, tb, sgn);
  } else if (dtype == SAF_F32)
    rope_slabs_kernel<float><<<blocks, 256, 0, st>>>(reinterpret_cast<float*>(x), ld, M, n_slabs, slab, T, cosT, sinT, tb, sgn);
  else
    rope_slabs_kernel<__nv_bfloat16><<<blocks, 256, 0, st>>>(reinterpret_cast<__nv_bfloat16*>(x), ld, M, n_slabs, slab, T,
                                                            cosT, sinT, tb, sgn);
  count_launch();
  return check_launch("rope_slabs_kernel");
}
int launch_logz(const float* alpha, const float* rho, float* z, int H, int S, int rows, cudaStream_t st) {
  const int64_t warps = (int64_t)H * S;
  const int64_t blocks = (warps * 32 + 255) / 256;
  logz_kernel<<<(unsigned)blocks, 256, 0, st>>>(alpha, rho, z, H, S, rows);
  count_launch();
  return check_launch("logz_kernel");
}

}  // namespace saf
