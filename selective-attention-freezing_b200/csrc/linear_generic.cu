// CUDA-core indexed linear (fp32 accumulate): forward for rows that are not whole 16-byte pieces / shapes the
// tensor-core GEMM does not take, and both backward products.  Weight rows are
// addressed in place through the slab table; no gathered weight copy exists
// (the reference builds one per call, kernel/indexed_linear.py:93).
//
//   fwd : out[m, n]  = sum_c x[m,c] W[n][c] + b[n]          (kernel/indexed_linear.py:28-38, 86-98)
//   dx  : dx[m, c]   = sum_n dout[m,n] W[n][c]              (:47-49, 107-109)
//   dw  : dW[n][c]   = sum_m dout[m,n] x[m,c], db[n] = sum_m dout[m,n]   (:50-55, 110-121)
// where n = g*slab + r addresses row (row0[g] + r) of weight matrix slab_weight[g].
// Also: the freeze-time row normaliser of decomposed patterns (kernel/fused_attn.py:101-116).
#include "linear_tables.cuh"
#include "saf_internal.h"
#include "sm100_prims.cuh"

namespace saf {
namespace {

constexpr int TM = 64, TN = 64, TK = 16, GNT = 256;

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

// Whether every row the product touches is made of whole 16-byte pieces and a 32-deep K slice stays inside one slab.
// A: the left operand (x, or dout in the backward); Cout is null for the weight gradient.
bool f32_rows_ok(const SafIndexedLinearArgs& a, const void* A, int64_t lda, const void* X, int64_t ldx, const void* Cout, int64_t ldc) {
  auto ok = [](const void* p, int64_t ld) { return ((uintptr_t)p & 15) == 0 && ld % 4 == 0; };
  if (a.slab % 32 || a.C % 4 || !ok(A, lda) || !ok(X, ldx) || !ok(Cout, ldc)) return false;
  for (int w = 0; w < a.n_weights; ++w)
    if (!ok(a.weights[w], a.ldw[w]) || (a.cdw[w] != 0 && a.cdw[w] != 1)) return false;
  return true;
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

// fp32, 16-byte accesses: one thread rotates 4 pairs of one slab of one row (2048 rows of 18 heads x 64: 10.5 -> 5 us)
__global__ void __launch_bounds__(256) rope_slabs_f32x4_kernel(float* __restrict__ out, int64_t ldo, uint32_t total, uint32_t n_slabs,
                                                               uint32_t slab, uint32_t Tlen, const float* __restrict__ cosT,
                                                               const float* __restrict__ sinT, const __grid_constant__ SlabTable tb, float sgn) {
  pdl_wait();
  pdl_trigger();
  const uint32_t half = slab >> 1, per_slab = half >> 2;
  for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
    const uint32_t q = idx / per_slab, d = (idx - q * per_slab) * 4, m = q / n_slabs, g = q - m * n_slabs;
    if (!tb.rope[g]) continue;
    float* p = out + (int64_t)m * ldo + (int64_t)g * slab + d;
    const int64_t at = (int64_t)(m % Tlen) * slab + d;
    const float4 x1 = *reinterpret_cast<const float4*>(p), x2 = *reinterpret_cast<const float4*>(p + half);
    const float4 c1 = *reinterpret_cast<const float4*>(cosT + at), c2 = *reinterpret_cast<const float4*>(cosT + at + half);
    const float4 s1 = *reinterpret_cast<const float4*>(sinT + at), s2 = *reinterpret_cast<const float4*>(sinT + at + half);
    *reinterpret_cast<float4*>(p) = make_float4(x1.x * c1.x - x2.x * (sgn * s1.x), x1.y * c1.y - x2.y * (sgn * s1.y),
                                                x1.z * c1.z - x2.z * (sgn * s1.z), x1.w * c1.w - x2.w * (sgn * s1.w));
    *reinterpret_cast<float4*>(p + half) = make_float4(x2.x * c2.x + x1.x * (sgn * s2.x), x2.y * c2.y + x1.y * (sgn * s2.y),
                                                       x2.z * c2.z + x1.z * (sgn * s2.z), x2.w * c2.w + x1.w * (sgn * s2.w));
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

// fp32 rows in place; rows, tables and slabs of whole 16-byte pieces go four pairs at a time
int rope_f32(float* x, int64_t ld, int M, int n_slabs, int slab, int T, const float* cosT, const float* sinT, const SlabTable& tb, float sgn,
             cudaStream_t st) {
  const int64_t pairs = (int64_t)M * n_slabs * (slab / 2);
  if (slab % 8 == 0 && ld % 4 == 0 && !(((uintptr_t)x | (uintptr_t)cosT | (uintptr_t)sinT) & 15) && pairs / 4 <= 0x7fffffff) {
    const int blocks = (int)std::min<int64_t>((pairs / 4 + 255) / 256, 148 * 32);
    return launch_pdl("rope_slabs_kernel", rope_slabs_f32x4_kernel, dim3(blocks), 256, 0, st, 1, x, ld, (uint32_t)(pairs / 4), (uint32_t)n_slabs,
                      (uint32_t)slab, (uint32_t)T, cosT, sinT, tb, sgn);
  }
  rope_slabs_kernel<float><<<(int)std::min<int64_t>((pairs + 255) / 256, 148 * 16), 256, 0, st>>>(x, ld, M, n_slabs, slab, T, cosT, sinT, tb, sgn);
  count_launch();
  return check_launch("rope_slabs_kernel");
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
      if ((rc = launch_linear_f32(0, a.x, a.ldx, nullptr, 0, a.out, a.ldo, a, ws, tb, st))) return rc;
    } else {
      linear_generic_kernel<T, 0><<<grid, GNT, 0, st>>>(reinterpret_cast<const T*>(a.x), a.ldx, nullptr, 0,
                                                        reinterpret_cast<T*>(a.out), a.ldo, a.M, a.C, N, a.slab, ws, tb);
      count_launch();
      if ((rc = check_launch("linear_generic_kernel<fwd>"))) return rc;
    }
    bool any_rope = false;
    for (int g = 0; g < a.n_slabs; ++g) any_rope |= tb.rope[g] != 0;
    if (any_rope && f32)
      return rope_f32(reinterpret_cast<float*>(a.out), a.ldo, a.M, a.n_slabs, a.slab, a.T, a.rope_cos, a.rope_sin, tb, 1.f, st);
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
      return launch_linear_f32(1, dout, lddo, bias, 0, dx, lddx, a, ws, tb, st);
    linear_generic_kernel<T, 1><<<grid, GNT, 0, st>>>(reinterpret_cast<const T*>(dout), lddo,
                                                      reinterpret_cast<const T*>(bias), 0,
                                                      reinterpret_cast<T*>(dx), lddx, a.M, a.C, N, a.slab, ws, tb);
    count_launch();
    if ((rc = check_launch("linear_generic_kernel<dx>"))) return rc;
  } else {
    dim3 grid((a.C + TN - 1) / TN, (N + TM - 1) / TM);
    if (f32 && f32_rows_ok(a, dout, lddo, a.x, a.ldx, nullptr, 0)) {
      if ((rc = launch_linear_f32(2, dout, lddo, a.x, a.ldx, nullptr, 0, a, ws, tb, st))) return rc;
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
                            const int32_t* __restrict__ states, int H, int S, int rows) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= H * S) return;
  const int h = warp / S, i = warp - h * S;
  if (i >= rows || (states && states[h] != SAF_DECOMP)) {
    if (lane == 0) z[(int64_t)h * S + i] = 0.f;
    return;
  }
  const float* al = alpha + (int64_t)h * S;
  const float* rh = rho + (int64_t)h * S;
  // the row's maximum first, then the sum against it: short chains instead of one that rescales as it goes
  // (12 heads, 2048 rows: 55 -> 42 us, now bound by the instructions of 25 M expf; of a layer with 3 decomposed heads only
  // theirs are computed)
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
  }
  if (dtype == SAF_F32) return rope_f32(reinterpret_cast<float*>(x), ld, M, n_slabs, slab, T, cosT, sinT, tb, sgn, st);
  rope_slabs_kernel<__nv_bfloat16><<<blocks, 256, 0, st>>>(reinterpret_cast<__nv_bfloat16*>(x), ld, M, n_slabs, slab, T,
                                                            cosT, sinT, tb, sgn);
  count_launch();
  return check_launch("rope_slabs_kernel");
}
int launch_logz(const float* alpha, const float* rho, float* z, const int32_t* states, int H, int S, int rows, cudaStream_t st) {
  const int64_t warps = (int64_t)H * S;
  const int64_t blocks = (warps * 32 + 255) / 256;
  logz_kernel<<<(unsigned)blocks, 256, 0, st>>>(alpha, rho, z, states, H, S, rows);
  count_launch();
  return check_launch("logz_kernel");
}

}  // namespace saf
