// fp32 attention of the live heads at head_dim 64: forward, dK / dV and dQ on the CUDA cores in true fp32.
//
// What bounds it: the FMA pipe (the tensor cores have no fp32 product), so everything else has to stay out of its way.  The
// any-type kernels beside this file read two operands from shared memory for every two FMAs and spend their time there.
// Here a thread owns 8 x 4 outputs of a 64 x 64 tile and reads its operands as float4 along the contraction index, or
// along the output columns where the operand is stored that way: 12 16-byte reads for 128 FMAs.  Every operand is used
// in the layout it has in memory (rows of 64 floats), so tiles arrive by cp.async and nothing is transposed.  Rows of a
// probability tile are written and read by the same half-warp: no block-wide barrier between the two products.
//
//   forward  CTA = 64 query rows, walks the key tiles; K of the next tile loads under softmax and P V, V under Q K^T
//   dK / dV  CTA = 64 keys, S^T = K Q^T and dP^T = V dO^T, then dV += P^T dO, dK += dS^T Q
//   dQ       CTA = 64 query rows, S, dP, dQ += dS K
// 9 live heads, T = 1024, B = 2 on a B200: forward 365 -> 151 us, dK / dV 581 -> 246, dQ 389 -> 192.
// The same split as the reference (kernel/fused_attn.py:228-289, 415-481, 483-540): no atomics, fixed order of sums.
#include "head_index.cuh"
#include "saf_internal.h"
#include "sm100_prims.cuh"

namespace saf {
namespace {

constexpr int FB = 64;          // rows, keys and columns of a tile
constexpr int FHD = 64;
constexpr int FLD = 68;         // row stride of operand tiles: float4 reads of 8 neighbouring rows hit all banks once
constexpr int FLP = 80;         // row stride of probability tiles: the two rows a warp writes lie 16 banks apart
constexpr int FNT = 128;
constexpr float F_LOG2E = 1.4426950408889634f;
constexpr int TILE_F = FB * FLD, PROB_F = FB * FLP;

// rows row0 .. row0+63 of one head -> dst[r * FLD + d]; rows from T on are zero
__device__ __forceinline__ void f32_tile(float* dst, const float* base, int64_t s_row, int row0, int T) {
#pragma unroll
  for (int q = 0; q < FB * FHD / 4 / FNT; ++q) {
    const int idx = threadIdx.x + q * FNT, r = idx >> 4, c = (idx & 15) * 4;
    const bool ok = row0 + r < T;
    cp_async16_zfill(dst + r * FLD + c, ok ? base + (int64_t)(row0 + r) * s_row + c : base, ok);
  }
}

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float comp(const float4& v, int e) { return e == 0 ? v.x : (e == 1 ? v.y : (e == 2 ? v.z : v.w)); }

// s[i][j] = sum_d A[ty + 8i][d] B[tx + 16j][d]
__device__ __forceinline__ void f32_dot(const float* A, const float* B, int ty, int tx, float (&s)[8][4]) {
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 4
  for (int d = 0; d < FHD; d += 4) {
    float4 b[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = ld4(B + (tx + 16 * j) * FLD + d);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float4 a = ld4(A + (ty + 8 * i) * FLD + d);
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int j = 0; j < 4; ++j) s[i][j] = fmaf(comp(a, e), comp(b[j], e), s[i][j]);
    }
  }
}

// acc[i][c] += sum_k P[ty + 8i][k] B[k][4 tx + c]
__device__ __forceinline__ void f32_acc(const float* P, const float* B, int ty, int tx, float (&acc)[8][4]) {
#pragma unroll 2
  for (int k = 0; k < FB; k += 4) {
    float4 b[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) b[e] = ld4(B + (k + e) * FLD + tx * 4);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float4 p = ld4(P + (ty + 8 * i) * FLP + k);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        acc[i][0] = fmaf(comp(p, e), b[e].x, acc[i][0]);
        acc[i][1] = fmaf(comp(p, e), b[e].y, acc[i][1]);
        acc[i][2] = fmaf(comp(p, e), b[e].z, acc[i][2]);
        acc[i][3] = fmaf(comp(p, e), b[e].w, acc[i][3]);
      }
    }
  }
}

__device__ __forceinline__ const float* f32_head(const SafTensor& t, int b, int h) {
  return reinterpret_cast<const float*>(t.ptr) + (int64_t)b * t.stride[0] + (int64_t)h * t.stride[1];
}
__device__ __forceinline__ void f32_store(const SafTensor& t, int b, int h, int row, int tx, const float (&v)[4], float f) {
  float* p = reinterpret_cast<float*>(t.ptr) + (int64_t)b * t.stride[0] + (int64_t)h * t.stride[1] + (int64_t)row * t.stride[2];
  *reinterpret_cast<float4*>(p + tx * 4) = make_float4(v[0] * f, v[1] * f, v[2] * f, v[3] * f);
}

// grid (B * H, row tiles): the longest tiles of all heads first
__global__ void __launch_bounds__(FNT, 3) f32_fwd_kernel(const __grid_constant__ SafMixedAttnArgs a) {
  extern __shared__ __align__(16) float f32_smem[];
  const HeadIdx hx = head_index(a, blockIdx.x);
  if (hx.state != SAF_LIVE) return;
  const int mt = gridDim.y - 1 - blockIdx.y, i0 = mt * FB, T = a.T;
  float *Qs = f32_smem, *Ks = Qs + TILE_F, *Vs = Ks + TILE_F, *Ps = Vs + TILE_F;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const float *qb = f32_head(a.q, hx.b, hx.hq), *kb = f32_head(a.k, hx.b, hx.hk), *vb = f32_head(a.v, hx.b, hx.hv);
  f32_tile(Qs, qb, a.q.stride[2], i0, T);
  f32_tile(Ks, kb, a.k.stride[2], 0, T);
  cp_async_commit();
  f32_tile(Vs, vb, a.v.stride[2], 0, T);
  cp_async_commit();
  float acc[8][4], m[8], l[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[i][c] = 0.f;
  }
  const float scale = a.sm_scale * F_LOG2E;
  for (int jt = 0; jt <= mt; ++jt) {
    const int j0 = jt * FB;
    cp_async_wait<1>();                       // Q, K of this tile; V may still be on its way
    __syncthreads();
    float s[8][4];
    f32_dot(Qs, Ks, ty, tx, s);
    __syncthreads();                          // K is read
    if (jt < mt) f32_tile(Ks, kb, a.k.stride[2], j0 + FB, T);
    cp_async_commit();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = ty + 8 * i;
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const bool ok = jt < mt || (tx + 16 * j <= r && j0 + tx + 16 * j < T);
        s[i][j] = ok ? s[i][j] * scale : -INFINITY;
        mx = fmaxf(mx, s[i][j]);
      }
#pragma unroll
      for (int off = 8; off; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
      const float m_new = fmaxf(m[i], mx), m_safe = (m_new == -INFINITY) ? 0.f : m_new;
      const float f = (m[i] == -INFINITY) ? 0.f : exp2f(m[i] - m_safe);
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float p = exp2f(s[i][j] - m_safe);
        Ps[r * FLP + tx + 16 * j] = p;
        sum += p;
      }
      l[i] = l[i] * f + sum;                  // this thread's columns; added over the row at the end
      m[i] = m_new;
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[i][c] *= f;
    }
    cp_async_wait<1>();                       // V of this tile; the next K may still be on its way
    __syncthreads();
    f32_acc(Ps, Vs, ty, tx, acc);
    __syncthreads();                          // V is read
    if (jt < mt) f32_tile(Vs, vb, a.v.stride[2], j0 + FB, T);
    cp_async_commit();
  }
  cp_async_wait<0>();
#pragma unroll
  for (int i = 0; i < 8; ++i) {
#pragma unroll
    for (int off = 8; off; off >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], off);
    const int t = i0 + ty + 8 * i;
    if (t >= T) continue;
    const float ls = l[i] == 0.f ? 1.f : l[i];
    f32_store(a.out, hx.b, hx.h, t, tx, acc[i], 1.f / ls);
    if (a.lse.ptr && tx == 0)
      reinterpret_cast<float*>(a.lse.ptr)[(int64_t)hx.b * a.lse.stride[0] + (int64_t)hx.h * a.lse.stride[1] + (int64_t)t * a.lse.stride[2]] =
          ((m[i] == -INFINITY) ? 0.f : m[i]) + log2f(ls);
  }
}

__global__ void __launch_bounds__(FNT, 2) f32_dkdv_kernel(const __grid_constant__ SafMixedAttnBwdArgs g) {
  extern __shared__ __align__(16) float f32_smem[];
  const SafMixedAttnArgs& a = g.fwd;
  const HeadIdx hx = head_index(a, blockIdx.x);
  if (hx.state != SAF_LIVE) return;
  const int j0 = blockIdx.y * FB, T = a.T;
  float *Ks = f32_smem, *Vs = Ks + TILE_F, *Qs = Vs + TILE_F, *Ds = Qs + TILE_F, *Pt = Ds + TILE_F, *St = Pt + PROB_F;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const float *qb = f32_head(a.q, hx.b, hx.hq), *dob = f32_head(g.dout, hx.b, hx.h);
  f32_tile(Ks, f32_head(a.k, hx.b, hx.hk), a.k.stride[2], j0, T);
  f32_tile(Vs, f32_head(a.v, hx.b, hx.hv), a.v.stride[2], j0, T);
  float dk[8][4], dv[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int c = 0; c < 4; ++c) dk[i][c] = dv[i][c] = 0.f;
  const float scale = a.sm_scale * F_LOG2E;
  const float* lse = f32_head(a.lse, hx.b, hx.h);
  const float* del = f32_head(g.delta, hx.b, hx.h);
  for (int i0 = j0; i0 < T; i0 += FB) {
    f32_tile(Qs, qb, a.q.stride[2], i0, T);
    f32_tile(Ds, dob, g.dout.stride[2], i0, T);
    cp_async_commit();
    float L[4], dl[4];                        // of query rows tx + 16 j
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int q = i0 + tx + 16 * j;
      L[j] = q < T ? lse[(int64_t)q * a.lse.stride[2]] : 0.f;
      dl[j] = q < T ? del[(int64_t)q * g.delta.stride[2]] : 0.f;
    }
    cp_async_wait<0>();
    __syncthreads();
    float s[8][4], dp[8][4];
    f32_dot(Ks, Qs, ty, tx, s);
    f32_dot(Vs, Ds, ty, tx, dp);
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = ty + 8 * i, r = tx + 16 * j;
        float p = 0.f, ds = 0.f;
        if (i0 + r < T && j0 + c <= i0 + r) {
          p = exp2f(s[i][j] * scale - L[j]);
          ds = p * (dp[i][j] - dl[j]) * a.sm_scale;
        }
        Pt[c * FLP + r] = p;
        St[c * FLP + r] = ds;
      }
    __syncwarp();
    f32_acc(Pt, Ds, ty, tx, dv);
    f32_acc(St, Qs, ty, tx, dk);
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int t = j0 + ty + 8 * i;
    if (t >= T) continue;
    f32_store(g.dv, hx.b, hx.hv, t, tx, dv[i], 1.f);
    f32_store(g.dk, hx.b, hx.hk, t, tx, dk[i], 1.f);
  }
}

__global__ void __launch_bounds__(FNT, 2) f32_dq_kernel(const __grid_constant__ SafMixedAttnBwdArgs g) {
  extern __shared__ __align__(16) float f32_smem[];
  const SafMixedAttnArgs& a = g.fwd;
  const HeadIdx hx = head_index(a, blockIdx.x);
  if (hx.state != SAF_LIVE) return;
  const int mt = gridDim.y - 1 - blockIdx.y, i0 = mt * FB, T = a.T;
  float *Qs = f32_smem, *Ds = Qs + TILE_F, *Ks = Ds + TILE_F, *Vs = Ks + TILE_F, *Ss = Vs + TILE_F;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const float *kb = f32_head(a.k, hx.b, hx.hk), *vb = f32_head(a.v, hx.b, hx.hv);
  f32_tile(Qs, f32_head(a.q, hx.b, hx.hq), a.q.stride[2], i0, T);
  f32_tile(Ds, f32_head(g.dout, hx.b, hx.h), g.dout.stride[2], i0, T);
  float dq[8][4], L[8], dl[8];
  const float* lse = f32_head(a.lse, hx.b, hx.h);
  const float* del = f32_head(g.delta, hx.b, hx.h);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int q = i0 + ty + 8 * i;
    L[i] = q < T ? lse[(int64_t)q * a.lse.stride[2]] : 0.f;
    dl[i] = q < T ? del[(int64_t)q * g.delta.stride[2]] : 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) dq[i][c] = 0.f;
  }
  const float scale = a.sm_scale * F_LOG2E;
  for (int jt = 0; jt <= mt; ++jt) {
    const int j0 = jt * FB;
    f32_tile(Ks, kb, a.k.stride[2], j0, T);
    f32_tile(Vs, vb, a.v.stride[2], j0, T);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    float s[8][4], dp[8][4];
    f32_dot(Qs, Ks, ty, tx, s);
    f32_dot(Ds, Vs, ty, tx, dp);
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int r = ty + 8 * i, c = tx + 16 * j;
        float ds = 0.f;
        if (i0 + r < T && j0 + c <= i0 + r) ds = exp2f(s[i][j] * scale - L[i]) * (dp[i][j] - dl[i]) * a.sm_scale;
        Ss[r * FLP + c] = ds;
      }
    __syncwarp();
    f32_acc(Ss, Ks, ty, tx, dq);
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (i0 + ty + 8 * i < T) f32_store(g.dq, hx.b, hx.hq, i0 + ty + 8 * i, tx, dq[i], 1.f);
}

// 16-byte rows: base, row, head and batch strides (an axis of one element is never stepped over)
bool f32_rows_ok(const SafTensor& t, int B, int Hn, int T) {
  return t.ptr && ((uintptr_t)t.ptr & 15) == 0 && t.stride[3] == 1 && (B < 2 || t.stride[0] % 4 == 0) && (Hn < 2 || t.stride[1] % 4 == 0) &&
         (T < 2 || t.stride[2] % 4 == 0);
}

bool f32_call_ok(const SafMixedAttnArgs& a) {
  const int kv = a.HKV > 0 ? a.HKV : 0;
  // (grid.y holds the row tiles)
  return a.dtype == SAF_F32 && a.HD == FHD && !a.rope && a.U > 0 && a.T <= 65535 * FB && f32_rows_ok(a.q, a.B, a.U, a.T) &&
         f32_rows_ok(a.k, a.B, kv ? kv : a.U, a.T) && f32_rows_ok(a.v, a.B, kv ? kv : a.H, a.T) && f32_rows_ok(a.out, a.B, a.H, a.T);
}

}  // namespace

// The live heads of an fp32 call whose rows are whole 16-byte pieces and come rotated already; everything else stays
// with the any-type kernels.
int launch_attn_f32_fwd(const SafMixedAttnArgs& a, cudaStream_t st) {
  if (!f32_call_ok(a)) return SAF_ERR_UNSUPPORTED;
  constexpr int smem = (3 * TILE_F + PROB_F) * 4;
  static PerDeviceOnce once;
  if (int rc = ensure_dyn_smem(f32_fwd_kernel, smem, once)) return rc;
  f32_fwd_kernel<<<dim3(a.B * a.H, (a.T + FB - 1) / FB), FNT, smem, st>>>(a);
  count_launch();
  return check_launch("f32_fwd_kernel");
}

// dK, dV and dQ; delta is filled already
int launch_attn_f32_bwd(const SafMixedAttnBwdArgs& g, cudaStream_t st) {
  const SafMixedAttnArgs& a = g.fwd;
  if (!f32_call_ok(a) || a.HKV > 0 || !f32_rows_ok(g.dout, a.B, a.H, a.T) || !f32_rows_ok(g.dv, a.B, a.H, a.T) ||
      !f32_rows_ok(g.dq, a.B, a.U, a.T) || !f32_rows_ok(g.dk, a.B, a.U, a.T))
    return SAF_ERR_UNSUPPORTED;
  const dim3 grid(a.B * a.H, (a.T + FB - 1) / FB);
  constexpr int smem_kv = (4 * TILE_F + 2 * PROB_F) * 4, smem_q = (4 * TILE_F + PROB_F) * 4;
  static PerDeviceOnce once_kv, once_q;
  if (int rc = ensure_dyn_smem(f32_dkdv_kernel, smem_kv, once_kv)) return rc;
  if (int rc = ensure_dyn_smem(f32_dq_kernel, smem_q, once_q)) return rc;
  f32_dkdv_kernel<<<grid, FNT, smem_kv, st>>>(g);
  count_launch();
  if (int rc = check_launch("f32_dkdv_kernel")) return rc;
  f32_dq_kernel<<<grid, FNT, smem_q, st>>>(g);
  count_launch();
  return check_launch("f32_dq_kernel");
}

}  // namespace saf
