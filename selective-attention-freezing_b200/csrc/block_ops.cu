// LayerNorm of the transformer block around the attention path (LayerNorm.forward, nanogpt/model.py:45-54):
// y = (x - mean) / sqrt(var + eps) * weight (+ bias), statistics in fp32, biased variance as F.layer_norm.
// rms = 1 gives the RMSNorm of the Qwen-shaped blocks instead (the norm the reference's grouped-query adapter
// leaves to the Hugging Face model, qwen/nanogpt/hybrid_prior_attention.py:522-523): no mean, no bias,
// y = x / sqrt(mean(x^2) + eps) * weight.
// HBM-bound: one warp per row, 16-byte loads, the row stays in registers between the two passes.
#include "saf_internal.h"
#include "sm100_prims.cuh"

namespace saf {
namespace {

constexpr int LN_WARPS = 8;
constexpr int LN_MAX_CHUNKS = 8;   // 16-byte chunks per lane held in registers: C <= 2048 on the vector path
// (the kernel is compiled per chunk count: with room for 8 chunks a 768-wide row held a third of its registers and
// the SM a third of the loads in flight)

__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    f[2 * e] = __uint_as_float(w[e] << 16);
    f[2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u);
  }
}

template <int NC>
__global__ void __launch_bounds__(LN_WARPS * 32) layernorm_bf16_kernel(const __nv_bfloat16* __restrict__ x, int64_t ldx,
                                                                       const __nv_bfloat16* __restrict__ w,
                                                                       const __nv_bfloat16* __restrict__ b,
                                                                       __nv_bfloat16* __restrict__ out, int64_t ldo, int M,
                                                                       int C, float eps, int rms) {
  const int row = blockIdx.x * LN_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  pdl_wait();
  pdl_trigger();
  if (row >= M) return;
  const int n_chunks = C >> 3;                     // 8 elements each
  const uint4* xr = reinterpret_cast<const uint4*>(x + (int64_t)row * ldx);
  float v[NC][8];
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < NC; ++k) {
    const int c = lane + 32 * k;
    if (c < n_chunks) {
      unpack8(xr[c], v[k]);
#pragma unroll
      for (int e = 0; e < 8; ++e) s += v[k][e];
    }
  }
#pragma unroll
  for (int off = 16; off; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  const float mean = rms ? 0.f : s / (float)C;
  float q = 0.f;
#pragma unroll
  for (int k = 0; k < NC; ++k) {
    if (lane + 32 * k < n_chunks) {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float d = v[k][e] - mean;
        q = fmaf(d, d, q);
      }
    }
  }
#pragma unroll
  for (int off = 16; off; off >>= 1) q += __shfl_xor_sync(0xffffffffu, q, off);
  const float rstd = rsqrtf(q / (float)C + eps);
  const uint4* wr = reinterpret_cast<const uint4*>(w);
  const uint4* br = reinterpret_cast<const uint4*>(b);
  uint4* orow = reinterpret_cast<uint4*>(out + (int64_t)row * ldo);
#pragma unroll
  for (int k = 0; k < NC; ++k) {
    const int c = lane + 32 * k;
    if (c < n_chunks) {
      float wv[8], bv[8];
      unpack8(wr[c], wv);
      if (b) unpack8(br[c], bv);
      uint32_t o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float y0 = (v[k][2 * e] - mean) * rstd * wv[2 * e], y1 = (v[k][2 * e + 1] - mean) * rstd * wv[2 * e + 1];
        if (b) {
          y0 += bv[2 * e];
          y1 += bv[2 * e + 1];
        }
        const __nv_bfloat162 h2 = __floats2bfloat162_rn(y0, y1);
        o[e] = *reinterpret_cast<const uint32_t*>(&h2);
      }
      orow[c] = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
}

// any dtype / width / alignment: one warp per row, three passes over the row
template <typename T>
__global__ void __launch_bounds__(LN_WARPS * 32) layernorm_generic_kernel(const T* __restrict__ x, int64_t ldx,
                                                                          const T* __restrict__ w, const T* __restrict__ b,
                                                                          T* __restrict__ out, int64_t ldo, int M, int C,
                                                                          float eps, int rms) {
  const int row = blockIdx.x * LN_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  pdl_wait();
  pdl_trigger();
  if (row >= M) return;
  const T* xr = x + (int64_t)row * ldx;
  float s = 0.f;
  for (int c = lane; c < C; c += 32) s += to_f<T>(xr[c]);
#pragma unroll
  for (int off = 16; off; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  const float mean = rms ? 0.f : s / (float)C;
  float q = 0.f;
  for (int c = lane; c < C; c += 32) {
    const float d = to_f<T>(xr[c]) - mean;
    q = fmaf(d, d, q);
  }
#pragma unroll
  for (int off = 16; off; off >>= 1) q += __shfl_xor_sync(0xffffffffu, q, off);
  const float rstd = rsqrtf(q / (float)C + eps);
  T* orow = out + (int64_t)row * ldo;
  for (int c = lane; c < C; c += 32) {
    float y = (to_f<T>(xr[c]) - mean) * rstd * to_f<T>(w[c]);
    if (b) y += to_f<T>(b[c]);
    orow[c] = from_f<T>(y);
  }
}

// fp32 -> bf16 of several arrays in one launch: the residual stream and the master weights of a training layer enter
// the tensor-core products this way once per pass.  Memory-bound: 32 bytes in and 16 out per thread and step.
constexpr int CAST_THREADS = 256, CAST_STEPS = 4;
constexpr int64_t CAST_BLOCK = (int64_t)CAST_THREADS * CAST_STEPS * 8;    // elements of one block
struct CastParams {
  CastSegment seg[MAX_CAST_SEGMENTS];
  unsigned block0[MAX_CAST_SEGMENTS + 1];
  int n;
};

__global__ void __launch_bounds__(CAST_THREADS) cast_bf16_kernel(const __grid_constant__ CastParams p) {
  pdl_wait();
  pdl_trigger();
  int s = 0;
  while (s + 1 < p.n && blockIdx.x >= p.block0[s + 1]) ++s;
  const float4* src = reinterpret_cast<const float4*>(p.seg[s].src);
  uint4* dst = reinterpret_cast<uint4*>(p.seg[s].dst);
  const int64_t n8 = p.seg[s].n >> 3;
  const int64_t i0 = (int64_t)(blockIdx.x - p.block0[s]) * (CAST_BLOCK / 8) + threadIdx.x;
  float4 a[CAST_STEPS], b[CAST_STEPS];
#pragma unroll
  for (int k = 0; k < CAST_STEPS; ++k) {
    const int64_t i = i0 + k * CAST_THREADS;
    if (i < n8) {
      a[k] = __ldcs(src + 2 * i);
      b[k] = __ldcs(src + 2 * i + 1);
    }
  }
#pragma unroll
  for (int k = 0; k < CAST_STEPS; ++k) {
    const int64_t i = i0 + k * CAST_THREADS;
    if (i < n8) {
      const __nv_bfloat162 w[4] = {__floats2bfloat162_rn(a[k].x, a[k].y), __floats2bfloat162_rn(a[k].z, a[k].w),
                                   __floats2bfloat162_rn(b[k].x, b[k].y), __floats2bfloat162_rn(b[k].z, b[k].w)};
      dst[i] = *reinterpret_cast<const uint4*>(w);
    }
  }
}

bool ln_al16(const void* p) { return ((uintptr_t)p & 15) == 0; }

}  // namespace

int launch_cast_bf16(const CastSegment* seg, int n, cudaStream_t st) {
  CastParams p;
  memset(&p, 0, sizeof(p));
  p.n = n;
  unsigned blocks = 0;
  for (int i = 0; i < n; ++i) {
    p.seg[i] = seg[i];
    p.block0[i] = blocks;
    blocks += (unsigned)((seg[i].n + CAST_BLOCK - 1) / CAST_BLOCK);
  }
  p.block0[n] = blocks;
  if (!blocks) return SAF_OK;
  return launch_pdl("cast_bf16_kernel", cast_bf16_kernel, dim3(blocks), CAST_THREADS, 0, st, 1, p);
}

int launch_layernorm(const void* x, int64_t ldx, const void* w, const void* b, void* out, int64_t ldo, int M, int C,
                     float eps, int dtype, int rms, cudaStream_t st) {
  const unsigned grid = (unsigned)((M + LN_WARPS - 1) / LN_WARPS);
  if (dtype == SAF_BF16) {
    const bool vec = C % 8 == 0 && C <= 256 * LN_MAX_CHUNKS && ldx % 8 == 0 && ldo % 8 == 0 && ln_al16(x) && ln_al16(w) &&
                     ln_al16(out) && (!b || ln_al16(b));
    if (vec) {
      const auto xb = reinterpret_cast<const __nv_bfloat16*>(x), wb = reinterpret_cast<const __nv_bfloat16*>(w),
                 bb = reinterpret_cast<const __nv_bfloat16*>(b);
      const auto ob = reinterpret_cast<__nv_bfloat16*>(out);
      auto go = [&](auto kernel) {
        return launch_pdl("layernorm_kernel", kernel, dim3(grid), LN_WARPS * 32, 0, st, 1, xb, ldx, wb, bb, ob, ldo, M, C, eps, rms);
      };
      switch ((C + 255) / 256) {
        case 1: return go(layernorm_bf16_kernel<1>);
        case 2: return go(layernorm_bf16_kernel<2>);
        case 3: return go(layernorm_bf16_kernel<3>);
        case 4: return go(layernorm_bf16_kernel<4>);
        case 5: case 6: return go(layernorm_bf16_kernel<6>);
        default: return go(layernorm_bf16_kernel<LN_MAX_CHUNKS>);
      }
    }
    return launch_pdl("layernorm_kernel", layernorm_generic_kernel<__nv_bfloat16>, dim3(grid), LN_WARPS * 32, 0, st, 1,
                      reinterpret_cast<const __nv_bfloat16*>(x), ldx, reinterpret_cast<const __nv_bfloat16*>(w),
                      reinterpret_cast<const __nv_bfloat16*>(b), reinterpret_cast<__nv_bfloat16*>(out), ldo, M, C, eps, rms);
  }
  return launch_pdl("layernorm_kernel", layernorm_generic_kernel<float>, dim3(grid), LN_WARPS * 32, 0, st, 1,
                    reinterpret_cast<const float*>(x), ldx, reinterpret_cast<const float*>(w), reinterpret_cast<const float*>(b),
                    reinterpret_cast<float*>(out), ldo, M, C, eps, rms);
}

}  // namespace saf
