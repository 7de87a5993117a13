// The attention layer as one call per direction: projection of live heads, mixed attention, output projection.
//
// A layer is three GEMM-or-attention launches at inference and about a dozen in training.  Issued one by one from the
// host language, every launch pays for an argument struct, an allocation and an autograd node of its own, and the
// pieces talk through whatever layout each of them likes best: gradients of q and k as separate tensors that are
// zero-filled, sliced and added, v in a third, weights and activations converted one by one.  Here the whole sequence
// is composed natively over ONE workspace the caller owns, and all of it works on the projection's own layout,
// rows of [Q live | K live | V all] (grouped-query: [Q live | K kv | V kv]):
//
//   forward   [fp32 -> bf16 of x and the four weights]  QKV GEMM (+bias, RoPE)  mixed attention  output GEMM (+residual)
//   backward  dY = dout Wo, dWo;  dQ, dK, dV of the attention written into one buffer of that layout;  adjoint RoPE of
//             its Q and K slabs;  dx = d[QKV] W and dW = d[QKV]^T x as ONE product each, fp32 when the tensor is fp32
//
// In fp32 (all tensors fp32) the same sequence with the fp32 products and attention: nothing is converted, the rotation is a
// launch of its own, dW goes straight to the gradients.
// (nanogpt/model.py:946-1077, the cheap path of the reference's module.)  Measured on a B200, forward and backward of one
// training layer under bf16 autocast: 12 x 64, T = 1024, B = 8 1.2-1.5 ms (41 launches, host-bound) -> 0.30 ms (14
// launches); 16 x 128, T = 8192, B = 2 4.16 -> 3.36 ms (0.8 ms of it were fills, copies, conversions and additions);
// one inference layer of 4 x 64, T = 512, B = 2 163 -> 41 us.
#include <string.h>

#include <algorithm>

#include "saf_internal.h"

namespace saf {
namespace {

constexpr int LAYER_MAX_HEADS = 256;
constexpr int LAYER_MAX_SLABS = 3 * LAYER_MAX_HEADS;     // of one product: heads of Q, K and V, or 64-row blocks of C
constexpr int MLP_MAX_BLOCKS = 1024;

int64_t up(int64_t n) { return (n + 255) & ~(int64_t)255; }

// workspace of the forward, kept until the backward; and the backward's own
struct FwdLayout {
  int64_t sched, x, w[4], qkv, y, lse, total;
};
struct BwdLayout {
  int64_t dy, dqkv, delta, dw, total;
};

struct Dims {
  int B, T, H, U, HD, C, kv, D;     // kv: heads of the K part (V: H or HKV); D: width of the attention output
  int n_q, n_k, n_v;                // heads of the three parts of the projection
  int es;                           // bytes of an element of the computation: 2, or 4 in fp32
  int64_t tok;
  int width() const { return (n_q + n_k + n_v) * HD; }
};

Dims dims_of(const SafAttnLayerArgs& a) {
  Dims d;
  d.B = a.attn.B; d.T = a.attn.T; d.H = a.attn.H; d.U = a.attn.U; d.HD = a.attn.HD; d.C = a.C;
  d.n_q = d.U;
  d.n_k = a.attn.HKV > 0 ? a.attn.HKV : d.U;
  d.n_v = a.attn.HKV > 0 ? a.attn.HKV : d.H;
  d.kv = d.n_k;
  d.D = d.H * d.HD;
  d.tok = (int64_t)d.B * d.T;
  d.es = dtype_size(a.attn.dtype);
  return d;
}

// rows and columns of weight i (q, k, v, o)
void weight_shape(const SafAttnLayerArgs& a, const Dims& d, int i, int* rows, int* cols) {
  const int kv = a.attn.HKV > 0 ? a.attn.HKV : d.H;
  *rows = i == 0 ? d.D : (i == 3 ? d.C : kv * d.HD);
  *cols = i == 3 ? d.D : d.C;
}

FwdLayout fwd_layout(const SafAttnLayerArgs& a, const Dims& d) {
  FwdLayout l;
  int64_t at = 256;
  l.sched = 0;
  l.x = at;
  if (a.x_dtype != a.attn.dtype) at += up(d.tok * d.C * 2);
  for (int i = 0; i < 4; ++i) {
    int r, c;
    weight_shape(a, d, i, &r, &c);
    l.w[i] = at;
    if (a.w_dtype != a.attn.dtype) at += up((int64_t)r * c * 2);
  }
  l.qkv = at;
  at += up(d.tok * d.width() * d.es);
  l.y = at;
  at += up(d.tok * d.D * d.es);
  l.lse = at;
  if (a.train) at += up((int64_t)d.B * d.H * d.T * 4);
  l.total = at;
  return l;
}

BwdLayout bwd_layout(const SafAttnLayerArgs& a, const Dims& d) {
  BwdLayout l;
  int64_t at = 0;
  l.dy = at;
  at += up(d.tok * d.D * d.es);
  l.dqkv = at;
  at += up(d.tok * d.width() * d.es);
  l.delta = at;
  at += up((int64_t)d.B * d.H * d.T * 4);
  l.dw = at;                         // the output projection's product is finished before the other one starts
  if (d.es == 2) at += up(std::max(gemm_dw_workspace_bytes(d.C, d.D, (int)d.tok), gemm_dw_workspace_bytes(d.width(), d.C, (int)d.tok)));
  l.total = at;
  return l;
}

int validate_layer(const SafAttnLayerArgs* a) {
  if (!a) return fail(SAF_ERR_INVALID, "null argument struct");
  if (a->struct_size != (int32_t)sizeof(SafAttnLayerArgs))
    return fail(SAF_ERR_INVALID, "SafAttnLayerArgs size mismatch: caller %d, library %d", a->struct_size,
                (int)sizeof(SafAttnLayerArgs));
  const SafMixedAttnArgs& t = a->attn;
  if (t.struct_size != (int32_t)sizeof(SafMixedAttnArgs)) return fail(SAF_ERR_INVALID, "SafMixedAttnArgs size mismatch");
  if (t.dtype != SAF_BF16 && (t.dtype != SAF_F32 || a->x_dtype != SAF_F32 || a->w_dtype != SAF_F32))
    return fail(SAF_ERR_UNSUPPORTED, "the layer entry computes in bf16, or in fp32 from fp32 tensors");
  if (t.B <= 0 || t.T <= 0 || t.H <= 0 || t.U < 0 || t.U > t.H || t.HD <= 0 || a->C <= 0 || t.HKV < 0)
    return fail(SAF_ERR_INVALID, "bad dimension");
  if (t.H > LAYER_MAX_HEADS || t.HKV > LAYER_MAX_HEADS) return fail(SAF_ERR_LIMIT, "more than %d heads", LAYER_MAX_HEADS);
  if (a->C > LAYER_MAX_SLABS * 64) return fail(SAF_ERR_LIMIT, "width %d exceeds the limit of %d", a->C, LAYER_MAX_SLABS * 64);
  if (t.HD % 32 || t.HD > 128 || a->C % 8) return fail(SAF_ERR_UNSUPPORTED, "head_dim %d, width %d", t.HD, a->C);
  if (t.rope || t.force_state >= 0) return fail(SAF_ERR_INVALID, "rope and force_state belong to the attention entry");
  if (!t.frozen || !t.frozen_host) return fail(SAF_ERR_INVALID, "frozen and frozen_host must be non-null");
  if (t.U > 0 && !a->live) return fail(SAF_ERR_INVALID, "live must be non-null");
  for (int i = 0; i < t.U; ++i)
    if (a->live[i] < 0 || a->live[i] >= t.H) return fail(SAF_ERR_INVALID, "live[%d] = %d", i, a->live[i]);
  if ((a->x_dtype != SAF_BF16 && a->x_dtype != SAF_F32) || (a->w_dtype != SAF_BF16 && a->w_dtype != SAF_F32))
    return fail(SAF_ERR_UNSUPPORTED, "x and the weights are fp32 or bf16");
  if (a->train && t.HKV > 0) return fail(SAF_ERR_UNSUPPORTED, "grouped-query attention has no backward");
  if ((a->rope_cos == nullptr) != (a->rope_sin == nullptr)) return fail(SAF_ERR_INVALID, "rope_cos and rope_sin come together");
  if ((int64_t)t.B * t.T > 0x7fffffff) return fail(SAF_ERR_LIMIT, "B * T");
  return SAF_OK;
}

// (B, heads, T, hd) inside token rows of ld elements of es bytes
SafTensor rows_view(void* base, int64_t first_col, int64_t ld, int T, int hd, int es) {
  SafTensor v;
  v.ptr = reinterpret_cast<uint8_t*>(base) + first_col * es;
  v.stride[0] = (int64_t)T * ld;
  v.stride[1] = hd;
  v.stride[2] = ld;
  v.stride[3] = 1;
  return v;
}

struct Slabs {
  int32_t weight[LAYER_MAX_SLABS], row0[LAYER_MAX_SLABS], rope[LAYER_MAX_SLABS];
  int n;
};
void qkv_slabs(const SafAttnLayerArgs& a, const Dims& d, Slabs* s) {
  int n = 0;
  for (int i = 0; i < d.n_q; ++i, ++n) { s->weight[n] = 0; s->row0[n] = a.live[i] * d.HD; s->rope[n] = 1; }
  for (int i = 0; i < d.n_k; ++i, ++n) { s->weight[n] = 1; s->row0[n] = (a.attn.HKV > 0 ? i : a.live[i]) * d.HD; s->rope[n] = 1; }
  for (int i = 0; i < d.n_v; ++i, ++n) { s->weight[n] = 2; s->row0[n] = i * d.HD; s->rope[n] = 0; }
  s->n = n;
}

// the weights as the products read them: converted copies in the workspace, or the caller's own
const void* weight_ptr(const SafAttnLayerArgs& a, const FwdLayout& l, int i) {
  if (a.w_dtype != a.attn.dtype) return reinterpret_cast<const uint8_t*>(a.work) + l.w[i];
  const void* w[4] = {a.wq, a.wk, a.wv, a.wo};
  return w[i];
}

// out projection / QKV projection as indexed-linear calls
void fill_linear(const SafAttnLayerArgs& a, const Dims& d, const FwdLayout& l, bool out_proj, Slabs* s, SafIndexedLinearArgs* g) {
  memset(g, 0, sizeof(*g));
  g->struct_size = (int32_t)sizeof(*g);
  g->dtype = a.attn.dtype;
  g->M = (int)d.tok;
  g->status = a.attn.status;
  uint8_t* work = reinterpret_cast<uint8_t*>(a.work);
  if (out_proj) {
    g->x = work + l.y;
    g->ldx = d.D;
    g->C = d.D;
    g->n_weights = 1;
    // whole matrix: 64-row blocks where the width allows, else one slab
    g->slab = d.C % 64 == 0 ? 64 : d.C;
    s->n = d.C / g->slab;
    for (int i = 0; i < s->n; ++i) { s->weight[i] = 0; s->row0[i] = i * g->slab; }
    g->weights[0] = weight_ptr(a, l, 3);
    g->biases[0] = a.bo;
    g->ldw[0] = d.D;
    g->rows_w[0] = d.C;
  } else {
    const bool converted = a.x_dtype != a.attn.dtype;
    g->x = converted ? work + l.x : a.x;
    g->ldx = converted ? d.C : a.ldx;
    g->C = d.C;
    g->n_weights = 3;
    g->slab = d.HD;
    qkv_slabs(a, d, s);
    const void* b[3] = {a.bq, a.bk, a.bv};
    for (int i = 0; i < 3; ++i) {
      int r, c;
      weight_shape(a, d, i, &r, &c);
      g->weights[i] = weight_ptr(a, l, i);
      g->biases[i] = b[i];
      g->ldw[i] = c;
      g->rows_w[i] = r;
    }
  }
  g->n_slabs = s->n;
  g->slab_weight = s->weight;
  g->slab_row0 = s->row0;
}

void attn_views(const SafAttnLayerArgs& a, const Dims& d, const FwdLayout& l, SafMixedAttnArgs* t) {
  uint8_t* work = reinterpret_cast<uint8_t*>(a.work);
  *t = a.attn;
  const int64_t W = d.width();
  if (d.U > 0) {
    t->q = rows_view(work + l.qkv, 0, W, d.T, d.HD, d.es);
    t->k = rows_view(work + l.qkv, (int64_t)d.n_q * d.HD, W, d.T, d.HD, d.es);
  }
  t->v = rows_view(work + l.qkv, (int64_t)(d.n_q + d.n_k) * d.HD, W, d.T, d.HD, d.es);
  t->out = rows_view(work + l.y, 0, d.D, d.T, d.HD, d.es);
  memset(&t->lse, 0, sizeof(t->lse));
  if (a.train) {
    t->lse.ptr = work + l.lse;
    t->lse.stride[0] = (int64_t)d.H * d.T;
    t->lse.stride[1] = d.T;
    t->lse.stride[2] = 1;
  }
  t->sched = d.U > 0 && d.es == 2 ? reinterpret_cast<int32_t*>(work + l.sched) : nullptr;
}

}  // namespace
}  // namespace saf

using namespace saf;

extern "C" {

int saf_attn_layer_workspace(const SafAttnLayerArgs* args, int64_t* out) {
  int rc = validate_layer(args);
  if (rc) return rc;
  if (!out) return fail(SAF_ERR_INVALID, "null pointer");
  const Dims d = dims_of(*args);
  const FwdLayout l = fwd_layout(*args, d);
  out[0] = l.total;
  out[1] = args->train ? bwd_layout(*args, d).total : 0;
  out[2] = l.qkv;
  out[3] = l.y;
  return SAF_OK;
}

int saf_attn_layer_fwd(const SafAttnLayerArgs* args, void* stream) {
  int rc = validate_layer(args);
  if (rc) return rc;
  const SafAttnLayerArgs& a = *args;
  const Dims d = dims_of(a);
  const FwdLayout l = fwd_layout(a, d);
  if (!a.x || !a.wq || !a.wk || !a.wv || !a.wo || !a.out || !a.work) return fail(SAF_ERR_INVALID, "null pointer");
  if (((uintptr_t)a.work & 255) || a.work_bytes < l.total) return fail(SAF_ERR_INVALID, "workspace too small or not aligned to 256 bytes");
  SafMixedAttnArgs t;
  attn_views(a, d, l, &t);
  if ((rc = validate_mixed_args(&t))) return rc;
  Slabs s, so;
  SafIndexedLinearArgs g, go;
  fill_linear(a, d, l, false, &s, &g);
  fill_linear(a, d, l, true, &so, &go);
  if (a.rope_cos) {
    g.slab_rope = s.rope;
    g.rope_cos = a.rope_cos;
    g.rope_sin = a.rope_sin;
    g.T = d.T;
  }
  if ((rc = validate_linear_args(&g)) || (rc = validate_linear_args(&go))) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  uint8_t* work = reinterpret_cast<uint8_t*>(a.work);
  CastSegment seg[MAX_CAST_SEGMENTS];
  int ns = 0;
  if (a.x_dtype == SAF_F32 && a.ldx != d.C) return fail(SAF_ERR_INVALID, "an fp32 x must be contiguous");
  if (d.es == 4 && a.residual) return fail(SAF_ERR_UNSUPPORTED, "the fp32 layer adds no residual");
  if (a.x_dtype != a.attn.dtype) {
    seg[ns++] = {reinterpret_cast<const float*>(a.x), work + l.x, d.tok * d.C};
  }
  if (a.w_dtype != a.attn.dtype) {
    const void* w[4] = {a.wq, a.wk, a.wv, a.wo};
    for (int i = 0; i < 4; ++i) {
      int r, c;
      weight_shape(a, d, i, &r, &c);
      seg[ns++] = {reinterpret_cast<const float*>(w[i]), work + l.w[i], (int64_t)r * c};
    }
  }
  for (int i = 0; i < ns; ++i)
    if (((uintptr_t)seg[i].src & 15) || seg[i].n % 8) return fail(SAF_ERR_INVALID, "fp32 tensors must be 16-byte aligned");
  if (ns && (rc = launch_cast_bf16(seg, ns, st))) return rc;
  g.out = work + l.qkv;
  g.ldo = d.width();
  // the projection also clears the attention launch's tile queue
  rc = launch_gemm_sm100(g, st, t.sched, a.w_dtype == SAF_BF16 && a.after_library_launch);
  if (rc == SAF_ERR_UNSUPPORTED) {
    t.sched = nullptr;
    rc = saf_indexed_linear_fwd(&g, stream);
  }
  if (rc) return rc;
  if (a.event_before && cudaEventRecord((cudaEvent_t)a.event_before, st) != cudaSuccess) return fail(SAF_ERR_CUDA, "cudaEventRecord");
  if ((rc = saf_mixed_attn_fwd(&t, stream))) return rc;
  if (a.event_after && cudaEventRecord((cudaEvent_t)a.event_after, st) != cudaSuccess) return fail(SAF_ERR_CUDA, "cudaEventRecord");
  go.out = a.out;
  go.ldo = a.ldo;
  go.residual = a.residual;
  go.ldr = a.ldr;
  // The caller's weights may be loaded while the attention launch still runs: it writes none, and whatever did was complete
  // and flushed before an earlier launch of this call passed its own wait.  Copies this call made itself are not relied on
  // that way.
  rc = launch_gemm_sm100(go, st, nullptr, a.w_dtype == SAF_BF16);
  return rc == SAF_ERR_UNSUPPORTED ? saf_indexed_linear_fwd(&go, stream) : rc;
}

int saf_attn_layer_bwd(const SafAttnLayerBwdArgs* args, void* stream) {
  if (!args) return fail(SAF_ERR_INVALID, "null argument struct");
  if (args->struct_size != (int32_t)sizeof(SafAttnLayerBwdArgs))
    return fail(SAF_ERR_INVALID, "SafAttnLayerBwdArgs size mismatch: caller %d, library %d", args->struct_size,
                (int)sizeof(SafAttnLayerBwdArgs));
  int rc = validate_layer(&args->fwd);
  if (rc) return rc;
  const SafAttnLayerArgs& a = args->fwd;
  if (!a.train) return fail(SAF_ERR_INVALID, "the forward call was not made for training");
  if (a.bq || a.bk || a.bv || a.bo) return fail(SAF_ERR_UNSUPPORTED, "bias gradients belong to the separate entries");
  const Dims d = dims_of(a);
  const FwdLayout l = fwd_layout(a, d);
  const BwdLayout b = bwd_layout(a, d);
  if (!a.x || !a.work || a.work_bytes < l.total || !args->dout || !args->work || ((uintptr_t)args->work & 255) || args->work_bytes < b.total)
    return fail(SAF_ERR_INVALID, "null pointer or workspace too small");
  cudaStream_t st = (cudaStream_t)stream;
  uint8_t* bw = reinterpret_cast<uint8_t*>(args->work);
  const bool f32 = d.es == 4, w32 = a.w_dtype == SAF_F32, x32 = a.x_dtype == SAF_F32;
  float* ws = reinterpret_cast<float*>(bw + b.dw);
  const int64_t ws_bytes = b.total - b.dw;
  Slabs s, so;
  SafIndexedLinearArgs g, go;
  fill_linear(a, d, l, false, &s, &g);
  fill_linear(a, d, l, true, &so, &go);
  if ((rc = validate_linear_args(&g)) || (rc = validate_linear_args(&go))) return rc;
  // ---- output projection: dY and dWo
  rc = f32 ? launch_gemm_bwd_dx(go, args->dout, args->lddo, bw + b.dy, d.D, nullptr, st)
           : launch_gemm_bwd_dx_sm100(go, args->dout, args->lddo, bw + b.dy, d.D, nullptr, false, st);
  if (rc) return rc;
  if (args->dwo) {
    SafIndexedLinearArgs gw = go;
    gw.weights[0] = args->dwo;
    rc = f32 ? launch_gemm_bwd_dw(gw, args->dout, args->lddo, st) : launch_gemm_bwd_dw_full_sm100(gw, args->dout, args->lddo, ws, ws_bytes, w32, st);
    if (rc) return rc;
  }
  if (!args->dx && !args->dwq && !args->need_dy) return SAF_OK;
  // ---- attention: every gradient lands in one buffer of the projection's layout
  SafMixedAttnBwdArgs m;
  memset(&m, 0, sizeof(m));
  m.struct_size = (int32_t)sizeof(m);
  attn_views(a, d, l, &m.fwd);
  m.fwd.sched = nullptr;
  const int64_t W = d.width();
  m.dout = rows_view(bw + b.dy, 0, d.D, d.T, d.HD, d.es);
  if (d.U > 0) {
    m.dq = rows_view(bw + b.dqkv, 0, W, d.T, d.HD, d.es);
    m.dk = rows_view(bw + b.dqkv, (int64_t)d.n_q * d.HD, W, d.T, d.HD, d.es);
  }
  m.dv = rows_view(bw + b.dqkv, (int64_t)(d.n_q + d.n_k) * d.HD, W, d.T, d.HD, d.es);
  m.delta.ptr = bw + b.delta;
  m.delta.stride[0] = (int64_t)d.H * d.T;
  m.delta.stride[1] = d.T;
  m.delta.stride[2] = 1;
  if (!args->dx && !args->dwq) return SAF_OK;
  if ((rc = saf_mixed_attn_bwd(&m, stream))) return rc;
  if (a.rope_cos && d.U > 0 &&
      (rc = launch_rope_slabs(bw + b.dqkv, W, (int)d.tok, d.n_q + d.n_k, d.HD, d.T, nullptr, a.rope_cos, a.rope_sin, a.attn.dtype, 1, st)))
    return rc;
  // ---- projection: dx and the three weight gradients, one product each
  if (args->dx) {
    rc = f32 ? launch_gemm_bwd_dx(g, bw + b.dqkv, W, args->dx, d.C, nullptr, st)
             : launch_gemm_bwd_dx_sm100(g, bw + b.dqkv, W, args->dx, d.C, nullptr, x32, st);
    if (rc) return rc;
  }
  if (args->dwq) {
    SafIndexedLinearArgs gw = g;
    gw.weights[0] = args->dwq;
    gw.weights[1] = args->dwk;
    gw.weights[2] = args->dwv;
    if (f32) {
      // rows of frozen heads belong to no slab of the product: exactly zero
      const size_t bytes = (size_t)d.D * d.C * 4;
      if (d.U < d.H && (cudaMemsetAsync(args->dwq, 0, bytes, st) != cudaSuccess || cudaMemsetAsync(args->dwk, 0, bytes, st) != cudaSuccess))
        return fail(SAF_ERR_CUDA, "cudaMemsetAsync");
      return launch_gemm_bwd_dw(gw, bw + b.dqkv, W, st);
    }
    if ((rc = launch_gemm_bwd_dw_full_sm100(gw, bw + b.dqkv, W, ws, ws_bytes, w32, st))) return rc;
  }
  return SAF_OK;
}

}  // extern "C"

// ---- the transformer block around the layer (inference) ----------------------------------------------------------------
namespace {

struct BlockLayout {       // (the layer's workspace comes first)
  int64_t normed, x1, hidden, total;
};
BlockLayout block_layout(const SafBlockArgs& b) {
  const Dims d = dims_of(b.layer);
  BlockLayout l;
  // The layer's part is read for the last time by its output projection, two launches before the first write of the MLP's
  // hidden rows, which may lie there.
  const int64_t layer = up(fwd_layout(b.layer, d).total), hidden = up(d.tok * b.hidden * 2);
  l.hidden = b.keep_projection ? layer : 0;
  int64_t at = b.keep_projection ? layer + hidden : std::max(layer, hidden);
  l.normed = at;
  at += up(d.tok * d.C * 2);
  l.x1 = at;
  at += up(d.tok * d.C * 2);
  l.total = at;
  return l;
}

int validate_block(const SafBlockArgs* b) {
  if (!b) return fail(SAF_ERR_INVALID, "null argument struct");
  if (b->struct_size != (int32_t)sizeof(SafBlockArgs))
    return fail(SAF_ERR_INVALID, "SafBlockArgs size mismatch: caller %d, library %d", b->struct_size, (int)sizeof(SafBlockArgs));
  if (int rc = validate_layer(&b->layer)) return rc;
  if (b->layer.attn.dtype != SAF_BF16 || b->layer.x_dtype != SAF_BF16 || b->layer.w_dtype != SAF_BF16 || b->layer.train)
    return fail(SAF_ERR_UNSUPPORTED, "the block entry is bf16 inference");
  if (b->hidden <= 0 || b->hidden % (b->gated ? 128 : 64) || b->layer.C % 64) return fail(SAF_ERR_UNSUPPORTED, "width %d, hidden %d", b->layer.C, b->hidden);
  if (b->hidden / 64 * (b->gated ? 2 : 1) > MLP_MAX_BLOCKS) return fail(SAF_ERR_LIMIT, "hidden %d", b->hidden);
  return SAF_OK;
}

// out = [residual +] act(x W^T + b) over whole matrices in 64-row blocks; gated: blocks of the two weights alternate
int mlp_linear(const void* x, int M, int K, const void* w0, const void* w1, const void* bias, int N, int act, const void* residual,
               int64_t ldr, void* out, int64_t ldo, int32_t* status, void* stream) {
  int32_t weight[MLP_MAX_BLOCKS], row0[MLP_MAX_BLOCKS];
  const int per = w1 ? 2 : 1, n = N / 64 * per;
  if (n > MLP_MAX_BLOCKS) return fail(SAF_ERR_LIMIT, "MLP width %d", N);
  for (int i = 0; i < n; ++i) {
    weight[i] = w1 ? i & 1 : 0;
    row0[i] = i / per * 64;
  }
  SafIndexedLinearArgs g;
  memset(&g, 0, sizeof(g));
  g.struct_size = (int32_t)sizeof(g);
  g.dtype = SAF_BF16;
  g.M = M; g.C = K;
  g.n_weights = per;
  g.slab = 64;
  g.n_slabs = n;
  g.x = x; g.ldx = K;
  g.weights[0] = w0; g.weights[1] = w1;
  g.biases[0] = bias;
  g.ldw[0] = g.ldw[1] = K;
  g.rows_w[0] = g.rows_w[1] = N;
  g.slab_weight = weight; g.slab_row0 = row0;
  g.out = out; g.ldo = ldo;
  g.status = status;
  g.act = act;
  g.residual = residual; g.ldr = ldr;
  if (int rc = validate_linear_args(&g)) return rc;
  const int rc = launch_gemm_sm100(g, (cudaStream_t)stream, nullptr, true);     // behind a norm or another product
  return rc == SAF_ERR_UNSUPPORTED ? saf_indexed_linear_fwd(&g, stream) : rc;
}

}  // namespace

extern "C" {

int saf_block_workspace(const SafBlockArgs* args, int64_t* bytes) {
  if (int rc = validate_block(args)) return rc;
  if (!bytes) return fail(SAF_ERR_INVALID, "null pointer");
  *bytes = block_layout(*args).total;
  return SAF_OK;
}

int saf_block_fwd(const SafBlockArgs* args, void* stream) {
  int rc = validate_block(args);
  if (rc) return rc;
  const SafBlockArgs& b = *args;
  const Dims d = dims_of(b.layer);
  const BlockLayout l = block_layout(b);
  if (!b.layer.x || !b.layer.out || !b.n1_w || !b.n2_w || !b.w_in || !b.w_out || (b.gated && !b.w_up)) return fail(SAF_ERR_INVALID, "null pointer");
  if (!b.layer.work || ((uintptr_t)b.layer.work & 255) || b.layer.work_bytes < l.total)
    return fail(SAF_ERR_INVALID, "workspace too small or not aligned to 256 bytes");
  if (b.rms && (b.n1_b || b.n2_b)) return fail(SAF_ERR_INVALID, "RMSNorm has no bias");
  cudaStream_t st = (cudaStream_t)stream;
  uint8_t* work = reinterpret_cast<uint8_t*>(b.layer.work);
  void *normed = work + l.normed, *x1 = work + l.x1, *hidden = work + l.hidden;
  const int M = (int)d.tok;
  if ((rc = launch_layernorm(b.layer.x, b.layer.ldx, b.n1_w, b.n1_b, normed, d.C, M, d.C, b.eps, SAF_BF16, b.rms, st))) return rc;
  SafAttnLayerArgs a = b.layer;
  a.x = normed;
  a.ldx = d.C;
  a.residual = b.layer.x;
  a.ldr = b.layer.ldx;
  a.out = x1;
  a.ldo = d.C;
  a.after_library_launch = 1;       // the norm, which writes no weights
  if ((rc = saf_attn_layer_fwd(&a, stream))) return rc;
  if ((rc = launch_layernorm(x1, d.C, b.n2_w, b.n2_b, normed, d.C, M, d.C, b.eps, SAF_BF16, b.rms, st))) return rc;
  int32_t* status = b.layer.attn.status;
  if ((rc = mlp_linear(normed, M, d.C, b.w_in, b.gated ? b.w_up : nullptr, b.b_in, b.hidden, b.gated ? SAF_ACT_SWIGLU : SAF_ACT_GELU,
                       nullptr, 0, hidden, b.hidden, status, stream)))
    return rc;
  return mlp_linear(hidden, M, b.hidden, b.w_out, nullptr, b.b_out, d.C, SAF_ACT_NONE, x1, d.C, b.layer.out, b.layer.ldo, status, stream);
}

}  // extern "C"
