"""The attention layer through `saf_attn_layer_fwd` / `saf_attn_layer_bwd`: one library call per direction over one
workspace, instead of an operator, an allocation and an autograd node for every product of the layer.

The forward's workspace holds the bf16 copies of fp32 inputs (autocast), the fused projection, the attention output and
the row statistics; a training call saves it for the backward, which works on the projection's own layout and returns
gradients in the dtypes of x and the weights.  Same mathematics as `linear_rows2` + `linear_rows` + `fused_mixed_attn` +
`linear_rows` with rotation fused (nanogpt/model.py:946-1077)."""
import ctypes as C

import torch

from . import ops
from ._cabi import SafAttnLayerArgs, SafAttnLayerBwdArgs, SafBlockArgs, SafMixedAttnArgs, lib, check, SAF_BF16, SAF_F32

_DT = {torch.float32: SAF_F32, torch.bfloat16: SAF_BF16}
HEAD_DIMS = (64, 96, 128)
MAX_BLOCKS = 160          # 64-row blocks of one backward product
MAX_HEADS = 256           # of the library's slab tables; the out projection's hold MAX_WIDTH / 64 blocks
MAX_WIDTH = 3 * MAX_HEADS * 64


class LayerPlan:
    """What a freeze set fixes on the host: head states and slots, and the argument struct with them filled in.  The
    struct points into this plan's own arrays, so a copied or unpickled plan is built anew from what made it."""

    def __init__(self, states, live, head_dim, width, n_kv=0):
        self._made_of = (list(states), list(live), head_dim, width, n_kv)
        H, U = len(states), len(live)
        self.H, self.U, self.hd, self.C, self.n_kv = H, U, head_dim, width, n_kv
        self._states = (C.c_int32 * H)(*states)
        self._live = (C.c_int32 * max(U, 1))(*live)
        a = SafAttnLayerArgs()
        a.struct_size = C.sizeof(SafAttnLayerArgs)
        a.C = width
        a.live = self._live
        t = a.attn
        t.struct_size = C.sizeof(SafMixedAttnArgs)
        t.dtype, t.H, t.U, t.HD, t.HKV, t.force_state = SAF_BF16, H, U, head_dim, n_kv, -1
        t.sm_scale = head_dim ** -0.5
        t.frozen_host = self._states
        self._template = bytes(a)
        kv = (n_kv or H) * head_dim
        self.weight_shapes = ((H * head_dim, width), (kv, width), (kv, width), (width, H * head_dim))
        self._sizes = {}

    def __reduce__(self):
        return LayerPlan, self._made_of

    def width(self):
        return (self.U + 2 * self.n_kv if self.n_kv else 2 * self.U + self.H) * self.hd

    def shapes_ok(self, training):
        """Sizes the tensor-core products of both directions take."""
        blocks = max(self.width(), self.C) // 64
        return (self.hd in HEAD_DIMS and 0 < self.U <= self.H <= MAX_HEADS and self.n_kv <= MAX_HEADS
                and self.C <= MAX_WIDTH and self.width() % 64 == 0 and self.C % 64 == 0
                and (not training or (blocks <= MAX_BLOCKS and self.H * self.hd % 64 == 0 and self.C + 3 * self.H * self.hd <= 32 * 1024)))

    def args(self, c):
        """The C struct of one call `c` (a _Call), every pointer taken from the tensors it holds now."""
        a = SafAttnLayerArgs.from_buffer_copy(self._template)
        t = a.attn
        x = c.x
        t.dtype = _DT[c.dt]
        t.B, t.T = c.B, c.T
        t.status = ops._status_ptr(x.device)
        t.frozen, t.hidx = c.frozen.data_ptr(), c.hidx.data_ptr()
        if c.kvidx is not None:
            t.kvidx = c.kvidx.data_ptr()
        if c.sink_decay is not None:
            t.sd_alpha, t.sd_rho = c.sink_decay[0].data_ptr(), c.sink_decay[1].data_ptr()
        if c.patt is not None:
            t.patt = ops._st(c.patt)
            t.S = c.patt.shape[1]
            t.patt_dtype = ops._dt(c.patt)
            if c.pidx is not None:
                t.pidx = c.pidx.data_ptr()
        if c.alpha is not None:
            t.alpha, t.rho, t.z = ops._st(c.alpha), ops._st(c.rho), ops._st(c.z)
            t.SD = c.alpha.shape[1]
            t.dec_dtype = ops._dt(c.alpha)
        a.x_dtype, a.w_dtype, a.train = _DT[x.dtype], _DT[c.w[0].dtype], c.train
        a.x, a.ldx = x.data_ptr(), _ld(x)
        a.wq, a.wk, a.wv, a.wo = [w.data_ptr() for w in c.w]
        if c.rope is not None:
            a.rope_cos, a.rope_sin = c.rope[0].data_ptr(), c.rope[1].data_ptr()
        return a

    def sizes(self, a):
        """(forward bytes, backward bytes, offset of the projection, offset of the attention output)."""
        t = a.attn
        key = (t.B, t.T, t.dtype, a.x_dtype, a.w_dtype, a.train)
        got = self._sizes.get(key)
        if got is None:
            out = (C.c_int64 * 4)()
            check(lib.saf_attn_layer_workspace(C.byref(a), out))
            if len(self._sizes) >= 64:
                self._sizes.clear()
            got = self._sizes[key] = tuple(out)
        return got


class _Call:
    """Tensors of one layer call, in the form the library reads them; dt is the dtype of the computation."""
    __slots__ = ("B", "T", "x", "w", "train", "rope", "frozen", "hidx", "kvidx", "sink_decay", "patt", "pidx", "alpha", "rho", "z",
                 "dt")

    def __init__(self, B, T, x, w, train, rope, frozen, hidx, kvidx=None, sink_decay=None, patt=None, pidx=None,
                 decomposed=(None, None, None), dt=torch.bfloat16):
        self.B, self.T, self.x, self.w, self.train, self.rope, self.dt = B, T, x, w, train, rope, dt
        self.frozen, self.hidx, self.kvidx, self.sink_decay = frozen, hidx, kvidx, sink_decay
        self.patt, self.pidx = patt, pidx
        self.alpha, self.rho, self.z = decomposed


def _plain(t, dtype, shape):
    """A tensor the library can take by its address and the plan's sizes."""
    return t.dtype is dtype and t.shape == shape and t.is_contiguous() and t.data_ptr() % 16 == 0


def usable(plan, x, weights, training):
    """True when the whole layer can run through the library's layer entry, which takes every size from the plan and the
    first two dimensions of x: other shapes stay with the operators (or are refused there)."""
    dt, shape = weights[0].dtype, x.shape
    if not (x.dtype in _DT and dt in _DT and len(shape) == 3 and shape[2] == plan.C and x.numel() > 0 and plan.shapes_ok(training)
            and x.data_ptr() % 16 == 0):
        return False
    for w, s in zip(weights, plan.weight_shapes):
        if not _plain(w, dt, s):
            return False
    return True


def _rows(x):
    """x as rows the library reads by TMA: 16-byte aligned, a whole number of 16-byte pieces and at least a row apart (an
    expanded tensor's rows are not); fp32 rows follow each other."""
    if x.is_contiguous() and x.data_ptr() % 16 == 0:
        return x
    x2 = ops._as_2d(x)
    step, C = _ld(x2), x2.shape[1]
    if x2.data_ptr() % 16 or (step != C if x2.dtype == torch.float32 else step % 8 or step < C):
        return x2.clone(memory_format=torch.contiguous_format)     # (.contiguous() keeps a misaligned contiguous tensor)
    return x2


def _ld(x):
    """Row stride of a contiguous tensor or a matrix (torch reports any stride for a single row)."""
    return x.shape[-1] if x.is_contiguous() else x.stride(0)


def _blob(n, device):
    return torch.empty(n, dtype=torch.uint8, device=device)


def _forward(plan, c, biases=None, residual=None):
    """Enqueues the layer; returns (out (tokens, C), workspace, sizes)."""
    a = plan.args(c)
    sz = plan.sizes(a)
    dev = c.x.device
    work = _blob(sz[0], dev)
    out = torch.empty((c.B * c.T, plan.C), dtype=c.dt, device=dev)
    a.out, a.ldo = out.data_ptr(), plan.C
    a.work, a.work_bytes = work.data_ptr(), sz[0]
    if biases is not None:
        a.bq, a.bk, a.bv, a.bo = [None if b is None else b.data_ptr() for b in biases]
    if residual is not None:
        a.residual, a.ldr = residual.data_ptr(), _ld(residual)
    events = ops.attention_event_pair()
    if events is not None:
        a.event_before, a.event_after = events
    ops._call(c.x, lib.saf_attn_layer_fwd, C.byref(a))
    return out, work, sz


def projection_views(plan, work, sz, B, T, dt=torch.bfloat16):
    """q, k, v (B, heads, T, hd) and the attention output y inside a forward workspace."""
    W, hd, es = plan.width(), plan.hd, dt.itemsize
    n = B * T * W
    qkv = work[sz[2]:sz[2] + es * n].view(dt).view(B, T, W // hd, hd)
    nk = plan.n_kv or plan.U
    y = work[sz[3]:sz[3] + es * B * T * plan.H * hd].view(dt).view(B, T, plan.H, hd)
    q, k, v = qkv[:, :, :plan.U], qkv[:, :, plan.U:plan.U + nk], qkv[:, :, plan.U + nk:]
    return q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2), y.transpose(1, 2)


class _LayerFunction(torch.autograd.Function):
    """(x, wq, wk, wv, wo, alpha, rho) -> layer output; alpha / rho are passed when they learn."""

    @staticmethod
    def forward(ctx, x, wq, wk, wv, wo, alpha_p, rho_p, plan, c, measure):
        out, work, sz = _forward(plan, c)
        if measure is not None:
            q, k, _, _ = projection_views(plan, work, sz, c.B, c.T, c.dt)
            measure(q, k)
        ctx.plan, ctx.sz, ctx.bt, ctx.dt = plan, sz, (c.B, c.T), c.dt
        ctx.x_like, ctx.w_cast = (x.shape, x.dtype), wq.dtype != c.dt
        # (converted tensors live in the workspace: the originals are not needed again)
        kept = [work, c.x if x.dtype == c.dt else None]
        kept += [None] * 4 if ctx.w_cast else [wq, wk, wv, wo]
        kept += [c.patt, c.pidx, c.alpha, c.rho, c.z, *(c.rope or (None, None))]
        ctx.save_for_backward(*kept, c.frozen, c.hidx, *(c.sink_decay or ()))
        ctx.w_like = [(w.shape, w.dtype) for w in (wq, wk, wv, wo)]
        ctx.learns = alpha_p is not None
        return out.view(*x.shape[:-1], plan.C)

    @staticmethod
    @torch.autograd.function.once_differentiable
    def backward(ctx, dout):
        saved = ctx.saved_tensors          # once: a checkpointed layer unpacks what it recomputed a single time
        work, x2, wq, wk, wv, wo, patt, pidx, alpha, rho, z, cos, sin, frozen, hidx = saved[:15]
        sink_decay = saved[15:] or None
        plan, sz = ctx.plan, ctx.sz
        B, T = ctx.bt
        dev = dout.device
        need = ctx.needs_input_grad
        d2 = _bf16_rows(dout) if ctx.dt == torch.bfloat16 else _rows(dout)
        x_shape, x_dtype = ctx.x_like
        # a converted tensor is read from the workspace; its argument only tells the dtype and layout
        x_arg = x2 if x2 is not None else work.view(torch.float32)[:plan.C].view(1, plan.C)
        w_arg = [wq, wk, wv, wo] if wq is not None else [work.view(torch.float32)] * 4
        c = _Call(B, T, x_arg, w_arg, 1, (cos, sin) if cos is not None else None, frozen, hidx, None, sink_decay, patt, pidx,
                  (alpha, rho, z), ctx.dt)
        g = SafAttnLayerBwdArgs()
        g.struct_size = C.sizeof(SafAttnLayerBwdArgs)
        g.fwd = plan.args(c)
        g.fwd.work, g.fwd.work_bytes = work.data_ptr(), sz[0]
        g.dout, g.lddo = d2.data_ptr(), _ld(d2)
        scratch = _blob(sz[1], dev)
        g.work, g.work_bytes = scratch.data_ptr(), sz[1]
        dx, dw = None, [None] * 4
        if need[0]:
            dx = torch.empty(x_shape, dtype=x_dtype, device=dev)
            g.dx = dx.data_ptr()
        if need[1] or need[2] or need[3]:
            for i in range(3):
                dw[i] = torch.empty(ctx.w_like[i][0], dtype=ctx.w_like[i][1], device=dev)
            g.dwq, g.dwk, g.dwv = [t.data_ptr() for t in dw[:3]]
        if need[4]:
            dw[3] = torch.empty(ctx.w_like[3][0], dtype=ctx.w_like[3][1], device=dev)
            g.dwo = dw[3].data_ptr()
        g.need_dy = int(ctx.learns)
        ops._call(d2, lib.saf_attn_layer_bwd, C.byref(g))
        da = dr = None
        if ctx.learns:
            from .trainable_patterns import pattern_param_grad
            _, _, v, y = projection_views(plan, work, sz, B, T, ctx.dt)
            dy = scratch[:ctx.dt.itemsize * B * T * plan.H * plan.hd].view(ctx.dt).view(B, T, plan.H, plan.hd).transpose(1, 2)
            da, dr = pattern_param_grad(dy, y, v, alpha, rho, z, frozen)
        return (dx, *[t if need[1 + i] else None for i, t in enumerate(dw)], da, dr, None, None, None)


def _bf16_rows(x):
    return _rows(x if x.dtype == torch.bfloat16 else x.to(torch.bfloat16))


def _residual_rows(residual, tokens, width):
    """`residual` as the output projection reads it; its map covers tokens x width whatever the tensor holds."""
    r2 = ops._as_2d(residual)
    if r2.shape != (tokens, width) or r2.dtype != torch.bfloat16:
        raise ValueError("residual must match the output")
    return _bf16_rows(r2)


def attention_layer(plan, x, weights, rope, frozen, hidx, *, kvidx=None, sink_decay=None, patt=None, pidx=None,
                    decomposed=(None, None, None), learn=None, biases=None, residual=None, measure=None, dtype=torch.bfloat16):
    """x (B, T, C) -> (B, T, C) in `dtype`, the dtype of the computation: bf16, or fp32 with everything in fp32.  weights:
    q, k, v, o; decomposed: (alpha, rho, z) buffers; learn: (alpha, rho) parameters that receive gradients (decomposed then
    holds their detached values and current normalisers); measure: called with the rotated q, k of the live heads.  Biases
    and residual go with inference, the residual with bf16."""
    enabled = torch.is_grad_enabled()
    grad = enabled and (x.requires_grad or learn is not None or any(w.requires_grad for w in weights))
    if residual is not None:
        residual = _residual_rows(residual, x.shape[0] * x.shape[1], plan.C)
    c = _Call(x.shape[0], x.shape[1], _rows(x.detach()), weights, int(grad), rope, frozen, hidx, kvidx, sink_decay, patt, pidx,
              decomposed, dtype)
    # (also when nothing wants a gradient: forward-mode tangents are refused there instead of getting lost)
    if grad or (enabled and biases is None and residual is None):
        ap, rp = learn if learn is not None else (None, None)
        return _LayerFunction.apply(x, *weights, ap, rp, plan, c, measure)
    out, work, sz = _forward(plan, c, biases, residual)
    if measure is not None:
        q, k, _, _ = projection_views(plan, work, sz, c.B, c.T, c.dt)
        measure(q, k)
    return out.view(c.B, c.T, plan.C)


_HOOKS = torch.nn.modules.module


def untouched(*modules):
    """Whether a block may read these sub-modules' parameters instead of calling them.  modules: (module, class) pairs.  A
    module of another class (a replaced MLP, a subclass) or with a forward of its own computes something else, and hooks on
    it, or on all modules, are to be called."""
    for m, cls in modules:
        if type(m) is not cls or m._forward_pre_hooks or m._forward_hooks or "forward" in m.__dict__:
            return False
    return not (_HOOKS._global_forward_pre_hooks or _HOOKS._global_forward_hooks)


def block_usable(plan, x, call, norm1, norm2, mlp, gated):
    """bf16 inference of the whole block: every weight and norm in bf16 and of the plan's width, widths in whole 64-row
    blocks.  Arguments as `block` takes them; `usable` has seen the call's weights."""
    dt, C, hidden = torch.bfloat16, plan.C, mlp[0].shape[0]
    if x.dtype is not dt or call["weights"][0].dtype is not dt or hidden % (128 if gated else 64) or hidden // 64 * (2 if gated else 1) > 288:
        return False
    for t in (*norm1, *norm2):
        if t is not None and not _plain(t, dt, (C,)):
            return False
    for t, s in zip(mlp, ((hidden, C), (hidden, C), (hidden,), (C, hidden), (C,))):
        if t is not None and not _plain(t, dt, s):
            return False
    for t, s in zip(call.get("biases", ()), plan.weight_shapes):
        if t is not None and not _plain(t, dt, s[:1]):
            return False
    return True


def block(plan, x, call, norm1, norm2, mlp, eps, *, rms=False, gated=False):
    """One pre-norm block, x (B, T, C) bf16 -> (B, T, C), in one library call.  call: the keyword arguments of
    `attention_layer`; norm: (weight, bias); mlp: (w_in, w_up, b_in, w_out, b_out)."""
    biases, measure = call.get("biases"), call.get("measure")
    c = _Call(x.shape[0], x.shape[1], _bf16_rows(x), call["weights"], 0, call["rope"], call["frozen"], call["hidx"], call.get("kvidx"),
              call.get("sink_decay"), call.get("patt"), call.get("pidx"), call.get("decomposed", (None, None, None)))
    g = SafBlockArgs()
    g.struct_size = C.sizeof(SafBlockArgs)
    g.rms, g.gated, g.hidden, g.eps = int(rms), int(gated), mlp[0].shape[0], eps
    a = plan.args(c)
    if biases is not None:
        a.bq, a.bk, a.bv, a.bo = [None if b is None else b.data_ptr() for b in biases]
    tok, Cw = c.B * c.T, plan.C
    dev = x.device
    g.keep_projection = int(measure is not None)
    key = ("block", c.B, c.T, g.hidden, g.keep_projection)
    n = plan._sizes.get(key)
    if n is None:
        g.layer = a
        out = C.c_int64()
        check(lib.saf_block_workspace(C.byref(g), C.byref(out)))
        if len(plan._sizes) >= 64:
            plan._sizes.clear()
        n = plan._sizes[key] = out.value
    work = _blob(n, dev)
    out = torch.empty((tok, Cw), dtype=torch.bfloat16, device=dev)
    a.out, a.ldo = out.data_ptr(), Cw
    a.work, a.work_bytes = work.data_ptr(), n
    events = ops.attention_event_pair()
    if events is not None:
        a.event_before, a.event_after = events
    g.layer = a
    g.n1_w, g.n1_b, g.n2_w, g.n2_b = [None if t is None else t.data_ptr() for t in (*norm1, *norm2)]
    g.w_in, g.w_up, g.b_in, g.w_out, g.b_out = [None if t is None else t.data_ptr() for t in mlp]
    ops._call(c.x, lib.saf_block_fwd, C.byref(g))
    if measure is not None:
        q, k, _, _ = projection_views(plan, work, plan.sizes(a), c.B, c.T)
        measure(q, k)
    return out.view(c.B, c.T, Cw)
