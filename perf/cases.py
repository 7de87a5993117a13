"""The work that users of this framework have it do, as cases that can be timed and compared.

`listed()` names a dozen of them, `draw()` gives more of the same ranges, `prepare()` makes what a user's program has in
hand before the call (module, weights, freeze state, inputs), `run()` is one pass through the public entry points,
`work()` the bytes and operations the path cannot do without, `tolerance()` what two correct implementations of it may
differ by.  A case is a dict of plain values:

  kind     "layer"   one attention layer of a prefill (bf16, inference)
           "block"   the transformer block around it (LayerNorms, MLP, residuals)
           "model"   token ids -> next-token logits through all blocks
           "gqa"     the grouped-query block (RMSNorms, gated MLP)
           "train"   forward and backward of one attention layer: bf16 autocast over fp32 master weights, or fp32
           "measure" a freeze controller's statistics of one layer, one batch merged into running moments
  heads, head_dim, frozen, T, B   as in the workload table (frozen = heads on a fixed pattern, 25 % in earnest)
  pattern  what the frozen heads hold: "sink" (sink weight + decay, two numbers a head), "dense" (a stored T x T
           matrix), "decomposed" (alpha_j + rho_{i-j}; while training the two vectors learn too)
"""
import math
import os
import sys
from types import SimpleNamespace

import torch

_PKG = os.path.join(os.getcwd(), "selective-attention-freezing_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from saf_b200 import gqa, synthetic, trainable_patterns  # noqa: E402
from saf_b200.attention import SafCausalSelfAttention, rope_tables  # noqa: E402
from saf_b200.block import SafBlock  # noqa: E402
from saf_b200.capture import AttentionMoments, LogitMoments  # noqa: E402
from saf_b200.model import SafGPT  # noqa: E402

DEV = "cuda"
VOCAB = 50257


def _case(kind, heads, head_dim, frozen, T, B, pattern="sink", dtype="bfloat16", **more):
    return dict(kind=kind, heads=heads, head_dim=head_dim, frozen=frozen, T=T, B=B, pattern=pattern, dtype=dtype, **more)


def listed():
    return [
        # the smallest call: one short layer of the test-sized workload; latency and launches are all there is
        dict(_case("layer", 4, 64, 1, 512, 2), name="layer tiny"),
        # one user's prompt through the whole 12-layer model, an odd length: next-token logits, launch after launch
        dict(_case("model", 12, 64, 3, 777, 1, layers=12), name="model one prompt"),
        # the single fp32 layer of the benchmark table, trained in fp32 (parity work, small studies)
        dict(_case("train", 12, 64, 3, 1024, 2, dtype="float32"), name="train fp32 layer"),
        # prefill of ordinary prompts in a batch: the whole 12 x 64 block at T = 4096, B = 16
        dict(_case("block", 12, 64, 3, 4096, 16), name="block prefill 4K"),
        # long-context prefill: the layer of the headline metric
        dict(_case("layer", 12, 64, 3, 16384, 4), name="layer prefill 16K"),
        # heads frozen on stored patterns (what a freeze controller installs first), a ragged length
        dict(_case("layer", 12, 64, 3, 1999, 8, pattern="dense"), name="layer dense ragged"),
        # grouped-query prefill at the table's sizes: 12 query heads on 2 KV heads x 128, gated MLP 8960
        dict(_case("gqa", 12, 128, 3, 8192, 8, kv=2, mlp=8960), name="gqa block 8K"),
        # training at a 124M model's own context length
        dict(_case("train", 12, 64, 3, 1024, 8), name="train 12x64 1K"),
        # training of the ~1B configuration: 16 heads x 128, T = 8192, micro-batch 2
        dict(_case("train", 16, 128, 4, 8192, 2), name="train 16x128 8K"),
        # the 16 x 96 recipe on one ragged sequence
        dict(_case("train", 16, 96, 4, 3001, 1), name="train 16x96 ragged"),
        # learnable decomposed patterns: the frozen heads' alpha and rho receive gradients too
        dict(_case("train", 12, 64, 3, 2048, 4, pattern="decomposed"), name="train patterns 2K"),
        # controller measurement between freeze events: attention and logit moments of 9 live heads
        dict(_case("measure", 12, 64, 3, 4096, 4), name="measure 4K"),
    ]


# ---- ranges -----------------------------------------------------------------------------------------------------------
def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _length(rng, lo, hi):
    """A sequence length, half of them whole multiples of 128 and half of them odd ones."""
    T = _log_int(rng, lo, hi)
    return max(lo, T // 128 * 128) if rng.random() < 0.5 else T | 1


def _heads(rng, shapes):
    heads, head_dim = rng.choice(shapes)
    return heads, head_dim, max(1, heads // 4)


def draw(rng):
    """One more case of the ranges above; the batch is what the token budget of the kind leaves."""
    kind = rng.choice(["layer", "layer", "block", "model", "gqa", "train", "train", "train", "measure"])
    if kind == "layer":
        pattern = rng.choice(["sink", "sink", "dense"])
        T = _length(rng, 256, 16384 if pattern == "sink" else 4096)
        B = min(32, max(1, _log_int(rng, 256, 65536) // T))
        return _case(kind, *_heads(rng, [(4, 64), (12, 64), (16, 96), (8, 128)]), T, B, pattern=pattern)
    if kind == "block":
        T = _length(rng, 256, 16384)
        return _case(kind, *_heads(rng, [(4, 64), (12, 64)]), T, min(32, max(1, _log_int(rng, 512, 65536) // T)))
    if kind == "model":
        return _case(kind, 12, 64, 3, _length(rng, 64, 2048), rng.choice([1, 1, 2, 4]), layers=rng.choice([6, 12]))
    if kind == "gqa":
        T = _length(rng, 256, 8192)
        return _case(kind, 12, 128, 3, T, min(8, max(1, _log_int(rng, 512, 32768) // T)), kv=2, mlp=8960)
    if kind == "measure":
        return _case(kind, *_heads(rng, [(12, 64), (8, 128)]), _length(rng, 512, 4096), rng.choice([1, 2, 4]))
    if rng.random() < 0.25:
        return _case(kind, 12, 64, 3, _length(rng, 128, 1024), rng.choice([1, 2]), dtype="float32")
    pattern = rng.choice(["sink", "sink", "decomposed"])
    shapes = [(12, 64), (16, 128)] if pattern == "decomposed" else [(12, 64), (16, 96), (16, 128)]
    T = _length(rng, 256, 8192 if pattern == "sink" else 2048)
    return _case(kind, *_heads(rng, shapes), T, min(16, max(1, _log_int(rng, 1024, 16384) // T)), pattern=pattern)


# ---- what a user's program has in hand before the call ----------------------------------------------------------------
def _config(c, **more):
    T = c["T"]
    # buffers of frozen patterns are made for the context length, a whole number of 64-row bands
    return SimpleNamespace(n_embd=c["heads"] * c["head_dim"], n_head=c["heads"], block_size=(T + 63) // 64 * 64, bias=False,
                           dropout=0.0, position_encoding="rope", freeze_pattern_dtype="bfloat16",
                           rand_attn_prior_repr="decomposed" if c["pattern"] == "decomposed" else "dense", **more)


def _weights(module, g):
    """Random-init weights N(0, 0.02^2) of every matrix and bias, drawn on the GPU; norms keep their ones."""
    with torch.no_grad():
        for name, p in module.named_parameters():
            if p.dim() >= 2 or name.endswith("bias"):
                p.normal_(0.0, 0.02, generator=g)


def _freeze(attn, c, seed):
    """The layer's frozen heads and what they hold, as a freeze controller leaves it."""
    T, nf = c["T"], c["frozen"]
    fz = synthetic.frozen_heads_for_layer(c["heads"], nf, seed, attn.layer_idx)
    a, r = synthetic.sink_decay_params(nf, seed + 1000 + attn.layer_idx)
    if c["pattern"] == "sink":
        attn.freeze_heads_sink_decay(fz, a.tolist(), r.tolist())
        return
    g = torch.Generator(device=DEV).manual_seed(seed + 17)
    if c["pattern"] == "dense":
        # a mean attention map: decay from the diagonal, some weight on the first key, noise; rows normalised at install
        d = torch.arange(T, device=DEV)
        d = (d[:, None] - d[None, :]).clamp_min(0).float()
        p = torch.rand(nf, T, T, device=DEV, generator=g)
        for i in range(nf):
            p[i] *= torch.exp(-d / (T / 8.0)) + 0.02
            p[i, :, 0] += float(a[i]) * T / 8.0
        attn.freeze_heads(fz, p)
    else:
        alpha = torch.randn(nf, T, device=DEV, generator=g) * 0.5
        rho = torch.randn(nf, T, device=DEV, generator=g) * 0.1
        rho -= torch.arange(T, device=DEV).float() * (8.0 / T)
        attn.freeze_heads_decomposed(fz, alpha, rho)


def _rope(c, base=10000.0):
    cos, sin = rope_tables(c["head_dim"], c["T"], base=base, device=DEV)
    return cos.view(1, 1, c["T"], -1), sin.view(1, 1, c["T"], -1)


def prepare(case, seed):
    c = case
    kind, T, B = c["kind"], c["T"], c["B"]
    g = torch.Generator(device=DEV).manual_seed(seed)
    s = SimpleNamespace(case=c)
    if kind == "gqa":
        cfg = SimpleNamespace(hidden_size=c["heads"] * c["head_dim"], num_attention_heads=c["heads"], num_key_value_heads=c["kv"],
                              head_dim=c["head_dim"], attention_bias=True, qk_norm=False, rms_norm_eps=1e-6,
                              intermediate_size=c["mlp"], max_position_embeddings=T)
        with torch.device(DEV):
            m = gqa.SafQwenBlock(cfg)
        _weights(m, g)
        s.module = m.to(torch.bfloat16).eval()
        fz = synthetic.frozen_heads_for_layer(c["heads"], c["frozen"], seed, 0)
        a, r = synthetic.sink_decay_params(len(fz), seed + 1000)
        m.self_attn.set_frozen(sink_decay=fz, sd_params=(a.tolist(), r.tolist()))
        s.rope = rope_tables(c["head_dim"], T, base=1000000.0, device=DEV)
        s.x = torch.randn(B, T, cfg.hidden_size, device=DEV, generator=g).bfloat16()
        return s
    if kind == "model":
        with torch.device(DEV):
            m = SafGPT(_config(c, n_layer=c["layers"], vocab_size=VOCAB, rope_base=10000.0))
        _weights(m, g)
        for blk in m.transformer.h:
            _freeze(blk.main_block, c, seed)
        s.module = m.to(torch.bfloat16).eval()
        s.ids = torch.randint(0, VOCAB, (B, T), device=DEV, generator=g)
        return s
    if kind == "measure":
        U, hd = c["heads"] - c["frozen"], c["head_dim"]
        # rotated q and k as the layer's projection lays them out: one token-major buffer
        qk = torch.randn(B, T, 2 * U, hd, device=DEV, generator=g).bfloat16()
        s.q, s.k = qk[:, :, :U].transpose(1, 2), qk[:, :, U:].transpose(1, 2)
        s.attn, s.logits = AttentionMoments(U, T, DEV), LogitMoments(U, T, DEV, with_var=True)
        # the measurement is under way: an earlier batch is in the running moments
        first = torch.randn(2, B, T, U, hd, device=DEV, generator=g).bfloat16().transpose(2, 3)
        s.attn.update(first[0], first[1])
        s.logits.update(first[0], first[1])
        return s
    cfg = _config(c)
    with torch.device(DEV):
        m = SafBlock(cfg) if kind == "block" else SafCausalSelfAttention(cfg)
    _weights(m, g)
    attn = m.main_block if kind == "block" else m
    _freeze(attn, c, seed)
    s.rope = _rope(c)
    x = torch.randn(B, T, cfg.n_embd, device=DEV, generator=g)
    if kind == "train":
        # the residual stream and the master weights are fp32; under autocast the layer's output and its gradient are bf16
        m.train()
        s.params = [m.q_proj.weight, m.k_proj.weight, m.v_proj.weight, m.c_proj.weight]
        if c["pattern"] == "decomposed":
            s.params += trainable_patterns.enable(m)
        s.x = x.requires_grad_(True)
        dt = torch.float32 if c["dtype"] == "float32" else torch.bfloat16
        s.dy = torch.randn(B, T, cfg.n_embd, device=DEV, generator=g).to(dt)
        s.module = m
        return s
    s.module = m.to(torch.bfloat16).eval()
    s.x = x.bfloat16()
    return s


# ---- one pass ---------------------------------------------------------------------------------------------------------
def run(state):
    s, c = state, state.case
    kind = c["kind"]
    if kind == "train":
        # parameters have moved since the last step, so normalisers of learnable patterns are recomputed, as the
        # optimizer's post-step hook arranges
        if c["pattern"] == "decomposed":
            trainable_patterns.clear_pattern_cache()
        with torch.autocast("cuda", dtype=torch.bfloat16, enabled=c["dtype"] == "bfloat16"):
            y = s.module(s.x, rope=s.rope)
        return [y.detach(), *torch.autograd.grad(y, [s.x, *s.params], s.dy)]
    with torch.inference_mode():
        if kind == "measure":
            s.attn.update(s.q, s.k)
            s.logits.update(s.q, s.k)
            return [s.attn.mean, s.attn.head_m2, s.attn.neg_entropy, s.logits.mean, s.logits.m2]
        if kind == "model":
            return s.module(s.ids)[0]
        if kind == "gqa":
            return s.module(s.x, s.rope)
        return s.module(s.x, rope=s.rope)


# ---- what the path cannot do without ----------------------------------------------------------------------------------
def work(case):
    c = case
    kind, H, hd, nf, T, B = c["kind"], c["heads"], c["head_dim"], c["frozen"], c["T"], c["B"]
    U, C, tok = H - nf, H * hd, B * T
    if kind == "measure":
        # lower triangle of the mean attention, whole squares of the logits' mean and centred squares, each read and
        # written once; causal attention scores are part of the whole square of scores
        return dict(bytes=2 * tok * U * hd * 2 + U * T * T * 4 * (1 + 2 + 2), flops=2 * B * U * T * T * hd)
    live = 2 * B * U * T * T * hd                               # causal half of the two products
    fixed = B * nf * T * T * hd if c["pattern"] != "sink" else 0
    stored = nf * T * T if c["pattern"] == "dense" else 0        # bf16, lower triangle: T^2 / 2 entries a head
    if kind == "gqa":
        HK, M = c["kv"], c["mlp"]
        nw = C * (U + 2 * HK) * hd + C * C + 3 * C * M
        return dict(bytes=4 * tok * C + 2 * nw, flops=live + 2 * tok * nw)
    nw = C * (2 * U + H) * hd + C * C                           # projection weights that take part
    if kind == "block":
        nw += 8 * C * C
    if kind == "model":
        L = c["layers"]
        nw = L * (nw + 8 * C * C)
        return dict(bytes=2 * (nw + VOCAB * C + tok * C) + 8 * tok + 2 * B * VOCAB, flops=L * live + 2 * tok * nw + 2 * B * C * VOCAB)
    if kind == "train":
        size = 4 if c["dtype"] == "float32" else 2              # activations in and out of the layer: x, dx fp32; y, dy
        return dict(bytes=tok * C * (4 + 4 + 2 * size) + 2 * 4 * nw,
                    flops=3 * 2 * tok * nw + 3.5 * live + (4 if c["pattern"] == "decomposed" else 2) * fixed)
    return dict(bytes=4 * tok * C + 2 * nw + stored, flops=live + fixed + 2 * tok * nw)


def tolerance(case):
    """About four times what the path was seen to differ by from the same computation in torch: fp32 for the bf16 cases
    (0.003 for a prefill layer, 0.007 for a training layer's gradients, 0.009 after twelve layers, single values of an
    input gradient by half the root mean square), fp64 for the fp32 layer (1.5e-6) and the statistics (3.5e-5)."""
    c = case
    if c["kind"] == "train":
        return {"rel": 6e-6, "max": 2e-4} if c["dtype"] == "float32" else {"rel": 2e-2, "max": 0.9}
    if c["kind"] == "measure":
        return {"rel": 1.5e-4, "max": 5e-4}
    return {"rel": 2e-2 if c["kind"] == "model" else 1.2e-2, "max": 0.4}
