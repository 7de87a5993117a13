"""fp32 layers through the layer entry against the operators they stand for: head widths, token counts, biases, no rotation,
every kind of frozen head (learning ones too), strided inputs, residuals, gradients of a part of the inputs."""
import random
from types import SimpleNamespace

import pytest
import torch

from tests.test_layer_forms_gpu import freeze, inputs, rel, weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", range(24))
def test_fp32_layer(seed, monkeypatch):
    from saf_b200 import layer, trainable_patterns
    from saf_b200.attention import SafCausalSelfAttention, rope_tables
    rng, g = random.Random(300 + seed), torch.Generator().manual_seed(seed)
    hd = rng.choice([64, 64, 96, 128])
    H = rng.choice([2, 4, 6]) if hd == 96 else rng.randrange(1, 7)
    B, T = rng.randrange(1, 4), rng.choice([1, 37, 64, 127, 129, 300, 640])
    train, bias = rng.random() < 0.7, rng.random() < 0.2
    C = H * hd
    cfg = SimpleNamespace(n_embd=C, n_head=H, block_size=(T + 63) // 64 * 64, bias=bias, dropout=0.0,
                          position_encoding=rng.choice(["rope", "rope", "none"]), rand_attn_prior_repr="decomposed",
                          freeze_pattern_dtype=rng.choice(["float32", "bfloat16"]))
    m = SafCausalSelfAttention(cfg)
    weights(m, seed)
    m = m.cuda()
    freeze(rng, m, H, T, g)
    learn = train and bool(m.dyn_decomp.any()) and rng.random() < 0.5
    if learn:
        trainable_patterns.enable(m)
    cos, sin = rope_tables(hd, T, device="cuda")
    rope = (cos.view(1, 1, T, hd), sin.view(1, 1, T, hd)) if cfg.position_encoding == "rope" else None
    x = inputs(rng, g, B, T, C, torch.float32)
    res = torch.randn(B, T, C, generator=g).cuda() if rng.random() < 0.5 else None
    dy = torch.randn(B, T, C, generator=g).cuda()
    params = [p for p in m.parameters() if rng.random() < 0.8]
    calls = []
    through = layer._forward
    monkeypatch.setattr(layer, "_forward", lambda *a, **k: (calls.append(1), through(*a, **k))[1])

    def run():
        with torch.set_grad_enabled(train):
            xx = x.detach().requires_grad_(train)
            y = m(xx, rope=rope, residual=res)
            return [y.detach()] + (list(torch.autograd.grad(y, [xx, *params], dy, allow_unused=True)) if train else [])

    got = run()
    entered = len(calls)
    monkeypatch.setattr(SafCausalSelfAttention, "_layer_call", lambda *a: None)
    want = run()
    # the entry takes every head width whose projection is whole 64-column blocks, and no bias gradients
    assert len(calls) == entered and entered == int(m._plan.shapes_ok(train) and not (train and bias))
    assert hd == 96 or m._plan.shapes_ok(train)
    # the same fp32 sums in another order at most (dx: one product over [Q | K | V] instead of two and an addition): a few
    # roundings of 2^-24 of sums of up to 1152 terms
    for a, b in zip(got, want):
        assert (a is None) == (b is None)
        if a is not None:
            assert a.dtype == b.dtype and a.shape == b.shape
            # (q and k of one key have no gradient: both are rounding)
            assert rel(a, b) <= 2e-6 or (a - b).norm() <= 1e-6 * got[1].norm(), a.shape
    if train and not bias:
        dead = [h for h in range(H) if h not in m._live]
        for p, gr in zip(params, got[2:]):
            if p is m.q_proj.weight or p is m.k_proj.weight:
                assert gr.view(H, hd, C)[dead].abs().sum() == 0
