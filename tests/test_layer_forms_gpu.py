"""The layer and block entries against the operators they stand for, over the forms of call they accept: head widths and
counts, biases, hidden sizes that are not heads x width, no rotation, every kind of frozen head, strided inputs, residuals,
autocast over fp32 weights.  Both sides round to bf16 at the same places in the forward (projection, attention output,
result), in sums of another order at most; the operators' gradients are rounded to bf16 once more."""
import random
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
FWD, BWD = 4e-3, 1.2e-2      # 2^-8; three roundings of 2^-8 along the operators' gradient chain


def rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-20)).item()


def weights(m, seed):
    g = torch.Generator().manual_seed(seed)
    with torch.no_grad():
        for p in m.parameters():
            p.copy_(torch.randn(p.shape, generator=g) * (p.shape[-1] ** -0.5 if p.dim() == 2 else 0.1))


def freeze(rng, m, H, T, g):
    """Some heads of every kind the module has, at least one live."""
    heads = rng.sample(range(H), rng.randrange(0, H))
    kinds = {h: rng.choice(["dense", "sink", "decomposed"]) for h in heads}
    dense, sink, dec = [[h for h in heads if kinds[h] == k] for k in ("dense", "sink", "decomposed")]
    patt = torch.rand(len(dense), T, T, generator=g).tril()
    a, r = [rng.uniform(0, 0.5) for _ in sink], [rng.uniform(0.3, 0.999) for _ in sink]
    alpha, rho = torch.randn(H, T, generator=g) * 0.5, torch.randn(H, T, generator=g) * 0.5
    if hasattr(m, "set_frozen"):
        m.set_frozen(dense=dense, patterns=patt if dense else None, decomposed=dec, decomp=(alpha.cuda(), rho.cuda()) if dec else None,
                     sink_decay=sink, sd_params=(a, r) if sink else None)
        return
    if dense:
        m.freeze_heads(dense, patt)
    if sink:
        m.freeze_heads_sink_decay(sink, a, r)
    if dec:
        m.freeze_heads_decomposed(dec, alpha[dec].cuda(), rho[dec].cuda())


def inputs(rng, g, B, T, C, dtype):
    x = torch.randn(B, T, C + 64, generator=g).cuda().to(dtype)
    return x[..., :C] if rng.random() < 0.3 else x[..., :C].contiguous()


@pytest.mark.parametrize("seed", range(24))
def test_dense_module(seed, monkeypatch):
    from saf_b200.attention import SafCausalSelfAttention, rope_tables
    rng, g = random.Random(seed), torch.Generator().manual_seed(seed)
    hd = rng.choice([64, 64, 96, 128])
    H = rng.choice([2, 4, 6]) if hd == 96 else rng.randrange(1, 7)
    B, T = rng.randrange(1, 4), rng.choice([1, 64, 127, 128, 200, 333, 640])
    train, bias = rng.random() < 0.5, rng.random() < 0.3
    C = H * hd
    cfg = SimpleNamespace(n_embd=C, n_head=H, block_size=(T + 63) // 64 * 64, bias=bias, dropout=0.0,
                          position_encoding=rng.choice(["rope", "rope", "none"]), rand_attn_prior_repr="decomposed",
                          freeze_pattern_dtype=rng.choice(["float32", "bfloat16"]))
    m = SafCausalSelfAttention(cfg)
    weights(m, seed)
    wdt = rng.choice([torch.float32, torch.bfloat16])
    m = m.cuda()
    if wdt == torch.bfloat16:
        for lin in (m.q_proj, m.k_proj, m.v_proj, m.c_proj):
            lin.to(wdt)
    freeze(rng, m, H, T, g)
    cos, sin = rope_tables(hd, T, device="cuda")
    rope = (cos.view(1, 1, T, hd), sin.view(1, 1, T, hd)) if cfg.position_encoding == "rope" else None
    xdt = wdt if train else rng.choice([torch.bfloat16, wdt])
    x = inputs(rng, g, B, T, C, xdt)
    res = torch.randn(B, T, C, generator=g).cuda().to(xdt) if rng.random() < 0.5 else None
    dy = torch.randn(B, T, C, generator=g).cuda().bfloat16()
    auto = xdt == torch.float32 or (train and wdt == torch.float32) or rng.random() < 0.3

    def run():
        with torch.set_grad_enabled(train), torch.autocast("cuda", dtype=torch.bfloat16, enabled=auto):
            xx = x.detach().requires_grad_(train)
            y = m(xx, rope=rope, residual=res)
            return [y.detach()] + (list(torch.autograd.grad(y, [xx, *m.parameters()], dy.to(y.dtype))) if train else [])

    got = run()
    monkeypatch.setattr(SafCausalSelfAttention, "_layer_call", lambda *a: None)
    want = run()
    assert rel(got[0], want[0]) <= FWD and got[0].dtype == want[0].dtype
    for a, b in zip(got[1:], want[1:]):
        # (q and k of one key have no gradient: both are rounding)
        assert a.dtype == b.dtype and (rel(a, b) <= BWD or (a.double() - b.double()).norm() <= 1e-3 * got[1].double().norm()), a.shape


@pytest.mark.parametrize("seed", range(16))
def test_grouped_module_and_block(seed, monkeypatch):
    from saf_b200.attention import rope_tables
    from saf_b200.gqa import SafGqaAttention, SafQwenBlock
    rng, g = random.Random(100 + seed), torch.Generator().manual_seed(seed)
    hd = rng.choice([64, 96, 128])
    kv = rng.choice([2, 4]) if hd == 96 else rng.randrange(1, 4)
    H = kv * rng.choice([1, 2, 3])
    hidden = rng.choice([H * hd, 192, 256, 448]) if H * hd % 64 == 0 else 256
    B, T = rng.randrange(1, 3), rng.choice([1, 100, 128, 257, 500])
    cfg = SimpleNamespace(hidden_size=hidden, num_attention_heads=H, num_key_value_heads=kv, head_dim=hd,
                          attention_bias=rng.random() < 0.5, intermediate_size=rng.choice([128, 384, 200]))
    block = rng.random() < 0.6
    m = SafQwenBlock(cfg) if block else SafGqaAttention(cfg)
    weights(m, seed)
    m = m.cuda().bfloat16().eval()
    freeze(rng, m.self_attn if block else m, H, T, g)
    rope = rope_tables(hd, T, base=1e6, device="cuda")
    x = inputs(rng, g, B, T, hidden, torch.bfloat16)
    kw = {} if block or rng.random() < 0.5 else dict(residual=torch.randn(B, T, hidden, generator=g).cuda().bfloat16())
    if block and cfg.intermediate_size % 64:
        m.mlp = m.mlp.to(torch.bfloat16)
    with torch.inference_mode():
        y = m(x, rope, **kw)
        monkeypatch.setattr(SafGqaAttention, "_layer_call", lambda *a: None)
        z = m(x, rope, **kw)
    assert rel(y, z) <= (3 * FWD if block else FWD)      # (a block: attention, MLP and result one after the other)


@pytest.mark.parametrize("seed", range(12))
def test_dense_block(seed, monkeypatch):
    from saf_b200.attention import SafCausalSelfAttention, rope_tables
    from saf_b200.block import SafBlock
    rng, g = random.Random(200 + seed), torch.Generator().manual_seed(seed)
    hd = rng.choice([64, 96, 128])
    H = rng.choice([2, 4]) if hd == 96 else rng.randrange(1, 5)
    B, T = rng.randrange(1, 3), rng.choice([1, 100, 128, 257, 500])
    cfg = SimpleNamespace(n_embd=H * hd, n_head=H, block_size=(T + 63) // 64 * 64, bias=rng.random() < 0.5, dropout=0.0,
                          position_encoding="rope", rand_attn_prior_repr="decomposed")
    m = SafBlock(cfg)
    weights(m, seed)
    m = m.cuda().bfloat16().eval()
    freeze(rng, m.main_block, H, T, g)
    cos, sin = rope_tables(hd, T, device="cuda")
    x = inputs(rng, g, B, T, H * hd, torch.bfloat16)
    with torch.inference_mode():
        y = m(x, rope=(cos.view(1, 1, T, hd), sin.view(1, 1, T, hd)))
        monkeypatch.setattr(SafCausalSelfAttention, "_layer_call", lambda *a: None)
        z = m(x, rope=(cos.view(1, 1, T, hd), sin.view(1, 1, T, hd)))
    assert rel(y, z) <= 3 * FWD
